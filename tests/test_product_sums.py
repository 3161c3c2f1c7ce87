"""Which blocks of a product are cut along K, and into how many parts: this is the order of an output's fp32 sum, and with it its bits."""
import os

import pytest
import torch

from mindspeed_mm_b200.ops import build, native

DEV = "cuda"


def _cut(M, N, K, bn, sms=148):
    """(blocks of 128 x bn in one go, parts of each of the others): what is shortest on tiles of 128 rows, one for each SM."""
    tiles, kb = -(-M // 128) * -(-N // bn), -(-K // 64)
    full, rem = divmod(tiles, sms)
    best, unit, operands = (tiles, 1), kb * 0.44 * bn / 256, 2.0 * K * (M + N) / 6.2e6
    least = max(unit * (full + 1), operands) - 4.0
    for parts in range(2, 17):
        if not rem or kb // parts < 4:
            break
        t = max(unit * full + unit * -(-rem * parts // sms) / parts, operands) + 6.0 + rem * parts * (128 * bn * 8e-6 / 4.0)
        if t < least:
            least, best = t, (tiles - rem, parts)
    return best


@pytest.mark.skipif(not os.path.exists(build.lib_path()), reason="the library is not built")
@pytest.mark.parametrize("N,K", [(4608, 3584), (3584, 3584), (37888, 3584), (3584, 18944), (3840, 1280), (1280, 3456), (6912, 1280), (1536, 8960), (200, 8192)])
def test_what_is_cut_depends_on_128_row_tiles_alone(N, K):
    """Rows from 5 to 9000, products of several models' layers: a prompt's logits move by more than a bf16 rounding where another rule cuts."""
    bn = 256 if N >= 256 else 128
    for M in [*range(5, 600, 7), *range(600, 4000, 31), *range(4000, 9000, 127)]:
        full, parts = _cut(M, N, K, bn)
        want = (-(-M // 128) * -(-N // bn) - full) * parts * 128 * bn * 4 if parts > 1 else 0
        assert native.lib().mm_gemm_ws_bytes(M, N, K, 0, 0, bn) == want, (M, N, K)


@pytest.mark.skipif(not os.path.exists(build.lib_path()), reason="the library is not built")
@pytest.mark.parametrize("T,V,H", [(513, 512, 256), (600, 152064, 3584), (2048, 152064, 3584), (8192, 152064, 3584), (1, 256, 256)])
def test_the_workspace_of_a_loss_is_bounded_by_its_products(T, V, H):
    """fp32 sums of 16 parts for each tile of 512 rows (256 columns), of at most eight rounds on half of the SMs; short main loops have fewer."""
    for M, N, K, b_mn in ((T, V, H, 0), (T, H, V, 1)):
        got = native.lib().mm_gemm_rows_ws_bytes(M, N, K, 0, b_mn)
        tiles, parts = -(-M // 512) * -(-N // 256), min(16, -(-K // 64) // 4)
        assert got <= 256 + 512 * 256 * 4 * (min(8 * 74, min(73, tiles) * parts) if parts > 1 else 0), (M, N, K)
        if T == 600:                        # (they are held one after the other) no more than a quarter of the logits, which are 182 MB
            assert got <= T * V * 2 // 4


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("M,N,K", [(136, 200, 8200), (405, 3584, 37888), (1421, 3584, 3600), (520, 9480, 4104), (2533, 5752, 6480), (2400, 32008, 5208), (4096, 4864, 2568),
                                   (3118, 3304, 3760), (2560, 3840, 18944), (17232, 4608, 18192), (1100, 3584, 3584)])
def test_blocks_are_cut_as_the_rule_says_on_every_tile(layout, M, N, K):
    """2^30 first, then ones, then -2^30: a sum in one go loses the ones (32 for 16 of K is under half an ulp at 2^30); in parts, each but the
    first keeps its own.  Tiles of 128, 256 and 512 rows, halves of the last, tiles with blocks of both kinds; all sums are exact."""
    kb = -(-K // 64)
    row = torch.zeros(K)
    row[0], row[64:(kb - 1) * 64], row[K - 1] = 2.0 ** 15, 1.0, -(2.0 ** 15)
    col = torch.zeros(K)
    col[0], col[64:(kb - 1) * 64], col[K - 1] = 2.0 ** 15, 2.0, 2.0 ** 15
    a, col_of_a = row.bfloat16().to(DEV).expand(M, K).contiguous(), row.bfloat16().to(DEV)[:, None]
    b = col.bfloat16().to(DEV).expand(N, K).contiguous()
    got = {"nt": lambda: native.gemm_nt(a, b), "nn": lambda: native.gemm_nn(a, b.t().contiguous()),
           "tn": lambda: native.gemm_tn(col_of_a.expand(K, -(-M // 8) * 8).contiguous()[:, :M], b.t().contiguous())}[layout]()
    native.check_status()
    bn = 256 if N >= 256 else 128
    full, parts = _cut(M, N, K, bn)
    m_blocks, n_blocks = -(-M // 128), -(-N // bn)
    want = torch.zeros(m_blocks, n_blocks)
    kept = 128.0 * (kb - 1 - kb // parts) if parts > 1 else 0.0
    for t in range(full, m_blocks * n_blocks):             # groups of 8 row blocks, column by column
        first = t // (8 * n_blocks) * 8
        rows, at = min(8, m_blocks - first), t - first * n_blocks
        want[first + at % rows, at // rows] = kept
    want = want.bfloat16().to(DEV).repeat_interleave(128, 0)[:M].repeat_interleave(bn, 1)[:, :N]
    assert torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("T,widths", [(1421, (3584, 3584, 4096, 3584)), (405, (3584, 4608, 3584, 1536)), (3118, (3760, 3304, 3760, 1024)), (2560, (8192, 3840, 1280, 3840))])
def test_products_behind_one_another_repeat_to_the_bit(T, widths):
    """Each starts while the one in front drains and reads what that one, or the sums of its split tail, has written: the same results as with a wait
    between them.  Tiles of 128, 256 and 512 rows, cut and not."""
    torch.manual_seed(T)
    x = torch.randn(T, widths[0], device=DEV).bfloat16()
    weights = [(torch.randn(n, k, device=DEV) * k ** -0.5).bfloat16() for k, n in zip(widths, widths[1:])]
    want = [x]
    for w in weights:
        want.append(native.gemm_nt(want[-1], w))
        torch.cuda.synchronize()
    same = torch.ones((), dtype=torch.bool, device=DEV)
    for _ in range(60):
        rows = [x]
        for w in weights:
            rows.append(native.gemm_nt(rows[-1], w))
        back = native.gemm_nn(native.gemm_nn(rows[-1], weights[-1]), weights[-2])
        for a, b in zip(rows, want):
            same &= (a == b).all()
        del rows, back
    native.check_status()
    assert bool(same)


@pytest.mark.gpu
@pytest.mark.parametrize("T,H,V,valid,chunk", [(1600, 1024, 18944, 1421, 8192), (700, 512, 4096, 65, 256), (513, 256, 512, 0, 8192), (300, 1024, 8192, 200, 8192)])
def test_a_loss_repeats_to_the_bit(T, H, V, valid, chunk):
    """Its chain of products over counted rows, softmax, gathers and sums, many times without a wait."""
    torch.manual_seed(T)
    h = torch.randn(T, H, device=DEV).bfloat16().requires_grad_()
    w = (0.02 * torch.randn(V, H, device=DEV)).bfloat16().requires_grad_()
    lab = torch.full((T,), -100, device=DEV)
    lab[torch.randperm(T, device=DEV)[:valid]] = torch.randint(0, V, (valid,), device=DEV)

    def once():
        loss = native.linear_cross_entropy(h, w, lab, -100, chunk)[0]
        return (loss.detach(), *torch.autograd.grad(loss, [h, w]))

    torch.cuda.synchronize()
    want = [t.clone() for t in once()]
    same = torch.ones((), dtype=torch.bool, device=DEV)
    for _ in range(40):
        for a, b in zip(once(), want):
            same &= (a == b).all()
    native.check_status()
    assert bool(same)
