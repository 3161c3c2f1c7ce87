"""Kernels at the sizes where they can go wrong: edges of tiles, remainders, empty parts, the ends of each dispatch rule."""
import pytest
import torch

from mindspeed_mm_b200 import ops  # noqa: F401
from mindspeed_mm_b200.ops import native
from mindspeed_mm_b200.ops import reference as ref  # noqa: F401

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _close(a, b, rtol, atol):
    a, b = a.float(), b.float()
    assert a.shape == b.shape and bool(torch.isfinite(a).all())
    err = float((a - b).abs().max())
    assert err <= atol + rtol * float(b.abs().max()), err
    # results that cancel (a gate's gradient is a sum of 128 rounded terms) keep the absolute error of their terms: a quarter of
    # the largest allowed one on average
    assert float((a - b).norm()) <= rtol * float(b.norm()) + 0.25 * atol * a.numel() ** 0.5


@pytest.mark.parametrize("T,k,E", [(0, 2, 3), (1, 1, 1), (1, 8, 8), (37, 2, 5), (128, 8, 9), (513, 8, 128), (4096, 3, 300), (341, 3, 300), (40000, 8, 7),
                                   (40000, 8, 513), (300, 2, 6000), (300, 2, 6001), (70, 1, 20000)])
@pytest.mark.parametrize("skew", [False, True])
def test_moe_routing_matches_a_stable_sort(T, k, E, skew):
    """One chunk of pairs and several, more chunks than threads of the scan, blocks of eight warps and of one; all pairs of one expert."""
    g = torch.Generator().manual_seed(T)
    ids = torch.randint(0, max(1, E - 2), (T, k), generator=g)               # the last experts stay empty where E > 2
    if skew:
        ids[:] = E // 2
    off, row_of_pair, src_of_row, R = (t.cpu() if torch.is_tensor(t) else t for t in native.aligned_routing(ids.to(DEV), E))
    flat = ids.reshape(-1)
    counts = torch.bincount(flat, minlength=E)
    start = torch.nn.functional.pad(((counts + 127) // 128 * 128).cumsum(0), (1, 0))
    order = torch.sort(flat, stable=True).indices
    rows = start[flat[order]] + torch.arange(T * k) - torch.nn.functional.pad(counts.cumsum(0), (1, 0))[flat[order]]
    want_row, want_src = torch.empty(T * k, dtype=torch.int64), torch.full((R,), -1)
    want_row[order], want_src[rows] = rows, order // k
    assert torch.equal(off.long(), start) and torch.equal(row_of_pair.long(), want_row) and torch.equal(src_of_row.long(), want_src)


def test_moe_routing_refuses_expert_numbers_out_of_range():
    for wrong in (-1, 4, 2 ** 40):
        for before in (0, 3000):
            ids = torch.zeros(before + 1, 2, dtype=torch.int64, device=DEV)
            ids[-1, 1] = wrong
            with pytest.raises(RuntimeError):
                native.aligned_routing(ids, 4)


@pytest.mark.parametrize("K,N", [(256, 128), (128, 256), (384, 512)])
def test_grouped_gemm_gradients_with_empty_experts(K, N):
    """Weight gradients of experts without rows are zero (written, not pre-set) in both tile widths."""
    counts = [0, 128, 0, 0, 256, 0]
    off = torch.nn.functional.pad(torch.tensor(counts).cumsum(0), (1, 0)).to(torch.int32).to(DEV)
    R = 512                                                                  # the last 128 rows belong to nobody
    torch.manual_seed(0)
    x, w = torch.randn(R, K, device=DEV).bfloat16().requires_grad_(), torch.randn(6, K, N, device=DEV).bfloat16().requires_grad_()
    dy = torch.randn(R, N, device=DEV).bfloat16()
    poison = [torch.full_like(w, float("nan")) for _ in range(4)]            # what the allocator hands out next
    del poison
    y = native._AlignedGroupedGemm.apply(x, w, off)
    dx, dw = torch.autograd.grad(y, [x, w], dy)
    a = 0
    for e, c in enumerate(counts):
        xe, ge, we = x[a:a + c].detach().float(), dy[a:a + c].float(), w[e].detach().float()
        if not c:
            assert not dw[e].any()
            continue
        _close(y[a:a + c].detach(), xe @ we, rtol=2e-2, atol=2e-2 * K ** 0.5)
        _close(dx[a:a + c], ge @ we.t(), rtol=2e-2, atol=2e-2 * N ** 0.5)
        _close(dw[e], xe.t() @ ge, rtol=2e-2, atol=2e-2 * c ** 0.5)
        a += c


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (1, 136, 264), (2, 4608, 3584), (3, 24, 1032), (4, 256, 18944), (1, 3584, 18944), (5, 136, 264),
                                   (4, 18816, 264), (4, 18944, 264), (3, 18944, 264), (4, 9344, 264), (4, 9472, 264)])
@pytest.mark.parametrize("norm,ends", [(False, "none"), (True, "bias"), (False, "residual"), (True, "swiglu")])
def test_product_of_a_few_rows(M, N, K, norm, ends):
    """Both sides of the 4-row rule (5 rows run on tiles, and 4 rows against 18944 or more weight rows, which SwiGLU has twice of);
    4 x 18944 is close to the most that the kernel takes."""
    torch.manual_seed(M * 1000 + N)
    x, g = torch.randn(M, K, device=DEV).bfloat16(), (1 + 0.1 * torch.randn(K, device=DEV)).bfloat16()
    n = 2 * N if ends == "swiglu" else N
    wide = torch.randn(n, K + 8, device=DEV).bfloat16() / K ** 0.5
    w, b, r = wide[:, :K], torch.randn(n, device=DEV).bfloat16(), torch.randn(M, N, device=DEV).bfloat16()       # rows with a pitch
    h = ref.rms_norm(x, g, 1e-6).float() if norm else x.float()
    want = h @ w.float().t()
    with torch.no_grad():
        if ends == "swiglu":
            got, want = ops.norm_linear_swiglu(x, g, 1e-6, w), ref.swiglu(want)
        elif ends == "residual":
            got, want = ops.linear_add(x, w, r), want + r.float()
        elif ends == "bias":
            got, want = ops.norm_linear(x, g, 1e-6, w, b), want + b.float()
        else:
            got = ops.linear(x, w)
    # operands are the same bf16 values (the normalised rows may round differently by one ulp), sums are fp32: half an ulp of bf16
    _close(got, want, rtol=8e-3, atol=4e-3)


@pytest.mark.parametrize("M,K", [(1, 12208), (1, 12216), (1, 12288), (1, 12296), (2, 8144), (2, 8192), (2, 8200), (3, 6144), (4, 4912), (1, 57344), (2, 38224),
                                 (1, 57352), (2, 38232), (4, 20488)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_normalised_rows_around_the_shared_memory_limits(M, K, swiglu):
    """x and the norm's weight in shared memory: up to, at and beyond the 48 KB that need no opt-in, and both sides of the most a
    block can have (beyond it the norm and the product run apart; rows over 8192 are normalised by PyTorch then)."""
    torch.manual_seed(K)
    x, g, w = torch.randn(M, K, device=DEV).bfloat16(), (1 + 0.1 * torch.randn(K, device=DEV)).bfloat16(), torch.randn(256, K, device=DEV).bfloat16() / K ** 0.5
    want = ref.rms_norm(x, g, 1e-6).float() @ w.float().t()
    with torch.no_grad():
        got = ops.norm_linear_swiglu(x, g, 1e-6, w) if swiglu else ops.norm_linear(x, g, 1e-6, w)
    _close(got, ref.swiglu(want) if swiglu else want, rtol=8e-3, atol=4e-3)


@pytest.mark.parametrize("start,pitch", [(1, 64), (2, 64), (3, 72), (8, 71)])
def test_residual_of_a_few_rows_may_start_anywhere(start, pitch):
    x, w, buf = torch.randn(2, 256, device=DEV).bfloat16(), torch.randn(64, 256, device=DEV).bfloat16() / 16, torch.randn(200, device=DEV).bfloat16()
    r = buf[start:].as_strided((2, 64), (pitch, 1))
    with torch.no_grad():
        _close(ops.linear_add(x, w, r), x.float() @ w.float().t() + r.float(), rtol=8e-3, atol=4e-3)


def test_product_of_a_few_rows_keeps_infinities_and_nan_to_their_outputs():
    x, w = torch.zeros(1, 272, device=DEV).bfloat16(), torch.ones(16, 272, device=DEV).bfloat16()
    x[0, -1], w[3, 5], w[4, 271] = float("inf"), float("nan"), -1
    with torch.no_grad():
        y = ops.linear(x, w)[0].float()
    assert y[3].isnan() and y[4] == float("-inf") and (y[:3] == float("inf")).all() and (y[5:] == float("inf")).all()


@pytest.mark.parametrize("T,past,Nq,Nkv", [(1, 0, 28, 4), (1, 1, 28, 4), (1, 15, 16, 16), (1, 127, 64, 4), (2, 128, 28, 4), (1, 129, 8, 8),
                                           (4, 500, 8, 2), (1, 2047, 28, 4), (1, 9000, 28, 4), (3, 16383, 5, 1), (16, 40, 2, 2), (17, 40, 2, 2)])
@pytest.mark.parametrize("rotate", [False, True])
def test_attention_over_the_cache(T, past, Nq, Nkv, rotate):
    """Every split of the keys over warps and CTAs, one to all rows of a tile, both sides of the 16-row rule."""
    torch.manual_seed(past + T)
    D = 128
    qkv = torch.randn(T, (Nq + 2 * Nkv) * D, device=DEV).bfloat16()
    q, k, v = (t.view(T, -1, D) for t in qkv.split([Nq * D, Nkv * D, Nkv * D], -1))
    ang = torch.rand(T, D // 2, device=DEV).repeat(1, 2) * 6
    cos, sin = (ang.cos().bfloat16(), ang.sin().bfloat16()) if rotate else (None, None)
    old = {n: torch.randn(past, Nkv, D, device=DEV).bfloat16() for n in "kv"} if past else {}
    cache = dict(old)
    with torch.no_grad():
        o = ops.attention_cached(q, k, v, cache, cos, sin)
    qr, kr = (ref.rope_rotate_half(t, cos, sin) if rotate else t for t in (q, k))
    keys, values = (torch.cat([old[n], t]) if past else t for n, t in (("k", kr), ("v", v)))
    assert torch.equal(cache["v"], values) and cache["k"].shape == keys.shape
    _close(cache["k"], keys, rtol=8e-3, atol=1e-6)                            # the rotation may round differently by one ulp
    assert not past or torch.equal(cache["k"][:past], old["k"])
    cu_q, cu_k = torch.tensor([0, T], device=DEV), torch.tensor([0, past + T], device=DEV)
    want = ref.attention_varlen(qr.float(), keys.float(), values.float(), cu_q, cu_k, True)
    _close(o, want, rtol=1e-2, atol=4e-3)                                     # probabilities and results are bf16


@pytest.mark.parametrize("lens,H,gate", [([1], 1, 0.5), ([63, 64, 65], 2, 0.5), ([128], 3, 0.0), ([17, 1, 127, 200], 2, 4.0), ([70, 5], 1, 60.0)])
def test_gated_delta_rule_on_bf16_tensors(lens, H, gate):
    """Both prologue kernels: chunks of 1 .. 64 tokens, no decay, decay that underflows within a chunk; all five gradients."""
    torch.manual_seed(sum(lens))
    T, K = sum(lens), 128
    cu = [0] + torch.tensor(lens).cumsum(0).tolist()
    unit = lambda: torch.nn.functional.normalize(torch.randn(T, H, K, device=DEV), dim=-1).bfloat16().requires_grad_()  # noqa: E731
    q, k, v = unit(), unit(), torch.randn(T, H, K, device=DEV).bfloat16().requires_grad_()
    g, beta = (-gate * torch.rand(T, H, device=DEV)).requires_grad_(), torch.rand(T, H, device=DEV).requires_grad_()
    do = torch.randn(T, H, K, device=DEV).bfloat16()
    o = ops.gated_delta_rule_varlen(q, k, v, g, beta, cu, chunk=64)
    got = torch.autograd.grad(o, [q, k, v, g, beta], do)
    leaf = [t.detach().float().requires_grad_() for t in (q, k, v, g, beta)]
    want = torch.cat([ref.gated_delta_rule_recurrent(*(t[None, a:b] for t in leaf))[0][0] for a, b in zip(cu[:-1], cu[1:])])
    want_g = torch.autograd.grad(want, leaf, do.float())
    # operands of the state walk and all bf16 results: 2^-9 each, a few of them in a row
    _close(o.detach(), want.detach(), rtol=2e-2, atol=2e-3)
    for a, b, t in zip(got, want_g, (q, k, v, g, beta)):
        assert a.dtype == t.dtype
        _close(a, b, rtol=2.5e-2, atol=4e-3)
    with torch.no_grad():
        assert torch.equal(ops.gated_delta_rule_varlen(q, k, v, g, beta, cu, chunk=64), o)
    with pytest.raises(RuntimeError):
        ops.gated_delta_rule_varlen(q, k, v, g, beta, [0, T + 1], chunk=64)


def test_decay_of_a_chunk_is_an_fp32_exponential():
    """Gates whose sums are exact in fp32: what is left is the exponential's own error, 2 ulp and not one that grows with the sum."""
    H, K, z = 64, 128, dict(dtype=torch.bfloat16, device=DEV)
    q = torch.nn.functional.normalize(torch.randn(64, H, K, device=DEV), dim=-1).bfloat16()
    g = (-torch.arange(1, H + 1, device=DEV, dtype=torch.float32) / 64).expand(64, H).contiguous()      # sums of -1 .. -64
    beta, first, count = torch.ones_like(g), torch.tensor([0], dtype=torch.int32, device=DEV), torch.tensor([64], dtype=torch.int32, device=DEV)
    W, Qg, Kd, U, At = *(torch.empty(H, 1, 64, K, **z) for _ in range(4)), torch.empty(H, 1, 64, 64, **z)
    gamma = torch.empty(H, 1, device=DEV)
    pointers = [t.data_ptr() for t in (q, q, q, g, beta, first, count, W, Qg, Kd, At, U, gamma)]
    assert native.lib().mm_gdn_prologue(*pointers, H, 1, 1.0, native._st()) == 0
    want = (-torch.arange(1, H + 1, device=DEV, dtype=torch.float64)).exp()
    assert float((gamma[:, 0].double() / want - 1).abs().max()) <= 2.5 * 2 ** -23


@pytest.mark.parametrize("lens_q,lens_k,nq,nkv,D,causal,grow", [
    ([1024], [1024], 2, 2, 128, False, False), ([1023], [1023], 2, 2, 128, False, False),       # both sides of the key-length rule
    ([1025], [1025], 4, 2, 80, False, True), ([4000, 129, 1], [4000, 129, 1], 2, 1, 72, False, True),
    ([100, 1], [2047, 3], 4, 4, 128, False, True), ([1500, 40], [900, 1700], 2, 2, 8, False, False),
    ([3072], [3072], 2, 2, 128, True, True), ([3071], [3071], 2, 2, 128, True, False), ([6200, 1], [6200, 1], 2, 1, 128, True, True),
    ([130, 3], [6143, 300], 7, 1, 128, True, False)])
def test_attention_over_long_keys(lens_q, lens_k, nq, nkv, D, causal, grow):
    """Alternating softmax groups: odd and even numbers of key tiles, a last tile of any width, sequences with a single tile, and
    scores that grow along the keys, so that the reference maximum moves and O is rescaled again and again."""
    torch.manual_seed(sum(lens_q) + sum(lens_k))
    Tq, Tk = sum(lens_q), sum(lens_k)
    q, k, v = (torch.randn(t, n, D, device=DEV).bfloat16() for t, n in ((Tq, nq), (Tk, nkv), (Tk, nkv)))
    if grow:
        q = q.abs()
        k = (k + torch.linspace(0.0, 40.0 / D ** 0.5, Tk, device=DEV)[:, None, None]).bfloat16()
    cu = [torch.tensor([0] + l, device=DEV).cumsum(0).to(torch.int32) for l in (lens_q, lens_k)]
    out, lse = native.fmha_forward(q, k, v, cu[0], cu[1], causal, D ** -0.5)
    want, want_lse = ref.attention_varlen(q.float(), k.float(), v.float(), cu[0].cpu(), cu[1].cpu(), causal, return_lse=True)
    native.check_status()
    _close(out, want, rtol=1e-2, atol=4e-3)               # probabilities and results are bf16
    assert float((lse - want_lse.reshape(lse.shape)).abs().max()) < 2e-3 * (1 + float(want_lse.abs().max()))


@pytest.mark.parametrize("rows,cols,pitch", [(1, 8, 8), (3, 264, 264), (33, 256, 512), (8192, 1280, 1280), (1000, 6912, 6920), (40000, 16, 16), (9, 8, 16),
                                             (5000, 24, 32), (777, 128, 128), (777, 136, 136), (65000, 248, 256)])
def test_column_sums(rows, cols, pitch):
    """One to 32 lanes a row, the last row of a lane's eight, columns of a wider matrix."""
    torch.manual_seed(rows)
    x = torch.randn(rows, pitch, device=DEV).bfloat16()[:, :cols]
    # fp32 sums rounded once to bf16
    _close(native.column_sum(x), x.double().sum(0), rtol=4e-3, atol=1e-3)


@pytest.mark.parametrize("B,S,H", [(1, 1, 8), (2, 7, 264), (1, 7800, 1536), (3, 100, 5120), (70000, 1, 264), (300, 7, 264), (300, 8, 264), (2, 0, 64), (0, 3, 64)])
def test_gated_residual_gradients(B, S, H):
    """Both sides of the rule for short batches (7 and 8 rows); a gate per token is 70000 batches; without rows its gradient is zero."""
    torch.manual_seed(S)
    x, y, do = (torch.randn(B, S, H, device=DEV).bfloat16().requires_grad_(i < 2) for i in range(3))
    gate = torch.randn(B, 1, H, device=DEV).bfloat16().requires_grad_()
    dx, dy, dg = torch.autograd.grad(ops.gated_residual(x, y, gate), [x, y, gate], do)
    assert torch.equal(dx, do) and torch.equal(dy, do * gate.detach())
    if not x.numel():
        assert dg.shape == gate.shape and not dg.any()
        return
    _close(dg, (do.double() * y.detach().double()).sum(1, keepdim=True), rtol=4e-3, atol=1e-3)


@pytest.mark.parametrize("n", [8, 16, 40, 4096 + 8])
@pytest.mark.parametrize("scale", [1.0, 1.0 / 3, float("inf")])
def test_scaling_in_place(n, scale):
    x = torch.randn(n, device=DEV).bfloat16()
    want = (x.float() * torch.tensor(scale, device=DEV)).bfloat16()
    s = torch.tensor([scale], device=DEV)
    assert native.lib().mm_scale_bf16(x.data_ptr(), n, s.data_ptr(), native._st()) == 0
    assert torch.equal(x, want)


def test_cross_entropy_refuses_a_second_backward():
    h, w = torch.randn(16, 64, device=DEV).bfloat16().requires_grad_(), torch.randn(256, 64, device=DEV).bfloat16().requires_grad_()
    loss, _ = ops.linear_cross_entropy(h, w, torch.arange(16, device=DEV))
    loss.backward(retain_graph=True)
    with pytest.raises(RuntimeError):
        loss.backward()


@pytest.mark.parametrize("T,H", [(1, 264), (5, 264), (300, 1536), (64, 3584), (7, 5120), (3, 8192)])
def test_rms_norm_of_columns_of_a_wider_matrix(T, H):
    """Rows that lie apart are normalised in place, with the gradients of a dense matrix."""
    torch.manual_seed(H)
    wide, w = torch.randn(T, 3 * H, device=DEV).bfloat16().requires_grad_(), (1 + 0.1 * torch.randn(H, device=DEV)).bfloat16().requires_grad_()
    dy = torch.randn(T, H, device=DEV).bfloat16()
    got = ops.rms_norm(wide[:, H:2 * H], w)
    dwide, dw = torch.autograd.grad(got, [wide, w], dy)
    dense = wide.detach()[:, H:2 * H].contiguous().requires_grad_()
    want = ops.rms_norm(dense, w)
    ddense, dw2 = torch.autograd.grad(want, [dense, w], dy)
    assert torch.equal(got, want) and torch.equal(dwide[:, H:2 * H], ddense) and torch.equal(dw, dw2)
    assert not dwide[:, :H].any() and not dwide[:, 2 * H:].any()


@pytest.mark.parametrize("B,S,H", [(2, 5, 64 * 8), (1, 777, 2048), (1, 40, 2056), (2, 33, 4104), (1, 3, 8192), (18, 32, 264), (19, 32, 264), (700, 2, 264)])
def test_layer_norm_modulate_gradients(B, S, H):
    """Each number of vectors per thread of the backward kernel; both folds of its partial sums, over 32 and 31 to one rows."""
    torch.manual_seed(H)
    x, sc, sh = torch.randn(B, S, H, device=DEV).bfloat16(), torch.randn(B, 1, H, device=DEV).bfloat16(), torch.randn(B, 1, H, device=DEV).bfloat16()
    dy = torch.randn(B, S, H, device=DEV).bfloat16()
    leaf = [t.clone().requires_grad_() for t in (x, sc, sh)]
    got = torch.autograd.grad(ops.layer_norm_modulate(*leaf), leaf, dy)
    leaf = [t.float().requires_grad_() for t in (x, sc, sh)]
    want = torch.autograd.grad(ref.layer_norm_modulate(*leaf), leaf, dy.float())
    for a, b in zip(got, want):
        _close(a, b, rtol=1e-2, atol=4e-3)


@pytest.mark.parametrize("lens,causal", [([64] * 9, False), ([1] * 300, False), ([127, 1, 128, 129, 0, 5, 300], False), ([1, 255, 257, 0, 128, 700], True),
                                         ([3] * 5000, False), ([2] * 4500, True)])
def test_attention_tile_lists(lens, causal):
    """Packed and plain tile lists: empty sequences, exact multiples of a tile, more sequences than the cached offsets."""
    torch.manual_seed(len(lens))
    T, D, N = sum(lens), 64, 2
    q, k, v = (torch.randn(T, N, D, device=DEV).bfloat16().requires_grad_() for _ in range(3))
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    do = torch.randn(T, N, D, device=DEV).bfloat16()
    o = ops.attention_varlen(q, k, v, cu, cu, max(lens), max(lens), causal=causal)
    got = torch.autograd.grad(o, [q, k, v], do)
    # one masked product over all tokens states the same
    seq = torch.repeat_interleave(torch.arange(len(lens), device=DEV), torch.tensor(lens, device=DEV))
    leaf = [t.detach().float().requires_grad_() for t in (q, k, v)]
    mask = seq[:, None] == seq[None]
    if causal:
        mask &= torch.arange(T, device=DEV)[:, None] >= torch.arange(T, device=DEV)[None]
    s = (torch.einsum("qnd,knd->nqk", leaf[0], leaf[1]) * D ** -0.5).masked_fill(~mask, float("-inf"))
    want = torch.einsum("nqk,knd->qnd", s.softmax(-1), leaf[2])
    _close(o.detach(), want.detach(), rtol=1e-2, atol=8e-3)
    for a, b in zip(got, torch.autograd.grad(want, leaf, do.float())):
        _close(a, b, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("D", [8, 24, 40, 80, 88, 120, 128])
@pytest.mark.parametrize("lens,nq,nkv,causal", [([1, 130, 257], 6, 2, True), ([300], 3, 3, False)])
def test_attention_gradients_of_narrow_heads(D, lens, nq, nkv, causal):
    """Depth steps of 16 that a head fills, half fills and does not have; row products and sums over a group's heads at odd row counts."""
    torch.manual_seed(D)
    T = sum(lens)
    q, k, v = (torch.randn(T, n, D, device=DEV).bfloat16().requires_grad_() for n in (nq, nkv, nkv))
    do = torch.randn(T, nq, D, device=DEV).bfloat16()
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    o = ops.attention_varlen(q, k, v, cu, cu, max(lens), max(lens), causal=causal)
    got = torch.autograd.grad(o, [q, k, v], do)
    leaf = [t.detach().float().requires_grad_() for t in (q, k, v)]
    seq = torch.repeat_interleave(torch.arange(len(lens), device=DEV), torch.tensor(lens, device=DEV))
    mask = seq[:, None] == seq[None]
    if causal:
        mask &= torch.arange(T, device=DEV)[:, None] >= torch.arange(T, device=DEV)[None]
    kk, vv = (t.repeat_interleave(nq // nkv, 1) for t in leaf[1:])
    s = (torch.einsum("qnd,knd->nqk", leaf[0], kk) * D ** -0.5).masked_fill(~mask, float("-inf"))
    want = torch.einsum("nqk,knd->qnd", s.softmax(-1), vv)
    _close(o.detach(), want.detach(), rtol=1e-2, atol=8e-3)
    for a, b in zip(got, torch.autograd.grad(want, leaf, do.float())):
        _close(a, b, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("M,N,K,splits", [(1421, 3584, 3600, True), (1409, 3592, 4104, True), (1, 264, 18952, None), (5, 8, 18944, True), (136, 520, 8200, True),
                                          (128 * 148, 256, 8192, False), (128 * 149, 256, 8192, True), (128, 256, 256, False), (85, 25368, 8200, False)])
def test_products_with_a_split_tail(layout, M, N, K, splits):
    """Ragged rows, columns and depths, a lone tail and one behind whole rounds; both sides of the rule (one row of tiles over a large
    weight is bound by its bytes and stays whole)."""
    if layout == "tn" and M % 8:
        M = M // 8 * 8 + 8                                        # the rows are the contiguous dimension there
    torch.manual_seed(M)
    a = torch.randn((K, M) if layout == "tn" else (M, K), device=DEV).bfloat16()
    b = torch.randn((N, K) if layout == "nt" else (K, N), device=DEV).bfloat16()
    bias = torch.randn(N, device=DEV).bfloat16() if layout == "nt" else None
    nbytes = native.lib().mm_gemm_ws_bytes(M, N, K, int(layout == "tn"), int(layout != "nt"), 256 if N >= 256 else 128)
    assert splits is None or (nbytes > 0) == splits
    got = {"nt": lambda: native.gemm_nt(a, b, bias), "nn": lambda: native.gemm_nn(a, b), "tn": lambda: native.gemm_tn(a, b)}[layout]()
    want = (a.float().t() if layout == "tn" else a.float()) @ (b.float().t() if layout == "nt" else b.float())
    if bias is not None:
        want += bias.float()
    native.check_status()
    # exact products, fp32 sums (of any order), one rounding to bf16: half an ulp, and the order's error at K = 18952
    _close(got, want, rtol=4.5e-3, atol=2e-3 * K ** 0.5 / 100)


@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("M,N,K,rows", [(128, 256, 64, 128), (136, 264, 8, 128), (256, 1000, 72, 128), (264, 9480, 320, 128), (4600, 3848, 328, 128),
                                        (264, 256, 384, 128), (264, 256, 392, 256), (384, 4096, 704, None),
                                        (520, 9480, 4104, None), (1000, 9472, 2056, 512), (4600, 3840, 4104, 512), (4096, 4864, 2568, 512),
                                        (2560, 3840, 18944, 512)])
def test_products_on_pairs_of_sms(layout, M, N, K, rows):
    """Tiles of one SM and of a pair, 256 and 512 rows: few rows, ragged rows, columns and depths, a main loop of fewer steps than the ring
    has slots, several tiles a pair, whole and cut along K; shallow products, which stay on one SM, at the ends of their staging's range."""
    torch.manual_seed(M + K)
    a = torch.randn((K, M) if layout == "tn" else (M, K), device=DEV).bfloat16()
    b = torch.randn((N, K) if layout == "nt" else (K, N), device=DEV).bfloat16()
    bias = torch.randn(N + 1, device=DEV).bfloat16()[K // 64 % 2:][:N] if layout == "nt" else None     # aligned and not
    if rows is not None:
        assert native.lib().mm_gemm_tile_rows(M, N, K, 256) == rows
    got = {"nt": lambda: native.gemm_nt(a, b, bias), "nn": lambda: native.gemm_nn(a, b), "tn": lambda: native.gemm_tn(a, b)}[layout]()
    want = (a.float().t() if layout == "tn" else a.float()) @ (b.float().t() if layout == "nt" else b.float())
    if bias is not None:
        want += bias.float()
    native.check_status()
    # exact products, fp32 sums (of any order), one rounding to bf16: half an ulp, and the order's error
    _close(got, want, rtol=4.5e-3, atol=2e-3 * K ** 0.5 / 100)


@pytest.mark.parametrize("T,nq,nk,D,pitch", [(1, 1, 1, 16, 0), (37, 4, 2, 80, 0), (130, 28, 4, 128, 8), (257, 16, 16, 80, 0), (3, 5, 1, 48, 16), (33, 2, 2, 72, 0),
                                             (65, 3, 3, 128, 4)])
@pytest.mark.parametrize("graph", [False, True])
def test_rotation_of_a_fused_projection(T, nq, nk, D, pitch, graph):
    """Heads whose half is a multiple of 8 and not, rows that lie apart (aligned and not), one token and one head: the separate
    rotations to the bit, gradients too; create_graph keeps the values' part differentiable."""
    torch.manual_seed(T)
    wide = torch.randn(T, (nq + 2 * nk) * D + pitch, device=DEV).bfloat16()
    qkv = wide[:, :(nq + 2 * nk) * D].detach().requires_grad_()
    ang = torch.randn(T, D, device=DEV)
    cos, sin = ang.cos().bfloat16(), ang.sin().bfloat16()
    outs = ops.split_rope(qkv, nq, nk, cos, sin)
    parts = [t.reshape(T, n, D) for t, n in zip(qkv.split([nq * D, nk * D, nk * D], 1), (nq, nk, nk))]
    want = [ops.rope_rotate_half(parts[0].contiguous(), cos, sin), ops.rope_rotate_half(parts[1].contiguous(), cos, sin), parts[2]]
    dys = [torch.randn_like(t).requires_grad_(graph) for t in want]
    got_g = torch.autograd.grad(outs, qkv, dys, create_graph=graph)[0]
    want_g = torch.autograd.grad(want, qkv, dys, create_graph=graph)[0]
    for a, b in zip((*outs, got_g), (*want, want_g)):
        assert torch.equal(a, b)
    if graph:
        assert torch.equal(torch.autograd.grad(got_g.float().sum(), dys[2])[0], torch.ones_like(dys[2]))
    with torch.no_grad():
        for a, b in zip(ops.split_rope(qkv, nq, nk, cos, sin), want):
            assert torch.equal(a, b)
    _close(outs[0].detach(), ref.rope_rotate_half(parts[0].detach(), cos, sin), rtol=4e-3, atol=1e-3)


@pytest.mark.parametrize("T,N,D", [(1, 1, 8), (77, 12, 128), (33, 3, 24)])
def test_interleaved_rotation(T, N, D):
    x = torch.randn(T, N, D, device=DEV).bfloat16().requires_grad_()
    ang = torch.randn(T, D // 2, device=DEV)
    y = ops.rope_interleaved(x, ang.cos(), ang.sin())
    dy = torch.randn_like(y)
    xr = x.detach().float().requires_grad_()
    yr = ref.rope_interleaved(xr, ang.cos(), ang.sin())
    _close(y.detach(), yr.detach(), rtol=4e-3, atol=1e-3)
    _close(torch.autograd.grad(y, x, dy)[0], torch.autograd.grad(yr, xr, dy.float())[0], rtol=4e-3, atol=1e-3)


@pytest.mark.parametrize("lens,D", [([512] * 16, 80), ([1564, 1276, 2048], 80), ([512] * 16, 128)])
def test_attention_backward_many_times_over(lens, D):
    """Back to back, so that a CTA's warps fall out of step now and then: the same gradients to the bit, and no wait that gives up."""
    torch.manual_seed(D)
    T, N = sum(lens), 16
    q, k, v, do = (torch.randn(T, N, D, device=DEV).bfloat16() for _ in range(4))
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    o, lse = native.fmha_forward(q, k, v, cu, cu, False, D ** -0.5)
    want = [t.clone() for t in native.fmha_backward(do, q, k, v, o, lse, cu, cu, False, D ** -0.5)]
    for _ in range(40):
        for _ in range(30):
            got = native.fmha_backward(do, q, k, v, o, lse, cu, cu, False, D ** -0.5)
        native.check_status()
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("T,H,V,valid,chunk", [(512, 256, 512, 100, 8192), (513, 256, 512, 0, 8192), (513, 264, 520, 513, 8192), (600, 256, 1000, 1, 8192),
                                               (700, 512, 4096, 64, 8192), (700, 512, 4096, 65, 256), (8300, 256, 512, 5000, 8192),
                                               (8300, 256, 512, 130, 4096), (1600, 3584, 18944, 1421, 8192)])
def test_loss_over_the_rows_with_a_target(T, H, V, valid, chunk):
    """No target at all, one, all; lists that end at and behind a step of 64 and in the first of several chunks, and a tail that is cut
    along K by the kernel's own plan.  Rows without a target get a gradient of exactly zero."""
    torch.manual_seed(T + valid)
    h = torch.randn(T, H, device=DEV).bfloat16().requires_grad_()
    w = (0.02 * torch.randn(V, H, device=DEV)).bfloat16().requires_grad_()
    lab = torch.full((T,), -100, device=DEV)
    use = torch.randperm(T, device=DEV)[:valid]
    lab[use] = torch.randint(0, V, (valid,), device=DEV)
    poison = [torch.full((T, max(H, V)), float("nan"), device=DEV, dtype=torch.bfloat16) for _ in range(3)]      # what the allocator hands out next
    del poison
    loss = native.linear_cross_entropy(h, w, lab, -100, chunk)[0]
    dh, dw = torch.autograd.grad(loss, [h, w])
    native.check_status()
    hr, wr = h.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    want = torch.nn.functional.cross_entropy(hr @ wr.t(), lab, reduction="sum", ignore_index=-100)
    eh, ew = torch.autograd.grad(want, [hr, wr])
    assert abs(float(loss) - float(want)) <= 2e-3 * abs(float(want)) + 1e-6
    assert not dh[lab == -100].any()
    # logits and their gradient are rounded to bf16 (2^-9 of each term), the sums to bf16 once more
    _close(dh, eh, rtol=2e-2, atol=1e-4)
    _close(dw, ew, rtol=2e-2, atol=2e-3 * max(valid, 1) ** 0.5)


@pytest.mark.parametrize("T,D,section,theta", [(1, 128, (16, 24, 24), 1e6), (77, 64, (8, 12, 12), 1e4), (3, 16, (2, 1, 1), 1e7), (5000, 128, (16, 24, 20), 1e6)])
def test_rotary_tables(T, D, section, theta):
    """Positions up to 130 000: the table is that of a 64-bit angle, rounded once."""
    pos = torch.randint(0, 130000, (3, T), device=DEV)
    cos, sin = ops.mrope_tables(pos, D, theta, section, torch.bfloat16)
    i = torch.arange(D // 2, device=DEV)
    axis = (i >= section[0]).long() + (i >= section[0] + section[1]).long()
    axis[i >= sum(section)] = 0
    ang = pos.double()[axis].t() * theta ** (-i.double() / (D // 2))
    ang = torch.cat([ang, ang], -1)
    # one rounding (two where the 64-bit value is rounded to 32 bits first)
    for got, want in ((cos, ang.cos()), (sin, ang.sin())):
        assert float((got.double() - want).abs().max()) <= 2 ** -9 + 1e-6


@pytest.mark.parametrize("T,hk,hv,dv", [(1, 1, 1, 8), (130, 2, 6, 128), (65, 16, 32, 128), (3, 3, 3, 72), (257, 1, 5, 24)])
def test_delta_heads(T, hk, hv, dv):
    """One head, odd repeats, values narrower than a warp's share: against the same steps in fp32."""
    torch.manual_seed(T)
    x = torch.randn(T, 2 * hk * 128 + hv * dv, device=DEV).bfloat16()
    x[0, :128] = 0                                                # a row without a norm
    x.requires_grad_()
    leaf = x.detach().float().requires_grad_()
    assert native.delta_heads_supported(x, hk, hv, 128, dv)
    got = ops.delta_heads(x, hk, hv, 128, dv)
    rows = ref.l2_norm(leaf[:, :2 * hk * 128].reshape(T, 2, hk, 128)).repeat_interleave(hv // hk, dim=2)
    want = (rows[:, 0], rows[:, 1], leaf[:, 2 * hk * 128:].reshape(T, hv, dv))
    for a, b in zip(got, want):
        _close(a.detach(), b.detach(), rtol=2 ** -8, atol=0)      # one rounding to bf16
    do = [torch.randn_like(t) for t in got]
    do[0][0] = 0                                                  # (its gradient is 1000 times the others')
    (a,), (b,) = torch.autograd.grad(got, [x], do), torch.autograd.grad(want, [leaf], [t.float() for t in do])
    # one rounding of the result; y is read rounded: 2^-9 of |g| |y| over the row's norm
    _close(a, b, rtol=2 ** -7, atol=0)


@pytest.mark.parametrize("T,D,extra", [(1, 8, 0), (1, 64, 3), (1, 264, 8), (70, 264, 8), (33, 1032, 24), (129, 64, 3)])
def test_convolution_and_gate_on_columns_of_a_wider_matrix(T, D, extra):
    """Columns read in place (and copied where their pitch or their start does not allow it) give what dense ones give."""
    torch.manual_seed(T)
    wide = torch.randn(T, D + extra, device=DEV).bfloat16()
    cu = torch.tensor([0, T // 3, T], device=DEV)
    w = torch.randn(D, 4, device=DEV).bfloat16()
    for lo in sorted({0, extra // 2, extra}):
        outs = []
        for x in (wide[:, lo:lo + D], wide[:, lo:lo + D].clone()):
            x = x.detach().requires_grad_()
            y = ops.causal_conv1d(x, w, None, "silu", cu)
            outs.append([y.detach(), *torch.autograd.grad(y, [x], torch.ones_like(y))])
            z = x.detach().view(T, -1, 8).requires_grad_()
            o = torch.linspace(-2, 2, T * D, device=DEV).bfloat16().view(T, -1, 8)
            y = ops.gated_rms_norm(o, z, w.view(-1)[:8])
            outs[-1] += [y.detach(), *torch.autograd.grad(y, [z], torch.ones_like(y))]
        assert all(torch.equal(a, b) for a, b in zip(*outs))


@pytest.mark.parametrize("lens,D,K,silu", [([1], 8, 1, True), ([100, 27], 136, 8, True), ([31, 1, 0, 97], 264, 2, False), ([129, 2, 169], 72, 5, True),
                                           ([32] * 5, 128, 4, True)])
def test_convolution_backward_at_strip_edges(lens, D, K, silu):
    """Strips of 32 tokens, four a block, 128 channels a warp: short tails, sequences that end at and around the edges, every K."""
    torch.manual_seed(K)
    T = sum(lens)
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0)
    x, dy = (torch.randn(T, D, device=DEV).bfloat16() for _ in range(2))
    w = torch.randn(D, K, device=DEV).bfloat16()
    leaf, want = [], []
    for cast, f in ((lambda t: t, ops.causal_conv1d), (lambda t: t.float(), ref.causal_conv1d)):
        leaf = [cast(t).detach().requires_grad_() for t in (x, w)]
        y = f(*leaf, None, "silu" if silu else None, cu if cast(x) is x else cu.unique().tolist())     # (the oracle takes no empty sequence)
        want.append(torch.autograd.grad(y, leaf, cast(dy)))
    for a, b in zip(*want):
        _close(a, b, rtol=2 ** -8, atol=1e-5)                     # fp32 sums, one rounding to bf16


@pytest.mark.parametrize("T,h", [(0, 4), (5, 0), (0, 0)])
def test_gate_without_rows(T, h):
    """No tokens or no heads: nothing to do, forward and backward."""
    x, z = (torch.randn(T, h, 64, device=DEV).bfloat16().requires_grad_() for _ in range(2))
    y = ops.gated_rms_norm(x, z, torch.ones(64, device=DEV).bfloat16())
    dx, dz = torch.autograd.grad(y, [x, z], torch.ones_like(y))
    assert y.shape == dx.shape == dz.shape == (T, h, 64)


@pytest.mark.parametrize("name", ["product", "attention", "tables", "experts", "swiglu"])
def test_a_recorded_trace_computes_again(name):
    """A trace of a call that keeps no graph runs the kernels on the inputs of its replay."""
    bf = lambda *s: torch.randn(*s, device=DEV).bfloat16()  # noqa: E731
    w, g, gate_up, down, tab, probs = bf(64, 256), bf(256), bf(4, 256, 512) / 16, bf(4, 256, 256) / 16, bf(1, 128), torch.rand(64, 2, device=DEV).bfloat16()
    f, make = {"product": (lambda x: ops.norm_linear(x, g, 1e-6, w), lambda: (bf(2, 256),)),
               "attention": (lambda q, k, v: ops.attention_cached(q, k, v, {}, tab, tab), lambda: (bf(1, 4, 128), bf(1, 2, 128), bf(1, 2, 128))),
               "tables": (lambda p: ops.mrope_tables(p, 128, 1e6, (16, 24, 24), torch.bfloat16)[0], lambda: (torch.randint(0, 99, (3, 7), device=DEV),)),
               "experts": (lambda x, i: native.moe_experts(x, i, probs, gate_up, down), lambda: (bf(64, 256), torch.randint(0, 4, (64, 2), device=DEV))),
               "swiglu": (lambda x: ops.linear_swiglu(x, gate_up[0]), lambda: (bf(8, 512),))}[name]
    with torch.no_grad():
        m, args = torch.jit.trace(f, make(), check_trace=False), make()
        # the tables' general path computes its angles in 32 bits
        _close(m(*args), f(*args), rtol=8e-3, atol=4e-3)


def test_forward_mode_is_refused_where_no_rule_for_it_exists():
    with torch.autograd.forward_ad.dual_level(), pytest.raises(NotImplementedError):
        x = torch.autograd.forward_ad.make_dual(torch.randn(1, 256, device=DEV).bfloat16(), torch.randn(1, 256, device=DEV).bfloat16())
        ops.norm_linear(x, torch.ones(256, device=DEV).bfloat16(), 1e-6, torch.randn(64, 256, device=DEV).bfloat16())


@pytest.mark.parametrize("n", [1, 31, 32, 33, 257, 4096, 4097])
@pytest.mark.parametrize("longest", [1, 300, 2000])
def test_tile_lists_name_every_tile_once_longest_first(n, longest):
    """The list as the planner writes it: one to all positions kept by ballot, both places where the sequences left are kept."""
    g = torch.Generator().manual_seed(n + longest)
    lens = torch.randint(0, longest + 1, (n,), generator=g) * (torch.rand(n, generator=g) < 0.7)
    if longest == 2000 and n > 300:
        lens[60:] = lens[60:] % 130                                          # a few long ones among many short ones
    lens[0] = longest
    T, cu = int(lens.sum()), torch.nn.functional.pad(lens.cumsum(0), (1, 0)).to(torch.int32).to(DEV)
    L, q = native.lib(), torch.randn(T, 1, 8, device=DEV).bfloat16()
    most = L.mm_fmha_max_tiles(T, n)
    plan, o, lse = torch.full((3 * most + 1,), -1, dtype=torch.int32, device=DEV), torch.empty_like(q), torch.empty(1, T, device=DEV)
    assert L.mm_fmha_fwd(q.data_ptr(), q.data_ptr(), q.data_ptr(), o.data_ptr(), lse.data_ptr(), cu.data_ptr(), cu.data_ptr(), plan.data_ptr(), T, T, n, 1, 1,
                         8, 8, 8, 8, 1, 1.0, native.status_word(q.device).data_ptr(), native._st()) == 0
    native.check_status()
    count = int(plan[2 * most])
    seq, row = plan[:count].tolist(), plan[most:most + count].tolist()
    assert sorted(zip(seq, row)) == [(b, r) for b, l in enumerate(lens.tolist()) for r in range(0, l, 128)]
    assert row == sorted(row, reverse=True) and set(plan[2 * most + 1:2 * most + 1 + count].tolist()) == {1}


def test_planning_many_short_sequences_takes_no_longer_than_their_attention_by_orders():
    """4096 causal sequences of 2: 0.6 ms on one thread, 41 ms where each tile counted the tiles of every sequence."""
    q, cu = torch.randn(8192, 2, 64, device=DEV).bfloat16(), torch.arange(0, 8193, 2, dtype=torch.int32, device=DEV)
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    native.fmha_forward(q, q, q, cu, cu, True, 0.125)
    a.record()
    native.fmha_forward(q, q, q, cu, cu, True, 0.125)
    b.record()
    torch.cuda.synchronize()
    assert a.elapsed_time(b) < 5


@pytest.mark.parametrize("name", ["bias", "loss", "unpermute", "gate"])
def test_gradients_that_are_linear_in_the_incoming_one_can_be_differentiated(name):
    """create_graph: the derivative of a gradient by a factor in front of the op's result is the gradient itself."""
    bf = lambda *s: torch.randn(*s, device=DEV).bfloat16().requires_grad_()  # noqa: E731
    s = torch.ones((), device=DEV, requires_grad=True)
    x, w, b, h, vocab, y, gate = bf(16, 64), bf(32, 64), bf(32), bf(16, 64), bf(256, 64), bf(128, 64), bf(2, 1, 64)
    probs, rows = torch.rand(64, 2, device=DEV).bfloat16().requires_grad_(), torch.arange(128, device=DEV, dtype=torch.int32).flip(0)
    c = torch.randn(8192, device=DEV)
    out, leaves = {"bias": lambda: (ops.linear(x, w, b), [b]), "loss": lambda: (ops.linear_cross_entropy(h, vocab, torch.arange(16, device=DEV))[0], [h, vocab]),
                   "unpermute": lambda: (native._AlignedUnpermute.apply(y, rows, probs), [y, probs]),
                   "gate": lambda: (ops.gated_residual(y.view(2, 64, 64), y.view(2, 64, 64), gate), [gate])}[name]()
    plain = torch.autograd.grad((out.float().view(-1) * c[:out.numel()] if out.dim() else out * 1.0).sum(), leaves, retain_graph=name != "loss")
    if name == "loss":                       # its gradients are scaled in place: once per forward
        out = ops.linear_cross_entropy(h, vocab, torch.arange(16, device=DEV))[0]
    grads = torch.autograd.grad((out.float().view(-1) * c[:out.numel()] * s if out.dim() else out * s).sum(), leaves, create_graph=True)
    for a, g in zip(plain, grads):
        _close(g.detach(), a, rtol=8e-3, atol=4e-3)
        v = torch.randn_like(g)
        (ds,) = torch.autograd.grad(g, [s], v, retain_graph=True)
        want = (a.float() * v.float()).sum()
        assert float((ds - want).abs()) <= 2e-2 * float((a.float() * v.float()).norm()) + 1e-3


@pytest.mark.parametrize("lens_q,lens_k,causal", [([400], [100], True), ([10, 300, 10], [0, 300, 7], False), ([10, 300], [0, 4000], False),
                                                  ([4000, 10], [3500, 3500], True)])
@pytest.mark.parametrize("D", [72, 128])
def test_rows_that_see_no_key_are_zero(lens_q, lens_k, causal, D):
    """Whole tiles of them, too, in both forward kernels; their gradients are zero."""
    torch.manual_seed(sum(lens_q))
    q, k, v = (torch.randn(sum(t), 2, D, device=DEV).bfloat16().requires_grad_() for t in (lens_q, lens_k, lens_k))
    cu = [torch.tensor([0] + l, device=DEV).cumsum(0).to(torch.int32) for l in (lens_q, lens_k)]
    poison = [torch.full((sum(lens_q), 2, 128), float("nan"), device=DEV) for _ in range(4)]       # what the allocator hands out next
    del poison
    out, lse = native.fmha_forward(q.detach(), k.detach(), v.detach(), *cu, causal, D ** -0.5)
    want, want_lse = ref.attention_varlen(q.detach().float(), k.detach().float(), v.detach().float(), cu[0].cpu(), cu[1].cpu(), causal, return_lse=True)
    hidden = want_lse[0] == float("-inf")
    assert hidden.any() and torch.equal(lse == float("-inf"), want_lse == float("-inf")) and not out[hidden].any()
    _close(out[~hidden], want[~hidden], rtol=1e-2, atol=4e-3)
    o = ops.attention_varlen(q, k, v, *cu, max(lens_q), max(lens_k), causal=causal)
    dq, dk, dv = torch.autograd.grad(o, [q, k, v], torch.randn_like(o))
    native.check_status()
    assert not dq[hidden].any() and all(bool(t.isfinite().all()) for t in (dq, dk, dv))


@pytest.mark.parametrize("T,H", [(1, 64), (1, 264), (1, 3584), (3, 264)])
@pytest.mark.parametrize("start", [1, 3, 8])
def test_rms_norm_of_rows_that_start_anywhere(T, H, start):
    """A single row is contiguous wherever it starts; so is what a gradient may be a view of."""
    x, w, dy = (torch.randn(T * H + start, device=DEV).bfloat16()[start:].view(T, H) for _ in range(3))
    outs = []
    for a, b, g in ((x, w[0], dy), (x.clone(), w[0].clone(), dy.clone())):
        a, b = a.detach().requires_grad_(), b.detach().requires_grad_()
        y = ops.rms_norm(a, b)
        outs.append([y.detach(), *torch.autograd.grad(y, [a, b], g)])
    assert all(torch.equal(p, q) for p, q in zip(*outs))


def test_columns_of_a_wider_matrix_offloaded_to_the_host_and_back():
    """What is saved where it lies comes back dense; the gradients stay the same."""
    from mindspeed_mm_b200.runtime.features import ActivationOffload
    wide, w, cw, o = (torch.randn(*s, device=DEV).bfloat16() for s in ((33, 1536), (512,), (512, 4), (33, 4, 128)))
    outs = []
    for enabled in (False, True):
        x = wide[:, 512:1024].detach().requires_grad_()
        with ActivationOffload(enabled=enabled, min_bytes=0) as a:
            ys = [ops.rms_norm(x, w), ops.causal_conv1d(x, cw, None, "silu", None), ops.gated_rms_norm(o, x.view(33, 4, 128), w[:128])]
        assert (a.bytes_offloaded > 0) == enabled
        outs.append([g for y in ys for g in torch.autograd.grad(y, [x], torch.ones_like(y))])
    assert all(torch.equal(p, q) for p, q in zip(*outs))


def test_delta_rule_gradients_keep_a_graph_where_they_had_one():
    """create_graph: through the prologue of the delta rule, and through the values of its heads."""
    torch.manual_seed(0)
    T, H, cu = 130, 2, [0, 70, 130]
    unit = lambda: torch.nn.functional.normalize(torch.randn(T, H, 128, device=DEV), dim=-1).bfloat16().requires_grad_()  # noqa: E731
    leaves = [unit(), unit(), torch.randn(T, H, 128, device=DEV).bfloat16().requires_grad_(), (-torch.rand(T, H, device=DEV)).requires_grad_(),
              torch.rand(T, H, device=DEV).requires_grad_()]
    do = torch.randn(T, H, 128, device=DEV).bfloat16()
    plain = torch.autograd.grad(ops.gated_delta_rule_varlen(*leaves, cu, chunk=64), leaves, do)
    grads = torch.autograd.grad(ops.gated_delta_rule_varlen(*leaves, cu, chunk=64), leaves, do, create_graph=True)
    for a, b in zip(grads, plain):
        assert a.requires_grad and a.dtype == b.dtype
        _close(a.detach(), b, rtol=2.5e-2, atol=4e-3)
    (some,) = torch.autograd.grad(ops.gated_delta_rule_varlen(*leaves, cu, chunk=64), leaves[2:3], do, create_graph=True)
    assert some.requires_grad
    x, s = torch.randn(5, 384, device=DEV).bfloat16().requires_grad_(), torch.ones((), device=DEV, requires_grad=True)
    (dx,) = torch.autograd.grad((ops.delta_heads(x, 1, 1, 128, 128)[2].float() * s).sum(), [x], create_graph=True)
    assert float(torch.autograd.grad(dx.float().sum(), [s])[0]) == 5 * 128


@pytest.mark.parametrize("T,nq,nk,D", [(1, 1, 1, 16), (37, 4, 2, 80), (33, 2, 2, 72), (65, 3, 3, 128)])
def test_gradients_of_a_rotation_can_be_differentiated(T, nq, nk, D):
    """create_graph: a rotation's gradient is linear in the incoming one, so its derivative by that is the rotation itself, to the bit; the
    derivative after that is the gradient again."""
    torch.manual_seed(T)
    ang = torch.randn(T, D, device=DEV)
    cos, sin, half_cos, half_sin = ang.cos().bfloat16(), ang.sin().bfloat16(), ang[:, :D // 2].cos().contiguous(), ang[:, :D // 2].sin().contiguous()
    bf = lambda *s: torch.randn(*s, device=DEV).bfloat16()  # noqa: E731
    width = (nq + 2 * nk) * D
    for op, shape in ((lambda t: ops.split_rope(t, nq, nk, cos, sin), (T, width)), (lambda t: (ops.rope_rotate_half(t, cos, sin),), (T, nq, D)),
                      (lambda t: (ops.rope_interleaved(t, half_cos, half_sin),), (T, nq, D))):
        x, r = bf(*shape).requires_grad_(), bf(*shape)
        outs = op(x)
        dys = [bf(*o.shape).requires_grad_() for o in outs]
        (g,) = torch.autograd.grad(outs, x, dys, create_graph=True)
        seconds = torch.autograd.grad(g, dys, r.requires_grad_(), create_graph=True)
        for a, b in zip(seconds, op(r.detach())):
            assert torch.equal(a, b)
        (third,) = torch.autograd.grad(seconds, r, [d.detach() for d in dys])
        assert torch.equal(third, g)
