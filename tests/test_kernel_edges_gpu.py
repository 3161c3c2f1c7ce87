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


@pytest.mark.parametrize("T,k,E", [(1, 1, 1), (1, 8, 8), (37, 2, 5), (513, 8, 128), (4096, 3, 300)])
def test_moe_routing_matches_a_stable_sort(T, k, E):
    g = torch.Generator().manual_seed(T)
    ids = torch.randint(0, max(1, E - 2), (T, k), generator=g)               # the last experts stay empty where E > 2
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
    for wrong in (-1, 4):
        with pytest.raises(RuntimeError):
            native.aligned_routing(torch.tensor([[0, wrong]], device=DEV), 4)


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


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (1, 136, 264), (2, 4608, 3584), (3, 24, 1032), (4, 256, 18944), (1, 3584, 18944), (5, 136, 264)])
@pytest.mark.parametrize("norm,ends", [(False, "none"), (True, "bias"), (False, "residual"), (True, "swiglu")])
def test_product_of_a_few_rows(M, N, K, norm, ends):
    """Both sides of the 4-row rule (5 rows and a 4 x 18944 operand beyond the shared-memory bound run on tiles)."""
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
