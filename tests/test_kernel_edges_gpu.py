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
    assert float((a - b).norm()) <= rtol * float(b.norm()) + 1e-6


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
