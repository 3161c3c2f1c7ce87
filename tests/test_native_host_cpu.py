"""Host side of the native ops: when an op may skip its autograd function."""
import torch
import torch.autograd.forward_ad as fwad

from mindspeed_mm_b200.ops import native


class _Double(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, k):
        ctx.save_for_backward(x)
        ctx.k = k
        return x * k

    @staticmethod
    def backward(ctx, g):
        return g * ctx.k, None


def test_only_calls_without_graph_transform_or_tracer_skip_the_autograd_function():
    x, p = torch.ones(3), torch.ones(3, requires_grad=True)
    assert native._keeps_no_graph((x, 2)) and not native._keeps_no_graph((p, 2))
    with torch.no_grad():
        assert native._keeps_no_graph((p, 2))
    seen = []
    torch.func.vmap(lambda t: seen.append(native._keeps_no_graph((t, 2))) or t)(x)
    with fwad.dual_level():
        seen.append(native._keeps_no_graph((fwad.make_dual(x, x), 2)))
    torch.jit.trace(lambda t: seen.append(native._keeps_no_graph((t, 2))) or t, (x,), check_trace=False)     # its check runs untraced
    assert seen and not any(seen)
    y = native._run(_Double, p, 2)
    assert torch.equal(torch.autograd.grad(y.sum(), p)[0], torch.full((3,), 2.0))
    assert torch.equal(native._run(_Double, x, 2), x * 2) and not native._run(_Double, x, 2).requires_grad
