"""Host side of the native ops: when an op may skip its autograd function."""
import os

import pytest
import torch
import torch.autograd.forward_ad as fwad

from mindspeed_mm_b200.models.qwen2_5_vl import DecoderLayer, LMHead, TextConfig
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


def _rules():
    """The rules of the kernels that are called without an autograd function, each on a call that it takes."""
    bf = lambda *s: torch.randn(*s).bfloat16()  # noqa: E731
    x, w, q, kv, old, tab = bf(2, 256), bf(64, 256), bf(1, 4, 128), bf(1, 2, 128), bf(9, 2, 128), bf(1, 128)
    return {"product": (lambda t: native.skinny_supported(t, w, None), x),
            "product, norm weight": (lambda t: native.skinny_supported(x, w, norm=t), bf(256)),
            "cached attention": (lambda t: native.decode_attention_supported(t, kv, kv, old, old, tab, tab), q),
            "cached attention, tables": (lambda t: native.decode_attention_supported(q, kv, kv, old, old, tab, t), tab),
            "rotary tables": (lambda t: native.mrope_tables_supported(t, 128, (16, 24, 24), torch.bfloat16), torch.arange(21).view(3, 7))}


@pytest.mark.parametrize("name", list(_rules()))
def test_kernels_called_without_an_autograd_function_ask_for_a_plain_call(name):
    rule, t = _rules()[name]
    assert rule(t)
    seen = []
    torch.func.vmap(lambda u: seen.append(rule(u)) or u)(torch.stack([t, t]))
    torch.jit.trace(lambda u: seen.append(rule(u)) or u + 0, (t,), check_trace=False)
    if t.is_floating_point():
        with fwad.dual_level():
            seen.append(rule(fwad.make_dual(t, t.clone())))
        seen.append(rule(t.clone().requires_grad_()))
        with torch.no_grad():
            assert rule(t.clone().requires_grad_())
    assert len(seen) >= 2 and not any(seen)


@pytest.mark.parametrize("name,role", [("fmha_bwd.cu", "// two warpgroups of 128 threads: both own all 128 query rows"),
                                       ("fmha_bwd_dkv128.cuh", "- row threads (warps 2..9)"), ("fmha_fwd_alt.cuh", "- softmax (warps 4..11)")])
def test_waits_in_front_of_whole_warp_instructions_are_voted(name, role):
    """A bounded wait may give up in some lanes of a warp only; these threads then run __syncwarp, votes and tensor-memory accesses
    of the whole warp, so every one of their waits has to be decided by the warp.  Read off the source: the waits cannot be made to fail."""
    with open(os.path.join(os.path.dirname(native.__file__), "csrc", name)) as f:
        text = f.read()
    begin = text.index(role)
    waits = [ln for ln in text[begin:text.index("atomicExch(p.status, MM_TIMEOUT_EPI)", begin)].splitlines() if "mbar_wait(" in ln]
    assert len(waits) >= 2 and all("__all_sync(0xffffffffu, mbar_wait(" in ln for ln in waits)


@pytest.mark.parametrize("M,K,norm,takes", [(1, 57344, True, True), (1, 57352, True, False), (1, 57352, False, True), (2, 38224, True, True),
                                            (2, 38232, True, False), (4, 20480, False, True), (4, 20488, False, False), (3, 27304, True, True),
                                            (3, 27312, True, False), (5, 64, False, False)])
def test_products_of_a_few_rows_that_fit_shared_memory(M, K, norm, takes):
    """M * K up to 80 K elements, and (M + 1) * K up to 112 K where a norm's weight is held beside x."""
    x, w = torch.zeros(M, K, dtype=torch.bfloat16), torch.zeros(16, K, dtype=torch.bfloat16)
    assert native.skinny_supported(x, w, norm=torch.zeros(K, dtype=torch.bfloat16) if norm else None) is takes


@pytest.mark.parametrize("name", ["input_layernorm", "post_attention_layernorm", "qkv_proj", "o_proj", "down_proj", "norm"])
@pytest.mark.parametrize("how", ["forward", "forward_hook", "pre_hook", "backward_hook", "adapter"])
def test_wrapped_modules_are_called_in_the_generation_path(name, how):
    """The generation path uses the weights of plain modules; one that something was attached to is called."""
    torch.manual_seed(0)
    c = TextConfig(num_layers=1, hidden_size=32, intermediate_size=64, num_attention_heads=4, num_key_value_heads=2, vocab_size=48)
    layer, head = DecoderLayer(c), LMHead(c)
    for p in (*layer.parameters(), *head.parameters()):
        torch.nn.init.normal_(p, std=0.1)
    owner, calls = (head, []) if name == "norm" else (layer, [])
    m = getattr(owner, name)
    if how == "forward":
        inner = m.forward
        m.forward = lambda *a, **k: calls.append(1) or inner(*a, **k)
    elif how == "forward_hook":
        m.register_forward_hook(lambda *a: calls.append(1))
    elif how == "pre_hook":
        m.register_forward_pre_hook(lambda *a: calls.append(1))
    elif how == "backward_hook":
        m.register_full_backward_hook(lambda *a: calls.append(1))
    else:
        class Adapter(type(m)):
            def forward(self, *a, **k):
                calls.append(1)
                return super().forward(*a, **k)
        m.__class__ = Adapter
    x = torch.randn(3, 32, requires_grad=True)
    y = head(x) if name == "norm" else layer(x, torch.ones(3, 8), torch.zeros(3, 8), None, None, cache={})
    y.sum().backward()
    assert calls


def test_four_rows_against_a_wide_weight_take_tiles():
    x = torch.zeros(4, 16, dtype=torch.bfloat16)
    takes = [native.skinny_supported(x[:m], torch.zeros(n, 16, dtype=torch.bfloat16)) for m, n in ((4, 18936), (4, 18944), (3, 18944))]
    assert takes == [True, False, True]


@pytest.mark.parametrize("name", ["rms_norm", "causal_conv1d", "gated_rms_norm"])
def test_backward_reads_the_layout_of_what_the_hooks_give_back(name, monkeypatch):
    """Columns of a wider matrix are saved as they lie; saved-tensor hooks (activations offloaded to the host) return dense copies.
    The pitch that the backward kernel gets has to be the one of the tensor it gets."""
    calls = {}

    class Fake:
        def __getattr__(self, fn):
            return lambda *a: calls.__setitem__(fn, a) or (1 if fn.endswith("_grid") else 0)
    monkeypatch.setattr(native, "lib", lambda: Fake())
    monkeypatch.setattr(native, "_st", lambda: 0)
    wide = torch.randn(6, 3 * 512).bfloat16()
    x, w = wide[:, 512:1024].detach().requires_grad_(), torch.randn(512).bfloat16()
    back, given = [], {}
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: back.append(t.clone(memory_format=torch.contiguous_format)) or back[-1]):
        if name == "rms_norm":
            y, ld = native.rms_norm(x, w), lambda a: (a[0], a[1])
        elif name == "causal_conv1d":
            y, ld = native.causal_conv1d(x, torch.randn(512, 4).bfloat16(), "silu", None), lambda a: (a[0], a[1])
        else:
            z = x.detach().view(6, 4, 128).requires_grad_()
            y, ld = native.gated_rms_norm(torch.randn(6, 4, 128).bfloat16(), z, torch.randn(128).bfloat16()), lambda a: (a[2], a[9] if len(a) == 12 else a[12])
        assert ld(next(a for fn, a in calls.items() if "_fwd" in fn))[1] == 3 * 512           # read in place
        y.backward(torch.ones_like(y))
    pointer, pitch = ld(next(a for fn, a in calls.items() if "_bwd" in fn and not fn.endswith("_grid")))
    assert any(t.data_ptr() == pointer for t in back) and pitch == 512


def test_a_tensor_brought_back_from_the_host_lives_until_its_readers_are_done(monkeypatch):
    """It is allocated on the copy stream; the allocator has to know the stream that reads it, or the next copy takes its memory."""
    import contextlib
    from mindspeed_mm_b200.runtime.features import ActivationOffload

    class Recorder:
        def __init__(self):
            self.calls = []

        def __getattr__(self, name):
            return lambda *a, **k: self.calls.append((name, a)) or self
    reader, host, off = Recorder(), Recorder(), ActivationOffload(enabled=False)
    off.h2d = Recorder()
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: reader)
    assert off._unpack(("host", host, None, "cuda")) is host and ("record_stream", (reader,)) in host.calls
