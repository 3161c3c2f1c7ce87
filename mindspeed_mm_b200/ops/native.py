"""ctypes bindings and autograd wrappers for the sm_100a kernels in ``csrc/``.

The library is loaded from ``ops/_lib/libmm_b200_ops.so`` (built in-tree by ``ops/build.py``).  On a
GPU box a missing or stale library is an error, never a silent fallback.  Kernels take raw device
pointers and the current CUDA stream; tensors are kept alive by the autograd contexts / callers.
"""
from __future__ import annotations

import ctypes as C
import math
import os
from typing import Optional

import torch

from . import build as _build

_LIB = None
_STATUS: dict = {}
# forward attention kernel: 3 (default) = by key length, alternating softmax groups (csrc/fmha_fwd_alt.cuh) for long keys, else
# split softmax (csrc/fmha_fwd_split.cuh), both with O in tensor memory and lazy rescaling; 2 = always split softmax;
# 0 = one softmax warpgroup, O folded in registers (csrc/fmha_fwd.cu, fallback)
FMHA_FWD_VARIANT = int(os.environ.get("MM_B200_FMHA_FWD_VARIANT", "3"))
LAUNCHES = 0  # native kernel launches issued through this module (bench reports it)

_p, _i, _ll, _f = C.c_void_p, C.c_int, C.c_longlong, C.c_float


def lib():
    global _LIB
    if _LIB is None:
        path = _build.lib_path()
        if not os.path.exists(path):
            raise RuntimeError(f"native op library not built: {path} (run python -m mindspeed_mm_b200.ops.build)")
        _LIB = C.CDLL(path)
        _declare(_LIB)
        _LIB.mm_fmha_set_fwd_variant(FMHA_FWD_VARIANT)
    return _LIB


# Row norms: rows of up to 256 elements (per-head q/k norms, L2 norm of GDN heads) take a lane group per row
# (csrc/rownorm.cu: 0.94 of the copy bandwidth against 0.45 for a block per row); longer rows keep a block per row
# (csrc/elementwise.cu), which measured faster there (0.67 against 0.45 at 3584).
def _row_group(H: int) -> bool:
    return H <= 256 and H % 8 == 0


def _declare(L):
    sig = {
        "mm_rmsnorm_fwd_ld": [_p, _ll, _p, _p, _p, _i, _i, _f, _p],
        "mm_rmsnorm_bwd_ld": [_p, _ll, _p, _p, _p, _p, _p, _p, _i, _i, _p],
        "mm_column_splits": [_i, _i, _i, _i],
        "mm_column_sum": [_p, _p, _p, _i, _i, _ll, _p],
        "mm_gated_residual_bwd": [_p, _p, _p, _p, _p, _p, _i, _i, _i, _p],
        "mm_scale_bf16": [_p, _ll, _p, _p],
        "mm_rmsnorm_fwd": [_p, _p, _p, _p, _i, _i, _f, _p],
        "mm_rownorm_rms_fwd": [_p, _p, _p, _p, _ll, _i, _f, _p],
        "mm_rownorm_ln_mod_fwd": [_p, _p, _p, _p, _p, _p, _ll, _i, _i, _f, _p],
        "mm_rownorm_l2_fwd": [_p, _p, _p, _ll, _i, _f, _p],
        "mm_gated_rms_fwd": [_p, _i, _p, _p, _p, _p, _ll, _i, _i, _ll, _f, _p],
        "mm_gated_rms_bwd": [_p, _i, _p, _p, _p, _p, _p, _p, _p, _ll, _i, _i, _ll, _p],
        "mm_rmsnorm_bwd_grid": [_i],
        "mm_sq_norm_blocks": [],
        "mm_rmsnorm_set_v16": [_i],
        "mm_sq_norm": [_p, _ll, _p, _p],
        "mm_rmsnorm_bwd": [_p, _p, _p, _p, _p, _p, _p, _i, _i, _p],
        "mm_swiglu_fwd": [_p, _p, _ll, _i, _p],
        "mm_swiglu_bwd": [_p, _p, _p, _ll, _i, _p],
        "mm_gelu_fwd": [_p, _p, _ll, _i, _p],
        "mm_gelu_bwd": [_p, _p, _p, _ll, _i, _p],
        "mm_rope_half": [_p, _ll, _p, _p, _p, _i, _i, _i, _i, _p],
        "mm_rope_qkv": [_p, _ll, _p, _ll, _p, _ll, _p, _p, _p, _ll, _p, _ll, _p, _ll, _i, _i, _i, _i, _i, _i, _p],
        "mm_rope_interleaved": [_p, _ll, _p, _p, _p, _i, _i, _i, _i, _p],
        "mm_ln_mod_fwd": [_p, _p, _p, _p, _p, _p, _i, _i, _i, _f, _p],
        "mm_ln_mod_bwd_ctas": [_i, _i],
        "mm_ln_mod_bwd": [_p, _p, _p, _p, _p, _p, _p, _p, _p, _i, _i, _i, _p],
        "mm_gated_residual": [_p, _p, _p, _p, _ll, _i, _i, _p],
        "mm_adamw": [_p, _p, _p, _p, _i, _p, _ll, _ll, _f, _f, _f, _f, _f, _f, _f, _f, _p, _p],
        "mm_gemm_bf16_ws": [_p, _p, _p, _p, _i, _i, _i, _ll, _ll, _ll, _i, _i, _i, _p, _p, _ll, _p],
        "mm_gemm_ws_bytes": [_i, _i, _i, _i, _i, _i],
        "mm_gemm_tile_rows": [_i, _i, _i, _i],
        "mm_gemm_rows_ws_bytes": [_i, _i, _i, _i, _i],
        "mm_gemm_bf16_rows": [_p, _p, _p, _i, _i, _i, _ll, _ll, _ll, _i, _i, _p, _i, _p, _p, _ll, _p],
        "mm_gemm_swiglu_bf16": [_p, _p, _p, _i, _i, _i, _ll, _ll, _ll, _p, _p],
        "mm_gemv_bf16": [_p, _p, _p, _p, _p, _p, _i, _i, _i, _ll, _ll, _ll, _ll, _f, _i, _p],
        "mm_rotary_tables": [_p, _p, _p, _i, _i, _i, _i, _i, C.c_double, _p],
        "mm_decode_attention": [_p, _p, _p, _p, _p, _p, _p, _p, _p, _p, _i, _i, _i, _i, _ll, _ll, _ll, _f, _p],
        "mm_ce_fwd_bwd": [_p, _ll, _p, _p, _i, _i, _i, _p, _p, _i, _p],
        "mm_label_rows": [_p, _i, _i, _p, _p, _p, _p],
        "mm_fmha_max_tiles": [_i, _i],
        "mm_fmha_set_fwd_variant": [_i],
        "mm_fmha_fwd": [_p, _p, _p, _p, _p, _p, _p, _p, _i, _i, _i, _i, _i, _i, _ll, _ll, _ll, _i, _f, _p, _p],
        "mm_fmha_bwd_max_tiles": [_i, _i],
        "mm_fmha_sum_heads": [_p, _p, _p, _p, _i, _i, _i, _i, _p],
        "mm_fmha_bwd": [_p, _p, _p, _p, _p, _p, _p, _p, _p, _p, _p, _p, _p, _i, _i, _i, _i, _i, _i, _ll, _ll, _ll, _i, _f,
                        _i, _i, _p, _p],
        "mm_grouped_gemm_bf16": [_p, _p, _p, _p, _i, _i, _i, _i, _i, _p, _p],
        "mm_moe_permute": [_p, _p, _p, _i, _i, _p],
        "mm_moe_unpermute": [_p, _p, _p, _p, _i, _i, _i, _p],
        "mm_moe_unpermute_bwd": [_p, _p, _p, _p, _p, _p, _p, _i, _i, _i, _i, _p],
        "mm_moe_route": [_p, _i, _i, _i, _i, _p, _p, _p, _p, _p, _p],
        "mm_moe_route_scratch": [_i, _i],
        "mm_delta_heads_fwd": [_p, _p, _p, _p, _p, _i, _i, _i, _i, _f, _p],
        "mm_delta_heads_bwd": [_p, _p, _p, _p, _p, _p, _p, _i, _i, _i, _i, _p],
        "mm_conv1d_fwd": [_p, _ll, _p, _p, _p, _i, _i, _i, _i, _p],
        "mm_conv1d_bwd": [_p, _ll, _p, _p, _p, _p, _p, _p, _i, _i, _i, _i, _p],
        "mm_l2norm_fwd": [_p, _p, _p, _ll, _i, _f, _p],
        "mm_l2norm_bwd": [_p, _p, _p, _p, _ll, _i, _p],
        "mm_gdn_prologue": [_p, _p, _p, _p, _p, _p, _p, _p, _p, _p, _p, _p, _p, _i, _i, _f, _p],
        "mm_gdn_prologue_bwd": [_p] * 17 + [_i, _i, _f, _p],
        "mm_gdn_layout": [_p, _p, _p, _p, _i, _i, _i, _p],
        "mm_gdn_fwd": [_p, _p, _p, _p, _p, _p, _p, _p, _p, _p, _p, _i, _i, _i, _i, _p, _p],
        "mm_gdn_bwd": [_p, _p, _p, _p, _p, _p, _p, _p, _p, _i, _i, _i, _i, _p, _p],
        "mm_p2p_scatter_rows": [_p, _p, _p, _p, _p, _i, _i, _i, _p],
        "mm_p2p_gather_rows": [_p, _p, _p, _p, _i, _i, _i, _p],
        "mm_p2p_copy": [_p, _p, _ll, _i, _p],
        "mm_p2p_set_wait_limit": [_ll],
        "mm_p2p_flag_bytes": [],
        "mm_p2p_allgather": [_p, _p, _ll, _i, _i, _i, _p],
        "mm_p2p_allgather_ce": [_p, _p, _ll, _i, _i, _p],
        "mm_p2p_rs_adamw": [_p, _p, _ll, _i, _i, _i, C.c_uint, _f, _p, _p, _p, _p, _ll, _f, _f, _f, _f, _f, _f, _f,
                            _p, _i, _p],
        "mm_p2p_rs": [_p, _p, _ll, _i, _i, _i, C.c_uint, _f, _p, _i, _p, _i, _p],
        "mm_p2p_wait_done": [_p, _i, C.c_uint, _i, _i, _p, _p],
        "mm_p2p_barrier_bytes": [],
        "mm_p2p_barrier": [_p, _i, _i, C.c_uint, _p, _p],
    }
    for name, args in sig.items():
        if hasattr(L, name):
            fn = getattr(L, name)
            fn.argtypes = args
            fn.restype = _ll if name in ("mm_gemm_ws_bytes", "mm_gemm_rows_ws_bytes", "mm_moe_route_scratch") else _i
            _STATUS[name] = True
        else:
            _STATUS[name] = False


def status() -> dict:
    lib()
    return {"loaded": True, "path": _build.lib_path(), "symbols": dict(_STATUS)}


def _st():
    """Raw handle of the current stream (building a ``torch.cuda.Stream`` for it costs 3 us a launch)."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


class _NoGraph:
    """Context of an autograd function that is run without a graph: takes what forward keeps and drops it."""
    __slots__ = ()

    def save_for_backward(self, *tensors):
        pass

    def __setattr__(self, name, value):
        pass


_NO_GRAPH = _NoGraph()


# bound once: looking them up costs more than calling them, and a generation step asks some fifty times
_compiling, _transforms, _tracing = torch.compiler.is_compiling, torch._C._are_functorch_transforms_active, torch._C._get_tracing_state
_wrapped, _forward_ad, _grad_enabled = torch._C._functorch.is_functorch_wrapped_tensor, torch.autograd.forward_ad, torch.is_grad_enabled


def _plain_mode() -> bool:
    """No transform, forward-mode level, tracer or compiler is active."""
    return not (_compiling() or _transforms() or _forward_ad._current_level >= 0 or _tracing() is not None)


def _keeps_no_graph(args) -> bool:
    if not _plain_mode():
        return False
    grad = _grad_enabled()
    for a in args:
        if isinstance(a, torch.Tensor) and ((grad and a.requires_grad) or _wrapped(a)):
            return False
    return True


def _plain_bf16(tensors) -> bool:
    """:func:`_keeps_no_graph` of tensors (or None) that have to be bf16 on one device."""
    if not _plain_mode():
        return False
    grad, bf16, dev, tensor = _grad_enabled(), torch.bfloat16, tensors[0].get_device(), torch.Tensor
    for t in tensors:
        # (a functorch wrapper is never a Parameter, which most of these are)
        if t is not None and (t.dtype is not bf16 or t.get_device() != dev or (grad and t.requires_grad) or (type(t) is tensor and _wrapped(t))):
            return False
    return True


def _run(fn, *args):
    """``fn.apply(*args)``.  Where nothing asks for a gradient and no transform, forward-mode level or tracer is active, the
    forward is called directly: ``apply`` costs 15 us of host time a call, more than most kernels of a generation step or of a
    prompt of a thousand tokens take (one token through 8 layers: 1484 -> 1235 us, a prompt of 1020 tokens with an image: 6604 -> 5725 us)."""
    if _keeps_no_graph(args):
        return fn.forward(_NO_GRAPH, *args)
    return fn.apply(*args)


def _eager(op: str, x, why: str):
    """An op of this module was called with a shape its kernel does not take: count it (or refuse, in strict mode)
    through the front end's fallback register, then let the caller run the PyTorch form."""
    from .. import ops as _ops
    _ops._fallback(op, x, why)


SYNC_CHECK = False   # ops/sanitize.py: synchronise after every native call and read the status word, so that an
                     # asynchronous error is reported under the name of the op that launched it


def _check(rc: int, what: str):
    global LAUNCHES
    LAUNCHES += 1
    if rc != 0:
        raise RuntimeError(f"{what} failed with code {rc}")
    if SYNC_CHECK and torch.cuda.is_available():
        try:
            torch.cuda.synchronize()
        except RuntimeError as e:
            raise RuntimeError(f"{what}: device error surfaced after this launch: {e}") from e
        for key, word in _status_words.items():
            v = int(word.item())
            if v:
                word.zero_()
                raise RuntimeError(f"{what}: a bounded wait ran out on device {key} (status {v})")


_status_words: dict = {}


def status_word(device) -> torch.Tensor:
    """Device int the tcgen05 kernels write when a bounded wait ran out (0 = fine)."""
    key = torch.device(device).index or 0
    if key not in _status_words:
        _status_words[key] = torch.zeros(1, dtype=torch.int32, device=device)
    return _status_words[key]


def check_status(device=None) -> int:
    """Host-side read of the status word (synchronises); raises if a kernel reported a timeout."""
    dev = device if device is not None else torch.cuda.current_device()
    v = int(status_word(dev).item())
    if v != 0:
        status_word(dev).zero_()
        raise RuntimeError(f"a native kernel gave up a bounded wait (status {v})")
    return v


def _pitch(x) -> int:
    """Elements between the rows of a matrix (a single row's stride means nothing)."""
    return x.stride(0) if x.shape[0] > 1 else x.shape[1]


def _dense(t):
    """Contiguous and 16-byte aligned, as kernels with vector loads take it (a single row of a wider matrix is contiguous wherever
    it starts, and .contiguous() returns it as it is)."""
    return t if t.is_contiguous() and t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format)


# --------------------------------------------------------------------------- RMSNorm
class _RMSNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, eps):
        shape = x.shape
        H = shape[-1]
        x2 = x.reshape(-1, H)
        if _row_group(H) or not _ok2d(x2):
            x2 = _dense(x2)
        T = x2.shape[0]
        y = torch.empty(T, H, dtype=x.dtype, device=x.device)
        rstd = torch.empty(T, dtype=torch.float32, device=x.device)
        wc = _dense(w)
        if _row_group(H):
            rc = lib().mm_rownorm_rms_fwd(x2.data_ptr(), wc.data_ptr(), y.data_ptr(), rstd.data_ptr(), T, H, eps, _st())
        else:       # rows may lie apart (the query or key columns of a fused projection): no copy of them is made
            rc = lib().mm_rmsnorm_fwd_ld(x2.data_ptr(), _pitch(x2), wc.data_ptr(), y.data_ptr(), rstd.data_ptr(), T, H, eps, _st())
        _check(rc, "rmsnorm_fwd")
        ctx.save_for_backward(x2, wc, rstd)
        ctx.shape = shape
        return y.view(shape)

    @staticmethod
    def backward(ctx, dy):
        x2, w, rstd = ctx.saved_tensors
        T, H = x2.shape
        dy2 = _dense(dy.reshape(T, H))
        dx = torch.empty(T, H, dtype=x2.dtype, device=x2.device)
        dw = torch.empty_like(w)
        grid = lib().mm_rmsnorm_bwd_grid(T)
        partial = torch.empty(grid * H, dtype=torch.float32, device=x2.device)
        _check(lib().mm_rmsnorm_bwd_ld(x2.data_ptr(), _pitch(x2), w.data_ptr(), dy2.data_ptr(), rstd.data_ptr(), dx.data_ptr(),
                                    dw.data_ptr(), partial.data_ptr(), T, H, _st()), "rmsnorm_bwd")
        return dx.view(ctx.shape), dw, None


def rms_norm(x, w, eps=1e-6):
    if x.shape[-1] % 8 or x.shape[-1] > 8192:
        from . import reference
        _eager("rms_norm", x, f"H={x.shape[-1]}")
        return reference.rms_norm(x, w, eps)
    return _run(_RMSNorm, x, w, eps)


# --------------------------------------------------------------------------- SwiGLU
class _SwiGLU(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gu):
        F2 = gu.shape[-1]
        g2 = gu.reshape(-1, F2)
        if not g2.is_contiguous():
            g2 = g2.contiguous()
        T, F = g2.shape[0], F2 // 2
        out = torch.empty(T, F, dtype=gu.dtype, device=gu.device)
        _check(lib().mm_swiglu_fwd(g2.data_ptr(), out.data_ptr(), T, F, _st()), "swiglu_fwd")
        ctx.save_for_backward(g2)
        ctx.shape = gu.shape
        return out.view(*gu.shape[:-1], F)

    @staticmethod
    def backward(ctx, dout):
        (g2,) = ctx.saved_tensors
        T, F = g2.shape[0], g2.shape[1] // 2
        d2 = dout.reshape(T, F)
        if not d2.is_contiguous():
            d2 = d2.contiguous()
        din = torch.empty_like(g2)
        _check(lib().mm_swiglu_bwd(g2.data_ptr(), d2.data_ptr(), din.data_ptr(), T, F, _st()), "swiglu_bwd")
        return din.view(ctx.shape)


def swiglu(gu):
    if (gu.shape[-1] // 2) % 8:
        from . import reference
        _eager("swiglu", gu, f"F={gu.shape[-1] // 2}")
        return reference.swiglu(gu)
    return _run(_SwiGLU, gu)


# --------------------------------------------------------------------------- RoPE
class _Gelu(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, tanh):
        xc = x.contiguous()
        y = torch.empty_like(xc)
        _check(lib().mm_gelu_fwd(xc.data_ptr(), y.data_ptr(), xc.numel(), int(tanh), _st()), "gelu_fwd")
        ctx.save_for_backward(xc)
        ctx.tanh = tanh
        return y.view(x.shape)

    @staticmethod
    def backward(ctx, dy):
        (x,) = ctx.saved_tensors
        dyc = dy.contiguous()
        dx = torch.empty_like(x)
        _check(lib().mm_gelu_bwd(x.data_ptr(), dyc.data_ptr(), dx.data_ptr(), x.numel(), int(ctx.tanh), _st()), "gelu_bwd")
        return dx.view(dy.shape), None


def gelu(x, tanh: bool = True):
    """bf16 GELU (tanh approximation or exact erf form); element count a multiple of 8."""
    return _run(_Gelu, x, bool(tanh))


def _rope_call(x, cos, sin, interleaved, backward):
    # x: [T, N, D] whose last two dims are dense; the token stride may be larger (view into fused qkv)
    T, N, D = x.shape
    if x.stride(2) != 1 or x.stride(1) != D or x.stride(0) % 8 or x.data_ptr() % 16:
        x = x.contiguous()
    out = torch.empty(T, N, D, dtype=x.dtype, device=x.device)
    if interleaved:
        _check(lib().mm_rope_interleaved(x.data_ptr(), x.stride(0), cos.data_ptr(), sin.data_ptr(), out.data_ptr(),
                                         T, N, D, int(backward), _st()), "rope_interleaved")
    else:
        _check(lib().mm_rope_half(x.data_ptr(), x.stride(0), cos.data_ptr(), sin.data_ptr(), out.data_ptr(),
                                  T, N, D, int(backward), _st()), "rope_half")
    return out


class _Rope(torch.autograd.Function):
    """The rotation or, with ``back``, its transpose: each is the other's gradient, which can so be differentiated in its turn."""

    @staticmethod
    def forward(ctx, x, cos, sin, interleaved, back):
        ctx.save_for_backward(cos, sin)
        ctx.meta = interleaved, back
        return _rope_call(x, cos, sin, interleaved, back)

    @staticmethod
    def backward(ctx, dy):
        interleaved, back = ctx.meta
        return _run(_Rope, dy, *ctx.saved_tensors, interleaved, not back), None, None, None, None


def rope(x, cos, sin, interleaved: bool):
    T, N, D = x.shape
    if interleaved:
        if D % 8:
            from . import reference
            _eager("rope_interleaved", x, f"D={D}")
            return reference.rope_interleaved(x, cos, sin)
        cos, sin = cos.float().contiguous(), sin.float().contiguous()
    else:
        if D % 8:
            from . import reference
            _eager("rope_rotate_half", x, f"D={D}")
            return reference.rope_rotate_half(x, cos, sin)
        cos, sin = cos.to(torch.bfloat16).contiguous(), sin.to(torch.bfloat16).contiguous()
    return _run(_Rope, x, cos, sin, interleaved, False)


def _rope_parts(q, k, v, cos, sin, outs, backward):
    """Rotates q and k into ``outs[:2]`` and copies v (None: left alone) into ``outs[2]``; all [T, N, D]."""
    dense = lambda t: t if t is None else _dense(t) if t.data_ptr() % 16 else _dense_heads(t)  # noqa: E731
    q, k, v = dense(q), dense(k), dense(v)
    T, nq, D = q.shape
    pointers = [a for t in (q, k, v) for a in ((None, 0) if t is None else (t.data_ptr(), t.stride(0)))]
    targets = [a for t in outs for a in ((None, 0) if t is None else (t.data_ptr(), t.stride(0)))]
    _check(lib().mm_rope_qkv(*pointers, cos.data_ptr(), sin.data_ptr(), *targets, T, nq, k.shape[1], 0 if v is None else v.shape[1], D,
                             int(backward), _st()), "rope_qkv")


def rope_pair_supported(q, k, cos, sin) -> bool:
    """The queries and keys of the same tokens, heads of a multiple of 16, tables made for them."""
    T, _, D = q.shape
    return (q.dtype == torch.bfloat16 and k.dtype == q.dtype and D % 16 == 0 and k.shape[0] == T and k.shape[2] == D and q.device == k.device
            and tuple(cos.shape) == (T, D) and tuple(sin.shape) == (T, D))


def _tables(cos, sin):
    return _dense(cos.to(torch.bfloat16)), _dense(sin.to(torch.bfloat16))


def rope_pair(q, k, cos, sin):
    """Both rotated by one kernel.  No autograd: for calls that keep no graph."""
    cos, sin = _tables(cos, sin)
    outs = [torch.empty(t.shape, dtype=t.dtype, device=t.device) for t in (q, k)]
    _rope_parts(q, k, None, cos, sin, [*outs, None], False)
    return outs


class _SplitRope(torch.autograd.Function):
    """Rotated queries and keys, and the values as they lie, of a fused projection [T, (nq + 2 nk) D]; its gradient is written whole by one
    kernel (a rotation for each tensor and a stack or concatenation before)."""

    @staticmethod
    def forward(ctx, qkv, cos, sin, nq, nk):
        T, D = qkv.shape[0], qkv.shape[1] // (nq + 2 * nk)
        ctx.save_for_backward(cos, sin)
        ctx.heads = nq, nk, D
        q, k, v = (t.view(T, -1, D) for t in qkv.split([nq * D, nk * D, nk * D], dim=1))
        outs = [torch.empty(t.shape, dtype=t.dtype, device=t.device) for t in (q, k)]
        _rope_parts(q, k, None, cos, sin, [*outs, None], False)
        return (*outs, v)

    @staticmethod
    def backward(ctx, dq, dk, dv):
        cos, sin = ctx.saved_tensors
        nq, nk, D = ctx.heads
        T = dq.shape[0]
        if torch.is_grad_enabled():          # create_graph: all three parts are differentiated
            return torch.cat([*(_run(_Rope, t, cos, sin, False, True).view(T, -1) for t in (dq, dk)), dv.reshape(T, -1)], dim=1), None, None, None, None
        dqkv = torch.empty(T, (nq + 2 * nk) * D, dtype=dq.dtype, device=dq.device)
        _rope_parts(dq, dk, dv, cos, sin, [t.view(T, -1, D) for t in dqkv.split([nq * D, nk * D, nk * D], dim=1)], True)
        return dqkv, None, None, None, None


def split_rope_supported(qkv, nq, nk, cos, sin) -> bool:
    heads = nq + 2 * nk
    if qkv.dim() != 2 or qkv.dtype != torch.bfloat16 or qkv.shape[1] % heads or not _ok2d(qkv):
        return False
    T, D = qkv.shape[0], qkv.shape[1] // heads
    return T > 0 and D % 16 == 0 and tuple(cos.shape) == (T, D) and tuple(sin.shape) == (T, D) and not (cos.requires_grad or sin.requires_grad)


def split_rope(qkv, nq, nk, cos, sin):
    return _run(_SplitRope, qkv, *_tables(cos, sin), nq, nk)


# --------------------------------------------------------------------------- adaLN
class _LNMod(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, scale, shift, eps):
        B, S, H = x.shape
        xc, sc, sh = x.contiguous(), scale.reshape(B, H).contiguous(), shift.reshape(B, H).contiguous()
        y = torch.empty_like(xc)
        mean = torch.empty(B * S, dtype=torch.float32, device=x.device)
        rstd = torch.empty_like(mean)
        fn = lib().mm_rownorm_ln_mod_fwd if _row_group(H) else lib().mm_ln_mod_fwd
        _check(fn(xc.data_ptr(), sc.data_ptr(), sh.data_ptr(), y.data_ptr(), mean.data_ptr(), rstd.data_ptr(), B * S, S, H,
                  eps, _st()), "ln_mod_fwd")
        ctx.save_for_backward(xc, sc, mean, rstd)
        ctx.sshape = scale.shape
        return y

    @staticmethod
    def backward(ctx, dy):
        x, sc, mean, rstd = ctx.saved_tensors
        B, S, H = x.shape
        dyc = dy.contiguous()
        dx = torch.empty_like(x)
        dscale = torch.empty_like(sc)
        dshift = torch.empty_like(sc)
        per = lib().mm_ln_mod_bwd_ctas(B, S)
        partial = torch.empty(2 * B * per * H, dtype=torch.float32, device=x.device)
        _check(lib().mm_ln_mod_bwd(x.data_ptr(), sc.data_ptr(), dyc.data_ptr(), mean.data_ptr(), rstd.data_ptr(),
                                   dx.data_ptr(), dscale.data_ptr(), dshift.data_ptr(), partial.data_ptr(), B, S, H,
                                   _st()), "ln_mod_bwd")
        return dx, dscale.view(ctx.sshape), dshift.view(ctx.sshape), None


def layer_norm_modulate(x, scale, shift, eps=1e-6):
    """x: [B, S, H]; scale/shift: [B, 1, H] or [B, H]."""
    if x.dim() != 3 or x.shape[-1] % 8 or x.shape[-1] > 8192 or scale.numel() != x.shape[0] * x.shape[-1]:
        from . import reference
        _eager("layer_norm_modulate", x, f"x {tuple(x.shape)} scale {tuple(scale.shape)}")
        return reference.layer_norm_modulate(x, scale, shift, eps)
    return _run(_LNMod, x, scale.to(x.dtype), shift.to(x.dtype), eps)


def layer_norm(x, weight=None, bias=None, eps=1e-6):
    """LayerNorm over the last dim of a bf16 tensor through the LayerNorm-modulate kernels: all rows form one batch,
    ``scale = weight - 1`` and ``shift = bias`` (zeros when absent), so ``LN(x) * (1 + scale) + shift`` is the affine
    LayerNorm.  Gradients of weight / bias come out of the kernel's per-batch scale / shift reductions."""
    H = x.shape[-1]
    if weight is not None:
        scale = (weight.float() - 1.0).to(x.dtype).view(1, H)
    else:
        scale = torch.zeros(1, H, dtype=x.dtype, device=x.device)
    shift = bias.to(x.dtype).view(1, H) if bias is not None else torch.zeros(1, H, dtype=x.dtype, device=x.device)
    return _run(_LNMod, x.reshape(1, -1, H), scale, shift, eps).view(x.shape)


class _GatedResidual(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, y, gate):
        B, S, H = x.shape
        xc, yc, gc = x.contiguous(), y.contiguous(), gate.reshape(B, H).contiguous()
        out = torch.empty_like(xc)
        _check(lib().mm_gated_residual(xc.data_ptr(), yc.data_ptr(), gc.data_ptr(), out.data_ptr(), B * S, S, H,
                                       _st()), "gated_residual")
        ctx.save_for_backward(yc, gc)
        ctx.gshape = gate.shape
        return out

    @staticmethod
    def backward(ctx, dout):
        y, g = ctx.saved_tensors
        B, S, H = y.shape
        if torch.is_grad_enabled():          # create_graph: the gradient itself is differentiated
            return dout, dout * g.view(B, 1, H), (dout.float() * y.float()).sum(1).to(g.dtype).view(ctx.gshape)
        dc, y, g = (t if t.data_ptr() % 16 == 0 else t.clone() for t in (dout.contiguous(), y, g))
        dy, dg = torch.empty_like(y), torch.empty_like(g)
        partial = torch.empty(B * lib().mm_column_splits(S, H, B, 1) * H, dtype=torch.float32, device=y.device)
        _check(lib().mm_gated_residual_bwd(dc.data_ptr(), y.data_ptr(), g.data_ptr(), dy.data_ptr(), dg.data_ptr(), partial.data_ptr(),
                                           B, S, H, _st()), "gated_residual_bwd")
        return dout, dy, dg.view(ctx.gshape)


def gated_residual(x, y, gate):
    if x.dim() != 3 or x.shape[-1] % 8 or gate.numel() != x.shape[0] * x.shape[-1]:
        from . import reference
        _eager("gated_residual", x, f"x {tuple(x.shape)} gate {tuple(gate.shape)}")
        return reference.gated_residual(x, y, gate)
    return _run(_GatedResidual, x, y, gate.to(x.dtype))


# --------------------------------------------------------------------------- AdamW
def sq_norm(tensors) -> torch.Tensor:
    """Sum of squares over a list of fp32 CUDA tensors (the squared global gradient norm of flat shards): one launch per
    tensor into a fixed-order table of block partials, one reduction at the end."""
    nb = lib().mm_sq_norm_blocks()
    partials = torch.zeros(len(tensors), nb, dtype=torch.float32, device=tensors[0].device)
    st = _st()
    for i, t in enumerate(tensors):
        t = t.contiguous()
        if t.data_ptr() % 16:           # a view at an odd offset: the kernel reads 16-byte vectors
            t = t.clone()
        _check(lib().mm_sq_norm(t.data_ptr(), t.numel(), partials[i].data_ptr(), st), "sq_norm")
    return partials.sum()


def adamw_shard(master, exp_avg, exp_avg_sq, grad, p16, lr, b1, b2, eps, wd, step, split, grad_scale=1.0):
    n = master.numel()
    scale_ptr = None
    gs = 1.0
    if isinstance(grad_scale, torch.Tensor):
        scale_ptr = grad_scale.float().reshape(1)
        sp = scale_ptr.data_ptr()
    else:
        gs = float(grad_scale)
        sp = None
    bc1 = 1.0 - b1 ** step
    bc2 = 1.0 - b2 ** step
    g = grad if grad.dtype in (torch.bfloat16, torch.float32) else grad.float()
    _check(lib().mm_adamw(master.data_ptr(), exp_avg.data_ptr(), exp_avg_sq.data_ptr(), g.data_ptr(),
                          int(g.dtype == torch.bfloat16), p16.data_ptr(), n, int(split), lr, b1, b2, eps, wd, bc1, bc2,
                          gs, sp, _st()), "adamw")


# --------------------------------------------------------------------------- GEMM (tcgen05)
def _gemm_raw(a, b, out, bias, M, N, K, lda, ldb, ldc, a_mn, b_mn, bn=None):
    if bn is None:
        bn = 256 if N >= 256 else 128
    st = status_word(a.device)
    L = lib()
    nbytes = L.mm_gemm_ws_bytes(M, N, K, int(a_mn), int(b_mn), bn)
    ws = torch.empty(nbytes, dtype=torch.uint8, device=a.device) if nbytes else None
    rc = L.mm_gemm_bf16_ws(a.data_ptr(), b.data_ptr(), out.data_ptr(), None if bias is None else bias.data_ptr(), M, N, K, lda, ldb,
                           ldc, int(a_mn), int(b_mn), bn, st.data_ptr(), None if ws is None else ws.data_ptr(), nbytes, _st())
    _check(rc, "gemm_bf16")


def _ok2d(t):
    st = t.stride()
    return len(st) == 2 and st[1] == 1 and st[0] % 8 == 0 and t.data_ptr() % 16 == 0


def gemm_supported(x, w) -> bool:
    return (os.environ.get("MM_B200_GEMM", "1") == "1" and w.dtype == torch.bfloat16 and w.dim() == 2
            and w.shape[0] % 8 == 0 and w.shape[1] % 8 == 0)


def gemm_nt(a, b, bias=None, out=None):
    """a [M,K] @ b[N,K]^T (+bias) -> [M,N]."""
    if not _ok2d(a):
        a = a.contiguous()
    if not _ok2d(b):
        b = b.contiguous()
    M, K = a.shape
    N = b.shape[0]
    if out is None:
        out = torch.empty(M, N, dtype=torch.bfloat16, device=a.device)
    _gemm_raw(a, b, out, bias, M, N, K, a.stride(0), b.stride(0), out.stride(0), 0, 0)
    return out


def gemm_swiglu_supported(x, w) -> bool:
    return gemm_supported(x, w) and w.shape[0] % 256 == 0 and os.environ.get("MM_B200_GEMM_SWIGLU", "1") == "1"


def gemm_swiglu(x, w):
    """``silu(x W_gate^T) * (x W_up^T)`` for the fused ``w = [W_gate; W_up]`` ([2F, K]) in one kernel: the activation is the
    GEMM epilogue and the [T, 2F] pre-activation is never written.  No autograd: for passes that keep no graph."""
    shape = x.shape
    a = x.reshape(-1, shape[-1])
    if not _ok2d(a):
        a = a.contiguous()
    if not _ok2d(w):
        w = w.contiguous()
    M, K = a.shape
    F = w.shape[0] // 2
    out = torch.empty(M, F, dtype=torch.bfloat16, device=a.device)
    st = status_word(a.device)
    _check(lib().mm_gemm_swiglu_bf16(a.data_ptr(), w.data_ptr(), out.data_ptr(), M, F, K, a.stride(0), w.stride(0),
                                     out.stride(0), st.data_ptr(), _st()), "gemm_swiglu_bf16")
    return out.view(*shape[:-1], F)


# --------------------------------------------------------------------------- generation (csrc/decode.cu)
# These kernels are called outside of an autograd function, so each rule below asks for a call that keeps no graph.
def mrope_tables_supported(position_ids, head_dim, section, dtype) -> bool:
    return (dtype == torch.bfloat16 and position_ids.dtype == torch.int64 and position_ids.dim() == 2 and position_ids.shape[0] == 3
            and position_ids.shape[1] > 0 and head_dim % 2 == 0 and len(section) == 3 and _keeps_no_graph((position_ids,)))


def mrope_tables(position_ids, head_dim, theta, section):
    """bf16 rotary tables [T, head_dim] of int64 positions [3, T], computed in 64 bits by one kernel."""
    pos = position_ids.contiguous()
    T = pos.shape[1]
    cos, sin = (torch.empty(T, head_dim, dtype=torch.bfloat16, device=pos.device) for _ in range(2))
    _check(lib().mm_rotary_tables(pos.data_ptr(), cos.data_ptr(), sin.data_ptr(), T, head_dim // 2, *section, float(theta), _st()),
           "rotary_tables")
    return cos, sin


def skinny_supported(x, w, *tensors, norm=None) -> bool:
    """Up to 4 bf16 rows that keep no graph: the product kernel of csrc/decode.cu with its fused ends applies.  The sizes are
    mm_gemv_bf16's own rule: x, and with a norm its weight too, have to fit a block's shared memory; and four rows against a weight
    whose tiles keep half of the SMs busy are left to the tensor cores (``skinny`` in csrc/gemm.cu)."""
    if x.dim() != 2:
        return False
    M, K = x.shape
    if not 1 <= M <= 4 or K % 8 or M * K > 80 * 1024 or (norm is not None and (M + 1) * K > 112 * 1024) or (M == 4 and w.shape[0] >= 74 * 256):
        return False
    return _plain_bf16((x, w, norm, *tensors)) and _ok2d(x)


def skinny_linear(x, w, bias=None, norm=None, eps=0.0, residual=None, swiglu=False):
    """``act(rms_norm(x) @ w.T + bias) + residual`` for the rows :func:`skinny_supported` takes."""
    if not _ok2d(w):
        w = w.contiguous()
    if bias is not None:
        bias = bias.contiguous()
    if norm is not None:
        norm = _dense(norm)
    if residual is not None and not _ok2d(residual):
        residual = residual.clone(memory_format=torch.contiguous_format)     # also where it only starts off an aligned address
    M, K = x.shape
    N = w.shape[0] // 2 if swiglu else w.shape[0]
    out = torch.empty(M, N, dtype=torch.bfloat16, device=x.device)
    _check(lib().mm_gemv_bf16(x.data_ptr(), w.data_ptr(), None if bias is None else bias.data_ptr(),
                              None if norm is None else norm.data_ptr(), None if residual is None else residual.data_ptr(),
                              out.data_ptr(), M, N, K, x.stride(0), w.stride(0), 0 if residual is None else residual.stride(0),
                              out.stride(0), eps, int(swiglu), _st()), "gemv_bf16")
    return out


def decode_attention_supported(q, k, v, k_old, v_old, cos, sin=None) -> bool:
    """Head dim 128, the new tokens' query heads of a group fill at most one 16-row tile, nothing keeps a graph."""
    T, Nq, D = q.shape
    Tk, Nkv, Dk = k.shape
    if D != 128 or Dk != D or not 1 <= T == Tk or v.shape != k.shape or Nq % Nkv or T * (Nq // Nkv) > 16:
        return False
    if k_old is not None and (k_old.shape != v_old.shape or k_old.shape[1:] != k.shape[1:]):
        return False
    if cos is not None and tuple(cos.shape) != (T, D):
        return False
    return os.environ.get("MM_B200_FMHA", "1") == "1" and _plain_bf16((q, k, v, k_old, v_old)) and _keeps_no_graph((cos, sin))


def decode_attention(q, k, v, k_old, v_old, cos, sin):
    """Rotates q and k (unless ``cos`` is None), appends k / v to the cache and attends to all of it.  Returns (out, keys, values)."""
    q, k, v = _dense_heads(q), _dense_heads(k), _dense_heads(v)
    T, Nq, D = q.shape
    Nkv, past = k.shape[1], 0
    if cos is not None:
        cos, sin = _dense(cos.to(torch.bfloat16)), _dense(sin.to(torch.bfloat16))
    if k_old is not None:
        k_old, v_old, past = _dense(k_old), _dense(v_old), k_old.shape[0]
    k_new, v_new = (torch.empty(past + T, Nkv, D, dtype=torch.bfloat16, device=q.device) for _ in range(2))
    out = torch.empty(T, Nq, D, dtype=torch.bfloat16, device=q.device)
    ptr = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    _check(lib().mm_decode_attention(q.data_ptr(), k.data_ptr(), v.data_ptr(), ptr(cos), ptr(sin), ptr(k_old), ptr(v_old),
                                     k_new.data_ptr(), v_new.data_ptr(), out.data_ptr(), T, past, Nq, Nkv, q.stride(0), k.stride(0),
                                     v.stride(0), 1.0 / math.sqrt(D), _st()), "decode_attention")
    return out, k_new, v_new


def gemm_nn(a, b, out=None):
    """a [M,K] @ b[K,N] -> [M,N]  (b read N-contiguous: dgrad)."""
    if not _ok2d(a):
        a = a.contiguous()
    if not _ok2d(b):
        b = b.contiguous()
    M, K = a.shape
    N = b.shape[1]
    if out is None:
        out = torch.empty(M, N, dtype=torch.bfloat16, device=a.device)
    _gemm_raw(a, b, out, None, M, N, K, a.stride(0), b.stride(0), out.stride(0), 0, 1)
    return out


def gemm_tn(a, b, out=None):
    """a[K,M]^T @ b[K,N] -> [M,N]  (both read with the contraction dim strided: wgrad)."""
    if not _ok2d(a):
        a = a.contiguous()
    if not _ok2d(b):
        b = b.contiguous()
    K, M = a.shape
    N = b.shape[1]
    if out is None:
        out = torch.empty(M, N, dtype=torch.bfloat16, device=a.device)
    _gemm_raw(a, b, out, None, M, N, K, a.stride(0), b.stride(0), out.stride(0), 1, 1)
    return out


_BWD_NATIVE = os.environ.get("MM_B200_GEMM_BWD", "1") == "1"


def column_sum(x):
    """Sum over the rows of a bf16 matrix (a bias gradient), fp32 inside.  The four bias gradients of a vision block on 8192 patches
    (218 MB, out of L2 as they come): 94 us as ``torch.sum``, 69 us in these two kernels."""
    rows, cols = x.shape
    if rows < 1 or cols % 8 or not _ok2d(x):
        return torch.sum(x, 0, dtype=torch.float32).to(x.dtype)
    out = torch.empty(cols, dtype=x.dtype, device=x.device)
    partial = torch.empty(lib().mm_column_splits(rows, cols, 1, 0) * cols, dtype=torch.float32, device=x.device)
    _check(lib().mm_column_sum(x.data_ptr(), out.data_ptr(), partial.data_ptr(), rows, cols, x.stride(0), _st()), "column_sum")
    return out


class _Linear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, bias, skip_value=False):
        shape = x.shape
        x2 = x.reshape(-1, shape[-1])
        ctx.save_for_backward(x2, w)
        ctx.has_bias = bias is not None
        ctx.shape = shape
        if skip_value:
            # re-forward of a checkpointed unit whose last linear feeds only a residual add: the gradient needs the
            # operands, not the product, so the GEMM is not run again
            return torch.empty(*shape[:-1], w.shape[0], dtype=x.dtype, device=x.device)
        y = gemm_nt(x2, w, bias)
        return y.view(*shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, w = ctx.saved_tensors
        dy2 = dy.reshape(-1, w.shape[0])
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        dx = dw = db = None
        if ctx.needs_input_grad[0]:
            dx = (gemm_nn(dy2, w) if _BWD_NATIVE else dy2 @ w).view(ctx.shape)
        if ctx.needs_input_grad[1]:
            tgt = getattr(w, "_grad_flat", None)
            if tgt is not None and _BWD_NATIVE and w.grad is None:
                # the sharding engine offered this parameter's slice of the unit's flat gradient buffer: write the
                # weight gradient there (a fresh view each time, so autograd can adopt it as .grad without a copy)
                flat, off, numel, shape = tgt
                w._grad_flat = None                      # a second use of the same weight falls back to a new tensor
                dw = gemm_tn(dy2, x2, out=flat[off:off + numel].view(shape))
            else:
                dw = gemm_tn(dy2, x2) if _BWD_NATIVE else dy2.t() @ x2
        if ctx.has_bias and ctx.needs_input_grad[2]:
            # create_graph: the sum itself is differentiated
            db = torch.sum(dy2, 0, dtype=torch.float32).to(dy2.dtype) if torch.is_grad_enabled() else column_sum(dy2)
        return dx, dw, db, None


def linear(x, w, bias=None, skip_value=False):
    return _run(_Linear, x, w, bias, skip_value)


# --------------------------------------------------------------------------- not yet native
def fmha_supported(q, k, v) -> bool:
    """bf16, one head dim for q / k / v, at most 128 and a multiple of 8 (the kernels work on 128-wide tiles; a narrower
    head, e.g. the vision tower's 80, is zero-filled by the TMA loads, not padded in memory), GQA groups whole."""
    D = q.shape[-1]
    return (os.environ.get("MM_B200_FMHA", "1") == "1" and q.dtype == torch.bfloat16 and D <= 128 and D % 8 == 0
            and k.shape[-1] == D and v.shape[-1] == D and q.shape[1] % k.shape[1] == 0)


def _dense_heads(t):
    """[T, N, D] with unit stride on D, D between heads and an 8-element aligned token stride (views into a
    fused qkv tensor qualify); anything else is copied."""
    st = t.stride()
    if st[2] != 1 or st[1] != t.shape[2] or st[0] % 8 or t.data_ptr() % 16:
        t = t.contiguous()
    return t


def fmha_forward(q, k, v, cu_q, cu_k, causal, scale):
    """Returns (out [T, Nq, D] bf16, lse [Nq, T] fp32) from the tcgen05 kernel."""
    q, k, v = _dense_heads(q), _dense_heads(k), _dense_heads(v)
    T, Nq, D = q.shape
    Tk, Nkv = k.shape[0], k.shape[1]
    n_seqs = cu_q.numel() - 1
    out = torch.empty(T, Nq, D, dtype=q.dtype, device=q.device)
    lse = torch.empty(Nq, T, dtype=torch.float32, device=q.device)
    plan = torch.empty(3 * lib().mm_fmha_max_tiles(T, n_seqs) + 1, dtype=torch.int32, device=q.device)
    cu_q = cu_q.to(torch.int32)
    cu_k = cu_k.to(torch.int32)
    rc = lib().mm_fmha_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), cu_q.data_ptr(),
                           cu_k.data_ptr(), plan.data_ptr(), T, Tk, n_seqs, Nq, Nkv, D, q.stride(0), k.stride(0),
                           v.stride(0), int(causal), float(scale), status_word(q.device).data_ptr(), _st())
    _check(rc, "fmha_fwd")
    return out, lse


# backward kernels: dQ kernel + dK/dV kernel over 128-row query steps (5, default) or over 64-row steps (0, fallback)
FMHA_BWD_VARIANT = int(os.environ.get("MM_B200_FMHA_BWD_VARIANT", "5"))
FMHA_BWD = os.environ.get("MM_B200_FMHA_BWD", "native")     # "native" (tcgen05 kernels) or "flash" (flash-attn library)


def fmha_backward(do, q, k, v, out, lse, cu_q, cu_k, causal, scale):
    """dq, dk, dv from the tcgen05 backward kernels (dQ kernel + dK/dV kernel, no atomics)."""
    q, k, v = _dense_heads(q), _dense_heads(k), _dense_heads(v)
    do, out = do.contiguous(), out.contiguous()
    T, Nq, D = q.shape
    Tk, Nkv = k.shape[0], k.shape[1]
    n_seqs = cu_q.numel() - 1
    dev = q.device
    dq = torch.empty(T, Nq, D, dtype=q.dtype, device=dev)
    # GQA: one dK/dV CTA per QUERY head (more, shorter CTAs); the group's partials are summed afterwards
    split = Nq != Nkv
    dk = torch.empty(Tk, Nq if split else Nkv, D, dtype=q.dtype, device=dev)
    dv = torch.empty(Tk, Nq if split else Nkv, D, dtype=q.dtype, device=dev)
    delta = torch.empty(Nq, T, dtype=torch.float32, device=dev)
    L = lib()
    plan = torch.empty(3 * (L.mm_fmha_bwd_max_tiles(T, n_seqs) + L.mm_fmha_bwd_max_tiles(Tk, n_seqs)) + 2,
                       dtype=torch.int32, device=dev)
    cu_q, cu_k = cu_q.to(torch.int32), cu_k.to(torch.int32)
    rc = L.mm_fmha_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), do.data_ptr(), lse.data_ptr(),
                       delta.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), cu_q.data_ptr(), cu_k.data_ptr(),
                       plan.data_ptr(), T, Tk, n_seqs, Nq, Nkv, D, q.stride(0), k.stride(0), v.stride(0), int(causal),
                       float(scale), int(split), FMHA_BWD_VARIANT, status_word(dev).data_ptr(), _st())
    _check(rc, "fmha_bwd")
    global LAUNCHES
    LAUNCHES += 4
    if split:
        G = Nq // Nkv
        part_k, part_v = dk, dv
        dk, dv = (torch.empty(Tk, Nkv, D, dtype=q.dtype, device=dev) for _ in range(2))
        _check(L.mm_fmha_sum_heads(part_k.data_ptr(), part_v.data_ptr(), dk.data_ptr(), dv.data_ptr(), Tk, Nkv, G, D, _st()), "fmha_sum_heads")
    return dq, dk, dv


class _FMHA(torch.autograd.Function):
    """Forward and backward: tcgen05 kernels (``MM_B200_FMHA_BWD=flash`` switches the backward to flash-attn's
    varlen backward fed with this forward's out / lse, for comparison)."""

    @staticmethod
    def forward(ctx, q, k, v, cu_q, cu_k, max_q, max_k, causal, scale, precomputed=None):
        out, lse = precomputed if precomputed is not None else fmha_forward(q, k, v, cu_q, cu_k, causal, scale)
        ctx.save_for_backward(q, k, v, out, lse, cu_q, cu_k)
        ctx.meta = (max_q, max_k, causal, scale)
        ctx.lse_out = lse
        return out

    @staticmethod
    def backward(ctx, do):
        from flash_attn.flash_attn_interface import _flash_attn_varlen_backward
        q, k, v, out, lse, cu_q, cu_k = ctx.saved_tensors
        max_q, max_k, causal, scale = ctx.meta
        if FMHA_BWD == "native" and _STATUS.get("mm_fmha_bwd", False):
            dq, dk, dv = fmha_backward(do, q, k, v, out, lse, cu_q, cu_k, causal, scale)
            return dq, dk, dv, None, None, None, None, None, None, None
        dq, dk, dv = torch.empty(q.shape, dtype=q.dtype, device=q.device), torch.empty(k.shape, dtype=k.dtype, device=k.device), \
            torch.empty(v.shape, dtype=v.dtype, device=v.device)
        _flash_attn_varlen_backward(do.contiguous(), q, k, v, out, lse, dq, dk, dv, cu_q.to(torch.int32), cu_k.to(torch.int32),
                                    max_q, max_k, 0.0, scale, causal, -1, -1, 0.0, None, False)
        return dq, dk, dv, None, None, None, None, None, None, None


def attention_varlen(q, k, v, cu_q, cu_k, max_q, max_k, causal, scale, cache=None):
    """``cache`` = (store, mode) from :class:`ops.activation_cache`: under ``record`` (the no-grad first forward of a
    checkpointed unit) the output and log-sum-exp are kept, under ``replay`` (its re-forward) they are reused and the
    forward kernel is not run again."""
    scale = scale if scale is not None else 1.0 / math.sqrt(q.shape[-1])
    if cache is not None:
        store, mode = cache
        if mode == "record" and not torch.is_grad_enabled():
            out, lse = fmha_forward(q, k, v, cu_q, cu_k, bool(causal), float(scale))
            store.append((out, lse))
            return out
        if mode == "replay" and store:
            return _run(_FMHA, q, k, v, cu_q, cu_k, max_q, max_k, bool(causal), float(scale), store.pop(0))
    return _run(_FMHA, q, k, v, cu_q, cu_k, max_q, max_k, bool(causal), float(scale))


def lce_supported(h, w) -> bool:
    return gemm_supported(h, w) and h.dim() == 2


# Up to here a vocabulary product costs little less for fewer rows (its weight's bytes): with 70 % of the rows in use, 256 / 512 / 1024 / 8192
# rows take 928 / 1451 / 2695 / 19980 us over all of them and 1027 / 1460 / 2498 / 14990 over those.  Where all rows have a target the list is what
# it costs: 1024 / 2048 / 8192 rows 2764 / 5222 / 20490 us without it, 2819 / 5366 / 20460 with it.
_LIST_ROWS = 512


def _gemm_rows(a, b, out, a_mn, b_mn, count, base):
    """gemm_nt / gemm_nn / gemm_tn over the rows in use of ``a`` (and of ``b``, for the last): ``count`` (device int) less ``base``."""
    M, K = (a.shape[1], a.shape[0]) if a_mn else a.shape
    N = b.shape[1] if b_mn else b.shape[0]
    L = lib()
    nbytes = L.mm_gemm_rows_ws_bytes(M, N, K, a_mn, b_mn)
    ws = torch.empty(nbytes, dtype=torch.uint8, device=a.device)
    _check(L.mm_gemm_bf16_rows(a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), b.stride(0), out.stride(0), a_mn, b_mn,
                               count.data_ptr(), base, status_word(a.device).data_ptr(), ws.data_ptr(), nbytes, _st()), "gemm_bf16_rows")
    return out


class _LinearCE(torch.autograd.Function):
    """loss_sum = sum_t CE(h_t W^T, label_t).  Forward already produces both gradients:
    logits GEMM (tcgen05) -> in-place softmax-minus-onehot kernel -> dgrad and wgrad GEMMs (tcgen05);
    backward only scales them by the incoming scalar.  Rows are processed in chunks so that the bf16
    logits buffer stays a bounded slab (the reference chunks for the same reason:
    fsdp/features/memory/chunkloss/chunkloss.py:6-95).

    Rows without a target (prompts, images, padding) have neither loss nor gradient: the others are listed on the device, gathered,
    and the three products run over as many rows as the list has (which the host is not told).  8192 rows of which 70 % have
    a target, vocabulary 152064: 20.0 -> 15.0 ms; where all of 2048 have one, the list costs 5.22 -> 5.37 ms."""

    @staticmethod
    def forward(ctx, h, w, labels, ignore_index, chunk):
        T, H = h.shape
        V = w.shape[0]
        h, w_ = _dense(h), w if _ok2d(w) else w.contiguous()
        labels = labels.contiguous()
        dev, L, st = h.device, lib(), _st()
        row_loss = torch.empty(T, dtype=torch.float32, device=dev)
        dh = torch.empty_like(h)
        dw = torch.empty(w.shape, dtype=w.dtype, device=dev)
        listed = T > _LIST_ROWS and H >= 256 and V >= 256
        src = count = None
        x, dx = h, dh
        if listed:
            src, row, count = (torch.empty(n, dtype=torch.int32, device=dev) for n in (T, T, 1))
            _check(L.mm_label_rows(labels.data_ptr(), T, ignore_index, src.data_ptr(), row.data_ptr(), count.data_ptr(), st), "label_rows")
            x, dx = torch.empty_like(h), torch.empty_like(h)
            _check(L.mm_moe_permute(h.data_ptr(), src.data_ptr(), x.data_ptr(), T, H, st), "gather_rows")
        chunk = min(chunk, T)
        logits = torch.empty(chunk, V, dtype=torch.bfloat16, device=dev)
        dw_acc = None
        n_chunks = (T + chunk - 1) // chunk
        for c in range(n_chunks):
            a, b = c * chunk, min(T, (c + 1) * chunk)
            z = logits[: b - a]
            if listed:
                _gemm_rows(x[a:b], w_, z, 0, 0, count, a)
            else:
                gemm_nt(x[a:b], w_, out=z)
            _check(L.mm_ce_fwd_bwd(z.data_ptr(), z.stride(0), labels.data_ptr() if listed else labels[a:b].data_ptr(), row_loss[a:b].data_ptr(),
                                   b - a, V, ignore_index, src.data_ptr() if listed else None, count.data_ptr() if listed else None, a, st),
                   "ce_fwd_bwd")
            out = dw if n_chunks == 1 else torch.empty_like(dw)
            if listed:
                _gemm_rows(z, w_, dx[a:b], 0, 1, count, a)
                _gemm_rows(z, x[a:b], out, 1, 1, count, a)
            else:
                gemm_nn(z, w_, out=dx[a:b])
                gemm_tn(z, x[a:b], out=out)
            if n_chunks > 1:
                dw_acc = out.float() if dw_acc is None else dw_acc.add_(out)
        if dw_acc is not None:
            dw.copy_(dw_acc)
        if listed:
            _check(L.mm_moe_permute(dx.data_ptr(), row.data_ptr(), dh.data_ptr(), T, H, st), "scatter_rows")
        ctx.save_for_backward(dh, dw)
        return row_loss.sum()

    @staticmethod
    def backward(ctx, g):
        dh, dw = ctx.saved_tensors
        if torch.is_grad_enabled():          # create_graph: the scaling itself is differentiated
            gs = g.to(dh.dtype)
            return dh.mul_(gs), dw.mul_(gs), None, None, None
        gs = g.float().reshape(1)
        for t in (dh, dw):
            _check(lib().mm_scale_bf16(t.data_ptr(), t.numel(), gs.data_ptr(), _st()), "scale_bf16")
        # written behind autograd's back: a second backward through the same forward stays an error
        torch.autograd.graph.increment_version((dh, dw))
        return dh, dw, None, None, None


def linear_cross_entropy(h, w, labels, ignore_index=-100, chunk=8192):
    loss = _LinearCE.apply(h, w, labels, ignore_index, chunk)
    return loss, (labels != ignore_index).sum()


def grouped_gemm_supported(x, w) -> bool:
    return False      # the native MoE path works on the aligned layout: see moe_experts()


# --------------------------------------------------------------------------- MoE on the aligned layout
def moe_supported(tokens, gate_up, down) -> bool:
    return (os.environ.get("MM_B200_MOE", "1") == "1" and tokens.dtype == torch.bfloat16 and tokens.shape[-1] % 128 == 0
            and gate_up.shape[-1] % 256 == 0 and down.shape[-1] % 128 == 0)


class _Route(torch.autograd.Function):
    """Routing kernels as an autograd function, so that a tracer records them (there is nothing to differentiate)."""

    @staticmethod
    def forward(ctx, topk_ids, num_experts):
        T, k = topk_ids.shape
        dev, n = topk_ids.device, T * k
        ids = topk_ids.to(torch.int64).contiguous()
        R = (n + num_experts * 127 + 127) // 128 * 128            # static upper bound of off[E]
        off = torch.empty(num_experts + 1, dtype=torch.int32, device=dev)
        scratch = torch.empty(lib().mm_moe_route_scratch(n, num_experts), dtype=torch.int32, device=dev)
        rows = torch.zeros(n + 1, dtype=torch.int32, device=dev)                    # rows of the pairs, out-of-range flag
        row_of_pair, bad = rows[:n], rows[n:]
        src_of_row = torch.empty(R, dtype=torch.int32, device=dev)
        _check(lib().mm_moe_route(ids.data_ptr(), n, k, num_experts, R, scratch.data_ptr(), off.data_ptr(), row_of_pair.data_ptr(),
                                  src_of_row.data_ptr(), bad.data_ptr(), _st()), "moe_route")
        return off, row_of_pair, src_of_row, bad


def _route(topk_ids, num_experts: int):
    """Launches the routing kernels; returns (off, row_of_pair, src_of_row, R, check).  ``check()`` waits for them (not for
    work queued behind them) and raises if an expert number was out of range."""
    off, row_of_pair, src_of_row, flag = _run(_Route, topk_ids, int(num_experts))
    R = src_of_row.shape[0]
    bad = torch.empty(1, dtype=torch.int32, pin_memory=True)
    bad.copy_(flag, non_blocking=True)
    done = torch.cuda.Event()
    done.record()

    def check():
        done.synchronize()
        if int(bad):
            raise RuntimeError(f"expert numbers outside [0, {num_experts})")
    return off, row_of_pair, src_of_row, R, check


def aligned_routing(topk_ids, num_experts: int):
    """Plan of the aligned expert-major layout: every expert's rows start at a multiple of 128.  Returns (off [E+1] int32,
    row_of_pair [T*k] int32, src_of_row [R] int32 (-1 = pad), R)."""
    off, row_of_pair, src_of_row, R, check = _route(topk_ids, num_experts)
    check()
    return off, row_of_pair, src_of_row, R


class _AlignedPermute(torch.autograd.Function):
    @staticmethod
    def forward(ctx, tokens, src_of_row, row_of_pair, k):
        R, H = src_of_row.numel(), tokens.shape[1]
        out = torch.empty(R, H, dtype=tokens.dtype, device=tokens.device)
        _check(lib().mm_moe_permute(tokens.contiguous().data_ptr(), src_of_row.data_ptr(), out.data_ptr(), R, H, _st()),
               "moe_permute")
        ctx.save_for_backward(row_of_pair)
        ctx.k, ctx.T = k, tokens.shape[0]
        return out

    @staticmethod
    def backward(ctx, g):
        (row_of_pair,) = ctx.saved_tensors
        out = torch.empty(ctx.T, g.shape[1], dtype=g.dtype, device=g.device)
        _check(lib().mm_moe_unpermute(g.contiguous().data_ptr(), row_of_pair.data_ptr(), None, out.data_ptr(),
                                      ctx.T, ctx.k, g.shape[1], _st()), "moe_unpermute")
        return out, None, None, None


class _AlignedUnpermute(torch.autograd.Function):
    """``src_of_row`` names the pad rows of ``y`` (they get zero gradients); None: every row belongs to a pair."""

    @staticmethod
    def forward(ctx, y, row_of_pair, probs, src_of_row=None):
        T, k = probs.shape
        y = y.contiguous()
        out = torch.empty(T, y.shape[1], dtype=y.dtype, device=y.device)
        pc = probs.to(y.dtype).contiguous()
        _check(lib().mm_moe_unpermute(y.data_ptr(), row_of_pair.data_ptr(), pc.data_ptr(), out.data_ptr(), T, k,
                                      y.shape[1], _st()), "moe_unpermute")
        ctx.save_for_backward(y, row_of_pair, pc, src_of_row)
        return out

    @staticmethod
    def backward(ctx, g):
        y, row_of_pair, probs, src_of_row = ctx.saved_tensors
        T, k = probs.shape
        if torch.is_grad_enabled():          # create_graph: the gradient itself is differentiated
            ge = g.repeat_interleave(k, dim=0)
            dy = torch.zeros_like(y).index_copy(0, row_of_pair.long(), ge * probs.reshape(-1, 1))
            return dy, None, (ge.float() * y[row_of_pair.long()].float()).sum(-1).view(T, k).to(probs.dtype), None
        g = _dense(g)
        dy = torch.empty_like(y)
        dprobs = torch.empty_like(probs)
        _check(lib().mm_moe_unpermute_bwd(g.data_ptr(), y.data_ptr(), row_of_pair.data_ptr(),
                                          None if src_of_row is None else src_of_row.data_ptr(), probs.data_ptr(),
                                          dy.data_ptr(), dprobs.data_ptr(), T, k, y.shape[0], y.shape[1], _st()),
               "moe_unpermute_bwd")
        return dy, None, dprobs, None


def _grouped_raw(a, b, c, off, mode, K, N, E):
    _check(lib().mm_grouped_gemm_bf16(a.data_ptr(), b.data_ptr(), c.data_ptr(), off.data_ptr(), a.shape[0], E, K, N, mode,
                                      status_word(a.device).data_ptr(), _st()), "grouped_gemm")


class _AlignedGroupedGemm(torch.autograd.Function):
    """x [R, K] (aligned expert-major rows) x W [E, K, N] -> [R, N]; all three passes on tcgen05."""

    @staticmethod
    def forward(ctx, x, w, off):
        E, K, N = w.shape
        x = x.contiguous()
        y = torch.empty(x.shape[0], N, dtype=x.dtype, device=x.device)
        _grouped_raw(x, w, y, off, 0, K, N, E)
        ctx.save_for_backward(x, w, off)
        return y

    @staticmethod
    def backward(ctx, g):
        x, w, off = ctx.saved_tensors
        E, K, N = w.shape
        g = g.contiguous()
        dx = torch.empty_like(x)
        _grouped_raw(g, w, dx, off, 1, K, N, E)
        dw = torch.empty(E, K, N, dtype=w.dtype, device=w.device)
        _grouped_raw(x, g, dw, off, 2, K, N, E)
        return dx, dw, None


def moe_experts(tokens, topk_ids, probs, gate_up, down):
    """Routed SwiGLU experts: permute -> grouped GEMM -> SwiGLU -> grouped GEMM -> weighted un-permute."""
    E = gate_up.shape[0]
    off, row_of_pair, src_of_row, _, check = _route(topk_ids, E)
    x = _run(_AlignedPermute, tokens, src_of_row, row_of_pair, topk_ids.shape[1])
    h = _run(_AlignedGroupedGemm, x, gate_up, off)
    y = _run(_AlignedGroupedGemm, swiglu(h), down, off)
    out = _run(_AlignedUnpermute, y, row_of_pair, probs, src_of_row)
    check()                      # the routing is long done by now: the products queued behind it keep the GPU busy
    return out


# --------------------------------------------------------------------------- GDN
def _seq_bounds(cu_seqlens, T, device):
    """Per-token first index and one-past-last index of its sequence (int32 [T] each)."""
    if cu_seqlens is None:
        return (torch.zeros(T, dtype=torch.int32, device=device), torch.full((T,), T, dtype=torch.int32, device=device))
    cu = torch.as_tensor(cu_seqlens, device=device).to(torch.int64)
    seg = torch.bucketize(torch.arange(T, device=device), cu[1:], right=True)
    return cu[seg].int().contiguous(), cu[seg + 1].int().contiguous()


class _CausalConv1d(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, cu_seqlens, silu):
        T, D = x.shape
        K = w.shape[-1]
        # the convolution's columns of a fused projection are read where they are
        if x.stride(1) != 1 or _pitch(x) % 8 or x.data_ptr() % 16:
            x = _dense(x)
        w = w.contiguous()
        start, end = _seq_bounds(cu_seqlens, T, x.device)
        y = torch.empty(T, D, dtype=x.dtype, device=x.device)
        _check(lib().mm_conv1d_fwd(x.data_ptr(), _pitch(x), w.data_ptr(), start.data_ptr(), y.data_ptr(), T, D, K, int(silu), _st()),
               "conv1d_fwd")
        ctx.save_for_backward(x, w, start, end)
        ctx.silu = silu
        return y

    @staticmethod
    def backward(ctx, dy):
        x, w, start, end = ctx.saved_tensors
        T, D = x.shape
        K = w.shape[-1]
        dy = _dense(dy)
        dx = torch.empty(T, D, dtype=x.dtype, device=x.device)
        dw = torch.zeros(D, K, dtype=torch.float32, device=x.device)
        _check(lib().mm_conv1d_bwd(x.data_ptr(), _pitch(x), w.data_ptr(), start.data_ptr(), end.data_ptr(), dy.data_ptr(),
                                   dx.data_ptr(), dw.data_ptr(), T, D, K, int(ctx.silu), _st()), "conv1d_bwd")
        return dx, dw.to(w.dtype), None, None


def conv1d_supported(x, w) -> bool:
    return x.dim() == 2 and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and x.shape[1] % 8 == 0 \
        and w.shape[-1] <= 8


def causal_conv1d(x, w, activation, cu_seqlens):
    return _run(_CausalConv1d, x, w, cu_seqlens, activation == "silu")


class _L2Norm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, eps):
        D = x.shape[-1]
        x2 = x.reshape(-1, D).contiguous()
        y = torch.empty_like(x2)
        r = torch.empty(x2.shape[0], dtype=torch.float32, device=x.device)
        fn = lib().mm_l2norm_fwd if (D % 8 or not _row_group(D)) else lib().mm_rownorm_l2_fwd
        _check(fn(x2.data_ptr(), y.data_ptr(), r.data_ptr(), x2.shape[0], D, eps, _st()), "l2norm_fwd")
        ctx.save_for_backward(y, r)
        return y.view(x.shape)

    @staticmethod
    def backward(ctx, dy):
        y, r = ctx.saved_tensors
        D = y.shape[-1]
        dy2 = dy.reshape(-1, D).contiguous()
        dx = torch.empty_like(y)
        _check(lib().mm_l2norm_bwd(y.data_ptr(), dy2.data_ptr(), r.data_ptr(), dx.data_ptr(), y.shape[0], D, _st()),
               "l2norm_bwd")
        return dx.view(dy.shape), None


def l2_norm(x, eps=1e-6):
    return _run(_L2Norm, x, eps)


class _DeltaHeads(torch.autograd.Function):
    """``q | k | v`` columns to the delta rule's heads: q and k L2-normalised and repeated, v as it is, each dense."""

    @staticmethod
    def forward(ctx, x, hk, hv, dv, eps):
        T, dev = x.shape[0], x.device
        q, k = (torch.empty(T, hv, 128, dtype=torch.bfloat16, device=dev) for _ in range(2))
        v = torch.empty(T, hv, dv, dtype=torch.bfloat16, device=dev)
        r = torch.empty(T, 2 * hk, dtype=torch.float32, device=dev)
        _check(lib().mm_delta_heads_fwd(x.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), r.data_ptr(), T, hk, hv // hk, hv * dv,
                                        eps, _st()), "delta_heads_fwd")
        ctx.save_for_backward(q, k, r)
        return q, k, v

    @staticmethod
    def backward(ctx, dq, dk, dv):
        q, k, r = ctx.saved_tensors
        T, hk, v_width = q.shape[0], r.shape[1] // 2, dv.shape[1] * dv.shape[2]
        dq, dk, dv = _dense(dq), _dense(dk), _dense(dv)
        dx = torch.empty(T, 2 * hk * 128 + v_width, dtype=torch.bfloat16, device=q.device)
        _check(lib().mm_delta_heads_bwd(q.data_ptr(), k.data_ptr(), r.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(),
                                        dx.data_ptr(), T, hk, q.shape[1] // hk, v_width, _st()), "delta_heads_bwd")
        if torch.is_grad_enabled():          # create_graph: the values' columns are dv itself
            dx = torch.cat([dx[:, :2 * hk * 128], dv.reshape(T, v_width)], 1)
        return dx, None, None, None, None


def delta_heads_supported(x, hk, hv, dk, dv) -> bool:
    return (x.dim() == 2 and x.dtype == torch.bfloat16 and dk == 128 and hv % hk == 0 and dv % 8 == 0 and x.is_contiguous()
            and x.data_ptr() % 16 == 0 and x.shape[1] == 2 * hk * dk + hv * dv)


def delta_heads(x, hk, hv, dv, eps=1e-6):
    return _run(_DeltaHeads, x, hk, hv, dv, eps)


def _gate_rows(z, D):
    """The gate as the kernels read it: (tensor, rows a token, elements between tokens).  [tokens, heads, D] with dense heads may have
    its tokens apart (the gate's columns of a fused projection); anything else is dense rows."""
    st = z.stride()
    if len(st) == 3 and st[2] == 1 and st[1] == D and st[0] % 8 == 0 and z.data_ptr() % 16 == 0 and z.shape[0] * z.shape[1] < 2 ** 31:
        return z, max(1, z.shape[1]), st[0]
    return _dense(z.reshape(-1, D)), 1, D


class _GatedRMSNorm(torch.autograd.Function):
    """``rmsnorm(x) * w * silu(z)`` over the last dim (<= 256): x fp32 or bf16, z / w / result bf16."""

    @staticmethod
    def forward(ctx, x, z, w, eps):
        D = x.shape[-1]
        x2, wc = _dense(x.reshape(-1, D)), _dense(w)
        rows = x2.shape[0]
        z2, zh, ldz = _gate_rows(z, D)
        y = torch.empty(rows, D, dtype=torch.bfloat16, device=x.device)
        rstd = torch.empty(rows, dtype=torch.float32, device=x.device)
        _check(lib().mm_gated_rms_fwd(x2.data_ptr(), int(x2.dtype == torch.float32), z2.data_ptr(), wc.data_ptr(), y.data_ptr(),
                                      rstd.data_ptr(), rows, D, zh, ldz, eps, _st()), "gated_rms_fwd")
        ctx.save_for_backward(x2, z2, wc, rstd)
        ctx.shapes = (x.shape, z.shape)
        return y.view(z.shape)

    @staticmethod
    def backward(ctx, dy):
        x2, z2, wc, rstd = ctx.saved_tensors
        rows, D = x2.shape
        z2, zh, ldz = _gate_rows(z2, D)        # read off what was saved: a hook (offload to the host) gives back a dense copy
        dy2 = _dense(dy.reshape(rows, D))
        dx, dz = torch.empty_like(x2), torch.empty(rows, D, dtype=z2.dtype, device=z2.device)
        dw = torch.zeros(D, dtype=torch.float32, device=x2.device)
        _check(lib().mm_gated_rms_bwd(x2.data_ptr(), int(x2.dtype == torch.float32), z2.data_ptr(), wc.data_ptr(), dy2.data_ptr(),
                                      rstd.data_ptr(), dx.data_ptr(), dz.data_ptr(), dw.data_ptr(), rows, D, zh, ldz, _st()),
               "gated_rms_bwd")
        return dx.view(ctx.shapes[0]), dz.view(ctx.shapes[1]), dw.to(wc.dtype), None


def gated_rms_norm(x, z, w, eps=1e-6):
    return _run(_GatedRMSNorm, x, z, w, eps)


def gdn_supported(q, v, chunk) -> bool:
    from . import gdn
    lib()
    return _STATUS.get("mm_gdn_fwd", False) and gdn.supported(q, v, chunk)


def gated_delta_rule_varlen(q, k, v, g, beta, cu_seqlens, chunk, scale):
    from . import gdn
    return gdn.gated_delta_rule_varlen(q, k, v, g, beta, cu_seqlens, scale)
