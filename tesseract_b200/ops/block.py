"""A pre-norm decoder block as one autograd function: the launches of ``rms_norm``, ``linear``, ``rope_qkv``, ``flash_attention_packed`` and
``swiglu`` in the same order, issued by one native call per direction (``csrc/decoder_block.cu``; two backward, between which memory is given back). For training on CUDA with weights and
gradients in an arena; ``nn.TransformerBlock`` decides when it stands for the modules that it takes the place of."""
from __future__ import annotations

import ctypes

import torch

from .. import _native
from .._native import check, lib, stream_ptr
from .attention import _native_flash_available
from .gemm import _use_native

_native.register_signatures({
    "tsb_block_bytes": [_native.P, _native.I, _native.P],
    "tsb_block_forward": [_native.P, _native.P, _native.P, _native.I, _native.P],
    "tsb_block_backward": [_native.P, _native.P, _native.P, _native.I, _native.I, _native.I, _native.P],
})

_Shape, _Floats, _Bytes = ctypes.c_longlong * 7, ctypes.c_float * 3, ctypes.c_longlong * 4
_Fwd, _Bwd = ctypes.c_longlong * 14, ctypes.c_longlong * 23
LAUNCHES_FORWARD, LAUNCHES_BACKWARD = 9, 17     # backward: eight products, SwiGLU, rotation, three of attention, two per norm


def _ptr(t) -> int:
    return 0 if t is None else t.data_ptr()


def _rows(t: torch.Tensor) -> torch.Tensor:
    """Contiguous rows that start on 16 bytes."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


_SAVED_TYPES = (torch.bfloat16, torch.uint8, torch.uint8, torch.bfloat16)
_CAN_LET_GO = hasattr(torch.autograd.function.BackwardCFunction, "maybe_clear_saved_tensors")


def _kept(t: torch.Tensor, size: int, dtype: torch.dtype, device: torch.device) -> torch.Tensor:
    """A tensor that is somewhere else than in the forward pass (a hook on saved tensors brought it back, a weight's storage was exchanged), as the
    kernels read it."""
    if t.nbytes != size or t.dtype is not dtype or t.device != device:
        raise RuntimeError(f"decoder_block: a tensor kept for the backward pass came back as {tuple(t.shape)} {t.dtype} on {t.device} instead "
                           f"of {size} bytes of {dtype} on {device}")
    return _rows(t)


def _weight_bytes(B, S, W, H, Hkv, D, F):
    kv = 2 * Hkv * D * W
    return 2 * W, 2 * W * W, 2 * W * W, 2 * W, 2 * F * W, 2 * W * F, kv, kv, 2 * F * W


def _stack(*parts: torch.Tensor) -> torch.Tensor:
    """Matrices one behind the other in memory: the first where they lie so, else a copy."""
    at = parts[0].data_ptr()
    for t in parts:
        if t.data_ptr() != at:
            return torch.cat(parts)
        at += t.nbytes
    return parts[0]


class _BlockFn(torch.autograd.Function):
    """(out, res2) of x and the residual stream. ``weights`` and ``grads``: norm_1, q / k / v, o, norm_2, gate / up, down; of the stacked
    ones the first, which the others (``behind``: k, v, up, and their gradients) follow in memory. Activations are saved; weights, which the model
    holds anyway, are only kept: a hook on saved tensors would copy the tensor it is given and not what lies behind it."""

    @staticmethod
    def forward(ctx, x, res, norm_1, q, o, norm_2, gate, down, grads, behind, cos, sin, shape, floats, causal):
        ctx.set_materialize_grads(False)
        x = _rows(x)
        if res is not None:
            res = _rows(res)
        shape, floats = _Shape(*shape), _Floats(*floats)
        sizes = _Bytes()
        if lib().tsb_block_bytes(shape, int(res is not None), sizes) != 0:
            raise ValueError("decoder_block: a shape that the kernels do not serve")
        saved = torch.empty(sizes[0], device=x.device, dtype=torch.uint8)
        mid = torch.empty(sizes[1], device=x.device, dtype=torch.uint8)
        res2, out = torch.empty_like(x), torch.empty_like(x)
        weights = (norm_1, q, o, norm_2, gate, down)
        args = _Fwd(x.data_ptr(), _ptr(res), *(w.data_ptr() for w in weights), cos.data_ptr(), sin.data_ptr(), saved.data_ptr(),
                    mid.data_ptr(), res2.data_ptr(), out.data_ptr())
        check(lib().tsb_block_forward(shape, args, floats, int(causal), stream_ptr(x.device)), "tsb_block_forward")
        _native.add_launches(LAUNCHES_FORWARD - 1)
        keep = (res2, saved, mid) if res is not None else (res2, saved, mid, x)
        ctx.save_for_backward(*keep)
        ctx.saved_as = [t.data_ptr() for t in keep], [t.nbytes for t in keep]
        ctx.weights, ctx.versions = (*weights, *behind[:3]), (norm_1._version, o._version, norm_2._version, down._version)
        ctx.weights_at = [w.data_ptr() for w in ctx.weights]
        ctx.tables, ctx.grads, ctx.behind, ctx.args = (cos, sin), grads, behind[3:], (shape, floats, causal, sizes)
        return out, res2

    @staticmethod
    def backward(ctx, dout, dres2):
        back, (at, sizes) = ctx.saved_tensors, ctx.saved_as
        if [t.data_ptr() for t in back] != at or [t.nbytes for t in back] != sizes or not all([t.is_contiguous() for t in back]):
            device = (dres2 if dout is None else dout).device
            back = [_kept(t, size, dtype, device) for t, size, dtype in zip(back, sizes, _SAVED_TYPES)]
        res2, saved, mid, *x = back
        norm_1, q, o, norm_2, gate, down, k, v, up = weights = ctx.weights
        if (norm_1._version, o._version, norm_2._version, down._version) != ctx.versions:
            raise RuntimeError("decoder_block: a weight needed for gradient computation has been modified by an inplace operation")
        if [w.data_ptr() for w in weights] != ctx.weights_at:
            norm_1, q, o, norm_2, gate, down, k, v, up = (_kept(w, n, torch.bfloat16, res2.device)
                                                          for w, n in zip(weights, _weight_bytes(*ctx.args[0])))
            q, gate = _stack(q, k, v), _stack(gate, up)
        shape, floats, causal, (_, _, wide_bytes, rest_bytes) = ctx.args
        cos, sin = ctx.tables
        dout = torch.zeros_like(res2) if dout is None else _rows(dout)
        if dres2 is not None:
            dres2 = _rows(dres2)
        stream, has_res, causal = stream_ptr(res2.device), int(not x), int(causal)
        wide = torch.empty(wide_bytes, device=res2.device, dtype=torch.uint8)
        args = _Bwd(x[0].data_ptr() if x else 0, norm_1.data_ptr(), q.data_ptr(), o.data_ptr(), norm_2.data_ptr(), gate.data_ptr(), down.data_ptr(),
                    cos.data_ptr(), sin.data_ptr(), saved.data_ptr(), mid.data_ptr(), res2.data_ptr(), *[g.data_ptr() for g in ctx.grads],
                    dout.data_ptr(), _ptr(dres2), wide.data_ptr())
        check(lib().tsb_block_backward(shape, args, floats, has_res, causal, 1, stream), "tsb_block_backward")
        # unless the graph is kept for another pass, the widest activations go back to the allocator here, as they do between modules
        back = mid = None
        if _CAN_LET_GO:
            ctx.maybe_clear_saved_tensors()
        rest = torch.empty(rest_bytes, device=res2.device, dtype=torch.uint8)
        dx = torch.empty_like(res2)
        args[21], args[22] = rest.data_ptr(), dx.data_ptr()
        check(lib().tsb_block_backward(shape, args, floats, has_res, causal, 2, stream), "tsb_block_backward")
        _native.add_launches(LAUNCHES_BACKWARD - 2)
        return (dx, None if x else dx) + (None,) * 13


def block_kernels_ok(x: torch.Tensor) -> bool:
    """The settings choose the native product and attention, and the library has this file's entry points."""
    return _use_native(x) and _native_flash_available() and hasattr(lib(), "tsb_block_forward")


def decoder_block(x, res, weights, grads, cos, sin, shape, floats, causal, behind=None):
    """``(out, x [+ res] + attention)``; ``shape`` is (B, S, W, H, Hkv, D, F), ``floats`` both norms' eps and the softmax scale. The gradients of
    ``weights`` are added to ``grads``; both, and ``behind``, as in ``_BlockFn``."""
    if behind is None:
        _, _, W, H, Hkv, D, F = shape
        with torch.no_grad():
            behind = [torch.as_strided(t[i], (rows, W), (W, 1), t[i].storage_offset() + first * W)
                      for t in (weights, grads) for i, first, rows in ((1, H * D, Hkv * D), (1, (H + Hkv) * D, Hkv * D), (4, F, F))]
    return _BlockFn.apply(x, res, *weights, grads, behind, cos, sin, shape, floats, causal)
