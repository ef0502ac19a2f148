"""A pre-norm decoder block as one autograd function: the launches of ``rms_norm``, ``linear``, ``rope_qkv``, ``flash_attention_packed`` and
``swiglu`` in the same order, issued by one native call per direction (``csrc/decoder_block.cu``). For training on CUDA with weights and
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
    "tsb_block_backward_down": [_native.P, _native.P, _native.P],
    "tsb_block_backward": [_native.P, _native.P, _native.P, _native.I, _native.I, _native.P],
})

_Shape, _Floats, _Bytes = ctypes.c_longlong * 7, ctypes.c_float * 3, ctypes.c_longlong * 4
_Fwd, _Down, _Bwd = ctypes.c_longlong * 14, ctypes.c_longlong * 5, ctypes.c_longlong * 19
LAUNCHES_FORWARD, LAUNCHES_BACKWARD = 9, 17     # backward: eight products, SwiGLU, rotation, three of attention, two per norm


def _ptr(t) -> int:
    return 0 if t is None else t.data_ptr()


def _rows(t: torch.Tensor) -> torch.Tensor:
    """Contiguous rows that start on 16 bytes."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


_KEPT_TYPES = (torch.bfloat16, torch.uint8, torch.uint8, torch.float32, torch.float32) + (torch.bfloat16,) * 10
_CAN_LET_GO = hasattr(torch.autograd.function.BackwardCFunction, "maybe_clear_saved_tensors")


def _kept(t: torch.Tensor, size: int, dtype: torch.dtype, device: torch.device) -> torch.Tensor:
    """A saved tensor that a hook has brought back somewhere else, as the kernels read it."""
    if t.nbytes != size or t.dtype is not dtype or t.device != device:
        raise RuntimeError(f"decoder_block: a saved tensor came back as {tuple(t.shape)} {t.dtype} on {t.device} instead of {size} bytes of {dtype} "
                           f"on {device}")
    return _rows(t)


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
    ones the first, which the others (``behind``: k, v, up, and their gradients) follow in memory. All are saved: a hook that copies what is
    saved copies the tensor it is given and not what lies behind it."""

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
        keep = (res2, saved, mid, cos, sin, *weights, *behind[:3]) + ((x,) if res is None else ())
        ctx.save_for_backward(*keep)
        ctx.kept = [t.data_ptr() for t in keep], [t.nbytes for t in keep]
        ctx.grads, ctx.behind, ctx.has_res, ctx.args = grads, behind[3:], res is not None, (shape, floats, causal, sizes)
        return out, res2

    @staticmethod
    def backward(ctx, dout, dres2):
        back, (at, sizes) = ctx.saved_tensors, ctx.kept
        if [t.data_ptr() for t in back] != at or [t.nbytes for t in back] != sizes or not all([t.is_contiguous() for t in back]):
            device = (dres2 if dout is None else dout).device
            back = [_kept(t, size, dtype, device) for t, size, dtype in zip(back, sizes, _KEPT_TYPES)]
        res2, saved, mid, cos, sin, norm_1, q, o, norm_2, gate, down, k, v, up, *x = back
        shape, floats, causal, (_, _, wide_bytes, rest_bytes) = ctx.args
        grads = [g.data_ptr() for g in ctx.grads]
        dout = torch.zeros_like(res2) if dout is None else _rows(dout)
        if dres2 is not None:
            dres2 = _rows(dres2)
        stream = stream_ptr(res2.device)
        wide = torch.empty(wide_bytes, device=res2.device, dtype=torch.uint8)
        args = _Down(down.data_ptr(), mid.data_ptr(), grads.pop(), dout.data_ptr(), wide.data_ptr())
        check(lib().tsb_block_backward_down(shape, args, stream), "tsb_block_backward_down")
        # unless the graph is kept for another pass, the widest activations go back to the allocator here, as they do between modules
        back = mid = None
        if _CAN_LET_GO:
            ctx.maybe_clear_saved_tensors()
        rest = torch.empty(rest_bytes, device=res2.device, dtype=torch.uint8)
        dx = torch.empty_like(res2)
        weights = (norm_1, _stack(q, k, v), o, norm_2, _stack(gate, up))
        args = _Bwd(x[0].data_ptr() if x else 0, *(w.data_ptr() for w in weights), cos.data_ptr(), sin.data_ptr(), saved.data_ptr(), res2.data_ptr(),
                    *grads, _ptr(dres2), wide.data_ptr(), rest.data_ptr(), dx.data_ptr())
        check(lib().tsb_block_backward(shape, args, floats, int(ctx.has_res), int(causal), stream), "tsb_block_backward")
        _native.add_launches(LAUNCHES_BACKWARD - 2)
        return (dx, dx if ctx.has_res else None) + (None,) * 13


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
