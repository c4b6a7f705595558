"""Linear layers of the trunk under bf16 autocast without the per-call casts.

``torch.autocast`` casts every fp32 weight and bias to bf16 inside each ``F.linear`` call and casts every weight /
bias gradient back to fp32 afterwards: for the trunk of the reference (``AdaLNBlock``, models/transformer.py:228-316,
five Linear layers per block) that is some 600 small cast kernels per training step, a quarter of all launches once the
batch is split over eight GPUs.  Here each parameter keeps a bf16 copy that is refreshed for all layers at once at the
start of a forward pass (one multi-tensor copy), and the backward pass writes the weight gradient in fp32 straight out of
the GEMM and the bias gradient comes from this library's column-sum kernels (``mf_column_sums``: one read of the output
gradient, fixed order of additions).  The GEMMs themselves stay library calls (cuBLAS).
"""
from __future__ import annotations

from typing import Iterable, Optional, Sequence

import torch
import torch.nn.functional as F

from .fused import column_sums, column_sums_applies, gelu_tanh_applies, gelu_tanh_backward, gelu_tanh_forward

_SHADOW = "_mf_bf16_copy"  # attribute on the parameter: (bf16 tensor, parameter version it was made from)


def _bf16_autocast() -> bool:
    return torch.is_autocast_enabled("cuda") and torch.get_autocast_dtype("cuda") == torch.bfloat16


def linear_bf16_applies(x: torch.Tensor, weight: torch.Tensor) -> bool:
    """CUDA, an fp32 parameter, and bf16 arithmetic asked for (autocast or a bf16 input)."""
    return x.is_cuda and weight.is_cuda and weight.dtype == torch.float32 and (x.dtype == torch.bfloat16 or _bf16_autocast())


def _current(p: torch.Tensor) -> Optional[torch.Tensor]:
    entry = getattr(p, _SHADOW, None)
    if entry is None:
        return None
    copy, version = entry
    if version != p._version or copy.device != p.device or copy.shape != p.shape:
        return None
    return copy


def bf16_copy(p: torch.Tensor) -> torch.Tensor:
    """The parameter's bf16 copy, refreshed if the parameter changed since it was made."""
    copy = _current(p)
    if copy is None:
        entry = getattr(p, _SHADOW, None)
        copy = entry[0] if entry is not None and entry[0].device == p.device and entry[0].shape == p.shape else None
        with torch.no_grad():
            if copy is None:
                copy = p.detach().to(torch.bfloat16)
            else:
                copy.copy_(p.detach())
        setattr(p, _SHADOW, (copy, p._version))
    return copy


def has_bf16_copy(p: torch.Tensor) -> bool:
    return getattr(p, _SHADOW, None) is not None


def refresh_bf16_copies(params: Iterable[torch.Tensor], *, force: bool = False) -> None:
    """Bring the bf16 copies of ``params`` up to date with one multi-tensor copy.  ``force`` copies even when the version
    counters say nothing changed: a step captured in a CUDA graph must contain the copy, because a replay updates the
    parameters without running this Python code again."""
    stale_dst, stale_src = [], []
    for p in params:
        if p is None or not p.is_cuda or p.dtype != torch.float32:
            continue
        entry = getattr(p, _SHADOW, None)
        if entry is None or entry[0].device != p.device or entry[0].shape != p.shape:
            bf16_copy(p)  # first use: allocates
            if not force:
                continue
            entry = getattr(p, _SHADOW)
        if force or entry[1] != p._version:
            stale_dst.append(entry[0])
            stale_src.append(p.detach())
            setattr(p, _SHADOW, (entry[0], p._version))
    if stale_dst:
        with torch.no_grad():
            torch._foreach_copy_(stale_dst, stale_src)


_REFRESH_IN_CAPTURE = True


class no_refresh_in_capture:
    """For a captured evaluation whose owner brings the bf16 copies up to date itself, before each replay."""

    def __enter__(self):
        global _REFRESH_IN_CAPTURE
        self._before, _REFRESH_IN_CAPTURE = _REFRESH_IN_CAPTURE, False

    def __exit__(self, *exc):
        global _REFRESH_IN_CAPTURE
        _REFRESH_IN_CAPTURE = self._before


def refresh_must_be_captured() -> bool:
    return _REFRESH_IN_CAPTURE and torch.cuda.is_current_stream_capturing()


def stacked_bf16_copies(params: Sequence[torch.Tensor], stack: Optional[torch.Tensor]) -> torch.Tensor:
    """The bf16 copies of equally shaped parameters as one contiguous tensor, (len(params) * rows, ...): each parameter's
    copy is a view of it, so refreshing the copies refreshes the stack.  ``stack`` is returned as it is while it still holds
    them.  Freshly placed copies are filled by the next :func:`refresh_bf16_copies`, or here where that does not follow."""
    rows, first = params[0].shape[0], params[0]
    if stack is not None and stack.device == first.device:
        for i, p in enumerate(params):
            entry = getattr(p, _SHADOW, None)
            if entry is None or entry[0].data_ptr() != stack[i * rows :].data_ptr() or entry[0].shape != p.shape:
                break
        else:
            return stack
    with torch.no_grad():
        stack = torch.cat([p.detach().to(torch.bfloat16) for p in params])
    for i, p in enumerate(params):
        setattr(p, _SHADOW, (stack[i * rows : (i + 1) * rows], p._version))
    return stack


class _StackedModulation(torch.autograd.Function):
    """The adaptive-LayerNorm modulations of all layers from the one conditioning vector they share: one GEMM forward, three
    products backward, instead of those per layer.  ``params``: the layers' weights, then their biases."""

    @staticmethod
    def forward(ctx, x, weights, biases, layers, *params):
        with torch.autocast("cuda", enabled=False):
            mod = F.linear(x, weights, biases)
        B, C = x.shape[0], mod.shape[1] // (6 * layers)
        out = torch.empty((6 * layers, B, C), device=x.device, dtype=torch.float32)
        out.copy_(mod.view(B, 6 * layers, C).transpose(0, 1))
        ctx.save_for_backward(x, weights)
        ctx.layers = layers
        return tuple(out.unbind(0))

    @staticmethod
    def backward(ctx, *grads):
        x, weights = ctx.saved_tensors
        like = next(g for g in grads if g is not None)
        g = torch.stack([t if t is not None else torch.zeros_like(like) for t in grads], dim=1)  # (B, 6 L, C) fp32
        g = g.reshape(g.shape[0], -1).to(torch.bfloat16)
        with torch.autocast("cuda", enabled=False):
            dx = torch.mm(g, weights) if ctx.needs_input_grad[0] else None
            dw = _mm_f32(g.t(), x)
        db = column_sums(g) if column_sums_applies(g) else g.sum(0, dtype=torch.float32)
        return (dx, None, None, None, *dw.chunk(ctx.layers), *db.chunk(ctx.layers))


def stacked_modulation(x: torch.Tensor, weights: torch.Tensor, biases: torch.Tensor, params: Sequence[torch.Tensor],
                       layers: int) -> list:  # fmt: skip
    """Per layer the six fp32 (B, C) tensors ``shift_a, scale_a, gate_a, shift_m, scale_m, gate_m``; ``weights`` / ``biases``
    are the stacked bf16 copies of ``params``."""
    out = _StackedModulation.apply(x, weights, biases, layers, *params)
    return [out[6 * i : 6 * i + 6] for i in range(layers)]


_MM_OUT_DTYPE = True  # torch.mm(..., out_dtype=) exists; cleared on the first refusal


def _mm_f32(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    """a @ b for bf16 operands with the fp32 accumulator written out unrounded."""
    global _MM_OUT_DTYPE
    if _MM_OUT_DTYPE:
        try:
            return torch.mm(a, b, out_dtype=torch.float32)
        except (TypeError, RuntimeError):
            _MM_OUT_DTYPE = False
    return torch.mm(a, b).float()


class _LinearBf16(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias):
        w16 = bf16_copy(weight)
        b16 = bf16_copy(bias) if bias is not None else None
        ctx.save_for_backward(x, w16)
        ctx.has_bias = bias is not None
        with torch.autocast("cuda", enabled=False):
            return F.linear(x, w16, b16)

    @staticmethod
    def backward(ctx, dy):
        x, w16 = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1])
        if dy2.dtype != torch.bfloat16:
            dy2 = dy2.to(torch.bfloat16)
        dx = dw = db = None
        with torch.autocast("cuda", enabled=False):
            if ctx.needs_input_grad[0]:
                dx = torch.mm(dy2, w16).view(x.shape)
            if ctx.needs_input_grad[1]:
                dw = _mm_f32(dy2.t(), x.reshape(-1, x.shape[-1]))
            if ctx.has_bias and ctx.needs_input_grad[2]:
                dyc = dy2 if dy2.is_contiguous() else dy2.contiguous()
                db = column_sums(dyc) if column_sums_applies(dyc) else dyc.sum(0, dtype=torch.float32)
        return dx, dw, db


def linear_bf16(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor]) -> torch.Tensor:
    """``F.linear`` in bf16 on fp32 parameters (what autocast computes), returning bf16.  Falls back to ``F.linear``
    where :func:`linear_bf16_applies` says no.  A step that is captured into a CUDA graph and updates the parameters
    must call ``refresh_bf16_copies(params, force=True)`` inside the captured region before its first layer (the trunk
    does): the version counters this function checks do not advance during replays."""
    if not linear_bf16_applies(x, weight):
        return F.linear(x, weight, bias)
    if x.dtype != torch.bfloat16:
        x = x.to(torch.bfloat16)
    return _LinearBf16.apply(x, weight, bias)


class _LinearGeluBf16(torch.autograd.Function):
    """fc1 + GELU(tanh) of the block's MLP.  The backward pass forms the gradient of the pre-activation and the bias
    gradient in one sweep over (pre-activation, incoming gradient)."""

    @staticmethod
    def forward(ctx, x, weight, bias):
        w16 = bf16_copy(weight)
        b16 = bf16_copy(bias) if bias is not None else None
        with torch.autocast("cuda", enabled=False):
            pre = F.linear(x, w16, b16)
        ctx.save_for_backward(x, w16, pre)
        ctx.has_bias = bias is not None
        return gelu_tanh_forward(pre)

    @staticmethod
    def backward(ctx, dact):
        x, w16, pre = ctx.saved_tensors
        cols = pre.shape[-1]
        dact2 = dact.reshape(-1, cols)
        if dact2.dtype != torch.bfloat16:
            dact2 = dact2.to(torch.bfloat16)
        dpre, sums = gelu_tanh_backward(pre.reshape(-1, cols), dact2.contiguous())
        dx = dw = None
        with torch.autocast("cuda", enabled=False):
            if ctx.needs_input_grad[0]:
                dx = torch.mm(dpre, w16).view(x.shape)
            if ctx.needs_input_grad[1]:
                dw = _mm_f32(dpre.t(), x.reshape(-1, x.shape[-1]))
        return dx, dw, (sums if ctx.has_bias and ctx.needs_input_grad[2] else None)


def linear_gelu_bf16(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor]) -> torch.Tensor:
    """``gelu(F.linear(x, weight, bias), approximate="tanh")`` in bf16 on fp32 parameters; plain torch calls where
    :func:`linear_bf16_applies` says no."""
    if not (linear_bf16_applies(x, weight) and weight.shape[0] % 8 == 0):
        return F.gelu(F.linear(x, weight, bias), approximate="tanh")
    if x.dtype != torch.bfloat16:
        x = x.to(torch.bfloat16)
    return _LinearGeluBf16.apply(x.contiguous(), weight, bias)
