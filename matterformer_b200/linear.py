"""Linear layers of the trunk under bf16 autocast without the per-call casts.

``torch.autocast`` casts every fp32 weight and bias to bf16 inside each ``F.linear`` call and casts every weight /
bias gradient back to fp32 afterwards: for the trunk of the reference (``AdaLNBlock``, models/transformer.py:228-316,
five Linear layers per block) that is some 600 small cast kernels per training step, a quarter of all launches once the
batch is split over eight GPUs.  Here a forward pass makes the bf16 copies of all its layers at once (one multi-tensor
copy, :func:`bf16_copies`), and the backward pass writes the weight gradient in fp32 straight out of the GEMM and the
bias gradient comes from this library's column-sum kernels (``mf_column_sums``: one read of the output gradient, fixed
order of additions).  The GEMMs themselves stay library calls (cuBLAS).

The copies belong to the pass that made them.  They are not kept for the next one: a parameter's version counter does not
see every change (a replayed CUDA graph, a write through ``.data`` or through a flat buffer that the parameter is a view
of), so a copy that outlived its pass could not be told from a stale one.
"""
from __future__ import annotations

import contextlib
import threading
from typing import Iterable, Optional, Sequence

import torch
import torch.nn.functional as F

from . import _lib
from .fused import _ptr_array, column_sums, column_sums_applies, gelu_tanh_applies, gelu_tanh_backward, gelu_tanh_forward

_COPY = "_mf_bf16_copy"  # attribute on a parameter given to refresh_bf16_copies: (bf16 tensor, version it was made from)


def _bf16_autocast() -> bool:
    return torch.is_autocast_enabled("cuda") and torch.get_autocast_dtype("cuda") == torch.bfloat16


def linear_bf16_applies(x: torch.Tensor, weight: torch.Tensor) -> bool:
    """CUDA, an fp32 parameter, and bf16 arithmetic asked for (autocast or a bf16 input)."""
    return x.is_cuda and weight.is_cuda and weight.dtype == torch.float32 and (x.dtype == torch.bfloat16 or _bf16_autocast())


class _Pass(threading.local):
    """What the forward pass that this thread is in computes with."""

    copies: dict = {}  # id of a parameter -> (the parameter, its bf16 copy)
    kept: Optional["KeptBf16Copies"] = None


_PASS = _Pass()


def _takes_copy(p: Optional[torch.Tensor]) -> bool:
    return p is not None and p.is_cuda and p.dtype == torch.float32


class _CopySet:
    """bf16 copies of ``params`` and of the parameters of ``stacks``, made on construction and again by :meth:`refresh`.  They
    share one buffer, on 256-byte boundaries; a stack's lie one behind the other and are one matrix."""

    def __init__(self, params: Sequence[torch.Tensor], stacks: Sequence[Sequence[torch.Tensor]]) -> None:
        stacked = {id(p) for stack in stacks for p in stack}
        single = [p for p in params if _takes_copy(p) and id(p) not in stacked]
        device = next((p.device for p in (*single, *(stack[0] for stack in stacks))), None)
        whole = [p for p in single if p.numel() % 128 == 0 and p.device == device]
        other = [p for p in single if not (p.numel() % 128 == 0 and p.device == device)]
        self.params = [*whole, *other, *(p for stack in stacks for p in stack)]
        at = sum(p.numel() for p in whole)
        sizes = [sum(p.numel() for p in stack) for stack in stacks]
        with torch.no_grad():
            self.buffers = [torch.empty(p.shape, device=p.device, dtype=torch.bfloat16) for p in other]
            flat = torch.empty(at + sum(-(-n // 128) * 128 for n in sizes), device=device, dtype=torch.bfloat16)
            self.copies = [*torch._utils._unflatten_dense_tensors(flat[:at], whole), *self.buffers] if whole else list(self.buffers)
            self.buffers.append(flat)
            self.stacks = []
            for stack, n in zip(stacks, sizes):
                self.stacks.append(flat[at : at + n].view(-1, *stack[0].shape[1:]))
                self.copies += self.stacks[-1].split(stack[0].shape[0])
                at += -(-n // 128) * 128
        self.entries = {id(p): (p, c) for p, c in zip(self.params, self.copies)}
        self.refresh()

    def refresh(self) -> None:
        if self.params:
            with torch.no_grad():
                torch._foreach_copy_(self.copies, self.params)


class KeptBf16Copies:
    """Copies that outlive a pass, for the owner of a CUDA graph: ``with kept.in_use():`` around the warm-up and the capture of an
    evaluation makes its passes use (and on the first one make) the copies held here, and :meth:`refresh` brings them up to
    date before a replay, once for as many replays as the parameters stay as they are."""

    def __init__(self) -> None:
        self._sets: dict = {}

    def provide(self, params, stacks) -> _CopySet:
        key = (tuple(map(id, params)), tuple(tuple(map(id, stack)) for stack in stacks))
        if key not in self._sets:
            new = _CopySet(params, stacks)
            if torch.cuda.is_current_stream_capturing() or not all(isinstance(p, torch.nn.Parameter) for p in new.params):
                return new  # computed afresh by every pass, captured ones included
            self._sets[key] = new
        return self._sets[key]

    def refresh(self) -> None:
        for made in self._sets.values():
            made.refresh()
            for buffer in made.buffers:  # (allocated on the stream of the warm-up, read by the replays on this one)
                if buffer.is_cuda:
                    buffer.record_stream(torch.cuda.current_stream(buffer.device))

    @contextlib.contextmanager
    def in_use(self):
        outer, _PASS.kept = _PASS.kept, self
        try:
            yield
        finally:
            _PASS.kept = outer


@contextlib.contextmanager
def bf16_copies(params: Iterable[torch.Tensor], stacks: Sequence[Sequence[torch.Tensor]] = ()):
    """``with bf16_copies(params, stacks) as stacked:`` makes the bf16 copies that the :func:`linear_bf16` calls inside compute
    with.  ``stacks``: groups of equally shaped parameters whose copies are wanted as one matrix each, returned in ``stacked``.
    Seen by this thread alone, and by nothing after the block; what autograd saves keeps its own copies alive."""
    params, kept, outer = list(params), _PASS.kept, _PASS.copies
    made = kept.provide(params, stacks) if kept is not None else _CopySet(params, stacks)
    _PASS.copies = {**outer, **made.entries}
    try:
        yield made.stacks
    finally:
        _PASS.copies = outer


def bf16_copy(p: torch.Tensor) -> torch.Tensor:
    """The parameter in bf16: the enclosing pass's copy, else the one its owner refreshes, else a cast."""
    entry = _PASS.copies.get(id(p))
    if entry is not None and entry[0] is p:
        return entry[1]
    copy, version = getattr(p, _COPY, (None, None))
    if copy is not None and version == p._version and copy.device == p.device and copy.shape == p.shape:
        return copy
    return p.detach().to(torch.bfloat16)


def refresh_bf16_copies(params: Iterable[torch.Tensor], *, force: bool = False) -> None:
    """For callers of :func:`linear_bf16` with layers of their own: give ``params`` bf16 copies that stay with them, all made
    or brought up to date by one multi-tensor copy.  The caller vouches for them: without ``force`` only the parameters whose
    version counter has moved are copied, which misses changes made by a graph's replay or through ``.data``, and a step
    captured in a CUDA graph must contain a forced call.  (The trunk does not use these; see :func:`bf16_copies`.)"""
    stale_dst, stale_src = [], []
    for p in params:
        if not _takes_copy(p):
            continue
        copy, version = getattr(p, _COPY, (None, None))
        if copy is None or copy.device != p.device or copy.shape != p.shape:
            copy, version = torch.empty(p.shape, device=p.device, dtype=torch.bfloat16), None
        if force or version != p._version:
            stale_dst.append(copy)
            stale_src.append(p.detach())
            setattr(p, _COPY, (copy, p._version))
    if stale_dst:
        with torch.no_grad():
            torch._foreach_copy_(stale_dst, stale_src)


def _modulation_kernels_apply(mod: torch.Tensor, groups: int) -> bool:
    """A contiguous CUDA bf16 (B, groups * C) matrix of vectors that the split and merge kernels take."""
    C = mod.shape[1] // groups
    return mod.is_cuda and mod.dtype == torch.bfloat16 and mod.is_contiguous() and groups <= 128 and C % 8 == 0 and 8 <= C <= 4096


class _StackedModulation(torch.autograd.Function):
    """The adaptive-LayerNorm modulations of all layers from the one conditioning vector they share: one GEMM forward, three
    products backward, instead of those per layer.  ``params``: the layers' weights, then their biases."""

    @staticmethod
    def forward(ctx, x, weights, biases, layers, *params):
        with torch.autocast("cuda", enabled=False):
            mod = F.linear(x, weights, biases)
        B, C = x.shape[0], mod.shape[1] // (6 * layers)
        out = torch.empty((6 * layers, B, C), device=x.device, dtype=torch.float32)
        if _modulation_kernels_apply(mod, 6 * layers):
            _lib.launch(_lib.lib().mf_split_modulation, x.device, mod.data_ptr(), B, 6 * layers, C, out.data_ptr())
        else:
            out.copy_(mod.view(B, 6 * layers, C).transpose(0, 1))
        ctx.save_for_backward(x, weights)
        ctx.layers = layers
        return tuple(out.unbind(0))

    @staticmethod
    def backward(ctx, *grads):
        x, weights = ctx.saved_tensors
        like = next(g for g in grads if g is not None)
        B, C = like.shape
        g = torch.empty((B, len(grads) * C), device=x.device, dtype=torch.bfloat16)
        if _modulation_kernels_apply(g, len(grads)) and all(t is None or (t.dtype == torch.float32 and t.data_ptr() % 16 == 0) for t in grads):
            parts = [t.contiguous() if t is not None else None for t in grads]
            _lib.launch(_lib.lib().mf_merge_modulation, x.device, _ptr_array(parts), B, len(parts), C, g.data_ptr())
        else:
            g.copy_(torch.stack([t if t is not None else torch.zeros_like(like) for t in grads], dim=1).reshape(B, -1))  # (B, 6 L, C)
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


def _mm_f32(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    """a @ b for bf16 operands with the fp32 accumulator written out unrounded."""
    return torch.mm(a, b, out_dtype=torch.float32)


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
    where :func:`linear_bf16_applies` says no.  Casts the parameters unless the enclosing :func:`bf16_copies` or an
    earlier :func:`refresh_bf16_copies` has done so."""
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


class _PairLinear(torch.autograd.Function):
    """The two d-wide column blocks of a pair MLP's first Linear, applied once per atom."""

    @staticmethod
    def forward(ctx, x, weight, bias):
        d = x.shape[-1]
        w16, b16 = bf16_copy(weight), bf16_copy(bias)
        x = x.to(torch.bfloat16)
        ctx.save_for_backward(x, w16)
        ctx.columns = weight.shape[1]
        with torch.autocast("cuda", enabled=False):
            return F.linear(x, w16[:, :d]), F.linear(x, w16[:, d : 2 * d], b16)

    @staticmethod
    def backward(ctx, da, db):
        x, w16 = ctx.saved_tensors
        d = x.shape[-1]
        x2 = x.reshape(-1, d)
        da, db = (g.reshape(-1, g.shape[-1]).to(torch.bfloat16).contiguous() for g in (da, db))
        dx = dw = sums = None
        with torch.autocast("cuda", enabled=False):
            if ctx.needs_input_grad[0]:  # in fp32, as the sum of the two products' fp32 results
                dx = _mm_f32(da, w16[:, :d]).add_(_mm_f32(db, w16[:, d : 2 * d])).view(x.shape)
            if ctx.needs_input_grad[1]:
                dw = torch.zeros((da.shape[1], ctx.columns), device=x.device, dtype=torch.float32)
                dw[:, :d] = _mm_f32(da.t(), x2)
                dw[:, d : 2 * d] = _mm_f32(db.t(), x2)
            if ctx.needs_input_grad[2]:
                sums = column_sums(db) if column_sums_applies(db) else db.sum(0, dtype=torch.float32)
        return dx, dw, sums


def pair_linear_bf16(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor):
    """``F.linear(x, weight[:, :d])`` and ``F.linear(x, weight[:, d:2d], bias)`` in bf16 on fp32 parameters, x (B, N, d) fp32 or bf16."""
    return _PairLinear.apply(x, weight, bias)
