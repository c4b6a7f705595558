"""Fused element-wise passes of the trunk's adaptive-LayerNorm block on the C-ABI kernels.

``ln_modulate(x, shift, scale)`` = ``LayerNorm(x) * (1 + scale[:, None]) + shift[:, None]`` and
``gated_residual(x, gate, a)`` = ``x + gate[:, None] * a`` (AdaLNBlock.forward of the reference,
src/matterformer/models/transformer.py:242-253, 308-316), each one pass over the (B, N, C) tensor forward
and one backward instead of a chain of element-wise kernels.  ``x`` is the residual stream, fp32 or bf16
(bf16 is what autocast leaves it in); ``shift``, ``scale`` and ``gate`` are used in fp32 and their gradients
come back in their own dtype.
"""
from __future__ import annotations

import ctypes
from typing import Optional

import torch
from torch.autograd import forward_ad

from . import _lib

_CODE = {torch.float32: _lib.MF_DTYPE_F32, torch.bfloat16: _lib.MF_DTYPE_BF16}
MAX_CHANNELS = 1024


def _stream(device):
    return ctypes.c_void_p(torch.cuda.current_stream(device).cuda_stream)


def _bytes(mask: torch.Tensor) -> torch.Tensor:
    """A mask as the bytes the kernels read: a bool tensor's own, without a copy."""
    mask = mask.contiguous()
    return mask.view(torch.uint8) if mask.dtype == torch.bool else mask.to(torch.uint8)


def fused_applies(x: torch.Tensor) -> bool:
    """The kernels take a CUDA fp32 / bf16 (B, N, C) residual stream; C a multiple of 8, at most ``MAX_CHANNELS``."""
    return x.is_cuda and x.dtype in _CODE and x.ndim == 3 and x.shape[-1] <= MAX_CHANNELS and x.shape[-1] % 8 == 0


def _check_shapes(x: torch.Tensor, rows=(), vectors=(), pad: Optional[torch.Tensor] = None) -> None:
    """The kernels read ``rows`` as (B, N, C) like ``x``, ``vectors`` as (B, C) and ``pad`` as (B, N): nothing is broadcast."""
    B, N, C = x.shape
    fits = all(t.shape == x.shape and t.device == x.device for t in rows) and all(t.shape == (B, C) and t.device == x.device for t in vectors)
    if not fits or (pad is not None and (pad.shape != (B, N) or pad.device != x.device)):
        raise ValueError(f"expected operands of shapes {(B, N, C)}, {(B, C)} and {(B, N)} on {x.device}")


class _LnModulate(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, shift, scale, eps, out_dtype):
        ctx.param_dtypes = (shift.dtype, scale.dtype)
        x, shift, scale = x.contiguous(), shift.float().contiguous(), scale.float().contiguous()
        B, N, C = x.shape
        h = torch.empty((B, N, C), device=x.device, dtype=out_dtype)
        mean = torch.empty((B, N), device=x.device, dtype=torch.float32)
        rstd = torch.empty_like(mean)
        with torch.cuda.device(x.device):
            _lib.check(_lib.lib().mf_ln_modulate_fwd(x.data_ptr(), _CODE[x.dtype], shift.data_ptr(), scale.data_ptr(),
                                                     B, N, C, float(eps), _CODE[out_dtype], h.data_ptr(),
                                                     mean.data_ptr(), rstd.data_ptr(), _stream(x.device)))  # fmt: skip
        ctx.save_for_backward(x, scale, mean, rstd)
        return h

    @staticmethod
    def backward(ctx, dh):
        x, scale, mean, rstd = ctx.saved_tensors
        B, N, C = x.shape
        if dh.dtype not in _CODE:
            dh = dh.float()
        dh = dh.contiguous()
        dx = torch.empty_like(x)
        dshift = torch.empty((B, C), device=x.device, dtype=torch.float32)
        dscale = torch.empty_like(dshift)
        with torch.cuda.device(x.device):
            _lib.check(_lib.lib().mf_ln_modulate_bwd(dh.data_ptr(), _CODE[dh.dtype], x.data_ptr(), _CODE[x.dtype],
                                                     scale.data_ptr(), mean.data_ptr(), rstd.data_ptr(), B, N, C,
                                                     dx.data_ptr(), dshift.data_ptr(), dscale.data_ptr(),
                                                     _stream(x.device)))  # fmt: skip
        return dx, dshift.to(ctx.param_dtypes[0]), dscale.to(ctx.param_dtypes[1]), None, None


class _GatedResidual(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, gate, a, pad):
        ctx.gate_dtype = gate.dtype
        x, gate = x.contiguous(), gate.float().contiguous()
        if a.dtype not in _CODE:
            a = a.float()
        a = a.contiguous()
        pad = _bytes(pad) if pad is not None else None
        B, N, C = x.shape
        y = torch.empty_like(x)
        with torch.cuda.device(x.device):
            _lib.check(_lib.lib().mf_gated_residual_fwd(x.data_ptr(), _CODE[x.dtype], gate.data_ptr(), a.data_ptr(),
                                                        _CODE[a.dtype], pad.data_ptr() if pad is not None else None,
                                                        B, N, C, y.data_ptr(), _stream(x.device)))  # fmt: skip
        ctx.save_for_backward(gate, a, pad)
        return y

    @staticmethod
    def backward(ctx, dy):
        gate, a, pad = ctx.saved_tensors
        B, N, C = a.shape
        if dy.dtype not in _CODE:
            dy = dy.float()
        dy = dy.contiguous()
        da = torch.empty_like(a)
        dx = torch.empty_like(dy) if pad is not None else None
        dgate = torch.empty((B, C), device=a.device, dtype=torch.float32)
        with torch.cuda.device(a.device):
            _lib.check(_lib.lib().mf_gated_residual_bwd(dy.data_ptr(), _CODE[dy.dtype], gate.data_ptr(), a.data_ptr(),
                                                        _CODE[a.dtype], pad.data_ptr() if pad is not None else None,
                                                        B, N, C, da.data_ptr(), dx.data_ptr() if dx is not None else None,
                                                        dgate.data_ptr(), _stream(a.device)))  # fmt: skip
        return (dy if dx is None else dx), dgate.to(ctx.gate_dtype), da, None


def ln_modulate(x: torch.Tensor, shift: torch.Tensor, scale: torch.Tensor, *, eps: float,
                out_dtype: torch.dtype = torch.float32) -> torch.Tensor:  # fmt: skip
    """``LayerNorm(x) * (1 + scale[:, None, :]) + shift[:, None, :]`` in ``out_dtype`` (fp32 or bf16)."""
    _check_shapes(x, vectors=(shift, scale))
    return _LnModulate.apply(x, shift, scale, eps, out_dtype)


def gated_residual(x: torch.Tensor, gate: torch.Tensor, a: torch.Tensor,
                   pad_mask: Optional[torch.Tensor] = None) -> torch.Tensor:  # fmt: skip
    """``x + gate[:, None, :] * a`` in ``x``'s dtype; with ``pad_mask`` (B, N) bool, followed by
    ``.masked_fill(pad_mask[..., None], 0)`` in the same pass (forward and backward)."""
    _check_shapes(x, (a,), (gate,), pad_mask)
    return _GatedResidual.apply(x, gate, a, pad_mask)


class _GatedLnModulate(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, gate, a, pad, shift, scale, eps):
        x, a = x.contiguous(), a.contiguous()
        gate, shift, scale = gate.contiguous(), shift.contiguous(), scale.contiguous()
        pad = _bytes(pad) if pad is not None else None
        B, N, C = x.shape
        y, h = torch.empty_like(x), torch.empty_like(a)
        mean = torch.empty((B, N), device=x.device, dtype=torch.float32)
        rstd = torch.empty_like(mean)
        _lib.launch(_lib.lib().mf_gated_ln_modulate_fwd, x.device, x.data_ptr(), _CODE[x.dtype], gate.data_ptr(), a.data_ptr(),
                    pad.data_ptr() if pad is not None else None, shift.data_ptr(), scale.data_ptr(), B, N, C, float(eps),
                    _CODE[a.dtype], y.data_ptr(), h.data_ptr(), mean.data_ptr(), rstd.data_ptr())  # fmt: skip
        ctx.save_for_backward(gate, a, pad, scale, y, mean, rstd)
        return y, h

    @staticmethod
    def backward(ctx, dy, dh):
        gate, a, pad, scale, y, mean, rstd = ctx.saved_tensors
        B, N, C = y.shape
        dy, dh = dy.to(y.dtype).contiguous(), dh.to(a.dtype).contiguous()
        total, da = torch.empty_like(y), torch.empty_like(a)
        dx = torch.empty_like(y) if pad is not None else None
        dgate, dshift, dscale = torch.empty((3, B, C), device=y.device, dtype=torch.float32).unbind(0)
        _lib.launch(_lib.lib().mf_ln_modulate_add_bwd, y.device, dh.data_ptr(), _CODE[dh.dtype], y.data_ptr(), _CODE[y.dtype],
                    scale.data_ptr(), mean.data_ptr(), rstd.data_ptr(), dy.data_ptr(), B, N, C, total.data_ptr(),
                    dshift.data_ptr(), dscale.data_ptr())  # fmt: skip
        _lib.launch(_lib.lib().mf_gated_residual_bwd, y.device, total.data_ptr(), _CODE[total.dtype], gate.data_ptr(), a.data_ptr(),
                    _CODE[a.dtype], pad.data_ptr() if pad is not None else None, B, N, C, da.data_ptr(),
                    dx.data_ptr() if dx is not None else None, dgate.data_ptr())  # fmt: skip
        return total if dx is None else dx, dgate, da, None, dshift, dscale, None


def gated_ln_modulate(x: torch.Tensor, gate: torch.Tensor, a: torch.Tensor, pad_mask: Optional[torch.Tensor], shift: torch.Tensor,
                      scale: torch.Tensor, *, eps: float, out_dtype: torch.dtype) -> tuple:  # fmt: skip
    """``y = gated_residual(x, gate, a, pad_mask)`` and ``ln_modulate(y, shift, scale)``; one pass where ``a`` already has
    ``out_dtype`` and the modulation is fp32, the two operators otherwise."""
    if a.dtype == out_dtype and a.dtype in _CODE and all(t.dtype == torch.float32 for t in (gate, shift, scale)):
        _check_shapes(x, (a,), (gate, shift, scale), pad_mask)
        return _GatedLnModulate.apply(x, gate, a, pad_mask, shift, scale, eps)
    y = gated_residual(x, gate, a, pad_mask)
    return y, ln_modulate(y, shift, scale, eps=eps, out_dtype=out_dtype)


class _SplitModulation(torch.autograd.Function):
    """(B, 6 C) -> six contiguous fp32 (B, C) tensors in one copy; the backward pass gathers the six gradients in one
    concatenation and one cast."""

    @staticmethod
    def forward(ctx, mod):
        B, W = mod.shape
        ctx.in_dtype = mod.dtype
        out = torch.empty((6, B, W // 6), device=mod.device, dtype=torch.float32)
        out.copy_(mod.view(B, 6, W // 6).transpose(0, 1))
        return tuple(out.unbind(0))

    @staticmethod
    def backward(ctx, *grads):
        g = torch.stack([t if t is not None else torch.zeros_like(grads[0]) for t in grads], dim=1)  # (B, 6, C) fp32
        return g.reshape(g.shape[0], -1).to(ctx.in_dtype)


def split_modulation(mod: torch.Tensor):
    """The six AdaLN modulation vectors ``shift_a, scale_a, gate_a, shift_m, scale_m, gate_m`` of
    ``self.ada_ln(cond).chunk(6, dim=-1)`` (transformer.py:242-244) as contiguous fp32 tensors, which is what the fused
    LayerNorm-modulate and gated-residual kernels read."""
    if mod.ndim != 2 or mod.shape[1] % 6 != 0 or not mod.is_cuda:
        return mod.chunk(6, dim=-1)
    return _SplitModulation.apply(mod)


def column_sums_applies(x: torch.Tensor) -> bool:
    return (x.is_cuda and x.ndim == 2 and x.dtype in _CODE and x.is_contiguous() and x.shape[1] % 8 == 0
            and x.shape[1] >= 8 and x.data_ptr() % 16 == 0)  # fmt: skip


def column_sums(x: torch.Tensor) -> torch.Tensor:
    """``x.sum(0)`` of a (rows, cols) fp32 / bf16 matrix in fp32, in a fixed order of additions: the bias gradient of a
    Linear layer from its output gradient.  No autograd (it is used inside backward passes)."""
    if not column_sums_applies(x):
        raise ValueError("column_sums needs a contiguous CUDA fp32 / bf16 matrix with a multiple of 8 columns")
    L = _lib.lib()
    rows, cols = x.shape
    out = torch.empty(cols, device=x.device, dtype=torch.float32)
    need = L.mf_column_sums_workspace_bytes(rows, cols)
    ws = torch.empty(max(need, 16), device=x.device, dtype=torch.uint8)
    with torch.cuda.device(x.device):
        _lib.check(L.mf_column_sums(x.data_ptr(), _CODE[x.dtype], rows, cols, out.data_ptr(), ws.data_ptr(), need,
                                    _stream(x.device)))  # fmt: skip
    return out


def gelu_tanh_applies(x: torch.Tensor) -> bool:
    return (x.is_cuda and x.dtype in _CODE and x.is_contiguous() and x.ndim >= 1 and x.shape[-1] % 8 == 0
            and x.data_ptr() % 16 == 0)  # fmt: skip


def gelu_tanh_forward(x: torch.Tensor) -> torch.Tensor:
    """``F.gelu(x, approximate="tanh")`` (no autograd; see :func:`matterformer_b200.linear.linear_gelu_bf16`)."""
    if not gelu_tanh_applies(x):
        raise ValueError("gelu_tanh_forward needs a contiguous CUDA fp32 / bf16 tensor with a multiple of 8 columns")
    y = torch.empty_like(x)
    with torch.cuda.device(x.device):
        _lib.check(_lib.lib().mf_gelu_tanh_fwd(x.data_ptr(), _CODE[x.dtype], x.numel(), y.data_ptr(), _stream(x.device)))
    return y


def gelu_tanh_backward(pre: torch.Tensor, dy: torch.Tensor):
    """``(dy * gelu'(pre), column sums of that product in fp32)`` for (rows, cols) matrices: the gradient of the
    pre-activation and, in the same sweep, the bias gradient of the Linear layer that produced it."""
    if not (gelu_tanh_applies(pre) and gelu_tanh_applies(dy) and pre.ndim == 2 and pre.shape == dy.shape and pre.dtype == dy.dtype):
        raise ValueError("gelu_tanh_backward needs two contiguous CUDA matrices of one shape and type")
    L = _lib.lib()
    rows, cols = pre.shape
    dx = torch.empty_like(pre)
    sums = torch.empty(cols, device=pre.device, dtype=torch.float32)
    need = L.mf_column_sums_workspace_bytes(rows, cols)
    ws = torch.empty(max(need, 16), device=pre.device, dtype=torch.uint8)
    with torch.cuda.device(pre.device):
        _lib.check(L.mf_gelu_tanh_bwd(pre.data_ptr(), dy.data_ptr(), _CODE[pre.dtype], rows, cols, dx.data_ptr(),
                                      sums.data_ptr(), ws.data_ptr(), need, _stream(pre.device)))  # fmt: skip
    return dx, sums


def _ptr_array(tensors):
    arr = (ctypes.c_void_p * len(tensors))()
    for i, t in enumerate(tensors):
        arr[i] = t.data_ptr() if t is not None else None
    return arr


def _scale_array(scales, groups):
    if scales is None:
        return None
    arr = (ctypes.c_float * groups)()
    for i in range(groups):
        arr[i] = float(scales[i])
    return arr


def heads_layout_applies(packed: torch.Tensor, heads: int, groups: int) -> bool:
    """CUDA fp32 / bf16 (B, N, groups*heads*D) with head rows of a multiple of 16 bytes."""
    if not (packed.is_cuda and packed.dtype in _CODE and packed.ndim == 3 and 1 <= groups <= 8):
        return False
    width = packed.shape[-1]
    if width % (groups * heads):
        return False
    return ((width // (groups * heads)) * packed.element_size()) % 16 == 0


class _SplitHeads(torch.autograd.Function):
    @staticmethod
    def forward(ctx, packed, groups, heads, scales):
        packed = packed.contiguous()
        B, N, W = packed.shape
        D = W // (groups * heads)
        outs = torch.empty((groups, B, heads, N, D), device=packed.device, dtype=packed.dtype)
        views = list(outs.unbind(0))
        with torch.cuda.device(packed.device):
            _lib.check(_lib.lib().mf_split_heads(packed.data_ptr(), _ptr_array(views), _scale_array(scales, groups),
                                                 groups, B, N, heads, D, _CODE[packed.dtype],
                                                 _stream(packed.device)))  # fmt: skip
        ctx.meta = (groups, heads, scales, B, N, D, packed.dtype)
        return tuple(views)

    @staticmethod
    def backward(ctx, *grads):
        groups, heads, scales, B, N, D, dtype = ctx.meta
        gs = [g.to(dtype).contiguous() if g is not None else None for g in grads]
        dev = next(g.device for g in gs if g is not None)
        packed = torch.empty((B, N, groups * heads * D), device=dev, dtype=dtype)
        with torch.cuda.device(dev):
            _lib.check(_lib.lib().mf_merge_heads(_ptr_array(gs), _scale_array(scales, groups), packed.data_ptr(),
                                                 groups, B, N, heads, D, _CODE[dtype], _stream(dev)))  # fmt: skip
        return packed, None, None, None


class _MergeHeads(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        x = x.contiguous()
        B, H, N, D = x.shape
        packed = torch.empty((B, N, H * D), device=x.device, dtype=x.dtype)
        with torch.cuda.device(x.device):
            _lib.check(_lib.lib().mf_merge_heads(_ptr_array([x]), None, packed.data_ptr(), 1, B, N, H, D,
                                                 _CODE[x.dtype], _stream(x.device)))  # fmt: skip
        ctx.meta = (B, H, N, D)
        return packed

    @staticmethod
    def backward(ctx, g):
        B, H, N, D = ctx.meta
        g = g.contiguous()
        out = torch.empty((B, H, N, D), device=g.device, dtype=g.dtype)
        with torch.cuda.device(g.device):
            _lib.check(_lib.lib().mf_split_heads(g.data_ptr(), _ptr_array([out]), None, 1, B, N, H, D, _CODE[g.dtype],
                                                 _stream(g.device)))  # fmt: skip
        return out


def split_heads(packed: torch.Tensor, groups: int, heads: int, scales=None):
    """(B, N, groups*heads*D) -> ``groups`` contiguous tensors (B, heads, N, D); group g multiplied by ``scales[g]``."""
    return _SplitHeads.apply(packed, groups, heads, tuple(scales) if scales is not None else None)


def merge_heads(x: torch.Tensor) -> torch.Tensor:
    """(B, H, N, D) -> (B, N, H*D)."""
    return _MergeHeads.apply(x)


PAIR_HIDDEN, PAIR_RBF = 128, 16


def pair_head_applies(a: torch.Tensor, w_rbf: torch.Tensor) -> bool:
    """The coordinate-head kernel is built for a 128-wide pair MLP with 16 radial basis functions on CUDA fp32 / bf16."""
    return (a.is_cuda and a.dtype in _CODE and a.ndim == 3 and a.shape[-1] == PAIR_HIDDEN
            and tuple(w_rbf.shape) == (PAIR_HIDDEN, PAIR_RBF))  # fmt: skip


class _PairHead(torch.autograd.Function):
    @staticmethod
    def forward(ctx, a, b, coords, valid, w_rbf, w_out, b_out, centers, gamma):
        ctx.param_dtypes = (w_rbf.dtype, w_out.dtype, b_out.dtype)
        ctx.w_out_shape, ctx.b_out_shape = tuple(w_out.shape), tuple(b_out.shape)
        a = a.contiguous()
        b = b.to(a.dtype).contiguous()
        coords = coords.detach().float().contiguous()
        valid = _bytes(valid)
        w_rbf, w_out = w_rbf.detach().float().contiguous(), w_out.detach().float().reshape(-1).contiguous()
        b_out, centers = b_out.detach().float().reshape(-1).contiguous(), centers.detach().float().contiguous()
        B, N, _ = a.shape
        out = torch.empty((B, N, 3), device=a.device, dtype=torch.float32)
        args = _lib.MfPairHeadArgs(batch=B, tokens=N, hidden=PAIR_HIDDEN, n_rbf=PAIR_RBF, dtype=_CODE[a.dtype],
                                   gamma=float(gamma), a=a.data_ptr(), b=b.data_ptr(), coords=coords.data_ptr(),
                                   valid=valid.data_ptr(), w_rbf=w_rbf.data_ptr(), w_out=w_out.data_ptr(),
                                   b_out=b_out.data_ptr(), centers=centers.data_ptr(), out=out.data_ptr())  # fmt: skip
        with torch.cuda.device(a.device):
            _lib.check(_lib.lib().mf_pair_head_fwd(ctypes.byref(args), _stream(a.device)))
        ctx.save_for_backward(a, b, coords, valid, w_rbf, w_out, b_out, centers)
        ctx.gamma = float(gamma)
        return out

    @staticmethod
    def backward(ctx, grad_out):
        a, b, coords, valid, w_rbf, w_out, b_out, centers = ctx.saved_tensors
        B, N, _ = a.shape
        grad_out = grad_out.float().contiguous()
        da, db = torch.empty_like(a), torch.empty_like(b)
        dparams = torch.empty(PAIR_HIDDEN * PAIR_RBF + PAIR_HIDDEN + 4, device=a.device, dtype=torch.float32)
        d_w_rbf = dparams[: PAIR_HIDDEN * PAIR_RBF].view(PAIR_HIDDEN, PAIR_RBF)
        d_w_out = dparams[PAIR_HIDDEN * PAIR_RBF : PAIR_HIDDEN * PAIR_RBF + PAIR_HIDDEN]
        d_b_out = dparams[PAIR_HIDDEN * PAIR_RBF + PAIR_HIDDEN : PAIR_HIDDEN * PAIR_RBF + PAIR_HIDDEN + 1]
        args = _lib.MfPairHeadArgs(batch=B, tokens=N, hidden=PAIR_HIDDEN, n_rbf=PAIR_RBF, dtype=_CODE[a.dtype],
                                   gamma=ctx.gamma, a=a.data_ptr(), b=b.data_ptr(), coords=coords.data_ptr(),
                                   valid=valid.data_ptr(), w_rbf=w_rbf.data_ptr(), w_out=w_out.data_ptr(),
                                   b_out=b_out.data_ptr(), centers=centers.data_ptr(), grad_out=grad_out.data_ptr(),
                                   grad_a=da.data_ptr(), grad_b=db.data_ptr(), grad_w_rbf=d_w_rbf.data_ptr(),
                                   grad_w_out=d_w_out.data_ptr(), grad_b_out=d_b_out.data_ptr())  # fmt: skip
        with torch.cuda.device(a.device):
            need = int(_lib.lib().mf_pair_head_bwd_workspace_bytes(ctypes.byref(args)))
            ws = torch.empty(max(need, 16), device=a.device, dtype=torch.uint8)
            args.workspace, args.workspace_bytes = ws.data_ptr(), need
            _lib.check(_lib.lib().mf_pair_head_bwd(ctypes.byref(args), _stream(a.device)))
        dt = ctx.param_dtypes
        return (da, db, None, None, d_w_rbf.to(dt[0]), d_w_out.reshape(ctx.w_out_shape).to(dt[1]),
                d_b_out.reshape(ctx.b_out_shape).to(dt[2]), None, None)  # fmt: skip


def equivariant_pair_head(a: torch.Tensor, b: torch.Tensor, coords: torch.Tensor, valid: torch.Tensor,
                          w_rbf: torch.Tensor, w_out: torch.Tensor, b_out: torch.Tensor, centers: torch.Tensor,
                          gamma: float) -> torch.Tensor:  # fmt: skip
    """Coordinate update of ``QM9EDMModel._equivariant_coord_delta`` (src/matterformer/models/qm9.py:478-501).

    ``a`` / ``b`` (B, N, 128): the pair MLP's first Linear applied to the trunk output, split into its ``h_i`` and
    ``h_j`` column blocks (the bias goes with ``b``); ``w_rbf`` (128, 16) its radial-basis columns; ``w_out`` / ``b_out``
    the second Linear; ``coords`` (B, N, 3), ``valid`` (B, N) bool.  Returns (B, N, 3) fp32: per atom the weighted sum
    of displacements to the molecule's other real atoms, divided by their number, minus its mean over the molecule.
    Gradients flow to ``a``, ``b``, ``w_rbf``, ``w_out`` and ``b_out``; the coordinates are treated as data.
    """
    return _PairHead.apply(a, b, coords, valid, w_rbf, w_out, b_out, centers, gamma)


def masked_sum_applies(x: torch.Tensor, pad_mask: torch.Tensor, *others) -> bool:
    """CUDA fp32 (B, N, C) tensors of one shape and a (B, N) bool mask."""
    return (x.is_cuda and x.ndim == 3 and pad_mask.is_cuda and pad_mask.dtype == torch.bool and tuple(pad_mask.shape) == tuple(x.shape[:2])
            and all(t.dtype == torch.float32 and t.shape == x.shape and t.device == x.device for t in (x, *others)))  # fmt: skip


def masked_update(pad_mask, x, a=1.0, y=None, z=None, c=1.0, p=None, q=None, k=0.0, center=False) -> torch.Tensor:
    """``a x + c (y - z) + k (p - q)``, masked and centred as :func:`masked_sum` says; no autograd."""
    if not masked_sum_applies(x, pad_mask, *(t for t in (y, z, p, q) if t is not None)) or pad_mask.device != x.device:
        raise ValueError("masked sums take CUDA fp32 (B, N, C) tensors of one shape and a (B, N) bool mask, on one device")
    B, N, C = x.shape
    for t in (a, c):
        if isinstance(t, torch.Tensor) and not (t.shape == (B,) and t.dtype == torch.float32 and t.device == x.device and t.is_contiguous()):
            raise ValueError("masked sums take numbers or contiguous fp32 (B,) tensors as factors")
    pad_mask = pad_mask.contiguous()
    x, y, z, p, q = (t.contiguous() if t is not None else None for t in (x, y, z, p, q))
    out = torch.empty_like(x)
    at = lambda t: t.data_ptr() if isinstance(t, torch.Tensor) else None  # noqa: E731
    value = lambda t: 0.0 if isinstance(t, torch.Tensor) else float(t)  # noqa: E731
    args = _lib.MfMaskedSumArgs(B, N, C, int(center), at(x), at(y), at(z), at(p), at(q), at(a), at(c), at(pad_mask), at(out),
                                value(a), value(c), float(k))  # fmt: skip
    _lib.launch(_lib.lib().mf_masked_sum, x.device, ctypes.byref(args))
    return out


class _MaskedSum(torch.autograd.Function):
    """Mask and centring are one symmetric projection, which the gradient passes through as well."""

    @staticmethod
    def forward(ctx, pad_mask, x, a, y, z, c, center):
        ctx.save_for_backward(pad_mask, *(t for t in (a, c) if isinstance(t, torch.Tensor)))
        ctx.scales = tuple(None if isinstance(t, torch.Tensor) else t for t in (a, c))
        ctx.center = center
        return masked_update(pad_mask, x, a, y, z, c, center=center)

    @staticmethod
    def backward(ctx, grad):
        pad_mask, *arrays = ctx.saved_tensors
        a, c = (arrays.pop(0) if t is None else t for t in ctx.scales)
        need = ctx.needs_input_grad
        dx = masked_update(pad_mask, grad, a, center=ctx.center) if need[1] else None
        dy = masked_update(pad_mask, grad, c, center=ctx.center) if need[3] or need[4] else None
        return None, dx, None, dy if need[3] else None, -dy if need[4] else None, None, None


def masked_sum(pad_mask: torch.Tensor, x: torch.Tensor, *, a=1.0, y: Optional[torch.Tensor] = None, z: Optional[torch.Tensor] = None,
               c=1.0, center: bool = False) -> torch.Tensor:  # fmt: skip
    """``a x + c (y - z)`` in one pass, zeros on padded rows, with ``center`` minus its mean over the molecule's real rows (see
    :func:`masked_sum_applies`).  ``a``, ``c``: numbers or contiguous fp32 (B,) tensors without gradient; differentiable in
    ``x``, ``y`` and ``z``."""
    if torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in (x, y, z)):
        return _MaskedSum.apply(pad_mask, x, a, y, z, c, center)
    return masked_update(pad_mask, x, a, y, z, c, center=center)


def edm_scalings(sigma: torch.Tensor, sigma_data: float):
    """``c_skip, c_out, c_in`` of the EDM preconditioner (tasks/edm.py:34-81) for CUDA fp32 noise levels (B,); no autograd."""
    out = torch.empty((3, sigma.shape[0]), device=sigma.device, dtype=torch.float32)
    _lib.launch(_lib.lib().mf_edm_scalings, sigma.device, sigma.data_ptr(), sigma.shape[0], float(sigma_data), out.data_ptr(), None)
    return out.unbind(0)


def noise_channel(sigma: torch.Tensor) -> torch.Tensor:
    """``log(max(sigma, 1e-8)) / 4`` for CUDA fp32 noise levels (B,); no autograd."""
    out = torch.empty_like(sigma)
    _lib.launch(_lib.lib().mf_edm_scalings, sigma.device, sigma.data_ptr(), sigma.shape[0], 1.0, None, out.data_ptr())
    return out


def watched(*tensors: torch.Tensor) -> bool:
    """Something follows the torch operations on these tensors (a transform of ``torch.func``, forward-mode differentiation, tracing,
    compilation) and would not see a kernel launched past it: plain operations have to do."""
    if (torch.jit.is_tracing() or torch.compiler.is_compiling() or torch._C._len_torch_dispatch_stack() > 0
            or torch._C._functorch.peek_interpreter_stack() is not None):  # fmt: skip
        return True
    return forward_ad._current_level >= 0 and any(forward_ad.unpack_dual(t).tangent is not None for t in tensors)


def per_molecule_applies(t: torch.Tensor) -> bool:
    """What the one-launch forms of the conditioning take: a contiguous CUDA fp32 vector without gradient that nothing watches."""
    return t.is_cuda and t.ndim == 1 and t.dtype == torch.float32 and t.is_contiguous() and not t.requires_grad and not watched(t)


def time_embedding(t: torch.Tensor, half: int, dtype: torch.dtype) -> torch.Tensor:
    """``[cos, sin, cos, sin](2 pi t f)``: what ``TimeEmbedder`` feeds its MLP when both its levels are ``t`` (B,); no autograd."""
    out = torch.empty((t.shape[0], 4 * half), device=t.device, dtype=dtype)
    _lib.launch(_lib.lib().mf_time_embedding, t.device, t.data_ptr(), t.shape[0], half, _CODE[dtype], out.data_ptr())
    return out


def valid_and_counts(pad_mask: torch.Tensor):
    """``~pad_mask`` and its row sums in int32, for a CUDA bool (B, N) mask."""
    pad = pad_mask.contiguous()
    B, N = pad.shape
    valid, counts = torch.empty_like(pad), torch.empty(B, device=pad.device, dtype=torch.int32)
    _lib.launch(_lib.lib().mf_pad_counts, pad.device, pad.data_ptr(), B, N, valid.data_ptr(), counts.data_ptr())
    return valid, counts


def token_projection_applies(x: torch.Tensor, noise: torch.Tensor, pad_mask: torch.Tensor, weight: torch.Tensor,
                             bias: Optional[torch.Tensor]) -> bool:  # fmt: skip
    return (x.is_cuda and x.ndim == 3 and x.dtype == torch.float32 and not x.requires_grad and x.shape[2] < 8 and not watched(x)
            and per_molecule_applies(noise)
            and noise.shape[0] == x.shape[0] and pad_mask.dtype == torch.bool and pad_mask.shape == x.shape[:2] and bias is not None
            and weight.dtype == bias.dtype == torch.float32 and weight.shape[1] == x.shape[2] + 1 and weight.shape[0] % 64 == 0
            and 64 <= weight.shape[0] <= 1024 and all(t.device == x.device for t in (noise, pad_mask, weight, bias)))  # fmt: skip


class _TokenProjection(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, noise, pad_mask, weight, bias):
        x, pad = x.contiguous(), _bytes(pad_mask)
        w, b = weight.detach().contiguous(), bias.detach().contiguous()
        B, N, C = *x.shape[:2], w.shape[0]
        out = torch.empty((B, N, C), device=x.device, dtype=torch.bfloat16)
        _lib.launch(_lib.lib().mf_token_projection_fwd, x.device, x.data_ptr(), noise.data_ptr(), pad.data_ptr(), w.data_ptr(), b.data_ptr(),
                    B, N, w.shape[1], C, out.data_ptr())  # fmt: skip
        ctx.save_for_backward(x, noise, pad)
        return out

    @staticmethod
    def backward(ctx, dy):
        x, noise, pad = ctx.saved_tensors
        dy = dy.to(torch.bfloat16).contiguous()
        (B, N, C), K = dy.shape, x.shape[2] + 1
        L = _lib.lib()
        need = L.mf_token_projection_bwd_workspace_bytes(B, N, K, C)
        ws = torch.empty(max(need, 16), device=dy.device, dtype=torch.uint8)
        grads = torch.empty(C * (K + 1), device=dy.device, dtype=torch.float32)
        _lib.launch(L.mf_token_projection_bwd, dy.device, dy.data_ptr(), x.data_ptr(), noise.data_ptr(), pad.data_ptr(), B, N, K, C,
                    grads.data_ptr(), ws.data_ptr(), need)  # fmt: skip
        return None, None, None, grads[: C * K].view(C, K), grads[C * K :]


def token_projection(x: torch.Tensor, noise: torch.Tensor, pad_mask: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor) -> torch.Tensor:
    """The model's first Linear in bf16 on ``cat[x, noise]`` per token, padded rows cleared, without the concatenation; see
    :func:`token_projection_applies`.  Gradients flow to ``weight`` and ``bias``."""
    return _TokenProjection.apply(x, noise, pad_mask, weight, bias)


class _GatedLayerNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, gate, a, pad, eps):
        x, a, gate = x.contiguous(), a.contiguous(), gate.contiguous()
        pad = _bytes(pad) if pad is not None else None
        B, N, C = x.shape
        y, h = torch.empty_like(x), torch.empty((B, N, C), device=x.device, dtype=torch.float32)
        mean = torch.empty((B, N), device=x.device, dtype=torch.float32)
        rstd = torch.empty_like(mean)
        _lib.launch(_lib.lib().mf_gated_layer_norm_fwd, x.device, x.data_ptr(), _CODE[x.dtype], gate.data_ptr(), a.data_ptr(), _CODE[a.dtype],
                    pad.data_ptr() if pad is not None else None, B, N, C, float(eps), y.data_ptr(), h.data_ptr(), mean.data_ptr(),
                    rstd.data_ptr())  # fmt: skip
        ctx.save_for_backward(gate, a, pad, y, mean, rstd)
        return h

    @staticmethod
    def backward(ctx, dh):
        gate, a, pad, y, mean, rstd = ctx.saved_tensors
        B, N, C = y.shape
        dh = dh.float().contiguous()
        total, da = torch.empty_like(y), torch.empty_like(a)
        dx = torch.empty_like(y) if pad is not None else None
        sums = torch.empty((3, B, C), device=y.device, dtype=torch.float32)
        zeros = torch.zeros((B, C), device=y.device, dtype=torch.float32)
        _lib.launch(_lib.lib().mf_ln_modulate_bwd, y.device, dh.data_ptr(), _CODE[dh.dtype], y.data_ptr(), _CODE[y.dtype], zeros.data_ptr(),
                    mean.data_ptr(), rstd.data_ptr(), B, N, C, total.data_ptr(), sums[1].data_ptr(), sums[2].data_ptr())  # fmt: skip
        _lib.launch(_lib.lib().mf_gated_residual_bwd, y.device, total.data_ptr(), _CODE[total.dtype], gate.data_ptr(), a.data_ptr(),
                    _CODE[a.dtype], pad.data_ptr() if pad is not None else None, B, N, C, da.data_ptr(),
                    dx.data_ptr() if dx is not None else None, sums.data_ptr())  # fmt: skip
        return total if dx is None else dx, sums[0], da, None, None


def gated_layer_norm(x: torch.Tensor, gate: torch.Tensor, a: torch.Tensor, pad_mask: Optional[torch.Tensor], eps: float) -> torch.Tensor:
    """``LayerNorm(gated_residual(x, gate, a, pad_mask))`` without affine parameters, in fp32; ``gate`` is fp32.  Padded rows come out as
    zeros."""
    if gate.dtype != torch.float32 or a.dtype not in _CODE:
        gate, a = gate.float(), a if a.dtype in _CODE else a.float()
    _check_shapes(x, (a,), (gate,), pad_mask)
    return _GatedLayerNorm.apply(x, gate, a, pad_mask, eps)


class _LayerNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias, eps, out_dtype):
        x, w, b = x.contiguous(), weight.detach().float().contiguous(), bias.detach().float().contiguous()
        B, N, C = x.shape
        h = torch.empty((B, N, C), device=x.device, dtype=out_dtype)
        mean = torch.empty((B, N), device=x.device, dtype=torch.float32)
        rstd = torch.empty_like(mean)
        _lib.launch(_lib.lib().mf_layer_norm_fwd, x.device, x.data_ptr(), _CODE[x.dtype], w.data_ptr(), b.data_ptr(), B * N, C, float(eps),
                    _CODE[out_dtype], h.data_ptr(), mean.data_ptr(), rstd.data_ptr())  # fmt: skip
        ctx.dtypes = (weight.dtype, bias.dtype)
        # (values of its own: the weight may change before the backward pass)
        ctx.save_for_backward(x, w - 1.0 if any(ctx.needs_input_grad) else None, mean, rstd)
        return h

    @staticmethod
    def backward(ctx, dh):
        x, w1, mean, rstd = ctx.saved_tensors
        B, N, C = x.shape
        dh = (dh if dh.dtype in _CODE else dh.float()).contiguous()
        dx = torch.empty_like(x)
        sums = torch.empty((2, B, C), device=x.device, dtype=torch.float32)
        scale = w1.expand(B, C).contiguous()
        _lib.launch(_lib.lib().mf_ln_modulate_bwd, x.device, dh.data_ptr(), _CODE[dh.dtype], x.data_ptr(), _CODE[x.dtype], scale.data_ptr(),
                    mean.data_ptr(), rstd.data_ptr(), B, N, C, dx.data_ptr(), sums[0].data_ptr(), sums[1].data_ptr())  # fmt: skip
        db, dw = sums.sum(1)
        return dx, dw.to(ctx.dtypes[0]), db.to(ctx.dtypes[1]), None, None


def affine_layer_norm(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor, eps: float, out_dtype: torch.dtype) -> torch.Tensor:
    """``F.layer_norm`` over the channels of a (B, N, C) residual stream (see :func:`fused_applies`) in ``out_dtype``."""
    return _LayerNorm.apply(x, weight, bias, eps, out_dtype)
