"""What an expired device-side wait leaves behind: the status, zeros, and a device that goes on."""
import ctypes

import pytest
import torch

from matterformer_b200 import _lib

pytestmark = pytest.mark.gpu
B, H, N = 2, 2, 64  # 32 and 14 steps a tile: more than the stages of the bias operands


def _call(cls, backend="tcgen05_tiles", **outputs):
    g = torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    t = {n: rnd(B, H, N, 64).bfloat16() for n in ("q", "k1", "v1", "k2", "v2")}
    if backend == "tcgen05_tiles":  # the trilinear kernels
        t.update(u=rnd(B, H, N, N), v_bias=rnd(B, H, N, N), w=rnd(B, H, N, N), gate=rnd(B, H, N))
    valid = (torch.arange(N, device="cuda")[None] < torch.tensor([[N], [40]], device="cuda")).view(torch.uint8)
    t.update(query_valid=valid, pair_key_valid=valid, **outputs)
    a = cls(batch=B, heads=H, tokens=N, head_dim=64, dtype=_lib.MF_DTYPE_BF16, backend=_lib.MF_BACKEND[backend])
    for name, x in t.items():
        setattr(a, name, x.data_ptr())
    size = "mf_simplicial_fwd_workspace_bytes" if cls is _lib.MfSimplicialFwdArgs else "mf_simplicial_bwd_workspace_bytes"
    ws = torch.empty(getattr(_lib.lib(), size)(ctypes.byref(a)), dtype=torch.uint8, device="cuda")
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    return a, t, ws


@pytest.mark.parametrize("kernel,withheld", [*(("forward", i) for i in range(8)), *(("backward", i) for i in range(8)),
                                             *(("row-packed forward", i) for i in range(6))])  # fmt: skip
def test_a_hand_off_that_never_completes(kernel, withheld):
    backward = kernel == "backward"
    nan = lambda *s, dtype=torch.float32: torch.full(s, float("nan"), dtype=dtype, device="cuda")  # noqa: E731
    bf = dict(dtype=torch.bfloat16)
    if backward:
        outputs = {n: nan(B, H, N, 64, **bf) for n in ("dq", "dk1", "dv1", "dk2", "dv2")}
        outputs.update(du=nan(B, H, N, N), dv_bias=nan(B, H, N, N), dw=nan(B, H, N, N), dgate=nan(B, H, N))
        saved = dict(grad_out=torch.ones(B, H, N, 64, device="cuda", **bf), out=torch.zeros(B, H, N, 64, device="cuda"),
                     lse=torch.zeros(B, H, N, device="cuda"))  # fmt: skip
        a, keep, ws = _call(_lib.MfSimplicialBwdArgs, **outputs, **saved)
    else:
        outputs = dict(out=nan(B, H, N, 64), out_cast=nan(B, H, N, 64, **bf), lse=nan(B, H, N))
        a, keep, ws = _call(_lib.MfSimplicialFwdArgs, "tcgen05" if kernel == "row-packed forward" else "tcgen05_tiles", **outputs)
    ref, stream = ctypes.byref(a), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.lib().mf_selftest_simplicial_give_up(None if backward else ref, ref if backward else None, withheld, 20_000, stream))
    assert ws[:4].view(torch.int32).item() == _lib.MF_ERR_DEVICE_TIMEOUT
    for name, t in outputs.items():
        assert torch.equal(t, torch.zeros_like(t)), name
    # the same call with nothing withheld, on the same buffers
    _lib.check(getattr(_lib.lib(), "mf_simplicial_bwd" if backward else "mf_simplicial_fwd")(ref, stream))
    assert ws[:4].view(torch.int32).item() == _lib.MF_OK
    assert all(torch.isfinite(outputs[n]).all() for n in (("dq", "dk1", "dv1", "dk2", "dv2") if backward else outputs))
    del keep


@pytest.mark.parametrize("window", [32, 64, 128])
@pytest.mark.parametrize("backward", [False, True])
def test_band_tiles_that_never_arrive(window, backward):
    B, H, N = 16, 4, 200
    bf = dict(dtype=torch.bfloat16, device="cuda")
    rows = {n: torch.ones(B, H, N, 64, **bf) for n in ("q", "k", "v", "grad_out")}
    nan = {n: torch.full((B, H, N, 64), float("nan"), **bf) for n in (("dq", "dk", "dv") if backward else ("out",))}
    if backward:
        rows["out"] = torch.ones(B, H, N, 64, **bf)
    lse = torch.full((B, H, N), 0.0 if backward else float("nan"), device="cuda")
    n = torch.full((B,), N, dtype=torch.int32, device="cuda")
    n[1], n[2] = 0, 100
    ws = torch.empty(1 << 20, dtype=torch.uint8, device="cuda")
    a = _lib.MfSparseAttnArgs(batch=B, heads=H, tokens=N, head_dim=64, dtype=_lib.MF_DTYPE_BF16, window=window, scale=0.125)
    for name, x in {**rows, **nan, "lse": lse, "num_atoms": n, "workspace": ws}.items():
        setattr(a, name, x.data_ptr())
    a.workspace_bytes = ws.numel()
    ref, stream, status = ctypes.byref(a), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.c_int32(0)
    _lib.check(_lib.lib().mf_selftest_band_give_up(ref, int(backward), 20_000, ctypes.byref(status), stream))
    assert status.value == _lib.MF_ERR_DEVICE_TIMEOUT
    for name, t in (*nan.items(), *(() if backward else (("lse", lse),))):
        assert torch.equal(t, torch.zeros_like(t)), name
    # the same call with tiles that arrive, on the same buffers
    _lib.check(getattr(_lib.lib(), "mf_local_attn_bwd" if backward else "mf_local_attn_fwd")(ref, stream))
    _lib.check(_lib.lib().mf_sparse_attn_status(ctypes.byref(status), stream))
    assert status.value == _lib.MF_OK
    assert all(torch.isfinite(t).all() for t in nan.values())
    assert backward or (nan["out"][0].float() - 1).abs().max() < 2**-7  # a mean of ones with weights rounded to bf16
