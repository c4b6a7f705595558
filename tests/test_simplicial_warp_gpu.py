"""Warp-level simplicial kernels of 33 to 192 tokens, the fp32 kernels and the low-rank residuals at the edges of their ranges."""
import pytest
import torch

import matterformer_b200 as mfb
from conftest import bf16_allowance
from oracle.simplicial_ref import SimplicialInputs, simplicial_forward_backward
from test_simplicial_gpu import BIAS_NAMES, NAMES, RES_NAMES, assert_rel, run_cuda, run_cuda_bias
from test_simplicial_small_gpu import _case

pytestmark = pytest.mark.gpu


def _with_bias(inp, seed):
    g = torch.Generator().manual_seed(seed)
    B, H, N, _ = inp.q.shape
    for n in ("u", "v_bias", "w"):
        setattr(inp, n, (torch.randn(B, H, N, N, generator=g) * 0.5).bfloat16().float())
    inp.gate = torch.randn(B, H, N, generator=g).bfloat16().float()


def _with_holes(inp, seed):
    g = torch.Generator().manual_seed(seed)
    B, _, N, _ = inp.q.shape
    inp.pair_key_valid = inp.query_valid & (torch.rand(B, N, generator=g) < 0.8)
    inp.pair_key_valid[:, 0] = True
    inp.pair_valid = torch.rand(B, N, N, generator=g) < 0.7
    inp.pair_valid[:, 0, 0] = True


@pytest.mark.parametrize("B,H,N,holes,shift", [(2, 2, 33, False, 0), (2, 1, 48, False, 0), (3, 2, 49, True, 0), (2, 2, 64, False, 0),
                                               (1, 3, 65, True, 0), (1, 2, 96, False, 0), (1, 1, 191, True, 0), (1, 1, 192, False, 0),
                                               (2, 2, 50, False, 1.5), (2, 2, 50, False, -1.5)])  # fmt: skip
def test_against_oracle(B, H, N, holes, shift):
    """Around the 16- and 32-row blocks, with masks inside them, and logits that need the exact maximum (near +-216)."""
    inp, go = _case(B, H, N, seed=N, scale=0.2 if shift else 0.5, lo=N // 2, shift=shift)
    if holes:
        _with_holes(inp, N)
    out_ref, g_ref = simplicial_forward_backward(inp, go)
    tol = bf16_allowance(inp, go, out_ref, g_ref)
    out, _, grads, _ = run_cuda(inp, go, dtype=torch.bfloat16, precision="bf16_tc")
    assert_rel(out, out_ref, tol["out"], "out")
    for n in NAMES:
        assert_rel(grads[n], g_ref[n], tol[n], f"d{n}")


@pytest.mark.parametrize("B,H,N,holes", [(2, 2, 33, False), (40, 8, 48, False), (2, 3, 49, True), (1, 2, 65, False), (1, 1, 128, True),
                                         (2, 1, 131, False), (1, 1, 177, False), (1, 1, 192, True)])  # fmt: skip
def test_with_bias_against_oracle(B, H, N, holes):
    """One to four splits of the second keys, rounds that leave warps without a block, query blocks that span rounds."""
    inp, go = _case(B, H, N, seed=N, scale=0.5, lo=N // 2)
    _with_bias(inp, N)
    if holes:
        _with_holes(inp, N)
    out_ref, g_ref = simplicial_forward_backward(inp, go)
    y, grads = run_cuda_bias(inp, go, dtype=torch.bfloat16, precision="bf16_tc")
    assert_rel(y, out_ref, 2e-2, "out")
    for n in NAMES + BIAS_NAMES:
        assert_rel(grads[n], g_ref[n], 2.5e-2, f"d{n}")
    _, again = run_cuda_bias(inp, go, dtype=torch.bfloat16, precision="bf16_tc")
    assert all(torch.equal(grads[n], again[n]) for n in NAMES + BIAS_NAMES)


@pytest.mark.parametrize("N,D,holes", [(1, 64, False), (31, 32, True), (32, 64, False), (33, 64, True), (64, 32, False), (64, 64, True), (65, 64, False)])
def test_fp32_against_oracle(N, D, holes):
    inp, go = _case(2, 2, N, seed=N + D, scale=0.7, lo=max(1, N - 3))
    for n in NAMES:
        setattr(inp, n, getattr(inp, n)[..., :D].contiguous())
    go = go[..., :D].contiguous()
    if holes:
        _with_holes(inp, N)
    out_ref, g_ref = simplicial_forward_backward(inp, go)
    out, _, grads, _ = run_cuda(inp, go)
    assert_rel(out, out_ref, 1e-5, "out")
    for n in NAMES:
        assert_rel(grads[n], g_ref[n], 1e-5, f"d{n}")


@pytest.mark.parametrize("N,ra,rm,factorized", [(1, 1, 1, True), (16, 16, 17, True), (17, 3, 5, False), (29, 32, 8, True), (32, 31, 32, False)])
def test_bf16_residuals_against_oracle(N, ra, rm, factorized):
    B, H = 2, 3
    inp, go = _case(B, H, N, seed=N + ra, scale=0.5, lo=max(1, N - 5))
    g = torch.Generator().manual_seed(N)
    if factorized:
        _with_bias(inp, N)
    for n, r in (("angle_left", ra), ("angle_right", ra), ("message_left", rm), ("message_right", rm)):
        setattr(inp, n, torch.randn(B, H, N, N, r, generator=g) * r**-0.25)
    inp.angle_gate = torch.randn(B, H, N, generator=g) * 0.5
    inp.message_basis = torch.randn(H, rm, 64, generator=g) / 8
    out_ref, g_ref = simplicial_forward_backward(inp, go)
    names = NAMES + RES_NAMES + (BIAS_NAMES if factorized else ())
    t = {n: getattr(inp, n).to("cuda:0", torch.bfloat16 if n in NAMES else torch.float32).requires_grad_(True) for n in names}
    y = mfb.simplicial_attention_cuda(
        *[t[n] for n in NAMES], query_valid=inp.query_valid.cuda(), pair_key_valid=inp.pair_key_valid.cuda(), precision="bf16_tc",
        factorized_bias=tuple(t[n] for n in BIAS_NAMES) if factorized else None, angle_residual=tuple(t[n] for n in RES_NAMES[:3]),
        message_residual=tuple(t[n] for n in RES_NAMES[3:]))  # fmt: skip
    grads = dict(zip(names, torch.autograd.grad(y, [t[n] for n in names], go.to("cuda:0", torch.bfloat16))))
    assert_rel(y.detach().float().cpu(), out_ref, 2.5e-2, "out")
    largest = max(float(g_ref[n].abs().max()) for n in NAMES)
    for n in names:  # (a lone token has exact zeros: judge them on the scale of the others)
        err = float((grads[n].float().cpu() - g_ref[n]).abs().max())
        assert err <= max(3e-2 * float(g_ref[n].abs().max()), 1e-2 * largest), f"d{n}: {err}"


@pytest.mark.parametrize("B,N,R,D,dtype", [(1, 1, 1, 64, torch.float32), (7, 9, 16, 64, torch.bfloat16), (41, 25, 17, 64, torch.float16),
                                           (3, 171, 32, 128, torch.bfloat16), (10, 103, 8, 32, torch.float32)])  # fmt: skip
def test_basis_gradient_sums(B, N, R, D, dtype):
    """Rows around a round of the cluster (1024, and 512 for wide heads), ranks and channels that do not fill their lanes.  Each sum has
    B N products of fp32 factors: the largest error is B N 2^-24 of the sum of absolute values."""
    from matterformer_b200 import _lib
    H = 3
    g = torch.Generator("cuda").manual_seed(B)
    c = torch.randn(B, H, N, R, generator=g, device="cuda")
    go = torch.randn(B, H, N, D, generator=g, device="cuda").to(dtype)
    out = torch.empty(H, R, D, device="cuda")
    code = {torch.float32: _lib.MF_DTYPE_F32, torch.bfloat16: _lib.MF_DTYPE_BF16, torch.float16: _lib.MF_DTYPE_F16}[dtype]
    _lib.launch(_lib.lib().mf_simplicial_basis_grad, out.device, c.data_ptr(), go.data_ptr(), code, B, H, N, R, D, out.data_ptr())
    want = torch.einsum("bhir,bhid->hrd", c.double(), go.double())
    bound = B * N * 2.0**-24 * torch.einsum("bhir,bhid->hrd", c.double().abs(), go.double().abs())
    assert ((out.double() - want).abs() <= bound + 1e-30).all()
