"""Warp-level simplicial kernels (at most 32 tokens) at the edges of their tiles and of their softmax range."""
import pytest
import torch

from conftest import bf16_allowance
from oracle.simplicial_ref import SimplicialInputs, simplicial_forward_backward
from test_simplicial_gpu import BIAS_NAMES, NAMES, assert_rel, run_cuda, run_cuda_bias

pytestmark = pytest.mark.gpu


def _case(B, H, N, seed, scale, lo=1, shift=0.0):
    g = torch.Generator().manual_seed(seed)
    n = torch.randint(lo, N + 1, (B,), generator=g)
    n[0] = N
    valid = torch.arange(N)[None, :] < n[:, None]
    t = {name: (torch.randn(B, H, N, 64, generator=g) * scale).bfloat16().float() for name in NAMES}
    if shift:  # every logit near 64 * shift**3: far from zero, all of one sign
        for name, sign in (("q", 1.0), ("k1", 1.0), ("k2", 1.0 if shift > 0 else -1.0)):
            t[name] = (t[name] * 0.1 + sign * abs(shift)).bfloat16().float()
    go = torch.randn(B, H, N, 64, generator=g).bfloat16().float()
    return SimplicialInputs(**t, query_valid=valid, pair_key_valid=valid, pair_valid=None), go


@pytest.mark.parametrize("B,H,N,scale,shift", [(3, 3, 8, 0.5, 0), (2, 1, 9, 0.5, 0), (5, 2, 16, 0.5, 0), (2, 5, 17, 0.5, 0),
                                               (3, 2, 24, 0.5, 0), (2, 3, 25, 0.5, 0), (140, 8, 32, 0.3, 0), (4, 2, 29, 0.2, 1.5),
                                               (4, 2, 29, 0.2, -1.5), (3, 2, 1, 0.5, -1.5)])  # fmt: skip
def test_small_molecules_against_oracle(B, H, N, scale, shift):
    """Token counts around the 8 / 16-row tiles, one and several warps per molecule, and logits whose exponentials leave the
    range in which no maximum is needed (all near +-216)."""
    inp, go = _case(B, H, N, seed=7 * N + H, scale=scale, shift=shift)
    out_ref, g_ref = simplicial_forward_backward(inp, go)
    tol = bf16_allowance(inp, go, out_ref, g_ref)
    out, _, grads, y = run_cuda(inp, go, dtype=torch.bfloat16, precision="bf16_tc")
    assert_rel(out, out_ref, tol["out"], "out")
    largest = max(float(g_ref[n].abs().max()) for n in NAMES)
    for n in NAMES:  # (a lone token has dq = dk = 0 exactly: judge zeros on the scale of the others)
        err = float((grads[n] - g_ref[n]).abs().max())
        assert err <= max(tol[n] * float(g_ref[n].abs().max()), 1e-2 * largest), f"d{n}: {err}"


@pytest.mark.parametrize("B,H,N", [(3, 3, 8), (2, 2, 17), (3, 1, 25), (140, 8, 31)])
def test_small_molecules_with_bias_against_oracle(B, H, N):
    inp, go = _case(B, H, N, seed=11 * N, scale=0.5, lo=max(1, N - 6))
    g = torch.Generator().manual_seed(N)
    for n in ("u", "v_bias", "w"):
        setattr(inp, n, (torch.randn(B, H, N, N, generator=g) * 0.5).bfloat16().float())
    inp.gate = torch.randn(B, H, N, generator=g).bfloat16().float()
    out_ref, g_ref = simplicial_forward_backward(inp, go)
    y, grads = run_cuda_bias(inp, go, dtype=torch.bfloat16, precision="bf16_tc")
    assert_rel(y, out_ref, 2e-2, "out")
    for n in NAMES + BIAS_NAMES:
        assert_rel(grads[n], g_ref[n], 2.5e-2, f"d{n}")


@pytest.mark.parametrize("B,H,N,holes", [(3, 1, 9, False), (2, 6, 29, True), (5, 3, 17, False), (171, 6, 8, False)])
def test_packed_projection_serves_any_number_of_heads(B, H, N, holes):
    from matterformer_b200.simplicial import packed_projection_applies
    from test_simplicial_gpu import test_packed_projection_matches_the_head_major_call as compare

    assert packed_projection_applies(torch.empty(B, N, 5 * H * 64, device="cuda:0", dtype=torch.bfloat16), H, 64)
    compare(B, H, N, holes)
