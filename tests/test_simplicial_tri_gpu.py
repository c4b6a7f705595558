"""Trilinear tcgen05 kernels (factorized bias, 33 to 192 tokens): unequal extents, empty molecules, exact maxima, no workspace."""
from dataclasses import replace

import pytest
import torch

from conftest import bf16_allowance
from matterformer_b200 import _lib
from matterformer_b200.simplicial import cuda_simplicial_attention_backward, cuda_simplicial_attention_forward, set_backend
from oracle.simplicial_ref import simplicial_forward_backward
from test_simplicial_gpu import BIAS_NAMES, NAMES, assert_rel, run_cuda_bias
from test_simplicial_small_gpu import _case
from test_simplicial_warp_gpu import _with_bias

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def trilinear_forward():
    """The default backend keeps forward calls as short as these on the warp-level kernel."""
    before = set_backend("tcgen05_tiles")
    yield
    set_backend(before)


def _check(inp, go):
    out_ref, g_ref = simplicial_forward_backward(inp, go)
    y, grads = run_cuda_bias(inp, go, dtype=torch.bfloat16, precision="bf16_tc")
    assert_rel(y, out_ref, 2e-2, "out")  # operands, probabilities and their gradients rounded to 8 bits
    for n in NAMES + BIAS_NAMES:
        assert_rel(grads[n], g_ref[n], 2.5e-2, f"d{n}")


@pytest.mark.parametrize("N,queries,keys", [(40, 3, 40), (64, 64, 5), (97, 17, 97), (129, 129, 16), (192, 1, 130), (192, 192, 3), (190, 33, 161)])
def test_unequal_extents(N, queries, keys):
    """One to eight y per step, one to three chunks of columns (each of 16 to 64), rows of a tile that carry no pair."""
    inp, go = _case(2, 2, N, seed=N + queries, scale=0.5, lo=N)
    _with_bias(inp, N)
    at = torch.arange(N)[None, :]
    inp.query_valid = (at < queries).repeat(2, 1)
    inp.pair_key_valid = (at < keys).repeat(2, 1)
    inp.query_valid[1, 0] = queries > 1  # a hole in front
    inp.pair_key_valid[1, keys // 2] = keys == 1
    _check(inp, go)


def test_empty_molecules():
    inp, go = _case(4, 2, 50, seed=1, scale=0.5, lo=30)
    _with_bias(inp, 1)
    inp.query_valid[1] = False
    inp.pair_key_valid[2] = False
    _check(inp, go)


@pytest.mark.parametrize("shift", [1.5, -1.5])
def test_exact_maxima(shift):
    """Logits near +-216 leave the range of a softmax with shift 0: the tile is done again with its maxima."""
    inp, go = _case(2, 2, 70, seed=70, scale=0.2, lo=35, shift=shift)
    _with_bias(inp, 70)
    out_ref, g_ref = simplicial_forward_backward(inp, go)
    tol = bf16_allowance(inp, go, out_ref, g_ref)  # logits this large carry the rounding of their products
    y, grads = run_cuda_bias(inp, go, dtype=torch.bfloat16, precision="bf16_tc")
    assert_rel(y, out_ref, tol["out"], "out")
    for n in NAMES:
        assert_rel(grads[n], g_ref[n], tol[n], f"d{n}")


@pytest.mark.parametrize("shift", [1.5, -1.5])
def test_bias_gradients_of_sharp_logits(shift):
    """Each pass forms the logits from products of another pair of the three sets, rounded for itself: the gradients of gate and u come
    from other roundings than those of w and v.  Allowed is what the torch path in bf16, which rounds the logits too, makes of it."""
    inp, go = _case(2, 2, 70, seed=70, scale=0.2, lo=35, shift=shift)
    _with_bias(inp, 70)
    _, g_ref = simplicial_forward_backward(inp, go)
    low = replace(inp, **{n: getattr(inp, n).bfloat16() for n in NAMES})
    _, g_low = simplicial_forward_backward(low, go.bfloat16(), fp32_core=False)
    _, grads = run_cuda_bias(inp, go, dtype=torch.bfloat16, precision="bf16_tc")
    for n in BIAS_NAMES:
        allowed = (g_low[n].float() - g_ref[n]).abs().max() / g_ref[n].abs().max()
        assert_rel(grads[n], g_ref[n], max(2.5e-2, float(allowed)), f"d{n}")


def _run(t, valid, grad, need=(True,) * 4, pair_valid=None):
    """Forward and backward on device tensors {name: tensor}: every output as a list."""
    kw = dict(query_valid=valid, pair_key_valid=valid, pair_valid=pair_valid, **{n: t[n] for n in BIAS_NAMES})
    heads = [t[n] for n in NAMES]
    out, lse, out32 = cuda_simplicial_attention_forward(*heads, **kw)
    grads = cuda_simplicial_attention_backward(grad, *heads, out32, lse, **kw, **dict(zip(("need_du", "need_dv_bias", "need_dw", "need_dgate"), need)))
    return [out, lse, out32, *grads[:9]]


def _device_case(B, H, N, seed, lo):
    inp, go = _case(B, H, N, seed=seed, scale=0.4, lo=lo)
    _with_bias(inp, seed)
    t = {n: getattr(inp, n).cuda() for n in (*NAMES, *BIAS_NAMES)}
    t.update({n: t[n].bfloat16() for n in NAMES})
    return t, inp.query_valid.cuda(), go.cuda().bfloat16()


@pytest.mark.parametrize("fill", [float("nan"), float("inf")])
@pytest.mark.parametrize("N", [50, 132])
def test_padded_tokens_may_hold_anything(N, fill):
    """In the rows of the heads and of grad_out, and in every entry of the bias that a padded token has a part in."""
    t, valid, go = _device_case(3, 2, N, seed=N, lo=N // 3)
    valid[1, 2] = False  # a hole too: columns are then copied one by one
    clean = _run(t, valid, go)
    pad = ~valid[:, None, :]
    dirty = {n: x.masked_fill(pad[..., None], fill) for n, x in t.items() if x.ndim == 4 and n in NAMES}
    dirty.update({n: t[n].masked_fill(pad[..., None] | pad[..., None, :], fill) for n in ("u", "v_bias", "w")})
    dirty["gate"] = t["gate"].masked_fill(pad, fill)
    for a, b in zip(clean, _run(dirty, valid, go.masked_fill(pad[..., None], fill))):
        assert torch.equal(a, b)


@pytest.mark.parametrize("value", [torch.finfo(torch.float32).min, float("-inf")])
def test_a_bias_that_hides_pairs(value):
    """The lowest value of the type and minus infinity in w, under a positive gate, hide a pair of keys as the mask does."""
    inp, go = _case(2, 2, 90, seed=90, scale=0.4, lo=60)
    _with_bias(inp, 90)
    inp.gate = inp.gate.abs().clamp(0.05, 0.9)
    hidden = torch.rand(2, 1, 90, 90, generator=torch.Generator().manual_seed(9)) < 0.3
    hidden[:, :, 0] = False  # (every query keeps a pair)
    inp.w = inp.w.masked_fill(hidden, value)
    out_ref, g_ref = simplicial_forward_backward(inp, go)
    t = {n: getattr(inp, n).cuda() for n in (*NAMES, *BIAS_NAMES)}  # (the bias in fp32: the lowest value is infinite in bf16)
    t.update({n: t[n].bfloat16() for n in NAMES})
    _, _, y, *grads = (x.float().cpu() for x in _run(t, inp.query_valid.cuda(), go.cuda().bfloat16()))
    assert_rel(y, out_ref, 2e-2, "out")
    for n, got in zip(NAMES + BIAS_NAMES, grads):
        if n == "gate" and value == float("-inf"):  # 0 * infinity, as in the torch path
            assert got[g_ref[n].isfinite()].isfinite().all()
        else:
            assert_rel(got, g_ref[n], 2.5e-2, f"d{n}")


@pytest.mark.parametrize("B,H,N,pick", [(5, 2, 192, slice(2, 3)), (1100, 1, 36, slice(1030, 1037))])
def test_a_molecule_alone_and_in_a_batch(B, H, N, pick):
    """The same bits, also from a batch of more molecules than the schedule's block has threads."""
    t, valid, go = _device_case(B, H, N, seed=B, lo=1)
    valid[B // 2] = False
    whole = _run(t, valid, go)
    part = _run({n: x[pick].contiguous() for n, x in t.items()}, valid[pick].contiguous(), go[pick].contiguous())
    assert all(torch.isfinite(x).all() for x in whole)
    for a, b in zip(whole, part):
        assert torch.equal(a[pick], b)


def test_each_bias_gradient_alone():
    t, valid, go = _device_case(2, 2, 77, seed=3, lo=40)
    whole = _run(t, valid, go)
    for i in range(4):
        some = _run(t, valid, go, need=tuple(j == i for j in range(4)))
        for k, (a, b) in enumerate(zip(whole, some)):
            assert torch.equal(a, b) if k < 8 or k == 8 + i else b is None


def test_forward_without_workspace(monkeypatch):
    """A caller that gives no workspace gets the warp-level kernel."""
    inp, go = _case(2, 2, 77, seed=77, scale=0.5, lo=38)
    _with_bias(inp, 77)
    out_ref, _ = simplicial_forward_backward(inp, go)
    monkeypatch.setattr(_lib.lib(), "mf_simplicial_fwd_workspace_bytes", lambda ref: 0)
    out, _, _ = cuda_simplicial_attention_forward(
        *(getattr(inp, n).bfloat16().cuda() for n in NAMES), query_valid=inp.query_valid.cuda(), pair_key_valid=inp.pair_key_valid.cuda(),
        pair_valid=None, **{n: getattr(inp, n).cuda() for n in BIAS_NAMES})  # fmt: skip
    assert_rel(out.float().cpu(), out_ref, 2e-2, "out")


@pytest.mark.parametrize("B,H,N", [(1, 1, 101), (2, 9, 128), (6, 8, 140), (13, 8, 110), (28, 8, 103)])
def test_spread_tiles_against_oracle(B, H, N):
    """Six tiles, fewer and none besides the usual ones, forward on either side of its line: molecules of 1, 65, 101 and N atoms (the others
    repeat them), against the oracle."""
    inp, go = _case(4, H, N, seed=N, scale=0.5, lo=1)
    for i, n in enumerate((N, 101, 65, 1)):
        inp.query_valid[i] = inp.pair_key_valid[i] = torch.arange(N) < n
    _with_bias(inp, N)
    out_ref, g_ref = simplicial_forward_backward(inp, go)
    pick = torch.arange(B) % 4
    t = {n: getattr(inp, n)[pick].cuda() for n in (*NAMES, *BIAS_NAMES)}
    t.update({n: t[n].bfloat16() for n in NAMES})
    _, _, y, *grads = (x.float().cpu() for x in _run(t, inp.query_valid[pick].cuda(), go[pick].cuda().bfloat16()))
    keep = min(B, 4)
    assert_rel(y[:keep], out_ref[:keep], 2e-2, "out")
    for n, got in zip(NAMES + BIAS_NAMES, grads):
        assert_rel(got[:keep], g_ref[n][:keep], 2.5e-2, f"d{n}")
        if B > 4:
            assert torch.equal(got[4:8], got[: min(4, B - 4)])


@pytest.mark.parametrize("B,N", [(2, 128), (9, 128), (20, 128), (28, 128), (4, 192), (8, 192), (14, 110)])
def test_a_molecule_alone_and_in_batches_of_many_sizes(B, N):
    """The split into tiles depends on the molecule alone: the same bits from a call that leaves most of the chip idle and from one that
    fills it, for molecules of N, 101 and 65 atoms."""
    t, valid, go = _device_case(B, 8, N, seed=B + N, lo=N)
    if B > 2:
        valid[1] = torch.arange(N, device="cuda") < 101
        valid[2] = torch.arange(N, device="cuda") < 65
    whole = _run(t, valid, go)
    for i in range(min(B, 3)):
        part = _run({n: x[i : i + 1].contiguous() for n, x in t.items()}, valid[i : i + 1].contiguous(), go[i : i + 1].contiguous())
        for a, b in zip(whole, part):
            assert torch.equal(a[i : i + 1], b)
