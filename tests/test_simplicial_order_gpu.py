"""Heavy-first order of the kernels of at most 32 tokens: the results are those of the order given, bit for bit."""
import ctypes

import pytest
import torch

from matterformer_b200 import _lib
from matterformer_b200.simplicial import cuda_simplicial_attention_backward, cuda_simplicial_attention_forward, simplicial_attention_cuda, simplicial_attention_packed

pytestmark = pytest.mark.gpu


def _without(monkeypatch):
    for name in ("fwd", "bwd"):
        monkeypatch.setattr(_lib.lib(), f"mf_simplicial_{name}_workspace_bytes", lambda ref: 0)
        monkeypatch.setattr(_lib.lib(), f"mf_simplicial_packed_{name}_workspace_bytes", lambda ref: 0)


@pytest.mark.parametrize("B,H,N,rank", [(1025, 4, 7, 0), (600, 8, 32, 0), (129, 4, 20, 8)])
def test_same_bits_in_either_order(monkeypatch, B, H, N, rank):
    """Empty molecules, ties, batches beyond the order kernel's block; with the factorized bias and the residuals."""
    g = torch.Generator(device="cuda").manual_seed(N)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    heads = [randn(B, H, N, 64).bfloat16() for _ in range(5)]
    go = randn(B, H, N, 64).bfloat16()
    n = torch.randint(0, N + 1, (B,), generator=g, device="cuda")
    valid = torch.arange(N, device="cuda")[None] < n[:, None]
    kw = dict(query_valid=valid, pair_key_valid=valid, pair_valid=None, u=randn(B, H, N, N), v_bias=randn(B, H, N, N), w=randn(B, H, N, N),
              gate=randn(B, H, N))  # fmt: skip
    if rank:
        kw.update(angle_left=randn(B, H, N, N, rank), angle_right=randn(B, H, N, N, rank), angle_gate=randn(B, H, N))

    def run():
        out, lse, out32 = cuda_simplicial_attention_forward(*heads, **kw)
        grads = cuda_simplicial_attention_backward(go, *heads, out32, lse, **kw, need_du=True, need_dv_bias=True, need_dw=True, need_dgate=True)
        return [out, lse, *(t for t in grads if t is not None)]

    a = _lib.MfSimplicialBwdArgs(batch=B, heads=H, tokens=N, head_dim=64, dtype=1, angle_left=go.data_ptr() if rank else None)
    args = {f: go.data_ptr() for f in ("q", "k1", "v1", "k2", "v2", "grad_out", "out", "dq", "dk1", "dv1", "dk2", "dv2")}
    for f, v in args.items():
        setattr(a, f, v)
    assert _lib.lib().mf_simplicial_bwd_workspace_bytes(ctypes.byref(a)) > 0  # the order is used
    ordered = run()
    _without(monkeypatch)
    assert all(torch.equal(x, y) for x, y in zip(ordered, run()))


def test_packed_projection_in_either_order(monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(5)
    proj = torch.randn(600, 23, 5 * 8 * 64, generator=g, device="cuda").bfloat16().requires_grad_(True)
    valid = torch.arange(23, device="cuda")[None] < torch.randint(1, 24, (600,), generator=g, device="cuda")[:, None]

    def run():
        out = simplicial_attention_packed(proj, heads=8, query_valid=valid, pair_key_valid=valid)
        return [out, *torch.autograd.grad(out, [proj], torch.ones_like(out))]

    ordered = run()
    _without(monkeypatch)
    assert all(torch.equal(x, y) for x, y in zip(ordered, run()))


@pytest.mark.parametrize("B,H,N", [(1024, 2, 33), (40, 8, 64), (9, 8, 131), (8, 8, 192)])
def test_forward_above_32_tokens_in_either_order(monkeypatch, B, H, N):
    g = torch.Generator(device="cuda").manual_seed(N)
    heads = [torch.randn(B, H, N, 64, generator=g, device="cuda").bfloat16() for _ in range(5)]
    valid = torch.arange(N, device="cuda")[None] < torch.randint(0, N + 1, (B,), generator=g, device="cuda")[:, None]
    kw = dict(query_valid=valid, pair_key_valid=valid, pair_valid=None)
    a = _lib.MfSimplicialFwdArgs(batch=B, heads=H, tokens=N, head_dim=64, dtype=1)
    for f in ("q", "k1", "v1", "k2", "v2", "out"):
        setattr(a, f, heads[0].data_ptr())
    assert _lib.lib().mf_simplicial_fwd_workspace_bytes(ctypes.byref(a)) > 0  # the order is used
    ordered = cuda_simplicial_attention_forward(*heads, **kw)
    _without(monkeypatch)
    assert all(torch.equal(x, y) for x, y in zip(ordered, cuda_simplicial_attention_forward(*heads, **kw)))


@pytest.mark.parametrize("N,batch", [(29, 300), (64, 64)])
def test_a_caller_may_leave_the_list_out(N, batch):
    """Through the operators on heads and on the packed projection: no launch of a list, the same bits."""
    g = torch.Generator(device="cuda").manual_seed(2)
    heads = [torch.randn(batch, 8, N, 64, generator=g, device="cuda").bfloat16().requires_grad_(True) for _ in range(5)]
    valid = torch.arange(N, device="cuda")[None] < torch.randint(1, N + 1, (batch,), generator=g, device="cuda")[:, None]
    proj = torch.randn(batch, N, 5 * 8 * 64, generator=g, device="cuda").bfloat16().requires_grad_(True)
    kw = dict(query_valid=valid, pair_key_valid=valid)

    def run(heavy_first):
        out = simplicial_attention_cuda(*heads, **kw, heavy_first=heavy_first)
        results = [out, *torch.autograd.grad(out, heads, torch.ones_like(out))]
        if N <= 32:
            out = simplicial_attention_packed(proj, heads=8, **kw, heavy_first=heavy_first)
            results += [out, *torch.autograd.grad(out, [proj], torch.ones_like(out))]
        out, lse, out32 = cuda_simplicial_attention_forward(*heads, **kw, pair_valid=None, heavy_first=heavy_first)
        grads = cuda_simplicial_attention_backward(out, *heads, out32, lse, **kw, pair_valid=None, heavy_first=heavy_first)
        return [*results, out, lse, *grads[:5]]

    def lists(heavy_first):
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            results = run(heavy_first)
            torch.cuda.synchronize()
        return sum(e.count for e in prof.key_averages() if "_order_kernel" in e.key and "simplicial" in e.key), results

    run(True)
    made, ordered = lists(True)
    none, given = lists(False)
    assert made > 0 and none == 0
    assert all(torch.equal(a, b) for a, b in zip(ordered, given))
