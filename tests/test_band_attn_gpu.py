"""Band attention with the whole neighbourhood in shared memory (bf16, head_dim 64, windows 32 / 64 / 128)."""
import pytest
import torch

import matterformer_b200 as mfb
from matterformer_b200.sparse import local_window_attention_packed
from oracle import sparse_ref
from test_sparse_gpu import DEV, _attn_ref, _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,N,window,sharp", [(2, 2, 96, 64, 1.0), (2, 2, 129, 64, 1.0), (3, 1, 255, 32, 1.0), (1, 2, 257, 128, 1.0),
                                                (2, 2, 100, 128, 1.0), (90, 8, 130, 64, 1.0), (2, 2, 200, 64, 900.0), (3, 2, 2, 64, 1.0),
                                                (5, 3, 16, 64, 1.0), (4, 2, 17, 128, 1.0), (40, 8, 32, 64, 1.0), (3, 2, 32, 64, 900.0)])  # fmt: skip
def test_band_attention_vs_oracle(B, H, N, window, sharp):
    """Both tile heights, tile remainders, structures that end inside a tile, an empty and a one-token structure, and logits
    whose exponentials leave the range in which no maximum is needed; structures that fit one tile."""
    g = torch.Generator().manual_seed(N + window)
    q, k, v, go = (torch.randn(B, H, N, 64, generator=g).bfloat16() for _ in range(4))
    q = (q.float() * sharp / 8).bfloat16()
    n = torch.randint(1, N + 1, (B,), generator=g)
    n[0] = N
    if B > 2:
        n[1], n[2] = 0, 1
    t = [x.to(DEV).requires_grad_(True) for x in (q, k, v)]
    out = mfb.local_window_attention(*t, n.to(DEV, torch.int32), window=window)
    grads = torch.autograd.grad(out, t, go.to(DEV))
    vis = sparse_ref.band_visible(N, n, window)
    valid = (torch.arange(N)[None] < n[:, None])[:, None, :, None].float()
    ref = _attn_ref(q, k, v, go, vis, valid)
    assert not torch.isnan(out).any()
    for got, want, what in zip((out.detach(), *grads), ref, ("out", "dq", "dk", "dv")):
        _check(got, want, 2e-2, what)
    again = mfb.local_window_attention(*t, n.to(DEV, torch.int32), window=window)
    assert torch.equal(out, again)


def test_packed_projection_takes_the_same_kernels():
    B, H, N = 2, 4, 140
    g = torch.Generator().manual_seed(5)
    qkv = torch.randn(B, N, 3 * H * 64, generator=g).bfloat16().to(DEV).requires_grad_(True)
    go = torch.randn(B, N, H * 64, generator=g).bfloat16().to(DEV)
    n = torch.tensor([N, 77], device=DEV, dtype=torch.int32)
    out = local_window_attention_packed(qkv, H, n, window=64)
    (gp,) = torch.autograd.grad(out, [qkv], go)
    parts = [x.view(B, N, H, 64).transpose(1, 2).contiguous() for x in qkv.detach().chunk(3, dim=-1)]
    parts = [x.requires_grad_(True) for x in parts]
    y = mfb.local_window_attention(*parts, n, window=64)
    grads = torch.autograd.grad(y, parts, go.view(B, N, H, 64).transpose(1, 2).contiguous())
    assert torch.equal(out.view(B, N, H, 64).transpose(1, 2), y)
    assert torch.equal(gp, torch.cat([x.transpose(1, 2).reshape(B, N, -1) for x in grads], dim=-1))


@pytest.mark.parametrize("B,H,N,window", [(37, 4, 128, 128), (25, 6, 127, 128), (13, 8, 191, 128), (13, 8, 192, 128), (16, 8, 65, 64),
                                          (16, 8, 130, 64), (127, 1, 97, 32)])  # fmt: skip
def test_both_sides_of_the_selection_rules(B, H, N, window):
    """One wave of tiles and one tile more under a window of 128 below 192 tokens (band or walk), and both tile heights around
    128 wide tiles: every choice is the same operator."""
    test_band_attention_vs_oracle(B, H, N, window, 1.0)


def _kernels(call):
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    return [e.name for e in prof.events() if "band_" in e.name]


@pytest.mark.parametrize("N,window", [(140, 32), (257, 32), (140, 64), (257, 64), (200, 128), (257, 128)])
def test_wide_tiles(N, window):
    """At 128 wide tiles and more, rows at the strides of a packed projection: the bits of head-major operands, and of the 64-row tiles that
    serve the same structures two at a time.  Structures that end at, one short of and inside a tile and inside a halo; an empty one."""
    B, H = 16, 8
    g = torch.Generator().manual_seed(N + window)
    qkv = torch.randn(B, N, 3 * H * 64, generator=g).bfloat16().to(DEV).requires_grad_(True)
    go = torch.randn(B, N, H * 64, generator=g).bfloat16().to(DEV)
    n = torch.tensor([N, 128, 127, 129, 0, 1, 77, 128 - window // 2, 128 + window // 2, 139, N - 1, N, 64, 63, 2, 96], device=DEV, dtype=torch.int32)
    parts = [x.view(B, N, H, 64).transpose(1, 2).contiguous().requires_grad_(True) for x in qkv.detach().chunk(3, dim=-1)]
    heads_go = go.view(B, N, H, 64).transpose(1, 2).contiguous()
    got = {}

    def call():
        got["out"] = local_window_attention_packed(qkv, H, n, window=window)
        (got["grad"],) = torch.autograd.grad(got["out"], [qkv], go)
        got["y"] = mfb.local_window_attention(*parts, n, window=window)
        got["grads"] = torch.autograd.grad(got["y"], parts, heads_go)

    names = _kernels(call)
    for kernel in ("band_fwd_kernel", "band_bwd_kernel"):
        assert sum(f"{kernel}<{window}, 128>" in x for x in names) == 2, names
    assert torch.equal(got["out"].view(B, N, H, 64).transpose(1, 2), got["y"])
    assert torch.equal(got["grad"], torch.cat([x.transpose(1, 2).reshape(B, N, -1) for x in got["grads"]], dim=-1))
    for at in range(0, B, 2):
        some = [x[at : at + 2].detach().contiguous().requires_grad_(True) for x in parts]
        y = mfb.local_window_attention(*some, n[at : at + 2].contiguous(), window=window)
        assert torch.equal(y, got["y"][at : at + 2])
        for a, b in zip(torch.autograd.grad(y, some, heads_go[at : at + 2].contiguous()), got["grads"]):
            assert torch.equal(a, b[at : at + 2])


@pytest.mark.parametrize("fill", [float("nan"), float("inf")])
@pytest.mark.parametrize("window", [32, 64, 128])
def test_wide_tiles_ignore_what_padding_holds(window, fill):
    """Rows from a structure's end on, at a tile's edge, inside a tile and inside a halo, come with the tiles and are cleared."""
    B, H, N = 16, 8, 200
    g = torch.Generator().manual_seed(window)
    q, k, v, go = (torch.randn(B, H, N, 64, generator=g).bfloat16().to(DEV) for _ in range(4))
    n = torch.tensor([N, 128, 127, 129, 0, 1, 199, 128 - window // 2, 128 + window // 2, 130, 64, 100, 77, 16, 144, 143], device=DEV, dtype=torch.int32)
    pad = torch.arange(N, device=DEV)[None, :] >= n[:, None]
    results = []
    for value in (0.0, fill):
        t = [x.masked_fill(pad[:, None, :, None], value).requires_grad_(True) for x in (q, k, v)]
        out = mfb.local_window_attention(*t, n, window=window)
        results.append([out, *torch.autograd.grad(out, t, go.masked_fill(pad[:, None, :, None], value))])
    for a, b in zip(*results):
        assert torch.equal(a, b)
        assert b.masked_select(pad[:, None, :, None]).abs().max() == 0
