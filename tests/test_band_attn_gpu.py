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
