"""The one-launch forms of what surrounds the trunk against the element-wise operations they stand for."""
import math

import pytest
import torch
import torch.nn.functional as F

from matterformer_b200 import fused
from matterformer_b200.dp import build_edm_net
from matterformer_b200.linear import _StackedModulation, pair_linear_bf16
from matterformer_b200.trunk import AdaLNBlock, TransformerTrunk, layer_norm

pytestmark = pytest.mark.gpu
EPS16 = 2.0**-7  # spacing of bf16 at 1 (seven fraction bits); a rounded value is within half of it, relatively


def _rand(g, *shape, dtype=torch.float32):
    return torch.randn(*shape, generator=g, device="cuda").to(dtype)


@pytest.mark.parametrize("B", [1, 129])
def test_noise_levels(B):
    """The same operations in the same order: the same bits, but for the embedding's cosine and sine (two units in the last place)."""
    g = torch.Generator("cuda").manual_seed(B)
    sigma = torch.exp(3 * _rand(g, B))
    sigma[0] = 0.0
    sd = 0.5
    skip, out, scale = fused.edm_scalings(sigma, sd)
    assert torch.equal(skip, sd**2 / (sigma.square() + sd**2))
    assert torch.equal(out, sigma * sd / torch.sqrt(sigma.square() + sd**2))
    assert torch.equal(scale, 1.0 / torch.sqrt(sd**2 + sigma.square()))
    noise = fused.noise_channel(sigma)
    assert torch.equal(noise, torch.log(sigma.clamp_min(1e-8)) / 4.0)
    for half in (1, 128, 130):
        freqs = torch.exp(-math.log(10_000) * torch.arange(half, dtype=torch.float32, device="cuda") / half)
        args = 2.0 * math.pi * noise[:, None] * freqs[None, :]
        want = torch.cat([torch.cos(args), torch.sin(args)] * 2, dim=-1)
        # the argument's own rounding (an ulp of the frequency where half is no power of two) moves a value by |arg| 2^-22
        assert ((fused.time_embedding(noise, half, torch.float32) - want).abs() <= 2.0**-22 * (1 + args.abs().repeat(1, 4))).all()
        assert (fused.time_embedding(noise, half, torch.bfloat16).float() - want).abs().max() <= EPS16


@pytest.mark.parametrize("B,N,C,K", [(1, 1, 64, 7), (3, 29, 512, 7), (40, 31, 192, 1), (21, 33, 1024, 8)])
def test_token_projection(B, N, C, K):
    """A row, a band's edge, one input, the widest rows.  Forward: one rounding to bf16 of a sum of K fp32 products.  Backward: sums of
    up to B N exact products in fp32."""
    g = torch.Generator("cuda").manual_seed(C + K)
    x, noise, w, b = _rand(g, B, N, K - 1), _rand(g, B), _rand(g, C, K), _rand(g, C)
    pad = torch.arange(N, device="cuda")[None] >= torch.randint(0, N + 1, (B, 1), generator=g, device="cuda")
    dy = _rand(g, B, N, C, dtype=torch.bfloat16)
    dy[pad] = float("nan")  # what lies on padded rows counts for nothing
    w.requires_grad_(True), b.requires_grad_(True)
    assert fused.token_projection_applies(x, noise, pad, w, b)
    y = fused.token_projection(x, noise, pad, w, b)
    gw, gb = torch.autograd.grad(y, (w, b), dy)
    full = torch.cat([x, noise[:, None, None].expand(B, N, 1)], dim=-1).bfloat16().double()
    want = (full @ w.bfloat16().double().t() + b.bfloat16().double()).masked_fill(pad[..., None], 0.0)
    bound = (full.abs() @ w.abs().double().t() + b.abs().double()) * 2.0**-20 + want.abs() * EPS16 / 2
    assert ((y.double() - want).abs() <= bound * 1.01).all()
    d = dy.double().masked_fill(pad[..., None], 0.0).flatten(0, 1)
    f = full.masked_fill(pad[..., None], 0.0).flatten(0, 1)
    for got, ref, size in ((gw, d.t() @ f, d.abs().t() @ f.abs()), (gb, d.sum(0), d.abs().sum(0))):
        assert got.shape == ref.shape and ((got.double() - ref).abs() <= B * N * 2.0**-24 * size + 1e-30).all()


@pytest.mark.parametrize("B,layers,C", [(1, 1, 8), (65, 2, 512), (7, 12, 264)])
def test_modulation_vectors(B, layers, C):
    """Split and merge move and round values: exact.  (The products around them are GEMMs.)"""
    g = torch.Generator("cuda").manual_seed(C)
    x = _rand(g, B, 16, dtype=torch.bfloat16)
    ws = [_rand(g, 6 * C, 16).requires_grad_(True) for _ in range(layers)]
    bs = [_rand(g, 6 * C).requires_grad_(True) for _ in range(layers)]
    w16, b16 = torch.cat([w.detach() for w in ws]).bfloat16(), torch.cat([b.detach() for b in bs]).bfloat16()
    outs = _StackedModulation.apply(x, w16, b16, layers, *ws, *bs)
    mod = F.linear(x, w16, b16).float().view(B, 6 * layers, C)
    assert all(torch.equal(o, mod[:, i]) for i, o in enumerate(outs))
    grads = [_rand(g, B, C) for _ in outs]
    used = [o for i, o in enumerate(outs) if i != 1]  # a vector that nothing uses has no gradient
    db = torch.autograd.grad(used, bs, [t for i, t in enumerate(grads) if i != 1])
    grads[1].zero_()
    want = torch.stack(grads, dim=1).bfloat16().double().sum(0).flatten()
    # fp32 sums of B values of about one
    assert (torch.cat(db).double() - want).abs().max() <= B * 2.0**-22 * 4


@pytest.mark.parametrize("B,N,C,xtype,atype", [(1, 1, 8, torch.float32, torch.float32), (3, 29, 512, torch.bfloat16, torch.bfloat16),
                                               (2, 9, 1024, torch.float32, torch.bfloat16)])  # fmt: skip
def test_norms_behind_the_trunk(B, N, C, xtype, atype):
    """Output norm with the last gated residual, affine norm, padding counts.  fp32 sums over C channels; results in bf16 are rounded once;
    the residual is stored in x's type, as the two operators store it."""
    g = torch.Generator("cuda").manual_seed(C)
    pad = torch.arange(N, device="cuda")[None] >= torch.randint(1, N + 1, (B, 1), generator=g, device="cuda")
    valid, counts = fused.valid_and_counts(pad)
    assert torch.equal(valid, ~pad) and torch.equal(counts, (~pad).sum(1).to(torch.int32))
    x, gate, a = _rand(g, B, N, C, dtype=xtype), _rand(g, B, C), _rand(g, B, N, C, dtype=atype)
    leaves = [t.requires_grad_(True) for t in (x, gate, a)]
    dh = _rand(g, B, N, C)
    for mask in (pad, None):
        h = fused.gated_layer_norm(*leaves, mask, 1e-6)
        y = fused.gated_residual(*leaves, mask)
        want = F.layer_norm(y.float(), (C,), eps=1e-6)
        if mask is not None:
            want = want.masked_fill(mask[..., None], 0.0)
            assert (h[mask] == 0).all()
        torch.testing.assert_close(h, want, rtol=1e-5, atol=1e-5)
        for got, ref in zip(torch.autograd.grad(h, leaves, dh), torch.autograd.grad(want, leaves, dh)):
            tol = 1e-4 if xtype == atype == torch.float32 else 2 * EPS16  # gradients pass through x's and a's types
            assert got.dtype == ref.dtype and (got.float() - ref.float()).abs().max() <= tol * ref.float().abs().max()
    w, b = _rand(g, C).requires_grad_(True), _rand(g, C).requires_grad_(True)
    z = _rand(g, B, N, C).requires_grad_(True)
    for dtype in (torch.float32, torch.bfloat16):
        h = fused.affine_layer_norm(z, w, b, 1e-5, dtype)
        want = F.layer_norm(z, (C,), w, b, 1e-5)
        assert h.dtype == dtype and (h.float() - want).abs().max() <= (1e-5 if dtype == torch.float32 else EPS16 / 2) * want.abs().max()
        for got, ref in zip(torch.autograd.grad(h, (z, w, b), dh.to(dtype)), torch.autograd.grad(want, (z, w, b), dh.to(dtype).float())):
            assert (got - ref).abs().max() <= 1e-4 * ref.abs().max() + 1e-5


def test_pair_linear():
    g = torch.Generator("cuda").manual_seed(1)
    d = 64
    x, w, b = (_rand(g, 2, 9, d).requires_grad_(True), _rand(g, 128, 2 * d + 16).requires_grad_(True), _rand(g, 128).requires_grad_(True))
    da, db = _rand(g, 2, 9, 128, dtype=torch.bfloat16), _rand(g, 2, 9, 128, dtype=torch.bfloat16)
    got = pair_linear_bf16(x, w, b)
    x16, w16 = x.bfloat16().double(), w.bfloat16().double()
    want = (x16 @ w16[:, :d].t(), x16 @ w16[:, d : 2 * d].t() + b.bfloat16().double())
    for y, r in zip(got, want):  # one rounding to bf16
        assert (y.double() - r).abs().max() <= EPS16 * r.abs().max()
    for y, r in zip(torch.autograd.grad(got, (x, w, b), (da, db)), torch.autograd.grad(want, (x, w, b), (da.double(), db.double()))):
        assert (y.double() - r.double()).abs().max() <= EPS16 * r.abs().max()


def test_a_norm_whose_weight_changes_before_the_backward_pass():
    """The gradient is that of the weight that the forward pass used."""
    g = torch.Generator("cuda").manual_seed(2)
    x, norm, dh = _rand(g, 3, 7, 64).requires_grad_(True), torch.nn.LayerNorm(64).cuda(), _rand(g, 3, 7, 64)
    torch.nn.init.normal_(norm.weight)
    wants = torch.autograd.grad(layer_norm(x, norm), (x, norm.weight, norm.bias), dh)
    h = layer_norm(x, norm)
    with torch.no_grad():
        norm.weight.mul_(1.5)
    for got, want in zip(torch.autograd.grad(h, (x, norm.weight, norm.bias), dh), wants):
        assert torch.equal(got, want)


def _trunk_case():
    torch.manual_seed(1)
    trunk = TransformerTrunk(64, 1, ["mha", "mha"]).cuda()
    for block in trunk.blocks:
        torch.nn.init.normal_(block.ada_ln[-1].weight, std=0.1)
        torch.nn.init.normal_(block.ada_ln[-1].bias, std=0.5)
    x, cond = torch.randn(2, 24, 64, device="cuda"), torch.randn(2, 64, device="cuda")
    return trunk, x, cond, torch.arange(24, device="cuda")[None] >= torch.tensor([[24], [10]], device="cuda")


class _Weighted(AdaLNBlock):
    def forward(self, *args, **kwargs):
        return super().forward(*args, **kwargs) * torch.linspace(0.5, 2.0, 64, device="cuda")


def test_a_last_block_of_another_class():
    """What a derived last block makes of its output comes before the output norm: as in a trunk whose norm is applied by hand."""
    trunk, x, cond, pad = _trunk_case()
    trunk.blocks[1].__class__ = _Weighted
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        got, norm = trunk(x, cond, pad_mask=pad), trunk.norm_out
        trunk.norm_out = torch.nn.Identity()
        trunk.norm_out.normalized_shape = ()
        before = trunk(x, cond, pad_mask=pad)
    want = norm(before).masked_fill(pad[..., None], 0.0)
    assert (got - want).abs().max() <= 1e-5 * want.abs().max()


def test_an_output_norm_without_eps():
    """Padded rows come out as zeros, and no NaN of theirs reaches a gradient."""
    trunk, x, cond, pad = _trunk_case()
    trunk.norm_out.eps = 0.0
    x.requires_grad_(True)
    with torch.autocast("cuda", torch.bfloat16):
        out = trunk(x, cond, pad_mask=pad)
    assert (out[pad] == 0).all() and torch.isfinite(out).all()
    grads = torch.autograd.grad(out.square().sum() + out.sum(), [x, *(b.mlp.fc1.weight for b in trunk.blocks)])
    assert all(torch.isfinite(t[~pad] if t is grads[0] else t).all() for t in grads)


def test_a_pair_head_without_a_bias():
    """A first Linear without a bias is one whose bias is zero.  The halves are rounded to bf16 once either way, their products summed in
    fp32: two spacings of bf16."""
    net = build_edm_net(seed=0).cuda()
    head = net.model.pair_head
    torch.nn.init.normal_(head[2].weight)
    torch.nn.init.zeros_(head[0].bias)
    g = torch.Generator("cuda").manual_seed(3)
    atoms, coords, pad = _rand(g, 2, 9, 6), _rand(g, 2, 9, 3), torch.zeros(2, 9, dtype=torch.bool, device="cuda")

    def call():
        with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
            return net(atoms, coords, pad, torch.ones(2, device="cuda"))

    want = call()
    head[0].bias = None
    for got, ref in zip(call(), want):
        assert (got - ref).abs().max() <= 2 * EPS16 * ref.abs().max()


def test_a_data_scale_that_is_learned():
    """A tensor in the place of the number, as a program may put one there, keeps its gradient: that of the scalings written out."""
    from matterformer_b200.trunk import EDMPreconditioner

    g = torch.Generator("cuda").manual_seed(4)
    pre = EDMPreconditioner(lambda a, c, pad, sigma, lattice=None: (a * 0.5, c * 0.5))
    atoms, coords, pad = _rand(g, 3, 4, 6).double(), _rand(g, 3, 4, 3).double(), torch.zeros(3, 4, dtype=torch.bool, device="cuda")
    sigma, scale = torch.tensor([0.5, 1.0, 2.0], device="cuda"), torch.tensor(1.5, device="cuda", requires_grad=True)
    pre.sigma_data = scale
    got = torch.autograd.grad(pre(atoms, coords, pad, sigma)[0].sum(), scale)[0]
    s = sigma.double()[:, None, None]
    d = scale.detach().double().requires_grad_(True)
    written = d**2 / (s**2 + d**2) * atoms + s * d / (s**2 + d**2) * 0.5 * atoms
    want = torch.autograd.grad(written.sum(), d)[0]
    assert abs(got.item() - want.item()) <= 1e-5 * abs(want.item())
