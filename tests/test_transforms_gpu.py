"""Noise conditioning under forward-mode differentiation, torch.func and tracing: what these see, they see on CUDA as on the CPU."""
import pytest
import torch
import torch.autograd.forward_ad as forward_ad
from torch import nn
from torch.fx.experimental.proxy_tensor import make_fx

from matterformer_b200.trunk import EDMModel, EDMPreconditioner, TimeEmbedder

pytestmark = pytest.mark.gpu


class _Scaled(nn.Module):
    """A denoiser of plain operations: what is left of the preconditioner are its own scalings."""

    def forward(self, atoms, coords, pad_mask, sigma, lattice=None):
        return atoms * sigma[:, None, None], coords * sigma[:, None, None]


class _NoiseChannel(EDMModel):
    def _forward(self, atoms, coords, pad_mask, sigma_cond):
        return sigma_cond


def _cases(device):
    """The same three functions of five noise levels on either device; atoms and coordinates in fp64, which no kernel takes."""
    g = torch.Generator().manual_seed(0)
    with torch.random.fork_rng():
        torch.manual_seed(1)
        embed, channel = (m.to(device).requires_grad_(False) for m in (TimeEmbedder(64), _NoiseChannel(d_model=64, n_heads=1, n_layers=1)))
    atoms, coords = (torch.randn(5, 4, c, generator=g, dtype=torch.float64).to(device) for c in (6, 3))
    pad = torch.zeros(5, 4, dtype=torch.bool, device=device)
    pad[1, 3] = True
    scaled = EDMPreconditioner(_Scaled())
    return {"embedding": lambda t: embed(t, t), "scalings": lambda t: torch.cat([x.flatten(1) for x in scaled(atoms, coords, pad, t)], dim=1),
            "channel": lambda t: channel(atoms, coords, pad, t)}  # fmt: skip


LEVELS = torch.tensor([0.2, 0.4, 0.7, 1.1, 1.6])
# fp32 on both sides: cos and sin of angles up to 2 pi 1.6 scaled by 2 pi in a derivative, a few units in the last place each
TOL = dict(rtol=1e-4, atol=1e-4)


def _both(name, transform):
    """The transform of the function on CUDA and on the CPU, side by side."""
    got, want = (transform(_cases(d)[name], LEVELS.to(d)) for d in ("cuda", "cpu"))
    torch.testing.assert_close(got.cpu(), want, **TOL)


NAMES = ["embedding", "scalings", "channel"]


@pytest.mark.parametrize("name", NAMES)
def test_forward_mode(name):
    def tangent(f, t):
        with forward_ad.dual_level(), torch.no_grad():
            return forward_ad.unpack_dual(f(forward_ad.make_dual(t, torch.ones_like(t)))).tangent

    _both(name, tangent)
    _both(name, lambda f, t: torch.func.jvp(f, (t,), (torch.ones_like(t),))[1].detach())
    _both(name, lambda f, t: torch.func.jacfwd(f)(t).detach())


@pytest.mark.parametrize("name", NAMES)
def test_vmap(name):
    _both(name, lambda f, t: torch.func.vmap(f)(torch.stack([t, 2 * t])).detach())


@pytest.mark.parametrize("name", NAMES)
def test_tracing(name):
    """A trace made at one set of noise levels holds at another."""
    f, t = _cases("cuda")[name], LEVELS.cuda()
    with torch.no_grad():
        torch.testing.assert_close(make_fx(f)(t)(t + 1), f(t + 1), **TOL)
        traced = torch.jit.trace(lambda x: f(x), (t,), check_trace=False)
        torch.testing.assert_close(traced(t + 1), f(t + 1), **TOL)
