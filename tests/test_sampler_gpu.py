"""The sampler's CUDA branch (fused, rearranged updates) against its CPU branch, which the reference's golden samples pin."""
import pytest
import torch

from matterformer_b200.sampler import build_pad_mask, edm_sample

pytestmark = pytest.mark.gpu


class _Net(torch.nn.Module):
    """Only says where the run takes place and which noise levels it may use."""

    def __init__(self, device):
        super().__init__()
        self.p = torch.nn.Parameter(torch.zeros(1, device=device))


def _draws_on_the_cpu(monkeypatch):
    randn, randn_like = torch.randn, torch.randn_like
    monkeypatch.setattr(torch, "randn", lambda *size, device=None: randn(*size).to(device or "cpu"))
    monkeypatch.setattr(torch, "randn_like", lambda t: randn(t.shape, dtype=t.dtype).to(t.device) if t.is_cuda else randn_like(t))


@pytest.mark.parametrize("kw", [dict(num_steps=6), dict(num_steps=1), dict(num_steps=5, s_churn=0.0, sigma_max=5.0),
                                dict(num_steps=7, s_min=0.1, s_max=3.0, s_noise=1.1)])  # fmt: skip
def test_updates_on_cuda_equal_those_on_the_cpu(monkeypatch, kw):
    """The same draws and the same denoiser, one that is not linear in the sample, depends on the noise level, is not centred
    and writes into padded rows, so that a wrong slope, half step, mask or centring shows.

    Both branches round in fp32: fewer than 20 roundings of 2^-24 per update of values of at most the first noise level
    times 5 (draws) and steps that shrink the sample, whose slopes (x - D) / t carry them on with a factor dt / t below 1
    per step.  2e-5 of the largest value is 20 x 2^-24 x 16; an error in the algebra is of the order of the step itself."""
    _draws_on_the_cpu(monkeypatch)
    n = torch.tensor([9, 6, 1, 4, 9])

    def denoise(a, c, sigma):
        k = 1.0 / (1.0 + sigma * sigma)
        return k * a + 0.3 * torch.sin(a) + 0.1 * sigma, k * c + 0.2 * torch.cos(c) - 0.05

    outs = []
    for device in ("cpu", "cuda:0"):
        torch.manual_seed(11)
        outs.append(edm_sample(_Net(device), n, denoiser=denoise, **kw))
    pad = build_pad_mask(n)
    for x, y in zip(outs[0][:2], outs[1][:2]):
        y = y.cpu()
        assert y[pad].abs().max() == 0
        assert (x - y).abs().max() <= 2e-5 * max(1.0, x.abs().max().item(), kw.get("sigma_max", 10.0))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_a_denoiser_may_return_other_types_and_broadcast_shapes(dtype):
    """Its outputs enter the updates by value, as in element-wise operations."""
    n = torch.tensor([9, 6, 1, 4])
    outs = []
    for convert in (lambda t: t, lambda t: t.float()):
        torch.manual_seed(4)
        low = lambda a, c, sigma: (convert((0.5 * a[:1]).to(dtype)), convert((0.5 * c).to(dtype)))  # noqa: B023, E731
        outs.append(edm_sample(_Net("cuda:0"), n, denoiser=low, num_steps=4))
    for x, y in zip(outs[0][:2], outs[1][:2]):
        assert torch.equal(x, y) and torch.isfinite(x).all()


@pytest.mark.parametrize("name,kw", [("churn", dict(num_steps=5)), ("plain", dict(num_steps=3, s_churn=0.0, sigma_max=5.0))])
def test_sampler_on_cuda_matches_the_reference(golden, monkeypatch, name, kw):
    """The reference's own samples (fp32, as on the CPU), with the network and the updates on the GPU.  The network's fp32
    kernels are held to 1e-4 elsewhere; a run evaluates it up to nine times."""
    from test_trunk import _golden_net

    _draws_on_the_cpu(monkeypatch)
    net = _golden_net(golden("trunk_edm.npz"), "cuda", device="cuda:0")
    net.eval()
    g = golden("sampler_edm.npz")
    torch.manual_seed(77)
    atoms, coords, _ = edm_sample(net, g["num_atoms"].long(), atom_channels=6, use_cuda_graph=False, **kw)
    torch.testing.assert_close(atoms.cpu(), g[name + "_atoms"], atol=9e-4, rtol=9e-4)
    torch.testing.assert_close(coords.cpu(), g[name + "_coords"], atol=9e-4, rtol=9e-4)
