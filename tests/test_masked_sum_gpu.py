"""The one-pass masked, centred sums of the EDM preconditioner and sampler."""
import pytest
import torch

from matterformer_b200 import fused
from matterformer_b200.trunk import _masked_mean

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,C,center", [(1, 1, 3, True), (5, 29, 3, True), (3, 128, 3, True), (2, 333, 3, True), (4, 29, 7, False), (2, 300, 1, False)])
def test_masked_sum_against_torch(B, N, C, center):
    """One row, a CTA's threads exactly, more rows than threads, an empty molecule; per-molecule and plain scales; gradients."""
    g = torch.Generator(device="cuda").manual_seed(N)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    x, y, z, p, q = (rnd(B, N, C).requires_grad_(True) for _ in range(5))
    pad = torch.rand(B, N, device="cuda", generator=g) < 0.3
    pad[0] = B > 1  # an empty molecule unless it is the only one
    a, c = rnd(B), rnd(B)

    def ref(v):
        v = v.masked_fill(pad[..., None], 0.0)
        return (v - _masked_mean(v, pad)).masked_fill(pad[..., None], 0.0) if center else v

    want = ref(a[:, None, None] * x + c[:, None, None] * (y - z))
    got = fused.masked_sum(pad, x, a=a, y=y, z=z, c=c, center=center)
    torch.testing.assert_close(got, want, atol=1e-6, rtol=1e-5)
    go = rnd(B, N, C)
    for u, v in zip(torch.autograd.grad(got, [x, y, z], go), torch.autograd.grad(want, [x, y, z], go)):
        torch.testing.assert_close(u, v, atol=1e-6, rtol=1e-5)
    with torch.no_grad():
        want = ref(0.5 * x + 0.25 * y - 3.0 * (p - q))
        torch.testing.assert_close(fused.masked_update(pad, x, 0.5, y, None, 0.25, p, q, -3.0, center), want, atol=2e-6, rtol=1e-5)


def test_operands_of_other_types_shapes_and_places_are_refused():
    """The kernel reads them as they lie: a narrower type, a shorter factor or a host tensor would be read beyond its end."""
    x, pad = torch.zeros(4, 5, 3, device="cuda"), torch.zeros(4, 5, dtype=torch.bool, device="cuda")
    for bad in (dict(y=x.bfloat16()), dict(y=x[:1]), dict(y=x.cpu()), dict(y=x, z=x[:, :4]), dict(p=x, q=x.half(), k=1.0),
                dict(a=torch.ones(1, device="cuda")), dict(a=torch.ones(4, device="cuda", dtype=torch.float64)),
                dict(y=x, c=torch.ones(8, device="cuda")[::2]), dict(a=torch.ones(4))):  # fmt: skip
        with pytest.raises(ValueError, match="masked sums take"):
            fused.masked_update(pad, x, **bad)
    for args in ((pad.cpu(), x), (pad.float(), x), (pad[:, :4], x), (pad, x.cpu()), (pad, x.double())):
        with pytest.raises(ValueError, match="masked sums take"):
            fused.masked_update(*args)
