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
