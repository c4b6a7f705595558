"""The gated residual and the LayerNorm-modulate behind it in one pass, against the two operators."""
import pytest
import torch

from matterformer_b200 import fused

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,C,xd,hd,padded", [(1, 1, 8, torch.float32, torch.float32, True), (3, 29, 512, torch.bfloat16, torch.bfloat16, True),
                                                (2, 9, 264, torch.float32, torch.bfloat16, False), (700, 5, 1024, torch.bfloat16, torch.float32, True)])  # fmt: skip
def test_one_pass_equals_two_operators(B, N, C, xd, hd, padded):
    g = torch.Generator(device="cuda").manual_seed(C)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    x, a = rnd(B, N, C).to(xd).requires_grad_(True), rnd(B, N, C).to(hd).requires_grad_(True)
    gate, shift, scale = (rnd(B, C).requires_grad_(True) for _ in range(3))
    pad = (torch.rand(B, N, device="cuda", generator=g) < 0.3) if padded else None
    leaves = [x, gate, a, shift, scale]
    y0 = fused.gated_residual(x, gate, a, pad)
    h0 = fused.ln_modulate(y0, shift, scale, eps=1e-6, out_dtype=hd)
    y, h = fused.gated_ln_modulate(x, gate, a, pad, shift, scale, eps=1e-6, out_dtype=hd)
    assert torch.equal(y, y0) and torch.equal(h, h0)
    gy, gh = rnd(B, N, C).to(xd), rnd(B, N, C).to(hd)
    want = torch.autograd.grad([y0, h0], leaves, [gy, gh])
    for u, v, t in zip(torch.autograd.grad([y, h], leaves, [gy, gh]), want, leaves):
        tol = 2e-2 if torch.bfloat16 in (xd, hd) else 1e-5  # dx: one rounding of the sum instead of two
        torch.testing.assert_close(u.float(), v.float(), atol=tol * float(v.float().abs().max()), rtol=tol)


def test_operands_that_would_need_broadcasting_are_refused():
    """The kernels read one vector per molecule and one row per token where they expect them."""
    from matterformer_b200 import fused

    x, v, pad = torch.zeros(3, 4, 16, device="cuda"), torch.zeros(3, 16, device="cuda"), torch.zeros(3, 4, dtype=torch.bool, device="cuda")
    kw = dict(eps=1e-6, out_dtype=torch.float32)
    fused.gated_ln_modulate(x, v, x, pad, v, v, **kw)
    for args in ((x, v[:1], x, pad, v, v), (x, v, x[:1], pad, v, v), (x, v, x, pad[:1], v, v), (x, v, x, pad, v[:, :8], v),
                 (x, v, x, pad, v, v.cpu())):  # fmt: skip
        with pytest.raises(ValueError, match="expected operands"):
            fused.gated_ln_modulate(*args, **kw)
    for args in ((x, v[:1], v), (x, v, v[0])):
        with pytest.raises(ValueError, match="expected operands"):
            fused.ln_modulate(*args, **kw)
    for args in ((x, v[:2], x), (x, v, x[:, :1]), (x, v, x, pad[:, :1])):
        with pytest.raises(ValueError, match="expected operands"):
            fused.gated_residual(*args)
