"""The C++ host path of the differentiable operators against the Python one: same kernels, so the same bits."""
import pytest
import torch

import matterformer_b200 as mfb
from matterformer_b200 import _lib

pytestmark = pytest.mark.gpu


def _both(call, leaves, grad, monkeypatch):
    assert _lib.native() is not None
    results = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(_lib, "_NATIVE", [None])
        out = call()
        assert ("Backward" in type(out.grad_fn).__name__) == (not native)  # (a C++ node has another name)
        results.append([out, *torch.autograd.grad(out, leaves, grad)])
    for a, b in zip(*results):
        assert a.dtype == b.dtype and torch.equal(a, b)


@pytest.mark.parametrize("dtype,N,bias,rank,pair,frozen", [
    (torch.float32, 7, False, 0, False, ()), (torch.bfloat16, 40, False, 0, True, (1,)), (torch.bfloat16, 20, True, 0, True, (5, 8)),
    (torch.bfloat16, 40, True, 0, False, (6,)), (torch.bfloat16, 11, False, 5, False, (6,)), (torch.float32, 9, True, 4, True, ()),
])  # fmt: skip
def test_simplicial_attention(dtype, N, bias, rank, pair, frozen, monkeypatch):
    """With and without each optional operand, and with gradients that are not asked for."""
    g = torch.Generator("cuda").manual_seed(N)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    B, H, D = 2, 3, 64
    valid = torch.arange(N, device="cuda")[None] < torch.tensor([[N], [N - 2]], device="cuda")
    heads = [(rnd(B, H, N, D) / 8).to(dtype) for _ in range(5)]
    extra = {}
    if bias:
        extra["factorized_bias"] = (rnd(B, H, N, N), rnd(B, H, N, N), rnd(B, H, N, N), rnd(B, H, N))
    if rank:
        extra["angle_residual"] = (rnd(B, H, N, N, rank), rnd(B, H, N, N, rank), rnd(B, H, N))
        extra["message_residual"] = (rnd(B, H, N, N, rank), rnd(B, H, N, N, rank), rnd(H, rank, D))
    leaves = [*heads, *(t for group in extra.values() for t in group)]
    for i, t in enumerate(leaves):
        t.requires_grad_(i not in frozen)
    call = lambda: mfb.simplicial_attention_cuda(*heads, query_valid=valid, pair_key_valid=valid,  # noqa: E731
                                                 pair_valid=valid[:, :, None] & valid[:, None, :] if pair else None, **extra)  # fmt: skip
    _both(call, [t for t in leaves if t.requires_grad], rnd(B, H, N, D).to(dtype), monkeypatch)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sparse_attention(dtype, monkeypatch):
    g = torch.Generator("cuda").manual_seed(3)
    q, k, v = ((torch.randn(2, 2, 70, 64, generator=g, device="cuda") / 8).to(dtype).requires_grad_(True) for _ in range(3))
    n = torch.tensor([70, 41], device="cuda", dtype=torch.int32)
    grad = torch.randn(2, 2, 70, 64, generator=g, device="cuda").to(dtype)
    blocks = mfb.build_radius_blocks(torch.rand(2, 70, 3, generator=g, device="cuda"), torch.full((2, 6), 2.3, device="cuda") *
                                     torch.tensor([1, 1, 1, 0, 0, 0], device="cuda"), n, 4.0)  # fmt: skip
    _both(lambda: mfb.local_window_attention(q, k, v, n, window=16), [q, k, v], grad, monkeypatch)
    monkeypatch.undo()
    _both(lambda: mfb.radius_block_sparse_attention(q, k, v, blocks), [q, k, v], grad, monkeypatch)


def test_operands_that_need_converting_take_the_python_path():
    N = 9
    valid = torch.ones(1, N, device="cuda", dtype=torch.bool)
    t = [torch.randn(1, N, 2, 32, device="cuda").transpose(1, 2) for _ in range(5)]
    a = mfb.simplicial_attention_cuda(*t, query_valid=valid, pair_key_valid=valid.float())
    b = mfb.simplicial_attention_cuda(*(x.contiguous() for x in t), query_valid=valid, pair_key_valid=valid)
    assert torch.equal(a, b)
    with pytest.raises(ValueError, match="k1 must match q"):
        mfb.simplicial_attention_cuda(t[0], t[1][:, :1], *t[2:], query_valid=valid, pair_key_valid=valid)


@pytest.mark.parametrize("counts", [None, torch.int32, torch.int64])
@pytest.mark.parametrize("form", ["latent", "cell", "strided"])
def test_neighbour_and_block_lists(counts, form, monkeypatch):
    """Operands that the C++ functions take as they are and operands that need converting: the bits of the Python path."""
    g = torch.Generator("cuda").manual_seed(5)
    pos = torch.rand(3, 3, 70, generator=g, device="cuda").transpose(1, 2)
    pos = pos if form == "strided" else pos.contiguous()
    lattice = torch.tensor([2.3, 2.4, 2.5, 0.1, -0.05, 0.2], device="cuda").repeat(3, 1)
    lattice = mfb.lattice_latent_to_cell(lattice) if form == "cell" else lattice
    n = counts and torch.tensor([70, 41, 1], device="cuda", dtype=counts)
    results = []
    for native in (_lib.native(), None):
        monkeypatch.setattr(_lib, "_NATIVE", [native])
        b = mfb.build_radius_blocks(pos, lattice, n, 4.0)
        results.append([b.perm, b.block_count, b.block_cols, b.block_mask, b.num_atoms, *mfb.knn_topk(pos, lattice, n, k=7),
                        *mfb.knn_topk(pos, lattice, n, k=3, include_self=True)])  # fmt: skip
    for a, c in zip(*results):
        assert a.dtype == c.dtype and torch.equal(a, c)
    monkeypatch.undo()
    for bad in (0, 33):
        with pytest.raises(ValueError, match="k must be in"):
            mfb.knn_topk(pos, lattice, n, k=bad)
    with pytest.raises(ValueError, match="cutoff must be non-negative"):
        mfb.build_radius_blocks(pos, lattice, n, -1.0)
    with pytest.raises(ValueError, match="one count per structure"):
        mfb.build_radius_blocks(pos, lattice, torch.ones(2, device="cuda", dtype=torch.int32), 4.0)
