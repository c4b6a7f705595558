"""Block lists and neighbour search straight from lattice latents: cell, grid and binning inside the kernels."""
import pytest
import torch

import matterformer_b200 as mfb
from matterformer_b200 import synthetic
from matterformer_b200.sparse import cell_grid_dims
from oracle import geom_ref

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _crystals(B, N, seed, lo=8.0, hi=20.0, spread=1.0):
    g = torch.Generator().manual_seed(seed)
    lat = synthetic.random_triclinic_lattices(B, g, lo, hi)
    n = torch.randint(max(1, N // 2), N + 1, (B,), generator=g)
    n[0] = N
    return lat, torch.rand(B, N, 3, generator=g) * spread - (spread - 1) / 2, n


@pytest.mark.parametrize("B,N,cutoff,spread", [(3, 1, 3.0, 1.0), (2, 64, 3.0, 3.0), (2, 65, 9.0, 1.0), (6, 200, 4.5, 1.0), (1, 1025, 4.0, 1.0),
                                               (1, 2049, 2.0, 2.0)])  # fmt: skip
def test_block_list_from_latents_bit_exact(B, N, cutoff, spread):
    """Atoms per CTA and key-tile edges, cells smaller and larger than the cutoff, coordinates outside [0, 1)."""
    lat, frac, n = _crystals(B, N, seed=N, spread=spread)
    cell = mfb.lattice_latent_to_cell(lat.to(DEV)).cpu()
    blocks = mfb.build_radius_blocks(frac.to(DEV), lat.to(DEV), n.to(DEV), cutoff)
    perm, count, cols, mask = geom_ref.cell_sort_blocklist(frac, cell, n, cell_grid_dims(cell, cutoff), cutoff)
    for got, want in ((blocks.perm, perm), (blocks.block_count, count), (blocks.block_cols, cols), (blocks.block_mask, mask)):
        assert torch.equal(got.cpu(), want)


@pytest.mark.parametrize("B,N,k", [(3, 1, 4), (2, 33, 32), (2, 1025, 16), (1, 16384, 8), (1, 16385, 8)])
def test_knn_from_latents_matches_all_pairs(B, N, k):
    """One setup kernel per structure up to 16384 atoms, separate kernels beyond."""
    edge = (N / 0.1) ** (1 / 3)
    lat, frac, n = _crystals(B, N, seed=N + k, lo=edge, hi=1.3 * edge)
    args = (frac.to(DEV), lat.to(DEV), n.to(DEV))
    ic, dc = mfb.knn_topk(*args, k=k)
    ip, dp = mfb.knn_topk(*args, k=k, method="pairs")
    assert torch.equal(ic, ip) and torch.equal(dc, dp)


def test_equal_distances():
    """Atoms on a grid: distances that equal the cutoff, and neighbours that only their indices order."""
    axis = torch.arange(8) / 8.0
    frac = torch.stack(torch.meshgrid(axis, axis, axis, indexing="ij"), dim=-1).reshape(1, 512, 3)
    frac = frac[:, torch.randperm(512, generator=torch.Generator().manual_seed(3))]
    lat = torch.tensor([[16.0, 16.0, 16.0, 1.0, 1.0, 1.0]])
    lat = torch.cat([lat[:, :3].log(), torch.zeros(1, 3)], dim=1)
    n = torch.tensor([512])
    cell = mfb.lattice_latent_to_cell(lat.to(DEV)).cpu()
    for cutoff in (2.0, 4.0, 6.0, float(torch.tensor(8.0).sqrt()), 8.5):
        blocks = mfb.build_radius_blocks(frac.to(DEV), lat.to(DEV), n.to(DEV), cutoff)
        want = geom_ref.cell_sort_blocklist(frac, cell, n, cell_grid_dims(cell, cutoff), cutoff)
        for got, ref in zip((blocks.perm, blocks.block_count, blocks.block_cols, blocks.block_mask), want):
            assert torch.equal(got.cpu(), ref)
    args = (frac.to(DEV), lat.to(DEV), n.to(DEV))
    for k in (5, 16, 32):
        ic, dc = mfb.knn_topk(*args, k=k)
        ip, dp = mfb.knn_topk(*args, k=k, method="pairs")
        assert torch.equal(ic, ip) and torch.equal(dc, dp)


@pytest.mark.parametrize("k", [1, 8, 16, 17, 32])
@pytest.mark.parametrize("edges,N", [((13.0, 17.5, 60.0), 1300), ((14.0, 14.0, 14.0), 260), ((18.0, 18.0, 18.0), 577),
                                     ((9.0, 30.0, 30.0), 900), ((40.0, 40.0, 40.0), 385)])  # fmt: skip
def test_knn_search_paths_match_all_pairs(edges, N, k):
    """Three, four and more bins per axis (one pass over the neighbour bins, with and without crossing the boundary), fewer than
    three, lists of all atoms; half of the atoms of one structure in a corner: more candidates and survivors than the shared
    lists hold there, several shells elsewhere."""
    g = torch.Generator().manual_seed(N + k)
    lat = torch.tensor(edges).log().repeat(3, 1)
    lat = torch.cat([lat, torch.tensor([[0.0, 0.0, 0.0], [0.3, -0.2, 0.1], [0.0, 0.0, 0.0]])], dim=1)
    frac = torch.rand(3, N, 3, generator=g)
    frac[2, : N // 2] *= 0.2
    frac[1, 1] = frac[1, 0]  # two atoms in one place
    n = torch.tensor([N, N - 5, N])
    args = (frac.to(DEV), lat.to(DEV), n.to(DEV))
    for include_self in (False, True):
        ic, dc = mfb.knn_topk(*args, k=k, include_self=include_self)
        ip, dp = mfb.knn_topk(*args, k=k, include_self=include_self, method="pairs")
        assert torch.equal(ic, ip) and torch.equal(dc, dp)
