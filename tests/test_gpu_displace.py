"""Displacement's commit, which takes survivors that lie apart together,
against the oracle's one after another, on the GPU's own fields: rungs of
none, a few and thousands of survivors, dense enough that many lie near one
another, and spheres from a cell to a quarter of the box."""
import numpy as np
import pytest

from conftest import same_catalogue
from sif_gb300 import abi, synth

pytestmark = pytest.mark.gpu

N, BOX = 72, 180.0


@pytest.fixture(scope="module")
def dev(gpu_lib):
    from sif_gb300 import device

    return device


@pytest.mark.parametrize("threshold,overlap,minima", [(-0.4, 0.0, False), (-0.5, 0.5, False),
                                                      (-0.6, 1.0, True), (-0.8, 1.0, False)])
def test_displacement_matches_the_oracle(dev, oracle, threshold, overlap, minima):
    import torch

    opt = abi.SIF_FINDER_DISPLACE | (abi.SIF_FINDER_SEEDS_MINIMA if minima else 0)
    x, y, z = synth.zeldovich(N, BOX, 6.0, 77)
    xs = [torch.from_numpy(a).cuda() for a in (x, y, z)]
    grid = dev.cic(*xs, N, BOX)
    dev.density_contrast(grid)
    radii = np.sort(synth.ladder(3.0, 45.0, 0.15).astype(np.float32))[::-1]
    fields = torch.stack([dev.smooth(grid, N, BOX, float(r)) for r in radii])
    got = dev.exodus(grid, N, BOX, dev.chain_mesh(*xs, 18, BOX), 18, radii, threshold, overlap, opt,
                     inject=fields.reshape(-1))
    displaced = sum(r["n_displaced"] for r in dev.last_rung_stats())
    want = oracle.exodus(grid.cpu().numpy(), oracle.OracleMesh(x, y, z, 18, BOX), radii, N, BOX,
                         threshold, overlap, opt, n_threads=4, inject=fields.cpu().numpy())
    assert len(want[0]) > 20 and same_catalogue(got, want), (len(got[0]), len(want[0]), displaced)


# A lattice of small voids to start from, which candidates between its nodes
# clear at the rung's radius and reach at their own: survivors that each
# displace several voids (their order, the spheres painted back), in rungs of
# more survivors than the commit tests at once.
@pytest.mark.parametrize("spacing,r0,radii,threshold,overlap", [(9.0, 0.8, (6, 5, 4), -0.6, 0.0),
                                                                (7.5, 0.6, (6, 5, 4.5), -0.7, 0.5)])
def test_survivors_that_displace_several(dev, oracle, spacing, r0, radii, threshold, overlap):
    import torch

    x, y, z = synth.zeldovich(N, BOX, 6.0, 77)
    xs = [torch.from_numpy(a).cuda() for a in (x, y, z)]
    grid = dev.cic(*xs, N, BOX)
    dev.density_contrast(grid)
    radii = np.array(radii, np.float32)
    fields = torch.stack([dev.smooth(grid, N, BOX, float(r)) for r in radii])
    q = (np.arange(int(BOX / spacing)) + 0.5) * spacing
    prior = [v.reshape(-1).astype(np.float32) for v in np.meshgrid(q, q, q, indexing="ij")]
    prior.append(np.full(len(prior[0]), r0, np.float32))
    got = dev.exodus(grid, N, BOX, dev.chain_mesh(*xs, 18, BOX), 18, radii, threshold, overlap,
                     abi.SIF_FINDER_DISPLACE, inject=fields.reshape(-1), prior=prior)
    stats = dev.last_rung_stats()
    want = oracle.exodus(grid.cpu().numpy(), oracle.OracleMesh(x, y, z, 18, BOX), radii, N, BOX,
                         threshold, overlap, abi.SIF_FINDER_DISPLACE, n_threads=4,
                         inject=fields.cpu().numpy(), prior=prior)
    assert any(r["n_displaced"] > r["n_accepted"] and r["n_survivors"] > 32 for r in stats), stats
    assert same_catalogue(got, want), (len(got[0]), len(want[0]))
