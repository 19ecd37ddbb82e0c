"""The chain mesh's canonical order at the edges of its ranking: cells around
what a warp sorts in one to thirty-two registers, cells ranked through
shared memory in parts, empty cells, against a stable sort by cell."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOX = 64.0


@pytest.fixture(scope="module")
def dev(gpu_lib):
    from sif_gb300 import device

    return device


def _check(dev, pos, n_cells):
    import torch

    real = pos[0].dtype.type
    inv = real(1) / (real(BOX) / real(n_cells))
    idx = [np.minimum((a * inv).astype(np.int32), n_cells - 1).astype(np.int64) for a in pos]
    cell = (idx[0] * n_cells + idx[1]) * n_cells + idx[2]
    order = np.argsort(cell, kind="stable")
    offs = np.zeros(n_cells ** 3 + 1, np.int64)
    np.cumsum(np.bincount(cell, minlength=n_cells ** 3), out=offs[1:])
    xs = [torch.from_numpy(a).cuda() for a in pos]
    mx, my, mz, got_offs, orig = dev.chain_mesh(*xs, n_cells, BOX)
    assert np.array_equal(got_offs.cpu().numpy(), offs)
    assert np.array_equal(orig.cpu().numpy(), order)
    for got, a in zip((mx, my, mz), pos):
        assert np.array_equal(got.cpu().numpy(), a[order])


# One cell of `crowd` particles among others: around the 1,024 entries a warp
# sorts, and several times that.
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("crowd", [0, 1, 31, 255, 256, 257, 1023, 1024, 1025, 5000])
@pytest.mark.parametrize("n_cells", [1, 7, 23])
def test_order_is_the_stable_sort(dev, crowd, n_cells, dtype):
    rng = np.random.default_rng(crowd + n_cells)
    spread = rng.uniform(0, BOX, (3, 3001))
    lump = BOX / n_cells * (n_cells // 2 + rng.uniform(0.01, 0.99, (3, crowd)))
    pos = np.concatenate([spread, lump], axis=1)[:, rng.permutation(3001 + crowd)]
    _check(dev, [np.ascontiguousarray(np.minimum(a, BOX * 0.999999).astype(dtype)) for a in pos], n_cells)


# Nearly empty meshes, and every size about the sorts' register counts.
@pytest.mark.parametrize("counts", [[1024] * 5, [1024, 0, 1, 1025, 1023, 2], [3] * 300, [0] * 511 + [4],
                                    [31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513] * 3])
def test_runs_of_cells(dev, counts):
    n_cells = 8
    rng = np.random.default_rng(len(counts))
    cell = np.repeat(np.arange(len(counts)), counts)
    cell = cell[rng.permutation(len(cell))]
    side = BOX / n_cells
    pos = [((c + rng.uniform(0.05, 0.95, len(cell))) * side).astype(np.float32)
           for c in (cell // 64, cell // 8 % 8, cell % 8)]
    _check(dev, pos, n_cells)


# Neighbours of a few entries each, taken by a warp together up to 32 of them;
# empty cells among them; and cells past what the warp holds between.
@pytest.mark.parametrize("counts", [[1] * 512, [0, 1, 2] * 170, [4] * 8 + [0] * 100 + [16, 16, 1] * 60,
                                    [31, 1, 32, 0, 33, 1, 0, 0, 31, 2] * 50, [0] * 31 + [32] + [0] * 480])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_neighbours_taken_together(dev, counts, dtype):
    n_cells = 70  # enough for 32 neighbours a warp
    rng = np.random.default_rng(len(counts))
    cell = np.repeat(np.arange(len(counts)) + 7000, counts)
    cell = cell[rng.permutation(len(cell))]
    side = BOX / n_cells
    pos = [((c + rng.uniform(0.05, 0.95, len(cell))) * side).astype(dtype)
           for c in (cell // 4900, cell // 70 % 70, cell % 70)]
    _check(dev, pos, n_cells)


# The passes over the particles one and four a thread, about where they change.
@pytest.mark.parametrize("n", [(1 << 17) - 1, 1 << 17, (1 << 17) + 1])
@pytest.mark.parametrize("n_cells", [9, 100])
def test_few_and_many_particles(dev, n, n_cells):
    rng = np.random.default_rng(n)
    _check(dev, [(rng.uniform(0, BOX, n) * 0.999999).astype(np.float32) for _ in range(3)], n_cells)
