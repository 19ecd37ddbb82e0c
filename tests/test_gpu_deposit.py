"""The tiled deposit where a tile's one-word sums end: cells that reach 2^32
quanta (256 particles on one node) and the tiles done again with two words,
against an exact count and the FP64 oracle."""
import numpy as np
import pytest

from conftest import same_bits
from sif_gb300 import synth

pytestmark = pytest.mark.gpu

N, BOX = 40, 80.0  # nodes every 2 units: exact in float


@pytest.fixture(scope="module")
def dev(gpu_lib):
    from sif_gb300 import device

    return device


def _cic(dev, x, y, z):
    import torch

    xs = [torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda() for a in (x, y, z)]
    return dev.cic(*xs, N, BOX).cpu().numpy().reshape(N, N, N)


# Around the wrap of one 32-bit word, past 2^16 particles a tile (the carry
# form of the second kernel), and past what any tile's words can hold.
@pytest.mark.parametrize("count", [1, 255, 256, 257, 512, 65535, 65537, 256 * 17 ** 3 + 1])
@pytest.mark.parametrize("node", [(5, 6, 7), (16, 0, 31)], ids=["inside", "face"])
def test_particles_on_one_node_are_counted_exactly(dev, count, node):
    pos = [np.full(count, 2.0 * k, np.float32) for k in node]
    g = _cic(dev, *pos)
    want = np.zeros((N, N, N), np.float32)
    # count quanta-exact particles in a cell of volume 8, rounded once.
    want[node] = np.float32(np.float32(count) * np.float32(1.0 / 8.0))
    assert same_bits(g, want)


def test_dense_tiles_beside_sparse_ones(dev, oracle):
    x, y, z = synth.zeldovich(32, BOX, 3.0, 9)
    rng = np.random.default_rng(4)
    blob = rng.uniform(33.0, 35.0, (3, 40000))  # 5,000 a cell over a tile's face
    x, y, z = (np.concatenate([a, b]).astype(np.float32) for a, b in zip((x, y, z), blob))
    g = _cic(dev, x, y, z)
    perm = rng.permutation(len(x))
    assert same_bits(g, _cic(dev, x[perm], y[perm], z[perm]))
    want = oracle.cic_f64(x, y, z, N, BOX).reshape(N, N, N)
    # Each cell's sum is exact to half a quantum of 2^-24 a particle, of which
    # no more than len(blob) reach it, then rounded to float: 2^-24 relative.
    err = np.abs(g.astype(np.float64) - want) * 8.0
    assert (err <= 2.0 ** -24 * (want * 8.0) + 2.0 ** -24 * 8 * blob.shape[1]).all()
