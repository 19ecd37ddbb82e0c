"""Chain meshes of boxes so small that a cell's reciprocal is infinite: every
particle off zero in the mesh's last cell on that axis, zero in its first, as
a conversion that saturates and takes NaN to zero places them; and a box a
little larger, whose reciprocal is finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CELLS = 8


@pytest.mark.parametrize("dtype,box", [(np.float32, 1e-38), (np.float32, 1e-37), (np.float64, 1e-308),
                                       (np.float64, 1e-306)])
def test_cells_stay_in_the_mesh(gpu_lib, dtype, box):
    import torch

    from sif_gb300 import device

    rng = np.random.default_rng(5)
    side = dtype(box)
    pos = [(rng.integers(0, 1000, 3000) / 1000.0 * float(side)).astype(dtype) for _ in range(3)]
    pos[1][:100] = 0
    pos[2][50:200] = dtype(-0.0)
    with np.errstate(over="ignore", invalid="ignore"):
        inv = dtype(1) / (side / dtype(CELLS))
        u = [np.nan_to_num(a * inv, nan=0.0, posinf=CELLS) for a in pos]
    idx = [np.minimum(v, CELLS - 1).astype(np.int64) for v in u]
    cell = (idx[0] * CELLS + idx[1]) * CELLS + idx[2]
    order = np.argsort(cell, kind="stable")
    offs = np.concatenate([[0], np.cumsum(np.bincount(cell, minlength=CELLS ** 3))])
    xs = [torch.from_numpy(a).cuda() for a in pos]
    got = device.chain_mesh(*xs, CELLS, box)
    assert np.array_equal(got[3].cpu().numpy(), offs)
    assert np.array_equal(got[4].cpu().numpy(), order)
    for g, a in zip(got, pos):
        assert np.array_equal(g.cpu().numpy(), a[order])
