"""The search where its smoothings' lanes and scans change form -- two lanes with
scans of their own, two lanes and one list, one stream -- against the same
search on the same fields smoothed beforehand."""
import numpy as np
import pytest

from conftest import same_catalogue
from sif_gb300 import synth

pytestmark = pytest.mark.gpu

BOX, MESH = 200.0, 20


@pytest.mark.parametrize("n,dtype", [(256, np.float32), (264, np.float32), (264, np.float64),
                                     (330, np.float32), (648, np.float32)])
def test_lanes_find_what_the_fields_hold(gpu_lib, n, dtype):
    import torch

    from sif_gb300 import device

    xs = [torch.from_numpy(a.astype(dtype)).cuda() for a in synth.zeldovich(64, BOX, 7.0, 21)]
    grid = device.cic(*xs, n, BOX)
    device.density_contrast(grid)
    mesh = device.chain_mesh(*xs, MESH, BOX)
    radii = np.array([30.0, 22.0, 16.0, 12.0, 10.0], dtype)
    # A size's first search takes one stream, the ones after it a lane more each.
    got = [device.exodus(grid, n, BOX, mesh, MESH, radii, -0.75) for _ in range(4)]
    fields = torch.cat([device.smooth(grid, n, BOX, float(r)) for r in radii])
    want = device.exodus(grid, n, BOX, mesh, MESH, radii, -0.75, inject=fields)
    assert len(want[0]) > 5
    assert [same_catalogue(c, want) for c in got] == [True] * 4, [len(c[0]) for c in (*got, want)]
