"""The deposit's tiles of crowded cells, summed in two passes over their
particles: against the weighted deposit of weights of 1, which is the same
integers by two words a cell, and against the particles in another order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, BOX = 40, 80.0  # three tiles a side, the last of eight cells


# A crowd about one point: below and above a cell's 256, a tile taken for a
# dense one unseen (32,768 particles and four times the mean), one taken in two
# parts (past 2^20 - 1); inside a tile and across the corner of eight.
@pytest.mark.parametrize("count", [200, 3000, 32768, 32769, (1 << 20) - 1, 1 << 20, 1500001])
@pytest.mark.parametrize("at,spread", [((9.3, 50.1, 70.7), 0.4), ((32.0, 64.0, 0.0), 3.0)],
                         ids=["inside", "corner"])
def test_crowds_sum_exactly(gpu_lib, count, at, spread):
    import torch

    from sif_gb300 import device

    g = torch.Generator(device="cuda").manual_seed(count)
    pos = []
    for c in at:
        crowd = c + spread * torch.randn(count, generator=g, device="cuda")
        field = BOX * torch.rand(20000, generator=g, device="cuda")
        v = torch.remainder(torch.cat([crowd, field]), BOX)
        pos.append(torch.where(v >= BOX, torch.zeros_like(v), v))
    got = device.cic(*pos, N, BOX)
    ones = torch.ones_like(pos[0])
    assert torch.equal(got.view(torch.int32), device.cic_weighted(*pos, ones, N, BOX).view(torch.int32))
    p = torch.randperm(len(ones), generator=g, device="cuda")
    again = device.cic(*[v[p].contiguous() for v in pos], N, BOX)
    assert torch.equal(got.view(torch.int32), again.view(torch.int32))
    # Every particle is whole: the cells sum to the count, each rounded once.
    total = float(got.double().sum()) * (BOX / N) ** 3
    assert abs(total - len(ones)) <= 2.0 ** -23 * len(ones)
