"""last_timings()'s mesh_ms covers the whole build of a chain_mesh call, its
first pass over the particles among it: of a build of a millisecond and a half
and two launches' and one read's gaps of some 30 us, at least 93%."""
import pytest

pytestmark = pytest.mark.gpu


def test_mesh_time_is_the_whole_build(gpu_lib):
    import torch

    from sif_gb300 import device

    pos = [torch.rand(1 << 26, device="cuda") * 99.9 for _ in range(3)]
    a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    shares = []
    for _ in range(6):
        torch.cuda.synchronize()
        a.record(device.stream())
        device.chain_mesh(*pos, 100, 100.0)
        b.record(device.stream())
        b.synchronize()
        shares.append(device.last_timings()["mesh_ms"] / a.elapsed_time(b))
    assert 0.93 <= max(shares) <= 1.0, shares
