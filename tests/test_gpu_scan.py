"""The candidate scan's threshold test in both forms: counts against numpy at
grids whose cells fill the scan's chunks of 8,192 and leave a remainder, on
fields holding what a threshold can go wrong at. (The float form compares;
the FP64 form orders the values' bits.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev(gpu_lib):
    from sif_gb300 import device

    return device


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n", [20, 21, 32, 41])
@pytest.mark.parametrize("threshold", [-0.7, -1e-30])
def test_candidates_at_the_threshold(dev, n, dtype, threshold):
    import torch

    rng = np.random.default_rng(n)
    f = rng.uniform(-1.0, 1.0, n ** 3).astype(dtype)
    thr = np.dtype(dtype).type(threshold)
    special = [thr, np.nextafter(thr, -1, dtype=dtype), np.nextafter(thr, 1, dtype=dtype), 0.0, -0.0, np.nan,
               -np.nan, np.inf, -np.inf, np.finfo(dtype).tiny, -np.finfo(dtype).tiny]
    f[rng.permutation(n ** 3)[: 50 * len(special)]] = np.repeat(np.array(special, dtype), 50)
    f[-1] = thr
    xs = [torch.from_numpy(rng.uniform(0, 100.0, 4000).astype(dtype)).cuda() for _ in range(3)]
    mesh = dev.chain_mesh(*xs, 10, 100.0)
    dev.exodus(torch.zeros(n ** 3, dtype=getattr(torch, dtype), device="cuda"), n, 100.0, mesh, 10, [12.0],
               threshold, inject=torch.from_numpy(f).cuda())
    with np.errstate(invalid="ignore"):
        want = int((f <= thr).sum())
    assert dev.last_rung_stats()[0]["n_candidates"] == want
