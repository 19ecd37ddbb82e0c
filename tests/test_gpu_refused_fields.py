"""A field with particles outside the box is refused with their number, from
the build's own first pass, and what it counted does not reach the next call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOX = 50.0


@pytest.mark.parametrize("call", ["cic", "chain_mesh"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_a_refusal_leaves_nothing_behind(gpu_lib, call, dtype):
    import torch

    from sif_gb300 import device

    rng = np.random.default_rng(3)
    good = [rng.uniform(0, BOX * 0.999, 5000).astype(dtype) for _ in range(3)]
    bad = [a.copy() for a in good]
    bad[0][7], bad[1][4000], bad[2][9] = -1.0, 1.5 * BOX, np.nan
    f = getattr(device, call)
    run = lambda pos: f(*[torch.from_numpy(a).cuda() for a in pos], 12, BOX)
    want = run(good)
    for _ in range(2):
        with pytest.raises(ValueError, match="3 of 5000 particles outside"):
            run(bad)
    got = run(good)
    for a, b in zip(got if isinstance(got, tuple) else [got], want if isinstance(want, tuple) else [want]):
        assert torch.equal(a, b)
