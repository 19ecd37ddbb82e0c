"""A small rung's commit in one cluster launch against the rounds launched one
by one: the same catalogue, over ladders whose rungs run from none to more
survivors than the cluster takes, in every form it is chosen for."""
import numpy as np
import pytest

from conftest import same_catalogue, same_catalogue64
from sif_gb300 import abi, synth

pytestmark = pytest.mark.gpu

N, BOX = 112, 280.0


@pytest.fixture(scope="module")
def dev(gpu_lib):
    from sif_gb300 import device

    return device


def _catalogues(dev, xs, **kw):
    radii = synth.ladder(4.0, 60.0, 0.1).astype(np.float32 if xs[0].element_size() == 4 else np.float64)
    out = []
    for mode in (0, 1):
        dev.set_commit_mode(mode)
        try:
            out.append(dev.box(*xs, N, BOX, 28, radii, **kw))
            stats = dev.last_rung_stats()
        finally:
            dev.set_commit_mode(0)
    return out, stats


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("kw", [dict(threshold=-0.5), dict(threshold=-0.8, overlap=0.4),
                                dict(threshold=-0.6, options=abi.SIF_FINDER_LAGRANGIAN_OVERLAP),
                                dict(threshold=-0.6, options=abi.SIF_FINDER_SEEDS_MINIMA)],
                         ids=["many", "overlap", "lagrangian", "minima"])
def test_cluster_commit_is_the_rounds(dev, kw, dtype):
    import torch

    xs = [torch.from_numpy(a).cuda().to(getattr(torch, dtype)) for a in synth.zeldovich(N, BOX, 5.0, 31)]
    (small, rounds), stats = _catalogues(dev, xs, **kw)
    counts = [r["n_candidates"] for r in stats]
    assert any(0 < c <= 4096 for c in counts), counts
    if kw["threshold"] == -0.5:
        assert max(counts) > 4096, counts  # and rungs past the cluster's share
    assert len(small[0]) > 20
    assert (same_catalogue if dtype == "float32" else same_catalogue64)(small, rounds)


def test_long_chains_of_undecided_survivors(dev):
    """Voids in a row whose depths fall along it: each survivor waits for the
    one before it, more rounds than the counters' ring holds."""
    import torch

    n, box = 256, 256.0
    # A uniform lattice with nothing inside a thin tube: every node on its axis
    # is a candidate, and a rising field orders them along it. A void's radius
    # is about 1.64 of the tube's, so some seventy fit in a row.
    q = torch.arange(n, device="cuda", dtype=torch.float32) + 0.5
    x, y, z = (v.reshape(-1) for v in torch.meshgrid(q, q, q, indexing="ij"))
    keep = (x - 128) ** 2 + (y - 128) ** 2 > 2.0 ** 2
    xs = [v[keep].contiguous() for v in (x, y, z)]
    field = torch.ones((n, n, n), device="cuda")
    field[128, 128, 8:248] = torch.linspace(-0.99, -0.9, 240, device="cuda")
    mesh = dev.chain_mesh(*xs, 64, box)
    out = []
    for mode in (0, 1):
        dev.set_commit_mode(mode)
        try:
            out.append(dev.exodus(torch.zeros(n ** 3, device="cuda"), n, box, mesh, 64, [2.0], -0.5,
                                  overlap=0.9, inject=field.reshape(-1)))
            rounds = max(r["rounds"] for r in dev.last_rung_stats())
        finally:
            dev.set_commit_mode(0)
        assert rounds > 64
    assert same_catalogue(*out)
