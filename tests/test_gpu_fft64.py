"""The FP64 form's own transforms (128 and 256 cells a side) against numpy.

The bar, on white noise: two transforms of 3 log2(n) levels, each level's
rounding at most two units of 2^-53 of the values' rms (a rotation in two
fused multiply-adds, a butterfly), all in one direction -- and as much for
numpy's own.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOX, RADIUS = 100.0, 7.0


def _bar(n):
    return 2 * (2 * 3 * np.log2(n) * 2) * 2.0 ** -53


def _noise(n):
    return np.random.default_rng(n).standard_normal(n ** 3)


def _want(delta, n, filt, window):
    k = np.fft.fftfreq(n, 1.0 / n)
    kz = np.arange(n // 2 + 1)
    x = RADIUS * 2 * np.pi / BOX * np.sqrt(
        (k * k)[:, None, None] + (k * k)[None, :, None] + (kz * kz)[None, None, :])
    x[0, 0, 0] = 1.0
    w = 3 * (np.sin(x) - x * np.cos(x)) / x ** 3 if filt == "top-hat" else np.exp(-x * x / 2)
    w[0, 0, 0] = 1.0
    if window != "none":
        y = np.pi * np.abs(np.arange(n) - n * (np.arange(n) > n // 2)) / n
        s2 = np.sinc(y / np.pi) ** 2
        a = 1 / s2 if window == "full" else s2 / (1 - 2 * np.sin(y) ** 2 / 3)
        w = w * (a[:, None, None] * a[None, :, None] * a[None, None, : n // 2 + 1])
    return np.fft.irfftn(np.fft.rfftn(delta.reshape(n, n, n)) * w, s=(n, n, n), axes=(0, 1, 2)).reshape(-1)


@pytest.fixture(scope="module")
def dev(gpu_lib):
    from sif_gb300 import device

    return device


@pytest.mark.parametrize("n", [128, 256])
@pytest.mark.parametrize("filt,window", [("top-hat", "full"), ("top-hat", "none"),
                                         ("gaussian", "aliasing")])
def test_fp64_transforms_match_numpy(dev, n, filt, window):
    import torch

    delta = _noise(n)
    got = dev.smooth(torch.from_numpy(delta).cuda(), n, BOX, RADIUS, filter=filt, window=window)
    want = _want(delta, n, filt, window)
    rms = np.sqrt(np.mean((got.cpu().numpy() - want) ** 2) / np.mean(want * want))
    assert rms <= _bar(n), rms


@pytest.mark.parametrize("n", [128, 256])
def test_fp64_transforms_from_an_odd_double(dev, n):
    """A grid that starts on 8 bytes, not 16; the smoothing that changes nothing."""
    import torch

    delta = torch.from_numpy(np.concatenate([[7.0], _noise(n)])).cuda()[1:]
    assert delta.data_ptr() % 16 == 8
    got = dev.smooth(delta, n, BOX, 1e-7, window="none")
    rms = float((got - delta).pow(2).mean().sqrt())
    assert rms <= _bar(n) / 2, rms


@pytest.mark.parametrize("n", [128, 256])
def test_fp64_transforms_lose_no_bits(dev, n):
    """White noise there and back: a value's rounding at a level is a random
    step of rms 2^-53 of the values at most (a rotation, a butterfly and the
    constant between them, each uniform within half a unit), so the steps of 2
    * 3 log2(n) levels and four more of the packing add up as their root."""
    import torch

    delta = torch.from_numpy(_noise(n)).cuda()
    got = dev.smooth(delta, n, BOX, 1e-7, window="none")
    rms = float((got - delta).pow(2).mean().sqrt() / delta.pow(2).mean().sqrt())
    assert rms <= np.sqrt(2 * 3 * np.log2(n) + 4) * 2.0 ** -53, rms


# One wave each, at the modes where the rows' packing and the columns' filter
# change form, through a Gaussian: the wave times its factor, to what every
# level's two units give when all of them go one way.
@pytest.mark.parametrize("n", [128, 256])
def test_fp64_transforms_of_single_waves(dev, n):
    import torch

    h = n // 2
    i = torch.arange(n, dtype=torch.int64, device="cuda")
    for kx, ky, kz in [(0, 0, 1), (0, 0, n // 8), (1, 0, n // 8 + 1), (0, 3, n // 4), (5, h, n // 4 - 1),
                       (0, 0, h), (h, h, h), (h, 0, 0), (0, h, 0), (n - 1, 2, 0), (h - 1, h + 1, 3 * n // 8),
                       (7, n - 7, h - 1)]:
        turn = (kx * i[:, None, None] + ky * i[None, :, None] + kz * i[None, None, :]) % n
        wave = torch.cos(2 * np.pi / n * turn.double()).reshape(-1)
        got = dev.smooth(wave, n, BOX, RADIUS / 8, filter="gaussian", window="none")
        k = [min(v, n - v) for v in (kx, ky, kz)]
        factor = np.exp(-0.5 * (RADIUS / 8 * 2 * np.pi / BOX) ** 2 * sum(v * v for v in k))
        err = float((got - factor * wave).abs().max())
        assert err <= _bar(n) / 2, (kx, ky, kz, err)
