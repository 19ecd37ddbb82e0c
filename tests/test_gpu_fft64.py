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
