"""GPU: the envelope's Gaussian of float32 data is the FP64 sum rounded to
float32, axis by axis (what scipy stores), also where that sum lies next to the
middle of two floats.  Exact: no tolerance."""
import numpy as np
import pytest

from odtbrain_gb300 import apple as odt_apple

pytestmark = pytest.mark.gpu


def _axis(x, w, r, axis):
    """scipy's order of a symmetric correlation, in FP64, stored float32."""
    x = np.moveaxis(x, axis, 0).astype(np.float64)
    pad = np.zeros((r,) + x.shape[1:])
    x = np.concatenate([pad, x, pad])
    n = len(x) - 2 * r
    acc = x[r:r + n] * w[r]
    for j in range(r, 0, -1):
        acc = acc + (x[r + j:r + j + n] + x[r - j:r - j + n]) * w[r + j]
    return np.moveaxis(acc.astype(np.float32), 0, axis)


def _near_ties(rng, shape, w, r):
    """Columns along axis 0 whose sum at one position lies within a few
    2^-48 of the middle of two floats: the last tap's sample moves it there."""
    x = rng.uniform(0.25, 1, shape).astype(np.float32)
    x *= np.exp(rng.uniform(-4, 0, shape)).astype(np.float32)
    k = shape[0] // 2
    cols = x.reshape(shape[0], -1)
    cols[k + r] *= 2.0 ** -9
    cols = cols.astype(np.float64)

    def total():
        acc = cols[k] * w[r]
        for j in range(r, 0, -1):
            acc = acc + (cols[k + j] + cols[k - j]) * w[r + j]
        return acc
    for _ in range(3):
        s = total()
        f = s.astype(np.float32)
        up = np.nextafter(f, np.float32(np.inf))
        mid = (f.astype(np.float64) + up.astype(np.float64)) / 2
        off = rng.uniform(-4, 4, s.shape) * 2.0 ** -48 * s
        moved = cols[k + r] + (mid + off - s) / w[2 * r]
        cols[k + r] = np.maximum(moved, 0).astype(np.float32)
    return cols.astype(np.float32).reshape(shape)


def _filtered(x, w, r, shape):
    ref = x
    for axis in range(3):
        ref = _axis(ref, w, r, axis)
    return np.fft.ifftshift(ref)


@pytest.mark.parametrize("shape", [(48, 40, 48), (250, 24, 250),
                                   (500, 8, 500)])
def test_rounded_like_the_fp64_sum(cuda_ready, shape):
    rng = np.random.default_rng(shape[1])
    w, r = odt_apple._gauss_weights(shape)
    x = _near_ties(rng, shape, w, r)
    # FFT order in, FFT order out
    ft = np.fft.ifftshift(x).astype(np.complex64)
    got = odt_apple.envelope_gauss(ft, np.zeros(shape, dtype=bool))
    ref = _filtered(x, w, r, shape)
    assert got.dtype == np.float32
    bad = np.flatnonzero(got != ref)
    assert bad.size == 0, (bad.size, got.ravel()[bad[:3]], ref.ravel()[bad[:3]])


@pytest.mark.parametrize("kind", ["lobes", "tiny", "widest"])
def test_any_weights(cuda_ready, monkeypatch, kind):
    """Weights that scipy's Gaussian does not have: of both signs (sums that
    cancel), too small for floats, and the largest radius."""
    shape = (48, 40, 48)
    rng = np.random.default_rng(4)
    r = 64 if kind == "widest" else 5
    w = np.exp(-0.5 * (np.arange(-r, r + 1) / (0.3 * r)) ** 2)
    if kind == "lobes":
        w -= 0.35
    elif kind == "tiny":
        w *= 1e-40
    x = np.exp(rng.uniform(-3, 3, shape)).astype(np.float32)
    if kind == "tiny":
        x *= np.float32(1e37)
    monkeypatch.setattr(odt_apple, "_gauss_weights", lambda shape: (w, r))
    got = odt_apple.envelope_gauss(np.fft.ifftshift(x).astype(np.complex64),
                                   np.zeros(shape, dtype=bool))
    np.testing.assert_array_equal(got, _filtered(x, w, r, shape))
