"""Missing-apple-core correction at sizes where a CTA of the line transforms
takes several groups of lines, with a remainder: power-of-two and other
lengths on each axis, the loop ended by the iteration limit
and by the stopping test."""
import numpy as np
import pytest

from oracle import apple_oracle as ao

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,kw", [
    ((64, 128, 64), {"max_iter": 3, "min_diff": 0.0}),
    ((128, 64, 128), {"method": "other", "max_iter": 2, "min_diff": 0.0}),
    ((64, 70, 64), {"max_iter": 1, "enforce_envelope": 0}),
    ((90, 64, 90), {"max_iter": 30, "min_diff": 0.05}),
    ((256, 21, 256), {"max_iter": 2, "min_diff": 0.0}),
])
def test_lines_in_turn(cuda_ready, shape, kw):
    import odtbrain_gb300 as odt
    rng = np.random.default_rng(sum(shape))
    z, y, x = np.meshgrid(*[np.arange(s) - s / 2 for s in shape],
                          indexing="ij")
    f = np.exp(-(x ** 2 + y ** 2 + z ** 2) / (0.08 * shape[0] ** 2)) \
        + 0.05 * rng.standard_normal(shape)
    kw = dict(res=3.0, nm=1.333, **kw)
    ref = ao.correct(f, **kw)
    got = odt.apple.correct(f, **kw)
    # the oracle's own change for a 1e-7 relative change of its input, times
    # four, and no less than FP32 transforms of this size give
    other = ao.correct(f * (1 + 1e-7), **kw)
    scale = np.abs(ref).max()
    tol = max(2e-5, 4 * np.abs(other - ref).max() / scale)
    assert np.abs(got - ref).max() <= tol * scale


@pytest.mark.parametrize("scale", [1e-30, 1e-18, 1.0, 1e18, 1e30])
def test_envelope_over_the_float_range(cuda_ready, scale):
    """The envelope's Gaussian sums in float pairs hand over to FP64 where the
    pairs are not exact: magnitudes near both ends of float32."""
    import odtbrain_gb300 as odt
    rng = np.random.default_rng(3)
    shape = (36, 40, 36)
    ft = ((rng.standard_normal(shape) + 1j * rng.standard_normal(shape))
          * np.exp(rng.uniform(-3, 3, shape)) * scale).astype(np.complex64)
    core = odt.apple.apple_core_3d(shape, 3.0, 1.333)
    ref = ao.envelope_gauss(ft.copy(), core)
    got = np.asarray(odt.apple.envelope_gauss(ft.copy(), core))
    assert np.isfinite(ref).all() and ref.max() > 0
    # one rounding of the magnitudes and of each axis's float32 result
    assert np.abs(got - ref).max() <= 2e-6 * ref.max()
