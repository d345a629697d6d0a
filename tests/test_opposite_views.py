"""Opposite views that share a slab (``_geometry.opposite_units``, CPU): every
angle appears once, paired rotations are half a turn apart, and both views of
a unit make the same in/out decision for every output, by the FP64 comparison
scipy makes."""
import numpy as np
import pytest

from odtbrain_gb300 import _geometry as geom


def _inside(g, n):
    """scipy's decision for every output of the n x n plane."""
    oz, ox = np.arange(n).reshape(-1, 1), np.arange(n).reshape(1, -1)
    cz = (g[4] + g[0] * oz) + g[1] * ox
    cx = (g[5] + g[2] * oz) + g[3] * ox
    return (cz >= 0) & (cz <= n - 1) & (cx >= 0) & (cx <= n - 1)


def _angle_sets():
    rng = np.random.default_rng(3)
    half = rng.uniform(0, np.pi, 9)
    yield "full circle", np.linspace(0, 2 * np.pi, 40, endpoint=False), 20
    # the quarter turns of this set are exact for one view of the pair only
    yield "200 views", np.linspace(0, 2 * np.pi, 200, endpoint=False), None
    yield "odd count", np.linspace(0, 2 * np.pi, 9, endpoint=False), 9
    yield "wedge", np.linspace(0, 2.1, 12), 12
    yield "one view", np.array([0.3]), 1
    # duplicates: each view is used once
    yield "closed circle", np.linspace(0, 2 * np.pi, 9), 5
    yield "pairs and singles", rng.permutation(
        np.concatenate([half, half[:5] + np.pi, [7.0]])), 10
    # quarter turns that are not exact: some outputs lie on the boundary for
    # one view only
    yield "near quarter turns", np.array(
        [0.5 * np.pi + 1e-15, 1.5 * np.pi - 1e-15, 0.2, 0.2 + np.pi]), None


@pytest.mark.parametrize("n", [16, 33])
@pytest.mark.parametrize("kind", ["y", "2d"])
def test_units_decide_alike(n, kind):
    for name, ang, num in _angle_sets():
        geo = (geom.rotation_y_geometry(ang, n, n) if kind == "y"
               else geom.rotation_2d_geometry(ang, n))
        units = geom.opposite_units(geo, n)
        assert units.dtype == np.int32 and units.shape[1] == 2, name
        assert sorted(units[units >= 0]) == list(range(len(ang))), name
        assert (units[:, 0] >= 0).all(), name
        if num is not None:
            assert len(units) == num, (name, len(units))
        for a, b in units[units[:, 1] >= 0]:
            np.testing.assert_allclose(geo[a, :4], -geo[b, :4], atol=1e-12)
            # the shared slab is resampled with the first view's geometry
            np.testing.assert_array_equal(_inside(geo[a], n),
                                          _inside(geo[b], n), err_msg=name)
