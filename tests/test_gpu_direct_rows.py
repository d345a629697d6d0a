"""GPU: unpadded detector heights without a radix-8 transform, whose rows are
direct transforms of interleaved lines: one and several slots per thread, a
slot's last position, fewer rows than a CTA takes, power-of-two and direct
columns, both geometries and every prefilter against the FP64 oracle (the parity
tests' 1e-5 rel-L2)."""
import numpy as np
import pytest

from oracle import odt_oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(5, 64), (33, 64), (63, 30), (65, 18), (130, 17), (66, 128), (2, 21)]


@pytest.mark.parametrize("ny,nx", SIZES)
@pytest.mark.parametrize("kind,order", [("y", 1), ("y", 2), ("y", 5),
                                        ("tilted", 0), ("tilted", 3),
                                        ("tilted", 4), ("pairs", 3)])
def test_unpadded_heights(cuda_ready, ny, nx, kind, order):
    import odtbrain_gb300 as odt
    if kind == "tilted" and order >= 4 and ny < 4:
        pytest.skip("lines of at least 4 samples")
    rng = np.random.default_rng(ny + nx + order)
    A = 6
    sino = np.exp(1j * rng.normal(0, .4, (A, ny, nx))) - 1
    ang = (np.linspace(0, 2 * np.pi, A, endpoint=False) if kind == "pairs"
           else np.sort(rng.uniform(0, 2 * np.pi, A)))
    kw = dict(padding=(False, False), intp_order=order, lD=1.2)
    if kind == "tilted":
        kw["tilted_axis"] = [0.05, 1.0, 0.2]
        ref = O.backpropagate_3d_tilted(sino, ang, 2.5, 1.333, **kw)
        got = odt.backpropagate_3d_tilted(sino, ang, 2.5, 1.333, **kw)
    else:
        ref = O.backpropagate_3d(sino, ang, 2.5, 1.333, **kw)
        got = odt.backpropagate_3d(sino, ang, 2.5, 1.333, **kw)
    assert np.linalg.norm(ref) > 0
    assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)
