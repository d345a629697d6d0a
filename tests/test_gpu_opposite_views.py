"""GPU: reconstructions and gradients over units of opposite views against
the general path (one angle per slab) and the FP64 oracle.

Tolerance: both paths compute in FP32 and differ by the order of their
roundings, so results agree within twice the parity tests' 1e-5 rel-L2 bound
against the oracle; measured errors are a few 1e-7."""
import numpy as np
import pytest

from oracle import odt_oracle as O
from sino_gen import ellipsoid_phantom_sinogram

pytestmark = pytest.mark.gpu
REL = 2e-5


def _close(got, ref, what, rel=REL):
    got, ref = np.asarray(got), np.asarray(ref)
    err = np.linalg.norm(got - ref) / np.linalg.norm(ref)
    assert err <= rel, (what, err)


def _angles(A, singles=0):
    """A views of a full circle in pairs, the last ones without partner."""
    ang = np.linspace(0, 2 * np.pi, A - singles, endpoint=False)
    return np.concatenate([ang, 0.013 + 0.31 * np.arange(singles)])


def _alone(rec):
    """`rec` over single angles."""
    import torch
    rec._units = None
    rec.workspace = torch.empty(rec.plan.workspace_bytes, dtype=torch.uint8,
                                device=rec.device)
    return rec


# (A, singles, ny, nx, order, padval, onlyreal, workspace limit): every line
# type of the two FFT axes (64..512 and, unpadded, the direct DFT), the
# half-crop kernels, odd and even left pads, one and two poles, one and
# several batches
CASES = [
    (8, 0, 16, 22, 2, "edge", False, None),
    (9, 1, 20, 37, 3, 0.3 - 0.1j, False, None),
    (12, 4, 64, 64, 2, "edge", True, None),
    (8, 0, 128, 128, 2, "edge", False, None),
    (8, 2, 70, 150, 5, "edge", False, None),
    (8, 0, 256, 256, 2, "edge", False, 1 << 30),
    (10, 2, 33, 40, 1, 0, False, None),
    (12, 2, 48, 48, 2, "edge", False, 8 << 20),
    (8, 0, 17, 21, 4, None, False, None),
    (10, 2, 1, 50, 2, "edge", False, None),
    (40, 4, 1, 64, 3, None, False, 256 << 10),
]


@pytest.mark.parametrize("case", CASES)
def test_pairs_match_single_angles(cuda_ready, case):
    import torch
    from odtbrain_gb300._alg3d import Backprop3D
    A, singles, ny, nx, order, padval, onlyreal, limit = case
    ang = _angles(A, singles)
    rng = np.random.default_rng(A + nx)
    sino = np.exp(1j * rng.normal(0, .4, (A, ny, nx))) - 1
    pad = padval is not None
    kw = dict(padding=(pad, pad), padval=padval if pad else "edge",
              intp_order=order, onlyreal=onlyreal)
    d = torch.from_numpy(sino.astype(np.complex64)).to(cuda_ready)
    recs = [Backprop3D(sino.shape, ang, 2.3, 1.333, lD=1.5,
                       device=cuda_ready, workspace_limit=limit, **kw)
            for _ in range(2)]
    assert recs[0]._units.num == (A - singles) // 2 + singles
    pairs = recs[0](d)
    single = _alone(recs[1])(d)
    _close(pairs.cpu(), single.cpu(), "pairs / single angles")
    if A * ny * nx * nx < 2e7:
        ref = O.backpropagate_3d(sino.astype(np.complex64), ang, 2.3, 1.333,
                                 lD=1.5, **kw)
        _close(pairs.cpu(), ref, "pairs / oracle", 1e-5)


@pytest.mark.parametrize("A,singles,ny,nx,order", [
    (12, 2, 24, 20, 2), (8, 0, 1, 30, 2), (9, 1, 64, 64, 3),
    (8, 0, 128, 128, 2), (6, 2, 30, 21, 1)])
def test_pair_gains_and_gradients(cuda_ready, A, singles, ny, nx, order):
    """Gain maps without any symmetry: the mirrored spectrum takes its own
    view's gains at the mirrored frequency, and the gradients go back there."""
    import torch
    from odtbrain_gb300._alg3d import Backprop3D
    ang = _angles(A, singles)
    g = torch.Generator(device=cuda_ready)
    g.manual_seed(nx)

    def rand(shape, dtype=torch.complex64):
        return torch.randn(shape, generator=g, device=cuda_ready, dtype=dtype)
    sino = rand((A, ny, nx))
    recs = [Backprop3D((A, ny, nx), ang, 3.0, 1.333, intp_order=order,
                       device=cuda_ready) for _ in range(2)]
    assert recs[0]._units.num < A
    _alone(recs[1])
    shape = recs[0].gain_shape()
    gain = rand(shape, torch.float32)
    again = rand((A,) + shape)
    cot = rand(recs[0].volume_shape())
    vols, grads = [], []
    for rec in recs:
        vols.append(rec.forward_gain(sino, gain=gain, angle_gain=again))
        grads.append(rec.adjoint(sino, cot, gain=gain, need_gain=True,
                                 angle_gain=again, need_angle_gain=True))
    _close(vols[0].cpu(), vols[1].cpu(), "volume")
    for name, x, y in zip(("sino", "gain", "angle gain"), *grads):
        _close(x.cpu(), y.cpu(), name)


@pytest.mark.parametrize("A,singles,n,padval", [(10, 0, 22, 0),
                                                (9, 1, 64, None),
                                                (12, 0, 300, 0)])
def test_pairs_2d(cuda_ready, A, singles, n, padval):
    import torch
    from odtbrain_gb300._alg2d import Backprop2D
    ang = _angles(A, singles)
    rng = np.random.default_rng(n)
    sino = (np.exp(1j * rng.normal(0, .4, (A, n))) - 1).astype(np.complex64)
    rec = Backprop2D((A, n), ang, 3.0, 1.333, padval=padval,
                     device=cuda_ready)
    assert rec._units.num == (A - singles) // 2 + singles
    got = rec(torch.from_numpy(sino).to(cuda_ready)).cpu()
    ref = O.backpropagate_2d(sino, ang, 3.0, 1.333, padval=padval)
    _close(got, ref, "2d", 1e-5)


def test_pairs_refused(cuda_ready):
    """A limit that holds no unit, more units than angles, and the tilted
    geometry are refused, and the instance runs single angles instead."""
    from odtbrain_gb300._alg3d import Backprop3D
    ang = _angles(8)
    tight = Backprop3D((8, 32, 32), ang, 3.0, 1.333, device=cuda_ready,
                       workspace_limit=1 << 10)
    assert tight._units is None and tight.plan.workspace_bytes > 1 << 10
    tilted = Backprop3D((8, 32, 32), ang, 3.0, 1.333, device=cuda_ready,
                        tilted_axis=(0.1, 1, 0.2))
    assert tilted.plan.pair_workspace_bytes(4) is None
    rec = Backprop3D((8, 32, 32), ang, 3.0, 1.333, device=cuda_ready)
    with pytest.raises(ValueError):
        rec.plan.pair_workspace_bytes(9)
