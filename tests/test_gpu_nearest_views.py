"""GPU: nearest-neighbour resampling (order 0) of full circles.  Every view
takes its own nearest sample: views phi and phi + pi resample with coordinates
c and n-1-c, whose halves round to different samples, so they cannot share a
slab.  The angle sets hold views whose coordinates are half integers: multiples
of 30 degrees at odd widths, of 45 degrees at even widths.

Tolerance: the parity tests' 1e-5 rel-L2 against the FP64 oracle; one sample
beside the right one in 1e5 outputs breaks it."""
import ctypes

import numpy as np
import pytest

from oracle import odt_oracle as O

pytestmark = pytest.mark.gpu
REL = 1e-5

CASES = [(12, 9, 33, "edge"), (12, 1, 33, None), (40, 6, 64, "edge"),
         (40, 1, 64, 0), (60, 3, 65, None), (8, 20, 64, None)]


def _case(A, ny, nx, padval):
    ang = np.linspace(0, 2 * np.pi, A, endpoint=False)
    rng = np.random.default_rng(A + nx)
    sino = (np.exp(1j * rng.normal(0, .4, (A, ny, nx))) - 1) \
        .astype(np.complex64)
    pad = padval is not None
    kw = dict(padding=(pad, pad), padval=padval if pad else "edge",
              intp_order=0)
    return ang, sino, kw


@pytest.mark.parametrize("case", CASES)
def test_every_view_takes_its_own_sample(cuda_ready, case):
    import odtbrain_gb300 as odt
    ang, sino, kw = _case(*case)
    ref = O.backpropagate_3d(sino, ang, 2.3, 1.333, lD=1.5, **kw)
    got = odt.backpropagate_3d(sino, ang, 2.3, 1.333, lD=1.5, **kw)
    assert np.linalg.norm(got - ref) <= REL * np.linalg.norm(ref)


@pytest.mark.parametrize("case", CASES)
def test_gradient_goes_to_its_own_sample(cuda_ready, case):
    """<oracle(s), c> = <s, adjoint(c)> for c unit Gaussian: the left side's
    share of an error of rel-L2 REL in the volume is a Gaussian of that norm,
    so five of them bound it."""
    import torch
    from odtbrain_gb300._alg3d import Backprop3D
    ang, sino, kw = _case(*case)
    ref = O.backpropagate_3d(sino, ang, 2.3, 1.333, **kw)
    rec = Backprop3D(sino.shape, ang, 2.3, 1.333, device=cuda_ready, **kw)
    rng = np.random.default_rng(1)
    d = torch.from_numpy(sino).to(cuda_ready)
    for _ in range(4):
        c = (rng.standard_normal(ref.shape) + 1j
             * rng.standard_normal(ref.shape)).astype(np.complex64)
        grad, _ = rec.adjoint(d, torch.from_numpy(c).to(cuda_ready))
        lhs = np.vdot(c.astype(complex), ref)
        rhs = np.vdot(grad.cpu().numpy().astype(complex), sino)
        assert abs(lhs - rhs) <= 5 * REL * np.linalg.norm(ref), (lhs, rhs)


def test_pairs_refused(cuda_ready):
    """By the instance and by the C entries, with the units of a plan that
    takes them."""
    import torch
    from odtbrain_gb300 import _native
    from odtbrain_gb300._alg3d import Backprop3D
    ang = np.linspace(0, 2 * np.pi, 8, endpoint=False)
    rec, paired = (Backprop3D((8, 20, 32), ang, 3.0, 1.333, intp_order=order,
                              device=cuda_ready) for order in (0, 1))
    assert paired._units.num == 4
    assert rec._units is None
    assert rec.plan.pair_workspace_bytes(4) is None
    sino = torch.ones(rec.shape, dtype=torch.complex64, device=cuda_ready)
    vol = torch.empty(rec.volume_shape(), dtype=torch.complex64,
                      device=cuda_ready)
    room = paired.plan.pair_workspace_bytes(4)[1]
    ws = torch.empty(room, dtype=torch.uint8, device=cuda_ready)
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in (sino, vol, ws)]
    L, units = _native.lib(), ctypes.byref(paired._units.struct)
    assert L.odt_bpp3d_execute_pairs(
        rec.plan._h, units, ptr[0], None, None, None, ptr[1], ptr[2], None,
        None) == _native.ODT_ERR_UNSUPPORTED
    assert L.odt_bpp3d_adjoint_pairs(
        rec.plan._h, units, ptr[0], None, None, None, ptr[1], ptr[0], None,
        None, ptr[2], None) == _native.ODT_ERR_UNSUPPORTED
