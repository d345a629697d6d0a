"""GPU: more views than a grid's y and z extents hold (65535).  By linearity a
volume is the mean of the volumes of the two halves of its views, and a half's
gradient is twice the whole's.

Tolerance: both sides are FP32 sums over the same views; the parity tests'
1e-5 rel-L2 each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,ny,paired", [(1, 2, 0), (2, 2, 0), (1, 1, 0),
                                             (1, 2, 20000), (3, 2, 20000)])
def test_more_than_65535_views(cuda_ready, order, ny, paired):
    import torch
    from odtbrain_gb300._alg3d import Backprop3D
    half, nx = 35000, 4
    rng = np.random.default_rng(order)
    ang = rng.uniform(0, 2 * np.pi, (2, half))
    if paired:
        ang[:, paired // 2:paired] = ang[:, :paired // 2] + np.pi
    kw = dict(weight_angles=False, padding=(False, False), intp_order=order,
              device=cuda_ready)
    whole = Backprop3D((2 * half, ny, nx), ang.reshape(-1), 3.0, 1.333, **kw)
    halves = [Backprop3D((half, ny, nx), a, 3.0, 1.333, **kw) for a in ang]
    assert (whole._units is not None) == bool(paired)
    g = torch.Generator(device=cuda_ready)
    g.manual_seed(order)
    s = torch.randn((2 * half, ny, nx), generator=g, device=cuda_ready,
                    dtype=torch.complex64)
    v = whole(s)
    ref = (halves[0](s[:half]) + halves[1](s[half:])) / 2
    assert (v - ref).norm() <= 2e-5 * ref.norm()
    c = torch.randn(v.shape, generator=g, device=cuda_ready,
                    dtype=torch.complex64)
    grad, _ = whole.adjoint(s, c)
    ref = torch.cat([h.adjoint(t, c)[0] for h, t in
                     zip(halves, (s[:half], s[half:]))]) / 2
    assert (grad - ref).norm() <= 2e-5 * ref.norm()
