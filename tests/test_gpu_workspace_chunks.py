"""GPU: chunks of planes under workspace limits.  The chunk buffer may take a
quarter of the limit (64^2 views: planes of 66 x 128 complex64, 62 in 4 MiB, 48
in multiples of 16), and where not even one slab fits, chunks of two planes
remain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_chunks_under_limits(cuda_ready):
    import torch
    from odtbrain_gb300._alg3d import Backprop3D
    ang = np.linspace(0, np.pi, 60, endpoint=False)
    kw = dict(device=cuda_ready)
    free = Backprop3D((60, 64, 64), ang, 3.0, 1.333, **kw)
    lim = Backprop3D((60, 64, 64), ang, 3.0, 1.333,
                     workspace_limit=16 << 20, **kw)
    assert lim.plan.workspace_bytes <= 16 << 20
    # per batch of slabs: two launches per chunk, at most one short chunk, and
    # five others
    batches = -(-60 // lim.plan.angle_batch)
    assert lim.launches_per_call <= 2 * (-(-60 * 64 // 48) + batches) \
        + 5 * batches
    tight = Backprop3D((60, 64, 64), ang, 3.0, 1.333, workspace_limit=1 << 20,
                       **kw)
    assert tight.plan.angle_batch == 1
    assert tight.launches_per_call <= 60 * (64 + 5)
    g = torch.Generator(device=cuda_ready)
    g.manual_seed(1)
    s = torch.randn((60, 64, 64), generator=g, device=cuda_ready,
                    dtype=torch.complex64)
    ref = free(s)
    for rec in (lim, tight):
        assert (rec(s) - ref).norm() <= 2e-5 * ref.norm()
