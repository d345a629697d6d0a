"""GPU: sinogram preparations of frames with residues (whose later tree rounds
are one cooperative launch as large as the device) on two streams at once, from
two host threads, and beside a long kernel of another stream: bit for bit what
each gives alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fields(device):
    import torch
    rng = np.random.default_rng(9)
    y, x = np.mgrid[:90, :131]
    return [torch.tensor(np.exp(1j * (0.9 * x - 0.7 * y
                                      + s * rng.normal(size=(12, 90, 131)))),
                         device=device) for s in (1.5, 0.8)]


def test_two_streams_and_threads(cuda_ready):
    import torch
    from odtbrain_gb300 import _prepare_sino as ps
    fields = _fields(cuda_ready)
    preps = [ps.SinogramPrep(f.shape, single=False) for f in fields]
    want = [p(f).clone() for p, f in zip(preps, fields)]
    streams = [torch.cuda.Stream() for _ in fields]
    torch.cuda.synchronize()
    got, failed = [[], []], []

    def work(k):
        try:
            with torch.cuda.stream(streams[k]):
                got[k] = [preps[k](fields[k], check=False)
                          for _ in range(20)]
                preps[k](fields[k])
        except Exception as e:  # a device check that tripped
            failed.append(e)
    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed
    for k in (0, 1):
        assert len(got[k]) == 20
        for g in got[k]:
            assert torch.equal(g, want[k])


def test_beside_a_long_kernel(cuda_ready):
    import torch
    from odtbrain_gb300 import _prepare_sino as ps
    field = _fields(cuda_ready)[0]
    prep = ps.SinogramPrep(field.shape, single=False)
    want = prep(field).clone()
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(other):
        torch.cuda._sleep(1 << 30)  # about half a second on one SM
    got = prep(field)
    assert torch.equal(got, want)
    torch.cuda.synchronize()
