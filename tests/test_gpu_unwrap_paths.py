"""Frames without residues are unwrapped by running sums, the others by the
spanning tree: both must give the oracle's tree bit by bit, also side by side
in one call and where FP32 estimates cannot decide (equal weights, steps of
exactly pi, phases far outside one turn)."""
import numpy as np
import pytest

from oracle import unwrap_oracle as uo

pytestmark = pytest.mark.gpu


def _frames(kind, H, W, rng):
    y, x = np.mgrid[:H, :W]
    ramp = 0.9 * x - 0.7 * y
    wrap = lambda p: np.angle(np.exp(1j * p))  # noqa: E731
    if kind == "smooth":  # no residues
        return wrap(ramp + 0.01 * rng.normal(size=(H, W)))
    if kind == "flat":  # equal weights: the lowest edge index is first
        return np.where((y > H // 2) & (x > W // 3), 0.25, 0.25 + 0 * ramp)
    if kind == "planes":  # exact ties off zero, whole turns in x
        return wrap(np.round(8 * ramp) / 8)
    if kind == "pi":  # steps of exactly +-pi and just beside it
        step = np.pi * (x % 2) - np.pi / 2
        return step * (1 + 1e-9 * rng.integers(-1, 2, W))
    if kind == "noise":  # residues
        return wrap(ramp + 1.5 * rng.normal(size=(H, W)))
    if kind == "far":  # beyond what the estimates cover
        return 40 * np.sin(ramp / 9) + 7.0 * (x > W // 2)
    raise ValueError(kind)


KINDS = ("smooth", "flat", "planes", "pi", "noise", "far")


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("H,W", [(1, 1), (1, 40), (40, 1), (2, 2), (3, 3),
                                 (8, 32), (9, 33), (7, 31), (16, 65),
                                 (300, 5), (70, 261)])
def test_both_paths_match_the_tree(cuda_ready, H, W, dtype):
    from odtbrain_gb300 import _prepare_sino as ps
    rng = np.random.default_rng(H * 1000 + W)
    w = np.array([_frames(k, H, W, rng) for k in KINDS]).astype(dtype)
    got = ps.unwrap_frames(w)
    for k, g, f in zip(KINDS, got, w):
        ref = uo.unwrap_2d(f, anchor="first_edge").astype(dtype)
        assert np.array_equal(g, ref), (k, np.argwhere(g != ref)[:3])


def test_nan_frame_leaves_the_others(cuda_ready):
    from odtbrain_gb300 import _prepare_sino as ps
    rng = np.random.default_rng(5)
    w = np.array([_frames(k, 20, 45, rng) for k in KINDS])
    clean = ps.unwrap_frames(w)
    v = w.copy()
    v[0, 7, 9] = np.nan
    v[3] = np.nan
    got = ps.unwrap_frames(v)
    for a in (1, 2, 4, 5):
        assert np.array_equal(got[a], clean[a])
    assert np.array_equal(np.isnan(got), np.isnan(v))


@pytest.mark.parametrize("low", [-13.0, -40.0, 21.0, -0.5])
def test_alignment_shift_rounds_like_fp64(cuda_ready, low):
    """float32 phases minus the FP64 shift, through FP32 pairs: the same
    rounding as the FP64 difference, zeros and cancelling sums included.
    Equal angles have no steps between them, so the shift is the minimum's
    whole turns, a float32 product."""
    from odtbrain_gb300 import _prepare_sino as ps
    rng = np.random.default_rng(11)
    base = (low + rng.gamma(2, 3, size=(40, 33))).astype(np.float32)
    turn = np.float32(2 * np.pi)
    base[0, :8] = [max(low, 0), 1e-30, turn, -turn, -3 * turn, 1e8, 0.5, 30]
    base[1] = np.float32(low)
    base[2] = np.linspace(0, 1e-6, 33)
    base = np.maximum(base, np.float32(low))
    w = np.repeat(base[None], 5, axis=0)
    got = w.copy()
    ps.align_unwrapped(got)
    q = np.float32(np.round(np.median(w - got) / (2 * np.pi)))
    ref = (w.astype(np.float64) - np.float64(q * turn)).astype(np.float32)
    assert abs(q) >= (low < -1 or low > 7)
    assert np.array_equal(got, ref)
    assert np.array_equal(np.signbit(got), np.signbit(ref))


def test_capture_and_replay(cuda_ready):
    """The whole preparation in a CUDA graph, replayed on other data (frames
    with residues where the captured ones had none)."""
    import torch
    from odtbrain_gb300 import _prepare_sino as ps
    rng = np.random.default_rng(21)
    field = [torch.tensor(np.exp(1j * np.array(
        [_frames(k, 40, 70, rng) for k in kinds])), device="cuda")
        for kinds in (("smooth",) * 4, ("noise", "smooth", "noise", "noise"))]
    run = ps.SinogramPrep((4, 40, 70), kind="rytov", single=False)
    want = [run(f).clone() for f in field]
    static, out = field[0].clone(), torch.empty_like(field[0])
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        run(static, out=out, check=False)
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(static, out=out, check=False)
    for f, ref in ((field[1], want[1]), (field[0], want[0])):
        static.copy_(f)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, ref)
