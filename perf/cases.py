"""The calls a tomography user makes, as cases that can be timed.

A case goes through the package's public entry points: the drop-in
reconstruction functions (``backpropagate_3d``, ``backpropagate_3d_tilted``),
the prepared 2D reconstruction (``Backprop2D``), the differentiable
reconstruction, one training step of the learned filter gain, and the steps
either side of a reconstruction (``sinogram_as_rytov``, ``apple.correct``,
``odt_to_ri``).  Sinograms are those of seeded random ellipsoid phantoms with
log-amplitude noise, resident on the GPU as they are in a pipeline that goes
on from ``sinogram_as_rytov``.  Reconstructions are asked for in single
precision (``dtype=float32``), the precision the kernels compute in.

``exact`` restates every path in 64 bits with plain torch and numpy.
"""
import math

import numpy as np
import torch

import odtbrain_gb300 as odt
from odtbrain_gb300 import phantoms
from odtbrain_gb300._alg2d import Backprop2D
from odtbrain_gb300._alg3d import Backprop3D
from odtbrain_gb300.autograd import backpropagate_3d_autograd
from odtbrain_gb300.learned import GainMLP, LearnedFilter, wedge_angles

RES, NM = 3.0, 1.333          # pixels per wavelength, medium index
TILT = 0.2                    # of the rotation axis, from y toward z (rad)
C128 = torch.complex128
F64 = torch.float64


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest reconstruction: one line of a small detector, where
        # launches and host work count
        dict(name="bpp2d_128", kind="2d", A=60, n=128, pad="ramp"),
        # a slice from a full-size detector line
        dict(name="bpp2d_512", kind="2d", A=400, n=512, pad="ramp"),
        # a quick look at a cropped cell: 60 views of 64^2, double-precision
        # data as NumPy pipelines hand it over
        dict(name="bpp3d_64", kind="3d", A=60, ny=64, nx=64, order=2,
             pad="edge", onlyreal=False, double=True),
        # a detector region cut to the sample: rectangular, an odd number of
        # views, cubic splines, padded down to the medium's zero phase, the
        # real part only
        dict(name="bpp3d_ragged", kind="3d", A=121, ny=101, nx=150, order=3,
             pad="ramp", onlyreal=True, double=False),
        # the standard reconstruction: 200 views of 256^2
        dict(name="bpp3d_256", kind="3d", A=200, ny=256, nx=256, order=2,
             pad="edge", onlyreal=False, double=False),
        # a tilted rotation axis on a small rectangular region, the cheapest
        # (linear) interpolation
        dict(name="tilted_ragged", kind="tilted", A=75, ny=90, nx=111,
             order=1, pad="edge", onlyreal=False),
        # a tilted rotation axis at full size: 220 views of 200^2
        dict(name="tilted_200", kind="tilted", A=220, ny=200, nx=200,
             order=2, pad="edge", onlyreal=False),
        # iterative reconstruction: forward and gradients with respect to
        # the sinogram and the filter gain
        dict(name="vjp_128", kind="vjp", A=90, n=128),
        # training of the learned filter gain on a 120 degree wedge: network
        # forward, reconstruction, adjoint, network backward
        dict(name="train_128", kind="train", A=40, n=128),
        # the recorded fields to a Rytov sinogram (per-frame unwrapping)
        dict(name="rytov_256", kind="rytov", A=200, ny=256, nx=256),
        # the missing-apple-core correction of a reconstruction
        dict(name="apple_256", kind="apple", n=256),
        # the object function to refractive index
        dict(name="ri_256", kind="ri", n=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["2d", "3d", "3d", "3d", "tilted", "tilted", "vjp",
                       "train", "rytov", "apple", "ri"])
    pad = rng.choice(["edge", "edge", "ramp"])
    if kind == "2d":
        return dict(kind=kind, A=_log_int(rng, 20, 400),
                    n=_log_int(rng, 64, 512), pad=pad)
    if kind == "3d":
        return dict(kind=kind, A=_log_int(rng, 20, 200),
                    ny=_log_int(rng, 32, 256), nx=_log_int(rng, 32, 256),
                    order=rng.choice([1, 2, 2, 2, 3]), pad=pad,
                    onlyreal=rng.random() < 0.25, double=rng.random() < 0.25)
    if kind == "tilted":
        return dict(kind=kind, A=_log_int(rng, 20, 220),
                    ny=_log_int(rng, 32, 200), nx=_log_int(rng, 32, 200),
                    order=rng.choice([1, 2, 2, 3]), pad=pad,
                    onlyreal=rng.random() < 0.25)
    if kind == "vjp":
        return dict(kind=kind, A=_log_int(rng, 20, 90),
                    n=_log_int(rng, 32, 128))
    if kind == "train":
        return dict(kind=kind, A=_log_int(rng, 20, 60),
                    n=_log_int(rng, 48, 128))
    if kind == "rytov":
        return dict(kind=kind, A=_log_int(rng, 20, 200),
                    ny=_log_int(rng, 32, 256), nx=_log_int(rng, 32, 256))
    if kind == "apple":
        return dict(kind=kind, n=_log_int(rng, 32, 200))
    return dict(kind=kind, n=_log_int(rng, 32, 256))


# ------------------------------------------------------------------ inputs
def _circle(A):
    return np.linspace(0, 2 * np.pi, A, endpoint=False)


def _phantom(rng, n):
    """3-8 ellipsoids inside the inscribed sphere of n voxels."""
    return phantoms.random_ellipsoids(rng, n, (3, 8), (n / 32, n / 4.5))


def _sinogram(angles, ny, nx, seed, amp=0.01):
    """Complex64 Rytov sinogram (A, ny, nx) of a seeded phantom; the phase
    alone is its imaginary part without noise."""
    rng = np.random.default_rng(seed)
    ells = _phantom(rng, min(nx, ny) if ny > 1 else nx)
    return phantoms.project([ells], angles, nx, RES, NM, amp, seed=seed,
                            device="cuda", ny=ny)[0]


def _normal(seed, shape, dtype=torch.complex64):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return torch.randn(shape, generator=g, device="cuda", dtype=dtype)


def _uniform(seed, shape):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return torch.rand(shape, generator=g, device="cuda")


def _tilt_axis():
    return (0.0, math.cos(TILT), math.sin(TILT))


def _apple_core(n):
    """The missing apple core in FFT order (odtbrain/apple.py:8-53), axis 1
    the axis of symmetry."""
    km = 2 * np.pi * NM / RES
    f = np.fft.fftfreq(n)
    fx, fy, fz = f.reshape(-1, 1, 1), f.reshape(1, -1, 1), f.reshape(1, 1, -1)
    ky = 2 * np.pi * fy
    kxz = 2 * np.pi * np.sqrt(fx ** 2 + fz ** 2)
    kr = 2 * np.pi * np.sqrt(fx ** 2 + fy ** 2 + fz ** 2)
    root = 2 * km * kxz - kxz ** 2
    root[root < 0] = 0
    core = np.abs(ky) > np.sqrt(root)
    core &= ~(kr > np.sqrt(2) * km)
    return core


def _object_function(n, seed):
    """Complex64 object function of a seeded phantom: km^2 ((n/nm)^2 - 1)
    inside its ellipsoids."""
    rng = np.random.default_rng(seed)
    km2 = (2 * np.pi * NM / RES) ** 2
    x = torch.arange(n, device="cuda", dtype=torch.float32) - (n - 1) / 2
    f = torch.zeros((n, n, n), device="cuda")
    for c, s, R, idx in _phantom(rng, n):
        Q = torch.tensor(R @ np.diag(1 / np.asarray(s) ** 2) @ R.T,
                         dtype=torch.float32)
        dx = (x - float(c[0])).view(1, 1, n)
        dy = (x - float(c[1])).view(1, n, 1)
        dz = (x - float(c[2])).view(n, 1, 1)
        q = (Q[0, 0] * dx * dx + Q[1, 1] * dy * dy + Q[2, 2] * dz * dz
             + 2 * (Q[0, 1] * dx * dy + Q[0, 2] * dx * dz
                    + Q[1, 2] * dy * dz))
        f[q <= 1] = km2 * ((idx / NM) ** 2 - 1)
    noise = _normal(seed, (n, n, n)) * 0.002
    return noise + f


def _cored_volume(n, seed):
    """A reconstruction's object function: the phantom's with the spectrum
    of the missing apple core taken out."""
    f = torch.fft.fftn(_object_function(n, seed))
    f[torch.from_numpy(_apple_core(n)).to("cuda")] = 0
    return torch.fft.ifftn(f)


def _padval(case):
    return "edge" if case["pad"] == "edge" else 0


def prepare(case, seed):
    kind = case["kind"]
    if kind == "2d":
        ang = _circle(case["A"])
        sino = _sinogram(ang, 1, case["n"], seed)[:, 0, :].contiguous()
        rec = Backprop2D((case["A"], case["n"]), ang, RES, NM,
                         padval=None if case["pad"] == "edge" else 0)
        return dict(case=case, sino=sino, rec=rec)
    if kind in ("3d", "tilted"):
        ang = _circle(case["A"])
        sino = _sinogram(ang, case["ny"], case["nx"], seed)
        if case.get("double"):
            sino = sino.to(C128)
        return dict(case=case, sino=sino, angles=ang)
    if kind == "vjp":
        n, A = case["n"], case["A"]
        rec = Backprop3D((A, n, n), _circle(A), RES, NM)
        return dict(case=case, rec=rec, angles=_circle(A),
                    sino=_sinogram(_circle(A), n, n, seed),
                    gain=0.5 + _uniform(seed + 1, rec.gain_shape()),
                    grad=_normal(seed + 2, (n, n, n)))
    if kind == "train":
        n, A = case["n"], case["A"]
        rec = Backprop3D((A, n, n), wedge_angles(A), RES, NM)
        # the network a few steps into its training: the last layer has left
        # zero
        mlp = GainMLP(device="cuda", seed=seed)
        state = mlp.state()
        state["W4"] = 0.1 * np.random.default_rng(seed).normal(
            size=state["W4"].shape)
        mlp.load_state(state)
        return dict(case=case, rec=rec, mlp=mlp,
                    filt=LearnedFilter(rec, mlp),
                    sino=_sinogram(wedge_angles(A), n, n, seed),
                    target=_cored_volume(n, seed))
    if kind == "rytov":
        sino = _sinogram(_circle(case["A"]), case["ny"], case["nx"], seed)
        return dict(case=case, field=torch.exp(sino))
    if kind == "apple":
        return dict(case=case, f=_cored_volume(case["n"], seed))
    return dict(case=case, f=_object_function(case["n"], seed))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "2d":
        return state["rec"](state["sino"])
    if kind == "3d":
        return odt.backpropagate_3d(
            state["sino"], state["angles"], RES, NM, padval=_padval(case),
            intp_order=case["order"], onlyreal=case["onlyreal"],
            dtype=np.float32)
    if kind == "tilted":
        return odt.backpropagate_3d_tilted(
            state["sino"], state["angles"], RES, NM,
            tilted_axis=_tilt_axis(), padval=_padval(case),
            intp_order=case["order"], onlyreal=case["onlyreal"],
            dtype=np.float32)
    if kind == "vjp":
        sino = state["sino"].detach().requires_grad_()
        gain = state["gain"].detach().requires_grad_()
        vol = backpropagate_3d_autograd(sino, state["angles"], RES, NM,
                                        gain=gain, plan=state["rec"])
        gs, gg = torch.autograd.grad(vol, (sino, gain), state["grad"])
        return dict(volume=vol.detach(), sino_grad=gs, gain_grad=gg)
    if kind == "train":
        rec, mlp, filt = state["rec"], state["mlp"], state["filt"]
        mlp.bump()  # the optimiser has changed the weights
        gain = filt.gains()
        vol = rec.forward_gain(state["sino"], angle_gain=gain)
        tgt = state["target"]
        diff = vol - tgt
        nt = torch.linalg.vector_norm(tgt) ** 2
        loss = torch.linalg.vector_norm(diff) ** 2 / nt
        cot = (diff * (2.0 / nt)).to(torch.complex64)
        _s, _g, dgain = rec.adjoint(state["sino"], cot, angle_gain=gain,
                                    need_sino=False, need_angle_gain=True)
        grads = mlp.grads(filt.feat, dgain, positions=filt.positions)
        return dict(volume=vol, loss=loss, gain_grad=dgain, **grads)
    if kind == "rytov":
        return odt.sinogram_as_rytov(state["field"])
    if kind == "apple":
        return odt.apple.correct(state["f"], RES, NM)
    return odt.odt_to_ri(state["f"], RES, NM)


# ------------------------------------------------------------------ floors
def _pow2(v):
    return max(64, 2 ** math.ceil(math.log2(v)))


def _filter_flops(A, lny, lnx, pny, pnx, km):
    """Per angle the forward 2D transform and, per plane, the propagator
    multiply and the cropped backward 2D transform of the spectrum inside
    |k| < km (5 N log2 N per complex transform of N)."""
    cols = min(pnx, pnx * km / np.pi)
    inside = np.pi * km ** 2 / (4 * np.pi ** 2) * pny * pnx
    fwd = 5 * pny * pnx * math.log2(max(2, pny * pnx))
    plane = (6 * inside + cols * 5 * pny * math.log2(max(2, pny))
             + lny * 5 * pnx * math.log2(max(2, pnx)))
    return A * (fwd + lnx * plane)


def work(case):
    """Compulsory bytes: every input read and every output written once."""
    kind = case["kind"]
    km = 2 * np.pi * NM / RES
    if kind == "2d":
        A, n = case["A"], case["n"]
        return dict(bytes=8 * (A * n + n * n),
                    flops=_filter_flops(A, 1, n, 1, _pow2(2.1 * n), km)
                    + A * n * n * 2 * 2 * 16)
    if kind in ("3d", "tilted"):
        A, ny, nx, o = case["A"], case["ny"], case["nx"], case["order"]
        taps = (o + 1) ** (2 if kind == "3d" else 3)
        comp = 1 if case["onlyreal"] else 2
        return dict(bytes=(16 if case.get("double") else 8) * A * ny * nx
                    + 4 * comp * nx * ny * nx,
                    flops=_filter_flops(A, ny, nx, _pow2(1.75 * ny),
                                        _pow2(1.75 * nx), km)
                    + A * nx * ny * nx * taps * 2 * comp)
    if kind in ("vjp", "train"):
        A, n = case["A"], case["n"]
        p = _pow2(1.75 * n)
        fl = 2 * (_filter_flops(A, n, n, p, p, km) + A * n ** 3 * 36)
        if kind == "vjp":
            return dict(bytes=2 * 8 * A * n * n + 2 * 8 * n ** 3
                        + 2 * 4 * p * p, flops=fl)
        mlp = 2 * (4 * 64 + 2 * 64 * 64 + 64 * 2)
        pts = A * np.pi * km ** 2 / (4 * np.pi ** 2) * p * p
        return dict(bytes=8 * A * n * n + 2 * 8 * n ** 3,
                    flops=fl + pts * 4 * mlp)
    if kind == "rytov":
        m = case["A"] * case["ny"] * case["nx"]
        return dict(bytes=16 * m, flops=100 * m)
    if kind == "apple":
        m = case["n"] ** 3
        # some thirty iterations of a forward and a backward transform
        return dict(bytes=16 * m,
                    flops=30 * 2 * 5 * m * math.log2(max(2, m)))
    m = case["n"] ** 3
    return dict(bytes=16 * m, flops=30 * m)


# ------------------------------------------------- the same paths in 64 bits
def _angle_weights(angles):
    """odtbrain/util.py:4-67."""
    flat = (angles - angles.min()) % np.pi
    unq, back, cnt = np.unique(flat, return_inverse=True, return_counts=True)
    gap = (np.roll(unq, -1) - np.roll(unq, 1)) % np.pi
    total = np.sum(gap)
    return (gap / cnt / total * flat.size)[back]


def _pad_ends(t, dim, left, right, end):
    """np.pad along one axis: edge values, or a linear ramp to `end`."""
    n = t.shape[dim]
    lo, hi = t.narrow(dim, 0, 1), t.narrow(dim, n - 1, 1)
    shape = [1] * t.dim()

    def side(edge, width, flip):
        shape[dim] = width
        if end is None:
            r = torch.ones(width, dtype=F64, device=t.device)
        else:
            r = torch.arange(width, dtype=F64, device=t.device) / width
        if flip:
            r = r.flip(0)
        r = r.view(shape)
        e = 0.0 if end is None else end
        return e + (edge - e) * r
    return torch.cat([side(lo, left, False), t, side(hi, right, True)], dim)


def _mirror(i, n):
    if n == 1:
        return torch.zeros_like(i)
    p = 2 * n - 2
    i = torch.remainder(i, p)
    return torch.where(i > n - 1, p - i, i)


def _bspline(order, t):
    """Weights of the order + 1 taps for the fraction t of a coordinate: t
    from its floor (odd orders) or from its nearest sample (even orders),
    by the recursion over the degree."""
    # distance of the coordinate to the first tap
    x = t + order // 2
    w = []
    for k in range(order + 1):
        w.append(_bspline_at(order, x - k))
    return w


def _bspline_at(order, x):
    """Centred B-spline of the given degree at x (truncated powers)."""
    s = 0
    h = (order + 1) / 2
    for j in range(order + 2):
        u = torch.clamp(x + h - j, min=0)
        p = (u > 0).to(F64) if order == 0 else u ** order
        s = s + (-1) ** j * math.comb(order + 1, j) * p
    return s / math.factorial(order)


def _prefilter(n, order):
    """The n x n inverse of the mirrored B-spline sampling matrix."""
    if order < 2 or n == 1:
        return None
    taps = _bspline_at(order, torch.arange(-2, 3, dtype=F64)).numpy()
    M = np.zeros((n, n))
    for k in range(-2, 3):
        for i in range(n):
            p = 2 * n - 2
            m = (i + k) % p
            M[i, p - m if m > n - 1 else m] += taps[k + 2]
    return torch.from_numpy(np.linalg.inv(M)).to("cuda")


class _Exact:
    """One geometry in 64 bits; `volume_of(a, u)` is angle a's share."""

    def __init__(self, kind, angles, ny, nx, order, end):
        self.kind, self.ny, self.nx, self.order = kind, ny, nx, order
        self.end, A = end, len(angles)
        self.w = _angle_weights(angles)
        two = kind == "2d"
        if two:
            self.pny, self.pnx = 1, _pow2(2.1 * nx)
        else:
            self.pny, self.pnx = _pow2(1.75 * ny), _pow2(1.75 * nx)
        self.yl = -(-(self.pny - ny) // 2)
        self.xl = -(-(self.pnx - nx) // 2)
        km = 2 * np.pi * NM / RES
        kx = 2 * np.pi * np.fft.fftfreq(self.pnx).reshape(1, -1)
        ky = 2 * np.pi * np.fft.fftfreq(self.pny).reshape(-1, 1)
        inside = kx ** 2 + ky ** 2 < km ** 2
        M = np.sqrt((km ** 2 - kx ** 2 - ky ** 2) * inside) / km
        axis = _tilt_axis() if kind == "tilted" else (0.0, 1.0, 0.0)
        f = (-1j * km / (2 * np.pi) * 2 * np.pi / A
             * np.abs(kx * axis[1] + ky * axis[0]) * inside)
        self.filt = torch.from_numpy(f / (self.pnx * self.pny)).cuda()
        phase = torch.from_numpy(km * (M - 1)).cuda()
        z = torch.arange(nx, dtype=F64, device="cuda") - nx / 2
        if two:
            z = z + 0.5
        prop = torch.exp(1j * phase * z.view(-1, 1, 1))
        pz = _prefilter(nx, order)
        if pz is not None:
            r = torch.view_as_real(prop).reshape(nx, -1)
            prop = torch.view_as_complex((pz @ r).reshape(
                nx, self.pny, self.pnx, 2))
        self.prop = prop
        self.px = _prefilter(nx, order)
        self.py = _prefilter(ny, order) if kind == "tilted" else None
        self.geo = [self._geometry(float(p), angles) for p in angles]

    def _geometry(self, phi, angles):
        n = self.nx
        if self.kind != "tilted":
            # scipy.ndimage.rotate by -phi, cosine and sine exact at
            # multiples of 90 degrees
            deg = -phi * 180 / np.pi if self.kind == "2d" \
                else -np.rad2deg(phi)
            q = int(round(deg / 90))
            r = math.radians(deg - 90 * q)
            c, s = math.cos(r), math.sin(r)
            c, s = [(c, s), (-s, c), (-c, -s), (s, -c)][q % 4]
            mat = np.array([[c, s], [-s, c]])
            ctr = np.array([(n - 1) / 2] * 2)
            return mat, ctr - mat @ ctr
        # odtbrain/_alg3d_bppt.py:230-371 for an axis in the y-z plane
        _u, v, w = _tilt_axis()
        th = np.arccos(v)
        rx = np.array([[1, 0, 0], [0, np.cos(th), -np.sin(th)],
                       [0, np.sin(th), np.cos(th)]])

        def point(a):
            return rx @ (np.cos(th) * np.array(
                [np.sin(a - angles[0]), 0, np.cos(a - angles[0])]))
        pt = point(phi) - (point(angles[0]) - np.array([0, 0, 1]))
        pt = rx.T @ pt  # the axis becomes y
        ph = np.arctan2(pt[0], pt[2])
        t = -np.arctan2(pt[1], np.sqrt(pt[0] ** 2 + pt[2] ** 2))
        rt = np.array([[1, 0, 0], [0, np.cos(t), -np.sin(t)],
                       [0, np.sin(t), np.cos(t)]])
        rp = np.array([[np.cos(ph), 0, -np.sin(ph)], [0, 1, 0],
                       [np.sin(ph), 0, np.cos(ph)]])
        mat = rt.T @ rp.T
        ctr = 0.5 * np.array([n, self.ny, n]) - 0.5
        return mat, ctr - mat @ ctr

    def slab(self, a, u, gain=None):
        """Prefiltered coefficients [z][y][x] of angle a."""
        u = u.to(C128) * self.w[a]
        p = u
        if self.kind != "2d":
            p = _pad_ends(p, 0, self.yl, self.pny - self.ny - self.yl,
                          self.end)
        p = _pad_ends(p, 1, self.xl, self.pnx - self.nx - self.xl, self.end)
        spec = torch.fft.fft2(p) * self.filt
        if gain is not None:
            spec = spec * gain
        out = []
        for z0 in range(0, self.nx, 64):
            v = torch.fft.ifft2(spec * self.prop[z0:z0 + 64], norm="forward")
            out.append(v[:, self.yl:self.yl + self.ny,
                         self.xl:self.xl + self.nx])
        s = torch.cat(out)
        if self.px is not None:
            s = torch.complex(s.real.contiguous() @ self.px.T,
                              s.imag.contiguous() @ self.px.T)
        if self.py is not None:
            s = torch.complex(self.py @ s.real.contiguous(),
                              self.py @ s.imag.contiguous())
        return s

    def _taps(self, c, n):
        o = self.order
        s = torch.floor(c) if o % 2 else torch.floor(c + 0.5)
        w = _bspline(o, c - s)
        s = s.to(torch.int64) - o // 2
        inside = ((c >= 0) & (c <= n - 1)).to(F64)
        return [_mirror(s + k, n) for k in range(o + 1)], w, inside

    def resampled(self, a, s):
        """Angle a's coefficients in the volume's frame [z][y][x]."""
        mat, off = self.geo[a]
        nx, ny = self.nx, self.ny
        i = torch.arange(nx, dtype=F64, device="cuda")
        if self.kind != "tilted":
            oz, ox = i.view(-1, 1), i.view(1, -1)
            cz = (float(off[0]) + float(mat[0, 0]) * oz) \
                + float(mat[0, 1]) * ox
            cx = (float(off[1]) + float(mat[1, 0]) * oz) \
                + float(mat[1, 1]) * ox
            iz, wz, inz = self._taps(cz, nx)
            ix, wx, inx = self._taps(cx, nx)
            flat = s.permute(0, 2, 1).reshape(nx * nx, ny)
            acc = 0
            for j in range(self.order + 1):
                for k in range(self.order + 1):
                    w = (wz[j] * wx[k] * inz * inx).view(-1, 1)
                    acc = acc + w * flat[(iz[j] * nx + ix[k]).view(-1)]
            return acc.view(nx, nx, ny).permute(0, 2, 1)
        # the frame of the resampling is (x, -y, z)
        j = torch.arange(ny, dtype=F64, device="cuda")
        o0, o1, o2 = i.view(-1, 1, 1), j.view(1, -1, 1), i.view(1, 1, -1)
        taps, ins = [], 1.0
        for ax, n in enumerate((nx, ny, nx)):
            c = ((float(off[ax]) + float(mat[ax, 0]) * o0)
                 + float(mat[ax, 1]) * o1) + float(mat[ax, 2]) * o2
            t, w, inside = self._taps(c, n)
            taps.append((t, w))
            ins = ins * inside
        flat = s.permute(2, 1, 0).flip(1).reshape(-1)
        acc = 0
        for j0 in range(self.order + 1):
            for j1 in range(self.order + 1):
                base = (taps[0][0][j0] * ny + taps[1][0][j1]) * nx
                w01 = taps[0][1][j0] * taps[1][1][j1] * ins
                for j2 in range(self.order + 1):
                    acc = acc + (w01 * taps[2][1][j2]) \
                        * flat[base + taps[2][0][j2]]
        return acc.permute(2, 1, 0).flip(1)

    def volume_of(self, a, u, gain=None):
        return self.resampled(a, self.slab(a, u, gain))

    def volume(self, sino, gain=None):
        v = 0
        for a in range(sino.shape[0]):
            v = v + self.volume_of(a, sino[a],
                                   None if gain is None else gain[a])
        return v


def _exact_rytov(case, seed):
    ang, ny, nx = _circle(case["A"]), case["ny"], case["nx"]
    field = torch.exp(_sinogram(ang, ny, nx, seed)).to(C128)
    # the phase without its whole turns is known: the phantom's own, up to
    # the rounding of the field
    true = _sinogram(ang, ny, nx, seed).imag.to(F64)
    phase = torch.angle(field)
    phase = phase + 2 * np.pi * torch.round((true - phase) / (2 * np.pi))
    return torch.complex(torch.log(field.abs()), phase)


def _exact_apple(case, seed):
    n = case["n"]
    f = _cored_volume(n, seed).real.to(F64)
    core = torch.from_numpy(_apple_core(n)).cuda()
    orig = torch.fft.fftn(f)
    hull = torch.fft.fftshift(torch.where(core, math.nan, orig.abs()))
    score = torch.fft.fftshift(core)
    hull = torch.where(score, hull.transpose(0, 1), hull)
    if torch.isnan(hull).any():
        return None
    sigma = n / 100
    r = int(4 * sigma + 0.5)
    g = torch.exp(-0.5 * torch.arange(-r, r + 1, dtype=F64) ** 2 / sigma ** 2)
    g = (g / g.sum()).tolist()
    for ax in range(3):
        acc = torch.zeros_like(hull)
        for k in range(-r, r + 1):
            m = n - abs(k)
            if m > 0:
                acc.narrow(ax, max(0, -k), m).add_(
                    hull.narrow(ax, max(0, k), m), alpha=g[k + r])
        hull = acc
    envelope = torch.fft.ifftshift(hull)
    x = (torch.arange(n, dtype=F64, device="cuda") - n / 2) / (n / 2)
    outside = (x.view(-1, 1, 1) ** 2 + x.view(1, -1, 1) ** 2
               + x.view(1, 1, -1) ** 2) > 1
    data = f.to(C128)
    prev = orig[core].abs().sum() / data.numel()
    norm = None
    for i in range(100):
        re = torch.where(outside, 0.0, data.real).clamp(min=0)
        ft = torch.fft.fftn(re)
        ft = torch.where(ft.abs() > envelope, ft * 0.95, ft)
        ft = torch.where(core, ft, orig)
        data = torch.fft.ifftn(ft)
        cur = ft[core].abs().sum() / data.numel()
        diff = cur - prev
        if i == 0:
            norm = diff
        elif abs(float(diff / norm)) < 0.01:
            break
        prev = cur
    return data


def _exact_gains(params, feat, positions, pny, pnx):
    """1 + MLP at the listed spectrum positions, 1 elsewhere."""
    A = feat.shape[0]
    fx = 2 * np.pi * np.fft.fftfreq(pnx) / np.pi
    fy = 2 * np.pi * np.fft.fftfreq(pny) / np.pi
    grid = np.stack(np.broadcast_arrays(fx.reshape(1, -1),
                                        fy.reshape(-1, 1)), -1)
    grid = torch.from_numpy(grid.reshape(-1, 2)).cuda()[positions.long()]
    x = torch.cat([grid.repeat(A, 1),
                   feat.to(F64).repeat_interleave(grid.shape[0], 0)], 1)
    for i in (1, 2, 3):
        x = torch.nn.functional.silu(x @ params["W%d" % i].T
                                     + params["b%d" % i])
    y = x @ params["W4"].T + params["b4"]
    y = torch.complex(1 + y[:, 0], y[:, 1]).view(A, -1)
    out = torch.ones((A, pny * pnx), dtype=C128, device="cuda")
    return out.index_copy(1, positions.long(), y).view(A, pny, pnx)


def exact(case, seed):
    kind = case["kind"]
    if kind == "2d":
        sino = _sinogram(_circle(case["A"]), 1, case["n"], seed)
        e = _Exact("2d", _circle(case["A"]), 1, case["n"], 3,
                   None if case["pad"] == "edge" else 0.0)
        return e.volume(sino)[:, 0, :]
    if kind in ("3d", "tilted"):
        ang = _circle(case["A"])
        sino = _sinogram(ang, case["ny"], case["nx"], seed)
        e = _Exact(kind, ang, case["ny"], case["nx"], case["order"],
                   None if case["pad"] == "edge" else 0.0)
        v = e.volume(sino)
        return v.real if case["onlyreal"] else v
    if kind == "vjp":
        n, A = case["n"], case["A"]
        e = _Exact("3d", _circle(A), n, n, 2, None)
        sino = _sinogram(_circle(A), n, n, seed)
        shape = (e.pny, e.pnx)
        gain = (0.5 + _uniform(seed + 1, shape)).to(F64).requires_grad_()
        grad = _normal(seed + 2, (n, n, n)).to(C128)
        vol, gs, gg = 0, [], 0
        for a in range(A):
            u = sino[a].to(C128).requires_grad_()
            v = e.volume_of(a, u, gain)
            x, y = torch.autograd.grad(v, (u, gain), grad)
            vol, gg = vol + v.detach(), gg + y
            gs.append(x)
        return dict(volume=vol, sino_grad=torch.stack(gs), gain_grad=gg)
    if kind == "train":
        n, A = case["n"], case["A"]
        s = prepare(case, seed)
        e = _Exact("3d", wedge_angles(A), n, n, 2, None)
        params = {k: v.to(F64).requires_grad_()
                  for k, v in s["mlp"].params.items()}
        gain = _exact_gains(params, s["filt"].feat, s["filt"].positions,
                            e.pny, e.pnx)
        held = gain.detach().requires_grad_()
        with torch.no_grad():
            vol = e.volume(s["sino"], held)
        tgt = s["target"].to(C128)
        diff, nt = vol - tgt, torch.linalg.vector_norm(tgt) ** 2
        dgain = []
        for a in range(A):
            ga = held[a].detach().requires_grad_()
            v = e.volume_of(a, s["sino"][a], ga)
            dgain.append(torch.autograd.grad(v, ga, diff * (2.0 / nt))[0])
        names = sorted(params)
        g = torch.autograd.grad(gain, [params[k] for k in names],
                                torch.stack(dgain))
        return dict(volume=vol, loss=torch.linalg.vector_norm(diff) ** 2 / nt,
                    gain_grad=torch.stack(dgain), **dict(zip(names, g)))
    if kind == "rytov":
        return _exact_rytov(case, seed)
    if kind == "apple":
        return _exact_apple(case, seed)
    f = _object_function(case["n"], seed).to(C128)
    r = NM * torch.sqrt(f / (2 * np.pi * NM / RES) ** 2 + 1)
    return torch.where(r.real < 0, -r, r)
