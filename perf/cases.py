"""Performance cases: the calls a reconstruction program makes, over their range of sizes.

The kinds, each through the package's public entry points:

  conv2d      A^T A on a stack of slices through the Toeplitz PSF (sysmat2d)
  conv3d      A^T A on a laminography volume through the Toeplitz PSF (sysmat)
  forward2d   projection of a stack of slices onto a sinogram
  backproj2d  backprojection of a sinogram stack
  forward3d   laminography projection (data generation, alignment)
  backproj3d  laminography backprojection (the right-hand side of every solve)
  sb3d        Split-Bregman TV solve with a prepared PSF
  batch2d     many independent tomography slices of uneven size, solved together
  mbir2d      one tomography slice from host sinogram to host image
  mbir3d      one laminography volume, projections and result in device memory

Inputs are seeded ellipse and ellipsoid phantoms with 1 % noise: volumes are
sampled on the grid, projections come from the closed-form shadow of an
ellipsoid.  `exact` restates the operators in 64 bits with torch: non-uniform
sums as matrix products, the point spread function as its sum of Dirichlet
kernels, convolutions by FFT.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import laminocam_b200 as lc
from laminocam_b200 import _lib

DEV = "cuda"


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    # Two choices are made for the comparison with 64 bits.  Unregularised CG
    # is stopped early: its iterates depend on the rounding of any FP32 form
    # after more than about five iterations.  The projection cases avoid a tilt
    # of 30 degrees, where the band limit |q| <= pi passes exactly through
    # lattice points and rounding decides which of them are in.
    return [
        # one slice inside an interactive or streaming solve: three short kernels, launch-bound
        dict(name="conv2d_small", kind="conv2d", ns=1, n=255, ntheta=180),
        # a stack of full-width slices, as a tomography solve applies it every iteration
        dict(name="conv2d_stack", kind="conv2d", ns=8, n=1023, ntheta=720),
        # the laminography benchmark's operator (padded volume), mirror-symmetric scan
        dict(name="conv3d_lamino", kind="conv3d", n1=29, n2=721, n3=721, ntheta=360, nrows=721, ncols=721,
             gamma=-30.0, beta=0.0),
        # a scan with a second tilt and ragged sizes: no mirror symmetry in z
        dict(name="conv3d_tilted", kind="conv3d", n1=31, n2=360, n3=363, ntheta=120, nrows=361, ncols=363,
             gamma=-35.0, beta=3.0),
        # simulating the sinograms of a few slices
        dict(name="forward2d", kind="forward2d", ns=4, n=511, ntheta=360),
        # the right-hand side of a slice stack
        dict(name="backproj2d", kind="backproj2d", ns=4, n=1023, ntheta=720),
        # simulating a laminography scan
        dict(name="forward3d", kind="forward3d", n1=21, n2=361, n3=361, ntheta=180, nrows=361, ncols=361,
             gamma=-28.0, beta=0.0),
        # the right-hand side of a laminography solve at the benchmark's detector
        dict(name="backproj3d", kind="backproj3d", n1=21, n2=511, n3=511, ntheta=360, nrows=511, ncols=511,
             gamma=-32.0, beta=0.0),
        # a short TV solve with the PSF in hand (warm restart, parameter search), default schedule
        dict(name="sb3d", kind="sb3d", n1=29, n2=721, n3=721, ntheta=360, nrows=721, ncols=721,
             gamma=-30.0, beta=0.0, outer=20, refresh=1),
        # a queue of independent slices of uneven size
        dict(name="batch2d", kind="batch2d", jobs=16, lo=127, hi=1023, iters=5, mix=7),
        # one slice end to end: upload, backprojection, PSF, Split-Bregman, download
        dict(name="mbir2d", kind="mbir2d", ns=1, n=511, ntheta=360, outer=30),
        # the benchmark: one complete laminography reconstruction
        dict(name="mbir3d", kind="mbir3d", r1=21, r2=511, r3=511, ntheta=360, nrows=511, ncols=511,
             gamma=-30.0, outer=100, refresh=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["conv2d", "conv3d", "forward2d", "backproj2d", "forward3d", "backproj3d", "sb3d",
                       "batch2d", "mbir2d", "mbir3d"])
    if kind in ("conv2d", "forward2d", "backproj2d"):
        n = _log(rng, 63, 1535)
        ns = max(1, min(_log(rng, 1, 16), 8 * 1024 * 1024 // (n * n)))
        return dict(kind=kind, ns=ns, n=n, ntheta=_log(rng, 45, 1080))
    if kind in ("conv3d", "forward3d", "backproj3d", "sb3d"):
        n2 = _log(rng, 63, 721)
        n3 = min(721, max(63, int(n2 * rng.uniform(0.8, 1.25))))
        nr = min(721, max(63, int(n2 * rng.uniform(0.9, 1.1))))
        nc = min(721, max(63, int(n3 * rng.uniform(0.9, 1.1))))
        c = dict(kind=kind, n1=rng.randint(7, 45 if max(n2, n3) < 512 else 29), n2=n2, n3=n3,
                 ntheta=_log(rng, 60, 360), nrows=nr, ncols=nc, gamma=-(rng.randint(15, 44) + 0.5),
                 beta=rng.choice([0.0, 0.0, 2.5]))
        if kind in ("forward3d", "backproj3d"):
            c["ntheta"] = min(c["ntheta"], max(60, 94_000_000 // (nr * nc)))
        if kind == "sb3d":
            c["outer"] = rng.randint(5, 20)
            c["refresh"] = rng.choice([1, 4, 16])
        return c
    if kind == "batch2d":
        return dict(kind=kind, jobs=rng.randint(4, 24), lo=rng.randint(64, 200), hi=rng.randint(400, 1023),
                    iters=rng.randint(3, 5), mix=rng.randint(0, 10 ** 6))
    if kind == "mbir2d":
        n = _log(rng, 63, 1535)
        return dict(kind=kind, ns=max(1, min(_log(rng, 1, 8), 4 * 1024 * 1024 // (n * n))), n=n,
                    ntheta=_log(rng, 45, 1080), outer=rng.randint(10, 40))
    r2 = _log(rng, 63, 511)
    r3 = min(511, max(63, int(r2 * rng.uniform(0.8, 1.25))))
    return dict(kind=kind, r1=rng.randint(5, 21), r2=r2, r3=r3, ntheta=_log(rng, 60, 360), nrows=r2, ncols=r3,
                gamma=-(rng.randint(15, 44) + 0.5), outer=rng.randint(20, 100), refresh=rng.choice([1, 16]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return np.random.RandomState(seed % (2 ** 32 - 1))


def _noise(shape, scale, seed, device=DEV):
    g = torch.Generator(device).manual_seed(seed)
    return torch.randn(shape, generator=g, device=device) * scale


def _theta2d(ntheta):
    return np.arange(ntheta) * np.pi / ntheta


def _theta3d(ntheta):
    return np.arange(ntheta) * 2 * np.pi / ntheta


def _euler(a, b, c):
    ca, sa, cb, sb, cc, sc = np.cos(a), np.sin(a), np.cos(b), np.sin(b), np.cos(c), np.sin(c)
    return (np.array([[ca, -sa, 0], [sa, ca, 0], [0, 0, 1]]) @ np.array([[cb, 0, sb], [0, 1, 0], [-sb, 0, cb]])
            @ np.array([[cc, -sc, 0], [sc, cc, 0], [0, 0, 1]]))


def _ellipsoids(dims, rs, count=12):
    """(centre, shape matrix S, density) in voxels, x^T S^-1 x <= 1; axes ordered (x, y, z)."""
    half = np.array([dims[2], dims[1], max(dims[0], 1)]) / 2.0
    out = []
    for _ in range(count):
        c = rs.uniform(-0.6, 0.6, 3) * half
        ax = rs.uniform(0.08, 0.4, 3) * half
        if dims[0] == 1:
            R = _euler(rs.uniform(0, np.pi), 0.0, 0.0)
            c[2], ax[2] = 0.0, 1.0
        else:
            R = _euler(rs.uniform(0, np.pi), 0.0, 0.0)
        out.append((c, R @ np.diag(ax ** 2) @ R.T, rs.uniform(0.1, 1.0)))
    return out


def _volume(dims, seed):
    """{n1, n2, n3} phantom with 1 % noise; a slice stack (n1 slices) when every slice is its own image."""
    n1, n2, n3 = dims
    ax = [torch.arange(n, device=DEV, dtype=torch.float32) - n // 2 for n in (n3, n2, n1)]
    v = torch.zeros(dims, device=DEV)
    for c, S, d in _ellipsoids(dims, _gen(seed)):
        Q = np.linalg.inv(S)
        x, y, z = (ax[0] - c[0])[None, None, :], (ax[1] - c[1])[None, :, None], (ax[2] - c[2])[:, None, None]
        q = (Q[0, 0] * x * x + Q[1, 1] * y * y + 2 * Q[0, 1] * x * y + Q[2, 2] * z * z
             + 2 * Q[0, 2] * x * z + 2 * Q[1, 2] * y * z)
        v += d * (q <= 1.0)
    return (v + _noise(dims, 0.01, seed + 1)).contiguous()


def _slices(ns, n, seed):
    return torch.cat([_volume((1, n, n), seed * 131 + k) for k in range(ns)]).contiguous()


def _sinograms(ns, n, theta, seed):
    """{ns, ntheta, n} line integrals of one ellipse phantom per slice, maximum 1, 1 % noise."""
    t = torch.arange(n, device=DEV, dtype=torch.float32)[None, :] - n // 2
    cs = torch.tensor(np.cos(theta), device=DEV, dtype=torch.float32)[:, None]
    sn = torch.tensor(np.sin(theta), device=DEV, dtype=torch.float32)[:, None]
    out = torch.zeros((ns, len(theta), n), device=DEV)
    for k in range(ns):
        for c, S, d in _ellipsoids((1, n, n), _gen(seed * 131 + k)):
            T = S[0, 0] * cs * cs + S[1, 1] * sn * sn + 2 * S[0, 1] * cs * sn
            u = t - (c[0] * cs + c[1] * sn)
            det = S[0, 0] * S[1, 1] - S[0, 1] ** 2
            out[k] += 2 * d * math.sqrt(det) * torch.sqrt(torch.clamp(1 - u * u / T, min=0)) / torch.sqrt(T)
    out /= out.max()
    return (out + _noise(out.shape, 0.01, seed + 2)).contiguous()


def _rot_cols(theta, gamma, beta):
    """Detector axes in the volume frame: (x, y, z) of the column axis a and the row axis b per angle."""
    ct, st = np.cos(theta), np.sin(theta)
    cb, sb, cg, sg = math.cos(beta), math.sin(beta), math.cos(gamma), math.sin(gamma)
    a = np.stack([np.full_like(ct, cb * cg), np.full_like(ct, -cb * sg), np.full_like(ct, sb)], 1)
    b = np.stack([ct * sg + st * sb * cg, ct * cg - st * sb * sg, -st * cb], 1)
    return a, b


def _projections(c, dims, theta, seed):
    """{ntheta, nrows, ncols} shadows of an ellipsoid phantom, maximum 1, 1 % noise."""
    gamma, beta = math.radians(c["gamma"]), math.radians(c.get("beta", 0.0))
    a, b = _rot_cols(theta, gamma, beta)
    nr, nc = c["nrows"], c["ncols"]
    u = (torch.arange(nc, device=DEV, dtype=torch.float32) - nc // 2)[None, None, :]
    v = (torch.arange(nr, device=DEV, dtype=torch.float32) - nr // 2)[None, :, None]
    out = torch.zeros((len(theta), nr, nc), device=DEV)

    def col(x):
        return torch.tensor(np.asarray(x, dtype=np.float32), device=DEV)[:, None, None]

    for cen, S, d in _ellipsoids(dims, _gen(seed)):
        Saa, Sbb, Sab = (np.einsum("ti,ij,tj->t", p, S, q) for p, q in ((a, a), (b, b), (a, b)))
        det = Saa * Sbb - Sab ** 2
        du, dv = u - col(a @ cen), v - col(b @ cen)
        q = col(Sbb / det) * du * du + col(Saa / det) * dv * dv - col(2 * Sab / det) * du * dv
        out += col(2 * d * np.sqrt(np.linalg.det(S) / det)) * torch.sqrt(torch.clamp(1 - q, min=0))
        del du, dv, q
    out /= out.max()
    out += _noise(out.shape, 0.01, seed + 3)
    return out


def _rhs3d(c, seed):
    """Right-hand side of a solve: the phantom under the limit of A^T A for dense sampling, 2 ntheta / rho with
    rho the frequency's distance from the column axis, in the units of normalised projections."""
    dims = (c["n1"], c["n2"], c["n3"])
    x = _volume(dims, seed) / (0.25 * min(c["n2"], c["n3"]))
    g = math.radians(c["gamma"])
    P = [2 * n for n in dims]
    w = [torch.fft.fftfreq(n, device=DEV) * 2 * math.pi for n in P[:2]] + \
        [torch.fft.rfftfreq(P[2], device=DEV) * 2 * math.pi]
    u = math.sin(g) * w[2][None, :] + math.cos(g) * w[1][:, None]
    f = torch.fft.rfftn(x, s=P)
    for k in range(P[0]):
        f[k] *= 2 * c["ntheta"] / torch.clamp(torch.sqrt(u * u + w[0][k] ** 2), min=math.pi / c["nrows"])
    return torch.fft.irfftn(f, s=P)[:dims[0], :dims[1], :dims[2]].contiguous()


def _job_sizes(c):
    rs = _gen(c["mix"])
    out = []
    for _ in range(c["jobs"]):
        n = int(round(math.exp(rs.uniform(math.log(c["lo"]), math.log(c["hi"])))))
        out.append((n, int(rs.randint(90, 721))))
    return out


def _grid3d(c):
    theta = _theta3d(c["ntheta"])
    return lc.PolarGrid(theta, math.radians(c["gamma"]), math.radians(c.get("beta", 0.0)), c["nrows"], c["ncols"])


def prepare(case, seed):
    c, k = case, case["kind"]
    s = dict(case=c)
    if k in ("conv2d", "forward2d", "backproj2d"):
        s["pg"] = lc.PolarGrid2D(_theta2d(c["ntheta"]), c["n"])
        if k == "backproj2d":
            s["x"] = _sinograms(c["ns"], c["n"], _theta2d(c["ntheta"]), seed)
        else:
            s["x"] = _slices(c["ns"], c["n"], seed)
        if k == "conv2d":
            s["psf"] = lc.PointSpreadFunction2D(s["pg"], c["n"], c["ns"])
    elif k in ("conv3d", "forward3d", "backproj3d", "sb3d"):
        dims = (c["n1"], c["n2"], c["n3"])
        s["pg"] = _grid3d(c)
        if k == "backproj3d":
            s["x"] = _projections(c, dims, _theta3d(c["ntheta"]), seed)
        elif k == "sb3d":
            s["x"] = _rhs3d(c, seed)
            s["x0"] = torch.zeros_like(s["x"])
        else:
            s["x"] = _volume(dims, seed)
        if k in ("conv3d", "sb3d"):
            s["psf"] = lc.PointSpreadFunction(s["pg"], dims)
    elif k == "batch2d":
        s["jobs"] = []
        for i, (n, nth) in enumerate(_job_sizes(c)):
            th = _theta2d(nth)
            s["jobs"].append((_sinograms(1, n, th, seed * 1009 + i).cpu().numpy(), th, n))
        s["params"] = lc.ReconParams(max_iters=c["iters"], tol=0.0, xtol=0.0, use_graph=True)
    elif k == "mbir2d":
        s["theta"] = _theta2d(c["ntheta"])
        s["x"] = _sinograms(c["ns"], c["n"], s["theta"], seed).cpu().numpy()
        s["params"] = lc.ReconParams(regularizer="split_bregman", recon_dims=(c["ns"], c["n"], c["n"]),
                                     max_iters=c["outer"], inner_iters=1, lam=0.1, mu=10.0, tol=1e-5, xtol=0.0,
                                     use_graph=True)
    elif k == "mbir3d":
        s["theta"] = _theta3d(c["ntheta"])
        s["x"] = _projections(c, (c["r1"], c["r2"], c["r3"]), s["theta"], seed)
        s["gamma"] = np.full(c["ntheta"], math.radians(c["gamma"]))
        s["beta"] = np.zeros(c["ntheta"])
        s["ctx"] = lc.Context.default()
        s["params"] = lc.ReconParams(regularizer="split_bregman", recon_dims=(c["r1"], c["r2"], c["r3"]),
                                     max_iters=c["outer"], inner_iters=1, lam=0.1, mu=10.0, tol=1e-5, xtol=0.0,
                                     use_graph=True, residual_refresh=c["refresh"])
    else:
        raise ValueError(k)
    return s


def run(s):
    c, k = s["case"], s["case"]["kind"]
    if k == "conv2d":
        return lc.sysmat2d(s["x"], s["psf"])
    if k == "conv3d":
        return lc.sysmat(s["x"], s["psf"])
    if k == "forward2d":
        return lc.forward2d(s["x"], s["pg"])
    if k == "backproj2d":
        return lc.backproj2d(s["x"], s["pg"], (c["ns"], c["n"], c["n"]))
    if k == "forward3d":
        return lc.forward(s["x"], s["pg"])
    if k == "backproj3d":
        return lc.backproj(s["x"], s["pg"], (c["n1"], c["n2"], c["n3"]))
    if k == "sb3d":
        return lc.split_bregman(s["psf"], s["x"], s["x0"], 0.1, 10.0, c["outer"], 1, 1e-5, 0.0, use_graph=True,
                                residual_refresh=c["refresh"])
    if k == "batch2d":
        return lc.MBIR2D_batch(s["jobs"], s["params"])
    if k == "mbir2d":
        return lc.MBIR2D(s["x"], s["theta"], s["params"])
    # the device-memory form of MBIR (lc_mbir3d_device of the C interface)
    ctx, x = s["ctx"], s["x"]
    ctx.sync_stream()
    out = torch.empty(s["params"].recon_dims, device=x.device)
    dp = C.POINTER(C.c_double)
    rp, st = s["params"].to_c(), _lib.SolverStats()
    rc = ctx.lib.lc_mbir3d_device(ctx.handle, C.c_void_p(x.data_ptr()), *x.shape, s["theta"].ctypes.data_as(dp),
                                  s["gamma"].ctypes.data_as(dp), s["beta"].ctypes.data_as(dp), None,
                                  (C.c_int * 3)(*out.shape), C.byref(rp), C.c_void_p(out.data_ptr()), C.byref(st))
    if rc:
        raise RuntimeError(ctx.lib.lc_last_error(ctx.handle))
    return out


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _fft_flops(dims):
    """A real transform pair (forward and inverse) on the padded grid."""
    n = 1.0
    for d in dims:
        n *= 2 * d
    return 2 * 2.5 * n * math.log2(n)


def _spectrum_bytes(dims):
    n = 4.0
    for d in dims[:-1]:
        n *= 2 * d
    return n * (dims[-1] + 1)


def _padded(r):
    v = int(np.float32(r) * np.float32(1.4142))
    return v - 1 if v % 2 == 0 else v


W = 7  # kernel width at the default tolerance


def work(case):
    c, k = case, case["kind"]
    if k in ("conv2d", "forward2d", "backproj2d"):
        vol, sino = c["ns"] * c["n"] ** 2, c["ns"] * c["ntheta"] * c["n"]
        if k == "conv2d":
            d = (c["n"], c["n"])
            return dict(bytes=8.0 * vol + _spectrum_bytes(d), flops=c["ns"] * _fft_flops(d))
        return dict(bytes=4.0 * (vol + sino), flops=c["ns"] * _fft_flops((c["n"], c["n"])) / 2 + 4.0 * W * W * sino)
    if k in ("conv3d", "forward3d", "backproj3d", "sb3d"):
        d = (c["n1"], c["n2"], c["n3"])
        vol, pts = float(c["n1"] * c["n2"] * c["n3"]), float(c["ntheta"] * c["nrows"] * c["ncols"])
        if k == "conv3d":
            return dict(bytes=8.0 * vol + _spectrum_bytes(d), flops=_fft_flops(d))
        if k == "sb3d":
            return dict(bytes=12.0 * vol + _spectrum_bytes(d), flops=c["outer"] * (_fft_flops(d) + 120.0 * vol))
        return dict(bytes=4.0 * (vol + pts), flops=_fft_flops(d) / 2 + 4.0 * W ** 3 * pts)
    if k in ("batch2d", "mbir2d"):
        jobs = _job_sizes(c) if k == "batch2d" else [(c["n"], c["ntheta"])] * c["ns"]
        b = sum(4.0 * (n * t + n * n) for n, t in jobs)
        it = c["iters"] + 1 if k == "batch2d" else c["outer"]
        return dict(bytes=b, flops=sum(it * _fft_flops((n, n)) + 4.0 * W * W * n * t for n, t in jobs))
    r = (c["r1"], c["r2"], c["r3"])
    d = tuple(_padded(v) for v in r)
    pts = float(c["ntheta"]) * _padded(c["nrows"]) * _padded(c["ncols"])
    vol = float(d[0] * d[1] * d[2])
    return dict(bytes=4.0 * (c["ntheta"] * c["nrows"] * c["ncols"] + r[0] * r[1] * r[2]),
                flops=c["outer"] * (_fft_flops(d) + 120.0 * vol) + 4.0 * W ** 3 * pts)


def tolerance(case):
    k = case["kind"]
    # FP32 transforms (conv), the NUFFT tolerance 1e-6 (projections), and what
    # the iterations make of either: about four times the measured distance
    # from the 64-bit result.
    return {"conv2d": {"rel": 1e-6}, "conv3d": {"rel": 1e-6}, "forward2d": {"rel": 2.5e-6},
            "backproj2d": {"rel": 5e-6}, "forward3d": {"rel": 3.5e-6}, "backproj3d": {"rel": 1e-5},
            "sb3d": {"rel": 6e-6}, "batch2d": {"rel": 5e-5}, "mbir2d": {"rel": 4.5e-5},
            "mbir3d": {"rel": 1.5e-5}}[k]


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
F8, C16 = torch.float64, torch.complex128
FLOP_LIMIT = 2.5e14


def _modes(n):
    return torch.arange(n, device=DEV, dtype=F8) - n // 2


def _radial(n):
    return (torch.arange(n, device=DEV, dtype=F8) + 0.5) * (2 * math.pi / n) - math.pi


def _phase(a, b, sign):
    p = torch.outer(a, b)
    return torch.complex(torch.cos(p), sign * torch.sin(p))


def _rolled(y, s, dim):
    """v[m] = y[(m + s) mod n]"""
    return torch.roll(y, -s, dim)


def _detector(y, dim, pre, post, inverse):
    """v[m] = y[m + pre]; V = DFT(v); out[k] = V[k + post] (indices mod n), unnormalised."""
    n = y.shape[dim]
    v = _rolled(y, pre, dim)
    v = torch.fft.ifft(v, dim=dim) * n if inverse else torch.fft.fft(v, dim=dim)
    return _rolled(v, post, dim)


def _exact_forward2d(x, theta):
    ns, n2, n3 = x.shape
    r, ky, kx = _radial(n3), _modes(n2), _modes(n3)
    out = torch.empty((ns, len(theta), n3), device=DEV, dtype=F8)
    xd = x.to(C16)
    for i, t in enumerate(theta):
        ex, ey = _phase(r * math.cos(t), kx, -1), _phase(r * math.sin(t), ky, -1)
        for s in range(ns):
            cj = ((ex @ xd[s].T) * ey).sum(1)
            out[s, i] = _detector(cj, 0, (n3 + 1) // 2, n3 // 2, True).real / n3
    return out


def _exact_backproj2d(y, theta, n):
    ns, nth, nr = y.shape
    r, k = _radial(nr), _modes(n)
    cj = _detector(y.to(C16), 2, nr // 2, (nr + 1) // 2, False)
    out = torch.zeros((ns, n, n), device=DEV, dtype=C16)
    for i, t in enumerate(theta):
        ex, ey = _phase(k, r * math.cos(t), +1), _phase(k, r * math.sin(t), +1)
        for s in range(ns):
            out[s] += (ey * cj[s, i]) @ ex.T
    return out.real / nr


def _detector_axes(c):
    gamma, beta = math.radians(c["gamma"]), math.radians(c.get("beta", 0.0))
    return _rot_cols(_theta3d(c["ntheta"]), gamma, beta)


def _exact_backproj3d(y, c, dims):
    """Row by row: with no second tilt a detector row has one z, so its points sum into one plane."""
    nth, nr, nc = y.shape
    n1, n2, n3 = dims
    if c.get("beta", 0.0) != 0.0 or 8.0 * nth * nr * nc * n2 * n3 > FLOP_LIMIT:
        return None
    a, b = _detector_axes(c)
    qx, qy = _radial(nc), _radial(nr)
    kz, ky, kx = _modes(n1), _modes(n2), _modes(n3)
    out = torch.zeros((n1, n2 * n3), device=DEV, dtype=C16)
    step = max(1, min(nr, int(2.0e9 / (16.0 * (nc * (n2 + n3) + n2 * n3)))))
    for i in range(nth):
        cj = _detector(y[i].to(C16), 1, nc // 2, (nc + 1) // 2, False)
        cj = _detector(cj, 0, nr // 2, (nr + 1) // 2, False)
        for r0 in range(0, nr, step):
            q = qy[r0:r0 + step, None]
            px, py, pz = (a[i][m] * qx[None, :] + b[i][m] * q for m in range(3))
            m = (px.abs() <= math.pi) & (py.abs() <= math.pi) & (pz.abs() <= math.pi)
            ey = py[:, None, :] * ky[None, :, None]
            ey = torch.complex(torch.cos(ey), torch.sin(ey)) * (cj[r0:r0 + step] * m)[:, None, :]
            ex = px[:, :, None] * kx[None, None, :]
            ex = torch.complex(torch.cos(ex), torch.sin(ex))
            out += _phase(kz, pz[:, 0], +1) @ torch.bmm(ey, ex).reshape(len(q), n2 * n3)
    return out.real.reshape(dims) / (nr * nc)


def _exact_forward3d(x, c):
    n1, n2, n3 = x.shape
    nth, nr, nc = c["ntheta"], c["nrows"], c["ncols"]
    if c.get("beta", 0.0) != 0.0 or 8.0 * nth * nr * nc * n2 * n3 > FLOP_LIMIT:
        return None
    a, b = _detector_axes(c)
    qx, qy = _radial(nc), _radial(nr)
    kz, ky, kx = _modes(n1), _modes(n2), _modes(n3)
    xd = x.to(C16).reshape(n1, n2 * n3)
    out = torch.empty((nth, nr, nc), device=DEV, dtype=F8)
    step = max(1, min(nr, int(2.0e9 / (16.0 * (nc * (n2 + n3) + n2 * n3)))))
    for i in range(nth):
        cj = torch.empty((nr, nc), device=DEV, dtype=C16)
        for r0 in range(0, nr, step):
            q = qy[r0:r0 + step, None]
            px, py, pz = (a[i][m] * qx[None, :] + b[i][m] * q for m in range(3))
            m = (px.abs() <= math.pi) & (py.abs() <= math.pi) & (pz.abs() <= math.pi)
            g = (_phase(pz[:, 0], kz, -1) @ xd).reshape(len(q), n2, n3)
            ex = px[:, None, :] * kx[None, :, None]
            t = torch.bmm(g, torch.complex(torch.cos(ex), -torch.sin(ex)))
            ey = py[:, None, :] * ky[None, :, None]
            cj[r0:r0 + step] = (t * torch.complex(torch.cos(ey), -torch.sin(ey))).sum(1) * m
        cj = _detector(cj, 1, nc // 2, (nc + 1) // 2, True)
        cj = _detector(cj, 0, nr // 2, (nr + 1) // 2, True)
        out[i] = cj.real / (nr * nc)
    return out


def _dirichlet(u, n):
    """sum over m of exp(i u r_m), r_m the n symmetric samples of [-pi, pi]."""
    q = torch.round(u / n)
    d = u - q * n
    den = torch.sin(d * (math.pi / n))
    v = torch.where(den.abs() < 1e-9, torch.full_like(d, float(n)), torch.sin(math.pi * d) / den)
    return v if n % 2 == 1 else v * (1 - 2 * torch.remainder(q, 2))


def _wrap_kernel(P, lags):
    """FFT indices of the lags -(n-1) .. n-1 on a grid of P."""
    return torch.remainder(lags, P).to(torch.long)


class _Conv2d:
    def __init__(self, n, theta, nr):
        self.n, self.P = n, 2 * n
        lag = torch.arange(-(n - 1), n, device=DEV, dtype=F8)
        k = torch.zeros((2 * n - 1, 2 * n - 1), device=DEV, dtype=F8)
        for t in theta:
            k += _dirichlet(math.cos(t) * lag[None, :] + math.sin(t) * lag[:, None], nr)
        full = torch.zeros((self.P, self.P), device=DEV, dtype=F8)
        i = _wrap_kernel(self.P, lag)
        full[i[:, None], i[None, :]] = k / nr
        self.f = torch.fft.rfft2(full)

    def __call__(self, x):
        n, P = self.n, self.P
        return torch.fft.irfft2(torch.fft.rfft2(x, s=(P, P)) * self.f, s=(P, P))[..., :n, :n]


class _Conv3d:
    def __init__(self, c, dims):
        self.dims, self.P = dims, tuple(2 * n for n in dims)
        a, b = _detector_axes(c)
        lag = [torch.arange(-(n - 1), n, device=DEV, dtype=F8) for n in dims]
        idx = [_wrap_kernel(P, v) for P, v in zip(self.P, lag)]
        same_a = bool(np.all(a == a[0]))
        full = torch.zeros(self.P, device=DEV, dtype=F8)
        ky, kx = lag[1][:, None], lag[2][None, :]
        for z in range(dims[0]):  # planes z >= 0; the others by K(-k) = K(k)
            k = torch.zeros((len(lag[1]), len(lag[2])), device=DEV, dtype=F8)
            dx = None
            for i in range(c["ntheta"]):
                if dx is None or not same_a:
                    dx = _dirichlet(a[i][0] * kx + a[i][1] * ky + a[i][2] * z, c["ncols"])
                dy = _dirichlet(b[i][0] * kx + b[i][1] * ky + b[i][2] * z, c["nrows"])
                k += dy if same_a else dx * dy
            if same_a:
                k *= dx
            k /= dims[1] * dims[2]
            full[z][idx[1][:, None], idx[2][None, :]] = k
            if z:
                full[-z][idx[1][:, None], idx[2][None, :]] = k.flip(0, 1)
        self.f = torch.fft.rfftn(full)

    def __call__(self, x):
        y = torch.fft.rfftn(x, s=self.P)
        y *= self.f
        return torch.fft.irfftn(y, s=self.P)[:self.dims[0], :self.dims[1], :self.dims[2]].contiguous()


def _cdiff(u, dim):
    v = torch.zeros_like(u)
    n = u.shape[dim]
    if n > 1:
        v.narrow(dim, 0, n - 1).add_(u.narrow(dim, 1, n - 1))
        v.narrow(dim, 1, n - 1).sub_(u.narrow(dim, 0, n - 1))
    return v * 0.5


def _exact_cg(A, y, iters):
    x = torch.zeros_like(y)
    r = y.clone()
    p = r.clone()
    rs = (r * r).sum()
    for _ in range(iters):
        ap = A(p)
        al = rs / (p * ap).sum()
        x = x + al * p
        r = r - al * ap
        rn = (r * r).sum()
        p = r + (rn / rs) * p
        rs = rn
    return x


def _exact_sb(A, y, lam, mu, outer):
    def div(v):
        return _cdiff(v[0], 2) + _cdiff(v[1], 1) + _cdiff(v[2], 0)

    def grad(u):
        return [_cdiff(u, 2), _cdiff(u, 1), _cdiff(u, 0)]

    def op(u):
        return A(u) - mu * div(grad(u))

    x = torch.zeros_like(y)
    d = [torch.zeros_like(y) for _ in range(3)]
    b = [torch.zeros_like(y) for _ in range(3)]
    for _ in range(outer):
        rhs = y - mu * div([d[i] - b[i] for i in range(3)])
        r = rhs - op(x)
        ap = op(r)
        x = x + (r * r).sum() / (r * ap).sum() * r
        g = grad(x)
        t = [g[i] + b[i] for i in range(3)]
        s = torch.sqrt(t[0] ** 2 + t[1] ** 2 + t[2] ** 2)
        f = torch.clamp(s - lam / mu, min=0) / (s + 1e-8)
        d = [f * t[i] for i in range(3)]
        b = [t[i] - d[i] for i in range(3)]
    return x


def exact(case, seed):
    c, k = case, case["kind"]
    if k == "conv2d":
        return _Conv2d(c["n"], _theta2d(c["ntheta"]), c["n"])(_slices(c["ns"], c["n"], seed).to(F8))
    if k == "forward2d":
        return _exact_forward2d(_slices(c["ns"], c["n"], seed), _theta2d(c["ntheta"]))
    if k == "backproj2d":
        th = _theta2d(c["ntheta"])
        return _exact_backproj2d(_sinograms(c["ns"], c["n"], th, seed), th, c["n"])
    if k in ("conv3d", "forward3d", "backproj3d", "sb3d"):
        dims = (c["n1"], c["n2"], c["n3"])
        if k == "conv3d":
            return _Conv3d(c, dims)(_volume(dims, seed).to(F8))
        if k == "forward3d":
            return _exact_forward3d(_volume(dims, seed), c)
        if k == "backproj3d":
            return _exact_backproj3d(_projections(c, dims, _theta3d(c["ntheta"]), seed), c, dims)
        return _exact_sb(_Conv3d(c, dims), _rhs3d(c, seed).to(F8), 0.1, 10.0, c["outer"])
    if k == "batch2d":
        out = []
        for i, (n, nth) in enumerate(_job_sizes(c)):
            th = _theta2d(nth)
            y = _exact_backproj2d(_sinograms(1, n, th, seed * 1009 + i), th, n)
            out.append(_exact_cg(_Conv2d(n, th, n), y, c["iters"]))
        return out
    if k == "mbir2d":
        th = _theta2d(c["ntheta"])
        y = _exact_backproj2d(_sinograms(c["ns"], c["n"], th, seed), th, c["n"])
        return _exact_sb(_Conv2d(c["n"], th, c["n"]), y, 0.1, 10.0, c["outer"])
    r = (c["r1"], c["r2"], c["r3"])
    dims = tuple(_padded(v) for v in r)
    pc = dict(c, nrows=_padded(c["nrows"]), ncols=_padded(c["ncols"]))
    if 8.0 * pc["ntheta"] * pc["nrows"] * pc["ncols"] * dims[1] * dims[2] > FLOP_LIMIT:
        return None
    p = _projections(c, r, _theta3d(c["ntheta"]), seed)
    full = torch.zeros((c["ntheta"], pc["nrows"], pc["ncols"]), device=DEV)
    o2, o3 = (pc["nrows"] - c["nrows"]) // 2, (pc["ncols"] - c["ncols"]) // 2
    full[:, o2:o2 + c["nrows"], o3:o3 + c["ncols"]] = p / p.max()
    x = _exact_sb(_Conv3d(pc, dims), _exact_backproj3d(full, pc, dims), 0.1, 10.0, c["outer"])
    o = [(a - b) // 2 for a, b in zip(dims, r)]
    return x[o[0]:o[0] + r[0], o[1]:o[1] + r[1], o[2]:o[2] + r[2]]
