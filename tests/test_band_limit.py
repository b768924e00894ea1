"""The forward projection on the band limit |q| <= pi.  At a tilt of 30 degrees
and angles of 30 degrees from the axes, lattice points of equal odd sides lie
exactly on the limit (2 m + 3 l = 2 n); rounding decides for each of them on its
own, and differently for some opposite pairs.  The projection is the real part
of the inverse transform, so a pair of which one member is inside counts half.

The half path (odd sides on the register plans) has to treat every such pair as
the path with all rows does, and both as the exact sums with the mask of the
pair averaged.  Tolerance: 1e-5, as the projection parity tests; one pair left
at the wrong weight changes its projection by about 1e-2."""
import os
import subprocess
import sys
import tempfile

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SIDES = [61, 63, 113]
ANGLES = np.deg2rad([30.0, 150.0, 210.0, 330.0, 47.0])


def grids(n):
    nth = len(ANGLES)
    return ANGLES, np.full(nth, -np.pi / 6), np.zeros(nth)


def volume(n):
    return np.random.default_rng(n).standard_normal((3, 10, 9)).astype(np.float32)


def spectrum(proj):
    """Lattice values whose Hermitian part the projection holds."""
    n = proj.shape[1]
    c = proj.astype(np.complex128)
    c = np.roll(np.roll(c, (n + 1) // 2, 1), (n + 1) // 2, 2)
    c = np.fft.fft2(c, axes=(1, 2))
    return np.roll(np.roll(c, n // 2, 1), n // 2, 2)


def projection(C):
    n = C.shape[1]
    c = O.fftshift_axis(O.fftshift_axis(C, 1), 2)
    c = np.fft.ifft2(c, axes=(1, 2))
    return O.ifftshift_axis(O.ifftshift_axis(c, 1), 2).real


def test_forward_on_the_band_limit(cuda):
    import laminocam_b200 as lc
    with tempfile.TemporaryDirectory() as td:
        out = os.path.join(td, "all_rows.npz")
        code = ("import numpy as np, laminocam_b200 as lc, test_band_limit as t\n"
                "r = {}\n"
                "for n in t.SIDES:\n"
                "    r[str(n)] = lc.forward(t.volume(n), lc.PolarGrid(*t.grids(n), n, n)).cpu().numpy()\n"
                f"np.savez({out!r}, **r)\n")
        env = dict(os.environ, LC_LINE_KERNELS="0",
                   PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests"), os.environ.get("PYTHONPATH", "")]))
        subprocess.run([sys.executable, "-c", code], check=True, timeout=300, env=env, cwd=ROOT)
        every = {int(k): v for k, v in np.load(out).items()}
    split = 0
    for n in SIDES:
        x, y, z, w = O.polar_grid3d(*grids(n), n, n)
        vol = volume(n)
        C = O.nudft2_3d(vol.astype(np.complex128), x, y, z, -1).reshape(x.shape)
        edge = np.zeros(x.shape, bool)
        for c in (x, y, z):
            edge |= np.abs(np.abs(c) - np.pi) < 1e-12
        edge |= edge[:, ::-1, ::-1]
        assert edge.any()
        # weight of each pair on the limit, from the path that keeps every row
        got = spectrum(every[n])
        wt = (w + w[:, ::-1, ::-1]) / 2
        wt[edge] = np.rint(2 * (got[edge] / C[edge]).real) / 2
        assert set(np.unique(wt[edge])) <= {0.0, 0.5, 1.0}
        split += int((wt[edge] == 0.5).sum())
        want = projection(wt * C)
        res = lc.forward(vol, lc.PolarGrid(*grids(n), n, n)).cpu().numpy()
        assert O.rel_l2(every[n], want) < 1e-5, n
        assert O.rel_l2(res, want) < 1e-5, n
    assert split > 0  # some pairs do disagree
