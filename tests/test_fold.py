"""The NUFFT plans handle one of each pair of opposite lattice points: both
parities of every lattice side (an odd lattice has a self-paired centre, an
even one gives values that are not Hermitian), the band limit on either member
of a pair, shifts and several volumes, against the exact non-uniform sums.

Tolerance: 1e-5 on the relative 2-norm, the bound of the parity tests, where
the sums do not cancel.  Of a single mode (n = 1: three values that cancel to
a twentieth of their size) the NUFFT tolerance bounds the error by 1e-6 of the
sum of the values' magnitudes, which is what that size is held to."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nth,ns", [(1, 3, 1), (2, 5, 1), (3, 1, 2), (16, 7, 1), (17, 7, 9), (40, 1, 1), (33, 64, 3)])
def test_2d(cuda, n, nth, ns):
    import laminocam_b200 as lc
    rng = np.random.default_rng(n)
    theta = rng.uniform(-4, 4, nth)
    pg = lc.PolarGrid2D(theta, n)
    y = rng.standard_normal((ns, nth, n)).astype(np.float32)
    got = lc.backproj2d(y, pg, (ns, n, n)).cpu().numpy()
    want = O.backproj2d(y, theta, (ns, n, n))
    if n == 1:
        assert np.abs(got - want).max() < 1e-6 * np.abs(y).sum()
    else:
        assert O.rel_l2(got, want) < 1e-5
    x = rng.standard_normal((ns, n, n)).astype(np.float32)
    assert O.rel_l2(lc.forward2d(x, pg).cpu().numpy(), O.forward2d(x, theta, n)) < 1e-5
    assert O.rel_l2(lc.sysmat2d(x, pg).cpu().numpy(), O.sysmat2d_nufft(x.astype(np.float64), theta, n)) < 1e-5


@pytest.mark.parametrize("rows,cols", [(1, 1), (1, 8), (9, 1), (8, 8), (8, 11), (11, 8), (11, 13)])
@pytest.mark.parametrize("shifted", [False, True])
def test_3d(cuda, rows, cols, shifted):
    import laminocam_b200 as lc
    rng = np.random.default_rng(rows * 100 + cols)
    nth, dims = 5, (5, 9, 8)
    theta, gamma, beta = rng.uniform(-3, 3, nth), rng.uniform(-1, 1, nth), rng.uniform(-0.3, 0.3, nth)
    sh = rng.uniform(-2, 2, (nth, 2)).astype(np.float32) if shifted else None
    pg = lc.PolarGrid(theta, gamma, beta, rows, cols, sh)
    g = O.Grid3D(theta, gamma, beta, rows, cols)
    y = rng.standard_normal((nth, rows, cols)).astype(np.float32)
    got = lc.backproj(y, pg, dims, shifts=shifted).cpu().numpy()
    assert O.rel_l2(got, O.backproj3d(y, g, dims, sh)) < 1e-5
    x = rng.standard_normal(dims).astype(np.float32)
    assert O.rel_l2(lc.forward(x, pg).cpu().numpy(), O.forward3d(x, g)) < 1e-5
    assert O.rel_l2(lc.sysmat(x, pg).cpu().numpy(), O.sysmat3d_nufft(x.astype(np.float64), g)) < 1e-5


# Angles whose lattices coincide share one set of points: theta and theta + 180
# degrees (opposite radii in 2D, mirrored rows in 3D without a second tilt) and
# repeated angles, in any order, each with its own shift.  Angle counts leave
# representatives with one, two and three members.
@pytest.mark.parametrize("n", [12, 17])
def test_2d_coinciding_angles(cuda, n):
    import laminocam_b200 as lc
    rng = np.random.default_rng(n)
    t = rng.uniform(-3, 3, 4)
    theta = np.concatenate([t, [t[0]], t[:3] + np.pi, [t[1] - np.pi]])
    pg = lc.PolarGrid2D(theta, n)
    y = rng.standard_normal((2, len(theta), n)).astype(np.float32)
    assert O.rel_l2(lc.backproj2d(y, pg, (2, n, n)).cpu().numpy(), O.backproj2d(y, theta, (2, n, n))) < 1e-5
    x = rng.standard_normal((2, n, n)).astype(np.float32)
    assert O.rel_l2(lc.forward2d(x, pg).cpu().numpy(), O.forward2d(x, theta, n)) < 1e-5


# 2D angles share points only where that saves two fifths of them: either side
# of the line, one coinciding pair, a full turn, both parities, and more slices
# than one chunk of the shared-memory tiles holds (eight).
@pytest.mark.parametrize("nth,saved", [(41, 1), (41, 16), (41, 17), (40, 20)])
@pytest.mark.parametrize("n,ns", [(20, 1), (21, 9), (20, 17)])
def test_2d_share_of_coinciding_angles(cuda, nth, saved, n, ns):
    import laminocam_b200 as lc
    rng = np.random.default_rng(100 * nth + saved + n)
    theta = rng.permutation(np.linspace(0.0, np.pi, nth - saved, endpoint=False))
    theta = np.concatenate([theta, theta[:saved] + np.pi * rng.integers(-1, 2, saved)])
    pg = lc.PolarGrid2D(theta, n)
    y = rng.standard_normal((ns, nth, n)).astype(np.float32)
    x = rng.standard_normal((ns, n, n)).astype(np.float32)
    assert O.rel_l2(lc.backproj2d(y, pg, (ns, n, n)).cpu().numpy(), O.backproj2d(y, theta, (ns, n, n))) < 1e-5
    assert O.rel_l2(lc.forward2d(x, pg).cpu().numpy(), O.forward2d(x, theta, n)) < 1e-5


@pytest.mark.parametrize("rows,cols", [(8, 9), (9, 8), (9, 11), (8, 8), (57, 61)])
@pytest.mark.parametrize("shifted", [False, True])
@pytest.mark.parametrize("beta", [0.0, 0.2])
def test_3d_coinciding_angles(cuda, rows, cols, shifted, beta):
    import laminocam_b200 as lc
    rng = np.random.default_rng(rows * 100 + cols)
    dims = (5, 9, 8)
    t = np.array([0.0, 0.7, np.pi / 2])
    theta = np.concatenate([t, t[::-1] + np.pi, [0.7], [2.9]])
    nth = len(theta)
    gamma, bt = np.full(nth, -0.61), np.full(nth, beta)
    sh = rng.uniform(-2, 2, (nth, 2)).astype(np.float32) if shifted else None
    pg = lc.PolarGrid(theta, gamma, bt, rows, cols, sh)
    g = O.Grid3D(theta, gamma, bt, rows, cols)
    y = rng.standard_normal((nth, rows, cols)).astype(np.float32)
    assert O.rel_l2(lc.backproj(y, pg, dims, shifts=shifted).cpu().numpy(), O.backproj3d(y, g, dims, sh)) < 1e-5
    x = rng.standard_normal(dims).astype(np.float32)
    assert O.rel_l2(lc.forward(x, pg).cpu().numpy(), O.forward3d(x, g)) < 1e-5
