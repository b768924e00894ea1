"""The fixed-point sums of the spreading at the ends of their range.

Crowded bins: an impulse at the detector's centre has a flat spectrum, so many
angles put values of one sign on the cells around the origin, where a 32-bit
tile sum comes closest to its bound; every kernel width, angles that share
their points and angles that do not.  A sum past the bound would wrap by 2^32
steps, an error of the order of the largest cell.  Tolerance: the NUFFT's, held
to 1e-5 from 1e-6 down and to ten times the requested one above.

A full cell: 1020 angles 1e-9 apart and a lattice of two points put 1020 equal
values on one cell centre, in one subproblem.  With weight 1 there and the
weight bound 0.1 % per axis above it, the cell's sum reaches 0.996 of 2^31.

Scales: the result is linear in the input, by powers of two exactly so, down to
values near the smallest normal float."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tol", [1e-3, 1e-4, 1e-5, 1e-6, 1e-8, 1e-11])  # widths 4, 5, 6, 7, 9, 12
@pytest.mark.parametrize("turn", [1.0, 2.0])  # angles over half a turn, and over a full one (pairs coincide)
def test_crowded_2d(cuda, tol, turn):
    import laminocam_b200 as lc
    n, nth = 48, 720
    theta = np.arange(nth) * (turn * np.pi / nth)
    y = np.zeros((1, nth, n), np.float32)
    y[:, :, n // 2] = 1.0
    got = lc.backproj2d(y, lc.PolarGrid2D(theta, n), (1, n, n), tol=tol).cpu().numpy()
    assert O.rel_l2(got, O.backproj2d(y, theta, (1, n, n))) < max(1e-5, 10 * tol)


@pytest.mark.parametrize("tol", [1e-3, 1e-6, 1e-11])
@pytest.mark.parametrize("beta", [0.0, 0.1])  # the pairs of a full turn coincide, or not
def test_crowded_3d(cuda, tol, beta):
    import laminocam_b200 as lc
    rows, cols, nth, dims = 24, 25, 360, (5, 12, 13)
    theta, gamma, bt = np.arange(nth) * (2 * np.pi / nth), np.full(nth, -0.6), np.full(nth, beta)
    y = np.zeros((nth, rows, cols), np.float32)
    y[:, rows // 2, cols // 2] = 1.0
    got = lc.backproj(y, lc.PolarGrid(theta, gamma, bt, rows, cols), dims, tol=tol).cpu().numpy()
    want = O.backproj3d(y, O.Grid3D(theta, gamma, bt, rows, cols), dims)
    assert O.rel_l2(got, want) < max(1e-5, 10 * tol)


@pytest.mark.parametrize("tol", [1e-3, 1e-5, 1e-6, 1e-11])
def test_full_cell_2d(cuda, tol):
    import laminocam_b200 as lc
    theta = np.arange(1020) * 1e-9
    y = np.ones((1, 1020, 2), np.float32)
    got = lc.backproj2d(y, lc.PolarGrid2D(theta, 2), (1, 2, 2), tol=tol).cpu().numpy()
    assert O.rel_l2(got, O.backproj2d(y, theta, (1, 2, 2))) < max(1e-5, 10 * tol)


@pytest.mark.parametrize("tol", [1e-3, 1e-5, 1e-6, 1e-11])
def test_full_cell_3d(cuda, tol):
    import laminocam_b200 as lc
    gamma, zero, dims = np.arange(1020) * 1e-9, np.zeros(1020), (3, 3, 2)
    y = np.ones((1020, 1, 2), np.float32)
    got = lc.backproj(y, lc.PolarGrid(zero, gamma, zero, 1, 2), dims, tol=tol).cpu().numpy()
    assert O.rel_l2(got, O.backproj3d(y, O.Grid3D(zero, gamma, zero, 1, 2), dims)) < max(1e-5, 10 * tol)


@pytest.mark.parametrize("e", [60, 0, -60, -90, -104, -108, -112, -116])
def test_scale(cuda, e):
    import laminocam_b200 as lc
    n, nth = 33, 12
    pg = lc.PolarGrid2D(np.arange(nth) * np.pi / nth, n)
    y = np.random.default_rng(3).standard_normal((1, nth, n)).astype(np.float32)
    want = lc.backproj2d(y, pg, (1, n, n)).cpu().numpy().astype(np.float64)
    got = lc.backproj2d((y.astype(np.float64) * 2.0 ** e).astype(np.float32), pg, (1, n, n)).cpu().numpy()
    # the sums are whole numbers of steps of at least 2^-126
    assert O.rel_l2(got.astype(np.float64) * 2.0 ** -e, want) < max(1e-6, 2.0 ** (-126 - e) * 100)
