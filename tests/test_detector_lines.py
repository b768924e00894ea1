"""Detector transforms on the Bluestein line kernels: real output (two lines to
one), real input, Hermitian halves (odd sides), even sides, and lengths whose
convolution length would be a power of three (37 .. 41, 109 .. 122, 325 .. 365,
1025), through the projections that use them, against the exact sums.
Tolerance: the NUFFT tolerance 1e-6 and FP32 transforms; 1e-5 is the bound of
the projection parity tests."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.mark.parametrize("n", [38, 41, 57, 58, 64, 65, 113, 122, 128, 363, 365, 1025])
def test_2d_lines(cuda, n):
    import laminocam_b200 as lc
    rng = np.random.default_rng(n)
    theta = np.array([0.1, 1.3, 2.9])
    pg = lc.PolarGrid2D(theta, n)
    x = rng.standard_normal((1, n, n)).astype(np.float32)
    assert O.rel_l2(lc.forward2d(x, pg).cpu().numpy(), O.forward2d(x, theta, n)) < TOL
    y = rng.standard_normal((1, 3, n)).astype(np.float32)
    assert O.rel_l2(lc.backproj2d(y, pg, (1, n, n)).cpu().numpy(), O.backproj2d(y, theta, (1, n, n))) < TOL


@pytest.mark.parametrize("rows,cols", [(57, 61), (57, 64), (64, 57), (64, 66), (113, 121), (41, 60), (59, 14), (363, 57)])
def test_3d_lines(cuda, rows, cols):
    import laminocam_b200 as lc
    rng = np.random.default_rng(rows + cols)
    nth, dims = 3, (3, 8, 9)
    theta, gamma, beta = rng.uniform(-3, 3, nth), np.full(nth, -0.52), np.full(nth, 0.04)
    pg = lc.PolarGrid(theta, gamma, beta, rows, cols)
    g = O.Grid3D(theta, gamma, beta, rows, cols)
    x = rng.standard_normal(dims).astype(np.float32)
    assert O.rel_l2(lc.forward(x, pg).cpu().numpy(), O.forward3d(x, g)) < TOL
    y = rng.standard_normal((nth, rows, cols)).astype(np.float32)
    assert O.rel_l2(lc.backproj(y, pg, dims).cpu().numpy(), O.backproj3d(y, g, dims)) < TOL
