"""NUFFT passes on the register plans: a size for every half length M of an even
fine grid (n = M, or M - 1 for the other parity), so that modes fill their half
exactly or leave a gap, with the kept window of rows (2D) and along both
in-plane axes (3D), against the exact sums.  Tolerance: as the projection
parity tests (NUFFT tolerance 1e-6, FP32 transforms)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

PLANS = [64, 72, 81, 96, 108, 128, 144, 162, 192, 216, 243, 256, 288, 324, 384, 432, 486, 512, 576, 648, 729, 768,
         864, 972, 1024, 1152, 1296]


@pytest.mark.parametrize("n", [m - (i % 2) for i, m in enumerate(PLANS)])
def test_2d_plans(cuda, n):
    import laminocam_b200 as lc
    rng = np.random.default_rng(n)
    theta = np.array([0.2, 1.9])
    pg = lc.PolarGrid2D(theta, n)
    x = rng.standard_normal((1, n, n)).astype(np.float32)
    assert O.rel_l2(lc.forward2d(x, pg).cpu().numpy(), O.forward2d(x, theta, n)) < 1e-5
    y = rng.standard_normal((1, 2, n)).astype(np.float32)
    assert O.rel_l2(lc.backproj2d(y, pg, (1, n, n)).cpu().numpy(), O.backproj2d(y, theta, (1, n, n))) < 1e-5


@pytest.mark.parametrize("dims", [(3, 64, 72), (4, 63, 81), (3, 80, 97), (66, 64, 64)])
def test_3d_plans(cuda, dims):
    import laminocam_b200 as lc
    rng = np.random.default_rng(dims[2])
    theta, gamma, beta = np.array([0.3, 2.2]), np.full(2, -0.5), np.zeros(2)
    pg = lc.PolarGrid(theta, gamma, beta, 13, 18)
    g = O.Grid3D(theta, gamma, beta, 13, 18)
    x = rng.standard_normal(dims).astype(np.float32)
    assert O.rel_l2(lc.forward(x, pg).cpu().numpy(), O.forward3d(x, g)) < 1e-5
    y = rng.standard_normal((2, 13, 18)).astype(np.float32)
    assert O.rel_l2(lc.backproj(y, pg, dims).cpu().numpy(), O.backproj3d(y, g, dims)) < 1e-5
