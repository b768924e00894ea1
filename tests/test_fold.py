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
