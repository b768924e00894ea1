"""Toeplitz applies whose padded row length is a power of three (81, 243, 729):
the x passes take real rows two to a complex line.  Row counts leave the last
line with one row and the last CTA with one line.  Against the oracle's FP64
FFT convolution with the device's own FP64 kernel, at the tolerance of the other
Toeplitz parity tests."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.mark.parametrize("n,P", [(38, 81), (41, 81), (109, 243), (122, 243), (325, 729), (365, 729)])
@pytest.mark.parametrize("ns", [1, 2, 3])
def test_odd_rows_2d(cuda, n, P, ns):
    import laminocam_b200 as lc
    rng = np.random.default_rng(n + ns)
    psf = lc.PointSpreadFunction2D(lc.PolarGrid2D(np.arange(9) * np.pi / 9, n), n, ns)
    assert psf.P[2] == P
    x = rng.standard_normal((ns, n, n)).astype(np.float32)
    K = psf.kernel()
    want = O.convolve2d(x, O.PSF2D(P, K, np.fft.rfft2(K)))
    assert O.rel_l2(psf.convolve(x).cpu().numpy().astype(np.float64), want) < TOL


def test_odd_rows_tilted_3d(cuda):
    import laminocam_b200 as lc
    rng = np.random.default_rng(5)
    dims = (5, 37, 115)
    pg = lc.PolarGrid(np.arange(7) * 2 * np.pi / 7, -0.5, 0.05, 37, 115)
    psf = lc.PointSpreadFunction(pg, dims)
    assert psf.P[2] == 243
    x = rng.standard_normal(dims).astype(np.float32)
    K = psf.kernel()
    want = O.convolve3d(x, O.PSF3D(tuple(psf.P), K, np.fft.rfftn(K)))
    assert O.rel_l2(psf.convolve(x).cpu().numpy().astype(np.float64), want) < TOL
