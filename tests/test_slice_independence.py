"""The slices of a stack are independent problems: a projection or an A^T A of
one slice does not change with what lies in the slices beside it, be it values
many orders larger (whose rounding errors would cover the slice) or NaN.  Odd
row counts, where a line that carries two real rows would reach into the next
slice.  Tolerance: the rounding of FP32 transforms against the same slice
alone, 1e-6."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-6


def stacks(rng, shape, beside):
    x = rng.standard_normal(shape).astype(np.float32)
    x[0::2] = np.nan if beside == "nan" else x[0::2] * np.float32(1e12)
    return x


@pytest.mark.parametrize("beside", ["large", "nan"])
@pytest.mark.parametrize("nth,n", [(1, 64), (3, 65), (5, 113), (4, 65)])
def test_forward2d(cuda, nth, n, beside):
    import laminocam_b200 as lc
    rng = np.random.default_rng(n + nth)
    pg = lc.PolarGrid2D(rng.uniform(-3, 3, nth), n)
    x = stacks(rng, (3, n, n), beside)
    got = lc.forward2d(x, pg).cpu().numpy()[1]
    want = lc.forward2d(x[1:2], pg).cpu().numpy()[0]
    assert np.isfinite(got).all()
    assert O.rel_l2(got, want.astype(np.float64)) < TOL


@pytest.mark.parametrize("beside", ["large", "nan"])
@pytest.mark.parametrize("n", [39, 41, 65, 111, 325])  # P = 81, 81, 144, 243, 729
def test_convolution(cuda, n, beside):
    import laminocam_b200 as lc
    rng = np.random.default_rng(n)
    pg = lc.PolarGrid2D(np.arange(7) * np.pi / 7, n)
    x = stacks(rng, (3, n, n), beside)
    got = lc.PointSpreadFunction2D(pg, n, 3).convolve(x).cpu().numpy()[1]
    want = lc.PointSpreadFunction2D(pg, n, 1).convolve(x[1:2]).cpu().numpy()[0]
    assert np.isfinite(got).all()
    assert O.rel_l2(got, want.astype(np.float64)) < TOL
