"""The server's footprint estimate of a job bounds what the job takes from the
device: the high-water mark of the allocation pool while the job runs alone.
Thin volumes with many projections, where the point data and the fine grid of
the backprojection (whose lengths go from 2187 to the next even 2304 cells)
outweigh everything else, ordinary volumes, and slices."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

USED_CURRENT, USED_HIGH = 7, 8  # CUmemPool_attribute


def pool(attr, reset=False):
    cu = ctypes.CDLL("libcuda.so.1")
    p, v = ctypes.c_void_p(), ctypes.c_uint64(0)
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(p), 0) == 0
    f = cu.cuMemPoolSetAttribute if reset else cu.cuMemPoolGetAttribute
    assert f(p, attr, ctypes.byref(v)) == 0
    return v.value


def run(lc, submit):
    with lc.Server(workers=1) as sv:
        before = pool(USED_CURRENT)
        pool(USED_HIGH, reset=True)
        r = sv.wait(submit(sv), 300.0)
        return r.device_bytes, pool(USED_HIGH) - before


@pytest.mark.parametrize("dims,nth,rows,beta", [((1, 1081, 1081), 220, 1081, 0.0), ((1, 1081, 1081), 220, 1081, 0.1),
                                                ((1, 361, 361), 1200, 361, 0.1), ((29, 181, 181), 60, 181, 0.0)])
def test_volume_job(cuda, dims, nth, rows, beta):
    import laminocam_b200 as lc
    projs = np.random.default_rng(0).random((nth, rows, dims[2]), dtype=np.float32)
    theta = np.arange(nth) * 2 * np.pi / nth
    p = lc.ReconParams(regularizer="unconstrained", recon_dims=dims, max_iters=1, tol=0, xtol=0, pad_factor=1.0)
    est, used = run(lc, lambda sv: sv.submit3d([lc.Dataset(projs, theta, -0.5, beta)], p))
    assert used <= est, (used, est)


@pytest.mark.parametrize("n,nth,ns", [(1081, 360, 1), (1081, 360, 5), (255, 1800, 9)])
def test_slice_job(cuda, n, nth, ns):
    import laminocam_b200 as lc
    sino = np.random.default_rng(0).random((ns, nth, n), dtype=np.float32)
    p = lc.ReconParams(regularizer="split_bregman", recon_dims=(ns, n, n), max_iters=1, tol=0, xtol=0)
    est, used = run(lc, lambda sv: sv.submit2d(sino, np.arange(nth) * 2 * np.pi / nth, p))
    assert used <= est, (used, est)
