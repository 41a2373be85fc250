"""The request server admits by an estimate of each request's device bytes: at the estimate's own surface density
(0.3 vertices per cell) it covers what the request takes at its peak, and is no more than half as much again.

The peak is the device memory pool's high-water mark over the request; the estimate is what the server reports as
its peak of admitted bytes after one request."""
import ctypes

import numpy as np
import pytest

from tmc_gb300 import native
from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu

USED_CURRENT, USED_HIGH = 7, 8  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT / _HIGH
FULL = native.OUT_POS_F64 | native.OUT_TRIANGLES | native.OUT_HALFEDGES


class Pool:
    def __init__(self):
        self.cuda = ctypes.CDLL("libcuda.so.1")
        self.pool = ctypes.c_void_p()
        assert self.cuda.cuDeviceGetDefaultMemPool(ctypes.byref(self.pool), 0) == 0

    def used(self, what):
        v = ctypes.c_uint64()
        assert self.cuda.cuMemPoolGetAttribute(self.pool, what, ctypes.byref(v)) == 0
        return v.value

    def restart(self):
        v = ctypes.c_uint64(0)
        assert self.cuda.cuMemPoolSetAttribute(self.pool, USED_HIGH, ctypes.byref(v)) == 0
        return self.used(USED_CURRENT)


@pytest.fixture(scope="module")
def vol():
    # 0.29 vertices per cell
    return V.Volume(V.periodic(161, 160, 159, 29.5), spacing=(0.01, 0.01, 0.01), iso=0.05)


@pytest.mark.parametrize("on_device", [True, False])
@pytest.mark.parametrize("algo,flags", [
    (native.ALGO_TMC, 0), (native.ALGO_TMC, native.OUT_POS_F64), (native.ALGO_TMC, native.OUT_HALFEDGES),
    (native.ALGO_DMC, 0), (native.ALGO_DMC, native.OUT_POS_F64 | native.OUT_LOCAL), (native.ALGO_DMC, native.OUT_TRIANGLES),
    (native.ALGO_DMC, native.OUT_HALFEDGES), (native.ALGO_DMC, native.DMC_SIMPLIFY), (native.ALGO_DMC, native.DMC_SIMPLIFY | FULL),
])
def test_estimate_covers_the_peak(vol, algo, flags, on_device):
    import torch
    field = torch.from_numpy(np.ascontiguousarray(vol.data)).cuda() if on_device else None
    torch.cuda.synchronize()
    v = native.make_volume(vol, field.data_ptr(), on_device=True) if on_device else native.make_volume(vol)
    srv = native.Server(0, workers=1)
    try:
        pool = Pool()
        before = pool.restart()
        m = srv.wait_raw(srv.submit(v, vol.iso, algo, flags))
        peak = pool.used(USED_HIGH) - before
        cells = (vol.dims[0] - 1) * (vol.dims[1] - 1) * (vol.dims[2] - 1)
        vertices, estimate = m.nr_v, srv.stats()[4]
        srv.release(m)
    finally:
        srv.close()
    print(f"{vertices / cells:.3f} vertices per cell, peak {peak / cells:.1f} B per cell, estimate {estimate / cells:.1f}")
    assert vertices <= 0.3 * cells
    assert peak <= estimate <= 1.5 * peak
