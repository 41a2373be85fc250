"""Device results of requests that the server batches are complete when their tickets are: read at once, on a
stream that knows nothing of the server's, they equal the meshes of the same requests extracted alone."""
import numpy as np
import pytest

from tmc_gb300 import native
from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu

SIDE = 260


def _array(ptr, count, kind):
    import torch

    class Array:
        __cuda_array_interface__ = {"data": (ptr, False), "shape": (count,), "typestr": kind, "version": 2}

    return torch.as_tensor(Array(), device="cuda")


def _copies(m):
    faces = _array(m.quads, 4 * m.nr_q, "<i4") if m.nr_q else _array(m.tris, 3 * m.nr_t, "<i4")
    return [x.clone() for x in (_array(m.v, 3 * m.nr_v, "<f4"), _array(m.n, 3 * m.nr_v, "<f4"), faces)]


@pytest.mark.parametrize("algo", [native.ALGO_DMC, native.ALGO_TMC])
def test_batched_device_results_are_complete(algo):
    import torch
    g = torch.Generator(device="cuda").manual_seed(5)
    # white noise: milliseconds of emission
    fields = [torch.randn((SIDE, SIDE, SIDE), generator=g, device="cuda") for _ in range(4)]
    vols = []
    for f in fields:
        v = native.make_volume(V.Volume(np.zeros((2, 2, 2), np.float32), spacing=(1.0, 1.0, 1.0)), f.data_ptr(), on_device=True)
        v.nx = v.ny = v.nz = SIDE
        vols.append(v)
    torch.cuda.synchronize()
    ctx = native.Context(0)
    want = []
    for v in vols:
        m = ctx.dmc_raw(v, 0.0, 0) if algo == native.ALGO_DMC else ctx.tmc_raw(v, 0.0, 0)
        want.append(_copies(m))
        torch.cuda.synchronize()
        ctx.free(m)
    ctx.close()
    srv = native.Server(0, workers=1, max_batch_cells=1 << 30)
    try:
        # the first request keeps the worker busy while the others are queued, which it takes as one batch
        tickets = [srv.submit(v, 0.0, algo, 0) for v in vols]
        for q in (1, 2, 3, 0):
            m = srv.wait_raw(tickets[q])
            for got, w in zip(_copies(m), want[q]):
                assert torch.equal(got, w), q
            srv.release(m)
        assert srv.stats()[5] >= 2  # largest batch
    finally:
        srv.close()
