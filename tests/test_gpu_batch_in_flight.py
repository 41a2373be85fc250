"""A batch with device results returns while its last kernels run; once one of its meshes is freed, they are done:
the caller may then free or rewrite the fields."""
import numpy as np
import pytest

from tmc_gb300 import native
from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", [native.ALGO_DMC, native.ALGO_TMC])
@pytest.mark.parametrize("first", [0, 1])
def test_the_batch_is_done_once_a_mesh_is_freed(algo, first):
    import torch
    g = torch.Generator(device="cuda").manual_seed(3)
    # white noise: milliseconds of emission after the call has returned
    fields = [torch.randn((300, 300, 300), generator=g, device="cuda") for _ in range(2)]
    vols = []
    for f in fields:
        v = native.make_volume(V.Volume(np.zeros((2, 2, 2), np.float32), spacing=(1.0, 1.0, 1.0)), f.data_ptr(), on_device=True)
        v.nx, v.ny, v.nz = f.shape[2], f.shape[1], f.shape[0]
        vols.append(v)
    torch.cuda.synchronize()
    ctx = native.Context(0)
    try:
        stream = torch.cuda.ExternalStream(ctx.stream)
        for _ in range(3):
            got = ctx.batch_raw(vols, [0.0] * 2, [algo] * 2, [0] * 2)
            ctx.free(got[first])
            assert stream.query()
            ctx.free(got[1 - first])
            torch.cuda.synchronize()
    finally:
        ctx.close()
