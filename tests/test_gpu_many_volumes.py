"""Batches of more volumes than a CUDA grid has rows (65,535): each volume's mesh is the one it has alone."""
import numpy as np
import pytest

from tmc_gb300 import native
from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu

KINDS = 61  # fields that the volumes take in turn
SIDE = 3


def _host(ptr, shape, kind):
    import torch

    class Array:
        __cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": kind, "version": 2}

    return torch.as_tensor(Array(), device="cuda").cpu().numpy()


@pytest.mark.parametrize("algo", [native.ALGO_DMC, native.ALGO_TMC])
@pytest.mark.parametrize("count", [65535, 65536, 70000])
def test_batch_of_many_volumes(algo, count):
    import torch
    data = np.random.Generator(np.random.PCG64(5)).standard_normal((KINDS, SIDE, SIDE, SIDE)).astype(np.float32)
    fields = torch.from_numpy(data).cuda()
    torch.cuda.synchronize()
    vols = [V.Volume(d, spacing=(1.0, 1.0, 1.0), iso=0.1) for d in data]
    ctx = native.Context(0)
    try:
        alone = [ctx.dmc(v) if algo == native.ALGO_DMC else ctx.tmc(v) for v in vols]
        structs = [native.make_volume(v, f.data_ptr(), on_device=True) for v, f in zip(vols, fields)]
        got = ctx.batch_raw([structs[q % KINDS] for q in range(count)], [0.1] * count, [algo] * count, [0] * count)
        ctx.synchronize()
        faces = "quads" if algo == native.ALGO_DMC else "tris"
        width, key = (4, "q") if algo == native.ALGO_DMC else (3, "t")
        for q, m in enumerate(got):
            want = alone[q % KINDS]
            assert (m.nr_v, m.nr_q + m.nr_t) == (want["v"].size // 3, want[key].size // width), q
        for q in list(range(0, 3 * KINDS)) + list(range(count - 3 * KINDS, count)):
            want, m = alone[q % KINDS], got[q]
            if want[key].size:
                np.testing.assert_array_equal(_host(m.v, (m.nr_v * 3,), "<f4"), want["v"])
                np.testing.assert_array_equal(_host(getattr(m, faces), (want[key].size,), "<i4"), want[key])
        for m in got:
            ctx.free(m)
    finally:
        ctx.close()
