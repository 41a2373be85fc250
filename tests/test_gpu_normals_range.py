"""Float32 normals of both algorithms on fields whose gradients' squares leave the float range, against the CPU
oracle's float64 normals: within 1e-5 per component, the bound of the float32 normals at any size."""
import numpy as np
import pytest

from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["dmc", "tmc"])
@pytest.mark.parametrize("scale", [1e-30, 1e-24, 1e-21, 1e-18, 1e-12, 1e12, 1e17, 1e20, 1e28, 1e36])
def test_normals_over_the_float_range(oracle, scale, algo):
    from tmc_gb300 import native
    f = V.blobs_volume(31, seed=4)
    vol = V.Volume((f.data.astype(np.float64) * scale).astype(np.float32), origin=f.origin, spacing=f.spacing, iso=0.5 * scale)
    want = oracle.dmc_front(vol) if algo == "dmc" else oracle.tmc(vol)
    ctx = native.Context(0)
    try:
        got = ctx.dmc(vol, 0) if algo == "dmc" else ctx.tmc(vol, 0)
    finally:
        ctx.close()
    assert want["n"].size > 0
    assert got["n"].shape == want["n"].shape
    np.testing.assert_allclose(got["n"], want["n"], rtol=0, atol=1e-5)
