"""DMC topology of fields whose values' products leave the float range, with an isovalue that is not zero, against
the CPU oracle: the asymptotic decider has to compare as float64 does.  Equal, without a tolerance."""
import numpy as np
import pytest

from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("part", [0.1, -0.37])
@pytest.mark.parametrize("scale", [1e-38, 1e-30, 1e-22, 1e-18, 1e-15, 1e-12, 1e12, 1e18, 1e22, 1e30, 1e37])
def test_topology_over_the_float_range(oracle, scale, part):
    from tmc_gb300 import native
    f = np.random.Generator(np.random.PCG64(3)).standard_normal((21, 22, 23)).astype(np.float32)
    data = (f.astype(np.float64) * scale).astype(np.float32)
    assert np.isfinite(data).all()
    vol = V.Volume(data, spacing=(0.1, 0.07, 0.13), iso=float(np.float32(part * scale)) * (1 + 2.0 ** -30))
    want = oracle.dmc_front(vol)
    ctx = native.Context(0)
    try:
        got = ctx.dmc(vol, native.OUT_POS_F64 | native.OUT_LOCAL)
    finally:
        ctx.close()
    for key, ref in (("q", want["q"]), ("vcell", want["vcell"]), ("vuvw", want["vuvw"]), ("v64", want["v"])):
        np.testing.assert_array_equal(got[key], ref)
