"""TMC float32 normals on steep fields (values over 25 decades side by side) against the CPU oracle: within 1e-5 per
component, the bound of the float32 normals on any field.  The inner vertices' normals there follow their
parameters' last digits."""
import numpy as np
import pytest

from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(6))
def test_normals_of_steep_fields(oracle, seed):
    from tmc_gb300 import native
    rng = np.random.Generator(np.random.PCG64(seed))
    shape = (40, 45 - seed, 50)
    data = (rng.standard_normal(shape) * np.exp(8 * rng.standard_normal(shape))).astype(np.float32)
    vol = V.Volume(data, spacing=(10.0 ** rng.uniform(-3, 1), 0.1, 0.05), iso=(0.0, 0.5, -0.37)[seed % 3])
    want = oracle.tmc(vol)
    ctx = native.Context(0)
    try:
        got = ctx.tmc(vol, 0)
    finally:
        ctx.close()
    np.testing.assert_array_equal(got["t"], want["t"])
    np.testing.assert_allclose(got["n"], want["n"], rtol=0, atol=1e-5)
