"""DMC float32 positions on grids whose spacing lies near the lower end of the float range: the roundings of the
oracle's float64 positions, without a tolerance."""
import numpy as np
import pytest

from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing", [(1e-20, 3e-24, 7e-25), (1e-30, 3e-31, 2e-32), (1e-34, 3e-36, 2e-35), (1e-38, 3e-38, 2e-39),
                                     (1e-41, 3e-43, 1e-45), (1.0, 1e-38, 1e-300)])
@pytest.mark.parametrize("origin", [0.0, 1e-33, 1.0])
def test_positions_of_fine_grids(oracle, spacing, origin):
    from tmc_gb300 import native
    vol = V.Volume(V.small_noise_volume(37, seed=4).data, spacing=spacing, origin=(origin, -origin, 2 * origin), iso=0.01)
    want = oracle.dmc_front(vol)
    ctx = native.Context(0)
    try:
        got = ctx.dmc(vol, 0)
    finally:
        ctx.close()
    np.testing.assert_array_equal(got["q"], want["q"])
    np.testing.assert_array_equal(got["v"], want["v"].astype(np.float32))
