"""The exact pass of the quad split over a list of several rounds per block, against the CPU oracle.

A white-noise volume has 1.4 quads per cell; with spacings of 1, 1e-3 and 1e-6 they are so thin that all of
them are listed for the exact pass, four times what its grid takes in one round.  The origin sets how many of a
round's quads a block keeps for its float64 step: about a fifth (carried from round to round), two thirds (a
full step every other round), all.  The split is a decision of the reference's own rounding: equal, without a
tolerance."""
import numpy as np
import pytest

from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("origin", [0.0, 3e3, 3e5])
def test_split_over_several_rounds(oracle, origin):
    import torch

    from tmc_gb300 import native
    n = 100
    data = np.random.Generator(np.random.PCG64(11)).standard_normal((n, n - 1, n - 3)).astype(np.float32)
    vol = V.Volume(data, spacing=(1.0, 1e-3, 1e-6), origin=(origin, -1.5 * origin, 0.5 * origin), iso=0.0)
    ctx = native.Context(0)
    try:
        got = ctx.dmc(vol, native.OUT_TRIANGLES)
    finally:
        ctx.close()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert got["q"].size // 4 > 3 * (8 * sms) * 256
    want = oracle.dmc(vol, 0)
    np.testing.assert_array_equal(got["q"], want["q"])
    np.testing.assert_array_equal(got["t"], want["t"])
