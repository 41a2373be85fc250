"""The quad -> triangle split where float positions leave it in doubt, against the CPU oracle.

A far origin, a fine spacing or a flat surface makes the float positions coarse beside the cells, so the
exact pass decides most quads, in whole and in partly filled blocks; symmetric fields give splits that are
equal up to rounding.  The split is a decision of the reference's own rounding: it is equal, without a
tolerance."""
import numpy as np
import pytest

from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu


def _cases():
    blobs = V.blobs_volume(24, seed=6).data
    noise = V.small_noise_volume(33, seed=9).data
    saw = (np.indices((9, 17, 17)).sum(0) % 3).astype(np.float32)
    return {
        "far": V.Volume(noise, spacing=(0.25, 0.5, 0.125), origin=(12345.5, -6789.25, 3.0), iso=0.0),
        "farther": V.Volume(blobs, spacing=(0.25, 0.5, 0.125), origin=(3e6, -5e6, 1e6), iso=0.5),
        "one_axis_far": V.Volume(noise, spacing=(1.0, 1.0, 1.0), origin=(0.0, 0.0, 2e5), iso=0.0),
        "fine": V.Volume(noise, spacing=(1e-6, 1.5e-6, 2e-6), iso=0.0),
        "finest": V.Volume(blobs, spacing=(1e-14, 1e-14, 1e-14), iso=0.5),
        "wide": V.Volume(blobs, spacing=(1e13, 1e13, 1e13), iso=0.5),
        "flat": V.Volume(blobs, spacing=(1.0, 1.0, 1e-4), origin=(1.0, 1.0, 1.0), iso=0.5),
        "regular": V.Volume(saw, spacing=(0.5, 0.5, 0.5), iso=0.5),
        "few": V.Volume(V.blobs_volume(6, seed=1).data, spacing=(0.1, 0.1, 0.1), origin=(900.0, 900.0, 900.0), iso=0.5),
    }


CASES = _cases()


@pytest.mark.parametrize("name", sorted(CASES))
def test_split_of_coarse_positions(oracle, name):
    from tmc_gb300 import native
    vol = CASES[name]
    want = oracle.dmc(vol, 0)
    ctx = native.Context(0)
    try:
        got = ctx.dmc(vol, native.OUT_TRIANGLES)
    finally:
        ctx.close()
    np.testing.assert_array_equal(got["q"], want["q"])
    np.testing.assert_array_equal(got["t"], want["t"])
    assert want["t"].size > 0
