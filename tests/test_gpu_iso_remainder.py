"""TMC float32 edge vertices where the isovalue is no float and the field's differences are small beside it.

The edge parameter is a quotient of a difference of floats (the isovalue as a float pair) and one of two floats:
three roundings of 2^-24 and the pair's own, so within 2^-22 of the oracle's; positions then within two float ulps
and 2^-22 of a cell."""
import numpy as np
import pytest

from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("base,size", [(1000.0, 1e-3), (1000.0, 1.0), (3e5, 0.25), (-70.0, 1e-4), (0.1, 1e-6)])
def test_positions_with_an_inexact_isovalue(oracle, base, size):
    from tmc_gb300 import native
    f = V.blobs_volume(34, seed=8).data.astype(np.float64)
    data = (base + size * f).astype(np.float32)
    iso = base + size * 0.4371  # not a float
    assert float(np.float32(iso)) != iso
    vol = V.Volume(data, origin=(-1.0, 0.5, 2.0), spacing=(0.1, 0.07, 0.13), iso=iso)
    want = oracle.tmc(vol)
    ctx = native.Context(0)
    try:
        got = ctx.tmc(vol, 0)
    finally:
        ctx.close()
    np.testing.assert_array_equal(got["t"], want["t"])
    w = want["v"].reshape(-1, 3)
    tol = 2 * np.spacing(np.abs(w).astype(np.float32)).astype(np.float64) + np.asarray(vol.spacing) * 2.0 ** -22
    assert w.size > 0
    assert np.all(np.abs(got["v"].reshape(-1, 3).astype(np.float64) - w) <= tol)
