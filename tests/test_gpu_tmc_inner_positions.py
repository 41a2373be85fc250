"""TMC float32 positions of inner vertices (ambiguous cells) against the CPU oracle: the roundings of its float64
positions, without a tolerance.  Checkerboards of nearly equal values have an inner vertex in most cells."""
import numpy as np
import pytest

from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu


def _checker(eps, seed, n=60, **grid):
    c = ((np.indices((n, n, n)).sum(0) % 2) * 2 - 1).astype(np.float32)
    r = np.random.Generator(np.random.PCG64(seed)).standard_normal(c.shape).astype(np.float32)
    return V.Volume((c * (1 + eps * r)).astype(np.float32), iso=0.0, **grid)


CASES = {
    "half": _checker(0.5, 7, spacing=(0.1, 0.1, 0.1)),
    "tenth": _checker(0.1, 7, spacing=(0.1, 0.1, 0.1)),
    "uneven": _checker(0.1, 8, spacing=(0.011, 0.043, 0.17), origin=(-0.3, -1.3, -5.0)),
    "thousandth": _checker(1e-3, 9, spacing=(0.5, 0.25, 0.125), origin=(1e4, -2e4, 0.0)),
    "fine": _checker(0.3, 10, n=40, spacing=(1e-34, 3e-36, 2e-38), origin=(0.0, 0.0, 0.0)),
    "fine_apart": _checker(0.3, 11, n=40, spacing=(1e-31, 1e-44, 1.0), origin=(1e-33, 1e-40, 0.0)),
    "white": V.Volume(np.random.Generator(np.random.PCG64(5)).standard_normal((50, 51, 52)).astype(np.float32),
                      spacing=(0.04, 0.04, 0.04), iso=0.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_inner_positions(oracle, name):
    from tmc_gb300 import native
    vol = CASES[name]
    want = oracle.tmc(vol)
    ctx = native.Context(0)
    try:
        got = ctx.tmc(vol, 0)
    finally:
        ctx.close()
    np.testing.assert_array_equal(got["t"], want["t"])
    v = want["v"].reshape(-1, 3)
    at = (v - np.asarray(vol.origin)) / np.asarray(vol.spacing)
    inner = (np.abs(at - np.round(at)) > 1e-6).sum(1) > 1
    assert inner.sum() > 1000
    np.testing.assert_array_equal(got["v"].reshape(-1, 3)[inner], v[inner].astype(np.float32))
