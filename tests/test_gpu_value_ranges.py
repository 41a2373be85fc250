"""Both algorithms against the CPU oracle on fields at the edges of the float-pair paths: values near the
ends of the float range, whole numbers (corners at the isovalue, exact ties, singular faces), a random
value per point (every case and ambiguity), flat, thin and odd grids."""
import numpy as np
import pytest

from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from tmc_gb300 import native
    c = native.Context(0)
    yield c
    c.close()


def _random(nx, ny, nz, seed, levels=None):
    rng = np.random.Generator(np.random.PCG64(seed))
    if levels:
        return rng.integers(-levels, levels + 1, size=(nz, ny, nx)).astype(np.float32)
    return rng.standard_normal(size=(nz, ny, nx)).astype(np.float32)


FIELDS = {
    "random": (_random(33, 17, 19, 1), 0.0),
    "random_iso": (_random(31, 18, 5, 2), 0.3),
    "levels": (_random(29, 23, 11, 3, levels=9), 0.0),
    "levels_between": (_random(29, 23, 11, 4, levels=40), 2.5),
    "tiny": (_random(21, 16, 13, 5) * np.float32(1e-30), 0.0),
    "subnormal": (_random(21, 16, 13, 5) * np.float32(1e-39), 0.0),
    "huge": (_random(21, 16, 13, 5) * np.float32(1e30), 0.0),
    "steep": (_random(21, 16, 13, 6) * np.exp(10 * _random(21, 16, 13, 7)).astype(np.float32), 0.0),
    "two_planes": (_random(40, 33, 2, 8), 0.1),
    "thin": (_random(2, 3, 70, 9), 0.0),
    "one_tile_and_one": (_random(130, 17, 2, 10), 0.0),  # 129 * 16 cells: 2048 + 16
}


@pytest.mark.parametrize("name", sorted(FIELDS))
def test_tmc_matches_the_oracle(ctx, oracle, name):
    from tmc_gb300 import native
    data, iso = FIELDS[name]
    vol = V.Volume(data, origin=(-1.0, 0.5, 2.0), spacing=(0.1, 0.07, 0.13), iso=iso)
    want = oracle.tmc(vol)
    got64 = ctx.tmc(vol, native.OUT_POS_F64)
    np.testing.assert_array_equal(got64["t"], want["t"])
    np.testing.assert_array_equal(got64["v64"], want["v"])
    got = ctx.tmc(vol, 0)
    np.testing.assert_array_equal(got["t"], want["t"])
    # float32 outputs: the edge parameter is a float32 quotient (2^-22 of a cell), the position a float
    tol = 2 * np.spacing(np.abs(want["v"]).astype(np.float32)).astype(np.float64) + 0.13 * 2.0 ** -22
    ok = np.isfinite(want["v"])
    assert np.all(np.abs(got["v"].astype(np.float64) - want["v"])[ok] <= tol[ok])


@pytest.mark.parametrize("name", sorted(FIELDS))
def test_dmc_matches_the_oracle(ctx, oracle, name):
    from tmc_gb300 import native
    data, iso = FIELDS[name]
    vol = V.Volume(data, origin=(-1.0, 0.5, 2.0), spacing=(0.1, 0.07, 0.13), iso=iso)
    want = oracle.dmc_front(vol)
    got = ctx.dmc(vol, native.OUT_POS_F64 | native.OUT_LOCAL)
    np.testing.assert_array_equal(got["q"], want["q"])
    np.testing.assert_array_equal(got["vuvw"], want["vuvw"])
    np.testing.assert_array_equal(got["v64"], want["v"])
