"""DMC float32 normals whose gradients cancel, against the float64 normals of the oracle's vertices.

Where the gradients at a cell's corners are more than 16 times the interpolated one (here: 20, so that a vertex
near the limit is left out) the float32 interpolation gives way, and the normal is the rounding of the float64 one:
central differences times the reciprocal of two spacings, interpolated along x, y, z and divided by the length, in
this order (where they cancel the order shows in the last bits).  Equal, without a tolerance."""
import numpy as np
import pytest

from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu


def _random(nx, ny, nz, seed):
    return np.random.Generator(np.random.PCG64(seed)).standard_normal(size=(nz, ny, nx)).astype(np.float32)


def _checker(eps, seed, n=50):
    c = ((np.indices((n, n, n)).sum(0) % 2) * 2 - 1).astype(np.float32)
    return (c * (1 + eps * _random(n, n, n, seed))).astype(np.float32)


UNEVEN = dict(origin=(-1.0, 0.7, 2.0), spacing=(0.011, 0.043, 0.17))
CASES = {
    "checker": V.Volume(_checker(0.01, 7), iso=0.0, spacing=(0.1, 0.1, 0.1)),
    "checker_uneven": V.Volume(_checker(1e-3, 7), iso=0.0, **UNEVEN),
    "levels": V.Volume(np.round(4 * _random(60, 60, 60, 4)).astype(np.float32), iso=0.5, spacing=(0.1, 0.1, 0.1)),
    "levels_uneven": V.Volume(np.round(4 * _random(60, 60, 60, 4)).astype(np.float32), iso=0.5, **UNEVEN),
    "white_uneven": V.Volume(_random(61, 47, 52, 2), iso=0.3, **UNEVEN),
    "saddle_uneven": V.Volume(V.saddle_slab(128, 60, 24, seed=3).data, iso=0.0, **UNEVEN),
    "tiny": V.Volume(_random(33, 31, 30, 5) * np.float32(1e-30), iso=0.0, **UNEVEN),
    "subnormal": V.Volume(_random(33, 31, 30, 6) * np.float32(1e-39), iso=0.0, **UNEVEN),
    "fine_spacing": V.Volume(_random(33, 31, 30, 10) * np.float32(1e-25), iso=0.0, spacing=(1e-30, 3e-28, 2e-36)),
    "wide_spacing": V.Volume(_random(33, 31, 30, 11), iso=0.0, spacing=(1e30, 3e31, 2e36)),
}


def _corner_gradients(f, spacing, i, j, k, sign):
    """estimateGradient at the eight corners: central differences, point 0 beyond either border."""
    nz, ny, nx = f.shape
    inv = [1.0 / (2 * h) for h in spacing]

    def index(x, n):
        return np.where(x < 0, 0, np.where(x >= n, n - x, x))

    out = []
    for q in range(8):
        a, b, c = i + (q & 1), j + (q >> 1 & 1), k + (q >> 2 & 1)
        out.append(sign * np.stack([(f[c, b, index(a + 1, nx)] - f[c, b, index(a - 1, nx)]) * inv[0],
                                    (f[c, index(b + 1, ny), a] - f[c, index(b - 1, ny), a]) * inv[1],
                                    (f[index(c + 1, nz), b, a] - f[index(c - 1, nz), b, a]) * inv[2]], -1))
    return out


@pytest.mark.parametrize("flip", [0, 1])
@pytest.mark.parametrize("name", sorted(CASES))
def test_cancelling_normals(oracle, name, flip):
    from tmc_gb300 import native
    vol = CASES[name]
    want = oracle.dmc_front(vol, flip)
    ctx = native.Context(0)
    try:
        got = ctx.dmc(vol, native.OUT_LOCAL | (native.GRAD_FLIP if flip else 0))
    finally:
        ctx.close()
    np.testing.assert_array_equal(got["q"], want["q"])
    nx, ny, _ = vol.dims
    cell, p = want["vcell"], want["vuvw"].reshape(-1, 3).astype(np.float64)
    i, j, k = cell % (nx - 1), cell // (nx - 1) % (ny - 1), cell // ((nx - 1) * (ny - 1))
    g = _corner_gradients(vol.data.astype(np.float64), vol.spacing, i, j, k, -1.0 if flip else 1.0)
    u, v, w = (p[:, d, None] for d in range(3))
    m = (1 - w) * ((1 - v) * ((1 - u) * g[0] + u * g[1]) + v * ((1 - u) * g[2] + u * g[3])) + w * (
        (1 - v) * ((1 - u) * g[4] + u * g[5]) + v * ((1 - u) * g[6] + u * g[7]))
    length = np.sqrt(m[:, 0] * m[:, 0] + m[:, 1] * m[:, 1] + m[:, 2] * m[:, 2])
    pick = np.max([np.abs(x).max(1) for x in g], axis=0) > 20 * length
    print(f"{name}: {pick.sum()} cancelling of {pick.size} vertices")
    n = (m[pick] / length[pick, None]).astype(np.float32)
    np.testing.assert_array_equal(got["n"].reshape(-1, 3)[pick], n)
