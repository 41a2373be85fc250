"""TMC normals that the float32 interpolation does not serve, against the CPU oracle's float64 normals.

With float64 positions every normal is the rounding of the float64 one.  With float32 outputs those of edge
vertices are wherever the ends' gradients cancel to below 1/16 of their size (here: 1/20, computed again in
float64, so that a vertex near the limit is left out).  Equal, without a tolerance."""
import numpy as np
import pytest

from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu


def _random(nx, ny, nz, seed):
    return np.random.Generator(np.random.PCG64(seed)).standard_normal(size=(nz, ny, nx)).astype(np.float32)


def _cases():
    saddle = V.saddle_slab(200, 60, 24, seed=3)
    uneven = dict(origin=(-1.0, 0.7, 2.0), spacing=(0.011, 0.043, 0.17))
    return {
        "noise": V.small_noise_volume(64, seed=5, coarse=7),
        "saddle": saddle,
        "saddle_uneven": V.Volume(saddle.data, iso=saddle.iso, **uneven),
        "white_uneven": V.Volume(_random(61, 47, 52, 2), iso=0.3, **uneven),
        "inexact_iso": V.Volume((1000 + _random(41, 37, 30, 3) * np.float32(2e-3)).astype(np.float32), iso=1000.00013, **uneven),
        "levels": V.Volume(np.round(4 * _random(45, 44, 43, 4)).astype(np.float32), iso=0.5, **uneven),
        "tiny": V.Volume(_random(33, 31, 30, 5) * np.float32(1e-30), iso=0.0, **uneven),
        "subnormal": V.Volume(_random(33, 31, 30, 6) * np.float32(1e-39), iso=0.0, **uneven),
        "huge": V.Volume(_random(33, 31, 30, 7) * np.float32(1e30), iso=0.0, **uneven),
        "steep": V.Volume((_random(33, 31, 30, 8) * np.exp(12 * _random(33, 31, 30, 9))).astype(np.float32), iso=0.0, **uneven),
        "fine_spacing": V.Volume(_random(33, 31, 30, 10) * np.float32(1e-25), iso=0.0, spacing=(1e-30, 3e-28, 2e-36)),
        "wide_spacing": V.Volume(_random(33, 31, 30, 11), iso=0.0, spacing=(1e30, 3e31, 2e36)),
        "thin": V.Volume(_random(2, 3, 70, 12), iso=0.1, **uneven),
    }


CASES = _cases()


def _gradient(f, spacing):
    """UGrid::gradient at every point: central differences, one-sided ones over one spacing at the border."""
    out = []
    for axis, h in zip((2, 1, 0), spacing):
        d = np.empty_like(f)
        s = np.moveaxis(f, axis, 0)
        o = np.moveaxis(d, axis, 0)
        o[1:-1] = (s[2:] - s[:-2]) / (2 * h)
        o[0], o[-1] = (s[1] - s[0]) / h, (s[-1] - s[-2]) / h
        out.append(d)
    return np.stack(out, -1)


def _cancelling(vol, v):
    """Edge vertices whose interpolated gradient is below 1/20 of the ends' largest component."""
    at = (v - np.asarray(vol.origin)) / np.asarray(vol.spacing)
    low = np.floor(at + 1e-7).astype(np.int64)
    off = np.abs(at - np.round(at)) > 1e-7
    edge = off.sum(1) == 1
    f = vol.data.astype(np.float64)
    g = _gradient(f, vol.spacing)
    low = np.minimum(low, np.asarray(vol.dims) - 1)
    high = np.minimum(low + off, np.asarray(vol.dims) - 1)
    a, b = g[low[:, 2], low[:, 1], low[:, 0]], g[high[:, 2], high[:, 1], high[:, 0]]
    l = np.where(off, at - low, 0).sum(1)[:, None]
    m = a + l * (b - a)
    return edge & (np.maximum(np.abs(a), np.abs(b)).max(1) > 20 * np.sqrt((m * m).sum(1)))


@pytest.mark.parametrize("name", sorted(CASES))
def test_tmc_normals(oracle, name):
    from tmc_gb300 import native
    vol = CASES[name]
    want = oracle.tmc(vol)
    n = want["n"].reshape(-1, 3).astype(np.float32)
    ctx = native.Context(0)
    try:
        got64 = ctx.tmc(vol, native.OUT_POS_F64)
        got = ctx.tmc(vol, 0)
    finally:
        ctx.close()
    np.testing.assert_array_equal(got64["v64"], want["v"])
    np.testing.assert_array_equal(got64["n"].reshape(-1, 3), n)
    if name in ("noise", "saddle", "saddle_uneven", "white_uneven", "inexact_iso", "levels", "thin"):
        pick = _cancelling(vol, want["v"].reshape(-1, 3))
        print(f"{name}: {pick.sum()} cancelling of {pick.size} vertices")
        np.testing.assert_array_equal(got["n"].reshape(-1, 3)[pick], n[pick])
