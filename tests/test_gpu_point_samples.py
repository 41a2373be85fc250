"""DMC vertices whose contours leave many samples of the projection open, against the CPU oracle.

The samples of a warp's 32 vertices are listed together, 256 at a time, short lists by their own lane and long
ones by the warp, so the cases vary how many there are: none but the first (smooth), a few (noise), dozens in
a few lanes or in all of them (saddles and flat or symmetric fields, one field per period of the lanes), and
vertex numbers around whole warps.  The sample taken decides the float64 position, which is exact."""
import numpy as np
import pytest

from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu


def _seeded(shape, every, seed):
    """A smooth field with strong saddles in every `every`-th cell."""
    rng = np.random.Generator(np.random.PCG64(seed))
    f = V.gaussian_blobs(*shape, rng).astype(np.float32)
    nz, ny, nx = f.shape
    n = 0
    for k in range(0, nz - 1, 2):
        for j in range(0, ny - 1, 2):
            for i in range(0, nx - 1, 2):
                n += 1
                if n % every == 0:
                    s = np.float32(rng.uniform(0.25, 1.0)) * np.array([[[1, -1], [-1, 1]], [[-1, 1], [1, -1]]], np.float32)
                    f[k:k + 2, j:j + 2, i:i + 2] = np.float32(0.5) + s * np.float32(rng.uniform(0.9, 1.1))
    return f


def _cases():
    rng = np.random.Generator(np.random.PCG64(21))
    c = {"smooth": (V.blobs_volume(20, seed=3).data, 0.5), "noise": (V.small_noise_volume(27, seed=2, coarse=5).data, 0.0),
         "white": (rng.standard_normal((19, 21, 23)).astype(np.float32), 0.0),
         "coarse_values": (np.round(rng.standard_normal((18, 18, 18)) * 2).astype(np.float32), 0.5),
         "checker": ((np.indices((9, 10, 11)).sum(0) % 2).astype(np.float32), 0.5),
         "one_cell": (np.array([[[0, 1], [1, 0]], [[1, 0], [0, 1]]], np.float32), 0.5)}
    for every in (1, 3, 16):
        c[f"saddles_{every}"] = (_seeded((21, 20, 19), every, 40 + every), 0.5)
    return c


CASES = _cases()


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("scale", [1.0, 3.0 * 2.0 ** -40])
def test_points_exact(oracle, name, scale):
    from tmc_gb300 import native
    data, iso = CASES[name]
    vol = V.Volume((data * np.float32(scale)).astype(np.float32), spacing=(0.5, 0.25, 1.0), origin=(1.0, 2.0, -3.0),
                   iso=iso * scale)
    want = oracle.dmc_front(vol, 0)
    ctx = native.Context(0)
    try:
        got = ctx.dmc(vol, native.OUT_POS_F64 | native.OUT_LOCAL)
    finally:
        ctx.close()
    np.testing.assert_array_equal(got["q"], want["q"])
    np.testing.assert_array_equal(got["vuvw"], want["vuvw"])
    np.testing.assert_array_equal(got["v64"], want["v"])
