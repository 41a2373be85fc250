"""TMC and DMC on fields with fewer and more ambiguous cells (TMC) and vertices (DMC) than the room planned
before their numbers are known, against the CPU oracle.

Room: one ambiguous cell in 64 (at least 4096, at most every cell), a vertex per cell.  White noise has about
10 % ambiguous cells and more vertices than cells, a checkerboard only ambiguous cells, blobs next to none.
Alone and in batches of them; all integers and the float64 positions are equal."""
import numpy as np
import pytest

from tmc_gb300 import native
from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu


def _white(shape, seed):
    return np.random.Generator(np.random.PCG64(seed)).standard_normal(shape).astype(np.float32)


VOLUMES = {
    "white_small": V.Volume(_white((12, 13, 14), 1), spacing=(1, 1, 1), iso=0.0),
    "white": V.Volume(_white((41, 37, 39), 2), spacing=(0.5, 1.0, 0.25), iso=0.0),
    "checker": V.Volume((np.indices((22, 21, 20)).sum(0) % 2).astype(np.float32), spacing=(1, 1, 1), iso=0.5),
    "blobs": V.blobs_volume(45, seed=3),
}


@pytest.fixture(scope="module")
def ctx():
    c = native.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("name", sorted(VOLUMES))
def test_room_alone(ctx, oracle, name):
    vol = VOLUMES[name]
    got = ctx.tmc(vol, native.OUT_POS_F64)
    want = oracle.tmc(vol)
    np.testing.assert_array_equal(got["t"], want["t"])
    np.testing.assert_array_equal(got["v64"], want["v"])
    got = ctx.dmc(vol, native.OUT_POS_F64)
    want = oracle.dmc_front(vol, 0)
    np.testing.assert_array_equal(got["q"], want["q"])
    np.testing.assert_array_equal(got["v64"], want["v"])


@pytest.mark.parametrize("names", [("blobs", "blobs"), ("white", "blobs"), ("checker", "white_small", "white")])
@pytest.mark.parametrize("algo", [native.ALGO_TMC, native.ALGO_DMC])
def test_room_in_a_batch(ctx, names, algo):
    vols = [VOLUMES[n] for n in names]
    got = ctx.batch(vols, [algo] * len(vols), [native.OUT_POS_F64] * len(vols))
    for vol, g in zip(vols, got):
        want = ctx.tmc(vol, native.OUT_POS_F64) if algo == native.ALGO_TMC else ctx.dmc(vol, native.OUT_POS_F64)
        for k in ("v64", "t", "q"):
            np.testing.assert_array_equal(g[k], want[k])
