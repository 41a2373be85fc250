"""The outputs of simplified DMC meshes do not depend on which of them are asked for.

The result's arrays are made after the passes in one allocation, the float64 positions only when they are
an output (the triangle split reads those of the mesh before compaction): every choice of passes and
outputs, on meshes that lose many faces, few and none, gives the arrays of the call with all outputs,
equal, and float32 positions that are the roundings of the float64 ones."""
import itertools

import numpy as np
import pytest

from tmc_gb300 import native
from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu

PASSES = {"colour": native.DMC_P3X3Y_COLOR, "isolated": native.DMC_P3X3Y_ISOLATED, "p3333": native.DMC_P3333}
OUTPUTS = [0, native.OUT_TRIANGLES, native.OUT_HALFEDGES, native.OUT_TRIANGLES | native.OUT_HALFEDGES,
           native.OUT_POS_F64, native.OUT_POS_F64 | native.OUT_TRIANGLES]
ALL = native.OUT_POS_F64 | native.OUT_TRIANGLES | native.OUT_HALFEDGES
VOLUMES = {
    "noise": V.small_noise_volume(29, seed=7, coarse=6),
    "blobs": V.blobs_volume(17, seed=2),
    # a flat surface: no vertex of valence 3 away from the border, nothing is removed
    "plane": V.Volume(np.broadcast_to(np.arange(9, dtype=np.float32)[:, None, None], (9, 8, 7)).copy(),
                      spacing=(0.5, 0.5, 0.5), iso=3.25),
    "cell": V.Volume(np.array([[[0, 1], [1, 0]], [[1, 0], [0, 1]]], np.float32), spacing=(1, 1, 1), iso=0.5),
    "empty": V.Volume(np.zeros((5, 6, 7), np.float32), spacing=(1, 1, 1), iso=0.5),
}
KEYS = ("v", "n", "q", "t", "he", "hv", "hf")


@pytest.fixture(scope="module")
def ctx():
    c = native.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("name", sorted(VOLUMES))
@pytest.mark.parametrize("passes", ["+".join(c) for n in (1, 2, 3) for c in itertools.combinations(PASSES, n)])
def test_outputs_do_not_depend_on_the_choice(ctx, name, passes):
    vol = VOLUMES[name]
    p = sum(PASSES[x] for x in passes.split("+"))
    want = ctx.dmc(vol, p | ALL)
    np.testing.assert_array_equal(want["v"], want["v64"].astype(np.float32))
    plain = ctx.dmc(vol, 0)
    assert want["q"].size <= plain["q"].size
    if name == "plane":
        np.testing.assert_array_equal(want["q"], plain["q"])
    for out in OUTPUTS:
        got = ctx.dmc(vol, p | out)
        for k in KEYS:
            if got.get(k) is not None and got[k].size:
                np.testing.assert_array_equal(got[k], want[k], err_msg=f"{k} with outputs {out:#x}")
        assert got["v"].size == want["v"].size and got["q"].size == want["q"].size
        assert got["stats"][4] == (want["stats"][4] if out & native.OUT_HALFEDGES else 0)
