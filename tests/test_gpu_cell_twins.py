"""Halfedges made from the cells (a single volume's) against the CPU oracle and the general build.

The twins come from each grid face's crossed edges.  Fields and shapes reach every case: faces with two and with
four crossed edges, edges of one to four halfedges, grid borders on every side (down to one cell thick), cells
all, some or none of whose contours are used, values on the isovalue.  All integers are equal.  The same volume in
a batch of two takes the general build."""
import numpy as np
import pytest

from tmc_gb300 import native
from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu

FLAGS = native.OUT_HALFEDGES | native.OUT_TRIANGLES


def _white(shape, seed, levels=0):
    f = np.random.Generator(np.random.PCG64(seed)).standard_normal(shape)
    return (np.round(f * levels) if levels else f).astype(np.float32)


SHAPES = [(2, 2, 2), (2, 9, 9), (9, 2, 9), (9, 9, 2), (3, 3, 3), (3, 17, 4), (4, 3, 40), (24, 23, 22)]
FIELDS = {
    "white": (lambda s: _white(s, 3), 0.0),
    "coarse": (lambda s: _white(s, 4, 2), 0.0),  # many values on the isovalue
    "checker": (lambda s: (np.indices(s).sum(0) % 2).astype(np.float32), 0.5),  # every face ambiguous
    "rows": (lambda s: (np.indices(s)[2] % 2).astype(np.float32), 0.5),
    "sparse": (lambda s: (_white(s, 5) > 1.5).astype(np.float32), 0.5),
    "dense": (lambda s: (_white(s, 6) < 1.2).astype(np.float32), 0.5),
}


@pytest.fixture(scope="module")
def ctx():
    c = native.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("simplify", [0, 1])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("field", sorted(FIELDS))
def test_halfedges_from_cells(ctx, oracle, field, shape, simplify):
    make, iso = FIELDS[field]
    vol = V.Volume(make(shape), spacing=(0.5, 0.25, 1.0), iso=iso)
    flags = FLAGS | (native.DMC_SIMPLIFY if simplify else 0)
    want = oracle.dmc(vol, simplify)
    got = ctx.dmc(vol, flags)
    np.testing.assert_array_equal(got["q"], want["q"])
    np.testing.assert_array_equal(got["he"].reshape(-1, 4), want["he"].reshape(-1, 5)[:, :4])
    np.testing.assert_array_equal(got["hv"], want["hv"])
    np.testing.assert_array_equal(got["hf"], want["hf"])
    np.testing.assert_array_equal(got["t"], want["t"])
    for b in ctx.batch([vol, vol], [native.ALGO_DMC] * 2, [flags] * 2):
        for k in ("q", "he", "hv", "hf", "t"):
            np.testing.assert_array_equal(b[k], got[k])
        assert b["stats"][4] == got["stats"][4]
