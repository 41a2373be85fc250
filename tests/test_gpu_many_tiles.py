"""Offsets over more tiles of cells than one block scans (8,192 of 2,048 cells), and around that number.

Isolated points above the isovalue make an octahedron each (TMC: six vertices, eight triangles), so what a wrong
offset anywhere would overwrite is known: the vertices are the expected positions, each once, in the order of
their cells, and every triangle joins three of one octahedron.  DMC makes a box of eight vertices and six
quads of each.  Exact."""
import numpy as np
import pytest

from tmc_gb300 import native
from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu

SHAPES = [(257, 257, 257), (257, 258, 257), (301, 259, 233)]  # z, y, x; 256^3 cells are 8,192 tiles


@pytest.mark.parametrize("shape", SHAPES)
def test_isolated_points(shape):
    rng = np.random.Generator(np.random.PCG64(5))
    nz, ny, nx = shape
    # one point in each chosen 3x3x3 block: never neighbours
    b = rng.permutation((nz // 3 - 1) * (ny // 3 - 1) * (nx // 3 - 1))[:60000]
    z, y, x = (1 + 3 * c for c in np.unravel_index(b, (nz // 3 - 1, ny // 3 - 1, nx // 3 - 1)))
    f = np.zeros(shape, np.float32)
    f[z, y, x] = 1.0
    n = b.size
    vol = V.Volume(f, spacing=(1.0, 1.0, 1.0), iso=0.5)
    ctx = native.Context(0)
    try:
        tmc, dmc = ctx.tmc(vol, native.OUT_POS_F64), ctx.dmc(vol, native.OUT_POS_F64)
    finally:
        ctx.close()
    # in grid units, exactly (whole origin, halves)
    v, t = tmc["v64"].reshape(-1, 3) - np.asarray(vol.origin), tmc["t"].reshape(-1, 3)
    assert v.shape[0] == 6 * n and t.shape[0] == 8 * n
    p = np.stack([x, y, z], 1).astype(np.float64)
    want = np.concatenate([p + s * d for d in np.eye(3) for s in (-0.5, 0.5)])
    order = lambda a: a[np.lexsort(a.T)]  # noqa: E731
    np.testing.assert_array_equal(order(v), order(want))
    np.testing.assert_array_equal(np.unique(t), np.arange(6 * n))
    centre = np.rint(v[t].mean(axis=1))  # the point: 1/6 off on every axis
    assert np.all(np.abs(v[t] - centre[:, None, :]).sum(axis=2) == 0.5)
    d, q = dmc["v64"].reshape(-1, 3) - np.asarray(vol.origin), dmc["q"].reshape(-1, 4)
    assert d.shape[0] == 8 * n and q.shape[0] == 6 * n
    cell = np.floor(d).astype(np.int64)
    lin = (cell[:, 2] * (ny - 1) + cell[:, 1]) * (nx - 1) + cell[:, 0]
    assert np.all(np.diff(lin) > 0)  # one vertex per crossed cell, in cell order
    np.testing.assert_array_equal(np.bincount(q.ravel(), minlength=8 * n), 3)
    assert np.all(np.ptp(cell[q], axis=1) <= 1)
