"""Kernels of a call are set up while the one before them runs; every result must still be the one of kernels
run one after another: small calls (where the overlap is largest) of changing sizes and kinds, repeated, from
several threads with a context each, give equal arrays every time."""
import threading

import numpy as np
import pytest

from tmc_gb300 import native
from tmc_gb300 import volumes as V

pytestmark = pytest.mark.gpu

FULL = native.OUT_POS_F64 | native.OUT_TRIANGLES | native.OUT_HALFEDGES


def _calls():
    vols = [V.small_noise_volume(n, seed=n) for n in (6, 19, 34)] + [V.blobs_volume(26, seed=1)]
    calls = []
    for v in vols:
        calls += [lambda c, v=v: c.dmc(v, 0), lambda c, v=v: c.dmc(v, native.DMC_SIMPLIFY | FULL),
                  lambda c, v=v: c.tmc(v, native.OUT_HALFEDGES, halfedge=True)]
    return calls


def _same(a, b):
    return all(np.array_equal(a[k], b[k]) for k in a if isinstance(a[k], np.ndarray))


@pytest.mark.parametrize("threads", [1, 3])
def test_repeated_small_calls_are_equal(threads):
    calls = _calls()
    ctx = native.Context(0)
    want = [c(ctx) for c in calls]
    ctx.close()
    bad = []

    def run(start):
        ctx = native.Context(0)
        try:
            for r in range(12):
                for i in range(len(calls)):
                    j = (i * (start + 1) + r) % len(calls)
                    if not _same(calls[j](ctx), want[j]):
                        bad.append((start, r, j))
        except Exception as e:  # shown by the assertion
            bad.append(e)
        finally:
            ctx.close()

    ts = [threading.Thread(target=run, args=(k,)) for k in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
