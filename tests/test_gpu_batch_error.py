"""A batch whose sort gave up, and the sort after it.

A sort's look-back words carry the number of the sort, so that they need no clearing.  A sort that
ends early must have used its number up: the next one would take the words it left for its own.
The error is planted from the host (the device's error word, which a wait that gives up sets); the
sort then ends before its repair.
"""
import numpy as np
import pytest

from adaptive_trees_b200 import _capi as C

from .gpu_util import to_np, tree_config
from .scenarios import uniform_cube

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("hilbert", [False, True])
def test_sort_after_one_that_gave_up(hilbert):
    import adaptive_trees_b200 as ab
    lib = C.load()
    sizes = (60_001, 0, 5_000, 120_007)
    # systems whose keys lie at opposite ends from one build to the next
    low = [[0.2 * a for a in uniform_cube(n, seed=n)] for n in sizes]
    high = [[0.7 + 0.3 * a for a in uniform_cube(n, seed=n + 1)] for n in sizes]
    dev = [[torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in s] for s in low]
    cfg = dict(bucket=16, hilbert=hilbert)
    ab.set_sort_autotune(False)
    try:
        b = ab.Batch(*[[d[k] for d in dev] for k in range(3)], tree_config(**cfg))
        b.build()
        for coords in (high, low, high):
            C.check(lib.ao_selftest_batch_error(b._h, 1))
            with pytest.raises(RuntimeError, match="gave up"):
                b.build()
            C.check(lib.ao_selftest_batch_error(b._h, 0))
            for d, s in zip(dev, coords):
                for a, h in zip(d, s):
                    a.copy_(torch.from_numpy(h))
            torch.cuda.synchronize()
            b.build()
            for k, d in enumerate(dev):
                if not d[0].numel():
                    continue
                t = ab.Tree(0, *d, tree_config(**cfg))
                t.build()
                for name in ("particleKeys_d", "perm_d", "cornerstone_d", "leafCounts_d"):
                    assert np.array_equal(to_np(b.get(k, name)), to_np(t.get(name))), (k, name)
                t.close()
        b.close()
    finally:
        ab.set_sort_autotune(True)
