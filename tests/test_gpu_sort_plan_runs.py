"""The plan sees the runs that many keys share.

A run of more than 256 keys is sorted by one CTA, which is meant for the rare run the sample misses: with
a tenth, or a hundredth, of the keys in one cell of 32 bits the plan has to take the digits that tell them
apart, or all of them.
"""
import ctypes

import numpy as np
import pytest

from adaptive_trees_b200 import _capi as C

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def plan_of(host):
    """(first pass run, long runs) of the pair sort of `host`, whose result is checked."""
    lib, n = C.load(), host.size
    keys = torch.from_numpy(host.view(np.int64)).cuda()
    out, vals = torch.empty_like(keys), torch.empty(n, dtype=torch.int32, device="cuda")
    size = ctypes.c_size_t()
    C.check(lib.ao_sort_pairs(None, ctypes.byref(size), None, None, None, None, n, 0, 64, None))
    scratch = torch.empty(size.value, dtype=torch.uint8, device="cuda")
    C.check(lib.ao_sort_pairs(scratch.data_ptr(), ctypes.byref(size), keys.data_ptr(), out.data_ptr(), None,
                              vals.data_ptr(), n, 0, 64, None))
    first, runs = ctypes.c_int(-1), ctypes.c_int(-1)
    C.check(lib.ao_selftest_sort_pairs_plan(scratch.data_ptr(), n, ctypes.byref(first), ctypes.byref(runs), None))
    assert np.array_equal(out.cpu().numpy().view(np.uint64), np.sort(host))
    return first.value, runs.value


@pytest.mark.parametrize("n,share", [(130_000, 0.1), (130_000, 0.03), (1_000_000, 0.03), (1_000_000, 0.012),
                                     (4_000_000, 0.012), (16_000_000, 0.012)])
def test_plan_tells_a_shared_cell_apart(n, share):
    r = np.random.default_rng(n)
    host = r.integers(0, 1 << 63, n, dtype=np.uint64)
    first, runs = plan_of(host)
    assert first >= 4 and runs == 0  # random keys: three or four digits are enough
    cell = r.random(n) < share
    host[cell] = (host[cell] & np.uint64(0xFFFFFFFF)) | np.uint64(0x1234567800000000)
    first, runs = plan_of(host)
    # five digits leave 256 runs of the cell's keys, each a CTA's where they are more than 256
    assert first == 0 and runs == 0 or first == 3 and runs == (256 if cell.sum() / 256 > 400 else 0), (first, runs)


def test_plan_of_clusters_in_every_part_of_a_batch_of_keys():
    """Clusters of a few hundred keys each, a third of the keys: the sample finds them in pairs, not in crowds."""
    n, size = 1_000_000, 400
    r = np.random.default_rng(7)
    host = r.integers(0, 1 << 63, n, dtype=np.uint64)
    centres = r.integers(0, 1 << 63, n // 3 // size, dtype=np.uint64) & ~np.uint64(0xFFFFFFFF)
    members = r.permutation(n)[: centres.size * size]
    host[members] = np.repeat(centres, size) | (host[members] & np.uint64(0xFFFFFFFF))
    first, runs = plan_of(host)
    assert first <= 3 and runs == 0, (first, runs)
