"""The repair of the planned sort under every plan.

A sort's result does not depend on its plan, so a test that looks at the result alone cannot tell
whether a repair ran.  Here the first pass is given (0 to 7), the sort reports it back with the number
of runs that were too long for the repair's tiles, and the runs are at the edges: of a tile, of the
longest run a tile orders, of the steps of a long run's own sort, of segments.
"""
import ctypes

import numpy as np
import pytest

from adaptive_trees_b200 import _capi as C

from .gpu_util import to_np, tree_config
from .scenarios import ESC64, uniform_cube

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TILE, RUN = 2048, 256
CONFIGS = [0, 1, 2]  # the 8-bit configurations: tiles of 2560, 4096 and 2048 keys


def clustered(n, members, seed):
    """Uniform particles; `members` more, spread over the others, within 1e-9 of one point: they share
    their key's first 7 digits (the point is not at a cell's edge)."""
    x = uniform_cube(n + members, seed=seed)
    r = np.random.default_rng(seed)
    at = r.permutation(n + members)[:members]
    for a in x:
        a[at] = 0.3123456789 + 1e-9 * r.random(members)
    return x


def stacked(n, copies, seed):
    base = uniform_cube(n // copies, seed=seed)
    order = np.random.default_rng(seed).permutation(n // copies * copies)
    return [np.repeat(a, copies)[order] for a in base]


def escaped(n, every, seed):
    x = uniform_cube(n, seed=seed)
    for a in x:
        a[::every] = ESC64
    return x


# particles, and whether first passes up to 4 (32 and more high bits) leave a run of more than RUN keys
CASES = {
    **{f"n={n}": (uniform_cube(n, seed=n), False) for n in (1, 2, TILE - 1, TILE, TILE + 1, 2 * TILE + RUN + 1, 30_011)},
    **{f"run of {m}": (clustered(40_000, m, m), m > RUN) for m in (RUN - 1, RUN, RUN + 1, 2 * TILE, 2 * TILE + 1, 9_001)},
    "stacks": (stacked(30_000, 300, 7), True), "pairs": (stacked(30_000, 2, 8), False),
    "escaped": (escaped(30_000, 3, 9), False), "all escaped": (escaped(3_000, 1, 10), False),
}


@pytest.fixture(autouse=True)
def as_before():
    yield
    import adaptive_trees_b200 as ab
    ab.force_sort_config(None)


def _plan(fn, handle, force):
    first, runs = ctypes.c_int(-1), ctypes.c_int(-1)
    C.check(fn(handle, force, ctypes.byref(first), ctypes.byref(runs)))
    return first.value, runs.value


def _sorted(kind, dev, curve):
    import adaptive_trees_b200 as ab
    keys = to_np(ab.compute_sfc_keys(kind, *dev, sfc_kind=curve))
    return keys, np.argsort(keys, kind="stable")


@pytest.mark.parametrize("config", CONFIGS)
@pytest.mark.parametrize("first", range(8))
def test_tree_sort_under_every_plan(first, config):
    import adaptive_trees_b200 as ab
    lib = C.load()
    ab.force_sort_config(config)
    stream = torch.cuda.Stream()
    for name, (x, long) in CASES.items():
        kind = len(name) % 2
        dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in x]
        keys, order = _sorted(kind, dev, ab.SfcKind.Hilbert)
        torch.cuda.synchronize()
        t = ab.Tree(kind, *dev, tree_config(bucket=64, hilbert=kind == 0), stream=stream)
        _plan(lib.ao_selftest_tree_sort_plan, t._h, first)

        def check(how):
            ran, runs = _plan(lib.ao_selftest_tree_sort_plan, t._h, first)
            assert ran == first, (name, how)
            if first == 0:
                assert runs == 0, (name, how)
            elif first <= 4:
                assert (runs > 0) == long, (name, how, runs)
            assert np.array_equal(to_np(t.get("particleKeys_d")), keys[order]), (name, how)
            assert np.array_equal(to_np(t.get("perm_d")), order.astype(np.uint32)), (name, how)

        with torch.cuda.stream(stream):
            t.build()  # passes and repair in one launch
            check("one launch")
            # the sample of the sorted keys, through the leaf counts that come from it
            corner, counts = to_np(t.get("cornerstone_d")), to_np(t.get("leafCounts_d"))
            assert np.array_equal(np.diff(np.searchsorted(keys[order], corner)), counts.astype(np.int64)), name
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            t.update()  # launch by launch
        graph.replay()
        torch.cuda.synchronize()
        check("launches")
        t.close()


@pytest.mark.parametrize("config", CONFIGS)
@pytest.mark.parametrize("first", range(8))
def test_batch_sort_under_every_plan(first, config):
    import adaptive_trees_b200 as ab
    lib = C.load()
    ab.force_sort_config(config)
    # systems that end inside a tile, equal neighbours, a long run across what was one tile
    systems = [uniform_cube(1, seed=1), [a[:0] for a in uniform_cube(1, seed=2)], uniform_cube(TILE + 1, seed=3),
               clustered(3_000, RUN, 4), clustered(3_000, RUN, 4), clustered(5_000, RUN + 1, 5),
               clustered(8_000, 2 * TILE + 1, 6), escaped(9_000, 2, 7), uniform_cube(20_011, seed=8)]
    dev = [[torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in s] for s in systems]
    b = ab.Batch(*[[d[k] for d in dev] for k in range(3)], tree_config(bucket=16, hilbert=True))
    _plan(lib.ao_selftest_batch_sort_plan, b._h, first)

    def check(how):
        ran, runs = _plan(lib.ao_selftest_batch_sort_plan, b._h, first)
        assert ran == first, how
        if first <= 4:
            assert runs == (2 if first else 0), (how, runs)
        for k, d in enumerate(dev):
            if d[0].numel():
                keys, order = _sorted(0, d, ab.SfcKind.Hilbert)
                assert np.array_equal(to_np(b.get(k, "particleKeys_d")), keys[order]), (k, how)
                assert np.array_equal(to_np(b.get(k, "perm_d")), order.astype(np.uint32)), (k, how)

    b.build()
    check("one launch")
    for d in dev:  # another order of the same particles
        for a in d:
            a.copy_(a.flip(0).clone())
    torch.cuda.synchronize()
    b.update()  # launch by launch (configuration 1: tiles in halves)
    b.doBuffersNeedResize()
    check("launches")
    b.close()


@pytest.mark.parametrize("config", CONFIGS)
@pytest.mark.parametrize("begin,end", [(0, 64), (5, 50), (0, 24)])
def test_pair_sort_under_every_plan(begin, end, config):
    lib = C.load()
    passes, r = (end - begin + 7) // 8, np.random.default_rng(end)
    for n, members in ((1, 1), (TILE + 1, 0), (20_001, RUN), (20_001, RUN + 1), (60_001, 9_001)):
        host = r.integers(0, 2 ** 64 - 1, n, dtype=np.uint64, endpoint=True)
        # equal keys but for the lowest digit that is sorted
        host[r.permutation(n)[:members]] = np.uint64(0x5A5A5A5A5A5A5A5A) ^ (
            r.integers(0, 256, members, dtype=np.uint64) << np.uint64(begin))
        mask = np.uint64((((1 << (end - begin)) - 1) << begin) & (2 ** 64 - 1))
        order = np.argsort(host & mask, kind="stable")
        keys = torch.from_numpy(host.view(np.int64)).cuda()
        out, vals = torch.empty_like(keys), torch.empty(n, dtype=torch.int32, device="cuda")
        size = ctypes.c_size_t()
        C.check(lib.ao_sort_pairs(None, ctypes.byref(size), None, None, None, None, n, begin, end, None))
        scratch = torch.empty(size.value, dtype=torch.uint8, device="cuda")
        stream = torch.cuda.Stream()
        for first in range(passes):
            def sort():
                C.check(lib.ao_selftest_sort_pairs(scratch.data_ptr(), ctypes.byref(size), keys.data_ptr(), out.data_ptr(),
                                                   None, vals.data_ptr(), n, begin, end, config, first,
                                                   ctypes.c_void_p(stream.cuda_stream)))

            for captured in (False, True):
                out.zero_(), vals.zero_()
                torch.cuda.synchronize()
                if captured:
                    graph = torch.cuda.CUDAGraph()
                    with torch.cuda.graph(graph, stream=stream):
                        sort()
                    graph.replay()
                else:
                    sort()
                torch.cuda.synchronize()
                got, runs = ctypes.c_int(-1), ctypes.c_int(-1)
                C.check(lib.ao_selftest_sort_pairs_plan(scratch.data_ptr(), n, ctypes.byref(got), ctypes.byref(runs),
                                                        ctypes.c_void_p(stream.cuda_stream)))
                assert got.value == first
                if first == 0 or members > RUN:
                    assert (runs.value > 0) == (first > 0), (n, first, runs.value)
                assert np.array_equal(out.cpu().numpy().view(np.uint64), host[order]), (n, first, captured)
                assert np.array_equal(vals.cpu().numpy(), order.astype(np.int32)), (n, first, captured)


def test_update_of_few_leaves_is_one_launch():
    """What test_gpu_update_fused.py compares are two paths: one launch behind the sort, and many."""
    import adaptive_trees_b200 as ab
    for kind in (0, 1):
        x = [torch.from_numpy(a).cuda() for a in uniform_cube(20_011, seed=kind)]
        torch.cuda.synchronize()
        t = ab.Tree(kind, *x, tree_config(bucket=64, iters=3))
        t.build()
        launches = []
        for timed in (False, True):
            t.setProfiling(timed)
            before = t.info().kernel_launches
            t.update()
            launches.append(t.info().kernel_launches - before)
        assert launches[0] == 4, launches  # plan, keys, sort, update
        assert launches[1] >= launches[0] + 10, launches
        t.close()
