"""The planned sort of the particle keys against a stable numpy sort.

The passes cover only the keys' high digits and a repair orders the runs that
share them, so the cases are runs of every kind: none, short ones that straddle
the repair's tiles, runs longer than its window, equal keys, escaped particles,
and inputs on which every pass runs.  All results are integers: equality.
"""
import numpy as np
import pytest

from tests import scenarios as S

pytestmark = pytest.mark.gpu

TILE, RUN = 2048, 256  # the repair's tile and its longest run


def uniform(n, seed):
    return S.uniform_cube(n, seed=seed)


def with_cluster(n, members, width, seed):
    """Uniform particles of which `members` lie within `width` of one point."""
    x = [a.copy() for a in S.uniform_cube(n, seed=seed)]
    r = np.random.default_rng(seed + 1)
    at = r.permutation(n)[:members]
    for a in x:
        a[at] = 0.3123456789 + width * r.random(members)
    return x


def stacked(n, copies, seed):
    """Every particle `copies` times, at shuffled positions."""
    base = S.uniform_cube(-(-n // copies), seed=seed)
    order = np.random.default_rng(seed + 1).permutation(-(-n // copies) * copies)[:n]
    return [np.repeat(a, copies)[order] for a in base]


def escaped(n, every, seed):
    x = [a.copy() for a in S.uniform_cube(n, seed=seed)]
    for a in x:
        a[::every] = S.ESC64
    return x


def in_order(n, seed):
    """Particles already stored along the curve (Morton order of a fine grid)."""
    x = S.uniform_cube(n, seed=seed)
    q = [(a * 1024).astype(np.int64) for a in x]
    key = np.zeros(n, np.int64)
    for b in range(10):
        for k, a in enumerate(q):
            key |= ((a >> b) & 1) << (3 * b + 2 - k)
    order = np.argsort(key, kind="stable")
    return [a[order] for a in x]


CASES = {
    "one": uniform(1, 1), "two": uniform(2, 2), "31": uniform(31, 3), "tile-1": uniform(TILE - 1, 4),
    "tile": uniform(TILE, 5), "tile+1": uniform(TILE + 1, 6), "tile+run": uniform(TILE + RUN, 7),
    "3tiles+run+1": uniform(3 * TILE + RUN + 1, 8), "40k": uniform(40_009, 9), "700k": uniform(700_001, 10),
    "plummer": S.plummer_sphere(500_003, seed=11, dtype=np.float32),
    "run of 200": with_cluster(300_000, 200, 1e-9, 12), "run of 256": with_cluster(300_000, RUN, 1e-9, 13),
    "run of 257": with_cluster(300_000, RUN + 1, 1e-9, 14), "run of 700": with_cluster(300_000, 700, 1e-9, 15),
    "run of 3000": with_cluster(1_000_000, 3000, 1e-6, 16), "run of 20000": with_cluster(4_000_000, 20_000, 1e-6, 17),
    # steps of a long run's sort: 2048 keys
    **{f"run of {k}": with_cluster(1_000_000, k, 1e-6, 50 + k) for k in (2047, 2048, 2049, 4097)},
    "one cluster": with_cluster(100_000, 100_000, 1e-5, 18),
    "pairs": stacked(200_000, 2, 19), "stacks of 100": stacked(200_000, 100, 20), "one point": stacked(50_000, 50_000, 21),
    "escaped": escaped(100_001, 3, 22), "all escaped": escaped(5_000, 1, 23), "few escaped": escaped(500_000, 1000, 24),
    "in order": in_order(600_000, 25),
}


@pytest.fixture(autouse=True, scope="module")
def untuned_afterwards():
    yield
    import adaptive_trees_b200 as ab
    ab.forget_sort_tuning()  # other tests start from an untuned library


@pytest.mark.parametrize("kind,hilbert", [(0, False), (0, True), (1, False)])
@pytest.mark.parametrize("name", list(CASES))
def test_planned_sort_is_the_stable_sort(name, kind, hilbert):
    import torch

    import adaptive_trees_b200 as ab
    xs = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in CASES[name]]
    curve = ab.SfcKind.Hilbert if hilbert else ab.SfcKind.Morton
    keys = ab.compute_sfc_keys(kind, *xs, sfc_kind=curve).view(torch.int64).cpu().numpy().view(np.uint64)
    order = np.argsort(keys, kind="stable")
    t = ab.Tree(kind, *xs, ab.TreeConfig(sfcKind=curve))
    for step in range(3):  # the first build times the sort configurations; the control block is used again
        t.build()
        got_k = t.get("particleKeys_d").view(torch.int64).cpu().numpy().view(np.uint64)
        got_p = t.get("perm_d").view(torch.int32).cpu().numpy().view(np.uint32)
        assert np.array_equal(got_k, keys[order]), (name, step)
        assert np.array_equal(got_p, order.astype(np.uint32)), (name, step)
        counts = t.get("leafCounts_d").view(torch.int32).cpu().numpy().view(np.uint32)
        corner = t.get("cornerstone_d").view(torch.int64).cpu().numpy().view(np.uint64)
        assert np.array_equal(np.diff(np.searchsorted(keys[order], corner)), counts.astype(np.int64)), (name, step)
    t.close()


SYSTEMS = {
    "odd sizes": [uniform(n, 100 + n) for n in (1, 0, 31, 2048, 2049, 7, 0, 5000, 257)],
    "the same system again": [with_cluster(30_000, 400, 1e-9, 31)] * 3,  # equal keys on both sides of a boundary
    "clusters": [with_cluster(60_000, 3000, 1e-7, 32), uniform(100_001, 33), with_cluster(9_000, 9_000, 1e-6, 34)],
    "points and escapes": [stacked(20_000, 300, 35), escaped(30_000, 2, 36), escaped(500, 1, 37), uniform(64, 38)],
    "one cluster each": [with_cluster(8_000, 8_000, 1e-5, 40 + k) for k in range(6)],
}


@pytest.mark.parametrize("hilbert", [False, True])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_planned_sort_of_a_batch_is_each_systems_stable_sort(name, hilbert):
    import torch

    import adaptive_trees_b200 as ab
    curve = ab.SfcKind.Hilbert if hilbert else ab.SfcKind.Morton
    dev = [[torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in x] for x in SYSTEMS[name]]
    b = ab.Batch(*[[d[k] for d in dev] for k in range(3)], ab.TreeConfig(sfcKind=curve))

    def check(step):
        for s, d in enumerate(dev):
            if not d[0].numel():
                continue
            keys = ab.compute_sfc_keys(0, *d, sfc_kind=curve).view(torch.int64).cpu().numpy().view(np.uint64)
            order = np.argsort(keys, kind="stable")
            got_k = b.get(s, "particleKeys_d").view(torch.int64).cpu().numpy().view(np.uint64)
            got_p = b.get(s, "perm_d").view(torch.int32).cpu().numpy().view(np.uint32)
            assert np.array_equal(got_k, keys[order]), (name, s, step)
            assert np.array_equal(got_p, order.astype(np.uint32)), (name, s, step)

    for step in ("first build (timed configurations)", "build in one launch", "build in one launch again"):
        b.build()
        check(step)
    for d in dev:  # an update sorts launch by launch
        for a in d:
            a.copy_(torch.where(a < 1, (a + 1e-3) % 1.0, a))
    torch.cuda.synchronize()
    b.update()
    b.doBuffersNeedResize()
    check("update")
    b.close()


def pair_keys(kind, n, seed):
    r = np.random.default_rng(seed)
    k = r.integers(0, 2 ** 64 - 1, size=n, dtype=np.uint64, endpoint=True)
    if kind == "low bits only":
        k &= np.uint64(0xFFFF)
    elif kind == "runs":  # high digits repeat, low ones tell apart; the all-ones prefix among them
        k = (k & np.uint64(0xFFFFFF)) | (np.uint64(0xFFFFFFFFFF) - (k >> np.uint64(40)) % np.uint64(max(1, n // 40)) << np.uint64(24))
    elif kind == "long run":
        k[: n // 3] = (k[: n // 3] & np.uint64(0xFFFFFFFF)) | np.uint64(0x1234567800000000)
        k = k[r.permutation(n)]
    elif kind == "equal":
        k[:] = k[0]
    return k


@pytest.mark.parametrize("begin,end", [(0, 64), (5, 50), (0, 32), (40, 64), (0, 17), (3, 11)])
@pytest.mark.parametrize("kind", ["random", "low bits only", "runs", "long run", "equal"])
@pytest.mark.parametrize("n,offset", [(1, 0), (2047, 0), (2305, 1), (60_001, 0), (600_000, 1)])
def test_planned_pair_sort_is_the_stable_sort(n, offset, kind, begin, end):
    import ctypes

    import torch

    from adaptive_trees_b200 import _capi as C
    lib = C.load()
    k = pair_keys(kind, n, n + begin)
    keys = torch.from_numpy(k.view(np.int64)).cuda()
    vals = torch.arange(n, dtype=torch.int32, device="cuda") * 7
    out_k = torch.zeros(n + 1, dtype=torch.int64, device="cuda")[offset:offset + n]  # 8-byte aligned only
    out_v = torch.zeros(n + 1, dtype=torch.int32, device="cuda")[offset:offset + n]
    size = ctypes.c_size_t()
    C.check(lib.ao_sort_pairs(None, ctypes.byref(size), None, None, None, None, n, begin, end, None))
    scratch = torch.full((size.value,), 0xA5, dtype=torch.uint8, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    mask = np.uint64((((1 << (end - begin)) - 1) << begin) & (2 ** 64 - 1))
    order = np.argsort(k & mask, kind="stable")
    for _ in range(2):  # the second call finds the first one's words in the scratch
        C.check(lib.ao_sort_pairs(scratch.data_ptr(), ctypes.byref(size), keys.data_ptr(), out_k.data_ptr(),
                                  vals.data_ptr(), out_v.data_ptr(), n, begin, end, stream))
        C.check(lib.ao_sort_pairs_check(scratch.data_ptr(), n, stream))
        assert np.array_equal(out_k.cpu().numpy().view(np.uint64), k[order])
        assert np.array_equal(out_v.cpu().numpy(), order.astype(np.int32) * 7)


@pytest.mark.parametrize("n", [1, 2047, 4097, 100_003, (1 << 21) + 1])
@pytest.mark.parametrize("bits", [(0, 64), (0, 16), (5, 46)])
def test_pair_sort_queued_and_captured(n, bits):
    """Small sorts run in one launch, or launch by launch under capture: both are the stable sort."""
    import ctypes

    import torch

    from adaptive_trees_b200 import _capi as C
    r = np.random.default_rng(n + bits[1])
    host = r.integers(0, 1 << 63, n, dtype=np.uint64) & ~np.uint64(0x3FF << 20)
    host[r.integers(0, n, n // 3)] = host[0]  # a stack of equal keys
    begin, end = bits
    mask = np.uint64(((1 << (end - begin)) - 1) << begin)
    order = np.argsort(host & mask, kind="stable")
    keys = torch.from_numpy(host.view(np.int64)).cuda()
    vals = torch.arange(n, dtype=torch.int32, device="cuda")
    out, out_vals = torch.empty_like(keys), torch.empty_like(vals)
    size = ctypes.c_size_t()
    lib = C.load()
    C.check(lib.ao_sort_pairs(None, ctypes.byref(size), None, None, None, None, n, begin, end, None))
    scratch = torch.empty(size.value, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()

    def sort():
        C.check(lib.ao_sort_pairs(scratch.data_ptr(), ctypes.byref(size), keys.data_ptr(), out.data_ptr(),
                                  vals.data_ptr(), out_vals.data_ptr(), n, begin, end,
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))

    def check(how):
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().view(np.uint64), host[order]), how
        assert np.array_equal(out_vals.cpu().numpy(), order.astype(np.int32)), how
        out.zero_(), out_vals.zero_()
        torch.cuda.synchronize()

    with torch.cuda.stream(stream):
        sort()
    check("queued")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        sort()
    graph.replay()
    check("replayed")
    graph.replay()
    check("replayed again")
