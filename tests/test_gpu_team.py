"""Launches by team: builds, small updates and small sorts whose CTAs wait for one another.

Only the CTAs that run at the same time take part, so work of another stream that holds part of the
GPU delays none of them, and their waits, all bounded, give up with an error status where what they
wait for never comes.
"""
import ctypes
import time

import numpy as np
import pytest

from adaptive_trees_b200 import _capi as C

from .gpu_util import to_dev, to_np, tree_config
from .scenarios import plummer_sphere, uniform_cube

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

AO_ERR_RUNTIME = 6
HOLD_MS = 300


@pytest.mark.parametrize("which", range(4), ids=["barrier", "roll", "octree_placement", "binary_placement"])
def test_team_wait_that_cannot_end_gives_up(which):
    lib = C.load()
    code = ctypes.c_int(-1)
    assert lib.ao_selftest_team_wait(which, 256, ctypes.byref(code)) == AO_ERR_RUNTIME, lib.ao_last_error().decode()
    assert code.value == 1
    assert "gave up" in lib.ao_last_error().decode()


def test_team_selftests_reject_bad_arguments():
    lib = C.load()
    assert lib.ao_selftest_team_wait(4, 256, None) == 1
    assert lib.ao_selftest_team_wait(-1, 256, None) == 1
    assert lib.ao_selftest_team_wait(0, 0, None) == 1
    assert lib.ao_selftest_team_wait(0, 1 << 20, None) == 1
    for sms, ms in ((0, 1), (1 << 20, 1), (1, 0), (1, 2001)):
        assert lib.ao_selftest_hold_sms(sms, ms, None) == 1


class Held:
    """`sms` SMs held by another stream while the block runs; the time the block took in ms."""

    def __init__(self, sms):
        self.sms, self.stream = sms, torch.cuda.Stream()

    def __enter__(self):
        torch.cuda.synchronize()
        C.check(C.load().ao_selftest_hold_sms(self.sms, HOLD_MS, ctypes.c_void_p(self.stream.cuda_stream)))
        time.sleep(0.01)  # (it has started)
        self.start = time.perf_counter()
        return self

    def __exit__(self, *_):
        self.ms = (time.perf_counter() - self.start) * 1e3
        torch.cuda.synchronize()


def _all_but(free):
    return torch.cuda.get_device_properties(0).multi_processor_count - free


# LeafCount and NFCount octrees and a k-d tree whose grids are the whole GPU's
TREES = {"leaf": (0, uniform_cube(700_001, seed=1), dict(bucket=64)),
         "leaf_small": (0, uniform_cube(20_011, seed=2), dict(bucket=16, hilbert=True)),
         "nf": (0, plummer_sphere(400_003, seed=3, dtype=np.float32), dict(bucket=512, nf=True, hilbert=True)),
         "binary": (1, uniform_cube(900_001, seed=4), dict(bucket=32))}


@pytest.mark.parametrize("free", [1, 40, 147])
@pytest.mark.parametrize("name", list(TREES))
def test_build_and_update_on_part_of_the_gpu(name, free):
    import adaptive_trees_b200 as ab
    kind, xyz, cfg = TREES[name]
    arrays = ["particleKeys_d", "perm_d", "cornerstone_d", "leafCounts_d"] + ["nearFieldCounts_d"] * cfg.get("nf", False)
    stream = torch.cuda.Stream()
    trees, coords, graphs, took = [], [], [], []
    for _ in range(2):  # one that shares the GPU, one that has it
        coords.append([to_dev(a) for a in xyz])
        torch.cuda.synchronize()
        t = ab.Tree(kind, *coords[-1], tree_config(**cfg), stream=stream)
        with torch.cuda.stream(stream):
            t.build()
            t.update()
            t.updateUntilConverged()  # (the kernels are loaded)
            t.doBuffersNeedResize()
        graphs.append(torch.cuda.CUDAGraph())
        torch.cuda.synchronize()
        with torch.cuda.graph(graphs[-1], stream=stream):
            t.update()
        graphs[-1].replay()
        trees.append(t)

    def step(do, k):
        with torch.cuda.stream(stream):
            do(k)
            return trees[k].doBuffersNeedResize()

    for do in (lambda k: trees[k].build(), lambda k: trees[k].update(), lambda k: graphs[k].replay(),
               lambda k: trees[k].updateUntilConverged()):
        for c in coords:
            for a, m in zip(c, (1.3e-3, 2.1e-3, 0.7e-3)):
                a.copy_((a + m) % 1.0)
        with Held(_all_but(free)) as held:
            needs = step(do, 0)
        assert needs == step(do, 1)
        for a in arrays:
            assert np.array_equal(to_np(trees[0].get(a)), to_np(trees[1].get(a))), a
        took.append(held.ms)
    assert max(took) < HOLD_MS / 2, took  # none waited for the SMs that are held
    for t in trees:
        t.close()


@pytest.mark.parametrize("free", [1, 147])
@pytest.mark.parametrize("n,bits", [(30_001, 64), (1_500_000, 64), (1_500_000, 16)])
def test_pair_sort_on_part_of_the_gpu(n, bits, free):
    lib = C.load()
    host = np.random.default_rng(n).integers(0, 1 << 63, n, dtype=np.uint64)
    order = np.argsort(host & np.uint64(2 ** bits - 1), kind="stable")
    keys = torch.from_numpy(host.view(np.int64)).cuda()
    out, vals = torch.empty_like(keys), torch.empty(n, dtype=torch.int32, device="cuda")
    size = ctypes.c_size_t()
    C.check(lib.ao_sort_pairs(None, ctypes.byref(size), None, None, None, None, n, 0, bits, None))
    scratch = torch.empty(size.value, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()

    def sort():
        C.check(lib.ao_sort_pairs(scratch.data_ptr(), ctypes.byref(size), keys.data_ptr(), out.data_ptr(), None,
                                  vals.data_ptr(), n, 0, bits, ctypes.c_void_p(stream.cuda_stream)))
        C.check(lib.ao_sort_pairs_check(scratch.data_ptr(), n, ctypes.c_void_p(stream.cuda_stream)))

    torch.cuda.synchronize()
    sort()
    out.zero_(), vals.zero_()
    with Held(_all_but(free)) as held:
        sort()
    assert np.array_equal(out.cpu().numpy().view(np.uint64), host[order])
    assert np.array_equal(vals.cpu().numpy(), order.astype(np.int32))
    assert held.ms < HOLD_MS / 2, held.ms


def test_trees_of_several_threads_and_priorities_at_once():
    """Teams of several streams share the SMs: each tree builds and updates as it does alone."""
    import threading

    import adaptive_trees_b200 as ab
    low, high = 0, -5
    work = [(low, 0, 300_001, 64), (high, 0, 300_001, 64), (low, 1, 400_003, 32), (high, 1, 400_003, 32),
            (high, 0, 20_011, 64), (low, 0, 700_001, 16)]
    failed = []

    def run(k, priority, kind, n, bucket):
        try:
            stream = torch.cuda.Stream(priority=priority)
            x = [to_dev(a) for a in uniform_cube(n, seed=20 + k)]
            torch.cuda.synchronize()
            t = ab.Tree(kind, *x, tree_config(bucket=bucket), stream=stream)
            first = None
            for _ in range(15):
                with torch.cuda.stream(stream):
                    t.build()
                    t.update()
                    assert not t.doBuffersNeedResize()
                    got = [to_np(t.get(a)) for a in ("perm_d", "cornerstone_d", "leafCounts_d")]
                first = first or got
                assert all(np.array_equal(a, b) for a, b in zip(first, got))
            t.close()
        except BaseException as e:  # noqa: BLE001 (reported by the test's own thread)
            failed.append((k, repr(e)))

    threads = [threading.Thread(target=run, args=(k, *w)) for k, w in enumerate(work)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
