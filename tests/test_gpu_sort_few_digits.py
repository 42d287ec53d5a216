"""Pair sorts of few digits: no plan, every pass, launch by launch or (four digits, middle sizes, not
captured) in one launch; at the edges of those rules, against the stable sort."""
import ctypes

import numpy as np
import pytest

from adaptive_trees_b200 import _capi as C

from .gpu_util import tree_config
from .scenarios import uniform_cube

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LOW, HIGH = 1 << 17, 1 << 20  # sorts without a plan in one launch


@pytest.fixture(scope="module")
def launches():
    """Kernel launches of the library so far."""
    import adaptive_trees_b200 as ab
    t = ab.Tree(0, *[torch.from_numpy(a).cuda() for a in uniform_cube(64, seed=1)], tree_config())
    yield lambda: t.info().kernel_launches
    t.close()


@pytest.mark.parametrize("begin,end", [(0, 8), (40, 64), (0, 32), (3, 30), (0, 33)])
@pytest.mark.parametrize("n", [2_561, LOW - 1, LOW, HIGH, HIGH + 1])
def test_pair_sort_of_few_digits(n, begin, end, launches):
    lib = C.load()
    r = np.random.default_rng(n + end)
    host = r.integers(0, 2 ** 64 - 1, n, dtype=np.uint64, endpoint=True)
    host[r.permutation(n)[: n // 4]] = host[0]
    mask = np.uint64((((1 << (end - begin)) - 1) << begin) & (2 ** 64 - 1))
    order = np.argsort(host & mask, kind="stable")
    keys = torch.from_numpy(host.view(np.int64)).cuda()
    out, vals = torch.empty_like(keys), torch.empty(n, dtype=torch.int32, device="cuda")
    size = ctypes.c_size_t()
    C.check(lib.ao_sort_pairs(None, ctypes.byref(size), None, None, None, None, n, begin, end, None))
    scratch = torch.full((size.value,), 0xFF, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()
    digits = (end - begin + 7) // 8

    def sort():
        C.check(lib.ao_sort_pairs(scratch.data_ptr(), ctypes.byref(size), keys.data_ptr(), out.data_ptr(), None,
                                  vals.data_ptr(), n, begin, end, ctypes.c_void_p(stream.cuda_stream)))

    def check(how):
        torch.cuda.synchronize()
        C.check(lib.ao_sort_pairs_check(scratch.data_ptr(), n, ctypes.c_void_p(stream.cuda_stream)))
        assert np.array_equal(out.cpu().numpy().view(np.uint64), host[order]), how
        assert np.array_equal(vals.cpu().numpy(), order.astype(np.int32)), how
        out.zero_(), vals.zero_()
        torch.cuda.synchronize()

    torch.cuda.synchronize()
    for how in ("queued", "queued again"):
        before = launches()
        sort()
        count = launches() - before
        if digits > 4:
            assert count == 2, count  # plan; passes and repair
        elif digits == 4 and LOW <= n <= HIGH:
            assert count == 1, count
        else:
            assert count == 2 + digits, count  # counts, their starts, passes
        check(how)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        sort()
    graph.replay()
    check("replayed")
