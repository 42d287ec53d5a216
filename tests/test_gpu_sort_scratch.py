"""The pair sort in scratch that starts at any 8-byte address: the alignment of its 64-bit words is
all it may ask for (a caller's own arena gives no more)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("config", [-1, 0, 3])
@pytest.mark.parametrize("n", [1, 2561, 60_001, (1 << 21) + 1])
@pytest.mark.parametrize("begin,end", [(0, 64), (5, 20)])
def test_pair_sort_in_scratch_at_8_bytes(n, begin, end, config, captured):
    import adaptive_trees_b200 as ab
    from adaptive_trees_b200 import _capi as C
    lib = C.load()
    r = np.random.default_rng(n + end)
    host = r.integers(0, 1 << 63, n, dtype=np.uint64)
    host[r.integers(0, n, n // 3)] = host[0]
    mask = np.uint64((((1 << (end - begin)) - 1) << begin) & (2 ** 64 - 1))
    order = np.argsort(host & mask, kind="stable")
    keys = torch.from_numpy(host.view(np.int64)).cuda()
    out = torch.empty_like(keys)
    out_vals = torch.empty(n, dtype=torch.int32, device="cuda")
    size = ctypes.c_size_t()
    C.check(lib.ao_sort_pairs(None, ctypes.byref(size), None, None, None, None, n, begin, end, None))
    block = torch.full((size.value + 256,), 0x5A, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()
    ab.force_sort_config(config)
    try:
        for offset in (0, 8, 24, 136):
            scratch = block[offset:offset + size.value]
            assert scratch.data_ptr() % 256 == offset

            def sort():
                C.check(lib.ao_sort_pairs(scratch.data_ptr(), ctypes.byref(size), keys.data_ptr(), out.data_ptr(), None,
                                          out_vals.data_ptr(), n, begin, end, ctypes.c_void_p(stream.cuda_stream)))

            out.zero_(), out_vals.zero_()
            torch.cuda.synchronize()
            if captured:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=stream):
                    sort()
                graph.replay()
            else:
                with torch.cuda.stream(stream):
                    sort()
            torch.cuda.synchronize()
            C.check(lib.ao_sort_pairs_check(scratch.data_ptr(), n, ctypes.c_void_p(stream.cuda_stream)))
            assert np.array_equal(out.cpu().numpy().view(np.uint64), host[order]), offset
            assert np.array_equal(out_vals.cpu().numpy(), order.astype(np.int32)), offset
    finally:
        ab.force_sort_config(-1)
