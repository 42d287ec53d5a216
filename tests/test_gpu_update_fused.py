"""update() in one launch after its sort against the same update launch by launch.

While stages are timed (setProfiling) every pass has launches of its own; otherwise
trees of few leaves refresh, pass and count in one cooperative launch.  Both follow
the same rules on the same integers, so every array, state word and resize request
is equal, queued directly and replayed from a graph.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

NAMES = ("particleKeys_d", "perm_d", "cornerstone_d", "leafCounts_d")
STATE = ("num_leaves", "num_active_particles", "leaf_capacity", "num_nodes")


def _bytes(t):
    return t.contiguous().view(torch.uint8).cpu().numpy() if t.numel() else np.empty(0, np.uint8)


@pytest.mark.parametrize("kind,n,bucket,iterations", [
    (0, 1, 4, 2), (0, 33, 32, 1), (0, 5_000, 1, 3), (0, 40_009, 16, 2), (0, 300_007, 64, 5),
    (1, 1, 4, 2), (1, 33, 32, 1), (1, 5_000, 1, 3), (1, 40_009, 16, 6), (1, 300_007, 32, 2)])
@pytest.mark.parametrize("captured", [False, True])
def test_update_in_one_launch(kind, n, bucket, iterations, captured):
    import adaptive_trees_b200 as ab
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n + bucket)
    start = [torch.rand(n, generator=gen, device="cuda") for _ in range(3)]
    stream = torch.cuda.Stream()
    trees, coords, replay = [], [], []
    torch.cuda.synchronize()
    for timed in (False, True):
        x = [a.clone() for a in start]
        torch.cuda.synchronize()
        t = ab.Tree(kind, *x, ab.TreeConfig(maxParticlesPerLeaf=bucket, updateIterations=iterations), stream=stream)
        t.setProfiling(timed)
        with torch.cuda.stream(stream):
            t.build()
        graph = None
        if captured:
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                t.update()
        trees.append(t), coords.append(x), replay.append(graph)
    # small moves, a collapse that splits past the capacity, the way back (merges)
    for step, move in enumerate((1e-3, 1e-3, None, "back", 0.0)):
        noise = [torch.randn(n, generator=gen, device="cuda") for _ in range(3)]
        for x in coords:
            for a, s, e in zip(x, start, noise):
                if move is None:
                    a.copy_((0.3 + 0.01 * e).clamp(0, 0.999))
                elif move == "back":
                    a.copy_(s)
                else:
                    a.copy_((a + move * e).clamp(0, 0.999))
        torch.cuda.synchronize()
        got = []
        for t, graph in zip(trees, replay):
            with torch.cuda.stream(stream):
                graph.replay() if graph is not None else t.update()
                needs = t.doBuffersNeedResize()
            torch.cuda.synchronize()
            info = t.info()
            got.append(([_bytes(t.get(k)) for k in NAMES], [needs] + [getattr(info, k) for k in STATE]))
        assert got[0][1] == got[1][1], step
        for name, a, b in zip(NAMES, got[0][0], got[1][0]):
            assert np.array_equal(a, b), (step, name)
    for t in trees:
        t.close()
