"""The two sorts of computeViews() take one launch each after the one that sets them up, where no graph is
being captured; captured they go launch by launch.  The views are the oracle's both ways."""
import pytest

from oracle import oracle as O

from .gpu_util import compare, oracle_config, tree_config
from .scenarios import uniform_cube

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("n", [500, 50_000, 300_000])
def test_view_sorts_in_one_launch(n, kind):
    import adaptive_trees_b200 as ab
    xyz = uniform_cube(n, seed=3)
    cfg = dict(bucket=64, views=(True, True, True))
    o = O.OracleTree(kind, *xyz, oracle_config(**cfg))
    o.build()
    dev = [torch.from_numpy(a).cuda() for a in xyz]
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    t = ab.Tree(kind, *dev, tree_config(**cfg), stream=stream)

    t.build()
    before = t.info().kernel_launches
    t.computeViews()
    direct = t.info().kernel_launches - before
    torch.cuda.synchronize()
    compare(t, o)
    before = t.info().kernel_launches
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        t.computeViews()
    captured = t.info().kernel_launches - before
    graph.replay()
    torch.cuda.synchronize()
    compare(t, o)
    # counts, their starts and a pass per digit (one digit, and eight) against a launch each
    assert captured - direct == (2 + 1 - 1) + (2 + 8 - 1), (captured, direct)
    del graph
    t.close()
