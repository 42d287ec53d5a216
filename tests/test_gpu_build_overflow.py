"""First builds that outgrow the unit arena and the leaf arrays they start with.

Pairs of particles at one point with a bucket of one split down to the last level,
so the tree holds far more units and leaves than its particle count suggests: the
build by levels grows its arena, places again, and must still equal the rounds.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("kind,n", [(0, 4_001), (0, 60_000), (1, 4_001), (1, 30_000)])
@pytest.mark.parametrize("hilbert", [False, True])
def test_stacked_pairs(kind, n, hilbert):
    import adaptive_trees_b200 as ab
    if kind == 1 and hilbert:
        pytest.skip("binary trees order by bisection")
    r = np.random.default_rng(n)
    xs = [torch.from_numpy(np.repeat(r.random(n // 2 + 1), 2)[:n]).cuda() for _ in range(3)]
    got = []
    for mode in (0, 1):
        t = ab.Tree(kind, *xs, ab.TreeConfig(maxParticlesPerLeaf=1,
                                             sfcKind=ab.SfcKind.Hilbert if hilbert else ab.SfcKind.Morton))
        t.setBuildMode(mode)
        t.build()
        assert t.buildPath()[0] == (mode == 0)
        needs, info = t.doBuffersNeedResize(), t.info()
        arrays = [t.get(k).view(torch.uint8).cpu().numpy()
                  for k in ("particleKeys_d", "perm_d", "cornerstone_d", "leafCounts_d")]
        got.append((arrays, [needs, info.num_leaves, info.leaf_capacity, info.num_nodes, t.buildPath()[1]]))
        t.close()
    assert got[0][1] == got[1][1]
    assert got[0][1][1] > 4 * n + 4096  # more leaves than a first build has room for
    for a, b in zip(got[0][0], got[1][0]):
        assert np.array_equal(a, b)
