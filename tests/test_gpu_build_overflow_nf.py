"""First builds of NFCount trees, large enough to refresh by units, that outgrow the unit arena and the
leaf arrays: the units stay where they are while the leaf arrays grow, and the tree equals the rounds'."""
import pytest

from .gpu_util import tree_config

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ARRAYS = ("particleKeys_d", "perm_d", "cornerstone_d", "leafCounts_d", "nearFieldCounts_d")


@pytest.mark.parametrize("bucket,hilbert", [(40, True), (64, False)])
def test_near_field_tree_of_more_leaves_than_particles(bucket, hilbert):
    import adaptive_trees_b200 as ab
    n = (1 << 22) + 3
    g = torch.Generator(device="cuda")
    g.manual_seed(bucket)
    x = [torch.rand(n, generator=g, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    trees = []
    for mode in (0, 1):
        t = ab.Tree(0, *x, tree_config(bucket=bucket, nf=True, hilbert=hilbert))
        t.setBuildMode(mode)
        t.build()
        assert t.buildPath()[0] == (mode == 0)
        trees.append(t)
    assert trees[0].info().num_leaves > n + 4096  # the leaf arrays a first build starts with
    for step in ("build", "update"):
        if step == "update":
            for a in x:
                a.copy_((a + 2e-4 * torch.randn(n, generator=g, device="cuda")).clamp(0, 0.999))
            torch.cuda.synchronize()
            for t in trees:
                t.update()
        assert trees[0].doBuffersNeedResize() == trees[1].doBuffersNeedResize()
        for name in ("num_leaves", "leaf_capacity", "num_active_particles"):
            assert getattr(trees[0].info(), name) == getattr(trees[1].info(), name), (step, name)
        for name in ARRAYS:
            a, b = (t.get(name).view(torch.uint8) for t in trees)
            assert torch.equal(a, b), (step, name)
    for t in trees:
        t.close()
