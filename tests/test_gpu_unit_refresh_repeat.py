"""update() by units again and again: the units of a standing tree are made by lanes of which the last
ones of a level have no child, and must not look at a unit that another warp is rewriting.  Levels
whose units do not fill their warps, many times over; every update of a frame gives the same arrays."""
import pytest

from .gpu_util import tree_config

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ARRAYS = ("cornerstone_d", "leafCounts_d", "nearFieldCounts_d")


@pytest.mark.parametrize("n,bucket,hilbert", [((1 << 22) + 1, 512, True), ((1 << 22) + 77_777, 300, False)])
def test_updates_by_units_repeat(n, bucket, hilbert):
    import adaptive_trees_b200 as ab
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    frames = [[torch.rand(n, generator=g, device="cuda").pow_(2) for _ in range(3)]]
    frames.append([(a + 1e-4 * torch.randn(n, generator=g, device="cuda")).clamp_(0, 0.999999) for a in frames[0]])
    x = [a.clone() for a in frames[0]]
    torch.cuda.synchronize()
    t = ab.Tree(0, *x, tree_config(bucket=bucket, nf=True, hilbert=hilbert, iters=8))

    def update(k):
        for a, b in zip(x, frames[k]):
            a.copy_(b)
        torch.cuda.synchronize()
        t.update()
        while t.doBuffersNeedResize():
            t.resizeBuffers()
            t.update()
        return [t.get(name).view(torch.uint8).clone() for name in ARRAYS]

    t.build()
    update(1), update(0)
    want = [update(1), update(0)]  # (converged from either frame)
    for step in range(40):
        for k in (1, 0):
            got = update(k)
            assert all(torch.equal(a, b) for a, b in zip(got, want[1 - k])), (step, k)
    t.close()
