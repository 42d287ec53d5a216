"""update() of NFCount trees large enough to refresh by units.

The near-field counts and group flags of the full refresh come from the
standing tree's internal nodes there.  A tree updated until nothing changes is
the tree of the particles alone, so it must equal one built from scratch by
the reference's rounds, whose near field goes leaf by leaf through the node
table.  All results are integers: equality.
"""
import numpy as np
import pytest

from tests.gpu_util import tree_config

pytestmark = pytest.mark.gpu

N = (1 << 22) + 12_345  # above the rule's line
ARRAYS = ("particleKeys_d", "perm_d", "cornerstone_d", "leafCounts_d", "nearFieldCounts_d")


def frames(dist, real, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    u = lambda: torch.rand(N, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    if dist == "uniform":
        x = [u() for _ in range(3)]
    elif dist == "plummer":
        r = 0.05 / torch.sqrt((u() * 0.985).clamp_(min=1e-12).pow(-2.0 / 3.0) - 1.0)
        v = torch.randn(3, N, generator=g, device="cuda", dtype=torch.float64)
        v *= r / v.norm(dim=0)
        x = [v[k] + 0.5 for k in range(3)]
    else:  # a tight cluster in a sparse background: leaves with hundreds of keys after the move
        x = [torch.where(torch.arange(N, device="cuda") % 4 == 0, u(), 0.25 + 1e-3 * u()) for _ in range(3)]
    y = [a + (3e-2 if dist == "cluster" else 2e-3) * torch.randn(N, generator=g, device="cuda", dtype=torch.float64)
         for a in x]
    return [[a.to(real).clamp_(0.0, 0.999999).contiguous() for a in f] for f in (x, y)]


@pytest.mark.parametrize("dist,bucket,hilbert,real", [("uniform", 512, False, "float32"), ("plummer", 512, True, "float32"),
                                                      ("plummer", 3000, False, "float64"), ("cluster", 512, True, "float64")])
def test_updated_tree_is_the_tree_of_the_moved_particles(dist, bucket, hilbert, real):
    import torch

    import adaptive_trees_b200 as ab
    first, second = frames(dist, getattr(torch, real), 7)
    cfg = tree_config(bucket=bucket, nf=True, hilbert=hilbert)
    moving = [a.clone() for a in first]
    a = ab.Tree(0, *moving, cfg)
    a.build()
    for m, s in zip(moving, second):
        m.copy_(s)
    torch.cuda.synchronize()
    for _ in range(8):
        a.updateUntilConverged(64)
        if not a.doBuffersNeedResize():
            break
        a.resizeBuffers()
    b = ab.Tree(0, *second, cfg)
    b.setBuildMode(1)
    b.build()
    for name in ARRAYS:
        x, y = a.get(name), b.get(name)
        assert x.numel() == y.numel(), name
        assert torch.equal(x.view(torch.uint8), y.view(torch.uint8)), name
    a.updateUntilConverged(4)  # nothing moved: the full refresh alone
    a.doBuffersNeedResize()
    for name in ARRAYS:
        assert torch.equal(a.get(name).view(torch.uint8), b.get(name).view(torch.uint8)), name
    a.close()
    b.close()


def test_captured_update_follows_the_particles():
    import torch

    import adaptive_trees_b200 as ab
    first, second = frames("plummer", torch.float32, 9)
    cfg = tree_config(bucket=512, nf=True, hilbert=True)
    moving = [a.clone() for a in first]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        a = ab.Tree(0, *moving, cfg, stream=stream)
        a.build()
        for frame in (second, first):
            for m, s in zip(moving, frame):
                m.copy_(s)
            a.update()
            while a.doBuffersNeedResize():
                a.resizeBuffers()
                a.update()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            a.update()
        direct = ab.Tree(0, *moving, cfg, stream=stream)
        direct.build()
        for frame in (second, first, second):
            for m, s in zip(moving, frame):
                m.copy_(s)
            graph.replay()
            assert not a.doBuffersNeedResize()
            direct.build()
            for name in ARRAYS[:4]:
                assert torch.equal(a.get(name).view(torch.uint8), direct.get(name).view(torch.uint8)), name
        del graph
    stream.synchronize()
    a.close()
    direct.close()
