"""The work a user of the tree engine has it do, as cases that can be timed.

An N-body or FMM program holds its particles on the GPU, builds a tree once, then moves the particles
and updates the tree every step, and reads the sorted keys, the permutation, the leaves and their counts
(and, where its traversal needs them, the views).  The cases go through the entry points such a program
calls (Tree, Batch, the pair sort), at sizes from one small system of a batch service to the largest
benchmark configurations, in both particle types, both curves, both split criteria and both tree kinds.

All results are integers that are determined by the inputs (keys, permutations, leaf boundaries, counts,
node links) or copies of inputs, so there is no rounding to compare with.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import adaptive_trees_b200 as ab
from adaptive_trees_b200 import _capi as C

LARGEST_TREE = 1 << 24        # particles of the largest single tree
BATCH_SIZES = (3.0, 6.0)      # log10 of the smallest and largest system of a batch
TREE_ARRAYS = ("particleKeys_d", "perm_d", "cornerstone_d", "leafCounts_d")
PARTICLE_ARRAYS = ("particleKeys_d", "perm_d", "sfcParticleIndex_d")  # one entry per particle
VIEW_ARRAYS = ("sfcBoxIndex_d", "hasBoxSplit_d", "boxDepth_d", "parentIndex_d", "childIndex_d", "levelOffset_d",
               "particleBeginIndex_d", "particleCounts_d", "sfcParticleIndex_d")


def _tree(op, n, dist, real, *, kind="octree", curve="morton", bucket=64, nf=False, **more):
    return dict(op=op, n=n, dist=dist, real=real, kind=kind, curve=curve, bucket=bucket, nf=nf, **more)


def listed():
    return [
        # one small system built on request: launches and host work, hardly any bytes
        _tree("build", 10_007, "plummer", "f32", curve="hilbert", name="build_10k"),
        # a mid-sized adaptive build whose caller then gathers its charges into key order (odd size)
        _tree("build", 300_007, "plummer", "f32", bucket=512, nf=True, gather=True, name="build_nf_300k"),
        # the plain octree configuration: 2^20 uniform doubles
        _tree("build", 1 << 20, "uniform", "f64", name="build_1Mi"),
        # the headline configuration: 16Mi Plummer floats, near-field refinement
        _tree("build", 1 << 24, "plummer", "f32", curve="hilbert", bucket=512, nf=True, name="build_nf_16Mi"),
        # the k-d tree configuration: 8Mi doubles from anisotropic Gaussians
        _tree("build", 1 << 23, "mixture", "f64", kind="binary", bucket=32, name="build_kd_8Mi"),
        # a time step of a small system: direct update() calls
        _tree("update", 30_011, "plummer", "f32", curve="hilbert", jitter=1e-3, name="update_30k"),
        # a time step with every view the traversal can ask for, replayed from a graph
        _tree("update", 1_000_003, "uniform", "f64", curve="hilbert", jitter=1e-3, graph=True, views=True,
              name="update_views_1M"),
        # a time step of the headline tree, replayed from a graph
        _tree("update", 1 << 24, "plummer", "f32", curve="hilbert", bucket=512, nf=True, jitter=1e-3, graph=True,
              name="update_nf_16Mi"),
        # a time step of the k-d tree
        _tree("update", 1 << 23, "mixture", "f64", kind="binary", bucket=32, jitter=5e-4, name="update_kd_8Mi"),
        # the batched configuration: 512 systems of 10^3 to 10^6 particles built together
        dict(op="batch_build", systems=512, sizes=4, real="f32", curve="morton", bucket=64, name="batch_build_512"),
        # a time step of a batch of systems, replayed from a graph
        dict(op="batch_update", systems=96, sizes=5, real="f32", curve="hilbert", bucket=64, jitter=1e-3,
             name="batch_update_96"),
        # the stand-alone pair sort on the particle keys, with the caller's values (odd size)
        dict(op="sort", n=3_000_017, dist="plummer", real="f32", curve="hilbert", name="sort_3M"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["build", "build", "build", "update", "update", "update", "batch_build", "batch_update", "sort"])
    curve, real = rng.choice(["morton", "hilbert"]), rng.choice(["f32", "f64"])
    dist = rng.choice(["uniform", "plummer", "mixture"])
    if op == "sort":
        return dict(op=op, n=_log_int(rng, 1_000, LARGEST_TREE), dist=dist, real=real, curve=curve)
    if op in ("batch_build", "batch_update"):
        case = dict(op=op, systems=_log_int(rng, 4, 256), sizes=rng.randrange(1 << 20), real="f32", curve=curve,
                    bucket=rng.choice([16, 32, 64, 100]))
        return dict(case, jitter=1e-3) if op == "batch_update" else case
    if rng.random() < 0.3:
        case = _tree(op, _log_int(rng, 2_000, 1 << 23), dist, real, kind="binary",
                     bucket=rng.choice([16, 32, 64]))
    elif rng.random() < 0.45:
        case = _tree(op, _log_int(rng, 5_000, LARGEST_TREE), dist, "f32", curve=curve, bucket=rng.choice([512, 1000]),
                     nf=True)
    else:
        case = _tree(op, _log_int(rng, 2_000, LARGEST_TREE // 2), dist, real, curve=curve,
                     bucket=rng.choice([16, 64, 100]))
    if op == "build":
        case["gather"] = rng.random() < 0.25
    else:
        case["jitter"] = rng.choice([1e-4, 5e-4, 1e-3])
        case["graph"] = rng.random() < 0.5
        # the views hold every node: only trees of few nodes have them
        case["views"] = rng.random() < 0.25 and not case["nf"] and case["n"] <= 2_000_000
    return case


def _dtype(case):
    return torch.float32 if case["real"] == "f32" else torch.float64


def _coordinates(n, dist, dtype, gen):
    """x, y, z in [0, 1): uniform, a Plummer sphere (a = 0.05, r <= 0.5) or a mixture of 8 Gaussians."""
    f64 = dict(dtype=torch.float64, device="cuda", generator=gen)
    upper = float(np.nextafter(np.float32(1.0), np.float32(0.0))) if dtype == torch.float32 else float(
        np.nextafter(1.0, 0.0))
    if dist == "uniform":
        axes = [torch.rand(n, **f64) for _ in range(3)]
    elif dist == "plummer":
        inside = (1.0 + (0.05 / 0.5) ** 2) ** -1.5  # mass fraction within r = 0.5
        u = torch.rand(n, **f64).mul_(inside).clamp_(min=1e-12)
        r = 0.05 / torch.sqrt(u.pow_(-2.0 / 3.0) - 1.0)
        v = torch.randn(3, n, **f64)
        v *= r / v.norm(dim=0)
        axes = [v[k] + 0.5 for k in range(3)]
    else:
        centres = torch.rand(3, 8, **f64) * 0.6 + 0.2
        sigmas = torch.exp(torch.rand(3, 8, **f64) * math.log(10.0) + math.log(0.005))
        which = torch.randint(0, 8, (n,), device="cuda", generator=gen)
        axes = [centres[k][which] + sigmas[k][which] * torch.randn(n, **f64) for k in range(3)]
    return [a.to(dtype).clamp_(0.0, upper).contiguous() for a in axes], upper


def _moved(axes, jitter, upper, gen):
    return [(a + jitter * torch.randn(a.shape, dtype=a.dtype, device="cuda", generator=gen)).clamp_(0.0, upper)
            for a in axes]


def _batch_sizes(case):
    r = np.random.default_rng(case["sizes"])
    sizes = np.floor(10.0 ** r.uniform(*BATCH_SIZES, case["systems"])).astype(np.int64)
    return [int(k) for k in sizes], [bool(p) for p in r.random(case["systems"]) < 0.5]


def _ints(t):
    """The same bytes as a signed type, which every torch operation knows."""
    return t.view({torch.uint64: torch.int64, torch.uint32: torch.int32}.get(t.dtype, t.dtype))


def _bound(case, n):
    """Entries a program reserves for the leaf (or node) arrays of such a tree."""
    return int(2.5 * n) + 4096 if case.get("nf") else n + 4096


def _keep(state, name, t):
    """The leaf arrays of this pass in the program's own arrays of fixed length (the tree reuses its buffers at the
    next step), zeros behind their end."""
    kept, used = state["kept"], state["used"]
    t, n, before = _ints(t), t.numel(), used.get(name, 0)
    if name not in kept:
        kept[name] = torch.zeros(state["bound"], dtype=t.dtype, device="cuda")
    kept[name][:n].copy_(t)
    if before > n:
        kept[name][n:before].zero_()
    used[name] = n
    return kept[name]


def _settle(handle, frames, coords, update):
    """Steps through both frames until the buffers hold either tree, as a program's first steps do."""
    for frame in (frames[1], frames[0], frames[1], frames[0]):
        for c, f in zip(coords, frame):
            c.copy_(f)
        update()
        while handle.doBuffersNeedResize():
            handle.resizeBuffers()
            update()


def _captured(update, stream):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        update()
    return graph


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    op = case["op"]
    stream = torch.cuda.Stream()
    state = dict(op=op, stream=stream, kept={}, used={})
    curve = ab.SfcKind.Hilbert if case.get("curve") == "hilbert" else ab.SfcKind.Morton
    if op == "sort":
        axes, _ = _coordinates(case["n"], case["dist"], _dtype(case), gen)
        n, keys = case["n"], ab.compute_sfc_keys(0, *axes, sfc_kind=curve)
        values = torch.randint(0, 1 << 31, (n,), dtype=torch.int32, device="cuda", generator=gen)
        size = ctypes.c_size_t()
        C.check(C.load().ao_sort_pairs(None, ctypes.byref(size), None, None, None, None, n, 0, 64, None))
        state.update(n=n, keys=keys, values=values, size=size, out=torch.empty_like(keys),
                     out_values=torch.empty_like(values),
                     scratch=torch.empty(size.value, dtype=torch.uint8, device="cuda"))
        torch.cuda.synchronize()
        return state
    if op in ("batch_build", "batch_update"):
        sizes, plummer = _batch_sizes(case)
        parts = [_coordinates(n, "plummer" if p else "uniform", _dtype(case), gen) for n, p in zip(sizes, plummer)]
        upper = parts[0][1]
        coords = [torch.cat([p[0][k] for p in parts]) for k in range(3)]
        offs = np.concatenate([[0], np.cumsum(sizes)])
        each = [[c[offs[i]:offs[i + 1]] for i in range(len(sizes))] for c in coords]
        torch.cuda.synchronize()
        handle = ab.Batch(*each, ab.TreeConfig(maxParticlesPerLeaf=case["bucket"], sfcKind=curve), stream=stream)
        state.update(handle=handle, systems=len(sizes), bound=_bound(case, int(offs[-1])), graph=None)
    else:
        coords, upper = _coordinates(case["n"], case["dist"], _dtype(case), gen)
        views = bool(case.get("views"))
        binary = case["kind"] == "binary"
        config = ab.TreeConfig(maxParticlesPerLeaf=case["bucket"], views=ab.ViewConfig(views, views, views),
                               splitCriterion=ab.SplitCriterion.NFCount if case["nf"] else ab.SplitCriterion.LeafCount,
                               sfcKind=ab.SfcKind.Morton if binary else curve)
        torch.cuda.synchronize()
        handle = ab.Tree(ab.TreeType.Binary if binary else ab.TreeType.Octree, *coords, config, stream=stream)
        arrays = TREE_ARRAYS + (("nearFieldCounts_d",) if case["nf"] else ()) + (VIEW_ARRAYS if views else ())
        state.update(handle=handle, arrays=arrays, bound=_bound(case, case["n"]), graph=None)
        if case.get("gather"):
            state["charges"] = torch.randn(case["n"], 4, device="cuda", generator=gen)
    if op in ("update", "batch_update"):
        frames = [[c.clone() for c in coords], _moved(coords, case["jitter"], upper, gen)]
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            handle.build()
            _settle(handle, frames, coords, handle.update)
        if case.get("graph") or op == "batch_update":
            state["graph"] = _captured(handle.update, stream)
        state.update(frames=frames, coords=coords, at=0)
    torch.cuda.synchronize()
    return state


def _batch_arrays(state):
    """Every array of all systems: the systems lie one after the other in the batch's buffers."""
    batch, out = state["handle"], []
    for name in TREE_ARRAYS:
        first, last = batch.get(0, name), batch.get(state["systems"] - 1, name)
        item = first.element_size()
        count = (last.data_ptr() - first.data_ptr()) // item + last.numel()
        whole = ab.device_tensor(first.data_ptr(), count, "<u8" if item == 8 else "<u4")
        out.append(_ints(whole) if name in PARTICLE_ARRAYS else _keep(state, name, whole))
    return out


def run(state):
    op, stream = state["op"], state["stream"]
    if op == "sort":
        C.check(C.load().ao_sort_pairs(state["scratch"].data_ptr(), ctypes.byref(state["size"]),
                                       state["keys"].data_ptr(), state["out"].data_ptr(), state["values"].data_ptr(),
                                       state["out_values"].data_ptr(), state["n"], 0, 64,
                                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return [_ints(state["out"]), state["out_values"]]
    handle = state["handle"]
    with torch.cuda.stream(stream):
        if op in ("build", "batch_build"):
            handle.build()
            if op == "batch_build":
                handle.doBuffersNeedResize()
        else:
            # the program moves its particles, updates the tree and asks whether its buffers held it
            state["at"] ^= 1
            for c, f in zip(state["coords"], state["frames"][state["at"]]):
                c.copy_(f)
            if state["graph"] is not None:
                state["graph"].replay()
            else:
                handle.update()
            if handle.doBuffersNeedResize():
                while True:
                    handle.resizeBuffers()
                    handle.update()
                    if not handle.doBuffersNeedResize():
                        break
                if state["graph"] is not None:
                    state["graph"] = _captured(handle.update, stream)
        if op in ("batch_build", "batch_update"):
            return _batch_arrays(state)
        out = [_ints(handle.get(name)) if name in PARTICLE_ARRAYS else _keep(state, name, handle.get(name))
               for name in state["arrays"]]
        if "charges" in state:
            out.append(handle.gather(state["charges"]))
        return out


def _leaves(case, n):
    """Leaves of a typical tree of these settings (about)."""
    if case.get("nf"):
        return 0.75 * n * math.sqrt(512.0 / case["bucket"])
    return (1.5 if case.get("kind") == "binary" else 2.5) * n / case["bucket"]


def work(case):
    op, real = case["op"], 4 if case["real"] == "f32" else 8
    if op == "sort":
        return {"bytes": 24 * case["n"], "flops": 0}  # key and value, in and out
    n = sum(_batch_sizes(case)[0]) if op.startswith("batch") else case["n"]
    leaves = _leaves(case, n)
    particle = 3 * real + 8 + 4                       # coordinates in; key and permutation out
    leaf = 8 + 4 + (4 if case.get("nf") else 0)       # boundary, count (and near-field count) out
    if op in ("update", "batch_update"):
        particle += 2 * 3 * real                      # the program's move: a frame in, coordinates out
        leaf += 8                                     # the old boundaries in
    if case.get("views"):
        nodes = leaves * (8.0 / 7.0)
        leaf += nodes / leaves * (8 + 1 + 1 + 4 + 4 + 4 + 4)
        particle += 8
    if case.get("gather"):
        particle += 2 * 16
    return {"bytes": particle * n + leaf * leaves, "flops": 0}
