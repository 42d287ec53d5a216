"""What a served tree holds is what the server counts against its budget."""
import numpy as np
import pytest

from .gpu_util import tree_config
from .scenarios import uniform_cube

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def block(bytes_):
    """Size class of a device block: the next 2^k or 1.5 * 2^k bytes."""
    top = 1 << (bytes_.bit_length() - 1)
    return bytes_ if bytes_ == top else top + top // 2 if bytes_ <= top + top // 2 else 2 * top


def test_binary_tree_counts_the_arena_of_its_build():
    import adaptive_trees_b200 as ab
    n = 100_003
    x = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in uniform_cube(n, seed=1)]
    torch.cuda.synchronize()
    server = ab.Server(slots=1)
    r = server.wait(server.build(0, *x, config=tree_config(bucket=1), kind=1))
    assert r["status"] == 0, r["message"]
    held = server.stats()["resident_bytes"]
    server.close()
    leaves, units = 4 * n + 4096, n + 4096  # capacities the build starts with
    particles = 5 * block(8 * n) + 2 * block(4 * n)           # coordinates, keys, permutation
    arrays = 2 * block(8 * (leaves + 1)) + 8 * block(4 * (leaves + 1))  # K; B, N, NF, offsets, dirty
    arena = block(48 * units) + block(32 * units) + block(8 * units) + 2 * block(4 * units)
    assert held >= particles + arrays + arena, (held, particles, arrays, arena)
