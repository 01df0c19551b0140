"""The tree read off the sorted keys, bit for bit the oracle's: sizes around a
warp and around the segments of the count (32 x 7,296 particles), capacities
from one to more than the particles, coincident particles, depth limits, a node
pool that overflows, a second build on fewer key digits."""
import numpy as np
import pytest

from conftest import TREE_EXACT

pytestmark = pytest.mark.gpu


def points(ic, shape, n):
    x, y, z, _, _, _, m = ic.plummer(n, seed=n)
    x, y, z, m = (np.asarray(a, np.float32).astype(np.float64) for a in (x, y, z, m))
    if shape == "pairs":  # every particle twice, and one place of a hundred
        x, y, z = (np.concatenate([a[:n // 2], a[:n - n // 2]]) for a in (x, y, z))
        x[:100], y[:100], z[:100] = 0.3, 0.1, -0.2
    return x, y, z, m


@pytest.mark.parametrize("shape,n,leaf,depth", [
    ("ball", 1, 1, 40), ("ball", 2, 1, 40), ("ball", 31, 8, 40), ("ball", 32, 1, 40), ("ball", 33, 32, 40),
    ("ball", 33, 33, 40), ("ball", 1000, 999, 40), ("ball", 5000, 1, 40), ("ball", 5000, 8, 0), ("ball", 5000, 8, 1),
    ("ball", 5000, 8, 3), ("ball", 20000, 100, 40), ("ball", 233471, 16, 40), ("ball", 233473, 16, 40),
    ("ball", 466945, 7, 40), ("pairs", 4000, 8, 10), ("pairs", 4000, 1, 6), ("pairs", 4000, 300, 40)])
def test_topology(pkg, oracle, ic, shape, n, leaf, depth):
    x, y, z, m = points(ic, shape, n)
    g = pkg.canonical(oracle.tree(x, y, z, m, leaf, depth))
    with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=0.05, theta=0.7), leaf_capacity=leaf, max_depth=depth) as sim:
        sim.set_particles(x, y, z, None, None, None, m)
        for again in (False, True):
            if again and n > 2000:
                sim.debug_shrink_pools(node_cap=max(64, len(g["level"]) // 3))
            sim.compute_accel()
            c = pkg.canonical(sim.debug_tree())
            for k in TREE_EXACT:
                assert np.array_equal(c[k], g[k]), k
            st = sim.stats()
            assert st["nodes"] == len(g["level"]) and st["leaves"] == int(np.sum(g["is_leaf"]))
            assert st["levels"] == g["level"].max()
            assert st["max_leaf_count"] == g["count"][g["is_leaf"] != 0].max()
