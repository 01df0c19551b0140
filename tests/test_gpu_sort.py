"""The key sort at the edges of its forms: one key, a warp, one CTA of 512 and of
1,024 threads, tiles beyond; odd and even numbers of passes; many equal keys.
The order equals a stable sort of the keys' sorted digits (kept between two
evaluations by the leaves), and the state follows it."""
import numpy as np
import pytest

from conftest import octant_keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("equal", [False, True])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 257, 4095, 4096, 4097, 8191, 8192, 8193, 12289, 70001])
def test_order(pkg, oracle, n, equal):
    rng = np.random.default_rng(n)
    x, y, z = (a.astype(np.float32).astype(np.float64) for a in rng.normal(size=(3, n)))
    if equal and n > 2:  # a third of the particles in one place
        x[::3], y[::3], z[::3] = 0.25, 0.5, -0.75
    m = np.full(n, 2.0 ** -17)
    with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=0.5, theta=0.8), leaf_capacity=8, max_depth=12) as sim:
        sim.set_particles(x, y, z, None, None, None, m)
        for _ in range(2):  # the full key, then the digits in use
            sim.compute_accel()
            t = sim.debug_tree()
            keys = octant_keys(x, y, z)
            assert np.array_equal(t["keys"], keys)
            assert np.array_equal(t["order"], oracle.tree(x, y, z, m, 8, 12)["order"])
        pos = np.stack(sim.state()[:3])
    assert np.array_equal(pos, np.stack([x, y, z]))
