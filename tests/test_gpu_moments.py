"""Leaf and internal moments at the edges of their work splits: leaves per warp
(4 to 32), members per leaf (1 to more than a mask of 64), leaves whose members
are all equally far from the centre of mass, trees whose levels go to the
cluster and to the grid.

The oracle's running FP64 sums over n insertions are good to n roundings, the
leaf sums here (double-float pairs) to 2^-46 of the coordinates, so a mass, a
centre and a radius may differ by (n + 64) 2^-52; the quadrupole tolerance is
the parity tests'."""
import numpy as np
import pytest

from conftest import TREE_EXACT

pytestmark = pytest.mark.gpu


def lattice(k):
    g = (np.arange(k) + 0.5) / k
    x, y, z = (a.ravel() for a in np.meshgrid(g, g, g, indexing="ij"))
    return x, y, z, np.full(k ** 3, 1.0 / k ** 3)


@pytest.mark.parametrize("shape,n,leaf", [
    ("ball", 1, 8), ("ball", 7, 8), ("ball", 9, 8), ("ball", 2431, 1), ("ball", 2433, 1), ("ball", 4865, 1),
    ("ball", 16383, 1), ("ball", 16385, 1), ("ball", 20000, 65), ("ball", 20000, 300), ("ball", 40000, 40000),
    ("ball", 1500000, 130), ("lattice", 32768, 8), ("lattice", 32768, 512), ("lattice", 262144, 8)])
def test_moments(pkg, oracle, ic, shape, n, leaf):
    x, y, z, m = lattice(round(n ** (1 / 3))) if shape == "lattice" else (ic.plummer(n, seed=n)[k] for k in (0, 1, 2, 6))
    x, y, z, m = (np.asarray(a, np.float32).astype(np.float64) for a in (x, y, z, m))
    if shape == "ball" and n > 9:
        m[::5] *= 2.0 ** -20
        m[:3] = 0.25
    with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=0.05, theta=0.7), leaf_capacity=leaf) as sim:
        sim.set_particles(x, y, z, None, None, None, m)
        sim.compute_accel()
        c = pkg.canonical(sim.debug_tree())
    g = pkg.canonical(oracle.tree(x, y, z, m, leaf))
    for k in TREE_EXACT:
        assert np.array_equal(c[k], g[k]), k
    eps = (n + 64) * 2.0 ** -52
    size = max(1.0, np.abs(g["com"]).max())
    np.testing.assert_allclose(c["mass"], g["mass"], rtol=eps, atol=0)
    np.testing.assert_allclose(c["com"], g["com"], rtol=0, atol=eps * size)
    np.testing.assert_allclose(c["max_radius"], g["max_radius"], rtol=0, atol=2 * eps * size)
    qs = g["mass"][:, None] * g["half"][:, None] ** 2
    assert np.all(np.abs(c["quad"] - g["quad"]) <= 1e-5 * qs + 1e-30)
