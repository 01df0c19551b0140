"""Keys by double-float cell numbers, bit for bit the FP64 octant recurrence:
particles on the faces of cells and a rounding beside them, systems far from the
origin, tiny and huge ones, and a plain FP32 state."""
import numpy as np
import pytest

from conftest import octant_keys

pytestmark = pytest.mark.gpu


def check(pkg, x, y, z, precision):
    m = np.full(len(x), 1.0 / len(x))
    if precision == pkg.PRECISION_PLAIN:
        x, y, z = (a.astype(np.float32).astype(np.float64) for a in (x, y, z))
    else:  # what a double-float pair holds
        x, y, z = ((h := a.astype(np.float32).astype(np.float64)) + (a - h).astype(np.float32) for a in (x, y, z))
    with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=0.05 * np.ptp(x), theta=0.7), precision=precision) as sim:
        sim.set_particles(x, y, z, None, None, None, m)
        sim.compute_accel()
        assert np.array_equal(sim.debug_tree()["keys"], octant_keys(x, y, z))


@pytest.mark.parametrize("precision", ["PRECISION_SPLIT", "PRECISION_PLAIN"])
@pytest.mark.parametrize("offset,size", [(0.0, 1.0), (0.3, 1.0), (100.0, 1.0), (3e4, 1.0), (2e6, 1.0), (0.0, 1e-8),
                                         (-5.0, 1e-3), (0.0, 1e12), (1e13, 1e12)])
def test_scattered(pkg, offset, size, precision):
    rng = np.random.default_rng(5)
    x, y, z = offset + size * rng.uniform(-1.0, 1.0, (3, 40000))
    check(pkg, x, y, z, getattr(pkg, precision))


@pytest.mark.parametrize("precision", ["PRECISION_SPLIT", "PRECISION_PLAIN"])
@pytest.mark.parametrize("level", [1, 4, 9, 15, 21])
def test_faces(pkg, level, precision):
    """Particles on, just below and just above faces of the cells of a level."""
    rng = np.random.default_rng(level)
    half = 1.001  # the root of a box [-1, 1]
    k = rng.integers(-(1 << (level - 1)), 1 << (level - 1), (3, 20000))
    face = np.clip(k * (2.0 * half / (1 << level)), -1.0, 1.0)
    near = face + rng.integers(-2, 3, face.shape) * 2.0 ** -rng.integers(30, 52, face.shape)
    x, y, z = np.clip(near, -1.0, 1.0)
    x[:2] = y[:2] = z[:2] = (-1.0, 1.0)
    check(pkg, x, y, z, getattr(pkg, precision))
