"""The evaluation kernel at the edges of its windows: source counts around
64, 128, 256 and 1,024 (windows, batches), target counts around a pass, leaves
larger than a batch, far lists around a list chunk.  Interaction counts equal
the oracle's; accelerations are within the parity bars (median 1e-5, max 1e-4)
of its FP64 sums over the same interactions."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

SPLIT, PLAIN = 1, 0


def check(pkg, oracle, arrs, eps, theta, leaf, precision=SPLIT, quadrupole=True, tile=0):
    x, y, z, m = (np.asarray(a, np.float32).astype(np.float64) for a in arrs)
    with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=eps, theta=theta), leaf_capacity=leaf, precision=precision,
                         quadrupole=quadrupole) as sim:
        sim.set_tuning(p2p_tile=tile, walk_stack=2048)
        sim.set_particles(x, y, z, None, None, None, m)
        a = sim.compute_accel()
        st = sim.stats()
    r = oracle.bh_accel(x, y, z, m, 1.0, eps, theta, leaf, quad=quadrupole, counters=True)
    assert (st["p2p_pairs"], st["p2c_terms"]) == (r[3]["p2p_pairs"], r[3]["p2c_terms"])
    if len(x) > 1:
        e = rel_err(*a, *r[:3])
        assert np.median(e) <= 1e-5 and e.max() <= 1e-4, (np.median(e), e.max())
    else:
        assert all(np.all(c == 0.0) for c in a)


@pytest.mark.parametrize("precision", [SPLIT, PLAIN])
@pytest.mark.parametrize("n", [1, 2, 20, 21, 40, 41, 63, 64, 65, 127, 129, 191, 193, 255, 256, 257, 1023, 1025, 2500])
def test_one_leaf(pkg, oracle, ic, n, precision):
    """Every particle in one leaf: n sources against n targets in passes."""
    x, y, z, _, _, _, m = ic.plummer(n, seed=n)
    check(pkg, oracle, (x, y, z, m), 0.05, 0.5, 4096, precision)


@pytest.mark.parametrize("tile", [0, 64, 128, 256])
@pytest.mark.parametrize("leaf", [1, 3, 8, 21, 64, 300, 1500])
def test_leaf_sizes_and_tiles(pkg, oracle, ic, leaf, tile):
    x, y, z, _, _, _, m = ic.plummer(3000, seed=leaf)
    check(pkg, oracle, (x, y, z, m), 0.02, 0.6, leaf, tile=tile)


@pytest.mark.parametrize("quadrupole", [True, False])
@pytest.mark.parametrize("precision", [SPLIT, PLAIN])
@pytest.mark.parametrize("theta", [0.25, 0.5, 1.5])
def test_far_lists(pkg, oracle, ic, theta, precision, quadrupole):
    x, y, z, _, _, _, m = ic.galaxy(5401, 600, seed=4)
    check(pkg, oracle, (x, y, z, m), 0.01, theta, 8, precision, quadrupole)


def test_unsoftened(pkg, oracle, ic):
    """eps = 0: the self pair is masked, window pads stay out of range."""
    x, y, z, _, _, _, m = ic.plummer(1500, seed=9)
    check(pkg, oracle, (x, y, z, m), 0.0, 0.5, 16)
