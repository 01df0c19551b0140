"""The per-particle walk at the edges of its slices, windows and batches:
particle counts around a slice of members, leaves of one particle up to
leaves larger than a batch, several systems in a slice, every precision and
softening.  Interaction counts equal the oracle's; accelerations are within
the parity bars (median 1e-5, max 1e-4) of its FP64 walk."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def check(pkg, oracle, arrs, eps, theta, leaf, precision=1, quadrupole=True):
    x, y, z, m = (np.asarray(a, np.float32).astype(np.float64) for a in arrs)
    with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=eps, theta=theta), leaf_capacity=leaf, precision=precision,
                         quadrupole=quadrupole, mac=pkg.MAC_RELATIVE) as sim:
        sim.set_particles(x, y, z, None, None, None, m)
        a = sim.compute_accel()  # no previous |a|: the geometric test per particle
        st = sim.stats()
    r = oracle.bh_pp_accel(x, y, z, m, 1.0, eps, theta, leaf, quad=quadrupole, counters=True)
    assert st["p2p_pairs"] == r[3][0] and st["p2c_terms"] == r[3][1]
    if len(x) > 1:
        e = rel_err(*a, *r[:3])
        assert np.median(e) <= 1e-5 and e.max() <= 1e-4, (np.median(e), e.max())
    else:
        assert all(np.all(c == 0.0) for c in a)


@pytest.mark.parametrize("leaf", [1, 8, 300])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 33, 64, 65, 129, 1001])
def test_counts_and_forces(pkg, oracle, ic, n, leaf):
    x, y, z, _, _, _, m = ic.plummer(n, seed=n)
    check(pkg, oracle, (x, y, z, m), 0.05, 0.6, leaf)


@pytest.mark.parametrize("quadrupole", [True, False])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("eps", [0.0, 0.01])
def test_options(pkg, oracle, ic, precision, quadrupole, eps):
    x, y, z, _, _, _, m = ic.galaxy(2701, 300, seed=2)
    check(pkg, oracle, (x, y, z, m), eps, 0.7, 8, precision, quadrupole)


def test_slices_across_systems(pkg, ic):
    """Systems of odd sizes share slices; each gets its own walk's result."""
    sizes = [1, 2, 5, 131, 3, 400]
    parts = [ic.plummer(k, seed=i) for i, k in enumerate(sizes)]
    arrs = [np.concatenate([p[c] for p in parts]) for c in range(7)]
    sp = pkg.StepParams(G=1.0, eps=0.05, theta=0.6)
    with pkg.NBodySystem(sp, mac=pkg.MAC_RELATIVE) as sim:
        sim.set_particles_f32(*arrs)
        sim.set_ensemble(np.concatenate([[0], np.cumsum(sizes)]))
        a = np.array(sim.compute_accel())
    at = 0
    for p, k in zip(parts, sizes):
        with pkg.NBodySystem(sp, mac=pkg.MAC_RELATIVE) as one:
            one.set_particles_f32(*p)
            b = np.array(one.compute_accel())
        # the same terms in another grouping: FP32 terms, compensated sums
        scale = np.maximum(np.sqrt(np.sum(b ** 2, axis=0)), 1e-30)
        assert np.max(np.sqrt(np.sum((a[:, at:at + k] - b) ** 2, axis=0)) / scale) <= 2e-6
        at += k
