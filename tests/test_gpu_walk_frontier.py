"""Walks whose frontier outgrows their stack: trees in which a few cells of
every level split and the rest wait, walked with nothing accepted.  Every
particle then meets every other one, so accelerations equal the direct sum and
steps the KDK step taken with it, whatever a walk does when its stack is full.
Accelerations are held to the parity bars (median 1e-5, max 1e-4); a step's
velocity change is a mean of two accelerations, so to the same."""
import itertools

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

EPS, DT = 0.05, 1e-3
OCTANTS = np.array(list(itertools.product((-1, 1), repeat=3)))[:, ::-1]  # x fastest, as in the keys


def nest(width, levels, per_leaf=1):
    """Positions in the lowest octant of the root cube, split once more into 64
    cells; of these, and of the cells that come of it, the `width` last in key
    order split into eight until there are `levels` levels below the octant.
    Every other cell is left with `per_leaf` (1 or 2) particles, two in opposite
    octants.  One particle more, at (1, 1, 1), holds the root cube."""
    half = 0.5005  # of the root cube: the particles span 0 to 1
    half /= 2
    cells, left = [np.full(3, 0.5 - half)], []
    for level in range(levels):
        split = cells if level < 2 else cells[-width:]
        left += [(c, half) for c in cells[:len(cells) - len(split)]]
        half /= 2
        cells = [c + half * o for c in split for o in OCTANTS]
    left += [(c, half) for c in cells]
    inside = (OCTANTS[0], OCTANTS[7]) if per_leaf == 2 else (0 * OCTANTS[0],)
    p = np.array([c + h / 2 * o for c, h in left for o in inside] + [np.ones(3)])
    p[np.argmin(p.sum(1))] = 0.0
    return p.T.copy(), np.random.default_rng(levels).uniform(0.5, 1.5, len(p)) / len(p)


def direct(x, m):
    a = np.empty_like(x)
    for i in range(x.shape[1]):
        d = x - x[:, i:i + 1]
        a[:, i] = (m * ((d * d).sum(0) + EPS ** 2) ** -1.5 * d).sum(1)
    return a


def bars(a, want):
    e = rel_err(*a, *want)
    assert np.median(e) <= 1e-5 and e.max() <= 1e-4, (np.median(e), e.max())


def system(pkg, x, m, theta=0.0, **kw):
    sim = pkg.NBodySystem(pkg.StepParams(G=1.0, eps=EPS, theta=theta), leaf_capacity=1, **kw)
    sim.set_particles(*x, None, None, None, m.astype(np.float32).astype(np.float64))
    return sim


@pytest.mark.parametrize("kind", ["relative", "block"])
@pytest.mark.parametrize("width,levels", [(32, 3), (32, 8), (40, 19)])
def test_per_particle_walk(pkg, kind, width, levels):
    """At 8 levels and at 19 more than the 1,024 nodes that a walk keeps would wait."""
    x, m = nest(width, levels)
    with system(pkg, x, m, mac=pkg.MAC_RELATIVE if kind == "relative" else pkg.MAC_GEOMETRIC) as sim:
        if kind == "relative":
            sim.set_mac_alpha(1e-30)  # the relative test accepts nothing either
        sim.prime()
        m = m.astype(np.float32).astype(np.float64)
        a0 = direct(x, m)
        bars(sim.accel(), a0)
        if kind == "relative":
            sim.step(1, DT)
        else:
            sim.block_step(DT, eta=1e3, max_rung=0)
        st = sim.stats()
        assert st["p2p_pairs"] == len(m) * (len(m) - 1) and st["p2c_terms"] == 0
        a1 = direct(x + DT * (0.5 * DT * a0), m)
        bars(sim.accel(), a1)
        bars(np.array(sim.state()[3:6]) / DT, 0.5 * (a0 + a1))


@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("stack,levels", [(1024, 8), (2048, 14)])
def test_grouped_walk_leaves_shared_memory(pkg, learned, stack, levels):
    """stack / 4 opened nodes fit in shared memory; these trees have more."""
    x, m = nest(8, levels, per_leaf=2)
    with system(pkg, x, m) as sim:
        sim.set_tuning(p2p_tile=0, walk_stack=stack)
        if learned:
            open_everything(pkg, sim, rho_hi=1e-6)
        bars(sim.compute_accel(), direct(x, m.astype(np.float32).astype(np.float64)))
        st = sim.stats()
    assert st["walk_stack_max"] > stack
    assert st["p2p_pairs"] == len(m) * (len(m) - 1) and st["p2c_terms"] == 0


def open_everything(pkg, sim, **opts):
    """The learned walk with a network that never decides (the geometric test
    does) and a band that starts at rho_lo = 0."""
    sim.lmac_set_model(np.zeros(1377, np.float32), np.ones(16, np.float32))
    sim.lmac_set_opts(gate=1e30, rho_lo=0.0, check_every=0, screen=0.0, **opts)
    sim.prime()  # the learned test reads accelerations
    sim.set_opts(mac=pkg.MAC_LEARNED)


def test_learned_walk_outgrows_the_global_stack(pkg):
    """A round that opens 4,096 nodes at once: the global-memory stack, 2,048
    opened nodes at first, is doubled."""
    x, m = nest(4096, 4, per_leaf=2)  # all 4,096 cells of a level split
    with system(pkg, x, m) as sim:
        open_everything(pkg, sim, rho_hi=1e30, rounds=8)
        bars(sim.compute_accel(), direct(x, m.astype(np.float32).astype(np.float64)))
        st = sim.stats()
    assert st["walk_stack_max"] > 4 * 2048
    assert st["p2p_pairs"] == len(m) * (len(m) - 1) and st["p2c_terms"] == 0
