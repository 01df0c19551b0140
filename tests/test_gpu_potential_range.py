"""The exact pair potential where masses, lengths or single pairs are far from
the rest: light particles round a heavy one in large units, coordinates at the
ends of FP32's range, a few pairs that carry the energy.  Compared with an FP64
pair sum (numpy, compensated over the rows) of the same float32 masses and
double-float positions.

Tolerance: 1e-14 of the sum.  An FP64 term is good to a few 2^-53 (the
reference's too) and both sides add up 10^7 terms of one sign per thousands of
partial sums: 1e-15 with room."""
import numpy as np
import pytest

from test_gpu_potential import pair_sum

pytestmark = pytest.mark.gpu

TOL = 1e-14


def check(pkg, x, y, z, m, eps, spline=False, sort=False, precision=1, tol=TOL):
    with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=eps, theta=0.6), leaf_capacity=16, precision=precision) as sim:
        if spline:
            sim.set_softening(pkg.SOFTENING_SPLINE)
        sim.set_particles(x, y, z, None, None, None, m)
        if sort:
            sim.prime()
        got = sim.diagnostics(exact_potential=1)
        st = sim.state()
    want = pair_sum(*st[:3], np.asarray(m, np.float32).astype(np.float64), eps, spline)
    assert got["potential_exact"] == 1 and np.isfinite(want)
    assert abs(got["potential"] - want) <= tol * abs(want), (got["potential"], want)


def plummer(ic, n, seed=4):
    x, y, z, _, _, _, _ = ic.plummer(n, seed=seed)
    return [np.float64(a) for a in (x, y, z)]


@pytest.mark.parametrize("at", [0, 40, 2600, 4999])
@pytest.mark.parametrize("length,heavy,light", [(1e9, 1.0, 1e-30), (5e11, 2e30, 1.0), (1e-9, 1e-3, 1e-33), (1.0, 1.0, 1e-37)])
def test_heavy_body_and_tracers(pkg, ic, length, heavy, light, at):
    """Tracers down to 1e-37 of the heavy body's mass, which is the first, one of
    the first or the last in the order of the pairs."""
    x, y, z = (a * length for a in plummer(ic, 5000))
    m = np.full(5000, light) * np.random.default_rng(1).uniform(0.5, 1.5, 5000)
    m[at] = heavy
    check(pkg, x, y, z, m, 0.01 * length)


@pytest.mark.parametrize("spline", [False, True])
@pytest.mark.parametrize("length", [1e30, 1e36, 1.5e37])
def test_extent_near_the_end_of_fp32(pkg, ic, length, spline):
    """Squares of the distances are past FP32's range, at 1.5e37 some differences too."""
    x, y, z = (a * length for a in plummer(ic, 5000))
    check(pkg, x, y, z, np.full(5000, 1.0 / 5000), 0.01 * length, spline)


def heavy_pair(ic, n, gap):
    """A wide set with bodies 1 and 20 `gap` of its extent apart."""
    x, y, z = plummer(ic, n)
    d = gap / 3 * max(np.abs(a).max() for a in (x, y, z))
    x[20], y[20], z[20] = x[1] + d, y[1] - 2 * d, z[1] + 2 * d * (1 + 1e-11)
    return x, y, z


@pytest.mark.parametrize("sort", [False, True])
@pytest.mark.parametrize("n", [4096, 5000, 9000])
@pytest.mark.parametrize("gap", [0.0442, 0.06, 0.1, 0.3])
def test_heavy_pair_in_a_wide_frame(pkg, ic, gap, n, sort):
    """Two bodies that carry nearly all of the energy, from just above the 1/16 of
    their frame's extent below which a pair is formed by itself."""
    m = np.full(n, 1e-9 / n)
    m[1], m[20] = 0.7, 0.3
    check(pkg, *heavy_pair(ic, n, gap), m, 0.0, sort=sort)


@pytest.mark.parametrize("gap", [0.0442, 0.06, 0.1, 0.3])
def test_masses_of_both_signs(pkg, ic, gap):
    """The same with a negative mass: what a pair's share is of the sum of sizes
    says nothing about its share of the sum."""
    m = np.random.default_rng(9).uniform(-1.0, 1.0, 5000) * 1e-9 / 5000
    m[1], m[20] = 0.7, -0.3
    check(pkg, *heavy_pair(ic, 5000, gap), m, 0.0)


@pytest.mark.parametrize("heavy", [3, 200])
def test_few_heavy_bodies(pkg, ic, heavy):
    """A handful of bodies, and a few hundred, with all but 1e-6 of the mass."""
    x, y, z = plummer(ic, 6000)
    rng = np.random.default_rng(heavy)
    m = rng.uniform(0.5, 1.5, 6000) * 1e-6 / 6000
    m[rng.choice(6000, heavy, replace=False)] = rng.uniform(0.5, 1.5, heavy) / heavy
    check(pkg, x, y, z, m, 1e-3, sort=True)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("eps", [0.002, 0.01, 0.05])
def test_errors_do_not_lean(pkg, ic, eps, precision):
    """Roundings that lean one way add up over the pairs.  The errors of FP64 sums
    at this size are 2e-16 to 4e-16 and independent (CPU emulation, 4,096 to
    16,384 bodies), so the mean of six has a deviation of 1.6e-16 at most; the bar
    is three of these."""
    errors = []
    for seed in range(6):
        x, y, z, _, _, _, m = ic.galaxy(5400, 600, seed=seed) if seed % 2 else ic.plummer(6000, seed=seed)
        x, y, z = (np.float64(a) + 1e-9 for a in (x, y, z))
        with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=eps, theta=0.6), leaf_capacity=16, precision=precision) as sim:
            sim.set_particles(x, y, z, None, None, None, m)
            sim.prime()
            got = sim.diagnostics(exact_potential=1)["potential"]
            st = sim.state()
        want = pair_sum(*st[:3], np.asarray(m, np.float32).astype(np.float64), eps, False)
        errors.append((got - want) / abs(want))
    assert abs(np.mean(errors)) <= 5e-16, errors
