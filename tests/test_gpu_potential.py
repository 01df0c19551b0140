"""The exact pair potential of the diagnostics against an FP64 pair sum
(numpy, compensated over the rows) of the state's own positions.

From 4,096 particles on, the terms are float pairs: 1/r to 2^-43 at worst (a
pair at 1/16 of its frame's extent, differences good to 2^-47 of that
extent), so the sum is within 2^-43 = 1.1e-13 of the FP64 one however the
errors align; below, FP64 terms."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1.2e-13


def phi(q):
    t = np.maximum(2.0 - q, 0.0)
    F = t ** 4 / 4 - t ** 5 / 5 + t ** 6 / 24
    inner = -(1.4 - 2 / 3 * q ** 2 + 0.3 * q ** 4 - 0.1 * q ** 5)
    with np.errstate(divide="ignore", invalid="ignore"):
        outer = -((1 - 4 * F) / q + t ** 4 / 2 - t ** 5 / 5)
    return np.where(q < 1, inner, outer)


def pair_sum(x, y, z, m, eps, spline):
    rows = []
    for i in range(len(x) - 1):
        r2 = (x[i + 1:] - x[i]) ** 2 + (y[i + 1:] - y[i]) ** 2 + (z[i + 1:] - z[i]) ** 2
        f = phi(np.sqrt(r2) / eps) / eps if spline else -1.0 / np.sqrt(r2 + eps * eps)
        rows.append(m[i] * float(np.sum(m[i + 1:] * f)))
    return math.fsum(rows)


def check(pkg, arrs, eps, spline=False, precision=None, sort=True, tol=TOL):
    x, y, z, vx, vy, vz, m = arrs
    with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=eps, theta=0.6), leaf_capacity=16,
                         precision=pkg.PRECISION_SPLIT if precision is None else precision) as sim:
        if spline:
            sim.set_softening(pkg.SOFTENING_SPLINE)
        sim.set_particles(x, y, z, vx, vy, vz, m)
        if sort:
            sim.prime()
        got = sim.diagnostics(exact_potential=1)
        st = sim.state()
    want = pair_sum(*st[:3], np.asarray(m, np.float32).astype(np.float64), eps, spline)
    assert got["potential_exact"] == 1
    assert abs(got["potential"] - want) <= tol * abs(want), (got["potential"], want)


@pytest.mark.parametrize("n", [1, 2, 33, 129, 2048, 4095, 4096, 4097, 9001])
def test_sizes(pkg, ic, n):
    arrs = [a.astype(np.float64) + 1e-9 for a in ic.plummer(n, seed=n)]  # low halves in use
    check(pkg, arrs, 0.01)


@pytest.mark.parametrize("spline", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("sort", [False, True])
@pytest.mark.parametrize("eps", [1e-4, 0.05, 3.0])
def test_softening_precision_order(pkg, ic, spline, precision, sort, eps):
    check(pkg, ic.galaxy(4500, 501, seed=3), eps, spline, precision, sort)


@pytest.mark.parametrize("length,mass", [(1e12, 1e30), (1e-12, 1e-30), (3e18, 1.0), (1e-18, 1.0)])
def test_units(pkg, ic, length, mass):
    """Units far from one: the frames are scaled, so nothing is lost."""
    x, y, z, vx, vy, vz, m = ic.plummer(5000, seed=2)
    check(pkg, [a * length for a in np.float64((x, y, z))] + [vx, vy, vz, m.astype(np.float64) * mass], 0.01 * length,
          sort=length < 1e15 and length > 1e-15)


def test_uneven_masses_and_close_pairs(pkg, ic):
    x, y, z, vx, vy, vz, m = (a.astype(np.float64) for a in ic.plummer(6000, seed=5))
    m = m * 10.0 ** np.random.default_rng(1).uniform(-12, 0, len(m))
    x[1::2], y[1::2], z[1::2] = x[::2] * (1 + 1e-11), y[::2] + 1e-12, z[::2]  # binaries at rounding distance
    check(pkg, (x, y, z, vx, vy, vz, m), 0.0, tol=1e-12)


def test_coincident_unsoftened_pair_is_infinite(pkg, ic):
    x, y, z, vx, vy, vz, m = ic.plummer(5000, seed=6)
    x[7], y[7], z[7] = x[4000], y[4000], z[4000]
    with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=0.0, theta=0.6), leaf_capacity=16) as sim:
        sim.set_particles(x, y, z, vx, vy, vz, m)
        assert sim.diagnostics(exact_potential=1)["potential"] == -np.inf
