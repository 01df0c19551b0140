"""Half-kicks in split precision: v + h a as a double-float pair, the product
exact, so a step's velocity change is that of FP64 to the pair's 2^-47 (three
roundings of a kick, two kicks; h and the accelerations are float32 numbers)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["geometric", "relative", "block"])
def test_kick_is_exact_to_the_pair(pkg, ic, kind):
    x, y, z, vx, vy, vz, m = ic.plummer(5003, seed=8)
    dt = 0.37
    with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=0.05, theta=0.6), leaf_capacity=16,
                         mac=pkg.MAC_RELATIVE if kind == "relative" else pkg.MAC_GEOMETRIC) as sim:
        sim.set_particles_f32(x, y, z, vx, vy, vz, m)
        sim.prime()
        v0, a0 = np.array(sim.state()[3:6]), np.array(sim.accel())
        if kind == "block":
            sim.block_step(dt, eta=1e3, max_rung=0)
        else:
            sim.step(1, dt)
        v1, a1 = np.array(sim.state()[3:6]), np.array(sim.accel())
    h = float(np.float32(0.5 * dt))
    want = v0 + h * a0 + h * a1
    size = np.maximum.reduce([np.abs(v0), np.abs(h * a0), np.abs(h * a1), np.abs(v0 + h * a0)])
    assert np.max(np.abs(v1 - want) / size) <= 6 * 2.0 ** -47
