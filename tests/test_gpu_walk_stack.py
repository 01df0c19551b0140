"""The grouped walk's stack of opened nodes: nodes with one to eight children,
more than a batch of opened nodes at once, frontiers that outgrow the smallest
stack.  The tests taken and the interactions found equal the oracle's, whatever
the stack."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stack", [1024, 2048, 4096])
@pytest.mark.parametrize("shape,n,leaf,theta", [
    ("ball", 2, 1, 0.5), ("ball", 9, 1, 0.5), ("ball", 65, 1, 1.5), ("ball", 700, 2, 0.0), ("ball", 4000, 1, 0.05),
    ("ball", 30000, 1, 0.25), ("ball", 30000, 32, 0.02),
    ("line", 2, 1, 0.5), ("line", 9, 1, 0.5), ("line", 65, 1, 1.5), ("line", 700, 2, 0.0), ("line", 30000, 32, 0.02)])
def test_counts(pkg, oracle, ic, shape, n, leaf, theta, stack):
    x, y, z, _, _, _, m = ic.plummer(n, seed=n + leaf)
    x, y, z, m = (np.asarray(a, np.float32).astype(np.float64) for a in (x, y, z, m))
    if shape == "line":  # at most two children per node, many levels
        y, z = np.zeros(n), np.zeros(n)
    with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=0.05, theta=theta), leaf_capacity=leaf) as sim:
        sim.set_tuning(p2p_tile=0, walk_stack=stack)
        sim.set_particles(x, y, z, None, None, None, m)
        sim.compute_accel()
        st = sim.stats()
    cnt = oracle.bh_accel(x, y, z, m, 1.0, 0.05, theta, leaf, counters=True)[3]
    keys = ("p2p_pairs", "p2c_terms", "mac_tests")
    assert [st[k] for k in keys] == [cnt[k] for k in keys]
