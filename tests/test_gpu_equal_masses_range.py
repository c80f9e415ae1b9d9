"""Equal masses and a softening far above the system's size, in units where r^-3 leaves
FP32's range though m r^-3 does not: the sums over unordered pairs, whose loop for equal
masses leaves the mass out, take the general loop there.

Tolerance, that of the mixed path: |a - a_ref| <= 1e-6 sum_j |pair term|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [1e-12, 1e-3, 1e10, 1e11, 3e11, 1e13, 3e14])
def test_softening_beyond_the_equal_mass_loop(nb, oracle, eps):
    n = 4300
    x, y, z, vx, vy, vz, _ = nb.plummer(n, seed=3)
    scale = max(1.0, min(eps, 1e10) / 10.0)
    x, y, z = x * scale, y * scale, z * scale
    m = np.full(n, 1e30 if eps > 1.0 else 1.0)
    ref, sabs = oracle.forces_naive(x, y, z, m, 1.0, eps), oracle.forces_abs_sum(x, y, z, m, 1.0, eps)
    cfg = nb.Config(method=nb.DIRECT_MIXED, G=1.0, softening=eps)
    with nb.Sim(cfg, capacity=n) as s:
        s.load(x, y, z, vx, vy, vz, m)
        s.compute_forces()
        got = [s.accelerations()]
    for flags in (0, nb.MIXED_UNSORTED):
        cfg.flags = flags
        with nb.Ensemble(cfg, [n]) as e:
            e.load(x, y, z, vx, vy, vz, m)
            e.compute_forces()
            st = e.read_state()
            got.append([st[k] for k in ("ax", "ay", "az")])
    for a in got:
        d = np.sqrt(sum((u - v) ** 2 for u, v in zip(a, ref)))
        assert (d <= 1e-6 * sabs).all(), (d / sabs).max()
