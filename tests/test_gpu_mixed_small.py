"""The mixed sum of a small system in one launch of clusters: partial tiles, warps and CTAs without a tile, and the most tiles per warp.

Tolerance, that of the mixed path: |a - a_ref| <= 1e-6 sum_j |pair term|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 65, 1000, 1023, 1025, 2047, 2048, 2049, 4095])
@pytest.mark.parametrize("eps", [0.0, 0.01])
def test_small_systems_by_clusters(nb, oracle, n, eps):
    x, y, z, vx, vy, vz, m = nb.plummer(n, seed=n)
    m *= np.linspace(0.5, 2.0, n)
    with nb.Sim(nb.Config(method=nb.DIRECT_MIXED, G=1.5, softening=eps), capacity=n) as s:
        s.load(x, y, z, vx, vy, vz, m)
        s.compute_forces()
        a = s.accelerations()
    ref = oracle.forces_naive(x, y, z, m, 1.5, eps)
    sabs = oracle.forces_abs_sum(x, y, z, m, 1.5, eps)
    d = np.sqrt(sum((u - v) ** 2 for u, v in zip(a, ref)))
    assert (d <= 1e-6 * sabs).all(), (d / np.maximum(sabs, 1e-300)).max()
