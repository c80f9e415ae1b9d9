"""The all-pairs mixed sum over unordered pairs at the sizes where it can go
wrong: the change from ordered pairs, the edges of the 64-body tiles, of the pairs
of tiles and of the 256-body blocks, odd and even numbers of blocks, tiles of one
mass and of several.

Tolerance, that of the mixed path: |a - a_ref| <= 1e-6 sum_j |pair term|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [4095, 4096, 4097, 4159, 4161, 4225, 4289, 4353, 4609, 6000, 8192, 16390]


@pytest.mark.parametrize("n", SIZES)
def test_unordered_pairs_at_tile_edges(nb, oracle, n):
    x, y, z, vx, vy, vz, m = nb.plummer(n, seed=n)
    for k, eps in enumerate((0.0, 0.01)):
        if k:  # half of the tiles of one mass, half of many
            m[: n // 2] *= np.linspace(0.5, 2.0, n // 2)
        cfg = nb.Config(method=nb.DIRECT_MIXED, G=1.5, softening=eps, flags=nb.MIXED_UNSORTED)
        with nb.Sim(cfg, capacity=n) as s:
            s.load(x, y, z, vx, vy, vz, m)
            s.compute_forces()
            a = s.accelerations()
            s.compute_forces()
            for u, v in zip(a, s.accelerations()):
                assert np.array_equal(u, v)
        ref = oracle.forces_naive(x, y, z, m, 1.5, eps)
        sabs = oracle.forces_abs_sum(x, y, z, m, 1.5, eps)
        d = np.sqrt(sum((u - v) ** 2 for u, v in zip(a, ref)))
        assert (d <= 1e-6 * sabs).all(), (n, eps, (d / sabs).max())
