"""The Hilbert-sorted direct sum over tile pairs at the sizes and masses where it
can go wrong: the edges of its 64-body tiles and 256-body blocks, odd and even
numbers of blocks, tiles of one mass (the equal-mass loop), of several and of
both kinds, and units in which r^-3 leaves FP32's range though m r^-3 does not (the
general loop: metres and kilograms, and a small-scale counterpart).

Tolerance, that of the mixed path: |a - a_ref| <= 1e-6 sum_j |pair term|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 63, 64, 65, 255, 256, 257, 511, 513, 767, 1025, 1600, 2303]


@pytest.mark.parametrize("masses", ["equal", "two_species", "mixed", "all_different"])
@pytest.mark.parametrize("scale, mass", [(1.0, 1.0), (1e12, 1e30), (1e-10, 1e-8)])
def test_sorted_forces_at_tile_edges(nb, oracle, masses, scale, mass):
    for n in SIZES:
        x, y, z, vx, vy, vz, m = (v[:n].copy() for v in nb.plummer(max(n, 3), seed=n))
        if n > 64:  # two clusters, so that most tile pairs are far
            x[::2] += 9.0
        if masses == "two_species":  # by place: tiles of one mass, unequal to the next's
            m[::2] *= 3.0
        elif masses == "mixed":
            m[: n // 3] *= np.linspace(0.5, 2.0, n // 3)
        elif masses == "all_different":
            m *= np.linspace(0.5, 2.0, n)
        x, y, z, m = x * scale, y * scale, z * scale, m * mass
        eps = 0.0 if n % 2 else 0.01 * scale
        cfg = nb.Config(method=nb.DIRECT_MIXED, G=1.5, softening=eps, flags=nb.MIXED_SORTED)
        with nb.Sim(cfg, capacity=n) as s:
            s.load(x, y, z, vx, vy, vz, m)
            s.compute_forces()
            a = s.accelerations()
        ref = oracle.forces_naive(x, y, z, m, 1.5, eps)
        sabs = oracle.forces_abs_sum(x, y, z, m, 1.5, eps)
        d = np.sqrt(sum(((u - v) / np.maximum(sabs, 1e-300)) ** 2 for u, v in zip(a, ref)))
        assert (d <= 1e-6).all(), (n, d.max())
