"""The FP64 block-pair kernels at the sizes where they can go wrong: the edges of
the 32-body tiles, odd and even numbers of blocks (an even number's last
diagonal is half filled), the change from one warp per body to block pairs,
and each number of tiles per block.

Tolerance, set before the first run: a term and a sum of n terms carry at most
(8 + log2 n + n / 1024) 2^-53 of sum |term| in any of the kernels' orders; the
oracle's serial sum carries at most n 2^-53.  Both together stay below
(n + 64) 2^-53 of S_i = sum_j |pair term|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 33, 512, 513, 544, 545, 1023, 1056, 2049, 3500, 7001, 13000]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("eps", [0.0, 0.02])
def test_fp64_forces_at_tile_edges(nb, oracle, n, eps):
    x, y, z, vx, vy, vz, m = nb.plummer(n, seed=n) if n > 2 else (
        np.array([0.5, -1.5][:n]), np.zeros(n), np.ones(n), *(np.zeros(n) for _ in range(3)),
        np.array([2.0, 3.0][:n]))
    m = m * np.linspace(0.5, 2.0, n)  # unequal masses: both sides of a pair differ
    with nb.Sim(nb.Config(method=nb.DIRECT_FP64, G=1.5, softening=eps), capacity=n) as s:
        s.load(x, y, z, vx, vy, vz, m)
        s.compute_forces()
        a = s.accelerations()
    ref = oracle.forces_naive(x, y, z, m, 1.5, eps)
    scale = oracle.forces_abs_sum(x, y, z, m, 1.5, eps)
    d = np.sqrt(sum((u - v) ** 2 for u, v in zip(a, ref)))
    assert (d <= (n + 64) * 2.0 ** -53 * scale).all(), (d / np.maximum(scale, 1e-300)).max()


def test_fp64_forces_of_extreme_scales(nb, oracle):
    """Separations far outside FP32's range: the seed works on exponents, and
    beyond its own range the library rsqrt is taken."""
    x, y, z, vx, vy, vz, m = nb.plummer(600, seed=1)
    for scale in (1e-60, 1e-30, 1e25, 1e60):
        p = [c * scale for c in (x, y, z)]
        with nb.Sim(nb.Config(method=nb.DIRECT_FP64), capacity=600) as s:
            s.load(*p, vx, vy, vz, m)
            s.compute_forces()
            a = s.accelerations()
        ref = oracle.forces_naive(*p, m, 1.0, 0.0)
        sabs = oracle.forces_abs_sum(*p, m, 1.0, 0.0)
        d = np.sqrt(sum(((u - v) / sabs) ** 2 for u, v in zip(a, ref)))
        assert (d <= 664 * 2.0 ** -53).all(), (scale, d.max())


@pytest.mark.parametrize("n", [1, 2, 33, 64, 65, 1000, 3500, 7001])
@pytest.mark.parametrize("eps", [0.0, 0.02])
def test_potential_at_tile_edges(nb, oracle, n, eps):
    """Every unordered pair once: against a sum over ordered pairs in NumPy."""
    x, y, z, vx, vy, vz, m = nb.plummer(max(n, 3), seed=n)
    st = [c[:n].copy() for c in (x, y, z, vx, vy, vz, m * np.linspace(0.5, 2.0, len(m)))]
    with nb.Sim(nb.Config(method=nb.DIRECT_FP64, G=1.5, softening=eps), capacity=n) as s:
        s.load(*st)
        d = s.diagnostics()
    p, mm = np.stack(st[:3]), st[6]
    want = [0.0, 0.0]
    for i in range(n - 1):
        r2 = ((p[:, i + 1:] - p[:, i:i + 1]) ** 2).sum(0)
        for k, e2 in enumerate((0.0, eps * eps)):
            want[k] -= 1.5 * mm[i] * (mm[i + 1:] / np.sqrt(r2 + e2)).sum()
    for got, w in zip((d["potential"], d["potential_softened"]), want):
        assert abs(got - w) <= (n + 64) * 2.0 ** -53 * abs(w)
