"""The batched block-pair kernel at the sizes where it can go wrong: the change
from row sums to block pairs, the edges of the 64-body tiles and 256-body blocks,
odd and even numbers of blocks (an even number's last diagonal is half filled).

Tolerance, that of the mixed path: |a - a_ref| <= 1e-6 sum_j |pair term| for every
body, and <= 1e-6 |a_ref| where that sum is at most ten times the force.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 33, 1025, 1311, 2047, 2048, 2049, 2112, 2304, 2305, 2335, 2560, 2817, 3841]
TOL = 1e-6


@pytest.mark.parametrize("eps", [0.0, 0.01])
@pytest.mark.parametrize("flags", [0, 8], ids=["sorted", "unsorted"])
def test_batch_forces_at_tile_edges(nb, oracle, flags, eps):
    st = nb.plummer_ensemble(np.maximum(SIZES, 3), seed=21)
    keep = np.concatenate([np.arange(n) + o for n, o in zip(
        SIZES, np.concatenate([[0], np.cumsum(np.maximum(SIZES, 3))]))])
    st = [v[keep].copy() for v in st]
    st[6] *= np.linspace(0.5, 2.0, len(keep))  # unequal masses: both sides differ
    cfg = nb.Config(method=nb.DIRECT_MIXED, G=1.5, softening=eps, flags=flags)
    with nb.Ensemble(cfg, SIZES) as e:
        e.load(*st)
        e.compute_forces()
        got = e.read_state()
        systems = [e.system(got, s) for s in range(len(SIZES))]
    for n, g in zip(SIZES, systems):
        args = (g["x"], g["y"], g["z"], g["m"], 1.5, eps)
        ref, sabs = oracle.forces_naive(*args), oracle.forces_abs_sum(*args)
        d = np.sqrt(sum((g[k] - r) ** 2 for k, r in zip(("ax", "ay", "az"), ref)))
        r = np.sqrt(sum(v * v for v in ref))
        assert (d <= TOL * sabs).all(), (n, (d / np.maximum(sabs, 1e-300)).max())
        well = sabs <= 10.0 * r
        assert (d[well] <= TOL * r[well]).all(), n
    for s in (3, 7, 12):  # alone, a system gives the bits it gave in the mix
        a = sum(SIZES[:s])
        with nb.Ensemble(cfg, [SIZES[s]]) as e:
            e.load(*[v[a:a + SIZES[s]] for v in st])
            e.compute_forces()
            one = e.read_state()
        for k in ("ax", "ay", "az"):
            assert np.array_equal(one[k], systems[s][k]), (SIZES[s], k)
