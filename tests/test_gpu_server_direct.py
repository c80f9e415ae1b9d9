"""A server's direct jobs on both sides of the size from which their pairs are summed
once: the accelerations after a step against the FP64 sum at the job's positions.

Tolerance, that of the mixed path: |a - a_ref| <= 1e-6 sum_j |pair term|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1024, 4095, 4096, 4161])
def test_direct_jobs_at_the_change_of_sums(nb, oracle, n):
    with nb.Server() as s:
        jobs = [s.submit(nb.disk_bulge(n, seed=n), 1), s.submit(nb.plummer(n, seed=n), 1)]
        s.run_until_idle()
        results = [s.result(j) for j in jobs]
    for r in results:
        args = (r["x"], r["y"], r["z"], r["m"], 1.0, 1e-3)
        ref, sabs = oracle.forces_naive(*args), oracle.forces_abs_sum(*args)
        d = np.sqrt(sum((r[k] - v) ** 2 for k, v in zip(("ax", "ay", "az"), ref)))
        assert (d <= 1e-6 * sabs).all(), (d / sabs).max()
