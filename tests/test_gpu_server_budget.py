"""A server's device memory against its budget: what the device lost while jobs of both
kinds ran stays within the budget and within what the server reports, with small slack for
streams, graphs and the allocator's 2 MiB pages."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

MIB = 1 << 20


def _run(nb, jobs, steps, **config):
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    most = 0
    with nb.Server(**config) as s:
        ids = [s.submit(j, steps) for j in jobs]
        while True:
            running, queued = s.tick()
            most = max(most, free - torch.cuda.mem_get_info()[0])
            if running == 0 and queued == 0:
                break
        results = [s.result(i) for i in ids]
        return results, most, s.stats()


def _bodies(nb, n, seed):
    return nb.disk_bulge(n, seed=seed) if seed % 2 else nb.plummer(n, seed=seed)


def test_a_small_budget_is_kept(nb):
    """8 trees of 200,000 bodies (470 bytes a body) and direct jobs that fill the pool: at
    320 bytes a body and with planes beside the budget they would take 1.1 GiB."""
    budget = 640 * MIB
    jobs = [_bodies(nb, 200_000, k) for k in range(8)] + [_bodies(nb, 16_000, k) for k in range(60)]
    _, most, st = _run(nb, jobs, 3, hbm_budget_bytes=budget, pool_bodies=1 << 20)
    assert st["jobs_finished"] == len(jobs) and st["jobs_failed"] == 0
    assert st["peak_device_bytes"] <= budget
    assert most <= st["peak_device_bytes"] + 128 * MIB, (most / MIB, st["peak_device_bytes"] / MIB)


def test_the_pool_may_take_the_whole_budget(nb):
    """No room for partial planes: direct jobs go by rows, and no tree is accepted."""
    pool = 1 << 17
    jobs = [_bodies(nb, 9_000, k) for k in range(10)]
    got, most, st = _run(nb, jobs, 2, hbm_budget_bytes=112 * pool, pool_bodies=pool)
    assert st["jobs_failed"] == 0 and most <= 112 * pool + 128 * MIB
    alone, _, _ = _run(nb, jobs[:1], 2, hbm_budget_bytes=112 * pool, pool_bodies=pool)
    assert all(np.array_equal(alone[0][k], got[0][k]) for k in alone[0])
    with nb.Server(hbm_budget_bytes=112 * pool, pool_bodies=pool) as s:
        with pytest.raises(nb.NBodyError) as e:
            s.submit(_bodies(nb, 20_000, 1), 1)
        assert e.value.status == 4


def test_an_accepted_job_runs(nb):
    """A tree that fits at 320 bytes a body, the condition of submission, and not at what it
    takes: it runs, alone among the trees."""
    pool, n = 1 << 14, 100_000
    jobs = [_bodies(nb, n, 1), _bodies(nb, 5_000, 2), _bodies(nb, n, 3)]
    got, _, st = _run(nb, jobs, 2, hbm_budget_bytes=112 * pool + 320 * n, pool_bodies=pool)
    assert st["jobs_failed"] == 0 and st["max_running"] <= 2
    alone, _, _ = _run(nb, jobs[2:], 2)
    assert all(np.array_equal(alone[0][k], got[2][k]) for k in alone[0])
