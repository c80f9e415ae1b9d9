"""A server's Barnes-Hut jobs on simulation objects that earlier jobs left: the
results and the interaction counts are those of a new server, for jobs of the same
size, a little smaller (an object with room to spare) and after a cancelled job."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(server, state, steps):
    job = server.submit(state, steps)
    before = server.stats()["interactions"]
    server.run_until_idle()
    result = server.result(job)
    server.release(job)
    return result, server.stats()["interactions"] - before


@pytest.mark.parametrize("n", [20_000, 17_000])
def test_reused_simulations_change_nothing(nb, n):
    state = nb.plummer(n, seed=n)
    with nb.Server() as fresh:
        want, count = _run(fresh, state, 3)
    with nb.Server() as s:
        _run(s, nb.disk_bulge(20_000, seed=1), 4)
        cancelled = s.submit(nb.disk_bulge(20_500, seed=2), 50)
        s.tick()
        s.cancel(cancelled)
        for _ in range(3):
            got, again = _run(s, state, 3)
            assert again == count
            assert all(np.array_equal(got[k], want[k]) for k in want)
