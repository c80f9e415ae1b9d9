"""A server whose trees go from few to many and back, so that their walks change between
the ordered and the serial one while they run: every job gives the bits it gives alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_walks_change_with_the_load(nb):
    states = [nb.disk_bulge(90_000 + k, seed=k) if k % 2 else nb.plummer(90_000 + k, seed=k)
              for k in range(8)]
    steps = [14, 4, 5, 6, 4, 5, 6, 4]

    def alone(k):
        with nb.Server() as s:
            job = s.submit(states[k], steps[k])
            s.run_until_idle()
            return s.result(job)

    with nb.Server() as s:
        jobs = [s.submit(states[0], steps[0])]  # few
        for _ in range(4):
            s.tick()
        jobs += [s.submit(states[k], steps[k]) for k in range(1, 8)]  # 720,000 bodies
        s.run_until_idle()  # the first is the last to end, alone again
        got = [s.result(j) for j in jobs]
    for k in range(8):
        want = alone(k)
        assert all(np.array_equal(got[k][c], want[c]) for c in want), k
