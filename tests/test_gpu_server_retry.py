"""A tick that fails because an allocation of the direct batch does has stepped nothing:
the next one carries on, and every job gives the bits it gives alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fail_at", [0, 1, 2, 3, 4, 5])
def test_a_failed_tick_can_be_repeated(nb, fail_at):
    states = [nb.plummer(5000, seed=1), nb.disk_bulge(1500, seed=2), nb.disk_bulge(20_000, seed=3)]

    def alone(state):
        with nb.Server() as s:
            job = s.submit(state, 3)
            s.run_until_idle()
            return s.result(job)

    with nb.Server() as s:
        tree = s.submit(states[2], 3)
        s.tick()  # its allocations are made
        jobs = [s.submit(states[0], 3), s.submit(states[1], 3)]
        nb.debug_fail_device_allocations(fail_at)
        try:
            s.tick()
        except nb.NBodyError as e:
            assert e.status == 3
        nb.debug_fail_device_allocations(-1)
        s.run_until_idle()
        got = [s.result(j) for j in jobs + [tree]]
        assert s.stats()["steps_done"] == 9
    for state, g in zip(states, got):
        want = alone(state)
        assert all(np.array_equal(g[k], want[k]) for k in want)
