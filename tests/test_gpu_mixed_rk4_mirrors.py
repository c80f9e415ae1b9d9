"""RK4 steps of the mixed path below 4096 bodies, where a stage's launch reads every
body's split position and writes the next stage's: the bits of a step put together
from force evaluations and the updates in NumPy, also beside other work on the GPU
(which delays some of a launch's clusters) and when the step is replayed as a graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

DT = 1e-3


def _by_hand(nb, cfg, state, steps):
    x, v, m = np.stack(state[:3]), np.stack(state[3:6]), state[6]
    with nb.Sim(cfg, capacity=len(m)) as s:
        def force(p):
            s.load(*p, *v, m)
            s.compute_forces()
            return np.stack(s.accelerations())

        for _ in range(steps):
            h = DT / 2.0
            a1 = force(x)
            v2 = v + a1 * h
            a2 = force(x + v * h)
            v3 = v + a2 * h
            a3 = force(x + v2 * h)
            v4 = v + a3 * DT
            a4 = force(x + v3 * DT)
            x = x + (((v + v2 * 2.0) + v3 * 2.0) + v4) * (DT / 6.0)
            v = v + (((a1 + a2 * 2.0) + a3 * 2.0) + a4) * (DT / 6.0)
    return np.concatenate([x, v])


@pytest.mark.parametrize("n", [33, 1000, 1025, 2049, 3000, 4095, 4097])
def test_rk4_stages_do_not_mix(nb, n):
    state = nb.plummer(n, seed=n)
    cfg = nb.Config(method=nb.DIRECT_MIXED, G=1.0, softening=0.01)
    want = _by_hand(nb, cfg, state, 4)
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    a = torch.rand(2048, 2048, device="cuda")
    for stream in [None, side.cuda_stream] + [side.cuda_stream] * 10:
        with torch.cuda.stream(other):
            for _ in range(8):
                a = torch.tanh(a @ a)
        with nb.Sim(cfg, capacity=n, stream=stream) as s:
            s.load(*state)
            s.step(nb.RK4, DT, 4)
            got = s.read_state()
        assert np.array_equal(np.stack([got[k] for k in ("x", "y", "z", "vx", "vy", "vz")]), want)
    torch.cuda.synchronize()
