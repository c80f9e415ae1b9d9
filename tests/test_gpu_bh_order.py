"""The Barnes-Hut walk's terms are added in one order, whatever computes it: the ordered
walk, also where a walk visits more groups than its log holds at a time (small theta,
small leaves, large trees under the reference's rule) or than the pool has room for,
and the serial walk.  All give the same bits, each time and beside other work."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _flags(nb, rule):
    return (nb.BH_QUADRUPOLE if "quad" in rule else 0) | (
        nb.BH_REFERENCE_OPENING if "ref" in rule else 0)


def _bodies(nb, model, n):
    if model == "cube":  # more groups a walk than the models the pool is sized by
        rng = np.random.default_rng(n)
        return (*rng.uniform(-1, 1, (3, n)), *np.zeros((3, n)), np.full(n, 1.0 / n))
    return nb.plummer(n, seed=n) if model == "plummer" else nb.disk_bulge(n, seed=n)


def _step(nb, state, rule, theta, leaf, eps=1e-3, stream=None):
    n = len(state[0])
    cfg = nb.Config(method=nb.BARNES_HUT, G=1.0, softening=eps, theta=theta,
                    leaf_capacity=leaf, flags=_flags(nb, rule))
    with nb.Sim(cfg, capacity=n, stream=stream) as s:
        s.load(*state)
        s.step(nb.LEAPFROG, 1e-3, 1)
        st, info = s.read_state(), s.bh_info()
    return (np.stack([st[k] for k in ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az")]),
            info["interactions_m2p"], info["interactions_p2p"])


CASES = [("disk", n, rule, theta, 8)
         for n in (16_500, 100_003) for rule in ("", "ref", "quad", "quad+ref")
         for theta in (0.2, 0.3, 0.4)]
CASES += [("plummer", 100_003, "", 0.3, 8), ("plummer", 400_003, "ref", 0.35, 8),
          ("disk", 400_003, "ref", 0.5, 8), ("disk", 100_003, "ref", 0.5, 1),
          ("disk", 100_003, "", 0.5, 1), ("cube", 200_001, "", 0.3, 8),
          ("cube", 100_003, "ref", 0.4, 2), ("plummer", 20_000, "", 0.0, 8)]


@pytest.mark.parametrize("model,n,rule,theta,leaf", CASES)
def test_one_order_of_summation(nb, monkeypatch, model, n, rule, theta, leaf):
    state = _bodies(nb, model, n)
    monkeypatch.setenv("NB_BH_WALK", "serial")
    want = _step(nb, state, rule, theta, leaf)
    monkeypatch.delenv("NB_BH_WALK")
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    a = torch.rand(2048, 2048, device="cuda")
    for k in range(3):
        if k:  # CTAs start in another order
            with torch.cuda.stream(other):
                for _ in range(10):
                    a = torch.tanh(a @ a)
        got = _step(nb, state, rule, theta, leaf, stream=side.cuda_stream if k else None)
        assert got[1:] == want[1:]
        assert np.array_equal(got[0], want[0])
    torch.cuda.synchronize()


def test_jobs_at_small_theta_alone_and_in_the_mix(nb):
    """A server's job gives the same bits beside others, at a theta whose walks are long."""
    jobs = [nb.plummer(60_000, seed=1), nb.disk_bulge(30_000, seed=2),
            nb.disk_bulge(70_000, seed=3), nb.plummer(5_000, seed=4)]

    def run(states):
        with nb.Server(theta=0.25) as s:
            ids = [s.submit(j, 2) for j in states]
            s.run_until_idle()
            return [s.result(i) for i in ids]

    for state, mixed in zip(jobs, run(jobs)):
        alone = run([state])[0]
        assert all(np.array_equal(alone[k], mixed[k]) for k in alone)
