"""The shared Barnes-Hut walk (2^k warps per 64 bodies) against the preorder walk.

Sizes around one CTA's 64 bodies, and one for each number of warps the launch
rule takes (16 under the reference's opening rule, 8, 4, 2, 1), with bodies that
share a position (leaves of more than 32 bodies) and without."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compare(nb, monkeypatch, n, flags, eps, theta):
    bits = (nb.BH_QUADRUPOLE if "quad" in flags else 0) | (
        nb.BH_REFERENCE_OPENING if "ref" in flags else 0)
    state = [np.array(v, copy=True) for v in nb.disk_bulge(n, seed=n)]
    if n > 1000:
        for v in state[:3]:
            v[100:300] = v[100]
    out = {}
    for walk in ("group", "preorder"):
        monkeypatch.setenv("NB_BH_WALK", walk)
        config = nb.Config(method=nb.BARNES_HUT, G=1.0, softening=eps, theta=theta, flags=bits)
        with nb.Sim(config, capacity=n) as s:
            s.load(*state)
            s.compute_forces()
            info = s.bh_info()
            out[walk] = (s.accelerations(), info["interactions_m2p"], info["interactions_p2p"])
    assert out["group"][1:] == out["preorder"][1:]
    a, b = out["group"][0], out["preorder"][0]
    mag = np.sqrt(sum(v * v for v in b))
    diff = np.sqrt(sum((u - v) ** 2 for u, v in zip(a, b)))
    assert all(np.isfinite(v).all() for v in a) and (mag > 0).all()
    assert diff.max() < 1e-4 * mag.max() and np.median(diff / mag) < 4e-6


@pytest.mark.parametrize("n", [2, 63, 64, 65, 4099, 200_001, 400_003, 700_001])
@pytest.mark.parametrize("flags", ["", "quad", "ref", "quad+ref"])
@pytest.mark.parametrize("eps", [1e-3, 0.0])
def test_shared_walk_equals_preorder_walk(nb, monkeypatch, n, flags, eps):
    """Equal monopole and body counts; forces equal up to the FP32 rounding of two
    orders of summation.  Each of two sums of T terms deviates by about 2^-24
    sqrt(T) of the sum of the terms' magnitudes; T is below 30,000 here, so 1e-5 of
    that sum each, and the magnitudes sum to at most the largest force but for
    cancellation, for which a factor of 10 is left: 1e-4 of the largest force, the
    bound of the walks' other comparison, as is the median's."""
    _compare(nb, monkeypatch, n, flags, eps, 0.5)


@pytest.mark.parametrize("theta", [0.1, 0.3])
def test_ordered_walk_without_room(nb, monkeypatch, theta):
    """The reference's rule at small theta: walks that visit more groups than a log
    holds (0.1), or than the pool has room for (0.3), go by the other walk."""
    _compare(nb, monkeypatch, 100_003, "ref", 1e-3, theta)
