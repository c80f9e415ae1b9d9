"""The i-bodies per lane that an ensemble reports are those of the kernels it launches: one
in the row sums of systems below 2048 bodies, four in the block pairs of larger ones."""
import pytest

pytestmark = pytest.mark.gpu


def test_reported_bodies_per_lane(nb):
    sizes = [40, 1500, 2048, 3000]
    with nb.Ensemble(nb.Config(method=nb.DIRECT_MIXED, softening=0.01), sizes) as e:
        e.load(*nb.plummer_ensemble(sizes, seed=1))
        tuned, info = e.tune(), e.info()["ipt_by_bucket"]
    assert list(tuned) == list(info)
    assert all(info[b] == 1 for b in range(11)) and all(info[b] == 4 for b in range(11, 20))
