"""A simulation that is taken off the caller's arrays (nb_bind_device with NULL) steps its
own: neither a captured step nor a kept tree of the caller's bodies is used again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

KEYS = ("x", "y", "z", "vx", "vy", "vz")


@pytest.mark.parametrize("method,flags", [("fp64", 0), ("mixed", 0), ("bh", 0), ("bh", 8 << 8)])
def test_steps_after_unbinding(nb, method, flags):
    n = 900
    cfg = nb.Config(method={"fp64": nb.DIRECT_FP64, "mixed": nb.DIRECT_MIXED,
                            "bh": nb.BARNES_HUT}[method], G=1.0, softening=0.01, flags=flags)
    own, other = nb.plummer(n, seed=1), nb.plummer(n, seed=2)
    side = torch.cuda.Stream()
    with nb.Sim(cfg, capacity=n, stream=side.cuda_stream) as s:
        s.load(*own)
        s.step(nb.RK4, 1e-3, 1)
        want = s.read_state()
    bound = torch.zeros(10, n, dtype=torch.float64, device="cuda")
    for row, v in zip((0, 1, 2, 3, 4, 5, 9), other):
        bound[row] = torch.from_numpy(v)
    torch.cuda.synchronize()
    with nb.Sim(cfg, capacity=n, stream=side.cuda_stream) as s:
        s.load(*own)
        rows = (nb.C.c_void_p * 10)(*[bound[k].data_ptr() for k in range(10)])
        assert nb.lib().nb_bind_device(s.handle, n, rows) == 0
        s.step(nb.RK4, 1e-3, 4)  # captured, and replayed
        s.synchronize()
        after = bound.clone()
        assert nb.lib().nb_bind_device(s.handle, 0, None) == 0
        s.step(nb.RK4, 1e-3, 1)
        got = s.read_state()
        assert torch.equal(bound, after)
    assert all(np.array_equal(got[k], want[k]) for k in KEYS)
