"""Below 4096 bodies the entry point that allocates nothing gives the bits of the
NB_DIRECT_MIXED method, as the header says."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 100, 1000, 1025, 2049, 4095])
@pytest.mark.parametrize("eps", [0.0, 1e-3])
def test_same_bits_as_the_allocating_path(nb, n, eps):
    state = nb.plummer(n, seed=n)
    cfg = nb.Config(method=nb.DIRECT_MIXED, G=1.5, softening=eps)
    with nb.Sim(cfg, capacity=n) as src, nb.Sim(cfg, capacity=n) as dst:
        src.load(*state)
        src.compute_forces()
        dst.load(*state)
        p, q = src.device_arrays(), dst.device_arrays()  # x y z vx vy vz ax ay az m
        rc = nb.lib().nb_direct_mixed_forces_noalloc(n, p[0], p[1], p[2], p[9], 1.5, eps, q[6],
                                                     q[7], q[8], None)
        assert rc == 0, nb.lib().nb_last_error()
        for a, b in zip(src.accelerations(), dst.accelerations()):
            assert np.array_equal(a, b)
