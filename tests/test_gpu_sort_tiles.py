"""The radix sort of the Barnes-Hut codes around the tile counts where a pass changes:
one tile and its edges, the last sizes whose scatter counts the next digit (64 tiles)
and adds up the tiles' counts itself (128), and beyond, where a kernel scans them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2047, 2049, 131_072, 131_073, 262_144, 262_145, 2_100_000])
def test_codes_and_order_at_tile_counts(nb, oracle, n):
    rng = np.random.default_rng(n)
    x, y, z = rng.standard_normal((3, n))
    x[: n // 3] = x[0]  # many equal digits
    zero = np.zeros(n)
    codes, _ = oracle.morton63(x, y, z)
    want, order = oracle.sort_codes(codes)
    with nb.Sim(nb.Config(method=nb.BARNES_HUT), capacity=n) as s:
        s.load(x, y, z, zero, zero, zero, np.ones(n))
        s.bh_build()
        got, got_order = s.bh_order()
    assert np.array_equal(got, want) and np.array_equal(got_order, order)
