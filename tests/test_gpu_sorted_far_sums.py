"""What the Hilbert-sorted direct sum keeps of a far sum: two clusters, each at one point,
a power of two apart, so that every term is m / R^2 without rounding; the masses are
integers whose runs of 32 fit FP32 and whose sums of 256 do not.  A partial sum of a
block pair is a Kahan pair, which holds such a sum exactly: 2^-40 leaves room for the
final additions in FP64 alone, and is far below the 2^-25 of one FP32 number.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _forces(nb, x, y, z, m):
    zero = np.zeros(len(m))
    cfg = nb.Config(method=nb.DIRECT_MIXED, G=1.0, softening=0.0, flags=nb.MIXED_SORTED)
    with nb.Sim(cfg, capacity=len(m)) as s:
        s.load(x, y, z, zero, zero, zero, m)
        s.compute_forces()
        return s.accelerations()


def test_far_sums_keep_their_compensation(nb):
    rng = np.random.default_rng(5)
    m = rng.integers(1 << 17, 1 << 18, 512).astype(float)
    for half in (m[:256], m[256:]):  # the last two of 26 bits: not in FP32
        half[0] += (1 - half.sum()) % 4
    x = np.repeat([0.0, 8.0], 256)
    ax, ay, az = _forces(nb, x, np.zeros(512), np.zeros(512), m)
    want = np.repeat([m[256:].sum() / 64.0, -m[:256].sum() / 64.0], 256)
    assert (np.abs(ax - want) <= 2.0 ** -40 * np.abs(want)).all(), (ax / want - 1.0)[[0, 511]]
    assert not ay.any() and not az.any()
