"""Two tiles, s apart, that share an origin in the Hilbert-sorted direct sum, and a third
0.13 s to 0.24 s from the second.  Relative to the middle of the first two, coordinates
of about s / 2 and 0.7 s round to FP32 by up to 2^-25 s each, 2^-24 s / 0.13 s = 4.6e-7
of the distance and twice that of the force.  A plain displacement without the Newton
step is for boxes at least a quarter of the origin's box away, so the third tile has to
be met otherwise: relative to a tile of its own size, the displacement rounds by 2^-24 of
itself (2^-23 of the force) and the term by 4 roundings and the Newton step's rest,
below 4e-7 in all.
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


def _worst_places(gap, rng):
    """Places of the second and third tile whose coordinates, relative to the middle of the
    first two, round apart the most."""
    x2 = 1.0 + rng.uniform(0.0, 1e-3, 4000)
    x3 = x2 + gap + rng.uniform(0.0, 1e-3, 4000)
    root = (0.0 + x3) / 2.0
    h1, h2 = np.float32(0.0 - root), np.float32(x2 - root)
    c = (np.float32(0.5) * (h1 + h2)).astype(float)
    off = [np.float32(v - root - c).astype(float) - (v - root - c) for v in (x2, x3)]
    k = np.abs(off[1] - off[0]).argmax()
    return x2[k], x3[k]


@pytest.mark.parametrize("gap", [0.13, 0.15, 0.2, 0.24])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_far_displacements_of_tiles_that_share_an_origin(nb, gap, axis, sign):
    rng = np.random.default_rng(int(100 * gap))
    x2, x3 = _worst_places(gap, rng)
    p = np.zeros((3, 192))
    p[axis] = sign * np.repeat([0.0, x2, x3], 64)
    m = np.repeat([1e-6, 1e-6, 1.0], 64)
    m *= np.linspace(0.9, 1.1, 192)
    a = np.stack(_forces(nb, *p, m))
    at = np.array([0.0, x2, x3])
    for t in range(2):  # bodies of a tile share a place and have no force on each other
        d = np.delete(at - at[t], t)
        ref = sign * (np.delete(m.reshape(3, 64).sum(1), t) * d / np.abs(d) ** 3).sum()
        err = np.abs(a[axis, 64 * t:64 * t + 64] - ref) / abs(ref)
        assert err.max() <= 4e-7, (t, err.max())
