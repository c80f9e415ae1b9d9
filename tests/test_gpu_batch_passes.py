"""Ensembles whose partial planes exceed one pass's buffer (1 GiB): a system that alone
does (its diagonals in passes), and many that do together.  The device memory stays
bounded, every system gives the bits it gives alone, and the large one is right.

Tolerance, that of the mixed path: |a - a_ref| <= 1e-6 sum_j |pair term|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

GIB = 1 << 30


def _forces(nb, cfg, sizes, state):
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with nb.Ensemble(cfg, sizes) as e:
        e.load(*state)
        e.compute_forces()
        e.synchronize()
        used = free - torch.cuda.mem_get_info()[0]
        st = e.read_state()
    return np.stack([st[k] for k in ("ax", "ay", "az")]), used


def _check(a, state, stride):
    p = torch.from_numpy(np.stack(state[:3])).cuda()
    m = torch.from_numpy(state[6].copy()).cuda()
    for i in range(0, len(m), stride):
        d = p - p[:, i:i + 1]
        t = 1.5 * m * d / ((d * d).sum(0) + 1e-6) ** 1.5
        ref, sabs = t.sum(1).cpu().numpy(), float((t * t).sum(0).sqrt().sum())
        assert np.sqrt(((a[:, i] - ref) ** 2).sum()) <= 1e-6 * sabs


@pytest.mark.parametrize("flags", [0, 8], ids=["sorted", "unsorted"])
def test_one_large_system(nb, flags):
    sizes = [3000, 150_000, 40]  # planes of 2.1 GB
    state = [np.concatenate(v) for v in zip(*(nb.plummer(n, seed=n) for n in sizes))]
    state[6] = state[6] * np.linspace(0.5, 2.0, sum(sizes))
    cfg = nb.Config(method=nb.DIRECT_MIXED, G=1.5, softening=1e-3, flags=flags)
    a, used = _forces(nb, cfg, sizes, state)
    assert used < 1.25 * GIB, used / GIB
    lo = 0
    for n in sizes:
        part = slice(lo, lo + n)
        alone, _ = _forces(nb, cfg, [n], [v[part] for v in state])
        assert np.array_equal(alone, a[:, part])
        lo += n
    _check(a[:, 3000:153_000], [v[3000:153_000] for v in state], 1171)


def test_many_systems(nb):
    n, count = 4096, 900  # planes of 1.5 GB together, two passes
    one = nb.plummer(n, seed=1)
    rng = np.random.default_rng(1)
    scale = rng.uniform(0.5, 2.0, count)
    state = [np.concatenate([v * s if k < 3 else v for s in scale]) for k, v in enumerate(one)]
    cfg = nb.Config(method=nb.DIRECT_MIXED, G=1.0, softening=1e-3)
    a, used = _forces(nb, cfg, [n] * count, state)
    assert used < 1.25 * GIB + 250 * n * count, used / GIB
    for s in (0, 1, 600, 700, count - 1):
        part = slice(s * n, (s + 1) * n)
        alone, _ = _forces(nb, cfg, [n], [v[part] for v in state])
        assert np.array_equal(alone, a[:, part])


def test_beyond_the_table_of_block_pairs(nb):
    n = (1 << 20) + 1  # by rows: no planes, no table of block pairs
    state = nb.plummer(n, seed=2)
    cfg = nb.Config(method=nb.DIRECT_MIXED, G=1.5, softening=1e-3)
    a, used = _forces(nb, cfg, [n], state)
    assert used < 0.5 * GIB, used / GIB
    _check(a, state, 50_021)
