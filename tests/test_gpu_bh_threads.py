"""Two host threads, each with a simulation of its own, whose Barnes-Hut walks take
different amounts of shared memory (16 and 8 warps, quadrupoles, the reference's rule):
neither disturbs the other's launches, and each gives the bits it gives alone.

A child process, since the bodies per lane are read once per process."""
import os
import subprocess
import sys

import pytest

from conftest import PKG_DIR, REPO

pytestmark = pytest.mark.gpu

CHILD = r'''
import sys, threading
sys.path.insert(0, sys.argv[1])
import numpy as np
import nbody_gb300 as nb
flags = nb.BH_QUADRUPOLE | nb.BH_REFERENCE_OPENING
cfg = nb.Config(method=nb.BARNES_HUT, G=1.0, softening=1e-3, theta=0.9, flags=flags)
cases = [(20_000, 300), (300_000, 60)]

def run(n, evals, out, k):
    try:
        with nb.Sim(cfg, capacity=n) as s:
            s.load(*nb.plummer(n, seed=n))
            for _ in range(evals):
                s.compute_forces()
            out[k] = np.stack(s.accelerations())
    except Exception as e:
        out[k] = e

alone, both = [None] * 2, [None] * 2
for k, (n, _) in enumerate(cases):
    run(n, 1, alone, k)
threads = [threading.Thread(target=run, args=(n, e, both, k)) for k, (n, e) in enumerate(cases)]
for t in threads: t.start()
for t in threads: t.join()
for a, b in zip(alone, both):
    for v in (a, b):
        if isinstance(v, Exception):
            raise v
    assert np.array_equal(a, b)
print("THREADS_OK")
'''


def test_two_threads_with_different_walks():
    env = dict(os.environ, NB_BH_WALK_PAIRS="2")
    r = subprocess.run([sys.executable, "-c", CHILD, PKG_DIR], env=env, cwd=REPO,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "THREADS_OK" in r.stdout, r.stderr[-3000:]
