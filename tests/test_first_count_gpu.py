"""The first pair count of a process loads the kernels it needs and not all there are:
it takes no longer than the first triplet count (of one module as well)."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = """
import time
from desi_b200 import api, catalog
c = api.Context(0)
a, b = (c.grid(catalog.uniform(3000, 250.0, seed=s, weights=%r), 250.0) for s in (1, 2))
a.info(), b.info()
def ms(f):
    t = time.perf_counter()
    f()
    return (time.perf_counter() - t) * 1e3
print(ms(lambda: c.count_triplets(a, bins=10, dmax=20.0)), ms(lambda: c.count_pairs(a, b, bins=30, dmax=80.0)))
"""


@pytest.mark.parametrize("weights", ["unit", "uniform"])
def test_pairs_after_triplets(weights):
    """(with all pair kernels in one module: 4 and 15 ms)"""
    best = None
    for _ in range(3):
        p = subprocess.run([sys.executable, "-c", CODE % weights], capture_output=True, text=True, cwd=ROOT,
                           timeout=300, env=dict(os.environ, CUDA_MODULE_LOADING="LAZY"))
        assert p.returncode == 0, p.stderr
        trip, pairs = (float(x) for x in p.stdout.split())
        best = min(best or 1e9, pairs / trip)
    assert best <= 2.0
