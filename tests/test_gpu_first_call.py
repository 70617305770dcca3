"""A process's first calls load the kernels they launch and not every other material's: a module is loaded whole, so how the
kernels lie in modules decides how long a first call waits."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CALLS = """
import json, time
import numpy as np
from nntc_b200 import materials
from nntc_b200.session import Session
mat = materials.small(1, 96, 64, textures=2, c0=2, c1=4)
rng = np.random.default_rng(0)
with Session(mat) as s:
    for i, p in enumerate(mat.planes):
        s.set_planes(i, rng.random(p[0] * p[1] * 2) * 2 - 1, rng.random(p[2] * p[3] * 4) * 2 - 1)
    s.set_decoder(rng.standard_normal((6, s.m.nin)) * 0.3, rng.random(6))
    s.set_grids(np.full(2, -1.0), np.full(2, 1.0), np.full(4, -1.0), np.full(4, 1.0))
    out = []
    for call in (s.objective, s.solve_decoder, lambda: s.block(False)):
        took = []
        for _ in range(3):
            t = time.perf_counter()
            call()
            took.append(time.perf_counter() - t)
        out.append(took[0] - min(took))
print(json.dumps(out))
"""


def test_first_calls_do_not_load_every_kernel():
    # with all of the assembly's kernels in two modules the decoder solve's first call took 20 ms more than its next, the
    # block's 18; the kernels they launch load in a few
    best = [1.0, 1.0, 1.0]
    for _ in range(3):
        run = subprocess.run([sys.executable, "-c", CALLS], cwd=ROOT, capture_output=True, text=True, check=True, timeout=120)
        best = [min(a, b) for a, b in zip(best, json.loads(run.stdout.splitlines()[-1]))]
    assert max(best) < 0.012, best
