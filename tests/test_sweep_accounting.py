"""What a timed launch of the quantised sweeps stands for: a colour, also where a whole sweep is one launch."""
import ctypes as C
import importlib.util
import os

import numpy as np
import pytest

from nntc_b200 import KERNELS, check, lib, materials
from nntc_b200.session import Session

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,sweeps", [(64, 48, 3), (400, 600, 2)])   # a launch a sweep; a launch a colour at level 0
def test_launches_are_colours(w, h, sweeps):
    mat = materials.small(w + h, w, h, textures=1, c0=2, c1=1)
    rng = np.random.default_rng(w)
    with Session(mat) as s:
        for i, p in enumerate(mat.planes):
            s.set_planes(i, rng.random(p[0] * p[1] * 2) * 2 - 1, rng.random(p[2] * p[3]) * 2 - 1)
        s.set_decoder(rng.standard_normal((3, s.m.nin)) * 0.3, rng.random(3))
        s.set_grids(np.full(2, -1.0), np.full(2, 1.0), np.full(1, -1.0), np.full(1, 1.0))
        check(lib().nntc_b200_kernel_timing(s.d, 1), "timing")
        for level0 in (False, True):
            check(lib().nntc_b200_kernel_stats(s.d, 0, None, None, 1), "reset")
            s.block(level0, sweeps=sweeps)
            n, ms = C.c_longlong(), C.c_double()
            check(lib().nntc_b200_kernel_stats(s.d, KERNELS.index("quant_sweep"), C.byref(n), C.byref(ms), 0), "stats")
            assert n.value == 4 * sweeps and ms.value > 0, level0


def test_bench_traffic_is_of_a_colour_launch():
    spec = importlib.util.spec_from_file_location("bench_module", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    for w, h, swept in ((64, 48, True), (416, 168, True), (512, 512, False)):
        mat = materials.small(1, w, h, textures=1, c0=4, c1=4)
        for form in ("plain", "adjoint"):
            roof = bench.roofline("quant_sweep", (8, 1.0), mat, 6000.0, 1500.0, "fallback", form)
            # the recorded DRAM bytes are of a launch of one colour
            assert (roof["traffic"] is None) == swept, (w, h, form)
            assert roof["bytes_per_launch"] == bench.algorithmic_bytes("quant_sweep", mat, form)
