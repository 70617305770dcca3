"""Several handles at once, each on a host thread of its own, whose launches of one kernel take different amounts of shared
memory: the most a kernel may take belongs to the function, so no call may leave it at what its own launch takes."""
import threading
import time

import numpy as np
import pytest

from nntc_b200 import abi, check, lib, materials
from nntc_b200.session import Session

pytestmark = pytest.mark.gpu

SECONDS = 5.0


def session(planes, channels, shaped):
    w, h = planes[0][:2]
    mat = materials.Material("two", [np.zeros((h, w, 3), np.uint8)], channels, channels)
    rng = np.random.default_rng(w)
    mat.planes, mat.per_site = planes, [1.0 / len(planes)] * len(planes)
    mat.chain = [rng.random((p[1], p[0], 3)).astype(np.float32) for p in planes]
    s = Session(mat)
    check(lib().nntc_b200_set_option(s.d, abi.OPT_REFERENCE_SHAPED_ASSEMBLY, shaped), "option")
    for i, p in enumerate(planes):
        s.set_planes(i, rng.random(p[0] * p[1] * channels) * 2 - 1, rng.random(p[2] * p[3] * channels) * 2 - 1)
    s.set_decoder(rng.standard_normal((3, s.m.nin)) * 0.3, rng.random(3))
    s.set_grids(np.full(channels, -1.0), np.full(channels, 1.0), np.full(channels, -1.0), np.full(channels, 1.0))
    return s


def percentiles(s, k):
    check(lib().nntc_b200_quantise_level1(s.d, abi.C.byref(s.m), 1, abi.u8_ptrs(s.u8_planes(1))), "quantise")


# one handle's launch takes more than 48 KB, the other's less: (call, planes, channels and K of each, option)
@pytest.mark.parametrize("call,large,small,shaped", [
    (lambda s, k: s.solve_decoder(k), ([(16, 16, 4, 4)] * 13, 2, 4), ([(16, 16, 4, 4)], 2, 4), 0),
    (lambda s, k: s.block(False, 1, k), ([(61, 45, 15, 11)], 2, 4), ([(13, 9, 3, 2)], 2, 4), 0),
    (lambda s, k: s.block(False, 1, k), ([(32, 16, 8, 4)], 2, 4), ([(32, 16, 8, 4)], 2, 1), 0),
    (lambda s, k: s.block(False, 1, k), ([(16, 16, 4, 4)], 4, 4), ([(16, 16, 4, 4)], 1, 4), 1),
    (percentiles, ([(16, 16, 4, 4)], 4, 4), ([(16, 16, 4, 4)], 1, 4), 0),
], ids=["decoder", "ragged tiles", "tabled tiles", "reference shape", "percentiles"])
def test_two_threads(call, large, small, shaped):
    failures = []

    def work(planes, channels, k, seconds):
        try:
            with session(planes, channels, shaped) as s:
                ready.wait(60)
                end = time.monotonic() + seconds
                while time.monotonic() < end and not failures:
                    call(s, k)
        except Exception as e:   # noqa: BLE001 (handed to the test's thread)
            failures.append(e)

    # the window between a limit and its launch is a microsecond of each call: six threads lower what one needs
    ready = threading.Barrier(7)
    threads = [threading.Thread(target=work, args=(large if i == 0 else small) + (SECONDS,)) for i in range(7)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[0]
