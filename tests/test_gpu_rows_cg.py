"""The conjugate gradients and the quantised sweeps of an FP32 stencil, formed a lane per row of a texel's blocks, at every
channel count, with symmetric blocks (weights of one) and blocks that are not, on planes whose last block and warp are
partly filled: one step of each recomputed from the downloaded stencil in FP64."""
import ctypes as C

import numpy as np
import pytest

from nntc_b200 import abi, check, lib, materials
from nntc_b200.session import Session
from test_gpu_adjoint import stencil_product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level0", [False, True])
@pytest.mark.parametrize("c0,c1,w,h,weights", [(4, 4, 68, 36, "one"), (4, 2, 61, 37, "mixed"), (2, 4, 40, 24, "mixed"),
                                               (3, 1, 45, 29, "one"), (2, 3, 64, 64, "one"), (1, 4, 33, 70, "mixed")])
def test_solve_residual_and_sweep(c0, c1, w, h, weights, level0):
    mat = materials.small(w + 9 * h, w, h, textures=2, c0=c0, c1=c1)
    rng = np.random.default_rng(w * h)
    cw = None if weights == "one" else list(0.3 + rng.random(6))
    c, bits = (c0 if level0 else c1), 8
    with Session(mat, model=abi.make_model(mat, cw=cw)) as s:
        check(lib().nntc_b200_set_option(s.d, abi.OPT_FP32_STENCIL, 1), "option")
        v0 = [rng.random(p[0] * p[1] * c0) * 2 - 1 for p in mat.planes]
        v1 = [rng.random(p[2] * p[3] * c1) * 2 - 1 for p in mat.planes]
        for i in range(len(mat.planes)):
            s.set_planes(i, v0[i], v1[i])
        s.set_decoder(rng.standard_normal((6, s.m.nin)) * 0.3, rng.random(6))
        s.set_grids(np.full(c0, -1.0), np.full(c0, 1.0), np.full(c1, -1.0), np.full(c1, 1.0))
        rep, _ = s.block(level0, ridge=1e-3)
        for i, p in enumerate(mat.planes):
            uw, uh = (p[0], p[1]) if level0 else (p[2], p[3])
            ws = s.workspace(i, level0)
            ax = stencil_product(ws["stencil"], ws["x"], uw, uh, c) + rep[i].lambda_ * ws["x"]
            # the recursive residual is below 1e-7 of the right-hand side when the iterations stop; FP64 recurrences over
            # at most 200 of them leave the true one within 1e-9 of it
            assert np.linalg.norm(ax + ws["grad"]) <= 1.1e-7 * np.linalg.norm(ws["grad"]), i
        for i in range(len(mat.planes)):
            s.set_planes(i, v0[i], v1[i])
        s.block(level0, sweeps=1, ridge=1e-3)
        for i, p in enumerate(mat.planes):
            uw, uh = (p[0], p[1]) if level0 else (p[2], p[3])
            ws = s.workspace(i, level0)
            S = ws["stencil"].reshape(uh, uw, 5, c, c)
            diag = S[:, :, 0]
            lam = 1e-3 * diag[..., range(c), range(c)].mean()
            # the last colour's texels ((1, 1) of each 2 x 2) met their neighbours' final corrections: the last channel
            # of each is the grid's nearest value to its one-variable minimum
            x = ws["x"].reshape(uh, uw, c)
            prev, g = ws["prev"].reshape(uh, uw, c).astype(np.float64), ws["grad"].reshape(uh, uw, c)
            full = stencil_product(ws["stencil"], ws["x"], uw, uh, c).reshape(uh, uw, c)
            q = c - 1
            a = diag[..., q, q]
            want = prev[..., q] - (g[..., q] + full[..., q] - a * x[..., q]) / (a + lam)
            got = prev[..., q] + x[..., q]
            step = 2.0 / ((1 << bits) - 1)
            sel = (slice(1, None, 2), slice(1, None, 2))
            # half a step, and the rounding of `want` to float before the grid's argmin
            assert np.all(np.abs(np.clip(want, -1, 1) - got)[sel] <= 0.5 * step + 1e-6), i
