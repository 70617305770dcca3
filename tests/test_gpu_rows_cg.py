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


@pytest.mark.parametrize("c0,c1,w,h,mip_min", [(4, 4, 68, 60, 8), (1, 4, 33, 29, 1), (3, 2, 130, 31, 8), (2, 3, 62, 57, 4),
                                               (2, 1, 400, 600, 8)])
@pytest.mark.parametrize("f32,sweeps", [(0, 1), (0, 4), (1, 3)])
def test_sweep_in_one_launch(c0, c1, w, h, mip_min, f32, sweeps):
    """A whole sweep per launch (few tiles) and a colour per launch (the last size, at level 0) against a plain walk of the
    four colours over the downloaded stencil, bit for bit: the tiles' margins give every texel the inputs it has there."""
    mat = materials.small(w + h, w, h, textures=1, c0=c0, c1=c1, mip_min=mip_min)
    mat.planes = [p for p in mat.planes if p[2] > 0 and p[3] > 0]
    rng = np.random.default_rng(w * h + sweeps)
    with Session(mat) as s:
        check(lib().nntc_b200_set_option(s.d, abi.OPT_FP32_STENCIL, f32), "option")
        for i, p in enumerate(mat.planes):
            s.set_planes(i, rng.random(p[0] * p[1] * c0) * 2 - 1, rng.random(p[2] * p[3] * c1) * 2 - 1)
        s.set_decoder(rng.standard_normal((3, s.m.nin)) * 0.3, rng.random(3))
        s.set_grids(np.full(c0, -1.0), np.full(c0, 1.0), np.full(c1, -0.9), np.full(c1, 1.1))
        for level0 in (False, True):
            rep, _ = s.block(level0, sweeps=sweeps)
            c = c0 if level0 else c1
            lo, hi = (-1.0, 1.0) if level0 else (np.float32(-0.9), np.float32(1.1))
            for i, p in enumerate(mat.planes):
                uw, uh = (p[0], p[1]) if level0 else (p[2], p[3])
                ws = s.workspace(i, level0)
                want = walk_sweeps(ws, uw, uh, c, rep[i].lambda_, float(lo), float(hi), sweeps)
                assert np.array_equal(ws["x"], want), (level0, i)


@pytest.mark.parametrize("c0,w,h", [(2, 171, 160), (2, 231, 180), (4, 171, 160), (3, 171, 160)])
def test_fp64_solve_residual(c0, w, h):
    """Block (c') on the FP64 stencil at two channels on either side of a block of texels per SM (148 blocks of 256), and at
    three and four: the solution against the downloaded stencil. The recursive residual is below 1e-10 of the right-hand
    side when the iterations stop, and FP64 recurrences over at most 200 of them leave the true one within 1e-9 of it."""
    mat = materials.small(w + h, w, h, textures=2, c0=c0, c1=2)
    rng = np.random.default_rng(w * h + c0)
    with Session(mat) as s:
        for i, p in enumerate(mat.planes):
            s.set_planes(i, rng.random(p[0] * p[1] * c0) * 2 - 1, rng.random(p[2] * p[3] * 2) * 2 - 1)
        s.set_decoder(rng.standard_normal((6, s.m.nin)) * 0.3, rng.random(6))
        s.set_grids(np.full(c0, -1.0), np.full(c0, 1.0), np.full(2, -1.0), np.full(2, 1.0))
        rep, _ = s.block(True, ridge=1e-3)
        for i, p in enumerate(mat.planes):
            ws = s.workspace(i, True)
            ax = stencil_product(ws["stencil"], ws["x"], p[0], p[1], c0) + rep[i].lambda_ * ws["x"]
            assert np.linalg.norm(ax + ws["grad"]) <= 1.1e-9 * np.linalg.norm(ws["grad"]), i


@pytest.mark.parametrize("w,h,weights", [(601, 611, "one"), (512, 750, "mixed"), (896, 600, "one")])
def test_colour_launches_of_either_residency(w, h, weights):
    """A colour of an FP32 stencil of four channels at about 480 and 500 blocks (four to an SM) and 700 (three), with symmetric
    blocks and blocks that are not, against the same walk, bit for bit."""
    mat = materials.small(w + h, w, h, textures=1, c0=4, c1=1)
    rng = np.random.default_rng(w * h)
    cw = None if weights == "one" else list(0.3 + rng.random(3))
    with Session(mat, model=abi.make_model(mat, cw=cw)) as s:
        check(lib().nntc_b200_set_option(s.d, abi.OPT_FP32_STENCIL, 1), "option")
        for i, p in enumerate(mat.planes):
            s.set_planes(i, rng.random(p[0] * p[1] * 4) * 2 - 1, rng.random(p[2] * p[3]) * 2 - 1)
        s.set_decoder(rng.standard_normal((3, s.m.nin)) * 0.3, rng.random(3))
        s.set_grids(np.full(4, -1.0), np.full(4, 1.0), np.full(1, -1.0), np.full(1, 1.0))
        rep, _ = s.block(True, sweeps=1)
        for i, p in enumerate(mat.planes):
            ws = s.workspace(i, True)
            assert np.array_equal(ws["x"], walk_sweeps(ws, p[0], p[1], 4, rep[i].lambda_, -1.0, 1.0, 1)), i


def walk_sweeps(ws, w, h, c, lam, lo, hi, sweeps):
    S, g = ws["stencil"].reshape(h, w, 5, c, c), ws["grad"].reshape(h, w, c)
    prev = ws["prev"].reshape(h, w, c).astype(np.float64)
    span = hi - lo
    values = (lo + (np.arange(256) / 255.0) * span).astype(np.float32).astype(np.float64)
    X = np.zeros((h, w, c))
    for _ in range(sweeps):
        for colour in range(4):
            cx, cy = colour & 1, colour >> 1
            ys, xs = np.meshgrid(np.arange(cy, h, 2), np.arange(cx, w, 2), indexing="ij")
            if ys.size == 0:
                continue
            nb = np.zeros(ys.shape + (c,))
            for slot, (dx, dy) in enumerate([(1, 0), (-1, 1), (0, 1), (1, 1)], 1):
                for sign in (1, -1):
                    fx, fy = xs + sign * dx, ys + sign * dy
                    ok = (fx >= 0) & (fx < w) & (fy >= 0) & (fy < h)
                    gx, gy = np.where(ok, fx, xs), np.where(ok, fy, ys)
                    block = S[ys, xs, slot] if sign > 0 else S[gy, gx, slot].swapaxes(-1, -2)
                    for i in range(c):
                        for j in range(c):
                            nb[..., i] = np.where(ok, nb[..., i] + block[..., i, j] * X[gy, gx, j], nb[..., i])
            for q in range(c):
                a = S[ys, xs, 0][..., q, q] + lam
                rest = nb[..., q].copy()
                for j in range(c):
                    if j != q:
                        rest = rest + S[ys, xs, 0][..., q, j] * X[ys, xs, j]
                want = (prev[ys, xs, q] - (g[ys, xs, q] + rest) / a).astype(np.float32).astype(np.float64)
                k = np.clip(((want - lo) / span * 255.0), 0.0, 255.0)
                k = np.clip((k + 0.5).astype(np.int64), 0, 255)
                best, dist = k, np.abs(want - values[k])
                for d in (-1, 1):
                    n = np.clip(k + d, 0, 255)
                    dn = np.abs(want - values[n])
                    better = (k + d >= 0) & (k + d <= 255) & ((dn < dist) | ((dn == dist) & (n < best)))
                    best, dist = np.where(better, n, best), np.where(better, dn, dist)
                X[ys, xs, q] = np.where(a > 0, values[best] - prev[ys, xs, q], X[ys, xs, q])
    return X.ravel()
