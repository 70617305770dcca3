"""The palette search over the channel counts it is compiled for, jointly and by coordinate sweeps, at odd sizes and each
K, against the method's own operations restated in order (float samples and decodes, double products and sums): level 0's
indices and values and the moved counts are bytes and must all be the same."""
import ctypes as C

import numpy as np
import pytest

import fp64_model as F
from nntc_b200 import abi, check, lib, materials
from nntc_b200.session import Session

pytestmark = pytest.mark.gpu

# (textures, c0, c1, w, h, bits, k): at most 8 bits in all is the joint enumeration
CASES = [(1, 2, 4, 29, 23, 3, 4), (2, 1, 1, 17, 33, 4, 4), (1, 2, 2, 21, 12, 4, 1), (1, 3, 3, 18, 15, 2, 2),
         (2, 4, 4, 16, 13, 2, 4), (1, 1, 4, 31, 9, 2, 0), (1, 3, 1, 15, 22, 3, 4), (6, 4, 2, 13, 16, 3, 4),
         (1, 4, 3, 12, 9, 4, 2)]


def tap(px, py, dx, dy, w0, h0, w, h):
    half = np.float32(0.5)
    x = px.astype(np.float32) + dx if w == w0 else ((px.astype(np.float32) + half + dx) * np.float32(w)) / np.float32(w0) - half
    y = py.astype(np.float32) + dy if h == h0 else ((py.astype(np.float32) + half + dy) * np.float32(h)) / np.float32(h0) - half
    xf, yf = np.floor(x), np.floor(y)
    fx, fy = x - xf, y - yf
    xs = [np.clip(xf.astype(int) + q, 0, w - 1) for q in (0, 1)]
    ys = [np.clip(yf.astype(int) + q, 0, h - 1) for q in (0, 1)]
    one = np.float32(1)
    wt = [(one - fx) * (one - fy), fx * (one - fy), (one - fx) * fy, fx * fy]
    return [(xs[q & 1], ys[q >> 1], wt[q]) for q in range(4)]


def blend(plane, taps):
    a, b, e, f = (wt[:, None] * plane[y, x] for x, y, wt in taps)
    return a + b + e + f


def quadratic(layout, src, v0, v1, dw, db, cw, c0, c1, k, tx, ty):
    """a0, a1, a2 of the texels (tx, ty), every candidate site's terms added in the method's order."""
    w0, h0, w1, h1 = layout
    nout, n = len(db), tx.size
    s0, t0, u1 = v0.reshape(h0, w0, c0), src.reshape(h0, w0, nout), v1.reshape(h1, w1, c1)
    q = np.zeros((1 + c0 + c0 * c0, n))
    for cand in range(9 * (k + 1)):
        pix, slot = divmod(cand, k + 1)
        px, py = tx + pix % 3 - 1, ty + pix // 3 - 1
        keep = (px >= 0) & (py >= 0) & (px < w0) & (py < h0)
        if slot == 0:
            keep &= pix == 4
        at = np.nonzero(keep)[0]
        if at.size == 0:
            continue
        x, y, gx, gy = px[at], py[at], tx[at], ty[at]
        dx = dy = np.zeros(at.size, np.float32)
        if slot:
            ox, oy = F.site_offsets(k, x, y)
            dx, dy = ox[slot - 1].astype(np.float32), oy[slot - 1].astype(np.float32)
        cbar = blend(u1, tap(x, y, dx, dy, w0, h0, w1, h1))
        beta = np.zeros((at.size, c0), np.float32)
        if slot == 0:
            alpha, target = np.ones(at.size, np.float32), t0[gy, gx]
        else:
            taps = tap(x, y, dx, dy, w0, h0, w0, h0)
            target = blend(t0, taps)
            alpha = np.zeros(at.size, np.float32)
            for qx, qy, wt in taps:
                own = (qx == gx) & (qy == gy)
                alpha = np.where(own, alpha + wt, alpha)
                beta = np.where(own[:, None], beta, beta + wt[:, None] * s0[qy, qx])
        g, s2 = np.zeros((c0, at.size)), np.zeros((c0, c0, at.size))
        a0 = []
        for r in range(nout):
            wr = dw[r]
            dec = np.full(at.size, db[r])
            for c in range(c1):
                dec = dec + wr[c] * cbar[:, c]
            slope = []
            for i in range(c0):
                sl = np.full(at.size, wr[c1 + i])
                for c in range(c1):
                    sl = sl + wr[c1 + c0 + i * c1 + c] * cbar[:, c]
                slope.append(sl)
                dec = dec + sl * beta[:, i]
            assert dec.dtype == np.float32 and target.dtype == np.float32
            res, wgt = (dec - target[:, r]).astype(np.float64), float(cw[r])
            a0.append(wgt * res * res)
            for i in range(c0):
                wq = wgt * slope[i].astype(np.float64)
                g[i] += wq * res
                for j in range(c0):
                    s2[i, j] += wq * slope[j].astype(np.float64)
        live = alpha > 0
        al = alpha.astype(np.float64)
        for r in range(nout):
            q[0, at[live]] += a0[r][live]
        for i in range(c0):
            q[1 + i, at[live]] += (al * g[i])[live]
            for j in range(c0):
                q[1 + c0 + i * c0 + j, at[live]] += (al * al * s2[i, j])[live]
    return q


def energy(q, x, c0):
    x = x.astype(np.float64)
    e = q[0].copy()
    for i in range(c0):
        e = e + 2.0 * x[:, i] * q[1 + i]
        for j in range(c0):
            e = e + x[:, i] * x[:, j] * q[1 + c0 + i * c0 + j]
    return e


def search(q, k0, pal, levels, joint, sweeps):
    """The states the texels take: a strict decrease to move, ties to the first in enumeration order."""
    c0 = len(pal)
    value = lambda idx: pal[np.arange(c0), idx]
    best = k0.copy()
    best_e = energy(q, value(best), c0)
    for chans in [list(range(c0))] if joint else [[c] for _ in range(sweeps) for c in range(c0)]:
        base = best.copy()
        low = np.full(len(base), np.inf)
        pick = base.copy()
        for n in range(levels ** len(chans)):
            idx = base.copy()
            for c in chans:
                idx[:, c] = n % levels
                n //= levels
            e = np.where((idx == base).all(1), np.inf, energy(q, value(idx), c0))
            better = e < low
            low = np.where(better, e, low)
            pick[better] = idx[better]
        move = low < best_e
        best[move] = pick[move]
        best_e = np.where(move, low, best_e)
    return best


@pytest.mark.parametrize("textures,c0,c1,w,h,bits,k", CASES)
def test_palette_search_matches_its_method(textures, c0, c1, w, h, bits, k):
    mat = materials.small(7 * w + h, w, h, textures=textures, c0=c0, c1=c1)
    nout, levels, sweeps = 3 * textures, 1 << bits, 2
    rng = np.random.default_rng(w * h + bits)
    cw = (0.5 + rng.random(nout)).astype(np.float32)
    m = abi.make_model(mat, l0_bc8=False, cw=list(cw))
    pal = np.sort(rng.random((c0, levels)).astype(np.float32) * 2 - 1, axis=1)
    for c in range(c0):
        m.bits0[c], m.palette0_len[c] = bits, levels
        for n in range(levels):
            m.palette0[c][n] = float(pal[c, n])
    dw = (rng.standard_normal((nout, m.nin)) * 0.4).astype(np.float32)
    db = rng.random(nout).astype(np.float32)
    k0 = [rng.integers(0, levels, (p[0] * p[1], c0)).astype(np.uint8) for p in mat.planes]
    v1 = [(rng.random(p[2] * p[3] * c1) * 2 - 1).astype(np.float32) for p in mat.planes]
    value = lambda idx: pal[np.arange(c0), idx]
    with Session(mat, model=m) as s:
        s.set_decoder(dw, db)
        check(lib().nntc_b200_upload_grids(s.d, C.byref(s.m)), "grids")
        for i in range(len(mat.planes)):
            s.set_planes(i, value(k0[i]).ravel(), v1[i])
            kk = np.ascontiguousarray(k0[i].ravel())
            check(lib().nntc_b200_level0_upload_indices(s.d, i, kk.ctypes.data_as(C.POINTER(C.c_uint8)), kk.size), "k0")
        rep = (abi.Level0Report * len(mat.planes))()
        ms = C.c_double()
        check(lib().nntc_b200_solve_level0_all(s.d, C.byref(s.m), k, sweeps, rep, C.byref(ms)), "palette search")
        got = [s.get_k0(i).reshape(-1, c0) for i in range(len(mat.planes))]
        vals = [s.get_v0(i).reshape(-1, c0) for i in range(len(mat.planes))]

    for i, p in enumerate(mat.planes):
        want = k0[i].copy()
        for colour in range(4):
            ty, tx = (a.ravel() for a in np.meshgrid(np.arange(colour >> 1, p[1], 2), np.arange(colour & 1, p[0], 2),
                                                     indexing="ij"))
            if tx.size == 0:
                continue
            mine = ty * p[0] + tx
            q = quadratic(p, np.asarray(mat.chain[i], np.float32), value(want), v1[i], dw, db, cw, c0, c1, k, tx, ty)
            want[mine] = search(q, want[mine], pal, levels, bits * c0 <= 8, sweeps)
        assert np.array_equal(got[i], want), (i, int((got[i] != want).any(1).sum()))
        assert np.array_equal(vals[i], value(want)), i
        assert rep[i].moved_total == int((want != k0[i]).any(1).sum()), i
