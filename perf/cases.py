"""Performance cases: the work a program has this encoder do, each case one pass through its public entry points.

Whole encodes (`Session.encode`) in both forms and in the palette mode, and the blocks an encode is made of, called one
by one as a host that drives the device seam calls them: the objective, the decoder solve, the two latents' conjugate
gradients and quantised sweeps, the BC pack with its refinement. A block's pass uploads the planes it starts from out of
pinned host memory, runs the block and downloads what it changed.

Materials are seeded, on the GPU: the correlated texture sets of the benchmark (colour, normal, roughness, occlusion,
metalness, displacement from one height field), and independent noise for a single texture. The latents a block starts
from are the kind the encoder itself starts from (level 1: block means of the source; level 0: luma and detail), and
the decoder is the least-squares fit of the source to them, so that residuals have the size they have in an encode.
"""
import ctypes as C
import math
import weakref

import numpy as np
import torch

from nntc_b200 import abi, check, lib, materials
from nntc_b200.session import Session

K = 4            # subtexel sites per texel
RIDGE = 1e-4     # the encoder's default ridge
SWEEPS = 4       # the encoder's default quantised sweeps per block
REFINE = 4       # the encoder's default refinement passes


# ---- the cases -------------------------------------------------------------------------------------------------------

def _case(name, what, textures, width, height, c0, c1, mixed):
    return {"name": name, "what": what, "textures": textures, "width": width, "height": height, "c0": c0, "c1": c1,
            "mixed": mixed}


def listed():
    return [
        # the smallest configuration of the benchmark, one texture: launches, synchronisations and host gaps count
        _case("encode_1x256x256", "encode", 1, 256, 256, 2, 4, False),
        # a whole encode of a four-texture set in the form the benchmark's headline is quoted in
        _case("encode_mixed_4x2048x1024", "encode", 4, 2048, 1024, 4, 4, True),
        # the palette mode on a small texture of no special size
        _case("encode_palette_1x100x76", "encode_palette", 1, 100, 76, 2, 4, False),
        # scoring a large six-texture material, the reference's arithmetic
        _case("objective_6x2048x2048", "objective", 6, 2048, 2048, 4, 4, False),
        # block (a), the default channel counts, FP64 sums
        _case("decoder_4x1024x1024", "decoder", 4, 1024, 1024, 2, 4, False),
        # block (a) of a large material on the tensor cores
        _case("decoder_mixed_6x2048x2048", "decoder", 6, 2048, 2048, 4, 4, True),
        # block (b)'s conjugate gradients on planes that are no power of two and divide unevenly down the chain
        _case("level1_solve_3x1000x756", "level1_solve", 3, 1000, 756, 2, 4, False),
        # block (c')'s conjugate gradients, both stencil types
        _case("level0_solve_4x1024x1024", "level0_solve", 4, 1024, 1024, 2, 4, False),
        _case("level0_solve_mixed_6x2048x2048", "level0_solve", 6, 2048, 2048, 4, 4, True),
        # the quantised sweeps of the frozen rounds, where an encode spends most of its rounds
        _case("level1_sweep_mixed_6x2048x2048", "level1_sweep", 6, 2048, 2048, 4, 4, True),
        _case("level0_sweep_4x2048x1024", "level0_sweep", 4, 2048, 1024, 4, 4, False),
        # the BC pack and its refinement, which every block-compressed asset goes through
        _case("refine_4x2048x1024", "refine", 4, 2048, 1024, 4, 4, False),
    ]


def draw(rng):
    """Any of the listed kinds at a size between 64 x 64 and 2048 x 2048 (whole encodes up to 1 Mpixel), one to six
    textures, two to four channels a level, most sizes no power of two."""
    what = rng.choice(["encode", "encode_palette", "objective", "decoder", "level1_solve", "level0_solve",
                       "level1_sweep", "level0_sweep", "refine"])
    top = {"encode": 2.0 ** 20, "encode_palette": 2.0 ** 14}.get(what, 2.0 ** 22)
    pixels = math.exp(rng.uniform(math.log(2.0 ** 12), math.log(top)))
    aspect = rng.choice([0.5, 1.0, 1.0, 1.5, 2.0])
    if rng.random() < 0.4:
        width = 1 << round(math.log2(math.sqrt(pixels * aspect)))
        height = 1 << round(math.log2(math.sqrt(pixels / aspect)))
    else:
        width = max(64, round(math.sqrt(pixels * aspect)))
        height = max(64, round(math.sqrt(pixels / aspect)))
    width, height = min(2048, max(64, width)), min(2048, max(64, height))
    c0 = rng.choice([2, 2, 3, 4, 4])
    c1 = rng.choice([2, 3, 4, 4, 4])
    if what == "encode_palette":
        c0 = 2
    return {"what": what, "textures": rng.randint(1, 6), "width": width, "height": height, "c0": c0, "c1": c1,
            "mixed": what not in ("encode_palette", "refine") and rng.random() < 0.5}


# ---- materials -------------------------------------------------------------------------------------------------------

def _noise(g, h, w, octaves, period):
    """Value noise in [0, 1]: smoothstep-interpolated random lattices, each octave half the period and amplitude."""
    out = torch.zeros(h, w, dtype=torch.float64, device="cuda")
    amp, total, p = 1.0, 0.0, float(period)
    for _ in range(octaves):
        lattice = torch.rand(math.ceil(h / p) + 2, math.ceil(w / p) + 2, generator=g, dtype=torch.float64,
                             device="cuda")
        fy = torch.arange(h, dtype=torch.float64, device="cuda") / p
        fx = torch.arange(w, dtype=torch.float64, device="cuda") / p
        iy, ix = fy.floor().long(), fx.floor().long()
        ty, tx = fy - iy, fx - ix
        sy, sx = (ty * ty * (3 - 2 * ty))[:, None], (tx * tx * (3 - 2 * tx))[None, :]
        top = lattice[iy][:, ix] * (1 - sx) + lattice[iy][:, ix + 1] * sx
        bot = lattice[iy + 1][:, ix] * (1 - sx) + lattice[iy + 1][:, ix + 1] * sx
        out += amp * (top * (1 - sy) + bot * sy)
        total += amp
        amp *= 0.5
        p = max(p / 2.0, 1.0)
    return out / total


def _base(case, seed):
    """The material's base level, h w 3T float32 in [0, 1], every value a byte over 255."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    h, w, T = case["height"], case["width"], case["textures"]
    period = max(16.0, min(h, w) / 8.0)
    if T == 1:
        img = torch.stack([_noise(g, h, w, 5, period) for _ in range(3)], -1)
        for _ in range(8):   # filled rectangles over the noise: hard edges
            r = torch.rand(7, generator=g, dtype=torch.float64, device="cuda").tolist()
            xa, xb = sorted((int(r[0] * w), int(r[1] * w)))
            ya, yb = sorted((int(r[2] * h), int(r[3] * h)))
            fill = torch.tensor(r[4:7], dtype=torch.float64, device="cuda")
            img[ya:yb, xa:xb] = 0.4 * img[ya:yb, xa:xb] + 0.6 * fill
        tex = [img * 255.0]
    else:
        H = _noise(g, h, w, 6, period)
        stops = torch.rand(3, 3, generator=g, dtype=torch.float64, device="cuda") * 255.0
        t = H * 2.0
        lo = t.long().clamp(max=1)
        f = (t - lo)[..., None]
        color = stops[lo] * (1 - f) + stops[lo + 1] * f
        color = color + 6.0 * torch.randn(h, w, 3, generator=g, dtype=torch.float64, device="cuda")
        gy, gx = torch.gradient(H)
        slope = 4.0 * period / 16.0
        n = torch.stack([-slope * gx, -slope * gy, torch.ones_like(H)], -1)
        n = n / n.norm(dim=-1, keepdim=True)
        blur = torch.nn.functional.avg_pool2d(torch.nn.functional.pad(H[None, None], (8, 8, 8, 8), mode="replicate"),
                                              17, 1)[0, 0]
        gray = lambda x: (255.0 * x)[..., None].expand(h, w, 3)   # noqa: E731
        tex = [color, (n + 1.0) * 127.5, gray(0.3 + 0.5 * H), gray(1.0 - 0.6 * (blur - H).clamp(min=0.0)),
               gray((H > 0.6).double()), gray(H)][:T]
    bytes_ = torch.cat(tex, -1).round().clamp(0, 255)
    return bytes_.float() * (torch.tensor(1.0) / torch.tensor(255.0)).item()


def _box(img):
    """One level of the default chain: the mean of 2 x 2, the last texel repeated where a side is one texel long."""
    h, w, _ = img.shape
    oh, ow = materials.mip_dim(h), materials.mip_dim(w)
    ya = (2 * torch.arange(oh, device="cuda")).clamp(max=h - 1)
    xa = (2 * torch.arange(ow, device="cuda")).clamp(max=w - 1)
    yb, xb = (ya + 1).clamp(max=h - 1), (xa + 1).clamp(max=w - 1)
    return 0.25 * ((img[ya][:, xa] + img[ya][:, xb]) + (img[yb][:, xa] + img[yb][:, xb]))


def _grid(v):
    """The nearest of the 256 values of an 8-bit grid on [-1, 1] and its index."""
    k = ((v.double() + 1.0) * 127.5).round().clamp(0, 255)
    return (-1.0 + k / 255.0 * 2.0).float(), k.to(torch.uint8)


def _inputs(case, seed):
    """Everything a case starts from, made from the seed alone: the source chain, both latents of every plane (on their
    grid where the call is one of the quantised phase) and the decoder fitted to them."""
    base = _base(case, seed)
    planes = materials.plane_sizes(case["width"], case["height"])
    chain = [base]
    for _ in range(1, len(planes)):
        chain.append(_box(chain[-1]))
    c0, c1, nout = case["c0"], case["c1"], base.shape[-1]
    quantised = case["what"] in ("level1_sweep", "level0_sweep", "refine")
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 7919)
    mix = torch.randn(nout, c0, generator=g, dtype=torch.float64, device="cuda") / math.sqrt(nout)
    v0, v1, k0, k1 = [], [], [], []
    for (w0, h0, w1, h1), src in zip(planes, chain):
        s = src.permute(2, 0, 1)[None].double()
        low = torch.nn.functional.adaptive_avg_pool2d(s, (h1, w1))
        take = [c % nout for c in range(c1)]
        a1 = (2.0 * low[0, take] - 1.0).permute(1, 2, 0)
        up = torch.nn.functional.interpolate(low, size=(h0, w0), mode="bilinear", align_corners=False)
        a0 = ((s - up)[0].permute(1, 2, 0) @ mix) * 4.0
        luma = s[0, 0] * 0.299 + s[0, 1] * 0.587 + s[0, 2] * 0.114
        a0[..., 0] = 2.0 * luma - 1.0
        a0, a1 = a0.clamp(-1, 1).float().contiguous(), a1.clamp(-1, 1).float().contiguous()
        g0, i0 = _grid(a0)
        g1, i1 = _grid(a1)
        v0.append(g0 if quantised else a0)
        v1.append(g1 if quantised else a1)
        k0.append(i0)
        k1.append(i1)
    # the decoder: least squares of the base level's source on the features at the texel centres
    w0, h0, w1, h1 = planes[0]
    step = max(1, int(math.sqrt(w0 * h0 / 65536)))
    py, px = torch.meshgrid(torch.arange(0, h0, step, device="cuda"), torch.arange(0, w0, step, device="cuda"),
                            indexing="ij")
    py, px = py.reshape(-1), px.reshape(-1)
    idx, wt = _taps(px, py, 0.0, 0.0, w0, h0, w1, h1)
    cbar = (v1[0].reshape(-1, c1).double()[idx] * wt[..., None]).sum(1)
    phi = _features(v0[0].double()[py, px], cbar)
    X = torch.cat([phi, torch.ones_like(phi[:, :1])], 1)
    A = X.T @ X
    A += 1e-6 * A.diagonal().mean() * torch.eye(A.shape[0], dtype=torch.float64, device="cuda")
    W = torch.linalg.solve(A, X.T @ base.double()[py, px]).T.float()
    return {"planes": planes, "chain": chain, "v0": v0, "v1": v1, "k0": k0, "k1": k1,
            "w": W[:, :-1].contiguous(), "b": W[:, -1].contiguous()}


# ---- a case's state --------------------------------------------------------------------------------------------------

class State:
    pass


def _pinned(t):
    return t.reshape(-1).cpu().pin_memory().numpy()


def _empty(n, dtype):
    return torch.empty(n, dtype=dtype, pin_memory=True).numpy()


def _ptr(a, ty):
    return a.ctypes.data_as(C.POINTER(ty))


def prepare(case, seed):
    inp = _inputs(case, seed)
    planes = inp["planes"]
    base = inp["chain"][0]
    mat = materials.Material("case", [np.empty((case["height"], case["width"], 3), np.uint8)] * case["textures"],
                             case["c0"], case["c1"], K)
    mat.planes, mat.chain = planes, [base.cpu().numpy()]
    mat.per_site = materials.mip_weights(planes, "pixels", 0.5, K)
    s = State()
    what = s.what = case["what"]
    s.session = Session(mat, model=abi.make_model(mat, l0_bc8=what != "encode_palette"), from_base=True)
    s.close = weakref.finalize(s, s.session.close)
    S, n = s.session, len(planes)
    if what in ("encode", "encode_palette"):
        s.args = abi.EncodeArgs()
        lib().nntc_b200_encode_defaults(C.byref(s.args))
        s.args.form = 1 if case["mixed"] else 0
        return s
    for opt in (abi.OPT_MIXED_PRECISION_GRAM, abi.OPT_MIXED_OBJECTIVE, abi.OPT_FP32_STENCIL):
        check(lib().nntc_b200_set_option(S.d, opt, 1 if case["mixed"] else 0), "option")
    S.set_decoder(inp["w"].cpu().numpy(), inp["b"].cpu().numpy())
    S.set_grids(np.full(case["c0"], -1.0), np.full(case["c0"], 1.0), np.full(case["c1"], -1.0),
                np.full(case["c1"], 1.0))
    s.v0, s.v1 = [_pinned(x) for x in inp["v0"]], [_pinned(x) for x in inp["v1"]]
    s.k0, s.k1 = [_pinned(x) for x in inp["k0"]], [_pinned(x) for x in inp["k1"]]
    for i in range(n):
        S.set_planes(i, s.v0[i], s.v1[i])
    f32, u8 = torch.float32, torch.uint8
    s.blocks = [((p[0] + 3) // 4) * ((p[1] + 3) // 4) for p in planes]
    c0, c1 = case["c0"], case["c1"]
    if what == "level1_solve":
        s.out = [_empty(p[2] * p[3] * c1, f32) for p in planes]
    elif what == "level0_solve":
        s.out = [_empty(p[0] * p[1] * c0, f32) for p in planes]
    elif what == "level1_sweep":
        s.out = [_empty(p[2] * p[3] * c1, u8) for p in planes]
    elif what == "level0_sweep":
        s.out = [_empty(p[0] * p[1] * c0, u8) for p in planes]
    elif what == "refine":
        s.ep = [_empty(b * c0 * 2, u8) for b in s.blocks]
        s.sel = [_empty(b * c0 * 16, u8) for b in s.blocks]
    return s


# ---- a pass ----------------------------------------------------------------------------------------------------------

def _encode(s):
    r, out = s.session.encode(s.args, outputs=True)
    w, b = s.session.decoder()
    got = {"k0": out["k0"], "k1": out["k1"], "w": w, "b": b,
           "e": np.array([r.e_init, r.e_after_rounds, r.e_ship, r.centre_mse, r.sampled_mse]),
           "psnr": np.array(r.psnr[:s.session.m.textures])}
    if out["ep"] is not None:
        got["ep"], got["sel"] = out["ep"], out["sel"]
    return got


def run(s):
    S, L, what = s.session, lib(), s.what
    n = S.m.nplanes
    if what in ("encode", "encode_palette"):
        return _encode(s)
    if what == "objective":
        r = S.objective(K)
        return {"e": np.array([r.e, r.centre_mse, r.sampled_mse]), "e_plane": np.array(r.e_plane[:n]),
                "centre_plane": np.array(r.centre_plane[:n])}
    if what == "decoder":
        S.m.has_decoder = 0
        S.solve_decoder(K)
        w, b = S.decoder()
        return {"w": w, "b": b}
    level0 = what in ("level0_solve", "level0_sweep", "refine")
    v, k = (s.v0, s.k0) if level0 else (s.v1, s.k1)
    for i in range(n):
        if level0:
            S.set_planes(i, v0=v[i])
        else:
            S.set_planes(i, v1=v[i])
    if what in ("level1_solve", "level0_solve"):
        S.block(level0, 0, K, RIDGE)
        get = L.nntc_b200_level0_download_values if level0 else L.nntc_b200_level1_download
        for i in range(n):
            check(get(S.d, i, _ptr(s.out[i], C.c_float), s.out[i].size), "download")
        return {"v": s.out}
    put = L.nntc_b200_level0_upload_indices if level0 else L.nntc_b200_level1_upload_indices
    for i in range(n):
        check(put(S.d, i, _ptr(k[i], C.c_uint8), k[i].size), "upload")
    if what == "refine":
        ms = C.c_double()
        rep = (abi.BcReport * REFINE)()
        check(L.nntc_b200_bc_pack_prepare(S.d, C.byref(S.m), K, 1, None, C.byref(ms)), "pack")
        check(L.nntc_b200_bc_refine(S.d, C.byref(S.m), REFINE, rep, C.byref(ms)), "refine")
        check(L.nntc_b200_bc_state_save(S.d, C.byref(S.m), abi.u8_ptrs(s.ep), abi.u8_ptrs(s.sel)), "save")
        return {"ep": s.ep, "sel": s.sel, "improved": np.array([r.improved for r in rep]),
                "delta_e": np.array([r.delta_e for r in rep])}
    rep, _ = S.block(level0, SWEEPS, K, RIDGE)
    get = L.nntc_b200_level0_download if level0 else L.nntc_b200_level1_download_indices
    for i in range(n):
        check(get(S.d, i, _ptr(s.out[i], C.c_uint8), s.out[i].size), "download")
    return {"k": s.out, "moved": np.array([r.moved for r in rep]), "ridge": np.array([r.lambda_ for r in rep])}


# ---- what a pass cannot do without -----------------------------------------------------------------------------------

def work(case):
    """Bytes: the source, the latents and the indices the pass reads and writes, each once. Flops: at every site of
    every plane the decode and what the pass forms from it; an encode is its default's passes over the sites."""
    planes = materials.plane_sizes(case["width"], case["height"])
    c0, c1, nout = case["c0"], case["c1"], 3 * case["textures"]
    p0, p1 = sum(p[0] * p[1] for p in planes), sum(p[2] * p[3] for p in planes)
    nin, sites = c0 + c1 + c0 * c1, p0 * (1 + K)
    source, l0, l1 = 4.0 * p0 * nout, 4.0 * p0 * c0, 4.0 * p1 * c1
    decode = 2.0 * sites * nin * nout
    mono0, mono1 = 1 + c1 + c1 * (c1 + 1) // 2, 1 + c0 + c0 * (c0 + 1) // 2

    def assemble(level0):
        # the gradient's term per site, then each site's monomials into the ten pairs of its four texels, then the
        # five blocks of every texel expanded
        c, mono, t = (c0, mono0, p0) if level0 else (c1, mono1, p1)
        return decode + 4.0 * sites * nout * c + 20.0 * sites * mono + 10.0 * t * mono * c * c

    def product(level0):   # one product with the assembled stencil, nine C x C blocks a texel
        c, t = (c0, p0) if level0 else (c1, p1)
        return 18.0 * t * c * c

    what = case["what"]
    if what == "objective":
        return {"bytes": source + l0 + l1, "flops": decode + 4.0 * sites * nout}
    if what == "decoder":
        return {"bytes": source + l0 + l1, "flops": sites * (nin + 1.0) * (nin + 2.0) + 2.0 * sites * (nin + 1) * nout}
    if what in ("level1_solve", "level0_solve"):
        lv0 = what == "level0_solve"
        return {"bytes": source + l0 + l1 + (l0 if lv0 else l1), "flops": assemble(lv0) + 10 * product(lv0)}
    if what in ("level1_sweep", "level0_sweep"):
        lv0 = what == "level0_sweep"
        own = l0 if lv0 else l1
        return {"bytes": source + l0 + l1 + 0.5 * own, "flops": assemble(lv0) + SWEEPS * product(lv0)}
    if what == "refine":
        return {"bytes": source + 2 * l0 + l1 + p0 * c0 * (1.0 + 2.0 / 16.0),
                "flops": assemble(True) + REFINE * 4 * product(True)}
    rounds = 8.0
    passes = assemble(False) + assemble(True) + 2 * SWEEPS * product(True) + 3 * decode
    shipped = p0 * c0 * 1.0 + p1 * c1 + p0 * c0 * (1.0 + 2.0 / 16.0)
    return {"bytes": rounds * source + shipped, "flops": rounds * passes}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------

def _offsets(j, px, py):
    """The offset of site j of every pixel: 0 the centre, then the rotated grid, a quarter turn per parity class."""
    z = torch.zeros(px.shape, dtype=torch.float64, device="cuda")
    if j == 0:
        return z, z
    ox, oy = [(-0.375, -0.125), (-0.125, 0.375), (0.125, -0.375), (0.375, 0.125)][j - 1]
    x, y = z + ox, z + oy
    turns = (py & 1) * 2 + (px & 1)
    for r in range(3):
        m = turns > r
        x, y = torch.where(m, -y, x), torch.where(m, x, y)
    return x, y


def _taps(px, py, dx, dy, w0, h0, w, h):
    """The four texels (row-major) of a w x h plane a site of a w0 x h0 plane reads, and their bilinear weights."""
    x = (px.double() + 0.5 + dx) * w / w0 - 0.5
    y = (py.double() + 0.5 + dy) * h / h0 - 0.5
    xf, yf = x.floor(), y.floor()
    fx, fy = x - xf, y - yf
    x0, x1 = xf.long().clamp(0, w - 1), (xf.long() + 1).clamp(0, w - 1)
    y0, y1 = yf.long().clamp(0, h - 1), (yf.long() + 1).clamp(0, h - 1)
    idx = torch.stack([y0 * w + x0, y0 * w + x1, y1 * w + x0, y1 * w + x1], 1)
    wt = torch.stack([(1 - fx) * (1 - fy), fx * (1 - fy), (1 - fx) * fy, fx * fy], 1)
    return idx, wt


def _features(s, c):
    return torch.cat([c, s, (s[:, :, None] * c[:, None, :]).reshape(s.shape[0], -1)], 1)


def _sites(inp, i, j):
    """Site j of every pixel of plane i: both latents' samples, the target, and the two tap sets."""
    w0, h0, w1, h1 = inp["planes"][i]
    n = torch.arange(w0 * h0, device="cuda")
    py, px = n // w0, n % w0
    dx, dy = _offsets(j, px, py)
    c0, c1 = inp["v0"][i].shape[-1], inp["v1"][i].shape[-1]
    t1 = _taps(px, py, dx, dy, w0, h0, w1, h1)
    t0 = _taps(px, py, dx, dy, w0, h0, w0, h0)

    def at(a, taps):
        out = torch.zeros(n.numel(), a.shape[-1], dtype=torch.float64, device="cuda")
        for q in range(4):
            out += a[taps[0][:, q]].double() * taps[1][:, q:q + 1]
        return out

    return (at(inp["v0"][i].reshape(-1, c0), t0), at(inp["v1"][i].reshape(-1, c1), t1),
            at(inp["chain"][i].reshape(w0 * h0, -1), t0), t0, t1)


def _exact_objective(inp):
    W, b = inp["w"].double(), inp["b"].double()
    weight = materials.mip_weights(inp["planes"], "pixels", 0.5, K)
    nout = W.shape[0]
    num = den = 0.0
    e_plane, c_plane, f_plane = [], [], []
    for i, p in enumerate(inp["planes"]):
        pix = p[0] * p[1]
        sums = []
        for j in range(K + 1):
            s, c, t, _, _ = _sites(inp, i, j)
            sums.append(float((_features(s, c) @ W.T + b - t).square().sum()))
        total, frac = sum(sums), sum(sums[1:])
        num += weight[i] * total
        den += weight[i] * pix * (1 + K)
        e_plane.append(total / (nout * pix * (1 + K)))
        c_plane.append(sums[0] / (nout * pix))
        f_plane.append(frac / (nout * pix * K))
    return [num / (nout * den), c_plane[0], f_plane[0]], e_plane, c_plane


def _exact_decoder(inp):
    weight = materials.mip_weights(inp["planes"], "pixels", 0.5, K)
    A = B = 0.0
    for i in range(len(inp["planes"])):
        for j in range(K + 1):
            s, c, t, _, _ = _sites(inp, i, j)
            f = _features(s, c)
            X = torch.cat([f, torch.ones_like(f[:, :1])], 1)
            A = A + weight[i] * (X.T @ X)
            B = B + weight[i] * (X.T @ t)
    A = A + 1e-9 * A.diagonal().mean() * torch.eye(A.shape[0], dtype=torch.float64, device="cuda")
    W = torch.linalg.solve(A, B).T
    return W[:, :-1], W[:, -1]


def _exact_solve(inp, i, level0):
    """Plane i's latent after its block: v + d, (H + lambda I) d = -J^T r, lambda the ridge times H's mean diagonal."""
    W, b = inp["w"].double(), inp["b"].double()
    nout = W.shape[0]
    v = inp["v0" if level0 else "v1"][i].double()
    c, c0, c1 = v.shape[-1], inp["v0"][i].shape[-1], inp["v1"][i].shape[-1]
    v = v.reshape(-1, c)
    M = W[:, c0 + c1:].reshape(nout, c0, c1)
    sets, grad, diag = [], torch.zeros_like(v), 0.0
    for j in range(K + 1):
        s, cb, t, t0, t1 = _sites(inp, i, j)
        r = _features(s, cb) @ W.T + b - t
        if level0:
            G = W[None, :, c1:c1 + c0] + torch.einsum("rij,nj->nri", M, cb)
        else:
            G = W[None, :, :c1] + torch.einsum("rij,ni->nrj", M, s)
        idx, wt = t0 if level0 else t1
        H = torch.einsum("nra,nrb->nab", G, G)
        g = torch.einsum("nra,nr->na", G, r)
        del G, r, s, cb, t
        # a texel met by several of a site's taps has their weights summed
        same = (idx[:, :, None] == idx[:, None, :]).double()
        diag += float((torch.einsum("nq,nqp,np->n", wt, same, wt) * H.diagonal(dim1=1, dim2=2).sum(1)).sum())
        for q in range(4):
            grad.index_add_(0, idx[:, q], g * wt[:, q:q + 1])
        sets.append((idx, wt, H))
    lam = RIDGE * diag / v.numel()

    def product(x):
        out = lam * x
        for idx, wt, H in sets:
            y = sum(x[idx[:, q]] * wt[:, q:q + 1] for q in range(4))
            z = torch.einsum("nab,nb->na", H, y)
            for q in range(4):
                out.index_add_(0, idx[:, q], z * wt[:, q:q + 1])
        return out

    # block-Jacobi preconditioned conjugate gradients to the rounding of 64 bits
    D = torch.zeros(v.shape[0], c, c, dtype=torch.float64, device="cuda")
    for idx, wt, H in sets:
        for q in range(4):
            D.index_add_(0, idx[:, q], H * (wt[:, q] ** 2)[:, None, None])
    D = torch.linalg.inv(D + lam * torch.eye(c, dtype=torch.float64, device="cuda"))
    x, r = torch.zeros_like(v), -grad
    z = torch.einsum("nab,nb->na", D, r)
    p, rz, stop = z.clone(), float((r * z).sum()), 1e-12 * float(grad.norm())
    for _ in range(400):
        if float(r.norm()) <= stop:
            break
        hp = product(p)
        a = rz / float((p * hp).sum())
        x += a * p
        r -= a * hp
        z = torch.einsum("nab,nb->na", D, r)
        new = float((r * z).sum())
        p = z + (new / rz) * p
        rz = new
    return v + x


def exact(case, seed):
    what = case["what"]
    if what not in ("objective", "decoder", "level1_solve", "level0_solve"):
        return None   # indices, selectors and whole encodes: decisions, which have no value in 64 bits
    inp = _inputs(case, seed)
    if what == "objective":
        e, e_plane, c_plane = _exact_objective(inp)
        return {"e": np.array(e), "e_plane": np.array(e_plane), "centre_plane": np.array(c_plane)}
    if what == "decoder":
        w, b = _exact_decoder(inp)
        return {"w": w, "b": b}
    level0 = what == "level0_solve"
    return {"v": [_exact_solve(inp, i, level0).reshape(-1) for i in range(len(inp["planes"]))]}
