// assemble.cu: the stencil and gradient assembly of blocks (b) and (c'), restructured for B200 - and bit-identical
// to the reference's per-texel gather (src/solve_level1.cu:259-581).
//
// The reference gives each texel one thread that walks every site whose bilinear footprint can reach it and, for each
// site that does, recomputes the whole site: its G (or Q) matrix, its residual and G^T diag(cw) r - about a thousand
// operations - then adds the site's monomials into five slots of fifteen sums. Every site is recomputed by each of the
// (up to four) texels it touches, and the 75 double accumulators of a thread spill.
//
// Two observations make it cheap without changing a single rounding:
//
//   - the gradient term of a site, t_s = G^T diag(cw) r, does not depend on which texel gathers it. One thread per
//     SITE computes it once, with the reference's arithmetic (rows in order, each column's sum over the rows in order,
//     no contraction), into a per-site buffer of doubles; the gather then adds w_self * t_s exactly as the reference
//     adds w_self * acc.
//   - the stencil's monomial sums need only the site's sample of the OTHER latent (a bilinear blend of four texels,
//     which k_site_terms also stores per site) and the tap weights - a few dozen operations. They are gathered per
//     (texel, slot): each slot's sums receive the same terms in the same site order as the reference's, so every sum,
//     and the expansion against the monomial matrices after it, is the same bits. gather.cu does it in tiles,
//     gather_any.cu for the planes whose visits are not tabled.
//
// Every plane of the chain is in each launch (nb::Planes); the per-site buffer holds every plane's sites.

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "footprint.cuh"
#include "gather.cuh"
#include "site_terms.cuh"

namespace nb
{

constexpr int SITE_THREADS = 256;
struct TargetOffsets
{
    long long site0[MAX_PLANES + 1];    // the first fractional site of each plane
};

// The float target of every fractional site (j > 0): the source blended at the site's four level-0 taps, in blend()'s
// order and arithmetic (src/solve_level1.cu:322-333). It depends on nothing but the source and K, neither of which an
// encode changes, so it is formed once per device model and K and then read by every k_site_terms launch.
template <int NOUT>
__global__ void __launch_bounds__(SITE_THREADS) k_site_targets(Planes P, float* tgt, const __grid_constant__ TargetOffsets O)
{
    const long long base = (long long)blockIdx.x * blockDim.x;
    const int pl = plane_of(P, base);
    const PlaneView& V = P.p[pl];
    const long long fi = base - P.start[pl] + threadIdx.x;
    const int kc = P.kc;
    if (fi >= (long long)V.w0 * V.h0 * kc)
        return;
    const long long pixel = fi / kc;
    const int j = 1 + (int)(fi % kc);
    const int px = (int)(pixel % V.w0), py = (int)(pixel / V.w0);
    float dx, dy;
    site_offset(kc, j, px, py, dx, dy);
    const Tap t0 = tap_at(px, py, dx, dy, V.w0, V.h0, V.w0, V.h0);
    float w0[4];
    tap_weights(t0, w0);
    float* out = tgt + (size_t)(O.site0[pl] + fi) * NOUT;
#pragma unroll
    for (int r = 0; r < NOUT; r++)
    {
        const float* s = V.src + r;
        out[r] = w0[0] * __ldg(s + ((size_t)t0.y0 * V.w0 + t0.x0) * NOUT) +
                 w0[1] * __ldg(s + ((size_t)t0.y0 * V.w0 + t0.x1) * NOUT) +
                 w0[2] * __ldg(s + ((size_t)t0.y1 * V.w0 + t0.x0) * NOUT) +
                 w0[3] * __ldg(s + ((size_t)t0.y1 * V.w0 + t0.x1) * NOUT);
    }
}

// One thread per site: t_s[a] = sum_r cw_r G[r][a] res_r (level 1, block b) or sum_r cw_r Q[r][a] res_r (level 0,
// block c'), in the reference's order of operations (src/solve_level1.cu:335-361, 518-544).
// ---- the gather's visit tables (gather.cuh)

// Every class's visits, in the reference's site order, for the FP64 sums (tab64) and the FP32 sums (tab32: the product
// of the weights rounded to float); off: each class's range per slot, the same in both.
template <bool LEVEL0>
static bool build_gather_table(int kc, std::vector<int4>& tab64, std::vector<int4>& tab32,
                               int (&off)[GATHER_CLASSES][SLOTS + 1])
{
    constexpr int AX = LEVEL0 ? AXIS_CLASSES0 : AXIS_CLASSES1, scale = LEVEL0 ? 1 : 4;
    // a texel of each axis class and the length of a plane it is one of
    const int at0[AXIS_CLASSES0] = { 0, 32, 33, 62, 63 }, len0[AXIS_CLASSES0] = { 64, 64, 64, 63, 64 };
    const int at1[AXIS_CLASSES1] = { 0, 32, 63 }, len1[AXIS_CLASSES1] = { 64, 64, 64 };
    tab64.clear();
    tab32.clear();
    for (int cls = 0; cls < AX * AX; cls++)
    {
        const int ax = cls % AX, ay = cls / AX;
        const int tx = LEVEL0 ? at0[ax] : at1[ax], w = LEVEL0 ? len0[ax] : len1[ax];
        const int ty = LEVEL0 ? at0[ay] : at1[ay], h = LEVEL0 ? len0[ay] : len1[ay];
        const int w0 = scale * w, h0 = scale * h;
        for (int slot = 0; slot < SLOTS; slot++)
        {
            off[cls][slot] = (int)tab64.size();
            int ox, oy;
            slot_offset(slot, ox, oy);
            const int nbx = tx + ox, nby = ty + oy;
            if (nbx < 0 || nbx >= w || nby >= h)
                continue;   // no neighbour: a zero block, no list
            int px_lo, px_hi, py_lo, py_hi, qx_lo, qx_hi, qy_lo, qy_hi;
            reach(tx, w0, w, px_lo, px_hi);
            reach(ty, h0, h, py_lo, py_hi);
            reach(nbx, w0, w, qx_lo, qx_hi);
            reach(nby, h0, h, qy_lo, qy_hi);
            px_lo = std::max(px_lo, qx_lo);
            px_hi = std::min(px_hi, qx_hi);
            py_lo = std::max(py_lo, qy_lo);
            py_hi = std::min(py_hi, qy_hi);
            for (int py = py_lo; py <= py_hi; py++)
                for (int px = px_lo; px <= px_hi; px++)
                    for (int j = 0; j <= kc; j++)
                    {
                        float ws, wo;
                        if (!site_touches<LEVEL0>(px, py, j, kc, tx, ty, nbx, nby, w0, h0, w, h, ws, wo))
                            continue;
                        const int dpx = px - scale * tx, dpy = py - scale * ty;
                        // the site's place from the lane's own: the lane's texel is TILE0's column cx of its pair
                        const int qx = LEVEL0 ? (tx & 1) + 1 + dpx : dpx + 2, qy = LEVEL0 ? dpy + 1 : dpy + 2;
                        if (qx < 0 || qy < 0 || qx > (LEVEL0 ? 3 : 7) || qy > (LEVEL0 ? 2 : 7))
                            return false;   // outside the tile's margin: not a visit these tiles hold
                        int4 e;
                        const int place = tile_site<LEVEL0>(qx, qy, j, 1 + kc) * (int)sizeof(float4);
                        e.x = place | (dpx + 2) << 16 | (dpy + 2) << 20 | j << 24;
                        std::memcpy(&e.y, &ws, sizeof(float));
                        const double s64 = (double)ws * (double)wo;
                        std::memcpy(&e.z, &s64, sizeof(double));
                        tab64.push_back(e);
                        const float s32 = ws * wo;
                        std::memcpy(&e.z, &s32, sizeof(float));
                        e.w = place;
                        tab32.push_back(e);
                    }
        }
        off[cls][SLOTS] = (int)tab64.size();
    }
    return true;
}

// The tiles of k_gather_any1 up to which it takes a level's planes that are not tabled; with more of them the walk does.
// The tiles test each pixel once for five warps, whatever comes of it, and stage its sites, which pays the more sites a
// pixel has; a thread a (texel, slot) waits longer but keeps more of them in flight, so that it gains as the launch
// grows. FP32 terms of four channels are staged side by side with the samples; an odd count of FP64 ones a value at a
// time. The diagonal blocks alone leave three of the five warps idle. Where the lines lie, from both at 179 to 57404 tiles
// (300 x 200 to 5500 x 4000), level 0 of two and of four channels: the assembly's time in the walk over that in tiles, at
// about 950, 2050, 5450 and 15700 tiles (31400 where it says so), mean of the two level-0 counts:
//   every slot     K = 0                 K = 1                 K = 2                 K = 4
//   FP64  1  .90 .82 .65 .61      1.16 1.06 .89 .83     1.40 1.17 1.00 .94    1.68 1.33 1.09 1.01 (1.04)
//         2  1.03 .91 .76 .71     1.33 1.16 .98 .93     1.51 1.32 1.10 1.04   1.89 1.54 1.27 1.19 (1.17)
//         3  .69 .62 .50 .46      1.00 .88 .73 .69      1.13 .97 .81 .76      1.33 1.08 .87 .79
//         4  .88 .77 .64 .60      1.17 1.01 .86 .82     1.36 1.17 1.00 .94    1.74 1.38 1.11 1.02 (1.00)
//   FP32 1-3 .91 .82 .63 .58      1.21 1.09 .87 .81     1.37 1.17 .96 .90     1.76 1.39 1.12 1.03 (1.00)
//         4  1.31 1.06 .88 .81    1.66 1.34 1.11 1.04   1.85 1.48 1.23 1.16   2.34 1.84 1.47 1.35 (1.32)
//   the diagonal blocks alone
//   FP64  1  .78 .57 .41 .36      .99 .74 .57 .51       1.19 .85 .67 .59      1.46 .94 .70 .61
//         2  .91 .69 .57 .50      1.12 .83 .73 .65      1.31 .99 .84 .74      1.67 1.15 .90 .79
//         3  .61 .44 .34 .30      .82 .62 .55 .49       .95 .72 .58 .51       1.14 .78 .59 .52
//         4  .71 .56 .55 .49      .94 .75 .71 .65       1.07 .90 .82 .74      1.55 1.02 .87 .78
//   FP32 1-3 .80 .60 .42 .34      1.05 .78 .62 .53      1.24 .87 .68 .57      1.59 1.00 .74 .61
//         4  .98 .84 .78 .67      1.21 1.02 .95 .82     1.39 1.13 1.06 .91    1.85 1.30 1.13 .98
static int any_tiles_line(bool f32, int c, int kc, bool every_slot)
{
    constexpr int ALL = 1 << 30;
    constexpr int LINE[2][5][4] = {   // the sums' type and channels as above, then K = 0, 1, 2, 4
        { { 700, 2500, 5000, ALL }, { 1000, 5000, ALL, ALL }, { 400, 1050, 1700, 2700 }, { 500, 1800, 4500, 30000 },
          { 700, 2800, 4000, 30000 } },
        { { 650, 950, 1350, 1800 }, { 800, 1300, 2000, 2800 }, { 500, 700, 850, 1300 }, { 600, 850, 1200, 2100 },
          { 700, 950, 1400, 2000 } }
    };
    constexpr int LINE_FP32_4[2][4] = { { 2500, ALL, ALL, ALL }, { 950, 1900, 5000, 10000 } };
    const int slots = every_slot ? 0 : 1, k = kc < 3 ? kc : 3;
    return f32 && c == MAX_CH ? LINE_FP32_4[slots][k] : LINE[slots][f32 ? 4 : c - 1][k];
}

// One of the gather's launches, for the other latent's channel count (ny).
#define NB_GATHER(launch, ...)                                                                                        \
    do                                                                                                                \
    {                                                                                                                 \
        switch (ny)                                                                                                   \
        {                                                                                                             \
        case 1: NB_TRY((launch<TS, 1>(__VA_ARGS__))); break;                                                          \
        case 2: NB_TRY((launch<TS, 2>(__VA_ARGS__))); break;                                                          \
        case 3: NB_TRY((launch<TS, 3>(__VA_ARGS__))); break;                                                          \
        default: NB_TRY((launch<TS, 4>(__VA_ARGS__))); break;                                                         \
        }                                                                                                             \
    } while (0)

// The gather of every plane: the tabled planes in one launch, the others in one more, or two.
template <typename TS>
static int gather_planes(nntc_b200_device* d, int level0, const Planes& P, int nmono, const double* mono, int slots)
{
    const int k = P.kc, ny = level0 ? d->c1 : d->c0, c = level0 ? d->c0 : d->c1;
    TileArgs<TS> A{};
    A.terms = d->site_terms;
    A.y = (const float4*)d->site_y;
    A.slots = slots;
    A.bc_copy = level0 && sizeof(TS) == sizeof(double) && d->bc_copy ? 1 : 0;
    d->bc_copied = A.bc_copy && slots == SLOTS;
    A.plain = 1;
    int q = 0;
    for (int L = 0; L < MAX_MONO; L++)
        if (mono_used(L, ny))
        {
            const double* mat = mono + (size_t)q++ * c * c;
            for (int i = 0; i < c; i++)
                for (int j = 0; j < c; j++)
                {
                    const TS v = (TS)mat[i * c + j];
                    A.mono[L][i * c + j] = v;
                    A.plain = A.plain && std::isfinite(v) && mat[i * c + j] == mat[j * c + i];
                }
        }
    d->sten_symmetric[level0] = A.plain != 0;   // symmetric matrices expand to symmetric blocks
    if (q != nmono)
    {
        set_error(NNTC_B200_ERR_STATE, "monomial layout and count disagree");
        return NNTC_B200_ERR_STATE;
    }
    if (d->gtab_kc[level0] != k)
    {
        std::vector<int4> tab64, tab32;
        int off[GATHER_CLASSES][SLOTS + 1] = {};
        if (!(level0 ? build_gather_table<true>(k, tab64, tab32, off)
                     : build_gather_table<false>(k, tab64, tab32, off)) ||
            tab64.size() > (size_t)GATHER_TABLE_MAX)
        {
            set_error(NNTC_B200_ERR_STATE, "the gather's visits outgrew their tiles or their table");
            return NNTC_B200_ERR_STATE;
        }
        int4* tab = (int4*)d->gtab[level0];
        NB_TRY(upload(d, tab, tab64.data(), tab64.size() * sizeof(int4)));
        NB_TRY(upload(d, tab + GATHER_TABLE_MAX, tab32.data(), tab32.size() * sizeof(int4)));
        static_assert(sizeof(d->gtab_off[0]) == sizeof(off), "visit table offsets");
        std::memcpy(d->gtab_off[level0], off, sizeof(off));
        d->gtab_kc[level0] = k;
    }
    A.tab = (const int4*)d->gtab[level0] + (sizeof(TS) == sizeof(double) ? 0 : GATHER_TABLE_MAX);
    std::memcpy(A.off, d->gtab_off[level0], sizeof(A.off));
    auto pow2 = [](int v) { return v > 0 && (v & (v - 1)) == 0; };
    // A level-1 plane that is not tabled goes to k_gather_any1 in tiles of the same texels, wherever a tile's sites fit
    // shared memory and the level has no more tiles than any_tiles_line. At K = 4 a tile of four pixels a texel takes 76.7 KB and those of an odd chain's planes up to
    // 80.3 KB: two to an SM either way, so that they share a launch. A launch of their own for the deepest planes' few
    // tiles costs a tile's whole walk on an idle GPU (us, both launches against one: 450 x 333 292 / 200, 1000 x 756 751 /
    // 638, 2047 x 1023 2073 / 1938). Planes whose tile leaves room for one alone are launched apart, or the others would
    // lose their second tile - in the same launch when there are too few tiles for that to matter.
    constexpr size_t SM_SHARED = 228 * 1024, BLOCK_RESERVED = 1024, ANY_STATIC = MAX_MONO * 32 * sizeof(TS);
    constexpr size_t ANY_SHARED = SM_SHARED / 2 - BLOCK_RESERVED - ANY_STATIC;
    constexpr int ANY_FEW = 2 * 148;
    AnyTiles R{};
    size_t any_bytes[MAX_PLANES] = {};
    auto widest = [](int n, int n0, int tile) {
        int most = 0;
        for (int t = 0; t < n; t += tile)
        {
            int lo, hi, other;
            reach(t, n0, n, lo, other);
            reach(std::min(t + tile, n) - 1, n0, n, other, hi);
            most = std::max(most, hi - lo + 1);
        }
        return most;
    };
    auto any_tiles_of = [&](int i) {
        return any_bytes[i] ? ((P.p[i].w + TILE1_W - 1) / TILE1_W) * ((P.p[i].h + TILE1_H - 1) / TILE1_H) : 0;
    };
    long long at = 0;
    int any_tiles = 0;
    for (int i = 0; i < P.n; i++)
    {
        const PlaneView& v = P.p[i];
        const bool tiled = v.w >= 2 && v.h >= 2 &&
                           (level0 || (v.w0 == 4 * v.w && v.h0 == 4 * v.h && pow2(v.w) && pow2(v.h)));
        A.site0[i] = at;
        at += (long long)v.w0 * v.h0 * (1 + k);
        const int tw = level0 ? TILE0_W : TILE1_W, th = level0 ? TILE0_H : TILE1_H;
        A.btiles[i] = tiled ? ((v.w + tw - 1) / tw) * ((v.h + th - 1) / th) : 0;
        if (!tiled && !level0)
        {
            R.px[i] = widest(v.w, v.w0, TILE1_W);
            R.py[i] = widest(v.h, v.h0, TILE1_H);
            const size_t bytes = any_tile_bytes(R.px[i], R.py[i], 1 + k);
            any_bytes[i] = bytes <= ANY_SHARED_MAX && R.px[i] * (1 + k) < 1024 ? bytes : 0;
            any_tiles += any_tiles_of(i);
        }
    }
    A.site0[P.n] = at;
    if (any_tiles > any_tiles_line(sizeof(TS) == sizeof(float), c, k, slots == SLOTS))
        any_tiles = 0;
    WalkBlocks B{};
    long long walk = 0;
    for (int i = 0; i < P.n; i++)
    {
        const PlaneView& v = P.p[i];
        const bool walked = A.btiles[i] == 0 && (any_bytes[i] == 0 || any_tiles == 0);
        B.start[i] = walk;
        const long long largest = (long long)((v.w + 1) / 2) * ((v.h + 1) / 2);   // colour 0
        walk += walked ? (largest + WALK_THREADS - 1) / WALK_THREADS * 4 * slots : 0;
    }
    B.start[P.n] = walk;
    int tiles = 0;
    for (int i = P.n - 1; i >= 0; i--)
        A.bend[i] = tiles += A.btiles[i];
    if (walk > 0)
        NB_GATHER(launch_gather_walk, d, level0, P, A, B);
    for (int group = 0; group < 2 && any_tiles > 0; group++)   // the larger tiles, then the others
    {
        TileArgs<TS> G = A;
        size_t shared = 0;
        int blocks = 0;
        for (int i = P.n - 1; i >= 0; i--)
        {
            const bool large = any_bytes[i] > ANY_SHARED || any_tiles <= ANY_FEW;
            G.btiles[i] = large == (group == 0) ? any_tiles_of(i) : 0;
            shared = G.btiles[i] ? std::max(shared, any_bytes[i]) : shared;
            G.bend[i] = blocks += G.btiles[i];
        }
        if (blocks > 0)
            NB_GATHER(launch_gather_any, d, P, G, R, (unsigned)blocks, shared);
    }
    if (tiles > 0)
        NB_GATHER(launch_gather_tiles, d, level0, P, A, (unsigned)tiles);
    return NNTC_B200_OK;
}

// The fractional sites' float targets at K in d->site_tgt ([fractional site][nout], planes in order), formed when the
// device does not hold them for this K yet: read by the assembly's site pass and the mixed-precision objective.
int ensure_site_targets(nntc_b200_device* d, int k, int level0)
{
    if (d->site_tgt_kc == k || k == 0)
        return NNTC_B200_OK;
    TargetOffsets O{};
    long long ft = 0;
    for (int i = 0; i < (int)d->planes.size(); i++)
    {
        O.site0[i] = ft;
        ft += (long long)d->planes[(size_t)i].w0 * d->planes[(size_t)i].h0 * k;
    }
    O.site0[d->planes.size()] = ft;
    Planes T = planes_for(d, level0, [&](int i) {
        const DevPlane& p = d->planes[(size_t)i];
        return (size_t)p.w0 * p.h0 * (size_t)k;
    });
    T.kc = k;
    const int tblocks = (int)(T.start[T.n] / SITE_THREADS);
#define NB_TARGETS(NO)                                                                                                \
    case NO:                                                                                                          \
        k_site_targets<NO><<<tblocks, SITE_THREADS, 0, d->stream>>>(T, d->site_tgt, O);                               \
        break;
    switch (d->nout)
    {
        NB_TARGETS(3)
        NB_TARGETS(6)
        NB_TARGETS(9)
        NB_TARGETS(12)
        NB_TARGETS(15)
        NB_TARGETS(18)
    default:
        set_error(NNTC_B200_ERR_STATE, "a material holds 1..6 RGB textures");
        return NNTC_B200_ERR_STATE;
    }
#undef NB_TARGETS
    NB_LAUNCHED();
    d->site_tgt_kc = k;
    return NNTC_B200_OK;
}

// Both passes for every plane: the per-site terms, then the gather.
int assemble_split(nntc_b200_device* d, int k, int level0, const Planes& P_texels, int nmono, const double* mono,
                   int slots, bool f32)
{
    Planes S = planes_for(d, level0, [&](int i) {
        const DevPlane& p = d->planes[(size_t)i];
        return (size_t)p.w0 * p.h0;
    });
    S.kc = k;
    SiteArgs A{ d->site_terms, (float4*)d->site_y, {} };
    long long at = 0;
    for (int i = 0; i < S.n; i++)
    {
        A.site0[i] = at;
        at += (long long)d->planes[(size_t)i].w0 * d->planes[(size_t)i].h0 * (1 + k);
    }
    A.site0[S.n] = at;
    // the fractional sites' targets, formed on the first assembly at this K
    A.tgt = d->site_tgt;
    {
        long long ft = 0;
        for (int i = 0; i < S.n; i++)
        {
            A.tsite0[i] = ft;
            ft += (long long)d->planes[(size_t)i].w0 * d->planes[(size_t)i].h0 * k;
        }
        A.tsite0[S.n] = ft;
    }
    NB_TRY(ensure_site_targets(d, k, level0));
#define NB_SITES(NO)                                                                                                  \
    case NO:                                                                                                          \
        if (f32)                                                                                                      \
            launch_site_terms<NO, true>(d, S, A, level0, d->stream);                                                  \
        else                                                                                                          \
            launch_site_terms<NO, false>(d, S, A, level0, d->stream);                                                 \
        break;
    switch (d->nout)
    {
        NB_SITES(3)
        NB_SITES(6)
        NB_SITES(9)
        NB_SITES(12)
        NB_SITES(15)
        NB_SITES(18)
    default:
        set_error(NNTC_B200_ERR_STATE, "a material holds 1..6 RGB textures");
        return NNTC_B200_ERR_STATE;
    }
#undef NB_SITES
    NB_LAUNCHED();
    return f32 ? gather_planes<float>(d, level0, P_texels, nmono, mono, slots)
               : gather_planes<double>(d, level0, P_texels, nmono, mono, slots);
}

}   // namespace nb
