// gather_any.cu: the gather of the stencil assembly (blocks (b) and (c')) for planes whose visits are not tabled
// (gather.cuh): level-1 planes in tiles (k_gather_any1), and a thread per texel and slot (k_gather_walk) for the rest.
//
// Compiled once per type of the sums and channel count of the other latent (NB_TYPE, NB_NY), a module each, as gather.cu.

#include <type_traits>

#include "footprint.cuh"
#include "gather.cuh"

namespace nb
{

// Level 1 planes of any other ratio or size: the tile's texels, warps and phases of k_gather_tile1, but no two texels
// share a visit list, so each lane walks the pixels its texel can meet and tests every site. What made that walk slow
// was recomputing each site's taps (two divisions, two floors and the subtexel's turns) in every (texel, slot) thread,
// reading the samples of the sites that pass from L2, and a branch around every site, so that nothing of the next site
// started before this one's sums were done. Here the taps are separable - the column tap of pixel px and site j depends
// on the pixel row's parity alone, and the other way round - so a block forms each column's and row's once, with
// tap_at's arithmetic, next to the staged samples; and a pixel's sites are taken side by side, one that misses the texel
// entering the sums with weight, sample and term zero, whose exact zeros leave them as they were (a sum is never -0).
struct __align__(16) AxisTap
{
    int a, b;        // the two texels, clamped
    float wa, wb;    // 1 - f, f
};

// The weight with which a site's two taps land on texel (x, y): the corner weights that do, summed in corner order
// (site_touches). Away from the plane's borders no tap is clamped and at most one corner does (EDGE false).
template <bool EDGE>
__device__ __forceinline__ float corner_weight(const AxisTap& ax, const AxisTap& ay, int x, int y, bool& touches)
{
    const bool x0 = ax.a == x, x1 = ax.b == x, y0 = ay.a == y, y1 = ay.b == y;
    touches = (x0 || x1) && (y0 || y1);
    if (!EDGE)
        return (x0 ? ax.wa : ax.wb) * (y0 ? ay.wa : ay.wb);
    float w = 0.0f;
    if (x0 && y0)
        w += ax.wa * ay.wa;
    if (x1 && y0)
        w += ax.wb * ay.wa;
    if (x0 && y1)
        w += ax.wa * ay.wb;
    if (x1 && y1)
        w += ax.wb * ay.wb;
    return w;
}

// PER: sites a pixel (1 + K), or 0 to take P.kc's.
template <typename TS, int NY, int PER>
__global__ void __launch_bounds__(TILE1_THREADS, 3) k_gather_any1(Planes P, const __grid_constant__ TileArgs<TS> A,
                                                                  const __grid_constant__ AnyTiles R)
{
    constexpr int SPLIT = NY == 4 ? 8 : (NY == 3 ? 7 : (NY == 2 ? 3 : 2));
    extern __shared__ float4 sy[];
    __shared__ TS other[MAX_MONO][32];
    int tile;
    const int pl = tile_plane(A, P.n, tile);
    const PlaneView& V = P.p[pl];
    const int w = V.w, h = V.h, kc = P.kc, per = PER ? PER : 1 + kc, c = P.c1;
    const int tiles_x = (w + TILE1_W - 1) / TILE1_W;
    const int x0 = tile % tiles_x * TILE1_W, y0 = tile / tiles_x * TILE1_H;
    const int rw = R.px[pl], rh = R.py[pl], quads = (rw + 3) / 4, run = rw * per, row = quads * 4 * per;
    const int inv = (65536 + per - 1) / per;
    int first_x, first_y, unused;
    reach(x0, V.w0, w, first_x, unused);
    reach(y0, V.h0, h, first_y, unused);
    // [column][j][row parity], then [row][j][column parity]; one entry of padding after every four columns, which lanes
    // are apart, keeps a warp's reads off one bank
    AxisTap* tap_x = reinterpret_cast<AxisTap*>(sy + (size_t)row * rh);
    AxisTap* tap_y = tap_x + any_taps(rw, per);
    auto place = [&](int qx, int qy, int j) { return ((qy * per + j) * 4 + (qx & 3)) * quads + (qx >> 2); };
    auto each_site = [&](auto f) {
        for (int r = threadIdx.x; r < run; r += TILE1_THREADS)
        {
            const int qx = (r * inv) >> 16, j = r - qx * per, px = first_x + qx;
            if (px >= V.w0)
                continue;
            const size_t site = (size_t)A.site0[pl] + ((size_t)first_y * V.w0 + px) * per + j;
            const int at = place(qx, 0, j);
#pragma unroll 4
            for (int qy = 0; qy < rh; qy++)
                if (first_y + qy < V.h0)
                    f(at + qy * row, site + (size_t)qy * V.w0 * per);
        }
    };
    each_site([&](int at, size_t site) { cp_async16(sy + at, A.y + site); });
    for (int i = threadIdx.x; i < (rw + rh) * per * 2; i += TILE1_THREADS)
    {
        const bool col = i < run * 2;
        const int q = col ? i : i - run * 2, cell = q >> 1, odd = q & 1, at = (cell * inv) >> 16, j = cell - at * per;
        const int px = col ? first_x + at : odd, py = col ? odd : first_y + at;
        float dx, dy;
        site_offset(kc, j, px, py, dx, dy);
        const Tap t = tap_at(px, py, dx, dy, V.w0, V.h0, w, h);
        (col ? tap_x : tap_y)[q + (at >> 2)] =
            col ? AxisTap{ t.x0, t.x1, 1.0f - t.fx, t.fx } : AxisTap{ t.y0, t.y1, 1.0f - t.fy, t.fy };
    }
    cp_async_wait_all();
    __syncthreads();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tx = x0 + (lane & (TILE1_W - 1)), ty = y0 + lane / TILE1_W;
    const bool active = tx < w && ty < h;
    const bool edge = __any_sync(0xffffffffu, active && (tx == 0 || ty == 0 || tx == w - 1 || ty == h - 1));
    const size_t T = (size_t)w * h, sp = active ? stencil_pos(tx, ty, w, h) : 0;
    // every site of the pixels that can meet both (tx, ty) and the slot's neighbour, in site order: f(j, place, whether
    // it touches both, w_self, w_other) for the sites of a pixel, then g() for the pixel
    auto pixels = [&](auto edges, int slot, auto f, auto g) {
        constexpr bool EDGE = decltype(edges)::value;
        int ox, oy;
        slot_offset(slot, ox, oy);
        const int nbx = tx + ox, nby = ty + oy;
        int px_lo, px_hi, py_lo, py_hi, qx_lo, qx_hi, qy_lo, qy_hi;
        reach(tx, V.w0, w, px_lo, px_hi);
        reach(ty, V.h0, h, py_lo, py_hi);
        reach(nbx, V.w0, w, qx_lo, qx_hi);
        reach(nby, V.h0, h, qy_lo, qy_hi);
        px_lo = max(px_lo, qx_lo);
        px_hi = min(px_hi, qx_hi);
        py_lo = max(py_lo, qy_lo);
        py_hi = min(py_hi, qy_hi);
        for (int py = py_lo; py <= py_hi; py++)
            for (int px = px_lo; px <= px_hi; px++)
            {
                const int qx = px - first_x, qy = py - first_y;
                const AxisTap* cols = tap_x + qx * per * 2 + (qx >> 2) + (py & 1);
                const AxisTap* rows = tap_y + qy * per * 2 + (qy >> 2) + (px & 1);
                const int at = place(qx, qy, 0);
#pragma unroll
                for (int j = 0; j < (PER ? PER : MAX_SITES); j++)
                {
                    if (!PER && j >= per)
                        break;
                    const AxisTap ax = cols[2 * j], ay = rows[2 * j];
                    bool self, both = true;
                    const float ws = corner_weight<EDGE>(ax, ay, tx, ty, self);
                    const float wo = slot ? corner_weight<EDGE>(ax, ay, nbx, nby, both) : ws;
                    f(j, at + j * 4 * quads, self && both, ws, wo);
                }
                g();
            }
    };
    TS sums[MAX_MONO];
#pragma unroll
    for (int i = 0; i < MAX_MONO; i++)
        sums[i] = (TS)0;
    auto sum_slot = [&](auto lo, auto hi, int slot) {
        constexpr int LO = decltype(lo)::value, HI = decltype(hi)::value;
        float4 y[MAX_SITES];
        TS scale[MAX_SITES];
        auto site = [&](int j, int at, bool hit, float ws, float wo) {
            const float4 v = sy[at];
            y[j] = hit ? v : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            scale[j] = hit ? (TS)ws * (TS)wo : (TS)0;
        };
        auto pixel = [&]() {
#pragma unroll
            for (int j = 0; j < (PER ? PER : MAX_SITES); j++)
                if (PER || j < per)
                    visit_sums<TS, NY, LO, HI>(sums, y[j], scale[j]);
        };
        if (edge)
            pixels(std::true_type{}, slot, site, pixel);
        else
            pixels(std::false_type{}, slot, site, pixel);
    };
    using Lo = std::integral_constant<int, 0>;
    using Mid = std::integral_constant<int, SPLIT>;
    using Hi = std::integral_constant<int, MAX_MONO>;
    if (active && warp == 0)
        sum_slot(Lo{}, Mid{}, 0);
    else if (active && warp == 4)
    {
        sum_slot(Mid{}, Hi{}, 0);
#pragma unroll
        for (int L = SPLIT; L < MAX_MONO; L++)
            if (mono_used(L, NY))
                other[L][lane] = sums[L];
    }
    else if (active)
    {
        const int s0 = warp == 1 ? 1 : (warp == 2 ? 3 : 2), s1 = warp == 3 ? 4 : s0;
#pragma unroll 1
        for (int slot = s0; slot <= s1 && slot < A.slots; slot += 2)
        {
            int ox, oy;
            slot_offset(slot, ox, oy);
            if (tx + ox < 0 || tx + ox >= w || ty + oy >= h)
            {
                store_zero_block<TS>(A, V, slot, c, tx, ty, T, sp);
                continue;
            }
#pragma unroll
            for (int i = 0; i < MAX_MONO; i++)
                sums[i] = (TS)0;
            sum_slot(Lo{}, Hi{}, slot);
            expand_block<TS, NY>(A, V, sums, slot, c, tx, ty, T, sp);
        }
    }
    __syncthreads();
    constexpr int CH = sizeof(TS) == sizeof(float) ? 4 : 2;
    for (int p = 0; p * CH < c; p++)
    {
        const int first = p * CH;
        stage_terms<TS>(A, sy, first, c, each_site);
        if (p == 0 && warp == 0 && active)
        {
#pragma unroll
            for (int L = SPLIT; L < MAX_MONO; L++)
                if (mono_used(L, NY))
                    sums[L] = other[L][lane];
            expand_block<TS, NY>(A, V, sums, 0, c, tx, ty, T, sp);
        }
        cp_async_wait_all();
        __syncthreads();
        const int ch = 2 * (warp - 1);
        if (active && ch >= first && ch < first + CH && ch < c)
        {
            using T2 = typename std::conditional<sizeof(TS) == sizeof(float), float2, double2>::type;
            double g0 = 0.0, g1 = 0.0;
            T2 t[MAX_SITES];
            float weight[MAX_SITES];
            auto site = [&](int j, int at, bool hit, float ws, float) {
                const T2 v = *reinterpret_cast<const T2*>(reinterpret_cast<const TS*>(sy + at) + (ch - first));
                t[j].x = hit ? v.x : 0;
                t[j].y = hit ? v.y : 0;
                weight[j] = hit ? ws : 0.0f;
            };
            auto pixel = [&]() {
#pragma unroll
                for (int j = 0; j < (PER ? PER : MAX_SITES); j++)
                    if (PER || j < per)
                    {
                        g0 += (double)weight[j] * (double)t[j].x;
                        g1 += (double)weight[j] * (double)t[j].y;
                    }
            };
            if (edge)
                pixels(std::true_type{}, 0, site, pixel);
            else
                pixels(std::false_type{}, 0, site, pixel);
            double* out = V.grad + ((size_t)ty * w + tx) * c + ch;
            out[0] = g0;
            if (ch + 1 < c)
                out[1] = g1;
        }
        __syncthreads();
    }
}

// The texel at position `pos` of the stencil's colour-major order (the inverse of stencil_pos).
__device__ __forceinline__ void stencil_texel(long long pos, int w, int h, int& x, int& y)
{
    const long long w0c = (w + 1) >> 1, w1c = w >> 1, h0c = (h + 1) >> 1, h1c = h >> 1;
    const long long n0 = w0c * h0c, n1 = w1c * h0c, n2 = w0c * h1c;
    int cx = 0, cy = 0;
    long long r = pos, rw = w0c;
    if (r >= n0 + n1 + n2)
    {
        r -= n0 + n1 + n2;
        cx = 1;
        cy = 1;
        rw = w1c;
    }
    else if (r >= n0 + n1)
    {
        r -= n0 + n1;
        cy = 1;
    }
    else if (r >= n0)
    {
        r -= n0;
        cx = 1;
        rw = w1c;
    }
    x = 2 * (int)(r % rw) + cx;
    y = 2 * (int)(r / rw) + cy;
}

// The gather of the planes no tile takes (planes one texel wide or high at level 0, level-1 planes whose tile would not
// fit shared memory or that are above any_tiles_line): one thread per (texel, slot) tests every site of the two texels' common
// footprint, in site order; the self-slot thread also gathers the gradient. Blocks run in (region, colour, slot) order,
// the slot fastest, so that the five slots of one run of texels and the four colours of one region run side by side
// and share the region's sites in L2.
template <bool LEVEL0, typename TS, int NY>
__global__ void __launch_bounds__(WALK_THREADS) k_gather_walk(Planes P, const __grid_constant__ TileArgs<TS> A,
                                                               const __grid_constant__ WalkBlocks B)
{
    using TT = TS;   // the terms' type
    int pl = 0;
    while (pl + 1 < P.n && B.start[pl + 1] <= (long long)blockIdx.x)
        pl++;
    const long long lb = (long long)blockIdx.x - B.start[pl];
    const int slot = (int)(lb % A.slots);
    const int colour = (int)((lb / A.slots) % 4);
    const long long region = lb / A.slots / 4;
    const PlaneView& V = P.p[pl];
    const int tw_ = V.w, th_ = V.h;
    const long long w0c = (tw_ + 1) >> 1, w1c = tw_ >> 1, h0c = (th_ + 1) >> 1, h1c = th_ >> 1;
    const long long n0 = w0c * h0c, n1 = w1c * h0c, n2 = w0c * h1c, n3 = w1c * h1c;
    const long long ncol = colour == 0 ? n0 : (colour == 1 ? n1 : (colour == 2 ? n2 : n3));
    const long long within = region * WALK_THREADS + threadIdx.x;
    if (within >= ncol)
        return;
    // the texel's place in the stencil's colour-major order
    const long long sp = within + (colour == 0 ? 0 : (colour == 1 ? n0 : (colour == 2 ? n0 + n1 : n0 + n1 + n2)));
    const int kc = P.kc, per = 1 + kc;
    const int c = LEVEL0 ? P.c0 : P.c1;
    int tx, ty;
    stencil_texel(sp, tw_, th_, tx, ty);
    int ox, oy;
    slot_offset(slot, ox, oy);
    const int nbx = tx + ox, nby = ty + oy;
    const size_t T = (size_t)tw_ * th_;
    if (nbx < 0 || nbx >= tw_ || nby >= th_)
    {
        store_zero_block<TS>(A, V, slot, c, tx, ty, T, (size_t)sp);
        return;
    }
    TS sums[MAX_MONO];
#pragma unroll
    for (int i = 0; i < MAX_MONO; i++)
        sums[i] = (TS)0;
    double g[MAX_CH];
#pragma unroll
    for (int a = 0; a < MAX_CH; a++)
        g[a] = 0.0;
    const TT* terms = (const TT*)A.terms + (size_t)A.site0[pl] * c;
    const float4* ys = A.y + A.site0[pl];
    // the pixel range of sites that can touch both texels: the intersection of their footprints
    int px_lo, px_hi, py_lo, py_hi, qx_lo, qx_hi, qy_lo, qy_hi;
    reach(tx, V.w0, tw_, px_lo, px_hi);
    reach(ty, V.h0, th_, py_lo, py_hi);
    reach(nbx, V.w0, tw_, qx_lo, qx_hi);
    reach(nby, V.h0, th_, qy_lo, qy_hi);
    px_lo = max(px_lo, qx_lo);
    px_hi = min(px_hi, qx_hi);
    py_lo = max(py_lo, qy_lo);
    py_hi = min(py_hi, qy_hi);
    for (int py = py_lo; py <= py_hi; py++)
        for (int px = px_lo; px <= px_hi; px++)
            for (int j = 0; j <= kc; j++)
            {
                float ws, wo;
                if (!site_touches<LEVEL0>(px, py, j, kc, tx, ty, nbx, nby, V.w0, V.h0, tw_, th_, ws, wo))
                    continue;
                const size_t site = ((size_t)py * V.w0 + px) * per + j;
                if (slot == 0)
                {
#pragma unroll
                    for (int a = 0; a < MAX_CH; a++)
                        if (a < c)
                            g[a] += (double)ws * (double)__ldg(terms + site * c + a);
                }
                visit_sums<TS, NY, 0, MAX_MONO>(sums, __ldg(ys + site), (TS)ws * (TS)wo);
            }
    expand_block<TS, NY>(A, V, sums, slot, c, tx, ty, T, (size_t)sp);
    if (slot == 0)
    {
#pragma unroll
        for (int a = 0; a < MAX_CH; a++)
            if (a < c)
                V.grad[((size_t)ty * tw_ + tx) * c + a] = g[a];
    }
}

template <typename TS, int NY>
int launch_gather_any(nntc_b200_device* d, const Planes& P, const TileArgs<TS>& A, const AnyTiles& S, unsigned grid,
                      size_t shared)
{
    void (*kernel)(Planes, const TileArgs<TS>, const AnyTiles) = P.kc == 4 ? k_gather_any1<TS, NY, 5> : k_gather_any1<TS, NY, 0>;
    NB_SHARED_LIMIT(kernel, ANY_SHARED_MAX);
    kernel<<<grid, TILE1_THREADS, shared, d->stream>>>(P, A, S);
    NB_LAUNCHED();
    return NNTC_B200_OK;
}

template <typename TS, int NY>
int launch_gather_walk(nntc_b200_device* d, int level0, const Planes& P, const TileArgs<TS>& A, const WalkBlocks& B)
{
    const unsigned grid = (unsigned)B.start[P.n];
    if (level0)
        k_gather_walk<true, TS, NY><<<grid, WALK_THREADS, 0, d->stream>>>(P, A, B);
    else
        k_gather_walk<false, TS, NY><<<grid, WALK_THREADS, 0, d->stream>>>(P, A, B);
    NB_LAUNCHED();
    return NNTC_B200_OK;
}

template int launch_gather_any<NB_TYPE, NB_NY>(nntc_b200_device*, const Planes&, const TileArgs<NB_TYPE>&, const AnyTiles&,
                                               unsigned, size_t);
template int launch_gather_walk<NB_TYPE, NB_NY>(nntc_b200_device*, int, const Planes&, const TileArgs<NB_TYPE>&,
                                                const WalkBlocks&);

}   // namespace nb
