// gather.cu: the tiled gather of the stencil assembly (blocks (b) and (c')), for planes whose visits are tabled.
//
// A block takes a tile of texels and stages the other latent's sample at every site the tile's texels meet (k_site_terms
// left them in global memory) in shared memory once; then each lane owns one texel and walks its class's visit list, one
// owned slot after another, adding every visit's monomials to the slot's sums in the reference's site order and
// expanding them into the slot's block. Every sum receives the same terms in the same order as the reference's
// per-texel gather, so the blocks are the same bits (FP64); the FP32 instantiation is the adjoint form's.
//
// Why this shape: one thread per (texel, slot) reading its private run of sites from L2 was bound by the latency and
// the sector traffic of those reads (a site is read by up to ten (texel, slot) threads, 16 of every 32 bytes used) at
// about half of the issue slots; a staged site is read from L2 once per tile, the visits' entries are one broadcast
// load, and the arithmetic (FP64: 41 visits x 40 operations + the expansions at level 0, 800 visits x 40 at level 1)
// is what is left. The smallest planes run first: their few blocks walk as long as any other's, and at the end of the
// launch nothing would run beside them.
//
// Compiled once per type of the sums and channel count of the other latent (NB_TYPE, NB_NY), a module each: a launch loads
// the kernels of its own counts alone (site_terms.cu).

#include <type_traits>

#include "gather.cuh"

namespace nb
{

constexpr int TILE0_THREADS = 256;   // a warp per texel row and x parity

template <typename TS>
__device__ __forceinline__ TS visit_scale(const int4& e);
template <>
__device__ __forceinline__ double visit_scale<double>(const int4& e)
{
    return __hiloint2double(e.w, e.z);
}
template <>
__device__ __forceinline__ float visit_scale<float>(const int4& e)
{
    return __int_as_float(e.z);
}

// The sums of one slot: every visit of the list, in order, GROUP samples loaded ahead of their additions and the next
// GROUP entries on their way meanwhile.
template <typename TS, int NY, int LO, int HI>
__device__ __forceinline__ void walk(const TileArgs<TS>& A, const float4* lane_sites, int e0, int e1,
                                     TS (&sums)[MAX_MONO])
{
    const char* sites = reinterpret_cast<const char*>(lane_sites);
    constexpr int GROUP = 4;
    int e = e0;
    int4 en[GROUP];
    if (e + GROUP <= e1)
    {
#pragma unroll
        for (int g = 0; g < GROUP; g++)
            en[g] = __ldg(A.tab + e + g);
    }
    for (; e + GROUP <= e1; e += GROUP)
    {
        float4 y[GROUP];
        TS scale[GROUP];
#pragma unroll
        for (int g = 0; g < GROUP; g++)
        {
            y[g] = *reinterpret_cast<const float4*>(sites + visit_place<TS>(en[g]));
            scale[g] = visit_scale<TS>(en[g]);
        }
        if (e + 2 * GROUP <= e1)
        {
#pragma unroll
            for (int g = 0; g < GROUP; g++)
                en[g] = __ldg(A.tab + e + GROUP + g);
        }
#pragma unroll
        for (int g = 0; g < GROUP; g++)
            visit_sums<TS, NY, LO, HI>(sums, y[g], scale[g]);
    }
    for (; e < e1; e++)
    {
        const int4 en = __ldg(A.tab + e);
        visit_sums<TS, NY, LO, HI>(sums, *reinterpret_cast<const float4*>(sites + visit_place<TS>(en)),
                                   visit_scale<TS>(en));
    }
}

// Level 0's gradient: the self slot's visits, each site's term weighted (in double in both forms), straight from global
// memory - a dozen and a half reads per texel, made while the samples of the tile are on their way.
template <typename TS>
__device__ __forceinline__ void gather_gradient0(const TileArgs<TS>& A, const PlaneView& V, int pl, int cls, int tx,
                                                 int ty, int w, int per, int c)
{
    const size_t site = A.site0[pl] + ((size_t)ty * w + tx) * per;
    double g[MAX_CH] = { 0.0, 0.0, 0.0, 0.0 };
    const int e1 = A.off[cls][1];
#pragma unroll 4
    for (int e = A.off[cls][0]; e < e1; e++)
    {
        const int4 en = __ldg(A.tab + e);
        const int dx = ((en.x >> 16) & 15) - 2, dy = ((en.x >> 20) & 15) - 2, j = en.x >> 24;
        const size_t s = (site + (ptrdiff_t)((dy * w + dx) * per + j)) * c;
        const double ws = (double)__int_as_float(en.y);
        if constexpr (sizeof(TS) == sizeof(float))
        {
            const float* t = (const float*)A.terms + s;
            if (c == MAX_CH)
            {
                const float4 t4 = __ldg((const float4*)t);
                g[0] += ws * (double)t4.x;
                g[1] += ws * (double)t4.y;
                g[2] += ws * (double)t4.z;
                g[3] += ws * (double)t4.w;
            }
            else
            {
#pragma unroll
                for (int a = 0; a < MAX_CH; a++)
                    if (a < c)
                        g[a] += ws * (double)__ldg(t + a);
            }
        }
        else
        {
            const double* t = (const double*)A.terms + s;
            if (c == MAX_CH)
            {
                const double2 t0 = __ldg((const double2*)t), t1 = __ldg((const double2*)t + 1);
                g[0] += ws * t0.x;
                g[1] += ws * t0.y;
                g[2] += ws * t1.x;
                g[3] += ws * t1.y;
            }
            else
            {
#pragma unroll
                for (int a = 0; a < MAX_CH; a++)
                    if (a < c)
                        g[a] += ws * __ldg(t + a);
            }
        }
    }
    double* out = V.grad + ((size_t)ty * w + tx) * c;
    if (c == MAX_CH)
    {
        reinterpret_cast<double2*>(out)[0] = make_double2(g[0], g[1]);
        reinterpret_cast<double2*>(out)[1] = make_double2(g[2], g[3]);
    }
    else
    {
#pragma unroll
        for (int a = 0; a < MAX_CH; a++)
            if (a < c)
                out[a] = g[a];
    }
}

// Level 0: a tile of 64 x 4 texels, a warp per (row, x parity): its 32 lanes share a class but at the borders.
template <typename TS, int NY>
__global__ void __launch_bounds__(TILE0_THREADS, (sizeof(TS) == sizeof(float) ? 4 : 2))
    k_gather_tile0(Planes P, const __grid_constant__ TileArgs<TS> A)
{
    extern __shared__ float4 sy[];
    int tile;
    const int pl = tile_plane(A, P.n, tile);
    const PlaneView& V = P.p[pl];
    const int w = V.w, h = V.h, per = 1 + P.kc, c = P.c0;
    const int tiles_x = (w + TILE0_W - 1) / TILE0_W;
    const int x0 = tile % tiles_x * TILE0_W, y0 = tile / tiles_x * TILE0_H;
    {
        const int run = TILE0_PX * per, inv = (65536 + per - 1) / per;   // r / per = (r inv) >> 16, r < 2^10
        for (int r = threadIdx.x; r < run; r += TILE0_THREADS)
        {
            const int qx = (r * inv) >> 16, j = r - qx * per, px = x0 - 1 + qx;
            if (px < 0 || px >= w)
                continue;
            const float4* from = A.y + A.site0[pl] + ((ptrdiff_t)(y0 - 1) * w + px) * per + j;
            float4* to = sy + tile_site<true>(qx, 0, j, per);
#pragma unroll
            for (int qy = 0; qy < TILE0_PY; qy++)
                if (y0 - 1 + qy >= 0 && y0 - 1 + qy < h)
                    cp_async16(to + qy * run, from + (ptrdiff_t)qy * w * per);
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cx = warp & 1, ry = warp >> 1;
    const int tx = x0 + 2 * lane + cx, ty = y0 + ry;
    const bool active = tx < w && ty < h;
    const int cls = active ? axis_class<true>(ty, h) * AXIS_CLASSES0 + axis_class<true>(tx, w) : 0;
    if (active)
        gather_gradient0(A, V, pl, cls, tx, ty, w, per, c);
    cp_async_wait_all();
    __syncthreads();
    if (!active)
        return;
    const size_t T = (size_t)w * h, sp = stencil_pos(tx, ty, w, h);
    const int base = tile_site<true>(0, ry, 0, per) + lane;
#pragma unroll 1
    for (int slot = 0; slot < A.slots; slot++)
    {
        int ox, oy;
        slot_offset(slot, ox, oy);
        if (tx + ox < 0 || tx + ox >= w || ty + oy >= h)
        {
            store_zero_block<TS>(A, V, slot, c, tx, ty, T, sp);
            continue;
        }
        TS sums[MAX_MONO];
#pragma unroll
        for (int i = 0; i < MAX_MONO; i++)
            sums[i] = (TS)0;
        walk<TS, NY, 0, MAX_MONO>(A, sy + base, A.off[cls][slot], A.off[cls][slot + 1], sums);
        expand_block<TS, NY>(A, V, sums, slot, c, tx, ty, T, sp);
    }
}

// Level 1: a tile of 8 x 4 texels, one per lane, and five warps of equal work: the self slot's visits (320 inside a
// plane) are walked by two warps, each summing half of the monomials, the right and the down slot's (160 each) by one
// warp each, the two diagonal slots' (80 each) by one. The gradient's terms, as many bytes again as the samples or
// twice that, then take the samples' place in shared memory, two channels (FP64) or all (FP32) at a time, and a warp
// sums two channels. (Reading the terms straight from global memory beside the visits, as level 0 does, cost 2.5 times
// the whole kernel: 320 reads a texel do not stay in what the tile leaves of L1.)
template <typename TS, int NY>
__global__ void __launch_bounds__(TILE1_THREADS, 3) k_gather_tile1(Planes P, const __grid_constant__ TileArgs<TS> A)
{
    // the monomials [0, SPLIT) to the self slot's first warp, the rest to its second
    constexpr int SPLIT = NY == 4 ? 8 : (NY == 3 ? 7 : (NY == 2 ? 3 : 2));
    extern __shared__ float4 sy[];
    __shared__ TS other[MAX_MONO][32];
    int tile;
    const int pl = tile_plane(A, P.n, tile);
    const PlaneView& V = P.p[pl];
    const int w = V.w, h = V.h, per = 1 + P.kc, c = P.c1;
    const int tiles_x = (w + TILE1_W - 1) / TILE1_W;
    const int x0 = tile % tiles_x * TILE1_W, y0 = tile / tiles_x * TILE1_H;
    const int run = TILE1_PX * per, inv = (65536 + per - 1) / per, first_x = 4 * x0 - 2, first_y = 4 * y0 - 2;
    // every site of the tile that the plane has, in f(place in the tile, site)
    auto each_site = [&](auto f) {
        for (int r = threadIdx.x; r < run; r += TILE1_THREADS)
        {
            const int qx = (r * inv) >> 16, j = r - qx * per, px = first_x + qx;
            if (px < 0 || px >= V.w0)
                continue;
            const ptrdiff_t site = (ptrdiff_t)A.site0[pl] + ((ptrdiff_t)first_y * V.w0 + px) * per + j;
            const int at = tile_site<false>(qx, 0, j, per);
#pragma unroll 4
            for (int qy = 0; qy < TILE1_PY; qy++)
                if (first_y + qy >= 0 && first_y + qy < V.h0)
                    f(at + qy * run, (size_t)(site + (ptrdiff_t)qy * V.w0 * per));
        }
    };
    each_site([&](int at, size_t site) { cp_async16(sy + at, A.y + site); });
    cp_async_wait_all();
    __syncthreads();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lx = lane & (TILE1_W - 1), ly = lane / TILE1_W;
    const int tx = x0 + lx, ty = y0 + ly;
    const bool active = tx < w && ty < h;
    const size_t T = (size_t)w * h, sp = active ? stencil_pos(tx, ty, w, h) : 0;
    const int cls = active ? axis_class<false>(ty, h) * AXIS_CLASSES1 + axis_class<false>(tx, w) : 0;
    const int base = tile_site<false>(0, 4 * ly, 0, per) + lx;
    TS sums[MAX_MONO];
#pragma unroll
    for (int i = 0; i < MAX_MONO; i++)
        sums[i] = (TS)0;
    if (active && warp == 0)
        walk<TS, NY, 0, SPLIT>(A, sy + base, A.off[cls][0], A.off[cls][1], sums);
    else if (active && warp == 4)
    {
        walk<TS, NY, SPLIT, MAX_MONO>(A, sy + base, A.off[cls][0], A.off[cls][1], sums);
#pragma unroll
        for (int L = SPLIT; L < MAX_MONO; L++)
            if (mono_used(L, NY))
                other[L][lane] = sums[L];
    }
    else if (active)
    {
        // the owned neighbours: warp 1 right, warp 2 down, warp 3 down-left then down-right
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
            walk<TS, NY, 0, MAX_MONO>(A, sy + base, A.off[cls][slot], A.off[cls][slot + 1], sums);
            expand_block<TS, NY>(A, V, sums, slot, c, tx, ty, T, sp);
        }
    }
    __syncthreads();   // the samples are spent; the second half of the self sums is in `other`

    // the gradient, in double in both forms: round p stages channels CH p .. CH p + CH - 1
    constexpr int CH = sizeof(TS) == sizeof(float) ? 4 : 2;
    const int e0 = A.off[cls][0], e1 = A.off[cls][1];
    for (int p = 0; p * CH < c; p++)
    {
        const int first = p * CH;
        stage_terms<TS>(A, sy, first, c, each_site);
        if (p == 0 && warp == 0 && active)
        {
            // the self slot's block, while the terms arrive
#pragma unroll
            for (int L = SPLIT; L < MAX_MONO; L++)
                if (mono_used(L, NY))
                    sums[L] = other[L][lane];
            expand_block<TS, NY>(A, V, sums, 0, c, tx, ty, T, sp);
        }
        cp_async_wait_all();
        __syncthreads();
        // a warp sums two channels (FP32: warps 1 and 2; FP64, round p: warp 1 + p), so that a visit's entry and weight
        // are read once for both
        const int pair = warp - 1, ch = 2 * pair;
        if (active && pair >= 0 && ch >= first && ch < first + CH && ch < c)
        {
            using TT = typename std::conditional<sizeof(TS) == sizeof(float), float, double>::type;
            using T2 = typename std::conditional<sizeof(TS) == sizeof(float), float2, double2>::type;
            const char* st = reinterpret_cast<const char*>(reinterpret_cast<const TT*>(sy + base) + (ch - first));
            double g0 = 0.0, g1 = 0.0;
#pragma unroll 8
            for (int e = e0; e < e1; e++)
            {
                const int2 en = __ldg(reinterpret_cast<const int2*>(A.tab + e));
                const T2 t = *reinterpret_cast<const T2*>(st + (en.x & 0xffff));
                const double ws = (double)__int_as_float(en.y);
                g0 += ws * (double)t.x;
                g1 += ws * (double)t.y;
            }
            double* out = V.grad + ((size_t)ty * w + tx) * c + ch;
            out[0] = g0;
            if (ch + 1 < c)
                out[1] = g1;
        }
        __syncthreads();
    }
}

template <typename TS, int NY>
int launch_gather_tiles(nntc_b200_device* d, int level0, const Planes& P, const TileArgs<TS>& A, unsigned grid)
{
    const int per = 1 + P.kc;
    const int site = (level0 ? TILE0_PX * TILE0_PY : TILE1_PX * TILE1_PY) * (int)sizeof(float4), shared = site * per;
    void (*kernel)(Planes, const TileArgs<TS>) = level0 ? k_gather_tile0<TS, NY> : k_gather_tile1<TS, NY>;
    NB_SHARED_LIMIT(kernel, site * MAX_SITES);
    kernel<<<grid, level0 ? TILE0_THREADS : TILE1_THREADS, shared, d->stream>>>(P, A);
    NB_LAUNCHED();
    return NNTC_B200_OK;
}

template int launch_gather_tiles<NB_TYPE, NB_NY>(nntc_b200_device*, int, const Planes&, const TileArgs<NB_TYPE>&, unsigned);

}   // namespace nb
