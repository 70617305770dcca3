// gather.cuh: what the two gathers of the stencil assembly share - the tiled gather of gather.cu (planes whose visits
// are tabled) and those of gather_any.cu (any other plane) - the monomial layout, the visit tables, the launch
// arguments and the expansion of a slot's sums into its stored block.
#pragma once

#include "device.cuh"

namespace nb
{

// The ten products y_i y_k (i <= k < 4) of the monomial layout, row by row: (0,0) (0,1) (0,2) (0,3) (1,1) (1,2)
// (1,3) (2,2) (2,3) (3,3). Functions rather than tables, so an unrolled index folds to a register name.
__host__ __device__ constexpr int pair_i(int p)
{
    return p < 4 ? 0 : (p < 7 ? 1 : (p < 9 ? 2 : 3));
}
__host__ __device__ constexpr int pair_k(int p)
{
    return p < 4 ? p : (p < 7 ? p - 3 : (p < 9 ? p - 5 : 3));
}

// Whether slot L of the fixed monomial layout (the constant, four linear terms, ten products) is a monomial of a
// latent with ny channels: the used slots, in slot order, are the reference's monomials in its order.
__host__ __device__ constexpr bool mono_used(int L, int ny)
{
    return L == 0 || (L <= MAX_CH ? L - 1 < ny : pair_k(L - 5) < ny);
}

// ---- the visit tables
//
// Which sites touch a texel and one of its neighbours, and with what weights, depends only on where the texel sits
// relative to the pixel grid and the plane's borders: for level 0 (the unknown at the pixels' own resolution, site
// positions px + dx exact in float) on the texel's parity, which decides the subtexel rotation of its pixels, and on
// whether it is a border texel; for level 1 at exactly a quarter of a power-of-two plane (site positions ((px + 0.5 +
// dx) w) / w0 - 0.5 exact in float) on whether it is a border texel alone. So the visits of every class are listed
// once, in the reference's site order, by running site_touches on a texel of that class; every texel of such a plane
// walks its list instead of testing every site of its footprint. A class is a pair of per-axis classes: level 1's are
// first / inner / last texel, level 0's first (even) / inner even / inner odd / last even / last odd. A plane one
// texel wide or high, whose one texel would be both first and last, is not tabled; level-1 planes that are not go to
// k_gather_any1 where its tiles fit and are the faster, the rest, and level 0's, to k_gather_walk.

constexpr int AXIS_CLASSES0 = 5, AXIS_CLASSES1 = 3;
constexpr int GATHER_CLASSES = AXIS_CLASSES0 * AXIS_CLASSES0;

template <bool LEVEL0>
__host__ __device__ __forceinline__ int axis_class(int t, int n)
{
    if (LEVEL0)
        return t == 0 ? 0 : ((t == n - 1 ? 3 : 1) + (t & 1));
    return t == 0 ? 0 : (t == n - 1 ? 2 : 1);
}

// The tiles of the tiled gather. Level 0: TILE0_W x TILE0_H texels, one pixel of margin; level 1: TILE1_W x TILE1_H
// texels, four pixels each and two of margin. A tile's sites are held row by row, the sites j of a pixel row apart, the
// pixels of one (row, j) split by their place relative to the lanes (two apart at level 0, four at level 1) so that the
// lanes of a warp, whose texels are that far apart, read consecutive 16-byte samples.
constexpr int TILE0_W = 64, TILE0_H = 4, TILE0_PX = TILE0_W + 2, TILE0_PY = TILE0_H + 2;
constexpr int TILE1_THREADS = 160;   // five warps: see k_gather_tile1
constexpr int TILE1_W = 8, TILE1_H = 4, TILE1_PX = 4 * TILE1_W + 4, TILE1_PY = 4 * TILE1_H + 4;

// Where site j of the tile's pixel (qx, qy) (from the margin's first pixel) sits in the tile.
template <bool LEVEL0>
__host__ __device__ __forceinline__ int tile_site(int qx, int qy, int j, int per)
{
    return LEVEL0 ? ((qy * per + j) * 2 + (qx & 1)) * (TILE0_PX / 2) + (qx >> 1)
                  : ((qy * per + j) * 4 + (qx & 3)) * (TILE1_PX / 4) + (qx >> 2);
}

// A visit: x the site's place in the tile from the lane's own, in bytes (bits 0..15) and its pixel and j relative to
// the texel's first pixel, (dpx + 2) << 16 | (dpy + 2) << 20 | j << 24; y w_self (float bits); z, w the product w_self
// w_other in double for the FP64 sums, or the FP32 product's bits in z and the place alone in w.
template <typename TS>
__device__ __forceinline__ int visit_place(const int4& e)
{
    return sizeof(TS) == sizeof(float) ? e.w : e.x & 0xffff;
}

template <typename TS>
struct TileArgs
{
    const void* terms;    // [site][c]: the gradient terms, doubles (FP64) or floats (FP32)
    const float4* y;      // [site]: the site's sample of the other latent
    const int4* tab;      // the visits, by class and slot
    // the monomial matrices (c x c, row-major) at their monomial's slot of the fixed layout, unused slots left out:
    // with the expansion unrolled every entry is a constant-bank operand, no loads
    TS mono[MAX_MONO][MAX_CH * MAX_CH];
    int off[GATHER_CLASSES][SLOTS + 1];
    long long site0[MAX_PLANES + 1];
    int bend[MAX_PLANES];   // one past each plane's last block, the planes in descending order (the smallest first)
    int btiles[MAX_PLANES]; // each plane's blocks (0: not of this launch)
    int slots;              // slots gathered: SLOTS, or 1 for the diagonal blocks and the gradient alone
    int bc_copy;            // level 0, FP64, for the BC refinement: each block also into the block-major copy
    int plain;              // every monomial matrix is symmetric bit for bit and finite
};

// Where coefficient e of slot `slot` of texel (x, y) sits in the block-major copy: block (y / 4, x / 4) of a plane
// bx blocks wide, then slot, coefficient and the texel's place in its 4x4 block.
__device__ __forceinline__ size_t bc_sten_pos(int x, int y, int bx, int slot, int cc, int e)
{
    const size_t blk = (size_t)(y >> 2) * bx + (x >> 2);
    return ((blk * SLOTS + slot) * cc + e) * 16 + (size_t)((y & 3) * 4 + (x & 3));
}

// Row and column of entry u of a C x C block: row by row, or the upper triangle's row by row (closed forms, so that an
// unrolled index folds to a constant).
__host__ __device__ constexpr int entry_row(int C, bool sym, int u)
{
    return !sym ? u / C : (u < C ? 0 : (u < 2 * C - 1 ? 1 : (u < 3 * C - 3 ? 2 : 3)));
}
__host__ __device__ constexpr int entry_col(int C, bool sym, int u)
{
    return !sym ? u % C
                : u - (entry_row(C, true, u) * C - entry_row(C, true, u) * (entry_row(C, true, u) - 1) / 2) +
                      entry_row(C, true, u);
}

// The slot's block from its sums, expanded against the monomial matrices in monomial order (src/solve_level1.cu:
// 382-399), and stored. SYM: the matrices are symmetric bit for bit (the outputs' weights all powers of two, the
// default) and finite. A symmetric block's upper triangle alone is expanded; and a monomial whose sum is zero, which
// the reference skips, may add its exact zeros, the same bits. Any other decoder takes the reference's steps.
template <typename TS, int NY, int C, bool SYM>
__device__ __forceinline__ void expand_store(const TileArgs<TS>& A, const PlaneView& V, const TS (&sums)[MAX_MONO],
                                             int slot, int tx, int ty, size_t T, size_t sp)
{
    constexpr int CC = C * C;
    constexpr int NE = SYM ? C * (C + 1) / 2 : CC;
    constexpr int PART = NE > 10 ? 8 : NE;
    const bool bc_copy = sizeof(TS) == sizeof(double) && A.bc_copy;
    TS keep[sizeof(TS) == sizeof(float) ? NE : 1];
#pragma unroll
    for (int p = 0; p < (NE + PART - 1) / PART; p++)
    {
        TS blk[PART];
#pragma unroll
        for (int q = 0; q < PART; q++)
            blk[q] = (TS)0;
#pragma unroll
        for (int L = 0; L < MAX_MONO; L++)
        {
            if (!mono_used(L, NY))
                continue;
            const TS s = sums[L];
            if (!SYM && s == (TS)0)
                continue;
#pragma unroll
            for (int q = 0; q < PART; q++)
                if (p * PART + q < NE)
                    blk[q] += s * A.mono[L][entry_row(C, SYM, p * PART + q) * C + entry_col(C, SYM, p * PART + q)];
        }
#pragma unroll
        for (int q = 0; q < PART; q++)
        {
            const int u = p * PART + q;
            if (u >= NE)
                continue;
            if constexpr (sizeof(TS) == sizeof(float))
                keep[u] = blk[q];
            else
            {
                const int e = entry_row(C, SYM, u) * C + entry_col(C, SYM, u);
                const int f = entry_col(C, SYM, u) * C + entry_row(C, SYM, u);
                V.stencil[sten_index<TS>(slot, e, CC, T, sp)] = blk[q];
                if (SYM && e != f)
                    V.stencil[sten_index<TS>(slot, f, CC, T, sp)] = blk[q];
                if (bc_copy)
                {
                    V.bc_sten[bc_sten_pos(tx, ty, (V.w + 3) >> 2, slot, CC, e)] = blk[q];
                    if (SYM && e != f)
                        V.bc_sten[bc_sten_pos(tx, ty, (V.w + 3) >> 2, slot, CC, f)] = blk[q];
                }
            }
        }
    }
    if constexpr (sizeof(TS) == sizeof(float))
    {
        // the FP32 stencil keeps a texel's block contiguous: whole 16-byte stores where the block is whole vectors
        auto entry = [&](int e) {
            const int i = e / C, j = e % C, lo = i < j ? i : j, hi = i < j ? j : i;
            return SYM ? keep[lo * C - lo * (lo - 1) / 2 + (hi - lo)] : keep[SYM ? 0 : e];
        };
        float* out = reinterpret_cast<float*>(V.stencil) + sten_index<float>(slot, 0, CC, T, sp);
        if constexpr (CC % 4 == 0)
        {
#pragma unroll
            for (int v = 0; v < CC / 4; v++)
                reinterpret_cast<float4*>(out)[v] =
                    make_float4(entry(4 * v), entry(4 * v + 1), entry(4 * v + 2), entry(4 * v + 3));
        }
        else
        {
#pragma unroll
            for (int e = 0; e < CC; e++)
                out[e] = entry(e);
        }
    }
}

template <typename TS, int NY>
__device__ __forceinline__ void expand_block(const TileArgs<TS>& A, const PlaneView& V, const TS (&sums)[MAX_MONO],
                                             int slot, int c, int tx, int ty, size_t T, size_t sp)
{
#define NB_EXPAND(C)                                                                                                  \
    if (A.plain)                                                                                                      \
        expand_store<TS, NY, C, true>(A, V, sums, slot, tx, ty, T, sp);                                               \
    else                                                                                                              \
        expand_store<TS, NY, C, false>(A, V, sums, slot, tx, ty, T, sp);                                              \
    break;
    switch (c)
    {
    case 1: NB_EXPAND(1)
    case 2: NB_EXPAND(2)
    case 3: NB_EXPAND(3)
    default: NB_EXPAND(4)
    }
#undef NB_EXPAND
}

// A block with no neighbour in its slot's direction: the reference's block is zero (no site touches both texels).
template <typename TS>
__device__ __forceinline__ void store_zero_block(const TileArgs<TS>& A, const PlaneView& V, int slot, int c, int tx,
                                                 int ty, size_t T, size_t sp)
{
    const int cc = c * c;
    for (int e = 0; e < cc; e++)
    {
        reinterpret_cast<TS*>(V.stencil)[sten_index<TS>(slot, e, cc, T, sp)] = (TS)0;
        if (sizeof(TS) == sizeof(double) && A.bc_copy)
            V.bc_sten[bc_sten_pos(tx, ty, (V.w + 3) >> 2, slot, cc, e)] = 0.0;
    }
}

// The monomials [LO, HI) of the fixed layout of one visit added to the sums: scale (the product of the two weights)
// times the constant, the four linear terms, then the ten products (i <= k) row by row; a narrower latent uses the
// entries whose indices are all below its channel count, which is the reference's order.
template <typename TS, int NY, int LO, int HI>
__device__ __forceinline__ void visit_sums(TS (&sums)[MAX_MONO], const float4& y4, TS scale)
{
    const TS y[MAX_CH] = { (TS)y4.x, (TS)y4.y, (TS)y4.z, (TS)y4.w };
#pragma unroll
    for (int L = LO; L < HI; L++)
    {
        if (!mono_used(L, NY))
            continue;
        const TS m = L == 0 ? (TS)1 : (L <= MAX_CH ? y[L <= MAX_CH && L > 0 ? L - 1 : 0]
                                                   : y[pair_i(L > MAX_CH ? L - 5 : 0)] * y[pair_k(L > MAX_CH ? L - 5 : 0)]);
        sums[L] += scale * m;
    }
}

constexpr int MAX_SITES = 5;   // sites of a pixel at the largest K the split assembly takes
constexpr size_t ANY_SHARED_MAX = 200 * 1024;   // the most a tile of k_gather_any1 may take

// Level 1 planes whose visits are not tabled, in tiles of the same texels (k_gather_any1): the pixels a tile's texels
// can meet on each axis, at most, per plane.
struct AnyTiles
{
    int px[MAX_PLANES], py[MAX_PLANES];
};

// The entries of n pixel columns' (or rows') taps, one of padding after every four.
__host__ __device__ inline int any_taps(int n, int per)
{
    return n * per * 2 + (n + 3) / 4;
}

// Shared memory of one such tile: every site's sample, then each pixel column's and row's taps.
inline size_t any_tile_bytes(int px, int py, int per)
{
    return (size_t)((px + 3) / 4 * 4) * py * per * sizeof(float4) +
           (size_t)(any_taps(px, per) + any_taps(py, per)) * 16;
}

constexpr int WALK_THREADS = 128;   // threads of a k_gather_walk block

struct WalkBlocks
{
    long long start[MAX_PLANES + 1];   // each plane's first block (a tiled plane has none)
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// The plane of a block (planes in descending order) and the block's number within the plane.
template <typename TS>
__device__ __forceinline__ int tile_plane(const TileArgs<TS>& A, int n, int& tile)
{
    int pl = n - 1;
    while ((int)blockIdx.x >= A.bend[pl])
        pl--;
    tile = (int)blockIdx.x - (A.bend[pl] - A.btiles[pl]);
    return pl;
}

// The gradient terms of channels first .. (two of FP64, four of FP32) in the samples' places, asynchronously where a
// site's are 16 aligned bytes.
template <typename TS, class Each>
__device__ __forceinline__ void stage_terms(const TileArgs<TS>& A, float4* sy, int first, int c, Each each_site)
{
    constexpr int CH = sizeof(TS) == sizeof(float) ? 4 : 2;
    if constexpr (sizeof(TS) == sizeof(float))
    {
        const float* t = (const float*)A.terms;
        if (c == MAX_CH)
            each_site([&](int at, size_t site) { cp_async16(sy + at, t + site * MAX_CH); });
        else
            each_site([&](int at, size_t site) {
                float* dst = reinterpret_cast<float*>(sy + at);
                for (int a = 0; a < c; a++)
                    dst[a] = __ldg(t + site * c + a);
            });
    }
    else
    {
        const double* t = (const double*)A.terms + first;
        if (c % 2 == 0)
            each_site([&](int at, size_t site) { cp_async16(sy + at, t + site * c); });
        else
            each_site([&](int at, size_t site) {
                double* dst = reinterpret_cast<double*>(sy + at);
                for (int a = 0; a < CH && first + a < c; a++)
                    dst[a] = __ldg(t + site * c + a);
            });
    }
}

// The launches, one module per type of the sums and channel count NY of the other latent (gather.cu, gather_any.cu).
template <typename TS, int NY>
int launch_gather_tiles(nntc_b200_device* d, int level0, const Planes& P, const TileArgs<TS>& A, unsigned grid);
template <typename TS, int NY>
int launch_gather_any(nntc_b200_device* d, const Planes& P, const TileArgs<TS>& A, const AnyTiles& S, unsigned grid,
                      size_t shared);
template <typename TS, int NY>
int launch_gather_walk(nntc_b200_device* d, int level0, const Planes& P, const TileArgs<TS>& A, const WalkBlocks& B);

}   // namespace nb
