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
//     and the expansion against the monomial matrices after it, is the same bits. gather.cu does it in tiles;
//     k_gather_walk below takes the few planes no tile fits.
//
// Every plane of the chain is in each launch (nb::Planes); the per-site buffer holds every plane's sites.

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "footprint.cuh"
#include "gather.cuh"

namespace nb
{

constexpr int SITE_THREADS = 256;
constexpr int SITE_BLOCK_MAX = 64 * 5;   // threads of a k_site_terms block at K = 4
// Pixels of one block (planes_for's unit, so that a block has one plane), in rounds that share its set-up; a launch of
// fewer than SITE_FEW pixels takes a block per round, which its SMs are too few blocks without (1 x 100 x 76: 3.9
// against 7.4 us; at 4 x 1024 x 1024 the rounds save 2%).
constexpr int SITE_PIXELS = THREADS, SITE_FEW = 148 * 6 * SITE_PIXELS;

struct SiteArgs
{
    void* terms;                        // [site][c] over every plane: doubles, or floats (MIXED)
    float4* y;                          // [site]: the site's sample of the other latent
    const float* tgt;                   // [fractional site][NOUT]: the targets of the sites j > 0 (k_site_targets)
    long long site0[MAX_PLANES + 1];    // the first site of each plane in `terms`
    long long tsite0[MAX_PLANES + 1];   // the first fractional site of each plane in `tgt`
    unsigned span;                      // pixels of one block
};

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
// The decoder as a launch parameter, each row at a fixed stride of 24 slots, [c_q (4)][s_i (4)][s_i c_q (4 x 4)]: with
// the row loop unrolled every weight is a constant-bank operand. Slots of channels the layout does not use are never
// read (the channel loops are guarded), so the arithmetic is the reference's operation for operation.
// Fused, every weight twice, side by side: the operand of a packed instruction.
template <bool MIXED>
struct SiteDecoder
{
    using Weight = typename std::conditional<MIXED, unsigned long long, float>::type;
    Weight w[MAX_NOUT * 24];
    Weight b[MAX_NOUT];
    Weight cw[MAX_NOUT];
    double cwd[MAX_NOUT];   // the outputs' weights in double (the FP64 terms)
};

// A lane's sites' values of one quantity. Packed: two side by side in a 64-bit register, for the packed FP32 instructions,
// which do both in one issue slot, each half rounded as the scalar instruction rounds it. The unfused form keeps scalar
// instructions: a packed multiply whose product is added by a packed add came back fused, whatever the rounding
// qualifiers (the assembly's own bits gave it away), and the plain form rounds every product.
template <bool PACKED>
struct Two;

template <>
struct Two<true>
{
    unsigned long long v;
    static __device__ __forceinline__ Two make(float a, float b)
    {
        Two r;
        asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
        return r;
    }
    static __device__ __forceinline__ Two weight(unsigned long long twice) { return Two{ twice }; }
    __device__ __forceinline__ void split(float& a, float& b) const
    {
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    }
    // a + b c
    static __device__ __forceinline__ Two madd(Two a, Two b, Two c)
    {
        Two r;
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(b.v), "l"(c.v), "l"(a.v));
        return r;
    }
    static __device__ __forceinline__ Two mul(Two a, Two b)
    {
        Two r;
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
        return r;
    }
    static __device__ __forceinline__ Two sub(Two a, float x, float y)
    {
        Two r, t = make(-x, -y);   // a sign flipped exactly, then added
        asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(t.v));
        return r;
    }
};

template <>
struct Two<false>   // one site
{
    float v;
    static __device__ __forceinline__ Two make(float a, float) { return Two{ a }; }
    static __device__ __forceinline__ Two weight(float w) { return Two{ w }; }
    __device__ __forceinline__ void split(float& a, float& b) const { a = b = v; }
    static __device__ __forceinline__ Two madd(Two a, Two b, Two c) { return Two{ __fadd_rn(a.v, __fmul_rn(b.v, c.v)) }; }
    static __device__ __forceinline__ Two mul(Two a, Two b) { return Two{ __fmul_rn(a.v, b.v) }; }
    static __device__ __forceinline__ Two sub(Two a, float x, float) { return Two{ a.v - x }; }
};

// MIXED (the adjoint form, whose stencil and sums are FP32): the same terms with fused multiply-adds and the gradient
// term summed and stored in FP32 - half the instructions of the reference's unfused float arithmetic, no FP64 work per
// output and half the bytes of the terms.
//
// A block takes A.span consecutive pixels of a plane in rounds, the last two warps their centre sites and the others
// their fractional sites, U to a lane: a warp's lanes agree on which kind they are, its targets are one contiguous run, staged in shared
// memory by 16-byte asynchronous copies while the lanes sample the latents, and a pixel's sites are written by one block
// (half-written sectors cost a read of DRAM each). A lane reading its own row of targets from global memory touches a
// line per lane and load, NOUT times over, which together with the 64-bit index divisions and the guards of run-time
// channel counts was most of the kernel: it is bound by issue, and these are instructions. Fused, a lane's two sites go
// through the packed FP32 instructions; unfused, one site a lane keeps the occupancy (two: 592 -> 683 us at 4 x 2048 x
// 1024). C0, C1: the channel counts, or 0, 0 to take the launch's (any count with guarded loops; the counts with C1 = 4,
// the encoder's default, have their own kernels).
template <bool LEVEL0, int NOUT, bool MIXED, int C0, int C1>
__global__ void __launch_bounds__(SITE_BLOCK_MAX) k_site_terms(Planes P, const __grid_constant__ SiteArgs A,
                                                               const __grid_constant__ SiteDecoder<MIXED> W)
{
    constexpr int U = MIXED ? 2 : 1, RUN = 32 * U, PIXELS = 64 * U;   // PIXELS: the pixels of one round of the block
    extern __shared__ __align__(16) float targets[];   // [warp][RUN][NOUT]
    const long long base = (long long)blockIdx.x * A.span;
    const int pl = plane_of(P, base);
    const PlaneView& V = P.p[pl];
    const int kc = P.kc, per = 1 + kc, c0 = C0 ? C0 : P.c0, c1 = C1 ? C1 : P.c1;
    const unsigned pixels = (unsigned)V.w0 * (unsigned)V.h0, pixel00 = (unsigned)(base - P.start[pl]);
    if (pixel00 >= pixels)
        return;
    const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool centre = warp >= 2 * (unsigned)kc;
    const unsigned each = centre ? 1 : (unsigned)kc;            // the warp's sites per pixel
    const unsigned first = (centre ? warp - 2 * (unsigned)kc : warp) * RUN;   // its first site of a round
    float* mine = targets + warp * RUN * NOUT;
    const float* all = centre ? V.src : A.tgt + (size_t)A.tsite0[pl] * NOUT;
    // a division by a power of two is the product with its exact reciprocal, the same bits; 0: not one
    const float inv_w = (V.w0 & (V.w0 - 1)) == 0 ? 1.0f / (float)V.w0 : 0.0f;
    const float inv_h = (V.h0 & (V.h0 - 1)) == 0 ? 1.0f / (float)V.h0 : 0.0f;
    const unsigned inv_each = (65536 + each - 1) / each;   // n / each = (n inv_each) >> 16, n < 2^10
    int row0 = (int)(pixel00 / (unsigned)V.w0), col0 = (int)(pixel00 - (unsigned)row0 * (unsigned)V.w0);
#pragma unroll 1
    for (unsigned pixel0 = pixel00; pixel0 < min(pixel00 + A.span, pixels); pixel0 += PIXELS, col0 += PIXELS)
    {
        const unsigned end = min((unsigned)PIXELS, pixels - pixel0) * each;   // the warp's kind of sites in this round
        if (first >= end)
            return;
        const unsigned run = min((unsigned)RUN, end - first) * NOUT;   // the warp's floats
        const float* from = all + ((size_t)pixel0 * each + first) * NOUT;
        __syncwarp();   // the last round's targets are spent
        if (((size_t)from & 15) == 0)
        {
            for (unsigned i = lane; i < run / 4; i += 32)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(mine + 4 * i)),
                             "l"(from + 4 * i)
                             : "memory");
            for (unsigned i = run / 4 * 4 + lane; i < run; i += 32)
                mine[i] = __ldg(from + i);
        }
        else
            for (unsigned i = lane; i < run; i += 32)
                mine[i] = __ldg(from + i);
        while (col0 >= V.w0)
        {
            col0 -= V.w0;
            row0++;
        }
        float s_[2][MAX_CH] = {}, c_[2][MAX_CH] = {};
        size_t site[2] = { 0, 0 };
#pragma unroll
        for (int u = 0; u < U; u++)
        {
            const unsigned n = min(first + lane + 32 * u, end - 1);   // past the end: the last site again, not stored
            const unsigned in = (n * inv_each) >> 16, pixel = pixel0 + in;
            const int j = centre ? 0 : 1 + (int)(n - in * each);
            int py = row0, px = col0 + (int)in;
            while (px >= V.w0)
            {
                px -= V.w0;
                py++;
            }
            float dx, dy;
            dx = dy = 0.0f;
            if (j > 0)
                subtexel_turned(kc, j - 1, px, py, dx, dy);
            const Tap tp = tap_scaled(px, py, dx, dy, V.w0, V.h0, V.w1, V.h1, inv_w, inv_h);
            if constexpr (C1 > 0)
                blend_c<C1>(V.v1, V.w1, tp, c_[u]);
            else
                blend_u<MAX_CH>(V.v1, V.w1, c1, tp, c_[u]);
            if (centre)
            {
#pragma unroll
                for (int i = 0; i < MAX_CH; i++)
                    if (i < c0)
                        s_[u][i] = __ldg(V.v0 + (size_t)pixel * c0 + i);
            }
            else
            {
                const Tap t0 = tap_at(px, py, dx, dy, V.w0, V.h0, V.w0, V.h0);
                if constexpr (C0 > 0)
                    blend_c<C0>(V.v0, V.w0, t0, s_[u]);
                else
                    blend_u<MAX_CH>(V.v0, V.w0, c0, t0, s_[u]);
            }
            site[u] = (size_t)A.site0[pl] + (size_t)pixel * per + j;
        }
        using F2 = Two<MIXED>;
        F2 sbar[MAX_CH], cbar[MAX_CH], accf[MAX_CH];
        double acc[MAX_CH];
#pragma unroll
        for (int a = 0; a < MAX_CH; a++)
        {
            sbar[a] = F2::make(s_[0][a], s_[1][a]);
            cbar[a] = F2::make(c_[0][a], c_[1][a]);
            accf[a] = F2::make(0.0f, 0.0f);
            acc[a] = 0.0;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        const float* tgt = mine + lane * NOUT;
        const float* tgt2 = mine + min(lane + 32 * (U - 1), end - 1 - first) * NOUT;
        // a + b c, unfused (the reference's rounding) or fused (MIXED)
        auto madd = [](F2 a, F2 b, F2 c) { return F2::madd(a, b, c); };
#pragma unroll
        for (int r = 0; r < NOUT; r++)
        {
            auto row = [&](int q) { return F2::weight(W.w[r * 24 + q]); };   // [c_q][s_i][s_i c_q]
            F2 out = F2::weight(W.b[r]);
            F2 col[MAX_CH];
            if (!LEVEL0)
            {
#pragma unroll
                for (int i = 0; i < MAX_CH; i++)
                    if (i < c0)
                        out = madd(out, row(4 + i), sbar[i]);
#pragma unroll
                for (int q = 0; q < MAX_CH; q++)
                    if (q < c1)
                    {
                        F2 gg = row(q);
#pragma unroll
                        for (int i = 0; i < MAX_CH; i++)
                            if (i < c0)
                                gg = madd(gg, sbar[i], row(8 + i * 4 + q));
                        col[q] = gg;
                        out = madd(out, gg, cbar[q]);
                    }
            }
            else
            {
#pragma unroll
                for (int q = 0; q < MAX_CH; q++)
                    if (q < c1)
                        out = madd(out, row(q), cbar[q]);
#pragma unroll
                for (int i = 0; i < MAX_CH; i++)
                    if (i < c0)
                    {
                        F2 qq = row(4 + i);
#pragma unroll
                        for (int q = 0; q < MAX_CH; q++)
                            if (q < c1)
                                qq = madd(qq, cbar[q], row(8 + i * 4 + q));
                        col[i] = qq;
                        out = madd(out, qq, sbar[i]);
                    }
            }
            const F2 res = F2::sub(out, tgt[r], tgt2[r]);
            const int c = LEVEL0 ? c0 : c1;
            if (MIXED)
            {
#pragma unroll
                for (int a = 0; a < MAX_CH; a++)
                    if (a < c)
                        accf[a] = madd(accf[a], F2::mul(F2::weight(W.cw[r]), col[a]), res);
            }
            else
            {
                float r0, g0, unused;
                res.split(r0, unused);
                const double d0 = (double)r0, cwd = W.cwd[r];
#pragma unroll
                for (int a = 0; a < MAX_CH; a++)
                    if (a < c)
                    {
                        col[a].split(g0, unused);
                        acc[a] += cwd * (double)g0 * d0;
                    }
            }
        }
        const int c = LEVEL0 ? c0 : c1, ny = LEVEL0 ? c1 : c0;
        float f_[2][MAX_CH];
#pragma unroll
        for (int a = 0; a < MAX_CH; a++)
            accf[a].split(f_[0][a], f_[1][a]);
#pragma unroll
        for (int u = 0; u < U; u++)
        {
            if (first + lane + 32 * u >= end)
                continue;
            if (MIXED)
            {
                float* out = static_cast<float*>(A.terms) + site[u] * c;
                if (c == MAX_CH)
                    *reinterpret_cast<float4*>(out) = make_float4(f_[u][0], f_[u][1], f_[u][2], f_[u][3]);
                else
                {
#pragma unroll
                    for (int a = 0; a < MAX_CH; a++)
                        if (a < c)
                            out[a] = f_[u][a];
                }
            }
            else
            {
                double* out = static_cast<double*>(A.terms) + site[u] * c;
                if (c == MAX_CH)
                {
                    reinterpret_cast<double2*>(out)[0] = make_double2(acc[0], acc[1]);
                    reinterpret_cast<double2*>(out)[1] = make_double2(acc[2], acc[3]);
                }
                else
                {
#pragma unroll
                    for (int a = 0; a < MAX_CH; a++)
                        if (a < c)
                            out[a] = acc[a];
                }
            }
            // the other latent's sample, which every (texel, slot) of the gather that meets this site needs again
            float y[MAX_CH];
#pragma unroll
            for (int i = 0; i < MAX_CH; i++)
                y[i] = i < ny ? (LEVEL0 ? c_[u][i] : s_[u][i]) : 0.0f;
            A.y[site[u]] = make_float4(y[0], y[1], y[2], y[3]);
        }
    }
}

template <bool LEVEL0, int NOUT, bool MIXED>
static void launch_site_terms(const nntc_b200_device* d, const Planes& S, SiteArgs A, cudaStream_t stream)
{
    using Weight = typename SiteDecoder<MIXED>::Weight;
    SiteDecoder<MIXED> W{};
    const int nin = d->nin, c0 = d->c0, c1 = d->c1;
    auto weight = [](float v) {
        if (!MIXED)
            return (Weight)v;
        unsigned bits;
        std::memcpy(&bits, &v, sizeof(bits));
        return (Weight)((unsigned long long)bits << 32 | bits);
    };
    for (int r = 0; r < d->nout; r++)
    {
        for (int q = 0; q < c1; q++)
            W.w[r * 24 + q] = weight(d->host_weights[(size_t)r * nin + q]);
        for (int i = 0; i < c0; i++)
            W.w[r * 24 + 4 + i] = weight(d->host_weights[(size_t)r * nin + c1 + i]);
        for (int i = 0; i < c0; i++)
            for (int q = 0; q < c1; q++)
                W.w[r * 24 + 8 + i * 4 + q] = weight(d->host_weights[(size_t)r * nin + c1 + c0 + i * c1 + q]);
        W.b[r] = weight(d->host_bias[r]);
        W.cw[r] = weight(d->m.cw[r]);
        W.cwd[r] = (double)d->m.cw[r];
    }
    constexpr int U = MIXED ? 2 : 1;
    A.span = S.start[S.n] < SITE_FEW ? 64 * U : SITE_PIXELS;
    const int blocks = (int)(S.start[S.n] / A.span), threads = 64 * (1 + S.kc);
    const size_t shared = (size_t)threads * U * NOUT * sizeof(float);
    if (S.c1 != MAX_CH)
        k_site_terms<LEVEL0, NOUT, MIXED, 0, 0><<<blocks, threads, shared, stream>>>(S, A, W);
    else if (S.c0 == 1)
        k_site_terms<LEVEL0, NOUT, MIXED, 1, 4><<<blocks, threads, shared, stream>>>(S, A, W);
    else if (S.c0 == 2)
        k_site_terms<LEVEL0, NOUT, MIXED, 2, 4><<<blocks, threads, shared, stream>>>(S, A, W);
    else if (S.c0 == 3)
        k_site_terms<LEVEL0, NOUT, MIXED, 3, 4><<<blocks, threads, shared, stream>>>(S, A, W);
    else
        k_site_terms<LEVEL0, NOUT, MIXED, 4, 4><<<blocks, threads, shared, stream>>>(S, A, W);
}

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
constexpr int WALK_THREADS = 128;

struct WalkBlocks
{
    long long start[MAX_PLANES + 1];   // each plane's first block (a tiled plane has none)
};

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

template <typename TS>
static int launch_walk(nntc_b200_device* d, int level0, const Planes& P, const TileArgs<TS>& A, const WalkBlocks& B)
{
    const unsigned grid = (unsigned)B.start[P.n];
    const int ny = level0 ? d->c1 : d->c0;
#define NB_WALK(NY)                                                                                                   \
    if (level0)                                                                                                       \
        k_gather_walk<true, TS, NY><<<grid, WALK_THREADS, 0, d->stream>>>(P, A, B);                                   \
    else                                                                                                              \
        k_gather_walk<false, TS, NY><<<grid, WALK_THREADS, 0, d->stream>>>(P, A, B);                                  \
    break;
    switch (ny)
    {
    case 1: NB_WALK(1)
    case 2: NB_WALK(2)
    case 3: NB_WALK(3)
    default: NB_WALK(4)
    }
#undef NB_WALK
    NB_LAUNCHED();
    return NNTC_B200_OK;
}

// The tiles of k_gather_any1 up to which it takes a level's planes that are not tabled; with more of them the walk does.
// The tiles test each pixel once for five warps, whatever comes of it, and stage its sites, which pays the more sites a
// pixel has; a thread a (texel, slot) waits longer but keeps more of them in flight, so that it gains as the launch
// grows. FP32 terms of four channels are staged side by side with the samples; an odd count of FP64 ones a value at a
// time. Measured (us, tiles / walk; at 950, 2050, 5460 and 15666 tiles: 700 x 500 to 3000 x 2000), every slot:
//   K = 0: FP64 2 channels 92 / 104, 159 / 150, 394 / 320, 1061 / 750; 3 channels 154 / 105, 262 / 154, 697 / 323,
//          1930 / 761; FP32 2 channels 99 / 90, 170 / 143, 463 / 296, 1270 / 700; 4 channels 85 / 128, 149 / 179, 378 / 360,
//          1034 / 895
//   K = 1: FP64 2 channels 132 / 197, 229 / 291, 571 / 625, 1528 / 1496; 3 channels 206 / 220, 367 / 312, 939 / 669,
//          2537 / 1624; FP32 2 channels 142 / 178, 242 / 282, 642 / 601, 1758 / 1448
//   K = 2: FP64 2 channels 172 / 306, 296 / 434, 739 / 934, 1983 / 2191; 3 channels 259 / 329, 457 / 447, 1162 / 945,
//          3200 / 2213; FP32 2 channels 182 / 258, 318 / 400, 810 / 849, 2229 / 1994
//   K = 4: FP64 2 channels (5460 and 15666) 1172 / 1731, 3150 / 3953; 3 channels 2060 / 1771, 5808 / 4011; FP32 2 channels
//          1265 / 1579, 3454 / 3685; 4 channels 1066 / 1835, 2913 / 4432
// The diagonal blocks alone leave three of the five warps idle (FP64 2 channels at 400, 2050 and 5460 tiles: K = 0 36 / 66,
// 139 / 89, 350 / 184; K = 2 69 / 197, 266 / 275, 666 / 570; K = 4 124 / 366, 431 / 532, 1119 / 1028).
static int any_tiles_line(bool f32, int c, int sites, bool every_slot)
{
    const bool staged = f32 && c == MAX_CH;
    const int base = staged ? 3200 : (!f32 && c % 2 != 0 ? 400 : 800);
    if (every_slot)
        return base * sites * sites;
    return staged ? base / 2 * sites * sites : base * 3 / 4 * sites;
}

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
    if (any_tiles > any_tiles_line(sizeof(TS) == sizeof(float), c, 1 + k, slots == SLOTS))
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
        NB_TRY(launch_walk<TS>(d, level0, P, A, B));
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
            NB_TRY(launch_gather_any(d, P, G, R, (unsigned)blocks, shared));
    }
    if (tiles > 0)
        NB_TRY(launch_gather_tiles(d, level0, P, A, (unsigned)tiles));
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
        if (level0)                                                                                                   \
        {                                                                                                             \
            if (f32)                                                                                                  \
                launch_site_terms<true, NO, true>(d, S, A, d->stream);                                                \
            else                                                                                                      \
                launch_site_terms<true, NO, false>(d, S, A, d->stream);                                               \
        }                                                                                                             \
        else if (f32)                                                                                                 \
            launch_site_terms<false, NO, true>(d, S, A, d->stream);                                                   \
        else                                                                                                          \
            launch_site_terms<false, NO, false>(d, S, A, d->stream);                                                  \
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
