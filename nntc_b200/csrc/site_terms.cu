// site_terms.cu: the site pass of the stencil assembly (assemble.cu): one lane per site forms the site's gradient term and
// its sample of the other latent.
//
// Compiled once per output count and form (NB_NOUT, NB_MIXED), a module each: the first launch of any of a module's kernels
// loads all of it. With every kernel of the assembly in two modules a process's first decoder solve and first block took
// 20 and 18 ms to load them (96 x 64, two textures); now 0.8 and 6 ms.

#include <cstring>
#include <type_traits>

#include "site_terms.cuh"

namespace nb
{

constexpr int SITE_BLOCK_MAX = 64 * 5;   // threads of a k_site_terms block at K = 4
// Pixels of one block (planes_for's unit, so that a block has one plane), in rounds that share its set-up; a launch of
// fewer than SITE_FEW pixels takes a block per round, which its SMs are too few blocks without (1 x 100 x 76: 3.9
// against 7.4 us; at 4 x 1024 x 1024 the rounds save 2%).
constexpr int SITE_PIXELS = THREADS, SITE_FEW = 148 * 6 * SITE_PIXELS;

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
static void launch_level(const nntc_b200_device* d, const Planes& S, SiteArgs A, cudaStream_t stream)
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

template <int NOUT, bool MIXED>
void launch_site_terms(const nntc_b200_device* d, const Planes& S, SiteArgs A, int level0, cudaStream_t stream)
{
    if (level0)
        launch_level<true, NOUT, MIXED>(d, S, A, stream);
    else
        launch_level<false, NOUT, MIXED>(d, S, A, stream);
}

template void launch_site_terms<NB_NOUT, NB_MIXED>(const nntc_b200_device*, const Planes&, SiteArgs, int, cudaStream_t);

}   // namespace nb
