// stencil.cu: blocks (b) and (c'), the latent planes as sparse weighted least squares (src/solve_level1.cu).
//
// Block (b) holds level 0 and the decoder and solves level 1; block (c') (--l0 bc8) holds level 1 and the decoder and
// solves level 0 as a continuous 8-bit plane. Both assemble a 9-point block stencil H (five owned C x C blocks per
// texel, the other four read as the neighbours' transposes) and a gradient by GATHER, one thread per texel of the
// unknown, exactly as src/solve_level1.cu:259-581 derives it; then either preconditioned conjugate gradients on
// (H + lambda I) d = -grad (src/solve_level1.cu:1222-1338) or four-colour quantised Gauss-Seidel sweeps with the exact
// per-value grid argmin (src/solve_level1.cu:1023-1098, 1343-1403).
//
// Per-texel arithmetic is the reference's, operation for operation, compiled without FMA contraction: given the same
// planes and decoder the stencil, the gradient, the preconditioner and every sweep decision are the same bits as the
// reference's. What differs is the B200 shape:
//
// - every plane of the chain in ONE launch (nb::Planes), one stream, no per-plane fan-out;
// - the FP64 stencil stored structure-of-arrays [slot][i][j][texel], coalesced for a warp of consecutive texels, the FP32
//   one by texel, whose kernels take a lane per row of a block;
// - the assembly is assemble.cu's; the reference-shaped one here, behind an option, keeps its 5 x nmono
//   monomial sums in shared memory (registers spill at C = 4);
// - the conjugate-gradient iteration is 5 launches (matvec + <p,Ap>, alpha, update + preconditioner + <r,r> +
//   <r,z>, beta, direction) and nothing else instead of 13, all planes in lockstep, and the stop is decided ON THE
//   DEVICE with the reference's rule (a plane leaves at an iteration that is a multiple of CG_PROBE once its residual is below the
//   tolerance); the host reads one active-plane count every CG_PROBE iterations, the reference's probe cadence.
// - every dot product is a fixed-order two-stage reduction: one partial per 256-texel block, added per plane in
//   block order.

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "device.cuh"

namespace nb
{

constexpr int ASM_THREADS = 128;

// ---- the gather (src/solve_level1.cu:259-581) ----------------------------------------------------------------------

struct AsmArgs
{
    const float* weights;
    const float* bias;
    const float* cw;
    const double* mono;   // nmono matrices of c x c
    int nmono;
};

// The monomials of a form in y: 1, y_i, y_i y_j (i <= j), in double (src/solve_level1.cu:142-152).
__device__ __forceinline__ void monomials(const float* y, int n, double* out)
{
    int k = 0;
    out[k++] = 1.0;
    for (int i = 0; i < n; i++)
        out[k++] = (double)y[i];
    for (int i = 0; i < n; i++)
        for (int j = i; j < n; j++)
            out[k++] = (double)y[i] * (double)y[j];
}

// The four corners of a tap merged by texel index, so a clamped duplicate adds its weight to one texel.
__device__ __forceinline__ int merge_taps(const Tap& t, int* nx, int* ny, float* tw)
{
    const int cx[4] = { t.x0, t.x1, t.x0, t.x1 };
    const int cy[4] = { t.y0, t.y0, t.y1, t.y1 };
    float cwt[4];
    tap_weights(t, cwt);
    int taps = 0;
    for (int q = 0; q < 4; q++)
    {
        int found = -1;
        for (int e = 0; e < taps; e++)
            if (nx[e] == cx[q] && ny[e] == cy[q])
                found = e;
        if (found >= 0)
            tw[found] += cwt[q];
        else
        {
            nx[taps] = cx[q];
            ny[taps] = cy[q];
            tw[taps] = cwt[q];
            taps++;
        }
    }
    return taps;
}

// The pixels whose bilinear footprint into an n1-wide plane can reach texel ti (src/solve_level1.cu:246-257).
__device__ __forceinline__ void footprint(int ti, int n0, int n1, int& lo, int& hi)
{
    const double r = (double)n0 / (double)n1;
    lo = (int)ceil(((double)ti - 0.5) * r - 1.0);
    hi = (int)ceil(((double)ti + 1.5) * r) - 1;
    lo = lo < 0 ? 0 : lo;
    hi = hi > n0 - 1 ? n0 - 1 : hi;
}

template <bool LEVEL0>
__global__ void __launch_bounds__(ASM_THREADS) k_assemble(Planes P, AsmArgs A)
{
    extern __shared__ double sums_sh[];   // [slot * nmono + i][thread]
    const long long base = (long long)blockIdx.x * blockDim.x;
    const int pl = plane_of(P, base);
    const PlaneView& V = P.p[pl];
    const long long ti = base - P.start[pl] + threadIdx.x;
    const int c0 = P.c0, c1 = P.c1, nin = P.nin, nout = P.nout, kc = P.kc, nmono = A.nmono;
    const int c = LEVEL0 ? c0 : c1;
    const int tw_ = V.w, th_ = V.h;
    if (ti >= (long long)tw_ * th_)
        return;
    const int tx = (int)(ti % tw_), ty = (int)(ti / tw_);
    double* sums = sums_sh + threadIdx.x;
    const int S = blockDim.x;
    for (int i = 0; i < SLOTS * nmono; i++)
        sums[i * S] = 0.0;
    double g[MAX_CH];
    for (int i = 0; i < c; i++)
        g[i] = 0.0;

    int px_lo, px_hi, py_lo, py_hi;
    if (LEVEL0)
    {
        footprint(tx, V.w0, V.w0, px_lo, px_hi);
        footprint(ty, V.h0, V.h0, py_lo, py_hi);
    }
    else
    {
        footprint(tx, V.w0, V.w1, px_lo, px_hi);
        footprint(ty, V.h0, V.h1, py_lo, py_hi);
    }

    for (int py = py_lo; py <= py_hi; py++)
        for (int px = px_lo; px <= px_hi; px++)
            for (int j = 0; j <= kc; j++)
            {
                float dx, dy;
                site_offset(kc, j, px, py, dx, dy);
                int nx[4], ny[4];
                float tw[4];
                int taps = 0;
                float sbar[MAX_CH], cbar[MAX_CH], target[MAX_NOUT];
                const Tap tp = tap_at(px, py, dx, dy, V.w0, V.h0, V.w1, V.h1);
                if (!LEVEL0)
                {
                    taps = merge_taps(tp, nx, ny, tw);
                    int self = -1;
                    for (int e = 0; e < taps; e++)
                        if (nx[e] == tx && ny[e] == ty)
                            self = e;
                    if (self < 0)
                        continue;
                    blend<MAX_CH>(V.v1, V.w1, c1, tp, cbar);
                    if (j == 0)
                    {
                        const size_t pi = (size_t)py * V.w0 + px;
                        for (int i = 0; i < c0; i++)
                            sbar[i] = V.v0[pi * c0 + i];
                        for (int r = 0; r < nout; r++)
                            target[r] = __ldg(V.src + pi * nout + r);
                    }
                    else
                    {
                        const Tap t0 = tap_at(px, py, dx, dy, V.w0, V.h0, V.w0, V.h0);
                        blend<MAX_CH>(V.v0, V.w0, c0, t0, sbar);
                        blend<MAX_NOUT>(V.src, V.w0, nout, t0, target);
                    }
                    // G = A + sum_i sbar_i M_i, residual r = b + B sbar + G cbar - t (src/solve_level1.cu:335-352)
                    float gmat[MAX_NOUT * MAX_CH], res[MAX_NOUT];
                    for (int r = 0; r < nout; r++)
                    {
                        const float* row = A.weights + (size_t)r * nin;
                        float out = A.bias[r];
                        for (int i = 0; i < c0; i++)
                            out += row[c1 + i] * sbar[i];
                        for (int q = 0; q < c1; q++)
                        {
                            float gg = row[q];
                            for (int i = 0; i < c0; i++)
                                gg += sbar[i] * row[c1 + c0 + i * c1 + q];
                            gmat[r * c1 + q] = gg;
                            out += gg * cbar[q];
                        }
                        res[r] = out - target[r];
                    }
                    double mono[MAX_MONO];
                    monomials(sbar, c0, mono);
                    const float w_self = tw[self];
                    for (int a = 0; a < c1; a++)
                    {
                        double acc = 0.0;
                        for (int r = 0; r < nout; r++)
                            acc += (double)A.cw[r] * (double)gmat[r * c1 + a] * (double)res[r];
                        g[a] += (double)w_self * acc;
                    }
                    for (int e = 0; e < taps; e++)
                    {
                        const int slot = slot_of(nx[e] - tx, ny[e] - ty);
                        if (slot < 0)
                            continue;
                        const double scale = (double)w_self * (double)tw[e];
                        double* dst = sums + (size_t)slot * nmono * S;
                        for (int i = 0; i < nmono; i++)
                            dst[i * S] += scale * mono[i];
                    }
                }
                else
                {
                    blend<MAX_CH>(V.v1, V.w1, c1, tp, cbar);
                    if (j == 0)
                    {
                        const size_t pi = (size_t)py * V.w0 + px;
                        nx[0] = px;
                        ny[0] = py;
                        tw[0] = 1.0f;
                        taps = 1;
                        for (int i = 0; i < c0; i++)
                            sbar[i] = V.v0[pi * c0 + i];
                        for (int r = 0; r < nout; r++)
                            target[r] = __ldg(V.src + pi * nout + r);
                    }
                    else
                    {
                        const Tap t0 = tap_at(px, py, dx, dy, V.w0, V.h0, V.w0, V.h0);
                        blend<MAX_CH>(V.v0, V.w0, c0, t0, sbar);
                        blend<MAX_NOUT>(V.src, V.w0, nout, t0, target);
                        taps = merge_taps(t0, nx, ny, tw);
                    }
                    int self = -1;
                    for (int e = 0; e < taps; e++)
                        if (nx[e] == tx && ny[e] == ty)
                            self = e;
                    if (self < 0)
                        continue;
                    // Q = B + sum_q cbar_q N_q, residual r = b + A cbar + Q sbar - t (src/solve_level1.cu:518-536)
                    float qmat[MAX_NOUT * MAX_CH], res[MAX_NOUT];
                    for (int r = 0; r < nout; r++)
                    {
                        const float* row = A.weights + (size_t)r * nin;
                        float out = A.bias[r];
                        for (int q = 0; q < c1; q++)
                            out += row[q] * cbar[q];
                        for (int i = 0; i < c0; i++)
                        {
                            float qq = row[c1 + i];
                            for (int q = 0; q < c1; q++)
                                qq += cbar[q] * row[c1 + c0 + i * c1 + q];
                            qmat[r * c0 + i] = qq;
                            out += qq * sbar[i];
                        }
                        res[r] = out - target[r];
                    }
                    double mono[MAX_MONO];
                    monomials(cbar, c1, mono);
                    const float w_self = tw[self];
                    for (int a = 0; a < c0; a++)
                    {
                        double acc = 0.0;
                        for (int r = 0; r < nout; r++)
                            acc += (double)A.cw[r] * (double)qmat[r * c0 + a] * (double)res[r];
                        g[a] += (double)w_self * acc;
                    }
                    for (int e = 0; e < taps; e++)
                    {
                        const int slot = slot_of(nx[e] - tx, ny[e] - ty);
                        if (slot < 0)
                            continue;
                        const double scale = (double)w_self * (double)tw[e];
                        double* dst = sums + (size_t)slot * nmono * S;
                        for (int i = 0; i < nmono; i++)
                            dst[i * S] += scale * mono[i];
                    }
                }
            }

    // The five blocks expanded once against the monomial matrices (src/solve_level1.cu:382-399), stored SoA.
    const size_t T = (size_t)tw_ * th_;
    const int cc = c * c;
    for (int slot = 0; slot < SLOTS; slot++)
    {
        double blk[MAX_CH * MAX_CH];
        for (int e = 0; e < cc; e++)
            blk[e] = 0.0;
        for (int i = 0; i < nmono; i++)
        {
            const double s = sums[(size_t)(slot * nmono + i) * S];
            if (s == 0.0)
                continue;
            const double* mat = A.mono + (size_t)i * cc;
            for (int e = 0; e < cc; e++)
                blk[e] += s * __ldg(mat + e);
        }
        for (int e = 0; e < cc; e++)
            V.stencil[(size_t)(slot * cc + e) * T + stencil_pos(tx, ty, tw_, th_)] = blk[e];
    }
    for (int i = 0; i < c; i++)
        V.grad[ti * c + i] = g[i];
}

// ---- reductions --------------------------------------------------------------------------------------------------

__device__ __forceinline__ double warp_sum(double v)
{
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_min(double v)
{
    for (int o = 16; o > 0; o >>= 1)
        v = fmin(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_max(double v)
{
    for (int o = 16; o > 0; o >>= 1)
        v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// Block-wide reduction of up to 3 values with a fixed shape (warp trees, then warps in order). kind: 0 sum, 1 min,
// 2 max. The result lands on thread 0.
template <int N>
__device__ __forceinline__ void block_reduce(double (&v)[N], const int (&kind)[N], double* sh)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int q = 0; q < N; q++)
        v[q] = kind[q] == 0 ? warp_sum(v[q]) : (kind[q] == 1 ? warp_min(v[q]) : warp_max(v[q]));
    __syncthreads();
    if (lane == 0)
        for (int q = 0; q < N; q++)
            sh[q * 32 + warp] = v[q];
    __syncthreads();
    if (threadIdx.x == 0)
        for (int q = 0; q < N; q++)
        {
            double s = sh[q * 32];
            for (int w = 1; w < nw; w++)
                s = kind[q] == 0 ? s + sh[q * 32 + w] : (kind[q] == 1 ? fmin(s, sh[q * 32 + w]) : fmax(s, sh[q * 32 + w]));
            v[q] = s;
        }
}

// The totals of ROWS rows of one plane's block partials, on every thread of a FOLD_THREADS block. Each row is folded
// by one warp in a fixed order - lane l adds partials l, l + 32, l + 64, ... of the plane, then the warp's tree - from
// shared memory, where the whole block stages the rows CHUNK partials at a time, the next chunk's loads in flight
// while this one is folded. A single warp walking the partials in global memory waited out one L2 latency per 32 of
// them: at 6 x 2048 x 2048 (21.8 k partials) the CG's two folds took 118 and 48 us an iteration; the chain of
// additions is now what bounds them.
constexpr int FOLD_THREADS = 256;

template <int ROWS>
__device__ __forceinline__ void plane_totals(const double* partial, size_t nblocks, long long b0, long long b1,
                                             const int (&row)[ROWS], const int (&kind)[ROWS], double (&out)[ROWS])
{
    constexpr int PER = ROWS < 3 ? 8 : 6, CHUNK = FOLD_THREADS * PER;   // within 48 KB of shared memory
    __shared__ double buf[ROWS][CHUNK];
    __shared__ double total[ROWS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long n = b1 - b0;
    double v[ROWS][PER];
    auto fetch = [&](long long at) {
#pragma unroll
        for (int q = 0; q < ROWS; q++)
#pragma unroll
            for (int i = 0; i < PER; i++)
            {
                const long long b = at + i * FOLD_THREADS + tid;
                v[q][i] = b < n ? __ldg(partial + (size_t)row[q] * nblocks + (size_t)(b0 + b)) : 0.0;
            }
    };
    int my_kind = 0;
#pragma unroll
    for (int q = 0; q < ROWS; q++)
        my_kind = warp == q ? kind[q] : my_kind;
    double s = my_kind == 0 ? 0.0 : (my_kind == 1 ? 1e300 : -1e300);
    fetch(0);
    for (long long at = 0; at < n; at += CHUNK)
    {
#pragma unroll
        for (int q = 0; q < ROWS; q++)
#pragma unroll
            for (int i = 0; i < PER; i++)
                buf[q][i * FOLD_THREADS + tid] = v[q][i];
        __syncthreads();
        fetch(at + CHUNK);
        if (warp < ROWS)
        {
            const int left = (int)(n - at < CHUNK ? n - at : CHUNK);
            const double* mine = buf[warp];
#pragma unroll 8
            for (int b = lane; b < left; b += 32)
            {
                const double x = mine[b];
                s = my_kind == 0 ? s + x : (my_kind == 1 ? fmin(s, x) : fmax(s, x));
            }
        }
        __syncthreads();
    }
    if (warp < ROWS)
    {
        s = my_kind == 0 ? warp_sum(s) : (my_kind == 1 ? warp_min(s) : warp_max(s));
        if (lane == 0)
            total[warp] = s;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < ROWS; q++)
        out[q] = total[q];
}

struct Red
{
    double* partial;      // [row][block]
    size_t nblocks;       // blocks of the launch (the row stride)
    double* scalars;      // [plane][S_COUNT]
};

// One coefficient of the stencil as stored: FP64 (the plain form) or FP32 (the adjoint form's quantised sweeps read a
// single-precision stencil, half the bytes), widened to double for the sums that read it.
template <typename TS>
__device__ __forceinline__ double sten(const PlaneView& V, size_t idx)
{
    return (double)reinterpret_cast<const TS*>(V.stencil)[idx];
}

// A texel's C x C block of slot `slot` (the texel at stencil position sp). An FP32 block of 16 (or 4) coefficients is
// read at once as 16-byte vector loads into registers; an FP64 block (and any other) is read a coefficient at a time
// where it is used, as the plain form always has (holding 16 doubles would cost its kernels occupancy).
template <int C, typename TS>
struct StenBlock
{
    static constexpr int cc = C * C;
    static constexpr bool vec = sizeof(TS) == sizeof(float) && cc % 4 == 0;
    float f[vec ? cc : 1];
    const TS* base;
    size_t T, sp;
    int slot;
    __device__ __forceinline__ StenBlock(const PlaneView& V, int slot_, size_t T_, size_t sp_)
        : base(reinterpret_cast<const TS*>(V.stencil)), T(T_), sp(sp_), slot(slot_)
    {
        if constexpr (vec)
        {
            const float4* q = reinterpret_cast<const float4*>(base + ((size_t)slot * T + sp) * cc);
#pragma unroll
            for (int v = 0; v < cc / 4; v++)
            {
                const float4 x = __ldg(q + v);
                f[4 * v] = x.x;
                f[4 * v + 1] = x.y;
                f[4 * v + 2] = x.z;
                f[4 * v + 3] = x.w;
            }
        }
    }
    __device__ __forceinline__ double operator[](int e) const
    {
        if constexpr (vec)
            return (double)f[e];
        else
            return (double)base[sten_index<TS>(slot, e, cc, T, sp)];
    }
};

// A texel's C consecutive doubles, as 16-byte accesses where they are whole vectors.
template <int C>
__device__ __forceinline__ void load_texel(const double* p, double* out)
{
    if constexpr (C % 2 == 0)
    {
#pragma unroll
        for (int q = 0; q < C / 2; q++)
        {
            const double2 v = reinterpret_cast<const double2*>(p)[q];
            out[2 * q] = v.x;
            out[2 * q + 1] = v.y;
        }
    }
    else
    {
#pragma unroll
        for (int q = 0; q < C; q++)
            out[q] = p[q];
    }
}
template <int C>
__device__ __forceinline__ void store_texel(double* p, const double* v)
{
    if constexpr (C % 2 == 0)
    {
#pragma unroll
        for (int q = 0; q < C / 2; q++)
            reinterpret_cast<double2*>(p)[q] = make_double2(v[2 * q], v[2 * q + 1]);
    }
    else
    {
#pragma unroll
        for (int q = 0; q < C; q++)
            p[q] = v[q];
    }
}

// ---- ridge, preconditioner ----------------------------------------------------------------------------------------

template <typename TS>
__global__ void __launch_bounds__(THREADS) k_diag(Planes P, Red R)
{
    __shared__ double sh[3 * 32];
    const long long base = (long long)blockIdx.x * blockDim.x;
    const int pl = plane_of(P, base);
    const PlaneView& V = P.p[pl];
    const long long t = base - P.start[pl] + threadIdx.x;
    const size_t T = (size_t)V.w * V.h;
    const int c = P.c;
    double v[3] = { 0.0, 1e300, -1e300 };
    const int kind[3] = { 0, 1, 2 };
    if (t < (long long)T)
        for (int a = 0; a < c; a++)
        {
            const double x = sten<TS>(V, sten_index<TS>(0, a * c + a, c * c, T, stencil_pos((int)(t % V.w), (int)(t / V.w), V.w, V.h)));
            v[0] += x;
            v[1] = x < v[1] ? x : v[1];
            v[2] = x > v[2] ? x : v[2];
        }
    block_reduce(v, kind, sh);
    if (threadIdx.x == 0)
        for (int q = 0; q < 3; q++)
            R.partial[(size_t)q * R.nblocks + blockIdx.x] = v[q];
}

__global__ void __launch_bounds__(FOLD_THREADS) k_diag_reduce(Planes P, Red R, double ridge)
{
    const int pl = blockIdx.x;
    const long long b0 = P.start[pl] / THREADS, b1 = P.start[pl + 1] / THREADS;
    double total[3];
    plane_totals<3>(R.partial, R.nblocks, b0, b1, { 0, 1, 2 }, { 0, 1, 2 }, total);
    if (threadIdx.x == 0)
    {
        const double sum = total[0], lo = total[1], hi = total[2];
        double* s = R.scalars + (size_t)pl * S_COUNT;
        const size_t unknowns = (size_t)P.p[pl].w * P.p[pl].h * P.c;
        s[S_DIAG_SUM] = sum;
        s[S_DIAG_MIN] = lo;
        s[S_DIAG_MAX] = hi;
        s[S_LAMBDA] = unknowns > 0 ? ridge * sum / (double)unknowns : 0.0;
    }
}

// Gauss-Jordan with partial pivoting on [a | I], n <= 4, in double (src/solve_level1.cu:689-740). Unrolled, a pivot row
// swapped in by selection: a row found at run time would put both matrices in local memory.
template <int n>
__device__ __forceinline__ bool invert(double (&a)[n * n], double (&inv)[n * n])
{
#pragma unroll
    for (int i = 0; i < n; i++)
#pragma unroll
        for (int j = 0; j < n; j++)
            inv[i * n + j] = i == j ? 1.0 : 0.0;
#pragma unroll
    for (int k = 0; k < n; k++)
    {
        int pivot = k;
        double best = fabs(a[k * n + k]);
#pragma unroll
        for (int i = k + 1; i < n; i++)
            if (fabs(a[i * n + k]) > best)
            {
                best = fabs(a[i * n + k]);
                pivot = i;
            }
        if (!(best > 0.0))
            return false;
#pragma unroll
        for (int i = k + 1; i < n; i++)
            if (pivot == i)
            {
#pragma unroll
                for (int j = 0; j < n; j++)
                {
                    double t = a[k * n + j];
                    a[k * n + j] = a[i * n + j];
                    a[i * n + j] = t;
                    t = inv[k * n + j];
                    inv[k * n + j] = inv[i * n + j];
                    inv[i * n + j] = t;
                }
            }
        const double s = 1.0 / a[k * n + k];
#pragma unroll
        for (int j = 0; j < n; j++)
        {
            a[k * n + j] *= s;
            inv[k * n + j] *= s;
        }
#pragma unroll
        for (int i = 0; i < n; i++)
        {
            if (i == k)
                continue;
            const double f = a[i * n + k];
            if (f == 0.0)
                continue;
#pragma unroll
            for (int j = 0; j < n; j++)
            {
                a[i * n + j] -= f * a[k * n + j];
                inv[i * n + j] -= f * inv[k * n + j];
            }
        }
    }
    return true;
}

__device__ __forceinline__ void apply_precond(const float* minv, const double* r, int c, double* z)
{
    for (int i = 0; i < c; i++)
    {
        double acc = 0.0;
        for (int j = 0; j < c; j++)
            acc += (double)minv[i * c + j] * r[j];
        z[i] = acc;
    }
}

// A neighbour's values in the product: whole vectors at four channels; at two the scalar loads measured faster (68
// against 77 us at 4 x 1024 x 1024: the vectors leave the compiler fewer loads in flight).
template <int C>
__device__ __forceinline__ void load_neighbour(const double* p, double* out)
{
    if constexpr (C == 4)
        load_texel<C>(p, out);
    else
    {
#pragma unroll
        for (int q = 0; q < C; q++)
            out[q] = p[q];
    }
}

// y_t = (H_tt + lambda I) x_t + sum of the owned slots' blocks times the forward neighbours + the transposes of the
// backward neighbours' blocks (src/solve_level1.cu:781-828), in the reference's order of accumulation.
template <int C, typename TS>
__device__ __forceinline__ void stencil_apply(const PlaneView& V, size_t T, long long t, double lambda, const double* x,
                                              double* acc)
{
    constexpr int cc = C * C;
    const int tx = (int)(t % V.w), ty = (int)(t / V.w);
    const size_t sp = stencil_pos(tx, ty, V.w, V.h);
    double xt[C];
    load_texel<C>(x + (size_t)t * C, xt);
    const StenBlock<C, TS> self(V, 0, T, sp);
#pragma unroll
    for (int i = 0; i < C; i++)
    {
        double s = lambda * xt[i];
#pragma unroll
        for (int j = 0; j < C; j++)
            s += self[i * C + j] * xt[j];
        acc[i] = s;
    }
    // Every neighbour's loads are issued whether or not the neighbour exists (from a clamped, in-range texel), and a
    // missing neighbour's products are replaced by -0.0, which leaves any sum, a signed zero included, exactly as it
    // was: the same bits as skipping those terms.
#pragma unroll
    for (int slot = 1; slot < SLOTS; slot++)
    {
        int dx, dy;
        slot_offset(slot, dx, dy);
        const int fx = tx + dx, fy = ty + dy;
        const bool fwd = fx >= 0 && fx < V.w && fy >= 0 && fy < V.h;
        const int gx = fwd ? fx : tx, gy = fwd ? fy : ty;
        double xn[C], xb[C];
        load_neighbour<C>(x + ((size_t)gy * V.w + gx) * C, xn);
        const StenBlock<C, TS> blk(V, slot, T, sp);
#pragma unroll
        for (int i = 0; i < C; i++)
#pragma unroll
            for (int j = 0; j < C; j++)
            {
                const double e = blk[i * C + j] * xn[j];
                acc[i] += fwd ? e : -0.0;
            }
        const int bx = tx - dx, by = ty - dy;
        const bool bwd = bx >= 0 && bx < V.w && by >= 0 && by < V.h;
        const int hx = bwd ? bx : tx, hy = bwd ? by : ty;
        const size_t nt = (size_t)hy * V.w + hx, np = stencil_pos(hx, hy, V.w, V.h);
        load_neighbour<C>(x + nt * C, xb);
        const StenBlock<C, TS> nbk(V, slot, T, np);
#pragma unroll
        for (int i = 0; i < C; i++)
#pragma unroll
            for (int j = 0; j < C; j++)
            {
                const double e = nbk[j * C + i] * xb[j];
                acc[i] += bwd ? e : -0.0;
            }
    }
}

// The channel count as a constant and every texel's values as whole vectors: scalar stores a texel apart wrote each
// sector of the five vectors and the preconditioner several times (5.0 GB of DRAM writes for 1.1 GB of results, 1915 us
// at 6 x 2048 x 2048).
template <int C, typename TS>
__global__ void __launch_bounds__(THREADS) k_precondition_init(Planes P, Red R)
{
    __shared__ double sh[2 * 32];
    const long long base = (long long)blockIdx.x * blockDim.x;
    const int pl = plane_of(P, base);
    const PlaneView& V = P.p[pl];
    const long long t = base - P.start[pl] + threadIdx.x;
    const size_t T = (size_t)V.w * V.h;
    constexpr int c = C;
    double v[2] = { 0.0, 0.0 };
    const int kind[2] = { 0, 0 };
    if (t < (long long)T)
    {
        const double lambda = R.scalars[(size_t)pl * S_COUNT + S_LAMBDA];
        double a[c * c], inv[c * c];
        const StenBlock<C, TS> self(V, 0, T, stencil_pos((int)(t % V.w), (int)(t / V.w), V.w, V.h));
#pragma unroll
        for (int i = 0; i < c; i++)
#pragma unroll
            for (int j = 0; j < c; j++)
                a[i * c + j] = self[i * c + j] + (i == j ? lambda : 0.0);
        const bool inverted = invert<C>(a, inv);
#pragma unroll
        for (int i = 0; i < c; i++)
#pragma unroll
            for (int j = 0; j < c; j++)
                inv[i * c + j] = inverted ? inv[i * c + j] : (i == j ? 1.0 : 0.0);
        float minv[c * c];
#pragma unroll
        for (int i = 0; i < c * c; i++)
            minv[i] = (float)inv[i];
        float* out = V.precond + (size_t)t * c * c;
        if constexpr (C % 2 == 0)
        {
#pragma unroll
            for (int i = 0; i < c * c / 4; i++)
                reinterpret_cast<float4*>(out)[i] =
                    make_float4(minv[4 * i], minv[4 * i + 1], minv[4 * i + 2], minv[4 * i + 3]);
        }
        else
        {
#pragma unroll
            for (int i = 0; i < c * c; i++)
                out[i] = minv[i];
        }
        // CG from d = 0: r = -grad, z = M r, p = z.
        double r[c], z[c], zero[c];
        load_texel<C>(V.grad + (size_t)t * c, r);
#pragma unroll
        for (int i = 0; i < c; i++)
        {
            r[i] = -r[i];
            zero[i] = 0.0;
        }
        store_texel<C>(V.x + (size_t)t * c, zero);
        store_texel<C>(V.r + (size_t)t * c, r);
        apply_precond(minv, r, c, z);
        store_texel<C>(V.z + (size_t)t * c, z);
        store_texel<C>(V.p + (size_t)t * c, z);
#pragma unroll
        for (int i = 0; i < c; i++)
        {
            v[0] += r[i] * r[i];
            v[1] += r[i] * z[i];
        }
    }
    block_reduce(v, kind, sh);
    if (threadIdx.x == 0)
    {
        R.partial[blockIdx.x] = v[0];
        R.partial[R.nblocks + blockIdx.x] = v[1];
    }
}

__global__ void __launch_bounds__(FOLD_THREADS) k_cg_start(Planes P, Red R)
{
    const int pl = blockIdx.x;
    const long long b0 = P.start[pl] / THREADS, b1 = P.start[pl + 1] / THREADS;
    double total[2];
    plane_totals<2>(R.partial, R.nblocks, b0, b1, { 0, 1 }, { 0, 0 }, total);
    if (threadIdx.x == 0)
    {
        double* s = R.scalars + (size_t)pl * S_COUNT;
        s[S_RHS2] = total[0];
        s[S_RZ] = total[1];
        s[S_ACTIVE] = 1.0;
        s[S_ITER] = 0.0;
        s[S_RESID] = 0.0;
    }
}

// The product with a thread per texel. PER_SM, the blocks an SM is to hold, weighs the loads a thread has in flight against
// the threads: an FP64 block of four channels needs the registers of three blocks an SM (four against three, us: 256 x 256
// 13.8 / 13.2, 1000 x 756 167 / 139, 2048 x 1024 428 / 355; two 524), two channels do with those of six (four against six:
// 256 x 256 6.06 / 5.92, 512 x 512 18.3 / 16.2, 2048 x 2048 236 / 211), three channels stay at four (1024 x 1024: three 133,
// four 106, five 117). A launch of at most a block an SM has nothing to hold more blocks with: two channels at 96 x 80 take
// 4.24 us at four and 4.57 at six.
template <int C, typename TS, int PER_SM = C == 4 ? 3 : 4>
__global__ void __launch_bounds__(THREADS, PER_SM) k_cg_matvec(Planes P, Red R)
{
    __shared__ double sh[32];
    const long long base = (long long)blockIdx.x * blockDim.x;
    const int pl = plane_of(P, base);
    const double* s = R.scalars + (size_t)pl * S_COUNT;
    if (s[S_ACTIVE] == 0.0)
        return;
    const PlaneView& V = P.p[pl];
    const long long t = base - P.start[pl] + threadIdx.x;
    const size_t T = (size_t)V.w * V.h;
    constexpr int c = C;
    double v[1] = { 0.0 };
    const int kind[1] = { 0 };
    if (t < (long long)T)
    {
        double acc[C], pt[C];
        stencil_apply<C, TS>(V, T, t, s[S_LAMBDA], V.p, acc);
        store_texel<C>(V.ap + (size_t)t * c, acc);
        load_texel<C>(V.p + (size_t)t * c, pt);
#pragma unroll
        for (int i = 0; i < c; i++)
            v[0] += pt[i] * acc[i];
    }
    block_reduce(v, kind, sh);
    if (threadIdx.x == 0)
        R.partial[blockIdx.x] = v[0];
}

// The product for an FP32 stencil of two or four channels with a lane per row (k_cg_matvec_rows): C lanes share a texel,
// lane i forms row i of the product - the same sums in the same order - and reads row i of each of the nine blocks as one
// vector, so that a warp's reads of a slot are contiguous runs. One thread per texel read each block's rows 64 bytes
// apart: the L1 served the same line four times, and that bound the kernel (97% of its wavefronts; 627 us at 6 x 2048 x
// 2048, against 330 us for its bytes; by rows 549 us, bound by the loads' latency: six blocks per SM, four take 690 us).
// A backward neighbour's transposed block is read by rows too where the blocks are symmetric bit for bit (symmetric
// != 0), else by columns. The FP64 stencil has a run per coefficient, which a thread per texel reads whole as it is.
template <int C>
__device__ __forceinline__ void load_row(const float* p, float (&r)[C])
{
    if constexpr (C == 4)
    {
        const float4 v = __ldg(reinterpret_cast<const float4*>(p));
        r[0] = v.x;
        r[1] = v.y;
        r[2] = v.z;
        r[3] = v.w;
    }
    else
    {
        const float2 v = __ldg(reinterpret_cast<const float2*>(p));
        r[0] = v.x;
        r[1] = v.y;
    }
}

// A texel's place among its neighbours, in 32-bit indices: the stencil positions of a row's even and odd texels (the
// colour-major order of stencil_pos) for its own row and the one above.
struct TexelPlace
{
    int tx, ty, t;               // column, row, row-major index
    unsigned even, odd;          // this row: position of texel x is (x & 1 ? odd : even) + x / 2
    unsigned even_up, odd_up;    // the row above (this row where there is none)
    __device__ __forceinline__ TexelPlace(int x, int y, int w, int h) : tx(x), ty(y), t(y * w + x)
    {
        const unsigned w0c = (unsigned)(w + 1) >> 1, w1c = (unsigned)w >> 1, h0c = (unsigned)(h + 1) >> 1;
        const unsigned h1c = (unsigned)h >> 1, odd_rows = (unsigned)w * h0c;
        auto row = [&](int r, unsigned& e, unsigned& o) {
            const unsigned half = (unsigned)r >> 1;
            e = (r & 1 ? odd_rows : 0u) + half * w0c;
            o = (r & 1 ? odd_rows + w0c * h1c : w0c * h0c) + half * w1c;
        };
        row(y, even, odd);
        row(y > 0 ? y - 1 : y, even_up, odd_up);
    }
    __device__ __forceinline__ unsigned at(int x) const { return (x & 1 ? odd : even) + ((unsigned)x >> 1); }
    __device__ __forceinline__ unsigned above(int x) const { return (x & 1 ? odd_up : even_up) + ((unsigned)x >> 1); }
};

// Row i of the four owned blocks times the forward neighbours plus the four backward neighbours' transposed blocks,
// added to acc in the order of stencil_apply. Every load is issued, a missing neighbour's from the texel itself, whose
// products are replaced by -0.0.
template <int C>
__device__ __forceinline__ void neighbour_rows(const PlaneView& V, unsigned T, const TexelPlace& at, int i, const double* x,
                                               int symmetric, double& acc)
{
    constexpr int cc = C * C;
    const float* S = reinterpret_cast<const float*>(V.stencil);
    const int w = V.w;
    const bool left = at.tx > 0, right = at.tx + 1 < w, up = at.ty > 0, down = at.ty + 1 < V.h;
    const unsigned sp = at.at(at.tx);
    // slots 1..4: right, down-left, down, down-right; backward: left, up-right, up, up-left
    const bool fwd[4] = { right, down && left, down, down && right }, bwd[4] = { left, up && right, up, up && left };
    const int ahead[4] = { 1, w - 1, w, w + 1 };
    const unsigned back[4] = { left ? at.at(at.tx - 1) : sp, up && right ? at.above(at.tx + 1) : sp,
                               up ? at.above(at.tx) : sp, up && left ? at.above(at.tx - 1) : sp };
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
        double xn[C], xb[C];
        float own[C], other[C];
        load_texel<C>(x + (size_t)(at.t + (fwd[q] ? ahead[q] : 0)) * C, xn);
        load_texel<C>(x + (size_t)(at.t - (bwd[q] ? ahead[q] : 0)) * C, xb);
        const float* slot = S + (size_t)(q + 1) * T * cc;
        load_row<C>(slot + (size_t)sp * cc + i * C, own);
        const float* nb = slot + (size_t)back[q] * cc;
        if (symmetric)
            load_row<C>(nb + i * C, other);
        else
        {
#pragma unroll
            for (int j = 0; j < C; j++)
                other[j] = __ldg(nb + j * C + i);
        }
#pragma unroll
        for (int j = 0; j < C; j++)
        {
            const double e = (double)own[j] * xn[j];
            acc += fwd[q] ? e : -0.0;
        }
#pragma unroll
        for (int j = 0; j < C; j++)
        {
            const double e = (double)other[j] * xb[j];
            acc += bwd[q] ? e : -0.0;
        }
    }
}

template <int C>
__global__ void __launch_bounds__(THREADS, 6) k_cg_matvec_rows(Planes P, Red R, int symmetric)
{
    __shared__ double sh[32];
    __shared__ double dot[THREADS];
    const long long base = (long long)blockIdx.x * blockDim.x;
    const int pl = plane_of(P, base);
    const double* s = R.scalars + (size_t)pl * S_COUNT;
    if (s[S_ACTIVE] == 0.0)
        return;
    const PlaneView& V = P.p[pl];
    const long long t0 = base - P.start[pl];
    const size_t T = (size_t)V.w * V.h;
    const double lambda = s[S_LAMBDA];
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int q = 0; q < C; q++)
    {
        const int local = (q * THREADS + (int)threadIdx.x) / C, i = (int)threadIdx.x % C;
        const long long t = t0 + local;
        double acc = 0.0, pq = 0.0;
        if (t < (long long)T)
        {
            const unsigned row = (unsigned)t / (unsigned)V.w;
            const TexelPlace at((int)((unsigned)t - row * (unsigned)V.w), (int)row, V.w, V.h);
            double xt[C];
            load_texel<C>(V.p + (size_t)t * C, xt);
            float self[C];
            load_row<C>(reinterpret_cast<const float*>(V.stencil) + (size_t)at.at(at.tx) * C * C + i * C, self);
#pragma unroll
            for (int j = 0; j < C; j++)
                pq = j == i ? xt[j] : pq;
            acc = lambda * pq;
#pragma unroll
            for (int j = 0; j < C; j++)
                acc += (double)self[j] * xt[j];
            neighbour_rows<C>(V, (unsigned)T, at, i, V.p, symmetric, acc);
            V.ap[(size_t)t * C + i] = acc;
        }
        // the texel's share of <p, Ap>, channel by channel
        const double e = pq * acc;
        double sum = 0.0;
#pragma unroll
        for (int j = 0; j < C; j++)
            sum += __shfl_sync(0xffffffffu, e, (lane & ~(C - 1)) + j);
        if (i == 0)
            dot[local] = sum;
    }
    __syncthreads();
    double v[1] = { dot[threadIdx.x] };
    const int kind[1] = { 0 };
    block_reduce(v, kind, sh);
    if (threadIdx.x == 0)
        R.partial[blockIdx.x] = v[0];
}

// alpha; block 0 also clears the count of planes that stay active, which k_cg_beta of this iteration adds up.
__global__ void __launch_bounds__(FOLD_THREADS) k_cg_alpha(Planes P, Red R, unsigned int* active_count)
{
    const int pl = blockIdx.x;
    double* s = R.scalars + (size_t)pl * S_COUNT;
    if (pl == 0 && threadIdx.x == 0)
        *active_count = 0;
    if (s[S_ACTIVE] == 0.0)
        return;
    const long long b0 = P.start[pl] / THREADS, b1 = P.start[pl + 1] / THREADS;
    double total[1];
    plane_totals<1>(R.partial, R.nblocks, b0, b1, { 0 }, { 0 }, total);
    if (threadIdx.x == 0)
    {
        const double pap = total[0];
        s[S_PAP] = pap;
        s[S_ALPHA] = pap > 0.0 ? s[S_RZ] / pap : 0.0;
    }
}

template <int C>
__global__ void __launch_bounds__(THREADS) k_cg_update(Planes P, Red R)
{
    __shared__ double sh[2 * 32];
    const long long base = (long long)blockIdx.x * blockDim.x;
    const int pl = plane_of(P, base);
    const double* s = R.scalars + (size_t)pl * S_COUNT;
    if (s[S_ACTIVE] == 0.0)
        return;
    const PlaneView& V = P.p[pl];
    const long long t = base - P.start[pl] + threadIdx.x;
    const size_t T = (size_t)V.w * V.h;
    constexpr int c = C;   // the channel count as a constant: r, z and the preconditioner stay in registers
    double v[2] = { 0.0, 0.0 };
    const int kind[2] = { 0, 0 };
    if (t < (long long)T)
    {
        const double alpha = s[S_ALPHA];
        double r[MAX_CH], z[MAX_CH];
#pragma unroll
        for (int i = 0; i < c; i++)
        {
            const size_t q = (size_t)t * c + i;
            V.x[q] += 1.0 * alpha * V.p[q];
            r[i] = V.r[q] + -1.0 * alpha * V.ap[q];
            V.r[q] = r[i];
        }
        float minv[MAX_CH * MAX_CH];
#pragma unroll
        for (int i = 0; i < c * c; i++)
            minv[i] = V.precond[(size_t)t * c * c + i];
#pragma unroll
        for (int i = 0; i < c; i++)
        {
            double acc = 0.0;
#pragma unroll
            for (int j = 0; j < c; j++)
                acc += (double)minv[i * c + j] * r[j];
            z[i] = acc;
        }
#pragma unroll
        for (int i = 0; i < c; i++)
        {
            V.z[(size_t)t * c + i] = z[i];
            v[0] += r[i] * r[i];
            v[1] += r[i] * z[i];
        }
    }
    block_reduce(v, kind, sh);
    if (threadIdx.x == 0)
    {
        R.partial[blockIdx.x] = v[0];
        R.partial[R.nblocks + blockIdx.x] = v[1];
    }
}

// k_cg_update for one, two or four channels with a lane per value: every vector is read and written in whole lines and
// lane i applies row i of the preconditioner to the texel's residuals, exchanged within the C lanes; the texels' sums go
// through shared memory to the block's reduction of one thread per texel. One thread per texel read each vector a texel
// apart (91% of the L1's wavefronts, 358 us at 6 x 2048 x 2048). Three channels, whose lanes would straddle warps, keep it.
template <int C>
__global__ void __launch_bounds__(THREADS) k_cg_update_rows(Planes P, Red R)
{
    __shared__ double sh[2 * 32];
    __shared__ double sums[2][THREADS];
    const long long base = (long long)blockIdx.x * blockDim.x;
    const int pl = plane_of(P, base);
    const double* s = R.scalars + (size_t)pl * S_COUNT;
    if (s[S_ACTIVE] == 0.0)
        return;
    const PlaneView& V = P.p[pl];
    const long long t0 = base - P.start[pl];
    const size_t T = (size_t)V.w * V.h;
    const double alpha = s[S_ALPHA];
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < C; q++)
    {
        const int local = (q * THREADS + (int)threadIdx.x) / C, i = (int)threadIdx.x % C;
        double r = 0.0, z = 0.0;
        float minv[C] = {};
        const size_t e = (size_t)t0 * C + q * THREADS + threadIdx.x;
        const bool ok = t0 + local < (long long)T;
        if (ok)
        {
            V.x[e] += 1.0 * alpha * V.p[e];
            r = V.r[e] + -1.0 * alpha * V.ap[e];
            V.r[e] = r;
            if constexpr (C == 1)
                minv[0] = V.precond[e];
            else
                load_row<C>(V.precond + e * C, minv);
        }
#pragma unroll
        for (int j = 0; j < C; j++)
            z += (double)minv[j] * __shfl_sync(0xffffffffu, r, (lane & ~(C - 1)) + j);
        if (ok)
            V.z[e] = z;
        const double rr = r * r, rz = r * z;
        double srr = 0.0, srz = 0.0;
#pragma unroll
        for (int j = 0; j < C; j++)
        {
            srr += __shfl_sync(0xffffffffu, rr, (lane & ~(C - 1)) + j);
            srz += __shfl_sync(0xffffffffu, rz, (lane & ~(C - 1)) + j);
        }
        if (i == 0)
        {
            sums[0][local] = srr;
            sums[1][local] = srz;
        }
    }
    __syncthreads();
    double v[2] = { sums[0][threadIdx.x], sums[1][threadIdx.x] };
    const int kind[2] = { 0, 0 };
    block_reduce(v, kind, sh);
    if (threadIdx.x == 0)
    {
        R.partial[blockIdx.x] = v[0];
        R.partial[R.nblocks + blockIdx.x] = v[1];
    }
}

// beta, the residual, and the device-side stop: at an iteration that is a multiple of CG_PROBE a plane whose residual
// is not at or above the tolerance leaves (the reference's host probe, src/solve_level1.cu:1288-1302): its direction
// is not updated again, which nothing reads.
__global__ void __launch_bounds__(FOLD_THREADS) k_cg_beta(Planes P, Red R, int it, unsigned int* active_count, double tol)
{
    const int pl = blockIdx.x;
    double* s = R.scalars + (size_t)pl * S_COUNT;
    if (s[S_ACTIVE] == 0.0)
        return;
    const long long b0 = P.start[pl] / THREADS, b1 = P.start[pl + 1] / THREADS;
    double total[2];
    plane_totals<2>(R.partial, R.nblocks, b0, b1, { 0, 1 }, { 0, 0 }, total);
    if (threadIdx.x == 0)
    {
        const double rr = total[0], rz_new = total[1];
        const double rz = s[S_RZ];
        s[S_RR] = rr;
        s[S_RZ_NEW] = rz_new;
        s[S_BETA] = rz != 0.0 ? rz_new / rz : 0.0;
        s[S_RZ] = rz_new;
        const double rhs2 = s[S_RHS2];
        s[S_RESID] = rhs2 > 0.0 ? sqrt((rr > 0.0 ? rr : 0.0) / rhs2) : 0.0;
        s[S_ITER] = (double)(it + 1);
        if ((it + 1) % CG_PROBE == 0 && !(s[S_RESID] >= tol))
            s[S_ACTIVE] = 0.0;
        else
            atomicAdd(active_count, 1u);
    }
}

__global__ void __launch_bounds__(THREADS) k_cg_direction(Planes P, Red R)
{
    const long long base = (long long)blockIdx.x * blockDim.x;
    const int pl = plane_of(P, base);
    const double* s = R.scalars + (size_t)pl * S_COUNT;
    if (s[S_ACTIVE] == 0.0)
        return;
    const PlaneView& V = P.p[pl];
    // the block's texels' values, a value a thread: whole lines
    const size_t first = (size_t)(base - P.start[pl]) * P.c, end = (size_t)V.w * V.h * P.c;
    const double beta = s[S_BETA];
    for (int i = 0; i < P.c; i++)
    {
        const size_t q = first + (size_t)i * THREADS + threadIdx.x;
        if (q < end)
            V.p[q] = V.z[q] + beta * V.p[q];
    }
}

// ---- the correction and the movement probe (src/solve_level1.cu:872-979) -------------------------------------------

__global__ void __launch_bounds__(THREADS) k_correct_range(Planes P, Red R)
{
    __shared__ double sh[2 * MAX_CH * 32];
    const long long base = (long long)blockIdx.x * blockDim.x;
    const int pl = plane_of(P, base);
    const PlaneView& V = P.p[pl];
    const long long t = base - P.start[pl] + threadIdx.x;
    const size_t T = (size_t)V.w * V.h;
    const int c = P.c;
    double v[2 * MAX_CH];
    int kind[2 * MAX_CH];
    for (int q = 0; q < MAX_CH; q++)
    {
        v[q] = 1e300;
        v[MAX_CH + q] = -1e300;
        kind[q] = 1;
        kind[MAX_CH + q] = 2;
    }
    if (t < (long long)T)
        for (int i = 0; i < c; i++)
        {
            const size_t q = (size_t)t * c + i;
            const float nv = (float)((double)V.v[q] + V.x[q]);
            V.v[q] = nv;
            v[i] = (double)nv;
            v[MAX_CH + i] = (double)nv;
        }
    block_reduce(v, kind, sh);
    if (threadIdx.x == 0)
        for (int q = 0; q < c; q++)
        {
            R.partial[(size_t)(3 + q) * R.nblocks + blockIdx.x] = v[q];
            R.partial[(size_t)(3 + MAX_CH + q) * R.nblocks + blockIdx.x] = v[MAX_CH + q];
        }
}

// One block per plane and channel (grid.y).
__global__ void __launch_bounds__(FOLD_THREADS) k_range_reduce(Planes P, Red R)
{
    const int pl = blockIdx.x, q = blockIdx.y;
    const long long b0 = P.start[pl] / THREADS, b1 = P.start[pl + 1] / THREADS;
    double total[2];
    plane_totals<2>(R.partial, R.nblocks, b0, b1, { 3 + q, 3 + MAX_CH + q }, { 1, 2 }, total);
    if (threadIdx.x == 0)
    {
        R.scalars[(size_t)pl * S_COUNT + S_LO + q] = total[0];
        R.scalars[(size_t)pl * S_COUNT + S_HI + q] = total[1];
    }
}

__global__ void __launch_bounds__(THREADS) k_movement(Planes P, Red R, int levels)
{
    __shared__ double sh[3 * 32];
    const long long base = (long long)blockIdx.x * blockDim.x;
    const int pl = plane_of(P, base);
    const PlaneView& V = P.p[pl];
    const double* s = R.scalars + (size_t)pl * S_COUNT;
    const long long t = base - P.start[pl] + threadIdx.x;
    const size_t T = (size_t)V.w * V.h;
    const int c = P.c;
    double v[3] = { 0.0, 0.0, 0.0 };
    const int kind[3] = { 0, 0, 0 };
    if (t < (long long)T)
        for (int i = 0; i < c; i++)
        {
            const size_t q = (size_t)t * c + i;
            const double step = (s[S_HI + i] - s[S_LO + i]) / (double)levels;
            const double dq = V.x[q];
            if (fabs(dq) > 0.5 * step)
                v[0] += 1.0;
            v[1] += dq * dq;
            v[2] += (double)V.v[q] * (double)V.v[q];
        }
    block_reduce(v, kind, sh);
    if (threadIdx.x == 0)
        for (int q = 0; q < 3; q++)
            R.partial[(size_t)q * R.nblocks + blockIdx.x] = v[q];
}

__global__ void __launch_bounds__(FOLD_THREADS) k_movement_reduce(Planes P, Red R)
{
    const int pl = blockIdx.x;
    const long long b0 = P.start[pl] / THREADS, b1 = P.start[pl + 1] / THREADS;
    double total[3];
    plane_totals<3>(R.partial, R.nblocks, b0, b1, { 0, 1, 2 }, { 0, 0, 0 }, total);
    if (threadIdx.x == 0)
    {
        double* s = R.scalars + (size_t)pl * S_COUNT;
        s[S_MOVED] = total[0];
        s[S_DELTA2] = total[1];
        s[S_PLANE2] = total[2];
    }
}

// ---- the quantised phase (src/solve_level1.cu:1023-1098) ----------------------------------------------------------

// The fractions rep(k) / 255 of a grid's values, formed once per block: grid_index and grid_value divide by 255 for each
// of the values they look at, four divisions a channel that nothing but the index decides.
constexpr int GRID_FRACTIONS = 256;
__device__ __forceinline__ void grid_fractions(double* frac, int bits)
{
    for (int k = threadIdx.x; k < (1 << bits); k += blockDim.x)
        frac[k] = (double)rep_index(k, bits) / 255.0;
}

// grid_index and the value of the index it finds, from the block's fractions: the same bits.
__device__ __forceinline__ int grid_nearest(float lo, float hi, int bits, float value, const double* frac, float& nearest)
{
    const double span = (double)hi - (double)lo;
    const int levels = (1 << bits) - 1;
    auto at = [&](int k) { return (float)__dadd_rn((double)lo, __dmul_rn(frac[k], span)); };
    int best = 0;
    if (span > 0.0)
    {
        double x = ((double)value - (double)lo) / span * (double)levels;
        x = x < 0.0 ? 0.0 : (x > (double)levels ? (double)levels : x);
        int k = (int)(x + 0.5);
        k = k < 0 ? 0 : (k > levels ? levels : k);
        best = k;
        double best_d = fabs((double)value - (double)at(k));
#pragma unroll
        for (int d = -1; d <= 1; d += 2)
        {
            const int n = k + d;
            if (n < 0 || n > levels)
                continue;
            const double dist = fabs((double)value - (double)at(n));
            if (dist < best_d || (dist == best_d && n < best))
            {
                best_d = dist;
                best = n;
            }
        }
    }
    nearest = at(best);
    return best;
}

struct ColourArgs
{
    const double* scalars;
    const float* lo;
    const float* hi;
    int bits;
    int cx, cy;
    int symmetric;         // the FP32 stencil's blocks are symmetric bit for bit
    unsigned int* moved;   // [plane]
};

// One colour of one sweep: the texels' couplings to their eight neighbours, then each texel's channels in turn. With an
// FP32 stencil of two or four channels the couplings are formed a lane per row (neighbour_rows) and handed to the
// texels' threads through shared memory, so that the stencil is read in whole lines; with an FP64 stencil (a plane of
// doubles per coefficient) a thread per texel already reads whole lines. The texel's own values are whole vectors.
// PER_SM: the blocks an SM is to hold, 0 for as many as the compiler's own choice of registers leaves (an explicit 1 lets
// it take 202 in FP64 where it takes 64: 6.2 -> 8.1 ms for the sweeps of 4 x 2048 x 1024). Each block waits out the same chain of loads, so a launch takes its waves of blocks
// times that: with an FP32 stencil of four channels about 21 us a wave at three blocks an SM (76 registers) and 27 at
// four (64, 48 bytes spilled). colour_per_sm takes the one whose waves hold fewer blocks (us a launch, three against four:
// 426 blocks 23.0 / 24.7, 583 blocks 41.7 / 30.7, 699 blocks 45.5 / 50.2, 984 blocks 65.8 / 57.7, 1365 blocks 83.0 / 79.4,
// 1930 blocks 111.3 / 109.6, 2730 blocks 147.2 / 138.2; the line misses two in a hundred at 1930).
constexpr int colour_per_sm(int blocks)
{
    constexpr int SMS = 148;
    return 4 * ((blocks + 4 * SMS - 1) / (4 * SMS)) <= 3 * ((blocks + 3 * SMS - 1) / (3 * SMS)) ? 4 : 3;
}

template <int C, typename TS, int PER_SM = 0>
__global__ void __launch_bounds__(THREADS, PER_SM) k_quant_colour(Planes P, ColourArgs A)
{
    constexpr bool ROWS = sizeof(TS) == sizeof(float) && C % 2 == 0;
    __shared__ __align__(16) double coupling[ROWS ? THREADS * C : 1];
    // (an FP64 stencil's kernel has no barrier to hide the fractions' set-up behind: with it 183 -> 201 us a colour)
    __shared__ double frac[ROWS ? GRID_FRACTIONS : 1];
    if (ROWS)
        grid_fractions(frac, A.bits);
    const long long base = (long long)blockIdx.x * blockDim.x;
    const int pl = plane_of(P, base);
    const PlaneView& V = P.p[pl];
    const int cwn = (V.w - A.cx + 1) / 2, chn = (V.h - A.cy + 1) / 2;
    const long long ci0 = base - P.start[pl], ci = ci0 + threadIdx.x, n = (long long)cwn * chn;
    const size_t T = (size_t)V.w * V.h;
    constexpr int c = C, cc = C * C;
    double nb[C];
#pragma unroll
    for (int i = 0; i < c; i++)
        nb[i] = 0.0;
    if constexpr (ROWS)
    {
#pragma unroll 1
        for (int q = 0; q < C; q++)
        {
            const long long at = ci0 + (q * THREADS + (int)threadIdx.x) / C;
            double acc = 0.0;
            if (at < n)
            {
                const unsigned row = (unsigned)at / (unsigned)cwn;
                const TexelPlace place(A.cx + 2 * (int)((unsigned)at - row * (unsigned)cwn), A.cy + 2 * (int)row, V.w, V.h);
                neighbour_rows<C>(V, (unsigned)T, place, (int)threadIdx.x % C, V.x, A.symmetric, acc);
            }
            coupling[q * THREADS + threadIdx.x] = acc;
        }
        __syncthreads();   // the fractions and the couplings
        load_texel<C>(coupling + threadIdx.x * C, nb);
    }
    if (ci >= n)
        return;
    const int tx = A.cx + 2 * (int)((unsigned)ci % (unsigned)cwn);
    const int ty = A.cy + 2 * (int)((unsigned)ci / (unsigned)cwn);
    const size_t t = (size_t)ty * V.w + tx;
    const size_t sp = stencil_pos(tx, ty, V.w, V.h);
    const double lambda = A.scalars[(size_t)pl * S_COUNT + S_LAMBDA];
    if constexpr (!ROWS)
    {
        // as in stencil_apply: every load issued, a missing neighbour's products replaced by -0.0 (an exact no-op)
#pragma unroll
        for (int slot = 1; slot < SLOTS; slot++)
        {
            int dx, dy;
            slot_offset(slot, dx, dy);
            const int fx = tx + dx, fy = ty + dy;
            const bool fwd = fx >= 0 && fx < V.w && fy >= 0 && fy < V.h;
            const int gx = fwd ? fx : tx, gy = fwd ? fy : ty;
            double xn[C], xb[C];
            load_texel<C>(V.x + ((size_t)gy * V.w + gx) * c, xn);
            const StenBlock<C, TS> blk(V, slot, T, sp);
#pragma unroll
            for (int i = 0; i < c; i++)
#pragma unroll
                for (int j = 0; j < c; j++)
                {
                    const double e = blk[i * c + j] * xn[j];
                    nb[i] += fwd ? e : -0.0;
                }
            const int bx = tx - dx, by = ty - dy;
            const bool bwd = bx >= 0 && bx < V.w && by >= 0 && by < V.h;
            const int hx = bwd ? bx : tx, hy = bwd ? by : ty;
            const size_t nt = (size_t)hy * V.w + hx, np = stencil_pos(hx, hy, V.w, V.h);
            load_texel<C>(V.x + nt * c, xb);
            const StenBlock<C, TS> nbk(V, slot, T, np);
#pragma unroll
            for (int i = 0; i < c; i++)
#pragma unroll
                for (int j = 0; j < c; j++)
                {
                    const double e = nbk[j * c + i] * xb[j];
                    nb[i] += bwd ? e : -0.0;
                }
        }
    }
    const StenBlock<C, TS> self(V, 0, T, sp);
    double x[C], grad[C];
    float prev[C];
    load_texel<C>(V.x + t * c, x);
    load_texel<C>(V.grad + t * c, grad);
    load_channels<C>(V.prev + t * c, prev);
    unsigned int changed = 0;
#pragma unroll
    for (int q = 0; q < c; q++)
    {
        const size_t idx = t * c + q;
        const float l = A.lo[q], span = A.hi[q] - A.lo[q];
        const double a = self[q * c + q] + lambda;
        if (!(a > 0.0) || !(span > 0.0f))
            continue;
        double rest = nb[q];
#pragma unroll
        for (int j = 0; j < c; j++)
            if (j != q)
                rest += self[q * c + j] * x[j];
        const double b = grad[q] + rest;
        const double want = (double)prev[q] - b / a;
        float value;
        int kk;
        if constexpr (ROWS)
            kk = grid_nearest(l, A.hi[q], A.bits, (float)want, frac, value);
        else
        {
            kk = grid_index(l, A.hi[q], A.bits, (float)want);
            value = grid_value(l, A.hi[q], A.bits, kk);
        }
        if ((int)V.k[idx] != kk)
        {
            V.k[idx] = (uint8_t)kk;
            changed++;
        }
        V.v[idx] = value;
        x[q] = (double)value - (double)prev[q];
    }
    // a channel that stayed out of the step keeps its correction: stored as it was read
    store_texel<C>(V.x + t * c, x);
    if (changed)
        atomicAdd(A.moved + pl, changed);
}

// A whole sweep, its four colours in order, in one launch, for planes of at most a tile an SM. A block takes a tile of
// SWEEP_W x SWEEP_H texels, holds the corrections of the tile and a margin in shared memory, and takes the colours one
// after another; what a later colour of the tile needs of the texels outside it is computed by the block itself, from the
// corrections before the sweep, so that every texel's step has exactly the inputs it has in four launches of one colour each,
// and blocks need not wait on one another. Across, colour 3 reads colour 2 one texel out, that colour 1 and that colour 0:
// colour 0 goes three texels out, colour 1 two, colour 2 one. Down, a tile starts and ends between an odd row and an even one:
// its rows of colours 2 and 3 read colours 0 and 1 in the row below it and nothing else that is new, and none reads above.
// The corrections are read from one vector and written to another (x and r in turn), and a tile's own texels alone are
// written.
//
// Where the line lies: a colour of few texels is a launch whose threads each wait out the same loads and divisions, so four
// of them in one launch save three rounds of that (1 x 256 x 256, level 1: 49 -> 32 us a sweep, level 0: 26 -> 17 us; 1 x
// 100 x 76: 58 -> 26 us). With more tiles than SMs the tiles' second wave costs as much again (175 k level-1 texels: 71
// against 35 us), and at level 0 of 4 x 2048 x 1024 the colours side by side, at four blocks an SM, read a quarter less from
// DRAM and still took 675 against 560 us (FP64: 1314 against 732 us), waiting at the colours' barriers.
constexpr int SWEEP_W = 32, SWEEP_H = 28, SWEEP_MARGIN_X = 4, SWEEP_MARGIN_Y = 2;   // (even: a cell's colour is its texel's)
constexpr int SWEEP_COLS = (SWEEP_W + 2 * SWEEP_MARGIN_X) / 2, SWEEP_ROWS = (SWEEP_H + 2 * SWEEP_MARGIN_Y) / 2;   // a colour's
constexpr int SWEEP_CELLS = SWEEP_COLS * SWEEP_ROWS;
constexpr int SWEEP_TILES = 148;
// Threads: a colour's texels in one pass (FP64), or its rows in two or three (FP32).
template <typename TS>
constexpr int SWEEP_THREADS = sizeof(TS) == sizeof(float) ? 512 : 320;

struct SweepArgs
{
    const double* scalars;
    const float* lo;
    const float* hi;
    int bits;
    int symmetric;         // the FP32 stencil's blocks are symmetric bit for bit
    int first;             // the first sweep: the corrections are zero
    int to_r;              // the corrections go to r and come from x, else the other way round
    int bend[MAX_PLANES];  // one past each plane's last block, the planes in descending order
    int btiles[MAX_PLANES];
    unsigned int* moved;   // [plane]
};

// The corrections of the tile and its margin: [pair of channels][colour][row][column].
template <int C>
struct TileX
{
    static constexpr int PAIRS = (C + 1) / 2;
    double2* cells;
    __device__ __forceinline__ int at(int rx, int ry) const
    {
        return ((rx & 1) + 2 * (ry & 1)) * SWEEP_CELLS + (ry >> 1) * SWEEP_COLS + (rx >> 1);
    }
    __device__ __forceinline__ void get(int rx, int ry, double* out) const
    {
        const int i = at(rx, ry);
#pragma unroll
        for (int q = 0; q < PAIRS; q++)
        {
            const double2 v = cells[q * 4 * SWEEP_CELLS + i];
            out[2 * q] = v.x;
            if (2 * q + 1 < C)
                out[2 * q + 1] = v.y;
        }
    }
    __device__ __forceinline__ void set(int rx, int ry, const double* v) const
    {
        const int i = at(rx, ry);
#pragma unroll
        for (int q = 0; q < PAIRS; q++)
            cells[q * 4 * SWEEP_CELLS + i] = make_double2(v[2 * q], 2 * q + 1 < C ? v[2 * q + 1] : 0.0);
    }
};

template <int C, typename TS, int COLOUR>
__device__ __forceinline__ unsigned sweep_colour(const PlaneView& V, const SweepArgs& A, double lambda, int x0, int y0,
                                                 const TileX<C>& X, const double* frac, double* coupling, double* xout)
{
    constexpr bool ROWS = sizeof(TS) == sizeof(float) && C % 2 == 0;
    constexpr int cx = COLOUR & 1, cy = COLOUR >> 1, cc = C * C;
    // this colour's texels of the tile and as far outside it as the later colours read
    constexpr int hx = COLOUR == 0 ? 3 : (COLOUR == 1 ? 2 : (COLOUR == 2 ? 1 : 0));
    constexpr int rx0 = SWEEP_MARGIN_X - hx + ((SWEEP_MARGIN_X - hx) % 2 != cx), ry0 = SWEEP_MARGIN_Y + cy;
    constexpr int nx = (SWEEP_MARGIN_X + SWEEP_W - 1 + hx - rx0) / 2 + 1, ny = SWEEP_H / 2 + (cy == 0 ? 1 : 0);
    static_assert(SWEEP_H % 2 == 0 && SWEEP_W % 2 == 0, "tiles start at even texels");
    constexpr int TASKS = nx * ny;
    const int w = V.w, h = V.h;
    const size_t T = (size_t)w * h;
    unsigned changed = 0;
#pragma unroll 1
    for (int batch = 0; batch < TASKS; batch += SWEEP_THREADS<TS>)
    {
        if constexpr (ROWS)
        {
            const float* S = reinterpret_cast<const float*>(V.stencil);
#pragma unroll 1
            for (int q = 0; q < C; q++)
            {
                const int task = batch + (q * SWEEP_THREADS<TS> + (int)threadIdx.x) / C, i = (int)threadIdx.x % C;
                const int rx = rx0 + 2 * (task % nx), ry = ry0 + 2 * (task / nx);
                const int gx = x0 - SWEEP_MARGIN_X + rx, gy = y0 - SWEEP_MARGIN_Y + ry;
                double acc = 0.0;
                if (task < TASKS && gx >= 0 && gx < w && gy >= 0 && gy < h)
                {
                    const TexelPlace at(gx, gy, w, h);
                    const bool left = gx > 0, right = gx + 1 < w, up = gy > 0, down = gy + 1 < h;
                    const unsigned sp = at.at(gx);
                    // slots 1..4: right, down-left, down, down-right; backward: left, up-right, up, up-left
                    const bool fwd[4] = { right, down && left, down, down && right };
                    const bool bwd[4] = { left, up && right, up, up && left };
                    const unsigned back[4] = { left ? at.at(gx - 1) : sp, up && right ? at.above(gx + 1) : sp,
                                               up ? at.above(gx) : sp, up && left ? at.above(gx - 1) : sp };
#pragma unroll
                    for (int d = 0; d < 4; d++)
                    {
                        int dx, dy;
                        slot_offset(d + 1, dx, dy);
                        float own[C], other[C];
                        const float* slot = S + (size_t)(d + 1) * T * cc;
                        load_row<C>(slot + (size_t)sp * cc + i * C, own);
                        const float* nb = slot + (size_t)back[d] * cc;
                        if (A.symmetric)
                            load_row<C>(nb + i * C, other);
                        else
                        {
#pragma unroll
                            for (int j = 0; j < C; j++)
                                other[j] = __ldg(nb + j * C + i);
                        }
                        double xn[C], xb[C];
                        X.get(rx + dx, ry + dy, xn);
                        X.get(rx - dx, ry - dy, xb);
#pragma unroll
                        for (int j = 0; j < C; j++)
                        {
                            const double e = (double)own[j] * xn[j];
                            acc += fwd[d] ? e : -0.0;
                        }
#pragma unroll
                        for (int j = 0; j < C; j++)
                        {
                            const double e = (double)other[j] * xb[j];
                            acc += bwd[d] ? e : -0.0;
                        }
                    }
                }
                coupling[q * SWEEP_THREADS<TS> + threadIdx.x] = acc;
            }
            __syncthreads();
        }
        const int task = batch + (int)threadIdx.x;
        const int rx = rx0 + 2 * (task % nx), ry = ry0 + 2 * (task / nx);
        const int gx = x0 - SWEEP_MARGIN_X + rx, gy = y0 - SWEEP_MARGIN_Y + ry;
        if (task < TASKS && gx >= 0 && gx < w && gy >= 0 && gy < h)
        {
            const size_t t = (size_t)gy * w + gx, sp = stencil_pos(gx, gy, w, h);
            const bool own = rx >= SWEEP_MARGIN_X && rx < SWEEP_MARGIN_X + SWEEP_W && ry >= SWEEP_MARGIN_Y &&
                             ry < SWEEP_MARGIN_Y + SWEEP_H;
            double nb[C];
            if constexpr (ROWS)
                load_texel<C>(coupling + threadIdx.x * C, nb);
            else
            {
#pragma unroll
                for (int i = 0; i < C; i++)
                    nb[i] = 0.0;
                // as in stencil_apply: every load issued, a missing neighbour's products replaced by -0.0 (an exact no-op)
#pragma unroll
                for (int slot = 1; slot < SLOTS; slot++)
                {
                    int dx, dy;
                    slot_offset(slot, dx, dy);
                    const bool fwd = gx + dx >= 0 && gx + dx < w && gy + dy < h;
                    const bool bwd = gx - dx >= 0 && gx - dx < w && gy - dy >= 0;
                    double xn[C], xb[C];
                    X.get(rx + dx, ry + dy, xn);
                    X.get(rx - dx, ry - dy, xb);
                    const StenBlock<C, TS> blk(V, slot, T, sp);
#pragma unroll
                    for (int i = 0; i < C; i++)
#pragma unroll
                        for (int j = 0; j < C; j++)
                        {
                            const double e = blk[i * C + j] * xn[j];
                            nb[i] += fwd ? e : -0.0;
                        }
                    const StenBlock<C, TS> nbk(V, slot, T, bwd ? stencil_pos(gx - dx, gy - dy, w, h) : sp);
#pragma unroll
                    for (int i = 0; i < C; i++)
#pragma unroll
                        for (int j = 0; j < C; j++)
                        {
                            const double e = nbk[j * C + i] * xb[j];
                            nb[i] += bwd ? e : -0.0;
                        }
                }
            }
            const StenBlock<C, TS> self(V, 0, T, sp);
            double x[2 * TileX<C>::PAIRS], grad[C];
            float prev[C];
            X.get(rx, ry, x);
            load_texel<C>(V.grad + t * C, grad);
            load_channels<C>(V.prev + t * C, prev);
#pragma unroll
            for (int q = 0; q < C; q++)
            {
                const float l = A.lo[q], span = A.hi[q] - A.lo[q];
                const double a = self[q * C + q] + lambda;
                if (!(a > 0.0) || !(span > 0.0f))
                    continue;
                double rest = nb[q];
#pragma unroll
                for (int j = 0; j < C; j++)
                    if (j != q)
                        rest += self[q * C + j] * x[j];
                const double b = grad[q] + rest;
                const double want = (double)prev[q] - b / a;
                float value;
                const int kk = grid_nearest(l, A.hi[q], A.bits, (float)want, frac, value);
                if (own)
                {
                    const size_t idx = t * C + q;
                    if ((int)V.k[idx] != kk)
                    {
                        V.k[idx] = (uint8_t)kk;
                        changed++;
                    }
                    V.v[idx] = value;
                }
                x[q] = (double)value - (double)prev[q];
            }
            X.set(rx, ry, x);
            if (own)
                store_texel<C>(xout + t * C, x);
        }
        __syncthreads();   // the couplings are spent; after the last batch, the colour is done
    }
    return changed;
}

template <int C, typename TS>
__global__ void __launch_bounds__(SWEEP_THREADS<TS>, 1) k_quant_sweep(Planes P, const __grid_constant__ SweepArgs A)
{
    extern __shared__ double2 sweep_sh[];
    __shared__ double frac[GRID_FRACTIONS];
    grid_fractions(frac, A.bits);
    const TileX<C> X{ sweep_sh };
    double* coupling = reinterpret_cast<double*>(sweep_sh + TileX<C>::PAIRS * 4 * SWEEP_CELLS);
    int pl = P.n - 1;
    while ((int)blockIdx.x >= A.bend[pl])
        pl--;
    const int tile = (int)blockIdx.x - (A.bend[pl] - A.btiles[pl]);
    const PlaneView& V = P.p[pl];
    const int tiles_x = (V.w + SWEEP_W - 1) / SWEEP_W;
    const int x0 = tile % tiles_x * SWEEP_W, y0 = tile / tiles_x * SWEEP_H;
    const double* xin = A.to_r ? V.x : V.r;
    double* xout = A.to_r ? V.r : V.x;
    for (int i = threadIdx.x; i < 4 * SWEEP_CELLS; i += SWEEP_THREADS<TS>)
    {
        const int rx = i % (2 * SWEEP_COLS), ry = i / (2 * SWEEP_COLS);
        const int gx = x0 - SWEEP_MARGIN_X + rx, gy = y0 - SWEEP_MARGIN_Y + ry;
        double x[2 * TileX<C>::PAIRS] = {};
        if (!A.first && gx >= 0 && gx < V.w && gy >= 0 && gy < V.h)
            load_texel<C>(xin + ((size_t)gy * V.w + gx) * C, x);
        X.set(rx, ry, x);
    }
    __syncthreads();
    const double lambda = A.scalars[(size_t)pl * S_COUNT + S_LAMBDA];
    unsigned changed = sweep_colour<C, TS, 0>(V, A, lambda, x0, y0, X, frac, coupling, xout);
    changed += sweep_colour<C, TS, 1>(V, A, lambda, x0, y0, X, frac, coupling, xout);
    changed += sweep_colour<C, TS, 2>(V, A, lambda, x0, y0, X, frac, coupling, xout);
    changed += sweep_colour<C, TS, 3>(V, A, lambda, x0, y0, X, frac, coupling, xout);
    if (changed)
        atomicAdd(A.moved + pl, changed);
}

template <int C, typename TS>
static int launch_sweep(nntc_b200_device* d, const Planes& P, const SweepArgs& A, int tiles)
{
    constexpr bool ROWS = sizeof(TS) == sizeof(float) && C % 2 == 0;
    const int shared =
        TileX<C>::PAIRS * 4 * SWEEP_CELLS * (int)sizeof(double2) + (ROWS ? SWEEP_THREADS<TS> * C * (int)sizeof(double) : 0);
    NB_SHARED_LIMIT((k_quant_sweep<C, TS>), shared);
    k_quant_sweep<C, TS><<<tiles, SWEEP_THREADS<TS>, shared, d->stream>>>(P, A);
    NB_LAUNCHED();
    return NNTC_B200_OK;
}

// prev = v, x = 0 (the quantised path and the refinement measure the correction from the plane as assembled).
__global__ void k_snapshot(Planes P)
{
    const long long base = (long long)blockIdx.x * blockDim.x;
    const int pl = plane_of(P, base);
    const PlaneView& V = P.p[pl];
    // the block's texels' values, a value a thread: whole lines
    const size_t first = (size_t)(base - P.start[pl]) * P.c, end = (size_t)V.w * V.h * P.c;
    for (int i = 0; i < P.c; i++)
    {
        const size_t q = first + (size_t)i * THREADS + threadIdx.x;
        if (q < end)
        {
            V.prev[q] = V.v[q];
            V.x[q] = 0.0;
        }
    }
}

// ---- host drivers ---------------------------------------------------------------------------------------------------

static Planes texel_planes(nntc_b200_device* d, int level0, int k)
{
    Planes P = planes_for(d, level0, [&](int i) { return d->planes[(size_t)i].work[level0 ? 1 : 0].texels(); });
    P.kc = k;
    return P;
}

static Red red_for(nntc_b200_device* d, const Planes& P)
{
    return Red{ d->partial, (size_t)(P.start[P.n] / THREADS), d->scalars };
}

int assemble_split(nntc_b200_device* d, int k, int level0, const Planes& P_texels, int nmono, const double* mono,
                   int slots, bool f32);
int matvec_free(nntc_b200_device* d, const Planes& P, double* partial, int level0);

// diag_only: the gradient and the diagonal blocks (slot 0) alone, what the matrix-free conjugate gradients of the
// adjoint form need (their products come from adjoint_cg.cu, not from the other four slots).
int assemble(nntc_b200_device* d, const nntc_b200_model* m, int k, double ridge, int level0, bool diag_only = false)
{
    if (level0 && !d->l0_bc8)
    {
        set_error(NNTC_B200_ERR_STATE, "block (c') runs only under --l0 bc8");
        return NNTC_B200_ERR_STATE;
    }
    std::vector<double> mono;
    build_monomials(*m, level0, mono);
    NB_TRY(upload_small(d, d->mono[level0], mono.data(), mono.size() * sizeof(double)));
    Planes P = texel_planes(d, level0, k);
    const int nmono = monomial_count(level0 ? d->c1 : d->c0);
    const int blocks = (int)(P.start[P.n] / ASM_THREADS);
    const size_t shared = (size_t)SLOTS * nmono * ASM_THREADS * sizeof(double);
    AsmArgs A{ d->weights, d->bias, d->cw, d->mono[level0], nmono };
    NB_TRY(ktimer_begin(d, level0 ? NNTC_B200_K_ASSEMBLE0 : NNTC_B200_K_ASSEMBLE1));
    const bool split = diag_only || (!d->reference_shaped_assembly && k <= 4);
    // the adjoint form stores the stencil in FP32 (the split form only; the reference-shaped kernel is FP64)
    d->sten_f32[level0] = split && d->mixed_stencil != 0;
    d->sten_symmetric[level0] = false;
    if (split)
        NB_TRY(assemble_split(d, k, level0, P, nmono, mono.data(), diag_only ? 1 : SLOTS, d->sten_f32[level0]));
    else if (level0)
    {
        NB_SHARED_LIMIT(k_assemble<true>, (size_t)SLOTS * MAX_MONO * ASM_THREADS * sizeof(double));
        k_assemble<true><<<blocks, ASM_THREADS, shared, d->stream>>>(P, A);
    }
    else
    {
        NB_SHARED_LIMIT(k_assemble<false>, (size_t)SLOTS * MAX_MONO * ASM_THREADS * sizeof(double));
        k_assemble<false><<<blocks, ASM_THREADS, shared, d->stream>>>(P, A);
    }
    NB_TRY(ktimer_end(d));
    if (!diag_only && (d->reference_shaped_assembly || k > 4))
        NB_LAUNCHED();
    const Red R = red_for(d, P);
    const int tblocks = (int)(P.start[P.n] / THREADS);
    if (d->sten_f32[level0])
        k_diag<float><<<tblocks, THREADS, 0, d->stream>>>(P, R);
    else
        k_diag<double><<<tblocks, THREADS, 0, d->stream>>>(P, R);
    NB_LAUNCHED();
    k_diag_reduce<<<P.n, FOLD_THREADS, 0, d->stream>>>(P, R, ridge);
    NB_LAUNCHED();
    return NNTC_B200_OK;
}

static void fill_report(const nntc_b200_device* d, int i, int channels, nntc_b200_plane_report& rep)
{
    const double* s = d->host_scalars + (size_t)i * S_COUNT;
    rep.lambda = s[S_LAMBDA];
    rep.min_diag = s[S_DIAG_MIN];
    rep.max_diag = s[S_DIAG_MAX];
    rep.residual = s[S_RESID];
    rep.moved_values = (long long)s[S_MOVED];
    rep.delta2 = s[S_DELTA2];
    rep.plane2 = s[S_PLANE2];
    for (int c = 0; c < channels; c++)
    {
        rep.lo[c] = (float)s[S_LO + c];
        rep.hi[c] = (float)s[S_HI + c];
    }
}

static int precondition_init(nntc_b200_device* d, const Planes& P, const Red& R, int tblocks, bool f32)
{
#define NB_PRECOND(C)                                                                                                 \
    if (f32)                                                                                                          \
        k_precondition_init<C, float><<<tblocks, THREADS, 0, d->stream>>>(P, R);                                      \
    else                                                                                                              \
        k_precondition_init<C, double><<<tblocks, THREADS, 0, d->stream>>>(P, R);                                     \
    break;
    switch (P.c)
    {
    case 1: NB_PRECOND(1)
    case 2: NB_PRECOND(2)
    case 3: NB_PRECOND(3)
    default: NB_PRECOND(4)
    }
#undef NB_PRECOND
    NB_LAUNCHED();
    return NNTC_B200_OK;
}

int solve_block(nntc_b200_device* d, const nntc_b200_model* m, int k, double ridge, int level0,
                nntc_b200_plane_report* rep, double* ms)
{
    const int np = (int)d->planes.size();
    const int nc = level0 ? d->c0 : d->c1;
    for (int i = 0; i < np; i++)
        rep[i] = nntc_b200_plane_report{};
    // the adjoint form: the gradient and the diagonal blocks assembled, the products matrix-free (adjoint_cg.cu)
    const bool adjoint = d->adjoint_cg != 0 && k <= 4;
    NB_TRY(block_begin(d));
    NB_TRY(assemble(d, m, k, ridge, level0, adjoint));
    NB_CUDA(cudaEventRecord(d->ev[2], d->stream));
    Planes P = texel_planes(d, level0, k);
    const Red R = red_for(d, P);
    const int tblocks = (int)(P.start[P.n] / THREADS);
    NB_TRY(precondition_init(d, P, R, tblocks, d->sten_f32[level0]));
    k_cg_start<<<P.n, FOLD_THREADS, 0, d->stream>>>(P, R);
    NB_LAUNCHED();
    NB_CUDA(cudaEventRecord(d->ev[3], d->stream));
    unsigned int* active = d->counters + CNT_ACTIVE;
    for (int it = 0; it < CG_MAX_IT; it++)
    {
        NB_TRY(ktimer_begin(d, level0 ? NNTC_B200_K_MATVEC0 : NNTC_B200_K_MATVEC));
        if (adjoint)
            NB_TRY(matvec_free(d, P, R.partial, level0));
        else
        {
            const int symmetric = d->sten_symmetric[level0] ? 1 : 0;
            const bool f32 = d->sten_f32[level0];
            switch (P.c)
            {
            case 1:
                if (f32)
                    k_cg_matvec<1, float><<<tblocks, THREADS, 0, d->stream>>>(P, R);
                else
                    k_cg_matvec<1, double><<<tblocks, THREADS, 0, d->stream>>>(P, R);
                break;
            case 2:
                if (f32)
                    k_cg_matvec_rows<2><<<tblocks, THREADS, 0, d->stream>>>(P, R, symmetric);
                else if (tblocks <= 148)
                    k_cg_matvec<2, double><<<tblocks, THREADS, 0, d->stream>>>(P, R);
                else
                    k_cg_matvec<2, double, 6><<<tblocks, THREADS, 0, d->stream>>>(P, R);
                break;
            case 3:
                if (f32)
                    k_cg_matvec<3, float><<<tblocks, THREADS, 0, d->stream>>>(P, R);
                else
                    k_cg_matvec<3, double><<<tblocks, THREADS, 0, d->stream>>>(P, R);
                break;
            default:
                if (f32)
                    k_cg_matvec_rows<4><<<tblocks, THREADS, 0, d->stream>>>(P, R, symmetric);
                else
                    k_cg_matvec<4, double><<<tblocks, THREADS, 0, d->stream>>>(P, R);
                break;
            }
            NB_LAUNCHED();
        }
        NB_TRY(ktimer_end(d));
        k_cg_alpha<<<P.n, FOLD_THREADS, 0, d->stream>>>(P, R, active + (it % CG_PROBE));
        NB_LAUNCHED();
        switch (P.c)
        {
        case 1: k_cg_update_rows<1><<<tblocks, THREADS, 0, d->stream>>>(P, R); break;
        case 2: k_cg_update_rows<2><<<tblocks, THREADS, 0, d->stream>>>(P, R); break;
        case 3: k_cg_update<3><<<tblocks, THREADS, 0, d->stream>>>(P, R); break;
        default: k_cg_update_rows<4><<<tblocks, THREADS, 0, d->stream>>>(P, R); break;
        }
        NB_LAUNCHED();
        k_cg_beta<<<P.n, FOLD_THREADS, 0, d->stream>>>(P, R, it, active + (it % CG_PROBE),
                                             adjoint || d->sten_f32[level0] ? CG_TOL_FP32 : CG_TOL);
        NB_LAUNCHED();
        k_cg_direction<<<tblocks, THREADS, 0, d->stream>>>(P, R);
        NB_LAUNCHED();
        if ((it + 1) % CG_PROBE != 0)
            continue;
        NB_TRY(fetch(d, FETCH_ACTIVE, active + (it % CG_PROBE), sizeof(unsigned int)));
        NB_CUDA(cudaStreamSynchronize(d->stream));
        if (*fetched<unsigned int>(d, FETCH_ACTIVE) == 0)
            break;
    }
    k_correct_range<<<tblocks, THREADS, 0, d->stream>>>(P, R);
    NB_LAUNCHED();
    k_range_reduce<<<dim3(P.n, P.c), FOLD_THREADS, 0, d->stream>>>(P, R);
    NB_LAUNCHED();
    const int levels = level0 ? 255 : (1 << m->bits1) - 1;
    k_movement<<<tblocks, THREADS, 0, d->stream>>>(P, R, levels);
    NB_LAUNCHED();
    k_movement_reduce<<<P.n, FOLD_THREADS, 0, d->stream>>>(P, R);
    NB_LAUNCHED();
    NB_CUDA(cudaMemcpyAsync(d->host_scalars, d->scalars, (size_t)np * S_COUNT * sizeof(double),
                            cudaMemcpyDeviceToHost, d->stream));
    double t = 0.0;
    NB_TRY(block_end(d, &t));
    float a_ms = 0.0f, p_ms = 0.0f, c_ms = 0.0f;
    NB_CUDA(cudaEventElapsedTime(&a_ms, d->ev[0], d->ev[2]));
    NB_CUDA(cudaEventElapsedTime(&p_ms, d->ev[2], d->ev[3]));
    NB_CUDA(cudaEventElapsedTime(&c_ms, d->ev[3], d->ev[1]));
    for (int i = 0; i < np; i++)
    {
        fill_report(d, i, nc, rep[i]);
        rep[i].iterations = (int)d->host_scalars[(size_t)i * S_COUNT + S_ITER];
        rep[i].quantised = 0;
        rep[i].ms_assemble = a_ms;
        rep[i].ms_precond = p_ms;
        rep[i].ms_cg = c_ms;
    }
    if (ms)
        *ms = t;
    return NNTC_B200_OK;
}

int sweep_block(nntc_b200_device* d, const nntc_b200_model* m, int k, double ridge, int sweeps, int level0,
                nntc_b200_plane_report* rep, double* ms)
{
    const int np = (int)d->planes.size();
    const int nc = level0 ? d->c0 : d->c1;
    for (int i = 0; i < np; i++)
        rep[i] = nntc_b200_plane_report{};
    // every slot assembled whatever the conjugate gradients' operator: a sweep step reads the texel's coupling to its
    // eight neighbours from the stencil (with the matrix-free option on, an assembly of the diagonal blocks alone
    // would leave the sweeps reading another block's off-diagonal slots)
    NB_TRY(block_begin(d));
    NB_TRY(assemble(d, m, k, ridge, level0, false));
    NB_CUDA(cudaEventRecord(d->ev[2], d->stream));
    Planes P = texel_planes(d, level0, k);
    k_snapshot<<<(int)(P.start[P.n] / THREADS), THREADS, 0, d->stream>>>(P);
    NB_LAUNCHED();
    NB_CUDA(cudaMemsetAsync(d->counters + CNT_SWEEP, 0, MAX_PLANES * sizeof(unsigned int), d->stream));
    const int bits = level0 ? 8 : m->bits1;
    SweepArgs S{ d->scalars, level0 ? d->lo0 : d->lo1, level0 ? d->hi0 : d->hi1, bits, d->sten_symmetric[level0] ? 1 : 0 };
    S.moved = d->counters + CNT_SWEEP;
    int tiles = 0;
    bool wide = false, high = false;
    for (int i = P.n - 1; i >= 0; i--)
    {
        wide = wide || P.p[i].w > 1;
        high = high || P.p[i].h > 1;
        S.btiles[i] = ((P.p[i].w + SWEEP_W - 1) / SWEEP_W) * ((P.p[i].h + SWEEP_H - 1) / SWEEP_H);
        S.bend[i] = tiles += S.btiles[i];
    }
    for (int s = 0; s < sweeps && tiles <= SWEEP_TILES; s++)
    {
        S.first = s == 0;
        S.to_r = (sweeps - 1 - s) & 1;   // the last sweep leaves the corrections in x
        NB_TRY(ktimer_begin(d, NNTC_B200_K_SWEEP, (wide ? 2 : 1) * (high ? 2 : 1)));   // the colours it has
#define NB_SWEEP(C)                                                                                                   \
    if (d->sten_f32[level0])                                                                                          \
        NB_TRY((launch_sweep<C, float>(d, P, S, tiles)));                                                             \
    else                                                                                                              \
        NB_TRY((launch_sweep<C, double>(d, P, S, tiles)));                                                            \
    break;
        switch (P.c)
        {
        case 1: NB_SWEEP(1)
        case 2: NB_SWEEP(2)
        case 3: NB_SWEEP(3)
        default: NB_SWEEP(4)
        }
#undef NB_SWEEP
        NB_TRY(ktimer_end(d));
    }
    for (int s = 0; s < sweeps && tiles > SWEEP_TILES; s++)
        for (int colour = 0; colour < 4; colour++)
        {
            const int cx = colour & 1, cy = colour >> 1;
            Planes C = planes_for(d, level0, [&](int i) {
                const Work& w = d->planes[(size_t)i].work[level0 ? 1 : 0];
                return (size_t)((w.w - cx + 1) / 2) * (size_t)((w.h - cy + 1) / 2);
            });
            C.kc = k;
            if (C.start[C.n] == 0)
                continue;
            ColourArgs A{ d->scalars, level0 ? d->lo0 : d->lo1, level0 ? d->hi0 : d->hi1, bits, cx, cy,
                         d->sten_symmetric[level0] ? 1 : 0, d->counters + CNT_SWEEP };
            NB_TRY(ktimer_begin(d, NNTC_B200_K_SWEEP));
            const int sblocks = (int)(C.start[C.n] / THREADS);
#define NB_SWEEP(TS)                                                                                                  \
    switch (C.c)                                                                                                      \
    {                                                                                                                 \
    case 1: k_quant_colour<1, TS><<<sblocks, THREADS, 0, d->stream>>>(C, A); break;                                    \
    case 2: k_quant_colour<2, TS><<<sblocks, THREADS, 0, d->stream>>>(C, A); break;                                    \
    case 3: k_quant_colour<3, TS><<<sblocks, THREADS, 0, d->stream>>>(C, A); break;                                    \
    default:                                                                                                           \
        if (sizeof(TS) == sizeof(float) && colour_per_sm(sblocks) == 4)                                                \
            k_quant_colour<4, TS, sizeof(TS) == sizeof(float) ? 4 : 0><<<sblocks, THREADS, 0, d->stream>>>(C, A);      \
        else                                                                                                           \
            k_quant_colour<4, TS><<<sblocks, THREADS, 0, d->stream>>>(C, A);                                           \
        break;                                                                                                         \
    }
            if (d->sten_f32[level0])
            {
                NB_SWEEP(float)
            }
            else
            {
                NB_SWEEP(double)
            }
#undef NB_SWEEP
            NB_TRY(ktimer_end(d));
            NB_LAUNCHED();
        }
    NB_CUDA(cudaEventRecord(d->ev[3], d->stream));
    NB_CUDA(cudaMemcpyAsync(d->host_scalars, d->scalars, (size_t)np * S_COUNT * sizeof(double),
                            cudaMemcpyDeviceToHost, d->stream));
    NB_CUDA(cudaMemcpyAsync(d->host_counters, d->counters, MAX_PLANES * sizeof(unsigned int),
                            cudaMemcpyDeviceToHost, d->stream));
    double t = 0.0;
    NB_TRY(block_end(d, &t));
    float a_ms = 0.0f, s_ms = 0.0f;
    NB_CUDA(cudaEventElapsedTime(&a_ms, d->ev[0], d->ev[2]));
    NB_CUDA(cudaEventElapsedTime(&s_ms, d->ev[2], d->ev[3]));
    for (int i = 0; i < np; i++)
    {
        fill_report(d, i, nc, rep[i]);
        rep[i].quantised = 1;
        rep[i].sweeps = sweeps;
        rep[i].ms_assemble = a_ms;
        rep[i].ms_sweeps = s_ms;
        // the fields only the continuous path writes are cleared (src/solve_level1.cu:1388-1397)
        rep[i].iterations = 0;
        rep[i].residual = 0.0;
        rep[i].moved_values = 0;
        rep[i].delta2 = 0.0;
        rep[i].plane2 = 0.0;
        rep[i].moved = (long long)d->host_counters[i];
    }
    if (ms)
        *ms = t;
    return NNTC_B200_OK;
}

// The gradient, the diagonal blocks and the preconditioned descent direction of one latent at its current plane:
// grad, z = -(H_tt + lambda I)^-1 grad texel by texel, prev = v (what the joint pass steps from).
int descent_direction(nntc_b200_device* d, const nntc_b200_model* m, int k, double ridge, int level0)
{
    NB_TRY(assemble(d, m, k, ridge, level0, true));
    Planes P = texel_planes(d, level0, k);
    const Red R = red_for(d, P);
    const int tblocks = (int)(P.start[P.n] / THREADS);
    NB_TRY(precondition_init(d, P, R, tblocks, d->sten_f32[level0]));
    k_snapshot<<<tblocks, THREADS, 0, d->stream>>>(P);
    NB_LAUNCHED();
    return NNTC_B200_OK;
}

// Level 0's stencil copied into the BC refinement's block-major layout (bc_sten: [block][slot][i][j][texel of the
// block]), one thread per texel; used when the assembly did not write the copy itself.
__global__ void k_bc_sten_copy(Planes P)
{
    const long long base = (long long)blockIdx.x * blockDim.x;
    const int pl = plane_of(P, base);
    const PlaneView& V = P.p[pl];
    const long long t = base - P.start[pl] + threadIdx.x;
    if (t >= (long long)V.w * V.h)
        return;
    const int x = (int)(t % V.w), y = (int)(t / V.w), cc = P.c * P.c;
    const size_t T = (size_t)V.w * V.h, sp = stencil_pos(x, y, V.w, V.h);
    const size_t blk = (size_t)(y >> 2) * (size_t)((V.w + 3) >> 2) + (size_t)(x >> 2);
    const int in = (y & 3) * 4 + (x & 3);
    for (int slot = 0; slot < SLOTS; slot++)
        for (int e = 0; e < cc; e++)
            V.bc_sten[((blk * SLOTS + slot) * cc + e) * 16 + in] = V.stencil[(size_t)(slot * cc + e) * T + sp];
}

// Block (c')'s assembly alone with no ridge, the correction measured from the plane as it stands (for refine_bc). The
// refinement's decisions are the reference's on an FP64 stencil, so this assembly is FP64 in either form.
int assemble_for_refine(nntc_b200_device* d, const nntc_b200_model* m, int k, double* ms)
{
    struct Fp64Scope
    {
        nntc_b200_device* d;
        int was;
        ~Fp64Scope()
        {
            d->mixed_stencil = was;
            d->bc_copy = 0;
        }
    } fp64{ d, d->mixed_stencil };
    d->mixed_stencil = 0;
    d->bc_copy = 1;   // the refinement reads the block-major copy the gather writes beside the stencil
    d->bc_copied = 0;
    NB_TRY(block_begin(d));
    NB_TRY(assemble(d, m, k, 0.0, 1));
    Planes P = texel_planes(d, 1, k);
    if (!d->bc_copied)
    {
        // the reference-shaped assembly wrote the stencil alone: the copy from it
        k_bc_sten_copy<<<(int)(P.start[P.n] / THREADS), THREADS, 0, d->stream>>>(P);
        NB_LAUNCHED();
    }
    k_snapshot<<<(int)(P.start[P.n] / THREADS), THREADS, 0, d->stream>>>(P);
    NB_LAUNCHED();
    return block_end(d, ms);
}

}   // namespace nb

using namespace nb;

extern "C"
{

int nntc_b200_set_option(nntc_b200_device* d, int option, int value)
{
    if (option == NNTC_B200_OPT_REFERENCE_SHAPED_ASSEMBLY)
    {
        d->reference_shaped_assembly = value != 0;
        return NNTC_B200_OK;
    }
    if (option == NNTC_B200_OPT_MIXED_PRECISION_GRAM)
    {
        d->mixed_gram = value != 0;
        return NNTC_B200_OK;
    }
    if (option == NNTC_B200_OPT_ADJOINT_CG)
    {
        d->adjoint_cg = value != 0;
        return NNTC_B200_OK;
    }
    if (option == NNTC_B200_OPT_MIXED_OBJECTIVE)
    {
        d->mixed_objective = value != 0;
        return NNTC_B200_OK;
    }
    if (option == NNTC_B200_OPT_FP32_STENCIL)
    {
        d->mixed_stencil = value != 0;
        return NNTC_B200_OK;
    }
    set_error(NNTC_B200_ERR_ARG, "no such option");
    return NNTC_B200_ERR_ARG;
}

int nntc_b200_solve_level1_all(nntc_b200_device* d, const nntc_b200_model* m, int k, double ridge,
                               nntc_b200_plane_report* rep, double* ms)
{
    return solve_block(d, m, k, ridge, 0, rep, ms);
}

int nntc_b200_sweep_level1_all(nntc_b200_device* d, const nntc_b200_model* m, int k, double ridge, int sweeps,
                               nntc_b200_plane_report* rep, double* ms)
{
    return sweep_block(d, m, k, ridge, sweeps, 0, rep, ms);
}

int nntc_b200_solve_level0_cont_all(nntc_b200_device* d, const nntc_b200_model* m, int k, double ridge,
                                    nntc_b200_plane_report* rep, double* ms)
{
    return solve_block(d, m, k, ridge, 1, rep, ms);
}

int nntc_b200_sweep_level0_cont_all(nntc_b200_device* d, const nntc_b200_model* m, int k, double ridge, int sweeps,
                                    nntc_b200_plane_report* rep, double* ms)
{
    return sweep_block(d, m, k, ridge, sweeps, 1, rep, ms);
}

int nntc_b200_assemble_level0_for_refine(nntc_b200_device* d, const nntc_b200_model* m, int k, double* ms)
{
    return assemble_for_refine(d, m, k, ms);
}

}   // extern "C"
