// row_stage.cuh: a warp's rows of targets in shared memory by asynchronous copies, for the kernels that take one pixel a
// lane and its 1 + K sites in turn (the objective, the normal equations).
//
// A pixel's targets at one site are a row of NOUT values; a lane that loads its own row from global memory touches a
// line of its own per load, NOUT times over, and the L1 then serves one line a cycle: that alone was 86% of the
// tensor-core normal equations' time and half of the objective's. Here the warp copies the 32 rows of one site together,
// in the widest copies their size allows, one site ahead of the lanes that read them.
#pragma once

#include "device.cuh"

namespace nb
{

// Rows of NOUT values of type T: the copies' unit and the row's stride in shared memory (an odd number of units, so that
// the lanes' reads of their own rows fall on different banks).
template <int NOUT, typename T>
struct RowShape
{
    static constexpr int BYTES = NOUT * (int)sizeof(T);
    static constexpr int UNIT = BYTES % 16 == 0 ? 16 : (BYTES % 8 == 0 ? 8 : 4);
    static constexpr int UNITS = BYTES / UNIT;
    static constexpr int STRIDE = (UNITS | 1) * UNIT;
};

template <int UNIT>
__device__ __forceinline__ void copy_unit(void* dst, const void* src)
{
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (UNIT == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src) : "memory");
    else if constexpr (UNIT == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(src) : "memory");
}

// `rows` rows (at most 32), `pitch` values apart in global memory, into the warp's buffer, one row a stride.
template <int NOUT, typename T>
__device__ __forceinline__ void stage_rows(char* buffer, const T* from, int pitch, int rows, int lane)
{
    using S = RowShape<NOUT, T>;
    const char* src = reinterpret_cast<const char*>(from);
    for (int i = lane; i < rows * S::UNITS; i += 32)
    {
        const int r = i / S::UNITS, q = i - r * S::UNITS;
        copy_unit<S::UNIT>(buffer + r * S::STRIDE + q * S::UNIT,
                           src + (size_t)r * pitch * sizeof(T) + q * S::UNIT);
    }
}

// The lane's own row into registers, in reads of the copies' unit.
template <int NOUT, typename T>
__device__ __forceinline__ void read_row(const char* buffer, int lane, T (&out)[NOUT])
{
    using S = RowShape<NOUT, T>;
    const char* row = buffer + lane * S::STRIDE;
    if constexpr (S::UNIT == 16)
    {
#pragma unroll
        for (int q = 0; q < S::UNITS; q++)
        {
            const float4 v = *reinterpret_cast<const float4*>(row + 16 * q);
            if constexpr (sizeof(T) == 4)
            {
                out[4 * q] = v.x;
                out[4 * q + 1] = v.y;
                out[4 * q + 2] = v.z;
                out[4 * q + 3] = v.w;
            }
            else
            {
                out[2 * q] = __hiloint2double(__float_as_int(v.y), __float_as_int(v.x));
                out[2 * q + 1] = __hiloint2double(__float_as_int(v.w), __float_as_int(v.z));
            }
        }
    }
    else if constexpr (S::UNIT == 8 && sizeof(T) == 4)
    {
#pragma unroll
        for (int q = 0; q < S::UNITS; q++)
        {
            const float2 v = *reinterpret_cast<const float2*>(row + 8 * q);
            out[2 * q] = v.x;
            out[2 * q + 1] = v.y;
        }
    }
    else
    {
#pragma unroll
        for (int r = 0; r < NOUT; r++)
            out[r] = reinterpret_cast<const T*>(row)[r];
    }
}

// blend_u with the channel loads of a tap one vector where the channel count is four or two (the same arithmetic).
__device__ __forceinline__ void blend_any(const float* plane, int w, int c, const Tap& t, float* out)
{
    if (c == 4)
        blend_c<4>(plane, w, t, out);
    else if (c == 2)
        blend_c<2>(plane, w, t, out);
    else
        blend_u<MAX_CH>(plane, w, c, t, out);
}

}   // namespace nb
