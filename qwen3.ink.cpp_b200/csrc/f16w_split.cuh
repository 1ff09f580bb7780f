// The fp32 activations of the fp16-weight products as two fp16 operands, shared by k_f16w_rows and k_f16w_split:
//   x = 2^-e * (h + l),   h = fp16(x * 2^e),   l = fp16(x * 2^e - h)
// with one e per row that takes the row's largest finite magnitude into [2^13, 2^14).  h + l carry 22 significant bits of the
// row's larger elements, and a finite row neither overflows nor loses elements below fp16's range: e goes from -114 (a
// largest value of 2^127) to 126, where even the subnormal x are multiples of 2^-23 after scaling, which h + l hold
// exactly; both 2^e and 2^-e are normal floats.  Infinities and NaNs stay what they are in h, with l = 0 beside an infinity
// (the difference would be a NaN), so that they act on the products as in an fp32 evaluation.
#pragma once
#include <cuda_fp16.h>
#include <float.h>

namespace inkq {

// Largest magnitude so far; a NaN in either argument stays.  A row without one, and without infinities, ends at or below FLT_MAX
__device__ __forceinline__ float absmax_nan(float amax, float v)
{
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(amax), "f"(fabsf(v)));
    return r;
}
__device__ __forceinline__ float absmax_nan(float amax, const float4 v)
{
    return absmax_nan(absmax_nan(absmax_nan(absmax_nan(amax, v.x), v.y), v.z), v.w);
}

// Largest finite magnitude of a row, by one warp: the second look at a row that holds infinities or NaNs
static __device__ __noinline__ float finite_absmax(const float4 *row, int n4, int lane)
{
    float amax = 0.f;
    for (int i = lane; i < n4; i += 32) {
        const float4 v = row[i];
        const float a[4] = {fabsf(v.x), fabsf(v.y), fabsf(v.z), fabsf(v.w)};
        for (int j = 0; j < 4; j++)
            if (a[j] <= FLT_MAX) amax = fmaxf(amax, a[j]);
    }
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    return amax;
}

// e for the largest finite magnitude of a row (0: the row is zero, whatever the scale)
__device__ __forceinline__ int split_exponent(float amax) { return amax > 0.f ? min(13 - ilogbf(amax), 126) : 0; }

// Four elements, `s` = 2^e; SPECIAL: the row holds infinities or NaNs
template <bool SPECIAL>
__device__ __forceinline__ void split4(const float4 v, float s, __half2 (&h2)[2], __half2 (&l2)[2])
{
    const float f[4] = {v.x * s, v.y * s, v.z * s, v.w * s};
    __half h[4], l[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        h[j] = __float2half_rn(f[j]);
        const float r = f[j] - __half2float(h[j]);   // exact in fp32
        l[j] = __float2half_rn(SPECIAL && !(fabsf(f[j]) <= FLT_MAX) ? 0.f : r);
    }
    h2[0] = __halves2half2(h[0], h[1]);
    h2[1] = __halves2half2(h[2], h[3]);
    l2[0] = __halves2half2(l[0], l[1]);
    l2[1] = __halves2half2(l[2], l[3]);
}

}  // namespace inkq
