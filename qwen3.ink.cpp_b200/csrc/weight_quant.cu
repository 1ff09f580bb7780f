// Offline weight quantizers on the GPU: fp32 weights [N][K] -> the reference's on-disk format
// (packed nibbles u8 [N][K/2] in the AWQ-interleaved order, scales and minima f32 [N][K/32],
// zero points i8 [N][K/32]), so that a checkpoint can be packed without the export notebooks.
//
// Restates notebooks/quantize_methods.py of the reference, operation for operation in fp32:
//   quantize_row_q41_tinyml (:68-125)  d = (max - min) / 15, m = min, id = d != 0 ? 1 / d : 0,
//                                      q = clip(rint((x - m) * id), 0, 15)      (np.round: ties to even), zp = 0
//   quantize_row_q40_tinyml (:13-66)   d = x[argmax |x|] / -8 (first index on ties), id likewise,
//                                      q = (uint8) clip(x * id + 8.5, 0, 15)    (truncation), m = 0, zp = 8
//   both: byte[32 g + e] = q[64 g + e] | q[64 g + 32 + e] << 4                  (:61-64, :120-123)
//
// Bound by memory: 4 bytes read and 0.78 written per weight.  Eight lanes share a pair of blocks (64 weights): a lane holds
// four consecutive elements of each, so both loads and the packed store of a warp are whole 128-byte lines, the reductions
// take three exchanges, and four pairs per lane keep eight 16-byte loads in flight.  (One element per lane and block, five
// exchanges and byte stores ran at 1.26 TB/s, 190 us for 12288 x 4096.)
#include "inkq_internal.h"

namespace inkq {

constexpr int WQ_PAIRS = 4;   // pairs of blocks per group of eight lanes

// Scale, minimum and the four codes (one per byte) of this lane's elements 4t .. 4t+3 of a block shared by eight lanes.
template <int FORMAT>   // 0: Q4_0, 1: Q4_1
__device__ __forceinline__ uint32_t quantize_block(const float4 x4, int t, float &dd, float &mm)
{
    const float x[4] = {x4.x, x4.y, x4.z, x4.w};
    float v[4];
    if (FORMAT == 1) {
        float mx = fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3])), mn = fminf(fminf(x[0], x[1]), fminf(x[2], x[3]));
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        }
        mm = mn;
        dd = __fdiv_rn(__fsub_rn(mx, mn), 15.0f);
        const float id = (dd != 0.0f) ? __fdiv_rn(1.0f, dd) : 0.0f;
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = rintf(__fmul_rn(__fsub_rn(x[i], mn), id));
    } else {
        // the value of the largest magnitude, lowest index on ties (np.argmax): the key orders by magnitude, then by
        // descending index, and carries the sign along
        unsigned long long key = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t bits = __float_as_uint(x[i]);
            const unsigned long long k = (static_cast<unsigned long long>(bits & 0x7fffffffu) << 6) | static_cast<unsigned>((31 - 4 * t - i) << 1) | (bits >> 31);
            key = k > key ? k : key;
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const unsigned long long k = __shfl_xor_sync(0xffffffffu, key, o);
            key = k > key ? k : key;
        }
        const float val = __uint_as_float(static_cast<uint32_t>(key >> 6) | (static_cast<uint32_t>(key & 1u) << 31));
        dd = __fdiv_rn(val, -8.0f);
        mm = 0.0f;
        const float id = (dd != 0.0f) ? __fdiv_rn(1.0f, dd) : 0.0f;
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = __fadd_rn(__fmul_rn(x[i], id), 8.5f);
    }
    uint32_t q = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) q |= static_cast<uint32_t>(fminf(fmaxf(v[i], 0.0f), 15.0f)) << (8 * i);   // truncation, as astype(np.uint8) of a value in [0, 15]
    return q;
}

// ALIGNED: every pointer suits the vector accesses (the callers' usual case); otherwise element by element.
template <int FORMAT, bool ALIGNED>
__global__ void __launch_bounds__(256) k_quantize_weight_q4(const float *__restrict__ w, long long pairs, uint8_t *__restrict__ nib, float *__restrict__ d,
                                                            float *__restrict__ m, int8_t *__restrict__ zp)
{
    // a pair is 64 consecutive floats of w, 32 consecutive bytes of nib and two consecutive entries of d, m and zp, so the
    // matrix is one long list of pairs; a warp takes 4 * WQ_PAIRS consecutive ones
    const int lane = threadIdx.x & 31, t = lane & 7;
    const long long p0 = (static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5)) * (4 * WQ_PAIRS) + (lane >> 3);
    float4 lo[WQ_PAIRS], hi[WQ_PAIRS];
#pragma unroll
    for (int u = 0; u < WQ_PAIRS; u++) {
        const long long p = p0 + 4 * u;
        lo[u] = hi[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p < pairs) {
            const float *src = w + p * 64 + 4 * t;
            if (ALIGNED) {
                lo[u] = __ldcs(reinterpret_cast<const float4 *>(src));
                hi[u] = __ldcs(reinterpret_cast<const float4 *>(src + 32));
            } else {
                lo[u] = make_float4(src[0], src[1], src[2], src[3]);
                hi[u] = make_float4(src[32], src[33], src[34], src[35]);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < WQ_PAIRS; u++) {
        const long long p = p0 + 4 * u;
        float2 dd, mm;
        const uint32_t q_lo = quantize_block<FORMAT>(lo[u], t, dd.x, mm.x);
        const uint32_t q_hi = quantize_block<FORMAT>(hi[u], t, dd.y, mm.y);
        if (p < pairs) {
            const uint32_t q = q_lo | (q_hi << 4);
            constexpr int z = (FORMAT == 0) ? 8 : 0;
            if (ALIGNED) {
                reinterpret_cast<uint32_t *>(nib)[p * 8 + t] = q;
                if (t == 0) {
                    reinterpret_cast<float2 *>(d)[p] = dd;
                    reinterpret_cast<float2 *>(m)[p] = mm;
                    if (zp != nullptr) reinterpret_cast<char2 *>(zp)[p] = make_char2(z, z);
                }
            } else {
                for (int i = 0; i < 4; i++) nib[p * 32 + 4 * t + i] = static_cast<uint8_t>(q >> (8 * i));
                if (t == 0) {
                    d[2 * p] = dd.x;
                    d[2 * p + 1] = dd.y;
                    m[2 * p] = mm.x;
                    m[2 * p + 1] = mm.y;
                    if (zp != nullptr) zp[2 * p] = zp[2 * p + 1] = z;
                }
            }
        }
    }
}

}  // namespace inkq

using namespace inkq;

extern "C" int inkq_weight_quantize_dev(inkq_ctx *ctx, int format, int N, int K, const float *w_dev, uint8_t *nib_dev, float *d_dev, float *m_dev,
                                        int8_t *zp_dev)
{
    if (ctx == nullptr) return fail(nullptr, INKQ_ERR_INVALID, "null context");
    INKQ_CUDA(ctx, cudaSetDevice(ctx->device));
    INKQ_REQUIRE(ctx, format == 0 || format == 1, "format must be 0 (Q4_0) or 1 (Q4_1)");
    INKQ_REQUIRE(ctx, N >= 1 && K >= 64 && K % 64 == 0, "K must be a positive multiple of 64");
    INKQ_REQUIRE(ctx, w_dev && nib_dev && d_dev && m_dev, "null pointer");
    const long long pairs = static_cast<long long>(N) * (K / 64);
    const bool aligned = ((reinterpret_cast<uintptr_t>(w_dev) & 15) | (reinterpret_cast<uintptr_t>(nib_dev) & 3) | (reinterpret_cast<uintptr_t>(d_dev) & 7) |
                          (reinterpret_cast<uintptr_t>(m_dev) & 7) | (reinterpret_cast<uintptr_t>(zp_dev) & 1)) == 0;
    const unsigned grid = static_cast<unsigned>((pairs + 32 * WQ_PAIRS - 1) / (32 * WQ_PAIRS));
    auto kernel = aligned ? (format == 1 ? k_quantize_weight_q4<1, true> : k_quantize_weight_q4<0, true>)
                          : (format == 1 ? k_quantize_weight_q4<1, false> : k_quantize_weight_q4<0, false>);
    kernel<<<grid, 256, 0, ctx->stream>>>(w_dev, pairs, nib_dev, d_dev, m_dev, zp_dev);
    return after_launch(ctx, "k_quantize_weight_q4");
}
