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
// four consecutive elements of each, so both loads and the packed store of a warp are whole 128-byte lines, and four pairs per
// lane keep eight 16-byte loads in flight.  (One element per lane and block, five exchanges and byte stores ran at 1.26 TB/s, 190 us
// for 12288 x 4096.)  The eight blocks of eight lanes are reduced together: each exchange hands half of the remaining blocks to the
// partner, seven exchanges in place of 24, after which lane t owns block t, divides once for all and hands the factors back.  With
// every lane reducing and dividing for every block, 12288 x 4096 took 45.6 us in Q4_1 and 60.8 in Q4_0 (whose 64-bit keys are now built
// only where a block's extremes tie); now 39.8 and 39.3 = 6.0 TB/s.
#include "inkq_internal.h"

namespace inkq {

constexpr int WQ_PAIRS = 4;   // pairs of blocks per group of eight lanes

// Reduces v[k] of eight lanes (t = 0 .. 7) for each of eight blocks k; lane t returns with block t's result
template <typename T, typename Op>
__device__ __forceinline__ T reduce_scatter8(T (&v)[8], int t, Op op)
{
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        const bool up = (t & o) != 0;
#pragma unroll
        for (int i = 0; i < o; i++) {
            const T keep = up ? v[i + o] : v[i], give = up ? v[i] : v[i + o];
            v[i] = op(keep, __shfl_xor_sync(0xffffffffu, give, o));
        }
    }
    return v[0];
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
    // block 2u: the low one of pair u, 2u + 1: its high one
    static_assert(WQ_PAIRS == 4, "eight blocks for eight lanes");
    float dd, mm = 0.0f;
    if (FORMAT == 1) {
        float mx[8], mn[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float4 x = (k & 1) ? hi[k >> 1] : lo[k >> 1];
            mx[k] = fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w));
            mn[k] = fminf(fminf(x.x, x.y), fminf(x.z, x.w));
        }
        mm = reduce_scatter8(mn, t, [](float a, float b) { return fminf(a, b); });
        dd = __fdiv_rn(__fsub_rn(reduce_scatter8(mx, t, [](float a, float b) { return fmaxf(a, b); }), mm), 15.0f);
    } else {
        // The value of the largest magnitude (as bits: a NaN is larger than any number): the larger of the positive and the negative
        // side's maximum
        int pos[8], neg[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float4 x = (k & 1) ? hi[k >> 1] : lo[k >> 1];
            const int b[4] = {__float_as_int(x.x), __float_as_int(x.y), __float_as_int(x.z), __float_as_int(x.w)};
            pos[k] = max(max(max(b[0], b[1]), max(b[2], b[3])), 0);
            constexpr int sign = static_cast<int>(0x80000000u);
            neg[k] = max(max(max(b[0] ^ sign, b[1] ^ sign), max(b[2] ^ sign, b[3] ^ sign)), 0);
        }
        const auto larger = [](int a, int b) { return max(a, b); };
        const int above = reduce_scatter8(pos, t, larger), below = reduce_scatter8(neg, t, larger);
        uint32_t val = above > below ? static_cast<uint32_t>(above) : static_cast<uint32_t>(below) | 0x80000000u;
        if (__any_sync(0xffffffffu, above == below)) {
            // Both sides reach it (or the block is zero): the lowest index decides (np.argmax).  The key orders by magnitude, then by
            // descending index, and carries the sign along
            unsigned long long key[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const float4 x4 = (k & 1) ? hi[k >> 1] : lo[k >> 1];
                const float x[4] = {x4.x, x4.y, x4.z, x4.w};
                key[k] = 0;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint32_t bits = __float_as_uint(x[i]);
                    const unsigned long long c = (static_cast<unsigned long long>(bits & 0x7fffffffu) << 6) | static_cast<unsigned>((31 - 4 * t - i) << 1) | (bits >> 31);
                    key[k] = c > key[k] ? c : key[k];
                }
            }
            const unsigned long long best = reduce_scatter8(key, t, [](unsigned long long a, unsigned long long b) { return a > b ? a : b; });
            val = static_cast<uint32_t>(best >> 6) | (static_cast<uint32_t>(best & 1u) << 31);
        }
        dd = __fdiv_rn(__uint_as_float(val), -8.0f);
    }
    const float id = (dd != 0.0f) ? __fdiv_rn(1.0f, dd) : 0.0f;
    const long long mine = p0 + 4 * (t >> 1);   // the pair of this lane's block
    if (mine < pairs) {
        const long long e = 2 * mine + (t & 1);
        d[e] = dd;
        m[e] = mm;
        if (zp != nullptr) zp[e] = (FORMAT == 0) ? 8 : 0;
    }
#pragma unroll
    for (int u = 0; u < WQ_PAIRS; u++) {
        uint32_t q[2] = {0u, 0u};
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int from = (lane & 24) + 2 * u + h;
            const float f = __shfl_sync(0xffffffffu, id, from), mn = (FORMAT == 1) ? __shfl_sync(0xffffffffu, mm, from) : 0.0f;
            const float4 x4 = h ? hi[u] : lo[u];
            const float x[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float v = (FORMAT == 1) ? rintf(__fmul_rn(__fsub_rn(x[i], mn), f)) : __fadd_rn(__fmul_rn(x[i], f), 8.5f);
                q[h] |= static_cast<uint32_t>(fminf(fmaxf(v, 0.0f), 15.0f)) << (8 * i);   // truncation, as astype(np.uint8) of a value in [0, 15]
            }
        }
        const long long p = p0 + 4 * u;
        if (p < pairs) {
            const uint32_t both = q[0] | (q[1] << 4);
            if (ALIGNED) {
                reinterpret_cast<uint32_t *>(nib)[p * 8 + t] = both;
            } else {
                for (int i = 0; i < 4; i++) nib[p * 32 + 4 * t + i] = static_cast<uint8_t>(both >> (8 * i));
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
