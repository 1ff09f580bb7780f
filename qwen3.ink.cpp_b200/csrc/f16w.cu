// fp16-weight matmul for few rows (lm_head: fp32 activations x fp16 weights, fp32 accumulate) and
// the CUDA-core weight-only W41 matmul (fp16 activations x dequantised Q4_1 weights).
//
// Neither has a C++ kernel in the reference.  lm_head follows the arithmetic of
// gemv_fp32_rcr_mt_impl_1 (qwen3/src/qwen/fp32_gemx_kernels_rcr.cc:494-507):
// logits[n] = sum_k x[k] * w[n][k].  Weight-only W41 follows
// notebooks/evaluate-qwen3_8b_W4.ipynb cell 13: the weight is replaced by
// w16 = fp16(q*d + m) and a stock fp16 linear with fp32 accumulation runs.
//
// k_f16w_rows (further down) serves rows of a multiple of 64 elements, k_f16w_gemv the others.
//
// k_f16w_gemv is bandwidth-bound: one warp per weight row, 128-bit streaming loads,
// eight loads in flight per lane, activations staged once per CTA in shared memory.
// Reduction order (fixed): lane l accumulates the 8-element chunks c with
// c % 32 == l in ascending order, then a 5-step xor-shuffle tree combines the lanes.
// Algorithmic bytes per launch: rows*K*2 weight bytes + M*K*4 activation bytes +
// M*rows*4 output bytes.
#include <cuda_fp16.h>

#include <type_traits>

#include "f16w_split.cuh"
#include "inkq_internal.h"
#include "ptx.cuh"

namespace inkq {

#ifndef INKQ_F16W_UNROLL
#define INKQ_F16W_UNROLL 8   // 16-byte loads in flight per lane (4: 5.3 TB/s, 8: 6.4 TB/s, 16: 6.0 TB/s on the 1.2 GB lm_head)
#endif
constexpr int F16W_UNROLL = INKQ_F16W_UNROLL;

template <int MT>
__global__ void __launch_bounds__(256) k_f16w_gemv(const uint16_t *__restrict__ w, const float *__restrict__ x, int m0, int M, int rows, int K,
                                                   float *__restrict__ C, int ldc, const ExtraDst extra)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float *xs = reinterpret_cast<float *>(smem_raw);  // [MT][K]
    const int mt = min(MT, M - m0);
    for (int i = threadIdx.x; i < MT * K / 4; i += blockDim.x) {
        const int r = (i * 4) / K;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < mt) v = reinterpret_cast<const float4 *>(x + static_cast<size_t>(m0) * K)[i];
        reinterpret_cast<float4 *>(xs)[i] = v;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int chunks = K / 8;
    for (int n = blockIdx.x * 8 + warp; n < rows; n += gridDim.x * 8) {
        const uint16_t *wrow = w + static_cast<size_t>(n) * K;
        float acc[MT];
#pragma unroll
        for (int j = 0; j < MT; j++) acc[j] = 0.0f;
        for (int c0 = lane; c0 < chunks; c0 += 32 * F16W_UNROLL) {
            uint4 v[F16W_UNROLL];
#pragma unroll
            for (int u = 0; u < F16W_UNROLL; u++) {
                const int c = c0 + u * 32;
                v[u] = (c < chunks) ? ldg_stream_v4(wrow + static_cast<size_t>(c) * 8) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < F16W_UNROLL; u++) {
                const int c = c0 + u * 32;
                if (c < chunks) {
                    const uint32_t wd[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
                    float wf[8];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&wd[i]));
                        wf[2 * i] = f.x;
                        wf[2 * i + 1] = f.y;
                    }
#pragma unroll
                    for (int j = 0; j < MT; j++) {
                        const float4 xa = *reinterpret_cast<const float4 *>(xs + j * K + c * 8);
                        const float4 xb = *reinterpret_cast<const float4 *>(xs + j * K + c * 8 + 4);
                        acc[j] = fmaf(xa.x, wf[0], acc[j]);
                        acc[j] = fmaf(xa.y, wf[1], acc[j]);
                        acc[j] = fmaf(xa.z, wf[2], acc[j]);
                        acc[j] = fmaf(xa.w, wf[3], acc[j]);
                        acc[j] = fmaf(xb.x, wf[4], acc[j]);
                        acc[j] = fmaf(xb.y, wf[5], acc[j]);
                        acc[j] = fmaf(xb.z, wf[6], acc[j]);
                        acc[j] = fmaf(xb.w, wf[7], acc[j]);
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < MT; j++) {
            float v = acc[j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
            if (lane == 0 && j < mt) {
                const size_t off = static_cast<size_t>(m0 + j) * ldc + n;
                C[off] = v;
#pragma unroll
                for (int e = 0; e < MAX_PEERS - 1; e++)   // further destinations (peers of a row-sharded matrix)
                    if (e < extra.n) extra.p[e][off] = v;
            }
        }
    }
}

// ---- up to 8 activation rows per pass, K a multiple of 64 ------------------------------------------------------------
// The CUDA-core kernel above needs, per weight and row, a conversion, an fp32 fma and its share of a 16-byte shared load: with
// four rows it is bound by instruction issue (4 rows 631 us for the 1.2 GB lm_head, 194 us with one).  Here 16 weight rows x 8
// activation rows x 16 k are one warp-level fp16 product with fp32 accumulation; the fp32 activations enter as an fp16 value and
// an fp16 remainder of the row scaled by a power of two (f16w_split.cuh: 22 significant bits), so both products are exact. Error
// against 64 bits, 2-norm: 1.2e-7 at K = 2048 and 4096, where the CUDA-core kernel's fp32 sums have 1.6e-7 and 2.1e-7.  A tile's
// K is split over the CTA's 16 warps, whose partial sums are added in ascending order.  A row's result does not depend on the
// rows beside it, and one row takes this kernel too: a batch gives the same bits as its rows one by one. Nine to 15 rows are two
// passes and read the weights twice (151936 x 4096: 9 rows 372 us, 15 rows 397, where 16 on the tensor cores take 280).
//
// Bound by the weight stream.  The weights come straight from global memory into A fragments: the order of k inside a product
// is free, so a lane takes 32 contiguous bytes of its two rows per 64 k - the fragments of four products, 128 bytes per row and
// request - and the activations are read alike.  Each lane keeps F16R_DEPTH such steps in flight across tile borders (128 KB
// per SM).  Measured (three matrices in turn): 151936 x 4096, 8 rows 1258 us on the CUDA cores, 230 with 64-byte pieces, 200 with
// slower preparation of the activations, 186 to 193 now (6.5 to 6.7 TB/s); one row 194 on the CUDA cores, 177 now (32000 x 4096:
// 54 -> 46, 151936 x 2048: 111 -> 102).
constexpr int F16R_WARPS = 16, F16R_DEPTH = 4, F16R_COLS = 8;

// bytes between two rows of the staged activations: 16 modulo 128, so that the 16-byte pieces of an 8-lane phase (two rows, every
// other piece of 128 bytes) fall into different banks
__host__ __device__ constexpr int f16r_pitch(int K) { return (K * 2 + 127) / 128 * 128 + 16; }

// One output in fp32, by one warp: for the outputs that the split operands cannot express
static __device__ __noinline__ float dot_f16w(const uint16_t *wrow, const float *xrow, int K, int lane)
{
    float acc = 0.0f;
    for (int i = lane; i < K / 4; i += 32) {
        const float4 v = reinterpret_cast<const float4 *>(xrow)[i];
        const __half2 *p = reinterpret_cast<const __half2 *>(wrow + i * 4);
        const float2 a = __half22float2(p[0]), b = __half22float2(p[1]);
        acc = fmaf(v.x, a.x, acc);
        acc = fmaf(v.y, a.y, acc);
        acc = fmaf(v.z, b.x, acc);
        acc = fmaf(v.w, b.y, acc);
    }
    for (int o = 16; o > 0; o >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, o));
    return acc;
}

__global__ void __launch_bounds__(F16R_WARPS * 32, 1)
    k_f16w_rows(const uint16_t *__restrict__ w, const float *__restrict__ x, int m0, int mt, int rows, int K, float *__restrict__ C, int ldc, const ExtraDst extra)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int pitch = f16r_pitch(K);
    unsigned char *xh = smem_raw, *xl = xh + F16R_COLS * pitch;                                  // [8][K] fp16 value and remainder
    float *part = reinterpret_cast<float *>(xl + F16R_COLS * pitch);                              // [2][warps][8 columns][16 rows]
    float *inv = part + 2 * F16R_WARPS * F16R_COLS * 16;                                           // [8] 2^-e of a row
    int *has_nan = reinterpret_cast<int *>(inv + F16R_COLS);                                       // [8]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int k64 = K / 64, steps = (k64 + F16R_WARPS - 1) / F16R_WARPS;                          // steps of 64 k per warp and tile
    const int tiles = (rows + 15) / 16;

    uint4 a[F16R_DEPTH][2][2];                                                                    // rows g and g + 8, 16 k each
    int ptile = blockIdx.x, ps = 0;                                                               // next step to request
    auto request = [&](uint4 (&v)[2][2]) {
        const int k = warp * steps + ps, r0 = ptile * 16 + g;
        v[0][0] = v[0][1] = v[1][0] = v[1][1] = make_uint4(0, 0, 0, 0);
        if (ptile < tiles && k < k64) {
            const uint16_t *src = w + static_cast<size_t>(r0) * K + k * 64 + t * 16;
            if (r0 < rows) ldg_stream_v8(src, v[0][0], v[0][1]);
            if (r0 + 8 < rows) ldg_stream_v8(src + static_cast<size_t>(8) * K, v[1][0], v[1][1]);
        }
        if (++ps == steps) {
            ps = 0;
            ptile += gridDim.x;
        }
    };
#pragma unroll
    for (int u = 0; u < F16R_DEPTH; u++) request(a[u]);
    // everything above reads weights only; below, the activations of the kernel before this one in the stream
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // 16, 8, 4 or 2 warps per row, whatever the number of rows leaves: scale and split (f16w_split.cuh).  Rows past mt stay
    // as they are: each only feeds its own column, which is not stored.  (Two warps per row whatever their number, each
    // scanning all of it: 3 us before the first product.)
    {
        const int wpr = F16R_WARPS / (mt > 4 ? 8 : mt > 2 ? 4 : mt), m = warp / wpr, n4 = K / 4, first = (warp % wpr) * 32 + lane;
        const float4 *row = reinterpret_cast<const float4 *>(x + static_cast<size_t>(m0 + m) * K);
        float amax = 0.f;
        if (m < mt) {
#pragma unroll 8
            for (int i = first; i < n4; i += wpr * 32) amax = absmax_nan(amax, row[i]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = absmax_nan(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        if (lane == 0) part[warp] = amax;   // (free until the first tile is complete)
        __syncthreads();
        amax = 0.f;
        for (int i = 0; i < wpr; i++) amax = absmax_nan(amax, part[m * wpr + i]);
        if (m < mt) {
            const bool special = !(amax <= FLT_MAX);
            if (first == 0) has_nan[m] = amax != amax;
            if (special) amax = finite_absmax(row, n4, lane);
            const int e = split_exponent(amax);
            const float sc = ldexpf(1.0f, e);
            if (first == 0) inv[m] = ldexpf(1.0f, -e);
            auto split_row = [&](auto with_special) {
#pragma unroll 4
                for (int i = first; i < n4; i += wpr * 32) {
                    __half2 h[2], l[2];
                    split4<decltype(with_special)::value>(row[i], sc, h, l);
                    __half2 *oh = reinterpret_cast<__half2 *>(xh + m * pitch + i * 8), *ol = reinterpret_cast<__half2 *>(xl + m * pitch + i * 8);
                    oh[0] = h[0];
                    oh[1] = h[1];
                    ol[0] = l[0];
                    ol[1] = l[1];
                }
            };
            if (special) split_row(std::true_type{});
            else split_row(std::false_type{});
        }
    }
    __syncthreads();

    const unsigned char *bh = xh + g * pitch + t * 32, *bl = xl + g * pitch + t * 32;            // column g of the activations
    int tile = blockIdx.x, s = 0, buf = 0;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    while (tile < tiles) {
#pragma unroll
        for (int u = 0; u < F16R_DEPTH; u++) {
            if (tile < tiles) {   // uniform over the CTA
                const int k = warp * steps + s;
                if (k < k64) {
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const uint4 h = *reinterpret_cast<const uint4 *>(bh + k * 128 + i * 16), l = *reinterpret_cast<const uint4 *>(bl + k * 128 + i * 16);
                        const uint4 &p = a[u][0][i], &q = a[u][1][i];
                        float sum[4] = {0.f, 0.f, 0.f, 0.f};   // the products' own accumulation truncates: 32 terms at a time, rounded sums beyond
                        mma_f16_16x8x16(sum, p.x, q.x, p.y, q.y, l.x, l.y);
                        mma_f16_16x8x16(sum, p.z, q.z, p.w, q.w, l.z, l.w);
                        mma_f16_16x8x16(sum, p.x, q.x, p.y, q.y, h.x, h.y);
                        mma_f16_16x8x16(sum, p.z, q.z, p.w, q.w, h.z, h.w);
#pragma unroll
                        for (int e = 0; e < 4; e++) acc[e] = __fadd_rn(acc[e], sum[e]);
                    }
                }
                request(a[u]);
                if (++s == steps) {   // the tile is complete: add the warps' partials
                    float *p = part + (buf * F16R_WARPS + warp) * (F16R_COLS * 16);
                    p[(2 * t) * 16 + g] = acc[0];
                    p[(2 * t + 1) * 16 + g] = acc[1];
                    p[(2 * t) * 16 + g + 8] = acc[2];
                    p[(2 * t + 1) * 16 + g + 8] = acc[3];
                    __syncthreads();
                    if (threadIdx.x < F16R_COLS * 16) {
                        const int c = threadIdx.x >> 4, n = tile * 16 + (threadIdx.x & 15);
                        const float *q = part + buf * F16R_WARPS * (F16R_COLS * 16) + threadIdx.x;
                        float v = q[0];
#pragma unroll
                        for (int i = 1; i < F16R_WARPS; i++) v = __fadd_rn(v, q[i * (F16R_COLS * 16)]);
                        const bool mine = c < mt && n < rows;
                        if (mine) v *= inv[c];   // exact: a power of two
                        // An infinite weight meets remainders of zero or of the other sign: a NaN that no fp32 evaluation has
                        for (unsigned redo = __ballot_sync(0xffffffffu, mine && v != v && has_nan[c] == 0); redo != 0; redo &= redo - 1) {
                            const int from = __ffs(redo) - 1;
                            const float y = dot_f16w(w + static_cast<size_t>(tile * 16 + (from & 15)) * K, x + static_cast<size_t>(m0 + warp * 2 + (from >> 4)) * K, K, lane);
                            if (lane == from) v = y;
                        }
                        if (mine) {
                            const size_t off = static_cast<size_t>(m0 + c) * ldc + n;
                            C[off] = v;
#pragma unroll
                            for (int e = 0; e < MAX_PEERS - 1; e++)
                                if (e < extra.n) extra.p[e][off] = v;
                        }
                    }
                    buf ^= 1;
                    s = 0;
                    tile += gridDim.x;
                    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
                }
            }
        }
    }
}

int launch_f16w_matmul(inkq_ctx *ctx, const F16W *w, const float *x, int M, float *C, int ldc, const ExtraDst *extra_in)
{
    ExtraDst extra = {};
    if (extra_in != nullptr) extra = *extra_in;
    const int grid = min((w->rows + 7) / 8, ctx->num_sms * 8);
    const size_t rows_smem = static_cast<size_t>(2 * F16R_COLS) * f16r_pitch(w->K) + sizeof(float) * (2 * F16R_WARPS * F16R_COLS * 16 + 2 * F16R_COLS);
    if (w->K % 64 == 0 && rows_smem <= 226 * 1024) {
        int rc = allow_smem<k_f16w_rows>(ctx);
        if (rc) return rc;
        const int tiles = (w->rows + 15) / 16;
        for (int m0 = 0; m0 < M; m0 += F16R_COLS) {
            const cudaError_t e = launch_pdl(k_f16w_rows, dim3(min(tiles, ctx->num_sms)), dim3(F16R_WARPS * 32), rows_smem, ctx->stream, w->w, x, m0,
                                             min(F16R_COLS, M - m0), w->rows, w->K, C, ldc, extra);
            if (e != cudaSuccess) return fail(ctx, INKQ_ERR_CUDA, std::string("k_f16w_rows launch: ") + cudaGetErrorString(e));
            if ((rc = after_launch(ctx, "k_f16w_rows"))) return rc;
        }
        return INKQ_OK;
    }
    // other row lengths: one or four rows per pass on the CUDA cores
    if (M == 1) {
        const size_t smem = static_cast<size_t>(w->K) * sizeof(float);
        const int rc = allow_smem<k_f16w_gemv<1>>(ctx);
        if (rc) return rc;
        k_f16w_gemv<1><<<grid, 256, smem, ctx->stream>>>(w->w, x, 0, M, w->rows, w->K, C, ldc, extra);
        return after_launch(ctx, "k_f16w_gemv");
    }
    const size_t smem = 4 * static_cast<size_t>(w->K) * sizeof(float);
    if (smem > 200 * 1024) return fail(ctx, INKQ_ERR_UNSUPPORTED, "K too large for the fp16-weight matmul");
    int rc = allow_smem<k_f16w_gemv<4>>(ctx);
    for (int m0 = 0; m0 < M && !rc; m0 += 4) {
        k_f16w_gemv<4><<<grid, 256, smem, ctx->stream>>>(w->w, x, m0, M, w->rows, w->K, C, ldc, extra);
        rc = after_launch(ctx, "k_f16w_gemv");
    }
    return rc;
}

// Weight-only W41 on the CUDA cores (cross-check of the tensor-core kernel): one output per thread,
// k ascending, fp32 accumulate: acc = fma(a16[k], w16, acc) with w16 = the half-precision fma q*d + m
// (one rounding), d and m the layer's fp16 scales.
__global__ void __launch_bounds__(256) k_gemm_w41_f16act(Weight w, const __half *__restrict__ a, int M, float *__restrict__ C, int ldc)
{
    const int n = blockIdx.x * 32 + (threadIdx.x & 31);
    const int m = blockIdx.y * 8 + (threadIdx.x >> 5);
    if (n >= w.rows || m >= M) return;
    const int t = n / TILE_N, r = n % TILE_N;
    const __half *arow = a + static_cast<size_t>(m) * w.K;
    float acc = 0.0f;
    for (int p = 0; p < w.pairs; p++) {
        const uint4 c0 = *reinterpret_cast<const uint4 *>(w.nibT + nib_offset(w.pairs, t, p, r, 0));
        const uint4 c1 = *reinterpret_cast<const uint4 *>(w.nibT + nib_offset(w.pairs, t, p, r, 1));
        const size_t rec = (static_cast<size_t>(t) * w.pairs + p) * TILE_N + r;
        const uint2 pk = w.sc16[rec];
        const __half2 d2 = *reinterpret_cast<const __half2 *>(&pk.x), m2 = *reinterpret_cast<const __half2 *>(&pk.y);
        const uint32_t wd[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
        for (int hi = 0; hi < 2; hi++) {
            const __half dd = hi ? __high2half(d2) : __low2half(d2), mm = hi ? __high2half(m2) : __low2half(m2);
#pragma unroll
            for (int e = 0; e < 32; e++) {
                const uint32_t nibble = (wd[e >> 2] >> (8 * (e & 3) + 4 * hi)) & 0xf;
                const float wv = __half2float(__hfma(__ushort2half_rn(static_cast<unsigned short>(nibble)), dd, mm));
                acc = fmaf(__half2float(arow[p * 64 + hi * 32 + e]), wv, acc);
            }
        }
    }
    C[static_cast<size_t>(m) * ldc + n] = acc;
}

int launch_gemm_w41_f16(inkq_ctx *ctx, const uint16_t *a16, int M, const Weight *w, float *C, int ldc)
{
    dim3 grid((w->rows + 31) / 32, (M + 7) / 8);
    k_gemm_w41_f16act<<<grid, 256, 0, ctx->stream>>>(*w, reinterpret_cast<const __half *>(a16), M, C, ldc);
    return after_launch(ctx, "k_gemm_w41_f16act");
}

}  // namespace inkq
