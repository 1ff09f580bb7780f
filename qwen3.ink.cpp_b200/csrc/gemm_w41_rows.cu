// Weight-only W41 for a few activation rows (up to 16; one row of a wide layer takes gemv_w41.cu): fp16 activations x Q4_1
// weights dequantised in registers, warp-level fp16 products with fp32 accumulation.
//
// No C++ kernel exists in the reference for this scheme; it follows notebooks/evaluate-qwen3_8b_W4.ipynb cell 13, like the
// tensor-core kernel (qgemm_w41_tc.cu), and dequantises alike:  w16[n][k] = fp16(q[n][k] * d[n][k/32] + m[n][k/32])  with one
// rounding, C[m][n] = sum_k a16[m][k] * w16[n][k].
//
// The least it has to move is the weight stream (0.625 bytes per weight), which it reaches a third of: 12288 x 4096 with 8 rows
// 13.6 us = 2.35 TB/s, with 16 rows 16.4; 24576 x 4096 24.6 = 2.6 TB/s; 4096 x 4096 5.3.  Dequantising and multiplying is 12.4k
// instructions per scheduler (6.3 us of the 13.6); for the rest the 16 warps of an SM wait for loads of 32 bytes per row and
// request.  The tensor-core kernel dequantises every stage for its tile whatever the number of rows: 29 us for 12288 x 4096 from
// 2 to 64 rows when this kernel took its place, 21 today.  Here the packed weights go from global memory straight into A
// fragments: the order of k inside a product is free, so a lane takes 8 contiguous bytes of its two rows per pair of blocks - 8
// weights of the low and 8 of the high block, the fragments of four products - and the activations, staged once per CTA in shared
// memory, are read alike.  A tile of 16 weight rows is split along K over the CTA's 16 warps, so the work is even to one tile per
// SM; each lane keeps DEPTH pairs in flight across tile borders. The products of one pair accumulate from zero and are added to
// the running sums in fp32 (the hardware's own accumulation truncates), the warps' partials are added in ascending order.
#include <cuda_fp16.h>

#include "inkq_internal.h"
#include "ptx.cuh"

namespace inkq {
namespace w41rows {

constexpr int WARPS = 16, DEPTH = 8;

// bytes between two rows of the staged activations: 64 modulo 128, so that the rows of an 8-lane phase fall into different banks
__host__ __device__ constexpr int pitch_for(int K) { return (K * 2 + 127) / 128 * 128 + 64; }

struct Step {   // one pair of blocks: 8 packed bytes and the fp16 {d_lo, d_hi, m_lo, m_hi} of rows g and g + 8
    uint2 w[2], sc[2];
};

// four nibbles (one per byte) -> four fp16 weights: 1024 + q by byte placement, - 1024 exact, one rounding of q * d + m
__device__ __forceinline__ void dequant4(uint32_t nib, __half2 d2, __half2 m2, uint32_t &o01, uint32_t &o23)
{
    const uint32_t h01 = __byte_perm(nib, 0x64646464u, 0x4140), h23 = __byte_perm(nib, 0x64646464u, 0x4342);
    const __half2 k1024 = __half2half2(__ushort_as_half(0x6400));
    const __half2 w01 = __hfma2(__hsub2(*reinterpret_cast<const __half2 *>(&h01), k1024), d2, m2);
    const __half2 w23 = __hfma2(__hsub2(*reinterpret_cast<const __half2 *>(&h23), k1024), d2, m2);
    o01 = *reinterpret_cast<const uint32_t *>(&w01);
    o23 = *reinterpret_cast<const uint32_t *>(&w23);
}

// NT: 8-row groups of activations.
template <int NT>
__global__ void __launch_bounds__(WARPS * 32, 1) k_gemm_w41_rows(const uint8_t *__restrict__ nibT, const uint2 *__restrict__ sc16, const uint16_t *__restrict__ a16,
                                                                 int M, int rows, int K, float *__restrict__ C, int ldc)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int pitch = pitch_for(K), pairs = K / 64, steps = (pairs + WARPS - 1) / WARPS;
    constexpr int TILE = 8 * NT * 16;                                                    // outputs of a tile
    unsigned char *xs = smem_raw;                                                        // [8 NT][K] fp16
    float *part = reinterpret_cast<float *>(xs + 8 * NT * pitch);                         // [2][warps][8 NT columns][16 rows]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int tiles = (rows + 15) / 16;

    Step st[DEPTH];
    int ptile = blockIdx.x, ps = 0;                                                      // next step to request
    auto request = [&](Step &v) {
        const int p = warp * steps + ps;
        v.w[0] = v.w[1] = v.sc[0] = v.sc[1] = make_uint2(0, 0);
        if (ptile < tiles && p < pairs) {   // (the layout pads rows to whole 128-row tiles)
            const int r = (ptile & 7) * 16 + g;
            const size_t rec = (static_cast<size_t>(ptile >> 3) * pairs + p) * TILE_N + r;
#pragma unroll
            for (int h = 0; h < 2; h++) {   // rows g + 8 h share the chunk swizzle bit of row g only up to (r >> 2) & 1
                const int swz = ((r + 8 * h) >> 2) & 1;
                v.w[h] = ldg_stream_v2(nibT + (rec + 8 * h) * 32 + (((t >> 1) ^ swz) << 4) + (t & 1) * 8);
                v.sc[h] = ldg_stream_v2(sc16 + rec + 8 * h);
            }
        }
        if (++ps == steps) {
            ps = 0;
            ptile += gridDim.x;
        }
    };
#pragma unroll
    for (int u = 0; u < DEPTH; u++) request(st[u]);
    // everything above reads weights only; below, the activations of the kernel before this one in the stream
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (int i = threadIdx.x; i < 8 * NT * (K / 8); i += WARPS * 32) {
        const int m = i / (K / 8), c = i % (K / 8);
        uint4 v = make_uint4(0, 0, 0, 0);
        if (m < M) v = *reinterpret_cast<const uint4 *>(a16 + static_cast<size_t>(m) * K + c * 8);
        *reinterpret_cast<uint4 *>(xs + m * pitch + c * 16) = v;
    }
    __syncthreads();

    const unsigned char *bx = xs + g * pitch + t * 16;                                   // column g of the first group
    int tile = blockIdx.x, s = 0, buf = 0;
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    while (tile < tiles) {
#pragma unroll
        for (int u = 0; u < DEPTH; u++) {
            if (tile < tiles) {   // uniform over the CTA
                const int p = warp * steps + s;
                if (p < pairs) {
                    uint32_t a[2][2][4];   // [block][row half][halves 8t .. 8t + 7]
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const __half2 d = *reinterpret_cast<const __half2 *>(&st[u].sc[h].x), m = *reinterpret_cast<const __half2 *>(&st[u].sc[h].y);
#pragma unroll
                        for (int b = 0; b < 2; b++) {
                            const __half2 d2 = b ? __high2half2(d) : __low2half2(d), m2 = b ? __high2half2(m) : __low2half2(m);
                            dequant4((b ? st[u].w[h].x >> 4 : st[u].w[h].x) & 0x0F0F0F0Fu, d2, m2, a[b][h][0], a[b][h][1]);
                            dequant4((b ? st[u].w[h].y >> 4 : st[u].w[h].y) & 0x0F0F0F0Fu, d2, m2, a[b][h][2], a[b][h][3]);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < NT; j++) {
                        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                        for (int b = 0; b < 2; b++) {
                            const uint4 x = *reinterpret_cast<const uint4 *>(bx + j * 8 * pitch + p * 128 + b * 64);
                            mma_f16_16x8x16(sum, a[b][0][0], a[b][1][0], a[b][0][1], a[b][1][1], x.x, x.y);
                            mma_f16_16x8x16(sum, a[b][0][2], a[b][1][2], a[b][0][3], a[b][1][3], x.z, x.w);
                        }
#pragma unroll
                        for (int i = 0; i < 4; i++) acc[j][i] = __fadd_rn(acc[j][i], sum[i]);
                    }
                }
                request(st[u]);
                if (++s == steps) {   // the tile is complete: add the warps' partials
                    float *q = part + (buf * WARPS + warp) * TILE;
#pragma unroll
                    for (int j = 0; j < NT; j++)
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            q[(j * 8 + 2 * t + (i & 1)) * 16 + g + 8 * (i >> 1)] = acc[j][i];
                            acc[j][i] = 0.f;
                        }
                    __syncthreads();
                    if (threadIdx.x < TILE) {
                        const int m = threadIdx.x >> 4, n = tile * 16 + (threadIdx.x & 15);
                        const float *r = part + buf * WARPS * TILE + threadIdx.x;
                        float v = r[0];
#pragma unroll
                        for (int i = 1; i < WARPS; i++) v = __fadd_rn(v, r[i * TILE]);
                        if (m < M && n < rows) C[static_cast<size_t>(m) * ldc + n] = v;
                    }
                    buf ^= 1;
                    s = 0;
                    tile += gridDim.x;
                }
            }
        }
    }
}

}  // namespace w41rows

bool gemm_w41_rows_fits(const uint16_t *a16, int M, int K)
{
    using namespace w41rows;
    const int nt = (M + 7) / 8;
    return nt <= 2 && (reinterpret_cast<uintptr_t>(a16) & 15) == 0 && 8 * nt * (pitch_for(K) + 2 * WARPS * 16 * static_cast<int>(sizeof(float))) <= 226 * 1024;
}

template <int NT>
static int launch_rows(inkq_ctx *ctx, const uint16_t *a16, int M, const Weight *w, float *C, int ldc)
{
    using namespace w41rows;
    const int rc = allow_smem<k_gemm_w41_rows<NT>>(ctx);
    if (rc) return rc;
    const int tiles = (w->rows + 15) / 16;
    const cudaError_t e = launch_pdl(k_gemm_w41_rows<NT>, dim3(tiles < ctx->num_sms ? tiles : ctx->num_sms), dim3(WARPS * 32),
                                     8 * NT * (pitch_for(w->K) + 2 * WARPS * 16 * static_cast<int>(sizeof(float))), ctx->stream, w->nibT, w->sc16, a16, M,
                                     w->rows, w->K, C, ldc);
    if (e != cudaSuccess) return fail(ctx, INKQ_ERR_CUDA, std::string("k_gemm_w41_rows launch: ") + cudaGetErrorString(e));
    return after_launch(ctx, "k_gemm_w41_rows");
}

int launch_gemm_w41_rows(inkq_ctx *ctx, const uint16_t *a16, int M, const Weight *w, float *C, int ldc)
{
    return M <= 8 ? launch_rows<1>(ctx, a16, M, w, C, ldc) : launch_rows<2>(ctx, a16, M, w, C, ldc);
}

}  // namespace inkq
