// QGEMM for a few activation rows (2 to 32: sequences decoded together, short prompts): warp-level int8 matrix products
// whose block dots are scaled where they appear, in registers.
//
// Stands in for gemm_repack_A81W41_fp32 (qwen3/src/qwen/quantized_gemx_kernels.cc:349-582)
// and gemm_repack_A80W40 (:195-347); A80W4Z has no reference kernel and follows the A80W40
// code with q_w = nibble - zp.  Same result bits as qgemm_tc.cu, which serves more rows.
//
//   C[m][n] = sum over 32-element blocks b of  d_a[m,b]*d_w[n,b]*I[m,n,b] + m_w[n,b]*s_a[m,b]
//   I[m,n,b] = sum_e q_a[m,32b+e] * q_w[n,32b+e]                       (exact int32)
//
// What bounds it: the weight stream, and for layers with few rows the chain of a warp's dependent instructions over K (the
// reference's order forbids splitting an output's sum).  mma.sync.m16n8k32 leaves the 16 x 8 dots of one block (K = 32)
// in the registers of the threads that scale them, so there is no tensor-memory round trip and no hand-shake between warps,
// which cost the tcgen05 kernel ~350 cycles per pair of blocks however narrow the tile.  Every warp owns 16 weight rows
// and all columns: each weight byte is fetched once.  Stages of four pairs (256 K-elements) are unrolled, so that
// the fragment loads and products of one pair overlap the scaling of the one before.  Measured (prefetched weights of
// distinct layers, A81W41): 24576 x 4096 with 5 rows 59 -> 15 us (4.2 TB/s), 4096 x 4096 with 5 rows 37 -> 8.5 us.
//
// Operands: the weights are the MMA's A side, the activation rows its B side.  A packed byte holds element e of both blocks of
// a pair, so one ldmatrix.x4 fetches the A fragments of two blocks.  Stages pass through a ring in shared memory: tiled TMA
// copies of the activations (128-byte swizzle, rows past M zero-filled) and of their planes d and s, bulk copies of the packed
// weights, their scale records and zero points.  Layers whose scales were rounded to fp16 read the 8-byte fp16 records, the
// others the 16-byte fp32 ones: the values are the same, the stream is 17 % shorter.  The warps take turns at issuing a
// stage's copies.  Every mbarrier wait is bounded; when one runs out the kernel sets a device flag, every later wait returns
// at once, all loops run to their end inside their buffers and the host reports INKQ_ERR_TIMEOUT with the context usable.
//
// Operation order per output (bit-identical to the reference): for each pair of blocks ascending:
// acc = fma((float)I_lo, d_a_lo*d_w_lo, acc); fma((float)I_hi, ...); acc = fma(m_lo, s_a_lo, acc); fma(m_hi, s_a_hi, acc).
#include <cuda.h>
#include <cuda_fp16.h>

#include <mutex>

#include "inkq_internal.h"
#include "ptx.cuh"

namespace inkq {
namespace qrows {

constexpr int SP = 4;             // pairs per stage
constexpr int MAX_STAGES = 8;
constexpr int SMEM_ONE_CTA = 116 * 1024;   // more than half of an SM's shared memory
constexpr int SMEM_CTA = 111 * 1024;       // two CTAs per SM

struct Params {
    const uint8_t *nibT;
    const unsigned char *sc;   // fp16 or fp32 scale records
    const uchar2 *zpT;
    float *C;
    ExtraDst extra;   // further destinations of every C element (peers of a column-sharded layer)
    int *flag;
    int M, rows, pairs, ldc;
};

// SCH: weight scheme; S16: fp16 scale records; WR: warps (16 weight rows each); NT: 8-column groups.
template <int SCH, bool S16, int WR, int NT>
struct Cfg {
    static constexpr int ROWS = 16 * WR, BM = 8 * NT, THREADS = 32 * WR;
    static constexpr int PLANES = (SCH == INKQ_A81W41) ? 2 : 1;
    static constexpr int Q_BYTES = BM * 64 * SP, PLANE_BYTES = 2 * SP * BM * 4;
    static constexpr int W_PAIR = ROWS * 32, SC_REC = S16 ? 8 : 16, SC_PAIR = ROWS * SC_REC, Z_PAIR = (SCH == INKQ_A80W4Z) ? ROWS * 2 : 0;
    static constexpr int W_OFF = Q_BYTES, SC_OFF = W_OFF + SP * W_PAIR, Z_OFF = SC_OFF + SP * SC_PAIR, D_OFF = Z_OFF + SP * Z_PAIR, S_OFF = D_OFF + PLANE_BYTES;
    static constexpr int STAGE_BYTES = (D_OFF + PLANES * PLANE_BYTES + 1023) / 1024 * 1024;
    static constexpr int FIT = (SMEM_CTA - 1024 - 256) / STAGE_BYTES, STAGES = FIT > MAX_STAGES ? MAX_STAGES : FIT;
    static constexpr int LEAD = STAGES >= 4 ? STAGES - 2 : STAGES - 1;   // stages requested ahead of the one being multiplied
    static constexpr int SMEM = 1024 + STAGES * STAGE_BYTES + 256;
    static_assert(STAGES >= 3, "shared memory budget");
    static_assert(TILE_N % ROWS == 0, "a CTA's rows lie inside one weight tile");
};

__device__ __forceinline__ void mma_block(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}

// Bounded wait: one probe in the common case, then probes until the phase completes, another warp has given up or the
// limit runs out.  Always returns; after an abort the warps finish their loops without waiting.
__device__ __forceinline__ void wait_bounded(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int *dev_flag)
{
    if (mbar_try_wait(bar, parity)) return;
    const long long t0 = clock64();
#pragma unroll 1
    for (uint32_t spin = 1;; spin++) {
        if (mbar_try_wait(bar, parity)) return;
        if ((spin & 31u) == 0u) {
            if (*abort_flag != 0) return;
            if (clock64() - t0 > INKQ_SPIN_LIMIT_CYCLES) {
                *abort_flag = 1;
                atomicExch(dev_flag, 1);
                return;
            }
        }
    }
}

template <int SCH, bool S16, int WR, int NT>
__global__ void __launch_bounds__(32 * WR, 2)
    k_qgemm_rows(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_d, const __grid_constant__ CUtensorMap map_s,
                 const Params prm)
{
    using G = Cfg<SCH, S16, WR, NT>;
    constexpr bool HAS_MIN = SCH == INKQ_A81W41;
    constexpr int STAGES = G::STAGES, LEAD = G::LEAD;
    extern __shared__ __align__(1024) unsigned char smem_dyn[];
    unsigned char *smem = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES * G::STAGE_BYTES), *empty = full + STAGES;
    volatile int *abort_flag = reinterpret_cast<volatile int *>(empty + STAGES);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row_base = blockIdx.x * G::ROWS, row_in_tile = row_base % TILE_N;   // first weight row of the CTA
    const size_t slab = static_cast<size_t>(row_base / TILE_N) * prm.pairs;
    const int k_stages = (prm.pairs + SP - 1) / SP;

    // `bytes` per row of pairs p0 .. p0 + np - 1 out of a [tile][pair][128 rows] array
    auto copy_rows = [&](unsigned char *dst, const void *src, int bytes, size_t p0, int np, uint64_t *bar) {
        const unsigned char *s = static_cast<const unsigned char *>(src) + (p0 * TILE_N + row_in_tile) * bytes;
        if (G::ROWS == TILE_N) tma_bulk_g2s(dst, s, np * (TILE_N * bytes), bar);   // the pairs are contiguous
        else
            for (int p = 0; p < np; p++) tma_bulk_g2s(dst + p * (G::ROWS * bytes), s + p * (TILE_N * bytes), G::ROWS * bytes, bar);
    };
    // the part of a stage that no earlier kernel of the stream writes
    auto issue_weights = [&](int ks, int slot) {
        const int np = min(SP, prm.pairs - ks * SP);
        unsigned char *st = smem + slot * G::STAGE_BYTES;
        mbar_arrive_expect_tx(&full[slot], G::Q_BYTES + G::PLANES * G::PLANE_BYTES + np * (G::W_PAIR + G::SC_PAIR + G::Z_PAIR));
        const size_t p0 = slab + static_cast<size_t>(ks) * SP;
        copy_rows(st + G::W_OFF, prm.nibT, 32, p0, np, &full[slot]);
        copy_rows(st + G::SC_OFF, prm.sc, G::SC_REC, p0, np, &full[slot]);
        if (SCH == INKQ_A80W4Z) copy_rows(st + G::Z_OFF, prm.zpT, 2, p0, np, &full[slot]);
    };
    auto issue_activations = [&](int ks, int slot) {   // boxes are always full size; parts out of range arrive as zeros
        unsigned char *st = smem + slot * G::STAGE_BYTES;
#pragma unroll
        for (int b = 0; b < SP / 2; b++) tma_tensor2d_g2s(st + b * (G::BM * 128), &map_q, ks * (64 * SP) + b * 128, 0, &full[slot]);
        tma_tensor2d_g2s(st + G::D_OFF, &map_d, 0, ks * (2 * SP), &full[slot]);
        if (G::PLANES == 2) tma_tensor2d_g2s(st + G::S_OFF, &map_s, 0, ks * (2 * SP), &full[slot]);
    };

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], WR);
        }
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&map_q);
        tma_prefetch_desc(&map_d);
        if (G::PLANES == 2) tma_prefetch_desc(&map_s);
        for (int ks = 0; ks < LEAD && ks < k_stages; ks++) issue_weights(ks, ks);
    }
    // Launched with programmatic stream serialization: everything above may overlap the tail of the kernel before this one
    // (normally the quantizer that writes the activations); nothing below may.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0) {
        for (int ks = 0; ks < LEAD && ks < k_stages; ks++) issue_activations(ks, ks);
    }
    __syncthreads();

    const int row0 = warp * 16;                              // the warp's first row inside the CTA's tile
    const int g = lane >> 2, t2 = (lane & 3) * 2;            // fragment coordinates: rows g, g + 8; columns t2, t2 + 1
    // ldmatrix row addresses.  A: matrices (rows 0-7, chunk 0), (rows 8-15, chunk 0), (rows 0-7, chunk 1), (rows 8-15, chunk 1)
    const int a_row = row0 + ((lane >> 3) & 1) * 8 + (lane & 7);
    const uint32_t a_off = G::W_OFF + a_row * 32 + ((((lane >> 4) & 1) ^ ((a_row >> 2) & 1)) << 4);
    // B: matrix j = 16-byte chunk j of a pair's 64 bytes (low block: chunks 0, 1; high block: 2, 3); rows of 128 B, swizzled;
    // the second pair of a row lies at this offset with bit 6 flipped
    const uint32_t b_off = (lane & 7) * 128 + (((lane >> 3) ^ (lane & 7)) << 4);
    const uint32_t base = smem_u32(smem);

    unsigned long long acc[NT][2];   // columns (t2, t2 + 1) of rows g and g + 8
#pragma unroll
    for (int j = 0; j < NT; j++) acc[j][0] = acc[j][1] = 0ull;

    auto multiply_pair = [&](int pj, uint32_t st) {
        uint32_t pk[4], alo[4], ahi[4];
        ldmatrix_x4(pk, st + a_off + pj * G::W_PAIR);
        float4 w[2];   // {d_lo, d_hi, m_lo, m_hi} of rows g and g + 8
        uint32_t z_lo[2] = {0u, 0u}, z_hi[2] = {0u, 0u};
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = row0 + g + 8 * h;
            if (S16) {
                const uint2 p = lds_u32x2(st + G::SC_OFF + pj * G::SC_PAIR + r * 8);
                const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&p.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&p.y));
                w[h] = make_float4(a.x, a.y, b.x, b.y);
            } else {
                w[h] = lds_f4(st + G::SC_OFF + pj * G::SC_PAIR + r * 16);
            }
            if (SCH == INKQ_A80W40) z_lo[h] = z_hi[h] = 0x08080808u;
            if (SCH == INKQ_A80W4Z) {
                const uint32_t z = lds_u16(st + G::Z_OFF + pj * G::Z_PAIR + r * 2);
                z_lo[h] = (z & 0xFFu) * 0x01010101u;
                z_hi[h] = (z >> 8) * 0x01010101u;
            }
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {   // registers 0, 2: row g; 1, 3: row g + 8
            alo[e] = pk[e] & 0x0F0F0F0Fu;
            ahi[e] = (pk[e] >> 4) & 0x0F0F0F0Fu;
            if (!HAS_MIN) {   // byte-wise (nibble - z) without borrows between bytes: set bit 7, subtract, clear
                alo[e] = ((alo[e] | 0x80808080u) - z_lo[e & 1]) ^ 0x80808080u;
                ahi[e] = ((ahi[e] | 0x80808080u) - z_hi[e & 1]) ^ 0x80808080u;
            }
        }
#pragma unroll
        for (int j = 0; j < NT; j++) {
            uint32_t b[4];
            ldmatrix_x4(b, st + (pj >> 1) * (G::BM * 128) + (b_off ^ ((pj & 1) << 6)) + j * (8 * 128));
            int lo[4], hi[4];
            mma_block(lo, alo, b[0], b[1]);
            mma_block(hi, ahi, b[2], b[3]);
            const uint32_t pl = st + (2 * pj) * (G::BM * 4) + (j * 8 + t2) * 4;
            const unsigned long long d_lo = lds_u64(pl + G::D_OFF), d_hi = lds_u64(pl + G::D_OFF + G::BM * 4);
            unsigned long long s_lo = 0ull, s_hi = 0ull;
            if (HAS_MIN) {
                s_lo = lds_u64(pl + G::S_OFF);
                s_hi = lds_u64(pl + G::S_OFF + G::BM * 4);
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                unsigned long long a = acc[j][h];
                a = fma2(cvt2_exact(lo[2 * h], lo[2 * h + 1]), mul2(d_lo, pack2(w[h].x, w[h].x)), a);
                a = fma2(cvt2_exact(hi[2 * h], hi[2 * h + 1]), mul2(d_hi, pack2(w[h].y, w[h].y)), a);
                if (HAS_MIN) {
                    a = fma2(pack2(w[h].z, w[h].z), s_lo, a);
                    a = fma2(pack2(w[h].w, w[h].w), s_hi, a);
                }
                acc[j][h] = a;
            }
        }
    };

    int slot = 0, fill = LEAD % STAGES, turn = 0;   // stage being multiplied, stage being filled, warp whose turn it is to fill
    uint32_t phase = 0, fill_phase = 1;
#pragma unroll 1
    for (int ks = 0; ks < k_stages; ks++) {
        if (ks + LEAD < k_stages && warp == turn && elect_one()) {
            if (ks + LEAD >= STAGES) wait_bounded(&empty[fill], fill_phase, abort_flag, prm.flag);
            issue_weights(ks + LEAD, fill);
            issue_activations(ks + LEAD, fill);
        }
        __syncwarp();
        if (++fill == STAGES) {
            fill = 0;
            fill_phase ^= 1;
        }
        if (++turn == WR) turn = 0;
        wait_bounded(&full[slot], phase, abort_flag, prm.flag);
        const uint32_t st = base + slot * G::STAGE_BYTES;
        const int np = min(SP, prm.pairs - ks * SP);
        if (np == SP) {
#pragma unroll
            for (int pj = 0; pj < SP; pj++) multiply_pair(pj, st);
        } else {
#pragma unroll 1
            for (int pj = 0; pj < np; pj++) multiply_pair(pj, st);
        }
        __syncwarp();
        if (elect_one()) mbar_arrive(&empty[slot]);
        if (++slot == STAGES) {
            slot = 0;
            phase ^= 1;
        }
    }
    if (*abort_flag != 0 && threadIdx.x == 0) {
        // copies of stages nobody waited for may still be in flight: wait (bounded) for the last fill of each slot
        for (int s = 0; s < STAGES && s < k_stages; s++) mbar_wait_drain(&full[s], ((k_stages - 1 - s) / STAGES) & 1);
    }
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const int m = j * 8 + t2 + c;
            if (m < prm.M) {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int n = row_base + row0 + h * 8 + g;
                    if (n < prm.rows) {
                        float v0, v1;
                        unpack2(acc[j][h], v0, v1);
                        const float v = c ? v1 : v0;
                        const size_t off = static_cast<size_t>(m) * prm.ldc + n;
                        prm.C[off] = v;
#pragma unroll
                        for (int e = 0; e < MAX_PEERS - 1; e++)   // static indices: the parameter array stays out of local memory
                            if (e < prm.extra.n) prm.extra.p[e][off] = v;
                    }
                }
            }
        }
}

constexpr int MAX_DEVICES = 64;

template <int SCH, bool S16, int WR, int NT>
static int launch_one(inkq_ctx *ctx, const Act *a, const Weight *w, int m_begin, const Params &prm)
{
    using G = Cfg<SCH, S16, WR, NT>;
    auto kernel = k_qgemm_rows<SCH, S16, WR, NT>;
    // The opt-in for large dynamic shared memory is a per-device function attribute: remembered per device and instantiation
    static std::mutex mu;
    static bool configured[MAX_DEVICES] = {};
    if (ctx->device < 0 || ctx->device >= MAX_DEVICES) return fail(ctx, INKQ_ERR_UNSUPPORTED, "device index beyond the launch table");
    {
        std::lock_guard<std::mutex> lk(mu);
        if (!configured[ctx->device]) {
            const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM < SMEM_ONE_CTA ? SMEM_ONE_CTA : G::SMEM);
            if (e != cudaSuccess) return fail(ctx, INKQ_ERR_CUDA, std::string("cudaFuncSetAttribute(k_qgemm_rows): ") + cudaGetErrorString(e));
            configured[ctx->device] = true;
        }
    }
    const int nb = a->K / QK;
    CUtensorMap mq, md, ms;
    // a row window starts m_begin rows into q and m_begin entries into every block's line of the planes
    int rc = encode_map_2d(ctx, &mq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a->q + static_cast<size_t>(m_begin) * a->K, a->K, prm.M, 128u, G::BM,
                           CU_TENSOR_MAP_SWIZZLE_128B, a->K);
    if (!rc) rc = encode_map_2d(ctx, &md, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a->d + m_begin, a->M_ld - m_begin, nb, G::BM, 2 * SP, CU_TENSOR_MAP_SWIZZLE_NONE,
                                a->M_ld);
    ms = md;
    if (!rc && G::PLANES == 2)
        rc = encode_map_2d(ctx, &ms, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a->s + m_begin, a->M_ld - m_begin, nb, G::BM, 2 * SP, CU_TENSOR_MAP_SWIZZLE_NONE, a->M_ld);
    if (rc) return rc;
    const int grid = (w->rows + G::ROWS - 1) / G::ROWS;
    // No more CTAs than SMs: one per SM.  The grid may be placed while the kernel before it still occupies SMs, and would
    // otherwise double up on the free ones (4096 x 12288 behind its quantizer: 95 -> 60 us with 77 rows in an earlier form).
    const int smem = grid <= ctx->num_sms && G::SMEM < SMEM_ONE_CTA ? SMEM_ONE_CTA : G::SMEM;
    const cudaError_t le = launch_pdl(kernel, dim3(grid), dim3(G::THREADS), smem, ctx->stream, mq, md, ms, prm);
    if (le != cudaSuccess) return fail(ctx, INKQ_ERR_CUDA, std::string("k_qgemm_rows launch: ") + cudaGetErrorString(le));
    return after_launch(ctx, "k_qgemm_rows");
}

template <int SCH, bool S16>
static int launch_sized(inkq_ctx *ctx, const Act *a, const Weight *w, int m_begin, const Params &prm)
{
    // 64 instead of 128 rows per CTA when the layer has too few 128-row tiles to occupy the SMs (measured: 6144 x 4096 with 24
    // rows 18.0 -> 13.4 us; 24576 x 4096 with 5 rows 16.3 against 23.1 us the other way round)
    const bool narrow = w->tiles * 2 <= ctx->num_sms;
    switch ((prm.M + 7) / 8) {
        case 1: return narrow ? launch_one<SCH, S16, 4, 1>(ctx, a, w, m_begin, prm) : launch_one<SCH, S16, 8, 1>(ctx, a, w, m_begin, prm);
        case 2: return narrow ? launch_one<SCH, S16, 4, 2>(ctx, a, w, m_begin, prm) : launch_one<SCH, S16, 8, 2>(ctx, a, w, m_begin, prm);
        case 3: return narrow ? launch_one<SCH, S16, 4, 3>(ctx, a, w, m_begin, prm) : launch_one<SCH, S16, 8, 3>(ctx, a, w, m_begin, prm);
        case 4: return narrow ? launch_one<SCH, S16, 4, 4>(ctx, a, w, m_begin, prm) : launch_one<SCH, S16, 8, 4>(ctx, a, w, m_begin, prm);
    }
    return fail(ctx, INKQ_ERR_INVALID, "internal: too many rows for k_qgemm_rows");
}

}  // namespace qrows

int launch_gemm_rows(inkq_ctx *ctx, const Act *a, const Weight *w, float *C, int ldc, const ExtraDst *extra, int m_begin, int m_count)
{
    using namespace qrows;
    const bool s16 = w->scale_mode == INKQ_SCALES_F16;
    Params prm;
    prm.nibT = w->nibT;
    prm.sc = s16 ? reinterpret_cast<const unsigned char *>(w->sc16) : reinterpret_cast<const unsigned char *>(w->sc32);
    prm.zpT = w->zpT;
    const size_t c_off = static_cast<size_t>(m_begin) * ldc;
    prm.C = C + c_off;
    prm.extra = ExtraDst{};
    if (extra != nullptr) {
        prm.extra = *extra;
        for (int e = 0; e < prm.extra.n; e++) prm.extra.p[e] += c_off;
    }
    prm.flag = ctx->dev_flag;
    prm.M = m_count;
    prm.rows = w->rows;
    prm.pairs = w->pairs;
    prm.ldc = ldc;
    if (w->scheme == INKQ_A81W41) return s16 ? launch_sized<INKQ_A81W41, true>(ctx, a, w, m_begin, prm) : launch_sized<INKQ_A81W41, false>(ctx, a, w, m_begin, prm);
    if (w->scheme == INKQ_A80W40) return s16 ? launch_sized<INKQ_A80W40, true>(ctx, a, w, m_begin, prm) : launch_sized<INKQ_A80W40, false>(ctx, a, w, m_begin, prm);
    return s16 ? launch_sized<INKQ_A80W4Z, true>(ctx, a, w, m_begin, prm) : launch_sized<INKQ_A80W4Z, false>(ctx, a, w, m_begin, prm);
}

}  // namespace inkq
