// QGEMM (2 and more activation rows: sequences decoded together, prompts): warp-level int8 matrix products whose block dots
// are scaled where they appear, in registers.
//
// Stands in for gemm_repack_A81W41_fp32 (qwen3/src/qwen/quantized_gemx_kernels.cc:349-582)
// and gemm_repack_A80W40 (:195-347); A80W4Z has no reference kernel and follows the A80W40
// code with q_w = nibble - zp.  Same result bits as qgemm_simt.cu.
//
//   C[m][n] = sum over 32-element blocks b of  d_a[m,b]*d_w[n,b]*I[m,n,b] + m_w[n,b]*s_a[m,b]
//   I[m,n,b] = sum_e q_a[m,32b+e] * q_w[n,32b+e]                       (exact int32)
//
// Why mma.sync: it leaves the 16 x 8 dots of one block (K = 32) in the registers of the threads that scale them.  Every block
// of every output needs its own fp32 conversion, scale product and one or two fused multiply-adds in the reference's order, so
// the CUDA cores bound this path and not the tensor cores: a tcgen05 form (block dots in tensor memory, or as e4m3 parts with
// the weights in tensor memory) keeps the tensor pipe ~90 % idle and pays for the way back to registers and for hand-shakes.
//
// What bounds it.  Up to 32 rows: the weight stream, and for layers with few rows the chain of a warp's dependent instructions
// over K (an output's sum may not be split).  Every warp owns 16 weight rows and all columns: each weight byte is fetched once.
// Stages of four pairs (256 K-elements) are unrolled, so that the fragment loads and products of one pair overlap the scaling of
// the one before.  More rows: conversions, register file and FMA pipe.  Alone in registers, with two warps of 32 x 56 dots a scheduler,
// a block's 16 x 8 dots (a product, four conversions, two packed multiplications and two packed multiply-adds, four with mins) take it
// 19 cycles, 23 with mins; 10.7 and 15.6 of them the packed operations, three operands of 64 bits each.  A block's
// chain (fragment loads, product, conversion, scaling) is long and an SM has few warps in a tile of this size, so stages of 4 to 8
// pairs are unrolled and one CTA of 8 warps gets up to 255 registers a thread.  The weights are read from L2 once per tile of
// columns (CTAs of one weight tile are neighbours).
// Measured (weights of distinct layers), A81W41: 24576 x 4096 with 5 rows 14 us (4.6 TB/s), 4096 x 4096 with 5 rows 6.6, 12288 x 4096
// with 24 rows 15.5, with 322 rows 99 (fp32 records), 24576 x 4096 with 322 rows 191; A80W40 12288 x 4096 with 2048 rows 502; A80W4Z 4096 x
// 12288 with 77 rows 36.  Slower: scalar multiplications (+12 %), the conversion by a bias in the product's accumulator operand (+20 %: it
// has to be moved there), fp16 operands with fp32 accumulators (+25 %), e4m3 parts (x2), the results staged in shared memory for whole-line
// stores (+1 to 2 %), a stage's pairs unrolled by two (+1 to 8 %), a resident CTA that requests its next tile's stages during the stores
// (K = 1024: -10 %, 322 and 77 rows at K = 4096 and 12288: +4 %, from the registers it takes).
// A tcgen05 form (kind::i8 with the weights in tensor memory, dots read back 16 x 256 bits at a time, a relay warp and named barriers in
// front of the scaling warps) takes 694 (A81W41) and 575 ns (A80W40) per pair of a 128 x 112 tile, exact fp16 operands 684 and 559, this
// kernel 706 and 612: the scaling bounds them all alike, two packed operations and a conversion per dot at ~0.55 instructions a cycle.
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

#include "inkq_internal.h"
#include "ptx.cuh"

namespace inkq {
namespace qrows {

constexpr int MAX_STAGES = 8;
constexpr int SMEM_ONE_CTA = 116 * 1024;   // more than half of an SM's shared memory
constexpr int SMEM_SM = 222 * 1024;        // for all CTAs of an SM

struct Params {
    const uint8_t *nibT;
    const unsigned char *sc;   // fp16 or fp32 scale records
    const uchar2 *zpT;
    float *C;
    int32_t *dots;    // DUMP: raw int32 block dots [M][rows][K/32] instead of C
    ExtraDst extra;   // further destinations of every C element (peers of a column-sharded layer)
    int *flag;
    int M, rows, pairs, ldc, tiles_m;
};

// Shape of a tile: WR x WC warps, each with MT groups of 16 weight rows and NT groups of 8 activation rows; SP pairs per stage;
// CTAS resident CTAs per SM; SHORT: the second column of warps has one group of activation rows less (each scheduler has a warp of both).
template <int WR_, int WC_, int MT_, int NT_, int SP_, int CTAS_ = 2, bool SHORT_ = false>
struct Tile {
    static constexpr int WR = WR_, WC = WC_, MT = MT_, NT = NT_, SP = SP_, CTAS = CTAS_, ROWS = 16 * WR * MT, COLS = 8 * (NT * WC - (SHORT_ ? 1 : 0));
    static constexpr bool SHORT = SHORT_;
    static_assert(!SHORT || (WC == 2 && WR == 4), "warps w and w + 4 share a scheduler");
};

// SCH: weight scheme; S16: fp16 scale records
template <int SCH, bool S16, class T>
struct Cfg {
    static constexpr int SP = T::SP, ROWS = T::ROWS, BM = T::COLS, WARPS = T::WR * T::WC, THREADS = 32 * WARPS;
    static constexpr int PLANES = (SCH == INKQ_A81W41) ? 2 : 1;
    static constexpr int Q_BYTES = BM * 64 * SP, PLANE_BYTES = 2 * SP * BM * 4;
    static constexpr int W_PAIR = ROWS * 32, SC_REC = S16 ? 8 : 16, SC_PAIR = ROWS * SC_REC, Z_PAIR = (SCH == INKQ_A80W4Z) ? ROWS * 2 : 0;
    static constexpr int W_OFF = Q_BYTES, SC_OFF = W_OFF + SP * W_PAIR, Z_OFF = SC_OFF + SP * SC_PAIR, D_OFF = Z_OFF + SP * Z_PAIR, S_OFF = D_OFF + PLANE_BYTES;
    static constexpr int STAGE_BYTES = (D_OFF + PLANES * PLANE_BYTES + 1023) / 1024 * 1024;
    static constexpr int FIT = (SMEM_SM / T::CTAS - 1024 - 256) / STAGE_BYTES, STAGES = FIT > MAX_STAGES ? MAX_STAGES : FIT;
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

template <int SCH, bool S16, class T, bool DUMP>
__global__ void __launch_bounds__(32 * T::WR * T::WC, T::CTAS)
    k_qgemm_rows(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_d, const __grid_constant__ CUtensorMap map_s,
                 const __grid_constant__ Params prm)
{
    using G = Cfg<SCH, S16, T>;
    constexpr int SP = T::SP, MT = T::MT, NT = T::NT;
    constexpr bool HAS_MIN = SCH == INKQ_A81W41;
    constexpr int STAGES = G::STAGES, LEAD = G::LEAD;
    extern __shared__ __align__(1024) unsigned char smem_dyn[];
    unsigned char *smem = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES * G::STAGE_BYTES), *empty = full + STAGES;
    volatile int *abort_flag = reinterpret_cast<volatile int *>(empty + STAGES);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tn = blockIdx.x / prm.tiles_m, m_base = (blockIdx.x - tn * prm.tiles_m) * G::BM;   // first activation row of the CTA
    const int row_base = tn * G::ROWS, row_in_tile = row_base % TILE_N;                          // and its first weight row
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
        for (int b = 0; b < SP / 2; b++) tma_tensor2d_g2s(st + b * (G::BM * 128), &map_q, ks * (64 * SP) + b * 128, m_base, &full[slot]);
        tma_tensor2d_g2s(st + G::D_OFF, &map_d, m_base, ks * (2 * SP), &full[slot]);
        if (G::PLANES == 2) tma_tensor2d_g2s(st + G::S_OFF, &map_s, m_base, ks * (2 * SP), &full[slot]);
    };

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], G::WARPS);
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

    const int row0 = (warp % T::WR) * (16 * MT), col0 = (warp / T::WR) * (8 * NT);   // the warp's first row and column inside the tile
    const bool is_short = T::SHORT && warp >= T::WR;         // this warp leaves its last group of activation rows out
    const int g = lane >> 2, t2 = (lane & 3) * 2;            // fragment coordinates: rows g, g + 8; columns t2, t2 + 1
    // ldmatrix row addresses.  A: matrices (rows 0-7, chunk 0), (rows 8-15, chunk 0), (rows 0-7, chunk 1), (rows 8-15, chunk 1)
    const int a_row = row0 + ((lane >> 3) & 1) * 8 + (lane & 7);
    const uint32_t a_off = G::W_OFF + a_row * 32 + ((((lane >> 4) & 1) ^ ((a_row >> 2) & 1)) << 4);
    // B: matrix j = 16-byte chunk j of a pair's 64 bytes (low block: chunks 0, 1; high block: 2, 3); rows of 128 B, swizzled;
    // the second pair of a row lies at this offset with bit 6 flipped
    const uint32_t b_off = (col0 + (lane & 7)) * 128 + (((lane >> 3) ^ (lane & 7)) << 4);
    const uint32_t base = smem_u32(smem);

    unsigned long long acc[MT][NT][2];   // columns (t2, t2 + 1) of rows g and g + 8
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++) acc[i][j][0] = acc[i][j][1] = 0ull;

    auto multiply_pair = [&](int p, int pj, uint32_t st) {   // pair p of the row, pj of the stage
        uint32_t alo[MT][4], ahi[MT][4];
        float4 w[MT][2];   // {d_lo, d_hi, m_lo, m_hi} of rows g and g + 8
#pragma unroll
        for (int i = 0; i < MT; i++) {
            uint32_t pk[4], z_lo[2] = {0u, 0u}, z_hi[2] = {0u, 0u};
            ldmatrix_x4(pk, st + a_off + pj * G::W_PAIR + i * (16 * 32));
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int r = row0 + i * 16 + g + 8 * h;
                if (S16) {
                    const uint2 v = lds_u32x2(st + G::SC_OFF + pj * G::SC_PAIR + r * 8);
                    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&v.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&v.y));
                    w[i][h] = make_float4(a.x, a.y, b.x, b.y);
                } else {
                    w[i][h] = lds_f4(st + G::SC_OFF + pj * G::SC_PAIR + r * 16);
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
                alo[i][e] = pk[e] & 0x0F0F0F0Fu;
                ahi[i][e] = (pk[e] >> 4) & 0x0F0F0F0Fu;
                if (!HAS_MIN) {   // byte-wise (nibble - z) without borrows between bytes: set bit 7, subtract, clear
                    alo[i][e] = ((alo[i][e] | 0x80808080u) - z_lo[e & 1]) ^ 0x80808080u;
                    ahi[i][e] = ((ahi[i][e] | 0x80808080u) - z_hi[e & 1]) ^ 0x80808080u;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < NT; j++) {
            if (T::SHORT && j == NT - 1 && is_short) break;
            uint32_t b[4];
            ldmatrix_x4(b, st + (pj >> 1) * (G::BM * 128) + (b_off ^ ((pj & 1) << 6)) + j * (8 * 128));
            const uint32_t pl = st + (2 * pj) * (G::BM * 4) + (col0 + j * 8 + t2) * 4;
            const unsigned long long d_lo = lds_u64(pl + G::D_OFF), d_hi = lds_u64(pl + G::D_OFF + G::BM * 4);
            unsigned long long s_lo = 0ull, s_hi = 0ull;
            if (HAS_MIN) {
                s_lo = lds_u64(pl + G::S_OFF);
                s_hi = lds_u64(pl + G::S_OFF + G::BM * 4);
            }
#pragma unroll
            for (int i = 0; i < MT; i++) {
                int lo[4], hi[4];
                mma_block(lo, alo[i], b[0], b[1]);
                mma_block(hi, ahi[i], b[2], b[3]);
                if (DUMP) {
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int n = row_base + row0 + i * 16 + g + (e >> 1) * 8, m = m_base + col0 + j * 8 + t2 + (e & 1);
                        if (n < prm.rows && m < prm.M) {
                            int32_t *o = prm.dots + (static_cast<size_t>(m) * prm.rows + n) * (2 * prm.pairs) + 2 * p;
                            o[0] = lo[e];
                            o[1] = hi[e];
                        }
                    }
                    continue;
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    unsigned long long a = acc[i][j][h];
                    a = fma2(cvt2_exact(lo[2 * h], lo[2 * h + 1]), mul2(d_lo, pack2(w[i][h].x, w[i][h].x)), a);
                    a = fma2(cvt2_exact(hi[2 * h], hi[2 * h + 1]), mul2(d_hi, pack2(w[i][h].y, w[i][h].y)), a);
                    if (HAS_MIN) {
                        a = fma2(pack2(w[i][h].z, w[i][h].z), s_lo, a);
                        a = fma2(pack2(w[i][h].w, w[i][h].w), s_hi, a);
                    }
                    acc[i][j][h] = a;
                }
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
        if (++turn == G::WARPS) turn = 0;
        wait_bounded(&full[slot], phase, abort_flag, prm.flag);
        const uint32_t st = base + slot * G::STAGE_BYTES;
        const int np = min(SP, prm.pairs - ks * SP);
        if (np == SP) {
#pragma unroll
            for (int pj = 0; pj < SP; pj++) multiply_pair(ks * SP + pj, pj, st);
        } else {
#pragma unroll 1
            for (int pj = 0; pj < np; pj++) multiply_pair(ks * SP + pj, pj, st);
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
    if (DUMP) return;
    // One copy of the stores for all destinations.  This code runs once per CTA and its instructions come from far away: with the seven
    // further destinations unrolled into each of up to 56 stores it took 5 to 8 us of a tile (12288 x 4096 with 322 rows 114 -> 99 us,
    // with 2048 rows 565 -> 528, 8192 x 1024 with 400 rows 39 -> 30)
    float *dst = prm.C;
#pragma unroll 1
    for (int e = 0;; e++) {
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int m = m_base + col0 + j * 8 + t2 + c;
                if (m < prm.M && !(T::SHORT && j == NT - 1 && is_short)) {
#pragma unroll
                    for (int i = 0; i < MT; i++)
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const int n = row_base + row0 + i * 16 + h * 8 + g;
                            float v0, v1;
                            unpack2(acc[i][j][h], v0, v1);
                            if (n < prm.rows) dst[static_cast<size_t>(m) * prm.ldc + n] = c ? v1 : v0;
                        }
                }
            }
        if (e >= prm.extra.n) break;
        dst = prm.extra.p[e];
    }
}

template <int SCH, bool S16, class T, bool DUMP = false>
static int launch_one(inkq_ctx *ctx, const Act *a, const Weight *w, int m_begin, Params prm)
{
    using G = Cfg<SCH, S16, T>;
    auto kernel = k_qgemm_rows<SCH, S16, T, DUMP>;
    int rc = allow_smem<k_qgemm_rows<SCH, S16, T, DUMP>>(ctx);
    if (rc) return rc;
    const int nb = a->K / QK;
    CUtensorMap mq, md, ms;
    // a row window starts m_begin rows into q and m_begin entries into every block's line of the planes
    rc = encode_map_2d(ctx, &mq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a->q + static_cast<size_t>(m_begin) * a->K, a->K, prm.M, 128u, G::BM,
                       CU_TENSOR_MAP_SWIZZLE_128B, a->K);
    if (!rc) rc = encode_map_2d(ctx, &md, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a->d + m_begin, a->M_ld - m_begin, nb, G::BM, 2 * G::SP, CU_TENSOR_MAP_SWIZZLE_NONE,
                                a->M_ld);
    ms = md;
    if (!rc && G::PLANES == 2)
        rc = encode_map_2d(ctx, &ms, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a->s + m_begin, a->M_ld - m_begin, nb, G::BM, 2 * G::SP, CU_TENSOR_MAP_SWIZZLE_NONE, a->M_ld);
    if (rc) return rc;
    prm.tiles_m = (prm.M + G::BM - 1) / G::BM;
    const int grid = (w->rows + G::ROWS - 1) / G::ROWS * prm.tiles_m;
    // Shared memory for no more CTAs per SM than an even spread needs.  The grid may be placed while the kernel before it
    // still occupies SMs, and would otherwise pile up on the free ones (4096 x 12288 behind its quantizer: 95 -> 60 us with 77
    // rows in an earlier form).
    const int per_sm = (grid + ctx->num_sms - 1) / ctx->num_sms, spread = per_sm == 1 ? SMEM_ONE_CTA : SMEM_SM / (per_sm < T::CTAS ? per_sm : T::CTAS);
    const int smem = spread > G::SMEM ? spread : G::SMEM;
    const cudaError_t le = launch_pdl(kernel, dim3(grid), dim3(G::THREADS), smem, ctx->stream, mq, md, ms, prm);
    if (le != cudaSuccess) return fail(ctx, INKQ_ERR_CUDA, std::string("k_qgemm_rows launch: ") + cudaGetErrorString(le));
    return after_launch(ctx, "k_qgemm_rows");
}

// Tiles for more than 32 activation rows: shape, the part of a launch's time (us) that does not depend on K, and for A81W41, A80W40 and
// A80W4Z, first with fp16 and then with fp32 scale records, the whole time at K = 4096; each with one and with two tiles on every SM and of
// every two tiles more (a third of the way from two to eight).  All measured in one way: 148 tiles of weight rows, as many tiles of columns
// as the count says, three layers in turn, the least of sixteen loops; two such measurements differ by 1 to 2 %.  The records' size makes up
// to 24 % of difference in either direction, by tile and scheme: it changes the ring's stages and the registers.  The fixed part is a CTA's
// set-up and its stores, from times at K = 512 and 4096; it hardly depends on scheme and records (their mean, mostly 0.3 us from each).
// Only the ratios matter.  Over 240 random layers each (33 to 2048 rows) the chosen tile takes 0.3 % more than the best one, at most 18 %
// (1248 x 1920 with 224 rows), for K from 1024 to 12288, and 1.5 %, at most 25 % (5360 x 576 with 42 rows: 4.2 us), for K from 64 to 1023.
// By the times at K = 4096 alone the latter took 5.7 % more, at most 80 %: two CTAs per SM hide set-up and stores behind each other's
// products, and short rows are little else (818 rows of 16832 x 384, A80W4Z with fp32 records: 49.8 -> 40.3 us).
// Mostly one CTA of 8 warps per SM with all the registers it wants and 4 to 8 unrolled pairs per stage: the fragment loads and products
// of several pairs overlap the scaling of the ones before (against two CTAs of 128 registers and two-pair stages: 64 x 48
// 17.9 -> 14.2, 128 x 112 72 -> 51).  Two such CTAs side by side remain for many tiles per SM, where one's set-up and stores hide behind
// the other's products.
// Per column the wide tiles cost least: fragments and scales of the weight rows are fetched once for more columns.
// Half- and quarter-height tiles split a layer with few weight rows over more SMs.  64 x 40 with one warp per scheduler costs less per
// column than 64 x 48 with two, which fetch and unpack every weight fragment twice (77 rows of 4096 x 12288, A80W4Z: 41 -> 36 us).
// Without mins, 8 warps of 16 rows by all columns instead of 4 x 2 of 32 rows by half of them, from 40 columns on: a column costs two loads of a
// plane less there, and the scales and fragments of twice the columns are cheaper than those of twice the weight rows.  One tile on every SM,
// us with 4 x 2 and with 8 x 1 warps: 48 columns A80W40 22.9, 21.6, A80W4Z 25.8, 22.7; 64: 28.1, 27.4 and 30.5, 28.2; 96: 37.6, 37.1 and
// 40.1, 37.7; 112: 42.2, 41.7 and 44.3, 43.6; and sizes between the multiples of 16 that two columns of warps have.  With mins it is the other
// way round: 48 columns 24.8, 26.5, 64: 31.6, 33.8; 322 rows of 4096 x 4096 47.1 with 96 columns by 4 x 2 warps, 48.2 with 88 by 8.
// With mins 88 columns are 48 for one column of warps and 40 for the other (41.5 us a tile, 96 columns 43.2; 322 rows of 4096 x 4096 47.1 -> 45.8,
// of 4096 x 12288 129.5 -> 126.1): the last group of the longer ones stands in a block of its own, which costs half of what is left out.  72
// columns take 36.3 us a tile (fp16 records; fp32 35.3) where 80 take 36.8 (36.3), 104 take 49.0 (49.6) and 112 48.7 (49.9).  With two bodies of code instead 88 columns take 58 us (instruction fetch).
// Layers with their quantizer: 12288 x 4096 with 2048 rows, A80W40 541 -> 518 us (128 x 104); 4096 x 12288 with 322 rows 113 -> 101, A80W4Z 120 -> 106 (128 x 88).
#define NEVER (0.f, 0.f, 0.f)   // a tile that a scheme does not have
#define QROWS_TILES(X)                                                                                                    \
    X(0, (2, 4, 1, 2, 8, 1), (2.2f, 3.6f, 3.2f), (12.2f, 24.1f, 23.7f), (11.6f, 22.7f, 22.3f), (13.5f, 26.6f, 26.3f),     \
      (12.6f, 24.4f, 24.0f), (11.6f, 22.4f, 22.0f), (13.6f, 26.8f, 26.4f))                                                \
    X(1, (4, 2, 1, 2, 8, 1), (2.0f, 3.3f, 2.9f), (13.1f, 25.7f, 25.2f), (12.4f, 24.4f, 23.8f), (14.5f, 28.6f, 28.1f),     \
      (13.2f, 26.1f, 25.5f), (12.2f, 24.0f, 23.5f), (14.6f, 28.8f, 28.2f))                                                \
    X(2, (4, 1, 2, 2, 4, 2), (2.1f, 2.1f, 1.0f), (13.3f, 19.8f, 18.4f), (12.7f, 18.7f, 17.4f), (14.4f, 21.5f, 20.3f),     \
      (15.6f, 21.0f, 19.8f), (15.8f, 20.9f, 20.0f), (17.2f, 23.9f, 22.4f))                                                \
    X(3, (4, 2, 1, 3, 8, 1), (2.0f, 3.8f, 3.4f), (15.8f, 30.9f, 30.3f), (13.9f, 27.2f, 26.8f), (16.1f, 31.6f, 31.2f),     \
      (15.9f, 31.4f, 30.9f), (13.8f, 27.0f, 26.4f), (15.8f, 31.1f, 30.6f))                                                \
    X(4, (4, 2, 1, 4, 6, 1), (2.6f, 4.9f, 4.5f), (19.4f, 38.5f, 38.0f), (17.9f, 35.5f, 35.0f), (20.1f, 39.9f, 39.3f),     \
      (19.9f, 39.5f, 39.1f), (16.8f, 33.5f, 32.8f), (19.1f, 37.8f, 37.2f))                                                \
    X(5, (4, 2, 1, 5, 6, 1), (2.7f, 5.2f, 4.6f), (23.0f, 45.8f, 45.2f), (19.5f, 38.6f, 38.0f), (21.4f, 42.4f, 41.9f),     \
      (26.1f, 51.5f, 51.6f), (19.5f, 38.7f, 38.1f), (21.1f, 41.9f, 41.4f))                                                \
    X(6, (4, 2, 1, 7, 4, 1), (2.7f, 5.1f, 4.9f), (29.6f, 59.0f, 58.3f), (25.5f, 50.4f, 49.9f), (27.8f, 54.9f, 54.4f),     \
      (30.1f, 59.9f, 59.4f), (25.4f, 50.2f, 49.3f), (27.7f, 54.9f, 54.2f))                                                \
    X(7, (4, 2, 2, 2, 8, 1), (2.1f, 3.4f, 2.5f), (19.2f, 36.8f, 35.5f), (18.3f, 35.2f, 33.9f), (20.9f, 40.3f, 38.9f),     \
      (18.3f, 34.8f, 33.4f), (18.4f, 35.2f, 33.7f), (21.0f, 40.2f, 38.6f))                                                \
    X(8, (4, 2, 2, 3, 6, 1), (2.7f, 4.4f, 3.6f), (24.8f, 48.4f, 47.4f), NEVER, NEVER,                                     \
      (24.5f, 47.6f, 46.2f), NEVER, NEVER)                                                                                \
    X(9, (4, 2, 2, 4, 4, 1), (2.7f, 4.5f, 3.7f), (31.6f, 61.9f, 61.0f), NEVER, NEVER,                                     \
      (30.7f, 59.8f, 58.8f), NEVER, NEVER)                                                                                \
    X(10, (4, 2, 2, 5, 4, 1), (3.0f, 5.0f, 4.2f), (36.6f, 72.3f, 71.3f), NEVER, NEVER,                                    \
      (36.1f, 71.0f, 70.0f), NEVER, NEVER)                                                                                \
    X(11, (4, 2, 2, 6, 4, 1), (3.2f, 5.4f, 4.9f), (43.2f, 85.5f, 84.7f), NEVER, NEVER,                                    \
      (41.6f, 82.0f, 81.0f), NEVER, NEVER)                                                                                \
    X(12, (4, 2, 2, 7, 4, 1), (3.3f, 5.5f, 5.3f), (48.4f, 95.7f, 94.9f), NEVER, NEVER,                                    \
      (49.6f, 99.0f, 97.9f), NEVER, NEVER)                                                                                \
    X(13, (4, 2, 1, 4, 2, 2), (2.7f, 2.7f, 2.5f), (23.2f, 37.5f, 35.8f), (20.5f, 32.3f, 31.2f), (24.3f, 36.6f, 35.5f),    \
      (22.5f, 37.2f, 36.0f), (20.7f, 32.5f, 31.4f), (23.6f, 35.7f, 34.7f))                                                \
    X(14, (4, 2, 1, 7, 2, 2), (2.4f, 2.9f, 2.3f), (31.8f, 56.7f, 54.6f), (28.2f, 48.4f, 46.2f), (30.8f, 50.7f, 48.8f),    \
      (32.1f, 57.7f, 55.3f), (27.6f, 47.2f, 45.2f), (30.0f, 49.9f, 47.9f))                                                \
    X(15, (4, 2, 2, 4, 2, 2), (2.2f, 2.7f, 1.9f), (34.4f, 61.4f, 58.1f), (31.3f, 54.9f, 52.0f), (34.2f, 60.3f, 57.6f),    \
      (34.4f, 60.3f, 56.8f), (31.2f, 54.7f, 51.7f), (33.6f, 59.6f, 56.4f))                                                \
    X(16, (4, 2, 2, 5, 2, 2), (2.3f, 3.1f, 1.9f), (42.4f, 76.0f, 72.2f), (36.3f, 64.5f, 61.4f), (39.0f, 69.7f, 66.2f),    \
      (42.7f, 75.8f, 71.8f), (36.0f, 63.9f, 60.5f), (38.1f, 68.9f, 65.3f))                                                \
    X(17, (4, 1, 1, 5, 8, 1), (2.3f, 4.1f, 3.6f), (14.9f, 29.1f, 28.7f), (13.3f, 26.2f, 25.8f), (15.3f, 30.0f, 29.6f),    \
      (14.8f, 28.9f, 28.3f), (12.6f, 24.7f, 24.2f), (14.4f, 28.2f, 27.8f))                                                \
    X(18, (8, 1, 1, 5, 6, 1), (2.7f, 4.2f, 3.5f), NEVER, (19.3f, 36.8f, 35.4f), (20.3f, 38.9f, 37.3f),                    \
      NEVER, (19.4f, 36.8f, 35.4f), (20.4f, 38.7f, 37.4f))                                                                \
    X(19, (8, 1, 1, 6, 6, 1), (2.7f, 4.3f, 3.6f), NEVER, (21.6f, 41.7f, 40.1f), (22.7f, 43.6f, 42.2f),                    \
      NEVER, (22.0f, 42.1f, 40.4f), (23.5f, 45.1f, 43.5f))                                                                \
    X(20, (8, 1, 1, 7, 6, 1), (2.8f, 4.6f, 3.9f), NEVER, (24.0f, 46.2f, 44.8f), (25.9f, 50.0f, 48.3f),                    \
      NEVER, (24.3f, 46.7f, 45.2f), (25.4f, 49.1f, 47.4f))                                                                \
    X(21, (8, 1, 1, 8, 4, 1), (2.6f, 4.3f, 3.6f), NEVER, (27.4f, 53.0f, 51.7f), (28.2f, 54.6f, 53.4f),                    \
      NEVER, (27.7f, 53.2f, 52.1f), (28.6f, 55.1f, 53.9f))                                                                \
    X(22, (8, 1, 1, 9, 4, 1), (2.8f, 4.6f, 4.0f), NEVER, (29.9f, 58.2f, 56.8f), (31.0f, 60.4f, 59.3f),                    \
      NEVER, (29.7f, 57.6f, 56.4f), (30.9f, 60.5f, 59.1f))                                                                \
    X(23, (8, 1, 1, 10, 4, 1), (2.9f, 4.8f, 4.2f), NEVER, (32.6f, 63.8f, 62.4f), (33.3f, 65.3f, 64.1f),                   \
      NEVER, (31.7f, 61.9f, 60.6f), (32.8f, 64.6f, 63.2f))                                                                \
    X(24, (8, 1, 1, 11, 4, 1), (3.1f, 5.1f, 4.5f), NEVER, (34.3f, 67.2f, 66.1f), (35.7f, 70.5f, 69.1f),                   \
      NEVER, (34.5f, 67.8f, 66.4f), (35.7f, 70.2f, 68.8f))                                                                \
    X(25, (8, 1, 1, 12, 4, 1), (3.2f, 5.4f, 4.9f), NEVER, (37.1f, 72.8f, 72.0f), (37.7f, 74.4f, 73.0f),                   \
      NEVER, (37.1f, 73.1f, 71.7f), (38.0f, 74.9f, 73.6f))                                                                \
    X(26, (8, 1, 1, 13, 4, 1), (3.3f, 5.6f, 5.2f), NEVER, (39.4f, 77.7f, 76.2f), (40.6f, 79.7f, 78.3f),                   \
      NEVER, (39.9f, 78.5f, 77.0f), (40.5f, 80.0f, 78.7f))                                                                \
    X(27, (8, 1, 1, 14, 4, 1), (3.3f, 5.7f, 5.5f), NEVER, (41.7f, 82.5f, 81.0f), (43.6f, 85.9f, 84.5f),                   \
      NEVER, (43.5f, 85.8f, 84.2f), (44.1f, 87.3f, 86.0f))                                                                \
    X(28, (8, 1, 1, 15, 4, 1), (3.4f, 5.8f, 5.8f), NEVER, (44.7f, 88.4f, 86.9f), (45.6f, 90.4f, 88.9f),                   \
      NEVER, (45.5f, 89.6f, 87.9f), (46.6f, 92.7f, 91.3f))                                                                \
    X(29, (4, 2, 2, 6, 4, 1, true), (2.7f, 4.3f, 3.7f), (41.5f, 81.7f, 80.2f), NEVER, NEVER,                              \
      (40.7f, 79.9f, 78.5f), NEVER, NEVER)

#define QROWS_UNWRAP(...) __VA_ARGS__
struct TileCost {
    int rows, cols;
    float fixed[3];        // part of the times below that does not depend on K
    float time[2][3][3];   // by scale records (fp16, fp32) and weight scheme (A81W41, A80W40, A80W4Z): one tile, two, every two more
};
static_assert(INKQ_A81W41 == 0 && INKQ_A80W40 == 1 && INKQ_A80W4Z == 2, "the schemes index the table");
static constexpr TileCost tile_costs[] = {
#define QROWS_COST(i, shape, fixed, h41, h40, h4z, f41, f40, f4z)                           \
    {Tile<QROWS_UNWRAP shape>::ROWS, Tile<QROWS_UNWRAP shape>::COLS, {QROWS_UNWRAP fixed}, \
     {{{QROWS_UNWRAP h41}, {QROWS_UNWRAP h40}, {QROWS_UNWRAP h4z}}, {{QROWS_UNWRAP f41}, {QROWS_UNWRAP f40}, {QROWS_UNWRAP f4z}}}},
    QROWS_TILES(QROWS_COST)
};
constexpr int TILES = static_cast<int>(sizeof(tile_costs) / sizeof(tile_costs[0]));
// What is compiled and what is chosen from: the tiles with times
static constexpr bool has_tile(int i, bool s16, int scheme) { return tile_costs[i].time[s16 ? 0 : 1][scheme][0] > 0.f; }

// The tile with the least time for M activation rows: a CTA takes one tile, so the busiest SM works through
// n = ceil(tiles / SMs) of them.
static int pick_tile(int num_sms, int scheme, bool s16, int rows, int pairs, int M)
{
    const float length = static_cast<float>(pairs) / 64.0f;   // of a row, in units of the K = 4096 of the table
    int best = -1;
    float best_time = 0.f;
    for (int i = 0; i < TILES; i++) {
        if (!has_tile(i, s16, scheme)) continue;
        const TileCost &c = tile_costs[i];
        const float *t = c.time[s16 ? 0 : 1][scheme];
        const long long total = static_cast<long long>((rows + c.rows - 1) / c.rows) * ((M + c.cols - 1) / c.cols);
        const long long n = (total + num_sms - 1) / num_sms;
        const float whole = t[(n - 1) % 2] + static_cast<float>((n - 1) / 2) * t[2];
        const float fixed = c.fixed[(n - 1) % 2] + static_cast<float>((n - 1) / 2) * c.fixed[2];
        const float time = fixed + (whole - fixed) * length;
        if (best < 0 || time < best_time) {
            best = i;
            best_time = time;
        }
    }
    return best;
}

template <int SCH, bool S16>
static int launch_sized(inkq_ctx *ctx, const Act *a, const Weight *w, int m_begin, const Params &prm)
{
    if (prm.M > 32) {
        const int tile = pick_tile(ctx->num_sms, SCH, S16, prm.rows, prm.pairs, prm.M);
        switch (tile) {
#define QROWS_CASE(i, shape, fixed, h41, h40, h4z, f41, f40, f4z)                                                             \
    case i:                                                                                                                   \
        if constexpr (has_tile(i, S16, SCH)) return launch_one<SCH, S16, Tile<QROWS_UNWRAP shape>>(ctx, a, w, m_begin, prm);  \
        break;
            QROWS_TILES(QROWS_CASE)
        }
    }
    // Up to 32 rows one tile holds all of them, so every weight byte is fetched once.  No more 128-row tiles than SMs: one CTA
    // per SM, stages of eight pairs, and 64 instead of 128 weight rows if that still leaves one CTA per SM (us, against 4 pairs and
    // two CTAs everywhere: 12288 x 4096 with 5 rows 10.6 -> 9.4, with 24 rows 18.8 -> 16.8; 6144 x 4096 with 5 rows 9.5 -> 7.3, with
    // 24 rows 13.3 -> 12.1).
    // More tiles, stages of four pairs: 64-row CTAs, three to an SM, as long as all of them are resident at once.  The busiest SM then
    // has 192 rows at most instead of the 256 of two 128-row CTAs.  Past that the fourth CTA of an SM is a second pass over K, and
    // 128-row CTAs are faster up to the widest layers.  us with 64- and 128-row CTAs, A81W41, K = 4096, fp16 records:
    //     weight rows (64-row CTAs)   8 activation rows   20 rows        32 rows
    //     24576 (384)                 13.9    15.2        22.8    28.8   30.2    35.1
    //     28416 (444)                 14.1    15.4        23.0    28.8   30.4    35.1
    //     28672 (448)                 20.1    15.4        32.3    29.0   52.5    35.1
    //     34816 (544)                 21.3    16.1        35.3    29.2   59.2    35.4
    //     51200 (800)                 26.6    29.4        44.5    44.1   59.9    53.1
    //     151936 (2374)               72.9    66.9       132     128    178     151
    // (640 CTAs, 8 to 20 rows of an A8xW4x layer without zero points, 3 to 13 % faster with 64: not worth a rule).  Up to four rows the
    // planes are narrower than the boxes of eight that fetch them, and with the two planes of A81W41 the larger number of
    // 64-row CTAs pays for that: 24576 x 4096 with 2 rows 16.4 against 15.5, with fp32 records 17.9 against 16.1; A80W40 15.5 and 15.5.
    const bool narrow = w->tiles * 2 <= ctx->num_sms, single = w->tiles <= ctx->num_sms;
    const bool half = (w->rows + 63) / 64 <= 3 * ctx->num_sms && (SCH != INKQ_A81W41 || prm.M > 4);
#define QROWS_SMALL(n)                                                                                              \
    case n:                                                                                                         \
        if (narrow) return launch_one<SCH, S16, Tile<4, 1, 1, n, 8, n == 1 ? 2 : 1>>(ctx, a, w, m_begin, prm);      \
        if (single) return launch_one<SCH, S16, Tile<8, 1, 1, n, 8, 1>>(ctx, a, w, m_begin, prm);                   \
        return half ? launch_one<SCH, S16, Tile<4, 1, 1, n, 4, 3>>(ctx, a, w, m_begin, prm) : launch_one<SCH, S16, Tile<8, 1, 1, n, 4, 2>>(ctx, a, w, m_begin, prm);
    switch ((prm.M + 7) / 8) {
        QROWS_SMALL(1)
        QROWS_SMALL(2)
        QROWS_SMALL(3)
        QROWS_SMALL(4)
    }
    return fail(ctx, INKQ_ERR_INVALID, "internal: too many rows for k_qgemm_rows");
}

}  // namespace qrows

void gemm_tile(int num_sms, int scheme, bool s16, int rows, int K, int M, int *tile)
{
    tile[0] = qrows::pick_tile(num_sms, scheme, s16, rows, K / (2 * QK), M);
    tile[1] = qrows::tile_costs[tile[0]].rows;
    tile[2] = qrows::tile_costs[tile[0]].cols;
}

int launch_gemm(inkq_ctx *ctx, const Act *a, const Weight *w, float *C, int ldc, int32_t *dots, const ExtraDst *extra, int m_begin, int m_count)
{
    using namespace qrows;
    if (m_count < 0) m_count = a->M - m_begin;   // default: every row from m_begin on
    if (m_begin < 0 || (m_begin & 3) != 0 || m_count < 1 || m_begin + m_count > a->M || (m_begin != 0 && dots != nullptr))
        return fail(ctx, INKQ_ERR_INVALID, "bad activation row window");
    if (ctx->encode_tiled == nullptr) return fail(ctx, INKQ_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled entry point not available");
    if (w->sc32 == nullptr) return fail(ctx, INKQ_ERR_INVALID, "this weight holds no fp32 scale records (weight-only layers use inkq_gemm_w41_f16act)");
    const bool s16 = w->scale_mode == INKQ_SCALES_F16 && dots == nullptr;
    Params prm;
    prm.nibT = w->nibT;
    prm.sc = s16 ? reinterpret_cast<const unsigned char *>(w->sc16) : reinterpret_cast<const unsigned char *>(w->sc32);
    prm.zpT = w->zpT;
    const size_t c_off = static_cast<size_t>(m_begin) * ldc;
    prm.C = (C != nullptr) ? C + c_off : nullptr;
    prm.dots = dots;
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
    if (dots != nullptr) {
        using T = Tile<4, 2, 1, 3, 2>;
        if (w->scheme == INKQ_A81W41) return launch_one<INKQ_A81W41, false, T, true>(ctx, a, w, m_begin, prm);
        if (w->scheme == INKQ_A80W40) return launch_one<INKQ_A80W40, false, T, true>(ctx, a, w, m_begin, prm);
        return launch_one<INKQ_A80W4Z, false, T, true>(ctx, a, w, m_begin, prm);
    }
    if (w->scheme == INKQ_A81W41) return s16 ? launch_sized<INKQ_A81W41, true>(ctx, a, w, m_begin, prm) : launch_sized<INKQ_A81W41, false>(ctx, a, w, m_begin, prm);
    if (w->scheme == INKQ_A80W40) return s16 ? launch_sized<INKQ_A80W40, true>(ctx, a, w, m_begin, prm) : launch_sized<INKQ_A80W40, false>(ctx, a, w, m_begin, prm);
    return s16 ? launch_sized<INKQ_A80W4Z, true>(ctx, a, w, m_begin, prm) : launch_sized<INKQ_A80W4Z, false>(ctx, a, w, m_begin, prm);
}

}  // namespace inkq
