// Weight-only W41 matmul on the 5th-generation tensor cores: fp16 activations x Q4_1 weights
// dequantised to fp16 on the fly, tcgen05.mma.kind::f16 with fp32 accumulators in tensor memory.
//
// No C++ kernel exists in the reference for this scheme; it follows
// notebooks/evaluate-qwen3_8b_W4.ipynb cell 13: the fp16 model's weight is replaced by the
// dequantised value and a stock fp16 linear with fp32 accumulation runs:
//   w16[n][k] = fp16(q[n][k] * d[n][k/32] + m[n][k/32])      (one rounding: a half-precision fma)
//   C[m][n]   = sum_k a16[m][k] * w16[n][k]                   (fp32 accumulate)
// Unlike the A8W4 schemes there is no per-block epilogue: the whole K extent accumulates inside
// tensor memory and the CUDA cores only dequantise (1.75 instructions per weight, once per tile of columns)
// and store the finished tile.
//
// "Swap-AB": the 128 weight rows of a tile are the UMMA M side (TMEM lanes), block_m = 16..256 activation rows
// the UMMA N side.  One stage = one pair of quantization blocks = 64 K-elements = four K=16 MMAs per weight tile.
// The dequantised weights go from registers straight into tensor memory and are the MMA's A operand there: with A in
// shared memory (16 KB written and read again per stage and tile) the shared-memory port was as busy as the tensor pipe.
// What bounds it: up to ~100 columns the turns of the dequantising warps and of the thread that issues the products (~260 cycles a
// stage of one weight tile: waits of ~60 cycles each, instruction fetch of six warps with different code on a scheduler, hand-over),
// above the tensor pipe.  Measured at K = 4096: 12288 rows x 17 columns 16.8 us, x 64 17.7 (21.4 and 22.1 before the waits' slow path left the
// loops and the issuing thread stopped waiting for the copies itself), x 322 32.4 (32.8: two weight tiles per CTA), x 2048 158 (157;
// 1.31 PFLOP/s); 4096 x 322 17.4 (22.4), 4096 x 12288 with 322 rows 44 (58).  Slower: A in shared memory with 8 dequantising warps (12288 x 322 53 us), one chunk per thread and
// turn (+15 %), the stores of a stage completing under the next one's arithmetic (+5 %: one slot less), two stages per copy (+10 %), the two
// chunks of a turn in a rolled loop (192 columns +8 %).
//
// Persistent, warp-specialised, one CTA per SM, 768 threads:
//   warps 0, 3   TMA producers (activations; weights): per stage one tiled 2-D copy of the fp16 activations
//                [block_m rows][64 halves = 128 B] (128-byte swizzle, rows beyond M zero-filled)
//                and per weight tile two untiled bulk copies: the pair's packed nibbles (4096 B) and its fp16
//                scales {d_lo, d_hi, m_lo, m_hi} per row (1024 B)
//   warp 1       MMA issuer (one elected thread); one commit per stage frees its shared memory and its weights' columns
//   warp 2       tensor-memory allocation / release
//   warps 4-19   dequantise: a thread takes one 16-byte chunk of a row = 16 weights of both blocks: byte pairs spread by
//                prmt, nibble -> 1024 + q as fp16 bits, minus 1024, fma.rn.f16x2 (one rounding of q*d + m), tcgen05.st.
//                Two chunks per turn: of two weight tiles every other stage, of one every fourth
//   warps 20-23  epilogue: tcgen05.ld of the finished fp32 tile, coalesced stores of C; the dequantising warps
//                help with a CTA's last tile
// Rings: as many raw stages as fit into shared memory, up to four slots of dequantised weights and one or two accumulators
// in tensor memory, whichever the tile's width leaves room for.
// Every mbarrier wait is bounded: when one runs out the kernel sets a device flag, every later wait returns at once, all
// loops run to their end inside their buffers and the host reports INKQ_ERR_TIMEOUT with the context usable.
//
// Algorithmic work per launch: 2*M*N*K flop; bytes: N*K*0.625 weights + M*K*2 activations (re-read
// from L2 once per weight tile) + M*N*4 output.
#include <cuda.h>
#include <cuda_fp16.h>

#include <math.h>

#include "inkq_internal.h"
#include "ptx.cuh"

namespace inkq {

namespace w41 {
constexpr int DEQ_WARPS = 16, EPI_WARPS = 4, THREADS = 32 * (4 + DEQ_WARPS + EPI_WARPS);
constexpr int RAW_W_BYTES = TILE_N * 32;                // packed nibbles of one (tile, pair): 4096
constexpr int RAW_S_BYTES = TILE_N * 8;                 // its fp16 scales: 1024
constexpr int A_COLS = 32;                              // tensor-memory columns of one dequantised (tile, pair): 64 halves per lane
constexpr int MAX_STAGES = 12, MAX_A_SLOTS = 4, MAX_ACC_SLOTS = 2;
constexpr int DONE_RING = 16;                           // "the MMAs of pair g have completed", indexed by g % DONE_RING
static_assert(MAX_STAGES < DONE_RING && MAX_A_SLOTS < DONE_RING, "rings");
constexpr int BAR_BYTES = 512, SMEM_BYTES = 226 * 1024;

// Weight tiles (of 128 rows) a CTA multiplies with one activation stage, and the activation rows of a stage.  Two weight
// tiles halve the activation bytes fetched from L2 per output.
struct Shape {
    int nt, block_m;
    constexpr int raw_bytes() const { return block_m * 128 + nt * (RAW_W_BYTES + RAW_S_BYTES); }
    constexpr int stages() const
    {
        const int fit = (SMEM_BYTES - 1024 - BAR_BYTES) / raw_bytes();
        return fit < MAX_STAGES ? fit : MAX_STAGES;
    }
    constexpr int acc_slots() const { return 2 * nt * block_m + 3 * nt * A_COLS <= 512 ? 2 : 1; }
    constexpr int a_slots() const
    {
        const int fit = (512 - acc_slots() * nt * block_m) / (nt * A_COLS);
        return fit < MAX_A_SLOTS ? fit / 2 * 2 : MAX_A_SLOTS;
    }
};
static_assert(Shape{2, 192}.a_slots() >= 2 && Shape{1, 256}.a_slots() >= 2 && Shape{1, 256}.stages() >= 2 && Shape{2, 192}.stages() >= 3, "shapes");

struct Params {
    const uint8_t *nibT;
    const uint2 *sc16;
    float *C;
    int *flag;
    int M, rows, pairs, tiles_n, groups_n, tiles_m, block_m, ldc;   // groups_n = ceil(tiles_n / NT)
    int stages, raw_bytes, a_slots, acc_slots;
};

struct Ring {
    uint32_t idx = 0, phase = 0, n;
    __device__ explicit Ring(uint32_t n_) : n(n_) {}
    __device__ __forceinline__ void advance()
    {
        if (++idx == n) {
            idx = 0;
            phase ^= 1;
        }
    }
};

// Bounded wait; always returns (after an abort the roles finish their loops without waiting).  The probes suspend the thread in
// hardware: probing in a loop, the roles that wait take issue slots from the dequantising warps (one more such warp: +10 %).
// Not inlined: the loops of all roles share the schedulers' small instruction caches, and a loop that spans fewer lines turns faster
// (one weight tile, a stage ~330 -> 260 cycles together with the shorter loop of the products).
__device__ __noinline__ void wait_slow(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int *dev_flag)
{
    const long long t0 = clock64();
#pragma unroll 1
    while (!mbar_try_wait_for(bar, parity, 10000u)) {
        if (*abort_flag != 0) return;
        if (clock64() - t0 > INKQ_SPIN_LIMIT_CYCLES) {
            *abort_flag = 1;
            atomicExch(dev_flag, 1);
            return;
        }
    }
}
__device__ __forceinline__ void wait_bounded(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int *dev_flag)
{
    if (__builtin_expect(!mbar_try_wait(bar, parity), 0)) wait_slow(bar, parity, abort_flag, dev_flag);
}

__device__ __forceinline__ uint32_t bits(__half2 h) { return *reinterpret_cast<const uint32_t *>(&h); }
__device__ __forceinline__ __half2 halves(uint32_t b) { return *reinterpret_cast<const __half2 *>(&b); }

// Four bytes (elements 4i .. 4i + 3 of both blocks of a pair) -> q*d + m of the low and of the high nibbles
__device__ __forceinline__ void dequant4(uint32_t v, __half2 d_lo, __half2 m_lo, __half2 d_hi, __half2 m_hi, uint32_t *lo, uint32_t *hi)
{
    const __half2 k1024 = halves(0x64006400u), k16th = halves(0x2C002C00u), k64 = halves(0xD400D400u);   // 1024, 1/16, -64
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const uint32_t p = __byte_perm(v, 0u, i ? 0x4342 : 0x4140);                     // two bytes, 16 bits apart
        // fp16 bits 0x6400 | b = 1024 + b exactly: 1024 + q, and 1024 + 16 q whose sixteenth minus 64 is q; all exact
        const __half2 ql = __hsub2(halves((p & 0x000F000Fu) | 0x64006400u), k1024);
        const __half2 qh = __hfma2(halves((p & 0x00F000F0u) | 0x64006400u), k16th, k64);
        lo[i] = bits(__hfma2(ql, d_lo, m_lo));
        hi[i] = bits(__hfma2(qh, d_hi, m_hi));
    }
}

// Worker `who` of `workers` warps of a lane quadrant stores its 16-column chunks of the tile at tensor-memory column `col`.
__device__ __forceinline__ void store_tile(const Params &prm, uint32_t col, int n, int m0, int quad, int who, int workers)
{
    for (int c0 = who * 16; c0 < prm.block_m; c0 += workers * 16) {
        uint32_t v[16];
        tmem_ld_x16(col + (static_cast<uint32_t>(quad * 32) << 16) + c0, v);
        tmem_ld_wait();
        if (n < prm.rows) {
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const int m = m0 + c0 + j;
                if (m < prm.M) prm.C[static_cast<size_t>(m) * prm.ldc + n] = __uint_as_float(v[j]);
            }
        }
    }
}

template <int NT>
__global__ void __launch_bounds__(THREADS, 1) k_gemm_w41_tc(const __grid_constant__ CUtensorMap map_a, const Params prm)
{
    extern __shared__ __align__(1024) unsigned char smem_dyn[];
    unsigned char *smem = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    uint64_t *raw_full = reinterpret_cast<uint64_t *>(smem + prm.stages * prm.raw_bytes);   // TMA bytes landed
    uint64_t *done = raw_full + MAX_STAGES, *a_full = done + DONE_RING;                     // a_full: dequantised
    uint64_t *acc_full = a_full + MAX_A_SLOTS, *acc_empty = acc_full + MAX_ACC_SLOTS, *drain = acc_empty + MAX_ACC_SLOTS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int total = prm.groups_n * prm.tiles_m;   // work items: (group of NT weight tiles, activation tile)
    const int q_bytes = prm.block_m * 128, w_off = q_bytes, s_off = w_off + NT * RAW_W_BYTES;

    if (threadIdx.x == 0) {
        for (int i = 0; i < prm.stages; i++) mbar_init(&raw_full[i], 2);
        for (int i = 0; i < DONE_RING; i++) mbar_init(&done[i], 1);
        for (int i = 0; i < prm.a_slots; i++) mbar_init(&a_full[i], DEQ_WARPS / (NT == 2 ? 2 : 4));
        for (int i = 0; i < prm.acc_slots; i++) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], prm.acc_slots == 1 ? DEQ_WARPS + EPI_WARPS : EPI_WARPS);
        }
        mbar_init(drain, 1);
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&map_a);
    }
    if (warp == 2) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot, tmem_a = tmem_base + prm.acc_slots * NT * prm.block_m;
    // Launched with programmatic stream serialization: everything above may overlap the tail of the kernel before this one
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (warp == 0 || warp == 3) {
        // ------------------------------ TMA producers: activations, weights ------------------------------
        if (elect_one()) {
            Ring raw(prm.stages);
            uint32_t g = 0;   // stages issued so far, over all tiles of this CTA
            for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
                const int tg = tile / prm.tiles_m, tm = tile % prm.tiles_m;
                const int nvalid = min(NT, prm.tiles_n - tg * NT);   // weight tiles of this group that exist
                for (int p = 0; p < prm.pairs; p++, g++) {
                    if (g >= static_cast<uint32_t>(prm.stages)) {   // the slot last held stage g - stages: free once its MMAs have completed
                        const uint32_t h = g - prm.stages;
                        wait_bounded(&done[h % DONE_RING], (h / DONE_RING) & 1u, abort_flag, prm.flag);
                    }
                    unsigned char *st = smem + raw.idx * prm.raw_bytes;
                    uint64_t *bar = &raw_full[raw.idx];
                    if (warp == 0) {
                        mbar_arrive_expect_tx(bar, q_bytes);
                        tma_tensor2d_g2s(st, &map_a, p * 64, tm * prm.block_m, bar);
                    } else {
                        mbar_arrive_expect_tx(bar, nvalid * (RAW_W_BYTES + RAW_S_BYTES));
                        for (int wt = 0; wt < nvalid; wt++) {
                            const size_t slab = static_cast<size_t>(tg * NT + wt) * prm.pairs + p;
                            tma_bulk_g2s(st + w_off + wt * RAW_W_BYTES, prm.nibT + slab * RAW_W_BYTES, RAW_W_BYTES, bar);
                            tma_bulk_g2s(st + s_off + wt * RAW_S_BYTES, reinterpret_cast<const unsigned char *>(prm.sc16) + slab * RAW_S_BYTES, RAW_S_BYTES, bar);
                        }
                    }
                    raw.advance();
                }
            }
            if (*abort_flag != 0) {   // copies nobody consumed may still be in flight: wait (bounded) for each stage's last fill
                for (uint32_t s = 0; s < static_cast<uint32_t>(prm.stages) && s < g; s++) mbar_wait_drain(&raw_full[s], s < raw.idx ? raw.phase : raw.phase ^ 1);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ------------------------------
        if (elect_one()) {
            const uint32_t idesc = umma_idesc_f16(TILE_N, prm.block_m);
            // A: lane = weight row, eight columns (16 halves) per MMA.  B: activations, 128-byte swizzled rows of 64 halves; slice j is the
            // j-th 32-byte part of the row; 8-row groups are 1024 B apart.  The start-address field counts 16-byte units.
            const uint64_t b_first = umma_smem_desc(smem_u32(smem), 16, 1024, 2);
            const uint32_t b_step = prm.raw_bytes >> 4;
            Ring as(prm.a_slots), acc(prm.acc_slots);
            uint32_t stage = 0, ring = 0;
            for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
                const bool both = NT == 2 && prm.tiles_n - (tile / prm.tiles_m) * NT > 1;
                wait_bounded(&acc_empty[acc.idx], acc.phase ^ 1, abort_flag, prm.flag);
                const uint32_t d = tmem_base + acc.idx * NT * prm.block_m;
#pragma unroll 1
                for (int p = 0; p < prm.pairs; p++) {
                    // The dequantising warps have waited for the whole stage, the activations among it, before they arrive here
                    wait_bounded(&a_full[as.idx], as.phase, abort_flag, prm.flag);
                    tc_fence_after_sync();
                    const uint64_t b0 = b_first + stage * b_step;
                    const uint32_t a0 = tmem_a + as.idx * NT * A_COLS;
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        umma_f16_ts(d, a0 + j * 8, b0 + static_cast<uint64_t>(j * 2), idesc, (p > 0 || j > 0) ? 1u : 0u);
                        if (both) umma_f16_ts(d + prm.block_m, a0 + A_COLS + j * 8, b0 + static_cast<uint64_t>(j * 2), idesc, (p > 0 || j > 0) ? 1u : 0u);
                    }
                    umma_commit(&done[ring]);   // the only commit of the pair
                    ring = (ring + 1) % DONE_RING;
                    if (++stage == static_cast<uint32_t>(prm.stages)) stage = 0;
                    as.advance();
                }
                umma_commit(&acc_full[acc.idx]);
                acc.advance();
            }
            umma_commit(drain);   // every MMA has completed before tensor memory is released
            mbar_wait_drain(drain, 0u);
        }
        __syncwarp();
    } else if (warp >= 4) {
        const int quad = warp & 3;                            // TMEM lane quadrant this warp may access
        const int r = quad * 32 + lane;                       // weight row inside the tile
        const int sub = (warp - 4) >> 2;                      // 0 .. 3: dequantise, 4: epilogue
        Ring acc(prm.acc_slots);
        // Two 16-byte chunks per thread and stage: two weight tiles: the same chunk of both, every other stage; one: both
        // chunks of a row, every fourth stage.  Fewer and longer turns: waiting, storing and handing over cost as many
        // instructions as one chunk.
        constexpr uint32_t STEP = (NT == 2) ? 2u : 4u;
        const int c = (NT == 2) ? sub & 1 : 0, swz = (r >> 2) & 1;
        const uint32_t t_row = tmem_a + (static_cast<uint32_t>(quad * 32) << 16) + c * 8;
        const uint32_t nib0 = w_off + r * 32 + ((c ^ swz) << 4), nib1 = (NT == 2) ? nib0 + RAW_W_BYTES : nib0 ^ 16u, sc0 = s_off + r * 8;
        const uint32_t mask = prm.a_slots - 1, base = smem_u32(smem);
        uint32_t g = (NT == 2) ? sub >> 1 : sub, end = 0, idx = g, phase = 0;   // this warp's next stage, over all tiles of the CTA
        if (idx >= static_cast<uint32_t>(prm.stages)) {
            idx -= prm.stages;
            phase = 1;
        }
        for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
            end += prm.pairs;
            // ------------------------------ dequantise ------------------------------
#pragma unroll 1
            for (; sub < 4 && g < end; g += STEP) {
                // A barrier's phase may be waited for only when the one before has completed.  With many stages the turns before
                // this one have seen to that
                if (static_cast<uint32_t>(prm.stages) < prm.a_slots + STEP && g >= static_cast<uint32_t>(prm.stages)) {
                    const uint32_t h = g - prm.stages;
                    wait_bounded(&done[h % DONE_RING], (h / DONE_RING) & 1u, abort_flag, prm.flag);
                }
                wait_bounded(&raw_full[idx], phase, abort_flag, prm.flag);
                const uint32_t st = base + idx * prm.raw_bytes;
                idx += STEP;
                if (idx >= static_cast<uint32_t>(prm.stages)) {
                    idx -= prm.stages;
                    phase ^= 1;
                }
                const uint4 v[2] = {lds_u32x4(st + nib0), lds_u32x4(st + nib1)};   // a missing tile's bytes are old ones: not used
                const uint2 sc[2] = {lds_u32x2(st + sc0), lds_u32x2(st + sc0 + (NT == 2 ? RAW_S_BYTES : 0))};   // {d_lo, d_hi | m_lo, m_hi}
                uint32_t lo[2][8], hi[2][8];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const __half2 d2 = halves(sc[u].x), m2 = halves(sc[u].y);
                    const __half2 d_lo = __low2half2(d2), d_hi = __high2half2(d2), m_lo = __low2half2(m2), m_hi = __high2half2(m2);
                    const uint32_t in[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
                    for (int i = 0; i < 4; i++) dequant4(in[i], d_lo, m_lo, d_hi, m_hi, &lo[u][2 * i], &hi[u][2 * i]);
                }
                if (g >= static_cast<uint32_t>(prm.a_slots)) {   // the columns last held stage g - a_slots
                    const uint32_t h = g - prm.a_slots;
                    wait_bounded(&done[h % DONE_RING], (h / DONE_RING) & 1u, abort_flag, prm.flag);
                }
                tc_fence_after_sync();
                const uint32_t t = t_row + (g & mask) * (NT * A_COLS);
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    tmem_st_x8(t + u * (NT == 2 ? A_COLS : 8), lo[u]);
                    tmem_st_x8(t + u * (NT == 2 ? A_COLS : 8) + 16, hi[u]);
                }
                tmem_st_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (elect_one()) mbar_arrive(&a_full[g & mask]);
            }
            // ------------------------------ epilogue ------------------------------
            // The dequantising warps help with the last tile, and with every tile when the next one's products wait for the stores
            // (a single accumulator).  Tiles of fewer than four stages: the warps may be further ahead than one phase of acc_full
            const bool help = prm.acc_slots == 1 || (tile + static_cast<int>(gridDim.x) >= total && prm.pairs >= 4);
            if (sub == 4 || help) {
                const int tg = tile / prm.tiles_m, tm = tile % prm.tiles_m;
                const int nvalid = min(NT, prm.tiles_n - tg * NT);
                wait_bounded(&acc_full[acc.idx], acc.phase, abort_flag, prm.flag);
                tc_fence_after_sync();
                for (int wt = 0; wt < nvalid; wt++)
                    store_tile(prm, tmem_base + (acc.idx * NT + wt) * prm.block_m, (tg * NT + wt) * TILE_N + r, tm * prm.block_m, quad, help ? sub : 0, help ? 5 : 1);
                tc_fence_before_sync();
                __syncwarp();
                if ((sub == 4 || prm.acc_slots == 1) && elect_one()) mbar_arrive(&acc_empty[acc.idx]);
            }
            acc.advance();
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}

template <int NT>
static int launch(inkq_ctx *ctx, const uint16_t *a16, int M, const Weight *w, float *C, int ldc, int block_m)
{
    const Shape sh{NT, block_m};
    CUtensorMap map;
    int rc = encode_map_2d(ctx, &map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a16, w->K, M, 64u, block_m, CU_TENSOR_MAP_SWIZZLE_128B, w->K);
    if (rc) return rc;
    Params prm;
    prm.nibT = w->nibT;
    prm.sc16 = w->sc16;
    prm.C = C;
    prm.flag = ctx->dev_flag;
    prm.M = M;
    prm.rows = w->rows;
    prm.pairs = w->pairs;
    prm.tiles_n = w->tiles;
    prm.groups_n = (w->tiles + NT - 1) / NT;
    prm.tiles_m = (M + block_m - 1) / block_m;
    prm.block_m = block_m;
    prm.ldc = ldc;
    prm.stages = sh.stages();
    prm.raw_bytes = sh.raw_bytes();
    prm.a_slots = sh.a_slots();
    prm.acc_slots = sh.acc_slots();
    if ((rc = allow_smem<k_gemm_w41_tc<NT>>(ctx))) return rc;
    const int total = prm.groups_n * prm.tiles_m;
    const cudaError_t e = launch_pdl(k_gemm_w41_tc<NT>, dim3(total < ctx->num_sms ? total : ctx->num_sms), dim3(THREADS), SMEM_BYTES, ctx->stream, map, prm);
    if (e != cudaSuccess) return fail(ctx, INKQ_ERR_CUDA, std::string("k_gemm_w41_tc launch: ") + cudaGetErrorString(e));
    return after_launch(ctx, "k_gemm_w41_tc");
}

}  // namespace w41

int launch_gemm_w41_tc(inkq_ctx *ctx, const uint16_t *a16, int M, const Weight *w, float *C, int ldc)
{
    using namespace w41;
    if (ctx->encode_tiled == nullptr) return fail(ctx, INKQ_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled entry point not available");
    if ((reinterpret_cast<uintptr_t>(a16) & 15) != 0) return fail(ctx, INKQ_ERR_INVALID, "the fp16 activations must be 16-byte aligned");
    // The split with the least time: waves x time of a wave (us at K = 4096, measured as what a second tile on every SM adds; it
    // is proportional to K).  Dequantising bounds narrow tiles (one weight tile
    // 13.4, two 26.4), the products wide ones.  One weight tile leaves fewer SMs idle where there are few tiles; two share the
    // activations, which pays beyond ~190 rows (192 rows: 22.6 twice against 42.6).
    Shape best{1, 0};
    float best_time = 0.f;
    for (int nt = 1; nt <= 2; nt++) {
        const int max_m = nt == 1 ? 256 : 192;
        for (int tm = (M + max_m - 1) / max_m; tm <= (M + 15) / 16; tm++) {
            const int bm = (((M + tm - 1) / tm) + 15) & ~15;
            const long long total = static_cast<long long>((w->tiles + nt - 1) / nt) * ((M + bm - 1) / bm);
            const float wave = nt == 1 ? fmaxf(13.4f, 5.0f + 0.098f * bm) : fmaxf(26.4f, 17.2f + 0.131f * bm);
            const float time = static_cast<float>((total + ctx->num_sms - 1) / ctx->num_sms) * wave;
            if (best_time == 0.f || time < best_time) {
                best = Shape{nt, bm};
                best_time = time;
            }
            if (total > 64LL * ctx->num_sms) break;   // many waves already: finer splits only dequantise more often
        }
    }
    return best.nt == 2 ? launch<2>(ctx, a16, M, w, C, ldc, best.block_m) : launch<1>(ctx, a16, M, w, C, ldc, best.block_m);
}

}  // namespace inkq
