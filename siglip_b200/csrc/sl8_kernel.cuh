// sl8_kernel.cuh -- the persistent, warp-specialised FP8 GEMM kernel with fused epilogues.
//
// One kernel template covers the three layers (patch-embed + periodic table add,
// FC1 + bias + GELU, FC2 + bias + residual) and every tile configuration.  It is the
// counterpart of the reference's persistent_gemm<EpilogueOp> (kernel_body.cuh:448-815) and
// epilogue_store (kernel_body.cuh:47-442), rebuilt around run-time M/N/K:
//
//   Every role walks its loop as a whole warp and issues through an elected lane (see the MMA role).
//
//   warp 0        TMA producer of A: streams A[128 x 128B] k-blocks into a ring of STAGES
//                 shared-memory stages (SWIZZLE_128B), one mbarrier pair (full / empty) per stage,
//                 and announces the stage's bytes.
//   warp 3 + EPI  TMA producer of B: streams B[TN/CG x 128B] k-blocks into the same stages.  Two
//                 issuing threads because a thread's next bulk-tensor copy is not accepted before the
//                 TMA unit has generated the requests of its previous one (2 cycles per 128-byte row:
//                 64 bytes per clock per issuing thread, measured), while the unit itself serves two
//                 threads at once at 128 bytes per clock: one thread cannot feed a 256 x 256 tile.
//   warp 1        one elected thread of the leader CTA's issues tcgen05.mma kind::f8f6f4 (E4M3 x E4M3 -> FP32 in TMEM), four K=32 steps per
//                 k-block (fewer in the K tail), and commits to the stage's empty barrier and,
//                 after the last k-block, to the accumulator's full barrier.
//   warps 2..     epilogue: tcgen05.ld of the finished accumulator (two accumulators in TMEM,
//                 so the MMA of tile i+1 overlaps the epilogue of tile i), dequantisation
//                 scale, fused bias / GELU / residual / table add, conversion to bf16 or
//                 e4m3 into swizzled shared staging, TMA tensor stores.  The residual / table
//                 values of a 32-row x 128-byte region are brought into that same staging buffer
//                 by a TMA load a few regions ahead, added in place and stored from there.
//
//   warp 2 + EPI  side-data loader (patch-embed, FC2): one lane issues the TMA loads that bring the table /
//                 residual regions into the epilogue warps' staging buffers as those become free, so
//                 the epilogue warps never wait for a TMA instruction to be accepted.
//
// CG == 2 runs a CTA pair per tile (cluster of two, tcgen05 cta_group::2): each CTA loads its
// own 128 rows of A and half of the tile's B rows, the leader issues 256 x TN MMAs that read
// both CTAs' shared memory and write both CTAs' tensor memory.
//
// Tiles are dealt round-robin (tile = cluster index + i * clusters) in N-fastest order, so
// the clusters running at any moment share a few A row-blocks and the whole of B in L2.
//
// Every wait is bounded: when a poll loop exceeds the budget it records where it was in the
// status block, raises a CTA-wide abort flag that every other wait loop checks, and all
// roles fall through to the common exit, which still frees tensor memory.
#pragma once

#include "sl8_ptx.cuh"

#ifndef SL8_SPIN_CRITICAL
#define SL8_SPIN_CRITICAL true
#endif

namespace sl8 {

enum : int { OP_PE = 0, OP_FC1 = 1, OP_FC2 = 2 };
enum : int { OUT_BF16 = 0, OUT_E4M3 = 1 };
// Measurement aids (skip one part of the kernel to time the rest).  They cost instructions in the
// hot loops, so they exist only in a library built with -DSL8_DIAG.
#ifdef SL8_DIAG
#define SL8_DBG(flags, bit) (((flags) & (bit)) != 0u)
#else
#define SL8_DBG(flags, bit) false
#endif

// FLAG_COARSE_TRACE (set by the library, never by a caller): with tracing on, record only the per-role totals; the
// roles then run their untimed code paths, so the totals are those of the kernel as it runs without tracing.
enum : unsigned { FLAG_BIAS_F32 = 1u, FLAG_PE_F32_ADD = 2u, FLAG_NO_ACTIVATION = 4u, FLAG_GELU_HW_TANH = 8u,
                  FLAG_COARSE_TRACE = 0x40000000u,
                  FLAG_TEST_DROP_B = 0x10000000u,  // test aid (set by the library from SL8_TEST_DROP_B): the B copy of k-block 1 of each cluster's first tile is
                                                   // never issued, so the MMA thread's bounded wait for that stage runs out
                  FLAG_SINGLE_ACC = 0x20000000u,   // measurement aid (set by the library from SL8_SINGLE_ACC): one accumulator, no MMA / epilogue overlap
                  DBG_SKIP_SIDE = 0x100u, DBG_SKIP_GELU = 0x200u, DBG_SKIP_BIAS = 0x400u, DBG_SKIP_STORE = 0x800u,
                  DBG_SKIP_LOAD = 0x1000u, DBG_SKIP_EPILOGUE = 0x2000u, DBG_SKIP_MMA = 0x4000u,
                  DBG_SKIP_A = 0x8000u, DBG_SKIP_B = 0x10000u, DBG_SKIP_TMEM_LD = 0x20000u, DBG_SKIP_MATH = 0x40000u,
                  DBG_COARSE_TRACE = 0x80000000u };   // record per-role totals only (the inner timers cost ~35 cycles each)

// status[0] codes: which role gave up.
enum : uint32_t {
    ST_OK = 0,
    ST_PRODUCER_EMPTY_WAIT = 1,
    ST_MMA_FULL_WAIT = 2,
    ST_MMA_TMEM_EMPTY_WAIT = 3,
    ST_EPI_TMEM_FULL_WAIT = 4,
    ST_EPI_SIDE_WAIT = 5,
    ST_SIDE_LOADER_WAIT = 6
};

// Tracing slots written per CTA when KernelParams::prof is set (cycles, clock64).
enum : int {
    PROF_PRODUCER_WAIT = 0,   // TMA producer waiting for a free stage
    PROF_PRODUCER_TOTAL = 1,
    PROF_MMA_WAIT_FULL = 2,   // MMA thread waiting for operands
    PROF_MMA_WAIT_TMEM = 3,   // MMA thread waiting for a free accumulator
    PROF_MMA_TOTAL = 4,
    PROF_EPI_WAIT_ACC = 5,    // epilogue warp 0 waiting for a finished accumulator
    PROF_EPI_TOTAL = 6,
    PROF_EPI_WAIT_STORE = 7,  // epilogue warp 0 waiting for staging to drain
    PROF_TILES = 8,
    PROF_EPI_WAIT_LD = 9,     // epilogue warp 0 waiting for tcgen05.ld
    PROF_EPI_MATH = 10,       // epilogue warp 0: transform + staging writes
    PROF_EPI_STORE_ISSUE = 11,// epilogue warp 0: proxy fence + TMA store issue
    PROF_EPI_REFILL = 12,     // epilogue warp 0: waiting until the previous store has read its staging buffer
    PROF_EPI_PREFETCH = 13,   // epilogue warp 0: issuing the side-data prefetch
    PROF_MMA_ISSUE = 14,      // MMA thread: issuing tcgen05.mma
    PROF_MMA_COMMIT = 15,     // MMA thread: issuing tcgen05.commit
    PROF_SLOTS = 16
};

struct KernelParams {
    long long M;
    int N;
    int K;
    int tiles_n;
    int num_tiles;
    unsigned tiles_n_magic;          // ceil(2^32 / tiles_n), 0 for tiles_n == 1 (see TileWalk)
    int step_m, step_n;              // what one round adds to a cluster's tile: clusters / tiles_n row-blocks, clusters % tiles_n columns
    int k_blocks;          // ceil(K / TILE_K)
    int last_kblock_mmas;  // K = 32 steps needed in the last k-block (1 .. TILE_K / 32)
    int tail_cols;         // columns of the last N tile: N - (tiles_n - 1) * TN, a multiple of 16 (== TN when N % TN == 0)
    const float* scale_a;
    const float* scale_b;
    const float* out_scale;
    const void* bias;                // bf16 [N] or fp32 [N] (FLAG_BIAS_F32); may be null
    const __nv_bfloat16* side;       // table [period, N] (patch-embed) or residual [M, N] (FC2)
    long long ld_side;               // elements
    int period;
    int row_phase;
    int table_rows;                  // rows the table holds: >= period; rows past period repeat it (patch-embed)
    void* D;
    long long ldd;                   // elements of the output type
    unsigned flags;
    unsigned wait_budget_us;         // budget of every device-side wait, microseconds
    uint32_t* status;                // 4 words: code, barrier/stage, tile, block
    long long* prof;                 // optional: PROF_SLOTS clock64 totals per CTA (null = tracing off)
};

template <int CG, int TN, int TK, int STAGES, int EPI_WARPS, int OUT, int NBUF>
struct KernelTraits {
    static_assert(CG == 1 || CG == 2, "one CTA or a CTA pair per tile");
    static_assert(TN == 64 || TN == 128 || TN == 192 || TN == 256, "tile N");
    static_assert(EPI_WARPS == 4 || EPI_WARPS == 8 || EPI_WARPS == 16, "one, two or four warps per TMEM lane quadrant");
    static_assert(NBUF >= 1 && NBUF <= 4, "staging buffers per epilogue warp");
    static constexpr int TILE_M_CTA = 128;                       // rows per CTA = TMEM lanes
    static_assert(TK == 128 || TK == 256, "bytes of K per stage: one or two 128-byte swizzle atoms");
    static constexpr int TILE_K = TK;                            // bytes of K per stage
    static constexpr int KATOMS = TK / 128;                      // 128-byte swizzle atoms per stage and operand
    static constexpr int B_ROWS = TN / CG;                       // B rows this CTA loads per stage
    // Where a CTA's share of B has 64 rows, the B producer brings the last 32 of A's 128 as well (boxes of 32 rows): an issuing
    // thread's copies take 2 cycles per row, so 96 + 96 rows take 192 cycles per k-block and 128 + 64 take 256.
    static constexpr bool SPLIT_A = (B_ROWS == 64 && KATOMS == 1);
    static constexpr int A_BOX_ROWS = SPLIT_A ? 32 : TILE_M_CTA; // rows of one copy of A: the box of map_a (VariantEntry::a_box_rows)
    static constexpr int A_ATOM_BYTES = TILE_M_CTA * 128;        // 16 KiB: 128 rows x 128 bytes
    static constexpr int B_ATOM_BYTES = B_ROWS * 128;
    static constexpr int A_BYTES = KATOMS * A_ATOM_BYTES;
    static constexpr int B_BYTES = KATOMS * B_ATOM_BYTES;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;        // also the bytes one CTA's TMA adds per stage
    static constexpr int ACC_STRIDE = TN;                        // TMEM columns between the two accumulators
    static constexpr int TMEM_COLS = (TN == 192) ? 512 : 2 * TN; // a power of two >= 32
    static constexpr int OUT_BYTES = (OUT == OUT_BF16) ? 2 : 1;
    static constexpr int COLS_PER_WARP = TN / (EPI_WARPS / 4);   // columns one epilogue warp covers
    // A staging row is 128 bytes (SWIZZLE_128B), or 64 (SWIZZLE_64B) where a warp's columns are no multiple of that: e4m3
    // output, 64 one-byte columns per warp (sixteen warps, 64-column tiles) or 192.
    static constexpr int REGION_ROW_BYTES = (COLS_PER_WARP * OUT_BYTES % 128 != 0) ? 64 : 128;
    static constexpr int REGION_COLS = REGION_ROW_BYTES / OUT_BYTES;   // output columns in one staging row
    static constexpr int REGION_BYTES = 32 * REGION_ROW_BYTES;   // 32 rows of one warp
    static constexpr int STAGING_BYTES = EPI_WARPS * NBUF * REGION_BYTES;
    static constexpr int REGIONS_PER_TILE = COLS_PER_WARP / REGION_COLS;
    static constexpr int CHUNKS_PER_REGION = REGION_COLS / 32;   // 32-column tcgen05.ld chunks per region
    static constexpr int BAR_BYTES = 512;                        // pipeline barriers + two per staging box
    // fp32 bias of the current tile: one copy per epilogue warp in shared memory (broadcast reads) where that fits;
    // a configuration that needs every byte for the operand ring keeps it in registers instead (lane l holds the
    // bias of column l of each 32-column chunk) and broadcasts by warp shuffle.
    static constexpr bool BIAS_IN_SMEM = 1024 + STAGES * STAGE_BYTES + STAGING_BYTES + EPI_WARPS * COLS_PER_WARP * 4 + 512 <= 232448;
    static constexpr int BIAS_BYTES = BIAS_IN_SMEM ? EPI_WARPS * COLS_PER_WARP * 4 : 0;
    static constexpr int THREADS = (4 + EPI_WARPS) * 32;         // A producer, MMA, epilogue warps, side-data loader, B producer
    static constexpr int SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + STAGING_BYTES + BIAS_BYTES + BAR_BYTES;
    static_assert(STAGE_BYTES % 1024 == 0, "every operand tile must start on a swizzle-atom boundary");
    static_assert(COLS_PER_WARP % REGION_COLS == 0, "a warp stores whole staging regions");
    static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KiB a CTA may use");
    // A launch that waits for the one ahead of it (pdl_wait) already holds tensor memory: it must not sit on that one's SMs.
    static_assert(!SPLIT_A || 96 + A_BOX_ROWS == TILE_M_CTA, "three boxes from one producer, the last one from the other");
    static_assert(2 * SMEM_BYTES > 228 * 1024, "two CTAs must not fit one SM");
};

// The tiles of one cluster: cluster, cluster + clusters, ... in N-fastest order.  No division: the first tile's number is
// small enough for a multiplication (exact for any tiles_n while there are no more than 2^16 clusters), later ones are steps.
struct TileWalk {
    int tile, tm, tn;
    __device__ __forceinline__ TileWalk(const KernelParams& p, int cluster)
        : tile(cluster), tm(p.tiles_n_magic ? static_cast<int>(static_cast<uint64_t>(cluster) * p.tiles_n_magic >> 32) : cluster) {
        tn = cluster - tm * p.tiles_n;
    }
    __device__ __forceinline__ void next(const KernelParams& p, int clusters) {
        tile += clusters;
        tm += p.step_m;
        tn += p.step_n;
        if (tn >= p.tiles_n) { tn -= p.tiles_n; tm++; }
    }
};

// Host side of TileWalk: the launch's clusters are known.
inline void set_tile_walk(KernelParams& p, int clusters) {
    p.tiles_n_magic = p.tiles_n > 1 ? static_cast<unsigned>((0x100000000ull + p.tiles_n - 1) / p.tiles_n) : 0u;
    p.step_m = clusters / p.tiles_n;
    p.step_n = clusters % p.tiles_n;
}

struct WaitCtx {
    volatile uint32_t* abort_flag;  // shared memory, one per CTA
    uint32_t peer_abort;            // shared::cluster address of the other CTA's flag in a CTA pair, else 0
    uint32_t* status;
    unsigned long long budget_ns;
    uint32_t tile;
};

// Polls `bar` until the phase with parity `parity` has completed.  Returns false if the CTA
// is aborting or the budget ran out (in which case it records `code` and raises the flag).
// All lanes of a warp call it together: a branch for one lane, its reconvergence and a second poll by the others cost 700 -
// 1 000 cycles where the barrier had long completed (embed of one image, from the last MMA to the first tcgen05.ld 2 000
// cycles, 400 as it stands; a block of 729 rows 46.9 -> 45.7 us).
// SPIN: poll without parking the warp (the roles on the critical path, whose wake-up latency is paid by the whole CTA
// pair); otherwise kPolls polls, and from then on each may park the warp until the phase completes (a parking poll costs
// several hundred cycles even on a barrier that is complete).
constexpr uint32_t kPolls = 64;
template <bool SPIN = false>
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, const WaitCtx& w, uint32_t code,
                                         uint32_t which) {
    if (mbar_test_wait(bar, parity) != 0u) return true;
    if constexpr (!SPIN) {
#pragma unroll 1
        for (uint32_t i = 0; i < kPolls; ++i)
            if (mbar_test_wait(bar, parity) != 0u) return true;
    }
    unsigned long long t0 = 0;
    for (uint32_t spins = 1;; ++spins) {
        if (SPIN ? (mbar_test_wait(bar, parity) != 0u) : mbar_try_wait(bar, parity)) return true;
        if ((spins & (SPIN ? 255u : 15u)) == 0) {   // each parked poll may have lasted up to 20 us
            if (*w.abort_flag) return false;
            const unsigned long long now = globaltimer_ns();
            if (t0 == 0) {
                t0 = now;
            } else if (now - t0 > w.budget_ns) {
                *w.abort_flag = 1u;
                // the other CTA of a pair would otherwise sit out its own full budget on barriers only this CTA feeds
                if (w.peer_abort) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(w.peer_abort), "r"(1u) : "memory");
                if (atomicCAS(w.status, 0u, code) == 0u) {
                    w.status[1] = which;
                    w.status[2] = w.tile;
                    w.status[3] = blockIdx.x;
                }
                return false;
            }
        }
    }
}

// tanh-form GELU of the reference (fc1_gelu.cu:16-19) written without the 1 + tanh
// cancellation: 0.5 x (1 + tanh u) == x * sigmoid(2u) == x / (1 + exp(-2u)), with
// u = sqrt(2/pi) (x + 0.044715 x^3).  Two SFU operations (ex2, rcp) per element; everything else
// runs two elements per instruction on packed fp32 pairs.
__device__ __forceinline__ uint64_t gelu_tanh_x2(uint64_t x) {
    constexpr float K0 = -2.0f * 0.7978845608f * 1.4426950408889634f;   // -2 sqrt(2/pi) log2(e)
    constexpr float K1 = K0 * 0.044715f;
    const uint64_t x2 = mul_f32x2(x, x);
    const uint64_t t = mul_f32x2(x, fma_f32x2(x2, pack_f32x2(K1, K1), pack_f32x2(K0, K0)));   // -2 u log2(e)
    float t0, t1;
    unpack_f32x2(t, t0, t1);
    const uint64_t d = add_f32x2(pack_f32x2(ex2_approx(t0), ex2_approx(t1)), pack_f32x2(1.0f, 1.0f));
    float d0, d1;
    unpack_f32x2(d, d0, d1);
    return mul_f32x2(x, pack_f32x2(rcp_approx(d0), rcp_approx(d1)));    // x / inf == 0
}

// The same GELU through the hardware tanh (tanh.approx.f32: one SFU operation per element instead of two, relative
// error about 2^-11, so |error| <= ~2.5e-4 |x|): 0.5 x (1 + tanh u) = h + h tanh u with h = x / 2.  Opt-in
// (SL8_FLAG_GELU_HW_TANH); inside the 1e-2 relative tolerance of bf16 outputs except where the result itself is within
// ~1e-3 of zero, but not bit-comparable to the exact form.
__device__ __forceinline__ uint64_t gelu_hw_tanh_x2(uint64_t x) {
    constexpr float C0 = 0.7978845608f, C1 = 0.7978845608f * 0.044715f;
    const uint64_t x2 = mul_f32x2(x, x);
    const uint64_t u = mul_f32x2(x, fma_f32x2(x2, pack_f32x2(C1, C1), pack_f32x2(C0, C0)));
    float u0, u1;
    unpack_f32x2(u, u0, u1);
    const uint64_t h = mul_f32x2(x, pack_f32x2(0.5f, 0.5f));
    return fma_f32x2(h, pack_f32x2(tanh_approx(u0), tanh_approx(u1)), h);
}

__device__ __forceinline__ void unpack8_bf16(const uint4& q, float (&f)[8]) {
    f[0] = bf16_lo_f32(q.x); f[1] = bf16_hi_f32(q.x);
    f[2] = bf16_lo_f32(q.y); f[3] = bf16_hi_f32(q.y);
    f[4] = bf16_lo_f32(q.z); f[5] = bf16_hi_f32(q.z);
    f[6] = bf16_lo_f32(q.w); f[7] = bf16_hi_f32(q.w);
}

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 r;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(addr));
    return r;
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// Per-warp epilogue constants.
struct EpiCtx {
    float scale;      // scale_a * scale_b
    float inv_out;    // 1 / out_scale
    uint32_t row_off; // lane * row bytes: byte offset of this lane's row inside a staging region
    uint32_t swz;     // XOR applied to the 16-byte piece index: lane & 7 (SWIZZLE_128B) or (lane >> 1) & 3 (SWIZZLE_64B)
    unsigned flags;
};

// Transforms 16 accumulator columns (v[16*H .. 16*H+15]) of this lane's row and writes them to the
// staging region at `region` (shared address), 16-byte pieces `piece0`.. of the lane's 128-byte row.
// bias16: the 16 fp32 bias values of these columns in shared memory (FC1 / FC2).  With side data
// (patch-embed table, FC2 residual) the 16 bf16 side values already sit in the staging region at the
// very place the result goes; they are read, combined and overwritten.
// Four consecutive bias values of the half-chunk: from the warp's shared copy, or (BSM false) from the chunk's
// bias register of lanes first .. first + 3.  Every lane of the warp must call it.
template <bool BSM>
__device__ __forceinline__ float4 bias_quad(const float* bias16, float breg, int first, int i) {
    if constexpr (BSM) {
        return *reinterpret_cast<const float4*>(bias16 + 4 * i);
    } else {
        float4 b;
        b.x = __shfl_sync(0xffffffffu, breg, first + 4 * i + 0);
        b.y = __shfl_sync(0xffffffffu, breg, first + 4 * i + 1);
        b.z = __shfl_sync(0xffffffffu, breg, first + 4 * i + 2);
        b.w = __shfl_sync(0xffffffffu, breg, first + 4 * i + 3);
        return b;
    }
}

template <int OP, int OUT, int H, bool BSM>
__device__ __forceinline__ void epilogue_16(const float (&v)[32], const EpiCtx& e, const float* bias16, float breg,
                                            uint32_t region, int piece0) {
    float x[16];
    uint32_t w[8];  // bf16: 8 words (16 values); e4m3: 4 words used
    const uint32_t a0 = region + e.row_off + (((piece0 + 0) ^ e.swz) << 4);
    const uint32_t a1 = region + e.row_off + (((piece0 + 1) ^ e.swz) << 4);

    if constexpr (OP == OP_PE) {
        const uint4 s0 = lds128(a0), s1 = lds128(a1);
#pragma unroll
        for (int i = 0; i < 16; i++) x[i] = v[16 * H + i] * e.scale;
        const uint32_t tw[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
        if (e.flags & FLAG_PE_F32_ADD) {
#pragma unroll
            for (int i = 0; i < 8; i++)
                w[i] = pack_bf16x2(x[2 * i] + bf16_lo_f32(tw[i]), x[2 * i + 1] + bf16_hi_f32(tw[i]));
        } else {
            // The reference's order: round the accumulator to bf16, then add in bf16 (patch_embed.cu:51-58).
#pragma unroll
            for (int i = 0; i < 8; i++) w[i] = add_bf16x2(pack_bf16x2(x[2 * i], x[2 * i + 1]), tw[i]);
        }
    } else if constexpr (OP == OP_FC1) {
        // acc * scale + bias, GELU and the output scaling on packed fp32 pairs; the bias comes from shared
        // memory, the same address in every lane (a broadcast read).
        const uint64_t scale2 = pack_f32x2(e.scale, e.scale);
        const uint64_t inv2 = pack_f32x2(e.inv_out, e.inv_out);
        uint64_t g[8];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 b = bias_quad<BSM>(bias16, breg, 16 * H, i);
            g[2 * i + 0] = fma_f32x2(pack_f32x2(v[16 * H + 4 * i + 0], v[16 * H + 4 * i + 1]), scale2, pack_f32x2(b.x, b.y));
            g[2 * i + 1] = fma_f32x2(pack_f32x2(v[16 * H + 4 * i + 2], v[16 * H + 4 * i + 3]), scale2, pack_f32x2(b.z, b.w));
        }
        if (e.flags & FLAG_GELU_HW_TANH) {                                           // warp-uniform branches
#pragma unroll
            for (int i = 0; i < 8; i++) g[i] = gelu_hw_tanh_x2(g[i]);
        } else if (!(e.flags & FLAG_NO_ACTIVATION) && !SL8_DBG(e.flags, DBG_SKIP_GELU)) {
#pragma unroll
            for (int i = 0; i < 8; i++) g[i] = gelu_tanh_x2(g[i]);
        }
        if constexpr (OUT == OUT_BF16) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                float lo, hi;
                unpack_f32x2(g[i], lo, hi);
                w[i] = pack_bf16x2(lo, hi);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                float a, b, c, d;
                unpack_f32x2(mul_f32x2(g[2 * i + 0], inv2), a, b);
                unpack_f32x2(mul_f32x2(g[2 * i + 1], inv2), c, d);
                w[i] = static_cast<uint32_t>(pack_e4m3x2(a, b)) | (static_cast<uint32_t>(pack_e4m3x2(c, d)) << 16);
            }
        }
    } else {  // OP_FC2: (acc * scale + bias) + residual, fc2.cu:27-46
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 b = bias_quad<BSM>(bias16, breg, 16 * H, i);
            x[4 * i + 0] = fmaf(v[16 * H + 4 * i + 0], e.scale, b.x);
            x[4 * i + 1] = fmaf(v[16 * H + 4 * i + 1], e.scale, b.y);
            x[4 * i + 2] = fmaf(v[16 * H + 4 * i + 2], e.scale, b.z);
            x[4 * i + 3] = fmaf(v[16 * H + 4 * i + 3], e.scale, b.w);
        }
        float r[8];
        unpack8_bf16(lds128(a0), r);
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] += r[i];
        unpack8_bf16(lds128(a1), r);
#pragma unroll
        for (int i = 0; i < 8; i++) x[8 + i] += r[i];
#pragma unroll
        for (int i = 0; i < 8; i++) w[i] = pack_bf16x2(x[2 * i], x[2 * i + 1]);
    }
    sts128(a0, w[0], w[1], w[2], w[3]);
    if constexpr (OUT == OUT_BF16) sts128(a1, w[4], w[5], w[6], w[7]);
}

// FC1 on a whole 32-column chunk at once: sixteen independent element pairs go through the GELU's special-function
// chain (ex2, rcp) together, which keeps that pipe fed with only two epilogue warps per scheduler.  Used by the variants
// with up to eight epilogue warps (with sixteen, four warps per scheduler hide the chain and registers are scarce).
template <int OUT, bool BSM>
__device__ __forceinline__ void epilogue_32_fc1(const float (&v)[32], const EpiCtx& e, const float* bias32, float breg,
                                                uint32_t region, int piece0) {
    const uint64_t scale2 = pack_f32x2(e.scale, e.scale);
    uint64_t g[16];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float4 b = bias_quad<BSM>(bias32, breg, 0, i);
        g[2 * i + 0] = fma_f32x2(pack_f32x2(v[4 * i + 0], v[4 * i + 1]), scale2, pack_f32x2(b.x, b.y));
        g[2 * i + 1] = fma_f32x2(pack_f32x2(v[4 * i + 2], v[4 * i + 3]), scale2, pack_f32x2(b.z, b.w));
    }
    if (e.flags & FLAG_GELU_HW_TANH) {                                           // warp-uniform branches
#pragma unroll
        for (int i = 0; i < 16; i++) g[i] = gelu_hw_tanh_x2(g[i]);
    } else if (!(e.flags & FLAG_NO_ACTIVATION) && !SL8_DBG(e.flags, DBG_SKIP_GELU)) {
#pragma unroll
        for (int i = 0; i < 16; i++) g[i] = gelu_tanh_x2(g[i]);
    }
    if constexpr (OUT == OUT_BF16) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            float lo, hi;
            unpack_f32x2(g[i], lo, hi);
            w[i] = pack_bf16x2(lo, hi);
        }
#pragma unroll
        for (int q = 0; q < 4; q++)
            sts128(region + e.row_off + (((piece0 + q) ^ e.swz) << 4), w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
    } else {
        const uint64_t inv2 = pack_f32x2(e.inv_out, e.inv_out);
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            float a, b, c, d;
            unpack_f32x2(mul_f32x2(g[2 * i + 0], inv2), a, b);
            unpack_f32x2(mul_f32x2(g[2 * i + 1], inv2), c, d);
            w[i] = static_cast<uint32_t>(pack_e4m3x2(a, b)) | (static_cast<uint32_t>(pack_e4m3x2(c, d)) << 16);
        }
#pragma unroll
        for (int q = 0; q < 2; q++)
            sts128(region + e.row_off + (((piece0 + q) ^ e.swz) << 4), w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
    }
}

// Bias values of columns col0 + lane + 32 i (i < NB) as fp32; zero past N or without a bias.
template <int NB>
__device__ __forceinline__ void load_bias(float (&b)[NB], const void* bias, unsigned flags, int col0, int lane, int N) {
#pragma unroll
    for (int i = 0; i < NB; i++) {
        const int col = col0 + lane + 32 * i;
        float val = 0.0f;
        if (bias != nullptr && col < N)
            val = (flags & FLAG_BIAS_F32) ? ld_f32(static_cast<const float*>(bias) + col) : ld_bf16(static_cast<const __nv_bfloat16*>(bias) + col);
        b[i] = val;
    }
}

template <int CG, int TN, int TK, int STAGES, int EPI_WARPS, int OP, int OUT, int NBUF>
__global__ void __launch_bounds__((4 + EPI_WARPS) * 32, 1)
sl8_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                const __grid_constant__ CUtensorMap map_bt, const __grid_constant__ CUtensorMap map_d,
                const __grid_constant__ CUtensorMap map_s, const KernelParams p) {
    using T = KernelTraits<CG, TN, TK, STAGES, EPI_WARPS, OUT, NBUF>;

    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_u32 = smem_u32(smem_raw);
    const uint32_t base = (raw_u32 + 1023u) & ~1023u;            // swizzle atoms are 1024-byte aligned
    uint8_t* const base_ptr = smem_raw + (base - raw_u32);

    const uint32_t staging_base = base + STAGES * T::STAGE_BYTES;
    const uint32_t bias_base = staging_base + T::STAGING_BYTES;
    const uint32_t bar_base = bias_base + T::BIAS_BYTES;
    // barrier block: full[STAGES] | empty[STAGES] | tmem_full[2] | tmem_empty[2] | tmem ptr | abort
    const uint32_t full_bar0 = bar_base;
    const uint32_t empty_bar0 = bar_base + 8 * STAGES;
    const uint32_t tfull_bar0 = bar_base + 16 * STAGES;
    const uint32_t tempty_bar0 = tfull_bar0 + 16;
    const uint32_t tmem_ptr_addr = tempty_bar0 + 16;
    uint8_t* const bar_ptr = base_ptr + (bar_base - base);
    volatile uint32_t* const tmem_ptr = reinterpret_cast<volatile uint32_t*>(bar_ptr + 16 * STAGES + 32);
    volatile uint32_t* const abort_flag = tmem_ptr + 1;
    const uint32_t side_bar0 = bar_base + 16 * STAGES + 48;     // (EPI_WARPS / 4) * NBUF barriers: side data landed
    const uint32_t side_free0 = side_bar0 + 8 * (EPI_WARPS / 4) * NBUF;   // ... and: staging box reusable
    static_assert(16 * STAGES + 48 + 16 * (EPI_WARPS / 4) * NBUF <= T::BAR_BYTES, "barrier block too small");

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    // Rank inside the CTA pair.  Clusters are (2,1,1) on a one-dimensional grid, so the rank is the parity of
    // blockIdx.x; taking it from there (not from %cluster_ctarank) lets the compiler see it as warp-uniform.
    const uint32_t cta_rank = (CG == 2) ? (blockIdx.x & 1u) : 0u;
    const int cluster_id = blockIdx.x / CG;
    const int num_clusters = gridDim.x / CG;

    WaitCtx wc;
    wc.abort_flag = abort_flag;
    wc.status = p.status;
    wc.budget_ns = static_cast<unsigned long long>(p.wait_budget_us) * 1000ull;
    wc.peer_abort = (CG == 2) ? map_to_cta(smem_u32(const_cast<uint32_t*>(abort_flag)), cta_rank ^ 1u) : 0u;
    wc.tile = 0;

    // ---------------------------------------------------------------- set-up
    // Each part by a warp of its own, and the roles begin before the parts are joined: what a role works out from the
    // parameters runs (and its code and constants are brought in) while the tensor memory is allocated and the pair's other
    // CTA arrives.  A CTA needs 0.8 (alone) to 1.2 us (pair) of set-up otherwise, all of it on the way where the kernel ahead
    // leaves no room for it: behind another GEMM.
    if (warp == 1) {
        // lane by lane: full[STAGES] empty[STAGES] tmem_full[2] tmem_empty[2] | side data landed, box reusable [boxes]
        constexpr int PIPE = 2 * STAGES + 4, BOXES = (EPI_WARPS / 4) * NBUF;
        static_assert(PIPE + 2 * BOXES <= 32, "one barrier per lane");
        if (lane < PIPE + 2 * BOXES) {
            // stages: one arrive.expect_tx (the leader's, for the whole pair) / one tcgen05.commit; accumulators: one commit /
            // one arrival per epilogue warp of the pair; boxes: one arrive (+ bytes) per fill / the group's four warps
            const uint32_t count = (lane < PIPE - 2) ? 1u : (lane < PIPE) ? EPI_WARPS * CG : (lane < PIPE + BOXES) ? 1u : 4u;
            mbar_init(bar_base + 8 * lane + (lane < PIPE ? 0 : 16), count);
            fence_mbar_init();
        }
    } else if (warp == 2) {
        tmem_alloc<CG>(tmem_ptr_addr, T::TMEM_COLS);
        tmem_relinquish<CG>();
    } else if (warp == 0) {
        if (elect_one()) {
            *abort_flag = 0u;
            prefetch_tensormap(&map_a);
        }
    } else if (warp == 3 + EPI_WARPS) {
        if (elect_one()) {
            prefetch_tensormap(&map_b);
            prefetch_tensormap(&map_bt);
        }
    } else if (warp == 2 + EPI_WARPS) {
        if (elect_one()) {
            prefetch_tensormap(&map_d);
            if constexpr (OP != OP_FC1) prefetch_tensormap(&map_s);
        }
    }
    __syncwarp();
    tc_fence_before();
    if constexpr (CG == 2) cluster_arrive();
    // Every warp calls this once, before it touches a barrier, shared memory or tensor memory.  Everything above it (and what a
    // role does before it calls pdl_wait(), directly in front of its first access to global memory) may run beside the tail of
    // the kernel ahead on the stream.  No two GEMM CTAs share an SM (each takes more than half its shared memory), so the next
    // GEMM's CTAs move in as these leave.
    const auto join_setup = [&]() {
        if constexpr (CG == 2) cluster_wait();
        else __syncthreads();
        tc_fence_after();
    };
    const auto tmem_address = [&]() { return __shfl_sync(0xffffffffu, *tmem_ptr, 0); };

    // ---------------------------------------------------------------- roles
    if (warp == 0 || warp == 3 + EPI_WARPS) {
        // ===== TMA producers: warp 0 brings A, the last warp brings B =====
        // Whole warps with an elected lane, like the MMA role: from a branch that only lane 0 takes, a k-block took 450 - 500
        // cycles to issue, more than the MMAs of a 128-column tile need (FC2 1152 x 4304 at 729 rows: 437 -> 373 cycles per k-block;
        // the whole loop inside one elected branch: 12 % slower than this).
        // Both wait for the stage to be free and then issue their own copies.  Only the A producer arrives on
        // the stage's full barrier (in a CTA pair: only the leader's), announcing the bytes of everything that
        // will land on it; the other copies just count down.  The transaction count may run negative until
        // that arrive lands, and the phase cannot complete before it.  A B copy can never be a whole phase
        // ahead of the arrive it belongs to: the stage is only handed back (empty barrier) after the MMAs have
        // read it, i.e. after the previous phase of the full barrier completed, arrive included.
        const bool is_a = (warp == 0);
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        const bool prof_total = p.prof != nullptr && is_a;
        const uint32_t full_bar_leader = (CG == 2) ? map_to_cta(full_bar0, 0) : full_bar0;
        long long t_wait = 0, t_begin = 0;
        bool waited = false;
        TileWalk walk(p, cluster_id);
        if (!is_a) {
            // The first tile's weights are asked into L2 before the kernel ahead has finished (a hint: were that kernel to write
            // them, L2 would hold what it wrote).  The row-blocks of the first round share the work: each asks for every
            // `sharing`-th k-block of its columns.  A model's weights come from HBM whenever a layer is reached, and a copy that
            // misses L2 takes 0.4 us longer, twice in a row where K is deep (block of 729 rows 45.1 -> 42.8 us, 1 568 rows
            // 42.5 -> 40.7; of 5 003 rows and more no difference).
            const int tm = walk.tm, tn = walk.tn;
            const int sharing = p.step_m + (p.step_n != 0 ? 1 : 0);
            const bool tail = (tn == p.tiles_n - 1) && (p.tail_cols != TN);
            const int nb = tn * TN + static_cast<int>(cta_rank) * (tail ? p.tail_cols / CG : T::B_ROWS);
            const CUtensorMap* const bmap = tail ? &map_bt : &map_b;
            for (int kb = tm; kb < p.k_blocks; kb += sharing) {
                if (elect_one()) {
#pragma unroll
                    for (int a = 0; a < T::KATOMS; a++) tma_prefetch_l2_2d(bmap, kb * T::TILE_K + 128 * a, nb);
                }
                __syncwarp();
            }
        }
        // The k-blocks kb .. end - 1 of a tile: wait for the stage, `issue` from one lane, go on.  What stands in this loop is what
        // paces a small tile (its MMAs need 170 - 290 cycles per k-block), so each producer has an instance of its own,
        // nothing in it is conditional on tracing or tests, and its clock is read only where it waits: 290 (A) and 340 cycles (B)
        // per k-block before that (FC2 1152 x 4304 at 729 rows on 256 x 128 pairs 9.4 -> 9.1 us, on 128 x 64 tiles 9.05 -> 8.15;
        // block of 729 rows 42.74 -> 42.33, 1 568 rows 40.6 -> 39.8).  One instance per producer, not one per tensor map:
        // the larger code cost what the shorter loop saved.
        const auto stream = [&](int kb, int end, auto&& issue) {
#pragma unroll 1
            for (; kb < end; kb++) {
                if (!__all_sync(0xffffffffu, mbar_test_wait(empty_bar0 + 8 * stage, phase ^ 1u) != 0u)) {
                    const long long t0 = clock64();
                    ok = __all_sync(0xffffffffu, wait_bar<SL8_SPIN_CRITICAL>(empty_bar0 + 8 * stage, phase ^ 1u, wc, ST_PRODUCER_EMPTY_WAIT, stage)) != 0;
                    t_wait += clock64() - t0;
                    if (!ok) return;
                }
                if (!waited) {
                    pdl_wait();
                    pdl_release();
                    waited = true;
                    t_begin = clock64();
                }
                if (elect_one()) issue(kb, base + stage * T::STAGE_BYTES, (CG == 2 ? full_bar_leader : full_bar0) + 8 * stage);
                __syncwarp();
                if (++stage == STAGES) { stage = 0; phase ^= 1u; }
            }
        };
        const auto load = [](uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
            if constexpr (CG == 2) tma_load_2d_pair(dst, map, x, y, bar);
            else tma_load_2d(dst, map, x, y, bar);
        };
        join_setup();            // ahead of the loop, like every role: a CTA without a tile joins too
        for (; ok && walk.tile < p.num_tiles; walk.next(p, num_clusters)) {
            wc.tile = walk.tile;
            const int tn = walk.tn;
            const int m0 = walk.tm * (T::TILE_M_CTA * CG) + static_cast<int>(cta_rank) * T::TILE_M_CTA;
            // The last N tile may be narrower: each CTA of a pair then holds tail_cols / CG rows of B,
            // brought by a tensor map whose box is that tall (map_bt), and the MMAs are issued with N = tail_cols.
            const bool tail = (tn == p.tiles_n - 1) && (p.tail_cols != TN);
            const int b_rows = tail ? p.tail_cols / CG : T::B_ROWS;
            const int nb = tn * TN + static_cast<int>(cta_rank) * b_rows;
            // (measurement builds: DBG_SKIP_A / DBG_SKIP_B leave one operand's copies out; the MMAs then read stale shared memory)
            const bool skip_a = SL8_DBG(p.flags, DBG_SKIP_LOAD | DBG_SKIP_A), skip_b = SL8_DBG(p.flags, DBG_SKIP_LOAD | DBG_SKIP_B);
            const uint32_t stage_tx = static_cast<uint32_t>((skip_a ? 0 : T::A_BYTES) + (skip_b ? 0 : T::KATOMS * b_rows * 128));
            if (is_a) {
                stream(0, p.k_blocks, [&](int kb, uint32_t a_dst, uint32_t bar) {
                    if (cta_rank == 0) {
                        if (skip_a && skip_b) mbar_arrive(full_bar0 + 8 * stage);   // measurement aid: MMAs run on whatever shared memory holds
                        else mbar_arrive_expect_tx(full_bar0 + 8 * stage, CG * stage_tx);
                    }
                    if (skip_a) return;
                    if constexpr (T::SPLIT_A) {
#pragma unroll
                        for (int r = 0; r < 96; r += T::A_BOX_ROWS) load(a_dst + r * 128, &map_a, kb * T::TILE_K, m0 + r, bar);
                    } else {
#pragma unroll
                        for (int a = 0; a < T::KATOMS; a++) load(a_dst + a * T::A_ATOM_BYTES, &map_a, kb * T::TILE_K + 128 * a, m0, bar);
                    }
                });
            } else {
                const auto b_loop = [&](int kb0, int end, const CUtensorMap* map) {
                    stream(kb0, end, [&](int kb, uint32_t a_dst, uint32_t bar) {
                        if constexpr (T::SPLIT_A) {
                            if (!skip_a) load(a_dst + 96 * 128, &map_a, kb * T::TILE_K, m0 + 96, bar);
                        }
                        if (skip_b) return;
#pragma unroll
                        for (int a = 0; a < T::KATOMS; a++) load(a_dst + T::A_BYTES + a * T::B_ATOM_BYTES, map, kb * T::TILE_K + 128 * a, nb, bar);
                    });
                };
                // (test aid: with FLAG_TEST_DROP_B k-block 1 of the first tile is never brought)
                int kb0 = 0, end = ((p.flags & FLAG_TEST_DROP_B) && walk.tile == cluster_id) ? 1 : p.k_blocks;
                for (;;) {
                    b_loop(kb0, end, tail ? &map_bt : &map_b);
                    if (!ok || end == p.k_blocks) break;
                    if (++stage == STAGES) { stage = 0; phase ^= 1u; }
                    kb0 = 2;
                    end = p.k_blocks;
                }
            }
        }
        if (prof_total && lane == 0) {
            long long* slot = p.prof + static_cast<size_t>(blockIdx.x) * PROF_SLOTS;
            slot[PROF_PRODUCER_WAIT] = t_wait;
            slot[PROF_PRODUCER_TOTAL] = clock64() - t_begin;
        }
        __syncwarp();
    } else if (warp == 1) {
        // ===== MMA issuer (leader CTA only) =====
        // The whole warp walks the loop and one elected lane issues: a tcgen05.mma takes its descriptors from uniform
        // registers, and in a branch that only one lane takes each of them is moved there instruction by instruction, which
        // cost ~110 cycles per MMA -- hidden behind the 128 cycles of a 256-column tile, but twice what a 128-column tile
        // needs (1152-wide FC2 at 729 rows on 128 x 128 tiles 14.5 -> 11.6 us; at 46 656 rows on 256 x 256 tiles 193 -> 186).
        // What else the loop executes per k-block counts too: the poll of the NEXT stage's barrier is issued before this
        // stage's MMAs and read after them
        // (the blocking wait runs only if that look-ahead failed), and k-blocks are taken several per loop iteration.
        if (cta_rank == 0) {
            const uint32_t idesc_full = make_idesc_e4m3_f32(T::TILE_M_CTA * CG, TN);
            const uint32_t idesc_tail = make_idesc_e4m3_f32(T::TILE_M_CTA * CG, p.tail_cols);   // the last, narrower N tile
            uint32_t idesc = idesc_full;
            // Descriptors differ between stages, atoms and K steps only in the 14-bit start-address
            // field: +2 there = 32 bytes = one K = 32 step inside the 128-byte row.
            const auto all_ok = [](bool lane_ok) { return __all_sync(0xffffffffu, lane_ok) != 0; };
            const uint64_t adesc0 = make_kmajor_sw128_desc(base);
            const uint64_t bdesc0 = make_kmajor_sw128_desc(base + T::A_BYTES);
            constexpr uint32_t STAGE_DESC = T::STAGE_BYTES >> 4;
            int stage = 0;
            uint32_t phase = 0;
            int acc = 0;
            uint32_t acc_phase = 0;
            bool ok = true;
            const bool prof_any = p.prof != nullptr;
            const bool prof = prof_any && !(p.flags & (FLAG_COARSE_TRACE | DBG_COARSE_TRACE));
            long long t_full = 0, t_tmem = 0, n_tiles = 0, t_mma = 0, t_commit = 0;
            TileWalk walk(p, cluster_id);
            join_setup();
            const uint32_t tmem_base = tmem_address();
            pdl_wait();              // nothing to wait for before that: the bounded waits start with the kernel's own work
            pdl_release();
            const long long t_begin = clock64();
            uint32_t ready = 0;      // look-ahead: the barrier of `stage` was already seen complete

            // All MMAs of one full k-block held in `st`; `fresh` = this k-block starts a tile (overwrite D).
            // (only inside `if (elect_one())`, which picks the same lane every time: a commit covers the MMAs its own thread issued)
            auto issue_full = [&](uint32_t d_tmem, int st, bool fresh) {
                const uint64_t adesc = adesc0 + static_cast<uint32_t>(st) * STAGE_DESC;
                const uint64_t bdesc = bdesc0 + static_cast<uint32_t>(st) * STAGE_DESC;
#pragma unroll
                for (int j = 0; j < 4 * T::KATOMS; j++) {
                    const uint32_t o = (j >> 2) * (T::A_ATOM_BYTES >> 4) + 2 * (j & 3);
                    const uint32_t ob = (j >> 2) * (T::B_ATOM_BYTES >> 4) + 2 * (j & 3);
                    mma_f8<CG>(d_tmem, adesc + o, bdesc + ob, idesc, (j == 0 && fresh) ? 0u : 1u);
                }
            };
            auto release_stage = [&](int st) {
                if constexpr (CG == 2) mma_commit_pair(empty_bar0 + 8 * st, 0x3);
                else mma_commit(empty_bar0 + 8 * st);
            };

            for (; ok && walk.tile < p.num_tiles; walk.next(p, num_clusters)) {
                wc.tile = walk.tile;
                long long t0 = prof_any ? clock64() : 0;     // once per tile: timed in the coarse mode too
                ok = all_ok(wait_bar<SL8_SPIN_CRITICAL>(tempty_bar0 + 8 * acc, acc_phase ^ 1u, wc, ST_MMA_TMEM_EMPTY_WAIT, acc));
                if (prof_any) t_tmem += clock64() - t0;
                n_tiles++;
                if (!ok) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * T::ACC_STRIDE;
                idesc = (walk.tn == p.tiles_n - 1) ? idesc_tail : idesc_full;
                int kb = 0;
                const int k_full = p.k_blocks - 1;           // k-blocks that hold all their MMAs
                if (!prof && !SL8_DBG(p.flags, DBG_SKIP_MMA)) {
                    // One k-block: wait (only if the look-ahead failed), look ahead, MMAs, release the stage.
                    // n < 4 * KATOMS only in the K tail.
                    auto step = [&](bool fresh, int n) -> bool {
                        if (!ready) {      // the look-ahead saw the stage still filling: counted, then waited for
                            t_full++;
                            if (!all_ok(wait_bar<SL8_SPIN_CRITICAL>(full_bar0 + 8 * stage, phase, wc, ST_MMA_FULL_WAIT, stage))) return false;
                        }
                        const int s1 = (stage + 1 == STAGES) ? 0 : stage + 1;
                        const uint32_t ph1 = (s1 == 0) ? (phase ^ 1u) : phase;
                        const uint32_t r1 = mbar_test_wait(full_bar0 + 8 * s1, ph1);
                        tc_fence_after();
                        if (elect_one()) {
                          if (n == 4 * T::KATOMS) {
                            issue_full(d_tmem, stage, fresh);
                          } else {
                            const uint64_t adesc = adesc0 + static_cast<uint32_t>(stage) * STAGE_DESC;
                            const uint64_t bdesc = bdesc0 + static_cast<uint32_t>(stage) * STAGE_DESC;
#pragma unroll
                            for (int j = 0; j < 4 * T::KATOMS - 1; j++) {
                                const uint32_t o = (j >> 2) * (T::A_ATOM_BYTES >> 4) + 2 * (j & 3);
                                const uint32_t ob = (j >> 2) * (T::B_ATOM_BYTES >> 4) + 2 * (j & 3);
                                if (j < n) mma_f8<CG>(d_tmem, adesc + o, bdesc + ob, idesc, (j == 0 && fresh) ? 0u : 1u);
                            }
                          }
                          release_stage(stage);
                        }
                        __syncwarp();
                        stage = s1;
                        phase = ph1;
                        ready = all_ok(r1 != 0u) ? 1u : 0u;
                        return true;
                    };
                    for (; ok && kb + 2 <= k_full; kb += 2) {      // two k-blocks per loop iteration
                        ok = step(kb == 0, 4 * T::KATOMS);
                        if (ok) ok = step(false, 4 * T::KATOMS);
                    }
                    if (ok && kb < k_full) {
                        ok = step(kb == 0, 4 * T::KATOMS);
                        kb++;
                    }
                    if (ok) {
                        ok = step(kb == 0, p.last_kblock_mmas);
                        kb++;
                    }
                    if (!ok) break;
                }
                for (; kb < p.k_blocks; kb++) {
                    if (prof) t0 = clock64();
                    if (!ready) ok = all_ok(wait_bar<SL8_SPIN_CRITICAL>(full_bar0 + 8 * stage, phase, wc, ST_MMA_FULL_WAIT, stage));
                    if (prof) t_full += clock64() - t0;
                    if (!ok) break;
                    const int s1 = (stage + 1 == STAGES) ? 0 : stage + 1;
                    const uint32_t ph1 = (s1 == 0) ? (phase ^ 1u) : phase;
                    ready = all_ok(mbar_test_wait(full_bar0 + 8 * s1, ph1) != 0u) ? 1u : 0u;
                    tc_fence_after();
                    long long t1 = prof ? clock64() : 0;
                    if (SL8_DBG(p.flags, DBG_SKIP_MMA)) {
                        // measurement aid: stages are released at once, the loads run at their own pace
                    } else if (elect_one()) {
                      if (kb < k_full) {
                        issue_full(d_tmem, stage, kb == 0);
                      } else {
                        const uint64_t adesc = adesc0 + static_cast<uint32_t>(stage) * STAGE_DESC;
                        const uint64_t bdesc = bdesc0 + static_cast<uint32_t>(stage) * STAGE_DESC;
                        for (int j = 0; j < p.last_kblock_mmas; j++) {
                            const uint32_t o = (j >> 2) * (T::A_ATOM_BYTES >> 4) + 2 * (j & 3);
                            const uint32_t ob = (j >> 2) * (T::B_ATOM_BYTES >> 4) + 2 * (j & 3);
                            mma_f8<CG>(d_tmem, adesc + o, bdesc + ob, idesc, (kb | j) != 0 ? 1u : 0u);
                        }
                      }
                    }
                    __syncwarp();
                    if (prof) { const long long t2 = clock64(); t_mma += t2 - t1; t1 = t2; }
                    if (elect_one()) release_stage(stage);
                    __syncwarp();
                    if (prof) t_commit += clock64() - t1;
                    stage = s1;
                    phase = ph1;
                }
                if (!ok) break;
                if (elect_one()) {
                    if constexpr (CG == 2) mma_commit_pair(tfull_bar0 + 8 * acc, 0x3);
                    else mma_commit(tfull_bar0 + 8 * acc);
                }
                __syncwarp();
                if (p.flags & FLAG_SINGLE_ACC) acc_phase ^= 1u;
                else { acc ^= 1; if (acc == 0) acc_phase ^= 1u; }
            }
            if (prof_any && lane == 0) {
                long long* slot = p.prof + static_cast<size_t>(blockIdx.x) * PROF_SLOTS;
                slot[PROF_MMA_WAIT_FULL] = t_full;
                slot[PROF_MMA_WAIT_TMEM] = t_tmem;
                slot[PROF_MMA_TOTAL] = clock64() - t_begin;
                slot[PROF_TILES] = n_tiles;
                slot[PROF_MMA_ISSUE] = t_mma;
                slot[PROF_MMA_COMMIT] = t_commit;
            }
        } else {
            join_setup();
        }
        __syncwarp();
    } else if (warp < 2 + EPI_WARPS) {
        // ===== epilogue =====
        const int ew = warp - 2;
        const int quad = warp & 3;                 // TMEM lane quadrant this warp may read
        const int col_part = ew >> 2;              // 0, or 0/1 with eight epilogue warps
        const int col_begin = col_part * T::COLS_PER_WARP;
        constexpr int RPT = T::REGIONS_PER_TILE;
        constexpr bool HAS_BIAS = (OP != OP_PE);
        constexpr bool HAS_SIDE = (OP != OP_FC1);
        static_assert(!HAS_SIDE || NBUF >= 2, "side data needs a buffer to land in while another is stored");

        EpiCtx e;
        e.flags = p.flags;
        e.swz = (T::REGION_ROW_BYTES == 128) ? (lane & 7) : ((lane >> 1) & 3);
        e.row_off = lane * T::REGION_ROW_BYTES;
        // Staging is organised per column group (the four quadrant warps that cover the same columns):
        // NBUF boxes of 128 rows x 128 bytes, of which this warp owns rows 32 * quad .. 32 * quad + 31.
        const uint32_t my_staging = staging_base + col_part * NBUF * 4 * T::REGION_BYTES + quad * T::REGION_BYTES;
        const long long warp_row_in_tile = static_cast<long long>(cta_rank) * T::TILE_M_CTA + quad * 32;

        const uint32_t my_side_bar = side_bar0 + 8 * col_part * NBUF;      // side data of the group's box b landed
        const uint32_t my_side_free = side_free0 + 8 * col_part * NBUF;    // the group's box b may be refilled

        constexpr int NB = T::COLS_PER_WARP / 32;  // bias values each lane stages per tile
        float* const bias_w = reinterpret_cast<float*>(base_ptr + (bias_base - base)) + ew * T::COLS_PER_WARP;
        constexpr bool BSM = T::BIAS_IN_SMEM;
        float bnext[NB], bcur[NB];
#pragma unroll
        for (int i = 0; i < NB; i++) bcur[i] = bnext[i] = 0.0f;
        bool ok = true;
        uint32_t seq = 0;                          // regions processed so far by this warp
        int acc = 0;
        uint32_t acc_phase = 0;
        const bool prof_total = p.prof != nullptr && ew == 0;
        const bool prof = prof_total && !(p.flags & (FLAG_COARSE_TRACE | DBG_COARSE_TRACE));   // inner timers cost ~35 cycles each
        long long t_acc = 0, t_store = 0, t_ld = 0, t_math = 0, t_issue = 0, t_refill = 0;
        TileWalk walk(p, cluster_id);
        join_setup();
        const uint32_t tmem_base = tmem_address();
        pdl_wait();
        pdl_release();
        const long long t_begin = clock64();
        e.scale = (p.scale_a ? ld_f32(p.scale_a) : 1.0f) * (p.scale_b ? ld_f32(p.scale_b) : 1.0f);
        e.inv_out = __frcp_rn(p.out_scale ? ld_f32(p.out_scale) : 1.0f);   // IEEE 1/x, as the CPU oracle computes it
        if constexpr (HAS_BIAS) {
            if (walk.tile < p.num_tiles) {
                load_bias<NB>(bnext, p.bias, p.flags, walk.tn * TN + col_begin, lane, p.N);
#pragma unroll
                for (int i = 0; i < NB; i++) {
                    if constexpr (BSM) bias_w[lane + 32 * i] = bnext[i];
                    else bcur[i] = bnext[i];
                }
                __syncwarp();
            }
        }
        while (ok && walk.tile < p.num_tiles) {
            wc.tile = walk.tile;
            const int tn = walk.tn;
            const long long m_warp = static_cast<long long>(walk.tm) * (T::TILE_M_CTA * CG) + warp_row_in_tile;
            const int n0 = tn * TN;

            // The next tile's bias travels to registers while this tile is processed.
            walk.next(p, num_clusters);
            const bool has_next = walk.tile < p.num_tiles;
            if constexpr (HAS_BIAS) {
                if (has_next) load_bias<NB>(bnext, p.bias, p.flags, walk.tn * TN + col_begin, lane, p.N);
            }

            long long t0 = prof_total ? clock64() : 0;       // once per tile: timed in the coarse mode too
            ok = wait_bar(tfull_bar0 + 8 * acc, acc_phase, wc, ST_EPI_TMEM_FULL_WAIT, acc);
            ok = __all_sync(0xffffffffu, ok);
            if (prof_total) t_acc += clock64() - t0;
            if (!ok) break;
            tc_fence_after();

            const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * T::ACC_STRIDE;
            const bool warp_rows_ok = m_warp < p.M;      // warp-uniform: any row of this warp inside M
            bool released = false;

#pragma unroll 1
            for (int r = 0; r < RPT; r++, seq++) {
                const int c0 = col_begin + r * T::REGION_COLS;       // first column of the region inside the tile
                const int col0 = n0 + c0;
                const uint32_t region = my_staging + (seq % NBUF) * 4 * T::REGION_BYTES;
                if (prof) t0 = clock64();
                if constexpr (HAS_SIDE) {
                    // this region's side values have landed
                    const uint32_t sbar = my_side_bar + 8 * (seq % NBUF);
                    const uint32_t spar = (seq / NBUF) & 1u;
                    ok = wait_bar(sbar, spar, wc, ST_EPI_SIDE_WAIT, seq % NBUF);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                } else {
                    if (elect_one()) tma_store_wait_read<NBUF - 1>();   // the buffer is no longer read by an older store
                    __syncwarp();
                }
                if (prof) t_store += clock64() - t0;

                const bool live = col0 < p.N && !SL8_DBG(p.flags, DBG_SKIP_EPILOGUE);   // warp-uniform
                if (live) {
#pragma unroll
                    for (int ch = 0; ch < T::CHUNKS_PER_REGION; ch++) {
                        const int c = c0 + 32 * ch;
                        if (n0 + c < p.N) {
                            float v[32];
                            if (SL8_DBG(p.flags, DBG_SKIP_TMEM_LD)) {   // measurement aid: the epilogue works on constants
#pragma unroll
                                for (int i = 0; i < 32; i++) v[i] = 1.0f;
                            } else {
                                tmem_ld_32x32(t_row + c, v);
                            }
                            if (prof) t0 = clock64();
                            if (!SL8_DBG(p.flags, DBG_SKIP_TMEM_LD)) tmem_ld_wait();
                            if (prof) t_ld += clock64() - t0;
                            if (r == RPT - 1 && ch == T::CHUNKS_PER_REGION - 1) {
                                // Last read of this accumulator: hand the TMEM buffer back before the math.
                                tc_fence_before();
                                __syncwarp();
                                if (elect_one()) {
                                    if constexpr (CG == 2) mbar_arrive_cluster(map_to_cta(tempty_bar0 + 8 * acc, 0));
                                    else mbar_arrive(tempty_bar0 + 8 * acc);
                                }
                                released = true;
                            }
                            if (prof) t0 = clock64();
                            const int piece0 = ch * 2 * T::OUT_BYTES;            // 32 columns = 2 (e4m3) or 4 (bf16) pieces
                            const float* bias32 = bias_w + (c - col_begin);
                            float breg = bcur[0];                       // this chunk's bias, one column per lane
                            if constexpr (!BSM) {
#pragma unroll
                                for (int i = 1; i < NB; i++)
                                    if (i == r * T::CHUNKS_PER_REGION + ch) breg = bcur[i];
                            }
                            if (!SL8_DBG(p.flags, DBG_SKIP_MATH)) {
                                if constexpr (OP == OP_FC1 && EPI_WARPS <= 8) {
                                    // (columns past N are computed on whatever the accumulator holds and clipped by the TMA store)
                                    epilogue_32_fc1<OUT, BSM>(v, e, bias32, breg, region, piece0);
                                } else {
                                    epilogue_16<OP, OUT, 0, BSM>(v, e, bias32, breg, region, piece0);
                                    if (n0 + c + 16 < p.N) epilogue_16<OP, OUT, 1, BSM>(v, e, bias32 + 16, breg, region, piece0 + T::OUT_BYTES);
                                }
                            }
                            if (prof) t_math += clock64() - t0;
                        }
                    }
                    if (prof) t0 = clock64();
                    if (!SL8_DBG(p.flags, DBG_SKIP_STORE)) {
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (warp_rows_ok && elect_one()) tma_store_2d(&map_d, region, col0, static_cast<int>(m_warp));
                    }
                    if (prof) t_issue += clock64() - t0;
                }
                if (elect_one()) tma_store_commit();       // one bulk group per region, possibly empty
                if constexpr (HAS_SIDE) {
                    // Once the PREVIOUS region's store has read its buffer, hand that buffer back to the
                    // side-data loader (this region's store may still be reading its own).
                    if (prof) t0 = clock64();
                    if (elect_one()) {
                        tma_store_wait_read<1>();
                        if (seq > 0) mbar_arrive(my_side_free + 8 * ((seq - 1) % NBUF));
                    }
                    if (prof) t_refill += clock64() - t0;
                }
            }

            if (!ok) break;
            if (!released) {                             // tile whose last region lies past N
                tc_fence_before();
                __syncwarp();
                if (elect_one()) {
                    if constexpr (CG == 2) mbar_arrive_cluster(map_to_cta(tempty_bar0 + 8 * acc, 0));
                    else mbar_arrive(tempty_bar0 + 8 * acc);
                }
            }
            if (p.flags & FLAG_SINGLE_ACC) acc_phase ^= 1u;
            else { acc ^= 1; if (acc == 0) acc_phase ^= 1u; }

            if constexpr (HAS_BIAS) {
                if (has_next) {
                    __syncwarp();                        // every lane has finished reading this tile's bias
#pragma unroll
                    for (int i = 0; i < NB; i++) {
                        if constexpr (BSM) bias_w[lane + 32 * i] = bnext[i];
                        else bcur[i] = bnext[i];
                    }
                    __syncwarp();
                }
            }
        }
        // The staging buffers must have been read before this CTA's shared memory is given back; the writes themselves
        // are complete for whoever is ordered after the kernel, as every write of a kernel is.
        if (elect_one()) tma_store_wait_read<0>();
        __syncwarp();
        if (prof_total && lane == 0) {
            long long* slot = p.prof + static_cast<size_t>(blockIdx.x) * PROF_SLOTS;
            slot[PROF_EPI_WAIT_ACC] = t_acc;
            slot[PROF_EPI_WAIT_STORE] = t_store;
            slot[PROF_EPI_WAIT_LD] = t_ld;
            slot[PROF_EPI_MATH] = t_math;
            slot[PROF_EPI_STORE_ISSUE] = t_issue;
            slot[PROF_EPI_REFILL] = t_refill;
            slot[PROF_EPI_TOTAL] = clock64() - t_begin;
        }
    } else {
        // ===== side-data loader =====
        // Region number s of a column group (RPT per tile, tiles in the order this cluster visits them)
        // -> 128 rows x 128 bytes of the table / residual (the rows of this CTA's tile, 64 bf16 columns)
        // into the group's staging box s % NBUF, in the swizzled layout the TMA stores of the result
        // expect; completion on the box's "landed" barrier.  One TMA load.  A positional table that holds
        // at least period + 127 rows (rows past the period repeating it) never needs anything else; with
        // an unpadded table the boxes that wrap around its end are copied row by row by the whole warp.
        if constexpr (OP != OP_FC1) {
            constexpr int RPT = T::REGIONS_PER_TILE;
            constexpr int GROUPS = EPI_WARPS / 4;
            constexpr uint32_t BOX_BYTES = 4 * T::REGION_BYTES;
            const bool skip_side = SL8_DBG(p.flags, DBG_SKIP_SIDE);
            bool ok = true, waited = false;
            TileWalk walk(p, cluster_id);
            join_setup();
            for (uint32_t s = 0; ok && walk.tile < p.num_tiles; s++) {
                const int tn = walk.tn;
                const long long m_cta = static_cast<long long>(walk.tm) * (T::TILE_M_CTA * CG) + cta_rank * T::TILE_M_CTA;
                wc.tile = walk.tile;
#pragma unroll 1
                for (int g = 0; g < GROUPS; g++) {
                    const uint32_t bsel = s % NBUF;
                    const uint32_t landed = side_bar0 + 8 * (g * NBUF + bsel);
                    const uint32_t freed = side_free0 + 8 * (g * NBUF + bsel);
                    const uint32_t buf = staging_base + (g * NBUF + bsel) * BOX_BYTES;
                    // the box's previous occupant (region s - NBUF) has been stored by all four warps
                    ok = __all_sync(0xffffffffu, wait_bar(freed, ((s / NBUF) & 1u) ^ 1u, wc, ST_SIDE_LOADER_WAIT, g)) != 0;
                    if (!ok) break;
                    const int col0 = tn * TN + g * T::COLS_PER_WARP + static_cast<int>(s % RPT) * T::REGION_COLS;
                    if (col0 >= p.N || skip_side) {
                        if (elect_one()) mbar_arrive(landed);
                        __syncwarp();
                        continue;
                    }
                    int y = static_cast<int>(m_cta);
                    bool wraps = false;
                    if constexpr (OP == OP_PE) {
                        y = static_cast<int>((static_cast<uint32_t>(m_cta) + static_cast<uint32_t>(p.row_phase)) % static_cast<uint32_t>(p.period));
                        wraps = y + T::TILE_M_CTA > p.table_rows;   // only a table without periodic padding wraps
                    }
                    if (!waited) {
                        pdl_wait();
                        pdl_release();
                        waited = true;
                    }
                    if (!wraps) {
                        if (elect_one()) {
                            mbar_arrive_expect_tx(landed, BOX_BYTES);
                            tma_load_2d(buf, &map_s, col0, y, landed);
                        }
                        __syncwarp();
                    } else {
                        const int piece = lane & 7;                 // 16-byte piece (8 bf16 columns) of the 128-byte row
                        const int col = col0 + piece * 8;
                        int t = y + (lane >> 3);
                        while (t >= p.period) t -= p.period;
                        // Eight rows' loads are asked for before the first of them is stored: a box is 32 trips to L2 otherwise
                        // (neither moves past the other in the compiler).  196 rows x 768 with a 196-row table 9.2 -> 8.2 us,
                        // 200 704 rows 335 -> 279; 46 656 x 1 152 with 729 rows 81.5 -> 71.8.
#pragma unroll 1
                        for (int i = 0; i < 32; i += 8) {
                            uint4 val[8];
#pragma unroll
                            for (int j = 0; j < 8; j++) {
                                val[j] = make_uint4(0, 0, 0, 0);
                                if (col < p.N) val[j] = ld_16(p.side + static_cast<long long>(t) * p.ld_side + col);
                                t += 4;
                                while (t >= p.period) t -= p.period;
                            }
#pragma unroll
                            for (int j = 0; j < 8; j++) {
                                const int r = (lane >> 3) + 4 * (i + j);      // staging row 0..127
                                sts128(buf + r * 128 + ((piece ^ (r & 7)) << 4), val[j].x, val[j].y, val[j].z, val[j].w);
                            }
                        }
                        __syncwarp();
                        if (elect_one()) mbar_arrive(landed);
                        __syncwarp();
                    }
                }
                if (s % RPT == RPT - 1) walk.next(p, num_clusters);
            }
        } else {
            join_setup();
        }
        __syncwarp();
    }

    // ---------------------------------------------------------------- exit
    tc_fence_before();
    if constexpr (CG == 2) {
        cluster_arrive();
        cluster_wait();
    } else {
        __syncthreads();
    }
    if (*abort_flag) {
        // Something gave up: let copies and MMAs already in flight land before the shared and
        // tensor memory they target is released.
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) {
        }
        __syncthreads();
    }
    if (warp == 2) {      // the warp that allocated
        tc_fence_after();
        tmem_dealloc<CG>(tmem_address(), T::TMEM_COLS);
    }
}

}  // namespace sl8
