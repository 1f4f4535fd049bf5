// sl8_prep.cu -- the producer-side steps of the C ABI (include/siglip_fp8.h): what feeds the GEMMs' A operand.
#include <cuda_bf16.h>

#include "sl8_internal.h"

namespace {

inline int fail(sl8_handle_t h, int code, const std::string& msg) { return sl8_fail(h, code, msg); }
inline int fail_cuda(sl8_handle_t h, cudaError_t e, const char* what) { return sl8_fail_cuda(h, e, what); }
inline bool aligned16(const void* p) { return sl8_aligned16(p); }
typedef Sl8DeviceGuard DeviceGuard;

}  // namespace

// =========================================================================== producer-side steps
// What feeds A: pixels -> patch rows (the Conv2d of the patch embedding written as a GEMM operand,
// docs/architecture.md:11-12 of the reference, which stops at the GEMM) with the per-tensor quantisation to
// e4m3 fused in, and the dynamic quantisation of a bf16 / fp32 activation (abs-max -> scale -> e4m3 codes)
// for a caller that has no static scale between FC1 and FC2.  Byte work bounded by HBM.

namespace {

__device__ __forceinline__ float prep_load(const float* p) { return sl8::ld_f32(p); }
__device__ __forceinline__ float prep_load(const __nv_bfloat16* p) { return sl8::ld_bf16(p); }
__device__ __forceinline__ uint8_t prep_e4m3(float v) { return static_cast<uint8_t>(sl8::pack_e4m3x2(v, 0.0f) & 0xFFu); }

// n / d for the small indices below, by one multiplication: exact while n * d < 2^32 (m = ceil(2^32 / d); d = 1: m = 0).
struct FastDiv {
    uint32_t m, d;
};
inline FastDiv fast_div(int d) { return FastDiv{d > 1 ? static_cast<uint32_t>((0x100000000ull + d - 1) / d) : 0u, static_cast<uint32_t>(d)}; }
__device__ __forceinline__ uint32_t operator/(uint32_t n, const FastDiv& f) { return f.m ? __umulhi(n, f.m) : n; }

__device__ __forceinline__ uint4 ld_once_16(const void* p) {         // 16 bytes that nothing reads again
    uint4 q;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w) : "l"(p) : "memory");
    return q;
}

// How the codes of one 16-byte chunk of pixels go to shared memory: byte by byte (odd patch, or rows that start on odd
// pixels), in pairs (even patch: a pair never straddles two patches), or whole (a patch is a whole number of chunks).
enum : int { UNFOLD_BYTES = 0, UNFOLD_PAIRS = 1, UNFOLD_CHUNKS = 2 };
constexpr int kUnfoldThreads = 256;     // at most: a whole number of image rows, chunk by chunk

__device__ __forceinline__ void sts_u8(uint32_t at, uint32_t v) { asm volatile("st.shared.u8 [%0], %1;" ::"r"(at), "r"(v) : "memory"); }
__device__ __forceinline__ void sts_u16(uint32_t at, uint16_t v) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(at), "h"(v) : "memory"); }
__device__ __forceinline__ void sts_u32(uint32_t at, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory"); }
__device__ __forceinline__ void sts_u64(uint32_t at, uint32_t lo, uint32_t hi) { asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at), "r"(lo), "r"(hi) : "memory"); }

// Offsets, inside the group's rows of A (pitch bytes apart), of the codes of the chunk that starts `x` pixels after the
// group's first one; `outside` for what lies outside the group.
template <int VP, int NO>
__device__ __forceinline__ void unfold_offsets(int (&to)[NO], int x, int len, int P, const FastDiv& by_patch, int pitch, int outside) {
#pragma unroll
    for (int j = 0; j < NO; j++) {
        const int xx = x + j * (VP / NO);
        const uint32_t gx = static_cast<uint32_t>(max(xx, 0)) / by_patch;
        to[j] = (xx < 0 || xx >= len) ? outside : static_cast<int>(gx) * pitch + (xx - static_cast<int>(gx) * P);
    }
}

// Quantises the 16 bytes of pixels in q and puts the codes where `to` says, relative to shared address dst.  SOME: a
// negative offset is dropped.
template <typename PT, int MODE, bool SOME, int NO>
__device__ __forceinline__ void unfold_put(const uint4& q, uint64_t inv2, uint32_t dst, const int (&to)[NO]) {
    constexpr int VP = 16 / sizeof(PT);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
    uint16_t code[VP / 2];                                // two codes each
#pragma unroll
    for (int j = 0; j < VP / 2; j++) {
        float lo, hi;
        if constexpr (sizeof(PT) == 4) { lo = __uint_as_float(w[2 * j]); hi = __uint_as_float(w[2 * j + 1]); }
        else { lo = __uint_as_float(w[j] << 16); hi = __uint_as_float(w[j] & 0xFFFF0000u); }
        sl8::unpack_f32x2(sl8::mul_f32x2(sl8::pack_f32x2(lo, hi), inv2), lo, hi);
        code[j] = sl8::pack_e4m3x2(lo, hi);
    }
    if constexpr (MODE == UNFOLD_CHUNKS) {
        const uint32_t lo = code[0] | (static_cast<uint32_t>(code[1]) << 16);
        if constexpr (VP == 4) sts_u32(dst + to[0], lo);
        else sts_u64(dst + to[0], lo, code[2] | (static_cast<uint32_t>(code[3]) << 16));
    } else {
#pragma unroll
        for (int j = 0; j < NO; j++) {
            if (SOME && to[j] < 0) continue;
            if constexpr (MODE == UNFOLD_PAIRS) sts_u16(dst + to[j], code[j]);
            else sts_u8(dst + to[j], static_cast<uint32_t>(code[j / 2]) >> (8 * (j & 1)));
        }
    }
}

// One block per (image, patch row, group of G patches).  The C * P image rows of the group are read in 16-byte chunks
// (aligned down from the first pixel; what lies outside the group is dropped), quantised, placed in shared memory at
// the position they have in the group's rows of A (column c * P * P + py * P + px, the flattening order of a Conv2d
// weight [N, C, P, P]) and those rows are then written whole, pad included.
// Bound by HBM where three things are seen to.  Bytes in flight: three, four or six 16-byte loads per thread (it was one load of
// two pixels), see unfold_batch.  Banks: rows of A are multiples of 128 bytes, so unpadded the same pixel of every patch falls into one bank; 16
// bytes of pad per row spread eight patches over all of them.  Instructions: a thread keeps its chunk position and walks
// down the image rows, so that where its codes go is worked out once (ALIGNED: every image row starts on a 16-byte
// boundary, and an image is less than 4 GiB) and a chunk costs its load, conversion, stores and a few additions; dividing
// for every pair of pixels took 24 instructions per pixel, and the kernel ran at a third of the bandwidth, issue-bound.
// 256 images of 384 x 384, patch 14: bf16 130 -> 65.5 us (5.3 TB/s), fp32 123 -> 89.5 us (6.2 TB/s); 32 images of 224 x 224,
// patch 16, fp32: 11.5 -> 4.3 us; one such image 7.1 -> 2.0 us.
template <typename PT, int MODE, bool ALIGNED, int BATCH>
__global__ void __launch_bounds__(kUnfoldThreads, 4)
patchify_quantize_kernel(const PT* pixels, long long total, int H, int W, int P, int C, int gh, int gw, int G, int groups,
                         int rows_per_step, FastDiv by_chunks, FastDiv by_patch, FastDiv by_vecs, const float* scale,
                         uint8_t* A, long long lda, int row_bytes) {
    extern __shared__ __align__(16) uint8_t prep_tile[];
    constexpr int VP = 16 / sizeof(PT);                   // pixels per chunk
    constexpr int NO = MODE == UNFOLD_CHUNKS ? 1 : MODE == UNFOLD_PAIRS ? VP / 2 : VP;    // stores per chunk
    const int strip = blockIdx.x / groups, g = blockIdx.x - strip * groups;
    const int img = strip / gh, gy = strip - img * gh;
    const int g0 = g * G, gn = min(G, gw - g0);           // patches of this block
    const int xs = g0 * P, len = gn * P;                  // ... and their pixels in an image row
    const int pitch = row_bytes + 16;
    const int CP = C * P;
    sl8::pdl_wait();
    sl8::pdl_release();
    const float inv = __frcp_rn(scale ? sl8::ld_f32(scale) : 1.0f);
    const uint64_t inv2 = sl8::pack_f32x2(inv, inv);
    const uint32_t tile = sl8::smem_u32(prep_tile);

    const int row0 = static_cast<int>(static_cast<uint32_t>(threadIdx.x) / by_chunks);    // first image row and chunk of this thread
    const int v = static_cast<int>(threadIdx.x) - row0 * static_cast<int>(by_chunks.d);
    const long long first0 = (static_cast<long long>(img) * C * H + gy * P) * W + xs;    // pixel (c = 0, py = 0) of the group
    int to[NO];
    if constexpr (ALIGNED) {
        if (row0 < rows_per_step && v * VP < len) {
            // (what the last chunk of a row has outside the group goes to a spare row behind the tile: a test for it, taken
            // by one lane of most warps, would run the conversion twice)
            unfold_offsets<VP, NO>(to, v * VP, len, P, by_patch, pitch, G * pitch);
            const char* const base = reinterpret_cast<const char*>(pixels + first0);
            const uint32_t row_step = static_cast<uint32_t>(rows_per_step) * W * sizeof(PT);
            const uint32_t plane_step = static_cast<uint32_t>(H - P) * W * sizeof(PT);   // from the last row of a channel's strip to the next one's first
            const uint32_t dst_step = static_cast<uint32_t>(rows_per_step) * P;
            int py = row0, left = CP - row0;              // row inside the channel; rows still to come, this one included
            uint32_t src = static_cast<uint32_t>(row0) * W * sizeof(PT) + 16u * v, dst = tile + row0 * P;
            while (py >= P) { py -= P; src += plane_step; }
            while (left > 0) {
                uint4 q[BATCH];
#pragma unroll
                for (int b = 0; b < BATCH; b++) {
                    if (left > b * rows_per_step) q[b] = ld_once_16(base + src);
                    src += row_step;
                    py += rows_per_step;
                    while (py >= P) { py -= P; src += plane_step; }
                }
#pragma unroll
                for (int b = 0; b < BATCH; b++) {
                    if (left > b * rows_per_step) unfold_put<PT, MODE, false, NO>(q[b], inv2, dst, to);
                    dst += dst_step;
                }
                left -= BATCH * rows_per_step;
            }
        }
    } else if (row0 < rows_per_step) {
        for (int cp0 = row0; cp0 < CP; cp0 += rows_per_step * BATCH) {
            uint4 q[BATCH];
            int x[BATCH];                          // first pixel of the chunk relative to the group
#pragma unroll
            for (int b = 0; b < BATCH; b++) {
                const int cp = cp0 + b * rows_per_step;
                x[b] = len;
                if (cp >= CP) continue;
                const int c = static_cast<int>(static_cast<uint32_t>(cp) / by_patch);
                const long long first = first0 + static_cast<long long>(cp + static_cast<long long>(c) * (H - P)) * W;
                x[b] = v * VP - static_cast<int>(first & (VP - 1));       // the row starts that many pixels past a chunk boundary
                if (x[b] >= len) continue;
                const long long at = first + x[b];
                if (at + VP <= total) {
                    q[b] = ld_once_16(pixels + at);
                } else {                                  // the last chunk of the tensor, when it is not a whole one
                    PT tail[VP] = {};
                    for (int j = 0; at + j < total; j++) tail[j] = pixels[at + j];
                    memcpy(&q[b], tail, 16);
                }
            }
#pragma unroll
            for (int b = 0; b < BATCH; b++) {
                if (x[b] >= len) continue;
                unfold_offsets<VP, NO>(to, x[b], len, P, by_patch, pitch, -1);
                unfold_put<PT, MODE, true, NO>(q[b], inv2, tile + (cp0 + b * rows_per_step) * P, to);
            }
        }
    }
    __syncthreads();
    // 16-byte vectors of the rows of A: a thread keeps its place in the row and walks down the rows.
    const int vecs = static_cast<int>(by_vecs.d);
    const int r0 = static_cast<int>(static_cast<uint32_t>(threadIdx.x) / by_vecs);
    const int steps = static_cast<int>(max(blockDim.x / by_vecs, 1u));
    if (r0 >= steps) return;
    const int K = CP * P;
    for (int vv = static_cast<int>(threadIdx.x) - r0 * vecs; vv < vecs; vv += blockDim.x) {
        const int keep = K - 16 * vv;                     // codes of this vector; the rest is the zero pad
        uint8_t* out = A + (static_cast<long long>(strip) * gw + g0 + r0) * lda + 16 * vv;
        for (int r = r0; r < gn; r += steps, out += steps * lda) {
            uint4 q = *reinterpret_cast<const uint4*>(prep_tile + r * pitch + 16 * vv);
            if (keep < 16) {
                uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int k = keep - 4 * j;
                    w[j] = k >= 4 ? w[j] : k <= 0 ? 0u : w[j] & (0xFFFFFFFFu >> (32 - 8 * k));
                }
                q = make_uint4(w[0], w[1], w[2], w[3]);
            }
            *reinterpret_cast<uint4*>(out) = q;
        }
    }
}

// Chunks a thread has in flight, of the `steps` it takes in all: as many as leave the fewest places of the last round empty, and of
// those the most; the fewest where patch rows are cut into groups, because there are hardly two blocks per SM.  A round that is not full is a trip to memory for less.  256 images of 384 x 384, patch 14 (9 steps bf16, 21 fp32):
// 3 / 4 / 6 in flight 65.5 / 70.6 / 73.5 us, 89.5 / 94.5 / 95.6; 512 of 224 x 224, patch 16, bf16 (6): 47.7 / 51.0 / 44.9; 32 of them, fp32 (12):
// 5.3 / 5.0 / 4.3; 976 of 128 x 160, patch 16 (4 and 8): 40.7 / 36.7 / 41.9, 50.5 / 48.2 / 58.1; cut into groups (6), 13 of 224 x 224, patch 16: 2.8 / 3.0 / 3.2.
inline int unfold_batch(int steps, bool cut) {
    int best = 3, idle = (3 - steps % 3) % 3;
    for (int b : {4, 6}) {
        const int i = (b - steps % b) % b;
        if (i < idle || (i == idle && !cut)) best = b, idle = i;
    }
    return best;
}

template <typename PT, int MODE, bool ALIGNED, int BATCH>
cudaError_t launch_unfold_batch(unsigned grid, unsigned threads, size_t smem, cudaStream_t s, const PT* pixels, long long total, int H, int W, int P, int C, int gh, int gw,
                                int G, int groups, int rows_per_step, int chunks, const float* scale, uint8_t* A, long long lda, int row_bytes) {
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(patchify_quantize_kernel<PT, MODE, ALIGNED, BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    return sl8_launch_chained(patchify_quantize_kernel<PT, MODE, ALIGNED, BATCH>, grid, threads, smem, s, pixels, total, H, W, P, C, gh, gw, G, groups, rows_per_step,
                              fast_div(chunks), fast_div(P), fast_div(row_bytes / 16), scale, A, lda, row_bytes);
}

template <typename PT, int MODE, bool ALIGNED>
cudaError_t launch_unfold(unsigned grid, size_t smem, cudaStream_t s, const PT* pixels, int images, int C, int H, int W, int P,
                          int gh, int gw, int G, int groups, int chunks, const float* scale, uint8_t* A, long long lda, int row_bytes) {
    const int rows_per_step = kUnfoldThreads / chunks;                       // image rows a step of the block covers
    const unsigned threads = static_cast<unsigned>((rows_per_step * chunks + 31) / 32 * 32);
    const long long total = static_cast<long long>(images) * C * H * W;
    const int batch = unfold_batch((C * P + rows_per_step - 1) / rows_per_step, groups > 1);
    auto go = [&](auto launch) { return launch(grid, threads, smem, s, pixels, total, H, W, P, C, gh, gw, G, groups, rows_per_step, chunks, scale, A, lda, row_bytes); };
    return batch == 3 ? go(launch_unfold_batch<PT, MODE, ALIGNED, 3>) : batch == 4 ? go(launch_unfold_batch<PT, MODE, ALIGNED, 4>) : go(launch_unfold_batch<PT, MODE, ALIGNED, 6>);
}

template <typename PT>
cudaError_t unfold(cudaStream_t s, const PT* pixels, int images, int C, int H, int W, int P, int gh, int gw, const float* scale,
                   uint8_t* A, long long lda, int row_bytes, int sm_count) {
    constexpr int VP = 16 / sizeof(PT);
    // A whole patch row per block is the cheapest per byte; where there are fewer of them than two blocks per SM, the
    // patch rows are cut into groups, down to one 128-byte line of an image row (one 224 x 224 image: 14 -> 98 blocks).
    // They are cut too where the group's rows of A leave no room for four blocks per SM, or where an image row of it has
    // more chunks than a block has threads.
    const long long strips = static_cast<long long>(images) * gh;
    const int line = (128 + P * (int)sizeof(PT) - 1) / (P * (int)sizeof(PT));
    auto chunks_of = [&](int G) {                                            // chunks an image row of a group can touch
        return (G * P + VP - 1) / VP + (W % VP == 0 && (G == gw || (G * P) % VP == 0) ? 0 : 1);
    };
    int G = gw;
    while (G > line && (strips * ((gw + G - 1) / G) < 2LL * sm_count || G * (row_bytes + 16) > 48 * 1024 || chunks_of(G) > kUnfoldThreads))
        G = (G + 1) / 2 < line ? line : (G + 1) / 2;
    const int groups = (gw + G - 1) / G;
    const int chunks = chunks_of(G);
    // The fast path wants 32-bit offsets inside an image and a spare row of A in shared memory.
    const bool aligned = W % VP == 0 && (groups == 1 || (G * P) % VP == 0) && static_cast<long long>(C) * H * W * sizeof(PT) < (1LL << 32) &&
                         (G + 1) * (row_bytes + 16) <= 100 * 1024;
    const size_t smem = static_cast<size_t>(aligned ? G + 1 : G) * (row_bytes + 16);
    const unsigned grid = static_cast<unsigned>(strips * groups);
#define SL8_UNFOLD(MODE, AL) launch_unfold<PT, MODE, AL>(grid, smem, s, pixels, images, C, H, W, P, gh, gw, G, groups, chunks, scale, A, lda, row_bytes)
    if (aligned && P % VP == 0) return SL8_UNFOLD(UNFOLD_CHUNKS, true);
    if (P % 2 == 0 && aligned) return SL8_UNFOLD(UNFOLD_PAIRS, true);
    if (P % 2 == 0 && W % 2 == 0) return SL8_UNFOLD(UNFOLD_PAIRS, false);
    if (aligned) return SL8_UNFOLD(UNFOLD_BYTES, true);
    return SL8_UNFOLD(UNFOLD_BYTES, false);
#undef SL8_UNFOLD
}

// 448 = largest e4m3 value; an all-zero tensor keeps scale 1
__device__ __forceinline__ float scale_from_amax(float a) { return a > 0.0f ? a / 448.0f : 1.0f; }

// |x| of non-negative floats orders like their bit patterns: one atomicMax on the bits per block.
template <typename T>
__device__ __forceinline__ float prep_absmax8(const T* p) {          // max |.| of eight consecutive elements, 16-byte loads
    float m;
    if constexpr (sizeof(T) == 4) {
        const uint4 a = sl8::ld_16(p), b = sl8::ld_16(p + 4);
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        m = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; i++) m = fmaxf(m, fabsf(__uint_as_float(w[i])));
    } else {
        const uint4 q = sl8::ld_16(p);
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        m = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; i++)
            m = fmaxf(m, fmaxf(fabsf(__uint_as_float(w[i] << 16)), fabsf(__uint_as_float(w[i] & 0xFFFF0000u))));
    }
    return m;
}

// Walks the 8-element vectors of a [rows, 8 * per_row] matrix, `stride` vectors at a time, without a division per step.
struct VecWalk {
    long long r;      // row
    int c;            // vector inside the row
    __device__ __forceinline__ void step(const VecWalk& by, int per_row) {
        r += by.r;
        c += by.c;
        if (c >= per_row) { c -= per_row; r++; }
    }
};
__device__ __forceinline__ VecWalk vec_walk(uint32_t i, uint32_t per_row) { return VecWalk{i / per_row, static_cast<int>(i % per_row)}; }     // (a grid has far fewer than 2^32 threads)
// A block of 256 threads takes BATCH * 256 consecutive vectors at a time, BATCH of them in flight per thread.  One each where a
// single wave of blocks covers the matrix; `several` where it is larger but still comes from L2, whose latency one load per
// thread does not cover; one again, and twice the blocks, where it comes from HBM (46 656 x 1 152 bf16 quantised with 1 / 2 / 4
// in flight: 29.0 / 32.3 / 37.4 us; 5 832 x 4 304: 11.6 / 10.8 / 12.5 us).
constexpr int kPrepThreads = 256;
inline int prep_batch(sl8_handle_t h, long long vectors, int vector_bytes, int several) {
    if (vectors <= static_cast<long long>(h->sm_count) * 8 * kPrepThreads || vectors * vector_bytes > (64ll << 20)) return 1;
    return several;
}

// `vectors` != 0: rows of cols = 8 * vectors_per_row elements on 16-byte boundaries, eight elements per load;
// otherwise element by element.  With `scale`, the block that finishes last also writes it: until then the word counts the
// finished blocks (zero_two_kernel cleared both), which saves the launch of a kernel for one division.
// Bound by L2 / HBM reads: 50 MB (5 832 x 4 304 bf16) with
// the scale 10.5 -> 6.7 us (7.5 TB/s), 46 656 x 1 152 20.6 -> 17.2, 729 x 1 152, where the launches count, 6.3 -> 4.1.
template <typename T, int BATCH>
__global__ void __launch_bounds__(kPrepThreads) amax_kernel(const T* x, long long rows, int cols, long long ld, int vectors, unsigned* amax_bits, float* scale) {
    sl8::pdl_wait();
    sl8::pdl_release();
    float m = 0.0f;
    if (vectors) {
        const int vpr = cols / 8;
        float part[BATCH];
        if (ld == cols) {                                   // one run of vectors: no rows to walk
            const long long total = rows * vpr;
            for (long long i = blockIdx.x * (BATCH * kPrepThreads) + threadIdx.x; i < total; i += static_cast<long long>(gridDim.x) * (BATCH * kPrepThreads)) {
#pragma unroll
                for (int b = 0; b < BATCH; b++) part[b] = i + b * kPrepThreads < total ? prep_absmax8(x + 8 * (i + b * kPrepThreads)) : 0.0f;
#pragma unroll
                for (int b = 0; b < BATCH; b++) m = fmaxf(m, part[b]);
            }
        } else {
            VecWalk at = vec_walk(blockIdx.x * (BATCH * kPrepThreads) + threadIdx.x, vpr);
            const VecWalk by = vec_walk(kPrepThreads, vpr), on = vec_walk((gridDim.x - 1) * (BATCH * kPrepThreads), vpr);
            while (at.r < rows) {
#pragma unroll
                for (int b = 0; b < BATCH; b++) {
                    part[b] = at.r < rows ? prep_absmax8(x + at.r * ld + 8 * at.c) : 0.0f;
                    at.step(by, vpr);
                }
#pragma unroll
                for (int b = 0; b < BATCH; b++) m = fmaxf(m, part[b]);
                at.step(on, vpr);
            }
        }
    } else {
        const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
        const long long first = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
        const long long total = rows * cols;
        for (long long i = first; i < total; i += stride) {
            const long long r = i / cols;
            m = fmaxf(m, fabsf(prep_load(x + r * ld + (i - r * cols))));
        }
    }
    unsigned b = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
    __shared__ unsigned warp_max[32];
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x < 32) {
        b = threadIdx.x < (blockDim.x + 31) / 32 ? warp_max[threadIdx.x] : 0u;
        b = __reduce_max_sync(0xffffffffu, b);
        if (threadIdx.x == 0) {
            atomicMax(amax_bits, b);
            if (scale) {
                __threadfence();
                if (atomicAdd(reinterpret_cast<unsigned*>(scale), 1u) == gridDim.x - 1) {
                    __threadfence();
                    *scale = scale_from_amax(__uint_as_float(atomicMax(amax_bits, 0u)));
                }
            }
        }
    }
}

// (chained like the others; a cudaMemsetAsync would wait for the kernel ahead to drain and hold up the one behind it)
__global__ void zero_two_kernel(unsigned* a, unsigned* b) {
    sl8::pdl_wait();
    sl8::pdl_release();
    *a = 0u;
    if (b) *b = 0u;
}

// A caller that keeps only the scale, in the word of the abs-max.
__global__ void scale_in_place_kernel(float* amax) {
    sl8::pdl_wait();
    sl8::pdl_release();
    *amax = scale_from_amax(sl8::ld_f32(amax));
}

template <typename T>
__device__ __forceinline__ void ln_load8(const T* p, float (&v)[8]);
template <>
__device__ __forceinline__ void ln_load8<float>(const float* p, float (&v)[8]) {
    const uint4 a = sl8::ld_16(p), b = sl8::ld_16(p + 4);
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __uint_as_float(w[i]);
}
template <>
__device__ __forceinline__ void ln_load8<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[8]) {
    const uint4 q = sl8::ld_16(p);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
}

__device__ __forceinline__ uint32_t prep_e4m3x4(float a, float b, float c, float d) {
    return static_cast<uint32_t>(sl8::pack_e4m3x2(a, b)) | (static_cast<uint32_t>(sl8::pack_e4m3x2(c, d)) << 16);
}

// BATCH > 0: cols a multiple of 8, rows of x on 16-byte and of out on 8-byte boundaries: eight elements per load and store.
// BATCH == 0: group by group, element by element where a group is cut off or misaligned.
// 46 656 x 1 152 bf16: 33.9 -> 29.0 us (5.6 TB/s); 5 003 x 1 152 4.4 -> 4.2.
template <typename T, int BATCH>
__global__ void __launch_bounds__(kPrepThreads) quantize_e4m3_kernel(const T* x, long long rows, int cols, long long ld, const float* scale, uint8_t* out, long long ld_out) {
    const int groups = (cols + 7) / 8;                      // eight columns per thread: one 8-byte store
    sl8::pdl_wait();
    sl8::pdl_release();
    const float inv = __frcp_rn(scale ? sl8::ld_f32(scale) : 1.0f);
    if constexpr (BATCH > 0) {
        VecWalk at = vec_walk(blockIdx.x * (BATCH * kPrepThreads) + threadIdx.x, groups);
        const VecWalk by = vec_walk(kPrepThreads, groups), on = vec_walk((gridDim.x - 1) * (BATCH * kPrepThreads), groups);
        while (at.r < rows) {
            VecWalk to[BATCH];
            float v[BATCH][8];
#pragma unroll
            for (int b = 0; b < BATCH; b++) {
                to[b] = at;
                if (at.r < rows) ln_load8<T>(x + at.r * ld + 8 * at.c, v[b]);
                at.step(by, groups);
            }
#pragma unroll
            for (int b = 0; b < BATCH; b++)
                if (to[b].r < rows)
                    *reinterpret_cast<uint2*>(out + to[b].r * ld_out + 8 * to[b].c) =
                        make_uint2(prep_e4m3x4(v[b][0] * inv, v[b][1] * inv, v[b][2] * inv, v[b][3] * inv),
                                   prep_e4m3x4(v[b][4] * inv, v[b][5] * inv, v[b][6] * inv, v[b][7] * inv));
            at.step(on, groups);
        }
    } else {
        const long long first = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
        const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
        const long long total = rows * groups;
        for (long long i = first; i < total; i += stride) {
            const long long r = i / groups;
            const int c0 = static_cast<int>(i - r * groups) * 8;
            const T* src = x + r * ld + c0;
            uint8_t* dst = out + r * ld_out + c0;
            if (c0 + 8 <= cols && (reinterpret_cast<uintptr_t>(dst) & 7u) == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
                float v[8];
                ln_load8<T>(src, v);
                *reinterpret_cast<uint2*>(dst) = make_uint2(prep_e4m3x4(v[0] * inv, v[1] * inv, v[2] * inv, v[3] * inv),
                                                            prep_e4m3x4(v[4] * inv, v[5] * inv, v[6] * inv, v[7] * inv));
            } else {
                float v[8];       // all loads first: a store between two keeps the second from being issued (fp32 46 656 x 1 155 85 -> 63 us)
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (c0 + j < cols) v[j] = prep_load(src + j);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (c0 + j < cols) dst[j] = prep_e4m3(v[j] * inv);
            }
        }
    }
}

// bf16 rows on 32-byte and codes on 16-byte boundaries: sixteen elements per load and store.  Half the instructions per byte, which
// is what bounds the eight-element form while the rows come from L2: 5 832 x 4 304 10.9 -> 8.0 us there, 16.4 -> 12.9 from HBM;
// 5 003 x 1 152 4.0 -> 3.1, 46 656 x 1 152 28.6 -> 25.2 (6.4 TB/s), 729 rows the same.  32 blocks per SM where one vector each is in flight
// (16: 26.1).  fp32 rows, two such loads per store, were 5 - 15 % slower up to 6 000 rows and 2 % faster from HBM: they keep the form above.
template <int BATCH>
__global__ void __launch_bounds__(kPrepThreads) quantize_bf16_wide_kernel(const __nv_bfloat16* x, long long rows, int cols, long long ld, const float* scale, uint8_t* out,
                                                                          long long ld_out) {
    const int groups = cols / 16;
    VecWalk at = vec_walk(blockIdx.x * (BATCH * kPrepThreads) + threadIdx.x, groups);
    const VecWalk by = vec_walk(kPrepThreads, groups), on = vec_walk((gridDim.x - 1) * (BATCH * kPrepThreads), groups);
    sl8::pdl_wait();
    sl8::pdl_release();
    const float inv = __frcp_rn(scale ? sl8::ld_f32(scale) : 1.0f);
    while (at.r < rows) {
        VecWalk to[BATCH];
        uint32_t w[BATCH][8];
#pragma unroll
        for (int b = 0; b < BATCH; b++) {
            to[b] = at;
            if (at.r < rows) sl8::ld_32(x + at.r * ld + 16 * at.c, w[b]);
            at.step(by, groups);
        }
#pragma unroll
        for (int b = 0; b < BATCH; b++)
            if (to[b].r < rows) {
                uint32_t q[4];
#pragma unroll
                for (int i = 0; i < 4; i++)
                    q[i] = prep_e4m3x4(sl8::bf16_lo_f32(w[b][2 * i]) * inv, sl8::bf16_hi_f32(w[b][2 * i]) * inv, sl8::bf16_lo_f32(w[b][2 * i + 1]) * inv,
                                       sl8::bf16_hi_f32(w[b][2 * i + 1]) * inv);
                *reinterpret_cast<uint4*>(out + to[b].r * ld_out + 16 * to[b].c) = make_uint4(q[0], q[1], q[2], q[3]);
            }
        at.step(on, groups);
    }
}

// Blocks for that many threads' worth of work, at most `per_sm` to an SM (eight fill it; more let the scheduler even out the end).
int prep_grid(sl8_handle_t h, long long work_items, int per_sm) {
    const long long want = (work_items + kPrepThreads - 1) / kPrepThreads;
    const long long cap = static_cast<long long>(h->sm_count > 0 ? h->sm_count : 148) * per_sm;
    return static_cast<int>(want < cap ? (want < 1 ? 1 : want) : cap);
}

}  // namespace

SL8_API int sl8_patchify_quantize_e4m3(sl8_handle_t h, const void* pixels, int pixel_dtype, int images, int channels,
                                       int height, int width, int patch, const float* scale, void* A, int64_t lda,
                                       sl8_stream_t stream) {
    if (!h) return SL8_ERR_INVALID_VALUE;
    if (!pixels || !A || images < 1 || channels < 1 || patch < 1 || height < patch || width < patch)
        return fail(h, SL8_ERR_INVALID_VALUE, "bad patchify arguments");
    if (pixel_dtype != SL8_DT_F32 && pixel_dtype != SL8_DT_BF16) return fail(h, SL8_ERR_INVALID_VALUE, "unknown pixel dtype");
    const int K = channels * patch * patch, gh = height / patch, gw = width / patch;
    if (lda < K) return fail(h, SL8_ERR_INVALID_VALUE, "lda smaller than channels * patch * patch");
    if (!aligned16(A) || lda % 16 != 0) return fail(h, SL8_ERR_ALIGNMENT, "A and lda must be multiples of 16 bytes");
    if (!aligned16(pixels)) return fail(h, SL8_ERR_ALIGNMENT, "pixels must be 16-byte aligned");
    // whole rows are written when the pad is short (K = 588 at pitch 640), else K rounded up to 16 bytes
    const int row_bytes = static_cast<int>(lda - K < 128 ? lda : (K + 15) / 16 * 16);
    const size_t smem = static_cast<size_t>(gw) * row_bytes;
    if (smem > 200 * 1024) return fail(h, SL8_ERR_UNSUPPORTED, "one strip of patches exceeds 200 KiB of shared memory");
    DeviceGuard guard(h->device);
    if (!guard.ok) return fail(h, SL8_ERR_CUDA, "cudaSetDevice failed");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const cudaError_t e =
        pixel_dtype == SL8_DT_F32
            ? unfold(s, static_cast<const float*>(pixels), images, channels, height, width, patch, gh, gw, scale, static_cast<uint8_t*>(A), lda, row_bytes, h->sm_count)
            : unfold(s, static_cast<const __nv_bfloat16*>(pixels), images, channels, height, width, patch, gh, gw, scale, static_cast<uint8_t*>(A), lda, row_bytes, h->sm_count);
    return e == cudaSuccess ? SL8_OK : fail_cuda(h, e, "patchify kernel launch");
}

SL8_API int sl8_amax_scale(sl8_handle_t h, const void* x, int dtype, int64_t rows, int cols, int64_t ld, float* amax,
                           float* scale, sl8_stream_t stream) {
    if (!h) return SL8_ERR_INVALID_VALUE;
    if (!x || !amax || rows < 1 || cols < 1 || ld < cols) return fail(h, SL8_ERR_INVALID_VALUE, "bad amax arguments");
    if (dtype != SL8_DT_F32 && dtype != SL8_DT_BF16) return fail(h, SL8_ERR_INVALID_VALUE, "unknown dtype");
    DeviceGuard guard(h->device);
    if (!guard.ok) return fail(h, SL8_ERR_CUDA, "cudaSetDevice failed");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool in_place = scale == amax;
    float* const ticket = in_place ? nullptr : scale;
    cudaError_t e = sl8_launch_chained(zero_two_kernel, 1, 1, 0, s, reinterpret_cast<unsigned*>(amax), reinterpret_cast<unsigned*>(ticket));
    if (e != cudaSuccess) return fail_cuda(h, e, "amax kernel launch");
    const int vectors = (cols % 8 == 0 && ld % 8 == 0 && aligned16(x)) ? 1 : 0;
    const int batch = vectors ? prep_batch(h, rows * cols / 8, dtype == SL8_DT_F32 ? 32 : 16, 4) : 1;
    const int grid = prep_grid(h, rows * cols / 8 / batch, batch > 1 ? 8 : 16);
    auto launch = [&](auto kernel, auto* src) {
        return sl8_launch_chained(kernel, grid, kPrepThreads, 0, s, src, rows, cols, ld, vectors, reinterpret_cast<unsigned*>(amax), ticket);
    };
    if (dtype == SL8_DT_F32) e = launch(batch == 1 ? amax_kernel<float, 1> : amax_kernel<float, 4>, static_cast<const float*>(x));
    else e = launch(batch == 1 ? amax_kernel<__nv_bfloat16, 1> : amax_kernel<__nv_bfloat16, 4>, static_cast<const __nv_bfloat16*>(x));
    if (in_place && e == cudaSuccess) e = sl8_launch_chained(scale_in_place_kernel, 1, 1, 0, s, amax);
    return e == cudaSuccess ? SL8_OK : fail_cuda(h, e, "amax kernel launch");
}

SL8_API int sl8_quantize_e4m3(sl8_handle_t h, const void* x, int dtype, int64_t rows, int cols, int64_t ld, const float* scale,
                              void* out, int64_t ld_out, sl8_stream_t stream) {
    if (!h) return SL8_ERR_INVALID_VALUE;
    if (!x || !out || rows < 1 || cols < 1 || ld < cols || ld_out < cols) return fail(h, SL8_ERR_INVALID_VALUE, "bad quantize arguments");
    if (dtype != SL8_DT_F32 && dtype != SL8_DT_BF16) return fail(h, SL8_ERR_INVALID_VALUE, "unknown dtype");
    DeviceGuard guard(h->device);
    if (!guard.ok) return fail(h, SL8_ERR_CUDA, "cudaSetDevice failed");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool vec = cols % 8 == 0 && ld % 8 == 0 && aligned16(x) && ld_out % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 7u) == 0;
    const int batch = vec ? prep_batch(h, rows * (cols / 8), dtype == SL8_DT_F32 ? 32 : 16, 2) : 0;
    const int grid = prep_grid(h, rows * ((cols + 7) / 8) / (vec ? batch : 1), 16);
    auto launch = [&](auto general, auto one, auto two, auto* src) {
        return sl8_launch_chained(batch == 0 ? general : batch == 1 ? one : two, grid, kPrepThreads, 0, s, src, rows, cols, ld, scale, static_cast<uint8_t*>(out), ld_out);
    };
    typedef __nv_bfloat16 bf16;
    if (dtype == SL8_DT_BF16 && cols % 16 == 0 && ld % 16 == 0 && (reinterpret_cast<uintptr_t>(x) & 31u) == 0 && ld_out % 16 == 0 && aligned16(out)) {
        const long long vectors = rows * (cols / 16);
        const bool two = prep_batch(h, vectors, 32, 2) == 2;
        const cudaError_t we = sl8_launch_chained(two ? quantize_bf16_wide_kernel<2> : quantize_bf16_wide_kernel<1>, prep_grid(h, vectors / (two ? 2 : 1), two ? 16 : 32),
                                                  kPrepThreads, 0, s, static_cast<const bf16*>(x), rows, cols, ld, scale, static_cast<uint8_t*>(out), ld_out);
        return we == cudaSuccess ? SL8_OK : fail_cuda(h, we, "quantize kernel launch");
    }
    const cudaError_t e = dtype == SL8_DT_F32
        ? launch(quantize_e4m3_kernel<float, 0>, quantize_e4m3_kernel<float, 1>, quantize_e4m3_kernel<float, 2>, static_cast<const float*>(x))
        : launch(quantize_e4m3_kernel<bf16, 0>, quantize_e4m3_kernel<bf16, 1>, quantize_e4m3_kernel<bf16, 2>, static_cast<const bf16*>(x));
    return e == cudaSuccess ? SL8_OK : fail_cuda(h, e, "quantize kernel launch");
}

// ---- LayerNorm -> quantise: the prologue of FC1 (docs/architecture.md:92-101 of the reference lists it as unstarted).
// One warp per row: mean, variance (two passes, fp32, the row stays in L1 after the first), then
// e4m3((x - mean) * rsqrt(var + eps) * gamma + beta) * (1 / scale), eight columns per lane and step.
namespace {

// 16-byte pieces of eight consecutive elements, as loaded, and their values.
template <typename T>
struct Raw8 {
    uint4 q[sizeof(T) / 2];
};
template <typename T>
__device__ __forceinline__ void raw_load(const T* p, Raw8<T>& x) {
#pragma unroll
    for (int i = 0; i < (int)sizeof(T) / 2; i++) x.q[i] = sl8::ld_16(p + 4 * i);
}
template <typename T>
__device__ __forceinline__ void raw_values(const Raw8<T>& x, float (&v)[8]) {
    const uint32_t w[4] = {x.q[0].x, x.q[0].y, x.q[0].z, x.q[0].w};
    if constexpr (sizeof(T) == 4) {
        const uint32_t u[4] = {x.q[1].x, x.q[1].y, x.q[1].z, x.q[1].w};
#pragma unroll
        for (int i = 0; i < 4; i++) { v[i] = __uint_as_float(w[i]); v[4 + i] = __uint_as_float(u[i]); }
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u); }
    }
}

// Eight elements: d = x - mean -> ((d * rstd) * gamma + beta) * (1 / scale) -> eight e4m3 codes, one 8-byte store.
__device__ __forceinline__ void ln_emit(const float (&d)[8], const float (&g)[8], const float (&b)[8], float rstd, float inv, uint8_t* out) {
    float y[8];
#pragma unroll
    for (int i = 0; i < 8; i++) y[i] = fmaf(d[i] * rstd, g[i], b[i]) * inv;
    *reinterpret_cast<uint2*>(out) = make_uint2(prep_e4m3x4(y[0], y[1], y[2], y[3]), prep_e4m3x4(y[4], y[5], y[6], y[7]));
}
__device__ __forceinline__ void ln_affine(const float* p, float otherwise, float (&v)[8]) {
    if (p) ln_load8<float>(p, v);
    else {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = otherwise;
    }
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

constexpr int kLnThreads = 128;

// cols <= 256 * CHUNKS: a warp keeps its columns' gamma and beta in registers, walks down the rows and has the next row on its
// way while it works on this one.  (Read per row, from L1, gamma and beta are four times the bytes of a bf16 row, and they were
// asked for only after the row's two reductions.)  Scalar fp32 arithmetic: the packed two-element forms were measured
// 20 - 40 % slower here.  bf16, 1 152 columns: 729 rows 3.6 -> 2.8 us,
// 5 003 rows 8.5 -> 5.5, 46 656 rows 49 -> 39.5 (4.1 TB/s); 1 600 columns, 5 003 rows 15.9 -> 7.8.  Gamma and beta read per row instead, and four
// blocks per SM for the registers that frees: 5 003 rows 7.5 us, 46 656 rows 42.  A ring of three rows in
// shared memory filled by cp.async was 10 % slower up to 12 000 rows and up to 60 % in fp32, 12 % faster from 46 656 bf16 rows.
// (2 048 columns: registers for the row only, gamma and beta a chunk ahead of their use.)
template <typename T, int CHUNKS>
struct LnShape {
    static constexpr bool KEEP = CHUNKS <= (sizeof(T) == 4 ? 5 : 7);
    static constexpr bool AHEAD = KEEP || sizeof(T) == 2;                    // the next row's loads are issued a row early
    static constexpr int PER_SM = CHUNKS > 5 ? 2 : sizeof(T) == 4 ? (CHUNKS <= 3 ? 3 : 2) : (CHUNKS <= 3 ? 4 : 3);
};
template <typename T, int CHUNKS>
__global__ void __launch_bounds__(kLnThreads, LnShape<T, CHUNKS>::PER_SM)
layernorm_quantize_kernel(const T* x, long long rows, int cols, long long ld, const float* gamma, const float* beta, float eps,
                          const float* scale, uint8_t* out, long long ld_out) {
    constexpr bool KEEP = LnShape<T, CHUNKS>::KEEP, AHEAD = LnShape<T, CHUNKS>::AHEAD;
    const int c0 = (threadIdx.x & 31) * 8;
    const long long warps = (static_cast<long long>(gridDim.x) * kLnThreads) >> 5;
    long long r = (static_cast<long long>(blockIdx.x) * kLnThreads + threadIdx.x) >> 5;
    const float inv_n = 1.0f / static_cast<float>(cols);
    sl8::pdl_wait();
    sl8::pdl_release();
    if (r >= rows) return;
    Raw8<T> next[CHUNKS];
    auto fetch = [&](long long row) {
#pragma unroll
        for (int j = 0; j < CHUNKS; j++)
            if (c0 + 256 * j < cols) raw_load<T>(x + row * ld + c0 + 256 * j, next[j]);
    };
    fetch(r);
    const float inv = __frcp_rn(scale ? sl8::ld_f32(scale) : 1.0f);
    constexpr int NG = KEEP ? CHUNKS : 2;
    float g[NG][8], b[NG][8];
    auto affine = [&](int j) {
        if (c0 + 256 * j < cols) {
            ln_affine(gamma ? gamma + c0 + 256 * j : nullptr, 1.0f, g[j % NG]);
            ln_affine(beta ? beta + c0 + 256 * j : nullptr, 0.0f, b[j % NG]);
        }
    };
#pragma unroll
    for (int j = 0; j < (KEEP ? CHUNKS : 1); j++) affine(j);
    for (; r < rows; r += warps) {
        float v[CHUNKS][8];
        float sum = 0.0f, sq = 0.0f;
#pragma unroll
        for (int j = 0; j < CHUNKS; j++)
            if (c0 + 256 * j < cols) {
                raw_values<T>(next[j], v[j]);
#pragma unroll
                for (int i = 0; i < 8; i++) sum += v[j][i];
            }
        if (AHEAD && r + warps < rows) fetch(r + warps);
        const float mean = warp_sum(sum) * inv_n;
#pragma unroll
        for (int j = 0; j < CHUNKS; j++)
            if (c0 + 256 * j < cols) {
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    v[j][i] -= mean;
                    sq = fmaf(v[j][i], v[j][i], sq);
                }
            }
        const float rstd = rsqrtf(warp_sum(sq) * inv_n + eps);
#pragma unroll
        for (int j = 0; j < CHUNKS; j++) {
            if (!KEEP && j + 1 < CHUNKS) affine(j + 1);
            if (c0 + 256 * j < cols) ln_emit(v[j], g[j % NG], b[j % NG], rstd, inv, out + r * ld_out + c0 + 256 * j);
            if (!KEEP && j + 1 == CHUNKS) affine(0);          // for the next row
        }
        if (!AHEAD && r + warps < rows) fetch(r + warps);
    }
}

// fp32 rows that come from HBM, without gamma and beta to keep: a row of registers per warp, and four times the warps, whose
// loads cover for one another.  46 656 x 1 152 48.0 -> 41.0 us (6.5 TB/s), 11 664 rows 14.1 -> 12.2; with gamma and beta,
// which every row would read again, 20 000 x 1 280 would go from 24.1 to 25.8.  Below 48 MiB the rows come from L2 in part: 5 003 rows 6.1 either way.
template <int CHUNKS>
__global__ void __launch_bounds__(kLnThreads) layernorm_quantize_plain_kernel(const float* x, long long rows, int cols, long long ld, float eps, const float* scale,
                                                                              uint8_t* out, long long ld_out) {
    const int c0 = (threadIdx.x & 31) * 8;
    const long long warps = (static_cast<long long>(gridDim.x) * kLnThreads) >> 5;
    sl8::pdl_wait();
    sl8::pdl_release();
    const float inv = __frcp_rn(scale ? sl8::ld_f32(scale) : 1.0f);
    const float inv_n = 1.0f / static_cast<float>(cols);
    for (long long r = (static_cast<long long>(blockIdx.x) * kLnThreads + threadIdx.x) >> 5; r < rows; r += warps) {
        float v[CHUNKS][8], sum = 0.0f, sq = 0.0f;
#pragma unroll
        for (int j = 0; j < CHUNKS; j++)
            if (c0 + 256 * j < cols) ln_load8<float>(x + r * ld + c0 + 256 * j, v[j]);
#pragma unroll
        for (int j = 0; j < CHUNKS; j++)
            if (c0 + 256 * j < cols) {
#pragma unroll
                for (int i = 0; i < 8; i++) sum += v[j][i];
            }
        const float mean = warp_sum(sum) * inv_n;
#pragma unroll
        for (int j = 0; j < CHUNKS; j++)
            if (c0 + 256 * j < cols) {
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    v[j][i] -= mean;
                    sq = fmaf(v[j][i], v[j][i], sq);
                }
            }
        const float rstd = rsqrtf(warp_sum(sq) * inv_n + eps);
        float g[8], b[8];
        ln_affine(nullptr, 1.0f, g);
        ln_affine(nullptr, 0.0f, b);
#pragma unroll
        for (int j = 0; j < CHUNKS; j++)
            if (c0 + 256 * j < cols) ln_emit(v[j], g, b, rstd, inv, out + r * ld_out + c0 + 256 * j);
    }
}

// Wider rows: a warp per row, three passes over it (the second and third hit L1 / L2).  Twice the blocks that are resident: their
// rows end at different times (20 000 bf16 rows of 2 304 / 4 304 / 8 192: 45.4 / 89.8 / 169.6 -> 41.9 / 85.4 / 158.2 us).
template <typename T>
__global__ void __launch_bounds__(kLnThreads) layernorm_quantize_wide_kernel(const T* x, long long rows, int cols, long long ld, const float* gamma,
                                                                             const float* beta, float eps, const float* scale, uint8_t* out, long long ld_out) {
    const int c0 = (threadIdx.x & 31) * 8;
    const long long warps = (static_cast<long long>(gridDim.x) * kLnThreads) >> 5;
    sl8::pdl_wait();
    sl8::pdl_release();
    const float inv = __frcp_rn(scale ? sl8::ld_f32(scale) : 1.0f);
    const float inv_n = 1.0f / static_cast<float>(cols);
    for (long long r = (static_cast<long long>(blockIdx.x) * kLnThreads + threadIdx.x) >> 5; r < rows; r += warps) {
        const T* row = x + r * ld;
        float v[8], sum = 0.0f, sq = 0.0f;
        for (int c = c0; c < cols; c += 256) {
            ln_load8<T>(row + c, v);
#pragma unroll
            for (int i = 0; i < 8; i++) sum += v[i];
        }
        const float mean = warp_sum(sum) * inv_n;
        for (int c = c0; c < cols; c += 256) {
            ln_load8<T>(row + c, v);
#pragma unroll
            for (int i = 0; i < 8; i++) sq = fmaf(v[i] - mean, v[i] - mean, sq);
        }
        const float rstd = rsqrtf(warp_sum(sq) * inv_n + eps);
        for (int c = c0; c < cols; c += 256) {
            float g[8], b[8];
            ln_load8<T>(row + c, v);
            ln_affine(gamma ? gamma + c : nullptr, 1.0f, g);
            ln_affine(beta ? beta + c : nullptr, 0.0f, b);
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] -= mean;
            ln_emit(v, g, b, rstd, inv, out + r * ld_out + c);
        }
    }
}

template <typename T>
cudaError_t launch_layernorm(int sm_count, cudaStream_t s, const T* x, long long rows, int cols, long long ld, const float* gamma,
                             const float* beta, float eps, const float* scale, uint8_t* out, long long ld_out) {
    auto launch = [&](auto kernel, int per_sm) {              // a warp per row, no more blocks than are resident at once
        const long long want = (rows + kLnThreads / 32 - 1) / (kLnThreads / 32), cap = static_cast<long long>(sm_count) * per_sm;
        return sl8_launch_chained(kernel, static_cast<unsigned>(want < cap ? want : cap), kLnThreads, 0, s, x, rows, cols, ld, gamma, beta, eps, scale, out, ld_out);
    };
    if constexpr (sizeof(T) == 4)
        if (!gamma && !beta && cols > 768 && cols <= 1280 && rows * cols > (12ll << 20)) {
            const long long want = (rows + kLnThreads / 32 - 1) / (kLnThreads / 32), cap = static_cast<long long>(sm_count) * 32;
            return sl8_launch_chained(layernorm_quantize_plain_kernel<5>, static_cast<unsigned>(want < cap ? want : cap), kLnThreads, 0, s, x, rows, cols, ld, eps, scale, out, ld_out);
        }
    if (cols <= 768) return launch(layernorm_quantize_kernel<T, 3>, LnShape<T, 3>::PER_SM);
    if (cols <= 1280) return launch(layernorm_quantize_kernel<T, 5>, LnShape<T, 5>::PER_SM);
    if (cols <= 1792) return launch(layernorm_quantize_kernel<T, 7>, LnShape<T, 7>::PER_SM);
    if (cols <= 2048) return launch(layernorm_quantize_kernel<T, 8>, LnShape<T, 8>::PER_SM);
    return launch(layernorm_quantize_wide_kernel<T>, 32);
}

}  // namespace

SL8_API int sl8_layernorm_quantize_e4m3(sl8_handle_t h, const void* x, int dtype, int64_t rows, int cols, int64_t ld,
                                        const float* gamma, const float* beta, float eps, const float* scale, void* out,
                                        int64_t ld_out, sl8_stream_t stream) {
    if (!h) return SL8_ERR_INVALID_VALUE;
    if (!x || !out || rows < 1 || cols < 1 || ld < cols || ld_out < cols || !(eps >= 0.0f))
        return fail(h, SL8_ERR_INVALID_VALUE, "bad layernorm arguments");
    if (dtype != SL8_DT_F32 && dtype != SL8_DT_BF16) return fail(h, SL8_ERR_INVALID_VALUE, "unknown dtype");
    if (cols % 8 != 0 || ld % 8 != 0 || ld_out % 8 != 0) return fail(h, SL8_ERR_UNSUPPORTED, "cols, ld and ld_out must be multiples of 8");
    if (!aligned16(x) || (reinterpret_cast<uintptr_t>(out) & 7u) != 0 || (gamma && !aligned16(gamma)) || (beta && !aligned16(beta)))
        return fail(h, SL8_ERR_ALIGNMENT, "x, gamma, beta must be 16-byte aligned and out 8-byte aligned");
    DeviceGuard guard(h->device);
    if (!guard.ok) return fail(h, SL8_ERR_CUDA, "cudaSetDevice failed");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaError_t e;
    if (dtype == SL8_DT_F32)
        e = launch_layernorm<float>(h->sm_count, s, static_cast<const float*>(x), rows, cols, ld, gamma, beta, eps, scale, static_cast<uint8_t*>(out), ld_out);
    else
        e = launch_layernorm<__nv_bfloat16>(h->sm_count, s, static_cast<const __nv_bfloat16*>(x), rows, cols, ld, gamma, beta, eps, scale,
                                        static_cast<uint8_t*>(out), ld_out);
    return e == cudaSuccess ? SL8_OK : fail_cuda(h, e, "layernorm kernel launch");
}
