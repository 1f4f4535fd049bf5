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
constexpr int kUnfoldBatch = 4;         // chunks a thread has in flight

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
// Bound by HBM where three things are seen to.  Bytes in flight: four 16-byte loads per thread (it was one load of two
// pixels).  Banks: rows of A are multiples of 128 bytes, so unpadded the same pixel of every patch falls into one bank; 16
// bytes of pad per row spread eight patches over all of them.  Instructions: a thread keeps its chunk position and walks
// down the image rows, so that where its codes go is worked out once (ALIGNED: every image row starts on a 16-byte
// boundary, and an image is less than 4 GiB) and a chunk costs its load, conversion, stores and a few additions; dividing
// for every pair of pixels took 24 instructions per pixel, and the kernel ran at a third of the bandwidth, issue-bound.
// 256 images of 384 x 384, patch 14: bf16 130 -> 70 us (4.9 TB/s), fp32 123 -> 97 us (5.7 TB/s); 32 images of 224 x 224,
// patch 16, fp32: 11.5 -> 5.0 us; one such image 7.1 -> 2.2 us.
template <typename PT, int MODE, bool ALIGNED>
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
                uint4 q[kUnfoldBatch];
#pragma unroll
                for (int b = 0; b < kUnfoldBatch; b++) {
                    if (left > b * rows_per_step) q[b] = ld_once_16(base + src);
                    src += row_step;
                    py += rows_per_step;
                    while (py >= P) { py -= P; src += plane_step; }
                }
#pragma unroll
                for (int b = 0; b < kUnfoldBatch; b++) {
                    if (left > b * rows_per_step) unfold_put<PT, MODE, false, NO>(q[b], inv2, dst, to);
                    dst += dst_step;
                }
                left -= kUnfoldBatch * rows_per_step;
            }
        }
    } else if (row0 < rows_per_step) {
        for (int cp0 = row0; cp0 < CP; cp0 += rows_per_step * kUnfoldBatch) {
            uint4 q[kUnfoldBatch];
            int x[kUnfoldBatch];                          // first pixel of the chunk relative to the group
#pragma unroll
            for (int b = 0; b < kUnfoldBatch; b++) {
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
            for (int b = 0; b < kUnfoldBatch; b++) {
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

template <typename PT, int MODE, bool ALIGNED>
cudaError_t launch_unfold(unsigned grid, size_t smem, cudaStream_t s, const PT* pixels, int images, int C, int H, int W, int P,
                          int gh, int gw, int G, int groups, int chunks, const float* scale, uint8_t* A, long long lda, int row_bytes) {
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(patchify_quantize_kernel<PT, MODE, ALIGNED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    const int rows_per_step = kUnfoldThreads / chunks;                       // image rows a step of the block covers
    const int threads = (rows_per_step * chunks + 31) / 32 * 32;
    const long long total = static_cast<long long>(images) * C * H * W;
    return sl8_launch_chained(patchify_quantize_kernel<PT, MODE, ALIGNED>, grid, threads, smem, s, pixels, total, H, W, P, C, gh, gw, G, groups, rows_per_step,
                              fast_div(chunks), fast_div(P), fast_div(row_bytes / 16), scale, A, lda, row_bytes);
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

// `vectors` != 0: rows of cols = 8 * vectors_per_row elements on 16-byte boundaries, eight elements per load;
// otherwise element by element.
template <typename T>
__global__ void amax_kernel(const T* x, long long rows, int cols, long long ld, int vectors,
                            unsigned* amax_bits) {
    sl8::pdl_wait();
    sl8::pdl_release();
    float m = 0.0f;
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    const long long first = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (vectors) {
        const int vpr = cols / 8;
        const long long total = rows * vpr;
        if (ld == cols) {
            for (long long i = first; i < total; i += stride) m = fmaxf(m, prep_absmax8(x + 8 * i));
        } else {
            for (long long i = first; i < total; i += stride) {
                const long long r = i / vpr;
                m = fmaxf(m, prep_absmax8(x + r * ld + 8 * (i - r * vpr)));
            }
        }
    } else {
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
        if (threadIdx.x == 0) atomicMax(amax_bits, b);
    }
}

__global__ void scale_from_amax_kernel(const float* amax, float* scale) {
    sl8::pdl_wait();
    sl8::pdl_release();
    const float a = sl8::ld_f32(amax);
    *scale = a > 0.0f ? a / 448.0f : 1.0f;                 // 448 = largest e4m3 value; an all-zero tensor keeps scale 1
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

template <typename T>
__global__ void quantize_e4m3_kernel(const T* x, long long rows, int cols, long long ld, const float* scale, uint8_t* out, long long ld_out) {
    sl8::pdl_wait();
    sl8::pdl_release();
    const float inv = __frcp_rn(scale ? sl8::ld_f32(scale) : 1.0f);
    const int groups = (cols + 7) / 8;                      // eight columns per thread: one 8-byte store
    const long long total = rows * groups;
    for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long r = i / groups;
        const int c0 = static_cast<int>(i - r * groups) * 8;
        const T* src = x + r * ld + c0;
        uint8_t* dst = out + r * ld_out + c0;
        if (c0 + 8 <= cols && (reinterpret_cast<uintptr_t>(dst) & 7u) == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
            float v[8];
            ln_load8<T>(src, v);
            uint32_t w[2];
#pragma unroll
            for (int h2 = 0; h2 < 2; h2++)
                w[h2] = static_cast<uint32_t>(sl8::pack_e4m3x2(v[4 * h2] * inv, v[4 * h2 + 1] * inv)) |
                        (static_cast<uint32_t>(sl8::pack_e4m3x2(v[4 * h2 + 2] * inv, v[4 * h2 + 3] * inv)) << 16);
            *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
        } else {
            for (int c = c0; c < cols && c < c0 + 8; c++) dst[c - c0] = prep_e4m3(prep_load(src + (c - c0)) * inv);
        }
    }
}

int prep_grid(sl8_handle_t h, long long work_items) {
    const long long want = (work_items + 255) / 256;
    const long long cap = static_cast<long long>(h->sm_count > 0 ? h->sm_count : 148) * 16;   // a multiple of the SM count
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
    cudaError_t e = cudaMemsetAsync(amax, 0, sizeof(float), s);
    if (e != cudaSuccess) return fail_cuda(h, e, "cudaMemsetAsync(amax)");
    const int grid = prep_grid(h, rows * cols / 8);
    const int vectors = (cols % 8 == 0 && ld % 8 == 0 && aligned16(x)) ? 1 : 0;
    if (dtype == SL8_DT_F32)
        e = sl8_launch_chained(amax_kernel<float>, grid, 256, 0, s, static_cast<const float*>(x), rows, cols, ld, vectors, reinterpret_cast<unsigned*>(amax));
    else
        e = sl8_launch_chained(amax_kernel<__nv_bfloat16>, grid, 256, 0, s, static_cast<const __nv_bfloat16*>(x), rows, cols, ld, vectors,
                               reinterpret_cast<unsigned*>(amax));
    if (scale && e == cudaSuccess) e = sl8_launch_chained(scale_from_amax_kernel, 1, 1, 0, s, amax, scale);
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
    const int grid = prep_grid(h, rows * ((cols + 7) / 8));
    cudaError_t e;
    if (dtype == SL8_DT_F32)
        e = sl8_launch_chained(quantize_e4m3_kernel<float>, grid, 256, 0, s, static_cast<const float*>(x), rows, cols, ld, scale, static_cast<uint8_t*>(out), ld_out);
    else
        e = sl8_launch_chained(quantize_e4m3_kernel<__nv_bfloat16>, grid, 256, 0, s, static_cast<const __nv_bfloat16*>(x), rows, cols, ld, scale,
                               static_cast<uint8_t*>(out), ld_out);
    return e == cudaSuccess ? SL8_OK : fail_cuda(h, e, "quantize kernel launch");
}

// ---- LayerNorm -> quantise: the prologue of FC1 (docs/architecture.md:92-101 of the reference lists it as unstarted).
// One warp per row: mean, variance (two passes, fp32, the row stays in L1 after the first), then
// e4m3((x - mean) * rsqrt(var + eps) * gamma + beta) * (1 / scale), eight columns per lane and step.
namespace {

// CHUNKS > 0: cols <= 256 * CHUNKS and the lane keeps its 8 * CHUNKS elements in registers (x is read once);
// CHUNKS == 0: any width, three passes over the row (the second and third hit L1 / L2).  Scalar fp32 arithmetic:
// the packed two-element forms were measured 20 - 40 % slower here.
template <typename T, int CHUNKS>
__global__ void __launch_bounds__(256, 3) layernorm_quantize_kernel(const T* x, long long rows, int cols, long long ld, const float* gamma,
                                          const float* beta, float eps, const float* scale, uint8_t* out, long long ld_out) {
    const int lane = threadIdx.x & 31;
    const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const long long warps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
    sl8::pdl_wait();
    sl8::pdl_release();
    const float inv = __frcp_rn(scale ? sl8::ld_f32(scale) : 1.0f);
    const float inv_n = 1.0f / static_cast<float>(cols);
    constexpr int NC = CHUNKS > 0 ? CHUNKS : 1;
    for (long long r = warp; r < rows; r += warps) {
        const T* row = x + r * ld;
        float v[NC][8];
        float sum = 0.0f;
        if constexpr (CHUNKS > 0) {
#pragma unroll
            for (int j = 0; j < NC; j++) {
                const int c = lane * 8 + 256 * j;
                if (c < cols) {
                    ln_load8<T>(row + c, v[j]);
#pragma unroll
                    for (int i = 0; i < 8; i++) sum += v[j][i];
                }
            }
        } else {
            for (int c = lane * 8; c < cols; c += 256) {
                ln_load8<T>(row + c, v[0]);
#pragma unroll
                for (int i = 0; i < 8; i++) sum += v[0][i];
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const float mean = sum * inv_n;
        float sq = 0.0f;
        if constexpr (CHUNKS > 0) {
#pragma unroll
            for (int j = 0; j < NC; j++)
                if (lane * 8 + 256 * j < cols) {
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        v[j][i] -= mean;                                   // x - mean, kept for the output pass
                        sq = fmaf(v[j][i], v[j][i], sq);
                    }
                }
        } else {
            for (int c = lane * 8; c < cols; c += 256) {
                ln_load8<T>(row + c, v[0]);
#pragma unroll
                for (int i = 0; i < 8; i++) sq = fmaf(v[0][i] - mean, v[0][i] - mean, sq);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        const float rstd = rsqrtf(sq * inv_n + eps);
        // d = x - mean -> ((d * rstd) * gamma + beta) * (1 / scale) -> eight e4m3 codes, one 8-byte store
        auto emit = [&](const float (&d)[8], int c) {
            float g[8], b[8], y[8];
            if (gamma) ln_load8<float>(gamma + c, g);
            if (beta) ln_load8<float>(beta + c, b);
#pragma unroll
            for (int i = 0; i < 8; i++) y[i] = fmaf(d[i] * rstd, gamma ? g[i] : 1.0f, beta ? b[i] : 0.0f) * inv;
            const uint32_t lo = static_cast<uint32_t>(sl8::pack_e4m3x2(y[0], y[1])) | (static_cast<uint32_t>(sl8::pack_e4m3x2(y[2], y[3])) << 16);
            const uint32_t hi = static_cast<uint32_t>(sl8::pack_e4m3x2(y[4], y[5])) | (static_cast<uint32_t>(sl8::pack_e4m3x2(y[6], y[7])) << 16);
            *reinterpret_cast<uint2*>(out + r * ld_out + c) = make_uint2(lo, hi);
        };
        if constexpr (CHUNKS > 0) {
#pragma unroll
            for (int j = 0; j < NC; j++)
                if (lane * 8 + 256 * j < cols) emit(v[j], lane * 8 + 256 * j);
        } else {
            for (int c = lane * 8; c < cols; c += 256) {
                ln_load8<T>(row + c, v[0]);
#pragma unroll
                for (int i = 0; i < 8; i++) v[0][i] -= mean;
                emit(v[0], c);
            }
        }
    }
}

template <typename T>
cudaError_t launch_layernorm(int grid, cudaStream_t s, const T* x, long long rows, int cols, long long ld, const float* gamma,
                      const float* beta, float eps, const float* scale, uint8_t* out, long long ld_out) {
    if (cols <= 1280) return sl8_launch_chained(layernorm_quantize_kernel<T, 5>, grid, 256, 0, s, x, rows, cols, ld, gamma, beta, eps, scale, out, ld_out);
    if (cols <= 2048) return sl8_launch_chained(layernorm_quantize_kernel<T, 8>, grid, 256, 0, s, x, rows, cols, ld, gamma, beta, eps, scale, out, ld_out);
    return sl8_launch_chained(layernorm_quantize_kernel<T, 0>, grid, 256, 0, s, x, rows, cols, ld, gamma, beta, eps, scale, out, ld_out);
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
    const int grid = prep_grid(h, rows * 32);            // one warp per row, eight warps per block
    cudaError_t e;
    if (dtype == SL8_DT_F32)
        e = launch_layernorm<float>(grid, s, static_cast<const float*>(x), rows, cols, ld, gamma, beta, eps, scale, static_cast<uint8_t*>(out), ld_out);
    else
        e = launch_layernorm<__nv_bfloat16>(grid, s, static_cast<const __nv_bfloat16*>(x), rows, cols, ld, gamma, beta, eps, scale,
                                        static_cast<uint8_t*>(out), ld_out);
    return e == cudaSuccess ? SL8_OK : fail_cuda(h, e, "layernorm kernel launch");
}
