// gemv_mma_r: tensor-core skinny kernel for Q6_K, Q8_0 and Q4_0 weights in the REPACKED row layout of halo_cuda_repack.
//
// Why a repacked layout: the GGUF blocks of these formats are 210 / 34 / 18 bytes, so their rows cannot be fetched by
// the copy engine (tile coordinates and row pitches must be multiples of 16 bytes) and their quant words are only
// 2-byte aligned.  The reference makes the same move for its Vulkan matvecs (include/halo/tensor/repack.h:11-36; the
// layout is a kernel variant, include/halo/backend/backend.h:178-183).  Repacking is a pure byte permutation of each
// 256-weight group (plus padding): every quant code and scale is bit-identical, which the tests check by unpacking the
// repacked rows back.  Layout of one group of 256 weights (rows are sequences of groups):
//   Q4_0r  144 B: d[8] fp16 | for chunk c<2, thread t<4: the quant word (bytes 4t..4t+3) of blocks 4c..4c+3
//   Q8_0r  272 B: d[8] fp16 | for chunk c<4, thread t<4: words (block 2c, k-step 0/1), (block 2c+1, k-step 0/1);
//                 a k-step is 16 elements, the word holds elements 16*step + 4t .. +3
//   Q6_Kr  224 B: scales[16] int8 | d fp16, 14 B pad | for half n<2, thread t<4: ql words (b, lh) = bytes
//                 64n + 32b + 16lh + 4t..+3 | for thread t<4: qh words (n, lh) = bytes 32n + 16lh + 4t..+3
// i.e. the four words one thread needs next to each other, so a fragment is one 16-byte shared-memory load.
//
// Arithmetic (the same scheme as gemv_mma_f16x2): A holds the unsigned quant code as an fp16 subnormal (code * 2^-24,
// exact), B holds x as fp16 hi + lo columns, one m16n8k16 MMA per 16 elements.  Every scale group (a 32-element block,
// or 16 elements of Q6_K) gets a fresh fp32 accumulator, and the group's scale and zero point are applied in fp32:
//     y += scale_g * (acc_g - zero * sum_g(x))        zero = 8 / 128 / 32, sum_g(x) in fp32 from the staging pass.
// Rows do not depend on the batch size; results are bounded against the CPU backend, not bitwise.
//
// Roofline: HBM.  Algorithmic bytes = rows * row_bytes + 4 * n_vec * cols + 4 * n_vec * rows.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "internal.h"
#include "mma_common.cuh"

namespace halo_cuda {
namespace {

using namespace mma;

// ---- repack: raw GGUF rows -> grouped rows (one thread per 32-bit output word) ---------------------------------------------
__device__ __forceinline__ uint32_t ld_u32_bytes(const uint8_t* p) {
    return static_cast<uint32_t>(p[0]) | (static_cast<uint32_t>(p[1]) << 8) | (static_cast<uint32_t>(p[2]) << 16) | (static_cast<uint32_t>(p[3]) << 24);
}

/// Word `wi` of repacked group `grp` of a row whose raw bytes start at `raw` (any alignment).
__device__ uint32_t repack_word(uint32_t wtype, const uint8_t* raw, uint32_t grp, uint32_t wi) {
    if (wtype == HALO_CUDA_T_Q4_0) {
        const uint8_t* g = raw + grp * 144u;  // 8 blocks of 18 bytes
        if (wi < 4) return static_cast<uint32_t>(g[(2 * wi) * 18]) | (static_cast<uint32_t>(g[(2 * wi) * 18 + 1]) << 8) |
                           (static_cast<uint32_t>(g[(2 * wi + 1) * 18]) << 16) | (static_cast<uint32_t>(g[(2 * wi + 1) * 18 + 1]) << 24);
        const uint32_t k = wi - 4, c = k >> 4, t = (k >> 2) & 3u, j = k & 3u;  // chunk, thread, block inside the chunk
        return ld_u32_bytes(g + (4 * c + j) * 18 + 2 + 4 * t);
    }
    if (wtype == HALO_CUDA_T_Q8_0) {
        const uint8_t* g = raw + grp * 272u;  // 8 blocks of 34 bytes
        if (wi < 4) return static_cast<uint32_t>(g[(2 * wi) * 34]) | (static_cast<uint32_t>(g[(2 * wi) * 34 + 1]) << 8) |
                           (static_cast<uint32_t>(g[(2 * wi + 1) * 34]) << 16) | (static_cast<uint32_t>(g[(2 * wi + 1) * 34 + 1]) << 24);
        const uint32_t k = wi - 4, c = k >> 4, t = (k >> 2) & 3u, j = k & 3u;  // j = (block parity) * 2 + k-step
        return ld_u32_bytes(g + (2 * c + (j >> 1)) * 34 + 2 + 16 * (j & 1u) + 4 * t);
    }
    // Q6_K: 210 raw bytes -> 224
    const uint8_t* g = raw + grp * 210u;
    if (wi < 4) return ld_u32_bytes(g + 192 + 4 * wi);                                                                  // scales
    if (wi == 4) return static_cast<uint32_t>(g[208]) | (static_cast<uint32_t>(g[209]) << 8);                          // d
    if (wi < 8) return 0u;                                                                                              // pad
    if (wi < 40) {
        const uint32_t k = wi - 8, n = k >> 4, t = (k >> 2) & 3u, j = k & 3u;  // j = b * 2 + lh
        return ld_u32_bytes(g + 64 * n + 32 * (j >> 1) + 16 * (j & 1u) + 4 * t);
    }
    const uint32_t k = wi - 40, t = k >> 2, j = k & 3u;  // j = n * 2 + lh
    return ld_u32_bytes(g + 128 + 32 * (j >> 1) + 16 * (j & 1u) + 4 * t);
}

// The tiled form: a block brings a run of whole groups into shared memory with 16-byte loads and writes them out as 16-byte words put
// together from 2-byte reads.  Bound by HBM (1 byte read and 1 - 1.07 written per raw byte).  A thread per output word that gathered its
// bytes from global memory ran at load-instruction rate: Q6_K 5120 x 17408 108.6 us, in this form 34.3 us (4.5 TB/s).
constexpr uint32_t kRepackThreads = 256;

__device__ __forceinline__ uint32_t lds_u32_a2(const uint8_t* p) {
    const uint16_t* q = reinterpret_cast<const uint16_t*>(p);
    return static_cast<uint32_t>(q[0]) | (static_cast<uint32_t>(q[1]) << 16);
}

template <uint32_t WT>
struct Repack;
template <>
struct Repack<HALO_CUDA_T_Q4_0> {
    static constexpr uint32_t kRaw = 144, kPacked = 144, kTile = 64;  // bytes of a raw and a repacked group, groups per block
    __device__ static uint4 quad(const uint8_t* g, uint32_t qi) {    // 16-byte word qi of the repacked group
        uint32_t w[4];
        if (qi == 0) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                w[j] = *reinterpret_cast<const uint16_t*>(g + 2 * j * 18) | (static_cast<uint32_t>(*reinterpret_cast<const uint16_t*>(g + (2 * j + 1) * 18)) << 16);
        } else {
            const uint32_t c = (qi - 1) >> 2, t = (qi - 1) & 3u;
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = lds_u32_a2(g + (4 * c + j) * 18 + 2 + 4 * t);
        }
        return make_uint4(w[0], w[1], w[2], w[3]);
    }
};
template <>
struct Repack<HALO_CUDA_T_Q8_0> {
    static constexpr uint32_t kRaw = 272, kPacked = 272, kTile = 32;
    __device__ static uint4 quad(const uint8_t* g, uint32_t qi) {
        uint32_t w[4];
        if (qi == 0) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                w[j] = *reinterpret_cast<const uint16_t*>(g + 2 * j * 34) | (static_cast<uint32_t>(*reinterpret_cast<const uint16_t*>(g + (2 * j + 1) * 34)) << 16);
        } else {
            const uint32_t c = (qi - 1) >> 2, t = (qi - 1) & 3u;
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = lds_u32_a2(g + (2 * c + (j >> 1)) * 34 + 2 + 16 * (j & 1) + 4 * t);
        }
        return make_uint4(w[0], w[1], w[2], w[3]);
    }
};
template <>
struct Repack<HALO_CUDA_T_Q6_K> {
    static constexpr uint32_t kRaw = 210, kPacked = 224, kTile = 40;
    __device__ static uint4 quad(const uint8_t* g, uint32_t qi) {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (qi == 0) w[j] = lds_u32_a2(g + 192 + 4 * j);                                                       // scales
            else if (qi == 1) w[j] = j == 0 ? *reinterpret_cast<const uint16_t*>(g + 208) : 0u;                    // d, pad
            else if (qi < 10) w[j] = lds_u32_a2(g + 64 * ((qi - 2) >> 2) + 32 * (j >> 1) + 16 * (j & 1) + 4 * ((qi - 2) & 3u));
            else w[j] = lds_u32_a2(g + 128 + 32 * (j >> 1) + 16 * (j & 1) + 4 * (qi - 10));
        }
        return make_uint4(w[0], w[1], w[2], w[3]);
    }
};

/// grid (blocks of kTile groups, rows): src rows 2-byte aligned, dst rows 16-byte aligned.  A dense matrix is passed as one row.
template <uint32_t WT>
__global__ void __launch_bounds__(kRepackThreads) repack_tiled_kernel(const uint8_t* __restrict__ src, uint64_t src_stride, uint8_t* __restrict__ dst,
                                                                      uint64_t dst_stride, uint64_t groups) {
    using R = Repack<WT>;
    __shared__ __align__(16) uint8_t buf[R::kTile * R::kRaw + 32];
    const uint64_t g0 = uint64_t{blockIdx.x} * R::kTile;
    const uint32_t n = static_cast<uint32_t>(groups - g0 < R::kTile ? groups - g0 : R::kTile), bytes = n * R::kRaw;
    const uint8_t* from = src + uint64_t{blockIdx.y} * src_stride + g0 * R::kRaw;
    const uint32_t lead = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(from) & 15u);  // the buffer keeps the source's phase
    const uint32_t head = min(bytes, (16u - lead) & 15u), quads = (bytes - head) / 16u, tail = bytes - head - quads * 16u;
    uint8_t* b = buf + lead;
    for (uint32_t i = threadIdx.x; i < quads; i += kRepackThreads)
        *reinterpret_cast<uint4*>(b + head + 16u * i) = __ldg(reinterpret_cast<const uint4*>(from + head) + i);
    if (threadIdx.x < (head + tail) / 2u) {  // the ragged ends, two bytes a thread
        const uint32_t at = 2u * threadIdx.x < head ? 2u * threadIdx.x : bytes - tail + 2u * threadIdx.x - head;
        *reinterpret_cast<uint16_t*>(b + at) = __ldg(reinterpret_cast<const uint16_t*>(from + at));
    }
    __syncthreads();
    uint4* to = reinterpret_cast<uint4*>(dst + uint64_t{blockIdx.y} * dst_stride + g0 * R::kPacked);
    constexpr uint32_t kQuads = R::kPacked / 16u;
    for (uint32_t i = threadIdx.x; i < n * kQuads; i += kRepackThreads) to[i] = R::quad(b + i / kQuads * R::kRaw, i % kQuads);
}

template <uint32_t WT>
int launch_repack_tiled(const uint8_t* src, uint64_t src_stride, uint8_t* dst, uint64_t dst_stride, uint64_t rows, uint64_t groups, cudaStream_t s) {
    using R = Repack<WT>;
    if (src_stride == groups * R::kRaw && dst_stride == groups * R::kPacked) groups *= rows, rows = 1;
    const uint64_t bx = (groups + R::kTile - 1) / R::kTile;
    for (uint64_t r0 = 0; r0 < rows; r0 += 65535u) {
        const uint32_t n = static_cast<uint32_t>(rows - r0 < 65535u ? rows - r0 : 65535u);
        repack_tiled_kernel<WT><<<dim3(static_cast<uint32_t>(bx), n), kRepackThreads, 0, s>>>(src + r0 * src_stride, src_stride, dst + r0 * dst_stride, dst_stride, groups);
    }
    HC_CUDA(cudaGetLastError());
    return 0;
}

__global__ void __launch_bounds__(256) repack_kernel(uint32_t wtype, const uint8_t* __restrict__ src, uint64_t src_stride, uint32_t* __restrict__ dst,
                                                     uint64_t dst_stride, uint32_t rows, uint32_t groups, uint32_t words_per_group) {
    const uint64_t total = uint64_t{rows} * groups * words_per_group;
    for (uint64_t i = uint64_t{blockIdx.x} * blockDim.x + threadIdx.x; i < total; i += uint64_t{gridDim.x} * blockDim.x) {
        const uint32_t wi = static_cast<uint32_t>(i % words_per_group);
        const uint64_t gr = i / words_per_group;
        const uint32_t grp = static_cast<uint32_t>(gr % groups), r = static_cast<uint32_t>(gr / groups);
        reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(dst) + uint64_t{r} * dst_stride)[grp * words_per_group + wi] =
            repack_word(wtype, src + uint64_t{r} * src_stride, grp, wi);
    }
}

uint32_t group_bytes(uint32_t wtype) {
    return wtype == HALO_CUDA_T_Q4_0 ? 144u : wtype == HALO_CUDA_T_Q8_0 ? 272u : wtype == HALO_CUDA_T_Q6_K ? 224u : 0u;
}

}  // namespace

uint64_t repacked_row_bytes(uint32_t wtype, uint64_t cols) { return cols / 256u * group_bytes(wtype); }

bool gemv_mma_r_supports(const GemvCall& c) {
    if (group_bytes(c.wtype) == 0 || c.cols == 0 || c.cols % 256u != 0) return false;
    if (reinterpret_cast<uintptr_t>(c.w) % 16 != 0 || c.w_stride % 16 != 0) return false;  // tensor-map base and pitch
    if (reinterpret_cast<uintptr_t>(c.x) % 16 != 0 || c.x_stride % 16 != 0) return false;  // float4 reads of x
    return (c.flags & HALO_CUDA_GEMV_FLAG_NO_SCRATCH) == 0;  // the kernels keep partial sums and staged x in context scratch
}

int launch_gemv_mma_r(HaloCudaCtx* ctx, const GemvCall& c, cudaStream_t s) {
    switch (c.wtype) {
        case HALO_CUDA_T_Q4_0: return launch_gemv_sk_q40r(ctx, c, s);
        case HALO_CUDA_T_Q8_0: return launch_gemv_sk_q80r(ctx, c, s);
        case HALO_CUDA_T_Q6_K: return launch_gemv_sk_q6kr(ctx, c, s);
        default: return fail(HALO_CUDA_E_UNSUPPORTED, "MATMUL: gemv_mma_r takes repacked Q4_0 / Q8_0 / Q6_K weights");
    }
}

int launch_repack(uint32_t wtype, const void* src, uint64_t src_stride, void* dst, uint64_t dst_stride, uint32_t rows, uint32_t cols, cudaStream_t s) {
    const uint32_t groups = cols / 256u, words = group_bytes(wtype) / 4u;
    const uint8_t* from = static_cast<const uint8_t*>(src);
    uint8_t* to = static_cast<uint8_t*>(dst);
    // Two-byte aligned rows (every GGUF tensor) take the tiled form, rows at odd addresses the word-by-word one -- and so do short rows of a
    // strided matrix, of which a tile holds one each: 151936 rows of one / two / four Q4_0 groups 26 / 50 / 100 us by words and 114 / 151 / 175
    // by tiles, of eight 197 and 183; Q8_0 and Q6_K cross between three and five groups, all three at about a kilobyte a row.
    const uint64_t raw_row = uint64_t{groups} * (wtype == HALO_CUDA_T_Q4_0 ? 144u : wtype == HALO_CUDA_T_Q8_0 ? 272u : 210u);
    const bool dense = src_stride == raw_row && dst_stride == uint64_t{groups} * words * 4u;
    if (reinterpret_cast<uintptr_t>(from) % 2 == 0 && src_stride % 2 == 0 && groups != 0 && (dense || rows == 1 || raw_row >= 1024u)) {
        switch (wtype) {
            case HALO_CUDA_T_Q4_0: return launch_repack_tiled<HALO_CUDA_T_Q4_0>(from, src_stride, to, dst_stride, rows, groups, s);
            case HALO_CUDA_T_Q8_0: return launch_repack_tiled<HALO_CUDA_T_Q8_0>(from, src_stride, to, dst_stride, rows, groups, s);
            case HALO_CUDA_T_Q6_K: return launch_repack_tiled<HALO_CUDA_T_Q6_K>(from, src_stride, to, dst_stride, rows, groups, s);
            default: break;
        }
    }
    const uint64_t total = uint64_t{rows} * groups * words;
    if (total == 0) return 0;
    const uint32_t blocks = static_cast<uint32_t>(total / 256 + 1 < 148 * 16 ? total / 256 + 1 : 148 * 16);
    repack_kernel<<<blocks, 256, 0, s>>>(wtype, from, src_stride, static_cast<uint32_t*>(dst), dst_stride, rows, groups, words);
    HC_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace halo_cuda
