// Bit-exact kernels: the CPU-order gemv (variant gemv_exact8), the GET_ROWS-shaped dequantizer and the
// two-stage argmax of the LM head.
//
// gemv_exact8 reproduces the reference's detail::dot (backends/cpu/kernel_common.h:16-27) on the device: eight
// lanes per W row hold the eight interleaved partial sums, lane j adds the products of elements i = j (mod 8)
// in increasing i with the multiply and the add rounded separately, and the lanes are combined as
// ((a0+a4)+(a1+a5))+((a2+a6)+(a3+a7)) followed by the sequential tail.  Its output is bitwise the CPU backend's.
// It is the acceptance anchor and the autotuner's validation reference, not the fast path: HBM traffic is the
// algorithmic minimum (every weight byte once per token tile) but the per-element unpacking is issue-bound.
#include "internal.h"
#include "quant_dev.cuh"

namespace halo_cuda {

namespace {

constexpr int kExactRowsPerBlock = 32;  // 32 rows x 8 lanes = 256 threads
constexpr int kExactTokens = 4;         // x rows sharing one unpacked weight

template <uint32_t WT>
__global__ void __launch_bounds__(256) gemv_exact8_kernel(const uint8_t* __restrict__ w, uint64_t w_stride,
                                                          const float* __restrict__ x, uint64_t x_stride,
                                                          float* __restrict__ y, uint64_t y_stride, uint32_t rows,
                                                          uint32_t cols, uint32_t n_vec, const float* __restrict__ gate_dt_bias,
                                                          const float* __restrict__ gate_a, uint32_t gate_n_v) {
    const uint32_t lane8 = threadIdx.x & 7u;
    const uint32_t n = blockIdx.x * kExactRowsPerBlock + (threadIdx.x >> 3);
    const uint32_t t0 = blockIdx.y * kExactTokens;
    // Rows past the end still take part in the shuffles below (with a clamped row), they only skip the store.
    const uint32_t nc = n < rows ? n : rows - 1;
    const uint8_t* row = w + uint64_t{nc} * w_stride;
    const float* xr[kExactTokens];
    float acc[kExactTokens];
#pragma unroll
    for (int t = 0; t < kExactTokens; ++t) {
        const uint32_t tt = t0 + t < n_vec ? t0 + t : n_vec - 1;
        xr[t] = reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(x) + uint64_t{tt} * x_stride);
        acc[t] = 0.0f;
    }
    const uint32_t k8 = cols & ~7u;
    for (uint32_t i = lane8; i < k8; i += 8) {
        const float wv = weight_elem<WT>(row, i);
#pragma unroll
        for (int t = 0; t < kExactTokens; ++t) acc[t] = __fadd_rn(acc[t], __fmul_rn(xr[t][i], wv));
    }
#pragma unroll
    for (int t = 0; t < kExactTokens; ++t) {
        float a = acc[t];
        a = __fadd_rn(a, __shfl_xor_sync(0xFFFFFFFFu, a, 4));  // a_j + a_{j+4}
        a = __fadd_rn(a, __shfl_xor_sync(0xFFFFFFFFu, a, 1));  // (a0+a4)+(a1+a5) | (a2+a6)+(a3+a7)
        a = __fadd_rn(a, __shfl_xor_sync(0xFFFFFFFFu, a, 2));
        float tail = 0.0f;
        for (uint32_t i = k8; i < cols; ++i) tail = __fadd_rn(tail, __fmul_rn(xr[t][i], weight_elem<WT>(row, i)));
        if (lane8 == 0 && n < rows && t0 + t < n_vec) {
            float* yr = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(y) + uint64_t{t0 + t} * y_stride);
            yr[n] = gated_value(__fadd_rn(a, tail), n, gate_n_v, gate_dt_bias, gate_a);
        }
    }
}

template <uint32_t WT>
__global__ void __launch_bounds__(256) get_rows_kernel(const uint8_t* __restrict__ table, uint64_t table_stride,
                                                       const int32_t* __restrict__ ids, float* __restrict__ out,
                                                       uint64_t out_stride, uint32_t n_rows, uint32_t cols,
                                                       uint32_t* __restrict__ status) {
    const uint32_t i = blockIdx.y;
    int64_t id = ids != nullptr ? ids[i] : static_cast<int64_t>(i);
    if (id < 0 || id >= static_cast<int64_t>(n_rows)) {
        if (threadIdx.x == 0 && blockIdx.x == 0 && status != nullptr) atomicOr(status, 8u);  // kStatusBadIndex
        return;
    }
    const uint8_t* row = table + static_cast<uint64_t>(id) * table_stride;
    float* o = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(out) + uint64_t{i} * out_stride);
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < cols; e += gridDim.x * blockDim.x) o[e] = weight_elem<WT>(row, e);
}

// ---- GET_ROWS, four elements a lane ---------------------------------------------------------------------------------
// Bound by the fp32 rows it writes (7 - 9 bytes out per byte in).  A lane takes four consecutive quant bytes (Q6_K: four
// positions of a 128-element half, all four of its 32-element runs) and decodes the scales it needs once for the 4 / 8 / 16
// elements these hold, so a warp's stores are whole 128-byte lines of float4.  One element a thread, each with its own scale
// decode and byte loads, ran at issue rate: 2048 rows of 5120 Q4_K elements 46.7 us, in this form 12.7 us (3.8 TB/s).
template <uint32_t WT>
struct RowItem;

template <bool A4>
__device__ __forceinline__ uint32_t ld_word(const uint8_t* p) {  // four bytes at a 4-byte (A4) or 2-byte aligned address
    if constexpr (A4) return __ldg(reinterpret_cast<const uint32_t*>(p));
    const uint16_t* q = reinterpret_cast<const uint16_t*>(p);
    return static_cast<uint32_t>(__ldg(q)) | (static_cast<uint32_t>(__ldg(q + 1)) << 16);
}
__device__ __forceinline__ float4 scaled(uint32_t bytes, int zero, float d) {  // (byte i - zero) * d
    float4 v;
    v.x = __fmul_rn(static_cast<float>(static_cast<int>(bytes & 0xFFu) - zero), d);
    v.y = __fmul_rn(static_cast<float>(static_cast<int>((bytes >> 8) & 0xFFu) - zero), d);
    v.z = __fmul_rn(static_cast<float>(static_cast<int>((bytes >> 16) & 0xFFu) - zero), d);
    v.w = __fmul_rn(static_cast<float>(static_cast<int>(bytes >> 24) - zero), d);
    return v;
}

template <>
struct RowItem<HALO_CUDA_T_Q4_K> {  // bytes 4i .. of a 64-element chunk: four low nibbles, and four high ones 32 elements on
    static constexpr uint32_t kPerBlock = 32, kBlockElems = 256, kAlign = 4, kRuns = 2;
    uint32_t dm, q, code[3];
    __device__ void fetch(const uint8_t* row, uint32_t i) {
        const uint8_t* blk = row + (i >> 5) * 144u;
        dm = ld_word<true>(blk), q = ld_word<true>(blk + 16 + (i & 31u) * 4u);
        code[0] = ld_word<true>(blk + 4), code[1] = ld_word<true>(blk + 8), code[2] = ld_word<true>(blk + 12);
    }
    __device__ static uint32_t first(uint32_t i) { return (i >> 5) * 256u + ((i >> 3) & 3u) * 64u + (i & 7u) * 4u; }
    __device__ float4 run(uint32_t i, int r) const {
        const uint32_t g = (i >> 3) & 3u, sub = 2 * g + r, sh = 8u * (sub & 3u);  // src/tensor/quant.cpp:236-244
        const uint32_t s0 = code[0] >> sh, s1 = code[1] >> sh, s2 = code[2] >> sh;
        const uint32_t sc = sub < 4 ? s0 & 63u : (s2 & 0x0Fu) | (((s0 >> 6) & 3u) << 4);
        const uint32_t mn = sub < 4 ? s1 & 63u : ((s2 >> 4) & 0x0Fu) | (((s1 >> 6) & 3u) << 4);
        const float d1 = __fmul_rn(f16_bits_to_f32(dm & 0xFFFFu), static_cast<float>(sc)), m1 = __fmul_rn(f16_bits_to_f32(dm >> 16), static_cast<float>(mn));
        float4 v = scaled((r ? q >> 4 : q) & 0x0F0F0F0Fu, 0, d1);
        v.x = __fsub_rn(v.x, m1), v.y = __fsub_rn(v.y, m1), v.z = __fsub_rn(v.z, m1), v.w = __fsub_rn(v.w, m1);
        return v;
    }
    __device__ static uint32_t at(int r) { return 32u * r; }
};
template <>
struct RowItem<HALO_CUDA_T_Q6_K> {
    static constexpr uint32_t kPerBlock = 16, kBlockElems = 256, kAlign = 2, kRuns = 4;
    uint32_t qa, qb, qh, d;
    int8_t sc[4];
    __device__ void fetch(const uint8_t* row, uint32_t i) {
        const uint32_t half = (i >> 3) & 1u, p = i & 7u;
        const uint8_t* blk = row + (i >> 4) * 210u;
        qa = ld_word<false>(blk + half * 64u + 4 * p), qb = ld_word<false>(blk + half * 64u + 32u + 4 * p), qh = ld_word<false>(blk + 128u + half * 32u + 4 * p);
        d = __ldg(reinterpret_cast<const uint16_t*>(blk + 208));
        const uint8_t* s = blk + 192 + half * 8u + (p >> 2);
#pragma unroll
        for (int r = 0; r < 4; ++r) sc[r] = static_cast<int8_t>(__ldg(s + 2 * r));
    }
    __device__ static uint32_t first(uint32_t i) { return (i >> 4) * 256u + ((i >> 3) & 1u) * 128u + (i & 7u) * 4u; }
    __device__ float4 run(uint32_t, int r) const {
        const uint32_t lo = (r & 1) ? qb : qa, nib = ((r & 2) ? lo >> 4 : lo) & 0x0F0F0F0Fu;
        return scaled(nib | (((qh >> (2 * r)) & 0x03030303u) << 4), 32, __fmul_rn(f16_bits_to_f32(d), static_cast<float>(sc[r])));
    }
    __device__ static uint32_t at(int r) { return 32u * r; }
};
template <>
struct RowItem<HALO_CUDA_T_Q8_0> {
    static constexpr uint32_t kPerBlock = 8, kBlockElems = 32, kAlign = 2, kRuns = 1;
    uint32_t q, d;
    __device__ void fetch(const uint8_t* row, uint32_t i) {
        const uint8_t* blk = row + (i >> 3) * 34u;
        q = ld_word<false>(blk + 2 + (i & 7u) * 4u), d = __ldg(reinterpret_cast<const uint16_t*>(blk));
    }
    __device__ static uint32_t first(uint32_t i) { return i * 4u; }
    __device__ float4 run(uint32_t, int) const { return scaled(q ^ 0x80808080u, 128, f16_bits_to_f32(d)); }
    __device__ static uint32_t at(int) { return 0u; }
};
template <>
struct RowItem<HALO_CUDA_T_Q4_0> {
    static constexpr uint32_t kPerBlock = 4, kBlockElems = 32, kAlign = 2, kRuns = 2;
    uint32_t q, d;
    __device__ void fetch(const uint8_t* row, uint32_t i) {
        const uint8_t* blk = row + (i >> 2) * 18u;
        q = ld_word<false>(blk + 2 + (i & 3u) * 4u), d = __ldg(reinterpret_cast<const uint16_t*>(blk));
    }
    __device__ static uint32_t first(uint32_t i) { return (i >> 2) * 32u + (i & 3u) * 4u; }
    __device__ float4 run(uint32_t, int r) const { return scaled((r ? q >> 4 : q) & 0x0F0F0F0Fu, 8, f16_bits_to_f32(d)); }
    __device__ static uint32_t at(int r) { return 16u * r; }
};

/// kRowItems: items a thread requests together -- two where there are many, one where the time is a thread's own instructions (one row of
/// 8192 Q6_K elements 2.41 us with two, 1.58 with one; 55 rows of 8192 Q8_0 elements 1.98 with two, 2.24 with one).
template <uint32_t WT, uint32_t kRowItems>
__global__ void __launch_bounds__(256) get_rows_wide_kernel(const uint8_t* __restrict__ table, uint64_t table_stride, const int32_t* __restrict__ ids,
                                                            float* __restrict__ out, uint64_t out_stride, uint32_t n_rows, uint32_t cols,
                                                            uint32_t* __restrict__ status) {
    using I = RowItem<WT>;
    const uint32_t i = blockIdx.y;
    const int64_t id = ids != nullptr ? ids[i] : static_cast<int64_t>(i);
    if (id < 0 || id >= static_cast<int64_t>(n_rows)) {
        if (threadIdx.x == 0 && blockIdx.x == 0 && status != nullptr) atomicOr(status, 8u);  // kStatusBadIndex
        return;
    }
    const uint8_t* row = table + static_cast<uint64_t>(id) * table_stride;
    float* o = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(out) + uint64_t{i} * out_stride);
    const uint32_t items = cols / I::kBlockElems * I::kPerBlock, it0 = blockIdx.x * blockDim.x * kRowItems + threadIdx.x;
    I v[kRowItems];
#pragma unroll
    for (uint32_t u = 0; u < kRowItems; ++u)
        if (it0 + u * blockDim.x < items) v[u].fetch(row, it0 + u * blockDim.x);
#pragma unroll
    for (uint32_t u = 0; u < kRowItems; ++u) {
        const uint32_t it = it0 + u * blockDim.x;
        if (it >= items) break;
        float* dst = o + I::first(it);
#pragma unroll
        for (int r = 0; r < static_cast<int>(I::kRuns); ++r) *reinterpret_cast<float4*>(dst + I::at(r)) = v[u].run(it, r);
    }
}

// ---- argmax ---------------------------------------------------------------------------------------------------
// "Larger value first, then lower index" is a strict total order (backends/cpu/matmul.cpp:19-22), so any reduction
// tree returns the index a sequential scan returns.  NaN is never ordered: it only raises the vector's flag.
struct ArgPart {
    float value;
    uint32_t index;  // 0xFFFFFFFF = no candidate
    uint32_t nan;
    uint32_t pad;
};
constexpr uint32_t kNoIndex = 0xFFFFFFFFu;
constexpr int kArgmaxThreads = 256;
constexpr uint32_t kArgmaxChunk = 8192;  // logits per first-stage block

__device__ __forceinline__ bool ranks_before(float va, uint32_t ia, float vb, uint32_t ib) {
    if (ia == kNoIndex) return false;
    if (ib == kNoIndex) return true;
    return va > vb || (va == vb && ia < ib);
}

__device__ __forceinline__ void block_reduce_part(float& v, uint32_t& idx, uint32_t& nan) {
    __shared__ float sv[kArgmaxThreads / 32];
    __shared__ uint32_t si[kArgmaxThreads / 32], sn[kArgmaxThreads / 32];
    for (int off = 16; off > 0; off >>= 1) {
        const float ov = __shfl_xor_sync(0xFFFFFFFFu, v, off);
        const uint32_t oi = __shfl_xor_sync(0xFFFFFFFFu, idx, off);
        nan |= __shfl_xor_sync(0xFFFFFFFFu, nan, off);
        if (ranks_before(ov, oi, v, idx)) {
            v = ov;
            idx = oi;
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        sv[warp] = v;
        si[warp] = idx;
        sn[warp] = nan;
    }
    __syncthreads();
    if (warp == 0) {
        v = lane < kArgmaxThreads / 32 ? sv[lane] : 0.0f;
        idx = lane < kArgmaxThreads / 32 ? si[lane] : kNoIndex;
        nan = lane < kArgmaxThreads / 32 ? sn[lane] : 0u;
        for (int off = 4; off > 0; off >>= 1) {
            const float ov = __shfl_xor_sync(0xFFFFFFFFu, v, off);
            const uint32_t oi = __shfl_xor_sync(0xFFFFFFFFu, idx, off);
            nan |= __shfl_xor_sync(0xFFFFFFFFu, nan, off);
            if (ranks_before(ov, oi, v, idx)) {
                v = ov;
                idx = oi;
            }
        }
    }
}

__global__ void __launch_bounds__(kArgmaxThreads) argmax_stage1(const float* __restrict__ logits, uint64_t stride, uint32_t n,
                                                                uint32_t limit, ArgPart* __restrict__ parts) {
    asm volatile("griddepcontrol.launch_dependents;");  // the kernel behind may start its prologue; the logits are the matmul's before
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t t = blockIdx.y;
    const float* row = logits + uint64_t{t} * stride;
    const uint32_t begin = blockIdx.x * kArgmaxChunk;
    const uint32_t end = min(n, begin + kArgmaxChunk);
    float v = 0.0f;
    uint32_t idx = kNoIndex, nan = 0;
    auto take = [&](float f, uint32_t c) {
        if (f != f) {
            nan = 1;
        } else if (c < limit && ranks_before(f, c, v, idx)) {
            v = f;
            idx = c;
        }
    };
    if (end - begin == kArgmaxChunk && (reinterpret_cast<uintptr_t>(row) & 15u) == 0) {
        // A whole aligned chunk: the thread's eight 16-byte loads are all in flight before the first is looked at (one 4-byte load at a
        // time left 304 blocks waiting out 32 latencies: 16 rows of 151936 logits 9.4 us).
        constexpr uint32_t kQuads = kArgmaxChunk / 4 / kArgmaxThreads;
        float4 f[kQuads];
#pragma unroll
        for (uint32_t u = 0; u < kQuads; ++u) f[u] = __ldcg(reinterpret_cast<const float4*>(row + begin) + u * kArgmaxThreads + threadIdx.x);
#pragma unroll
        for (uint32_t u = 0; u < kQuads; ++u) {
            const uint32_t c = begin + 4u * (u * kArgmaxThreads + threadIdx.x);
            take(f[u].x, c), take(f[u].y, c + 1), take(f[u].z, c + 2), take(f[u].w, c + 3);
        }
    } else {
#pragma unroll 8
        for (uint32_t c = begin + threadIdx.x; c < end; c += kArgmaxThreads) take(row[c], c);
    }
    block_reduce_part(v, idx, nan);
    if (threadIdx.x == 0) parts[uint64_t{t} * gridDim.x + blockIdx.x] = {v, idx, nan, 0u};
}

__global__ void __launch_bounds__(kArgmaxThreads) argmax_stage2(const ArgPart* __restrict__ parts, uint32_t n_parts, uint32_t row_offset,
                                                                uint32_t* __restrict__ result, int32_t* __restrict__ ids) {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t t = blockIdx.x;
    float v = 0.0f;
    uint32_t idx = kNoIndex, nan = 0;
    for (uint32_t p = threadIdx.x; p < n_parts; p += kArgmaxThreads) {
        const ArgPart a = parts[uint64_t{t} * n_parts + p];
        nan |= a.nan;
        if (ranks_before(a.value, a.index, v, idx)) {
            v = a.value;
            idx = a.index;
        }
    }
    block_reduce_part(v, idx, nan);
    if (threadIdx.x == 0) {
        // {index, value bits, nan}: a poisoned vector reports {-1, quiet NaN, 1} and the dense id 0
        // (src/backend/cpu_backend.cpp:751-758, 825-833).
        const bool poisoned = nan != 0;
        const uint32_t out_idx = poisoned || idx == kNoIndex ? kNoIndex : idx + row_offset;
        result[3 * t + 0] = out_idx;
        result[3 * t + 1] = poisoned ? 0x7FC00000u : __float_as_uint(v);
        result[3 * t + 2] = poisoned ? 1u : 0u;
        if (ids != nullptr) ids[t] = out_idx == kNoIndex ? 0 : static_cast<int32_t>(out_idx);
    }
}

template <uint32_t WT>
int launch_exact_t(const GemvCall& c, cudaStream_t s) {
    const dim3 grid((c.rows + kExactRowsPerBlock - 1) / kExactRowsPerBlock, (c.n_vec + kExactTokens - 1) / kExactTokens);
    gemv_exact8_kernel<WT><<<grid, 256, 0, s>>>(c.w, c.w_stride, c.x, c.x_stride, c.y, c.y_stride, c.rows, c.cols, c.n_vec, c.gate_dt_bias,
                                                c.gate_a, c.gate_n_v);
    HC_CUDA(cudaGetLastError());
    return 0;
}

constexpr uint64_t kManyRowItems = 148 * 256;  // eight warps of items an SM: where the two forms cross for all four formats

/// The wide form where its loads and stores are aligned (any GGUF tensor in a dense table with 16-byte aligned output rows), the
/// element form for everything else (F32 tables, odd addresses, unaligned outputs).
template <uint32_t WT>
int launch_get_rows_t(const HaloCudaGetRows& a, uint64_t ts, uint64_t os, cudaStream_t s) {
    const uint8_t* table = static_cast<const uint8_t*>(a.table);
    if constexpr (WT != HALO_CUDA_T_F32) {
        using I = RowItem<WT>;
        if (reinterpret_cast<uintptr_t>(table) % I::kAlign == 0 && ts % I::kAlign == 0 && reinterpret_cast<uintptr_t>(a.out) % 16 == 0 && os % 16 == 0) {
            const uint32_t items = a.cols / I::kBlockElems * I::kPerBlock;
            if (uint64_t{items} * a.n_ids < kManyRowItems) {
                get_rows_wide_kernel<WT, 1><<<dim3((items + 63u) / 64u, a.n_ids), 64, 0, s>>>(table, ts, a.ids, a.out, os, a.n_rows, a.cols, a.status);
            } else {
                const uint32_t threads = items < 256u ? 64u : 256u;
                get_rows_wide_kernel<WT, 2><<<dim3((items + threads * 2u - 1) / (threads * 2u), a.n_ids), threads, 0, s>>>(
                    table, ts, a.ids, a.out, os, a.n_rows, a.cols, a.status);
            }
            HC_CUDA(cudaGetLastError());
            return 0;
        }
    }
    const uint32_t bx = min((a.cols + 255u) / 256u, 64u);
    get_rows_kernel<WT><<<dim3(bx, a.n_ids), 256, 0, s>>>(table, ts, a.ids, a.out, os, a.n_rows, a.cols, a.status);
    HC_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace

int launch_gemv_exact8(const GemvCall& c, cudaStream_t s) {
    if (c.n_vec > 65535u * kExactTokens) return fail(HALO_CUDA_E_UNSUPPORTED, "MATMUL: n_vec %u exceeds the launch limit", c.n_vec);
    switch (c.wtype) {
        case HALO_CUDA_T_F32: return launch_exact_t<HALO_CUDA_T_F32>(c, s);
        case HALO_CUDA_T_Q4_0: return launch_exact_t<HALO_CUDA_T_Q4_0>(c, s);
        case HALO_CUDA_T_Q8_0: return launch_exact_t<HALO_CUDA_T_Q8_0>(c, s);
        case HALO_CUDA_T_Q4_K: return launch_exact_t<HALO_CUDA_T_Q4_K>(c, s);
        case HALO_CUDA_T_Q6_K: return launch_exact_t<HALO_CUDA_T_Q6_K>(c, s);
        default: return fail(HALO_CUDA_E_UNSUPPORTED, "MATMUL: weight type id %u", c.wtype);
    }
}

int launch_get_rows(const HaloCudaGetRows& a, uint64_t /*row_bytes*/, uint64_t ts, uint64_t os, cudaStream_t s) {
    if (a.n_ids > 65535u) return fail(HALO_CUDA_E_UNSUPPORTED, "GET_ROWS: n_ids %u exceeds the launch limit", a.n_ids);
    switch (a.type) {
        case HALO_CUDA_T_F32: return launch_get_rows_t<HALO_CUDA_T_F32>(a, ts, os, s);
        case HALO_CUDA_T_Q4_0: return launch_get_rows_t<HALO_CUDA_T_Q4_0>(a, ts, os, s);
        case HALO_CUDA_T_Q8_0: return launch_get_rows_t<HALO_CUDA_T_Q8_0>(a, ts, os, s);
        case HALO_CUDA_T_Q4_K: return launch_get_rows_t<HALO_CUDA_T_Q4_K>(a, ts, os, s);
        case HALO_CUDA_T_Q6_K: return launch_get_rows_t<HALO_CUDA_T_Q6_K>(a, ts, os, s);
        default: return fail(HALO_CUDA_E_UNSUPPORTED, "GET_ROWS: type id %u", a.type);
    }
}

uint64_t argmax_scratch_bytes(uint32_t n, uint32_t n_vec) {
    const uint64_t parts = (uint64_t{n} + kArgmaxChunk - 1) / kArgmaxChunk;
    return (parts == 0 ? 1 : parts) * n_vec * sizeof(ArgPart);
}

int launch_argmax(const float* logits, uint64_t stride_elems, uint32_t n, uint32_t n_vec, uint32_t valid, uint32_t row_offset,
                  uint32_t* result, int32_t* ids, void* scratch, cudaStream_t s) {
    if (n_vec > 65535u) return fail(HALO_CUDA_E_UNSUPPORTED, "LM_HEAD: n_vec %u exceeds the launch limit", n_vec);
    const uint32_t parts = (n + kArgmaxChunk - 1) / kArgmaxChunk;
    const uint32_t limit = valid > 0 && valid < n ? valid : n;
    ArgPart* p = static_cast<ArgPart*>(scratch);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(parts, n_vec), cfg.blockDim = dim3(kArgmaxThreads), cfg.stream = s, cfg.attrs = attr, cfg.numAttrs = 1;
    if (parts != 0) HC_CUDA(cudaLaunchKernelEx(&cfg, argmax_stage1, logits, stride_elems, n, limit, p));
    cfg.gridDim = dim3(n_vec);
    HC_CUDA(cudaLaunchKernelEx(&cfg, argmax_stage2, static_cast<const ArgPart*>(p), parts, row_offset, result, ids));
    return 0;
}

}  // namespace halo_cuda
