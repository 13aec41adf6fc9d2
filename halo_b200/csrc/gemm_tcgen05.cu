// gemm_tcgen05_{f16,bf16}[_r]: the prefill GEMM, Y[M x N] = X[M x K] * dequant(W)[N x K]^T, M >= 64, for raw Q4_K rows and
// (the _r variants) for Q6_K / Q8_0 / Q4_0 rows in the repacked layout of halo_cuda_repack_rows (gemv_mma_grouped.cu).
//
// The reference's own GEMM path rounds x and dequant(W) to fp16 and accumulates in fp32
// (backends/vulkan/shaders/common/matmul_cm_main.glsl:1-6); a caller opts in with GemvArgs::allow_gemm
// (include/halo/backend/backend.h:300-304).  Same numerics here: W is dequantized in fp32 exactly as
// tensor::dequantize_row does ((d*sc)*q - dmin*m, src/tensor/quant.cpp:247-269; (d*s)*(q-32), :302-327; d*q, :143-151;
// d*(q-8), :79-90) and rounded ONCE to the 16-bit type.
//
// Structure: a persistent grid of CTA pairs (clusters of two, one CTA per SM).  A pair's tile is 256 W rows x T tokens, W as the M
// operand of tcgen05.mma.cta_group::2 (128 rows in each CTA), X as its N operand (each CTA holds half of the tokens), fp32
// accumulators in TMEM (lane = W row, column = token).  T is a multiple of 32 up to 256 with two accumulators used in turn, so that a
// tile's epilogue runs under the next tile's MMAs, or a multiple of 64 up to 448 with both accumulators in one tile
// (Q8_0 up to 320, Q6_K up to 384: what leaves room for four stages beside two blocks of quants).
// Warps of a CTA (768 threads):
//   0       TMA: this CTA's half of the 16-bit X tile (64 K elements x T/2 tokens per stage, 128-byte swizzle)
//   1       TMEM allocation; in the leading CTA the tcgen05.mma issue
//   2       TMA: the quantized rows of the W tile, one 256-element block of 128 rows at a time, into a ring of their own
//   4-7     epilogue: tcgen05.ld -> y, a lane per W row, so that every store is 128 consecutive bytes of one token's y
//   8-23    dequantization: warp group j takes the j-th 64 elements of every 256-element block; a thread reads its row's quants from the
//           raw ring and writes the 128-byte swizzled row of the stage's W tile
// Barriers: full (X bytes of both CTAs, the dequant warps of both), empty and accumulator-full (tcgen05.commit to both CTAs),
// accumulator-empty (the epilogue warps of both).  Where the tiles alone do not fill the device, K is split: every split stores its
// partial sums to scratch and a second kernel adds them in split order.
//
// What bounds it: the tensor pipe where T is large (2*M*N*K flops per call), the issue slots of the dequantization (2 - 4 instructions a
// weight) where it is small, HBM below that.  A pair shares the dequantized W: a CTA converts 128 rows for T tokens, and its quants arrive
// by TMA instead of 16-byte gathers from 128 different rows.
//
// Measured against one 256 x 256 tile a CTA with gathered quants: Q4_K 17408 x 5120 at 512 / 2048 tokens 109 -> 74 / 393 -> 268 us
// (1.36 PFLOP/s; 34816 x 5120 1.45, where the power cap holds the clock), Q6_K 5120 x 17408 at 2048 tokens 1070 -> 312 us, Q8_0 and Q4_0
// 17408 x 5120 at 2048 tokens 262 us; at 64 tokens, Q4_0 / Q8_0 / Q4_K / Q6_K 17408 x 5120, 26 / 28 / 31 / 33 us.
//
// The K order inside every group of 8 elements is permuted to (0,2,1,3,4,6,5,7) in BOTH operands -- the cast kernel
// writes X that way -- because that is the order in which masked nibble pairs fall out of a 32-bit word.
//
// Every mbarrier wait is bounded; a role that gives up raises the context error word, and all roles of both CTAs still meet at
// the final barrier so that TMEM is released before the CTAs exit.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>

#include "internal.h"

namespace halo_cuda {
namespace {

constexpr uint32_t kPairRows = 256, kCtaRows = 128, kBK = 64;
constexpr uint32_t kTileW = kCtaRows * kBK * 2;      // dequantized W of a stage: 16 KiB
// A dequant group fills every fourth position of the stage ring and waits for a position's slot by the parity of its last use.  That it
// cannot see the use before the last one as the last (the parities agree) rests on its own previous position: slot p - S was free then, and
// p + 4 - 2S <= p - S holds for S >= 4 only.
constexpr uint32_t kMinStages = 4, kMaxStages = 8, kMaxRaw = 3;
constexpr uint32_t kEpiWarp = 4, kDeqWarp = 8, kDeqGroupWarps = 4, kDeqWarps = 16;
constexpr uint32_t kGemmThreads = (kDeqWarp + kDeqWarps) * 32;
constexpr uint32_t kGemmSmem = 227 * 1024;
constexpr uint32_t kSmemTiles = kGemmSmem - 1024 /*alignment slack*/ - 512 /*barriers*/;
constexpr uint32_t kGemmWaitSpins = 1u << 16;

struct GemmArgs {
    float* y;
    uint64_t y_stride;       // bytes
    uint32_t rows, n_vec, nb;
    uint32_t nt, nacc;       // tokens per accumulator, accumulators per tile
    uint32_t stages, raw_slots;
    uint32_t token_tiles, whole, splits, units;  // units: tiles [0, whole) over all of K, then `splits` shares of K of every further tile
    float* partials;         // splits > 1: [tile - whole][split][CTA of the pair][nacc * nt tokens][128 rows]
    uint32_t* error_word;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_to_leader(uint32_t addr) {  // the same shared-memory offset in the pair's first CTA
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void g_mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void g_mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void g_mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void g_mbar_arrive_cluster(uint32_t bar) {  // a barrier of either CTA of the pair
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool g_mbar_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kGemmWaitSpins; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ bool g_mbar_wait_warp(uint32_t bar, uint32_t parity) {
    return __all_sync(0xFFFFFFFFu, g_mbar_wait(bar, parity));
}
__device__ __forceinline__ void g_tma_2d(uint32_t dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
/// The same copy into this CTA's shared memory, counted on a barrier of the pair's first CTA.
__device__ __forceinline__ void g_tma_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}

// Shared-memory matrix descriptor of a K-major tile with 128-byte rows and 128-byte swizzle: start address / 16,
// leading byte offset (unused for swizzled K-major, 1), stride byte offset 1024 / 16 (one 8-row swizzle atom),
// descriptor version 1 (bits 46-47), layout type 2 = SWIZZLE_128B (bits 61-63).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    return static_cast<uint64_t>((addr & 0x3FFFFu) >> 4) | (uint64_t{1} << 16) | (uint64_t{64} << 32) | (uint64_t{1} << 46) |
           (uint64_t{2} << 61);
}

__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
/// Arrives on the barrier at this offset in both CTAs once the MMAs issued so far have finished.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"(static_cast<uint16_t>(3))
                 : "memory");
}

/// One lane of a converged warp.  The issuing warps run their loops with all lanes and branch on this around the issue alone: under a branch on
/// the lane id the compiler moves every operand of a copy or an MMA to the uniform registers one lane at a time, and an issuer that spent
/// 700 clocks on the four MMAs of a K step was what the whole kernel waited for.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

/// Position in a ring of n slots; the parity flips at every wrap.
struct RingPos {
    uint32_t slot, parity;
    __device__ __forceinline__ void advance(uint32_t by, uint32_t n) {
        slot += by;  // by <= n
        if (slot >= n) slot -= n, parity ^= 1u;
    }
};

/// fp32 -> 16-bit copy of X with the K order of every 8-element group permuted to (0,2,1,3,4,6,5,7).  HBM-bound; a thread has the 64 bytes
/// of two groups in flight.
template <bool BF16>
__global__ void __launch_bounds__(256) cast_x_kernel(const float* __restrict__ x, uint64_t x_stride, uint16_t* __restrict__ out,
                                                     uint32_t n_vec, uint32_t cols) {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t groups = cols / 8, g0 = blockIdx.x * 2u * blockDim.x + threadIdx.x;
    for (uint32_t t = blockIdx.y; t < n_vec; t += gridDim.y) {
        const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const uint8_t*>(x) + uint64_t{t} * x_stride);
        uint4* dst = reinterpret_cast<uint4*>(out + uint64_t{t} * cols);
        float4 a[2], b[2];
#pragma unroll
        for (uint32_t u = 0; u < 2; ++u) {
            const uint32_t g = g0 + u * blockDim.x;
            if (g < groups) a[u] = __ldg(src + 2 * g), b[u] = __ldg(src + 2 * g + 1);
        }
#pragma unroll
        for (uint32_t u = 0; u < 2; ++u) {
            const uint32_t g = g0 + u * blockDim.x;
            if (g >= groups) break;
            const float v[8] = {a[u].x, a[u].z, a[u].y, a[u].w, b[u].x, b[u].z, b[u].y, b[u].w};
            uint32_t p[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if constexpr (BF16) {
                    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
                    p[k] = *reinterpret_cast<const uint32_t*>(&h);
                } else {
                    const __half2 h = __floats2half2_rn(v[2 * k], v[2 * k + 1]);
                    p[k] = *reinterpret_cast<const uint32_t*>(&h);
                }
            }
            dst[g] = make_uint4(p[0], p[1], p[2], p[3]);
        }
    }
}

// ---- dequantization: what a thread does for 64 weights of one row -----------------------------------------------------------------------
// load() reads block row `row` (one 256-element block in shared memory) for K quarter j, fold() depends on every word it read; emit() writes the row's eight 16-byte chunks:
// chunk p holds weights 8p .. 8p+7 of the quarter in the order (0,2,1,3,4,6,5,7), which is how byte pairs (0,2) and (1,3) fall out of a
// masked 32-bit word.
__device__ __forceinline__ uint32_t fold4(const uint4& v) { return v.x ^ v.y ^ v.z ^ v.w; }
template <bool BF16>
__device__ __forceinline__ uint32_t pack2(uint64_t v) {  // two fp32 in a register pair -> one 16-bit pair, rounded once
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    if constexpr (BF16) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&h);
    } else {
        const __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
}
__device__ __forceinline__ uint64_t f32x2(float a, float b) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }
/// A pair of codes in the halves 1024 + u -> the two values u - zero (integers below 2048: exact).
__device__ __forceinline__ __half2 codes(uint32_t biased, uint32_t zero) { return __hsub2(as_half2(biased), as_half2(zero * 0x00010001u + 0x64006400u)); }
__device__ __forceinline__ uint64_t widen(__half2 q) {
    const float2 f = __half22float2(q);
    return f32x2(f.x, f.y);
}
/// scale * q with a scale that is exact in fp16: the product of two fp16 numbers is exact in fp32, so the fp16 multiply rounds the
/// same value once.
template <bool BF16>
__device__ __forceinline__ uint32_t scaled_pair(__half2 q, __half2 d16, uint64_t d32) {
    if constexpr (BF16) return pack2<true>(mul2(d32, widen(q)));
    return as_u32(__hmul2(d16, q));
}
/// Chunk `pos` of a 128-byte swizzled row; `at` is the shared-memory address of the row's chunk 0, whose bits 4-6 hold the row's xor.
__device__ __forceinline__ void store_chunk(uint32_t at, uint32_t pos, const uint4& v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at ^ (pos << 4)), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint32_t bytes02(uint32_t w) { return __byte_perm(w, 0x64646464u, 0x4240); }  // halves 1024 + byte 0, 1024 + byte 2
__device__ __forceinline__ uint32_t bytes13(uint32_t w) { return __byte_perm(w, 0x64646464u, 0x4341); }

struct GemmQ4K {  // raw rows of 144-byte super-blocks: quarter j = sub-blocks 2j (low nibbles) and 2j + 1 (high)
    static constexpr uint32_t kBlock = 144, kPitch = 144;
    static constexpr double kConvertNs = 350.0;  // to convert a stage
    struct Regs {
        uint4 h, q[2];
    };
    __device__ static __forceinline__ uint32_t fold(const Regs& r) { return fold4(r.h) ^ fold4(r.q[0]) ^ fold4(r.q[1]); }
    __device__ static __forceinline__ void load(Regs& r, const uint8_t* row, uint32_t j) {
        r.h = *reinterpret_cast<const uint4*>(row);
        r.q[0] = *reinterpret_cast<const uint4*>(row + 16 + j * 32);
        r.q[1] = *reinterpret_cast<const uint4*>(row + 32 + j * 32);
    }
    template <bool BF16>
    __device__ static __forceinline__ void emit(const Regs& r, uint32_t j, uint32_t at) {
        // 6-bit codes of sub-blocks 2j (low nibbles) and 2j+1 (high nibbles), src/tensor/quant.cpp:236-244
        const uint32_t s0 = r.h.y, s1 = r.h.z, s2 = r.h.w;
        uint32_t sc0, mn0, sc1, mn1;
        if (j < 2) {
            sc0 = (s0 >> (16 * j)) & 63u;       mn0 = (s1 >> (16 * j)) & 63u;
            sc1 = (s0 >> (16 * j + 8)) & 63u;   mn1 = (s1 >> (16 * j + 8)) & 63u;
        } else {
            const uint32_t sh = 16 * (j - 2);
            sc0 = ((s2 >> sh) & 0x0Fu) | (((s0 >> (sh + 6)) & 3u) << 4);
            mn0 = ((s2 >> (sh + 4)) & 0x0Fu) | (((s1 >> (sh + 6)) & 3u) << 4);
            sc1 = ((s2 >> (sh + 8)) & 0x0Fu) | (((s0 >> (sh + 14)) & 3u) << 4);
            mn1 = ((s2 >> (sh + 12)) & 0x0Fu) | (((s1 >> (sh + 14)) & 3u) << 4);
        }
        const float2 dd = __half22float2(as_half2(r.h.x));
        // d * sc * q is exact in fp32 (11-bit scale x 6-bit code x 4-bit quant), so the fused form rounds like mul-then-sub
        const float d1 = dd.x * static_cast<float>(sc0), m1 = -(dd.y * static_cast<float>(mn0));
        const float d2 = dd.x * static_cast<float>(sc1) * 0.0625f, m2 = -(dd.y * static_cast<float>(mn1));  // a high nibble arrives as 16 q
        const uint64_t dl = f32x2(d1, d1), ml = f32x2(m1, m1), dh = f32x2(d2, d2), mh = f32x2(m2, m2);
        const uint32_t q[8] = {r.q[0].x, r.q[0].y, r.q[0].z, r.q[0].w, r.q[1].x, r.q[1].y, r.q[1].z, r.q[1].w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {  // bytes 8c .. 8c+7: elements 8c .. of the low-nibble sub-block and of the high one
            uint32_t lo[4], hi[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t u = q[2 * c + (k >> 1)] >> (8 * (k & 1));
                lo[k] = pack2<BF16>(fma2(dl, widen(codes((u & 0x000F000Fu) | 0x64006400u, 0)), ml));
                hi[k] = pack2<BF16>(fma2(dh, widen(codes((u & 0x00F000F0u) | 0x64006400u, 0)), mh));
            }
            store_chunk(at, c, make_uint4(lo[0], lo[1], lo[2], lo[3]));
            store_chunk(at, c + 4, make_uint4(hi[0], hi[1], hi[2], hi[3]));
        }
    }
};

struct GemmQ80R {  // repacked groups of 272 B: d[8] fp16 | chunk c < 4, thread t < 4: words (block 2c, step 0/1), (block 2c+1, step 0/1)
    static constexpr uint32_t kBlock = 272, kPitch = 272;
    static constexpr double kConvertNs = 320.0;
    struct Regs {
        uint4 w[4];  // thread t: (block 2j, step 0), (2j, 1), (2j + 1, 0), (2j + 1, 1)
        uint32_t d;  // the scales of blocks 2j and 2j + 1
    };
    __device__ static __forceinline__ uint32_t fold(const Regs& r) { return fold4(r.w[0]) ^ fold4(r.w[1]) ^ fold4(r.w[2]) ^ fold4(r.w[3]) ^ r.d; }
    __device__ static __forceinline__ void load(Regs& r, const uint8_t* row, uint32_t j) {
#pragma unroll
        for (int t = 0; t < 4; ++t) r.w[t] = *reinterpret_cast<const uint4*>(row + 16 + j * 64 + t * 16);
        r.d = *reinterpret_cast<const uint32_t*>(row + 4 * j);
    }
    template <bool BF16>
    __device__ static __forceinline__ void emit(const Regs& r, uint32_t, uint32_t at) {
        const __half2 dd = as_half2(r.d);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const __half2 d16 = b ? __high2half2(dd) : __low2half2(dd);
            const uint64_t d32 = widen(d16);
#pragma unroll
            for (int g = 0; g < 4; ++g) {  // weights 8g .. 8g+7 of the block: step g / 2, threads 2 (g % 2) and + 1
                uint32_t v[4];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const uint4& w4 = r.w[2 * (g & 1) + k];
                    const uint32_t w = (b ? (g >> 1 ? w4.w : w4.z) : (g >> 1 ? w4.y : w4.x)) ^ 0x80808080u;  // int8 + 128
                    v[2 * k] = scaled_pair<BF16>(codes(bytes02(w), 128), d16, d32);
                    v[2 * k + 1] = scaled_pair<BF16>(codes(bytes13(w), 128), d16, d32);
                }
                store_chunk(at, 4 * b + g, make_uint4(v[0], v[1], v[2], v[3]));
            }
        }
    }
};

struct GemmQ40R {  // repacked groups of 144 B: d[8] fp16 | chunk c < 2, thread t < 4: the quant word (bytes 4t..4t+3) of blocks 4c..4c+3
    static constexpr uint32_t kBlock = 144, kPitch = 144;
    static constexpr double kConvertNs = 310.0;
    struct Regs {
        uint2 w[4];  // thread t's words of blocks 2j and 2j + 1: low nibbles = weights 4t.., high nibbles = weights 16 + 4t..
        uint32_t d;
    };
    __device__ static __forceinline__ uint32_t fold(const Regs& r) {
        return r.w[0].x ^ r.w[0].y ^ r.w[1].x ^ r.w[1].y ^ r.w[2].x ^ r.w[2].y ^ r.w[3].x ^ r.w[3].y ^ r.d;
    }
    __device__ static __forceinline__ void load(Regs& r, const uint8_t* row, uint32_t j) {
#pragma unroll
        for (int t = 0; t < 4; ++t) r.w[t] = *reinterpret_cast<const uint2*>(row + 16 + (j >> 1) * 64 + t * 16 + (j & 1) * 8);
        r.d = *reinterpret_cast<const uint32_t*>(row + 4 * j);
    }
    template <bool BF16>
    __device__ static __forceinline__ void emit(const Regs& r, uint32_t, uint32_t at) {
        const __half2 dd = as_half2(r.d);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const __half2 d16 = b ? __high2half2(dd) : __low2half2(dd);
            const uint64_t d32 = widen(d16);
#pragma unroll
            for (int g = 0; g < 4; ++g) {  // weights 8g .. 8g+7: g < 2 the low nibbles of words 2g, 2g+1; else the high nibbles of words 2(g-2), +1
                uint32_t v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint2& w2 = r.w[2 * (g & 1) + (k >> 1)];
                    const uint32_t u = (b ? w2.y : w2.x) >> (8 * (k & 1) + (g < 2 ? 0 : 4));
                    v[k] = scaled_pair<BF16>(codes((u & 0x000F000Fu) | 0x64006400u, 8), d16, d32);
                }
                store_chunk(at, 4 * b + g, make_uint4(v[0], v[1], v[2], v[3]));
            }
        }
    }
};

struct GemmQ6KR {  // repacked groups of 224 B: scales[16] int8 | d fp16, pad | half n < 2, thread t < 4: ql words (b, lh) | thread t: qh words (n, lh)
    // A slot row holds 16 bytes of the next group as well: at a pitch of 224 bytes (an even number of 16-byte units) the 16-byte loads of
    // eight rows met on four bank groups.
    static constexpr uint32_t kBlock = 224, kPitch = 240;
    static constexpr double kConvertNs = 380.0;
    struct Regs {
        uint4 ql[4];     // thread t: words (b 0, lh 0), (0, 1), (1, 0), (1, 1) of half j / 2
        uint2 qh[4];     // thread t: words (lh 0, lh 1)
        uint32_t sc, d;  // the scales of the quarter's four 16-weight groups
    };
    __device__ static __forceinline__ uint32_t fold(const Regs& r) {
        return fold4(r.ql[0]) ^ fold4(r.ql[1]) ^ fold4(r.ql[2]) ^ fold4(r.ql[3]) ^ r.qh[0].x ^ r.qh[0].y ^ r.qh[1].x ^ r.qh[1].y ^ r.qh[2].x ^ r.qh[2].y ^
               r.qh[3].x ^ r.qh[3].y ^ r.sc ^ r.d;
    }
    __device__ static __forceinline__ void load(Regs& r, const uint8_t* row, uint32_t j) {
        const uint32_t n = j >> 1;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            r.ql[t] = *reinterpret_cast<const uint4*>(row + 32 + n * 64 + t * 16);
            r.qh[t] = *reinterpret_cast<const uint2*>(row + 160 + n * 8 + t * 16);
        }
        r.sc = *reinterpret_cast<const uint32_t*>(row + 4 * j);
        r.d = *reinterpret_cast<const uint16_t*>(row + 16);
    }
    template <bool BF16>
    __device__ static __forceinline__ void emit(const Regs& r, uint32_t j, uint32_t at) {
        if (j & 1u) emit_half<BF16, 1>(r, at);
        else emit_half<BF16, 0>(r, at);
    }
    /// Runs 2 J and 2 J + 1 of a 128-weight half: ql words b = 0, 1, their nibbles J; qh bits 4 J + 2 b and + 1 of every byte.
    template <bool BF16, int J>
    __device__ static __forceinline__ void emit_half(const Regs& r, uint32_t at) {
        const float d = __half2float(__ushort_as_half(static_cast<uint16_t>(r.d)));
#pragma unroll
        for (int b = 0; b < 2; ++b) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {  // weights 8g .. 8g+7 of the run: lh = g / 2, threads 2 (g % 2) and + 1
                const int lh = g >> 1;
                const float ds = d * static_cast<float>(static_cast<int8_t>((r.sc >> (8 * (2 * b + lh))) & 0xFFu));
                const uint64_t ds2 = f32x2(ds, ds);
                uint32_t v[4];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const uint4& l4 = r.ql[2 * (g & 1) + k];
                    const uint2& h2 = r.qh[2 * (g & 1) + k];
                    const uint32_t l = b ? (lh ? l4.w : l4.z) : (lh ? l4.y : l4.x), h = lh ? h2.y : h2.x;
                    const uint32_t hi = J ? (b ? h >> 2 : h) : (b ? h << 2 : h << 4);  // the run's two bits at bits 4 and 5 of every byte
                    const uint32_t w = ((l >> (4 * J)) & 0x0F0F0F0Fu) | (hi & 0x30303030u);
                    // (d*s)*(q-32): 19-bit scale x 6-bit code is exact in fp32, rounded once to 16 bits
                    v[2 * k] = pack2<BF16>(mul2(ds2, widen(codes(bytes02(w), 32))));
                    v[2 * k + 1] = pack2<BF16>(mul2(ds2, widen(codes(bytes13(w), 32))));
                }
                store_chunk(at, 4 * b + g, make_uint4(v[0], v[1], v[2], v[3]));
            }
        }
    }
};

#define HC_TMEM_LD32(v, taddr)                                                                                                                   \
    asm volatile(                                                                                                                                \
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "                                                                                                \
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"        \
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),     \
          "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),       \
          "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),       \
          "=r"(v[31])                                                                                                                            \
        : "r"(taddr)                                                                                                                             \
        : "memory")

template <bool BF16, class F>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ GemmArgs a) {
    extern __shared__ uint8_t smem_raw[];
    constexpr uint32_t kRawTile = kCtaRows * F::kPitch;
    // tiles need 1024-byte alignment (one swizzle atom)
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t tiles = smem_u32(smem);
    const uint32_t x_bytes = (a.nt / 2u) * (kBK * 2u), stage_bytes = kTileW + a.nacc * x_bytes;  // x_bytes: one accumulator's half in this CTA
    const uint32_t raw_off = a.stages * stage_bytes;
    const uint32_t bars_off = raw_off + a.raw_slots * kRawTile, bars = tiles + bars_off;
    auto full = [&](uint32_t s) { return bars + s * 8u; };
    auto empty = [&](uint32_t s) { return bars + (kMaxStages + s) * 8u; };
    auto raw_full = [&](uint32_t s) { return bars + (2 * kMaxStages + s) * 8u; };
    auto raw_empty = [&](uint32_t s) { return bars + (2 * kMaxStages + kMaxRaw + s) * 8u; };
    auto acc_full = [&](uint32_t s) { return bars + (2 * kMaxStages + 2 * kMaxRaw + s) * 8u; };
    auto acc_empty = [&](uint32_t s) { return bars + (2 * kMaxStages + 2 * kMaxRaw + 2 + s) * 8u; };
    constexpr uint32_t kBarBytes = (2 * kMaxStages + 2 * kMaxRaw + 4) * 8u;
    volatile uint32_t* tmem_word = reinterpret_cast<volatile uint32_t*>(smem + bars_off + kBarBytes);
    volatile uint32_t* abort_word = tmem_word + 1;

    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31u;
    const uint32_t rank = cluster_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1, leader_bars = map_to_leader(bars);

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < a.stages; ++s) {
            g_mbar_init(full(s), 1 + 2 * kDeqGroupWarps);
            g_mbar_init(empty(s), 1);
        }
        for (uint32_t s = 0; s < a.raw_slots; ++s) {
            g_mbar_init(raw_full(s), 1);
            g_mbar_init(raw_empty(s), kDeqWarps);
        }
        for (uint32_t s = 0; s < 2; ++s) {
            g_mbar_init(acc_full(s), 1);
            g_mbar_init(acc_empty(s), 8);
        }
        *abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    cluster_sync();
    if (warp == 1) {  // TMEM: all 512 columns (two 128 x 256 fp32 accumulators) in both CTAs, which both run by now; one CTA per SM, so nobody else asks
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(const_cast<uint32_t*>(tmem_word))), "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_word;
    // the next kernel in the stream may start its prologue; nothing of an earlier kernel's is read or overwritten before the wait
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    struct Unit {
        uint32_t w_tile, t_tile, sb0, sb1, split, tile;
    };
    auto unit_of = [&](uint32_t u) {
        Unit r;
        r.tile = u, r.split = 0, r.sb0 = 0, r.sb1 = a.nb;
        if (u >= a.whole && a.splits > 1) {
            r.tile = a.whole + (u - a.whole) / a.splits, r.split = (u - a.whole) % a.splits;
            r.sb0 = static_cast<uint32_t>(uint64_t{a.nb} * r.split / a.splits);
            r.sb1 = static_cast<uint32_t>(uint64_t{a.nb} * (r.split + 1) / a.splits);
        }
        r.t_tile = r.tile % a.token_tiles, r.w_tile = r.tile / a.token_tiles;
        return r;
    };

    if (warp == 0) {
        // ---- TMA producer: X tiles (this CTA's half of every accumulator's tokens) ------------------------------------------
        RingPos st{0, 0};
        bool ok = true;
        for (uint32_t u = pair; u < a.units && ok; u += pairs) {
            const Unit un = unit_of(u);
            const uint32_t m0 = un.t_tile * a.nacc * a.nt + rank * (a.nt / 2u);
            for (uint32_t kb = un.sb0 * 4u; kb < un.sb1 * 4u; ++kb) {
                ok = g_mbar_wait_warp(empty(st.slot), st.parity ^ 1u);
                if (!ok) break;
                if (elect_one()) {
                    if (rank == 0) g_mbar_expect_tx(full(st.slot), 2u * a.nacc * x_bytes);
                    const uint32_t dst = tiles + st.slot * stage_bytes + kTileW, bar = leader_bars + st.slot * 8u;
                    g_tma_2d_pair(dst, &xmap, kb * kBK, m0, bar);
                    if (a.nacc == 2) g_tma_2d_pair(dst + x_bytes, &xmap, kb * kBK, m0 + a.nt, bar);
                }
                __syncwarp();
                st.advance(1, a.stages);
            }
        }
        // the leader's commits reach into both CTAs: neither leaves before the last one to each slot has arrived
        for (uint32_t s = 0; s < a.stages && ok; ++s) {
            ok = g_mbar_wait_warp(empty(st.slot), st.parity ^ 1u);
            st.advance(1, a.stages);
        }
        if (!ok && lane == 0) *abort_word = 1;
    } else if (warp == 1) {
        // ---- MMA issuer (the pair's first CTA, for both) ------------------------------------------------------------------------
        if (rank == 0) {
            // instruction descriptor: D = fp32 (bits 4-5 = 1), A / B format (bits 7-9 / 10-12: 0 = f16, 1 = bf16), both
            // K-major (bits 15, 16 = 0), N / 8 at bits 17-22, M / 16 at bits 24-28
            const uint32_t fmt = BF16 ? 1u : 0u;
            const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((a.nt >> 3) << 17) | ((kPairRows >> 4) << 24);
            bool ok = true;
            RingPos st{0, 0}, ac{0, 0};  // ac: the accumulator of the tile (its first of two), and the parity of its use
            for (uint32_t u = pair; u < a.units && ok; u += pairs) {
                const Unit un = unit_of(u);
                for (uint32_t acc = 0; acc < a.nacc && ok; ++acc) ok = g_mbar_wait_warp(acc_empty(ac.slot + acc), ac.parity ^ 1u);
                for (uint32_t kb = un.sb0 * 4u; kb < un.sb1 * 4u && ok; ++kb) {
                    ok = g_mbar_wait_warp(full(st.slot), st.parity);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elect_one()) {
                        const uint32_t more = kb == un.sb0 * 4u ? 0u : 1u, w_at = tiles + st.slot * stage_bytes, d = tmem_base + ac.slot * 256u;
                        const uint64_t wd = smem_desc(w_at), xd = smem_desc(w_at + kTileW);
#pragma unroll
                        for (uint32_t k = 0; k < kBK / 16; ++k)  // 16 elements = 32 bytes along K inside the swizzled row
                            umma_f16_pair(d, wd + k * 2u, xd + k * 2u, idesc, k == 0 ? more : 1u);
                        if (a.nacc == 2) {
                            const uint64_t xd2 = xd + (x_bytes >> 4);
#pragma unroll
                            for (uint32_t k = 0; k < kBK / 16; ++k) umma_f16_pair(d + 256u, wd + k * 2u, xd2 + k * 2u, idesc, k == 0 ? more : 1u);
                        }
                        umma_commit_pair(empty(st.slot));  // arrives once the MMAs above have finished reading this stage
                        if (kb + 1u == un.sb1 * 4u) {
                            umma_commit_pair(acc_full(ac.slot));
                            if (a.nacc == 2) umma_commit_pair(acc_full(1));
                        }
                    }
                    __syncwarp();
                    st.advance(1, a.stages);
                }
                ac.advance(a.nacc, 2);
            }
            if (!ok && lane == 0) *abort_word = 1;
        }
    } else if (warp == 2) {
        // ---- TMA producer: quantized W rows of this CTA -----------------------------------------------------------------------
        RingPos rw{0, 0};
        bool ok = true;
        for (uint32_t u = pair; u < a.units && ok; u += pairs) {
            const Unit un = unit_of(u);
            const uint32_t row0 = un.w_tile * kPairRows + rank * kCtaRows;
            for (uint32_t sb = un.sb0; sb < un.sb1; ++sb) {
                ok = g_mbar_wait_warp(raw_empty(rw.slot), rw.parity ^ 1u);
                if (!ok) break;
                if (elect_one()) {
                    g_mbar_expect_tx(raw_full(rw.slot), kRawTile);
                    g_tma_2d(tiles + raw_off + rw.slot * kRawTile, &wmap, sb * (F::kBlock / 4u), row0, raw_full(rw.slot));
                }
                __syncwarp();
                rw.advance(1, a.raw_slots);
            }
        }
        if (!ok && lane == 0) *abort_word = 1;
    } else if (warp >= kDeqWarp) {
        // ---- dequantization ----------------------------------------------------------------------------------------------------
        const uint32_t j = (warp - kDeqWarp) / kDeqGroupWarps, r = ((warp - kDeqWarp) % kDeqGroupWarps) * 32u + lane;
        const uint32_t row_at = tiles + r * (kBK * 2u) + ((r & 7u) << 4);
        bool ok = true;
        RingPos rw{0, 0}, st{0, 0};
        st.advance(j, a.stages);
        for (uint32_t u = pair; u < a.units && ok; u += pairs) {
            const Unit un = unit_of(u);
            for (uint32_t sb = un.sb0; sb < un.sb1; ++sb) {
                ok = g_mbar_wait_warp(raw_full(rw.slot), rw.parity);
                if (!ok) break;
                typename F::Regs regs;
                F::load(regs, smem + raw_off + rw.slot * kRawTile + r * F::kPitch, j);
                // The slot may be refilled once every lane's words are in registers: the vote cannot be taken before (an arrival behind the
                // load instructions alone let the copy engine overwrite the first rows of a slow warp).
                const uint32_t others = __ballot_sync(0xFFFFFFFFu, F::fold(regs) != 0x9E3779B9u);
                if (lane == (others == 0 ? 1u : 0u)) g_mbar_arrive(raw_empty(rw.slot));
                rw.advance(1, a.raw_slots);
                ok = g_mbar_wait_warp(empty(st.slot), st.parity ^ 1u);
                if (!ok) break;
                F::template emit<BF16>(regs, j, row_at + st.slot * stage_bytes);
                // make the generic-proxy stores visible to the tensor core's (async-proxy) reads, then one arrival per warp
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) g_mbar_arrive_cluster(leader_bars + st.slot * 8u);
                st.advance(4, a.stages);
            }
        }
        if (!ok && lane == 0) *abort_word = 1;
    } else if (warp >= kEpiWarp) {
        // ---- epilogue: TMEM -> registers -> y (or this split's partial sums) -------------------------------------------------------
        const uint32_t quarter = warp & 3u;  // TMEM lanes 32 * quarter .. (fixed by warp id % 4)
        bool ok = true;
        RingPos ac{0, 0};
        for (uint32_t u = pair; u < a.units && ok; u += pairs) {
            const Unit un = unit_of(u);
            const uint32_t row = un.w_tile * kPairRows + rank * kCtaRows + quarter * 32u + lane;
            const uint32_t tile_tokens = a.nacc * a.nt;
            const uint64_t part_floats = uint64_t{tile_tokens} * kCtaRows;
            const bool shared = a.splits > 1 && un.tile >= a.whole;  // this unit is a share of its tile's K
            float* part = shared ? a.partials + ((uint64_t{un.tile - a.whole} * a.splits + un.split) * 2u + rank) * part_floats + quarter * 32u + lane : nullptr;
            for (uint32_t acc = 0; acc < a.nacc; ++acc) {
                const uint32_t which = ac.slot + acc;
                ok = g_mbar_wait_warp(acc_full(which), ac.parity);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t t0 = un.t_tile * tile_tokens + acc * a.nt;
#pragma unroll 1
                for (uint32_t c = 0; c < a.nt && t0 + c < a.n_vec; c += 32u) {
                    uint32_t v[32];
                    HC_TMEM_LD32(v, tmem_base + ((quarter * 32u) << 16) + which * 256u + c);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (shared) {
                        float* p = part + uint64_t{acc * a.nt + c} * kCtaRows;
#pragma unroll
                        for (uint32_t k = 0; k < 32u; ++k) p[k * kCtaRows] = __uint_as_float(v[k]);
                    } else if (row < a.rows) {
                        uint8_t* yp = reinterpret_cast<uint8_t*>(a.y + row) + uint64_t{t0 + c} * a.y_stride;
                        const uint32_t left = a.n_vec - (t0 + c);
                        if (left >= 32u) {
#pragma unroll
                            for (uint32_t k = 0; k < 32u; ++k) *reinterpret_cast<uint32_t*>(yp + k * a.y_stride) = v[k];
                        } else {
#pragma unroll
                            for (uint32_t k = 0; k < 32u; ++k)
                                if (k < left) *reinterpret_cast<uint32_t*>(yp + k * a.y_stride) = v[k];
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) g_mbar_arrive_cluster(leader_bars + (acc_empty(which) - bars));
            }
            if (!ok) break;
            ac.advance(a.nacc, 2);
        }
        if (!ok && lane == 0) *abort_word = 1;
    }
    // ---- everyone meets here, also after a failed wait, so that TMEM is always released and no CTA leaves while its pair still needs it --
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();
    if (threadIdx.x == 0 && *abort_word != 0 && a.error_word != nullptr) atomicOr(a.error_word, 2u);
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
    __syncwarp();
    cluster_sync();
}

/// y of the split tiles = their partial sums added in split order.  grid (128-row halves of the tiles from `whole` on, tokens / 8), 32 x 4
/// threads: a lane takes four consecutive W rows of two tokens.  (The last CTA to finish a tile adding them itself had 128 threads' loads in
/// flight for what the whole device does here.)
__global__ void __launch_bounds__(128) add_splits_kernel(const float* __restrict__ partials, float* __restrict__ y, uint64_t y_stride, uint32_t rows, uint32_t n_vec,
                                                         uint32_t tile_tokens, uint32_t token_tiles, uint32_t whole, uint32_t splits) {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t rest = blockIdx.x >> 1, half = blockIdx.x & 1u, w_tile = (whole + rest) / token_tiles, t_tile = (whole + rest) % token_tiles;
    const uint32_t r = (threadIdx.x & 31u) * 4u, row = w_tile * kPairRows + half * kCtaRows + r;
    const uint64_t part_floats = uint64_t{tile_tokens} * kCtaRows;
#pragma unroll
    for (uint32_t u = 0; u < 2; ++u) {
        const uint32_t in = blockIdx.y * 8u + u * 4u + (threadIdx.x >> 5), t = t_tile * tile_tokens + in;
        if (t >= n_vec) break;
        const float* p = partials + (uint64_t{rest} * splits * 2u + half) * part_floats + uint64_t{in} * kCtaRows + r;
        float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
        for (uint32_t s = 0; s < splits; ++s) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(p + uint64_t{s} * 2u * part_floats));
            sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
        }
        float* yp = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(y) + uint64_t{t} * y_stride) + row;
        if (row + 4u <= rows && (reinterpret_cast<uintptr_t>(yp) & 15u) == 0) {
            *reinterpret_cast<float4*>(yp) = sum;
        } else {
            if (row < rows) yp[0] = sum.x;
            if (row + 1u < rows) yp[1] = sum.y;
            if (row + 2u < rows) yp[2] = sum.z;
            if (row + 3u < rows) yp[3] = sum.w;
        }
    }
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int encode_2d(CUtensorMapDataType type, const void* base, uint64_t inner, uint64_t outer, uint64_t stride, uint32_t box_inner, uint32_t box_outer,
              CUtensorMapSwizzle swizzle, const char* what, CUtensorMap* out) {
    static EncodeTiledFn encode = nullptr;
    if (encode == nullptr) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        HC_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
        if (fn == nullptr || qres != cudaDriverEntryPointSuccess) return fail(HALO_CUDA_E_BACKEND, "cuTensorMapEncodeTiled is not available");
        encode = reinterpret_cast<EncodeTiledFn>(fn);
    }
    const cuuint64_t dims[2] = {inner, outer};
    const cuuint64_t strides[1] = {stride};
    const cuuint32_t box[2] = {box_inner, box_outer};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = encode(out, type, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(HALO_CUDA_E_KERNEL, "MATMUL: cannot describe %s to the copy engine (CUresult %d)", what, (int)r);
    return 0;
}

/// How a call is cut into units of (256 W rows, T tokens, a share of K).
struct GemmPlan {
    uint32_t nt, nacc, stages, raw_slots, w_tiles, token_tiles, splits;
    uint64_t whole, units;  // tiles over all of K; units of work
    uint64_t split_tiles() const { return uint64_t{w_tiles} * token_tiles - whole; }
};

template <class F>
void ring_sizes(GemmPlan* p) {
    const uint32_t raw = kCtaRows * F::kPitch, stage = kTileW + p->nacc * (p->nt / 2u) * (kBK * 2u);
    p->raw_slots = 2;
    p->stages = std::min((kSmemTiles - 2u * raw) / stage, kMaxStages);
    if (p->stages * stage + 3u * raw <= kSmemTiles) p->raw_slots = 3;
}

/// The cheapest (T, splits) by a model of the measured times (ns): a K step of 64 costs 1.42 a token for its MMAs and the format's
/// conversion, which overlap but for the issue slots and the shared memory they compete for (the fourth-power mean fits T from 64 to 448);
/// storing a tile's y costs 31 a token, under the next tile's MMAs where T <= 256.  Every pair gets as many whole tiles as there are for
/// all; the K of the tiles left over is split, and a split stores and adds 2 x 4 bytes an output.
template <class F>
GemmPlan plan_gemm(uint32_t rows, uint32_t cols, uint32_t n_vec, uint32_t pairs, bool may_split) {
    const uint32_t nb = cols / 256u, w_tiles = (rows + kPairRows - 1) / kPairRows;
    const double reread = 0.3 * (double(rows) * nb * F::kBlock / 6000.0);  // what a further token tile's pass over W (in L2) costs beyond its conversion
    GemmPlan best{};
    double best_cost = 0;
    for (uint32_t t = 32; t <= 448; t += t < 256 ? 32 : 64) {
        GemmPlan p{};
        p.nacc = t > 256 ? 2 : 1, p.nt = t / p.nacc;
        p.w_tiles = w_tiles, p.token_tiles = (n_vec + t - 1) / t;
        ring_sizes<F>(&p);
        if (p.stages < kMinStages) break;
        const double mma = 1.42 * t, a = mma * mma, b = F::kConvertNs * F::kConvertNs, step = std::sqrt(std::sqrt(a * a + b * b));
        const double store = 31.0 * std::min(t, n_vec);
        auto waves_of = [&](uint64_t waves, uint32_t blocks) {
            const double main = step * 4.0 * blocks;
            return waves * (p.nacc == 1 ? std::max(main, store) : main + store);
        };
        const uint64_t tiles = uint64_t{w_tiles} * p.token_tiles, whole = tiles / pairs * pairs, rest = tiles - whole;
        for (uint32_t s = 1; s <= (may_split && rest != 0 ? std::min(nb, 16u) : 1u); ++s) {
            p.splits = s, p.whole = s > 1 ? whole : tiles, p.units = p.whole + (s > 1 ? rest * s : 0);
            double cost = waves_of(whole / pairs, nb) + waves_of((rest * s + pairs - 1) / pairs, (nb + s - 1) / s) + store + reread * p.token_tiles;
            if (s > 1) cost += 3000.0 + 8.0 * s * rest * kPairRows * std::min(t, n_vec) / 5000.0;
            if (best_cost == 0 || cost < best_cost) best_cost = cost, best = p;
        }
        if (t >= n_vec) break;  // nothing but padding beyond this
    }
    return best;
}

cudaLaunchConfig_t dependent_launch(dim3 grid, uint32_t threads, uint32_t smem, cudaStream_t s, cudaLaunchAttribute* attr) {
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid, cfg.blockDim = dim3(threads), cfg.dynamicSmemBytes = smem, cfg.stream = s, cfg.attrs = attr, cfg.numAttrs = 1;
    return cfg;
}

template <bool BF16, class F>
int launch_t(HaloCudaCtx* ctx, const GemvCall& c, cudaStream_t s) {
    const uint32_t pairs_max = static_cast<uint32_t>(ctx->prop.multiProcessorCount) / 2u;
    GemmPlan p = plan_gemm<F>(c.rows, c.cols, c.n_vec, pairs_max, (c.flags & HALO_CUDA_GEMV_FLAG_NO_SCRATCH) == 0);
    if (uint64_t{p.w_tiles} * p.token_tiles > 0x7FFFFFFFu) return fail(HALO_CUDA_E_UNSUPPORTED, "MATMUL: %u x %u outputs exceed the launch limit", c.n_vec, c.rows);
    void* ws = nullptr;
    if (int rc = workspace(ctx, 0, uint64_t{c.n_vec} * c.cols * 2, s, &ws)) return rc;
    // The splits' partial sums: also while the stream is being captured, so that a prompt's plan, and with it its bits, do not depend on what the
    // stream ran before.  A device without the memory runs the cheapest plan that needs none.
    void* partials = nullptr;
    if (p.splits > 1) {
        const int rc = workspace(ctx, 4, p.split_tiles() * p.splits * p.nacc * p.nt * kPairRows * 4u, s, &partials, /*zeroed=*/false, /*while_capturing=*/true);
        if (rc == HALO_CUDA_E_MEMORY) p = plan_gemm<F>(c.rows, c.cols, c.n_vec, pairs_max, false);
        else if (rc != 0) return rc;
    }
    CUtensorMap xmap, wmap;
    if (int rc = encode_2d(BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, ws, c.cols, c.n_vec, uint64_t{c.cols} * 2, kBK, p.nt / 2u,
                           CU_TENSOR_MAP_SWIZZLE_128B, "x", &xmap))
        return rc;
    // (the pitch of a one-row matrix is never used, but has to be a valid one: at least a row, below 2^40)
    if (int rc = encode_2d(CU_TENSOR_MAP_DATA_TYPE_UINT32, c.w, c.row_bytes / 4u, c.rows, c.rows > 1 ? c.w_stride : c.row_bytes, F::kPitch / 4u, kCtaRows,
                           CU_TENSOR_MAP_SWIZZLE_NONE, "the weight matrix", &wmap))
        return rc;
    cudaLaunchAttribute attr[1];
    const uint32_t groups = c.cols / 8u, chunks = (groups + 511u) / 512u, cast_threads = ((groups + 2u * chunks - 1u) / (2u * chunks) + 31u) & ~31u;
    const cudaLaunchConfig_t cast_cfg = dependent_launch(dim3(chunks, std::min(c.n_vec, 65535u)), cast_threads, 0, s, attr);
    HC_CUDA(cudaLaunchKernelEx(&cast_cfg, cast_x_kernel<BF16>, c.x, c.x_stride, static_cast<uint16_t*>(ws), c.n_vec, c.cols));
    auto kern = gemm_tcgen05_kernel<BF16, F>;
    if (int rc = allow_dynamic_smem(ctx, reinterpret_cast<const void*>(kern), kGemmSmem)) return rc;
    const GemmArgs args{c.y, c.y_stride, c.rows, c.n_vec, c.cols / 256u, p.nt, p.nacc, p.stages, p.raw_slots, p.token_tiles, static_cast<uint32_t>(p.whole), p.splits, static_cast<uint32_t>(p.units),
                        static_cast<float*>(partials), ctx->error_word_dev};
    const cudaLaunchConfig_t cfg = dependent_launch(dim3(2u * static_cast<uint32_t>(std::min<uint64_t>(p.units, pairs_max))), kGemmThreads, kGemmSmem, s, attr);
    HC_CUDA(cudaLaunchKernelEx(&cfg, kern, xmap, wmap, args));
    if (p.splits > 1) {
        const cudaLaunchConfig_t add_cfg = dependent_launch(dim3(2u * static_cast<uint32_t>(p.split_tiles()), p.nacc * p.nt / 8u), 128, 0, s, attr);
        HC_CUDA(cudaLaunchKernelEx(&add_cfg, add_splits_kernel, static_cast<const float*>(partials), c.y, c.y_stride, c.rows, c.n_vec, p.nacc * p.nt, p.token_tiles, static_cast<uint32_t>(p.whole), p.splits));
    }
    return 0;
}

template <class F>
int launch_f(HaloCudaCtx* ctx, const GemvCall& c, bool bf16, cudaStream_t s) {
    return bf16 ? launch_t<true, F>(ctx, c, s) : launch_t<false, F>(ctx, c, s);
}

}  // namespace

/// repacked: W is in the layout of halo_cuda_repack_rows (Q6_K / Q8_0 / Q4_0); else raw Q4_K rows.
bool gemm_tcgen05_supports(const GemvCall& c, bool repacked) {
    const bool type_ok = repacked ? (c.wtype == HALO_CUDA_T_Q6_K || c.wtype == HALO_CUDA_T_Q8_0 || c.wtype == HALO_CUDA_T_Q4_0) : c.wtype == HALO_CUDA_T_Q4_K;
    if (!type_ok || c.cols == 0 || c.rows == 0 || c.cols % 256u != 0) return false;
    if (reinterpret_cast<uintptr_t>(c.w) % 16 != 0 || c.w_stride % 16 != 0) return false;  // 16-byte block loads
    if (reinterpret_cast<uintptr_t>(c.x) % 16 != 0 || c.x_stride % 16 != 0) return false;  // float4 reads of x
    return c.n_vec <= 65535u * 256u;
}

int launch_gemm_tcgen05(HaloCudaCtx* ctx, const GemvCall& c, bool bf16, bool repacked, cudaStream_t s) {
    if (!repacked) return launch_f<GemmQ4K>(ctx, c, bf16, s);
    switch (c.wtype) {
        case HALO_CUDA_T_Q6_K: return launch_f<GemmQ6KR>(ctx, c, bf16, s);
        case HALO_CUDA_T_Q8_0: return launch_f<GemmQ80R>(ctx, c, bf16, s);
        case HALO_CUDA_T_Q4_0: return launch_f<GemmQ40R>(ctx, c, bf16, s);
        default: return fail(HALO_CUDA_E_UNSUPPORTED, "MATMUL: no repacked GEMM for weight type id %u", c.wtype);
    }
}

int gemm_plan(uint32_t wtype, uint32_t rows, uint32_t cols, uint32_t n_vec, uint32_t sm_count, bool may_split, HaloCudaGemmPlan* out) {
    auto describe = [&](const GemmPlan& p) {
        *out = HaloCudaGemmPlan{p.nt * p.nacc, p.nacc, p.stages, p.raw_slots, p.w_tiles, p.token_tiles, p.splits, sm_count / 2u, p.whole, p.units};
        return 0;
    };
    switch (wtype) {
        case HALO_CUDA_T_Q4_K: return describe(plan_gemm<GemmQ4K>(rows, cols, n_vec, sm_count / 2u, may_split));
        case HALO_CUDA_T_Q6_K: return describe(plan_gemm<GemmQ6KR>(rows, cols, n_vec, sm_count / 2u, may_split));
        case HALO_CUDA_T_Q8_0: return describe(plan_gemm<GemmQ80R>(rows, cols, n_vec, sm_count / 2u, may_split));
        case HALO_CUDA_T_Q4_0: return describe(plan_gemm<GemmQ40R>(rows, cols, n_vec, sm_count / 2u, may_split));
        default: return fail(HALO_CUDA_E_UNSUPPORTED, "MATMUL: no prefill GEMM for weight type id %u", wtype);
    }
}

}  // namespace halo_cuda
