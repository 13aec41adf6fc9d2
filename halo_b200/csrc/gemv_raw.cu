// gemv_warp_f32 over raw Q8_0 / Q4_0 / Q6_K rows: the fp32 kernel a host without the repacking loader runs, and the GDN gate rows.
//
// The 34 / 18 / 210-byte blocks start at any even address, so a lane that reads its block from global memory needs a 2-byte load per two
// quants.  Here a warp copies 2048 weights of a row at a time into its own ring of shared-memory slots with 16-byte cp.async (a slot keeps
// the source's phase within 16 bytes), x sits in shared memory for the whole CTA, and a lane takes 64 consecutive weights: it reads 4-byte
// words, puts misaligned ones together with a funnel shift, turns quants into fp32 by placing the byte under the exponent of 2^23, and
// multiplies two at a time (fma.rn.f32x2).
//
// Arithmetic of one (row, x row), the same for every batch size and every launch shape, so that a row's bits do not depend on either
// (include/halo/backend/backend.h:300-304): per scale group of 32 (Q6_K: 16) weights an even and an odd fp32 sum of q * x, added; the
// lane's total takes d * that by one fma, group after group in K order; the 32 lane totals are added by a xor-shuffle tree.
//
// What bounds it: one x row, the issue slots and the shared-memory reads of x, near HBM for the 8-bit formats (16 warps an SM with four
// slots of up to 2.2 KB in flight each; 8 warps with eight slots took 33 % longer at Q8_0 5120 x 17408); batches, the fp32 pipe and the decode:
// four (two) rows of W share each x value read, four (two) x rows share each decoded weight.  Measured, us, two-byte loads -> this form:
// Q8_0 5120 x 17408 at 1 / 8 / 16 rows 66 -> 27 (3.5 TB/s), 361 -> 113, 698 -> 218; Q6_K 46 -> 29, 190 -> 120 (8 rows); Q4_0 17408 x 5120 at
// 1 / 4 / 16 rows 91 -> 24, 327 -> 48, 1274 -> 161; 96 gate rows of K = 5120 at 1 / 512 / 2048 rows 6.1 -> 3.3, 125 -> 36, 494 -> 132.
#include <algorithm>

#include "internal.h"
#include "quant_dev.cuh"

namespace halo_cuda {
namespace {

constexpr uint32_t kSmemMax = 227 * 1024;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ int lds_s8(uint32_t a) {
    int v;
    asm volatile("ld.shared.s8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
struct X4 {
    uint64_t lo, hi;  // elements 0, 1 and 2, 3 as fp32 pairs
};
__device__ __forceinline__ X4 lds_x4(uint32_t a) {
    X4 v;
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v.lo), "=l"(v.hi) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t pack(float a, float b) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float sum2(uint64_t a) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a));
    return lo + hi;
}
/// Four unsigned bytes -> (byte - zero) as fp32: the byte under the exponent of 2^23, minus 2^23 + zero (exact).
__device__ __forceinline__ X4 widen4(uint32_t w, int zero) {
    const uint32_t e = 0x4B000000u;
    const float f0 = __uint_as_float(__byte_perm(w, e, 0x7440)), f1 = __uint_as_float(__byte_perm(w, e, 0x7441));
    const float f2 = __uint_as_float(__byte_perm(w, e, 0x7442)), f3 = __uint_as_float(__byte_perm(w, e, 0x7443));
    const float z = -(8388608.0f + static_cast<float>(zero));
    return {add2(pack(f0, f1), pack(z, z)), add2(pack(f2, f3), pack(z, z))};
}
template <int N>
__device__ __forceinline__ void lds_words(uint32_t (&w)[N], uint32_t at) {  // N words from a 2-byte aligned address
    const uint32_t base = at & ~3u, sh = (at & 2u) * 8u;
    uint32_t a = lds32(base);
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const uint32_t b = lds32(base + 4 * (k + 1));
        w[k] = __funnelshift_r(a, b, sh);
        a = b;
    }
}

// ---- formats: a lane's 64 weights ("item") of a slot ------------------------------------------------------------------------------------
// Groups of kQuads * 4 weights share a scale; quad q of a group is four consecutive x elements.  item_of maps a float4 of an x row to
// (item, position within the item).
struct RawQ80 {
    static constexpr uint32_t kSlotBytes = 2176, kGroups = 2, kQuads = 8;
    static constexpr bool kSharedWords = false;  // every group has words of its own
    struct Words {
        uint32_t w[8];
        float d;
    };
    __device__ static __forceinline__ void load(Words& r, uint32_t slot, uint32_t lane, uint32_t g) {
        const uint32_t at = slot + lane * 68u + g * 34u;
        r.d = f16_bits_to_f32(lds16(at));
        lds_words<8>(r.w, at + 2);
    }
    __device__ static __forceinline__ X4 quad(const Words& r, uint32_t, int q) { return widen4(r.w[q] ^ 0x80808080u, 128); }
    __device__ static __forceinline__ float scale(const Words& r, uint32_t) { return r.d; }
    __device__ static __forceinline__ void item_of(uint32_t f, uint32_t& item, uint32_t& i4) { item = f >> 4, i4 = f & 15u; }
    __device__ static __forceinline__ uint32_t groups_in(uint32_t item, uint32_t cols) {  // whole groups of an item inside the row
        return item * 64u + 64u <= cols ? 2u : item * 64u + 32u <= cols ? 1u : 0u;
    }
};
struct RawQ40 {
    static constexpr uint32_t kSlotBytes = 1152, kGroups = 2, kQuads = 8;
    static constexpr bool kSharedWords = false;
    struct Words {
        uint32_t w[4];
        float d;
    };
    __device__ static __forceinline__ void load(Words& r, uint32_t slot, uint32_t lane, uint32_t g) {
        const uint32_t at = slot + lane * 36u + g * 18u;
        r.d = f16_bits_to_f32(lds16(at));
        lds_words<4>(r.w, at + 2);
    }
    __device__ static __forceinline__ X4 quad(const Words& r, uint32_t, int q) { return widen4((r.w[q & 3] >> (q < 4 ? 0 : 4)) & 0x0F0F0F0Fu, 8); }
    __device__ static __forceinline__ float scale(const Words& r, uint32_t) { return r.d; }
    __device__ static __forceinline__ void item_of(uint32_t f, uint32_t& item, uint32_t& i4) { item = f >> 4, i4 = f & 15u; }
    __device__ static __forceinline__ uint32_t groups_in(uint32_t item, uint32_t cols) { return RawQ80::groups_in(item, cols); }
};
struct RawQ6K {  // item = (block, 128-weight half, run half h): 16 positions of each of the half's four 32-weight runs, one scale a run
    static constexpr uint32_t kSlotBytes = 1680, kGroups = 4, kQuads = 4;
    static constexpr bool kSharedWords = true;  // the words of an item serve all of its groups
    struct Words {
        uint32_t qa[4], qb[4], qh[4];
        float d[4];
    };
    __device__ static __forceinline__ void load(Words& r, uint32_t slot, uint32_t lane, uint32_t) {
        const uint32_t blk = slot + (lane >> 2) * 210u, half = (lane >> 1) & 1u, h = lane & 1u;
        lds_words<4>(r.qa, blk + half * 64u + h * 16u);
        lds_words<4>(r.qb, blk + half * 64u + 32u + h * 16u);
        lds_words<4>(r.qh, blk + 128u + half * 32u + h * 16u);
        const float d = f16_bits_to_f32(lds16(blk + 208u));
#pragma unroll
        for (uint32_t g = 0; g < 4; ++g) r.d[g] = d * static_cast<float>(lds_s8(blk + 192u + half * 8u + 2 * g + h));
    }
    __device__ static __forceinline__ X4 quad(const Words& r, uint32_t g, int q) {
        const uint32_t l = (g & 1u) ? r.qb[q] : r.qa[q];
        return widen4(((l >> (g & 2u ? 4 : 0)) & 0x0F0F0F0Fu) | (((r.qh[q] >> (2 * g)) & 0x03030303u) << 4), 32);
    }
    __device__ static __forceinline__ float scale(const Words& r, uint32_t g) { return r.d[g]; }
    __device__ static __forceinline__ void item_of(uint32_t f, uint32_t& item, uint32_t& i4) {
        item = (f >> 6) * 4u + ((f >> 5) & 1u) * 2u + ((f >> 2) & 1u), i4 = ((f >> 3) & 3u) * 4u + (f & 3u);
    }
    __device__ static __forceinline__ uint32_t groups_in(uint32_t item, uint32_t cols) { return item * 64u < cols ? 4u : 0u; }
};

template <class F>
constexpr uint32_t slot_pitch() { return (F::kSlotBytes + 32u + 15u) & ~15u; }  // room for the phase and for the word behind the last

struct RawArgs {
    const uint8_t *w, *w_end;
    uint64_t w_stride, row_bytes;
    const float* x;
    uint64_t x_stride;
    float* y;
    uint64_t y_stride;
    uint32_t rows, cols, n_vec, items_pad;
    const float *gate_dt_bias, *gate_a;
    uint32_t gate_n_v;
};

/// Copies 2048 weights (or what the row has left) of `row` from slot column `chunk` on into a slot.
template <class F>
__device__ __forceinline__ void fill_slot(const RawArgs& a, uint32_t row, uint32_t chunk, uint8_t* slot, uint32_t lane) {
    const uint64_t off = uint64_t{chunk} * F::kSlotBytes;
    const uint8_t* from = a.w + uint64_t{row} * a.w_stride + off;
    const uint32_t n = static_cast<uint32_t>(a.row_bytes - off < F::kSlotBytes ? a.row_bytes - off : F::kSlotBytes);
    const uint32_t lead = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(from) & 15u), quads = (lead + n + 15u) / 16u;
    const uint8_t* q0 = from - lead;
    if (q0 >= a.w && q0 + 16u * quads <= a.w_end) {
        const uint32_t dst = smem_addr(slot) + 16u * lane;
        const uint8_t* src = q0 + 16u * lane;
#pragma unroll
        for (uint32_t i = 0; i < (slot_pitch<F>() / 16u + 31u) / 32u; ++i)
            if (lane + 32u * i < quads) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 512u * i), "l"(src + 512u * i) : "memory");
        return;
    }
    for (uint32_t i = lane; i < quads; i += 32u) {  // the matrix's first and last bytes: never outside of the operand
        const uint8_t* src = q0 + 16u * i;
        if (src >= a.w && src + 16 <= a.w_end) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(slot + 16u * i)), "l"(src) : "memory");
        } else {
            for (uint32_t b = 0; b < 16u; b += 2u)
                if (src + b >= from && src + b + 2 <= from + n)
                    *reinterpret_cast<uint16_t*>(slot + 16u * i + b) = *reinterpret_cast<const uint16_t*>(src + b);
        }
    }
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait_pending() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

/// Adds a lane's item of R rows (at slot[0 .. R)) times MT x rows to acc.
template <class F, int R, int MT>
__device__ __forceinline__ void add_items(const uint32_t (&slot)[R], uint32_t lane, uint32_t xs, uint32_t x_pitch, uint32_t items_pad, uint32_t item, uint32_t groups,
                                          float (&acc)[R][MT]) {
    const uint32_t xi = min(item, items_pad - 1u);
    typename F::Words w[R];
    if constexpr (F::kSharedWords) {
#pragma unroll
        for (int r = 0; r < R; ++r) F::load(w[r], slot[r], lane, 0);
    }
#pragma unroll
    for (uint32_t g = 0; g < F::kGroups; ++g) {
        if constexpr (!F::kSharedWords) {
#pragma unroll
            for (int r = 0; r < R; ++r) F::load(w[r], slot[r], lane, g);
        }
        uint64_t s[R][MT];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int t = 0; t < MT; ++t) s[r][t] = 0;
#pragma unroll
        for (int q = 0; q < static_cast<int>(F::kQuads); ++q) {
            const uint32_t i4 = g * F::kQuads + q;
            X4 x[MT];
#pragma unroll
            for (int t = 0; t < MT; ++t) x[t] = lds_x4(xs + t * x_pitch + (i4 * items_pad + (xi ^ (i4 & 7u))) * 16u);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const X4 v = F::quad(w[r], g, q);
#pragma unroll
                for (int t = 0; t < MT; ++t) s[r][t] = fma2(v.hi, x[t].hi, fma2(v.lo, x[t].lo, s[r][t]));
            }
        }
        if (g < groups) {  // (a lane behind the row's end has read another row's bytes: its sums are dropped)
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int t = 0; t < MT; ++t) acc[r][t] = fmaf(F::scale(w[r], g), sum2(s[r][t]), acc[r][t]);
        }
    }
}

/// One pass: rows [row0, row0 + R) against the MT x rows from t0 on.
template <class F, int R, int MT, int NS, class Next>
__device__ __forceinline__ void run_pass(const RawArgs& a, uint32_t row0, uint32_t t0, uint32_t chunks, uint8_t* ring, uint32_t& head, uint32_t lane, uint32_t xs,
                                         uint32_t x_pitch, Next&& fill_next) {
    float acc[R][MT];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int t = 0; t < MT; ++t) acc[r][t] = 0.0f;
    for (uint32_t c = 0; c < chunks; ++c) {
        wait_pending<NS - R>();
        __syncwarp();
        uint32_t slot[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint8_t* from = a.w + uint64_t{row0 + r} * a.w_stride + uint64_t{c} * F::kSlotBytes;
            slot[r] = smem_addr(ring + ((head + r) % NS) * slot_pitch<F>()) + static_cast<uint32_t>(reinterpret_cast<uintptr_t>(from) & 15u);
        }
        const uint32_t item = c * 32u + lane, groups = F::groups_in(item, a.cols);
        add_items<F, R, MT>(slot, lane, xs, x_pitch, a.items_pad, item, groups, acc);
        __syncwarp();
#pragma unroll
        for (int r = 0; r < R; ++r) fill_next();
        head = (head + R) % NS;
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int t = 0; t < MT; ++t) {
            float v = acc[r][t];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
            if (lane == 0 && t0 + t < a.n_vec)
                reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(a.y) + uint64_t{t0 + t} * a.y_stride)[row0 + r] =
                    gated_value(v, row0 + r, a.gate_n_v, a.gate_dt_bias, a.gate_a);
        }
}

/// grid (row ranges, tiles of MT x rows).  A warp walks its rows in passes of up to NR rows through a ring of NS slots.
template <class F, int MT, int NR, int NS, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1) gemv_raw_kernel(const __grid_constant__ RawArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr uint32_t kWarps = WARPS, kThreads = WARPS * 32;
    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31u;
    uint8_t* ring = smem + warp * (NS * slot_pitch<F>());
    uint8_t* xbuf = smem + kWarps * NS * slot_pitch<F>();
    const uint32_t x_pitch = a.items_pad * 256u, chunks = (a.cols + 2047u) / 2048u, t0 = blockIdx.y * MT;
    // the CTA's rows, then the warp's, as even contiguous shares
    const uint32_t c0 = static_cast<uint32_t>(uint64_t{a.rows} * blockIdx.x / gridDim.x), cn = static_cast<uint32_t>(uint64_t{a.rows} * (blockIdx.x + 1) / gridDim.x) - c0;
    const uint32_t r0 = c0 + static_cast<uint32_t>(uint64_t{cn} * warp / kWarps), n = c0 + static_cast<uint32_t>(uint64_t{cn} * (warp + 1) / kWarps) - r0;
    const uint32_t passes = n / NR + (n % NR != 0 ? 1u : 0u);
    auto pass_row = [&](uint32_t p) { return r0 + static_cast<uint32_t>(uint64_t{n} * p / passes); };
    uint32_t fp = 0, fc = 0, fr = 0, fslot = 0;  // the next slot to fill: pass, chunk, row of the pass
    uint32_t f_first = r0, f_rows = passes != 0 ? pass_row(1) - r0 : 0;
    auto fill_next = [&]() {
        if (fp < passes) {
            fill_slot<F>(a, f_first + fr, fc, ring + fslot * slot_pitch<F>(), lane);
            if (++fr == f_rows) {
                fr = 0;
                if (++fc == chunks) {
                    fc = 0, ++fp;
                    if (fp < passes) f_first = pass_row(fp), f_rows = pass_row(fp + 1) - f_first;
                }
            }
        }
        commit();  // an empty group where nothing is left: the counting stays the same
        fslot = fslot + 1 == NS ? 0 : fslot + 1;
    };
#pragma unroll 1
    for (int i = 0; i < NS; ++i) fill_next();
    for (uint32_t t = 0; t < MT; ++t) {  // x, laid out so that the 32 lanes' float4 of one position are on different banks
        const uint32_t tt = min(t0 + t, a.n_vec - 1u);
        const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const uint8_t*>(a.x) + uint64_t{tt} * a.x_stride);
        for (uint32_t f = threadIdx.x; f < a.cols / 4u; f += kThreads) {
            uint32_t item, i4;
            F::item_of(f, item, i4);
            *reinterpret_cast<float4*>(xbuf + t * x_pitch + (i4 * a.items_pad + (item ^ (i4 & 7u))) * 16u) = __ldg(src + f);
        }
    }
    __syncthreads();
    const uint32_t xs = smem_addr(xbuf);
    uint32_t head = 0;
    for (uint32_t p = 0; p < passes; ++p) {
        const uint32_t row = pass_row(p), rows = pass_row(p + 1) - row;
        switch (rows) {
            case 1: run_pass<F, 1, MT, NS>(a, row, t0, chunks, ring, head, lane, xs, x_pitch, fill_next); break;
            case 2:
                if constexpr (NR >= 2) run_pass<F, 2, MT, NS>(a, row, t0, chunks, ring, head, lane, xs, x_pitch, fill_next);
                break;
            case 3:
                if constexpr (NR >= 3) run_pass<F, 3, MT, NS>(a, row, t0, chunks, ring, head, lane, xs, x_pitch, fill_next);
                break;
            default:
                if constexpr (NR >= 4) run_pass<F, 4, MT, NS>(a, row, t0, chunks, ring, head, lane, xs, x_pitch, fill_next);
                break;
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

template <class F>
uint32_t smem_of(uint32_t items_pad, uint32_t mt, uint32_t slots) {  // slots: of all warps
    return slots * slot_pitch<F>() + mt * items_pad * 256u;
}

uint32_t padded_items(uint32_t cols) { return ((cols + 63u) / 64u + 7u) & ~7u; }

template <class F, int MT, int NR, int NS, int WARPS>
int launch_cfg(HaloCudaCtx* ctx, const GemvCall& c, cudaStream_t s) {
    RawArgs a{};
    a.w = c.w, a.w_stride = c.w_stride, a.row_bytes = c.row_bytes, a.w_end = c.w + (uint64_t{c.rows} - 1) * c.w_stride + c.row_bytes;
    a.x = c.x, a.x_stride = c.x_stride, a.y = c.y, a.y_stride = c.y_stride;
    a.rows = c.rows, a.cols = c.cols, a.n_vec = c.n_vec, a.items_pad = padded_items(c.cols);
    a.gate_dt_bias = c.gate_dt_bias, a.gate_a = c.gate_a, a.gate_n_v = c.gate_n_v;
    auto kern = gemv_raw_kernel<F, MT, NR, NS, WARPS>;
    if (int rc = allow_dynamic_smem(ctx, reinterpret_cast<const void*>(kern), kSmemMax)) return rc;
    // Row ranges: every CTA brings MT x rows into shared memory (about the time of twelve of its rows), and one CTA runs on an SM at a
    // time; the count with the least (waves * (rows of a CTA + 12)).
    const uint32_t sms = static_cast<uint32_t>(ctx->prop.multiProcessorCount), tiles = c.n_vec / MT + (c.n_vec % MT != 0 ? 1u : 0u);
    uint32_t gx = 1;
    uint64_t best = UINT64_MAX;
    for (uint32_t g = 1; g <= std::min(c.rows, sms); ++g) {
        const uint64_t waves = (uint64_t{g} * tiles + sms - 1) / sms, cost = waves * (uint64_t{c.rows / g} + (c.rows % g != 0 ? 1u : 0u) + 12u);
        if (cost < best) best = cost, gx = g;
    }
    for (uint32_t y0 = 0; y0 < tiles; y0 += 65535u) {
        const uint32_t n = std::min(tiles - y0, 65535u);
        RawArgs part = a;
        part.x = reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(a.x) + uint64_t{y0} * MT * a.x_stride);
        part.y = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(a.y) + uint64_t{y0} * MT * a.y_stride);
        part.n_vec = a.n_vec - y0 * MT;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(gx, n), cfg.blockDim = dim3(WARPS * 32), cfg.dynamicSmemBytes = smem_of<F>(a.items_pad, MT, NS * WARPS), cfg.stream = s, cfg.attrs = attr, cfg.numAttrs = 1;
        HC_CUDA(cudaLaunchKernelEx(&cfg, kern, part));
    }
    return 0;
}

/// Four x rows a CTA where they fit beside a ring of four rows (K up to 5632 for Q8_0, 9728 for Q4_0, 7680 for Q6_K), else four or two rows beside a ring of two,
/// else one.  A row's arithmetic is the same in all of them.
template <class F>
int launch_format(HaloCudaCtx* ctx, const GemvCall& c, cudaStream_t s) {
    const uint32_t ip = padded_items(c.cols);
    if (c.n_vec >= 3 && smem_of<F>(ip, 4, 64) <= kSmemMax) return launch_cfg<F, 4, 4, 8, 8>(ctx, c, s);
    if (c.n_vec >= 3 && smem_of<F>(ip, 4, 32) <= kSmemMax) return launch_cfg<F, 4, 2, 4, 8>(ctx, c, s);
    if (c.n_vec >= 2 && smem_of<F>(ip, 2, 32) <= kSmemMax) return launch_cfg<F, 2, 2, 4, 8>(ctx, c, s);
    if (smem_of<F>(ip, 1, 64) <= kSmemMax) return launch_cfg<F, 1, 2, 4, 16>(ctx, c, s);
    return launch_cfg<F, 1, 2, 4, 8>(ctx, c, s);
}

/// A lane's 64 weights leave most of a warp without work where K is short, and the kernel that reads both operands from global memory (16 - 32
/// weights a lane and step) is faster there: over 32 - 34816 rows and 1 - 64 x rows the geometric mean of this form's time over that one's is
/// Q8_0 1.02 - 1.07 at K = 512 and 0.83 - 0.98 at 640 (256: 1.1 - 1.7), Q4_0 1.0 - 1.1 at 256 and 0.75 - 1.0 at 384, Q6_K 0.85 - 1.44 at 1024
/// (above 1 from 1024 rows on) and 0.74 - 1.12 at 1280.  (Q6_K batches stay slower where a last slot is nearly empty, 10000 x 2304 at four rows 1.5
/// times, and where one x row fills the memory beside the ring, 1024 x 28672 at sixteen 1.26 times; one row is as fast or four times faster.)  The line depends on the type and K alone, since the two add in other orders: a row's bits
/// depend neither on the batch nor on how many rows of W a device holds.
uint32_t least_cols(uint32_t wtype) { return wtype == HALO_CUDA_T_Q8_0 ? 640u : wtype == HALO_CUDA_T_Q4_0 ? 384u : 1280u; }

}  // namespace

/// Raw Q8_0 / Q4_0 / Q6_K rows at even addresses, one x row beside the smallest ring (K up to 40448 for Q8_0, 48640 for Q4_0, 44032 for
/// Q6_K); a longer or a shorter K keeps the kernel that reads both operands from global memory.
bool gemv_raw_supports(const GemvCall& c) {
    if (c.cols == 0 || c.rows == 0 || c.n_vec == 0 || reinterpret_cast<uintptr_t>(c.w) % 2 != 0 || c.w_stride % 2 != 0) return false;
    if (reinterpret_cast<uintptr_t>(c.x) % 16 != 0 || c.x_stride % 16 != 0) return false;
    if (c.cols < least_cols(c.wtype) || c.cols > (1u << 20)) return false;
    const uint32_t ip = padded_items(c.cols);
    switch (c.wtype) {
        case HALO_CUDA_T_Q8_0: return smem_of<RawQ80>(ip, 1, 32) <= kSmemMax;
        case HALO_CUDA_T_Q4_0: return smem_of<RawQ40>(ip, 1, 32) <= kSmemMax;
        case HALO_CUDA_T_Q6_K: return smem_of<RawQ6K>(ip, 1, 32) <= kSmemMax;
        default: return false;
    }
}

int launch_gemv_raw(HaloCudaCtx* ctx, const GemvCall& c, cudaStream_t s) {
    if (c.n_vec / 4 > 65535u) return fail(HALO_CUDA_E_UNSUPPORTED, "MATMUL: n_vec %u exceeds the launch limit", c.n_vec);
    switch (c.wtype) {
        case HALO_CUDA_T_Q8_0: return launch_format<RawQ80>(ctx, c, s);
        case HALO_CUDA_T_Q4_0: return launch_format<RawQ40>(ctx, c, s);
        case HALO_CUDA_T_Q6_K: return launch_format<RawQ6K>(ctx, c, s);
        default: return fail(HALO_CUDA_E_UNSUPPORTED, "MATMUL: gemv_raw takes raw Q8_0 / Q4_0 / Q6_K weights");
    }
}

}  // namespace halo_cuda
