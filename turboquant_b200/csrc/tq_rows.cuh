// Quantization of 16-bit rows padded to 64, 128 or 256, a lane (two lanes of one of 256) a row: the cache write of large 16-bit writes at head sizes other than
// 128 (tq_write_rows.cu) and the flat quantizer of many rows (tq_flat_quant.cu).
//
// The arithmetic is the torch quantizer's (turboquant/quantizer.py:77-91 in the reference) for every element, as in tq_write.cu: eight
// interleaved sum-of-squares accumulators without FMA, IEEE sqrt and division, signs, butterflies h = 1 .. PD / 2 in order, code = number of
// boundaries below.  Compiled with -fmad=false.
//
// Mapping: a lane owns a row of up to 128 (two lanes one of 256) in registers, so that norm and butterflies are local and, but for stage h = 1, packed in
// pairs (f32x2).  A warp takes 32 (16) rows, in the cache write a box of neighbouring heads and tokens; the box arrives by tiled tensor
// copies (128-byte swizzle; short rows and missing ones as zeros), unit n + 2 while the warp works on unit n.  What is not done per element:
//   * x / norm is q = x r, e = fma(-q, norm, x), q' = fma(e, r, q) with r the correctly rounded reciprocal, which equals the IEEE quotient
//     while the intermediates stay normal and the norm's significand is not all ones.  Rows where they may not (a nonzero |x| < 2^-63, a norm
//     outside [2^-40, 2^40], infinities, NaN) are left out and done by the whole warp with divisions, see slow_row.
//   * The multiplication by 1 / sqrt(PD): the transform w is compared with the largest w whose rounded product is not above the boundary.
//   * The search: bins of w (whose standard deviation is about 1) hold at most one boundary each; {that boundary, boundaries in lower bins}
//     is one 8-byte lookup, 16 columns (served half a warp at a time: no two lanes meet in a bank).
//   * Rows of 96: the stages below 64 leave the 32 zeros of the padding alone.
// What bounds it is instruction issue (54 - 62 % of the active cycles in writes of 96, 256 and 64) and the FMA pipe's heavy half (49 - 57 %) at five (64) and
// three warps a scheduler; the flat quantizer of 65536 rows, two units a warp at most, waits for its first copies.  An instance for the cache write of
// 128, not kept (61 us for 32768 x 8), took 34 us with copies and stores alone, 2 - 6 % more with rows by 16-byte asynchronous copies in place of the
// tensor copies, and 17 % more with two lanes a row (five warps a scheduler).
#pragma once

#include <cuda.h>  // CUtensorMap and its enums only

#include <cmath>
#include <cstring>
#include <type_traits>

#include "tq_common.cuh"

namespace tq {

// bin(w) = round(64 w / sqrt(128)) + kRowBinZero: |w| <= sqrt(PD) <= 16 is bin 91 at most
constexpr int kRowBinZero = 96, kRowBins = 2 * kRowBinZero + 1;
constexpr float kRowBinMagic = 8388608.0f + (float)kRowBinZero;

struct LaneRowsParams {
    alignas(64) CUtensorMap map[2];   // K, V as [tokens][heads][head_dim], boxes of 64 elements x box_heads x rows / box_heads; flat: [rows][1][dim]
    uint8_t* dst;                     // the cache; flat: packed codes, rows dense
    float* norms;                     // flat
    const void* slot_mapping;
    const float* signs;
    int64_t num_tokens, slab_bytes, total_slots;      // flat: num_tokens rows of one head
    int heads, head_dim, slot_bytes, pad_end;   // pad_end: zero the slot's bytes from its norms to here (0: leave them)
    int box_heads, box_shift, head_boxes;       // heads of a box (a power of two), its logarithm, boxes that make up the heads
    int slot_is_i64;
    int bits, cache_order, count;     // flat: bits of a code, first value of a byte in its high bits; count of boundaries
    float bin_scale, scale;
    float2 bins[kRowBins];            // {the largest w not above the bin's boundary (or +inf), the bits of: boundaries in lower bins}
    float bounds[15];                 // +inf from count on
};

template <int PD>
struct LaneRowsShape {
    static constexpr int kLanes = PD == 256 ? 2 : 1, kRows = 32 / kLanes, kPairs = PD / kLanes / 2;   // lanes of a row, rows of a unit, packed pairs a lane
    static constexpr int kWarps = kPairs == 32 ? 20 : 12, kThreads = 32 * kWarps;                          // 64 values a lane: 96 registers, 128: 168
    static constexpr int kBoxes = PD / 64, kBoxBytes = kRows * 128, kStage = kBoxes * kBoxBytes;
    static constexpr uint32_t kTableBytes = kRowBins * 128, kMaskBytes = PD * 2 + 32, kSlotBytes = kWarps * 512;
    static constexpr size_t kSmem = 1024 + 2 * kWarps * kStage + kTableBytes + kMaskBytes + kSlotBytes + 2 * kWarps * 8;
    static_assert(kSmem <= 232448, "shared memory");
};

// Tokens that the cache write dropped (slot outside the cache), and copies of rows that never landed; read back by tq_fault_counts.
static __device__ int32_t g_rows_dropped = 0;

template <typename T>
struct RowWord;
template <>
struct RowWord<__nv_bfloat16> {
    static constexpr bool kTiny = true;      // holds values whose squares are no normal numbers
    static __device__ __forceinline__ P2 unpack(uint32_t w) { return pk(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
};
template <>
struct RowWord<__half> {
    static constexpr bool kTiny = false;
    static __device__ __forceinline__ P2 unpack(uint32_t w) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
        return pk(f.x, f.y);
    }
};

__device__ __forceinline__ void box_g2s_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ uint4 lds_u4(uint32_t at) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t at) {
    uint32_t v;
    asm volatile("{\n\t.reg .u16 t;\n\tld.shared.u16 t, [%1];\n\tcvt.u32.u16 %0, t;\n\t}" : "=r"(v) : "r"(at) : "memory");
    return v;
}

// The code of w at bit `at` of a word: the table entry's count, and one more above its boundary.
__device__ __forceinline__ void code_into(uint32_t& word, float w, uint32_t entry, int at) {
    float most;
    uint32_t below;
    asm("ld.shared.v2.b32 {%0,%1}, [%2];" : "=f"(most), "=r"(below) : "r"(entry));
    word += below << at;
    asm("{\n\t.reg .pred q;\n\tsetp.gt.f32 q, %1, %2;\n\t@q add.u32 %0, %0, %3;\n\t}" : "+r"(word) : "f"(w), "f"(most), "r"(1u << at));
}

// One row by the whole warp, for what the common path leaves out (a row at a time: where all rows are such ones the call takes two to four times what
// the kernels take that divide for every element, 8000 x 8 rows of 96 with an infinity 179 us against 46, 60000 x 128 with signs of 1.5 82 against 15).  Lane l on elements E l .. E l + E - 1, with divisions and with the signs as factors; the codes, four bits each in the order of
// code_into, replace the row's first PD / 2 bytes in `row`.  elem(i): shared-memory address of element i.
template <typename T, int PD, bool FLAT, typename F>
__device__ __noinline__ void slow_row(const LaneRowsParams& p, F elem, uint32_t row, float norm, int lane) {
    constexpr int E = PD / 32;
    constexpr uint32_t kAll = 0xffffffffu;
    float x[E];
#pragma unroll
    for (int i = 0; i < E; i++) {
        const uint32_t h = lds_u16(elem(E * lane + i));
        float a, b;
        up(RowWord<T>::unpack(h), a, b);
        // the sign vector is as long as the padded row; the padding itself is zero
        x[i] = E * lane + i < p.head_dim ? __fmul_rn(__fdiv_rn(a, norm), p.signs[E * lane + i]) : 0.0f;
    }
    __syncwarp();      // the row has been read
#pragma unroll
    for (int h = 1; h < E; h <<= 1)
#pragma unroll
        for (int i = 0; i < E; i++)
            if (!(i & h)) {
                const float a = x[i], c = x[i + h];
                x[i] = __fadd_rn(a, c);
                x[i + h] = __fsub_rn(a, c);
            }
#pragma unroll
    for (int d = 1; d < 32; d <<= 1)
#pragma unroll
        for (int i = 0; i < E; i++) {
            const float o = __shfl_xor_sync(kAll, x[i], d);
            x[i] = (lane & d) ? __fsub_rn(o, x[i]) : __fadd_rn(x[i], o);
        }
    uint32_t codes = 0;
#pragma unroll
    for (int i = 0; i < E; i++) {
        const float y = __fmul_rn(x[i], p.scale);
        uint32_t c = 0;
#pragma unroll
        for (int k = 0; k < 15; k++) c += p.bounds[k] < y ? 1u : 0u;      // fewer bits: the rest are +inf
        if (y != y) c = FLAT ? p.count : 15;      // torch's bucketize sends NaN to the last bucket
        codes |= c << (4 * (FLAT ? i : i ^ 1));
    }
    const uint32_t at = row + lane * (E / 2);
    if constexpr (E == 2) asm volatile("st.shared.u8 [%0], %1;" ::"r"(at), "r"(codes) : "memory");
    else if constexpr (E == 4) asm volatile("st.shared.u16 [%0], %1;" ::"r"(at), "h"((unsigned short)codes) : "memory");
    else asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(codes) : "memory");
}

// Words of eight 4-bit codes, first value of a byte low, as a row of `bits`-bit codes in either order: bits 3 and 4 word by word, 2 and 1 into half and a quarter
// of the words.
template <int N>
__device__ __forceinline__ void pack_codes(uint32_t (&w)[N], int bits, bool high_first) {
    if (bits >= 3) {
        const uint32_t mask = bits == 4 ? 0x0F0F0F0Fu : 0x07070707u;
        if (bits == 4 && !high_first) return;
#pragma unroll
        for (int i = 0; i < N; i++) {
            const uint32_t first = w[i] & mask, second = (w[i] >> 4) & mask;
            w[i] = high_first ? (first << bits) | second : first | (second << bits);
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < N; i++) {      // a byte's two codes side by side, then two bytes' in one
        const uint32_t a = w[i] & 0x0F0F0F0Fu, b = (w[i] >> 4) & 0x0F0F0F0Fu;
        const uint32_t two = high_first ? (a << bits) | b : a | (b << bits), c = two & 0x00FF00FFu, d = (two >> 8) & 0x00FF00FFu;
        const uint32_t four = high_first ? (c << (2 * bits)) | d : c | (d << (2 * bits));      // in bytes 0 and 2
        if (bits == 2) {
            w[i] = (four & 0xFFu) | ((four >> 8) & 0xFF00u);
        } else {
            const uint32_t e = four & 0xFFu, f = four >> 16;
            w[i] = high_first ? (e << 4) | f : e | (f << 4);
        }
    }
    if (bits == 2) {
#pragma unroll
        for (int i = 0; i < N / 2; i++) w[i] = w[2 * i] | (w[2 * i + 1] << 16);
    } else {
#pragma unroll
        for (int i = 0; i < N / 4; i++) w[i] = w[4 * i] | (w[4 * i + 1] << 8) | (w[4 * i + 2] << 16) | (w[4 * i + 3] << 24);
    }
}

// HD: elements of an input row, 0: p.head_dim.  FLAT: rows to rows, else K and V into the cache.
template <typename T, int PD, int HD, bool FLAT>
__global__ void __launch_bounds__(LaneRowsShape<PD>::kThreads, 1) lane_rows_kernel(const __grid_constant__ LaneRowsParams p) {
    using S = LaneRowsShape<PD>;
    using W = RowWord<T>;
    constexpr int kLive = HD && S::kLanes == 1 ? HD / 2 : S::kPairs;      // pairs that hold more than padding
    constexpr uint32_t kAll = 0xffffffffu;
    extern __shared__ uint8_t wr_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m = lane / S::kRows, row = lane % S::kRows;      // the eight lanes served together are of different rows
    const uint32_t raw = smem_u32(wr_smem), smem0 = (raw + 1023u) & ~1023u;      // the swizzle is a function of the address
    const uint32_t ring = smem0 + (uint32_t)warp * 2 * S::kStage, table = smem0 + 2 * S::kWarps * S::kStage, masks = table + S::kTableBytes;
    const uint32_t my_slot = masks + S::kMaskBytes + (uint32_t)warp * 512 + 8u * lane;
    uint64_t* const bar = reinterpret_cast<uint64_t*>(wr_smem + (masks + S::kMaskBytes + S::kSlotBytes - raw)) + 2 * warp;

    grid_launch_dependents();
    if (lane == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_barrier_init();
    }
    for (int i = tid; i < kRowBins * 8; i += S::kThreads) {
        const float2 e = p.bins[i >> 3];
        asm volatile("st.shared.v4.f32 [%0], {%1,%2,%1,%2};" ::"r"(table + 16u * i), "f"(e.x), "f"(e.y) : "memory");
    }
    if (FLAT) grid_dependency_wait();
    // The signs (in the cache write constants of the context like the table, hence ahead of the wait) as masks of word pairs; a second lane's start 16 bytes
    // on and have their last half changed (see the last stage).  Signs other than +-1 are factors: then all rows go by slow_row.
    bool odd_sign = false;
    for (int i = tid; i < PD / 2; i += S::kThreads) {
        const bool in0 = 2 * i < p.head_dim, in1 = 2 * i + 1 < p.head_dim;
        const float a = in0 ? p.signs[2 * i] : 1.0f, b = in1 ? p.signs[2 * i + 1] : 1.0f;
        odd_sign |= fabsf(a) != 1.0f || fabsf(b) != 1.0f;
        uint32_t w = (a < 0.0f ? 0x8000u : 0u) | (b < 0.0f ? 0x80000000u : 0u);
        if (S::kLanes == 2 && i >= PD * 3 / 8) w ^= 0x80008000u;
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(masks + 4u * i + (S::kLanes == 2 && i >= PD / 4 ? 16u : 0u)), "r"(w) : "memory");
    }
    if (!FLAT) grid_dependency_wait();  // K, V, the slots and the cache belong to earlier kernels
    const bool all_slow = __syncthreads_or(odd_sign);

    // ---- units: box_heads heads x kRows / box_heads tokens of K or V, K and V in turn (flat: kRows rows); neighbouring units go to different SMs ----
    const int box_tokens = S::kRows >> p.box_shift;
    const int64_t token_boxes = (p.num_tokens + box_tokens - 1) / box_tokens, units = (FLAT ? 1 : 2) * token_boxes * p.head_boxes;
    const int64_t step = (int64_t)gridDim.x * S::kWarps;
    int64_t unit = (int64_t)warp * gridDim.x + blockIdx.x;
    // first token and head of unit u
    auto place = [&](int64_t u, int& t0, int& h0) {
        const int64_t k = FLAT ? u : u >> 1;
        int64_t tb = k;
        h0 = 0;
        if (p.head_boxes > 1) {
            tb = k < 0x7fffffff ? (int64_t)((uint32_t)k / (uint32_t)p.head_boxes) : k / p.head_boxes;
            h0 = (int)(k - tb * p.head_boxes) << p.box_shift;
        }
        t0 = (int)(tb * box_tokens);      // num_tokens fits the copy's 32-bit coordinate
    };
    // The box of unit u and the slots of its rows on their way to stage s.  (The slots go by shared memory too: in registers they were spilled, which waits for them.)
    auto fetch = [&](int64_t u, int s) {
        if (u < units) {
            int t0, h0;
            place(u, t0, h0);
            __syncwarp();
            fence_proxy_async();   // the stage has been read out by ordinary loads
            if (lane == 0) {
                mbar_arrive_expect_tx(&bar[s], S::kStage);
#pragma unroll
                for (int b = 0; b < S::kBoxes; b++) box_g2s_3d(ring + s * S::kStage + b * S::kBoxBytes, &p.map[FLAT ? 0 : u & 1], 64 * b, h0, t0, &bar[s]);
            }
            const int64_t t = (int64_t)t0 + (row >> p.box_shift);
            if (!FLAT && t < p.num_tokens) {
                if (p.slot_is_i64) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(my_slot + s * 256), "l"(reinterpret_cast<const int64_t*>(p.slot_mapping) + t) : "memory");
                else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(my_slot + s * 256), "l"(reinterpret_cast<const int32_t*>(p.slot_mapping) + t) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    const uint32_t table_lane = table + 8u * (lane & 15) - 0x80000000u;      // (the bits of 2^23 + k) * 128 = 2^31 + 128 k modulo 2^32
    const uint32_t my_masks = masks + (uint32_t)m * (PD + 16);
    fetch(unit, 0);
    fetch(unit + step, 1);
    uint32_t phases = 0;
    for (int s = 0; unit < units; unit += step, s ^= 1) {
        if (!__all_sync(kAll, mbar_wait(&bar[s], (phases >> s) & 1))) {
            copy_lost(&g_rows_dropped, lane, &bar[s], (phases >> s) & 1, unit + step < units, &bar[s ^ 1], (phases >> (s ^ 1)) & 1);
            return;
        }
        phases ^= 1u << s;
        const uint32_t stage = ring + s * S::kStage;
        // 16-byte piece c (8 elements) of this lane's values
        const uint32_t my_row = stage + (uint32_t)m * (S::kBoxes / 2) * S::kBoxBytes + row * 128 + ((row & 7) << 4);
        auto piece = [&](int c) { return (my_row ^ ((c & 7) << 4)) + (c >> 3) * S::kBoxBytes; };

        // ---- the row with its signs, and the norm ----
        P2 x[S::kPairs], acc[4];
        uint32_t least = 0x7f7f7f7fu;      // smallest magnitudes of the even and of the odd elements
#pragma unroll
        for (int k = 0; k < 4; k++) acc[k] = pk(0.0f, 0.0f);
#pragma unroll
        for (int c = 0; c < kLive / 4; c++) {
            const uint4 v = lds_u4(piece(c)), g = lds_u4(my_masks + 16 * c);
            const uint32_t w[4] = {v.x ^ g.x, v.y ^ g.y, v.z ^ g.z, v.w ^ g.w};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (W::kTiny && (HD || 8 * c + (S::kLanes == 2 ? PD / 2 * m : 0) < p.head_dim))      // (the padding's zeros do not count)
                    asm("min.xorsign.abs.bf16x2 %0, %0, %1;" : "+r"(least) : "r"(w[k]));
                x[4 * c + k] = W::unpack(w[k]);
                acc[k] = fma2(x[4 * c + k], x[4 * c + k], acc[k]);      // squares of 16-bit values are exact: one rounding, that of the sum
            }
        }
        if constexpr (S::kLanes == 2) {      // the second lane's sums go on from the first's
#pragma unroll
            for (int k = 0; k < 4; k++) {
                float a, b;
                up(acc[k], a, b);
                a = __shfl_xor_sync(kAll, a, 16);
                b = __shfl_xor_sync(kAll, b, 16);
                acc[k] = m ? pk(a, b) : pk(0.0f, 0.0f);
            }
#pragma unroll
            for (int c = 0; c < S::kPairs / 4; c++)
#pragma unroll
                for (int k = 0; k < 4; k++) acc[k] = fma2(x[4 * c + k], x[4 * c + k], acc[k]);
        }
        float sum, a1;
        up(acc[0], sum, a1);
        sum = __fadd_rn(sum, a1);
#pragma unroll
        for (int k = 1; k < 4; k++) {
            float a, b;
            up(acc[k], a, b);
            sum = __fadd_rn(__fadd_rn(sum, a), b);
        }
        if constexpr (S::kLanes == 2) sum = __shfl_sync(kAll, sum, lane | 16);
        float norm = __fsqrt_rn(sum);
        // clamp(min=1e-8); a NaN stays a NaN, in the canonical quiet pattern torch produces
        if (!(norm >= 1e-8f)) norm = (norm != norm) ? __uint_as_float(0x7fc00000u) : 1e-8f;
        bool slow = all_slow || !(norm >= 9.0949470e-13f && norm <= 1.0995116e12f) || (__float_as_uint(norm) & 0x7fffffu) == 0x7fffffu;
        if (W::kTiny) {
            const bool small = (least & 0x7fffu) < 0x2000u || ((least >> 16) & 0x7fffu) < 0x2000u;      // 2^-63
            if (__any_sync(kAll, small)) {      // zeros are no trouble
                bool tiny = false;
#pragma unroll
                for (int i = 0; i < kLive; i++) {
                    float a, b;
                    up(x[i], a, b);
                    tiny |= (a != 0.0f && fabsf(a) < 1.0842022e-19f) || (b != 0.0f && fabsf(b) < 1.0842022e-19f);
                }
                if (S::kLanes == 2) tiny |= __shfl_xor_sync(kAll, (int)tiny, 16) != 0;
                slow |= tiny;
            }
        }
        if (__any_sync(kAll, slow)) {      // such a row forms no lookup address
            if (slow) {
#pragma unroll
                for (int i = 0; i < kLive; i++) x[i] = pk(0.0f, 0.0f);
            }
        }

        // ---- x / norm, butterflies ----
        {
            const float rcp = __frcp_rn(slow ? 1.0f : norm);
            const P2 rcp2 = pk(rcp, rcp), nneg2 = pk(-norm, -norm);
#pragma unroll
            for (int i = 0; i < kLive; i++) {
                const P2 q = mul2(x[i], rcp2);
                float a, b;
                up(fma2(fma2(q, slow ? rcp2 : nneg2, x[i]), rcp2, q), a, b);      // x - q norm is exact
                x[i] = pk(__fadd_rn(a, b), __fsub_rn(a, b));
            }
        }
#pragma unroll
        for (int h = 1; h < S::kPairs; h <<= 1)
#pragma unroll
            for (int i = 0; i < S::kPairs; i++)
                if (!(i & h) && (i < kLive || 4 * h > S::kPairs)) {      // sets of padding up to the stage that meets it
                    if (kLive < S::kPairs && 4 * h == S::kPairs && i + h >= kLive) {
                        x[i + h] = x[i];      // x + 0 and x - 0
                        continue;
                    }
                    const P2 a = x[i], b = x[i + h];
                    x[i] = add2(a, b);
                    x[i + h] = sub2(a, b);
                }
        if constexpr (S::kLanes == 2) {
            // The last stage is between the lanes: each keeps its first half of values and sends the other.  For that the second lane holds its values
            // with the halves exchanged, as it does when the inputs of the second half change sign (equal values; zeros may change sign, which no code depends on).
            const P2 flip = m ? pk(-1.0f, -1.0f) : pk(1.0f, 1.0f);
            constexpr int kHalf = S::kPairs / 2;
#pragma unroll
            for (int i = 0; i < kHalf; i++) {
                float a, b;
                up(x[kHalf + i], a, b);
                const P2 mine = x[i], other = pk(__shfl_xor_sync(kAll, a, 16), __shfl_xor_sync(kAll, b, 16));
                x[i] = add2(mine, other);
                x[kHalf + i] = mul2(sub2(mine, other), flip);
            }
        }
        // codes: words of 8 dims, the even dim of a byte in its high nibble (flat: in its low one, for now)
        uint32_t codes[S::kPairs / 4];
        const P2 bin_scale2 = pk(p.bin_scale, p.bin_scale), magic2 = pk(kRowBinMagic, kRowBinMagic);
#pragma unroll
        for (int c = 0; c < S::kPairs / 4; c++) codes[c] = 0;
#pragma unroll
        for (int i = 0; i < S::kPairs; i++) {
            float w0, w1, k0, k1;
            up(x[i], w0, w1);
            up(fma2(x[i], bin_scale2, magic2), k0, k1);
            code_into(codes[i / 4], w0, __float_as_uint(k0) * 128u + table_lane, 8 * (i & 3) + (FLAT ? 0 : 4));
            code_into(codes[i / 4], w1, __float_as_uint(k1) * 128u + table_lane, 8 * (i & 3) + (FLAT ? 4 : 0));
        }

        // where 16 code bytes of the lane lie in the row's: two lanes hold a quarter of its lower and of its upper half each
        auto part = [m](int c) {
            constexpr int kHalf = S::kPairs / 32;
            return S::kLanes == 2 ? PD / 4 * (c / kHalf) + PD / 8 * m + 16 * (c % kHalf) : 16 * c;
        };
        // ---- rows left out ----
        int t0, h0;
        place(unit, t0, h0);
        const int which = FLAT ? 0 : (int)(unit & 1), h = h0 + (row & (p.box_heads - 1));
        int64_t slot = t0 + row;      // flat: the row
        if constexpr (!FLAT) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");      // all but the next unit's (a lane reads what it copied itself)
            uint32_t slot_lo, slot_hi;
            asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(slot_lo), "=r"(slot_hi) : "r"(my_slot + s * 256) : "memory");
            slot = p.slot_is_i64 ? (int64_t)(((uint64_t)slot_hi << 32) | slot_lo) : (int64_t)(int32_t)slot_lo;
        }
        if (t0 + (row >> p.box_shift) >= p.num_tokens) slot = -1;
        if (!FLAT && slot >= p.total_slots) {
            if (m == 0 && h == 0 && which == 0) atomicAdd(&g_rows_dropped, 1);  // once per token
            slot = -1;
        }
        uint32_t todo = __ballot_sync(kAll, slow && slot >= 0 && m == 0);
        if (todo) {
            const bool mine = slow;
            while (todo) {
                const int r = __ffs(todo) - 1;
                todo &= todo - 1;
                slow_row<T, PD, FLAT>(p, [&](int i) { return stage + (i >> 6) * S::kBoxBytes + r * 128 + ((((i >> 3) ^ r) & 7) << 4) + (i & 7) * 2; },
                                stage + r * 128, __shfl_sync(kAll, norm, r), lane);
            }
            __syncwarp();
            if (mine) {
#pragma unroll
                for (int c = 0; c < S::kPairs / 16; c++) {
                    const uint4 v = lds_u4(stage + row * 128 + part(c));
                    codes[4 * c] = v.x; codes[4 * c + 1] = v.y; codes[4 * c + 2] = v.z; codes[4 * c + 3] = v.w;
                }
            }
        }

        if (!FLAT && slot >= 0) {
            // slot = block * block_size + entry and the cache is [block][entry][head][slot_bytes]
            uint8_t* dst = p.dst + (size_t)which * p.slab_bytes + ((size_t)slot * p.heads + h) * p.slot_bytes;
#pragma unroll
            for (int c = 0; c < S::kPairs / 16; c++)
                *reinterpret_cast<uint4*>(dst + part(c)) =
                    make_uint4(codes[4 * c], codes[4 * c + 1], codes[4 * c + 2], codes[4 * c + 3]);
            if (m == 0) {
                const uint32_t nh = (norm != norm) ? 0x7e00u : (uint32_t)__half_as_ushort(__float2half_rn(norm));
                if constexpr (PD == 64) *reinterpret_cast<uint16_t*>(dst + 32) = (uint16_t)nh;
                else if constexpr (PD == 128) *reinterpret_cast<uint32_t*>(dst + 64) = nh | (nh << 16);
                else *reinterpret_cast<uint2*>(dst + 128) = make_uint2(nh | (nh << 16), nh | (nh << 16));
                for (int b = PD / 2 + 2 * (PD / 64); b < p.pad_end; b += 2) *reinterpret_cast<uint16_t*>(dst + b) = 0;
            }
        }
        if constexpr (FLAT) {
            pack_codes(codes, p.bits, p.cache_order);
            if (slot >= 0) {
                const int fewer = p.bits == 2 ? 1 : p.bits == 1 ? 2 : 0;      // a row is PD / 2 bytes, or half or a quarter of it
                uint8_t* dst = p.dst + slot * (int64_t)(PD / 2 >> fewer);
                if (S::kLanes == 2) {      // a quarter of the row's lower and of its upper half
                    constexpr int kHalf = S::kPairs / 8;      // words of four bits
                    dst += PD / 8 * m >> fewer;
                    uint8_t* const upper = dst + (PD / 4 >> fewer);
                    if (fewer == 0) {
#pragma unroll
                        for (int c = 0; c < kHalf; c += 4) {
                            *reinterpret_cast<uint4*>(dst + 4 * c) = make_uint4(codes[c], codes[c + 1], codes[c + 2], codes[c + 3]);
                            *reinterpret_cast<uint4*>(upper + 4 * c) = make_uint4(codes[kHalf + c], codes[kHalf + c + 1], codes[kHalf + c + 2], codes[kHalf + c + 3]);
                        }
                    } else if (fewer == 1) {
                        *reinterpret_cast<uint4*>(dst) = make_uint4(codes[0], codes[1], codes[2], codes[3]);
                        *reinterpret_cast<uint4*>(upper) = make_uint4(codes[4], codes[5], codes[6], codes[7]);
                    } else {
                        *reinterpret_cast<uint2*>(dst) = make_uint2(codes[0], codes[1]);
                        *reinterpret_cast<uint2*>(upper) = make_uint2(codes[2], codes[3]);
                    }
                } else {
                    constexpr int kWords = S::kPairs / 4;
#pragma unroll
                    for (int c = 0; c < kWords; c += 2)
                        if (c < (kWords >> fewer)) {
                            if (c + 4 <= (kWords >> fewer) && c % 4 == 0) *reinterpret_cast<uint4*>(dst + 4 * c) = make_uint4(codes[c], codes[c + 1], codes[c + 2], codes[c + 3]);
                            else if (c % 4 == 0) *reinterpret_cast<uint2*>(dst + 4 * c) = make_uint2(codes[c], codes[c + 1]);
                        }
                }
                if (m == 0) p.norms[slot] = norm;
            }
        }
        fetch(unit + 2 * step, s);
    }
}

int device_sm_count(int* out);
bool encode_tensor_map(CUtensorMap* map, CUtensorMapDataType type, int rank, const void* base, const cuuint64_t* dims, const cuuint64_t* strides,
                       const cuuint32_t* box, CUtensorMapSwizzle swizzle);

// The search's table for one padded size and width, made once by the kernel's own float operations.
struct RowBins {
    float2 bins[kRowBins];
    float bounds[15], bin_scale, scale;
    bool ok;
};
static RowBins make_row_bins(int padded, int bits) {
    RowBins r{};
    float cen[16];
    const int count = (1 << bits) - 1;
    host_codebook(padded, bits, cen, r.bounds);
    r.scale = (float)(1.0 / std::sqrt((double)padded));
    r.bin_scale = (float)(64.0 / std::sqrt(128.0));
    r.ok = true;
    auto product = [&](float w) { volatile float y = w * r.scale; return (float)y; };
    float most[15];
    int bin_of[15];
    for (int i = 0; i < count; i++) {
        float w = r.bounds[i] / r.scale;      // the largest w with product(w) <= bounds[i]
        while (product(w) > r.bounds[i]) w = std::nextafterf(w, -INFINITY);
        while (product(std::nextafterf(w, INFINITY)) <= r.bounds[i]) w = std::nextafterf(w, INFINITY);
        most[i] = w;
        volatile float kf = fmaf(w, r.bin_scale, kRowBinMagic);
        const float k = kf;
        uint32_t bits;
        memcpy(&bits, &k, 4);
        bin_of[i] = (int)(bits - 0x4B000000u);
        if (bin_of[i] < 0 || bin_of[i] >= kRowBins || (i > 0 && bin_of[i] <= bin_of[i - 1])) r.ok = false;
    }
    for (int k = 0; k < kRowBins; k++) {
        uint32_t below = 0;
        float inside = INFINITY;      // no boundary in this bin: the comparison is never true
        for (int i = 0; i < count; i++) {
            if (bin_of[i] < k) below++;
            if (bin_of[i] == k) inside = most[i];
        }
        float bits;
        memcpy(&bits, &below, 4);
        r.bins[k] = make_float2(inside, bits);
    }
    for (int i = count; i < 15; i++) r.bounds[i] = INFINITY;
    return r;
}
template <typename T, int PD, int HD, bool FLAT>
static int launch_lane_rows(const LaneRowsParams& p, int sms, cudaStream_t stream) {
    using S = LaneRowsShape<PD>;
    static bool configured[64] = {};  // per template instance and device
    int dev = 0;
    TQ_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        TQ_CUDA(cudaFuncSetAttribute(lane_rows_kernel<T, PD, HD, FLAT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const int tokens = S::kRows >> p.box_shift;
    const int64_t units = (FLAT ? 1 : 2) * ((p.num_tokens + tokens - 1) / tokens) * p.head_boxes;
    TQ_CUDA(launch_serialized(lane_rows_kernel<T, PD, HD, FLAT>, dim3((unsigned)(units < sms ? units : sms)), dim3(S::kThreads), S::kSmem, stream, p));
    return TQ_OK;
}
inline int lane_rows_of(int padded) { return padded == 256 ? LaneRowsShape<256>::kRows : LaneRowsShape<64>::kRows; }

}  // namespace tq
