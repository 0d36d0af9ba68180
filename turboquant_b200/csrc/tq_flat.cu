// Flat (non-paged) quantizer API kernels: TurboQuantMSE.quantize / dequantize and the
// Walsh-Hadamard rotation for any head size up to 256 and 1..4 bits
// (turboquant/quantizer.py:77-106, turboquant/hadamard.py:21-78 in the reference).
//
// These back the Python algorithm API; the paged cache write has its own specialised kernel.
// One warp owns one row, staged in a per-warp shared buffer; the arithmetic order is the same
// as in the cache-write kernel (eight interleaved no-FMA accumulators for the norm, IEEE
// division, butterflies in stage order, one scale multiply), so 4-bit codes agree with it
// bit for bit.  Compiled with -fmad=false.
#include <cmath>
#include <cstring>

#include "tq_common.cuh"

namespace tq {

constexpr int kMaxDim = 256;
constexpr int kFlatWarps = 4;

struct FlatParams {
    const void* x;         // quantize: input rows; fwht: fp32 input
    const float* signs;    // [padded] (pre-rotation signs); may be null for fwht
    const float* post_signs;
    uint8_t* packed;
    float* norms;
    float* out;
    int64_t n;
    int dim, padded, out_dim, bits, cache_order;
    float scale;           // (float)(1/sqrt(padded))
    float table[16];       // boundaries (quantize) or centroids (dequantize)
};

__device__ __forceinline__ void warp_fwht(float* buf, int padded, int lane) {
    for (int h = 1; h < padded; h <<= 1) {
        for (int idx = lane; idx < padded / 2; idx += 32) {
            const int i = (idx / h) * 2 * h + (idx % h);
            const float a = buf[i], b = buf[i + h];
            buf[i] = __fadd_rn(a, b);
            buf[i + h] = __fsub_rn(a, b);
        }
        __syncwarp();
    }
}

template <typename T>
__global__ void __launch_bounds__(kFlatWarps * 32) quantize_flat_kernel(const __grid_constant__ FlatParams p) {
    __shared__ float buf_s[kFlatWarps][kMaxDim];
    __shared__ uint8_t idx_s[kFlatWarps][kMaxDim];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* buf = buf_s[warp];
    uint8_t* idx = idx_s[warp];
    const int nb = (1 << p.bits) - 1;
    const int vpb = 8 / p.bits;
    const int nbytes = (p.padded + vpb - 1) / vpb;
    for (int64_t r = (int64_t)blockIdx.x * kFlatWarps + warp; r < p.n; r += (int64_t)gridDim.x * kFlatWarps) {
        const T* row = reinterpret_cast<const T*>(p.x) + r * p.dim;
        for (int i = lane; i < p.padded; i += 32) buf[i] = i < p.dim ? to_f32(row[i]) : 0.0f;
        __syncwarp();
        // norm: eight interleaved accumulators over the first dim & ~7 elements, then the tail
        float acc = 0.0f;
        const int full = p.dim & ~7;
        if (lane < 8)
            for (int j = lane; j < full; j += 8) acc = __fadd_rn(acc, __fmul_rn(buf[j], buf[j]));
        float s = 0.0f;
        for (int k = 0; k < 8; k++) {
            const float a = __shfl_sync(0xffffffffu, acc, k);
            s = k == 0 ? a : __fadd_rn(s, a);
        }
        for (int j = full; j < p.dim; j++) s = __fadd_rn(s, __fmul_rn(buf[j], buf[j]));
        float norm = __fsqrt_rn(s);
        if (!(norm >= 1e-8f)) norm = (norm != norm) ? __uint_as_float(0x7fc00000u) : 1e-8f;
        for (int i = lane; i < p.padded; i += 32)
            buf[i] = i < p.dim ? __fmul_rn(__fdiv_rn(buf[i], norm), p.signs[i]) : 0.0f;
        __syncwarp();
        warp_fwht(buf, p.padded, lane);
        for (int i = lane; i < p.padded; i += 32) {
            const float y = __fmul_rn(buf[i], p.scale);
            int c = 0;
            for (int k = 0; k < nb; k++) c += (p.table[k] < y) ? 1 : 0;
            if (y != y) c = nb;  // torch's lower bound puts NaN in the last bucket
            idx[i] = (uint8_t)c;
        }
        __syncwarp();
        uint8_t* dst = p.packed + r * nbytes;
        for (int b = lane; b < nbytes; b += 32) {
            uint32_t v = 0;
            for (int i = 0; i < vpb; i++) {
                const int e = b * vpb + i;
                const uint32_t code = e < p.padded ? idx[e] : 0u;
                if (p.cache_order) v |= code << ((vpb - 1 - i) * p.bits);
                else v |= code << (i * p.bits);
            }
            dst[b] = (uint8_t)v;
        }
        if (lane == 0) p.norms[r] = norm;
        __syncwarp();
    }
}

__global__ void __launch_bounds__(kFlatWarps * 32) dequantize_flat_kernel(const __grid_constant__ FlatParams p) {
    __shared__ float buf_s[kFlatWarps][kMaxDim];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* buf = buf_s[warp];
    const int vpb = 8 / p.bits, mask = (1 << p.bits) - 1;
    const int nbytes = (p.padded + vpb - 1) / vpb;
    for (int64_t r = (int64_t)blockIdx.x * kFlatWarps + warp; r < p.n; r += (int64_t)gridDim.x * kFlatWarps) {
        const uint8_t* src = p.packed + r * nbytes;
        for (int e = lane; e < p.padded; e += 32) {
            const int i = e % vpb;
            const int sh = p.cache_order ? (vpb - 1 - i) * p.bits : i * p.bits;
            buf[e] = p.table[(src[e / vpb] >> sh) & mask];
        }
        __syncwarp();
        warp_fwht(buf, p.padded, lane);
        const float norm = p.norms[r];
        for (int e = lane; e < p.dim; e += 32)
            p.out[r * p.dim + e] = __fmul_rn(__fmul_rn(__fmul_rn(buf[e], p.scale), p.signs[e]), norm);
        __syncwarp();
    }
}

__global__ void __launch_bounds__(kFlatWarps * 32) fwht_kernel(const __grid_constant__ FlatParams p) {
    __shared__ float buf_s[kFlatWarps][kMaxDim];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* buf = buf_s[warp];
    const float* x = reinterpret_cast<const float*>(p.x);
    for (int64_t r = (int64_t)blockIdx.x * kFlatWarps + warp; r < p.n; r += (int64_t)gridDim.x * kFlatWarps) {
        for (int i = lane; i < p.padded; i += 32) {
            float v = i < p.dim ? x[r * p.dim + i] : 0.0f;
            if (p.signs) v = __fmul_rn(v, p.signs[i]);
            buf[i] = v;
        }
        __syncwarp();
        warp_fwht(buf, p.padded, lane);
        for (int i = lane; i < p.out_dim; i += 32) {
            float v = __fmul_rn(buf[i], p.scale);
            if (p.post_signs) v = __fmul_rn(v, p.post_signs[i]);
            p.out[r * p.out_dim + i] = v;
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------------------------
// Rows padded to 64, 128 or 256 whose length is a multiple of eight (every head size in use): four lanes a row, eight rows a warp.
//
// Lane m of a row holds elements 8 j + 2 m, 8 j + 2 m + 1 for j = 0 ... E - 1 (E = padded / 8) as packed pairs: two of the norm's
// eight interleaved accumulators (each a running sum over j in one register half), butterfly stage 1 inside a pair, stages 2 and 4 as
// one shuffle per element, stages from 8 up between registers, and the two codes of every pair.  Arithmetic in the order of the
// plain kernels below, which stay for other lengths; the quotient is the FMA-refined reciprocal with their division as the
// exception (see tq_write.cu).  The code of a value comes from a table over bins that hold at most one boundary each (the search
// of the cache write, with bins scaled to the row's length).
// 65536 rows of 128, 4 bits: quantize 107 us with the plain kernel (a warp a row, butterflies in shared memory, a
// compare per boundary: 20 times the memory floor) -> 16 us here (dequantize 77 -> 14 us); the limits are instruction issue and the shuffles of stages 2 and 4.
// That many rows come here from fp32 only: many 16-bit ones go to codes a lane a row by tq_flat_quant.cu (10 - 12 us), codes to rows by tq_flat_rows.cu (11).
// ---------------------------------------------------------------------------------------------
constexpr int kRowsWarps = 8, kRowsThreads = kRowsWarps * 32;
constexpr int kFlatBinZero = 144, kFlatBins = 2 * kFlatBinZero + 1;      // |y| <= 1.5 in bins of sqrt(128 / padded) / 64: 136 at 256
constexpr int kFlatCols = 16;                                            // copies of a table: an 8-byte load serves half a warp at a time

struct FlatRowsParams {
    FlatParams f;
    float bin_scale, bin_magic;           // bin of y = low mantissa bits of fma(y, bin_scale, bin_magic)
    float2 bins[kFlatBins];               // quantize: {boundary inside the bin or +inf, boundaries in lower bins}
};

template <typename T>
__device__ __forceinline__ P2 load_pair(const T* p);
template <>
__device__ __forceinline__ P2 load_pair<float>(const float* p) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    return pk(v.x, v.y);
}
template <>
__device__ __forceinline__ P2 load_pair<__nv_bfloat16>(const __nv_bfloat16* p) {
    const uint32_t w = *reinterpret_cast<const uint32_t*>(p);
    return pk(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
template <>
__device__ __forceinline__ P2 load_pair<__half>(const __half* p) {
    const uint32_t w = *reinterpret_cast<const uint32_t*>(p);
    const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w));
    return pk(v.x, v.y);
}

// butterflies in stage order on the four lanes of a row
template <int E>
__device__ __forceinline__ void rows_fwht(P2 (&x)[E], int m) {
#pragma unroll
    for (int j = 0; j < E; j++) {
        float a, b;
        up(x[j], a, b);
        x[j] = pk(__fadd_rn(a, b), __fsub_rn(a, b));
    }
#pragma unroll
    for (int d = 1; d < 4; d <<= 1) {
        // upper partner: other - mine, lower partner: mine + other; one FMA with +-1 does both (the product is exact)
        const float sgn = (m & d) ? -1.0f : 1.0f;
        const P2 sgn2 = pk(sgn, sgn);
#pragma unroll
        for (int j = 0; j < E; j++) {
            float a, b;
            up(x[j], a, b);
            const float oa = __shfl_xor_sync(0xffffffffu, a, d), ob = __shfl_xor_sync(0xffffffffu, b, d);
            x[j] = fma2(x[j], sgn2, pk(oa, ob));
        }
    }
#pragma unroll
    for (int h = 1; h < E; h <<= 1) {
#pragma unroll
        for (int j = 0; j < E; j++) {
            if (!(j & h)) {
                const P2 a = x[j], b = x[j + h];
                x[j] = add2(a, b);
                x[j + h] = sub2(a, b);
            }
        }
    }
}

// packed bytes of a row: a pair of codes fills a byte at 4 and 3 bits, two pairs at 2, four at 1
__host__ __device__ constexpr int flat_row_bytes(int padded, int bits) { return bits >= 3 ? padded / 2 : padded * bits / 8; }

template <typename T, int E, int BITS>
__global__ void __launch_bounds__(kRowsThreads, E == 8 ? 4 : E == 16 ? 3 : 2) quantize_rows_kernel(const __grid_constant__ FlatRowsParams p) {
    constexpr int kPd = 8 * E, kNb = flat_row_bytes(kPd, BITS), kPitch = kNb + 4;      // rows of a pass in different banks
    constexpr float kLast = (float)((1 << BITS) - 1);
    __shared__ float2 bins_s[kFlatBins * kFlatCols];
    __shared__ __align__(8) float sign_s[kPd];
    __shared__ __align__(16) uint8_t out_s[kRowsWarps][8 * kPitch + 12];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m = lane & 3, rw = lane >> 2;
    const int dim = p.f.dim;
    grid_launch_dependents();
    for (int i = threadIdx.x; i < kFlatBins * kFlatCols; i += kRowsThreads) bins_s[i] = p.bins[i / kFlatCols];
    grid_dependency_wait();      // only the table is made ahead of it
    bool beyond = false;
    for (int i = threadIdx.x; i < kPd; i += kRowsThreads) {
        const float sg = i < dim ? p.f.signs[i] : 1.0f;
        sign_s[i] = sg;
        beyond |= !(fabsf(sg) <= 1.0f);
    }
    // A normalized row keeps |y| <= 1, well inside the table, as long as no sign exceeds one.  Any other vector is taken too (infinities and
    // NaN among them): its values are brought inside the table first, beyond every boundary all the same.
    const bool wild = __syncthreads_or(beyond);
    // (the bit pattern of 2^23 + k) * 128 = 2^31 + 128 k modulo 2^32: entry k of this lane's column
    const uint32_t table_lane = smem_u32(bins_s) + 8u * (lane & (kFlatCols - 1)) - 0x80000000u;
    const P2 bin_scale2 = pk(p.bin_scale, p.bin_scale), bin_magic2 = pk(p.bin_magic, p.bin_magic), scale2 = pk(p.f.scale, p.f.scale);
    uint8_t* const tile = out_s[warp];
    auto code_of = [&](float y, float kf) -> float {
        float bnd, below;
        asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(bnd), "=f"(below) : "r"(__float_as_uint(kf) * 128u + table_lane));
        return y > bnd ? __fadd_rn(below, 1.0f) : below;
    };

    for (int64_t row0 = ((int64_t)blockIdx.x * kRowsWarps + warp) * 8; row0 < p.f.n; row0 += (int64_t)gridDim.x * kRowsWarps * 8) {
        // a lane without a row works on the last one again and stores nothing: the shuffles take every lane
        const int64_t last = p.f.n - 1, row = row0 + rw < p.f.n ? row0 + rw : last;
        const T* src = reinterpret_cast<const T*>(p.f.x) + row * dim + 2 * m;
        P2 x[E], acc = pk(0.0f, 0.0f);
        float minsq = 1.0f;
#pragma unroll
        for (int j = 0; j < E; j++) x[j] = 8 * j < dim ? load_pair<T>(src + 8 * j) : pk(0.0f, 0.0f);
#pragma unroll
        for (int j = 0; j < E; j++) {
            const P2 sq = mul2(x[j], x[j]);
            float s0, s1;
            up(sq, s0, s1);
            if (8 * j < dim) {      // the padding adds nothing and does not count as a small square
                acc = add2(acc, sq);
                asm("min.f32 %0, %0, %1, %2;" : "+f"(minsq) : "f"(s0), "f"(s1));
            }
        }
        // combine the eight accumulators left to right: lane m holds 2 m and 2 m + 1
        float a0, a1;
        up(acc, a0, a1);
        float s = __shfl_sync(0xffffffffu, a0, 0, 4);
        s = __fadd_rn(s, __shfl_sync(0xffffffffu, a1, 0, 4));
#pragma unroll
        for (int k = 1; k < 4; k++) {
            s = __fadd_rn(s, __shfl_sync(0xffffffffu, a0, k, 4));
            s = __fadd_rn(s, __shfl_sync(0xffffffffu, a1, k, 4));
        }
        minsq = fminf(minsq, __shfl_xor_sync(0xffffffffu, minsq, 1));
        minsq = fminf(minsq, __shfl_xor_sync(0xffffffffu, minsq, 2));
        float norm = __fsqrt_rn(s);
        if (!(norm >= 1e-8f)) norm = (norm != norm) ? __uint_as_float(0x7fc00000u) : 1e-8f;
        const bool fast = minsq >= 1.1754944e-38f && norm >= 9.0949470e-13f && norm <= 1.0995116e12f &&
                          (__float_as_uint(norm) & 0x7fffffu) != 0x7fffffu;
        if (fast) {
            const float rcp = __frcp_rn(norm);
            const P2 rcp2 = pk(rcp, rcp), nneg2 = pk(-norm, -norm);
#pragma unroll
            for (int j = 0; j < E; j++) {
                const P2 q = mul2(x[j], rcp2);
                x[j] = fma2(fma2(q, nneg2, x[j]), rcp2, q);      // x - q norm is exact
            }
        } else {
#pragma unroll
            for (int j = 0; j < E; j++) {
                float a, b;
                up(x[j], a, b);
                x[j] = 8 * j < dim ? pk(__fdiv_rn(a, norm), __fdiv_rn(b, norm)) : pk(0.0f, 0.0f);
            }
        }
#pragma unroll
        for (int j = 0; j < E; j++) {
            const float2 sg = *reinterpret_cast<const float2*>(&sign_s[8 * j + 2 * m]);
            x[j] = mul2(x[j], pk(sg.x, sg.y));
        }
        rows_fwht<E>(x, m);
        if (wild) {
            const float most = 1.5f / p.f.scale;
            auto inside = [most](float v) { return v < most ? fmaxf(v, -most) : most; };      // NaN: the last code
#pragma unroll
            for (int j = 0; j < E; j++) {
                float a, b;
                up(x[j], a, b);
                x[j] = pk(inside(a), inside(b));
            }
        }
        // codes.  A NaN row is NaN in every element (each output takes every input): torch puts NaN in the last bucket.
        float y0, y1;
        up(mul2(x[0], scale2), y0, y1);
        const bool all_nan = y0 != y0;
        __syncwarp();      // the pass before has been read out of the tile
#pragma unroll
        for (int j = 0; j < E; j++) {
            float c0 = kLast, c1 = kLast;
            if (!all_nan) {
                const P2 y = mul2(x[j], scale2);
                float k0, k1;
                up(y, y0, y1);
                up(fma2(y, bin_scale2, bin_magic2), k0, k1);
                c0 = code_of(y0, k0);
                c1 = code_of(y1, k1);
            }
            // first value in the low bits (cache order: in the high bits); sums of small whole numbers are exact
            const float lo = p.f.cache_order ? c1 : c0, hi = p.f.cache_order ? c0 : c1;
            float pair = __fmaf_rn(hi, (float)(1 << BITS), lo);
            if constexpr (BITS == 2) {
                const float other = __shfl_xor_sync(0xffffffffu, pair, 1);
                pair = p.f.cache_order ? __fmaf_rn(pair, 16.0f, other) : __fmaf_rn(other, 16.0f, pair);      // even lanes hold the byte
            } else if constexpr (BITS == 1) {
                float other = __shfl_xor_sync(0xffffffffu, pair, 1);
                pair = p.f.cache_order ? __fmaf_rn(pair, 4.0f, other) : __fmaf_rn(other, 4.0f, pair);
                other = __shfl_xor_sync(0xffffffffu, pair, 2);
                pair = p.f.cache_order ? __fmaf_rn(pair, 16.0f, other) : __fmaf_rn(other, 16.0f, pair);      // lane 0 holds it
            }
            const uint8_t byte = (uint8_t)__float_as_uint(__fadd_rn(pair, 8388608.0f));
            if constexpr (BITS >= 3) tile[rw * kPitch + 4 * j + m] = byte;
            else if constexpr (BITS == 2) { if ((m & 1) == 0) tile[rw * kPitch + 2 * j + (m >> 1)] = byte; }
            else { if (m == 0) tile[rw * kPitch + j] = byte; }
        }
        __syncwarp();
        // rows of the pass are consecutive in memory: 4-byte words, whole warps at a time
        uint32_t* const dst = reinterpret_cast<uint32_t*>(p.f.packed + row0 * kNb);
        const int words = (int)((p.f.n - row0 < 8 ? p.f.n - row0 : 8) * (kNb / 4));
        for (int i = lane; i < words; i += 32) {
            const int r = i / (kNb / 4), c = i % (kNb / 4);
            dst[i] = *reinterpret_cast<const uint32_t*>(tile + r * kPitch + 4 * c);
        }
        if (m == 0 && row0 + rw < p.f.n) p.f.norms[row] = norm;
    }
}

// pair value -> {centroid of the first, of the second}
template <int E, int BITS>
__global__ void __launch_bounds__(kRowsThreads, E == 8 ? 5 : E == 16 ? 4 : 2) dequantize_rows_kernel(const __grid_constant__ FlatParams p) {
    constexpr int kPd = 8 * E, kNb = flat_row_bytes(kPd, BITS), kEntries = 1 << (2 * BITS);
    __shared__ float2 pair_s[kEntries * kFlatCols];
    __shared__ __align__(8) float sign_s[kPd];
    __shared__ float cent_s[16];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m = lane & 3, rw = lane >> 2;
    grid_launch_dependents();
    if (threadIdx.x < 16) cent_s[threadIdx.x] = p.table[threadIdx.x];
    __syncthreads();
    for (int i = threadIdx.x; i < kEntries * kFlatCols; i += kRowsThreads) {
        const int v = i / kFlatCols, lo = v & ((1 << BITS) - 1), hi = v >> BITS;
        pair_s[i] = p.cache_order ? make_float2(cent_s[hi], cent_s[lo]) : make_float2(cent_s[lo], cent_s[hi]);
    }
    grid_dependency_wait();
    for (int i = threadIdx.x; i < kPd; i += kRowsThreads) sign_s[i] = i < p.dim ? p.signs[i] : 0.0f;
    __syncthreads();
    const uint32_t pair_lane = smem_u32(pair_s) + 8u * (lane & (kFlatCols - 1));
    const P2 scale2 = pk(p.scale, p.scale);
    for (int64_t row0 = ((int64_t)blockIdx.x * kRowsWarps + warp) * 8; row0 < p.n; row0 += (int64_t)gridDim.x * kRowsWarps * 8) {
        const int64_t row = row0 + rw < p.n ? row0 + rw : p.n - 1;
        const uint32_t* src = reinterpret_cast<const uint32_t*>(p.packed + row * kNb);
        uint32_t w[kNb / 4];      // the four lanes of a row read the same words
#pragma unroll
        for (int i = 0; i < kNb / 4; i++) w[i] = src[i];
        const float norm = p.norms[row];
        P2 x[E];
#pragma unroll
        for (int j = 0; j < E; j++) {
            // this lane's pair of elements 8 j + 2 m, + 1: a byte, a nibble or two bits
            uint32_t v;
            if constexpr (BITS >= 3) v = (w[j] >> (8 * m)) & (uint32_t)(kEntries - 1);
            else if constexpr (BITS == 2) v = (w[j / 2] >> (16 * (j & 1) + 8 * (m >> 1) + 4 * ((m & 1) ^ (p.cache_order ? 1 : 0)))) & 15u;
            else v = (w[j / 4] >> (8 * (j & 3) + 2 * (p.cache_order ? 3 - m : m))) & 3u;
            float a, b;
            asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(a), "=f"(b) : "r"(v * (8u * kFlatCols) + pair_lane));
            x[j] = pk(a, b);
        }
        rows_fwht<E>(x, m);
        if (row0 + rw >= p.n) continue;
        const P2 norm2 = pk(norm, norm);
        float* dst = p.out + row * p.dim + 2 * m;
#pragma unroll
        for (int j = 0; j < E; j++) {
            if (8 * j >= p.dim) break;
            const float2 sg = *reinterpret_cast<const float2*>(&sign_s[8 * j + 2 * m]);
            float a, b;
            up(mul2(mul2(mul2(x[j], scale2), pk(sg.x, sg.y)), norm2), a, b);
            *reinterpret_cast<float2*>(dst + 8 * j) = make_float2(a, b);
        }
    }
}

bool dequantize_lanes(const uint8_t* packed, const float* norms, int64_t n, int dim, int padded, const float* signs, int bits, bool cache_order, float* out,
                      void* stream, int* rc);

bool quantize_lanes(const void* x, int x_dtype, int64_t n, int dim, int padded, const float* signs, int bits, bool cache_order, uint8_t* packed, float* norms,
                    void* stream, int* rc);

static int next_pow2(int n) {
    int p = 1;
    while (p < n) p <<= 1;
    return p;
}

static unsigned flat_grid(int64_t n) {
    const int64_t blocks = (n + kFlatWarps - 1) / kFlatWarps;
    return (unsigned)(blocks < 148 * 16 ? (blocks > 0 ? blocks : 1) : 148 * 16);
}

// Rows the four-lane kernels take: padded to 64, 128 or 256, whole groups of eight, pairs that can be loaded and stored at once.
static bool rows_kernel_takes(int dim, int padded, const void* a, int a_align, const void* b, int b_align) {
    return padded >= 64 && dim % 8 == 0 && (uintptr_t)a % a_align == 0 && (uintptr_t)b % b_align == 0;
}

// one wave of resident blocks, or as many as there are eight-row passes for eight warps
template <typename K, typename P>
static int launch_rows(K kernel, int64_t n, int blocks_per_sm, const P& p, cudaStream_t s) {
    const int64_t blocks = (n + 8 * kRowsWarps - 1) / (8 * kRowsWarps), most = (int64_t)148 * blocks_per_sm;
    TQ_CUDA(launch_serialized(kernel, dim3((unsigned)(blocks < most ? blocks : most)), dim3(kRowsThreads), 0, s, p));
    return TQ_OK;
}

template <typename T, int E>
static int launch_quantize_rows(const FlatRowsParams& p, cudaStream_t s) {
    constexpr int kPerSm = E == 8 ? 4 : E == 16 ? 3 : 2;
    switch (p.f.bits) {
        case 1: return launch_rows(quantize_rows_kernel<T, E, 1>, p.f.n, kPerSm, p, s);
        case 2: return launch_rows(quantize_rows_kernel<T, E, 2>, p.f.n, kPerSm, p, s);
        case 3: return launch_rows(quantize_rows_kernel<T, E, 3>, p.f.n, kPerSm, p, s);
        default: return launch_rows(quantize_rows_kernel<T, E, 4>, p.f.n, kPerSm, p, s);
    }
}
template <typename T>
static int launch_quantize_rows(const FlatRowsParams& p, cudaStream_t s) {
    switch (p.f.padded) {
        case 64: return launch_quantize_rows<T, 8>(p, s);
        case 128: return launch_quantize_rows<T, 16>(p, s);
        default: return launch_quantize_rows<T, 32>(p, s);
    }
}
template <int E>
static int launch_dequantize_rows(const FlatParams& p, cudaStream_t s) {
    constexpr int kPerSm = E == 8 ? 5 : E == 16 ? 4 : 2;
    switch (p.bits) {
        case 1: return launch_rows(dequantize_rows_kernel<E, 1>, p.n, kPerSm, p, s);
        case 2: return launch_rows(dequantize_rows_kernel<E, 2>, p.n, kPerSm, p, s);
        case 3: return launch_rows(dequantize_rows_kernel<E, 3>, p.n, kPerSm, p, s);
        default: return launch_rows(dequantize_rows_kernel<E, 4>, p.n, kPerSm, p, s);
    }
}

// The table of the code search for (padded, bits), binned by the kernel's own float operations; made once each.
struct FlatBinTable {
    float scale;
    float2 bins[kFlatBins];
    bool ok;
};
static const FlatBinTable& flat_bins(int padded, int bits) {
    struct All {
        FlatBinTable t[3][4];
        All() {
            for (int e = 0; e < 3; e++) {
                for (int b = 1; b <= 4; b++) {
                    FlatBinTable& t = this->t[e][b - 1];
                    const int pd = 64 << e, nb = (1 << b) - 1;
                    float cen[16], bnd[15];
                    host_codebook(pd, b, cen, bnd);
                    t.scale = (float)(64.0 * std::sqrt(pd / 128.0));
                    t.ok = true;
                    int bin_of[15];
                    for (int i = 0; i < nb; i++) {
                        volatile float kf = fmaf(bnd[i], t.scale, 8388608.0f + kFlatBinZero);
                        float k = kf;
                        uint32_t word;
                        memcpy(&word, &k, 4);
                        bin_of[i] = (int)(word - 0x4B000000u);
                        if (bin_of[i] < 0 || bin_of[i] >= kFlatBins || (i && bin_of[i] <= bin_of[i - 1])) t.ok = false;
                    }
                    for (int k = 0; k < kFlatBins; k++) {
                        int below = 0;
                        float inside = INFINITY;
                        for (int i = 0; i < nb; i++) {
                            below += bin_of[i] < k;
                            if (bin_of[i] == k) inside = bnd[i];
                        }
                        t.bins[k] = make_float2(inside, (float)below);
                    }
                }
            }
        }
    };
    static const All all;
    return all.t[padded == 64 ? 0 : padded == 128 ? 1 : 2][bits - 1];
}

}  // namespace tq

extern "C" int tq_quantize_flat(const void* x, int x_dtype, int64_t n, int dim, const float* signs,
                                int bits, int pack_order, uint8_t* packed, float* norms,
                                void* stream) {
    using namespace tq;
    if (n == 0) return TQ_OK;
    TQ_REQUIRE(x && signs && packed && norms, TQ_ERR_INVALID, "null pointer");
    TQ_REQUIRE(n > 0 && dim >= 1 && dim <= kMaxDim, TQ_ERR_INVALID, "dim must be 1..%d", kMaxDim);
    TQ_REQUIRE(bits >= 1 && bits <= 4, TQ_ERR_INVALID, "bits must be 1..4");
    FlatParams p{};
    p.x = x; p.signs = signs; p.packed = packed; p.norms = norms; p.n = n; p.dim = dim;
    p.padded = next_pow2(dim); p.bits = bits; p.cache_order = pack_order == TQ_PACK_CACHE;
    p.scale = (float)(1.0 / std::sqrt((double)p.padded));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int rc = TQ_OK;
    if (quantize_lanes(x, x_dtype, n, dim, p.padded, signs, bits, p.cache_order, packed, norms, stream, &rc)) return rc;
    if (rows_kernel_takes(dim, p.padded, x, x_dtype == TQ_F32 ? 8 : 4, packed, 4) && x_dtype >= TQ_F32 && x_dtype <= TQ_BF16) {
        const FlatBinTable& t = flat_bins(p.padded, bits);
        if (t.ok) {
            FlatRowsParams r;
            r.f = p;
            r.bin_scale = t.scale;
            r.bin_magic = 8388608.0f + kFlatBinZero;
            memcpy(r.bins, t.bins, sizeof(r.bins));
            return x_dtype == TQ_F32 ? launch_quantize_rows<float>(r, s) : x_dtype == TQ_F16 ? launch_quantize_rows<__half>(r, s)
                                                                                             : launch_quantize_rows<__nv_bfloat16>(r, s);
        }
    }
    float cen[16];
    host_codebook(p.padded, bits, cen, p.table);
    switch (x_dtype) {
        case TQ_F32: quantize_flat_kernel<float><<<flat_grid(n), kFlatWarps * 32, 0, s>>>(p); break;
        case TQ_F16: quantize_flat_kernel<__half><<<flat_grid(n), kFlatWarps * 32, 0, s>>>(p); break;
        case TQ_BF16: quantize_flat_kernel<__nv_bfloat16><<<flat_grid(n), kFlatWarps * 32, 0, s>>>(p); break;
        default: return fail(TQ_ERR_INVALID, "bad x_dtype %d", x_dtype);
    }
    TQ_CUDA(cudaGetLastError());
    return TQ_OK;
}

extern "C" int tq_dequantize_flat(const uint8_t* packed, const float* norms, int64_t n, int dim,
                                  const float* signs, int bits, int pack_order, float* out,
                                  void* stream) {
    using namespace tq;
    if (n == 0) return TQ_OK;
    TQ_REQUIRE(packed && norms && signs && out, TQ_ERR_INVALID, "null pointer");
    TQ_REQUIRE(n > 0 && dim >= 1 && dim <= kMaxDim, TQ_ERR_INVALID, "dim must be 1..%d", kMaxDim);
    TQ_REQUIRE(bits >= 1 && bits <= 4, TQ_ERR_INVALID, "bits must be 1..4");
    FlatParams p{};
    p.packed = const_cast<uint8_t*>(packed); p.norms = const_cast<float*>(norms); p.signs = signs;
    p.out = out; p.n = n; p.dim = dim; p.padded = next_pow2(dim); p.bits = bits;
    p.cache_order = pack_order == TQ_PACK_CACHE;
    p.scale = (float)(1.0 / std::sqrt((double)p.padded));
    float bnd[15];
    host_codebook(p.padded, bits, p.table, bnd);
    int rc = TQ_OK;
    if (dequantize_lanes(packed, norms, n, dim, p.padded, signs, bits, p.cache_order, out, stream, &rc)) return rc;
    if (rows_kernel_takes(dim, p.padded, packed, 4, out, 8)) {
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        switch (p.padded) {
            case 64: return launch_dequantize_rows<8>(p, s);
            case 128: return launch_dequantize_rows<16>(p, s);
            default: return launch_dequantize_rows<32>(p, s);
        }
    }
    dequantize_flat_kernel<<<flat_grid(n), kFlatWarps * 32, 0, static_cast<cudaStream_t>(stream)>>>(p);
    TQ_CUDA(cudaGetLastError());
    return TQ_OK;
}

extern "C" int tq_fwht(const float* x, int64_t n, int in_dim, int padded_dim, int out_dim,
                       const float* pre_signs, const float* post_signs, float* out, void* stream) {
    using namespace tq;
    if (n == 0) return TQ_OK;
    TQ_REQUIRE(x && out, TQ_ERR_INVALID, "null pointer");
    TQ_REQUIRE(padded_dim >= 1 && padded_dim <= kMaxDim && (padded_dim & (padded_dim - 1)) == 0,
               TQ_ERR_INVALID, "padded_dim must be a power of two <= %d, got %d", kMaxDim, padded_dim);
    TQ_REQUIRE(in_dim >= 1 && in_dim <= padded_dim && out_dim >= 1 && out_dim <= padded_dim,
               TQ_ERR_INVALID, "in_dim/out_dim must be within padded_dim");
    FlatParams p{};
    p.x = x; p.signs = pre_signs; p.post_signs = post_signs; p.out = out; p.n = n; p.dim = in_dim;
    p.padded = padded_dim; p.out_dim = out_dim;
    p.scale = (float)(1.0 / std::sqrt((double)padded_dim));
    fwht_kernel<<<flat_grid(n), kFlatWarps * 32, 0, static_cast<cudaStream_t>(stream)>>>(p);
    TQ_CUDA(cudaGetLastError());
    return TQ_OK;
}
