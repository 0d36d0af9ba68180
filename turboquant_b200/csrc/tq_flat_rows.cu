// Flat dequantizer for many rows: a lane owns a row (two lanes one of 256), as in the bulk dequantization of tq_dequant.cu.
//
// The arithmetic of the plain kernel in tq_flat.cu, in its order, each step rounded to fp32 (turboquant/quantizer.py:93-106 in the reference): centroids,
// butterflies h = 1 .. PD / 2, times 1 / sqrt(PD), times the sign, times the norm.  Compiled with -fmad=false.  The first butterfly stages come out of the
// lookup table (one per code byte: h = 1 of its two values at 3 and 4 bits, h = 1 and 2 of its four at 2 bits), the others are packed
// register adds, and the rows leave through shared memory so that a store instruction covers whole ones.  65536 rows of 128, 4 bits: 13.7 -> 10.8 us
// (floor 5.8); what is left is the table, two units a warp at most one after the other, and lookups (short scoreboard 2.3 stalls an issue, L1 51 %).
#include <cmath>

#include "tq_common.cuh"

namespace tq {

int device_sm_count(int* out);
int device_shared_window_fits(uint32_t below, bool* fits);

struct DequantRowsParams {
    const uint8_t* packed;
    const float* norms;
    const float* signs;
    float* out;
    int64_t n;
    int dim, cache_order;     // cache_order: the first value of a byte in its high bits
    float scale;
    float cen[16];
};

template <int PD, int BITS>
struct DequantRowsShape {
    static constexpr int kLanes = PD == 256 ? 2 : 1, kRows = 32 / kLanes, kPairs = PD / kLanes / 2;   // lanes of a row, rows of a unit, packed pairs a lane
    static constexpr int kWarps = PD == 64 ? 20 : 12, kThreads = 32 * kWarps;                          // 64 values a lane: 96 registers, 128: 168
    static constexpr int kRowBytes = BITS == 2 ? PD / 4 : PD / 2, kPieces = kRowBytes / 16;            // of codes; 16-byte pieces of it
    static constexpr int kLaneWords = kRowBytes / 4 / kLanes;
    static constexpr int kStage = kRows * kRowBytes;
    // Output passes: 32 or 64 dims of every row of one lane, a quarter or half (64 + 64) of a row of two.
    static constexpr int kPassDims = PD == 64 ? 32 : PD == 128 ? 64 : 128, kLaneDims = kPassDims / kLanes;
    static constexpr int kPitch = kPassDims * 4, kOut = kRows * kPitch;
    // The table at 64 KB with 256 bytes a code byte, so that one byte permute makes an entry's address: 16 columns of 8 bytes (served half a warp at a
    // time) or 8 of 16 (a quarter at a time), no two lanes meet in a bank.
    static constexpr uint32_t kTable = 65536, kSignBytes = PD * 4 + 64;
    static constexpr uint32_t kBelow = 2 * kWarps * kStage + 2 * kThreads * 4 + kSignBytes;
    static constexpr uint32_t kSmem = 2 * kTable + kWarps * kOut - 1024;      // from offset 1024 (the system's part)
    static_assert(kBelow + 1024 + 128 <= kTable && kSmem <= 232448, "shared memory");
};

// Launches that did nothing (their blocks' shared window started elsewhere than the device said); read back by tq_fault_counts.
static __device__ int32_t g_flat_rows_unfit = 0;
int flat_rows_fault_count(int32_t* out) {
    TQ_CUDA(cudaMemcpyFromSymbol(out, g_flat_rows_unfit, sizeof(int32_t)));
    return TQ_OK;
}

template <int PD, int BITS>
__global__ void __launch_bounds__(DequantRowsShape<PD, BITS>::kThreads, 1) dequantize_lanes_kernel(const __grid_constant__ DequantRowsParams p) {
    using S = DequantRowsShape<PD, BITS>;
    constexpr uint32_t kAll = 0xffffffffu;
    extern __shared__ __align__(128) uint8_t fr_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m = lane & (S::kLanes - 1), row = lane / S::kLanes;
    const uint32_t smem0 = (smem_u32(fr_smem) + 127u) & ~127u;
    if (smem0 + S::kBelow > S::kTable || smem0 < 1024) {
        grid_dependency_wait();
        if (tid == 0 && blockIdx.x == 0) atomicAdd(&g_flat_rows_unfit, 1);
        return;
    }
    const uint32_t ring = smem0 + (uint32_t)warp * 2 * S::kStage, norms = smem0 + 2 * S::kWarps * S::kStage + (uint32_t)warp * 256 + 4 * lane;
    const uint32_t sgn = smem0 + 2 * S::kWarps * S::kStage + 2 * S::kThreads * 4;
    grid_launch_dependents();
    for (int i = tid; i < 256 * 8; i += S::kThreads) {
        const int v = i >> 3;
        const uint32_t at = S::kTable + 256u * v + 16u * (i & 7);
        if constexpr (BITS == 2) {
            float c[4];
#pragma unroll
            for (int k = 0; k < 4; k++) c[k] = p.cen[(v >> (2 * (p.cache_order ? 3 - k : k))) & 3];
            const float a = __fadd_rn(c[0], c[1]), b = __fsub_rn(c[0], c[1]), d = __fadd_rn(c[2], c[3]), e = __fsub_rn(c[2], c[3]);
            asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(at), "f"(__fadd_rn(a, d)), "f"(__fadd_rn(b, e)), "f"(__fsub_rn(a, d)), "f"(__fsub_rn(b, e)) : "memory");
        } else {
            constexpr int kMask = (1 << BITS) - 1;
            const float lo = p.cen[v & kMask], hi = p.cen[(v >> BITS) & kMask], a = p.cache_order ? hi : lo, b = p.cache_order ? lo : hi;
            asm volatile("st.shared.v4.f32 [%0], {%1,%2,%1,%2};" ::"r"(at), "f"(__fadd_rn(a, b)), "f"(__fsub_rn(a, b)) : "memory");
        }
    }
    grid_dependency_wait();      // only the table is made ahead of it
    for (int d = tid; d < PD; d += S::kThreads) {
        const float v = d < p.dim ? p.signs[d] : 0.0f;
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(sgn + 4u * d + (S::kLanes == 2 ? 16u * (d / (PD / 4)) : 0u)), "f"(v) : "memory");
    }
    __syncthreads();

    const int64_t units = (p.n + S::kRows - 1) / S::kRows, step = (int64_t)gridDim.x * S::kWarps;
    // 16-byte piece pc of row r of a stage: the eight lanes served together (rows, or both halves of four) meet no bank twice
    auto code_piece = [](int r, int pc) {
        const int key = S::kPieces >= 8 ? r : S::kPieces == 4 ? r >> 1 : S::kPieces == 2 ? r >> 2 : 0;
        return (uint32_t)(r * S::kRowBytes + ((pc ^ key) & (S::kPieces < 8 ? S::kPieces - 1 : 7)) * 16);
    };
    auto fetch = [&](int64_t u, int s) {
        __syncwarp();      // the stage has been read out
        if (u < units) {
            const int64_t r0 = u * S::kRows;
            const int left = p.n - r0 < S::kRows ? (int)(p.n - r0) : S::kRows;
            const uint8_t* src = p.packed + r0 * S::kRowBytes;
#pragma unroll
            for (int i = 0; i < (S::kRows * S::kPieces + 31) / 32; i++) {
                const int q = lane + 32 * i, r = q / S::kPieces;
                if (r < left)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ring + s * S::kStage + code_piece(r, q % S::kPieces)), "l"(src + q * 16) : "memory");
            }
            if (row < left) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(norms + s * 128), "l"(p.norms + r0 + row) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    constexpr int lane_pieces = S::kLaneDims / 4, pass_pieces = S::kPassDims / 4;
    const uint32_t staging = 2 * S::kTable + (uint32_t)warp * S::kOut, my_part = staging + lane * (S::kPitch / S::kLanes) + ((lane & 7) << 4);
    const uint32_t table_lane = S::kTable + (BITS == 2 ? 16u * (lane & 7) : 8u * (lane & 15));
    const P2 scale2 = pk(p.scale, p.scale);
    int64_t u = (int64_t)warp * gridDim.x + blockIdx.x;      // neighbouring units go to different SMs
    fetch(u, 0);
    fetch(u + step, 1);
    for (int s = 0; u < units; u += step, s ^= 1) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");      // all but the next unit's
        __syncwarp();
        P2 x[S::kPairs];      // pairs of neighbouring dims of the lane's values
        float norm;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(norm) : "r"(norms + s * 128) : "memory");
#pragma unroll
        for (int j = 0; j < S::kLaneWords / 4; j++) {
            uint32_t w[4];
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                         : "r"(ring + s * S::kStage + code_piece(row, m * (S::kPieces / S::kLanes) + j)) : "memory");
#pragma unroll
            for (int e = 0; e < 16; e++) {
                uint32_t at;      // byte e & 3 of the word becomes byte 1 of the address: row of the table
                asm("prmt.b32 %0, %1, %2, %3;" : "=r"(at) : "r"(w[e >> 2]), "r"(table_lane), "r"(0x7604u | (uint32_t)((e & 3) << 4)));
                if constexpr (BITS == 2) asm("ld.shared.v2.b64 {%0,%1}, [%2];" : "=l"(x[2 * (16 * j + e)].v), "=l"(x[2 * (16 * j + e) + 1].v) : "r"(at));
                else asm("ld.shared.b64 %0, [%1];" : "=l"(x[16 * j + e].v) : "r"(at));
            }
        }
        if constexpr (S::kLanes == 2) {      // see the last stage
            const P2 flip = m ? pk(-1.0f, -1.0f) : pk(1.0f, 1.0f);
#pragma unroll
            for (int e = S::kPairs / 2; e < S::kPairs; e++) x[e] = mul2(x[e], flip);
        }
#pragma unroll
        for (int h = BITS == 2 ? 2 : 1; h < S::kPairs; h <<= 1)
#pragma unroll
            for (int e = 0; e < S::kPairs; e++)
                if (!(e & h)) {
                    const P2 a = x[e], c = x[e + h];
                    x[e] = add2(a, c);
                    x[e + h] = sub2(a, c);
                }
        if constexpr (S::kLanes == 2) {
            // The last stage is between the lanes: each keeps its first half of values and sends the other.  For that the second lane holds its values
            // with the halves exchanged, as it does when the inputs of the second half change sign; bit for bit: a sum with an unchanged first half that
            // cancels is +0 whatever the second's zero.  Upper outputs are mine - other or, in that lane, other - mine (not its negative, which is
            // -0 where the two are equal).
            constexpr int kHalf = S::kPairs / 2;
            const P2 mine_sign = m ? pk(-1.0f, -1.0f) : pk(1.0f, 1.0f), other_sign = m ? pk(1.0f, 1.0f) : pk(-1.0f, -1.0f);
#pragma unroll
            for (int e = 0; e < kHalf; e++) {
                float a, c;
                up(x[kHalf + e], a, c);
                const P2 mine = x[e], other = pk(__shfl_xor_sync(kAll, a, 1), __shfl_xor_sync(kAll, c, 1));
                x[e] = add2(mine, other);
                x[kHalf + e] = fma2(other, other_sign, mul2(mine, mine_sign));      // exact products: one rounding, that of the difference
            }
        }
        const P2 norm2 = pk(norm, norm);
        const int64_t r0 = u * S::kRows;
        const int left = p.n - r0 < S::kRows ? (int)(p.n - r0) : S::kRows;
#pragma unroll
        for (int pass = 0; pass < PD / S::kPassDims; pass++) {
            const int d0 = pass * S::kPassDims;
            if (d0 >= p.dim) break;
            const uint32_t sgn_part = sgn + (S::kLanes == 2 ? (2 * pass + m) * (PD + 16) : d0 * 4);
#pragma unroll
            for (int c = 0; c < lane_pieces; c++) {
                const int e = (pass * S::kLaneDims + 4 * c) / 2;
                float4 sg;
                asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(sg.x), "=f"(sg.y), "=f"(sg.z), "=f"(sg.w) : "r"(sgn_part + 16u * c));
                const P2 y0 = mul2(mul2(mul2(x[e], scale2), pk(sg.x, sg.y)), norm2), y1 = mul2(mul2(mul2(x[e + 1], scale2), pk(sg.z, sg.w)), norm2);
                asm volatile("st.shared.v2.b64 [%0], {%1,%2};" ::"r"((my_part ^ ((c & 7) << 4)) + (c >> 3) * 128), "l"(y0.v), "l"(y1.v) : "memory");
            }
            __syncwarp();
            // whole rows of the pass, from where their pieces were staged (piece i of a lane's part at (i ^ lane) & 7 of its 128 bytes)
            const int pieces = (p.dim - d0 < S::kPassDims ? p.dim - d0 : S::kPassDims) / 4;
            float* dst = p.out + r0 * p.dim + d0;
            if (pieces == pass_pieces) {
                constexpr int kAtOnce = 32 / pass_pieces > 0 ? 32 / pass_pieces : 1;      // rows of an instruction
                const int rr = lane / pass_pieces, pc = lane % pass_pieces;
                const uint32_t first = staging + rr * S::kPitch + (pc >> 3) * 128 + (((pc ^ (rr * S::kLanes + pc / lane_pieces)) & 7) << 4);
#pragma unroll
                for (int i = 0; i < S::kRows / kAtOnce; i++) {
                    float4 v;
                    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                                 : "r"((first ^ ((i * kAtOnce * S::kLanes & 7) << 4)) + i * kAtOnce * S::kPitch) : "memory");
                    if (rr + i * kAtOnce < left) *reinterpret_cast<float4*>(dst + (int64_t)(rr + i * kAtOnce) * p.dim + pc * 4) = v;
                }
            } else {
                for (int q = lane; q < left * pieces; q += 32) {
                    const int rr = q / pieces, pc = q - rr * pieces;
                    float4 v;
                    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                                 : "r"(staging + rr * S::kPitch + (pc >> 3) * 128 + (((pc ^ (rr * S::kLanes + pc / lane_pieces)) & 7) << 4)) : "memory");
                    *reinterpret_cast<float4*>(dst + (int64_t)rr * p.dim + pc * 4) = v;
                }
            }
            __syncwarp();
        }
        fetch(u + 2 * step, s);
    }
}

template <int PD, int BITS>
static int launch_dequantize_lanes(const DequantRowsParams& p, int sms, cudaStream_t stream) {
    using S = DequantRowsShape<PD, BITS>;
    static bool configured[64] = {};  // per template instance and device
    int dev = 0;
    TQ_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        TQ_CUDA(cudaFuncSetAttribute(dequantize_lanes_kernel<PD, BITS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const int64_t units = (p.n + S::kRows - 1) / S::kRows;
    TQ_CUDA(launch_serialized(dequantize_lanes_kernel<PD, BITS>, dim3((unsigned)(units < sms ? units : sms)), dim3(S::kThreads), S::kSmem, stream, p));
    return TQ_OK;
}
template <int PD>
static int launch_dequantize_lanes(const DequantRowsParams& p, int bits, int sms, cudaStream_t stream) {
    return bits == 4 ? launch_dequantize_lanes<PD, 4>(p, sms, stream) : bits == 3 ? launch_dequantize_lanes<PD, 3>(p, sms, stream) : launch_dequantize_lanes<PD, 2>(p, sms, stream);
}

// Rows an SM above which this kernel is the faster one (us on 148 SMs, the four-lane kernel first).  128 wide: up to 64 an SM the blocks of 64 rows of that one
// are a wave (4 bits, 9472 rows 3.1 / 4.1; 10000 5.9 / 4.1, 60000 13.7 / 10.7; 72 wide 9472 2.8 / 3.8, 10000 4.6 / 3.8).  At 2 bits its output
// is what counts there, so only whole rows (9472 3.3 / 4.8, 12500 3.9 / 4.9, 16000 5.7 / 5.0, 48000 9.9 / 7.2; 72 wide 60000 7.8 / 9.5, 96 wide
// 10.0 / 10.7).  256 wide: 2048 rows 5.1 / 3.5, 60000 25 / 16; 136 ... 192 wide at 2 bits 4736 rows 4.1 / 4.4, 7200 5.8 / 4.6.  64 wide: 49152
// 5.5 / 4.1, 131072 12.5 / 8.6.
static int lanes_from(int dim, int padded, int bits) {
    if (padded == 64) return 332;
    if (padded == 128) return bits > 2 ? 64 : dim == 128 ? 96 : -1;
    return bits > 2 || dim == 256 ? 13 : 32;
}
static uint32_t lanes_below(int padded, int bits) {
    return padded == 64 ? (bits == 2 ? DequantRowsShape<64, 2>::kBelow : DequantRowsShape<64, 4>::kBelow)
         : padded == 128 ? (bits == 2 ? DequantRowsShape<128, 2>::kBelow : DequantRowsShape<128, 4>::kBelow)
                         : (bits == 2 ? DequantRowsShape<256, 2>::kBelow : DequantRowsShape<256, 4>::kBelow);
}
// Calls that this kernel takes: many rows of a multiple of 8 elements padded to 64, 128 or 256, 2 to 4 bits, codes and output on 16 bytes, on a device
// whose shared window has room for the table's place.  Returns false, having done nothing, for others.
bool dequantize_lanes(const uint8_t* packed, const float* norms, int64_t n, int dim, int padded, const float* signs, int bits, bool cache_order, float* out,
                      void* stream, int* rc) {
    if (padded < 64 || dim % 8 != 0 || bits < 2 || (uintptr_t)packed % 16 != 0 || (uintptr_t)out % 16 != 0 || (uintptr_t)norms % 4 != 0)
        return false;
    int sms = 0;
    *rc = device_sm_count(&sms);
    if (*rc != TQ_OK) return true;
    const int from = lanes_from(dim, padded, bits);
    if (from < 0 || n <= (int64_t)from * sms) return false;
    bool fits = false;
    *rc = device_shared_window_fits(lanes_below(padded, bits), &fits);
    if (*rc != TQ_OK) return true;
    if (!fits) return false;
    DequantRowsParams p{};
    p.packed = packed;
    p.norms = norms;
    p.signs = signs;
    p.out = out;
    p.n = n;
    p.dim = dim;
    p.cache_order = cache_order;
    p.scale = (float)(1.0 / std::sqrt((double)padded));
    float bnd[15];
    host_codebook(padded, bits, p.cen, bnd);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    *rc = padded == 64 ? launch_dequantize_lanes<64>(p, bits, sms, s) : padded == 128 ? launch_dequantize_lanes<128>(p, bits, sms, s) : launch_dequantize_lanes<256>(p, bits, sms, s);
    return true;
}

}  // namespace tq
