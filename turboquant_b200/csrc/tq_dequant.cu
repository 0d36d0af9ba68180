// Bulk dequantization of paged cache contents into dense K / V tensors.
//
// Used when a chunk of new query tokens has to attend to KV that already sits quantized in the
// cache (continuation of a prefill): the cached tokens of every sequence are gathered through the
// block table, dequantized (centroid lookup, inverse rotation, times the stored fp16 norm) and
// written as varlen-packed [total_tokens][num_kv_heads][128] K and V, the layout a varlen
// attention kernel takes.  The reference's backend ignores the cache during prefill
// (turboquant/vllm_backend_fused.py:336-369); its per-row arithmetic for this is
// TurboQuantMSE.dequantize (turboquant/quantizer.py:93-106) with the fp16 norm of the cache slot,
// as in its dequant-attention check (tests/test_fused_integration.py:127-159).
//
// Arithmetic, in this order, each step rounded to fp32: y[d] = (float)(C[idx[d]] / sqrt(128));
// butterflies h = 1..64; times (float)(1/sqrt(128)); times signs[d]; times float(fp16 norm).
// With fp32 output the result equals the CPU restatement bit for bit; fp16/bf16 outputs are its
// correctly rounded values.
//
// Mapping: a lane owns a row (two lanes a row of 256), a warp 32 / lanes-per-row consecutive rows of a page (its K rows, then its V rows).
// The butterflies are then register-local and packed in pairs (f32x2): stage h = 1 comes out of the lookup table, h = 2 .. 64 are
// whole-register adds.  Rows reach and leave the registers through shared memory: each warp copies the slots of unit n + 2 there while it works
// on unit n, and stages its output so that a store instruction covers whole rows.
//   8 ragged sequences of 5000 .. 13000 tokens x 8 heads of 128 -> bf16 (336 MB): 100 us with two lanes a row (a shuffle per element for
//   h = 64, on the pipe of the lookups and stores; 4 warps a scheduler, work found row by row) -> 70.4 us = 73 % of the copy rate.  Heads of 64, 8 x 1000 .. 8000 tokens (28300): 40.1 -> 18.0 us,
//   of 256, 8 x 1000 .. 4000 (20100): 89.0 -> 47.4, of 96, 3 x 1000 .. 16000 (31400) x 32 heads: 191 -> 104 (eight and two lanes a row before).  What bounds
//   it now is that pipe (74 % busy: 128 wavefronts of lookups, 192 of output, 32 of signs in about 430 a unit) at three warps a scheduler.
//   Output by tensor copies of 16 rows x 128 bytes in place of the read-back: 123 us.
#include <cmath>

#include "tq_common.cuh"

namespace tq {

int device_sm_count(int* out);
int device_shared_window_fits(uint32_t below, bool* fits);

constexpr int kDqDim = 128;
constexpr int kDqChunks = 256;      // parts of the sequences in a block's table of pages (a power of two; no more than a block's threads)

struct DequantParams {
    const uint8_t* kv_cache;
    int64_t slab_bytes;
    int64_t num_blocks;           // page ids outside [0, num_blocks) are skipped and counted
    const int32_t* page_indices;
    const int32_t* page_indptr;   // null: dense block table [batch][max_pages]
    const int32_t* seq_lens;
    const int32_t* cu_seqlens;    // [batch + 1]: first output row of every sequence
    const float* signs;
    void* out[2];                 // K, V: [total_tokens][H][head_dim]
    int64_t out_token_stride;     // elements between tokens
    int max_pages, H, head_shift, block_size, slot_bytes, batch;  // head_shift: log2(H) or -1
    float cen[16];                // (float)(C[i] / sqrt(padded))
    float scale;                  // (float)(1 / sqrt(padded))
};

// Page halves skipped because the page id lay outside the cache or the sequence was longer than
// its page list, copies of slots that never landed, and launches that did nothing; read back by tq_fault_counts.
static __device__ int32_t g_dequant_skipped = 0;

// HD: elements of an output row; PD: of the rotated row (HD rounded up to a power of two).  SMALL: jobs of a few units a scheduler.  With
// rows of 128 over two lanes a unit takes half as long, and the blocks leave room for the next kernel's beside them.
template <int DT, int PD, int HD, bool SMALL>
struct DqShape {
    static constexpr int kEsz = DT == TQ_F32 ? 4 : 2;
    static constexpr int kLanes = PD == 256 || (SMALL && PD == 128) ? 2 : 1, kRows = 32 / kLanes;    // lanes of a row, rows of a unit
    static constexpr int kPairs = PD / kLanes / 2;                           // packed pairs of values a lane
    static constexpr int kWarps = SMALL ? 8 : PD == 64 ? 20 : 12, kThreads = 32 * kWarps;      // 128 values a lane: 168 registers, 64: 96
    static constexpr int kCodes = PD / 2, kRow = (kCodes + 2 * (PD / 64) + 15) & ~15;   // staged bytes of a slot: 48, 80, 144
    static constexpr int kStage = kRows * kRow;
    // Output leaves in passes of 32 to 128 dims of every row.  A lane holds kLaneDims of them.
    static constexpr int kPassDims = kLanes == 2 ? PD / 2 : PD == 64 ? 128 / kEsz : 256 / kEsz, kLaneDims = kPassDims / kLanes;
    static constexpr int kPasses = (HD + kPassDims - 1) / kPassDims;
    static constexpr int kPitch = kPassDims * kEsz, kOut = kRows * kPitch;
    // Shared memory: rings, barriers, signs, the work list's table; the lookup table, 16 columns of 8 bytes a code byte (served half a warp at a time: no two lanes meet in a
    // bank); the output staging.  Large jobs have the table at 64 KB with a 256-byte row a code byte, so that one byte permute makes an entry's address.
    static constexpr uint32_t kSignBytes = PD * 4 + 64;                     // blocks of a pass's dims 16 bytes apart: two lanes of a row meet no bank
    static constexpr uint32_t kListBytes = (kDqChunks + 1 + kDqChunks / 32) * 8;
    static constexpr uint32_t kBelow = 2 * kWarps * kStage + ((2 * kWarps * 8 + kSignBytes + kListBytes + 127) & ~127);
    static constexpr uint32_t kEntry = SMALL ? 128 : 256, kTable = 65536;
    static constexpr uint32_t kSmem = SMALL ? 128 + kBelow + 256 * kEntry + kWarps * kOut : 2 * kTable + kWarps * kOut - 1024;   // from offset 1024 (the system's part)
    static_assert(SMALL || (kBelow + 1024 + 128 <= kTable && kSmem <= 232448), "shared memory");
};

template <int DT, int PD, int HD, bool SMALL>
__global__ void __launch_bounds__(DqShape<DT, PD, HD, SMALL>::kThreads, SMALL && PD != 256 ? 2 : 1) dequant_paged_kernel(const __grid_constant__ DequantParams p) {
    using S = DqShape<DT, PD, HD, SMALL>;
    constexpr uint32_t kAll = 0xffffffffu;
    extern __shared__ __align__(128) uint8_t dq_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t smem0 = (smem_u32(dq_smem) + 127u) & ~127u;
    const uint32_t bars = smem0 + 2 * S::kWarps * S::kStage, sgn = bars + 2 * S::kWarps * 8;
    const uint32_t table = SMALL ? smem0 + S::kBelow : S::kTable, stagings = table + 256 * S::kEntry;
    if (!SMALL && (smem0 + S::kBelow > S::kTable || smem0 < 1024)) {      // the shared window starts elsewhere than the device said
        grid_dependency_wait();
        if (tid == 0 && blockIdx.x == 0) atomicAdd(&g_dequant_skipped, 1);
        return;
    }
    uint8_t* const ring = dq_smem + (smem0 - smem_u32(dq_smem)) + warp * 2 * S::kStage;
    uint64_t* const bar = reinterpret_cast<uint64_t*>(dq_smem + (bars - smem_u32(dq_smem))) + 2 * warp;
    grid_launch_dependents();
    if (lane == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_barrier_init();
    }
    // byte -> {high + low, high - low}: butterfly stage h = 1 of the two centroids
    for (int i = tid; i < 256 * 8; i += S::kThreads) {
        const int v = i >> 3;
        const float hi = p.cen[v >> 4], lo = p.cen[v & 15];
        asm volatile("st.shared.v4.f32 [%0], {%1,%2,%1,%2};" ::"r"(table + S::kEntry * v + 16u * (i & 7)), "f"(__fadd_rn(hi, lo)), "f"(__fsub_rn(hi, lo)) : "memory");
    }
    grid_dependency_wait();  // the cache, the page table and the lengths belong to earlier kernels
    for (int d = tid; d < PD; d += S::kThreads) {
        const float v = d < HD ? __fmul_rn(p.signs[d], p.scale) : 0.0f;  // exact: the sign is +-1, or the scale a power of two
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(sgn + 4u * d + (S::kLanes == 2 ? 16u * (d / (PD / 4)) : 0u)), "f"(v) : "memory");
    }
    // The work list: units of 32 or 16 rows (a page's K rows, then its V rows) that hold a row of a token, all of a sequence's pages but its last and what
    // is live of that.  A warp takes every workers-th unit; its lanes look 32 of them up at a time, each its own: in a table of the units ahead of every
    // 256th part of the sequences, made here by the block, then sequence by sequence.  (With every warp going through all sequences for each 32 units of
    // whole pages 1024 x 20 tokens x 8 heads of 128 took 78 us and 4096 x 100 1053, against 49 and 622 item by item of a dense table; now 27 and 376.)
    const int half_rows = p.block_size * p.H, units = (2 * half_rows + S::kRows - 1) / S::kRows;
    const int chunk = (p.batch + kDqChunks - 1) / kDqChunks;
    int64_t* const starts = reinterpret_cast<int64_t*>(dq_smem + (sgn + S::kSignBytes - smem_u32(dq_smem)));
    // The live units of a page's first n tokens: k_units from the page's first, v_units from v_first.
    auto live = [&](int n, int& k_units, int& v_first) {
        k_units = (n * p.H + S::kRows - 1) / S::kRows;
        v_first = half_rows / S::kRows;
        if (v_first < k_units) v_first = k_units;      // a unit of K and V rows counts once
        return (half_rows + n * p.H + S::kRows - 1) / S::kRows - v_first;
    };
    // Pages of sequence b but its last live one, and that one's tokens; the count of its units.
    auto units_of = [&](int b, int& whole_pages, int& rest) -> int64_t {
        const int len = b < p.batch ? p.seq_lens[b] : 0;
        whole_pages = rest = 0;
        if (len <= 0 || p.max_pages <= 0) return 0;
        whole_pages = (len - 1) / p.block_size;
        rest = len - whole_pages * p.block_size;
        if (whole_pages >= p.max_pages) {      // longer than its page list
            whole_pages = p.max_pages - 1;
            rest = p.block_size;
        }
        int k_units, v_first;
        const int v_units = live(rest, k_units, v_first);
        return (int64_t)whole_pages * units + k_units + v_units;
    };
    {
        int64_t* const totals = starts + kDqChunks + 1;      // of the 32 chunks of a warp
        int64_t sum = 0;
        if (tid < kDqChunks) {
            int whole_pages, rest;
            for (int j = 0; j < chunk; j++) sum += units_of(tid * chunk + j, whole_pages, rest);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t t = __shfl_up_sync(kAll, sum, o);
                if (lane >= o) sum += t;
            }
            if (lane == 31) totals[warp] = sum;
        }
        __syncthreads();
        if (tid < kDqChunks) {
            for (int i = 0; i < warp; i++) sum += totals[i];
            starts[tid + 1] = sum;
            if (tid == 0) starts[0] = 0;
        }
        __syncthreads();
    }
    const int workers = (int)gridDim.x * S::kWarps;
    int64_t first = (int64_t)warp * gridDim.x + blockIdx.x;      // lane 0's unit; neighbouring units go to different SMs
    uint64_t src;       // this lane's unit: where its slots begin (0: nothing to do, 1: the end of the work; else a multiple of 16) ...
    int unit, ntok;     // ... which of the page's units, tokens in the page ...
    int row0;           // ... and the output row (token) of the page's first token
    auto look_up = [&]() {
        const int64_t at = first + (int64_t)lane * workers;
        src = 1;
        unit = 0;
        if (at < starts[kDqChunks]) {
            int c = 0;      // the part of the sequences that unit `at` lies in: the last that starts at or ahead of it
#pragma unroll
            for (int step = kDqChunks / 2; step > 0; step >>= 1)
                if (starts[c + step] <= at) c += step;
            int64_t rem = at - starts[c];
            int b = c * chunk, whole_pages, rest;
            int64_t n = units_of(b, whole_pages, rest);
            for (int j = 1; j < chunk && rem >= n; j++) {
                rem -= n;
                n = units_of(++b, whole_pages, rest);
            }
            src = 0;
            if (rem < n) {
                const int64_t pg = rem / units < whole_pages ? rem / units : whole_pages;
                unit = (int)(rem - pg * units);
                ntok = p.block_size;
                if (pg == whole_pages) {
                    int k_units, v_first;
                    live(rest, k_units, v_first);
                    if (unit >= k_units) unit += v_first - k_units;
                    ntok = rest;
                }
                row0 = p.cu_seqlens[b] + (int)pg * p.block_size;
                const int64_t tbl = p.page_indptr ? (int64_t)p.page_indptr[b] : (int64_t)b * p.max_pages;
                const int64_t page = !p.page_indptr || tbl + pg < (int64_t)p.page_indptr[b + 1] ? (int64_t)p.page_indices[tbl + pg] : -1;
                if ((uint64_t)page < (uint64_t)p.num_blocks) src = reinterpret_cast<uint64_t>(p.kv_cache) + (uint64_t)page * half_rows * p.slot_bytes;
                // else never form an address from it: the rows stay unwritten (the last two units are looked up again)
                else if (unit == 0 && lane < 30) atomicAdd(&g_dequant_skipped, 1);
            }
        }
        __syncwarp();
    };
    // The slots of unit i into stage s: neighbouring rows are neighbours in the cache, so one copy for the K and one for the V rows.
    auto issue = [&](int i, int s) {
        const uint64_t k0 = __shfl_sync(kAll, src, i);
        if (k0 <= 1) return;
        const int r0 = S::kRows * __shfl_sync(kAll, unit, i);
        const int rows = 2 * half_rows - r0 < S::kRows ? 2 * half_rows - r0 : S::kRows;
        uint8_t* dst = ring + s * S::kStage;
        __syncwarp();
        fence_proxy_async();   // the stage has been read out by ordinary loads
        if (p.slot_bytes == S::kRow) {
            if (lane == 0) {
                const int nk = half_rows - r0 < 0 ? 0 : half_rows - r0 < rows ? half_rows - r0 : rows;
                const uint8_t* from = reinterpret_cast<const uint8_t*>(k0) + (int64_t)r0 * S::kRow;
                mbar_arrive_expect_tx(&bar[s], (uint32_t)(rows * S::kRow));
                if (nk > 0) bulk_g2s(dst, from, (uint32_t)(nk * S::kRow), &bar[s]);
                if (nk < rows) bulk_g2s(dst + nk * S::kRow, from + p.slab_bytes + (int64_t)(nk - half_rows) * S::kRow, (uint32_t)((rows - nk) * S::kRow), &bar[s]);
            }
        } else {      // slots with more behind them: row by row
            if (lane == 0) mbar_arrive_expect_tx(&bar[s], (uint32_t)(rows * S::kRow));
            __syncwarp();
            const int r = r0 + lane;
            if (lane < rows)
                bulk_g2s(dst + lane * S::kRow, reinterpret_cast<const uint8_t*>(k0) + (r < half_rows ? (int64_t)r * p.slot_bytes : p.slab_bytes + (int64_t)(r - half_rows) * p.slot_bytes),
                         S::kRow, &bar[s]);
        }
    };

    // Of a pass, 16-byte piece i of a row (a lane's part of it is lane_pieces) is staged with the low three bits of i changed by the part's number, or
    // the row's where a part is half of 128 bytes: the eight lanes served together meet no bank twice, writing and reading.
    const int m = lane & (S::kLanes - 1);
    constexpr int kPer = 16 / S::kEsz, lane_pieces = S::kLaneDims / kPer;      // dims of a piece
    const uint32_t staging = stagings + (uint32_t)warp * S::kOut;
    auto staged = [&](int row, int pc) {
        const int key = lane_pieces >= 8 ? row * S::kLanes + pc / lane_pieces : row;
        return staging + row * S::kPitch + (pc >> 3) * 128 + (((pc ^ key) & 7) << 4);
    };
    const uint32_t my_part = staged(lane / S::kLanes, m * lane_pieces);
    const uint32_t table_lane = table + 8u * (lane & 15);
    const bool dense = p.out_token_stride == (int64_t)p.H * HD;

    look_up();
    issue(0, 0);
    issue(1, 1);
    uint32_t phases = 0;
    for (int i = 0, s = 0;; i++, s ^= 1) {
        if (i == 30) {      // the next units: this one becomes the first
            first += 30 * (int64_t)workers;
            look_up();
            i = 0;
        }
        const uint64_t k0 = __shfl_sync(kAll, src, i);
        if (k0 == 1) break;
        if (k0 != 0) {
            if (!__all_sync(kAll, mbar_wait(&bar[s], (phases >> s) & 1))) {
                copy_lost(&g_dequant_skipped, lane, &bar[s], (phases >> s) & 1, __shfl_sync(kAll, src, i + 1) > 1, &bar[s ^ 1], (phases >> (s ^ 1)) & 1);
                return;
            }
            phases ^= 1u << s;
            const uint32_t slot = smem_u32(ring) + s * S::kStage + (uint32_t)(lane / S::kLanes) * S::kRow;
            P2 x[S::kPairs];   // x[i] = dims 2 i, 2 i + 1 = code byte i (two lanes: of the row's half m)
#pragma unroll
            for (int j = 0; j < S::kPairs / 16; j++) {
                uint32_t w[4];
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(slot + (PD / 4) * m + 16 * j));
                if (S::kLanes == 2 && j >= S::kPairs / 32) {      // see the last stage
#pragma unroll
                    for (int e = 0; e < 4; e++) w[e] ^= 0u - m;
                }
#pragma unroll
                for (int e = 0; e < 16; e++) {
                    uint32_t at;      // byte e & 3 of the word becomes byte 1 of the address: row of the table
                    if constexpr (!SMALL) asm("prmt.b32 %0, %1, %2, %3;" : "=r"(at) : "r"(w[e >> 2]), "r"(table_lane), "r"(0x7604u | (uint32_t)((e & 3) << 4)));
                    else at = __byte_perm(w[e >> 2], 0, 0x4440 | (e & 3)) * S::kEntry + table_lane;
                    asm("ld.shared.b64 %0, [%1];" : "=l"(x[16 * j + e].v) : "r"(at));
                }
            }
            uint32_t nh;
            asm volatile("{\n\t.reg .u16 t;\n\tld.shared.u16 t, [%1];\n\tcvt.u32.u16 %0, t;\n\t}" : "=r"(nh) : "r"(slot + S::kCodes));
            const float norm = __half2float(__ushort_as_half((unsigned short)nh));
#pragma unroll
            for (int h = 1; h < S::kPairs; h <<= 1)
#pragma unroll
                for (int e = 0; e < S::kPairs; e++)
                    if (!(e & h)) {
                        const P2 a = x[e], c = x[e + h];
                        x[e] = add2(a, c);
                        x[e + h] = sub2(a, c);
                    }
            if constexpr (S::kLanes == 2) {
                // The last stage is between the lanes: each keeps its first half of values and sends the other, half the shuffles of sending all.  For that
                // the upper lane has to hold its values with the halves exchanged, which it does when the inputs of the second half change sign (the transform
                // of (-1)^[e >= n / 2] x is that of x at e ^ (n / 2)); the codebook is symmetric, so the complement of a code is its
                // negative.  Bit for bit: sums that cancel are +0 either way, and no input is a zero.  Lower outputs are mine + other, upper ones mine - other
                // or, in the upper lane, other - mine (not its negative, which is -0 where the two are equal).
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
            const P2 n2 = pk(norm, norm);
            const int r0 = S::kRows * __shfl_sync(kAll, unit, i), left = __shfl_sync(kAll, ntok, i);
            const int64_t out0 = __shfl_sync(kAll, row0, i);
            const bool in_v = r0 >= half_rows;
            // All rows are K rows or all V rows, and neighbours in the output.
            const bool whole = dense && (in_v ? r0 - half_rows : r0) + S::kRows <= left * p.H;
#pragma unroll
            for (int pass = 0; pass < S::kPasses; pass++) {
                // pieces of a row that are kept
                const int d0 = pass * S::kPassDims, dims = HD - d0 < S::kPassDims ? HD - d0 : S::kPassDims, pieces = dims / kPer;
                const uint32_t sgn_part = sgn + (S::kLanes == 2 ? (2 * pass + m) * (PD + 16) : 0);
#pragma unroll
                for (int c = 0; c < lane_pieces; c++) {
                    if (S::kLanes == 1 && c >= pieces) break;
                    uint32_t w[4];
#pragma unroll
                    for (int q = 0; q < kPer / 4; q++) {
                        const int d = pass * S::kLaneDims + c * kPer + 4 * q;      // of the lane's values
                        const int sd = S::kLanes == 2 ? c * kPer + 4 * q : d;
                        float4 sg;
                        asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(sg.x), "=f"(sg.y), "=f"(sg.z), "=f"(sg.w) : "r"(sgn_part + 4u * sd));
                        // (w * scale) * sign == w * (scale * sign) exactly; then the norm
                        float a, b, f, g;
                        up(mul2(mul2(x[d / 2], pk(sg.x, sg.y)), n2), a, b);
                        up(mul2(mul2(x[d / 2 + 1], pk(sg.z, sg.w)), n2), f, g);
                        if constexpr (DT == TQ_F32) {
                            w[0] = __float_as_uint(a); w[1] = __float_as_uint(b); w[2] = __float_as_uint(f); w[3] = __float_as_uint(g);
                        } else if constexpr (DT == TQ_F16) {
                            const __half2 u = __floats2half2_rn(a, b), v = __floats2half2_rn(f, g);
                            w[2 * q] = *reinterpret_cast<const uint32_t*>(&u); w[2 * q + 1] = *reinterpret_cast<const uint32_t*>(&v);
                        } else {
                            const __nv_bfloat162 u = __floats2bfloat162_rn(a, b), v = __floats2bfloat162_rn(f, g);
                            w[2 * q] = *reinterpret_cast<const uint32_t*>(&u); w[2 * q + 1] = *reinterpret_cast<const uint32_t*>(&v);
                        }
                    }
                    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"((my_part ^ ((c & 7) << 4)) + (c >> 3) * 128), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
                }
                __syncwarp();
                // piece lane + 32 e of the pass in row order, from where it was staged
                int row = lane / pieces, pc = lane - row * pieces;
                if (whole) {
                    const uint32_t first_piece = staged(row, pc);
                    uint8_t* dst = static_cast<uint8_t*>(p.out[in_v]) + ((out0 * p.H + r0 - (in_v ? half_rows : 0)) * HD + d0) * S::kEsz +
                                   row * (HD * S::kEsz) + pc * 16;
#pragma unroll
                    for (int e = 0; e < pieces / S::kLanes; e++) {
                        // 32 is a multiple of the pieces, or (96-wide rows, 12 pieces) they wrap within it
                        const int q_row = 32 % pieces ? (lane + 32 * e) / pieces : row + e * (32 / pieces), q_pc = 32 % pieces ? (lane + 32 * e) % pieces : pc;
                        const uint32_t at = 32 % pieces ? staged(q_row, q_pc) : (first_piece ^ ((e * (32 / pieces) * (lane_pieces >= 8 ? S::kLanes : 1) & 7) << 4)) + e * (32 / pieces) * S::kPitch;
                        uint4 v;
                        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
                        *reinterpret_cast<uint4*>(dst + ((q_row - row) * (HD * S::kEsz) + (q_pc - pc) * 16)) = v;
                    }
                } else {
#pragma unroll 1
                    for (int e = 0; e < pieces / S::kLanes; e++) {
                        const int r = r0 + row, v_row = r >= half_rows, rr = v_row ? r - half_rows : r;
                        const int t = p.head_shift >= 0 ? rr >> p.head_shift : rr / p.H;
                        uint4 v;
                        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                                     : "r"(staged(row, pc)) : "memory");
                        if (r < 2 * half_rows && t < left)
                            *reinterpret_cast<uint4*>(static_cast<uint8_t*>(p.out[v_row]) + ((out0 + t) * p.out_token_stride + (rr - t * p.H) * HD + d0) * S::kEsz + pc * 16) = v;
                        row += 32 / pieces;
                        pc += 32 % pieces;
                        if (pc >= pieces) { pc -= pieces; row++; }
                    }
                }
                __syncwarp();
            }
        }
        issue(i + 2, s);
    }
}

template <int DT, int PD, int HD, bool SMALL>
static int launch_dequant(const DequantParams& p, int64_t grid, cudaStream_t stream) {
    using S = DqShape<DT, PD, HD, SMALL>;
    static bool configured[64] = {};  // per template instance and device
    int dev = 0;
    TQ_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        TQ_CUDA(cudaFuncSetAttribute(dequant_paged_kernel<DT, PD, HD, SMALL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    TQ_CUDA(launch_serialized(dequant_paged_kernel<DT, PD, HD, SMALL>, dim3((unsigned)grid), dim3(S::kThreads), S::kSmem, stream, p));
    return TQ_OK;
}
// Up to this many units of 32 rows an SM (two a warp of the large kernel) the small blocks are faster: 8 heads of 128, 4800 tokens (16 units an
// SM) 8.2 us against 8.9; 16 ragged rows x 600, 4 heads 5.3 / 6.1; at 2400 tokens both 5.8; heads of 256, 3600 tokens 12.8 / 13.2.
constexpr int kDqSmallUnits = 24;

template <int DT, int PD, int HD>
static int launch_dequant(const DequantParams& p, int sms, cudaStream_t stream) {
    // The lengths are on the device: the table's width bounds the units of 32 rows.
    const int64_t units = (int64_t)p.batch * p.max_pages * ((2 * (int64_t)p.block_size * p.H + 31) / 32);
    // A device whose shared window leaves no room under the large blocks' table has the small blocks do all.
    bool fits = false;
    const int rc = device_shared_window_fits(DqShape<DT, PD, HD, false>::kBelow, &fits);
    if (rc != TQ_OK) return rc;
    if (!fits || units <= (int64_t)kDqSmallUnits * sms) {
        const int64_t most = (int64_t)sms * (PD == 256 ? 1 : 2), count = units * DqShape<DT, PD, HD, true>::kLanes;
        return launch_dequant<DT, PD, HD, true>(p, count < most ? count : most, stream);
    }
    return launch_dequant<DT, PD, HD, false>(p, units < sms ? units : sms, stream);
}
template <int PD, int HD>
static int launch_dequant(const DequantParams& p, int out_dtype, int sms, cudaStream_t stream) {
    switch (out_dtype) {
        case TQ_F32: return launch_dequant<TQ_F32, PD, HD>(p, sms, stream);
        case TQ_F16: return launch_dequant<TQ_F16, PD, HD>(p, sms, stream);
        default: return launch_dequant<TQ_BF16, PD, HD>(p, sms, stream);
    }
}
void host_codebook(int dim, int bits, float* centroids, float* boundaries);

int generic_dequant(const void* kv_cache, int64_t num_blocks, int block_size, int num_kv_heads, int slot_bytes,
                    const int32_t* page_indices, const int32_t* page_indptr, int max_pages, const int32_t* seq_lens,
                    const int32_t* cu_seqlens, int batch, const float* signs, int head_dim, void* k_out, void* v_out,
                    int out_dtype, int64_t out_token_stride, void* stream);
int generic_fault_counts(int32_t* write_dropped, int32_t* dequant_skipped);
int flat_rows_fault_count(int32_t* out);

int dequant_fault_count(int32_t* out) {
    int32_t a = 0, b = 0, c = 0, d = 0;
    TQ_CUDA(cudaMemcpyFromSymbol(&a, g_dequant_skipped, sizeof(int32_t)));
    int rc = generic_fault_counts(&b, &c);
    if (rc != TQ_OK) return rc;
    rc = flat_rows_fault_count(&d);
    if (rc != TQ_OK) return rc;
    *out = a + c + d;
    return TQ_OK;
}

}  // namespace tq

extern "C" int tq_dequant_paged(const void* kv_cache, int64_t num_blocks, int block_size, int num_kv_heads,
                                int slot_bytes, const int32_t* page_indices, const int32_t* page_indptr,
                                int max_pages, const int32_t* seq_lens, const int32_t* cu_seqlens, int batch,
                                const float* signs, int head_dim, void* k_out, void* v_out, int out_dtype,
                                int64_t out_token_stride, void* stream) {
    using namespace tq;
    TQ_REQUIRE(batch >= 0 && num_blocks >= 0, TQ_ERR_INVALID, "negative size");
    if (batch == 0 || max_pages == 0) return TQ_OK;
    TQ_REQUIRE(kv_cache && page_indices && seq_lens && cu_seqlens && signs && k_out && v_out, TQ_ERR_INVALID, "null pointer");
    const bool wide = head_dim == kDqDim || head_dim == 96;      // the sizes that take nothing but aligned slots and rows
    const int esz = out_dtype == TQ_F32 ? 4 : 2;
    const bool aligned = slot_bytes % 16 == 0 && (uintptr_t)kv_cache % 16 == 0 && (uintptr_t)k_out % 16 == 0 && (uintptr_t)v_out % 16 == 0 &&
                         out_token_stride * esz % 16 == 0;
    const bool second = (head_dim == 64 || head_dim == 256) && aligned && block_size == 16 && slot_bytes >= (head_dim == 64 ? 48 : 144);
    if (!wide && !second) {  // other head sizes, slots that are no multiple of 16 bytes: the plain kernel
        TQ_REQUIRE(num_kv_heads >= 1 && out_dtype >= TQ_F32 && out_dtype <= TQ_BF16 &&
                       out_token_stride >= (int64_t)num_kv_heads * head_dim, TQ_ERR_INVALID, "bad geometry");
        return generic_dequant(kv_cache, num_blocks, block_size, num_kv_heads, slot_bytes, page_indices, page_indptr, max_pages,
                               seq_lens, cu_seqlens, batch, signs, head_dim, k_out, v_out, out_dtype, out_token_stride, stream);
    }
    TQ_REQUIRE(!wide || (slot_bytes >= 80 && slot_bytes % 16 == 0), TQ_ERR_INVALID, "slot_bytes must be a multiple of 16 and >= 80");
    TQ_REQUIRE(block_size >= 1 && num_kv_heads >= 1 && max_pages >= 1 && batch >= 1, TQ_ERR_INVALID, "bad geometry");
    TQ_REQUIRE(out_dtype >= TQ_F32 && out_dtype <= TQ_BF16, TQ_ERR_INVALID, "bad out_dtype");
    TQ_REQUIRE(out_token_stride >= (int64_t)num_kv_heads * head_dim && (!wide || out_token_stride % 8 == 0), TQ_ERR_INVALID,
               "out_token_stride must cover one token and keep rows 16-byte aligned");
    TQ_REQUIRE(((uintptr_t)kv_cache % 16) == 0 && ((uintptr_t)k_out % 16) == 0 && ((uintptr_t)v_out % 16) == 0,
               TQ_ERR_INVALID, "kv_cache, k_out and v_out must be 16-byte aligned");
    DequantParams p{};
    p.kv_cache = static_cast<const uint8_t*>(kv_cache);
    p.slab_bytes = num_blocks * block_size * (int64_t)num_kv_heads * slot_bytes;
    p.num_blocks = num_blocks;
    p.page_indices = page_indices;
    p.page_indptr = page_indptr;
    p.seq_lens = seq_lens;
    p.cu_seqlens = cu_seqlens;
    p.signs = signs;
    p.out[0] = k_out;
    p.out[1] = v_out;
    p.out_token_stride = out_token_stride;
    p.max_pages = max_pages;
    p.H = num_kv_heads;
    p.head_shift = -1;
    for (int sft = 0; sft < 16; sft++)
        if ((1 << sft) == num_kv_heads) p.head_shift = sft;
    p.block_size = block_size;
    p.slot_bytes = slot_bytes;
    p.batch = batch;
    float bnd[15];
    const int padded = wide ? kDqDim : head_dim;
    host_codebook(padded, 4, p.cen, bnd);
    p.scale = (float)(1.0 / std::sqrt((double)padded));
    int sms = 0;
    int rc = device_sm_count(&sms);
    if (rc != TQ_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (head_dim) {
        case 64: return launch_dequant<64, 64>(p, out_dtype, sms, s);
        case 96: return launch_dequant<128, 96>(p, out_dtype, sms, s);
        case 256: return launch_dequant<256, 256>(p, out_dtype, sms, s);
        default: return launch_dequant<128, 128>(p, out_dtype, sms, s);
    }
}
