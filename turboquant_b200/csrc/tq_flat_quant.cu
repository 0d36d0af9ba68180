// Flat quantizer for many 16-bit rows (kernel and mapping: tq_rows.cuh).
#include "tq_rows.cuh"

namespace tq {

// Rows an SM above which this kernel is the faster one (us on 148 SMs, 4 bits, the four-lane kernel first).  128 wide: up to 64 an SM the blocks of 64 rows of that
// one are a wave (9472 rows 5.4 / 4.8, at 2 bits 4.7 / 5.8, bf16 4.5 / 5.8; 10000 6.8 / 4.8, 2 bits 6.9 / 5.8, bf16 6.7 / 6.2; 56832 13.4 / 8.4).  64 wide:
// 16384 rows 5.1 / 3.4, 49152 8.1 / 5.0.  256 wide: 4096 rows 7.1 / 6.0, 20000 12.2 / 9.1 (136 wide).  The time of one unit bounds fewer.
static int quantize_lanes_from(int padded) { return padded == 64 ? 110 : padded == 128 ? 64 : 27; }
// Calls that this kernel takes: many 16-bit rows of a multiple of 8 elements padded to 64, 128 or 256, input and codes on 16 bytes, and a map that can be made.
// Returns false, having done nothing, for others.
bool quantize_lanes(const void* x, int x_dtype, int64_t n, int dim, int padded, const float* signs, int bits, bool cache_order, uint8_t* packed, float* norms,
                    void* stream, int* rc) {
    if (padded < 64 || n >= 0x7fffff00 || (x_dtype != TQ_F16 && x_dtype != TQ_BF16) || dim % 8 != 0 || (uintptr_t)x % 16 != 0 ||
        (uintptr_t)packed % 16 != 0 || (uintptr_t)norms % 4 != 0)
        return false;
    int sms = 0;
    *rc = device_sm_count(&sms);
    if (*rc != TQ_OK) return true;
    if (n <= (int64_t)quantize_lanes_from(padded) * sms) return false;
    struct Tables {
        RowBins t[3][4];
        Tables() {
            for (int e = 0; e < 3; e++)
                for (int b = 0; b < 4; b++) t[e][b] = make_row_bins(64 << e, b + 1);
        }
    };
    static const Tables tables;
    const RowBins& t = tables.t[padded == 64 ? 0 : padded == 128 ? 1 : 2][bits - 1];
    if (!t.ok) return false;
    LaneRowsParams p{};
    const cuuint64_t dims[3] = {(cuuint64_t)dim, 1u, (cuuint64_t)n};
    const cuuint64_t strides[2] = {(cuuint64_t)dim * 2, (cuuint64_t)dim * 2};
    const cuuint32_t box[3] = {64u, 1u, (cuuint32_t)lane_rows_of(padded)};
    if (!encode_tensor_map(&p.map[0], x_dtype == TQ_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, x, dims, strides, box,
                           CU_TENSOR_MAP_SWIZZLE_128B))
        return false;
    p.dst = packed;
    p.norms = norms;
    p.signs = signs;
    p.num_tokens = n;
    p.heads = p.box_heads = p.head_boxes = 1;
    p.head_dim = dim;
    p.bits = bits;
    p.cache_order = cache_order;
    p.count = (1 << bits) - 1;
    p.bin_scale = t.bin_scale;
    p.scale = t.scale;
    memcpy(p.bins, t.bins, sizeof(p.bins));
    memcpy(p.bounds, t.bounds, sizeof(p.bounds));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool bf = x_dtype == TQ_BF16;
    if (padded == 64) *rc = bf ? launch_lane_rows<__nv_bfloat16, 64, 0, true>(p, sms, s) : launch_lane_rows<__half, 64, 0, true>(p, sms, s);
    else if (dim == 96) *rc = bf ? launch_lane_rows<__nv_bfloat16, 128, 96, true>(p, sms, s) : launch_lane_rows<__half, 128, 96, true>(p, sms, s);
    else if (padded == 128) *rc = bf ? launch_lane_rows<__nv_bfloat16, 128, 0, true>(p, sms, s) : launch_lane_rows<__half, 128, 0, true>(p, sms, s);
    else *rc = bf ? launch_lane_rows<__nv_bfloat16, 256, 0, true>(p, sms, s) : launch_lane_rows<__half, 256, 0, true>(p, sms, s);
    return true;
}

int flat_quant_fault_count(int32_t* out) {
    TQ_CUDA(cudaMemcpyFromSymbol(out, g_rows_dropped, sizeof(int32_t)));
    return TQ_OK;
}

}  // namespace tq
