// Cache write of large 16-bit K / V at head sizes 96, and padded 64 and 256 (kernel and mapping: tq_rows.cuh).
//   32768 tokens x 8 heads of 64, bf16: 91 us with eight lanes a row (a shuffle per element for each of stages 1, 2, 4, a four-step search) -> 32.4;
//   16384 x 8 of 256: 167 -> 65.8 (floors 14 and 26).  Heads of 96: 2048 x 32 fp16 19.0 -> 13.7, 16384 x 8 bf16 33.0 -> 25.3 (two lanes
//   a row of 128 before; the tensor-core kernel of tq_write.cu, padded, 38.7).  Heads of 128 this way, in an instance that was not kept, took 61 us (32768 x 8);
//   the tensor-core kernel takes 55.8.
#include "tq_rows.cuh"

namespace tq {

// Writes that this kernel takes: more than 8192 16-bit rows of a multiple of 8 elements, padded to 64 or 256 (16384 of 96), rows and slots on 16 bytes, 32-bit token
// numbers, and maps that can be made.  Returns false, having done nothing, for others.  Up to 8192 rows the kernel with a warp per row (256) is the faster
// one (300 tokens x 8: 6.6 us and 6.7; 600: 13.0 and 6.2), or a single call takes longer here for the maps (64, 350 tokens x 8: 5.2 and 4.1 us in a row,
// 13.3 and 14.7 alone); at 96 the kernel with two lanes a row does as well up to 16384 (1000 x 8: 4.8 and 4.8).
bool write_rows(void* kv_cache, int64_t num_blocks, int block_size, int num_kv_heads, int slot_bytes, const void* key, const void* value, int in_dtype,
                int64_t num_tokens, int64_t k_token_stride, int64_t v_token_stride, const float* signs, const void* slot_mapping, int slot_dtype,
                int head_dim, int flags, void* stream, int* rc) {
    const int padded = head_dim <= 64 ? 64 : head_dim == 96 ? 128 : 256;
    if (2 * num_tokens * num_kv_heads <= (head_dim == 96 ? 16384 : 8192) || num_tokens >= 0x7fffff00 || in_dtype == TQ_F32 || head_dim <= 32 || (head_dim > 64 && head_dim <= 128 && head_dim != 96) ||
        head_dim > 256 || head_dim % 8 != 0 || slot_bytes % 16 != 0 ||
        k_token_stride % 8 != 0 || v_token_stride % 8 != 0 || (uintptr_t)kv_cache % 16 != 0 || (uintptr_t)key % 16 != 0 || (uintptr_t)value % 16 != 0)
        return false;
    static const RowBins tables[3] = {make_row_bins(64, 4), make_row_bins(128, 4), make_row_bins(256, 4)};
    const RowBins& t = tables[padded == 64 ? 0 : padded == 128 ? 1 : 2];
    if (!t.ok) return false;
    LaneRowsParams p{};
    const int rows = lane_rows_of(padded);
    p.box_heads = 1;
    p.box_shift = 0;
    while (p.box_heads < rows && num_kv_heads % (2 * p.box_heads) == 0) {
        p.box_heads *= 2;
        p.box_shift++;
    }
    p.head_boxes = num_kv_heads / p.box_heads;
    for (int i = 0; i < 2; i++) {
        const int64_t stride = i ? v_token_stride : k_token_stride;
        const cuuint64_t dims[3] = {(cuuint64_t)head_dim, (cuuint64_t)num_kv_heads, (cuuint64_t)num_tokens};
        const cuuint64_t strides[2] = {(cuuint64_t)head_dim * 2, (cuuint64_t)stride * 2};
        const cuuint32_t box[3] = {64u, (cuuint32_t)p.box_heads, (cuuint32_t)(rows / p.box_heads)};
        if (!encode_tensor_map(&p.map[i], in_dtype == TQ_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, i ? value : key, dims,
                               strides, box, CU_TENSOR_MAP_SWIZZLE_128B))
            return false;
    }
    p.dst = static_cast<uint8_t*>(kv_cache);
    p.slot_mapping = slot_mapping;
    p.signs = signs;
    p.num_tokens = num_tokens;
    p.slab_bytes = num_blocks * block_size * (int64_t)num_kv_heads * slot_bytes;
    p.total_slots = num_blocks * (int64_t)block_size;
    p.heads = num_kv_heads;
    p.head_dim = head_dim;
    p.slot_bytes = slot_bytes;
    p.pad_end = (flags & TQ_WRITE_ZERO_PAD) == 0 ? 0 : head_dim == 96 ? 80 : slot_bytes;
    p.slot_is_i64 = slot_dtype == TQ_I64;
    p.bin_scale = t.bin_scale;
    p.scale = t.scale;
    memcpy(p.bins, t.bins, sizeof(p.bins));
    memcpy(p.bounds, t.bounds, sizeof(p.bounds));
    int sms = 0;
    *rc = device_sm_count(&sms);
    if (*rc != TQ_OK) return true;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool bf = in_dtype == TQ_BF16;
    if (padded == 64) *rc = bf ? launch_lane_rows<__nv_bfloat16, 64, 0, false>(p, sms, s) : launch_lane_rows<__half, 64, 0, false>(p, sms, s);
    else if (padded == 128) *rc = bf ? launch_lane_rows<__nv_bfloat16, 128, 96, false>(p, sms, s) : launch_lane_rows<__half, 128, 96, false>(p, sms, s);
    else *rc = bf ? launch_lane_rows<__nv_bfloat16, 256, 0, false>(p, sms, s) : launch_lane_rows<__half, 256, 0, false>(p, sms, s);
    return true;
}

int write_rows_fault_count(int32_t* out) {
    TQ_CUDA(cudaMemcpyFromSymbol(out, g_rows_dropped, sizeof(int32_t)));
    return TQ_OK;
}

}  // namespace tq
