// Paged decode attention split over (sequence, KV head, page range): every padded head size (64, 128, 256).
//
// The streaming kernel of tq_decode.cu gives a block all KV heads of a page range, which is what a long uniform context of
// 128-wide heads wants (whole page halves in a few bulk copies) and what a short one does not: 1024 cached tokens are
// eight blocks of four pages per warp, and the merge reads one partial per block, head and page lane.  Here a group of
// warps takes ONE head of a page range.  Work that fits the chip in one page per warp is spread that wide; anything larger is cut into
// equal ranges whatever the batch looks like, with the heads of a range side by side in one block.
//
//   * One block per SM = kGroups groups of kGroupWarps warps around one lookup table.  A group works alone (its own
//     named barrier); the table, the longest part of a block's prologue, is filled before the dependency wait.
//   * Plan on the device, by every warp for itself from seq_lens (no barrier): see SplitPlan.
//   * A warp takes whole pages of its head: one tiled tensor copy (16 rows of the head's slot from K and 16 from V; see kSlabs) into its
//     own ring of stages (eleven 16-byte asynchronous copies a lane filled the load/store queue: 40 / 8 heads, 32 ragged
//     sequences 34.4 -> 27.5 us a step, head size 64 34 -> 28, 256 37 -> 32), codes looked up straight
//     into mma.sync.m16n8k16 fragments (the scheme of tq_decode.cu: K bytes are A fragments of S = K^ Q^T, V nibbles of
//     two tokens zipped into bytes are A fragments of O^T += V^^T P).  Up to 32 query columns (128-wide heads) are up to four
//     MMA column tiles over one dequantization; see SplitShape for how registers are found for them.
//   * The group's warps combine in shared memory.  A head whose whole sequence the group covered is finished there
//     (inverse rotation, cast, store); only a head that was cut leaves partials for the merge kernel, which replans
//     while the decode kernel runs (it is launched when every decode block is past its own wait) and has two dependent
//     round trips to memory left after its wait.
#include <cmath>
#include <cstring>

#include <cuda.h>  // CUtensorMap and its enums only: the encoder is looked up at run time

#include "tq_decode_common.cuh"

namespace tq {

constexpr int kSplitMaxGroup = 8;     // query columns per KV head, and with the wide tiles of 128-wide heads
constexpr int kSplitMaxWide = 32;

// NT: tiles of eight query columns (MMA columns) a warp carries through one dequantization of its page.
template <int PD, int NT>
struct SplitShape {
    static constexpr int kCols = 8 * NT;
    static constexpr int kE = PD / 32;                       // elements per lane of a row
    static constexpr int kKBytes = PD / 8, kVBytes = PD / 16;  // code bytes per lane and token, K and V
    static constexpr int kRow = ((PD / 2 + 2 * (PD / 64)) + 15) & ~15;   // staged bytes of a slot: 48 / 80 / 144
    // A stage is a page's K box, then its V box: 16 dense rows each.  V loads (four rows, 32 bytes each) meet no bank twice at
    // any of the three pitches; the K loads (16 bytes a lane, two rows at a time) of 80-byte rows take two wavefronts a quarter for
    // one (8 a page of about 130), those of 144-byte rows one.
    static constexpr int kHalfBytes = 16 * kRow, kStageBytes = 2 * kHalfBytes;
    static_assert(kHalfBytes % 128 == 0, "boxes start on 128 bytes");
    // Wide tiles (128-wide heads): 32 accumulators a thread and tile.  Two tiles: 12 warps of 168 registers.  Three or four tiles would
    // leave 8 warps of 255, so two warps go as a pair: each works out the probabilities of its own page and accumulates half of the
    // dims of both (12 warps again).  Batch 8 x 32768 causal, 32 query / 8 KV heads: 8 queries a row 194 -> 181 us, 6: 171 -> 159 us,
    // 32 ragged sequences x 4096, 8 queries: 87 -> 71 us; as a pair two tiles are slower (124 -> 140 us).
    static constexpr bool kPair = NT >= 3;
    static constexpr int kStages = NT > 1 ? 4 : PD == 256 ? 2 : 3;
    // Slabs of a tensor copy's box: K and V of a page in one is up to 3 % faster (us, two boxes first: 10 x 2199 tokens, 32 / 8 heads of 96 18.1 / 17.6; 3 x 101 ...
    // 406, 40 heads 12.34 / 12.12; 18 x 1156 ... 37010, 2 causal queries 74.6 / 73.7).  For pairs of warps it is neither (8 x 32768, 8 queries 167.3 / 169.3; 18 x
    // 1156 ... 37010, 6 queries 117.8 / 115.6; 32 x 100 ... 4096, 8 queries 58.3 / 58.7): they keep two.
    static constexpr int kSlabs = kPair ? 1 : 2;
    static constexpr int kRingBytes = kStages * kStageBytes;
    // registers decide the warps per SM: 16 accumulator + 8 query registers at head 64 (80 a thread), 32 + 16 at 128
    // (128), 64 + 32 at 256 (168)
    static constexpr int kGroups = kPair ? 2 : 4, kGroupWarps = kPair ? 6 : NT == 2 ? 3 : PD == 64 ? 5 : PD == 128 ? 4 : 3;
    // query fragments kept in registers; the other tiles' are read from shared memory on every page (16 wavefronts a tile beside the
    // page's 64 lookups; in registers they spill: 8 queries 181 -> 185 us with one tile, 234 with two)
    static constexpr int kRegTiles = NT == 4 ? 0 : NT == 3 ? 2 : NT;
    static constexpr int kWarps = kGroups * kGroupWarps, kThreads = kWarps * 32;
    static constexpr int kRingsBelow = NT > 1 ? 5 : PD == 64 ? 13 : PD == 128 ? 7 : 6;   // rings below the table at 64 KB, the rest above it
    // What starting an item (a sequence's set of heads) costs a group, in pages of it: page ids, queries to rotate, a ring to fill, a combine.
    // Too little makes the blocks that hold many short sequences the last ones. 32 / 8 heads, 64 sequences of 64 ... 16384 tokens (log-
    // uniform): cost 6 / 10 / 14 / 20 / 26 / 32 gives 103 / 83 / 71 / 64 / 66 / 67 us; 16 columns 16 / 26 / 40 / 60 / 80: 140 / 110 /
    // 99 / 106 / 110; 24 columns 16 / 32 / 40 / 60: 214 / 148 / 130 / 136; 32 columns 32 / 40 / 60 / 80: 184 / 164 / 158 / 170; head size
    // 64, 6 / 10 / 16: 76 / 61 / 50 (but 16 x 8192 uniform 35 / 35 / 43); 256, 6 / 10 / 16: 127 / 102 / 104.
    static constexpr int kItemCost = PD != 128 ? 10 : NT == 1 ? 20 : NT < 4 ? 40 : 60;
    static constexpr bool kNormScale = NT > 1 || PD == 256;      // see kVNormMost
    // What the warps of a pair hand each other: the probabilities of a page as fragments, two pages' worth in turn.
    static constexpr int kHandBytes = kPair ? (NT + 1) / 2 * 512 : 0, kHandAt = (kWarps - kRingsBelow) * kRingBytes;
    static constexpr size_t kSmem = kLutAddr + kLutSpan + (size_t)kHandAt + 2 * kWarps * kHandBytes - 1024;   // from offset 1024 (the system's part): ample
    static_assert(kRingBytes >= kCols * PD * (kPair ? 2 : 4), "a warp's partial output goes through its ring");
    // in the unused upper halves of the table's rows: rotated queries, the warps' plans
    static constexpr uint32_t kPlanAt = kGroups * kCols * PD * 2;
    static_assert(kPlanAt + kWarps * 512 <= kLutSpan / 2, "the upper halves hold 32 KB");
    static_assert(NT == 1 || PD == 128, "wide tiles are for 128-wide heads");
};

struct SplitParams {
    alignas(64) CUtensorMap cache_map;   // uint8 [2][num_blocks * 16][H * slot], boxes of [kSlabs][16][kRow]
    const void* q;
    const uint8_t* kv_cache;
    const int32_t* page_indices;
    const int32_t* page_indptr;
    const int32_t* seq_lens;
    const float* signs;
    int32_t* header;        // workspace word 0: sticky status
    float* partial_lse;     // [2 x groups of the grid][group columns], base 2
    float* partial_o;       // [2 x groups of the grid][group columns][PD], normalized, rotated domain
    void* out;
    float* out_lse;
    int64_t num_blocks, kv_begin, kv_end;
    int batch, kv_heads, group, max_pages, q_dtype, out_dtype, emit_rotated;
    int nq, real_heads, real_group, head_dim, slot_bytes;
    int causal;             // query i of nq sees the first len - (nq - 1 - i) tokens
    int grid, head_set, head_sets;   // blocks of the decode launch; heads side by side in a block when the work is cut evenly, and kv_heads / head_set
    int item_cost;          // virtual pages that starting an item is worth (SplitShape::kItemCost)
    float inv_warps;        // 1 / warps of the grid
    int all_or_nothing;     // a sequence longer than its table empties the whole batch (128-wide heads), or only itself
    float k_scale, v_scale, scale;
    uint16_t centroid_h[16];
};

// ---------------------------------------------------------------------------------------------
// The plan: which (sequence, head, page range) a worker takes, and which workers a head's partials come from.  Both kernels
// compute it from seq_lens, every warp for itself: a lane holds one sequence of a batch of 32.
//   pieces: every head is cut into equal pieces of at most kGroupWarps x `tiles` pages, with the smallest number of tiles (pages per
//           warp) for which all pieces fit the groups of the grid; a worker is a group and takes one piece.  One start and one combine per
//           group, and a head that fits a piece is not cut at all; but the pieces of a ragged batch are of many sizes.
//   even:   the list of all pages (sequence, head set, page) is cut into equal ranges, one per worker and none of them empty, with
//           item_cost virtual pages in front of every item for what starting it costs (queries to rotate, a combine).  The head_set groups of a worker
//           take neighbouring heads of the same pages, so that the slots they read share their DRAM lines.
// Pieces are taken when their tiles exceed the even share by at most kSplitSlackTiles (about what a second start costs a group).
// ---------------------------------------------------------------------------------------------
constexpr int kSplitSlackTiles = 3;
// The running maximum before any score: finite, so that a column whose tokens are all masked so far has exp2(-inf - m) = 0.
constexpr float kNoMax = -3.402823466e38f;
// P times the V norm is rounded to fp16 as the MMA's operand; 1 / sqrt(128) is taken out in fp32 at the combine (ahead of the rounding it cost V rows of
// norm 1e-3 under 16 ... 32 causal columns 7 ... 8.7e-4 of error against 64 bits, now 4.9e-4 at any norm).  Norms are any fp16 value; a
// page whose largest exceeds kVNormMost (2^kRaiseThreshold times that is still finite in fp16) would overflow.
//   One column tile of padded size 64 / 128: that page's norms are brought to [256, 512) and the accumulators scaled down and up again around
//   it, so that other pages pay a maximum and a comparison (head size 64, 22 x 14327: 67 us as with a fixed scale, 75 with the one below).
//   Else: the warp keeps a power of two for the norms, 16 at first, and lowers it with the accumulators; a word in shared memory, for a register
//   more spills, and so does the code of the other form (8 x 32768 causal, 8 queries 162.6 us with a fixed scale, 163.2 so, 166 the other
//   way; one sequence of 1048576 567 / 577 / 587; head size 256, 1 x 1917 13.0 / 13.3 / 13.4).
constexpr float kVNormMost = 1000.0f, kVScaleStart = 16.0f;

// n / d for 0 <= n < 2^24, d > 0: a reciprocal, then the quotient put right.  (The plan is repeated by every warp, and the compiler's
// division is three times as long.)
__device__ __forceinline__ int split_div(int n, int d) {
    int q = (int)((float)n * __frcp_rn((float)d));
    const int r = n - q * d;
    q += r >= d ? 1 : r < 0 ? -1 : 0;
    return q;
}
// ceil(n / d), as above
__device__ __forceinline__ int split_div_up(int n, int d) { return split_div(n + d - 1, d); }

// the list position where worker c's range begins: c total / workers
__device__ __forceinline__ int split_cut(int c, int total, int workers) {
    if (total < (1 << 20) && workers < (1 << 12)) return (int)((uint32_t)c * (uint32_t)total / (uint32_t)workers);
    return (int)((int64_t)c * total / workers);
}

struct SplitPlan {
    int lane, base;          // this batch of 32 starts at sequence `base`
    int np, len;             // the lane's sequence: pages inside the window, tokens up to the window's end
    int vstart, vend;        // its span in the list, in units of pieces or of virtual pages (even)
    int run;                 // end of the span of the last sequence before this batch
    int ends;                // of many sequences: the list position where the lane's bin of them ends
    int total, workers, head_set;
    int piece;               // pages of a piece at most, 0: the even cut
    bool too_long;           // some sequence is longer than its page table
    bool void_batch;         // ... and that empties the batch
};

__device__ __forceinline__ int split_pages(const SplitParams& p, int b, int& len_out, bool& too_long) {
    int64_t len = p.seq_lens[b];
    if (p.kv_end >= 0 && p.kv_end < len) len = p.kv_end;
    const int first = (int)(p.kv_begin / kPageTokens);
    const int64_t last = (len + kPageTokens - 1) / kPageTokens;
    len_out = (int)len;
    int np = last > first ? (int)(last - first) : 0;
    const int have = p.page_indptr ? p.page_indptr[b + 1] - p.page_indptr[b] : p.max_pages;
    if (np > 0 && first + np > have) {
        too_long = true;
        np = 0;
    }
    return np;
}

__device__ __forceinline__ void split_load(const SplitParams& p, SplitPlan& s, int base, int run, bool keep) {
    bool dummy = false;
    if (!keep) {
        s.np = 0;
        if (base + s.lane < p.batch && !s.void_batch) s.np = split_pages(p, base + s.lane, s.len, dummy);
    }
    s.base = base;
    s.run = run;
    int v = 0;
    if (s.np > 0) v = s.piece ? p.kv_heads * split_div_up(s.np, s.piece) : p.head_sets * (s.np + p.item_cost);
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (s.lane >= o) incl += t;
    }
    s.vstart = run + incl - v;
    s.vend = run + incl;
}

// The cut of a work list of `pages` pages in `nonempty` sequences (and, in pieces, the piece and their number).
template <int NG>
__device__ __forceinline__ void split_cut_list(const SplitParams& p, SplitPlan& s, int pages, int nonempty, int pieces) {
    s.head_set = s.piece ? 1 : p.head_set;
    s.workers = p.grid * (s.head_set == 1 ? NG : s.head_set == 2 ? NG / 2 : NG / 4);
    s.total = s.piece ? pieces * p.kv_heads : p.head_sets * (pages + nonempty * p.item_cost);
    // Every worker of the even cut has a position of the list: one with an empty range would write no partial, and the merge counts
    // all workers between a head's first and last as its parts.  (A short list is cut too: many sequences of which few hold tokens.)
    if (!s.piece && s.workers > s.total) s.workers = s.total;
}
// Up to kSplitSelf sequences: every warp of both kernels plans for itself, and walks the list a batch of 32 at a time.
constexpr int kSplitSelf = 64;
template <int GW, int NG>
__device__ __forceinline__ void split_plan(const SplitParams& p, SplitPlan& s, int lane) {
    s.lane = lane;
    s.too_long = s.void_batch = false;
    s.len = 0;
    int pages = 0, nonempty = 0, np_first = 0, len_first = 0;
    for (int base = 0; base < p.batch; base += 32) {
        int np = 0, len = 0;
        if (base + lane < p.batch) np = split_pages(p, base + lane, len, s.too_long);
        if (base == 0) { np_first = np; len_first = len; }
        nonempty += __popc(__ballot_sync(0xffffffffu, np > 0));
        pages += __reduce_add_sync(0xffffffffu, np);
    }
    s.too_long = __any_sync(0xffffffffu, s.too_long);
    s.void_batch = s.too_long && p.all_or_nothing;
    if (s.void_batch) pages = nonempty = np_first = 0;
    s.np = np_first;
    s.len = len_first;
    // the smallest number of tiles whose pieces fit, from the even share on
    const int groups = p.grid * NG;
    const float even = (float)pages * (float)p.kv_heads * p.inv_warps;     // pages per warp (rounding it either way is fine)
    const int share = (int)even + (even > (float)(int)even ? 1 : 0);
    s.piece = 0;
    int pieces = 0;
    for (int t = share < 1 ? 1 : share; t <= share + kSplitSlackTiles; t++) {
        const int size = t * GW;
        pieces = __reduce_add_sync(0xffffffffu, split_div_up(np_first, size));
        for (int base = 32; base < p.batch && !s.void_batch; base += 32) {
            int len;
            bool dummy;
            const int np = base + lane < p.batch ? split_pages(p, base + lane, len, dummy) : 0;
            pieces += __reduce_add_sync(0xffffffffu, split_div_up(np, size));
        }
        if (pieces * p.kv_heads <= groups) {
            s.piece = size;
            break;
        }
    }
    split_cut_list<NG>(p, s, pages, nonempty, pieces);
    split_load(p, s, 0, 0, true);
}

// More sequences: the decode kernel's warps load the lengths of 256 at a time and remember where each of up to 32 bins of sequences ends in the list (a
// bin is one batch of 32, or as many as make 32 bins do), to find their place in one step.  Up to 256 may be cut in pieces (beyond that it measured slower: 512 of 2048
// tokens, ragged, 8 heads on one 29 -> 41 us).  The merge,
// whose blocks are more than fit the chip at once, reads this plan from the workspace (words 1 ... 4 and 8 ... 39) after its wait.
// The plan above costs a warp two trips over the lengths and half of a third one, in every block of the merge too: 8 heads on one, head size 64, 1000
// sequences of 500 tokens 75 -> 42 us with this one, 2000 of 64 157 -> 52; 64 / 8 heads, 256 ragged ones x 1024 98 -> 56.  At 64
// sequences and fewer the one above is faster by up to 8 %.
__device__ __forceinline__ int split_bin(const SplitParams& p) { return (p.batch + 1023) >> 10; }     // batches of 32 in a bin

template <int GW, int NG>
__device__ __forceinline__ void split_plan_many(const SplitParams& p, SplitPlan& s, int lane) {
    constexpr int kAhead = 8;
    s.lane = lane;
    s.too_long = s.void_batch = false;
    s.np = s.len = 0;
    const int span = split_bin(p);
    int np[kAhead], pages = 0, nonempty = 0, bin_pages = 0, bin_live = 0, bin = 0, in_bin = 0;
    for (int g0 = 0; 32 * g0 < p.batch; g0 += kAhead) {
#pragma unroll
        for (int u = 0; u < kAhead; u++) {
            const int b = 32 * (g0 + u) + lane;
            int len = 0;
            np[u] = b < p.batch ? split_pages(p, b, len, s.too_long) : 0;
        }
#pragma unroll
        for (int u = 0; u < kAhead; u++) {
            if (32 * (g0 + u) >= p.batch) break;
            const int sum = __reduce_add_sync(0xffffffffu, np[u]), live = __popc(__ballot_sync(0xffffffffu, np[u] > 0));
            if (lane == bin) { bin_pages += sum; bin_live += live; }
            if (++in_bin == span) { in_bin = 0; bin++; }
            pages += sum;
            nonempty += live;
        }
    }
    s.too_long = __any_sync(0xffffffffu, s.too_long);
    s.void_batch = s.too_long && p.all_or_nothing;
    if (s.void_batch) {
        pages = nonempty = bin_pages = bin_live = 0;
#pragma unroll
        for (int u = 0; u < kAhead; u++) np[u] = 0;
    }
    const int groups = p.grid * NG;
    const float even = (float)pages * (float)p.kv_heads * p.inv_warps;
    const int share = (int)even + (even > (float)(int)even ? 1 : 0);
    s.piece = 0;
    int pieces = 0, bin_pieces = 0;
    for (int t = share < 1 ? 1 : share; t <= share + kSplitSlackTiles && p.batch <= 32 * kAhead; t++) {      // np has them all
        const int size = t * GW;
        pieces = 0;
#pragma unroll
        for (int u = 0; u < kAhead; u++) {
            if (32 * u >= p.batch) break;
            const int sum = __reduce_add_sync(0xffffffffu, split_div_up(np[u], size));
            if (lane == u) bin_pieces = sum;
            pieces += sum;
        }
        if (pieces * p.kv_heads <= groups) {
            s.piece = size;
            break;
        }
    }
    split_cut_list<NG>(p, s, pages, nonempty, pieces);
    s.ends = s.piece ? p.kv_heads * bin_pieces : p.head_sets * (bin_pages + bin_live * p.item_cost);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, s.ends, o);
        if (lane >= o) s.ends += t;
    }
}
// to the first sequences of bin i
__device__ __forceinline__ void split_jump(const SplitParams& p, SplitPlan& s, int i) {
    const int before = __shfl_sync(0xffffffffu, s.ends, (i - 1) & 31);
    split_load(p, s, 32 * split_bin(p) * i, i > 0 ? before : 0, false);
}
__device__ __forceinline__ void split_keep_plan(const SplitParams& p, const SplitPlan& s) {
    if (s.lane == 0) {
        p.header[1] = s.total;
        p.header[2] = s.workers;
        p.header[3] = s.piece;
        p.header[4] = s.void_batch;
    }
    p.header[8 + s.lane] = s.ends;
}
__device__ __forceinline__ void split_kept_plan(const SplitParams& p, SplitPlan& s, int lane) {
    s.lane = lane;
    s.total = p.header[1];
    s.workers = p.header[2];
    s.piece = p.header[3];
    s.void_batch = p.header[4] != 0;
    s.ends = p.header[8 + lane];
    s.head_set = s.piece ? 1 : p.head_set;
    s.len = 0;
}

// One box of the cache into shared memory: bytes x ... of 16 token rows from row y of slab z (0: K, 1: V), or of both.  No multicast; x is a
// multiple of the slot, hence of 16.
__device__ __forceinline__ void split_box(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
__device__ __forceinline__ void split_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool split_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// A value the compiler cannot work out again: a lane's constants stay in registers through the page loop instead of being recomputed
// from the thread index in every iteration.
__device__ __forceinline__ uint32_t split_keep(uint32_t v) {
    asm volatile("" : "+r"(v));
    return v;
}
// BYTES (4, 8, 16 or 32) of a staged code row into words
template <int BYTES>
__device__ __forceinline__ void split_lds(uint32_t addr, uint32_t (&w)[BYTES / 4]) {
    if constexpr (BYTES == 4) {
        w[0] = lds32(addr);
    } else if constexpr (BYTES == 8) {
        const uint2 v = lds64(addr);
        w[0] = v.x; w[1] = v.y;
    } else {
#pragma unroll
        for (int i = 0; i < BYTES / 16; i++) {
            const uint4 v = lds128(addr + 16 * i);
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
    }
}

// Hadamard butterflies of a row over a warp: lane l holds elements E l ... E l + E - 1.
template <int E>
__device__ __forceinline__ void split_fwht(float (&v)[E], int lane) {
#pragma unroll
    for (int h = 1; h < E; h <<= 1) {
#pragma unroll
        for (int i = 0; i < E; i++) {
            if ((i & h) == 0) {
                const float a = v[i], b = v[i + h];
                v[i] = a + b;
                v[i + h] = a - b;
            }
        }
    }
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
#pragma unroll
        for (int i = 0; i < E; i++) {
            const float o = __shfl_xor_sync(0xffffffffu, v[i], m);
            v[i] = (lane & m) ? o - v[i] : v[i] + o;
        }
    }
}

// E consecutive elements of a 16- or 32-bit row as fp32; `at` is the element index of the first one, rows hold `dim` elements
template <int E>
__device__ __forceinline__ void split_load_row(const void* base, int dtype, int64_t row, int dim, int d0, float (&v)[E]) {
    const int64_t at = row * dim + d0;
    if (dtype != TQ_F32 && dim % E == 0 && (reinterpret_cast<uintptr_t>(base) & 15) == 0) {   // E 16-bit elements: 4, 8 or 16 bytes
        if (d0 >= dim) {
#pragma unroll
            for (int i = 0; i < E; i++) v[i] = 0.0f;
            return;
        }
        uint32_t w[E / 2];
        const uint16_t* src = reinterpret_cast<const uint16_t*>(base) + at;
        if constexpr (E == 2) w[0] = *reinterpret_cast<const uint32_t*>(src);
        else if constexpr (E == 4) { const uint2 t = *reinterpret_cast<const uint2*>(src); w[0] = t.x; w[1] = t.y; }
        else { const uint4 t = *reinterpret_cast<const uint4*>(src); w[0] = t.x; w[1] = t.y; w[2] = t.z; w[3] = t.w; }
#pragma unroll
        for (int i = 0; i < E / 2; i++) {
            if (dtype == TQ_BF16) {
                v[2 * i] = __uint_as_float(w[i] << 16);
                v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
            } else {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
                v[2 * i] = f.x;
                v[2 * i + 1] = f.y;
            }
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < E; i++) v[i] = d0 + i < dim ? load_q(base, dtype, at + i) : 0.0f;
}

// A finished row (normalized, rotated domain): back through the rotation and out, or out as it is.
template <int PD>
__device__ __forceinline__ void split_finish(const SplitParams& p, const float* signs, int b, int head, int col, float (&o)[PD / 32], float lse2, int lane) {
    constexpr int E = PD / 32;
    const int qi = col / p.real_group, hh = col - qi * p.real_group;
    const int64_t orow = ((int64_t)b * p.nq + qi) * p.real_heads + head * p.real_group + hh;
    const int d0 = lane * E;
    if (p.emit_rotated) {
        float* dst = reinterpret_cast<float*>(p.out) + orow * PD + d0;
#pragma unroll
        for (int i = 0; i < E; i++) dst[i] = o[i];
        if (p.out_lse && lane == 0) p.out_lse[orow] = lse2;
        return;
    }
    split_fwht<E>(o, lane);
    const int dim = p.head_dim;
#pragma unroll
    for (int i = 0; i < E; i++) o[i] *= p.scale * signs[d0 + i];
    const int64_t at = orow * dim + d0;
    if (p.out_dtype != TQ_F32 && dim % E == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0) {
        if (d0 < dim) {
            uint32_t w[E / 2];
#pragma unroll
            for (int i = 0; i < E / 2; i++) {
                if (p.out_dtype == TQ_BF16) {
                    const __nv_bfloat162 t = __floats2bfloat162_rn(o[2 * i], o[2 * i + 1]);
                    w[i] = *reinterpret_cast<const uint32_t*>(&t);
                } else {
                    w[i] = pack_half2(o[2 * i], o[2 * i + 1]);
                }
            }
            uint16_t* dst = reinterpret_cast<uint16_t*>(p.out) + at;
            if constexpr (E == 2) *reinterpret_cast<uint32_t*>(dst) = w[0];
            else if constexpr (E == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
            else *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    } else {
#pragma unroll
        for (int i = 0; i < E; i++) {
            if (d0 + i >= dim) continue;
            if (p.out_dtype == TQ_BF16) reinterpret_cast<__nv_bfloat16*>(p.out)[at + i] = __float2bfloat16_rn(o[i]);
            else if (p.out_dtype == TQ_F16) reinterpret_cast<__half*>(p.out)[at + i] = __float2half_rn(o[i]);
            else reinterpret_cast<float*>(p.out)[at + i] = o[i];
        }
    }
    if (p.out_lse && lane == 0) p.out_lse[orow] = lse2 * 0.6931471805599453f;
}

// MANY: more than kSplitSelf sequences (the plan's registers would spill in the page loop of a kernel that has both)
template <int PD, int NT, bool MANY>
__global__ void __launch_bounds__(SplitShape<PD, NT>::kThreads, 1) decode_split_kernel(const __grid_constant__ SplitParams p) {
    using F = SplitShape<PD, NT>;
    constexpr int E = F::kE, NG = F::kGroups, GW = F::kGroupWarps;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float m_s[NG][GW][F::kCols], l_s[NG][GW][F::kCols], v_s[NG][GW];
    __shared__ float sign_s[PD];
    __shared__ float max_s[F::kPair ? F::kWarps : 1][F::kCols + 1];  // a pair's maxima of a page that raises them (and its largest V norm), and whether it does
    __shared__ int raise_s[2][F::kPair ? F::kWarps : 1];
    __shared__ uint64_t full_s[F::kWarps][F::kStages + F::kNormScale];   // a stage's page has landed; and a word for the warp's scale of the V norms
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int gg = warp / GW, wg = warp % GW;      // group of the block, warp of the group
    const int g = lane >> 2, tg = lane & 3;
    const uint32_t smem_base = smem_u32(smem);
    const int G = p.group;
    if (smem_base + F::kRingsBelow * F::kRingBytes > kLutAddr) {   // the map does not fit
        grid_dependency_wait();
        if (tid == 0) {
            p.header[1] = 0;      // no plan for the merge
            atomicExch(&p.header[0], 3);
        }
        return;
    }
    uint8_t* const ring = smem + (warp < F::kRingsBelow ? (uint32_t)warp * F::kRingBytes
                                                       : kLutAddr + kLutSpan - smem_base + (uint32_t)(warp - F::kRingsBelow) * F::kRingBytes);
    const uint32_t ring_at = smem_u32(ring);
    uint8_t* const lut = smem + (kLutAddr - smem_base);
    // byte `off` of row r of the group's rotated queries (PD fp16), in the unused upper halves of the table's 256-byte rows, in the
    // order of B fragments: piece (tile j = r / 8, i) of 512 bytes holds, 16 bytes a lane (g = r % 8, tg), bytes 16 i ... of quarter tg
    auto q_ptr = [&](int r, uint32_t off) -> uint8_t* {
        const uint32_t tg = off / (PD / 2), i = off % (PD / 2) / 16;
        const uint32_t at = (uint32_t)gg * F::kCols * (PD * 2) + ((r >> 3) * (PD / 32) + i) * 512u + ((r & 7) * 4 + tg) * 16u + off % 16;
        return lut + ((at >> 7) << 8) + 128u + (at & 127u);
    };
    auto group_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + gg), "r"(GW * 32) : "memory"); };

    // lookup table: entry v, column c = {centroid(v & 15), centroid(v >> 4)}; a warp writes whole rows
    {
        // a warp's store covers four rows, 16 bytes a lane
        const uint32_t mine = p.centroid_h[lane & 15];
        for (int v = 4 * warp + (lane >> 3); v < 256; v += 4 * F::kWarps) {
            const uint32_t e = __shfl_sync(0xffffffffu, mine, v & 15) | (__shfl_sync(0xffffffffu, mine, v >> 4) << 16);
            *reinterpret_cast<uint4*>(lut + v * 256 + 16 * (lane & 7)) = make_uint4(e, e, e, e);
        }
    }
    // the signs are a constant of the context (as in the cache write): read ahead of the wait
    for (int i = tid; i < PD; i += F::kThreads) sign_s[i] = p.signs[i];
    if (tid == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(&p.cache_map) : "memory");
    if (lane < F::kStages) mbar_init(&full_s[warp][lane], 1);
    fence_barrier_init();
    // The small inputs into L2 while the kernel before this one drains: a whole KV stream may have passed since they were last
    // touched, and a prefetch hands no value over.
    if (blockIdx.x == 0 && tid * 32 < p.batch) prefetch_l2(p.seq_lens + tid * 32);
    if (!p.page_indptr)
        for (int64_t i = ((int64_t)blockIdx.x * F::kThreads + tid) * 32; i < (int64_t)p.batch * p.max_pages && i < (2 << 20); i += (int64_t)gridDim.x * F::kThreads * 32)
            prefetch_l2(p.page_indices + i);
    __syncthreads();
    grid_dependency_wait();      // seq_lens, the page table, Q, the cache and the workspace belong to earlier kernels
    grid_launch_dependents();    // the merge may now be scheduled: it reads seq_lens ahead of its own wait

    SplitPlan s;
    if constexpr (MANY) split_plan_many<GW, NG>(p, s, lane);
    else split_plan<GW, NG>(p, s, lane);
    if (s.too_long && blockIdx.x == 0 && tid == 0) atomicExch(&p.header[0], kStatusSeqTooLong);
    const int hs = s.head_set;
    const int sub = hs == 1 ? gg : hs == 2 ? gg >> 1 : gg >> 2, hsub = gg - sub * hs;
    const int worker = sub * p.grid + (int)blockIdx.x;   // neighbouring workers sit on different SMs
    int pos = 0, hi = 0;
    if (s.piece) {
        pos = worker;
        hi = worker < s.total ? worker + 1 : worker;
    } else if (worker < s.workers) {
        pos = split_cut(worker, s.total, s.workers);
        hi = split_cut(worker + 1, s.total, s.workers);
    }
    if constexpr (MANY) {
        if (blockIdx.x == 0 && warp == 0) split_keep_plan(p, s);
        split_jump(p, s, pos < hi ? __ffs(__ballot_sync(0xffffffffu, s.ends > pos)) - 1 : 0);      // a range lies inside the list
    }
    // the lane's sequence of the plan waits in shared memory while pages are worked on (registers are what the loop is short of)
    auto plan_at = [&]() -> uint8_t* {
        const uint32_t at = F::kPlanAt + (uint32_t)warp * 512u + (uint32_t)lane * 16u;
        return lut + ((at >> 7) << 8) + 128u + (at & 127u);
    };
    *reinterpret_cast<int4*>(plan_at()) = make_int4(s.np, s.len, s.vstart, s.vend);
    const int piece = s.piece;
    int base = MANY ? s.base : 0;
    const uint32_t lut_lane = split_keep(smem_u32(lut) + 4u * lane);
    const int fp = (int)(p.kv_begin / kPageTokens);
    // this lane's places in a stage: fragment rows g, g + 8 of K are tokens ta, tb
    const int ta = g, tb = g + 8;
    const uint32_t k_at = split_keep(ring_at + g * F::kRow + tg * F::kKBytes), kn_at = split_keep(ring_at + g * F::kRow + PD / 2);
    const uint32_t v_at = split_keep(ring_at + F::kHalfBytes + 2 * tg * F::kRow + g * F::kVBytes), vn_at = kn_at + F::kHalfBytes;
    const uint32_t full_at = split_keep(smem_u32(&full_s[warp][0]));
    const uint32_t frag_at = split_keep(smem_u32(lut) + ((uint32_t)gg * F::kCols * PD * 4) + 128u + ((uint32_t)(lane >> 3) << 8) + 16u * (lane & 7));
    constexpr int kVNext = F::kRow;      // from token 2 tg to token 2 tg + 1
    // The ring goes on from segment to segment: a stage's barrier completes once per page, in turn.
    uint32_t stage = 0, parity = 0;
    bool lost = false;                    // a wait ran out: nothing is copied or waited for from then on
    bool bad_page = false;

    while (pos < hi) {
        // ---- the next segment: a page range of one head -------------------------------------------------
        int4 e = *reinterpret_cast<const int4*>(plan_at());
        int run_end = __shfl_sync(0xffffffffu, e.w, 31);
        while (pos >= run_end && base + 32 < p.batch) {
            base += 32;
            s.piece = piece;
            s.head_set = hs;
            split_load(p, s, base, run_end, false);
            e = make_int4(s.np, s.len, s.vstart, s.vend);
            *reinterpret_cast<int4*>(plan_at()) = e;
            run_end = __shfl_sync(0xffffffffu, e.w, 31);
        }
        const uint32_t ahead = __ballot_sync(0xffffffffu, e.w > pos);
        if (ahead == 0) break;
        const int bl = __ffs(ahead) - 1, b = base + bl;
        const int np = __shfl_sync(0xffffffffu, e.x, bl), rel = pos - __shfl_sync(0xffffffffu, e.z, bl);
        const int len = __shfl_sync(0xffffffffu, e.y, bl);
        int hset, p0, p1;
        if (piece) {
            const int pieces = split_div_up(np, piece);
            hset = split_div(rel, pieces);
            const int j = rel - hset * pieces, size = split_div(np, pieces), more = np - size * pieces;
            p0 = j * size + (j < more ? j : more);           // the first `more` pieces take a page more
            p1 = p0 + size + (j < more ? 1 : 0);
            pos = hi;
        } else {
            const int item = np + p.item_cost;
            hset = split_div(rel, item);
            const int off = rel - hset * item;
            const int left = hi - pos, rest = item - off;      // up to the end of the range or of the item
            const int take = left < rest ? left : rest;
            p0 = off > p.item_cost ? off - p.item_cost : 0;
            p1 = off + take - p.item_cost;
            pos += take;
            if (p1 <= p0) continue;
        }
        const int head = hset * hs + hsub;

        // ---- page ids, the first stages' copies, the queries ------------------------------------------------
        const int n = p1 - p0 > wg ? (p1 - p0 - wg + GW - 1) / GW : 0;      // this warp's pages: p0 + wg + GW i
        const int32_t* ids = p.page_indices + (p.page_indptr ? (int64_t)p.page_indptr[b] : (int64_t)b * p.max_pages) + fp + p0 + wg;
        auto fetch_ids = [&](int i) -> int {
            int id = 0;
            if (i + lane < n) {
                id = ids[(i + lane) * GW];
                if ((uint64_t)(int64_t)id >= (uint64_t)p.num_blocks) {       // no address is formed from it: page 0 in its place
                    id = 0;
                    bad_page = true;
                }
            }
            return id;
        };
        int id_now = fetch_ids(0), id_next = n > 32 ? fetch_ids(32) : 0;
        // this warp's query rows wg, wg + GW, ... (a third one at head 256 below)
        constexpr int kQRows = NT == 1 ? 2 : (F::kCols + GW - 1) / GW;
        float qv[kQRows][E];
        const float* sign = sign_s + lane * E;
        auto q_row = [&](int r) -> int64_t {
            const int qi = r / p.real_group, hh = r - qi * p.real_group;
            return ((int64_t)b * p.nq + qi) * p.real_heads + head * p.real_group + hh;
        };
#pragma unroll
        for (int i = 0; i < kQRows; i++)
            if (wg + i * GW < G) {
                split_load_row<E>(p.q, p.q_dtype, q_row(wg + i * GW), p.head_dim, lane * E, qv[i]);
            } else {
#pragma unroll
                for (int e = 0; e < E; e++) qv[i][e] = 0.0f;
            }
        const int turns = F::kPair ? (p1 - p0 > (wg & ~1) ? (p1 - p0 - (wg & ~1) + GW - 1) / GW : 0) : n;      // the pair's
        const int x = head * p.slot_bytes;
        auto issue = [&](int i, uint32_t to) {       // page i of this warp into stage `to`
            const int id = __shfl_sync(0xffffffffu, id_now, i & 31);
            if (lane == 0 && i < turns && !lost) {
                const uint32_t bar = full_at + 8 * to, dst = ring_at + to * F::kStageBytes;
                split_expect(bar, i < n ? F::kStageBytes : 0);      // no page: the warps of a pair stay at the same stage
                if (i < n) {
#pragma unroll
                    for (int z = 0; z < 2; z += F::kSlabs) split_box(dst + z * F::kHalfBytes, &p.cache_map, x, id * kPageTokens, z, bar);
                }
            }
        };
#pragma unroll
        for (int i = 0; i < F::kStages - 1; i++) issue(i, stage + i < F::kStages ? stage + i : stage + i - F::kStages);
        auto put_q = [&](int r, float (&v)[E]) {
#pragma unroll
            for (int i = 0; i < E; i++) v[i] *= sign[i];
            split_fwht<E>(v, lane);
            // each (even, odd) pair swapped: a code byte dequantizes to {low half: odd dim, high half: even dim}
#pragma unroll
            for (int i = 0; i < E / 2; i++)
                *reinterpret_cast<uint32_t*>(q_ptr(r, (uint32_t)(lane * E + 2 * i) * 2u)) = pack_half2(v[2 * i + 1] * p.scale, v[2 * i] * p.scale);
        };
#pragma unroll
        for (int i = 0; i < kQRows; i++)
            if (wg + i * GW < F::kCols) put_q(wg + i * GW, qv[i]);
        for (int r = wg + kQRows * GW; r < G; r += GW) {
            split_load_row<E>(p.q, p.q_dtype, q_row(r), p.head_dim, lane * E, qv[0]);
            put_q(r, qv[0]);
        }
        auto v_norm_scale = [&]() -> float {
            if constexpr (F::kNormScale) return __uint_as_float(lds32(full_at + 8 * F::kStages));
            else return 1.0f;
        };
        auto set_v_norm_scale = [&](float v) {
            if (F::kNormScale && lane == 0) asm volatile("st.shared.u32 [%0], %1;" ::"r"(full_at + 8 * F::kStages), "r"(__float_as_uint(v)) : "memory");
        };
        set_v_norm_scale(kVScaleStart);
        group_sync();
        uint32_t qf[F::kRegTiles > 0 ? F::kRegTiles : 1][PD / 8];    // B fragments of Q^T: dims 2 x (code bytes tg PD/8 ...) of query column 8 j + g
#pragma unroll
        for (int j = 0; j < F::kRegTiles; j++)
#pragma unroll
            for (int i = 0; i < PD / 32; i++) {
                const uint4 t = 8 * j + g < G ? lds128(frag_at + 1024u * (j * (PD / 32) + i)) : make_uint4(0u, 0u, 0u, 0u);
                qf[j][4 * i] = t.x; qf[j][4 * i + 1] = t.y; qf[j][4 * i + 2] = t.z; qf[j][4 * i + 3] = t.w;
            }

        // ---- pages -----------------------------------------------------------------------------------------
        constexpr int kAccTiles = F::kPair ? PD / 32 : PD / 16;       // a warp of a pair keeps half of the dims
        float o_acc[NT][kAccTiles][4], m0[NT], m1[NT], l0[NT], l1[NT];
#pragma unroll
        for (int t = 0; t < NT; t++) {
#pragma unroll
            for (int i = 0; i < kAccTiles; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) o_acc[t][i][j] = 0.0f;
            m0[t] = m1[t] = kNoMax;
            l0[t] = l1[t] = 0.0f;
        }
        // S = K^ Q^T of the page in stage `st`: rows g, g + 8 are tokens ta, tb, columns 8 t + 2 tg, + 1 query heads; and the V norms
        auto scores = [&](uint32_t st, int left, float (&s_acc)[NT][4], float& vfa, float& vfb) {
            uint32_t ka[F::kKBytes / 4], kb[F::kKBytes / 4];
            split_lds<F::kKBytes>(k_at + st, ka);
            split_lds<F::kKBytes>(k_at + st + 8 * F::kRow, kb);
            float s_acc2[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int t = 0; t < NT; t++)
#pragma unroll
                for (int i = 0; i < 4; i++) s_acc[t][i] = 0.0f;
#pragma unroll
            for (int w = 0; w < F::kKBytes / 4; w++) {
                uint32_t ra[4], rb[4];
                dequant8(ka[w], lut_lane, ra);
                dequant8(kb[w], lut_lane, rb);
                if constexpr (NT == 1) {       // two chains
                    mma16816(s_acc[0], ra[0], rb[0], ra[1], rb[1], qf[0][4 * w], qf[0][4 * w + 1]);
                    mma16816(s_acc2, ra[2], rb[2], ra[3], rb[3], qf[0][4 * w + 2], qf[0][4 * w + 3]);
                } else {
                    uint32_t qs[NT][4];
#pragma unroll
                    for (int t = 0; t < NT; t++) {
                        if (t < F::kRegTiles) {
#pragma unroll
                            for (int i = 0; i < 4; i++) qs[t][i] = qf[t][4 * w + i];
                        } else {
                            const uint4 v = lds128(frag_at + 1024u * (t * (PD / 32) + w));
                            qs[t][0] = v.x; qs[t][1] = v.y; qs[t][2] = v.z; qs[t][3] = v.w;
                        }
                    }
#pragma unroll
                    for (int t = 0; t < NT; t++) mma16816(s_acc[t], ra[0], rb[0], ra[1], rb[1], qs[t][0], qs[t][1]);
#pragma unroll
                    for (int t = 0; t < NT; t++) mma16816(s_acc[t], ra[2], rb[2], ra[3], rb[3], qs[t][2], qs[t][3]);
                }
            }
            if constexpr (NT == 1) {
#pragma unroll
                for (int i = 0; i < 4; i++) s_acc[0][i] += s_acc2[i];
            }
            // Only the last page of a sequence holds tokens past the window: their norms are zeroed (whatever the unwritten
            // slots contain) and their scores biased to -inf.
            float kfa = lds_half(kn_at + st) * p.k_scale, kfb = lds_half(kn_at + st + 8 * F::kRow) * p.k_scale;
            const float v_norm = v_norm_scale();
            vfa = lds_half(vn_at + st) * v_norm, vfb = lds_half(vn_at + st + 8 * F::kRow) * v_norm;
            float bias_a = 0.0f, bias_b = 0.0f;
            if (left < kPageTokens) {
                if (ta >= left) { kfa = 0.0f; vfa = 0.0f; bias_a = -INFINITY; }
                if (tb >= left) { kfb = 0.0f; vfb = 0.0f; bias_b = -INFINITY; }
            }
#pragma unroll
            for (int t = 0; t < NT; t++) {
                float (&x)[4] = s_acc[t];
                x[0] = fmaf(x[0], kfa, bias_a);
                x[1] = fmaf(x[1], kfa, bias_a);
                x[2] = fmaf(x[2], kfb, bias_b);
                x[3] = fmaf(x[3], kfb, bias_b);
            }
            if (p.causal && left < kPageTokens + p.nq - 1) {       // a page that some query sees in part, or not at all
#pragma unroll
                for (int t = 0; t < NT; t++) {
                    const int s0 = left + 1 - p.nq + (8 * t + 2 * tg) / p.real_group, s1 = left + 1 - p.nq + (8 * t + 2 * tg + 1) / p.real_group;
                    if (ta >= s0) s_acc[t][0] = -INFINITY;
                    if (ta >= s1) s_acc[t][1] = -INFINITY;
                    if (tb >= s0) s_acc[t][2] = -INFINITY;
                    if (tb >= s1) s_acc[t][3] = -INFINITY;
                }
            }
        };
        // ---- online softmax (base 2) with a maximum that is raised only when a score exceeds it by kRaiseThreshold
        auto exceeds = [&](const float (&s_acc)[NT][4], float vfa, float vfb) {
            bool over = fmaxf(fabsf(vfa), fabsf(vfb)) > kVNormMost;
#pragma unroll
            for (int t = 0; t < NT; t++)
                over |= fmaxf(s_acc[t][0], s_acc[t][2]) > m0[t] + kRaiseThreshold || fmaxf(s_acc[t][1], s_acc[t][3]) > m1[t] + kRaiseThreshold;
            return __any_sync(0xffffffffu, over) != 0;
        };
        auto page_max = [&](const float (&x)[4], float& mx0, float& mx1) {
            mx0 = fmaxf(x[0], x[2]);
            mx1 = fmaxf(x[1], x[3]);
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
                mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
            }
        };
        // the largest V norm of the page if it is beyond the limit, else zero; and the power of two that brings it to [256, 512)
        auto norm_max = [&](float vfa, float vfb) {
            float v = fmaxf(fabsf(vfa), fabsf(vfb));
            if (!__any_sync(0xffffffffu, v > kVNormMost)) return 0.0f;
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
            return v;
        };
        auto norm_factor = [](float v) { return v > kVNormMost ? __uint_as_float((127 + 8 + 127 - (__float_as_uint(v) >> 23)) << 23) : 1.0f; };
        auto power_inverse = [](float f) { return __uint_as_float(0x7f000000u - __float_as_uint(f)); };      // of a power of two
        auto scale_sums = [&](float f) {
#pragma unroll
            for (int t = 0; t < NT; t++)
#pragma unroll
                for (int i = 0; i < kAccTiles; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) o_acc[t][i][j] *= f;
        };
        auto raise_to = [&](int t, float mx0, float mx1, float f) {
            const bool raise0 = mx0 > m0[t] + kRaiseThreshold, raise1 = mx1 > m1[t] + kRaiseThreshold;
            const float c0 = raise0 ? fast_exp2(m0[t] - mx0) : 1.0f, c1 = raise1 ? fast_exp2(m1[t] - mx1) : 1.0f;
            if (raise0) m0[t] = mx0;
            if (raise1) m1[t] = mx1;
            l0[t] *= c0;
            l1[t] *= c1;
            const float f0 = c0 * f, f1 = c1 * f;
#pragma unroll
            for (int i = 0; i < kAccTiles; i++) {
                o_acc[t][i][0] *= f0; o_acc[t][i][1] *= f1; o_acc[t][i][2] *= f0; o_acc[t][i][3] *= f1;
            }
        };
        // P = exp2(x - m) times the V norm as B fragments, and its column sums over this lane's two tokens
        auto probabilities = [&](const float (&s_acc)[NT][4], float vfa, float vfb, uint32_t (&pb0)[NT], uint32_t (&pb1)[NT], float (&a0)[NT], float (&a1)[NT]) {
#pragma unroll
            for (int t = 0; t < NT; t++) {
                const float e0 = fast_exp2(s_acc[t][0] - m0[t]), e1 = fast_exp2(s_acc[t][1] - m1[t]);
                const float e2 = fast_exp2(s_acc[t][2] - m0[t]), e3 = fast_exp2(s_acc[t][3] - m1[t]);
                a0[t] = e0 + e2;
                a1[t] = e1 + e3;
                pb0[t] = movmatrix_trans(pack_half2(e0 * vfa, e1 * vfa));
                pb1[t] = movmatrix_trans(pack_half2(e2 * vfb, e3 * vfb));
            }
        };
        // ---- O^T += V^^T P: four code bytes of four tokens, V^ rows g <- odd dim, g + 8 <- even dim of code byte 4 w + j
        auto accumulate = [&](int w, uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3, const uint32_t (&pb0)[NT], const uint32_t (&pb1)[NT]) {
            const uint32_t lo01 = (v0 & 0x0F0F0F0Fu) | ((v1 << 4) & 0xF0F0F0F0u);      // odd dims
            const uint32_t hi01 = ((v0 >> 4) & 0x0F0F0F0Fu) | (v1 & 0xF0F0F0F0u);      // even dims
            const uint32_t lo23 = (v2 & 0x0F0F0F0Fu) | ((v3 << 4) & 0xF0F0F0F0u);
            const uint32_t hi23 = ((v2 >> 4) & 0x0F0F0F0Fu) | (v3 & 0xF0F0F0F0u);
            uint32_t a_lo01[4], a_hi01[4], a_lo23[4], a_hi23[4];
            dequant8(lo01, lut_lane, a_lo01);
            dequant8(hi01, lut_lane, a_hi01);
            dequant8(lo23, lut_lane, a_lo23);
            dequant8(hi23, lut_lane, a_hi23);
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int t = 0; t < NT; t++) mma16816(o_acc[t][4 * w + j], a_lo01[j], a_hi01[j], a_lo23[j], a_hi23[j], pb0[t], pb1[t]);
        };
        uint32_t st = stage * F::kStageBytes;                                // offset of the stage in turn
        int left = len - (fp + p0 + wg) * kPageTokens;                       // tokens from this warp's page on
        auto copy_ahead = [&](int it) {
            const int ahead_i = it + F::kStages - 1;
            if ((ahead_i & 31) == 0) {          // the ids of the next 32 pages, and the load of those after them
                id_now = id_next;
                id_next = ahead_i + 32 < n ? fetch_ids(ahead_i + 32) : 0;
            }
            issue(ahead_i, stage == 0 ? F::kStages - 1 : stage - 1);
        };
        auto wait_page = [&] {
            if (!lost) {
                bool there = false;
                for (uint32_t i = 0; i < kSpinLimit && !there; i++) there = split_try_wait(full_at + 8 * stage, parity);
                if (!__all_sync(0xffffffffu, there)) {
                    lost = true;      // the output is void; what is still in flight gets its time to land
                    if (lane == 0) atomicExch(&p.header[0], 1);
                    for (uint32_t k = 1; k < F::kStages; k++) {
                        const bool wraps = stage + k >= F::kStages;
                        for (uint32_t i = 0; i < kSpinLimit / 64; i++)
                            if (split_try_wait(full_at + 8 * (wraps ? stage + k - F::kStages : stage + k), wraps ? parity ^ 1 : parity)) break;
                    }
                }
            }
            __syncwarp();
        };
        auto next_stage = [&] {
            if (++stage == F::kStages) {
                stage = 0;
                parity ^= 1;
            }
            st = stage * F::kStageBytes;
        };
        if constexpr (!F::kPair) {
            for (int it = 0; it < n; it++, left -= GW * kPageTokens) {
                copy_ahead(it);
                wait_page();
                // the V codes too, ahead of the vote below
                uint32_t v0[F::kVBytes / 4], v1[F::kVBytes / 4], v2[F::kVBytes / 4], v3[F::kVBytes / 4];
                split_lds<F::kVBytes>(v_at + st, v0);
                split_lds<F::kVBytes>(v_at + st + kVNext, v1);
                split_lds<F::kVBytes>(v_at + st + 8 * F::kRow, v2);
                split_lds<F::kVBytes>(v_at + st + 8 * F::kRow + kVNext, v3);
                float s_acc[NT][4], vfa, vfb, a0[NT], a1[NT];
                uint32_t pb0[NT], pb1[NT];
                scores(st, left, s_acc, vfa, vfb);
                if (exceeds(s_acc, vfa, vfb)) {
                    const float f = norm_factor(norm_max(vfa, vfb));
#pragma unroll
                    for (int t = 0; t < NT; t++) {
                        float mx0, mx1;
                        page_max(s_acc[t], mx0, mx1);
                        raise_to(t, mx0, mx1, F::kNormScale ? f : 1.0f);
                    }
                    if constexpr (!F::kNormScale) {
                        if (f < 1.0f) {
                            probabilities(s_acc, vfa * f, vfb * f, pb0, pb1, a0, a1);
                            scale_sums(f);
#pragma unroll
                            for (int w = 0; w < F::kVBytes / 4; w++) accumulate(w, v0[w], v1[w], v2[w], v3[w], pb0, pb1);
                            scale_sums(power_inverse(f));
                            l0[0] += a0[0];
                            l1[0] += a1[0];
                            __syncwarp();
                            next_stage();
                            continue;
                        }
                    } else if (f < 1.0f) {
                        vfa *= f;
                        vfb *= f;
                        set_v_norm_scale(v_norm_scale() * f);
                    }
                }
                probabilities(s_acc, vfa, vfb, pb0, pb1, a0, a1);
#pragma unroll
                for (int t = 0; t < NT; t++) {
                    l0[t] += a0[t];
                    l1[t] += a1[t];
                }
#pragma unroll
                for (int w = 0; w < F::kVBytes / 4; w++) accumulate(w, v0[w], v1[w], v2[w], v3[w], pb0, pb1);
                __syncwarp();      // every lane has read the stage before a later iteration copies into it
                next_stage();
            }
        } else {
            // A pair's turn is two pages, one a warp: scores and probabilities of its own, then half of the dims of both.  One
            // barrier a turn, at which the probabilities are in shared memory and both pages' copies have landed; it also tells
            // that the pair is through with the turn before, whose stage and whose hand-over buffer are written next.
            const uint32_t hand = smem_u32(smem) + (kLutAddr + kLutSpan - smem_base) + F::kHandAt + 16u * lane;
            const uint32_t mine = split_keep(hand + warp * 2 * F::kHandBytes), other = split_keep(hand + (warp ^ 1) * 2 * F::kHandBytes);
            const int ow = warp ^ 1;
            const uint32_t other_ring = smem_base + (ow < F::kRingsBelow ? (uint32_t)ow * F::kRingBytes
                                                                         : kLutAddr + kLutSpan - smem_base + (uint32_t)(ow - F::kRingsBelow) * F::kRingBytes);
            const uint32_t v_off = F::kHalfBytes + 2 * tg * F::kRow + 32 * (wg & 1) + 4 * g;
            const uint32_t v_own = split_keep(ring_at + v_off), v_other = split_keep(other_ring + v_off);
            auto pair_sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + NG + (warp >> 1)) : "memory"); };
            auto put = [&](uint32_t at, const uint32_t (&pb0)[NT], const uint32_t (&pb1)[NT]) {
#pragma unroll
                for (int t = 0; t < NT; t += 2)
                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at + 256u * t), "r"(pb0[t]), "r"(pb1[t]), "r"(t + 1 < NT ? pb0[(t + 1) % NT] : 0u),
                                 "r"(t + 1 < NT ? pb1[(t + 1) % NT] : 0u) : "memory");
            };
            for (int it = 0; it < turns; it++, left -= GW * kPageTokens) {
                wait_page();
                float s_acc[NT][4], vfa, vfb, a0[NT], a1[NT];
                uint32_t pb0[NT], pb1[NT];
                scores(st, it < n ? left : 0, s_acc, vfa, vfb);      // past its last page a warp has no tokens: P = 0
                const uint32_t turn = (uint32_t)(it & 1) * F::kHandBytes;
                const bool over = exceeds(s_acc, vfa, vfb);
                probabilities(s_acc, vfa, vfb, pb0, pb1, a0, a1);
                put(mine + turn, pb0, pb1);
                if (lane == 0) raise_s[it & 1][warp] = over;
                pair_sync();
                if (over || raise_s[it & 1][ow]) {      // rare: both warps raise to the maximum of both pages, and the probabilities again
                    float mx0[NT], mx1[NT];
#pragma unroll
                    for (int t = 0; t < NT; t++) {
                        page_max(s_acc[t], mx0[t], mx1[t]);
                        if (g == 0) {
                            max_s[warp][8 * t + 2 * tg] = mx0[t];
                            max_s[warp][8 * t + 2 * tg + 1] = mx1[t];
                        }
                    }
                    const float v_max = norm_max(vfa, vfb);
                    if (lane == 0) max_s[warp][F::kCols] = v_max;
                    pair_sync();
                    const float f = norm_factor(fmaxf(v_max, max_s[ow][F::kCols]));
#pragma unroll
                    for (int t = 0; t < NT; t++) raise_to(t, fmaxf(mx0[t], max_s[ow][8 * t + 2 * tg]), fmaxf(mx1[t], max_s[ow][8 * t + 2 * tg + 1]), f);
                    if (f < 1.0f) {
                        vfa *= f;
                        vfb *= f;
                        set_v_norm_scale(v_norm_scale() * f);
                    }
                    probabilities(s_acc, vfa, vfb, pb0, pb1, a0, a1);
                    put(mine + turn, pb0, pb1);
                    pair_sync();
                }
                copy_ahead(it);
#pragma unroll
                for (int t = 0; t < NT; t++) {
                    l0[t] += a0[t];
                    l1[t] += a1[t];
                }
                accumulate(0, lds32(v_own + st), lds32(v_own + st + kVNext), lds32(v_own + st + 8 * F::kRow), lds32(v_own + st + 8 * F::kRow + kVNext), pb0, pb1);
#pragma unroll
                for (int t = 0; t < NT; t += 2) {
                    const uint4 v = lds128(other + turn + 256u * t);
                    pb0[t] = v.x;
                    pb1[t] = v.y;
                    if (t + 1 < NT) {
                        pb0[(t + 1) % NT] = v.z;
                        pb1[(t + 1) % NT] = v.w;
                    }
                }
                accumulate(0, lds32(v_other + st), lds32(v_other + st + kVNext), lds32(v_other + st + 8 * F::kRow), lds32(v_other + st + 8 * F::kRow + kVNext), pb0, pb1);
                next_stage();
            }
        }
        if constexpr (F::kPair) group_sync();      // the other warp has read this one's last stage

        // ---- combine the group's warps ------------------------------------------------------------------------
#pragma unroll
        for (int t = 0; t < NT; t++) {
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                l0[t] += __shfl_xor_sync(0xffffffffu, l0[t], o);
                l1[t] += __shfl_xor_sync(0xffffffffu, l1[t], o);
            }
            if (g == 0) {
                m_s[gg][wg][8 * t + 2 * tg] = m0[t];      // columns past the group are zero queries: nobody reads them
                m_s[gg][wg][8 * t + 2 * tg + 1] = m1[t];
                l_s[gg][wg][8 * t + 2 * tg] = l0[t];
                l_s[gg][wg][8 * t + 2 * tg + 1] = l1[t];
            }
        }
        if (lane == 0) v_s[gg][wg] = p.v_scale * power_inverse(v_norm_scale());
        // The warp's accumulators as rows of PD floats (a pair: half rows, half of the dims each) in its own ring (the copies have landed and
        // been read).  The 16-byte pieces of a row are swapped by the column, which keeps the columns a quarter warp stores at a time in
        // different banks.
        __syncwarp();
        float* const mine = reinterpret_cast<float*>(ring);
        constexpr int kRowFloats = F::kPair ? PD / 2 : PD;
        auto swap_of = [](int c) -> int { return F::kPair ? (c & 1) | ((c & 2) << 1) : c; };     // of column pair c
        if (turns > 0) {
#pragma unroll
            for (int w = 0; w < kAccTiles / 2; w++) {      // bytes 2 w, 2 w + 1 of this lane: dims d ... d + 3
                const int piece = (g * kAccTiles + 2 * w) / 2;
#pragma unroll
                for (int t = 0; t < NT; t++) {
                    const int c = 8 * t + 2 * tg;
                    const float(&a)[4] = o_acc[t][2 * w], (&b4)[4] = o_acc[t][2 * w + 1];
                    if (c < G) *reinterpret_cast<float4*>(mine + c * kRowFloats + 4 * (piece ^ swap_of(tg))) = make_float4(a[2], a[0], b4[2], b4[0]);
                    if (c + 1 < G) *reinterpret_cast<float4*>(mine + (c + 1) * kRowFloats + 4 * (piece ^ swap_of(tg))) = make_float4(a[3], a[1], b4[3], b4[1]);
                }
            }
        }
        group_sync();
        const bool whole = p0 == 0 && p1 == np;
        const int slot = (worker * 2 + (p0 == 0 ? 1 : 0)) * hs + hsub;
        for (int r = wg; r < G; r += GW) {
            float mm = -INFINITY;
#pragma unroll
            for (int w = 0; w < GW; w++) mm = fmaxf(mm, m_s[gg][w][r]);
            float o[E], ll = 0.0f;
#pragma unroll
            for (int i = 0; i < E; i++) o[i] = 0.0f;
            constexpr int kStep = F::kPair ? 2 : 1;
#pragma unroll
            for (int w = 0; w < GW; w += kStep) {
                const float mw = m_s[gg][w][r];
                if (mw > kNoMax) {            // a warp without a page has stored nothing
                    const float cl = fast_exp2(mw - mm), c = cl * v_s[gg][w];
                    ll += cl * (F::kPair ? l_s[gg][w][r] + l_s[gg][w + kStep - 1][r] : l_s[gg][w][r]);
                    const int other = gg * GW + w + (F::kPair ? lane >> 4 : 0);      // a pair: dims 64 ... are the second warp's
                    const float* row = reinterpret_cast<const float*>(
                                           smem + (other < F::kRingsBelow ? (uint32_t)other * F::kRingBytes
                                                                         : kLutAddr + kLutSpan - smem_base + (uint32_t)(other - F::kRingsBelow) * F::kRingBytes)) + r * kRowFloats;
                    const int at = F::kPair ? lane & 15 : lane, swap = swap_of((r & 7) >> 1);
                    if constexpr (E == 2) {
                        const float2 t = *reinterpret_cast<const float2*>(row + 4 * ((at >> 1) ^ swap) + 2 * (at & 1));
                        o[0] += c * t.x; o[1] += c * t.y;
                    } else {
#pragma unroll
                        for (int i = 0; i < E / 4; i++) {
                            const float4 t = *reinterpret_cast<const float4*>(row + 4 * ((at * (E / 4) + i) ^ swap));
                            o[4 * i] += c * t.x; o[4 * i + 1] += c * t.y; o[4 * i + 2] += c * t.z; o[4 * i + 3] += c * t.w;
                        }
                    }
                }
            }
            const float inv = ll > 0.0f ? 1.0f / ll : 0.0f, lse2 = ll > 0.0f ? mm + log2f(ll) : -INFINITY;
#pragma unroll
            for (int i = 0; i < E; i++) o[i] *= inv;
            if (whole) {
                split_finish<PD>(p, sign_s, b, head, r, o, lse2, lane);
            } else {
                const int64_t at = (int64_t)slot * G + r;
                float* dst = p.partial_o + at * PD + lane * E;
                if constexpr (E == 2) {
                    *reinterpret_cast<float2*>(dst) = make_float2(o[0], o[1]);
                } else {
#pragma unroll
                    for (int i = 0; i < E / 4; i++)
                        *reinterpret_cast<float4*>(dst + 4 * i) = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
                }
                if (lane == 0) p.partial_lse[at] = lse2;
            }
        }
        if (pos < hi) {
            fence_proxy_async();       // the ring was written and read as rows
            group_sync();              // rings and query rows are free again
        }
    }
    if (bad_page) atomicExch(&p.header[0], kStatusBadPage);
}

// ---------------------------------------------------------------------------------------------
// Merge of the heads that were cut: RW warps per row (sequence, KV head, column) share its parts.  The plan is made ahead of
// the wait.  An empty sequence's rows become zeros here; a head that one group covered is finished already.
// ---------------------------------------------------------------------------------------------

template <int PD, int NT, int RW>
__global__ void __launch_bounds__(RW == 16 ? 512 : 128) merge_split_kernel(const __grid_constant__ SplitParams p) {
    using F = SplitShape<PD, NT>;
    constexpr int E = F::kE, GW = F::kGroupWarps, NG = F::kGroups, kRows = RW == 1 ? 4 : 1;      // rows of the block
    __shared__ float acc_s[RW][PD], m_s[RW], w_s[RW], sign_s[PD];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int part_warp = RW == 1 ? 0 : warp;
    const int G = p.group;
    grid_launch_dependents();
    const int row = blockIdx.x * kRows + (RW == 1 ? warp : 0);
    const int bh = row / G, r = row - bh * G, b = bh / p.kv_heads, head = bh - b * p.kv_heads;
    for (int i = threadIdx.x; i < PD; i += RW == 16 ? 512 : 128) sign_s[i] = p.signs[i];
    if (RW == 1) __syncthreads();
    SplitPlan s;
    const bool many = p.batch > kSplitSelf;
    if (many) {
        grid_dependency_wait();
        split_kept_plan(p, s, lane);
        split_jump(p, s, b < p.batch ? b / (32 * split_bin(p)) : 0);
    } else {
        split_plan<GW, NG>(p, s, lane);     // every decode block is past its wait: the lengths are final
    }
    while (s.base + 32 <= b && b < p.batch) split_load(p, s, s.base + 32, __shfl_sync(0xffffffffu, s.vend, 31), false);
    const int np = __shfl_sync(0xffffffffu, s.np, (b - s.base) & 31), vstart = __shfl_sync(0xffffffffu, s.vstart, (b - s.base) & 31);
    const int hs = s.head_set, hset = head / hs, hsub = head - hset * hs;
    int first = 0, count = 0;           // workers of this head's parts
    if (np > 0 && s.total > 0) {
        if (s.piece) {
            count = split_div_up(np, s.piece);
            first = vstart + hset * count;
        } else {
            const int64_t at = vstart + (int64_t)hset * (np + p.item_cost) + p.item_cost, end = at + np;   // its pages in the list
            first = (int)(((at + 1) * s.workers + s.total - 1) / s.total) - 1;
            count = (int)((end * s.workers + s.total - 1) / s.total) - first;
        }
    }
    if (!many) grid_dependency_wait();
    if (count == 1 || b >= p.batch) return;
    // part i: worker first + i; the first part starts its sequence (odd slot of the worker), the others continue it
    auto slot_row = [&](int i) -> int64_t { return ((int64_t)((first + i) * 2 + (i == 0 ? 1 : 0)) * hs + hsub) * G + r; };
    float m = -INFINITY, wsum = 0.0f, acc[E];
#pragma unroll
    for (int e = 0; e < E; e++) acc[e] = 0.0f;
    for (int i0 = part_warp; i0 < count; i0 += 8 * RW) {        // parts i0, i0 + RW, ...: eight payloads and their LSEs in flight together
        float o[8][E], lse[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int i = i0 + RW * j;
            lse[j] = -INFINITY;
#pragma unroll
            for (int e = 0; e < E; e++) o[j][e] = 0.0f;
            if (i < count) {
                const int64_t at = slot_row(i);
                lse[j] = p.partial_lse[at];
                const float* src = p.partial_o + at * PD + lane * E;
                if constexpr (E == 2) {
                    const float2 t = *reinterpret_cast<const float2*>(src);
                    o[j][0] = t.x; o[j][1] = t.y;
                } else {
#pragma unroll
                    for (int e = 0; e < E / 4; e++) {
                        const float4 t = *reinterpret_cast<const float4*>(src + 4 * e);
                        o[j][4 * e] = t.x; o[j][4 * e + 1] = t.y; o[j][4 * e + 2] = t.z; o[j][4 * e + 3] = t.w;
                    }
                }
            }
        }
        float mx = m;
#pragma unroll
        for (int j = 0; j < 8; j++) mx = fmaxf(mx, lse[j]);
        if (mx == -INFINITY) continue;
        const float c = fast_exp2(m - mx);
        wsum *= c;
#pragma unroll
        for (int e = 0; e < E; e++) acc[e] *= c;
        m = mx;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float w = fast_exp2(lse[j] - mx);
            if (w > 0.0f) {      // an empty part's payload is never trusted
                wsum += w;
#pragma unroll
                for (int e = 0; e < E; e++) acc[e] = fmaf(w, o[j][e], acc[e]);
            }
        }
    }
    float o[E], mm = m, wtot = wsum;
#pragma unroll
    for (int e = 0; e < E; e++) o[e] = acc[e];
    if constexpr (RW > 1) {
#pragma unroll
        for (int e = 0; e < E; e++) acc_s[warp][lane * E + e] = acc[e];
        if (lane == 0) { m_s[warp] = m; w_s[warp] = wsum; }
        __syncthreads();
        if (warp != 0) return;
#pragma unroll
        for (int w = 1; w < RW; w++) mm = fmaxf(mm, m_s[w]);
        wtot = 0.0f;
#pragma unroll
        for (int e = 0; e < E; e++) o[e] = 0.0f;
        if (mm > -INFINITY) {
#pragma unroll
            for (int w = 0; w < RW; w++) {
                const float c = fast_exp2(m_s[w] - mm);
                if (c > 0.0f) {
                    wtot += c * w_s[w];
#pragma unroll
                    for (int e = 0; e < E; e++) o[e] = fmaf(c, acc_s[w][lane * E + e], o[e]);
                }
            }
        }
    }
    const float inv = wtot > 0.0f ? 1.0f / wtot : 0.0f;
#pragma unroll
    for (int e = 0; e < E; e++) o[e] *= inv;
    split_finish<PD>(p, sign_s, b, head, r, o, wtot > 0.0f ? mm + log2f(wtot) : -INFINITY, lane);
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
int device_sm_count(int* out);
cudaEvent_t decode_event(int i);
int encode_cache_map(CUtensorMap* map, const void* kv_cache, int64_t num_blocks, int64_t row_bytes, int box_bytes, int slabs);

static size_t split_up(size_t x) { return (x + 255) & ~(size_t)255; }

// partial slots: two per group of the grid, each with the columns of one KV head
size_t split_workspace_bytes(int columns, int padded, int ctas) {
    const size_t rows = (size_t)2 * ctas * 4 * columns;
    return 256 + split_up(rows * sizeof(float)) + split_up(rows * padded * sizeof(float));
}

template <int PD, int NT, bool MANY>
static int launch_split_kernel(const SplitParams& p, cudaStream_t s) {
    using F = SplitShape<PD, NT>;
    static bool configured[64] = {};
    int dev = 0;
    TQ_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        TQ_CUDA(cudaFuncSetAttribute(decode_split_kernel<PD, NT, MANY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F::kSmem));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    TQ_CUDA(launch_serialized(decode_split_kernel<PD, NT, MANY>, dim3((unsigned)p.grid), dim3(F::kThreads), F::kSmem, s, p));
    return TQ_OK;
}

template <int PD, int NT>
static int launch_split(SplitParams& p, int ctas, cudaStream_t s) {
    using F = SplitShape<PD, NT>;
    static_assert(F::kGroups <= 4, "split_workspace_bytes counts four groups a block");
    p.grid = ctas;
    p.head_set = F::kGroups == 4 && p.kv_heads % 4 == 0 ? 4 : p.kv_heads % 2 == 0 ? 2 : 1;
    p.head_sets = p.kv_heads / p.head_set;
    p.item_cost = F::kItemCost;
    p.inv_warps = 1.0f / (float)(ctas * F::kWarps);
    int rc = encode_cache_map(&p.cache_map, p.kv_cache, p.num_blocks, (int64_t)p.kv_heads * p.slot_bytes, F::kRow, F::kSlabs);
    if (rc != TQ_OK) return rc;
    rc = p.batch > kSplitSelf ? launch_split_kernel<PD, NT, true>(p, s) : launch_split_kernel<PD, NT, false>(p, s);
    if (rc != TQ_OK) return rc;
    if (cudaEvent_t mid = decode_event(1)) TQ_CUDA(cudaEventRecord(mid, s));
    // A head has about groups / (sequences x heads) parts at most: a warp fetches eight at a time, so up to eight go to one warp
    // (a block takes four rows), more to four or sixteen warps.
    const int rows = p.batch * p.kv_heads * p.group, parts = p.grid * F::kGroups / (p.batch * p.kv_heads);
    if (parts > 32) TQ_CUDA(launch_serialized(merge_split_kernel<PD, NT, 16>, dim3((unsigned)rows), dim3(512), 0, s, p));
    else if (parts > 8) TQ_CUDA(launch_serialized(merge_split_kernel<PD, NT, 4>, dim3((unsigned)rows), dim3(128), 0, s, p));
    else TQ_CUDA(launch_serialized(merge_split_kernel<PD, NT, 1>, dim3((unsigned)(rows + 3) / 4), dim3(128), 0, s, p));
    return TQ_OK;
}

// The caller has checked pointers, types and geometry: slots a multiple of 16 bytes, padded head size 64 / 128 / 256.
int split_decode(const void* q, int q_dtype, int batch, int nq, int real_q_heads, int num_kv_heads, int head_dim, int padded,
                 const void* kv_cache, int64_t num_blocks, int slot_bytes, const int32_t* page_indices, const int32_t* page_indptr,
                 int max_pages, const int32_t* seq_lens, int64_t kv_begin, int64_t kv_end, const float* signs, float sm_scale,
                 void* workspace, size_t workspace_bytes, void* out, int out_dtype, float* out_lse, int emit_rotated,
                 int all_or_nothing, int causal, int ctas, cudaStream_t s) {
    SplitParams p{};
    p.group = nq * (real_q_heads / num_kv_heads);
    TQ_REQUIRE(p.group <= (padded == 128 ? kSplitMaxWide : kSplitMaxGroup), TQ_ERR_UNSUPPORTED, "too many query columns: %d", p.group);
    const size_t need = split_workspace_bytes(p.group, padded, ctas);
    TQ_REQUIRE(workspace_bytes >= need, TQ_ERR_WORKSPACE, "workspace too small: %zu < %zu", workspace_bytes, need);
    TQ_REQUIRE((int64_t)batch * num_kv_heads * p.group < (int64_t)1 << 31, TQ_ERR_UNSUPPORTED, "too many rows for one launch");
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    p.q = q;
    p.kv_cache = static_cast<const uint8_t*>(kv_cache);
    p.page_indices = page_indices;
    p.page_indptr = page_indptr;
    p.seq_lens = seq_lens;
    p.signs = signs;
    p.header = reinterpret_cast<int32_t*>(ws);
    p.partial_lse = reinterpret_cast<float*>(ws + 256);
    p.partial_o = reinterpret_cast<float*>(ws + 256 + split_up((size_t)2 * ctas * 4 * p.group * sizeof(float)));
    p.out = out;
    p.out_lse = out_lse;
    p.num_blocks = num_blocks;
    p.kv_begin = kv_begin;
    p.kv_end = kv_end;
    p.batch = batch;
    p.kv_heads = num_kv_heads;
    p.max_pages = max_pages;
    p.q_dtype = q_dtype;
    p.out_dtype = out_dtype;
    p.emit_rotated = emit_rotated;
    p.nq = nq;
    p.real_heads = real_q_heads;
    p.real_group = real_q_heads / num_kv_heads;
    p.head_dim = head_dim;
    p.slot_bytes = slot_bytes;
    p.all_or_nothing = all_or_nothing;
    p.causal = causal;
    const double inv = 1.0 / std::sqrt((double)padded);
    p.scale = (float)inv;
    // The table is fp16 and so is P times the V norm.  Heads of 128 / 96 share the N(0, 1) centroids with the streaming kernel and have
    // 1 / sqrt(d) in the scales; other sizes have it in their own centroids, as the plain kernel does.  Error of the output against 64 bits,
    // N(0, 1) queries and keys, with the N(0, 1) centroids / with their own: head size 80 4.7 ... 5.6e-4 / 3.6e-4; V rows of norm 1e-3 at head size
    // 64 6.8e-4 / 4.7e-4, 256 7.0e-4 / 4.7e-4 (the scale brings P times the norm 8 and 16 times nearer to fp16's subnormals).
    const bool own_table = head_dim != kHeadDim && head_dim != 96;
    float cen[16], bnd[15];
    host_codebook(padded, 4, cen, bnd);
    for (int k = 0; k < 16; k++) {
        const __half h = __float2half_rn(own_table ? cen[k] : (float)kCentroidsN01_4bit[k]);
        memcpy(&p.centroid_h[k], &h, 2);
    }
    p.v_scale = own_table ? 1.0f : (float)inv;
    p.k_scale = (float)((own_table ? 1.0 : inv) * (double)sm_scale * 1.4426950408889634);
    switch (padded) {
        case 64: return launch_split<64, 1>(p, ctas, s);
        case 128:
            switch ((p.group + 7) / 8) {
                case 1: return launch_split<128, 1>(p, ctas, s);
                case 2: return launch_split<128, 2>(p, ctas, s);
                case 3: return launch_split<128, 3>(p, ctas, s);
                default: return launch_split<128, 4>(p, ctas, s);
            }
        default: return launch_split<256, 1>(p, ctas, s);
    }
}

}  // namespace tq
