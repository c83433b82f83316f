// attn_decode.cu — one query token per sequence on the 5th-generation tensor cores (sm_100a), for
// head_dim 64, 128, 256 and 512: query norm and rotation, K/V append (single-sequence steps), split
// attention over the cache, merge and epilogue in ONE launch.
//
// Replaces attention_decode, attention_decode_split and attention_decode_merge
// (Sources/HydraMetal/Shaders/attention.metal:132-242, 307-452) together with the rms_norm_heads,
// rope_apply and kv_cache_write launches in front of them.
//
// A decode row tile has at most 16 real rows (the query heads of one kv head), so the contractions are
// turned round: the 128 keys of a tile are the M side of S^T = K Q^T (N = 16) and the head_dim
// columns the M side of O^T = V^T P^T.  K and V are the operands as they lie in the cache (V transposed by its
// descriptor), the query tile costs 32 bytes per element of head_dim instead of 256, an accumulator
// costs 16 columns of tensor memory, and what is left of shared memory (128 to 192 KB) holds rings of K
// and V boxes in flight, which is what a kernel bound by HBM latency x bandwidth needs (one 128-row
// query tile and single K/V stages took 37 us for 67 MB of head_dim 256 cache, 1.8 TB/s).
// The tensor core gives an accumulator element the same bits whichever operand plays M (measured),
// so a tile's partial is the prefill kernels' bit for bit.
//
//   warp 0       TMA producer: boxes of 128 keys x 64 columns into a K ring and a V ring
//   warp 1       issues S^T, up to four tiles ahead
//   warp 2       issues O^T
//   warp 3       queries of later items: norm, rotation, rounding, into the operand layout; with a fused
//                append, also the token's own K and V rows, ahead of the load of their tile
//   warps 4-7, 8-11   softmax of alternate tiles, thread = key: maximum over the keys of a tile by a
//                warp reduction and shared memory, weights rounded to bf16 into the P operand
//   warps 12-15  fold, thread = head_dim column: the tile partials of an item into its segment, partials
//                out, and the merge
//
// Two ways to cut a launch (tc_plan_decode):
//   a line     the rows (sequence, kv head) with their key tiles lie one behind the other, and every thread block takes
//              an equal stretch of the line, cut at segment boundaries.  A row that lies inside one stretch
//              is finished there; the others leave one partial per segment in global memory.  (Dealing
//              out runs of segments round robin left the last thread block of 64 ragged sequences 25 % behind
//              the average; equal stretches leave half a segment.)
//   clusters   few long rows: the 2 to 16 thread blocks of a cluster share a row, or a span of its segments, and
//              every tile's partial is pushed, value by value, into the shared memory of the block
//              that folds that slice of the columns: no partial touches global memory, no
//              thread block folds more than its slice, and a row that fits a cluster needs no ticket.
// Cut rows end in tickets that count tiles: the thread block whose tiles complete a row (or a slice of it) folds what
// the others left.  Nobody waits for anybody.  It also puts the ticket back to zero.
//
// Every wait on an mbarrier is bounded (see tc_ptx.cuh).

#include <algorithm>

#include "internal.hpp"
#include "prologue.cuh"
#include "tc_common.cuh"
#include "tc_ptx.cuh"

namespace hc {
namespace {

constexpr int kBoxBytes = kTileKeys * 128;      // 128 keys x 64 columns of bf16
constexpr int kQRows = 16;                      // N of both contractions
constexpr int kSBuf = 4;                        // S^T accumulators in tensor memory
constexpr int kPBytes = kQRows * 128 * 2;       // one P^T operand: 16 rows x 128 keys
constexpr int kPushBytes = 32 * 1024;           // room for the tile partials pushed to a block of a cluster
constexpr int kPushTiles = 256;                 // and their number

template <int D>
struct DecLayout {
    static constexpr int kBlocks = D / 64;                        // 64-column blocks of a row
    // K and V have a ring each: two warps consume them, and a stage's phase bit means something only to a
    // consumer that sees every use of the stage.  A K stage is one box; a V stage two side by side (M = 128).
    static constexpr int kVBoxes = D == 64 ? 1 : 2;
    static constexpr int kVStageBytes = kVBoxes * kBoxBytes;
    static constexpr int kVTileStages = kBlocks / kVBoxes;        // V stages of one tile
    static constexpr int kKStages = 4;
    static constexpr int kVStages = D == 64 ? 5 : D == 512 ? 2 : 3;
    static constexpr int kMBlocks = D <= 128 ? 1 : D / 128;       // 128-row blocks of O^T
    static constexpr bool kSumOnTensor = D == 64;                 // rows 64.. of O^T: the row sums, by a block of ones
    static constexpr int kQBlock = kQRows * 128;                  // 64 columns of the query tile
    static constexpr int kQBytes = kBlocks * kQBlock;
    static constexpr int kOCol = kSBuf * kQRows;
    static constexpr int kOCols = kMBlocks * kQRows;
    static constexpr int kTmemCols = kOCol + 2 * kOCols <= 128 ? 128 : 256;
    static constexpr int kOnesBytes = kSumOnTensor ? kBoxBytes : 0;
    static constexpr int kKRingBytes = kKStages * kBoxBytes;
    static constexpr int kRingBytes = kKRingBytes + kVStages * kVStageBytes;
    static constexpr int kStateBytes = kPushBytes;    // pushed partials, or the second fold of a whole-row item
    static_assert(kMBlocks * kQRows * 128 * 4 <= kStateBytes, "the second fold fits");
    static constexpr int kSmemBytes = 1024 + kRingBytes + kOnesBytes + 2 * kQBytes + 2 * kPBytes + kStateBytes;
};

struct DecArgs {
    // The query (and the token's own k, v when they are appended here) as they come.
    const void* q;
    const void* k_new;               // null: the rows are in the cache already
    const void* v_new;
    int src_dtype;
    int q_head_stride;               // 2 d for an interleaved gate
    int norm_q, norm_k, norm_v;
    const uint16_t* q_weight;
    const uint16_t* k_weight;
    float eps;
    const float* cos;                // null: no rotation
    const float* sin;
    int table_positions;
    CacheView cache;
    int q_heads;
    int log_group;
    int window;
    float c;
    const uint16_t* sinks;
    int count_sink;
    EpilogueArgs ep;
    int* status;
    // The cut (see TcDecodePlan): a line of n_tiles tiles over the thread blocks, or clusters of `cluster` blocks per
    // span of seq_run[b] segments.
    int n_seq;
    int cluster;                     // 1: a line
    int slots;                       // partial slots per row: segments
    float* part_o;                   // fp32 [rows][slots][d]
    float* part_ml;                  // fp32 [rows][slots][2]
    unsigned* tickets;               // [n_seq * kv_heads][cluster]: tiles whose partials are there
    int n_tiles;
    int start[kMaxBatch + 1];        // line: tiles (of all kv heads) before sequence b; clusters: spans before it
    unsigned short seq_run[kMaxBatch];
    unsigned short seq_spans[kMaxBatch];
    BatchMeta meta;
};

struct DecItem {
    int b, kv_head;
    int tile_first, n_tiles;         // key tiles, `world` apart
    bool last;                       // holds the row's last key tile: the one the token's own key lies in
    bool whole;                      // line: all of the row, finished by this block
};

// b with start[b] <= index < start[b + 1]
__host__ __device__ __forceinline__ int dec_search(const DecArgs& args, int index) {
    int lo = 0, hi = args.n_seq;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (index >= args.start[mid]) lo = mid; else hi = mid;
    }
    return lo;
}

// Rows of a tile or two are never cut, not at a segment's boundary either: the merge costs more than their tiles
// (8 sequences x 8 kv heads of a 128-key window, some rows across a boundary: 12.3 us cut there, 7.1 whole).
constexpr int kDecUncut = 2;

// Where the stretch of the line begins that block c of `blocks` takes: a row and a tile of it, the equal share's end moved to
// the nearest segment boundary.  (The host asks too, for the rows that the longest list holds.)
struct DecPlace {
    int row, t;
};
__host__ __device__ __forceinline__ DecPlace dec_place(const DecArgs& args, int c, int blocks) {
    DecPlace p;
    p.row = args.n_seq * args.cache.kv_heads;
    p.t = 0;
    if (c >= blocks) return p;
    const int at = int((long long)c * args.n_tiles / blocks);
    const int b = dec_search(args, at);
    const int world = args.cache.map.world > 1 ? args.cache.map.world : 1;
    const int log_segment = args.cache.map.log_segment;
    const TileRange row = row_tiles(args.cache.map, args.meta.pos[b], args.meta.pos[b], args.window);
    if (row.count <= 0) return p;                        // (an empty launch)
    const int head = (at - args.start[b]) / row.count;
    const int t = at - args.start[b] - head * row.count;
    const int segment_tile = ((row.first + t * world) >> log_segment) << log_segment;
    int before = segment_tile <= row.first ? 0 : (segment_tile - row.first + world - 1) / world;
    const int next = (segment_tile + (1 << log_segment) - row.first + world - 1) / world;
    int after = next < row.count ? next : row.count;
    if (row.count <= kDecUncut) {
        before = 0;
        after = row.count;
    }
    p.row = b * args.cache.kv_heads + head;
    p.t = t - before <= after - t ? before : after;
    if (p.t == row.count) {
        p.t = 0;
        ++p.row;
    }
    return p;
}
// The list of the block that starts at `from` and ends at `to`.
__host__ __device__ __forceinline__ int dec_items(const DecPlace& from, const DecPlace& to) {
    return to.row - from.row + (to.t > 0 ? 1 : 0);
}

// A thread block's items, worked out once by all its threads side by side (finding an item takes a search and
// a few divisions, thousands of clocks for a single thread, and every role needs every item) and packed
// into twelve bytes each; a tile's index takes 24 bits, positions being ints.  (Eight bytes, with the first tile worked
// out from the position again by every reader: batches of 64 long sequences 2 % slower.)
constexpr int kDecItems = 340;       // of one thread block, at most: what head_dim 256 leaves of shared memory
struct DecPacked {
    uint32_t what;                   // sequence, kv head, flags
    int tile_first, n_tiles;
};
static_assert(kMaxBatch <= 64, "the sequence has six bits");
struct DecList {
    DecPacked packed[kDecItems];
    int pos[kMaxBatch], seq[kMaxBatch];
    int count;
    int span_first, span_tiles;      // of the cluster
};
__device__ __forceinline__ DecPacked dec_pack(const DecItem& w) {
    DecPacked p;
    p.what = uint32_t(w.b) | (uint32_t(w.kv_head) << 6) | (w.whole ? 0x40000000u : 0u) | (w.last ? 0x80000000u : 0u);
    p.tile_first = w.tile_first;
    p.n_tiles = w.n_tiles;
    return p;
}
__device__ __forceinline__ DecItem dec_unpack(const DecPacked& p) {
    DecItem w;
    w.b = int(p.what & 0x3fu);
    w.kv_head = int((p.what >> 6) & 0xffffffu);
    w.whole = (p.what & 0x40000000u) != 0;
    w.last = (p.what >> 31) != 0;
    w.tile_first = p.tile_first;
    w.n_tiles = p.n_tiles;
    return w;
}
__device__ __forceinline__ void dec_list_build(const DecArgs& args, DecList* list) {
    const int world = args.cache.map.world > 1 ? args.cache.map.world : 1;
    for (int i = threadIdx.x; i < args.n_seq; i += kTcThreads) {
        list->pos[i] = args.meta.pos[i];
        list->seq[i] = args.meta.seq[i];
    }
    if (args.cluster > 1) {
        if (threadIdx.x != 0) return;
        // This block's share of the cluster's span.
        const int span = int(blockIdx.x) / args.cluster, rank = int(blockIdx.x) & (args.cluster - 1);
        DecItem w;
        w.b = dec_search(args, span);
        const int spans = args.seq_spans[w.b], run = args.seq_run[w.b], pos = args.meta.pos[w.b];
        w.kv_head = (span - args.start[w.b]) / spans;
        const int ordinal = span - args.start[w.b] - w.kv_head * spans;
        const TileRange tiles = segment_run_tiles(args.cache.map, pos, pos, args.window, ordinal * run, run);
        const int share = (max(tiles.count, 0) + args.cluster - 1) / args.cluster;
        w.n_tiles = max(min(share, tiles.count - rank * share), 0);
        w.tile_first = tiles.first + rank * share * world;
        w.last = w.n_tiles > 0 && w.tile_first + (w.n_tiles - 1) * world == pos / kTileKeys;
        w.whole = false;
        list->packed[0] = dec_pack(w);
        list->count = 1;
        list->span_first = tiles.first;
        list->span_tiles = max(tiles.count, 0);
        return;
    }
    const DecPlace from = dec_place(args, int(blockIdx.x), int(gridDim.x)), to = dec_place(args, int(blockIdx.x) + 1, int(gridDim.x));
    const int count = min(dec_items(from, to), kDecItems);
    if (threadIdx.x == 0) list->count = count;
    for (int i = threadIdx.x; i < count; i += kTcThreads) {
        DecItem w;
        const int r = from.row + i;
        w.b = r / args.cache.kv_heads;
        w.kv_head = r - w.b * args.cache.kv_heads;
        const int pos = args.meta.pos[w.b];
        const TileRange row = row_tiles(args.cache.map, pos, pos, args.window);
        const int t0 = i == 0 ? from.t : 0, t1 = r == to.row ? to.t : max(row.count, 0);
        w.tile_first = row.first + t0 * world;
        w.n_tiles = t1 - t0;
        w.last = w.n_tiles > 0 && t1 == row.count && row.first + (row.count - 1) * world == pos / kTileKeys;
        w.whole = t0 == 0 && t1 == row.count;
        list->packed[i] = dec_pack(w);
    }
}

// The walk over the list; items without tiles (sequence shards) are passed over.
struct DecIter {
    int i, count;
    DecItem w;
    __device__ __forceinline__ bool more() const { return i < count; }
};
__device__ __forceinline__ void dec_seek(const DecList* list, DecIter& it) {
    for (; it.i < it.count; ++it.i) {
        it.w = dec_unpack(list->packed[it.i]);
        if (it.w.n_tiles > 0) return;
    }
}
__device__ __forceinline__ DecIter dec_begin(const DecList* list) {
    DecIter it;
    it.i = 0;
    it.count = list->count;
    it.w = DecItem{};
    dec_seek(list, it);
    return it;
}
__device__ __forceinline__ void dec_next(const DecList* list, DecIter& it) {
    ++it.i;
    dec_seek(list, it);
}

struct DecBarriers {
    uint64_t k_full[6], k_empty[6], v_full[6], v_empty[6];
    uint64_t q_first, q_full[2], q_empty[2];
    uint64_t s_full[kSBuf], s_free[kSBuf];
    uint64_t p_full[2], p_free[2];
    uint64_t o_full[2], o_free[2];
    uint64_t merge_full[2];
    uint32_t tmem_base;
    int abort_flag;
    int n_work;                             // rows that this block completes
    int cut;                                // line: some item is not a whole row
    uint32_t staged;                        // items whose queries and appended rows are written
    __align__(16) float red[2][2][4][kQRows];           // per softmax group, alternate tiles: the warps' maxima
    __align__(16) float mm[4][kQRows];                  // scaled maxima of a tile, softmax -> fold (ring of 4 tiles)
    __align__(16) float lsum[4][4][kQRows];             // sums of 32 weights, softmax -> fold
    __align__(16) float2 coef[4][kQRows];               // per fold warp: the fold's coefficients of the tile
    __align__(16) float denom[2][kQRows];               // a row's L, to all fold threads (alternate items)
    float push_m[kPushTiles], push_l[kPushTiles];       // [tile][row of the slice]: a pushed partial's maximum and sum
    uint32_t n_last;                                    // outcome of a slice's ticket
};

// ---- queries (and appended rows) of one item: passes first, first + stride, .. of the item's vectors ----
template <int D, int NV>
__device__ __forceinline__ void dec_stage(const DecArgs& args, const DecList* list, const DecItem& w, unsigned char* q_dst, int first,
                                          int stride) {
    using HL = HeadLanes<D>;
    const int lane = threadIdx.x & 31;
    const int sub = lane / HL::kLanes, m = lane % HL::kLanes;
    const int G = 1 << args.log_group;
    const bool append = args.k_new != nullptr && w.last;
    const int total = G + (append ? 2 : 0);
    const int passes = (total + HL::kPerWarp - 1) / HL::kPerWarp;
    if (first >= passes) return;
    const bool rotate = args.cos != nullptr;
    const bool any_norm = (args.norm_q | (append ? args.norm_k | args.norm_v : 0)) != 0;
    float c[HL::kElems], s[HL::kElems];
    if (rotate) {
        const int table_row = min(list->pos[w.b], args.table_positions - 1);
        load_rotation<D>(args.cos + size_t(table_row) * (D / 2), args.sin + size_t(table_row) * (D / 2), m, c, s);
    }
    for (int p0 = first; p0 < passes; p0 += stride * NV) {
        float lo[NV][HL::kElems], hi[NV][HL::kElems];
        #pragma unroll
        for (int u = 0; u < NV; ++u) {
            const int vec = min((p0 + u * stride) * HL::kPerWarp + sub, total - 1);
            const void* src = vec < G ? args.q : vec == G ? args.k_new : args.v_new;
            const size_t base = vec < G
                ? (size_t(w.b) * args.q_heads + size_t(w.kv_head) * G + vec) * args.q_head_stride
                : (size_t(w.b) * args.cache.kv_heads + w.kv_head) * D;
            load_head<D>(src, base, args.src_dtype, m, lo[u], hi[u]);
        }
        #pragma unroll
        for (int u = 0; u < NV; ++u) {
            if (p0 + u * stride >= passes) break;                 // warp-uniform
            const int vec = (p0 + u * stride) * HL::kPerWarp + sub;
            const int norm = vec < G ? args.norm_q : vec == G ? args.norm_k : args.norm_v;
            float wl[HL::kElems], wh[HL::kElems];
            if (norm == 1) load_head<D>(vec < G ? args.q_weight : args.k_weight, 0, 1, m, wl, wh);
            prepare_head<D>(lo[u], hi[u], norm, wl, wh, args.eps, rotate && vec <= G, c, s, any_norm);
            if (vec >= total) continue;
            #pragma unroll
            for (int x = 0; x < HL::kVecs; ++x) {
                const float a[4] = {lo[u][4 * x], lo[u][4 * x + 1], lo[u][4 * x + 2], lo[u][4 * x + 3]};
                const float b[4] = {hi[u][4 * x], hi[u][4 * x + 1], hi[u][4 * x + 2], hi[u][4 * x + 3]};
                #pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int e = h * (D / 2) + 4 * (m + x * HL::kLanes);
                    const uint2 packed = pack_bf16x4(h == 0 ? a : b);
                    if (vec < G) {
                        unsigned char* at = q_dst + (e >> 6) * (kQRows * 128) + vec * 128 + ((((e & 63) >> 3) ^ (vec & 7)) << 4) + (e & 7) * 2;
                        *reinterpret_cast<uint2*>(at) = packed;
                    } else {
                        uint16_t* rows = vec == G ? args.cache.k : args.cache.v;
                        const int seq = list->seq[w.b];
                        const size_t row = size_t(cache_plane(args.cache.map, seq, args.cache.kv_heads, w.kv_head)) * args.cache.capacity +
                                           cache_row(args.cache.map, seq, list->pos[w.b]);
                        *reinterpret_cast<uint2*>(rows + row * D + e) = packed;
                    }
                }
            }
        }
    }
    // Both the operand tile (shared) and the appended rows (global) are read by the async proxy next; the fence
    // that covers global memory waits for the rows to get there, seven hundred clocks.
    if (append) asm volatile("fence.proxy.async;" ::: "memory");
    else fence_proxy_async();
}

// ---- merge -------------------------------------------------------------------------------------------------
__device__ __forceinline__ bool dec_segment_present(const DecArgs& args, int pos, int ordinal) {
    return args.cache.map.world <= 1 || group_tiles(args.cache.map, pos, pos, args.window, ordinal, args.cache.map.log_segment).count > 0;
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ float dec_sink(const DecArgs& args, int head) {
    return __fmul_rn(bf16_bits_to_float(args.sinks ? args.sinks[head] : kNoSinkBits), kLog2e);
}
// One value of a finished row (or of a shard's partial), column col of head row `vec`.
__device__ __forceinline__ void dec_write(const DecArgs& args, int d, size_t vec, int col, float A, float M, float L) {
    if (args.ep.write_partial) {
        float* dst = reinterpret_cast<float*>(args.ep.out) + vec * size_t(d + 2);
        dst[col] = A;
        if (col == 0) {
            dst[d] = M;
            dst[d + 1] = L;
        }
        return;
    }
    const bool gated = args.ep.gate_layout != HC_GATE_NONE;
    const size_t gate_at = (args.ep.gate_layout == HC_GATE_INTERLEAVED ? vec * size_t(2 * d) + d : vec * size_t(d)) + col;
    const float gv = gated ? load_io(args.ep.gate, gate_at, args.ep.io_dtype) : 0.0f;
    store_io(args.ep.out, vec * d + col, args.ep.io_dtype, finish_value(A, L, gated, gv));
}

// A fold's coefficients depend on the maxima alone.  A warp computes those of up to 32 consecutive partials at once,
// lane = partial (lanes that have none pass -inf): the prefix maximum from `carry` on, which it moves along.
// Prefix maxima are exact, so these are the bits that fold_coefficients gives one after the other.
__device__ __forceinline__ float2 warp_fold_coefficients(float m, float& carry) {
    const int lane = threadIdx.x & 31;
    float prefix = fmaxf(m, carry);
    #pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
        const float other = __shfl_up_sync(0xffffffffu, prefix, offset);
        if (lane >= offset) prefix = fmaxf(prefix, other);
    }
    float before = __shfl_up_sync(0xffffffffu, prefix, 1);
    if (lane == 0) before = carry;
    carry = __shfl_sync(0xffffffffu, prefix, 31);
    return make_float2(ex2(__fsub_rn(before, prefix)), ex2(__fsub_rn(m, prefix)));
}

// Scratch of the merges, in the P operands' place.
struct DecMerge {
    union {
        struct {
            float2 coef[kQRows][32];     // dec_fold: a row's coefficients over a piece of up to 32 segments
            float l[kQRows][32];         // and the partials' row sums
        } rows;
        struct {
            float2 coef[kPushTiles];     // dec_fold_slice: [row of the slice][tile]
            float2 end[kPushTiles];      // [row of the slice][segment]: the step that ends a segment
        } slice;
    };
    float M[kQRows], L[kQRows];
};
static_assert(sizeof(DecMerge) <= 2 * kPBytes, "fits in the P operands' place");

// The second fold over the segment partials of one (batch entry, kv head), by the whole block.  The rings are free by
// then and take the partials, up to 32 slots at a time, two such pieces in flight, one bulk copy per row (a
// row's slots are contiguous); per partial and value that leaves two multiplies and an add.
template <int D, int NG>
__device__ __forceinline__ void dec_fold(const DecArgs& args, const DecItem& w, int pos, float* ring, DecMerge* sm,
                                         uint64_t* bars, uint32_t& loads, volatile int* abort_flag) {
    constexpr int kCols = NG * D / kTcThreads > 0 ? NG * D / kTcThreads : 1;      // values of a thread
    constexpr int kHalfFloats = DecLayout<D>::kRingBytes / 8;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int G = 1 << args.log_group;
    const bool shard = args.cache.map.world > 1;           // segments without a tile of this rank were never written
    const int count = visible_groups(pos, pos, args.window, args.cache.map.log_segment);
    const size_t row0 = size_t(w.b) * args.q_heads + size_t(w.kv_head) * G;
    const float* part_o = args.part_o + row0 * args.slots * D;
    const float* part_ml = args.part_ml + row0 * args.slots * 2;
    const int most = min(32, kHalfFloats / (G * D));
    float2 ml_next = make_float2(0.0f, 0.0f);
    auto fetch = [&](int s, int n) {                      // piece [s, s + n): into the half that `loads` points at
        float* dst = ring + (loads & 1) * kHalfFloats;
        uint64_t* bar = bars + (loads & 1);
        if (tid == 0) {
            mbar_expect_tx(bar, uint32_t(G * n * D * 4));
            #pragma unroll 1
            for (int g = 0; g < G; ++g) bulk_load(dst + g * n * D, part_o + (size_t(g) * args.slots + s) * D, uint32_t(n * D * 4), bar);
        }
        if (warp < G && lane < n) ml_next = __ldcg(reinterpret_cast<const float2*>(part_ml + (size_t(warp) * args.slots + s + lane) * 2));
        ++loads;
    };
    float A[kCols], L = args.count_sink ? 1.0f : 0.0f;     // L: of row tid, in the first G threads
    float M = kEmptyMax;                                   // of row `warp`, in its warp
    #pragma unroll
    for (int i = 0; i < kCols; ++i) A[i] = 0.0f;
    if (args.count_sink && warp < G) M = dec_sink(args, w.kv_head * G + warp);
    if (tid == 0) asm volatile("fence.proxy.async;" ::: "memory");
    int n = min(most, count);
    fetch(0, n);
    #pragma unroll 1
    for (int s0 = 0; s0 < count;) {
        const float* part = ring + ((loads - 1) & 1) * kHalfFloats;
        uint64_t* bar = bars + ((loads - 1) & 1);
        const uint32_t parity = ((loads - 1) >> 1) & 1;
        const float2 ml = ml_next;
        const int after = s0 + n;
        const int n_after = min(most, count - after);
        if (n_after > 0) fetch(after, n_after);
        if (warp < G) {
            const bool there = lane < n && (!shard || dec_segment_present(args, pos, s0 + lane));
            sm->rows.coef[warp][lane] = warp_fold_coefficients(there ? ml.x : __int_as_float(0xff800000), M);
            sm->rows.l[warp][lane] = ml.y;
        }
        mbar_wait(bar, parity, abort_flag, args.status, 53);
        __syncthreads();
        #pragma unroll 2
        for (int u = 0; u < n; ++u) {
            if (shard && !dec_segment_present(args, pos, s0 + u)) continue;
            #pragma unroll
            for (int i = 0; i < kCols; ++i) {
                const int index = tid + i * kTcThreads;
                const int row = min(index / D, G - 1);
                const float2 c = sm->rows.coef[row][u];
                A[i] = fold_value(A[i], c.x, part[(row * n + u) * D + index % D], c.y);
            }
            if (tid < G) {
                const float2 c = sm->rows.coef[tid][u];
                L = __fmaf_rn(L, c.x, __fmul_rn(sm->rows.l[tid][u], c.y));
            }
        }
        __syncthreads();                                  // before the half and the coefficients are written again
        s0 = after;
        n = n_after;
    }
    if (warp < G && lane == 0) sm->M[warp] = M;
    if (tid < G) sm->L[tid] = L;
    __syncthreads();
    #pragma unroll
    for (int i = 0; i < kCols; ++i) {
        const int index = tid + i * kTcThreads;
        const int row = index / D;
        if (row < G) dec_write(args, D, row0 + row, index % D, A[i], sm->M[row], sm->L[row]);
    }
    __syncthreads();
}

// Counts tiles on a ticket; true for whoever completes the row.
__device__ __forceinline__ bool dec_last_ticket(unsigned* ticket, int tiles, int of) {
    if (atomicAdd(ticket, unsigned(tiles)) + unsigned(tiles) != unsigned(of)) return false;
    atomicExch(ticket, 0u);
    return true;
}

// A line's block that has written its partials counts them on its rows' tickets (all at once, a thread each), and folds
// the rows that this completes.
template <int D, int NG>
__device__ __forceinline__ void dec_close(const DecArgs& args, const DecList* list, float* ring, DecMerge* sm, int* work, int* n_work,
                                          uint64_t* bars, volatile int* abort_flag) {
    uint32_t loads = 0;
    __threadfence();                                    // the partials, before the tickets
    __syncthreads();
    for (int i = threadIdx.x; i < list->count; i += kTcThreads) {
        const DecItem w = dec_unpack(list->packed[i]);
        if (w.n_tiles == 0 || w.whole) continue;
        const int pos = list->pos[w.b];
        if (dec_last_ticket(args.tickets + w.b * args.cache.kv_heads + w.kv_head, w.n_tiles,
                            row_tiles(args.cache.map, pos, pos, args.window).count)) {
            work[atomicAdd(n_work, 1)] = i;
        }
    }
    __threadfence();
    __syncthreads();
    const int todo = *n_work;
    #pragma unroll 1
    for (int k = 0; k < todo; ++k) {
        const DecItem w = dec_unpack(list->packed[work[k]]);
        dec_fold<D, NG>(args, w, list->pos[w.b], ring, sm, bars, loads, abort_flag);
    }
}

// ---- clusters ----------------------------------------------------------------------------------------------
// The G x D values of a row group are cut into as many slices as the cluster has blocks, G D / cluster consecutive
// values each: part of one row, or several whole rows.
__device__ __forceinline__ void cluster_store(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
// This block's slice: both folds over the span's pushed tile partials when the span is the whole row, otherwise the
// first fold of every segment, and the second by the slice's last span.
template <int D>
__device__ __forceinline__ void dec_fold_slice(const DecArgs& args, const DecList* list, const float* pushed, const float* push_m,
                                               const float* push_l, DecMerge* sm, uint32_t* n_last) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int G = 1 << args.log_group;
    const int world = args.cache.map.world > 1 ? args.cache.map.world : 1;
    const int log_segment = args.cache.map.log_segment;
    const int rank = int(blockIdx.x) & (args.cluster - 1);
    const DecItem w = dec_unpack(list->packed[0]);
    const int pos = list->pos[w.b];
    const int tiles = list->span_tiles, tile0 = list->span_first;
    const int width = G * D / args.cluster;                // values of the slice
    const int rows = width > D ? width / D : 1;
    const int first_row = rank * width / D;
    const int first_segment = first_visible_tile(pos, args.window) >> log_segment;
    const int base_segment = (tile0 >> log_segment) - first_segment;         // ordinal of the span's first segment
    const bool whole = args.seq_spans[w.b] == 1;
    const size_t row0 = size_t(w.b) * args.q_heads + size_t(w.kv_head) * G;
    const size_t slot0 = (row0 + first_row) * args.slots;                    // partial slot 0 of the slice's first row
    const int segments = tiles > 0 ? ((tile0 + (tiles - 1) * world) >> log_segment) - (tile0 >> log_segment) + 1 : 0;
    // Partials before the running segment's end: the tiles of one segment, 32 at most.
    auto run_of = [&](int s) -> int {
        const int tile = tile0 + s * world;
        const int end = ((tile >> log_segment) + 1) << log_segment;
        return min(tiles - s, (end - tile + world - 1) / world);
    };
    if (warp < rows) {
        float M = args.count_sink ? dec_sink(args, w.kv_head * G + first_row + warp) : kEmptyMax;
        #pragma unroll 1
        for (int s = 0; s < tiles;) {
            const int n = run_of(s);
            const int segment = ((tile0 + s * world) >> log_segment) - (tile0 >> log_segment);
            float m1 = kEmptyMax;
            const float2 c = warp_fold_coefficients(lane < n ? push_m[(s + lane) * rows + warp] : __int_as_float(0xff800000), m1);
            if (lane < n) sm->slice.coef[warp * tiles + s + lane] = c;
            float Mn, a, b;
            fold_coefficients(M, m1, Mn, a, b);
            M = Mn;
            if (lane == 0) {
                sm->slice.end[warp * segments + segment] = make_float2(a, b);
                if (!whole) args.part_ml[(slot0 + size_t(warp) * args.slots + base_segment + segment) * 2] = m1;
            }
            s += n;
        }
        if (lane == 0) sm->M[warp] = M;
    }
    __syncthreads();
    // Values, and behind them the row sums, which fold the same way.
    #pragma unroll 1
    for (int i = tid; i < width + rows; i += kTcThreads) {
        const bool is_sum = i >= width;
        const int row = is_sum ? i - width : (width > D ? i / D : 0);
        const int col = (rank * width + i) % D;
        const float* src = is_sum ? push_l + row : pushed + i;
        const int stride = is_sum ? rows : width;
        const float2* coef = sm->slice.coef + row * tiles;
        float A = is_sum && args.count_sink ? 1.0f : 0.0f, a1 = 0.0f;
        int segment = 0;
        #pragma unroll 1
        for (int s = 0; s < tiles;) {
            const int end = s + run_of(s);
            #pragma unroll 4
            for (; s < end; ++s) a1 = fold_value(a1, coef[s].x, src[s * stride], coef[s].y);
            if (whole) {
                const float2 c = sm->slice.end[row * segments + segment];
                A = fold_value(A, c.x, a1, c.y);
            } else {
                const size_t at = slot0 + size_t(row) * args.slots + base_segment + segment;
                if (is_sum) args.part_ml[at * 2 + 1] = a1;
                else args.part_o[at * D + col] = a1;
            }
            a1 = 0.0f;
            ++segment;
        }
        if (is_sum) sm->L[row] = A;
        else if (whole) const_cast<float*>(pushed)[i] = A;
    }
    if (whole) {
        __syncthreads();
        #pragma unroll 1
        for (int i = tid; i < width; i += kTcThreads) {
            const int row = width > D ? i / D : 0;
            dec_write(args, D, row0 + first_row + row, (rank * width + i) % D, pushed[i], sm->M[row], sm->L[row]);
        }
        return;
    }
    // The slice's ticket.
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        *n_last = tiles > 0 && dec_last_ticket(args.tickets + (w.b * args.cache.kv_heads + w.kv_head) * args.cluster + rank, tiles,
                                               row_tiles(args.cache.map, pos, pos, args.window).count) ? 1u : 0u;
        __threadfence();
    }
    __syncthreads();
    if (*n_last == 0) return;
    // The second fold over the slice's segments, up to 32 at a time: the values' loads go out before the coefficients,
    // which a warp per row works out, are there.
    const int count = visible_groups(pos, pos, args.window, log_segment);
    float M = kEmptyMax, L = args.count_sink ? 1.0f : 0.0f;                  // of row `warp`, in its warp
    if (args.count_sink && warp < rows) M = dec_sink(args, w.kv_head * G + first_row + warp);
    #pragma unroll 1
    for (int s0 = 0; s0 < count; s0 += 32) {
        const int n = min(32, count - s0);
        float2 ml = make_float2(0.0f, 0.0f);
        if (warp < rows && lane < n) ml = __ldcg(reinterpret_cast<const float2*>(args.part_ml + (slot0 + size_t(warp) * args.slots + s0 + lane) * 2));
        float v[16];
        auto load = [&](int i, int u0) {
            const int row = width > D ? i / D : 0;
            const float* src = args.part_o + (slot0 + size_t(row) * args.slots + s0 + u0) * D + (rank * width + i) % D;
            #pragma unroll
            for (int u = 0; u < 16; ++u) v[u] = u0 + u < n ? __ldcg(src + size_t(u) * D) : 0.0f;
        };
        if (tid < width) load(tid, 0);
        if (warp < rows) {
            const bool there = lane < n && dec_segment_present(args, pos, s0 + lane);
            const float2 c = warp_fold_coefficients(there ? ml.x : __int_as_float(0xff800000), M);
            sm->slice.coef[warp * 32 + lane] = c;
            const float lb = there ? __fmul_rn(ml.y, c.y) : 0.0f;
            #pragma unroll 1
            for (int u = 0; u < n; ++u) L = __fmaf_rn(L, __shfl_sync(0xffffffffu, c.x, u), __shfl_sync(0xffffffffu, lb, u));
            if (lane == 0) {
                sm->M[warp] = M;
                sm->L[warp] = L;
            }
        }
        __syncthreads();
        #pragma unroll 1
        for (int i = tid; i < width; i += kTcThreads) {
            const float2* coef = sm->slice.coef + (width > D ? i / D : 0) * 32;
            float A = s0 == 0 ? 0.0f : pushed[i];
            #pragma unroll 1
            for (int u0 = 0; u0 < n; u0 += 16) {
                if (i != tid || u0 != 0) load(i, u0);
                #pragma unroll
                for (int u = 0; u < 16; ++u) {
                    if (u0 + u >= n || !dec_segment_present(args, pos, s0 + u0 + u)) continue;
                    const float2 c = coef[u0 + u];
                    A = fold_value(A, c.x, v[u], c.y);
                }
            }
            const_cast<float*>(pushed)[i] = A;
        }
        __syncthreads();
    }
    #pragma unroll 1
    for (int i = tid; i < width; i += kTcThreads) {
        const int row = width > D ? i / D : 0;
        dec_write(args, D, row0 + first_row + row, (rank * width + i) % D, pushed[i], sm->M[row], sm->L[row]);
    }
}

// Rows that this rank of a sequence shard holds no key of are nobody's item: the seed is their result.
template <int D, int NG>
__device__ __forceinline__ void dec_seed_rows(const DecArgs& args) {
    const int G = 1 << args.log_group;
    for (int r = blockIdx.x; r < args.n_seq * args.cache.kv_heads; r += gridDim.x) {
        const int b = r / args.cache.kv_heads;
        const int pos = args.meta.pos[b];
        if (row_tiles(args.cache.map, pos, pos, args.window).count > 0) continue;
        for (int i = threadIdx.x; i < G * D; i += kTcThreads) {
            const int row = i / D, col = i % D;
            const int head = (r - b * args.cache.kv_heads) * G + row;
            const size_t vec = size_t(b) * args.q_heads + head;
            const float L = args.count_sink ? 1.0f : 0.0f;
            if (args.ep.write_partial) {
                float* dst = reinterpret_cast<float*>(args.ep.out) + vec * size_t(D + 2);
                dst[col] = 0.0f;
                if (col == 0) {
                    dst[D] = args.count_sink ? __fmul_rn(bf16_bits_to_float(args.sinks ? args.sinks[head] : kNoSinkBits), kLog2e) : kEmptyMax;
                    dst[D + 1] = L;
                }
            } else {
                store_io(args.ep.out, vec * D + col, args.ep.io_dtype, 0.0f);
            }
        }
    }
}

// S^T or O^T columns of this lane: 8 or 16 of them.
template <int N>
__device__ __forceinline__ void tmem_ld_cols(uint32_t addr, uint32_t (&v)[N]) {
    static_assert(N == 8 || N == 16, "8 or 16 columns");
    if constexpr (N == 8) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                     : "r"(addr) : "memory");
    } else {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                       "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                     : "r"(addr) : "memory");
    }
}
__device__ __forceinline__ float warp_max(float v) {
    float m;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(m) : "f"(v));
    return m;
}
template <int N>
__device__ __forceinline__ void load_row(const float* src, float (&v)[N]) {
    #pragma unroll
    for (int i = 0; i < N; i += 4) {
        const float4 x = *reinterpret_cast<const float4*>(src + i);
        v[i] = x.x; v[i + 1] = x.y; v[i + 2] = x.z; v[i + 3] = x.w;
    }
}

// Instruction descriptor of the two contractions: M 128, N 16; `a_mn` for V (columns are the M side).
__host__ __device__ constexpr uint32_t dec_idesc(bool a_mn) { return instr_desc(kQRows, false) | (a_mn ? (1u << 15) : 0u); }

// NG: query heads per kv head, rounded up to 8 or 16 (what the softmax and fold threads hold).
template <int D, int NG>
__global__ void __launch_bounds__(kTcThreads, 1)
attention_decode_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                        const DecArgs args) {
    using DL = DecLayout<D>;
    extern __shared__ unsigned char raw_smem[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw_smem) + 1023) & ~uintptr_t(1023));
    unsigned char* q_smem = base;                                    // two query tiles
    unsigned char* k_ring = q_smem + 2 * DL::kQBytes;
    unsigned char* v_ring = k_ring + DL::kKRingBytes;
    unsigned char* ones_smem = k_ring + DL::kRingBytes;
    unsigned char* p_smem = ones_smem + DL::kOnesBytes;
    float* state = reinterpret_cast<float*>(p_smem + 2 * kPBytes);
    DecBarriers* bars = reinterpret_cast<DecBarriers*>(p_smem + 2 * kPBytes + DL::kStateBytes);
    DecList* list = reinterpret_cast<DecList*>(bars + 1);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int G = 1 << args.log_group;
    const int world = max(args.cache.map.world, 1);
    volatile int* abort_flag = &bars->abort_flag;

    pdl_launch_dependents();
    if (args.cluster > 1) cluster_arrive();       // the peers are told that this block runs, and may be written to
    if (warp == 0) {
        // One lane per barrier (the arrays of the struct lie one behind the other).
        constexpr int kSingles = 24;                              // the rings' barriers: one arrival each
        if (lane < kSingles) mbar_init(&bars->k_full[0] + lane, 1);
        if (lane < 2) {
            mbar_init(&bars->q_full[lane], 1);
            mbar_init(&bars->q_empty[lane], 1);
            mbar_init(&bars->p_full[lane], 4);
            mbar_init(&bars->p_free[lane], 1);
            mbar_init(&bars->o_full[lane], 1);
            mbar_init(&bars->o_free[lane], 4);
        }
        if (lane < kSBuf) {
            mbar_init(&bars->s_full[lane], 1);
            mbar_init(&bars->s_free[lane], 4);
        }
        if (lane == 0) {
            mbar_init(&bars->q_first, 12);
            bars->abort_flag = 0;
            bars->staged = 0;
            bars->n_work = 0;
            bars->cut = 0;
            mbar_init(&bars->merge_full[0], 1);
            mbar_init(&bars->merge_full[1], 1);
        }
        fence_barrier_init();
    }
    if (DL::kSumOnTensor) {
        for (int i = threadIdx.x; i < DL::kOnesBytes / 4; i += kTcThreads) reinterpret_cast<uint32_t*>(ones_smem)[i] = 0x3F803F80u;
        fence_proxy_async();
    }
    dec_list_build(args, list);
    __syncwarp();
    if (warp == 1) tmem_alloc(&bars->tmem_base, DL::kTmemCols);
    if (warp == 0 && lane == 0) {
        prefetch_tensormap(&tmap_k);
        prefetch_tensormap(&tmap_v);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    const DecIter start = dec_begin(list);
    if (args.cluster > 1) cluster_wait();
    pdl_wait();        // from here on the kernel reads what earlier kernels of the stream wrote

    // The first item's queries (and appended rows) are prepared by the twelve warps that have nothing to do yet
    // while its key tiles are on their way; later items' by warp 3, up to two items ahead.
    if (warp >= 4) {
        if (start.more()) dec_stage<D, 1>(args, list, start.w, q_smem, warp - 4, 12);
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->q_first);
    }
    auto queries_parity = [](uint32_t it) -> uint32_t { return ((it >> 1) - ((it & 1) ? 0u : 1u)) & 1; };   // it >= 1

    if (warp == 0) {
        // ===== producer: one thread feeds both rings, each with its own walk over the items, whichever has a free
        // stage. =====
        if (lane == 0) {
            struct Cursor {
                DecIter walk;
                uint32_t it;               // item index
                int j, part;               // tile of the item, stage of the tile
                uint32_t n;                // stage index of the stream
                int row0, plane;
            };
            Cursor ck, cv;
            auto enter_tile = [&](Cursor& c) {
                const DecItem& w = c.walk.w;
                const int seq = list->seq[w.b];
                c.plane = cache_plane(args.cache.map, seq, args.cache.kv_heads, w.kv_head);
                c.row0 = cache_row(args.cache.map, seq, (w.tile_first + c.j * world) * kTileKeys);
            };
            auto advance = [&](Cursor& c, int parts) {
                ++c.n;
                if (++c.part < parts) return;
                c.part = 0;
                if (++c.j == c.walk.w.n_tiles) {
                    c.j = 0;
                    ++c.it;
                    dec_next(list, c.walk);
                }
                if (c.walk.more()) enter_tile(c);
            };
            // The tile that the token's own rows go to is read after they are written.  (For later items a count:
            // this thread may be several uses of an item's barrier ahead.)
            auto rows_ready = [&](const Cursor& c) -> bool {
                if (args.k_new == nullptr || !c.walk.w.last || c.j != c.walk.w.n_tiles - 1) return true;
                if (c.it == 0) return mbar_test(&bars->q_first, 0);
                uint32_t staged;
                asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(staged) : "r"(smem_u32(&bars->staged)) : "memory");
                return staged > c.it;
            };
            ck.walk = start;
            ck.it = ck.n = 0;
            ck.j = ck.part = ck.row0 = ck.plane = 0;
            if (start.more()) enter_tile(ck);
            cv = ck;
            long long idle_since = 0;
            while (ck.walk.more() || cv.walk.more()) {
                bool moved = false;
                if (ck.walk.more()) {
                    const int slot = int(ck.n % DL::kKStages);
                    const uint32_t round = ck.n / DL::kKStages;
                    if ((round == 0 || mbar_test(&bars->k_empty[slot], (round - 1) & 1)) && (ck.part > 0 || rows_ready(ck))) {
                        mbar_expect_tx(&bars->k_full[slot], kBoxBytes);
                        tma_load_3d(k_ring + slot * kBoxBytes, &tmap_k, &bars->k_full[slot], ck.part * 64, ck.row0, ck.plane);
                        advance(ck, DL::kBlocks);
                        moved = true;
                    }
                }
                if (cv.walk.more()) {
                    const int slot = int(cv.n % DL::kVStages);
                    const uint32_t round = cv.n / DL::kVStages;
                    if ((round == 0 || mbar_test(&bars->v_empty[slot], (round - 1) & 1)) && (cv.part > 0 || rows_ready(cv))) {
                        mbar_expect_tx(&bars->v_full[slot], DL::kVStageBytes);
                        #pragma unroll
                        for (int b = 0; b < DL::kVBoxes; ++b) {
                            tma_load_3d(v_ring + slot * DL::kVStageBytes + b * kBoxBytes, &tmap_v, &bars->v_full[slot],
                                        (cv.part * DL::kVBoxes + b) * 64, cv.row0, cv.plane);
                        }
                        advance(cv, DL::kVTileStages);
                        moved = true;
                    }
                }
                if (moved) {
                    idle_since = 0;
                    continue;
                }
                if (*abort_flag != 0) break;
                const long long now = clock64();
                if (idle_since == 0) idle_since = now;
                if (static_cast<unsigned long long>(now - idle_since) > kWaitCycles) {
                    *abort_flag = 1;
                    report_status(args.status, 0x100 + 42);
                    break;
                }
                __nanosleep(20);
            }
        }
    } else if (warp == 1) {
        // ===== S^T = K Q^T.  The warp walks converged and one elected lane issues. =====
        constexpr uint32_t idesc = dec_idesc(false);
        const uint64_t q_desc0 = smem_desc(smem_u32(q_smem), 16);
        const uint64_t k_desc0 = smem_desc(smem_u32(k_ring), 16);
        uint32_t t = 0, it = 0, n = 0;
        bool ok = true;
        for (DecIter walk = start; ok && walk.more(); dec_next(list, walk), ++it) {
            const int n_tiles = walk.w.n_tiles;
            ok = it == 0 ? mbar_wait(&bars->q_first, 0, abort_flag, args.status, 43)
                         : mbar_wait(&bars->q_full[it & 1], queries_parity(it), abort_flag, args.status, 43);
            for (int j = 0; ok && j < n_tiles; ++j, ++t) {
                const int sb = int(t % kSBuf);
                if (t >= kSBuf && !mbar_wait(&bars->s_free[sb], (t / kSBuf - 1) & 1, abort_flag, args.status, 44)) { ok = false; break; }
                #pragma unroll 1
                for (int block = 0; block < DL::kBlocks; ++block, ++n) {
                    const int slot = int(n % DL::kKStages);
                    if (!mbar_wait(&bars->k_full[slot], (n / DL::kKStages) & 1, abort_flag, args.status, 45)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t k_desc = warp_uniform(k_desc0 + uint64_t((slot * kBoxBytes) >> 4));
                    const uint64_t q_desc = warp_uniform(q_desc0 + uint64_t(((it & 1) * DL::kQBytes + block * DL::kQBlock) >> 4));
                    const uint32_t d_tmem = warp_uniform(tmem + sb * kQRows);
                    if (elect_one()) {
                        #pragma unroll
                        for (int ks = 0; ks < 4; ++ks) {
                            mma_ss(d_tmem, k_desc + uint64_t((ks * 32) >> 4), q_desc + uint64_t((ks * 32) >> 4), idesc,
                                   ks != 0 ? 1u : uint32_t(block != 0));
                        }
                        tc_commit(&bars->k_empty[slot]);
                        if (block == DL::kBlocks - 1) {
                            tc_commit(&bars->s_full[sb]);
                            if (j + 1 == n_tiles) tc_commit(&bars->q_empty[it & 1]);
                        }
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp == 2) {
        // ===== O^T = V^T P^T, with the row sums as rows 64.. of it when head_dim is 64 (the second 64-column
        // block of V is then a block of ones). =====
        constexpr uint32_t idesc = dec_idesc(true);
        const uint64_t p_desc0 = smem_desc(smem_u32(p_smem), 16);
        const uint32_t ones_addr = smem_u32(ones_smem), ring_addr = smem_u32(v_ring);
        uint32_t t = 0, n = 0;
        bool ok = true;
        for (DecIter walk = start; ok && walk.more(); dec_next(list, walk)) {
            const int n_tiles = walk.w.n_tiles;
            for (int j = 0; ok && j < n_tiles; ++j, ++t) {
                const int ob = int(t & 1);
                if (!mbar_wait(&bars->p_full[ob], (t >> 1) & 1, abort_flag, args.status, 46)) { ok = false; break; }
                if (t >= 2 && !mbar_wait(&bars->o_free[ob], ((t >> 1) - 1) & 1, abort_flag, args.status, 47)) { ok = false; break; }
                #pragma unroll 1
                for (int part = 0; part < DL::kVTileStages; ++part, ++n) {
                    const int slot = int(n % DL::kVStages);
                    if (!mbar_wait(&bars->v_full[slot], (n / DL::kVStages) & 1, abort_flag, args.status, 48)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t v_addr = ring_addr + slot * DL::kVStageBytes;
                    const uint64_t v_desc = warp_uniform(smem_desc(v_addr, DL::kSumOnTensor ? ones_addr - v_addr : uint32_t(kBoxBytes)));
                    const uint64_t p_desc = warp_uniform(p_desc0 + uint64_t((ob * kPBytes) >> 4));
                    const uint32_t o_tmem = warp_uniform(tmem + DL::kOCol + ob * DL::kOCols + part * kQRows);
                    if (elect_one()) {
                        #pragma unroll
                        for (int ks = 0; ks < kTileKeys / 16; ++ks) {
                            mma_ss(o_tmem, v_desc + uint64_t((ks * 2048) >> 4), p_desc + uint64_t(((ks >> 2) * (kQRows * 128) + (ks & 3) * 32) >> 4),
                                   idesc, ks != 0 ? 1u : 0u);
                        }
                        tc_commit(&bars->v_empty[slot]);
                        if (part == DL::kVTileStages - 1) {
                            tc_commit(&bars->o_full[ob]);
                            tc_commit(&bars->p_free[ob]);
                        }
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp == 3) {
        // ===== queries of the items after the first =====
        DecIter walk = start;
        if (walk.more()) dec_next(list, walk);
        for (uint32_t it = 1; walk.more(); dec_next(list, walk), ++it) {
            if (it >= 2 && !mbar_wait(&bars->q_empty[it & 1], ((it >> 1) - 1) & 1, abort_flag, args.status, 49)) break;
            dec_stage<D, (D <= 256 ? 4 : 2)>(args, list, walk.w, q_smem + (it & 1) * DL::kQBytes, 0, 1);
            __syncwarp();
            if (lane == 0) {
                asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_u32(&bars->staged)), "r"(it + 1) : "memory");
                mbar_arrive(&bars->q_full[it & 1]);
            }
        }
    } else if (warp < 12) {
        // ===== softmax: thread = key; the two warpgroups take alternate tiles.  The warps of a group meet at named
        // barriers, so none of them may leave early: a wait that gives up is not acted on (the fold
        // warps do the same), the walk goes on over whatever is in the buffers, in bounds, and the
        // status word tells. =====
        const int par = (warp >> 2) - 1;
        const int quad = warp & 3;
        const int key = quad * 32 + lane;
        const uint32_t lane_base = uint32_t(quad * 32) << 16;
        const float neg_inf = __int_as_float(0xff800000);
        uint32_t t = 0;
        for (DecIter walk = start; walk.more(); dec_next(list, walk)) {
            const DecItem& w = walk.w;
            const int pos = list->pos[w.b];
            const int lo = args.window > 0 ? max(0, pos - args.window + 1) : 0;
            for (int j = 0; j < w.n_tiles; ++j, ++t) {
                if (int(t & 1) != par) continue;
                const int sb = int(t % kSBuf);
                mbar_wait(&bars->s_full[sb], (t / kSBuf) & 1, abort_flag, args.status, 50);
                tc_fence_after();
                uint32_t s[NG];
                tmem_ld_cols<NG>(tmem + lane_base + sb * kQRows, s);
                tc_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->s_free[sb]);
                const int at = (w.tile_first + j * world) * kTileKeys + key;
                const bool visible = at >= lo && at <= pos;
                float (&red)[4][kQRows] = bars->red[par][(t >> 1) & 1];
                float m[NG];
                #pragma unroll
                for (int q = 0; q < NG; ++q) {
                    if (!visible) s[q] = __float_as_uint(neg_inf);
                    m[q] = warp_max(__uint_as_float(s[q]));
                }
                if (lane == 0) {
                    #pragma unroll
                    for (int q = 0; q < NG; q += 4) *reinterpret_cast<float4*>(&red[quad][q]) = make_float4(m[q], m[q + 1], m[q + 2], m[q + 3]);
                }
                named_barrier(1 + par, 128);
                #pragma unroll
                for (int u = 0; u < 4; ++u) {
                    float other[NG];
                    load_row<NG>(red[u], other);
                    #pragma unroll
                    for (int q = 0; q < NG; ++q) m[q] = fmaxf(m[q], other[q]);
                }
                // P^T: row q holds the weights of the tile's 128 keys, in two 64-key blocks.
                if (t >= 2) mbar_wait(&bars->p_free[par], ((t >> 1) - 1) & 1, abort_flag, args.status, 51);
                unsigned char* p_key = p_smem + par * kPBytes + (key >> 6) * (kQRows * 128) + (key & 7) * 2;
                const int chunk = (key & 63) >> 3;
                float weight[NG];
                #pragma unroll
                for (int q = 0; q < NG; ++q) {
                    const float neg_mc = -__fmul_rn((m[q] == neg_inf) ? 0.0f : m[q], args.c);
                    const uint16_t bits = float_to_bf16_bits(tile_weight_raw(__uint_as_float(s[q]), neg_mc, args.c));
                    *reinterpret_cast<uint16_t*>(p_key + q * 128 + ((chunk ^ (q & 7)) << 4)) = bits;
                    weight[q] = bf16_bits_to_float(bits);
                }
                if (!DL::kSumOnTensor) {
                    // Sums of this warp's 32 weights per row by the butterfly tree (i with i + 16, then + 8, + 4, + 2,
                    // + 1).  The first steps halve the rows a lane carries: a lane keeps the rows its lane bit selects.
                    #pragma unroll
                    for (int step = 0; step < 3; ++step) {
                        const int half = NG >> (step + 1);
                        const bool upper = (lane & (16 >> step)) != 0;
                        #pragma unroll
                        for (int q = 0; q < half; ++q) {
                            const float give = upper ? weight[q] : weight[q + half];
                            const float keep = upper ? weight[q + half] : weight[q];
                            weight[q] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, 16 >> step));
                        }
                    }
                    constexpr int kLeft = NG >> 3;
                    #pragma unroll
                    for (int q = 0; q < kLeft; ++q) {
                        weight[q] = __fadd_rn(weight[q], __shfl_xor_sync(0xffffffffu, weight[q], 2));
                        weight[q] = __fadd_rn(weight[q], __shfl_xor_sync(0xffffffffu, weight[q], 1));
                    }
                    if ((lane & 3) == 0) {
                        const int row0 = ((lane >> 4) & 1) * (NG / 2) + ((lane >> 3) & 1) * (NG / 4) + ((lane >> 2) & 1) * (NG / 8);
                        #pragma unroll
                        for (int q = 0; q < kLeft; ++q) bars->lsum[t & 3][quad][row0 + q] = weight[q];
                    }
                }
                if (quad == 0 && lane == 0) {
                    #pragma unroll
                    for (int q = 0; q < NG; q += 4) {
                        *reinterpret_cast<float4*>(&bars->mm[t & 3][q]) = make_float4(__fmul_rn(m[q], args.c), __fmul_rn(m[q + 1], args.c),
                                                                                     __fmul_rn(m[q + 2], args.c), __fmul_rn(m[q + 3], args.c));
                    }
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->p_full[par]);
            }
        }
    } else {
        // ===== fold: thread = column of head_dim (and, at head_dim 64, threads 64.. the row sums).  A wait that
        // gives up is not acted on here: whatever is in the buffers is folded, in bounds, and the tickets
        // stay in step; the status word tells. =====
        const int tid = threadIdx.x & 127;
        const int quad = warp & 3;
        const uint32_t lane_base = uint32_t(quad * 32) << 16;
        const int q_self = lane & (NG - 1);                  // the row whose (M, L) chain this lane carries
        const bool holds_value = !DL::kSumOnTensor || tid < 64;
        float2* coef = bars->coef[quad];
        // (a, b) of this lane's row to all lanes of the warp.
        auto share = [&](float a, float b, float (&av)[NG], float (&bv)[NG]) {
            __syncwarp();
            if (lane < NG) coef[lane] = make_float2(a, b);
            __syncwarp();
            #pragma unroll
            for (int q = 0; q < NG; q += 2) {
                const float4 x = *reinterpret_cast<const float4*>(&coef[q]);
                av[q] = x.x; bv[q] = x.y; av[q + 1] = x.z; bv[q + 1] = x.w;
            }
        };
        uint32_t t = 0, it = 0;
        for (DecIter walk = start; walk.more(); dec_next(list, walk), ++it) {
            const DecItem w = walk.w;
            const int pos = list->pos[w.b];
            const int log_segment = args.cache.map.log_segment;
            const int first_segment = first_visible_tile(pos, args.window) >> log_segment;
            const size_t row0 = size_t(w.b) * args.q_heads + size_t(w.kv_head) * G;
            float A[DL::kMBlocks][NG];
            float M = kEmptyMax, L = 0.0f;
            float M2 = kEmptyMax, L2 = 0.0f;
            #pragma unroll
            for (int mb = 0; mb < DL::kMBlocks; ++mb) {
                #pragma unroll
                for (int q = 0; q < NG; ++q) A[mb][q] = 0.0f;
            }
            if (w.whole) {
                // The second fold's seed.
                if (args.count_sink) {
                    const uint16_t bits = args.sinks && q_self < G ? args.sinks[w.kv_head * G + q_self] : kNoSinkBits;
                    M2 = __fmul_rn(bf16_bits_to_float(bits), kLog2e);
                    L2 = 1.0f;
                }
                const float seed = holds_value ? 0.0f : L2;
                #pragma unroll
                for (int mb = 0; mb < DL::kMBlocks; ++mb) {
                    #pragma unroll
                    for (int q = 0; q < NG; ++q) state[(mb * NG + q) * 128 + tid] = seed;
                }
            }
            if (tid == 0 && !w.whole) bars->cut = 1;
            for (int j = 0; j < w.n_tiles; ++j, ++t) {
                const int ob = int(t & 1);
                const int tile = w.tile_first + j * world;
                mbar_wait(&bars->o_full[ob], (t >> 1) & 1, abort_flag, args.status, 52);
                tc_fence_after();
                const uint32_t o_tmem = tmem + lane_base + DL::kOCol + ob * DL::kOCols;
                uint32_t o[DL::kMBlocks][NG];
                #pragma unroll
                for (int mb = 0; mb < DL::kMBlocks; ++mb) tmem_ld_cols<NG>(o_tmem + mb * kQRows, o[mb]);
                const float mm = bars->mm[t & 3][q_self];
                float l = 0.0f;
                if (!DL::kSumOnTensor) {
                    const float g0 = bars->lsum[t & 3][0][q_self], g1 = bars->lsum[t & 3][1][q_self];
                    const float g2 = bars->lsum[t & 3][2][q_self], g3 = bars->lsum[t & 3][3][q_self];
                    l = D == 128 ? __fadd_rn(__fadd_rn(g0, g1), __fadd_rn(g2, g3)) : __fadd_rn(__fadd_rn(__fadd_rn(g0, g1), g2), g3);
                }
                if (args.cluster > 1) {
                    // The tile's partial to the blocks that fold its slices.
                    tc_wait_ld();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars->o_free[ob]);
                    const int rank = int(blockIdx.x) & (args.cluster - 1);
                    const int at = rank * ((list->span_tiles + args.cluster - 1) / args.cluster) + j;       // tile of the span
                    const int width = G * D / args.cluster, log_width = __ffs(width) - 1;
                    const int rows = width > D ? width / D : 1;
                    #pragma unroll
                    for (int q = 0; q < NG; ++q) {
                        if (q >= G) continue;
                        if (holds_value) {
                            #pragma unroll
                            for (int mb = 0; mb < DL::kMBlocks; ++mb) {
                                const int index = q * D + mb * 128 + tid;
                                const int to = index >> log_width;
                                cluster_store(cluster_addr(state + at * width + (index & (width - 1)), to), __uint_as_float(o[mb][q]));
                            }
                        } else if (tid == 64) {
                            for (int to = (q * D) >> log_width; to * width < (q + 1) * D; ++to) {
                                cluster_store(cluster_addr(&bars->push_l[at * rows + (rows > 1 ? q - to * rows : 0)], to), __uint_as_float(o[0][q]));
                            }
                        }
                    }
                    if (tid < G) {
                        for (int to = (tid * D) >> log_width; to * width < (tid + 1) * D; ++to) {
                            const int slot = at * rows + (rows > 1 ? tid - to * rows : 0);
                            cluster_store(cluster_addr(&bars->push_m[slot], to), mm);
                            if (!DL::kSumOnTensor) cluster_store(cluster_addr(&bars->push_l[slot], to), l);
                        }
                    }
                    continue;
                }
                float Mn, a, b, av[NG], bv[NG];
                fold_coefficients(M, mm, Mn, a, b);
                L = __fmaf_rn(L, a, __fmul_rn(l, b));
                M = Mn;
                share(a, b, av, bv);
                tc_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->o_free[ob]);
                #pragma unroll
                for (int mb = 0; mb < DL::kMBlocks; ++mb) {
                    #pragma unroll
                    for (int q = 0; q < NG; ++q) A[mb][q] = fold_value(A[mb][q], av[q], __uint_as_float(o[mb][q]), bv[q]);
                }
                const int segment = tile >> log_segment;
                if (j + 1 < w.n_tiles && ((tile + world) >> log_segment) == segment) continue;
                // The segment's last tile here: its partial is complete.
                if (w.whole) {
                    fold_coefficients(M2, M, Mn, a, b);
                    L2 = __fmaf_rn(L2, a, __fmul_rn(L, b));
                    M2 = Mn;
                    share(a, b, av, bv);
                    #pragma unroll
                    for (int mb = 0; mb < DL::kMBlocks; ++mb) {
                        #pragma unroll
                        for (int q = 0; q < NG; ++q) {
                            float& before = state[(mb * NG + q) * 128 + tid];
                            before = fold_value(before, av[q], A[mb][q], bv[q]);
                            A[mb][q] = 0.0f;
                        }
                    }
                } else {
                    const int slot = segment - first_segment;
                    #pragma unroll
                    for (int q = 0; q < NG; ++q) {
                        if (q >= G) continue;
                        const size_t at = (row0 + q) * args.slots + slot;
                        if (holds_value) {
                            #pragma unroll
                            for (int mb = 0; mb < DL::kMBlocks; ++mb) args.part_o[at * D + mb * 128 + tid] = A[mb][q];
                        } else if (tid == 64) {
                            args.part_ml[at * 2 + 1] = A[0][q];
                        }
                    }
                    if (tid < G) {
                        args.part_ml[((row0 + tid) * args.slots + slot) * 2] = M;
                        if (!DL::kSumOnTensor) args.part_ml[((row0 + tid) * args.slots + slot) * 2 + 1] = L;
                    }
                    #pragma unroll
                    for (int mb = 0; mb < DL::kMBlocks; ++mb) {
                        #pragma unroll
                        for (int q = 0; q < NG; ++q) A[mb][q] = 0.0f;
                    }
                }
                M = kEmptyMax;
                L = 0.0f;
            }
            if (w.whole) {
                // The row's denominators to all threads, then the epilogue.
                float* denom = bars->denom[it & 1];
                if (DL::kSumOnTensor) {
                    if (tid == 64) {
                        #pragma unroll
                        for (int q = 0; q < NG; ++q) denom[q] = state[q * 128 + tid];
                    }
                } else if (tid < NG) {
                    denom[tid] = L2;
                }
                named_barrier(3, 128);
                if (args.ep.write_partial && tid < G) {
                    float* dst = reinterpret_cast<float*>(args.ep.out) + (row0 + tid) * size_t(D + 2);
                    dst[D] = M2;
                    dst[D + 1] = denom[tid];
                }
                #pragma unroll 1                         // run once per item: short code, not fast code
                for (int q = 0; q < (holds_value ? G : 0); ++q) {
                    #pragma unroll 1
                    for (int mb = 0; mb < DL::kMBlocks; ++mb) {
                        const float value = state[(mb * NG + q) * 128 + tid];
                        const int col = mb * 128 + tid;
                        if (args.ep.write_partial) {
                            reinterpret_cast<float*>(args.ep.out)[(row0 + q) * size_t(D + 2) + col] = value;
                        } else {
                            const bool gated = args.ep.gate_layout != HC_GATE_NONE;
                            float gv = 0.0f;
                            if (args.ep.gate_layout == HC_GATE_INTERLEAVED) gv = load_io(args.ep.gate, (row0 + q) * size_t(2 * D) + D + col, args.ep.io_dtype);
                            else if (gated) gv = load_io(args.ep.gate, (row0 + q) * size_t(D) + col, args.ep.io_dtype);
                            store_io(args.ep.out, (row0 + q) * D + col, args.ep.io_dtype, finish_value(value, denom[q], gated, gv));
                        }
                    }
                }
            }
        }
    }

    // Teardown.  On the abort path the producer first lets its copies in flight land (bounded).
    if (warp == 0 && lane == 0 && *abort_flag != 0) {
        const long long begin = clock64();
        while (static_cast<unsigned long long>(clock64() - begin) < 200000000ull) { }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, DL::kTmemCols);
    if (args.cluster > 1) {
        cluster_arrive();
        cluster_wait();                // every partial of the span has been pushed
        dec_fold_slice<D>(args, list, state, bars->push_m, bars->push_l, reinterpret_cast<DecMerge*>(p_smem), &bars->n_last);
    } else if (bars->cut) {
        dec_close<D, NG>(args, list, reinterpret_cast<float*>(k_ring), reinterpret_cast<DecMerge*>(p_smem),
                         reinterpret_cast<int*>(state), &bars->n_work, bars->merge_full, abort_flag);
    }
    if (world > 1) dec_seed_rows<D, NG>(args);
}

template <int D, int NG>
constexpr int decode_smem() {
    return DecLayout<D>::kSmemBytes + int(sizeof(DecBarriers) + sizeof(DecList));
}

template <int D, int NG>
hc_status configure_decode_kernel(hc_context* ctx) {
    static_assert(decode_smem<D, NG>() <= 227 * 1024, "shared memory of one thread block");
    static bool configured[64] = {};                 // per device: the attributes are set once
    if (configured[ctx->device & 63]) return HC_OK;
    cudaError_t err = cudaFuncSetAttribute(attention_decode_kernel<D, NG>, cudaFuncAttributeMaxDynamicSharedMemorySize, decode_smem<D, NG>());
    if (err == cudaSuccess) err = cudaFuncSetAttribute(attention_decode_kernel<D, NG>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (err != cudaSuccess) return check_cuda(err, "attention_decode_kernel attributes");
    configured[ctx->device & 63] = true;
    return HC_OK;
}

template <int D, int NG>
hc_status launch_decode_kernel(hc_context* ctx, const DecArgs& args, int grid, const hc_layer_store& layer, cudaStream_t stream) {
    const hc_status st = configure_decode_kernel<D, NG>(ctx);
    if (st != HC_OK) return st;
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = kTcThreads;
    config.dynamicSmemBytes = decode_smem<D, NG>();
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[0].val.programmaticStreamSerializationAllowed = 1;
    attribute[1].id = cudaLaunchAttributeClusterDimension;
    attribute[1].val.clusterDim.x = unsigned(args.cluster);
    attribute[1].val.clusterDim.y = 1;
    attribute[1].val.clusterDim.z = 1;
    config.attrs = attribute;
    config.numAttrs = args.cluster > 1 ? 2 : 1;
    const cudaError_t launched = cudaLaunchKernelEx(&config, attention_decode_kernel<D, NG>, *static_cast<const CUtensorMap*>(layer.tmap_k),
                                                    *static_cast<const CUtensorMap*>(layer.tmap_v), args);
    ctx->launches += 1;
    return check_cuda(launched, "attention_decode_kernel launch");
}

template <int D>
hc_status launch_decode_dim(hc_context* ctx, const DecArgs& args, int grid, const hc_layer_store& layer, cudaStream_t stream) {
    return args.log_group <= 3 ? launch_decode_kernel<D, 8>(ctx, args, grid, layer, stream)
                               : launch_decode_kernel<D, 16>(ctx, args, grid, layer, stream);
}

}  // namespace

// Thread blocks that can be resident at once in clusters of 2, 4, 8 and 16 (the decode kernel takes an SM's whole
// shared memory whatever the head_dim): a cluster lives in one GPC, and what is left over of its SMs idles.
hc_status decode_cluster_slots(hc_context* ctx) {
    const hc_status st = configure_decode_kernel<64, 8>(ctx);
    if (st != HC_OK) return st;
    for (int i = 0; i < 4; ++i) {
        cudaLaunchConfig_t config = {};
        config.gridDim = 2u << i;
        config.blockDim = kTcThreads;
        config.dynamicSmemBytes = decode_smem<64, 8>();
        cudaLaunchAttribute attribute;
        attribute.id = cudaLaunchAttributeClusterDimension;
        attribute.val.clusterDim.x = 2u << i;
        attribute.val.clusterDim.y = 1;
        attribute.val.clusterDim.z = 1;
        config.attrs = &attribute;
        config.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, attention_decode_kernel<64, 8>, &config) != cudaSuccess) {
            cudaGetLastError();
            clusters = 0;
        }
        ctx->cluster_slots[i] = clusters * (2 << i);
    }
    return HC_OK;
}

// How a launch cuts its rows, by the time of its busiest thread block in units of one key tile (about 0.75 us of
// HBM at head_dim 64, proportional to it).  A launch's (or a wave of clusters') ramp is about 1.3 us, the merge
// 1.5 us inside a cluster, 3.5 us when it goes over global memory and tickets, whatever the head_dim.
TcDecodePlan tc_plan_decode(const hc_context* ctx, const AttnShape& shape, const RowMap& map, const BatchMeta& meta, int n_seq) {
    const int sms = std::max(ctx->sm_count, 1);
    TcDecodePlan plan{};
    int most_tiles = 1, most_segments = 1;
    long long tiles = 0, segments = 0;
    for (int b = 0; b < n_seq; ++b) {
        const int n = row_tiles(map, meta.pos[b], meta.pos[b], shape.window).count;
        most_tiles = std::max(most_tiles, n);
        tiles += std::max(n, 0);
        const int g = visible_groups(meta.pos[b], meta.pos[b], shape.window, map.log_segment);
        most_segments = std::max(most_segments, g);
        segments += n <= kDecUncut ? 1 : g;
    }
    const int d = shape.head_dim;
    const int segment_tiles = 1 << map.log_segment;
    const double us = 85.0 / d;                     // tiles per microsecond
    // A line over all SMs, or over as many thread blocks as there are segments.
    const long long all_segments = segments * shape.kv_heads;
    plan.cluster = 1;
    plan.blocks = int(std::max(1LL, std::min<long long>(sms, all_segments)));
    plan.run_segments = 1;
    plan.slots = most_segments;
    const bool rows_cut = (long long)n_seq * shape.kv_heads < plan.blocks || most_segments > 1;
    const double even = double(tiles) * shape.kv_heads / plan.blocks;
    double best = std::max(even + (all_segments > plan.blocks ? 0.5 * std::min(most_tiles, segment_tiles) : 0.0),
                           double(std::min(most_tiles, segment_tiles))) + (rows_cut ? 3.5 * us : 0.0) + 1.3 * us;
    if (most_tiles > 2) {
        for (int i = 0; i < 4; ++i) {
            const int cluster = 2 << i;
            const int resident = ctx->cluster_slots[i] / cluster;
            const int width = shape.group * d / cluster;
            if (resident < 1 || width < 4) continue;
            const int slice_rows = std::max(1, width / d);
            const int most_span = std::min(kPushBytes / 4 / width, kPushTiles / slice_rows);
            // A whole row per cluster, or spans of as many segments as fit, evened out.
            int run = most_segments;
            if (most_tiles > most_span) {
                const int fit = most_span / segment_tiles;
                if (fit < 1) continue;
                const int spans = (most_segments + fit - 1) / fit;
                if (spans > 0xffff) continue;                          // (DecArgs counts a row's spans in 16 bits)
                run = (most_segments + spans - 1) / spans;
            }
            long long clusters = 0;
            for (int b = 0; b < n_seq; ++b) {
                const int g = visible_groups(meta.pos[b], meta.pos[b], shape.window, map.log_segment);
                clusters += (g + run - 1) / run;
            }
            clusters *= shape.kv_heads;
            const int span_tiles = std::min(most_tiles, run * segment_tiles);
            const long long waves = (clusters + resident - 1) / resident;
            // The slice's last span folds width x segments values that others left, 512 at a time.
            const double merge = run == most_segments ? 1.5 : 3.5 + (width * most_segments >> 9) * 0.04;
            const double t = double(waves) * ((span_tiles + cluster - 1) / cluster + 1.3 * us) + merge * us;
            if (t < best) {
                best = t;
                plan.cluster = cluster;
                plan.blocks = int(std::min<long long>(clusters * cluster, 1 << 30));
                plan.run_segments = run;
            }
        }
    }
    const size_t q_rows = size_t(n_seq) * shape.q_heads;
    plan.part_o_floats = q_rows * plan.slots * d;
    plan.part_ml_floats = (q_rows * plan.slots * 2 + 3) & ~size_t(3);
    plan.tickets = size_t(n_seq) * shape.kv_heads * plan.cluster;
    return plan;
}

// A launch's arguments as far as they follow from its rows: where the rows lie on the line, or in clusters.
static long long dec_lay_out(DecArgs& args, const TcDecodePlan& plan, const BatchMeta& meta, int n_seq, const AttnShape& shape) {
    args.n_seq = n_seq;
    args.cluster = plan.cluster;
    args.slots = plan.slots;
    args.meta = meta;
    long long next = 0;
    for (int b = 0; b < n_seq; ++b) {
        args.start[b] = int(std::min(next, 0x7fffffffLL));
        if (plan.cluster == 1) {
            next += (long long)std::max(row_tiles(args.cache.map, meta.pos[b], meta.pos[b], shape.window).count, 0) * shape.kv_heads;
        } else {
            // Spans of one size, plan.run_segments each at most.
            const int segments = visible_groups(meta.pos[b], meta.pos[b], shape.window, args.cache.map.log_segment);
            const int want = (segments + plan.run_segments - 1) / plan.run_segments;
            const int run = (segments + want - 1) / want;
            args.seq_run[b] = static_cast<unsigned short>(run);
            args.seq_spans[b] = static_cast<unsigned short>((segments + run - 1) / run);
            next += (long long)args.seq_spans[b] * shape.kv_heads;
        }
    }
    for (int b = n_seq; b <= kMaxBatch; ++b) args.start[b] = int(std::min(next, 0x7fffffffLL));
    args.n_tiles = args.start[n_seq];
    return next;
}

// Whether the longest of the blocks' lists has room in shared memory.
static bool dec_lists_fit(const DecArgs& args, int blocks, const AttnShape& shape) {
    // (Most launches: no more rows than a list holds, or no more tiles to a stretch, where every row has one.)
    const long long rows = (long long)args.n_seq * shape.kv_heads;
    if (args.cluster > 1 || rows <= kDecItems) return true;
    if (args.cache.map.world <= 1 && args.n_tiles / blocks + 2 * (1 << args.cache.map.log_segment) + 2 <= kDecItems) return true;
    DecPlace from = dec_place(args, 0, blocks);
    for (int c = 0; c < blocks; ++c) {
        const DecPlace to = dec_place(args, c + 1, blocks);
        if (dec_items(from, to) > kDecItems) return false;
        from = to;
    }
    return true;
}

hc_status tc_decode(hc_context* ctx, const AttnShape& shape, const hc_layer_store& layer, const CacheView& cache,
                    const BatchMeta& meta, int n_seq, const DecodeSource& src, const Workspace& ws, const EpilogueArgs& ep,
                    cudaStream_t stream, int* served) {
    *served = 0;
    if (!layer.tmap_k || !layer.tmap_v) return fail(HC_UNSUPPORTED, "this layer has no tensor maps");
    if (n_seq <= 0) return HC_OK;
    DecArgs args{};
    args.q = src.q;
    args.k_new = src.k;
    args.v_new = src.v;
    args.src_dtype = src.dtype;
    args.q_head_stride = src.q_head_stride;
    args.norm_q = src.norm_q;
    args.norm_k = src.norm_k;
    args.norm_v = src.norm_v;
    args.q_weight = src.q_weight;
    args.k_weight = src.k_weight;
    args.eps = src.eps;
    args.cos = src.cos;
    args.sin = src.sin;
    args.table_positions = src.table_positions;
    args.cache = cache;
    args.q_heads = shape.q_heads;
    while ((1 << args.log_group) < shape.group) ++args.log_group;
    args.window = shape.window;
    args.c = shape.c;
    args.sinks = shape.sinks;
    args.count_sink = shape.count_sink;
    args.ep = ep;
    args.status = ctx->status_dev;
    args.part_o = ws.part_o;
    args.part_ml = ws.part_ml;
    args.tickets = ws.tickets;
    // As many of the rows as the workspace has partials for and the blocks' lists hold: all of them, but for many rows
    // of a cache that was made for few sequences, or for thousands of short ones.
    TcDecodePlan plan{};
    for (;; n_seq = (n_seq + 1) / 2) {
        plan = tc_plan_decode(ctx, shape, cache.map, meta, n_seq);
        const bool room = plan.part_o_floats <= ws.part_o_floats && plan.part_ml_floats <= ws.part_ml_floats && plan.tickets <= ws.n_tickets;
        if (!room && n_seq == 1) return fail(HC_KV_OVERFLOW, "decode: the split-attention workspace is too small for this call");
        if (!room) continue;
        const long long tiles = dec_lay_out(args, plan, meta, n_seq, shape);
        if (tiles <= 0x7fffffffLL && dec_lists_fit(args, plan.blocks, shape)) break;
        if (n_seq == 1) return fail(HC_UNSUPPORTED, "decode: too many key tiles or rows for one launch");
    }
    *served = n_seq;
    const int grid = plan.blocks;
    switch (shape.head_dim) {
        case 64: return launch_decode_dim<64>(ctx, args, grid, layer, stream);
        case 128: return launch_decode_dim<128>(ctx, args, grid, layer, stream);
        case 256: return launch_decode_dim<256>(ctx, args, grid, layer, stream);
        default: return launch_decode_dim<512>(ctx, args, grid, layer, stream);
    }
}

}  // namespace hc
