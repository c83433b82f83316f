// tc_common.cuh — what the tcgen05 attention kernels share: the kernel arguments, the work-item list a
// persistent CTA walks, and small helpers.
#pragma once

#include "internal.hpp"
#include "tc_ptx.cuh"

namespace hc {
namespace {

struct TcArgs {
    const uint16_t* q;        // bf16 [rows][q_heads][d], prepared
    int tokens;
    int first_position;
    int q_heads;
    int kv_heads;
    int log_group;
    int window;
    float c;
    const uint16_t* sinks;
    int count_sink;
    int seq;
    RowMap map;
    EpilogueArgs ep;
    int* status;
    int n_items;              // work items in the list
    int mtiles;               // row tiles per kv head
    // How a launch cuts its rows' keys into items (the bits are the same whichever the host picks):
    //   finish != 0       an item is all the key tiles of one row tile and kv head.  The kernel runs both folds
    //                     and the epilogue, keeping the second fold's values between segments in row_state
    //                     (head_dim 64: in shared memory).
    //   otherwise         an item is one segment of those and leaves its partial in the workspace, `slots`
    //                     per row at most (slot = ordinal of the segment); a merge kernel finishes the rows.
    int slots;
    int finish;
    float* part_o;            // fp32 [rows][slots][d]
    float* part_ml;           // fp32 [rows][slots][2]
    float* row_state;         // fp32 [thread blocks][d][128], finish only
    // Multipliers for the divisions of tc_item (see fast_div); 0 = divide the ordinary way.
    uint32_t magic_slots, magic_kv_heads;
    // With bidirectional blocks an item reaches to the end of its last token's chunk; rows that see nothing of a tile fold
    // its empty partial, a no-op.
    Blocks blocks;
};

// n / d for the small operands of the item list: with magic = ceil(2^32 / d) the high word of
// n * magic is the quotient whenever n * d < 2^32, which the host checks before it sets a magic.
__host__ __device__ inline uint32_t division_magic(uint32_t d, uint32_t n_max) {
    if (d <= 1 || uint64_t(n_max) * d >= (1ull << 32)) return 0;
    return uint32_t(((1ull << 32) + d - 1) / d);
}
__device__ __forceinline__ int fast_div(int n, int d, uint32_t magic) {
    return magic != 0 ? int(__umulhi(uint32_t(n), magic)) : n / d;
}


struct TcItem {
    int kv_head;
    int row0;          // first row of q / out (token index of the chunk)
    int valid_tokens;  // query tokens in this row tile
    int first_pos;     // position of the first query token
    int tile_first;    // absolute index of the first key tile
    int n_tiles;       // key tiles to visit (stride `world` apart); <= 0: nothing to do
    int first_segment; // absolute index of the first segment the rows see (segment partials go to
                       // slot = segment - first_segment)
};

__device__ __forceinline__ TcItem tc_item(const TcArgs& args, int index) {
    TcItem w;
    const int tokens_per_tile = kRows >> args.log_group;
    // Longest key ranges first: descending row tile; a row tile's segments and kv heads adjacent.
    const int rest = fast_div(index, args.slots, args.magic_slots);
    const int slot = index - rest * args.slots;
    const int tile_index = fast_div(rest, args.kv_heads, args.magic_kv_heads);
    w.kv_head = rest - tile_index * args.kv_heads;
    const int mtile = args.mtiles - 1 - tile_index;
    w.row0 = mtile * tokens_per_tile;
    w.valid_tokens = min(tokens_per_tile, args.tokens - w.row0);
    w.first_pos = args.first_position + w.row0;
    int last_pos = w.first_pos + w.valid_tokens - 1;
    if (args.blocks.ends != nullptr) last_pos = args.blocks.reach(last_pos) - 1;
    const TileRange tiles = args.finish ? row_tiles(args.map, w.first_pos, last_pos, args.window)
                                        : group_tiles(args.map, w.first_pos, last_pos, args.window, slot, args.map.log_segment);
    w.tile_first = tiles.first;
    w.n_tiles = tiles.count;
    w.first_segment = first_visible_tile(w.first_pos, args.window) >> args.map.log_segment;
    return w;
}

// A worker's way through a list of items, longest first: forwards through the workers in one round, backwards in the
// next, so that the first of them does not get the longest item of every round.
struct Snake {
    int item, step, twice;
    __device__ __forceinline__ Snake(int worker, int workers) : item(worker), step(2 * (workers - worker) - 1), twice(2 * workers) {}
    __device__ __forceinline__ void next() {
        item += step;
        step = twice - step;
    }
};

// The walk over a CTA's items: each item is decoded once per role (its decoding costs a few integer
// divisions, which a role pays on its critical path at every item boundary).
struct TcItemIter {
    Snake at;
    int item;          // index in the work list, or n_items at the end
    TcItem w;
};
__device__ __forceinline__ void items_seek(const TcArgs& args, TcItemIter& it) {
    for (; it.at.item < args.n_items; it.at.next()) {
        it.item = it.at.item;
        it.w = tc_item(args, it.item);
        if (it.w.n_tiles > 0) return;
    }
    it.item = args.n_items;
}
__device__ __forceinline__ TcItemIter items_begin(const TcArgs& args) {
    TcItemIter it{Snake(int(blockIdx.x), int(gridDim.x)), 0, TcItem{}};
    items_seek(args, it);
    return it;
}
__device__ __forceinline__ void items_next(const TcArgs& args, TcItemIter& it) {
    it.at.next();
    items_seek(args, it);
}

// bf16x2 of two softmax weights: `lo` in the low half (the earlier key), `hi` in the high half.
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    uint32_t packed;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(packed) : "f"(hi), "f"(lo));
    return packed;
}


// (x0, x1) <- (x0 * c + d, x1 * c + d), each rounded once, as one packed instruction.
__device__ __forceinline__ void fma2_inplace(uint32_t& x0, uint32_t& x1, float c, float d) {
    uint64_t x = uint64_t(x0) | (uint64_t(x1) << 32);
    const uint64_t cc = uint64_t(__float_as_uint(c)) | (uint64_t(__float_as_uint(c)) << 32);
    const uint64_t dd = uint64_t(__float_as_uint(d)) | (uint64_t(__float_as_uint(d)) << 32);
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(x) : "l"(x), "l"(cc), "l"(dd));
    x0 = uint32_t(x);
    x1 = uint32_t(x >> 32);
}

// Eight words to a 16-byte boundary, in one store where it is a 32-byte one (all of a launch's rows lie alike).
__device__ __forceinline__ void store_32bytes(void* dst, const uint32_t (&v)[8]) {
    if ((reinterpret_cast<uintptr_t>(dst) & 31) == 0) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                     ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
    } else {
        *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
        *(reinterpret_cast<uint4*>(dst) + 1) = make_uint4(v[4], v[5], v[6], v[7]);
    }
}

// (x0, x1) <- (x0 * c, x1 * c).
__device__ __forceinline__ void mul2_inplace(float& x0, float& x1, float c) {
    uint64_t x = uint64_t(__float_as_uint(x0)) | (uint64_t(__float_as_uint(x1)) << 32);
    const uint64_t cc = uint64_t(__float_as_uint(c)) | (uint64_t(__float_as_uint(c)) << 32);
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(x) : "l"(cc));
    x0 = __uint_as_float(uint32_t(x));
    x1 = __uint_as_float(uint32_t(x >> 32));
}

// Two steps of the fold at once: (A0, A1) <- (A0 * a + (o0 * b), A1 * a + (o1 * b)), every product
// and sum rounded exactly as fold_value does, in two packed instructions instead of four.
__device__ __forceinline__ void fold_value2(float& A0, float& A1, float a, uint32_t o0, uint32_t o1, float b) {
    uint64_t acc = uint64_t(__float_as_uint(A0)) | (uint64_t(__float_as_uint(A1)) << 32);
    const uint64_t o = uint64_t(o0) | (uint64_t(o1) << 32);
    const uint64_t aa = uint64_t(__float_as_uint(a)) | (uint64_t(__float_as_uint(a)) << 32);
    const uint64_t bb = uint64_t(__float_as_uint(b)) | (uint64_t(__float_as_uint(b)) << 32);
    uint64_t ob;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(ob) : "l"(o), "l"(bb));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(acc) : "l"(acc), "l"(aa), "l"(ob));
    A0 = __uint_as_float(uint32_t(acc));
    A1 = __uint_as_float(uint32_t(acc >> 32));
}

}  // namespace
}  // namespace hc
