// attn_pair.cu — prefill attention for head_dim 256 and 512 (Gemma- and Qwen-shaped layers) on pairs of SMs.
//
// Same arithmetic as attn_tc.cu; what changes is how a wide row tile fits the machine.  Two CTAs form a cluster and
// share every MMA (cta_group::2): 256 query rows, 128 in each CTA, against key and value tiles of which each
// CTA loads half.  A 128-key tile then costs an SM 64 KB of loads and 2048 clocks of tensor pipe at head_dim
// 256, 32 bytes a clock; one CTA per 128 rows needed twice that, more than L2 gives 148 SMs at once,
// and with single 64 KB K and V stages each tile's load was exposed too (measured 0.21 of the bf16
// peak on an 8192-token prompt through six layers).
//
// Tensor memory holds two S buffers (2 x 128 columns) and ONE O buffer of 256 columns: all 512.  Head_dim 512 has
// twice as many columns of O, so there a work item is a row tile's 256-column half, and the logits are
// computed once for each half (a third more MMA work than a layout that kept 512 columns would need).
// Shared memory holds one Q tile (64 or 128 KB) and a ring of 16 KB stages through which K and V tiles
// pass in the order the MMAs take them: K0 K1 V0 K2 V1 .., across item boundaries.
//
//   warpgroup 0    warp 0 loads K and V, warp 1 of the leading CTA issues the MMAs, warp 2 works the items out and
//                  loads Q (all TMA)
//   warpgroups 1-2 softmax, thread = row; each group takes 64 of a tile's 128 columns.  With two S buffers the loop
//                  S -> softmax -> P V -> next S of the buffer sets the pace, so what counts is the softmax's
//                  latency (whole tiles in turn: 3100 clocks of it, 3250 a tile)
//   warpgroups 3-4 fold: a row of O is 256 floats, too many for one thread, so each folds a 128-column half
//
// The code of a tile is kept short: every launch fetches it cold, and straight-line code for 128 columns of softmax took
// 11000 clocks on its first pass.
// Registers per thread after setmaxnreg: 32 / 64 / 64 / 160 / 160.  Every mbarrier wait is bounded.

#include <algorithm>

#include "internal.hpp"
#include "tc_common.cuh"
#include "tc_ptx.cuh"

namespace hc {
namespace {

constexpr int kPairThreads = 640;                    // five warpgroups
constexpr int kPairRows = 2 * kRows;                 // query rows of a pair
constexpr int kPairO = 256;                          // O columns of an item
constexpr int kPairOCol = 2 * kTileKeys;             // their place in tensor memory
constexpr int kPairPCol = 32;                        // P of keys 32 .. 63 (of 64) begins in the columns of their S
constexpr int kPairStageBytes = 16 * 1024;           // K: 64 keys x 128 of head_dim; V: 128 keys x 64 columns; per CTA
constexpr int kPairBoxBytes = 64 * 128;              // a box of 64 rows x 64 elements
constexpr int kPairStoreBytes = 32 * 64;

template <int D>
struct PairLayout {
    static constexpr int kHalves = D / kPairO;               // items per row tile
    static constexpr int kQBytes = kRows * D * 2;
    static constexpr int kStages = D == 256 ? 8 : 4;
    static constexpr int kKChunks = D / 128;                 // stages of a K tile
    // The epilogue's stores go through 2 KB per fold warp: 32 rows x 64 bytes.
    static constexpr int kSmemBytes = 1024 + kQBytes + kStages * kPairStageBytes + 8 * kPairStoreBytes;
};

struct PairItem {
    int kv_head;
    int half;          // 256-column half of O (head_dim 512)
    int row0;          // first token of the row tile in the call
    int valid_tokens;
    int first_pos;
    int tile_first, n_tiles;
    int slot;          // ordinal of the item's segment among those the rows see (segment partials)
};
// BLOCKS: the launch has bidirectional blocks.
template <int D, bool BLOCKS>
__device__ __forceinline__ PairItem pair_item(const TcArgs& args, int index) {
    PairItem w;
    const int tokens_per_tile = kPairRows >> args.log_group;
    // Longest key ranges first: descending row tile; a row tile's halves, segments and kv heads adjacent.
    w.half = PairLayout<D>::kHalves > 1 ? index % PairLayout<D>::kHalves : 0;
    const int rest = index / PairLayout<D>::kHalves;
    const int rows = rest / args.slots;
    w.slot = rest - rows * args.slots;
    const int tile_index = rows / args.kv_heads;
    w.kv_head = rows - tile_index * args.kv_heads;
    const int mtile = args.mtiles - 1 - tile_index;
    w.row0 = mtile * tokens_per_tile;
    w.valid_tokens = min(tokens_per_tile, args.tokens - w.row0);
    w.first_pos = args.first_position + w.row0;
    int last_pos = w.first_pos + w.valid_tokens - 1;
    if (BLOCKS) last_pos = args.blocks.reach(last_pos) - 1;
    const TileRange tiles = args.finish ? row_tiles(args.map, w.first_pos, last_pos, args.window)
                                        : group_tiles(args.map, w.first_pos, last_pos, args.window, w.slot, args.map.log_segment);
    w.tile_first = tiles.first;
    w.n_tiles = tiles.count;
    return w;
}

// A pair's items, worked out by the warp that loads Q and read by every other role (as in attn_tc.cu: the divisions, in each
// role's own path, stood between two items).  The readers are never 16 items apart: what lies between the Q loader and
// the fold is one item's Q and fewer than ten tiles.
constexpr int kPairItems = 16;

struct PairBarriers {
    uint64_t q_full, q_empty;
    uint64_t full[9], empty[9];
    uint64_t s_full[2], p_full[2], m_full[4], o_full[2], o_free[2];
    uint64_t item_full[kPairItems];
    PairItem item[kPairItems];
    uint32_t tmem_base;
    int abort_flag;
    int more[2][4];                     // alternate items, per quadrant: whether there is one (softmax)
    float red[2][2][kRows];             // alternate tiles: the two halves' row maxima
    float mm[4][kRows];                 // scaled maxima, softmax -> fold (ring of 4 tiles, like m_full and l)
    float l[4][3][kRows];               // row sums: columns 0-63, 64-95, 96-127
    float m2[2][kRows], l2[2][kRows];   // the rows' second fold between segments, per half
};

// (x0 + y0, x1 + y1) of two bf16 pairs, as one packed addition.
__device__ __forceinline__ uint64_t unpack_pair(uint32_t w) { return uint64_t(w << 16) | (uint64_t(w & 0xffff0000u) << 32); }
__device__ __forceinline__ uint64_t add2(uint64_t x, uint64_t y) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    return r;
}

// MODE: what becomes of an item's rows, a template argument so that a launch carries the code (and the registers) of its
// own way only: bf16 rows (or, sequence-sharded, row partials); rows with a gate or in fp32; segment partials.
constexpr int kPairRowsOut = 0, kPairGatedOut = 1, kPairSegments = 2;
template <int D, int MODE, bool BLOCKS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
attention_pair_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                      const __grid_constant__ CUtensorMap tmap_q, const TcArgs args) {
    using PL = PairLayout<D>;
    extern __shared__ unsigned char raw_smem[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw_smem) + 1023) & ~uintptr_t(1023));
    unsigned char* q_smem = base;
    unsigned char* ring = q_smem + PL::kQBytes;
    unsigned char* store_smem = ring + PL::kStages * kPairStageBytes;
    PairBarriers* bars = reinterpret_cast<PairBarriers*>(store_smem + 8 * kPairStoreBytes);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int wg = warp >> 2;
    const int G = 1 << args.log_group;
    const int world = max(args.map.world, 1);
    const int rank = int(cluster_rank());
    const int token0 = rank * (kRows >> args.log_group);     // the first token of this CTA's half of a row tile
    volatile int* abort_flag = &bars->abort_flag;
    // Item `it` of this pair into w; false behind the last one, or on abort.
    auto read_item = [&](uint32_t it, PairItem& w) -> bool {
        if (!mbar_wait(&bars->item_full[it % kPairItems], (it / kPairItems) & 1, abort_flag, args.status, 13)) return false;
        w = bars->item[it % kPairItems];
        return w.n_tiles > 0;
    };
    // The walk tile by tile.
    struct Cursor {
        PairItem w;
        uint32_t it;
        int j;
        bool more;
    };
    auto begin = [&](Cursor& c) {
        c.it = 0;
        c.j = 0;
        c.more = read_item(0, c.w);
    };
    auto next = [&](Cursor& c) {
        if (++c.j == c.w.n_tiles) {
            c.j = 0;
            c.more = read_item(++c.it, c.w);
        }
    };

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        mbar_init(&bars->q_full, 1);
        mbar_init(&bars->q_empty, 1);
        for (int i = 0; i < PL::kStages; ++i) {
            mbar_init(&bars->full[i], 1);
            mbar_init(&bars->empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->s_full[i], 1);
            mbar_init(&bars->p_full[i], 16);                 // the softmax warps of both CTAs
            mbar_init(&bars->o_full[i], 1);
            mbar_init(&bars->o_free[i], 8);                  // a half's fold warps of both CTAs
        }
        for (int i = 0; i < 4; ++i) mbar_init(&bars->m_full[i], 8);      // those of this one
        for (int i = 0; i < kPairItems; ++i) mbar_init(&bars->item_full[i], 1);
        bars->abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc_pair(&bars->tmem_base, 512);
    if (warp == 0 && lane == 0) {
        prefetch_tensormap(&tmap_k);
        prefetch_tensormap(&tmap_v);
        prefetch_tensormap(&tmap_q);
    }
    tc_fence_before();
    __syncthreads();
    cluster_arrive();
    cluster_wait();        // the peer's barriers are there
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    pdl_wait();            // set-up done; from here on the kernel reads what earlier kernels wrote

    if (wg == 0) {
    reg_dealloc<32>();
    if (warp == 0) {
        // ===== producer: this CTA's halves of the tiles, in the order of the MMAs; the leader's barriers count
        // both CTAs' loads. =====
        if (lane == 0) {
            uint32_t n = 0;
            bool ok = true;
            auto load = [&](const CUtensorMap* map, int col0, int row, int plane, bool two_boxes) {
                const int slot = int(n % PL::kStages);
                const uint32_t round = n / PL::kStages;
                ++n;
                if (round > 0 && !mbar_wait(&bars->empty[slot], (round - 1) & 1, abort_flag, args.status, 1)) { ok = false; return; }
                if (rank == 0) mbar_expect_tx(&bars->full[slot], 2 * kPairStageBytes);
                const uint32_t full = cluster_addr(&bars->full[slot], 0);
                unsigned char* dst = ring + slot * kPairStageBytes;
                tma_load_3d_pair(dst, map, full, col0, row, plane);
                if (two_boxes) tma_load_3d_pair(dst + kPairBoxBytes, map, full, col0 + 64, row, plane);
            };
            // K one tile ahead of V.
            Cursor keys, values;
            begin(keys);
            begin(values);
            auto load_keys = [&]() {                         // this CTA's 64 keys of the tile
                const PairItem& w = keys.w;
                const int plane = cache_plane(args.map, args.seq, args.kv_heads, w.kv_head);
                const int row = cache_row(args.map, args.seq, (w.tile_first + keys.j * world) * kTileKeys) + rank * 64;
                for (int c = 0; ok && c < PL::kKChunks; ++c) load(&tmap_k, c * 128, row, plane, true);
                next(keys);
            };
            if (keys.more) load_keys();
            while (ok && values.more) {
                if (keys.more) load_keys();
                const PairItem& w = values.w;                // this CTA's 64 columns of each half of O
                const int plane = cache_plane(args.map, args.seq, args.kv_heads, w.kv_head);
                const int row = cache_row(args.map, args.seq, (w.tile_first + values.j * world) * kTileKeys);
                for (int h = 0; ok && h < 2; ++h) load(&tmap_v, w.half * kPairO + h * 128 + rank * 64, row, plane, false);
                next(values);
            }
        }
    } else if (warp == 1) {
        // ===== MMA issuer of the pair: S of the next tile (of the next item, at an item's end) is issued before P of
        // this one is awaited.  The whole warp walks the loop and waits, so control flow stays
        // warp-uniform; one elected lane issues the tcgen05 instructions. =====
        if (rank == 0) {
            constexpr uint32_t idesc_qk = instr_desc_pair(kTileKeys, false);
            constexpr uint32_t idesc_pv = instr_desc_pair(kPairO / 2, true);
            const uint64_t q_desc0 = smem_desc(smem_u32(q_smem), 16);
            const uint64_t k_desc0 = smem_desc(smem_u32(ring), 16);
            const uint64_t v_desc0 = smem_desc(smem_u32(ring), 16);
            uint32_t n = 0;
            Cursor ahead;
            begin(ahead);
            uint32_t ta = 0;                                 // tile of S
            auto issue_qk = [&]() -> bool {
                const uint32_t t = ta;
                const bool last = ahead.j + 1 == ahead.w.n_tiles;
                if (ahead.j == 0 && !mbar_wait(&bars->q_full, ahead.it & 1, abort_flag, args.status, 4)) return false;
                const uint32_t s_tmem = tmem + (t & 1) * kTileKeys;
                #pragma unroll 1
                for (int c = 0; c < PL::kKChunks; ++c, ++n) {
                    const int slot = int(n % PL::kStages);
                    if (!mbar_wait(&bars->full[slot], (n / PL::kStages) & 1, abort_flag, args.status, 3)) return false;
                    tc_fence_after();
                    const uint64_t q_desc = warp_uniform(q_desc0 + uint64_t((2 * c * (kRows * 128)) >> 4));
                    const uint64_t k_desc = warp_uniform(k_desc0 + uint64_t((slot * kPairStageBytes) >> 4));
                    const uint32_t d_tmem = warp_uniform(s_tmem);
                    if (elect_one()) {
                        #pragma unroll
                        for (int b = 0; b < 2; ++b) {
                            #pragma unroll
                            for (int ks = 0; ks < 4; ++ks) {
                                mma_ss_pair(d_tmem, q_desc + uint64_t((b * (kRows * 128) + ks * 32) >> 4),
                                            k_desc + uint64_t((b * kPairBoxBytes + ks * 32) >> 4), idesc_qk,
                                            (b | ks) != 0 ? 1u : uint32_t(c != 0));
                            }
                        }
                        tc_commit_pair(&bars->empty[slot]);
                        if (c == PL::kKChunks - 1) {
                            tc_commit_pair(&bars->s_full[t & 1]);
                            if (last) tc_commit_pair(&bars->q_empty);
                        }
                    }
                    __syncwarp();
                }
                ++ta;
                next(ahead);
                return true;
            };
            bool ok = !ahead.more || issue_qk();
            for (uint32_t t = 0; ok && t < ta; ++t) {
                if (ahead.more && !issue_qk()) break;
                if (!mbar_wait(&bars->p_full[t & 1], (t >> 1) & 1, abort_flag, args.status, 5)) break;
                const uint32_t p_tmem = tmem + (t & 1) * kTileKeys;
                // The two halves of O one after the other: one is folded while the other is computed.
                #pragma unroll 1
                for (int h = 0; h < 2; ++h, ++n) {
                    const int slot = int(n % PL::kStages);
                    if (t > 0 && !mbar_wait(&bars->o_free[h], (t - 1) & 1, abort_flag, args.status, 7)) { ok = false; break; }
                    if (!mbar_wait(&bars->full[slot], (n / PL::kStages) & 1, abort_flag, args.status, 6)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t v_desc = warp_uniform(v_desc0 + uint64_t((slot * kPairStageBytes) >> 4));
                    const uint32_t d_tmem = warp_uniform(tmem + kPairOCol + h * 128), a_tmem = warp_uniform(p_tmem);
                    if (elect_one()) {
                        #pragma unroll
                        for (int ks = 0; ks < kTileKeys / 16; ++ks) {
                            mma_ts_pair(d_tmem, a_tmem + (ks & 1) * 8 + ((ks >> 1) & 1) * kPairPCol + (ks >> 2) * 64, v_desc + uint64_t((ks * 2048) >> 4), idesc_pv,
                                        ks != 0 ? 1u : 0u);
                        }
                        tc_commit_pair(&bars->empty[slot]);
                        tc_commit_pair(&bars->o_full[h]);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp == 2) {
        // ===== Q loader: this CTA's 128 rows (128 / G tokens x G heads) of the prepared queries =====
        if (lane == 0) {
            uint32_t it = 0;
            const uint32_t q_full = cluster_addr(&bars->q_full, 0);
            for (Snake at(int(blockIdx.x) >> 1, int(gridDim.x) >> 1);; at.next()) {
                const bool more = at.item < args.n_items;
                PairItem& entry = bars->item[it % kPairItems];
                entry.n_tiles = 0;
                if (more) entry = pair_item<D, BLOCKS>(args, at.item);
                if (more && entry.n_tiles <= 0) continue;
                mbar_arrive(&bars->item_full[it % kPairItems]);
                if (!more) break;
                if (it > 0 && !mbar_wait(&bars->q_empty, (it - 1) & 1, abort_flag, args.status, 10)) break;
                if (rank == 0) mbar_expect_tx(&bars->q_full, 2 * PL::kQBytes);
                for (int b = 0; b < D / 64; ++b) {
                    tma_load_3d_pair(q_smem + b * (kRows * 128), &tmap_q, q_full, b * 64, entry.kv_head * G, entry.row0 + token0);
                }
                ++it;
            }
        }
    }
    } else if (wg <= 2) {
        // ===== softmax: thread = row, 64 columns.  The two warps of a row meet at a named barrier, so none leaves early: a
        // wait that gives up is not acted on, and the walk goes on over whatever is in the buffers, in bounds. =====
        reg_dealloc<64>();
        const int cols = wg - 1;                             // columns 64 cols .. 64 cols + 63
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        const int t_local = token0 + (row >> args.log_group);
        const uint32_t s_base = tmem + (uint32_t(quad * 32) << 16) + cols * 64;
        const uint32_t p_full[2] = {cluster_addr(&bars->p_full[0], 0), cluster_addr(&bars->p_full[1], 0)};
        const float neg_inf = __int_as_float(0xff800000);
        uint32_t t = 0;
        for (uint32_t it = 0;; ++it) {
            // Both warps of a row go by what the first of them reads.
            PairItem w;
            int* more = &bars->more[it & 1][quad];
            if (cols == 0) {
                const bool there = read_item(it, w);
                if (lane == 0) *more = there ? 1 : 0;
            }
            named_barrier(1 + quad, 64);
            if (*more == 0) break;
            if (cols != 0) w = bars->item[it % kPairItems];
            const bool valid = t_local < w.valid_tokens;
            const bool warp_has_rows = quad * 32 < ((w.valid_tokens - token0) << args.log_group);
            int pos = valid ? w.first_pos + t_local : -1;
            const int lo = args.window > 0 ? max(0, pos - args.window + 1) : 0;
            // From here on the last key the row sees: its own, or the end of its bidirectional block.
            if (BLOCKS && valid) {
                pos = max(pos, min(__ldg(args.blocks.ends + (w.first_pos - args.first_position) + t_local), args.blocks.reach(pos)) - 1);
            }
            for (int j = 0; j < w.n_tiles; ++j, ++t) {
                const int sb = int(t & 1);
                mbar_wait(&bars->s_full[sb], (t >> 1) & 1, abort_flag, args.status, 8);
                tc_fence_after();
                if (warp_has_rows) {
                    const uint32_t s_tmem = s_base + sb * kTileKeys;
                    const int key0 = (w.tile_first + j * world) * kTileKeys + cols * 64;
                    const int c_lo = lo - key0;
                    const int c_hi = pos - key0;
                    const bool full = c_lo <= 0 && c_hi >= 63;
                    // By bits of a word for each 32 columns (two comparisons a column were twice the code, fetched cold).
                    auto mask = [&](uint32_t (&s)[32], int base_col) {
                        const int from = min(max(c_lo - base_col, 0), 32), to = min(max(c_hi + 1 - base_col, 0), 32);
                        const uint32_t visible = uint32_t((1ull << to) - 1) & ~uint32_t((1ull << from) - 1);
                        #pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            if (((visible >> i) & 1u) == 0) s[i] = __float_as_uint(neg_inf);
                        }
                    };
                    auto maximum = [&](const uint32_t (&s)[32]) -> float {
                        float mx[4];
                        #pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            mx[u] = fmax3(__uint_as_float(s[u]), __uint_as_float(s[u + 4]), __uint_as_float(s[u + 8]));
                            mx[u] = fmax3(mx[u], __uint_as_float(s[u + 12]), __uint_as_float(s[u + 16]));
                            mx[u] = fmax3(mx[u], __uint_as_float(s[u + 20]), __uint_as_float(s[u + 24]));
                            mx[u] = fmaxf(mx[u], __uint_as_float(s[u + 28]));
                        }
                        return fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                    };
                    auto weights = [&](uint32_t (&s)[32], uint32_t (&packed)[16], float neg_mc) {
                        #pragma unroll
                        for (int i = 0; i < 16; ++i) fma2_inplace(s[2 * i], s[2 * i + 1], args.c, neg_mc);
                        #pragma unroll
                        for (int i = 0; i < 16; ++i) packed[i] = pack_bf16x2(ex2(__uint_as_float(s[2 * i])), ex2(__uint_as_float(s[2 * i + 1])));
                    };
                    // The row sum has a fixed shape: groups of 32 columns by the butterfly tree (i with i + 16, then + 8,
                    // + 4, + 2, + 1; two columns an addition), the four groups in order (the last two are added by the fold).
                    auto sum = [&](const uint32_t (&packed)[16]) -> float {
                        uint64_t a[2];
                        #pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            auto level = [&](int n) -> uint64_t { return add2(unpack_pair(packed[n]), unpack_pair(packed[n + 8])); };
                            a[i] = add2(add2(level(i), level(i + 4)), add2(level(i + 2), level(i + 6)));
                        }
                        a[0] = add2(a[0], a[1]);
                        return __fadd_rn(__uint_as_float(uint32_t(a[0])), __uint_as_float(uint32_t(a[0] >> 32)));
                    };
                    // A tile's time here is what one of prompts too short for the power limit takes, so as little as may be stands in a
                    // row: the second 32 columns stay in the registers between the passes, the first ones come back behind the sums
                    // of the others, and their own sum follows P (777 tokens behind 1291, 16 heads of 256: the launch 43.0 us, now 39.3).
                    uint32_t s[32], packed[16];
                    HC_TMEM_LD32(s_tmem, s);
                    tc_wait_ld();
                    if (!full) mask(s, 0);
                    float m = maximum(s);
                    HC_TMEM_LD32(s_tmem + 32, s);
                    tc_wait_ld();
                    if (!full) mask(s, 32);
                    m = fmaxf(m, maximum(s));
                    bars->red[sb][cols][row] = m;
                    named_barrier(1 + quad, 64);
                    m = fmaxf(m, bars->red[sb][cols ^ 1][row]);
                    const float neg_mc = -__fmul_rn((m == neg_inf) ? 0.0f : m, args.c);
                    weights(s, packed, neg_mc);
                    HC_TMEM_ST16(s_tmem + kPairPCol, packed);            // P in place of S columns already consumed
                    HC_TMEM_LD32(s_tmem, s);
                    const float sum1 = sum(packed);
                    tc_wait_ld();
                    if (!full) mask(s, 0);
                    weights(s, packed, neg_mc);
                    HC_TMEM_ST16(s_tmem, packed);
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster_relaxed(p_full[sb]);  // (P itself is ordered by the fences around tensor memory)
                    const float sum0 = sum(packed);
                    if (cols == 0) {
                        bars->mm[t & 3][row] = __fmul_rn(m, args.c);
                        bars->l[t & 3][0][row] = __fadd_rn(sum0, sum1);
                    } else {
                        bars->l[t & 3][1][row] = sum0;
                        bars->l[t & 3][2][row] = sum1;
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars->m_full[t & 3]);        // the maxima and sums, to this CTA's fold
                } else if (lane == 0) {
                    mbar_arrive_cluster_relaxed(p_full[sb]);
                    mbar_arrive(&bars->m_full[t & 3]);
                }
            }
        }
    } else {
        // ===== fold + epilogue: two threads per row, one per 128-column half of O =====
        reg_alloc<160>();
        const int half = wg - 3;
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        const int t_local = token0 + (row >> args.log_group);
        const int g = row & (G - 1);
        const uint32_t o_tmem = tmem + (uint32_t(quad * 32) << 16) + kPairOCol + half * 128;
        const uint32_t o_free = cluster_addr(&bars->o_free[half], 0);
        // This thread's values between segments: 32 groups of four, a row's group beside the next row's.
        float4* const state = reinterpret_cast<float4*>(args.row_state + size_t(blockIdx.x) * (kPairO * kRows)) + half * 32 * kRows + row;
        // (M, L) the second fold stands at: what the last segment end left, or the seed.
        auto second_fold_state = [&](bool state_holds, uint16_t sink, float& M2, float& L2) {
            if (state_holds) {
                M2 = bars->m2[half][row];
                L2 = bars->l2[half][row];
            } else if (args.count_sink) {
                M2 = __fmul_rn(bf16_bits_to_float(sink), kLog2e);
                L2 = 1.0f;
            } else {
                M2 = kEmptyMax;
                L2 = 0.0f;
            }
        };
        auto free_o = [&]() {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster_relaxed(o_free);      // nothing but tensor memory was read
        };
        // Four values of the row's state, zeros before its first segment is complete.
        auto state4 = [&](bool holds, int i) -> float4 { return holds ? state[(i >> 2) * kRows] : make_float4(0.0f, 0.0f, 0.0f, 0.0f); };
        // x[0..3] <- before * a + x * b
        auto join = [&](uint32_t* x, const float4& before, float a, float b) {
            float y[4] = {before.x, before.y, before.z, before.w};
            fold_value2(y[0], y[1], a, x[0], x[1], b);
            fold_value2(y[2], y[3], a, x[2], x[3], b);
            #pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = __float_as_uint(y[u]);
        };
        uint32_t t = 0, it = 0;
        bool ok = true;
        PairItem w;
        for (; ok && read_item(it, w); ++it) {
            // The head's sink, in time for the item's (or a segment's) end.
            uint16_t sink = kNoSinkBits;
            if (MODE != kPairSegments && args.count_sink && args.sinks != nullptr) sink = __ldg(args.sinks + w.kv_head * G + g);
            const bool valid = t_local < w.valid_tokens;
            const bool warp_has_rows = quad * 32 < ((w.valid_tokens - token0) << args.log_group);
            // The running segment's partial: a fold over its tiles from the empty state (both halves of
            // the row carry M and L, the same chain, the same bits).
            float M = kEmptyMax, L = 0.0f;
            float A[128];
            #pragma unroll
            for (int i = 0; i < 128; ++i) A[i] = 0.0f;
            bool state_holds = false;
            for (int j = 0; j < w.n_tiles; ++j, ++t) {
                const int tile = w.tile_first + j * world;
                const bool last = j + 1 == w.n_tiles;
                const bool ends = last || (MODE != kPairSegments && (tile >> args.map.log_segment) != ((tile + world) >> args.map.log_segment));
                // The coefficients while O is on its way.
                if (!mbar_wait(&bars->m_full[t & 3], (t >> 2) & 1, abort_flag, args.status, 11)) { ok = false; break; }
                float Mn, a, b;
                fold_coefficients(M, bars->mm[t & 3][row], Mn, a, b);
                L = __fmaf_rn(L, a, __fmul_rn(__fadd_rn(__fadd_rn(bars->l[t & 3][0][row], bars->l[t & 3][1][row]), bars->l[t & 3][2][row]), b));
                M = Mn;
                if (!mbar_wait(&bars->o_full[half], t & 1, abort_flag, args.status, 9)) { ok = false; break; }
                tc_fence_after();
                if (!warp_has_rows) {
                    if (lane == 0) mbar_arrive_cluster_relaxed(o_free);
                    continue;
                }
                #pragma unroll
                for (int chunk = 0; chunk < 8; ++chunk) {
                    uint32_t o[16];
                    HC_TMEM_LD16(o_tmem + chunk * 16, o);
                    tc_wait_ld();
                    if (chunk == 7 && !ends) free_o();
                    #pragma unroll
                    for (int i = 0; i < 16; i += 2) fold_value2(A[chunk * 16 + i], A[chunk * 16 + i + 1], a, o[i], o[i + 1], b);
                }
                if (!ends) continue;
                // A segment or the item ends.  Its values go back to tensor memory, in place of the O that was folded last, so
                // that what is done with them can be a rolled loop over the columns, short code with few registers (straight-line
                // over the 128 registers an item's end took 10800 clocks and spilled, now 6300; 777 gated fp32 tokens behind
                // 1291, 16 heads of 256: 76 us, now 58; 8192 tokens with a window of 1024: 160, now 147).
                #pragma unroll
                for (int i = 0; i < 128; i += 16) {
                    uint32_t v[16];
                    #pragma unroll
                    for (int u = 0; u < 16; ++u) v[u] = __float_as_uint(A[i + u]);
                    HC_TMEM_ST16(o_tmem + i, v);
                }
                tc_wait_st();
                if (last) {
                    ++t;
                    break;
                }
                // Another segment follows: this one joins the row's state, which is kept out of the registers ((M2, L2) in
                // shared memory, the values in global memory).
                float M2, L2;
                second_fold_state(state_holds, sink, M2, L2);
                fold_coefficients(M2, M, Mn, a, b);
                bars->m2[half][row] = Mn;
                bars->l2[half][row] = __fmaf_rn(L2, a, __fmul_rn(L, b));
                float4 before[8];
                #pragma unroll
                for (int u = 0; u < 8; ++u) before[u] = state4(state_holds, 4 * u);
                #pragma unroll 1
                for (int i = 0; i < 128; i += 32) {
                    uint32_t v[32];
                    HC_TMEM_LD32(o_tmem + i, v);
                    float4 after[8];
                    #pragma unroll
                    for (int u = 0; u < 8; ++u) after[u] = state4(state_holds && i < 96, i + 32 + 4 * u);
                    tc_wait_ld();
                    #pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        join(v + 4 * u, before[u], a, b);
                        state[(i / 4 + u) * kRows] = make_float4(__uint_as_float(v[4 * u]), __uint_as_float(v[4 * u + 1]), __uint_as_float(v[4 * u + 2]),
                                                                 __uint_as_float(v[4 * u + 3]));
                        before[u] = after[u];
                    }
                }
                free_o();
                #pragma unroll
                for (int i = 0; i < 128; ++i) A[i] = 0.0f;
                M = kEmptyMax;
                L = 0.0f;
                state_holds = true;
            }
            if (!ok) break;
            if (!warp_has_rows) continue;
            const size_t vec = size_t(w.row0 + t_local) * args.q_heads + w.kv_head * G + g;
            const int col0 = w.half * kPairO + half * 128;
            if constexpr (MODE == kPairSegments) {
                // The segment's partial goes to the workspace (a merge kernel runs the second fold).
                const size_t prow = vec * args.slots + w.slot;
                float* dst = args.part_o + prow * D + col0;
                #pragma unroll 1
                for (int i = 0; i < 128; i += 32) {
                    uint32_t v[32];
                    HC_TMEM_LD32(o_tmem + i, v);
                    tc_wait_ld();
                    #pragma unroll
                    for (int u = 0; valid && u < 32; u += 4) *reinterpret_cast<uint4*>(dst + i + u) = make_uint4(v[u], v[u + 1], v[u + 2], v[u + 3]);
                }
                free_o();
                if (valid && half == 0 && w.half == 0) *reinterpret_cast<float2*>(args.part_ml + prow * 2) = make_float2(M, L);
                continue;
            }
            // The row's last segment: the last step of the second fold, which started from the sink (or
            // from the empty state).
            float a, b;
            {
                float M2, L2, Mn;
                second_fold_state(state_holds, sink, M2, L2);
                fold_coefficients(M2, M, Mn, a, b);
                L = __fmaf_rn(L2, a, __fmul_rn(L, b));
                M = Mn;
            }
            const float inverse = __frcp_rn(L);
            if constexpr (MODE == kPairGatedOut) {
                // With a gate, or fp32 rows: thread = row, with registers to spare for the next 16 columns' gates.
                const bool gated = args.ep.gate_layout != HC_GATE_NONE, fp32 = args.ep.io_dtype == HC_F32;
                const int bytes = fp32 ? 4 : 2;
                const size_t gate_at = args.ep.gate_layout == HC_GATE_INTERLEAVED ? vec * size_t(2 * D) + D : vec * size_t(D);
                const unsigned char* gate = static_cast<const unsigned char*>(args.ep.gate) + (gate_at + col0) * bytes;
                unsigned char* out = static_cast<unsigned char*>(args.ep.out) + (vec * D + col0) * bytes;
                const bool aligned = (reinterpret_cast<uintptr_t>(gate) & 15) == 0;
                // Four columns of the thread's row as fp32.
                auto gate4 = [&](int i) -> float4 {
                    if (!gated || !valid) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (fp32) {
                        const float* from = reinterpret_cast<const float*>(gate) + i;
                        return aligned ? *reinterpret_cast<const float4*>(from) : make_float4(from[0], from[1], from[2], from[3]);
                    }
                    const uint16_t* from = reinterpret_cast<const uint16_t*>(gate) + i;
                    const uint2 two = aligned ? *reinterpret_cast<const uint2*>(from)
                                              : make_uint2(from[0] | uint32_t(from[1]) << 16, from[2] | uint32_t(from[3]) << 16);
                    return make_float4(__uint_as_float(two.x << 16), __uint_as_float(two.x & 0xffff0000u),
                                       __uint_as_float(two.y << 16), __uint_as_float(two.y & 0xffff0000u));
                };
                float4 now[4], next[4], before[4], after[4];
                #pragma unroll
                for (int u = 0; u < 4; ++u) {
                    now[u] = gate4(4 * u);
                    before[u] = state4(state_holds, 4 * u);
                }
                #pragma unroll 1
                for (int i = 0; i < 128; i += 16) {
                    uint32_t v[16];
                    HC_TMEM_LD16(o_tmem + i, v);
                    #pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        next[u] = gate4(i < 112 ? i + 16 + 4 * u : 0);
                        after[u] = state4(state_holds && i < 112, i + 16 + 4 * u);
                    }
                    tc_wait_ld();
                    if (i == 112) free_o();
                    #pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        join(v + 4 * u, before[u], a, b);
                        float r[4];
                        #pragma unroll
                        for (int x = 0; x < 4; ++x) r[x] = __fmul_rn(__uint_as_float(v[4 * u + x]), inverse);
                        if (gated) {
                            r[0] = __fmul_rn(r[0], sigmoid_gate(now[u].x));
                            r[1] = __fmul_rn(r[1], sigmoid_gate(now[u].y));
                            r[2] = __fmul_rn(r[2], sigmoid_gate(now[u].z));
                            r[3] = __fmul_rn(r[3], sigmoid_gate(now[u].w));
                        }
                        now[u] = next[u];
                        before[u] = after[u];
                        if (!valid) continue;
                        if (fp32) {
                            *reinterpret_cast<float4*>(out + (i + 4 * u) * 4) = make_float4(r[0], r[1], r[2], r[3]);
                        } else {
                            *reinterpret_cast<uint2*>(out + (i + 4 * u) * 2) = make_uint2(pack_bf16x2(r[0], r[1]), pack_bf16x2(r[2], r[3]));
                        }
                    }
                }
                continue;
            }
            // bf16 rows leave through shared memory, 64 bytes of each at a time, so that a store instruction touches 8
            // lines and not 32 (a thread storing its own row took 4300 clocks an item).  Lane l moves piece l % 4 of
            // rows l / 4, l / 4 + 8, ..  Row partials (a sequence-sharded cache) are stored by their own threads.
            unsigned char* stage = store_smem + (warp - 12) * kPairStoreBytes;
            auto piece = [&](int r, int c) -> uint4* { return reinterpret_cast<uint4*>(stage + r * 64 + ((c ^ ((r >> 1) & 3)) << 4)); };
            const int c = lane & 3;
            uint16_t* rows_out[4];
            #pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int r = quad * 32 + k * 8 + (lane >> 2);
                const int token = token0 + (r >> args.log_group);
                const size_t out_row = size_t(w.row0 + token) * args.q_heads + size_t(w.kv_head) * G + (r & (G - 1));
                rows_out[k] = token < w.valid_tokens ? reinterpret_cast<uint16_t*>(args.ep.out) + out_row * D + col0 + c * 8 : nullptr;
            }
            float* partial = reinterpret_cast<float*>(args.ep.out) + vec * size_t(D + 2) + col0;
            const bool partials = args.ep.write_partial != 0;
            float4 before[8];
            #pragma unroll
            for (int u = 0; u < 8; ++u) before[u] = state4(state_holds, 4 * u);
            #pragma unroll 1
            for (int i = 0; i < 128; i += 32) {
                uint32_t v[32];
                HC_TMEM_LD32(o_tmem + i, v);
                float4 after[8];
                #pragma unroll
                for (int u = 0; u < 8; ++u) after[u] = state4(state_holds && i < 96, i + 32 + 4 * u);
                tc_wait_ld();
                if (i == 96) free_o();
                #pragma unroll
                for (int u = 0; u < 8; ++u) {
                    join(v + 4 * u, before[u], a, b);
                    before[u] = after[u];
                }
                if (partials) {
                    #pragma unroll
                    for (int u = 0; valid && u < 32; u += 2) *reinterpret_cast<uint2*>(partial + i + u) = make_uint2(v[u], v[u + 1]);
                    continue;
                }
                #pragma unroll
                for (int u = 0; u < 4; ++u) {
                    uint32_t p[4];
                    #pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        p[x] = pack_bf16x2(__fmul_rn(__uint_as_float(v[8 * u + 2 * x]), inverse), __fmul_rn(__uint_as_float(v[8 * u + 2 * x + 1]), inverse));
                    }
                    *piece(lane, u) = make_uint4(p[0], p[1], p[2], p[3]);
                }
                __syncwarp();
                #pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (rows_out[k] != nullptr) *reinterpret_cast<uint4*>(rows_out[k] + i) = *piece(k * 8 + (lane >> 2), c);
                }
                __syncwarp();
            }
            if (partials && valid && half == 0 && w.half == 0) *reinterpret_cast<float2*>(partial + D) = make_float2(M, L);
        }
    }

    // Teardown.  On the abort path the producer first lets its copies in flight land (bounded).
    if (warp == 0 && lane == 0 && *abort_flag != 0) {
        const long long start = clock64();
        while (static_cast<unsigned long long>(clock64() - start) < 200000000ull) { }
    }
    tc_fence_before();
    __syncthreads();
    cluster_arrive();
    cluster_wait();        // neither CTA leaves while the other's MMAs or arrivals may still name it
    if (warp == 1) tmem_dealloc_pair(tmem, 512);
}

template <int D, int MODE, bool BLOCKS>
hc_status launch_pair_kernel(hc_context* ctx, const hc_layer_store& layer, const CUtensorMap& tmap_q, const TcArgs& args, cudaStream_t stream) {
    constexpr int smem = PairLayout<D>::kSmemBytes + int(sizeof(PairBarriers));
    static_assert(smem <= 227 * 1024, "shared memory of one CTA");
    static bool configured[64] = {};
    if (!configured[ctx->device & 63]) {
        const cudaError_t err = cudaFuncSetAttribute(attention_pair_kernel<D, MODE, BLOCKS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (err != cudaSuccess) return check_cuda(err, "attention_pair_kernel shared memory");
        configured[ctx->device & 63] = true;
    }
    const int grid = 2 * std::max(1, std::min(args.n_items, std::max(ctx->sm_count / 2, 1)));
    const cudaError_t launched = launch_pdl(attention_pair_kernel<D, MODE, BLOCKS>, grid, kPairThreads, size_t(smem), stream,
                                            *static_cast<const CUtensorMap*>(layer.tmap_k64),
                                            *static_cast<const CUtensorMap*>(layer.tmap_v), tmap_q, args);
    ctx->launches += 1;
    return check_cuda(launched, "attention_pair_kernel launch");
}

template <bool BLOCKS>
hc_status launch_pair(hc_context* ctx, const hc_layer_store& layer, const CUtensorMap& tmap_q, const TcArgs& args, int head_dim, bool gated,
                      cudaStream_t stream) {
    const bool wide = head_dim == 512;
    auto launch = !args.finish ? (wide ? launch_pair_kernel<512, kPairSegments, BLOCKS> : launch_pair_kernel<256, kPairSegments, BLOCKS>)
                : gated        ? (wide ? launch_pair_kernel<512, kPairGatedOut, BLOCKS> : launch_pair_kernel<256, kPairGatedOut, BLOCKS>)
                               : (wide ? launch_pair_kernel<512, kPairRowsOut, BLOCKS> : launch_pair_kernel<256, kPairRowsOut, BLOCKS>);
    return launch(ctx, layer, tmap_q, args, stream);
}

}  // namespace

int pair_items_per_row_tile(int head_dim) { return head_dim / kPairO; }

hc_status launch_attention_pair(hc_context* ctx, const hc_layer_store& layer, const void* args_ptr, int head_dim, cudaStream_t stream) {
    const TcArgs& args = *static_cast<const TcArgs*>(args_ptr);
    // A CTA's Q tile is a box of 64 columns x G heads x 128 / G tokens; rows beyond the last token are zeros.
    CUtensorMap tmap_q;
    const int group = 1 << args.log_group;
    const hc_status st = tc_encode_3d(&tmap_q, args.q, uint64_t(head_dim), uint64_t(args.q_heads), uint64_t(args.tokens), uint32_t(group),
                                      uint32_t(kRows / group));
    if (st != HC_OK) return st;
    const bool gated = !args.ep.write_partial && (args.ep.gate_layout != HC_GATE_NONE || args.ep.io_dtype == HC_F32);
    return args.blocks.ends ? launch_pair<true>(ctx, layer, tmap_q, args, head_dim, gated, stream)
                            : launch_pair<false>(ctx, layer, tmap_q, args, head_dim, gated, stream);
}

}  // namespace hc
