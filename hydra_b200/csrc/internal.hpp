// internal.hpp — host-side objects behind the opaque handles of hydra_cuda.h, and the launchers
// each .cu file exports to api.cu.  Nothing here is visible outside the shared library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <memory>
#include <string>
#include <vector>

#include "../../include/hydra_cuda.h"
#include "common.cuh"

namespace hc {

// At most this many sequences share one decode launch; larger batches are cut into launches.
constexpr int kMaxBatch = 64;

struct BatchMeta {
    int seq[kMaxBatch];
    int pos[kMaxBatch];
};

// One head's rows of one layer, as the kernels address them.
struct CacheView {
    uint16_t* k;       // bf16 [max_seqs][kv_heads][capacity][head_dim]
    uint16_t* v;
    int capacity;      // rows per (sequence, head)
    int kv_heads;
    RowMap map;
};

struct AttnShape {
    int q_heads;
    int kv_heads;
    int head_dim;
    int group;          // q_heads / kv_heads
    int window;         // 0 = full
    float c;            // sm_scale * log2(e)
    const uint16_t* sinks;  // bf16 [q_heads] or null
    int count_sink;     // 0 on ranks > 0 of a sequence-sharded cache
};

// Launch with programmatic stream serialisation allowed (see pdl_wait in common.cuh).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              Args&&... args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, static_cast<KArgs>(args)...);
}

// What the prologue does to one of q, k, v.
struct PrepJob {
    const void* src;
    int src_dtype;
    int heads;
    long long token_stride;  // elements between tokens in src
    int head_stride;         // elements between heads in src (2 * d for an interleaved gate)
    int norm;                // 0 none, 1 weighted, 2 weightless
    const uint16_t* weight;
    int rope;                // 0 / 1
    int kind;                // 0: dense bf16 [tokens][heads][d]; 1: K rows; 2: V rows; 3: in place
    void* dst;
};
struct PrepArgs {
    PrepJob job[3];
    int n_jobs;
    int head_dim;
    float eps;
    const float* cos;        // fp32 [table_positions][head_dim / 2]
    const float* sin;
    int table_positions;
    int tokens;
    int first_position;      // position of token 0 when batched == 0
    int batched;             // 1: token t is sequence meta.seq[t] at position meta.pos[t]
    int seq;                 // sequence when batched == 0
    CacheView cache;         // for kinds 1 and 2
    // Rows at positions from also_from on go here too (a prompt whose keys attend outside its ring); 0 rows: nowhere.
    CacheView also;
    int also_from;
    int also_seq;
    BatchMeta meta;
};

struct EpilogueArgs {
    void* out;               // [rows][q_heads][d] io dtype, or fp32 partial [rows][q_heads][d + 2]
    int io_dtype;
    int write_partial;       // 1: write (A, M, L) instead of the finished value
    int gate_layout;
    const void* gate;        // HC_GATE_SEPARATE: [rows][q_heads][d]; INTERLEAVED: q_proj output
};

struct Workspace {
    uint16_t* qprep = nullptr;   // bf16 [qprep_capacity][q_heads][d]
    int qprep_capacity = 0;
    int qprep_tokens = 0;        // what the host-buffer calls take at once: max(prefill_chunk, max_seqs)
    float* part_o = nullptr;     // fp32 [rows][slots][d]: segment partials, rows and slots those of the call
    float* part_ml = nullptr;    // fp32 [rows][slots][2]
    size_t part_o_floats = 0;    // capacities
    size_t part_ml_floats = 0;
    // Counters by which the last thread block of a decode row (or of a row's segment) to finish knows that it
    // is the last; zero between launches.
    unsigned* tickets = nullptr;
    size_t n_tickets = 0;
};

// What the tcgen05 decode kernel prepares itself: the queries as the caller has them and, when k is set, the
// tokens' own key and value rows on their way into the cache.
struct DecodeSource {
    const void* q;
    const void* k;
    const void* v;
    int dtype;               // hc_dtype of the three
    int q_head_stride;       // elements between heads of q (2 d for an interleaved gate)
    int norm_q, norm_k, norm_v;
    const uint16_t* q_weight;
    const uint16_t* k_weight;
    float eps;
    const float* cos;        // null: no rotation
    const float* sin;
    int table_positions;
};

}  // namespace hc

struct hc_context {
    int device = 0;
    int sm_count = 0;
    uint64_t launches = 0;
    int* status_host = nullptr;   // one word the kernels may set on a bounded-wait timeout, in pinned host memory:
    int* status_dev = nullptr;    // a check is a synchronisation and a read; its address on the device
    int cluster_slots[4] = {};    // thread blocks resident at once in clusters of 2, 4, 8, 16 (see attn_decode.cu)
    float* static_scratch = nullptr;   // device address of the fixed scratch of hc_attention_decode_static
};

struct hc_rope_table {
    int device = 0;
    float* cos = nullptr;
    float* sin = nullptr;
    int positions = 0;
    int pairs = 0;
};

struct hc_layer_store {
    hc_layer_desc desc{};
    uint16_t* k = nullptr;
    uint16_t* v = nullptr;
    int ring = 0;                 // rows of the ring as stored (0: linear); positions map to pos % ring
    int ring_margin = 0;          // the reference's ring is window + ring_margin rows: what a chunk may
                                  // append at once and how far a rewind may reach
    int capacity = 0;
    int log_segment = 0;          // key tiles per segment, as a power of two (see common.cuh)
    int log_segment_general = 0;  // the grouping that hc_attention_decode_static's limit is stated in
    bool keeps_history = false;
    void* tmap_k = nullptr;       // tensor maps of the tcgen05 path (host copies), or null
    void* tmap_v = nullptr;
    void* tmap_k64 = nullptr;     // keys in boxes of 64 rows: what a CTA of a pair loads (head_dim 256, 512)
    // A ring holds too little of a prompt beside its window, so a longer one attends in the workspace: a ring of one sequence
    // with room for the window and a whole call's tokens, used by one call at a time like the rest of the workspace.  Null where
    // no call is longer than that, or the store did not fit: the prompts take the ring in pieces.
    std::unique_ptr<hc_layer_store> prompt;
};

struct hc_kv_cache {
    hc_context* ctx = nullptr;
    std::vector<hc_layer_store> layers;
    int context_length = 0;
    int prefill_chunk = 0;
    int max_seqs = 0;
    hc_shard_desc shard{HC_SHARD_NONE, 0, 1};
    std::vector<int> lengths;
    // Paged storage (hc_kv_cache_create_paged): the linear layers are pools of total_pages pages of 128
    // rows shared by all sequences; one page table for all layers, [max_seqs][pages_per_seq], -1 =
    // not assigned (the device copy holds 0 there: a valid page that no visible key maps to).
    int total_pages = 0;
    int pages_per_seq = 0;
    int* pages_dev = nullptr;
    int* pages_host = nullptr;    // pinned mirror, the source of the asynchronous updates
    std::vector<int> free_pages;
    hc::Workspace ws;
    // hc_layer_step_host / hc_prefill_host: two device staging slots, a stream for the copies in and
    // one for the copies out, and the events that order them against the caller's stream.
    void* workspace_dev = nullptr;   // ws and the staging slots
    void* stage_dev = nullptr;
    size_t stage_bytes = 0;       // of one slot
    cudaStream_t copy_in = nullptr;
    cudaStream_t copy_out = nullptr;
    cudaEvent_t in_done[2] = {nullptr, nullptr};
    cudaEvent_t step_done[2] = {nullptr, nullptr};
    cudaEvent_t out_done[2] = {nullptr, nullptr};
    cudaEvent_t entry = nullptr;
};

namespace hc {

// Sets the thread's error message and returns `status`.
hc_status fail(hc_status status, const std::string& message);
hc_status check_cuda(cudaError_t err, const char* what);

// prologue.cu
hc_status launch_prepare(hc_context* ctx, const PrepArgs& args, cudaStream_t stream);
// The rows of positions [first, end) of `from_seq` in `from`, keys and values, into sequence 0 of `to`, and zeros to the values
// there from call_end to the end of its key tile.
hc_status launch_copy_rows(hc_context* ctx, const CacheView& from, int from_seq, const CacheView& to, int first, int end, int call_end,
                           int d, cudaStream_t stream);
// `count` floats, a multiple of 4 on 16-byte boundaries, one side possibly in pinned host memory.
hc_status launch_copy_floats(hc_context* ctx, float* dst, const float* src, size_t count, cudaStream_t stream);
hc_status launch_rms_norm_rows(hc_context* ctx, const void* x, const uint16_t* scale, void* out, int tokens, int width,
                               float eps, int x_dtype, int out_dtype, cudaStream_t stream);
hc_status launch_split_query_gate(hc_context* ctx, const void* combined, void* query, void* gate,
                                  int tokens, int heads, int d, int dtype, cudaStream_t stream);
hc_status launch_output_gate(hc_context* ctx, void* output, const void* gate, size_t count,
                             int dtype, cudaStream_t stream);

// attn_simt.cu
hc_status simt_prefill(hc_context* ctx, const AttnShape& shape, const CacheView& cache, int seq,
                       const uint16_t* q, int tokens, int first_position, const EpilogueArgs& ep,
                       cudaStream_t stream, const Blocks& blocks);
hc_status simt_decode(hc_context* ctx, const AttnShape& shape, const CacheView& cache,
                      const BatchMeta& meta, int n_seq, const uint16_t* q, const Workspace& ws,
                      const EpilogueArgs& ep, cudaStream_t stream);
// How a decode launch cuts its rows' keys (see TcArgs in tc_common.cuh for the three ways).
struct DecodePlan {
    int finish;          // whole rows per item, finished by the kernel itself
    int log_run;         // tile partials: items are aligned runs of 2^log_run tiles
    int run_segments;    // segment partials: about this many segments per item
    int tile_partials;   // the kernel writes one partial per tile (log_run < log_segment) rather than per segment
    int slots;           // partial slots per row
    int tiles;           // key tiles of the longest row (on this rank)
};
// The coarsest cut that gives at least target_items items, runs of max_run_segments segments at most.
DecodePlan plan_decode(const AttnShape& shape, const RowMap& map, const BatchMeta& meta, int n_seq, int target_items,
                       bool allow_whole, int max_run_segments);
// The cut simt_decode makes.
DecodePlan simt_plan_decode(const hc_context* ctx, const AttnShape& shape, const RowMap& map, const BatchMeta& meta, int n_seq);
// Both folds (tile partials) or the second fold (segment partials) over the partials in `ws`, then the
// epilogue: for the rows of a decode batch, or for the query tokens of a prefill chunk.
hc_status launch_merge_decode(hc_context* ctx, const AttnShape& shape, const RowMap& map, const BatchMeta& meta,
                              int n_seq, const Workspace& ws, const DecodePlan& plan, const EpilogueArgs& ep,
                              cudaStream_t stream);
hc_status launch_merge_prefill(hc_context* ctx, const AttnShape& shape, const RowMap& map, int tokens,
                               int first_position, int tokens_per_tile, const Blocks& blocks, const Workspace& ws, int slots,
                               const EpilogueArgs& ep, cudaStream_t stream);
hc_status launch_combine(hc_context* ctx, const float* gathered, int world, int rows, int q_heads,
                         int d, const EpilogueArgs& ep, cudaStream_t stream);
// Device address of the fixed scratch array on `device` (which must be current).
hc_status static_scratch_prepare(int device, float** address);

// attn_tc.cu
// A tensor map (CUtensorMap behind `map`) over a row-major bf16 matrix: boxes of 64 columns x box_rows
// rows, 128-byte swizzle, zeros beyond the edges.
hc_status tc_encode_2d(void* map, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows);
// The same with the 64-column blocks as a third dimension: boxes of box_blocks of them, [block][row][64 columns] in shared memory.
hc_status tc_encode_blocks(void* map, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, uint32_t box_blocks);
// The same over [planes][rows][cols]: boxes of 64 columns x box_rows x box_planes.
hc_status tc_encode_3d(void* map, const void* base, uint64_t cols, uint64_t rows, uint64_t planes, uint32_t box_rows, uint32_t box_planes);
bool tc_supported(const AttnShape& shape);
hc_status tc_prefill(hc_context* ctx, const AttnShape& shape, const hc_layer_store& layer,
                     const CacheView& cache, int seq, const uint16_t* q, int tokens,
                     int first_position, const Workspace& ws, const EpilogueArgs& ep, cudaStream_t stream, const Blocks& blocks);
// attn_decode.cu
// How a tcgen05 decode launch cuts its rows' keys, and the workspace that takes.
struct TcDecodePlan {
    int cluster;             // thread blocks that share a span of run_segments segments; 1: equal stretches of all rows
    int blocks;              // thread blocks
    int run_segments;
    int slots;               // partial slots per row: segments
    size_t part_o_floats, part_ml_floats, tickets;
};
hc_status decode_cluster_slots(hc_context* ctx);
TcDecodePlan tc_plan_decode(const hc_context* ctx, const AttnShape& shape, const RowMap& map, const BatchMeta& meta, int n_seq);
// One launch, for the first *served of the n_seq rows: as many as it takes (see there); the caller comes back for the rest.
hc_status tc_decode(hc_context* ctx, const AttnShape& shape, const hc_layer_store& layer,
                    const CacheView& cache, const BatchMeta& meta, int n_seq, const DecodeSource& src,
                    const Workspace& ws, const EpilogueArgs& ep, cudaStream_t stream, int* served);
// linear_tc.cu
// n_jobs (1 to 4) projections of the same x in one launch; bias / residual may be null, or hold nulls.
hc_status linear_tc(hc_context* ctx, const void* x, int n_jobs, const void* const* w, const void* const* bias,
                    const float* const* residual, void* const* y, const int* out_features, int tokens, int in_features,
                    int y_dtype, cudaStream_t stream);
// attn_pair.cu (args_ptr: the TcArgs of tc_common.cuh)
int pair_items_per_row_tile(int head_dim);
hc_status launch_attention_pair(hc_context* ctx, const hc_layer_store& layer, const void* args_ptr, int head_dim, cudaStream_t stream);
hc_status tc_make_tensor_maps(hc_layer_store& layer, size_t planes);
void tc_free_tensor_maps(hc_layer_store& layer);

}  // namespace hc
