// linear_tc.cu — the projections around the attention path on the 5th-generation tensor cores:
// y[t][o] = sum_i x[t][i] * w[o][i] (+ bias[o]), bf16 x bf16 -> fp32.
//
// Replaces bf16_gemv (Sources/HydraMetal/Shaders/dense.metal:14-60) and its batched and tiled
// forms (Sources/HydraMetal/Shaders/batch.metal:36-88, tiled.metal:48-120) for the Q, K, V and O
// projections; the CPU statement is ReferenceLayer.matVec
// (Sources/HydraReference/ReferenceLayer.swift:104-113).  The weight keeps the reference's layout:
// row-major [out_features][in_features] bf16, so both operands are K-major and no transpose is
// needed.  Where the reference gives every output row its own threadgroup that streams that row
// of the weight once per token, a weight tile fetched by TMA serves up to 256 tokens here.
//
// Two kernels.  A call of up to 128 tokens reads the weights once and little else: linear_few_kernel, one CTA
// per SM, narrow output tiles, up to nine 16 to 40 KB stages in flight.  Prompts are bound by the tensor pipe:
// linear_pair_kernel, where two SMs share a 256-row output tile (cta_group::2: each loads its own 128
// rows of x and half of the weight tile, so a K step brings 24 to 32 KB into each SM for 256 x BN outputs where a
// CTA of its own needed 48 KB for 128 x 256), six to eight stages, two accumulators in tensor memory.
//   warp 0      TMA producer: x tile and w tile per K step of 64 into the ring
//               (a launch may carry up to four projections of the same x: one list of tiles)
//   warp 1      MMA issuer (of the leading CTA): four tcgen05.mma per K step into one of two accumulators
//   warps 4-7   epilogue: the finished accumulator from tensor memory, + bias (+ residual), to y (fp32 or bf16),
//               thread = row, while the next tile's MMAs fill the other accumulator
// Every mbarrier wait is bounded and reports through the context's status word.

#include <algorithm>

#include "internal.hpp"
#include "linear_plan.hpp"
#include "tc_ptx.cuh"

namespace hc {
namespace {

constexpr int kLinM = 128;
constexpr int kLinK = 64;                       // one 128-byte swizzled row of bf16
constexpr int kLinABytes = kLinM * kLinK * 2;   // 16 KB
constexpr int kLinThreads = 256;

// Few tokens: the work is reading the weight once.  Column tiles of BN weight rows, as narrow as gives every SM one tile
// and none two (a second tile doubles the call's time; columns cost little), and stages of `subs` K steps of
// 64 each: with one K step a stage the waits and the issue around its four MMAs took longer than they did
// (137 clocks an MMA against the 41 it takes), with four they do not.
constexpr int kFewMaxStages = 9;
constexpr int kFewSmemBytes = 208 * 1024;       // ring and the x tile's overhang (see launch_few)
constexpr int kFewTmemCols = 128;               // two accumulators of up to 64 columns

// Pairs: 256 x BN tiles, each CTA holding 128 rows of x and BN / 2 rows of w per stage.  An output element is the same
// sum in the same order in every shape, so a token projected alone and inside a prompt gets the same bits.
template <int BN>
struct PairShape {
    static constexpr int kStages = BN >= 224 ? 6 : BN >= 160 ? 7 : 8;
    static constexpr int kBBytes = BN / 2 * kLinK * 2;
    static constexpr int kTmemCols = 2 * BN <= 256 ? 256 : 512;
    static constexpr int kSmemBytes = 1024 + kStages * (kLinABytes + kBBytes);
};

constexpr int kLinMaxStages = 9;
struct LinBarriers {
    uint64_t full[kLinMaxStages], empty[kLinMaxStages];
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    int abort_flag;
    int pad[2];
};
static_assert(sizeof(LinBarriers) % 16 == 0, "the staging behind it is 16-byte aligned");

// One launch may carry several projections of the same x (q, k and v of a layer): their output tiles
// form one list, job after job.
struct LinJob {
    const uint16_t* bias;     // bf16 [out_features] or null
    const float* residual;    // fp32 [tokens][out_features] added to the result, or null (may be y itself)
    void* y;                  // [tokens][out_features]
    int out_features;
    int first_tile;           // of this job in the launch's list; its tiles: column tile major, row tiles adjacent
};

struct LinArgs {
    LinJob job[kLinJobs];
    int n_jobs;
    int y_dtype;              // HC_F32 or HC_BF16
    int tokens;
    int tiles_m, n_tiles, k_steps;   // tiles of 128 rows (few tokens) or 256 (pairs)
    int n_wide;               // pairs, 256 columns: the first n_wide tiles are that wide, the others half of it
    int a_bytes;              // few tokens: of one x box, as many rows of 128 bytes as there are tokens (rounded up to 8)
    int stages;               // few tokens
    int* status;
};

struct LinTile {
    int job, tn, tm;
};
__device__ __forceinline__ LinTile decode_tile(const LinArgs& args, int tile) {
    LinTile t;
    t.job = 0;
    #pragma unroll
    for (int j = 1; j < kLinJobs; ++j) {
        if (j < args.n_jobs && tile >= args.job[j].first_tile) t.job = j;
    }
    const int local = tile - args.job[t.job].first_tile;
    t.tn = local / args.tiles_m;
    t.tm = local - t.tn * args.tiles_m;
    return t;
}

// 32 accumulator columns of a warp's 32 rows (lane = row in `v`): + bias (+ residual), to y.  The block goes through
// 4 KB of shared memory so that a store instruction writes four rows' whole 128-byte lines (64 for bf16)
// instead of 16 bytes of 32 rows, and the residual is read the same way, a block ahead: it may be y itself, so the
// compiler may not move a load across a store, and a block's eight loads one after the other cost more
// than its MMAs (o_proj of 4096 tokens: 141 us).
constexpr int kLinStageBytes = 32 * 128;
// A tile's bias, eight columns a lane in one load while the tile is computed, and the four of them that a lane adds in a block
// of 32 columns.  (Loaded block by block, one ahead, they were 1.4 us of a 256-column tile.)
__device__ __forceinline__ uint4 load_bias(const LinJob& job, int col0) {
    const int col = col0 + (threadIdx.x & 31) * 8;
    if (job.bias == nullptr || col >= job.out_features) return make_uint4(0, 0, 0, 0);
    if (col + 8 <= job.out_features && (reinterpret_cast<uintptr_t>(job.bias) & 15) == 0) return __ldg(reinterpret_cast<const uint4*>(job.bias + col));
    uint32_t b[8];
    #pragma unroll
    for (int i = 0; i < 8; ++i) b[i] = col + i < job.out_features ? __ldg(job.bias + col + i) : 0u;
    return make_uint4(b[0] | b[1] << 16, b[2] | b[3] << 16, b[4] | b[5] << 16, b[6] | b[7] << 16);
}
__device__ __forceinline__ float4 block_bias(const uint4& tile, int block) {
    const int lane = threadIdx.x & 31, from = block * 4 + ((lane & 7) >> 1);
    const uint32_t x = __shfl_sync(0xffffffffu, tile.x, from), y = __shfl_sync(0xffffffffu, tile.y, from);
    const uint32_t z = __shfl_sync(0xffffffffu, tile.z, from), w = __shfl_sync(0xffffffffu, tile.w, from);
    const uint32_t lo = (lane & 1) ? z : x, hi = (lane & 1) ? w : y;
    return make_float4(__uint_as_float(lo << 16), __uint_as_float(lo & 0xffff0000u), __uint_as_float(hi << 16), __uint_as_float(hi & 0xffff0000u));
}
__device__ __forceinline__ void load_residual(const LinJob& job, int row0, int row_end, int col0, float4 (&z)[8]) {
    if (job.residual == nullptr) return;                                        // z is not looked at
    #pragma unroll
    for (int k = 0; k < 8; ++k) z[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int lane = threadIdx.x & 31;
    const int col = col0 + (lane & 7) * 4;
    if (col + 4 > job.out_features || (job.out_features & 3) != 0) return;      // read element by element when it is added
    const bool aligned = (reinterpret_cast<uintptr_t>(job.residual) & 15) == 0;
    #pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int row = row0 + k * 4 + (lane >> 3);
        if (row >= row_end) continue;
        const float* src = job.residual + size_t(row) * job.out_features + col;
        if (aligned) z[k] = *reinterpret_cast<const float4*>(src);
        else z[k] = make_float4(src[0], src[1], src[2], src[3]);
    }
}
__device__ __forceinline__ float2 add2(float x0, float x1, float y0, float y1) {
    uint64_t x = uint64_t(__float_as_uint(x0)) | (uint64_t(__float_as_uint(x1)) << 32);
    const uint64_t y = uint64_t(__float_as_uint(y0)) | (uint64_t(__float_as_uint(y1)) << 32);
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(x) : "l"(y));
    return make_float2(__uint_as_float(uint32_t(x)), __uint_as_float(uint32_t(x >> 32)));
}
// A block of a job whose rows start on 8- or 16-byte boundaries.  One warp a scheduler walks the epilogue, so what it costs is
// its instructions one after the other (five to seven clocks each): with a branch and an address for every row they were 420 a
// block, 1500 ns, and a launch of one round of tiles took longer than without the pairs (400 tokens to 9216 columns 21.2
// us before the pairs, 24.6 with them, 16.7 now; 64 -> 2560 features of 4096 tokens 27.5, 37.4 and 15.5).
template <bool kFp32, bool kResidual>
__device__ __forceinline__ void store_rows(const LinJob& job, const uint32_t (&v)[32], const float4& bias, const float4 (&z)[8],
                                           int row0, int row_end, int col0, unsigned char* stage, int width) {
    const int lane = threadIdx.x & 31;
    #pragma unroll
    for (int c = 0; c < 8; ++c) {
        *reinterpret_cast<uint4*>(stage + lane * 128 + ((c ^ (lane & 7)) << 4)) = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
    }
    __syncwarp();
    const int chunk = lane & 7, r0 = lane >> 3;
    float4 x[8];
    #pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = *reinterpret_cast<const float4*>(stage + (k * 4 + r0) * 128 + ((chunk ^ ((k & 1) * 4 + r0)) << 4));
    const size_t at = size_t(row0 + r0) * job.out_features + col0 + chunk * 4;
    unsigned char* dst = static_cast<unsigned char*>(job.y) + at * (kFp32 ? 4 : 2);
    const size_t step = size_t(job.out_features) * (kFp32 ? 16 : 8);
    const int rows = chunk * 4 < width && col0 + chunk * 4 < job.out_features ? row_end - row0 - r0 : 0;      // k * 4 of them
    #pragma unroll
    for (int k = 0; k < 8; ++k) {
        float2 lo = add2(x[k].x, x[k].y, bias.x, bias.y), hi = add2(x[k].z, x[k].w, bias.z, bias.w);
        if (kResidual) {
            lo = add2(lo.x, lo.y, z[k].x, z[k].y);
            hi = add2(hi.x, hi.y, z[k].z, z[k].w);
        }
        if (kFp32) {
            if (k * 4 < rows) *reinterpret_cast<float4*>(dst) = make_float4(lo.x, lo.y, hi.x, hi.y);
        } else {
            uint2 packed;
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(packed.x) : "f"(lo.y), "f"(lo.x));
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(packed.y) : "f"(hi.y), "f"(hi.x));
            if (k * 4 < rows) *reinterpret_cast<uint2*>(dst) = packed;
        }
        dst += step;
    }
    __syncwarp();
}
// (Rows up to row_end.)
__device__ __forceinline__ void store_block(const LinArgs& args, const LinJob& job, const uint32_t (&v)[32], const float4& bias, const float4 (&z)[8], int row0,
                                            int row_end, int col0, unsigned char* stage, int width = 32) {
    if (col0 >= job.out_features || row0 >= row_end) return;              // warp-uniform, as the next
    if ((job.out_features & 3) == 0) {
        if (args.y_dtype != HC_F32) store_rows<false, false>(job, v, bias, z, row0, row_end, col0, stage, width);
        else if (job.residual != nullptr) store_rows<true, true>(job, v, bias, z, row0, row_end, col0, stage, width);
        else store_rows<true, false>(job, v, bias, z, row0, row_end, col0, stage, width);
        return;
    }
    const int lane = threadIdx.x & 31;
    #pragma unroll
    for (int c = 0; c < 8; ++c) {
        *reinterpret_cast<uint4*>(stage + lane * 128 + ((c ^ (lane & 7)) << 4)) = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
    }
    __syncwarp();
    const int chunk = lane & 7, col = col0 + chunk * 4;
    #pragma unroll 1
    for (int k = 0; k < 8; ++k) {
        const int r = k * 4 + (lane >> 3);
        if (row0 + r >= row_end || chunk * 4 >= width) continue;
        const float4 x = *reinterpret_cast<const float4*>(stage + r * 128 + ((chunk ^ (r & 7)) << 4));
        const float y[4] = {__fadd_rn(x.x, bias.x), __fadd_rn(x.y, bias.y), __fadd_rn(x.z, bias.z), __fadd_rn(x.w, bias.w)};
        const size_t at = size_t(row0 + r) * job.out_features + col;
        #pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (col + i >= job.out_features) continue;
            store_io(job.y, at + i, args.y_dtype, job.residual != nullptr ? __fadd_rn(y[i], job.residual[at + i]) : y[i]);
        }
    }
    __syncwarp();
}

__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap* map, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global [%0, {%1, %2, %3}];"
                 ::"l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}

// ROWS: of the MMA, 128 or 64.  An MMA of so few columns takes as long as its operands take out of shared memory, 32 clocks for
// 128 rows of x and BN / 4 for the weights, and the chain of K steps is what a launch of one token lasts (256 MMAs at o_proj): up to
// 64 tokens go as 64 rows.  Their accumulators lie in the first 16 lanes of each warp's quarter of tensor memory.
template <int BN, int SUBS, int ROWS>
__global__ void __launch_bounds__(kLinThreads, 1)
linear_few_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w0,
                  const __grid_constant__ CUtensorMap tmap_w1, const __grid_constant__ CUtensorMap tmap_w2,
                  const __grid_constant__ CUtensorMap tmap_w3, const LinArgs args) {
    constexpr int kWBytes = BN * kLinK * 2;                         // weight rows of a K step
    extern __shared__ unsigned char raw_smem[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw_smem) + 1023) & ~uintptr_t(1023));
    const int a_stage = SUBS * args.a_bytes, w_stage = SUBS * kWBytes;
    unsigned char* a_smem = base;                                   // [stages][subs][x rows x 64]
    unsigned char* w_smem = a_smem + args.stages * a_stage;         // [stages][subs][BN x 64]
    LinBarriers* bars = reinterpret_cast<LinBarriers*>(base + kFewSmemBytes);        // and the epilogue's staging
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    volatile int* abort_flag = &bars->abort_flag;
    const int n_tiles = args.n_tiles, k_steps = args.k_steps;
    auto weight_map = [&](int job) { return job == 0 ? &tmap_w0 : job == 1 ? &tmap_w1 : job == 2 ? &tmap_w2 : &tmap_w3; };

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int i = 0; i < kFewMaxStages; ++i) {
            mbar_init(&bars->full[i], 1);
            mbar_init(&bars->empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->acc_full[i], 1);
            mbar_init(&bars->acc_empty[i], 4);
        }
        bars->abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc(&bars->tmem_base, kFewTmemCols);
    if (warp == 2 && int(blockIdx.x) < n_tiles) {
        // While the kernel before this one finishes, the weights come into L2 (where it may still change them: nothing
        // is read into this CTA before the wait below).
        const LinTile where = decode_tile(args, blockIdx.x);
        for (int k = lane * SUBS; k < k_steps; k += 32 * SUBS) tma_prefetch_3d(weight_map(where.job), 0, where.tn * BN, k);
    }
    if (warp == 0 && lane == 0) prefetch_tensormap(&tmap_x);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    pdl_wait();

    if (warp == 0) {
        // ===== producer =====
        if (lane == 0) {
            int slot = 0;
            uint32_t round = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < n_tiles; tile += gridDim.x) {
                const LinTile where = decode_tile(args, tile);
                const CUtensorMap* tmap_w = weight_map(where.job);
                for (int k = 0; k < k_steps; k += SUBS) {
                    if (round > 0 && !mbar_wait(&bars->empty[slot], (round - 1) & 1, abort_flag, args.status, 21)) { ok = false; break; }
                    // A stage's K steps in one copy each: the maps have them as a third dimension (zeros behind the last, which
                    // count).  Step by step a launch of one token was 128 copies from one thread.
                    mbar_expect_tx(&bars->full[slot], uint32_t(w_stage + a_stage));
                    tma_load_3d(w_smem + slot * w_stage, tmap_w, &bars->full[slot], 0, where.tn * BN, k);
                    tma_load_3d(a_smem + slot * a_stage, &tmap_x, &bars->full[slot], 0, 0, k);
                    if (++slot == args.stages) {
                        slot = 0;
                        ++round;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ===== MMA issuer (the warp walks the loop converged; one elected lane issues) =====
        constexpr uint32_t idesc = (instr_desc(BN, false) & ~(0x1fu << 24)) | (uint32_t(ROWS >> 4) << 24);
        const uint64_t a_desc0 = smem_desc(smem_u32(a_smem), 16);
        const uint64_t w_desc0 = smem_desc(smem_u32(w_smem), 16);
        int slot = 0;
        uint32_t round = 0, count = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < n_tiles; tile += gridDim.x, ++count) {
            const int acc = int(count & 1);
            // The epilogue must have taken this accumulator's previous tile out.
            if (count >= 2 && !mbar_wait(&bars->acc_empty[acc], ((count >> 1) - 1) & 1, abort_flag, args.status, 22)) break;
            tc_fence_after();
            for (int k = 0; k < k_steps; k += SUBS) {
                if (!mbar_wait(&bars->full[slot], round & 1, abort_flag, args.status, 23)) { ok = false; break; }
                tc_fence_after();
                const uint64_t a_desc = warp_uniform(a_desc0 + uint64_t((slot * a_stage) >> 4));
                const uint64_t w_desc = warp_uniform(w_desc0 + uint64_t((slot * w_stage) >> 4));
                const uint32_t x_step = warp_uniform(uint32_t(args.a_bytes >> 4)), d_tmem = warp_uniform(tmem + acc * 64);
                const int n = min(SUBS, k_steps - k);
                if (elect_one()) {
                    #pragma unroll
                    for (int u = 0; u < SUBS; ++u) {
                        if (u < n) {
                            #pragma unroll
                            for (int ks = 0; ks < kLinK / 16; ++ks) {
                                mma_ss(d_tmem, a_desc + uint64_t(u * x_step + ((ks * 32) >> 4)), w_desc + uint64_t((u * kWBytes + ks * 32) >> 4), idesc,
                                       (u | ks) != 0 ? 1u : uint32_t(k != 0));
                            }
                        }
                    }
                    tc_commit(&bars->empty[slot]);
                    if (k + n == k_steps) tc_commit(&bars->acc_full[acc]);
                }
                __syncwarp();
                if (++slot == args.stages) {
                    slot = 0;
                    ++round;
                }
            }
        }
    } else if (warp >= 4) {
        // ===== epilogue: thread = token (of 64 rows: every other 16 threads) =====
        const int quad = warp & 3;
        unsigned char* stage = reinterpret_cast<unsigned char*>(bars + 1) + quad * kLinStageBytes;
        const uint32_t lane_base = uint32_t(quad * 32) << 16;
        uint32_t count = 0;
        for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++count) {
            const LinTile where = decode_tile(args, tile);
            const LinJob& job = args.job[where.job];
            const int acc = int(count & 1);
            constexpr int kQuadRows = ROWS / 4;
            const int row0 = quad * kQuadRows, row_end = min(args.tokens, row0 + kQuadRows);
            const bool rows = row0 < row_end;                       // warp-uniform
            float4 z[8];
            if (rows) load_residual(job, row0, row_end, where.tn * BN, z);
            const uint4 bias = load_bias(job, where.tn * BN);
            if (!mbar_wait(&bars->acc_full[acc], (count >> 1) & 1, abort_flag, args.status, 24)) break;
            tc_fence_after();
            #pragma unroll 1
            for (int col = 0; rows && col < BN; col += 32) {
                uint32_t v[32];
                HC_TMEM_LD32(tmem + lane_base + acc * 64 + col, v);
                tc_wait_ld();
                if (col > 0) load_residual(job, row0, row_end, where.tn * BN + col, z);
                store_block(args, job, v, block_bias(bias, col >> 5), z, row0, row_end, where.tn * BN + col, stage, BN - col);
                __syncwarp();          // the next tcgen05.ld is warp-wide
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->acc_empty[acc]);
        }
    }

    // Teardown.  On the abort path the producer first lets its copies in flight land (bounded).
    if (warp == 0 && lane == 0 && *abort_flag != 0) {
        const long long start = clock64();
        while (static_cast<unsigned long long>(clock64() - start) < 200000000ull) { }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, kFewTmemCols);
}

// Two SMs per 256 x BN tile (BN 256: of tiles of 128 columns too, see decode_wide); see the head of the file.  The leading
// CTA's barriers count both CTAs' loads.
template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kLinThreads, 1)
linear_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w0,
                   const __grid_constant__ CUtensorMap tmap_w1, const __grid_constant__ CUtensorMap tmap_w2,
                   const __grid_constant__ CUtensorMap tmap_w3, const LinArgs args) {
    using PS = PairShape<BN>;
    extern __shared__ unsigned char raw_smem[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw_smem) + 1023) & ~uintptr_t(1023));
    unsigned char* a_smem = base;                                   // [stages][128 x 64]
    unsigned char* b_smem = a_smem + PS::kStages * kLinABytes;      // [stages][BN / 2 x 64]
    LinBarriers* bars = reinterpret_cast<LinBarriers*>(b_smem + PS::kStages * PS::kBBytes);      // and the epilogue's staging
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int rank = int(cluster_rank());
    const int pair = int(blockIdx.x) >> 1, pairs = int(gridDim.x) >> 1;
    volatile int* abort_flag = &bars->abort_flag;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int i = 0; i < PS::kStages; ++i) {
            mbar_init(&bars->full[i], 1);
            mbar_init(&bars->empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->acc_full[i], 1);
            mbar_init(&bars->acc_empty[i], 8);                      // the epilogue warps of both CTAs
        }
        bars->abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc_pair(&bars->tmem_base, PS::kTmemCols);
    if (warp == 0 && lane == 0) {
        prefetch_tensormap(&tmap_x);
        prefetch_tensormap(&tmap_w0);
    }
    tc_fence_before();
    __syncthreads();
    cluster_arrive();
    cluster_wait();                 // the peer's barriers are there
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    pdl_wait();

    const int n_tiles = args.n_tiles;
    constexpr bool kTwoWidths = BN == 256;
    auto tile_at = [&](int tile) -> LinWide {
        if constexpr (kTwoWidths) return decode_wide<BN>(args, tile);
        const LinTile where = decode_tile(args, tile);
        return LinWide{where.job, where.tn * BN, where.tm, BN};
    };
    if (warp == 0) {
        // ===== producer: this CTA's rows of x and its half of the weight tile, counted by the leader =====
        if (lane == 0) {
            uint32_t step = 0;
            bool ok = true;
            for (int tile = pair; ok && tile < n_tiles; tile += pairs) {
                const LinWide where = tile_at(tile);
                const int tm = where.tm, w_row = where.col + rank * (where.width / 2);
                const CUtensorMap* tmap_w = where.job == 0 ? &tmap_w0 : where.job == 1 ? &tmap_w1 : where.job == 2 ? &tmap_w2 : &tmap_w3;
                for (int k = 0; k < args.k_steps; ++k, ++step) {
                    const int slot = int(step % PS::kStages);
                    const uint32_t round = step / PS::kStages;
                    if (round > 0 && !mbar_wait(&bars->empty[slot], (round - 1) & 1, abort_flag, args.status, 21)) { ok = false; break; }
                    const uint32_t full = cluster_addr(&bars->full[slot], 0);
                    if (rank == 0) mbar_expect_tx(&bars->full[slot], 2 * (kLinABytes + where.width / 2 * kLinK * 2));
                    tma_load_2d_pair(a_smem + slot * kLinABytes, &tmap_x, full, k * kLinK, tm * (2 * kLinM) + rank * kLinM);
                    tma_load_2d_pair(b_smem + slot * PS::kBBytes, tmap_w, full, k * kLinK, w_row);
                    if (kTwoWidths && where.width == BN) {       // (boxes of 64 rows)
                        tma_load_2d_pair(b_smem + slot * PS::kBBytes + PS::kBBytes / 2, tmap_w, full, k * kLinK, w_row + BN / 4);
                    }
                }
            }
        }
    } else if (warp == 1 && rank == 0) {
        // ===== MMA issuer (the warp walks the loop converged; one elected lane issues) =====
        const uint64_t a_desc0 = smem_desc(smem_u32(a_smem), 16);
        const uint64_t b_desc0 = smem_desc(smem_u32(b_smem), 16);
        uint32_t step = 0, count = 0;
        bool ok = true;
        for (int tile = pair; ok && tile < n_tiles; tile += pairs, ++count) {
            const int acc = int(count & 1);
            // The epilogues must have taken this accumulator's previous tile out.
            if (count >= 2 && !mbar_wait(&bars->acc_empty[acc], ((count >> 1) - 1) & 1, abort_flag, args.status, 22)) break;
            tc_fence_after();
            const uint32_t idesc = kTwoWidths && tile >= args.n_wide ? instr_desc_pair(BN / 2, false) : instr_desc_pair(BN, false);
            for (int k = 0; k < args.k_steps; ++k, ++step) {
                const int slot = int(step % PS::kStages);
                if (!mbar_wait(&bars->full[slot], (step / PS::kStages) & 1, abort_flag, args.status, 23)) { ok = false; break; }
                tc_fence_after();
                const uint64_t a_desc = warp_uniform(a_desc0 + uint64_t((slot * kLinABytes) >> 4));
                const uint64_t b_desc = warp_uniform(b_desc0 + uint64_t((slot * PS::kBBytes) >> 4));
                if (elect_one()) {
                    #pragma unroll
                    for (int ks = 0; ks < kLinK / 16; ++ks) {
                        mma_ss_pair(tmem + acc * BN, a_desc + uint64_t((ks * 32) >> 4), b_desc + uint64_t((ks * 32) >> 4), idesc,
                                    (k | ks) != 0 ? 1u : 0u);
                    }
                    tc_commit_pair(&bars->empty[slot]);
                    if (k + 1 == args.k_steps) tc_commit_pair(&bars->acc_full[acc]);
                }
                __syncwarp();
            }
        }
    } else if (warp >= 4) {
        // ===== epilogue: thread = row of this CTA's half of the tile =====
        const int quad = warp & 3;
        unsigned char* stage = reinterpret_cast<unsigned char*>(bars + 1) + quad * kLinStageBytes;
        const uint32_t lane_base = uint32_t(quad * 32) << 16;
        uint32_t count = 0;
        for (int tile = pair; tile < n_tiles; tile += pairs, ++count) {
            const LinWide where = tile_at(tile);
            const LinJob& job = args.job[where.job];
            const int row0 = where.tm * (2 * kLinM) + rank * kLinM + quad * 32;
            const int acc = int(count & 1);
            float4 z[8], z_next[8];
            load_residual(job, row0, args.tokens, where.col, z);
            const uint4 bias = load_bias(job, where.col);
            if (!mbar_wait(&bars->acc_full[acc], (count >> 1) & 1, abort_flag, args.status, 24)) break;
            tc_fence_after();
            #pragma unroll 1
            for (int chunk = 0; chunk < where.width / 32; ++chunk) {
                uint32_t v[32];
                HC_TMEM_LD32(tmem + lane_base + acc * BN + chunk * 32, v);
                if (chunk + 1 < where.width / 32) load_residual(job, row0, args.tokens, where.col + (chunk + 1) * 32, z_next);
                tc_wait_ld();
                store_block(args, job, v, block_bias(bias, chunk), z, row0, args.tokens, where.col + chunk * 32, stage);
                if (job.residual != nullptr) {
                    #pragma unroll
                    for (int k = 0; k < 8; ++k) z[k] = z_next[k];
                }
                __syncwarp();          // the next tcgen05.ld is warp-wide
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(cluster_addr(&bars->acc_empty[acc], 0));
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
    cluster_wait();                 // neither CTA leaves while the other's MMAs or arrivals may still name it
    if (warp == 1) tmem_dealloc_pair(tmem, PS::kTmemCols);
}

}  // namespace

// Encoding a tensor map costs a few microseconds of host time, as much as a decode-sized call's
// kernel; weights and activation buffers recur from call to call, so the last maps are kept, keyed
// by what determines them.  One caller thread per context: the cache is per thread.
// k_blocks: 0, boxes of one K step; or so many of them in a box.
static hc_status cached_map(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, uint32_t k_blocks) {
    struct Entry {
        const void* base;
        uint64_t rows, cols;
        uint32_t box_rows, k_blocks;
        CUtensorMap map;
    };
    constexpr int kEntries = 32;
    static thread_local Entry entries[kEntries];
    static thread_local int used = 0, next = 0;
    for (int i = 0; i < used; ++i) {
        const Entry& e = entries[i];
        if (e.base == base && e.rows == rows && e.cols == cols && e.box_rows == box_rows && e.k_blocks == k_blocks) {
            *out = e.map;
            return HC_OK;
        }
    }
    Entry& e = entries[next];
    const hc_status st = k_blocks == 0 ? tc_encode_2d(&e.map, base, rows, cols, box_rows) : tc_encode_blocks(&e.map, base, rows, cols, box_rows, k_blocks);
    if (st != HC_OK) {
        e.base = nullptr;
        return st;
    }
    e.base = base;
    e.rows = rows;
    e.cols = cols;
    e.box_rows = box_rows;
    e.k_blocks = k_blocks;
    *out = e.map;
    next = (next + 1) % kEntries;
    used = std::min(used + 1, kEntries);
    return HC_OK;
}

// Tensor maps and the tile list of a launch with column tiles of `bn` and row tiles of `bm` over boxes of x_rows and
// w_rows rows (and k_blocks K steps).
struct LinMaps {
    CUtensorMap x, w[kLinJobs];
};
static hc_status prepare_linear(LinMaps& maps, const void* x, const void* const* w, LinArgs& args, int in_features, int bm, int bn,
                                int x_rows, int w_rows, int k_blocks) {
    hc_status st = cached_map(&maps.x, x, uint64_t(args.tokens), uint64_t(in_features), uint32_t(x_rows), uint32_t(k_blocks));
    args.tiles_m = (args.tokens + bm - 1) / bm;
    int tiles = 0;
    for (int j = 0; j < kLinJobs && st == HC_OK; ++j) {
        const int source = j < args.n_jobs ? j : 0;            // unused maps repeat the first
        st = cached_map(&maps.w[j], w[source], uint64_t(args.job[source].out_features), uint64_t(in_features), uint32_t(w_rows), uint32_t(k_blocks));
        if (j < args.n_jobs) {
            args.job[j].first_tile = tiles;
            tiles += args.tiles_m * ((args.job[j].out_features + bn - 1) / bn);
        }
    }
    args.n_tiles = tiles;
    return st;
}

template <typename Kernel>
static hc_status launch_linear_kernel(hc_context* ctx, Kernel kernel, bool (&configured)[64], int grid, int smem, const LinMaps& maps,
                                      const LinArgs& args, cudaStream_t stream) {
    if (!configured[ctx->device & 63]) {
        const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (err != cudaSuccess) return check_cuda(err, "linear kernel shared memory");
        configured[ctx->device & 63] = true;
    }
    const cudaError_t launched = launch_pdl(kernel, grid, kLinThreads, size_t(smem), stream, maps.x, maps.w[0], maps.w[1], maps.w[2],
                                            maps.w[3], args);
    ctx->launches += 1;
    return check_cuda(launched, "linear kernel launch");
}

template <int BN, int ROWS>
static hc_status launch_few(hc_context* ctx, const void* x, const void* const* w, LinArgs args, int in_features, cudaStream_t stream) {
    LinMaps maps;
    // A box that reaches past the last token is filled with zeros, and that fill measured slower than
    // reading real rows (one token: 21 us against 13 us for 128): a call of few tokens loads only the
    // rows it has.  The rows of the 128-row operand tile it leaves unwritten are whatever lies behind it in shared memory
    // and feed accumulator rows that are never stored (a row of the result depends on its own row of x alone).
    const int x_rows = std::min(kLinM, (args.tokens + 7) & ~7);
    args.a_bytes = x_rows * kLinK * 2;
    // Stages of four K steps while there is room for four of them, of two beyond; the last x tile's overhang
    // stays inside the ring (there are at least 16 KB of weights behind the x tiles, or room).
    const int step_bytes = args.a_bytes + BN * kLinK * 2;
    const int room = kFewSmemBytes - kLinABytes;
    const int subs = 16 * step_bytes <= room ? 4 : 2;
    args.stages = std::max(1, std::min(kFewMaxStages, room / (subs * step_bytes)));
    const hc_status st = prepare_linear(maps, x, w, args, in_features, kLinM, BN, x_rows, BN, subs);
    if (st != HC_OK) return st;
    static bool configured4[64] = {}, configured2[64] = {};
    const int grid = std::max(1, std::min(args.n_tiles, std::max(ctx->sm_count, 1)));
    constexpr int smem = 1024 + kFewSmemBytes + int(sizeof(LinBarriers)) + 4 * kLinStageBytes;
    static_assert(smem <= 227 * 1024, "shared memory of one CTA");
    return subs == 4 ? launch_linear_kernel(ctx, linear_few_kernel<BN, 4, ROWS>, configured4, grid, smem, maps, args, stream)
                     : launch_linear_kernel(ctx, linear_few_kernel<BN, 2, ROWS>, configured2, grid, smem, maps, args, stream);
}

template <int BN>
static hc_status launch_pair(hc_context* ctx, const void* x, const void* const* w, LinArgs args, int in_features, cudaStream_t stream,
                             int n_wide = 0, int n_tiles = 0) {
    LinMaps maps;
    const hc_status st = prepare_linear(maps, x, w, args, in_features, 2 * kLinM, BN, kLinM, BN == 256 ? BN / 4 : BN / 2, 0);
    if (st != HC_OK) return st;
    if (BN == 256) {
        args.n_wide = n_wide;
        args.n_tiles = n_tiles;
    }
    static bool configured[64] = {};
    constexpr int smem = PairShape<BN>::kSmemBytes + int(sizeof(LinBarriers)) + 4 * kLinStageBytes;
    static_assert(smem <= 227 * 1024, "shared memory of one CTA");
    const int grid = 2 * std::max(1, std::min(args.n_tiles, std::max(ctx->sm_count / 2, 1)));
    return launch_linear_kernel(ctx, linear_pair_kernel<BN>, configured, grid, smem, maps, args, stream);
}

hc_status linear_tc(hc_context* ctx, const void* x, int n_jobs, const void* const* w, const void* const* bias,
                    const float* const* residual, void* const* y, const int* out_features, int tokens, int in_features,
                    int y_dtype, cudaStream_t stream) {
    LinArgs args{};
    args.n_jobs = n_jobs;
    for (int j = 0; j < n_jobs; ++j) {
        args.job[j].bias = bias ? static_cast<const uint16_t*>(bias[j]) : nullptr;
        args.job[j].residual = residual ? residual[j] : nullptr;
        args.job[j].y = y[j];
        args.job[j].out_features = out_features[j];
    }
    args.y_dtype = y_dtype;
    args.tokens = tokens;
    args.k_steps = in_features / kLinK;
    args.status = ctx->status_dev;
    if (tokens <= kLinM) {
        const int sms = std::max(ctx->sm_count, 1);
        auto tiles = [&](int bn) {
            int n = 0;
            for (int j = 0; j < n_jobs; ++j) n += (out_features[j] + bn - 1) / bn;
            return n;
        };
        if (tokens <= 64) {                                  // (64 rows take columns in eights)
            if (tiles(16) <= sms) return launch_few<16, 64>(ctx, x, w, args, in_features, stream);
            if (tiles(24) <= sms) return launch_few<24, 64>(ctx, x, w, args, in_features, stream);
            if (tiles(32) <= sms) return launch_few<32, 64>(ctx, x, w, args, in_features, stream);
            if (tiles(40) <= sms) return launch_few<40, 64>(ctx, x, w, args, in_features, stream);
            if (tiles(48) <= sms) return launch_few<48, 64>(ctx, x, w, args, in_features, stream);
            return launch_few<64, 64>(ctx, x, w, args, in_features, stream);
        }
        if (tiles(16) <= sms) return launch_few<16, 128>(ctx, x, w, args, in_features, stream);
        if (tiles(32) <= sms) return launch_few<32, 128>(ctx, x, w, args, in_features, stream);
        if (tiles(48) <= sms) return launch_few<48, 128>(ctx, x, w, args, in_features, stream);
        return launch_few<64, 128>(ctx, x, w, args, in_features, stream);
    }
    const LinPlan plan = plan_pairs(out_features, n_jobs, (tokens + 2 * kLinM - 1) / (2 * kLinM), std::max(ctx->sm_count / 2, 1));
    switch (plan.width) {
        case 256: return launch_pair<256>(ctx, x, w, args, in_features, stream, int(plan.n_wide), int(plan.n_tiles));
        case 192: return launch_pair<192>(ctx, x, w, args, in_features, stream);
        case 160: return launch_pair<160>(ctx, x, w, args, in_features, stream);
        default: return launch_pair<128>(ctx, x, w, args, in_features, stream);
    }
}

}  // namespace hc
