// prologue.cu — everything that happens to q, k and v before attention, in one kernel:
// per-head RMSNorm, half-split rotation, rounding to bf16 and, for k and v, the store into the
// cache.  Also the stand-alone element-wise kernels of the protocol.
//
// Replaces, fused: rms_norm_heads (Sources/HydraMetal/Shaders/gemma.metal:785-821), rope_apply /
// rope_apply_batch / rope_apply_batched (attention.metal:48-72, batch.metal:224-251,
// gemma.metal:961-984) and kv_cache_write / kv_cache_write_batch (dense.metal:66-86,
// batch.metal:254-277).  The order is the reference's: norm, then rotation, then the cast
// (Sources/HydraReference/Gemma4ReferenceLayer.swift:154-157, 234-246); v is normalised without a
// weight and never rotated.
//
// HBM-bound and tiny: a chunk of 512 tokens moves a few MB, so what matters is how many bytes each
// warp has in flight.

#include <algorithm>

#include "internal.hpp"
#include "prologue.cuh"

namespace hc {
namespace {

constexpr int kPrepWarps = 8;
constexpr int kMaxHeadDim = 512;

// A key or value row's second place (PrepArgs::also).
__device__ __forceinline__ uint16_t* also_row(const PrepArgs& args, int kind, int head, int position, int d) {
    return (kind == 1 ? args.also.k : args.also.v) +
           (size_t(cache_plane(args.also.map, args.also_seq, args.also.kv_heads, head)) * args.also.capacity +
            cache_row(args.also.map, args.also_seq, position)) * d;
}

// The kernel for head_dim 64, 128, 256 and 512.  A warp stays with its heads and walks over tokens, so what to do, where
// from and where to, and the norm weights are worked out once; the next token's vectors are on their way while this one's
// are worked on.  What bounds it is its instructions, so a lane owns sixteen elements (8 m .. 8 m + 7 of each half, 16-byte
// accesses; head_dim 512 as in HeadLanes): a warp has two vectors of 256 at a time, and reduces, and takes the root and the
// addresses, once for both (8192 tokens of 32 x 256 with norms and rotation: 90 us with a vector a warp, a division by
// head_dim and a remainder per cached row, 64 without the prefetch into L2, now 55).  The bits are HeadLanes' and
// prepare_head's: a lane keeps the sums of two of their lanes apart until the last step of the butterfly.
// The launcher checks the alignment this needs and otherwise uses the general kernel below.
template <int D>
struct WideLanes {
    static constexpr bool kContiguous = D <= 256;
    static constexpr int kLanes = D / 16;
    static constexpr int kPerWarp = 32 / kLanes;
    // Where elements 4 u .. 4 u + 3 of a lane's half lie in it.
    __device__ static constexpr int at(int m, int u) { return kContiguous ? 8 * m + 4 * u : 4 * (m + u * kLanes); }
};
// A lane's elements as they come: [half][4 u ..].
template <int D, bool F32>
struct RawHead {
    uint4 x[2][F32 ? 2 : 1];
    __device__ __forceinline__ void load(const unsigned char* src, int m) {
        using WL = WideLanes<D>;
        #pragma unroll
        for (int h = 0; h < 2; ++h) {
            if constexpr (F32) {
                #pragma unroll
                for (int u = 0; u < 2; ++u) x[h][u] = *reinterpret_cast<const uint4*>(src + (h * (D / 2) + WL::at(m, u)) * 4);
            } else if constexpr (WL::kContiguous) {
                x[h][0] = *reinterpret_cast<const uint4*>(src + (h * (D / 2) + WL::at(m, 0)) * 2);
            } else {
                const uint2 a = *reinterpret_cast<const uint2*>(src + (h * (D / 2) + WL::at(m, 0)) * 2);
                const uint2 b = *reinterpret_cast<const uint2*>(src + (h * (D / 2) + WL::at(m, 1)) * 2);
                x[h][0] = make_uint4(a.x, a.y, b.x, b.y);
            }
        }
    }
    __device__ __forceinline__ void unpack(int h, float (&v)[8]) const {
        const uint32_t w[4] = {x[h][0].x, x[h][0].y, x[h][0].z, x[h][0].w};
        if constexpr (F32) {
            const uint32_t w2[4] = {x[h][1].x, x[h][1].y, x[h][1].z, x[h][1].w};
            #pragma unroll
            for (int i = 0; i < 4; ++i) { v[i] = __uint_as_float(w[i]); v[4 + i] = __uint_as_float(w2[i]); }
        } else {
            #pragma unroll
            for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
        }
    }
};
// Eight values of a half to a row of bf16.
template <int D>
__device__ __forceinline__ void store_half(uint16_t* row, int h, int m, const float (&v)[8]) {
    using WL = WideLanes<D>;
    const float a[4] = {v[0], v[1], v[2], v[3]}, b[4] = {v[4], v[5], v[6], v[7]};
    const uint2 pa = pack_bf16x4(a), pb = pack_bf16x4(b);
    uint16_t* at = row + h * (D / 2);
    if constexpr (WL::kContiguous) {
        *reinterpret_cast<uint4*>(at + WL::at(m, 0)) = make_uint4(pa.x, pa.y, pb.x, pb.y);
    } else {
        *reinterpret_cast<uint2*>(at + WL::at(m, 0)) = pa;
        *reinterpret_cast<uint2*>(at + WL::at(m, 1)) = pb;
    }
}

__device__ __forceinline__ void store8(void* dst, const float (&v)[8]) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}

// Thread blocks an SM holds.
constexpr int prep_blocks(bool fp32) { return fp32 ? 2 : 3; }

template <int D, bool F32>
__global__ void __launch_bounds__(kPrepWarps * 32, prep_blocks(F32))
prepare_heads_vec_kernel(const PrepArgs args, int total_heads, int prefetch) {
    using WL = WideLanes<D>;
    constexpr int kBytes = F32 ? 4 : 2;
    pdl_launch_dependents();
    const unsigned warp = blockIdx.x * kPrepWarps + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    const int sub = lane / WL::kLanes;
    const int m = lane % WL::kLanes;
    const bool any_norm = (args.job[0].norm | (args.n_jobs > 1 ? args.job[1].norm : 0) | (args.n_jobs > 2 ? args.job[2].norm : 0)) != 0;
    // Warps side by side take the heads of a token.
    const unsigned head_groups = unsigned(total_heads + WL::kPerWarp - 1) / WL::kPerWarp;
    const unsigned step = gridDim.x * kPrepWarps / head_groups;
    unsigned token = warp / head_groups;
    int head = int(warp - token * head_groups) * WL::kPerWarp + sub;
    const bool in_range = head < total_heads;
    if (!in_range) head = total_heads - 1;               // keeps the lane's loads legal; nothing is stored
    int job_index = 0;
    while (head >= args.job[job_index].heads) {
        head -= args.job[job_index].heads;
        ++job_index;
    }
    const PrepJob& job = args.job[job_index];
    const int norm = job.norm, kind = job.kind;
    const bool rope = job.rope != 0, cached = kind == 1 || kind == 2;
    const RowMap& map = args.cache.map;
    pdl_wait();
    if (token >= step || token >= unsigned(args.tokens)) return;
    float wl[8], wh[8];
    if (norm == 1) {
        RawHead<D, false> w;
        w.load(reinterpret_cast<const unsigned char*>(job.weight), m);
        w.unpack(0, wl);
        w.unpack(1, wh);
    }
    const size_t src_step = size_t(step) * size_t(job.token_stride) * kBytes;
    unsigned char* src = const_cast<unsigned char*>(static_cast<const unsigned char*>(job.src)) +
                         (size_t(token) * size_t(job.token_stride) + size_t(head) * job.head_stride) * kBytes;
    // Rows of a ring or of linear storage are counted along; other storage is asked for every row.
    const bool counted = cached && args.batched == 0 && map.pages == nullptr && map.world <= 1;
    uint16_t* dst = nullptr;
    size_t dst_step = 0;
    int row = 0, row_step = int(step);
    if (kind == 0) {
        dst = static_cast<uint16_t*>(job.dst) + (size_t(token) * job.heads + head) * D;
        dst_step = size_t(step) * job.heads * D;
    } else if (cached) {
        dst = kind == 1 ? args.cache.k : args.cache.v;
        if (counted) {
            dst += size_t(cache_plane(map, args.seq, args.cache.kv_heads, head)) * args.cache.capacity * D;
            row = args.first_position + int(token);
            if (map.ring > 0) {
                row %= map.ring;
                row_step %= map.ring;
            }
        }
    }
    RawHead<D, F32> now, ahead;
    const bool by32 = (reinterpret_cast<uintptr_t>(src) & 31) == 0;      // (of all vectors or none)
    now.load(src, m);
    for (;;) {
        const bool more = token + step < unsigned(args.tokens);
        if (more) ahead.load(src + src_step, m);
        if ((!F32 || prefetch) && token + 3 * step < unsigned(args.tokens)) {              // two further on their way into L2
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                asm volatile("prefetch.global.L2 [%0];" ::"l"(src + 3 * src_step + (h * (D / 2) + WL::at(m, 0)) * kBytes));
            }
        }
        const int position = args.batched ? args.meta.pos[token] : args.first_position + int(token);
        float c[8], s[8];
        if (rope) {
            const size_t table = size_t(min(position, args.table_positions - 1)) * (D / 2);
            #pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float4 cv = *reinterpret_cast<const float4*>(args.cos + table + WL::at(m, u));
                const float4 sv = *reinterpret_cast<const float4*>(args.sin + table + WL::at(m, u));
                c[4 * u] = cv.x; c[4 * u + 1] = cv.y; c[4 * u + 2] = cv.z; c[4 * u + 3] = cv.w;
                s[4 * u] = sv.x; s[4 * u + 1] = sv.y; s[4 * u + 2] = sv.z; s[4 * u + 3] = sv.w;
            }
        }
        // Where to: of fp32 rows while the loads are on their way (1000 x 16 x 256 in place 6.1 us behind the sums, so 5.8), of bf16
        // ones behind the sums (ahead of them they spill: 4000 x 64 x 256 56.3 us, so 53.4).
        uint16_t* to = dst;
        bool active = in_range;
        auto where_to = [&]() {
            if (counted) {
                to = dst + size_t(row) * D;
                row += row_step;
                if (map.ring > 0 && row >= map.ring) row -= map.ring;
            } else if (cached) {
                active = active && row_is_local(map, position);           // else another rank's tile
                const int seq = args.batched ? args.meta.seq[token] : args.seq;
                if (active) to = dst + (size_t(cache_plane(map, seq, args.cache.kv_heads, head)) * args.cache.capacity + cache_row(map, seq, position)) * D;
            }
        };
        if constexpr (F32) where_to();
        float lo[8], hi[8];
        now.unpack(0, lo);
        now.unpack(1, hi);
        if (any_norm) {                                  // warp-uniform
            float part[2] = {0.0f, 0.0f};
            constexpr int kParts = WL::kContiguous ? 2 : 1, kEach = 8 / kParts;
            #pragma unroll
            for (int p = 0; p < kParts; ++p) {
                #pragma unroll
                for (int i = 0; i < kEach; ++i) part[p] = __fmaf_rn(lo[kEach * p + i], lo[kEach * p + i], part[p]);
                #pragma unroll
                for (int i = 0; i < kEach; ++i) part[p] = __fmaf_rn(hi[kEach * p + i], hi[kEach * p + i], part[p]);
            }
            #pragma unroll
            for (int offset = WL::kLanes / 2; offset > 0; offset >>= 1) {
                #pragma unroll
                for (int p = 0; p < kParts; ++p) part[p] = __fadd_rn(part[p], __shfl_xor_sync(0xffffffffu, part[p], offset));
            }
            if (norm != 0) {
                // (Dividing by a power of two and multiplying by its inverse round alike.)
                const float mean = __fmul_rn(kParts == 2 ? __fadd_rn(part[0], part[1]) : part[0], 1.0f / float(D));
                const float inverse = __frsqrt_rn(__fadd_rn(mean, args.eps));
                #pragma unroll
                for (int i = 0; i < 8; ++i) {
                    lo[i] = __fmul_rn(lo[i], inverse);
                    hi[i] = __fmul_rn(hi[i], inverse);
                }
                if (norm == 1) {
                    #pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        lo[i] = __fmul_rn(lo[i], wl[i]);
                        hi[i] = __fmul_rn(hi[i], wh[i]);
                    }
                }
            }
        }
        if (rope) {
            #pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float a = lo[i], b = hi[i];
                lo[i] = __fmaf_rn(a, c[i], -__fmul_rn(b, s[i]));
                hi[i] = __fmaf_rn(b, c[i], __fmul_rn(a, s[i]));
            }
        }
        if constexpr (!F32) where_to();
        if (active) {
            if (kind == 3 && F32) {
                if (WL::kContiguous && by32) {               // (by halves of them 2000 x 16 x 256 take 12.5 us, so 8.4)
                    store8(src + WL::at(m, 0) * 4, lo);
                    store8(src + (D / 2 + WL::at(m, 0)) * 4, hi);
                } else {
                    #pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        *reinterpret_cast<float4*>(src + WL::at(m, u) * 4) = make_float4(lo[4 * u], lo[4 * u + 1], lo[4 * u + 2], lo[4 * u + 3]);
                        *reinterpret_cast<float4*>(src + (D / 2 + WL::at(m, u)) * 4) = make_float4(hi[4 * u], hi[4 * u + 1], hi[4 * u + 2], hi[4 * u + 3]);
                    }
                }
            } else {
                if (kind == 3) to = reinterpret_cast<uint16_t*>(src);
                store_half<D>(to, 0, m, lo);
                store_half<D>(to, 1, m, hi);
                if (cached && args.also.capacity > 0 && position >= args.also_from) {
                    uint16_t* also = also_row(args, kind, head, position, D);
                    store_half<D>(also, 0, m, lo);
                    store_half<D>(also, 1, m, hi);
                }
            }
        }
        if (!more) break;
        now = ahead;
        token += step;
        src += src_step;
        if (kind == 0) dst += dst_step;
    }
}

__device__ __forceinline__ void store_io4(void* base, size_t index, int dtype, const float (&v)[4]) {
    if (dtype == 0) {
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(base) + index) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
        *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(base) + index) = pack_bf16x4(v);
    }
}

// The same where every warp has one token: what counts there is the time of one vector, so a lane has half as many elements
// (HeadLanes; head_dim 512 as many) and nothing is prepared for a walk.  All of the job is read ahead of the wait, and the loop,
// which goes round once, keeps the norm weights' load ahead of the sum that is worked out meanwhile (without it a row of 2 x 512
// appended behind another took 1.8 us, now 1.55; 8 x 64 1.56 and 1.4; one wave of 64 x 256 3.0, by the kernel above, and 2.25).
template <int D>
__global__ void __launch_bounds__(kPrepWarps * 32)
prepare_heads_few_kernel(const PrepArgs args, int total_heads) {
    using HL = HeadLanes<D>;
    pdl_launch_dependents();
    const unsigned warp = blockIdx.x * kPrepWarps + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    const int sub = lane / HL::kLanes;
    const int m = lane % HL::kLanes;
    const bool any_norm = (args.job[0].norm | (args.n_jobs > 1 ? args.job[1].norm : 0) | (args.n_jobs > 2 ? args.job[2].norm : 0)) != 0;
    // Warps side by side take the heads of a token.
    const unsigned head_groups = unsigned(total_heads + HL::kPerWarp - 1) / HL::kPerWarp;
    const unsigned step = gridDim.x * kPrepWarps / head_groups;
    const unsigned first_token = warp / head_groups;
    int head = int(warp - first_token * head_groups) * HL::kPerWarp + sub;
    const bool in_range = head < total_heads;
    if (!in_range) head = total_heads - 1;               // keeps the lane's loads legal; nothing is stored
    int job_index = 0;
    while (head >= args.job[job_index].heads) {
        head -= args.job[job_index].heads;
        ++job_index;
    }
    const PrepJob& job = args.job[job_index];
    const int norm = job.norm, kind = job.kind, dtype = job.src_dtype, heads = job.heads;
    const bool rope = job.rope != 0;
    const void* src = job.src;
    const long long token_stride = job.token_stride;
    const size_t head_offset = size_t(head) * job.head_stride;
    void* dst = kind == 1 ? args.cache.k : kind == 2 ? args.cache.v : job.dst;
    const uint16_t* weight = job.weight;
    pdl_wait();
    float wl[HL::kElems], wh[HL::kElems];
    if (first_token >= step || first_token >= unsigned(args.tokens)) return;
    if (norm == 1) load_head<D>(weight, 0, 1, m, wl, wh);
    for (unsigned token = first_token; token < unsigned(args.tokens); token += step) {
        const int position = args.batched ? args.meta.pos[token] : args.first_position + int(token);
        const size_t src_base = size_t(token) * size_t(token_stride) + head_offset;
        float lo[HL::kElems], hi[HL::kElems], c[HL::kElems], s[HL::kElems];
        load_head<D>(src, src_base, dtype, m, lo, hi);
        if (rope) {
            const int table_row = min(position, args.table_positions - 1);
            load_rotation<D>(args.cos + size_t(table_row) * (D / 2), args.sin + size_t(table_row) * (D / 2), m, c, s);
        }
        size_t base = src_base;
        bool active = in_range;
        if (kind == 0) {
            base = (size_t(token) * heads + head) * D;
        } else if (kind != 3) {
            active = active && row_is_local(args.cache.map, position);           // else another rank's tile
            const int seq = args.batched ? args.meta.seq[token] : args.seq;
            if (active) {
                base = (size_t(cache_plane(args.cache.map, seq, args.cache.kv_heads, head)) * args.cache.capacity +
                        cache_row(args.cache.map, seq, position)) * D;
            }
        }
        prepare_head<D>(lo, hi, norm, wl, wh, args.eps, rope, c, s, any_norm);
        if (!active) continue;
        #pragma unroll
        for (int u = 0; u < HL::kVecs; ++u) {
            const float a[4] = {lo[4 * u], lo[4 * u + 1], lo[4 * u + 2], lo[4 * u + 3]};
            const float b[4] = {hi[4 * u], hi[4 * u + 1], hi[4 * u + 2], hi[4 * u + 3]};
            const size_t at = base + 4 * (m + u * HL::kLanes);
            if (kind == 3 && (D == 512 || dtype == HC_F32)) {
                store_io4(dst, at, dtype, a);
                store_io4(dst, at + D / 2, dtype, b);
            } else {
                *reinterpret_cast<uint2*>(static_cast<uint16_t*>(dst) + at) = pack_bf16x4(a);
                *reinterpret_cast<uint2*>(static_cast<uint16_t*>(dst) + at + D / 2) = pack_bf16x4(b);
            }
        }
    }
}

// The general kernel: any even head_dim up to 512, any alignment.  One warp per head vector, staged
// in shared memory.
__global__ void __launch_bounds__(kPrepWarps * 32)
prepare_heads_kernel(const PrepArgs args) {
    __shared__ float stage[kPrepWarps][kMaxHeadDim];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int d = args.head_dim;
    const int half = d >> 1;

    int total_heads = 0;
    for (int j = 0; j < args.n_jobs; ++j) total_heads += args.job[j].heads;
    // Warps stride over the (token, head) vectors of the call.
    // 32-bit indices: a launch covers at most 32768 tokens x a few hundred heads.
    const unsigned vectors = unsigned(args.tokens) * unsigned(total_heads);
    const unsigned stride = gridDim.x * kPrepWarps;
    for (unsigned vec = blockIdx.x * kPrepWarps + warp; vec < vectors; vec += stride) {
    const int token = int(vec / unsigned(total_heads));
    const int slot = int(vec - unsigned(token) * unsigned(total_heads));
    int job_index = 0, head = slot;
    while (head >= args.job[job_index].heads) {
        head -= args.job[job_index].heads;
        ++job_index;
    }
    const PrepJob& job = args.job[job_index];

    const int position = args.batched ? args.meta.pos[token] : args.first_position + token;
    const int seq = args.batched ? args.meta.seq[token] : args.seq;
    if (job.kind == 1 || job.kind == 2) {
        if (!row_is_local(args.cache.map, position)) continue;   // another rank owns this key tile
    }

    const size_t src_base = size_t(token) * size_t(job.token_stride) + size_t(head) * job.head_stride;
    const bool rotate = job.rope != 0;
    const int table_row = position < args.table_positions ? position : args.table_positions - 1;
    // Destination of this head vector.
    uint16_t *dst16 = nullptr, *also = nullptr;
    if (job.kind == 0) {
        dst16 = reinterpret_cast<uint16_t*>(job.dst) + (size_t(token) * job.heads + head) * d;
    } else if (job.kind == 1 || job.kind == 2) {
        const int row = cache_row(args.cache.map, seq, position);
        uint16_t* base = job.kind == 1 ? args.cache.k : args.cache.v;
        dst16 = base + (size_t(cache_plane(args.cache.map, seq, args.cache.kv_heads, head)) * args.cache.capacity + row) * d;
        if (args.also.capacity > 0 && position >= args.also_from) also = also_row(args, job.kind, head, position, d);
    }

    // Stage the vector in shared memory.
    __syncwarp();                                  // the staging row is reused
    float* x = stage[warp];
    float sum = 0.0f;
    for (int i = lane; i < d; i += 32) {
        const float value = load_io(job.src, src_base + i, job.src_dtype);
        x[i] = value;
        sum = __fmaf_rn(value, value, sum);
    }
    if (job.norm != 0) {
        #pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) {
            sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, offset));
        }
        const float inverse = __frsqrt_rn(__fadd_rn(__fdiv_rn(sum, float(d)), args.eps));
        for (int i = lane; i < d; i += 32) {
            float value = __fmul_rn(x[i], inverse);
            if (job.norm == 1) value = __fmul_rn(value, bf16_bits_to_float(job.weight[i]));
            x[i] = value;
        }
    }
    __syncwarp();
    for (int i = lane; i < half; i += 32) {
        float x1 = x[i], x2 = x[half + i];
        if (rotate) {
            const float c = args.cos[size_t(table_row) * half + i];
            const float s = args.sin[size_t(table_row) * half + i];
            const float r1 = __fmaf_rn(x1, c, -__fmul_rn(x2, s));
            const float r2 = __fmaf_rn(x2, c, __fmul_rn(x1, s));
            x1 = r1;
            x2 = r2;
        }
        if (job.kind == 3) {
            store_io(job.dst, src_base + i, job.src_dtype, x1);
            store_io(job.dst, src_base + half + i, job.src_dtype, x2);
        } else {
            dst16[i] = float_to_bf16_bits(x1);
            dst16[half + i] = float_to_bf16_bits(x2);
            if (also != nullptr) {
                also[i] = dst16[i];
                also[half + i] = dst16[half + i];
            }
        }
    }
    }
}

// Rows [first, end) of one sequence from one storage to another, and zeros to the values of [clear, clear_end) there, a thread
// per 16 bytes (a row is 2 head_dim bytes, a multiple of 16).
__global__ void __launch_bounds__(256)
copy_rows_kernel(const CacheView from, int from_seq, const CacheView to, int first, int end, int clear, int clear_end, int pieces) {
    pdl_launch_dependents();
    pdl_wait();
    const int heads = from.kv_heads, copied = end - first;
    const unsigned total = unsigned(copied + clear_end - clear) * unsigned(heads) * unsigned(pieces);
    for (unsigned i = blockIdx.x * 256 + threadIdx.x; i < total; i += gridDim.x * 256) {
        const unsigned row = i / unsigned(pieces), piece = i - row * unsigned(pieces);
        const int at = int(row / unsigned(heads)), head = int(row % unsigned(heads));
        const int position = at < copied ? first + at : clear + (at - copied);
        const size_t dst = (size_t(cache_plane(to.map, 0, heads, head)) * to.capacity + cache_row(to.map, 0, position)) * pieces + piece;
        if (at >= copied) {
            reinterpret_cast<uint4*>(to.v)[dst] = make_uint4(0, 0, 0, 0);
            continue;
        }
        const size_t src = (size_t(cache_plane(from.map, from_seq, heads, head)) * from.capacity + cache_row(from.map, from_seq, position)) * pieces + piece;
        const uint4 k = reinterpret_cast<const uint4*>(from.k)[src], v = reinterpret_cast<const uint4*>(from.v)[src];
        reinterpret_cast<uint4*>(to.k)[dst] = k;
        reinterpret_cast<uint4*>(to.v)[dst] = v;
    }
}

// A multiple of four floats, either side in pinned host memory.
__global__ void __launch_bounds__(256) copy_floats_kernel(float4* dst, const float4* src, int count) {
    pdl_launch_dependents();
    pdl_wait();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < count) dst[i] = src[i];
}

// RMSNorm of whole rows (the layer's input norm): out = x * rsqrt(mean(x^2) + eps) * scale.  One block
// per token; replaces rms_norm and rms_norm_batch (Sources/HydraMetal/Shaders/attention.metal:9-43,
// batch.metal:184-218).  The output may be bf16, ready to be the A operand of hc_linear.
// Rows whose width is a multiple of 4 (and at most 4096) are read once, four elements per load, and
// kept in registers between the sum and the scaling: all of a thread's loads are in flight together,
// where an element-by-element loop with the dtype looked up per element paid one memory round trip
// after the other (12 us for one 2880-wide row).  The sum's order is fixed by the width alone.
constexpr int kNormVecs = 4;      // float4 per thread held in registers: 256 threads x 16 values

__device__ __forceinline__ float4 load_vec4(const void* p, size_t index, int dtype) {
    if (dtype == HC_F32) return *reinterpret_cast<const float4*>(static_cast<const float*>(p) + index);
    const uint2 bits = *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(p) + index);
    return make_float4(__uint_as_float(bits.x << 16), __uint_as_float(bits.x & 0xffff0000u),
                       __uint_as_float(bits.y << 16), __uint_as_float(bits.y & 0xffff0000u));
}

__global__ void __launch_bounds__(256)
rms_norm_rows_kernel(const void* __restrict__ x, const uint16_t* __restrict__ scale, void* __restrict__ out, int width,
                     float eps, int x_dtype, int out_dtype, int vectors) {
    __shared__ float warp_sum[8];
    __shared__ float inverse;
    pdl_launch_dependents();
    pdl_wait();
    const size_t base = size_t(blockIdx.x) * width;
    float partial = 0.0f;
    float4 held[kNormVecs];
    if (vectors) {
        #pragma unroll
        for (int u = 0; u < kNormVecs; ++u) {
            const int i = (threadIdx.x + u * 256) * 4;
            held[u] = i < width ? load_vec4(x, base + i, x_dtype) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        #pragma unroll
        for (int u = 0; u < kNormVecs; ++u) {
            partial = __fmaf_rn(held[u].x, held[u].x, partial);
            partial = __fmaf_rn(held[u].y, held[u].y, partial);
            partial = __fmaf_rn(held[u].z, held[u].z, partial);
            partial = __fmaf_rn(held[u].w, held[u].w, partial);
        }
    } else {
        for (int i = threadIdx.x; i < width; i += blockDim.x) {
            const float v = load_io(x, base + i, x_dtype);
            partial = __fmaf_rn(v, v, partial);
        }
    }
    #pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) partial += __shfl_xor_sync(0xffffffffu, partial, offset);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = partial;
    __syncthreads();
    if (threadIdx.x == 0) {
        float total = 0.0f;
        for (int w = 0; w < int(blockDim.x >> 5); ++w) total += warp_sum[w];
        inverse = rsqrtf(total / float(width) + eps);
    }
    __syncthreads();
    const float inv = inverse;
    if (vectors) {
        #pragma unroll
        for (int u = 0; u < kNormVecs; ++u) {
            const int i = (threadIdx.x + u * 256) * 4;
            if (i >= width) continue;
            float w[4] = {1.0f, 1.0f, 1.0f, 1.0f};
            if (scale != nullptr) {
                const uint2 bits = *reinterpret_cast<const uint2*>(scale + i);
                w[0] = __uint_as_float(bits.x << 16);
                w[1] = __uint_as_float(bits.x & 0xffff0000u);
                w[2] = __uint_as_float(bits.y << 16);
                w[3] = __uint_as_float(bits.y & 0xffff0000u);
            }
            const float r0 = __fmul_rn(__fmul_rn(held[u].x, inv), w[0]), r1 = __fmul_rn(__fmul_rn(held[u].y, inv), w[1]);
            const float r2 = __fmul_rn(__fmul_rn(held[u].z, inv), w[2]), r3 = __fmul_rn(__fmul_rn(held[u].w, inv), w[3]);
            if (out_dtype == HC_F32) {
                *reinterpret_cast<float4*>(static_cast<float*>(out) + base + i) = make_float4(r0, r1, r2, r3);
            } else {
                uint2 packed;
                packed.x = uint32_t(float_to_bf16_bits(r0)) | (uint32_t(float_to_bf16_bits(r1)) << 16);
                packed.y = uint32_t(float_to_bf16_bits(r2)) | (uint32_t(float_to_bf16_bits(r3)) << 16);
                *reinterpret_cast<uint2*>(static_cast<uint16_t*>(out) + base + i) = packed;
            }
        }
        return;
    }
    for (int i = threadIdx.x; i < width; i += blockDim.x) {
        const float v = load_io(x, base + i, x_dtype);
        const float w = scale != nullptr ? bf16_bits_to_float(scale[i]) : 1.0f;
        store_io(out, base + i, out_dtype, __fmul_rn(__fmul_rn(v, inv), w));
    }
}

__global__ void split_query_gate_kernel(const void* combined, void* query, void* gate, size_t count,
                                        int d, int dtype) {
    // count = tokens * heads * d; element e = (token*heads + head) * d + i
    const size_t e = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= count) return;
    const size_t vec = e / d;
    const int i = int(e % d);
    store_io(query, e, dtype, load_io(combined, vec * 2 * d + i, dtype));
    store_io(gate, e, dtype, load_io(combined, vec * 2 * d + d + i, dtype));
}

__global__ void output_gate_kernel(void* output, const void* gate, size_t count, int dtype) {
    const size_t e = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= count) return;
    const float value = load_io(output, e, dtype);
    store_io(output, e, dtype, __fmul_rn(value, sigmoid_gate(load_io(gate, e, dtype))));
}

}  // namespace

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

hc_status launch_prepare(hc_context* ctx, const PrepArgs& args, cudaStream_t stream) {
    int total_heads = 0;
    for (int j = 0; j < args.n_jobs; ++j) total_heads += args.job[j].heads;
    if (total_heads == 0 || args.tokens == 0) return HC_OK;
    const long long vectors = (long long)args.tokens * total_heads;
    const int d = args.head_dim;
    const long long cap = (long long)std::max(ctx->sm_count, 1) * 16;
    // The vector kernel needs 16-byte aligned rows everywhere it touches.
    bool vector_ok = d == 64 || d == 128 || d == 256 || d == 512;
    for (int j = 0; j < args.n_jobs && vector_ok; ++j) {
        const PrepJob& job = args.job[j];
        if (job.heads == 0) continue;
        vector_ok = aligned16(job.src) && job.token_stride % 8 == 0 && job.head_stride % 8 == 0 &&
                    (job.norm != 1 || aligned16(job.weight)) && job.src_dtype == args.job[0].src_dtype &&
                    ((job.kind != 0 && job.kind != 3) || aligned16(job.dst));
    }
    const bool fp32 = args.job[0].src_dtype == HC_F32;
    const bool large = size_t(vectors) * d * (fp32 ? 4 : 2) > (size_t(64) << 20);      // does not stay in L2
    auto groups_of = [&](int per_warp) -> long long { return (total_heads + per_warp - 1) / per_warp; };     // of a token
    const long long sms = std::max(ctx->sm_count, 1);
    const int few_blocks = d == 512 ? 3 : 4;             // thread blocks of the few kernel an SM holds
    const long long few = groups_of(std::max(256 / d, 1));
    // What one wave holds goes a token a warp, at 16 x 64 up to 1184 tokens (1000 of them 2.4 us, by the other kernel 2.9; 2000 3.7
    // and 3.4), and so do, in a walk, fp32 rows of 512 that come from and go to DRAM (8000 x 16 59 us, by the other 68).
    if (vector_ok && args.also.capacity == 0 && (args.tokens * few <= sms * few_blocks * kPrepWarps || (fp32 && d == 512 && large))) {
        const int grid = int((std::max(std::min(args.tokens * few, cap * kPrepWarps), few) + kPrepWarps - 1) / kPrepWarps);
        auto kernel = d == 64 ? prepare_heads_few_kernel<64> : d == 128 ? prepare_heads_few_kernel<128>
                    : d == 256 ? prepare_heads_few_kernel<256> : prepare_heads_few_kernel<512>;
        launch_pdl(kernel, grid, kPrepWarps * 32, 0, stream, args, total_heads);
    } else if (vector_ok) {
        const long long groups = groups_of(512 / d);
        // (A warp stays with its heads, so there are never fewer warps than a token has groups of them.)
        const int grid = int((std::max(std::min(args.tokens * groups, sms * prep_blocks(fp32) * kPrepWarps), groups) + kPrepWarps - 1) / kPrepWarps);
        // Prefetched bf16 rows are 64 us -> 55 (above).  Of fp32 rows a warp has enough on its way without (appends of 8000 x 64 x 256
        // 146 us with, 130 without, of 1000 x 64 x 256 15.7 and 14.7; in place 8000 x 16 x 256 47.5 and 43.2), but for queries and
        // rows in place that L2 keeps (2000 x 16 x 256 in place 12.4 with, 13.4 without; a prompt of 777 gated tokens 58.7 and 59).
        const int prefetch = !fp32 || (args.job[0].kind != 1 && !large) ? 1 : 0;
        auto kernel = d == 64 ? (fp32 ? prepare_heads_vec_kernel<64, true> : prepare_heads_vec_kernel<64, false>)
                    : d == 128 ? (fp32 ? prepare_heads_vec_kernel<128, true> : prepare_heads_vec_kernel<128, false>)
                    : d == 256 ? (fp32 ? prepare_heads_vec_kernel<256, true> : prepare_heads_vec_kernel<256, false>)
                               : (fp32 ? prepare_heads_vec_kernel<512, true> : prepare_heads_vec_kernel<512, false>);
        launch_pdl(kernel, grid, kPrepWarps * 32, 0, stream, args, total_heads, prefetch);
    } else {
        const long long wanted = (vectors + kPrepWarps - 1) / kPrepWarps;
        const int grid = int(std::min<long long>(wanted, cap));
        launch_pdl(prepare_heads_kernel, grid, kPrepWarps * 32, 0, stream, args);
    }
    ctx->launches += 1;
    return check_cuda(cudaGetLastError(), "prepare_heads_kernel launch");
}

hc_status launch_copy_rows(hc_context* ctx, const CacheView& from, int from_seq, const CacheView& to, int first, int end, int call_end,
                           int d, cudaStream_t stream) {
    const int clear_end = (call_end + kTileKeys - 1) / kTileKeys * kTileKeys;
    const long long total = (long long)(end - first + clear_end - call_end) * from.kv_heads * (d / 8);
    if (total == 0) return HC_OK;
    const int grid = int(std::min<long long>((total + 255) / 256, (long long)std::max(ctx->sm_count, 1) * 8));
    launch_pdl(copy_rows_kernel, grid, 256, 0, stream, from, from_seq, to, first, end, call_end, clear_end, d / 8);
    ctx->launches += 1;
    return check_cuda(cudaGetLastError(), "copy_rows_kernel launch");
}

hc_status launch_copy_floats(hc_context* ctx, float* dst, const float* src, size_t count, cudaStream_t stream) {
    const int vectors = int(count / 4);
    launch_pdl(copy_floats_kernel, (vectors + 255) / 256, 256, 0, stream, reinterpret_cast<float4*>(dst), reinterpret_cast<const float4*>(src), vectors);
    ctx->launches += 1;
    return check_cuda(cudaGetLastError(), "copy_floats_kernel launch");
}

hc_status launch_rms_norm_rows(hc_context* ctx, const void* x, const uint16_t* scale, void* out, int tokens, int width,
                               float eps, int x_dtype, int out_dtype, cudaStream_t stream) {
    if (tokens <= 0) return HC_OK;
    // Four elements per load where every row starts on a 16-byte boundary in every buffer it touches.
    const bool vectors = width % 4 == 0 && width <= 256 * 4 * 4 && aligned16(x) && aligned16(out) &&
                         (scale == nullptr || (reinterpret_cast<uintptr_t>(scale) & 7u) == 0) &&
                         (width % 8 == 0 || (x_dtype == HC_F32 && out_dtype == HC_F32));
    launch_pdl(rms_norm_rows_kernel, dim3(unsigned(tokens)), dim3(256), 0, stream, x, scale, out, width, eps, x_dtype, out_dtype,
               vectors ? 1 : 0);
    ctx->launches += 1;
    return check_cuda(cudaGetLastError(), "rms_norm_rows_kernel launch");
}

hc_status launch_split_query_gate(hc_context* ctx, const void* combined, void* query, void* gate,
                                  int tokens, int heads, int d, int dtype, cudaStream_t stream) {
    const size_t count = size_t(tokens) * heads * d;
    if (count == 0) return HC_OK;
    split_query_gate_kernel<<<unsigned((count + 255) / 256), 256, 0, stream>>>(combined, query, gate,
                                                                               count, d, dtype);
    ctx->launches += 1;
    return check_cuda(cudaGetLastError(), "split_query_gate_kernel launch");
}

hc_status launch_output_gate(hc_context* ctx, void* output, const void* gate, size_t count,
                             int dtype, cudaStream_t stream) {
    if (count == 0) return HC_OK;
    output_gate_kernel<<<unsigned((count + 255) / 256), 256, 0, stream>>>(output, gate, count, dtype);
    ctx->launches += 1;
    return check_cuda(cudaGetLastError(), "output_gate_kernel launch");
}

}  // namespace hc
