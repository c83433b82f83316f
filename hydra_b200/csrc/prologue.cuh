// prologue.cuh — what happens to one head vector of q, k or v before attention (per-head RMSNorm,
// half-split rotation, rounding to bf16), for the head dims whose vectors are spread over the lanes
// of a warp with 8- and 16-byte accesses.  Shared by the prologue kernel and the decode kernel, so a
// token gets the same bits whichever prepares it.
#pragma once

#include "common.cuh"

namespace hc {
namespace {

// Four consecutive elements of an activation row as fp32 (8-byte load for bf16, 16-byte for fp32).
__device__ __forceinline__ void load_io4(const void* base, size_t index, int dtype, float (&out)[4]) {
    if (dtype == 0) {
        const float4 v = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + index);
        out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
    } else {
        const uint2 v = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(base) + index);
        out[0] = bf16_bits_to_float(uint16_t(v.x & 0xffffu));
        out[1] = bf16_bits_to_float(uint16_t(v.x >> 16));
        out[2] = bf16_bits_to_float(uint16_t(v.y & 0xffffu));
        out[3] = bf16_bits_to_float(uint16_t(v.y >> 16));
    }
}
__device__ __forceinline__ uint2 pack_bf16x4(const float (&v)[4]) {
    uint2 r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r.x) : "f"(v[1]), "f"(v[0]));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r.y) : "f"(v[3]), "f"(v[2]));
    return r;
}

// How a D-element vector lies over lanes: kLanes lanes per vector (a warp holds 32 / kLanes vectors at a
// time), lane m owning kVecs groups of four elements of EACH half, group u at element 4 (m + u kLanes),
// which keeps both members of every rotation pair (i, i + D/2) in one lane.
template <int D>
struct HeadLanes {
    static constexpr int kLanes = D <= 256 ? D / 8 : 32;
    static constexpr int kVecs = D / (8 * kLanes);
    static constexpr int kPerWarp = 32 / kLanes;
    static constexpr int kElems = 4 * kVecs;            // per half
};

template <int D>
__device__ __forceinline__ void load_head(const void* src, size_t base, int dtype, int m,
                                          float (&lo)[HeadLanes<D>::kElems], float (&hi)[HeadLanes<D>::kElems]) {
    #pragma unroll
    for (int u = 0; u < HeadLanes<D>::kVecs; ++u) {
        float a[4], b[4];
        load_io4(src, base + 4 * (m + u * HeadLanes<D>::kLanes), dtype, a);
        load_io4(src, base + D / 2 + 4 * (m + u * HeadLanes<D>::kLanes), dtype, b);
        #pragma unroll
        for (int j = 0; j < 4; ++j) { lo[4 * u + j] = a[j]; hi[4 * u + j] = b[j]; }
    }
}
template <int D>
__device__ __forceinline__ void load_rotation(const float* cos_row, const float* sin_row, int m,
                                              float (&c)[HeadLanes<D>::kElems], float (&s)[HeadLanes<D>::kElems]) {
    #pragma unroll
    for (int u = 0; u < HeadLanes<D>::kVecs; ++u) {
        const float4 cv = *reinterpret_cast<const float4*>(cos_row + 4 * (m + u * HeadLanes<D>::kLanes));
        const float4 sv = *reinterpret_cast<const float4*>(sin_row + 4 * (m + u * HeadLanes<D>::kLanes));
        c[4 * u] = cv.x; c[4 * u + 1] = cv.y; c[4 * u + 2] = cv.z; c[4 * u + 3] = cv.w;
        s[4 * u] = sv.x; s[4 * u + 1] = sv.y; s[4 * u + 2] = sv.z; s[4 * u + 3] = sv.w;
    }
}

// In place: the norm (0 none, 1 with `weight`, 2 weightless), then the rotation when `rope`.  The lanes of
// a warp may hold vectors with different settings: the shuffles are executed by all of them.
// wl, wh: the weight's elements of this lane (norm 1).
template <int D>
__device__ __forceinline__ void prepare_head(float (&lo)[HeadLanes<D>::kElems], float (&hi)[HeadLanes<D>::kElems], int norm,
                                             const float (&wl)[HeadLanes<D>::kElems], const float (&wh)[HeadLanes<D>::kElems],
                                             float eps, bool rope,
                                             const float (&c)[HeadLanes<D>::kElems], const float (&s)[HeadLanes<D>::kElems],
                                             bool any_norm) {
    constexpr int kElems = HeadLanes<D>::kElems, kLanes = HeadLanes<D>::kLanes;
    if (any_norm) {                                  // warp-uniform
        float sum = 0.0f;
        #pragma unroll
        for (int j = 0; j < kElems; ++j) sum = __fmaf_rn(lo[j], lo[j], sum);
        #pragma unroll
        for (int j = 0; j < kElems; ++j) sum = __fmaf_rn(hi[j], hi[j], sum);
        #pragma unroll
        for (int offset = kLanes / 2; offset > 0; offset >>= 1) {
            sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, offset));
        }
        if (norm != 0) {
            const float inverse = __frsqrt_rn(__fadd_rn(__fdiv_rn(sum, float(D)), eps));
            #pragma unroll
            for (int j = 0; j < kElems; ++j) { lo[j] = __fmul_rn(lo[j], inverse); hi[j] = __fmul_rn(hi[j], inverse); }
            if (norm == 1) {
                #pragma unroll
                for (int j = 0; j < kElems; ++j) { lo[j] = __fmul_rn(lo[j], wl[j]); hi[j] = __fmul_rn(hi[j], wh[j]); }
            }
        }
    }
    if (rope) {
        #pragma unroll
        for (int j = 0; j < kElems; ++j) {
            const float a = lo[j], b = hi[j];
            lo[j] = __fmaf_rn(a, c[j], -__fmul_rn(b, s[j]));
            hi[j] = __fmaf_rn(b, c[j], __fmul_rn(a, s[j]));
        }
    }
}

}  // namespace
}  // namespace hc
