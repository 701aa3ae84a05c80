// RMS norm + activation quantisation, one pass per token row.
//
// The integer matrix kernels multiply weights by activations quantised exactly as the reference
// CPU engine quantises them, so that the block dot products are the same integers:
//   quantize_q8_0 (src/quant.cpp:115-142): d = amax/127 (f32), q = rint(x * (1/d)), stored scale = half(d)
//   quantize_q8_k (src/quant.cpp:146-194): inverse = -127/x_extreme (first of equal magnitudes),
//                                          d = 1/inverse, q = min(127, rint(inverse*x)), sums of 16
//   rms_norm      (src/model.cpp:87-97):   squares in f32, sum in f64, y = x * (1/sqrt(mean+eps)) * w
// All divisions and roots are IEEE-rounded; products are separate roundings (no contraction).
//
// Latency-bound: a few tokens' rows are a few kilobytes each. A thread owns eight consecutive values in registers, so four
// lanes hold a Q8_0 block and a warp a Q8_K super-block and nothing goes through shared memory; a row is split over CTAs
// of 2048 values, each of which sums the whole row for itself when there is a norm. Measured, one multiply's preparation at
// 9 tokens: the 9-token step of the 7B shape 6.32 -> 6.08 ms against one CTA per row with the row in shared
// memory, the 512-token prompt of the 0.6B shape 7.40 -> 7.16 ms.
#include "kernels.h"
#include "pdl.cuh"
#include "rowops.cuh"

namespace bk {
namespace {

constexpr uint32_t kThreads = 256, kSegment = kThreads * 8;

__global__ void __launch_bounds__(kThreads) norm_quant_kernel(const float* __restrict__ x, uint32_t ldx, const float* __restrict__ weight,
                                                              float eps, uint32_t cols, DevActMut act, int want0, int wantk) {
    __shared__ double red[32];
    wait_for_previous();
    release_next();
    const uint32_t t = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const float* xr = x + size_t(t) * ldx;
    const float scale = weight != nullptr ? cta_rms_scale(xr, cols, eps, red) : 1.0f;
    for (uint32_t i0 = blockIdx.y * kSegment; i0 < cols; i0 += gridDim.y * kSegment) {
        const uint32_t i = i0 + tid * 8;
        const bool mine = i < cols;  // whole blocks: a row length is a multiple of 32 (256 where Q8_K is wanted)
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = 0.0f;
        if (mine) {
            const float4 a = *reinterpret_cast<const float4*>(xr + i), b = *reinterpret_cast<const float4*>(xr + i + 4);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
            if (weight != nullptr) {
                const float4 wa = *reinterpret_cast<const float4*>(weight + i), wb = *reinterpret_cast<const float4*>(weight + i + 4);
                const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = __fmul_rn(__fmul_rn(v[k], scale), w[k]);
            }
            if (act.f32 != nullptr) {
                float4* o = reinterpret_cast<float4*>(act.f32 + size_t(t) * cols + i);
                o[0] = make_float4(v[0], v[1], v[2], v[3]);
                o[1] = make_float4(v[4], v[5], v[6], v[7]);
            }
        }
        if (want0) {  // four lanes per block of 32
            float d;
            int sum;
            const uint2 packed = quad_quantize_q8_0(v, d, sum);
            if (mine) {
                *reinterpret_cast<uint2*>(act.q0 + size_t(t) * cols + i) = packed;
                if ((lane & 3) == 0) {
                    act.d0[size_t(t) * (cols / 32) + i / 32] = d;
                    act.s0[size_t(t) * (cols / 32) + i / 32] = sum;
                }
            }
        }
        if (wantk && i0 + (tid & ~31u) * 8 < cols) {  // a warp per super-block of 256
            warp_quantize_q8_k(v, act.qk + size_t(t) * cols + i, act.dk + size_t(t) * (cols / 256) + i / 256, act.bs + size_t(t) * (cols / 16) + i / 16);
        }
    }
}

}  // namespace

void launch_norm_quant(const float* x, uint32_t ldx, const float* weight, float eps, uint32_t n, uint32_t cols,
                       const DevActMut& act, bool want0, bool wantk, cudaStream_t s) {
    // x may be act.f32: then one CTA takes the whole row, so that nobody still sums what another has overwritten
    const uint32_t segments = x == act.f32 ? 1u : (cols + kSegment - 1) / kSegment;
    launch_dependent(norm_quant_kernel, dim3(n, segments), dim3(kThreads), 0, s, x, ldx, weight, eps, cols, act, want0 ? 1 : 0, wantk ? 1 : 0);
}

}  // namespace bk
