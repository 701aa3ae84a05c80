// Log-probability of the token that follows each row of logits: Engine::log_likelihood's inner loop
// (src/engine.cpp:10-33) on the device, so that scoring a text returns eight bytes a token instead of a
// vocabulary-sized row that the host then walks three times.
//
// Bound by the rows' trip through L2 and the f64 exps. A row (0.1-1 MB) is spread over a cluster of eight CTAs which
// exchange its maximum and its sum through distributed shared memory: one launch for up to 64 rows, two passes over a row
// of which the second hits L2. Measured on B200 (333 tokens, vocabulary 151 936, Q8_0 0.6B shape): the whole call 146 ms
// with the host's softmax over copied rows, 8.9 ms with this kernel and the layers in prompt-sized batches.
#include <cooperative_groups.h>

#include "kernels.h"

namespace bk {
namespace {

constexpr uint32_t kRowCtas = 8, kRowThreads = 256;

__global__ void __cluster_dims__(kRowCtas, 1, 1) __launch_bounds__(kRowThreads)
    row_logp_kernel(const float* __restrict__ logits, uint32_t vocab, const int32_t* __restrict__ targets, double* __restrict__ out) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ float warp_mx[kRowThreads / 32];
    __shared__ double warp_total[kRowThreads / 32];
    __shared__ float cta_mx;
    __shared__ double cta_total;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = blockIdx.x, row = blockIdx.y;
    const float* x = logits + size_t(row) * vocab;
    float mx = -INFINITY;
    for (uint32_t i = rank * kRowThreads + tid; i < vocab; i += kRowCtas * kRowThreads) mx = fmaxf(mx, x[i]);
    mx = warp_max(mx);
    if (lane == 0) warp_mx[warp] = mx;
    __syncthreads();
    if (tid == 0) {
        for (uint32_t w = 1; w < kRowThreads / 32; ++w) mx = fmaxf(mx, warp_mx[w]);
        cta_mx = mx;
    }
    cluster.sync();
    mx = *cluster.map_shared_rank(&cta_mx, 0);
    for (uint32_t r = 1; r < kRowCtas; ++r) mx = fmaxf(mx, *cluster.map_shared_rank(&cta_mx, r));
    // as the reference: the difference in f32, its exp and the sum in f64
    double part = 0.0;
    for (uint32_t i = rank * kRowThreads + tid; i < vocab; i += kRowCtas * kRowThreads) part += exp(double(__fsub_rn(x[i], mx)));
    part = warp_sum(part);
    if (lane == 0) warp_total[warp] = part;
    __syncthreads();
    if (tid == 0) {
        for (uint32_t w = 1; w < kRowThreads / 32; ++w) part += warp_total[w];
        cta_total = part;
    }
    cluster.sync();
    if (rank == 0 && tid == 0) {
        double total = 0.0;
        for (uint32_t r = 0; r < kRowCtas; ++r) total += *cluster.map_shared_rank(&cta_total, r);
        out[row] = double(__fsub_rn(x[targets[row]], mx)) - log(total);
    }
    cluster.sync();  // no CTA leaves while its shared memory is still read
}

}  // namespace

void launch_row_logp(const float* logits, uint32_t vocab, uint32_t rows, const int32_t* targets, double* out, cudaStream_t s) {
    row_logp_kernel<<<dim3(kRowCtas, rows), kRowThreads, 0, s>>>(logits, vocab, targets, out);
    BK_CUDA(cudaGetLastError());
}

}  // namespace bk
