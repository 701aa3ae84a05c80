// Weighted sum of attention for 2..24 tokens at once (one token: attn_decode.cu), arranged around the one thing the reference's
// order of operations does not let anybody parallelise: out[i] = ((p[0]*v_0[i] + p[1]*v_1[i]) + p[2]*v_2[i]) + ... is a chain
// of dependent f32 additions per (token, head, i), one per visible position (src/kernels_f32.cpp:265-273), and the result has
// to be that chain's, bit for bit, because the 8-bit re-quantisation that follows turns a 1-ulp difference into a different
// integer every so often. The probabilities come from the scores and softmax kernels of attn_prompt.cu.
//
//   CTA    32 values of a K/V head, ROWS of its (token, query head) rows, tokens outermost: one warp per row, one value per
//          lane. The rows share the V they read; with a CTA per row or two and all of a head's values every CTA streams the
//          whole head's V, 18 of them the same lines at a time.
//   tiles  128 positions: the values' slices of V (64 bytes a row) and the rows' probabilities come with cp.async through a
//          ring of four stages, so that no context is too long
//   chain  per position a lane loads its value (one shared wavefront a warp), widens it, multiplies by the probability (read
//          four positions at a time) and adds: 4.25 issue slots, two warps a scheduler hide one another's latencies
//
// Measured, 9 tokens at 2064 positions of the 7B shape 25 us with either form (its eight warps an SM share the shared-memory
// pipe, which a probability read, broadcast or not, holds for four cycles), 23 tokens at 53 positions 7.0 -> 4.1 us, 9-token step
// of the 1B Q4_K_M shape at 1000 positions 1.79 -> 1.65 ms. Two values a lane and half the warps: 32 us, a lone warp on its
// scheduler waits out every load.
#include "kernels.h"
#include "pdl.cuh"
#include "rowops.cuh"

namespace bk {
namespace {

constexpr uint32_t kTile = 128, kStages = 4, kBatch = 16, kValues = 32;

struct ChainParams {
    const float* probs;    // [n][heads][max_context]
    const __half* v_cache; // [kv][max_context][dim]
    float* out;            // [n][heads * dim]
    DevActMut quant;       // where q0 is set: the same as Q8_0 planes
    const uint32_t* position;
    uint32_t n, heads, kv_heads, dim, max_context, window;
};

// grid: (dim / 32, K/V heads, row groups)
template <int ROWS>
__global__ void __launch_bounds__(ROWS * 32) attn_chain_kernel(const ChainParams a) {
    constexpr uint32_t kThreads = ROWS * 32;
    __shared__ __align__(16) __half vs[kStages][kTile][kValues];
    __shared__ __align__(16) float ps[kStages][ROWS][kTile];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t group = a.heads / a.kv_heads, kvh = blockIdx.y, rows = a.n * group, col0 = blockIdx.x * kValues;
    const uint32_t r0 = blockIdx.z * ROWS, last = min(r0 + ROWS, rows) - 1, row = min(r0 + warp, last);  // a warp past the last row repeats it
    const uint32_t token = row / group, h = kvh * group + row % group;
    wait_for_previous();
    // Where the rows end in planes, the multiply that takes them starts when the chains are done; released here, its CTAs would sit
    // beside these for the whole walk.
    if (a.quant.q0 == nullptr) release_next();
    const uint32_t position = *a.position;
    // a sliding-window layer attends to the last `window` positions only (src/model.cpp:1084-1091)
    auto start_of = [&](uint32_t visible) { return a.window != 0 && visible > a.window ? visible - a.window : 0u; };
    const uint32_t visible = position + token + 1, start = start_of(visible);
    const uint32_t all_visible = position + last / group + 1, first = start_of(position + r0 / group + 1) / kTile, tiles = (all_visible + kTile - 1) / kTile;
    const __half* vbase = a.v_cache + size_t(kvh) * a.max_context * a.dim + col0;
    const float* prow = a.probs + (size_t(token) * a.heads + h) * a.max_context;
    const bool aligned = a.max_context % 4 == 0;  // probability rows start on 16-byte boundaries

    auto request = [&](uint32_t tile) {
        if (tile < tiles) {
            const uint32_t base = tile * kTile, stage = tile % kStages;
            for (uint32_t i = tid; i < kTile * 4; i += kThreads) {  // 16-byte pieces of V
                const uint32_t p = base + i / 4, c = i % 4;
                if (p < all_visible) {
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(&vs[stage][i / 4][c * 8]))),
                                 "l"(vbase + size_t(p) * a.dim + c * 8)
                                 : "memory");
                }
            }
            const uint32_t p = base + lane * 4, dst = uint32_t(__cvta_generic_to_shared(&ps[stage][warp][lane * 4]));
            if (aligned) {
                if (p < visible) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(prow + p) : "memory");
            } else {
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    if (p + k < visible) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * k), "l"(prow + p + k) : "memory");
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (uint32_t s = 0; s + 1 < kStages; ++s) request(first + s);

    float acc = 0.0f;
    auto add = [&](float p, __half v) { acc = __fadd_rn(acc, __fmul_rn(p, __half2float(v))); };
    for (uint32_t tile = first; tile < tiles; ++tile) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();  // the stage has landed for every thread, and the one requested next is no longer read
        request(tile + kStages - 1);
        const uint32_t base = tile * kTile, stage = tile % kStages;
        const uint32_t lo = start > base ? min(kTile, start - base) : 0, hi = visible > base ? min(kTile, visible - base) : 0;
        const __half* v = &vs[stage][0][lane];
        const float* p = ps[stage][warp];
        // Batches of 16 positions in two register sets named apart: the loads of one are in flight while the other's additions -
        // the dependent chain - run.
        __half v0[kBatch], v1[kBatch];
        float4 p0[kBatch / 4], p1[kBatch / 4];
        auto load = [&](uint32_t i, __half (&vv)[kBatch], float4 (&pp)[kBatch / 4]) {
#pragma unroll
            for (uint32_t u = 0; u < kBatch; ++u) vv[u] = v[(i + u) * 32];
#pragma unroll
            for (uint32_t u = 0; u < kBatch / 4; ++u) pp[u] = *reinterpret_cast<const float4*>(p + i + 4 * u);
        };
        auto run = [&](const __half (&vv)[kBatch], const float4 (&pp)[kBatch / 4]) {
#pragma unroll
            for (uint32_t u = 0; u < kBatch / 4; ++u) {
                add(pp[u].x, vv[4 * u]);
                add(pp[u].y, vv[4 * u + 1]);
                add(pp[u].z, vv[4 * u + 2]);
                add(pp[u].w, vv[4 * u + 3]);
            }
        };
        uint32_t i = lo;
        for (; i < hi && i % kBatch != 0; ++i) add(p[i], v[i * 32]);
        uint32_t batches = i < hi ? (hi - i) / kBatch : 0;
        if (batches > 0) {
            load(i, v0, p0);
#pragma unroll 1
            for (; batches > 2; batches -= 2, i += 2 * kBatch) {
                load(i + kBatch, v1, p1);
                run(v0, p0);
                load(i + 2 * kBatch, v0, p0);
                run(v1, p1);
            }
            if (batches == 2) {
                load(i + kBatch, v1, p1);
                run(v0, p0);
                run(v1, p1);
            } else {
                run(v0, p0);
            }
            i += batches * kBatch;
        }
        if (i < hi) {  // fewer than a batch: the rest of it adds -0.0, which changes nothing
            load(i, v0, p0);
            const uint32_t left = hi - i;
            const float pv[kBatch] = {p0[0].x, p0[0].y, p0[0].z, p0[0].w, p0[1].x, p0[1].y, p0[1].z, p0[1].w, p0[2].x, p0[2].y, p0[2].z, p0[2].w, p0[3].x, p0[3].y, p0[3].z, p0[3].w};
#pragma unroll
            for (uint32_t u = 0; u < kBatch; ++u) {
                const float product = __fmul_rn(pv[u], __half2float(v0[u]));
                acc = __fadd_rn(acc, u < left ? product : -0.0f);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (a.quant.q0 != nullptr) release_next();
    const size_t at = (size_t(token) * a.heads + h) * a.dim + col0;
    if (r0 + warp <= last) a.out[at + lane] = acc;
    if (a.quant.q0 != nullptr) {  // the warp's 32 values are a block of the next multiply's input
        int sum;
        float d;
        const int q = warp_quantize_q8_0(acc, d, sum);
        if (r0 + warp <= last) {
            a.quant.q0[at + lane] = int8_t(q);
            if (lane == 0) {
                a.quant.d0[at / 32] = d;
                a.quant.s0[at / 32] = sum;
            }
        }
    }
}

template <int ROWS>
void launch_rows(const ChainParams& p, uint32_t groups, cudaStream_t s) {
    launch_dependent(attn_chain_kernel<ROWS>, dim3(p.dim / kValues, p.kv_heads, groups), dim3(ROWS * 32), 0, s, p);
}

}  // namespace

// a.scores holds the probabilities of the n tokens (rows of max_context floats); a.out receives the attended rows.
void launch_attn_chain(const AttnArgs& a, const DevActMut* planes, uint32_t sms, cudaStream_t s) {
    ChainParams p{};
    p.probs = a.scores; p.v_cache = a.v_cache; p.out = a.out; p.position = a.position;
    p.n = a.n; p.heads = a.heads; p.kv_heads = a.kv_heads; p.dim = a.dim; p.max_context = a.max_context; p.window = a.window;
    if (planes != nullptr) p.quant = *planes;
    const uint32_t rows = a.n * (a.heads / a.kv_heads);
    // The rows a CTA takes: whichever leaves the busiest SM with fewer warps, the more of them on a tie (less V traffic).
    auto groups = [&](uint32_t per_cta) { return (rows + per_cta - 1) / per_cta; };
    auto busiest = [&](uint32_t per_cta) { return (uint64_t(groups(per_cta)) * a.kv_heads * (a.dim / kValues) + sms - 1) / sms * per_cta; };
    if (busiest(8) <= busiest(4)) launch_rows<8>(p, groups(8), s);
    else launch_rows<4>(p, groups(4), s);
}

}  // namespace bk
