// Attention of the single new token in two kernels, or one up to 512 positions, bit-identical to the CPU engine's (src/model.cpp:1022-1093; the orders
// of the float operations are those of attn_prompt.cu). They are launched with programmatic dependent launch and request
// the K rows and V tiles of earlier positions before the results they depend on are complete.
//
//   scores  a CTA takes 256 positions of one K/V head and all of its query heads: per-head norm and RoPE of q (and, where the
//           token's own position lies, of the new k, with the f16 cache store), then the dots. Two lanes share two positions,
//           each with half of the 16 partial sums, and two heads share every widened K value.
//   sum     a CTA takes 32 values of one head: softmax of the head's scores, then the position-ordered weighted sum - a
//           chain of dependent f32 additions (src/kernels_f32.cpp:265-273), 4.1 cycles each at best, that bounds the kernel.
//           One warp runs the 32 chains; eight warps on the other schedulers produce p[pos] * v[pos][i] into a pair of
//           tiles, four positions of a value side by side, so that a chain lane reads them with one 16-byte load and adds
//           them one after the other. A producer warp asks for its own pieces of V three tiles ahead with cp.async; chain
//           and producers meet at named barriers. Shared-memory traffic, 3.5 wavefronts a position, is what keeps it at 5.3
//           cycles (one load a position, and loads that queue behind a producer on the same scheduler, made it 8.3).
//
// Short contexts are all latency, so what can be is off the chain of dependent steps: norm weights and RoPE values are asked for
// before the wait (three trips to L2 one after the other otherwise), the cache rows of the new position are stored beside the
// scores instead of ahead of them (their V loads alone were four more trips), the division by the softmax's sum is folded into
// the products, and the sum's last batch is filled up with -0.0. Measured, us a layer: 0.6B shape at 181 positions (one kernel)
// 6.5 -> 4.2, at 530 8.4 -> 6.7, ternary 2B at 530 8.9 -> 7.3, Gemma 1B in its 512-position window 9.6 -> 7.5, 1B shape at 1040
// 10.0 -> 9.0, 7B shape at 2064 18.1 -> 17.0, at 8200 39.0 -> 36.3. Eight producers instead of four are 1 to 3 us of the last two
// (5.6 cycles a position then, 5.3 now). One kernel for both, a cluster of CTAs per K/V head that exchanges the softmax through
// distributed shared memory, was measured too: 46-64 us at 8000 positions of the 7B shape. Three cluster barriers cost it about
// 3 us, and this GPU places only 7 clusters of 16 (15 of 8) at a CTA per SM, so one of the 7B shape's has to share its SMs.
#include <algorithm>

#include "attn_decode.h"
#include "decode_body.cuh"
#include "exact_math.h"
#include "packed.cuh"
#include "pdl.cuh"

namespace bk {
namespace {

constexpr uint32_t kScoreThreads = 256, kSumThreads = 512, kSumWarps = kSumThreads / 32;
constexpr uint32_t kTileFloats = 4096;                  // 128 positions of 32 values
constexpr uint32_t kProducers = 8;                      // warps
constexpr uint32_t kPieces = 16, kDepth = 4;            // pieces of 8 positions x 32 values per tile; tiles in flight
constexpr uint32_t kItems = kPieces / kProducers;       // pieces per producer warp and tile
constexpr uint32_t kPieceBytes = 9 * 64;                // a staged piece: rows of 64 bytes, the second four shifted by one row (banks)
constexpr uint32_t kRingBytes = kDepth * kPieces * kPieceBytes;

constexpr uint32_t kTile = kTileFloats / 32, kBatch = 32;  // positions per tile, and that a chain lane loads ahead

// The new position's K and V rows of a K/V head into the f16 cache, by one warp, `k` normed and rotated. Beside the scores, not
// before them: every score waits for the warp that makes k.
template <int DIM>
__device__ __forceinline__ void store_new_kv(const DecAttnParams& a, uint32_t kvh, uint32_t pos, const float* k) {
    const uint32_t lane = threadIdx.x & 31;
    const size_t base = (size_t(kvh) * a.max_context + pos) * DIM;
    float v[DIM / 32];
#pragma unroll
    for (int i = 0; i < DIM / 32; ++i) {
        v[i] = __ldcg(a.v + size_t(kvh) * DIM + i * 32 + lane);
        if (a.v_bias != nullptr) v[i] = __fadd_rn(v[i], a.v_bias[size_t(kvh) * DIM + i * 32 + lane]);
    }
#pragma unroll
    for (int i = 0; i < DIM / 32; ++i) {
        a.k_cache[base + i * 32 + lane] = __float2half_rn(k[i * 32 + lane]);
        a.v_cache[base + i * 32 + lane] = __float2half_rn(v[i]);
    }
}

template <int DIM>
__global__ void __launch_bounds__(kScoreThreads, 2) decode_scores_kernel(const DecAttnParams a, float one) {
    constexpr int kSteps = DIM / 16;
    constexpr int POS = DIM > 128 ? 1 : 2;  // positions of a pair of lanes: a 256-wide row takes the registers of two
    constexpr uint32_t kPositions = kScoreThreads / 2 * POS;
    extern __shared__ __align__(16) float qs[];  // [group][DIM], then the new k [DIM]
    const uint32_t group = a.heads / a.kv_heads, kvh = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t pos = *a.position, visible = pos + 1, first = blockIdx.x * kPositions;
    if (first >= visible) return;
    const uint32_t mine = min(kPositions, visible - first);
    const bool owner = pos - first < mine;
    // Half a warp apart, so that the halves of a row's 32-byte sectors are asked for by one instruction.
    const uint32_t half = lane >> 4, in_cta = warp * 16 + (lane & 15);
    const __half* kbase = a.k_cache + (size_t(kvh) * a.max_context + first) * DIM + half * 8;
    uint4 raw[POS][kSteps];
#pragma unroll
    for (int j = 0; j < POS; ++j) {
        const uint32_t i = in_cta + j * (kScoreThreads / 2);
        if (i < mine && first + i != pos) {
            const uint4* kr = reinterpret_cast<const uint4*>(kbase + size_t(i) * DIM);
#pragma unroll
            for (int s = 0; s < kSteps; ++s) raw[j][s] = kr[2 * s];
        }
    }
    HeadConstants<DIM / 32> constants;  // of this warp's first task
    warp_head_constants<DIM / 32>(warp < group ? a.q_norm : a.k_norm, a.rope + size_t(pos) * DIM, a.neox, constants);
    wait_for_previous();
    release_next();
    for (uint32_t task = warp; task <= group; task += kScoreThreads / 32) {
        if (task != warp) warp_head_constants<DIM / 32>(task < group ? a.q_norm : a.k_norm, a.rope + size_t(pos) * DIM, a.neox, constants);
        if (task < group) {
            const uint32_t h = kvh * group + task;
            warp_norm_rope_head<DIM / 32>(a.q + size_t(h) * DIM, a.q_bias ? a.q_bias + size_t(h) * DIM : nullptr, a.q_norm != nullptr, constants, a.eps, a.neox, qs + task * DIM);
        } else if (owner) {
            float* knew = qs + group * DIM;
            warp_norm_rope_head<DIM / 32>(a.k + size_t(kvh) * DIM, a.k_bias ? a.k_bias + size_t(kvh) * DIM : nullptr, a.k_norm != nullptr, constants, a.eps, a.neox, knew);
        }
    }
    __syncthreads();
    if (owner && warp == kScoreThreads / 32 - 1) store_new_kv<DIM>(a, kvh, pos, qs + group * DIM);
#pragma unroll
    for (int j = 0; j < POS; ++j) {
        const uint32_t i = in_cta + j * (kScoreThreads / 2);
        if (i < mine && first + i == pos) {  // the token's own row: the f16 values just stored
            const float* knew = qs + group * DIM + half * 8;
#pragma unroll
            for (int s = 0; s < kSteps; ++s) {
                __half2 h[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) h[k] = __floats2half2_rn(knew[s * 16 + 2 * k], knew[s * 16 + 2 * k + 1]);
                raw[j][s] = *reinterpret_cast<const uint4*>(h);
            }
        }
    }
    const f32x2 one2 = pack2(one, one);
#pragma unroll 1
    for (uint32_t g = 0; g < group; g += 2) {  // two heads at a time share a widened value (the last of an odd group goes twice)
        const uint32_t g1 = min(g + 1, group - 1);
        // widened again for every pair of heads: hoisted out of this loop the rows would take twice the registers
#pragma unroll
        for (int j = 0; j < POS; ++j)
#pragma unroll
            for (int k = 0; k < kSteps; ++k) asm volatile("" : "+r"(raw[j][k].x), "+r"(raw[j][k].y), "+r"(raw[j][k].z), "+r"(raw[j][k].w));
        const ulonglong2* qa = reinterpret_cast<const ulonglong2*>(qs + g * DIM + half * 8);
        const ulonglong2* qb = reinterpret_cast<const ulonglong2*>(qs + g1 * DIM + half * 8);
        f32x2 part[2][POS][4];
#pragma unroll
        for (int j = 0; j < POS; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) part[0][j][k] = part[1][j][k] = 0ull;
#pragma unroll
        for (int s = 0; s < kSteps; ++s) {
            const ulonglong2 a0 = qa[s * 4], a1 = qa[s * 4 + 1], b0 = qb[s * 4], b1 = qb[s * 4 + 1];
            const f32x2 va[4] = {a0.x, a0.y, a1.x, a1.y}, vb[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
            for (int j = 0; j < POS; ++j) {
                const __half2* h = reinterpret_cast<const __half2*>(&raw[j][s]);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float2 f = __half22float2(h[k]);
                    const f32x2 k2 = pack2(f.x, f.y);
                    part[0][j][k] = fma2(mul2(va[k], k2), one2, part[0][j][k]);
                    part[1][j][k] = fma2(mul2(vb[k], k2), one2, part[1][j][k]);
                }
            }
        }
        float sum[2][POS];
        auto add_parts = [&] {
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int hd = 0; hd < 2; ++hd)
#pragma unroll
                    for (int j = 0; j < POS; ++j) {
                        float x, y;
                        unpack2(part[hd][j][k], x, y);
                        sum[hd][j] = __fadd_rn(__fadd_rn(sum[hd][j], x), y);
                    }
        };
#pragma unroll
        for (int j = 0; j < POS; ++j) sum[0][j] = sum[1][j] = 0.0f;
        add_parts();
#pragma unroll
        for (int j = 0; j < POS; ++j) {  // the upper half-warp goes on from its partner's sums of the first eight
            sum[0][j] = __shfl_sync(0xffffffffu, sum[0][j], lane & 15);
            sum[1][j] = __shfl_sync(0xffffffffu, sum[1][j], lane & 15);
        }
        if (half == 1) {
            add_parts();
#pragma unroll
            for (int j = 0; j < POS; ++j) {
                const uint32_t i = in_cta + j * (kScoreThreads / 2);
                if (i < mine) {
                    a.scores[size_t(kvh * group + g) * a.max_context + first + i] = __fmul_rn(sum[0][j], a.scale);
                    a.scores[size_t(kvh * group + g1) * a.max_context + first + i] = __fmul_rn(sum[1][j], a.scale);
                }
            }
        }
    }
}

// Producer warps leave the chain warp's scheduler (warp mod 4) to it: its loads would queue behind theirs.
__device__ __forceinline__ uint32_t producer_number(uint32_t warp) { return warp % 4 == 0 || warp > 10 ? kProducers : warp - warp / 4 - 1; }  // kProducers: none
__device__ __forceinline__ void tile_sync(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kProducers * 32 + 32) : "memory"); }
__device__ __forceinline__ void tile_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(kProducers * 32 + 32) : "memory"); }

// grid: heads x dim / 32. ps_floats: room for the visible positions' probabilities, a multiple of 4.
// DIM = 0: the scores are there. DIM = 64, 128: every CTA computes its head's scores itself, which saves the kernel before it
// for as long as the K rows (each read by group x dim / 32 CTAs, the first 512 positions' before the wait) cost less.
template <int DIM>
__global__ void __launch_bounds__(kSumThreads, 1) decode_sum_kernel(const DecAttnParams a, uint32_t window, uint32_t ps_floats, float one) {
    constexpr bool kScores = DIM != 0;
    constexpr int kSteps = kScores ? DIM / 16 : 1, POS = 2;  // as in the scores kernel
    __shared__ __align__(16) float q_row[kScores ? DIM : 4], k_new[kScores ? DIM : 4];
    __shared__ __align__(4) __half v_new[32];  // the token's own V slice: its cache row is another CTA's store
    extern __shared__ __align__(16) unsigned char smem[];
    float* ps = reinterpret_cast<float*>(smem);
    float* tiles = ps + ps_floats;
    unsigned char* ring = reinterpret_cast<unsigned char*>(tiles + 2 * kTileFloats);
    __shared__ float redf[kSumWarps];
    __shared__ double redd[kSumWarps];
    __shared__ uint64_t exp_table[32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, dim = a.dim, slices = dim / 32;
    const uint32_t h = blockIdx.x / slices, col0 = blockIdx.x % slices * 32, kvh = h / (a.heads / a.kv_heads);
    const uint32_t visible = *a.position + 1, start = window != 0 && visible > window ? visible - window : 0, cnt = visible - start;
    const __half* vbase = a.v_cache + (size_t(kvh) * a.max_context + start) * dim + col0;

    const uint32_t producer = producer_number(warp);
    auto piece_at = [&](uint32_t tile, uint32_t i) { return ring + (tile % kDepth * kPieces + i * kProducers + producer) * kPieceBytes; };
    auto request = [&](uint32_t tile, uint32_t from, uint32_t to) {  // rows [from, to) of the sequence that lie in `tile`
        const uint32_t r = lane >> 2, c = lane & 3;
#pragma unroll
        for (uint32_t i = 0; i < kItems; ++i) {
            const uint32_t piece = i * kProducers + producer, p = tile * kTile + piece * 8 + r;
            if (p >= from && p < to) {
                const uint32_t dst = uint32_t(__cvta_generic_to_shared(piece_at(tile, i) + r * 64 + (r >> 2) * 64 + c * 16));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(vbase + size_t(p) * dim + c * 8) : "memory");
            }
        }
    };
    if (producer < kProducers) {
        for (uint32_t t = 0; t + 1 < kDepth; ++t) {
            request(t, 0, cnt - 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    }
    if (tid < 32) exp_table[tid] = exp2_table_device()[tid];
    const uint32_t half = lane >> 4, in_cta = warp * 16 + (lane & 15);
    uint4 raw[POS][kSteps];
    auto load_k = [&](uint32_t p0) {
        const __half* kbase = a.k_cache + (size_t(kvh) * a.max_context + start) * DIM + half * 8;
#pragma unroll
        for (int j = 0; j < POS; ++j) {
            const uint32_t i = p0 + in_cta + j * (kSumThreads / 2);
            if (i < cnt - 1) {
                const uint4* kr = reinterpret_cast<const uint4*>(kbase + size_t(i) * DIM);
#pragma unroll
                for (int s = 0; s < kSteps; ++s) raw[j][s] = kr[2 * s];
            }
        }
    };
    if constexpr (kScores) load_k(0);
    HeadConstants<kScores ? DIM / 32 : 2> constants;
    if (kScores && warp < 2) warp_head_constants(warp == 0 ? a.q_norm : a.k_norm, a.rope + size_t(visible - 1) * DIM, a.neox, constants);
    wait_for_previous();
    release_next();
    float m = -INFINITY;
    if constexpr (kScores) {
        const uint32_t pos = visible - 1;
        if (warp == 0) {
            warp_norm_rope_head<DIM / 32>(a.q + size_t(h) * DIM, a.q_bias ? a.q_bias + size_t(h) * DIM : nullptr, a.q_norm != nullptr, constants, a.eps, a.neox, q_row);
        } else if (warp == 1) {
            warp_norm_rope_head<DIM / 32>(a.k + size_t(kvh) * DIM, a.k_bias ? a.k_bias + size_t(kvh) * DIM : nullptr, a.k_norm != nullptr, constants, a.eps, a.neox, k_new);
        } else if (warp == 2) {
            float v = __ldcg(a.v + size_t(kvh) * DIM + col0 + lane);
            if (a.v_bias != nullptr) v = __fadd_rn(v, a.v_bias[size_t(kvh) * DIM + col0 + lane]);
            v_new[lane] = __float2half_rn(v);
        }
        __syncthreads();
        if (h % (a.heads / a.kv_heads) == 0 && col0 == 0 && warp == kSumWarps - 1) store_new_kv<DIM>(a, kvh, pos, k_new);
        const f32x2 one2 = pack2(one, one);
        const ulonglong2* q2 = reinterpret_cast<const ulonglong2*>(q_row + half * 8);
        // `count` of the lane's POS positions from p0 on
        auto score = [&](uint32_t p0, auto count) {
            constexpr int N = decltype(count)::value;
            f32x2 part[N][4];
#pragma unroll
            for (int j = 0; j < N; ++j) {
                if (p0 + in_cta + j * (kSumThreads / 2) == cnt - 1) {  // the token's own row, as the cache holds it
#pragma unroll
                    for (int s = 0; s < kSteps; ++s) {
                        __half2 hv[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) hv[k] = __floats2half2_rn(k_new[s * 16 + half * 8 + 2 * k], k_new[s * 16 + half * 8 + 2 * k + 1]);
                        raw[j][s] = *reinterpret_cast<const uint4*>(hv);
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) part[j][k] = 0ull;
            }
#pragma unroll
            for (int s = 0; s < kSteps; ++s) {
                const ulonglong2 q0 = q2[s * 4], q1 = q2[s * 4 + 1];
                const f32x2 qv[4] = {q0.x, q0.y, q1.x, q1.y};
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    const __half2* hv = reinterpret_cast<const __half2*>(&raw[j][s]);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float2 f = __half22float2(hv[k]);
                        part[j][k] = fma2(mul2(qv[k], pack2(f.x, f.y)), one2, part[j][k]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < N; ++j) {
                float sum = 0.0f;
                auto add_parts = [&] {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        float x, y;
                        unpack2(part[j][k], x, y);
                        sum = __fadd_rn(__fadd_rn(sum, x), y);
                    }
                };
                add_parts();
                sum = __shfl_sync(0xffffffffu, sum, lane & 15);  // the upper half-warp goes on from its partner's sum of the first eight
                const uint32_t i = p0 + in_cta + j * (kSumThreads / 2);
                if (half == 1 && i < cnt) {
                    add_parts();
                    const float v = __fmul_rn(sum, a.scale);
                    ps[i] = v;
                    m = fmaxf(m, v);
                }
            }
        };
        // A warp without positions leaves the schedulers to the others: 2560 -> 1300 cycles for the scores of 180 positions.
        for (uint32_t p0 = 0; p0 + warp * 16 < cnt; p0 += kSumThreads / 2 * POS) {
            if (p0 != 0) load_k(p0);
            if (p0 + warp * 16 + kSumThreads / 2 < cnt) score(p0, std::integral_constant<int, 2>{});
            else score(p0, std::integral_constant<int, 1>{});
        }
    }

    // ---- softmax (src/kernels_f32.cpp:275-284): e = expf(s - max), f64 sum, p = e * float(1 / sum) ----
    const float* s = a.scores + size_t(h) * a.max_context + start;
    if constexpr (!kScores) for (uint32_t p0 = tid; p0 < cnt; p0 += 8 * kSumThreads) {  // eight loads in flight
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = p0 + u * kSumThreads < cnt ? __ldcg(s + p0 + u * kSumThreads) : -INFINITY;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (p0 + u * kSumThreads < cnt) ps[p0 + u * kSumThreads] = v[u];
            m = fmaxf(m, v[u]);
        }
    }
    m = warp_max(m);
    if (lane == 0) redf[warp] = m;
    __syncthreads();
    m = warp_max(redf[lane & (kSumWarps - 1)]);
    double part = 0.0;
    // N at a time: one exp is a long chain of f64 operations (1040 positions one after the other: 1200 cycles, 700 so).
    auto exps = [&](uint32_t p0, auto count, auto whole) {  // whole: no position past the last among them
        constexpr int N = decltype(count)::value;
        constexpr bool kWhole = decltype(whole)::value;
        float e[N];
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const uint32_t p = p0 + u * kSumThreads + tid;
            e[u] = exact_expf_flat(kWhole || p < cnt ? __fsub_rn(ps[p], m) : 0.0f, exp_table);
        }
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const uint32_t p = p0 + u * kSumThreads + tid;
            if (kWhole || p < cnt) {
                ps[p] = e[u];
                part += double(e[u]);
            }
        }
    };
    uint32_t p0 = 0;
    for (; p0 + 4 * kSumThreads <= cnt; p0 += 4 * kSumThreads) exps(p0, std::integral_constant<int, 4>{}, std::true_type{});
    if (p0 + 2 * kSumThreads + warp * 32 < cnt) exps(p0, std::integral_constant<int, 4>{}, std::false_type{});
    else if (p0 + kSumThreads + warp * 32 < cnt) exps(p0, std::integral_constant<int, 2>{}, std::false_type{});
    else if (p0 + warp * 32 < cnt) exps(p0, std::integral_constant<int, 1>{}, std::false_type{});
    part = warp_sum(part);
    if (lane == 0) redd[warp] = part;
    __syncthreads();
    static_assert(kSumWarps == 16);
    double total = redd[lane & (kSumWarps - 1)];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    const float inv = float(1.0 / total);

    // ---- weighted sum: p = e * inv where it is used ----
    const uint32_t chunks = (cnt + kTile - 1) / kTile;
    if (producer < kProducers) {
        if (!kScores && (cnt - 1) / kTile + 1 < kDepth) {  // a short context: the own row belongs to a tile requested above
            request((cnt - 1) / kTile, cnt - 1, cnt);
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
#pragma unroll 1
        for (uint32_t c = 0; c < chunks; ++c) {
            const uint32_t b = c & 1, dp = lane & 15, pg = lane >> 4;  // this lane: values 2 dp, 2 dp + 1 of positions 4 pg .. 4 pg + 3
            request(c + kDepth - 1, 0, kScores ? cnt - 1 : cnt);
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 1) : "memory");
            __syncwarp();  // tile c's pieces of this warp have landed
            uint32_t v[kItems][4];
            float4 pr[kItems];
#pragma unroll
            for (uint32_t i = 0; i < kItems; ++i) {
                const unsigned char* at = piece_at(c, i) + pg * 5 * 64 + dp * 4;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[i][j] = *reinterpret_cast<const uint32_t*>(at + j * 64);
                    if (kScores && c * kTile + (i * kProducers + producer) * 8 + pg * 4 + j == cnt - 1) v[i][j] = *reinterpret_cast<const uint32_t*>(v_new + 2 * dp);
                }
                pr[i] = *reinterpret_cast<const float4*>(ps + min(c * kTile + (i * kProducers + producer) * 8 + pg * 4, ps_floats - 4));
            }
            if (c >= 2) tile_sync(3 + b);  // the chains are done with this buffer's previous tile
            float* tile = tiles + size_t(b) * kTileFloats;
#pragma unroll
            for (uint32_t i = 0; i < kItems; ++i) {
                const uint32_t piece = i * kProducers + producer;
                pr[i] = make_float4(__fmul_rn(pr[i].x, inv), __fmul_rn(pr[i].y, inv), __fmul_rn(pr[i].z, inv), __fmul_rn(pr[i].w, inv));
                float2 f[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) f[j] = __half22float2(*reinterpret_cast<const __half2*>(&v[i][j]));
                float4 lo = make_float4(__fmul_rn(pr[i].x, f[0].x), __fmul_rn(pr[i].y, f[1].x), __fmul_rn(pr[i].z, f[2].x), __fmul_rn(pr[i].w, f[3].x));
                float4 hi = make_float4(__fmul_rn(pr[i].x, f[0].y), __fmul_rn(pr[i].y, f[1].y), __fmul_rn(pr[i].z, f[2].y), __fmul_rn(pr[i].w, f[3].y));
                if (c + 1 == chunks) {  // Past the last position: x + -0.0 is x, whatever x is, so the chains add whole batches.
                    const uint32_t p = c * kTile + piece * 8 + pg * 4;
                    if (p >= cnt) lo.x = hi.x = -0.0f;
                    if (p + 1 >= cnt) lo.y = hi.y = -0.0f;
                    if (p + 2 >= cnt) lo.z = hi.z = -0.0f;
                    if (p + 3 >= cnt) lo.w = hi.w = -0.0f;
                }
                float4* at = reinterpret_cast<float4*>(tile) + (piece * 2 + pg) * 32 + 2 * dp;
                const bool swap = (dp & 4) != 0;  // every other quad of lanes stores its values the other way round: no bank conflict
                at[swap ? 1 : 0] = swap ? hi : lo;
                at[swap ? 0 : 1] = swap ? lo : hi;
            }
            __syncwarp();  // the pieces may be overwritten
            tile_arrive(1 + b);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else if (warp == 0) {
        float acc = 0.0f;
        const float4* tile0 = reinterpret_cast<const float4*>(tiles) + lane;
        constexpr uint32_t kTileVecs = kTileFloats / 4, kVecs = kBatch / 4;
        // Two register sets: while one set's products are added, one load between every four additions fills the other. The
        // order is written down because the compiler left to itself moves the loads behind the additions that hide them.
        float4 s0[kVecs], s1[kVecs];
        auto load = [&](const float4* src, float4& v) {
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                         : "r"(uint32_t(__cvta_generic_to_shared(src)))
                         : "memory");
        };
        auto add4 = [&](const float4& v) {
            asm volatile("add.rn.f32 %0, %0, %1;\n\tadd.rn.f32 %0, %0, %2;\n\tadd.rn.f32 %0, %0, %3;\n\tadd.rn.f32 %0, %0, %4;"
                         : "+f"(acc)
                         : "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w));
        };
        auto load_and_add = [&](const float4* src, float4 (&dst)[kVecs], const float4 (&sum)[kVecs]) {
#pragma unroll
            for (uint32_t u = 0; u < kVecs; ++u) {
                load(src + u * 32, dst[u]);
                add4(sum[u]);
            }
        };
        // Batches of 32 positions, four to a tile; the last one is filled up with -0.0 (see the producers). One position after the
        // other, what a last batch of fewer had left took 1600 cycles at 53 positions.
        constexpr uint32_t kBatchVecs = kVecs * 32;
        static_assert(kTile == 4 * kBatch);
        tile_sync(1);
#pragma unroll
        for (uint32_t u = 0; u < kVecs; ++u) load(tile0 + u * 32, s0[u]);
#pragma unroll 1
        for (uint32_t c = 0; c + 1 < chunks; ++c) {  // s0 holds the tile's first batch
            const float4* src = tile0 + (c & 1) * kTileVecs;
            load_and_add(src + kBatchVecs, s1, s0);
            load_and_add(src + 2 * kBatchVecs, s0, s1);
            load_and_add(src + 3 * kBatchVecs, s1, s0);
            tile_sync(1 + ((c + 1) & 1));  // the next tile's first batch, before this tile's last additions
            load_and_add(tile0 + ((c + 1) & 1) * kTileVecs, s0, s1);
            if (c + 2 < chunks) tile_arrive(3 + (c & 1));  // a producer waits for exactly these
        }
        const float4* src = tile0 + ((chunks - 1) & 1) * kTileVecs;
        const uint32_t batches = (cnt - (chunks - 1) * kTile + kBatch - 1) / kBatch;
#pragma unroll 1
        for (uint32_t b = 0; b < batches; b += 2) {
            if (b + 1 < batches) load_and_add(src + (b + 1) * kBatchVecs, s1, s0);
            else {
#pragma unroll
                for (uint32_t u = 0; u < kVecs; ++u) add4(s0[u]);
                break;
            }
            if (b + 2 < batches) load_and_add(src + (b + 2) * kBatchVecs, s0, s1);
            else {
#pragma unroll
                for (uint32_t u = 0; u < kVecs; ++u) add4(s1[u]);
            }
        }
        a.out[size_t(h) * dim + col0 + lane] = acc;
    }
}

template <int DIM>
void launch_scores(const DecAttnParams& a, uint32_t max_visible, cudaStream_t s) {
    constexpr uint32_t kPositions = DIM > 128 ? 128 : 256;
    launch_dependent(decode_scores_kernel<DIM>, dim3((max_visible + kPositions - 1) / kPositions, a.kv_heads), dim3(kScoreThreads),
                     size_t(a.heads / a.kv_heads + 1) * DIM * sizeof(float), s, a, 1.0f);
}

size_t sum_smem(uint32_t positions) { return size_t((positions + 3) & ~3u) * 4 + 2 * kTileFloats * 4 + kRingBytes; }

}  // namespace

bool attn_decode_fits(uint32_t dim, uint32_t positions) { return (dim == 64 || dim == 128 || dim == 256) && sum_smem(positions) <= 200 * 1024; }

template <int DIM>
static void launch_sum(const DecAttnParams& a, uint32_t window, cudaStream_t s) {
    static DeviceOnce once;
    if (once.first()) BK_CUDA(cudaFuncSetAttribute(decode_sum_kernel<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    const uint32_t positions = window != 0 ? std::min(window, a.max_context) : a.max_context;
    launch_dependent(decode_sum_kernel<DIM>, dim3(a.heads * (a.dim / 32)), dim3(kSumThreads), sum_smem(positions), s, a, window, (positions + 3) & ~3u, 1.0f);
}

int launch_attn_decode(const DecAttnParams& a, uint32_t window, bool fused, cudaStream_t s) {
    if (fused && a.dim == 64) launch_sum<64>(a, window, s);
    else if (fused && a.dim == 128) launch_sum<128>(a, window, s);
    else {
        if (a.dim == 64) launch_scores<64>(a, a.max_context, s);
        else if (a.dim == 128) launch_scores<128>(a, a.max_context, s);
        else launch_scores<256>(a, a.max_context, s);
        launch_sum<0>(a, window, s);
        return 2;
    }
    return 1;
}

}  // namespace bk
