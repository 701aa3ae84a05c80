// Causal attention of a batch of tokens over cached positions, in the reference's own order of float operations
// (src/model.cpp:1050-1093 over src/kernels_f32.cpp:231-284), so that the result is bit-identical to the CPU engine's and
// the 8-bit re-quantisation that follows sees the same values:
//   scores   s[p] = dot_f32(q, k_p) * scale, dot_f32 = 16 interleaved partial sums, then their sum in order
//   softmax  e[p] = expf(s[p] - max) (glibc's expf, see exact_math.h), sum in f64, p[p] = e[p] * float(1/sum)
//   output   out[i] = ((p[0]*v_0[i] + p[1]*v_1[i]) + p[2]*v_2[i]) + ...   one position after the other
//
// Bound: the f32 pipe. Every multiply-add is two roundings (no fused multiply-add, no tensor core: the order of every sum
// is fixed), so 2 * 2 * pairs * heads * head_dim lane operations are what an attention costs at least - 2 x 440 us for the
// last 512 tokens of a 4096-token prompt of the 7B shape. Packed f32x2 instructions halve the issue slots of that
// arithmetic (not its pipe time) and leave room for the shared-memory reads. Their sum is an fma by `one`, a kernel
// parameter: a packed multiply feeding a packed add would be contracted into a single rounding by the assembler.
//
// All three kernels work on ROWS: the (token, query head) pairs of one K/V head, tokens outermost. Rows of a tile share
// every cached K and V row they read, so grouped-query heads cost no extra cache traffic, and a tile of few tokens wastes
// little at the causal edge.
#include <algorithm>

#include "exact_math.h"
#include "kernels.h"
#include "packed.cuh"
#include "pdl.cuh"

namespace bk {
namespace {

// ---- scores -------------------------------------------------------------------------------------------------------
// grid of both forms: (position chunks, K/V heads, row tiles), the row tile outermost and latest first: late tiles see the
// most.
//
// Heads of 64 and 128 values: a thread owns one cached position, its K row in registers as packed f32 pairs, and scores it
// against the tile's rows one after the other (q broadcast from shared memory, 16 bytes a read). Measured, the last 512
// tokens of a 4096-token prompt of the 7B shape: 763 us with scalar arithmetic, 668 us now (70 % of the f32 pipe).
// Four positions shared by the lanes of a quad, which reads q a quarter as often, measured 762: what it saves in reads it
// pays in exchanging partial sums.
template <int DIM>
__global__ void __launch_bounds__(128) attn_scores_kernel(const AttnArgs a, uint32_t tile_rows, float one) {
    constexpr int kSteps = DIM / 16;
    extern __shared__ __align__(16) float qs[];  // [tile_rows][DIM]
    const uint32_t group = a.heads / a.kv_heads, kvh = blockIdx.y, rows = a.n * group, tid = threadIdx.x;
    const uint32_t r0 = (gridDim.z - 1 - blockIdx.z) * tile_rows, rn = min(tile_rows, rows - r0);
    wait_for_previous();
    const uint32_t position = *a.position;
    const uint32_t last_visible = position + (r0 + rn - 1) / group + 1;
    if (blockIdx.x * 128 >= last_visible) return;
    for (uint32_t i = tid; i < rn * (DIM / 4); i += 128) {
        const uint32_t r = r0 + i / (DIM / 4), piece = i % (DIM / 4);
        reinterpret_cast<float4*>(qs)[i] = *reinterpret_cast<const float4*>(a.q + (size_t(r / group) * a.heads + kvh * group + r % group) * DIM + piece * 4);
    }
    const uint32_t p = blockIdx.x * 128 + tid;
    // threads past the end read a valid row and store nothing
    const uint4* kr = reinterpret_cast<const uint4*>(a.k_cache + (size_t(kvh) * a.max_context + min(p, last_visible - 1)) * DIM);
    f32x2 k2[kSteps][8];
#pragma unroll
    for (int s = 0; s < kSteps; ++s) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint4 raw = kr[2 * s + u];
            const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = __half22float2(h[j]);
                k2[s][u * 4 + j] = pack2(f.x, f.y);
            }
        }
    }
    __syncthreads();
    const f32x2 one2 = pack2(one, one);
    uint32_t token = r0 / group, g = r0 % group;
    for (uint32_t r = 0; r < rn; ++r) {
        const ulonglong2* q2 = reinterpret_cast<const ulonglong2*>(qs + r * DIM);
        f32x2 part[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) part[j] = 0ull;
#pragma unroll
        for (int s = 0; s < kSteps; ++s) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const ulonglong2 q = q2[s * 4 + j];
                part[2 * j] = fma2(mul2(q.x, k2[s][2 * j]), one2, part[2 * j]);
                part[2 * j + 1] = fma2(mul2(q.y, k2[s][2 * j + 1]), one2, part[2 * j + 1]);
            }
        }
        float sum = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float x, y;
            unpack2(part[j], x, y);
            sum = __fadd_rn(__fadd_rn(sum, x), y);
        }
        if (p < position + token + 1) a.scores[(size_t(token) * a.heads + kvh * group + g) * a.max_context + p] = __fmul_rn(sum, a.scale);
        if (++g == group) {
            g = 0;
            ++token;
        }
    }
    release_next();
}

// Heads of 256 values: a K row does not fit a thread's registers. Four lanes share two cached positions: lane k of a quad
// holds partial sums 4k .. 4k + 3 of both, that is the values 16s + 4k .. 16s + 4k + 3 of their rows. At the end of a row the
// pairs of lanes exchange sums so that each works on one position, and the quad's second pair goes on with the first one's
// sum.
__global__ void __launch_bounds__(128) attn_scores_wide_kernel(const AttnArgs a, uint32_t tile_rows, float one) {
    constexpr int POS = 2, DIM = 256, kSteps = DIM / 16;
    constexpr uint32_t kPositions = 32 * POS;  // per CTA
    extern __shared__ __align__(16) float qs[];  // [tile_rows][DIM]
    const uint32_t group = a.heads / a.kv_heads, kvh = blockIdx.y, rows = a.n * group;
    const uint32_t r0 = (gridDim.z - 1 - blockIdx.z) * tile_rows, rn = min(tile_rows, rows - r0);
    wait_for_previous();
    const uint32_t position = *a.position;
    const uint32_t last_visible = position + (r0 + rn - 1) / group + 1;
    if (blockIdx.x * kPositions >= last_visible) return;
    const uint32_t tid = threadIdx.x, k = tid & 3;
    for (uint32_t i = tid; i < rn * (DIM / 4); i += 128) {
        const uint32_t r = r0 + i / (DIM / 4), piece = i % (DIM / 4);
        reinterpret_cast<float4*>(qs)[i] = *reinterpret_cast<const float4*>(a.q + (size_t(r / group) * a.heads + kvh * group + r % group) * DIM + piece * 4);
    }
    const uint32_t p0 = blockIdx.x * kPositions + (tid >> 2) * POS;  // the quad's first position
    f32x2 k2[POS][kSteps][2];
#pragma unroll
    for (int j = 0; j < POS; ++j) {
        // positions past the end read a valid row and store nothing
        const __half* kr = a.k_cache + (size_t(kvh) * a.max_context + min(p0 + j, last_visible - 1)) * DIM + 4 * k;
#pragma unroll
        for (int s = 0; s < kSteps; ++s) {
            const uint2 raw = *reinterpret_cast<const uint2*>(kr + s * 16);
            const float2 f0 = __half22float2(reinterpret_cast<const __half2*>(&raw)[0]), f1 = __half22float2(reinterpret_cast<const __half2*>(&raw)[1]);
            k2[j][s][0] = pack2(f0.x, f0.y);
            k2[j][s][1] = pack2(f1.x, f1.y);
        }
    }
    __syncthreads();
    const f32x2 one2 = pack2(one, one);
    const bool odd = (k & 1) != 0, high = (k & 2) != 0;
    const uint32_t mine = p0 + (k & 1);  // the position this lane finishes
    uint32_t token = r0 / group, g = r0 % group;
    for (uint32_t r = 0; r < rn; ++r) {
        const ulonglong2* q2 = reinterpret_cast<const ulonglong2*>(qs + r * DIM + 4 * k);
        f32x2 part[POS][2];
#pragma unroll
        for (int j = 0; j < POS; ++j) part[j][0] = part[j][1] = 0ull;
#pragma unroll
        for (int s = 0; s < kSteps; ++s) {
            const ulonglong2 q = q2[s * 4];
#pragma unroll
            for (int j = 0; j < POS; ++j) {
                part[j][0] = fma2(mul2(q.x, k2[j][s][0]), one2, part[j][0]);
                part[j][1] = fma2(mul2(q.y, k2[j][s][1]), one2, part[j][1]);
            }
        }
        // an even lane keeps the even position's sums, an odd lane the odd one's; low / up: what the pair's even and odd lane had
        f32x2 low[2], up[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const f32x2 keep = odd ? part[1][u] : part[0][u];
            const f32x2 got = __shfl_xor_sync(0xffffffffu, odd ? part[0][u] : part[1][u], 1);
            low[u] = odd ? got : keep;
            up[u] = odd ? keep : got;
        }
        float sum = 0.0f;
        auto add8 = [&] {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                float x, y;
                unpack2(u < 2 ? low[u] : up[u - 2], x, y);
                sum = __fadd_rn(__fadd_rn(sum, x), y);
            }
        };
        add8();
        sum = __shfl_xor_sync(0xffffffffu, sum, 2);  // of use in the high lanes: their partner's sum of 0-7
        add8();
        if (high && mine < position + token + 1) a.scores[(size_t(token) * a.heads + kvh * group + g) * a.max_context + mine] = __fmul_rn(sum, a.scale);
        if (++g == group) {
            g = 0;
            ++token;
        }
    }
    release_next();
}

// ---- softmax ------------------------------------------------------------------------------------------------------
// Bound by the exps (f64, exact_math.h) and the rows' trip through L2. Scores stay in registers between the passes, so a
// row is read and written once: THREADS = 32 is a warp per row (rows of up to 1024 positions), 256 a CTA per row, which
// reads again what lies beyond its 16 scores a thread.
template <int THREADS, int HELD>
__global__ void __launch_bounds__(256) attn_softmax_kernel(const AttnArgs a) {
    constexpr uint32_t kRows = 256 / THREADS;
    wait_for_previous();
    __shared__ float redf[8];
    __shared__ double redd[8];
    const uint32_t row = blockIdx.x * kRows + threadIdx.x / THREADS, tid = threadIdx.x % THREADS;
    if (row >= a.n * a.heads) return;  // whole warps, and never with THREADS = 256
    const uint32_t visible = *a.position + row / a.heads + 1;
    // a sliding-window layer normalises over the last `window` positions only (src/model.cpp:1084-1088)
    const uint32_t start = a.window != 0 && visible > a.window ? visible - a.window : 0;
    const uint32_t count = visible - start;
    float* s = a.scores + size_t(row) * a.max_context + start;
    float held[HELD];
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < HELD; ++i) {
        const uint32_t p = tid + i * THREADS;
        held[i] = p < count ? s[p] : -INFINITY;
    }
#pragma unroll
    for (int i = 0; i < HELD; ++i) mx = fmaxf(mx, held[i]);
    for (uint32_t p = tid + HELD * THREADS; p < count; p += THREADS) mx = fmaxf(mx, s[p]);
    mx = warp_max(mx);
    if constexpr (THREADS > 32) {
        if ((tid & 31) == 0) redf[tid >> 5] = mx;
        __syncthreads();
        mx = redf[0];
#pragma unroll
        for (int w = 1; w < 8; ++w) mx = fmaxf(mx, redf[w]);
    }
    double part = 0.0;
#pragma unroll
    for (int i = 0; i < HELD; ++i) {
        if (uint32_t(i * THREADS) >= count) break;
        if (tid + i * THREADS < count) {
            held[i] = exact_expf(__fsub_rn(held[i], mx));
            part += double(held[i]);
        }
    }
    for (uint32_t p = tid + HELD * THREADS; p < count; p += THREADS) {
        const float e = exact_expf(__fsub_rn(s[p], mx));
        s[p] = e;
        part += double(e);
    }
    double total = warp_sum(part);
    if constexpr (THREADS > 32) {
        if ((tid & 31) == 0) redd[tid >> 5] = total;
        __syncthreads();
        total = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) total += redd[w];
    }
    const float inv = float(1.0 / total);
    release_next();
#pragma unroll
    for (int i = 0; i < HELD; ++i) {
        const uint32_t p = tid + i * THREADS;
        if (p < count) s[p] = __fmul_rn(held[i], inv);
    }
    for (uint32_t p = tid + HELD * THREADS; p < count; p += THREADS) s[p] = __fmul_rn(s[p], inv);
}

// ---- weighted sum -------------------------------------------------------------------------------------------------
// A lane owns four values of the head and R rows, two rows to a packed accumulator, and walks the positions in order: one
// warp covers R rows of a 128-wide head (2 R rows of a 64-wide one; a 256-wide head is summed as two independent 128-wide
// parts). Four values per lane because a probability read from shared memory then meets four of them - with one, the
// broadcast reads bound the kernel, see the scores. V rows and the rows' probabilities - transposed, so that four rows of a
// position are one 16-byte read - are staged in chunks of 32 positions; while one is summed the next chunk's V is on its way
// (cp.async) and its probabilities are loaded into registers.
// A position past a row's causal limit (or before its window) must not touch the row's sum: positions that every row of
// the tile sees go through the plain loop, the few at the edges through one with a test per row.
// Measured as above: 845 us with one value per thread and scalar arithmetic, 736 us now.
// grid (parts, K/V heads, row tiles), the row tile outermost and latest first.
constexpr uint32_t kChunk = 32;

template <int R>
__global__ void __launch_bounds__(128) attn_weighted_kernel(const AttnArgs a, float one) {
    extern __shared__ __align__(16) unsigned char smem[];  // V [2][kChunk][width] f16 | probabilities [kChunk][pitch] f32
    __shared__ uint32_t visible[8 * R];                    // per row of the tile
    const uint32_t parts = gridDim.x, width = a.dim / parts, lanes = width / 4;  // width: the 64 or 128 values this CTA sums
    const uint32_t tile_rows = R * (128 / lanes), pitch = tile_rows + 4;
    const uint32_t group = a.heads / a.kv_heads, kvh = blockIdx.y, doff = blockIdx.x * width, tid = threadIdx.x;
    const uint32_t rows = a.n * group, r0 = (gridDim.z - 1 - blockIdx.z) * tile_rows, rn = min(tile_rows, rows - r0);
    const uint32_t col = tid % lanes * 4, mine = tid / lanes * R;  // this lane's first value, the first of its rows
    wait_for_previous();
    const uint32_t position = *a.position, win = a.window;
    const uint32_t base_visible = position + r0 / group + 1, last_visible = position + (r0 + rn - 1) / group + 1;
    const uint32_t start_first = win != 0 && base_visible > win ? base_visible - win : 0;
    const uint32_t start_last = win != 0 && last_visible > win ? last_visible - win : 0;
    for (uint32_t i = tid; i < tile_rows; i += 128) visible[i] = i < rn ? position + (r0 + i) / group + 1 : 0;
    __half* vs = reinterpret_cast<__half*>(smem);
    float* ws = reinterpret_cast<float*>(smem + size_t(2) * kChunk * width * sizeof(__half));
    const __half* vbase = a.v_cache + size_t(kvh) * a.max_context * a.dim + doff;
    const uint32_t row_pieces = width / 8;  // 16-byte pieces of a staged V row

    f32x2 acc[R / 2][4];
#pragma unroll
    for (int i = 0; i < R / 2; ++i)
#pragma unroll
        for (int d = 0; d < 4; ++d) acc[i][d] = 0ull;
    const f32x2 one2 = pack2(one, one);

    auto request_v = [&](uint32_t c0, uint32_t buffer) {
        const uint32_t cn = min(kChunk, last_visible - c0);
        const uint32_t dst = uint32_t(__cvta_generic_to_shared(vs + buffer * kChunk * width));
        for (uint32_t i = tid; i < cn * row_pieces; i += 128) {
            const __half* src = vbase + size_t(c0 + i / row_pieces) * a.dim + i % row_pieces * 8;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 16), "l"(src) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // This thread's share of a chunk's probabilities: runs of four positions of one row, piece_step positions apart.
    constexpr int kItems = 2 * R * 4 * (kChunk / 4) / 128;  // enough for 64-wide heads, which have twice the rows
    const uint32_t items = tile_rows * (kChunk / 4) / 128, piece_row = tid % tile_rows, piece_pos = tid / tile_rows * 4, piece_step = 128 / tile_rows * 4;
    const uint32_t prow = r0 + min(piece_row, rn - 1);
    const float* wsrc = a.scores + (size_t(prow / group) * a.heads + kvh * group + prow % group) * a.max_context;
    float next[kItems][4];
    const bool whole = a.max_context % 4 == 0;  // rows start on 16-byte boundaries, and a run never leaves its row
    auto request_w = [&](uint32_t c0) {
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
            if (uint32_t(i) >= items) break;
            const uint32_t p = c0 + piece_pos + i * piece_step;
            if (whole) {
                const float4 v = p < last_visible ? *reinterpret_cast<const float4*>(wsrc + p) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                next[i][0] = v.x; next[i][1] = v.y; next[i][2] = v.z; next[i][3] = v.w;
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) next[i][k] = p + k < last_visible ? wsrc[p + k] : 0.0f;
            }
        }
    };
    const uint32_t first = start_first / kChunk * kChunk;
    request_v(first, 0);
    request_w(first);
    uint32_t buffer = 0;
    for (uint32_t c0 = first; c0 < last_visible; c0 += kChunk, buffer ^= 1) {
        const uint32_t cn = min(kChunk, last_visible - c0);
        __syncthreads();  // the previous chunk's probabilities and the other V buffer are fully consumed
        if (c0 + kChunk < last_visible) request_v(c0 + kChunk, buffer ^ 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (uint32_t(i) < items) ws[(piece_pos + i * piece_step + k) * pitch + piece_row] = next[i][k];
            }
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        if (c0 + kChunk < last_visible) request_w(c0 + kChunk);
        const __half* v = vs + buffer * kChunk * width + col;
        auto values = [&](uint32_t pp, float (&f)[4]) {
            const uint2 raw = *reinterpret_cast<const uint2*>(v + pp * width);
            const float2 f0 = __half22float2(reinterpret_cast<const __half2*>(&raw)[0]), f1 = __half22float2(reinterpret_cast<const __half2*>(&raw)[1]);
            f[0] = f0.x; f[1] = f0.y; f[2] = f1.x; f[3] = f1.y;
        };
        // positions of this chunk that every row sees: [lo, hi)
        const uint32_t lo = start_last > c0 ? min(cn, start_last - c0) : 0, hi = base_visible > c0 ? min(cn, base_visible - c0) : 0;
        auto edge = [&](uint32_t begin, uint32_t end) {
            for (uint32_t pp = begin; pp < end; ++pp) {
                float f[4];
                values(pp, f);
                const uint32_t p = c0 + pp;
#pragma unroll
                for (int i = 0; i < R / 2; ++i) {
                    const uint32_t vx = visible[mine + 2 * i], vy = visible[mine + 2 * i + 1];
                    const bool sees_x = p < vx && (win == 0 || p + win >= vx), sees_y = p < vy && (win == 0 || p + win >= vy);
                    const float wx = ws[pp * pitch + mine + 2 * i], wy = ws[pp * pitch + mine + 2 * i + 1];
#pragma unroll
                    for (int d = 0; d < 4; ++d) {
                        float x, y;
                        unpack2(acc[i][d], x, y);
                        if (sees_x) x = __fadd_rn(x, __fmul_rn(wx, f[d]));
                        if (sees_y) y = __fadd_rn(y, __fmul_rn(wy, f[d]));
                        acc[i][d] = pack2(x, y);
                    }
                }
            }
        };
        edge(0, min(lo, cn));
        if (lo < hi) {
#pragma unroll 2
            for (uint32_t pp = lo; pp < hi; ++pp) {
                float f[4];
                values(pp, f);
                const ulonglong2* w = reinterpret_cast<const ulonglong2*>(ws + pp * pitch + mine);
#pragma unroll
                for (int i = 0; i < R / 4; ++i) {
                    const ulonglong2 w4 = w[i];
#pragma unroll
                    for (int d = 0; d < 4; ++d) {
                        const f32x2 v2 = pack2(f[d], f[d]);
                        acc[2 * i][d] = fma2(mul2(w4.x, v2), one2, acc[2 * i][d]);
                        acc[2 * i + 1][d] = fma2(mul2(w4.y, v2), one2, acc[2 * i + 1][d]);
                    }
                }
            }
        }
        edge(max(lo, hi), cn);
    }
    release_next();
#pragma unroll
    for (int i = 0; i < R; ++i) {
        if (mine + i >= rn) continue;
        const uint32_t r = r0 + mine + i;
        float o[4];
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            float x, y;
            unpack2(acc[i / 2][d], x, y);
            o[d] = i & 1 ? y : x;
        }
        *reinterpret_cast<float4*>(a.out + (size_t(r / group) * a.heads + kvh * group + r % group) * a.dim + doff + col) = make_float4(o[0], o[1], o[2], o[3]);
    }
}

template <int DIM>
void launch_scores(const AttnArgs& a, uint32_t sms, cudaStream_t s) {
    constexpr uint32_t kPerCta = DIM > 128 ? 64 : 128;
    const auto kernel = [] {
        if constexpr (DIM > 128) return attn_scores_wide_kernel;
        else return attn_scores_kernel<DIM>;
    }();
    const uint32_t rows = a.n * (a.heads / a.kv_heads), chunks = (a.max_visible + kPerCta - 1) / kPerCta;
    // More rows per tile reuse the K row a thread has widened; fewer fill the GPU: the largest tile that leaves four CTAs
    // an SM, half of which the causal edge may leave without work. Few tokens have no such edge, and re-reading the K rows is
    // what they pay for: most of an SM's CTA each is enough (9 tokens at 2064 positions, 7B shape: tiles of 8 rows 18.9 us, of
    // all 36 15.4).
    const uint64_t enough = a.n <= kChainMaxTokens ? sms * 4ull / 5 : 4ull * sms;
    uint32_t tile = 64;
    while (tile > 8 && uint64_t(chunks) * a.kv_heads * ((rows + tile - 1) / tile) < enough) tile /= 2;
    static DeviceOnce once;
    if (once.first()) BK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(64 * DIM * sizeof(float))));
    launch_dependent(kernel, dim3(chunks, a.kv_heads, (rows + tile - 1) / tile), dim3(128), size_t(tile) * DIM * sizeof(float), s, a, tile, 1.0f);
}

template <int R>
void launch_weighted(const AttnArgs& a, uint32_t tiles, uint32_t parts, cudaStream_t s) {
    const uint32_t width = a.dim / parts, tile_rows = R * (512 / width);
    const size_t smem = size_t(2) * kChunk * width * sizeof(__half) + size_t(kChunk) * (tile_rows + 4) * sizeof(float);
    launch_dependent(attn_weighted_kernel<R>, dim3(parts, a.kv_heads, tiles), dim3(128), smem, s, a, 1.0f);
}

}  // namespace

void launch_attn_scores(const AttnArgs& a, uint32_t sms, cudaStream_t s) {
    if (a.dim == 64) launch_scores<64>(a, sms, s);
    else if (a.dim == 128) launch_scores<128>(a, sms, s);
    else launch_scores<256>(a, sms, s);
}

void launch_attn_softmax(const AttnArgs& a, uint32_t sms, cudaStream_t s) {
    const uint32_t softmax_rows = a.n * a.heads, widest = a.window != 0 ? std::min(a.window, a.max_visible) : a.max_visible;
    const bool many = softmax_rows >= 16 * sms;  // enough rows for a warp each (1000 positions, 144 rows: 8.7 us so, 4 with a CTA each)
    if (widest <= 512 && (many || widest <= 128)) launch_dependent(attn_softmax_kernel<32, 16>, dim3((softmax_rows + 7) / 8), dim3(256), 0, s, a);
    else if (widest <= 1024 && many) launch_dependent(attn_softmax_kernel<32, 32>, dim3((softmax_rows + 7) / 8), dim3(256), 0, s, a);
    else launch_dependent(attn_softmax_kernel<256, 16>, dim3(softmax_rows), dim3(256), 0, s, a);
}

void launch_attn_weighted(const AttnArgs& a, uint32_t sms, cudaStream_t s) {
    // More rows per lane reuse the V row it has widened (16 rows: 736 us for the case above, 8: 921), fewer fill the GPU: the
    // most that still leave one and a half CTAs an SM.
    const uint32_t rows = a.n * (a.heads / a.kv_heads), parts = (a.dim + 127) / 128, groups = 512 / (a.dim / parts);
    auto tiles = [&](uint32_t per_lane) { return (rows + per_lane * groups - 1) / (per_lane * groups); };
    auto enough = [&](uint32_t per_lane) { return uint64_t(tiles(per_lane)) * a.kv_heads * parts * 2 >= 3ull * sms; };
    if (enough(16)) launch_weighted<16>(a, tiles(16), parts, s);
    else if (enough(8)) launch_weighted<8>(a, tiles(8), parts, s);
    else launch_weighted<4>(a, tiles(4), parts, s);
}

}  // namespace bk
