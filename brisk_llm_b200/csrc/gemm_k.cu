// Multiply of a few to some hundred tokens (and, with few rows, more; gemm_k_tc.cu takes the rest) on int8 tensor cores for the
// 256-value super-block formats (Q4_K, Q5_K, Q6_K, TQ2_0) against Q8_K
// activations, with the reference's integer arithmetic and float order (src/quant.cpp:500-596):
//
//   TQ2_0  acc   = sum over the super-block of q*x            (8 MMAs of k = 32 chained in int32)
//          term  = (x.d * w.d) * float(acc - sum(x))
//   Q4_K, Q5_K  per 32-value sub-block sb: dot_sb = q*x (one MMA)   weighted += scale[sb] * dot_sb
//                                                              offsets  += min[sb] * (bsum[2sb] + bsum[2sb+1])
//          term  = x.d * (w.d * float(weighted) - w.dmin * float(offsets))
//   Q6_K   per 16-value group g: dot_g = q6*x (one k = 16 MMA) weighted += scale[g] * (dot_g - 32 * bsum[g])
//          term  = (x.d * w.d) * float(weighted)
//   out[token][row] = sum of the terms over super-blocks, in order, by the one thread that owns the output.
//
// Everything before the float expression is exact integer work, so results are bit-identical to the CPU kernels.
//
// Bound: integer multiply-adds and the shared-memory reads that feed them, not the tensor pipe. So what depends on the token
// alone is worked out once per super-block when the stage is filled - sum(x) for TQ2_0, -32 * bsum[g] for Q6_K, where it is
// the C operand of the group's MMA, and for Q4_K / Q5_K the sums of 32 as two 6-bit digits, so that two k = 16 MMAs against
// the row's eight minimums replace eight multiply-adds per output. Measured (before gemm_k_tc.cu took
// prompts of these sizes): 777 tokens, ternary 2B shape
// 30.0 -> 27.1 ms, Q5_K_M 1B shape (its Q5_K matrices went through the streaming kernel) 119.7 -> 18.6 ms; 1023 tokens of
// the Q4_K_M 1B shape 21.5 -> 20.0 ms.
// Tiling as in gemm.cu: the tile is picked from rows, tokens and row length (launch_type); stages of one super-block come
// through a cp.async ring, and targets of one type share a launch.
#include <algorithm>

#include "kernels.h"
#include "pdl.cuh"

namespace bk {
namespace {

__device__ __forceinline__ void cp16(void* smem, const void* gmem) {
    const uint32_t a = uint32_t(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(gmem) : "memory");
}
__device__ __forceinline__ void mma_k32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0));
}

// d = a x b + {c0, c1, c0, c1}: the two token columns of a thread's results start from their own values
__device__ __forceinline__ void mma_k16_from(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, int c0, int c1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%7,%8};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a0), "r"(a1), "r"(b0), "r"(c0), "r"(c1));
}
// four bits -> bit 4 of four bytes
__device__ __forceinline__ uint32_t fifth_bits(uint32_t bits) { return (((bits & 0xFu) * 0x00204081u) & 0x01010101u) << 4; }

struct KParams {
    DevMatrix m[3];
    float* out[3];
    uint32_t ldo[3];
    uint32_t first_tile[4];  // row tiles of target i: [first_tile[i], first_tile[i + 1])
    DevAct act;
    uint32_t n;
    int count, epi;
};

// Shared-memory stage of one super-block. Row strides carry 16 bytes of padding so that the 8 rows a warp's fragment
// loads touch fall into different banks.
template <int TYPE, int KM, int KN>
struct KStage {
    static constexpr bool kMins = TYPE == T_Q4_K || TYPE == T_Q5_K;
    static constexpr int kQ = TYPE == T_TQ2_0 ? 64 : TYPE == T_Q4_K ? 128 : TYPE == T_Q5_K ? 160 : 192;  // quant bytes per row and super-block
    static constexpr int kARow = kQ + 16;
    static constexpr int kA = KM * kARow;
    static constexpr int kSc = TYPE == T_TQ2_0 ? 0 : KM * 16;  // sub-block scales (and mins)
    static constexpr int kD = KM * 4;                          // d (and dmin) as f16
    static constexpr int kBRow = 256 + 16;
    static constexpr int kB = KN * kBRow;
    static constexpr int kBd = KN * 4;
    // per token: sum(x) | two runs of eight digits | 16 values -32 * bsum[g], [g][token] so that a thread's two columns are one read
    static constexpr int kBs = TYPE == T_TQ2_0 ? KN * 4 : kMins ? KN * 16 : KN * 64;
    static constexpr int kBytes = kA + kSc + kD + kB + kBd + kBs;
};

// Warps of 16 MI rows x 8 NI tokens, WR of them along the rows and WT along the tokens.
//
// KS > 1, for few tokens and long rows: KS warps on the same rows and tokens take every KS-th super-block, each with stages
// of its own. Only the sum of a row's terms is serial: the terms of a round meet in shared memory and every thread adds those
// of its outputs in super-block order. (One warp walks a super-block in 1.4 us, 2048 x 8192 Q6_K in 44 us whatever the tile.)
template <int TYPE, int MI, int NI, int WR, int WT, int KS, int STAGES, int RESIDENT>
__global__ void __launch_bounds__(WR * WT * KS * 32, RESIDENT) gemm_k_kernel(const __grid_constant__ KParams p) {
    static_assert(KS == 1 || (WR == 1 && WT == 1), "a split row has one warp per share");
    constexpr uint32_t KM = 16 * MI * WR, KN = 8 * NI * WT, ALL = WR * WT * KS * 32, THREADS = ALL / KS;  // THREADS fill a stage
    using S = KStage<TYPE, KM, KN>;
    static_assert(KM <= THREADS && KN <= THREADS, "a thread stages one row's and one token's scales at most");
    extern __shared__ __align__(16) unsigned char smem_all[];
    const uint32_t tid = threadIdx.x % THREADS, ks = threadIdx.x / THREADS, lane = tid & 31, warp = tid >> 5;
    unsigned char* smem = smem_all + size_t(ks) * STAGES * S::kBytes;
    constexpr uint32_t kOutputs = MI * NI * 128, kMine = KS > 1 ? kOutputs / ALL : 1;  // split rows: outputs of the CTA and of a thread
    float* terms = reinterpret_cast<float*>(smem_all + size_t(KS) * STAGES * S::kBytes);  // [2][KS][kOutputs]
    const uint32_t g = lane >> 2, t = lane & 3;
    int target = 0;
    if (p.count > 1 && blockIdx.x >= p.first_tile[1]) target = 1;
    if (p.count > 2 && blockIdx.x >= p.first_tile[2]) target = 2;
    const DevMatrix& m = p.m[target];
    const uint32_t row_base = (blockIdx.x - p.first_tile[target]) * KM, tok_base = blockIdx.y * KN;
    const uint32_t wr = warp % WR * (16 * MI), wt = warp / WR * (8 * NI);
    const uint32_t nsb = m.blocks, rounds = (nsb + KS - 1) / KS;  // super-blocks per row
    auto block_of = [&](uint32_t round) { return round * KS + ks; };

    auto load_weights = [&](uint32_t slot, uint32_t sb) {
        unsigned char* base = smem + size_t(slot) * S::kBytes;
        constexpr uint32_t kPieces = S::kQ / 16;
        for (uint32_t i = tid; i < KM * kPieces; i += THREADS) {
            const uint32_t r = i / kPieces, piece = i % kPieces;
            const size_t at = size_t(min(row_base + r, m.rows - 1)) * nsb + sb;
            const unsigned char* src;
            if (TYPE == T_Q6_K) {  // three planes of 64 bytes per super-block: qa | qb | qc
                const uint8_t* plane = piece < 4 ? m.qa : piece < 8 ? m.qb : m.qc;
                src = plane + at * 64 + (piece & 3) * 16;
            } else if (TYPE == T_Q5_K && piece >= 8) {
                src = m.qb + at * 32 + (piece - 8) * 16;  // the units' fifth bits, one u32 each
            } else if (TYPE == T_Q5_K) {
                src = m.qa + at * 128 + piece * 16;
            } else {
                src = m.qa + at * S::kQ + piece * 16;
            }
            cp16(base + r * S::kARow + piece * 16, src);
        }
        if (TYPE != T_TQ2_0 && tid < KM) cp16(base + S::kA + tid * 16, m.sc + (size_t(min(row_base + tid, m.rows - 1)) * nsb + sb) * 16);
    };
    auto load_tokens = [&](uint32_t slot, uint32_t sb) {
        unsigned char* bq = smem + size_t(slot) * S::kBytes + S::kA + S::kSc + S::kD;
        for (uint32_t i = tid; i < KN * 16; i += THREADS) {
            const uint32_t r = i >> 4, piece = i & 15;
            // Tokens past the last are left out: their columns of the MMAs hold whatever was there and are never stored. (A copy of
            // the last token in their place made 2 tokens slower than 16: every CTA read the same few lines over and over.)
            if (tok_base + r < p.n) cp16(bq + r * S::kBRow + piece * 16, p.act.qk + size_t(tok_base + r) * p.act.cols + sb * 256 + piece * 16);
        }
    };
    // What is too small or too raw for cp.async goes through registers, loaded a super-block before it is stored: the row's d
    // (and dmin), the token's scale and its sums of 16.
    const uint32_t srow = min(row_base + tid, m.rows - 1), stok = tok_base + tid;
    uint32_t next_d = 0;
    float next_dx = 0.0f;
    uint4 next_lo{}, next_hi{};
    auto fetch_row = [&](uint32_t sb) {
        if (tid < KM && sb < nsb) {
            if (S::kMins) next_d = reinterpret_cast<const uint32_t*>(m.d)[size_t(srow) * nsb + sb];
            else next_d = reinterpret_cast<const uint16_t*>(m.d)[size_t(srow) * nsb + sb];
        }
    };
    auto fetch_token = [&](uint32_t sb) {
        if (tid < KN && stok < p.n && sb < nsb) {
            next_dx = p.act.dk[size_t(stok) * nsb + sb];
            const uint4* sums = reinterpret_cast<const uint4*>(p.act.bs + (size_t(stok) * nsb + sb) * 16);
            next_lo = sums[0];
            next_hi = sums[1];
        }
    };
    auto store_scales = [&](uint32_t slot) {
        unsigned char* base = smem + size_t(slot) * S::kBytes;
        if (tid < KM) reinterpret_cast<uint32_t*>(base + S::kA + S::kSc)[tid] = next_d;
        if (tid < KN) {
            float* bd = reinterpret_cast<float*>(base + S::kA + S::kSc + S::kD + S::kB);
            unsigned char* bs = reinterpret_cast<unsigned char*>(bd) + S::kBd;
            const uint32_t r = tid;
            bd[r] = next_dx;
            const uint32_t w[8] = {next_lo.x, next_lo.y, next_lo.z, next_lo.w, next_hi.x, next_hi.y, next_hi.z, next_hi.w};  // two sums of 16 each
            if constexpr (TYPE == T_Q6_K) {
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    reinterpret_cast<int*>(bs)[(2 * k) * KN + r] = -32 * int(int16_t(w[k] & 0xFFFF));
                    reinterpret_cast<int*>(bs)[(2 * k + 1) * KN + r] = -32 * int(int16_t(w[k] >> 16));
                }
            } else if constexpr (TYPE == T_TQ2_0) {
                int total = 0;
#pragma unroll
                for (int k = 0; k < 8; ++k) total += int(int16_t(w[k] & 0xFFFF)) + int(int16_t(w[k] >> 16));
                reinterpret_cast<int*>(bs)[r] = total;
            } else {  // a sum of 32 is 64 * high + low with both in s8
                uint32_t low[2] = {0u, 0u}, high[2] = {0u, 0u};
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int sum = int(int16_t(w[k] & 0xFFFF)) + int(int16_t(w[k] >> 16)), l = ((sum + 32) & 63) - 32;
                    low[k >> 2] |= uint32_t(l & 0xFF) << (8 * (k & 3));
                    high[k >> 2] |= uint32_t(((sum - l) >> 6) & 0xFF) << (8 * (k & 3));
                }
                *reinterpret_cast<uint4*>(bs + r * 16) = make_uint4(low[0], low[1], high[0], high[1]);
            }
        }
    };

    float sums[kMine] = {};  // split rows
    float acc[MI][NI][4];
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < NI; ++ni)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[mi][ni][j] = 0.0f;

    // the weights of the first stages before the activations are there
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i) {
        if (block_of(i) < nsb) load_weights(i, block_of(i));
    }
    fetch_row(block_of(0));
    wait_for_previous();
    if (p.n <= 64) release_next();  // few CTAs will wait beside this kernel
    fetch_token(block_of(0));
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i) {
        if (block_of(i) < nsb) {
            load_tokens(i, block_of(i));
            store_scales(i);
        }
        fetch_row(block_of(i + 1));
        fetch_token(block_of(i + 1));
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    uint32_t slot = 0, fill = STAGES - 1;
    for (uint32_t round = 0; round < rounds; ++round) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        // the stage has landed for every thread that reads it, and the slot filled next is no longer read
        if constexpr (KS == 1) __syncthreads();
        else __syncwarp();
        if (block_of(round + STAGES - 1) < nsb) {
            load_weights(fill, block_of(round + STAGES - 1));
            load_tokens(fill, block_of(round + STAGES - 1));
            store_scales(fill);
            fetch_row(block_of(round + STAGES));
            fetch_token(block_of(round + STAGES));
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        fill = fill + 1 == STAGES ? 0 : fill + 1;
        const unsigned char* base = smem + size_t(slot) * S::kBytes;
        slot = slot + 1 == STAGES ? 0 : slot + 1;
        const bool here = block_of(round) < nsb;  // the last round of a split row may leave warps without a super-block
        if (here) {
        const unsigned char* aq = base;
        const unsigned char* asc = base + S::kA;
        const __half* ad = reinterpret_cast<const __half*>(base + S::kA + S::kSc);
        const unsigned char* bq = base + S::kA + S::kSc + S::kD;
        const float* bd = reinterpret_cast<const float*>(bq + S::kB);
        const unsigned char* bs = bq + S::kB + S::kBd;

        // integer accumulators of this super-block: [row tile][token tile][4 results]
        int weighted[MI][NI][4], offsets[MI][NI][4];  // offsets: Q4_K / Q5_K only
#pragma unroll
        for (int mi = 0; mi < MI; ++mi)
#pragma unroll
            for (int ni = 0; ni < NI; ++ni)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    weighted[mi][ni][j] = 0;
                    offsets[mi][ni][j] = 0;
                }

        if constexpr (TYPE == T_TQ2_0) {
#pragma unroll
            for (int jj = 0; jj < 2; ++jj) {  // halves of 128 values: units 2jj (k 0..15 of each run) and 2jj+1 (k 16..31)
                uint32_t w0[MI][2], w1[MI][2];
#pragma unroll
                for (int mi = 0; mi < MI; ++mi) {
                    const uint32_t r0 = wr + mi * 16 + g, r1 = r0 + 8;
                    w0[mi][0] = *reinterpret_cast<const uint32_t*>(aq + r0 * S::kARow + (2 * jj) * 16 + 4 * t);
                    w0[mi][1] = *reinterpret_cast<const uint32_t*>(aq + r0 * S::kARow + (2 * jj + 1) * 16 + 4 * t);
                    w1[mi][0] = *reinterpret_cast<const uint32_t*>(aq + r1 * S::kARow + (2 * jj) * 16 + 4 * t);
                    w1[mi][1] = *reinterpret_cast<const uint32_t*>(aq + r1 * S::kARow + (2 * jj + 1) * 16 + 4 * t);
                }
#pragma unroll
                for (int l = 0; l < 4; ++l) {  // run l: values jj*128 + 32l .. +31
                    const int kofs = jj * 128 + l * 32;
#pragma unroll
                    for (int ni = 0; ni < NI; ++ni) {
                        const unsigned char* brow = bq + (wt + ni * 8 + g) * S::kBRow + kofs;
                        const uint32_t b0 = *reinterpret_cast<const uint32_t*>(brow + 4 * t);
                        const uint32_t b1 = *reinterpret_cast<const uint32_t*>(brow + 16 + 4 * t);
#pragma unroll
                        for (int mi = 0; mi < MI; ++mi) {
                            mma_k32(weighted[mi][ni], (w0[mi][0] >> (2 * l)) & 0x03030303u, (w1[mi][0] >> (2 * l)) & 0x03030303u,
                                    (w0[mi][1] >> (2 * l)) & 0x03030303u, (w1[mi][1] >> (2 * l)) & 0x03030303u, b0, b1);
                        }
                    }
                }
            }
        } else if constexpr (S::kMins) {
#pragma unroll
            for (int ch = 0; ch < 4; ++ch) {  // 64-value chunk: sub-blocks 2ch (low nibbles) and 2ch+1 (high nibbles)
                uint32_t w0[MI][2], w1[MI][2];
                uint32_t f0[MI][2], f1[MI][2];   // Q5_K: the fifth bits of rows g and g + 8, this thread's four of each half
                int sc[MI][2][2];               // [row tile][row g / g+8][sub-block low / high]
#pragma unroll
                for (int mi = 0; mi < MI; ++mi) {
                    const uint32_t r0 = wr + mi * 16 + g, r1 = r0 + 8;
                    w0[mi][0] = *reinterpret_cast<const uint32_t*>(aq + r0 * S::kARow + (2 * ch) * 16 + 4 * t);
                    w0[mi][1] = *reinterpret_cast<const uint32_t*>(aq + r0 * S::kARow + (2 * ch + 1) * 16 + 4 * t);
                    w1[mi][0] = *reinterpret_cast<const uint32_t*>(aq + r1 * S::kARow + (2 * ch) * 16 + 4 * t);
                    w1[mi][1] = *reinterpret_cast<const uint32_t*>(aq + r1 * S::kARow + (2 * ch + 1) * 16 + 4 * t);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        sc[mi][0][h] = asc[r0 * 16 + 2 * ch + h];
                        sc[mi][1][h] = asc[r1 * 16 + 2 * ch + h];
                    }
                    if constexpr (TYPE == T_Q5_K) {
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            f0[mi][u] = *reinterpret_cast<const uint32_t*>(aq + r0 * S::kARow + 128 + (2 * ch + u) * 4) >> (4 * t);
                            f1[mi][u] = *reinterpret_cast<const uint32_t*>(aq + r1 * S::kARow + 128 + (2 * ch + u) * 4) >> (4 * t);
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int sbk = 2 * ch + h;
                    uint32_t v[MI][4];
#pragma unroll
                    for (int mi = 0; mi < MI; ++mi) {
                        v[mi][0] = (w0[mi][0] >> (4 * h)) & 0x0F0F0F0Fu;
                        v[mi][1] = (w1[mi][0] >> (4 * h)) & 0x0F0F0F0Fu;
                        v[mi][2] = (w0[mi][1] >> (4 * h)) & 0x0F0F0F0Fu;
                        v[mi][3] = (w1[mi][1] >> (4 * h)) & 0x0F0F0F0Fu;
                        if constexpr (TYPE == T_Q5_K) {
                            v[mi][0] |= fifth_bits(f0[mi][0] >> (16 * h));
                            v[mi][1] |= fifth_bits(f1[mi][0] >> (16 * h));
                            v[mi][2] |= fifth_bits(f0[mi][1] >> (16 * h));
                            v[mi][3] |= fifth_bits(f1[mi][1] >> (16 * h));
                        }
                    }
#pragma unroll
                    for (int ni = 0; ni < NI; ++ni) {
                        const unsigned char* brow = bq + (wt + ni * 8 + g) * S::kBRow + sbk * 32;
                        const uint32_t b0 = *reinterpret_cast<const uint32_t*>(brow + 4 * t);
                        const uint32_t b1 = *reinterpret_cast<const uint32_t*>(brow + 16 + 4 * t);
#pragma unroll
                        for (int mi = 0; mi < MI; ++mi) {
                            int c[4] = {0, 0, 0, 0};
                            mma_k32(c, v[mi][0], v[mi][1], v[mi][2], v[mi][3], b0, b1);
                            weighted[mi][ni][0] += sc[mi][0][h] * c[0];
                            weighted[mi][ni][1] += sc[mi][0][h] * c[1];
                            weighted[mi][ni][2] += sc[mi][1][h] * c[2];
                            weighted[mi][ni][3] += sc[mi][1][h] * c[3];
                        }
                    }
                }
            }
            // offsets = sum over the eight sub-blocks of min * sum(x): the minimums against both digits (k = 0 .. 7 of 16)
#pragma unroll
            for (int mi = 0; mi < MI; ++mi) {
                const uint32_t r0 = wr + mi * 16 + g, r1 = r0 + 8;
                const uint32_t m0 = t < 2 ? *reinterpret_cast<const uint32_t*>(asc + r0 * 16 + 8 + 4 * t) : 0u;
                const uint32_t m1 = t < 2 ? *reinterpret_cast<const uint32_t*>(asc + r1 * 16 + 8 + 4 * t) : 0u;
#pragma unroll
                for (int ni = 0; ni < NI; ++ni) {
                    const unsigned char* digits = bs + (wt + ni * 8 + g) * 16 + 4 * (t & 1);
                    int high[4] = {0, 0, 0, 0};
                    mma_k16(high, m0, m1, *reinterpret_cast<const uint32_t*>(digits + 8));
                    mma_k16(offsets[mi][ni], m0, m1, *reinterpret_cast<const uint32_t*>(digits));
#pragma unroll
                    for (int j = 0; j < 4; ++j) offsets[mi][ni][j] += 64 * high[j];
                }
            }
        } else {  // Q6_K
#pragma unroll
            for (int u = 0; u < 4; ++u) {  // unit u: 64 values = four runs of 16: k-th run at (u>>1)*128 + 32k + (u&1)*16
                uint32_t a[MI][2], b[MI][2], cc[MI][2];
#pragma unroll
                for (int mi = 0; mi < MI; ++mi) {
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {
                        const uint32_t r = wr + mi * 16 + g + hh * 8;
                        a[mi][hh] = *reinterpret_cast<const uint32_t*>(aq + r * S::kARow + u * 16 + 4 * t);
                        b[mi][hh] = *reinterpret_cast<const uint32_t*>(aq + r * S::kARow + 64 + u * 16 + 4 * t);
                        cc[mi][hh] = *reinterpret_cast<const uint32_t*>(aq + r * S::kARow + 128 + u * 16 + 4 * t);
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int grp = (u >> 1) * 8 + 2 * k + (u & 1);  // 16-value group inside the super-block
                    const int kofs = (u >> 1) * 128 + 32 * k + (u & 1) * 16;
                    uint32_t v[MI][2];
                    int sc[MI][2];
#pragma unroll
                    for (int mi = 0; mi < MI; ++mi) {
#pragma unroll
                        for (int hh = 0; hh < 2; ++hh) {
                            const uint32_t L = 0x0F0F0F0Fu, H = 0x30303030u;
                            const uint32_t lo = k == 0 ? (a[mi][hh] & L) : k == 1 ? (b[mi][hh] & L) : k == 2 ? ((a[mi][hh] >> 4) & L) : ((b[mi][hh] >> 4) & L);
                            const uint32_t hi = k == 0 ? ((cc[mi][hh] << 4) & H) : k == 1 ? ((cc[mi][hh] << 2) & H) : k == 2 ? (cc[mi][hh] & H) : ((cc[mi][hh] >> 2) & H);
                            v[mi][hh] = lo | hi;
                            sc[mi][hh] = reinterpret_cast<const int8_t*>(asc)[(wr + mi * 16 + g + hh * 8) * 16 + grp];
                        }
                    }
#pragma unroll
                    for (int ni = 0; ni < NI; ++ni) {
                        const uint32_t tb = wt + ni * 8;
                        const uint32_t b0 = *reinterpret_cast<const uint32_t*>(bq + (tb + g) * S::kBRow + kofs + 4 * t);
                        const int2 o = *reinterpret_cast<const int2*>(reinterpret_cast<const int*>(bs) + grp * KN + tb + 2 * t);
#pragma unroll
                        for (int mi = 0; mi < MI; ++mi) {
                            int c[4];
                            mma_k16_from(c, v[mi][0], v[mi][1], b0, o.x, o.y);
                            weighted[mi][ni][0] += sc[mi][0] * c[0];
                            weighted[mi][ni][1] += sc[mi][0] * c[1];
                            weighted[mi][ni][2] += sc[mi][1] * c[2];
                            weighted[mi][ni][3] += sc[mi][1] * c[3];
                        }
                    }
                }
            }
        }

        // the super-block's float term, added to the running sums in super-block order
#pragma unroll
        for (int mi = 0; mi < MI; ++mi) {
            const uint32_t r0 = wr + mi * 16 + g, r1 = r0 + 8;
            const float dw0 = __half2float(ad[2 * r0]), dw1 = __half2float(ad[2 * r1]);
            const float dm0 = S::kMins ? __half2float(ad[2 * r0 + 1]) : 0.0f, dm1 = S::kMins ? __half2float(ad[2 * r1 + 1]) : 0.0f;
#pragma unroll
            for (int ni = 0; ni < NI; ++ni) {
                const uint32_t c0 = wt + ni * 8 + 2 * t, c1 = c0 + 1;
                const float dx0 = bd[c0], dx1 = bd[c1];
                float term[4];
                if constexpr (S::kMins) {
                    term[0] = __fmul_rn(dx0, __fsub_rn(__fmul_rn(dw0, float(weighted[mi][ni][0])), __fmul_rn(dm0, float(offsets[mi][ni][0]))));
                    term[1] = __fmul_rn(dx1, __fsub_rn(__fmul_rn(dw0, float(weighted[mi][ni][1])), __fmul_rn(dm0, float(offsets[mi][ni][1]))));
                    term[2] = __fmul_rn(dx0, __fsub_rn(__fmul_rn(dw1, float(weighted[mi][ni][2])), __fmul_rn(dm1, float(offsets[mi][ni][2]))));
                    term[3] = __fmul_rn(dx1, __fsub_rn(__fmul_rn(dw1, float(weighted[mi][ni][3])), __fmul_rn(dm1, float(offsets[mi][ni][3]))));
                } else {
                    int xs0 = 0, xs1 = 0;
                    if constexpr (TYPE == T_TQ2_0) {  // sum((q-1)*x) = sum(q*x) - sum(x)
                        xs0 = reinterpret_cast<const int*>(bs)[c0];
                        xs1 = reinterpret_cast<const int*>(bs)[c1];
                    }
                    term[0] = __fmul_rn(__fmul_rn(dx0, dw0), float(weighted[mi][ni][0] - xs0));
                    term[1] = __fmul_rn(__fmul_rn(dx1, dw0), float(weighted[mi][ni][1] - xs1));
                    term[2] = __fmul_rn(__fmul_rn(dx0, dw1), float(weighted[mi][ni][2] - xs0));
                    term[3] = __fmul_rn(__fmul_rn(dx1, dw1), float(weighted[mi][ni][3] - xs1));
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if constexpr (KS == 1) acc[mi][ni][j] = __fadd_rn(acc[mi][ni][j], term[j]);
                    else terms[((round & 1) * KS + ks) * kOutputs + ((mi * NI + ni) * 4 + j) * 32 + lane] = term[j];
                }
            }
        }
        }
        if constexpr (KS > 1) {
            __syncthreads();  // the round's terms are there; those of the round before last are no longer read
            const uint32_t valid = min(uint32_t(KS), nsb - round * KS);
#pragma unroll
            for (uint32_t e = 0; e < kMine; ++e) {
                const float* mine = terms + (round & 1) * KS * kOutputs + threadIdx.x + e * ALL;
#pragma unroll
                for (int k = 0; k < KS; ++k) {
                    if (uint32_t(k) < valid) sums[e] = __fadd_rn(sums[e], mine[k * kOutputs]);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (p.n > 64) release_next();
    auto store = [&](uint32_t row, uint32_t tok, float value) {
        if (row < m.rows && tok < p.n) {
            float* o = p.out[target] + size_t(tok) * p.ldo[target] + row;
            *o = p.epi == EPI_ADD ? __fadd_rn(*o, value) : value;
        }
    };
    if constexpr (KS > 1) {
#pragma unroll
        for (uint32_t e = 0; e < kMine; ++e) {
            const uint32_t f = threadIdx.x + e * ALL, l = f & 31, j = (f >> 5) & 3, ni = (f >> 7) % NI, mi = (f >> 7) / NI;
            store(row_base + mi * 16 + (l >> 2) + (j >= 2 ? 8 : 0), tok_base + ni * 8 + 2 * (l & 3) + (j & 1), sums[e]);
        }
        return;
    }

#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < NI; ++ni)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                store(row_base + wr + mi * 16 + g + (j >= 2 ? 8 : 0), tok_base + wt + ni * 8 + 2 * t + (j & 1), acc[mi][ni][j]);
            }
}

struct KTile {
    uint32_t rows, tokens, split, threads, resident, smem;
    uint64_t alone, shared;  // ns of a super-block of Q4_K: of one CTA by itself, and per CTA of a full SM
    uint64_t percent;        // of them that this type takes
    void (*kernel)(KParams);
    mutable DeviceOnce allowed{};  // its shared memory
};

template <int TYPE, int MI, int NI, int WR, int WT, int KS, int STAGES, int RESIDENT>
KTile tile_of(uint64_t alone, uint64_t shared, uint64_t q5_k, uint64_t q6_k, uint64_t tq2_0) {
    const uint32_t stages = KS * STAGES * KStage<TYPE, 16 * MI * WR, 8 * NI * WT>::kBytes, terms = KS > 1 ? 2 * KS * MI * NI * 128 * 4 : 0;
    const uint64_t percent = TYPE == T_Q4_K ? 100 : TYPE == T_Q5_K ? q5_k : TYPE == T_Q6_K ? q6_k : tq2_0;
    return KTile{16 * MI * WR, 8 * NI * WT, KS, WR * WT * KS * 32, RESIDENT, stages + terms, alone, shared, percent,
                 gemm_k_kernel<TYPE, MI, NI, WR, WT, KS, STAGES, RESIDENT>};
}

// The tile whose busiest SM is done first, as in gemm.cu, and its time in ns; 800 ns for what a CTA does besides its super-blocks.
// Measured, Q4_K: 2048 x 8192 at 9 tokens 25 (64 x 16 tiles) / 7.9 us (16 x 16, split), 14336 x 4096 at 9 tokens 20 / 24.
template <int TYPE>
const KTile& fastest_tile(const MatTarget* targets, int count, uint32_t n, uint32_t sms, uint64_t& ns) {
    static const KTile tiles[] = {
        tile_of<TYPE, 1, 4, 4, 2, 1, 2, 2>(1250, 1060, 122, 172, 74), tile_of<TYPE, 1, 2, 4, 1, 1, 4, 4>(770, 540, 125, 143, 65),
        tile_of<TYPE, 1, 2, 1, 1, 8, 2, 1>(210, 230, 118, 137, 85), tile_of<TYPE, 1, 1, 1, 1, 4, 3, 3>(200, 137, 110, 135, 85),
    };
    const KTile* pick = nullptr;
    uint64_t best = 0;
    for (const KTile& tile : tiles) {
        uint64_t ctas = 0;
        for (int i = 0; i < count; ++i) ctas += (targets[i].m.rows + tile.rows - 1) / tile.rows;
        ctas *= (n + tile.tokens - 1) / tile.tokens;
        const uint64_t per_sm = (ctas + sms - 1) / sms, rounds = (per_sm + tile.resident - 1) / tile.resident;
        const uint64_t blocks = (targets[0].m.blocks + tile.split - 1) / tile.split * tile.split;
        const uint64_t cost = std::max(rounds * (tile.alone * blocks + 800), per_sm * tile.shared * blocks);
        if (pick == nullptr || cost < best) {
            pick = &tile;
            best = cost;
        }
    }
    ns = best * pick->percent / 100;
    return *pick;
}

const KTile& fastest_tile(const MatTarget* targets, int count, uint32_t n, uint32_t sms, uint64_t& ns) {
    switch (targets[0].m.type) {
        case T_Q4_K: return fastest_tile<T_Q4_K>(targets, count, n, sms, ns);
        case T_Q5_K: return fastest_tile<T_Q5_K>(targets, count, n, sms, ns);
        case T_Q6_K: return fastest_tile<T_Q6_K>(targets, count, n, sms, ns);
        case T_TQ2_0: return fastest_tile<T_TQ2_0>(targets, count, n, sms, ns);
        default: throw CudaError("cuda: no super-block tensor kernel for this type");
    }
}

}  // namespace

// gemm_k_tc.cu: the multiply in tensor memory, in tiles of `tokens` tokens, what it is expected to take and with which tile
void launch_gemm_k_tc(const MatTarget* targets, int count, const DevAct& act, uint32_t n, Epilogue epi, uint32_t tokens, const WaitBound& bound, uint32_t sms, cudaStream_t s);
uint64_t gemm_k_tc_ns(const MatTarget* targets, int count, uint32_t n, bool pair, uint32_t sms, uint32_t& tokens);

bool gemm_k_supports(int type) { return type == T_Q4_K || type == T_Q5_K || type == T_Q6_K || type == T_TQ2_0; }

// The kernel in tensor memory takes tiles of 128 rows and needs about 5 us around its super-blocks, so few rows or tokens stay here
// (2048 x 2048 Q4_K at 128 tokens 9.6 us here, 12.2 there; 14336 x 4096 at 64 tokens 34 and 21): whichever is estimated to be done sooner.
uint32_t super_block_tokens(const MatTarget* targets, int count, uint32_t n, bool pair, uint32_t sms) {
    uint64_t here_ns = 0;
    fastest_tile(targets, count, n, sms, here_ns);
    uint32_t tokens = 0;
    uint64_t there_ns = gemm_k_tc_ns(targets, count, n, pair, sms, tokens);
    if (pair) {
        // Here the activation is a launch of its own (a 3 us launch, 22 us for 512 x 8192 values): the tensor-memory kernel applies it
        // as it stores. The two matrices are asked about as the caller would send them.
        const uint64_t activation_ns = 3000 + uint64_t(n) * targets[0].m.rows / 220;
        there_ns = there_ns > activation_ns ? there_ns - activation_ns : 0;
    }
    return there_ns < here_ns ? tokens : 0;
}

// False, nothing launched: a gate/up pair that the caller multiplies separately.
bool launch_gemm_k(const MatTarget* targets, int count, const DevAct& act, uint32_t n, Epilogue epi, const WaitBound& bound, uint32_t sms, cudaStream_t s) {
    const bool pair = epi == EPI_SILU_MUL || epi == EPI_RELU2_MUL;
    if (const uint32_t tokens = super_block_tokens(targets, count, n, pair, sms)) {
        launch_gemm_k_tc(targets, count, act, n, epi, tokens, bound, sms, s);
        return true;
    }
    if (pair) return false;
    KParams p{};
    uint64_t ns = 0;
    const KTile& tile = fastest_tile(targets, count, n, sms, ns);
    uint32_t row_tiles = 0;
    for (int i = 0; i < count; ++i) {
        p.m[i] = targets[i].m;
        p.out[i] = targets[i].out;
        p.ldo[i] = targets[i].ldo;
        p.first_tile[i] = row_tiles;
        row_tiles += (p.m[i].rows + tile.rows - 1) / tile.rows;
    }
    p.act = act;
    p.n = n;
    p.count = count;
    p.epi = int(epi);
    if (tile.allowed.first()) BK_CUDA(cudaFuncSetAttribute(tile.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(tile.smem)));
    launch_dependent(tile.kernel, dim3(row_tiles, (n + tile.tokens - 1) / tile.tokens), dim3(tile.threads), tile.smem, s, p);
    return true;
}

}  // namespace bk
