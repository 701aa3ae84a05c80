// Prompt multiply of the 256-value super-block formats (Q4_K, Q5_K, Q6_K, TQ2_0) on the fifth-generation tensor cores, with the
// reference's integers and float order (see gemm_k.cu), so the results are the CPU's bit for bit.
//
// A sub-block's scale is an integer, and so is weighted = sum of scale[sb] * q * x over a super-block: what an MMA per sub-block
// and a scale-and-add per output on the CUDA cores compute is one contraction of length 256 over the products scale * q. Those
// take 10 to 14 bits, so they go in as two 8-bit digits (Q6_K: p = 256 high + low, Q4_K and Q5_K: 8 high + low): 16 MMAs of k = 32 accumulate the two
// digit sums of a super-block in tensor memory, and an output meets the CUDA cores once per 256 values instead of once per 32
// (Q6_K: 16). The minimums of Q4_K / Q5_K times the sums of 16 activations are exact in f16, and their sum (below 2^24) in the
// MMA's f32: one MMA of kind::f16 gives float(offsets) itself. Ternary weights need one digit and no scales.
//
// CTA tile: 128 weight rows (of one matrix, or 64 gate and 64 up rows) x 64 or 128 tokens, a CTA per SM that walks tiles until
// none are left; the roles run ahead of one another across tiles and meet only at mbarriers (bounded waits, error word: tc.cuh):
//
//   8 loader warps    thread = row = tensor-memory lane, a half super-block each: quants times scales four or two at a time, the digits
//                     in registers until the MMAs of the half before are done, then into tensor memory as the A operand. (In
//                     shared memory the digits' 64 KB per super-block, written and read, would take its bandwidth.) The
//                     minimums as f16.
//   3 helper warps    weights by TMA into one ring; activations by TMA, sums of 16 as f16 and scales into another
//   1 MMA warp        an elected lane issues. Tokens go in halves of 64 with their own accumulators, of which there are two sets:
//                     while the epilogue reads one, the other fills
//   8 epilogue warps  per super-block: accumulators as mma-style fragments (4 rows x 8 tokens a thread, so that a scale read
//                     from shared memory meets 4 or 8 outputs), the digits joined, one conversion, the reference's roundings
//
// Measured, 512 tokens, us against the tiles of gemm_k.cu: 14336 x 4096 Q4_K 228 -> 108, Q5_K 269 -> 114, Q6_K 364 -> 115, TQ2_0
// 168 -> 72; 2048 x 8192 Q4_K 67 -> 36, Q6_K 118 -> 42. Bound: not the MMAs (16 of 32 cycles each, plus one, in the 1900 cycles a
// super-block and 64 tokens take; 1400 in tiles of 128; the tensor pipe is active 11 to 26 % of the time, the issue slots 30 to 57)
// but the hand-overs around them. By cycle stamps in a copy of the kernel a wait on an mbarrier costs 71 cycles even when it is long
// complete (111 where lanes wait for several), and with neither arithmetic nor MMAs the same hand-overs take 900 cycles: the tensor
// memory beside two sets of accumulators holds the digits of one super-block only. Tiles of 128 tokens, one expansion for two
// sets, are the better ones where they fill the GPU.
#include <algorithm>

#include "formats.cuh"
#include "kernels.h"
#include "packed.cuh"
#include "pdl.cuh"
#include "tc.cuh"

namespace bk {
namespace {

constexpr uint32_t kRows = 128, kTokens = 64, kBox = 64;  // kBox: rows of a TMA box
constexpr uint32_t kLoadWarps = 8, kEpiWarps = 8, kHelpWarps = 3;
constexpr uint32_t kMmaWarp = kLoadWarps + kEpiWarps, kHelpWarp = kMmaWarp + 1, kThreads = (kHelpWarp + kHelpWarps) * 32;
constexpr uint32_t kSlots = 3;
constexpr uint32_t kACol = 384;  // tensor memory: two sets of accumulators below, two half super-blocks of digits from here on

template <int TYPE, int NT>
struct Shape {
    static constexpr bool kMins = TYPE == T_Q4_K || TYPE == T_Q5_K, kScales = TYPE != T_TQ2_0;
    static constexpr int kDigits = TYPE == T_TQ2_0 ? 1 : 2, kDigitBits = kMins ? 3 : 8;  // product = (high << kDigitBits) + low
    static constexpr uint32_t kSet = kTokens * (kDigits + (kMins ? 1 : 0));  // columns of one set: low | high | offsets
    // A weight slot: up to three planes of quants [row][kPlane bytes of a super-block], swizzled, then [row][16 scale bytes].
    static constexpr int kPlanes = TYPE == T_Q6_K ? 3 : TYPE == T_Q5_K ? 2 : 1;
    static constexpr uint32_t plane(int i) { return TYPE == T_Q4_K || (TYPE == T_Q5_K && i == 0) ? 128 : TYPE == T_Q5_K ? 32 : 64; }
    static constexpr uint32_t kQ = plane(0) + (kPlanes > 1 ? plane(1) : 0) + (kPlanes > 2 ? plane(2) : 0);  // quant bytes per row
    static constexpr uint32_t kWSlot = kRows * (kQ + (kScales ? 16 : 0));
    // A token slot: activations (two swizzled tiles of 128 values) | sums of 16 | token scales | row scales
    static constexpr uint32_t kB = NT * kTokens * 256, kSums = kMins ? NT * kTokens * 32 : 0, kMn = kMins ? kRows * 32 : 0, kXd = NT * kTokens * 4, kDw = kRows * 8;
    static constexpr uint32_t kSlot = (kB + kSums + kXd + kDw + 1023) / 1024 * 1024;
    // at least half of an SM's: a second CTA beside the first would only wait for its tensor memory
    static constexpr uint32_t smem(bool pair) { return std::max(1024 + kSlots * (kWSlot + kSlot) + 4 * kMn + (pair ? 16384u : 0u), 120u * 1024); }
    static_assert(2 * kSet <= kACol && kWSlot % 1024 == 0);
};

struct KtParams {
    CUtensorMap quants[3][3], scales[3], tokens;  // [target][plane]
    DevMatrix m[3];
    float* out[3];
    uint32_t ldo[3];
    uint32_t first_tile[4];  // row tiles of target i: [first_tile[i], first_tile[i + 1])
    DevAct act;
    uint32_t n, tok_tiles, tiles;
    int count, epi;
    float one;
    WaitBound bound;
};

// Four products of 16 bits, in even and odd bytes' order -> the four low bytes and the four high bytes.
__device__ __forceinline__ void digits(uint32_t even, uint32_t odd, uint32_t& low, uint32_t& high) {
    low = __byte_perm(even, odd, 0x6240);
    high = __byte_perm(even, odd, 0x7351);
}

// 16 bytes of a swizzled plane of `width` bytes per row: piece `c` of row `r`.
__device__ __forceinline__ uint4 piece(const unsigned char* plane, uint32_t width, uint32_t r, uint32_t c) {
    const uint32_t turned = width == 128 ? c ^ (r & 7) : width == 64 ? c ^ ((r >> 1) & 3) : c ^ ((r >> 2) & 1);
    return *reinterpret_cast<const uint4*>(plane + r * width + turned * 16);
}

// Row r's half super-block h (values 128 h ..) of the slot: the digits of four sub-blocks of 32, 8 registers each.
template <int TYPE, class S>
__device__ __forceinline__ void expand_half(const unsigned char* slot, uint32_t r, uint32_t h, uint32_t (&lo)[32], uint32_t (&hi)[32]) {
    uint4 sc{};
    if (S::kScales) sc = *reinterpret_cast<const uint4*>(slot + kRows * S::kQ + r * 16);
    if constexpr (S::kMins) {
        // scale = 8 high + low, six bits: either digit times q stays below 256, so a multiplication makes four products at once
        const uint32_t s4 = h == 0 ? sc.x : sc.y;
        uint32_t f[4] = {};  // Q5_K: the fifth bits of four units
        if constexpr (TYPE == T_Q5_K) {
            const uint4 f4 = piece(slot + kRows * 128, 32, r, h);
            f[0] = f4.x; f[1] = f4.y; f[2] = f4.z; f[3] = f4.w;
        }
        // four bits -> bit 4 of four bytes
        auto fifth = [](uint32_t bits) { return ((bits & 0xFu) * 0x02040810u) & 0x10101010u; };
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const uint32_t s0 = (s4 >> (16 * g)) & 0x3F, s1 = (s4 >> (16 * g + 8)) & 0x3F;
            const uint4 a = piece(slot, 128, r, h * 4 + 2 * g), b = piece(slot, 128, r, h * 4 + 2 * g + 1);
            const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                uint32_t v0 = w[i] & 0x0F0F0F0Fu, v1 = (w[i] >> 4) & 0x0F0F0F0Fu;
                if constexpr (TYPE == T_Q5_K) {
                    v0 |= fifth(f[2 * g + i / 4] >> (4 * (i & 3)));
                    v1 |= fifth(f[2 * g + i / 4] >> (16 + 4 * (i & 3)));
                }
                lo[16 * g + i] = v0 * (s0 & 7);
                hi[16 * g + i] = v0 * (s0 >> 3);
                lo[16 * g + 8 + i] = v1 * (s1 & 7);
                hi[16 * g + 8 + i] = v1 * (s1 >> 3);
            }
        }
    } else if constexpr (TYPE == T_Q6_K) {
        const uint32_t s8[2] = {h == 0 ? sc.x : sc.z, h == 0 ? sc.y : sc.w};  // scales of the half's eight groups of 16
#pragma unroll
        for (int u = 0; u < 2; ++u) {  // the units that hold the first and the last 16 values of each sub-block
            const uint4 av = piece(slot, 64, r, h * 2 + u), bv = piece(slot + kRows * 64, 64, r, h * 2 + u), cv = piece(slot + kRows * 128, 64, r, h * 2 + u);
            const uint32_t a[4] = {av.x, av.y, av.z, av.w}, b[4] = {bv.x, bv.y, bv.z, bv.w}, c[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {  // sub-block k
                const int s = int(int8_t(s8[k >> 1] >> (8 * (2 * (k & 1) + u))));
                // scale * (q - 32) + 2^15 in each 16-bit lane, never negative: the high byte's top bit flipped makes it signed
                const uint32_t offset = uint32_t(32768 - 32 * s) * 0x00010001u;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t base = k & 1 ? b[i] : a[i];
                    const uint32_t low4 = k < 2 ? base & 0x0F0F0F0Fu : (base >> 4) & 0x0F0F0F0Fu;
                    const uint32_t top2 = (k == 0 ? c[i] << 4 : k == 1 ? c[i] << 2 : k == 2 ? c[i] : c[i] >> 2) & 0x30303030u;
                    const uint32_t v = low4 | top2;
                    const int at = 8 * k + 4 * u + i;
                    digits((v & 0x00FF00FFu) * uint32_t(s) + offset, __byte_perm(v, 0, 0x4341) * uint32_t(s) + offset, lo[at], hi[at]);
                    hi[at] ^= 0x80808080u;
                }
            }
        }
    } else {  // ternary: q - 1 as signed bytes
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint4 q = piece(slot, 64, r, h * 2 + u);
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int l = 0; l < 4; ++l)
#pragma unroll
                for (int i = 0; i < 4; ++i) lo[8 * l + 4 * u + i] = (((w[i] >> (2 * l)) & 0x03030303u) + 0x7F7F7F7Fu) ^ 0x80808080u;
        }
    }
}

template <int TYPE, int NT, bool PAIR>
__global__ void __launch_bounds__(kThreads, 1) gemm_kt_kernel(const __grid_constant__ KtParams p) {
    using S = Shape<TYPE, NT>;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t a_full[2], a_free[2], d_full[2], d_free[2], w_full[kSlots], w_free[kSlots], b_full[kSlots], b_free[kSlots];
    __shared__ __align__(8) uint64_t drained;
    __shared__ uint32_t tmem_slot, stored;
    unsigned char* const weights = smem_raw + (1024 - saddr(smem_raw) % 1024) % 1024;  // swizzled tiles lie on 1024-byte boundaries
    unsigned char* const slots = weights + kSlots * S::kWSlot;
    unsigned char* const minimums = slots + kSlots * S::kSlot;  // of the rows, as an f16 operand, for four super-blocks
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t nsb = p.m[0].blocks;  // super-blocks per row, the same for every target
    const uint32_t my_tiles = (p.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x, total = my_tiles * nsb;

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&a_full[i], kLoadWarps / 2);
            mbar_init(&a_free[i], 1);
            mbar_init(&d_full[i], 1);
            mbar_init(&d_free[i], kEpiWarps);
        }
        for (uint32_t i = 0; i < kSlots; ++i) {
            mbar_init(&w_full[i], 1);
            mbar_init(&w_free[i], kLoadWarps);
            mbar_init(&b_full[i], kHelpWarps);  // two warps that store, one copy
            mbar_init(&b_free[i], 1 + kEpiWarps);
        }
        mbar_init(&drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {  // all 512 columns: one CTA per SM
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_slot);
    bool dead = false;  // a wait of this lane gave up
    auto report = [&] { atomicOr(p.bound.error, 1u); };
    // Of a thread that asked for copies or MMAs: the barriers on which they are counted, and how often.
    uint64_t* asked_on = &drained;
    uint32_t asked = 0;

    auto target_of = [&](uint32_t row_tile) {
        int target = 0;
        if (!PAIR) {
            if (p.count > 1 && row_tile >= p.first_tile[1]) target = 1;
            if (p.count > 2 && row_tile >= p.first_tile[2]) target = 2;
        }
        return target;
    };
    // This CTA's super-blocks one after the other, tile after tile.
    struct Walk {
        uint32_t tile, sb;
        __device__ bool next(uint32_t nsb) {  // true: a new tile begins
            if (++sb < nsb) return false;
            sb = 0;
            tile += gridDim.x;
            return true;
        }
    };

    if (warp < kLoadWarps) {
        // ---- loaders ----
        const uint32_t h = warp >> 2, r = (warp & 3) * 32 + lane, ta = tmem + (((warp & 3) * 32) << 16) + kACol + h * 64;
        for (uint32_t it = 0; it < total; ++it) {
            const uint32_t w = it % kSlots;
            mbar_wait(&w_full[w], (it / kSlots) & 1, dead, p.bound.cycles);
            uint32_t lo[32], hi[32];
            expand_half<TYPE, S>(weights + w * S::kWSlot, r, h, lo, hi);
            if constexpr (S::kMins) {  // this half's four minimums, each twice: for the sums of 16 on either side of a sub-block.
                // (The MMA that read this place is four super-blocks old: the one after it has been waited for.)
                const uint32_t m4 = *reinterpret_cast<const uint32_t*>(weights + w * S::kWSlot + kRows * S::kQ + r * 16 + 8 + h * 4);
                uint32_t v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t bits = 0x64006400u | ((m4 >> (8 * j)) & 0xFFu) * 0x00010001u;  // 1024 + min, exact in f16
                    const __half2 f = __hsub2(*reinterpret_cast<const __half2*>(&bits), __half2half2(__ushort_as_half(0x6400)));
                    v[j] = *reinterpret_cast<const uint32_t*>(&f);
                }
                *reinterpret_cast<uint4*>(minimums + (it & 3) * S::kMn + h * (kRows * 16) + r * 16) = make_uint4(v[0], v[1], v[2], v[3]);
                async_proxy_fence();
            }
            if (it > 0) mbar_wait(&a_free[h], (it - 1) & 1, dead, p.bound.cycles);
            __syncwarp();
            tc_fence_after();
            tmem_st16(ta, *reinterpret_cast<const uint32_t(*)[16]>(lo));
            tmem_st16(ta + 16, *reinterpret_cast<const uint32_t(*)[16]>(lo + 16));
            if (S::kDigits == 2) {
                tmem_st16(ta + 32, *reinterpret_cast<const uint32_t(*)[16]>(hi));
                tmem_st16(ta + 48, *reinterpret_cast<const uint32_t(*)[16]>(hi + 16));
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && !dead) {
                mbar_arrive(&a_full[h]);
                mbar_arrive(&w_free[w]);
            }
        }
        if (dead) report();
    } else if (warp >= kHelpWarp) {
        // ---- helpers ----
        // One warp copies: weights by TMA. The other two: a thread has two rows' d, two runs of eight sums and a token's scale,
        // loaded a super-block ahead; their first thread asks for the activations.
        Walk at{blockIdx.x, 0};
        const bool leader = elect_one();
        if (warp == kHelpWarp) {
            asked_on = w_full;
            for (uint32_t it = 0; it < total && it != p.bound.withheld; ++it, at.next(nsb)) {
                const uint32_t w = it % kSlots;
                if (it >= kSlots) mbar_wait(&w_free[w], (it / kSlots - 1) & 1, dead, p.bound.cycles);
                __syncwarp();
                const uint32_t row_tile = at.tile / p.tok_tiles;
                const int target = target_of(row_tile);
                const uint32_t row = (row_tile - p.first_tile[target]) * (PAIR ? kRows / 2 : kRows);
                if (leader && !dead) {
                    ++asked;
                    mbar_expect(&w_full[w], S::kWSlot);
#pragma unroll
                    for (uint32_t half = 0; half < 2; ++half) {
                        const int m = PAIR ? int(half) : target;
                        const uint32_t y = PAIR ? row : row + half * kBox;
                        uint32_t dst = saddr(weights + w * S::kWSlot);
#pragma unroll
                        for (int i = 0; i < S::kPlanes; ++i) {
                            tma_load(dst + half * kBox * S::plane(i), &p.quants[m][i], at.sb * S::plane(i), y, &w_full[w]);
                            dst += kRows * S::plane(i);
                        }
                        if (S::kScales) tma_load(dst + half * kBox * 16, &p.scales[m], at.sb * 16, y, &w_full[w]);
                    }
                }
                __syncwarp();
            }
        } else {
            const uint32_t hid = tid - (kHelpWarp + 1) * 32;
            const uint8_t* row_d[2];  // of this thread's rows, at the tile's first super-block
            constexpr uint32_t kDBytes = S::kMins ? 4 : 2;
            auto enter_tile = [&] {
                const uint32_t row_tile = at.tile / p.tok_tiles;
                const int target = target_of(row_tile);
#pragma unroll
                for (uint32_t k = 0; k < 2; ++k) {
                    const uint32_t row = (row_tile - p.first_tile[target]) * (PAIR ? kRows / 2 : kRows) + (PAIR ? 0 : k * 64) + hid;
                    const DevMatrix& m = p.m[PAIR ? int(k) : target];
                    row_d[k] = reinterpret_cast<const uint8_t*>(m.d) + size_t(min(row, m.rows - 1)) * nsb * kDBytes;
                }
            };
            uint32_t d[2] = {0u, 0u};
            uint4 sums[2 * NT];
            float xd[NT];
#pragma unroll
            for (uint32_t k = 0; k < 2 * NT; ++k) sums[k] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (uint32_t k = 0; k < NT; ++k) xd[k] = 0.0f;
            auto fetch_rows = [&] {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    if (S::kMins) d[k] = __ldg(reinterpret_cast<const uint32_t*>(row_d[k]) + at.sb);
                    else d[k] = __ldg(reinterpret_cast<const uint16_t*>(row_d[k]) + at.sb);
                }
            };
            auto fetch_tokens = [&] {
                const uint32_t tok_base = at.tile % p.tok_tiles * (kTokens * NT);
#pragma unroll
                for (uint32_t k = 0; k < NT; ++k) {
                    const uint32_t tok = tok_base + k * 64 + hid;
                    if (tok < p.n) xd[k] = p.act.dk[size_t(tok) * nsb + at.sb];
                }
                if constexpr (S::kMins) {
#pragma unroll
                    for (uint32_t k = 0; k < 2 * NT; ++k) {
                        const uint32_t tok = tok_base + k * 32 + (hid >> 1);
                        if (tok < p.n) sums[k] = *reinterpret_cast<const uint4*>(p.act.bs + (size_t(tok) * nsb + at.sb) * 16 + (hid & 1) * 8);
                    }
                }
            };
            enter_tile();
            fetch_rows();
            wait_for_previous();
            fetch_tokens();
            for (uint32_t it = 0; it < total; ++it) {
                const uint32_t b = it % kSlots;
                if (it >= kSlots) mbar_wait(&b_free[b], (it / kSlots - 1) & 1, dead, p.bound.cycles);
                __syncwarp();
                unsigned char* bslot = slots + b * S::kSlot;
                if (warp == kHelpWarp + 1 && leader && !dead) {
                    mbar_expect(&b_full[b], S::kB);
                    const uint32_t y = at.tile % p.tok_tiles * (kTokens * NT);
#pragma unroll
                    for (uint32_t k = 0; k < 2 * NT; ++k) tma_load(saddr(bslot) + k * (kTokens * 128), &p.tokens, at.sb * 256 + (k & 1) * 128, y + (k >> 1) * kTokens, &b_full[b]);
                }
                __syncwarp();
#pragma unroll
                for (uint32_t k = 0; k < 2; ++k) {
                    reinterpret_cast<float2*>(bslot + S::kB + S::kSums + S::kXd)[k * 64 + hid] = __half22float2(*reinterpret_cast<const __half2*>(&d[k]));
                }
#pragma unroll
                for (uint32_t k = 0; k < NT; ++k) reinterpret_cast<float*>(bslot + S::kB + S::kSums)[k * 64 + hid] = xd[k];
                if constexpr (S::kMins) {
#pragma unroll
                    for (uint32_t k = 0; k < 2 * NT; ++k) {
                        const uint32_t w[4] = {sums[k].x, sums[k].y, sums[k].z, sums[k].w}, token = k * 32 + (hid >> 1);
                        uint32_t v[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {  // at most 16 * 128 in magnitude: exact in f16
                            const __half2 f = __halves2half2(__short2half_rn(short(w[j] & 0xFFFF)), __short2half_rn(short(w[j] >> 16)));
                            v[j] = *reinterpret_cast<const uint32_t*>(&f);
                        }
                        *reinterpret_cast<uint4*>(bslot + S::kB + token / 64 * (kTokens * 32) + (hid & 1) * (kTokens * 16) + token % 64 * 16) = make_uint4(v[0], v[1], v[2], v[3]);
                    }
                }
                if (S::kMins) async_proxy_fence();
                __syncwarp();
                if (leader && !dead) {
                    mbar_arrive(&b_full[b]);
                    ++asked;
                }
                const bool new_tile = at.next(nsb);
                if (it + 1 < total) {
                    if (new_tile) enter_tile();
                    fetch_rows();
                    fetch_tokens();
                }
            }
            // A slot is full once both warps have arrived. Should the other one have given up first, its arrivals are made here.
            if (warp != kHelpWarp + 1 && leader) stored = asked;
            __syncwarp();
            asm volatile("bar.sync 3, 64;" ::: "memory");
            if (warp == kHelpWarp + 1) {
                asked_on = b_full;
                if (leader) for (uint32_t i = *reinterpret_cast<volatile uint32_t*>(&stored); i < asked; ++i) mbar_arrive(&b_full[i % kSlots]);
            } else {
                asked = 0;
            }
        }
        if (dead) report();
    } else if (warp == kMmaWarp) {
        // ---- MMAs: one elected lane ----
        constexpr uint32_t kLow = instr_i8(TYPE == T_TQ2_0, kTokens), kHigh = instr_i8(TYPE == T_Q6_K, kTokens);
        const bool leader = elect_one();
        auto issue = [&] {
            for (uint32_t it = 0; it < total; ++it) {
                const uint32_t b = it % kSlots, base = saddr(slots + b * S::kSlot);
#pragma unroll
                for (uint32_t nt = 0; nt < NT; ++nt) {
                    const uint32_t i = it * NT + nt, set = i & 1, d = tmem + set * S::kSet;
                    const uint64_t bd = smem_desc_swizzled(base + nt * (kTokens * 256));
                    // a free set of accumulators (from the third use on), the activations, the first half's digits
                    if (!mbar_wait_all(lane == 0 ? &d_free[set] : lane == 1 ? &a_full[0] : &b_full[b], lane == 0 ? ((i >> 1) - 1) & 1 : lane == 1 ? it & 1 : (it / kSlots) & 1, i >= 2 ? 0 : 1,
                                       nt == 0 ? 3 : 1, p.bound.cycles)) {
                        if (lane == 0) report();
                        return;
                    }
#pragma unroll
                    for (uint32_t h = 0; h < 2; ++h) {
                        if (nt == 0 && h == 1) {
                            mbar_wait(&a_full[1], it & 1, dead, p.bound.cycles);
                            __syncwarp();
                        }
                        tc_fence_after();
                        // (Where the wait for the digits gave up, these MMAs run on what is there, and the next wait ends the walk: asking
                        // here as well took 0.2 % of a Q4_K prompt, 1.7 % of a ternary one.)
                        if (leader) {
                            asked = 1;
                            if (S::kMins && h == 1) {
                                mma_f16_ss(d + 2 * kTokens, smem_desc(saddr(minimums + (it & 3) * S::kMn), kRows * 16, 128),
                                           smem_desc(base + S::kB + nt * (kTokens * 32), kTokens * 16, 128), instr_f16(kTokens));
                            }
#pragma unroll
                            for (uint32_t j = 0; j < 4; ++j) {
                                const uint32_t a = tmem + kACol + h * 64 + j * 8;
                                mma_i8_ts(d, a, bd + (h * (kTokens * 128) + j * 32) / 16, kLow, h + j != 0);
                                if (S::kDigits == 2) mma_i8_ts(d + kTokens, a + 32, bd + (h * (kTokens * 128) + j * 32) / 16, kHigh, h + j != 0);
                            }
                            if (nt + 1 == NT) mma_commit(&a_free[h]);
                            if (h == 1) mma_commit(&d_full[set]);
                            if (h == 1 && nt + 1 == NT) mma_commit(&b_free[b]);
                        }
                        __syncwarp();
                    }
                }
            }
        };
        issue();
        if (dead) report();
        // One commit behind all others: the MMAs, and the arrivals of the last commits (which nobody else waits for), are through.
        if (asked != 0) mma_commit(&drained);
    } else {
        // ---- epilogue ----
        const uint32_t quarter = warp & 3, part = (warp - kLoadWarps) >> 2;  // tensor-memory lanes 32 quarter .., token columns 32 part ..
        const uint32_t g = lane >> 2, t = lane & 3;
        const uint32_t mine = tmem + ((quarter * 32) << 16) + part * 32;
        const f32x2 one2 = pack2(p.one, p.one), minus2 = pack2(-p.one, -p.one);
        wait_for_previous();
        uint32_t it = 0;
        auto finish = [&] {
            for (uint32_t tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
                f32x2 acc[NT][2][4][2];  // [tokens 64 ..][16 lanes][8 columns][lane g / g + 8]
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int c = 0; c < 4; ++c) acc[nt][h][c][0] = acc[nt][h][c][1] = 0ull;
                for (uint32_t sb = 0; sb < nsb; ++sb, ++it) {
                    const uint32_t b = it % kSlots;
                    const unsigned char* bslot = slots + b * S::kSlot;
                    const float2* dw = reinterpret_cast<const float2*>(bslot + S::kB + S::kSums + S::kXd) + quarter * 32 + g;
                    float2 rs[2][2];
#pragma unroll
                    for (uint32_t nt = 0; nt < NT; ++nt) {
                        const uint32_t i = it * NT + nt, set = i & 1, at = mine + set * S::kSet;
                        // the accumulators and the scales
                        if (!mbar_wait_all(lane == 0 ? &d_full[set] : &b_full[b], lane == 0 ? (i >> 1) & 1 : (it / kSlots) & 1, 0, nt == 0 ? 2 : 1, p.bound.cycles)) {
                            if (lane == 0) report();
                            if (PAIR) {  // the warps of a pair meet at barriers: twice for every tile and half of its tokens
                                for (uint32_t left = tile; left < p.tiles; left += gridDim.x) {
                                    for (int k = 0; k < 2 * NT; ++k) asm volatile("bar.sync 2, 256;" ::: "memory");
                                }
                            }
                            return;
                        }
                        tc_fence_after();
                        const f32x2* xd = reinterpret_cast<const f32x2*>(bslot + S::kB + S::kSums) + nt * 32 + part * 16 + t;
                        if (nt == 0) {
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                rs[h][0] = dw[h * 16];
                                rs[h][1] = dw[h * 16 + 8];
                            }
                        }
                        f32x2 xs[4];
#pragma unroll
                        for (int c = 0; c < 4; ++c) xs[c] = xd[c * 4];
#pragma unroll
                        for (int k = 0; k < 8; ++k) {  // 16 lanes x 8 columns at a time
                            const int h = k >> 2, c = k & 3;
                            const uint32_t from = at + (uint32_t(h * 16) << 16) + c * 8;
                            uint32_t low[4], high[4], off[4];
                            tmem_ld_frag1(from, low);
                            if (S::kDigits == 2) tmem_ld_frag1(from + kTokens, high);
                            if (S::kMins) tmem_ld_frag1(from + 2 * kTokens, off);
                            tmem_wait_ld();
                            if (k == 7) {
                                tc_fence_before();
                                __syncwarp();
                                if (lane == 0) {
                                    mbar_arrive(&d_free[set]);
                                    if (nt + 1 == NT) mbar_arrive(&b_free[b]);  // the scales are in registers
                                }
                            }
#pragma unroll
                            for (int r = 0; r < 2; ++r) {
                                auto joined = [&](int e) { return float(int(S::kDigits == 2 ? (high[2 * r + e] << S::kDigitBits) + low[2 * r + e] : low[2 * r + e])); };
                                const f32x2 sum2 = pack2(joined(0), joined(1)), dw2 = pack2(rs[h][r].x, rs[h][r].x);
                                f32x2 term;
                                if constexpr (S::kMins) {  // x.d * (d * weighted - dmin * offsets)
                                    term = mul2(xs[c], fma2(mul2(pack2(rs[h][r].y, rs[h][r].y), pack2(off[2 * r], off[2 * r + 1])), minus2, mul2(dw2, sum2)));
                                } else {  // (x.d * d) * weighted
                                    term = mul2(mul2(xs[c], dw2), sum2);
                                }
                                acc[nt][h][c][r] = fma2(term, one2, acc[nt][h][c][r]);
                            }
                        }
                    }
                }
                const uint32_t row_tile = tile / p.tok_tiles, tok_base = tile % p.tok_tiles * (kTokens * NT);
                const int target = target_of(row_tile);
                if (tile + gridDim.x >= p.tiles) release_next();
                // (a pair: lanes 0 - 15 of a quarter's gate rows are finished there, 16 - 31 on the up side)
                const uint32_t row_base = (row_tile - p.first_tile[target]) * (PAIR ? kRows / 2 : kRows) + (PAIR ? (quarter & 1) * 32 + (quarter >> 1) * 16 : quarter * 32) + g;
                if constexpr (PAIR) {
                    // Gate rows are with quarters 0 and 1, the same up rows with 2 and 3. Each side sends the other half of its sums and
                    // applies the activation to the rest: sums 0 .. 7 of a token half stay on the gate side, 8 .. 15 go to the up side.
                    f32x2* exchange = reinterpret_cast<f32x2*>(minimums + 4 * S::kMn) + part * 64 + (quarter & 1) * 32 + lane;
                    const bool up_side = quarter >= 2;
                    __syncwarp();
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            const f32x2 low = acc[nt][0][(k >> 1) & 3][k & 1], high = acc[nt][1][(k >> 1) & 3][k & 1];
                            exchange[(up_side ? k : 8 + k) * 128] = up_side ? low : high;
                        }
                        asm volatile("bar.sync 2, 256;" ::: "memory");
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            const f32x2 mine2 = up_side ? acc[nt][1][(k >> 1) & 3][k & 1] : acc[nt][0][(k >> 1) & 3][k & 1], other2 = exchange[(up_side ? 8 + k : k) * 128];
                            float g0, g1, u0, u1;
                            unpack2(up_side ? other2 : mine2, g0, g1);
                            unpack2(up_side ? mine2 : other2, u0, u1);
                            if (tok_base + nt * 64 + part * 32 + (k >> 1) * 8 < p.n) {  // of these eight tokens, some exist
                                acc[nt][0][(k >> 1) & 3][k & 1] =
                                    p.epi == EPI_SILU_MUL ? pack2(silu_mul(g0, u0), silu_mul(g1, u1)) : pack2(relu2_mul(g0, u0), relu2_mul(g1, u1));
                            }
                        }
                        asm volatile("bar.sync 2, 256;" ::: "memory");  // the exchange may be overwritten
                    }
                }
                float* const out = p.out[target];
                const uint32_t rows = p.m[target].rows, ldo = p.ldo[target];
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const uint32_t tok = tok_base + nt * 64 + part * 32 + c * 8 + 2 * t + e;
                            if (tok >= p.n) continue;
                            float* o = out + size_t(tok) * ldo;
#pragma unroll
                            for (int h = 0; h < (PAIR ? 1 : 2); ++h)
#pragma unroll
                                for (int r = 0; r < 2; ++r) {
                                    const uint32_t row = row_base + h * 16 + r * 8;
                                    float x, y;
                                    unpack2(acc[nt][h][c][r], x, y);
                                    const float value = e == 0 ? x : y;
                                    if (row < rows) o[row] = p.epi == EPI_ADD ? __fadd_rn(o[row], value) : value;
                                }
                        }
            }
        };
        finish();
    }
    // Copies are complete by now unless a wait gave up; MMAs and their commits' arrivals in any case only behind this.
    for (uint32_t i = asked < kSlots ? 0 : asked - kSlots; i < asked; ++i) mbar_drain(&asked_on[i % kSlots], (i / kSlots) & 1);
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

template <int TYPE, int NT, bool PAIR>
void launch_tile(KtParams& p, uint32_t sms, cudaStream_t s) {
    using S = Shape<TYPE, NT>;
    constexpr uint32_t smem = S::smem(PAIR);
    static_assert(smem <= 226 * 1024);
    static DeviceOnce once;
    if (once.first()) BK_CUDA(cudaFuncSetAttribute(gemm_kt_kernel<TYPE, NT, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    p.tok_tiles = (p.n + kTokens * NT - 1) / (kTokens * NT);
    uint32_t row_tiles = 0;
    const uint32_t per_tile = PAIR ? kRows / 2 : kRows;
    for (int i = 0; i < p.count; ++i) {
        const DevMatrix& m = p.m[i];
        if (i == 0 || !PAIR) {
            p.first_tile[i] = row_tiles;
            row_tiles += (m.rows + per_tile - 1) / per_tile;
        }
        const uint8_t* planes[3] = {m.qa, m.qb, m.qc};
        for (int k = 0; k < S::kPlanes; ++k) p.quants[i][k] = tensor_map(planes[k], uint64_t(m.blocks) * S::plane(k), m.rows, S::plane(k), kBox);
        if (S::kScales) p.scales[i] = tensor_map(m.sc, uint64_t(m.blocks) * 16, m.rows, 16, kBox);
    }
    p.tokens = tensor_map(p.act.qk, p.act.cols, p.n, 128, kTokens);
    p.tiles = row_tiles * p.tok_tiles;
    launch_dependent(gemm_kt_kernel<TYPE, NT, PAIR>, dim3(std::min(p.tiles, sms)), dim3(kThreads), smem, s, p);
}

template <int TYPE>
void launch_type(KtParams& p, bool pair, int halves, uint32_t sms, cudaStream_t s) {
    if (halves == 2) pair ? launch_tile<TYPE, 2, true>(p, sms, s) : launch_tile<TYPE, 2, false>(p, sms, s);
    else pair ? launch_tile<TYPE, 1, true>(p, sms, s) : launch_tile<TYPE, 1, false>(p, sms, s);
}

}  // namespace

CUtensorMap tensor_map(const void* base, uint64_t row_bytes, uint64_t rows, uint32_t box_bytes, uint32_t box_rows) {
    using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult found{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess) fn = nullptr;
        return reinterpret_cast<Encode>(fn);
    }();
    if (encode == nullptr) throw CudaError("cuda: the driver has no cuTensorMapEncodeTiled");
    CUtensorMap map;
    const cuuint64_t dims[2] = {row_bytes, rows}, strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_bytes, box_rows}, steps[2] = {1, 1};
    const CUtensorMapSwizzle swizzle = box_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : box_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : box_bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE;
    if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
        throw CudaError("cuda: cuTensorMapEncodeTiled refused a matrix");
    }
    return map;
}

// ns that `count` targets (a pair: gate and up) take with tiles of 64 `halves` tokens: the busiest SM's tiles one after the other.
// Measured: ns of a super-block in either tile, 1.2 us of activation for every 64 tokens of a pair's tile, and 5 us before the first
// and after the last (3.5 where the same multiply is repeated; among other kernels its start overlaps less of theirs).
static uint64_t tile_ns(const MatTarget* targets, int count, uint32_t n, bool pair, int halves, uint32_t sms) {
    const int type = targets[0].m.type;
    const uint64_t one = type == T_Q4_K ? 1020 : type == T_Q5_K ? 1070 : type == T_Q6_K ? 1130 : 610;
    const uint64_t two = type == T_Q4_K ? 1480 : type == T_Q5_K ? 1610 : type == T_Q6_K ? 1600 : 880;
    uint64_t tiles = 0;
    for (int i = 0; i < (pair ? 1 : count); ++i) tiles += (targets[i].m.rows + (pair ? kRows / 2 : kRows) - 1) / (pair ? kRows / 2 : kRows);
    tiles *= (n + kTokens * halves - 1) / (kTokens * halves);
    return (tiles + sms - 1) / sms * (targets[0].m.blocks * (halves == 2 ? two : one) + (pair ? 1200 * halves : 0)) + 5000;
}

uint64_t gemm_k_tc_ns(const MatTarget* targets, int count, uint32_t n, bool pair, uint32_t sms, uint32_t& tokens) {
    const uint64_t one = tile_ns(targets, count, n, pair, 1, sms), two = tile_ns(targets, count, n, pair, 2, sms);
    tokens = two < one ? 2 * kTokens : kTokens;
    return std::min(one, two);
}

void launch_gemm_k_tc(const MatTarget* targets, int count, const DevAct& act, uint32_t n, Epilogue epi, uint32_t tokens, const WaitBound& bound, uint32_t sms, cudaStream_t s) {
    KtParams p{};
    for (int i = 0; i < count; ++i) {
        p.m[i] = targets[i].m;
        p.out[i] = targets[i].out;
        p.ldo[i] = targets[i].ldo;
    }
    p.act = act;
    p.n = n;
    p.count = count;
    p.epi = int(epi);
    p.one = 1.0f;
    p.bound = bound;
    const bool pair = epi == EPI_SILU_MUL || epi == EPI_RELU2_MUL;
    const int halves = int(tokens / kTokens);
    switch (targets[0].m.type) {
        case T_Q4_K: launch_type<T_Q4_K>(p, pair, halves, sms, s); break;
        case T_Q5_K: launch_type<T_Q5_K>(p, pair, halves, sms, s); break;
        case T_Q6_K: launch_type<T_Q6_K>(p, pair, halves, sms, s); break;
        case T_TQ2_0: launch_type<T_TQ2_0>(p, pair, halves, sms, s); break;
        default: throw CudaError("cuda: no super-block tensor kernel for this type");
    }
}

}  // namespace bk
