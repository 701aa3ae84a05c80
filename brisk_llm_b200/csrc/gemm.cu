// Multiply of a few to many tokens by Q4_0 / Q8_0 matrices: int8 tensor-core MMA on Q8_0-quantised activations, with the
// reference's per-block arithmetic kept intact.
//
// The reference computes, per (row, token), the sum over 32-value blocks IN ORDER of float(int_dot) * d_w * d_x
// (src/quant.cpp:445-482). One m16n8k32 s8 MMA yields the integer block dots of 16 tokens x 8 rows; each thread scales
// the dots it holds and adds them to f32 accumulators it alone owns, walking the blocks in order - the same sequence of
// roundings as the CPU, so results are bit-identical and the next 8-bit re-quantisation sees the same values. K is never
// split across threads.
//
// Bound: the f32 pipe. A term costs three roundings the reference makes (dot * d_w, * d_x, + sum), and nothing else may
// go through that pipe if the rest is to keep out of the way:
//   - the MMA's C operand is the bit pattern of 1.5 * 2^23, so a result read as a float is 1.5 * 2^23 + dot exactly, and
//     fma(result, d_w, -1.5 * 2^23 * d_w) is dot * d_w rounded once (the addend has 13 significant bits: it is exact) -
//     conversion and first multiply in one instruction;
//   - packed f32x2 instructions work on two outputs each. They do not raise the f32 rate (measured: 0.49 of them per
//     cycle and scheduler against 0.98 scalar ones) but halve the issue slots, which the fragment loads and MMAs need. The
//     sum is an fma by 1.0 taken from the kernel's parameters: a packed multiply feeding a packed add is contracted into
//     one fused multiply-add by the assembler, and the reference does not fuse;
//   - tokens are the MMA's M side and weight rows its N side, so a thread's packed pair is two rows of one token: the pair
//     of weight scales is what two adjacent scale rows hold, and the token's scale is one value twice;
//   - Q4_0 nibbles become signed bytes as 16 * (q - 8) - the nibble in the byte's upper half with its top bit flipped: one
//     logic operation for four weights. Sums come out 16 times as large, exactly, and are scaled once at the end.
//
// Tiling: a CTA of four warps side by side along the rows; a warp covers 16 MI tokens x 8 NI rows (big tiles reuse
// fragments, small ones fill the GPU; the rule is at pick_tile). Weights, activations and their scales come through a ring
// of cp.async stages of four blocks. Row pitches carry 16 bytes of padding: fragment reads are conflict-free. For a
// gate/up pair half of a warp's rows are gate rows and half the up rows at the same place, and the activation is applied
// in the epilogue. Measured: 4096 x 14336 Q4_0 at 512 tokens 282 -> 225 us (134 TMAC/s), 1024 x 3072 25 -> 21 us; at 9
// tokens 43 -> 24 us (and 14336 x 4096 35 -> 17 us) against a kernel whose warps split a stage and add terms up through
// shared memory.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "formats.cuh"
#include "kernels.h"
#include "packed.cuh"
#include "pdl.cuh"

namespace bk {
namespace {

constexpr int KB = 4, GWARPS = 4;  // blocks per stage, warps per CTA

// One stage of a CTA tile of RT rows x TT tokens; WB: bytes of quants per block and row, 16 (Q4_0) or 32 (Q8_0).
template <int WB, int RT, int TT>
struct Stage {
    static constexpr int kWRow = KB * WB + 16;
    static constexpr int kXRow = KB * 32 + 16;
    static constexpr int kW = RT * kWRow;
    static constexpr int kWd = RT * KB * 2;  // weight scales [row][block], f16
    static constexpr int kX = TT * kXRow;
    static constexpr int kXd = TT * KB * 4;  // activation scales [token][block], f32
    static constexpr int kBytes = kW + kWd + kX + kXd;
};

struct GemmParams {
    DevMatrix m[3];
    float* out[3];
    uint32_t ldo[3];
    uint32_t first_tile[4];  // row tiles of target i: [first_tile[i], first_tile[i + 1])
    DevAct act;
    uint32_t n;
    int count, epi;
    int early;  // release the next kernel at once: with few tokens it has few CTAs to wait beside this one
    float one;  // 1.0f
};

__device__ __forceinline__ void cp_async8(uint32_t smem, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}

constexpr int kMagicBits = 0x4B400000;  // 1.5 * 2^23 as a float; |dot| <= 16 * 32 * 8 * 127 or 32 * 128 * 127, both < 2^22
constexpr float kMagic = 12582912.0f;

// d = a x b + kMagicBits in every element
__device__ __forceinline__ void mma_s8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(kMagicBits));
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <class T> __device__ __forceinline__ T lds(uint32_t addr);
template <> __device__ __forceinline__ uint32_t lds<uint32_t>(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
template <> __device__ __forceinline__ float lds<float>(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
template <> __device__ __forceinline__ uint4 lds<uint4>(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}

template <int WB, int MI, int NI, bool PAIR, int STAGES, int MINB>
__global__ void __launch_bounds__(GWARPS * 32, MINB) gemm_q8_kernel(const __grid_constant__ GemmParams p) {
    constexpr int RT = GWARPS * 8 * NI, TT = 16 * MI, THREADS = GWARPS * 32;
    using S = Stage<WB, RT, TT>;
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t sbase = uint32_t(__cvta_generic_to_shared(smem));
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t g = lane >> 2, t = lane & 3;
    const uint32_t tok_base = blockIdx.x * TT;
    int target = 0;
    if (!PAIR) {
        if (p.count > 1 && blockIdx.y >= p.first_tile[1]) target = 1;
        if (p.count > 2 && blockIdx.y >= p.first_tile[2]) target = 2;
    }
    const DevMatrix& m = p.m[target];
    const uint32_t nb = m.blocks, chunks = nb / KB;
    // Rows of the tile: RT of one matrix, or (pair) RT / 2 of the gate matrix and the same RT / 2 of the up matrix.
    const uint32_t row_base = (blockIdx.y - p.first_tile[target]) * (PAIR ? RT / 2 : RT);

    // What this thread copies into every stage: 16-byte pieces of quants, an 8-byte run of weight scales, 16 bytes of
    // activation scales. The places are worked out once; a stage advances them by a constant.
    constexpr int kWParts = KB * WB / 16;                                      // pieces per row and stage
    constexpr int kWPieces = (RT * kWParts + THREADS - 1) / THREADS, kXPieces = TT * 8 / THREADS;
    static_assert(RT * kWParts % THREADS == 0 && TT * 8 % THREADS == 0 && RT <= THREADS && TT <= THREADS, "whole pieces per thread");
    const uint8_t* wsrc[kWPieces];
    const int8_t* xsrc[kXPieces];
    auto row_of = [&](uint32_t r, const DevMatrix*& mat) {  // tile row r -> its matrix and row there (clamped)
        mat = &m;
        uint32_t row = row_base + r;
        if (PAIR && r >= RT / 2) {
            mat = &p.m[1];
            row -= RT / 2;
        }
        return min(row, m.rows - 1);
    };
#pragma unroll
    for (int i = 0; i < kWPieces; ++i) {
        const uint32_t at = tid + i * THREADS, r = at / kWParts;
        const DevMatrix* mat;
        const uint32_t row = row_of(r, mat);
        wsrc[i] = mat->qa + size_t(row) * nb * WB + (at % kWParts) * 16;
    }
#pragma unroll
    for (int i = 0; i < kXPieces; ++i) {
        const uint32_t at = tid + i * THREADS, tok = tok_base + at / 8;
        xsrc[i] = tok < p.n ? p.act.q0 + size_t(tok) * p.act.cols + (at % 8) * 16 : nullptr;
    }
    const __half* dsrc = nullptr;
    if (tid < RT) {
        const DevMatrix* mat;
        const uint32_t row = row_of(tid, mat);
        dsrc = mat->d + size_t(row) * nb;
    }
    const bool scales = tid < TT && tok_base + tid < p.n;  // this thread copies a token's scales
    const float* xdsrc = p.act.d0 + size_t(scales ? tok_base + tid : 0) * nb;
    auto load_weights = [&](uint32_t slot, uint32_t chunk) {
        const uint32_t at = sbase + slot * S::kBytes;
#pragma unroll
        for (int i = 0; i < kWPieces; ++i) {
            const uint32_t piece = tid + i * THREADS;
            cp_async16(at + piece / kWParts * S::kWRow + piece % kWParts * 16, wsrc[i] + size_t(chunk) * (KB * WB));
        }
        if (tid < RT) cp_async8(at + S::kW + tid * (KB * 2), dsrc + size_t(chunk) * KB);
    };
    auto load_tokens = [&](uint32_t slot, uint32_t chunk) {
        const uint32_t at = sbase + slot * S::kBytes;
#pragma unroll
        for (int i = 0; i < kXPieces; ++i) {
            const uint32_t piece = tid + i * THREADS;
            // Tokens past the last are left out: their rows of the MMAs hold whatever was there and are never stored. (A copy
            // of the last token in their place had every CTA read the same few lines of L2 over and over.)
            if (xsrc[i] != nullptr) cp_async16(at + S::kW + S::kWd + piece / 8 * S::kXRow + piece % 8 * 16, xsrc[i] + size_t(chunk) * (KB * 32));
        }
        if (scales) cp_async16(at + S::kW + S::kWd + S::kX + tid * (KB * 4), xdsrc + size_t(chunk) * KB);
    };

    f32x2 acc[MI][NI][2];  // [..][0]: rows 2t, 2t + 1 of token g, [..][1]: of token g + 8
#pragma unroll
    for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < NI; ++ni) acc[mi][ni][0] = acc[mi][ni][1] = 0ull;
    const f32x2 one2 = pack2(p.one, p.one), minus_magic2 = pack2(-kMagic, -kMagic);
    // first tile row of this warp's row tile ni
    auto tile_row = [&](int ni) -> uint32_t {
        if constexpr (PAIR) return (ni / (NI / 2)) * (RT / 2) + warp * (4 * NI) + (ni % (NI / 2)) * 8;
        else return warp * (8 * NI) + ni * 8;
    };

#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (uint32_t(s) < chunks) load_weights(s, s);
    }
    wait_for_previous();  // the activations
    if (p.early) release_next();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (uint32_t(s) < chunks) load_tokens(s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    uint32_t slot = 0, fill = STAGES - 1;
    for (uint32_t chunk = 0; chunk < chunks; ++chunk) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();  // the stage has landed for every thread, and the slot filled next is no longer read
        if (chunk + STAGES - 1 < chunks) {
            load_weights(fill, chunk + STAGES - 1);
            load_tokens(fill, chunk + STAGES - 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        fill = fill + 1 == STAGES ? 0 : fill + 1;
        const uint32_t at = sbase + slot * S::kBytes;
        slot = slot + 1 == STAGES ? 0 : slot + 1;

        uint4 dw[NI];  // scales of rows 2t and 2t + 1, four blocks each
#pragma unroll
        for (int ni = 0; ni < NI; ++ni) dw[ni] = lds<uint4>(at + S::kW + (tile_row(ni) + 2 * t) * (KB * 2));
        const uint32_t xfrag = at + S::kW + S::kWd + ((lane & 7) + ((lane >> 3) & 1) * 8) * S::kXRow + (lane >> 4) * 16;
        const uint32_t xscale = at + S::kW + S::kWd + S::kX + g * (KB * 4);
        const uint32_t wfrag = at + g * S::kWRow + 4 * t;
#pragma unroll
        for (int b = 0; b < KB; ++b) {
            uint32_t a[MI][4];
            f32x2 dx2[MI][2];
#pragma unroll
            for (int mi = 0; mi < MI; ++mi) {
                ldmatrix4(a[mi], xfrag + mi * 16 * S::kXRow + b * 32);
                const float d0 = lds<float>(xscale + (mi * 16) * (KB * 4) + b * 4), d1 = lds<float>(xscale + (mi * 16 + 8) * (KB * 4) + b * 4);
                dx2[mi][0] = pack2(d0, d0);
                dx2[mi][1] = pack2(d1, d1);
            }
#pragma unroll
            for (int ni = 0; ni < NI; ++ni) {
                uint32_t b0, b1;
                if (WB == 16) {
                    const uint32_t w = lds<uint32_t>(wfrag + tile_row(ni) * S::kWRow + b * 16);
                    b0 = ((w << 4) ^ 0x80808080u) & 0xF0F0F0F0u;
                    b1 = (w ^ 0x80808080u) & 0xF0F0F0F0u;
                } else {
                    b0 = lds<uint32_t>(wfrag + tile_row(ni) * S::kWRow + b * 32);
                    b1 = lds<uint32_t>(wfrag + tile_row(ni) * S::kWRow + b * 32 + 16);
                }
                const uint32_t lo = b < 2 ? dw[ni].x : dw[ni].y, hi = b < 2 ? dw[ni].z : dw[ni].w;
                const f32x2 dw2 = pack2(__half2float(__ushort_as_half(uint16_t(b & 1 ? lo >> 16 : lo & 0xFFFF))),
                                        __half2float(__ushort_as_half(uint16_t(b & 1 ? hi >> 16 : hi & 0xFFFF))));
                const f32x2 off2 = mul2(dw2, minus_magic2);
#pragma unroll
                for (int mi = 0; mi < MI; ++mi) {
                    int c[4];
                    mma_s8(c, a[mi], b0, b1);
                    acc[mi][ni][0] = fma2(mul2(fma2(pack2(c[0], c[1]), dw2, off2), dx2[mi][0]), one2, acc[mi][ni][0]);
                    acc[mi][ni][1] = fma2(mul2(fma2(pack2(c[2], c[3]), dw2, off2), dx2[mi][1]), one2, acc[mi][ni][1]);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (!p.early) release_next();

    constexpr float kScale = WB == 16 ? 0.0625f : 1.0f;  // exact
    float* const out = p.out[target];
    const uint32_t ldo = p.ldo[target];
    const bool even = (ldo & 1) == 0;
#pragma unroll
    for (int mi = 0; mi < MI; ++mi) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const uint32_t tok = tok_base + mi * 16 + half * 8 + g;
            if (tok >= p.n) continue;
#pragma unroll
            for (int ni = 0; ni < (PAIR ? NI / 2 : NI); ++ni) {
                const uint32_t row = row_base + tile_row(ni) + 2 * t;
                if (row >= m.rows) continue;
                float v0, v1;
                unpack2(acc[mi][ni][half], v0, v1);
                v0 *= kScale;
                v1 *= kScale;
                if constexpr (PAIR) {
                    float u0, u1;
                    unpack2(acc[mi][ni + NI / 2][half], u0, u1);
                    u0 *= kScale;
                    u1 *= kScale;
                    v0 = p.epi == EPI_SILU_MUL ? silu_mul(v0, u0) : relu2_mul(v0, u0);
                    v1 = p.epi == EPI_SILU_MUL ? silu_mul(v1, u1) : relu2_mul(v1, u1);
                }
                float* o = out + size_t(tok) * ldo + row;
                if (even && row + 1 < m.rows) {
                    float2 v = make_float2(v0, v1);
                    if (p.epi == EPI_ADD) {
                        const float2 old = *reinterpret_cast<const float2*>(o);
                        v = make_float2(__fadd_rn(old.x, v0), __fadd_rn(old.y, v1));
                    }
                    *reinterpret_cast<float2*>(o) = v;
                } else {
                    o[0] = p.epi == EPI_ADD ? __fadd_rn(o[0], v0) : v0;
                    if (row + 1 < m.rows) o[1] = p.epi == EPI_ADD ? __fadd_rn(o[1], v1) : v1;
                }
            }
        }
    }
}

// A tile shape and what it costs: cycles of one block of its K loop when nothing shares the scheduler (the dependent
// chain fragment - MMA - three roundings) and when the scheduler is full (issue and f32 pipe), measured on B200 with the
// 4096 x 14336 Q4_0 matrix at 9 to 512 tokens.
struct Tile {
    int mi, ni, alone, shared, resident;
    void (*kernel)(GemmParams);
    uint32_t smem;
    uint32_t rows() const { return uint32_t(GWARPS * 8 * ni); }
    uint32_t tokens() const { return uint32_t(16 * mi); }
};

template <int WB, bool PAIR, int MI, int NI, int STAGES, int RESIDENT>
Tile tile_of(int alone, int shared) {
    return Tile{MI, NI, alone, shared, RESIDENT, gemm_q8_kernel<WB, MI, NI, PAIR, STAGES, RESIDENT>, uint32_t(STAGES * Stage<WB, GWARPS * 8 * NI, 16 * MI>::kBytes)};
}
template <int WB, bool PAIR>
const std::vector<Tile>& tiles_of() {
    static const std::vector<Tile> list = [] {
        std::vector<Tile> v = {tile_of<WB, PAIR, 4, 2, 3, 3>(305, 240), tile_of<WB, PAIR, 2, 2, 5, 4>(210, 135), tile_of<WB, PAIR, 1, 2, 6, 6>(166, 90)};
        if constexpr (!PAIR) {
            v.push_back(tile_of<WB, PAIR, 2, 1, 5, 4>(186, 79));
            v.push_back(tile_of<WB, PAIR, 1, 1, 8, 5>(127, 52));
        }
        return v;
    }();
    return list;
}

// The tile whose busiest SM is done first: it runs ceil(tiles / SMs) CTAs, `resident` of them at a time, and a round of
// CTAs takes the longer of one warp's chain and what the scheduler's warps need together. Few rows or tokens favour small
// tiles (1024 x 2048 at 23 tokens: 6.4 us against 14.6 with the largest), a full GPU large ones (4096 x 14336 at 512
// tokens: 225 us against 351 with the smallest).
const Tile& pick_tile(const std::vector<Tile>& list, const GemmParams& p, bool pair, uint32_t sms) {
    const Tile* best = nullptr;
    uint64_t best_cost = 0;
    for (const Tile& tile : list) {
        uint64_t tiles = 0;
        const uint32_t rows = pair ? tile.rows() / 2 : tile.rows();
        for (int i = 0; i < (pair ? 1 : p.count); ++i) tiles += (p.m[i].rows + rows - 1) / rows;
        tiles *= (p.n + tile.tokens() - 1) / tile.tokens();
        const uint64_t per_sm = (tiles + sms - 1) / sms, rounds = (per_sm + tile.resident - 1) / tile.resident;
        const uint64_t cost = std::max<uint64_t>(rounds * uint64_t(tile.alone), per_sm * uint64_t(tile.shared));
        if (best == nullptr || cost < best_cost) {
            best = &tile;
            best_cost = cost;
        }
    }
    return *best;
}

template <int WB, bool PAIR>
void launch_q8(GemmParams& p, uint32_t sms, cudaStream_t s) {
    static DeviceOnce once;
    if (once.first()) {
        for (const Tile& tile : tiles_of<WB, PAIR>()) {
            BK_CUDA(cudaFuncSetAttribute(tile.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(tile.smem)));
            BK_CUDA(cudaFuncSetAttribute(tile.kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        }
    }
    const Tile& tile = pick_tile(tiles_of<WB, PAIR>(), p, PAIR, sms);
    uint32_t tiles = 0;
    const uint32_t rows = PAIR ? tile.rows() / 2 : tile.rows();
    for (int i = 0; i < (PAIR ? 1 : p.count); ++i) {
        p.first_tile[i] = tiles;
        tiles += (p.m[i].rows + rows - 1) / rows;
    }
    // A grid of one to four CTAs an SM is launched in plain order: started while the kernel before it drains, its CTAs pile up
    // on the SMs that are free first (1024 x 3072 at 512 tokens: 28 us -> 40). Fewer do not share an SM's time, more even out.
    const dim3 grid((p.n + tile.tokens() - 1) / tile.tokens(), tiles);
    const uint64_t ctas = uint64_t(grid.x) * grid.y;
    if (ctas > sms && ctas < 4ull * sms && !p.early) {
        tile.kernel<<<grid, GWARPS * 32, tile.smem, s>>>(p);
        BK_CUDA(cudaGetLastError());
    } else {
        launch_dependent(tile.kernel, grid, dim3(GWARPS * 32), tile.smem, s, p);
    }
}

uint32_t sm_count() {
    static const uint32_t sms = [] {
        int dev = 0, count = 148;
        if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
        return uint32_t(count);
    }();
    return sms;
}

}  // namespace

bool gemm_tc_supports(int type, uint32_t cols);  // gemm_tc.cu: the same arithmetic on tcgen05 / tensor memory
void launch_gemm_tc(const MatTarget& tg, const DevAct& act, uint32_t n, Epilogue epi, const WaitBound& bound, cudaStream_t s);
// BRISK_CUDA_GEMM=tc / mma picks the prompt GEMM of Q4_0 / Q8_0 matrices (read at every call); unset: kGemmTcDefault. Measured,
// 512 tokens, us here / gemm_tc.cu: 1024 x 3072 Q4_0 21 / 37, 2048 x 8192 76 / 89, 4096 x 14336 228 / 287, Q8_0 241 / 322.
constexpr bool kGemmTcDefault = false;
static bool gemm_tc_on() {
    const char* env = std::getenv("BRISK_CUDA_GEMM");
    return env == nullptr ? kGemmTcDefault : std::strcmp(env, "tc") == 0;
}
bool gemm_k_supports(int type);  // gemm_k.cu: the 256-value super-block formats
bool launch_gemm_k(const MatTarget* targets, int count, const DevAct& act, uint32_t n, Epilogue epi, const WaitBound& bound, uint32_t sms, cudaStream_t s);

// From 2 tokens on: Q4_0 / Q8_0 rows of a multiple of 4 blocks (128 values), and the super-block formats.
static bool gemm_supports(int type, uint32_t cols, uint32_t n) {
    return n >= 2 && (type == T_Q4_0 || type == T_Q8_0 ? cols % (32 * KB) == 0 : gemm_k_supports(type));
}

WaitBound wait_bound(unsigned int* word_on_device, cudaStream_t s) {
    const char* env = std::getenv("BRISK_CUDA_TEST_TC_TIMEOUT");
    const int test = env != nullptr ? std::atoi(env) : 0;
    const unsigned int start = test == 1 ? 1u : 0u;
    BK_CUDA(cudaMemcpyAsync(word_on_device, &start, sizeof start, cudaMemcpyHostToDevice, s));
    BK_CUDA(cudaStreamSynchronize(s));
    WaitBound bound;
    bound.error = word_on_device;
    if (test >= 2) {
        bound.cycles = 100000;
        bound.withheld = uint32_t(test - 2);
    }
    return bound;
}

int launch_gemm(const MatTarget* targets, int count, const DevAct& act, uint32_t n, Epilogue epi, const WaitBound& bound, cudaStream_t s) {
    const bool pair = epi == EPI_SILU_MUL || epi == EPI_RELU2_MUL;
    for (int i = 0; i < count; ++i) {
        if (!gemm_supports(targets[i].m.type, targets[i].m.cols, n)) return 0;
    }
    const int type = targets[0].m.type;
    if (type != T_Q4_0 && type != T_Q8_0) {
        return launch_gemm_k(targets, count, act, n, epi, bound, sm_count(), s) ? 1 : 0;
    }
    if (!pair && n >= 32 && gemm_tc_on() && gemm_tc_supports(type, targets[0].m.cols)) {
        for (int i = 0; i < count; ++i) launch_gemm_tc(targets[i], act, n, epi, bound, s);
        return count;
    }
    GemmParams p{};
    for (int i = 0; i < count; ++i) {
        p.m[i] = targets[i].m;
        p.out[i] = targets[i].out;
        p.ldo[i] = targets[i].ldo;
    }
    p.act = act;
    p.n = n;
    p.count = count;
    p.epi = int(epi);
    p.early = n <= 64;
    p.one = 1.0f;
    if (type == T_Q4_0) pair ? launch_q8<16, true>(p, sm_count(), s) : launch_q8<16, false>(p, sm_count(), s);
    else pair ? launch_q8<32, true>(p, sm_count(), s) : launch_q8<32, false>(p, sm_count(), s);
    return 1;
}

}  // namespace bk
