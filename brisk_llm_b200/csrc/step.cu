// The whole single-token step of every layer as ONE persistent kernel: one 512-thread CTA per SM, the layer operations
// as phases inside it instead of kernels of their own.
//
//   per layer:  q/k/v multiply | scores (+ per-head norm, RoPE, K/V store) | softmax + weighted sum | output
//               projection (+residual) | gate/up (+activation) | down (+residual)
//
// Why: at batch 1 a layer operation of a 0.6B-class model moves a few megabytes and lasts 3-5 us as its own kernel, of
// which the weight stream is a fraction - the rest is launch and drain, the scheduling gap between graph nodes, and the
// first-load latency of every CTA. Inside one kernel a CTA requests what does not depend on the previous operation (its
// weight rows, cached K rows, V rows, RoPE row, norm weights) before that operation's results exist.
//
// The phases call the same device bodies as the one-kernel-per-operation path (decode_body.cuh): the arithmetic and its
// order are unchanged, results stay bit-identical to the CPU engine.
//
// How the operations hand their results on (default): TAGGED PAIRS, see TaggedIo in decode_body.cuh - every element of
// the small vectors between operations is an 8-byte {value, tag} written with one store; a consumer re-reads until the
// pairs it needs carry the tag of this token, layer and operation. No barrier, no fence, no counter: measured one-way
// latency between two SMs 0.28 us, against 0.50 us for a release/acquire counter. Every poll loop is bounded
// (kPollLimit re-reads); when one runs out the CTA sets the error word and goes on, so the kernel always ends, and the
// host checks the word after the step and raises.
//
// For comparison (BRISK_CUDA_STEP_SYNC=barrier) the same kernel runs with ordinary vectors and grid barriers: a
// monotonic arrival counter, barrier k opens when it reaches k x CTAs. Every CTA arrives once per phase and waits once
// per barrier, also when it has no work in a phase (otherwise its early arrivals would open a later barrier too soon).
// The last CTA to leave the kernel zeroes the counter for the next launch. Waits are bounded as well: after kSpinLimit
// polls the CTA sets the error word and adds a huge constant to the counter, which opens this and every later barrier.
// About 10 % slower than the tagged form.
//
// The launch is cooperative, so the CTAs are co-resident or the launch itself fails.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <memory>
#include <utility>

#include "decode_body.cuh"

namespace bk {

struct alignas(16) StepLayerDesc {
    DecMatParams qkv, o, gate_up, down;
    DecAttnParams attn;
};
static_assert(sizeof(StepLayerDesc) % 16 == 0, "copied in 16-byte pieces");

namespace {

constexpr uint32_t kStepThreads = kDecWarps * 32;
constexpr uint32_t kSpinLimit = 1u << 21;
constexpr unsigned int kOpenAll = 1u << 30;  // far above any arrival count of one launch

struct StepParams {
    const StepLayerDesc* layers;
    uint32_t n_layers;
    unsigned int* sync;   // [0] arrivals, [1] exits, [2] error
    uint32_t tile_offset; // bytes from the start of dynamic shared memory to the transpose tile (after the widest activation row)
    unsigned long long* trace;  // optional (BRISK_CUDA_STEP_TRACE): per phase, CTA 0's time of entry, of passing the barrier, of finishing, and its polls
    // tagged exchange (see TaggedIo): the tags of this launch start above tag_base; the residual stream comes in and
    // goes out as ordinary floats in plain_hidden and lives in between as tagged pairs in tagged_hidden
    uint32_t tag_base;
    uint32_t fault_layer;  // test only: this layer's q/k/v multiply expects a tag nobody writes (0xffffffff: none)
    float* plain_hidden;
    uint2* tagged_hidden;
    uint32_t hidden_size;
};

struct NoGate {  // tagged exchange: nothing to wait for, the data itself says when it is there
    __device__ __forceinline__ void wait() {}
    __device__ __forceinline__ void prologue_done() {}
};

// `count` tagged values (a multiple of 2) from src into shared memory at dst, by one warp; bounded re-reads.
__device__ __forceinline__ void warp_fetch_tagged(const uint2* src, float* dst, uint32_t count, uint32_t tag, unsigned int* error) {
    const uint32_t lane = threadIdx.x & 31;
    const uint4* src2 = reinterpret_cast<const uint4*>(src);
    for (uint32_t base = 0; base < count / 2; base += 32 * 4) {
        uint4 v[4];
        for (uint32_t spin = 0;; ++spin) {
            bool complete = true;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t i = base + lane + 32 * k;
                v[k] = i < count / 2 ? ld_pairs2(src2 + i) : make_uint4(0u, tag, 0u, tag);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) complete = complete && v[k].y == tag && v[k].w == tag;
            if (complete) break;
            if (spin == kPollLimit || poll_abandoned(spin, error)) {
                poll_failed(error);
                break;
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t i = base + lane + 32 * k;
            if (i < count / 2) {
                dst[2 * i] = __uint_as_float(v[k].x);
                dst[2 * i + 1] = __uint_as_float(v[k].z);
            }
        }
    }
}

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release_add(unsigned int* p, unsigned int v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

struct GridGate {
    unsigned int* sync;
    unsigned int target;  // arrivals that open the next barrier
    unsigned int nctas;
    bool waited;          // this phase's barrier has been passed (or the phase needs none)
    unsigned long long* trace;  // CTA 0 only, else nullptr: four words per phase
    int* open_flag;       // shared memory: the result of enter()'s single poll

    // Start of a phase: ONE poll before the phase requests anything. An acquire load does not complete while the
    // thread's earlier loads are in flight, so a poll issued after the weight prefetch would wait for the prefetch; a
    // CTA that finds its barrier open already (the usual case for the CTAs that arrive last) skips the wait entirely
    // and its prefetch overlaps the activation prologue instead.
    __device__ __forceinline__ void enter() {
        if (waited) return;
        if (threadIdx.x == 0) *open_flag = int(ld_acquire(sync) - target) >= 0 ? 1 : 0;
        __syncthreads();
        if (*open_flag != 0) {
            waited = true;
            if (trace != nullptr && threadIdx.x == 0) {
                trace[1] = now_ns();
                trace[3] = 0;
            }
        }
    }

    // Thread 0 polls with acquire loads; the barrier that follows orders every other thread of the CTA behind it.
    __device__ __forceinline__ void wait() {
        if (waited) return;
        waited = true;
        if (threadIdx.x == 0) {
            unsigned int spins = 0;
            while (int(ld_acquire(sync) - target) < 0) {
                if (++spins > kSpinLimit) {  // give up: flag it and open this and every later barrier for every CTA
                    atomicExch(sync + 2, 1u);
                    atomicAdd(sync, kOpenAll);
                    break;
                }
            }
            if (trace != nullptr) {
                trace[1] = now_ns();
                trace[3] = spins;
            }
        }
        __syncthreads();
    }
    __device__ __forceinline__ void prologue_done() {}
    // End of a phase: make sure this phase's barrier was passed, publish the phase's results, arm the next barrier.
    // The release reduction of thread 0, after the CTA barrier, publishes the stores of all of the CTA's threads.
    __device__ __forceinline__ void arrive() {
        if (trace != nullptr && threadIdx.x == 0) trace[2] = now_ns();
        wait();
        __syncthreads();  // every thread's stores of this phase are issued
        if (threadIdx.x == 0) {
            red_release_add(sync, 1u);
            if (trace != nullptr) {
                trace += 4;
                trace[0] = now_ns();
            }
        }
        target += nctas;
        waited = false;
    }
};

// Scores of the new token against every visible position, as WARP tasks of (query head, 32 positions) dealt round-robin
// over the CTAs (a 600-position context of 16 heads gives 304 tasks: two or three warps on every SM), so that the K
// rows come in over every SM's memory pipe at once (the heads of a group read the same rows; the second read hits L2). A warp needs no CTA barrier: it copies its 32 K rows into its own slice of
// shared memory with cp.async (requested BEFORE the grid barrier; rows padded by 16 bytes so that the 16-byte reads of
// a quarter warp fall into distinct banks), norms and rotates the group's query heads into the same slice, and each
// lane then owns one position. The task that covers the token's own position also norms, rotates and stores the new
// K and V rows. Arithmetic and order per (head, position) are those of the per-operation scores kernel.
constexpr uint32_t kMaxGroup = 8;
__host__ __device__ inline size_t step_scores_warp_smem(uint32_t group, uint32_t dim) {
    return size_t(group + 1) * dim * sizeof(float) + size_t(32) * (dim * 2 + 16);
}

struct ScoreTags {
    uint32_t in, out;  // tag of q/k/v, tag of the scores
    unsigned int* error;
};

template <int VPL, bool NEOX, bool TAGGED, class Gate>
__device__ __forceinline__ void step_scores(const DecAttnParams& a, const uint32_t cta, const uint32_t nctas, unsigned char* sm, Gate& gate, const ScoreTags& tags) {
    constexpr uint32_t dim = VPL * 32;
    const uint32_t group = a.heads / a.kv_heads;
    const uint32_t pos = *a.position, visible = pos + 1;
    const uint32_t chunks = (visible + 31) / 32;
    const uint32_t tasks = a.heads * chunks;  // (query head, 32 positions)
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char* mine = sm + size_t(warp) * step_scores_warp_smem(group, dim);
    float* qs = reinterpret_cast<float*>(mine);
    float* knew = qs + dim;
    const uint4* krow = reinterpret_cast<const uint4*>(mine + size_t(group + 1) * dim * sizeof(float) + size_t(lane) * (dim * 2 + 16));
    const float* rope = a.rope + size_t(pos) * dim;

    auto request_row = [&](uint32_t task) {  // this lane's cached K row of the task, if it has one
        const uint32_t kvh = (task / chunks) / group, p = (task % chunks) * 32 + lane;
        if (p < visible && p != pos) {
            const __half* kr = a.k_cache + (size_t(kvh) * a.max_context + p) * dim;
            const uint32_t dst = uint32_t(__cvta_generic_to_shared(krow));
#pragma unroll
            for (uint32_t i = 0; i < dim / 8; ++i) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 16), "l"(kr + i * 8) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const uint32_t first = cta + warp * nctas, stride = nctas * kDecWarps;
    dec_stamp(a.trace, cta, 0);
    if (first < tasks) {
        request_row(first);
        // The RoPE row of this position and the per-head norm weights do not depend on the projections either: pull
        // their cache lines in now, so that the loads behind the poll hit L1.
        if (lane * 32 < dim) {
            asm volatile("prefetch.global.L1 [%0];" ::"l"(rope + lane * 32));
            if (a.q_norm != nullptr) asm volatile("prefetch.global.L1 [%0];" ::"l"(a.q_norm + lane * 32));
            if (a.k_norm != nullptr) asm volatile("prefetch.global.L1 [%0];" ::"l"(a.k_norm + lane * 32));
        }
    }
    gate.wait();
    dec_stamp(a.trace, cta, 1);
    for (uint32_t task = first; task < tasks; task += stride) {
        if (task != first) request_row(task);
        const uint32_t head = task / chunks, kvh = head / group, begin = (task % chunks) * 32;
        const uint32_t p = begin + lane;
        const bool cached = p < visible && p != pos;
        // The raw query head and, for the tasks that cover the token's own position, the raw new K row: into the slice
        // through L2, then norm + RoPE in place (a lane rewrites exactly the elements it read). Every head of the group
        // prepares the new K row for its own score; the group's first head also stores it (and V) to the cache.
        const bool owner = pos >= begin && pos < begin + 32;
        if constexpr (TAGGED) {
            warp_fetch_tagged(reinterpret_cast<const uint2*>(a.q) + size_t(head) * dim, qs, dim, tags.in, tags.error);
            if (owner) warp_fetch_tagged(reinterpret_cast<const uint2*>(a.k) + size_t(kvh) * dim, knew, dim, tags.in, tags.error);
        } else {
            const float* qsrc = a.q + size_t(head) * dim;
            const uint32_t qdst = uint32_t(__cvta_generic_to_shared(qs));
            for (uint32_t i = lane; i < dim / 4; i += 32) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(qdst + i * 16), "l"(qsrc + i * 4) : "memory");
            }
            if (owner) {
                const float* ksrc = a.k + size_t(kvh) * dim;
                const uint32_t kdst = uint32_t(__cvta_generic_to_shared(knew));
                for (uint32_t i = lane; i < dim / 4; i += 32) {
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(kdst + i * 16), "l"(ksrc + i * 4) : "memory");
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");  // the raw heads, and this lane's K row requested earlier
        __syncwarp();
        dec_stamp(a.trace, cta, 2);
        if (owner) {
            float kv[VPL];
#pragma unroll
            for (int k = 0; k < VPL; ++k) {
                const uint32_t i = NEOX ? lane + 32 * k : VPL * lane + k;
                kv[k] = knew[i];
                if (a.k_bias != nullptr) kv[k] = __fadd_rn(kv[k], a.k_bias[size_t(kvh) * dim + i]);  // add_bias, src/model.cpp:1026-1030
            }
            warp_head_norm_rope<VPL, NEOX>(kv, a.k_norm, rope, a.eps, knew);
            __syncwarp();
            const bool stores = head % group == 0;
            const size_t row = (size_t(kvh) * a.max_context + pos) * dim;
            for (uint32_t i = lane; i < dim; i += 32) {  // as warp_store_new_kv
                const __half kh = __float2half_rn(knew[i]);
                knew[i] = __half2float(kh);  // the score of the own position uses the cache's f16 value
                if (stores) {
                    a.k_cache[row + i] = kh;
                    float v;
                    if constexpr (TAGGED) v = poll_pair(reinterpret_cast<const uint2*>(a.v) + size_t(kvh) * dim + i, tags.in, tags.error);
                    else v = __ldcg(a.v + size_t(kvh) * dim + i);
                    if (a.v_bias != nullptr) v = __fadd_rn(v, a.v_bias[size_t(kvh) * dim + i]);
                    a.v_cache[row + i] = __float2half_rn(v);
                }
            }
        }
        {
            float v[VPL];
#pragma unroll
            for (int k = 0; k < VPL; ++k) {
                const uint32_t i = NEOX ? lane + 32 * k : VPL * lane + k;
                v[k] = qs[i];
                if (a.q_bias != nullptr) v[k] = __fadd_rn(v[k], a.q_bias[size_t(head) * dim + i]);
            }
            warp_head_norm_rope<VPL, NEOX>(v, a.q_norm, rope, a.eps, qs);
        }
        __syncwarp();
        dec_stamp(a.trace, cta, 3);
        if (p < visible) {
            float lanes[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) lanes[j] = 0.0f;
#pragma unroll
            for (uint32_t i = 0; i < dim; i += 16) {
                float kf[16];
                if (!cached) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) kf[j] = knew[i + j];
                } else {
                    const uint4 r0 = krow[i / 8], r1 = krow[i / 8 + 1];
                    const __half2* h0 = reinterpret_cast<const __half2*>(&r0);
                    const __half2* h1 = reinterpret_cast<const __half2*>(&r1);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 f0 = __half22float2(h0[j]), f1 = __half22float2(h1[j]);
                        kf[2 * j] = f0.x; kf[2 * j + 1] = f0.y; kf[8 + 2 * j] = f1.x; kf[8 + 2 * j + 1] = f1.y;
                    }
                }
                const float4* q4 = reinterpret_cast<const float4*>(qs + i);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 q = q4[j];
                    lanes[4 * j + 0] = __fadd_rn(lanes[4 * j + 0], __fmul_rn(q.x, kf[4 * j + 0]));
                    lanes[4 * j + 1] = __fadd_rn(lanes[4 * j + 1], __fmul_rn(q.y, kf[4 * j + 1]));
                    lanes[4 * j + 2] = __fadd_rn(lanes[4 * j + 2], __fmul_rn(q.z, kf[4 * j + 2]));
                    lanes[4 * j + 3] = __fadd_rn(lanes[4 * j + 3], __fmul_rn(q.w, kf[4 * j + 3]));
                }
            }
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < 16; ++j) sum = __fadd_rn(sum, lanes[j]);
            const size_t at = size_t(head) * a.max_context + p;
            if constexpr (TAGGED) st_pair(reinterpret_cast<uint2*>(a.scores) + at, __fmul_rn(sum, a.scale), tags.out);
            else a.scores[at] = __fmul_rn(sum, a.scale);
        }
        __syncwarp();  // the slice is rewritten by the warp's next task
        dec_stamp(a.trace, cta, 4);
    }
}

constexpr int ring_depth(int regs_per_iter, bool deep) { return !deep ? 1 : regs_per_iter * 4 <= 48 ? 4 : regs_per_iter * 2 <= 48 ? 2 : 1; }

template <class F, int RWA, int RWO, int RWG, int RWD, bool DEEP, bool TAGGED>
__global__ void __launch_bounds__(kStepThreads, 1) step_kernel(const StepParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double red[32];
    __shared__ float redf[kDecWarps];
    __shared__ uint64_t exp_table[32];  // 2^(i/32) for the softmax's exps: the kernel keeps almost no L1, a global table means an L2 trip per exp
    if (threadIdx.x < 32) exp_table[threadIdx.x] = exp2_table_device()[threadIdx.x];  // ordered before its first use by the barriers of the first phases
    constexpr int kWordsPerUnit = F::kRegs;
    float* tile = reinterpret_cast<float*>(smem + P.tile_offset);
    const uint32_t cta = blockIdx.x, nctas = gridDim.x;
    // The layer's descriptor (pointers, shapes, row-group tables) is read many times on the way to the first weight
    // load of a phase; from global memory those dependent reads cost more than a microsecond per phase. Each layer's
    // descriptor is therefore copied into shared memory while the previous layer runs.
    __shared__ StepLayerDesc desc[2];
    constexpr uint32_t kDescPieces = sizeof(StepLayerDesc) / 16;
    auto fetch_desc = [&](uint32_t layer) {
        if (threadIdx.x < kDescPieces) {
            const uint32_t dst = uint32_t(__cvta_generic_to_shared(reinterpret_cast<unsigned char*>(&desc[layer & 1]) + threadIdx.x * 16));
            const unsigned char* src = reinterpret_cast<const unsigned char*>(P.layers + layer) + threadIdx.x * 16;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    static_assert(kDescPieces <= kStepThreads, "one piece per thread");
    fetch_desc(0);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if constexpr (TAGGED) {
        // ---- tagged exchange: no barriers, every operation polls its own inputs --------------------------------
        unsigned int* error = P.sync + 2;
        unsigned long long* trace = cta == 0 ? P.trace : nullptr;
        auto enter = [&] {
            if (trace != nullptr && threadIdx.x == 0) trace[0] = trace[1] = now_ns();
        };
        auto leave = [&] {
            __syncthreads();  // shared memory (activation row, tiles, descriptor buffers) changes hands between operations
            if (trace != nullptr && threadIdx.x == 0) {
                trace[2] = now_ns();
                trace += 4;
            }
        };
        NoGate gate;
        const uint32_t tag_in = P.tag_base + 1;
        if (cta == 0) {  // the token's embedding row arrives as ordinary floats: hand it to every CTA as tagged pairs
            for (uint32_t i = threadIdx.x; i < P.hidden_size; i += kStepThreads) st_pair(P.tagged_hidden + i, __ldcg(P.plain_hidden + i), tag_in);
        }
        for (uint32_t l = 0; l < P.n_layers; ++l) {
            const StepLayerDesc& L = desc[l & 1];
            if (l + 1 < P.n_layers) fetch_desc(l + 1);
            const uint32_t t0 = P.tag_base + 2 + l * 6;  // tags of this layer's six operations: t0 .. t0 + 5
            const uint32_t tag_residual = l == 0 ? tag_in : t0 - 1;  // the previous layer's down projection
            const uint32_t tag_qkv_in = l == P.fault_layer ? (tag_residual ^ 0x40000000u) : tag_residual;
            const bool last = l + 1 == P.n_layers;

            enter();
            dec_multiply_body<F, RWA, false, ring_depth(RWA * kWordsPerUnit, DEEP)>(L.qkv, cta, nctas, smem, tile, red, gate,
                                                                                    TaggedIo{tag_qkv_in, 0u, t0, error, nullptr});
            leave();

            enter();
            {
                const ScoreTags tags{t0, t0 + 1, error};
                if (L.attn.dim == 128) {
                    if (L.attn.neox) step_scores<4, true, true>(L.attn, cta, nctas, smem, gate, tags);
                    else step_scores<4, false, true>(L.attn, cta, nctas, smem, gate, tags);
                } else {
                    if (L.attn.neox) step_scores<2, true, true>(L.attn, cta, nctas, smem, gate, tags);
                    else step_scores<2, false, true>(L.attn, cta, nctas, smem, gate, tags);
                }
            }
            leave();

            enter();
            {
                const uint32_t slices = L.attn.dim / L.attn.slice_width;
                for (uint32_t task = cta; task < L.attn.heads * slices; task += nctas) {
                    dec_attn_out_body<kStepThreads>(L.attn, task / slices, task % slices, smem, redf, red, gate, TaggedAttnIo{t0 + 1, t0, t0 + 2, error}, exp_table);
                    __syncthreads();
                }
            }
            leave();

            enter();
            dec_multiply_body<F, RWO, false, ring_depth(RWO * kWordsPerUnit, DEEP)>(L.o, cta, nctas, smem, tile, red, gate,
                                                                                    TaggedIo{t0 + 2, tag_residual, t0 + 3, error, nullptr});
            leave();

            enter();
            dec_multiply_body<F, RWG, true, ring_depth(2 * RWG * kWordsPerUnit, DEEP)>(L.gate_up, cta, nctas, smem, tile, red, gate,
                                                                                       TaggedIo{t0 + 3, 0u, t0 + 4, error, nullptr});
            leave();

            enter();
            dec_multiply_body<F, RWD, false, ring_depth(RWD * kWordsPerUnit, DEEP)>(L.down, cta, nctas, smem, tile, red, gate,
                                                                                    TaggedIo{t0 + 4, t0 + 3, t0 + 5, error, last ? P.plain_hidden : nullptr});
            asm volatile("cp.async.wait_group 0;" ::: "memory");  // the next layer's descriptor
            leave();
        }
    } else {
        __shared__ int open_flag;
        GridGate gate{P.sync, 0u, nctas, true, cta == 0 ? P.trace : nullptr, &open_flag};  // the first phase reads what earlier kernels wrote: no barrier
        if (gate.trace != nullptr && threadIdx.x == 0) gate.trace[0] = now_ns();

        for (uint32_t l = 0; l < P.n_layers; ++l) {
            const StepLayerDesc& L = desc[l & 1];
            if (l + 1 < P.n_layers) fetch_desc(l + 1);  // the other buffer's layer finished behind the barrier of its last arrive
            gate.enter();
            dec_multiply_body<F, RWA, false, ring_depth(RWA * kWordsPerUnit, DEEP)>(L.qkv, cta, nctas, smem, tile, red, gate);
            gate.arrive();

            gate.enter();
            if (L.attn.dim == 128) {
                if (L.attn.neox) step_scores<4, true, false>(L.attn, cta, nctas, smem, gate, ScoreTags{});
                else step_scores<4, false, false>(L.attn, cta, nctas, smem, gate, ScoreTags{});
            } else {
                if (L.attn.neox) step_scores<2, true, false>(L.attn, cta, nctas, smem, gate, ScoreTags{});
                else step_scores<2, false, false>(L.attn, cta, nctas, smem, gate, ScoreTags{});
            }
            gate.arrive();

            gate.enter();
            {
                const uint32_t slices = L.attn.dim / L.attn.slice_width;
                for (uint32_t task = cta; task < L.attn.heads * slices; task += nctas) {
                    dec_attn_out_body<kStepThreads>(L.attn, task / slices, task % slices, smem, redf, red, gate, PlainIo{}, exp_table);
                    __syncthreads();  // the shared-memory row of probabilities is rewritten for the CTA's next task
                }
            }
            gate.arrive();

            gate.enter();
            dec_multiply_body<F, RWO, false, ring_depth(RWO * kWordsPerUnit, DEEP)>(L.o, cta, nctas, smem, tile, red, gate);
            gate.arrive();

            gate.enter();
            dec_multiply_body<F, RWG, true, ring_depth(2 * RWG * kWordsPerUnit, DEEP)>(L.gate_up, cta, nctas, smem, tile, red, gate);
            gate.arrive();

            gate.enter();
            dec_multiply_body<F, RWD, false, ring_depth(RWD * kWordsPerUnit, DEEP)>(L.down, cta, nctas, smem, tile, red, gate);
            asm volatile("cp.async.wait_group 0;" ::: "memory");  // the next layer's descriptor (long since landed); arrive's barrier publishes it
            if (l + 1 < P.n_layers) gate.arrive();
        }
        if (gate.trace != nullptr && threadIdx.x == 0) gate.trace[2] = now_ns();

        // Leave: the last CTA out re-arms the counters for the next launch (every CTA is past all of its waits by then).
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            const unsigned int before = atomicAdd(P.sync + 1, 1u);
            if (before + 1 == nctas) {
                P.sync[0] = 0;
                P.sync[1] = 0;
                __threadfence();
            }
        }
    }
}

using StepKernel = void (*)(StepParams);

struct Variant {
    int rw[4];  // rows per warp of the q/k/v, output, gate/up and down multiplies
    StepKernel tagged, barrier;
};

template <class F>
const Variant* variants(int& count) {
    constexpr bool heavy = sizeof(typename F::W) > 32;  // K-quants hold many registers per row
    if constexpr (heavy) {
        static const Variant v[] = {{{2, 2, 1, 2}, step_kernel<F, 2, 2, 1, 2, true, true>, step_kernel<F, 2, 2, 1, 2, true, false>},
                                    {{2, 1, 1, 1}, step_kernel<F, 2, 1, 1, 1, false, true>, step_kernel<F, 2, 1, 1, 1, false, false>},
                                    {{1, 1, 1, 1}, step_kernel<F, 1, 1, 1, 1, false, true>, step_kernel<F, 1, 1, 1, 1, false, false>}};
        count = 3;
        return v;
    } else {
        static const Variant v[] = {{{4, 2, 4, 2}, step_kernel<F, 4, 2, 4, 2, true, true>, step_kernel<F, 4, 2, 4, 2, true, false>},
                                    {{2, 1, 2, 1}, step_kernel<F, 2, 1, 2, 1, false, true>, step_kernel<F, 2, 1, 2, 1, false, false>},
                                    {{1, 1, 1, 1}, step_kernel<F, 1, 1, 1, 1, false, true>, step_kernel<F, 1, 1, 1, 1, false, false>}};
        count = 3;
        return v;
    }
}

const Variant* variants_of(int type, int& count) {
    switch (type) {
        case T_Q4_0: return variants<FQ4_0>(count);
        case T_Q8_0: return variants<FQ8_0>(count);
        case T_Q4_K: return variants<FQ4_K>(count);
        case T_Q6_K: return variants<FQ6_K>(count);
        case T_TQ2_0: return variants<FTQ2_0>(count);
        default: count = 0; return nullptr;
    }
}

// Rows per warp one multiply would like: more rows share the activation loads and the serial adds, as long as about
// half of all warps still get a row group (the rule of the one-kernel-per-operation path).
int wanted_rows_per_warp(const DecMatParams& p, bool pair, uint32_t sms) {
    uint32_t rows = 0;
    bool div4 = true, div2 = true;
    for (int i = 0; i < (pair ? 1 : p.count); ++i) rows += p.m[i].rows;
    for (int i = 0; i < p.count; ++i) {
        div4 = div4 && p.m[i].rows % 4 == 0;
        div2 = div2 && p.m[i].rows % 2 == 0;
    }
    const uint32_t enough = sms * kDecWarps / 2;
    if (div4 && rows / 4 >= enough) return 4;
    if (div2 && rows / 2 >= enough) return 2;
    return 1;
}

}  // namespace

struct StepPlan::Impl {
    StepKernel kernel = nullptr;
    bool tagged = true;
    StepLayerDesc* layers_dev = nullptr;
    unsigned int* sync_dev = nullptr;
    uint2* pairs_dev = nullptr;  // tagged exchange: hidden | q | k | v | scores | attended | gated, as {value, tag} pairs
    size_t pairs = 0;
    uint2* tagged_hidden = nullptr;
    float* plain_hidden = nullptr;
    uint32_t hidden_size = 0;
    uint32_t epoch = 0;          // launches so far; tags of a launch start above epoch * tags_per_launch
    uint32_t tags_per_launch = 0;
    uint32_t n_layers = 0, grid = 0, tile_offset = 0;
    uint32_t fault_layer = 0xffffffffu;
    size_t smem = 0;
    unsigned long long* trace = nullptr;
};

StepPlan::StepPlan() = default;
StepPlan::~StepPlan() {
    if (impl_ != nullptr) {
        if (impl_->layers_dev) cudaFree(impl_->layers_dev);
        if (impl_->sync_dev) cudaFree(impl_->sync_dev);
        if (impl_->pairs_dev) cudaFree(impl_->pairs_dev);
        delete impl_;
    }
}

bool StepPlan::build(const std::vector<StepLayerArgs>& layers, const StepShared& shared, uint32_t sms, cudaStream_t s, std::string& why_not) {
    StepShared sh = shared;
    if (layers.empty()) {
        why_not = "no layers";
        return false;
    }
    const int type = layers[0].q.type;
    for (const StepLayerArgs& L : layers) {
        for (const DevMatrix* m : {&L.q, &L.k, &L.v, &L.o, &L.gate, &L.up, &L.down}) {
            if (m->type != type) {
                why_not = "the layer matrices are not all of one type";
                return false;
            }
        }
    }
    int count = 0;
    const Variant* list = variants_of(type, count);
    if (list == nullptr) {
        why_not = "no persistent kernel for this weight type";
        return false;
    }
    if (sh.dim != 64 && sh.dim != 128) {
        why_not = "head size is not 64 or 128";
        return false;
    }
    // Measured on B200 (decode tok/s, persistent vs one kernel per operation): 0.6B-class Q4_0 (rows up to 3072 values)
    // 1282 vs 1135; 2B-class TQ2_0 (up to 6912) 664 vs 698; 7B-class Q4_0 (up to 14336, context 8192) 177 vs 198. Every
    // CTA re-reads the whole activation row of an operation, as tagged pairs twice the bytes: beyond a few thousand values
    // that traffic outweighs the saved launches. BRISK_CUDA_STEP=force overrides (tests use it to cover the wide variants).
    const uint32_t widest_row = std::max(std::max(sh.hidden_size, sh.heads * sh.dim), sh.ffn_size);
    const char* force = std::getenv("BRISK_CUDA_STEP");
    if (widest_row > 4096 && !(force != nullptr && std::strcmp(force, "force") == 0)) {
        why_not = "activation rows wider than 4096 values (the per-operation kernels are faster there)";
        return false;
    }
    const uint32_t group = sh.heads / sh.kv_heads;
    if (group > kMaxGroup) {
        why_not = "more than 8 query heads per K/V head";
        return false;
    }

    // BRISK_CUDA_STEP_SYNC=barrier keeps ordinary vectors and grid barriers between the operations (for comparison);
    // the default is the tagged exchange.
    const char* mode = std::getenv("BRISK_CUDA_STEP_SYNC");
    const bool tagged = !(mode != nullptr && std::strcmp(mode, "barrier") == 0);
    struct Freer {
        void operator()(void* p) const { cudaFree(p); }
    };
    std::unique_ptr<void, Freer> pairs_guard;
    uint2* pairs_dev = nullptr;
    const size_t q_dim = size_t(sh.heads) * sh.dim, kv_dim = size_t(sh.kv_heads) * sh.dim;
    const size_t pairs = sh.hidden_size + q_dim + 2 * kv_dim + size_t(sh.heads) * sh.max_context + q_dim + sh.ffn_size;
    uint2* tagged_hidden = nullptr;
    if (tagged) {
        BK_CUDA(cudaMalloc(&pairs_dev, pairs * sizeof(uint2)));
        pairs_guard.reset(pairs_dev);
        BK_CUDA(cudaMemsetAsync(pairs_dev, 0, pairs * sizeof(uint2), s));  // tag 0 is never expected
        uint2* at = pairs_dev;
        auto take = [&](size_t n) {
            float* p = reinterpret_cast<float*>(at);
            at += n;
            return p;
        };
        tagged_hidden = at;
        sh.hidden = take(sh.hidden_size);
        sh.q = take(q_dim);
        sh.k = take(kv_dim);
        sh.v = take(kv_dim);
        sh.scores = take(size_t(sh.heads) * sh.max_context);
        sh.attended = take(q_dim);
        sh.gated = take(sh.ffn_size);
    }

    std::vector<StepLayerDesc> descs(layers.size());
    for (size_t l = 0; l < layers.size(); ++l) {
        const StepLayerArgs& L = layers[l];
        StepLayerDesc& d = descs[l];
        std::memset(static_cast<void*>(&d), 0, sizeof(d));
        auto fill = [&](DecMatParams& p, std::initializer_list<std::pair<const DevMatrix*, float*>> targets, const float* x, const float* w, uint32_t cols, int epi) {
            p.count = 0;
            for (const auto& t : targets) {
                p.m[p.count] = *t.first;
                p.out[p.count] = t.second;
                ++p.count;
            }
            p.epi = epi; p.x = x; p.weight = w; p.eps = sh.eps; p.cols = cols; p.trace = nullptr; p.pdl = 0;
        };
        fill(d.qkv, {{&L.q, sh.q}, {&L.k, sh.k}, {&L.v, sh.v}}, sh.hidden, L.attn_norm, sh.hidden_size, EPI_STORE);
        fill(d.o, {{&L.o, sh.hidden}}, sh.attended, L.attn_sub_norm, sh.heads * sh.dim, EPI_ADD);
        fill(d.gate_up, {{&L.gate, sh.gated}, {&L.up, nullptr}}, sh.hidden, L.ffn_norm, sh.hidden_size, sh.act_epi);
        fill(d.down, {{&L.down, sh.hidden}}, sh.gated, L.ffn_sub_norm, sh.ffn_size, EPI_ADD);
        DecAttnParams& a = d.attn;
        a.q = sh.q; a.k = sh.k; a.v = sh.v; a.q_norm = L.q_norm; a.k_norm = L.k_norm; a.rope = sh.rope;
        a.q_bias = L.q_bias; a.k_bias = L.k_bias; a.v_bias = L.v_bias;
        a.k_cache = L.k_cache; a.v_cache = L.v_cache; a.scores = sh.scores; a.out = sh.attended; a.position = sh.position;
        a.heads = sh.heads; a.kv_heads = sh.kv_heads; a.dim = sh.dim; a.max_context = sh.max_context;
        a.eps = sh.eps; a.scale = sh.scale; a.neox = sh.neox; a.pdl = 0;
        a.slice_width = dec_attn_slice_width(sh.heads, sh.dim, sms);
    }
    if (sh.body_trace != nullptr) {
        StepLayerDesc& d = descs[std::min<size_t>(5, descs.size() - 1)];
        d.qkv.trace = sh.body_trace;
        d.o.trace = sh.body_trace + 8;
        d.gate_up.trace = sh.body_trace + 16;
        d.down.trace = sh.body_trace + 24;
        d.attn.trace = sh.body_trace + 32;
    }
    // One variant for all layers: the rows per warp every layer can take.
    int want[4] = {4, 4, 4, 4};
    for (StepLayerDesc& d : descs) {
        want[0] = std::min(want[0], wanted_rows_per_warp(d.qkv, false, sms));
        want[1] = std::min(want[1], wanted_rows_per_warp(d.o, false, sms));
        want[2] = std::min(want[2], wanted_rows_per_warp(d.gate_up, true, sms));
        want[3] = std::min(want[3], wanted_rows_per_warp(d.down, false, sms));
    }
    const Variant* pick = nullptr;
    for (int i = 0; i < count && pick == nullptr; ++i) {
        bool fits = true;
        for (int k = 0; k < 4; ++k) fits = fits && list[i].rw[k] <= want[k];
        if (fits) pick = &list[i];
    }
    if (pick == nullptr) {
        why_not = "no kernel variant fits the row counts";
        return false;
    }
    for (StepLayerDesc& d : descs) {
        dec_assign_groups(d.qkv, pick->rw[0], false);
        dec_assign_groups(d.o, pick->rw[1], false);
        dec_assign_groups(d.gate_up, pick->rw[2], true);
        dec_assign_groups(d.down, pick->rw[3], false);
    }

    const uint32_t widest = std::max(std::max(sh.hidden_size, sh.heads * sh.dim), sh.ffn_size);
    const size_t act = (dec_act_smem(widest) + 15) & ~size_t(15);
    const size_t multiply = act + dec_tile_floats(8) * sizeof(float);
    const size_t attention = std::max(dec_attn_out_smem(sh.max_context, dec_attn_slice_width(sh.heads, sh.dim, sms)), size_t(kDecWarps) * step_scores_warp_smem(group, sh.dim));
    const size_t smem = std::max(multiply, attention);
    int dev = 0, limit = 0, coop = 0;
    BK_CUDA(cudaGetDevice(&dev));
    BK_CUDA(cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    BK_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (coop == 0) {
        why_not = "the device has no cooperative launch";
        return false;
    }
    if (smem + 1024 > size_t(limit)) {
        why_not = "the context is too long for the persistent kernel's shared memory";
        return false;
    }
    const StepKernel kernel = tagged ? pick->tagged : pick->barrier;
    BK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    int per_sm = 0;
    BK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, int(kStepThreads), smem));
    if (per_sm < 1) {
        why_not = "the persistent kernel does not fit an SM";
        return false;
    }

    impl_ = new Impl();
    impl_->kernel = kernel;
    impl_->tagged = tagged;
    impl_->pairs_dev = static_cast<uint2*>(pairs_guard.release());
    impl_->pairs = pairs;
    impl_->tagged_hidden = tagged_hidden;
    impl_->plain_hidden = shared.hidden;
    impl_->hidden_size = shared.hidden_size;
    impl_->tags_per_launch = uint32_t(descs.size()) * 6 + 2;
    // BRISK_CUDA_TEST_POLL_TIMEOUT=1 (tests only): the second layer's first multiply waits for a tag nobody writes and every
    // wait gives up after 64 re-reads - the kernel ends at once with the error word set, and the host must raise, keep the
    // position and carry on with the per-operation kernels. Every access stays in bounds; nothing faults or hangs. The barrier
    // form has the word set from the start instead, as a barrier that ran out leaves it.
    const char* env = std::getenv("BRISK_CUDA_TEST_POLL_TIMEOUT");
    const bool inject = env != nullptr && std::strcmp(env, "1") == 0;
    {
        impl_->fault_layer = inject && tagged ? std::min<uint32_t>(1u, uint32_t(descs.size()) - 1) : 0xffffffffu;
        const uint32_t limit = inject && tagged ? 64u : kPollLimitDefault;
        BK_CUDA(cudaMemcpyToSymbolAsync(c_poll_limit, &limit, sizeof(limit), 0, cudaMemcpyHostToDevice, s));
    }
    impl_->n_layers = uint32_t(descs.size());
    impl_->grid = sms;
    impl_->tile_offset = uint32_t(act);
    impl_->smem = smem;
    BK_CUDA(cudaMalloc(&impl_->layers_dev, descs.size() * sizeof(StepLayerDesc)));
    BK_CUDA(cudaMalloc(&impl_->sync_dev, 64));
    BK_CUDA(cudaMemcpyAsync(impl_->layers_dev, descs.data(), descs.size() * sizeof(StepLayerDesc), cudaMemcpyHostToDevice, s));
    BK_CUDA(cudaMemsetAsync(impl_->sync_dev, 0, 64, s));
    if (inject && !tagged) BK_CUDA(cudaMemsetAsync(impl_->sync_dev + 2, 1, sizeof(unsigned int), s));
    BK_CUDA(cudaStreamSynchronize(s));  // descs goes out of scope
    char text[96];
    std::snprintf(text, sizeof text, "%s, rows per warp %d/%d/%d/%d, %u CTAs, %zu KB shared", tagged ? "tagged exchange" : "grid barriers", pick->rw[0],
                  pick->rw[1], pick->rw[2], pick->rw[3], sms, smem / 1024);
    description_ = text;
    return true;
}

void StepPlan::launch(cudaStream_t s) {
    StepParams P{};
    P.layers = impl_->layers_dev;
    P.n_layers = impl_->n_layers;
    P.sync = impl_->sync_dev;
    P.tile_offset = impl_->tile_offset;
    P.trace = impl_->trace;
    if (impl_->tagged) {
        // Tags must never repeat while old pairs are still in the buffers: when the 32-bit range runs out, wipe them.
        if (uint64_t(impl_->epoch + 2) * impl_->tags_per_launch >= (uint64_t(1) << 32)) {
            BK_CUDA(cudaMemsetAsync(impl_->pairs_dev, 0, impl_->pairs * sizeof(uint2), s));
            impl_->epoch = 0;
        }
        ++impl_->epoch;
        P.tag_base = impl_->epoch * impl_->tags_per_launch;
        P.fault_layer = impl_->fault_layer;
        P.plain_hidden = impl_->plain_hidden;
        P.tagged_hidden = impl_->tagged_hidden;
        P.hidden_size = impl_->hidden_size;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(impl_->grid);
    cfg.blockDim = dim3(kStepThreads);
    cfg.dynamicSmemBytes = impl_->smem;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    BK_CUDA(cudaLaunchKernelEx(&cfg, impl_->kernel, P));
}

bool StepPlan::graph_safe() const { return impl_ == nullptr || !impl_->tagged; }

void StepPlan::set_trace(unsigned long long* words) { impl_->trace = words; }

const unsigned int* StepPlan::error_word() const { return impl_->sync_dev + 2; }

void StepPlan::rearm(cudaStream_t s) {
    impl_->fault_layer = 0xffffffffu;
    BK_CUDA(cudaMemsetAsync(impl_->sync_dev, 0, 64, s));
    BK_CUDA(cudaStreamSynchronize(s));
}

}  // namespace bk
