// Decode path: the layer for a batch of at most eight tokens as one persistent kernel plus the combine.
//
// With a handful of tokens every active expert has at most eight rows, the layer is nothing
// but streaming the active experts' weights once (44 MB per expert), and what the staged
// chain of kernels spends between those streams -- kernel boundaries, the permute, the padding of every
// expert to a 128-row tensor-core tile, TMEM set-up -- costs more than the streams themselves.  Here:
//   * every CTA routes the (<= 8) tokens itself, with the same selection as the staged chain, and derives
//     the same active-expert table, so nothing has to be exchanged before the first weight byte is
//     requested;
//   * phase 1 (GEMM1 + SwiGLU): a unit is 8 SwiGLU columns of one active expert = 8 linear +
//     8 gated rows of W1, i.e. exactly one 16-row A tile of the warp-level
//     mma.sync.m16n8k32 (e4m3 x e4m3 -> fp32), with the expert's <= 8 token rows as the 8-wide
//     B tile.  The weights arrive by TMA, 16 rows x 1 KB per step (two boxes of 8 rows in
//     phase 1, one of 16 in phase 2) through a ring of four or five steps per half CTA, fed by a
//     producer warp per half; eight warps split a step along K, promote per 128-K block with the two scales
//     like the staged kernel, and meet in shared memory.  (Per-thread loads and per-row bulk copies both
//     left the HBM two thirds idle: the first for the loads in flight a thread can hold, the second for the
//     rate at which one thread can issue sixteen copies per step.  A consumer thread as producer left it
//     at 5.3 TB/s: freed slots waited for that thread's own share of the step and of the unit's sum.)
//     In the accumulator layout a thread owns the linear and the gated value of the same
//     (column, token), so SwiGLU needs no exchange.  v = silu(gate) * lin goes to a small
//     fp32 scratch (the 1x128 requantisation needs whole 128-column blocks, which span units);
//   * phase 2 (GEMM2): a worker waits for its expert's rows in the scratch, requantises them (same arithmetic as
//     the staged epilogue), streams 16 rows of W2 per unit the same way, and writes bf16 y rows; the first
//     weights are requested before that wait, so the wait and the requantisation hide behind their latency;
//   * the weighted combine is a kernel of its own (decode_combine_kernel): it is resident before this one ends,
//     so its start costs no more than a grid barrier would, and meanwhile the CTAs of the next
//     layer's decode kernel, which need this one's shared memory, can move in.
// Every wait on memory or an mbarrier is bounded; the named barrier of a half is met by all of its warps or none.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <cstdint>

#include "decode.cuh"
#include "layer.cuh"
#include "ptx.cuh"
#include "route_token.cuh"

namespace moe {

namespace {

constexpr int kDecWarps = 16;                           // consumer warps; two producer warps follow
constexpr int kConsumers = kDecWarps * 32;
constexpr int kDecThreads = kConsumers + 64;
constexpr int kHalfWarps = 8;                           // the CTA works as two halves of 8 warps
constexpr int kHalfThreads = kHalfWarps * 32;
constexpr int kDecMaxActive = kDecodeMaxTokens * kTopK; // 64 (token, expert) pairs at most
constexpr int kHidStride = kHidden + 64;                // row strides that spread rows over the banks
constexpr int kG1Cols = 8;                              // SwiGLU columns of a phase-1 unit
constexpr int kG1Units = kInter / kG1Cols;              // 256 per expert
constexpr int kG2Cols = 16;                             // output columns of a phase-2 unit
constexpr int kG2Units = kHidden / kG2Cols;             // 448 per expert
// A step = 16 weight rows x 1 KB of K (8 K blocks, one per warp of the half).
constexpr int kStepRows = 16;
constexpr int kStepK = kHalfWarps * kBlock;             // 1024 bytes of every row
constexpr int kStepStride = kStepK;                     // rows of a step lie densely, as TMA writes them
constexpr int kStepBytes = kStepRows * kStepK;          // 16 KB arrive per step
constexpr int kG1Steps = kHidden / kStepK;              // 7 per phase-1 unit
constexpr int kG2Steps = kInter / kStepK;               // 2 per phase-2 unit
constexpr int kRing = 4;                                // steps in flight per half ...
constexpr int kRingFew = 5;                             // ... and with at most kFewTokens tokens, whose rows leave room
constexpr int kFewTokens = 4;
constexpr int kCoopRouteTokens = 3;                     // up to here the CTA's warps route the tokens together
static_assert(kHidden % kStepK == 0 && kInter % kStepK == 0, "K splits into whole steps");

// Shared-memory pool: the hidden rows of all tokens, then the two weight rings.
__host__ __device__ constexpr int rows_tokens(int T) { return T <= kFewTokens ? kFewTokens : kDecodeMaxTokens; }
constexpr int kPoolFew = kFewTokens * kHidStride + 2 * kRingFew * kStepBytes;
constexpr int kPoolAll = kDecodeMaxTokens * kHidStride + 2 * kRing * kStepBytes;
constexpr int kPoolBytes = kPoolFew > kPoolAll ? kPoolFew : kPoolAll;
static_assert(kDecodeMaxTokens * kHidStride % 128 == 0 && kFewTokens * kHidStride % 128 == 0, "ring slots are 128-byte aligned");
static_assert(2 * kDecodeMaxTokens * kNumExperts * 4 <= 2 * kRing * kStepBytes, "routing scratch fits the idle rings");

struct DecodeShared {
    int abort;
    int pair_count[kDecodeMaxTokens];
    int pair_le[kDecMaxActive];                            // [token][pair] local expert, -1 past the token's pairs
    int pair_first[kDecMaxActive];                         // entry of that expert's first use
    float pair_w[kDecMaxActive];
    int act_expert[kDecMaxActive], act_m[kDecMaxActive], act_row0[kDecMaxActive];
    int act_tok[kDecMaxActive][kDecodeMaxTokens];
    int expert_m[kMaxLocalExperts];
    // routing scratch
    float r_gscore[kDecodeMaxTokens][kNumGroups];
    int r_kept[kDecodeMaxTokens][kTopKGroup];
    int r_count[kDecodeMaxTokens][kTopKGroup][32];
    int r_idx[kDecodeMaxTokens][kTopK];
    float r_sel[kDecodeMaxTokens][kTopK];
    float hid_scale[kDecodeMaxTokens][kHiddenBlocks];      // [token][kb]
    int stop_at[2];                                        // per half: ring position (2 slot + parity) no step will fill, or -1
    alignas(16) int4 step_desc[2][kRingFew];               // {unit, step, next unit or -1, -}; unit -1: no more
    alignas(8) uint64_t full_bar[2][kRingFew];
    alignas(8) uint64_t empty_bar[2][kRingFew];
    alignas(8) uint64_t hid_bar;
    alignas(16) float red[2][2][kHalfWarps][128];          // per half, by unit parity: the warps' partial sums
    alignas(128) uint8_t pool[kPoolBytes];
};
static_assert(sizeof(DecodeShared) <= 227 * 1024, "decode kernel shared memory");

__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// The SwiGLU scratch is its own flag: between launches every word holds kAbsent, a NaN that no arithmetic here
// produces (the hardware's NaN results are 0x7fffffff); phase 2 re-reads a word until it holds something else.
// A flag per expert would need a fence behind every unit's stores (measured: 20 % of the kernel).
constexpr uint32_t kAbsent = 0xffffffffu;
__device__ __forceinline__ float4 ld_relaxed_gpu(const float* p) {
    float4 v;
    asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_gpu(float* p, float v) {
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ bool is_there(const float4& v) {
    return __float_as_uint(v.x) != kAbsent && __float_as_uint(v.y) != kAbsent && __float_as_uint(v.z) != kAbsent &&
           __float_as_uint(v.w) != kAbsent;
}

// Untiled bulk copy global -> shared memory of this CTA, completion counted on an mbarrier.
// Both addresses and the size are multiples of 16 bytes.  No multicast.
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void mma_e4m3(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// One 128-K block of the warp-level MMA tile: `arow` points at this K block in weight row r of
// the staged step (row r + 8 lies 8 strides further), `brow` at the same K block of token slot
// r's row; r = lane / 4, c = lane % 4.  A thread takes bytes [16c, 16c+16) and [64+16c, 64+16c+16)
// of the block from each; which 4 bytes feed which k index of the MMA is the same for A and B,
// and a dot product does not care about more.  (The choice cannot depend on the row: a product
// pairs the A bytes of one lane group with the B bytes of another.  The weight rows are 1 KB apart,
// so rows r and r + 1, which share a shared-memory access phase, collide two-way; that is cheap.)
__device__ __forceinline__ void mma_half(float (&acc)[4], const uint8_t* arow, const uint4& b) {
    const uint4 lo = *reinterpret_cast<const uint4*>(arow);
    const uint4 hi = *reinterpret_cast<const uint4*>(arow + 8 * kStepStride);
    mma_e4m3(acc, lo.x, hi.x, lo.y, hi.y, b.x, b.y);
    mma_e4m3(acc, lo.z, hi.z, lo.w, hi.w, b.z, b.w);
}
__device__ __forceinline__ void mma_block(float (&acc)[4], const uint8_t* arow, const uint8_t* brow) {
    mma_half(acc, arow, *reinterpret_cast<const uint4*>(brow));
    mma_half(acc, arow + 64, *reinterpret_cast<const uint4*>(brow + 64));
}

// How the work is drawn.  Workers (half CTAs) draw tickets from a counter; a ticket stands for a run of
// consecutive units.  Of each phase the first tickets, one per worker, stand for long runs (seven eighths of
// the phase: few changes of expert, whose rows phase 2 has to requantise again), the rest for short ones that
// even out how fast the workers get their weights.  All of phase 1 is drawn before phase 2, and phase 2 waits
// only for phase-1 units, i.e. for workers that are running: the waits end whatever part of the grid is
// resident, so the launch needs no co-residency guarantee (a cooperative launch starts 3 us later here: it does
// not overlap its predecessor's end).
struct PhasePlan {
    int units, in_runs, runs, rest_run, tickets;
    __device__ __forceinline__ void make(int n, int workers) {
        units = n;
        in_runs = n >= 2 * workers ? n / 8 * 7 : 0;
        runs = in_runs > 0 ? workers : 0;
        const int rest = n - in_runs;
        rest_run = rest / (workers * 4);
        if (rest_run < 1) rest_run = 1;
        tickets = runs + (rest + rest_run - 1) / rest_run;
    }
    __device__ __forceinline__ void range(int ticket, int& begin, int& end) const {
        if (ticket < runs) {
            begin = (int)((long long)in_runs * ticket / runs);
            end = (int)((long long)in_runs * (ticket + 1) / runs);
        } else {
            begin = in_runs + (ticket - runs) * rest_run;
            end = begin + rest_run < units ? begin + rest_run : units;
        }
    }
};
constexpr int kPhase2Bit = 1 << 20;   // unit numbers of phase 2 carry it

__global__ void __launch_bounds__(kDecThreads, 1) decode_layer_kernel(
    DecodeArgs a, const __grid_constant__ CUtensorMap tmap_w1, const __grid_constant__ CUtensorMap tmap_w2, Workspace ws)
{
    extern __shared__ __align__(128) uint8_t smem_raw[];
    DecodeShared* sh = reinterpret_cast<DecodeShared*>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r = lane >> 2, c = lane & 3;   // MMA fragment coordinates
    const int T = a.T, E = a.num_local_experts;
    const bool clocked = blockIdx.x == 0 && tid == 0;
    auto stamp = [&](int i) { if (clocked) ws.ctrl->dec_time[i] = global_timer_ns(); };
    volatile int* abort_flag = &sh->abort;

    // Set-up that depends on no earlier kernel, while the predecessor in the stream drains: barriers, and
    // requests that bring the call's small inputs from HBM into L2 (the weights of the layers before have
    // pushed them out; a prefetch returns no value, so it may run ahead of the kernel that writes them).
    pdl_launch_dependents();
    if (tid == 0) {
        sh->abort = 0;
        sh->stop_at[0] = sh->stop_at[1] = -1;
        prefetch_tmap(&tmap_w1);
        prefetch_tmap(&tmap_w2);
        mbar_init(smem_u32(&sh->hid_bar), 1);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < kRingFew; ++j) {
                mbar_init(smem_u32(&sh->full_bar[h][j]), 1);
                mbar_init(smem_u32(&sh->empty_bar[h][j]), kHalfWarps);
            }
        fence_mbar_init();
    }
    if (tid < T * 8) prefetch_l2(a.logits + (size_t)tid * 32);
    else if (tid >= 64 && tid < 68) prefetch_l2(a.bias + (size_t)(tid - 64) * 64);
    else if (tid >= 128 && tid < 128 + kHiddenBlocks) prefetch_l2(a.hscale + (size_t)(tid - 128) * T);
    else if (tid >= 192 && tid < 192 + kHidden / 128) {
        for (int t = 0; t < T; ++t) prefetch_l2(a.hidden + (size_t)t * kHidden + (size_t)(tid - 192) * 128);
    }
    pdl_wait();
    // the first ticket travels while the tables are made (an unused one does no harm)
    int first_ticket = 0;
    if (warp >= kDecWarps && lane == 0) first_ticket = (int)atomicAdd(&ws.ctrl->dec_ticket, 1u);
    // A failure that an earlier launch recorded stays in the status word until the host has read it
    // (moe_fp8_b200_check clears it; the next run then clears counter and scratch).  Until then this kernel does
    // nothing: with a stale counter it would leave units out, with stale words phase 2 would not wait.
    // Every CTA reads the same word; within one launch it can only change after a full wait limit.
    if (__ldcg(&ws.ctrl->status) != kStatusOk) return;
    stamp(0);

    // The tokens' hidden rows start moving before anything else: nothing depends on routing here.
    if (tid == 0) {
        const uint32_t hb = smem_u32(&sh->hid_bar);
        mbar_expect_tx(hb, (uint32_t)T * kHidden);
        for (int t = 0; t < T; ++t)
            bulk_g2s(smem_u32(sh->pool + t * kHidStride), a.hidden + (size_t)t * kHidden, kHidden, hb);
    }
    for (int q = tid; q < T * kHiddenBlocks; q += kDecThreads) {
        const int t = q % T, kb = q / T;
        sh->hid_scale[t][kb] = __ldg(a.hscale + q);   // [56, T] -> [token][kb]
    }

    // ------------------------------------------------------------------ routing (every CTA)
    // For up to three tokens: the same selection as route_token_warp (route_token.cuh), spread over the CTA's
    // warps (2.6 us for one token, 1.1 us more for each further one, where a warp per token takes 5 us for any
    // number of them).  Scores and their order-preserving keys go to
    // shared memory; one warp per (token, group) forms the group score; one thread per token keeps
    // the four best groups; then the eight argmax rounds are replaced by counting, for each of the
    // 128 live scores, how many of the others beat it (higher key, or equal key and earlier in the
    // reference's tie order): the score with count k is the k-th pick.  Same picks, same order.
    if (tid < kMaxLocalExperts) sh->expert_m[tid] = 0;
    if (tid < kDecMaxActive) sh->pair_le[tid] = -1;
    float* r_s = reinterpret_cast<float*>(sh->pool + rows_tokens(T) * kHidStride);        // [T][256], idle ring
    uint32_t* r_key = reinterpret_cast<uint32_t*>(r_s + kDecodeMaxTokens * kNumExperts);  // [T][256]
    stamp(12);
    if (T <= kCoopRouteTokens) {
        for (int q = tid; q < T * kNumExperts; q += kDecThreads) {
            const float l = __ldg(a.logits + q);
            const float sig = 1.0f / (1.0f + __expf(-l));
            r_s[q] = sig;
            r_key[q] = float_to_ordered(sig + __bfloat162float(a.bias[q & (kNumExperts - 1)]));
        }
        for (int q = tid; q < T * kTopKGroup * 32; q += kDecThreads) (&sh->r_count[0][0][0])[q] = 0;
        __syncthreads();
        for (int task = warp; task < T * kNumGroups; task += kDecThreads / 32) {   // group score = two largest of the group
            const uint32_t key = r_key[task * 32 + lane];
            const uint32_t k1 = __reduce_max_sync(0xffffffffu, key);
            const uint32_t holders = __ballot_sync(0xffffffffu, key == k1);
            uint32_t k2 = k1;
            if (__popc(holders) < 2) k2 = __reduce_max_sync(0xffffffffu, key == k1 ? 0u : key);
            if (lane == 0) sh->r_gscore[task / kNumGroups][task % kNumGroups] = ordered_to_float(k1) + ordered_to_float(k2);
        }
        __syncthreads();
        if (tid < T) {   // four best groups, lowest index first on ties
            uint32_t kept_mask = 0;
            for (int k = 0; k < kTopKGroup; ++k) {
                float best = kNegSentinel;
                int best_i = -1;
#pragma unroll
                for (int i = 0; i < kNumGroups; ++i) {
                    const float gsc = sh->r_gscore[tid][i];
                    if (!((kept_mask >> i) & 1u) && gsc > best) { best = gsc; best_i = i; }
                }
                if (best_i >= 0) {
                    kept_mask |= 1u << best_i;
                    sh->r_kept[tid][k] = best_i;
                } else {
                    sh->r_kept[tid][k] = k;   // unreachable with finite scores; keeps the indices valid
                }
            }
        }
        __syncthreads();
        // count[t][j][lane]: how many live scores beat score `lane` of the j-th kept group; the work of one
        // (token, group) is split over four warps, one per opposing group
        for (int task = warp; task < T * kTopKGroup * kTopKGroup; task += kDecThreads / 32) {
            const int t = task / (kTopKGroup * kTopKGroup), j = (task / kTopKGroup) % kTopKGroup, part = task % kTopKGroup;
            const int g = sh->r_kept[t][j], g2 = sh->r_kept[t][part];
            const uint32_t key = r_key[t * kNumExperts + g * 32 + lane];
            const uint32_t tie = (uint32_t)g * 32u + (__brev((uint32_t)lane) >> 27);
            const uint32_t* other = r_key + t * kNumExperts + g2 * 32;
            int beat = 0;
#pragma unroll 8
            for (int l2 = 0; l2 < 32; ++l2) {
                const uint32_t key2 = other[l2];
                const uint32_t tie2 = (uint32_t)g2 * 32u + (__brev((uint32_t)l2) >> 27);
                beat += (key2 > key || (key2 == key && tie2 < tie)) ? 1 : 0;
            }
            atomicAdd(&sh->r_count[t][j][lane], beat);
        }
        __syncthreads();
        for (int task = warp; task < T * kTopKGroup; task += kDecThreads / 32) {
            const int t = task / kTopKGroup, j = task % kTopKGroup;
            const int rank = sh->r_count[t][j][lane];
            if (rank < kTopK) {
                const int ge = sh->r_kept[t][j] * 32 + lane;
                sh->r_idx[t][rank] = ge;
                sh->r_sel[t][rank] = r_s[t * kNumExperts + ge];
            }
        }
        // The scratch lies in half 0's first ring slots, which TMA writes next: ordinary accesses and the async
        // proxy's to the same bytes want this fence, by every thread that made them, in front of the barrier.
        fence_proxy_async_smem();
    } else if (warp < T) {
        // more tokens than that: one warp per token runs the staged chain's routine, the tokens in parallel
        int idx[kTopK];
        float wn[kTopK];
        route_token_warp(a.logits + (size_t)warp * kNumExperts, a.bias, lane, idx, wn);
#pragma unroll
        for (int k = 0; k < kTopK; ++k)
            if (k == lane) { sh->r_idx[warp][k] = idx[k]; sh->r_sel[warp][k] = wn[k]; }   // already normalised
    }
    __syncthreads();
    stamp(8);
    // Dispatch, one warp per token: lane s applies the policy to 32-expert shard s, and a lane's pairs follow
    // those of the lanes before it.
    if (warp < T) {
        const int t = warp;
        int idx[kTopK];
        float wn[kTopK];
        float sumw = 1e-20f;
#pragma unroll
        for (int k = 0; k < kTopK; ++k) { idx[k] = sh->r_idx[t][k]; sumw += sh->r_sel[t][k]; }
        const float inv = 1.0f / sumw;
#pragma unroll
        for (int k = 0; k < kTopK; ++k) wn[k] = T <= kCoopRouteTokens ? sh->r_sel[t][k] * inv : sh->r_sel[t][k];
        if (blockIdx.x == 0 && lane < kTopK) {
            ws.topk_idx[(size_t)t * kTopK + lane] = sh->r_idx[t][lane];
            ws.topk_weight[(size_t)t * kTopK + lane] = T <= kCoopRouteTokens ? sh->r_sel[t][lane] * inv : sh->r_sel[t][lane];
        }
        int n_pairs = 0;
        int p_le[kTopK];
        float p_w[kTopK];
#pragma unroll
        for (int i = 0; i < kTopK; ++i) { p_le[i] = 0; p_w[i] = 0.0f; }
        if (lane < E / kShardExperts) dispatch_one_shard(idx, wn, lane, a.local_expert_offset, a.pol, a.rsf, n_pairs, p_le, p_w);
        int incl = n_pairs;
#pragma unroll
        for (int off = 1; off < 8; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += y;
        }
        const int pair_base = incl - n_pairs;
#pragma unroll
        for (int i = 0; i < kTopK; ++i) {
            if (i < n_pairs) {
                sh->pair_le[t * kTopK + pair_base + i] = p_le[i];
                sh->pair_w[t * kTopK + pair_base + i] = p_w[i];
            }
        }
        if (lane == 7) sh->pair_count[t] = incl;
        stamp(9);
    }
    __syncthreads();
    // Active experts in order of first use, rows of an expert in token order: the same in every CTA, so unit u
    // means the same thing everywhere.  One thread per (token, pair) entry looks the others over.
    const int n_entries = T * kTopK;
    const int my_le = tid < n_entries ? sh->pair_le[tid] : -1;
    int my_first = kDecMaxActive, my_slot = 0, my_m = 0;
    if (my_le >= 0) {
        for (int j = 0; j < n_entries; ++j) {
            if (sh->pair_le[j] == my_le) {
                ++my_m;
                if (j < tid) ++my_slot;
                if (my_first == kDecMaxActive) my_first = j;
            }
        }
    }
    if (tid < n_entries) sh->pair_first[tid] = my_first;
    const int n_active = __syncthreads_count(my_le >= 0 && my_first == tid);
    if (my_le >= 0) {
        int ai = 0, row0 = 0;
        for (int j = 0; j < n_entries; ++j) {
            const int f = sh->pair_first[j];
            if (f < my_first) { ++row0; ai += f == j ? 1 : 0; }
        }
        if (my_first == tid) {
            sh->act_expert[ai] = my_le;
            sh->act_m[ai] = my_m;
            sh->act_row0[ai] = row0;
            sh->expert_m[my_le] = my_m;
        }
        sh->act_tok[ai][my_slot] = tid / kTopK;
        if (blockIdx.x == 0) {   // the tables that the combine, other entry points and the tests read
            ws.pair_code[tid] = ((uint32_t)my_le << 24) | (uint32_t)my_slot;
            ws.pair_weight[tid] = sh->pair_w[tid];
        }
        if (blockIdx.x == 0) ws.pair_row[tid] = row0 + my_slot;
    } else if (blockIdx.x == 0 && tid < n_entries) {
        ws.pair_row[tid] = -1;
    }
    if (blockIdx.x == 0 && tid < T) ws.pair_count[tid] = sh->pair_count[tid];
    stamp(10);
    __syncthreads();
    if (blockIdx.x == 0 && tid < E) ws.ctrl->expert_rows[tid] = sh->expert_m[tid];
    stamp(11);
    stamp(1);
    float* act = ws.dec_act;   // [rows, 2048] fp32 SwiGLU output

    // The 16 consumer warps work as two independent halves of 8 (named barriers 1 and 2): a half is one
    // worker with its own weight ring and reduction buffer, so an SM always has two
    // units in flight and the work is dealt twice as finely.  A producer warp per half (one lane) draws the units
    // and requests a step (16 rows x 1 KB) as soon as its ring slot is free -- of the next unit and of the next
    // phase as well.  Warp hw of the half consumes K block hw of every step.
    const bool producer = warp >= kDecWarps;
    const int half = producer ? warp - kDecWarps : warp >> 3, hw = warp & (kHalfWarps - 1), htid = tid & (kHalfThreads - 1);
    const int workers = (int)gridDim.x * 2;
    const int bar_id = 1 + half;
    const int ring = T <= kFewTokens ? kRingFew : kRing;
    uint8_t* const wring = sh->pool + rows_tokens(T) * kHidStride + half * ring * kStepBytes;
    uint64_t* const full_bar = sh->full_bar[half];
    uint64_t* const empty_bar = sh->empty_bar[half];

    if (producer) {
        if (lane != 0) return;
        PhasePlan p1, p2;
        p1.make(n_active * kG1Units, workers);
        p2.make(n_active * kG2Units, workers);
        const int tickets = p1.tickets + p2.tickets;
        int slot = 0, issued = 0;
        uint32_t phase = 1;   // the first pass over the ring finds every slot free
        bool ok = true;
        auto range_of = [&](int ticket, int& begin, int& end, int& bit) {
            if (ticket < p1.tickets) { p1.range(ticket, begin, end); bit = 0; }
            else { p2.range(ticket - p1.tickets, begin, end); bit = kPhase2Bit; }
        };
        int ticket = first_ticket;
        while (ok && ticket < tickets) {
            int u, end, bit;
            range_of(ticket, u, end, bit);
            int next_ticket = tickets;
            for (; ok && u < end; ++u) {
                const int steps = bit ? kG2Steps : kG1Steps;
                const int ai = bit ? u / kG2Units : u / kG1Units;
                const int in = bit ? u - ai * kG2Units : u - ai * kG1Units;
                const int row = bit ? sh->act_expert[ai] * kHidden + in * kG2Cols : sh->act_expert[ai] * kGemm1Out + in * kG1Cols;
                // The next ticket is drawn with the run's last unit: early enough for its round trip to pass while
                // that unit's steps are requested, and not before (a ticket drawn with a long run still ahead
                // would be held for that long).
                if (u + 1 == end) next_ticket = (int)atomicAdd(&ws.ctrl->dec_ticket, 1u);
                for (int i = 0; i < steps; ++i) {
                    if (!mbar_wait(smem_u32(&empty_bar[slot]), phase, abort_flag)) { ok = false; break; }
                    int next = u + 1 < end ? u + 1 + bit : -1;
                    if (u + 1 == end && i >= (steps > 2 ? 2 : steps - 1) && next_ticket < tickets) {
                        // by now the next ticket is there: the run's last unit names the first of the next run
                        int nb, ne, nbit;
                        range_of(next_ticket, nb, ne, nbit);
                        next = nb + nbit;
                    }
                    sh->step_desc[half][slot] = make_int4(u + bit, i, next, 0);
                    const uint32_t bar = smem_u32(&full_bar[slot]);
                    const uint32_t dst = smem_u32(wring + slot * kStepBytes);
                    mbar_expect_tx(bar, kStepBytes);
                    if (!bit) {
                        tma_load_2d(dst, &tmap_w1, bar, i * (kStepK / 4), row);                              // 8 linear rows
                        tma_load_2d(dst + 8 * kStepStride, &tmap_w1, bar, i * (kStepK / 4), row + kInter);   // 8 gated rows
                    } else {
                        tma_load_2d(dst, &tmap_w2, bar, i * (kStepK / 4), row);
                    }
                    ++issued;
                    if (++slot == ring) { slot = 0; phase ^= 1u; }
                }
            }
            ticket = next_ticket;
        }
        if (ok && mbar_wait(smem_u32(&empty_bar[slot]), phase, abort_flag)) {
            sh->step_desc[half][slot] = make_int4(-1, 0, -1, 0);
            mbar_arrive(smem_u32(&full_bar[slot]));
        } else {
            // This is where the half stops: the consumers take every step issued so far and find the position here.
            *(volatile int*)&sh->stop_at[half] = 2 * slot + (int)(phase ^ 1u);
            // leave only after the copies in flight have landed (bounded)
            for (int g = issued > ring ? issued - ring : 0; g < issued; ++g) {
                const uint32_t bar = smem_u32(&full_bar[g % ring]);
                const uint64_t t0 = global_timer_ns();
                while (!mbar_try_wait(bar, (uint32_t)((g / ring) & 1)) && global_timer_ns() - t0 < kWaitLimitNs) {}
            }
        }
        return;
    }

    int slot = 0;            // ring slot and parity of the next step to consume
    uint32_t phase = 0;
    bool ok = true;
    auto release = [&]() {
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&empty_bar[slot]));
        if (++slot == ring) { slot = 0; phase ^= 1u; }
    };
    // Waits for the next step; false: the half ends here.  The eight warps meet once per unit at a named barrier,
    // which has no limit of its own, so all of them must end at the same step.  Their producer alone decides which:
    // it issues a step or, when one of its waits runs out or the CTA's abort flag is up, names the ring position where
    // it stopped; a step that was issued arrives.  (No other position has that slot and parity: the producer is at
    // most one ring ahead.)  The abort flag itself is not looked at here, since one warp might find its step arrived
    // and another one the flag.  The limit behind it is for a copy that never lands: longer than any wait of the
    // producer, and then no warp of the half gets past that step.
    const volatile int* stop_at = &sh->stop_at[half];
    auto arrived = [&]() -> bool {
        const uint32_t bar = smem_u32(&full_bar[slot]);
        if (mbar_try_wait(bar, phase)) return true;
        const uint64_t t0 = global_timer_ns();
        for (uint32_t it = 1;; ++it) {
            if (mbar_try_wait(bar, phase)) return true;
            if ((it & 0xffu) == 0u && (*stop_at == 2 * slot + (int)phase || global_timer_ns() - t0 > 4 * kWaitLimitNs)) return false;
        }
    };
    // the first step of the next unit and what the producer wrote about it ({-1, ...} once there is no more work)
    int4 d = make_int4(-1, 0, -1, 0);
    auto next_unit = [&]() {
        ok = ok && arrived();
        d.x = -1;
        if (ok) d = sh->step_desc[half][slot];
    };
    // The weight scales of a unit's K blocks sit in lanes of the warp that uses them (phase 1: lanes 0..13, 7
    // linear and 7 gated; phase 2: lanes 0 and 1), fetched one unit ahead so that no step waits for them.
    auto unit_scales = [&](int unit) -> float {
        float v = 0.0f;
        if (unit & kPhase2Bit) {
            const int u = unit - kPhase2Bit;
            if (lane < kG2Steps) {
                const int e = sh->act_expert[u / kG2Units], hh = u % kG2Units;
                v = __ldg(a.s2 + ((size_t)e * kHiddenBlocks + hh / (kBlock / kG2Cols)) * kInterBlocks + hw + kHalfWarps * lane);
            }
        } else if (lane < 2 * kG1Steps) {
            const int e = sh->act_expert[unit / kG1Units], gg = unit % kG1Units;
            const int blk = gg / (kBlock / kG1Cols) + (lane >= kG1Steps ? kInter / kBlock : 0);
            const int kb = hw + kHalfWarps * (lane % kG1Steps);
            v = __ldg(a.s1 + ((size_t)e * (kGemm1Out / kBlock) + blk) * kHiddenBlocks + kb);
        }
        return v;
    };
    // the hidden rows must have landed before the first MMA (a wait that fails sets the abort flag and is reported at
    // the end: a warp does not leave its half, see arrived)
    mbar_wait(smem_u32(&sh->hid_bar), 0u, abort_flag);

    float sc_next = 0.0f;
    int loaded_for = -1;   // unit that sc_next belongs to
    int parity = 0;
    // ------------------------------------------------------------------ phase 1: GEMM1 + SwiGLU
    for (next_unit(); d.x >= 0 && !(d.x & kPhase2Bit); next_unit()) {
        const int ai = d.x / kG1Units, g = d.x % kG1Units, m = sh->act_m[ai];
        const float sc_cur = loaded_for == d.x ? sc_next : unit_scales(d.x);
        const uint8_t* brow = sh->pool + sh->act_tok[ai][r < m ? r : 0] * kHidStride + hw * kBlock + 16 * c;
        const float* sc0 = sh->hid_scale[sh->act_tok[ai][2 * c < m ? 2 * c : 0]] + hw;
        const float* sc1 = sh->hid_scale[sh->act_tok[ai][2 * c + 1 < m ? 2 * c + 1 : 0]] + hw;
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        int next = -1;
#pragma unroll
        for (int i = 0; i < kG1Steps; ++i) {
            if (i > 0 && !arrived()) { ok = false; break; }
            float raw[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            mma_block(raw, wring + slot * kStepBytes + r * kStepStride + hw * kBlock + 16 * c, brow + i * kHalfWarps * kBlock);
            if (i == kG1Steps - 1) next = sh->step_desc[half][slot].z;
            release();
            const float sl = __shfl_sync(0xffffffffu, sc_cur, i), sg = __shfl_sync(0xffffffffu, sc_cur, kG1Steps + i);
            const float sa0 = sc0[i * kHalfWarps], sa1 = sc1[i * kHalfWarps];
            acc[0] = fmaf(raw[0], sa0 * sl, acc[0]);
            acc[1] = fmaf(raw[1], sa1 * sl, acc[1]);
            acc[2] = fmaf(raw[2], sa0 * sg, acc[2]);
            acc[3] = fmaf(raw[3], sa1 * sg, acc[3]);
        }
        if (!ok) break;
        if (next >= 0) { sc_next = unit_scales(next); loaded_for = next; }
        // the unit is complete: add the eight warps' partial sums
        float* red = &sh->red[half][parity][0][0];
        parity ^= 1;
        *reinterpret_cast<float4*>(red + hw * 128 + lane * 4) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        named_bar_sync(bar_id, kHalfThreads);
        if (htid < 64) {
            const int l = htid & 31, jj = htid >> 5;
            float lin = 0.0f, gate = 0.0f;
#pragma unroll
            for (int w = 0; w < kHalfWarps; ++w) {
                lin += red[w * 128 + l * 4 + jj];
                gate += red[w * 128 + l * 4 + 2 + jj];
            }
            const int row = 2 * (l & 3) + jj, col = g * kG1Cols + (l >> 2);
            if (row < m) {
                const float x1 = round_bf16(lin), x2 = round_bf16(gate);
                const float silu = a.silu_exact ? x2 / (1.0f + __expf(-x2))
                                                : x2 * (0.5f * (x2 * rsqrtf(fmaf(x2, x2, 4.0f)) + 1.0f));
                st_relaxed_gpu(act + (size_t)(sh->act_row0[ai] + row) * kInter + col, silu * x1);
            }
        }
    }

    // ------------------------------------------------------------------ phase 2: requantisation + GEMM2
    stamp(2);
    int staged = -1;
    uint4 bfrag[kG2Steps][2];      // this warp's K blocks of the staged expert's rows
    float bscale[kG2Steps][2];     // ... and the scales of rows 2c and 2c + 1
    for (; ok && d.x >= 0; next_unit()) {
        const int u = d.x - kPhase2Bit, ai = u / kG2Units, hg = u % kG2Units, m = sh->act_m[ai];
        if (ai != staged) {
            // 1x128 requantisation as in the staged GEMM1 epilogue: scale = amax / 448 (1 if the block is
            // zero), payload e4m3(v * (1 / scale)).  A warp needs its own two K blocks only and keeps them
            // in registers as B fragments, so the warps take another expert up without meeting.
#pragma unroll
            for (int k2 = 0; k2 < kG2Steps; ++k2) {
                const float* src = act + (size_t)sh->act_row0[ai] * kInter + (hw + kHalfWarps * k2) * kBlock + lane * 4;
                bfrag[k2][0] = bfrag[k2][1] = make_uint4(0u, 0u, 0u, 0u);
                bscale[k2][0] = bscale[k2][1] = 0.0f;
#pragma unroll
                for (int j0 = 0; j0 < kDecodeMaxTokens; j0 += 4) {
                    if (j0 >= m) break;
                    float4 v[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (j0 + j < m) v[j] = ld_relaxed_gpu(src + (size_t)(j0 + j) * kInter);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (j0 + j >= m) break;
                        if (!__all_sync(0xffffffffu, is_there(v[j]))) {   // phase-1 units still under way elsewhere
                            const uint64_t t0 = global_timer_ns();
                            do {
                                if (!is_there(v[j])) v[j] = ld_relaxed_gpu(src + (size_t)(j0 + j) * kInter);
                                if (*abort_flag != 0 || global_timer_ns() - t0 > kWaitLimitNs) sh->abort = 1;
                            } while (!__all_sync(0xffffffffu, is_there(v[j]) || *abort_flag != 0));
                        }
                        float amax = fmaxf(fmaxf(fabsf(v[j].x), fabsf(v[j].y)), fmaxf(fabsf(v[j].z), fabsf(v[j].w)));
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
                        const float sc = amax > 0.0f ? amax / 448.0f : 1.0f;
                        const float inv = 1.0f / sc;
                        const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[j].x * inv, v[j].y * inv), __NV_SATFINITE, __NV_E4M3);
                        const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[j].z * inv, v[j].w * inv), __NV_SATFINITE, __NV_E4M3);
                        const uint32_t w = lo | (hi << 16);   // bytes 4 lane .. 4 lane + 3 of the row's block
                        // lanes of fragment row j0 + j take bytes 16c .. 16c+15 and 64+16c .. 64+16c+15
                        uint32_t g[8];
#pragma unroll
                        for (int q = 0; q < 8; ++q) g[q] = __shfl_sync(0xffffffffu, w, (q >> 2) * 16 + 4 * c + (q & 3));
                        if (r == j0 + j) {
                            bfrag[k2][0] = make_uint4(g[0], g[1], g[2], g[3]);
                            bfrag[k2][1] = make_uint4(g[4], g[5], g[6], g[7]);
                        }
                        if (2 * c == j0 + j) bscale[k2][0] = sc;
                        if (2 * c + 1 == j0 + j) bscale[k2][1] = sc;
                    }
                }
            }
            if (staged < 0) stamp(3);
            staged = ai;
        }
        const float sc_cur = loaded_for == d.x ? sc_next : unit_scales(d.x);
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        int next = -1;
#pragma unroll
        for (int i = 0; i < kG2Steps; ++i) {
            if (i > 0 && !arrived()) { ok = false; break; }
            float raw[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            const uint8_t* arow = wring + slot * kStepBytes + r * kStepStride + hw * kBlock + 16 * c;
            mma_half(raw, arow, bfrag[i][0]);
            mma_half(raw, arow + 64, bfrag[i][1]);
            if (i == kG2Steps - 1) next = sh->step_desc[half][slot].z;
            release();
            const float sw = __shfl_sync(0xffffffffu, sc_cur, i);
            const float sa0 = bscale[i][0] * sw, sa1 = bscale[i][1] * sw;
            acc[0] = fmaf(raw[0], sa0, acc[0]);
            acc[1] = fmaf(raw[1], sa1, acc[1]);
            acc[2] = fmaf(raw[2], sa0, acc[2]);
            acc[3] = fmaf(raw[3], sa1, acc[3]);
        }
        if (!ok) break;
        if (next >= 0) { sc_next = unit_scales(next); loaded_for = next; }
        float* red = &sh->red[half][parity][0][0];
        parity ^= 1;
        *reinterpret_cast<float4*>(red + hw * 128 + lane * 4) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        named_bar_sync(bar_id, kHalfThreads);
        if (htid < 128) {
            const int l = htid >> 2, q = htid & 3;
            const int row = 2 * (l & 3) + (q & 1), hrow = hg * kG2Cols + (l >> 2) + 8 * (q >> 1);
            float sum = 0.0f;
#pragma unroll
            for (int w = 0; w < kHalfWarps; ++w) sum += red[w * 128 + l * 4 + q];
            if (row < m) ws.y[(size_t)(sh->act_row0[ai] + row) * kHidden + hrow] = __float2bfloat16_rn(sum);
        }
    }
    if (staged < 0) stamp(3);   // no phase-2 unit came this way
    if (*abort_flag != 0) ok = false;
    if (!ok) {
        // a half that gave up on a wait says so; the producers let their copies land before they leave
        atomicCAS(&ws.ctrl->status, kStatusOk, kStatusDecodeTimeout);
        sh->abort = 1;
    }
    stamp(4);
}

// The weighted combine of the decode kernel's rows: same arithmetic and pair order as combine_kernel, the rows
// found through pair_row (one load instead of pair code -> expert offset), all requested at once.  Small CTAs
// (a seventh of a row each), so that they fit beside a running decode CTA's registers.
constexpr int kDecCombineThreads = 128;
constexpr int kDecCombineParts = kHidden / 8 / kDecCombineThreads;   // 7
static_assert(kDecCombineParts * kDecCombineThreads * 8 == kHidden, "a row splits into whole CTAs");
__global__ void __launch_bounds__(kDecCombineThreads) decode_combine_kernel(Workspace ws, __nv_bfloat16* __restrict__ out)
{
    const int t = blockIdx.y, ch = blockIdx.x * kDecCombineThreads + threadIdx.x;
    const bool clocked = t == 0 && blockIdx.x == 0 && threadIdx.x == 0;
    pdl_launch_dependents();
    pdl_wait();
    // the decode kernel has completed: its counter and (below) its scratch are put back for the next launch
    if (clocked) { ws.ctrl->dec_ticket = 0; ws.ctrl->dec_time[5] = global_timer_ns(); }
    const int4* pr = reinterpret_cast<const int4*>(ws.pair_row + (size_t)t * kTopK);
    const float4* pw = reinterpret_cast<const float4*>(ws.pair_weight + (size_t)t * kTopK);
    const int status = __ldcg(&ws.ctrl->status);
    const int4 ra = __ldcg(pr), rb = __ldcg(pr + 1);
    const float4 wa = __ldcg(pw), wb = __ldcg(pw + 1);
    if (status != kStatusOk) return;   // the rows are not there (see decode_layer_kernel)
    const int rows[kTopK] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, rb.w};
    const float wts[kTopK] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
    uint4 raw[kTopK];
#pragma unroll
    for (int p = 0; p < kTopK; ++p)
        if (rows[p] >= 0) raw[p] = __ldcg(reinterpret_cast<const uint4*>(ws.y + (size_t)rows[p] * kHidden) + ch);
    if (ch < kInter / 4) {
#pragma unroll
        for (int p = 0; p < kTopK; ++p)
            if (rows[p] >= 0)
                reinterpret_cast<uint4*>(ws.dec_act + (size_t)rows[p] * kInter)[ch] = make_uint4(kAbsent, kAbsent, kAbsent, kAbsent);
    }
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.0f;
#pragma unroll
    for (int p = 0; p < kTopK; ++p) {
        if (rows[p] >= 0) {
            const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw[p]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = __bfloat1622float2(h2[j]);
                acc[2 * j] += f.x * wts[p];
                acc[2 * j + 1] += f.y * wts[p];
            }
        }
    }
    uint4 packed;
    __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
    for (int j = 0; j < 4; ++j) o2[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
    reinterpret_cast<uint4*>(out + (size_t)t * kHidden)[ch] = packed;
    if (clocked) ws.ctrl->dec_time[6] = global_timer_ns();
}

}  // namespace

int decode_max_ctas_per_sm()
{
    if (cudaFuncSetAttribute(decode_layer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(DecodeShared)) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, decode_layer_kernel, kDecThreads, sizeof(DecodeShared)) !=
        cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

cudaError_t launch_decode_layer(const DecodeArgs& args, const void* tmap_w1, const void* tmap_w2, const Workspace& ws,
                                int num_ctas, cudaStream_t stream)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(num_ctas);
    cfg.blockDim = dim3(kDecThreads);
    cfg.dynamicSmemBytes = sizeof(DecodeShared);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // set-up under the predecessor's tail
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, decode_layer_kernel, args, *static_cast<const CUtensorMap*>(tmap_w1),
                                             *static_cast<const CUtensorMap*>(tmap_w2), ws);
    if (e != cudaSuccess) return e;
    cfg.gridDim = dim3(kDecCombineParts, args.T);
    cfg.blockDim = dim3(kDecCombineThreads);
    cfg.dynamicSmemBytes = 0;
    return cudaLaunchKernelEx(&cfg, decode_combine_kernel, ws, args.out);
}

}  // namespace moe
