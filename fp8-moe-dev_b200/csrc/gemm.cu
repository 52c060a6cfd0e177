// The two FP8 block-scaled grouped GEMMs for batches of at most four tokens (split along K), and what both
// GEMM forms need on the host: tensor maps, the pre-laid-out weight scales, the tile-ordered weight copies.
// expert_gemms.cu states the arithmetic and holds the kernel for larger batches.
//
// Such a batch has at most 32 rows and fewer tiles than SMs, so every tile's K range is cut into units and
// all SMs stream weights; units park their partial rows in global scratch and the last one (a ticket) sums
// them in split order and runs the epilogue.  One CTA (384 threads, one per SM, 128 x 256 tile):
//   warp 0      TMA producer: 128x128 B A tile + 256x128 B weight tile per 128-wide K block, ring of four
//               stages, SWIZZLE_128B, one mbarrier pair per stage
//   warp 1      MMA issuer: 4 x tcgen05.mma (M128 N256 K32, e4m3 -> fp32) per K block into one
//               of two 256-column TMEM accumulator stages, overwrite mode on the first
//   warp 2      TMEM allocation / release
//   warps 4-11  promotion (scale and add into fp32 registers), split-K hand-over, epilogue
// Every mbarrier wait is bounded; a wait that runs out sets the CTA's abort flag, all roles unwind, TMEM is
// released and the error is reported through Control::status.
#include <cuda.h>
#include <cuda_fp8.h>

#include "gemm_tile.cuh"

namespace moe {

constexpr int kSplitKMaxRows = 4;    // split-K is used for batches of at most this many tokens
constexpr int kSplitKMaxSplit = 14;  // 56 K blocks / 4

static_assert(kHiddenBlocks / 4 <= kSplitKMaxSplit, "split-K register array too small");

constexpr int kStages = 4;
struct GemmShared {
    uint64_t full[kStages];
    uint64_t empty[kStages];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];
    uint64_t amax_bar[2];
    uint64_t splitk_bar;
    uint32_t tmem_base;
    int abort;
    int splitk_last;
};
struct GemmScratch {
    alignas(16) float splitk_sum[kSplitKMaxRows][256];   // read and written as float4
    float amax[2][2][kTileM];
};
constexpr size_t kGemmCoreBytes = 1024;   // GemmShared, padded
static_assert(sizeof(GemmShared) <= kGemmCoreBytes, "barrier block grew");

constexpr size_t kSplitKSmemBytes = 1024 + (size_t)kStages * kStageBytes + kGemmCoreBytes + sizeof(GemmScratch);
static_assert(kSplitKSmemBytes <= 227 * 1024, "shared memory");

// Tile id -> (expert, n tile, first packed row, valid rows).  Tiles of one expert are
// numbered n-major / m-minor so that CTAs working on neighbouring ids share a weight tile.
__device__ __forceinline__ TileCoord decode_tile(const Workspace& ws, int id, int n_tiles_n) {
    // one 16-byte record per tile: {expert, first tile of the expert, its tile count, its rows}
    const int4 info = ws.tile_info[id / n_tiles_n];
    const int local = id - info.y * n_tiles_n;
    const int n = local / info.z;
    const int j = local - n * info.z;
    const int left = info.w - j * kTileM;
    TileCoord c;
    c.e = info.x;
    c.n = n;
    c.row0 = (info.y + j) * kTileM;
    c.rows = left < kTileM ? left : kTileM;
    return c;
}

// Work units.  Where there are fewer tiles than CTAs every tile is cut into `split` K ranges so that all SMs
// stream weights; the partial tiles are summed by the last unit to finish.
struct UnitPlan {
    int units, split;
};
__device__ __forceinline__ UnitPlan plan_units(int KBLOCKS, int total_tiles, int num_ctas) {
    UnitPlan p;
    p.split = 1;
    if (total_tiles > 0 && total_tiles < num_ctas) {
        // rounds x (K blocks per unit + reduction overhead, about six K blocks' worth), units capped
        // by the scratch slots; ties keep the smaller split
        int best = KBLOCKS;
        for (int s = 2; s <= KBLOCKS / 4 && s <= kSplitKMaxSplit && total_tiles * s <= kSplitKSlots; ++s) {
            const int rounds = (total_tiles * s + num_ctas - 1) / num_ctas;
            const int cost = rounds * ((KBLOCKS + s - 1) / s + 6);
            if (cost < best) { best = cost; p.split = s; }
        }
    }
    p.units = total_tiles * p.split;
    return p;
}
// K-block range [kb0, kb1) of split `s` out of `split`
__device__ __forceinline__ void unit_range(int KBLOCKS, int s, int split, int& kb0, int& kb1) {
    kb0 = (KBLOCKS * s) / split;
    kb1 = (KBLOCKS * (s + 1)) / split;
}

// Split-K: sums the partial rows of one tile over its `split` units into shared memory.  Called by
// the 256 promotion threads of the last unit to finish; thread `et` owns one float4 of the
// (kSplitKMaxRows x 256) block, all splits' loads are in flight together and are added in split
// order.  Kept out of line so that its registers do not weigh on the K loop.
__device__ __noinline__ void splitk_sum_partials(const float* partial, float* sum_smem, int tile_id, int split,
                                                 int rows, int et)
{
    const int r = et >> 6, c4 = et & 63;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows) {
        const float4* src =
            reinterpret_cast<const float4*>(partial + ((size_t)(tile_id * split) * kSplitKMaxRows + r) * 256) + c4;
        float4 v[kSplitKMaxSplit];
#pragma unroll
        for (int sp = 0; sp < kSplitKMaxSplit; ++sp)
            if (sp < split) v[sp] = __ldcg(src + (size_t)sp * (kSplitKMaxRows * 256 / 4));
#pragma unroll
        for (int sp = 0; sp < kSplitKMaxSplit; ++sp)
            if (sp < split) { sum.x += v[sp].x; sum.y += v[sp].y; sum.z += v[sp].z; sum.w += v[sp].w; }
    }
    reinterpret_cast<float4*>(sum_smem)[et] = sum;
}

// Scale load that the compiler cannot sink towards its use: issued (as volatile asm) one
// K block ahead, so that its L2 latency is covered by the whole block's promotion work.
__device__ __forceinline__ float ld_scale_early(const float* p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ float round_bf16(float x) {
    return __bfloat162float(__float2bfloat16_rn(x));
}

// MODE 1: GEMM1 + SwiGLU + requant (K = 7168).  MODE 2: GEMM2 -> bf16 Y (K = 2048).
template <int MODE>
__global__ void __launch_bounds__(kGemmThreads, 1) splitk_gemm_kernel(
    const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, Workspace ws,
    const float* __restrict__ w_scale, int silu_exact)
{
    constexpr int hidden = kHidden, inter = kInter;
    constexpr int kKBlocks = ((MODE == 1) ? hidden : inter) / kBlock;               // 56 / 16
    constexpr int kTilesN = (MODE == 1) ? (inter / kBlock) : (hidden / kTileN);     // 16 / 28

    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    GemmShared* sh = reinterpret_cast<GemmShared*>(smem_raw + (base - raw_addr) + (size_t)kStages * kStageBytes);
    GemmScratch* sc = reinterpret_cast<GemmScratch*>(reinterpret_cast<uint8_t*>(sh) + kGemmCoreBytes);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&sh->full[s]), 1);
            mbar_init(smem_u32(&sh->empty[s]), 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&sh->acc_full[s]), 1);
            mbar_init(smem_u32(&sh->acc_empty[s]), kEpilogueWarps);
            mbar_init(smem_u32(&sh->amax_bar[s]), kEpilogueThreads);
        }
        mbar_init(smem_u32(&sh->splitk_bar), kEpilogueThreads);
        sh->abort = 0;
        fence_mbar_init();
    }
    if (warp == 0 && lane == 0) {
        prefetch_tmap(&tmap_a);
        prefetch_tmap(&tmap_b);
    }
    // Everything above is independent of earlier kernels; from here on their results are read.
    pdl_wait();
    const int total_tiles = ws.num_tiles[0] * kTilesN;
    const UnitPlan plan = plan_units(kKBlocks, total_tiles, (int)gridDim.x);
    if ((int)blockIdx.x >= plan.units) return;  // nothing for this CTA: leave before touching TMEM
    if (warp == 2) {
        tmem_alloc(smem_u32(&sh->tmem_base), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = sh->tmem_base;
    volatile int* abort_flag = &sh->abort;

    if (warp < 4) {
        // register split: 56 per thread for the producer warpgroup, 224 for the two promotion
        // warpgroups (128 * 56 + 256 * 224 <= 64 K registers per SM)
        setmaxnreg_dec<56>();
        if (warp == 0 && lane == 0) {
            // ------------------------------------------------------------ TMA producer
            uint32_t it = 0;
            bool ok = true;
            for (int u = blockIdx.x; ok && u < plan.units; u += gridDim.x) {
                const TileCoord tc = decode_tile(ws, u / plan.split, kTilesN);
                int kb0, kb1;
                unit_range(kKBlocks, u % plan.split, plan.split, kb0, kb1);
                for (int kb = kb0; kb < kb1; ++kb, ++it) {
                    const uint32_t s = it % kStages;
                    const uint32_t ph = (it / kStages) & 1u;
                    if (!mbar_wait(smem_u32(&sh->empty[s]), ph ^ 1u, abort_flag)) { ok = false; break; }
                    const uint32_t full = smem_u32(&sh->full[s]);
                    mbar_expect_tx(full, kStageBytes);
                    const uint32_t a_dst = base + s * kStageBytes;
                    const uint32_t b_dst = a_dst + kATileBytes;
                    tma_load_2d(a_dst, &tmap_a, full, kb * kBlock, tc.row0);
                    if (ws.w_tiled) {
                        // tile-ordered copy of the weights: the operand of (expert, n tile, K block) is one
                        // contiguous 32 KB piece
                        tma_load_2d(b_dst, &tmap_b, full, 0, ((tc.e * kTilesN + tc.n) * kKBlocks + kb) * kTileN);
                    } else if (MODE == 1) {
                        tma_load_3d(b_dst, &tmap_b, full, kb * kBlock, tc.n * kBlock, tc.e);
                        tma_load_3d(b_dst + kBTileBytes / 2, &tmap_b, full, kb * kBlock, inter + tc.n * kBlock, tc.e);
                    } else {
                        tma_load_3d(b_dst, &tmap_b, full, kb * kBlock, tc.n * kTileN, tc.e);
                    }
                }
            }
            if (!ok) {
                // Leave only after this thread's copies in flight have landed (bounded).
                const uint32_t pending = it < (uint32_t)kStages ? it : (uint32_t)kStages;
                for (uint32_t j = 1; j <= pending; ++j) {
                    const uint32_t jt = it - j;
                    const uint32_t s = jt % kStages;
                    const uint32_t ph = (jt / kStages) & 1u;
                    const uint64_t t0 = global_timer_ns();
                    while (!mbar_try_wait(smem_u32(&sh->full[s]), ph)) {
                        if (global_timer_ns() - t0 > kWaitLimitNs / 4) break;
                    }
                }
            }
        } else if (warp == 1 && lane == 0) {
            // ------------------------------------------------------------ MMA issuer
            const uint32_t idesc = make_idesc_e4m3(kTileM, kTileN);
            uint32_t it = 0;
            bool ok = true;
            bool next_full_ready = false;
            for (int u = blockIdx.x; ok && u < plan.units; u += gridDim.x) {
                int kb0, kb1;
                unit_range(kKBlocks, u % plan.split, plan.split, kb0, kb1);
                for (int kb = kb0; kb < kb1; ++kb, ++it) {
                    const uint32_t as = it & 1u;
                    const uint32_t aph = (it >> 1) & 1u;
                    const uint32_t s = it % kStages;
                    const uint32_t ph = (it / kStages) & 1u;
                    // The operand stage is normally long since loaded; its barrier was already
                    // probed while the previous block's MMAs ran (next_full_ready), which keeps
                    // that probe's latency off the release -> issue chain below.
                    if (!next_full_ready && !mbar_wait(smem_u32(&sh->full[s]), ph, abort_flag)) { ok = false; break; }
                    const uint32_t a_addr = base + s * kStageBytes;
                    const uint64_t adesc = make_kmajor_sw128_desc(a_addr);
                    const uint64_t bdesc = make_kmajor_sw128_desc(a_addr + kATileBytes);
                    const uint32_t d = tmem_base + as * kTileN;
                    if (!mbar_wait(smem_u32(&sh->acc_empty[as]), aph ^ 1u, abort_flag)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (int k = 0; k < kBlock / 32; ++k) {
                        // 32 e4m3 = 32 B along K inside the 128 B swizzled row: +2 in 16 B units.
                        umma_f8(d, adesc + 2 * k, bdesc + 2 * k, idesc, k > 0 ? 1u : 0u);
                    }
                    tc_commit(smem_u32(&sh->empty[s]));
                    tc_commit(smem_u32(&sh->acc_full[as]));
                    {
                        const uint32_t nit = it + 1;
                        next_full_ready = mbar_try_wait(smem_u32(&sh->full[nit % kStages]), (nit / kStages) & 1u);
                    }
                }
            }
        }
    } else {
        // ---------------------------------------------------------------- promotion + epilogue
        setmaxnreg_inc<224>();
        const int ew = warp - 4;
        const int h = ew >> 2;       // which 128 of the tile's 256 accumulator columns
        const int q = warp & 3;      // TMEM lane quarter this warp may read
        const int row = q * 32 + lane;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
        // accumulator column of the four 32-column chunks this thread promotes: columns 64h..64h+63 of the
        // tile's first 128-column half and 128+64h..128+64h+63 of its second (GEMM1: linear and gated branch)
        const uint32_t c0 = (uint32_t)(64 * h);
        const uint32_t c1 = c0 + 32;
        const uint32_t c2 = (uint32_t)(128 + 64 * h);
        const uint32_t c3 = c2 + 32;

        uint32_t it = 0;
        uint32_t tile_iter = 0;
        bool ok = true;
        uint32_t splitk_uses = 0;
        for (int u = blockIdx.x; ok && u < plan.units; u += gridDim.x) {
            const int tile_id = u / plan.split;
            const TileCoord tc = decode_tile(ws, tile_id, kTilesN);
            int kb0, kb1;
            unit_range(kKBlocks, u % plan.split, plan.split, kb0, kb1);
            const int grow = tc.row0 + row;
            const float* sfa = ((MODE == 1) ? ws.sfa1 : ws.sfa2) + grow;
            // The tile's weight-block scales for all K blocks: lane l keeps the entries of K blocks l and l + 32,
            // a K block's pair then comes from a shuffle instead of two dependent global loads.
            const ScaleRows sw = weight_scale_rows(w_scale, ws.scales_in_place != 0, MODE == 1, tc.e, tc.n, kTilesN, kKBlocks);
            const float2 sw_a = (lane < kKBlocks) ? sw.at(lane) : make_float2(0.0f, 0.0f);
            const float2 sw_b = (kKBlocks > 32 && lane + 32 < kKBlocks) ? sw.at(lane + 32) : make_float2(0.0f, 0.0f);
            // .x scales the tile's first 128-column block (GEMM1: linear branch), .y its second (gated branch)
            const float mine_a = sw_a.x, other_a = sw_a.y;
            const float mine_b = sw_b.x, other_b = sw_b.y;
            float acc[128];
#pragma unroll
            for (int j = 0; j < 128; ++j) acc[j] = 0.0f;
            const bool warp_has_rows = q * 32 < tc.rows;

            float sa_n = ld_scale_early(sfa + (size_t)kb0 * ws.m_cap);
            for (int kb = kb0; kb < kb1; ++kb, ++it) {
                const float lo_w = __shfl_sync(0xffffffffu, (kKBlocks > 32 && kb >= 32) ? mine_b : mine_a, kb & 31);
                const float hi_w = __shfl_sync(0xffffffffu, (kb >= 32) ? other_b : other_a, kb & 31);
                const float s_lo = sa_n * lo_w;
                const float s_hi = sa_n * hi_w;
                if (kb + 1 < kb1) sa_n = ld_scale_early(sfa + (size_t)(kb + 1) * ws.m_cap);
                const uint32_t as = it & 1u;
                const uint32_t aph = (it >> 1) & 1u;
                ok = mbar_wait(smem_u32(&sh->acc_full[as]), aph, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                if (!warp_has_rows) {
                    // none of this warp's 32 rows is a routed row (short expert tail): nothing to
                    // promote, release the accumulator stage at once
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&sh->acc_empty[as]));
                    continue;
                }
                const uint32_t t = lane_addr + as * kTileN;
                uint32_t r0[32], r1[32];
                tmem_ld_32x32(t + c0, r0);
                tmem_ld_32x32(t + c1, r1);
                tmem_ld_wait2(r0, r1);
                promote32<0>(acc, r0, s_lo);
                tmem_ld_32x32(t + c2, r0);
                promote32<32>(acc, r1, s_lo);
                tmem_ld_32x32(t + c3, r1);
                tmem_ld_wait2(r0, r1);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sh->acc_empty[as]));
                promote32<64>(acc, r0, s_hi);
                promote32<96>(acc, r1, s_hi);
            }
            if (!ok) break;

            const bool valid = row < tc.rows;
            if (plan.split > 1) {
                // Split-K reduction (batches of at most kSplitKMaxRows tokens, so a tile has at most
                // that many routed rows).  Every unit parks its partial rows in global scratch and
                // takes a ticket; the last unit of the tile sums all partials -- one float4 per
                // thread, all splits' loads in flight together, fixed split order -- into shared
                // memory, from where the owning threads pick up their accumulators again.
                float4* mine = reinterpret_cast<float4*>(ws.splitk_partial + ((size_t)u * kSplitKMaxRows + row) * 256 +
                                                         (size_t)h * 128);
                if (valid) {
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        __stcg(mine + j, make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]));
                    __threadfence();
                }
                const uint32_t bar = smem_u32(&sh->splitk_bar);
                mbar_arrive(bar);
                ok = mbar_wait(bar, splitk_uses & 1u, abort_flag);
                ++splitk_uses;
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                if (threadIdx.x == 4 * 32) {
                    const int ticket = atomicAdd(&ws.ctrl->splitk_ticket[tile_id], 1);
                    const int last = (ticket == plan.split - 1) ? 1 : 0;
                    if (last) ws.ctrl->splitk_ticket[tile_id] = 0;
                    sh->splitk_last = last;
                }
                mbar_arrive(bar);
                ok = mbar_wait(bar, splitk_uses & 1u, abort_flag);
                ++splitk_uses;
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                if (!sh->splitk_last) continue;
                __threadfence();
                splitk_sum_partials(ws.splitk_partial, &sc->splitk_sum[0][0], tile_id, plan.split, tc.rows,
                                    (int)threadIdx.x - 4 * 32);
                mbar_arrive(bar);
                ok = mbar_wait(bar, splitk_uses & 1u, abort_flag);
                ++splitk_uses;
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                if (valid) {
                    const float4* src = reinterpret_cast<const float4*>(&sc->splitk_sum[row][h * 128]);
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float4 v = src[j];
                        acc[4 * j] = v.x; acc[4 * j + 1] = v.y; acc[4 * j + 2] = v.z; acc[4 * j + 3] = v.w;
                    }
                }
            }
            if (MODE == 1) {
                // D is rounded to bf16 (the reference materialises it in bf16), then
                // v = silu(x2) * x1 in fp32, absmax over the row's 128-column block.
                float amax = 0.0f;
#pragma unroll
                for (int j = 0; j < 64; ++j) {
                    const float x1 = round_bf16(acc[j]);
                    const float x2 = round_bf16(acc[64 + j]);
                    const float silu = silu_exact ? x2 / (1.0f + __expf(-x2))
                                                  : x2 * (0.5f * (x2 * rsqrtf(fmaf(x2, x2, 4.0f)) + 1.0f));
                    const float v = silu * x1;
                    acc[j] = v;
                    amax = fmaxf(amax, fabsf(v));
                }
                const uint32_t tp = tile_iter & 1u;
                sc->amax[tp][h][row] = amax;
                mbar_arrive(smem_u32(&sh->amax_bar[tp]));
                ok = mbar_wait(smem_u32(&sh->amax_bar[tp]), (tile_iter >> 1) & 1u, abort_flag);
                ++tile_iter;
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                const float maxv = fmaxf(amax, sc->amax[tp][h ^ 1][row]);
                const float scale = (maxv > 0.0f) ? (maxv / 448.0f) : 1.0f;
                const float inv_scale = 1.0f / scale;
                if (valid) {
                    uint4* dst = reinterpret_cast<uint4*>(ws.a2 + (size_t)grow * inter + tc.n * kBlock + 64 * h);
#pragma unroll
                    for (int v8 = 0; v8 < 2; ++v8) {
                        uint4 pk[2];
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            uint32_t wd[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const int j = (v8 * 2 + q) * 16 + i * 4;
                                const uint32_t lo = __nv_cvt_float2_to_fp8x2(
                                    make_float2(acc[j] * inv_scale, acc[j + 1] * inv_scale), __NV_SATFINITE, __NV_E4M3);
                                const uint32_t hi = __nv_cvt_float2_to_fp8x2(
                                    make_float2(acc[j + 2] * inv_scale, acc[j + 3] * inv_scale), __NV_SATFINITE, __NV_E4M3);
                                wd[i] = lo | (hi << 16);
                            }
                            pk[q] = make_uint4(wd[0], wd[1], wd[2], wd[3]);
                        }
                        st_global_32B(dst + 2 * v8, pk[0], pk[1]);
                    }
                    if (h == 0) ws.sfa2[(size_t)tc.n * ws.m_cap + grow] = scale;
                }
            } else {
                if (valid) {
                    // acc[0..63] are columns 64h.., acc[64..127] columns 128 + 64h.. of the tile
                    uint4* dst = reinterpret_cast<uint4*>(ws.y + (size_t)grow * hidden + tc.n * kTileN + 64 * h);
#pragma unroll
                    for (int v8 = 0; v8 < 8; ++v8) {
                        uint4 pk[2];
#pragma unroll
                        for (int q2 = 0; q2 < 2; ++q2) {
                            __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&pk[q2]);
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                h2[i] = __floats2bfloat162_rn(acc[v8 * 16 + q2 * 8 + 2 * i], acc[v8 * 16 + q2 * 8 + 2 * i + 1]);
                        }
                        st_global_32B(dst + (v8 < 4 ? 0 : 8) + 2 * v8, pk[0], pk[1]);
                    }
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
    if (threadIdx.x == 0 && sh->abort != 0) {
        atomicCAS(&ws.ctrl->status, kStatusOk, MODE == 1 ? kStatusGemm1Timeout : kStatusGemm2Timeout);
    }
}

// ---------------------------------------------------------------------------------------
// Weight-scale pre-layout, run once per pair of scale tensors (the handle remembers their
// addresses; not used where the scales are read in place): the promotion wants, per output tile and K block, the two 128x128-block scales the
// tile's 256 accumulator columns use.  In the operator's layout those lie kInterBlocks rows apart
// (GEMM1: [E, 32, 56], linear-branch block n and gated-branch block 16 + n) or in neighbouring
// rows (GEMM2: [E, 56, 16], blocks 2n and 2n + 1); here they become one float2 per (expert, tile,
// K block), the order the promotion walks.  This is the counterpart of the reference's cached
// scale transposes (kernel/moe_fp8.cu:981-994, cached per scale pointer at :3007-3014, 3501-3508).
// ---------------------------------------------------------------------------------------
__global__ void repack_weight_scales_kernel(const float* __restrict__ s1, const float* __restrict__ s2,
                                            float2* __restrict__ p1, float2* __restrict__ p2, int num_experts,
                                            Geometry geo)
{
    const int hb = geo.hidden / kBlock, ib = geo.inter / kBlock;   // 56 / 16 K blocks
    const int kN1 = ib;                    // 16 GEMM1 tiles per expert
    const int kN2 = geo.hidden / kTileN;   // 28 GEMM2 tiles per expert
    const int per1 = kN1 * hb, per2 = kN2 * ib;
    const int total = num_experts * (per1 + per2);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int e = i / (per1 + per2);
        const int r = i - e * (per1 + per2);
        if (r < per1) {
            const int n = r / hb, kb = r - n * hb;
            const float* src = s1 + ((size_t)e * (2 * kN1) + n) * hb + kb;
            p1[(size_t)e * per1 + r] = make_float2(src[0], src[(size_t)kN1 * hb]);
        } else {
            const int r2 = r - per1;
            const int n = r2 / ib, kb = r2 - n * ib;
            const float* src = s2 + ((size_t)e * hb + 2 * n) * ib + kb;
            p2[(size_t)e * per2 + r2] = make_float2(src[0], src[ib]);
        }
    }
}

size_t packed_scale_floats(int mode, int num_experts, const Geometry& geo)
{
    const size_t hb = geo.hidden / kBlock, ib = geo.inter / kBlock;
    return 2 * (size_t)num_experts * (mode == 1 ? ib * hb : (size_t)(geo.hidden / kTileN) * ib);
}

cudaError_t launch_repack_weight_scales(const float* s1, const float* s2, float* p1, float* p2, int num_experts,
                                        const Geometry& geo, cudaStream_t stream)
{
    repack_weight_scales_kernel<<<64, 256, 0, stream>>>(s1, s2, reinterpret_cast<float2*>(p1), reinterpret_cast<float2*>(p2),
                                                        num_experts, geo);
    return cudaGetLastError();
}

// Tile-ordered copy of one weight tensor: for every (expert, n tile, K block) the 256 x 128-byte
// operand the K loop loads becomes one contiguous 32 KB piece (GEMM1: 128 linear rows of the n
// tile, then its 128 gated rows), so that a TMA box reads whole DRAM pages instead of 256 pieces
// of 128 bytes that lie a weight row apart.  One warp per source row, read once front to back.
// The reference keeps such a per-pointer pre-layout of W1 (kernel/moe_fp8.cu:981-994, 3007-3014).
__global__ void __launch_bounds__(256) tile_weights_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst,
                                                           int mode, int num_experts, Geometry geo)
{
    const int k_bytes = mode == 1 ? geo.hidden : geo.inter;
    const int rows = mode == 1 ? 2 * geo.inter : geo.hidden;
    const int kblocks = k_bytes / kBlock;
    const int tiles_n = rows / kTileN;
    const int lane = threadIdx.x & 31;
    const long long total_rows = (long long)num_experts * rows;
    for (long long gr = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); gr < total_rows; gr += (long long)gridDim.x * 8) {
        const int e = (int)(gr / rows);
        const int r = (int)(gr - (long long)e * rows);
        int n, in_tile;
        if (mode == 1) {
            const int half = r >= geo.inter;
            const int rr = r - half * geo.inter;
            n = rr / kBlock;
            in_tile = half * kBlock + (rr - n * kBlock);
        } else {
            n = r / kTileN;
            in_tile = r - n * kTileN;
        }
        const uint4* s4 = reinterpret_cast<const uint4*>(src + (size_t)gr * k_bytes);
        uint8_t* tile0 = dst + ((size_t)(e * tiles_n + n) * kblocks * kTileN + in_tile) * kBlock;
        for (int c = lane; c < k_bytes / 16; c += 32) {
            const int kb = c >> 3;
            *reinterpret_cast<uint4*>(tile0 + (size_t)kb * kTileN * kBlock + (c & 7) * 16) = __ldg(s4 + c);
        }
    }
}

cudaError_t launch_tile_weights(int mode, const void* src, void* dst, int num_experts, const Geometry& geo, int num_sms,
                                cudaStream_t stream)
{
    tile_weights_kernel<<<num_sms * 8, 256, 0, stream>>>(static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst), mode,
                                                         num_experts, geo);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------
// Host side: tensor maps and launch.
// ---------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (fn) return fn;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
        return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(p);
    return fn;
}

// rows x K bytes (K contiguous), optionally batched over experts; box = 128 B x box_rows.
int encode_kmajor_u8_map(void* out_map, const void* base, uint64_t k_bytes, uint64_t rows, uint64_t batch,
                         uint32_t box_rows)
{
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return -1;
    CUtensorMap* m = static_cast<CUtensorMap*>(out_map);
    CUresult r;
    if (batch == 0) {
        const cuuint64_t dims[2] = {k_bytes, rows};
        const cuuint64_t strides[1] = {k_bytes};
        const cuuint32_t box[2] = {(cuuint32_t)kBlock, box_rows};
        const cuuint32_t es[2] = {1, 1};
        r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    } else {
        const cuuint64_t dims[3] = {k_bytes, rows, batch};
        const cuuint64_t strides[2] = {k_bytes, k_bytes * rows};
        const cuuint32_t box[3] = {(cuuint32_t)kBlock, box_rows, 1};
        const cuuint32_t es[3] = {1, 1, 1};
        r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    return r == CUDA_SUCCESS ? 0 : (int)r;
}

// rows x row_bytes viewed as 32-bit words, no swizzle; box = 1 KB of a row x box_rows rows
// (the decode kernel's weight steps).
int encode_rows_1k_map(void* out_map, const void* base, uint64_t row_bytes, uint64_t rows, uint32_t box_rows)
{
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return -1;
    CUtensorMap* m = static_cast<CUtensorMap*>(out_map);
    const cuuint64_t dims[2] = {row_bytes / 4, rows};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {256, box_rows};
    const cuuint32_t es[2] = {1, 1};
    const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(base), dims, strides, box, es,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : (int)r;
}

// bf16 [rows, cols] row-major output; box = 64 columns x 128 rows with the 128-byte swizzle (one panel
// of GEMM2's finished tile).
int encode_out_bf16_map(void* out_map, void* base, uint64_t cols, uint64_t rows)
{
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return -1;
    CUtensorMap* m = static_cast<CUtensorMap*>(out_map);
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kPanelCols, (cuuint32_t)kTileM};
    const cuuint32_t es[2] = {1, 1};
    const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : (int)r;
}

size_t tensor_map_bytes() { return sizeof(CUtensorMap); }

cudaError_t configure_gemm_kernels()
{
    cudaError_t e = cudaFuncSetAttribute(splitk_gemm_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSplitKSmemBytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(splitk_gemm_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSplitKSmemBytes);
    return e;
}

cudaError_t launch_splitk_gemm(int mode, const GemmMaps& maps, const Workspace& ws, const float* w_scale, int silu_exact,
                               int num_ctas, cudaStream_t stream)
{
    const CUtensorMap* ma = static_cast<const CUtensorMap*>(mode == 1 ? maps.a1 : maps.a2);
    const CUtensorMap* mb = static_cast<const CUtensorMap*>(mode == 1 ? maps.w1 : maps.w2);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(num_ctas < 1 ? 1 : num_ctas);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = kSplitKSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (mode == 1) return cudaLaunchKernelEx(&cfg, splitk_gemm_kernel<1>, *ma, *mb, ws, w_scale, silu_exact);
    return cudaLaunchKernelEx(&cfg, splitk_gemm_kernel<2>, *ma, *mb, ws, w_scale, silu_exact);
}

}  // namespace moe
