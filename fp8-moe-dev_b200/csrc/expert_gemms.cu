// Both grouped GEMMs of the layer as ONE persistent kernel of warp-specialised CTAs (batches of more than
// four tokens; gemm.cu holds the split-K form for fewer).
//
//   GEMM1  D[m, 0:4096] = sum_kb (A1[m, kb] . W1[e, :, kb]^T) * (sA1[kb, m] * sW1[e, n/128, kb])
//          epilogue: bf16 rounding of D, SwiGLU (x1 = D[:, n], x2 = D[:, 2048 + n]), per-row 1x128
//          absmax, e4m3 requantisation -> A2, sA2
//   GEMM2  Y[m, 0:7168] = sum_kb (A2[m, kb] . W2[e, :, kb]^T) * (sA2[kb, m] * sW2[e, h/128, kb]) -> bf16
//
// The arithmetic (what is accumulated in fp32, where bf16 / e4m3 rounding happens) follows the reference's
// readable statement of the same math: kernel/moe_fp8.cu:1239-1312 (GEMM1), :1801-1837 (SwiGLU +
// requantisation), :2055-2110 (GEMM2).
//
// Work units.  A unit is one 128-row x 256-column output tile over its whole K range: first all GEMM1 units
// (expert by expert, n-major / m-minor inside an expert, so that CTAs on neighbouring units share a weight
// tile in L2), then all GEMM2 units in the same order.  CTAs draw unit numbers from a counter.  A GEMM2 unit
// needs the GEMM1 units of its 128 rows, which count themselves done per row tile; since units are drawn in
// order, what a CTA waits for has always been drawn by a CTA that is running, so the waits end whatever part
// of the grid is resident.  One kernel instead of two because a batch that only streams weights (up to about
// a thousand tokens per 32 experts) runs at the memory's rate only while every SM has a tile: as two
// launches, the partly filled last round of GEMM1's 40 us tiles, the drain, the second launch and its
// refill left the memory idle for a quarter of the time; here CTAs that find no GEMM1 unit left go on with
// GEMM2 units, and the last units to be drawn are the short ones.
//
// Roles (384 threads, one CTA per SM):
//   warp 0      producer: draws units, waits for a GEMM2 unit's rows (its first weight blocks are requested
//               before that), publishes the unit to the other roles through a four-slot queue, and loads per
//               128-wide K block 128 x 128 B of activations and 256 x 128 B of weights by TMA (SWIZZLE_128B)
//               into a ring of three stages (four with 64-row activation boxes)
//   warp 1      MMA issuer: 4 x tcgen05.mma (M128 N256 K32, e4m3 -> fp32) per K block into one of two
//               256-column TMEM accumulator stages, overwriting on the first
//   warps 2-3   tile epilogue, one unit behind (warp 2 also owns the TMEM allocation)
//   warps 4-11  promotion: tcgen05.ld of the raw block product, times row scale x weight-block scale, added
//               into fp32 registers (arbitrary fp32 scales rule the block-scaled MMA kinds out); a thread
//               owns one row and 128 of the 256 columns.  At the end of a unit's K loop they hand a bf16 tile
//               over in shared memory and go on with the next unit
// Host-resident calls whose output is written in place give a few CTAs another role (see zero_empty_rows).
// Every wait is bounded; one that runs out sets the CTA's abort flag, all roles unwind, TMEM is released and
// the failure is reported through Control::status.
#include "gemm_tile.cuh"

namespace moe {

namespace {

constexpr int kUnitSlots = 4;
constexpr int kMaxStages = 4;
struct UnitDesc {
    int mode;         // 1 GEMM1, 2 GEMM2, 0 no more work
    int e, n;         // local expert, n tile
    int row0, rows;   // first packed row of the 128-row tile, its valid rows
};
struct FusedShared {
    uint64_t full[kMaxStages];
    uint64_t empty[kMaxStages];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];
    uint64_t tile_full;                // the bf16 tile in shared memory is complete (8 promotion warps arrive)
    uint64_t tile_empty;               // the two epilogue warps are done with it
    uint64_t unit_full[kUnitSlots];    // a unit has been published
    uint64_t unit_empty[kUnitSlots];   // issuer, two epilogue warps and eight promotion warps have read it
    alignas(16) int4 unit_a[kUnitSlots];   // {mode | e << 8, n, row0, rows}
    uint32_t tmem_base;
    int abort;
};
constexpr int kUnitReaders = 1 + 2 + kEpilogueWarps;
constexpr size_t kCoreBytes = 1024;   // FusedShared, padded: the panels want 1 KB alignment
static_assert(sizeof(FusedShared) <= kCoreBytes, "barrier block grew");

// Batches of at most 64 tokens: an expert has at most 64 rows, so the activation box is 64 rows high (8 KB instead
// of 16 KB per stage; the MMAs still multiply 128 rows, the upper 64 read whatever follows and are never stored)
// and the room goes to a fourth operand stage: 128 KB instead of 96 KB of weights in flight per SM.
template <bool SMALLA> __host__ __device__ constexpr int ring_stages() { return SMALLA ? 4 : 3; }
template <bool SMALLA> __host__ __device__ constexpr int a_bytes() { return SMALLA ? kATileBytes / 2 : kATileBytes; }
template <bool SMALLA> constexpr size_t smem_bytes() {
    return 1024 + (size_t)ring_stages<SMALLA>() * (a_bytes<SMALLA>() + kBTileBytes) + kCoreBytes + kTileStageBytes;
}
static_assert(smem_bytes<false>() <= 227 * 1024 && smem_bytes<true>() <= 227 * 1024, "shared memory");

__device__ __forceinline__ uint32_t ld_acquire_gpu_u32(const unsigned* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

// Row scale of the next K block: volatile, so that the compiler cannot sink it towards its use.  A plain
// (coherent) load: GEMM2's scales are written by this very kernel.
__device__ __forceinline__ float ld_scale(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}

// Unit number -> tile.  `info` is the record of the unit's row tile: {expert, first tile of the expert, its
// tile count, its rows}.
__device__ __forceinline__ UnitDesc unit_from_record(const int4& info, int local, int mode) {
    UnitDesc d;
    d.mode = mode;
    d.e = info.x;
    d.n = local / info.z;
    const int j = local - d.n * info.z;
    const int left = info.w - j * kTileM;
    d.row0 = (info.y + j) * kTileM;
    d.rows = left < kTileM ? left : kTileM;
    return d;
}

// A reader's view of the unit queue: waits for the next unit and releases its slot.  Whole warps call it
// together (ONE = false) or a single thread does (ONE = true).
template <bool ONE>
__device__ __forceinline__ bool next_unit(FusedShared* sh, uint32_t ui, volatile int* abort_flag, UnitDesc& d) {
    const uint32_t slot = ui % kUnitSlots;
    bool ok = mbar_wait(smem_u32(&sh->unit_full[slot]), (ui / kUnitSlots) & 1u, abort_flag);
    if (!ONE) ok = __all_sync(0xffffffffu, ok);
    if (!ok) return false;
    const int4 a = sh->unit_a[slot];
    d.mode = a.x & 0xff;
    d.e = a.x >> 8;
    d.n = a.y;
    d.row0 = a.z;
    d.rows = a.w;
    if (!ONE) __syncwarp();
    if (ONE || (threadIdx.x & 31) == 0) mbar_arrive(smem_u32(&sh->unit_empty[slot]));
    return d.mode != 0;
}

// Output rows of the tokens that have no expert here (most of them where a GPU holds one shard of eight), written to
// pinned host memory while the other CTAs' GEMMs run.  Behind the permute: beside it, its read requests would queue
// behind these writes on their way out (host call on 32 experts, beside / behind: T=512 369 / 337 us, T=1024 520 /
// 474).  Bound by PCIe, which few CTAs of plain stores fill (52 GB/s; cudaMemcpyAsync 56.7) if they do not share an SM:
// as CTAs of this launch each has its own.  A warp per row.
__device__ __forceinline__ void zero_empty_rows(const Workspace& ws, const EmptyRows& rows) {
    const int lane = threadIdx.x & 31, warps = rows.ctas * (kGemmThreads / 32);
    const bool none = ws.num_tiles[0] == 0;
    const int vecs = ws.geo.hidden * 2 / 16;
    for (int t = (int)blockIdx.x * (kGemmThreads / 32) + (int)(threadIdx.x >> 5); t < rows.T; t += warps) {
        if (!none && ws.pair_count[t] != 0) continue;
        uint4* row = reinterpret_cast<uint4*>(rows.out) + (size_t)t * vecs;
        for (int i = lane; i < vecs; i += 32) row[i] = make_uint4(0u, 0u, 0u, 0u);
    }
}

}  // namespace

// GENERIC takes hidden / intermediate from Workspace::geo (hidden a multiple of 256, intermediate of 128, at
// most 64 K blocks each) instead of the reference's 7168 / 2048.  SMALLA: 64-row activation boxes, see above.
// `phases`: 3 = both GEMMs; 1 / 2 = only the GEMM1 / GEMM2 units, for callers that time or cut the chain
// between the two.
template <bool GENERIC, bool SMALLA>
__global__ void __launch_bounds__(kGemmThreads, 1) expert_gemms_kernel(
    const __grid_constant__ CUtensorMap tmap_a1, const __grid_constant__ CUtensorMap tmap_w1,
    const __grid_constant__ CUtensorMap tmap_a2, const __grid_constant__ CUtensorMap tmap_w2,
    const __grid_constant__ CUtensorMap tmap_y, Workspace ws, const float* __restrict__ w1_scale,
    const float* __restrict__ w2_scale, int silu_exact, int phases, EmptyRows empty_rows)
{
    static_assert(!(SMALLA && GENERIC), "the 64-row activation box is a variant of the reference's geometry");
    const int hidden = GENERIC ? ws.geo.hidden : kHidden;
    const int inter = GENERIC ? ws.geo.inter : kInter;
    const int kb_gemm1 = hidden / kBlock, kb_gemm2 = inter / kBlock;        // 56, 16 K blocks
    const int tiles_n1 = inter / kBlock, tiles_n2 = hidden / kTileN;        // 16, 28 column tiles
    constexpr int kStages = ring_stages<SMALLA>();
    constexpr int kABytes = a_bytes<SMALLA>();
    constexpr int kStageSize = kABytes + kBTileBytes;

    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    FusedShared* sh = reinterpret_cast<FusedShared*>(smem_raw + (base - raw_addr) + (size_t)kStages * kStageSize);
    uint8_t* tile_stage = reinterpret_cast<uint8_t*>(sh) + kCoreBytes;   // the bf16 tile (64 KB), 1 KB aligned

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    pdl_launch_dependents();
    if ((int)blockIdx.x < empty_rows.ctas) {   // whole CTAs, before any barrier or TMEM is set up
        pdl_wait();
        zero_empty_rows(ws, empty_rows);
        return;
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&sh->full[s]), 1);
            mbar_init(smem_u32(&sh->empty[s]), 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&sh->acc_full[s]), 1);
            mbar_init(smem_u32(&sh->acc_empty[s]), kEpilogueWarps);
        }
        for (int s = 0; s < kUnitSlots; ++s) {
            mbar_init(smem_u32(&sh->unit_full[s]), 1);
            mbar_init(smem_u32(&sh->unit_empty[s]), kUnitReaders);
        }
        mbar_init(smem_u32(&sh->tile_full), kEpilogueWarps);
        mbar_init(smem_u32(&sh->tile_empty), 2);
        sh->abort = 0;
        fence_mbar_init();
        prefetch_tmap(&tmap_a1);
        prefetch_tmap(&tmap_w1);
        prefetch_tmap(&tmap_a2);
        prefetch_tmap(&tmap_w2);
        prefetch_tmap(&tmap_y);
    }
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
        // register split: 56 per thread for this warpgroup, 224 for the two promotion warpgroups
        // (128 * 56 + 256 * 224 <= 64 K registers per SM)
        setmaxnreg_dec<56>();
        if (warp == 0 && lane == 0) {
            // ------------------------------------------------------------ producer
            // The kernel in front of this one in the chain (permute, or the GEMM1 half) triggers the launch only
            // once the routing kernel's results are complete, so units can be drawn and looked up and the first
            // weights requested while it still runs; its own results are read after pdl_wait().
            int* ticket = &ws.ctrl->unit_ticket[phases == 2 ? 1 : 0];
            const int row_tiles = __ldcg(ws.num_tiles);
            const int first_ticket = atomicAdd(ticket, 1);
            const int units1 = row_tiles * tiles_n1, units_all = units1 + row_tiles * tiles_n2;
            const int unit_begin = phases == 2 ? units1 : 0, unit_end = phases == 1 ? units1 : units_all;
            const unsigned done_count = 2u * (unsigned)tiles_n1;   // both epilogue warps of every GEMM1 unit of the row tile
            uint32_t it = 0, ui = 0;
            bool ok = true;
            auto record_of = [&](int id) {
                return id < units1 ? __ldcg(ws.tile_info + id / tiles_n1) : __ldcg(ws.tile_info + (id - units1) / tiles_n2);
            };
            auto desc_of = [&](const int4& info, int id) {
                return id < units1 ? unit_from_record(info, id - info.y * tiles_n1, 1)
                                   : unit_from_record(info, id - units1 - info.y * tiles_n2, 2);
            };
            auto publish = [&](const UnitDesc& d) -> bool {
                const uint32_t slot = ui % kUnitSlots;
                if (!mbar_wait(smem_u32(&sh->unit_empty[slot]), ((ui / kUnitSlots) & 1u) ^ 1u, abort_flag)) return false;
                sh->unit_a[slot] = make_int4(d.mode | (d.e << 8), d.n, d.row0, d.rows);
                mbar_arrive(smem_u32(&sh->unit_full[slot]));
                ++ui;
                return true;
            };
            int id = unit_begin + first_ticket;
            UnitDesc d;
            d.mode = 0;
            if (id < unit_end) d = desc_of(record_of(id), id);
            bool rows_ready = phases == 2;   // an earlier launch finished all GEMM1 units
            bool first = true;
            while (ok && id < unit_end) {
                const bool g1 = d.mode == 1;
                const CUtensorMap* map_a = g1 ? &tmap_a1 : &tmap_a2;
                const CUtensorMap* map_w = g1 ? &tmap_w1 : &tmap_w2;
                const int kblocks = g1 ? kb_gemm1 : kb_gemm2;
                // arms K block kb's stage and requests its weights
                auto load_weights = [&](int kb) {
                    const uint32_t s = (it + kb) % kStages;
                    const uint32_t full = smem_u32(&sh->full[s]);
                    mbar_expect_tx(full, kStageSize);
                    const uint32_t b_dst = base + s * kStageSize + kABytes;
                    if (ws.w_tiled) {
                        // tile-ordered copy of the weights: the operand of (expert, n tile, K block) is one
                        // contiguous 32 KB piece
                        tma_load_2d(b_dst, map_w, full, 0, ((d.e * (g1 ? tiles_n1 : tiles_n2) + d.n) * kblocks + kb) * kTileN);
                    } else if (g1) {
                        tma_load_3d(b_dst, map_w, full, kb * kBlock, d.n * kBlock, d.e);
                        tma_load_3d(b_dst + kBTileBytes / 2, map_w, full, kb * kBlock, inter + d.n * kBlock, d.e);
                    } else {
                        tma_load_3d(b_dst, map_w, full, kb * kBlock, d.n * kTileN, d.e);
                    }
                };
                int pre = 0;   // K blocks whose weights have been requested ahead of the rows
                const int lim = kblocks < kStages ? kblocks : kStages;
                if (first) {
                    while (pre < lim) load_weights(pre++);
                    pdl_wait();
                    first = false;
                }
                if (!g1) {
                    if (!rows_ready) {
                        const unsigned* done = ws.tile_done + d.row0 / kTileM;
                        const uint64_t t0 = global_timer_ns();
                        while (ld_acquire_gpu_u32(done) < done_count) {
                            if (pre < lim) {
                                const uint32_t j = it + pre;
                                if (mbar_try_wait(smem_u32(&sh->empty[j % kStages]), ((j / kStages) & 1u) ^ 1u)) load_weights(pre++);
                            }
                            if (*abort_flag != 0 || global_timer_ns() - t0 > kWaitLimitNs) { *abort_flag = 1; ok = false; break; }
                        }
                        if (!ok) { it += pre; break; }
                    }
                    fence_proxy_async_global();   // the rows were written through the generic proxy, TMA reads them
                }
                if (!publish(d)) { ok = false; it += pre; break; }
                // The next unit is drawn and looked up while this one loads: each step below is a round trip
                // to L2 that the ring's loads in flight cover.
                const int next_id = unit_begin + atomicAdd(ticket, 1);
                int4 next_info = make_int4(0, 0, 1, 0);
                UnitDesc nd;
                nd.mode = 0;
                bool next_ready = phases == 2;
                for (int kb = 0; kb < kblocks; ++kb) {
                    const uint32_t j = it + kb, s = j % kStages;
                    if (kb >= pre) {
                        if (!mbar_wait(smem_u32(&sh->empty[s]), ((j / kStages) & 1u) ^ 1u, abort_flag)) { ok = false; it += kb > pre ? kb : pre; break; }
                        load_weights(kb);
                    }
                    tma_load_2d(base + s * kStageSize, map_a, smem_u32(&sh->full[s]), kb * kBlock, d.row0);
                    const bool last = kb == kblocks - 1;
                    if ((kb == 1 || (last && kb < 1)) && next_id < unit_end) next_info = record_of(next_id);
                    if ((kb == 2 || (last && kb < 2)) && next_id < unit_end) nd = desc_of(next_info, next_id);
                    if (last && nd.mode == 2 && !next_ready)
                        next_ready = ld_acquire_gpu_u32(ws.tile_done + nd.row0 / kTileM) >= done_count;
                }
                if (!ok) break;
                it += kblocks;
                id = next_id;
                d = nd;
                rows_ready = next_ready;
            }
            if (ok) {
                UnitDesc none;
                none.mode = none.e = none.n = none.row0 = none.rows = 0;
                ok = publish(none);
            }
            if (!ok) {
                // Leave only after this thread's copies in flight have landed (bounded).
                const uint32_t pending = it < (uint32_t)kStages ? it : (uint32_t)kStages;
                for (uint32_t j = 1; j <= pending; ++j) {
                    const uint32_t jt = it - j;
                    const uint64_t t0 = global_timer_ns();
                    while (!mbar_try_wait(smem_u32(&sh->full[jt % kStages]), (jt / kStages) & 1u)) {
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
            UnitDesc d;
            for (uint32_t ui = 0; ok && next_unit<true>(sh, ui, abort_flag, d); ++ui) {
                const int kblocks = d.mode == 1 ? kb_gemm1 : kb_gemm2;
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const uint32_t as = it & 1u;
                    const uint32_t aph = (it >> 1) & 1u;
                    const uint32_t s = it % kStages;
                    const uint32_t ph = (it / kStages) & 1u;
                    // The operand stage is normally long since loaded; its barrier was already
                    // probed while the previous block's MMAs ran (next_full_ready), which keeps
                    // that probe's latency off the release -> issue chain below.
                    if (!next_full_ready && !mbar_wait(smem_u32(&sh->full[s]), ph, abort_flag)) { ok = false; break; }
                    const uint32_t a_addr = base + s * kStageSize;
                    const uint64_t adesc = make_kmajor_sw128_desc(a_addr);
                    const uint64_t bdesc = make_kmajor_sw128_desc(a_addr + kABytes);
                    const uint32_t acc = tmem_base + as * kTileN;
                    if (!mbar_wait(smem_u32(&sh->acc_empty[as]), aph ^ 1u, abort_flag)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (int k = 0; k < kBlock / 32; ++k) {
                        // 32 e4m3 = 32 B along K inside the 128 B swizzled row: +2 in 16 B units.
                        umma_f8(acc, adesc + 2 * k, bdesc + 2 * k, idesc, k > 0 ? 1u : 0u);
                    }
                    tc_commit(smem_u32(&sh->empty[s]));
                    tc_commit(smem_u32(&sh->acc_full[as]));
                    {
                        const uint32_t nit = it + 1;
                        next_full_ready = mbar_try_wait(smem_u32(&sh->full[nit % kStages]), (nit / kStages) & 1u);
                    }
                }
            }
        } else if (warp >= 2) {
            // ------------------------------------------------------------ tile epilogue
            // Runs one unit behind the promotion warps, while they are in the next unit's K loop.
            const int ew = warp - 2;
            bool ok = true;
            UnitDesc d;
            for (uint32_t ui = 0; next_unit<false>(sh, ui, abort_flag, d); ++ui) {
                ok = mbar_wait(smem_u32(&sh->tile_full), ui & 1u, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                if (d.mode == 2) {
                    // Y: four 128-row x 64-column tile stores, two per warp.  Rows past the tile's valid rows
                    // land in the expert's padding, which nobody reads.
                    if (lane == 0) {
#pragma unroll
                        for (int p = 0; p < kTilePanels / 2; ++p)
                            tma_store_2d(&tmap_y, smem_u32(tile_stage + (2 * ew + p) * kPanelBytes),
                                         d.n * kTileN + (2 * ew + p) * kPanelCols, d.row0);
                        bulk_commit_group();
                        bulk_wait_group_read<0>();   // the panels have been read: they may be overwritten
                        mbar_arrive(smem_u32(&sh->tile_empty));
                    }
                    __syncwarp();
                } else {
                    // GEMM1: D was rounded to bf16 on its way here (the reference materialises it in
                    // bf16).  A warp takes four rows per pass, eight lanes each: a lane owns SwiGLU columns
                    // 16*l8 .. 16*l8+15 of the tile's 128-column block, x1 from panels 0-1 (linear branch),
                    // x2 from panels 2-3 (gated branch); v = silu(x2) * x1 in fp32, row absmax by three
                    // shuffles, scale = amax / 448 (1 for an all-zero block), e4m3 codes -> one 16-byte
                    // store per lane, 128 coalesced bytes per row.  Latency-bound: one row per pass and 32
                    // lanes took 20 us for a full tile (five shuffles and a division per row in one chain),
                    // time that the GEMM2 tiles of the expert wait for behind the last GEMM1 tile.
                    const int r_begin = ew * (kTileM / 2);
                    const int r_end = d.rows < (ew + 1) * (kTileM / 2) ? d.rows : (ew + 1) * (kTileM / 2);
                    const int l8 = lane & 7;
                    const uint32_t pan = (uint32_t)(l8 >> 2) * kPanelBytes;
                    // lanes 4-7 read their two 16-byte chunks in the other order: panels 0 and 1 lie on the
                    // same banks, so a quarter warp (one row) then touches all eight chunks of a row
                    const uint32_t c0 = 2u * (uint32_t)(l8 & 3) + (uint32_t)(l8 >> 2), c1 = c0 ^ 1u;
                    const bool swapped = l8 >= 4;
                    for (int r0 = r_begin; r0 < r_end; r0 += 4) {
                        const int r = r0 + (lane >> 3);   // < 128: rows past r_end hold stale data and are not stored
                        const uint8_t* src = tile_stage + pan + r * 128;
                        const uint32_t o0 = (c0 ^ (uint32_t)(r & 7)) << 4, o1 = (c1 ^ (uint32_t)(r & 7)) << 4;
                        float v[16];
                        float amax = 0.0f;
#pragma unroll
                        for (int hf = 0; hf < 2; ++hf) {
                            const uint4 l1 = *reinterpret_cast<const uint4*>(src + (hf ? o1 : o0));
                            const uint4 l2 = *reinterpret_cast<const uint4*>(src + 2 * kPanelBytes + (hf ? o1 : o0));
                            const uint32_t w1[4] = {l1.x, l1.y, l1.z, l1.w}, w2[4] = {l2.x, l2.y, l2.z, l2.w};
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                const uint32_t b1 = w1[j >> 1], b2 = w2[j >> 1];
                                const float x1 = __uint_as_float((j & 1) ? (b1 & 0xffff0000u) : (b1 << 16));
                                const float x2 = __uint_as_float((j & 1) ? (b2 & 0xffff0000u) : (b2 << 16));
                                const float silu = silu_exact ? x2 / (1.0f + __expf(-x2))
                                                              : x2 * (0.5f * (x2 * rsqrtf(fmaf(x2, x2, 4.0f)) + 1.0f));
                                v[8 * hf + j] = silu * x1;
                                amax = fmaxf(amax, fabsf(v[8 * hf + j]));
                            }
                        }
#pragma unroll
                        for (int off = 4; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
                        const float scale = (amax > 0.0f) ? (amax / 448.0f) : 1.0f;
                        const float inv_scale = 1.0f / scale;
                        uint32_t q[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            q[i] = (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(v[4 * i] * inv_scale, v[4 * i + 1] * inv_scale),
                                                                      __NV_SATFINITE, __NV_E4M3) |
                                   ((uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(v[4 * i + 2] * inv_scale, v[4 * i + 3] * inv_scale),
                                                                       __NV_SATFINITE, __NV_E4M3) << 16);
                        if (r < r_end) {
                            const int grow = d.row0 + r;
                            const uint4 out = swapped ? make_uint4(q[2], q[3], q[0], q[1]) : make_uint4(q[0], q[1], q[2], q[3]);
                            *reinterpret_cast<uint4*>(ws.a2 + (size_t)grow * inter + d.n * kBlock + 16 * l8) = out;
                            if (l8 == 0) ws.sfa2[(size_t)d.n * ws.m_cap + grow] = scale;
                        }
                    }
                    // The rows' codes and scales are read by TMA and by the promotion warps of whichever CTAs draw
                    // the GEMM2 units: make them visible (to the async proxy too) before counting this unit done.
                    fence_proxy_async_global();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(smem_u32(&sh->tile_empty));
                        __threadfence();
                        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ws.tile_done + d.row0 / kTileM) : "memory");
                    }
                }
            }
            if (lane == 0) bulk_wait_group<0>();   // stores performed before the CTA leaves
        }
    } else {
        // ---------------------------------------------------------------- promotion
        setmaxnreg_inc<224>();
        pdl_wait();   // the packed rows' scales
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
        bool ok = true;
        UnitDesc d;
        for (uint32_t ui = 0; next_unit<false>(sh, ui, abort_flag, d); ++ui) {
            const bool g1 = d.mode == 1;
            const int kblocks = g1 ? kb_gemm1 : kb_gemm2;
            const float* sfa = (g1 ? ws.sfa1 : ws.sfa2) + d.row0 + row;
            // The tile's weight-block scales for all K blocks: lane l keeps the entries of K blocks l and l + 32,
            // a K block's pair then comes from a shuffle instead of two dependent global loads.
            const ScaleRows sw = weight_scale_rows(g1 ? w1_scale : w2_scale, ws.scales_in_place != 0, g1, d.e, d.n,
                                                   g1 ? tiles_n1 : tiles_n2, kblocks);
            const float2 sw_a = (lane < kblocks) ? sw.at(lane) : make_float2(0.0f, 0.0f);
            const float2 sw_b = (lane + 32 < kblocks) ? sw.at(lane + 32) : make_float2(0.0f, 0.0f);
            // .x scales the tile's first 128-column block (GEMM1: linear branch), .y its second (gated branch)
            float acc[128];
#pragma unroll
            for (int j = 0; j < 128; ++j) acc[j] = 0.0f;
            const bool warp_has_rows = q * 32 < d.rows;

            float sa_n = ld_scale(sfa);
            for (int kb = 0; kb < kblocks; ++kb, ++it) {
                const float lo_w = __shfl_sync(0xffffffffu, kb >= 32 ? sw_b.x : sw_a.x, kb & 31);
                const float hi_w = __shfl_sync(0xffffffffu, kb >= 32 ? sw_b.y : sw_a.y, kb & 31);
                const float s_lo = sa_n * lo_w;
                const float s_hi = sa_n * hi_w;
                if (kb + 1 < kblocks) sa_n = ld_scale(sfa + (size_t)(kb + 1) * ws.m_cap);
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

            // Hand the tile to the epilogue warps: accumulators rounded to bf16 (what both the GEMM1 and the
            // GEMM2 result are rounded to anyway) into the shared-memory panels, a thread's first 64 columns
            // into panel h, its other 64 into panel 2 + h.  The panels were released a whole K loop ago, so
            // the wait below does not block in practice.
            if (ui > 0) {
                ok = mbar_wait(smem_u32(&sh->tile_empty), (ui - 1) & 1u, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
            }
            if (warp_has_rows) {
                uint8_t* ra = tile_stage + h * kPanelBytes + row * 128;
                uint8_t* rb = tile_stage + (2 + h) * kPanelBytes + row * 128;
                const uint32_t swz = (uint32_t)(row & 7);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    uint4 pk;
                    __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
                    for (int i = 0; i < 4; ++i) h2[i] = __floats2bfloat162_rn(acc[8 * c + 2 * i], acc[8 * c + 2 * i + 1]);
                    *reinterpret_cast<uint4*>(ra + (((uint32_t)c ^ swz) << 4)) = pk;
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        h2[i] = __floats2bfloat162_rn(acc[64 + 8 * c + 2 * i], acc[64 + 8 * c + 2 * i + 1]);
                    *reinterpret_cast<uint4*>(rb + (((uint32_t)c ^ swz) << 4)) = pk;
                }
                if (!g1) fence_proxy_async_smem();   // the TMA stores read these writes
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&sh->tile_full));
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
    if (threadIdx.x == 0 && sh->abort != 0) atomicCAS(&ws.ctrl->status, kStatusOk, kStatusGemm1Timeout);
}

template <bool GENERIC, bool SMALLA>
static cudaError_t configure_one()
{
    return cudaFuncSetAttribute(expert_gemms_kernel<GENERIC, SMALLA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem_bytes<SMALLA>());
}

cudaError_t configure_expert_gemms()
{
    cudaError_t e = configure_one<false, false>();
    if (e == cudaSuccess) e = configure_one<true, false>();
    if (e == cudaSuccess) e = configure_one<false, true>();
    return e;
}

// `small_a` (reference geometry, at most 64 tokens): maps.a1 / maps.a2 are the 64-row views of the packed rows.
cudaError_t launch_expert_gemms(const GemmMaps& maps, const Workspace& ws, const float* w1_scale, const float* w2_scale,
                                int silu_exact, int phases, int num_ctas, int small_a, const EmptyRows& empty_rows,
                                cudaStream_t stream)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(num_ctas < 1 ? 1 : num_ctas);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = small_a ? smem_bytes<true>() : smem_bytes<false>();
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto map = [](const void* p) { return *static_cast<const CUtensorMap*>(p); };
    auto go = [&](auto* kernel) {
        return cudaLaunchKernelEx(&cfg, kernel, map(maps.a1), map(maps.w1), map(maps.a2), map(maps.w2), map(maps.y), ws,
                                  w1_scale, w2_scale, silu_exact, phases, empty_rows);
    };
    if (!ws.geo.is_reference()) return go(expert_gemms_kernel<true, false>);
    return small_a ? go(expert_gemms_kernel<false, true>) : go(expert_gemms_kernel<false, false>);
}

}  // namespace moe
