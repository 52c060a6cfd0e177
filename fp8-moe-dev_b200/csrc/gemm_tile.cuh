// Building blocks shared by the grouped-GEMM kernels: tile geometry, the promotion step (raw TMEM block
// product x scale, added into fp32 registers) and the layout of a finished tile in shared memory.
#pragma once
#include <cuda.h>
#include <cuda_fp8.h>

#include "layer.cuh"
#include "ptx.cuh"

namespace moe {

constexpr int kGemmThreads = 384;
constexpr int kTileN = 256;
constexpr int kATileBytes = kTileM * kBlock;   // 16384
constexpr int kBTileBytes = kTileN * kBlock;   // 32768
constexpr int kStageBytes = kATileBytes + kBTileBytes;
constexpr int kTmemCols = 512;
constexpr int kEpilogueWarps = 8;
constexpr int kEpilogueThreads = kEpilogueWarps * 32;

// The finished tile on its way to the epilogue warps: 128 rows x 256 bf16 columns as four panels of
// 64 columns.  A panel is 128 rows of 128 bytes in the 128-byte swizzle (16-byte chunk index XOR
// row mod 8): what a TMA tile store with SWIZZLE_128B reads, and conflict-free both for the
// promotion threads (one row each) and for the epilogue warps (one row per warp).
constexpr int kPanelCols = 64;
constexpr int kPanelBytes = kTileM * kPanelCols * 2;                // 16 KB
constexpr int kTilePanels = kTileN / kPanelCols;                    // 4
constexpr int kTileStageBytes = kTilePanels * kPanelBytes;          // 64 KB

struct TileCoord {
    int e, n, row0, rows;
};

// Where the two weight-block scales of an output tile lie, K block after K block: .lo scales its first 128 columns
// (GEMM1: linear branch), .hi its second (gated branch).  In the handle's copy (repack_weight_scales_kernel) a
// K block's two lie side by side; in the operator's own layout, where both tensors have 2 tiles_n rows per expert,
// they are two rows contiguous in the K block: n and tiles_n + n of GEMM1's tensor, 2n and 2n + 1 of GEMM2's.  A
// warp reads a unit's scales once, ahead of its K loop, so either form serves.
struct ScaleRows {
    const float *lo, *hi;
    int step;
    __device__ __forceinline__ float2 at(int kb) const { return make_float2(__ldg(lo + kb * step), __ldg(hi + kb * step)); }
};
__device__ __forceinline__ ScaleRows weight_scale_rows(const float* base, bool in_place, bool gemm1, int e, int n, int tiles_n,
                                                       int kblocks) {
    ScaleRows r;
    if (in_place) {
        r.lo = base + ((size_t)e * 2 * tiles_n + (gemm1 ? n : 2 * n)) * kblocks;
        r.hi = r.lo + (size_t)(gemm1 ? tiles_n : 1) * kblocks;
        r.step = 1;
    } else {
        r.lo = base + ((size_t)e * tiles_n + n) * kblocks * 2;
        r.hi = r.lo + 1;
        r.step = 2;
    }
    return r;
}

// tcgen05.wait::ld with the destination registers as in/out operands, so that the
// compiler cannot move a use of them above the wait.
__device__ __forceinline__ void tmem_ld_wait2(uint32_t (&a)[32], uint32_t (&b)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                   "+r"(a[8]), "+r"(a[9]), "+r"(a[10]), "+r"(a[11]), "+r"(a[12]), "+r"(a[13]), "+r"(a[14]),
                   "+r"(a[15]), "+r"(a[16]), "+r"(a[17]), "+r"(a[18]), "+r"(a[19]), "+r"(a[20]), "+r"(a[21]),
                   "+r"(a[22]), "+r"(a[23]), "+r"(a[24]), "+r"(a[25]), "+r"(a[26]), "+r"(a[27]), "+r"(a[28]),
                   "+r"(a[29]), "+r"(a[30]), "+r"(a[31]), "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3]),
                   "+r"(b[4]), "+r"(b[5]), "+r"(b[6]), "+r"(b[7]), "+r"(b[8]), "+r"(b[9]), "+r"(b[10]),
                   "+r"(b[11]), "+r"(b[12]), "+r"(b[13]), "+r"(b[14]), "+r"(b[15]), "+r"(b[16]), "+r"(b[17]),
                   "+r"(b[18]), "+r"(b[19]), "+r"(b[20]), "+r"(b[21]), "+r"(b[22]), "+r"(b[23]), "+r"(b[24]),
                   "+r"(b[25]), "+r"(b[26]), "+r"(b[27]), "+r"(b[28]), "+r"(b[29]), "+r"(b[30]), "+r"(b[31])
                 :
                 : "memory");
}

// acc[OFF + j] += raw[j] * s for 32 accumulator columns, by the two-wide fp32 FMA of sm_100: same IEEE result per element and the same FMA-pipe time, but half the issue slots.
// That matters because the MMA-issuing thread shares its scheduler with two of these warps: long
// bursts of scalar FMAs starve it (measured: 728 -> 592 cycles per K block in an isolated
// two-stage pipeline when the promotion uses the packed form).
template <int OFF>
__device__ __forceinline__ void promote32(float (&acc)[128], const uint32_t (&r)[32], float s) {
    const float2 s2 = make_float2(s, s);
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
        const float2 d = __ffma2_rn(make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])), s2,
                                    make_float2(acc[OFF + j], acc[OFF + j + 1]));
        acc[OFF + j] = d.x;
        acc[OFF + j + 1] = d.y;
    }
}

}  // namespace moe
