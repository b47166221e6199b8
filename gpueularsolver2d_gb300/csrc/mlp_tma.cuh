// mlp_tma.cuh -- what the TMA / tcgen05 kernels of the warm-start MLP share
// (descriptors, barriers, tensor-map copies), and the weight gradient of the
// hidden layers with the bias sums.  The forward pass and the data gradient
// are in mlp_chain.cuh.  No reference counterpart.
#pragma once

#include <cuda.h>

#include "mlp_kernels.cuh"

namespace e2d {
namespace mlp {
namespace ws {

constexpr int ND = 256, BM = 128;            // output width, rows per tile
constexpr int KC = 64;                       // K columns per A slice: one 128-byte swizzle row of bf16
constexpr int SLICE_BYTES = BM * KC * 2;     // 16 KB
constexpr int WSLICE_BYTES = ND * KC * 2;    // 32 KB
constexpr int NEPI = 16;                     // epilogue warps: 4 per 32-lane quarter of tensor memory
constexpr int THREADS = 32 * (2 + NEPI);
constexpr uint32_t TMEM_COLS = 512;          // two 256-column FP32 accumulators
constexpr int WAIT_LIMIT = 1 << 22;          // try_wait calls before giving up
constexpr int MAXL = 16;                     // hidden layers

// instruction descriptor: FP32 D, BF16 A and B, both K-major, N = 256, M = 128
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(ND >> 3) << 17) |
                           ((uint32_t)(BM >> 4) << 24);

// Shared-memory matrix descriptor of a K-major operand in the 128-byte swizzle
// layout TMA writes: rows of 128 bytes (64 bf16 of K), 8-row groups 1024 bytes
// apart (SBO), version 1, layout type 2 (128-byte swizzle).  A K = 16 step
// inside the 64-column slice advances the start address by 32 bytes.
__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity) {
    for (int it = 0; it < WAIT_LIMIT; it++) {
        uint32_t done;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                     " selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" :: "r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" :: "r"(bar) : "memory");
}

// 2D tiled TMA load of box (x, y) of the tensor map into shared memory,
// completing on bar.  x is a multiple of 64 elements (128 bytes).
__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
                 :: "r"(dst), "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar) : "memory");
}

// 2D tiled TMA store of a shared-memory box to (x, y) of the tensor map, in
// the calling thread's bulk group.
__device__ __forceinline__ void tma_store(const CUtensorMap *map, uint32_t src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];\n"
                 :: "l"((uint64_t)map), "r"(x), "r"(y), "r"(src) : "memory");
}

__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" :: "r"(bar)
                 : "memory");
}

// ---------------------------------------------------------------------------
// Weight gradient of a 256 x 256 hidden layer, split over the batch:
//   part[split][m][n] = sum over the split's rows b of dZ[b][m] H[b][n]
// (the batch, the reduction index, is the slow index of both operands, so
// both are MN-major).  CTA `split` takes WROWS consecutive rows in 64-row
// chunks: warp 0 loads each chunk of dZ and of H as four 64 x 64 boxes apiece
// (TMA, 128-byte swizzle) into a three-stage ring, warp 1 accumulates the two
// 128-row halves of the 256 x 256 product in tensor memory (all 512
// columns), and eight warps write the FP32 partial.  While the MMAs run, the
// same eight warps sum each column of dZ over the split's rows from the
// staged boxes (thread m: column m), the bias gradient's partial
// bpart[split][m]; a stage is released when its MMAs and these reads are
// done.
constexpr int WROWS = 512;                      // batch rows per split (a multiple of WCH)
constexpr int WCH = 64;                         // rows per chunk
constexpr int WBOX = 64 * WCH * 2;              // one 64 (MN) x 64 (K) box: 8 KB
constexpr int WSTAGE = 8 * WBOX;                // dZ and H boxes of one chunk: 64 KB
constexpr int WNST = 3;
constexpr int WSMEM = WNST * WSTAGE + 1024;
constexpr int WEPI = 8;
constexpr int WTHREADS = 32 * (2 + WEPI);

// MN-major operand in the 128-byte swizzle layout: 64-element (128-byte) rows
// along MN, one per K index; 8-row K groups 1024 bytes apart (SBO), the next
// 64 MN elements one box (8 KB) further (LBO); a K = 16 step advances the
// start by two K groups (2048 bytes).
__device__ __forceinline__ uint64_t desc_sw128_mn(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)(WBOX >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// The partials are written through mapPart: FP32 [splits * 256][64 NH], boxes
// of 32 x 32 with the 128-byte swizzle.  After the last MMA the ring is free
// and each epilogue warp stages its 32 rows there, up to 128 columns at a time
// (four boxes), for TMA stores.  Instruction descriptor: FP32 D, BF16 A and B,
// both MN-major (bits 15 / 16), N = 64 NH, M = 128.
// One launch covers gridDim.y layers: layer l0 + blockIdx.y.
struct WgradMaps {
    CUtensorMap dz[MAXL], h[MAXL], part[MAXL];
    float *bpart[MAXL];
};
template <int NH>
__global__ void __launch_bounds__(WTHREADS, 1)
    k_wgrad_ws(const __grid_constant__ WgradMaps maps, int l0, int M, int rows, int *flag) {
    const int layer = l0 + (int)blockIdx.y;
    const CUtensorMap &mapDz = maps.dz[layer], &mapH = maps.h[layer], &mapPart = maps.part[layer];
    float *bpart = maps.bpart[layer];
    // N = 64 NH columns of H (4 boxes for a 256-wide layer, 1 for the first
    // layer's inputs padded to 64); tensor memory: two M halves of N columns
    constexpr int NCOL = 64 * NH, PASSES = NCOL >= 128 ? NCOL / 128 : 1, PCOLS = NCOL / PASSES;
    constexpr uint32_t TCOLS = 2 * NCOL;
    constexpr uint32_t IDESC_W = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                                 ((uint32_t)(NCOL >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    constexpr uint32_t STAGE_TX = (4 + NH) * WBOX;
    extern __shared__ unsigned char ws_raw[];
    __shared__ __align__(8) uint64_t full[WNST], empty[WNST], tfull, mdone;
    __shared__ uint32_t tmem_sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_u32(ws_raw) + 1023u) & ~1023u;
    const int r0 = blockIdx.x * rows, nch = rows / WCH;
    if (tid == 0) {
        for (int s = 0; s < WNST; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(smem_u32(&full[s])));
            // released by the MMAs' commit and by each column-sum warp
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" :: "r"(smem_u32(&empty[s])), "n"(1 + WEPI));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(smem_u32(&tfull)));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(smem_u32(&mdone)));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     :: "r"(smem_u32(&tmem_sh)), "r"(TCOLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem = tmem_sh;
    if (warp == 0 && lane == 0) {
        // ---- producer: boxes 0..3 dZ columns 64j.., boxes 4..7 H columns 64j.. ----
        bool ok = true;
        int c = 0;
        for (; c < nch && r0 + c * WCH < M; c++) {
            const int st = c % WNST;
            if (!wait(smem_u32(&empty[st]), ((c / WNST) & 1) ^ 1)) { ok = false; break; }
            expect_tx(smem_u32(&full[st]), STAGE_TX);
            const uint32_t dst = base + st * WSTAGE;
            for (int j = 0; j < 4; j++) tma_load(dst + j * WBOX, &mapDz, 64 * j, r0 + c * WCH, smem_u32(&full[st]));
            for (int j = 0; j < NH; j++)
                tma_load(dst + (4 + j) * WBOX, &mapH, 64 * j, r0 + c * WCH, smem_u32(&full[st]));
        }
        if (!ok) atomicExch(flag, 1);
        for (int k = c - WNST > 0 ? c - WNST : 0; k < c; k++) wait(smem_u32(&full[k % WNST]), (k / WNST) & 1);
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issuer: D_h (columns 256 h..) += dZ[:, 128 h..]^T H ----
        bool ok = true;
        for (int c = 0; c < nch && r0 + c * WCH < M && ok; c++) {
            const int st = c % WNST;
            if (!wait(smem_u32(&full[st]), (c / WNST) & 1)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;\n");
            const uint32_t src = base + st * WSTAGE;
#pragma unroll
            for (int kk = 0; kk < WCH / 16; kk++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint64_t ad = desc_sw128_mn(src + (2 * h) * WBOX + kk * 2048);
                    const uint64_t bd = desc_sw128_mn(src + 4 * WBOX + kk * 2048);
                    const uint32_t accumulate = (c > 0 || kk > 0) ? 1u : 0u;
                    asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
                                 " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                                 :: "r"(tmem + (uint32_t)(h * NCOL)), "l"(ad), "l"(bd), "r"(IDESC_W), "r"(accumulate));
                }
            commit(smem_u32(&empty[st]));
        }
        if (ok) commit(smem_u32(&tfull));
        else atomicExch(flag, 1);
        commit(smem_u32(&mdone));
        wait(smem_u32(&mdone), 0);
    } else if (warp >= 2) {
        // ---- column sums of dZ while the MMAs run (thread e: column e) ----
        const int e = tid - 64;
        const int bj = e >> 6, chunk = (e & 63) >> 3, elem = e & 7;
        float bsum = 0.0f;
        int okw = 1;
        for (int c = 0; c < nch && r0 + c * WCH < M; c++) {
            const int st = c % WNST;
            okw = lane == 0 ? (int)wait(smem_u32(&full[st]), (c / WNST) & 1) : 0;
            okw = __shfl_sync(0xffffffffu, okw, 0);
            if (!okw) break;
            // box bj of dZ: row k at 128 k bytes, its 16-byte chunks swizzled by k % 8
            const unsigned char *box = ws_raw + (base - smem_u32(ws_raw)) + st * WSTAGE + bj * WBOX;
#pragma unroll 8
            for (int k = 0; k < WCH; k++)
                bsum += __bfloat162float(*(const bf16 *)(box + k * 128 + ((chunk ^ (k & 7)) << 4) + elem * 2));
            __syncwarp();
            if (lane == 0) arrive(smem_u32(&empty[st]));
        }
        if (okw) bpart[(size_t)blockIdx.x * ND + e] = bsum;
        // the ring is reused for staging below: every column-sum warp has
        // finished reading it (named barrier 1 over the WEPI epilogue warps)
        asm volatile("bar.sync 1, %0;\n" :: "n"(WEPI * 32) : "memory");
        // ---- epilogue: warp -> (32-lane quarter, half of the rows' M-half) ----
        const int quarter = warp & 3, h = (warp - 2) >> 2;
        if (okw) okw = lane == 0 ? (int)wait(smem_u32(&tfull), 0) : 0;
        okw = __shfl_sync(0xffffffffu, okw, 0);
        if (okw) {
            asm volatile("tcgen05.fence::after_thread_sync;\n");
            // the ring is free: every stage has been consumed by the MMAs and
            // the column sums; 16 KB of it per warp
            const uint32_t stg = base + (uint32_t)((warp - 2) * 4 * 4096);
            const int prow = blockIdx.x * ND + h * BM + quarter * 32;
#pragma unroll 1
            for (int pass = 0; pass < PASSES; pass++) {
                if (pass == 1) {
                    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
                    __syncwarp();
                }
#pragma unroll 1
                for (int ch = 0; ch < PCOLS / 16; ch++) {
                    uint32_t v[16];
                    const uint32_t taddr =
                        tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(h * NCOL + pass * PCOLS + ch * 16);
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                        "[%16];\n"
                        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                          "=r"(v[14]), "=r"(v[15])
                        : "r"(taddr));
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                    // box ch / 2 (32 columns), 16-byte units 4 (ch % 2) .. of row lane,
                    // swizzled by lane % 8 (conflict-free per quarter-warp)
                    const uint32_t bx = stg + (uint32_t)((ch >> 1) * 4096 + lane * 128);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const int u = (ch & 1) * 4 + j;
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n"
                                     :: "r"(bx + (uint32_t)((u ^ (lane & 7)) << 4)), "r"(v[4 * j]), "r"(v[4 * j + 1]),
                                        "r"(v[4 * j + 2]), "r"(v[4 * j + 3]) : "memory");
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    for (int j = 0; j < PCOLS / 32; j++)
                        tma_store(&mapPart, stg + j * 4096, pass * PCOLS + j * 32, prow);
                    asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                }
            }
            if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
            __syncwarp();
        } else if (lane == 0) {
            atomicExch(flag, 1);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" :: "r"(tmem), "r"(TCOLS));
}

}  // namespace ws
}  // namespace mlp
}  // namespace e2d
