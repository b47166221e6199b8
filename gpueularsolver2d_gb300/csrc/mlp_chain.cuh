// mlp_chain.cuh -- the hidden layers of the warm-start MLP as one launch per
// direction: the forward pass (bias + GELU) and the data gradient (GELU') of
// every layer, a batch tile staying on its SM from the first layer to the
// last.  No reference counterpart.
//
// A 128-row tile is carried through the layers in shared memory: the epilogue
// of a step writes the next step's A operand in place.  One CTA per SM walks its
// tiles, two at a time when there are more tiles than SMs: one's MMAs run while
// the other's epilogue does.
//   warp 0  (one thread) streams the operands through a ring of 32 KB slots by
//           TMA: the tile's own input for the first step, then each step's
//           weights in four slices of 64 columns of K; three slots with two
//           tiles in shared memory, five with one;
//   warp 1  (one thread) issues tcgen05.mma (kind::f16, M = 128, N = 256, K =
//           16, FP32 accumulate) into one of two 256-column accumulators;
//   warps 2-17 take 32 rows x 64 columns each from tensor memory, apply the
//           epilogue, write the bf16 result over their own part of the A
//           operand (128-byte swizzle, the layout both the next MMA and the TMA
//           store read), store it, and release it to the MMA thread.  gelu'(z)
//           is written (forward) or read ahead (data gradient) from registers, 32
//           bytes per lane, so that it takes no shared memory; between two
//           layers of the chain it is kept in the order of the accesses (a
//           warp's 1 KB together: stored row by row, 32 sectors to a store, a
//           step took 2 us longer), and row-major for the last layer, where the
//           output layer reads it.
// What one launch per layer cost: start-up (barriers, tensor memory, 128 KB of
// weights, an empty pipeline) of about 6 us, and a round trip of the tile
// through L2.  The accumulation order and the roundings are those of the
// per-tile kernel's layers.
// Every wait is bounded: a timed-out thread sets *flag and leaves its loop;
// the producer then waits (bounded) for the copies it issued, the MMA thread
// for the MMAs it issued, and the tensor memory is freed on every path.
#pragma once

#include "mlp_tma.cuh"

namespace e2d {
namespace mlp {
namespace ws {

constexpr int A_BYTES = 4 * SLICE_BYTES;     // a tile: 4 slices of 128 rows x 64 columns
template <int TILES> struct Chain {
    static constexpr int RSLOT = TILES == 2 ? 3 : 5;
    static constexpr int SMEM = TILES * A_BYTES + RSLOT * WSLICE_BYTES + 1024;
};

// Step k of a chain, A = the tile of `in` (k = 0) or step k - 1's output: out =
// epilogue(A . w[k]^T) forward (weights [N][K], K-major boxes of 256 x 64), out =
// epilogue(A . w[k]) for the data gradient (weights [K][N], N-major boxes of 64
// 64, four to a slice).
struct ChainMaps {
    CUtensorMap in;  // boxes of 128 rows x 64 columns
    CUtensorMap w[MAXL], out[MAXL];  // out: boxes of 32 rows x 64 columns
};
struct ChainArgs {
    int M, steps;              // rows (a multiple of 128), steps
    int first;                 // 64-column slices of the first step's K (1 or 4)
    int keep;                  // forward: first step whose outputs are stored (earlier ones stay on chip)
    int store_aux;             // forward: store gelu'(z)
    bf16 *aux[MAXL];           // gelu'(z) of each step, M x 256, written (forward) or read
    const float *bias[MAXL];   // forward
    int *flag;                 // set to 1 when a wait gave up
};

// 32-byte accesses of one lane (global memory, 32-byte aligned)
__device__ __forceinline__ void load32(const void *p, uint4 &a, uint4 &b) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void store32(void *p, const uint4 &a, const uint4 &b) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n"
                 :: "l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}

// The order in which a CTA takes its tiles' steps (its items): tiles blockIdx.x
// + j gridDim.x in groups of TILES, and within a group step by step, the tiles in
// turn.
template <int TILES> struct Items {
    int ntiles, steps, t0 = (int)blockIdx.x, k = 0, x = 0;
    __device__ __forceinline__ Items(int n, int s) : ntiles(n), steps(s) {}
    __device__ __forceinline__ bool more() const { return t0 < ntiles; }
    __device__ __forceinline__ bool paired() const { return TILES == 2 && t0 + (int)gridDim.x < ntiles; }
    __device__ __forceinline__ int tile() const { return t0 + x * (int)gridDim.x; }
    __device__ __forceinline__ void next() {
        if (x == 0 && paired()) { x = 1; return; }
        x = 0;
        if (++k < steps) return;
        k = 0;
        t0 += TILES * (int)gridDim.x;
    }
};

template <int EPI, int TILES>
__global__ void __launch_bounds__(THREADS, 1) k_chain(const __grid_constant__ ChainMaps maps, const ChainArgs g) {
    constexpr int RSLOT = Chain<TILES>::RSLOT;
    extern __shared__ unsigned char ws_raw[];
    __shared__ __align__(8) uint64_t full[RSLOT], empty[RSLOT], tfull[2], ready[2], mdone;
    __shared__ uint32_t tmem_sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // 1024-byte aligned base: the swizzle pattern is taken from address bits
    const uint32_t Asm = (smem_u32(ws_raw) + 1023u) & ~1023u;
    const uint32_t Rsm = Asm + TILES * A_BYTES;
    Items<TILES> it(g.M / BM, g.steps);
    if (tid == 0) {
        for (int s = 0; s < RSLOT; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(smem_u32(&full[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(smem_u32(&empty[s])));
        }
        for (int a = 0; a < 2; a++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(smem_u32(&tfull[a])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" :: "r"(smem_u32(&ready[a])), "n"(NEPI));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(smem_u32(&mdone)));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     :: "r"(smem_u32(&tmem_sh)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    const uint32_t tmem = tmem_sh;

    if (warp == 0 && lane == 0) {
        // ---- producer ----
        bool ok = true;
        int q = 0;
        auto claim = [&](int bytes) {  // the next slot
            const int slot = q % RSLOT;
            ok = ok && wait(smem_u32(&empty[slot]), ((q / RSLOT) & 1) ^ 1);
            if (ok) expect_tx(smem_u32(&full[slot]), bytes);
            return slot;
        };
        for (; it.more() && ok; it.next())
            for (int s = 0; s < (it.k == 0 ? g.first : 4) && ok; s++) {
                if (it.k == 0) {
                    const int a = claim(SLICE_BYTES);
                    if (!ok) break;
                    tma_load(Rsm + a * WSLICE_BYTES, &maps.in, s * KC, it.tile() * BM, smem_u32(&full[a]));
                    q++;
                }
                const int b = claim(WSLICE_BYTES);
                if (!ok) break;
                const uint32_t dst = Rsm + b * WSLICE_BYTES;
                if (EPI == EPI_BIAS_GELU) tma_load(dst, &maps.w[it.k], s * KC, 0, smem_u32(&full[b]));
                else
                    for (int j = 0; j < 4; j++)
                        tma_load(dst + j * WBOX, &maps.w[it.k], 64 * j, s * KC, smem_u32(&full[b]));
                q++;
            }
        if (!ok) atomicExch(g.flag, 1);
        // every copy issued lands before the CTA can leave
        for (int j = q - RSLOT > 0 ? q - RSLOT : 0; j < q; j++) wait(smem_u32(&full[j % RSLOT]), (j / RSLOT) & 1);
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issuer ----
        bool ok = true;
        int q = 0, li = 0;  // ring slots taken, items issued
        for (; it.more() && ok; it.next(), li++) {
            const int acc = li & 1;
            // the item two back has read this accumulator; it is also the
            // tile's step before when two tiles alternate.  With one tile
            // that step is the item before, whose epilogue has written A.
            if (it.k > 0 && !it.paired()) ok = wait(smem_u32(&ready[acc ^ 1]), ((li - 1) >> 1) & 1);
            else ok = wait(smem_u32(&ready[acc]), ((li >> 1) & 1) ^ 1);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n");
            const uint32_t dt = tmem + (uint32_t)(acc * ND);
            const int slices = it.k == 0 ? g.first : 4;
            for (int s = 0; s < slices && ok; s++) {
                uint32_t a = Asm + it.x * A_BYTES + s * SLICE_BYTES;
                int sa = -1;
                if (it.k == 0) {
                    sa = q % RSLOT;
                    ok = wait(smem_u32(&full[sa]), (q / RSLOT) & 1);
                    a = Rsm + sa * WSLICE_BYTES;
                    q++;
                }
                const int sw = q % RSLOT;
                ok = ok && wait(smem_u32(&full[sw]), (q / RSLOT) & 1);
                q++;
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n");
#pragma unroll
                for (int kk = 0; kk < KC / 16; kk++) {
                    const uint64_t ad = desc_sw128(a + kk * 32);
                    const uint32_t b = Rsm + sw * WSLICE_BYTES;
                    const uint64_t bd = EPI == EPI_BIAS_GELU ? desc_sw128(b + kk * 32) : desc_sw128_mn(b + kk * 2048);
                    constexpr uint32_t idesc = EPI == EPI_BIAS_GELU ? IDESC : IDESC | (1u << 16);  // B N-major
                    const uint32_t accumulate = (s > 0 || kk > 0) ? 1u : 0u;
                    asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
                                 " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                                 :: "r"(dt), "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate));
                }
                if (sa >= 0) commit(smem_u32(&empty[sa]));
                commit(smem_u32(&empty[sw]));
            }
            if (ok) commit(smem_u32(&tfull[acc]));
        }
        if (!ok) atomicExch(g.flag, 1);
        // every MMA issued completes before the tensor memory is freed
        commit(smem_u32(&mdone));
        wait(smem_u32(&mdone), 0);
    } else if (warp >= 2) {
        // ---- epilogue: rows 32 quarter .. and columns 64 group .. of the tile ----
        const int quarter = warp & 3, group = (warp - 2) >> 2, col0 = group * 64;
        const uint32_t own0 = Asm + (uint32_t)(group * SLICE_BYTES + quarter * 32 * 128);  // 32 rows of 128 bytes
        const int sw = lane & 7;  // 16-byte unit u of a row is at ((u ^ sw) << 4)
        // where this lane's 16 values of a chunk of gelu'(z) are
        auto aux_at = [&](const Items<TILES> &i, int ch) {
            if (EPI == EPI_BIAS_GELU && i.k == g.steps - 1)
                return g.aux[i.k] + (size_t)(i.tile() * BM + quarter * 32 + lane) * ND + col0 + 16 * ch;
            return g.aux[i.k] + (size_t)i.tile() * BM * ND + (((warp - 2) * 4 + ch) * 32 + lane) * 16;
        };
        uint4 za[4], zb[4];  // data gradient: this lane's gelu'(z) factors, requested an item ahead
        if (EPI == EPI_GELU_BWD && it.more())
#pragma unroll
            for (int c = 0; c < 4; c++) load32(aux_at(it, c), za[c], zb[c]);
        bool ok = true;
        for (int li = 0; it.more(); li++) {
            const int acc = li & 1, row0 = it.tile() * BM + quarter * 32;
            const uint32_t own = own0 + it.x * A_BYTES, row = own + (uint32_t)(lane * 128);
            // one lane waits and the warp follows its answer, so that the warp
            // stays converged for the collective tensor-memory loads; this
            // tile's earlier stores have read A
            int okw = 1;
            if (lane == 0) {
                okw = (int)wait(smem_u32(&tfull[acc]), (li >> 1) & 1);
                if (it.paired()) asm volatile("cp.async.bulk.wait_group.read 1;\n" ::: "memory");  // the other tile's
                else asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
            }
            okw = __shfl_sync(0xffffffffu, okw, 0);
            if (!okw) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n");
#pragma unroll
            for (int ch = 0; ch < 4; ch++) {  // 16 columns at a time
                const int n0 = col0 + ch * 16;
                uint32_t v[16];
                const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * ND + n0);
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                    "[%16];\n"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                      "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                      "=r"(v[14]), "=r"(v[15])
                    : "r"(taddr));
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                __align__(16) __nv_bfloat162 o2[8];
                if (EPI == EPI_BIAS_GELU) {
                    __align__(16) __nv_bfloat162 z2[8];
                    const float4 *bias = (const float4 *)(g.bias[it.k] + n0);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float4 b4 = __ldg(bias + (j >> 1));
                        const float2 bb = j & 1 ? make_float2(b4.z, b4.w) : make_float2(b4.x, b4.y);
                        const float2 z = __fadd2_rn(make_float2(__uint_as_float(v[2 * j]),
                                                                __uint_as_float(v[2 * j + 1])), bb);
                        float2 hh, gg;
                        gelu_and_grad2(z, hh, gg);
                        o2[j] = __floats2bfloat162_rn(hh.x, hh.y);
                        z2[j] = __floats2bfloat162_rn(gg.x, gg.y);
                    }
                    if (g.store_aux) store32(aux_at(it, ch), ((const uint4 *)z2)[0], ((const uint4 *)z2)[1]);
                } else {
                    const __align__(16) uint4 zz[2] = {za[ch], zb[ch]};
                    const __nv_bfloat162 *z2 = (const __nv_bfloat162 *)zz;
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float2 d = __fmul2_rn(make_float2(__uint_as_float(v[2 * j]),
                                                                __uint_as_float(v[2 * j + 1])),
                                                    __bfloat1622float2(z2[j]));
                        o2[j] = __floats2bfloat162_rn(d.x, d.y);
                    }
                }
                const uint4 *po = (const uint4 *)o2;
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n"
                             :: "r"(row + (uint32_t)(((2 * ch) ^ sw) << 4)), "r"(po[0].x), "r"(po[0].y),
                                "r"(po[0].z), "r"(po[0].w) : "memory");
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n"
                             :: "r"(row + (uint32_t)(((2 * ch + 1) ^ sw) << 4)), "r"(po[1].x), "r"(po[1].y),
                                "r"(po[1].z), "r"(po[1].w) : "memory");
            }
            // the accumulator has been read and A written: visible to the
            // async proxy (the next step's MMAs and the store)
            asm volatile("tcgen05.fence::before_thread_sync;\n");
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                arrive(smem_u32(&ready[acc]));
                if (EPI != EPI_BIAS_GELU || it.k >= g.keep) tma_store(&maps.out[it.k], own, col0, row0);
                asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
            }
            it.next();
            if (EPI == EPI_GELU_BWD && it.more())
#pragma unroll
                for (int c = 0; c < 4; c++) load32(aux_at(it, c), za[c], zb[c]);
        }
        if (!ok && lane == 0) atomicExch(g.flag, 1);
        // the stores have completed before the CTA leaves
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
        __syncwarp();
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" :: "r"(tmem), "r"(TMEM_COLS));
}

}  // namespace ws
}  // namespace mlp
}  // namespace e2d
