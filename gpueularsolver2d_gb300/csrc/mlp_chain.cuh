// mlp_chain.cuh -- the hidden layers of the warm-start MLP as one launch per
// direction: the forward pass (bias + GELU) and the data gradient (GELU') of
// every layer, a batch tile staying on its SM from the first layer to the
// last.  No reference counterpart.
//
// A 128-row tile is carried through the layers in shared memory: the epilogue
// of a step writes the next step's A operand in place.  One CTA per SM walks
// the tiles:
//   warp 0  (one thread) streams the operands through a ring of three 32 KB
//           slots by TMA: the tile's own input for the first step, then each
//           step's weights in four slices of 64 columns of K; the slices of
//           the next step arrive while the epilogue of this one runs;
//   warp 1  (one thread) issues tcgen05.mma (kind::f16, M = 128, N = 256, K =
//           16, FP32 accumulate) into one of two 256-column accumulators;
//   warps 2-17 take 32 rows x 64 columns each from tensor memory, apply the
//           epilogue, write the bf16 result over their own part of the A
//           operand (128-byte swizzle, the layout both the next MMA and the TMA
//           store read), store it, and release it to the MMA thread.  gelu'(z)
//           goes out (forward) or comes in (data gradient) through two 32 x 32
//           slabs per warp.
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

constexpr int RSLOT = 3;                     // ring slots
constexpr int A_BYTES = 4 * SLICE_BYTES;     // the tile: 4 slices of 128 rows x 64 columns
constexpr int CHAIN_SMEM = A_BYTES + RSLOT * WSLICE_BYTES + SLABS_BYTES + 1024;

// Step k of a chain, A = the tile of `in` (k = 0) or step k - 1's output: out =
// epilogue(A . w[k]^T) forward (weights [N][K], K-major boxes of 256 x 64), out =
// epilogue(A . w[k]) for the data gradient (weights [K][N], N-major boxes of 64
// x 64, four to a slice).  aux: gelu'(z), written (forward) or read.
struct ChainMaps {
    CUtensorMap in;  // boxes of 128 rows x 64 columns
    CUtensorMap w[MAXL], out[MAXL], aux[MAXL];  // out 32 x 64, aux 32 x 32
};
struct ChainArgs {
    int M, steps;              // rows (a multiple of 128), steps
    int first;                 // 64-column slices of the first step's K (1 or 4)
    int keep;                  // forward: first step whose outputs are stored (earlier ones stay on chip)
    int aux;                   // forward: store gelu'(z)
    const float *bias[MAXL];   // forward
    int *flag;                 // set to 1 when a wait gave up
};

template <int EPI>
__global__ void __launch_bounds__(THREADS, 1) k_chain(const __grid_constant__ ChainMaps maps, const ChainArgs g) {
    extern __shared__ unsigned char ws_raw[];
    __shared__ __align__(8) uint64_t full[RSLOT], empty[RSLOT], tfull[2], ready[2], mdone, auxbar[NEPI];
    __shared__ uint32_t tmem_sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // 1024-byte aligned base: the swizzle pattern is taken from address bits
    const uint32_t Asm = (smem_u32(ws_raw) + 1023u) & ~1023u;
    const uint32_t Rsm = Asm + A_BYTES, Ssm = Rsm + RSLOT * WSLICE_BYTES;
    const int ntiles = g.M / BM;
    if (tid == 0) {
        for (int e = 0; e < NEPI; e++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(smem_u32(&auxbar[e])));
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
        auto claim = [&](int bytes) {  // the next slot, as a barrier and an address
            const int slot = q % RSLOT;
            ok = ok && wait(smem_u32(&empty[slot]), ((q / RSLOT) & 1) ^ 1);
            if (ok) expect_tx(smem_u32(&full[slot]), bytes);
            return slot;
        };
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x)
            for (int k = 0; k < g.steps && ok; k++)
                for (int s = 0; s < (k == 0 ? g.first : 4) && ok; s++) {
                    if (k == 0) {
                        const int a = claim(SLICE_BYTES);
                        if (!ok) break;
                        tma_load(Rsm + a * WSLICE_BYTES, &maps.in, s * KC, t * BM, smem_u32(&full[a]));
                        q++;
                    }
                    const int b = claim(WSLICE_BYTES);
                    if (!ok) break;
                    const uint32_t dst = Rsm + b * WSLICE_BYTES;
                    if (EPI == EPI_BIAS_GELU) tma_load(dst, &maps.w[k], s * KC, 0, smem_u32(&full[b]));
                    else
                        for (int j = 0; j < 4; j++)
                            tma_load(dst + j * WBOX, &maps.w[k], 64 * j, s * KC, smem_u32(&full[b]));
                    q++;
                }
        if (!ok) atomicExch(g.flag, 1);
        // every copy issued lands before the CTA can leave
        for (int j = q - RSLOT > 0 ? q - RSLOT : 0; j < q; j++) wait(smem_u32(&full[j % RSLOT]), (j / RSLOT) & 1);
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issuer ----
        bool ok = true;
        int q = 0, li = 0;  // ring items taken, steps issued
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x)
            for (int k = 0; k < g.steps && ok; k++, li++) {
                const int acc = li & 1;
                // k > 0: the step before has written A (and so has read the
                // accumulator of the one before it).  k = 0: A comes through
                // the ring; the accumulator has been read by step li - 2.
                if (k > 0) ok = wait(smem_u32(&ready[acc ^ 1]), ((li - 1) >> 1) & 1);
                else ok = wait(smem_u32(&ready[acc]), ((li >> 1) & 1) ^ 1);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n");
                const uint32_t dt = tmem + (uint32_t)(acc * ND);
                const int slices = k == 0 ? g.first : 4;
                for (int s = 0; s < slices && ok; s++) {
                    uint32_t a = Asm + s * SLICE_BYTES;
                    int sa = -1;
                    if (k == 0) {
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
        const int quarter = warp & 3, ew = warp - 2, group = ew >> 2;
        const uint32_t own = Asm + (uint32_t)(group * SLICE_BYTES + quarter * 32 * 128);  // 32 rows of 128 bytes
        const uint32_t slab = Ssm + (uint32_t)(ew * 2 * SLAB);
        const uint32_t abar = smem_u32(&auxbar[ew]);
        const int col0 = group * 64;
        const uint32_t row = own + (uint32_t)(lane * 128);
        const int sw = lane & 7;  // 16-byte unit u of the row is at ((u ^ sw) << 4)
        bool ok = true;
        int li = 0, asked = 0;
        auto ask = [&](int t, int k) {  // lane 0: the gelu'(z) factors of a step
            expect_tx(abar, 2 * SLAB);
            tma_load(slab, &maps.aux[k], col0, t * BM + quarter * 32, abar);
            tma_load(slab + SLAB, &maps.aux[k], col0 + 32, t * BM + quarter * 32, abar);
        };
        if (EPI == EPI_GELU_BWD && (int)blockIdx.x < ntiles) {
            if (lane == 0) ask(blockIdx.x, 0);
            asked = 1;
        }
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
            const int row0 = t * BM + quarter * 32;
            for (int k = 0; k < g.steps; k++, li++) {
                const int acc = li & 1;
                // one lane waits and the warp follows its answer, so that the
                // warp stays converged for the collective tensor-memory loads;
                // the stores issued so far have read A and the slabs
                int okw = 1;
                if (lane == 0) {
                    okw = (int)wait(smem_u32(&tfull[acc]), (li >> 1) & 1);
                    asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
                }
                okw = __shfl_sync(0xffffffffu, okw, 0);
                // every lane observes the copy's completion before reading the slabs
                if (EPI == EPI_GELU_BWD) okw = __all_sync(0xffffffffu, okw && wait(abar, li & 1));
                if (!okw) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n");
                const bool store = EPI != EPI_BIAS_GELU || k >= g.keep;
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
                    const uint32_t sl = slab + (uint32_t)((ch >> 1) * SLAB);
                    const uint32_t o0 = slab_off(lane, 2 * (ch & 1)), o1 = slab_off(lane, 2 * (ch & 1) + 1);
                    __align__(16) __nv_bfloat162 o2[8];
                    if (EPI == EPI_BIAS_GELU) {
                        __align__(16) __nv_bfloat162 z2[8];
                        const float4 *bias = (const float4 *)(g.bias[k] + n0);
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
                        if (g.aux) {
                            const uint4 *pz = (const uint4 *)z2;
                            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" :: "r"(sl + o0), "r"(pz[0].x),
                                         "r"(pz[0].y), "r"(pz[0].z), "r"(pz[0].w) : "memory");
                            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" :: "r"(sl + o1), "r"(pz[1].x),
                                         "r"(pz[1].y), "r"(pz[1].z), "r"(pz[1].w) : "memory");
                        }
                    } else {
                        __align__(16) uint4 zz[2];
                        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];\n"
                                     : "=r"(zz[0].x), "=r"(zz[0].y), "=r"(zz[0].z), "=r"(zz[0].w) : "r"(sl + o0) : "memory");
                        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];\n"
                                     : "=r"(zz[1].x), "=r"(zz[1].y), "=r"(zz[1].z), "=r"(zz[1].w) : "r"(sl + o1) : "memory");
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
                // async proxy (the next step's MMAs and the stores)
                asm volatile("tcgen05.fence::before_thread_sync;\n");
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    arrive(smem_u32(&ready[acc]));
                    if (store) tma_store(&maps.out[k], own, col0, row0);
                    if (EPI == EPI_BIAS_GELU && store && g.aux) {
                        tma_store(&maps.aux[k], slab, col0, row0);
                        tma_store(&maps.aux[k], slab + SLAB, col0 + 32, row0);
                    }
                    asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                }
                if (EPI == EPI_GELU_BWD) {
                    // the next step's factors, into the slabs just read
                    const int k1 = k + 1 < g.steps ? k + 1 : 0, t1 = k1 ? t : t + (int)gridDim.x;
                    if (t1 < ntiles) {
                        if (lane == 0) ask(t1, k1);
                        asked++;
                    }
                }
            }
        }
        if (!ok && lane == 0) {
            atomicExch(g.flag, 1);
            // a gelu'(z) copy may still be in flight: let it land (bounded)
            if (EPI == EPI_GELU_BWD && asked) wait(abar, (asked - 1) & 1);
        }
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
