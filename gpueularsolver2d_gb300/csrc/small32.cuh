// small32.cuh -- whole iterations of a small FP32 mesh in one launch.
//
// Up to kSmallCells cells the passes of an iteration are launch bound: 8192
// cells took 2.2 us for each of 21 launches.  Here one cluster of 16 CTAs holds
// the mesh: every thread keeps one or two cells (geometry, face codes, start
// state, residual) in registers, the arrays that neighbours read (state, face
// states, residual, sweeps) lie in the CTAs' shared memory and are gathered
// through distributed shared memory, and the passes are separated by cluster
// barriers.  A sixteenth of the cells, a multiple of 128, belongs to each CTA,
// so that the residual's partial sums group as in the other path; a warp of CTA
// 0 that holds no cells folds them while the next iteration's first pass, which
// changes no state, already runs.  Same operations per cell, same bits.
#pragma once

#include "kernels.cuh"
#include "resid.cuh"

namespace e2d {

constexpr int kSmallCtas = 16;        // the largest (non-portable) cluster
constexpr int kSmallThreads = 512;    // threads with cells at most; one more warp for the residual
constexpr int kSmallPerCta = 1024;    // cells of a CTA at most: two per thread
constexpr int kSmallCells = kSmallCtas * kSmallPerCta;
constexpr int kSmallParts = kSmallCells / 128;

struct SmallArgs {
    MeshDev<float> m;
    Flow<float> f;
    V4<float> *W;    // start state and result
    V4<float> *phi;
    Ctl *ctl;
    double *hist;
    int hist_cap, stages, sweeps, cells, iters;  // cells of a CTA; iterations of the launch at most
    float rk[8];
};

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
// The address in CTA rank of this CTA's shared address a.
__device__ __forceinline__ uint32_t map_shared(uint32_t a, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ V4<float> load_cluster(uint32_t a) {
    V4<float> v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ int load_cluster_int(uint32_t a) {
    int v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];\n" : "=r"(v) : "r"(a) : "memory");
    return v;
}

// Dynamic shared memory: [cells] state, [3 cells] face states, [cells]
// residual, [cells] or [2 cells] sweeps.
inline size_t small_smem(int cells, int sweeps) { return (size_t)cells * sizeof(V4<float>) * (sweeps > 2 ? 7 : 6); }

template <bool OPT, int CPT>
__global__ void __launch_bounds__(kSmallThreads + 32, 1) k_small32(const __grid_constant__ SmallArgs g) {
    extern __shared__ __align__(32) unsigned char smem[];
    __shared__ Ctl ctl;                          // CTA 0: the control block
    __shared__ float2 parts[kSmallParts];        // CTA 0: squares of each 128 cells
    __shared__ int bads[kSmallParts];            // CTA 0: unphysical cells of each 128
    __shared__ float2 wsq[CPT][kSmallThreads / 32];
    __shared__ int wbad[CPT][kSmallThreads / 32];
    if (g.ctl->halt) return;  // the same for every CTA
    const int C = g.cells, t = threadIdx.x, warp = t >> 5, lane = t & 31, n = g.m.n;
    const int TH = blockDim.x - 32;  // threads with cells: C / CPT, a multiple of 128
    const int rank = (int)cluster_rank();
    const bool worker = t < TH;
    V4<float> *Ws = reinterpret_cast<V4<float> *>(smem), *FSs = Ws + C, *RES = FSs + 3 * C, *SM = RES + C;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem), row = (uint32_t)C * 16u;
    const uint32_t off_res = 4 * row, off_sm = 5 * row;
    const uint32_t ctl0 = map_shared((uint32_t)__cvta_generic_to_shared(&ctl), 0);
    const uint32_t parts0 = map_shared((uint32_t)__cvta_generic_to_shared(parts), 0);
    const uint32_t bads0 = map_shared((uint32_t)__cvta_generic_to_shared(bads), 0);
    if (rank == 0 && t == 0) ctl = *g.ctl;

    bool live[CPT];
    int id[CPT], at[CPT], code[CPT][3], clog[CPT];
    uint32_t nb[CPT][3];  // the neighbours' places in the cluster's arrays
    V2<float> S[CPT][3];
    V4<float> w0[CPT], r[CPT];
    float area[CPT], dt[CPT];
#pragma unroll
    for (int j = 0; j < CPT; j++) {
        at[j] = j * TH + t;
        id[j] = rank * C + at[j];
        live[j] = worker && at[j] < C && id[j] < n;
        clog[j] = 0;
        area[j] = 1.f;
        w0[j] = r[j] = V4<float>{};
#pragma unroll
        for (int k = 0; k < 3; k++) { code[j][k] = -2; nb[j][k] = base; S[j][k] = V2<float>{}; }
        if (!live[j]) continue;
        const int4 tp = g.m.topo[id[j]];
        code[j][0] = tp.x; code[j][1] = tp.y; code[j][2] = tp.z;
        clog[j] = tp.w;
        area[j] = g.m.area[id[j]];
        w0[j] = g.W[id[j]];
        Ws[at[j]] = w0[j];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            S[j][k] = g.m.S[k * n + id[j]];
            if (code[j][k] < 0) continue;
            const int c = code[j][k] >> 3;
            nb[j][k] = map_shared(base, c / C) + (uint32_t)(c % C) * 16u;
        }
    }
    // the residual of the iteration done: partial sums in the order of k_resid
    auto fold = [&] {
        if (rank != 0 || worker) return;
        const int np = (n + 127) / 128;
        double v[4];
        int bad = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int k = lane + 32 * q;
            v[q] = k < np ? (double)parts[k].x + (double)parts[k].y : 0.0;
            if (k < np) bad += bads[k];
        }
        double s = (v[0] + v[2]) + (v[1] + v[3]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s += __shfl_down_sync(0xffffffffu, s, o);
            bad += __shfl_down_sync(0xffffffffu, bad, o);
        }
        if (lane == 0) {
            ctl.nbad += bad;
            resid_finish(0.0 + s, &ctl, g.hist, g.hist_cap);
        }
    };
    cluster_sync();
    // the control block as this thread last saw it
    int frozen = OPT ? load_cluster_int(ctl0 + offsetof(Ctl, frozen)) : 0;
    int step = OPT ? load_cluster_int(ctl0 + offsetof(Ctl, step)) : 0;
    bool pending = false, halted = false;
    for (int it = 0; it < g.iters && !halted; it++) {
        for (int st = 0; st < g.stages; st++) {
            const bool last = st == g.stages - 1;
            // A: face states and time step
            const bool first = OPT && step < g.f.first_order;
#pragma unroll
            for (int j = 0; j < CPT; j++) {
                if (!live[j]) continue;
                const V4<float> U = Ws[at[j]];
                V4<float> nbv[3];
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    if (code[j][k] >= 0) nbv[k] = load_cluster(nb[j][k]);
                    else FSs[k * C + at[j]] = nbv[k] = ghost(code[j][k], U, S[j][k].x, S[j][k].y, g.f);
                }
                dt[j] = faces_cell32<OPT>(g.m, g.f, id[j], code[j], S[j], U, nbv, g.phi, frozen, first,
                                          [&](int k, const V4<float> &o) { FSs[k * C + at[j]] = o; });
            }
            if (st == 0 && pending) fold();
            cluster_sync();
            if (st == 0 && pending) {
                pending = false;
                halted = load_cluster_int(ctl0 + offsetof(Ctl, halt)) != 0;
                if (halted) break;
            }
            // B: fluxes
#pragma unroll
            for (int j = 0; j < CPT; j++) {
                if (!live[j]) continue;
                V4<float> own[3], oth[3];
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    own[k] = code[j][k] >= 0 ? FSs[k * C + at[j]] : Ws[at[j]];
                    if (code[j][k] >= 0) oth[k] = load_cluster(nb[j][k] + (1 + (code[j][k] & 3)) * row);
                    else oth[k] = FSs[k * C + at[j]];
                }
                V4<float> s = {};
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    bool right;
                    const V4<float> F = face_flux_of(g.f, code[j][k], S[j][k], own[k], oth[k], right);
                    add_flux(s, F, right);
                }
                r[j] = s;
                RES[at[j]] = s;
            }
            cluster_sync();
            // C: smoothing sweeps but the last
            auto nb_values = [&](int j, uint32_t off) {
                V4<float> d = {};
#pragma unroll
                for (int k = 0; k < 3; k++)
                    if (code[j][k] >= 0) {
                        const V4<float> v = load_cluster(nb[j][k] + off);
                        d.x += v.x; d.y += v.y; d.z += v.z; d.w += v.w;
                    }
                return d;
            };
            uint32_t src = off_res;
            for (int sw = 0; sw + 1 < g.sweeps; sw++) {
                V4<float> *dst = SM + (sw & 1) * C;
#pragma unroll
                for (int j = 0; j < CPT; j++)
                    if (live[j]) dst[at[j]] = smooth_value(g.f.irs_eps, clog[j], nb_values(j, src), r[j]);
                cluster_sync();
                src = off_sm + (sw & 1) * row;
            }
            // D: last sweep and update
#pragma unroll
            for (int j = 0; j < CPT; j++) {
                float drho = 0.f;
                int bad = 0;
                if (live[j]) {
                    V4<float> d = {};
                    if (g.sweeps > 0) d = nb_values(j, src);
                    const V4<float> w = update_value(g.f.irs_eps, g.rk[st], g.sweeps > 0 ? 1 : 0, clog[j], r[j], d, dt[j],
                                                     area[j], w0[j], last, drho, bad);
                    Ws[at[j]] = w;
                    if (last) w0[j] = w;
                }
                if (last && worker) {
                    const float2 sq = warp_squares(drho);
                    const unsigned mask = __ballot_sync(0xffffffffu, bad);
                    if (lane == 0) {
                        wsq[j][warp] = sq;
                        wbad[j][warp] = __popc(mask);
                    }
                }
            }
            if (last) {
                __syncthreads();
                // the sums of each 128 cells, to CTA 0
                const int j = t / (TH / 128), q = t % (TH / 128) * 4;
                const int part = rank * (C / 128) + t;
                if (j < CPT && t < C / 128 && part < kSmallParts) {
                    float sh = 0.f, sl = 0.f;
                    int b = 0;
                    for (int k = 0; k < 4; k++) {
                        pair_add(sh, sl, wsq[j][q + k].x, wsq[j][q + k].y);
                        b += wbad[j][q + k];
                    }
                    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};\n" :: "r"(parts0 + part * 8), "f"(sh),
                                 "f"(sl) : "memory");
                    asm volatile("st.shared::cluster.u32 [%0], %1;\n" :: "r"(bads0 + part * 4), "r"(b) : "memory");
                }
            }
            cluster_sync();
        }
        if (halted) break;
        pending = true;
        if (OPT) {  // the next iteration's first pass depends on the step and on the freezing
            fold();
            cluster_sync();
            pending = false;
            frozen = load_cluster_int(ctl0 + offsetof(Ctl, frozen));
            step = load_cluster_int(ctl0 + offsetof(Ctl, step));
            halted = load_cluster_int(ctl0 + offsetof(Ctl, halt)) != 0;
        }
    }
    if (pending) fold();
#pragma unroll
    for (int j = 0; j < CPT; j++)
        if (live[j]) g.W[id[j]] = w0[j];
    cluster_sync();  // the last reads of other CTAs' shared memory are done
    if (rank == 0 && t == 0) *g.ctl = ctl;
}

template <bool OPT, int CPT> bool small_launch(const SmallArgs &a, cudaStream_t s, bool probe) {
    auto *kern = &k_small32<OPT, CPT>;
    const size_t bytes = small_smem(a.cells, a.sweeps);
    if (probe && (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
                  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)small_smem(kSmallPerCta, 3)) != cudaSuccess))
        return false;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = kSmallCtas;
    cfg.blockDim = a.cells / CPT + 32;
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kSmallCtas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (probe) {
        int clusters = 0;
        return cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters > 0;
    }
    return cudaLaunchKernelEx(&cfg, kern, a) == cudaSuccess;
}

// us per iteration of 4 stages, this against one launch per pass: 2k cells 14.7 and
// 35.6; 8k 21.2 and 36.4, with the cell-wise limiter 27.5 and 38.9; 12k 29.1 and 36.3;
// 16k 33.6 and 37.8 (two cells to a thread
// spill with the options: they stop at one).  A pass more costs a launch about 1.5
// us and this kernel 0.75, a stage's flux and reconstruction of two cells per thread
// more than the launches: above 768 cells to a CTA the launches win with less than
// two sweeps and more than three stages.  16k cells (and 12.3k) in file order, without
// smoothing: 3 stages 20.4 and 20.0 (20.2, 20.5), 4 stages 26.7 and 25.4 (26.5, 25.6),
// 8 stages 51.8 and 46.5 (51.5, 46.8); one sweep, 4 stages 28.1 and 27.4 (28.4, 27.7);
// two sweeps, 8 stages 60.5 and 62.5 (61.6, 62.3).  12288 cells, 4 stages, without
// smoothing: 22.8 and 24.9.
bool small_iterations(const Plan<float> &p, int iters, cudaStream_t s, bool probe) {
    const bool opt = faces_options(p.f, p.phi);
    if (p.m.n > (opt ? kSmallCtas * kSmallThreads : kSmallCells) || p.block != 128 || p.f.global_dt) return false;
    if (p.m.n > small_dense_cells && p.sweeps < 2 && p.stages > 3) return false;
    SmallArgs a;
    a.m = p.m; a.f = p.f; a.W = p.W[0]; a.phi = p.phi; a.ctl = p.ctl; a.hist = p.hist; a.hist_cap = p.hist_cap;
    a.stages = p.stages; a.sweeps = p.sweeps; a.iters = iters;
    for (int k = 0; k < 8; k++) a.rk[k] = p.rk[k];
    const int per = (p.m.n + kSmallCtas - 1) / kSmallCtas;
    const bool two = per > kSmallThreads;
    a.cells = two ? (per + 255) / 256 * 256 : (per + 127) / 128 * 128;
    bool ok;
    if (opt) ok = small_launch<true, 1>(a, s, probe);
    else ok = two ? small_launch<false, 2>(a, s, probe) : small_launch<false, 1>(a, s, probe);
    if (probe) cudaGetLastError();  // a GPU without the feature takes the other path
    return ok;
}

}  // namespace e2d
