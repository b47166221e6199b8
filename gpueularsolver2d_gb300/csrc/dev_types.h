// dev_types.h -- types shared by the host solver and the kernel translation
// units, and the per-precision launch entry points.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace e2d {

template <typename T> struct alignas(4 * sizeof(T)) V4 { T x, y, z, w; };
template <typename T> struct alignas(2 * sizeof(T)) V2 { T x, y; };

// Device-side iteration control, one per solver (or per batched case).
struct Ctl {
    int step;        // iterations completed
    int halt;        // nonzero: every kernel returns at once (1 done, 2 diverged)
    int target;      // halt when step reaches this
    int check_epsl;  // halt when Resd <= epsl
    int nbad;        // cells with rho <= 0, p <= 0 or NaN after the last iteration
    int fixed_norm;  // epsm given by the caller
    double epsl, epsm, resd;
    int freeze_after;  // > 0: freeze the limiter once step reaches this (option; 0 = reference)
    int frozen;        // limiter values are frozen (set by the residual kernel)
    double freeze_resd;  // > 0: freeze the limiter once Resd falls to this (option)
    // Global time-step option: the smallest local step of RK stage k, as the
    // bits of a non-negative double (whose order is that of the integers), so
    // that blocks fold into it with atomicMin.  kDtNone between iterations.
    unsigned long long dtmin[8];
    unsigned int fold_count;  // blocks of the residual fold done this iteration (0 between iterations)
};

constexpr unsigned long long kDtNone = 0x7FF0000000000000ULL;  // +inf

// Flow constants of one case (gpu_init.cu:63-93).
template <typename T> struct Flow {
    T gamma, ui, vi, ain, tin, vin, R, pis, cfl, dt_cap, eps_entropy, irs_eps;
    T venk_k3;    // K^3 of the Venkatakrishnan option
    int limiter;  // 0 reference, 1 Venkatakrishnan
    int global_dt;  // 1: every cell advances with the smallest local step (option)
    int first_order;  // > 0: first-order faces while fewer iterations are done (option)
    int positivity;   // 1: a non-physical reconstructed face side falls back to the cell state (option)
};

// Cell-local mesh data in internal order (n cells).
//   topo[i] = {f0, f1, f2, clog}; face code f >= 0: (nb << 3) | (right << 2) | slot,
//   -1 far field, -2 wall.  slot = face index of this edge in the neighbour;
//   right = this cell is the edge's right cell in the reference numbering.
//   S[k*n+i] = outward normal of face k in the cell's own node order,
//              (vectory, vectorx) of gpu_init.cu:153-154, so |S| = face length.
//   R[k*n+i] = face midpoint minus cell centroid.
template <typename T> struct MeshDev {
    int n;
    const int4 *__restrict__ topo;
    const V2<T> *__restrict__ S;
    const V2<T> *__restrict__ R;
    const T *__restrict__ area;
};

// Every face once (FP64 on large meshes), in the order of the left cells:
// at[j] = {entry k * n + i of the left (or boundary) cell i, the right cell's entry
// or -1 on a boundary face, i, the right cell}; geo: unit normal, half the length,
// face vector and its square, [6][count]; radius: [3n] a face's spectral radius at
// its left cell's entry.
struct FaceList {
    const int4 *at;
    double *geo, *radius;
    int count;  // 0: passes A and B work in tiles of cells
};

// Cells above which an FP64 mesh, or batch in all, takes a face list.  Below, a launch is as
// long as one thread's chain, and the list's extra launch costs more than it saves.
// us per iteration in tiles and with the list: 8k cells 141 and 152, 12.8k 158 and
// 152, 20k 186 and 185, 34k 220 and 207, 80k 436 and 353, 252k 1059 and 907.
constexpr int face_list_cells = 12000;

// Everything one iteration needs.
template <typename T> struct Plan {
    MeshDev<T> m;
    Flow<T> f;
    V4<T> *W[2];   // W[0] holds the iteration's start state and its result
    V4<T> *FS;     // [3n] face-side states
    V4<T> *phi;    // [3n] limiter values (limiter-freeze option), else null
    T *dt;         // [n]
    V4<T> *res;    // [n]
    V4<T> *sm[2];  // [n] smoothing sweeps (ping-pong)
    double *part;  // [blocks] FP64 partials of sum (rho - rho0)^2
    Ctl *ctl;
    double *hist;
    int hist_cap;
    int stages;
    T rk[8];
    int sweeps;
    int block;
    FaceList faces;
};

template <typename T> int launches_per_iteration(const Plan<T> &p) {
    return p.stages * (3 + (p.faces.count ? 1 : 0) + (p.sweeps > 1 ? p.sweeps - 1 : 0)) + 1;
}

// Batched cases: the cells of all cases in one array, case c in
// [off_c, off_c + n_c) with off_c a multiple of kChunk, so that a tile of B
// cells (B dividing kChunk) lies in one case.  Padding cells are skipped.
constexpr int kChunk = 256;

template <typename T> struct BatchDev {
    const Flow<T> *flows;    // [ncase]
    const int *chunk_case;   // [n / kChunk] case of each chunk
    int *live;               // [n / kChunk] the same, or -1 while the case is halted
    const int *case_end;     // [ncase] one past the last real cell
    Ctl *ctl;                // [ncase]
};

template <typename T> struct BPlan {
    MeshDev<T> m;            // concatenated mesh (n includes padding)
    Flow<T> f;               // parameters shared by all cases (gamma, irs_eps, ...)
    BatchDev<T> b;
    V4<T> *W[2];
    V4<T> *FS;
    V4<T> *phi;              // [3n] limiter values (limiter-freeze option), else null
    T *dt;
    V4<T> *res;
    V4<T> *sm[2];
    double *part;            // [tiles] one partial per tile
    int ncase;
    const int2 *case_tiles;  // [ncase] {first tile, tile count}
    double *hist;            // [ncase * hist_cap]
    int hist_cap;
    int stages;
    T rk[8];
    int sweeps;
    int block;               // cells per tile = threads per CTA
    bool options = true;     // some case uses a scheme option (pass-A option variant)
    int grid;                // CTAs per launch (persistent when < tiles)
    FaceList faces;          // of all cases (FP64)
};

template <typename T> int launches_per_iteration(const BPlan<T> &p) {
    return p.stages * (3 + (p.faces.count ? 1 : 0) + (p.sweeps > 1 ? p.sweeps - 1 : 0)) + 1;
}

template <typename T> void enqueue_batch_iteration(const BPlan<T> &p, cudaStream_t s);

// pairs: the partials are float2 pairs (FP32 stencil) rather than doubles.
void enqueue_batch_resid(double *part, const int2 *case_tiles, int ncase, Ctl *ctl, double *hist,
                         int hist_cap, bool pairs, int *live, int block, cudaStream_t s);
// The chunks' live table from the cases' halt flags; before the first iteration
// after the host has set them.
void enqueue_batch_live(const int *chunk_case, int *live, int nchunk, const Ctl *ctl, cudaStream_t s);

// Enqueue one iteration (all RK stages + the residual) on a stream.
// Instantiated for double in kernels_f64.cu and for float in kernels_f32.cu.
template <typename T> void enqueue_iteration(const Plan<T> &p, cudaStream_t s);

// Up to `iters` iterations of a small FP32 mesh in one launch (small32.cuh); it
// stops by itself like the passes do.  False when it does not apply to the plan
// (probe: asked once, nothing is launched) or the launch failed.
bool small_iterations(const Plan<float> &p, int iters, cudaStream_t s, bool probe);

// Cells up to which that is the faster way for every scheme and number of
// iterations (768 to a CTA).  Above, not for schemes that small_iterations leaves
// out, nor for a call of a single iteration, which has the kernel's loads of the
// mesh to itself: us per call at 16k cells, in one launch and in passes, 72 and 64
// for one iteration, 99 and 101 for two, 164 and 174 for four.
constexpr int small_dense_cells = 12288;

// Same, with an event pair around every launch (per-pass timing).
template <typename T> int enqueue_iteration_timed(const Plan<T> &p, cudaStream_t s, cudaEvent_t *ev, int *kind);

// FP64 file-order state <-> T internal-order state (perm[i] = file index).
template <typename T>
void enqueue_import(int n, const int *perm, const double *wfile, V4<T> *W, cudaStream_t s);
template <typename T>
void enqueue_export(int n, const int *perm, const V4<T> *W, double *wfile, cudaStream_t s);

// The states of cells[0 .. cnt), FP64.
template <typename T>
void enqueue_export_cells(int cnt, const int *cells, const V4<T> *W, double *w, cudaStream_t s);

// Geometry of a face list from the mesh's face vectors.
void enqueue_face_geometry(const MeshDev<double> &m, const FaceList &l, cudaStream_t s);

// Residual kernel launcher (resid.cu).
void enqueue_resid(double *part, int nparts, Ctl *ctl, double *hist, int hist_cap, bool pairs,
                   cudaStream_t s);

}  // namespace e2d
