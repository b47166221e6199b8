// kernels.cuh -- the solve-path kernels for sm_103a, templated on the stencil
// precision T (double or float).
//
// One RK stage is four passes over the cells (a grid-wide dependency
// separates each pair):
//   A  k_faces : boundary ghosts + Green-Gauss gradient + neighbour min/max
//                + per-face limited reconstruction of the cell's own side of
//                its three faces + spectral radius sum -> local time step
//   B  k_flux  : per cell, Roe flux of its three faces from the two face-side
//                states, summed with the reference's signs and face order
//   C  k_smooth: implicit residual smoothing sweep (all but the last sweep)
//   D  k_update: last smoothing sweep + magnitude clamp + RK update, and on
//                the last stage the (rho - rho0)^2 block partials
// and k_resid folds the partials into Resd on the last stage.
//
// Every cell gathers its own faces, so nothing is accumulated with atomics
// and the result does not depend on scheduling.  An interior face inside one
// block's tile of cells is evaluated once; a face between two tiles is
// evaluated by both cells from identical inputs, so both see the same value.
// (Large FP64 meshes evaluate every face once from a list and split pass B in
// two: k_face_flux, k_face_sum.)  The arithmetic of each quantity follows the reference kernel
// it replaces operation by operation (cited per function); compiled without
// FMA contraction, the FP64 instantiation reproduces the CPU oracle bit for
// bit.
#pragma once

#include "dev_types.h"
#include "fp64_alu.cuh"
#include "pdl.cuh"

namespace e2d {

// Occupancy targets (minimum resident 256-thread blocks per SM) of the two
// gather kernels; the register budget follows from them.  Build-time knobs.
// 0 leaves the choice to the compiler.  Both kernels are latency bound.
// Pass A: 6 (40 registers); on the 4.2M-cell mesh 6 beat the compiler's own
// 48-register choice by 12 % (sweep over 1, 4, 5, 6 at 128 and 256 threads
// per block).  Pass B requests the inputs of all three faces before its
// first flux, which needs 63 registers: 4 blocks (99.7 -> 89.2 us per launch
// against the one-face-at-a-time form at 6 blocks; 94.4 us at 5 blocks,
// where it spills).
#ifndef E2D_MINB_FACES
#define E2D_MINB_FACES 6
#endif
#ifndef E2D_MINB_FLUX
#define E2D_MINB_FLUX 4
#endif
// The targets apply to the FP32 kernels; the FP64 (parity) kernels keep two
// blocks, enough registers for their ~100 live doubles without spilling.
template <typename T> struct MinBlocks { static constexpr int faces = 2, flux = 2; };
template <> struct MinBlocks<float> {
    static constexpr int faces = E2D_MINB_FACES > 0 ? E2D_MINB_FACES : 1;
    static constexpr int flux = E2D_MINB_FLUX > 0 ? E2D_MINB_FLUX : 1;
};
// FP32 pass A with the scheme options needs 64 registers not to spill (at 40 it
// spilled 148 / 416 bytes per thread): an iteration of 131k cells with the
// cell-wise limiter 63.2 -> 60.5 us, of 24 batched cases of 33k cells with the
// smooth limiter (48 registers before) 295 -> 281 us.
constexpr int kOptBlocks = 4;
// The batched (persistent, tile-walking) FP32 kernels hold a few more live
// values across their tile loop: one block fewer per SM, so that they do not
// spill (at the single-case targets ptxas spilled 144 / 60 bytes per thread).
template <typename T> struct BatchMinBlocks {
    static constexpr int faces = MinBlocks<T>::faces > 2 ? MinBlocks<T>::faces - 1 : MinBlocks<T>::faces;
    static constexpr int flux = MinBlocks<T>::flux > 2 ? MinBlocks<T>::flux - 1 : MinBlocks<T>::flux;
};

// Pass B variant.  FP64 evaluates each interior face inside a block's tile of
// cells once (flux_tile): the FP64 Roe flux is arithmetic bound on this GPU,
// and evaluating about half as many pays for the tile's list (1.75 against 1.27
// ms for an iteration on a 51.8k-cell mesh when it was introduced).  FP32 is bound by memory latency, where the
// tile's work list and barriers cost more than they save (0.152 against
// 0.110 ms per launch on 4.2M cells), so every cell evaluates its own three
// faces (flux_cell).  Either way both cells of a face use the same flux bits.
template <typename T> struct FluxTiled { static constexpr bool value = sizeof(T) == 8; };
#define E2D_LB_FLUX __launch_bounds__(256, MinBlocks<T>::flux)

template <typename T> __device__ __forceinline__ T tabs(T v) { return fabs(v); }
template <typename T> __device__ __forceinline__ T tsqrt(T v) { return sqrt(v); }
template <> __device__ __forceinline__ double tsqrt<double>(double v) { return dsqrt(v); }
// |x| < |y| (FP64: fp64_alu.cuh)
__device__ __forceinline__ bool abs_less(float x, float y) { return fabsf(y) > fabsf(x); }
template <typename T> __device__ __forceinline__ T tmin(T a, T b) { return fmin(a, b); }
template <typename T> __device__ __forceinline__ T tmax(T a, T b) { return fmax(a, b); }

// a * b + c: two roundings in FP64 (the oracle's arithmetic; the FP64 units
// are built without contraction), one fused multiply-add in FP32.  Explicit,
// so the FP32 result does not depend on where the compiler contracts.
template <typename T> __device__ __forceinline__ T madd(T a, T b, T c) { return a * b + c; }
template <> __device__ __forceinline__ float madd<float>(float a, float b, float c) { return fmaf(a, b, c); }

// Divisions and square roots of the stencil's hot paths: in FP64 the IEEE
// results (bit parity with the oracle) from the integer units, fp64_alu.cuh; in FP32 the special-function unit's approximate
// reciprocal, reciprocal square root and square root (rcp / rsqrt /
// sqrt.approx.f32, a few ulp), one instruction each where the IEEE forms take
// a refinement sequence: the FP32 gather passes are issue bound.
__device__ __forceinline__ float frcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float frsqrt(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float fsqrt(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
template <typename T> __device__ __forceinline__ T fdiv(T a, T b) { return a / b; }
template <> __device__ __forceinline__ float fdiv<float>(float a, float b) { return a * frcp(b); }
template <> __device__ __forceinline__ double fdiv<double>(double a, double b) { return ddiv(a, b); }
// The same with several numerators over one divisor.  FP64: FastOps, whose user
// does its formula again with IeeeOps where an operand was out of range.
struct Ops32 {
    __device__ __forceinline__ float over(float b) { return frcp(b); }
    __device__ __forceinline__ float by(float a, float r) { return a * r; }
};
template <typename T> struct OpsFor { typedef Ops32 type; };
template <> struct OpsFor<double> { typedef FastOps type; };
template <typename T> using OpsOf = typename OpsFor<T>::type;
// Divisions of the boundary ghosts: the compiler's in FP32.
template <typename T> __device__ __forceinline__ T gdiv(T a, T b) { return a / b; }
template <> __device__ __forceinline__ double gdiv<double>(double a, double b) { return ddiv(a, b); }
template <typename T> struct GOver {
    T b;
    __device__ __forceinline__ explicit GOver(T v) : b(v) {}
    __device__ __forceinline__ T operator()(T a) const { return a / b; }
};
template <> struct GOver<double> {
    Divisor d;
    __device__ __forceinline__ explicit GOver(double v) : d(divisor(v)) {}
    __device__ __forceinline__ double operator()(double a) const { return div_by(a, d); }
};

template <typename T> __device__ __forceinline__ T comp(const V4<T> &v, int k) {
    return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w;
}

// gpu_solver.cu:49-60 (kernel_CalculationPTA): pressure and sound speed
template <typename T> __device__ __forceinline__ void pta(const V4<T> &w, T g, T &P, T &A) {
    const GOver<T> by(w.x);
    T U = by(w.y);
    T V = by(w.z);
    T E = by(w.w) - T(0.5) * (U * U + V * V);
    P = (g - T(1.0)) * w.x * E;
    A = tsqrt(by(g * P));
}

// gpu_solver.cu:62-135 (kernel_Far_Boundary): far-field ghost state from the
// interior state dw (with its P, A) and the face vector (vectorx, vectory).
template <typename T>
__device__ __noinline__ V4<T> far_ghost(const V4<T> dw, T P, T A, T vectorx, T vectory,
                                        const Flow<T> f) {
    const T g = f.gamma;
    T nn = tsqrt(vectorx * vectorx + vectory * vectory);
    T nx = gdiv(vectory, nn);
    T ny = gdiv(vectorx, nn);
    T UD = gdiv(dw.y, dw.x);
    T VD = gdiv(dw.z, dw.x);
    T Un = tabs(f.ui * nx + f.vi * ny);
    T Uncell = UD * nx + VD * ny;
    V4<T> w0 = dw;
    if (gdiv(Un, f.ain) > T(1.0)) {
        if (!(Uncell > T(0.0))) {
            w0.x = T(1.0);
            w0.y = f.ui;
            w0.z = f.vi;
            w0.w = gdiv(gdiv(f.R * f.tin, f.vin * f.vin), g - T(1.0)) + T(0.50);
        }
    } else {
        T PA = f.pis, PD = P, AD = A, ROUD = dw.x, PB, UB, VB;
        if (Uncell > T(0.0)) {
            PB = PA;
            w0.x = ROUD + gdiv(gdiv(PB - PD, AD), AD);
            UB = UD + gdiv(gdiv(nx * (PD - PB), ROUD), AD);
            VB = VD + gdiv(gdiv(ny * (PD - PB), ROUD), AD);
        } else {
            PB = T(0.5) * (PA + PD - ROUD * AD * (nx * (f.ui - UD) + ny * (f.vi - VD)));
            w0.x = T(1.0) + gdiv(gdiv(PB - PA, AD), AD);
            UB = f.ui - gdiv(gdiv(nx * (PA - PB), ROUD), AD);
            VB = f.vi - gdiv(gdiv(ny * (PA - PB), ROUD), AD);
        }
        w0.y = UB * w0.x;
        w0.z = VB * w0.x;
        w0.w = gdiv(PB, g - T(1.0)) + T(0.5) * (UB * UB + VB * VB) * w0.x;
    }
    return w0;
}

// FP64: the same operations; divisions by one divisor share its preparation,
// and the supersonic test's quotient exceeds 1 only where Un > AIN.
template <>
inline __device__ __noinline__ V4<double> far_ghost<double>(const V4<double> dw, double P, double A, double vectorx,
                                                     double vectory, const Flow<double> f) {
    const double g = f.gamma;
    const Divisor dn = divisor(tsqrt(vectorx * vectorx + vectory * vectory)), dr = divisor(dw.x);
    const double nx = div_by(vectory, dn), ny = div_by(vectorx, dn);
    const double UD = div_by(dw.y, dr), VD = div_by(dw.z, dr);
    const double Un = fabs(f.ui * nx + f.vi * ny);
    const double Uncell = UD * nx + VD * ny;
    V4<double> w0 = dw;
    if (Un > f.ain && ddiv(Un, f.ain) > 1.0) {
        if (!(Uncell > 0.0)) {
            w0.x = 1.0;
            w0.y = f.ui;
            w0.z = f.vi;
            w0.w = ddiv(ddiv(f.R * f.tin, f.vin * f.vin), g - 1.0) + 0.50;
        }
    } else {
        const Divisor da = divisor(A);
        const bool out = Uncell > 0.0;
        // outflow: the ghost's pressure is the free stream's, its state follows
        // from the cell's; inflow: from the free stream's (gpu_solver.cu:98-130)
        const double PA = f.pis;
        double PB = PA;
        if (!out) PB = 0.5 * (PA + P - dw.x * A * (nx * (f.ui - UD) + ny * (f.vi - VD)));
        const double dp = out ? PB - P : PB - PA, pd = out ? P - PB : PA - PB;
        w0.x = (out ? dw.x : 1.0) + div_by(div_by(dp, da), da);
        const double du = div_by(div_by(nx * pd, dr), da), dv = div_by(div_by(ny * pd, dr), da);
        const double UB = out ? UD + du : f.ui - du, VB = out ? VD + dv : f.vi - dv;
        w0.y = UB * w0.x;
        w0.z = VB * w0.x;
        w0.w = ddiv(PB, g - 1.0) + 0.5 * (UB * UB + VB * VB) * w0.x;
    }
    return w0;
}

// gpu_solver.cu:188-221: slip-wall ghost (velocity mirrored in the face)
template <typename T>
__device__ __forceinline__ V4<T> wall_ghost(const V4<T> &dw, T vectorx, T vectory, T vectorn) {
    const GOver<T> n(vectorn), r(dw.x);
    T nij0 = n(vectory);
    T nij1 = n(vectorx);
    T UU = r(dw.y);
    T VV = r(dw.z);
    T UV = UU * nij0 + VV * nij1;
    UU = UU - T(2) * UV * nij0;
    VV = VV - T(2) * UV * nij1;
    V4<T> o = dw;
    o.y = dw.x * UU;
    o.z = dw.x * VV;
    return o;
}

// Ghost state across a boundary face code (-1 far, -2 wall).
template <typename T>
__device__ __forceinline__ V4<T> ghost(int code, const V4<T> &U, T Sx, T Sy, const Flow<T> &f) {
    if (code == -1) {
        T P, A;
        pta(U, f.gamma, P, A);
        return far_ghost(U, P, A, Sy, Sx, f);
    }
    T vn = tsqrt(Sy * Sy + Sx * Sx);
    return wall_ghost(U, Sy, Sx, vn);
}

// gpu_solver.cu:385-454 (kernel_deltT): face spectral radius from the mean of
// the two unreconstructed states.  Symmetric in (a, b) and in the sign of S.
// The reference halves the sums of the two states (rou = sum / 2, u = sum_u /
// rou / 2, p = rou EE (g - 1)); here the halves are left out where they cancel
// exactly (a power of two goes through a rounding unchanged), and a half that
// is subtracted is a fused multiply-add with an exact product.  19 FP64
// additions and multiplications where the reference's form issues about 30.
template <typename T> __device__ T spectral_radius(const V4<T> &a, const V4<T> &b, T vectorx, T vectory, T g);
// FP64, with the face vector's square q given.
template <class O>
__device__ __forceinline__ double spectral_radius64(O &o, const V4<double> &a, const V4<double> &b, double vectorx,
                                                    double vectory, double q, double g) {
    const double rou2 = a.x + b.x;  // 2 rou
    const auto d = o.over(rou2);
    const double u = o.by(a.y + b.y, d);
    const double v = o.by(a.z + b.z, d);
    const double EE = fma(-0.5, u * u + v * v, o.by(a.w + b.w, d));
    const double VC = u * vectory + v * vectorx;
    const double p2 = rou2 * EE * (g - 1.0);  // 2 p
    const double CS = o.sqrt(o.by(g * p2, d) * q);
    return tabs(VC) + CS;
}
static __device__ __noinline__ double spectral_radius_ieee(const V4<double> a, const V4<double> b, double vectorx,
                                                           double vectory, double q, double g) {
    IeeeOps o;
    return spectral_radius64(o, a, b, vectorx, vectory, q, g);
}
template <>
__device__ __forceinline__ double spectral_radius<double>(const V4<double> &a, const V4<double> &b, double vectorx,
                                                         double vectory, double g) {
    FastOps o;
    const double q = vectorx * vectorx + vectory * vectory;
    const double r = spectral_radius64(o, a, b, vectorx, vectory, q, g);
    return o.bad ? spectral_radius_ieee(a, b, vectorx, vectory, q, g) : r;
}

// FP32: the same quantity with one reciprocal and fused multiply-adds.
template <>
__device__ __forceinline__ float spectral_radius<float>(const V4<float> &a, const V4<float> &b, float vectorx,
                                                       float vectory, float g) {
    const float2 s01 = __fadd2_rn(make_float2(a.x, a.y), make_float2(b.x, b.y));
    const float2 s23 = __fadd2_rn(make_float2(a.z, a.w), make_float2(b.z, b.w));
    const float rou = s01.x * 0.5f, ir = frcp(rou);
    const float u = s01.y * (0.5f * ir), v = s23.x * (0.5f * ir);
    const float EE = fmaf(s23.y * 0.5f, ir, -0.5f * fmaf(u, u, v * v));
    const float VC = fmaf(u, vectory, v * vectorx);
    const float p = rou * EE * (g - 1.0f);
    const float CS = fsqrt(g * p * ir * fmaf(vectorx, vectorx, vectory * vectory));
    return fabsf(VC) + CS;
}

// gpu_solver.cu:569-647 (kernel_ROE_SCHEME): Roe flux with Harten's entropy
// fix of width eps through the unit normal (nx, ny).
template <typename T>
__device__ V4<T> roe(const V4<T> &LW, const V4<T> &RW, T nx, T ny, T g, T epsilon);

// |v| of the Harten fix (gpu_solver.cu:603-616): (v^2 + eps^2) / (2 eps) below
// eps.
template <class O> __device__ __forceinline__ double harten(O &o, const double v, const double epsilon) {
    if (!abs_less(v, epsilon)) return fabs(v);
    return o.div(v * v + epsilon * epsilon, 2.0 * epsilon);
}

__device__ __forceinline__ double twice(double b) { return 2.0 * b; }
__device__ __forceinline__ Divisor twice(Divisor d) {  // (exponent 2046 becomes one that is not prepared)
    d.b = 2.0 * d.b;
    d.e = d.e ? d.e + 1 : 0;
    return d;
}

// Which products go to the integer units (IM, o.mul): on meshes that fill the GPU
// the FP64 pipe is the bound (81 % busy is the most seen) and the integer units
// have most of their issue slots left.  us per launch at 1.05M cells: pass A with
// none / 12 / 24 / 36 of its 68 there 281 / 261 / 256 / 261, the flux and the radii
// with 42 / 48 / 52 of the flux's 78: 406 / 413 / 419, pass C with none / 1 / 2 of 4:
// 45 / 43 / 41.  On small meshes a launch is as long as one thread's chain, which
// forty instructions for one only lengthen (8k cells: pass B 19 -> 24).
// FP64: the reference's operations in its order (calc_function,
// gpu_solver.cu:552-566, and the flux), times the face length 2 hv.  Powers of two
// move through the roundings: x - 0.5 y is one fused multiply-add (its product
// is exact), 2 AB AB is twice AB AB and shares its divisor, and the flux's
// factor 0.5 goes into the face length.
// IM: some of the products (o.mul) on the integer units.
template <bool IM, class O>
__device__ __forceinline__ V4<double> roe_scaled(O &o, const V4<double> &LW, const V4<double> &RW, const double nx,
                                                const double ny, const double g, const double epsilon,
                                                const double hv) {
    const double gm1 = g - 1.0;
    const double t0 = o.div(1.0, LW.x), t1 = o.div(1.0, RW.x);
    const double U0 = o.template mul<IM>(LW.y, t0), V0 = o.template mul<IM>(LW.z, t0), e0 = o.template mul<IM>(LW.w, t0);
    const double U1 = o.template mul<IM>(RW.y, t1), V1 = o.template mul<IM>(RW.z, t1), e1 = o.template mul<IM>(RW.w, t1);
    const double P0 = o.template mul<IM>(gm1, LW.x) * fma(-0.5, o.template mul<IM>(U0, U0) + V0 * V0, e0);
    const double P1 = o.template mul<IM>(gm1, RW.x) * fma(-0.5, o.template mul<IM>(U1, U1) + V1 * V1, e1);
    const double H0 = e0 + o.template mul<IM>(P0, t0), H1 = e1 + o.template mul<IM>(P1, t1);
    const double M0 = o.template mul<IM>(U0, nx) + V0 * ny, M1 = o.template mul<IM>(U1, nx) + V1 * ny;
    const double DVC = M1 - M0;
    const double sl = o.sqrt(LW.x), sr = o.sqrt(RW.x);
    const double ROUB = o.template mul<IM>(sl, sr);
    const auto ds = o.over(sl + sr);
    const double UB = o.by(U0 * sl + U1 * sr, ds);
    const double VB = o.by(V0 * sl + V1 * sr, ds);
    const double HB = o.by(H0 * sl + H1 * sr, ds);
    const double QB = o.template mul<IM>(UB, UB) + VB * VB;
    const double AB = o.sqrt(gm1 * fma(-0.5, QB, HB));
    const double VC = o.template mul<IM>(UB, nx) + VB * ny;
    const double AD0 = harten(o, VC - AB, epsilon), AD1 = harten(o, VC, epsilon), AD2 = harten(o, VC + AB, epsilon);
    const double dP = P1 - P0, RAD = o.template mul<IM>(ROUB, AB) * DVC;
    const double a2 = o.template mul<IM>(AB, AB);
    const auto da = o.over(a2), da2 = twice(da);
    const double F00 = o.by(o.template mul<IM>(AD0, dP - RAD), da2);
    const double F20 = o.by(o.template mul<IM>(AD2, dP + RAD), da2);
    const double F10 = AD1 * ((RW.x - LW.x) - o.by(dP, da));
    const double anx = o.template mul<IM>(AB, nx), any = o.template mul<IM>(AB, ny), avc = o.template mul<IM>(AB, VC);
    const double dU = U1 - U0, dV = V1 - V0, aR = o.template mul<IM>(AD1, ROUB);
    const double F11 = o.template mul<IM>(F10, UB) + aR * (dU - o.template mul<IM>(DVC, nx));
    const double F12 = o.template mul<IM>(F10, VB) + aR * (dV - o.template mul<IM>(DVC, ny));
    const double F13 = fma(o.template mul<IM>(F10, QB), 0.5, aR * (o.template mul<IM>(UB, dU) + VB * dV - o.template mul<IM>(DVC, VC)));
    const double WL0 = o.template mul<IM>(LW.x, M0), WR0 = o.template mul<IM>(RW.x, M1);
    V4<double> F;
    F.x = ((WL0 + WR0) - (F00 + F10 + F20)) * hv;
    F.y = ((o.template mul<IM>(U0, WL0) + o.template mul<IM>(nx, P0)) + (o.template mul<IM>(U1, WR0) + nx * P1) - (F00 * (UB - anx) + F11 + F20 * (UB + anx))) * hv;
    F.z = ((o.template mul<IM>(V0, WL0) + o.template mul<IM>(ny, P0)) + (o.template mul<IM>(V1, WR0) + ny * P1) - (F00 * (VB - any) + F12 + F20 * (VB + any))) * hv;
    F.w = ((o.template mul<IM>(WL0, H0) + o.template mul<IM>(WR0, H1)) - (F00 * (HB - avc) + F13 + F20 * (HB + avc))) * hv;
    return F;
}

// FP32: the same flux, algebraically identical, arranged for the FP32 units
// (shared reciprocals, explicit fused multiply-adds); the FP32 pass is issue
// bound, not memory bound.  Rounding differs from the generic form at FP32
// level only.
template <>
__device__ __forceinline__ V4<float> roe<float>(const V4<float> &LW, const V4<float> &RW, float nx, float ny,
                                               float g, float epsilon) {
    const float gm1 = g - 1.0f;
    // The left / right quantities as pairs on the packed FP32 units (two
    // lanes per instruction, each with the scalar form's operation order, so
    // the bits are those of the scalar expressions); one reciprocal square
    // root per density gives both its square root and its reciprocal.
    const float2 rho = make_float2(LW.x, RW.x), en = make_float2(LW.w, RW.w);
    const float2 rs = make_float2(frsqrt(LW.x), frsqrt(RW.x));
    const float2 iv = __fmul2_rn(rs, rs);
    const float2 Up = __fmul2_rn(make_float2(LW.y, RW.y), iv), Vp = __fmul2_rn(make_float2(LW.z, RW.z), iv);
    const float2 Pp = __fmul2_rn(make_float2(gm1, gm1),
                                 __ffma2_rn(__fmul2_rn(make_float2(-0.5f, -0.5f), rho),
                                            __ffma2_rn(Up, Up, __fmul2_rn(Vp, Vp)), en));
    const float2 Hp = __fmul2_rn(__fadd2_rn(en, Pp), iv);
    const float2 nx2 = make_float2(nx, nx), ny2 = make_float2(ny, ny);
    const float2 Mp = __ffma2_rn(Up, nx2, __fmul2_rn(Vp, ny2));
    const float2 sp = __fmul2_rn(rho, rs);
    const float U0 = Up.x, U1 = Up.y, V0 = Vp.x, V1 = Vp.y, P0 = Pp.x, P1 = Pp.y, H0 = Hp.x, H1 = Hp.y;
    const float M0 = Mp.x, M1 = Mp.y;
    const float DVC = M1 - M0;
    const float sl = sp.x, sr = sp.y;
    const float ROUB = sl * sr, is = frcp(sl + sr);
    const float UB = fmaf(U0, sl, U1 * sr) * is;
    const float VB = fmaf(V0, sl, V1 * sr) * is;
    const float HB = fmaf(H0, sl, H1 * sr) * is;
    const float QB = fmaf(UB, UB, VB * VB);
    // c^2 of the Roe average: AB = sqrt(c^2) and 1 / AB^2 from one rsqrt
    const float c2 = gm1 * fmaf(-0.5f, QB, HB), rc = frsqrt(c2);
    const float AB = c2 * rc;
    const float VC = fmaf(UB, nx, VB * ny);
    const float e2 = epsilon * epsilon, ie = 0.5f / epsilon;
    // the two acoustic waves (eigenvalues VC -+ AB) as a pair
    const float2 abs2 = make_float2(-AB, AB);
    const float2 lp = __fadd2_rn(make_float2(VC, VC), abs2);  // (VC - AB, VC + AB)
    const float2 lh = __fmul2_rn(__ffma2_rn(lp, lp, make_float2(e2, e2)), make_float2(ie, ie));
    const float AD0 = fabsf(lp.x) < epsilon ? lh.x : fabsf(lp.x);
    const float AD1 = fabsf(VC) < epsilon ? fmaf(VC, VC, e2) * ie : fabsf(VC);
    const float AD2 = fabsf(lp.y) < epsilon ? lh.y : fabsf(lp.y);
    const float dP = P1 - P0, ia2 = rc * rc, rad = ROUB * AB * DVC, h2 = 0.5f * ia2;
    const float2 FA = __fmul2_rn(__fmul2_rn(make_float2(AD0, AD2), __fadd2_rn(make_float2(dP, dP), make_float2(-rad, rad))),
                                 make_float2(h2, h2));  // (F00, F20)
    const float F00 = FA.x, F20 = FA.y;
    const float F10 = AD1 * fmaf(-dP, ia2, RW.x - LW.x);
    const float du = U1 - U0, dv = V1 - V0, aR = AD1 * ROUB;
    const float2 Fk1 = __fmul2_rn(FA, __ffma2_rn(abs2, nx2, make_float2(UB, UB)));  // (F01, F21)
    const float2 Fk2 = __fmul2_rn(FA, __ffma2_rn(abs2, ny2, make_float2(VB, VB)));  // (F02, F22)
    const float2 Fk3 = __fmul2_rn(FA, __ffma2_rn(abs2, make_float2(VC, VC), make_float2(HB, HB)));  // (F03, F23)
    const float F01 = Fk1.x, F21 = Fk1.y, F02 = Fk2.x, F22 = Fk2.y, F03 = Fk3.x, F23 = Fk3.y;
    const float F11 = fmaf(F10, UB, aR * fmaf(-DVC, nx, du));
    const float F12 = fmaf(F10, VB, aR * fmaf(-DVC, ny, dv));
    const float F13 = fmaf(F10 * 0.5f, QB, aR * fmaf(UB, du, fmaf(VB, dv, -DVC * VC)));
    const float2 W0 = __fmul2_rn(rho, Mp);
    const float2 W1 = __ffma2_rn(Up, W0, __fmul2_rn(nx2, Pp));
    const float2 W2 = __ffma2_rn(Vp, W0, __fmul2_rn(ny2, Pp));
    const float2 W3 = __fmul2_rn(W0, Hp);
    const float WL0 = W0.x, WR0 = W0.y, WL1 = W1.x, WR1 = W1.y, WL2 = W2.x, WR2 = W2.y, WL3 = W3.x, WR3 = W3.y;
    V4<float> F;
    F.x = 0.5f * ((WL0 + WR0) - (F00 + F10 + F20));
    F.y = 0.5f * ((WL1 + WR1) - (F01 + F11 + F21));
    F.z = 0.5f * ((WL2 + WR2) - (F02 + F12 + F22));
    F.w = 0.5f * ((WL3 + WR3) - (F03 + F13 + F23));
    return F;
}

// ---------------------------------------------------------------------------
// Pass A: gpu_solver.cu:137-223 (kernel_Boundary), 225-383 (kernel_Gradient),
// 385-454 (kernel_deltT), 456-549 (kernel_Limiter / kernel_LBJinterpolate),
// and the dt part of 768-878 (kernel_Flux_e2c).
// FS[k*n+i] receives the state on the cell's own side of face k, the limited
// reconstruction, for an interior face, and the ghost state for a boundary face
// (the reference's boundary faces are first order: the cell's own side is the
// cell state, and pass B would evaluate the ghost again from it: on small
// O-grids most warps hold a boundary cell.  us per iteration without and with
// this: FP32 2k cells in one launch 18.4 and 14.7, 131k 54.3 and 52.6, 4.2M 926 and
// 929 (pass A 76.9 and 78.1, pass B 81.5 and 79.9); FP64 33.6k cells 252 and 243).
//
// Limiter freezing (an option with no reference counterpart, off when phi is
// null): while not frozen the limiter values of every face are recorded in
// phi; once frozen they are reused instead of re-evaluated, which makes the
// residual a smooth function of the state so that it can converge below the
// limiter's chatter floor.
// Face midpoint minus cell centroid of face k.  FP64 reads the value the host
// computed with the reference's formulas (midpoint and centroid averages,
// gpu_init.cu:100-228), which keeps the FP64 parity bit for bit.  FP32
// (offset32) derives it from the face vectors already in registers instead of
// reading 24 bytes per cell: with e_j = (-S_j.y, S_j.x) the edge opposite node
// j, mid_k - centroid = (e_{k+2} - e_{k+1}) / 6 exactly.

// Cell area: FP64 reads the host value (Calc_area, gpu_init.cu:95-98); FP32
// takes half the cross product of two edge vectors, (S_1.x S_2.y - S_1.y S_2.x) / 2
// with the edges e_j = (-S_j.y, S_j.x) of a counter-clockwise cell.
template <typename T>
__device__ __forceinline__ T cell_area(const MeshDev<T> &m, const V2<T> *S, int i) {
    return m.area[i];
}
template <>
__device__ __forceinline__ float cell_area<float>(const MeshDev<float> &m, const V2<float> *S, int i) {
    return 0.5f * fmaf(S[1].x, S[2].y, -(S[1].y * S[2].x));
}

// Limiter value of one component on one face side from its reconstruction
// difference delt2: kind 0 the reference's min(1, (Umax - U) / delt2) for
// delt2 > 0, min(1, (Umin - U) / delt2) for delt2 < 0, 1 for delt2 == 0
// (gpu_solver.cu:456-494; the bound is selected first so a warp divides once
// whatever the signs of its lanes, and a NaN delt2 makes the face state NaN
// whatever the value); kind 1 the Venkatakrishnan form on the same
// differences (option).
template <typename T>
__device__ __forceinline__ T face_limiter(const int kind, const Flow<T> &f, const T A, const T umax, const T umin,
                                          const T u, const T delt2) {
    if (kind == 1) {
        const T e2 = f.venk_k3 * A * tsqrt(A);
        const T d1 = delt2 > T(0) ? umax - u : umin - u;
        return delt2 == T(0) ? T(1.0)
                             : fdiv(d1 * d1 + e2 + T(2) * delt2 * d1, d1 * d1 + T(2) * delt2 * delt2 + d1 * delt2 + e2);
    }
    const T bound = delt2 > T(0) ? umax : umin;
    return delt2 == T(0) ? T(1.0) : tmin(fdiv(bound - u, delt2), T(1.0));
}

// FP32 pass A.  The component pairs (rho, rho u) and (rho v, rho E) run on the
// packed FP32 units (two lanes per instruction, each with the scalar operation
// order): the gradient sums, the gradients, the reconstruction differences,
// the limiter quotients and the face states.

// Gradient and bounds of one cell: what its face states are reconstructed from.
struct Recon32 {
    float2 U01, U23, gxa, gxb, gya, gyb;
    float umax[4], umin[4];
};

// From the cell's state U, its face vectors S and its neighbours' (or ghost)
// states nbv; SR: also the sum of the three face spectral radii.
template <bool SR>
__device__ __forceinline__ Recon32 reconstruct32(const Flow<float> &f, const V4<float> &U, const V2<float> *S,
                                                 const V4<float> *nbv, const float A, float &Tsum) {
    Recon32 c;
    c.U01 = make_float2(U.x, U.y);
    c.U23 = make_float2(U.z, U.w);
    const float2 half = make_float2(0.5f, 0.5f);
    float2 g0a = make_float2(0.f, 0.f), g0b = g0a, g1a = g0a, g1b = g0a;
    float jmax[4], jmin[4];
    Tsum = 0.f;
#pragma unroll
    for (int k = 0; k < 3; k++) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float v = comp(nbv[k], q);
            if (k == 0) { jmax[q] = v; jmin[q] = v; }
            else {
                if (v < jmin[q]) jmin[q] = v;
                if (v > jmax[q]) jmax[q] = v;
            }
        }
        const float2 ha = __fmul2_rn(half, __fadd2_rn(c.U01, make_float2(nbv[k].x, nbv[k].y)));
        const float2 hb = __fmul2_rn(half, __fadd2_rn(c.U23, make_float2(nbv[k].z, nbv[k].w)));
        const float2 sx = make_float2(S[k].x, S[k].x), sy = make_float2(S[k].y, S[k].y);
        g0a = __ffma2_rn(ha, sx, g0a);
        g0b = __ffma2_rn(hb, sx, g0b);
        g1a = __ffma2_rn(ha, sy, g1a);
        g1b = __ffma2_rn(hb, sy, g1b);
        if (SR) Tsum += spectral_radius(U, nbv[k], S[k].y, S[k].x, f.gamma);
    }
    const float rA = fdiv(1.0f, A);
    const float2 rA2 = make_float2(rA, rA);
    c.gxa = __fmul2_rn(g0a, rA2);
    c.gxb = __fmul2_rn(g0b, rA2);
    c.gya = __fmul2_rn(g1a, rA2);
    c.gyb = __fmul2_rn(g1b, rA2);
#pragma unroll
    for (int q = 0; q < 4; q++) {
        c.umax[q] = tmax(comp(U, q), jmax[q]);
        c.umin[q] = tmin(comp(U, q), jmin[q]);
    }
    return c;
}

// How a cell limits its face states under the scheme options.
struct Limit32 {
    bool reuse;     // frozen values from phi
    bool cellwise;  // one value per cell and component (options 2, 3)
    float A;
    float phic[4];
};

// State on the cell's side of the face with midpoint offset r: the limited
// reconstruction.  ph: the limiter values (in: the frozen ones when reused).
template <bool OPT>
__device__ __forceinline__ V4<float> face_state32(const Recon32 &c, const Flow<float> &f, const Limit32 &lim,
                                                  const V2<float> r, V4<float> &ph) {
    const float2 rx = make_float2(r.x, r.x), ry = make_float2(r.y, r.y);
    const float2 da = __ffma2_rn(c.gxa, rx, __fmul2_rn(c.gya, ry));  // delt2 of components 0, 1
    const float2 db = __ffma2_rn(c.gxb, rx, __fmul2_rn(c.gyb, ry));  // and 2, 3
    float2 fa, fb;
    if (OPT && lim.reuse) {
        fa = make_float2(ph.x, ph.y);
        fb = make_float2(ph.z, ph.w);
    } else if (OPT && lim.cellwise) {
        fa = make_float2(lim.phic[0], lim.phic[1]);
        fb = make_float2(lim.phic[2], lim.phic[3]);
    } else if (OPT && f.limiter == 1) {
        fa = make_float2(face_limiter(1, f, lim.A, c.umax[0], c.umin[0], c.U01.x, da.x),
                         face_limiter(1, f, lim.A, c.umax[1], c.umin[1], c.U01.y, da.y));
        fb = make_float2(face_limiter(1, f, lim.A, c.umax[2], c.umin[2], c.U23.x, db.x),
                         face_limiter(1, f, lim.A, c.umax[3], c.umin[3], c.U23.y, db.y));
    } else {
        // limiter (kind 0): min(1, (bound - u) / delt2), bound - u as
        // u * (-1) + bound (one rounding, the same bits)
        const float2 mone = make_float2(-1.0f, -1.0f);
        const float2 na = __ffma2_rn(c.U01, mone, make_float2(da.x > 0.f ? c.umax[0] : c.umin[0],
                                                              da.y > 0.f ? c.umax[1] : c.umin[1]));
        const float2 nb = __ffma2_rn(c.U23, mone, make_float2(db.x > 0.f ? c.umax[2] : c.umin[2],
                                                              db.y > 0.f ? c.umax[3] : c.umin[3]));
        const float2 qa = __fmul2_rn(na, make_float2(frcp(da.x), frcp(da.y)));
        const float2 qb = __fmul2_rn(nb, make_float2(frcp(db.x), frcp(db.y)));
        fa = make_float2(da.x == 0.f ? 1.0f : tmin(qa.x, 1.0f), da.y == 0.f ? 1.0f : tmin(qa.y, 1.0f));
        fb = make_float2(db.x == 0.f ? 1.0f : tmin(qb.x, 1.0f), db.y == 0.f ? 1.0f : tmin(qb.y, 1.0f));
    }
    const float2 wa = __ffma2_rn(da, fa, c.U01), wb = __ffma2_rn(db, fb, c.U23);
    V4<float> o;
    o.x = wa.x; o.y = wa.y; o.z = wb.x; o.w = wb.y;
    ph.x = fa.x; ph.y = fa.y; ph.z = fb.x; ph.w = fb.y;
    if (OPT && f.positivity) {
        // positivity fallback (option): a face side with a density or
        // pressure that is not positive takes the cell state
        const float q = 0.5f * (o.y * o.y + o.z * o.z) / o.x;
        if (!(o.x > 0.f) || !((f.gamma - 1.0f) * (o.w - q) > 0.f)) {
            o.x = c.U01.x; o.y = c.U01.y; o.z = c.U23.x; o.w = c.U23.y;
        }
    }
    return o;
}

// Face offsets of a cell from its face vectors (face_offset, FP32).
__device__ __forceinline__ V2<float> offset32(const V2<float> a, const V2<float> b) {
    V2<float> r;
    r.x = (a.y - b.y) * (1.0f / 6.0f);
    r.y = (b.x - a.x) * (1.0f / 6.0f);
    return r;
}

// The limiter settings of a cell; the cell-wise options (2, 3) take the
// smallest of the per-face values (reference form, Venkatakrishnan form) of
// the cell's interior faces.
template <bool OPT>
__device__ __forceinline__ Limit32 limits32(const Recon32 &c, const Flow<float> &f, const int *code,
                                            const V2<float> *S, const float A, const bool reuse, const bool first) {
    Limit32 lim;
    lim.reuse = reuse;
    lim.cellwise = OPT && f.limiter >= 2;
    lim.A = A;
    if (lim.cellwise && !reuse && !first) {
#pragma unroll
        for (int q = 0; q < 4; q++) lim.phic[q] = INFINITY;
        const float2 u[2] = {c.U01, c.U23};
#pragma unroll
        for (int k = 0; k < 3; k++) {
            if (code[k] < 0) continue;
            const V2<float> r = offset32(S[(k + 1) % 3], S[(k + 2) % 3]);
            const float2 rx = make_float2(r.x, r.x), ry = make_float2(r.y, r.y);
            const float2 d[2] = {__ffma2_rn(c.gxa, rx, __fmul2_rn(c.gya, ry)),
                                 __ffma2_rn(c.gxb, rx, __fmul2_rn(c.gyb, ry))};
#pragma unroll
            for (int q = 0; q < 4; q++)
                lim.phic[q] = tmin(lim.phic[q],
                                   face_limiter(f.limiter - 2, f, A, c.umax[q], c.umin[q],
                                                q & 1 ? u[q >> 1].y : u[q >> 1].x, q & 1 ? d[q >> 1].y : d[q >> 1].x));
        }
    }
    return lim;
}

// Pass A of one cell from its neighbours' (or ghost) states: the states of its
// interior faces go to out(k, state), its local time step is returned.  (On a
// boundary face the cell's side is the cell state itself; what pass B needs
// there is the ghost, which the caller leaves in the face's place.)  OPT compiles in
// the scheme options (smooth limiter, frozen limiter values, first-order faces,
// positivity fallback); without them the reference configuration runs in fewer
// registers.  first: this iteration uses first-order faces.  Without the options a
// boundary face's state is evaluated like the others and only not stored: with a
// branch around each face the launch spilled 32 bytes per thread instead of 20 (12
// instead of none in a batch) and took 80.2 instead of 78.1 us at 4.2M cells (an
// iteration 937 and 929 us, of 60 batched cases 480 and 473).
template <bool OPT, typename Out>
__device__ __forceinline__ float faces_cell32(const MeshDev<float> &m, const Flow<float> &f, const int i,
                                              const int *code, const V2<float> *S, const V4<float> &U,
                                              const V4<float> *nbv, V4<float> *__restrict__ phi, const int frozen,
                                              const bool first, Out out) {
    const int n = m.n;
    const float A = cell_area(m, S, i);
    float Tsum;
    const Recon32 c = reconstruct32<true>(f, U, S, nbv, A, Tsum);
    const bool reuse = OPT && phi && frozen;
    const Limit32 lim = limits32<OPT>(c, f, code, S, A, reuse, first);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (OPT && code[k] < 0) continue;
        V4<float> o = U;
        if (!(OPT && first)) {
            V4<float> ph;
            if (reuse) ph = phi[k * n + i];
            o = face_state32<OPT>(c, f, lim, offset32(S[(k + 1) % 3], S[(k + 2) % 3]), ph);
            if (OPT && phi && !frozen) phi[k * n + i] = ph;
        }
        if (code[k] >= 0) out(k, o);
    }
    return tmin(fdiv(A * f.cfl, Tsum), f.dt_cap);
}

// The same from global memory; the face states go to FS, the step to dt[i].
template <bool OPT>
__device__ __forceinline__ float faces_cell(const MeshDev<float> &m, const Flow<float> &f, const int i,
                                            const V4<float> *__restrict__ W, V4<float> *__restrict__ FS,
                                            float *__restrict__ dt, V4<float> *__restrict__ phi, const int frozen,
                                            const bool first, const int4 tp) {
    const int n = m.n;
    const int code[3] = {tp.x, tp.y, tp.z};
    const V4<float> U = W[i];
    V2<float> S[3];
#pragma unroll
    for (int k = 0; k < 3; k++) S[k] = m.S[k * n + i];
    V4<float> nbv[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (code[k] >= 0) nbv[k] = W[code[k] >> 3];
        else FS[k * n + i] = nbv[k] = ghost(code[k], U, S[k].x, S[k].y, f);
    }
    const float dti = faces_cell32<OPT>(m, f, i, code, S, U, nbv, phi, frozen, first,
                                        [&](int k, const V4<float> &o) { FS[k * n + i] = o; });
    dt[i] = dti;
    return dti;
}

// Bounds of component values over a cell and its neighbours, minus the cell's
// own value: x = max - u, y = min - u (gpu_solver.cu:330-375), ordered on
// integer keys.  (A NaN among them makes the gradient, and with it the
// component's face states, NaN whatever the bounds.)
__device__ __forceinline__ double2 cell_bounds(const double c0, const double c1, const double c2, const double u) {
    const int64_t k0 = order_key(c0), k1 = order_key(c1), k2 = order_key(c2), ku = order_key(u);
    const int64_t a = k0 > k1 ? k0 : k1, b = k2 > ku ? k2 : ku, c = k0 < k1 ? k0 : k1, d = k2 < ku ? k2 : ku;
    return make_double2(key_value(a > b ? a : b) - u, key_value(c < d ? c : d) - u);
}

// Limiter value of one component on one face side (face_limiter) in FP64, from
// the bounds minus the cell value.  Kind 0, min(1, bound / delt2): the bound
// has delt2's sign, so a correctly rounded quotient of |bound| >= |delt2| is
// >= 1 and only smaller bounds divide.  Kind 1, the Venkatakrishnan form with
// its doubled products as exact fused multiply-adds.
template <class O>
__device__ __forceinline__ double face_limiter64(O &o, const int kind, const double e2, const double2 bnd,
                                                 const double delt2) {
    const double d1 = (int64_t)bits_of(delt2) > 0 ? bnd.x : bnd.y;
    if (kind == 1) {
        if (delt2 == 0.0) return 1.0;
        const double q = d1 * d1, p = delt2 * d1;
        return o.div(fma(2.0, p, q + e2), fma(2.0, delt2 * delt2, q) + p + e2);
    }
    const bool need = abs_less(d1, delt2);  // else a quotient of at least 1 (or of 0 by 0)
    const double q = o.div(d1, need ? delt2 : 1.0);
    return need ? q : 1.0;
}

// The face states of the FP64 form of faces_cell, by LPC lanes per cell: lane part
// takes the NQ = 4 / LPC components from part NQ on.  It issues about 160 FP64 additions and
// multiplications per cell in the reference configuration: the reference's
// halves of the neighbour means are taken into the face vectors (exact), the
// first term of a sum is not added to zero, the bounds are subtracted once per
// component and divisions, comparisons and selections run on the integer units.
// gs: the ghost states of the cell's boundary faces, gstep apart.
// IM: 24 of the 68 products on the integer units (see roe_scaled).
template <bool OPT, int LPC, bool IM, class O>
__device__ __forceinline__ void faces_cell64(O &o, const MeshDev<double> &m, const Flow<double> &f, const int i,
                                               const int part, const V4<double> *__restrict__ W,
                                               V4<double> *FS, V4<double> *__restrict__ phi, const int frozen,
                                               const bool first, const V4<double> *__restrict__ Uc, const int4 tp,
                                               const V4<double> *gs, const int gstep) {
    constexpr int NQ = 4 / LPC;
    const int n = m.n, q0 = part * NQ;
    const int code[3] = {tp.x, tp.y, tp.z};
    auto values = [&](const V4<double> *p, double *v) {
        const double *d = reinterpret_cast<const double *>(p) + q0;
#pragma unroll
        for (int q = 0; q < NQ; q++) v[q] = d[q];
    };
    auto store = [&](V4<double> *p, const double *v) {
        double *d = reinterpret_cast<double *>(p) + q0;
#pragma unroll
        for (int q = 0; q < NQ; q++) d[q] = v[q];
    };
    V2<double> h[3];  // halves of the face vectors
    double u[NQ], nb[3][NQ];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const V2<double> S = m.S[k * n + i];
        h[k].x = o.half(S.x);
        h[k].y = o.half(S.y);
        values(code[k] >= 0 ? W + (code[k] >> 3) : gs + k * gstep, nb[k]);
    }
    values(Uc, u);
    const double A = m.area[i];
    const double rA = o.div(1.0, A);
    double gx[NQ], gy[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const double s = u[q] + nb[k][q];
            const double px = o.template mul<IM>(s, h[k].x), py = s * h[k].y;
            gx[q] = k == 0 ? px : gx[q] + px;
            gy[q] = k == 0 ? py : gy[q] + py;
        }
        gx[q] *= rA;
        gy[q] *= rA;
    }
    const bool reuse = OPT && phi && frozen;
    double2 bnd[NQ];
    if (!reuse && !(OPT && first)) {
#pragma unroll
        for (int q = 0; q < NQ; q++) bnd[q] = cell_bounds(nb[0][q], nb[1][q], nb[2][q], u[q]);
    }
    const int kind = OPT ? f.limiter & 1 : 0;
    const double e2 = OPT && kind == 1 && !reuse ? f.venk_k3 * A * o.sqrt(A) : 0.0;
    // cell-wise limiter options (2, 3): see limits32
    const bool cellwise = OPT && f.limiter >= 2;
    double phic[NQ];
    if (cellwise && !reuse && !first) {
#pragma unroll
        for (int q = 0; q < NQ; q++) phic[q] = (double)INFINITY;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            if (code[k] < 0) continue;
            const V2<double> r = m.R[k * n + i];
#pragma unroll
            for (int q = 0; q < NQ; q++)
                phic[q] = fmin(phic[q], face_limiter64(o, kind, e2, bnd[q], o.template mul<IM>(gx[q], r.x) + gy[q] * r.y));
        }
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        double d[NQ];
        if (!(OPT && first)) {
            const V2<double> r = m.R[k * n + i];
            double ph[NQ];
            if (reuse) values(phi + k * n + i, ph);
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                const double delt2 = o.template mul<IM>(gx[q], r.x) + gy[q] * r.y;
                if (cellwise && !reuse) ph[q] = phic[q];
                else if (!reuse) ph[q] = face_limiter64(o, kind, e2, bnd[q], delt2);
                d[q] = delt2 * ph[q] + u[q];
            }
            if constexpr (OPT && LPC == 1)
                if (f.positivity) {
                    // positivity fallback (option): see face_state32
                    const double q = o.div(0.5 * (d[1] * d[1] + d[2] * d[2]), d[0]);
                    if (!(d[0] > 0.0) || !((f.gamma - 1.0) * (d[3] - q) > 0.0))
                        for (int c = 0; c < 4; c++) d[c] = u[c];
                }
            if (OPT && phi && !frozen && code[k] >= 0) store(phi + k * n + i, ph);
        } else {
#pragma unroll
            for (int q = 0; q < NQ; q++) d[q] = u[q];
        }
        // a boundary face's place takes the ghost (for pass B)
#pragma unroll
        for (int q = 0; q < NQ; q++) d[q] = code[k] < 0 ? nb[k][q] : d[q];
        store(FS + k * n + i, d);
    }
}

template <bool OPT, int LPC>
static __device__ __noinline__ void faces_cell64_ieee(const MeshDev<double> m, const Flow<double> f, const int i,
                                                      const int part, const V4<double> *W, V4<double> *FS,
                                                      V4<double> *phi, const int frozen, const bool first,
                                                      const V4<double> *Uc, const int4 tp, const V4<double> *gs,
                                                      const int gstep) {
    IeeeOps o;
    faces_cell64<OPT, LPC, false>(o, m, f, i, part, W, FS, phi, frozen, first, Uc, tp, gs, gstep);
}
template <bool OPT, int LPC, bool IM = (LPC < 4)>
__device__ __forceinline__ void faces_cell64(const MeshDev<double> &m, const Flow<double> &f, const int i,
                                             const int part, const V4<double> *__restrict__ W, V4<double> *FS,
                                             V4<double> *__restrict__ phi, const int frozen, const bool first,
                                             const V4<double> *__restrict__ Uc, const int4 tp, const V4<double> *gs,
                                             const int gstep) {
    FastOps o;
    faces_cell64<OPT, LPC, IM>(o, m, f, i, part, W, FS, phi, frozen, first, Uc, tp, gs, gstep);
    if (o.bad) faces_cell64_ieee<OPT, LPC>(m, f, i, part, W, FS, phi, frozen, first, Uc, tp, gs, gstep);
}

// Local time step of a cell from the sum of its faces' spectral radii.
__device__ __forceinline__ double local_dt(const MeshDev<double> &m, const Flow<double> &f, const int i,
                                           const double Tsum) {
    return tmin(ddiv(m.area[i] * f.cfl, Tsum), f.dt_cap);
}

// Pass A in FP64 for one tile of cells [base, base + nvalid), nvalid <=
// blockDim.x / LPC, each interior face's spectral radius evaluated once: the tile
// lists the radii it must evaluate (boundary faces, faces to cells outside the
// tile, and inside faces from their left cell only, as flux_tile does for the
// Roe flux), spreads that list over its threads with the cell states in shared
// memory (boundary faces leave their ghost states there), then every cell sums
// its three radii in face order and LPC lanes run faces_cell64.  The radius is
// symmetric in its two states and in the sign of the face vector, and the two
// cells of a face hold exactly negated face vectors, so each cell gets the bits
// of its own evaluation.  Returns the cell's time step (+inf for other lanes).
// LPC 2 and 4 shorten the chain of a thread where a mesh leaves the GPU's
// schedulers with few warps (faces_lanes).
struct FacesSmem {
    V4<double> *Us, *Gs;    // [cells] states, [3 cells] ghost states
    double *SRs;            // [3 cells] spectral radii
    int4 *tps;              // [cells] face codes
    unsigned short *items;  // [3 cells] radii to evaluate
    static constexpr size_t per_cell = 4 * sizeof(V4<double>) + 3 * sizeof(double) + sizeof(int4) + 3 * sizeof(unsigned short);
    __device__ __forceinline__ FacesSmem(unsigned char *p, int cells)
        : Us(reinterpret_cast<V4<double> *>(p)), Gs(Us + cells), SRs(reinterpret_cast<double *>(Gs + 3 * cells)),
          tps(reinterpret_cast<int4 *>(SRs + 3 * cells)), items(reinterpret_cast<unsigned short *>(tps + cells)) {}
};
template <bool OPT, int LPC>
__device__ __forceinline__ double faces_tile(const MeshDev<double> &m, const Flow<double> &f, const int base,
                                             const int nvalid, const V4<double> *__restrict__ W,
                                             V4<double> *__restrict__ FS, double *__restrict__ dt,
                                             V4<double> *__restrict__ phi, const int frozen, const bool first,
                                             unsigned char *smem) {
    using T = double;
    __shared__ int wtot[8];
    const FacesSmem sm(smem, blockDim.x / LPC);
    V4<T> *Us = sm.Us, *Gs = sm.Gs;
    T *SRs = sm.SRs;
    int4 *tps = sm.tps;
    unsigned short *items = sm.items;
    const int n = m.n, t = threadIdx.x;
    const bool owner = t < nvalid;
    __syncthreads();  // the previous tile of this block may still read the shared arrays
    unsigned mask = 0;
    if (owner) {
        const int4 tp = m.topo[base + t];
        tps[t] = tp;
        Us[t] = W[base + t];
        const int code[3] = {tp.x, tp.y, tp.z};
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const int c = code[k];
            const bool inside = c >= 0 && (unsigned)((c >> 3) - base) < (unsigned)nvalid;
            if (!inside || !((c >> 2) & 1)) mask |= 1u << k;
        }
    }
    // exclusive prefix sum of the per-cell counts over the block
    const int cnt = __popc(mask), lane = t & 31, wid = t >> 5;
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) wtot[wid] = incl;
    __syncthreads();
    int off = incl - cnt, total = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
        if (w < wid) off += wtot[w];
        total += wtot[w];
    }
#pragma unroll
    for (int k = 0; k < 3; k++)
        if (mask & (1u << k)) items[off++] = (unsigned short)((t << 2) | k);
    __syncthreads();
    for (int j = t; j < total; j += blockDim.x) {
        const int it = items[j], tt = it >> 2, k = it & 3;
        const int4 q = tps[tt];
        const int c = k == 0 ? q.x : k == 1 ? q.y : q.z;
        const V4<T> Uo = Us[tt];
        const V2<T> S = m.S[k * n + base + tt];
        V4<T> nb;
        if (c >= 0) {
            const int nj = c >> 3;
            nb = (unsigned)(nj - base) < (unsigned)nvalid ? Us[nj - base] : W[nj];
        } else {
            nb = ghost(c, Uo, S.x, S.y, f);
            Gs[tt * 3 + k] = nb;
        }
        SRs[tt * 3 + k] = spectral_radius(Uo, nb, S.y, S.x, f.gamma);
    }
    __syncthreads();
    const int tt = t / LPC;
    if (tt >= nvalid) return (double)INFINITY;
    const int4 tp = tps[tt];
    const int code[3] = {tp.x, tp.y, tp.z};
    T Tsum = T(0);
    if (t % LPC == 0) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            // an inside face of which the cell is the right one: its left cell has it
            const int c = code[k], q = (c >> 3) - base;
            const bool other = c >= 0 && (unsigned)q < (unsigned)nvalid && ((c >> 2) & 1);
            const T r = other ? SRs[q * 3 + (c & 3)] : SRs[tt * 3 + k];
            Tsum = k == 0 ? r : Tsum + r;
        }
    }
    faces_cell64<OPT, LPC>(m, f, base + tt, t % LPC, W, FS, phi, frozen, first, Us + tt, tp, Gs + tt * 3, 1);
    if (t % LPC != 0) return (double)INFINITY;
    return dt[base + tt] = local_dt(m, f, base + tt, Tsum);
}

// Global time-step option: the block's smallest step folded into *slot.
// Every thread of the block must call it (v = +inf for no cell).  A time
// step is non-negative, so its bits order like the integers and min over
// them is exact and independent of the order of the blocks.
__device__ __forceinline__ void block_min_dt(double v, unsigned long long *slot) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_down_sync(0xffffffffu, v, o));
    __shared__ double wm[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();  // wm may still be read by the previous use in this block
    if (lane == 0) wm[wid] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = wm[0];
        for (int k = 1; k < (int)(blockDim.x >> 5); k++) b = fmin(b, wm[k]);
        atomicMin(slot, (unsigned long long)__double_as_longlong(b));
    }
}

// FP64: pass A in tiles of blockDim.x / LPC cells (faces_tile).
template <bool OPT, int LPC>
__global__ void __launch_bounds__(256, 2) k_faces_tile(MeshDev<double> m, Flow<double> f,
                                                       const V4<double> *__restrict__ W,
                                                       V4<double> *__restrict__ FS, double *__restrict__ dt,
                                                       Ctl *__restrict__ ctl, V4<double> *__restrict__ phi,
                                                       const int st) {
    extern __shared__ __align__(32) unsigned char smem[];
    wait_prior_grid();
    if (ctl->halt) return;
    const int tile = blockDim.x / LPC, base = blockIdx.x * tile;
    const double v = faces_tile<OPT, LPC>(m, f, base, min(tile, m.n - base), W, FS, dt, phi,
                                          OPT && phi ? ctl->frozen : 0, OPT && ctl->step < f.first_order, smem);
    if (OPT && f.global_dt) block_min_dt(v, &ctl->dtmin[st]);
}

// FP64 with a face list: the face states only, LPC threads per cell without tiles;
// the radii are taken with the fluxes (k_face_flux) and the steps with their sums.
// Every thread of the warp calls it (live: it has a cell).
template <bool OPT, int LPC>
__device__ __forceinline__ void faces_listed(const MeshDev<double> &m, const Flow<double> &f, const int i,
                                             const int part, const bool live, const int4 tp,
                                             const V4<double> *__restrict__ W, V4<double> *FS,
                                             V4<double> *__restrict__ phi, const int frozen, const bool first) {
    const int n = m.n;
    if (live && (tp.x | tp.y | tp.z) < 0 && part == 0) {
#pragma unroll 1
        for (int k = 0; k < 3; k++) {
            const int c = k == 0 ? tp.x : k == 1 ? tp.y : tp.z;
            const V2<double> S = m.S[k * n + i];
            if (c < 0) FS[k * n + i] = ghost(c, W[i], S.x, S.y, f);
        }
    }
    if (LPC > 1) __syncwarp();  // the cell's other threads read the ghosts
    if (live) faces_cell64<OPT, LPC>(m, f, i, part, W, FS, phi, frozen, first, W + i, tp, FS + i, n);
}
template <bool OPT, int LPC>
__global__ void __launch_bounds__(256, 2) k_faces_cells(MeshDev<double> m, Flow<double> f,
                                                        const V4<double> *__restrict__ W, V4<double> *FS,
                                                        const Ctl *__restrict__ ctl, V4<double> *__restrict__ phi) {
    wait_prior_grid();
    if (ctl->halt) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x, i = t / LPC;
    const bool live = i < m.n;
    faces_listed<OPT, LPC>(m, f, i, t % LPC, live, live ? m.topo[i] : make_int4(0, 0, 0, 0), W, FS, phi,
                           OPT && phi ? ctl->frozen : 0, OPT && ctl->step < f.first_order);
}

// FP32.  OPT: the variant with the scheme options (smooth limiter, limiter
// freezing, global time step); faces_options picks it.
template <typename T, bool OPT>
__global__ void __launch_bounds__(256, OPT ? kOptBlocks : MinBlocks<T>::faces) k_faces(MeshDev<T> m, Flow<T> f, const V4<T> *__restrict__ W,
                                     V4<T> *__restrict__ FS, T *__restrict__ dt,
                                     Ctl *__restrict__ ctl, V4<T> *__restrict__ phi, const int st) {
    wait_prior_grid();
    if (ctl->halt) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool first = OPT && ctl->step < f.first_order;
    if (!OPT || !f.global_dt) {
        if (i >= m.n) return;
        faces_cell<OPT>(m, f, i, W, FS, dt, phi, OPT && phi ? ctl->frozen : 0, first, m.topo[i]);
        return;
    }
    double v = __longlong_as_double((long long)kDtNone);
    if (i < m.n) v = (double)faces_cell<OPT>(m, f, i, W, FS, dt, phi, phi ? ctl->frozen : 0, first, m.topo[i]);
    block_min_dt(v, &ctl->dtmin[st]);
}

// The FP64 pass-A kernel, in tiles and with a face list.
inline auto faces_tile_kernel(bool opt, int lanes) {
    if (lanes == 4) return opt ? &k_faces_tile<true, 4> : &k_faces_tile<false, 4>;
    if (lanes == 2) return opt ? &k_faces_tile<true, 2> : &k_faces_tile<false, 2>;
    return opt ? &k_faces_tile<true, 1> : &k_faces_tile<false, 1>;
}
inline auto faces_cells_kernel(bool opt, int lanes) {
    if (lanes == 4) return opt ? &k_faces_cells<true, 4> : &k_faces_cells<false, 4>;
    if (lanes == 2) return opt ? &k_faces_cells<true, 2> : &k_faces_cells<false, 2>;
    return opt ? &k_faces_cells<true, 1> : &k_faces_cells<false, 1>;
}

// True when a pass-A launch needs the option variant.
template <typename T> inline bool faces_options(const Flow<T> &f, const void *phi) {
    return phi != nullptr || f.limiter != 0 || f.global_dt != 0 || f.first_order > 0 || f.positivity != 0;
}

// Time step of cell i in RK stage st: its own, or with the global option the
// smallest of its case.
template <typename T>
__device__ __forceinline__ T stage_dt(const Flow<T> &f, const Ctl *ctl, const int st, const T *dt, const int i) {
    return f.global_dt ? (T)__longlong_as_double((long long)ctl->dtmin[st]) : dt[i];
}

// ---------------------------------------------------------------------------
// Pass B: gpu_solver.cu:651-764 (kernel_Flux2) evaluated per cell for its
// three faces, summed as gpu_solver.cu:798-825 (+F where the cell is the
// edge's left cell, -F where it is the right cell, in face order).
template <typename T>
__device__ __forceinline__ void add_flux(V4<T> &r, const V4<T> &F, const bool right) {
    if constexpr (sizeof(T) == 4) {
        // r +- F as r + (+-1) F: the product is exact, one rounding, the
        // same bits as the add or subtract; two packed instructions
        const float sg = right ? -1.0f : 1.0f;
        const float2 xy = __ffma2_rn(make_float2(F.x, F.y), make_float2(sg, sg), make_float2(r.x, r.y));
        const float2 zw = __ffma2_rn(make_float2(F.z, F.w), make_float2(sg, sg), make_float2(r.z, r.w));
        r.x = xy.x; r.y = xy.y; r.z = zw.x; r.w = zw.y;
    } else {
        // the sign on the integer units: r - F as r + (-F), one addition for a
        // warp whose lanes differ (1.05M cells: k_face_sum 61 -> 38 us)
        const uint64_t sg = right ? 0x8000000000000000ULL : 0;
        r.x += double_of(bits_of(F.x) ^ sg); r.y += double_of(bits_of(F.y) ^ sg);
        r.z += double_of(bits_of(F.z) ^ sg); r.w += double_of(bits_of(F.w) ^ sg);
    }
}

template <typename T>
__device__ __forceinline__ void flux_cell(const MeshDev<T> &m, const Flow<T> &f, const int i,
                                          const V4<T> *__restrict__ W, const V4<T> *__restrict__ FS,
                                          V4<T> *__restrict__ res, const int4 tp) {
    const int n = m.n;
    const int code[3] = {tp.x, tp.y, tp.z};
    V4<T> r;
    r.x = T(0.0); r.y = T(0.0); r.z = T(0.0); r.w = T(0.0);
    // every input of the three faces is requested before the first flux
    V2<T> S[3];
    V4<T> own[3], oth[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        S[k] = m.S[k * n + i];
        own[k] = code[k] >= 0 ? FS[k * n + i] : W[i];
        oth[k] = FS[code[k] >= 0 ? (code[k] & 3) * n + (code[k] >> 3) : k * n + i];
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        bool right;
        const V4<T> F = face_flux_of(f, code[k], S[k], own[k], oth[k], right);
        add_flux(r, F, right);
    }
    res[i] = r;
}

// Length vn of the face vector S and the unit normal S / vn: IEEE in FP64; in
// FP32 from one reciprocal square root of |S|^2 (the other cell of the face,
// with S negated, gets the exact negative).
template <class O>
__device__ __forceinline__ void unit_normal(O &o, const V2<double> S, double &nx, double &ny, double &vn) {
    vn = o.sqrt(S.y * S.y + S.x * S.x);
    const auto by = o.over(vn);
    nx = o.by(S.x, by);
    ny = o.by(S.y, by);
}
__device__ __forceinline__ void unit_normal(Ops32 &, const V2<float> S, float &nx, float &ny, float &vn) {
    const float q = fmaf(S.y, S.y, S.x * S.x), r = frsqrt(q);
    vn = q * r;
    const float2 nn = __fmul2_rn(make_float2(S.x, S.y), make_float2(r, r));
    nx = nn.x;
    ny = nn.y;
}

// Inputs of the Roe flux of one face in the edge's orientation: left state a,
// right state b (oth: the neighbour's side, the ghost of a boundary face), unit normal (nx, ny) of
// the edge and the face length vn; *right tells whether the cell is the
// edge's right cell.
template <typename T, class O>
__device__ __forceinline__ void face_inputs(O &o, const int code, const V2<T> S, const V4<T> own, const V4<T> oth, V4<T> &a,
                                            V4<T> &b, T &nx, T &ny, T &vn, bool &right) {
    unit_normal(o, S, nx, ny, vn);
    // the left state first: both cells of a face run the same instructions on
    // the same inputs (their normals are exact negatives), so they get the
    // same bits
    a = own;
    b = oth;
    right = code >= 0 && ((code >> 2) & 1);
    if (right) { a = oth; b = own; nx = -nx; ny = -ny; }
}

// Flux of face k of cell i, times |S|, in the edge's orientation (the
// reference's Res_e.left of gpu_solver.cu:738-745); *right tells whether cell
// i is the edge's right cell.
__device__ __forceinline__ V4<float> face_flux_of(const Flow<float> &f, const int code, const V2<float> S,
                                                  const V4<float> own, const V4<float> oth, bool &right) {
    Ops32 o;
    V4<float> a, b;
    float nx, ny, vn;
    face_inputs(o, code, S, own, oth, a, b, nx, ny, vn, right);
    V4<float> F = roe(a, b, nx, ny, f.gamma, f.eps_entropy);
    // two packed multiplies, the same products
    const float2 xy = __fmul2_rn(make_float2(F.x, F.y), make_float2(vn, vn));
    const float2 zw = __fmul2_rn(make_float2(F.z, F.w), make_float2(vn, vn));
    F.x = xy.x; F.y = xy.y; F.z = zw.x; F.w = zw.y;
    return F;
}

// The same in FP64, from global memory.
template <bool IM, class O>
__device__ __forceinline__ V4<double> face_flux64(O &o, const MeshDev<double> &m, const Flow<double> &f, const int i,
                                                  const int k, const int code, const V4<double> *W,
                                                  const V4<double> *FS) {
    const int n = m.n;
    const V2<double> S = m.S[k * n + i];
    const V4<double> own = code >= 0 ? FS[k * n + i] : W[i];
    const V4<double> oth = code >= 0 ? FS[(code & 3) * n + (code >> 3)] : FS[k * n + i];
    V4<double> a, b;
    double nx, ny, vn;
    bool right;
    face_inputs(o, code, S, own, oth, a, b, nx, ny, vn, right);
    return roe_scaled<IM>(o, a, b, nx, ny, f.gamma, f.eps_entropy, 0.5 * vn);
}
static __device__ __noinline__ V4<double> face_flux_ieee(const MeshDev<double> m, const Flow<double> f, const int i,
                                                         const int k, const int code, const V4<double> *W,
                                                         const V4<double> *FS) {
    IeeeOps o;
    return face_flux64<false>(o, m, f, i, k, code, W, FS);
}

// Pass B for one tile of cells [base, base + nvalid) with each interior face
// inside the tile evaluated once: the tile lists the faces it must evaluate
// (boundary faces, faces to cells outside the tile, and inside faces from
// their left cell only), spreads that list over its threads, keeps the
// fluxes in shared memory, and then every cell sums its three faces in face
// order with the reference's signs.  The fluxes are the same bits as in
// flux_cell and are summed in the same order.  nvalid <= blockDim.x / R,
// blockDim.x <= 256: with R = 2 the list (about 1.7 faces per cell) takes the
// threads once instead of twice.
template <typename T, int R = 1, bool IM = true>
__device__ __forceinline__ void flux_tile(const MeshDev<T> &m, const Flow<T> &f, const int base, const int nvalid,
                                          const V4<T> *__restrict__ W, const V4<T> *__restrict__ FS,
                                          V4<T> *__restrict__ res) {
    constexpr int CELLS = 256 / R;
    __shared__ V4<T> Fs[CELLS * 3];
    __shared__ int4 tps[CELLS];
    __shared__ unsigned short items[CELLS * 3];
    __shared__ int wtot[8];
    const int t = threadIdx.x, i = base + t;
    const bool live = t < nvalid;
    const int4 tp = live ? m.topo[i] : make_int4(-3, -3, -3, 0);
    if (live) tps[t] = tp;
    const int code[3] = {tp.x, tp.y, tp.z};
    unsigned mask = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (!live) continue;
        const int c = code[k];
        if (c < 0) { mask |= 1u << k; continue; }
        const bool inside = (unsigned)((c >> 3) - base) < (unsigned)nvalid;
        if (!inside || !((c >> 2) & 1)) mask |= 1u << k;
    }
    // exclusive prefix sum of the per-cell counts over the block
    const int cnt = __popc(mask), lane = t & 31, wid = t >> 5;
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) wtot[wid] = incl;
    __syncthreads();
    int off = incl - cnt, total = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
        if (w < wid) off += wtot[w];
        total += wtot[w];
    }
#pragma unroll
    for (int k = 0; k < 3; k++)
        if (mask & (1u << k)) items[off++] = (unsigned short)((t << 2) | k);
    __syncthreads();
    for (int j = t; j < total; j += blockDim.x) {
        const int it = items[j], tt = it >> 2, k = it & 3;
        const int4 q = tps[tt];
        const int c = k == 0 ? q.x : k == 1 ? q.y : q.z;
        FastOps o;
        V4<T> F = face_flux64<IM>(o, m, f, base + tt, k, c, W, FS);
        if (o.bad) F = face_flux_ieee(m, f, base + tt, k, c, W, FS);
        Fs[tt * 3 + k] = F;
    }
    __syncthreads();
    if (!live) return;
    V4<T> r;
    r.x = T(0.0); r.y = T(0.0); r.z = T(0.0); r.w = T(0.0);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int c = code[k];
        V4<T> F;
        bool right;
        if (mask & (1u << k)) {
            F = Fs[t * 3 + k];
            right = c >= 0 && ((c >> 2) & 1);
        } else {  // inside face evaluated by its left cell
            F = Fs[((c >> 3) - base) * 3 + (c & 3)];
            right = true;
        }
        add_flux(r, F, right);
    }
    res[i] = r;
}

template <typename T>
__global__ void E2D_LB_FLUX k_flux_tile(MeshDev<T> m, Flow<T> f, const V4<T> *__restrict__ W,
                                        const V4<T> *__restrict__ FS,
                                        V4<T> *__restrict__ res, const Ctl *__restrict__ ctl) {
    wait_prior_grid();
    if (ctl->halt) return;
    const int tile = blockDim.x / 2, base = blockIdx.x * tile;
    flux_tile<T, 2, false>(m, f, base, min(tile, m.n - base), W, FS, res);
}

template <typename T>
__global__ void E2D_LB_FLUX k_flux(MeshDev<T> m, Flow<T> f, const V4<T> *__restrict__ W,
                                   const V4<T> *__restrict__ FS,
                                   V4<T> *__restrict__ res, const Ctl *__restrict__ ctl) {
    wait_prior_grid();
    if (ctl->halt) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.n) return;
    flux_cell(m, f, i, W, FS, res, m.topo[i]);
}

// Pass B in FP64 with a face list, in two launches.  First every face once, one
// thread each: its spectral radius, and its flux, which takes the place of the
// left cell's side in FS (a face's two sides are read by its thread alone).  Then
// every cell sums its three in face order with the reference's signs.  Same bits as
// flux_tile and faces_tile, whose tiles of 128 cells evaluate 1.75 rounds of
// faces per warp of cells (faces between tiles twice, the last round partly filled)
// and wait for their slowest warp; this is 1.5, without barriers, and the
// normals are the list's.  1.05M cells, when it was introduced: pass A 401 ->
// 301 us, pass B 527 -> 480.
template <typename T> __global__ void __launch_bounds__(256) k_face_geometry(const V2<T> *__restrict__ S, FaceList l) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= l.count) return;
    const V2<T> v = S[l.at[j].x];
    T nx, ny, vn;
    IeeeOps o;
    unit_normal(o, v, nx, ny, vn);
    const T g[6] = {nx, ny, 0.5 * vn, v.x, v.y, v.y * v.y + v.x * v.x};
    for (int k = 0; k < 6; k++) l.geo[(size_t)k * l.count + j] = g[k];
}

template <bool IM, class O>
__device__ __forceinline__ V4<double> listed_face(O &o, const FaceList &l, const Flow<double> &f, const int j,
                                                  const int4 at, const V4<double> *W, const V4<double> *FS,
                                                  double &radius) {
    const double *g = l.geo + j;
    const size_t nf = l.count;
    const bool inner = at.y >= 0;
    const V4<double> Wa = W[at.z], b = FS[inner ? at.y : at.x], a = inner ? FS[at.x] : Wa;
    radius = spectral_radius64(o, Wa, inner ? W[at.w] : b, g[4 * nf], g[3 * nf], g[5 * nf], f.gamma);
    return roe_scaled<IM>(o, a, b, g[0], g[nf], f.gamma, f.eps_entropy, g[2 * nf]);
}
static __device__ __noinline__ V4<double> listed_face_ieee(const FaceList l, const Flow<double> f, const int j,
                                                           const V4<double> *W, const V4<double> *FS) {
    IeeeOps o;
    double r;
    const int4 at = l.at[j];
    const V4<double> F = listed_face<false>(o, l, f, j, at, W, FS, r);
    l.radius[at.x] = r;
    return F;
}
__device__ __forceinline__ void face_listed(const FaceList &l, const Flow<double> &f, const int j, const int4 at,
                                            const V4<double> *__restrict__ W, V4<double> *FS) {
    FastOps o;
    double r;
    V4<double> F = listed_face<true>(o, l, f, j, at, W, FS, r);
    l.radius[at.x] = r;
    if (o.bad) F = listed_face_ieee(l, f, j, W, FS);
    FS[at.x] = F;
}
template <typename T>
__global__ void __launch_bounds__(256, 2) k_face_flux(FaceList l, Flow<T> f, const V4<T> *__restrict__ W, V4<T> *FS,
                                                      const Ctl *__restrict__ ctl) {
    wait_prior_grid();
    if (ctl->halt) return;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < l.count) face_listed(l, f, j, l.at[j], W, FS);
}

template <typename T>
__device__ __forceinline__ T face_sum(const MeshDev<T> &m, const Flow<T> &f, const int i, const int4 tp,
                                      const V4<T> *__restrict__ F, const T *__restrict__ radius,
                                      V4<T> *__restrict__ res, T *__restrict__ dt) {
    const int n = m.n;
    const int code[3] = {tp.x, tp.y, tp.z};
    V4<T> v[3], r = {};
    T q[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int c = code[k], j = c >= 0 && ((c >> 2) & 1) ? (c & 3) * n + (c >> 3) : k * n + i;
        v[k] = F[j];
        q[k] = radius[j];
    }
#pragma unroll
    for (int k = 0; k < 3; k++) add_flux(r, v[k], code[k] >= 0 && ((code[k] >> 2) & 1));
    res[i] = r;
    return dt[i] = local_dt(m, f, i, q[0] + q[1] + q[2]);
}
template <typename T>
__global__ void __launch_bounds__(256) k_face_sum(MeshDev<T> m, Flow<T> f, const V4<T> *__restrict__ F,
                                                  const T *__restrict__ radius, V4<T> *__restrict__ res,
                                                  T *__restrict__ dt, Ctl *ctl, const int st) {
    wait_prior_grid();
    if (ctl->halt) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    T dti = T(INFINITY);
    if (i < m.n) dti = face_sum(m, f, i, m.topo[i], F, radius, res, dt);
    if (f.global_dt) block_min_dt(dti, &ctl->dtmin[st]);
}

// Threads per cell of pass A.  FP32: one.  FP64: a mesh of up to some 100k cells
// has one to five warps for each of the GPU's 608 schedulers, and a launch takes as
// long as one thread's chain of some 2500 instructions, so the cell's components
// are spread over more threads; on large meshes that only repeats loads and the
// work per cell.  us per iteration with 1 / 2 / 4 and a face list: 12.8k cells 177 /
// 162 / 152, 34k 221 / 207 / 214, 80k 376 / 353 / 362, 131k 497 / 493 / 512 (with the
// cell-wise limiter 633 / 658 / 668), 252k 908 / 907 / 938.  In tiles (at most
// 12k cells, and the allocation-free iteration's 33k) four, then two; pass B's
// tiles are half a block, one thread per listed face (8k: 22 us a launch, 33 with
// tiles of a block).  (The positivity option compares a cell's components: one.)
template <typename T> int faces_lanes(const Plan<T> &p) {
    const int n = p.m.n;
    if (sizeof(T) == 4 || p.f.positivity) return 1;
    if (p.faces.count) return n > 100000 ? 1 : n > 16000 ? 2 : 4;
    return n > 12000 ? 2 : 4;
}

// Sum of the interior neighbours' values in face order (gpu_solver.cu:1658-1666)
template <typename T>
__device__ __forceinline__ V4<T> nb_sum(const int4 tp, const V4<T> *__restrict__ src) {
    V4<T> d;
    d.x = T(0.0); d.y = T(0.0); d.z = T(0.0); d.w = T(0.0);
    const int code[3] = {tp.x, tp.y, tp.z};
#pragma unroll
    for (int k = 0; k < 3; k++)
        if (code[k] >= 0) {
            const V4<T> v = src[code[k] >> 3];
            if (sizeof(T) == 8 && k == 0) { d = v; continue; }  // no addition to zero
            d.x += v.x; d.y += v.y; d.z += v.z; d.w += v.w;
        }
    return d;
}

// ---------------------------------------------------------------------------
// Pass C: gpu_solver.cu:1635-1673 (kernel_Smooth1): one Jacobi-type sweep
// dst = (eps * sum_interior src + res) / (1 + eps * CLog).
template <typename T, class O>
__device__ __forceinline__ V4<T> smooth_with(O &q, const T eps, const int clog, const V4<T> &d, const V4<T> &r0) {
    const auto den = q.over(T(1.0) + (eps) * T(clog));
    V4<T> o;
    if constexpr (sizeof(T) == 8) {  // two products on each kind of unit (1.05M cells: 45 -> 41 us, pass D 70 -> 67)
        o.x = q.by(q.template mul<true>(d.x, eps) + r0.x, den);
        o.y = q.by(q.template mul<true>(d.y, eps) + r0.y, den);
    } else {
        o.x = q.by(madd(d.x, eps, r0.x), den);
        o.y = q.by(madd(d.y, eps, r0.y), den);
    }
    o.z = q.by(madd(d.z, eps, r0.z), den);
    o.w = q.by(madd(d.w, eps, r0.w), den);
    return o;
}
static __device__ __noinline__ V4<double> smooth_ieee(const double eps, const int clog, const V4<double> d,
                                                      const V4<double> r0) {
    IeeeOps o;
    return smooth_with(o, eps, clog, d, r0);
}
template <typename T>
__device__ __forceinline__ V4<T> smooth_value(const T eps, const int clog, const V4<T> &d, const V4<T> &r0) {
    OpsOf<T> o;
    V4<T> v = smooth_with(o, eps, clog, d, r0);
    if constexpr (sizeof(T) == 8)
        if (o.bad) v = smooth_ieee(eps, clog, d, r0);
    return v;
}

template <typename T>
__device__ __forceinline__ void smooth_cell(const MeshDev<T> &m, const T eps, const int i,
                                            const V4<T> *__restrict__ src, const V4<T> *__restrict__ res,
                                            V4<T> *__restrict__ dst) {
    const int4 tp = m.topo[i];
    dst[i] = smooth_value(eps, tp.w, nb_sum(tp, src), res[i]);
}

template <typename T>
__global__ void __launch_bounds__(256) k_smooth(MeshDev<T> m, T eps, const V4<T> *__restrict__ src,
                                                const V4<T> *__restrict__ res, V4<T> *__restrict__ dst,
                                                const Ctl *__restrict__ ctl) {
    wait_prior_grid();
    if (ctl->halt) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.n) return;
    smooth_cell(m, eps, i, src, res, dst);
}

// ---------------------------------------------------------------------------
// Pass D: gpu_solver.cu:1675-1720 (kernel_Smooth2, last sweep + clamp) fused
// with 938-966 (kernel_RKStep); on the last stage also 968-1020 (kernel_drou)
// as FP64 block partials and a count of unphysical cells.
// The new state from the start state w0, the residual r and (smooth) the sum d of
// the neighbours' smoothed residuals; want: also rho - rho0 and whether the state
// is unphysical.
template <typename T, class O>
__device__ __forceinline__ V4<T> update_with(O &o, const T eps, const T rk, const int smooth, const int clog, V4<T> r,
                                             const V4<T> &d, const T dti, const T area, const V4<T> &w0) {
    if (smooth) {
        const V4<T> s = smooth_with(o, eps, clog, d, r);
        if (abs_less(s.x, r.x)) r.x = s.x;
        if (abs_less(s.y, r.y)) r.y = s.y;
        if (abs_less(s.z, r.z)) r.z = s.z;
        if (abs_less(s.w, r.w)) r.w = s.w;
    }
    T RK = rk;
    RK *= dti;
    const auto A = o.over(area);
    V4<T> w;
    w.x = w0.x - o.by(RK * r.x, A);
    w.y = w0.y - o.by(RK * r.y, A);
    w.z = w0.z - o.by(RK * r.z, A);
    w.w = w0.w - o.by(RK * r.w, A);
    return w;
}
static __device__ __noinline__ V4<double> update_ieee(const double eps, const double rk, const int smooth,
                                                      const int clog, const V4<double> r, const V4<double> d,
                                                      const double dti, const double area, const V4<double> w0) {
    IeeeOps o;
    return update_with(o, eps, rk, smooth, clog, r, d, dti, area, w0);
}
template <typename T>
__device__ __forceinline__ V4<T> update_value(const T eps, const T rk, const int smooth, const int clog, const V4<T> &r,
                                              const V4<T> &d, const T dti, const T area, const V4<T> &w0,
                                              const bool want, T &drho, int &bad) {
    OpsOf<T> o;
    V4<T> w = update_with(o, eps, rk, smooth, clog, r, d, dti, area, w0);
    if constexpr (sizeof(T) == 8)
        if (o.bad) w = update_ieee(eps, rk, smooth, clog, r, d, dti, area, w0);
    if (want) {
        // rho - rho0 in the stencil's precision: exact in FP32 as long as the
        // two densities are within a factor of two (Sterbenz)
        drho = w.x - w0.x;
        const T q = gdiv(T(0.5) * (w.y * w.y + w.z * w.z), w.x);
        bad = !(w.x > T(0)) || !(w.w - q > T(0));
    }
    return w;
}

template <typename T>
__device__ __forceinline__ void update_cell(const MeshDev<T> &m, const Flow<T> &f, const T rk,
                                            const int smooth, const int i, const V4<T> *__restrict__ src,
                                            const V4<T> *__restrict__ res, const T dti,
                                            const V4<T> *W0, V4<T> *Wout, const bool want, T &drho,
                                            int &bad) {
    const int4 tp = m.topo[i];
    V4<T> d = {};
    if (smooth) d = nb_sum(tp, src);
    Wout[i] = update_value(f.irs_eps, rk, smooth, tp.w, res[i], d, dti, m.area[i], W0[i], want, drho, bad);
}

// Deterministic block sum of (rho - rho0)^2 (fixed shuffle tree, then the
// warps in order) into *slot, and the count of unphysical cells added to
// *nbad.  Every thread of the block must call it.  FP64 stencil: an FP64 sum.
// FP32 stencil: the squares and sums as unevaluated pairs of floats (exact
// square by a fused multiply-add, two-sum additions), about 48 bits, so that
// pass D issues no FP64 instruction (FP64 throughput is a small fraction of
// FP32 on this GPU and the FP64 tree took ~25 us per iteration at 4.2M
// cells); *slot then holds the pair as a float2 that the residual kernel
// widens to FP64.
__device__ __forceinline__ void block_partial(double drho, int bad, double *slot, int *nbad) {
    double d2 = drho * drho;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d2 += __shfl_down_sync(0xffffffffu, d2, o);
    unsigned badmask = __ballot_sync(0xffffffffu, bad);
    __shared__ double ws[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();  // ws may still be read by the previous use in this block
    if (lane == 0) {
        ws[wid] = d2;
        if (badmask) atomicAdd(nbad, __popc(badmask));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) s += ws[k];
        *slot = s;
    }
}

// a + b for unevaluated float pairs (a.x + a.y): two-sum of the leading
// parts, the trailing parts and its error added, renormalised.  The terms
// summed here are non-negative, so there is no cancellation.
__device__ __forceinline__ void pair_add(float &ah, float &al, const float bh, const float bl) {
    const float s = ah + bh;
    const float bb = s - ah;
    const float e = (ah - (s - bb)) + (bh - bb);
    const float t = e + (al + bl);
    ah = s + t;
    al = t - (ah - s);
}

// The warp's sum of drho^2 as a pair, in lane 0.
__device__ __forceinline__ float2 warp_squares(const float drho) {
    float hi = drho * drho;
    float lo = fmaf(drho, drho, -hi);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float bh = __shfl_down_sync(0xffffffffu, hi, o), bl = __shfl_down_sync(0xffffffffu, lo, o);
        pair_add(hi, lo, bh, bl);
    }
    return make_float2(hi, lo);
}

__device__ __forceinline__ void block_partial(float drho, int bad, double *slot, int *nbad) {
    const float2 sq = warp_squares(drho);
    unsigned badmask = __ballot_sync(0xffffffffu, bad);
    __shared__ float2 wsf[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();  // wsf may still be read by the previous use in this block
    if (lane == 0) {
        wsf[wid] = sq;
        if (badmask) atomicAdd(nbad, __popc(badmask));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float sh = 0.0f, sl = 0.0f;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) pair_add(sh, sl, wsf[k].x, wsf[k].y);
        *reinterpret_cast<float2 *>(slot) = make_float2(sh, sl);
    }
}

// GDT: the global time-step option (its FP64 slot is converted per thread, an
// FP64-pipe instruction the local-step variant does without).
template <typename T, bool GDT>
__global__ void __launch_bounds__(256) k_update(MeshDev<T> m, Flow<T> f, T rk, int smooth,
                                                const V4<T> *__restrict__ src, const V4<T> *__restrict__ res,
                                                const T *__restrict__ dt, const V4<T> *W0, V4<T> *Wout,
                                                double *__restrict__ part, Ctl *ctl, const int st) {
    wait_prior_grid();
    if (ctl->halt) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    T drho = T(0.0);
    int bad = 0;
    if (i < m.n)
        update_cell(m, f, rk, smooth, i, src, res,
                    GDT ? (T)__longlong_as_double((long long)ctl->dtmin[st]) : dt[i], W0, Wout, part != nullptr,
                    drho, bad);
    if (!part) return;
    block_partial(drho, bad, part + blockIdx.x, &ctl->nbad);
}

// ---------------------------------------------------------------------------
// Batched cases: the same per-cell work as the kernels above, by persistent
// CTAs that walk the tiles of all cases (tile = blockDim.x consecutive cells,
// all of one case: cases are padded to kChunk cells and a block has at most
// kChunk threads).  The tile's case, or that it is halted (converged), is one load
// beside the cell's face codes, so the cell's gathers wait for no more than in a
// single case; its flow constants are read beside them, and padding cells have a
// mark in their face codes.  (With the case, then its halt flag and last cell, read
// before the gathers an iteration of 60 cases, 1.85M cells, took 507 us; so 453;
// 24 cases of 33k cells with the smooth limiter 255 -> 241 us.)  With a CTA for every
// tile (LOOP false, the default launch shape) there is no loop to keep values for
// and pass B has its single-case registers (540 -> 508 us).
// In FP64 kb_faces and kb_flux serve batches of at most 12000 cells (above, a face
// list).  kb_faces with options spills 212 bytes per thread there, at the 128
// registers of two blocks; 4 cases of 4096 cells in tiles took 196 us an iteration
// without options, 222 with the smooth limiter.

template <typename T, bool OPT, bool LOOP>
__global__ void __launch_bounds__(256, OPT && sizeof(T) == 4 ? kOptBlocks : BatchMinBlocks<T>::faces) kb_faces(MeshDev<T> m, BatchDev<T> b, int ntiles, const V4<T> *__restrict__ W,
                                      V4<T> *__restrict__ FS, T *__restrict__ dt, V4<T> *__restrict__ phi,
                                      const int st) {
    extern __shared__ __align__(32) unsigned char smem[];
    wait_prior_grid();
    for (int t = blockIdx.x; t < ntiles; t += LOOP ? gridDim.x : ntiles) {
        const int base = t * blockDim.x, i = base + threadIdx.x;
        int4 tp;  // requested with the lookup, not after it
        if (sizeof(T) == 4) tp = m.topo[i];
        const int tc = b.live[base / kChunk];  // the tile's case
        if (tc < 0) continue;                  // uniform over the block
        const Flow<T> &f = b.flows[tc];
        double v = __longlong_as_double((long long)kDtNone);
        const int frozen = OPT && phi ? b.ctl[tc].frozen : 0;
        const bool first = OPT && b.ctl[tc].step < f.first_order;
        if constexpr (sizeof(T) == 8)
            v = faces_tile<OPT, 1>(m, f, base, max(0, min((int)blockDim.x, b.case_end[tc] - base)), W, FS, dt, phi,
                                frozen, first, smem);
        else if (tp.w >= 0)
            v = (double)faces_cell<OPT>(m, f, i, W, FS, dt, phi, frozen, first, tp);
        if (OPT && f.global_dt) block_min_dt(v, &b.ctl[tc].dtmin[st]);  // uniform over the block
    }
}

template <typename T, bool LOOP>
__global__ void __launch_bounds__(256, LOOP ? BatchMinBlocks<T>::flux : MinBlocks<T>::flux) kb_flux(MeshDev<T> m, BatchDev<T> b, int ntiles, const V4<T> *__restrict__ W, const V4<T> *__restrict__ FS,
                                    V4<T> *__restrict__ res) {
    wait_prior_grid();
    for (int t = blockIdx.x; t < ntiles; t += LOOP ? gridDim.x : ntiles) {
        const int base = t * blockDim.x, i = base + threadIdx.x;
        int4 tp;  // requested with the lookup, not after it
        if (!FluxTiled<T>::value) tp = m.topo[i];
        const int tc = b.live[base / kChunk];  // every cell of a tile is in one case
        if (tc < 0) continue;                  // uniform over the block
        const Flow<T> &f = b.flows[tc];
        if constexpr (FluxTiled<T>::value) {
            flux_tile(m, f, base, max(0, min((int)blockDim.x, b.case_end[tc] - base)), W, FS, res);
        } else {
            if (tp.w >= 0) flux_cell(m, f, i, W, FS, res, tp);
        }
    }
}

// FP64 with a face list of all cases: passes A and B as in a single mesh, a thread
// per cell or face whatever the launch shape.  A block's cells are in one case.
// An iteration of 60 cases, 1.85M cells, in tiles and so: 7243 and 5763 us; 24 cases of
// 33k cells with the smooth limiter 3764 and 3164.
template <bool OPT, int LPC>
__global__ void __launch_bounds__(256, 2) kb_faces_cells(MeshDev<double> m, BatchDev<double> b,
                                                         const V4<double> *__restrict__ W, V4<double> *FS,
                                                         V4<double> *__restrict__ phi) {
    wait_prior_grid();
    const int t = blockIdx.x * blockDim.x + threadIdx.x, i = t / LPC;
    if (i >= m.n) return;  // whole warps: n is a multiple of kChunk
    const int4 tp = m.topo[i];
    const int tc = b.live[i / kChunk];
    if (tc < 0) return;
    const Flow<double> &f = b.flows[tc];
    faces_listed<OPT, LPC>(m, f, i, t % LPC, tp.w >= 0, tp, W, FS, phi, OPT && phi ? b.ctl[tc].frozen : 0,
                           OPT && b.ctl[tc].step < f.first_order);
}

template <typename T>
__global__ void __launch_bounds__(256, 2) kb_face_flux(FaceList l, BatchDev<T> b, const V4<T> *__restrict__ W,
                                                       V4<T> *FS) {
    wait_prior_grid();
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= l.count) return;
    const int4 at = l.at[j];
    const int tc = b.live[at.z / kChunk];
    if (tc >= 0) face_listed(l, b.flows[tc], j, at, W, FS);
}

template <typename T>
__global__ void __launch_bounds__(256) kb_face_sum(MeshDev<T> m, BatchDev<T> b, const V4<T> *__restrict__ F,
                                                   const T *__restrict__ radius, V4<T> *__restrict__ res,
                                                   T *__restrict__ dt, const int st) {
    wait_prior_grid();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.n) return;  // whole blocks
    const int4 tp = m.topo[i];
    const int tc = b.live[i / kChunk];
    if (tc < 0) return;  // uniform over the block
    const Flow<T> &f = b.flows[tc];
    T dti = T(INFINITY);
    if (tp.w >= 0) dti = face_sum(m, f, i, tp, F, radius, res, dt);
    if (f.global_dt) block_min_dt(dti, &b.ctl[tc].dtmin[st]);
}

template <typename T, bool LOOP>
__global__ void __launch_bounds__(256) kb_smooth(MeshDev<T> m, BatchDev<T> b, int ntiles, T eps,
                                                 const V4<T> *__restrict__ src, const V4<T> *__restrict__ res,
                                                 V4<T> *__restrict__ dst) {
    wait_prior_grid();
    for (int t = blockIdx.x; t < ntiles; t += LOOP ? gridDim.x : ntiles) {
        const int base = t * blockDim.x, i = base + threadIdx.x;
        const int4 tp = m.topo[i];  // requested with the lookup, not after it
        const V4<T> r = res[i];
        if (b.live[base / kChunk] < 0) continue;
        if (tp.w >= 0) dst[i] = smooth_value(eps, tp.w, nb_sum(tp, src), r);
    }
}

// GDT: some case uses the global time-step option (read per case); without
// it the FP32 build issues no FP64 conversion.
template <typename T, bool GDT, bool LOOP>
__global__ void __launch_bounds__(256) kb_update(MeshDev<T> m, BatchDev<T> b, int ntiles, T rk, int smooth,
                                                 const V4<T> *__restrict__ src, const V4<T> *__restrict__ res,
                                                 const T *__restrict__ dt, const V4<T> *W0, V4<T> *Wout,
                                                 double *__restrict__ part, const int st) {
    wait_prior_grid();
    for (int t = blockIdx.x; t < ntiles; t += LOOP ? gridDim.x : ntiles) {
        const int base = t * blockDim.x, i = base + threadIdx.x;
        const int4 tp = m.topo[i];  // requested with the lookup, not after it
        const int tc = b.live[base / kChunk];  // the tile's case
        if (tc < 0) continue;                  // uniform over the block
        T drho = T(0.0);
        int bad = 0;
        if (tp.w >= 0) {
            V4<T> d = {};
            if (smooth) d = nb_sum(tp, src);
            const T dti = GDT ? stage_dt(b.flows[tc], &b.ctl[tc], st, dt, i) : dt[i];
            Wout[i] = update_value(b.flows[tc].irs_eps, rk, smooth, tp.w, res[i], d, dti, m.area[i], W0[i],
                                   part != nullptr, drho, bad);
        }
        if (part) block_partial(drho, bad, part + t, &b.ctl[tc].nbad);
    }
}

// One iteration of every case that has not halted; the same stage / buffer
// sequence as enqueue_iteration.
template <typename T, bool LOOP> void enqueue_batch_passes(const BPlan<T> &p, cudaStream_t s) {
    const int B = p.block, NT = (p.m.n + B - 1) / B, G = p.grid;
    for (int st = 0; st < p.stages; st++) {
        const bool last = st == p.stages - 1;
        V4<T> *Wcur = st == 0 ? p.W[0] : p.W[1];
        V4<T> *Wout = last ? p.W[0] : p.W[1];
        if (sizeof(T) == 8 && p.faces.count) {
            if constexpr (sizeof(T) == 8) {
                // positivity: one thread per cell (faces_lanes); a case may ask for it
                const int lanes = p.options || p.m.n > 100000 ? 1 : 2;
                launch_chained(p.options ? kb_faces_cells<true, 1>
                               : lanes == 1 ? kb_faces_cells<false, 1> : kb_faces_cells<false, 2>,
                               NT * lanes, B, s, p.m, p.b, Wcur, p.FS, p.phi);
                launch_chained(kb_face_flux<T>, (p.faces.count + B - 1) / B, B, s, p.faces, p.b, Wcur, p.FS);
                launch_chained(kb_face_sum<T>, NT, B, s, p.m, p.b, p.FS, p.faces.radius, p.res, p.dt, st);
            }
        } else {
            launch_chained_smem(p.options ? kb_faces<T, true, LOOP> : kb_faces<T, false, LOOP>, G, B,
                                sizeof(T) == 8 ? B * FacesSmem::per_cell : 0, s, p.m, p.b, NT, Wcur, p.FS, p.dt, p.phi,
                                st);
            launch_chained(kb_flux<T, LOOP>, G, B, s, p.m, p.b, NT, Wcur, p.FS, p.res);
        }
        const V4<T> *src = p.res;
        for (int sw = 0; sw + 1 < p.sweeps; sw++) {
            V4<T> *dst = p.sm[sw & 1];
            launch_chained(kb_smooth<T, LOOP>, G, B, s, p.m, p.b, NT, p.f.irs_eps, src, p.res, dst);
            src = dst;
        }
        launch_chained(p.options ? kb_update<T, true, LOOP> : kb_update<T, false, LOOP>, G, B, s, p.m, p.b, NT,
                       p.rk[st], p.sweeps > 0 ? 1 : 0, src, p.res, p.dt, p.W[0], Wout, last ? p.part : nullptr, st);
    }
    enqueue_batch_resid(p.part, p.case_tiles, p.ncase, p.b.ctl, p.hist, p.hist_cap, sizeof(T) == 4, p.b.live, B, s);
}

template <typename T> void enqueue_batch_iteration(const BPlan<T> &p, cudaStream_t s) {
    if (p.grid >= (p.m.n + p.block - 1) / p.block) enqueue_batch_passes<T, false>(p, s);
    else enqueue_batch_passes<T, true>(p, s);
}

// ---------------------------------------------------------------------------
// State exchange with the caller: FP64 in file order <-> T in internal order.
template <typename T>
__global__ void k_import(int n, const int *__restrict__ perm, const double *__restrict__ wfile,
                         V4<T> *__restrict__ W) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double *s = wfile + 4 * (size_t)perm[i];
    V4<T> o;
    o.x = (T)s[0]; o.y = (T)s[1]; o.z = (T)s[2]; o.w = (T)s[3];
    W[i] = o;
}

template <typename T>
__global__ void k_export(int n, const int *__restrict__ perm, const V4<T> *__restrict__ W,
                         double *__restrict__ wfile) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const V4<T> v = W[i];
    double *d = wfile + 4 * (size_t)perm[i];
    d[0] = (double)v.x; d[1] = (double)v.y; d[2] = (double)v.z; d[3] = (double)v.w;
}

// The states of a list of cells (the wall cells of the forces), FP64.
template <typename T>
__global__ void k_export_cells(int cnt, const int *__restrict__ cells, const V4<T> *__restrict__ W,
                               double *__restrict__ w) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cnt) return;
    const V4<T> v = W[cells[j]];
    double *d = w + 4 * (size_t)j;
    d[0] = (double)v.x; d[1] = (double)v.y; d[2] = (double)v.z; d[3] = (double)v.w;
}

template <typename T>
void enqueue_export_cells(int cnt, const int *cells, const V4<T> *W, double *w, cudaStream_t s) {
    if (cnt > 0) k_export_cells<T><<<(cnt + 255) / 256, 256, 0, s>>>(cnt, cells, W, w);
}

template <typename T>
void enqueue_import(int n, const int *perm, const double *wfile, V4<T> *W, cudaStream_t s) {
    k_import<T><<<(n + 255) / 256, 256, 0, s>>>(n, perm, wfile, W);
}

template <typename T>
void enqueue_export(int n, const int *perm, const V4<T> *W, double *wfile, cudaStream_t s) {
    k_export<T><<<(n + 255) / 256, 256, 0, s>>>(n, perm, W, wfile);
}

// ---------------------------------------------------------------------------
// One iteration: gpu_solver.cu:2200-2434 without the W -> W0 copies.  W[0]
// holds the start state; stage 0 reads it and writes W[1], middle stages
// update W[1] in place, and the last stage writes the result back into W[0]
// (each cell reads its own W0 before overwriting it), so W[0] is also the
// next iteration's W0.
// mark(kind) and done() bracket each launch (kind: 0 faces, 1 flux, 2 smooth,
// 3 update, 4 resid).
template <typename T, typename Mark, typename Done>
void enqueue_passes(const Plan<T> &p, cudaStream_t s, Mark mark, Done done) {
    const int n = p.m.n, B = p.block, G = (n + B - 1) / B;
    const bool opt = faces_options(p.f, p.phi);
    const int lanes = faces_lanes(p);
    const auto grid = [&](int per_cell) { return (n + B / per_cell - 1) / (B / per_cell); };
    for (int st = 0; st < p.stages; st++) {
        const bool last = st == p.stages - 1;
        V4<T> *Wcur = st == 0 ? p.W[0] : p.W[1];
        V4<T> *Wout = last ? p.W[0] : p.W[1];
        mark(0);
        if constexpr (sizeof(T) == 4) {
            launch_chained(opt ? k_faces<T, true> : k_faces<T, false>, G, B, s, p.m, p.f, Wcur, p.FS, p.dt, p.ctl,
                           p.phi, st);
            done();
            mark(1);
            launch_chained(k_flux<T>, G, B, s, p.m, p.f, Wcur, p.FS, p.res, p.ctl);
        } else if (p.faces.count) {
            launch_chained(faces_cells_kernel(opt, lanes), grid(lanes), B, s, p.m, p.f, Wcur, p.FS, p.ctl, p.phi);
            done();
            mark(1);
            launch_chained(k_face_flux<T>, (p.faces.count + B - 1) / B, B, s, p.faces, p.f, Wcur, p.FS, p.ctl);
            done();
            mark(1);
            launch_chained(k_face_sum<T>, G, B, s, p.m, p.f, p.FS, p.faces.radius, p.res, p.dt, p.ctl, st);
        } else {
            launch_chained_smem(faces_tile_kernel(opt, lanes), grid(lanes), B, B / lanes * FacesSmem::per_cell, s, p.m,
                                p.f, Wcur, p.FS, p.dt, p.ctl, p.phi, st);
            done();
            mark(1);
            launch_chained(k_flux_tile<T>, grid(2), B, s, p.m, p.f, Wcur, p.FS, p.res, p.ctl);
        }
        done();
        const V4<T> *src = p.res;
        for (int sw = 0; sw + 1 < p.sweeps; sw++) {
            V4<T> *dst = p.sm[sw & 1];
            mark(2);
            launch_chained(k_smooth<T>, G, B, s, p.m, p.f.irs_eps, src, p.res, dst, p.ctl);
            done();
            src = dst;
        }
        mark(3);
        launch_chained(p.f.global_dt ? k_update<T, true> : k_update<T, false>, G, B, s, p.m, p.f, p.rk[st],
                       p.sweeps > 0 ? 1 : 0, src, p.res, p.dt, p.W[0], Wout, last ? p.part : nullptr, p.ctl, st);
        done();
    }
    mark(4);
    enqueue_resid(p.part, G, p.ctl, p.hist, p.hist_cap, sizeof(T) == 4, s);
    done();
}

template <typename T> void enqueue_iteration(const Plan<T> &p, cudaStream_t s) {
    enqueue_passes(p, s, [](int) {}, [] {});
}

// Same launches as enqueue_iteration, with events recorded around each one.
// ev[2*j], ev[2*j+1] bracket launch j; kind[j] is its kind.  Returns the
// number of launches.
template <typename T>
int enqueue_iteration_timed(const Plan<T> &p, cudaStream_t s, cudaEvent_t *ev, int *kind) {
    int j = 0;
    enqueue_passes(
        p, s, [&](int k) { kind[j] = k; cudaEventRecord(ev[2 * j], s); },
        [&] { cudaEventRecord(ev[2 * j + 1], s); j++; });
    return j;
}

}  // namespace e2d
