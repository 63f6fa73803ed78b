// stage_common.cuh -- device helpers of the stage kernels (stage.cu):
// periodic indices, the precision-dependent fast operations and the RK update
// (reference src/cu/pde.cu:640-720; solver.cu:14-93).
#pragma once

#include <math.h>

#include "wf_internal.h"

namespace wf {
namespace {

__device__ __forceinline__ int wrap_p(int v, int n)
{
    // periodic index with period n = N-1 for v in [-2, 2n+1] (pde.cu:227-234)
    if (v >= n) v -= n;
    if (v >= n) v -= n;
    if (v < 0) v += n;
    return v;
}

template <class R> __device__ __forceinline__ R rmax(R a, R b) { return (a > b) ? a : b; }
template <class R> __device__ __forceinline__ R rmin(R a, R b) { return (a < b) ? a : b; }

// Square root and quotient.  The FP64 path keeps the reference's correctly rounded
// operations; the FP32 stencil path uses the PTX approximations (sqrt.approx,
// rcp.approx: about 1 ulp, no slow path; results below 2^-126 are 0), well inside
// its 1e-5 error budget against FP64: in the strain and its viscosity, the wall friction,
// the Arrhenius exponent, and in the Sutherland laws and the convective exchange, whose
// powers 3/2 and 1/4 are square roots (error of a step with all of them against 64 bits
// 8.6e-7; with powf and IEEE quotients 8.8e-7).  FP64 takes those powers by square roots
// too, and constants that the model divides by as products with their reciprocals: Phi on
// 191 x 96 x 50 is 2.1e-15 from 64-bit arithmetic in the model's order, 1.6e-15 before.
__device__ __forceinline__ double rsqrt_(double x) { return sqrt(x); }
__device__ __forceinline__ float rsqrt_(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ double fdiv(double a, double b) { return a / b; }
__device__ __forceinline__ float fdiv(float a, float b)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    return a * r;
}
__device__ __forceinline__ double rexp(double x) { return exp(x); }
__device__ __forceinline__ float rexp(float x) { return expf(x); }
__device__ __forceinline__ double rpow(double x, double y) { return pow(x, y); }
__device__ __forceinline__ float rpow(float x, float y) { return powf(x, y); }
__device__ __forceinline__ double rfabs(double x) { return fabs(x); }
__device__ __forceinline__ float rfabs(float x) { return fabsf(x); }

// Van Driest damping f_w = 1 - exp(-z+ / A_VD).  Below the cut-off the
// exponential is smaller than half an ulp of 1 and the result is exactly 1.
__device__ __forceinline__ double van_driest(double x) { return x < -37.5 ? 1.0 : 1.0 - exp(x); }
__device__ __forceinline__ float van_driest(float x) { return x < -17.5f ? 1.0f : 1.0f - expf(x); }
template <class R> struct VanDriestCut;
template <> struct VanDriestCut<double> { static constexpr double v = 37.5; };
template <> struct VanDriestCut<float> { static constexpr float v = 17.5f; };
// Arrhenius rate A exp(-T_act/T) H(T - T_pc) (pde.cu:665): exactly 0 below
// the phase change.
template <class R> __device__ __forceinline__ R arrhenius(const PhysR<R> &p, R T)
{
    R K_T = R(0);
    if (T > p.T_pc) K_T = p.A * rexp(-fdiv(p.T_act, T));
    return K_T;
}

// RK update of one value: returns the next-stage (or final) value, updates acc.
//   operator test (method 3): k_s itself;
//   Euler (solver.cu:14-21): y_n + a k;
//   RK2 (solver.cu:23-30, 65-74): acc = k1, y_n + a k1; then y_n + a (acc + k2);
//   RK4 (solver.cu:32-39, 76-93): acc = k1, then acc + 2 k2, acc + 2 k3 with
//   y_n + a k_s; last y_n + a (acc + k4).
// Written as three fused multiply-adds with coefficients of the method and
// stage (uniform over the launch, so computed once), without branches per
// value: t = k + cA acc, out = a t + cY y_n, acc' = cK k + cB acc.  Each is the
// rounding of the contracted expression above (1 and 0 coefficients are exact).
template <class R>
__device__ __forceinline__ R rk_update(int method, int stage, R kv, R yv, R &accv, R a_next)
{
    const bool kstore = method == 3;
    const bool last = (method == 1 && stage == 2) || (method == 2 && stage == 4);
    const bool first = (method == 1 || method == 2) && stage == 1;
    const R cA = last ? R(1) : R(0), cY = kstore ? R(0) : R(1), an = kstore ? R(1) : a_next;
    const R cB = first ? R(0) : R(1), cK = (method == 2 && stage > 1 && stage < 4) ? R(2) : R(1);
    const R t = fma(cA, accv, kv);
    const R out = fma(an, t, cY * yv);
    accv = fma(cK, kv, cB * accv);
    return out;
}

__host__ __device__ __forceinline__ bool stage_keeps_acc(int method, int stage)
{
    return (method == 1 && stage == 1) || (method == 2 && stage < 4);
}
__host__ __device__ __forceinline__ bool stage_reads_acc(int method, int stage)
{
    return (method == 1 && stage == 2) || (method == 2 && stage > 1);
}

}  // namespace
}  // namespace wf
