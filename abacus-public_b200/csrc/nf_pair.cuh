// nf_pair.cuh -- per-pair softened gravity on the B200 FP32 pipe.
//
// Softening formulas follow singlestep/Direct/DirectGPUKernels.cuh:20-174
// (Plummer :144-174, single spline :68-108, cubic spline :20-66, cubic
// Plummer :110-143).  Differences from the reference GPU kernel, all in the
// direction of accuracy:
//   * rsqrt is the hardware estimate (rsqrt.approx.ftz.f32) followed by one
//     Newton-Raphson step, applied to the cube:
//       y = rsqrt(r2); q = r2*y^2 (1 up to the estimate's error)
//       r2^-3/2 ~= y^3 * (1 - 1.5 (q - 1)) = y^3 * (q - 5/3) * (-3/2)
//     The one-sided engine writes the step as y^3 - 1.5 (q - 1) y^3, five
//     instructions, 3.8e-8 RMS.  The mutual engine uses the product above,
//     four instructions, 4.6e-8 RMS (q - 5/3 rounds to 2^-25 at 2/3), with
//     the constant factor left out of the pair (Step::SHORT): sums are in
//     units of NEWTON_UNIT = 1 - float(5/3), divided out once per sink.  Its
//     64-bit sums are nearer to FP64 than the one-sided engine's compensated
//     FP32 all the same (uniform boxes of 3000 and 20000 particles: 3.0e-7 and
//     1.8e-7 beside 3.4e-7 and 2.6e-7; isolated pairs, where nothing is summed:
//     Plummer 1.07e-7 beside 1.03e-7, single spline 1.24e-7 beside 1.45e-7),
//     and the fifth instruction costs it 3-4 % of a sweep (clustered 256^3
//     90.0 -> 93.3 ms, uniform 160^3 12.1 -> 12.6) and 10 % of a single slab;
//     the one-sided engine pays 1 % (uniform 160^3 15.75 -> 15.91 ms).
//   * the single spline is accumulated in far units, g = f_ref / eps^3
//     (r^-3 in the far branch), and the sum is multiplied by eps^3 once per
//     sink.  Chunks of sources that hold none within the spline's reach of a
//     tile's sinks use the far branch alone; the others the full formula.
//   * the cubic kernels are free of branches and divisions (cubic spline,
//     uniform 75^3: 3.26 -> 1.43 ms a sweep beside the scalar form with an
//     IEEE division and three-way branch).  Error against FP64 beside that
//     form, uniform boxes of 20000: cubic spline 6.9e-7 -> 1.7e-7, cubic
//     Plummer 2.6e-7 -> 1.7e-7 (2.6e-7 both in the one-sided engine).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>

#include "nf_capi.h"

namespace nf {

enum { SOFT_PLUMMER = 0, SOFT_SINGLE_SPLINE = 1, SOFT_CUBIC_SPLINE = 2, SOFT_CUBIC_PLUMMER = 3 };

// Hardware reciprocal square root estimate (one MUFU.RSQ).
__device__ __forceinline__ float rsqrt_est(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The Newton step's constant and the unit it leaves the pair sums in (1 - K
// with K as the float it is, so the step has no bias at q = 1).
constexpr float NEWTON_K = 5.0f / 3.0f;
constexpr double NEWTON_UNIT = 1.0 - (double)NEWTON_K;

// How the Newton step on the cube is written: in unit 1, or four instructions
// in NEWTON_UNIT.
enum class Step { FULL, SHORT };

// y^3 with the step, from the estimate y of r2^-1/2.
template <Step STEP>
__device__ __forceinline__ float cube_step(float r2, float y) {
    const float y2 = y * y;
    const float y3 = y2 * y;
    if constexpr (STEP == Step::SHORT) return y3 * fmaf(r2, y2, -NEWTON_K);
    return fmaf(y3 * fmaf(r2, y2, -1.0f), -1.5f, y3);
}

// y with one Newton step.
__device__ __forceinline__ float rsqrt_step(float r2, float y) {
    return fmaf(-0.5f * fmaf(r2, y * y, -1.0f), y, y);
}
// The same from c = r2 y^2 - K: y (c / -2 + M).
constexpr float NEWTON_M = (float)(0.5 * (3.0 - (double)NEWTON_K));

// Hardware reciprocal estimate (one MUFU.RCP).
__device__ __forceinline__ float rcp_est(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// TwoSum (Knuth): s + err == a + b exactly.
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &err) {
    s = a + b;
    float bb = s - a;
    err = (a - (s - bb)) + (b - bb);
}

// Kernel constants shared by every pair of a launch.
struct PairConst {
    float eps;        // the reference kernel parameter (eps^2, 1/eps^2, 1/eps, eps^3)
    float b2;         // FOF density radius^2 (0 = off)
    // single spline near branch in far units (g = f_ref / eps^3):
    //   (-15 u + 6 u^2 + 10) / eps^3 with u = r/eps = r^2 y / eps
    //   = (c1 y + c2) r^2 + c3,  c1 = -15 eps^-4, c2 = 6 eps^-5, c3 = 10 eps^-3,
    // cubic spline: c3 = eps^-3; all in the unit of the step
    float c1, c2, c3;
};

// What r^2 = |d|^2 carries on top: Plummer eps^2; cubic Plummer the
// reference's TAU2 (DirectGPUKernels.cuh:124); the splines a floor far below
// any eps^2, so that a zero separation stays finite.
template <int SOFT>
__device__ __host__ __forceinline__ float r2_add(const PairConst &pc) {
    return SOFT == SOFT_PLUMMER ? pc.eps : SOFT == SOFT_CUBIC_PLUMMER ? 1e-16f : 1e-25f;
}

// Splines near a sink.  The reference writes the single spline as
// min(f^3, (-15 f + 6) dr2 + 10) in eps units (DirectCPUKernels.cc:71; the
// GPU's branch on dr2 > 1, DirectGPUKernels.cuh:94-98, selects the same value
// because the two branches touch to second order at u = 1 and the polynomial
// is the smaller one for u < 1).  Here it is evaluated in far units with the
// Newton-corrected yn = 1/r:
//   g = min(r^-3, (c1 yn + c2) r^2 + c3)
// (in NEWTON_UNIT, which is negative, the smaller is the maximum).
// A self pair (d = 0, r^2 = 1e-25 floor) gives a finite g times d = 0; a
// padding record far away gives an infinite polynomial and g ~ 0.
// The cubic spline (Hernquist & Katz, DirectGPUKernels.cuh:31-65) is r^-3
// beyond u = r/eps = 2, r^-3 (-1/15 + u^3 (8/3 - 3 u + 6/5 u^2 - u^3/6)) down
// to u = 1 and eps^-3 (4/3 - 6/5 u^2 + u^3/2) below.  The bracket is 1 at
// u = 2 to fourth order,
//   1 - (2 - u)^4 (1/15 + 2 u / 15 + u^2 / 6),
// and evaluated in that form: the powers of u cancel to a part in 40 at
// u = 2, and cost up to 2e-6 there (FP32 model, RMS over u in [1.75, 2));
// this form keeps 6e-8, at one more instruction (uniform 75^3 1.389 -> 1.405
// ms a sweep).
// Only sources within near_width() of a tile's sinks need these; all others
// are evaluated as r^-3.

// g of a += g * d from r^2 (r2_add included), in the unit of the step.  NEAR:
// the splines' full formula; otherwise their far branch.
template <int SOFT, bool NEAR, Step STEP>
__device__ __forceinline__ float pair_g(float r2, const PairConst &pc) {
    const float y = rsqrt_est(r2);
    if constexpr (SOFT == SOFT_CUBIC_PLUMMER) {
        // 1 / (r^3 + eps^3): reciprocal estimate and one Newton step written on
        // the residual, so that only the last addition rounds; the clamp keeps
        // t * (1/t) defined for padding records
        const float t = fminf(fmaf(r2 * r2, rsqrt_step(r2, y), pc.eps), 1e37f);
        const float g = rcp_est(t);
        return fmaf(fmaf(-t, g, 1.0f), g, g);
    } else if constexpr (!NEAR || SOFT == SOFT_PLUMMER) {
        return cube_step<STEP>(r2, y);
    } else {
        if constexpr (SOFT == SOFT_SINGLE_SPLINE && STEP == Step::SHORT) {
            // one c for both, written out: with the two steps above, left to the
            // compiler to share, clustered 256^3 took 91.2 ms instead of 89.9
            const float y2 = y * y;
            const float c = fmaf(r2, y2, -NEWTON_K);
            const float yn = y * fmaf(c, -0.5f, NEWTON_M);
            const float gfar = (y2 * y) * c;
            return fmaxf(gfar, fmaf(fmaf(pc.c1, yn, pc.c2), r2, pc.c3));
        }
        const float gfar = cube_step<STEP>(r2, y);
        const float yn = rsqrt_step(r2, y);
        if constexpr (SOFT == SOFT_SINGLE_SPLINE) {
            return fminf(gfar, fmaf(fmaf(pc.c1, yn, pc.c2), r2, pc.c3));
        } else {
            const float u = r2 * yn * pc.eps;
            const float u2 = u * u, w = 2.f - u, w2 = w * w;
            const float p = fmaf(u, fmaf(u, -1.f / 6.f, -2.f / 15.f), -1.f / 15.f);
            const float mid = fmaf(w2 * w2, p, 1.f);
            const float near = fmaf(u2, fmaf(u, 0.5f, -1.2f), 4.f / 3.f);
            return u >= 2.f ? gfar : u >= 1.f ? gfar * mid : pc.c3 * near;
        }
    }
}

// ---------------------------------------------------------------------------
// Two sinks per instruction.  sm_100 executes FP32 add/mul/fma on register
// pairs (f32x2): one issue slot for two results, the same per-component
// rounding as the scalar instruction.  The pair loop is issue-bound in
// scalar form (~15 issue slots per pair against 14 FP32 results), so pairing
// the sinks of a lane moves the bound to the FP32 pipe itself.  Each helper
// below is the component-wise twin of the scalar code above, operation for
// operation, so a paired evaluation is bit-identical to the scalar one.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }

// cube_step and rsqrt_step on a pair.
template <Step STEP>
__device__ __forceinline__ float2 cube_step_x2(float2 r2, float2 y) {
    const float2 y2 = mul2(y, y);
    const float2 y3 = mul2(y2, y);
    if constexpr (STEP == Step::SHORT) return mul2(y3, fma2(r2, y2, dup2(-NEWTON_K)));
    return fma2(mul2(y3, fma2(r2, y2, dup2(-1.0f))), dup2(-1.5f), y3);
}
__device__ __forceinline__ float2 rsqrt_step_x2(float2 r2, float2 y) {
    return fma2(mul2(dup2(-0.5f), fma2(r2, mul2(y, y), dup2(-1.0f))), y, y);
}

// r^2 (+ the kernel's additive constant a2) of a pair of separations.
__device__ __forceinline__ float2 r2_x2(float2 dx, float2 dy, float2 dz, float a2) {
    return fma2(dz, dz, fma2(dy, dy, fma2(dx, dx, dup2(a2))));
}

// pair_g on a pair.
template <int SOFT, bool NEAR, Step STEP>
__device__ __forceinline__ float2 pair_g_x2(float2 r2, const PairConst &pc) {
    const float2 y = make_float2(rsqrt_est(r2.x), rsqrt_est(r2.y));
    if constexpr (SOFT == SOFT_CUBIC_PLUMMER) {
        const float2 t0 = fma2(mul2(r2, r2), rsqrt_step_x2(r2, y), dup2(pc.eps));
        const float2 t = make_float2(fminf(t0.x, 1e37f), fminf(t0.y, 1e37f));
        const float2 g = make_float2(rcp_est(t.x), rcp_est(t.y));
        return fma2(fma2(mul2(t, dup2(-1.0f)), g, dup2(1.0f)), g, g);
    } else if constexpr (!NEAR || SOFT == SOFT_PLUMMER) {
        return cube_step_x2<STEP>(r2, y);
    } else {
        if constexpr (SOFT == SOFT_SINGLE_SPLINE && STEP == Step::SHORT) {
            const float2 y2 = mul2(y, y);
            const float2 c = fma2(r2, y2, dup2(-NEWTON_K));
            const float2 yn = mul2(y, fma2(c, dup2(-0.5f), dup2(NEWTON_M)));
            const float2 gfar = mul2(mul2(y2, y), c);
            const float2 gnear = fma2(fma2(dup2(pc.c1), yn, dup2(pc.c2)), r2, dup2(pc.c3));
            return make_float2(fmaxf(gfar.x, gnear.x), fmaxf(gfar.y, gnear.y));
        }
        const float2 gfar = cube_step_x2<STEP>(r2, y);
        const float2 yn = rsqrt_step_x2(r2, y);
        if constexpr (SOFT == SOFT_SINGLE_SPLINE) {
            const float2 gnear = fma2(fma2(dup2(pc.c1), yn, dup2(pc.c2)), r2, dup2(pc.c3));
            return make_float2(fminf(gfar.x, gnear.x), fminf(gfar.y, gnear.y));
        } else {
            const float2 u = mul2(mul2(r2, yn), dup2(pc.eps));
            const float2 u2 = mul2(u, u), w = fma2(u, dup2(-1.f), dup2(2.f)), w2 = mul2(w, w);
            const float2 p = fma2(u, fma2(u, dup2(-1.f / 6.f), dup2(-2.f / 15.f)), dup2(-1.f / 15.f));
            const float2 mid = mul2(gfar, fma2(mul2(w2, w2), p, dup2(1.f)));
            const float2 near =
                mul2(dup2(pc.c3), fma2(u2, fma2(u, dup2(0.5f), dup2(-1.2f)), dup2(4.f / 3.f)));
            return make_float2(u.x >= 2.f ? gfar.x : u.x >= 1.f ? mid.x : near.x,
                               u.y >= 2.f ? gfar.y : u.y >= 1.f ? mid.y : near.y);
        }
    }
}

__host__ __device__ __forceinline__ int wrapc(int i, int cpd) {
    return i < 0 ? i + cpd : (i >= cpd ? i - cpd : i);
}

// 1 if source t lies inside a box: x in [b.x, b.y], y in [b.z, b.w], z in
// [zlo, zhi]; else 0.
__device__ __forceinline__ float inside(const float4 &t, const float4 &b, float zlo, float zhi) {
    return (t.x >= b.x && t.x <= b.y && t.y >= b.z && t.y <= b.w && t.z >= zlo && t.z <= zhi) ? 1.f : 0.f;
}

// Fold a partial p into the running compensated sum (h, l) and clear it
// (plain: one FP32 running sum).  Kahan's compensated summation with the
// correction kept as the low part to add (the sum is h + l):
//   y = p + l;  t = h + y;  l = y - (t - h);  h = t
// four paired instructions per component and sink pair.  Scalar and paired
// (two sinks) forms; a - b is formed as fma(b, -1, a), which rounds exactly
// like a subtraction.
__device__ __forceinline__ void fold1(float &h, float &l, float &p, bool plain) {
    if (plain) {
        h += p;
    } else {
        float y = p + l;
        float t = h + y;
        l = y - (t - h);
        h = t;
    }
    p = 0.f;
}

__device__ __forceinline__ void fold2(float2 &h, float2 &l, float2 &p, bool plain) {
    if (plain) {
        h = add2(h, p);
    } else {
        const float2 m1 = dup2(-1.0f);
        float2 y = add2(p, l);
        float2 t = add2(h, y);
        l = fma2(fma2(h, m1, t), m1, y);  // y - (t - h)
        h = t;
    }
    p = make_float2(0.f, 0.f);
}

// Unsoftened r^2 for the FOF density sum (w += b2 - r^2 if r^2 < b2).
__device__ __forceinline__ float dens_term(float dx, float dy, float dz, float b2) {
    float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    return r2 < b2 ? b2 - r2 : 0.0f;
}

// The unit the pair sums of a softening are accumulated in.
inline double pair_unit(int soft, Step step) {
    return soft == SOFT_CUBIC_PLUMMER || step == Step::FULL ? 1.0 : NEWTON_UNIT;
}

// The pair constants of a launch; eps: the softening parameter (0: the configuration's).
inline PairConst pair_const(const nf_config &cfg, float eps, Step step) {
    const double unit = pair_unit(cfg.softening, step);
    PairConst pc{};
    if (!(eps > 0.f)) eps = cfg.eps;
    pc.eps = eps;
    pc.b2 = cfg.b2;
    if (cfg.softening == SOFT_SINGLE_SPLINE) {
        const double ie2 = (double)eps;  // eps_int^-2
        pc.c1 = (float)(-15.0 * ie2 * ie2 * unit);
        pc.c2 = (float)(6.0 * pow(ie2, 2.5) * unit);
        pc.c3 = (float)(10.0 * pow(ie2, 1.5) * unit);
    } else if (cfg.softening == SOFT_CUBIC_SPLINE) {
        pc.c3 = (float)((double)eps * eps * eps * unit);
    }
    return pc;
}

// Whether a kernel comes in several shapes (either engine): the density
// channel and the cubic softenings have shape 0 only.
inline bool tunable(int soft, bool dens) {
    return !dens && (soft == SOFT_PLUMMER || soft == SOFT_SINGLE_SPLINE);
}

// Whether sources are told near from far for a softening.
__host__ __device__ constexpr bool has_near(int soft) {
    return soft == SOFT_SINGLE_SPLINE || soft == SOFT_CUBIC_SPLINE;
}

// Margin of the near test: the separation up to which the spline is not
// r^-3, eps_int (single) or 2 eps_int (cubic), +1% and a rounding allowance.
inline float near_width(const nf_config &cfg, float eps, int cpd) {
    if (!(eps > 0.f)) eps = cfg.eps;
    const double e = cfg.softening == SOFT_SINGLE_SPLINE  ? 1.0 / sqrt((double)eps)
                     : cfg.softening == SOFT_CUBIC_SPLINE ? 2.0 / (double)eps
                                                          : 0.0;
    return (float)(e * 1.01 + 1e-6 / (double)cpd);
}

}  // namespace nf
