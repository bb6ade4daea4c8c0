// Small-step Kepler drift in float-float (FP32 pipe).
//
// A drift whose step is a small part of the local dynamical time
// (tau^2 = dt^2 mu / r0^3 < SMALL_DRIFT_TAU2) moves the particle by
//   r' = r + dt v + ((f - 1) r + (g - dt) v),
//   v' = v + (fd r + (gd - 1) v),
// where f - 1, gd - 1 ~ tau^2 / 2, g / dt - 1 ~ tau^2 / 6 and fd r ~ tau v are
// small next to what they are added to, so the ~47 bits of a float-float reach
// past the double's last place.  GB300 issues FP64 at 1/64 of the FP32 rate:
// the corrections are formed on the FP32 pipe and twelve FP64 instructions
// remain in a step (dt v, the sums into r and v, |r'|^2), where the general
// drift (kepler.cuh) and kick execute 44.
//
// Kepler's equation, dimensionless.  With s = (dt/r0)(1 + w), X = u dt/(2 r0^2)
// (u = r.v), A = alpha dt^2/r0^2, Y = (tau^2 - A)/6:
//   R(w) = w + X (1+w)^2 2c2(x) + Y (1+w)^3 6c3(x) = 0,   x = A (1+w)^2,
// from r0 G1 + u G2 + mu G3 = dt.  Every term is a correction of the size of
// w itself (~ e tau / 2).  w starts from the fourth-order reversion, takes one
// FP32 Newton step (to ~1e-9) and one whose residual R is float-float: what is
// left is quadratic in 1e-9.  Then, with 1 + q2 = (1+w)^2 2c2 and
// 1 + q3 = (1+w)^3 6c3,
//   f - 1  = -H / r0,   gd - 1 = -H / r',   H = mu G2 = (mu dt^2/2r0^2)(1 + q2),
//   g / dt = 1 - p,     p = (tau^2 / 6)(1 + q3),
//   fd     = -mu G1 / (r0 r'),  G1 r0 / dt = 1 - X (1 + q2) - p  by Kepler's
//            equation itself: fd needs ~2^-46, and this form multiplies the
//            errors of q2 and q3 by X and tau^2 / 6.
//
// Bound: issue (about 1,400 instructions a step with four planets, 11 cycles of
// the 128 lanes, at 80 % of the issue slots; twelve FP64 instructions are 6 cycles
// of the FP64 pipe).  Packed pairs (fma.rn.f32x2) do not help: each takes two
// issue cycles.  The line at tau^2 = 1e-3: up to there the error of a drift is that
// of FP64 (position 6e-17 rms of |r| against 6e-17, velocity 5e-17 to 1.4e-16 of
// |v| against 7e-17 for the coefficients correctly rounded); at 1e-3..2e-3 it is
// 3.4e-16.  Measured on GB300, before (every drift general) and after: 1e6
// particles x 1,024 steps with four giants 98.6 -> 45.5 ms; 2e6 planet crossers
// x 100 steps 16.6 -> 5.8 ms; 2,000 particles x 128 steps 643 -> 333 us;
// 256 ensembles, 1.5e6 particles x 512 steps, 80 -> 35.5 ms.  Position error of
// those blocks against long double: giants 1.49e-14 -> 1.01e-14 rms, belt
// 2.34e-14 -> 1.64e-14, crossers 8.6e-16 -> 7.2e-16, scattered disk
// 3.5e-15 -> 3.0e-15.
#pragma once
#include "fastmath.cuh"

namespace glisser {

// Bounds on tau^2 of the small-step drift and of its solution of Kepler's
// equation for a drift applied in FP64.  A warp that holds drifts on both sides of
// a bound runs both paths.  Where most warps do, around 1e-3, that gives back the
// gain: 150,000 belt particles x 128 steps take 0.67 ms at dt = 300 d (1.74 with every
// drift general), 1.86 at 600 d, tau^2 of 6e-4 to 2e-3 (1.80), 1.34 at 900 d (2.30);
// with the FP64 kick 1.10 (2.15), 2.38 (2.22), 1.89 (2.73); 4,000 with the FP64
// kick at 600 d 686 us (568).
constexpr float SMALL_DRIFT_TAU2 = 1e-3f;
constexpr float MEDIUM_DRIFT_TAU2 = 1e-2f;

// Least tau^2 / 2 of a small step.  It only keeps the chain of products within a
// float's range: 2^-34 does for any mu, dt and r, and where the ranges of these
// are checked (run_tile: |r|^2 in 2^-40..2^44, mu dt^2 / 2 in 2^-40..2^30, dt in
// 2^-24..2^24) tau^2 / 2 is 2^-106 at least, and what underflows is below 2^-70 of what
// it is added to.  A particle below the bound takes the general drift at every step and
// holds its warp: with 2^-30 (1,700 au at dt = 180 d), one in 500 of a scattered disk,
// 1,000 particles x 128 steps took 706 us, with 2^-34 449, 16,000 867 and 604, 500,000
// 5.12 and 4.23 ms; and with 2^-34 150,000 at dt = 10 d, where it lies at 630 au, took
// 2.53 ms (1.74 with every drift general, 0.72 without a bound).
constexpr float TINY_DRIFT_TH = 0x1p-34f, FAR_DRIFT_TH = 0x1p-110f;

// --- float-float without the renormalising step: hi + lo with |lo| up to a
// few units in hi's last place.  Sums and products of them lose ~2^-46; a
// result is renormalised (ff_norm) where a longer chain follows.
__device__ __forceinline__ ff ff_norm(ff a) { return ff_fast_two_sum(a.hi, a.lo); }

__device__ __forceinline__ ff ff_mul_u(ff a, ff b)
{
    const float p = __fmul_rn(a.hi, b.hi);
    float e = __fmaf_rn(a.hi, b.hi, -p);
    e = __fmaf_rn(a.hi, b.lo, e);
    return { p, __fmaf_rn(a.lo, b.hi, e) };
}

__device__ __forceinline__ ff ff_sqr_u(ff a)
{
    const float p = __fmul_rn(a.hi, a.hi);
    const float e = __fmaf_rn(a.hi, a.hi, -p);
    return { p, __fmaf_rn(__fadd_rn(a.hi, a.hi), a.lo, e) };
}

__device__ __forceinline__ ff ff_sqr_lo(ff a)       // the same with lo^2
{
    const ff s = ff_sqr_u(a);
    return { s.hi, __fmaf_rn(a.lo, a.lo, s.lo) };
}

__device__ __forceinline__ ff ff_add_u(ff a, ff b)
{
    const ff s = ff_two_sum(a.hi, b.hi);
    return { s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)) };
}

// a . b and |a|^2 of 3-vectors
__device__ __forceinline__ ff ff_sum3(ff p, ff q, ff r)
{
    const ff s = ff_two_sum(p.hi, q.hi);
    const ff t = ff_two_sum(s.hi, r.hi);
    return { t.hi, __fadd_rn(__fadd_rn(s.lo, t.lo), __fadd_rn(__fadd_rn(p.lo, q.lo), r.lo)) };
}

__device__ __forceinline__ ff ff_dot3(ff ax, ff ay, ff az, ff bx, ff by, ff bz)
{
    return ff_sum3(ff_mul_u(ax, bx), ff_mul_u(ay, by), ff_mul_u(az, bz));
}

__device__ __forceinline__ ff ff_sqr3(ff x, ff y, ff z) { return ff_sum3(ff_sqr_u(x), ff_sqr_u(y), ff_sqr_u(z)); }

// The rare halves of ff_split_fast and ff_widen, as calls: inlined, the compiler
// turns their branches into predicated instructions that every step issues
// (ff_widen's FP64 conversions and addition, so issued, made the crossers'
// block 1.9x longer).  Zero is not left to them: a planar swarm's z is zero at
// every step.  No FP64 instruction in the split's.
static __device__ __noinline__ ff ff_split_rare(double d)
{
    const unsigned e = ((unsigned)__double2hiint(d) >> 20) & 0x7ffu;
    ff f = ff_split(d);                       // infinite from 2^128 on, for NaN too
    if (e >= 1023u + 128u) f.lo = 0.0f;
    const unsigned m = ((unsigned)__double2hiint(d) << 12) | (unsigned)__double2loint(d);
    if (e == 0x7ffu && m != 0u) f.hi = f.lo = __int_as_float(0x7fc00000);
    return f;
}
static __device__ __noinline__ double ff_widen_rare(float hi, float lo) { return (double)hi + (double)lo; }

// A double as a float-float on the integer and FP32 pipes: hi = d rounded to
// 24 significant bits, lo = the (signed) rest rounded to 24: |d - hi - lo| <
// 2^-49 |d|, for 2^-70 <= |d| < 2^127.  ff_split counts leading zeros to place
// lo; here the conversion instruction does.  Zero and |d| < 2^-70 (where lo's unit
// would leave the float range), |d| >= 2^127, the infinities and NaN (whose
// exponents would wrap into a float's) are rare: they take ff_split_rare.
__device__ __forceinline__ bool split_is_rare(double d)
{
    // both ends in one unsigned comparison, the sign shifted out
    return 2u * (unsigned)__double2hiint(d) - ((1023u - 70u) << 21) >= (127u + 70u) << 21;
}

__device__ __forceinline__ ff split_common(double d)
{
    const unsigned hw = (unsigned)__double2hiint(d), lw = (unsigned)__double2loint(d);
    // exponent and top 23 significand bits in a float's places; rebiasing from
    // 1023 to 127 adds -896 << 23, 0x40000000 modulo 2^32; bit 28 rounds
    const unsigned f = __funnelshift_l(lw, hw, 3);
    const unsigned h = ((f + 0x40000000u + ((lw >> 28) & 1u)) & 0x7fffffffu) | (hw & 0x80000000u);
    // the rest: the low 29 bits, signed, in units of 2^(e - 52); as the top of a
    // 32-bit integer in units of 2^(e - 55), with d's sign
    const float rest = (float)(int)(lw << 3);
    const unsigned unit = (((f & 0x7f800000u) + (0x40000000u - (55u << 23))) & 0x7fffffffu) | (hw & 0x80000000u);
    return { __uint_as_float(h), __fmul_rn(rest, __uint_as_float(unit)) };
}

__device__ __forceinline__ ff ff_split_fast(double d)
{
    if (split_is_rare(d)) return ff_split_rare(d);
    return split_common(d);
}

// A rare one of three components.
__device__ __forceinline__ ff split_uncommon(double d)
{
    if ((((unsigned)__double2hiint(d) & 0x7fffffffu) | (unsigned)__double2loint(d)) == 0u) return { 0.0f, 0.0f };
    return ff_split_rare(d);
}

// Three at once, with one branch for the rare ones.
__device__ __forceinline__ void ff_split3(double x, double y, double z, ff& fx, ff& fy, ff& fz)
{
    fx = split_common(x);
    fy = split_common(y);
    fz = split_common(z);
    if (split_is_rare(x) || split_is_rare(y) || split_is_rare(z)) {
        if (split_is_rare(x)) fx = split_uncommon(x);
        if (split_is_rare(y)) fy = split_uncommon(y);
        if (split_is_rare(z)) fz = split_uncommon(z);
    }
}

// hi + lo as a double on the integer and FP32 pipes, to ~2^-47 of it (lo
// enters in units of 2^-46 of hi's binade), for a renormalised pair: hi widened
// exactly, lo's multiple of the unit added to the magnitude bits.  hi a power
// of two (the sum may fall into the binade below, whose unit is another), zero,
// below 2^-76, infinite or NaN is rare: it takes the FP64 addition.
__device__ __forceinline__ bool widen_is_rare(ff x)
{
    const unsigned b = __float_as_uint(x.hi);
    return (b & 0x007fffffu) == 0u || !(fabsf(x.hi) >= 0x1p-76f);
}

__device__ __forceinline__ double widen_common(ff x)
{
    const unsigned b = __float_as_uint(x.hi);
    // 2^(46 - e) with hi's sign, so that the multiple is relative to hi's; the
    // FMA rounds it to an integer in the last places of 1.5 * 2^23
    const float scale = __uint_as_float(((127u + 46u + 127u) << 23) - (b & 0xff800000u));
    const int k = __float_as_int(__fmaf_rn(x.lo, scale, 12582912.0f)) - 0x4b400000;
    const unsigned hw = ((b & 0x7fffffffu) >> 3) + ((1023u - 127u) << 20) + (b & 0x80000000u);
    return __longlong_as_double((long long)((unsigned long long)hw << 32 | (b << 29)) + ((long long)k << 6));
}

__device__ __forceinline__ double ff_widen(ff x)
{
    if (widen_is_rare(x)) return ff_widen_rare(x.hi, x.lo);
    return widen_common(x);
}

__device__ __forceinline__ double widen_uncommon(ff x)
{
    if (x.hi == 0.0f && x.lo == 0.0f) return 0.0;
    return ff_widen_rare(x.hi, x.lo);
}

__device__ __forceinline__ void ff_widen3(ff x, ff y, ff z, double& dx, double& dy, double& dz)
{
    dx = widen_common(x);
    dy = widen_common(y);
    dz = widen_common(z);
    if (widen_is_rare(x) || widen_is_rare(y) || widen_is_rare(z)) {
        if (widen_is_rare(x)) dx = widen_uncommon(x);
        if (widen_is_rare(y)) dy = widen_uncommon(y);
        if (widen_is_rare(z)) dz = widen_uncommon(z);
    }
}

// 1/x by the special-function unit (~1 unit in the last place)
__device__ __forceinline__ float rcp_approx(float x)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return 1.0f / x;
#endif
}

// e = 1 - x y^2 for the seed y of 1/sqrt(x): the product's leading part cancels
// against 1 inside the first FMA, so each of the three roundings is of a
// number of e's own size (2^-22), below 2^-47
__device__ __forceinline__ float rsqrt_residual(ff x, float y)
{
    const ff y2 = ff_two_prod(y, y);
    return __fmaf_rn(-x.lo, y2.hi, __fmaf_rn(-x.hi, y2.lo, __fmaf_rn(-x.hi, y2.hi, 1.0f)));
}

// 1/sqrt(x) of a float-float, to ~2^-48: y (1 + e/2 + 3e^2/8) with e = 1 - x y^2 as
// a float-float (1 - x.hi y^2.hi is exact, the rest some 2^-24) and y e/2 as an
// exact product
__device__ __forceinline__ ff ff_rsqrt(ff x)
{
    const float y = rsqrtf(x.hi), h = 0.5f * y;
    const ff y2 = ff_two_prod(y, y), t = ff_two_prod(x.hi, y2.hi);
    const ff e = ff_two_sum(__fsub_rn(1.0f, t.hi), -__fmaf_rn(x.lo, y2.hi, __fmaf_rn(x.hi, y2.lo, t.lo)));
    const ff d = ff_two_prod(h, e.hi);
    const ff s = ff_fast_two_sum(y, d.hi);
    return { s.hi, __fadd_rn(s.lo, __fmaf_rn(h, __fmaf_rn(0.75f * e.hi, e.hi, e.lo), d.lo)) };
}

// 1/x of a float-float, the same way: y (1 + e + e^2), e = 1 - x y
__device__ __forceinline__ ff ff_rcp(ff x)
{
    const float y = rcp_approx(x.hi);
    const ff t = ff_two_prod(x.hi, y);
    const ff e = ff_two_sum(__fsub_rn(1.0f, t.hi), -__fmaf_rn(x.lo, y, t.lo));
    const ff d = ff_two_prod(y, e.hi);
    const ff s = ff_fast_two_sum(y, d.hi);
    return { s.hi, __fadd_rn(s.lo, __fmaf_rn(y, __fmaf_rn(e.hi, e.hi, e.lo), d.lo)) };
}

// Constants of a launch's step dt.
struct SmallStepDt {
    ff dt2, dt_half, neg_dt;      // dt^2, dt / 2, -dt
    float th_min = TINY_DRIFT_TH; // the least tau^2 / 2: FAR_DRIFT_TH where the ranges are checked
};

// Constants of the central mass mu and the step dt: mu dt^2 / 2, mu dt.  Rounded
// (ff_split_fast), not truncated: their error is the same at every step of a run,
// and a truncation (7e-15 at most, 1.5e-15 in the mean) is a weaker Sun throughout.
struct SmallStepMu {
    ff muh, mudt;
};

__device__ __forceinline__ SmallStepMu small_step_mu(double mu, double dt)
{
    return { ff_split_fast(0.5 * mu * dt * dt), ff_split_fast(mu * dt) };
}

// What a drift's solution leaves: DRIFT_SMALL, its coefficients f - 1, g - dt, H
// (gd - 1 = -H / r') and fd r'; DRIFT_MEDIUM, its q2, q3 and e = 1 - G1 r0 / dt
// for the G-functions.
struct SmallDrift {
    ff f1, gdt, h, fdr;
};
enum DriftTier : int { DRIFT_GENERAL = 0, DRIFT_SMALL = 1, DRIFT_MEDIUM = 2 };

// R'(w) = 1 + 2X (1+w) c1(x) + 3Y (1+w)^2 2c2(x) in FP32, its reciprocal
__device__ __forceinline__ float kepler_slope_rcp(float x, float y, float s, float s2, float xx)
{
    return rcp_approx(__fmaf_rn(2.0f * x * s, __fmaf_rn(xx, -1.0f / 6.0f, 1.0f),
                                __fmaf_rn(3.0f * y * s2, __fmaf_rn(xx, -1.0f / 12.0f, 1.0f), 1.0f)));
}

// R(w) in float-float from q2 and q3 at w
__device__ __forceinline__ float kepler_residual(ff X, ff Y, float w, ff q2, ff q3, ff& xq)
{
    xq = ff_mul_u(X, q2);
    const ff e1 = ff_two_sum(X.hi, w);
    const ff e2 = ff_two_sum(e1.hi, xq.hi);
    const ff yq = ff_mul_u(Y, q3);
    const ff e3 = ff_two_sum(e2.hi, Y.hi);
    const float lows = __fadd_rn(__fadd_rn(__fadd_rn(e1.lo, e2.lo), __fadd_rn(e3.lo, xq.lo)),
                                 __fadd_rn(__fadd_rn(X.lo, Y.lo), yq.lo));
    return __fadd_rn(__fadd_rn(e3.hi, yq.hi), lows);
}

// Solves one drift from the float-float split of its state, of r0^2 and 1/r0
// (muh = mu dt^2 / 2, mudt = mu dt).  DRIFT_GENERAL (nothing solved) for tau^2 at or
// above the tier's bound, a state not bound beyond the energy's rounding, or a
// value outside the range that float-float covers (run_tile puts a NaN in 1/r0
// where |r|^2 leaves it; a NaN or an infinity in any input leaves tau^2 or the
// energy's A NaN or -infinity, which no comparison below accepts).  The
// decision is each particle's own, so that its path does not depend on the
// particles that share its warp.
//
// MEDIUM: tau^2 up to MEDIUM_DRIFT_TAU2.  There the corrections are too large for a
// float-float velocity, but Kepler's equation can still be solved here: the FP64
// G-functions are T (1 - e), (T^2/2)(1 + q2), (T^3/6)(1 + q3) with T = dt / r0, and
// e, q2, q3 of 0.2 at most.  It spares the general solution's invariants, FP64
// residual and Stumpff series (about 30 FP64 instructions).  An instance of its own:
// with one code for both tiers (the shared half not repeated) the scattered disk
// took 6.19 instead of 6.47 ms, but its registers cost the planet crossers 2 % and
// the ensembles 5 %.  The line at 1e-2: e, q2 and q3 at 2^-46 then change
// r by 2^-55 and v by 2^-53 at most, and the series end below 2^-46.  300,000
// scattered-disk particles x 256 steps, 0.9 % of their drifts here and 0.1 % beyond,
// but spread over the warps: 7.19 -> 6.47 ms (5.15 with tau^2 / 2 down to 2^-34; 5.31
// since the conversions tell both ends of their range and zero apart), error against
// long double 3.1e-15 before and after; 1e6 particles x 64 steps with the learned
// starter 5.94 -> 5.21 ms.
template <bool MEDIUM>
__device__ __forceinline__ int small_drift(ff rx, ff ry, ff rz, ff vx, ff vy, ff vz, ff r2, ff rinv, ff muh, ff mudt,
                                           const SmallStepDt& c, SmallDrift& d)
{
    const ff u = ff_dot3(rx, ry, rz, vx, vy, vz);
    const ff v2 = ff_sqr3(vx, vy, vz);
    // 1/r0^2 from r0^2, not from 1/r0: the square of a float-float drops its lo^2,
    // below its last place and so never rounded up to it -- a bias of 8e-16 in the
    // Sun's pull, which adds up over the steps
    const ff ri2 = ff_rcp(r2);
    const ff m2 = ff_mul_u(muh, ri2);                                 // mu dt^2 / (2 r0^2)
    const ff th = ff_mul_u(m2, rinv);                                 // tau^2 / 2
    const ff b = ff_mul_u(ff_mul_u(c.dt2, ri2), v2);                  // (v dt / r0)^2
    const ff X = ff_mul(ff_mul_u(c.dt_half, ri2), u);
    // A = 2 tau^2 - b and 6 Y = tau^2 - A = b - tau^2
    const ff A = ff_add_u(ff_scale(th, 4.0f), ff_neg(b));
    const ff Y = ff_mul_u(ff_add_u(b, ff_scale(th, -2.0f)), ff_sixth());
    const float a = A.hi, x = X.hi, y = Y.hi;
    const bool inside = th.hi < 0.5f * (MEDIUM ? MEDIUM_DRIFT_TAU2 : SMALL_DRIFT_TAU2) && th.hi > c.th_min &&
                        a > 0x1p-20f * th.hi;
    if (!inside) return DRIFT_GENERAL;

    // FP32: fourth-order start and one Newton step
    float w = __fmaf_rn(x, __fmaf_rn(a, 1.0f / 12.0f, __fmaf_rn(__fmaf_rn(-5.0f, x, 2.0f), x, __fmaf_rn(5.0f, y, -1.0f))), -y);
    float s = 1.0f + w, s2 = s * s, xx = a * s2;
    float rp = kepler_slope_rcp(x, y, s, s2, xx);
    const float res = __fmaf_rn(x * s2, __fmaf_rn(xx, __fmaf_rn(xx, 1.0f / 360.0f, -1.0f / 12.0f), 1.0f),
                                __fmaf_rn(y * s2 * s, __fmaf_rn(xx, -1.0f / 20.0f, 1.0f), w));
    w = __fmaf_rn(-res, rp, w);

    // with z = (1+w)^2 - 1 the float-float residual at w and the second Newton step
    const ff ww = ff_two_prod(w, w);
    ff z = ff_fast_two_sum(2.0f * w, ww.hi);
    z.lo += ww.lo;
    s = 1.0f + w;
    s2 = 1.0f + z.hi;
    xx = a * s2;
    ff q2, q3, xq;
    float dw;
    if constexpr (!MEDIUM) {
        // q2 = z - (A/12) (1 + 2z) + [ -(A/12) z^2 + A^2/360 (1+w)^6 - A^3/20160 (1+w)^8 ],
        // q3 = 3w + 3w^2 + [ w^3 + (1+w)^3 (6c3 - 1) ], the brackets in FP32
        const ff A12 = ff_mul_u(A, ff_twelfth());
        const ff az = ff_mul_u(A12, ff_scale(z, 2.0f));
        const float rest2 = __fmaf_rn(-A12.hi * z.hi, z.hi,
                                      s2 * xx * xx * __fmaf_rn(xx, -1.0f / 20160.0f, 1.0f / 360.0f));
        const ff t1 = ff_two_sum(z.hi, -A12.hi);
        const ff t2 = ff_fast_two_sum(t1.hi, -az.hi);
        q2 = { t2.hi, __fadd_rn(__fadd_rn(__fadd_rn(t1.lo, t2.lo), __fsub_rn(z.lo, A12.lo)), __fsub_rn(rest2, az.lo)) };
        const float w3 = 3.0f * w, ww3 = 3.0f * ww.hi;
        q3 = ff_fast_two_sum(w3, ww3);
        q3.lo = (q3.lo + (__fmaf_rn(3.0f, w, -w3) + __fmaf_rn(3.0f, ww.hi, -ww3))) +
                __fmaf_rn(ww.hi, w, s2 * s * xx * __fmaf_rn(xx, __fmaf_rn(xx, -1.0f / 60480.0f, 1.0f / 840.0f),
                                                           -1.0f / 20.0f));
        dw = -kepler_residual(X, Y, w, q2, q3, xq) * rp;
        q2.lo = __fmaf_rn(2.0f * s, dw, q2.lo);
        q3.lo = __fmaf_rn(3.0f * s2, dw, q3.lo);
        xq.lo = __fmaf_rn(2.0f * s * x, dw, xq.lo);
    } else {
        // the same with every term above 2^-24 of q2, q3 in float-float and the slope
        // taken anew: x = A (1+w)^2, 1 - 2c2 = x/12 (1 - x/30 (1 - x/56 (1 - x/90))),
        // 1 - 6c3 = x/20 (1 - x/42 (1 - x/72))
        rp = kepler_slope_rcp(x, y, s, s2, xx);
        const ff xf = ff_add_u(A, ff_mul_u(A, z));
        ff t = ff_mul_u(xf, ff_30th());
        t.lo = __fmaf_rn(-t.hi * xx * (1.0f / 56.0f), __fmaf_rn(xx, -1.0f / 90.0f, 1.0f), t.lo);
        const ff g = ff_mul_u(xf, ff_twelfth());
        const ff k2 = ff_add_u(g, ff_neg(ff_mul_u(g, t)));            // 1 - 2c2
        q2 = ff_add_u(ff_add_u(z, ff_neg(k2)), ff_neg(ff_mul_u(k2, z)));
        const ff wf = { w, 0.0f };
        const ff s3 = ff_add_u(ff_add_u(z, wf), ff_mul_u(z, wf));     // (1+w)^3 - 1
        ff k3 = ff_mul_u(xf, ff_20th());                              // 1 - 6c3
        k3.lo = __fmaf_rn(-k3.hi * xx * (1.0f / 42.0f), __fmaf_rn(xx, -1.0f / 72.0f, 1.0f), k3.lo);
        q3 = ff_add_u(ff_add_u(s3, ff_neg(k3)), ff_neg(ff_mul_u(k3, s3)));
        dw = -kepler_residual(X, Y, w, q2, q3, xq) * rp;
        // q2' = 2 (1+w) c1, q3' = 3 (1+w)^2 2c2
        const float dq2 = 2.0f * s * __fmaf_rn(xx, __fmaf_rn(xx, 1.0f / 120.0f, -1.0f / 6.0f), 1.0f) * dw;
        q2.lo += dq2;
        q3.lo = __fmaf_rn(3.0f * s2 * __fmaf_rn(xx, -1.0f / 12.0f, 1.0f), dw, q3.lo);
        xq.lo = __fmaf_rn(x, dq2, xq.lo);
    }

    // p = (tau^2 / 6) (1 + q3), e = X + X q2 + p
    const ff o3 = ff_fast_two_sum(1.0f, q3.hi);
    const ff p = ff_mul(ff_mul_u(th, ff_third()), ff{ o3.hi, o3.lo + q3.lo });
    const ff xs = ff_two_sum(x, xq.hi);
    const ff ps = ff_two_sum(xs.hi, p.hi);
    const float el = __fadd_rn(__fadd_rn(xs.lo, ps.lo), __fadd_rn(__fadd_rn(X.lo, xq.lo), p.lo));
    if constexpr (MEDIUM) {
        d.f1 = ff_norm(q2);
        d.gdt = ff_norm(q3);
        d.h = ff_norm(ff{ ps.hi, el });
        return DRIFT_MEDIUM;
    }
    const ff o2 = ff_fast_two_sum(1.0f, q2.hi);
    d.h = ff_mul_u(m2, ff{ o2.hi, o2.lo + q2.lo });
    d.f1 = ff_neg(ff_mul_u(d.h, rinv));
    d.gdt = ff_mul_u(c.neg_dt, p);
    // fd r' = -(mu dt / r0^2) (1 - e)
    const ff os = ff_fast_two_sum(1.0f, -ps.hi);
    d.fdr = ff_mul(ff_neg(ff_mul_u(mudt, ri2)), ff{ os.hi, __fsub_rn(os.lo, el) });
    return DRIFT_SMALL;
}

// The G-functions of a DRIFT_MEDIUM solution, with T = dt / r0 in FP64:
// G1 = T (1 - e), G2 = (T^2 / 2)(1 + q2), G3 = (T^3 / 6)(1 + q3).
__device__ __forceinline__ void medium_gfuns(const SmallDrift& d, double T, double& g1, double& g2, double& g3)
{
    const double h = f64_half(T * T), t3 = T * h * (1.0 / 3.0);
    g1 = fma(-ff_widen(d.h), T, T);
    g2 = fma(ff_widen(d.f1), h, h);
    g3 = fma(ff_widen(d.gdt), t3, t3);
}

}  // namespace glisser
