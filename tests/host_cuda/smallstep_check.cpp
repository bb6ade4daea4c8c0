// C entries over the device routines of smallstep.cuh, for ctypes.
#include "smallstep.cuh"

using namespace glisser;

static ff ff_of(double d) { const float h = (float)d; return { h, (float)(d - (double)h) }; }

extern "C" {

void split(int n, const double* d, float* hi, float* lo)
{
    for (int i = 0; i < n; i++) { const ff x = ff_split_fast(d[i]); hi[i] = x.hi; lo[i] = x.lo; }
}

void widen(int n, const float* hi, const float* lo, double* d)
{
    for (int i = 0; i < n; i++) d[i] = ff_widen(ff{ hi[i], lo[i] });
}

void inverses(int n, const double* x, float* sh, float* sl, float* rh, float* rl)
{
    for (int i = 0; i < n; i++) {
        const ff f = ff_split_fast(x[i]), s = ff_rsqrt(f), r = ff_rcp(f);
        sh[i] = s.hi; sl[i] = s.lo; rh[i] = r.hi; rl[i] = r.lo;
    }
}

// One drift of each state (rv [n][6]) in place, as the time-block kernel applies
// it; ok[i] = 0 and the state untouched outside the small-step domain.
void drift(int n, double dt, double mu, double* rv, int* ok)
{
    const SmallStepDt c = { ff_of(dt * dt), ff_of(0.5 * dt), ff_of(-dt) };
    const ff muh = ff_split_fast(0.5 * mu * dt * dt), mudt = ff_split_fast(mu * dt);
    for (int i = 0; i < n; i++) {
        double* r = rv + 6 * i;
        double* v = r + 3;
        ff f[3], w[3];
        for (int k = 0; k < 3; k++) { f[k] = ff_split_fast(r[k]); w[k] = ff_split_fast(v[k]); }
        const ff r2 = ff_split_fast(std::fma(r[0], r[0], std::fma(r[1], r[1], r[2] * r[2])));
        SmallDrift d;
        ok[i] = small_drift<false>(f[0], f[1], f[2], w[0], w[1], w[2], r2, ff_rsqrt(r2), muh, mudt, c, d) == DRIFT_SMALL;
        if (!ok[i]) continue;
        for (int k = 0; k < 3; k++)
            r[k] += std::fma(dt, v[k], ff_widen(ff_norm(ff_add_u(ff_mul_u(d.f1, f[k]), ff_mul_u(d.gdt, w[k])))));
        const ff n2 = ff_split_fast(std::fma(r[0], r[0], std::fma(r[1], r[1], r[2] * r[2])));
        const ff ri = ff_rsqrt(n2), gd1 = ff_neg(ff_mul_u(d.h, ri)), fd = ff_mul_u(d.fdr, ri);
        for (int k = 0; k < 3; k++) v[k] += ff_widen(ff_norm(ff_add_u(ff_mul_u(fd, f[k]), ff_mul_u(gd1, w[k]))));
    }
}

// The G-functions of each state's drift (g [n][3]) by the medium solution;
// tier[i] is what the two tiers returned.
void gfuns_medium(int n, double dt, double mu, const double* rv, int* tier, double* g)
{
    const SmallStepDt c = { ff_of(dt * dt), ff_of(0.5 * dt), ff_of(-dt) };
    const ff muh = ff_split_fast(0.5 * mu * dt * dt), mudt = ff_split_fast(mu * dt);
    for (int i = 0; i < n; i++) {
        const double* r = rv + 6 * i;
        const double* v = r + 3;
        ff f[3], w[3];
        for (int k = 0; k < 3; k++) { f[k] = ff_split_fast(r[k]); w[k] = ff_split_fast(v[k]); }
        const double r2d = std::fma(r[0], r[0], std::fma(r[1], r[1], r[2] * r[2]));
        const ff r2 = ff_split_fast(r2d);
        SmallDrift d;
        const ff ri = ff_rsqrt(r2);
        tier[i] = small_drift<false>(f[0], f[1], f[2], w[0], w[1], w[2], r2, ri, muh, mudt, c, d);
        if (tier[i] == DRIFT_GENERAL) tier[i] = small_drift<true>(f[0], f[1], f[2], w[0], w[1], w[2], r2, ri, muh, mudt, c, d);
        if (tier[i] == DRIFT_MEDIUM) medium_gfuns(d, dt / std::sqrt(r2d), g[3 * i], g[3 * i + 1], g[3 * i + 2]);
    }
}

}
