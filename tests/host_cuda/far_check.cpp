// C entry over the small-step drift with the kernels' lower bound, for ctypes.
#include "smallstep.cuh"

using namespace glisser;

static ff ff_of(double d) { const float h = (float)d; return { h, (float)(d - (double)h) }; }

// One drift of each state (rv [n][6]) in place; ok[i] = 0 outside the domain.
extern "C" void drift_far(int n, double dt, double mu, double* rv, int* ok)
{
    const SmallStepDt c = { ff_of(dt * dt), ff_of(0.5 * dt), ff_of(-dt), FAR_DRIFT_TH };
    const SmallStepMu m = small_step_mu(mu, dt);
    for (int i = 0; i < n; i++) {
        double* r = rv + 6 * i;
        double* v = r + 3;
        ff f[3], w[3], u[3];
        ff_split3(r[0], r[1], r[2], f[0], f[1], f[2]);
        ff_split3(v[0], v[1], v[2], w[0], w[1], w[2]);
        const ff r2 = ff_split_fast(std::fma(r[0], r[0], std::fma(r[1], r[1], r[2] * r[2])));
        SmallDrift d;
        ok[i] = small_drift<false>(f[0], f[1], f[2], w[0], w[1], w[2], r2, ff_rsqrt(r2), m.muh, m.mudt, c, d) == DRIFT_SMALL;
        if (!ok[i]) continue;
        double x[3];
        for (int k = 0; k < 3; k++) u[k] = ff_norm(ff_add_u(ff_mul_u(d.f1, f[k]), ff_mul_u(d.gdt, w[k])));
        ff_widen3(u[0], u[1], u[2], x[0], x[1], x[2]);
        for (int k = 0; k < 3; k++) r[k] += std::fma(dt, v[k], x[k]);
        const ff n2 = ff_split_fast(std::fma(r[0], r[0], std::fma(r[1], r[1], r[2] * r[2])));
        const ff ri = ff_rsqrt(n2), gd1 = ff_neg(ff_mul_u(d.h, ri)), fd = ff_mul_u(d.fdr, ri);
        for (int k = 0; k < 3; k++) u[k] = ff_norm(ff_add_u(ff_mul_u(fd, f[k]), ff_mul_u(gd1, w[k])));
        ff_widen3(u[0], u[1], u[2], x[0], x[1], x[2]);
        for (int k = 0; k < 3; k++) v[k] += x[k];
    }
}
