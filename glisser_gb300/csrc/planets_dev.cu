// Device planet WH for ensembles: every system's planets integrated over a
// time block by one warp, lane j holding planet j (the Sun in lane 0), and
// the block's planet log written straight into the buffer the ensemble
// kernel stages by TMA.  Replaces the host planet step (planets.cpp
// PlanetIntegrator::step, restating src/wh.cpp:1027-1067 with the Jacobi
// bookkeeping of :19-43 and :696-756) and the per-block upload of the logs.
//
// Bound: the serial chain of a step.  A block's steps follow one another, a
// system fills a part of one warp, and an FP64 instruction holds its scheduler's
// FP64 unit for 64 cycles however many lanes are active: the kernel's time is
// the FP64 instructions of one step times 64 cycles plus the FP32 and shuffle
// latencies between them, whatever the number of systems, and with few systems
// it is the ensemble's whole block time.  Hence the fewest FP64 instructions:
// the Kepler drift in universal variables (FP32 start, one FP64 pass, where the
// eccentric-anomaly iteration's sin/cos passes took ~700), reciprocal roots from
// the FP32 seed, masses and Jacobi factors divided once per block, a lane per
// vector component and per inverse cube (planet_wh_lanes), and one warp per CTA,
// so that systems spread over the SMs.  Measured, four planets on GB300: 31.4 us
// a step with a lane per planet and the eccentric-anomaly iteration, 8.8 us
// with a lane per planet, 4.6 us with a lane per component.
//
// Prefix sums over planets (Jacobi velocities, heliocentric positions, the
// indirect terms) run sequentially in the host's order, each lane reading the
// others' values by warp shuffles, and this translation unit is compiled
// without FMA contraction; results differ from the host's by rounding.
#include "planets_dev.h"

#include "kepler.cuh"

namespace glisser {
namespace {

constexpr double PI_D = 3.14159265358979323846;
constexpr unsigned FULL = 0xffffffffu;

// Elliptic Kepler drift of a Jacobi orbit (planets.cpp kepler_drift_planet,
// src/wh.cpp:875-957): 0 ok, 1 unbound, 2 not converged in ten passes.
__device__ int kepler_drift_planet(double mu, double dt, double& rx, double& ry, double& rz, double& vx, double& vy,
                                   double& vz)
{
    const double dist = sqrt(rx * rx + ry * ry + rz * rz);
    const double vdotr = vx * rx + vy * ry + vz * rz;
    const double energy = (vx * vx + vy * vy + vz * vz) * 0.5 - mu / dist;
    if (energy >= 0) return 1;
    const double a = -0.5 * mu / energy;
    const double n = sqrt(mu / (a * a * a));
    const double ecosE0 = 1.0 - dist / a;
    const double esinE0 = vdotr / (n * a * a);
    // whole orbits removed as (int)(dt n / pi * 2) turns (the reference's
    // unparenthesised M_2PI, src/types.h:8)
    const double dM = dt * n - (PI_D * 2) * (int)(dt * n / PI_D * 2);
    const double adv = dM / n;
    double dE = dM - esinE0 + esinE0 * cos(dM) + ecosE0 * sin(dM);
    double s = sin(dE), c = cos(dE);
    bool converged = false;
    for (int k = 0; k < 10; k++) {
        const double f = dE - ecosE0 * s + esinE0 * (1. - c) - dM;
        const double fp = 1. - ecosE0 * c + esinE0 * s;
        const double delta = -f / fp;
        if (fabs(delta) < 1e-14) {
            converged = true;
            break;
        }
        dE += delta;
        s = sin(dE);
        c = cos(dE);
    }
    if (!converged) return 2;
    const double fp = 1.0 - ecosE0 * c + esinE0 * s;
    const double ff = 1.0 + a * (c - 1.0) / dist;
    const double gg = adv + (s - dE) / n;
    const double fd = -n * s * a / (dist * fp);
    const double gd = 1.0 + (c - 1.0) / fp;
    const double r0x = rx, r0y = ry, r0z = rz, v0x = vx, v0y = vy, v0z = vz;
    rx = r0x * ff + v0x * gg;
    ry = r0y * ff + v0y * gg;
    rz = r0z * ff + v0z * gg;
    vx = r0x * fd + v0x * gd;
    vy = r0y * fd + v0y * gd;
    vz = r0z * fd + v0z * gd;
    return 0;
}

// The drift in universal variables, for steps that are a modest part of an
// orbit: A = alpha dt^2 / r0^2 and tau^2 = dt^2 mu / r0^3 below 0.25 and |X| below
// 0.15 (X = u dt / 2 r0^2; some thirteen steps an orbit, where the eccentric-
// anomaly iteration always converges too).  Kepler's equation in the
// dimensionless form R(w) = 0 of smallstep.cuh, s = (dt / r0)(1 + w): its
// fourth-order reversion and three FP32 Newton steps leave s within ~1e-7, one
// FP64 evaluation of the G-functions (|x| < 0.4, for inbound orbits at the bounds:
// stumpff_small's next term is 1.4e-16 of c2, which mu G2 / r0 < 0.13 carries into
// the position as 2e-17) with the second-order Newton correction folded in does the
// rest.
// Wider steps, other orbits and values outside a float's range (mu itself, which
// the correction's second-order term takes in FP32: G Msun in cm^3/yr^2 is above
// it) take kepler_drift_planet, whose refusals stay.
constexpr float JACOBI_MU_MAX = 1e37f;       // alpha r0, below 2 mu, stays a float too

__device__ __forceinline__ bool jacobi_start(float t, float u, float rinv, float alpha, float mu_r, float mu, float& w)
{
    const float tau2 = t * t * mu_r;
    const float X = 0.5f * u * rinv * t, A = alpha * t * t, Y = (tau2 - A) * (1.0f / 6.0f);
    w = fmaf(X, fmaf(A, 1.0f / 12.0f, fmaf(fmaf(-5.0f, X, 2.0f), X, fmaf(5.0f, Y, -1.0f))), -Y);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float s = 1.0f + w, s2 = s * s, x = A * s2;
        const float c2 = fmaf(x * (-1.0f / 12.0f), fmaf(x * (-1.0f / 30.0f), fmaf(x, -1.0f / 56.0f, 1.0f), 1.0f), 1.0f);
        const float c3 = fmaf(x * (-1.0f / 20.0f), fmaf(x * (-1.0f / 42.0f), fmaf(x, -1.0f / 72.0f, 1.0f), 1.0f), 1.0f);
        const float R = fmaf(X * s2, c2, fmaf(Y * s2 * s, c3, w));
        const float Rp = fmaf(2.0f * X * s, fmaf(x * (-1.0f / 6.0f), c3, 1.0f), fmaf(3.0f * Y * s2, c2, 1.0f));
        w -= __fdividef(R, Rp);
    }
    return A > 1e-12f && A < 0.25f && tau2 < 0.25f && fabsf(X) < 0.15f && mu < JACOBI_MU_MAX;
}

// The Newton correction ds of s from f, f' and G0, G1: h = f / f' from the FP32
// reciprocal and one correction, ds = -h (1 + f'' h / 2f') with
// f'' = (mu - alpha r0) G1 + u G0 in FP32.
__device__ __forceinline__ double jacobi_correction(double f, double fp, float r0, float u, float mu, float alpha,
                                                    double g0, double g1)
{
    const float yf = __fdividef(1.0f, f32_trunc(fp));
    const double y = f64_of_f32(yf);
    double h = f * y;
    h = fma(fma(-fp, h, f), y, h);
    const float a = 0.5f * f32_trunc(h) * yf * fmaf(fmaf(-alpha, r0, mu), f32_trunc(g1), u * f32_trunc(g0));
    return fma(-h, f64_of_f32(a), -h);
}

__device__ __forceinline__ int kepler_drift_jacobi(double mu, double dt, double& rx, double& ry, double& rz,
                                                   double& vx, double& vy, double& vz)
{
    const double r2 = fma(rx, rx, fma(ry, ry, rz * rz));
    const double rinv = rsqrt_fast(r2);
    const double r0 = r2 * rinv, u = fma(rx, vx, fma(ry, vy, rz * vz)), mu_r = mu * rinv, T = dt * rinv;
    const double alpha = fma(2.0, mu_r, -fma(vx, vx, fma(vy, vy, vz * vz)));
    const float uf = f32_trunc(u), af = f32_trunc(alpha), muf = f32_trunc(mu);
    float w;
    if (!jacobi_start(f32_trunc(T), uf, f32_trunc(rinv), af, f32_trunc(mu_r), muf, w))
        return kepler_drift_planet(mu, dt, rx, ry, rz, vx, vy, vz);
    const double s = fma(T, f64_of_f32(w), T), s2 = s * s, x = alpha * s2;
    double c2, c3;
    stumpff_small(x, c2, c3);
    const double g2 = s2 * c2, g3 = s * (s2 * c3), g1 = fma(-alpha, g3, s), g0 = fma(-alpha, g2, 1.0);
    const double f = fma(r0, g1, fma(u, g2, fma(mu, g3, -dt)));
    const double fp = fma(r0, g0, fma(u, g1, mu * g2));
    const double ds = jacobi_correction(f, fp, f32_trunc(r0), uf, muf, af, g0, g1), hd = 0.5 * ds;
    const double n3 = fma(ds, fma(hd, g1, g2), g3), n2 = fma(ds, fma(hd, g0, g1), g2);
    const double n1 = fma(ds, fma(-alpha * hd, g1, g0), g1);
    const double ff = fma(-mu_r, n2, 1.0), gg = fma(-mu, n3, dt);
    const double nx = fma(ff, rx, gg * vx), ny = fma(ff, ry, gg * vy), nz = fma(ff, rz, gg * vz);
    const double ninv = rsqrt_fast(fma(nx, nx, fma(ny, ny, nz * nz)));
    const double fd = -mu_r * n1 * ninv, gd = fma(-mu * n2, ninv, 1.0);
    vx = fma(fd, rx, gd * vx);
    vy = fma(fd, ry, gd * vy);
    vz = fma(fd, rz, gd * vz);
    rx = nx; ry = ny; rz = nz;
    return 0;
}

__device__ __forceinline__ double inv_cube(double x, double y, double z)
{
    const double i = rsqrt_fast(fma(x, x, fma(y, y, z * z)));
    return i * i * i;
}

// Semi-major axis and eccentricity as the host's to_elements computes them
// (orbits.cpp, restating src/convert.cpp:310-463).
__device__ void elements_ae(double mu, double x, double y, double z, double vx, double vy, double vz, double& a,
                            double& e)
{
    const double prec = 1.0e-13;
    const double hx = y * vz - z * vy, hy = z * vx - x * vz, hz = x * vy - y * vx;
    const double hsq = hx * hx + hy * hy + hz * hz;
    if (!(hsq > prec)) {
        a = sqrt(x * x + y * y + z * z);
        e = HUGE_VAL;
        return;
    }
    const double vsq = vx * vx + vy * vy + vz * vz;
    const double vdotr = x * vx + y * vy + z * vz;
    const double rr = sqrt(x * x + y * y + z * z);
    const double xh = x / rr, yh = y / rr, zh = z / rr;
    const double fac = vsq * rr - mu;
    const double px = fac * xh - vdotr * vx, py = fac * yh - vdotr * vy, pz = fac * zh - vdotr * vz;
    e = sqrt(px * px + py * py + pz * pz) / mu;
    const double energy = vsq / 2.0 - mu / rr;
    a = fabs(energy) < prec ? 0.5 * hsq / mu : -0.5 * mu / energy;
}

__device__ __forceinline__ double shfl(double v, uint32_t lane) { return __shfl_sync(FULL, v, (int)lane); }

// Encounter radii of the block's start state (encounter_radii), body j of the
// system whose arrays start at `first`.
__device__ __forceinline__ void write_radii(const PlanetSysDev& ps, size_t first, uint32_t npl, uint32_t j, double cull,
                                            double rhf, double* rh_out)
{
    if (j >= npl) return;
    const size_t at = first + j;
    double rh = cull;
    if (j >= 1 && fabs(rhf) > 1e-6) {
        double a, e;
        elements_ae(ps.m[first] + ps.m[at], ps.rx[at], ps.ry[at], ps.rz[at], ps.vx[at], ps.vy[at], ps.vz[at], a, e);
        rh = rhf * a * (1 - e) * pow(ps.m[at] / (3 * ps.m[first]), 1. / 3);
    }
    rh_out[at] = rh;
}

// Any number of planets: lane j holds planet j's vectors.
__global__ void __launch_bounds__(32)
    planet_wh_kernel(PlanetSysDev ps, uint32_t npl, uint32_t len, double dt, double cull, double rhf,
                     double* __restrict__ log, size_t stride, double* __restrict__ rh_out)
{
    const uint32_t s = blockIdx.x;
    const uint32_t j = threadIdx.x & 31u;
    const bool body = j < npl;
    const bool pl = body && j >= 1;
    const size_t at = (size_t)s * npl + (body ? j : 0);
    double rx = 0, ry = 0, rz = 0, vx = 0, vy = 0, vz = 0, ax = 0, ay = 0, az = 0, jx = 0, jy = 0, jz = 0;
    double m = 0, eta = 1;
    if (body) {
        rx = ps.rx[at]; ry = ps.ry[at]; rz = ps.rz[at];
        vx = ps.vx[at]; vy = ps.vy[at]; vz = ps.vz[at];
        ax = ps.ax[at]; ay = ps.ay[at]; az = ps.az[at];
        jx = ps.jx[at]; jy = ps.jy[at]; jz = ps.jz[at];
        m = ps.m[at];
        eta = ps.eta[at];
    }
    const double m0 = shfl(m, 0);
    const double eta_prev = shfl(eta, j >= 1 ? j - 1 : 0);

    write_radii(ps, (size_t)s * npl, npl, j, cull, rhf, rh_out);

    const double hdt = dt / 2;
    uint32_t status = 0;
    // the masses' factors of the step, once per block
    const double rcp_eta = 1.0 / eta_prev, mu_j = m0 * eta / eta_prev, f_j = m / eta, g_j = m * m0 / eta_prev;
    double* rec = log + (size_t)s * stride;
    for (uint32_t k = 0; k < len; k++, rec += 3 * (size_t)npl) {
        if (pl) {
            vx += ax * hdt; vy += ay * hdt; vz += az * hdt;
        }
        // heliocentric -> Jacobi velocities (psum over planets 1..j-1)
        double wx = vx, wy = vy, wz = vz;
        {
            const double px = vx * m, py = vy * m, pz = vz * m;
            double sx = 0, sy = 0, sz = 0;
            for (uint32_t q = 1; q + 1 < npl; q++) {
                const double tx = shfl(px, q), ty = shfl(py, q), tz = shfl(pz, q);
                if (q < j) {
                    sx += tx; sy += ty; sz += tz;
                }
            }
            if (pl && j >= 2) {
                wx = vx - sx * rcp_eta; wy = vy - sy * rcp_eta; wz = vz - sz * rcp_eta;
            }
        }
        // Kepler drift of each Jacobi orbit
        if (pl) {
            const int rc = kepler_drift_jacobi(mu_j, dt, jx, jy, jz, wx, wy, wz);
            if (rc && !status) status = 0x100u * j + (uint32_t)rc;
        }
        // Jacobi -> heliocentric
        {
            const double ux = jx * f_j, uy = jy * f_j, uz = jz * f_j;
            const double qx = wx * f_j, qy = wy * f_j, qz = wz * f_j;
            double rsx = 0, rsy = 0, rsz = 0, vsx = 0, vsy = 0, vsz = 0;
            for (uint32_t q = 1; q + 1 < npl; q++) {
                const double a1 = shfl(ux, q), a2 = shfl(uy, q), a3 = shfl(uz, q);
                const double b1 = shfl(qx, q), b2 = shfl(qy, q), b3 = shfl(qz, q);
                if (q < j) {
                    rsx += a1; rsy += a2; rsz += a3;
                    vsx += b1; vsy += b2; vsz += b3;
                }
            }
            if (pl) {
                if (j == 1) {
                    rx = jx; ry = jy; rz = jz; vx = wx; vy = wy; vz = wz;
                } else {
                    rx = jx + rsx; ry = jy + rsy; rz = jz + rsz;
                    vx = wx + vsx; vy = wy + vsy; vz = wz + vsz;
                }
            }
        }
        // accelerations and h0 (PlanetIntegrator::accelerations)
        double invh = 0, invj = 0;
        if (pl) {
            invh = inv_cube(rx, ry, rz);
            invj = inv_cube(jx, jy, jz);
        }
        double cx = 0, cy = 0, cz = 0;
        const double gh = pl ? m * invh : 0.0;
        const double hx = rx * gh, hy = ry * gh, hz = rz * gh;
        for (uint32_t q = 2; q < npl; q++) {
            cx -= shfl(hx, q); cy -= shfl(hy, q); cz -= shfl(hz, q);
        }
        double h0x = cx, h0y = cy, h0z = cz;
        if (npl > 1) {
            h0x -= shfl(hx, 1); h0y -= shfl(hy, 1); h0z -= shfl(hz, 1);
        }
        ax = cx; ay = cy; az = cz;
        if (pl && j >= 2) {
            ax += (jx * invj - rx * invh) * m0;
            ay += (jy * invj - ry * invh) * m0;
            az += (jz * invj - rz * invh) * m0;
        }
        {
            const double g = pl ? g_j * invj : 0.0;
            const double ux = jx * g, uy = jy * g, uz = jz * g;
            double sx = 0, sy = 0, sz = 0;
            for (uint32_t q = 2; q < npl; q++) {
                const double a1 = shfl(ux, q), a2 = shfl(uy, q), a3 = shfl(uz, q);
                if (q <= j) {
                    sx += a1; sy += a2; sz += a3;
                }
            }
            if (pl && j >= 2) {
                ax += sx; ay += sy; az += sz;
            }
        }
        // direct planet-planet terms, each planet's sources in ascending order
        for (uint32_t q = 1; q < npl; q++) {
            const double dx = shfl(rx, q) - rx, dy = shfl(ry, q) - ry, dz = shfl(rz, q) - rz, mq = shfl(m, q);
            if (!pl || q == j) continue;
            const double g = mq * inv_cube(dx, dy, dz);
            ax += dx * g; ay += dy * g; az += dz * g;
        }
        if (pl) {
            vx += ax * hdt; vy += ay * hdt; vz += az * hdt;
            rec[3 * j] = rx; rec[3 * j + 1] = ry; rec[3 * j + 2] = rz;
        }
        if (j == 0) {
            rec[0] = h0x; rec[1] = h0y; rec[2] = h0z;
        }
    }
    if (body) {
        ps.rx[at] = rx; ps.ry[at] = ry; ps.rz[at] = rz;
        ps.vx[at] = vx; ps.vy[at] = vy; ps.vz[at] = vz;
        ps.ax[at] = ax; ps.ay[at] = ay; ps.az[at] = az;
        ps.jx[at] = jx; ps.jy[at] = jy; ps.jz[at] = jz;
    }
    // first failing planet of the system
    const unsigned bad = __ballot_sync(FULL, status != 0);
    if (bad && j == (uint32_t)(__ffs(bad) - 1)) ps.status[s] = status;
}

// One to five planets: a lane per vector component.
//
// Lane l of each half of the warp holds component c = l % 3 of planet l / 3 + 1
// (both halves the same state), so a vector operation is one instruction, not
// three; scalars that are needed together (r.r, r.v, v.v; r0, mu/r0, dt/r0; the
// two Stumpff series; f and f'; the folded G-functions) are computed on the
// three lanes of a planet at once, each lane its own; positions and velocities
// return to heliocentric on the two halves at once; and every inverse cube of
// the accelerations -- heliocentric, Jacobi, pairs -- has a lane.  89 FP64
// instructions a step where a lane per planet takes ~190.
__device__ __forceinline__ double pick3(uint32_t c, double a0, double a1, double a2)
{
    return c == 0 ? a0 : c == 1 ? a1 : a2;
}

template <int NP>
__global__ void __launch_bounds__(32)
    planet_wh_lanes(PlanetSysDev ps, uint32_t len, double dt, double cull, double rhf, double* __restrict__ log,
                    size_t stride, double* __restrict__ rh_out)
{
    static_assert(NP >= 1 && NP <= 5, "three lanes per planet in half a warp");
    constexpr uint32_t NPL = NP + 1;
    const uint32_t s = blockIdx.x, lane = threadIdx.x & 31u, half = lane >> 4, l = lane & 15u;
    const uint32_t p = l < 3u * NP ? l / 3u : 0, c = l < 3u * NP ? l % 3u : 0;
    const uint32_t base = (lane & 16u) + 3u * p;          // the planet's first lane in this half
    const bool active = l < 3u * NP;
    const size_t first = (size_t)s * NPL, at = first + p + 1;
    write_radii(ps, first, NPL, lane, cull, rhf, rh_out);

    double r = pick3(c, ps.rx[at], ps.ry[at], ps.rz[at]), v = pick3(c, ps.vx[at], ps.vy[at], ps.vz[at]);
    double a = pick3(c, ps.ax[at], ps.ay[at], ps.az[at]), jr = pick3(c, ps.jx[at], ps.jy[at], ps.jz[at]);
    const double m0 = ps.m[first], m = ps.m[at], eta = ps.eta[at], eta_prev = ps.eta[at - 1];
    const double rcp_eta = 1.0 / eta_prev, mu = m0 * eta / eta_prev, f_j = m / eta;
    // the step's m / |r|^3 of this half: m for the heliocentric terms, m m0 / eta
    // for the Jacobi ones
    const double g_half = half ? m * m0 / eta_prev : m;
    const double hdt = dt / 2;
    const float muf = f32_trunc(mu);
    // Horner coefficients of this lane's Stumpff series: c3 on lane 1 of a planet
    const bool third = c == 1;
    const double k6 = third ? 1.0 / 1307674368000.0 : 1.0 / 87178291200.0,
                 k5 = third ? -1.0 / 6227020800.0 : -1.0 / 479001600.0,
                 k4 = third ? 1.0 / 39916800.0 : 1.0 / 3628800.0, k3 = third ? -1.0 / 362880.0 : -1.0 / 40320.0,
                 k2 = third ? 1.0 / 5040.0 : 1.0 / 720.0, k1 = third ? -1.0 / 120.0 : -1.0 / 24.0,
                 k0 = third ? 1.0 / 6.0 : 0.5;
    // the lane's inverse cube: heliocentric planet, Jacobi planet, or pair (i < k)
    const bool jac = lane >= NP && lane < 2u * NP;
    uint32_t ci = lane < NP ? lane : jac ? lane - NP : 0, ck = ci;
    const bool pair = lane >= 2u * NP && lane < 2u * NP + NP * (NP - 1) / 2;
    if (pair) {
        uint32_t q = lane - 2u * NP;
        for (ci = 0; q >= NP - 1 - ci; ci++) q -= NP - 1 - ci;
        ck = ci + 1 + q;
    }
    uint32_t status = 0;
    double* rec = log + (size_t)s * stride;
    for (uint32_t step = 0; step < len; step++, rec += 3 * (size_t)NPL) {
        v = fma(a, hdt, v);
        // heliocentric -> Jacobi velocities
        double w = v;
        if constexpr (NP > 1) {
            const double pm = v * m;
            double sum = 0;
#pragma unroll
            for (uint32_t q = 0; q + 1 < NP; q++) {
                const double t = shfl(pm, 3u * q + c);
                if (q < p) sum += t;
            }
            if (p > 0) w = fma(-sum, rcp_eta, v);
        }
        // Kepler drift of each Jacobi orbit
        const double r_0 = shfl(jr, base), r_1 = shfl(jr, base + 1), r_2 = shfl(jr, base + 2);
        const double w_0 = shfl(w, base), w_1 = shfl(w, base + 1), w_2 = shfl(w, base + 2);
        double nr, nw;
        {
            const bool cv = c == 2, cr = c == 0;      // r.r on lane 0, r.v on lane 1, v.v on lane 2
            const double dot = fma(cv ? w_0 : r_0, cr ? r_0 : w_0,
                                   fma(cv ? w_1 : r_1, cr ? r_1 : w_1, (cv ? w_2 : r_2) * (cr ? r_2 : w_2)));
            const double r2 = shfl(dot, base), u = shfl(dot, base + 1), v2 = shfl(dot, base + 2);
            const double rinv = rsqrt_fast(r2);
            const double by_r = pick3(c, r2, mu, dt) * rinv;
            const double r0 = shfl(by_r, base), mu_r = shfl(by_r, base + 1), T = shfl(by_r, base + 2);
            const double alpha = fma(2.0, mu_r, -v2);
            const float uf = f32_trunc(u), af = f32_trunc(alpha);
            float wf;
            const bool inside = jacobi_start(f32_trunc(T), uf, f32_trunc(rinv), af, f32_trunc(mu_r), muf, wf);
            const double sv = fma(T, f64_of_f32(wf), T), s2 = sv * sv, x = alpha * s2;
            double h = fma(x, k6, k5);
            h = fma(x, h, k4);
            h = fma(x, h, k3);
            h = fma(x, h, k2);
            h = fma(x, h, k1);
            h = fma(x, h, k0);
            const double sh = s2 * h;
            const double g2 = shfl(sh, base), g3 = shfl(sv * sh, base + 1);
            const double e01 = fma(-alpha, cr ? g2 : g3, cr ? 1.0 : sv);
            const double g0 = shfl(e01, base), g1 = shfl(e01, base + 1);
            const double ffp = fma(r0, cr ? g1 : g0, fma(u, cr ? g2 : g1, fma(mu, cr ? g3 : g2, cr ? -dt : 0.0)));
            const double f = shfl(ffp, base), fp = shfl(ffp, base + 1);
            const double ds = jacobi_correction(f, fp, f32_trunc(r0), uf, muf, af, g0, g1), hd = 0.5 * ds;
            const double ah = -alpha * hd;
            const double gn = fma(ds, fma(cr ? ah : hd, third ? g0 : g1, pick3(c, g0, g1, g2)), pick3(c, g1, g2, g3));
            const double n1 = shfl(gn, base), n2 = shfl(gn, base + 1), n3 = shfl(gn, base + 2);
            const double fg = fma(cr ? -mu_r : -mu, cr ? n2 : n3, cr ? 1.0 : dt);
            nr = fma(shfl(fg, base), jr, shfl(fg, base + 1) * w);
            const double x_0 = shfl(nr, base), x_1 = shfl(nr, base + 1), x_2 = shfl(nr, base + 2);
            const double ninv = rsqrt_fast(fma(x_0, x_0, fma(x_1, x_1, x_2 * x_2)));
            const double fgd = fma((cr ? -mu_r : -mu) * (cr ? n1 : n2), ninv, cr ? 0.0 : 1.0);
            nw = fma(shfl(fgd, base), jr, shfl(fgd, base + 1) * w);
            if (!inside) {
                double x0 = r_0, x1 = r_1, x2 = r_2, y0 = w_0, y1 = w_1, y2 = w_2;
                const int rc = kepler_drift_planet(mu, dt, x0, x1, x2, y0, y1, y2);
                if (rc && !status) status = 0x100u * (p + 1) + (uint32_t)rc;
                nr = pick3(c, x0, x1, x2);
                nw = pick3(c, y0, y1, y2);
            }
        }
        jr = nr;
        // Jacobi -> heliocentric: positions on the lower half, velocities on the upper
        {
            const double q_own = half ? nw : nr;
            double h = q_own;
            if constexpr (NP > 1) {
                const double uq = q_own * f_j;
                double sum = 0;
#pragma unroll
                for (uint32_t q = 0; q + 1 < NP; q++) {
                    const double t = shfl(uq, (lane & 16u) + 3u * q + c);
                    if (q < p) sum += t;
                }
                if (p > 0) h = q_own + sum;
            }
            r = shfl(h, l < 3u * NP ? l : 0);
            v = shfl(h, 16u + (l < 3u * NP ? l : 0));
        }
        // accelerations and h0: the inverse cubes
        double gx, gy, gz, i3;
        {
            const double a_0 = shfl(r, 3u * ci), a_1 = shfl(r, 3u * ci + 1), a_2 = shfl(r, 3u * ci + 2);
            const double b_0 = shfl(r, 3u * ck), b_1 = shfl(r, 3u * ck + 1), b_2 = shfl(r, 3u * ck + 2);
            const double j_0 = shfl(jr, 3u * ci), j_1 = shfl(jr, 3u * ci + 1), j_2 = shfl(jr, 3u * ci + 2);
            const double d_0 = pair ? b_0 - a_0 : jac ? j_0 : a_0, d_1 = pair ? b_1 - a_1 : jac ? j_1 : a_1,
                         d_2 = pair ? b_2 - a_2 : jac ? j_2 : a_2;
            const double i = rsqrt_fast(fma(d_0, d_0, fma(d_1, d_1, d_2 * d_2)));
            i3 = i * i * i;
            gx = d_0 * i3; gy = d_1 * i3; gz = d_2 * i3;
        }
        const double invh = shfl(i3, p), invj = shfl(i3, NP + p);
        // heliocentric pulls m r / |r|^3 (lower half) and the Jacobi terms (upper)
        const double term = (half ? jr : r) * (g_half * (half ? invj : invh));
        // minus the pulls of planets 2 .. (lower), the Jacobi terms of planets 2 .. this one (upper)
        double sum = 0;
#pragma unroll
        for (uint32_t q = 1; q < NP; q++) {
            const double t = shfl(term, (lane & 16u) + 3u * q + c);
            if (!half || q <= p) sum += half ? t : -t;
        }
        const double common = shfl(sum, l < 3u * NP ? l : 0);
        const double h0 = common - shfl(term, c);
        a = common;
        if constexpr (NP > 1) {
            const double accum = shfl(sum, 16u + (l < 3u * NP ? l : 0));
            if (p > 0) a = fma(fma(jr, invj, -(r * invh)), m0, common) + accum;
            // direct planet-planet terms, each planet's sources in ascending order
#pragma unroll
            for (uint32_t k = 0; k < NP - 1; k++) {
                const uint32_t q = k + (k >= p ? 1u : 0u), lo = q < p ? q : p, hi = q < p ? p : q;
                const uint32_t src = 2u * NP + lo * (2u * NP - lo - 1u) / 2u + (hi - lo - 1u);
                const double g = pick3(c, shfl(gx, src), shfl(gy, src), shfl(gz, src));
                const double mq = shfl(m, 3u * q);
                a = fma(q < p ? -mq : mq, g, a);
            }
        }
        v = fma(a, hdt, v);
        if (active && !half) {
            rec[3 * (p + 1) + c] = r;
            if (p == 0) rec[c] = h0;
        }
    }
    if (active && !half) {
        double* const out[4][3] = { { ps.rx, ps.ry, ps.rz }, { ps.vx, ps.vy, ps.vz }, { ps.ax, ps.ay, ps.az },
                                    { ps.jx, ps.jy, ps.jz } };
        const double val[4] = { r, v, a, jr };
#pragma unroll
        for (int k = 0; k < 4; k++) (c == 0 ? out[k][0] : c == 1 ? out[k][1] : out[k][2])[at] = val[k];
    }
    // first failing planet of the system
    const unsigned bad = __ballot_sync(FULL, status != 0);
    if (bad && lane == (uint32_t)(__ffs(bad) - 1)) ps.status[s] = status;
}

}  // namespace

cudaError_t launch_planet_wh(const PlanetSysDev& ps, uint32_t systems, uint32_t npl, uint32_t len, double dt,
                             double cull_radius, double rh_factor, double* log, size_t log_stride, double* rh,
                             cudaStream_t stream)
{
    if (npl < 1 || npl > PLANET_WH_MAX_NPL) return cudaErrorInvalidValue;
    if (systems == 0) return cudaSuccess;
#define GLISSER_PLANET_WH(n)                                                                                      \
    planet_wh_lanes<n><<<systems, 32, 0, stream>>>(ps, len, dt, cull_radius, rh_factor, log, log_stride, rh)
    switch (npl) {
    case 2: GLISSER_PLANET_WH(1); break;
    case 3: GLISSER_PLANET_WH(2); break;
    case 4: GLISSER_PLANET_WH(3); break;
    case 5: GLISSER_PLANET_WH(4); break;
    case 6: GLISSER_PLANET_WH(5); break;
    default:
        planet_wh_kernel<<<systems, 32, 0, stream>>>(ps, npl, len, dt, cull_radius, rh_factor, log, log_stride, rh);
    }
#undef GLISSER_PLANET_WH
    return cudaGetLastError();
}

}  // namespace glisser
