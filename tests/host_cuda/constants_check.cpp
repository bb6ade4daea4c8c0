// C entry over the small-step drift's constants of the central mass, for ctypes.
#include "smallstep.cuh"

using namespace glisser;

extern "C" void sun_constants(int n, const double* mu, const double* dt, float* muh, float* mudt)
{
    for (int i = 0; i < n; i++) {
        const SmallStepMu c = small_step_mu(mu[i], dt[i]);
        muh[2 * i] = c.muh.hi; muh[2 * i + 1] = c.muh.lo;
        mudt[2 * i] = c.mudt.hi; mudt[2 * i + 1] = c.mudt.lo;
    }
}
