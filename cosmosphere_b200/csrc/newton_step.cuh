/*
 * newton_step.cuh -- the Newton-Raphson step of one particle, shared by the Newton kernels.
 */
#pragma once

#include "common.cuh"

namespace cosmo {

// Newton-Raphson step of one particle from its un-normalised sums (src/density_base.cu:
// 294-333): rho, d(rho)/dh, the new h (clamped to +-20%) and whether |dh/h| < tolh.
// Returns true while the particle stays unconverged.
__device__ __forceinline__ bool newton_step(double rhoi, double gradhi, double hi, double pmass, double hfact,
                                           double tolh, double& rhoOut, double& gradOut, double& hOut, int& conv)
{
    const double hi1 = 1.0 / hi;
    const double hi31 = hi1 * hi1 * hi1;
    const double hi41 = hi31 * hi1;
    const double rho_i = rhoi * kCnormk * pmass * hi31;
    const double grad_i = gradhi * kCnormk * pmass * hi41;
    if (!(rho_i > 0.0))
    {
        rhoOut = 0.0;
        gradOut = 0.0;
        hOut = hi;
        conv = 0;
        return true;
    }
    const double rhoh_i = pmass * (hfact * hi1) * (hfact * hi1) * (hfact * hi1);
    const double funci = rhoh_i - rho_i;
    const double dhdrhoi = -hi / (3.0 * rhoh_i);
    const double omegai = 1.0 - dhdrhoi * grad_i;
    const double safe = (omegai > 0.0) ? omegai : fabs(omegai + 1e-300);
    const double hraw = hi - funci * dhdrhoi / safe;
    double hnew;
    if (hraw > 1.2 * hi) hnew = 1.2 * hi;
    else if (hraw < 0.8 * hi) hnew = 0.8 * hi;
    else hnew = hraw;
    rhoOut = rho_i;
    gradOut = grad_i;
    hOut = hnew;
    conv = (fabs((hnew - hi) / hi) < tolh) ? 1 : 0;
    return !conv;
}

} // namespace cosmo
