// When the BiCGStab kernels that predict their scalars (krylov.cu, krylov_small.cu) have to restart.
//
// On convective systems (rp, r) falls to the round-off of its own terms long before r does, and the
// iteration goes on with noise for rho.  That is harmless until rho comes out almost zero: the next
// beta goes with 1 / rho and throws r up by orders of magnitude, for good.  Summed over the cells,
// rho is a multiple of its terms' last place, such a rho is an exact zero, the next direction is
// NaN and the solve restarts from the true residual; predicted as (rp, s) - omega (rp, t) it is an ordinary
// small number.  So a rho below BI_FLOOR |rp| |r| restarts the process explicitly.
//
// Of 280 upwind convection-diffusion systems each on 64x64, 20x20x20 and 40x36x30 cells (Peclet numbers
// to 1000, lognormal conductances) these reach 1e-9 within 4000 iterations: 255, 225 and 156
// with rho summed over the cells, 176, 194 and 128 predicted without this rule, 266, 221 and 156 with it.  In 120
// such systems on the CPU floors from 1e-18 to 1e-16 converge alike; from 1e-14 on restarts come too often.
//
// Large lattices need it most: the p' systems of a sphere in a channel, one step from rest (six solves to
// 1e-8), iterations with rho summed and predicted with the rule: 240x160x164 21,357 and 16,315, 288x192x192 34,508 and
// 21,447, 384x256x256 56,811 and 33,596 (1.74 and 1.04 ms each); without the rule the first two end
// at maxit with relative residuals above 1.
#pragma once
#include "common.cuh"

namespace cb {

constexpr double BI_FLOOR = 3.4694469519536142e-18;   // 2^-58

// rho = (rp, r), rp2 = (rp, rp), rr = (r, r).  The squares decide nearly always; the roots where they come close,
// underflow or overflow.
__device__ __forceinline__ bool bi_sound(double rho, double rp2, double rr) {
    return rho * rho > 2. * BI_FLOOR * BI_FLOOR * (rp2 * fabs(rr)) || fabs(rho) > BI_FLOOR * (sqrt(rp2) * sqrt(fabs(rr)));
}

}  // namespace cb
