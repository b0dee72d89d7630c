// One RK stage of the plain FP64 form over the digit-product transforms (stage_f64.cu).
#pragma once

#include "ops.h"

namespace sg {

// z lengths that have digit-product transforms
bool f64_stage_ok(const Plan &P);
// stage o from vin (RK-step start cold) into vout; E: spectra of the unit laplace_z profiles
int f64_stage(Plan &P, const StageParams &sp, int o, const void *const vin[4], const void *const cold[4],
              void *const vout[4], void *pr, void *const E[2]);

// sol_project's pieces with a Dirichlet target on vz: the Poisson potential d and the velocity without its
// gradient, theta's filter beside it when th is given, and the laplace_z coefficients of every column
// (coef[2 * (ky * nxh + kx) + 0, 1]); the harmonic profile on the physical rows, or with its derivative on all
int f64_poisson(Plan &P, void *vx, void *vy, void *vz, void *d, void *th, double2 *coef);
int f64_profile(Plan &P, const double2 *coef, void *prof, void *deriv);

}  // namespace sg
