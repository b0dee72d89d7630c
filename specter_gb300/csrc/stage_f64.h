// One RK stage of the plain FP64 form over the digit-product transforms (stage_f64.cu).
#pragma once

#include "ops.h"

namespace sg {

// z lengths that have digit-product transforms
bool f64_stage_ok(const Plan &P);
// stage o from vin (RK-step start cold) into vout; E: spectra of the unit laplace_z profiles
int f64_stage(Plan &P, const StageParams &sp, int o, const void *const vin[4], const void *const cold[4],
              void *const vout[4], void *pr, void *const E[2]);

}  // namespace sg
