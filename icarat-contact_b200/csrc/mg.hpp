// mg.hpp -- geometric multigrid preconditioner and the mixed-precision solve.
#pragma once
#include "problem.hpp"

namespace icb
{
/// coarse planes a thread of the 3D restriction takes: 0 (the default) by its rule,
/// else as many on every grid (option mg_restrict_planes)
int mg_restrict_planes();
void set_mg_restrict_planes(int n);
/// GMG-preconditioned CG in FP64 (precision ICB_FP64) or FP32 inner GMG-PCG
/// inside FP64 defect correction (precision ICB_MIXED).
int solve_multigrid(icb_problem p, const icb_solve_opts &o, const double *b,
                    icb_solve_info *info);
} // namespace icb
