// The separable preconditioner of the pressure and velocity systems (separable.cu).
#pragma once
#include "solver.h"

namespace cuibm {

constexpr int kRowBlocks = 608;  // blocks of the Krylov kernels there at most (four an SM): S.partials holds 4 sums of each
void setup_separable(Context &c, LinearSystem &S);  // S.sep stays null where it does not apply
// digits: the caller has split `in` already (the row kernels of separable.cu)
void launch_separable_apply(Context &c, LinearSystem &S, const double *in, double *out, bool digits = false);
void launch_separable_transposed(Context &c, LinearSystem &S, const TransposeList &T, const double *in, double *out);
void launch_separable_solve(Context &c, LinearSystem &S, const double *b, double *x, bool in_graph);
long long separable_body_launches(const LinearSystem &S, int runs);
double separable_bytes(const LinearSystem &S, int it);
void free_separable(LinearSystem &S);

}  // namespace cuibm
