// Direct solve of the FP64 coarsest level by its planes (coarse_direct.cu).
#pragma once
#include "common.cuh"

struct pmgb_solver;

namespace pmgb {

struct DirectState;

// Device bytes of a level's factors and work, 0 where it does not fit.
size_t direct_bytes(Grid g);
// Factors the reference's band matrix of the coarsest level: 1; 0 where it does
// not fit, is not positive definite or is no 27-point operator; -1 (an error)
// where a wait of the factor ran out.
int direct_prepare(pmgb_solver* s);
int launch_direct_solve(pmgb_solver* s, cudaStream_t st, const double* b, double* x);
void direct_destroy(DirectState* d);

}  // namespace pmgb
