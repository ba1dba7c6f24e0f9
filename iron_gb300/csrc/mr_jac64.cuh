// mr_jac64.cuh -- FP64 element Jacobians of the Q2/Q1 Mooney-Rivlin element (mr_jac64.cu).
#pragma once

#include "gfe_internal.cuh"

namespace mr64 {

// Element matrices Kel[e][89][89] of the elements elems[0..n_elem) in FP64; exact: the consistent
// tangent, else Iron's analytic Jacobian.  Allocates and frees its Gauss-point blocks on `s`; adds the
// kernels launched to *launches.
int element_matrices(bool exact, int32_t n_elem, const int32_t* elems, const int32_t* eq2, const int32_t* elin,
                     int32_t nq2, const double* xg, const double* dep, const double* cpar, double* Kel,
                     cudaStream_t s, unsigned* err, int* launches);

}  // namespace mr64
