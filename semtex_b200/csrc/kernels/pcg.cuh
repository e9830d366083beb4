// Jacobi-preconditioned conjugate gradients on the globally numbered
// vectors of every plane.
#pragma once

#include "device.hpp"

namespace stx {

// Vectors of plane k at v + k vstride: [0, nglobal) element-boundary nodes,
// then nel blocks of nint interior nodes in boundary-major order.
struct PcgVectors {
  double* r;   // assembled right-hand side on entry, residual on exit
  double* x;   // initial guess on entry, solution on exit
  double* q;   // scratch
  double* p0;  // scratch
  double* p1;  // scratch
  double* scal;  // scratch, pcg_scalar_doubles(nz)
  int vstride, npts;
  int2* out;   // [nz] (iterations, 1 when step_max was reached); entries of planes not solved are not written
};

size_t pcg_scalar_doubles(int nz);

// Iterate every plane to its own stopping test.  Asynchronous on st, unless
// the iteration runs as launches (then the host reads back every eight
// iterations whether a plane is still at work).
cudaError_t pcg_iterate(const DevGeom& g, const DevNumbering& N, const DevModal& S, const PcgVectors& v,
                        double tol_rel, int step_max, cudaStream_t st);

}  // namespace stx
