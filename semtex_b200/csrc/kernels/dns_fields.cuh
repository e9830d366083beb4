// The field passes of a DNS step over every velocity component at once
// (asynchronous on the given stream).  Field arguments are nz planes of
// plane_size doubles; D is the np x np derivative matrix on the host.
#pragma once

#include "device.hpp"

namespace stx {

// N[i] of every component i from the physical velocity U (dns/nonlinear.cpp):
// minus the convective form U . grad U_i (form 1), the conservative form
// div(U_i U) (2) or their mean (0).  Tc[i] = dU_i/dz and Tk[i] = d(U_i U_2)/dz
// are the z parts of the two (null where there is none).
struct NonlinearFields {
  int ncom, form;
  const double* U[3];
  const double* Tc[3];
  const double* Tk[3];
  double* N[3];
};
cudaError_t dns_nonlinear_fields(const DevGeom& g, const double* D, const NonlinearFields& a, cudaStream_t st);

// out[i] = sum_q c[q] p[i][q] (waveProp, dns/integrate.cpp:204-239) and
// div = (the divergence of out) inv_dt (setPForce, :242-257).
struct WaveFields {
  int ncom, n, z3;
  double c[6];
  const double* p[3][6];
  double* out[3];
  double* div;
  double inv_dt, beta;
};
cudaError_t dns_wave_fields(const DevGeom& g, const double* D, const WaveFields& a, cudaStream_t st);

// io[i] = alpha io[i] + b dp/dx_i (project, dns/integrate.cpp:260-289), no
// derivative for a component 2 of a 2D flow; the Nyquist planes of clear[i]
// are zeroed.
struct ProjectFields {
  int ncom, z3;
  const double* p;
  double* io[3];
  double* clear[3];
  double alpha, b, beta;
};
cudaError_t dns_project_fields(const DevGeom& g, const double* D, const ProjectFields& a, cudaStream_t st);

}  // namespace stx
