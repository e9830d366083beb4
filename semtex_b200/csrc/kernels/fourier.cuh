// z-direction real DFTs of batches of fields, with the z-derivative and the
// 3/2-rule padding of the DNS step folded in.
#pragma once

#include "device.hpp"

namespace stx {

// Up to kZBatch fields transformed by one launch.
constexpr int kZBatch = 4;
struct ZBatch {
  int count = 0;
  const double* in[kZBatch];
  const double* mul[kZBatch];  // z_product_dz: the second factor
  double* out[kZBatch];
  double* dz[kZBatch];         // z_inverse_dz: the z-derivative
  void add(const double* i, double* o, const double* m = nullptr, double* d = nullptr) {
    in[count] = i;
    out[count] = o;
    mul[count] = m;
    dz[count++] = d;
  }
};

// Whether the batched transforms below cover lines of n points (n even, of
// prime factors 2, 3, 5 and 7, n > 2, within the shared memory); otherwise
// z_transform and separate passes apply.
bool z_batch_supported(int n);

// out planes [0, nout) = the packed spectrum of in's n planes, scaled by 1/n
// (out may be in).
cudaError_t z_forward(const ZBatch& b, int n, int nout, int plane_size, const double* twiddle, cudaStream_t st,
                      bool pdl);
// out's n planes = the values of in's packed spectrum of nin <= n planes,
// taken as zero past them (out may be in).
cudaError_t z_inverse(const ZBatch& b, int nin, int n, int plane_size, const double* twiddle, cudaStream_t st,
                      bool pdl);
// The same, and dz's n planes = the values of the z-derivative (planes 0
// and 1 of the spectrum have none).
cudaError_t z_inverse_dz(const ZBatch& b, int nin, int n, int plane_size, const double* twiddle, double beta,
                         cudaStream_t st, bool pdl);
// out's n planes = the z-derivative of in x mul, modes from `keep` on dropped.
cudaError_t z_product_dz(const ZBatch& b, int n, int keep, int plane_size, const double* twiddle, double beta,
                         cudaStream_t st, bool pdl);

}  // namespace stx
