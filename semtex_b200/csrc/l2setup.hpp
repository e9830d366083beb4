// Device setup of the two-level skeleton matrices (see l2setup.cu).
#pragma once

#include <cuda_runtime.h>

#include <memory>
#include <vector>

#include "host/mesh.hpp"
#include "host/patch.hpp"
#include "host/session.hpp"

namespace stx {

// Form, on the device, every mode's packed S_II^-1 (per patch family, at
// fam_off[m * nfamily + f]), G (at g_off[...]) and interface inverse (at
// if_off[m]) into d_pack (FP64, zeroed by the caller), from the element Schur
// complements hbb [nmodes][mesh families][next][next] and the pinned
// interface id of each mode (-1: none).  Synchronises `st`; throws when a
// system is not positive definite.  Temporaries stay within budget_bytes
// (modes are processed in chunks).
void l2_device_setup_guarded(const Mesh& M, const Numbering& N, const Patching& P, const std::vector<double>& hbb,
                             int nmodes, const std::vector<int>& pin, const std::vector<long long>& fam_off,
                             const std::vector<long long>& g_off, const std::vector<long long>& if_off,
                             double* d_pack, cudaStream_t st, size_t budget_bytes = size_t(2) << 30);

// The patching of a numbering for the two-level direct solve, or null when
// the single banded factor is used: token STX_TWOLEVEL = 0, element boundaries
// of more than 64 nodes, or an interface too large for a dense inverse at
// every patch size.  The patch size is the one of {8, 16, 36, 64, all}
// elements with the least estimated time: the matrix bytes of every mode (the
// interface inverse and, per patch family, S_II^-1 and G = S_II^-1 S_IB once
// each) at the products' rate, and the interface's three launches where there
// is an interface.  One patch has none unless its system can be singular, so
// a small problem's solve is four launches instead of seven.
std::unique_ptr<Patching> choose_patching(const Session& S, const Mesh& M, const Numbering& N);

}  // namespace stx
