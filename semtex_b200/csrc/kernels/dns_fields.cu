// Field passes of a DNS step (Cartesian), every velocity component in one
// kernel: nonlinear terms, waveProp + setPForce, project.
//
// A block holds one element on up to PP planes in shared memory.  Global
// memory is read and written in storage order (coalesced); between, thread
// (plane, line) forms the s derivatives of one element column, then the r
// derivatives of one element row, its values in registers and the entries of
// D as constant operands (D is a kernel parameter and the loops are unrolled
// for the compile-time N_P), so an element plane's derivative costs 2 N_P^3
// multiply-adds and four shared-memory accesses a node.  The tensor-core form
// (m8n8k4 tiles, elemderiv.cuh) pads N_P = 9 to 16 x 16 x 12: 4.2 times the
// multiply-adds at the same FP64 rate.
//
// Bound: HBM.  Fields of F bytes: nonlinear terms 12 F in the skew form
// (velocities and both z terms in, N out), 9 F in the others, waveProp and
// setPForce 22 F (N_TIME = 3), project 7 F.  us, 24 x 24 x 96, N_P = 9 (F = 36
// MB; B200): 95 (skew), 156 and 64 against 340, 258 and 130 for a launch per
// component; with the loads of a pass not batched (the compiler keeps them
// behind the stores before them) 227, 179 and 81.  At larger N_P a block has
// more registers (192 to 240 for N_P 12 to 16) and shared memory, and the step
// is still the faster: us a step, a launch per component on the tensor cores
// and an unfused z direction / so, 32 planes: 10 x 10 elements, N_P = 12 406 /
// 260, N_P = 14 575 / 327; 8 x 8, N_P = 15 558 / 269, N_P = 16 460 / 340; one
// plane of 16 x 16, N_P = 16 171 / 124.
#include "dns_fields.cuh"

#include <algorithm>
#include <type_traits>
#include <utility>

#include "launch.hpp"
#include "ptx.cuh"

namespace stx {

namespace {

template <int NP>
struct DMat {
  double d[NP * NP];
};

// Planes per block and threads: one thread per (plane, line), an even number
// of planes (the Re and Im planes of a mode stay together), planes spread
// evenly over the blocks.
constexpr int kLineThreads = 128;
struct FieldPlan {
  int pp, threads;
  dim3 grid;
};
FieldPlan field_plan(const DevGeom& g) {
  FieldPlan P;
  const int most = std::max(2, kLineThreads / g.np / 2 * 2);
  const int nb = (g.nz + most - 1) / most;
  P.pp = g.nz == 1 ? 1 : ((g.nz + nb - 1) / nb + 1) / 2 * 2;
  P.threads = (P.pp * g.np + 31) / 32 * 32;  // at least pp np: BlockPoints
  P.grid = dim3(g.nel, (g.nz + P.pp - 1) / P.pp);
  return P;
}

// out[a] = sum_b D[a][b] f[b]
template <int NP>
__device__ __forceinline__ double d_row(const DMat<NP>& D, int a, const double (&f)[NP]) {
  double v = D.d[a * NP] * f[0];
#pragma unroll
  for (int b = 1; b < NP; ++b) v = fma(D.d[a * NP + b], f[b], v);
  return v;
}

// The geometric factors of element e: [drdx | drdy | dsdx | dsdy].
template <int NP>
__device__ __forceinline__ void load_geom(const DevGeom& g, int e, double* geo) {
  constexpr int NN = NP * NP;
  for (int t = threadIdx.x; t < NN; t += blockDim.x) {
    geo[t] = __ldg(g.drdx + e * NN + t);
    geo[NN + t] = __ldg(g.drdy + e * NN + t);
    geo[2 * NN + t] = __ldg(g.dsdx + e * NN + t);
    geo[3 * NN + t] = __ldg(g.dsdy + e * NN + t);
  }
}

// The points of a block's planes in storage order, NP or fewer a thread (the
// block has at least pn NP threads): point it of this thread is entry
// threadIdx.x + it blockDim.x, in batches whose loads are all in flight
// before the first is used (the fields of a pass may alias, so the compiler
// cannot move loads over stores by itself).
struct BlockPoints {
  int total, plane_size;
  __device__ __forceinline__ int index(int it) const { return threadIdx.x + it * blockDim.x; }
  // offset of entry i from the block's first point
  template <int NN>
  __device__ __forceinline__ size_t offset(int i) const {
    const int p = i / NN;
    return static_cast<size_t>(p) * plane_size + (i - p * NN);
  }
};

// A pass over the lines of one direction: element offset of point b of this
// thread's line.
template <int NP, bool kRow>
__device__ __forceinline__ int at(int line, int b) {
  return kRow ? line * NP + b : b * NP + line;
}

template <int NP, bool W, bool kRow>
__device__ __forceinline__ void nonlinear_lines(const DMat<NP>& D, const double* geo, const double* U, double* O,
                                                int pn, int p, int line, int form) {
  constexpr int NN = NP * NP, NC = W ? 3 : 2;
  const double* gx = geo + (kRow ? 0 : 2 * NN);
  const double* gy = gx + NN;
  double f[NC][NP];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int b = 0; b < NP; ++b) f[c][b] = U[(c * pn + p) * NN + at<NP, kRow>(line, b)];
  auto put = [&](int c, int t, double v) {
    double* o = O + (c * pn + p) * NN + t;
    *o = kRow ? *o + v : v;
  };
  const double w = form == 0 ? 0.5 : 1.0;
  if (form != 2) {  // (u dr/dx + v dr/dy) dU_c/dr and the same in s
#pragma unroll
    for (int a = 0; a < NP; ++a) {
      const int t = at<NP, kRow>(line, a);
      const double adv = w * (f[0][a] * gx[t] + f[1][a] * gy[t]);
#pragma unroll
      for (int c = 0; c < NC; ++c) put(c, t, adv * d_row<NP>(D, a, f[c]));
    }
  }
  if (form != 1) {  // d(U_c u)/dr dr/dx + d(U_c v)/dr dr/dy and the same in s
    double q[2 * NC - 1][NP];  // uu, uv, vv, (uw, vw)
#pragma unroll
    for (int b = 0; b < NP; ++b) {
      q[0][b] = f[0][b] * f[0][b];
      q[1][b] = f[0][b] * f[1][b];
      q[2][b] = f[1][b] * f[1][b];
      if constexpr (W) {
        q[3][b] = f[0][b] * f[2][b];
        q[4][b] = f[1][b] * f[2][b];
      }
    }
#pragma unroll
    for (int a = 0; a < NP; ++a) {
      const int t = at<NP, kRow>(line, a);
      const double x = w * gx[t], y = w * gy[t];
      double d[2 * NC - 1];
#pragma unroll
      for (int k = 0; k < 2 * NC - 1; ++k) d[k] = d_row<NP>(D, a, q[k]);
      double v[3] = {d[0] * x + d[1] * y, d[1] * x + d[2] * y, 0.0};
      if constexpr (W) v[2] = d[3] * x + d[4] * y;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        double* o = O + (c * pn + p) * NN + t;
        *o = (kRow || form == 0) ? *o + v[c] : v[c];
      }
    }
  }
}

template <int NP, bool W>
__global__ void __launch_bounds__(kLineThreads) k_nonlinear_fields(DevGeom g, DMat<NP> D, NonlinearFields a, int pp) {
  pdl_trigger();
  pdl_wait();
  constexpr int NN = NP * NP, NC = W ? 3 : 2;
  extern __shared__ __align__(16) double sm[];
  const int e = blockIdx.x, k0 = blockIdx.y * pp, pn = min(pp, g.nz - k0);
  double* geo = sm;
  double* U = geo + 4 * NN;       // [NC][pn][NN]
  double* O = U + NC * pp * NN;   // [NC][pn][NN]
  const size_t base = static_cast<size_t>(k0) * g.plane_size + static_cast<size_t>(e) * NN;
  load_geom<NP>(g, e, geo);
  const BlockPoints B{pn * NN, g.plane_size};
  {
    double v[NP][NC];
#pragma unroll
    for (int it = 0; it < NP; ++it) {
      const int i = B.index(it);
      const size_t x = base + B.offset<NN>(i);
#pragma unroll
      for (int c = 0; c < NC; ++c) v[it][c] = i < B.total ? a.U[c][x] : 0.0;
    }
#pragma unroll
    for (int it = 0; it < NP; ++it) {
      const int i = B.index(it);
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (i < B.total) U[c * pn * NN + i] = v[it][c];
    }
  }
  __syncthreads();
  const int p = threadIdx.x / NP, line = threadIdx.x - p * NP;
  if (p < pn) nonlinear_lines<NP, W, false>(D, geo, U, O, pn, p, line, a.form);
  __syncthreads();
  if (p < pn) nonlinear_lines<NP, W, true>(D, geo, U, O, pn, p, line, a.form);
  __syncthreads();
  const double w = a.form == 0 ? 0.5 : 1.0;
  constexpr int kB = (NP + 2) / 3;  // a third of the points together
#pragma unroll
  for (int it0 = 0; it0 < NP; it0 += kB) {
    double tc[kB][NC], tk[kB][NC];
#pragma unroll
    for (int j = 0; j < kB; ++j) {
      const int i = B.index(it0 + j);
      const size_t x = base + B.offset<NN>(i);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        tc[j][c] = (W && a.Tc[c] && i < B.total) ? a.Tc[c][x] : 0.0;
        tk[j][c] = (W && a.Tk[c] && i < B.total) ? a.Tk[c][x] : 0.0;
      }
    }
#pragma unroll
    for (int j = 0; j < kB; ++j) {
      const int i = B.index(it0 + j);
      if (i >= B.total) break;
      const size_t x = base + B.offset<NN>(i);
      const double uw = W ? w * U[2 * pn * NN + i] : 0.0;
#pragma unroll
      for (int c = 0; c < NC; ++c) a.N[c][x] = -(O[c * pn * NN + i] + uw * tc[j][c] + w * tk[j][c]);
    }
  }
}

template <int NP>
__global__ void __launch_bounds__(kLineThreads) k_wave_fields(DevGeom g, DMat<NP> D, WaveFields a, int pp) {
  pdl_trigger();
  pdl_wait();
  constexpr int NN = NP * NP;
  extern __shared__ __align__(16) double sm[];
  const int e = blockIdx.x, k0 = blockIdx.y * pp, pn = min(pp, g.nz - k0);
  double* geo = sm;
  double* V = geo + 4 * NN;      // [3][pn][NN]
  double* O = V + 3 * pp * NN;   // [pn][NN]
  const size_t base = static_cast<size_t>(k0) * g.plane_size + static_cast<size_t>(e) * NN;
  load_geom<NP>(g, e, geo);
  const BlockPoints B{pn * NN, g.plane_size};
  constexpr int kB = (NP + 2) / 3;
  for (int c = 0; c < a.ncom; ++c) {
#pragma unroll
    for (int it0 = 0; it0 < NP; it0 += kB) {
      double v[kB][6];
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        const int i = B.index(it0 + j);
        const size_t x = base + B.offset<NN>(i);
#pragma unroll
        for (int q = 0; q < 6; ++q) v[j][q] = (q < a.n && i < B.total) ? a.p[c][q][x] : 0.0;
      }
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        const int i = B.index(it0 + j);
        if (i >= B.total) break;
        double r = 0.0;
#pragma unroll
        for (int q = 0; q < 6; ++q) r += a.c[q] * v[j][q];  // c is zero past n
        a.out[c][base + B.offset<NN>(i)] = r;
        V[c * pn * NN + i] = r;
      }
    }
  }
  __syncthreads();
  const int p = threadIdx.x / NP, line = threadIdx.x - p * NP;
  if (p < pn) {
    double f[2][NP];
#pragma unroll
    for (int b = 0; b < NP; ++b)
#pragma unroll
      for (int c = 0; c < 2; ++c) f[c][b] = V[(c * pn + p) * NN + at<NP, false>(line, b)];
#pragma unroll
    for (int r = 0; r < NP; ++r) {
      const int t = at<NP, false>(line, r);
      O[p * NN + t] = d_row<NP>(D, r, f[0]) * geo[2 * NN + t] + d_row<NP>(D, r, f[1]) * geo[3 * NN + t];
    }
  }
  __syncthreads();
  if (p < pn) {
    double f[2][NP];
#pragma unroll
    for (int b = 0; b < NP; ++b)
#pragma unroll
      for (int c = 0; c < 2; ++c) f[c][b] = V[(c * pn + p) * NN + at<NP, true>(line, b)];
#pragma unroll
    for (int r = 0; r < NP; ++r) {
      const int t = at<NP, true>(line, r);
      O[p * NN + t] += d_row<NP>(D, r, f[0]) * geo[t] + d_row<NP>(D, r, f[1]) * geo[NN + t];
    }
  }
  __syncthreads();
  const double* Wv = V + 2 * pn * NN;
  for (int i = threadIdx.x; i < pn * NN; i += blockDim.x) {
    const int q = i / NN, t = i - q * NN, k = k0 + q;
    double v = O[i];
    if (a.z3 && k >= 2) v += a.beta * (k >> 1) * ((k & 1) ? Wv[i - NN] : -Wv[i + NN]);
    a.div[base + static_cast<size_t>(q) * g.plane_size + t] = v * a.inv_dt;
  }
}

template <int NP>
__global__ void __launch_bounds__(kLineThreads) k_project_fields(DevGeom g, DMat<NP> D, ProjectFields a, int pp) {
  pdl_trigger();
  pdl_wait();
  constexpr int NN = NP * NP;
  extern __shared__ __align__(16) double sm[];
  const int e = blockIdx.x, k0 = blockIdx.y * pp, pn = min(pp, g.nz - k0);
  double* geo = sm;
  double* P = geo + 4 * NN;   // [pn][NN] each
  double* X = P + pp * NN;
  double* Y = X + pp * NN;
  const size_t base = static_cast<size_t>(k0) * g.plane_size + static_cast<size_t>(e) * NN;
  load_geom<NP>(g, e, geo);
  const BlockPoints B{pn * NN, g.plane_size};
  {
    double v[NP];
#pragma unroll
    for (int it = 0; it < NP; ++it) {
      const int i = B.index(it);
      v[it] = i < B.total ? a.p[base + B.offset<NN>(i)] : 0.0;
    }
#pragma unroll
    for (int it = 0; it < NP; ++it) {
      const int i = B.index(it);
      if (i < B.total) P[i] = v[it];
    }
  }
  __syncthreads();
  const int p = threadIdx.x / NP, line = threadIdx.x - p * NP;
  if (p < pn) {
    double f[NP];
#pragma unroll
    for (int b = 0; b < NP; ++b) f[b] = P[p * NN + at<NP, false>(line, b)];
#pragma unroll
    for (int r = 0; r < NP; ++r) X[p * NN + at<NP, false>(line, r)] = d_row<NP>(D, r, f);
  }
  __syncthreads();
  if (p < pn) {
    double f[NP];
#pragma unroll
    for (int b = 0; b < NP; ++b) f[b] = P[p * NN + at<NP, true>(line, b)];
#pragma unroll
    for (int r = 0; r < NP; ++r) {
      const int t = at<NP, true>(line, r);
      const double dr = d_row<NP>(D, r, f), ds = X[p * NN + t];
      X[p * NN + t] = dr * geo[t] + ds * geo[2 * NN + t];
      Y[p * NN + t] = dr * geo[NN + t] + ds * geo[3 * NN + t];
    }
  }
  __syncthreads();
  constexpr int kB = (NP + 2) / 3;
#pragma unroll
  for (int it0 = 0; it0 < NP; it0 += kB) {
    double v[kB][3];
#pragma unroll
    for (int j = 0; j < kB; ++j) {
      const int i = B.index(it0 + j);
      const size_t x = base + B.offset<NN>(i);
#pragma unroll
      for (int c = 0; c < 3; ++c) v[j][c] = (c < a.ncom && i < B.total) ? a.io[c][x] : 0.0;
    }
#pragma unroll
    for (int j = 0; j < kB; ++j) {
      const int i = B.index(it0 + j);
      if (i >= B.total) break;
      const size_t x = base + B.offset<NN>(i);
      const int k = k0 + i / NN;
      double z = 0.0;
      if (a.z3 && k >= 2) z = a.beta * (k >> 1) * ((k & 1) ? P[i - NN] : -P[i + NN]);
      const double d[3] = {X[i], Y[i], z};
#pragma unroll
      for (int c = 0; c < 3; ++c)
        if (c < a.ncom) {
          a.io[c][x] = a.alpha * v[j][c] + a.b * d[c];
          if (k == 1) a.clear[c][x] = 0.0;
        }
    }
  }
}

// Call f(NP) with the compile-time number of points (2..16).
template <int NP, class F>
cudaError_t np_dispatch_from(int np, F&& f) {
  if constexpr (NP > 16) {
    return cudaErrorInvalidValue;
  } else {
    if (np == NP) return f(std::integral_constant<int, NP>{});
    return np_dispatch_from<NP + 1>(np, std::forward<F>(f));
  }
}

template <int NP, class Args>
cudaError_t field_launch(void (*kernel)(DevGeom, DMat<NP>, Args, int), const DevGeom& g, const double* D,
                         const Args& a, int fields, cudaStream_t st) {
  DMat<NP> M;
  std::copy(D, D + NP * NP, M.d);
  const FieldPlan P = field_plan(g);
  const size_t smem = sizeof(double) * NP * NP * (4 + static_cast<size_t>(fields) * P.pp);
  raise_smem_limit(reinterpret_cast<const void*>(kernel), smem);
  const cudaError_t err = launch_ex(g.pdl != 0, kernel, P.grid, dim3(P.threads), smem, st, g, M, a, P.pp);
  return err != cudaSuccess ? err : cudaGetLastError();
}

}  // namespace

cudaError_t dns_nonlinear_fields(const DevGeom& g, const double* D, const NonlinearFields& a, cudaStream_t st) {
  return np_dispatch_from<2>(g.np, [&](auto np_) {
    constexpr int NP = decltype(np_)::value;
    return a.ncom == 3 ? field_launch<NP>(k_nonlinear_fields<NP, true>, g, D, a, 6, st)
                       : field_launch<NP>(k_nonlinear_fields<NP, false>, g, D, a, 4, st);
  });
}

cudaError_t dns_wave_fields(const DevGeom& g, const double* D, const WaveFields& a, cudaStream_t st) {
  return np_dispatch_from<2>(g.np, [&](auto np_) {
    constexpr int NP = decltype(np_)::value;
    return field_launch<NP>(k_wave_fields<NP>, g, D, a, 4, st);
  });
}

cudaError_t dns_project_fields(const DevGeom& g, const double* D, const ProjectFields& a, cudaStream_t st) {
  return np_dispatch_from<2>(g.np, [&](auto np_) {
    constexpr int NP = decltype(np_)::value;
    return field_launch<NP>(k_project_fields<NP>, g, D, a, 3, st);
  });
}

}  // namespace stx
