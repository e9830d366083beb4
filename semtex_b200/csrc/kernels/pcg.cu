// The iteration of Field::solve JACPCG (src/field.cpp:711-805).
//
// One cluster of thread blocks per plane runs that plane's whole iteration:
// the planes share nothing, so a plane stops when its own test says so, and
// nothing returns to the host between iterations.  Two cluster barriers an
// iteration separate
//   (1) per element (one warp each): p = z + beta p at its nodes, q = H p
//       scattered to the global vector, and the element's part of p . H p;
//   (2) per vector entry: x += alpha p, r -= alpha q, and the sums r . z and
//       r . r, z = PC r formed on the fly.
// The sums travel as one partial per warp, written into every block's shared
// memory (distributed shared memory) before the barrier; every warp then adds
// the same numbers in the same order, so all threads of a cluster take the
// same branches.  Vectors other blocks wrote are read past the L1.
//
// Bound: latency.  An iteration moves a few hundred KB a plane, all of it in
// the L2, and is two barriers and three dependent rounds of loads.  As
// launches (a dozen kernels and memsets an iteration, a host read-back every
// eight) the 8 x 8, N_P = 9, N_Z = 16 problem took 53 us an iteration
// (15.5 ms for 288), now 7.4 (2.1 ms for 282); see pcg_cluster.
#include "pcg.cuh"

#include <algorithm>

#include "elemderiv.cuh"
#include "launch.hpp"

namespace stx {

namespace {

constexpr int kPcgWarps = 8;
constexpr int kPcgThreads = 32 * kPcgWarps;
constexpr int kPcgMaxCluster = 16;
constexpr int kPcgPortable = 8;  // blocks of a cluster that every device places
constexpr int kPcgBatch = 4;  // entries a thread loads together

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Store v at the same shared-memory offset as `p` in block `rank` of the cluster.
__device__ __forceinline__ void st_cluster(const double* p, unsigned rank, double v) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// Partial sums of a cluster: [parity][value][block of the cluster][warp].  The parity
// alternates, so that a block still reading one sum's partials is not
// overtaken by the next sum's.
struct PcgShared {
  double part[2][2][kPcgMaxCluster][kPcgWarps];
};

// Cluster-wide sums of two values; every thread gets both.  Includes the
// cluster barrier (and so orders the global writes before it).
__device__ __forceinline__ void cluster_sum2(PcgShared& sh, int& parity, unsigned rank, unsigned nrank, double& a,
                                             double& b) {
  const int ln = threadIdx.x & 31, wp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if (ln < static_cast<int>(nrank)) {
    st_cluster(&sh.part[parity][0][rank][wp], ln, a);
    st_cluster(&sh.part[parity][1][rank][wp], ln, b);
  }
  __syncwarp();
  cluster_barrier();
  double va = 0.0, vb = 0.0;
  for (int i = ln; i < static_cast<int>(nrank) * kPcgWarps; i += 32) {
    va += sh.part[parity][0][i / kPcgWarps][i % kPcgWarps];
    vb += sh.part[parity][1][i / kPcgWarps][i % kPcgWarps];
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    va += __shfl_xor_sync(0xffffffffu, va, o);
    vb += __shfl_xor_sync(0xffffffffu, vb, o);
  }
  a = va;
  b = vb;
  parity ^= 1;
}

// out(t, (H u)[t]) for the nodes of element e this lane holds, u in su
// (Element::HelmholtzOp, src/element.cpp:1484-1529); su, sR, sS are the warp's.
// MT > 0: on the FP64 tensor cores (np <= 8 MT); MT = 0: any np.
template <int MT, int KS>
struct HelmholtzOp {
  ElemMma<MT, KS> M;
  double dt[MT][KS];  // D[4 s + t][8 x + g]: D^T as A operand, D as B operand
  __device__ __forceinline__ void load(const double* sD, int np) {
    M.load_d(sD, np);
    const int ln = threadIdx.x & 31, g8 = ln >> 2, t4 = ln & 3;
#pragma unroll
    for (int x = 0; x < MT; ++x)
#pragma unroll
      for (int s = 0; s < KS; ++s) {
        const int r = 4 * s + t4, c = 8 * x + g8;
        dt[x][s] = (r < np && c < np) ? sD[r * np + c] : 0.0;
      }
  }
  template <class F>
  __device__ __forceinline__ void apply(const DevGeom& g, int e, double hcon, const double* su, double* sR,
                                        double* sS, const double* /*sD*/, F&& out) const {
    const int np = g.np, ln = threadIdx.x & 31, g8 = ln >> 2, t4 = ln & 3;
    const size_t o = static_cast<size_t>(e) * g.npnp;
    double ur[MT][MT][2], us[MT][MT][2];
    M.grad(su, np, ur, us);
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < MT; ++n)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int i = 8 * m + g8, j = 8 * n + 2 * t4 + c;
          if (i < np && j < np) {
            const int t = i * np + j;
            const double q1 = __ldg(g.Q1 + o + t), q2 = __ldg(g.Q2 + o + t), q3 = __ldg(g.Q3 + o + t);
            sR[t] = q1 * ur[m][n][c] + q3 * us[m][n][c];
            sS[t] = q2 * us[m][n][c] + q3 * ur[m][n][c];
          }
        }
    __syncwarp();
    double ra[MT][KS], sb[KS][MT];
#pragma unroll
    for (int x = 0; x < MT; ++x)
#pragma unroll
      for (int s = 0; s < KS; ++s) {
        const int k = 4 * s + t4, i = 8 * x + g8;
        ra[x][s] = (i < np && k < np) ? sR[i * np + k] : 0.0;
        sb[s][x] = (i < np && k < np) ? sS[k * np + i] : 0.0;
      }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < MT; ++n) {
        double h[2] = {0.0, 0.0};
#pragma unroll
        for (int s = 0; s < KS; ++s) {
          dmma_8x8x4(h[0], h[1], dt[m][s], sb[s][n]);  // D^T S
          dmma_8x8x4(h[0], h[1], ra[m][s], dt[n][s]);  // R D
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int i = 8 * m + g8, j = 8 * n + 2 * t4 + c;
          if (i < np && j < np) {
            const int t = i * np + j;
            out(t, h[c] + __ldg(g.Q4 + o + t) * su[t] * hcon);
          }
        }
      }
  }
};

template <>
struct HelmholtzOp<0, 0> {
  __device__ __forceinline__ void load(const double*, int) {}
  template <class F>
  __device__ __forceinline__ void apply(const DevGeom& g, int e, double hcon, const double* su, double* sR,
                                        double* sS, const double* sD, F&& out) const {
    const int np = g.np;
    const size_t o = static_cast<size_t>(e) * g.npnp;
    for (int t = threadIdx.x & 31; t < g.npnp; t += 32) {
      const int i = t / np, j = t - i * np;
      double r = 0.0, s = 0.0;
      for (int k = 0; k < np; ++k) {
        r += su[i * np + k] * sD[j * np + k];
        s += sD[i * np + k] * su[k * np + j];
      }
      const double q1 = g.Q1[o + t], q2 = g.Q2[o + t], q3 = g.Q3[o + t];
      sR[t] = q1 * r + q3 * s;
      sS[t] = q2 * s + q3 * r;
    }
    __syncwarp();
    for (int t = threadIdx.x & 31; t < g.npnp; t += 32) {
      const int i = t / np, j = t - i * np;
      double h = g.Q4[o + t] * su[t] * hcon;
      for (int k = 0; k < np; ++k) {
        h += sD[k * np + i] * sS[k * np + j];
        h += sR[i * np + k] * sD[k * np + j];
      }
      out(t, h);
    }
  }
};

template <int MT, int KS>
__global__ void __launch_bounds__(kPcgThreads, 2)
    k_pcg(DevGeom g, DevNumbering N, DevModal S, PcgVectors v, double tol_rel, int step_max) {
  extern __shared__ __align__(16) double sm[];
  __shared__ PcgShared sh;
  unsigned rank, nrank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(nrank));
  const int j = blockIdx.x / nrank;
  const int k = (g.nz > 1 && j > 0) ? j + 1 : j;  // the Nyquist plane (1) is never solved
  const int m = k >> 1, np = g.np, nn = g.npnp, next = g.next, nint = g.nint;
  const int ng = N.nglobal, ns = S.nsolve[m];
  const double hcon = S.lambda2[m] + S.betak2[m];
  const int wp = threadIdx.x >> 5, ln = threadIdx.x & 31;
  const size_t off = static_cast<size_t>(k) * v.vstride;
  double *r = v.r + off, *x = v.x + off, *q = v.q + off, *pn = v.p0 + off, *po = v.p1 + off;
  const double* pc = S.pc + static_cast<size_t>(m) * S.npts;
  double* sD = sm;
  double* su = sD + np * np + static_cast<size_t>(wp) * 3 * nn;
  double* sR = su + nn;
  double* sS = sR + nn;
  for (int t = threadIdx.x; t < np * np; t += kPcgThreads) sD[t] = S.D[t];
  __syncthreads();
  // every block of the cluster has started before any writes into another's
  // shared memory
  cluster_barrier();
  HelmholtzOp<MT, KS> op;
  op.load(sD, np);
  int parity = 0;
  const int i0 = rank * kPcgThreads + threadIdx.x, istep = nrank * kPcgThreads;
  const int e0 = rank * kPcgWarps + wp, estep = nrank * kPcgWarps;

  // q += H u per element, node(i, u) giving u at global positions i; the
  // element's u . H u summed into dot.  `keep` (may be null) receives u.
  auto apply = [&](auto&& node, double* keep, double& dot) {
    for (int e = e0; e < g.nel; e += estep) {
      const int* bt = N.btog + static_cast<size_t>(e) * next;
      const int ibase = ng + e * nint - next;  // + boundary-major position
      // a few nodes a lane at a time, their loads in flight together
      for (int a0 = ln; a0 < nn; a0 += 32 * kPcgBatch) {
        int i[kPcgBatch];
        double u[kPcgBatch];
#pragma unroll
        for (int b = 0; b < kPcgBatch; ++b) {
          const int a = min(a0 + 32 * b, nn - 1);
          i[b] = a < next ? __ldg(bt + a) : ibase + a;
        }
        node(i, u);
#pragma unroll
        for (int b = 0; b < kPcgBatch; ++b) {
          const int a = a0 + 32 * b;
          if (a >= nn) break;
          if (keep) __stcg(keep + i[b], u[b]);
          su[__ldg(g.emap + a)] = u[b];
        }
      }
      __syncwarp();
      op.apply(g, e, hcon, su, sR, sS, sD, [&](int t, double h) {
        dot += su[t] * h;
        const int a = __ldg(g.pmap + t);
        if (a < next) atomicAdd(q + __ldg(bt + a), h);
        else __stcg(q + ibase + a, h);
      });
      __syncwarp();
    }
  };
  // <K u, w> on mixed-BC edges (Mixed::augmentOp, src/condition.cpp:379-407)
  auto mixed = [&](int i, double u) { return (N.mixdiag && i < ng) ? N.mixdiag[i] * u : 0.0; };

  // the essential (and pinned) entries of the right-hand side and the guess
  // are zero; q's boundary part is zero before every operator apply
  double bb = 0.0, none = 0.0;
  for (int i = i0; i < v.npts; i += istep) {
    const bool fixed = i >= ns && i < ng;
    const double rv = fixed ? 0.0 : r[i];
    if (fixed) {
      r[i] = 0.0;
      x[i] = 0.0;
    }
    if (i < ng) __stcg(q + i, 0.0);
    bb += rv * rv;
  }
  cluster_sum2(sh, parity, rank, nrank, bb, none);
  double dot = 0.0;
  apply(
      [&](const int(&i)[kPcgBatch], double(&u)[kPcgBatch]) {
#pragma unroll
        for (int b = 0; b < kPcgBatch; ++b) u[b] = __ldcg(x + i[b]);
      },
      nullptr, dot);
  cluster_barrier();
  double rho = 0.0, r2 = 0.0, rho_old = 0.0;
  for (int i = i0; i < v.npts; i += istep) {
    const bool fixed = i >= ns && i < ng;
    const double qv = __ldcg(q + i) + mixed(i, x[i]);
    if (i < ng) __stcg(q + i, 0.0);
    const double rv = fixed ? 0.0 : r[i] - qv;
    __stcg(r + i, rv);
    rho += pc[i] * rv * rv;
    r2 += rv * rv;
  }
  cluster_sum2(sh, parity, rank, nrank, rho, r2);

  const double eps = tol_rel * sqrt(bb), eps2 = eps * eps;
  int iter = 0, hit = 0;
  while (r2 > eps2) {
    if (++iter >= step_max) {
      hit = 1;
      break;
    }
    const bool first = iter == 1;
    const double beta = first ? 0.0 : rho / rho_old;
    auto direction = [&](const int(&i)[kPcgBatch], double(&u)[kPcgBatch]) {
      double z[kPcgBatch], c[kPcgBatch];
#pragma unroll
      for (int b = 0; b < kPcgBatch; ++b) {
        c[b] = __ldg(pc + i[b]);
        z[b] = __ldcg(r + i[b]);
        u[b] = first ? 0.0 : __ldcg(po + i[b]);
      }
#pragma unroll
      for (int b = 0; b < kPcgBatch; ++b) u[b] = first ? c[b] * z[b] : c[b] * z[b] + beta * u[b];
    };
    double pq = 0.0;
    apply(direction, pn, pq);
    if (N.mixdiag)
      for (int i = i0; i < ng; i += istep) {
        const double z = __ldg(pc + i) * __ldcg(r + i), p = first ? z : z + beta * __ldcg(po + i);
        pq += N.mixdiag[i] * p * p;
      }
    cluster_sum2(sh, parity, rank, nrank, pq, none);
    const double alpha = rho / pq;
    rho_old = rho;
    rho = r2 = 0.0;
    for (int ib = i0; ib < v.npts; ib += istep * kPcgBatch) {
      double p[kPcgBatch], qv[kPcgBatch], rv[kPcgBatch], xv[kPcgBatch], cv[kPcgBatch];
#pragma unroll
      for (int b = 0; b < kPcgBatch; ++b) {
        const int i = min(ib + b * istep, v.npts - 1);
        p[b] = __ldcg(pn + i);
        qv[b] = __ldcg(q + i);
        rv[b] = __ldcg(r + i);
        xv[b] = x[i];
        cv[b] = __ldg(pc + i);
      }
#pragma unroll
      for (int b = 0; b < kPcgBatch; ++b) {
        const int i = ib + b * istep;
        if (i >= v.npts) break;
        const bool fixed = i >= ns && i < ng;
        const double rn = fixed ? 0.0 : rv[b] - alpha * (qv[b] + mixed(i, p[b]));
        if (i < ng) __stcg(q + i, 0.0);
        x[i] = xv[b] + alpha * p[b];
        __stcg(r + i, rn);
        rho += cv[b] * rn * rn;
        r2 += rn * rn;
      }
    }
    cluster_sum2(sh, parity, rank, nrank, rho, r2);
    double* t = pn;
    pn = po;
    po = t;
  }
  if (rank == 0 && threadIdx.x == 0) v.out[k] = make_int2(iter, hit);
}

// ---------------------------------------------------------------------------
// The same iteration as a chain of launches over all planes, for few planes
// of many elements: a cluster is at most 16 blocks, so a plane's warps then
// have dozens of elements each while most SMs are idle.  Every plane has its
// own scalars and stopping test; every eighth iteration the host reads back
// whether any plane is still at work.
// ---------------------------------------------------------------------------

struct PcgScalars {
  double rho2, r2, eps;
  int iter, active, hit_max, solved;
};

// y = H x (Field::HelmholtzOperator, src/field.cpp:855-940) per (element,
// plane); y's boundary part must be zero on entry.
__global__ void k_global_op(DevGeom g, DevNumbering N, DevModal S, const double* __restrict__ X,
                            double* __restrict__ Y, int vstride, const PcgScalars* sc) {
  extern __shared__ double smem[];
  const int nn = g.npnp, np = g.np;
  double* sD = smem;
  double* su = sD + np * np;
  double* sR = su + nn;
  double* sS = sR + nn;
  const int e = blockIdx.x, k = blockIdx.y, t = threadIdx.x;
  if (!sc[k].active) return;
  const int m = k >> 1;
  const double hcon = S.lambda2[m] + S.betak2[m];
  const double* x = X + static_cast<size_t>(k) * vstride;
  double* y = Y + static_cast<size_t>(k) * vstride;
  if (N.mixdiag && e == 0)  // <K x, w> on mixed-BC edges (Mixed::augmentOp, src/condition.cpp:379-407)
    for (int q = t; q < N.nglobal; q += blockDim.x) atomicAdd(&y[q], N.mixdiag[q] * x[q]);
  for (int q = t; q < np * np; q += blockDim.x) sD[q] = S.D[q];
  if (t < g.next) su[g.emap[t]] = x[N.btog[e * g.next + t]];
  if (t < g.nint) su[g.emap[g.next + t]] = x[N.nglobal + static_cast<size_t>(e) * g.nint + t];
  __syncthreads();
  const int i = t / np, j = t - (t / np) * np;
  if (t < nn) {
    double r = 0.0, s = 0.0;
    for (int q = 0; q < np; ++q) {
      r += su[i * np + q] * sD[j * np + q];
      s += sD[i * np + q] * su[q * np + j];
    }
    const double q1 = g.Q1[e * nn + t], q2 = g.Q2[e * nn + t], q3 = g.Q3[e * nn + t];
    sR[t] = q1 * r + q3 * s;
    sS[t] = q2 * s + q3 * r;
  }
  __syncthreads();
  if (t < nn) {
    double h = g.Q4[e * nn + t] * su[t] * hcon;
    for (int q = 0; q < np; ++q) {
      h += sD[q * np + i] * sS[q * np + j];
      h += sR[i * np + q] * sD[q * np + j];
    }
    const int b = g.pmap[t];
    if (b < g.next)
      atomicAdd(&y[N.btog[e * g.next + b]], h);
    else
      y[N.nglobal + static_cast<size_t>(e) * g.nint + (b - g.next)] = h;
  }
}

// Zero entries [nsolve, hi) of each plane's vector (essential and pinned ones).
__global__ void k_zero_fixed(double* V, int vstride, const int* nsolve, int hi) {
  const int k = blockIdx.y;
  for (int i = nsolve[k >> 1] + blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += gridDim.x * blockDim.x)
    V[static_cast<size_t>(k) * vstride + i] = 0.0;
}

// out[k] += sum_i a[k][i] * b[k][i] over active (or all, if force) planes.
__global__ void k_dot(const double* __restrict__ A, const double* __restrict__ B, int n, int vstride, double* out,
                      const PcgScalars* sc, int force) {
  const int k = blockIdx.y;
  if (!force && !sc[k].active) return;
  double s = 0.0;
  const double* a = A + static_cast<size_t>(k) * vstride;
  const double* b = B + static_cast<size_t>(k) * vstride;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) s += a[i] * b[i];
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double ws[32];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = threadIdx.x < (blockDim.x >> 5) ? ws[threadIdx.x] : 0.0;
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) atomicAdd(&out[k], s);
  }
}

// r -= p on solved planes.
__global__ void k_sub(double* __restrict__ R, const double* __restrict__ P, int n, int vstride,
                      const PcgScalars* sc) {
  const int k = blockIdx.y;
  if (!sc[k].solved) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    R[static_cast<size_t>(k) * vstride + i] -= P[static_cast<size_t>(k) * vstride + i];
}

__global__ void k_pcg_init(PcgScalars* sc, const double* bb, const double* rr, double tol, int nz) {
  const int k = threadIdx.x;
  if (k >= nz) return;
  PcgScalars s{};
  const double e = tol * sqrt(bb[k]);
  s.eps = e * e;
  s.r2 = rr[k];
  s.solved = s.active = !(nz > 1 && k == 1);
  sc[k] = s;
}

// Loop head `while (r2 > epsb2 && ++i < StepMax)`.
__global__ void k_pcg_head(PcgScalars* sc, int step_max, int nz, int* any_active) {
  const int k = threadIdx.x;
  if (k >= nz) return;
  PcgScalars& s = sc[k];
  if (s.active) {
    if (s.r2 > s.eps) {
      s.iter += 1;
      if (s.iter >= step_max) {
        s.active = 0;
        s.hit_max = 1;
      }
    } else {
      s.active = 0;
    }
  }
  if (s.active) atomicOr(any_active, 1);
}

__global__ void k_pcg_precond(const double* __restrict__ PC, int npts, const double* __restrict__ R,
                              double* __restrict__ Z, int vstride, const PcgScalars* sc) {
  const int k = blockIdx.y;
  if (!sc[k].active) return;
  const double* pc = PC + static_cast<size_t>(k >> 1) * npts;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npts; i += gridDim.x * blockDim.x)
    Z[static_cast<size_t>(k) * vstride + i] = pc[i] * R[static_cast<size_t>(k) * vstride + i];
}

__global__ void k_pcg_dir(const double* __restrict__ Z, double* __restrict__ P, int n, int vstride,
                          const PcgScalars* sc, const double* rho1) {
  const int k = blockIdx.y;
  if (!sc[k].active) return;
  const bool first = sc[k].iter == 1;
  const double beta = first ? 0.0 : rho1[k] / sc[k].rho2;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const size_t o = static_cast<size_t>(k) * vstride + i;
    P[o] = first ? Z[o] : Z[o] + beta * P[o];
  }
}

__global__ void k_pcg_step(double* __restrict__ X, double* __restrict__ R, const double* __restrict__ P,
                           const double* __restrict__ Q, int n, int vstride, const PcgScalars* sc,
                           const double* rho1, const double* dotp) {
  const int k = blockIdx.y;
  if (!sc[k].active) return;
  const double alpha = rho1[k] / dotp[k];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const size_t o = static_cast<size_t>(k) * vstride + i;
    X[o] += alpha * P[o];
    R[o] -= alpha * Q[o];
  }
}

__global__ void k_pcg_tail(PcgScalars* sc, const double* rho1, const double* r2, int nz) {
  const int k = threadIdx.x;
  if (k >= nz || !sc[k].active) return;
  sc[k].rho2 = rho1[k];
  sc[k].r2 = r2[k];
}

__global__ void k_pcg_out(const PcgScalars* sc, int nz, int2* out) {
  const int k = threadIdx.x;
  if (k < nz) out[k] = make_int2(sc[k].iter, sc[k].hit_max);
}

constexpr int kPcgMaxPlanes = 1024;  // one thread a plane in the scalar kernels

cudaError_t pcg_launches(const DevGeom& g, const DevNumbering& N, const DevModal& S, const PcgVectors& v,
                         double tol_rel, int step_max, cudaStream_t st) {
  const int nz = g.nz, npts = v.npts, vs = v.vstride;
  double *r = v.r, *x = v.x, *q = v.q, *p = v.p0, *z = v.p1;
  double *rho1 = v.scal, *dotp = rho1 + nz, *r2 = dotp + nz, *bb = r2 + nz;
  int* flag = reinterpret_cast<int*>(bb + nz);
  PcgScalars* sc = reinterpret_cast<PcgScalars*>(bb + 2 * nz);
  const int nzt = (nz + 31) / 32 * 32;
  const int threads = std::max(64, (g.npnp + 31) / 32 * 32);
  const size_t shm = sizeof(double) * (static_cast<size_t>(g.np) * g.np + 3 * g.npnp);
  const size_t plane_bytes = sizeof(double) * static_cast<size_t>(vs) * nz;
  const dim3 egrid(g.nel, nz);
  const dim3 vgrid(std::min(1024, (npts + 255) / 256), nz);
  const dim3 zgrid(std::max(1, std::min(64, (N.nglobal + 255) / 256)), nz);
  cudaError_t err = cudaMemsetAsync(v.scal, 0, sizeof(double) * pcg_scalar_doubles(nz), st);
  if (err == cudaSuccess) err = cudaMemsetAsync(p, 0, plane_bytes, st);
  if (err != cudaSuccess) return err;
  k_zero_fixed<<<zgrid, 256, 0, st>>>(r, vs, S.nsolve, N.nglobal);
  k_dot<<<vgrid, 256, 0, st>>>(r, r, npts, vs, bb, sc, 1);
  // the essential entries of the guess are zero; r -= H x
  k_zero_fixed<<<zgrid, 256, 0, st>>>(x, vs, S.nsolve, N.nglobal);
  k_pcg_init<<<1, nzt, 0, st>>>(sc, bb, bb, tol_rel, nz);
  k_global_op<<<egrid, threads, shm, st>>>(g, N, S, x, p, vs, sc);
  k_zero_fixed<<<zgrid, 256, 0, st>>>(p, vs, S.nsolve, N.nglobal);
  k_sub<<<vgrid, 256, 0, st>>>(r, p, npts, vs, sc);
  k_dot<<<vgrid, 256, 0, st>>>(r, r, npts, vs, r2, sc, 1);
  k_pcg_init<<<1, nzt, 0, st>>>(sc, bb, r2, tol_rel, nz);
  for (int it = 0; it < step_max + 1; ++it) {
    cudaMemsetAsync(flag, 0, sizeof(int), st);
    k_pcg_head<<<1, nzt, 0, st>>>(sc, step_max, nz, flag);
    if ((it & 7) == 0) {
      int active = 0;
      cudaMemcpyAsync(&active, flag, sizeof(int), cudaMemcpyDeviceToHost, st);
      err = cudaStreamSynchronize(st);
      if (err != cudaSuccess) return err;
      if (!active) break;
    }
    k_pcg_precond<<<vgrid, 256, 0, st>>>(S.pc, S.npts, r, z, vs, sc);
    cudaMemsetAsync(rho1, 0, sizeof(double) * nz, st);
    k_dot<<<vgrid, 256, 0, st>>>(r, z, npts, vs, rho1, sc, 0);
    k_pcg_dir<<<vgrid, 256, 0, st>>>(z, p, npts, vs, sc, rho1);
    cudaMemsetAsync(q, 0, plane_bytes, st);
    k_global_op<<<egrid, threads, shm, st>>>(g, N, S, p, q, vs, sc);
    k_zero_fixed<<<zgrid, 256, 0, st>>>(q, vs, S.nsolve, N.nglobal);
    cudaMemsetAsync(dotp, 0, sizeof(double) * nz, st);
    k_dot<<<vgrid, 256, 0, st>>>(p, q, npts, vs, dotp, sc, 0);
    k_pcg_step<<<vgrid, 256, 0, st>>>(x, r, p, q, npts, vs, sc, rho1, dotp);
    cudaMemsetAsync(r2, 0, sizeof(double) * nz, st);
    k_dot<<<vgrid, 256, 0, st>>>(r, r, npts, vs, r2, sc, 0);
    k_pcg_tail<<<1, nzt, 0, st>>>(sc, rho1, r2, nz);
  }
  k_pcg_out<<<1, nzt, 0, st>>>(sc, nz, v.out);
  return cudaGetLastError();
}

// Blocks per plane: enough warps for one element each, up to 8 blocks, or 16
// while every plane's 16 have an SM of their own and the device can place
// such a cluster (16 is past the portable size; launch_pcg asks).  us an iteration (B200, 4 / 8
// / 16 blocks of 8 warps a plane): 8 x 8 elements, N_P = 9, 15 planes 13.3 /
// 7.4 / 15.0; 12 x 12, N_P = 13, 23 planes 45.8 / 27.6 / 39.2; 12 x 12, N_P =
// 8, 3 planes 14.2 / 8.3 / 6.9; 12 x 10, N_P = 11, 1 plane 29.1 / 13.7 / 9.2;
// 24 x 24, N_P = 9, 95 planes 179 / 124 / 167.  Blocks of 16 warps: 9.6 (8 x
// 8), 40.4 and 7.7 (12 x 12), 166 (24 x 24) at 8 a plane.
int pcg_cluster(int nel, int planes) {
  const int want = (nel + kPcgWarps - 1) / kPcgWarps;
  int device = 0, sms = 0;
  cudaGetDevice(&device);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  const int room = planes * kPcgMaxCluster <= sms ? kPcgMaxCluster : kPcgPortable;
  int c = 1;
  while (c < want && c < room) c *= 2;
  return c;
}

// Whether the iteration runs as launches: where they are estimated faster than
// one cluster a plane.  us an iteration, launches / clusters (B200): one plane
// of 24 x 24 elements, N_P = 9 54 / 23, 44 x 44 58 / 66, 60 x 60 64 / 116, 100
// x 100, N_P = 7 67 / 146, 80 x 60, N_P = 5 56 / 66, 24 x 24, N_P = 16 67 /
// 43, N_P = 18 63 / 129; 3 planes 40 x 40, N_P = 9 64 / 55, 50 x 50 77 / 82, 32 x 32, N_P = 16
// 137 / 70; 9 planes 40 x 40, N_P = 9 101 / 63; 11 planes 60 x 60 208 / 279;
// 15 planes 64 x 64, N_P = 6 153 / 126; 31 planes 32 x 32, N_P = 9 177 / 86.
// The estimates: a cluster's warps each do their elements in turn (products
// padded to 8 or 16 nodes a side, above that without the tensor cores), the
// launches go over all points.
bool pcg_by_launches(const DevGeom& g, const DevModal& S, int planes) {
  if (g.nz > kPcgMaxPlanes || S.pcg_launches == 0) return false;
  if (S.pcg_launches == 1) return true;
  const double elements_a_warp = static_cast<double>(g.nel) / (kPcgWarps * pcg_cluster(g.nel, planes));
  const double element_us = g.np <= 8 ? 1.8 : g.np <= 16 ? 2.1 + 0.0234 * g.npnp : 0.085 * g.npnp;
  const double point_us = g.np < 16 ? 5e-5 : g.np == 16 ? 1e-4 : 7e-5;
  return 52.0 + point_us * g.nel * g.npnp * planes < 5.0 + elements_a_warp * element_us;
}

template <int MT, int KS>
cudaError_t launch_pcg(const DevGeom& g, const DevNumbering& N, const DevModal& S, const PcgVectors& v,
                       double tol_rel, int step_max, cudaStream_t st) {
  const int planes = g.nz > 1 ? g.nz - 1 : 1;
  int c = pcg_cluster(g.nel, planes);
  const size_t smem = sizeof(double) * (static_cast<size_t>(g.np) * g.np + 3 * static_cast<size_t>(kPcgWarps) * g.npnp);
  auto kernel = k_pcg<MT, KS>;
  raise_smem_limit(reinterpret_cast<const void*>(kernel), smem);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(planes * c);
  cfg.blockDim = dim3(kPcgThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = c;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (c > kPcgPortable) {
    int fit = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) != cudaSuccess || fit < 1) {
      cudaGetLastError();  // not an error of the solve
      c = kPcgPortable;
      cfg.gridDim = dim3(planes * c);
      attr[0].val.clusterDim.x = c;
    }
  }
  return cudaLaunchKernelEx(&cfg, kernel, g, N, S, v, tol_rel, step_max);
}

}  // namespace

size_t pcg_scalar_doubles(int nz) {
  return (6 * sizeof(double) + sizeof(PcgScalars)) * static_cast<size_t>(nz) / sizeof(double);
}

cudaError_t pcg_iterate(const DevGeom& g, const DevNumbering& N, const DevModal& S, const PcgVectors& v,
                        double tol_rel, int step_max, cudaStream_t st) {
  if (pcg_by_launches(g, S, g.nz > 1 ? g.nz - 1 : 1)) return pcg_launches(g, N, S, v, tol_rel, step_max, st);
  if (g.np <= 4) return launch_pcg<1, 1>(g, N, S, v, tol_rel, step_max, st);
  if (g.np <= 8) return launch_pcg<1, 2>(g, N, S, v, tol_rel, step_max, st);
  if (g.np <= 12) return launch_pcg<2, 3>(g, N, S, v, tol_rel, step_max, st);
  if (g.np <= 16) return launch_pcg<2, 4>(g, N, S, v, tol_rel, step_max, st);
  return launch_pcg<0, 0>(g, N, S, v, tol_rel, step_max, st);
}

}  // namespace stx
