// z-direction real DFT of field planes (AuxField::transform,
// src/auxfield.cpp:1157-1194, contract of femlib/fourier.c:40-165).
//
// Forward (sign +1), scaled by 1/nz:  c_k = (1/nz) sum_n x_n exp(-2 pi i k n / nz),
// packed per point as [Re c_0, Re c_{nz/2}, Re c_1, Im c_1, Re c_2, ...].
// Inverse (sign -1):  x_n = c_0 + c_{nz/2} (-1)^n + 2 sum_k (Re c_k cos - Im c_k sin).
// nz == 2 follows the reference special case (forward zeroes plane 1,
// inverse copies plane 0 to plane 1).
//
// The reference layout keeps the z-lines strided by plane_size, so a block
// owns 32 consecutive points of every plane: loads and stores of each plane
// row are coalesced, and the transform runs out of shared memory.  The DNS
// step's z work is folded in (k_z): both the values and the z-derivative of
// a spectrum from one read of it, the z-derivative of a product of two fields
// without its spectrum ever leaving the block, the zero padding and the
// truncation of the 3/2 rule, and the three velocity components in one
// launch.
#include "fourier.cuh"

#include <algorithm>
#include <vector>

#include "helmholtz.cuh"
#include "launch.hpp"
#include "ptx.cuh"

namespace stx {

namespace {

constexpr int kTP = 32;  // points per block

__global__ void k_dft(double* __restrict__ data, int nz, int plane_size, int sign,
                      const double* __restrict__ twiddle) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ double sm[];
  double* x = sm;             // [nz][kTP]
  double* tw = sm + nz * kTP; // [2][nz]
  const int p0 = blockIdx.x * kTP;
  for (int t = threadIdx.x; t < 2 * nz; t += blockDim.x) tw[t] = twiddle[t];
  for (int t = threadIdx.x; t < nz * kTP; t += blockDim.x) {
    const int k = t / kTP, p = t - k * kTP;
    x[t] = (p0 + p < plane_size) ? data[static_cast<size_t>(k) * plane_size + p0 + p] : 0.0;
  }
  __syncthreads();
  const int half = nz >> 1;
  const double scale = 1.0 / nz;
  for (int t = threadIdx.x; t < nz * kTP; t += blockDim.x) {
    const int q = t / kTP, p = t - q * kTP;
    double v = 0.0;
    if (sign > 0) {
      const int kf = q == 0 ? 0 : (q == 1 ? half : q >> 1);
      const bool im = q >= 2 && (q & 1);
      int idx = 0;
      for (int n = 0; n < nz; ++n) {
        v += x[n * kTP + p] * (im ? -tw[nz + idx] : tw[idx]);
        idx += kf;
        if (idx >= nz) idx -= nz;
      }
      v *= scale;
    } else {
      const int n = q;
      v = x[p] + ((n & 1) ? -x[kTP + p] : x[kTP + p]);
      int idx = n, step = n;
      for (int k = 1; k < half; ++k) {
        v += 2.0 * (x[(2 * k) * kTP + p] * tw[idx] - x[(2 * k + 1) * kTP + p] * tw[nz + idx]);
        idx += step;
        if (idx >= nz) idx -= nz;
      }
    }
    sm[nz * kTP + 2 * nz + t] = v;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < nz * kTP; t += blockDim.x) {
    const int k = t / kTP, p = t - k * kTP;
    if (p0 + p < plane_size)
      data[static_cast<size_t>(k) * plane_size + p0 + p] = sm[nz * kTP + 2 * nz + t];
  }
}

// ---------------------------------------------------------------------------
// Mixed-radix Stockham FFT of the z-lines of 2 TPC consecutive points per
// block, two real lines (columns q and q + TPC of the block) as one complex
// line z = x + i x'.  Few, large radices (up to 8) keep a line's points in
// registers: a transform of 96 points is three passes over shared memory, the
// first reading global memory (or the landed spectrum), the last writing it.
// Twiddles w^m = exp(-2 pi i m / n) come from the same host-computed table as
// the DFT's.
//
// Bound: HBM (a read and a write of each plane), as far as enough lines are
// in flight.  Three fields of 46656 x 96 points (107 MB; B200): forward 58 us,
// inverse 81 us, inverse with z-derivative 130 us, z-derivative of a product
// 87 us, where a pass per field and operation took 29 us a transform, 12 us a
// copy, 15 us a derivative and 16 us a product (88, 126, 261 and 313 us).
// 32 points a block and radices up to 8 in 80 registers (which spill 72 to 312
// bytes a thread, by instance) measured best: radix 12 (two passes, 128
// registers, two blocks an SM) 65 / 101 / 155 / 87 us, 16 points a block 63 /
// 89 / 141 / 88 (radix 12) and 67 / 89 / 153 / 102 us.
// ---------------------------------------------------------------------------

// Radices of the passes, 4 bits each from the lowest (read with shifts: a
// kernel parameter indexed at run time would be copied to local memory).
struct FftPlan {
  int nf;
  unsigned long long radices;
  __device__ int dradix(int f) const { return static_cast<int>((radices >> (4 * f)) & 15u); }
};

// cos(2 pi m / 24), sin(2 pi m / 24): the twiddles inside radices 6 and 8.
__host__ __device__ constexpr double cos24(int m) {
  m = m % 24;
  if (m < 0) m += 24;
  if (m > 12) m = 24 - m;
  const double c[7] = {1.0, 0.96592582628906828675, 0.86602540378443864676, 0.70710678118654752440, 0.5,
                       0.25881904510252076235, 0.0};
  return m <= 6 ? c[m] : -c[12 - m];
}
__host__ __device__ constexpr double sin24(int m) { return cos24(m - 6); }

// In-place length-R DFT of (vr, vi), exponent sign S (-1 forward, +1 inverse).
template <int R, int S>
struct Dft;

template <int S>
struct Dft<2, S> {
  static __device__ __forceinline__ void run(double* vr, double* vi) {
    const double ar = vr[0], ai = vi[0];
    vr[0] = ar + vr[1];
    vi[0] = ai + vi[1];
    vr[1] = ar - vr[1];
    vi[1] = ai - vi[1];
  }
};

template <int S>
struct Dft<3, S> {
  static __device__ __forceinline__ void run(double* vr, double* vi) {
    constexpr double c = -0.5, sn = S * 0.86602540378443864676;  // sin(2 pi / 3)
    const double sr = vr[1] + vr[2], si = vi[1] + vi[2];
    const double dr = vr[1] - vr[2], di = vi[1] - vi[2];
    const double ar = vr[0] + c * sr, ai = vi[0] + c * si;
    vr[0] += sr;
    vi[0] += si;
    // (dr + i di) * (i sn) = -sn di + i sn dr
    vr[1] = ar - sn * di;
    vi[1] = ai + sn * dr;
    vr[2] = ar + sn * di;
    vi[2] = ai - sn * dr;
  }
};

template <int S>
struct Dft<4, S> {
  static __device__ __forceinline__ void run(double* vr, double* vi) {
    const double t0r = vr[0] + vr[2], t0i = vi[0] + vi[2];
    const double t1r = vr[0] - vr[2], t1i = vi[0] - vi[2];
    const double t2r = vr[1] + vr[3], t2i = vi[1] + vi[3];
    const double t3r = vr[1] - vr[3], t3i = vi[1] - vi[3];
    // multiply t3 by S i: (x + iy) * (S i) = -S y + i S x
    const double ur = -S * t3i, ui = S * t3r;
    vr[0] = t0r + t2r;
    vi[0] = t0i + t2i;
    vr[2] = t0r - t2r;
    vi[2] = t0i - t2i;
    vr[1] = t1r + ur;
    vi[1] = t1i + ui;
    vr[3] = t1r - ur;
    vi[3] = t1i - ui;
  }
};

template <int S>
struct Dft<5, S> {
  static __device__ __forceinline__ void run(double* vr, double* vi) {
    constexpr double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;   // cos(2pi/5), cos(4pi/5)
    constexpr double s1 = S * 0.95105651629515357212, s2 = S * 0.58778525229247312917;  // sin(2pi/5), sin(4pi/5)
    const double a1r = vr[1] + vr[4], a1i = vi[1] + vi[4], b1r = vr[1] - vr[4], b1i = vi[1] - vi[4];
    const double a2r = vr[2] + vr[3], a2i = vi[2] + vi[3], b2r = vr[2] - vr[3], b2i = vi[2] - vi[3];
    const double x0r = vr[0], x0i = vi[0];
    const double p1r = x0r + c1 * a1r + c2 * a2r, p1i = x0i + c1 * a1i + c2 * a2i;
    const double p2r = x0r + c2 * a1r + c1 * a2r, p2i = x0i + c2 * a1i + c1 * a2i;
    // q = i * (s1 b1 + s2 b2), r = i * (s2 b1 - s1 b2)
    const double q1r = -(s1 * b1i + s2 * b2i), q1i = s1 * b1r + s2 * b2r;
    const double q2r = -(s2 * b1i - s1 * b2i), q2i = s2 * b1r - s1 * b2r;
    vr[0] = x0r + a1r + a2r;
    vi[0] = x0i + a1i + a2i;
    vr[1] = p1r + q1r;
    vi[1] = p1i + q1i;
    vr[4] = p1r - q1r;
    vi[4] = p1i - q1i;
    vr[2] = p2r + q2r;
    vi[2] = p2i + q2i;
    vr[3] = p2r - q2r;
    vi[3] = p2i - q2i;
  }
};

// R = R1 R2 dividing 24: the points n = R2 n1 + n2 by R1-point transforms
// over n1, twiddles, R2-point transforms over n2; X at k1 + R1 k2.
template <int R1, int R2, int S>
struct DftPair {
  static __device__ __forceinline__ void run(double* vr, double* vi) {
    constexpr int R = R1 * R2;
    double yr[R], yi[R];
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) {
      double tr[R1], ti[R1];
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) {
        tr[n1] = vr[R2 * n1 + n2];
        ti[n1] = vi[R2 * n1 + n2];
      }
      Dft<R1, S>::run(tr, ti);
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) {
        const double c = cos24(n2 * k1 * (24 / R)), s = S * sin24(n2 * k1 * (24 / R));
        if (n2 * k1 == 0) {
          yr[n2 * R1 + k1] = tr[k1];
          yi[n2 * R1 + k1] = ti[k1];
        } else {
          yr[n2 * R1 + k1] = tr[k1] * c - ti[k1] * s;
          yi[n2 * R1 + k1] = ti[k1] * c + tr[k1] * s;
        }
      }
    }
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) {
      double tr[R2], ti[R2];
#pragma unroll
      for (int n2 = 0; n2 < R2; ++n2) {
        tr[n2] = yr[n2 * R1 + k1];
        ti[n2] = yi[n2 * R1 + k1];
      }
      Dft<R2, S>::run(tr, ti);
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) {
        vr[k1 + R1 * k2] = tr[k2];
        vi[k1 + R1 * k2] = ti[k2];
      }
    }
  }
};

template <int S>
struct Dft<6, S> : DftPair<2, 3, S> {};
template <int S>
struct Dft<8, S> : DftPair<2, 4, S> {};

// A prime R without a formula of its own (7): the sums themselves,
// twiddles from the table of the whole length N.
template <int R, int S>
__device__ __forceinline__ void prime_dft(double* vr, double* vi, const double* tw, int N) {
  double yr[R], yi[R];
  const int step = N / R;
#pragma unroll
  for (int c = 0; c < R; ++c) {
    double ar = vr[0], ai = vi[0];
#pragma unroll
    for (int r = 1; r < R; ++r) {
      const int m = (r * c % R) * step;
      const double wr = tw[m], wi = S * tw[N + m];
      ar += vr[r] * wr - vi[r] * wi;
      ai += vi[r] * wr + vr[r] * wi;
    }
    yr[c] = ar;
    yi[c] = ai;
  }
#pragma unroll
  for (int c = 0; c < R; ++c) {
    vr[c] = yr[c];
    vi[c] = yi[c];
  }
}

// One radix-R pass over TPC complex lines of N points, Ns of them already
// transformed: ld(n, q, re, im) reads point n of line q, st(n, q, re, im)
// writes it.
template <int R, int S, int TPC, class Ld, class St>
__device__ __forceinline__ void fft_pass_r(int N, int Ns, const double* tw, Ld& ld, St& st) {
  const int nj = N / R;
  for (int w = threadIdx.x; w < nj * TPC; w += blockDim.x) {
    const int j = w / TPC, q = w - j * TPC;
    const int k = Ns == 1 ? 0 : (Ns == nj ? j : j % Ns);
    double vr[R], vi[R];
#pragma unroll
    for (int r = 0; r < R; ++r) ld(j + r * nj, q, vr[r], vi[r]);
    if (k) {
      // twiddle exp(S 2 pi i r k / (Ns R)) = table entry r k N / (Ns R) (< N)
      const int step = k * (nj / Ns);
#pragma unroll
      for (int r = 1; r < R; ++r) {
        const double c = tw[r * step], s = S * tw[N + r * step];
        const double t = vr[r] * c - vi[r] * s;
        vi[r] = vi[r] * c + vr[r] * s;
        vr[r] = t;
      }
    }
    if constexpr (R == 7) prime_dft<R, S>(vr, vi, tw, N);
    else Dft<R, S>::run(vr, vi);
    const int base = (j - k) * R + k;  // (j / Ns) Ns R + k
#pragma unroll
    for (int r = 0; r < R; ++r) st(base + r * Ns, q, vr[r], vi[r]);
  }
}

template <int S, int TPC, class Ld, class St>
__device__ __forceinline__ void fft_pass(int R, int N, int Ns, const double* tw, Ld ld, St st) {
  switch (R) {
    case 2: fft_pass_r<2, S, TPC>(N, Ns, tw, ld, st); break;
    case 3: fft_pass_r<3, S, TPC>(N, Ns, tw, ld, st); break;
    case 4: fft_pass_r<4, S, TPC>(N, Ns, tw, ld, st); break;
    case 5: fft_pass_r<5, S, TPC>(N, Ns, tw, ld, st); break;
    case 6: fft_pass_r<6, S, TPC>(N, Ns, tw, ld, st); break;
    case 7: fft_pass_r<7, S, TPC>(N, Ns, tw, ld, st); break;
    default: fft_pass_r<8, S, TPC>(N, Ns, tw, ld, st); break;
  }
  __syncthreads();
}

// A whole transform (at least two passes): the first pass by `ld`, the last
// by `st`, between them shared-memory buffers a, b in turn ([n][2 TPC]).
template <int S, int TPC, class Ld, class St>
__device__ __forceinline__ void fft_run(const FftPlan& plan, int N, const double* tw, double* a, double* b, Ld ld,
                                        St st) {
  constexpr int LD = 2 * TPC;
  auto to = [](double* y) {
    return [y](int n, int q, double re, double im) {
      y[n * LD + q] = re;
      y[n * LD + q + TPC] = im;
    };
  };
  auto from = [](const double* x) {
    return [x](int n, int q, double& re, double& im) {
      re = x[n * LD + q];
      im = x[n * LD + q + TPC];
    };
  };
  int Ns = plan.dradix(0);
  fft_pass<S, TPC>(Ns, N, 1, tw, ld, to(a));
  for (int f = 1; f + 1 < plan.nf; ++f) {
    const int R = plan.dradix(f);
    fft_pass<S, TPC>(R, N, Ns, tw, from(a), to(b));
    Ns *= R;
    double* t = a;
    a = b;
    b = t;
  }
  fft_pass<S, TPC>(plan.dradix(plan.nf - 1), N, Ns, tw, from(a), st);
}

// Set when a bounded wait for bulk copies expired (the block then leaves its
// lines untransformed).
__device__ int g_fft_timeout = 0;

enum { kZForward = 0, kZInverse = 1, kZInverseDz = 2, kZProductDz = 3 };

struct ZArgs {
  ZBatch b;
  int n, nin, nout, keep, plane_size, bulk;
  double beta;
  const double* twiddle;
  FftPlan plan;
};

template <int OP, int TPC>
__global__ void __launch_bounds__(256, 3) k_z(ZArgs z) {
  pdl_trigger();
  pdl_wait();
  constexpr int LD = 2 * TPC;
  extern __shared__ __align__(16) double sm[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm);
  const int N = z.n, half = N / 2, f = blockIdx.y;
  double* tw = sm + 2;      // [2][N]
  double* A = tw + 2 * N;   // [N][LD] each
  double* B = A + N * LD;
  double* C = B + N * LD;   // kZInverseDz of three or more passes
  const int p0 = blockIdx.x * LD, cnt = min(LD, z.plane_size - p0);
  const size_t ps = z.plane_size;
  const double* in = z.b.in[f];
  double* out = z.b.out[f];
  for (int t = threadIdx.x; t < 2 * N; t += blockDim.x) tw[t] = z.twiddle[t];

  // real lines q, q + TPC of a physical field
  auto put_lines = [&](double* dst) {
    return [=](int n, int q, double re, double im) {
      double* row = dst + n * ps + p0;
      if (q < cnt) row[q] = re;
      if (q + TPC < cnt) row[q + TPC] = im;
    };
  };

  if constexpr (OP == kZForward || OP == kZProductDz) {
    __syncthreads();  // twiddles
    const double* mul = OP == kZProductDz ? z.b.mul[f] : nullptr;
    double* X = z.plan.nf & 1 ? A : B;  // where the last pass of the forward transform lands
    double* Y = z.plan.nf & 1 ? B : A;
    fft_run<-1, TPC>(
        z.plan, N, tw, A, B,
        [&](int n, int q, double& re, double& im) {
          const size_t o = n * ps + p0 + q;
          re = q < cnt ? in[o] : 0.0;
          im = q + TPC < cnt ? in[o + TPC] : 0.0;
          if (OP == kZProductDz) {
            re *= q < cnt ? mul[o] : 0.0;
            im *= q + TPC < cnt ? mul[o + TPC] : 0.0;
          }
        },
        [=](int n, int q, double re, double im) {
          X[n * LD + q] = re;
          X[n * LD + q + TPC] = im;
        });
    if constexpr (OP == kZForward) {
      // X_k = (Z_k + conj Z_{N-k}) / 2, X'_k = (Z_k - conj Z_{N-k}) / 2i, packed and scaled
      const double scale = 0.5 / N;
      for (int t = threadIdx.x; t < z.nout * TPC; t += blockDim.x) {
        const int n = t / TPC, q = t - n * TPC;
        const int k = n == 0 ? 0 : (n == 1 ? half : n >> 1);
        const bool im = n >= 2 && (n & 1);
        const int kn = k == 0 ? 0 : N - k;
        const double zr = X[k * LD + q], zi = X[k * LD + q + TPC];
        const double wr = X[kn * LD + q], wi = X[kn * LD + q + TPC];
        const double v0 = im ? (zi - wi) : (zr + wr);   // line q
        const double v1 = im ? (wr - zr) : (zi + wi);   // line q + TPC
        double* row = out + n * ps + p0;
        if (q < cnt) row[q] = v0 * scale;
        if (q + TPC < cnt) row[q + TPC] = v1 * scale;
      }
    } else {
      // the derivative is linear and real, so it acts on the complex line as
      // a whole: Z_k -> i k beta Z_k / N
      const double c = z.beta / N;
      const int keep = z.keep;
      fft_run<1, TPC>(
          z.plan, N, tw, Y, X,
          [=](int k, int q, double& re, double& im) {
            const int kk = k <= half ? k : k - N;
            const double s = (kk < keep && kk > -keep) ? kk * c : 0.0;
            re = -s * X[k * LD + q + TPC];
            im = s * X[k * LD + q];
          },
          put_lines(out));
    }
  } else {
    // the packed spectra land in B
    const int nin = z.nin;
    if (z.bulk) {
      if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(bar, static_cast<unsigned>(sizeof(double) * nin * cnt));
      }
      __syncthreads();  // armed before any copy can complete
      if (threadIdx.x < 32)
        for (int n = threadIdx.x; n < nin; n += 32)
          bulk_g2s(B + n * LD, in + n * ps + p0, static_cast<unsigned>(sizeof(double) * cnt), bar);
      if (cnt < LD)
        for (int t = threadIdx.x; t < nin * LD; t += blockDim.x)
          if (t % LD >= cnt) B[t] = 0.0;  // columns no copy writes
      const bool ok = __syncthreads_and(mbar_wait(bar, 0));
      if (!ok) {
        if (threadIdx.x == 0) atomicExch(&g_fft_timeout, 1);
        mbar_wait(bar, 0);
        return;
      }
    } else {
      for (int t = threadIdx.x; t < nin * LD; t += blockDim.x) {
        const int n = t / LD, c = t - n * LD;
        B[t] = (c < cnt) ? in[n * ps + p0 + c] : 0.0;
      }
      __syncthreads();
    }
    // X_k of column c (plane 0 = Re X_0, 1 = Re X_{N/2}, 2k / 2k+1 = Re / Im
    // X_k, zero from plane nin on; X_{N-k} = conj X_k)
    auto spectrum = [=](int k, int c, double& re, double& im) {
      if (k == 0 || k == half) {
        re = B[(k ? LD : 0) + c];
        im = 0.0;
      } else {
        const int m = k < half ? k : N - k;
        const bool have = 2 * m < nin;
        re = have ? B[(2 * m) * LD + c] : 0.0;
        im = have ? B[(2 * m + 1) * LD + c] : 0.0;
        if (k > half) im = -im;
      }
    };
    // Z_k = X_k + i X'_k of columns q and q + TPC
    fft_run<1, TPC>(
        z.plan, N, tw, A, OP == kZInverseDz ? C : B,
        [=](int k, int q, double& re, double& im) {
          double r0, i0, r1, i1;
          spectrum(k, q, r0, i0);
          spectrum(k, q + TPC, r1, i1);
          re = r0 - i1;
          im = i0 + r1;
        },
        put_lines(out));
    if constexpr (OP == kZInverseDz) {
      const double beta = z.beta;
      fft_run<1, TPC>(
          z.plan, N, tw, A, C,
          [=](int k, int q, double& re, double& im) {
            double r0, i0, r1, i1;
            spectrum(k, q, r0, i0);
            spectrum(k, q + TPC, r1, i1);
            const double s = k == half ? 0.0 : beta * (k < half ? k : k - N);
            re = -s * (i0 + r1);
            im = s * (r0 - i1);
          },
          put_lines(z.b.dz[f]));
    }
  }
}

__global__ void k_nz2(double* data, int plane_size, int sign) {
  pdl_trigger();
  pdl_wait();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= plane_size) return;
  data[plane_size + p] = sign > 0 ? 0.0 : data[p];
}

// The fewest passes over the radices there are; of equal ones the one whose
// largest radix is least (even passes).  nf = 0: n has another prime factor or would
// be a single pass.
FftPlan find_plan(int n) {
  constexpr int radix[] = {8, 7, 6, 5, 4, 3, 2};  // a plan's first is its largest
  FftPlan best{};
  auto search = [&](auto&& self, int left, int from, FftPlan p) -> void {
    if (left == 1) {
      if (p.nf >= 2 && (best.nf == 0 || p.nf < best.nf || (p.radices & 15u) < (best.radices & 15u))) best = p;
      return;
    }
    if (p.nf >= 15 || (best.nf && p.nf >= best.nf)) return;
    for (int r = from; r < 7; ++r)
      if (left % radix[r] == 0) {
        FftPlan q = p;
        q.radices |= static_cast<unsigned long long>(radix[r]) << (4 * q.nf++);
        self(self, left / radix[r], r, q);
      }
  };
  if (n > 2 && n % 2 == 0) search(search, n, 0, FftPlan{});
  return best;
}

// The plans of every length the shared memory admits, made once.
FftPlan fft_plan(int n) {
  static const std::vector<FftPlan> plans = [] {
    std::vector<FftPlan> p(2561);
    for (int k = 4; k < static_cast<int>(p.size()); k += 2) p[k] = find_plan(k);
    return p;
  }();
  return n > 0 && n < static_cast<int>(plans.size()) ? plans[n] : FftPlan{};
}

size_t z_smem(int n, int tpc, int buffers) {
  return sizeof(double) * (2 + 2 * static_cast<size_t>(n) + static_cast<size_t>(buffers) * n * 2 * tpc);
}

constexpr size_t kZSmemLimit = 200 * 1024;
constexpr size_t kZTwoBlocks = 112 * 1024;

template <int OP>
cudaError_t z_launch(ZArgs z, cudaStream_t st, bool pdl) {
  z.plan = fft_plan(z.n);
  if (z.plan.nf == 0 || z.b.count < 1 || z.b.count > kZBatch) return cudaErrorInvalidValue;
  const int buffers = OP == kZInverseDz && z.plan.nf > 2 ? 3 : 2;
  // 32 points a block (256-byte rows) while two blocks fit an SM, then 16, 8
  // and 4.  us forward / inverse of 5184 points a plane, with 4 points where
  // 32 do not fit / so: 216 planes 16.5 and 26.8 / 11.7 and 16.6, 256 planes
  // 18.6 and 30.9 / 12.4 and 18.6, 512 planes 33.5 and 57.5 / 23.9 and 50.7;
  // a DNS step of 8 x 8, N_P = 9, 256 planes 494 / 426
  int tpc = 16;
  while (tpc > 2 && z_smem(z.n, tpc, buffers) > kZTwoBlocks) tpc /= 2;
  const size_t smem = z_smem(z.n, tpc, buffers);
  if (smem > kZSmemLimit) return cudaErrorInvalidValue;
  // bulk row copies need 16-byte aligned rows: aligned bases and an even
  // plane size
  z.bulk = z.plane_size % 2 == 0;
  for (int i = 0; i < z.b.count; ++i) z.bulk = z.bulk && reinterpret_cast<uintptr_t>(z.b.in[i]) % 16 == 0;
  int rmin = 16;
  for (int f = 0; f < z.plan.nf; ++f) rmin = std::min(rmin, static_cast<int>((z.plan.radices >> (4 * f)) & 15u));
  const int threads = std::max(64, std::min(256, (z.n / rmin * tpc + 31) / 32 * 32));
  const dim3 grid((z.plane_size + 2 * tpc - 1) / (2 * tpc), z.b.count);
  auto go = [&](auto kernel) {
    raise_smem_limit(reinterpret_cast<const void*>(kernel), smem);
    return launch_ex(pdl, kernel, grid, dim3(threads), smem, st, z);
  };
  const cudaError_t err = tpc == 16  ? go(k_z<OP, 16>)
                          : tpc == 8 ? go(k_z<OP, 8>)
                          : tpc == 4 ? go(k_z<OP, 4>)
                                     : go(k_z<OP, 2>);
  return err != cudaSuccess ? err : cudaGetLastError();
}

ZArgs z_args(const ZBatch& b, int n, int plane_size, const double* twiddle) {
  ZArgs z{};
  z.b = b;
  z.n = z.nin = z.nout = n;
  z.plane_size = plane_size;
  z.twiddle = twiddle;
  return z;
}

}  // namespace

int fft_timeout_flag() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_fft_timeout, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

const int* fft_timeout_address() {
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, g_fft_timeout) != cudaSuccess) return nullptr;
  return static_cast<const int*>(p);
}

bool z_batch_supported(int n) { return fft_plan(n).nf > 0 && z_smem(n, 2, 3) <= kZSmemLimit; }

cudaError_t z_forward(const ZBatch& b, int n, int nout, int plane_size, const double* twiddle, cudaStream_t st,
                      bool pdl) {
  ZArgs z = z_args(b, n, plane_size, twiddle);
  z.nout = nout;
  return z_launch<kZForward>(z, st, pdl);
}

cudaError_t z_inverse(const ZBatch& b, int nin, int n, int plane_size, const double* twiddle, cudaStream_t st,
                      bool pdl) {
  ZArgs z = z_args(b, n, plane_size, twiddle);
  z.nin = nin;
  return z_launch<kZInverse>(z, st, pdl);
}

cudaError_t z_inverse_dz(const ZBatch& b, int nin, int n, int plane_size, const double* twiddle, double beta,
                         cudaStream_t st, bool pdl) {
  ZArgs z = z_args(b, n, plane_size, twiddle);
  z.nin = nin;
  z.beta = beta;
  return z_launch<kZInverseDz>(z, st, pdl);
}

cudaError_t z_product_dz(const ZBatch& b, int n, int keep, int plane_size, const double* twiddle, double beta,
                         cudaStream_t st, bool pdl) {
  ZArgs z = z_args(b, n, plane_size, twiddle);
  z.keep = keep;
  z.beta = beta;
  return z_launch<kZProductDz>(z, st, pdl);
}

cudaError_t z_transform(double* data, int nz, int plane_size, int sign, const double* twiddle,
                        double* /*work*/, cudaStream_t st, bool pdl) {
  if (nz < 2) return cudaSuccess;
  if (nz == 2) {
    launch_ex(pdl, k_nz2, dim3((plane_size + 255) / 256), dim3(256), 0, st, data, plane_size, sign);
    return cudaGetLastError();
  }
  if (fft_plan(nz).nf > 0 && z_smem(nz, 2, 2) <= kZSmemLimit) {
    ZBatch b;
    b.add(data, data);
    return sign > 0 ? z_forward(b, nz, nz, plane_size, twiddle, st, pdl)
                    : z_inverse(b, nz, nz, plane_size, twiddle, st, pdl);
  }
  raise_smem_limit(reinterpret_cast<const void*>(k_dft), 200 * 1024);
  const size_t shm = sizeof(double) * (2 * static_cast<size_t>(nz) * kTP + 2 * nz);
  launch_ex(pdl, k_dft, dim3((plane_size + kTP - 1) / kTP), dim3(256), shm, st, data, nz, plane_size, sign, twiddle);
  return cudaGetLastError();
}

}  // namespace stx
