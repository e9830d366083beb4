// Two-level condensed solve of the skeleton system (all planes at once).
//
// After the element-level condensation has produced the skeleton right-hand
// side R (Element::local2globalSumSC, src/element.cpp:326-365), the reference
// solves the banded skeleton system with dpbtrs (src/field.cpp:693).  Here
// the same linear system is solved by block elimination over patches of
// elements: with I the skeleton unknowns interior to a patch and B those on
// patch interfaces,
//   y_I = S_II^-1 R_I                    (per patch)
//   r_B = R_B - S_BI y_I                 (per element: S is assembled from
//                                         the element Schur complements)
//   x_B = A^-1 r_B                       (A = S_BB - S_BI S_II^-1 S_IB)
//   x_I = y_I - G x_B                    (per patch, G = S_II^-1 S_IB)
// S_II^-1 and A^-1 are symmetric and stored packed, G in tiles
// (symtile.hpp); each product streams its tiles with bulk copies, the Re and
// Im planes of a mode sharing every tile read, a symmetric tile applied as
// itself and as its transpose.  Tiles are read as doubles, or as floats for
// the mixed-precision solve (the same layout; sums in FP64 either way).
#include "twolevel.cuh"

#include <algorithm>
#include <type_traits>

#include "element.cuh"
#include "launch.hpp"
#include "ptx.cuh"
#include "symtile.hpp"

namespace stx {

namespace {

// Warps per block of the packed products: DevModal::sym_warps (token
// STX_SYM_WARPS, 1..8, default 4: measured faster than 6 for one field).
constexpr int kSymWarpsMax = 8;
constexpr int kSymStages = 1;  // tile buffers per warp
constexpr int kTileDoubles = kSymTile * kSymLd;

// Shared memory per warp: barriers, tile ring, x entries of each buffered
// tile (32 of its column block, 32 of its row block, both planes).
struct SymWarpSmem {
  uint64_t bar[kSymStages];
  double2 x[kSymStages][2 * kSymTile];
  double tile[kSymStages][kTileDoubles];
};
constexpr size_t sym_smem(int warps) { return warps * sizeof(SymWarpSmem); }

// Position of a warp in the tiles of its problems.
struct SymCursor {
  int p, q, I, J, nt, tc;
  SymProblem P;
  __device__ void load(const SymProblem* probs, int prob, int tile) {
    p = prob;
    q = tile;
    P = probs[p];
    if (P.ncol) {
      tc = sym_tiles(P.ncol);
      nt = sym_tiles(P.n) * tc;
      I = q / tc;
      J = q - I * tc;
    } else {
      tc = 0;
      nt = sym_ntiles(P.n);
      sym_tile_at(q, I, J);
    }
  }
  __device__ bool row_last() const { return P.ncol ? J == tc - 1 : J == I; }
  __device__ long long offset() const {
    return P.ncol ? gen_tile_offset(P.n, P.ncol, I, J) : sym_tile_offset(P.n, I, J);
  }
  __device__ void next(const SymProblem* probs, bool more) {
    if (++q == nt) {
      if (more) load(probs, p + 1, 0);
    } else if (row_last()) {
      ++I;
      J = 0;
    } else {
      ++J;
    }
  }
};

// Column of a tile held in position q (0..3) by a lane of column group cq
// (0..7): two 16-byte pairs, 2 cq and 16 + 2 cq, so that the eight lanes
// reading one tile row cover it in one conflict-free 128-byte access each.
__host__ __device__ inline int col_of(int cq, int q) { return 16 * (q >> 1) + 2 * cq + (q & 1); }

// The lane's four entries of a tile row in shared memory (zero when the row
// is past the matrix).
__device__ __forceinline__ void tile_row4(const double* row, int cq, bool ok, double (&e)[4]) {
  if (ok) {
    const double2 u = *reinterpret_cast<const double2*>(row + 2 * cq);
    const double2 v = *reinterpret_cast<const double2*>(row + 16 + 2 * cq);
    e[0] = u.x;
    e[1] = u.y;
    e[2] = v.x;
    e[3] = v.y;
  } else {
    e[0] = e[1] = e[2] = e[3] = 0.0;
  }
}
__device__ __forceinline__ void tile_row4(const float* row, int cq, bool ok, double (&e)[4]) {
  if (ok) {
    const float2 u = *reinterpret_cast<const float2*>(row + 2 * cq);
    const float2 v = *reinterpret_cast<const float2*>(row + 16 + 2 * cq);
    e[0] = u.x;
    e[1] = u.y;
    e[2] = v.x;
    e[3] = v.y;
  } else {
    e[0] = e[1] = e[2] = e[3] = 0.0;
  }
}

// The last two halving exchanges (lane bits 1, 0) of a sum over the 8 lanes
// that share (lane >> 3): v[i] holds, after the first exchange (bit 2), the
// pair sums of row group i (lanes with bit 2 set: the upper row of the
// pair); lane l ends with the sum for position l & 7.
__device__ __forceinline__ double reduce_scatter4_low(const double (&w)[4], int ln) {
  double u[2];
  const bool h1 = ln & 2, h0 = ln & 1;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double send = h1 ? w[i] : w[2 + i], keep = h1 ? w[2 + i] : w[i];
    u[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
  }
  const double send = h0 ? u[0] : u[1], keep = h0 ? u[1] : u[0];
  return keep + __shfl_xor_sync(0xffffffffu, send, 1);
}

// Sum over the 4 lanes that share (lane & 7) of v[q], q = 0..3: lane l ends
// with the sum for q = l >> 3 (halving exchanges over lane bits 4, 3).
__device__ __forceinline__ double reduce_scatter4_high(const double (&v)[4], int ln) {
  double w[2];
  const bool h4 = ln & 16, h3 = ln & 8;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double send = h4 ? v[i] : v[2 + i], keep = h4 ? v[2 + i] : v[i];
    w[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
  const double send = h3 ? w[0] : w[1], keep = h3 ? w[1] : w[0];
  return keep + __shfl_xor_sync(0xffffffffu, send, 8);
}

// y[idx] += scale A x[idx] for every problem: each warp streams its run of tiles
// (SymWarp) through a ring of kSymStages buffers.  For a tile, lane 0
// bulk-copies the tile and every lane copies (cp.async) the x entries of the
// tile's column and row blocks, all completing on the buffer's mbarrier (count 1 + 32).
// Per tile (I, J) every lane reads its 8 x 4 entries of the tile once from
// shared memory (eight lanes cover a tile row with 16-byte reads) and forms
// both products from registers: the direct part y_I += A_IJ x_J as partial
// row sums over its four columns, summed over the eight lanes of a row by a
// halving exchange of warp shuffles (one row per lane, accumulated along the
// tile row and added at its end), and for J < I the transposed part
// y_J += A_IJ^T x_I as partial column sums over its eight rows, summed over
// the four lanes of a column the same way.  Waits are bounded; on expiry `status` is set and the
// warp stops.  Two builds (DevModal::sym_regcap chooses): CAP 0, blocks of
// up to 4 warps and the registers the code wants (no minimum block count:
// giving one lets the compiler take up to 255); CAP 1, blocks of up to 8
// warps and at most 80 registers (three such blocks per SM), a few spilled,
// more resident warps.
template <class T, int CAP>
__global__ void __launch_bounds__(CAP ? 32 * kSymWarpsMax : 128, CAP ? 2 : 4)
    k_psymv(const T* __restrict__ pack, const SymProblem* __restrict__ probs, const SymWarp* __restrict__ warps,
            int nwarps, const double* __restrict__ X, double* __restrict__ Y, int rstride, int nz, int* status, unsigned long long wait_ns) {
  extern __shared__ __align__(16) unsigned char sraw[];
  pdl_trigger();
  const int wp = threadIdx.x >> 5, ln = threadIdx.x & 31;
  const int gw = blockIdx.x * (blockDim.x >> 5) + wp;
  if (gw >= nwarps) {  // the warps of a block never synchronise with each other
    pdl_wait();
    return;
  }
  SymWarpSmem& sm = reinterpret_cast<SymWarpSmem*>(sraw)[wp];
  const SymWarp W = warps[gw];
  SymCursor ic, cc;  // issue and consume cursors
  ic.load(probs, W.prob, W.q);
  cc = ic;
  if (ln == 0) {
    for (int s = 0; s < kSymStages; ++s) mbar_init(&sm.bar[s], 1 + 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  int issued = 0;
  // positions in the plane vectors of the x entries of the next tile to
  // issue (column block, row block), loaded one issue ahead
  int pf[2];
  auto prefetch = [&]() {
    const int i = kSymTile * ic.J + ln;  // column block
    if (ic.P.ncol) {
      pf[0] = i < ic.P.ncol ? __ldg(ic.P.idx_col + i) : -1;
      pf[1] = -1;  // general products have no transposed part
    } else {
      pf[0] = (i < ic.P.n && i != ic.P.pin) ? __ldg(ic.P.idx + i) : -1;
      const int r = kSymTile * ic.I + ln;  // row block
      pf[1] = (r < ic.P.n && r != ic.P.pin) ? __ldg(ic.P.idx + r) : -1;
    }
  };
  prefetch();
  auto issue = [&](int s) {
    const int n = ic.P.n, m = ic.P.mode;
    const bool two = nz > 1 && m > 0;
    if (ln == 0) {
      const unsigned bytes = static_cast<unsigned>(sizeof(T) * kSymLd * sym_rows_stored(n, ic.I));
      mbar_expect_tx(&sm.bar[s], bytes);
      bulk_g2s(sm.tile[s], pack + ic.P.moff + ic.offset(), bytes, &sm.bar[s]);
    }
    // the matrix tiles are set-up data; the x entries (and the y atomics
    // after them) depend on the previous kernel
    if (issued == 0) pdl_wait();
    const double* X0 = X + static_cast<size_t>(2 * m) * rstride;
    const double* X1 = X0 + rstride;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int gi = pf[h];
      double2* d = &sm.x[s][kSymTile * h + ln];
      if (gi >= 0) {
        cp_async8(&d->x, X0 + gi);
        if (two) cp_async8(&d->y, X1 + gi);
        else d->y = 0.0;
      } else {
        *d = make_double2(0.0, 0.0);
      }
    }
    cp_async_arrive_noinc(&sm.bar[s]);
    ++issued;
    ic.next(probs, issued < W.count);
    if (issued < W.count) prefetch();
  };
  for (int s = 0; s < kSymStages && s < W.count; ++s) issue(s);
  if (W.count == 0) pdl_wait();
  // lane (rho, cq) = (lane >> 3, lane & 7): rows 4 t + rho (t = 0..7) and
  // columns col_of(cq, q) (q = 0..3) of every tile; it collects row
  // 4 cq + rho of the direct part and column col_of(cq, rho) of the
  // transposed part
  const int rho = ln >> 3, cq = ln & 7;
  double d0 = 0.0, d1 = 0.0;  // direct part of row 32 I + 4 cq + rho
  int done = 0;
  for (; done < W.count; ++done) {
    const int s = done % kSymStages;
    if (!__all_sync(0xffffffffu, mbar_wait(&sm.bar[s], (done / kSymStages) & 1, wait_ns))) {
      if (ln == 0 && status) atomicExch(status, 4);
      break;
    }
    const int n = cc.P.n, m = cc.P.mode, I = cc.I, J = cc.J;
    const bool two = nz > 1 && m > 0, sym = cc.P.ncol == 0, trans = sym && J < I;
    const double scale = cc.P.scale;
    const T* A = reinterpret_cast<const T*>(sm.tile[s]);
    const double2* xs = sm.x[s];
    const int h = sym_rows(n, I);
    // output positions (the column this lane collects for the transposed
    // part, the row it collects where the tile row ends), loaded before the
    // products to overlap their latency
    const bool row_end = cc.row_last() || done + 1 == W.count;
    const int rrow = 4 * cq + rho;
    const int g_col = trans ? __ldg(cc.P.idx + kSymTile * J + col_of(cq, rho)) : 0;  // J < I: a full block
    const int g_row = (row_end && rrow < h) ? __ldg(cc.P.idx + kSymTile * I + rrow) : 0;
    double* Y0 = Y + static_cast<size_t>(2 * m) * rstride;
    double* Y1 = Y0 + rstride;
    double2 xc[4];  // x of the lane's four columns (column block)
#pragma unroll
    for (int q = 0; q < 4; ++q) xc[q] = xs[col_of(cq, q)];
    double w0[4], w1[4], tp0[4] = {0.0, 0.0, 0.0, 0.0}, tp1[4] = {0.0, 0.0, 0.0, 0.0};
    const bool h2 = ln & 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      // rows 4 i + rho and 16 + 4 i + rho, their direct partial sums
      // combined at once over lane bit 2 (the first halving exchange)
      double dp[2][2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int r = 16 * k + 4 * i + rho;
        double e[4];
        tile_row4(A + r * kSymLd, cq, r < h, e);
        dp[k][0] = fma(e[0], xc[0].x, fma(e[1], xc[1].x, fma(e[2], xc[2].x, e[3] * xc[3].x)));
        dp[k][1] = fma(e[0], xc[0].y, fma(e[1], xc[1].y, fma(e[2], xc[2].y, e[3] * xc[3].y)));
        if (trans) {
          const double2 xr = xs[kSymTile + r];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            tp0[q] = fma(e[q], xr.x, tp0[q]);
            tp1[q] = fma(e[q], xr.y, tp1[q]);
          }
        }
      }
      w0[i] = (h2 ? dp[1][0] : dp[0][0]) + __shfl_xor_sync(0xffffffffu, h2 ? dp[0][0] : dp[1][0], 4);
      w1[i] = (h2 ? dp[1][1] : dp[0][1]) + __shfl_xor_sync(0xffffffffu, h2 ? dp[0][1] : dp[1][1], 4);
    }
    d0 += reduce_scatter4_low(w0, ln);
    d1 += reduce_scatter4_low(w1, ln);
    if (trans) {
      const double s0 = reduce_scatter4_high(tp0, ln), s1 = reduce_scatter4_high(tp1, ln);
      atomicAdd(&Y0[g_col], scale * s0);
      if (two) atomicAdd(&Y1[g_col], scale * s1);
    }
    if (row_end) {
      if (rrow < h) {
        atomicAdd(&Y0[g_row], scale * d0);
        if (two) atomicAdd(&Y1[g_row], scale * d1);
      }
      d0 = d1 = 0.0;
    }
    __syncwarp();
    if (issued < W.count) issue(s);  // the buffer's reads are complete (syncwarp)
    cc.next(probs, done + 1 < W.count);
  }
  // leave no copy in flight (only after an expired wait; default bound)
  for (int k = done; k < issued; ++k) mbar_wait(&sm.bar[k % kSymStages], (k / kSymStages) & 1);
}

// The same products for NF (2, 3) fields at once on the FP64 tensor cores: the
// planes of the fields are the columns of m8n8k4 products (2 NF of 8), so that
// a tile costs its fragment reads and 64 products where k_psymv spends 128 NF
// multiply-adds a lane, the x entries and the sums' exchanges (at three fields
// four fifths of the shared-memory pipe: 24 x 24 x 96, three fields, the
// interface product of half the modes, 226 MB, 103 us; 73 here).  Tile rows are copied kMmaLd entries
// apart and the x entries kept [column][entry], so that fragments of the tile,
// of its transpose and of x are read without bank conflicts.
constexpr int kMmaLd = 36;
constexpr int kMmaX = 2 * kSymTile + 4;
struct MmaWarpSmem {
  uint64_t bar[2];  // [0] used; 16-byte alignment of what follows
  double tile[kSymTile * kMmaLd];
  double x[8 * kMmaX];  // [2 f + plane][column block | row block]
};
constexpr size_t mma_smem(int warps) { return warps * sizeof(MmaWarpSmem); }

template <int NF>
__global__ void __launch_bounds__(32 * kSymWarpsMax, 2)
    k_psymv_mma(const double* __restrict__ pack, const SymProblem* __restrict__ probs,
                const SymWarp* __restrict__ warps, int nwarps, const double* __restrict__ X, double* __restrict__ Y,
                int rstride, size_t fstride, int nz, int* status, unsigned long long wait_ns) {
  extern __shared__ __align__(16) unsigned char sraw[];
  pdl_trigger();
  const int wp = threadIdx.x >> 5, ln = threadIdx.x & 31, g8 = ln >> 2, t4 = ln & 3;
  const int gw = blockIdx.x * (blockDim.x >> 5) + wp;
  if (gw >= nwarps) {  // the warps of a block never synchronise with each other
    pdl_wait();
    return;
  }
  MmaWarpSmem& sm = reinterpret_cast<MmaWarpSmem*>(sraw)[wp];
  const SymWarp W = warps[gw];
  // rows past a last tile and columns past the fields stay finite
  for (int i = ln; i < kSymTile * kMmaLd; i += 32) sm.tile[i] = 0.0;
  for (int i = ln; i < 8 * kMmaX; i += 32) sm.x[i] = 0.0;
  if (ln == 0) {
    mbar_init(&sm.bar[0], 1 + 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  SymCursor ic, cc;  // issue and consume cursors
  ic.load(probs, W.prob, W.q);
  cc = ic;
  int issued = 0, pf[2];
  auto prefetch = [&]() {
    const int i = kSymTile * ic.J + ln;  // column block
    if (ic.P.ncol) {
      pf[0] = i < ic.P.ncol ? __ldg(ic.P.idx_col + i) : -1;
      pf[1] = -1;  // general products have no transposed part
    } else {
      pf[0] = (i < ic.P.n && i != ic.P.pin) ? __ldg(ic.P.idx + i) : -1;
      const int r = kSymTile * ic.I + ln;  // row block
      pf[1] = (r < ic.P.n && r != ic.P.pin) ? __ldg(ic.P.idx + r) : -1;
    }
  };
  auto issue = [&]() {
    const int rows = sym_rows_stored(ic.P.n, ic.I);
    const bool two = nz > 1 && ic.P.mode > 0;
    if (ln == 0) mbar_expect_tx(&sm.bar[0], static_cast<unsigned>(sizeof(double)) * kSymLd * rows);
    if (ln < rows)
      bulk_g2s(sm.tile + ln * kMmaLd, pack + ic.P.moff + ic.offset() + ln * kSymLd,
               static_cast<unsigned>(sizeof(double)) * kSymLd, &sm.bar[0]);
    // the matrix tiles are set-up data; the x entries (and the y atomics
    // after them) depend on the previous kernel
    if (issued == 0) pdl_wait();
    const double* X0 = X + static_cast<size_t>(2 * ic.P.mode) * rstride;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      double* d = sm.x + kSymTile * h + ln;
#pragma unroll
      for (int f = 0; f < NF; ++f)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          if (pf[h] >= 0 && (r == 0 || two)) cp_async8(d + (2 * f + r) * kMmaX, X0 + f * fstride + (r ? rstride : 0) + pf[h]);
          else d[(2 * f + r) * kMmaX] = 0.0;
        }
    }
    cp_async_arrive_noinc(&sm.bar[0]);
    ++issued;
    ic.next(probs, issued < W.count);
    if (issued < W.count) prefetch();
  };
  if (W.count == 0) {
    pdl_wait();
    return;
  }
  prefetch();
  issue();
  double acc[4][2];  // rows 8 i + g8 of the tile row, planes of field t4
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0.0;
  for (int done = 0; done < W.count; ++done) {
    if (!__all_sync(0xffffffffu, mbar_wait(&sm.bar[0], done & 1, wait_ns))) {
      if (ln == 0 && status) atomicExch(status, 4);
      mbar_wait(&sm.bar[0], done & 1);  // leave no copy in flight (default bound)
      break;
    }
    __syncwarp();
    const int I = cc.I, J = cc.J, h = sym_rows(cc.P.n, I);
    const bool trans = cc.P.ncol == 0 && J < I, two = nz > 1 && cc.P.mode > 0;
    const bool row_end = cc.row_last() || done + 1 == W.count;
    const double scale = cc.P.scale;
    double* Yf = Y + t4 * fstride + static_cast<size_t>(2 * cc.P.mode) * rstride;
    int gi[4], gj[4];  // output positions, loaded before the products to overlap their latency
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      gi[i] = row_end && t4 < NF && 8 * i + g8 < h ? __ldg(cc.P.idx + kSymTile * I + 8 * i + g8) : -1;
      gj[i] = trans && t4 < NF ? __ldg(cc.P.idx + kSymTile * J + 8 * i + g8) : -1;  // J < I: a full block
    }
    const double* xb = sm.x + g8 * kMmaX + t4;
#pragma unroll
    for (int k = 0; k < kSymTile / 4; ++k) {
      const double b = xb[4 * k];
#pragma unroll
      for (int i = 0; i < 4; ++i) dmma_8x8x4(acc[i][0], acc[i][1], sm.tile[(8 * i + g8) * kMmaLd + 4 * k + t4], b);
    }
    if (trans) {
      double tr[4][2];
#pragma unroll
      for (int j = 0; j < 4; ++j) tr[j][0] = tr[j][1] = 0.0;
#pragma unroll
      for (int k = 0; k < kSymTile / 4; ++k) {
        const double b = xb[kSymTile + 4 * k];
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma_8x8x4(tr[j][0], tr[j][1], sm.tile[(4 * k + t4) * kMmaLd + 8 * j + g8], b);
      }
      __syncwarp();  // the buffer's reads are complete
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      if (issued < W.count) issue();
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (gj[j] >= 0) {
          atomicAdd(Yf + gj[j], scale * tr[j][0]);
          if (two) atomicAdd(Yf + rstride + gj[j], scale * tr[j][1]);
        }
    } else {
      __syncwarp();
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      if (issued < W.count) issue();
    }
    if (row_end) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (gi[i] >= 0) {
          atomicAdd(Yf + gi[i], scale * acc[i][0]);
          if (two) atomicAdd(Yf + rstride + gi[i], scale * acc[i][1]);
        }
        acc[i][0] = acc[i][1] = 0.0;
      }
    }
    cc.next(probs, done + 1 < W.count);
  }
}

template <int CAP>
void configure_psymv_as() {
  raise_smem_limit(reinterpret_cast<const void*>(k_psymv<double, CAP>), sym_smem(kSymWarpsMax));
  raise_smem_limit(reinterpret_cast<const void*>(k_psymv<float, CAP>), sym_smem(kSymWarpsMax));
}

void configure_psymv() {
  configure_psymv_as<0>();
  configure_psymv_as<1>();
  raise_smem_limit(reinterpret_cast<const void*>(k_psymv_mma<2>), mma_smem(kSymWarpsMax));
  raise_smem_limit(reinterpret_cast<const void*>(k_psymv_mma<3>), mma_smem(kSymWarpsMax));
}

template <class T>
void launch_psymv_as(const DevModal& S, const T* pack, const SymProblem* probs, const SymWarp* warps, int nwarps,
                     const double* X, double* Y, int rstride, int nz, cudaStream_t st) {
  const int wpb = S.sym_warps;
  const dim3 blocks((nwarps + wpb - 1) / wpb), threads(32 * wpb);
  if (S.sym_regcap)
    launch_ex(S.pdl != 0, k_psymv<T, 1>, blocks, threads, sym_smem(wpb), st, pack, probs, warps, nwarps, X, Y,
              rstride, nz, S.status, S.wait_ns);
  else
    launch_ex(S.pdl != 0, k_psymv<T, 0>, blocks, threads, sym_smem(wpb), st, pack, probs, warps, nwarps, X, Y,
              rstride, nz, S.status, S.wait_ns);
}

cudaError_t launch_psymv(const DevModal& S, const SymProblem* probs, const SymWarp* warps, int nwarps,
                         const double* X, double* Y, int rstride, int nz, bool fp32, cudaStream_t st, int nf = 1,
                         size_t fstride = 0) {
  if (nwarps <= 0) return cudaSuccess;
  configure_psymv();
  const int wpb = S.sym_warps;
  const dim3 blocks((nwarps + wpb - 1) / wpb), threads(32 * wpb);
  if (fp32)
    launch_psymv_as<float>(S, S.l2_pack32, probs, warps, nwarps, X, Y, rstride, nz, st);
  else if (nf == 3)
    launch_ex(S.pdl != 0, k_psymv_mma<3>, blocks, threads, mma_smem(wpb), st, S.l2_pack, probs, warps, nwarps, X, Y,
              rstride, fstride, nz, S.status, S.wait_ns);
  else if (nf == 2)
    launch_ex(S.pdl != 0, k_psymv_mma<2>, blocks, threads, mma_smem(wpb), st, S.l2_pack, probs, warps, nwarps, X, Y,
              rstride, fstride, nz, S.status, S.wait_ns);
  else
    launch_psymv_as<double>(S, S.l2_pack, probs, warps, nwarps, X, Y, rstride, nz, st);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Patch products batched over the patches of a family: Y_I = S_II^-1 X_I or
// Y_I -= G X_B for every (patch, field, plane) of a family's patches in one
// mode as the columns of a matrix product on the FP64 tensor cores (m8n8k4).
// A block owns 64 rows and 8 NT columns over the whole inner dimension, so
// its results are stored, not summed: per inner tile of 32 the block's two
// matrix tiles (one 256-byte bulk copy a row, rows kGemmLd doubles apart in
// shared memory so that a fragment of the tile or of its transpose is read
// without bank conflicts) and the gathered columns (8-byte asynchronous
// copies) land in one of kGemmStages buffers while the tensor cores work on
// the others.  The upper triangle of the packed S_II^-1 is read as the
// transposed lower one.
//
// Bound: the FP64 tensor cores (16 cycles a m8n8k4 product and scheduler).
// Three stages and two measured alike.
// ---------------------------------------------------------------------------
constexpr int kGemmLd = 36;
constexpr int kGemmStages = 3;
constexpr int kGemmRows = 64;
constexpr int kGemmWarps = kGemmRows / 8;
constexpr int kGemmMaxNt = 6;

__host__ __device__ constexpr size_t gemm_stage_doubles(int nt) { return (kGemmRows + 8 * static_cast<size_t>(nt)) * kGemmLd; }
constexpr size_t gemm_smem(int nt) { return 64 + sizeof(double) * kGemmStages * gemm_stage_doubles(nt); }

template <int NT>
__global__ void __launch_bounds__(32 * kGemmWarps, 2)
    k_patch_gemm(DevModal S, int general, const double* X, double* Y, int rstride, size_t fstride, int nf,
                 int nz) {
  extern __shared__ __align__(16) unsigned char sraw[];
  pdl_trigger();
  const PatchGroup G = S.pgroups[blockIdx.y];
  const int n = G.n, K = general ? G.nb : n, TK = sym_tiles(K), T = sym_tiles(n);
  const int nr = nz > 1 && G.mode > 0 ? 2 : 1, per = nf * nr, ncol = G.npatch * per;
  const int I0 = 2 * blockIdx.x, c0 = 8 * NT * blockIdx.z;
  if (I0 >= T || c0 >= ncol || K <= 0) {  // the whole block
    pdl_wait();
    return;
  }
  uint64_t* full = reinterpret_cast<uint64_t*>(sraw);
  double* ring = reinterpret_cast<double*>(sraw + 64);
  constexpr size_t kStage = gemm_stage_doubles(NT);
  const int wp = threadIdx.x >> 5, ln = threadIdx.x & 31, g8 = ln >> 2, t4 = ln & 3;
  // rows past the matrix and columns past the group stay finite
  for (int i = threadIdx.x; i < static_cast<int>(kStage * kGemmStages); i += 32 * kGemmWarps) ring[i] = 0.0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kGemmStages; ++s) mbar_init(&full[s], 1 + 32 * kGemmWarps);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  const double* A = S.l2_pack + (general ? G.g_off : G.s_off);
  // tile of block row I (0, 1) and inner tile J: its rows in storage
  auto tile_rows = [&](int I, int J) {
    if (I >= T) return 0;
    return sym_rows_stored(n, general || J <= I ? I : J);
  };
  auto issue_matrix = [&](int J) {
    double* a = ring + (J % kGemmStages) * kStage;
    uint64_t* bar = &full[J % kGemmStages];
    if (threadIdx.x == 0)
      mbar_expect_tx(bar, 256u * static_cast<unsigned>(tile_rows(I0, J) + tile_rows(I0 + 1, J)));
    if (threadIdx.x < kGemmRows) {
      const int I = I0 + (threadIdx.x >> 5), r = threadIdx.x & 31;
      if (r < tile_rows(I, J)) {
        const long long o = general  ? gen_tile_offset(n, K, I, J)
                            : J <= I ? sym_tile_offset(n, I, J)
                                     : sym_tile_offset(n, J, I);
        bulk_g2s(a + threadIdx.x * kGemmLd, A + o + r * kSymLd, 256u, bar);
      }
    }
  };
  // the warp gathers columns c0 + NT wp + u
  const double* xp[NT];
  const int* xi[NT];
  const int imax = general ? S.nB_max : S.nI_max;
  const int* ids = general ? S.p_Bgid : S.p_Igid;
#pragma unroll
  for (int u = 0; u < NT; ++u) {
    const int c = c0 + NT * wp + u;
    xi[u] = nullptr;
    xp[u] = X;
    if (c < ncol) {
      const int p = c / per, f = (c - p * per) / nr, r = c - p * per - f * nr;
      xi[u] = ids + static_cast<size_t>(__ldg(S.group_patch + G.patch0 + p)) * imax;
      xp[u] = X + f * fstride + static_cast<size_t>(2 * G.mode + r) * rstride;
    }
  }
  int id[NT];  // positions of the next gather, loaded one tile ahead
  auto prefetch = [&](int J) {
    const int k = kSymTile * J + ln;
#pragma unroll
    for (int u = 0; u < NT; ++u) id[u] = xi[u] && k < K ? __ldg(xi[u] + k) : -1;
  };
  auto issue_columns = [&](int J) {
    double* x = ring + (J % kGemmStages) * kStage + kGemmRows * kGemmLd;
#pragma unroll
    for (int u = 0; u < NT; ++u) {
      double* d = x + (NT * wp + u) * kGemmLd + ln;
      if (id[u] >= 0) cp_async8(d, xp[u] + id[u]);
      else *d = 0.0;
    }
    cp_async_arrive_noinc(&full[J % kGemmStages]);
    if (J + 1 < TK) prefetch(J + 1);
  };
  const int lead = min(kGemmStages, TK);
  prefetch(0);
  for (int J = 0; J < lead; ++J) issue_matrix(J);
  pdl_wait();  // the matrices and indices are set-up data, the vectors are not
  for (int J = 0; J < lead; ++J) issue_columns(J);
  double acc[NT][2];
#pragma unroll
  for (int u = 0; u < NT; ++u) acc[u][0] = acc[u][1] = 0.0;
  const int I = I0 + (wp >> 2), i8 = 8 * (wp & 3);
  for (int J = 0; J < TK; ++J) {
    // tile J has landed, and every warp is done with tile J - 1
    if (!__syncthreads_and(mbar_wait(&full[J % kGemmStages], (J / kGemmStages) & 1, S.wait_ns))) {
      if (threadIdx.x == 0 && S.status) atomicExch(S.status, 4);
      // leave no copy in flight
      const int issued = J == 0 ? lead : min(TK, J - 1 + kGemmStages);
      for (int t = J; t < issued; ++t) mbar_wait(&full[t % kGemmStages], (t / kGemmStages) & 1);
      return;
    }
    if (J > 0 && J - 1 + kGemmStages < TK) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      issue_matrix(J - 1 + kGemmStages);
      issue_columns(J - 1 + kGemmStages);
    }
    const double* a = ring + (J % kGemmStages) * kStage;
    const double* x = a + kGemmRows * kGemmLd + g8 * kGemmLd + t4;
    a += (wp >> 2) * kSymTile * kGemmLd;
    const bool direct = general || J <= I;
    const double* ap = direct ? a + (i8 + g8) * kGemmLd + t4 : a + t4 * kGemmLd + i8 + g8;
    const int step = direct ? 4 : 4 * kGemmLd;
#pragma unroll
    for (int k = 0; k < kSymTile / 4; ++k) {
      const double av = ap[k * step];
#pragma unroll
      for (int u = 0; u < NT; ++u) dmma_8x8x4(acc[u][0], acc[u][1], av, x[8 * u * kGemmLd + 4 * k]);
    }
  }
  // every position and old value before the first store (y may alias what is
  // still to be read, as far as the compiler knows)
  const int row = kSymTile * I + i8 + g8;
  if (row >= n) return;
  double* y[NT][2];
#pragma unroll
  for (int u = 0; u < NT; ++u)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int c = c0 + 8 * u + 2 * t4 + q;
      y[u][q] = nullptr;
      if (c < ncol) {
        const int p = c / per, f = (c - p * per) / nr, r = c - p * per - f * nr;
        const int gi = __ldg(S.p_Igid + static_cast<size_t>(__ldg(S.group_patch + G.patch0 + p)) * S.nI_max + row);
        y[u][q] = Y + f * fstride + static_cast<size_t>(2 * G.mode + r) * rstride + gi;
      }
    }
  if (general) {
#pragma unroll
    for (int u = 0; u < NT; ++u)
#pragma unroll
      for (int q = 0; q < 2; ++q) acc[u][q] = (y[u][q] ? *y[u][q] : 0.0) - acc[u][q];
  }
#pragma unroll
  for (int u = 0; u < NT; ++u)
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (y[u][q]) *y[u][q] = acc[u][q];
}

struct GemmShape {
  int nt;
  dim3 grid;
};
GemmShape gemm_shape(const DevModal& S, int nf, int nz) {
  const int cols = S.pg_npatch * nf * (nz > 1 ? 2 : 1);
  const int blocks = (cols + 8 * kGemmMaxNt - 1) / (8 * kGemmMaxNt);  // column blocks, evenly filled
  return {(cols + 8 * blocks - 1) / (8 * blocks), dim3((sym_tiles(S.nI_max) + 1) / 2, S.npgroup, blocks)};
}

// Whether the patch products of nf fields go through k_patch_gemm rather than
// k_psymv, which reads a matrix once a patch and plane pair (token
// STX_PATCH_GEMM: 0 never, 1 always).  It pays where a family's matrices have
// eight columns or more on average, and its blocks of 64 rows are enough to
// fill the SMs.  us a DNS step with / without (B200): 24 x 24 x 96, N_P = 9
// (16 patches of one family: 96 and 32 columns, 336 blocks a mode group) 1508
// / 1739; 16 x 16 x 64 (8 patches: 48 and 16 columns, 112 blocks) 536 / 573;
// channel 16 x 8 x 32 (4 patches a family: 24 columns, 48 blocks) 281 / 272;
// always: the 16 x 16 x 64, N_P = 11 Dirichlet solve (1 to 4 patches a family,
// 2 to 8 columns) 157 / 131.
bool patch_gemm_pays(const DevModal& S, int nf, int nz) {
  if (!S.pgroups || S.pfam <= 0 || S.patch_gemm == 0) return false;
  const dim3 g = gemm_shape(S, nf, nz).grid;
  if (g.y > 65535) return false;  // families x modes past the grid's limit
  if (S.patch_gemm == 1) return true;
  return S.npatch * nf * (nz > 1 ? 2 : 1) >= 8 * S.pfam && g.x * g.y * g.z >= 96;
}

cudaError_t launch_patch_gemm(const DevModal& S, bool general, const double* X, double* Y, int rstride,
                              size_t fstride, int nf, int nz, cudaStream_t st) {
  const GemmShape h = gemm_shape(S, nf, nz);
  auto go = [&](auto nt_) {
    constexpr int NT = decltype(nt_)::value;
    raise_smem_limit(reinterpret_cast<const void*>(k_patch_gemm<NT>), gemm_smem(NT));
    return launch_ex(S.pdl != 0, k_patch_gemm<NT>, h.grid, dim3(32 * kGemmWarps), gemm_smem(NT), st, S,
                     general ? 1 : 0, X, Y, rstride, fstride, nf, nz);
  };
  switch (h.nt) {
    case 1: return go(std::integral_constant<int, 1>{});
    case 2: return go(std::integral_constant<int, 2>{});
    case 3: return go(std::integral_constant<int, 3>{});
    case 4: return go(std::integral_constant<int, 4>{});
    case 5: return go(std::integral_constant<int, 5>{});
    default: return go(std::integral_constant<int, 6>{});
  }
}

// y_I = S_II^-1 x_I into zeroed y, or (general) y_I -= G x_B.
cudaError_t patch_product(const DevModal& S, bool general, const double* X, double* Y, int rstride, int nz,
                          bool fp32, cudaStream_t st, int nf = 1, size_t fstride = 0) {
  if (!fp32 && patch_gemm_pays(S, nf, nz))
    return launch_patch_gemm(S, general, X, Y, rstride, fstride, nf, nz, st);
  return general ? launch_psymv(S, S.prob_gen, S.warp_gen, S.nwarp_gen, X, Y, rstride, nz, fp32, st, nf, fstride)
                 : launch_psymv(S, S.prob_patch, S.warp_patch, S.nwarp_patch, X, Y, rstride, nz, fp32, st, nf,
                                fstride);
}

}  // namespace

namespace {

__global__ void k_zero_ranges(ZeroRanges z, size_t total) {
  pdl_trigger();
  pdl_wait();
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    size_t j = i;
    int r = 0;
    while (r + 1 < z.count && j >= z.n[r]) j -= z.n[r++];
    z.p[r][j] = 0.0;
  }
}

}  // namespace

cudaError_t zero_ranges(bool pdl, const ZeroRanges& z, cudaStream_t st) {
  size_t n = 0;
  for (int r = 0; r < z.count; ++r) n += z.n[r];
  if (n == 0) return cudaSuccess;
  const unsigned blocks = static_cast<unsigned>(std::min<size_t>((n + 255) / 256, 148 * 8));
  return launch_ex(pdl, k_zero_ranges, dim3(blocks), dim3(256), 0, st, z, n);
}

cudaError_t zero_ranges(bool pdl, double* a, size_t na, double* b, size_t nb, cudaStream_t st) {
  ZeroRanges z;
  z.add(a, na);
  z.add(b, nb);
  return zero_ranges(pdl, z, st);
}

size_t twolevel_workspace_doubles(int rstride, int nz) { return static_cast<size_t>(rstride) * nz; }

cudaError_t twolevel_solve(const DevModal& S, const DevGeom& g, double* R, int rstride, double* work, int nz,
                           cudaStream_t st, cudaEvent_t mid, bool fp32, bool y_zeroed) {
  double* Yv = twolevel_solution(work, rstride, nz);  // y_I, then the whole skeleton solution
  // planes of the launch's modes
  const int k0 = nz > 1 ? 2 * S.mode0 : 0, k1 = nz > 1 ? std::min(nz, 2 * (S.mode0 + S.nmodes)) : 1;
  cudaError_t err = y_zeroed ? cudaSuccess
                             : zero_ranges(S.pdl != 0, Yv + static_cast<size_t>(rstride) * k0,
                                           static_cast<size_t>(rstride) * (k1 - k0), nullptr, 0, st);
  if (err != cudaSuccess) return err;
  // y_I = S_II^-1 R_I; r_B = R_B - S_BI y_I
  err = patch_product(S, false, R, Yv, rstride, nz, fp32, st);
  if (err != cudaSuccess) return err;
  if (S.niface > 0) element_schur_apply(0, g, S, Yv, R, rstride, 1, 0, st);
  // x_B = A^-1 r_B (into the interface positions of Y)
  err = launch_psymv(S, S.prob_iface, S.warp_iface, S.nwarp_iface, R, Yv, rstride, nz, fp32, st);
  if (err != cudaSuccess) return err;
  if (mid) cudaEventRecord(mid, st);
  // x_I = y_I - G x_B, G = S_II^-1 S_IB
  err = patch_product(S, true, Yv, Yv, rstride, nz, fp32, st);
  if (err != cudaSuccess) return err;
  return cudaGetLastError();
}

cudaError_t twolevel_solve_fields(const DevModal& S, const DevGeom& g, double* R, double* Y, size_t fstride, int nf,
                                  int rstride, int nz, cudaStream_t st, bool y_zeroed) {
  if (nf < 1 || nf > 3 || S.refine > 0 || S.l2_pack32) return cudaErrorInvalidValue;
  const int k0 = nz > 1 ? 2 * S.mode0 : 0, k1 = nz > 1 ? std::min(nz, 2 * (S.mode0 + S.nmodes)) : 1;
  cudaError_t err = cudaSuccess;
  if (!y_zeroed) {
    ZeroRanges z;
    for (int f = 0; f < nf; ++f)
      z.add(Y + f * fstride + static_cast<size_t>(rstride) * k0, static_cast<size_t>(rstride) * (k1 - k0));
    err = zero_ranges(S.pdl != 0, z, st);
  }
  if (err != cudaSuccess) return err;
  err = patch_product(S, false, R, Y, rstride, nz, false, st, nf, fstride);
  if (err != cudaSuccess) return err;
  if (S.niface > 0) element_schur_apply(0, g, S, Y, R, rstride, nf, fstride, st);
  err = launch_psymv(S, S.prob_iface, S.warp_iface, S.nwarp_iface, R, Y, rstride, nz, false, st, nf, fstride);
  if (err != cudaSuccess) return err;
  err = patch_product(S, true, Y, Y, rstride, nz, false, st, nf, fstride);
  if (err != cudaSuccess) return err;
  return cudaGetLastError();
}

int twolevel_launches(const DevModal& S) {
  return (S.nwarp_patch > 0 ? 1 : 0) + (S.nwarp_iface > 0 ? 1 : 0) + (S.nwarp_gen > 0 ? 1 : 0) + (S.niface > 0 ? 1 : 0);
}

static int prob_ntiles(const SymProblem& P) { return P.ncol ? gen_ntiles(P.n, P.ncol) : sym_ntiles(P.n); }

std::vector<SymWarp> sym_schedule(const std::vector<SymProblem>& probs, int device, int wpb, int occ_pct,
                                  int regcap) {
  std::vector<SymWarp> out;
  long long total = 0;
  for (const auto& P : probs) total += prob_ntiles(P);
  if (total == 0) return out;
  int sms = 148, per_sm = 1;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  configure_psymv();
  const void* kern = regcap ? reinterpret_cast<const void*>(k_psymv<double, 1>)
                            : reinterpret_cast<const void*>(k_psymv<double, 0>);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * wpb, sym_smem(wpb)) != cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  // warps of one full wave at the kernel's occupancy, times occ_pct / 100
  const long long wave = static_cast<long long>(sms) * per_sm * wpb;
  // a warp's fixed cost (its barrier, its first wait) is paid by two tiles or
  // more (16 uneven 2D problems in one graph 151 -> 134 us)
  const long long nw = std::max<long long>(1, std::min<long long>((total + 1) / 2, wave * occ_pct / 100));
  size_t p = 0;
  long long before = 0;  // tiles of problems [0, p)
  for (long long w = 0; w < nw; ++w) {
    const long long t0 = total * w / nw, t1 = total * (w + 1) / nw;
    while (before + prob_ntiles(probs[p]) <= t0) before += prob_ntiles(probs[p++]);
    out.push_back(SymWarp{static_cast<int>(p), static_cast<int>(t0 - before), static_cast<int>(t1 - t0)});
  }
  return out;
}

}  // namespace stx
