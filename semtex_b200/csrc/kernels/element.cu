// Element kernels: a block takes up to 16 same-family elements (a part of a
// chunk), the Re and Im planes of one Fourier mode and a block of rows of the
// family's operator, and applies the operator to the elements' columns on the
// FP64 tensor cores (m8n8k4), for one or several fields in turn.  Columns and
// operators are in natural node order, so a column is read from the forcing
// as it lies (boundary rows of the recovery from the skeleton solution),
// scaled by -Q4 on the way into shared memory; the condensation's operator
// (I | -hbi hii^-1) leaves the sums to add to the skeleton right-hand side, the
// recovery's (-(hbi hii^-1)^T | hii^-1) the interior values, both taken to
// global memory from the accumulators.  The operator rows are bulk-copied
// alongside.  Essential values g enter the recovery as boundary rows of its
// columns, and the condensation as -S_e g, S_e the element's Schur complement:
// what the operators make of the lift term H g, without forming it.  (Forming
// it in two warps of a block took 126 us to 376 us a solve for 16 x 16 x 64,
// N_P = 11 with values on the walls, and was the less accurate; now 119 and
// 150.)
//
// Bound: the FP64 tensor cores and the latency of one round of loads a block,
// so the rest is kept out of the way: a warp reads an element with constant
// offsets (no index arithmetic a node), enough blocks share an SM to hide the
// loads, nothing is staged on the way out.  us a launch (B200; all fields of a
// solve, half the modes): recovery of 24 x 24 x 96, N_P = 9, three fields 58
// (73 with 64 staged columns a block, index tables and write-out passes),
// condensation 37 (45); 16 x 16 x 64, N_P = 11, one field 24.7 and 14.4 (25
// and 23).  The same kernels at 128 registers with the next field's loads
// under a field's product: 70 and 51; eight warps a block throughout, two row
// blocks at N_P = 11: 36 and 18.
#include "element.cuh"

#include <algorithm>

#include "launch.hpp"
#include "ptx.cuh"

namespace stx {

namespace {

constexpr int kColBatch = 4;    // columns per warp whose index loads are in flight together (Schur couplings)
constexpr int kSchurParts = 2;  // blocks per chunk and mode of the Schur couplings (latency-bound)
constexpr int kUnitTiles = 4;   // 8x8 tiles per warp unit of the Schur products: 8 rows x 32 columns
constexpr int kElemThreads = 512;  // most threads of a block
constexpr int kElemCols = 32;   // most columns of a block: elements x planes
constexpr int kElemRounds = 3;  // nodes per lane and plane whose loads are in flight together

__device__ __forceinline__ void col_slot(int col, int cnt, int& slot, int& l) {
  slot = col >= cnt ? 1 : 0;  // at most two planes (Re, Im) per mode
  l = col - slot * cnt;
}

struct ElemSmem {
  size_t a, b, out, el, tab, bytes;
};

// [mbarrier | operator rows | columns | output offsets | the part's elements |
//  their btog (condensation) or the interior nodes (recovery)]
__host__ __device__ inline ElemSmem elem_layout(int rows, int cols, int ld, int tab) {
  ElemSmem L;
  L.a = 16;
  L.b = L.a + sizeof(double) * static_cast<size_t>(rows) * ld;
  L.out = L.b + sizeof(double) * static_cast<size_t>(cols) * ld;
  L.el = L.out + sizeof(size_t) * kElemCols;
  L.tab = L.el + sizeof(int) * kElemCols;
  L.bytes = (L.tab + sizeof(int) * static_cast<size_t>(tab) + 15) / 16 * 16;
  return L;
}

// Entries of the table: the recovery's interior nodes, or the elements' rows.
__host__ __device__ inline int elem_tab(bool recover, int rows, int pe) { return recover ? rows : pe * rows; }

// Thread 0: initialise the mbarrier and start the bulk copy of the operator
// rows (bytes a multiple of 16, 16-byte aligned source).
__device__ __forceinline__ void stage_rows(uint64_t* bar, double* sA, const double* src, unsigned bytes) {
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(bar, bytes);
    const char* s = reinterpret_cast<const char*>(src);
    char* d = reinterpret_cast<char*>(sA);
    for (unsigned off = 0; off < bytes; off += 32768u) bulk_g2s(d + off, s + off, min(32768u, bytes - off), bar);
  }
}

// All threads: wait, bounded by `limit_ns`, for the operator rows; false
// (uniformly) when the bound expired, after the error is recorded and a
// second wait (bounded by the default 2 s) for the copy still in flight.
__device__ __forceinline__ bool rows_ready(uint64_t* bar, int* status, unsigned long long limit_ns) {
  const bool ok = __syncthreads_and(mbar_wait(bar, 0, limit_ns));
  if (!ok) {
    if (threadIdx.x == 0 && status) atomicExch(status, 3);
    mbar_wait(bar, 0);
  }
  return ok;
}

// R -= S_e g of one element and nr planes, S_e its Schur complement (one row of
// it a node with an essential value, lanes over the rows of the result: S_e is
// symmetric), g the essential values among its boundary nodes bt.  One warp.
// Out of line: most elements have none, and its registers are not the loads'.
__device__ __noinline__ void lift_element(const double* __restrict__ Se, int ld, const int* __restrict__ bt, int next,
                                          int ness, const double* g0, double* r0, int rstride, int nr) {
  const int ln = threadIdx.x & 31;
  for (int r = 0; r < nr; ++r, g0 += rstride, r0 += rstride)
    for (int b0 = 0; b0 < next; b0 += 64) {
      double acc[2] = {0.0, 0.0};
      for (int a0 = 0; a0 < next; a0 += 32) {
        const int gi = a0 + ln < next ? __ldg(bt + a0 + ln) : -1;
        const double g = gi >= ness ? g0[gi] : 0.0;
        if (!__any_sync(0xffffffffu, g != 0.0)) continue;
        const int na = min(32, next - a0);
#pragma unroll 8
        for (int a = 0; a < na; ++a) {
          const double v = __shfl_sync(0xffffffffu, g, a);
          const double* row = Se + static_cast<size_t>(a0 + a) * ld + b0 + ln;
#pragma unroll
          for (int q = 0; q < 2; ++q)
            if (b0 + 32 * q + ln < next) acc[q] = fma(__ldg(row + 32 * q), v, acc[q]);
        }
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int b = b0 + 32 * q + ln;
        if (b < next && __ldg(bt + b) < ness) atomicAdd(r0 + __ldg(bt + b), -acc[q]);
      }
    }
}

// acc[j] = rows [8 strip, + 8) of the operator times columns [8 (j0 + j), + 8),
// over K rows of the columns (a multiple of 4).  Rows and columns past the
// ends are clamped, their results discarded.
template <int NT>
__device__ __forceinline__ void strip_product(double (&acc)[4][2], const double* sA, int ld, int rows, int strip,
                                              const double* sB, int ncol, int j0, int K) {
  const int ln = threadIdx.x & 31, g8 = ln >> 2, t4 = ln & 3;
  const double* ap = sA + min(strip * 8 + g8, rows - 1) * ld + t4;
  const double* bp[NT];
#pragma unroll
  for (int j = 0; j < NT; ++j) bp[j] = sB + min((j0 + j) * 8 + g8, ncol - 1) * ld + t4;
#pragma unroll
  for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = 0.0;
#pragma unroll 4
  for (int k0 = 0; k0 < K; k0 += 4) {
    const double a = ap[k0];
#pragma unroll
    for (int j = 0; j < NT; ++j) dmma_8x8x4(acc[j][0], acc[j][1], a, bp[j][k0]);
  }
}

// A lane's nodes t0 + 32 u of an element: their global numbers (-1 inside the
// element, -2 past its nodes) and -Q4.
struct ElemNodes {
  int gi[kElemRounds];
  double w[kElemRounds];
  __device__ __forceinline__ void load(const double* __restrict__ q4, const int* __restrict__ gid, int t0, int nn) {
#pragma unroll
    for (int u = 0; u < kElemRounds; ++u) {
      const bool in = t0 + 32 * u < nn;
      gi[u] = in ? __ldg(gid + t0 + 32 * u) : -2;
      w[u] = in ? -__ldg(q4 + t0 + 32 * u) : 0.0;
    }
  }
};

// The same nodes' column entries (NR planes of the mode) into shared memory:
// every load is in flight before the first is used, every address a base plus
// a constant.  f0, u0: the element in the mode's first plane of F, U; y0, g0:
// the plane vectors.  lifted: whether a node has an essential value that is
// not zero.
template <bool kRecover, int NR>
__device__ __forceinline__ void load_nodes(const ElemNodes& E, const double* __restrict__ f0, double* u0,
                                           const double* __restrict__ y0, const double* __restrict__ g0, size_t ps,
                                           int rstride, int t0, int nsolve, int ness, bool write_u, double* b0,
                                           double* b1, bool& lifted) {
  double v[kElemRounds][NR];
#pragma unroll
  for (int u = 0; u < kElemRounds; ++u)
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      if (kRecover) {
        v[u][r] = 0.0;
        if (E.gi[u] == -1) v[u][r] = f0[r * ps + t0 + 32 * u];
        else if (E.gi[u] >= 0 && E.gi[u] < nsolve) v[u][r] = y0[static_cast<size_t>(r) * rstride + E.gi[u]];
      } else {
        v[u][r] = E.gi[u] != -2 ? f0[r * ps + t0 + 32 * u] : 0.0;
      }
    }
#pragma unroll
  for (int u = 0; u < kElemRounds; ++u) {
    if (E.gi[u] == -2) break;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      double* b = r ? b1 : b0;
      double gv = 0.0;
      if (g0 && E.gi[u] >= ness) {
        gv = g0[static_cast<size_t>(r) * rstride + E.gi[u]];
        lifted = lifted || gv != 0.0;
      }
      if (kRecover && E.gi[u] >= 0) {
        const double ub = E.gi[u] >= ness ? gv : v[u][r];
        b[t0 + 32 * u] = ub;
        if (write_u) u0[r * ps + t0 + 32 * u] = ub;
      } else {
        b[t0 + 32 * u] = E.w[u] * v[u][r];
      }
    }
  }
}

// kRecover: U of the elements' nodes (essential and pinned ones included);
// otherwise R += the condensed forcing.  Block (part of a chunk, mode, row
// block and first of the block's `fpb` fields).
template <bool kRecover>
__global__ void __launch_bounds__(kElemThreads, 2)
    k_elem(DevGeom g, SolveFields B, DevModal S, int rstride, ElementShape P, int parts, int fpb) {
  extern __shared__ __align__(16) unsigned char sraw[];
  pdl_trigger();
  const int chunk = blockIdx.x / parts, part = blockIdx.x - chunk * parts, m = S.mode0 + blockIdx.y;
  const int rb = blockIdx.z % P.nrb, f0 = blockIdx.z / P.nrb * fpb, f1 = min(f0 + fpb, B.n);
  const int nr = (g.nz > 1 && m > 0) ? 2 : 1, pe = P.pe;
  const int wp = threadIdx.x >> 5, ln = threadIdx.x & 31, nwp = blockDim.x >> 5;
  const int nn = g.npnp, next = g.next, nint = g.nint;
  const int4 cd = __ldg(g.chunk_desc + chunk);  // start, count, family
  const int cnt = min(pe, cd.y - part * pe), ncol = nr * cnt;
  if (cnt <= 0) {  // the whole block
    pdl_wait();
    return;
  }
  const int ld = S.ew_ld, nrow = kRecover ? nint : next;
  const int r_lo = rb * P.rows, rows = min(P.rows, nrow - r_lo);
  const ElemSmem L = elem_layout(P.rows, g.nz > 1 ? 2 * pe : pe, ld, elem_tab(kRecover, P.rows, pe));
  uint64_t* bar = reinterpret_cast<uint64_t*>(sraw);
  double* sA = reinterpret_cast<double*>(sraw + L.a);
  double* sB = reinterpret_cast<double*>(sraw + L.b);
  size_t* sOut = reinterpret_cast<size_t*>(sraw + L.out);  // offset of each column's results in U or R
  int* sEl = reinterpret_cast<int*>(sraw + L.el);
  int* sTab = reinterpret_cast<int*>(sraw + L.tab);
  const size_t fm = static_cast<size_t>(m) * S.nfamily + cd.z, ps = g.plane_size;
  stage_rows(bar, sA, (kRecover ? S.ew : S.eb) + (fm * nrow + r_lo) * ld,
             static_cast<unsigned>(sizeof(double) * rows * ld));
  const int* el = g.elem_sorted + cd.x + part * pe;
  const DevNumbering& N0 = B.f[f0].N;  // the fields of a solve share their numbering
  if (threadIdx.x < cnt) sEl[threadIdx.x] = __ldg(el + threadIdx.x);
  if (threadIdx.x < ncol) {
    int slot, l;
    col_slot(threadIdx.x, cnt, slot, l);
    const size_t k = 2 * m + slot;
    sOut[threadIdx.x] = kRecover ? k * ps + static_cast<size_t>(__ldg(el + l)) * nn : k * rstride;
  }
  if (kRecover) {
    for (int i = threadIdx.x; i < rows; i += blockDim.x) sTab[i] = __ldg(g.emap + next + r_lo + i);
  } else {
    for (int i = threadIdx.x; i < cnt * rows; i += blockDim.x) {
      const int l = i / rows;
      sTab[i] = __ldg(N0.btog + static_cast<size_t>(__ldg(el + l)) * next + r_lo + i - l * rows);
    }
  }
  for (int c = wp; c < ncol; c += nwp)  // padding rows of every column
    if (nn + ln < ld) sB[c * ld + nn + ln] = 0.0;
  __syncthreads();
  const int nsolve = S.nsolve[m];
  const int strips = (rows + 7) / 8, ntile = (ncol + 7) / 8, K = (nn + 3) / 4 * 4;
  // column tiles per warp unit: four, fewer where that leaves half the warps idle
  int tiles = 4;
  while (tiles > 1 && 2 * strips * ((ntile + tiles - 1) / tiles) <= nwp) tiles >>= 1;
  const int groups = (ntile + tiles - 1) / tiles;
  ElemNodes E;
  if (wp < cnt) E.load(g.Q4 + static_cast<size_t>(sEl[wp]) * nn, N0.node_gid + static_cast<size_t>(sEl[wp]) * nn, ln, nn);
  pdl_wait();  // the operators and numbering are set-up data; the vectors come from earlier kernels
  bool first = true;
  for (int f = f0; f < f1; ++f) {
    const SolveField& fl = B.f[f];
    const size_t p0 = static_cast<size_t>(2 * m) * ps, v0 = static_cast<size_t>(2 * m) * rstride;
    const double *y0 = kRecover ? fl.Y + v0 : nullptr, *g0 = fl.G ? fl.G + v0 : nullptr;
    for (int l = wp; l < cnt; l += nwp) {
      const size_t o = static_cast<size_t>(sEl[l]) * nn;
      double *b0 = sB + l * ld, *b1 = sB + (cnt + l) * ld;
      bool lifted = false;
      for (int t0 = ln; t0 - ln < nn; t0 += 32 * kElemRounds) {
        if (!first) E.load(g.Q4 + o, N0.node_gid + o, t0, nn);
        first = false;
        if (nr == 2)
          load_nodes<kRecover, 2>(E, fl.F + p0 + o, fl.U + p0 + o, y0, g0, ps, rstride, t0, nsolve, N0.nsolve, rb == 0, b0,
                                  b1, lifted);
        else
          load_nodes<kRecover, 1>(E, fl.F + p0 + o, fl.U + p0 + o, y0, g0, ps, rstride, t0, nsolve, N0.nsolve, rb == 0, b0,
                                  b1, lifted);
      }
      // the condensed lift term (the recovery's operator applies it to the
      // column's essential values)
      if (!kRecover && rb == 0 && __any_sync(0xffffffffu, lifted))
        lift_element(S.sc + fm * next * S.sc_ld, S.sc_ld, N0.btog + static_cast<size_t>(sEl[l]) * next, next, N0.nsolve,
                     g0, fl.R + v0, rstride, nr);
    }
    __syncthreads();
    if (f == f0 && !rows_ready(bar, S.status, S.wait_ns)) return;
    for (int unit = wp; unit < strips * groups; unit += nwp) {
      const int strip = unit / groups, j0 = (unit - strip * groups) * tiles;
      double acc[4][2];
      const int nt = min(tiles, ntile - j0);
      if (nt == 4) strip_product<4>(acc, sA, ld, rows, strip, sB, ncol, j0, K);
      else if (nt == 3) strip_product<3>(acc, sA, ld, rows, strip, sB, ncol, j0, K);
      else if (nt == 2) strip_product<2>(acc, sA, ld, rows, strip, sB, ncol, j0, K);
      else strip_product<1>(acc, sA, ld, rows, strip, sB, ncol, j0, K);
      const int row = strip * 8 + (ln >> 2);
      if (row >= rows) continue;
      double* out = kRecover ? fl.U + sTab[row] : fl.R;
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int col = (j0 + j) * 8 + 2 * (ln & 3) + i;
          if (j >= nt || col >= ncol) break;
          if (kRecover) out[sOut[col]] = acc[j][i];
          else atomicAdd(out + sOut[col] + sTab[(col >= cnt ? col - cnt : col) * rows + row], acc[j][i]);
        }
    }
    if (f + 1 < f1) __syncthreads();  // every read of the columns is done
  }
}

// acc[j] = tile j0+j (8x8) of the warp's 8-row strip: A[strip rows][0:K)
// B[tile columns][boff : boff + K), K a multiple of 4; rows and columns past
// the ends are clamped (their results are discarded).
__device__ __forceinline__ void unit_product(double (&acc)[kUnitTiles][2], const double* sA, int lda, int rows,
                                             int strip, const double* sB, int ldb, int ncol, int j0, int ntile,
                                             int boff, int K) {
  const int ln = threadIdx.x & 31, g8 = ln >> 2, t4 = ln & 3;
  const double* ap = sA + min(strip * 8 + g8, rows - 1) * lda + t4;
  const double* bp[kUnitTiles];
#pragma unroll
  for (int j = 0; j < kUnitTiles; ++j) bp[j] = sB + min((j0 + j) * 8 + g8, ncol - 1) * ldb + boff + t4;
#pragma unroll
  for (int j = 0; j < kUnitTiles; ++j) acc[j][0] = acc[j][1] = 0.0;
#pragma unroll 4
  for (int k0 = 0; k0 < K; k0 += 4) {
    const double a = ap[k0];
#pragma unroll
    for (int j = 0; j < kUnitTiles; ++j)
      if (j0 + j < ntile) dmma_8x8x4(acc[j][0], acc[j][1], a, bp[j][k0]);
  }
}

// Element Schur complement products: one block per (chunk, mode).  The
// family-mode matrix S_e (rows padded) and the chunk's input columns (the
// source values at the element nodes of the taken class, zero elsewhere)
// in shared memory; out = S_e x on the tensor cores; the rows of the put
// class are subtracted from dst.  dir 0: patch-interior -> interface,
// 1: interface -> patch-interior, 2: every non-essential node both ways
// (dst -= S x, the skeleton residual).
__global__ void __launch_bounds__(256)
    k_elem_schur(int dir, DevGeom g, DevModal S, const double* __restrict__ src, double* __restrict__ dst, int rstride,
                 size_t fstride) {
  extern __shared__ __align__(16) unsigned char sraw[];
  pdl_trigger();
  src += (blockIdx.z / kSchurParts) * fstride;
  dst += (blockIdx.z / kSchurParts) * fstride;
  const int part = blockIdx.z % kSchurParts;
  const int c = blockIdx.x, m = S.mode0 + blockIdx.y;
  const int nr = (g.nz > 1 && m > 0) ? 2 : 1;
  // this block's part of the chunk: elements [e0, e0 + cnt)
  const int4 cd = __ldg(g.chunk_desc + c);  // start, count, family
  const int e0 = cd.y * part / kSchurParts, cnt = cd.y * (part + 1) / kSchurParts - e0;
  const int next = g.next, ncol = nr * cnt;
  const int lda = S.sc_ld, ldb = element_ld(next);
  double* sA = reinterpret_cast<double*>(sraw);               // [next][lda]
  double* sB = sA + next * lda;                               // [2 cm][ldb]
  int* sN = reinterpret_cast<int*>(sB + 2 * g.chunk_max * ldb);  // [cm][next] skeleton id << 2 | class
  const int take = dir == 0 ? 1 : 2, put = dir == 0 ? 2 : 1;
  const bool every = dir == 2;
  const double* A = S.sc + (static_cast<size_t>(m) * S.nfamily + cd.z) * next * lda;
  for (int i = threadIdx.x; i < next * lda; i += blockDim.x) sA[i] = __ldg(A + i);
  const int wp = threadIdx.x >> 5, ln = threadIdx.x & 31, nwp = blockDim.x >> 5;
  const int* code = S.l2_ncode + static_cast<size_t>(cd.x + e0) * next;
  for (int i = threadIdx.x; i < cnt * next; i += blockDim.x) sN[i] = __ldg(code + i);
  __syncthreads();
  pdl_wait();  // S_e and the node codes are set-up data; src and dst are not
  // input columns, loads of kColBatch columns per warp in flight together
  for (int c0 = wp; c0 < ncol; c0 += nwp * kColBatch) {
    double v[kColBatch][2];
#pragma unroll
    for (int j = 0; j < kColBatch; ++j) {
      const int col = c0 + j * nwp;
      int slot, l;
      col_slot(min(col, ncol - 1), cnt, slot, l);
      const double* sp = src + static_cast<size_t>(2 * m + slot) * rstride;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int a = ln + 32 * h;
        const int code_v = (col < ncol && a < next) ? sN[l * next + a] : 0;
        v[j][h] = (every ? (code_v & 3) != 0 : (code_v & 3) == take) ? sp[code_v >> 2] : 0.0;
      }
    }
#pragma unroll
    for (int j = 0; j < kColBatch; ++j) {
      const int col = c0 + j * nwp;
      if (col >= ncol) continue;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (ln + 32 * h < next) sB[col * ldb + ln + 32 * h] = v[j][h];
    }
  }
  __syncthreads();
  const int ntile = (ncol + 7) / 8, strips = (next + 7) / 8;
  const int ncg = (ntile + kUnitTiles - 1) / kUnitTiles;
  for (int unit = wp; unit < strips * ncg; unit += nwp) {
    const int strip = unit / ncg, j0 = (unit - strip * ncg) * kUnitTiles;
    double acc[kUnitTiles][2];
    unit_product(acc, sA, lda, next, strip, sB, ldb, ncol, j0, ntile, 0, next);
    const int row = strip * 8 + (ln >> 2);
#pragma unroll
    for (int j = 0; j < kUnitTiles; ++j)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int col = (j0 + j) * 8 + 2 * (ln & 3) + i;
        if (j0 + j < ntile && row < next && col < ncol) {
          int slot, l;
          col_slot(col, cnt, slot, l);
          const int code_v = sN[l * next + row];
          if (every ? (code_v & 3) != 0 : (code_v & 3) == put)
            atomicAdd(&dst[static_cast<size_t>(2 * m + slot) * rstride + (code_v >> 2)], -acc[j][i]);
        }
      }
  }
}

// Elements, operator rows and threads per block of a kernel with nrow operator
// rows.  Two blocks of 16 warps an SM or more (113 KB): all rows and 16, 12 or
// 8 elements (32 in one plane), or two balanced row blocks; failing that one
// block an SM.  Close to the limit (16 elements at N_P = 11 and 13) fewer elements
// a block while there are not 100 blocks (us a solve alone, 12 / 16 elements: 5 x
// 9 x 20, N_P = 13 43.8 / 45.5; 8 x 6 x 24, N_P = 11 38.1 / 40.3; 16 x 16 x 64,
// where there are, 148 / 142).  Filling the SMs with smaller row blocks where there are few
// chunks (one plane) shortens one solve (20 x 20, N_P = 8: 43 to 38 us alone)
// and costs many at once more: 16 uneven 2D problems in a graph 110 us, 120
// with at least 37 blocks a launch, 134 with 74.
bool elem_shape(bool recover, int nrow, const DevGeom& g, const DevModal& S, ElementShape& P,
                bool one_row_block = false) {
  const int planes = g.nz > 1 ? 2 : 1, ld = S.ew_ld, most = std::min(g.chunk_max, kElemCols / planes);
  auto bytes = [&](int rows, int pe) {
    return elem_layout(rows, pe * planes, ld, elem_tab(recover, rows, pe)).bytes;
  };
  constexpr size_t kTwoBlocks = 113 * 1024, kOneBlock = 226 * 1024;
  P.nrb = 0;
  for (int q = 4; q >= 2 && !P.nrb; --q) {
    const int pe = std::max(1, most * q / 4);
    const size_t b = bytes(nrow, pe);
    const int blocks = g.nchunk * ((g.chunk_max + pe - 1) / pe) * S.nmodes;
    if (b <= 104 * 1024 || (b <= kTwoBlocks && (blocks >= 100 || q == 2))) P = ElementShape{pe, nrow, 1};
  }
  if (one_row_block) {
    for (int q = 4; q >= 1 && !P.nrb; --q) {
      const int pe = std::max(1, most * q / 4);
      if (bytes(nrow, pe) <= kOneBlock) P = ElementShape{pe, nrow, 1};
    }
    if (!P.nrb) return false;
  }
  for (size_t cap : {kTwoBlocks, kOneBlock})
    for (int nrb = cap == kTwoBlocks ? 2 : 1; !P.nrb; ++nrb) {
      const int rows = nrb == 1 ? nrow : ((nrow + nrb - 1) / nrb + 7) / 8 * 8;
      if (bytes(rows, most) <= cap) P = ElementShape{most, rows, (nrow + rows - 1) / rows};
      else if (rows <= 8 || (cap == kTwoBlocks && nrb == 2)) break;
    }
  if (!P.nrb) return false;
  const int parts = (g.chunk_max + P.pe - 1) / P.pe;
  P.pe = (g.chunk_max + parts - 1) / parts;  // even parts
  return true;
}

template <bool kRecover>
void elem_launch(const ElementShape& P, const DevGeom& g, const SolveFields& B, const DevModal& S,
                 int rstride, cudaStream_t st) {
  const int parts = (g.chunk_max + P.pe - 1) / P.pe;
  // every field of a solve in the same block (its operator rows read once)
  // where the blocks still fill the SMs, else a block each
  const int fpb = g.nchunk * parts * S.nmodes * P.nrb >= 4 * 148 ? B.n : 1;
  const size_t smem =
      elem_layout(P.rows, P.pe * (g.nz > 1 ? 2 : 1), S.ew_ld, elem_tab(kRecover, P.rows, P.pe)).bytes;
  // eight warps where four blocks share an SM, else sixteen.  Close to the limit
  // of shared memory (N_P = 9 and 10) eight only if there is a block an SM: us a
  // step, sixteen below that / eight always: channel 5 x 14 x 14, N_P = 10 77.7 /
  // 83.1, 8 x 6 x 16, N_P = 9 44.9 / 49.2, 16 x 8 x 32 116.6 / 117.1; vortex 5 x 5
  // x 22, N_P = 10 71.6 / 73.5.  (Sixteen for every small grid: one solve alone 5
  // to 10 % faster, several side by side 3 to 7 % slower.)
  const int blocks = g.nchunk * parts * S.nmodes * P.nrb * ((B.n + fpb - 1) / fpb);
  const bool four = smem <= 52 * 1024 || (smem <= 56 * 1024 && blocks >= 100);
  const int threads = four ? kElemThreads / 2 : kElemThreads;
  raise_smem_limit(reinterpret_cast<const void*>(k_elem<kRecover>), smem);
  launch_ex(S.pdl != 0, k_elem<kRecover>, dim3(g.nchunk * parts, S.nmodes, P.nrb * ((B.n + fpb - 1) / fpb)),
            dim3(threads), smem, st, g, B, S, rstride, P, parts, fpb);
}

}  // namespace

ElementPlan element_plan(const DevGeom& g, const DevModal& S) {
  ElementPlan P;
  if (g.nchunk <= 0 || !S.ew || !S.eb || !S.sc || S.ew_ld <= 0 || g.nint <= 0) return P;
  P.ok = elem_shape(false, g.next, g, S, P.cond) && elem_shape(true, g.nint, g, S, P.rec);
  return P;
}

bool element_plan_in_place(const DevGeom& g, const DevModal& S, ElementPlan& P) {
  return P.rec.nrb == 1 || elem_shape(true, g.nint, g, S, P.rec, true);
}

void element_condense(const ElementPlan& P, const DevGeom& g, const SolveFields& B, const DevModal& S, int rstride,
                      cudaStream_t st) {
  elem_launch<false>(P.cond, g, B, S, rstride, st);
}

void element_recover(const ElementPlan& P, const DevGeom& g, const SolveFields& B, const DevModal& S, int rstride,
                     cudaStream_t st) {
  elem_launch<true>(P.rec, g, B, S, rstride, st);
}

void element_schur_apply(int dir, const DevGeom& g, const DevModal& S, const double* src, double* dst, int rstride,
                         int nf, size_t fstride, cudaStream_t st) {
  const size_t smem = sizeof(double) * (static_cast<size_t>(g.next) * S.sc_ld +
                                        2 * static_cast<size_t>(g.chunk_max) * element_ld(g.next)) +
                      sizeof(int) * static_cast<size_t>(g.chunk_max) * g.next;
  raise_smem_limit(reinterpret_cast<const void*>(k_elem_schur), smem);
  launch_ex(S.pdl != 0, k_elem_schur, dim3(g.nchunk, S.nmodes, kSchurParts * nf), dim3(256), smem, st, dir, g, S, src,
            dst, rstride, fstride);
}

}  // namespace stx
