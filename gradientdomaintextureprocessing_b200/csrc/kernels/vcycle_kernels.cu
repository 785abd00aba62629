// V-cycle kernels: colour-run Gauss-Seidel, residual, transfer operators,
// exact boundary-block solve, coarsest dense solve, FP64 refinement.
// Reference operators restated (same arithmetic, different work partition):
//   deep update      IterativeSolvers.inl:449-463   x = rhs*c4 - sum_{k!=4} c_k x_k
//   deep residual    IterativeSolvers.inl:479-493   r = rhs - (sum_{k!=4} c_k x_k + x) * c9
//   restriction      IterativeSolvers.inl:1037-1053 full weighting 1, 1/2, 1/4 (+ sparse boundary rows)
//   prolongation     IterativeSolvers.inl:1128-1151 bilinear 1/2, 1/4 with aligned-start parity
//   boundary relax   IterativeSolvers.inl:414-430   x_B = BB^-1 (rhs_B - BD x)
//   boundary residual IterativeSolvers.inl:549-555  r_B = rhs_B - BD x - BB x_B
//   raw operator     IterativeSolvers.inl:881-950   y = A x (MultiplyBySystemMatrix_NoReciprocals)
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "vcycle.cuh"
#include "vcycle_kernels.h"
#include "vcycle_ops.cuh"

namespace cg = cooperative_groups;

namespace gdtp {
namespace dev {

// ----------------------------------------------------------------------------
// Gauss-Seidel on one colour: x = rhs*c4 - sum_{k!=4} c_k x_k
// ----------------------------------------------------------------------------
template <typename T, int W>
__global__ void __launch_bounds__(256) k_gs_colour(const ColourRun* __restrict__ runs, int nRuns, const T* __restrict__ coef,
                                                   int planeStride, const T* __restrict__ rhs, T* __restrict__ x, int KP, int G,
                                                   int skip, int rhsEarly) {
  // What the previous launch cannot have written is loaded before waiting for
  // it, so that these loads overlap its tail: the run and its coefficients
  // (written at set-up), and the right-hand side when the previous launch is a
  // colour pass of the same smoothing step (rhsEarly).  x is read after the
  // wait.  The arithmetic is gs_item's, in the same order.
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int per = 32 * G;
  const long long r = t / per;
  const int rem = int(t - r * per);
  const int m = rem / G, q = rem - m * G;
  ColourRun R;
  R.len = 0;
  if (r < nRuns) R = runs[r];
  const bool active = r < nRuns && m < R.len;
  T w[10];
  Vec<T, W> b;
  int pos = 0, pp = 0, pn = 0;
  const int off = q * W;
  if (active) {
    pos = R.pos0 + 2 * m, pp = R.prev0 + 2 * m, pn = R.next0 + 2 * m;
    const T* c = coef + R.coef0 + m;
#pragma unroll
    for (int k = 0; k < 9; k++) w[k] = c[k * planeStride];
    if (rhsEarly) b = vload<T, W>(rhs + (long long)pos * KP + off);
  }
  grid_dependency_wait();
  grid_launch_dependents();
  if (!active) return;
  if (!rhsEarly) b = vload<T, W>(rhs + (long long)pos * KP + off);
  Vec<T, W> acc;
#pragma unroll
  for (int k = 0; k < W; k++) acc.v[k] = 0;
  if (!(skip & 1)) axpy(acc, w[0], vload<T, W>(x + (long long)(pp - 1) * KP + off));
  if (!(skip & 2)) axpy(acc, w[1], vload<T, W>(x + (long long)(pp)*KP + off));
  if (!(skip & 4)) axpy(acc, w[2], vload<T, W>(x + (long long)(pp + 1) * KP + off));
  if (!(skip & 8)) axpy(acc, w[3], vload<T, W>(x + (long long)(pos - 1) * KP + off));
  if (!(skip & 32)) axpy(acc, w[5], vload<T, W>(x + (long long)(pos + 1) * KP + off));
  if (!(skip & 64)) axpy(acc, w[6], vload<T, W>(x + (long long)(pn - 1) * KP + off));
  if (!(skip & 128)) axpy(acc, w[7], vload<T, W>(x + (long long)(pn)*KP + off));
  if (!(skip & 256)) axpy(acc, w[8], vload<T, W>(x + (long long)(pn + 1) * KP + off));
  Vec<T, W> out;
#pragma unroll
  for (int k = 0; k < W; k++) out.v[k] = b.v[k] * w[4] - acc.v[k];
  vstore<T, W>(x + (long long)pos * KP + off, out);
}

// Two colour passes of one row parity (launch_gs_rows).  Colours 0 and 1 hold
// the even rows, 2 and 3 the odd rows, and the 9-point stencil of a row reaches
// only its own row and the two rows of the other parity.  So the passes of one
// row parity update each raster line independently: the first colour (A) from
// the line's old values, then the second (B) from A's new values in the line.
// A block holds whole lines; thread q of a line owns its texels 2q and 2q + 1
// (A texel oA + 2q, B texel oB + 2q), which it stages with the rows above and
// below into shared memory (slot 0 of a line: texel -1, slot len + 1: texel
// len, the line's non-deep neighbours).  Coefficients and (rhsEarly) the
// right-hand side are loaded before the dependency wait, as in k_gs_colour; A
// texels of a line are consecutive in the colour-run planes, as are B texels.
// Each update is gs_item's sum in gs_item's order.
// blocks of BS threads per SM the row smoother is compiled for (registers)
template <typename T>
constexpr int rows_min_blocks(int bs) {
  return (sizeof(T) == 4 ? 1280 : 768) / bs > 0 ? (sizeof(T) == 4 ? 1280 : 768) / bs : 1;
}
template <typename T, int W, int BS>
__global__ void __launch_bounds__(BS) k_gs_rows(const RowLine* __restrict__ lines, const int* __restrict__ lineOf,
                                                           const T* __restrict__ coef, int planeStride, const T* __restrict__ rhs,
                                                           T* __restrict__ x, int KP, int slots, int oddFirst, int skip,
                                                           int rhsEarly) {
  extern __shared__ __align__(32) unsigned char smem_raw[];
  Vec<T, W>* up = reinterpret_cast<Vec<T, W>*>(smem_raw);
  Vec<T, W>* mid = up + slots;
  Vec<T, W>* dn = mid + slots;
  const int li = lineOf[(long long)blockIdx.x * BS + threadIdx.x];
  const int off = blockIdx.y * W;
  RowLine Ln;
  Ln.len = 0;
  int q = 0, a = 0, b = 0, s0 = 0, H = 0;
  bool hasA = false, hasB = false;
  T wA[9], wB[9];
  Vec<T, W> bA, bB;
  if (li >= 0) {
    Ln = lines[li];
    q = int(threadIdx.x) - (Ln.meta & 2047);
    s0 = (Ln.meta >> 11) & 8191;
    H = (Ln.len + 3) >> 1;
    const int oA = ((Ln.meta >> 24) & 1) ^ oddFirst;
    a = oA + 2 * q;
    b = (oA ^ 1) + 2 * q;
    hasA = a < Ln.len;
    hasB = b < Ln.len;
    const T* cA = coef + (oddFirst ? Ln.cOdd : Ln.cEven) + q;
    const T* cB = coef + (oddFirst ? Ln.cEven : Ln.cOdd) + q;
    if (hasA) {
#pragma unroll
      for (int k = 0; k < 9; k++) wA[k] = cA[k * planeStride];
      if (rhsEarly) bA = vload<T, W>(rhs + (long long)(Ln.pos + a) * KP + off);
    }
    if (hasB) {
#pragma unroll
      for (int k = 0; k < 9; k++) wB[k] = cB[k * planeStride];
      if (rhsEarly) bB = vload<T, W>(rhs + (long long)(Ln.pos + b) * KP + off);
    }
  }
  // shared slot of line texel i (-1 .. len): texels of even and odd i + 1 in
  // two halves, so that consecutive threads touch consecutive slots
  auto slot = [&](int i) { return s0 + (((i + 1) & 1) ? H + ((i + 1) >> 1) : ((i + 1) >> 1)); };
  grid_dependency_wait();
  grid_launch_dependents();
  const bool rowsA = !(skip & 1), rowsB = !(skip & 4);
  if (li >= 0) {
    const bool rows = rowsA || rowsB;
    auto stage = [&](int i) {
      const int sl = slot(i);
      mid[sl] = vload<T, W>(x + (long long)(Ln.pos + i) * KP + off);
      if (rows) {
        up[sl] = vload<T, W>(x + (long long)(Ln.prev + i) * KP + off);
        dn[sl] = vload<T, W>(x + (long long)(Ln.next + i) * KP + off);
      }
    };
    // the pair of texels (2q, 2q + 1) of the three rows, and the line's ends:
    // the first thread texel -1, the last thread texel len
    stage(2 * q);
    if (2 * q + 1 < Ln.len) stage(2 * q + 1);
    if (q == 0) stage(-1);
    if (2 * q + 2 >= Ln.len) stage(Ln.len);
    if (!rhsEarly) {
      if (hasA) bA = vload<T, W>(rhs + (long long)(Ln.pos + a) * KP + off);
      if (hasB) bB = vload<T, W>(rhs + (long long)(Ln.pos + b) * KP + off);
    }
  }
  __syncthreads();
  Vec<T, W> xa, xb;
  if (hasA) {
    const int sm = slot(a - 1), sc = slot(a), sp = slot(a + 1);
    Vec<T, W> acc;
#pragma unroll
    for (int k = 0; k < W; k++) acc.v[k] = 0;
    if (rowsA) {
      axpy(acc, wA[0], up[sm]);
      axpy(acc, wA[1], up[sc]);
      axpy(acc, wA[2], up[sp]);
    }
    if (!(skip & 2)) {
      axpy(acc, wA[3], mid[sm]);
      axpy(acc, wA[5], mid[sp]);
    }
    if (rowsA) {
      axpy(acc, wA[6], dn[sm]);
      axpy(acc, wA[7], dn[sc]);
      axpy(acc, wA[8], dn[sp]);
    }
#pragma unroll
    for (int k = 0; k < W; k++) xa.v[k] = bA.v[k] * wA[4] - acc.v[k];
    mid[sc] = xa;  // A slots are read only by B updates, after the barrier
  }
  __syncthreads();
  if (hasB) {
    const int sm = slot(b - 1), sc = slot(b), sp = slot(b + 1);
    Vec<T, W> acc;
#pragma unroll
    for (int k = 0; k < W; k++) acc.v[k] = 0;
    if (rowsB) {
      axpy(acc, wB[0], up[sm]);
      axpy(acc, wB[1], up[sc]);
      axpy(acc, wB[2], up[sp]);
    }
    if (!(skip & 8)) {
      axpy(acc, wB[3], mid[sm]);
      axpy(acc, wB[5], mid[sp]);
    }
    if (rowsB) {
      axpy(acc, wB[6], dn[sm]);
      axpy(acc, wB[7], dn[sc]);
      axpy(acc, wB[8], dn[sp]);
    }
#pragma unroll
    for (int k = 0; k < W; k++) xb.v[k] = bB.v[k] * wB[4] - acc.v[k];
  }
  // texels 2q and 2q + 1 of the line, in address order
  if (a < b) {
    if (hasA) vstore<T, W>(x + (long long)(Ln.pos + a) * KP + off, xa);
    if (hasB) vstore<T, W>(x + (long long)(Ln.pos + b) * KP + off, xb);
  } else {
    if (hasB) vstore<T, W>(x + (long long)(Ln.pos + b) * KP + off, xb);
    if (hasA) vstore<T, W>(x + (long long)(Ln.pos + a) * KP + off, xa);
  }
}

// Every sweep of one smoothing step on one chart per block: the colour passes
// of a chart only read texels of that chart (deep) or boundary texels, which
// the sweeps do not change, so block barriers order the passes.  The chart's
// texel span of x is staged in shared memory for all passes (the smoothing of
// a small level is a chain of dependent memory latencies, and shared memory
// has the shortest); the updated deep texels are written back at the end.  The
// arithmetic is gs_item's, so the result is the launch path's, bit for bit.
constexpr int kGroupBlockMax = 1024;
template <typename T, int W>
__global__ void __launch_bounds__(kGroupBlockMax, 1) k_gs_groups(const ColourRun* __restrict__ runs, const int* __restrict__ groups,
                                                               const T* __restrict__ coef, int planeStride, const T* __restrict__ rhs,
                                                               T* __restrict__ x, int KP, int G, int sweeps, int reverse) {
  grid_dependency_wait();
  grid_launch_dependents();
  extern __shared__ __align__(32) unsigned char smem_raw[];
  T* xs = reinterpret_cast<T*>(smem_raw);
  const int* g = groups + 10 * blockIdx.x;
  const int lo = g[8], span = g[9];
  const int nt = blockDim.x;
  for (long long i = threadIdx.x; i < (long long)span * KP; i += nt) xs[i] = x[(long long)lo * KP + i];
  __syncthreads();
  for (int sw = 0; sw < sweeps; sw++)
    for (int cc = 0; cc < 4; cc++) {
      const int c = reverse ? 3 - cc : cc;
      const int nr = g[4 + c];
      const ColourRun* rc = runs + g[c];
      for (long long t = threadIdx.x; t < (long long)nr * 32 * G; t += nt) {
        const int per = 32 * G;
        const int r = int(t / per), rem = int(t - (long long)r * per);
        const int m = rem / G, q = rem - m * G;
        const ColourRun R = rc[r];
        if (m >= R.len) continue;
        // gs_item with positions relative to the span
        const int pos = R.pos0 + 2 * m - lo, pp = R.prev0 + 2 * m - lo, pn = R.next0 + 2 * m - lo;
        const T* cf = coef + R.coef0 + m;
        const int off = q * W;
        Vec<T, W> acc;
#pragma unroll
        for (int k = 0; k < W; k++) acc.v[k] = 0;
        axpy(acc, cf[0 * planeStride], vload<T, W>(xs + (pp - 1) * KP + off));
        axpy(acc, cf[1 * planeStride], vload<T, W>(xs + (pp)*KP + off));
        axpy(acc, cf[2 * planeStride], vload<T, W>(xs + (pp + 1) * KP + off));
        axpy(acc, cf[3 * planeStride], vload<T, W>(xs + (pos - 1) * KP + off));
        axpy(acc, cf[5 * planeStride], vload<T, W>(xs + (pos + 1) * KP + off));
        axpy(acc, cf[6 * planeStride], vload<T, W>(xs + (pn - 1) * KP + off));
        axpy(acc, cf[7 * planeStride], vload<T, W>(xs + (pn)*KP + off));
        axpy(acc, cf[8 * planeStride], vload<T, W>(xs + (pn + 1) * KP + off));
        const T c4 = cf[4 * planeStride];
        const Vec<T, W> bv = vload<T, W>(rhs + (long long)(pos + lo) * KP + off);
        Vec<T, W> out;
#pragma unroll
        for (int k = 0; k < W; k++) out.v[k] = bv.v[k] * c4 - acc.v[k];
        vstore<T, W>(xs + pos * KP + off, out);
      }
      __syncthreads();
    }
  // write back the chart's deep texels (the rest of the span is unchanged and
  // may not be written: boundary texels belong to the boundary solve's order)
  for (int c = 0; c < 4; c++) {
    const int nr = g[4 + c];
    const ColourRun* rc = runs + g[c];
    for (long long t = threadIdx.x; t < (long long)nr * 32; t += nt) {
      const int r = int(t >> 5), m = int(t & 31);
      const ColourRun R = rc[r];
      if (m >= R.len) continue;
      const int pos = R.pos0 + 2 * m;
      for (int k = 0; k < KP; k++) x[(long long)pos * KP + k] = xs[(pos - lo) * KP + k];
    }
  }
}

// ----------------------------------------------------------------------------
// Residual: deep rows by runs (all colours), boundary rows by CSR (global cols).
// Blocks [0, deepBlocks) handle deep texels, the rest boundary rows.
// ----------------------------------------------------------------------------
template <typename T, int W>
__global__ void __launch_bounds__(256) k_residual(const ColourRun* __restrict__ runs, int nRuns, const T* __restrict__ coef,
                                                  int planeStride, int deepBlocks, const int* __restrict__ bPtr,
                                                  const int* __restrict__ bCol, const T* __restrict__ bVal,
                                                  const int* __restrict__ bGlobal, int nB, const T* __restrict__ rhs,
                                                  const T* __restrict__ x, T* __restrict__ res, int KP, int G, int rhsEarly, int rowLanes) {
  if ((int)blockIdx.x >= deepBlocks) {
    const long long t = (long long)(blockIdx.x - deepBlocks) * blockDim.x + threadIdx.x;
    if (rowLanes == 1) {  // a thread per row and group (row_lanes)
      grid_dependency_wait();
      grid_launch_dependents();
      residual_boundary_item<T, W, LoadDefault>(bPtr, bCol, bVal, bGlobal, nB, rhs, x, res, KP, G, t);
      return;
    }
    // residual_boundary_item's sum on 8 lanes, its first entries loaded before the wait
    const long long row = t >> 3;
    const int lane8 = int(t & 7), off = 0;
    const bool valid = row < nB;
    const int g = valid ? bGlobal[row] : 0;
    OrderedRow8<T, W, 2> entries(bCol, bVal, valid ? bPtr[row] : 0, valid ? bPtr[row + 1] : 0, lane8);
    grid_dependency_wait();
    grid_launch_dependents();
    Vec<T, W> acc = vload<T, W>(rhs + (long long)g * KP + off);
    entries.add_to(acc, true, bCol, bVal, lane8, [&](int c) { return vload<T, W>(x + (long long)c * KP + off); });
    if (valid && lane8 == 0) vstore<T, W>(res + (long long)g * KP + off, acc);
    return;
  }
  // deep items (residual_deep_item's arithmetic, same order): the run and its
  // coefficients (set-up data), and rhs when the previous launch does not
  // write it (rhsEarly), are loaded before waiting for the previous launch
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int per = 32 * G;
  const long long r = t / per;
  const int rem = int(t - r * per);
  const int m = rem / G, q = rem - m * G;
  ColourRun R;
  R.len = 0;
  if (r < nRuns) R = runs[r];
  const bool active = r < nRuns && m < R.len;
  T w[10];
  Vec<T, W> b;
  int pos = 0, pp = 0, pn = 0;
  const int off = q * W;
  if (active) {
    pos = R.pos0 + 2 * m, pp = R.prev0 + 2 * m, pn = R.next0 + 2 * m;
    const T* c = coef + R.coef0 + m;
#pragma unroll
    for (int k = 0; k < 10; k++)
      if (k != 4) w[k] = c[k * planeStride];
    if (rhsEarly) b = vload<T, W>(rhs + (long long)pos * KP + off);
  }
  grid_dependency_wait();
  grid_launch_dependents();
  if (!active) return;
  if (!rhsEarly) b = vload<T, W>(rhs + (long long)pos * KP + off);
  Vec<T, W> acc = vload<T, W>(x + (long long)pos * KP + off);
  axpy(acc, w[0], vload<T, W>(x + (long long)(pp - 1) * KP + off));
  axpy(acc, w[1], vload<T, W>(x + (long long)(pp)*KP + off));
  axpy(acc, w[2], vload<T, W>(x + (long long)(pp + 1) * KP + off));
  axpy(acc, w[3], vload<T, W>(x + (long long)(pos - 1) * KP + off));
  axpy(acc, w[5], vload<T, W>(x + (long long)(pos + 1) * KP + off));
  axpy(acc, w[6], vload<T, W>(x + (long long)(pn - 1) * KP + off));
  axpy(acc, w[7], vload<T, W>(x + (long long)(pn)*KP + off));
  axpy(acc, w[8], vload<T, W>(x + (long long)(pn + 1) * KP + off));
  Vec<T, W> out;
#pragma unroll
  for (int k = 0; k < W; k++) out.v[k] = b.v[k] - acc.v[k] * w[9];
  vstore<T, W>(res + (long long)pos * KP + off, out);
}

// ----------------------------------------------------------------------------
// Restriction of the residual to the coarse right-hand side.
// ----------------------------------------------------------------------------
template <typename T, int W>
__global__ void __launch_bounds__(256) k_restrict(const RestrictRun* __restrict__ runs, int nRuns, int deepBlocks,
                                                  const int* __restrict__ rPtr, const int* __restrict__ rCol,
                                                  const T* __restrict__ rVal, const int* __restrict__ rOut, int nB,
                                                  const T* __restrict__ res, T* __restrict__ coarseRhs, T* __restrict__ coarseX,
                                                  long long coarseVals, int KP, int G, int rowLanes) {
  // the coarse iterate starts from zero: cleared here (grid-stride), before
  // waiting for the previous launch (the residual of this level, which does
  // not touch the coarse level)
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < coarseVals; i += (long long)gridDim.x * blockDim.x)
    coarseX[i] = T(0);
  if ((int)blockIdx.x < deepBlocks) {
    grid_dependency_wait();
    grid_launch_dependents();
    restrict_deep_item<T, W, LoadDefault>(runs, nRuns, res, coarseRhs, KP, G, (long long)blockIdx.x * blockDim.x + threadIdx.x);
    return;
  }
  const long long t = (long long)(blockIdx.x - deepBlocks) * blockDim.x + threadIdx.x;
  if (rowLanes == 1) {
    grid_dependency_wait();
    grid_launch_dependents();
    restrict_boundary_item<T, W, LoadDefault>(rPtr, rCol, rVal, rOut, nB, res, coarseRhs, KP, G, t);
    return;
  }
  // restrict_boundary_item's sum on 8 lanes, its first entries loaded before the wait
  const long long row = t >> 3;
  const int lane8 = int(t & 7), off = 0;
  const bool valid = row < nB;
  const int o = valid ? rOut[row] : 0;
  OrderedRow8<T, W, 2> entries(rCol, rVal, valid ? rPtr[row] : 0, valid ? rPtr[row + 1] : 0, lane8);
  grid_dependency_wait();
  grid_launch_dependents();
  Vec<T, W> acc;
#pragma unroll
  for (int k = 0; k < W; k++) acc.v[k] = 0;
  entries.add_to(acc, false, rCol, rVal, lane8, [&](int c) { return vload<T, W>(res + (long long)c * KP + off); });
  if (valid && lane8 == 0) vstore<T, W>(coarseRhs + (long long)o * KP + off, acc);
}

// ----------------------------------------------------------------------------
// Prolongation of the coarse correction, added to the fine iterate.
// ----------------------------------------------------------------------------
template <typename T, int W>
__global__ void __launch_bounds__(256) k_prolong_add(const ProlongRun* __restrict__ runs, int nRuns, const T* __restrict__ coarse,
                                                     T* __restrict__ fine, int KP, int G) {
  // prolong_item's arithmetic; the run and the fine value (this level's iterate,
  // which the previous launch, on the coarse level, does not write) are loaded
  // before waiting for it, the coarse values after
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int per = 32 * G;
  const long long r = t / per;
  const int rem = int(t - r * per);
  const int m = rem / G, q = rem - m * G;
  ProlongRun R{};
  if (r < nRuns) R = runs[r];
  const bool active = r < nRuns && m < R.len;
  const int off = q * W;
  T* dst = active ? fine + (long long)(R.f0 + m) * KP + off : nullptr;
  Vec<T, W> acc;
  if (active) acc = vload<T, W>(dst);
  grid_dependency_wait();
  grid_launch_dependents();
  if (!active) return;
  const int i = R.i0 + m, o = R.aligned ? 0 : 1;
  const int p = (i + o) / 2, n = (i + o + 1) / 2;
  if (R.center >= 0) {
    const Vec<T, W> a = vload<T, W>(coarse + (long long)(R.center + p) * KP + off),
                    b = vload<T, W>(coarse + (long long)(R.center + n) * KP + off);
#pragma unroll
    for (int k = 0; k < W; k++) acc.v[k] += (a.v[k] + b.v[k]) * T(0.5);
  } else {
    const Vec<T, W> a = vload<T, W>(coarse + (long long)(R.prev + p) * KP + off),
                    b = vload<T, W>(coarse + (long long)(R.prev + n) * KP + off),
                    c = vload<T, W>(coarse + (long long)(R.next + p) * KP + off),
                    d = vload<T, W>(coarse + (long long)(R.next + n) * KP + off);
#pragma unroll
    for (int k = 0; k < W; k++) acc.v[k] += (a.v[k] + b.v[k] + c.v[k] + d.v[k]) * T(0.25);
  }
  vstore<T, W>(dst, acc);
}

// ----------------------------------------------------------------------------
// Exact boundary-block solve  x_B = BB^-1 (rhs_B - BD x) over the subdomain /
// separator split (scaled by s = BB_ii^-1/2), four launches per level:
//   k_bs_prep:          r^ = s (rhs - BD x) for every boundary position
//   k_bs_dense mode 0:  y  = Inv_p r^_I
//   k_bs_dense mode 1:  xs = Sinv t,      t  = r^_S - A_SI y built in the prologue;
//                       x_S = s xs
//   k_bs_back:          x_I = s (y - W_p xs),  W_p = Inv_p A_{I_p,S} (m x t_p)
// The sparse row sums run on 8 lanes per row (group8_sum in vcycle_ops.cuh).
// The dense products stream the symmetric inverses, stored row-major with rows
// padded to a multiple of 4: lane l of a warp reads rows 4l..4l+3 of matrix row j
// with one vector load, so a warp reads contiguous memory.  The j range of a row
// group (128 rows of one matrix) is cut into nch chunks, which keeps the
// dependent-load chain of each warp short on the small levels (8 warps interleave
// a chunk's j); partial sums are added warps first, then chunks, in order, so the
// result does not depend on scheduling.
// ----------------------------------------------------------------------------

// Chunks of one row group share a cluster of up to kBsClusterMax CTAs: CTA r takes
// chunks r, r + CS, ..., one per group of 8 warps (blockDim / 256 groups, then the
// next round), and stores each partial sum into the shared memory of the CTA that
// will write the row (distributed shared memory); after one cluster barrier every
// CTA adds its rows' chunks, in order, from its own.
// What bounds it: on every level but the finest a product is a few MB behind a chain
// of latencies, so what is set-up data (task, first matrix rows, couplings) is
// loaded before the dependency wait, and the chunks' sums no longer go through
// global memory, fences and an arrival counter (the last CTA then read them back: two
// more trips).  Per refinement step with the early loads of k_bs_prep and k_bs_back:
// 256^2 torus 134 -> 124 us, 1024^2 genus-2 (one channel) 153 -> 149, 1024^2
// icosphere 334 -> 315, 2048^2 672 -> 655, 15 right-hand sides 490 -> 435.  Storing
// the sums where they are added, instead of reading them there (a trip and a second
// barrier), and accumulators without bank conflicts (16-way before): 120, 146, 310,
// 653 and 414 us.
// Shared memory: vin [groups][Q][chunk], red [groups][8][128 W], recv [chunks][values
// this CTA writes].  A row group's values are numbered (row % 4, row / 4, channel), so
// that a warp's accumulators go to shared memory without bank conflicts.
constexpr int kBsClusterMax = 8;
constexpr size_t kBsDenseSmemMax = 200 * 1024;
// Threads a CTA is compiled for: with the couplings in registers the separator
// product (mode 1) spills at the 64 registers of 1024 threads
template <typename T>
constexpr int bs_dense_threads(int Q, int mode) { return sizeof(T) == 4 && Q == 1 ? (mode == 0 ? 1024 : 768) : 512; }
template <typename T, int W, int Q, int mode>
__global__ void __launch_bounds__(bs_dense_threads<T>(Q, mode)) k_bs_dense(BoundaryDev<T> B, int nch, int clen0, T* __restrict__ x,
                                                                     int KP) {
  extern __shared__ __align__(32) unsigned char smem_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int CS = gridDim.y, rank = blockIdx.y, groups = blockDim.x >> 8, grp = threadIdx.x >> 8, tg = threadIdx.x & 255;
  constexpr int kRowVals = 128 * W;  // values of one channel group of the task's rows
  Vec<T, W>* vin = reinterpret_cast<Vec<T, W>*>(smem_raw) + size_t(grp) * Q * clen0;
  T* redAll = reinterpret_cast<T*>(reinterpret_cast<Vec<T, W>*>(smem_raw) + size_t(groups) * Q * clen0);
  T* red = redAll + size_t(grp) * 8 * kRowVals;
  T* recv = redAll + size_t(groups) * 8 * kRowVals;
  const int share = (Q * kRowVals + CS - 1) / CS;  // CTA r writes values [r share, (r + 1) share)
  // the CTAs of the cluster are running once this barrier's wait returns (before
  // the first remote store)
  if (CS > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  // the block's task, its matrix and its rows of it are set-up data: read (and
  // the rows prefetched into L2) before waiting for the previous launch
  const int4 task = (mode == 0 ? B.subTasks : B.schurTasks)[blockIdx.x];
  const int warp = tg >> 5, lane = tg & 31, rq = task.y + lane;
  const int r0 = mode == 0 ? B.subPtr[task.x] : 0;
  const int m = mode == 0 ? B.subPtr[task.x + 1] - r0 : B.nS, mp = (m + 3) & ~3;
  const T* M = mode == 0 ? B.inv + B.invOff[task.x] : B.sinv;
  const int clen = (m + nch - 1) / nch;
  const int c0 = blockIdx.z * Q * W;  // first channel
  if (blockIdx.z == 0) {
    // rows of this group's chunks, columns 4 task.y .. 4 task.y + 127 (clipped to the padded row)
    const int col0 = 4 * task.y, cols = max(0, min(mp - col0, 128));
    if (lane * 32 < cols * (int)sizeof(T))
      for (int ch = rank + CS * grp; ch < nch; ch += CS * groups) {
        const int j0 = min(m, ch * clen), j1 = min(m, j0 + clen);
        for (int j = j0 + warp; j < j1; j += 8)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(M + (long long)j * mp + col0) + lane * 32));
      }
  }
  // the first rows of this warp's first chunk into registers; mode 1: the first
  // row's couplings
  const bool active = 4 * rq < m;
  constexpr int kPre = W == 1 ? 4 : sizeof(T) == 4 ? 2 : 1;
  Quad<T> pre[kPre];
  constexpr int kPreA = W == 1 ? 4 : 3;
  T aw[kPreA];
  int ac[kPreA], ae0 = 0, ae1 = 0;
  {
    const int ch = rank + CS * grp, j0 = min(m, ch * clen), j1 = min(m, j0 + clen);
    if (active)
#pragma unroll
      for (int u = 0; u < kPre; u++)
        if (j0 + warp + 8 * u < j1) pre[u] = *reinterpret_cast<const Quad<T>*>(M + (long long)(j0 + warp + 8 * u) * mp + 4 * rq);
    if (mode == 1 && j0 + (tg >> 3) < j1) {
      ae0 = B.asiPtr[j0 + (tg >> 3)] + (tg & 7);
      ae1 = B.asiPtr[j0 + (tg >> 3) + 1];
#pragma unroll
      for (int u = 0; u < kPreA; u++)
        if (ae0 + 8 * u < ae1) {
          aw[u] = B.asiVal[ae0 + 8 * u];
          ac[u] = B.asiCol[ae0 + 8 * u];
        }
    }
  }
  grid_dependency_wait();
  grid_launch_dependents();
  const int rounds = (nch - rank + CS * groups - 1) / (CS * groups);  // the same for every group of the CTA
  for (int rd = 0; rd < rounds; rd++) {
    const int ch = rank + CS * (grp + groups * rd);
    const bool has = ch < nch;
    const int j0 = has ? min(m, ch * clen) : 0, j1 = has ? min(m, j0 + clen) : 0;
    // the chunk's input vector (mode 0: the scaled right-hand side from k_bs_prep;
    // mode 1: minus the coupling to the interior solution)
    if (mode == 0) {
      for (int i = tg; i < (j1 - j0) * Q; i += 256) {
        const int j = Q == 1 ? i : i / Q, q = Q == 1 ? 0 : i - j * Q;
        vin[q * clen0 + j] = vload<T, W>(B.rhat + (long long)(r0 + j0 + j) * KP + c0 + q * W);
      }
    } else {
      const int lane8 = tg & 7, row = tg >> 3;
      for (int q = 0; q < Q; q++)
        for (int jb = j0; jb < j1; jb += 32) {  // 32 groups of 8 lanes
          const int j = jb + row;
          Vec<T, W> v;
          if (rd == 0 && jb == j0) {
            // bs_schur_input_group's sums from the couplings loaded above
            Vec<T, W> sum, y[kPreA], r;
#pragma unroll
            for (int c = 0; c < W; c++) sum.v[c] = 0;
            if (j < j1 && lane8 == 0) r = vload<T, W>(B.rhat + (long long)(B.nI + j) * KP + c0 + q * W);
#pragma unroll
            for (int u = 0; u < kPreA; u++)
              if (ae0 + 8 * u < ae1) y[u] = vload<T, W>(B.y + (long long)ac[u] * KP + c0 + q * W);
#pragma unroll
            for (int u = 0; u < kPreA; u++)
              if (ae0 + 8 * u < ae1) fma_to(sum, aw[u], y[u]);
            for (int e = ae0 + 8 * kPreA; e < ae1; e += 8) fma_to(sum, B.asiVal[e], vload<T, W>(B.y + (long long)B.asiCol[e] * KP + c0 + q * W));
            sum = group8_sum(sum);
#pragma unroll
            for (int c = 0; c < W; c++) v.v[c] = r.v[c] - sum.v[c];
          } else {
            v = bs_schur_input_group<T, W, LoadDefault>(B, j, j < j1, KP, c0 + q * W, lane8);
          }
          if (j < j1 && lane8 == 0) vin[q * clen0 + j - j0] = v;
        }
    }
    __syncthreads();
    T acc[4][Q * W];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int c = 0; c < Q * W; c++) acc[a][c] = 0;
    if (active) {
      auto add = [&](const Quad<T>& mq, int j) {
#pragma unroll
        for (int q = 0; q < Q; q++) {
          const Vec<T, W> v = vin[q * clen0 + j - j0];
#pragma unroll
          for (int a = 0; a < 4; a++)
#pragma unroll
            for (int c = 0; c < W; c++) acc[a][q * W + c] = fma(mq.v[a], v.v[c], acc[a][q * W + c]);
        }
      };
      int j = j0 + warp;
      if (rd == 0) {
#pragma unroll
        for (int u = 0; u < kPre; u++)
          if (j + 8 * u < j1) add(pre[u], j + 8 * u);
        j += 8 * kPre;
      }
      constexpr int kAhead = sizeof(T) == 4 ? 4 : 6;
#pragma unroll kAhead
      for (; j < j1; j += 8) add(*reinterpret_cast<const Quad<T>*>(M + (long long)j * mp + 4 * rq), j);
    }
    if (CS > 1 && rd == 0) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
#pragma unroll
    for (int q = 0; q < Q; q++) {
      if (q) __syncthreads();
#pragma unroll
      for (int a = 0; a < 4; a++) {
        Vec<T, W> v;
#pragma unroll
        for (int c = 0; c < W; c++) v.v[c] = acc[a][q * W + c];
        vstore<T, W>(red + warp * kRowVals + (a * 32 + lane) * W, v);
      }
      __syncthreads();
      for (int o = tg; o < kRowVals; o += 256) {
        T v = 0;
#pragma unroll
        for (int w = 0; w < 8; w++) v += red[w * kRowVals + o];
        if (has) {
          const int i = q * kRowVals + o, r = i / share;
          T* dst = CS > 1 ? cluster.map_shared_rank(recv, r) : recv;
          dst[(size_t)ch * share + (i - r * share)] = v;
        }
      }
    }
    __syncthreads();
  }
  // the chunks of this CTA's values, in order
  if (CS > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  for (int j = threadIdx.x; j < share; j += blockDim.x) {
    const int i = rank * share + j;
    if (i >= Q * kRowVals) break;
    const int q = i / kRowVals, o = i - q * kRowVals, rw = o / W, c = o - rw * W, row = 4 * (task.y + (rw & 31)) + (rw >> 5);
    if (row >= m) continue;
    T sum = recv[j];
    if (nch > 1) {
      sum = T(0) + sum;
#pragma unroll 4
      for (int k = 1; k < nch; k++) sum += recv[(size_t)k * share + j];
    }
    const int ch = c0 + q * W + c;
    if (mode == 0) {
      B.y[(long long)(r0 + row) * KP + ch] = sum;
    } else {
      B.xs[(long long)row * KP + ch] = sum;
      x[(long long)B.posGlobal[B.nI + row] * KP + ch] = sum * B.scale[B.nI + row];
    }
  }
}

// The same products with a CTA per chunk of a row group and the chunks' sums in global
// memory; the last CTA of a row group to finish adds them in chunk order.  The same bits.
template <typename T, int W>
__global__ void __launch_bounds__(256, 3) k_bs_chunks(BoundaryDev<T> B, int mode, T* __restrict__ x, int KP, int G) {
  __shared__ T red[8][32][4 * W];
  __shared__ Vec<T, W> vin[kBoundaryChunkMax];
  __shared__ int lastFlag;
  // the block's task, its matrix and its rows of it are set-up data: read (and
  // the rows prefetched into L2) before waiting for the previous launch
  const int4 task = (mode == 0 ? B.subTasks : B.schurTasks)[blockIdx.x];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rq = task.y + lane;
  const int r0 = mode == 0 ? B.subPtr[task.x] : 0;
  const int m = mode == 0 ? B.subPtr[task.x + 1] - r0 : B.nS, mp = (m + 3) & ~3;
  const T* M = mode == 0 ? B.inv + B.invOff[task.x] : B.sinv;
  const int nch = gridDim.y, chunk = blockIdx.y;
  const int clen = (m + nch - 1) / nch, j0 = min(m, chunk * clen), j1 = min(m, j0 + clen);
  {
    // rows j0..j1 of columns 4 task.y .. 4 task.y + 127 (clipped to the padded row)
    const int col0 = 4 * task.y, cols = max(0, min(mp - col0, 128));
    if (lane * 32 < cols * (int)sizeof(T))
      for (int j = j0 + warp; j < j1; j += 8)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(M + (long long)j * mp + col0) + lane * 32));
  }
  grid_dependency_wait();
  grid_launch_dependents();
  const bool active = 4 * rq < m;
  T* part = mode == 0 ? B.subPart : B.schurPart;
  auto store = [&](int row, int off, Vec<T, W> sum) {
    if (mode == 0) {
      vstore<T, W>(B.y + (long long)(r0 + row) * KP + off, sum);
    } else {
      vstore<T, W>(B.xs + (long long)row * KP + off, sum);
      const T sc = B.scale[B.nI + row];
#pragma unroll
      for (int c = 0; c < W; c++) sum.v[c] *= sc;
      vstore<T, W>(x + (long long)B.posGlobal[B.nI + row] * KP + off, sum);
    }
  };
  for (int q = 0; q < G; q++) {
    const int off = q * W;
    // the chunk's input vector (mode 0: the scaled right-hand side from k_bs_prep;
    // mode 1: minus the coupling to the interior solution)
    if (mode == 0) {
      for (int j = j0 + (int)threadIdx.x; j < j1; j += blockDim.x) vin[j - j0] = vload<T, W>(B.rhat + (long long)(r0 + j) * KP + off);
    } else {
      const int lane8 = threadIdx.x & 7, grp = threadIdx.x >> 3;
      for (int jb = j0; jb < j1; jb += 32) {  // 32 groups of 8 lanes
        const int j = jb + grp;
        const Vec<T, W> v = bs_schur_input_group<T, W, LoadDefault>(B, j, j < j1, KP, off, lane8);
        if (j < j1 && lane8 == 0) vin[j - j0] = v;
      }
    }
    __syncthreads();
    T acc[4][W];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int c = 0; c < W; c++) acc[a][c] = 0;
    if (active) {
#pragma unroll 8
      for (int j = j0 + warp; j < j1; j += 8) {
        const Quad<T> mq = *reinterpret_cast<const Quad<T>*>(M + (long long)j * mp + 4 * rq);
        const Vec<T, W> v = vin[j - j0];
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
          for (int c = 0; c < W; c++) acc[a][c] = fma(mq.v[a], v.v[c], acc[a][c]);
      }
    }
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int c = 0; c < W; c++) red[warp][lane][a * W + c] = acc[a][c];
    __syncthreads();
    if (warp == 0 && active) {
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const int row = 4 * rq + a;
        if (row >= m) continue;
        Vec<T, W> sum;
#pragma unroll
        for (int c = 0; c < W; c++) {
          T v = 0;
          for (int w = 0; w < 8; w++) v += red[w][lane][a * W + c];
          sum.v[c] = v;
        }
        if (nch > 1) vstore<T, W>(part + (((long long)blockIdx.x * nch + chunk) * 128 + 4 * lane + a) * KP + off, sum);
        else store(row, off, sum);
      }
    }
    __syncthreads();
  }
  if (nch == 1) return;
  __threadfence();
  __syncthreads();
  int* counter = (mode == 0 ? B.subCount : B.schurCount) + blockIdx.x;
  if (threadIdx.x == 0) {
    const int prev = atomicAdd(counter, 1);
    lastFlag = prev == nch - 1;
    if (lastFlag) *counter = 0;  // ready for the next launch
  }
  __syncthreads();
  if (!lastFlag) return;
  __threadfence();
  for (int it = threadIdx.x; it < 128 * G; it += blockDim.x) {
    const int rt = it / G, q = it - rt * G, row = 4 * task.y + rt, off = q * W;
    if (row >= m) continue;
    Vec<T, W> sum;
#pragma unroll
    for (int c = 0; c < W; c++) sum.v[c] = 0;
#pragma unroll 4
    for (int ch = 0; ch < nch; ch++) {
      const T* src = part + (((long long)blockIdx.x * nch + ch) * 128 + rt) * KP + off;
#pragma unroll
      for (int c = 0; c < W; c++) sum.v[c] += __ldcg(src + c);
    }
    store(row, off, sum);
  }
}

// x_I = s (y - W_p xs[touch_p]) for every interior position (W_p column-major,
// so a warp reads consecutive rows of one column)
template <typename T, int W>
__global__ void __launch_bounds__(256) k_bs_back(BoundaryDev<T> B, T* __restrict__ x, int KP, int G, int yEarly) {
  // bs_back_group's arithmetic.  Before waiting for the previous launch (the
  // separator product, which writes xs): the row's subdomain, its W_p column
  // range and scale (set-up data), and y when yEarly (then y comes from the
  // subdomain product, which the previous launch itself waited for)
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long gi = t >> 3;
  const int lane8 = int(t & 7);
  const long long i = gi / G;
  const int q = int(gi - i * G), off = q * W;
  const bool valid = i < B.nI;
  int m = 0, e0 = 0, e1 = 0;
  const T* Wp = nullptr;
  Vec<T, W> yv;
  T sc = T(0);
  int g = 0;
  if (valid) {
    const int p = B.rowSub[i];
    const int b0 = B.subPtr[p];
    m = B.subPtr[p + 1] - b0;
    Wp = B.wt + B.wOff[p] + (int(i) - b0);
    e0 = B.touchPtr[p];
    e1 = B.touchPtr[p + 1];
    if (lane8 == 0) {
      if (yEarly) yv = vload<T, W>(B.y + i * KP + off);
      sc = B.scale[i];
      g = B.posGlobal[i];
    }
  }
  // the first columns of this lane's part of the row (set-up data)
  constexpr int kAhead = 4;
  T w[kAhead];
  int col[kAhead];
#pragma unroll
  for (int u = 0; u < kAhead; u++) {
    const int e = e0 + lane8 + 8 * u;
    if (e < e1) {
      w[u] = Wp[(long long)(e - e0) * m];
      col[u] = B.touch[e];
    }
  }
  grid_dependency_wait();
  grid_launch_dependents();
  if (valid && lane8 == 0 && !yEarly) yv = vload<T, W>(B.y + i * KP + off);
  Vec<T, W> acc;
#pragma unroll
  for (int c = 0; c < W; c++) acc.v[c] = 0;
  if (valid) {
    Vec<T, W> v[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; u++)
      if (e0 + lane8 + 8 * u < e1) v[u] = vload<T, W>(B.xs + (long long)col[u] * KP + off);
#pragma unroll
    for (int u = 0; u < kAhead; u++)
      if (e0 + lane8 + 8 * u < e1) fma_to(acc, w[u], v[u]);
    // (the columns after those four at a time: with the next columns' loads behind the
    // sums of these, a row of a 1024^2 atlas of 1024 charts, some 100 columns, took 1701 us
    // per step with 3 channels, now 1635)
#pragma unroll 4
    for (int e = e0 + lane8 + 8 * kAhead; e < e1; e += 8) fma_to(acc, Wp[(long long)(e - e0) * m], vload<T, W>(B.xs + (long long)B.touch[e] * KP + off));
  }
  acc = group8_sum(acc);
  if (valid && lane8 == 0) {
#pragma unroll
    for (int c = 0; c < W; c++) yv.v[c] = (yv.v[c] - acc.v[c]) * sc;
    vstore<T, W>(x + (long long)g * KP + off, yv);
  }
}

// rhat = s (rhs - BD x) for every boundary position, 8 lanes per position
template <typename T, int W>
__global__ void __launch_bounds__(256) k_bs_prep(BoundaryDev<T> B, const T* __restrict__ rhs, const T* __restrict__ x, int KP, int G,
                                                 int rhsEarly) {
  // bs_prep_group's arithmetic.  Before waiting for the previous launch: the
  // row's BD range, position and scale (set-up data), and rhs when the previous
  // launch does not write it (rhsEarly: the prolongation before a boundary solve
  // after the coarse correction)
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long gi = t >> 3;
  const int lane8 = int(t & 7);
  const long long k = gi / G;
  const int q = int(gi - k * G), off = q * W;
  const bool valid = k < B.nb;
  int e0 = 0, e1 = 0, g = 0;
  T sc = T(0);
  Vec<T, W> r;
  if (valid) {
    e0 = B.bdPtr[k];
    e1 = B.bdPtr[k + 1];
    if (lane8 == 0) {
      g = B.posGlobal[k];
      sc = B.scale[k];
      if (rhsEarly) r = vload<T, W>(rhs + (long long)g * KP + off);
    }
  }
  // this lane's first entries of the row (set-up data)
  constexpr int kAhead = 2;
  T w[kAhead];
  int col[kAhead];
#pragma unroll
  for (int u = 0; u < kAhead; u++) {
    const int e = e0 + lane8 + 8 * u;
    if (e < e1) {
      w[u] = B.bdVal[e];
      col[u] = B.bdCol[e];
    }
  }
  grid_dependency_wait();
  grid_launch_dependents();
  Vec<T, W> acc, v[kAhead];
#pragma unroll
  for (int c = 0; c < W; c++) acc.v[c] = 0;
#pragma unroll
  for (int u = 0; u < kAhead; u++)
    if (e0 + lane8 + 8 * u < e1) v[u] = vload<T, W>(x + (long long)col[u] * KP + off);
#pragma unroll
  for (int u = 0; u < kAhead; u++)
    if (e0 + lane8 + 8 * u < e1) fma_to(acc, w[u], v[u]);
  for (int e = e0 + lane8 + 8 * kAhead; e < e1; e += 8) fma_to(acc, B.bdVal[e], vload<T, W>(x + (long long)B.bdCol[e] * KP + off));
  acc = group8_sum(acc);
  if (valid && lane8 == 0) {
    if (!rhsEarly) r = vload<T, W>(rhs + (long long)g * KP + off);
#pragma unroll
    for (int c = 0; c < W; c++) r.v[c] = (r.v[c] - acc.v[c]) * sc;
    vstore<T, W>(B.rhat + k * KP + off, r);
  }
}

// L2 prefetch of [p, p + bytes) by the threads of a block (128-byte lines);
// used for set-up matrices before a kernel waits for the previous launch
__device__ __forceinline__ void prefetch_l2_block(const void* p, long long bytes) {
  const char* c = static_cast<const char*>(p);
  for (long long o = (long long)threadIdx.x * 128; o < bytes; o += (long long)blockDim.x * 128)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(c + o));
}

// Sums of N values over the warp's lanes, each in the order of a shuffle-down tree
// (lanes l and l + 16, then l + 8, ...).  While a lane holds several values it keeps
// half of them and hands the other half over, so the whole takes N - 1 + log2(32 / N)
// shuffles (N <= 32), not 5 N.  Afterwards value i is in v[i % own] of lane (i / own)
// lanes, with own = max(1, N / 32) and lanes = max(1, 32 / N).
template <int N>
__device__ __forceinline__ void warp_sums(double (&v)[N], int lane) {
  static_assert(N >= 1 && N <= 64 && (N & (N - 1)) == 0, "a power of two");
#pragma unroll
  for (int step = 0; step < 5; step++) {
    const int s = 16 >> step, half = (N >> step) / 2;
    if (half > 0) {
      const bool upper = lane & s;
#pragma unroll
      for (int i = 0; i < N / 2; i++)
        if (i < half) {
          const double give = upper ? v[i] : v[i + half], keep = upper ? v[i + half] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, give, s);
        }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], s);
    }
  }
}

// ----------------------------------------------------------------------------
// Coarsest level: x = D Ainv^ D rhs with the scaled dense inverse (FP64): a
// stream of the n x n inverse.  A block takes 2 R rows, a warp one part of the
// j range (coarse_part's partition and order, so the same bits) of R rows and Q
// channel groups: a value of the inverse is used for Q W channels, and a
// right-hand side value, widened to FP64 once, for R rows.  What bounds it is
// the loads in flight: a lane loads U of its j at once, before their updates.
// With several channel groups it was the lines that a load touched (a lane's row of
// the right-hand side) and the shuffles of R Q W sums: with the rows staged and
// warp_sums, per refinement step at 1024^2, 64 right-hand sides 2120 -> 2078 us (17 of
// it warp_sums), 32 1096 -> 1075, 16 653 -> 648; 725 x 611 with 15 397 -> 394; up to 4
// no difference.
// ----------------------------------------------------------------------------
template <typename T, int W, int R, int Q, int U>
__global__ void __launch_bounds__(256, Q == 1 ? 2 : 1) k_coarse_solve(int n, const double* __restrict__ ainv, const double* __restrict__ scale,
                                                      const T* __restrict__ rhs, T* __restrict__ x, int KP) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rl = warp / kCoarseParts, p = warp % kCoarseParts;
  const int b0 = blockIdx.x * 2 * R, row0 = b0 + rl * R;
  // this block's rows of the inverse (set-up data) start moving into L2 while
  // the previous launch finishes
  if (b0 < n && blockIdx.y == 0) prefetch_l2_block(ainv + (long long)b0 * n, (long long)min(2 * R, n - b0) * n * sizeof(double));
  grid_dependency_wait();
  grid_launch_dependents();
  __shared__ double part[2][R][kCoarseParts][Q * W];
  const int c0 = blockIdx.y * Q * W;
  const int len = ((n + kCoarseParts - 1) / kCoarseParts + 31) & ~31;
  const int j0 = p * len, j1 = min(n, j0 + len);
  double acc[R][Q * W];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int c = 0; c < Q * W; c++) acc[r][c] = 0;
  const double* arow[R];
#pragma unroll
  for (int r = 0; r < R; r++) arow[r] = ainv + (long long)min(row0 + r, n - 1) * n;  // rows past n: computed, not stored
  if constexpr (Q > 1 && sizeof(T) == 4) {
    // several FP32 channel groups: a chunk of 32 rows of the right-hand side comes in
    // contiguous pieces (a lane reading its whole row touches 32 lines per load), one
    // chunk ahead, and each lane takes its row from shared memory
    constexpr int kRow = Q * W * int(sizeof(T)), kPieces = kRow / 16, kPitch = kRow + 16;
    static_assert(kRow % 16 == 0, "16-byte pieces");
    __shared__ __align__(16) unsigned char stage[8][2][32 * kPitch];
    auto queue = [&](int j, int buf) {  // rows j .. j + 31 below j1
#pragma unroll
      for (int u = 0; u < kPieces; u++) {
        const int e = lane + 32 * u, row = e / kPieces, piece = e % kPieces;
        if (j + row < j1)
          copy_async<16, true>(&stage[warp][buf][row * kPitch + piece * 16],
                               reinterpret_cast<const char*>(rhs + (long long)(j + row) * KP + c0) + piece * 16);
      }
      copies_commit();
    };
    double wn[R], scn = 0;
    auto fetch = [&](int j) {
      if (j < j1) {
#pragma unroll
        for (int r = 0; r < R; r++) wn[r] = __ldg(arow[r] + j);
        scn = scale[j];
      }
    };
    if (j0 < j1) queue(j0, 0);
    fetch(j0 + lane);
    for (int jb = j0, buf = 0; jb < j1; jb += 32, buf ^= 1) {
      const int j = jb + lane;
      double w[R];
#pragma unroll
      for (int r = 0; r < R; r++) w[r] = wn[r] * scn;
      if (jb + 32 < j1) {
        queue(jb + 32, buf ^ 1);
        fetch(j + 32);
        copies_wait<1>();
      } else {
        copies_wait<0>();
      }
      __syncwarp();
      if (j < j1)
#pragma unroll
        for (int q = 0; q < Q; q++) {
          const Vec<T, W> v = *reinterpret_cast<const Vec<T, W>*>(&stage[warp][buf][lane * kPitch + q * W * int(sizeof(T))]);
#pragma unroll
          for (int c = 0; c < W; c++) {
            const double d = double(v.v[c]);
#pragma unroll
            for (int r = 0; r < R; r++) acc[r][q * W + c] = fma(w[r], d, acc[r][q * W + c]);
          }
        }
      __syncwarp();  // before this buffer is filled again
    }
  } else {
    for (int j = j0 + lane; j < j1; j += 32 * U) {
      double w[U][R], sc[U];
      Vec<T, W> v[U][Q];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int ju = j + 32 * u;
        if (ju < j1) {
#pragma unroll
          for (int r = 0; r < R; r++) w[u][r] = __ldg(arow[r] + ju);
          sc[u] = scale[ju];
#pragma unroll
          for (int q = 0; q < Q; q++) v[u][q] = vload<T, W>(rhs + (long long)ju * KP + c0 + q * W);
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++)
        if (j + 32 * u < j1) {
#pragma unroll
          for (int r = 0; r < R; r++) w[u][r] = w[u][r] * sc[u];
#pragma unroll
          for (int q = 0; q < Q; q++)
#pragma unroll
            for (int c = 0; c < W; c++) {
              const double d = double(v[u][q].v[c]);
#pragma unroll
              for (int r = 0; r < R; r++) acc[r][q * W + c] += w[u][r] * d;
            }
        }
    }
  }
  constexpr int kValues = R * Q * W, kOwn = kValues > 32 ? kValues / 32 : 1, kLanes = kValues > 32 ? 1 : 32 / kValues;
  double sums[kValues];
#pragma unroll
  for (int i = 0; i < kValues; i++) sums[i] = acc[i / (Q * W)][i % (Q * W)];
  warp_sums(sums, lane);
  if (lane % kLanes == 0)
#pragma unroll
    for (int u = 0; u < kOwn; u++) {
      const int i = lane / kLanes * kOwn + u;
      part[rl][i / (Q * W)][p][i % (Q * W)] = sums[u];
    }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * R * Q * W; i += blockDim.x) {
    const int rr = i / (Q * W), c = i % (Q * W), row = b0 + rr;
    if (row >= n) continue;
    double sum = 0;
    for (int pp = 0; pp < kCoarseParts; pp++) sum += part[rr / R][rr % R][pp][c];
    x[(long long)row * KP + c0 + c] = T(sum * scale[row]);
  }
}

// ----------------------------------------------------------------------------
// Reduction of the per-block partial sums, in a fixed order: sum c is the sum
// over a tree of 256 thread sums (thread t takes blocks t, t + 256, ...; the
// tree adds t and t + 128, + 64, ... + 1).  Up to kSumWide sums are reduced side
// by side, a block per kSumWide sums.
// It is a chain of latencies over 1184 x 2K doubles, so the loads of a thread
// are issued together, and what used to follow as launches of their own is done
// here: the sums' copy for the host and the flexible-CG scalar.  One block for
// all 2K sums took 57 us at K = 15 and 230 us at K = 64, the blocks here 12 us at
// K = 64.  Reducing in the last block of the kernel that writes the partials
// was measured slower (its fences and arrivals: the operator 77 -> 97 us at
// 2048^2, against 7 us for this launch).
// ----------------------------------------------------------------------------
constexpr int kSumWide = 8;
constexpr int kSumThreads = 256;

// sums [c0, c0 + count) of 2K by a block of kSumThreads threads, into total[]
// (shared) and `sums` / `host` (optional, mapped host memory)
__device__ __forceinline__ void reduce_partials(const double* __restrict__ partials, int nBlocks, int K, int c0, int count, double* sums,
                                                double* host, double (*sh)[kSumThreads], double* total) {
  double s[kSumWide];
#pragma unroll
  for (int c = 0; c < kSumWide; c++) s[c] = 0;
  constexpr int kAhead = 4;
  for (int b = threadIdx.x; b < nBlocks; b += kAhead * kSumThreads) {
    double v[kAhead][kSumWide];
#pragma unroll
    for (int u = 0; u < kAhead; u++)
#pragma unroll
      for (int c = 0; c < kSumWide; c++)
        if (b + u * kSumThreads < nBlocks && c < count) v[u][c] = partials[(long long)(b + u * kSumThreads) * 2 * K + c0 + c];
#pragma unroll
    for (int u = 0; u < kAhead; u++)
#pragma unroll
      for (int c = 0; c < kSumWide; c++)
        if (b + u * kSumThreads < nBlocks && c < count) s[c] += v[u][c];
  }
  // four sums at a time: 256 thread sums -> 32 in shared memory (+128, +64, +32),
  // then one warp's shuffles (+16 ... +1)
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int h = 0; h < kSumWide; h += 4) {
    if (h >= count) break;
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 4; c++) sh[c][threadIdx.x] = s[h + c];
    __syncthreads();
    if (w < 4) {
      const double* a = sh[w];
      double v = ((a[l] + a[l + 128]) + (a[l + 64] + a[l + 192])) + ((a[l + 32] + a[l + 160]) + (a[l + 96] + a[l + 224]));
#pragma unroll
      for (int d = 16; d >= 1; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
      if (l == 0 && h + w < count) {
        total[h + w] = v;
        sums[c0 + h + w] = v;
        if (host) host[c0 + h + w] = v;
      }
    }
  }
  __syncthreads();
}

// beta = -alpha_old (z . q_old) / rho_old (0 on a (re)start, rho_old = 0); rho = z . r
__device__ __forceinline__ void fcg_beta(int K, int c, double rho, double gamma, double* sc) {
  const double rhoOld = sc[3 * K + c];
  sc[K + c] = rhoOld != 0.0 ? -sc[c] * gamma / rhoOld : 0.0;
  sc[2 * K + c] = rho;
  sc[3 * K + c] = rho;
}
// alpha = rho / (p . A p), 0 for frozen right-hand sides
__device__ __forceinline__ void fcg_alpha(int K, int c, double pq, const int* frozen, double* sc) {
  sc[c] = (frozen && frozen[c]) || !(pq > 0) ? 0.0 : sc[2 * K + c] / pq;
}

// scalar: 1 beta and rho, 2 alpha (K <= kSumWide / 2: one block holds every sum)
__global__ void __launch_bounds__(kSumThreads) k_sum_partials(const double* __restrict__ partials, int nBlocks, int K,
                                                             double* __restrict__ sums, double* __restrict__ host, int scalar,
                                                             double* __restrict__ sc, const int* __restrict__ frozen) {
  grid_dependency_wait();
  grid_launch_dependents();
  __shared__ double sh[4][kSumThreads];
  __shared__ double total[kSumWide];
  const int c0 = blockIdx.x * kSumWide;
  reduce_partials(partials, nBlocks, K, c0, min(kSumWide, 2 * K - c0), sums, host, sh, total);
  const int c = threadIdx.x;
  if (scalar == 1 && c < K) fcg_beta(K, c, total[c], total[K + c], sc);
  if (scalar == 2 && c < K) fcg_alpha(K, c, total[c], frozen, sc);
}

// Per-block sums of two per-channel accumulators into partials[block][0..K) and
// [K..2K): lanes l and l^s (s >= G) hold the same channel group, then the warps
// are added in a fixed order (deterministic).  All threads of the block call it.
template <int NCH = 4>
__device__ __forceinline__ void block_partials(double (&ra)[4], double (&rb)[4], int G, int K, double* partials) {
  __shared__ double red[8][2][64];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int ch = 0; ch < NCH; ch++)
    for (int s = 16; s >= G; s >>= 1) {
      ra[ch] += __shfl_xor_sync(0xffffffffu, ra[ch], s);
      rb[ch] += __shfl_xor_sync(0xffffffffu, rb[ch], s);
    }
  if (lane < G)
#pragma unroll
    for (int ch = 0; ch < NCH; ch++)
      if (4 * lane + ch < K) { red[warp][0][4 * lane + ch] = ra[ch]; red[warp][1][4 * lane + ch] = rb[ch]; }
  __syncthreads();
  if ((int)threadIdx.x < K) {
    double a = 0, c = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) { a += red[w][0][threadIdx.x]; c += red[w][1][threadIdx.x]; }
    partials[(long long)blockIdx.x * 2 * K + threadIdx.x] = a;
    partials[(long long)blockIdx.x * 2 * K + K + threadIdx.x] = c;
  }
}

// ----------------------------------------------------------------------------
// FP64 raw operator: res = b - A x (mode 0), y = A x (mode 1), y = A x with
// the partial sums of x . y instead of y . y (mode 2), or res = b for x = 0
// (mode 3: the stencil and x are not read; A 0 sums signed zeros to +0, so
// mode 0 on x = 0 gives these bits) on tight n x K vectors.  Deep rows use 9 raw coefficients per run texel (line runs:
// up to 32 consecutive deep texels of a raster line), boundary rows
// the merged BD/BB CSR.  A thread handles one texel and up to 4 channels
// (group q of G = KP/4 groups, or G = 1 for K = 1).  Per-block sums of res^2
// and b^2 per channel go to `partials` for a deterministic norm reduction.
// ----------------------------------------------------------------------------
// Any K (k_raw_few below for K <= 4).  V4: K is a multiple of 4 and every vector
// 32-byte aligned, so that a thread's 4 channels are one access (as four, each of them
// touched every sector of the warp's texels): per refinement step at 1024^2, 64
// right-hand sides 2077 -> 1954 us, 32 1075 -> 1020, 16 648 -> 620; 725 x 611 with 16
// 405 -> 392.
template <bool V4>
__global__ void __launch_bounds__(256) k_raw_operator(const ColourRun* __restrict__ runs, int nRuns, const double* __restrict__ coef,
                                                      int planeStride, const int* __restrict__ bPtr, const int* __restrict__ bCol,
                                                      const double* __restrict__ bVal, const int* __restrict__ bGlobal, int nB,
                                                      const double* __restrict__ b, const double* __restrict__ x,
                                                      double* __restrict__ out, int K, int G, int mode, double* __restrict__ partials,
                                                      float* __restrict__ out32, int KP) {
  grid_dependency_wait();
  grid_launch_dependents();
  // grid-stride over deep items (runs x 32 x G) then boundary items (rows x G);
  // the stride is a multiple of G, so every thread keeps one channel group q
  const long long nDeepItems = (long long)nRuns * 32 * G, nItems = nDeepItems + (long long)nB * G;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int q = int(t0 % G);
  double rr[4] = {0, 0, 0, 0}, bb[4] = {0, 0, 0, 0};
  auto add = [K](double (&acc)[4], double w, const double* xs, int q) {
    if constexpr (V4) {
      const Vec<double, 4> v = vload<double, 4>(xs);
#pragma unroll
      for (int ch = 0; ch < 4; ch++) acc[ch] = fma(w, v.v[ch], acc[ch]);
    } else {
#pragma unroll
      for (int ch = 0; ch < 4; ch++)
        if (4 * q + ch < K) acc[ch] = fma(w, xs[ch], acc[ch]);
    }
  };
  const bool pad = V4 && 4 * q >= K;  // K need not fill its G groups
  for (long long t = pad && !out32 ? nItems : t0; t < nItems; t += stride) {
    double acc[4] = {0, 0, 0, 0};
    int g = -1;
    if (t < nDeepItems) {
      const long long r = t / (32 * G);
      const int m = int(t - r * 32 * G) / G;
      const ColourRun R = runs[r];
      if (m < R.len && (mode == 3 || pad)) {
        g = R.pos0 + m;
      } else if (m < R.len) {  // line runs: consecutive texels
        const int pos = R.pos0 + m, pp = R.prev0 + m, pn = R.next0 + m;
        const double* c = coef + R.coef0 + m;
        const int nb[9] = {pp - 1, pp, pp + 1, pos - 1, pos, pos + 1, pn - 1, pn, pn + 1};
#pragma unroll
        for (int s = 0; s < 9; s++) {
          const double w = c[s * planeStride];
          add(acc, w, x + (long long)nb[s] * K + 4 * q, q);
        }
        g = pos;
      }
    } else {
      const long long row = (t - nDeepItems) / G;
      for (int k = mode == 3 || pad ? bPtr[row + 1] : bPtr[row]; k < bPtr[row + 1]; k++) {
        const double w = bVal[k];
        add(acc, w, x + (long long)bCol[k] * K + 4 * q, q);
      }
      g = bGlobal[row];
    }
    if (V4 && pad) {
      if (g >= 0 && 4 * q < KP) vstore<float, 4>(out32 + (long long)g * KP + 4 * q, Vec<float, 4>{});
    } else if (V4 && g >= 0) {
      const long long at = (long long)g * K + 4 * q;
      Vec<double, 4> bv, xc, v;
#pragma unroll
      for (int ch = 0; ch < 4; ch++) bv.v[ch] = xc.v[ch] = 0.0;
      if (b) bv = vload<double, 4>(b + at);
      if (mode == 2) xc = vload<double, 4>(x + at);
      Vec<float, 4> f;
#pragma unroll
      for (int ch = 0; ch < 4; ch++) {
        v.v[ch] = (mode == 0 || mode == 3) ? bv.v[ch] - acc[ch] : acc[ch];
        f.v[ch] = float(v.v[ch]);
        rr[ch] += mode == 2 ? xc.v[ch] * v.v[ch] : v.v[ch] * v.v[ch];  // mode 2: x . A x
        bb[ch] += bv.v[ch] * bv.v[ch];
      }
      if (out32) vstore<float, 4>(out32 + (long long)g * KP + 4 * q, f);
      else vstore<double, 4>(out + at, v);
    } else if (g >= 0) {
#pragma unroll
      for (int ch = 0; ch < 4; ch++) {
        const int c = 4 * q + ch;
        if (c >= K) continue;
        const double bv = b ? b[(long long)g * K + c] : 0.0;
        const double v = (mode == 0 || mode == 3) ? bv - acc[ch] : acc[ch];
        if (out32) out32[(long long)g * KP + c] = float(v);
        else out[(long long)g * K + c] = v;
        rr[ch] += mode == 2 ? x[(long long)g * K + c] * v : v * v;  // mode 2: x . A x
        bb[ch] += bv * bv;
      }
      if (out32)  // zero the padding channels of this group
        for (int c = max(K, 4 * q); c < min(KP, 4 * q + 4); c++) out32[(long long)g * KP + c] = 0.f;
    }
  }
  if (!partials) return;
  block_partials(rr, bb, G, K, partials);
}

// The same for K = KT <= 4 right-hand sides.
//  * A warp takes a run, its header loaded during the run before.
//  * Boundary rows come before the deep rows, whose loads hide their trips.  A warp takes 4
//    of them (FEW: at most kRawRowsFew, one pass of the chip) or 32, the warps dealt to the
//    blocks in turn, since blocks that are launched early share few SMs (rows in the first
//    blocks: 42.5 instead of 19 us at 1024^2).  The threads that add a row to the norms are
//    the same for every KT: so are the norms, whatever is solved together.  One right-hand
//    side of few rows takes 8 lanes a row with the first entries loaded ahead; with more,
//    handing the terms round costs more than the trips it saves.  Per step, 8 lanes always
//    / now: 3 right-hand sides, 256^2 torus 115.5 / 110 us, 1013 x 1187 genus-2 170.6 / 167,
//    icospheres of 28 k rows 277.8 / 276.2, of 60 k 632 / 617, 16 x 16 charts of 123 k rows 631
//    / 591; one, 256^2 torus 85.5 / 83.8, 640 x 480 183.8 / 185.6, 16 x 16 charts 467 / 452 (a
//    thread per row also where there are few: genus-2 of 15 k rows 134.2 / 135.5, of 29 k
//    197 / 200.8).
// What bounds it at 2048^2 (65 us for 203 MB; read when every row ran on 8 lanes, 77 us):
// half the warps (64 registers), each a long-scoreboard wait of 10.6 of 17.9 cycles per
// issue, and 58 % of the first-level cache's cycles; a lane per value instead of per texel
// (consecutive addresses, but the coefficients read for every channel) took 85 us.
template <int KT, bool FEW>
__global__ void __launch_bounds__(256, 4) k_raw_few(const ColourRun* __restrict__ runs, int nRuns, const double* __restrict__ coef,
                                                    int planeStride, const int* __restrict__ bPtr, const int* __restrict__ bCol,
                                                    const double* __restrict__ bVal, const int* __restrict__ bGlobal, int nB,
                                                    const double* __restrict__ b, const double* __restrict__ x, double* __restrict__ out,
                                                    int mode, double* __restrict__ partials, float* __restrict__ out32, int KP) {
  const int lane = threadIdx.x & 31;
  const int warp0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = (gridDim.x * blockDim.x) >> 5;
  double rr[4] = {0, 0, 0, 0}, bb[4] = {0, 0, 0, 0};
  // row g: its value from the sums, its share of the norms
  auto finish = [&](int g, const double (&acc)[KT]) {
#pragma unroll
    for (int ch = 0; ch < KT; ch++) {
      const double bv = b ? b[(long long)g * KT + ch] : 0.0;
      const double v = (mode == 0 || mode == 3) ? bv - acc[ch] : acc[ch];
      if (out32) out32[(long long)g * KP + ch] = float(v);
      else out[(long long)g * KT + ch] = v;
      rr[ch] += mode == 2 ? x[(long long)g * KT + ch] * v : v * v;  // mode 2: x . A x
      bb[ch] += bv * bv;
    }
    if (out32)  // zero the padding channels
      for (int c = KT; c < KP; c++) out32[(long long)g * KP + c] = 0.f;
  };
  const int rowWarp = blockIdx.x + gridDim.x * (threadIdx.x >> 5);
  if constexpr (FEW && KT == 1) {
    const int lane8 = lane & 7;
    int row = rowWarp * 4 + (lane >> 3), k0, k1, g;
    auto range = [&] {
      const bool valid = row < nB;
      g = valid ? bGlobal[row] : 0;
      k0 = valid && mode != 3 ? bPtr[row] : 0;
      k1 = valid && mode != 3 ? bPtr[row + 1] : 0;
    };
    range();
    OrderedRow8<double, KT, 2> entries(bCol, bVal, k0, k1, lane8);
    grid_dependency_wait();
    grid_launch_dependents();
    for (int first = rowWarp * 4; first < nB; first += warps * 4) {
      Vec<double, KT> acc;
      acc.v[0] = 0;
      entries.add_to(acc, false, bCol, bVal, lane8, [&](int c) {
        Vec<double, KT> v;
        v.v[0] = x[c];
        return v;
      });
      if (row < nB && lane8 == 0) finish(g, acc.v);
      row += warps * 4;
      range();
      entries = OrderedRow8<double, KT, 2>(bCol, bVal, k0, k1, lane8);
    }
  } else {
    grid_dependency_wait();
    grid_launch_dependents();
    if (!FEW || (lane & 7) == 0)
      for (int row = FEW ? rowWarp * 4 + (lane >> 3) : rowWarp * 32 + lane; row < nB; row += warps * (FEW ? 4 : 32)) {
        double acc[KT];
#pragma unroll
        for (int ch = 0; ch < KT; ch++) acc[ch] = 0;
        for (int k = mode == 3 ? bPtr[row + 1] : bPtr[row]; k < bPtr[row + 1]; k++) {
          const double w = bVal[k];
          const double* xs = x + (long long)bCol[k] * KT;
#pragma unroll
          for (int ch = 0; ch < KT; ch++) acc[ch] = fma(w, xs[ch], acc[ch]);
        }
        finish(bGlobal[row], acc);
      }
  }
  ColourRun R;
  R.len = 0;
  if (warp0 < nRuns) R = runs[warp0];
  for (int r = warp0; r < nRuns; r += warps) {
    ColourRun next;
    next.len = 0;
    if (r + warps < nRuns) next = runs[r + warps];  // on its way during this run
    if (lane < R.len) {
      double acc[KT];
#pragma unroll
      for (int ch = 0; ch < KT; ch++) acc[ch] = 0;
      const int pos = R.pos0 + lane;
      if (mode != 3) {
        const double* c = coef + R.coef0 + lane;
        const int nb[3] = {R.prev0 + lane, pos, R.next0 + lane};
#pragma unroll
        for (int k = 0; k < 9; k++) {
          const double w = c[k * planeStride];
          const double* xs = x + (long long)(nb[k / 3] + k % 3 - 1) * KT;
#pragma unroll
          for (int ch = 0; ch < KT; ch++) acc[ch] = fma(w, xs[ch], acc[ch]);
        }
      }
      finish(pos, acc);
    }
    R = next;
  }
  if (!partials) return;
  block_partials<KT>(rr, bb, 1, KT, partials);
}

// The solve loops' per-right-hand-side flags come in as a kernel argument (and
// the norms go out through mapped pinned host memory, SumTarget::host): small
// exchanges kept off the copy engines, which a streaming solve keeps busy with
// whole vectors.
__global__ void k_set_flags(int* __restrict__ flags, unsigned long long mask, int k) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int c = threadIdx.x;
  if (c < k) flags[c] = int((mask >> c) & 1ull);
}

// ----------------------------------------------------------------------------
// Flexible preconditioned conjugate gradients around the FP32 V-cycle (FP64
// vectors, tight n x K; per right-hand side scalars in `sc`: alpha [0,K),
// beta [K,2K), rho [2K,3K), previous rho [3K,4K)).  Items are texels x channel
// groups of 4 over a fixed grid, so the partial sums have a fixed order.
// ----------------------------------------------------------------------------
// z = e (V-cycle output, FP32 padded), e cleared; partials: z . r and z . q
__global__ void __launch_bounds__(256) k_fcg_precond(long long n, int K, int KP, int G, float* __restrict__ e,
                                                     const double* __restrict__ r, const double* __restrict__ q,
                                                     double* __restrict__ z, double* __restrict__ partials) {
  grid_dependency_wait();
  grid_launch_dependents();
  const long long stride = (long long)gridDim.x * blockDim.x, t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int qg = int(t0 % G);
  double a[4] = {0, 0, 0, 0}, b[4] = {0, 0, 0, 0};
  for (long long t = t0; t < n * G; t += stride) {
    const long long i = t / G;
#pragma unroll
    for (int ch = 0; ch < 4; ch++) {
      const int c = 4 * qg + ch;
      if (c >= K) continue;
      const double v = double(e[i * KP + c]);
      e[i * KP + c] = 0.f;
      z[i * K + c] = v;
      a[ch] += v * r[i * K + c];
      b[ch] += v * q[i * K + c];
    }
  }
  block_partials(a, b, G, K, partials);
}

// the scalars as launches of their own (more right-hand sides than one block sums)
__global__ void k_fcg_beta(int K, const double* __restrict__ sums, double* __restrict__ sc) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int c = threadIdx.x;
  if (c < K) fcg_beta(K, c, sums[c], sums[K + c], sc);
}

// p = z + beta p
__global__ void __launch_bounds__(256) k_fcg_direction(long long n, int K, const double* __restrict__ z, const double* __restrict__ sc,
                                                       double* __restrict__ p) {
  grid_dependency_wait();
  grid_launch_dependents();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * K) return;
  const int c = int(t % K);
  p[t] = z[t] + sc[K + c] * p[t];
}

__global__ void k_fcg_alpha(int K, const double* __restrict__ sums, const int* __restrict__ frozen, double* __restrict__ sc) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int c = threadIdx.x;
  if (c < K) fcg_alpha(K, c, sums[c], frozen, sc);
}

// x += alpha p, r -= alpha q, r packed into the next V-cycle's FP32 right-hand
// side; partials: r . r and 0
__global__ void __launch_bounds__(256) k_fcg_update(long long n, int K, int KP, int G, const double* __restrict__ sc,
                                                    const double* __restrict__ p, const double* __restrict__ q, double* __restrict__ x,
                                                    double* __restrict__ r, float* __restrict__ rhs32, double* __restrict__ partials) {
  grid_dependency_wait();
  grid_launch_dependents();
  const long long stride = (long long)gridDim.x * blockDim.x, t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int qg = int(t0 % G);
  double a[4] = {0, 0, 0, 0}, b[4] = {0, 0, 0, 0};
  for (long long t = t0; t < n * G; t += stride) {
    const long long i = t / G;
#pragma unroll
    for (int ch = 0; ch < 4; ch++) {
      const int c = 4 * qg + ch;
      if (c >= K) continue;
      const double al = sc[c];
      x[i * K + c] += al * p[i * K + c];
      const double rv = r[i * K + c] - al * q[i * K + c];
      r[i * K + c] = rv;
      rhs32[i * KP + c] = float(rv);
      a[ch] += rv * rv;
    }
  }
  block_partials(a, b, G, K, partials);
}

// out = a x + b y (the system operator's planes from the mass and stiffness planes)
__global__ void k_axpby(double* __restrict__ out, double a, const double* __restrict__ x, double b, const double* __restrict__ y,
                        long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = a * x[i] + b * y[i];
}

// n*K, tight -> n*KP, padded with zeros: the FP64 residual as a right-hand side, or
// the caller's vectors
template <typename S, typename T>
__global__ void k_pack(const S* __restrict__ r, T* __restrict__ rhs, long long n, int K, int KP) {
  grid_dependency_wait();
  grid_launch_dependents();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * KP) return;
  const long long i = t / KP;
  const int c = int(t - i * KP);
  rhs[t] = c < K ? T(r[i * K + c]) : T(0);
}
template <typename T>
__global__ void k_unpack(const T* __restrict__ padded, T* __restrict__ tight, long long n, int K, int KP) {
  grid_dependency_wait();
  grid_launch_dependents();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * K) return;
  const long long i = t / K;
  tight[t] = padded[i * KP + (t - i * K)];
}
// x64 += e (padded FP32/FP64 correction); e is cleared for the next V-cycle
// (its padding lanes stay zero through the V-cycle).  Columns with frozen[c]
// set keep their x: a right-hand side that has converged stops changing, so
// its result does not depend on what it was solved together with.
// PER values per thread, their loads issued together, and 32-bit divisions (small:
// n K < 2^32).  Four values where that still fills the chip: per refinement step 64
// right-hand sides at 1024^2 1961 -> 1942 us, 16 623 -> 617, 2048^2 644 -> 640.5, FP64
// values at 1024^2 392.6 -> 388; one below (256^2 torus 116.2, with four 116.8).
template <typename T, int PER>
__global__ void __launch_bounds__(256) k_add_correction(double* __restrict__ x, T* __restrict__ e, long long n, int K, int KP,
                                                        const int* __restrict__ frozen, int small) {
  grid_dependency_wait();
  grid_launch_dependents();
  const long long t0 = (long long)blockIdx.x * (256 * PER) + threadIdx.x, total = n * K;
  double xv[PER];
  T ev[PER];
  long long at[PER];
  bool go[PER];
#pragma unroll
  for (int u = 0; u < PER; u++) {
    const long long t = t0 + 256 * u;
    go[u] = false;
    if (t >= total) continue;
    const long long i = small ? (long long)((unsigned)t / (unsigned)K) : t / K;
    const int c = int(t - i * K);
    at[u] = i * KP + c;
    go[u] = !frozen || !frozen[c];
    if (go[u]) {
      xv[u] = x[t];
      ev[u] = e[at[u]];
    }
  }
#pragma unroll
  for (int u = 0; u < PER; u++) {
    const long long t = t0 + 256 * u;
    if (t >= total) continue;
    if (go[u]) x[t] = xv[u] + double(ev[u]);
    e[at[u]] = T(0);
  }
}

// ----------------------------------------------------------------------------
// launch wrappers
// ----------------------------------------------------------------------------
static inline int nblk(long long threads) { return int((threads + 255) / 256); }

static bool g_programmatic = true;
void set_programmatic_launch(bool on) { g_programmatic = on; }
bool programmatic_launch() { return g_programmatic; }
int device_sms() {
  static std::atomic<int> slots[kMaxDevices];
  static const bool init = [] {
    for (auto& a : slots) a.store(kUnset);
    return true;
  }();
  (void)init;
  return per_device_once(slots, [] {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return sms;
  });
}

// Every V-cycle kernel is launched with programmatic stream serialization:
// inside a captured graph consecutive kernels get programmatic edges, so a
// kernel is scheduled while its predecessor drains (each kernel waits in
// grid_dependency_wait() before touching memory).
template <typename... P, typename... A>
static void launch(void (*kernel)(P...), dim3 grid, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_programmatic ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <typename T, int W>
void launch_gs_colour(const ColourRun* runs, int nRuns, const T* coef, int planeStride, const T* rhs, T* x, int KP,
                      cudaStream_t s, int skip, bool rhsEarly) {
  if (nRuns == 0) return;
  const int G = KP / W;
  launch(k_gs_colour<T, W>, dim3(nblk((long long)nRuns * 32 * G)), s, runs, nRuns, coef, planeStride, rhs, x, KP, G, skip,
         rhsEarly ? 1 : 0);
}
template <typename T, int W>
size_t gs_rows_smem(const LevelDev<T>& D) {
  return size_t(3) * D.rowSlots * sizeof(Vec<T, W>);  // three rows
}
// The row smoother's shared memory fits this device (its attribute set): 1, else 0.
template <typename T, int W, int BS>
static int gs_rows_ready() {
  static std::atomic<int> slots[kMaxDevices];
  static const bool init = [] {
    for (auto& v : slots) v.store(kUnset);
    return true;
  }();
  (void)init;
  return per_device_once(slots, [] {
    const int smem = int(3 * row_slot_cap(BS) * sizeof(Vec<T, W>));
    if (cudaFuncSetAttribute(k_gs_rows<T, W, BS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return 1;
  });
}
template <typename T, int W, int BS>
static bool launch_gs_rows_bs(const LevelDev<T>& D, int rows, bool oddFirst, int KP, cudaStream_t s, int skip, bool rhsEarly) {
  if (gs_rows_ready<T, W, BS>() <= 0) return false;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(D.nRowBins[rows]), unsigned(KP / W));
  cfg.blockDim = dim3(BS);
  cfg.dynamicSmemBytes = gs_rows_smem<T, W>(D);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = g_programmatic ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k_gs_rows<T, W, BS>, D.rowLines[rows], D.rowLineOf[rows], D.coef, D.planeStride,
                     static_cast<const T*>(D.b), D.x, KP, D.rowSlots, oddFirst ? 1 : 0, skip, rhsEarly ? 1 : 0);
  return true;
}
template <typename T, int W>
bool gs_rows_available(const LevelDev<T>& D) {
  if (D.rowBlock == 256) return gs_rows_ready<T, W, 256>() > 0;
  if (D.rowBlock == 512) return gs_rows_ready<T, W, 512>() > 0;
  if (D.rowBlock == 1024) return gs_rows_ready<T, W, 1024>() > 0;
  return false;
}
template <typename T, int W>
bool launch_gs_rows(const LevelDev<T>& D, int rows, bool oddFirst, int KP, cudaStream_t s, int skip, bool rhsEarly) {
  if (D.nRowBins[rows] == 0) return true;
  if (D.rowBlock == 256) return launch_gs_rows_bs<T, W, 256>(D, rows, oddFirst, KP, s, skip, rhsEarly);
  if (D.rowBlock == 512) return launch_gs_rows_bs<T, W, 512>(D, rows, oddFirst, KP, s, skip, rhsEarly);
  if (D.rowBlock == 1024) return launch_gs_rows_bs<T, W, 1024>(D, rows, oddFirst, KP, s, skip, rhsEarly);
  return false;
}
template <typename T, int W>
size_t gs_groups_smem(const LevelDev<T>& D, int KP) {
  return size_t(D.maxGroupSpan) * KP * sizeof(T);
}
template <typename T, int W>
bool launch_gs_groups(const LevelDev<T>& D, int sweeps, bool reverse, int KP, cudaStream_t s) {
  if (D.nGroups == 0 || sweeps <= 0) return true;
  const size_t smem = gs_groups_smem<T, W>(D, KP);
  if (smem > kGroupSmemMax) return false;
  static std::atomic<int> attr[kMaxDevices];
  static const bool init = [] {
    for (auto& a : attr) a.store(kUnset);
    return true;
  }();
  (void)init;
  const int ok = per_device_once(attr, [] {
    return cudaFuncSetAttribute(k_gs_groups<T, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kGroupSmemMax)) == cudaSuccess ? 1
                                                                                                                              : 0;
  });
  if (!ok) return false;
  const int G = KP / W;
  // threads: the largest colour pass of a chart, in warps, at most 1024
  const int items = 32 * G * std::max(1, (D.maxGroupDeep / 4 + 31) / 32 + 1);
  const int nt = std::min(kGroupBlockMax, std::max(128, (items + 31) / 32 * 32));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(D.nGroups);
  cfg.blockDim = dim3(nt);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = g_programmatic ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k_gs_groups<T, W>, D.runs, D.groups, (const T*)D.coef, D.planeStride, (const T*)D.b, D.x, KP, G,
                            sweeps, reverse ? 1 : 0) == cudaSuccess;
}
// Lanes per boundary row of the residual and the restriction: 8 for one channel group
// (a row one term after another was the launch's time: residual and restriction of a
// 256^2 torus 4.7 and 3.9 us, 140 -> 152 us per step without the 8 lanes for a 1013 x 1187
// genus-2), as long as the rows do not fill the chip by themselves: 8 lanes hand every
// term round, (1 + W) words of it, so `limit` is in rows times words.  With several groups
// the threads of a row's groups read its texels' values contiguously.  Per step, 8 lanes
// everywhere / the residual's rows on one: 28 k rows of 4 floats 279 / 292 us, 60 k 633 / 631,
// 123 k 625 / 617, 229 k 1709 / 1686, of 4 doubles 2766 / 2736; the restriction's on one: 60 k
// 633 / 643, 229 k 1709 / 1707, of 4 doubles 2766 / 2711.  With the operator's rows
// (k_raw_few): 1024^2 of 1024 charts, 3 channels 1755 -> 1689 us, 256 charts 631 -> 591, 64
// charts 491 -> 479, 2048^2 icosphere 632 -> 617.
constexpr long long kResidualRows8 = 200000, kRestrictRows8 = 1200000;
template <typename T, int W>
static int row_lanes(int nB, int G, long long limit) {
  return G == 1 && nB * (1 + W) * (long long)sizeof(T) / 4 <= limit ? 8 : 1;
}
template <typename T, int W>
void launch_residual(const ColourRun* runs, int nRuns, const T* coef, int planeStride, const int* bPtr, const int* bCol,
                     const T* bVal, const int* bGlobal, int nB, const T* rhs, const T* x, T* res, int KP, cudaStream_t s,
                     bool rhsEarly) {
  const int G = KP / W;
  const int lanes = row_lanes<T, W>(nB, G, kResidualRows8), db = nblk((long long)nRuns * 32 * G), bb = nblk((long long)nB * G * lanes);
  if (db + bb == 0) return;
  launch(k_residual<T, W>, dim3(db + bb), s, runs, nRuns, coef, planeStride, db, bPtr, bCol, bVal, bGlobal, nB, rhs, x, res, KP, G,
         rhsEarly ? 1 : 0, lanes);
}
template <typename T, int W>
void launch_restrict(const RestrictRun* runs, int nRuns, const int* rPtr, const int* rCol, const T* rVal, const int* rOut,
                     int nB, const T* res, T* coarseRhs, T* coarseX, long long coarseTexels, int KP, cudaStream_t s) {
  const int G = KP / W;
  const int lanes = row_lanes<T, W>(nB, G, kRestrictRows8), db = nblk((long long)nRuns * 32 * G), bb = nblk((long long)nB * G * lanes);
  if (db + bb == 0 && coarseTexels == 0) return;
  launch(k_restrict<T, W>, dim3(std::max(1, db + bb)), s, runs, nRuns, db, rPtr, rCol, rVal, rOut, nB, res, coarseRhs, coarseX,
         coarseTexels * KP, KP, G, lanes);
}
template <typename T, int W>
void launch_prolong_add(const ProlongRun* runs, int nRuns, const T* coarse, T* fine, int KP, cudaStream_t s) {
  if (nRuns == 0) return;
  const int G = KP / W;
  launch(k_prolong_add<T, W>, dim3(nblk((long long)nRuns * 32 * G)), s, runs, nRuns, coarse, fine, KP, G);
}
// One dense product of the boundary solve (mode 0: subdomains, 1: separator) on clusters.
// Channel groups per CTA: as many as the registers hold (a matrix value read once
// for them); warp groups per CTA: one per chunk while the registers last.
template <typename T, int W, int Q, int mode>
struct BsDense {
  int nch, tasks, CS, groups, clen;
  unsigned z;
  size_t smem;
  BsDense(const BoundaryDev<T>& B, int KP)
      : nch(mode == 0 ? B.subChunks : B.schurChunks), tasks(mode == 0 ? B.nSubTasks : B.nSchurTasks), z(unsigned(KP / W / Q)) {
    CS = std::min(kBsClusterMax, nch);
    groups = std::min(bs_dense_threads<T>(Q, mode) / 256, (nch + CS - 1) / CS);
    clen = ((mode == 0 ? kBoundaryChunkMax : B.nS) + nch - 1) / nch;
    smem = size_t(groups) * Q * clen * sizeof(Vec<T, W>) + size_t(groups) * 8 * 128 * W * sizeof(T) +
           size_t(nch) * ((Q * 128 * W + CS - 1) / CS) * sizeof(T);
  }
  static bool ready() {
    static std::atomic<int> attr[kMaxDevices];
    static const bool init = [] {
      for (auto& a : attr) a.store(kUnset);
      return true;
    }();
    (void)init;
    return per_device_once(attr, [] {
             return cudaFuncSetAttribute(k_bs_dense<T, W, Q, mode>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kBsDenseSmemMax)) ==
                            cudaSuccess
                        ? 1
                        : 0;
           }) != 0;
  }
  bool fits() const { return smem <= kBsDenseSmemMax && ready(); }
  void config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&at)[2], cudaStream_t s) const {
    cfg.gridDim = dim3(unsigned(tasks), unsigned(CS), z);
    cfg.blockDim = dim3(unsigned(256 * groups));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {1, unsigned(CS), 1};
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = g_programmatic ? 2 : 1;
  }
  // clusters of this launch that run at the same time (0: none can)
  int resident() const {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    config(cfg, at, nullptr);
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k_bs_dense<T, W, Q, mode>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return clusters;
  }
  bool launch(const BoundaryDev<T>& B, T* x, int KP, cudaStream_t s) const {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    config(cfg, at, s);
    return cudaLaunchKernelEx(&cfg, k_bs_dense<T, W, Q, mode>, B, nch, clen, x, KP) == cudaSuccess;
  }
};
// f(the variant for this width); false where none fits
template <typename T, int W, int mode, typename F>
static bool bs_dense_variant(const BoundaryDev<T>& B, int KP, const F& f) {
  if constexpr (W > 1) {
    const int G = KP / W;
    if constexpr (sizeof(T) == 4)
      if (const BsDense<T, W, 4, mode> d(B, KP); G % 4 == 0 && d.fits()) return f(d, 4);
    if (const BsDense<T, W, 2, mode> d(B, KP); G % 2 == 0 && d.fits()) return f(d, 2);
  }
  const BsDense<T, W, 1, mode> d(B, KP);
  return d.fits() && f(d, 1);
}
// On clusters: the subdomains' product where a row group has several chunks or a CTA
// several channel groups; the separator's where its clusters of one channel group set are
// resident together (15 at 8 CTAs: up to some 1900 rows).  Beyond, a CTA per chunk with
// three CTAs an SM and 8 rows ahead keeps more of the matrix in flight than the clusters'
// one or two.  Measured without overlap, FP32 of 4 channels, clusters / a CTA per chunk:
//   separator    1228 rows 14.6 / 15.8 us, 1919 16.4 / 18.3, 2550 39 / 24, 4347 105 / 41,
//                12017 594 / 254; 16 channels 1228 28.9 / 38.7, 2550 76 / 57, 12017 1240 / 715
//   subdomains   112 row groups (3 chunks) 11.2 / 12.4, 263 (2) 17.6 / 19.2, 366 (1) 25.3 /
//                16.6, 1851 (1) 86.7 / 69.7; 16 channels 450 (1) 42.4 / 41.0, 1851 139 / 178
// Per refinement step, a 1024^2 atlas of 1024 charts, 1 / 3 / 9 channels: 2278 -> 1477, 2740
// -> 1777, 6716 -> 5078 us, FP64 values 3880 -> 2898; 256 charts 756 -> 639; 2048^2
// icosphere 640 -> 631.
template <typename T, int W>
bool bs_dense_on_clusters(const BoundaryDev<T>& B, int KP, int mode) {
  auto rule = [mode](const auto& d, int Q) { return mode == 0 ? (d.nch > 1 || Q > 1) && d.resident() > 0 : d.tasks <= d.resident(); };
  return mode == 0 ? bs_dense_variant<T, W, 0>(B, KP, rule) : bs_dense_variant<T, W, 1>(B, KP, rule);
}
template <typename T, int W, int mode>
static void launch_bs_dense(const BoundaryDev<T>& B, T* x, int KP, cudaStream_t s) {
  const int tasks = mode == 0 ? B.nSubTasks : B.nSchurTasks, nch = mode == 0 ? B.subChunks : B.schurChunks;
  if (mode == 0 ? B.subPart : B.schurPart)
    launch(k_bs_chunks<T, W>, dim3(tasks, nch), s, B, mode, x, KP, KP / W);
  else
    bs_dense_variant<T, W, mode>(B, KP, [&](const auto& d, int) { return d.launch(B, x, KP, s); });
}
template <typename T, int W>
void launch_boundary_solve(const BoundaryDev<T>& B, const T* rhs, T* x, int KP, cudaStream_t s, bool rhsEarly) {
  if (B.nb == 0) return;
  const int G = KP / W;
  launch(k_bs_prep<T, W>, dim3(nblk((long long)B.nb * G * 8)), s, B, rhs, x, KP, G, rhsEarly ? 1 : 0);
  if (B.nSubTasks > 0) launch_bs_dense<T, W, 0>(B, x, KP, s);
  if (B.nS > 0) launch_bs_dense<T, W, 1>(B, x, KP, s);
  // y comes from the subdomain product: read early only when the separator
  // product sits between the two launches
  if (B.nI > 0) launch(k_bs_back<T, W>, dim3(nblk((long long)B.nI * G * 8)), s, B, x, KP, G, B.nS > 0 ? 1 : 0);
}
// Rows per warp R and channel groups per warp Q.  One group: the fewest rows that
// fit the blocks on one wave of two per SM, so that a small level's rows spread and
// a large one reuses the right-hand side (n = 2316: 14.9 us with R = 4, 17.5 with
// R = 2 in 1.3 waves, 21.8 with R = 8 and fewer loads in flight, 23.6 before, a
// warp per part of one row; n = 1024, R = 2: 5.0 us, 5.8 before).  Several groups:
// the inverse read once for up to 4 (n = 2219, 16 groups: 152 us with R = Q = 4,
// 187 with R = 2 and twice the loads ahead, 423 before, a read per group).
template <typename T, int W>
void launch_coarse_solve(int n, const double* ainv, const double* scale, const T* rhs, T* x, int KP, cudaStream_t s) {
  if (n == 0) return;
  const int G = KP / W;
  auto go = [&](auto kernel, int R, int Q) { launch(kernel, dim3((n + 2 * R - 1) / (2 * R), G / Q), s, n, ainv, scale, rhs, x, KP); };
  if constexpr (W > 1) {
    if (G % 4 == 0) return go(k_coarse_solve<T, W, 4, 4, 1>, 4, 4);
    if (G % 2 == 0) return go(k_coarse_solve<T, W, 2, 2, 4>, 2, 2);
  }
  const int wave = 2 * device_sms();
  if (n <= 2 * wave) return go(k_coarse_solve<T, W, 1, 1, 4>, 1, 1);
  if (n <= 4 * wave) return go(k_coarse_solve<T, W, 2, 1, 4>, 2, 1);
  go(k_coarse_solve<T, W, 4, 1, 4>, 4, 1);
}

static inline int raw_groups(int K) { int G = 1; while (4 * G < K) G *= 2; return G; }
// fixed grid (grid-stride): bounded number of partial sums, launch-shape-independent order
// Fixed grid of the FP64 operator and its reductions: 8 blocks per SM of the
// device (its partial sums are added in block order, so one device always gives
// the same bits), at most kRawMaxBlocks.
static int raw_blocks() {
  const int sms = device_sms();
  return sms > 0 ? std::min(kRawMaxBlocks, 8 * sms) : kRawMaxBlocks;
}
// The 2K sums of a launch of `blocks` blocks; scalar: true when the reduction
// evaluated it too (it holds every sum in one block)
static bool launch_sums(const SumTarget& t, int blocks, int K, cudaStream_t s, int scalar = 0, double* sc = nullptr,
                        const int* frozen = nullptr) {
  const bool one = 2 * K <= kSumWide;
  launch(k_sum_partials, dim3((2 * K + kSumWide - 1) / kSumWide), s, (const double*)t.partials, blocks, K, t.sums, t.host, one ? scalar : 0,
         sc, frozen);
  return one;
}
// Launches the operator for K right-hand sides; returns its blocks (a grid of at
// most 8 per SM).  K <= 4 against the kernel for any K, per step: LIC on a 1024^2
// genus-2 134 -> 129 us, its filtering at 1013 x 1187 140 -> 134, 1024^2 icosphere 307
// -> 303; half the blocks (one wave) 127, 136 and 306.
constexpr int kRawRowsFew = 32000;
static int launch_raw(const ColourRun* runs, int nRuns, const double* coef, int planeStride, const int* bPtr, const int* bCol,
                      const double* bVal, const int* bGlobal, int nB, const double* b, const double* x, double* out, int K, int mode,
                      double* partials, float* out32, int KP, cudaStream_t s) {
  const int G = raw_groups(K);
  if (K > 4) {
    const int blocks = int(std::min<long long>(raw_blocks(), nblk((long long)nRuns * 32 * G + (long long)nB * G)));
    auto aligned = [](const void* p, size_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; };
    auto go = [&](auto kernel) {
      launch(kernel, dim3(blocks), s, runs, nRuns, coef, planeStride, bPtr, bCol, bVal, bGlobal, nB, b, x, out, K, G, mode, partials, out32, KP);
    };
    if (K % 4 == 0 && aligned(b, 32) && aligned(x, 32) && aligned(out, 32) && aligned(out32, 16)) go(k_raw_operator<true>);
    else go(k_raw_operator<false>);
    return blocks;
  }
  const int blocks = int(std::min<long long>(raw_blocks(), nblk(32LL * std::max((long long)nRuns, (nB + 3) / 4LL))));
  auto go = [&](auto kernel) {
    launch(kernel, dim3(blocks), s, runs, nRuns, coef, planeStride, bPtr, bCol, bVal, bGlobal, nB, b, x, out, mode, partials, out32, KP);
  };
  const bool few = nB <= kRawRowsFew;
  if (K == 1) few ? go(k_raw_few<1, true>) : go(k_raw_few<1, false>);
  else if (K == 2) few ? go(k_raw_few<2, true>) : go(k_raw_few<2, false>);
  else if (K == 3) few ? go(k_raw_few<3, true>) : go(k_raw_few<3, false>);
  else few ? go(k_raw_few<4, true>) : go(k_raw_few<4, false>);
  return blocks;
}
void launch_raw_operator(const ColourRun* runs, int nRuns, const double* coef, int planeStride, const int* bPtr, const int* bCol,
                         const double* bVal, const int* bGlobal, int nB, const double* b, const double* x, double* out, int K,
                         int mode, const SumTarget& t, cudaStream_t s) {
  if (nRuns == 0 && nB == 0) return;
  const int blocks = launch_raw(runs, nRuns, coef, planeStride, bPtr, bCol, bVal, bGlobal, nB, b, x, out, K, mode, t.partials, nullptr, 0, s);
  if (t.partials && t.sums) launch_sums(t, blocks, K, s);
}
int raw_operator_blocks(int nRuns, int nB, int K) { return raw_blocks(); }
void launch_raw_residual_f32(const ColourRun* runs, int nRuns, const double* coef, int planeStride, const int* bPtr,
                             const int* bCol, const double* bVal, const int* bGlobal, int nB, const double* b, const double* x,
                             float* rhs32, int K, int KP, const SumTarget& t, cudaStream_t s, bool xZero) {
  if (nRuns == 0 && nB == 0) return;
  const int blocks = launch_raw(runs, nRuns, coef, planeStride, bPtr, bCol, bVal, bGlobal, nB, b, x, nullptr, K, xZero ? 3 : 0, t.partials, rhs32, KP, s);
  launch_sums(t, blocks, K, s);
}

// ---- flexible CG steps (fixed grids: partial sums in a fixed order)
static inline int fcg_blocks(long long n, int G) { return int(std::min<long long>(raw_blocks(), nblk(n * G))); }
void launch_fcg_precond(long long n, int K, int KP, float* e, const double* r, const double* q, double* z, const SumTarget& t,
                        double* sc, cudaStream_t s) {
  const int G = raw_groups(K), blocks = fcg_blocks(n, G);
  launch(k_fcg_precond, dim3(blocks), s, n, K, KP, G, e, r, q, z, t.partials);
  if (!launch_sums(t, blocks, K, s, 1, sc)) launch(k_fcg_beta, dim3(1), s, K, (const double*)t.sums, sc);
}
void launch_fcg_direction(long long n, int K, const double* z, const double* sc, double* p, cudaStream_t s) {
  launch(k_fcg_direction, dim3(nblk(n * K)), s, n, K, z, sc, p);
}
void launch_fcg_update(long long n, int K, int KP, const double* sc, const double* p, const double* q, double* x, double* r, float* rhs32,
                       const SumTarget& t, cudaStream_t s) {
  const int G = raw_groups(K), blocks = fcg_blocks(n, G);
  launch(k_fcg_update, dim3(blocks), s, n, K, KP, G, sc, p, q, x, r, rhs32, t.partials);
  launch_sums(t, blocks, K, s);
}
void launch_raw_apply_dot(const ColourRun* runs, int nRuns, const double* coef, int planeStride, const int* bPtr, const int* bCol,
                          const double* bVal, const int* bGlobal, int nB, const double* x, double* out, int K, const int* frozen,
                          double* sc, const SumTarget& t, cudaStream_t s) {
  if (nRuns == 0 && nB == 0) return;
  const int blocks = launch_raw(runs, nRuns, coef, planeStride, bPtr, bCol, bVal, bGlobal, nB, nullptr, x, out, K, 2, t.partials, nullptr, 0, s);
  if (!launch_sums(t, blocks, K, s, 2, sc, frozen)) launch(k_fcg_alpha, dim3(1), s, K, (const double*)t.sums, frozen, sc);
}

void launch_axpby(double* out, double a, const double* x, double b, const double* y, long long n, cudaStream_t s) {
  if (n > 0) k_axpby<<<nblk(n), 256, 0, s>>>(out, a, x, b, y, n);
}
template <typename T>
void launch_pack_rhs(const double* r, T* rhs, long long n, int K, int KP, cudaStream_t s) {
  launch(k_pack<double, T>, dim3(nblk(n * KP)), s, r, rhs, n, K, KP);
}
template <typename T>
void launch_pad_vector(const T* tight, T* padded, long long n, int K, int KP, cudaStream_t s) {
  launch(k_pack<T, T>, dim3(nblk(n * KP)), s, tight, padded, n, K, KP);
}
template <typename T>
void launch_unpad_vector(const T* padded, T* tight, long long n, int K, int KP, cudaStream_t s) {
  launch(k_unpack<T>, dim3(nblk(n * K)), s, padded, tight, n, K, KP);
}
void launch_set_flags(int* flags, unsigned long long mask, int k, cudaStream_t s) {
  launch(k_set_flags, dim3(1), s, flags, mask, k);
}
template <typename T>
void launch_add_correction(double* x, T* e, long long n, int K, int KP, cudaStream_t s, const int* frozen) {
  const long long total = n * K;
  const int small = total <= 0xffffffffLL ? 1 : 0;
  // one value per thread up to two waves of threads (2048 an SM)
  if (total <= 2 * 2048LL * device_sms()) launch(k_add_correction<T, 1>, dim3(nblk(total)), s, x, e, n, K, KP, frozen, small);
  else launch(k_add_correction<T, 4>, dim3(nblk((total + 3) / 4)), s, x, e, n, K, KP, frozen, small);
}

#define GDTP_INSTANTIATE(T, W)                                                                                             \
  template void launch_gs_colour<T, W>(const ColourRun*, int, const T*, int, const T*, T*, int, cudaStream_t, int, bool); \
  template bool launch_gs_rows<T, W>(const LevelDev<T>&, int, bool, int, cudaStream_t, int, bool);                       \
  template bool gs_rows_available<T, W>(const LevelDev<T>&);                                                             \
  template size_t gs_rows_smem<T, W>(const LevelDev<T>&);                                                                \
  template bool launch_gs_groups<T, W>(const LevelDev<T>&, int, bool, int, cudaStream_t);                                \
  template bool bs_dense_on_clusters<T, W>(const BoundaryDev<T>&, int, int);                                              \
  template void launch_residual<T, W>(const ColourRun*, int, const T*, int, const int*, const int*, const T*, const int*, \
                                      int, const T*, const T*, T*, int, cudaStream_t, bool);                             \
  template void launch_restrict<T, W>(const RestrictRun*, int, const int*, const int*, const T*, const int*, int,        \
                                      const T*, T*, T*, long long, int, cudaStream_t);                                   \
  template void launch_prolong_add<T, W>(const ProlongRun*, int, const T*, T*, int, cudaStream_t);                       \
  template void launch_boundary_solve<T, W>(const BoundaryDev<T>&, const T*, T*, int, cudaStream_t, bool);               \
  template void launch_coarse_solve<T, W>(int, const double*, const double*, const T*, T*, int, cudaStream_t);
GDTP_INSTANTIATE(float, 1)
GDTP_INSTANTIATE(float, 4)
GDTP_INSTANTIATE(double, 1)
GDTP_INSTANTIATE(double, 4)
template void launch_pad_vector<float>(const float*, float*, long long, int, int, cudaStream_t);
template void launch_pad_vector<double>(const double*, double*, long long, int, int, cudaStream_t);
template void launch_unpad_vector<float>(const float*, float*, long long, int, int, cudaStream_t);
template void launch_unpad_vector<double>(const double*, double*, long long, int, int, cudaStream_t);
template void launch_pack_rhs<float>(const double*, float*, long long, int, int, cudaStream_t);
template void launch_pack_rhs<double>(const double*, double*, long long, int, int, cudaStream_t);
template void launch_add_correction<float>(double*, float*, long long, int, int, cudaStream_t, const int*);
template void launch_add_correction<double>(double*, double*, long long, int, int, cudaStream_t, const int*);

}  // namespace dev
}  // namespace gdtp
