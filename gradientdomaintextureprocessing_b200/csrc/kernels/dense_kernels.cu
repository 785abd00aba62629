// Dense FP64 set-up products on the device: the inverses and products of the
// exact boundary-block solve and the coarsest-level inverse (setup/bsolve.cpp,
// system.cu), which the reference factorises with Eigen's SimplicialLDLT
// (UpdateCoefficients.inl:402-439, Solver.h:144-259).
//
// Inverse: blocked Gauss-Jordan elimination without pivoting (the matrices are
// symmetric positive definite, so every pivot block is a principal block of a
// Schur complement, itself SPD).  Step k takes the 64 pivot rows and columns
// K = [64k, 64k + 64):
//   P    = A[K,K]^-1              (k_bgj_first, then by the update of step k - 1)
//   R    = P [A[K,:] with A[K,K] replaced by I]       (k_bgj_panel, row tiles)
//   Cold = A[:,K] with rows K zeroed; A[i,K] = 0, i not in K (k_bgj_panel)
//   A[K,:] = R;  A -= Cold R                          (k_bgj_update, rank-64 update)
// after which A[K,K] = P, A[K,j] = P A[K,j], A[i,K] = -A[i,K] P and
// A[i,j] -= A[i,K] P A[K,j]: the n/64 steps leave A^-1.  Every matrix of a
// batch takes part in the steps k < ceil(m/64); the update is 2 n^3 flops in
// 64 x 64 register-tiled FP64 tiles.  A non-positive pivot sets an error flag
// (and the result is discarded).  The result is made exactly symmetric by
// averaging with its transpose.
//
// What bounds it: the steps are a chain, so a lone matrix pays each step's latency
// (pivot inverse, panel, update) and a batch or a large matrix the update's products.
// Steps of a 2240 x 2240 matrix (the coarsest level of a 1024^2 atlas): 49 us each
// (panel 8.7, update 40.2 with the next pivot's inverse in it), before 95 (panel 21,
// update 74 with the selects and 16-wide chunks) and, with the pivot in a launch of its
// own, 160; new weights and a solve there 9.4 -> 5.3 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>
#include <vector>

#include "vcycle.cuh"
#include "vcycle_kernels.h"

namespace gdtp {
namespace dev {
namespace {

constexpr int kPB = 64;  // pivot block of the blocked Gauss-Jordan elimination

// C (M x N) = op(A) B over a batch of tasks (blockIdx.z); op(A)
// is A (M x K, leading dimension lda) or, with transA, the transpose of A
// stored K x M.  64 x 64 tiles, 256 threads of 4 x 4 outputs each (rows ty +
// 16 r, columns tx + 16 c), K in chunks of 16 through shared memory.
__global__ void __launch_bounds__(256) k_gemm(const GemmTask* __restrict__ tasks, const double* __restrict__ A,
                                              const double* __restrict__ B, double* __restrict__ C) {
  const GemmTask T = tasks[blockIdx.z];
  const int row0 = blockIdx.y * 64, col0 = blockIdx.x * 64;
  if (row0 >= T.M || col0 >= T.N) return;
  __shared__ double As[16][64 + 1], Bs[16][64];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  double acc[4][4];
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) acc[r][c] = 0.0;
  const double* Ab = A + T.a;
  const double* Bb = B + T.b;
  // the next chunk of K is loaded into registers while this one is multiplied
  double an[4], bn[4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int e = tid + 256 * q;
      an[q] = 0.0;
      if (T.transA) {  // A stored K x M: consecutive threads along the rows of the tile
        const int gr = row0 + (e & 63), gk = k0 + (e >> 6);
        if (gr < T.M && gk < T.K) an[q] = Ab[(long long)gk * T.lda + gr];
      } else {  // A stored M x K: consecutive threads along k
        const int gr = row0 + (e >> 4), gk = k0 + (e & 15);
        if (gr < T.M && gk < T.K) an[q] = Ab[(long long)gr * T.lda + gk];
      }
      const int gk = k0 + (e >> 6), gc = col0 + (e & 63);
      bn[q] = (gk < T.K && gc < T.N) ? Bb[(long long)gk * T.ldb + gc] : 0.0;
    }
  };
  fetch(0);
  for (int k0 = 0; k0 < T.K; k0 += 16) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int e = tid + 256 * q;
      if (T.transA) As[e >> 6][e & 63] = an[q];
      else As[e & 15][e >> 4] = an[q];
      Bs[e >> 6][e & 63] = bn[q];
    }
    __syncthreads();
    if (k0 + 16 < T.K) fetch(k0 + 16);
#pragma unroll
    for (int kk = 0; kk < 16; kk++) {
      double a[4], b[4];
#pragma unroll
      for (int r = 0; r < 4; r++) a[r] = As[kk][ty + 16 * r];
#pragma unroll
      for (int c = 0; c < 4; c++) b[c] = Bs[kk][tx + 16 * c];
#pragma unroll
      for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[r][c] = fma(a[r], b[c], acc[r][c]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int gr = row0 + ty + 16 * r;
    if (gr >= T.M) continue;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int gc = col0 + tx + 16 * c;
      if (gc >= T.N) continue;
      C[T.c + (long long)gr * T.ldc + gc] = acc[r][c] + 0.0;  // (no negative zeros)
    }
  }
}

// Product of two 64 x 64 tiles, the part [K0, K1) of the inner dimension, on 128
// threads of 8 x 4 outputs each (rows ty + 8 r, columns tx + 16 c): 16 shared-memory
// reads for 64 products.
constexpr int kEThreads = 128;
constexpr int kPitchA = kPB + 2;  // the two rows that a warp reads lie in different banks
constexpr size_t kETile = (size_t(kPB) * kPitchA + size_t(kPB) * kPB) * sizeof(double);
__device__ __forceinline__ void tile_product(double (&acc)[8][4], const double* As, const double* Bs, int tx, int ty, int K0, int K1) {
#pragma unroll 4
  for (int kk = K0; kk < K1; kk += 2) {
    double2 a[8];
#pragma unroll
    for (int r = 0; r < 8; r++) a[r] = *reinterpret_cast<const double2*>(As + (ty + 8 * r) * kPitchA + kk);
    double b[4];
#pragma unroll
    for (int c = 0; c < 4; c++) b[c] = Bs[kk * kPB + tx + 16 * c];
#pragma unroll
    for (int r = 0; r < 8; r++)
#pragma unroll
      for (int c = 0; c < 4; c++) acc[r][c] = fma(a[r].x, b[c], acc[r][c]);
#pragma unroll
    for (int c = 0; c < 4; c++) b[c] = Bs[(kk + 1) * kPB + tx + 16 * c];
#pragma unroll
    for (int r = 0; r < 8; r++)
#pragma unroll
      for (int c = 0; c < 4; c++) acc[r][c] = fma(a[r].y, b[c], acc[r][c]);
  }
}

// queue the inner part [K0, K0 + 32) of the tiles: A rows [0, rows) (64 wide, 16-byte
// aligned) and B rows below K, columns [0, cols) (leading dimension ldb)
__device__ __forceinline__ void queue_half(double* As, double* Bs, const double* A, int rows, const double* B, int ldb, int K, int cols, int K0) {
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const int e = threadIdx.x + kEThreads * q, r = e >> 4, c = K0 + 2 * (e & 15);
    copy_async_or_zero<16>(As + r * kPitchA + c, r < rows ? A + r * kPB + c : A, r < rows);
  }
#pragma unroll
  for (int q = 0; q < 16; q++) {
    const int e = threadIdx.x + kEThreads * q, r = K0 + (e >> 6), c = e & 63;
    const bool in = r < K && c < cols;
    copy_async_or_zero<8>(Bs + r * kPB + c, in ? B + (long long)r * ldb + c : B, in);
  }
  copies_commit();
}

// Unblocked Gauss-Jordan inverse of the bs x bs block (bs <= 64) whose entries (ty +
// 8 r, tx + 16 c) thread (ty, tx) of 8 x 16 holds in P[r][c] (zeros past bs), in
// registers.  The pivot row and column of each step go through shared memory (sm:
// 2 x 3 x 64 doubles), double-buffered so that one barrier per step orders them, with
// the next diagonal entry, so that the next pivot's reciprocal is taken beside this
// step's update.  The steps are a chain: s = 8 sr + sy with sr unrolled fixes at
// compile time which of a thread's entries can be in the pivot row or column (selects
// over all 32, and the division between the barrier and the update: 0.55 us a step).
__device__ __forceinline__ void invert_block(double (&P)[8][4], int bs, double* sm, int* __restrict__ bad) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  if (threadIdx.x == 0) sm[3 * kPB + 2 * kPB] = P[0][0];  // the second buffer's diagonal slot
  __syncthreads();
  auto reciprocal = [&](double p) {
    if (!(p > 0.0)) {
      if (threadIdx.x == 0) atomicExch(bad, 1);
      p = 1.0;
    }
    return 1.0 / p;
  };
  double ip = reciprocal(sm[3 * kPB + 2 * kPB]);
#pragma unroll
  for (int sr = 0; sr < 8; sr++) {
    constexpr int kLast = 7;
    for (int sy = 0; sy < 8; sy++) {
      const int s = 8 * sr + sy;
      if (s >= bs) break;
      double* rowS = sm + (s & 1) * 3 * kPB;
      double* colS = rowS + kPB;
      double* diag = colS + kPB;
      const int sx = 8 * (sr & 1) + sy;  // s & 15
      const bool row = ty == sy, col = tx == sx;
      // the pivot row s and column s as they stand before step s
      if (row)
#pragma unroll
        for (int c = 0; c < 4; c++) rowS[tx + 16 * c] = P[sr][c];
      if (col)
#pragma unroll
        for (int r = 0; r < 8; r++) colS[ty + 8 * r] = P[r][sr >> 1];
      if (ty == ((sy + 1) & 7) && tx == ((s + 1) & 15)) {
        if (sy < 7) *diag = P[sr][sr >> 1];
        else if (sr < kLast) *diag = P[sr < kLast ? sr + 1 : sr][(sr < kLast ? sr + 1 : sr) >> 1];
      }
      __syncthreads();
      double tb[4];
#pragma unroll
      for (int c = 0; c < 4; c++) tb[c] = rowS[tx + 16 * c] * ip;
      // the next pivot as this step leaves it
      double next = 1.0;
      if (s + 1 < bs) next = fma(-colS[s + 1], rowS[s + 1] * ip, *diag);
      const double ipn = reciprocal(next);
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const double ca = colS[ty + 8 * r];
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const double v = fma(-ca, tb[c], P[r][c]);
          const bool inRow = r == sr && row, inCol = c == (sr >> 1) && col;
          P[r][c] = inRow ? (inCol ? ip : tb[c]) : (inCol ? -ca * ip : v);
        }
      }
      ip = ipn;
    }
  }
}

__device__ __forceinline__ void store_inverse(const double (&P)[8][4], double* __restrict__ Pq) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) Pq[(ty + 8 * r) * kPB + tx + 16 * c] = P[r][c];
}

// P_q = A_q[0:64, 0:64]^-1, the first pivot block of every matrix q (one CTA each;
// the later ones are inverted by the update before them)
__global__ void __launch_bounds__(kEThreads) k_bgj_first(const long long* __restrict__ off, const int* __restrict__ size,
                                                         const double* __restrict__ A, double* __restrict__ Pinv, int* __restrict__ bad) {
  const int q = blockIdx.x, m = size[q], bs = min(kPB, m), tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  if (m <= 0) return;
  __shared__ double sm[6 * kPB];
  const double* Aq = A + off[q];
  double P[8][4];
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int i = ty + 8 * r, j = tx + 16 * c;
      P[r][c] = (i < bs && j < bs) ? Aq[(long long)i * m + j] : 0.0;
    }
  invert_block(P, bs, sm, bad);
  store_inverse(P, Pinv + (long long)q * kPB * kPB);
}

// blockIdx.y == 0: row tile t of R = P [A[K,:], A[K,K] -> I], written to R
// (64 x m per matrix) and to A[K,:].  blockIdx.y == 1: row tile t of
// Cold = A[:,K] (rows K zeroed, 64 columns per row), A[i,K] = 0 for i not in K.
// The two roles touch disjoint entries of A (rows K, and columns K outside rows K).
__global__ void __launch_bounds__(kEThreads, 3) k_bgj_panel(int k, const long long* __restrict__ off, const int* __restrict__ size,
                                                            const long long* __restrict__ wsOff, double* A,
                                                            const double* __restrict__ Pinv, double* __restrict__ R, double* __restrict__ Cold) {
  const int q = blockIdx.z, m = size[q], kb = k * kPB;
  if (kb >= m) return;
  const int bs = min(kPB, m - kb), t0 = blockIdx.x * kPB;
  if (t0 >= m) return;
  double* Aq = A + off[q];
  if (blockIdx.y == 1) {
    double* Cq = Cold + wsOff[q];
#pragma unroll
    for (int h = 0; h < 4; h++) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int e = threadIdx.x + kEThreads * (8 * h + u), i = t0 + (e >> 6), c = e & 63;
        v[u] = 0.0;
        if (i < m && c < bs && (i < kb || i >= kb + bs)) v[u] = Aq[(long long)i * m + kb + c];
      }
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int e = threadIdx.x + kEThreads * (8 * h + u), i = t0 + (e >> 6), c = e & 63;
        if (i >= m) continue;
        if (c < bs && (i < kb || i >= kb + bs)) Aq[(long long)i * m + kb + c] = 0.0;
        Cq[(long long)i * kPB + c] = v[u];
      }
    }
    return;
  }
  extern __shared__ __align__(16) double sm[];
  double *As = sm, *Bs = sm + kPB * kPitchA;
  const double* Pq = Pinv + (long long)q * kPB * kPB;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4, cols = t0 == kb ? 0 : m - t0;
  const double* X = Aq + (long long)kb * m + t0;
  queue_half(As, Bs, Pq, kPB, X, m, bs, cols, 0);
  queue_half(As, Bs, Pq, kPB, X, m, bs, cols, kPB / 2);
  double acc[8][4];
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) acc[r][c] = 0.0;
  if (t0 == kb) {  // columns K: the identity
    copies_wait<0>();
    __syncthreads();
    if (threadIdx.x < bs) Bs[threadIdx.x * (kPB + 1)] = 1.0;
  }
  copies_wait<1>();
  __syncthreads();
  tile_product(acc, As, Bs, tx, ty, 0, kPB / 2);
  copies_wait<0>();
  __syncthreads();
  tile_product(acc, As, Bs, tx, ty, kPB / 2, kPB);
  double* Rq = R + wsOff[q];
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int rr = ty + 8 * r, j = t0 + tx + 16 * c;
      if (rr >= bs || j >= m) continue;
      Rq[(long long)rr * m + j] = acc[r][c];
      Aq[(long long)(kb + rr) * m + j] = acc[r][c];
    }
}

// A_q -= Cold_q R_q (64 x 64 tiles, one per CTA) over the step's tasks, the rank-64
// update of elimination step kNext - 1.  The whole inner dimension is copied to shared
// memory at once, in two halves, so that a tile waits for memory once or twice, not
// for every 16 of the 64.  The tile of the next pivot block, taken by the task's first
// CTA, goes on to be inverted: the inversion, a chain of 64 barriers, runs beside the
// other tiles instead of in a launch of its own.
__global__ void __launch_bounds__(kEThreads, 3) k_bgj_update(const GemmTask* __restrict__ tasks, const double* __restrict__ Cold,
                                                             const double* __restrict__ R, double* __restrict__ A, int kNext,
                                                             double* __restrict__ Pinv, int* __restrict__ bad) {
  const GemmTask T = tasks[blockIdx.z];
  int bx = blockIdx.x, by = blockIdx.y;
  bool pivot = false;
  if (kNext * kPB < T.M) {  // the next pivot block's tile changes places with the first
    pivot = bx == 0 && by == 0;
    if (pivot) bx = by = kNext;
    else if (bx == kNext && by == kNext) bx = by = 0;
  }
  const int row0 = by * kPB, col0 = bx * kPB;
  if (row0 >= T.M || col0 >= T.N) return;
  extern __shared__ __align__(16) double sm[];
  double *As = sm, *Bs = sm + kPB * kPitchA;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const double* At = Cold + T.a + (long long)row0 * kPB;
  const double* Bt = R + T.b + col0;
  queue_half(As, Bs, At, T.M - row0, Bt, T.ldb, T.K, T.N - col0, 0);
  queue_half(As, Bs, At, T.M - row0, Bt, T.ldb, T.K, T.N - col0, kPB / 2);
  double acc[8][4];
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) acc[r][c] = 0.0;
  copies_wait<1>();
  __syncthreads();
  tile_product(acc, As, Bs, tx, ty, 0, kPB / 2);
  copies_wait<0>();
  __syncthreads();
  tile_product(acc, As, Bs, tx, ty, kPB / 2, kPB);
  double* Ct = A + T.c + (long long)(row0 + ty) * T.ldc + col0 + tx;
  double P[8][4];
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) P[r][c] = (row0 + ty + 8 * r < T.M && col0 + tx + 16 * c < T.N) ? Ct[(long long)(8 * r) * T.ldc + 16 * c] : 0.0;
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      P[r][c] -= acc[r][c];
      if (row0 + ty + 8 * r < T.M && col0 + tx + 16 * c < T.N) Ct[(long long)(8 * r) * T.ldc + 16 * c] = P[r][c];
    }
  if (!pivot) return;
  __syncthreads();  // As is free
  invert_block(P, min(kPB, T.M - row0), As, bad);
  store_inverse(P, Pinv + (long long)T.matrix * kPB * kPB);
}

// out = (in + in^T) / 2, a 32 x 32 tile per CTA (32 x 8 threads) with its transpose
// turned in shared memory: both are read along rows (an element per thread with the
// transpose read down a column took 79 us on a 2240 x 2240 matrix, 40 MB).
constexpr int kSymTile = 32;
__global__ void __launch_bounds__(256) k_symmetrise(const long long* __restrict__ off, const int* __restrict__ size,
                                                    const double* __restrict__ in, double* __restrict__ out) {
  const int m = size[blockIdx.z], i0 = blockIdx.y * kSymTile, j0 = blockIdx.x * kSymTile;
  if (i0 >= m || j0 >= m) return;
  __shared__ double t[kSymTile][kSymTile + 1];
  const double* A = in + off[blockIdx.z];
  double* O = out + off[blockIdx.z];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  double v[4];
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int i = i0 + y + 8 * r, j = j0 + x, ti = j0 + y + 8 * r, tj = i0 + x;
    v[r] = i < m && j < m ? A[(long long)i * m + j] : 0.0;
    t[y + 8 * r][x] = ti < m && tj < m ? A[(long long)ti * m + tj] : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int i = i0 + y + 8 * r, j = j0 + x;
    if (i < m && j < m) O[(long long)i * m + j] = 0.5 * (v[r] + t[x][y + 8 * r]);
  }
}

// stream-ordered scratch (no device-wide synchronisation on release, so the
// set-up of one system does not wait for the solves of others)
struct Buf {
  void* p = nullptr;
  cudaStream_t s = nullptr;
  ~Buf() {
    if (p) cudaFreeAsync(p, s);
  }
  template <class T>
  T* as() const { return static_cast<T*>(p); }
};

bool check(cudaError_t e, const char* what, std::string& err) {
  if (e == cudaSuccess) return true;
  err = std::string(what) + ": " + cudaGetErrorString(e);
  return false;
}

bool alloc(Buf& b, size_t bytes, cudaStream_t s, std::string& err) {
  b.s = s;
  return check(cudaMallocAsync(&b.p, std::max<size_t>(16, bytes), s), "cudaMallocAsync", err);
}

template <class T>
bool upload(Buf& b, const T* v, size_t n, cudaStream_t s, std::string& err) {
  if (!alloc(b, n * sizeof(T), s, err)) return false;
  return n == 0 || check(cudaMemcpyAsync(b.p, v, n * sizeof(T), cudaMemcpyHostToDevice, s), "h2d", err);
}
template <class T>
bool upload(Buf& b, const std::vector<T>& v, cudaStream_t s, std::string& err) {
  return upload(b, v.data(), v.size(), s, err);
}

constexpr int kMaxGridZ = 65535;

}  // namespace

void launch_gemm_batch(const GemmTask* dTasks, int nTasks, int maxM, int maxN, const double* A, const double* B, double* C,
                       cudaStream_t s) {
  for (int t0 = 0; t0 < nTasks; t0 += kMaxGridZ) {
    const dim3 grid(unsigned((maxN + 63) / 64), unsigned((maxM + 63) / 64), unsigned(std::min(kMaxGridZ, nTasks - t0)));
    k_gemm<<<grid, 256, 0, s>>>(dTasks + t0, A, B, C);
  }
}

bool spd_inverse_layout(const std::vector<int64_t>& offsets, const std::vector<int>& sizes, SpdInverseLayout& L, std::string& err) {
  L = SpdInverseLayout();
  L.nMat = (int)sizes.size();
  if (L.nMat > kMaxGridZ) {
    err = "more dense blocks than one launch holds";
    return false;
  }
  L.offsets = offsets;
  L.sizes = sizes;
  L.ws.resize(L.nMat);
  int mMax = 0;
  for (int q = 0; q < L.nMat; q++) {
    L.ws[q] = L.wsTotal;
    L.wsTotal += (long long)kPB * sizes[q];
    L.elems = std::max<long long>(L.elems, offsets[q] + (long long)sizes[q] * sizes[q]);
    mMax = std::max(mMax, sizes[q]);
  }
  L.steps = (mMax + kPB - 1) / kPB;
  // rank-64 update tasks of every step: A_q -= Cold_q R_q over the matrices still eliminating
  L.taskStart.assign(L.steps + 1, 0);
  L.stepMax.assign(L.steps, 0);
  for (int k = 0; k < L.steps; k++) {
    for (int q = 0; q < L.nMat; q++) {
      const int m = sizes[q], kb = k * kPB;
      if (kb >= m) continue;
      GemmTask T{};
      T.a = L.ws[q];
      T.b = L.ws[q];
      T.c = offsets[q];
      T.M = T.N = m;
      T.K = std::min(kPB, m - kb);
      T.ldb = m;
      T.ldc = m;
      T.matrix = q;
      L.tasks.push_back(T);
      L.stepMax[k] = std::max(L.stepMax[k], m);
    }
    L.taskStart[k + 1] = (int)L.tasks.size();
  }
  return true;
}

size_t spd_inverse_scratch_doubles(const SpdInverseLayout& L) { return size_t(L.nMat) * kPB * kPB + 2 * size_t(L.wsTotal); }

bool launch_spd_inverse(const SpdInverseLayout& L, const SpdInverseDevice& D, double* A, double* out, double* scratch, int* bad,
                        cudaStream_t s) {
  if (L.nMat == 0 || L.steps == 0) return true;
  for (const void* f : {reinterpret_cast<const void*>(k_bgj_panel), reinterpret_cast<const void*>(k_bgj_update)})
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kETile)) != cudaSuccess) return false;
  double* pinv = scratch;
  double* rw = pinv + size_t(L.nMat) * kPB * kPB;
  double* cw = rw + L.wsTotal;  // 64 doubles a row, as pinv: rows stay 16-byte aligned
  k_bgj_first<<<L.nMat, kEThreads, 0, s>>>(D.off, D.size, A, pinv, bad);
  for (int k = 0; k < L.steps; k++) {
    // matrices of size m <= 64k, and tiles past a matrix's own size, return at once
    const unsigned tiles = unsigned((L.stepMax[k] + kPB - 1) / kPB);
    k_bgj_panel<<<dim3(tiles, 2, unsigned(L.nMat)), kEThreads, kETile, s>>>(k, D.off, D.size, D.ws, A, pinv, rw, cw);
    k_bgj_update<<<dim3(tiles, tiles, unsigned(L.taskStart[k + 1] - L.taskStart[k])), kEThreads, kETile, s>>>(D.tasks + L.taskStart[k], cw, rw, A,
                                                                                                            k + 1, pinv, bad);
  }
  const unsigned tiles = unsigned((L.stepMax[0] + kSymTile - 1) / kSymTile);
  k_symmetrise<<<dim3(tiles, tiles, unsigned(L.nMat)), 256, 0, s>>>(D.off, D.size, A, out);
  return cudaGetLastError() == cudaSuccess;
}

namespace {

// device copies of a layout's arrays in stream-ordered scratch
struct LayoutUpload {
  Buf off, size, ws, tasks;
  SpdInverseDevice dev;
  bool run(const SpdInverseLayout& L, cudaStream_t s, std::string& err) {
    if (!upload(off, L.offsets, s, err) || !upload(size, L.sizes, s, err) ||
        !upload(ws, L.ws, s, err) || !upload(tasks, L.tasks, s, err))
      return false;
    dev = {off.as<long long>(), size.as<int>(), ws.as<long long>(), tasks.as<GemmTask>()};
    return true;
  }
};

}  // namespace

bool gpu_spd_inverse_batched(double* data, const std::vector<int64_t>& offsets, const std::vector<int>& sizes, cudaStream_t s,
                             std::string& err) {
  SpdInverseLayout L;
  if (!spd_inverse_layout(offsets, sizes, L, err)) return false;
  if (L.nMat == 0 || L.steps == 0) return true;
  LayoutUpload U;
  Buf a, b, bad, scratch;
  if (!U.run(L, s, err) || !upload(a, data, size_t(L.elems), s, err) || !alloc(b, size_t(L.elems) * sizeof(double), s, err) ||
      !upload(bad, std::vector<int>(1, 0), s, err) || !alloc(scratch, spd_inverse_scratch_doubles(L) * sizeof(double), s, err))
    return false;
  if (!launch_spd_inverse(L, U.dev, a.as<double>(), b.as<double>(), scratch.as<double>(), bad.as<int>(), s)) {
    err = std::string("Gauss-Jordan: ") + cudaGetErrorString(cudaGetLastError());
    return false;
  }
  int badHost = 0;
  if (!check(cudaMemcpyAsync(&badHost, bad.p, sizeof(int), cudaMemcpyDeviceToHost, s), "d2h", err) ||
      !check(cudaStreamSynchronize(s), "Gauss-Jordan", err))
    return false;
  if (badHost) {
    err = "dense block is not positive definite";
    return false;
  }
  for (int q = 0; q < L.nMat; q++) {
    const size_t bytes = size_t(sizes[q]) * sizes[q] * sizeof(double);
    if (bytes && !check(cudaMemcpyAsync(data + offsets[q], b.as<double>() + offsets[q], bytes, cudaMemcpyDeviceToHost, s), "d2h", err))
      return false;
  }
  return check(cudaStreamSynchronize(s), "Gauss-Jordan", err);
}

void schur_product_tasks(const std::vector<int64_t>& invOff, const std::vector<int>& m, const std::vector<int64_t>& cOff,
                         const std::vector<int>& t, const std::vector<int64_t>& localOff, std::vector<GemmTask>& gTasks,
                         std::vector<GemmTask>& lTasks, int& maxM, int& maxT) {
  gTasks.clear();
  lTasks.clear();
  maxM = maxT = 1;
  for (size_t p = 0; p < m.size(); p++) {
    if (t[p] == 0 || m[p] == 0) continue;
    GemmTask g{};  // G = Inv C   (m x t)
    g.a = invOff[p];
    g.b = cOff[p];
    g.c = cOff[p];
    g.M = m[p];
    g.N = t[p];
    g.K = m[p];
    g.lda = m[p];
    g.ldb = t[p];
    g.ldc = t[p];
    gTasks.push_back(g);
    GemmTask l{};  // local = C^T G   (t x t)
    l.a = cOff[p];
    l.b = cOff[p];
    l.c = localOff[p];
    l.M = t[p];
    l.N = t[p];
    l.K = m[p];
    l.lda = t[p];
    l.ldb = t[p];
    l.ldc = t[p];
    l.transA = 1;
    lTasks.push_back(l);
    maxM = std::max(maxM, m[p]);
    maxT = std::max(maxT, t[p]);
  }
}

bool gpu_schur_products(const std::vector<double>& inv, const std::vector<int64_t>& invOff, const std::vector<int>& m,
                        const std::vector<double>& C, const std::vector<int64_t>& cOff, const std::vector<int>& t, std::vector<double>& G,
                        std::vector<double>& local, const std::vector<int64_t>& localOff, cudaStream_t s, std::string& err) {
  const int nSub = (int)m.size();
  G.assign(C.size(), 0.0);
  long long localTotal = 0;
  for (int p = 0; p < nSub; p++) localTotal = std::max<long long>(localTotal, localOff[p] + (long long)t[p] * t[p]);
  local.assign(size_t(localTotal), 0.0);
  std::vector<GemmTask> gTasks, lTasks;
  int maxM = 1, maxT = 1;
  schur_product_tasks(invOff, m, cOff, t, localOff, gTasks, lTasks, maxM, maxT);
  if (gTasks.empty()) return true;
  Buf dInv, dC, dG, dL, dgt, dlt;
  if (!upload(dInv, inv, s, err) || !upload(dC, C, s, err) || !alloc(dG, C.size() * sizeof(double), s, err) ||
      !alloc(dL, size_t(localTotal) * sizeof(double), s, err) || !upload(dgt, gTasks, s, err) || !upload(dlt, lTasks, s, err))
    return false;
  launch_gemm_batch(dgt.as<GemmTask>(), (int)gTasks.size(), maxM, maxT, dInv.as<double>(), dC.as<double>(), dG.as<double>(), s);
  launch_gemm_batch(dlt.as<GemmTask>(), (int)lTasks.size(), maxT, maxT, dC.as<double>(), dG.as<double>(), dL.as<double>(), s);
  if (!check(cudaGetLastError(), "products", err) ||
      !check(cudaMemcpyAsync(G.data(), dG.p, G.size() * sizeof(double), cudaMemcpyDeviceToHost, s), "d2h", err) ||
      !check(cudaMemcpyAsync(local.data(), dL.p, local.size() * sizeof(double), cudaMemcpyDeviceToHost, s), "d2h", err) ||
      !check(cudaStreamSynchronize(s), "products", err))
    return false;
  return true;
}

}  // namespace dev
}  // namespace gdtp
