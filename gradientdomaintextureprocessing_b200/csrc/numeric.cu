// Numeric set-up of the multigrid on the device (numeric.h).
#include "numeric.h"

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cmath>
#include <memory>

#include "system.h"

namespace gdtp {
namespace {

constexpr int kThreads = 256;
inline unsigned blocks_for(long long n) { return unsigned(std::max<long long>(1, (n + kThreads - 1) / kThreads)); }

// screen M + stiffness S, each product and the sum rounded once (the host's
// csr_axpby / update arithmetic, without contraction into a fused multiply-add)
__device__ __forceinline__ double combine_rn(double a, double m, double b, double s) { return __dadd_rn(__dmul_rn(a, m), __dmul_rn(b, s)); }

__global__ void k_combine(long long n, double a, const double* __restrict__ M, double b, const double* __restrict__ S, double* __restrict__ V) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) V[i] = combine_rn(a, M[i], b, S[i]);
}

// reciprocal planes of the smoother: planes[k][i] = c_k / c_4 (k != 4),
// planes[4][i] = 1 / c_4, planes[9][i] = c_4, c of run texel i's deep texel
template <typename T>
__global__ void k_planes(int count, const int* __restrict__ runTexel, const double* __restrict__ M, const double* __restrict__ S, double a,
                         double b, T* __restrict__ planes) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const long long d = 10LL * runTexel[i];
  const double c4 = combine_rn(a, M[d + 4], b, S[d + 4]), inv = 1.0 / c4;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const double c = combine_rn(a, M[d + k], b, S[d + k]);
    planes[(long long)k * count + i] = T(k == 4 ? inv : __dmul_rn(c, inv));
  }
  planes[9LL * count + i] = T(c4);
}

template <typename T>
__global__ void k_gather_rows(long long n, const int* __restrict__ src, const double* __restrict__ bdV, const double* __restrict__ bbV,
                              T* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int c = src[i];
  out[i] = T(c >= 0 ? bdV[c] : bbV[-1 - c]);
}

// s_k = 1 / sqrt(diagonal of the row at position k)
__global__ void k_scale_pos(int nb, const int* __restrict__ order, const int* __restrict__ diagEntry, const double* __restrict__ bbV,
                            double* __restrict__ scale) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < nb) scale[k] = 1.0 / sqrt(bbV[diagEntry[order[k]]]);
}

struct Scaled {
  const double* bbV;
  const int *bbRow, *bbCol, *pos;
  const double* scale;
  __device__ __forceinline__ double operator()(int e) const {
    return __dmul_rn(__dmul_rn(bbV[e], scale[pos[bbRow[e]]]), scale[pos[bbCol[e]]]);
  }
};

__global__ void k_scatter_scaled(long long n, const int* __restrict__ entry, const long long* __restrict__ dest, Scaled sc,
                                 double* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[dest[i]] = sc(entry[i]);
}

template <typename T>
__global__ void k_scaled_values(long long n, const int* __restrict__ entry, Scaled sc, T* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = T(sc(entry[i]));
}

template <typename T>
__global__ void k_gather_values(long long n, const int* __restrict__ entry, const double* __restrict__ V, T* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = T(V[entry[i]]);
}

template <typename T>
__global__ void k_convert(long long n, const double* __restrict__ src, T* __restrict__ dst) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = T(src[i]);
}

// S -= sum_p scatter(local_p) in subdomain order: a block owns kRowsPerBlock
// separator rows and applies the subdomains one after the other, so every
// entry sees its contributions in the same order from run to run
constexpr int kRowsPerBlock = 16;
__global__ void k_schur_subtract(int nS, int nSub, const int* __restrict__ touchPtr, const int* __restrict__ touch,
                                 const long long* __restrict__ lOff, const double* __restrict__ local, double* __restrict__ S) {
  const int r0 = blockIdx.x * kRowsPerBlock, r1 = min(nS, r0 + kRowsPerBlock);
  for (int p = 0; p < nSub; p++) {
    const int* tp = touch + touchPtr[p];
    const int t = touchPtr[p + 1] - touchPtr[p];
    // the touch list is sorted: its entries in [r0, r1)
    int lo = 0, hi = t;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (tp[mid] < r0) lo = mid + 1; else hi = mid;
    }
    int end = lo;
    while (end < t && tp[end] < r1) end++;
    const int rows = end - lo;
    const double* Lp = local + lOff[p];
    for (int e = threadIdx.x; e < rows * t; e += blockDim.x) {
      const int c1 = lo + e / t, c2 = e % t;
      S[(long long)tp[c1] * nS + tp[c2]] -= Lp[(long long)c1 * t + c2];
    }
    __syncthreads();
  }
}

// S = (S + S^T) / 2 below and above the diagonal
__global__ void k_symmetrise_pairs(int n, double* __restrict__ S) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)n * n) return;
  const int a = int(e / n), c = int(e - (long long)a * n);
  if (c >= a) return;
  const double v = 0.5 * (S[(long long)a * n + c] + S[(long long)c * n + a]);
  S[(long long)a * n + c] = v;
  S[(long long)c * n + a] = v;
}

// subdomain inverses, rows padded to a multiple of 4 (zeros past m): kPadBlocks
// blocks per subdomain, a warp per row (one block per subdomain with a 64-bit
// division per entry took 340 us on level 0 at 1024^2)
constexpr int kPadBlocks = 12;
template <typename T>
__global__ void k_pad_blocks(const int* __restrict__ subPtr, const long long* __restrict__ invOff, const long long* __restrict__ invOffPad,
                             const double* __restrict__ src, T* __restrict__ dst) {
  const int p = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int m = subPtr[p + 1] - subPtr[p], mp = (m + 3) & ~3;
  const double* s = src + invOff[p];
  T* d = dst + invOffPad[p];
  for (int j = blockIdx.y * warps + warp; j < m; j += gridDim.y * warps)
    for (int a = lane; a < mp; a += 32) d[(long long)j * mp + a] = a < m ? T(s[(long long)j * m + a]) : T(0);
}

template <typename T>
__global__ void k_pad_square(int n, int np, const double* __restrict__ src, T* __restrict__ dst) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)n * np) return;
  const int j = int(e / np), a = int(e - (long long)j * np);
  dst[e] = a < n ? T(src[(long long)j * n + a]) : T(0);
}

// back-substitution blocks: W_p (m x t, column-major) from G_p (m x t, row-major),
// kPadBlocks blocks per subdomain, a warp per column
template <typename T>
__global__ void k_wt(const int* __restrict__ subPtr, const int* __restrict__ touchPtr, const long long* __restrict__ wOff,
                     const double* __restrict__ G, T* __restrict__ wt) {
  const int p = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int m = subPtr[p + 1] - subPtr[p], t = touchPtr[p + 1] - touchPtr[p];
  const double* g = G + wOff[p];
  T* w = wt + wOff[p];
  for (int c = blockIdx.y * warps + warp; c < t; c += gridDim.y * warps)
    for (int a = lane; a < m; a += 32) w[(long long)c * m + a] = T(g[(long long)a * t + c]);
}

// coarsest level: a source is kind << 40 | index (0 deep coefficient, 1 bd, 2 bb)
struct Sources {
  double a, b;
  const double *deepM, *deepS, *bdV, *bbV;
  __device__ __forceinline__ double operator()(long long src) const {
    const int kind = int(src >> 40);
    const long long i = src & ((1LL << 40) - 1);
    return kind == 0 ? combine_rn(a, deepM[i], b, deepS[i]) : kind == 1 ? bdV[i] : bbV[i];
  }
};

__global__ void k_coarse_scale(int n, const long long* __restrict__ diagSrc, Sources v, double* __restrict__ scale) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) scale[i] = 1.0 / sqrt(v(diagSrc[i]));
}

__global__ void k_coarse_fill(long long nD, int n, const long long* __restrict__ src, const int* __restrict__ row, const int* __restrict__ col,
                              Sources v, const double* __restrict__ scale, double* __restrict__ dense) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nD) return;
  const int r = row[e], c = col[e];
  dense[(long long)r * n + c] = __dmul_rn(__dmul_rn(v(src[e]), scale[r]), scale[c]);
}

template <class T>
std::vector<int> as_int(const std::vector<T>& v) {
  std::vector<int> out(v.size());
  for (size_t i = 0; i < v.size(); i++) out[i] = int(v[i]);
  return out;
}

std::vector<long long> as_ll(const std::vector<int64_t>& v) { return std::vector<long long>(v.begin(), v.end()); }

__global__ void k_gather_planes(int count, const int* __restrict__ texel, const double* __restrict__ deep, double* __restrict__ planes) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const double* c = deep + 10LL * texel[i];
#pragma unroll
  for (int k = 0; k < 9; k++) planes[(long long)k * count + i] = c[k];
}

}  // namespace

void launch_gather_planes(int count, const int* texel, const double* deep, double* planes, cudaStream_t s) {
  k_gather_planes<<<blocks_for(count), kThreads, 0, s>>>(count, texel, deep, planes);
}

NumericPlan::~NumericPlan() {
  for (LevelStream& ls : streams_) {
    for (cudaEvent_t e : ls.mark)
      if (e) cudaEventDestroy(e);
    if (ls.s) cudaStreamDestroy(ls.s);
  }
  if (ready_) cudaEventDestroy(ready_);
  delete arena_;
}

size_t NumericPlan::deviceBytes() const { return arena_ ? arena_->total : 0; }

namespace {
// host side of one level's plan, built for all levels in parallel before the uploads
struct LevelHost {
  Csr bbS, bdS;                           // S aligned to the union patterns (N.bb, N.bd hold M)
  std::vector<int> bsrc;
  std::vector<long long> denseSrc, diagSrc;
  std::vector<int> denseRow, denseCol, m, t;
  std::string err;
};
}  // namespace

bool NumericPlan::build(const Hierarchy& h, int L_, const FineSystem& fine, const std::vector<LevelCoefficients>& coM,
                        const std::vector<LevelCoefficients>& coS, const double* deep0M, const double* deep0S, int maxBlock_,
                        int denseMax_, cudaStream_t s, std::string& err) {
  (void)s;
  delete arena_;
  arena_ = new DeviceArena();
  DeviceArena& A = *arena_;
  L = L_;
  maxBlock = maxBlock_;
  denseMax = denseMax_;
  levels.assign(L, NumericLevel());
  std::vector<LevelHost> host(L);
  // ---- structure of every level (host, levels in parallel)
#pragma omp parallel for schedule(dynamic, 1)
  for (int l = 0; l < L; l++) {
    const GridLevel& G = h.levels[l];
    NumericLevel& N = levels[l];
    LevelHost& H = host[l];
    N.n = G.numTexels;
    N.nDeep = G.numDeep;
    N.nB = G.numBoundary;
    N.coarsest = (l == L - 1);
    const Csr& bbM = l == 0 ? fine.bbMass : coM[l].bb;
    const Csr& bbS = l == 0 ? fine.bbStiffness : coS[l].bb;
    Csr bdM = l == 0 ? fine.bdMass : coM[l].bd, bdS = l == 0 ? fine.bdStiffness : coS[l].bd;
    bdM.cols = bdS.cols = G.numTexels;
    // union patterns, M and S aligned to them
    N.bb = csr_axpby(1.0, bbM, 0.0, bbS);
    H.bbS = csr_axpby(0.0, bbM, 1.0, bbS);
    N.bd = csr_axpby(1.0, bdM, 0.0, bdS);
    H.bdS = csr_axpby(0.0, bdM, 1.0, bdS);
    N.nBB = (long long)N.bb.col.size();
    N.nBD = (long long)N.bd.col.size();
    if (N.coarsest) {
      // dense entries: deep rows' 3x3 stencils, boundary rows' bd and bb entries
      // (the layout of full_matrix, galerkin.cpp)
      H.diagSrc.assign(G.numTexels, -1);
      for (int d = 0; d < G.numDeep; d++) {
        const int r = G.deepGlobal[d];
        const NodeInfo& nd = G.nodes[r];
        const GridChart& gc = G.charts[nd.chart];
        for (int oy = -1; oy <= 1; oy++)
          for (int ox = -1; ox <= 1; ox++) {
            const int c = gc.texel[gc.at(nd.ci + ox, nd.cj + oy)];
            const long long sIdx = 10LL * d + (oy + 1) * 3 + (ox + 1);
            H.denseRow.push_back(r);
            H.denseCol.push_back(c);
            H.denseSrc.push_back(sIdx);
            if (c == r) H.diagSrc[r] = sIdx;
          }
      }
      for (int b = 0; b < G.numBoundary; b++) {
        const int r = G.boundaryGlobal[b];
        for (int k = N.bd.ptr[b]; k < N.bd.ptr[b + 1]; k++) {
          H.denseRow.push_back(r);
          H.denseCol.push_back(N.bd.col[k]);
          H.denseSrc.push_back((1LL << 40) | k);
          if (N.bd.col[k] == r) H.diagSrc[r] = (1LL << 40) | k;
        }
        for (int k = N.bb.ptr[b]; k < N.bb.ptr[b + 1]; k++) {
          const int c = G.boundaryGlobal[N.bb.col[k]];
          H.denseRow.push_back(r);
          H.denseCol.push_back(c);
          H.denseSrc.push_back((2LL << 40) | k);
          if (c == r) H.diagSrc[r] = (2LL << 40) | k;
        }
      }
      for (int i = 0; i < G.numTexels && H.err.empty(); i++)
        if (H.diagSrc[i] < 0) H.err = "coarsest level: texel without a diagonal entry";
      for (int c : H.denseCol)
        if (H.err.empty() && (c < 0 || c >= G.numTexels)) H.err = "coarsest level: stencil column outside the level";
      if (H.err.empty())
        dev::spd_inverse_layout(std::vector<int64_t>(1, 0), std::vector<int>(1, G.numTexels), N.coarseLayout, H.err);
      continue;
    }
    // boundary rows of the smoother
    N.bPtr.assign(1, 0);
    for (int b = 0; b < G.numBoundary; b++) {
      for (int k = N.bd.ptr[b]; k < N.bd.ptr[b + 1]; k++) { N.bCol.push_back(N.bd.col[k]); H.bsrc.push_back(k); }
      for (int k = N.bb.ptr[b]; k < N.bb.ptr[b + 1]; k++) { N.bCol.push_back(G.boundaryGlobal[N.bb.col[k]]); H.bsrc.push_back(-1 - k); }
      N.bPtr.push_back((int)N.bCol.size());
    }
    N.nBRow = (long long)H.bsrc.size();
    // boundary solver structure
    BoundarySymbolic& sym = N.sym;
    if (!build_boundary_symbolic(N.bb, N.bd, maxBlock, denseMax, sym, H.err)) {
      H.err = "level " + std::to_string(l) + ": " + H.err;
      continue;
    }
    if (sym.nb == 0) continue;
    N.invOffPadHost.assign(sym.nSub + 1, 0);
    H.m.resize(sym.nSub);
    H.t.resize(sym.nSub);
    for (int p = 0; p < sym.nSub; p++) {
      H.m[p] = sym.subPtr[p + 1] - sym.subPtr[p];
      H.t[p] = sym.touchPtr[p + 1] - sym.touchPtr[p];
      N.invOffPadHost[p + 1] = N.invOffPadHost[p] + (long long)H.m[p] * ((H.m[p] + 3) & ~3);
    }
    std::vector<int64_t> invOff(sym.invOff.begin(), sym.invOff.end() - 1);
    if (!dev::spd_inverse_layout(invOff, H.m, N.subLayout, H.err)) continue;
    if (sym.nS > 0 && !dev::spd_inverse_layout(std::vector<int64_t>(1, 0), std::vector<int>(1, sym.nS), N.schurLayout, H.err)) continue;
    std::vector<int64_t> cOff(sym.wOff.begin(), sym.wOff.end() - 1), lOff(sym.lOff.begin(), sym.lOff.end() - 1);
    dev::schur_product_tasks(invOff, H.m, cOff, H.t, lOff, N.gTasks, N.lTasks, N.maxM, N.maxT);
  }
  for (const LevelHost& H : host)
    if (!H.err.empty()) {
      err = H.err;
      return false;
    }
  // ---- resident sources and structure arrays (device)
  auto layout_dev = [&](const dev::SpdInverseLayout& Ly) -> dev::SpdInverseDevice {
    return {A.upload(as_ll(Ly.offsets)), A.upload(Ly.sizes), A.upload(as_ll(Ly.ws)), A.upload(Ly.tasks)};
  };
  for (int l = 0; l < L; l++) {
    NumericLevel& N = levels[l];
    const LevelHost& H = host[l];
    N.deepM = (l == 0 && deep0M) ? deep0M : A.upload(l == 0 ? fine.deepMass : coM[l].deep);
    N.deepS = (l == 0 && deep0S) ? deep0S : A.upload(l == 0 ? fine.deepStiffness : coS[l].deep);
    N.bbM = A.upload(N.bb.val);
    N.bbS = A.upload(H.bbS.val);
    N.bdM = A.upload(N.bd.val);
    N.bdS = A.upload(H.bdS.val);
    N.bbV = static_cast<double*>(A.alloc(std::max<long long>(1, N.nBB) * sizeof(double)));
    N.bdV = static_cast<double*>(A.alloc(std::max<long long>(1, N.nBD) * sizeof(double)));
    if (N.coarsest) {
      N.nDense = (long long)H.denseSrc.size();
      N.denseSrc = A.upload(H.denseSrc);
      N.diagSrc = A.upload(H.diagSrc);
      N.denseRow = A.upload(H.denseRow);
      N.denseCol = A.upload(H.denseCol);
      N.coarseDev = layout_dev(N.coarseLayout);
      continue;
    }
    N.bSrc = A.upload(H.bsrc);
    const BoundarySymbolic& sym = N.sym;
    if (sym.nb == 0) continue;
    N.pos = A.upload(sym.pos);
    N.order = A.upload(sym.order);
    N.bbRow = A.upload(sym.bbRow);
    N.bbCol = A.upload(N.bb.col);
    N.diagEntry = A.upload(sym.diagEntry);
    N.fillEntry = A.upload(sym.fillEntry);
    N.fillDest = A.upload(as_ll(sym.fillDest));
    N.ssEntry = A.upload(sym.ssEntry);
    N.ssDest = A.upload(as_ll(sym.ssDest));
    N.aisEntry = A.upload(as_int(sym.AIS.val));
    N.aisDest = A.upload(as_ll(sym.aisDest));
    N.asiEntry = A.upload(as_int(sym.ASI.val));
    N.bdEntry = A.upload(as_int(sym.BD.val));
    N.subPtr = A.upload(sym.subPtr);
    N.touchPtr = A.upload(sym.touchPtr);
    N.touch = A.upload(sym.touch);
    N.wOff = A.upload(as_ll(sym.wOff));
    N.lOff = A.upload(as_ll(sym.lOff));
    N.invOff = A.upload(as_ll(sym.invOff));
    N.invOffPad = A.upload(N.invOffPadHost);
    N.subDev = layout_dev(N.subLayout);
    if (sym.nS > 0) N.schurDev = layout_dev(N.schurLayout);
    N.gTasksDev = A.upload(N.gTasks);
    N.lTasksDev = A.upload(N.lTasks);
  }
  if (A.last != cudaSuccess) {
    err = std::string("numeric plan upload: ") + cudaGetErrorString(A.last);
    return false;
  }
  return true;
}

bool NumericPlan::set_run_order(int l, const std::vector<int>& runTexel, std::string& err) {
  NumericLevel& N = levels[l];
  if (N.runTexel && N.runCount == (int)runTexel.size()) return true;  // the runs are a function of the level's structure
  N.runTexel = arena_->upload(runTexel);
  N.runCount = (int)runTexel.size();
  if (arena_->last != cudaSuccess) {
    err = std::string("run order upload: ") + cudaGetErrorString(arena_->last);
    return false;
  }
  return true;
}

bool NumericPlan::combine(double a, double b, cudaStream_t s, std::string& err) {
  screen = a;
  stiffness = b;
  for (NumericLevel& N : levels) {
    if (N.nBB) k_combine<<<blocks_for(N.nBB), kThreads, 0, s>>>(N.nBB, a, N.bbM, b, N.bbS, N.bbV);
    if (N.nBD) k_combine<<<blocks_for(N.nBD), kThreads, 0, s>>>(N.nBD, a, N.bdM, b, N.bdS, N.bdV);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) err = std::string("combine: ") + cudaGetErrorString(e);
  return e == cudaSuccess;
}

bool NumericPlan::fill_raw_rows(double* bVal, cudaStream_t s, std::string& err) {
  const NumericLevel& N = levels[0];
  if (N.nBRow) k_gather_rows<double><<<blocks_for(N.nBRow), kThreads, 0, s>>>(N.nBRow, N.bSrc, N.bdV, N.bbV, bVal);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) err = std::string("operator rows: ") + cudaGetErrorString(e);
  return e == cudaSuccess;
}

namespace {

template <typename T>
void convert_boundary(const NumericLevel& N, const BoundarySymbolic& sym, const Scaled& sc, const double* invS, const double* G,
                      const double* Ss, const double* scale64, const LevelValues<T>& v, cudaStream_t s) {
  if (sym.nSub > 0) {
    k_pad_blocks<T><<<dim3(sym.nSub, kPadBlocks), kThreads, 0, s>>>(N.subPtr, N.invOff, N.invOffPad, invS, v.inv);
    k_wt<T><<<dim3(sym.nSub, kPadBlocks), kThreads, 0, s>>>(N.subPtr, N.touchPtr, N.wOff, G, v.wt);
  }
  if (sym.nS > 0) {
    const long long e = (long long)sym.nS * v.nSp;
    k_pad_square<T><<<blocks_for(e), kThreads, 0, s>>>(sym.nS, v.nSp, Ss, v.sinv);
  }
  k_convert<T><<<blocks_for(sym.nb), kThreads, 0, s>>>(sym.nb, scale64, v.scale);
  const long long nAsi = (long long)sym.ASI.col.size(), nBd = (long long)sym.BD.col.size();
  if (nAsi) k_scaled_values<T><<<blocks_for(nAsi), kThreads, 0, s>>>(nAsi, N.asiEntry, sc, v.asiVal);
  if (nBd) k_gather_values<T><<<blocks_for(nBd), kThreads, 0, s>>>(nBd, N.bdEntry, N.bdV, v.bdVal);
}

}  // namespace

void keep_pool_memory() {
  static std::atomic<int> slots[dev::kMaxDevices];
  static const bool init = [] {
    for (auto& a : slots) a.store(dev::kUnset);
    return true;
  }();
  (void)init;
  dev::per_device_once(slots, [] {
    int d = 0;
    cudaMemPool_t pool;
    if (cudaGetDevice(&d) != cudaSuccess || cudaDeviceGetDefaultMemPool(&pool, d) != cudaSuccess) return 1;
    uint64_t keep = ~0ULL;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    return 1;
  });
}

// One level's work in flight: its scratch (released in its stream's order), its
// error words on the device {subdomain inverses, Schur complement or coarsest
// inverse}, and the first launch error.
struct NumericPlan::LevelJob {
  StreamScratch S;
  LevelStream& ls;
  int* bad = nullptr;
  bool launchOk = true;
  explicit LevelJob(LevelStream& stream) : S(stream.s), ls(stream) {}
};

bool NumericPlan::ensure_streams(std::string& err) {
  cudaError_t e = cudaSuccess;
  if (!ready_) e = cudaEventCreateWithFlags(&ready_, cudaEventDisableTiming);
  if ((int)streams_.size() < L) streams_.resize(L);
  for (LevelStream& ls : streams_) {
    if (e == cudaSuccess && !ls.s) e = cudaStreamCreateWithFlags(&ls.s, cudaStreamNonBlocking);
    for (cudaEvent_t& m : ls.mark)
      if (e == cudaSuccess && !m) e = cudaEventCreate(&m);
  }
  if (e != cudaSuccess) err = std::string("set-up streams: ") + cudaGetErrorString(e);
  return e == cudaSuccess;
}

// Marks: 0 start, 1 values, 2 subdomain inverses, 3 Schur products, 4 Schur
// complement inverse, 5 end (the coarsest level: 0, 1, 5)
void NumericPlan::queue_level(int l, const LevelValues<float>* f32, const LevelValues<double>* f64, LevelJob& job) {
  const NumericLevel& N = levels[l];
  StreamScratch& S = job.S;
  cudaStream_t s = job.ls.s;
  auto mark = [&](int i) { cudaEventRecord(job.ls.mark[i], s); };
  mark(0);
  cudaMemsetAsync(job.bad, 0, 2 * sizeof(int), s);
  const Sources src{screen, stiffness, N.deepM, N.deepS, N.bdV, N.bbV};
  if (N.coarsest) {
    const int n = N.n;
    double* scale = f64 ? f64->coarseScale : f32->coarseScale;
    double* inv = f64 ? f64->coarseInv : f32->coarseInv;
    double* dense = S.get<double>(size_t(n) * n);
    double* scratch = S.get<double>(dev::spd_inverse_scratch_doubles(N.coarseLayout));
    if (dense && scratch) {
      k_coarse_scale<<<blocks_for(n), kThreads, 0, s>>>(n, N.diagSrc, src, scale);
      cudaMemsetAsync(dense, 0, size_t(n) * n * sizeof(double), s);
      k_coarse_fill<<<blocks_for(N.nDense), kThreads, 0, s>>>(N.nDense, n, N.denseSrc, N.denseRow, N.denseCol, src, scale, dense);
      mark(1);
      job.launchOk = dev::launch_spd_inverse(N.coarseLayout, N.coarseDev, dense, inv, scratch, job.bad + 1, s);
      if (f64 && f32) {
        cudaMemcpyAsync(f32->coarseInv, inv, size_t(n) * n * sizeof(double), cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(f32->coarseScale, scale, size_t(n) * sizeof(double), cudaMemcpyDeviceToDevice, s);
      }
    }
    mark(5);
    return;
  }
  // smoother planes and boundary rows
  if (N.runCount > 0) {
    if (f32) k_planes<float><<<blocks_for(N.runCount), kThreads, 0, s>>>(N.runCount, N.runTexel, N.deepM, N.deepS, screen, stiffness, f32->planes);
    if (f64) k_planes<double><<<blocks_for(N.runCount), kThreads, 0, s>>>(N.runCount, N.runTexel, N.deepM, N.deepS, screen, stiffness, f64->planes);
  }
  if (N.nBRow) {
    if (f32) k_gather_rows<float><<<blocks_for(N.nBRow), kThreads, 0, s>>>(N.nBRow, N.bSrc, N.bdV, N.bbV, f32->bVal);
    if (f64) k_gather_rows<double><<<blocks_for(N.nBRow), kThreads, 0, s>>>(N.nBRow, N.bSrc, N.bdV, N.bbV, f64->bVal);
  }
  const BoundarySymbolic& sym = N.sym;
  const int nS = sym.nb > 0 ? sym.nS : 0;
  // boundary solver: scaled subdomain blocks, their inverses
  const long long elems = std::max<long long>(1, N.subLayout.elems);
  const long long wTotal = sym.nb > 0 ? std::max<int64_t>(1, sym.wOff.back()) : 1, lTotal = sym.nb > 0 ? std::max<int64_t>(1, sym.lOff.back()) : 1;
  double *scale64 = nullptr, *blk = nullptr, *invS = nullptr, *C = nullptr, *G = nullptr, *Lc = nullptr, *subScratch = nullptr;
  double *Ss = nullptr, *Sm = nullptr, *schurScratch = nullptr;
  if (sym.nb > 0) {
    scale64 = S.get<double>(sym.nb);
    blk = S.get<double>(elems);
    invS = S.get<double>(elems);
    C = S.get<double>(wTotal);
    G = S.get<double>(wTotal);
    Lc = S.get<double>(lTotal);
    subScratch = S.get<double>(std::max<size_t>(1, dev::spd_inverse_scratch_doubles(N.subLayout)));
    if (nS > 0) {
      Sm = S.get<double>(size_t(nS) * nS);
      Ss = S.get<double>(size_t(nS) * nS);
      schurScratch = S.get<double>(dev::spd_inverse_scratch_doubles(N.schurLayout));
    }
  }
  if (sym.nb == 0 || S.last != cudaSuccess) {
    for (int i = 1; i < kMarks; i++) mark(i);
    return;
  }
  k_scale_pos<<<blocks_for(sym.nb), kThreads, 0, s>>>(sym.nb, N.order, N.diagEntry, N.bbV, scale64);
  const Scaled sc{N.bbV, N.bbRow, N.bbCol, N.pos, scale64};
  cudaMemsetAsync(blk, 0, size_t(elems) * sizeof(double), s);
  const long long nFill = (long long)sym.fillEntry.size();
  if (nFill) k_scatter_scaled<<<blocks_for(nFill), kThreads, 0, s>>>(nFill, N.fillEntry, N.fillDest, sc, blk);
  mark(1);
  job.launchOk = dev::launch_spd_inverse(N.subLayout, N.subDev, blk, invS, subScratch, job.bad, s);
  mark(2);
  // couplings, back-substitution blocks G_p = Inv_p C_p, Schur complement
  cudaMemsetAsync(C, 0, size_t(wTotal) * sizeof(double), s);
  const long long nAis = (long long)sym.aisDest.size();
  if (nAis) k_scatter_scaled<<<blocks_for(nAis), kThreads, 0, s>>>(nAis, N.aisEntry, N.aisDest, sc, C);
  dev::launch_gemm_batch(N.gTasksDev, (int)N.gTasks.size(), N.maxM, N.maxT, invS, C, G, s);
  if (nS > 0) {
    dev::launch_gemm_batch(N.lTasksDev, (int)N.lTasks.size(), N.maxT, N.maxT, C, G, Lc, s);
    cudaMemsetAsync(Sm, 0, size_t(nS) * nS * sizeof(double), s);
    const long long nSS = (long long)sym.ssEntry.size();
    if (nSS) k_scatter_scaled<<<blocks_for(nSS), kThreads, 0, s>>>(nSS, N.ssEntry, N.ssDest, sc, Sm);
    if (sym.nSub > 0) k_schur_subtract<<<(nS + kRowsPerBlock - 1) / kRowsPerBlock, kThreads, 0, s>>>(nS, sym.nSub, N.touchPtr, N.touch, N.lOff, Lc, Sm);
    k_symmetrise_pairs<<<blocks_for((long long)nS * nS), kThreads, 0, s>>>(nS, Sm);
  }
  mark(3);
  if (nS > 0) job.launchOk = dev::launch_spd_inverse(N.schurLayout, N.schurDev, Sm, Ss, schurScratch, job.bad + 1, s) && job.launchOk;
  mark(4);
  if (f32) convert_boundary(N, sym, sc, invS, G, Ss, scale64, *f32, s);
  if (f64) convert_boundary(N, sym, sc, invS, G, Ss, scale64, *f64, s);
  mark(5);
}

// What bounds it: each level is a chain of small dependent launches (an
// elimination step of the coarsest matrix is two), some 100 in all for 1024^2, and
// the levels in turn left most of the chip idle.  Side by side the chains of level 0
// and of the coarsest level, queued first, hide the others: re-weighting and solve
// 13.35 -> 9.4 ms (5.0 with the later, faster inverses).  The coarsest level's stream
// at a higher priority: 5.35, level 0 waits.
bool NumericPlan::fill_levels(const std::vector<LevelValues<float>>& f32, const std::vector<LevelValues<double>>& f64, cudaStream_t s,
                              std::string& err) {
  if (!ensure_streams(err)) return false;
  std::vector<int> badHost(2 * size_t(L), 0);
  std::vector<std::unique_ptr<LevelJob>> jobs(L);
  StreamScratch words(s);
  int* bad = words.get<int>(2 * size_t(L));
  if (!bad) {
    cudaGetLastError();
    err = std::string("numeric scratch: ") + cudaGetErrorString(words.last);
    return false;
  }
  // a level on its stream, after the work queued on s
  auto queue = [&](int l) -> cudaError_t {
    const cudaError_t w = cudaStreamWaitEvent(streams_[l].s, ready_, 0);
    if (w != cudaSuccess) return w;
    jobs[l].reset(new LevelJob(streams_[l]));
    jobs[l]->bad = bad + 2 * l;
    queue_level(l, f32.empty() ? nullptr : &f32[l], f64.empty() ? nullptr : &f64[l], *jobs[l]);
    return cudaSuccess;
  };
  // s continues after every level that was queued, also after an error; the error words
  auto finish = [&](cudaError_t e) -> cudaError_t {
    for (int l = 0; l < L; l++)
      if (jobs[l]) {
        const cudaError_t w = cudaStreamWaitEvent(s, streams_[l].mark[kMarks - 1], 0);
        if (e == cudaSuccess) e = w;
      }
    const cudaError_t d = cudaMemcpyAsync(badHost.data(), bad, badHost.size() * sizeof(int), cudaMemcpyDeviceToHost, s);
    const cudaError_t y = cudaStreamSynchronize(s);
    const cudaError_t last = cudaGetLastError();
    for (cudaError_t q : {d, y, last})
      if (e == cudaSuccess) e = q;
    return e;
  };
  auto order = [this](int i) { return i == 0 ? L - 1 : i - 1; };  // the longest chain first
  auto scratch_failed = [&] {
    for (int l = 0; l < L; l++)
      if (jobs[l] && jobs[l]->S.last != cudaSuccess) return l;
    return -1;
  };
  cudaError_t e = cudaEventRecord(ready_, s);
  for (int i = 0; i < L && e == cudaSuccess; i++) e = queue(order(i));
  e = finish(e);
  if (scratch_failed() >= 0) {
    // no room for the scratch of all levels at once (their sum): in turn, each giving its
    // scratch back before the next, so that the largest level's is enough
    e = cudaSuccess;
    for (int i = 0; i < L && e == cudaSuccess && (i == 0 || scratch_failed() < 0); i++) {
      for (int l = 0; l < L; l++) {
        jobs[l].reset();
        if (e == cudaSuccess) e = cudaStreamSynchronize(streams_[l].s);
      }
      int device = 0;
      cudaMemPool_t pool;
      if (cudaGetDevice(&device) == cudaSuccess && cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) cudaMemPoolTrimTo(pool, 0);
      if (e == cudaSuccess) e = queue(order(i));
      e = finish(e);
      const int l = order(i);
      if (jobs[l] && scratch_failed() < 0 && !jobs[l]->launchOk) break;
      if (badHost[2 * size_t(l)] || badHost[2 * size_t(l) + 1]) break;
    }
  }
  const int starved = scratch_failed();
  for (int l = 0; l < L; l++) {
    const std::string where = l == L - 1 ? "coarsest level: " : "level " + std::to_string(l) + ": ";
    if (l == starved) {
      err = where + "scratch: " + cudaGetErrorString(jobs[l]->S.last);
      return false;
    }
    if (jobs[l] && e == cudaSuccess && !jobs[l]->launchOk) {
      err = where + "inverse launch failed";
      return false;
    }
  }
  if (e != cudaSuccess) {
    err = std::string("numeric set-up: ") + cudaGetErrorString(e);
    return false;
  }
  for (int l = 0; l < L; l++)
    for (int w = 0; w < 2; w++)
      if (badHost[2 * size_t(l) + w]) {
        err = (l == L - 1 ? std::string("coarsest level: coarsest inverse") : "level " + std::to_string(l) + ": " +
               (w == 0 ? "boundary subdomain inverses" : "boundary Schur complement inverse")) + ": not positive definite";
        return false;
      }
  // phases, from the marks
  std::fill(ms, ms + 4, 0.0);
  boundaryMs = coarseMs = 0;
  auto between = [&](cudaEvent_t a, cudaEvent_t b) {
    float t = 0;
    return cudaEventElapsedTime(&t, a, b) == cudaSuccess ? double(t) : 0.0;
  };
  const cudaEvent_t first = streams_[L - 1].mark[0];
  for (int l = 0; l + 1 < L; l++) {
    const cudaEvent_t* m = streams_[l].mark;
    ms[0] += between(m[0], m[1]) + between(m[4], m[5]);
    for (int q = 1; q < 4; q++) ms[q] += between(m[q], m[q + 1]);
    boundaryMs = std::max(boundaryMs, between(first, m[5]));
  }
  coarseMs = std::max(0.0, between(first, streams_[L - 1].mark[5]) - boundaryMs);
  // the levels overlap: the phases as shares of the time they took together
  const double sum = ms[0] + ms[1] + ms[2] + ms[3];
  if (sum > boundaryMs)
    for (double& t : ms) t *= boundaryMs / sum;
  return true;
}

}  // namespace gdtp
