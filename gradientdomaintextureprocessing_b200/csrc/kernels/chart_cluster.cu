// Chart smoother on a thread-block cluster: every sweep of one smoothing step
// (IterativeSolvers.inl:174-395 restated as 4-colour Gauss-Seidel) in one launch,
// a chart on the CTAs of a cluster (charts that need few of them share one).
//
// Deep texels of different charts never neighbour each other and the sweeps do
// not change boundary texels, so a chart is independent of the others.  The
// chart's rows are dealt to its CTAs (contiguous rows, balanced by
// texels); a CTA keeps its rows' x, with the row above and the row below, in
// shared memory (the slab), and its coefficients and right-hand side in
// registers or shared memory, for all sweeps.  One half sweep updates the rows of
// one parity (their 9-point stencils reach only their own row and the other
// parity's): first colour, block barrier, second colour.  Updates in a CTA's
// first or last row are also stored into the neighbouring CTA's slab (distributed
// shared memory), and a cluster barrier ends the half sweep.
//
// Races: in a half sweep of parity p a neighbour's slab receives rows of parity p
// next to its own rows of parity 1 - p, which read them in the next half sweep,
// after the barrier.  The first half sweep's stores come after the barrier that
// follows the slab loads; the last half sweep stores nothing remotely, so no CTA
// is written after its last barrier.
//
// Every update is gs_item's sum in gs_item's order: the result is the colour
// passes', bit for bit.
//
// What bounds it: on the levels below the finest, and on whole problems up to about
// 1024^2, a sweep is a chain of latencies, not bytes.  As two row launches it took
// 5.5 us (launch, x through L2, two block barriers, each time); a sweep more in here
// takes 1.9 us (256^2 torus, 8 CTAs a chart), and a smoothing step of 3 sweeps 12
// instead of 22 us.  Per refinement step: 256^2 torus 187 -> 134 us, 1024^2 genus-2
// (one channel) 209 -> 153 us.
// Which charts: up to 512 pairs of one row parity in each of 8 CTAs, the coefficients
// in registers; larger ones, up to 1024 pairs with the coefficients in shared memory
// (one CTA per SM), where one wave holds every cluster: 15 are resident, and a second
// wave takes as long as the row launches (42 us against 36 for 3 sweeps).  Smaller
// charts share a cluster's CTAs (build_chart_clusters): the 8 large and 8 small charts
// of a 1024^2 icosphere atlas are 12 clusters, not 16, so its level 0 runs in one wave:
// 305 -> 275 us per refinement step.  Fewer CTAs for small charts elsewhere: 725 x 611
// with 15 right-hand sides 413 -> 400, 256^2 torus 117 -> 112, 1024^2 genus-2 (one
// channel) 130.4 -> 127.7, FP64 values at 1024^2 399 -> 393 us.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "vcycle.cuh"
#include "vcycle_kernels.h"
#include "vcycle_ops.cuh"

namespace cg = cooperative_groups;

namespace gdtp {
namespace dev {
namespace {

// Slab slot of texel i: threads of a line touch every other texel, so the lowest
// bit is mixed with the one that would bring two of them onto one bank.  Texels 2j
// and 2j + 1 may swap places, so a slab holds an even number of entries.
template <typename T, int W>
__device__ __forceinline__ int slab_slot(int i) {
  constexpr int kShift = sizeof(Vec<T, W>) == 4 ? 5 : sizeof(Vec<T, W>) == 8 ? 4 : sizeof(Vec<T, W>) == 16 ? 3 : 2;
  return i ^ ((i >> kShift) & 1);
}

// A thread's pair of texels of one row parity, first-updated colour A, then B
struct PairPos {
  int mA = 0;               // slab index of A
  int dB = 0;               // B = A + dB (+1 or -1)
  int up = 0, dn = 0;       // distance to the rows above and below
  int flags = 0;            // 1: A, 2: B, 4: push up, 8: push down
  int cA = 0, cB = 0;       // coefficient indices
};

__device__ __forceinline__ PairPos load_pair(const ClusterItem& it, int lo, int oddFirst) {
  PairPos p;
  const int has1 = (it.pos >> kItemPairBit) & 1, odd = (it.pos >> kItemOddBit) & 1;
  const int a = (odd == oddFirst) ? 0 : 1;  // texel of the pair with the first colour
  p.mA = (it.pos & kItemPosMask) - lo + a;
  p.dB = 1 - 2 * a;
  p.up = it.dist & 0xffff;
  p.dn = (it.dist >> 16) & 0xffff;
  p.flags = ((a == 0 || has1) ? 1 : 0) | ((a == 1 || has1) ? 2 : 0) | (((it.pos >> kItemUpBit) & 3) << 2);
  p.cA = a ? it.c1 : it.c0;
  p.cB = a ? it.c0 : it.c1;
  return p;
}

// an asynchronous copy of a texel's values
template <typename T, int W>
__device__ __forceinline__ void async_vec(Vec<T, W>* dst, const T* src) {
  constexpr int kBytes = sizeof(Vec<T, W>), kStep = kBytes < 16 ? kBytes : 16;
#pragma unroll
  for (int b = 0; b < kBytes; b += kStep) copy_async<kStep>(reinterpret_cast<char*>(dst) + b, reinterpret_cast<const char*>(src) + b);
}

template <typename T, int W>
struct Slab {
  Vec<T, W>* x;             // this CTA's slab
  Vec<T, W>* xUp;           // the neighbours' (the CTAs of the rows above and below)
  Vec<T, W>* xDn;
  int upShift, dnShift;     // slab index here -> slab index there
  int upCount, dnCount;
  __device__ __forceinline__ Vec<T, W> at(int i) const { return x[slab_slot<T, W>(i)]; }
  __device__ __forceinline__ void put(int i, const Vec<T, W>& v, int flags, bool push) const {
    x[slab_slot<T, W>(i)] = v;
    if (!push) return;
    if (flags & 4) {
      const int j = i + upShift;
      if (j >= 0 && j < upCount) xUp[slab_slot<T, W>(j)] = v;
    }
    if (flags & 8) {
      const int j = i + dnShift;
      if (j >= 0 && j < dnCount) xDn[slab_slot<T, W>(j)] = v;
    }
  }
};

// One half sweep of a thread's pair; w(k): coefficient k of A (k < 9) or of B
// (9 + k); rhs(0), rhs(1): the right-hand side of A and B.  EARLY: B's row below is
// read before the barrier too (registers allowing)
template <typename T, int W, bool EARLY, typename Coef, typename Rhs>
__device__ __forceinline__ void half_sweep(const Slab<T, W>& s, const PairPos& p, const Coef& w, const Rhs& rhs, bool push) {
  const int mA = p.mA, mB = p.mA + p.dB;
  if (p.flags & 1) {
    Vec<T, W> acc;
#pragma unroll
    for (int k = 0; k < W; k++) acc.v[k] = 0;
    fma_to(acc, w(0), s.at(mA - p.up - 1));
    fma_to(acc, w(1), s.at(mA - p.up));
    fma_to(acc, w(2), s.at(mA - p.up + 1));
    fma_to(acc, w(3), s.at(mA - 1));
    fma_to(acc, w(5), s.at(mA + 1));
    fma_to(acc, w(6), s.at(mA + p.dn - 1));
    fma_to(acc, w(7), s.at(mA + p.dn));
    fma_to(acc, w(8), s.at(mA + p.dn + 1));
    const Vec<T, W> b = rhs(0);
    const T c4 = w(4);
    Vec<T, W> out;
#pragma unroll
    for (int k = 0; k < W; k++) out.v[k] = fma(b.v[k], c4, -acc.v[k]);
    s.put(mA, out, p.flags, push);
  }
  // B's rows above and below do not change: read before the barrier
  Vec<T, W> acc, d0, d1, d2;
#pragma unroll
  for (int k = 0; k < W; k++) acc.v[k] = 0;
  if (p.flags & 2) {
    fma_to(acc, w(9 + 0), s.at(mB - p.up - 1));
    fma_to(acc, w(9 + 1), s.at(mB - p.up));
    fma_to(acc, w(9 + 2), s.at(mB - p.up + 1));
    if (EARLY) {
      d0 = s.at(mB + p.dn - 1);
      d1 = s.at(mB + p.dn);
      d2 = s.at(mB + p.dn + 1);
    }
  }
  __syncthreads();
  if (p.flags & 2) {
    if (!EARLY) {
      d0 = s.at(mB + p.dn - 1);
      d1 = s.at(mB + p.dn);
      d2 = s.at(mB + p.dn + 1);
    }
    fma_to(acc, w(9 + 3), s.at(mB - 1));
    fma_to(acc, w(9 + 5), s.at(mB + 1));
    fma_to(acc, w(9 + 6), d0);
    fma_to(acc, w(9 + 7), d1);
    fma_to(acc, w(9 + 8), d2);
    const Vec<T, W> b = rhs(1);
    const T c4 = w(9 + 4);
    Vec<T, W> out;
#pragma unroll
    for (int k = 0; k < W; k++) out.v[k] = fma(b.v[k], c4, -acc.v[k]);
    s.put(mB, out, p.flags, push);
  }
}

// CREG / BREG: coefficients / right-hand side in registers (else in shared memory);
// MINB: CTAs per SM the registers are limited for
template <typename T, int W, int MAXT, int MINB, bool CREG, bool BREG>
__global__ void __launch_bounds__(MAXT, MINB) k_gs_cluster(const ClusterPart* __restrict__ parts, const ClusterItem* __restrict__ items,
                                                       int slabMax, const T* __restrict__ coef, int planeStride,
                                                       const T* __restrict__ rhs, T* __restrict__ x, int KP, int sweeps, int reverse,
                                                       int zeroStart, int rhsEarly) {
  extern __shared__ __align__(32) unsigned char smem_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int nt = blockDim.x, tid = threadIdx.x;
  const ClusterPart& part = parts[blockIdx.x];
  struct { int lo, count, upLo, upCount, dnLo, dnCount; } P = {part.lo, part.count, part.upLo, part.upCount, part.dnLo, part.dnCount};
  const int off = blockIdx.y * W;
  Slab<T, W> slab;
  slab.x = reinterpret_cast<Vec<T, W>*>(smem_raw);
  slab.xUp = rank > 0 ? cluster.map_shared_rank(slab.x, rank - 1) : slab.x;
  slab.xDn = rank + 1 < C ? cluster.map_shared_rank(slab.x, rank + 1) : slab.x;
  slab.upShift = P.lo - P.upLo;
  slab.dnShift = P.lo - P.dnLo;
  slab.upCount = P.upCount;
  slab.dnCount = P.dnCount;
  Vec<T, W>* sb = slab.x + slabMax;                                       // [4][nt] unless BREG
  T* sw = reinterpret_cast<T*>(sb + (BREG ? 0 : 4 * (size_t)nt));         // [36][nt] unless CREG

  // set-up data, and the right-hand side when the previous launch does not write
  // it, before waiting for that launch
  const int first = reverse ? 1 : 0;  // row parity of the first half sweep
  PairPos pos[2];
  T wr[2][CREG ? 18 : 1];
  Vec<T, W> br[2][BREG ? 2 : 1];
  auto load_rhs = [&](int h) {
    const long long gA = (long long)(P.lo + pos[h].mA) * KP + off, gB = (long long)(P.lo + pos[h].mA + pos[h].dB) * KP + off;
    if (pos[h].flags & 1) {
      if constexpr (BREG) br[h][0] = vload<T, W>(rhs + gA);
      else async_vec<T, W>(&sb[(2 * h) * nt + tid], rhs + gA);
    }
    if (pos[h].flags & 2) {
      if constexpr (BREG) br[h][1] = vload<T, W>(rhs + gB);
      else async_vec<T, W>(&sb[(2 * h + 1) * nt + tid], rhs + gB);
    }
  };
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int par = h ? 1 - first : first;
    if (tid < part.nItems[par]) {
      pos[h] = load_pair(items[part.item0[par] + tid], P.lo, reverse);
      const T *cA = coef + pos[h].cA, *cB = coef + pos[h].cB;
#pragma unroll
      for (int k = 0; k < 9; k++) {
        if constexpr (CREG) {
          if (pos[h].flags & 1) wr[h][k] = cA[(long long)k * planeStride];
          if (pos[h].flags & 2) wr[h][9 + k] = cB[(long long)k * planeStride];
        } else {
          if (pos[h].flags & 1) copy_async<sizeof(T)>(&sw[(18 * h + k) * nt + tid], cA + (long long)k * planeStride);
          if (pos[h].flags & 2) copy_async<sizeof(T)>(&sw[(18 * h + 9 + k) * nt + tid], cB + (long long)k * planeStride);
        }
      }
      if (rhsEarly) load_rhs(h);
    }
  }
  grid_dependency_wait();
  grid_launch_dependents();
  if (zeroStart) {
    Vec<T, W> z;
#pragma unroll
    for (int k = 0; k < W; k++) z.v[k] = 0;
    for (int i = tid; i < P.count; i += nt) slab.x[slab_slot<T, W>(i)] = z;
  } else {
    for (int i = tid; i < P.count; i += nt) async_vec<T, W>(&slab.x[slab_slot<T, W>(i)], x + (long long)(P.lo + i) * KP + off);
  }
  if (!rhsEarly) {
    load_rhs(0);
    load_rhs(1);
  }
  copies_wait_all();  // this thread's copies; the barrier then orders every thread's
  if (C > 1) cluster.sync(); else __syncthreads();

  auto half = [&](auto hc, bool push) {
    constexpr int h = decltype(hc)::value;
    half_sweep<T, W, (MINB == 1 && MAXT <= kClusterMaxThreads)>(
        slab, pos[h], [&](int k) -> T { return CREG ? wr[h][CREG ? k : 0] : sw[(18 * h + k) * nt + tid]; },
        [&](int k) -> Vec<T, W> { return BREG ? br[h][BREG ? k : 0] : sb[(2 * h + k) * nt + tid]; }, push);
  };
  for (int sweep = 0; sweep < sweeps; sweep++) {
    half(std::integral_constant<int, 0>(), C > 1);
    if (C > 1) cluster.sync(); else __syncthreads();
    const bool last = sweep == sweeps - 1;
    half(std::integral_constant<int, 1>(), C > 1 && !last);
    if (last) break;
    if (C > 1) cluster.sync(); else __syncthreads();
  }
  // this thread's own texels (their last update is its own store)
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int mA = pos[h].mA, mB = mA + pos[h].dB;
    if (pos[h].flags & 1) vstore<T, W>(x + (long long)(P.lo + mA) * KP + off, slab.at(mA));
    if (pos[h].flags & 2) vstore<T, W>(x + (long long)(P.lo + mB) * KP + off, slab.at(mB));
  }
}

template <typename T, int W, bool CREG, bool BREG>
size_t cluster_smem(int slabMax, int threads) {
  return size_t(slabMax) * sizeof(Vec<T, W>) + (BREG ? 0 : size_t(4) * threads * sizeof(Vec<T, W>)) + (CREG ? 0 : size_t(36) * threads * sizeof(T));
}

// shared memory attribute set, and the clusters resident at the largest size (per
// device, once)
template <typename T, int W, int MAXT, int MINB, bool CREG, bool BREG>
int cluster_ready() {
  static std::atomic<int> slots[kMaxDevices];
  static const bool init = [] {
    for (auto& v : slots) v.store(kUnset);
    return true;
  }();
  (void)init;
  return per_device_once(slots, [] {
    auto kern = k_gs_cluster<T, W, MAXT, MINB, CREG, BREG>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kClusterSmemMax)) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(8);
    cfg.blockDim = dim3(MAXT);
    cfg.dynamicSmemBytes = kClusterSmemMax;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {8, 1, 1};
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return clusters;
  });
}

// Most CTAs per SM of one launch with several channel groups, each of which loads the
// coefficients again, or with FP64 charts of more than one CTA: beyond a few waves the
// colour passes keep up (64 right-hand sides at 1024^2, level 1: 92 us against 80; 256
// charts of a 1024^2 atlas in FP64 270 against 261).  FP32 values of up to 4 channels and
// charts of one CTA have no limit: 3 pre- and 3 post-sweeps of level 0 at 1024^2 in 1024
// charts 72 us with clusters, 143 with a block per chart (3 channels; FP64 178 and 247), in
// 576 charts 89 against 134 with the row launches, in 256 106 against 132.  Per refinement
// step of 3 channels: 1024 charts 2853 -> 2740 us, 576 1629 -> 1558, 256 806 -> 756.
constexpr int kClusterMaxCtasPerSm = 4;

template <typename T, int W, int MAXT, int MINB, bool CREG, bool BREG>
bool cluster_fits(const LevelDev<T>& D) {
  return D.clusterThreads > 0 && D.clusterThreads <= MAXT &&
         cluster_smem<T, W, CREG, BREG>(D.clusterSlab, D.clusterThreads) <= kClusterSmemMax && cluster_ready<T, W, MAXT, MINB, CREG, BREG>() > 0;
}

template <typename T, int W, int MAXT, int MINB, bool CREG, bool BREG>
bool launch_variant(const LevelDev<T>& D, int sweeps, bool reverse, bool zeroStart, int KP, cudaStream_t s, bool rhsEarly) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(D.nClusterParts), unsigned(KP / W));
  cfg.blockDim = dim3(unsigned(D.clusterThreads));
  cfg.dynamicSmemBytes = cluster_smem<T, W, CREG, BREG>(D.clusterSlab, D.clusterThreads);
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim = {unsigned(D.clusterSize), 1, 1};
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = programmatic_launch() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, k_gs_cluster<T, W, MAXT, MINB, CREG, BREG>, D.clusterParts, D.clusterItems, D.clusterSlab, D.coef, D.planeStride,
                            static_cast<const T*>(D.b), D.x, KP, sweeps, reverse ? 1 : 0, zeroStart ? 1 : 0,
                            rhsEarly ? 1 : 0) == cudaSuccess;
}

}  // namespace

// the large layout: in one wave (one CTA per SM), its coefficients in shared memory
template <typename T, int W>
static bool large_in_one_wave(const LevelDev<T>& D, int KP) {
  return cluster_fits<T, W, kClusterLargeThreads, 1, false, true>(D) &&
         (long long)(D.nClusterParts / D.clusterSize) * (KP / W) <= cluster_ready<T, W, kClusterLargeThreads, 1, false, true>();
}

template <typename T, int W>
bool gs_cluster_available(const LevelDev<T>& D, int KP) {
  if (D.clusterThreads == 0) return false;
  const bool limited = KP / W > 1 || (sizeof(T) == 8 && D.clusterSize > 1);
  if (limited && (long long)D.nClusterParts * (KP / W) > (long long)kClusterMaxCtasPerSm * device_sms()) return false;
  if constexpr (std::is_same<T, float>::value)
    return cluster_fits<T, W, 320, 2, true, false>(D) || cluster_fits<T, W, 512, 1, true, true>(D) || large_in_one_wave<T, W>(D, KP);
  else
    return cluster_fits<T, W, 512, 1, false, false>(D);
}

// Up to 320 pairs: registers limited to 96, so that two CTAs share an SM and the
// resident clusters double (a 1024^2 genus-2 step with one channel 155 -> 153 us, no
// difference with four); up to 512: one CTA per SM, the right-hand side in registers
// too.  FP64 values keep both in shared memory.
template <typename T, int W>
bool launch_gs_cluster(const LevelDev<T>& D, int sweeps, bool reverse, bool zeroStart, int KP, cudaStream_t s, bool rhsEarly) {
  if (sweeps <= 0) return true;
  if constexpr (std::is_same<T, float>::value) {
    if (cluster_fits<T, W, 320, 2, true, false>(D)) return launch_variant<T, W, 320, 2, true, false>(D, sweeps, reverse, zeroStart, KP, s, rhsEarly);
    if (cluster_fits<T, W, 512, 1, true, true>(D)) return launch_variant<T, W, 512, 1, true, true>(D, sweeps, reverse, zeroStart, KP, s, rhsEarly);
    if (large_in_one_wave<T, W>(D, KP))
      return launch_variant<T, W, kClusterLargeThreads, 1, false, true>(D, sweeps, reverse, zeroStart, KP, s, rhsEarly);
  } else {
    if (cluster_fits<T, W, 512, 1, false, false>(D)) return launch_variant<T, W, 512, 1, false, false>(D, sweeps, reverse, zeroStart, KP, s, rhsEarly);
  }
  return false;
}

#define GDTP_CLUSTER(T, W)                                                                       \
  template bool gs_cluster_available<T, W>(const LevelDev<T>&, int);                             \
  template bool launch_gs_cluster<T, W>(const LevelDev<T>&, int, bool, bool, int, cudaStream_t, bool);
GDTP_CLUSTER(float, 1)
GDTP_CLUSTER(float, 4)
GDTP_CLUSTER(double, 1)
GDTP_CLUSTER(double, 4)

}  // namespace dev
}  // namespace gdtp
