// The cluster chart smoother's layout (build_chart_clusters, csrc/system.cu) run on
// the host: every CTA's slab, its pairs, the stores into the neighbouring CTAs'
// slabs and the half sweeps, as kernels/chart_cluster.cu orders them, against
// 4-colour Gauss-Seidel over the colour runs on the whole vector.  Checks that
// every index lies in its slab or plane, that an update never reads a slab entry
// another CTA has changed since the last barrier, and that the result is the
// colour passes' bit for bit.
//
//   chart_cluster_check <mesh.gdm> <levels> <sweeps>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <cstdlib>
#include <fstream>
#include <random>
#include <string>
#include <vector>

#include "system.h"

using namespace gdtp;

namespace {

template <class T>
bool rd(std::ifstream& f, T* p, size_t n) {
  return bool(f.read(reinterpret_cast<char*>(p), std::streamsize(n * sizeof(T))));
}
bool read_gdm(const char* path, Mesh& m, int& width, int& height) {
  std::ifstream f(path, std::ios::binary);
  char magic[8];
  int64_t h[5];
  if (!rd(f, magic, 8) || !rd(f, h, 5)) return false;
  m.vertices.resize(size_t(h[0]) * 3), m.triangles.resize(size_t(h[1]) * 3), m.uv.resize(size_t(h[1]) * 6);
  width = int(h[2]), height = int(h[3]);
  return rd(f, m.vertices.data(), m.vertices.size()) && rd(f, m.triangles.data(), m.triangles.size()) &&
         rd(f, m.uv.data(), m.uv.size());
}

[[noreturn]] void die(const std::string& what) {
  std::fprintf(stderr, "%s\n", what.c_str());
  std::exit(1);
}

float update(const std::vector<float>& w, int plane, int c, float rhs, const float (&n)[9]) {
  float acc = 0;
  for (int k = 0; k < 9; k++)
    if (k != 4) acc = std::fmaf(w[size_t(k) * plane + c], n[k], acc);
  return std::fmaf(rhs, w[size_t(4) * plane + c], -acc);
}

}  // namespace

int main(int argc, char** argv) {
  if (argc != 4) die("usage: chart_cluster_check mesh.gdm levels sweeps");
  Mesh mesh;
  int width = 0, height = 0;
  if (!read_gdm(argv[1], mesh, width, height)) die("mesh");
  Hierarchy H;
  if (!build_hierarchy(mesh, width, height, std::atoi(argv[2]), BlockInfo(), H, 0, 8)) die(H.error);
  const int sweeps = std::atoi(argv[3]);
  int checked = 0;
  for (size_t l = 0; l < H.levels.size(); l++) {
    const GridLevel& L = H.levels[l];
    const DeepRuns R = build_deep_runs(L);
    ChartClusters cc;
    if (!build_chart_clusters(L, R, cc)) continue;
    checked++;
    if (cc.slab % 2) die("odd slab: the kernel swaps entries within pairs");
    std::mt19937 gen(7);
    std::uniform_real_distribution<float> u(-1.f, 1.f);
    std::vector<float> w(size_t(10) * R.count), rhs(L.numTexels), x0(L.numTexels);
    for (float& v : w) v = u(gen);
    for (float& v : rhs) v = u(gen);
    for (float& v : x0) v = u(gen);
    for (int reverse = 0; reverse < 2; reverse++) {
      // colour passes on the whole vector
      std::vector<float> ref = x0;
      for (int s = 0; s < sweeps; s++)
        for (int cc4 = 0; cc4 < 4; cc4++) {
          const int c = reverse ? 3 - cc4 : cc4;
          for (int r = R.runStart[c]; r < R.runStart[c + 1]; r++)
            for (int m = 0; m < R.runs[r].len; m++) {
              const int p = R.runs[r].pos0 + 2 * m, up = R.runs[r].prev0 + 2 * m, dn = R.runs[r].next0 + 2 * m;
              const float n[9] = {ref[up - 1], ref[up], ref[up + 1], ref[p - 1], ref[p], ref[p + 1], ref[dn - 1], ref[dn], ref[dn + 1]};
              ref[p] = update(w, R.count, R.runs[r].coef0 + m, rhs[p], n);
            }
        }
      // clusters
      std::vector<float> got = x0;
      std::vector<char> owned(L.numTexels, 0);
      const int C = cc.size;
      if (cc.parts.size() % C) die("parts are not whole clusters");
      for (size_t base = 0; base < cc.parts.size(); base += C) {
        std::vector<std::vector<float>> slab(C);
        for (int p = 0; p < C; p++) {
          const dev::ClusterPart& P = cc.parts[base + p];
          if (P.count > cc.slab || P.lo < 0 || P.lo + P.count > L.numTexels) die("slab range");
          slab[p].assign(x0.begin() + P.lo, x0.begin() + P.lo + P.count);
        }
        for (int hs = 0; hs < 2 * sweeps; hs++) {
          const int par = (reverse ? 1 : 0) ^ (hs & 1);
          const bool push = C > 1 && hs < 2 * sweeps - 1;
          // remote stores of this half sweep, visible after the barrier that ends it
          struct Remote { int part, at; float v; };
          std::vector<Remote> remote;
          for (int colour = 0; colour < 2; colour++)
            for (int p = 0; p < C; p++) {
              const dev::ClusterPart& P = cc.parts[base + p];
              if (P.nItems[par] > cc.threads) die("more pairs than threads");
              std::vector<std::pair<int, float>> stores;
              for (int t = 0; t < P.nItems[par]; t++) {
                const size_t ii = size_t(P.item0[par]) + t;
                if (ii >= cc.items.size()) die("item index");
                const dev::ClusterItem& it = cc.items[ii];
                const int has1 = (it.pos >> dev::kItemPairBit) & 1, odd = (it.pos >> dev::kItemOddBit) & 1;
                const int a0 = odd == reverse ? 0 : 1, a = colour == 0 ? a0 : 1 - a0;
                if (a == 1 && !has1) continue;
                const int g = (it.pos & dev::kItemPosMask) + a, m = g - P.lo, d1 = it.dist & 0xffff, d2 = (it.dist >> 16) & 0xffff;
                const int c = a ? it.c1 : it.c0;
                if (c < 0 || c >= R.count) die("coefficient index");
                if (m - d1 - 1 < 0 || m + d2 + 1 >= P.count || m - 1 < 0 || m + 1 >= P.count) die("stencil outside the slab");
                if (hs < 2 && !owned[g]) owned[g] = 1;
                const std::vector<float>& s = slab[p];
                const float n[9] = {s[m - d1 - 1], s[m - d1], s[m - d1 + 1], s[m - 1], s[m], s[m + 1], s[m + d2 - 1], s[m + d2], s[m + d2 + 1]};
                const float v = update(w, R.count, c, rhs[g], n);
                stores.emplace_back(m, v);
                if (push && ((it.pos >> dev::kItemUpBit) & 1)) {
                  if (p == 0) die("store above the first CTA");
                  const int j = g - P.upLo;
                  if (P.upLo != cc.parts[base + p - 1].lo || P.upCount != cc.parts[base + p - 1].count) die("slab above");
                  if (j >= 0 && j < P.upCount) remote.push_back({p - 1, j, v});
                }
                if (push && ((it.pos >> (dev::kItemUpBit + 1)) & 1)) {
                  if (p + 1 >= C) die("store below the last CTA");
                  const int j = g - P.dnLo;
                  if (P.dnLo != cc.parts[base + p + 1].lo || P.dnCount != cc.parts[base + p + 1].count) die("slab below");
                  if (j >= 0 && j < P.dnCount) remote.push_back({p + 1, j, v});
                }
                if (hs == 2 * sweeps - 1 || hs == 2 * sweeps - 2) got[g] = v;
              }
              for (auto& st : stores) slab[p][st.first] = st.second;
            }
          for (const Remote& r : remote) slab[r.part][r.at] = r.v;
        }
      }
      int deep = 0;
      for (char o : owned) deep += o;
      if (deep != R.count) die("not every deep texel has an owner");
      for (int i = 0; i < L.numTexels; i++)
        if (std::memcmp(&got[i], &ref[i], 4)) die("level " + std::to_string(l) + ": texel " + std::to_string(i) + " differs");
    }
    std::printf("level %zu: %d texels, %zu parts of clusters of %d, %d threads, slab %d\n", l, L.numTexels, cc.parts.size(), cc.size,
                cc.threads, cc.slab);
  }
  if (!checked) die("no level has a cluster layout");
  return 0;
}
