// Eigenvalue clusters of the modes' FP64 refinement: the labels, written against the Team abstraction
// (khp_core.cuh) so that they are checked on a machine without a GPU too.
#pragma once

#include "khp_core.cuh"

namespace khp {

// The clusters are the connected components of the graph joining eigenvalues closer than kClusterTol
// max|mu|.  Inside a cluster a first-order step converges
// slowly or not at all (its correction E_ij / (mu_j - mu_i) is not small), so every cluster of
// 2..kClusterMax members takes the exact eigen-decomposition of its block of diag(mu) + E instead.
// A component larger than kClusterMax (a chain of close eigenvalues) is split again at a third of
// the distance, up to kClusterLevels times; what is still too large is treated member by member.
constexpr double kClusterTol = 1e-3;
constexpr int kClusterMax = 12;
constexpr int kClusterLevels = 4;

// *p = min(*p, v) among the threads of a team.
KHP_HD void label_min(int* p, int v) {
#ifdef __CUDA_ARCH__
  atomicMin(p, v);
#else
  if (v < *p) *p = v;
#endif
}

// Labels of the n eigenvalues m, big = max|m|: lb[i] becomes the smallest index of i's component, so
// lb[lb[i]] == lb[i], and sz[i] the component's size.  act: n ints of scratch; changed: one int shared by the
// team.  kRounded: mf holds the eigenvalues rounded to FP32, and distances are taken in FP32 where that
// decides as FP64 would.
template <bool kRounded, class Team>
KHP_HD void cluster_labels(const Team& t, int n, const cplx<double>* m, const cplx<float>* mf, double big, int* lb,
                           int* sz, int* act, int* changed) {
  double tol = kClusterTol * big;
  for (int level = 0; level < kClusterLevels; ++level, tol *= (1.0 / 3.0)) {
    if (t.tid() == 0) *changed = 0;
    t.sync();
    for (int i = t.tid(); i < n; i += t.size()) {
      act[i] = level == 0 || sz[i] > kClusterMax;
      if (act[i]) {
        lb[i] = i;
        *changed = 1;
      }
    }
    t.sync();
    if (!*changed) break;
    t.sync();
    const double tol2 = tol * tol;
    const float margin = (float)(1e-6 * big / tol) + 1e-6f;  // (of d2: twice that of d, rounded up)
    const float lo2 = (1.f - margin) * (float)tol2, hi2 = (1.f + margin) * (float)tol2;
    const bool scaled = lo2 > 1e-30f && hi2 < 1e30f;  // FP32 squares in range
    auto close64 = [&](int i, int j) -> bool {
      const double dr = m[j].re - m[i].re, di = m[j].im - m[i].im;
      return dr * dr + di * di < tol2;
    };
    // Connected components among the columns being split.  A round gives every column the smallest
    // label among its neighbours' and passes it on to the column its old label names, so that a whole chain's
    // worth of columns follows at once; without that a label moves one neighbour a round.  After
    // round r every column within r neighbours of its component's smallest index holds that index: n
    // rounds settle any component (few are needed).
    for (int it = 0; it < n; ++it) {
      if (t.tid() == 0) *changed = 0;
      t.sync();
      for (int i = t.tid(); i < n; i += t.size()) {
        if (!act[i]) continue;
        const int old = lb[i];
        int best = old;
        if (kRounded && scaled) {  // eight columns' loads at a time (a label read a little early is only older)
          const cplx<float> mi = mf[i];
          for (int j0 = 0; j0 < n; j0 += 8) {
            cplx<float> q[8];
            int a[8], l[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const int j = j0 + u < n ? j0 + u : n - 1;
              q[u] = mf[j];
              a[u] = act[j];
              l[u] = lb[j];
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const float dr = q[u].re - mi.re, di = q[u].im - mi.im, d2 = dr * dr + di * di;
              if (!a[u] || l[u] >= best || d2 > hi2) continue;
              if (d2 < lo2 || close64(i, j0 + u < n ? j0 + u : n - 1)) best = l[u];
            }
          }
        } else {
          for (int j = 0; j < n; ++j)
            if (act[j] && lb[j] < best && close64(i, j)) best = lb[j];
        }
        const int next = lb[best];
        if (next < best) best = next;
        if (best < old) {
          // (a label passed to i in between may be lost here: another round follows)
          lb[i] = best;
          if (old != i) label_min(lb + old, best);
          *changed = 1;
        }
      }
      t.sync();
      if (!*changed) break;
      t.sync();
    }
    // component sizes of the columns just labelled (a label is the smallest index of its
    // component, so it never equals the label of a column outside it)
    for (int i = t.tid(); i < n; i += t.size()) {
      if (!act[i]) continue;
      int c = 0;
      for (int j = 0; j < n; ++j) c += lb[j] == lb[i];
      sz[i] = c;
    }
    t.sync();
  }
}

}  // namespace khp
