// Host build of the eigenvalue-cluster labels (khp_clusters.cuh) for the CPU tests, by a team of one.
#include <algorithm>
#include <cmath>
#include <vector>

#include "khp_clusters.cuh"

using namespace khp;

extern "C" void host_cluster_labels(int n, const double* mu, int fp32, int* lb, int* sz) {
  const cplx<double>* m = reinterpret_cast<const cplx<double>*>(mu);
  std::vector<cplx<float>> mf(n);
  std::vector<int> act(n);
  double big = 0.0;
  for (int i = 0; i < n; ++i) {
    big = std::max(big, norm2(m[i]));
    mf[i] = mk((float)m[i].re, (float)m[i].im);
    lb[i] = i;
  }
  int changed = 0;
  if (fp32)
    cluster_labels<true>(TeamSerial(), n, m, mf.data(), std::sqrt(big), lb, sz, act.data(), &changed);
  else
    cluster_labels<false>(TeamSerial(), n, m, mf.data(), std::sqrt(big), lb, sz, act.data(), &changed);
}
