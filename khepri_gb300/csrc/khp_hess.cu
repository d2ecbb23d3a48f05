// Hessenberg reduction H = Q^H A Q of batched FP32 complex matrices with each matrix in the shared
// memory of a thread-block cluster, and Q from its reflectors.
//
// Reflector k: P = I - tau v v^H, v = 0 up to row k, 1 in row k + 1, chosen so that P^H annihilates
// column k below row k + 1 (the convention of team_gehrd, khp_dense.cuh).
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "khepri_gb300.h"
#include "khp_core.cuh"
#include "khp_launch.h"

namespace khp {
namespace {

namespace cg = cooperative_groups;
using cf = cplx<float>;

constexpr int kHessThreads = 256;
constexpr int kHessWarps = kHessThreads / 32;
constexpr int kHessMaxSmem = 220 * 1024;

// rows of the matrix per CTA, then vectors of n: x (the column), v, z (this CTA's part of v^H A), g,
// and one entry per row
constexpr size_t hess_smem(int n, int C) {
  const size_t rows = (n + C - 1) / C;
  return sizeof(cf) * (rows * n + 4 * (size_t)n + rows);
}

// CTA r of a cluster of C holds rows r, r + C, ..  A column: its entries go to every CTA (distributed
// shared memory), each forms the reflector for itself; y = A v for its rows (a warp per row) and its
// part of v^H A (a thread per column); the parts are summed from all CTAs; then the rank-2 update
//   A - v (conj(tau) v^H A - |tau|^2 (v^H A v) v^H) - (tau A v) v^H
// of its rows.  Two cluster barriers per column.  Bound by those and by three passes over the rows in
// shared memory; global memory sees the matrix once in and once out.  H and Q of one matrix, against one
// CTA per matrix in global memory: n = 50 0.58 -> 0.25 ms, n = 98 1.37 -> 0.65, n = 242 10.9 -> 1.4,
// n = 578 159 -> 6.5; 152 matrices of n = 242 11.5 -> 5.9; 912 of them 33.4 -> 34.2, as fast.
__global__ void __launch_bounds__(kHessThreads, 3) k_gehrd_cluster(int n, int C, cf* A, int64_t lda, int64_t bsA,
                                                                    cf* V, int64_t ldv, int64_t bsV) {
  extern __shared__ __align__(16) unsigned char dyn_h[];
  __shared__ float red[2][kHessWarps];
  const cg::cluster_group cl = cg::this_cluster();
  const int rank = C > 1 ? (int)cl.block_rank() : 0;
  const int64_t b = blockIdx.x / C;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cap = (n + C - 1) / C, nr = (n - rank + C - 1) / C;  // rows held at most, here
  cf* As = reinterpret_cast<cf*>(dyn_h);
  cf* x = As + (size_t)cap * n;
  cf* v = x + n;
  cf* z = v + n;
  cf* g = z + n;
  cf* y = g + n;
  cf* Ab = A + b * bsA;
  cf* Vb = V + b * bsV;
  auto cluster_sync = [&]() {
    if (C > 1) cl.sync();
    else __syncthreads();
  };
  for (int m = warp; m < nr; m += kHessWarps)
    for (int j = lane; j < n; j += 32) As[(size_t)m * n + j] = Ab[(int64_t)(rank + C * m) * lda + j];
  cluster_sync();  // (every CTA of the cluster runs before its shared memory is written)
  for (int k = 0; k + 2 < n; ++k) {
    // column k, rows k + 1 .., to every CTA
    for (int e = tid; e < nr * C; e += kHessThreads) {
      const int m = e / C, d = e - m * C, i = rank + C * m;
      if (i > k) {
        cf* dst = C > 1 ? cl.map_shared_rank(x, d) : x;
        dst[i] = As[(size_t)m * n + k];
      }
    }
    cluster_sync();
    // every warp of every CTA forms the same reflector from the same values
    float s = 0.f;
    for (int i = k + 2 + lane; i < n; i += 32) s += norm2(x[i]);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const cf alpha = x[k + 1];
    const bool skip = s == 0.f && alpha.im == 0.f;  // already reduced (tau = 0)
    const float beta = -copysignf(sqrtf(norm2(alpha) + s), alpha.re);
    const cf tau = skip ? mk(0.f) : mk((beta - alpha.re) / beta, -alpha.im / beta);
    const cf scal = skip ? mk(0.f) : cdiv(mk(1.f), alpha - mk(beta));
    for (int i = tid; i < n; i += kHessThreads) {
      const cf vi = skip || i <= k ? mk(0.f) : i == k + 1 ? mk(1.f) : x[i] * scal;
      v[i] = vi;
      if (rank == k % C) Vb[(int64_t)k * ldv + i] = vi;
    }
    if (tid == 0 && rank == k % C) Vb[(int64_t)(n - 2) * ldv + k] = tau;
    __syncthreads();
    if (skip) {  // the same in the whole cluster
      cluster_sync();  // every CTA has read x
      continue;
    }
    // y = A v of this CTA's rows, four of a warp's rows at a time (one load of v for all)
    for (int m = warp; m < nr; m += 4 * kHessWarps) {
      const cf* row[4];
      cf acc[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        row[q] = As + (size_t)min(m + q * kHessWarps, nr - 1) * n;
        acc[q] = mk(0.f);
      }
#pragma unroll 2
      for (int j = ((k + 1) & ~31) + lane; j < n; j += 32) {  // (v is 0 up to k)
        const cf vj = v[j];
#pragma unroll
        for (int q = 0; q < 4; ++q) fma_acc(acc[q], row[q][j], vj);
      }
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          acc[q].re += __shfl_xor_sync(0xffffffffu, acc[q].re, o);
          acc[q].im += __shfl_xor_sync(0xffffffffu, acc[q].im, o);
        }
      if (lane == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (m + q * kHessWarps < nr) y[m + q * kHessWarps] = tau * acc[q];
      }
    }
    // this CTA's part of v^H A
    const int m0 = k + 1 > rank ? (k + 1 - rank + C - 1) / C : 0;  // first row > k
    for (int j = k + 1 + tid; j < n; j += kHessThreads) {
      cf acc[4] = {mk(0.f), mk(0.f), mk(0.f), mk(0.f)};
      int m = m0;
      for (; m + 3 < nr; m += 4)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] += conj_mul(v[rank + C * (m + q)], As[(size_t)(m + q) * n + j]);
      for (; m < nr; ++m) acc[0] += conj_mul(v[rank + C * m], As[(size_t)m * n + j]);
      z[j] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    }
    cluster_sync();
    // v^H A from all parts, and v^H A v
    cf dot = mk(0.f);
    for (int j = k + 1 + tid; j < n; j += kHessThreads) {
      cf zj = mk(0.f);
      if (C > 1) {
#pragma unroll 4
        for (int d = 0; d < C; ++d) zj += cl.map_shared_rank(z, d)[j];
      } else {
        zj = z[j];
      }
      fma_acc(dot, zj, v[j]);
      g[j] = conj(tau) * zj;
    }
    for (int o = 16; o > 0; o >>= 1) {
      dot.re += __shfl_xor_sync(0xffffffffu, dot.re, o);
      dot.im += __shfl_xor_sync(0xffffffffu, dot.im, o);
    }
    if (lane == 0) {
      red[0][warp] = dot.re;
      red[1][warp] = dot.im;
    }
    __syncthreads();
    dot = mk(0.f);
#pragma unroll
    for (int q = 0; q < kHessWarps; ++q) dot += mk(red[0][q], red[1][q]);
    const cf tt = norm2(tau) * dot;
    // A[i][j] -= v_i (g_j - tt conj(v_j)) + y_i conj(v_j)
    for (int m = warp; m < nr; m += 4 * kHessWarps) {
      cf* row[4];
      cf vi[4], yi[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int mq = m + q * kHessWarps, i = rank + C * mq;
        const bool has = mq < nr;
        row[q] = As + (size_t)min(mq, nr - 1) * n;
        vi[q] = has ? v[i] : mk(0.f);
        yi[q] = has ? y[mq] - vi[q] * tt : mk(0.f);
      }
      const int nq = (nr - m + kHessWarps - 1) / kHessWarps;  // rows of this group
#pragma unroll 2
      for (int j = ((k + 1) & ~31) + lane; j < n; j += 32) {
        if (j <= k) continue;
        const cf gj = g[j], vj = v[j];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (q < nq) {
            cf a = row[q][j];
            fms_acc(a, vi[q], gj);
            a -= mul_conj(yi[q], vj);
            row[q][j] = a;
          }
        }
      }
      if (lane < 4 && lane < nq) {
        const int mq = m + lane * kHessWarps, i = rank + C * mq;
        if (i > k) As[(size_t)mq * n + k] = i == k + 1 ? mk(beta) : mk(0.f);
      }
    }
    __syncthreads();
  }
  for (int m = warp; m < nr; m += kHessWarps)
    for (int j = lane; j < n; j += 32) Ab[(int64_t)(rank + C * m) * lda + j] = As[(size_t)m * n + j];
  cluster_sync();  // no CTA leaves while another may still read its shared memory
}

// Z = Q = P_0 P_1 ..: every row of Q by itself, z <- z - tau_k (z v_k) v_k^H, RW rows per warp in
// registers (lane l holds columns l, l + 32, ..; reflector k leaves the columns up to k alone).  The
// reflectors come through shared memory, kQStage at a time for the CTA's 8 warps, the next ones loading
// meanwhile (6.6 ms for 912 matrices of n = 242, 7.0 with every warp reading them from L2 for
// itself).  Bound by the reductions over the lanes beside n^3 complex FMAs, spread over all SMs.
constexpr int kQStage = 4;
constexpr int kQWarps = 8;
template <int EPL, int RW>
__global__ void __launch_bounds__(32 * kQWarps) k_gehrd_q(int n, const cf* __restrict__ V, int64_t ldv, int64_t bsV,
                                                           cf* Z, int64_t boff) {
  __shared__ cf vs[2][kQStage][32 * EPL];
  __shared__ cf taus[2][kQStage];
  const int64_t b = boff + blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31;
  const int r0 = (blockIdx.x * kQWarps + (tid >> 5)) * RW;
  const cf* Vb = V + b * bsV;
  cf q[RW][EPL];
#pragma unroll
  for (int r = 0; r < RW; ++r)
#pragma unroll
    for (int e = 0; e < EPL; ++e) q[r][e] = mk(lane + 32 * e == r0 + r ? 1.f : 0.f);
  const int K = n - 2;  // reflectors
  auto stage = [&](int k0, int buf) {
    for (int e = tid; e < kQStage * 32 * EPL; e += 32 * kQWarps) {
      const int k = k0 + e / (32 * EPL), j = e % (32 * EPL);
      cf* d = &vs[buf][0][0] + e;
      if (k < K && j < n) {
        const unsigned sa = (unsigned)__cvta_generic_to_shared(d);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(Vb + (int64_t)k * ldv + j) : "memory");
      } else {
        *d = mk(0.f);
      }
    }
    if (tid < kQStage) taus[buf][tid] = k0 + tid < K ? Vb[(int64_t)(n - 2) * ldv + k0 + tid] : mk(0.f);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  stage(0, 0);
  for (int k0 = 0, buf = 0; k0 < K; k0 += kQStage, buf ^= 1) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();  // this stage is in; every warp is done with the other buffer
    if (k0 + kQStage < K) stage(k0 + kQStage, buf ^ 1);
#pragma unroll 1
    for (int kk = 0; kk < kQStage; ++kk) {
      const int k = k0 + kk;
      const cf* v = vs[buf][kk] + lane;
      cf d[RW];
#pragma unroll
      for (int r = 0; r < RW; ++r) d[r] = mk(0.f);
#pragma unroll
      for (int e = 0; e < EPL; ++e)
        if (32 * e + 31 > k) {
          const cf ve = v[32 * e];
#pragma unroll
          for (int r = 0; r < RW; ++r) fma_acc(d[r], q[r][e], ve);
        }
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          d[r].re += __shfl_xor_sync(0xffffffffu, d[r].re, o);
          d[r].im += __shfl_xor_sync(0xffffffffu, d[r].im, o);
        }
#pragma unroll
      for (int r = 0; r < RW; ++r) d[r] = taus[buf][kk] * d[r];
#pragma unroll
      for (int e = 0; e < EPL; ++e)
        if (32 * e + 31 > k) {
          const cf ve = v[32 * e];
#pragma unroll
          for (int r = 0; r < RW; ++r) q[r][e] -= mul_conj(d[r], ve);
        }
    }
  }
  cf* Zb = Z + b * (int64_t)n * n;
#pragma unroll
  for (int r = 0; r < RW; ++r)
    if (r0 + r < n) {
#pragma unroll
      for (int e = 0; e < EPL; ++e)
        if (lane + 32 * e < n) Zb[(int64_t)(r0 + r) * n + lane + 32 * e] = q[r][e];
    }
}

// Cluster size for n: the smallest of 1, 2, 4, 8, 16 whose CTAs hold their rows in about a third of an
// SM's shared memory (three CTAs share an SM's barriers' waits); 8 and 16 up to what a whole SM holds.
// 0: too large.
int hess_cluster(int n) {
  for (int C = 1; C <= 8; C *= 2)
    if (hess_smem(n, C) <= 74 * 1024) return C;
  for (int C = 8; C <= 16; C *= 2)
    if (hess_smem(n, C) <= (size_t)kHessMaxSmem) return C;
  return 0;
}

template <int EPL, int RW>
int form_q(int64_t batch, int n, const cf* V, int64_t ldv, int64_t bsV, cf* Z, cudaStream_t s) {
  const unsigned gx = (unsigned)((n + kQWarps * RW - 1) / (kQWarps * RW));
  for (int64_t off = 0; off < batch; off += 65535) {
    const unsigned nb = (unsigned)std::min<int64_t>(batch - off, 65535);
    k_gehrd_q<EPL, RW><<<dim3(gx, nb), 32 * kQWarps, 0, s>>>(n, V, ldv, bsV, Z, off);
    count_launches(1);
  }
  return cuda_status();
}

}  // namespace

bool gehrd_cluster_fits(int64_t batch, int n) {
  const int C = n >= 3 ? hess_cluster(n) : 0;
  // a CTA that fills its SM runs alone there: hundreds of such matrices are faster one per CTA, three to an
  // SM (k_gehrd; n = 338, 304 matrices: 46 ms against 52; n = 578, 64: 207 against 61)
  if (C == 8 && hess_smem(n, C) > 74 * 1024 && batch > 256) return false;
  if (C < 16) return C > 0;
  // a cluster of 16 is beyond the portable size: ask whether the device can hold one (once per device; callers
  // of several threads may all ask, and get the same answer)
  constexpr int kDevices = 64;
  static std::atomic<int> can16[kDevices];  // 0: not asked, 1: no, 2: yes
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return false;
  int can = can16[dev].load(std::memory_order_relaxed);
  if (can == 0) {
    int ok = 0;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {16, 1, 1};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(kHessThreads);
    cfg.dynamicSmemBytes = kHessMaxSmem;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(k_gehrd_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(k_gehrd_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, kHessMaxSmem) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&ok, k_gehrd_cluster, &cfg) != cudaSuccess) {
      cudaGetLastError();
      ok = 0;
    }
    can = ok > 0 ? 2 : 1;
    can16[dev].store(can, std::memory_order_relaxed);
  }
  return can == 2;
}

int launch_gehrd_cluster(int64_t batch, int n, cplx<float>* A, int64_t lda, int64_t bsA, cplx<float>* V, int64_t ldv,
                         int64_t bsV, cplx<float>* Z, cudaStream_t s) {
  if (batch <= 0) return KHP_OK;
  const int C = hess_cluster(n);
  if (C <= 0) return KHP_ERR_TOO_LARGE;
  const size_t smem = hess_smem(n, C);
  if (cudaFuncSetAttribute(k_gehrd_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, kHessMaxSmem) != cudaSuccess)
    return KHP_ERR_CUDA;
  if (C > 8 &&
      cudaFuncSetAttribute(k_gehrd_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return KHP_ERR_CUDA;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim = {(unsigned)C, 1, 1};
  cfg.gridDim = dim3((unsigned)(batch * C));
  cfg.blockDim = dim3(kHessThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, k_gehrd_cluster, n, C, A, lda, bsA, V, ldv, bsV) != cudaSuccess) return KHP_ERR_CUDA;
  count_launches(1);
  if (n <= 64) return form_q<2, 4>(batch, n, V, ldv, bsV, Z, s);
  if (n <= 128) return form_q<4, 4>(batch, n, V, ldv, bsV, Z, s);
  if (n <= 192) return form_q<6, 4>(batch, n, V, ldv, bsV, Z, s);
  if (n <= 256) return form_q<8, 4>(batch, n, V, ldv, bsV, Z, s);
  if (n <= 384) return form_q<12, 2>(batch, n, V, ldv, bsV, Z, s);
  if (n <= 512) return form_q<16, 2>(batch, n, V, ldv, bsV, Z, s);
  return form_q<22, 1>(batch, n, V, ldv, bsV, Z, s);
}

}  // namespace khp
