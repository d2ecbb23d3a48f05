// Batched explicit inverse by Gauss-Jordan elimination with partial pivoting.
//
// Two forms, by size:
//   * k_inv_reg: the whole matrix in one CTA's registers (FP32 up to n = 128), one launch;
//   * k_gj_panel + k_gj_update: panels of up to 32 columns eliminated by one CTA per matrix, each
//     followed by one rank-w update of the whole matrix spread over the SMs.
// Both leave the rows (columns) where they are: pivots are recorded, and the interchange of the
// result's rows and columns happens as the inverse is written.
#include <algorithm>
#include <utility>

#include "khepri_gb300.h"
#include "khp_core.cuh"
#include "khp_launch.h"

namespace khp {
namespace {

constexpr int64_t kMaxGridY = 65535;

// Magnitude |re| + |im| of a pivot candidate as an ordered integer: 0 for NaN (never chosen while a
// number is left), 1 for zero, larger for larger magnitudes (FP64: by the 20 leading bits of the
// mantissa; of candidates that agree in them the first is taken).
__device__ __forceinline__ unsigned pivot_key(cplx<float> v) {
  const float x = abs1(v);
  return x == x ? __float_as_uint(x) + 1u : 0u;
}
__device__ __forceinline__ unsigned pivot_key(cplx<double> v) {
  const double x = abs1(v);
  if (!(x == x)) return 0u;
  return x == 0.0 ? 1u : max((unsigned)__double2hiint(x), 1u) + 1u;
}
// Status of a step from its best candidate's key, 0 for a nonzero finite pivot.  (An infinite one would
// eliminate with a reciprocal of 0 and leave a finite "inverse" of a matrix that has none.)
template <typename T>
__device__ __forceinline__ int pivot_status(unsigned best) {
  constexpr unsigned kInf = (sizeof(T) == 4 ? 0x7f800000u : 0x7ff00000u) + 1u;
  if (best - 2u < kInf - 2u) return 0;  // (one comparison on the elimination's chain)
  return best == 1u ? KHP_BIT_SINGULAR : KHP_BIT_NONFINITE;
}

// 1/p for a pivot (nonzero): conj(p)/|p|^2 with p scaled by a power of two to a modulus of 1 to 2^1.5, one
// division.  (khp_core.cuh's cdiv takes three divisions in a row and a branch, which every elimination
// step waits for: in FP64, where a warp's instruction takes 16 cycles of the SM's pipe, 2.5 to 5K cycles of
// a step's 5.3 to 9.6K.)  FP64 refines the FP32 reciprocal by two Newton steps (2^-22, 2^-44, rounding).
__device__ __forceinline__ cplx<float> pivot_recip(cplx<float> p) {
  const unsigned e = __float_as_uint(fmaxf(fabsf(p.re), fabsf(p.im))) >> 23;
  const float sc = __uint_as_float((254u - min(e, 253u)) << 23);
  const float x = p.re * sc, y = p.im * sc;
  const float r = sc / (x * x + y * y);
  return e < 255u ? mk(x * r, -y * r) : mk(0.f);  // (0 for an infinite pivot)
}
__device__ __forceinline__ cplx<double> pivot_recip(cplx<double> p) {
  const int e = max(__double2hiint(fabs(p.re)), __double2hiint(fabs(p.im))) >> 20;
  const double sc = __hiloint2double((2046 - min(e, 2045)) << 20, 0);
  const double x = p.re * sc, y = p.im * sc;
  const double d = x * x + y * y;
  double r = (double)(1.0f / (float)d);
  r = fma(r, fma(-d, r, 1.0), r);
  r = fma(r, fma(-d, r, 1.0), r);
  r *= sc;
  return e < 2047 ? mk(x * r, -y * r) : mk(0.0);
}

// ------------------------------------------------------------------------------------------
// Whole matrix in registers.  Warp w of NW holds rows w, w + NW, ..; lane l columns l, l + 32, ..:
// element (w + NW j, l + 32 i) of the matrix in a[i][j].  Step k takes row k, picks the largest
// |a| among the columns not yet used (one warp, REDUX), and eliminates row k from every other
// column: a[., c] -= a[k][c] / a[k][p] a[., p], in place.  Row k reaches the other warps through
// shared memory (double-buffered, one barrier per step); column p stays inside each warp (a lane's
// registers, by shuffles).  The warp that owns row k + 1 updates that row first and publishes its
// pivot before the rest of its update, so the search and the division run beside the other warps'
// FMAs.  With B the array after n steps and p_k the column of step k: inv[p_r][k] = B[r][p_k].
//
// Bound by FP32 issue (n^3 complex FMAs, 4 n^3 FFMA, of one SM) plus ~0.15 us of dependent steps per
// row.  152 matrices: n = 50 251 -> 48 us, n = 126 702 -> 155 us (blocked LU and substitutions, 25 and 50
// launches, before).
// ------------------------------------------------------------------------------------------
template <int TR, int TC, int NW>
__global__ void __launch_bounds__(32 * NW) k_inv_reg(int n, const cplx<float>* __restrict__ A, int64_t lda,
                                                      int64_t bsA, cplx<float>* Ainv, int64_t ldi, int64_t bsI,
                                                      int* info) {
  using cf = cplx<float>;
  __shared__ cf frow[2][32 * TR];
  __shared__ cf pinv_s[2];
  __shared__ int pcol_s[2];
  __shared__ int pcol[NW * TC];
  __shared__ int kinv[32 * TR];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const cf* Ab = A + blockIdx.x * bsA;
  cf a[TR][TC];
#pragma unroll
  for (int j = 0; j < TC; ++j)
#pragma unroll
    for (int i = 0; i < TR; ++i) {
      const int r = warp + NW * j, c = lane + 32 * i;
      a[i][j] = (r < n && c < n) ? Ab[(int64_t)r * lda + c] : mk(0.f);
    }
  unsigned used = 0;  // bit i: column lane + 32 i has been a pivot
#pragma unroll
  for (int i = 0; i < TR; ++i)
    if (lane + 32 * i >= n) used |= 1u << i;
  int st = 0;
  // row `j` of this warp: pick its pivot and publish it with the row (step buffer `buf`)
  auto publish = [&](const cf (&row)[TR], int k, int buf) __attribute__((always_inline)) {
    unsigned key = 0;
    int col = 0x7fffffff;
    cf pv = mk(0.f);  // the lane's best candidate
#pragma unroll
    for (int i = TR - 1; i >= 0; --i) {  // ties to the lowest column
      const unsigned q = pivot_key(row[i]);
      if (!((used >> i) & 1u)) {
        if (q >= key) { key = q; col = lane + 32 * i; pv = row[i]; }
      }
      frow[buf][lane + 32 * i] = row[i];
    }
    const unsigned best = __reduce_max_sync(0xffffffffu, key);
    const int p = __reduce_min_sync(0xffffffffu, key == best ? col : 0x7fffffff);
    pv.re = __shfl_sync(0xffffffffu, pv.re, p & 31);
    pv.im = __shfl_sync(0xffffffffu, pv.im, p & 31);
    const bool ok = best > 1u;  // 1: every candidate is 0; 0: every candidate is NaN
    if (lane == 0) {
      pinv_s[buf] = ok ? pivot_recip(pv) : mk(0.f);
      pcol_s[buf] = ok ? p : ~p;  // ~p: the column is spent but nothing is eliminated
      pcol[k] = p;
      kinv[p] = k;
      st |= pivot_status<float>(best);
    }
  };
  if (warp == 0) {
    cf row[TR];
#pragma unroll
    for (int i = 0; i < TR; ++i) row[i] = a[i][0];
    publish(row, 0, 0);
  }
#pragma unroll
  for (int jj = 0; jj < TC; ++jj) {
#pragma unroll 1
    for (int w = 0; w < NW; ++w) {
      const int k = jj * NW + w;
      if (k >= n) break;
      const int buf = k & 1;
      __syncthreads();
      const int ps = pcol_s[buf];
      const int p = ps < 0 ? ~ps : ps;
      const cf pinv = pinv_s[buf];
      const int pl = p & 31, pi = p >> 5;
      const bool elim = ps >= 0;
      cf s[TC], f[TR];
#pragma unroll
      for (int i = 0; i < TR; ++i) f[i] = frow[buf][lane + 32 * i];
#pragma unroll
      for (int i = 0; i < TR; ++i)
        if (pi == i) {  // (uniform over the CTA)
#pragma unroll
          for (int j = 0; j < TC; ++j) {
            s[j].re = __shfl_sync(0xffffffffu, a[i][j].re, pl);
            s[j].im = __shfl_sync(0xffffffffu, a[i][j].im, pl);
          }
          if (lane == pl) {
            used |= 1u << i;
            if (elim) {
              f[i] = mk(-1.f);
#pragma unroll
              for (int j = 0; j < TC; ++j) a[i][j] = mk(0.f);
            }
          }
        }
      if (elim) {
#pragma unroll
        for (int j = 0; j < TC; ++j) s[j] = s[j] * pinv;
        if (warp == w) {
          s[jj] = pinv;
#pragma unroll
          for (int i = 0; i < TR; ++i) a[i][jj] = mk(0.f);
        }
      } else {
#pragma unroll
        for (int j = 0; j < TC; ++j) s[j] = mk(0.f);
      }
      // the next row's owner: its row first, published before the rest of its update
      if (k + 1 < n) {
        if (w + 1 < NW) {
          if (warp == w + 1) {
            cf row[TR];
#pragma unroll
            for (int i = 0; i < TR; ++i) {
              row[i] = a[i][jj];
              fms_acc(row[i], f[i], s[jj]);
            }
            publish(row, k + 1, buf ^ 1);
          }
        } else if (warp == 0) {
          constexpr int J = TC - 1;
          const int jn = jj + 1 < TC ? jj + 1 : J;
          cf row[TR];
#pragma unroll
          for (int i = 0; i < TR; ++i) {
            row[i] = a[i][jn];
            fms_acc(row[i], f[i], s[jn]);
          }
          publish(row, k + 1, buf ^ 1);
        }
      }
#pragma unroll
      for (int j = 0; j < TC; ++j)
#pragma unroll
        for (int i = 0; i < TR; ++i) fms_acc(a[i][j], f[i], s[j]);
    }
  }
  __syncthreads();
  cf* Ib = Ainv + blockIdx.x * bsI;
#pragma unroll
  for (int j = 0; j < TC; ++j) {
    const int r = warp + NW * j;
    if (r < n) {
      cf* out = Ib + (int64_t)pcol[r] * ldi;
#pragma unroll
      for (int i = 0; i < TR; ++i)
        if (lane + 32 * i < n) out[kinv[lane + 32 * i]] = a[i][j];
    }
  }
  if (lane == 0 && st) atomicOr(info + blockIdx.x, st);
}

// ------------------------------------------------------------------------------------------
// Panels of rows.  With P the pivot columns of a panel of rows J, D = A[J, P]: the panel becomes
//   G[:, P] = D^-1,  G[:, j] = -D^-1 A[J, j] (other columns),
// and every other row A[i, .] <- (P's columns 0, the others kept) + A[i, P] G.  k_gj_panel makes G in
// place (scalar Gauss-Jordan steps, partial pivoting over the columns not yet used); k_gj_update
// applies it, from one of the two buffers A and inv(A) to the other, so that its tiles read the pivot
// columns' old values themselves (copied aside by the panel's CTA, an entry per sector, they took half of
// the panel's time for 912 matrices and a quarter for one).  (Pivots are searched along rows because
// rows are contiguous, and because the matrices inverted most are eigenvector matrices, whose columns
// have unit norm: the inverse's error there is 0.86 to 0.94 of the row-pivoted LU's at n = 162 to 338,
// with column panels 1.2 to 1.3.)
//
// The panel lives in shared memory row by row (conflict-free for a thread per column) and is
// eliminated in sub-panels of 8 rows held in registers, a column per thread: a step is one barrier
// (every warp's best candidate column goes to shared memory with its key, every thread then picks the
// winner) and 8 complex FMAs per column; the other rows of the panel follow as a rank-8 update.
// Bound by that chain of barriers (n = 242: ~30 us for one matrix, two thirds of it the steps).
// An inverse with its updates, against the blocked LU with substitutions on the identity: one n = 242
// 1349 -> 318 us, 912 7.2 -> 4.16 ms.
// ------------------------------------------------------------------------------------------
constexpr int kGjW = 32;   // panel width
constexpr int kGjSub = 8;  // sub-panel width

template <typename T>
constexpr size_t gj_panel_smem(int n, int w, int threads) {
  // candidate columns and their reciprocals [2][warps][8 + 1], pivot columns of a sub-panel [w][8],
  // panel [w][n], used flags [n], pivot columns of the panel
  return sizeof(cplx<T>) * ((size_t)2 * (threads / 32) * (kGjSub + 1) + (size_t)kGjSub * w + (size_t)w * n) +
         sizeof(int) * ((size_t)n + kGjW);
}

template <typename T, int MAXT>
__global__ void __launch_bounds__(MAXT) k_gj_panel(int n, int kb, int w, cplx<T>* A, int64_t lda, int64_t bsA,
                                                    int* piv, int* info) {
  using ct = cplx<T>;
  extern __shared__ __align__(16) unsigned char dyn_gj[];
  __shared__ unsigned ckey[2][32];
  __shared__ int crow[2][32];
  const int nw = blockDim.x >> 5;
  ct* cand = reinterpret_cast<ct*>(dyn_gj);   // [2][warps][8]
  ct* cinv = cand + 2 * nw * kGjSub;          // [2][warps]
  ct* Us = cinv + 2 * nw;                     // [w][8]
  ct* P = Us + kGjSub * w;                    // P[c n + r]: row kb + c, column r
  int* used = reinterpret_cast<int*>(P + (size_t)w * n);
  int* pcol = used + n;                       // pivot column of every panel row
  const int64_t b = blockIdx.x;
  ct* Ab = A + b * bsA;
  int* pv = piv + b * n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r = tid;  // this thread's column (blockDim.x >= n)
  if (r < n) {
#pragma unroll 8
    for (int c = 0; c < w; ++c) P[c * n + r] = Ab[(int64_t)(kb + c) * lda + r];
    used[r] = 0;
  }
  __syncthreads();
  for (int k = tid; k < kb; k += blockDim.x) used[pv[k]] = 1;
  __syncthreads();
  bool free_col = r < n && !used[r];
  int st = 0;
  for (int c0 = 0; c0 < w; c0 += kGjSub) {
    const int cw = min(kGjSub, w - c0);
    ct a[kGjSub];
#pragma unroll
    for (int c = 0; c < kGjSub; ++c) a[c] = (r < n && c < cw) ? P[(c0 + c) * n + r] : mk(T(0));
    bool mine = false;  // this column is a pivot of the sub-panel
#pragma unroll
    for (int c = 0; c < kGjSub; ++c) {
      if (c >= cw) break;
      const int buf = c & 1;
      // the warp's best candidate (ties to the lower column), its column and its reciprocal; a warp
      // without a free column has key 0 and crow -1
      const unsigned key = free_col ? pivot_key(a[c]) : 0u;
      const unsigned best = __reduce_max_sync(0xffffffffu, key);
      const unsigned who = __ballot_sync(0xffffffffu, free_col && key == best);
      const int src = __ffs(who) - 1;
      if (lane == src) {
        ct* q = cand + (buf * nw + warp) * kGjSub;
#pragma unroll
        for (int z = 0; z < kGjSub; ++z) q[z] = a[z];
        if (best > 1u) cinv[buf * nw + warp] = pivot_recip(a[c]);
      }
      if (lane == 0) {
        ckey[buf][warp] = best;
        crow[buf][warp] = src < 0 ? -1 : warp * 32 + src;
      }
      __syncthreads();
      const int kr = lane < nw ? crow[buf][lane] : -1;
      const unsigned kk = kr >= 0 ? ckey[buf][lane] : 0u;
      const unsigned top = __reduce_max_sync(0xffffffffu, kk);
      const int bw = __ffs(__ballot_sync(0xffffffffu, kr >= 0 && kk == top)) - 1;
      const int br = __shfl_sync(0xffffffffu, kr, bw);
      st |= pivot_status<T>(top);
      if (tid == 0) pcol[c0 + c] = br;
      const bool pivot = r == br;
      if (pivot) { mine = true; free_col = false; }
      if (top > 1u) {
        // a <- a - f (pivot column / pivot), with f = -1 and a = 0 in the pivot column itself
        const ct* q = cand + (buf * nw + bw) * kGjSub;
        const ct pinv = cinv[buf * nw + bw];
        const ct f = pivot ? mk(T(-1)) : a[c];
        if (pivot) {
#pragma unroll
          for (int z = 0; z < kGjSub; ++z) a[z] = mk(T(0));
        }
        a[c] = mk(T(0));
        const ct fp = f * pinv;
#pragma unroll
        for (int z = 0; z < kGjSub; ++z) {
          if (z == c) a[z] = -fp;
          else fms_acc(a[z], fp, q[z]);
        }
      }
    }
    // the other rows of the panel: old values at the sub-panel's pivot columns, then rank-8 update
    __syncthreads();
    for (int e = tid; e < kGjSub * w; e += blockDim.x) {
      const int c = e & (kGjSub - 1), j = e / kGjSub;
      Us[e] = c < cw ? P[j * n + pcol[c0 + c]] : mk(T(0));
    }
    __syncthreads();
    if (r < n) {
#pragma unroll 4
      for (int j = 0; j < w; ++j) {
        if (j >= c0 && j < c0 + cw) continue;
        ct acc = mine ? mk(T(0)) : P[j * n + r];
#pragma unroll
        for (int c = 0; c < kGjSub; ++c) fma_acc(acc, a[c], Us[j * kGjSub + c]);
        P[j * n + r] = acc;
      }
#pragma unroll
      for (int c = 0; c < kGjSub; ++c)
        if (c < cw) P[(c0 + c) * n + r] = a[c];
    }
    __syncthreads();
  }
  if (tid < w) pv[kb + tid] = pcol[tid];
  if (r < n)
    for (int c = 0; c < w; ++c) Ab[(int64_t)(kb + c) * lda + r] = P[c * n + r];
  if (tid == 0 && st) info[b] |= st;
}

// The update by the panel of rows [kb, kb + w), from A to out (panel rows copied); for the last panel
// with the inverse's rows and columns interchanged (inv[p_r][k] = B[r][p_k]).  Tiles of 16 TM x 16 TN,
// TM x TN outputs per thread, the whole rank in one pass through shared memory: 64 x 64 in FP32; 16 x 16 in
// FP64, whose pipe is so slow (2 FMAs per clock and SM) that padding and idle SMs cost more than the extra
// loads.  FP32 products as packed pairs of neighbouring columns (the same FMAs in the same order, half
// the instructions): 152 matrices of n = 242 895 -> 869 us, 912 4.23 -> 4.16 ms an inverse.  Bound by reading and
// writing the matrix once per panel (0.86 GB for those 912, 2.4 TB/s with the gathered pivot entries).
// Slower or no faster: 128 threads with 8 x 4 outputs each (161 against 139 us for 304), a CTA per row of
// tiles with its pivot entries gathered once (4.21 ms).
template <typename T, int TM, int TN>
constexpr size_t gj_update_smem() {
  // (FP32: a pivot column's entry twice, as the packed products take it)
  return sizeof(cplx<T>) * kGjW * (16 * TN + (16 * TM + 1) * (sizeof(T) == 4 ? 2 : 1)) +
         16 * (TM + TN) * sizeof(int);
}

// d = a b + d on two FP32 values each (one instruction for two FMAs, at the FP32 pipe's rate).
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  return v;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}

template <typename T, int TM, int TN>
__global__ void __launch_bounds__(256, 3) k_gj_update(
    int n, int kb, int w, const cplx<T>* __restrict__ A, int64_t lda, int64_t bsA, const int* __restrict__ piv,
    cplx<T>* __restrict__ out, int64_t ldo, int64_t bsO, int last, int64_t boff) {
  using ct = cplx<T>;
  struct alignas(2 * sizeof(ct)) Pair { ct a, b; };
  constexpr int BM = 16 * TM, BN = 16 * TN, LU = BM + 1;
  extern __shared__ __align__(32) unsigned char dyn_gu[];
  constexpr bool kPacked = sizeof(T) == 4;
  ct* Gs = reinterpret_cast<ct*>(dyn_gu);  // [w][BN]; packed: real parts [w][BN], then imaginary parts
  T* Gi = reinterpret_cast<T*>(Gs) + kGjW * BN;
  // [w][LU]: the tile's rows of the pivot columns; packed: {re, re, im, im}
  ct* Us = Gs + kGjW * BN;
  int* col_k = reinterpret_cast<int*>(Us + kGjW * LU * (kPacked ? 2 : 1));  // [BN]: step of the column in this panel (or, last, overall)
  int* row_p = col_k + BN;                              // [BM]: last panel: pivot column of the row's step
  const int64_t b = blockIdx.z + boff;
  const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;  // rows ty + 16 i
  auto col = [&](int j) { return TN == 1 ? tx : 2 * tx + (j & 1) + 32 * (j >> 1); };
  const ct* Ab = A + b * bsA;
  ct* Ob = out + b * bsO;
  const int* pv = piv + b * n;
  {  // a row's pivot columns by neighbouring lanes: they share its lines
    const int lw = w <= 8 ? 3 : 5, c = tid & ((1 << lw) - 1);
    if (c < w) {
      const int p = pv[kb + c];
#pragma unroll 4
      for (int i = tid >> lw; i < BM; i += 256 >> lw) {
        const ct u = row0 + i < n ? Ab[(int64_t)(row0 + i) * lda + p] : mk(T(0));
        if constexpr (kPacked) reinterpret_cast<float4*>(Us)[c * LU + i] = make_float4(u.re, u.re, u.im, u.im);
        else Us[c * LU + i] = u;
      }
    }
  }
  if (tid < BN) col_k[tid] = -1;
  for (int e = tid; e < w * BN; e += 256) {
    const int c = e / BN, i = e % BN;
    const ct g = col0 + i < n ? Ab[(int64_t)(kb + c) * lda + col0 + i] : mk(T(0));
    if constexpr (kPacked) {
      reinterpret_cast<T*>(Gs)[e] = g.re;
      Gi[e] = g.im;
    } else {
      Gs[e] = g;
    }
  }
  ct acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int r = row0 + ty + 16 * i, c = col0 + col(j);
      acc[i][j] = (r < n && c < n) ? Ab[(int64_t)r * lda + c] : mk(T(0));
    }
  if (last && tid < BM && row0 + tid < n) row_p[tid] = pv[row0 + tid];
  __syncthreads();
  for (int k = (last ? 0 : kb) + tid; k < kb + w; k += 256) {
    const int c = pv[k] - col0;
    if (c >= 0 && c < BN) col_k[c] = k;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < TN; ++j)
    if (col_k[col(j)] >= kb) {  // a pivot column of this panel
#pragma unroll
      for (int i = 0; i < TM; ++i) acc[i][j] = mk(T(0));
    }
  if constexpr (kPacked) {
    using u64 = unsigned long long;
    u64 re[TM][TN / 2], im[TM][TN / 2];  // of two neighbouring columns
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) {
        re[i][j] = pack2(acc[i][2 * j].re, acc[i][2 * j + 1].re);
        im[i][j] = pack2(acc[i][2 * j].im, acc[i][2 * j + 1].im);
      }
#pragma unroll 2
    for (int c = 0; c < w; ++c) {
      u64 gr[TN / 2], gi[TN / 2], ngi[TN / 2];
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) {
        gr[j] = *reinterpret_cast<const u64*>(reinterpret_cast<const T*>(Gs) + c * BN + 2 * tx + 32 * j);
        gi[j] = *reinterpret_cast<const u64*>(Gi + c * BN + 2 * tx + 32 * j);
        ngi[j] = gi[j] ^ 0x8000000080000000ull;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const ulonglong2 u = reinterpret_cast<const ulonglong2*>(Us)[c * LU + ty + 16 * i];
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) {
          fma2(re[i][j], u.x, gr[j]);
          fma2(re[i][j], u.y, ngi[j]);
          fma2(im[i][j], u.x, gi[j]);
          fma2(im[i][j], u.y, gr[j]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) {
        const float2 a = unpack2(re[i][j]), b = unpack2(im[i][j]);
        acc[i][2 * j] = mk(a.x, b.x);
        acc[i][2 * j + 1] = mk(a.y, b.y);
      }
  } else {
#pragma unroll 4
    for (int c = 0; c < w; ++c) {
      ct u[TM], g[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) u[i] = Us[c * LU + ty + 16 * i];
      if constexpr (TN == 1) {
        g[0] = Gs[c * BN + tx];
      } else {
#pragma unroll
        for (int j = 0; j < TN; j += 2) {
          const Pair p = *reinterpret_cast<const Pair*>(Gs + c * BN + 2 * tx + 16 * j);
          g[j] = p.a;
          g[j + 1] = p.b;
        }
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) fma_acc(acc[i][j], u[i], g[j]);
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int rl = ty + 16 * i, r = row0 + rl;
    if (r >= n) continue;
    const bool panel = r >= kb && r < kb + w;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int cl = col(j), c = col0 + cl;
      if (c >= n) continue;
      ct v = acc[i][j];
      if (panel) {
        const int e = (r - kb) * BN + cl;
        if constexpr (kPacked) v = mk(reinterpret_cast<const T*>(Gs)[e], Gi[e]);
        else v = Gs[e];
      }
      if (last) Ob[(int64_t)row_p[rl] * ldo + col_k[cl]] = v;
      else Ob[(int64_t)r * ldo + c] = v;
    }
  }
}

template <int TR, int TC, int NW>
void inv_reg(int64_t batch, int n, const cplx<float>* A, int64_t lda, int64_t bsA, cplx<float>* Ainv, int64_t ldi,
             int64_t bsI, int* info, cudaStream_t s) {
  k_inv_reg<TR, TC, NW><<<(unsigned)batch, 32 * NW, 0, s>>>(n, A, lda, bsA, Ainv, ldi, bsI, info);
}

// Largest n of the panel form: a thread per column.
constexpr int kGjMaxN = 1024;
constexpr int kGjPanelSmem = 200 * 1024;

template <typename T>
int inverse_panels(int64_t batch, int n, cplx<T>* A, int64_t lda, int64_t bsA, cplx<T>* Ainv, int64_t ldi, int64_t bsI,
                   int* piv, int* info, cudaStream_t s) {
  const int threads = (n + 31) / 32 * 32;
  // panel width: 32 rows in FP32, fewer while the panel does not fit in shared memory; 8 in FP64, where
  // the panel's own n w^2 FMAs on one SM are its cost (one n = 98
  // inverse: 1.10 ms with 32 rows, 0.45 with 8, 1.41 by the one-CTA LU before; n = 242: 3.7, 1.6 and 10.8)
  int w = sizeof(T) == 4 ? kGjW : kGjSub;
  while (w > kGjSub && gj_panel_smem<T>(n, w, threads) > (size_t)kGjPanelSmem) w -= kGjSub;
  w = std::min(w, n);
  const size_t psmem = gj_panel_smem<T>(n, w, threads);
  constexpr int TT = sizeof(T) == 4 ? 4 : 1;
  constexpr size_t usmem = gj_update_smem<T, TT, TT>();
  auto panel = threads <= 512 ? k_gj_panel<T, 512> : k_gj_panel<T, 1024>;
  auto update = k_gj_update<T, TT, TT>;
  if (cudaFuncSetAttribute(panel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGjPanelSmem) != cudaSuccess ||
      cudaFuncSetAttribute(update, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)usmem) != cudaSuccess)
    return KHP_ERR_CUDA;
  const int tiles = (n + 16 * TT - 1) / (16 * TT);
  // an odd number of panels, so that the last one goes from A to Ainv: with an even one the first w rows
  // are taken as two panels
  const bool odd = (n + w - 1) / w % 2 == 1;
  cplx<T>* src = A;
  cplx<T>* dst = Ainv;
  int64_t lds = lda, bss = bsA, ldd = ldi, bsd = bsI;
  for (int kb = 0; kb < n;) {
    const int cw = !odd && kb == 0 ? w / 2 : !odd && kb < w ? w - kb : std::min(w, n - kb);
    const int last = kb + cw >= n ? 1 : 0;
    panel<<<(unsigned)batch, threads, psmem, s>>>(n, kb, cw, src, lds, bss, piv, info);
    for (int64_t off = 0; off < batch; off += kMaxGridY) {
      const unsigned nb = (unsigned)std::min<int64_t>(batch - off, kMaxGridY);
      update<<<dim3(tiles, tiles, nb), 256, usmem, s>>>(n, kb, cw, src, lds, bss, piv, dst, ldd, bsd, last, off);
      count_launches(1);
    }
    count_launches(1);
    kb += cw;
    std::swap(src, dst);
    std::swap(lds, ldd);
    std::swap(bss, bsd);
  }
  return cuda_status();
}

}  // namespace

template <typename T>
int launch_inverse_blocked(int64_t batch, int n, cplx<T>* A, int64_t lda, int64_t bsA, cplx<T>* Ainv, int64_t ldi,
                           int64_t bsI, int* piv, int* info, cudaStream_t s) {
  if (batch <= 0) return KHP_OK;
  if constexpr (sizeof(T) == 4) {
    // registers while a thread's share of the matrix fits beside its temporaries: 4 x 8 entries at
    // n = 128; the 5 x 10 of n = 160 spill (12 KB a thread).  152 matrices: 155 us at n = 126 here,
    // 350 us at n = 162 by panels
    if (n <= 128) {
#define KHP_REG(TR, TC, NW) inv_reg<TR, TC, NW>(batch, n, A, lda, bsA, Ainv, ldi, bsI, info, s)
      if (n <= 32) KHP_REG(1, 8, 4);
      else if (n <= 56) KHP_REG(2, 7, 8);
      else if (n <= 64) KHP_REG(2, 8, 8);
      else if (n <= 80) KHP_REG(3, 5, 16);
      else if (n <= 96) KHP_REG(3, 6, 16);
      else if (n <= 112) KHP_REG(4, 7, 16);
      else KHP_REG(4, 8, 16);
#undef KHP_REG
      count_launches(1);
      return cuda_status();
    }
  }
  if (n <= kGjMaxN) return inverse_panels<T>(batch, n, A, lda, bsA, Ainv, ldi, bsI, piv, info, s);
  // (beyond 12800 rows not even one panel column fits in shared memory)
  if ((size_t)n * sizeof(cplx<T>) <= 200 * 1024)
    return launch_inverse_lu<T>(batch, n, A, lda, bsA, Ainv, ldi, bsI, piv, info, s);
  return launch_inverse<T>(batch, n, A, lda, bsA, Ainv, ldi, bsI, piv, info, s);
}

template int launch_inverse_blocked<double>(int64_t, int, cplx<double>*, int64_t, int64_t, cplx<double>*, int64_t,
                                            int64_t, int*, int*, cudaStream_t);
template int launch_inverse_blocked<float>(int64_t, int, cplx<float>*, int64_t, int64_t, cplx<float>*, int64_t,
                                           int64_t, int*, int*, cudaStream_t);

}  // namespace khp

extern "C" {

int khp_inverse_gj(int64_t batch, int32_t n, int32_t precision, void* A, int64_t a_stride, void* Ainv,
                   int64_t inv_stride, int32_t* status, void* workspace, size_t ws_bytes, void* stream) {
  using namespace khp;
  if (batch < 0 || n < 1 || (precision != 0 && precision != 1) || !A || !Ainv || !status ||
      a_stride < (int64_t)n * n || inv_stride < (int64_t)n * n)
    return KHP_ERR_INVALID_ARG;
  if (batch == 0) return KHP_OK;
  if (!workspace || ws_bytes < khp_inverse_workspace(batch, n)) return KHP_ERR_WORKSPACE;
  int* piv = static_cast<int*>(workspace);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (precision == 0)
    return launch_inverse_blocked<double>(batch, n, static_cast<cplx<double>*>(A), n, a_stride,
                                          static_cast<cplx<double>*>(Ainv), n, inv_stride, piv, status, s);
  return launch_inverse_blocked<float>(batch, n, static_cast<cplx<float>*>(A), n, a_stride,
                                       static_cast<cplx<float>*>(Ainv), n, inv_stride, piv, status, s);
}

}  // extern "C"
