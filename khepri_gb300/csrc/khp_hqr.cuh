// Complex Schur form of an upper Hessenberg matrix by one CTA: the single-shift QR of
// team_hqr_win (khp_dense.cuh: same deflation test, shifts, iteration cap and rotations, in the same
// order for every element), with the chase of a window held in one warp's registers.
#pragma once

#include "khp_dense.cuh"

namespace khp {

constexpr int kHqrCols = 32;            // window columns: one per lane
constexpr int kHqrRot = kHqrCols - 1;   // rotations of a full window
constexpr int kHqrLd = kHqrCols + 1;    // stride of a window row and of a strip (odd: conflict-free)
constexpr int kHqrMaxStrips = 640;      // strips staged at a time
constexpr int kHqrSpareThreads = 512;   // more threads than this leave warp 0's scheduler to it

// Fixed shared memory of cta_hqr (one per CTA); beside it hqr_strips(n) strips of kHqrLd entries.
// Windows, leading strips and rotations are double-buffered by the window's parity.
template <typename T>
struct HqrShared {
  cplx<T> win[2][(kHqrCols + 1) * kHqrLd];  // rows k0 .. k1 + 1, columns k0 .. k1
  cplx<T> lead[2][kHqrRot * kHqrLd];        // the columns k1 + 1 .. k1 + 31, rows k0 .. k1
  HqrRot<T> rot[2][kHqrCols];               // identity beyond the window's rotations
  int best[2][32];
};
KHP_HD constexpr int hqr_strips(int n) { return n < kHqrMaxStrips ? n : kHqrMaxStrips; }
template <typename T>
constexpr size_t hqr_strip_smem(int n) { return sizeof(cplx<T>) * kHqrLd * (size_t)hqr_strips(n); }

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ float rsqrt_ftz(float v) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

// givens() (FP32) without branches: an x whose square underflows is taken as 1e-18 (c ~ 0 and s of
// modulus 1 if y is larger), which against the deflation tolerance is an exact 0.
__device__ __forceinline__ void givens_chain(cplx<float> x, cplx<float> y, float& c, cplx<float>& s, cplx<float>& r) {
  float ax2 = x.re * x.re + x.im * x.im;
  const float ay2 = y.re * y.re + y.im * y.im;
  const bool tiny = ax2 < 1e-36f;
  ax2 = tiny ? 1e-36f : ax2;
  x.re = tiny ? 1e-18f : x.re;
  x.im = tiny ? 0.f : x.im;
  const float t2 = ax2 + ay2;
  const float q = rsqrt_ftz(ax2) * rsqrt_ftz(t2);
  c = ax2 * q;
  s = (x * conj(y)) * q;
  r = x * (t2 * q);
}

template <typename T>
__device__ __forceinline__ cplx<T> shfl(cplx<T> v, int src) {
  return mk(__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src));
}

__device__ __forceinline__ void named_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

// The strip p (kHqrCols entries) rolled through the rotations u0 .. of rot (identity beyond the
// window's): columns take them from the left (sg = 1), rows from the right (sg = -1: conj(s)).
// With kStore false only the running entry is formed.  Returns it after all rotations.
template <bool kStore, bool kFrom, typename T>
__device__ __forceinline__ cplx<T> roll_strip(cplx<T>* p, const HqrRot<T>* rot, T sg, int u0) {
  constexpr int RB = 8;  // loads of a chunk before its stores (which would order the next loads)
  cplx<T> a = p[0];
#pragma unroll
  for (int q0 = 0; q0 < kHqrRot; q0 += RB) {
    cplx<T> v[RB];
#pragma unroll
    for (int u = 0; u < RB; ++u)
      if (q0 + u < kHqrRot) v[u] = p[q0 + u + 1];
#pragma unroll
    for (int u = 0; u < RB; ++u)
      if (q0 + u < kHqrRot) {
        HqrRot<T> g = rot[q0 + u];
        if (kFrom && q0 + u < u0) {  // not this row's yet
          g.c = T(1);
          g.sre = g.sim = T(0);
        }
        const cplx<T> s = mk(g.sre, sg * g.sim), b = v[u];
        v[u] = g.c * a + s * b;
        a = g.c * b - conj_mul(s, a);
      }
    if (kStore) {
#pragma unroll
      for (int u = 0; u < RB; ++u)
        if (q0 + u < kHqrRot) p[q0 + u] = v[u];
    }
  }
  if (kStore) p[kHqrRot] = a;
  return a;
}

// The chase of one window by one warp: rotations into rot, the window's rows (without the right
// rotations from their own on) and r's into win; x, y: column k - 1 of rows k, k + 1 on entry and exit.
// first_r receives the first step's r, corner (in every lane) the entries of rows k1, k1 + 1 in a full
// window's last column, the next window's first.
template <typename T>
__device__ __forceinline__ void hqr_chase(cplx<T>* win, HqrRot<T>* rot, int nrot, cplx<T>& x, cplx<T>& y,
                                          cplx<T>& first_r, cplx<T> (&corner)[2]) {
  const int lane = threadIdx.x & 31;
  cplx<T>* w = win + lane;
  cplx<T> h0 = w[0], h1 = w[kHqrLd], h2 = w[2 * kHqrLd];
  const cplx<T>* sub = win + 2 * kHqrLd + 1;  // H[k+2][k+1] of the next step
  cplx<T> u = *sub;
  T mc = T(1);  // lane t keeps step t's rotation and r (a branch to store them costs 54 cycles a step)
  cplx<T> ms = mk(T(0)), mr = mk(T(0));
#pragma unroll 1
  for (int t = 0; t < nrot; ++t) {
    // for the next step: row k + 3 and H[k+3][k+2] (past the window's last row: not used)
    const cplx<T> next = w[min(t + 3, kHqrCols) * kHqrLd];
    sub += kHqrLd + 1;
    const cplx<T> unext = t + 3 <= kHqrCols ? *sub : mk(T(0));
    T c;
    cplx<T> s, r;
    givens_chain(x, y, c, s, r);
    // left, rows k and k + 1
    const cplx<T> l0 = c * h0 + s * h1, l1 = c * h1 - conj_mul(s, h0);
    // right, rows k + 1 and k + 2 (H[k+2][k] is 0 before)
    const cplx<T> p = shfl(l1, t), q = shfl(l1, t + 1);
    if (lane >= t) w[t * kHqrLd] = l0;
    const bool at = lane == t, at1 = lane == t + 1;
    mc = at ? c : mc;
    ms.re = at ? s.re : ms.re;
    ms.im = at ? s.im : ms.im;
    mr.re = at ? r.re : mr.re;
    mr.im = at ? r.im : mr.im;
    x = c * p + mul_conj(q, s);
    y = mul_conj(u, s);
    const cplx<T> n1 = c * q - s * p, n2 = c * u;
    h0.re = at1 ? n1.re : l1.re;
    h0.im = at1 ? n1.im : l1.im;
    h1.re = at1 ? n2.re : h2.re;
    h1.im = at1 ? n2.im : h2.im;
    h2 = next;
    u = unext;
  }
  HqrRot<T> g;
  g.c = mc;
  g.sre = ms.re;
  g.sim = ms.im;
  g.pad = T(0);
  rot[lane] = g;
  first_r = shfl(mr, 0);
  corner[0] = shfl(h0, kHqrRot);
  corner[1] = shfl(h1, kHqrRot);
  if (lane > 0 && lane < nrot) win[lane * kHqrLd + lane - 1] = mr;
  if (lane >= nrot - 1) {
    w[nrot * kHqrLd] = lane == nrot - 1 ? x : h0;
    w[(nrot + 1) * kHqrLd] = lane == nrot - 1 ? y : h1;
  }
}

// One sweep over the active block [lo, hi] with shift mu, in windows of at most 31 rotations.
//
// The chase is the serial chain of the whole eigensolver.  Warp 0 runs it with a column of the
// window per lane and the rows the bulge touches in registers: the left rotation of step k (rows k,
// k + 1) is lane-local; of the right one (columns k, k + 1) only rows k + 1 and k + 2 feed the chain,
// and only lane k + 1 keeps them (column k's entries are the next step's x and y, which every lane forms
// from lanes k and k + 1 by shuffle, then r and 0).  A step is one rotation, one shuffle and two complex
// products deep.  The right rotations of window row i from its own on are left for later.
//
// The other warps run one window behind: a thread per strip (a column right of the window or a row above
// it, 32 entries, in shared memory) or window row rolls it through the window's rotations, the results go
// back to H, and the next window's strips and untouched rows come in (cp.async, along rows of H).  Warp 0
// rolls its own copy of the next 31 columns' strips to complete the next window's first row.  One
// CTA barrier per window.  Bound by the chase for a few matrices (n = 242: 48K rotations, 0.26 us each
// with everything else) and by what a window moves between H and shared memory for many (two CTAs per
// SM).  Against the chase through shared memory with three warp barriers a step and strips from global
// memory after it (both with the triangular factor's eigenvectors): n = 50 1.35 -> 0.54 ms, n = 98,
// 64 matrices 3.9 -> 1.72, n = 242 31.0 -> 9.0, 912 matrices 89 -> 43, n = 578 222 -> 72.
template <typename T>
__device__ __forceinline__ void cta_hqr_sweep(cplx<T>* H, int64_t ld, int n, int lo, int hi, cplx<T> mu,
                                              HqrShared<T>& sh, cplx<T>* strips, HqrRot<T>* log) {
  static_assert(sizeof(cplx<T>) == 8, "strips are staged in 8-byte copies");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // threads and warps beside warp 0; in the largest CTAs the warps that share its scheduler stay idle
  const int aw = (blockDim.x >> 5) - 1;
  const bool spare = blockDim.x > kHqrSpareThreads, idle = spare && warp > 0 && (warp & 3) == 0;
  const int nw = spare ? aw - aw / 4 : aw, wt = 32 * nw;
  const int vw = spare ? warp - 1 - warp / 4 : warp - 1, vt = 32 * vw + lane;
  const int cap = hqr_strips(n);
  const int nwin = (hi - lo + kHqrRot - 1) / kHqrRot;
  cplx<T> x = mk(T(0)), y = mk(T(0));  // warp 0: column k - 1 of rows k, k + 1
  cplx<T> corner[2] = {x, x};
  // window 0
  {
    const int nrot = min(kHqrRot, hi - lo);
    for (int e = tid; e < (nrot + 2) * kHqrCols; e += blockDim.x) {
      const int i = e >> 5, j = e & 31;
      sh.win[0][i * kHqrLd + j] = (lo + i <= hi && j <= nrot) ? H[(int64_t)(lo + i) * ld + lo + j] : mk(T(0));
    }
  }
  for (int w = 0; w <= nwin; ++w) {
    __syncthreads();
    if (idle) continue;
    if (warp == 0) {
      if (w == nwin) continue;
      cplx<T>* win = sh.win[w & 1];
      const int k0 = lo + w * kHqrRot, nrot = min(kHqrRot, hi - k0);
      if (w == 0) {
        x = win[0] - mu;
        y = win[kHqrLd];
      } else {
        // first row: the leading strips' last entries; first column: from the window before
        cplx<T> a = mk(T(0));
        if (lane < kHqrRot) a = roll_strip<false, false>(sh.lead[(w - 1) & 1] + lane * kHqrLd, sh.rot[(w - 1) & 1], T(1), 0);
        if (lane < kHqrRot) win[lane + 1] = lane < nrot ? a : mk(T(0));
        if (lane == 0) {
          win[0] = corner[0];
          win[kHqrLd] = corner[1];
        }
        __syncwarp();
      }
      cplx<T> r0;
      hqr_chase(win, sh.rot[w & 1], nrot, x, y, r0, corner);
      if (lane == 0 && w > 0) {
        H[(int64_t)k0 * ld + k0 - 1] = r0;
        H[(int64_t)(k0 + 1) * ld + k0 - 1] = mk(T(0));
      }
      continue;
    }
    if (w > 0) {
      // window w - 1: roll, write back
      cplx<T>* win = sh.win[(w - 1) & 1];
      const HqrRot<T>* rot = sh.rot[(w - 1) & 1];
      const int k0 = lo + (w - 1) * kHqrRot, k1 = min(k0 + kHqrRot, hi), nrot = k1 - k0;
      // strip t < right: column k1 + 1 + t, rows k0 .. k1; else row t - right, columns k0 .. k1
      const int right = n - 1 - k1, items = right + k0;
      if (log)
        for (int u = vt; u < nrot; u += wt) log[k0 - lo + u] = rot[u];
      for (int t0 = 0; t0 == 0 || t0 < items; t0 += cap) {
        const int t1 = min(items, t0 + cap), tr = min(t1, right);
        if (t0 > 0) {  // strips beyond those staged ahead
          named_sync(1, wt);
          for (int u = vw; u <= nrot; u += nw)
            for (int t = t0 + lane; t < tr; t += 32)
              strips[(t - t0) * kHqrLd + u] = H[(int64_t)(k0 + u) * ld + k1 + 1 + t];
          if (lane <= nrot)
            for (int t = max(t0, right) + vw; t < t1; t += nw)
              strips[(t - t0) * kHqrLd + lane] = H[(int64_t)(t - right) * ld + k0 + lane];
          named_sync(1, wt);
        }
        for (int t = t0 + vt; t < t1; t += wt)
          roll_strip<true, false>(strips + (t - t0) * kHqrLd, rot, t < right ? T(1) : T(-1), 0);
        if (t0 == 0) {  // window rows, from the far end of the threads
          const int i = wt - 1 - vt;
          if (i < nrot) roll_strip<true, true>(win + i * kHqrLd, rot, T(-1), i);
        }
        named_sync(1, wt);
        for (int u = vw; u <= nrot; u += nw) {
          cplx<T>* hr = H + (int64_t)(k0 + u) * ld + k1 + 1;
          for (int t = t0 + lane; t < tr; t += 32) hr[t] = strips[(t - t0) * kHqrLd + u];
        }
        if (lane <= nrot)
          for (int t = max(t0, right) + vw; t < t1; t += nw)
            H[(int64_t)(t - right) * ld + k0 + lane] = strips[(t - t0) * kHqrLd + lane];
      }
      // (the bulge's column k1 - 1 of rows k1, k1 + 1 belongs to the next window's first step)
      for (int i = vw; i < nrot + 2; i += nw)
        if (k0 + i <= hi && lane <= nrot && !(k1 < hi && i >= nrot && lane == nrot - 1))
          H[(int64_t)(k0 + i) * ld + k0 + lane] = win[i * kHqrLd + lane];
      named_sync(1, wt);
    }
    if (w < nwin) {
      // window w's strips, their first 31 columns again for warp 0, and window w + 1's untouched rows
      const int k0 = lo + w * kHqrRot, k1 = min(k0 + kHqrRot, hi), nrot = k1 - k0;
      const int right = n - 1 - k1, t1 = min(right + k0, cap), tr = min(t1, right);
      const bool more = k1 < hi;
      for (int u = vw; u <= nrot; u += nw) {
        const cplx<T>* hr = H + (int64_t)(k0 + u) * ld + k1 + 1;
        for (int t = lane; t < tr; t += 32) cp_async8(strips + t * kHqrLd + u, hr + t);
        if (more && lane < min(kHqrRot, right)) cp_async8(sh.lead[w & 1] + lane * kHqrLd + u, hr + lane);
      }
      if (lane <= nrot)
        for (int t = right + vw; t < t1; t += nw)
          cp_async8(strips + t * kHqrLd + lane, H + (int64_t)(t - right) * ld + k0 + lane);
      if (more) {
        cplx<T>* nx = sh.win[(w + 1) & 1];
        const int m = min(kHqrRot, hi - k1);
        for (int i = 1 + vw; i < kHqrCols + 1; i += nw) {
          cplx<T>* d = nx + i * kHqrLd + lane;
          if (lane > 0 && lane <= m && k1 + i <= hi) cp_async8(d, H + (int64_t)(k1 + i) * ld + k1 + lane);
          else *d = mk(T(0));
        }
      }
      asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    }
  }
  __syncthreads();
}

// The whole QR, Z through the rotation log as team_hqr_win (log->cap_rot >= n - 1).  Every thread
// follows the same control flow from its own copy of the state.  Returns status bits.
template <typename T>
__device__ __forceinline__ int cta_hqr(cplx<T>* H, int64_t ld, int n, cplx<T>* Z, int64_t ldz, HqrShared<T>& sh, cplx<T>* strips,
                       const HqrLog<T>& log) {
  const TeamCta t;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = (nt + 31) >> 5;
  const T smlnum = Eps<T>::safemin * (T(n) / Eps<T>::ulp);
  const int cap = 30 * n + 60;
  int hi = n - 1, its = 0, total = 0, st = 0, buf = 0;
  int nsw = 0, nrot = 0;  // sweeps and rotations in the log
  // strip entries beyond a short window's rotations take part in products with 0: no stale NaN there
  for (int e = tid; e < hqr_strips(n) * kHqrLd; e += nt) strips[e] = mk(T(0));
  for (int e = tid; e < 2 * kHqrRot * kHqrLd; e += nt) sh.lead[0][e] = mk(T(0));
  __syncthreads();
  while (hi >= 0) {
    // largest k in [1, hi] with a negligible subdiagonal H[k][k-1]
    int l = 0;
    for (int k = 1 + tid; k <= hi; k += nt)
      if (hqr_negligible(H, ld, k, hi, smlnum)) l = k;
    l = __reduce_max_sync(0xffffffffu, l);
    buf ^= 1;
    if (lane == 0) sh.best[buf][warp] = l;
    __syncthreads();
    l = lane < nw ? sh.best[buf][lane] : 0;
    l = __reduce_max_sync(0xffffffffu, l);
    if (l > 0 && tid == 0) H[(int64_t)l * ld + l - 1] = mk(T(0));
    if (l == hi) {
      hi -= 1;
      its = 0;
      continue;
    }
    ++its;
    if (++total > cap) {
      st |= KHP_BIT_NOT_CONVERGED;
      break;
    }
    const cplx<T> mu = hqr_shift(H, ld, l, hi, its);
    __syncthreads();  // every thread has read the shift's entries before the sweep changes them
    if (nrot + (hi - l) > log.cap_rot) {
      // no room for this sweep: the team applies what is logged, and the log starts again
      hqr_log_flush(t, log, nsw, Z, ldz, n);
      nsw = 0;
      nrot = 0;
    }
    if (tid == 0) {
      log.sweeps[2 * nsw] = l;
      log.sweeps[2 * nsw + 1] = hi;
    }
    cta_hqr_sweep(H, ld, n, l, hi, mu, sh, strips, log.rot + nrot);
    ++nsw;
    nrot += hi - l;
  }
  __syncthreads();
  if (tid == 0) {
    log.head[0] = nsw;
    log.head[1] = nrot;
  }
  __syncthreads();
  return st;
}

}  // namespace khp
