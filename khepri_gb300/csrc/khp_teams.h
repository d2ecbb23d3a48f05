// Threads per CTA of the eigensolver's one-CTA-per-matrix kernels (host only).
#pragma once

#include <algorithm>
#include <cstdint>

namespace khp {

constexpr int kTeamThreads = 256;
constexpr int64_t kSms = 152;

// Hessenberg reduction and window QR: the caller's choice (khp_tune; 0: none), else by precision and size.  FP64:
// smaller teams for small matrices, whose barriers and reductions are most of a step (one n = 18 1.64 ms with 256
// threads, 1.55 with 64; n = 50 8.96, 8.76 with 128; n = 98 the fastest with 256).
inline int eig_team(bool fp64, int n, int tuned) {
  if (tuned > 0) return tuned;
  return !fp64 || n > 64 ? kTeamThreads : n > 32 ? 128 : 64;
}

// FP32 QR with a rotation log (cta_hqr: a warp for the chase, the others for the strips): the caller's choice,
// at least a warp for each, else by size and matrices per SM.  While a matrix has an SM to itself more threads
// than strips shorten their way to and from H (one n = 242: 256 threads 11.2 ms, 288 10.5, 352 9.4, 480
// 9.3, 544 with the warps on the chase's scheduler idle 9.0, 480 so 9.2; n = 162: 4.87, 4.83, 4.09, 4.15, 3.94,
// 4.21; n = 50: 557, 561, 542, 547, 555, 558 us).  Up to two matrices per SM two CTAs
// fit with 256 (304 of n = 98: 192 threads 2.67 ms, 256 2.41, 352 3.44).  Beyond, three of 192 where their
// shared memory fits (456 of n = 98: 192 threads 3.22, 256 4.48; of n = 150: 7.17, 8.87), else two of 288
// (456 of n = 162: 192 threads 13.8, 256 12.2, 288 11.0; of n = 242: 32.1, 29.5, 25.3).  Small matrices: 512
// of n = 18 with 128 threads 284 us, 160 270, 192 368.
inline int chase_team(int n, int64_t batch, int tuned) {
  if (tuned > 0) return std::max(64, tuned);
  if (n <= 32) return 160;
  if (batch <= kSms) return n <= 64 ? 352 : 544;
  if (batch <= 2 * kSms) return kTeamThreads;
  return n <= 150 ? 192 : kTeamThreads + 32;
}

}  // namespace khp
