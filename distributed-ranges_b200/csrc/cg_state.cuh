// cg_state.cuh -- the device-side state of a conjugate-gradient solve, shared
// by the launch-per-step loop (cg.cu) and the one-launch loop
// (cg_resident.cu).
#pragma once

#include "drb_internal.cuh"

namespace drb {

enum : int { kRunning = 0, kConverged = 1, kBreakdown = 2, kMaxIters = 3 };

struct CgState {
  double rr;   // r.r of the current residual
  double pq;   // p.Ap of the current iteration (written by the SpMV)
  double beta; // rr' / rr of the last update
  double bb;   // b.b
  double tol2; // rtol^2 * b.b
  int64_t iters, max_iters;
  int done; // kRunning, kConverged, kBreakdown, kMaxIters
  int pad;
};

// Rows of the largest solve that runs in one launch (beyond it little of the
// vectors fits the SMs, and three kernels on four CTAs per SM stream as fast: 64
// iterations on a g x g Laplacian, launch per step / one launch, f64 g = 1900
// 6013 / 5189 us, f32 1800 3954 / 3677, 2048 4785 / 4779, 2700 7914 / 8748),
// and how much of the matrix it asks L2 to keep between iterations.
constexpr int64_t kResMaxRows = 3670016;
constexpr int64_t kResKeepBytes = (int64_t)72 << 20;

// The whole matrix up to kResKeepBytes; above that what the four vectors leave of
// it, possibly nothing.  64 iterations, f64 g = 1250 / 1448 / 1800 and
// f32 1448 / 1600 / 1800, with a fixed amount kept of a matrix that does not fit:
// none 2256 / 3062 / 4719, 2550 / 2984 / 3435 us; 24 MB 2188 / 2986 / 5221, 2451 /
// 2883 / 3353; 56 MB 2263 / 3163 / 5527, 2383 / 2826 / 3492; 72 MB slower still
// except where all of it fits (f64 1024: 56 MB 1522, 72 MB 1501).  With the rule
// 2188 / 3017 / 4722, 2416 / 2857 / 3358.
inline float resident_keep(int64_t matrix_bytes, int64_t vector_bytes) {
  if (matrix_bytes <= kResKeepBytes) return 1.0f;
  const int64_t left = kResKeepBytes - vector_bytes;
  return left > 0 ? (float)left / (float)matrix_bytes : 0.0f;
}

bool cg_resident_wanted(const Csr &A);
size_t cg_resident_sync_bytes();
// One launch of the loop (at most 1024 iterations; `first`: from x, else from
// the state, r and p that the previous launch left).  *launched = false when
// the grid cannot be resident at once.  sync: cg_resident_sync_bytes() of
// device memory.  A device-side timeout is left in the handle's error word.
template <class T>
drb_status cg_resident_launch(Csr &A, const T *b, T *x, T *r, T *p, T *q, CgState *st,
                              void *sync, double rtol, int64_t max_iters, bool first,
                              bool *launched, cudaStream_t s);

} // namespace drb
