// cg_state.cuh -- the device-side state of a conjugate-gradient solve, shared
// by the launch-per-step loop (cg.cu) and the one-launch loop
// (cg_resident.cu).
#pragma once

#include <algorithm>

#include "drb_internal.cuh"

namespace drb {

enum : int {
  kRunning = 0,
  kConverged = 1,
  kBreakdown = 2,
  kMaxIters = 3,
  kNotStarted = 4, // one-launch loop: its CTAs did not all get an SM; nothing has changed
};

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
// it, possibly nothing, in the sixteenths of the matrix that a cache policy tells
// apart (rounded up by the hardware, 0.4% of g = 1530 cost 5%).  64 iterations, us,
// nothing kept of a matrix that does not fit / this rule: f64 g = 1140
// 2074 / 1971, 1250 2086 / 1997, 1448 3014 / 2991, 1530 2964 / 2963; f32 1400
// 2303 / 2104, 1448 2377 / 2202, 1600 2741 / 2610, 1800 3026 / 3005.  A fixed amount
// fits some sizes only: 40 MB 1893 at g = 1140, but 3522 at 1530 and 5399 (4419) at 1800.
inline float resident_keep(int64_t matrix_bytes, int64_t vector_bytes) {
  if (matrix_bytes <= kResKeepBytes) return 1.0f;
  const int64_t left = std::max<int64_t>(kResKeepBytes - vector_bytes, 0);
  return (float)(16 * left / matrix_bytes) / 16.0f;
}

bool cg_resident_wanted(const Csr &A);
// CTAs of such a launch (all of them want an SM at once).
template <class T> drb_status cg_resident_grid(const Csr &A, int *ctas);
size_t cg_resident_sync_bytes();
// One launch of the loop (at most 1024 iterations; `first`: from x, else from
// the state, r and p that the previous launch left).  *launched = false when
// the grid cannot be resident at once.  sync: cg_resident_sync_bytes() of
// device memory.  A device-side timeout is left in the handle's error word;
// kNotStarted in the state: CTAs that started waited CgWait::start_ns for others
// that other kernels kept from an SM, and the launch ended without an effect.
template <class T>
drb_status cg_resident_launch(Csr &A, const T *b, T *x, T *r, T *p, T *q, CgState *st,
                              void *sync, double rtol, int64_t max_iters, bool first,
                              bool *launched, cudaStream_t s);

} // namespace drb
