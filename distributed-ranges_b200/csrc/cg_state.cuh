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
// and the matrix size up to which that launch asks L2 to keep the matrix between
// iterations.
constexpr int64_t kResMaxRows = 3670016;
constexpr int64_t kResKeepBytes = (int64_t)72 << 20;

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
