// cg_resident.cu -- the whole conjugate-gradient loop in one cooperative
// launch, for matrices on their sliced-ELL copy.
//
// What bounds the launch-per-step loop (cg.cu) below HBM-size vectors: three
// kernels an iteration, each with a ramp, a tail and a grid-wide reduction, and
// x, r, q written and read back between them.  Here every CTA (one per SM) owns
// a contiguous range of 32-row slices for the whole solve.  Its parts of r, q, x
// and p stay in shared memory as far as they fit (in this order: the order of
// the traffic each saves), so an iteration moves the matrix, the gathered p
// and one write of p:
//
//   q = A p, p.q        -> exchange of the CTAs' sums
//   x += alpha p, r -= alpha q, r.r -> exchange
//   p = r + beta p      -> grid barrier (p is gathered by other CTAs next)
//
// Measured (64 iterations on a g x g Laplacian, us, launch per step -> here):
// f64 g = 48 787 -> 478, 512 1455 -> 812, 1024 2386 -> 1339, 1448 3672 -> 2991,
// 1800 5462 -> 4367; f32 300 1088 -> 680, 1024 2134 -> 1307, 1448 2979 -> 2151.
// What is left at small sizes is the chain of three grid-wide steps (about 5 us
// of 11 an iteration on all SMs), at large ones the matrix's bytes.
//
// Exchange: CTA b publishes its sum as two 64-bit words of 32 payload bits and
// the exchange's number each, so a reader knows from the word itself that it
// is the new one: no fence and no second round trip.  Up to kResDirect CTAs read
// all sums themselves; of more, CTA 0 does and publishes the total the same way,
// in eight copies (148 CTAs polling 148 words each got in their own way:
// measured 3.9 us a sum, 1.9 through CTA 0, 2.3 by a counter and a second
// read; 8 CTAs: 0.9 direct, 1.6 through CTA 0).  Sums are added in CTA order:
// the same bits everywhere, repeatable.  The barrier is a counter with one
// polling thread per CTA (1.3 us; a flag per CTA read by all: 5.1).
//
// The CTAs wait for one another, so all have to be resident: a cooperative launch,
// which was seen to start only when all its CTAs fit beside the kernels of other
// streams.  Should some start without the others all the same (other processes
// under MPS), until the first exchange ends, which changes nothing that counts,
// a wait of more than start_ns (100 ms) ends the launch, and the host goes on
// with a kernel per step.  All CTAs agree
// on it through one word: each counts itself in as it starts, and giving up is a
// compare-and-swap that succeeds only while the count is short; a CTA that starts
// after it leaves at once.  From then on all CTAs run, and a wait that takes ten
// seconds of %globaltimer all the same is an error (DRB_ERR_TIMEOUT in the
// handle's error word).
#include <algorithm>

#include "drb_internal.cuh"
#include "cg_state.cuh"
#include "tma.cuh"

namespace drb {
namespace {

// Threads per CTA.  f64 needs 80 registers; f32 fits 64 and gains from more
// warps once each has several slices a phase (64 iterations at g = 1024 1419 ->
// 1307 us, 1448 2655 -> 2353; g = 300 726 -> 763).
constexpr int kResNT = 768, kResNTMany = 1024;
constexpr int kResManySlices = 64; // slices per CTA from which f32 takes 1024
constexpr uint64_t kResWaitNs = 10 * tma::kWaitNs;
constexpr int kResMinSlices = 16;  // slices per CTA at least, for small systems
constexpr int kResMaxCtas = 256;   // exchange slots
constexpr int kResDirect = 32;     // CTAs that read each other's sums directly
constexpr int kResCopies = 8;      // copies of a published total, 128 bytes apart
constexpr int kResLaunchIters = 1024; // iterations of one launch

template <class T> struct ResArgs {
  const T *vals;
  const int *cols;
  const int64_t *off;
  int64_t m, ns;
  const T *b;
  T *x, *r, *p, *q; // global vectors; r and q, x only where not resident
  CgState *st;
  ulonglong2 *slots; // [2][kResMaxCtas] exchange words, [2][kResCopies][8] totals
  unsigned *count;   // barrier arrivals
  int *err;
  double rtol;
  int64_t max_iters;
  int cap;   // slices a CTA may own (shared-memory rows = 32 * cap)
  int nres;  // vectors held in shared memory: r, q, x, p in this order
  int first; // this launch starts the solve
  float keep; // share of the matrix that L2 is asked to keep between iterations
  unsigned *start;   // CTAs that started; kGaveUp
  uint64_t start_ns; // limit of the wait for them
  int stall_cta;     // failure-detection hook: this CTA stays away (-1: none)
};
constexpr unsigned kGaveUp = 0x80000000u;

__device__ __forceinline__ double warp_down(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float ld_mat(const float *p, uint64_t pol) {
  float r;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(r) : "l"(p), "l"(pol));
  return r;
}
__device__ __forceinline__ double ld_mat(const double *p, uint64_t pol) {
  double r;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(r) : "l"(p), "l"(pol));
  return r;
}
__device__ __forceinline__ int ld_mat(const int *p, uint64_t pol) {
  int r;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(r) : "l"(p), "l"(pol));
  return r;
}

// The grid's CTAs as one group (all resident: cooperative launch).
template <int NT> struct Grid {
  static constexpr int W = NT / 32;
  ulonglong2 *slots;
  unsigned *count;
  int *err;
  double *s_red;  // [W]
  double *s_sum;  // [kResMaxCtas / 32]
  int *s_stop;
  unsigned *start;
  uint64_t start_ns;
  CgState *st;
  unsigned epoch = 0, arrived = 0; // exchanges, barrier arrivals so far

  // Thread 0 counts the CTA in as it starts (the answer, in `ticket`, is not
  // waited for until the first exchange) ...
  unsigned ticket = 0;
  __device__ void enter() { ticket = atomicAdd(start, 1u); }
  // ... and before it takes part in one finds out: false, the others have given up.
  __device__ bool entered() {
    const bool in = !(ticket & kGaveUp);
    __threadfence(); // counted before its sum can be seen
    return in;
  }
  // After start_ns without all CTAs: true when the launch is given up.
  __device__ bool give_up() {
    unsigned v = atomicAdd(start, 0u);
    while (!(v & kGaveUp) && v < gridDim.x) {
      const unsigned was = atomicCAS(start, v, v | kGaveUp);
      if (was == v) {
        st->done = kNotStarted;
        v |= kGaveUp;
      } else {
        v = was;
      }
    }
    return v & kGaveUp;
  }
  // One step of a wait: true when it has to be given up.
  __device__ bool expired(uint64_t &t0, int spins) {
    if ((spins & 63) != 63) // (reading the timer takes as long as a poll)
      return false;
    if (spins == 63) {
      t0 = tma::globaltimer();
    } else {
      const uint64_t waited = tma::globaltimer() - t0;
      if (epoch == 1 && waited > start_ns && give_up()) {
        *s_stop = 1;
        return true;
      }
      if (waited > kResWaitNs)
        atomicExch(err, DRB_ERR_TIMEOUT);
    }
    if (!*(volatile int *)err)
      return false;
    *s_stop = 1;
    return true;
  }
  __device__ static void publish(ulonglong2 *d, double v, unsigned epoch) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v);
    const unsigned long long e = (unsigned long long)epoch << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(d),
                 "l"((u & 0xffffffffull) | e), "l"((u >> 32) | e)
                 : "memory");
  }
  __device__ double collect(const ulonglong2 *d) {
    unsigned long long w0, w1;
    uint64_t t0 = 0;
    for (int i = 0;; i++) {
      asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];"
                   : "=l"(w0), "=l"(w1)
                   : "l"(d)
                   : "memory");
      if ((unsigned)(w0 >> 32) == epoch && (unsigned)(w1 >> 32) == epoch)
        break;
      if (expired(t0, i))
        break;
    }
    return __longlong_as_double((long long)((w0 & 0xffffffffull) | (w1 << 32)));
  }

  // The sum of v over all threads of the grid, in every thread; false: a wait
  // ran out.
  __device__ bool sum(double v, double &total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int G = gridDim.x;
    epoch++;
    v = warp_down(v);
    if (lane == 0)
      s_red[warp] = v;
    __syncthreads();
    ulonglong2 *slot = slots + (epoch & 1) * kResMaxCtas;
    ulonglong2 *copies = slots + 2 * kResMaxCtas + (epoch & 1) * kResCopies * 8;
    if (warp == 0) {
      const double t = warp_down(lane < W ? s_red[lane] : 0.0);
      if (lane == 0) {
        if (G == 1)
          s_sum[0] = t;
        else if (epoch > 1 || entered())
          publish(slot + blockIdx.x, t, epoch);
        else
          *s_stop = 1;
      }
    }
    const bool reads = G > 1 && (G <= kResDirect || blockIdx.x == 0);
    int np = 1; // words of s_sum
    if (reads) {
      np = (G + 31) / 32;
      if (warp < np) {
        const double t = warp_down((int)threadIdx.x < G ? collect(slot + threadIdx.x) : 0.0);
        if (lane == 0)
          s_sum[warp] = t;
      }
    } else if (G > 1 && threadIdx.x == 0) {
      s_sum[0] = collect(copies + (blockIdx.x % kResCopies) * 8);
    }
    __syncthreads();
    const bool complete = *(volatile int *)s_stop == 0; // (else there is no total)
    double t = 0.0;
    for (int i = 0; i < np; i++)
      t += s_sum[i];
    total = t;
    if (G > kResDirect && blockIdx.x == 0 && threadIdx.x < kResCopies && complete)
      publish(copies + threadIdx.x * 8, t, epoch);
    return complete;
  }

  // Global writes of every thread before are seen by every thread after.
  __device__ bool barrier() {
    arrived += gridDim.x;
    __syncthreads();
    if (gridDim.x == 1)
      return true;
    if (threadIdx.x == 0) {
      __threadfence();
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
      uint64_t t0 = 0;
      for (int i = 0;; i++) {
        unsigned c;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(count) : "memory");
        if ((int)(c - arrived) >= 0)
          break;
        if (expired(t0, i))
          break;
      }
      __threadfence();
    }
    __syncthreads();
    return *(volatile int *)s_stop == 0;
  }
};

template <class T, int NT>
__global__ void __launch_bounds__(NT, 1) cg_resident(const ResArgs<T> a) {
  constexpr int W = NT / 32;
  extern __shared__ __align__(16) unsigned char res_mem[];
  __shared__ double s_red[W], s_sum[(kResMaxCtas + 31) / 32];
  __shared__ int s_stop;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t s0 = a.ns * blockIdx.x / gridDim.x, s1 = a.ns * (blockIdx.x + 1) / gridDim.x;
  const int nsl = (int)(s1 - s0);
  const int64_t row0 = 32 * s0;
  const int rows = (int)(min(a.m, 32 * s1) - row0); // rows of this CTA
  T *sm = reinterpret_cast<T *>(res_mem);
  const int64_t vs = 32 * (int64_t)a.cap;
  int *soff = reinterpret_cast<int *>(sm + a.nres * vs); // [nsl + 1] slice starts from s0's
  // this CTA's part of each vector, in shared or global memory
  T *const vr = a.nres > 0 ? sm : a.r + row0;
  T *const vq = a.nres > 1 ? sm + vs : a.q + row0;
  T *const vx = a.nres > 2 ? sm + 2 * vs : a.x + row0;
  T *const pg = a.p + row0;
  T *const vp = a.nres > 3 ? sm + 3 * vs : pg;
  const int64_t obase = a.off[s0];
  Grid<NT> G{a.slots, a.count, a.err, s_red, s_sum, &s_stop, a.start, a.start_ns, a.st};
  if (tid == 0) {
    s_stop = (int)blockIdx.x == a.stall_cta;
    if (!s_stop)
      G.enter();
    else if (gridDim.x == 1)
      a.st->done = kNotStarted;
  }
  for (int i = tid; i <= nsl; i += NT)
    soff[i] = (int)(a.off[s0 + i] - obase);
  const uint64_t pol = a.keep > 0.0f ? ptx::policy_keep(a.keep) : ptx::policy_evict_first();
  __syncthreads();
  if (s_stop)
    return;

  // The matrix runs ahead of its use: a slice's first K entries per row load
  // while the previous slice's gathers are in flight, those of the warp's first
  // slice while the CTA waits for the others' part of the vector.
  constexpr int K = 6;
  struct Part {
    T e[K];
    int c[K];
  };
  auto fetch = [&](Part &s, int i, int k0) {
    const int o = soff[i], w = ((soff[i + 1] - o) >> 5) - k0;
    const T *va = a.vals + obase + o + 32 * k0 + lane;
    const int *ca = a.cols + obase + o + 32 * k0 + lane;
#pragma unroll
    for (int k = 0; k < K; k++) {
      s.e[k] = T(0);
      s.c[k] = -1;
      if (k < w) {
        s.e[k] = ld_mat(va + 32 * k, pol);
        s.c[k] = ld_mat(ca + 32 * k, pol);
      }
    }
  };
  Part ahead;
  auto fetch_first = [&]() {
    if (warp < nsl)
      fetch(ahead, warp, 0);
  };
  // f(local row, (A v)_row) for this CTA's rows, after fetch_first(); plain loads
  // of v: other CTAs wrote it before the last barrier
  auto spmv = [&](const T *v, auto f) {
    auto add = [&](const Part &s, T &acc) {
      T g[K];
#pragma unroll
      for (int k = 0; k < K; k++)
        g[k] = s.c[k] >= 0 ? v[s.c[k]] : T(0);
#pragma unroll
      for (int k = 0; k < K; k++)
        if (s.c[k] >= 0)
          acc += s.e[k] * g[k];
    };
    for (int i = warp; i < nsl; i += W) {
      Part cur = ahead;
      if (i + W < nsl)
        fetch(ahead, i + W, 0);
      T acc = 0;
      add(cur, acc);
      const int w = (soff[i + 1] - soff[i]) >> 5;
      for (int k0 = K; k0 < w; k0 += K) { // rows of more than K entries
        fetch(cur, i, k0);
        add(cur, acc);
      }
      const int row = 32 * i + lane;
      if (row < rows)
        f(row, acc);
    }
  };
  // f(local row) over this CTA's rows, U at a time: load(row, u) first
  constexpr int U = sizeof(T) == 4 ? 4 : 2; // (64 registers per thread)
  auto each = [&](auto load, auto f) {
    for (int i = tid; i < rows; i += U * NT) {
#pragma unroll
      for (int u = 0; u < U; u++)
        if (i + u * NT < rows)
          load(i + u * NT, u);
#pragma unroll
      for (int u = 0; u < U; u++)
        if (i + u * NT < rows)
          f(i + u * NT, u);
    }
  };

  double rr, tol2;
  int64_t it;
  int done;
  if (a.first) {
    double s_rr = 0.0, s_bb = 0.0, bb;
    fetch_first();
    spmv(a.x, [&](int i, T q) {
      const T bi = a.b[row0 + i];
      const T ri = bi - q;
      vr[i] = ri;
      pg[i] = ri;
      if (a.nres > 3)
        vp[i] = ri;
      s_rr += (double)ri * (double)ri;
      s_bb += (double)bi * (double)bi;
    });
    if (a.nres > 2)
      for (int i = tid; i < rows; i += NT)
        vx[i] = a.x[row0 + i];
    if (!G.sum(s_rr, rr) || !G.sum(s_bb, bb))
      return;
    tol2 = a.rtol * a.rtol * bb;
    it = 0;
    done = rr <= tol2 ? kConverged : (a.max_iters <= 0 ? kMaxIters : kRunning);
    if (blockIdx.x == 0 && tid == 0) {
      a.st->bb = bb;
      a.st->tol2 = tol2;
      a.st->pq = a.st->beta = 0.0;
      a.st->max_iters = a.max_iters;
    }
    fetch_first();
    if (done == kRunning && !G.barrier())
      return;
  } else {
    fetch_first();
    rr = a.st->rr;
    tol2 = a.st->tol2;
    it = a.st->iters;
    done = kRunning;
    for (int i = tid; i < rows; i += NT) {
      if (a.nres > 0)
        vr[i] = a.r[row0 + i];
      if (a.nres > 2)
        vx[i] = a.x[row0 + i];
      if (a.nres > 3)
        vp[i] = pg[i];
    }
    __syncthreads();
    // every CTA has read the state before CTA 0 rewrites it below
    double none;
    if (!G.sum(0.0, none))
      return;
  }

  const int64_t last = it + kResLaunchIters;
  while (done == kRunning && it < last) {
    double acc = 0.0, pq, rr1;
    spmv(a.p, [&](int i, T q) {
      vq[i] = q;
      acc += (double)q * (double)vp[i];
    });
    if (!G.sum(acc, pq))
      return;
    const double alpha = rr / pq;
    if (!(pq > 0.0) || !isfinite(alpha)) {
      done = kBreakdown; // x and r stay as they were
      break;
    }
    acc = 0.0;
    {
      T pv[U], xv[U], rv[U];
      each(
          [&](int i, int u) {
            pv[u] = vp[i];
            xv[u] = vx[i];
            rv[u] = vr[i];
          },
          [&](int i, int u) {
            vx[i] = (T)((double)xv[u] + alpha * (double)pv[u]);
            const T ri = (T)((double)rv[u] - alpha * (double)vq[i]);
            vr[i] = ri;
            acc += (double)ri * (double)ri;
          });
    }
    if (!G.sum(acc, rr1))
      return;
    it++;
    const double beta = rr1 / rr;
    rr = rr1;
    done = rr1 <= tol2 ? kConverged : (it >= a.max_iters ? kMaxIters : kRunning);
    if (done == kRunning) {
      T pv[U];
      each([&](int i, int u) { pv[u] = vp[i]; },
           [&](int i, int u) {
             const T pi = (T)((double)vr[i] + beta * (double)pv[u]);
             pg[i] = pi;
             if (a.nres > 3)
               vp[i] = pi;
           });
      fetch_first();
      if (!G.barrier())
        return;
    }
  }

  for (int i = tid; i < rows; i += NT) {
    if (a.nres > 2)
      a.x[row0 + i] = vx[i];
    if (a.nres > 0 && done == kRunning)
      a.r[row0 + i] = vr[i];
  }
  if (blockIdx.x == 0 && tid == 0) {
    a.st->rr = rr;
    a.st->iters = it;
    a.st->done = done;
  }
}

constexpr size_t kSyncBytes =
    (2 * kResMaxCtas + 2 * kResCopies * 8) * sizeof(ulonglong2) + 2 * sizeof(unsigned);

template <class T> struct ResShape {
  const void *kernel = nullptr;
  int grid = 0, threads = 0, cap = 0, nres = 0;
  size_t smem = 0;
};

template <class T, int NT> drb_status res_shape(const Csr &A, ResShape<T> &S) {
  static std::atomic<unsigned long long> allowed[64];
  static std::atomic<int> dyn_of[64]; // shared memory that a CTA may have
  std::atomic<int> &dyn = dyn_of[A.device < 64 ? A.device : 0];
  int sms = 0;
  DRB_TRY(device_sms(A.device, &sms));
  DRB_TRY(once_per_context(allowed, A.device, [&]() -> drb_status {
    int optin = 0;
    DRB_CUDA_TRY(
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, A.device));
    cudaFuncAttributes fa;
    DRB_CUDA_TRY(cudaFuncGetAttributes(&fa, cg_resident<T, NT>));
    dyn.store(optin - (int)fa.sharedSizeBytes);
    DRB_CUDA_TRY(cudaFuncSetAttribute(
        cg_resident<T, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn.load()));
    return DRB_OK;
  }));
  const int64_t ns = A.sell.nslices;
  S.kernel = reinterpret_cast<const void *>(cg_resident<T, NT>);
  S.threads = NT;
  S.grid = (int)std::max<int64_t>(
      1, std::min<int64_t>(std::min(sms, kResMaxCtas), ns / kResMinSlices));
  S.cap = (int)((ns + S.grid - 1) / S.grid);
  const int64_t vec = 32 * (int64_t)S.cap * (int64_t)sizeof(T);
  const int64_t room = dyn.load() - 4 * ((int64_t)S.cap + 1);
  S.nres = (int)std::max<int64_t>(0, std::min<int64_t>(4, room / vec));
  S.smem = (size_t)(S.nres * vec + 4 * ((int64_t)S.cap + 1));
  return DRB_OK;
}

} // namespace

bool cg_resident_wanted(const Csr &A) {
  // The sliced-ELL copy only (its rows map to threads one to one).  Solves of
  // under 32 slices keep the graph, whose launches per iteration callers may
  // count (drb_launch_count), although one launch is faster there too (40 iterations
  // on a g x g Laplacian, f64, us, graph / one launch: g = 8 520 / 134, 16 509 / 133, 24
  // 517 / 149, 31 577 / 180).
  return A.sell.on && A.sell.nslices >= 32 && A.m <= kResMaxRows;
}

size_t cg_resident_sync_bytes() { return kSyncBytes; }

template <class T> drb_status shape_of(const Csr &A, ResShape<T> &S) {
  DRB_TRY((res_shape<T, kResNT>(A, S)));
  if constexpr (sizeof(T) == 4)
    if (S.cap >= kResManySlices)
      DRB_TRY((res_shape<T, kResNTMany>(A, S)));
  return DRB_OK;
}

template <class T> drb_status cg_resident_grid(const Csr &A, int *ctas) {
  ResShape<T> S;
  DRB_TRY(shape_of<T>(A, S));
  *ctas = S.grid;
  return DRB_OK;
}
template drb_status cg_resident_grid<float>(const Csr &, int *);
template drb_status cg_resident_grid<double>(const Csr &, int *);

template <class T>
drb_status cg_resident_launch(Csr &A, const T *b, T *x, T *r, T *p, T *q, CgState *st,
                              void *sync, double rtol, int64_t max_iters, bool first,
                              bool *launched, cudaStream_t s) {
  *launched = false;
  ResShape<T> S;
  DRB_TRY(shape_of<T>(A, S));
  ResArgs<T> a;
  a.vals = A.sell.vals.as<T>();
  a.cols = A.sell.cols.as<int>();
  a.off = A.sell.off.as<int64_t>();
  a.m = A.m;
  a.ns = A.sell.nslices;
  a.b = b;
  a.x = x;
  a.r = r;
  a.p = p;
  a.q = q;
  a.st = st;
  a.slots = static_cast<ulonglong2 *>(sync);
  a.count = reinterpret_cast<unsigned *>(a.slots + 2 * kResMaxCtas + 2 * kResCopies * 8);
  a.start = a.count + 1;
  a.start_ns = A.cg_start_ns;
  a.stall_cta = A.cg_stall_cta;
  a.err = A.pipe.err.as<int>();
  a.rtol = rtol;
  a.max_iters = max_iters;
  a.cap = S.cap;
  a.nres = S.nres;
  a.first = first ? 1 : 0;
  a.keep = resident_keep(A.sell.padded * (int64_t)(sizeof(T) + 4), 4 * A.m * (int64_t)sizeof(T));
  DRB_CUDA_TRY(cudaMemsetAsync(sync, 0, kSyncBytes, s));
  void *args[] = {&a};
  const cudaError_t e = cudaLaunchCooperativeKernel(
      S.kernel, dim3((unsigned)S.grid), dim3((unsigned)S.threads), args, S.smem, s);
  if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
    cudaGetLastError(); // fewer SMs than the device reports: the graph path
    return DRB_OK;
  }
  DRB_CUDA_TRY(e);
  note_launch();
  *launched = true;
  return DRB_OK;
}

template drb_status cg_resident_launch<float>(Csr &, const float *, float *, float *, float *,
                                              float *, CgState *, void *, double, int64_t, bool,
                                              bool *, cudaStream_t);
template drb_status cg_resident_launch<double>(Csr &, const double *, double *, double *,
                                               double *, double *, CgState *, void *, double,
                                               int64_t, bool, bool *, cudaStream_t);

} // namespace drb
