// dense_reduce.cu -- dense row-major gemv (one right-hand side; several:
// dense_panel.cu) and the deterministic dot/norm reduction.
//
// Dense gemv has no dr::mp counterpart (dr::mp::gemv only takes
// distributed_sparse_matrix, include/dr/mp/algorithms/matrix/gemv.hpp:16-71);
// it is shaped after the sparse call over a row-major matrix, the layout of
// dr::sp::distributed_dense_matrix tiles
// (include/dr/sp/containers/distributed_dense_matrix.hpp:205-219).
// The dot product replaces mp::reduce over zip(a, b) | transform(mul)
// (include/dr/mp/algorithms/reduce.hpp:58-107,
// benchmarks/gbench/common/dot_product.cpp:33-52) with one launch and a
// fixed summation order.
#include <algorithm>
#include <mutex>

#include "drb_internal.cuh"

namespace drb {
namespace {

constexpr int kDenseNT = 256;

template <class V> __device__ __forceinline__ V warp_sum_d(V v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// One right-hand side: HBM-bound, A streamed once.  The work is cut into
// steps of one row x 32 * U pieces (16 bytes, or single elements where A's rows
// or x do not start on 16 bytes), 2 KB or 4 KB of a row, so a warp reads long
// contiguous runs.
// CTAs take equal consecutive shares of the steps (LOCAL: of the rows), their
// warps equal shares of those.  A row that falls to one warp goes straight to y,
// the parts of a row cut between warps meet in shared memory in step order, and
// the parts of a row cut between CTAs go to frag (slot 0: the part does not start
// its row; slot 1: it does), which dense_row_join adds, a warp per row.  (Whole
// 32 KB row slabs per warp, the earlier unit, left 8192 rows on 7104 warps: some
// did two while the others had finished one.)
// A lane sums a step's products (16 to 32) by themselves and adds the steps'
// sums: one chain over its share of a row grew the error with the row (N(0, 1)
// rows of 16384 columns, 2-norm over the result's: f32 2.6e-7, f64 4.9e-16, now
// 1.3e-7 and 2.6e-16).
// U pieces per lane and step: 8, but 4 for rows under 8 KB, whose last step would be
// mostly empty (us, U = 4 / 8: f32 20000 x 500 10.2 / 11.7, 10000 x 2000 16.3 / 16.1, 4096^2
// 13.2 / 12.6, 8192^2 43.3 / 42.5, 32768^2 622 / 606; f64 16384 x 128 6.3 / 7.9, 10000 x 500
// 10.5 / 11.8, 16384 x 1000 23.7 / 24.0, 5000 x 4000 28.4 / 27.5), and 16 single elements.
constexpr int64_t kLongRowBytes = 8192;
constexpr int64_t kUneven = 48 * 1024;
// CTAs per SM: as many as leave the registers for a step's loads to go out at once.
// Rows of 16-byte pieces, us, 4 / 3 / 2: f32 8192^2 45.0 / 43.1 / 41.9 (0.99 of the
// measured HBM rate; the slab kernel 53.5), 32768^2 656 / 617 / 604 (slabs 626), f64
// 8192^2 91.3 / 84.4 / 81.9, 20000^2 509 / 476 / 460.  Single elements: f32 4001^2 15.8
// / 16.3 with 4 / 3 CTAs, f64 5003 x 3001 23.9 / 22.4.
template <class V, bool VEC> constexpr int kRowCtas = VEC ? 2 : sizeof(V) == 4 ? 4 : 3;

struct RowShare { // the steps [s0, s1) of share w of W over `steps`, from `base`
  int64_t s0, s1;
  __device__ RowShare(int64_t base, int64_t steps, int64_t w, int64_t W)
      : s0(base + steps * w / W), s1(base + steps * (w + 1) / W) {}
};

template <class V, bool VEC, bool LOCAL, int U>
__global__ void __launch_bounds__(kDenseNT, kRowCtas<V, VEC>)
    dense_row_kernel(int64_t m, int64_t n, const V *__restrict__ A, int64_t lda,
                     const V *__restrict__ x, V *__restrict__ y, int64_t spr, V *frag) {
  constexpr int PER = VEC ? 16 / (int)sizeof(V) : 1;
  constexpr int NW = kDenseNT / 32;
  __shared__ V s_frag[2 * NW];
  ptx::grid_dependents_start();
  ptx::grid_dependency_wait(A, x);
  const uint64_t pol_s = ptx::policy_evict_first();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const RowShare cta = LOCAL ? RowShare(0, m, blockIdx.x, gridDim.x)
                             : RowShare(0, m * spr, blockIdx.x, gridDim.x);
  const int64_t c0 = LOCAL ? cta.s0 * spr : cta.s0, c1 = LOCAL ? cta.s1 * spr : cta.s1;
  const RowShare me(c0, c1 - c0, warp, NW);
  const int64_t ng = n / PER; // whole pieces of a row
  int64_t row = me.s0 / spr, q = me.s0 - row * spr;
  bool inside = q != 0; // the current part does not start its row
  V acc = 0;
  for (int64_t s = me.s0; s < me.s1; s++) {
    const V *Ar = A + row * lda;
    const int64_t g0 = q * (32 * U) + lane;
    V part = 0; // this step's products
    if constexpr (VEC) {
      union G16 {
        uint4 u;
        V t[PER];
      };
      G16 a[U];
      if ((q + 1) * (32 * U) <= ng) { // no predicates: all loads go out at once
#pragma unroll
        for (int i = 0; i < U; i++)
          a[i].u = ptx::ld_stream16(Ar + (g0 + 32 * i) * PER, pol_s);
#pragma unroll
        for (int i = 0; i < U; i++) {
          G16 xv;
          xv.u = reinterpret_cast<const uint4 *>(x)[g0 + 32 * i];
#pragma unroll
          for (int e = 0; e < PER; e++)
            part += a[i].t[e] * xv.t[e];
        }
      } else {
#pragma unroll
        for (int i = 0; i < U; i++) {
          a[i].u = make_uint4(0, 0, 0, 0);
          if (g0 + 32 * i < ng)
            a[i].u = ptx::ld_stream16(Ar + (g0 + 32 * i) * PER, pol_s);
        }
#pragma unroll
        for (int i = 0; i < U; i++)
          if (g0 + 32 * i < ng) {
            G16 xv;
            xv.u = reinterpret_cast<const uint4 *>(x)[g0 + 32 * i];
#pragma unroll
            for (int e = 0; e < PER; e++)
              part += a[i].t[e] * xv.t[e];
          }
      }
      if (q + 1 == spr && ng * PER + lane < n) // the elements after the last piece
        part += Ar[ng * PER + lane] * x[ng * PER + lane];
    } else {
      V a[U];
#pragma unroll
      for (int i = 0; i < U; i++)
        a[i] = g0 + 32 * i < ng ? __ldcs(Ar + g0 + 32 * i) : V(0);
#pragma unroll
      for (int i = 0; i < U; i++)
        if (g0 + 32 * i < ng)
          part += a[i] * x[g0 + 32 * i];
    }
    acc += part;
    q++;
    if (q == spr || s + 1 == me.s1) {
      const V t = warp_sum_d(acc);
      if (lane == 0) {
        if (q == spr && !inside)
          y[row] = t;
        else
          s_frag[2 * warp + (inside ? 0 : 1)] = t;
      }
      acc = 0;
      row++;
      q = 0;
      inside = false;
    }
  }
  __syncthreads();
  if (threadIdx.x >= NW)
    return;
  // what the CTA's warps have of the row up to step `end`, from warp v on
  auto rest = [&](int v, int64_t end, V sum) {
    for (; v < NW; v++) {
      const RowShare o(c0, c1 - c0, v, NW);
      if (o.s0 >= end)
        break;
      if (o.s1 > o.s0)
        sum += s_frag[2 * v];
    }
    return sum;
  };
  const RowShare mine(c0, c1 - c0, threadIdx.x, NW);
  const int64_t cut = mine.s1 / spr; // the row that this warp started and did not finish
  if (mine.s1 % spr != 0 && cut * spr >= mine.s0) {
    const V sum = rest(threadIdx.x + 1, (cut + 1) * spr, s_frag[2 * threadIdx.x + 1]);
    if (LOCAL || (cut + 1) * spr <= c1)
      y[cut] = sum;
    else
      frag[2 * blockIdx.x + 1] = sum;
  }
  if (!LOCAL && threadIdx.x == 0 && c0 % spr != 0) // the row that an earlier CTA started
    frag[2 * blockIdx.x] = rest(0, (c0 / spr + 1) * spr, V(0));
}

// The rows cut between the G CTAs: a warp per CTA that started one and did not
// finish it adds its part and the later CTAs'.
template <class V>
__global__ void __launch_bounds__(kDenseNT)
    dense_row_join(int64_t steps, int64_t spr, int64_t G, const V *frag, V *y) {
  ptx::grid_dependents_start();
  ptx::grid_dependency_wait(frag);
  const int lane = threadIdx.x & 31;
  const int64_t b = ((int64_t)blockIdx.x * kDenseNT + threadIdx.x) >> 5;
  if (b >= G)
    return;
  const RowShare me(0, steps, b, G);
  const int64_t row = me.s1 / spr;
  if (me.s1 % spr == 0 || row * spr < me.s0)
    return;
  const int64_t last = ((row + 1) * spr * G - 1) / steps; // the CTA of the row's last step
  V s = 0;
  for (int64_t v = b + 1 + lane; v <= last; v += 32)
    s += frag[2 * v];
  s = warp_sum_d(s);
  if (lane == 0)
    y[row] = frag[2 * b + 1] + s;
}

template <class V, bool VEC, int U>
drb_status dense_row_call(int64_t m, int64_t n, const V *A, int64_t lda, const V *x, V *y,
                          cudaStream_t s) {
  constexpr int PER = VEC ? 16 / (int)sizeof(V) : 1;
  constexpr int64_t STEP = 32 * U; // pieces per step
  static int grid_cache[64] = {0};
  int dev = 0;
  DRB_CUDA_TRY(cudaGetDevice(&dev));
  int &full = grid_cache[dev < 64 ? dev : 0];
  if (full == 0) {
    int occ = 0, sms = 0;
    DRB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &occ, dense_row_kernel<V, VEC, true, U>, kDenseNT, 0));
    DRB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    full = std::max(1, occ) * sms;
  }
  const int64_t spr = std::max<int64_t>(1, (n / PER + STEP - 1) / STEP);
  const int64_t steps = m * spr;
  constexpr int NW = kDenseNT / 32;
  const int64_t gl = std::min<int64_t>(full, m), gs = std::min<int64_t>(full, (steps + NW - 1) / NW);
  // Whole rows per CTA, unless the CTA with the most rows then reads more than
  // kUneven bytes above an equal share: that takes longer than the second launch
  // and its scratch do.  (us, whole rows / shared steps, f32: 1 row of 0.25 MB
  // 7.4 / 4.5, of 4 MB 184 / 6.1; 4 rows of 64 KB 3.6 / 4.7; 32 rows, 2 MB 5.9 / 5.8,
  // 4 MB 9.2 / 6.0; 100 rows, 8 MB 7.7 / 6.3; 148 rows, 8 MB 6.2 / 6.4; 592 rows,
  // 16 MB 6.0 / 7.8.  The slab kernel that came before: 1 row of 4 MB 22.)
  const int64_t row_bytes = n * (int64_t)sizeof(V);
  const bool local = (m + gl - 1) / gl * row_bytes - m * row_bytes / full <= kUneven;
  cudaError_t e;
  if (local) {
    e = launch_overlapped(dense_row_kernel<V, VEC, true, U>, dim3((unsigned)gl), dim3(kDenseNT), 0,
                          s, m, n, A, lda, x, y, spr, (V *)nullptr);
    note_launch();
  } else {
    V *frag = nullptr;
    DRB_TRY(scratch_alloc(reinterpret_cast<void **>(&frag), sizeof(V) * 2 * (size_t)gs, s));
    e = launch_overlapped(dense_row_kernel<V, VEC, false, U>, dim3((unsigned)gs), dim3(kDenseNT),
                          0, s, m, n, A, lda, x, y, spr, frag);
    note_launch();
    if (e == cudaSuccess) {
      e = launch_overlapped(dense_row_join<V>, dim3((unsigned)((gs + NW - 1) / NW)),
                            dim3(kDenseNT), 0, s, steps, spr, gs, (const V *)frag, y);
      note_launch();
    }
    scratch_free(frag, s);
  }
  if (e != cudaSuccess) {
    set_error("dense gemv launch: %s", cudaGetErrorString(e));
    return DRB_ERR_CUDA;
  }
  return DRB_OK;
}

template <class V>
drb_status dense_row(int64_t m, int64_t n, const V *A, int64_t lda, const V *x, V *y,
                     cudaStream_t s) {
  const bool vec = reinterpret_cast<uintptr_t>(A) % 16 == 0 &&
                   reinterpret_cast<uintptr_t>(x) % 16 == 0 && lda * sizeof(V) % 16 == 0;
  if (!vec)
    return dense_row_call<V, false, 16>(m, n, A, lda, x, y, s);
  if (n * (int64_t)sizeof(V) < kLongRowBytes)
    return dense_row_call<V, true, 4>(m, n, A, lda, x, y, s);
  return dense_row_call<V, true, 8>(m, n, A, lda, x, y, s);
}

// ---- dot -------------------------------------------------------------------------
constexpr int kDotNT = 256;
constexpr int kDotGrid = 592; // at most; a function of n only: the order must not vary
// 16-byte loads in flight per vector per thread.  (f64, 3 / 4: two vectors of 40 MB
// 12.5 / 15.3 us, of 240 MB 70.0 / 70.5; f32 16.9 / 13.6 and 74.9 / 71.0.)
template <class V> constexpr int kDotUnroll = sizeof(V) == 8 ? 3 : 4;

// The CTA's sum of v, in thread 0.
__device__ __forceinline__ double dot_cta_sum(double v) {
  __shared__ double s_red[kDotNT / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum_d(v);
  __syncthreads(); // (an earlier sum's values have been read)
  if (lane == 0)
    s_red[warp] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kDotNT / 32; w++)
      s += s_red[w];
  return s;
}

// The partials of a dot in a fixed order, in thread 0.
__device__ __forceinline__ double dot_partials_sum(const double *partials, int count) {
  double s = 0.0;
  for (int i = threadIdx.x; i < count; i += kDotNT)
    s += __ldcg(&partials[i]);
  return dot_cta_sum(s);
}

// HBM-bound (two streams, 2 n sizeof(T) bytes).  Every trip issues all its loads
// first, the last, partial one too: left to single loads it was up to three
// more memory latencies, a sixth of the time at 40 MB a vector.  With TICKET the
// last CTA adds the partials; without it dot_finish does, whose launch overlaps
// this kernel (a ticket needs a memset before every call: a launch and its gap,
// about 2 us).  One CTA writes the result itself.
template <class V, bool TICKET>
__global__ void __launch_bounds__(kDotNT)
    dot_kernel(int64_t n, const V *__restrict__ a, const V *__restrict__ b,
               double *partials, int *ticket, double *out) {
  constexpr int PER = 16 / sizeof(V), U = kDotUnroll<V>;
  if (!TICKET) {
    ptx::grid_dependents_start();
    ptx::grid_dependency_wait(a, b);
  }
  const uint64_t pol_s = ptx::policy_evict_first();
  double acc = 0.0;
  const int64_t tid = (int64_t)blockIdx.x * kDotNT + threadIdx.x;
  const int64_t nth = (int64_t)gridDim.x * kDotNT;
  const bool vec = (reinterpret_cast<uintptr_t>(a) % 16 == 0) &&
                   (reinterpret_cast<uintptr_t>(b) % 16 == 0);
  int64_t done = 0;
  if (vec) {
    union W {
      uint4 u;
      V t[PER];
    };
    const int64_t nv = n / PER;
    auto add = [&](const W (&wa)[U], const W (&wb)[U]) {
#pragma unroll
      for (int u = 0; u < U; u++)
#pragma unroll
        for (int q = 0; q < PER; q++)
          acc += (double)wa[u].t[q] * (double)wb[u].t[q];
    };
    int64_t i = tid;
    if (a == b) { // a squared norm: one stream
      for (; i + (U - 1) * nth < nv; i += U * nth) {
        W wa[U];
#pragma unroll
        for (int u = 0; u < U; u++)
          wa[u].u = ptx::ld_stream16(a + (i + u * nth) * PER, pol_s);
        add(wa, wa);
      }
    } else {
      for (; i + (U - 1) * nth < nv; i += U * nth) {
        W wa[U], wb[U];
#pragma unroll
        for (int u = 0; u < U; u++)
          wa[u].u = ptx::ld_stream16(a + (i + u * nth) * PER, pol_s);
#pragma unroll
        for (int u = 0; u < U; u++)
          wb[u].u = ptx::ld_stream16(b + (i + u * nth) * PER, pol_s);
        add(wa, wb);
      }
    }
    if (i < nv) { // the last trip: places past the end count as 0
      W wa[U], wb[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int64_t at = i + u * nth < nv ? i + u * nth : i;
        wa[u].u = ptx::ld_stream16(a + at * PER, pol_s);
        wb[u].u = ptx::ld_stream16(b + at * PER, pol_s);
      }
#pragma unroll
      for (int u = 1; u < U; u++)
        if (i + u * nth >= nv)
          wa[u].u = wb[u].u = make_uint4(0, 0, 0, 0);
      add(wa, wb);
    }
    done = nv * PER;
  }
  for (int64_t i = done + tid; i < n; i += nth)
    acc += (double)a[i] * (double)b[i];
  const double cta = dot_cta_sum(acc);
  if (gridDim.x == 1 || !TICKET) {
    if (threadIdx.x == 0)
      *(gridDim.x == 1 ? out : partials + blockIdx.x) = cta;
    return;
  }
  __shared__ int s_last;
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = cta;
    __threadfence();
    s_last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last)
    return;
  __threadfence();
  const double t = dot_partials_sum(partials, (int)gridDim.x);
  if (threadIdx.x == 0) {
    *out = t;
    *ticket = 0;
  }
}

__global__ void __launch_bounds__(kDotNT)
    dot_finish(const double *partials, int count, double *out) {
  ptx::grid_dependents_start();
  ptx::grid_dependency_wait(partials);
  const double t = dot_partials_sum(partials, count);
  if (threadIdx.x == 0)
    *out = t;
}

// ---- dot without allocation --------------------------------------------------
// Scratch of drb_dot_noalloc: one f64 partial per CTA plus the ticket, in a
// file-scope device array that every GPU loading the library keeps until
// process exit (kNoAllocSlots * 8 bytes + 256 = 512.25 KiB).  Each CTA covers
// kNoAllocBlock elements, so the largest vector is kNoAllocSlots *
// kNoAllocBlock elements.
constexpr int kNoAllocBlock = kDotNT * 32;   // 8192 elements per CTA
constexpr int kNoAllocSlots = 65536;         // partials (one per CTA)
constexpr int64_t kNoAllocMaxN = (int64_t)kNoAllocBlock * kNoAllocSlots; // 2^29
static __device__ __align__(256) double g_dot_noalloc_scratch[kNoAllocSlots + 32];

std::mutex g_noalloc_mu;
struct NoAllocAddr {
  unsigned long long ctx = 0; // id of the context the address belongs to
  void *addr = nullptr;
};
NoAllocAddr g_noalloc_addr[64];

// Device address of the scratch array in the current device's context.  Host
// code only sees a host-side stand-in under that name, so the address is
// looked up with cudaGetSymbolAddress on the first call in each context (the
// first call on a device, and the first after its context was destroyed and
// created again) and cached under the context's id.
drb_status noalloc_scratch(double **out) {
  int dev = 0;
  DRB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    set_error("drb_dot_noalloc: device %d out of range", dev);
    return DRB_ERR_UNSUPPORTED;
  }
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  unsigned long long id = 0;
  DRB_TRY(current_context(&id));
  NoAllocAddr &e = g_noalloc_addr[dev];
  if (id == 0 || e.ctx != id || !e.addr) {
    void *p = nullptr;
    DRB_CUDA_TRY(cudaGetSymbolAddress(&p, g_dot_noalloc_scratch)); // makes the context
    DRB_TRY(current_context(&id));
    e.ctx = id;
    e.addr = p;
  }
  *out = static_cast<double *>(e.addr);
  return DRB_OK;
}

} // namespace

int64_t dot_noalloc_max_n() { return kNoAllocMaxN; }

drb_status dot_noalloc_launch(int64_t n, const void *a, const void *b,
                              drb_dtype dt, double *out, cudaStream_t s) {
  if (n > kNoAllocMaxN) {
    set_error("drb_dot_noalloc: n = %lld exceeds the maximum %lld elements that its "
              "static scratch covers; use drb_dot",
              (long long)n, (long long)kNoAllocMaxN);
    return DRB_ERR_INVALID_ARG;
  }
  if (dt != DRB_F32 && dt != DRB_F64) {
    set_error("drb_dot_noalloc: dtype %d not supported", (int)dt);
    return DRB_ERR_UNSUPPORTED;
  }
  double *scratch = nullptr;
  DRB_TRY(noalloc_scratch(&scratch));
  int *ticket = reinterpret_cast<int *>(scratch + kNoAllocSlots);
  // the array keeps the previous call's contents: the ticket must start at 0
  DRB_CUDA_TRY(cudaMemsetAsync(ticket, 0, sizeof(int), s));
  const int64_t grid = std::max<int64_t>(1, (n + kNoAllocBlock - 1) / kNoAllocBlock);
  if (dt == DRB_F32)
    dot_kernel<float, true><<<(unsigned)grid, kDotNT, 0, s>>>(
        n, (const float *)a, (const float *)b, scratch, ticket, out);
  else
    dot_kernel<double, true><<<(unsigned)grid, kDotNT, 0, s>>>(
        n, (const double *)a, (const double *)b, scratch, ticket, out);
  note_launch();
  DRB_CUDA_TRY(cudaGetLastError());
  return DRB_OK;
}

drb_status dense_launch(int64_t m, int64_t n, const void *A, int64_t lda,
                        const void *x, void *y, int64_t k, drb_layout layout,
                        drb_dtype dt, cudaStream_t s) {
  if (m == 0 || k == 0)
    return DRB_OK;
  if (n == 0) {
    DRB_CUDA_TRY(cudaMemsetAsync(y, 0, (size_t)dtype_bytes(dt) * m * k, s));
    return DRB_OK;
  }
  if (dt == DRB_F32 || dt == DRB_F64) {
    if (k > 1)
      return dense_panel_launch(m, n, A, lda, x, y, k, layout, dt, s);
    if (dt == DRB_F32)
      return dense_row<float>(m, n, (const float *)A, lda, (const float *)x, (float *)y, s);
    return dense_row<double>(m, n, (const double *)A, lda, (const double *)x, (double *)y, s);
  }
  set_error("dense gemv: dtype %d not supported", (int)dt);
  return DRB_ERR_UNSUPPORTED;
}

drb_status dot_launch(int64_t n, const void *a, const void *b, drb_dtype dt,
                      double *out, cudaStream_t s) {
  if (dt != DRB_F32 && dt != DRB_F64) {
    set_error("dot: dtype %d not supported", (int)dt);
    return DRB_ERR_UNSUPPORTED;
  }
  // one CTA up to 16384 elements (its result needs no scratch and no second
  // pass), then one per 4096 up to four per SM
  const int grid = (int)(n <= 16384 ? 1 : std::min<int64_t>(kDotGrid, (n + 4095) / 4096));
  void *scratch = nullptr;
  if (grid > 1)
    DRB_TRY(scratch_alloc(&scratch, sizeof(double) * kDotGrid, s));
  double *partials = static_cast<double *>(scratch);
  cudaError_t e;
  if (dt == DRB_F32)
    e = launch_overlapped(dot_kernel<float, false>, dim3(grid), dim3(kDotNT), 0, s, n,
                          (const float *)a, (const float *)b, partials, (int *)nullptr, out);
  else
    e = launch_overlapped(dot_kernel<double, false>, dim3(grid), dim3(kDotNT), 0, s, n,
                          (const double *)a, (const double *)b, partials, (int *)nullptr, out);
  note_launch();
  if (e == cudaSuccess && grid > 1) {
    e = launch_overlapped(dot_finish, dim3(1), dim3(kDotNT), 0, s,
                          (const double *)partials, grid, out);
    note_launch();
  }
  if (scratch)
    scratch_free(scratch, s);
  if (e != cudaSuccess) {
    set_error("dot launch: %s", cudaGetErrorString(e));
    return DRB_ERR_CUDA;
  }
  return DRB_OK;
}

} // namespace drb
