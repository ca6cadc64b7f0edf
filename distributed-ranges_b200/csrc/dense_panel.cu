// dense_panel.cu -- dense row-major product with several right-hand sides:
// one pass over A for up to kPanelCols of them.
//
// What bounds it: A streams once from HBM (k is small), but every element of A
// meets k elements of X, so the operand path from shared memory to registers
// and the FMA pipes run close to the HBM rate as well (20 right-hand sides:
// 10 flop per byte of an f32 A, 5 of an f64 A).  Reading A once per block of
// eight right-hand sides, as a gemv repeated over column blocks does, costs
// ceil(k / 8) passes over HBM, and rows that do not start on 16 bytes went
// through single-element loads with few of them in flight.
//
// Measured (us), a gemv repeated over column blocks -> here: 5003 x 3001 f64 with 20
// right-hand sides 253 -> 50, f32 445 -> 38; 8192^2 f32 with 20 342 -> 102, with 8
// 138 -> 61, with 4 63 -> 53; 4096 x 8192 f64 with 32 437 -> 106.  (One CTA of 16 warps per SM with tiles twice as high
// ran the f64 case in 57: all warps loaded, waited and multiplied in step.)
//
// Tiles and split.  A CTA of 8 warps owns a tile of BM rows and walks along the
// columns in chunks of KC; the chunks of A and of X come through a
// STAGES-deep cp.async ring in 16-byte pieces.  Where rows of A or columns of X
// do not start on 16 bytes (odd sizes), a row is copied from the boundary below
// its start and read from its own offset in shared memory: copies of single
// elements ran at a third of the speed.  All chunks of all tiles form one list
// that is cut into equal consecutive shares, one per CTA, so the chip is full
// whatever the shape; a tile cut between CTAs leaves one partial per CTA, and
// panel_sum adds them in chunk order (deterministic).
//
//   f32: a warp has R rows; a lane takes every 16th column of A and one half of
//        the right-hand sides: R x C/2 sums per lane (an X value read from shared
//        memory serves R rows, an A value C/2 right-hand sides), so the FMA pipes
//        and the shared-memory path are about equally busy.  The lanes' sums
//        meet in a halving tree at the end of a tile.  Scalar fused multiply-adds:
//        the packed f32x2 form kept the pipe busy for four cycles each, half the
//        scalar rate.
//   f64: mma.sync m8n8k4: a warp has 16 rows x 8 NT right-hand sides and one
//        half of each chunk's columns (the halves meet in shared memory at the
//        end of a tile).  CUDA cores would need 2 (R + C) shared-memory cycles
//        for R C fused multiply-adds at half rate, and 4 R C registers.
#include <algorithm>

#include "drb_internal.cuh"

namespace drb {
namespace {

constexpr int kNT = 256;
constexpr int kCtas = 2; // per SM: one computes while the other waits for its loads
constexpr int kWarps = kNT / 32;
constexpr int kPanelCols = 32; // right-hand sides of one pass
constexpr int64_t kLongShare = 6; // see Shape
constexpr int64_t kTurnElems = (int64_t)1 << 21; // A above this: row-major X is transposed first

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// BYTES from global to shared memory, the last BYTES - n of them zeros.
template <int BYTES>
__device__ __forceinline__ void cp_zfill(uint32_t dst, const void *src, int n = BYTES) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;" ::"r"(dst), "l"(src), "r"(n),
                 "n"(BYTES)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N> __device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

struct PanelArgs {
  const void *A;
  const void *x;
  void *y;
  void *part; // [CTA][2][BM][CP] partial sums of cut tiles
  int64_t m, n, lda;
  int64_t x_cs, x_js; // address of X(c, j): c * x_cs + j * x_js
  int64_t y_ld, y_js; // address of Y(r, j): r * y_ld + j * y_js
  int k;
  int64_t cpt, chunks, share; // chunks per tile, in all, per CTA
};

// Tile shapes: BM rows, KC columns a chunk, AS / XS elements between the rows of
// a staged A / X chunk: a 16-byte multiple with room for the offset of a
// shifted row.  The rows of one shared-memory load hit different banks: f32
// right-hand sides of the two half-warps are 64 bytes apart modulo 128, f64 rows
// 64 bytes for the 16-byte fragment loads of aligned rows and 32 bytes for the
// 8-byte loads of shifted ones.
// LONG chunks are twice as wide in a ring of two: half the waits and longer runs
// of a row per copy, for shares of many chunks (a short share is over before
// they pay, and its last chunk is mostly padding; f64 with more than 16
// right-hand sides does not gain: its tensor pipe is as busy as the loads).
// Measured, us, short / long: 8192^2 f32 k = 20 105 / 94, 8191^2 k = 3 83 / 69,
// 8191 x 4095 f64 k = 5 80 / 70; 16000 x 300 f32 k = 12 9.9 / 11.1, 5003 x 3001
// f64 k = 20 49.7 / 51.3.
// FOLD chunks: a sum runs over 32 products (a lane's in f32, a warp's mma chain in
// f64) before it joins the tile's, since one chain over a whole tile grew its error
// with the row: N(0, 1) entries, 2-norm over the result's, blocks of columns before /
// one chain / folded: 16384 x 4096, k = 20, f32 2.1e-7 / 2.4e-7 / 1.3e-7, k = 32 2.1e-7 /
// 2.7e-7 / 1.3e-7, f64 3.0e-16 / 1.2e-15 / 3.0e-16; 16384 x 1024 f32 1.20e-7 / 1.30e-7 /
// 1.14e-7, f64 2.2e-16 / 6.0e-16 / 2.4e-16.  (Under 512 columns the shorter trees
// leave it 1.13 times the old one in f32, 1.45 in f64, whose chains of 16 would be
// 1.2.)  It costs, us: 5003 x 3001 k = 20 f64 48.2 -> 49.8, f32 37.3 -> 37.5; 8192^2 k = 20
// f32 92.6 -> 101.7, f64 122 -> 138; 8192 x 4096 k = 32 f32 78.7 -> 82.1, f64 93.3 -> 100.1.
// f64 keeps three short chunks per CTA in the ring, with more than 24 right-hand
// sides two (three / two, us: 8192 x 4096 k = 20 66 / 71, k = 32 100 / 95; 8192 x 1024
// k = 32 38 / 33, 5003 x 3001 k = 32 58 / 57).  Three CTAs of two chunks (8192 x 4096
// k = 20: 80) and warps of 32 rows (81; k = 32 105) measured slower.
template <class V, int P, bool SH, bool LONG> struct Shape;
template <int C, bool SH, bool LONG>
struct Shape<float, C, SH, LONG> { // C right-hand sides
  static constexpr int R = C <= 20 ? 8 : 4;
  static constexpr int BM = kWarps * R, KC = LONG ? 128 : 64, AS = KC + 4, XS = KC + 16, CP = C;
  static constexpr int STAGES = LONG ? 2 : 4, MERGE = 0, FOLD = 32 * 16 / KC;
};
template <int NT, bool SH, bool LONG>
struct Shape<double, NT, SH, LONG> { // 8 NT right-hand sides
  static constexpr int R = 16;
  static constexpr int BM = kWarps / 2 * R, KC = LONG ? 64 : 32, AS = KC + (SH ? 4 : 8), XS = AS;
  static constexpr int CP = 8 * NT, STAGES = LONG || NT == 4 ? 2 : 3;
  static constexpr int MERGE = BM * CP; // the second half's sums of a tile
  static constexpr int FOLD = LONG ? 1 : 2;
};
template <class V, int P> constexpr bool may_be_long() { return sizeof(V) == 4 || P <= 2; }
template <class V, int P, bool SH, bool LONG> constexpr size_t panel_smem() {
  using S = Shape<V, P, SH, LONG>;
  return ((size_t)S::STAGES * (S::BM * S::AS + S::CP * S::XS) + S::MERGE) * sizeof(V);
}

// Elements from the 16-byte boundary at or below p to p.
template <class V> __device__ __forceinline__ int shift_of(const V *p) {
  return (int)((reinterpret_cast<uintptr_t>(p) & 15) / sizeof(V));
}

// One 16-byte piece of a shifted row: element e0 of the row (kb - its offset +
// a multiple of a piece) lands at dst.  Zeros from element n on; elements below
// kb are not wanted.  [lo, hi) is the whole array: a piece that reaches
// outside it is copied element by element.
template <class V>
__device__ __forceinline__ void copy_edge_piece(uint32_t dst, const V *row, int64_t e0, int64_t kb,
                                                int64_t n, const V *lo, const V *hi) {
  constexpr int PER = 16 / (int)sizeof(V);
  const V *src = row + e0;
  if (e0 >= n) {
    // (nothing is read, but the address has to be a piece's)
    cp_zfill<16>(dst, reinterpret_cast<const void *>(reinterpret_cast<uintptr_t>(lo) & ~(uintptr_t)15),
                 0);
  } else if (src >= lo && src + PER <= hi) {
    cp_zfill<16>(dst, src, (int)min((int64_t)PER, n - e0) * (int)sizeof(V));
  } else {
    for (int i = 0; i < PER; i++)
      if (e0 + i >= kb)
        cp_zfill<sizeof(V)>(dst + i * (uint32_t)sizeof(V), e0 + i < n ? src + i : lo,
                            e0 + i < n ? (int)sizeof(V) : 0);
  }
}

template <class V, int P, bool SH, bool LONG>
__global__ void __launch_bounds__(kNT, kCtas) dense_panel(const PanelArgs a) {
  using S = Shape<V, P, SH, LONG>;
  constexpr int BM = S::BM, KC = S::KC, AS = S::AS, XS = S::XS, CP = S::CP, ST = S::STAGES;
  constexpr int PER = 16 / (int)sizeof(V), GR = KC / PER, RP = kNT / GR;
  extern __shared__ __align__(16) unsigned char panel_mem[];
  ptx::grid_dependents_start();
  ptx::grid_dependency_wait();
  V *sa = reinterpret_cast<V *>(panel_mem);
  V *sx = sa + (size_t)ST * BM * AS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const V *A = static_cast<const V *>(a.A);
  const V *X = static_cast<const V *>(a.x);
  const V *Aend = A + (a.m - 1) * a.lda + a.n;
  const V *Xend = X + (a.k - 1) * a.x_js + a.n;
  const int64_t c0 = (int64_t)blockIdx.x * a.share, c1 = min(a.chunks, c0 + a.share);
  const int cpt = (int)a.cpt;

  // The next chunk of the share -> ring slot st.  A thread's piece column is
  // fixed and its rows step by a constant, so a whole chunk costs one address
  // addition per piece.
  const int ar = tid / GR, ag = (tid % GR) * PER; // first row, piece column
  // A shifted row's offset depends on its index modulo a piece, which tiles,
  // warps' rows and a thread's row steps are multiples of: fixed per thread.
  const int sha = SH ? shift_of(A + ar * a.lda) : 0;
  const int sha_end = SH ? shift_of(A + tid * a.lda) : 0;
  const int shx = SH && a.x_cs == 1 ? shift_of(X + ar * a.x_js) : 0;
  const int shx_end = SH && a.x_cs == 1 ? shift_of(X + tid * a.x_js) : 0;
  int64_t lt = c0 / cpt; // tile and chunk of the next load
  int lc = (int)(c0 - lt * cpt);
  auto load = [&](int st) {
    const int64_t kb = (int64_t)lc * KC, r0 = lt * BM;
    // every piece lies in A (shifted rows: also what precedes the first one
    // and follows the last)
    const bool inside =
        kb + KC <= a.n && r0 + BM <= a.m &&
        (!SH || ((lt > 0 || lc > 0) && (r0 + BM < a.m || kb + KC + PER <= a.n)));
    if (++lc == cpt) {
      lc = 0;
      lt++;
    }
    const uint32_t s0 = smem_u32(sa + (size_t)st * BM * AS);
    const uint32_t da = s0 + (uint32_t)((ar * AS + ag) * sizeof(V));
    const V *row = A + (r0 + ar) * a.lda;
    const int64_t step = RP * a.lda;
    if (inside) {
      const V *src = row + kb + ag - sha;
#pragma unroll
      for (int p = 0; p < BM / RP; p++, src += step)
        cp_zfill<16>(da + (uint32_t)(p * RP * AS * sizeof(V)), src);
    } else {
#pragma unroll 1
      for (int p = 0; p < BM / RP; p++, row += step)
        if (r0 + ar + p * RP < a.m)
          copy_edge_piece<V>(da + (uint32_t)(p * RP * AS * sizeof(V)), row,
                             kb + ag - sha, kb, a.n, A, Aend);
    }
    if (SH && tid < BM && sha_end > 0 && r0 + tid < a.m) { // the piece past the chunk
      const V *rw = A + (r0 + tid) * a.lda;
      const uint32_t d = s0 + (uint32_t)((tid * AS + KC) * sizeof(V));
      if (inside)
        cp_zfill<16>(d, rw + kb + KC - sha_end);
      else
        copy_edge_piece<V>(d, rw, kb + KC - sha_end, kb, a.n, A, Aend);
    }
    const uint32_t dx = smem_u32(sx + (size_t)st * CP * XS);
    if (a.x_cs == 1) {
      const bool xin = SH ? kb > 0 && kb + KC + PER <= a.n : kb + KC <= a.n;
      for (int j = ar; j < a.k; j += RP) {
        const V *xc = X + j * a.x_js;
        const int64_t e0 = kb + ag - shx;
        const uint32_t d = dx + (uint32_t)((j * XS + ag) * sizeof(V));
        if (xin)
          cp_zfill<16>(d, xc + e0);
        else
          copy_edge_piece<V>(d, xc, e0, kb, a.n, X, Xend);
      }
      if (SH && tid < a.k && shx_end > 0) {
        const V *xc = X + tid * a.x_js;
        const uint32_t d = dx + (uint32_t)((tid * XS + KC) * sizeof(V));
        if (xin)
          cp_zfill<16>(d, xc + kb + KC - shx_end);
        else
          copy_edge_piece<V>(d, xc, kb + KC - shx_end, kb, a.n, X, Xend);
      }
    } else { // row-major X: 32-byte runs of right-hand sides, few bank conflicts
      constexpr int JL = 32 / (int)sizeof(V), CL = 32 / JL; // lanes over j, over c
      const int kn = (int)min((int64_t)KC, a.n - kb);
      const int jl = lane % JL;
      for (int c = warp * CL + lane / JL; c < KC; c += kWarps * CL)
        for (int j = jl; j < a.k; j += JL)
          cp_zfill<sizeof(V)>(dx + (uint32_t)((j * XS + c) * sizeof(V)),
                              c < kn ? X + (kb + c) * a.x_cs + j : X,
                              c < kn ? (int)sizeof(V) : 0);
    }
  };
  // first row of this warp; f64: its half of a chunk's columns
  const int wr = (sizeof(V) == 4 ? warp : warp % (kWarps / 2)) * S::R;
  const int kh = sizeof(V) == 4 ? 0 : warp / (kWarps / 2) * (KC / 2);
  // offsets of this lane's rows and columns in a staged chunk
  auto ashift = [&](int r) { return SH ? shift_of(A + r * a.lda) : 0; };
  auto xshift = [&](int j) { return SH && a.x_cs == 1 ? shift_of(X + j * a.x_js) : 0; };
  static_assert(BM % PER == 0 && RP % PER == 0 && S::R % PER == 0, "offsets repeat");
  int ra[PER], xj[2];
#pragma unroll
  for (int q = 0; q < PER; q++)
    ra[q] = sizeof(V) == 4 ? ashift(q) : ashift(lane >> 2);
#pragma unroll
  for (int q = 0; q < 2; q++) // (f32: columns cg, cg + 2, ...: four apart share an offset)
    xj[q] = sizeof(V) == 4 ? (lane >> 4) * XS + xshift((lane >> 4) + 2 * q) : xshift(lane >> 2);
  // this thread's sums of the current tile
  constexpr int R = S::R;
  constexpr int NACC = sizeof(V) == 4 ? R * CP / 2 : 2 * (CP / 8);
  float accf[sizeof(V) == 4 ? NACC : 1], sumf[sizeof(V) == 4 ? NACC / 16 : 1];
  double accd[sizeof(V) == 8 ? NACC : 1][2], sumd[sizeof(V) == 8 ? NACC : 1][2];
  auto clear = [&]() {
    if constexpr (sizeof(V) == 4) {
#pragma unroll
      for (int i = 0; i < NACC; i++)
        accf[i] = 0.0f;
    } else {
#pragma unroll
      for (int i = 0; i < NACC; i++)
        accd[i][0] = accd[i][1] = 0.0;
    }
  };
  auto clear_sums = [&]() {
    if constexpr (sizeof(V) == 4) {
#pragma unroll
      for (int i = 0; i < NACC / 16; i++)
        sumf[i] = 0.0f;
    } else {
#pragma unroll
      for (int i = 0; i < NACC; i++)
        sumd[i][0] = sumd[i][1] = 0.0;
    }
  };
  // The sums since the last fold join the tile's.  f32: the 16 lanes' sums
  // meet in a halving tree, which leaves a sixteenth of them in each lane.
  auto fold = [&]() {
    if constexpr (sizeof(V) == 4) {
      constexpr int N = NACC;
      static_assert(N % 16 == 0, "the halving tree needs a multiple of 16 sums");
      // each step a lane keeps one half of its sums and passes the other on
#pragma unroll
      for (int s = 0; s < 4; s++) {
        const int off = 8 >> s, h = N >> (s + 1);
        const bool up = lane & off;
#pragma unroll
        for (int i = 0; i < N / 2; i++)
          if (i < h) {
            const float keep = up ? accf[i + h] : accf[i], send = up ? accf[i] : accf[i + h];
            accf[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
          }
      }
#pragma unroll
      for (int i = 0; i < N / 16; i++)
        sumf[i] += accf[i];
    } else {
#pragma unroll
      for (int i = 0; i < NACC; i++) {
        sumd[i][0] += accd[i][0];
        sumd[i][1] += accd[i][1];
      }
    }
  };
  auto compute = [&](int st, bool fold_first) {
    const V *As = sa + (size_t)st * BM * AS + wr * AS;
    const V *Xs = sx + (size_t)st * CP * XS;
    if constexpr (sizeof(V) == 4) {
      constexpr int CH = CP / 2;
#pragma unroll 2
      for (int c = lane & 15; c < KC; c += 16) {
        float av[R];
#pragma unroll
        for (int r = 0; r < R; r++)
          av[r] = As[r * AS + ra[r % PER] + c];
#pragma unroll
        for (int j = 0; j < CH; j++) {
          const float xv = Xs[2 * j * XS + xj[j % 2] + c];
#pragma unroll
          for (int r = 0; r < R; r++)
            accf[r * CH + j] = fmaf(av[r], xv, accf[r * CH + j]);
        }
      }
    } else {
      constexpr int NT = CP / 8;
      const int fr = lane >> 2;
      // k order inside a step of eight: a lane's pair (aligned rows) or the
      // lane's column of either half (shifted rows); the same for A and X
      const int fk = SH ? (lane & 3) : 2 * (lane & 3);
      const V *Ap[2], *Xp = Xs + fr * XS + fk + xj[0] + kh; // 8 columns on: the same offset
#pragma unroll
      for (int i = 0; i < 2; i++)
        Ap[i] = As + (i * 8 + fr) * AS + fk + kh + ra[0];
#pragma unroll
      for (int c = 0; c < KC / 2; c += 8) {
        double2 av[2], bv[NT];
#pragma unroll
        for (int i = 0; i < 2; i++) {
          if constexpr (SH)
            av[i] = make_double2(Ap[i][c], Ap[i][c + 4]);
          else
            av[i] = *reinterpret_cast<const double2 *>(Ap[i] + c);
        }
#pragma unroll
        for (int t = 0; t < NT; t++) {
          if constexpr (SH)
            bv[t] = make_double2(Xp[t * 8 * XS + c], Xp[t * 8 * XS + c + 4]);
          else
            bv[t] = *reinterpret_cast<const double2 *>(Xp + t * 8 * XS + c);
        }
        if (c == 0 && fold_first) {
          fold();
          clear();
        }
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int t = 0; t < NT; t++)
            dmma(accd[i * NT + t], av[i].x, bv[t].x);
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int t = 0; t < NT; t++)
            dmma(accd[i * NT + t], av[i].y, bv[t].y);
      }
    }
  };
  // the tile's sums to Y (all its chunks were this CTA's) or to the partials
  auto emit = [&](int64_t tile) {
    const int64_t t0 = tile * cpt, t1 = t0 + cpt;
    const bool whole = t0 >= c0 && t1 <= c1;
    V *P0 = static_cast<V *>(a.part) +
            ((int64_t)blockIdx.x * 2 + (tile == c0 / cpt ? 0 : 1)) * BM * CP;
    V *Y = static_cast<V *>(a.y);
    auto put = [&](int r, int j, V v) {
      if (!whole)
        P0[r * CP + j] = v;
      else if (tile * BM + r < a.m && j < a.k)
        Y[(tile * BM + r) * a.y_ld + j * a.y_js] = v;
    };
    if constexpr (sizeof(V) == 4) {
      constexpr int CH = CP / 2, N = R * CH;
      int f0 = 0;
#pragma unroll
      for (int s = 0; s < 4; s++)
        if (lane & (8 >> s))
          f0 += N >> (s + 1);
#pragma unroll
      for (int i = 0; i < N / 16; i++)
        put(wr + (f0 + i) / CH, (lane >> 4) + 2 * ((f0 + i) % CH), sumf[i]);
    } else {
      // the second half's warps hand their sums over
      constexpr int NT = CP / 8;
      double *mine = sx + (size_t)ST * CP * XS + wr * CP;
      auto at = [&](int i, int t, int e) {
        return (i * 8 + (lane >> 2)) * CP + t * 8 + 2 * (lane & 3) + e;
      };
      if (kh) {
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int t = 0; t < NT; t++)
            *reinterpret_cast<double2 *>(mine + at(i, t, 0)) =
                make_double2(sumd[i * NT + t][0], sumd[i * NT + t][1]);
      }
      __syncthreads();
      if (!kh) {
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int t = 0; t < NT; t++)
#pragma unroll
            for (int e = 0; e < 2; e++)
              put(wr + i * 8 + (lane >> 2), t * 8 + 2 * (lane & 3) + e,
                  sumd[i * NT + t][e] + mine[at(i, t, e)]);
      }
    }
  };

  int64_t ct = c0 / cpt;                      // current tile
  int left = cpt - (int)(c0 - ct * cpt);      // chunks left in it
  if (c1 - c0 < left)
    left = (int)(c1 - c0); // (of this CTA's)
  int run = min(left, S::FOLD); // chunks until the next fold
  bool fold_next = false; // f64: fold in the next chunk, behind whose loads the adds hide
#pragma unroll
  for (int s = 0; s < ST - 1; s++) {
    if (c0 + s < c1)
      load(s);
    cp_commit();
  }
  clear();
  clear_sums();
  int st = 0;
  for (int64_t q = c0; q < c1; q++) {
    cp_wait<ST - 2>();
    __syncthreads(); // chunk q landed; slot st - 1 is free
    const int fill = st == 0 ? ST - 1 : st - 1;
    if (q + ST - 1 < c1)
      load(fill);
    cp_commit();
    compute(st, fold_next);
    left--;
    fold_next = false;
    if (--run == 0) {
      if (sizeof(V) == 4 || left == 0) {
        fold();
        clear();
      } else {
        fold_next = true;
      }
      if (left == 0) {
        emit(ct);
        clear_sums();
        left = (int)min((int64_t)cpt, c1 - q - 1);
        ct++;
      }
      run = min(left, S::FOLD);
    }
    st = st + 1 == ST ? 0 : st + 1;
  }
  cp_wait<0>();
}

// Y of the tiles cut between CTAs: their partials added in a fixed order.  A
// group of PW threads (in different warps, so that a warp reads consecutive
// partials) takes every PW-th piece of an output and thread 0 of the group adds
// the groups' sums: one piece after another, a 300 x 16000 matrix's tiles, cut
// into 59 pieces, kept the pass busy longer than the product.
template <class V, int PW>
__global__ void __launch_bounds__(256) panel_sum(const PanelArgs a, int BM, int CP) {
  __shared__ V s_sum[256];
  ptx::grid_dependency_wait();
  constexpr int OUT = 256 / PW; // outputs per CTA
  const V *part = static_cast<const V *>(a.part);
  V *Y = static_cast<V *>(a.y);
  const int w = threadIdx.x / OUT, o = threadIdx.x % OUT;
  for (int64_t i0 = (int64_t)blockIdx.x * OUT; i0 < a.m * a.k; i0 += (int64_t)gridDim.x * OUT) {
    const int64_t i = i0 + o;
    const bool in = i < a.m * a.k;
    int64_t r = 0;
    int j = 0;
    if (in && a.y_ld == 1) { // consecutive threads write consecutive addresses
      j = (int)(i / a.m);
      r = i - (int64_t)j * a.m;
    } else if (in) {
      r = i / a.k;
      j = (int)(i - r * a.k);
    }
    const int64_t tile = r / BM;
    const int64_t b0 = tile * a.cpt / a.share, b1 = ((tile + 1) * a.cpt - 1) / a.share;
    const bool cut = in && b0 != b1; // else one CTA had the whole tile
    V s = 0;
    if (cut) {
      // every piece but the first opens its CTA's share (slot 0)
      const V *p = part + (r - tile * BM) * CP + j;
      const int64_t step = 2 * (int64_t)BM * CP;
      const int slot0 = tile == b0 * a.share / a.cpt ? 0 : 1;
      int64_t b = b0 + w;
      if (w == 0) {
        s = p[b * step + slot0 * (int64_t)BM * CP];
        b += PW;
      }
#pragma unroll 4
      for (; b <= b1; b += PW)
        s += p[b * step];
    }
    if constexpr (PW > 1) {
      __syncthreads(); // (the previous outputs' sums have been read)
      s_sum[threadIdx.x] = s;
      __syncthreads();
      if (w > 0)
        continue;
#pragma unroll
      for (int q = 1; q < PW; q++)
        s += s_sum[q * OUT + o];
    }
    if (cut && w == 0)
      Y[r * a.y_ld + j * a.y_js] = s;
  }
}

template <class V, int P, bool SH, bool LONG>
drb_status panel_run(PanelArgs a, cudaStream_t s) {
  using S = Shape<V, P, SH, LONG>;
  constexpr size_t smem = panel_smem<V, P, SH, LONG>();
  static std::atomic<unsigned long long> allowed[64];
  int dev = 0, sms = 0;
  DRB_CUDA_TRY(cudaGetDevice(&dev));
  DRB_TRY(device_sms(dev, &sms));
  DRB_TRY(once_per_context(allowed, dev, [&]() -> drb_status {
    DRB_CUDA_TRY(cudaFuncSetAttribute(dense_panel<V, P, SH, LONG>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return DRB_OK;
  }));
  const int64_t tiles = (a.m + S::BM - 1) / S::BM;
  a.cpt = (a.n + S::KC - 1) / S::KC;
  a.chunks = tiles * a.cpt;
  // Equal shares over the resident CTAs, of at least kMinShare chunks: a
  // shorter share is over before the ring is full, and a tile cut into more
  // pieces only adds partials.
  constexpr int64_t kMinShare = 4;
  const int64_t ctas = (int64_t)kCtas * sms;
  a.share = std::max((a.chunks + ctas - 1) / ctas, std::min(kMinShare, a.cpt));
  // Shares of many tiles end on a tile: the rounding costs under 1/16, the
  // partials and their pass are saved.
  if (a.share >= 16 * a.cpt)
    a.share = (a.share + a.cpt - 1) / a.cpt * a.cpt;
  const int64_t grid = (a.chunks + a.share - 1) / a.share;
  const bool cut = a.share % a.cpt != 0;
  a.part = nullptr;
  if (cut)
    DRB_TRY(scratch_alloc(&a.part, sizeof(V) * 2 * (size_t)grid * S::BM * S::CP, s));
  cudaError_t e =
      launch_overlapped(dense_panel<V, P, SH, LONG>, dim3((unsigned)grid), dim3(kNT), smem, s, a);
  note_launch();
  if (e == cudaSuccess && cut) {
    const bool many = a.cpt > 4 * a.share; // pieces of a tile
    const int out = many ? 32 : 256;
    const unsigned g = (unsigned)std::max<int64_t>(
        1, std::min<int64_t>(8 * (int64_t)sms, (a.m * a.k + out - 1) / out));
    e = many ? launch_overlapped(panel_sum<V, 8>, dim3(g), dim3(256), 0, s, a, S::BM, S::CP)
             : launch_overlapped(panel_sum<V, 1>, dim3(g), dim3(256), 0, s, a, S::BM, S::CP);
    note_launch();
  }
  if (a.part)
    scratch_free(a.part, s);
  if (e != cudaSuccess) {
    set_error("dense gemv launch: %s", cudaGetErrorString(e));
    return DRB_ERR_CUDA;
  }
  return DRB_OK;
}

template <class V, int P> drb_status panel_align(const PanelArgs &a, cudaStream_t s) {
  const bool aligned = reinterpret_cast<uintptr_t>(a.A) % 16 == 0 &&
                       a.lda * sizeof(V) % 16 == 0 &&
                       (a.x_cs != 1 || (reinterpret_cast<uintptr_t>(a.x) % 16 == 0 &&
                                        a.x_js * sizeof(V) % 16 == 0));
  if constexpr (may_be_long<V, P>()) {
    // at least kLongShare long chunks for every CTA of the GPU
    int dev = 0, sms = 0;
    DRB_CUDA_TRY(cudaGetDevice(&dev));
    DRB_TRY(device_sms(dev, &sms));
    using S = Shape<V, P, false, true>;
    const int64_t chunks = (a.m + S::BM - 1) / S::BM * ((a.n + S::KC - 1) / S::KC);
    if (a.n >= 8 * S::KC && chunks >= kLongShare * kCtas * sms)
      return aligned ? panel_run<V, P, false, true>(a, s) : panel_run<V, P, true, true>(a, s);
  }
  return aligned ? panel_run<V, P, false, false>(a, s) : panel_run<V, P, true, false>(a, s);
}

drb_status panel_cols(const PanelArgs &a, float, cudaStream_t s) {
  if (a.k <= 4)
    return panel_align<float, 4>(a, s);
  if (a.k <= 8)
    return panel_align<float, 8>(a, s);
  if (a.k <= 12)
    return panel_align<float, 12>(a, s);
  if (a.k <= 16)
    return panel_align<float, 16>(a, s);
  if (a.k <= 20)
    return panel_align<float, 20>(a, s);
  if (a.k <= 24)
    return panel_align<float, 24>(a, s);
  return panel_align<float, 32>(a, s);
}
drb_status panel_cols(const PanelArgs &a, double, cudaStream_t s) {
  if (a.k <= 8)
    return panel_align<double, 1>(a, s);
  if (a.k <= 16)
    return panel_align<double, 2>(a, s);
  if (a.k <= 24)
    return panel_align<double, 3>(a, s);
  return panel_align<double, 4>(a, s);
}

template <class V>
drb_status panel_typed(int64_t m, int64_t n, const V *A, int64_t lda, const V *x, V *y,
                       int64_t k, drb_layout layout, cudaStream_t s) {
  const bool rm = layout == DRB_ROW_MAJOR;
  if (rm && (n + 31) / 32 > 65535) { // the limit of the layout transposes
    set_error("transpose: %lld rows exceed the grid limit", (long long)n);
    return DRB_ERR_UNSUPPORTED;
  }
  // Row-major X is gathered element by element in every chunk, which a large A
  // pays for more than one transpose of X (a launch) costs.
  const bool turn = rm && m * n > kTurnElems;
  void *xt = nullptr;
  if (turn) {
    DRB_TRY(scratch_alloc(&xt, sizeof(V) * (size_t)n * k, s));
    const drb_status st = transpose_launch(x, xt, n, k, sizeof(V), s);
    if (st != DRB_OK) {
      scratch_free(xt, s);
      return st;
    }
    x = static_cast<const V *>(xt);
  }
  PanelArgs a{};
  a.A = A;
  a.m = m;
  a.n = n;
  a.lda = lda;
  a.x_cs = rm && !turn ? k : 1;
  a.x_js = rm && !turn ? 1 : n;
  a.y_ld = rm ? k : 1;
  a.y_js = rm ? 1 : m;
  // more right-hand sides than one pass takes: equal blocks
  const int64_t nb = (k + kPanelCols - 1) / kPanelCols, kb = (k + nb - 1) / nb;
  for (int64_t j = 0; j < k; j += kb) {
    a.k = (int)std::min(kb, k - j);
    a.x = x + j * a.x_js;
    a.y = y + j * a.y_js;
    const drb_status st = panel_cols(a, V(0), s);
    if (st != DRB_OK) {
      if (xt)
        scratch_free(xt, s);
      return st;
    }
  }
  if (xt)
    scratch_free(xt, s);
  return DRB_OK;
}

} // namespace

drb_status dense_panel_launch(int64_t m, int64_t n, const void *A, int64_t lda, const void *x,
                              void *y, int64_t k, drb_layout layout, drb_dtype dt,
                              cudaStream_t s) {
  if (dt == DRB_F32)
    return panel_typed<float>(m, n, static_cast<const float *>(A), lda,
                              static_cast<const float *>(x), static_cast<float *>(y), k, layout,
                              s);
  return panel_typed<double>(m, n, static_cast<const double *>(A), lda,
                             static_cast<const double *>(x), static_cast<double *>(y), k, layout,
                             s);
}

} // namespace drb
