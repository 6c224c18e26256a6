// gemm_dmma.cu -- batched FP64 GEMM items (N > 32) on the FP64 tensor-core
// instruction mma.sync.m16n8k4.f64 (DMMA).
//
// The plain FP64 path (the reference's arithmetic: dgemm in the leaf solve's
// blocked LU, the reduce V^T [d | u] of gemm.cc:315-384 and the broadcast
// d -= u eta of gemm.cc:417-478) runs every wide product through this kernel:
//   C = beta Cin + alpha sum_s op(A_s) B_s,  op(A) = A (M x K) or A^T (A K x M).
// One CTA computes a BM x BN tile of one item, WM x WN warps of 16 MT x 32
// outputs each; K advances 16 at a time through a 3-stage cp.async ring, one
// barrier per stage.  The kernel is bound by the FP64 pipe: 37.0 TFLOP/s of
// m16n8k4 on this part, reached by one warp per SM quarter (measured with
// registers only; k8 and k16 forms run at the same rate), so what matters is
// that no quarter waits for copies.  Hence
//   * the copies of a stage advance per-thread pointers (no per-copy 64-bit
//     address arithmetic); rows beyond the item repeat its last row, whose
//     products land in outputs that are never stored, so that only the last,
//     partial stage of a K segment needs per-element bounds;
//   * operands off a 16-byte boundary (odd leading dimensions or row
//     offsets: any system whose leaves do not start on even rows) take
//     8-byte copies through the same pointers;
//   * small tiles: two to four CTAs per SM, one's C loads and stores under
//     another's products (K is only 32..128 in the leaf updates and r in the
//     broadcast, so a tile's prologue and epilogue are a third of its life).
// Shared-memory layouts (doubles):
//   op(A) = A:    As[k][m], row stride BM + 4   (m contiguous, like A)
//   op(A) = A^T:  As[m][k], row stride 20       (k contiguous, like A)
//   B:            Bs[n][k], row stride 20       (k contiguous, like B)
// The strides put the 16 lanes of each half-warp's fragment loads in 16
// distinct 8-byte bank slots.  For the in-place updates (alpha = +-1,
// beta = 1) the accumulators start from alpha * Cin, so the C tile's loads
// overlap the main loop: alpha * (alpha * c + s) == c + alpha * s exactly.
#include <type_traits>

#include "common.cuh"
#include "gemm_dmma.cuh"
#include "warp_f64.cuh"

namespace hodlr {

namespace {

constexpr int BK = 16, kStages = 3;
constexpr int LDK = BK + 4;  // k-contiguous row stride (doubles)

__device__ inline void cpa16(double *dst, const double *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src));
}
__device__ inline void cpa8(double *dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src));
}
// 8 bytes, or zero without `ok` (src must be readable memory either way)
__device__ inline void cpa8z(double *dst, const double *src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(ok ? 8 : 0));
}
__device__ inline void cpa_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ inline void cpa_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

template <int BM, bool TRANS>
constexpr int a_stage_doubles() {
  return TRANS ? BM * LDK : BK * (BM + 4);
}
template <int BN>
constexpr int b_stage_doubles() { return BN * LDK; }
template <int BM, int BN, bool TRANS>
constexpr size_t tile_smem() {
  return (size_t)kStages * (a_stage_doubles<BM, TRANS>() + b_stage_doubles<BN>()) * sizeof(double);
}

// Copies of a k-contiguous operand (ROWS rows of BK doubles, row r at
// base + (row0 + r) ld + k): thread tid's share as 16-byte pairs, pair
// kv = 2 (tid % 8) of the rows tid / 8, tid / 8 + THREADS / 8, ...
template <int ROWS, int THREADS>
struct KRows {
  static constexpr int STEP = THREADS / (BK / 2);
  static constexpr int NC = (ROWS + STEP - 1) / STEP;
  const double *p[NC];
  bool vec;
  __device__ void start(const double *base, long long ld, int row0, int rows) {
    const int r = threadIdx.x / (BK / 2), kv = 2 * (threadIdx.x % (BK / 2));
    vec = ((reinterpret_cast<uintptr_t>(base) & 15) == 0) && ((ld & 1) == 0);
#pragma unroll
    for (int i = 0; i < NC; ++i)
      p[i] = base + kv + (long long)min(row0 + r + i * STEP, rows - 1) * ld;
  }
  // the stage at the pointers, `left` k-values of the segment remaining
  __device__ void copy(double *s, int left) {
    const int r = threadIdx.x / (BK / 2), kv = 2 * (threadIdx.x % (BK / 2));
    double *d = s + r * LDK + kv;
    if (left >= BK) {
      if (vec) {
#pragma unroll
        for (int i = 0; i < NC; ++i)
          if (ROWS % STEP == 0 || r + i * STEP < ROWS) cpa16(d + i * STEP * LDK, p[i]);
      } else {
#pragma unroll
        for (int i = 0; i < NC; ++i)
          if (ROWS % STEP == 0 || r + i * STEP < ROWS) {
            cpa8(d + i * STEP * LDK, p[i]);
            cpa8(d + i * STEP * LDK + 1, p[i] + 1);
          }
      }
    } else {
#pragma unroll
      for (int i = 0; i < NC; ++i)
        if (ROWS % STEP == 0 || r + i * STEP < ROWS) {
          const bool ok0 = kv < left, ok1 = kv + 1 < left;
          cpa8z(d + i * STEP * LDK, ok0 ? p[i] : p[i] - kv, ok0);
          cpa8z(d + i * STEP * LDK + 1, ok1 ? p[i] + 1 : p[i] - kv, ok1);
        }
    }
#pragma unroll
    for (int i = 0; i < NC; ++i) p[i] += BK;
  }
};

// Copies of an m-contiguous operand (BK columns of BM doubles, column k at
// base + m0 + k ld): pair mv of the columns k = tid / (BM / 2), ...
template <int BM, int THREADS>
struct MCols {
  static constexpr int STEP = THREADS / (BM / 2);
  static constexpr int NC = BK / STEP;
  static_assert(STEP >= 1 && THREADS % (BM / 2) == 0 && BK % STEP == 0, "whole columns per pass");
  const double *p;
  long long ld;
  bool vec, one;  // pair on a 16-byte boundary; the pair's second row is outside
  __device__ void start(const double *base, long long ld_, int m0, int rows) {
    const int k = threadIdx.x / (BM / 2), mv = 2 * (threadIdx.x % (BM / 2));
    const int m = min(m0 + mv, rows - 1);
    ld = ld_;
    one = m + 1 >= rows;
    vec = ((reinterpret_cast<uintptr_t>(base) & 15) == 0) && ((ld & 1) == 0) && ((m & 1) == 0) &&
          !one;
    p = base + m + (long long)k * ld;
  }
  // only the rows [lo, hi)
  __device__ void copy(double *s, int left, int lo = 0, int hi = BM) {
    const int k = threadIdx.x / (BM / 2), mv = 2 * (threadIdx.x % (BM / 2));
    double *d = s + k * (BM + 4) + mv;
    const int u = one ? 0 : 1;
    if (mv < lo || mv >= hi) {
    } else if (left >= BK) {
      if (vec) {
#pragma unroll
        for (int i = 0; i < NC; ++i) cpa16(d + i * STEP * (BM + 4), p + i * STEP * ld);
      } else {
#pragma unroll
        for (int i = 0; i < NC; ++i) {
          cpa8(d + i * STEP * (BM + 4), p + i * STEP * ld);
          cpa8(d + i * STEP * (BM + 4) + 1, p + i * STEP * ld + u);
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        const bool ok = k + i * STEP < left;
        const double *q = ok ? p + i * STEP * ld : p - k * ld;
        cpa8z(d + i * STEP * (BM + 4), q, ok);
        cpa8z(d + i * STEP * (BM + 4) + 1, q + u, ok);
      }
    }
    p += BK * ld;
  }
};

template <int WM, int WN, int MT, bool TRANS>
__global__ void __launch_bounds__(WM *WN * 32, WM * WN == 4 ? 3 : 2)
    gemm_dmma_tile_kernel(const GemmItem<double, double> *__restrict__ items,
                          const GemmSeg<double> *__restrict__ segs, double alpha, double beta,
                          int mtiles, int ntiles) {
  constexpr int THREADS = WM * WN * 32, BM = WM * MT * 16, BN = WN * 32;
  constexpr int AP = BM + 4;  // As[k][m] row stride (non-trans)
  constexpr int AS = a_stage_doubles<BM, TRANS>(), BS = b_stage_doubles<BN>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *As = reinterpret_cast<double *>(smem_raw);
  double *Bs = As + (size_t)kStages * AS;
  // one-dimensional grid, the tiles of an item consecutive (column tiles
  // fastest): CTAs resident together share the item's A rows and B columns
  // through L2
  const int per = mtiles * ntiles;
  const int itx = blockIdx.x / per, rem = blockIdx.x - itx * per;
  const GemmItem<double, double> it = items[itx];
  const int m0 = (rem / ntiles) * BM, n0 = (rem % ntiles) * BN;
  if (m0 >= it.M || n0 >= it.N) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wn = (warp % WN) * 32;
  // tile row of the warp's row fragment mt: fragments w and 2 WM - 1 - w, so
  // that a triangular A gives every warp (each on its own SM quarter) the same
  // number of products
  auto frow = [&](int mt) {
    return 16 * (mt & 1 ? MT * WM - 1 - warp / WN : warp / WN);
  };
  static_assert(MT <= 2, "two fragments mirror each other");

  // the item's K stages, flattened over its segments
  KRows<BN, THREADS> cb;
  std::conditional_t<TRANS, KRows<BM, THREADS>, MCols<BM, THREADS>> ca;
  int seg = it.seg_begin;
  const int seg_end = it.seg_begin + it.seg_count;
  int left = 0;  // k-values of the current segment not yet copied
  auto settle = [&]() {
    for (; seg < seg_end; ++seg) {
      const GemmSeg<double> sg = segs[seg];
      if (sg.K <= 0) continue;
      left = sg.K;
      ca.start(sg.A, sg.lda, m0, it.M);
      cb.start(sg.B, sg.ldb, n0, it.N);
      ++seg;
      return;
    }
  };
  // A's zero half (the leaf LU's block-row solves) is neither copied nor
  // multiplied: stage i of a lower (upper) triangle holds values only in the
  // rows from (up to) its 16-row fragment i.  N = 262144, leaf 512, r = 64,
  // m = 16: block solves and inverses 2.76 -> 2.45 ms, the backward solve
  // 3.60 -> 3.38 ms, the solve 21.9 -> 21.4 ms.
  const int tri = !TRANS && it.seg_count == 1 ? segs[seg].tri : 0;
  int copied = 0;  // stages
  int stages = 0;
  for (int s = seg; s < seg_end; ++s) stages += (max(segs[s].K, 0) + BK - 1) / BK;
  auto load = [&](int st) {
    if (left <= 0) settle();
    if (left > 0) {
      if constexpr (TRANS)
        ca.copy(As + (size_t)st * AS, left);
      else
        ca.copy(As + (size_t)st * AS, left, tri == 1 ? BK * copied : 0,
                tri == 2 ? BK * (copied + 1) : BM);
      ++copied;
      cb.copy(Bs + (size_t)st * BS, left);
      left -= BK;
    }
    cpa_commit();
  };
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) load(i);

  double acc[MT][4][4];
  const bool preload = it.Cin && beta == 1.0 && (alpha == 1.0 || alpha == -1.0);
  // Cin at this thread's outputs of row fragment mt, every load issued before
  // any is used (rows and columns outside the item repeat its last ones, for
  // outputs that are not stored)
  auto load_cin = [&](int mt, double (&c)[4][4]) {
    const int row = m0 + frow(mt) + g;
    const double *c0 = it.Cin + min(row, it.M - 1), *c1 = it.Cin + min(row + 8, it.M - 1);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const long long o = min(n0 + wn + nt * 8 + 2 * t + u, it.N - 1) * it.ldcin;
        c[nt][u] = c0[o];
        c[nt][2 + u] = c1[o];
      }
  };
  if (preload) {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) load_cin(mt, acc[mt]);
    if (alpha != 1.0) {
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int v = 0; v < 4; ++v) acc[mt][nt][v] = -acc[mt][nt][v];
    }
  } else {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[mt][nt][v] = 0.0;
  }

  auto run = [&](auto triangular) {
    constexpr bool TRI = decltype(triangular)::value;
    int st = 0, lst = kStages - 1;
    for (int i = 0; i < stages; ++i) {
      cpa_wait<kStages - 2>();  // this thread's copies of stage i have landed
      __syncthreads();          // ... and everybody's; slot lst (stage i - 1) is free
      load(lst);
      lst = lst + 1 == kStages ? 0 : lst + 1;
      const double *a = As + (size_t)st * AS;
      const double *b = Bs + (size_t)st * BS;
#pragma unroll
      for (int ks = 0; ks < BK; ks += 4) {
        double bv[4];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) bv[nt] = b[(wn + nt * 8 + g) * LDK + ks + t];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          if (TRI && (tri == 1 ? frow(mt) < BK * i : frow(mt) > BK * i)) continue;
          const int mr = frow(mt) + g;
          const double a0 = TRANS ? a[mr * LDK + ks + t] : a[(ks + t) * AP + mr];
          const double a1 = TRANS ? a[(mr + 8) * LDK + ks + t] : a[(ks + t) * AP + mr + 8];
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) dmma(acc[mt][nt], a0, a1, bv[nt]);
        }
      }
      st = st + 1 == kStages ? 0 : st + 1;
    }
  };
  if constexpr (TRANS) {
    run(std::false_type{});
  } else {
    if (tri) run(std::true_type{});
    else run(std::false_type{});
  }
  cpa_wait<0>();

  const bool add = it.Cin && !preload;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    double (&x)[4][4] = acc[mt];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int v = 0; v < 4; ++v) x[nt][v] *= alpha;
    if (add) {
      double c[4][4];
      load_cin(mt, c);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int v = 0; v < 4; ++v) x[nt][v] += beta * c[nt][v];
    }
    const int row = m0 + frow(mt) + g;
    const bool ok0 = row < it.M, ok1 = row + 8 < it.M;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int col = n0 + wn + nt * 8 + 2 * t + u;
        double *d = it.C + row + col * it.ldc;
        if (ok0 && col < it.N) d[0] = x[nt][u];
        if (ok1 && col < it.N) d[8] = x[nt][2 + u];
      }
  }
}

template <int WM, int WN, int MT>
void launch_tile(const GemmItem<double, double> *items, const GemmSeg<double> *segs, int nitems,
                 int max_m, int max_n, bool trans, double alpha, double beta, cudaStream_t s) {
  constexpr int BM = WM * MT * 16, BN = WN * 32;
  const int mt = cdiv(max_m, BM), nt = cdiv(max_n, BN);
  const long long total = (long long)nitems * mt * nt;
  if (total > 0x7fffffffLL) throw CudaError{cudaErrorInvalidConfiguration};
  auto go = [&](auto kern, size_t smem) {
    raise_smem_limit(reinterpret_cast<const void *>(kern), smem);
    kern<<<(unsigned)total, WM * WN * 32, smem, s>>>(items, segs, alpha, beta, mt, nt);
  };
  if (trans) go(gemm_dmma_tile_kernel<WM, WN, MT, true>, tile_smem<BM, BN, true>());
  else go(gemm_dmma_tile_kernel<WM, WN, MT, false>, tile_smem<BM, BN, false>());
  HODLR_LAUNCH_CHECK();
}

}  // namespace

void launch_dmma_tile(const GemmItem<double, double> *items, const GemmSeg<double> *segs,
                      int nitems, int max_m, int max_n, bool trans, double alpha, double beta,
                      cudaStream_t s) {
  if (nitems <= 0 || max_m <= 0 || max_n <= 0) return;
  // Non-transposed items of at most 128 rows run as one tile row: the leaf
  // LU's block-row solves compute C = L^{-1} C in place (C is also the B
  // operand), which is only correct when a single CTA reads all of C's rows
  // before it writes any.  Taller items (the trailing updates, the
  // broadcast) and transposed ones (the reduce) are never in place.
  //
  // Tiles (N = 262144, leaf 512, r = 64, m = 16, FP64 solve with 128-column
  // leaf blocks): 64 x 64 at three CTAs of four warps per SM runs the
  // broadcast in 4.14 ms and the leaf updates in 4.08 ms; 64 x 128 at two
  // CTAs of eight warps 4.98 / 4.45 ms, 128 x 64 4.21 / 4.47 ms (and the
  // reduce in 7.36 instead of 3.76 ms, half of its rows being padding at
  // r = 64), 64 x 64 at four CTAs (128 registers) 4.38 / 4.15 ms.
  // Launches of fewer 64 x 64 tiles than SMs run 32-row tiles: at such sizes
  // a tile's own products, one SM's share of the FP64 pipe, are the time.
  const bool inplace = !trans && max_m <= 128;
  const long long tiles = (long long)nitems * cdiv(max_m, 64) * cdiv(max_n, 64);
  if (max_m <= 32 || (!inplace && tiles < 148))
    launch_tile<2, 2, 1>(items, segs, nitems, max_m, max_n, trans, alpha, beta, s);
  else if (max_m <= 64 || max_m > 128)
    launch_tile<2, 2, 2>(items, segs, nitems, max_m, max_n, trans, alpha, beta, s);
  else if (trans)
    launch_tile<4, 2, 2>(items, segs, nitems, max_m, max_n, trans, alpha, beta, s);
  else
    launch_tile<4, 1, 2>(items, segs, nitems, max_m, max_n, trans, alpha, beta, s);
}

}  // namespace hodlr
