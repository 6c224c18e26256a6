// leaf_blocked.cu -- batched blocked leaf factorization on [D | X].
//
// The leaf task body (src/solver/solver_tasks.cc:424-450) is dgesv(D, X) on
// all m + r*L columns of the leaf.  On the GPU every leaf of the tree is
// factored at once, panel by panel (NB columns), as a right-looking blocked
// LU of the augmented matrix [D | X]:
//
//   for each panel k0:
//     leaf_panel_reg_kernel  one CTA per leaf: LU with partial pivoting of
//                         D[k0:n, k0:k0+NB] in registers (LAPACK idamax
//                         tie rule), written back; the inverses of the
//                         panel's unit-lower and upper diagonal blocks are
//                         formed for the solves; ipiv / perm updated,
//                         per-leaf "had interchanges" flag
//     leaf_laswp_kernel   the panel's row interchanges on every other column
//                         of D (LAPACK layout) and of X; a no-op for leaves
//                         whose panel pivoted on the diagonal
//     leaf_panel_solve    U12 = L11^{-1} A12 (in place, D and X columns; FP32: an
//                         item of the batched GEMM)
//     batched GEMM        A22 -= L21 U12 (D trailing block and X rows below)
//   then for each panel from the last: X[k] = U_kk^{-1} X[k];
//                                      X[0:k0] -= U[0:k0, k] X[k]
// so D ends as LAPACK's P L U factors, X as D^{-1} X.  The GEMMs are items of
// the batched GEMM engine (gemm_simt.cu), one launch per step for all leaves.
// FP64 solves use the triangles' inverses only where these are well-conditioned
// (ill_conditioned below), substitution elsewhere.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "common.cuh"
#include "leaf_blocked.cuh"
#include "warp_f64.cuh"

namespace hodlr {

namespace {

constexpr int kThreads = 256;

// 16-byte vector of T
template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
  using V = float4;
};
template <>
struct Vec16<double> {
  using V = double2;
};

// Register-resident panel LU in LAPACK's dgetf2 pivot order, with implicit row
// interchanges (rows stay in their threads, each tracking its current
// position), and the inverses of the diagonal block's triangles.
// Thread t owns panel rows t + threads q (q < RPT) in registers.
//
// What bounds it is one column's serial chain (search, publish, barrier,
// combine, eliminate), so that chain is kept short.  The columns go in
// sub-blocks of SB = 8: a column's elimination touches its own sub-block
// only, and the columns behind it are updated once per sub-block, the
// sub-block's pivot rows solved against each other first (one thread per
// column).  Every element still gets its updates in column order, each one
// fused multiply-add, so the factors are those of the column-by-column
// elimination bit for bit.  Per column: every warp finds its best candidate (largest |a|,
// lowest current position on ties) with one warp reduction and one ballot
// unless several rows tie in the reduced bits, each thread having formed its
// candidate's reciprocal beside the search, and the winning lane publishes
// its SB values; one barrier; every warp finds the best warp the same way
// and eliminates its rows.  Warps without live rows only keep the barriers
// and share the inverses.  A column takes 780 (FP64) / 630 (FP32) cycles with
// one live warp where the column-by-column form (every warp reducing full
// keys, whole rows published and updated per column) took ~2500; a 256-row
// panel with its inverses 27 us (FP64, 32 columns) and 41 us (FP32, 64) where
// it took 50 and 87 us.
constexpr int kRegThreads = 512;
// columns of a triangle's inverse per warp
template <int NB>
__host__ __device__ constexpr int panel_sub() {
  return NB < 32 ? NB : 32;
}

// |a| as an integer that orders like it, plus one; 0 for a NaN (never a
// candidate, as idamax skips it)
__device__ inline unsigned abs_key(float a) {
  const unsigned b = __float_as_uint(a) & 0x7fffffffu;
  return b <= 0x7f800000u ? b + 1u : 0u;
}
__device__ inline unsigned long long abs_key(double a) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(a) & 0x7fffffffffffffffull;
  return b <= 0x7ff0000000000000ull ? b + 1ull : 0ull;
}
__device__ inline unsigned key_high(unsigned k) { return k; }
__device__ inline unsigned key_high(unsigned long long k) { return (unsigned)(k >> 32); }
__device__ inline unsigned key_low(unsigned) { return 0u; }
__device__ inline unsigned key_low(unsigned long long k) { return (unsigned)k; }

template <typename T, int NB, int RPT>
__global__ void __launch_bounds__(kRegThreads, 1)
    leaf_panel_reg_kernel(const LeafFactorTask<T> *__restrict__ tasks, int k0, int panel,
                          int *info) {
  constexpr int NW = kRegThreads / 32;
  constexpr int SB = 8, NSB = NB / SB;
  constexpr int VW = 16 / sizeof(T);
  using V = typename Vec16<T>::V;
  __shared__ __align__(16) T wrow[2][NW][SB];  // a warp's candidate row, its sub-block
  __shared__ T wrcp[2][NW];                    // 1 / candidate
  __shared__ int4 wmeta[2][NW];                // its key (high, low), position, row
  __shared__ __align__(16) T Us[SB][NB];           // the pivot rows behind the sub-block
  __shared__ T Ls[SB][SB + 1];                     // their multipliers
  // the diagonal block's triangles, both as lower ones, column-major: U with
  // rows and columns reversed
  __shared__ __align__(16) T Lk[NB * NB], Uk[NB * NB];
  __shared__ T udr[NB];  // 1 / U's diagonal, reversed
  __shared__ int pv[NB];
  const LeafFactorTask<T> tk = tasks[blockIdx.x];
  const int n = tk.n;
  if (k0 >= n) return;
  const int kb = min(NB, n - k0);
  const int R = n - k0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nthr = blockDim.x, nw = nthr >> 5;
  const int nlive = min(nw, (R + 31) >> 5);        // warps with live rows
  T *D = tk.D;
  const long long ldd = tk.ldd;
  T a[RPT][NB];
  int pos[RPT];
  bool live[RPT], act[RPT];  // a row of the panel; one not yet pivotal
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    const int i = tid + q * nthr;
    live[q] = act[q] = i < R;
    pos[q] = i;
    // every load issued before any is used: rows beyond the leaf repeat its
    // last row, columns beyond the panel its last column
    const T *src = D + (k0 + min(i, R - 1)) + (long long)k0 * ldd;
    if (kb == NB) {
#pragma unroll
      for (int c = 0; c < NB; ++c) a[q][c] = src[(long long)c * ldd];
    } else {
#pragma unroll
      for (int c = 0; c < NB; ++c) a[q][c] = src[(long long)min(c, kb - 1) * ldd];
#pragma unroll
      for (int c = 0; c < NB; ++c)
        if (c >= kb) a[q][c] = T(0);
    }
  }
  const bool warp_live = warp < nlive;
  int info_local = 0;
  bool swaps = false;
  // Before sub-block h every row is rotated left by h SB, so the sub-block's
  // columns sit at register positions 0 .. SB - 1; positions SB ..
  // NB - h SB - 1 hold the later columns, the rest the finished ones.
#pragma unroll 1
  for (int h = 0; h < NSB; ++h) {
    const int j0 = h * SB;
    const int behind = NB - j0 - SB;  // columns behind the sub-block
    unsigned zero_piv = 0;            // columns without a pivot: no update (uniform)
#pragma unroll
    for (int jj = 0; jj < SB; ++jj) {
      const int j = j0 + jj;  // panel column
      if (j >= kb) break;
      const int slot = jj & 1;
      if (warp_live) {
        auto best = abs_key(a[0][jj]);
        if (!act[0]) best = 0;
        int bp = pos[0], bq = 0;
        T cand = a[0][jj];
#pragma unroll
        for (int q = 1; q < RPT; ++q) {
          auto k = abs_key(a[q][jj]);
          if (!act[q]) k = 0;
          if (k > best || (k == best && pos[q] < bp)) {
            best = k; bp = pos[q]; bq = q; cand = a[q][jj];
          }
        }
        const unsigned mx = __reduce_max_sync(0xffffffffu, key_high(best));
        const T rc = sizeof(T) == 4 ? T(__frcp_rn(float(cand))) : T(__drcp_rn(double(cand)));
        const unsigned win = __ballot_sync(0xffffffffu, key_high(best) == mx);
        int wl = __ffs(win) - 1;
        if (win & (win - 1)) wl = tied_lane(key_high(best), mx, key_low(best), bp);
        if (lane == wl) {
          wmeta[slot][warp] = make_int4((int)key_high(best), (int)key_low(best), bp,
                                        tid + bq * nthr);
          wrcp[slot][warp] = rc;
          V *dst = reinterpret_cast<V *>(wrow[slot][warp]);
#pragma unroll
          for (int cv = jj / VW; cv < SB / VW; ++cv) {
            V v;
            T *vp = reinterpret_cast<T *>(&v);
#pragma unroll
            for (int u = 0; u < VW; ++u) {
              vp[u] = a[0][cv * VW + u];
#pragma unroll
              for (int q = 1; q < RPT; ++q)
                if (q == bq) vp[u] = a[q][cv * VW + u];
            }
            dst[cv] = v;
          }
        }
      }
      __syncthreads();
      if (warp_live) {
        // the best warp (every warp, same result)
        const unsigned key = lane < nlive ? (unsigned)wmeta[slot][lane].x : 0u;
        const unsigned mx = __reduce_max_sync(0xffffffffu, key);
        const unsigned win = __ballot_sync(0xffffffffu, key == mx);
        int pw = __ffs(win) - 1;
        if (win & (win - 1)) {
          const int4 m = wmeta[slot][lane < nlive ? lane : 0];
          pw = tied_lane(key, mx, (unsigned)m.y, lane < nlive ? m.z : 0x7fffffff);
        }
        const int4 m = wmeta[slot][pw];
        const T rinv = wrcp[slot][pw];
        const V *prow = reinterpret_cast<const V *>(wrow[slot][pw]);
        T u[SB];
#pragma unroll
        for (int cv = jj / VW; cv < SB / VW; ++cv) {
          const V v = prow[cv];
          const T *vp = reinterpret_cast<const T *>(&v);
#pragma unroll
          for (int x = 0; x < VW; ++x) u[cv * VW + x] = vp[x];
        }
        // no candidate (FP64: its key's words are both 0): position j keeps its row
        const bool any = (m.x | (sizeof(T) == 8 ? m.y : 0)) != 0;
        const int p = any ? m.z : j, pc = any ? m.w : -1;
        if (tid == 0) pv[j] = p;
        swaps |= p != j;
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
          const bool me = tid + q * nthr == pc;
          if (!me && pos[q] == j) pos[q] = p;
          if (me) pos[q] = j;
          act[q] = act[q] && pos[q] != j;
        }
        if (any && u[jj] != T(0)) {
#pragma unroll
          for (int q = 0; q < RPT; ++q) {
            if (act[q]) {
              const T l = a[q][jj] * rinv;
              a[q][jj] = l;
#pragma unroll
              for (int c = jj + 1; c < SB; ++c) a[q][c] -= l * u[c];
            }
          }
        } else {
          zero_piv |= 1u << jj;
          if (info_local == 0) info_local = k0 + j + 1;
        }
      }
    }
    if (behind > 0 && j0 + SB < kb) {
      // the sub-block's pivot rows, un-updated behind it, and their multipliers
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        const int k = pos[q] - j0;
        if (live[q] && k >= 0 && k < SB) {
          V *dst = reinterpret_cast<V *>(Us[k]);
#pragma unroll
          for (int cv = SB / VW; cv < NB / VW; ++cv) {
            V v;
            T *vp = reinterpret_cast<T *>(&v);
#pragma unroll
            for (int x = 0; x < VW; ++x) vp[x] = a[q][cv * VW + x];
            dst[cv] = v;
          }
#pragma unroll
          for (int c = 0; c < SB; ++c) Ls[k][c] = zero_piv >> c & 1 ? T(0) : a[q][c];
        }
      }
      __syncthreads();
      if (tid < behind && warp_live) {
        T u[SB];
#pragma unroll
        for (int k = 0; k < SB; ++k) u[k] = Us[k][SB + tid];
#pragma unroll
        for (int k = 0; k < SB - 1; ++k) {
#pragma unroll
          for (int i = k + 1; i < SB; ++i) u[i] -= Ls[i][k] * u[k];
        }
#pragma unroll
        for (int k = 0; k < SB; ++k) Us[k][SB + tid] = u[k];
      }
      __syncthreads();
      if (warp_live) {
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
          if (live[q] && pos[q] >= j0 + SB) {
#pragma unroll
            for (int g = 1; g < NSB; ++g) {
              if (g * SB > behind) break;  // uniform: finished columns from here
#pragma unroll
              for (int k = 0; k < SB; ++k) {
                const T l = zero_piv >> k & 1 ? T(0) : a[q][k];
                const V *ur = reinterpret_cast<const V *>(&Us[k][g * SB]);
#pragma unroll
                for (int cv = 0; cv < SB / VW; ++cv) {
                  const V v = ur[cv];
                  const T *vp = reinterpret_cast<const T *>(&v);
                  T *ac = &a[q][g * SB + cv * VW];
                  if constexpr (sizeof(T) == 4) {
                    // the packed FP32 FMA, each half rounded as a - l u
                    const float2 nl = make_float2(-float(l), -float(l));
#pragma unroll
                    for (int x = 0; x < VW; x += 2) {
                      const float2 r = __ffma2_rn(nl, make_float2(vp[x], vp[x + 1]),
                                                  make_float2(ac[x], ac[x + 1]));
                      ac[x] = r.x;
                      ac[x + 1] = r.y;
                    }
                  } else {
#pragma unroll
                    for (int x = 0; x < VW; ++x) ac[x] -= l * vp[x];
                  }
                }
              }
            }
          } else if (live[q] && pos[q] >= j0) {  // this sub-block's pivot rows
            const V *ur = reinterpret_cast<const V *>(Us[pos[q] - j0]);
#pragma unroll
            for (int cv = SB / VW; cv < NB / VW; ++cv) {
              if (cv * VW >= SB + behind) break;  // uniform: finished columns from here
              const V v = ur[cv];
              const T *vp = reinterpret_cast<const T *>(&v);
#pragma unroll
              for (int x = 0; x < VW; ++x) a[q][cv * VW + x] = vp[x];
            }
          }
        }
      }
    }
    // rotate every row left by SB (after NSB rotations the order is restored)
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      T t[SB];
#pragma unroll
      for (int c = 0; c < SB; ++c) t[c] = a[q][c];
#pragma unroll
      for (int c = 0; c < NB - SB; ++c) a[q][c] = a[q][c + SB];
#pragma unroll
      for (int c = 0; c < SB; ++c) a[q][NB - SB + c] = t[c];
    }
  }
  // rows to their final positions; diagonal block rows to shared memory
  int pold[RPT];
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    pold[q] = live[q] ? tk.perm[k0 + tid + q * nthr] : 0;
    if (live[q]) {
      T *dst = D + (k0 + pos[q]) + (long long)k0 * ldd;
#pragma unroll
      for (int c = 0; c < NB; ++c)
        if (c < kb) dst[(long long)c * ldd] = a[q][c];
      if (pos[q] < kb) {
        const int r = pos[q];
#pragma unroll
        for (int c = 0; c < NB; ++c) {
          Lk[c * NB + r] = c < r ? a[q][c] : (c == r ? T(1) : T(0));
          Uk[(NB - 1 - c) * NB + NB - 1 - r] = c >= r ? a[q][c] : T(0);
        }
      }
    }
  }
  for (int r = kb + tid; r < NB; r += nthr) {
    for (int c = 0; c < NB; ++c) {
      Lk[c * NB + r] = c == r ? T(1) : T(0);
      Uk[(NB - 1 - c) * NB + NB - 1 - r] = c == r ? T(1) : T(0);
    }
  }
  __syncthreads();  // every thread has read its perm entry and written its rows
#pragma unroll
  for (int q = 0; q < RPT; ++q)
    if (live[q]) tk.perm[k0 + pos[q]] = pold[q];
  for (int j = tid; j < kb; j += nthr) tk.ipiv[k0 + j] = k0 + pv[j] + 1;
  for (int r = tid; r < NB; r += nthr) udr[r] = T(1) / Uk[r * NB + r];
  if (tid == 0) {
    tk.swapflag[panel] = swaps ? 1 : 0;
    if (info_local && info && info[tk.info_slot] == 0) info[tk.info_slot] = info_local;
  }
  __syncthreads();
  // Inverses of the diagonal block's triangles, every column by substitution: a
  // warp per 32 columns of a triangle, a lane per column, RB rows at a time in
  // registers; A's columns are read as broadcasts.  (With lanes as rows and x_k
  // passed by shuffles the shuffles took 9.5 k cycles per 32 x 32 FP64 pair and
  // 17.5 k per 64 x 64 FP32 pair; with all rows in registers the straight-line
  // code's instruction fetches took 5 us per FP64 panel.)  The columns are not put
  // together from the inverses of half blocks, -A22^{-1} (A21 A11^{-1}): that
  // squares the triangle's condition number in the residual of a solve.
  constexpr int CB = panel_sub<NB>(), NT = NB / CB, RB = 16;
  T *Lout = tk.Linv + (size_t)panel * NB * NB;
  T *Uout = tk.Uinv + (size_t)panel * NB * NB;
  for (int job = warp; job < 2 * NT; job += nw) {
    const bool upper = job >= NT;
    const int cb = job % NT * CB;  // the warp's columns cb, cb + 1, ..
    const int j = cb + lane % CB;  // this lane's
    T *A = upper ? Uk : Lk;
    T *out = upper ? Uout + (NB - RB) + (size_t)(NB - 1 - j) * NB : Lout + (size_t)j * NB;
#pragma unroll 1
    for (int o = 0; o < NB; o += RB) {
      T x[RB];
#pragma unroll
      for (int i = 0; i < RB; ++i) x[i] = o + i == j ? T(1) : T(0);
      // less A's part left of the diagonal times the rows above, which are kept
      // on and above A's diagonal (x_k of column j in A's row j, column k >= j)
#pragma unroll 4
      for (int k = cb; k < o; ++k) {
        const T xk = j <= k ? A[k * NB + j] : T(0);
#pragma unroll
        for (int cv = 0; cv < RB / VW; ++cv) {
          const V v = reinterpret_cast<const V *>(A + k * NB + o)[cv];
          const T *vp = reinterpret_cast<const T *>(&v);
#pragma unroll
          for (int u = 0; u < VW; ++u) x[cv * VW + u] -= vp[u] * xk;
        }
      }
      if (o + RB > cb) {
#pragma unroll
        for (int k = 0; k < RB; ++k) {
          __syncwarp();  // A's columns are read as needed (read ahead, they spill)
          if (upper) x[k] *= udr[o + k];
#pragma unroll
          for (int cv = (k + 1) / VW; cv < RB / VW; ++cv) {
            const V v = reinterpret_cast<const V *>(A + (o + k) * NB + o)[cv];
            const T *vp = reinterpret_cast<const T *>(&v);
#pragma unroll
            for (int u = 0; u < VW; ++u)
              if (cv * VW + u > k) x[cv * VW + u] -= vp[u] * x[k];
          }
        }
      }
      __syncwarp();
      if (lane < CB) {
#pragma unroll
        for (int cv = 0; cv < RB / VW; ++cv) {
          V w;
          T *wp = reinterpret_cast<T *>(&w);
#pragma unroll
          for (int u = 0; u < VW; ++u) wp[u] = x[upper ? RB - 1 - cv * VW - u : cv * VW + u];
          reinterpret_cast<V *>(out + (upper ? -o : o))[cv] = w;
        }
#pragma unroll
        for (int k = 0; k < RB; ++k)
          if (j <= o + k) A[(o + k) * NB + j] = x[k];
      }
      __syncwarp();
    }
  }
}

// Row interchanges of panels [p0, p0 + np) (in order) on the D columns
// [a0, a1) and [b0, b1) (clamped to the leaf) and, with with_x, on the
// leaf's X columns.  grid (column block, leaf); thread = column.
template <typename T>
__global__ void __launch_bounds__(kThreads)
    leaf_laswp_kernel(const LeafFactorTask<T> *__restrict__ tasks, int p0, int np, int nb,
                      int a0, int a1, int b0, int b1, int with_x) {
  const LeafFactorTask<T> tk = tasks[blockIdx.y];
  const int n = tk.n;
  if (p0 * nb >= n) return;
  bool any = false;
  for (int q = p0; q < p0 + np && q * nb < n; ++q) any |= tk.swapflag[q] != 0;
  if (!any) return;
  const int na = max(0, min(a1, n) - a0);
  const int nbr = max(0, min(b1, n) - b0);
  const int c = blockIdx.x * kThreads + threadIdx.x;
  T *col;
  if (c < na) {
    col = tk.D + (long long)(a0 + c) * tk.ldd;
  } else if (c < na + nbr) {
    col = tk.D + (long long)(b0 + c - na) * tk.ldd;
  } else if (with_x && c < na + nbr + tk.ncols) {
    col = tk.X + (long long)(c - na - nbr) * tk.ldx;
  } else {
    return;
  }
  for (int q = p0; q < p0 + np; ++q) {
    const int k0 = q * nb;
    if (k0 >= n) break;
    if (tk.swapflag[q] == 0) continue;
    const int kb = min(nb, n - k0);
    for (int j = 0; j < kb; ++j) {
      const int p = tk.ipiv[k0 + j] - 1;
      if (p != k0 + j) {
        const T t = col[k0 + j];
        col[k0 + j] = col[p];
        col[p] = t;
      }
    }
  }
}

template <typename T>
__global__ void leaf_init_kernel(const LeafFactorTask<T> *__restrict__ tasks, int *info) {
  const LeafFactorTask<T> tk = tasks[blockIdx.x];
  for (int i = threadIdx.x; i < tk.n; i += blockDim.x) tk.perm[i] = i;
  if (threadIdx.x == 0 && info) info[tk.info_slot] = 0;
}

// ---- apply: X <- U^{-1} L^{-1} P X with the stored blocked factors.
//
// One CTA per (column chunk of MC right-hand sides, leaf).  The rows of P X
// live in registers for the whole solve; panel by panel (forward with L, then
// backward with U) the owners of the panel's rows publish them, they are
// multiplied by the diagonal block's explicit inverse, and every row still to
// come subtracts its row of the block column, streamed from global memory
// once, coalesced along the rows and loaded ahead of the barriers it does not
// depend on.  Two barriers per panel.
//
// FP32: rows in threads, two per thread, so that a broadcast read of the
// panel's values feeds two rows (with the chunk of X in shared memory and one
// row per thread the kernel was bound by those reads).  FP64: 16-row tiles in
// warps on the DMMA pipe.
//   FP32, 512 leaves of 512 rows, 16 columns: 407 -> 320 us;
//   FP32, 128 leaves of 512 rows, 8 columns: 172 -> 78 us;
//   FP64, 256 leaves of 512 rows, 16 columns: 587 -> 251 us.

// Stage the diagonal-block inverse Ainv (kb x kb, column-major, ld nb) into
// shared memory `As` (ld kb + 1) with asynchronous copies (one commit group).
__device__ inline void stage_inverse(const float *__restrict__ Ainv, int nb, int kb, float *As) {
  const int lds = kb + 1;
  for (int e = threadIdx.x; e < kb * kb; e += blockDim.x) {
    const int i = e % kb, k = e / kb;
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(As + i + k * lds));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(Ainv + i + (size_t)k * nb));
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

constexpr int kApplyNB = 64;  // largest panel

template <int MC>
constexpr int apply32_smem() {
  return (2 * kApplyNB * (kApplyNB + 1) + 2 * kApplyNB * MC) * (int)sizeof(float);
}

// THREADS >= half the rows of the largest leaf, a multiple of 4 kApplyNB
template <int MC, int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS)
    leaf_apply32_kernel(const LeafFactorTask<float> *__restrict__ tasks, int nb) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int CH = MC == 32 ? 8 : 16;            // k-values of a row loaded ahead
  constexpr int CG = THREADS / kApplyNB, CW = MC / CG;  // column groups of the diagonal product
  static_assert(CW * CG == MC, "whole column groups");
  const LeafFactorTask<float> tk = tasks[blockIdx.y];
  const int n = tk.n;
  const int c0 = blockIdx.x * MC;
  if (c0 >= tk.ncols || n <= 0) return;
  const int mc = min(MC, tk.ncols - c0);
  const int tid = threadIdx.x;
  float *As0 = reinterpret_cast<float *>(smem_raw);  // two staged inverses
  const int as_stride = kApplyNB * (kApplyNB + 1);
  float *ys = As0 + 2 * as_stride;                   // the panel's rows, published
  float *yo = ys + kApplyNB * MC;                    // ... times the inverse
  float *X = tk.X + (long long)c0 * tk.ldx;
  const long long ldx = tk.ldx, ldd = tk.ldd;
  const int np = (n + nb - 1) / nb;
  // step st < np: forward panel st with Linv; else backward panel 2 np - 1 - st
  // with Uinv
  auto panel_of = [&](int st) { return st < np ? st : 2 * np - 1 - st; };
  auto stage = [&](int st) {
    const int p = panel_of(st), kb = min(nb, n - p * nb);
    stage_inverse((st < np ? tk.Linv : tk.Uinv) + (size_t)p * nb * nb, nb, kb,
                  As0 + (st & 1) * as_stride);
  };
  stage(0);
  float acc[2][MC];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const float *x = X + tk.perm[min(tid + q * THREADS, n - 1)];
#pragma unroll
    for (int j = 0; j < MC; ++j) acc[q][j] = x[(long long)min(j, mc - 1) * ldx];
  }
  for (int st = 0; st < 2 * np; ++st) {
    const int p = panel_of(st), k0 = p * nb, kb = min(nb, n - k0);
    const bool fwd = st < np;
    bool act[2];
    const float *ap[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int i = tid + q * THREADS;
      act[q] = fwd ? i >= k0 + kb && i < n : i < k0;
      ap[q] = tk.D + min(i, n - 1) + (long long)k0 * ldd;
    }
    // the first k-values of this thread's rows, before the barriers
    float a[2][CH];
    auto load = [&](int q, int kk) {  // the next CH columns (the last one repeated)
      const float *x = ap[q] + (long long)kk * ldd;
      if (kk + CH <= kb) {
#pragma unroll
        for (int u = 0; u < CH; ++u, x += ldd) a[q][u] = *x;
      } else {
#pragma unroll
        for (int u = 0; u < CH; ++u) {
          a[q][u] = *x;
          if (kk + u + 1 < kb) x += ldd;
        }
      }
    };
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (act[q]) load(q, 0);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int i = tid + q * THREADS - k0;
      if (i >= 0 && i < kb) {
#pragma unroll
        for (int j = 0; j < MC; j += 4)
          *reinterpret_cast<float4 *>(ys + i * MC + j) =
              make_float4(acc[q][j], acc[q][j + 1], acc[q][j + 2], acc[q][j + 3]);
      }
    }
    if (st + 1 < 2 * np) {
      stage(st + 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    {
      const int i = tid % kApplyNB, cg = tid / kApplyNB * CW;
      const float *As = As0 + (st & 1) * as_stride;
      float o[CW];
#pragma unroll
      for (int c = 0; c < CW; ++c) o[c] = 0.f;
      if (i < kb) {
#pragma unroll 8
        for (int k = 0; k < kb; ++k) {
          const float m = As[i + k * (kb + 1)];
#pragma unroll
          for (int c = 0; c < CW; ++c) o[c] += m * ys[k * MC + cg + c];
        }
      }
      if (i < nb) {
#pragma unroll
        for (int c = 0; c < CW; ++c) yo[i * MC + cg + c] = o[c];  // 0 beyond kb
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int i = tid + q * THREADS - k0;
      if (i >= 0 && i < kb) {
#pragma unroll
        for (int j = 0; j < MC; ++j) acc[q][j] = yo[i * MC + j];
      }
    }
    // rows still to come: acc -= D[row][panel] y
    auto update = [&](auto Q0, auto Q1) {
      for (int kk = 0; kk < kb; kk += CH) {
        float c[2][CH];
#pragma unroll
        for (int q = Q0; q < Q1; ++q)
#pragma unroll
          for (int u = 0; u < CH; ++u) c[q][u] = a[q][u];
        if (kk + CH < kb) {
#pragma unroll
          for (int q = Q0; q < Q1; ++q) load(q, kk + CH);
        }
        const float *y = yo + kk * MC;
#pragma unroll
        for (int u = 0; u < CH; ++u)
#pragma unroll
          for (int j = 0; j < MC; j += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(y + u * MC + j);
#pragma unroll
            for (int q = Q0; q < Q1; ++q) {
              acc[q][j] -= c[q][u] * v.x;
              acc[q][j + 1] -= c[q][u] * v.y;
              acc[q][j + 2] -= c[q][u] * v.z;
              acc[q][j + 3] -= c[q][u] * v.w;
            }
          }
      }
    };
    using std::integral_constant;
    if (act[0] && act[1]) update(integral_constant<int, 0>{}, integral_constant<int, 2>{});
    else if (act[0]) update(integral_constant<int, 0>{}, integral_constant<int, 1>{});
    else if (act[1]) update(integral_constant<int, 1>{}, integral_constant<int, 2>{});
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int i = tid + q * THREADS;
    if (i < n) {
#pragma unroll
      for (int j = 0; j < MC; ++j)
        if (j < mc) X[i + (long long)j * ldx] = acc[q][j];
    }
  }
}

// NT blocks of 8 columns; TPW 16-row tiles per warp (16 warps: 256 TPW rows)
template <int NT, int TPW>
__global__ void __launch_bounds__(512, 1)
    leaf_apply64_kernel(const LeafFactorTask<double> *__restrict__ tasks, int nb) {
  constexpr int MC = 8 * NT, XS = MC + 4, NBM = 32;  // row stride: conflict-free fragments
  __shared__ __align__(16) double ys[NBM * XS], yo[NBM * XS];
  const LeafFactorTask<double> tk = tasks[blockIdx.y];
  const int n = tk.n;
  const int c0 = blockIdx.x * MC;
  if (c0 >= tk.ncols || n <= 0) return;
  const int mc = min(MC, tk.ncols - c0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  double *X = tk.X + (long long)c0 * tk.ldx;
  const long long ldx = tk.ldx, ldd = tk.ldd;
  const int np = (n + nb - 1) / nb;
  // tile j of this warp: rows 16 (warp + 16 j) .. + 15
  double acc[TPW][NT][4];
#pragma unroll
  for (int j = 0; j < TPW; ++j)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const double *x = X + tk.perm[min(16 * (warp + 16 * j) + g + (v >> 1) * 8, n - 1)];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
        acc[j][nt][v] = x[(long long)min(8 * nt + 2 * t + (v & 1), mc - 1) * ldx];
    }
  for (int st = 0; st < 2 * np; ++st) {
    const bool fwd = st < np;
    const int p = fwd ? st : 2 * np - 1 - st, k0 = p * nb, kb = min(nb, n - k0);
    const int t0 = k0 / 16, t1 = t0 + nb / 16;  // the panel's tiles
    auto active = [&](int j) {
      const int tile = warp + 16 * j;
      return fwd ? tile >= t1 && 16 * tile < n : tile < t0;
    };
    // fragments of 16 of the panel's columns in the tile's rows; columns beyond
    // the leaf meet zero rows of y
    double a[4][2];
    auto load = [&](int j, int h) {
      const int r = 16 * (warp + 16 * j) + g;
      const double *p0 = tk.D + min(r, n - 1), *p1 = tk.D + min(r + 8, n - 1);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const long long o = (long long)min(k0 + 16 * h + 4 * k + t, n - 1) * ldd;
        a[k][0] = p0[o];
        a[k][1] = p1[o];
      }
    };
    // the diagonal product's tile of this warp, then the first block tile
    const int dm = warp % 2, dn = warp / 2;  // 16-row and 8-column block
    const bool diag = dm < nb / 16 && dn < NT;
    double d[NBM / 4][2];
    if (diag) {
      const double *inv = (fwd ? tk.Linv : tk.Uinv) + (size_t)p * nb * nb + 16 * dm + g;
#pragma unroll
      for (int k = 0; k < NBM / 4; ++k) {
        if (4 * k >= nb) break;
        d[k][0] = inv[(4 * k + t) * nb];
        d[k][1] = inv[(4 * k + t) * nb + 8];
      }
    }
    int first = TPW;
#pragma unroll
    for (int j = TPW - 1; j >= 0; --j)
      if (active(j)) first = j;
    if (first < TPW) load(first, 0);
#pragma unroll
    for (int j = 0; j < TPW; ++j) {
      const int tile = warp + 16 * j;
      if (tile >= t0 && tile < t1) {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int r = 16 * (tile - t0) + g + (v >> 1) * 8;
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
            ys[r * XS + 8 * nt + 2 * t + (v & 1)] = r < kb ? acc[j][nt][v] : 0.0;
        }
      }
    }
    __syncthreads();
    if (diag) {
      double c[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int k = 0; k < NBM / 4; ++k) {
        if (4 * k >= nb) break;
        dmma(c, d[k][0], d[k][1], ys[(4 * k + t) * XS + 8 * dn + g]);
      }
#pragma unroll
      for (int v = 0; v < 4; ++v)  // kept negated: the updates subtract
        yo[(16 * dm + g + (v >> 1) * 8) * XS + 8 * dn + 2 * t + (v & 1)] = -c[v];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < TPW; ++j) {
      const int tile = warp + 16 * j;
      if (tile >= t0 && tile < t1) {
#pragma unroll
        for (int v = 0; v < 4; ++v)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
            acc[j][nt][v] =
                -yo[(16 * (tile - t0) + g + (v >> 1) * 8) * XS + 8 * nt + 2 * t + (v & 1)];
      }
      if (active(j)) {
        for (int h = 0; h < nb / 16; ++h) {
          double c[4][2];
#pragma unroll
          for (int k = 0; k < 4; ++k) { c[k][0] = a[k][0]; c[k][1] = a[k][1]; }
          if (16 * (h + 1) < nb) load(j, h + 1);
          else if (j + 1 < TPW && active(j + 1)) load(j + 1, 0);
          const double *y = yo + (16 * h + t) * XS + g;
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
              dmma(acc[j][nt], c[k][0], c[k][1], y[4 * k * XS + 8 * nt]);
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < TPW; ++j)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int r = 16 * (warp + 16 * j) + g + (v >> 1) * 8;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int c = 8 * nt + 2 * t + (v & 1);
        if (r < n && c < mc) X[r + (long long)c * ldx] = acc[j][nt][v];
      }
    }
}

// Whether an FP64 triangle T with the explicit inverse Y is solved by
// substitution instead: max|T| max|Y| of about 64 or more, from the high words
// of the two (their binary exponents; NaN and infinity count as largest).  A
// product with Y leaves a residual of up to |T| |Y| rounding errors where
// substitution leaves one.  On smooth-kernel leaves (Gaussian kernels, 100 to
// 1000 rows) products alone left backward errors of up to 2e12 u, with this
// bound they stay within four times substitution's 0.2 to 0.4 u; Gaussian
// random leaves of 512 rows reach 20, so ordinary leaves keep the products.
__device__ inline unsigned high_abs(double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; }
__device__ inline bool ill_conditioned(unsigned tri, unsigned inv) {
  const unsigned et = tri >> 20, ei = inv >> 20;
  return et == 2047 || ei == 2047 || et + ei >= 2 * 1023 + 6;
}
// The same over a CTA: every thread's high words go in, the caller's barrier, and
// every thread has the answer.  slots: one per warp.
__device__ inline void publish_largest(uint2 *slots, unsigned tri, unsigned inv) {
  tri = __reduce_max_sync(0xffffffffu, tri);
  inv = __reduce_max_sync(0xffffffffu, inv);
  if ((threadIdx.x & 31) == 0) slots[threadIdx.x >> 5] = make_uint2(tri, inv);
}
template <int WARPS>
__device__ inline bool ill_conditioned_cta(const uint2 *slots) {
  unsigned tri = 0, inv = 0;
#pragma unroll
  for (int w = 0; w < WARPS; ++w) {
    tri = max(tri, slots[w].x);
    inv = max(inv, slots[w].y);
  }
  return ill_conditioned(tri, inv);
}

// ---- inverses of the outer diagonal blocks (two-level factorization).
//
// Outer block J (rows / columns j0 .. j0 + obe of a leaf) starts as its
// panels' own inverses on the diagonal and L's (U's) blocks beside them, and
// diagonal blocks are merged pairwise, in place:
//   lower: X21 = -X22 (L21 X11),    upper: Y12 = -Y11 (U12 Y22),
// with blocks of NB, 2 NB, ... columns: two products and two barriers per
// doubling.  One CTA per leaf, block and triangle; the matrix (column-major,
// padded), and the inner product live in shared memory, FP64 products on the
// DMMA pipe, tiles skipping the triangular operand's zeros.  Built panel by
// panel, with P (P - 1) (P + 1) / 3 products one after another and a staged
// block for each, the five launches of an FP64 solve (N = 262144, 512 leaves
// of 512 rows, blocks of four panels) took 1.64 ms; this takes 0.8 ms.  FP32
// blocks are two panels, two products either way (0.47 -> 0.45 ms).
constexpr int kInvThreads = 256;

// Which operand of a product is triangular: the lower or the upper one of A or
// B.  A tile of C skips the k for which that operand's rows (columns) of the
// tile are zero.
enum Tri { kLowerA, kUpperA, kLowerB, kUpperB };
template <Tri TRI>
__device__ inline void tri_range(int m0, int m1, int n0, int n1, int K, int &k0, int &k1) {
  k0 = TRI == kUpperA ? m0 : TRI == kLowerB ? n0 : 0;
  k1 = TRI == kLowerA ? m1 : TRI == kUpperB ? n1 : K;
}

// C (M x N) = alpha A B (A M x K, B K x N), all column-major in shared memory,
// M and N multiples of 16 R
template <int R, Tri TRI>
__device__ inline void block_mm(int M, int N, int K, const float *A, int lda, const float *B,
                                int ldb, float *C, int ldc, float alpha) {
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  for (int m0 = 0; m0 < M; m0 += 16 * R)
    for (int n0 = 0; n0 < N; n0 += 16 * R) {
      int k0, k1;
      tri_range<TRI>(m0, m0 + 16 * R, n0, n0 + 16 * R, K, k0, k1);
      float c[R][R];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int q = 0; q < R; ++q) c[r][q] = 0.f;
#pragma unroll 8
      for (int k = k0; k < k1; ++k) {
        float a[R], b[R];
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = A[(m0 + ty * R + r) + k * lda];
#pragma unroll
        for (int q = 0; q < R; ++q) b[q] = B[k + (n0 + tx * R + q) * ldb];
        // packed two-wide FMAs, each half rounded as c + a b
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int q = 0; q < R; q += 2) {
            const float2 v = __ffma2_rn(make_float2(a[r], a[r]), make_float2(b[q], b[q + 1]),
                                        make_float2(c[r][q], c[r][q + 1]));
            c[r][q] = v.x;
            c[r][q + 1] = v.y;
          }
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int q = 0; q < R; ++q)
          C[(m0 + ty * R + r) + (n0 + tx * R + q) * ldc] = alpha * c[r][q];
    }
}
template <Tri TRI>
__device__ inline void block_product(int M, int N, int K, const float *A, int lda, const float *B,
                                     int ldb, float *C, int ldc, float alpha) {
  block_mm<2, TRI>(M, N, K, A, lda, B, ldb, C, ldc, alpha);
}
// FP64: warps take 16 x 8 tiles in turn
template <Tri TRI>
__device__ inline void block_product(int M, int N, int K, const double *A, int lda,
                                     const double *B, int ldb, double *C, int ldc, double alpha) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int tm = M / 16, tn = N / 8;
  for (int tile = threadIdx.x >> 5; tile < tm * tn; tile += kInvThreads / 32) {
    const int m = (tile % tm) * 16 + g, n = (tile / tm) * 8;
    int k0, k1;
    tri_range<TRI>(m - g, m - g + 16, n, n + 8, K, k0, k1);
    double c[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
    for (int k = k0 + t; k < k1; k += 4) {
      const double a0 = A[m + k * lda], a1 = A[m + 8 + k * lda], b = B[k + (n + g) * ldb];
      dmma(c, a0, a1, b);
    }
#pragma unroll
    for (int v = 0; v < 4; ++v)
      C[m + (v >> 1) * 8 + (n + 2 * t + (v & 1)) * ldc] = alpha * c[v];
  }
}

// column strides: FP64 4 modulo 16 (conflict-free DMMA fragments), FP32 odd
template <typename T>
__host__ __device__ constexpr int inv_ld(int n) { return n + (sizeof(T) == 8 ? 4 : 1); }
// largest inner product: a block of half the next power of two's size
template <typename T>
__host__ __device__ inline size_t inv_words(int ob, int nb) {
  int h = nb;
  while (2 * h < ob) h *= 2;
  return (size_t)inv_ld<T>(ob) * ob + (size_t)inv_ld<T>(h) * h;
}

// grid (leaf, block J0, J0 + 1, ...)
template <typename T, int NB>
__global__ void __launch_bounds__(kInvThreads)
    leaf_block_inverse_kernel(const LeafFactorTask<T> *__restrict__ tasks, int ob, int J0, int slots,
                              int upper) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const LeafFactorTask<T> tk = tasks[blockIdx.x];
  const int n = tk.n;
  const int J = J0 + (int)blockIdx.y;
  const int j0 = J * ob;
  if (j0 >= n) return;
  const int obe = min(ob, n - j0);
  const int pbase = j0 / NB, live = (obe + NB - 1) / NB * NB;  // whole panels
  const int ld = inv_ld<T>(ob);
  T *X = reinterpret_cast<T *>(smem_raw);
  T *Tt = X + (size_t)ld * ob;
  const int tid = threadIdx.x;
  const T *inv = upper ? tk.Uinv : tk.Linv;
  const int lane = tid & 31, warp = tid >> 5;
  // a warp per column, every load unconditional (an address inside the leaf's
  // own data), so that a thread's loads overlap
  const T *safe = tk.D + j0 + (long long)j0 * tk.ldd;
  constexpr int kAhead = sizeof(T) == 8 ? 2 : 4;  // columns whose loads overlap
  unsigned largest = 0, largest_t = 0;  // FP64: high words of max|inverse|, max|triangle|
  constexpr int kTri = 128 * NB / kInvThreads;
  T tri[kTri];
  if constexpr (sizeof(T) == 8) {
    // U's part inside the panels, whose inverses stand in for it below: loads
    // under way during the main ones
    if (upper) {
#pragma unroll
      for (int q = 0; q < kTri; ++q) {
        const int e = min(tid + q * kInvThreads, ob * NB - 1);
        const int c = min(e / NB, obe - 1), i = min(c / NB * NB + e % NB, c);
        tri[q] = tk.D[j0 + i + (long long)(j0 + c) * tk.ldd];
      }
    }
  }
#pragma unroll kAhead
  for (int c = warp; c < ob; c += kInvThreads / 32) {
    const int pc = c / NB;
    const T *dcol = tk.D + j0 + (long long)(j0 + c) * tk.ldd;
    const T *icol = inv + (size_t)(pbase + pc) * NB * NB + (c - pc * NB) * NB - pc * NB;
    T v[4];
    bool in[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = lane + 32 * q, pi = i / NB;
      const bool diag = pi == pc;
      in[q] = diag ? i < live : (upper ? pi < pc : pi > pc) && i < obe && c < obe;
      v[q] = *(in[q] ? (diag ? icol : dcol) + i : safe);
    }
    if constexpr (sizeof(T) == 8) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const bool diag = (lane + 32 * q) / NB == pc;
        largest_t = max(largest_t, in[q] && !diag ? high_abs(v[q]) : 0u);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (lane + 32 * q < ob) X[lane + 32 * q + c * ld] = in[q] ? v[q] : T(0);
  }
  if constexpr (sizeof(T) == 8) {
    if (upper) {
#pragma unroll
      for (int q = 0; q < kTri; ++q) largest_t = max(largest_t, high_abs(tri[q]));
    }
  }
  __syncthreads();
  for (int b = NB; b < ob; b *= 2) {
    for (int o = 0; o + b < live; o += 2 * b) {
      const int h = min(b, ob - o - b);  // the second block's size
      T *X11 = X + o + o * ld, *X22 = X + (o + b) + (o + b) * ld;
      T *off = upper ? X + o + (o + b) * ld : X + (o + b) + o * ld;
      const int lt = inv_ld<T>(upper ? b : h);
      if (upper) block_product<kUpperB>(b, h, h, off, ld, X22, ld, Tt, lt, T(1));
      else block_product<kLowerB>(h, b, b, off, ld, X11, ld, Tt, lt, T(1));
      __syncthreads();
      if (upper) block_product<kUpperA>(b, h, b, X11, ld, Tt, lt, off, ld, T(-1));
      else block_product<kLowerA>(h, b, h, X22, ld, Tt, lt, off, ld, T(-1));
      __syncthreads();
    }
  }
  // zero outside the leaf's part of the block (rows / columns >= obe)
  T *dst = tk.Binv + (size_t)(J % slots) * ob * ob;
  for (int c = warp; c < ob; c += kInvThreads / 32)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = lane + 32 * q;
      const T v = i < obe && c < obe ? X[i + c * ld] : T(0);
      if (i < ob) dst[i + c * ob] = v;
      if constexpr (sizeof(T) == 8) largest = max(largest, high_abs(v));
    }
  if constexpr (sizeof(T) == 8) {
    __shared__ uint2 slots[kInvThreads / 32];
    publish_largest(slots, upper ? largest_t : 1023u << 20, largest);  // max|L| = 1
    __syncthreads();
    const bool ill = ill_conditioned_cta<kInvThreads / 32>(slots);
    if (tid == 0) tk.ill_b[2 * J + upper] = ill;
    if (ill)  // leaf_block_solve_kernel solves, the product with this copies
      for (int e = tid; e < ob * ob; e += kInvThreads)
        dst[e] = e % ob == e / ob && e / ob < obe ? T(1) : T(0);
  }
}

// ---- FP64 solves with a diagonal triangle.

constexpr int kSolveThreads = 128;

// x <- T^{-1} x by substitution, a thread per column (x: this thread's, or
// null), T (order x order, unit-lower or upper) column-major in global memory
// and staged as 32 x 32 blocks in Ts.  All kSolveThreads threads call it.  Only
// ill-conditioned triangles come here: 32 rows at a time in registers.
template <bool UPPER>
__device__ void substitute_columns(const double *T, long long ldt, int order, double *x,
                                   double *Ts) {
  const int nblk = (order + 31) / 32;
  auto stage = [&](int bi, int bk) {  // the identity beyond the triangle's order
    __syncthreads();  // the previous block's reads are done
    for (int e = threadIdx.x; e < 32 * 32; e += kSolveThreads) {
      const int i = 32 * bi + e % 32, k = 32 * bk + e / 32;
      Ts[e] = i < order && k < order ? T[i + k * ldt] : i == k ? 1.0 : 0.0;
    }
    __syncthreads();
  };
  for (int s = 0; s < nblk; ++s) {
    const int bi = UPPER ? nblk - 1 - s : s;
    double v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = x && 32 * bi + i < order ? x[32 * bi + i] : 0.0;
    for (int q = 0; q < s; ++q) {
      const int bk = UPPER ? nblk - 1 - q : q;
      stage(bi, bk);
      for (int k = 0; k < 32; ++k) {
        const double xk = x && 32 * bk + k < order ? x[32 * bk + k] : 0.0;
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] -= Ts[i + 32 * k] * xk;
      }
    }
    stage(bi, bi);
#pragma unroll
    for (int kk = 0; kk < 32; ++kk) {
      const int k = UPPER ? 31 - kk : kk;
      if (UPPER) v[k] /= Ts[k + 32 * k];
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (UPPER ? i < k : i > k) v[i] -= Ts[i + 32 * k] * v[k];
    }
    if (x) {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (32 * bi + i < order) x[32 * bi + i] = v[i];
    }
  }
}

// The panel's rows of a chunk of 64 columns times the inverse of the panel's
// triangle, in place: one rank-NB DMMA product of operands that are all read
// before the first store.  grid (column chunk, leaf).  Against items of the tile
// GEMM, which cannot substitute: 5.5 instead of 5.7 us a launch for one leaf of
// 512 rows and 592 columns, 125 instead of 157 us in all inside the outer blocks
// of 512 such leaves.  Every CTA decides from the inverse it loads anyway (marks
// left by the panel kernel took that 1.5 us each).
constexpr int kSolveCols = 64;

template <int NB, bool UPPER>
__global__ void __launch_bounds__(kSolveThreads)
    leaf_panel_solve_kernel(const LeafFactorTask<double> *__restrict__ tasks, int panel, int b0,
                            int b1, int with_x) {
  constexpr int LD = NB + 4;                  // conflict-free fragments
  constexpr int WM = NB / 16, WN = 4 / WM;    // warps over rows, columns
  constexpr int NT = kSolveCols / WN / 8;     // column blocks of a warp
  constexpr int PER = kSolveCols / 4 * NB / 32;  // values of a thread
  __shared__ __align__(16) double xs[kSolveCols * LD > 32 * 32 ? kSolveCols * LD : 32 * 32];
  const LeafFactorTask<double> tk = tasks[blockIdx.y];
  const int n = tk.n, k0 = panel * NB;
  if (k0 >= n) return;
  const int kb = min(NB, n - k0);
  const int nd = max(0, min(b1, n) - b0), total = nd + (with_x ? tk.ncols : 0);
  const int c0 = blockIdx.x * kSolveCols;
  if (c0 >= total) return;
  // column c of this CTA (the last one repeated), at the panel's first row
  auto column = [&](int c) {
    const int q = min(c0 + c, total - 1);
    return q < nd ? tk.D + k0 + (long long)(b0 + q) * tk.ldd
                  : tk.X + k0 + (long long)(q - nd) * tk.ldx;
  };
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wm = warp % WM * 16, wn = warp / WM * (8 * NT);
  const double *inv = (UPPER ? tk.Uinv : tk.Linv) + (size_t)panel * NB * NB + wm + g;
  double a[NB / 4][2], v[PER], tri[NB * NB / kSolveThreads];
  const int row = lane % NB, c1 = warp * (kSolveCols / 4) + lane / NB;
#pragma unroll
  for (int u = 0; u < PER; ++u) v[u] = column(c1 + u * (32 / NB))[min(row, kb - 1)];
#pragma unroll
  for (int k = 0; k < NB / 4; ++k) {
    a[k][0] = inv[(4 * k + t) * NB];
    a[k][1] = inv[(4 * k + t) * NB + 8];
  }
  unsigned largest = 0, largest_t = 1023u << 20;  // max|L| = 1
  if (UPPER) {
#pragma unroll
    for (int q = 0; q < NB * NB / kSolveThreads; ++q) {
      const int e = tid + q * kSolveThreads, j = min(e / NB, kb - 1), i = min(e % NB, j);
      tri[q] = tk.D[k0 + i + (long long)(k0 + j) * tk.ldd];
    }
    largest_t = 0;
#pragma unroll
    for (int q = 0; q < NB * NB / kSolveThreads; ++q) largest_t = max(largest_t, high_abs(tri[q]));
  }
#pragma unroll
  for (int q = 0; q < PER; ++q) xs[(c1 + q * (32 / NB)) * LD + row] = row < kb ? v[q] : 0.0;
#pragma unroll
  for (int k = 0; k < NB / 4; ++k) largest = max(largest, max(high_abs(a[k][0]), high_abs(a[k][1])));
  __shared__ uint2 slots[kSolveThreads / 32];
  publish_largest(slots, largest_t, largest);
  __syncthreads();
  double c[NT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int q = 0; q < 4; ++q) c[nt][q] = 0.0;
#pragma unroll
  for (int k = 0; k < NB / 4; ++k)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
      dmma(c[nt], a[k][0], a[k][1], xs[(wn + 8 * nt + g) * LD + 4 * k + t]);
  if (ill_conditioned_cta<kSolveThreads / 32>(slots)) {
    double *x = tid < kSolveCols && c0 + tid < total ? column(tid) : nullptr;
    substitute_columns<UPPER>(tk.D + k0 + k0 * tk.ldd, tk.ldd, kb, x, xs);
    return;
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int col = wn + 8 * nt + 2 * t + u;
      if (c0 + col >= total) continue;
      double *d = column(col) + wm + g;
      if (wm + g < kb) d[0] = c[nt][u];
      if (wm + g + 8 < kb) d[8] = c[nt][2 + u];
    }
}

// The CTAs of a leaf (grid (CTAs, leaf)) take its chunks of kSolveThreads
// columns in turn.
template <bool UPPER>
__global__ void __launch_bounds__(kSolveThreads)
    leaf_block_solve_kernel(const LeafFactorTask<double> *__restrict__ tasks, int ob, int J) {
  __shared__ __align__(16) double Ts[32 * 32];
  const LeafFactorTask<double> &tk = tasks[blockIdx.y];
  const int n = tk.n, j0 = J * ob;
  if (j0 >= n || !tk.ill_b[2 * J + UPPER]) return;
  const int obe = min(ob, n - j0);
  const int nd = UPPER ? 0 : n - j0 - obe, total = nd + tk.ncols;
  for (int c0 = blockIdx.x * kSolveThreads; c0 < total; c0 += gridDim.x * kSolveThreads) {
    const int c = c0 + (int)threadIdx.x;
    double *x = nullptr;
    if (c < nd) x = tk.D + j0 + (long long)(j0 + obe + c) * tk.ldd;
    else if (c < total) x = tk.X + j0 + (long long)(c - nd) * tk.ldx;
    substitute_columns<UPPER>(tk.D + j0 + j0 * tk.ldd, tk.ldd, obe, x, Ts);
  }
}

}  // namespace

template <typename T>
void launch_leaf_init(const LeafFactorTask<T> *tasks, int count, int *info, cudaStream_t s) {
  if (count <= 0) return;
  leaf_init_kernel<T><<<count, kThreads, 0, s>>>(tasks, info);
  HODLR_LAUNCH_CHECK();
}

template <typename T, int NB, int RPT>
void launch_leaf_panel_reg(const LeafFactorTask<T> *tasks, int count, int rows, int k0,
                           int panel, int *info, cudaStream_t s) {
  // one thread per RPT live rows of the largest leaf's panel, and a warp for
  // each of the inverses' column blocks
  constexpr int blocks = 2 * NB / panel_sub<NB>();
  const int threads = std::min(kRegThreads, std::max(32 * blocks, cdiv(cdiv(rows, RPT), 32) * 32));
  leaf_panel_reg_kernel<T, NB, RPT><<<count, threads, 0, s>>>(tasks, k0, panel, info);
  HODLR_LAUNCH_CHECK();
}

template <typename T>
void launch_leaf_panel(const LeafFactorTask<T> *tasks, int count, int max_n, int nb, int k0,
                       int panel, int *info, cudaStream_t s) {
  if (count <= 0) return;
  // register-resident panel: rows <= 512 RPT with 64 values per thread
  const int rows = max_n - k0;
  if constexpr (sizeof(T) == 4) {
    if (nb == 64 && rows <= kRegThreads)
      return launch_leaf_panel_reg<T, 64, 1>(tasks, count, rows, k0, panel, info, s);
    if (nb == 32 && rows <= 2 * kRegThreads)
      return launch_leaf_panel_reg<T, 32, 2>(tasks, count, rows, k0, panel, info, s);
  } else {
    if (nb == 32 && rows <= kRegThreads)
      return launch_leaf_panel_reg<T, 32, 1>(tasks, count, rows, k0, panel, info, s);
    if (nb == 16 && rows <= 2 * kRegThreads)
      return launch_leaf_panel_reg<T, 16, 2>(tasks, count, rows, k0, panel, info, s);
  }
  throw CudaError{cudaErrorInvalidValue};  // no such panel: leaves have at most 1024 rows
}

template <typename T>
void launch_leaf_laswp(const LeafFactorTask<T> *tasks, int count, int max_cols, int nb, int p0,
                       int np, int a0, int a1, int b0, int b1, bool with_x, cudaStream_t s) {
  if (count <= 0 || max_cols <= 0 || np <= 0) return;
  dim3 grid(cdiv(max_cols, kThreads), count);
  leaf_laswp_kernel<T><<<grid, kThreads, 0, s>>>(tasks, p0, np, nb, a0, a1, b0, b1,
                                                 with_x ? 1 : 0);
  HODLR_LAUNCH_CHECK();
}

template <typename T>
void launch_leaf_apply(const LeafFactorTask<T> *tasks, int count, int max_n, int max_cols, int nb,
                       cudaStream_t s) {
  if (count <= 0 || max_cols <= 0 || max_n <= 0) return;
  if (max_n > 1024 || nb > (sizeof(T) == 8 ? 32 : kApplyNB) || nb % 16)
    throw CudaError{cudaErrorInvalidValue};
  auto go = [&](auto kern, int mc, int threads, size_t smem) {
    raise_smem_limit(reinterpret_cast<const void *>(kern), smem);
    kern<<<dim3(cdiv(max_cols, mc), count), threads, smem, s>>>(tasks, nb);
  };
  const bool tall = max_n > 512;
  if constexpr (sizeof(T) == 4) {
    auto pick = [&](auto mcv) {
      constexpr int MC = decltype(mcv)::value;
      if (tall) go(leaf_apply32_kernel<MC, 512>, MC, 512, apply32_smem<MC>());
      else go(leaf_apply32_kernel<MC, 256>, MC, 256, apply32_smem<MC>());
    };
    if (max_cols <= 8) pick(std::integral_constant<int, 8>{});
    else if (max_cols <= 16) pick(std::integral_constant<int, 16>{});
    else pick(std::integral_constant<int, 32>{});
  } else {
    // 32 columns of a leaf above 512 rows do not fit the registers
    if (max_cols <= 8) tall ? go(leaf_apply64_kernel<1, 4>, 8, 512, 0) : go(leaf_apply64_kernel<1, 2>, 8, 512, 0);
    else if (tall) go(leaf_apply64_kernel<2, 4>, 16, 512, 0);
    else if (max_cols <= 16) go(leaf_apply64_kernel<2, 2>, 16, 512, 0);
    else go(leaf_apply64_kernel<4, 2>, 32, 512, 0);
  }
  HODLR_LAUNCH_CHECK();
}

template <typename T>
void launch_leaf_block_inverse(const LeafFactorTask<T> *tasks, int count, int nb, int ob, int J0,
                               int blocks, int slots, bool upper, cudaStream_t s) {
  if (count <= 0 || blocks <= 0) return;
  if (ob > 128 || ob % nb || blocks > slots) throw CudaError{cudaErrorInvalidValue};
  dim3 grid(count, blocks);
  const size_t smem = inv_words<T>(ob, nb) * sizeof(T);
  auto go = [&](auto kern) {
    raise_smem_limit(reinterpret_cast<const void *>(kern), smem);
    kern<<<grid, kInvThreads, smem, s>>>(tasks, ob, J0, slots, upper ? 1 : 0);
  };
  if (nb == 64) go(leaf_block_inverse_kernel<T, 64>);
  else if (nb == 32) go(leaf_block_inverse_kernel<T, 32>);
  else if (nb == 16) go(leaf_block_inverse_kernel<T, 16>);
  else throw CudaError{cudaErrorInvalidValue};
  HODLR_LAUNCH_CHECK();
}

void launch_leaf_panel_solve(const LeafFactorTask<double> *tasks, int count, int max_cols, int nb,
                             int panel, int b0, int b1, bool with_x, bool upper, cudaStream_t s) {
  if (count <= 0 || max_cols <= 0) return;
  const dim3 grid(cdiv(max_cols, kSolveCols), count);
  auto go = [&](auto kern) {
    kern<<<grid, kSolveThreads, 0, s>>>(tasks, panel, b0, b1, with_x ? 1 : 0);
  };
  if (nb == 32) upper ? go(leaf_panel_solve_kernel<32, true>) : go(leaf_panel_solve_kernel<32, false>);
  else if (nb == 16) upper ? go(leaf_panel_solve_kernel<16, true>) : go(leaf_panel_solve_kernel<16, false>);
  else throw CudaError{cudaErrorInvalidValue};
  HODLR_LAUNCH_CHECK();
}

void launch_leaf_block_solve(const LeafFactorTask<double> *tasks, int count, int max_cols, int ob,
                             int J, bool upper, cudaStream_t s) {
  if (count <= 0 || max_cols <= 0) return;
  // few CTAs per leaf where there are many leaves: nearly always they have nothing to do
  const dim3 grid(std::min(cdiv(max_cols, kSolveThreads), std::max(1, 1024 / count)), count);
  if (upper) leaf_block_solve_kernel<true><<<grid, kSolveThreads, 0, s>>>(tasks, ob, J);
  else leaf_block_solve_kernel<false><<<grid, kSolveThreads, 0, s>>>(tasks, ob, J);
  HODLR_LAUNCH_CHECK();
}

template void launch_leaf_block_inverse<double>(const LeafFactorTask<double> *, int, int, int, int,
                                                int, int, bool, cudaStream_t);
template void launch_leaf_block_inverse<float>(const LeafFactorTask<float> *, int, int, int, int,
                                               int, int, bool, cudaStream_t);

template void launch_leaf_apply<double>(const LeafFactorTask<double> *, int, int, int, int,
                                        cudaStream_t);
template void launch_leaf_apply<float>(const LeafFactorTask<float> *, int, int, int, int,
                                       cudaStream_t);
template void launch_leaf_init<double>(const LeafFactorTask<double> *, int, int *, cudaStream_t);
template void launch_leaf_init<float>(const LeafFactorTask<float> *, int, int *, cudaStream_t);
template void launch_leaf_panel<double>(const LeafFactorTask<double> *, int, int, int, int, int,
                                        int *, cudaStream_t);
template void launch_leaf_panel<float>(const LeafFactorTask<float> *, int, int, int, int, int,
                                       int *, cudaStream_t);
template void launch_leaf_laswp<double>(const LeafFactorTask<double> *, int, int, int, int, int,
                                        int, int, int, int, bool, cudaStream_t);
template void launch_leaf_laswp<float>(const LeafFactorTask<float> *, int, int, int, int, int,
                                       int, int, int, int, bool, cudaStream_t);

}  // namespace hodlr
