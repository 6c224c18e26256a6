// node.cu -- capacitance (node) factorization, FP64, batched over a tree level.
//
// GPU restatement of LUSolveTask::cpu_task (src/solver/solver_tasks.cc:
// 139-305) and of the 2r x 2r Schur system of serial_leaf_solve's internal
// branch (solver_tasks.cc:483-535).  For a node with children b0, b1 and the
// summed reduce results W0 = [V0Td0 | V0Tu0], W1 = [V1Td1 | V1Tu1] the
// reference computes, per column block of the d part,
//
//   T    = V1Td1 - V1Tu1 V0Td0          (dgemm at 236)
//   eta0 = S^{-1} T,  S = I - V1Tu1 V0Tu0   (dgemm at 261, dgesv at 281)
//   eta1 = V0Td0 - V0Tu0 eta0           (dgemm at 299)
//
// which is linear in [V0Td0; V1Td1]:
//
//   [eta0; eta1] = M [V0Td0; V1Td1],
//   M = [[ -S^{-1} V1Tu1,            S^{-1}         ],
//        [ I + V0Tu0 S^{-1} V1Tu1,  -V0Tu0 S^{-1}   ]]
//
// (form 1, the 2r x 2r system [[V0Tu0, I], [I, V1Tu1]] of the leaf-internal
// branch: M is that matrix's inverse).  node_factor_kernel forms M once per
// node, one CTA per node: S on the DMMA pipe, S^{-1} by blocked Gauss-Jordan
// elimination with partial pivoting (pivot = largest |a|, lowest row on ties,
// as LAPACK's idamax), the three products on the DMMA pipe.  The solver
// applies M to every column block as one batched GEMM per level (the same
// engine as the reduce and broadcast), for the fused pass and for every later
// solve with the same factors.  INFO > 0 reports an exactly zero pivot
// (singular S), as dgesv.
#include <algorithm>

#include "common.cuh"
#include "node.cuh"
#include "warp_f64.cuh"

namespace hodlr {

namespace {

constexpr int kNodeThreads = 512;
constexpr int kNodeWarps = kNodeThreads / 32;
constexpr int PB = 8;         // columns per panel of the elimination
constexpr int kXld = PB + 4;  // row stride of the panel's multipliers (conflict-free fragments)
constexpr size_t kSmemLimit = 227 * 1024 - 4096;  // a CTA's shared memory less the static arrays

__host__ __device__ constexpr int up(int x, int m) { return (x + m - 1) / m * m; }
// Row stride (doubles) of the eliminated matrix: whole panels, and 8 modulo
// 16, so that two rows' 64-byte column pairs share no bank.
__host__ __device__ constexpr int node_lda(int s) { return up(s + 8, 16) - 8; }
// Column stride of a staged V^T u block with `rows` rows: whole fragment
// rows plus a shift that spreads the columns over the banks.
template <typename TW>
__host__ __device__ constexpr int node_ldw(int rows) { return up(rows, 16) + (sizeof(TW) == 4 ? 8 : 4); }

// Shared-memory layout of a launch (bytes from the start).
struct NodeSmem {
  int lda, ldb;
  size_t x, b, ints, w0, w1, total;
};
template <typename TW>
__host__ __device__ inline NodeSmem node_smem(int max_s, int max_r, bool stage) {
  NodeSmem m{};
  const int s16 = up(max_s, 16);
  m.lda = node_lda(max_s);
  m.ldb = m.lda + 12;  // 4 modulo 16
  m.x = sizeof(double) * s16 * m.lda;
  m.b = m.x + sizeof(double) * s16 * kXld;
  m.ints = m.b + sizeof(double) * PB * m.ldb;
  m.w0 = m.ints + sizeof(int) * up(3 * s16 + PB, 4);
  m.w1 = m.w0 + (stage ? sizeof(TW) * node_ldw<TW>(max_r) * up(max_r, 8) : 0);
  m.total = m.w1 + (stage ? sizeof(TW) * node_ldw<TW>(max_r) * up(max_r, 8) : 0);
  return m;
}

// out(i, j, sum_k a(i, k) b(k, j)) for i < rows, j < cols on the FP64 tensor
// pipe, every warp taking 16 x 8 tiles in turn.  a and b are read up to the
// next multiples of 16 rows, 8 columns and 4 k; a(i, k) b(k, j) must be 0 for
// k >= K.
template <typename FA, typename FB, typename FO>
__device__ inline void node_product(int rows, int cols, int K, FA a, FB b, FO out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int tm = (rows + 15) / 16, tn = (cols + 7) / 8;
  for (int tile = warp; tile < tm * tn; tile += kNodeWarps) {
    const int m0 = (tile % tm) * 16 + g, n0 = (tile / tm) * 8;
    double c[4] = {0.0, 0.0, 0.0, 0.0};
    int k = t;
    for (; k - t + 16 <= K; k += 16) {
      double a0[4], a1[4], bv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        a0[u] = a(m0, k + 4 * u);
        a1[u] = a(m0 + 8, k + 4 * u);
        bv[u] = b(k + 4 * u, n0 + g);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) dmma(c, a0[u], a1[u], bv[u]);
    }
    for (; k - t < K; k += 4) dmma(c, a(m0, k), a(m0 + 8, k), b(k, n0 + g));
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int i = m0 + (v >> 1) * 8, j = n0 + 2 * t + (v & 1);
      if (i < rows && j < cols) out(i, j, c[v]);
    }
  }
}

// Inverse of the s x s matrix A (row-major, row stride lda, zero up to the
// next multiples of 16 rows and 8 columns) by Gauss-Jordan elimination with
// partial pivoting and implicit row interchanges, PB = 8 columns at a time:
//   1. the panel's columns are eliminated on their own, one row per thread in
//      registers (every row, also those already pivotal), with one barrier of
//      the row warps per column: search by one warp reduction and one ballot
//      unless keys tie, the winner publishes its 8 values and its reciprocal.
//      What is left are every row's multipliers, X; those of a pivot row before
//      its own column go to Lp;
//   2. the panel's pivot rows, each as it is at its own column: as before the
//      panel, in the panel's own columns (now the inverse's) the unit rows, less
//      Lp times the ones before them;
//   3. every column: A = (pivot rows and own columns: 0, others: A) + X (those
//      rows), one rank-8 DMMA product.
// So every element goes through the steps of the column-by-column elimination.
// (With X the panel's part of the inverse and the pivot rows as they were before
// the panel the products multiply with explicit inverses of 8 x 8 pivot blocks:
// on smooth-kernel systems of order 16 to 144 the residual of the solution grew
// up to 1e8-fold.)
// What bounds it is the serial chain of a column (~700 cycles: search,
// publish, barrier, combine), no longer the re-reading of the matrix: column
// by column it took 1.9 k cycles with the matrix in registers (s <= 64) and
// ~3.5 k in shared memory.
// On return A[at[i]][src[j]] is the inverse's entry (i, j).  Returns 0 or the
// first zero pivot (1-based), uniform over the CTA.
__device__ inline int gauss_jordan(double *A, int lda, int s, double *X, double *Bb, int ldb,
                                   int *at, int *src, int *mark, int *prow) {
  __shared__ __align__(16) double wrow[2][kNodeWarps][PB];
  __shared__ double wrcp[2][kNodeWarps];
  __shared__ int4 wmeta[2][kNodeWarps];
  __shared__ double Lp[PB][PB];
  __shared__ int s_info;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int nrw = (s + 31) >> 5;  // warps with rows
  const int tm = (s + 15) / 16, tn = (s + 7) / 8;
  const bool rowok = tid < s;
  int pos = tid;        // current position of this row (LAPACK interchange order)
  bool act = rowok;     // not yet pivotal
  if (tid == 0) s_info = 0;
  for (int k0 = 0; k0 < s; k0 += PB) {
    const int nb = min(PB, s - k0);
    if (warp < nrw) {
      double a[PB];
      const double2 *ar = reinterpret_cast<const double2 *>(A + min(tid, s - 1) * lda + k0);
#pragma unroll
      for (int c = 0; c < PB / 2; ++c) {
        const double2 v = ar[c];
        a[2 * c] = v.x;
        a[2 * c + 1] = v.y;
      }
      bool bad = false;
#pragma unroll
      for (int jj = 0; jj < PB; ++jj) {
        if (jj >= nb || bad) break;
        const int k = k0 + jj, slot = jj & 1;
        const unsigned long long bits =
            (unsigned long long)__double_as_longlong(a[jj]) & 0x7fffffffffffffffull;
        // NaN is never a candidate (as idamax, which skips it)
        const unsigned long long key = act && bits <= 0x7ff0000000000000ull ? bits + 1ull : 0ull;
        const unsigned hi = (unsigned)(key >> 32);
        const unsigned mx = __reduce_max_sync(0xffffffffu, hi);
        const double rc = 1.0 / a[jj];
        const unsigned win = __ballot_sync(0xffffffffu, hi == mx);
        int wl = __ffs(win) - 1;
        if (win & (win - 1)) wl = tied_lane(hi, mx, (unsigned)key, pos);
        if (lane == wl) {
          wmeta[slot][warp] = make_int4((int)hi, (int)(unsigned)key, pos, tid);
          wrcp[slot][warp] = rc;
          double2 *d = reinterpret_cast<double2 *>(wrow[slot][warp]);
#pragma unroll
          for (int c = jj / 2; c < PB / 2; ++c) d[c] = make_double2(a[2 * c], a[2 * c + 1]);
        }
        asm volatile("bar.sync 1, %0;\n" ::"r"(nrw * 32) : "memory");
        const unsigned wkey = lane < nrw ? (unsigned)wmeta[slot][lane].x : 0u;
        const unsigned wmx = __reduce_max_sync(0xffffffffu, wkey);
        const unsigned wwin = __ballot_sync(0xffffffffu, wkey == wmx);
        int pw = __ffs(wwin) - 1;
        if (wwin & (wwin - 1)) {
          const int4 m = wmeta[slot][lane < nrw ? lane : 0];
          pw = tied_lane(wkey, wmx, (unsigned)m.y, lane < nrw ? m.z : 0x7fffffff);
        }
        const int4 m = wmeta[slot][pw];
        const double rinv = wrcp[slot][pw];
        double u[PB];
        const double2 *ur = reinterpret_cast<const double2 *>(wrow[slot][pw]);
#pragma unroll
        for (int c = jj / 2; c < PB / 2; ++c) {
          const double2 v = ur[c];
          u[2 * c] = v.x;
          u[2 * c + 1] = v.y;
        }
        if ((m.x | m.y) == 0 || u[jj] == 0.0) {  // exactly singular (or a NaN column)
          if (tid == 0) s_info = k + 1;
          bad = true;
        } else if (tid == m.w) {
          pos = k;
          act = false;
          mark[tid] = k0;
          prow[jj] = tid;
          a[jj] = rinv;
#pragma unroll
          for (int c = jj + 1; c < PB; ++c) a[c] *= rinv;
        } else {
          if (pos == k) pos = m.z;
          a[jj] = -(a[jj] * rinv);
#pragma unroll
          for (int c = jj + 1; c < PB; ++c) a[c] += a[jj] * u[c];
        }
      }
      if (rowok) {
        const int own = act ? 0 : max(pos - k0, 0);  // the column here whose pivot this row is
        if (own > 0) {
#pragma unroll
          for (int c = 0; c < PB; ++c) Lp[own][c] = a[c];
        }
        double2 *xr = reinterpret_cast<double2 *>(X + tid * kXld);
#pragma unroll
        for (int c = 0; c < PB; ++c)
          if (c < own || c >= nb) a[c] = 0.0;
#pragma unroll
        for (int c = 0; c < PB / 2; ++c) xr[c] = make_double2(a[2 * c], a[2 * c + 1]);
      }
    }
    __syncthreads();
    if (s_info != 0) return s_info;  // uniform
    if (const int c = tid; c < tn * 8) {
      static_assert(kMaxNodeS <= kNodeThreads, "a thread per column");
      double u[PB];
#pragma unroll
      for (int jj = 0; jj < PB; ++jj) u[jj] = jj < nb ? A[prow[jj] * lda + c] : 0.0;
      if (c >= k0 && c < k0 + PB) {
#pragma unroll
        for (int jj = 0; jj < PB; ++jj) u[jj] = c == k0 + jj ? 1.0 : 0.0;
      }
#pragma unroll
      for (int jj = 0; jj < PB; ++jj) {
        Bb[jj * ldb + c] = u[jj];
#pragma unroll
        for (int k = jj + 1; k < PB; ++k)
          if (k < nb) u[k] += Lp[k][jj] * u[jj];
      }
    }
    __syncthreads();
    for (int tile = warp; tile < tm * tn; tile += kNodeWarps) {
      const int mt = tile % tm, nt = tile / tm;
      const bool own = nt == k0 / PB;
      const int ra = mt * 16 + g, rb = ra + 8;
      double2 *p0 = reinterpret_cast<double2 *>(A + ra * lda + nt * 8 + 2 * t);
      double2 *p1 = reinterpret_cast<double2 *>(A + rb * lda + nt * 8 + 2 * t);
      const double2 v0 = *p0, v1 = *p1;
      const bool z0 = own || mark[ra] == k0, z1 = own || mark[rb] == k0;  // pivot rows here
      double c[4] = {z0 ? 0.0 : v0.x, z0 ? 0.0 : v0.y, z1 ? 0.0 : v1.x, z1 ? 0.0 : v1.y};
      const double *x0 = X + ra * kXld + t, *x1 = X + rb * kXld + t;
      const double *bp = Bb + t * ldb + nt * 8 + g;
      dmma(c, x0[0], x1[0], bp[0]);
      dmma(c, x0[4], x1[4], bp[4 * ldb]);
      *p0 = make_double2(c[0], c[1]);
      *p1 = make_double2(c[2], c[3]);
    }
    __syncthreads();
  }
  // row interchanges of the elimination are column interchanges of the inverse
  if (rowok) {
    at[pos] = tid;
    src[tid] = pos;
  }
  __syncthreads();
  return 0;
}

template <typename TW, typename TE, bool STAGE>
__global__ void __launch_bounds__(kNodeThreads, 2)
    node_factor_kernel(const NodeTask<TW, TE> *tasks, int form, int max_s, int max_r, int *info) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const NodeTask<TW, TE> tk = tasks[blockIdx.x];
  const int tid = threadIdx.x;
  const int r0 = tk.r0, r1 = tk.r1, s2 = r0 + r1;
  const int s = form == 0 ? r0 : s2, s16 = up(s, 16);
  const NodeSmem sm = node_smem<TW>(max_s, max_r, STAGE);
  const int lda = sm.lda;
  double *A = reinterpret_cast<double *>(smem_raw);  // s x s, row-major
  double *X = reinterpret_cast<double *>(smem_raw + sm.x);
  double *Bb = reinterpret_cast<double *>(smem_raw + sm.b);
  int *at = reinterpret_cast<int *>(smem_raw + sm.ints);  // s16 each; prow: PB
  int *src = at + s16, *mark = src + s16, *prow = mark + s16;
  TW *W0s = reinterpret_cast<TW *>(smem_raw + sm.w0), *W1s = reinterpret_cast<TW *>(smem_raw + sm.w1);
  const TW *W0u = tk.W0u, *W1u = tk.W1u;
  const long long l0 = tk.ldw0u, l1 = tk.ldw1u;
  const int ld0 = node_ldw<TW>(r1), ld1 = node_ldw<TW>(r0);

  for (int e = tid; e < s16 * lda; e += kNodeThreads) A[e] = 0.0;
  for (int e = tid; e < s16 * kXld; e += kNodeThreads) X[e] = 0.0;
  for (int e = tid; e < s16; e += kNodeThreads) { at[e] = src[e] = 0; mark[e] = -1; }
  if constexpr (STAGE) {
    if (form == 0) {
      // V0Tu0 and V1Tu1 in their own precision (FP32 values convert exactly
      // at each operand load), zero outside
      auto stage = [&](TW *dst, int ld, const TW *W, long long ldw, int rows, int cols) {
        for (int e = tid; e < ld * up(cols, 8); e += kNodeThreads) {
          const int i = e % ld, j = e / ld;
          dst[e] = i < rows && j < cols ? W[i + (long long)j * ldw] : TW(0);
        }
      };
      stage(W0s, ld0, W0u, l0, r1, r0);
      stage(W1s, ld1, W1u, l1, r0, r1);
    }
  }
  __syncthreads();
  // the blocks' entries, 0 outside
  auto w0 = [&](int i, int j) -> double {
    if constexpr (STAGE) return double(W0s[i + j * ld0]);
    else return i < r1 && j < r0 ? double(W0u[i + j * l0]) : 0.0;
  };
  auto w1 = [&](int i, int j) -> double {
    if constexpr (STAGE) return double(W1s[i + j * ld1]);
    else return i < r0 && j < r1 ? double(W1u[i + j * l1]) : 0.0;
  };
  if (form == 0) {
    // S = I - V1Tu1 V0Tu0 (the dgemm at solver_tasks.cc:261)
    node_product(r0, r0, r1, w1, w0, [&](int i, int j, double v) {
      A[i * lda + j] = (i == j ? 1.0 : 0.0) - v;
    });
  } else {
    for (int e = tid; e < s * s; e += kNodeThreads) {
      const int i = e % s, c = e / s;
      double v = (i == (r1 + c) % s) ? 1.0 : 0.0;
      if (i < r1 && c < r0) v = double(W0u[i + (long long)c * l0]);
      else if (i >= r1 && c >= r0) v = double(W1u[(i - r1) + (long long)(c - r0) * l1]);
      A[i * lda + c] = v;
    }
  }
  __syncthreads();
  const int bad = gauss_jordan(A, lda, s, X, Bb, sm.ldb, at, src, mark, prow);
  if (tid == 0 && info) info[tk.info_slot] = bad;
  if (bad) return;  // singular: no solve matrix
  const long long ldm = s2;
  TE *M = tk.M;
  const int cs = form == 0 ? r1 : 0;  // S^{-1}'s (or, form 1, the inverse's) first column of M
  for (int e = tid; e < s * s; e += kNodeThreads) {
    const int i = e % s, j = e / s;
    M[i + (long long)(cs + j) * ldm] = TE(A[at[i] * lda + src[j]]);
  }
  if (form == 1) return;
  auto inv = [&](int i, int j) -> double { return A[at[i] * lda + src[j]]; };
  double *F = tk.F;
  // F = -V0Tu0 S^{-1} (r1 x r0): M's lower right block and FP64 work copy
  node_product(r1, r0, r0, w0, inv, [&](int i, int j, double v) {
    F[i + (long long)j * r1] = -v;
    M[(r0 + i) + (long long)(r1 + j) * ldm] = TE(-v);
  });
  // -S^{-1} V1Tu1 (r0 x r1): M's upper left block
  node_product(r0, r1, r0, inv, w1, [&](int i, int j, double v) { M[i + (long long)j * ldm] = TE(-v); });
  __syncthreads();  // F (global) visible to the whole CTA
  // I + V0Tu0 S^{-1} V1Tu1 = I - F V1Tu1 (r1 x r1): M's lower left block
  node_product(
      r1, r1, r0, [&](int i, int k) { return F[min(i, r1 - 1) + (long long)min(k, r0 - 1) * r1]; },
      w1, [&](int i, int j, double v) {
        M[(r0 + i) + (long long)j * ldm] = TE((i == j ? 1.0 : 0.0) - v);
      });
}

}  // namespace

template <typename TW, typename TE>
void launch_node_factor(const NodeTask<TW, TE> *tasks, int count, int max_s, int max_r, int form,
                        int *info, cudaStream_t s) {
  if (count <= 0) return;
  auto go = [&](auto kern, size_t smem) {
    raise_smem_limit(reinterpret_cast<const void *>(kern), smem);
    // the largest shared-memory carveout: two CTAs of up to ~110 KB per SM
    HODLR_CUDA_TRY(cudaFuncSetAttribute(reinterpret_cast<const void *>(kern),
                                        cudaFuncAttributePreferredSharedMemoryCarveout,
                                        cudaSharedmemCarveoutMaxShared));
    kern<<<count, kNodeThreads, smem, s>>>(tasks, form, max_s, max_r, info);
  };
  // V0Tu0 and V1Tu1 in shared memory where they fit beside the matrix (FP32 up to
  // r = 104, FP64 up to r = 88), also where that leaves one CTA per SM (FP64 above
  // r = 56); beyond, the products read them from L2.  All levels of 131072 rows,
  // leaves of 512, staged / not: FP64 r = 30 225 / 232 us, 56 434 / 449, 64 509 / 560,
  // 88 924 / 1021; mixed r = 64 504 / 572, 80 749 / 899, 104 1212 / 1458.
  const size_t staged = node_smem<TW>(max_s, max_r, true).total;
  if (form == 0 && staged <= kSmemLimit) go(node_factor_kernel<TW, TE, true>, staged);
  else go(node_factor_kernel<TW, TE, false>, node_smem<TW>(max_s, max_r, false).total);
  HODLR_LAUNCH_CHECK();
}

template void launch_node_factor<double, double>(const NodeTask<double, double> *, int, int,
                                                 int, int, int *, cudaStream_t);
template void launch_node_factor<float, float>(const NodeTask<float, float> *, int, int, int,
                                               int, int *, cudaStream_t);

}  // namespace hodlr
