// skinny_units.cuh -- CTA-level building blocks of the skinny GEMM items
// (at most 32 columns: the refinement sweeps' reduce, node apply and
// broadcast), shared by the one-launch-per-step kernels of gemm_skinny.cu and
// the persistent level-walk kernel of sweep.cu.  Every unit is executed by all
// threads of a CTA together (it synchronizes the CTA) and returns early only
// CTA-uniformly.
#pragma once
#include <type_traits>

#include "common.cuh"

namespace hodlr {
namespace sk {

constexpr int kSkStages = 3;

__device__ inline void cpa(void *dst, const void *src, int bytes, bool ok) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  const int n = ok ? bytes : 0;
  if (bytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n));
  else if (bytes == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(n));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(n));
}
__device__ inline void cpa_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ inline void cpa_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// The K tiles of an item, flattened over its segments (zero-length ones skipped).
template <typename T>
struct TileIter {
  const GemmSeg<T> *segs;
  int s, s_end, k0;
  GemmSeg<T> sg;
  bool valid;
  __device__ void init(const GemmSeg<T> *sp, int b, int c) {
    segs = sp;
    s = b;
    s_end = b + c;
    k0 = 0;
    settle();
  }
  __device__ void settle() {
    valid = false;
    for (; s < s_end; ++s) {
      sg = segs[s];
      if (sg.K > 0) { valid = true; return; }
    }
  }
  __device__ void next(int kt) {
    k0 += kt;
    if (k0 < sg.K) return;
    k0 = 0;
    ++s;
    settle();
  }
};

// Global loads of the units.  CG = false: the read-only path (__ldg), for
// one-step kernels whose inputs are never written by the same launch.
// CG = true: L2-only loads (__ldcg), for the persistent level-walk kernel,
// whose later steps read what other CTAs wrote in earlier steps of the same
// launch (an L1 or read-only-cache copy of an earlier step's value would be
// stale).
template <bool CG, typename T>
__device__ inline T ldg_unit(const T *p) {
  if constexpr (CG) return __ldcg(p);
  else return __ldg(p);
}

// ---------------------------------------------------------------- NN (rows)
constexpr int kRowThreads = 128;
constexpr int kNnSlab = 128;  // k-values of B in shared memory

// The k-values [k0, k0 + kNnSlab) of B (K x N) as Bs[k][NC], zero beyond K and
// N.  All threads of the CTA; the caller synchronizes.
template <int NC, bool CG>
__device__ inline void load_b_slab(float *Bs, const GemmSeg<float> &sg, int N, int k0) {
  constexpr int KS = kNnSlab, PER = NC < 16 ? NC : 16;
  static_assert(KS == kRowThreads, "a thread per k-value");
  const int k = threadIdx.x;
  const bool in = k0 + k < sg.K;
  const float *p = sg.B + k0 + (in ? k : 0);
#pragma unroll
  for (int n0 = 0; n0 < NC; n0 += PER) {
    float v[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) v[u] = ldg_unit<CG>(p + (long long)min(n0 + u, N - 1) * sg.ldb);
#pragma unroll
    for (int u = 0; u < PER; u += 4) {
      float w[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) w[x] = in && n0 + u + x < N ? v[u + x] : 0.f;
      *reinterpret_cast<float4 *>(Bs + k * NC + n0 + u) = make_float4(w[0], w[1], w[2], w[3]);
    }
  }
}

// FP32 C (M x N <= NC) = beta Cin + alpha sum_s A_s B_s, one row per thread,
// for short items (the node products, M = 2r): A straight from global memory,
// the next 16 k-values of a row loading while the current ones are used.
// One CTA (kRowThreads threads) computes rows [rb kRowThreads, ...) of item
// `item`; Bs holds kNnSlab NC floats.  CTA-uniform.  An item of at most
// kRowThreads rows may be in place (C also its B): its one unit has read all
// of B before it writes.
template <int NC, bool CG = false>
__device__ inline void nn_rows_unit(const GemmItem<float, float> *__restrict__ items,
                                    const GemmSeg<float> *__restrict__ segs, float alpha,
                                    float beta, int item, int rb, float *Bs) {
  constexpr int CH = NC == 32 ? 8 : 16, KS = kNnSlab;
  const GemmItem<float, float> it = items[item];
  const int row0 = rb * kRowThreads;
  if (row0 >= it.M) return;
  const int N = it.N;
  const int row = min(row0 + (int)threadIdx.x, it.M - 1);  // (beyond: not stored)
  float acc[NC];
#pragma unroll
  for (int n = 0; n < NC; ++n) acc[n] = 0.f;
  for (int sidx = it.seg_begin; sidx < it.seg_begin + it.seg_count; ++sidx) {
    const GemmSeg<float> sg = segs[sidx];
    const int K = sg.K;
    if (K <= 0) continue;
    float a[CH];
    auto load = [&](int kk) {  // (the last k-value repeated)
#pragma unroll
      for (int u = 0; u < CH; ++u)
        a[u] = ldg_unit<CG>(sg.A + row + (long long)min(kk + u, K - 1) * sg.lda);
    };
    load(0);
    for (int k0 = 0; k0 < K; k0 += KS) {
      const int ks = min(KS, K - k0);
      __syncthreads();  // the previous slab's reads are done
      load_b_slab<NC, CG>(Bs, sg, N, k0);
      __syncthreads();
      for (int kk = 0; kk < ks; kk += CH) {
        float c[CH];
#pragma unroll
        for (int u = 0; u < CH; ++u) c[u] = a[u];
        if (k0 + kk + CH < K) load(k0 + kk + CH);
#pragma unroll
        for (int u = 0; u < CH; ++u)
#pragma unroll
          for (int n = 0; n < NC; n += 4) {
            const float4 b = *reinterpret_cast<const float4 *>(Bs + (kk + u) * NC + n);
            acc[n] += c[u] * b.x;
            acc[n + 1] += c[u] * b.y;
            acc[n + 2] += c[u] * b.z;
            acc[n + 3] += c[u] * b.w;
          }
      }
    }
  }
  // all of the row's Cin values before any store: C may be Cin
  float cin[NC];
  if (it.Cin) {
#pragma unroll
    for (int n = 0; n < NC; ++n) cin[n] = ldg_unit<CG>(it.Cin + row + (long long)min(n, N - 1) * it.ldcin);
  }
  if (row0 + (int)threadIdx.x >= it.M) return;
#pragma unroll
  for (int n = 0; n < NC; ++n) {
    if (n >= N) break;
    float v = alpha * acc[n];
    if (it.Cin) v += beta * cin[n];
    it.C[row + (long long)n * it.ldc] = v;
  }
}

// The same for tall items (the broadcast d -= u eta): 256 rows per unit, A
// through a cp.async ring of kRingK k-values per stage, which keeps 40 KB per
// CTA in flight from the unit's start.  Each thread has 4 adjacent rows (at 8
// columns; 4 + 4 at more) x NC / 4 columns (8: 4), so that up to 16 shared
// values feed 64 FMAs: with whole rows per thread the broadcast reads of B,
// a register write of 16 bytes per lane each, took twice the FMAs' time.  Cin
// is fetched into L2 meanwhile and moves 16 bytes at a time.
constexpr int kRingRows = 2 * kRowThreads, kRingK = 8, kRingStages = 6;

template <int NC>
__host__ __device__ constexpr size_t nn_ring_smem() {
  return ((size_t)kRingStages * kRingK * kRingRows + (size_t)kNnSlab * NC) * sizeof(float);
}

template <int NC, bool CG = false>
__device__ inline void nn_ring_unit(const GemmItem<float, float> *__restrict__ items,
                                    const GemmSeg<float> *__restrict__ segs, float alpha,
                                    float beta, int item, int rb, unsigned char *smem_raw) {
  constexpr int KS = kNnSlab, RK = kRingK, ROWS = kRingRows, ST = kRingStages;
  float *As = reinterpret_cast<float *>(smem_raw);  // [stage][RK][ROWS]
  float *Bs = As + ST * RK * ROWS;                  // [KS][NC]
  const GemmItem<float, float> it = items[item];
  const int row0 = rb * ROWS;
  if (row0 >= it.M) return;
  const int tid = threadIdx.x, N = it.N;
  const int rows = min(ROWS, it.M - row0);
  if (it.Cin) {  // a 128-byte line per lane: 8 lines of every column
    const int r = tid % 8 * 32;
    if (r < rows)
      for (int n = tid / 8; n < N; n += kRowThreads / 8)
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(it.Cin + row0 + r + (long long)n * it.ldcin));
  }
  // rows rr + 128 h + 0 .. 3 and columns cc .. cc + CW - 1 of this thread
  constexpr int H = NC == 8 ? 1 : 2, CW = NC == 8 ? 4 : NC / 4;
  const int lane = tid & 31, warp = tid >> 5;
  const int rr = 4 * lane + (NC == 8 ? 128 * (warp >> 1) : 0);
  const int cc = CW * (NC == 8 ? warp & 1 : warp);
  float acc[H][4][CW];
#pragma unroll
  for (int h = 0; h < H; ++h)
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int c = 0; c < CW; ++c) acc[h][q][c] = 0.f;
  for (int sidx = it.seg_begin; sidx < it.seg_begin + it.seg_count; ++sidx) {
    const GemmSeg<float> sg = segs[sidx];
    const int K = sg.K;
    const float *A = sg.A + row0;
    const bool vec = rows == ROWS && ((reinterpret_cast<uintptr_t>(A) & 15) == 0) && sg.lda % 4 == 0;
    // stage i: k-values i RK .. of the rows, zero beyond K (A is never written
    // by the launch, so its copies may go through L1)
    auto load = [&](int i) {
      float *d = As + i % ST * (RK * ROWS);
      if (i * RK < K) {
        if (vec) {
#pragma unroll
          for (int u = 0; u < RK * ROWS / 4 / kRowThreads; ++u) {
            const int e = tid + u * kRowThreads, k = e / (ROWS / 4), r = e % (ROWS / 4) * 4;
            const bool ok = i * RK + k < K;
            cpa(d + k * ROWS + r, A + r + (long long)(ok ? i * RK + k : 0) * sg.lda, 16, ok);
          }
        } else {
#pragma unroll
          for (int u = 0; u < RK * ROWS / kRowThreads; ++u) {
            const int e = tid + u * kRowThreads, k = e / ROWS, r = e % ROWS;
            const bool ok = i * RK + k < K && r < rows;
            cpa(d + k * ROWS + r, ok ? A + r + (long long)(i * RK + k) * sg.lda : sg.A, 4, ok);
          }
        }
      }
      cpa_commit();
    };
    __syncthreads();  // the previous segment's (or unit's) reads are done
#pragma unroll
    for (int i = 0; i < ST - 1; ++i) load(i);
    for (int k0 = 0; k0 < K; k0 += KS) {
      if (k0 > 0) __syncthreads();
      load_b_slab<NC, CG>(Bs, sg, N, k0);
      for (int kk = 0; kk < KS && k0 + kk < K; kk += RK) {
        const int i = (k0 + kk) / RK;
        cpa_wait<ST - 2>();
        __syncthreads();  // stage i (and the slab) visible; slot of stage i - 1 free
        load(i + ST - 1);
        const float *a = As + i % ST * (RK * ROWS) + rr;
        constexpr int UN = NC == 32 ? 2 : RK;
#pragma unroll UN
        for (int u = 0; u < RK; ++u) {
          float4 v[H], w[CW / 4];
#pragma unroll
          for (int h = 0; h < H; ++h)
            v[h] = *reinterpret_cast<const float4 *>(a + u * ROWS + 128 * h);
#pragma unroll
          for (int x = 0; x < CW / 4; ++x)
            w[x] = *reinterpret_cast<const float4 *>(Bs + (kk + u) * NC + cc + 4 * x);
          const float *b = reinterpret_cast<const float *>(w);
#pragma unroll
          for (int h = 0; h < H; ++h)
#pragma unroll
            for (int c = 0; c < CW; ++c) {
              acc[h][0][c] += v[h].x * b[c];
              acc[h][1][c] += v[h].y * b[c];
              acc[h][2][c] += v[h].z * b[c];
              acc[h][3][c] += v[h].w * b[c];
            }
        }
      }
    }
    cpa_wait<0>();
  }
  // Cin values before the stores (C may be Cin, so a load after a store would
  // wait for it)
  auto aligned = [](const float *p, long long ld) {
    return ((reinterpret_cast<uintptr_t>(p) & 15) == 0) && ld % 4 == 0;
  };
  const bool vec = aligned(it.C + row0, it.ldc) && (!it.Cin || aligned(it.Cin + row0, it.ldcin));
#pragma unroll
  for (int h = 0; h < H; ++h) {
    const int r = rr + 128 * h;
    if (r >= rows) continue;
    if (vec && r + 4 <= rows) {
#pragma unroll
      for (int c0 = 0; c0 < CW; c0 += CW < 4 ? CW : 4) {
        constexpr int CB = CW < 4 ? CW : 4;
        float4 cin[CB];
        if (it.Cin) {
#pragma unroll
          for (int c = 0; c < CB; ++c) {
            const float4 *cp = reinterpret_cast<const float4 *>(
                it.Cin + row0 + r + (long long)min(cc + c0 + c, N - 1) * it.ldcin);
            cin[c] = CG ? __ldcg(cp) : *cp;
          }
        }
#pragma unroll
        for (int c = 0; c < CB; ++c) {
          const int n = c0 + c;
          if (cc + n >= N) break;
          float4 v = make_float4(alpha * acc[h][0][n], alpha * acc[h][1][n], alpha * acc[h][2][n],
                                 alpha * acc[h][3][n]);
          if (it.Cin) {
            v.x += beta * cin[c].x;
            v.y += beta * cin[c].y;
            v.z += beta * cin[c].z;
            v.w += beta * cin[c].w;
          }
          *reinterpret_cast<float4 *>(it.C + row0 + r + (long long)(cc + n) * it.ldc) = v;
        }
      }
    } else {
      float cin[4][CW];
      if (it.Cin) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int c = 0; c < CW; ++c)
            cin[q][c] = ldg_unit<CG>(it.Cin + row0 + min(r + q, rows - 1) +
                                     (long long)min(cc + c, N - 1) * it.ldcin);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int c = 0; c < CW; ++c) {
          if (r + q >= rows || cc + c >= N) continue;
          float v = alpha * acc[h][q][c];
          if (it.Cin) v += beta * cin[q][c];
          it.C[row0 + r + q + (long long)(cc + c) * it.ldc] = v;
        }
    }
  }
}

// ---------------------------------------------------------------- TN
// FP32 C (64 x NC block) = beta Cin + alpha sum_s A_s^T B_s over all of an
// item's K, 128 k-values of both operands at a time in shared memory
// (k-contiguous, as in memory): all of a sweep's slot at once.  Each of the
// four warps takes a quarter of the k-values for the whole block, a lane
// having 8 rows x NC / 4 columns (NC = 8: 4 x 4), so that a vector read feeds
// up to 16 FMAs; the warps' sums are added in order.  (With 2 x 4 outputs per
// thread and 16-column blocks the shared-memory reads bounded the kernel, and
// right-hand sides above 16 columns read A twice.)
constexpr int kTNThreads = 128;
constexpr int kTnK = 128, kTnLd = kTnK + 4;

template <int NC>
__host__ __device__ constexpr size_t tn_smem() { return (size_t)(64 + NC) * kTnLd * sizeof(float); }

// One CTA (kTNThreads threads): rows 64 mt .. of item `item`; smem holds
// tn_smem<NC>() bytes.  CTA-uniform.
template <int NC, bool CG = false>
__device__ inline void tn_unit(const GemmItem<float, float> *__restrict__ items,
                               const GemmSeg<float> *__restrict__ segs, float alpha, float beta,
                               int item, int mt, unsigned char *smem_raw) {
  constexpr int TM = 64, R = NC == 8 ? 4 : 8, MG = TM / R, NG = 32 / MG, CW = NC / NG;
  constexpr int KR = kTnK / (kTNThreads / 32);
  float *As = reinterpret_cast<float *>(smem_raw);  // [TM][kTnLd]
  float *Bs = As + TM * kTnLd;                      // [NC][kTnLd]
  const GemmItem<float, float> it = items[item];
  const int m0 = mt * TM;
  if (m0 >= it.M) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int mg = lane % MG, ng = lane / MG;  // rows mg + MG j, columns ng + NG c
  const int rows = min(TM, it.M - m0);
  float acc[R][CW];
#pragma unroll
  for (int j = 0; j < R; ++j)
#pragma unroll
    for (int c = 0; c < CW; ++c) acc[j][c] = 0.f;
  // k-values k0 .. k0 + kTnK of `cols` columns from c0 (zero beyond K and, up
  // to `pad` columns, beyond cols) into dst[col][kTnLd].  fresh: values that
  // this launch may have written (not through L1)
  auto load_block = [&](float *dst, const float *base, long long ld, int k0, int K, int c0,
                        int cols, int pad, bool fresh) {
    const float *p0 = base + k0 + (long long)c0 * ld;
    const bool vec = ((reinterpret_cast<uintptr_t>(p0) & 15) == 0) && (ld % 4 == 0);
    if (vec && k0 + kTnK <= K) {
      for (int e = tid; e < cols * (kTnK / 4); e += kTNThreads) {
        const int c = e / (kTnK / 4), k = e % (kTnK / 4) * 4;
        cpa(dst + c * kTnLd + k, p0 + k + (long long)c * ld, 16, true);
      }
    } else {
      // a thread per k-value, eight columns in flight
      const bool in = k0 + tid < K;
      const float *p = p0 + (in ? tid : 0);
      for (int c = 0; c < cols; c += 8) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const float *q = p + (long long)min(c + u, cols - 1) * ld;
          v[u] = fresh ? __ldcg(q) : __ldg(q);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (c + u < cols) dst[(c + u) * kTnLd + tid] = in ? v[u] : 0.f;
      }
    }
    for (int c = cols; c < pad; ++c) dst[c * kTnLd + tid] = 0.f;
  };
  static_assert(kTnK == kTNThreads, "a thread per k-value");
  for (int sidx = it.seg_begin; sidx < it.seg_begin + it.seg_count; ++sidx) {
    const GemmSeg<float> sg = segs[sidx];
    for (int k0 = 0; k0 < sg.K; k0 += kTnK) {
      __syncthreads();  // the previous block's (or unit's) reads are done
      load_block(As, sg.A, sg.lda, k0, sg.K, m0, rows, (rows + MG - 1) / MG * MG, false);
      load_block(Bs, sg.B, sg.ldb, k0, sg.K, 0, it.N, NC, CG);
      cpa_commit();
      cpa_wait<0>();
      __syncthreads();
      const float *a = As + mg * kTnLd + warp * KR, *b = Bs + ng * kTnLd + warp * KR;
      constexpr int UN = NC == 32 ? 1 : 2;
#pragma unroll UN
      for (int k = 0; k < KR; k += 4) {
        float4 bv[CW];
#pragma unroll
        for (int c = 0; c < CW; ++c)
          bv[c] = *reinterpret_cast<const float4 *>(b + NG * c * kTnLd + k);
#pragma unroll
        for (int j = 0; j < R; ++j) {
          if (MG * j >= rows) break;  // uniform
          const float4 av = *reinterpret_cast<const float4 *>(a + MG * j * kTnLd + k);
#pragma unroll
          for (int c = 0; c < CW; ++c) {
            acc[j][c] += av.x * bv[c].x;
            acc[j][c] += av.y * bv[c].y;
            acc[j][c] += av.z * bv[c].z;
            acc[j][c] += av.w * bv[c].w;
          }
        }
      }
    }
  }
  // the warps' sums in order, every thread TM NC / 128 outputs of a column
  __syncthreads();
  float *red = As;  // [4][NC][TM]
  static_assert(4 * NC <= kTnLd, "the sums fit the block's operands");
#pragma unroll
  for (int j = 0; j < R; ++j)
#pragma unroll
    for (int c = 0; c < CW; ++c) red[(warp * NC + ng + NG * c) * TM + mg + MG * j] = acc[j][c];
  __syncthreads();
  const int gm = m0 + tid % TM;
  constexpr int PER = TM * NC / kTNThreads;  // columns tid / TM, tid / TM + 2, ...
  float v[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int n = tid / TM + 2 * u;
    const float *r = red + n * TM + tid % TM;
    float x = r[0];
#pragma unroll
    for (int w = 1; w < 4; ++w) x += r[w * NC * TM];
    v[u] = alpha * x;
  }
  if (it.Cin) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int n = tid / TM + 2 * u;
      const float *cp = it.Cin + min(gm, it.M - 1) + (long long)min(n, it.N - 1) * it.ldcin;
      v[u] += beta * ldg_unit<CG>(cp);
    }
  }
  if (gm < it.M) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int n = tid / TM + 2 * u;
      if (n < it.N) it.C[gm + (long long)n * it.ldc] = v[u];
    }
  }
}

}  // namespace sk
}  // namespace hodlr
