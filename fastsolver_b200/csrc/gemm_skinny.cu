// gemm_skinny.cu -- batched GEMM items with at most 32 columns (the m
// right-hand sides): the refinement sweeps' reduce / broadcast and the FP64
// HODLR matvec (gemm_simt.cu routes them here).
//
// These products stream a tall operand (V, U or D, up to a few GB per
// launch) against a small one, so they are bound by HBM bandwidth once their
// shared-memory reads are: the FP32 units are those of skinny_units.cuh, the
// FP64 kernels run on the DMMA pipe out of a 3-stage cp.async ring.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "gemm_skinny.cuh"
#include "skinny_units.cuh"
#include "warp_f64.cuh"

namespace hodlr {

namespace {

using namespace sk;

// ---------------------------------------------------------------- FP32
// The resident CTAs (three per SM) take the units (item, row block)
// u = blockIdx.x, blockIdx.x + gridDim.x, ...: at N = 262144 the root's
// m-column broadcast has 2048 blocks of 128 rows, which as one CTA each ran in
// 4.6 waves of short CTAs.
template <int NC>
__global__ void __launch_bounds__(kRowThreads, 3)
    skinny_nn_rows_kernel(const GemmItem<float, float> *__restrict__ items,
                          const GemmSeg<float> *__restrict__ segs, float alpha, float beta,
                          int nunits, int rbn) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  for (int u = blockIdx.x; u < nunits; u += gridDim.x)
    nn_rows_unit<NC>(items, segs, alpha, beta, u / rbn, u % rbn, reinterpret_cast<float *>(smem_raw));
}
template <int NC>
__global__ void __launch_bounds__(kRowThreads, 3)
    skinny_nn_ring_kernel(const GemmItem<float, float> *__restrict__ items,
                          const GemmSeg<float> *__restrict__ segs, float alpha, float beta,
                          int nunits, int rbn) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  for (int u = blockIdx.x; u < nunits; u += gridDim.x)
    nn_ring_unit<NC>(items, segs, alpha, beta, u / rbn, u % rbn, smem_raw);
}

// CTA per (item, 64-row block)
template <int NC>
__global__ void __launch_bounds__(kTNThreads, 3)
    skinny_tn_kernel(const GemmItem<float, float> *__restrict__ items,
                     const GemmSeg<float> *__restrict__ segs, float alpha, float beta) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  tn_unit<NC>(items, segs, alpha, beta, blockIdx.x, blockIdx.y, smem_raw);
}

// ---------------------------------------------------------------- FP64 on the DMMA pipe
// FP64 items (at most 32 columns: the HODLR matvec's D x + U t and V^T x, the node
// products, the leaves' block rows of few right-hand sides) run on the FP64
// tensor-core instruction mma.m16n8k4.f64 (warp_f64.cuh): one instruction per
// 16 x 8 x 4 block instead of 512 FMAs, so the kernels stay bound by the operand
// stream instead of by instruction issue.

// NN: C (M x N) = beta Cin + alpha sum_s A_s B_s, A_s column-major; one CTA
// per (item, ROWS-row block) and all of an item's columns (8 NT8; with two
// passes of 16 the tall operand, all of D and U in a matvec, was read twice
// above 16 columns: 9.0 instead of 7.5 ms at N = 1048576, 32 columns, where
// the DMMA pipe's floor is 4.9 ms), KT
// k-values per stage.  Large: 512 rows (256 above 16 columns, for the
// accumulators), 8 warps, 8 k; small: 128 rows, 4 warps, 16 k, for launches
// that leave SMs without a large block and for items that fill a quarter of one.
template <int NT8, bool SMALL>
struct NnDmma {
  static constexpr int NCS = 8 * NT8;
  static constexpr int ROWS = SMALL ? 128 : NT8 > 2 ? 256 : 512, THREADS = SMALL ? 128 : 256;
  static constexpr int KT = SMALL ? 16 : 8;
  static constexpr int AP = ROWS + 8;              // padded k-row stride (doubles)
  static constexpr int BP = NCS + 4;              // conflict-free fragments
  static constexpr int STAGES = 3;                // (five above 16 columns: no gain)
  static constexpr size_t smem() {
    return (size_t)STAGES * KT * (AP + BP) * sizeof(double);
  }
};

template <int NT8, bool SMALL>
__global__ void __launch_bounds__(NnDmma<NT8, SMALL>::THREADS, 2)
    skinny_nn_dmma_kernel(const GemmItem<double, double> *__restrict__ items,
                          const GemmSeg<double> *__restrict__ segs, double alpha, double beta) {
  using Cfg = NnDmma<NT8, SMALL>;
  constexpr int KT = Cfg::KT, ROWS = Cfg::ROWS, AP = Cfg::AP, THREADS = Cfg::THREADS;
  constexpr int NCS = Cfg::NCS, BP = Cfg::BP, STAGES = Cfg::STAGES;
  constexpr int MT = ROWS / (THREADS / 32) / 16;  // 16-row fragments per warp
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *As = reinterpret_cast<double *>(smem_raw);      // [stage][KT][AP]
  double *Bs = As + (size_t)STAGES * KT * AP;         // [stage][KT][BP]
  const GemmItem<double, double> it = items[blockIdx.x];
  const int row0 = blockIdx.y * ROWS;
  if (row0 >= it.M) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int N = it.N;

  auto load = [&](const TileIter<double> &p, int st) {
    if (p.valid) {
      const GemmSeg<double> &sg = p.sg;
      double *a = As + (size_t)st * KT * AP;
      double *b = Bs + (size_t)st * KT * BP;
      const double *abase = sg.A + row0 + (long long)p.k0 * sg.lda;
      const bool vec = ((reinterpret_cast<uintptr_t>(abase) & 15) == 0) && ((sg.lda & 1) == 0);
      for (int e = tid; e < KT * (ROWS / 2); e += THREADS) {
        const int k = e / (ROWS / 2), rv = e % (ROWS / 2);
        const int r = row0 + 2 * rv;
        const bool kin = p.k0 + k < sg.K;
        const double *src = abase + 2 * rv + (long long)k * sg.lda;
        double *dst = a + k * AP + 2 * rv;
        if (vec && kin && r + 2 <= it.M) {
          cpa(dst, src, 16, true);
        } else {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const bool ok = kin && r + u < it.M;
            cpa(dst + u, ok ? src + u : sg.A, 8, ok);
          }
        }
      }
      for (int e = tid; e < KT * NCS; e += THREADS) {
        const int k = e % KT, n = e / KT;
        const bool ok = (p.k0 + k < sg.K) && n < N;
        cpa(b + k * BP + n, ok ? sg.B + (p.k0 + k) + (long long)n * sg.ldb : sg.B, 8,
            ok);
      }
    }
    cpa_commit();
  };

  double acc[MT][NT8][4];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[mt][nt][v] = 0.0;
  TileIter<double> ld, cp;
  ld.init(segs, it.seg_begin, it.seg_count);
  cp = ld;
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) {
    load(ld, i);
    if (ld.valid) ld.next(KT);
  }
  int st = 0, lst = STAGES - 1;
  const int wrow = warp * 16 * MT;
  while (cp.valid) {
    load(ld, lst);
    if (ld.valid) ld.next(KT);
    lst = (lst + 1) % STAGES;
    cpa_wait<STAGES - 1>();
    __syncthreads();
    const double *a = As + (size_t)st * KT * AP;
    const double *b = Bs + (size_t)st * KT * BP;
#pragma unroll
    for (int ks = 0; ks < KT; ks += 4) {
      const double *ak = a + (ks + t) * AP + wrow + g;
      double bv[NT8];
#pragma unroll
      for (int nt = 0; nt < NT8; ++nt) bv[nt] = b[(ks + t) * BP + nt * 8 + g];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const double a0 = ak[mt * 16], a1 = ak[mt * 16 + 8];
#pragma unroll
        for (int nt = 0; nt < NT8; ++nt) dmma(acc[mt][nt], a0, a1, bv[nt]);
      }
    }
    __syncthreads();  // stage st is refilled STAGES - 1 tiles later
    st = (st + 1) % STAGES;
    cp.next(KT);
  }
  cpa_wait<0>();
  // per 16-row fragment: its Cin values before its stores (C may alias Cin,
  // so a load after a store would wait for it)
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    double cin[NT8][4];
#pragma unroll
    for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int row = row0 + wrow + mt * 16 + g + (v >> 1) * 8;
        const int c = nt * 8 + 2 * t + (v & 1);
        cin[nt][v] = (it.Cin && row < it.M && c < N) ? it.Cin[row + c * (long long)it.ldcin]
                                                      : 0.0;
      }
#pragma unroll
    for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int row = row0 + wrow + mt * 16 + g + (v >> 1) * 8;
        const int c = nt * 8 + 2 * t + (v & 1);
        if (row < it.M && c < N) {
          const long long col = c;
          double val = alpha * acc[mt][nt][v];
          if (it.Cin) val += beta * cin[nt][v];
          it.C[row + col * it.ldc] = val;
        }
      }
  }
}

// TN: C (64 rows of an item and all of its 8 NT8 columns, over all K) =
// beta Cin + alpha sum_s A_s^T B_s
constexpr int kDmmaKC = 32;
constexpr int kDmmaLDK = kDmmaKC + 4;  // padded k stride (doubles): conflict-free fragments

template <int NT8>
constexpr size_t tn_dmma_smem() {
  return (size_t)kSkStages * (64 + 8 * NT8) * kDmmaLDK * sizeof(double);
}

template <int NT8>
__global__ void __launch_bounds__(kTNThreads)
    skinny_tn_dmma_kernel(const GemmItem<double, double> *__restrict__ items,
                          const GemmSeg<double> *__restrict__ segs, double alpha, double beta) {
  constexpr int TM = 64, TN = 8 * NT8, KC = kDmmaKC, LDK = kDmmaLDK;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *As = reinterpret_cast<double *>(smem_raw);   // [stage][TM][LDK]
  double *Bs = As + (size_t)kSkStages * TM * LDK;      // [stage][TN][LDK]
  const GemmItem<double, double> it = items[blockIdx.x];
  const int m0 = blockIdx.y * TM;
  if (m0 >= it.M) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;

  auto load_block = [&](double *dst, const double *base, long long ld, int k0, int K, int c0,
                        int ncols, int cmax) {
    const double *p0 = base + k0 + (long long)c0 * ld;
    const bool vec = ((reinterpret_cast<uintptr_t>(p0) & 15) == 0) && ((ld & 1) == 0);
    for (int e = tid; e < ncols * (KC / 2); e += kTNThreads) {
      const int c = e / (KC / 2), kv = e % (KC / 2);
      const int k = k0 + 2 * kv;
      const bool colok = c0 + c < cmax;
      const double *src = p0 + 2 * kv + (long long)c * ld;
      double *d = dst + c * LDK + 2 * kv;
      if (vec && colok && k + 2 <= K) {
        cpa(d, src, 16, true);
      } else {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const bool ok = colok && k + u < K;
          cpa(d + u, ok ? src + u : base, 8, ok);
        }
      }
    }
  };
  auto load = [&](const TileIter<double> &p, int st) {
    if (p.valid) {
      load_block(As + (size_t)st * TM * LDK, p.sg.A, p.sg.lda, p.k0, p.sg.K, m0, TM, it.M);
      load_block(Bs + (size_t)st * TN * LDK, p.sg.B, p.sg.ldb, p.k0, p.sg.K, 0, TN, it.N);
    }
    cpa_commit();
  };

  double acc[NT8][4];
#pragma unroll
  for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[nt][v] = 0.0;
  TileIter<double> ld, cp;
  ld.init(segs, it.seg_begin, it.seg_count);
  cp = ld;
#pragma unroll
  for (int i = 0; i < kSkStages - 1; ++i) {
    load(ld, i);
    if (ld.valid) ld.next(KC);
  }
  int st = 0, lst = kSkStages - 1;
  while (cp.valid) {
    load(ld, lst);
    if (ld.valid) ld.next(KC);
    lst = (lst + 1) % kSkStages;
    cpa_wait<kSkStages - 1>();
    __syncthreads();
    const double *a = As + (size_t)st * TM * LDK + (warp * 16 + g) * LDK + t;
    const double *b = Bs + (size_t)st * TN * LDK + g * LDK + t;
#pragma unroll
    for (int ks = 0; ks < KC; ks += 4) {
      const double a0 = a[ks], a1 = a[8 * LDK + ks];
#pragma unroll
      for (int nt = 0; nt < NT8; ++nt) dmma(acc[nt], a0, a1, b[8 * nt * LDK + ks]);
    }
    __syncthreads();
    st = (st + 1) % kSkStages;
    cp.next(KC);
  }
  cpa_wait<0>();
  // every Cin value before any store (C may alias Cin)
  double cin[NT8][4];
#pragma unroll
  for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int gm = m0 + warp * 16 + g + (v >> 1) * 8;
      const int gn = nt * 8 + 2 * t + (v & 1);
      cin[nt][v] = (it.Cin && gm < it.M && gn < it.N) ? it.Cin[gm + (long long)gn * it.ldcin] : 0.0;
    }
#pragma unroll
  for (int nt = 0; nt < NT8; ++nt)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int gm = m0 + warp * 16 + g + (v >> 1) * 8;
      const int gn = nt * 8 + 2 * t + (v & 1);
      if (gm < it.M && gn < it.N) {
        double val = alpha * acc[nt][v];
        if (it.Cin) val += beta * cin[nt][v];
        it.C[gm + (long long)gn * it.ldc] = val;
      }
    }
}

// f(blocks of 8 columns of the widest item)
template <typename F>
void dmma_by_width(int max_n, F &&f) {
  if (max_n <= 8) f(std::integral_constant<int, 1>{});
  else if (max_n <= 16) f(std::integral_constant<int, 2>{});
  else if (max_n <= 24) f(std::integral_constant<int, 3>{});
  else f(std::integral_constant<int, 4>{});
}

}  // namespace

template <typename T>
void launch_skinny(const GemmItem<T, T> *items, const GemmSeg<T> *segs, int nitems, int max_m,
                   int max_n, bool trans, T alpha, T beta, cudaStream_t s) {
  if (nitems <= 0 || max_m <= 0 || max_n <= 0) return;
  if constexpr (sizeof(T) == 8) {
    // FP64 products run on the FP64 tensor pipe (DMMA)
    if (trans) {
      dmma_by_width(max_n, [&](auto w) {
        constexpr int NT8 = decltype(w)::value;
        auto kern = skinny_tn_dmma_kernel<NT8>;
        raise_smem_limit(reinterpret_cast<const void *>(kern), tn_dmma_smem<NT8>());
        kern<<<dim3(nitems, cdiv(max_m, 64)), kTNThreads, tn_dmma_smem<NT8>(), s>>>(items, segs,
                                                                                  alpha, beta);
      });
    } else {
      // Small blocks where large ones would leave SMs idle or mostly empty:
      // matvec of 4096 rows 88 -> 36 us, 60001 rows 201 -> 184 us, node
      // products of 128 rows 233 -> 129 us per solve; above, large ones stream
      // faster (131072 rows: 346 us large, 404 us small).
      const bool small = max_m <= 256 || (long long)nitems * cdiv(max_m, 512) < 148;
      auto go = [&](auto kern, auto cfg) {
        using Cfg = decltype(cfg);
        raise_smem_limit(reinterpret_cast<const void *>(kern), Cfg::smem());
        const dim3 grid(nitems, cdiv(max_m, Cfg::ROWS));
        kern<<<grid, Cfg::THREADS, Cfg::smem(), s>>>(items, segs, alpha, beta);
      };
      dmma_by_width(max_n, [&](auto w) {
        constexpr int NT8 = decltype(w)::value;
        if (small) go(skinny_nn_dmma_kernel<NT8, true>, NnDmma<NT8, true>{});
        else go(skinny_nn_dmma_kernel<NT8, false>, NnDmma<NT8, false>{});
      });
    }
    HODLR_LAUNCH_CHECK();
    return;
  }
  if constexpr (sizeof(T) == 4) {
    auto by_width = [&](auto &&f) {
      if (max_n <= 8) f(std::integral_constant<int, 8>{});
      else if (max_n <= 16) f(std::integral_constant<int, 16>{});
      else f(std::integral_constant<int, 32>{});
    };
    by_width([&](auto w) {
      constexpr int NC = decltype(w)::value;
      if (trans) {
        auto kern = skinny_tn_kernel<NC>;
        raise_smem_limit(reinterpret_cast<const void *>(kern), tn_smem<NC>());
        kern<<<dim3(nitems, cdiv(max_m, 64)), kTNThreads, tn_smem<NC>(), s>>>(items, segs, alpha,
                                                                              beta);
        return;
      }
      int sms = 148, dev = 0;
      if (cudaGetDevice(&dev) == cudaSuccess)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      cudaGetLastError();
      auto units = [&](auto kern, int rows, size_t smem) {
        const int rbn = cdiv(max_m, rows);
        const long long nunits = (long long)nitems * rbn;
        if (nunits > 0x7fffffffLL) throw CudaError{cudaErrorInvalidValue};
        const int grid = (int)std::min<long long>(nunits, 3LL * sms);
        raise_smem_limit(reinterpret_cast<const void *>(kern), smem);
        kern<<<grid, kRowThreads, smem, s>>>(items, segs, alpha, beta, (int)nunits, rbn);
      };
      // short items (the node products) a row per thread, tall ones by the ring
      if (max_m <= kRowThreads)
        units(skinny_nn_rows_kernel<NC>, kRowThreads, (size_t)kNnSlab * NC * sizeof(float));
      else
        units(skinny_nn_ring_kernel<NC>, kRingRows, nn_ring_smem<NC>());
    });
    HODLR_LAUNCH_CHECK();
  }
}

template void launch_skinny<double>(const GemmItem<double, double> *, const GemmSeg<double> *,
                                    int, int, int, bool, double, double, cudaStream_t);
template void launch_skinny<float>(const GemmItem<float, float> *, const GemmSeg<float> *, int,
                                   int, int, bool, float, float, cudaStream_t);

}  // namespace hodlr
