// solver.cu -- device-resident HODLR system and its level schedule.
//
// The reference launches one Legion task per leaf and per (node, leaf) pair
// and lets region privileges order them (src/solver/fast_solver.cc:136-255).
// Here the same dependence structure is a fixed schedule on one stream:
//   1. every leaf at once: getrf + getrs (solver_tasks.cc:424-450);
//   2. for each depth d from the deepest internal level up to the root, every
//      internal node of depth d at once:
//        reduce  V_c^T [d_c | u_c] for both children (gemm.cc:208-229, as
//                split-K partial sums, summed in a fixed order by the node
//                kernel instead of REDOP_ADD atomics),
//        node    capacitance LU and eta (solver_tasks.cc:139-305),
//        bcast   d_c -= u_c eta (gemm.cc:232-284).
// Nodes of equal depth touch disjoint rows, so batching them does not change
// any operation's inputs; the leaf solves have no inputs from other tasks.
// All launch descriptors are built once per system and live on the device,
// so a solve is a fixed sequence of launches (capturable in a CUDA graph).
#include <algorithm>
#include <type_traits>
#include <cmath>
#include <cstring>

#include "gemm_simt.cuh"
#include "leaf_blocked.cuh"
#include "node.cuh"
#include "solver.h"

namespace hodlr {

namespace {

template <typename T, typename TE>
struct PathSpec {
  T *X = nullptr;           // d columns (and the U columns on factor paths)
  long long ldx = 0;
  const T *Usrc = nullptr;  // transformed U columns (== X on factor paths)
  long long ldu = 0;
  T *D = nullptr;           // leaf LU factors
  long long ldd = 0;
  int *ipiv = nullptr, *perm = nullptr;
  const T *V = nullptr;
  long long ldv = 0;
  T *part = nullptr;   // split-K partial slots
  T *wfin = nullptr;   // summed W per child (when a child has several slots)
  TE *eta = nullptr;
  TE *M = nullptr;     // per-node solve matrices, (2r)^2 each
  NodeStore *ns = nullptr;
  const LeafPlan<T> *factors = nullptr;  // apply paths: the blocked leaf factors
  std::shared_ptr<LeafPlan<T>> leaf;     // factor paths: a built leaf plan to share, or null
  int nb_force = 0;                      // leaf panel width (0: by the largest leaf)
  int ob = 0;                            // leaf outer block width (0: one level)
  bool factor = false;
  int red_chunk = 512, bc_chunk = 512;
  int max_slots = 64;  // split-K slots per child at most
  int leaf_size = 1;  // nodes with at most this many real leaves use the 2r x 2r form
};

// Rows per split-K slot of a child with `nrow` rows: at least `chunk` rows,
// at most `max_slots` slots (the slots are summed into one W per child).
// The factor passes use up to 64 slots of >= 512 rows (wide products, few
// long tiles per SM); the FP32 refinement sweeps, whose products have only
// m columns, up to 1024 slots of >= 128 rows, so that the persistent sweep
// kernel's reduce step has many short units instead of a few long ones.
constexpr int kMaxSlots = 64;
constexpr int kSweepChunk = 128, kSweepMaxSlots = 1024;
inline int slot_rows(int nrow, int chunk, int max_slots = kMaxSlots) {
  const int ns = std::max(1, std::min(cdiv(nrow, chunk), max_slots));
  return cdiv(cdiv(nrow, ns), 16) * 16;
}

// Partial-sum, summed-W and eta workspace (elements) of a path's largest level.
void path_need(const Tree &t, bool factor, int chunk, size_t &part, size_t &wfin, size_t &eta,
               int max_slots = kMaxSlots) {
  part = wfin = eta = 0;
  for (int d = t.max_depth - 1; d >= 0; --d) {
    size_t p = 0, w = 0, e = 0;
    for (int id : t.internal_at_depth[d]) {
      const Node &P = t.nodes[id];
      const Node &c0 = t.nodes[P.lchild], &c1 = t.nodes[P.rchild];
      const int cw = factor ? c0.col_beg : t.nrhs;
      for (const Node *c : {&c0, &c1}) {
        const int NW = factor ? c->col_beg + c->ncol : t.nrhs;
        const int ns = cdiv(c->nrow, slot_rows(c->nrow, chunk, max_slots));
        p += (size_t)ns * c->vncol * NW;
        if (ns > 1) w += (size_t)c->vncol * NW;
      }
      e += (size_t)(c0.ncol + c1.ncol) * cw;
    }
    part = std::max(part, p);
    wfin = std::max(wfin, w);
    eta = std::max(eta, e);
  }
}


// One step of the two-level blocked leaf factorization (see LeafPlan and
// leaf_blocked.cu) with its GEMM items on the host.
template <typename T>
struct HostStep : LeafPlan<T>::StepInfo {
  std::vector<GemmItem<T, T>> it;
  std::vector<GemmSeg<T>> sg;
  void add(T *C, long long ldc, int M, int N, const T *A, long long lda, const T *B,
           long long ldb, int K, bool inplace, int tri = 0) {
    if (M <= 0 || N <= 0 || K <= 0) return;
    GemmSeg<T> g{A, B, lda, ldb, K, tri};
    GemmItem<T, T> i{C, inplace ? C : nullptr, ldc, inplace ? ldc : 0, M, N, (int)sg.size(), 1};
    sg.push_back(g);
    it.push_back(i);
  }
};

// The steps of the blocked factorization of `tasks` (panels of NB columns in
// outer blocks of OB, a multiple of NB): forward steps on [D | X], then the
// backward solve on X, each one merged launch over all leaves; a leaf without
// work in a step contributes no item.  binv: block-row solves by the inverses
// of the outer diagonal blocks, in place on the block's rows, which one GEMM
// tile row (128) covers (the GEMM launchers run launches of items of at most
// 128 rows as one tile row).  FP64 steps solve with the triangles themselves
// where these are ill-conditioned.
template <typename T>
void leaf_steps(const std::vector<LeafFactorTask<T>> &tasks, int NB, int OB, int nblocks, bool binv,
                int slots, std::vector<HostStep<T>> &fwd, std::vector<HostStep<T>> &bwd) {
  using Plan = LeafPlan<T>;
  const int P = OB / NB;
  auto step = [](typename Plan::Kind kind) {
    HostStep<T> st;
    st.kind = kind;
    return st;
  };
  auto laswp_step = [&](int p0, int np, int a0, int a1, int b0, int b1, bool with_x) {
    HostStep<T> st = step(Plan::kLaswp);
    st.panel = p0;
    st.np = np;
    st.a0 = a0; st.a1 = a1; st.b0 = b0; st.b1 = b1;
    st.with_x = with_x;
    return st;
  };
  constexpr int kAll = 1 << 30;
  constexpr bool kSubst = std::is_same<T, double>::value;
  // the panel's rows of the D columns [b0, b1) and X by its triangle
  auto panel_solve = [&](int panel, int b0, int b1, bool with_x, bool upper) {
    HostStep<T> st = step(Plan::kPanelSolve);
    st.panel = panel;
    st.b0 = b0; st.b1 = b1;
    st.with_x = with_x;
    st.upper = upper;
    for (const LeafFactorTask<T> &k : tasks)
      if (panel * NB < k.n)
        st.cols = std::max(st.cols, std::max(0, std::min(b1, k.n) - b0) + (with_x ? k.ncols : 0));
    return st;
  };
  auto block_solve = [&](int J, bool upper) {
    HostStep<T> st = step(Plan::kBlockSolve);
    st.block = J;
    st.upper = upper;
    for (const LeafFactorTask<T> &k : tasks)
      if (J * OB < k.n)
        st.cols = std::max(st.cols, (upper ? 0 : std::max(0, k.n - J * OB - OB)) + k.ncols);
    return st;
  };
  for (int J = 0; J < nblocks; ++J) {
    const int j0 = J * OB;
    // the block's panels: factor, interchange and update inside the block columns
    for (int p = 0; p < P; ++p) {
      const int pi = J * P + p, k0 = pi * NB;
      HostStep<T> pan = step(Plan::kPanel);
      pan.k0 = k0;
      pan.panel = pi;
      fwd.push_back(pan);
      fwd.push_back(laswp_step(pi, 1, j0, k0, k0 + NB, j0 + OB, false));
      HostStep<T> tr = step(Plan::kTrsm), up = step(Plan::kUpdate);
      for (const LeafFactorTask<T> &k : tasks) {
        if (k0 >= k.n) continue;
        const int kb = std::min(NB, k.n - k0);
        const int N = std::min(j0 + OB, k.n) - (k0 + kb);
        const int rest = k.n - k0 - kb;
        const T *Li = k.Linv + (size_t)pi * NB * NB;
        T *U12 = k.D + k0 + (long long)(k0 + kb) * k.ldd;
        if (!kSubst) tr.add(U12, k.ldd, kb, N, Li, NB, U12, k.ldd, kb, false);
        up.add(k.D + (k0 + kb) + (long long)(k0 + kb) * k.ldd, k.ldd, rest, N,
               k.D + (k0 + kb) + (long long)k0 * k.ldd, k.ldd, U12, k.ldd, kb, true);
      }
      fwd.push_back(kSubst ? panel_solve(pi, k0 + NB, j0 + OB, false, false) : std::move(tr));
      fwd.push_back(std::move(up));
    }
    // the block's interchanges on the columns left and right of it and on X
    fwd.push_back(laswp_step(J * P, P, 0, j0, j0 + OB, kAll, true));
    if (binv) {
      // block rows: U12 = L11^{-1} A12 on R = (D right of the block | X), one
      // product with the inverse of the block's unit-lower triangle
      HostStep<T> inv = step(Plan::kBlockInv);
      inv.block = J;
      fwd.push_back(inv);
      HostStep<T> tr = step(Plan::kTrsm);
      for (const LeafFactorTask<T> &k : tasks) {
        if (j0 >= k.n) continue;
        const int obe = std::min(OB, k.n - j0);
        const T *Li = k.Binv + (size_t)(J % slots) * OB * OB;
        T *Dr = k.D + j0 + (long long)(j0 + obe) * k.ldd;
        T *Xr = k.X + j0;
        tr.add(Dr, k.ldd, obe, k.n - j0 - obe, Li, OB, Dr, k.ldd, obe, false, 1);
        tr.add(Xr, k.ldx, obe, k.ncols, Li, OB, Xr, k.ldx, obe, false, 1);
      }
      fwd.push_back(std::move(tr));
      if (kSubst) fwd.push_back(block_solve(J, false));
    }
    // block rows: U12 = L11^{-1} A12 by panels on R = (D right of the block | X)
    for (int p = 0; p < (binv ? 0 : P); ++p) {
      const int pi = J * P + p, k0 = pi * NB;
      HostStep<T> tr = step(Plan::kTrsm), up = step(Plan::kUpdate);
      for (const LeafFactorTask<T> &k : tasks) {
        if (k0 >= k.n) continue;
        const int kb = std::min(NB, k.n - k0);
        const int obe = std::min(OB, k.n - j0);
        const int nd = k.n - j0 - obe;           // D columns right of the block
        const int below = j0 + obe - k0 - kb;    // block rows below this panel
        const T *Li = k.Linv + (size_t)pi * NB * NB;
        T *Dr = k.D + k0 + (long long)(j0 + obe) * k.ldd;
        T *Xr = k.X + k0;
        if (!kSubst) {
          tr.add(Dr, k.ldd, kb, nd, Li, NB, Dr, k.ldd, kb, false);
          tr.add(Xr, k.ldx, kb, k.ncols, Li, NB, Xr, k.ldx, kb, false);
        }
        const T *L = k.D + (k0 + kb) + (long long)k0 * k.ldd;
        up.add(Dr + kb, k.ldd, below, nd, L, k.ldd, Dr, k.ldd, kb, true);
        up.add(Xr + kb, k.ldx, below, k.ncols, L, k.ldd, Xr, k.ldx, kb, true);
      }
      fwd.push_back(kSubst ? panel_solve(pi, j0 + OB, kAll, true, false) : std::move(tr));
      fwd.push_back(std::move(up));
    }
    // trailing update of depth OB: A22 -= L21 U12 on R, rows below the block
    HostStep<T> big = step(Plan::kUpdate);
    for (const LeafFactorTask<T> &k : tasks) {
      if (j0 >= k.n) continue;
      const int obe = std::min(OB, k.n - j0);
      const int rest = k.n - j0 - obe;
      const T *L21 = k.D + (j0 + obe) + (long long)j0 * k.ldd;
      big.add(k.D + (j0 + obe) + (long long)(j0 + obe) * k.ldd, k.ldd, rest, rest, L21, k.ldd,
              k.D + j0 + (long long)(j0 + obe) * k.ldd, k.ldd, obe, true);
      big.add(k.X + (j0 + obe), k.ldx, rest, k.ncols, L21, k.ldd, k.X + j0, k.ldx, obe, true);
    }
    fwd.push_back(std::move(big));
  }
  // backward solve on X, last block first
  for (int J = nblocks - 1; J >= 0; --J) {
    const int j0 = J * OB;
    if (binv) {
      // X[block] = U11^{-1} X[block]: one product with the block's upper inverse
      HostStep<T> tr = step(Plan::kTrsm);
      for (const LeafFactorTask<T> &k : tasks) {
        if (j0 >= k.n) continue;
        const int obe = std::min(OB, k.n - j0);
        T *Xk = k.X + j0;
        tr.add(Xk, k.ldx, obe, k.ncols, k.Binv + (size_t)(J % slots) * OB * OB, OB, Xk, k.ldx, obe,
               false, 2);
      }
      bwd.push_back(std::move(tr));
      if (kSubst) bwd.push_back(block_solve(J, true));
    }
    for (int p = binv ? -1 : P - 1; p >= 0; --p) {
      const int pi = J * P + p, k0 = pi * NB;
      HostStep<T> tr = step(Plan::kTrsm), up = step(Plan::kUpdate);
      for (const LeafFactorTask<T> &k : tasks) {
        if (k0 >= k.n) continue;
        const int kb = std::min(NB, k.n - k0);
        T *Xk = k.X + k0;
        if (!kSubst)
          tr.add(Xk, k.ldx, kb, k.ncols, k.Uinv + (size_t)pi * NB * NB, NB, Xk, k.ldx, kb, false);
        up.add(k.X + j0, k.ldx, k0 - j0, k.ncols, k.D + j0 + (long long)k0 * k.ldd, k.ldd, Xk,
               k.ldx, kb, true);
      }
      bwd.push_back(kSubst ? panel_solve(pi, 0, 0, true, true) : std::move(tr));
      bwd.push_back(std::move(up));
    }
    HostStep<T> big = step(Plan::kUpdate);
    for (const LeafFactorTask<T> &k : tasks) {
      if (j0 >= k.n) continue;
      const int obe = std::min(OB, k.n - j0);
      big.add(k.X, k.ldx, j0, k.ncols, k.D + (long long)j0 * k.ldd, k.ldd, k.X + j0, k.ldx, obe,
              true);
    }
    bwd.push_back(std::move(big));
  }
}

// FP64 outer block width without a request, for `rows` rows in leaves of at
// most max_n: 0 (one level) or 128.  Blocks of 128 read and write the trailing
// matrix a quarter as often but lengthen the chain of launches by the blocks'
// triangular inverses, so they pay once a factorization is bound by its
// updates: whole FP64 solves on one level / with 128, in ms: 4096 rows in
// leaves of 256 0.60 / 0.65, of 512 0.96 / 1.04; 12000 rows in leaves of 375
// 1.25 / 1.29; 16384 rows of 512 1.68 / 1.62; 60001 rows of 469 4.18 / 3.76;
// 262144 rows of 512 27.5 / 22.0.  Above 512 rows panels are 16 wide, and one
// level means 16-deep updates: 6000 rows in leaves of 750 2.02 / 1.89.
int leaf_ob_auto64(long long rows, int max_n) {
  return max_n > 512 || (max_n > 128 && rows * max_n >= (8 << 20)) ? 128 : 0;
}

// Slots of outer-block inverses per leaf.  FP32: all blocks, so that the upper
// inverses are one launch.  FP64: as many as fit in 32 MB over all leaves, at
// least one; lower and upper ones of all blocks took 0.5 GB at N = 262144 (512
// leaves of 512 rows), where one launch per block instead of one for all costs 0.4 %
// of the solve.
template <typename T>
int binv_slots(long long leaves, int nblocks, int ob) {
  if (sizeof(T) == 4) return nblocks;
  const long long fit = (32LL << 20) / std::max(1LL, leaves * ob * ob * (long long)sizeof(T));
  return (int)std::min<long long>(nblocks, std::max(1LL, fit));
}

// The blocked factorization of every leaf of a tree as uploaded steps.
template <typename T>
void build_leaf_plan(const Tree &t, T *Dbase, long long ldd, T *Xbase, long long ldx,
                     int *ipiv, int *perm, bool factor_cols_all, int m, LeafPlan<T> &lp,
                     int nb_force, int ob_req) {
  using Step = typename LeafPlan<T>::Step;
  const int nleaf = (int)t.leaves.size();
  lp.max_n = 0;
  for (int id : t.leaves) lp.max_n = std::max(lp.max_n, t.nodes[id].nrow);
  const int NB = nb_force > 0 ? nb_force : leaf_nb<T>(lp.max_n);
  const int OB = ob_req >= NB ? ob_req / NB * NB : NB;
  const int P = OB / NB;
  lp.nb = NB;
  lp.ob = OB;
  const int max_panels = cdiv(lp.max_n, NB);
  lp.nblocks = cdiv(lp.max_n, OB);
  lp.Linv.ensure((size_t)nleaf * max_panels * NB * NB);
  lp.Uinv.ensure((size_t)nleaf * max_panels * NB * NB);
  const bool binv = P > 1 && OB <= 128;
  lp.binv = binv;
  if (binv) {
    lp.slots = binv_slots<T>(nleaf, lp.nblocks, OB);
    lp.Binv.ensure((size_t)nleaf * lp.slots * OB * OB);
  }
  lp.swapflag.ensure((size_t)nleaf * max_panels);
  if (binv && std::is_same<T, double>::value) lp.ill_b.ensure((size_t)nleaf * lp.nblocks * 2);
  std::vector<LeafFactorTask<T>> tasks(nleaf);
  lp.laswp_cols = 0;
  for (int q = 0; q < nleaf; ++q) {
    const Node &nd = t.nodes[t.leaves[q]];
    LeafFactorTask<T> &k = tasks[q];
    k.D = Dbase + nd.row_beg;
    k.ldd = ldd;
    k.X = Xbase + nd.row_beg;
    k.ldx = ldx;
    k.ipiv = ipiv + nd.row_beg;
    k.perm = perm + nd.row_beg;
    k.Linv = lp.Linv.p + (size_t)q * max_panels * NB * NB;
    k.Uinv = lp.Uinv.p + (size_t)q * max_panels * NB * NB;
    k.swapflag = lp.swapflag.p + (size_t)q * max_panels;
    k.ill_b = lp.ill_b.p ? lp.ill_b.p + (size_t)q * lp.nblocks * 2 : nullptr;
    k.Binv = binv ? lp.Binv.p + (size_t)q * lp.slots * OB * OB : nullptr;
    k.n = nd.nrow;
    k.ncols = factor_cols_all ? nd.col_beg + nd.ncol : m;
    k.info_slot = q;
    lp.laswp_cols = std::max(lp.laswp_cols, k.n + k.ncols);
  }
  lp.tasks.upload(tasks);
  lp.host_tasks = tasks;
  lp.nleaf = nleaf;
  lp.fwd.clear();
  lp.bwd.clear();
  std::vector<HostStep<T>> fwd, bwd;
  leaf_steps<T>(tasks, NB, OB, lp.nblocks, binv, lp.slots, fwd, bwd);
  auto upload = [](const std::vector<HostStep<T>> &src, std::vector<std::unique_ptr<Step>> &dst) {
    for (const HostStep<T> &h : src) {
      auto st = std::make_unique<Step>();
      static_cast<typename LeafPlan<T>::StepInfo &>(*st) = h;
      if (h.kind == LeafPlan<T>::kTrsm || h.kind == LeafPlan<T>::kUpdate) st->g.set(h.it, h.sg);
      dst.push_back(std::move(st));
    }
  };
  upload(fwd, lp.fwd);
  upload(bwd, lp.bwd);
  lp.fwd_per_block = (int)lp.fwd.size() / std::max(lp.nblocks, 1);
  lp.bwd_per_block = (int)lp.bwd.size() / std::max(lp.nblocks, 1);
}

template <typename TA, typename TC, typename TACC>
void run_gemm(const GemmLaunch<TA, TC> &g, bool trans, TACC alpha, TACC beta, cudaStream_t s) {
  launch_gemm_items<TA, TC, TACC>(g.items.p, g.segs.p, g.n, g.max_m, g.max_n, trans, alpha, beta,
                                  s);
}

template <typename T>
void run_leaf_plan(Profiler &pf, const LeafPlan<T> &lp, int *info, cudaStream_t s);

// The level descriptors of an FP32 apply path for the persistent sweep
// kernel, when every level's products have at most 32 columns.
template <typename T, typename TE>
void build_sweep(PathPlan<T, TE> &plan) {
  plan.sweep_ok = false;
  if constexpr (std::is_same<T, float>::value && std::is_same<TE, float>::value) {
    if (plan.factor || plan.levels.empty()) return;
    std::vector<SweepLevel> v;
    int mx = 0;
    for (const auto &Lp : plan.levels) {
      const LevelPlan<T, TE> &L = *Lp;
      if (L.red_max_n > 32 || L.ap_max_n > 32 || L.bc_max_n > 32) return;
      SweepLevel d{};
      d.red_items = L.red_items.p;
      d.red_segs = L.red_segs.p;
      d.n_red = L.n_red;
      d.red_mt = cdiv(std::max(L.red_max_m, 1), 64);
      d.sums = L.sums.p;
      d.n_sums = L.n_sums;
      d.sum_units = (int)cdiv<long long>(std::max<long long>(L.sum_max_len, 1), kSweepSumChunk);
      d.sum_max_slots = L.sum_max_slots;
      d.ap_items = L.ap_items.p;
      d.ap_segs = L.ap_segs.p;
      d.n_ap = L.n_ap;
      d.ap_rb = cdiv(std::max(L.ap_max_m, 1), 128);
      d.bc_items = L.bc_items.p;
      d.bc_segs = L.bc_segs.p;
      d.n_bc = L.n_bc;
      d.bc_rb = cdiv(std::max(L.bc_max_m, 1), 256);
      mx = std::max({mx, L.red_max_n, L.ap_max_n, L.bc_max_n});
      v.push_back(d);
    }
    plan.sweep.upload(v);
    plan.sweep_bar.ensure(kSweepBarWords);
    plan.sweep_max_n = std::max(mx, 1);
    plan.sweep_ok = true;
  }
}

template <typename T, typename TE>
void build_path(const Tree &t, const PathSpec<T, TE> &sp, PathPlan<T, TE> &plan, int form) {
  plan.levels.clear();
  plan.factor = sp.factor;
  plan.nleaf = (int)t.leaves.size();
  const int m = t.nrhs;
  if (sp.factor) {
    if (sp.leaf) {
      plan.leaf = sp.leaf;
    } else {
      if (!plan.leaf) plan.leaf = std::make_shared<LeafPlan<T>>();
      build_leaf_plan<T>(t, sp.D, sp.ldd, sp.X, sp.ldx, sp.ipiv, sp.perm, true, m, *plan.leaf,
                         sp.nb_force, sp.ob);
    }
  } else {
    std::vector<LeafFactorTask<T>> at = sp.factors->host_tasks;
    for (size_t q = 0; q < at.size(); ++q) {
      const Node &n = t.nodes[t.leaves[q]];
      at[q].X = sp.X + n.row_beg;
      at[q].ldx = sp.ldx;
      at[q].ncols = m;
    }
    plan.apply_tasks.upload(at);
    plan.apply_nb = sp.factors->nb;
    plan.apply_max_n = sp.factors->max_n;
    plan.apply_max_cols = m;
  }
  const int nleaf = (int)t.leaves.size();

  for (int d = t.max_depth - 1; d >= 0; --d) {
    const auto &ids = t.internal_at_depth[d];
    if (ids.empty()) continue;
    auto L = std::make_unique<LevelPlan<T, TE>>();
    std::vector<GemmItem<T, T>> ri, bi;
    std::vector<GemmSeg<T>> rs, bs;
    std::vector<NodeTask<T, TE>> nt[2];
    std::vector<SumTask<T>> su;
    std::vector<GemmItem<T, T>> ai;
    std::vector<GemmSeg<T>> as;
    size_t poff = 0, woff = 0, eoff = 0;
    L->v_lo = 1 << 30;
    for (int p : ids) {
      const Node &P = t.nodes[p];
      const Node &c0 = t.nodes[P.lchild], &c1 = t.nodes[P.rchild];
      const int cw = sp.factor ? c0.col_beg : m;
      for (const Node *c : {&c0, &c1}) {
        L->v_lo = std::min(L->v_lo, c->col_beg - m);
        L->v_hi = std::max(L->v_hi, c->col_beg - m + c->vncol);
      }
      NodeTask<T, TE> k{};
      const T *W0d = nullptr, *W1d = nullptr;
      long long ldw0d = 0, ldw1d = 0;
      for (int side = 0; side < 2; ++side) {
        const Node &c = side ? c1 : c0;
        const int NW = sp.factor ? c.col_beg + c.ncol : m;
        const int M = c.vncol;
        const int rows_per = slot_rows(c.nrow, sp.red_chunk, sp.max_slots);
        const int nslots = cdiv(c.nrow, rows_per);
        T *slot0 = sp.part + poff;
        for (int q = 0; q < nslots; ++q) {
          const int rb = c.row_beg + q * rows_per;
          const int rows = std::min(rows_per, c.row_beg + c.nrow - rb);
          GemmSeg<T> sg{};
          sg.A = sp.V + rb + (long long)(c.col_beg - m) * sp.ldv;
          sg.B = sp.X + rb;
          sg.lda = sp.ldv;
          sg.ldb = sp.ldx;
          sg.K = rows;
          GemmItem<T, T> it{};
          it.C = slot0 + (size_t)q * M * NW;
          it.Cin = nullptr;
          it.ldc = M;
          it.M = M;
          it.N = NW;
          it.seg_begin = (int)rs.size();
          it.seg_count = 1;
          rs.push_back(sg);
          ri.push_back(it);
          L->red_max_m = std::max(L->red_max_m, M);
          L->red_max_n = std::max(L->red_max_n, NW);
        }
        poff += (size_t)nslots * M * NW;
        T *W = slot0;
        if (nslots > 1) {
          W = sp.wfin + woff;
          woff += (size_t)M * NW;
          SumTask<T> st{};
          st.dst = W;
          st.src = slot0;
          st.len = (long long)M * NW;
          st.stride = (long long)M * NW;
          st.nslots = nslots;
          su.push_back(st);
          L->sum_max_len = std::max(L->sum_max_len, st.len);
          L->sum_max_slots = std::max(L->sum_max_slots, nslots);
        }
        if (side == 0) {
          W0d = W; k.W0u = W + (size_t)M * (NW - c.ncol);
          ldw0d = k.ldw0u = M;
        } else {
          W1d = W; k.W1u = W + (size_t)M * (NW - c.ncol);
          ldw1d = k.ldw1u = M;
        }
      }
      const int r0 = c0.ncol, r1 = c1.ncol, s2 = r0 + r1;
      k.r0 = r0;
      k.r1 = r1;
      // eta = [eta0; eta1] (s2 x cw, ld s2): eta0 feeds child 0, eta1 child 1
      TE *eta = sp.eta + eoff;
      eoff += (size_t)s2 * cw;
      k.F = sp.ns->F.p + (size_t)p * sp.ns->rr;
      k.M = sp.M + (size_t)p * sp.ns->mm;
      k.info_slot = nleaf + p;
      // the node's form: 1 everywhere when asked for, else 1 inside a Legion leaf
      const int nform = (form == 1 || inside_legion_leaf(t, p, sp.leaf_size)) ? 1 : 0;
      nt[nform].push_back(k);
      const int s = nform == 0 ? r0 : s2;
      L->max_s[nform] = std::max(L->max_s[nform], s);
      L->max_r[nform] = std::max(L->max_r[nform], std::max(r0, r1));
      if (cw > 0) {
        // [eta0; eta1] = M [V0Td0; V1Td1]: one item, two K segments
        GemmSeg<T> a0{}, a1{};
        a0.A = reinterpret_cast<const T *>(k.M);
        a0.lda = s2;
        a0.B = W0d;
        a0.ldb = ldw0d;
        a0.K = r1;
        a1.A = reinterpret_cast<const T *>(k.M) + (size_t)r1 * s2;
        a1.lda = s2;
        a1.B = W1d;
        a1.ldb = ldw1d;
        a1.K = r0;
        GemmItem<T, T> it{};
        it.C = reinterpret_cast<T *>(eta);
        it.ldc = s2;
        it.M = s2;
        it.N = cw;
        it.seg_begin = (int)as.size();
        it.seg_count = 2;
        as.push_back(a0);
        as.push_back(a1);
        ai.push_back(it);
        L->ap_max_m = std::max(L->ap_max_m, s2);
        L->ap_max_n = std::max(L->ap_max_n, cw);
      }
      // broadcast d_c -= u_c eta into both children
      for (int side = 0; side < 2; ++side) {
        const Node &c = side ? c1 : c0;
        const TE *eta_c = side ? eta + r0 : eta;
        if (cw == 0) continue;
        for (int rb = c.row_beg; rb < c.row_beg + c.nrow; rb += sp.bc_chunk) {
          const int rows = std::min(sp.bc_chunk, c.row_beg + c.nrow - rb);
          GemmSeg<T> sg{};
          sg.A = sp.Usrc + rb + (long long)c.col_beg * sp.ldu;
          sg.B = reinterpret_cast<const T *>(eta_c);
          sg.lda = sp.ldu;
          sg.ldb = s2;
          sg.K = c.ncol;
          GemmItem<T, T> it{};
          it.C = sp.X + rb;
          it.Cin = sp.X + rb;
          it.ldc = it.ldcin = sp.ldx;
          it.M = rows;
          it.N = cw;
          it.seg_begin = (int)bs.size();
          it.seg_count = 1;
          bs.push_back(sg);
          bi.push_back(it);
          L->bc_max_m = std::max(L->bc_max_m, rows);
          L->bc_max_n = std::max(L->bc_max_n, cw);
        }
      }
    }
    L->red_items.upload(ri);
    L->red_segs.upload(rs);
    L->n_red = (int)ri.size();
    L->sums.upload(su);
    L->n_sums = (int)su.size();
    for (int f = 0; f < 2; ++f) {
      L->node_tasks[f].upload(nt[f]);
      L->n_nodes[f] = (int)nt[f].size();
    }
    L->ap_items.upload(ai);
    L->ap_segs.upload(as);
    L->n_ap = (int)ai.size();
    L->bc_items.upload(bi);
    L->bc_segs.upload(bs);
    L->n_bc = (int)bi.size();
    plan.levels.push_back(std::move(L));
  }
  build_sweep(plan);
  plan.built = true;
}

// RAII phase marker: records a CUDA event pair when profiling is on.
struct PhaseScope {
  Profiler &p;
  int ph;
  cudaStream_t s;
  cudaEvent_t a = nullptr;
  PhaseScope(Profiler &p_, int ph_, cudaStream_t s_) : p(p_), ph(ph_), s(s_) {
    if (p.on) p.begin(ph, s, a);
  }
  ~PhaseScope() {
    if (p.on) p.end(ph, s, a);
  }
};

// What a step of the leaf factorization launches over.
template <typename T>
struct LeafSet {
  const LeafFactorTask<T> *tasks;
  int nleaf, max_n, laswp_cols, nb, ob, slots;
};

// Enqueues one step (a plan's Step or a HostStep) with its GEMM items on the
// device (n of them, at most max_m x max_n).
template <typename T, typename S>
void run_leaf_step(Profiler &pf, const LeafSet<T> &L, const S &st, const GemmItem<T, T> *items,
                   const GemmSeg<T> *segs, int n, int max_m, int max_n, int *info,
                   cudaStream_t s) {
  using Plan = LeafPlan<T>;
  const bool solve = st.kind == Plan::kTrsm;
  switch (st.kind) {
    case Plan::kPanel: {
      PhaseScope pp(pf, PH_LEAF_PANEL, s);
      launch_leaf_panel<T>(L.tasks, L.nleaf, L.max_n, L.nb, st.k0, st.panel, info, s);
      break;
    }
    case Plan::kLaswp: {
      if (st.a1 <= st.a0 && st.b1 <= st.b0 && !st.with_x) break;  // no columns
      PhaseScope pp(pf, PH_LEAF_PANEL, s);
      launch_leaf_laswp<T>(L.tasks, L.nleaf, L.laswp_cols, L.nb, st.panel, st.np, st.a0, st.a1,
                           st.b0, st.b1, st.with_x, s);
      break;
    }
    case Plan::kBlockInv: {
      PhaseScope pt(pf, PH_LEAF_TRSM, s);
      launch_leaf_block_inverse<T>(L.tasks, L.nleaf, L.nb, L.ob, st.block, 1, L.slots, false, s);
      break;
    }
    case Plan::kPanelSolve:
    case Plan::kBlockSolve: {
      if constexpr (std::is_same<T, double>::value) {
        if (st.cols == 0) break;
        PhaseScope pt(pf, PH_LEAF_TRSM, s);
        if (st.kind == Plan::kPanelSolve)
          launch_leaf_panel_solve(L.tasks, L.nleaf, st.cols, L.nb, st.panel, st.b0, st.b1,
                                  st.with_x, st.upper, s);
        else
          launch_leaf_block_solve(L.tasks, L.nleaf, st.cols, L.ob, st.block, st.upper, s);
      }
      break;
    }
    case Plan::kTrsm:
    case Plan::kUpdate: {
      if (n == 0) break;
      PhaseScope pg(pf, solve ? PH_LEAF_TRSM : PH_LEAF_UPDATE, s);
      launch_gemm_items<T, T, T>(items, segs, n, max_m, max_n, false, solve ? T(1) : T(-1),
                                 solve ? T(0) : T(1), s);
      break;
    }
  }
}

// Before the backward steps of block J of nblocks: the upper inverses of it and
// the blocks before it, as many as there are slots, unless they are there.
template <typename T>
void run_upper_inverses(const LeafSet<T> &L, int J, int nblocks, cudaStream_t s) {
  if ((nblocks - 1 - J) % L.slots != 0) return;
  const int J0 = std::max(0, J - L.slots + 1);
  launch_leaf_block_inverse<T>(L.tasks, L.nleaf, L.nb, L.ob, J0, J - J0 + 1, L.slots, true, s);
}

template <typename T>
void run_leaf_plan(Profiler &pf, const LeafPlan<T> &lp, int *info, cudaStream_t s) {
  const LeafSet<T> L{lp.tasks.p, lp.nleaf, lp.max_n, lp.laswp_cols, lp.nb, lp.ob, lp.slots};
  {
    PhaseScope ps(pf, PH_GETRF, s);
    launch_leaf_init<T>(lp.tasks.p, lp.nleaf, info, s);
    for (const auto &st : lp.fwd)
      run_leaf_step<T>(pf, L, *st, st->g.items.p, st->g.segs.p, st->g.n, st->g.max_m, st->g.max_n,
                       info, s);
  }
  {
    PhaseScope ps(pf, PH_GETRS, s);
    Profiler off;  // (the backward solve's steps count as PH_GETRS alone)
    for (size_t i = 0; i < lp.bwd.size(); ++i) {
      const auto &st = lp.bwd[i];
      if (lp.binv && i % lp.bwd_per_block == 0)
        run_upper_inverses(L, lp.nblocks - 1 - (int)i / lp.bwd_per_block, lp.nblocks, s);
      run_leaf_step<T>(off, L, *st, st->g.items.p, st->g.segs.p, st->g.n, st->g.max_m, st->g.max_n,
                       info, s);
    }
  }
}

// parts: kPathLeaves (the leaf solves / factorization), kPathLevels (the
// tree levels), or both; the levels read nothing of V before their first
// reduce, so a caller can let V arrive in between
template <typename T, typename TE>
void run_path(Profiler &pf, const PathPlan<T, TE> &plan, int form, int *info, cudaStream_t s,
              int parts = kPathLeaves | kPathLevels, const LevelHook *hook = nullptr) {
  if (!(parts & kPathLeaves)) {
  } else if (plan.factor) {
    run_leaf_plan<T>(pf, *plan.leaf, info, s);
  } else {
    PhaseScope ps(pf, PH_GETRS, s);
    launch_leaf_apply<T>(plan.apply_tasks.p, plan.nleaf, plan.apply_max_n, plan.apply_max_cols,
                         plan.apply_nb, s);
  }
  if (!(parts & kPathLevels)) return;
  if (!plan.factor && plan.sweep_ok && sweep_persistent_enabled()) {
    PhaseScope ps(pf, PH_SWEEP_LEVELS, s);
    launch_sweep_levels(plan.sweep.p, (int)plan.levels.size(), plan.sweep_max_n,
                        plan.sweep_bar.p, s);
    return;
  }
  int li = 0;
  for (const auto &Lp : plan.levels) {
    const LevelPlan<T, TE> &L = *Lp;
    if (hook) (*hook)(li, L.v_lo, L.v_hi);
    ++li;
    {
      PhaseScope ps(pf, PH_REDUCE, s);
      launch_gemm_items<T, T, T>(L.red_items.p, L.red_segs.p, L.n_red, L.red_max_m,
                                 L.red_max_n, true, T(1), T(0), s);
      launch_sum_slots<T>(L.sums.p, L.n_sums, L.sum_max_len, s);
    }
    if (plan.factor) {
      PhaseScope ps(pf, PH_NODE_FACTOR, s);
      for (int f = 0; f < 2; ++f)
        if (L.n_nodes[f] > 0)
          launch_node_factor<T, TE>(L.node_tasks[f].p, L.n_nodes[f], L.max_s[f], L.max_r[f], f,
                                    info, s);
    }
    {
      PhaseScope ps(pf, PH_NODE_APPLY, s);
      launch_gemm_items<T, T, T>(L.ap_items.p, L.ap_segs.p, L.n_ap, L.ap_max_m, L.ap_max_n,
                                 false, T(1), T(0), s);
    }
    {
      PhaseScope ps(pf, PH_BCAST, s);
      launch_gemm_items<T, T, T>(L.bc_items.p, L.bc_segs.p, L.n_bc, L.bc_max_m, L.bc_max_n,
                                 false, T(-1), T(1), s);
    }
  }
}

void alloc_node_store(NodeStore &ns, const Tree &t, bool fp64) {
  const int r = t.rank;
  ns.rr = r * r;
  ns.mm = 4 * r * r;
  const size_t nn = t.nodes.size();
  ns.F.ensure(nn * ns.rr);
  if (fp64) ns.M64.ensure(nn * ns.mm);
  else ns.M32.ensure(nn * ns.mm);
}

void build_matvec(System &S, const double *x, MatvecPlan &mv) {
  const Tree &t = S.tree;
  const int m = S.m;
  const long long N = S.N;
  // rows per split-K slot: 1024, fewer where that would leave the reduce of
  // all levels below four CTAs per SM
  const int chunk = std::min(1024, std::max(128, (int)((long long)N * t.max_depth / 592 / 64 * 64)));
  std::vector<GemmItem<double, double>> ri, ai;
  std::vector<GemmSeg<double>> rs, as;
  std::vector<SumTask<double>> su;
  std::vector<size_t> toff(t.nodes.size(), 0);
  size_t poff = 0, tsz = 0;
  for (size_t i = 1; i < t.nodes.size(); ++i) {
    const Node &c = t.nodes[i];
    toff[i] = tsz;
    tsz += (size_t)c.vncol * m;
  }
  size_t pneed = 0;
  for (size_t i = 1; i < t.nodes.size(); ++i) {
    const int rp = slot_rows(t.nodes[i].nrow, chunk);
    pneed += (size_t)cdiv(t.nodes[i].nrow, rp) * t.nodes[i].vncol * m;
  }
  S.tbuf.ensure(std::max<size_t>(tsz, 1));
  S.mvpart.ensure(std::max<size_t>(pneed, 1));
  mv.red_max_m = mv.red_max_n = 0;
  for (size_t i = 1; i < t.nodes.size(); ++i) {
    const Node &c = t.nodes[i];
    const int M = c.vncol;
    const int rows_per = slot_rows(c.nrow, chunk);
    const int nslots = cdiv(c.nrow, rows_per);
    double *slot0 = S.mvpart.p + poff;
    for (int q = 0; q < nslots; ++q) {
      const int rb = c.row_beg + q * rows_per;
      const int rows = std::min(rows_per, c.row_beg + c.nrow - rb);
      GemmSeg<double> sg{};
      sg.A = S.V.p + rb + (long long)(c.col_beg - m) * N;
      sg.B = x + rb;
      sg.lda = N;
      sg.ldb = N;
      sg.K = rows;
      GemmItem<double, double> it{};
      it.C = slot0 + (size_t)q * M * m;
      it.ldc = M;
      it.M = M;
      it.N = m;
      it.seg_begin = (int)rs.size();
      it.seg_count = 1;
      rs.push_back(sg);
      ri.push_back(it);
      mv.red_max_m = std::max(mv.red_max_m, M);
      mv.red_max_n = std::max(mv.red_max_n, m);
    }
    SumTask<double> st{};
    st.dst = S.tbuf.p + toff[i];
    st.src = slot0;
    st.len = (long long)M * m;
    st.stride = (long long)M * m;
    st.nslots = nslots;
    su.push_back(st);
    mv.sum_max_len = std::max(mv.sum_max_len, st.len);
    poff += (size_t)nslots * M * m;
  }
  mv.ap_max_m = mv.ap_max_n = 0;
  for (int leaf : t.leaves) {
    const Node &n = t.nodes[leaf];
    GemmItem<double, double> it{};
    it.C = S.R64.p + n.row_beg;
    it.Cin = S.B.p + n.row_beg;
    it.ldc = N;
    it.ldcin = N;
    it.M = n.nrow;
    it.N = m;
    it.seg_begin = (int)as.size();
    GemmSeg<double> sd{};
    sd.A = S.D.p + n.row_beg;
    sd.lda = N;
    sd.B = x + n.row_beg;
    sd.ldb = N;
    sd.K = n.nrow;
    as.push_back(sd);
    for (int a = leaf; a > 0; a = t.nodes[a].parent) {
      const Node &an = t.nodes[a];
      const Node &pa = t.nodes[an.parent];
      const int sib = (pa.lchild == a) ? pa.rchild : pa.lchild;
      GemmSeg<double> su_{};
      su_.A = S.U.p + n.row_beg + (long long)(an.col_beg - m) * N;
      su_.lda = N;
      su_.B = S.tbuf.p + toff[sib];
      su_.ldb = an.ncol;
      su_.K = an.ncol;
      as.push_back(su_);
    }
    it.seg_count = (int)as.size() - it.seg_begin;
    ai.push_back(it);
    mv.ap_max_m = std::max(mv.ap_max_m, n.nrow);
    mv.ap_max_n = std::max(mv.ap_max_n, m);
  }
  mv.red_items.upload(ri);
  mv.red_segs.upload(rs);
  mv.n_red = (int)ri.size();
  mv.sums.upload(su);
  mv.n_sums = (int)su.size();
  mv.ap_items.upload(ai);
  mv.ap_segs.upload(as);
  mv.n_ap = (int)ai.size();
  mv.built = true;
}

// ---- merging the plans of several systems into one batch schedule.  All
// descriptors hold absolute device pointers into their own system's buffers,
// so merging is concatenation: item lists shift their segment indices, INFO
// slots shift by the system's offset in the batch's INFO array.

template <typename TA, typename TC>
struct ItemAcc {
  std::vector<GemmItem<TA, TC>> it;
  std::vector<GemmSeg<TA>> sg;
  int max_m = 0, max_n = 0;
  void add(const std::vector<GemmItem<TA, TC>> &items, const std::vector<GemmSeg<TA>> &segs) {
    const int off = (int)sg.size();
    for (GemmItem<TA, TC> x : items) {
      x.seg_begin += off;
      it.push_back(x);
      max_m = std::max(max_m, x.M);
      max_n = std::max(max_n, x.N);
    }
    sg.insert(sg.end(), segs.begin(), segs.end());
  }
  void add(const GemmLaunch<TA, TC> &g) { add(g.items.h, g.segs.h); }
  void store(GemmLaunch<TA, TC> &g) const { g.set(it, sg); }
  void store(DevBuf<GemmItem<TA, TC>> &items, DevBuf<GemmSeg<TA>> &segs, int &n, int &mm,
             int &mn) const {
    items.upload(it);
    segs.upload(sg);
    n = (int)it.size();
    mm = max_m;
    mn = max_n;
  }
};

template <typename T>
void merge_leaf_plans(const std::vector<const LeafPlan<T> *> &src, const std::vector<int> &info_off,
                      LeafPlan<T> &dst) {
  using Step = typename LeafPlan<T>::Step;
  std::vector<LeafFactorTask<T>> tasks;
  dst.max_n = dst.laswp_cols = 0;
  dst.nb = src.empty() ? 0 : src[0]->nb;
  dst.ob = src.empty() ? 0 : src[0]->ob;
  dst.nblocks = 0;
  for (size_t k = 0; k < src.size(); ++k) {
    const LeafPlan<T> &lp = *src[k];
    if (lp.nb != dst.nb || lp.ob != dst.ob) throw CudaError{cudaErrorInvalidValue};
    for (LeafFactorTask<T> t : lp.host_tasks) {
      t.info_slot += info_off[k];
      tasks.push_back(t);
    }
    dst.max_n = std::max(dst.max_n, lp.max_n);
    dst.laswp_cols = std::max(dst.laswp_cols, lp.laswp_cols);
    dst.nblocks = std::max(dst.nblocks, lp.nblocks);
  }
  dst.fwd_per_block = src[0]->fwd_per_block;
  dst.bwd_per_block = src[0]->bwd_per_block;
  dst.binv = src[0]->binv;
  dst.slots = dst.nblocks;  // FP32: every system has a slot per block
  dst.tasks.upload(tasks);
  dst.host_tasks = tasks;
  dst.nleaf = (int)tasks.size();
  dst.fwd.clear();
  dst.bwd.clear();
  // the step lists have the same shape per block in every system (same nb
  // and ob): step i of block J merges the systems that have block J; the
  // backward lists start at each system's own last block
  auto merge_step = [&](const Step &proto, const std::vector<const Step *> &parts) {
    auto st = std::make_unique<Step>();
    static_cast<typename LeafPlan<T>::StepInfo &>(*st) = proto;
    for (const Step *p : parts) st->cols = std::max(st->cols, p->cols);
    if (proto.kind == LeafPlan<T>::kTrsm || proto.kind == LeafPlan<T>::kUpdate) {
      ItemAcc<T, T> acc;
      for (const Step *p : parts) acc.add(p->g);
      acc.store(st->g);
    }
    return st;
  };
  for (int J = 0; J < dst.nblocks; ++J)
    for (int i = 0; i < dst.fwd_per_block; ++i) {
      std::vector<const Step *> parts;
      for (const LeafPlan<T> *lp : src)
        if (J < lp->nblocks) parts.push_back(lp->fwd[(size_t)J * dst.fwd_per_block + i].get());
      dst.fwd.push_back(merge_step(*parts[0], parts));
    }
  for (int J = dst.nblocks - 1; J >= 0; --J)
    for (int i = 0; i < dst.bwd_per_block; ++i) {
      std::vector<const Step *> parts;
      for (const LeafPlan<T> *lp : src)
        if (J < lp->nblocks)
          parts.push_back(lp->bwd[(size_t)(lp->nblocks - 1 - J) * dst.bwd_per_block + i].get());
      dst.bwd.push_back(merge_step(*parts[0], parts));
    }
}

// Level j of the merged plan is level j (deepest first) of every system
// that has one: each system still walks its own levels bottom-up.
template <typename T, typename TE>
void merge_paths(const std::vector<const PathPlan<T, TE> *> &src, const std::vector<int> &info_off,
                 PathPlan<T, TE> &dst) {
  dst.levels.clear();
  dst.factor = src[0]->factor;
  dst.nleaf = 0;
  dst.apply_nb = dst.apply_max_n = dst.apply_max_cols = 0;
  if (dst.factor) {
    std::vector<const LeafPlan<T> *> lps;
    for (const auto *p : src) lps.push_back(p->leaf.get());
    dst.leaf = std::make_shared<LeafPlan<T>>();
    merge_leaf_plans<T>(lps, info_off, *dst.leaf);
    dst.nleaf = dst.leaf->nleaf;
  } else {
    std::vector<LeafFactorTask<T>> at;
    for (const auto *p : src) {
      at.insert(at.end(), p->apply_tasks.h.begin(), p->apply_tasks.h.end());
      if (p->apply_nb != src[0]->apply_nb) throw CudaError{cudaErrorInvalidValue};
      dst.apply_max_n = std::max(dst.apply_max_n, p->apply_max_n);
      dst.apply_max_cols = std::max(dst.apply_max_cols, p->apply_max_cols);
    }
    dst.apply_tasks.upload(at);
    dst.apply_nb = src[0]->apply_nb;
    dst.nleaf = (int)at.size();
  }
  size_t nlev = 0;
  for (const auto *p : src) nlev = std::max(nlev, p->levels.size());
  for (size_t j = 0; j < nlev; ++j) {
    auto L = std::make_unique<LevelPlan<T, TE>>();
    ItemAcc<T, T> red, ap, bc;
    std::vector<SumTask<T>> su;
    std::vector<NodeTask<T, TE>> nt[2];
    for (size_t k = 0; k < src.size(); ++k) {
      if (j >= src[k]->levels.size()) continue;
      const LevelPlan<T, TE> &S = *src[k]->levels[j];
      red.add(S.red_items.h, S.red_segs.h);
      ap.add(S.ap_items.h, S.ap_segs.h);
      bc.add(S.bc_items.h, S.bc_segs.h);
      su.insert(su.end(), S.sums.h.begin(), S.sums.h.end());
      L->sum_max_len = std::max(L->sum_max_len, S.sum_max_len);
      L->sum_max_slots = std::max(L->sum_max_slots, S.sum_max_slots);
      for (int f = 0; f < 2; ++f) {
        for (NodeTask<T, TE> t : S.node_tasks[f].h) {
          t.info_slot += info_off[k];
          nt[f].push_back(t);
        }
        L->max_s[f] = std::max(L->max_s[f], S.max_s[f]);
        L->max_r[f] = std::max(L->max_r[f], S.max_r[f]);
      }
    }
    red.store(L->red_items, L->red_segs, L->n_red, L->red_max_m, L->red_max_n);
    ap.store(L->ap_items, L->ap_segs, L->n_ap, L->ap_max_m, L->ap_max_n);
    bc.store(L->bc_items, L->bc_segs, L->n_bc, L->bc_max_m, L->bc_max_n);
    L->sums.upload(su);
    L->n_sums = (int)su.size();
    for (int f = 0; f < 2; ++f) {
      L->node_tasks[f].upload(nt[f]);
      L->n_nodes[f] = (int)nt[f].size();
    }
    dst.levels.push_back(std::move(L));
  }
  build_sweep(dst);
  dst.built = true;
}

void merge_matvecs(const std::vector<const MatvecPlan *> &src, MatvecPlan &dst) {
  ItemAcc<double, double> red, ap;
  std::vector<SumTask<double>> su;
  dst.sum_max_len = 0;
  for (const MatvecPlan *p : src) {
    red.add(p->red_items.h, p->red_segs.h);
    ap.add(p->ap_items.h, p->ap_segs.h);
    su.insert(su.end(), p->sums.h.begin(), p->sums.h.end());
    dst.sum_max_len = std::max(dst.sum_max_len, p->sum_max_len);
  }
  red.store(dst.red_items, dst.red_segs, dst.n_red, dst.red_max_m, dst.red_max_n);
  ap.store(dst.ap_items, dst.ap_segs, dst.n_ap, dst.ap_max_m, dst.ap_max_n);
  dst.sums.upload(su);
  dst.n_sums = (int)su.size();
  dst.built = true;
}

void matvec_launches(Profiler &pf, const MatvecPlan &p, double alpha, double beta,
                     cudaStream_t s) {
  PhaseScope ps(pf, PH_MATVEC, s);
  launch_gemm_items<double, double, double>(p.red_items.p, p.red_segs.p, p.n_red, p.red_max_m,
                                            p.red_max_n, true, 1.0, 0.0, s);
  launch_sum_slots<double>(p.sums.p, p.n_sums, p.sum_max_len, s);
  launch_gemm_items<double, double, double>(p.ap_items.p, p.ap_segs.p, p.n_ap, p.ap_max_m,
                                            p.ap_max_n, false, alpha, beta, s);
}

// Bytes of a vector, rounded up so that what follows stays 16-byte aligned.
template <typename E>
size_t padded_bytes(const std::vector<E> &v) {
  return (v.size() * sizeof(E) + 15) & ~size_t(15);
}

}  // namespace

LeafBodyShape leaf_body_shape(long long leaves, int max_n) {
  LeafBodyShape S;
  S.max_n = max_n;
  S.nb = leaf_nb<double>(max_n);
  S.ob = std::max(S.nb, leaf_ob_auto64(leaves * max_n, max_n));
  S.nblocks = cdiv(max_n, S.ob);
  // the leaves of a group: as many as fit in the scratch with one slot of block
  // inverses, and then as many slots as still fit
  S.slots = 1;
  const long long base = S.leaf_bytes(), cap = kLeafBodyScratch;
  S.group = (int)std::max(1LL, std::min(leaves, cap / base));
  if (S.ob > S.nb) {
    const long long more = (cap / S.group - base) / ((long long)sizeof(double) * S.ob * S.ob);
    S.slots = (int)std::min<long long>(S.nblocks, 1 + std::max(0LL, more));
  }
  return S;
}

size_t LeafBodyShape::leaf_words() const {
  // panel inverses, block inverses, then as ints: row order, pivots, interchange
  // flags, marks (doubles; even, so that every leaf's inverses start on 16 bytes)
  const size_t np = (size_t)nblocks * (ob / nb);
  const size_t ints = (2 * (size_t)max_n + np + 2 * nblocks + 3) / 4 * 2;
  return 2 * np * nb * nb + (ob > nb ? (size_t)slots * ob * ob : 0) + ints;
}

size_t LeafBodyShape::leaf_bytes() const {
  // the task and at most four GEMM items per panel and six per outer block
  const size_t items = 4 * (size_t)nblocks * (ob / nb) + 6 * (size_t)nblocks;
  return sizeof(double) * leaf_words() + sizeof(LeafFactorTask<double>) +
         items * (sizeof(GemmItem<double, double>) + sizeof(GemmSeg<double>));
}

void run_leaf_bodies(std::vector<LeafFactorTask<double>> tasks, const LeafBodyShape &S, int *info,
                     cudaStream_t s, const std::function<void *(size_t)> &scratch) {
  using T = double;
  using Item = GemmItem<T, T>;
  using Seg = GemmSeg<T>;
  if (tasks.empty()) return;
  int cols = 0;
  for (const auto &k : tasks) cols = std::max(cols, k.n + k.ncols);
  const int NB = S.nb, OB = S.ob, nblocks = S.nblocks, slots = S.slots, max_n = S.max_n;
  const bool binv = OB > NB;
  const size_t np = (size_t)nblocks * (OB / NB), w_inv = np * NB * NB;
  const size_t w_blk = binv ? (size_t)slots * OB * OB : 0, per = S.leaf_words();
  double *w = static_cast<double *>(scratch(std::max<size_t>(sizeof(T) * per * tasks.size(), 16)));
  for (size_t q = 0; q < tasks.size(); ++q) {
    LeafFactorTask<T> &k = tasks[q];
    double *b = w + q * per;
    k.Linv = b;
    k.Uinv = b + w_inv;
    k.Binv = binv ? b + 2 * w_inv : nullptr;
    int *ip = reinterpret_cast<int *>(b + 2 * w_inv + w_blk);
    if (!k.perm) k.perm = ip;
    if (!k.ipiv) k.ipiv = ip + max_n;
    k.swapflag = ip + 2 * max_n;
    k.ill_b = k.swapflag + np;
  }
  std::vector<HostStep<T>> fwd, bwd;
  leaf_steps<T>(tasks, NB, OB, nblocks, binv, slots, fwd, bwd);
  // one block of descriptors: tasks | items | segments
  std::vector<Item> items;
  std::vector<Seg> segs;
  for (auto *v : {&fwd, &bwd})
    for (const HostStep<T> &h : *v) {
      items.insert(items.end(), h.it.begin(), h.it.end());
      segs.insert(segs.end(), h.sg.begin(), h.sg.end());
    }
  const size_t o_items = padded_bytes(tasks), o_segs = o_items + padded_bytes(items);
  std::vector<char> blob(o_segs + padded_bytes(segs));
  std::memcpy(blob.data(), tasks.data(), sizeof(tasks[0]) * tasks.size());
  if (!items.empty()) {
    std::memcpy(blob.data() + o_items, items.data(), sizeof(Item) * items.size());
    std::memcpy(blob.data() + o_segs, segs.data(), sizeof(Seg) * segs.size());
  }
  char *dev = static_cast<char *>(scratch(blob.size()));
  if (blob.size() <= 64 * 1024)
    launch_param_copy(dev, blob.data(), blob.size(), s);
  else
    HODLR_CUDA_TRY(cudaMemcpyAsync(dev, blob.data(), blob.size(), cudaMemcpyHostToDevice, s));
  Profiler off;
  const LeafSet<T> L{reinterpret_cast<const LeafFactorTask<T> *>(dev), (int)tasks.size(), max_n,
                     cols, NB, OB, slots};
  const Item *di = reinterpret_cast<const Item *>(dev + o_items);
  const Seg *ds = reinterpret_cast<const Seg *>(dev + o_segs);
  auto run = [&](const HostStep<T> &h) {
    int mm = 0, mn = 0;
    for (const Item &x : h.it) {
      mm = std::max(mm, x.M);
      mn = std::max(mn, x.N);
    }
    run_leaf_step<T>(off, L, h, di, ds, (int)h.it.size(), mm, mn, info, s);
    di += h.it.size();
    ds += h.sg.size();
  };
  launch_leaf_init<T>(L.tasks, L.nleaf, info, s);
  for (const HostStep<T> &h : fwd) run(h);
  const size_t per_block = bwd.size() / std::max(nblocks, 1);
  for (size_t i = 0; i < bwd.size(); ++i) {
    if (binv && i % per_block == 0)
      run_upper_inverses(L, nblocks - 1 - (int)(i / per_block), nblocks, s);
    run(bwd[i]);
  }
}

void Profiler::begin(int ph, cudaStream_t s, cudaEvent_t &a) {
  HODLR_CUDA_TRY(cudaEventCreate(&a));
  HODLR_CUDA_TRY(cudaEventRecord(a, s));
  (void)ph;
}
void Profiler::end(int ph, cudaStream_t s, cudaEvent_t a) {
  cudaEvent_t b;
  HODLR_CUDA_TRY(cudaEventCreate(&b));
  HODLR_CUDA_TRY(cudaEventRecord(b, s));
  recs.push_back({ph, a, b});
}
void Profiler::collect() {
  for (auto &r : recs) {
    HODLR_CUDA_TRY(cudaEventSynchronize(r.b));
    float t = 0.f;
    HODLR_CUDA_TRY(cudaEventElapsedTime(&t, r.a, r.b));
    ms[r.phase] += t;
    launches[r.phase] += 1;
    cudaEventDestroy(r.a);
    cudaEventDestroy(r.b);
  }
  recs.clear();
}
void Profiler::reset() {
  collect();
  for (int i = 0; i < PH_COUNT; ++i) { ms[i] = 0; launches[i] = 0; }
}

int System::init(int N_, int nrhs, int rank, int threshold) {
  int rc = build_tree(N_, nrhs, rank, threshold, tree);
  if (rc) return rc;
  if (2 * rank > kMaxNodeS && rank > kMaxNodeS) return -3;
  N = N_;
  m = nrhs;
  r = rank;
  C = tree.ncols;
  vc = tree.vcols();
  nmax = tree.max_leaf;
  const size_t n = (size_t)N;
  D.ensure(n * nmax);
  U.ensure(n * std::max(vc, 1));
  V.ensure(n * std::max(vc, 1));
  B.ensure(n * m);
  Xsol.ensure(n * m);
  R64.ensure(n * m);
  MVx.ensure(n * m);
  relres_dev.ensure(m);
  ratio_part.ensure((size_t)m * kRatioChunks * 2);
  n_info = (int)(tree.leaves.size() + tree.nodes.size());
  info.ensure(n_info);
  HODLR_CUDA_TRY(cudaMemset(info.p, 0, sizeof(int) * n_info));
  HODLR_CUDA_TRY(cudaMemset(D.p, 0, sizeof(double) * n * nmax));
  HODLR_CUDA_TRY(cudaMemset(U.p, 0, sizeof(double) * n * std::max(vc, 1)));
  HODLR_CUDA_TRY(cudaMemset(V.p, 0, sizeof(double) * n * std::max(vc, 1)));
  HODLR_CUDA_TRY(cudaMemset(B.p, 0, sizeof(double) * n * m));
  HODLR_CUDA_TRY(cudaMemset(Xsol.p, 0, sizeof(double) * n * m));
  build_matvec(*this, Xsol.p, mv_sol);
  build_matvec(*this, MVx.p, mv_usr);
  return 0;
}

void System::ensure_fp64() {
  if (fused64[0].built) return;
  const size_t n = (size_t)N;
  X64.ensure(n * C);
  DLU64.ensure(n * nmax);
  Y64.ensure(n * m);
  ipiv64.ensure(n);
  perm64.ensure(n);
  alloc_node_store(ns64, tree, true);
  size_t pf, wf, ef, pa, wa, ea;
  path_need(tree, true, red_chunk, pf, wf, ef);
  path_need(tree, false, red_chunk, pa, wa, ea);
  part64.ensure(std::max<size_t>(std::max(pf, pa), 1));
  wfin64.ensure(std::max<size_t>(std::max(wf, wa), 1));
  eta64.ensure(std::max<size_t>(std::max(ef, ea), 1));
  for (int form = 0; form < 2; ++form) {
    if (form == 1 && 2 * r > kMaxNodeS) continue;
    PathSpec<double, double> f;
    f.X = X64.p; f.ldx = N; f.Usrc = X64.p; f.ldu = N;
    f.D = DLU64.p; f.ldd = N; f.ipiv = ipiv64.p; f.perm = perm64.p;
    f.V = V.p; f.ldv = N; f.part = part64.p; f.wfin = wfin64.p; f.eta = eta64.p; f.M = ns64.M64.p; f.ns = &ns64;
    f.factor = true; f.red_chunk = red_chunk; f.bc_chunk = bc_chunk;
    f.ob = ob64 > 0 ? ob64 : leaf_ob_auto64(N, nmax);
    f.leaf_size = leaf_size;
    if (form == 1) f.leaf = fused64[0].leaf;
    build_path(tree, f, fused64[form], form);
    PathSpec<double, double> a = f;
    a.X = Y64.p; a.factor = false; a.factors = fused64[form].leaf.get();
    build_path(tree, a, apply64[form], form);
  }
}

void System::ensure_mixed() {
  if (fused32.built) return;
  const size_t n = (size_t)N;
  X32.ensure(n * C);
  D32.ensure(n * nmax);
  V32.ensure(n * std::max(vc, 1));
  Y32.ensure(n * m);
  ipiv32.ensure(n);
  perm32.ensure(n);
  alloc_node_store(ns32, tree, false);
  size_t pf, wf, ef, pa, wa, ea;
  path_need(tree, true, red_chunk, pf, wf, ef);
  path_need(tree, false, kSweepChunk, pa, wa, ea, kSweepMaxSlots);
  part32.ensure(std::max<size_t>(std::max(pf, pa), 1));
  wfin32.ensure(std::max<size_t>(std::max(wf, wa), 1));
  eta32.ensure(std::max<size_t>(std::max(ef, ea), 1));
  PathSpec<float, float> f;
  f.X = X32.p; f.ldx = N; f.Usrc = X32.p; f.ldu = N;
  f.D = D32.p; f.ldd = N; f.ipiv = ipiv32.p; f.perm = perm32.p;
  f.V = V32.p; f.ldv = N; f.part = part32.p; f.wfin = wfin32.p; f.eta = eta32.p; f.M = ns32.M32.p; f.ns = &ns32;
  f.factor = true; f.red_chunk = red_chunk; f.bc_chunk = bc_chunk; f.nb_force = nb32;
  f.ob = ob32;
  build_path(tree, f, fused32, 0);
  PathSpec<float, float> a = f;
  a.X = Y32.p; a.factor = false; a.factors = fused32.leaf.get();
  a.red_chunk = kSweepChunk;
  a.max_slots = kSweepMaxSlots;
  build_path(tree, a, apply32, 0);
}

void System::run_fused64(int form, cudaStream_t s) {
  ensure_fp64();
  const size_t n = (size_t)N;
  HODLR_CUDA_TRY(cudaMemcpyAsync(DLU64.p, D.p, sizeof(double) * n * nmax, cudaMemcpyDeviceToDevice, s));
  HODLR_CUDA_TRY(cudaMemcpyAsync(X64.p, B.p, sizeof(double) * n * m, cudaMemcpyDeviceToDevice, s));
  if (vc > 0)
    HODLR_CUDA_TRY(cudaMemcpyAsync(X64.p + n * m, U.p, sizeof(double) * n * vc,
                                   cudaMemcpyDeviceToDevice, s));
  run_path(prof, fused64[form], form, info.p, s);
  HODLR_CUDA_TRY(cudaMemcpyAsync(Xsol.p, X64.p, sizeof(double) * n * m, cudaMemcpyDeviceToDevice, s));
  factored = HODLR_PREC_FP64;
  factored_form = form;
}

void System::run_apply64(cudaStream_t s) {
  run_path(prof, apply64[factored_form], factored_form, nullptr, s);
}

void System::run_factor32(cudaStream_t s) {
  run_factor32_part(kPathLeaves | kPathLevels, s);
}

void System::run_factor32_part(int parts, cudaStream_t s) {
  convert32(parts, s);
  run_path(prof, fused32, 0, info.p, s, parts);
  if (parts & kPathLevels) {
    factored = HODLR_PREC_MIXED;
    factored_form = 0;
  }
}

void System::run_factor32_levels_hooked(const LevelHook &hook, cudaStream_t s) {
  ensure_mixed();
  run_path(prof, fused32, 0, info.p, s, kPathLevels, &hook);
  factored = HODLR_PREC_MIXED;
  factored_form = 0;
}

void System::convert_v32(int lo, int hi, cudaStream_t s) {
  if (hi <= lo) return;
  PhaseScope ps(prof, PH_CONVERT, s);
  launch_convert2d<double, float>(V.p + (size_t)lo * N, N, V32.p + (size_t)lo * N, N, N, hi - lo, s);
}

void System::convert32(int parts, cudaStream_t s) {
  ensure_mixed();
  const long long n = N;
  {
    PhaseScope ps(prof, PH_CONVERT, s);
    if (parts & kPathLeaves) {  // what the leaf factorization reads: D and [b | U]
      launch_convert2d<double, float>(D.p, n, D32.p, n, n, nmax, s);
      launch_convert2d<double, float>(B.p, n, X32.p, n, n, m, s);
      if (vc > 0) launch_convert2d<double, float>(U.p, n, X32.p + (size_t)n * m, n, n, vc, s);
    }
    if ((parts & kPathLevels) && vc > 0)  // V, first read by the levels' reduce
      launch_convert2d<double, float>(V.p, n, V32.p, n, n, vc, s);
  }
}

void System::run_apply32(cudaStream_t s) { run_path(prof, apply32, 0, nullptr, s); }

void System::run_matvec(const MatvecPlan &p, double alpha, double beta, cudaStream_t s) {
  matvec_launches(prof, p, alpha, beta, s);
}

int System::check_info(cudaStream_t s) {
  std::vector<int> h(n_info);
  HODLR_CUDA_TRY(cudaMemcpyAsync(h.data(), info.p, sizeof(int) * n_info, cudaMemcpyDeviceToHost, s));
  HODLR_CUDA_TRY(cudaStreamSynchronize(s));
  const int nleaf = (int)tree.leaves.size();
  for (int i = 0; i < n_info; ++i)
    if (h[i] != 0) return i < nleaf ? h[i] : 100000 + h[i];
  return 0;
}

void System::relres_enqueue(cudaStream_t s) {
  run_matvec(mv_sol, -1.0, 1.0, s);
  launch_colratio(R64.p, N, B.p, N, N, m, ratio_part.p, relres_dev.p, s);
}

double System::relres(cudaStream_t s) {
  relres_enqueue(s);
  return relres_read(s);
}

double System::relres_read(cudaStream_t s) {
  std::vector<double> h(m);
  HODLR_CUDA_TRY(cudaMemcpyAsync(h.data(), relres_dev.p, sizeof(double) * m,
                                 cudaMemcpyDeviceToHost, s));
  HODLR_CUDA_TRY(cudaStreamSynchronize(s));
  double mx = 0.0;
  for (double v : h) mx = std::max(mx, std::isnan(v) ? INFINITY : v);
  return mx;
}

// ---- Batch

void Batch::build(const std::vector<System *> &systems) {
  if (systems.empty()) throw CudaError{cudaErrorInvalidValue};
  sys = systems;
  groups.clear();
  for (size_t k = 0; k < sys.size(); ++k) {
    System *S = sys[k];
    S->ensure_mixed();
    const int nbk = S->fused32.leaf->nb, obk = S->fused32.leaf->ob;
    const bool wide = S->m > 16;
    Group *g = nullptr;
    for (auto &q : groups)
      if (q->nb == nbk && q->ob == obk && q->wide == wide) g = q.get();
    if (!g) {
      groups.push_back(std::make_unique<Group>());
      g = groups.back().get();
      g->nb = nbk;
      g->ob = obk;
      g->wide = wide;
    }
    g->members.push_back((int)k);
  }
  info_off.clear();
  rr_off.clear();
  n_info = 0;
  int n_rr = 0;
  max_m = 0;
  std::vector<const MatvecPlan *> mp;
  std::vector<Ew2DTask<double, float>> cin, cres;
  std::vector<Ew2DTask<float, double>> cx0, addy;
  std::vector<RatioTask> rt;
  for (System *S : sys) {
    info_off.push_back(n_info);
    n_info += S->n_info;
    rr_off.push_back(n_rr);
    n_rr += S->m;
    max_m = std::max(max_m, S->m);
    mp.push_back(&S->mv_sol);
    const long long n = S->N;
    auto add_in = [&](const double *src, float *dst, long long cols) {
      if (cols > 0) cin.push_back({src, n, dst, n, n, cols, 0});
    };
    add_in(S->D.p, S->D32.p, S->nmax);
    add_in(S->B.p, S->X32.p, S->m);
    add_in(S->U.p, S->X32.p + (size_t)n * S->m, S->vc);
    add_in(S->V.p, S->V32.p, S->vc);
    cres.push_back({S->R64.p, n, S->Y32.p, n, n, S->m, 0});
    cx0.push_back({S->X32.p, n, S->Xsol.p, n, n, S->m, 0});
    addy.push_back({S->Y32.p, n, S->Xsol.p, n, n, S->m, 0});
  }
  t_in = ew2d_prefix(cin);
  t_res = ew2d_prefix(cres);
  t_x0 = ew2d_prefix(cx0);
  ew2d_prefix(addy);
  rr.ensure(std::max(n_rr, 1));
  for (size_t k = 0; k < sys.size(); ++k) {
    System *S = sys[k];
    RatioTask t{};
    t.r = S->R64.p;
    t.ldr = S->N;
    t.b = S->B.p;
    t.ldb = S->N;
    t.rows = S->N;
    t.out = rr.p + rr_off[k];
    t.cols = S->m;
    rt.push_back(t);
  }
  for (auto &g : groups) {
    std::vector<const PathPlan<float, float> *> fp, ap;
    std::vector<int> off;
    for (int k : g->members) {
      fp.push_back(&sys[k]->fused32);
      ap.push_back(&sys[k]->apply32);
      off.push_back(info_off[k]);
    }
    merge_paths<float, float>(fp, off, g->fused32);
    merge_paths<float, float>(ap, off, g->apply32);
  }
  merge_matvecs(mp, mv);
  cv_in.upload(cin);
  cv_res.upload(cres);
  cv_x0.upload(cx0);
  add_y.upload(addy);
  ratios.upload(rt);
  info.ensure(n_info);
  HODLR_CUDA_TRY(cudaMemset(info.p, 0, sizeof(int) * n_info));
  g_factor.reset();
  g_sweep.reset();
}

void Batch::residuals(cudaStream_t s) {
  matvec_launches(prof, mv, -1.0, 1.0, s);
  launch_colratio_batched(ratios.p, (int)sys.size(), max_m, s);
}

void Batch::run_factor(cudaStream_t s) {
  {
    PhaseScope ps(prof, PH_CONVERT, s);
    launch_ew2d_batched<double, float>(cv_in.p, (int)cv_in.h.size(), t_in, false, s);
  }
  for (auto &g : groups) run_path(prof, g->fused32, 0, info.p, s);
  launch_ew2d_batched<float, double>(cv_x0.p, (int)cv_x0.h.size(), t_x0, false, s);
  residuals(s);
}

void Batch::run_sweep(cudaStream_t s) {
  launch_ew2d_batched<double, float>(cv_res.p, (int)cv_res.h.size(), t_res, false, s);
  for (auto &g : groups) run_path(prof, g->apply32, 0, nullptr, s);
  launch_ew2d_batched<float, double>(add_y.p, (int)add_y.h.size(), t_x0, true, s);
  residuals(s);
}

int Batch::check_info(cudaStream_t s, int *failed) {
  std::vector<int> h(n_info);
  HODLR_CUDA_TRY(cudaMemcpyAsync(h.data(), info.p, sizeof(int) * n_info, cudaMemcpyDeviceToHost, s));
  HODLR_CUDA_TRY(cudaStreamSynchronize(s));
  if (failed) *failed = -1;
  for (size_t k = 0; k < sys.size(); ++k) {
    const int nl = (int)sys[k]->tree.leaves.size();
    for (int i = 0; i < sys[k]->n_info; ++i) {
      const int v = h[info_off[k] + i];
      if (v == 0) continue;
      if (failed) *failed = (int)k;
      return i < nl ? v : 100000 + v;
    }
  }
  return 0;
}

double Batch::relres_read(cudaStream_t s, std::vector<double> *per_system) {
  const int n_rr = rr_off.back() + sys.back()->m;
  std::vector<double> h(n_rr);
  HODLR_CUDA_TRY(cudaMemcpyAsync(h.data(), rr.p, sizeof(double) * n_rr, cudaMemcpyDeviceToHost, s));
  HODLR_CUDA_TRY(cudaStreamSynchronize(s));
  double mx = 0.0;
  if (per_system) per_system->assign(sys.size(), 0.0);
  for (size_t k = 0; k < sys.size(); ++k) {
    double mk = 0.0;
    for (int c = 0; c < sys[k]->m; ++c) {
      const double v = h[rr_off[k] + c];
      mk = std::max(mk, std::isnan(v) ? INFINITY : v);
    }
    if (per_system) (*per_system)[k] = mk;
    mx = std::max(mx, mk);
  }
  return mx;
}

}  // namespace hodlr
