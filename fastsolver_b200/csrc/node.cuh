// node.cuh -- launcher of the capacitance (node) factorization (node.cu).
#pragma once
#include "common.cuh"

namespace hodlr {

// Largest capacitance system kept in shared memory (s = r or 2r).
constexpr int kMaxNodeS = 144;

// One CTA per node: S = I - V1Tu1 V0Tu0, S^{-1} (Gauss-Jordan, partial
// pivoting) and the node's solve matrix M; info[task.info_slot] = 0 or the
// first zero pivot (1-based).  max_s / max_r: the largest system (r0, form 1:
// r0 + r1; at most kMaxNodeS) and the largest of r0 and r1 in the launch.
template <typename TW, typename TE>
void launch_node_factor(const NodeTask<TW, TE> *tasks, int count, int max_s, int max_r, int form,
                        int *info, cudaStream_t s);

}  // namespace hodlr
