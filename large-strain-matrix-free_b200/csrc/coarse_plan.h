// Work distribution of the coarse-level solver: a level small enough that
// one CTA per SM takes all its cells (one batch per warp, and their records
// in shared memory) is solved by
// one cooperative kernel (coarse_kernels.cuh).  Every CTA keeps a compact
// group of cells, sums their contributions to its nodes in shared memory and
// exchanges only the sums of the nodes it shares with other CTAs.
#pragma once
#include <cuda_runtime.h>

#include "lsmf_internal.h"

namespace lsmf {

constexpr int COARSE_THREADS = 256;  // threads of a CTA
constexpr int COARSE_MAX_WARPS = COARSE_THREADS / 32;

// sizes that depend on the kernel (degree, number type, variant)
struct CoarseShape {
  int cells = 0;           // cells of a CTA
  int batch = 0;           // cells of a warp
  size_t unit_bytes = 0;   // shared memory of a working warp
  size_t out_offset = 0;   // ... and where its cells' results lie in it (bytes)
};

// Per CTA (rows of fixed length): its cells (a negative entry -1 - c repeats
// cell c without contributing), the local node of every cell node, the
// global nodes (2 * node + 1 for the CTA that stores the node), the exchange
// slot of a shared node (else -1), the shared-memory places of a node's (at
// most 8) contributions, and its items: the slots of the other CTAs' sums of
// its shared nodes, each with its place in the receive array.  The sums of a
// shared node stand there in CTA order, the CTA's own among them: every CTA
// adds the same sums in the same order, so its copies of a shared node's
// values stay bitwise equal to the others'.  Local nodes are ordered by the
// number of CTAs that share them, then of contributions, both falling.
struct CoarsePlan {
  bool usable = false;
  int n_cta = 0, warps = 0, cells_per_cta = 0, max_nodes = 0, max_items = 0, max_sums = 0, n_slots = 0, packets = 0;
  size_t unit_bytes = 0, smem = 0;
  // device arrays, parts of one buffer
  const int *counts = nullptr;           // [cta][4]: cells, nodes, items, 0
  const int *cells = nullptr;            // [cta][cells_per_cta]
  const unsigned *nodes = nullptr;       // [cta][max_nodes]
  const int *send = nullptr;             // [cta][max_nodes]
  const int *item_slot = nullptr;        // [cta][max_items]
  const uint16_t *lid = nullptr;         // [cta][cells_per_cta][NN]
  const uint16_t *contrib = nullptr;     // [cta][max_nodes][8], element offsets, 0xffff: none
  const uint16_t *item_place = nullptr;  // [cta][max_items]
  const uint16_t *first = nullptr;       // [cta][max_nodes]: first sum of a shared node in the receive array
  const uint8_t *sums = nullptr;         // [cta][max_nodes]: number of its sums | place of the own one << 4 (0: not shared)
  DevBuf<uint8_t> lists;
  mutable DevBuf<ulonglong2> xbuf;  // two exchange buffers of n_slots * packets, two of 8 * n_cta (reductions)
};

// The CG of an eigenvalue estimate: mean of the start vector's integers i mod
// 11, tolerance max(tol_abs, tol_rel * initial residual), and where its
// history (alpha, beta, squared residual per iteration) and iteration count go
struct CoarseEig {
  double mean = 0, tol_abs = 0, tol_rel = 0;
  int max_it = 0;
  double *alpha = nullptr, *beta = nullptr, *res2 = nullptr;
  int *its = nullptr;
};

// shared memory of a CTA beside its units
size_t coarse_tail_bytes(int max_nodes, int max_sums, size_t elem);

// Build the plan for op's level (plan.usable says whether the solver can take
// it: the smallest number of working warps whose cells fit on `sms` SMs and
// whose records fit in smem_limit bytes).
lsmf_status build_coarse_plan(const lsmf_op *op, int sms, size_t smem_limit, CoarsePlan &plan);

}  // namespace lsmf
