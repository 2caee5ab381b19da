// Launchers of the matrix-free tangent operator (cache, vmult, diagonal,
// Jacobi) and the small element-wise kernels around the cell loops.  The
// cell-loop kernels themselves are templates in op_kernels.cuh, compiled per
// degree and precision in op_p<P>_<f64|f32>.cu and reached through
// ops_for().
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

#include "cell_kernels.cuh"
#include "lsmf_internal.h"
#include "op_dispatch.h"

namespace lsmf {

namespace {

// ------------------------------------------------------ element-wise ops
// dst += src on the constrained dofs.  No cell loop adds to those, so one
// launched as its programmatic dependent may start at once.
template <typename T>
__global__ void constrained_add_kernel(T *dst, const T *src, const int *idx, int n) {
  asm volatile("griddepcontrol.launch_dependents;");
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int k = idx[i];
    dst[k] += src[k];
  }
}
// dst = src on the constrained dofs and zero elsewhere, for the dofs first ..
// last - 1: the zeroing and the identity rows of a vmult in one launch (the
// cell loop adds nothing to constrained dofs).  Every thread writes aligned
// 16-byte groups of dst; the ends of the range are written value by value.
// It lets a cell loop launched as its programmatic dependent start at once.
template <typename T>
__global__ void identity_rows_kernel(T *__restrict__ dst, const T *__restrict__ src, const uint8_t *__restrict__ cmask,
                                     size_t first, size_t last) {
  asm volatile("griddepcontrol.launch_dependents;");
  constexpr int W = 16 / sizeof(T);
  const size_t shift = ((size_t)dst / sizeof(T)) % W;  // dst + i is aligned where (i + shift) % W == 0
  const size_t g0 = (first + shift) / W, g1 = (last + shift + W - 1) / W;
  for (size_t g = g0 + blockIdx.x * (size_t)blockDim.x + threadIdx.x; g < g1; g += (size_t)gridDim.x * blockDim.x) {
    const size_t a = g * W < shift ? 0 : g * W - shift, b = g * W + W - shift;
    if (g * W >= first + shift && b <= last) {
      alignas(16) T v[W];
#pragma unroll
      for (int k = 0; k < W; ++k) v[k] = __ldg(cmask + a + k) ? src[a + k] : T(0);
      *(float4 *)(dst + a) = *(const float4 *)v;
    } else {
      for (size_t i = a > first ? a : first; i < (b < last ? b : last); ++i) dst[i] = cmask[i] ? src[i] : T(0);
    }
  }
}
template <typename T>
__global__ void constrained_set_kernel(T *dst, const int *idx, int n, T val) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[idx[i]] = val;
}
template <typename T>
__global__ void invert_kernel(T *inv, const T *d, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    inv[i] = T(1) / d[i];
}
template <typename T>
__global__ void scaled_mul_kernel(T *dst, const T *a, const T *b, T s, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    dst[i] = s * a[i] * b[i];
}

int g_num_sms = 0;
int num_sms() {
  if (!g_num_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 148;
  }
  return g_num_sms;
}

const OpsTable *table_of(const lsmf_op *op) {
  const Level &L = op->L();
  const OpsTable *t = L.q == L.p + 1 ? ops_for(L.p, op->precision == LSMF_FP32) : nullptr;
  if (!t) set_error("unsupported (degree, n_q_points_1d): only q = p + 1, p = 1..4");
  return t;
}

lsmf_status identity_rows(const lsmf_op *op, void *dst, const void *src, size_t first, size_t last, cudaStream_t st) {
  if (last <= first) return LSMF_OK;
  const size_t per = 16 / op->elem(), groups = (last - first + per - 1) / per + 1;
  const int g = (int)std::min<size_t>((groups + 255) / 256, (size_t)8 * num_sms());
  const uint8_t *cm = op->L().d_cmask.ptr;
  if (op->precision == LSMF_FP64)
    identity_rows_kernel<double><<<g, 256, 0, st>>>((double *)dst, (const double *)src, cm, first, last);
  else
    identity_rows_kernel<float><<<g, 256, 0, st>>>((float *)dst, (const float *)src, cm, first, last);
  LSMF_CUDA(cudaGetLastError());
  return LSMF_OK;
}

// node-sum scatter: dst (+)= the sum over the node's cells, in increasing
// cell order, of the node's slot in the per-cell buffer (a fixed order: the
// result is the same from call to call), and with `rows` the identity rows:
// the slots of constrained dofs hold zeros, src is added there (as a launch of
// their own after this one the rows cost 1-2 us on small levels and 8 of 365
// us at 60^3 Q2 tensor4 FP64)
template <typename T>
__global__ void node_sum_kernel(T *dst, const T *__restrict__ buf, const int *__restrict__ off,
                                const int *__restrict__ ent, int n_nodes, int add, const T *__restrict__ src,
                                const uint8_t *__restrict__ cmask, int rows) {
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < n_nodes; n += gridDim.x * blockDim.x) {
    T s[3] = {T(0), T(0), T(0)};
    const int e1 = __ldg(off + n + 1);
    for (int e = __ldg(off + n); e < e1; ++e) {
      const int b = __ldg(ent + e);
#pragma unroll
      for (int i = 0; i < 3; ++i) s[i] += buf[b + i];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const size_t d = 3 * (size_t)n + i;
      if (rows && __ldg(cmask + d)) s[i] += __ldg(src + d);
      dst[d] = add ? dst[d] + s[i] : s[i];
    }
  }
}

}  // namespace

int record_components(int caching) {
  if (caching == LSMF_CACHE_TENSOR4) return variant_ncomp(VAR_TENSOR4);
  if (caching == LSMF_CACHE_TENSOR2) return variant_ncomp(VAR_TENSOR2);
  if (caching == LSMF_CACHE_SCALAR_REFERENTIAL) return variant_ncomp(VAR_SCALAR_REF);
  if (caching == LSMF_CACHE_TENSOR4_NS) return variant_ncomp(VAR_TENSOR4_NS);
  return variant_ncomp(VAR_SCALAR_F1);
}

// metric 9 + tau/J 6 + the full 6x6 C; metric 9 + the full 9x9 dP/dF
int table_components(int caching) {
  if (caching == LSMF_CACHE_TENSOR4) return 9 + 6 + 36;
  if (caching == LSMF_CACHE_TENSOR4_NS) return 9 + 81;
  return record_components(caching);
}

int cells_per_batch(int p, lsmf_precision precision) {
  const int halves = precision == LSMF_FP32 ? 2 : 1;
  return 32 / ((p + 1) * (p + 1)) * halves;
}

size_t record_index(const lsmf_op *op, int cell, int comp, int q) {
  auto at = [&](auto layout) -> size_t {
    using RL = decltype(layout);
    return RL::base(cell, op->batch_elems) + (size_t)comp * RL::CS + RL::q_off(q, op->slice_elems);
  };
  const bool f = op->precision == LSMF_FP32;
  switch (op->L().p) {
    case 1: return f ? at(RecLayout<1, 2, 2>{}) : at(RecLayout<1, 2, 1>{});
    case 2: return f ? at(RecLayout<2, 3, 2>{}) : at(RecLayout<2, 3, 1>{});
    case 3: return f ? at(RecLayout<3, 4, 2>{}) : at(RecLayout<3, 4, 1>{});
    default: return f ? at(RecLayout<4, 5, 2>{}) : at(RecLayout<4, 5, 1>{});
  }
}

lsmf_status launch_cache(lsmf_op *op) {
  const OpsTable *t = table_of(op);
  if (!t) return LSMF_ERR_UNSUPPORTED;
  LSMF_CUDA(cudaMemsetAsync(op->d_flag.ptr, 0, sizeof(int), op->stream));
  return t->cache(op);
}

// Run a cell loop f(range) over all cells with atomic scatter, or, with the
// colour8 scatter option, once per lattice colour in the fixed order 0..7
// (the launches are ordered on the operator's stream, so every node sums
// its cell contributions in the same order on every call).
template <typename F>
lsmf_status for_cell_ranges(const Level &L, int scatter, F &&f) {
  // the node-sum scatter serves the full vmult cell loop; every other cell
  // loop of a node-sum operator runs the (equally deterministic) colours
  if (scatter != LSMF_SCATTER_ATOMIC) {
    for (int c = 0; c < 8; ++c) {
      CellRange r;
      r.cells = L.d_colour_cells.ptr + L.colour_off[c];
      r.n_list = L.colour_off[c + 1] - L.colour_off[c];
      r.plain = true;
      if (r.n_list > 0) LSMF_TRY(f(r));
    }
    return LSMF_OK;
  }
  return f(CellRange{});
}

// The cell ranges of a vmult cell loop (the node-sum path's production loops
// go through apply_node_sum).  The production kernel of a colour8 operator
// takes whole batches of cells, in groups that share no
// node, so that its records are read as contiguous slices; the basic kernel
// takes the cells of the lattice colours.
template <typename F>
static lsmf_status for_apply_ranges(const lsmf_op *op, unsigned mask, F &&f) {
  const unsigned all = LSMF_MASK_RW | LSMF_MASK_SF | LSMF_MASK_QD;
  const bool production = !op->basic && (mask & all) == all && !(mask & MASK_INHOM_BIT);
  if (op->scatter != LSMF_SCATTER_COLOUR8 || !production) return for_cell_ranges(op->L(), op->scatter, f);
  const Level::BatchGroups &g = op->L().batch_groups[op->precision == LSMF_FP32];
  for (size_t c = 0; c + 1 < g.off.size(); ++c) {
    CellRange r;
    r.cells = g.list.ptr + g.off[c];
    r.n_list = g.off[c + 1] - g.off[c];
    r.plain = r.batches = true;
    r.dependent = c > 0;
    LSMF_TRY(f(r));
  }
  return LSMF_OK;
}

// Groups of the level's batches: each batch, in order, joins the first group
// none of whose batches has one of its nodes (a bit per group and node, 64
// groups at a time; 8 to 12 groups on the meshes in use).
static lsmf_status build_batch_groups(Level &L, int B, Level::BatchGroups &g) {
  const int nb = (L.n_cells + B - 1) / B, ncn = L.ncn();
  std::vector<std::vector<uint64_t>> used;
  std::vector<int> group(nb);
  int n_groups = 0;
  for (int b = 0; b < nb; ++b) {
    const int *n0 = &L.cell_nodes[(size_t)b * B * ncn], *n1 = n0 + (size_t)std::min(B, L.n_cells - b * B) * ncn;
    for (size_t l = 0;; ++l) {
      if (l == used.size()) used.emplace_back(L.n_nodes, 0);
      uint64_t taken = 0;
      for (const int *n = n0; n < n1; ++n) taken |= used[l][*n];
      if (taken == ~0ull) continue;
      const int bit = __builtin_ctzll(~taken);
      for (const int *n = n0; n < n1; ++n) used[l][*n] |= 1ull << bit;
      group[b] = 64 * (int)l + bit;
      break;
    }
    n_groups = std::max(n_groups, group[b] + 1);
  }
  std::vector<int> off(n_groups + 1, 0), list(nb);
  for (int b = 0; b < nb; ++b) ++off[group[b] + 1];
  for (int c = 0; c < n_groups; ++c) off[c + 1] += off[c];
  std::vector<int> pos(off.begin(), off.end() - 1);
  for (int b = 0; b < nb; ++b) list[pos[group[b]]++] = b;
  LSMF_TRY(g.list.upload(list.data(), list.size()));
  g.off = off;
  return LSMF_OK;
}

// the node-sum path applies: the operator asks for it and the launch is the
// full production cell loop
static bool node_sum_path(const lsmf_op *op, unsigned mask) {
  const unsigned all = LSMF_MASK_RW | LSMF_MASK_SF | LSMF_MASK_QD;
  return op->scatter == LSMF_SCATTER_NODESUM && !op->basic && (mask & all) == all && !(mask & MASK_INHOM_BIT);
}

// cell loop into the operator's cell buffer, then dst (+)= node sums
static lsmf_status apply_node_sum(const lsmf_op *op, const OpsTable *t, void *dst, const void *src, unsigned mask,
                                  bool add, bool rows) {
  const Level &L = op->L();
  if (!op->d_cellbuf.ptr || !L.d_node_cell_off.ptr) {
    set_error("node-sum scatter selected without its buffers");
    return LSMF_ERR_NOT_INITIALIZED;
  }
  CellRange r;
  r.cellbuf = op->d_cellbuf.ptr;
  LSMF_TRY(t->apply(op, dst, src, mask, r));
  const int g = std::min((L.n_nodes + 255) / 256, 8 * num_sms());
  auto sum = [&](auto zero) {
    using T = decltype(zero);
    node_sum_kernel<T><<<g, 256, 0, op->stream>>>((T *)dst, (const T *)op->d_cellbuf.ptr, L.d_node_cell_off.ptr,
                                                  L.d_node_cell_ent.ptr, L.n_nodes, add, (const T *)src, L.d_cmask.ptr, rows);
  };
  if (op->precision == LSMF_FP64) sum(0.0);
  else sum(0.0f);
  LSMF_CUDA(cudaGetLastError());
  return LSMF_OK;
}

lsmf_status set_scatter_mode(lsmf_op *op, int mode) {
  if (mode != LSMF_SCATTER_ATOMIC && mode != LSMF_SCATTER_COLOUR8 && mode != LSMF_SCATTER_NODESUM) {
    set_error("scatter must be 0 (atomic), 1 (colour8) or 2 (nodesum)");
    return LSMF_ERR_INVALID_ARG;
  }
  if (mode == LSMF_SCATTER_COLOUR8) {
    Level::BatchGroups &g = op->L().batch_groups[op->precision == LSMF_FP32];
    if (g.off.empty()) LSMF_TRY(build_batch_groups(op->L(), cells_per_batch(op->L().p, op->precision), g));
  }
  if (mode == LSMF_SCATTER_NODESUM) {
    Level &L = op->L();
    const int ncn = L.ncn();
    if ((double)L.n_cells * ncn * 3 > 2147483647.0) {
      set_error("the node-sum scatter indexes its cell buffer with 32-bit offsets; this level is too large");
      return LSMF_ERR_UNSUPPORTED;
    }
    if (!L.d_node_cell_off.ptr) {
      // counting sort of the (cell, local node) slots by node, cells in
      // increasing order within a node
      std::vector<int> off(L.n_nodes + 1, 0), ent((size_t)L.n_cells * ncn);
      for (size_t k = 0; k < ent.size(); ++k) ++off[L.cell_nodes[k] + 1];
      for (int n = 0; n < L.n_nodes; ++n) off[n + 1] += off[n];
      std::vector<int> pos(off.begin(), off.end() - 1);
      for (int c = 0; c < L.n_cells; ++c)
        for (int a = 0; a < ncn; ++a) ent[pos[L.cell_nodes[(size_t)c * ncn + a]]++] = (c * ncn + a) * 3;
      LSMF_TRY(L.d_node_cell_off.upload(off.data(), off.size()));
      LSMF_TRY(L.d_node_cell_ent.upload(ent.data(), ent.size()));
    }
    LSMF_TRY(op->d_cellbuf.alloc((size_t)L.n_cells * ncn * 3 * op->elem()));
  }
  op->scatter = mode;
  return LSMF_OK;
}

// Chunks of an operator's atomic-scatter cell loop: the option, or the
// measured choice (vmult time on B200 against one launch, at 60^3 Q2, 96^3
// Q1, 40^3 Q3 and 36^3 Q4): from 131,072 cells 8 for the referential variants
// (scalar_referential -3 %, tensor4_ns -2 %), 4 for the others (tensor4
// -0.5 %, scalar -2 %; degree 4 -2 to -4 %), from 32,768 cells 2; tensor2 and
// fewer cells run in one launch (60^3 Q2 tensor2 229 us against 235 in 4).
static int chunk_count(const lsmf_op *op) {
  if (op->chunks > 0) return op->chunks;
  const int n = op->L().n_cells;
  if (op->caching == LSMF_CACHE_TENSOR2 || n < 32768) return 1;
  if (n < 131072) return 2;
  return op->caching == LSMF_CACHE_TENSOR4_NS || op->caching == LSMF_CACHE_SCALAR_REFERENTIAL ? 8 : 4;
}

// The operator's plan for k chunks (*out = nullptr where it does not apply:
// k < 2, fewer than 1024 cells per chunk, or a chunk whose cells reach past
// the next chunk's node range).  Cells and nodes are numbered z-slowest, so
// contiguous cell chunks touch nearly contiguous node ranges; chunk c owns
// the nodes from the lowest one its cells touch up to the next chunk's.
static lsmf_status chunk_plan(const lsmf_op *op, int k, const ChunkPlan **out) {
  *out = nullptr;
  if (k < 2) return LSMF_OK;
  if (op->chunk_plan && op->chunk_plan->requested == k) {
    if (op->chunk_plan->k) *out = op->chunk_plan.get();
    return LSMF_OK;
  }
  auto plan = std::make_unique<ChunkPlan>();
  plan->requested = k;
  const Level &L = op->L();
  const int ncn = L.ncn();
  bool ok = k <= 8 && L.n_cells >= 1024 * k;
  if (ok) {
    plan->cell0.resize(k + 1);
    plan->node0.resize(k + 1);
    std::vector<int> nmax(k);
    // chunks start at whole batches of the cell records
    const int B = cells_per_batch(L.p, op->precision);
    for (int c = 0; c <= k; ++c) plan->cell0[c] = c == k ? L.n_cells : (int)((long long)L.n_cells * c / k) / B * B;
    for (int c = 0; c < k; ++c) {
      int lo = L.n_nodes, hi = -1;
      for (size_t i = (size_t)plan->cell0[c] * ncn; i < (size_t)plan->cell0[c + 1] * ncn; ++i) {
        lo = std::min(lo, L.cell_nodes[i]);
        hi = std::max(hi, L.cell_nodes[i]);
      }
      plan->node0[c] = c == 0 ? 0 : lo;
      nmax[c] = hi;
    }
    plan->node0[k] = L.n_nodes;
    for (int c = 0; c < k && ok; ++c) {
      ok = plan->node0[c] <= plan->node0[c + 1];
      if (c + 2 <= k) ok = ok && nmax[c] < plan->node0[c + 2];
    }
  }
  if (ok) {
    for (int c = 0; c < k; ++c) {
      LSMF_CUDA(cudaStreamCreateWithFlags(&plan->stream[c], cudaStreamNonBlocking));
      LSMF_CUDA(cudaEventCreateWithFlags(&plan->zero[c], cudaEventDisableTiming));
      LSMF_CUDA(cudaEventCreateWithFlags(&plan->done[c], cudaEventDisableTiming));
    }
    LSMF_CUDA(cudaEventCreateWithFlags(&plan->fork, cudaEventDisableTiming));
    plan->k = k;
  }
  op->chunk_plan = std::move(plan);
  if (op->chunk_plan->k) *out = op->chunk_plan.get();
  return LSMF_OK;
}

// the chunked path applies: atomic scatter, fast kernels, the full cell loop
static bool chunkable(const lsmf_op *op, unsigned mask) {
  const unsigned all = LSMF_MASK_RW | LSMF_MASK_SF | LSMF_MASK_QD;
  return op->scatter == LSMF_SCATTER_ATOMIC && !op->basic && (mask & all) == all && !(mask & MASK_INHOM_BIT);
}

// chunks the operator's next full vmult cell loop runs in (1: one launch)
lsmf_status effective_chunks(const lsmf_op *op, int *k) {
  *k = 1;
  if (!chunkable(op, LSMF_MASK_RW | LSMF_MASK_SF | LSMF_MASK_QD)) return LSMF_OK;
  const ChunkPlan *cp = nullptr;
  LSMF_TRY(chunk_plan(op, chunk_count(op), &cp));
  if (cp) *k = cp->k;
  return LSMF_OK;
}


// The vmult over the plan's chunks, forked from and joined back into the
// operator's stream: chunk c zeroes its node range of dst (zero) and sets, or
// without it adds, the identity rows of the constrained dofs there, then runs its
// cells once chunk c + 1 has zeroed its range (its cells add into that
// range's first node layer).  The scatter skips constrained components, so
// the identity rows are never touched by another chunk.
static lsmf_status apply_chunked(const lsmf_op *op, const OpsTable *t, const ChunkPlan &cp, void *dst,
                                 const void *src, unsigned mask, bool zero) {
  const Level &L = op->L();
  const int g_max = 4 * num_sms();
  LSMF_CUDA(cudaEventRecord(cp.fork, op->stream));
  for (int c = 0; c < cp.k; ++c) {
    cudaStream_t st = cp.stream[c];
    LSMF_CUDA(cudaStreamWaitEvent(st, cp.fork, 0));
    const size_t d0 = 3 * (size_t)cp.node0[c], d1 = 3 * (size_t)cp.node0[c + 1];
    if (zero) {
      LSMF_TRY(identity_rows(op, dst, src, d0, d1, st));
    } else {
      // L.constrained is in increasing dof order
      const int a0 = (int)(std::lower_bound(L.constrained.begin(), L.constrained.end(), (int)d0) - L.constrained.begin());
      const int a1 = (int)(std::lower_bound(L.constrained.begin(), L.constrained.end(), (int)d1) - L.constrained.begin());
      const int nc = a1 - a0;
      if (nc > 0) {
        const int g = (nc + 255) / 256 < g_max ? (nc + 255) / 256 : g_max;
        if (op->precision == LSMF_FP64)
          constrained_add_kernel<double><<<g, 256, 0, st>>>((double *)dst, (const double *)src, L.d_constrained.ptr + a0, nc);
        else
          constrained_add_kernel<float><<<g, 256, 0, st>>>((float *)dst, (const float *)src, L.d_constrained.ptr + a0, nc);
        LSMF_CUDA(cudaGetLastError());
      }
    }
    LSMF_CUDA(cudaEventRecord(cp.zero[c], st));
  }
  for (int c = 0; c < cp.k; ++c) {
    if (c + 1 < cp.k) LSMF_CUDA(cudaStreamWaitEvent(cp.stream[c], cp.zero[c + 1], 0));
    CellRange r;
    r.first = cp.cell0[c];
    r.count = cp.cell0[c + 1] - cp.cell0[c];
    r.stream = cp.stream[c];
    LSMF_TRY(t->apply(op, dst, src, mask, r));
    LSMF_CUDA(cudaEventRecord(cp.done[c], cp.stream[c]));
  }
  for (int c = 0; c < cp.k; ++c) LSMF_CUDA(cudaStreamWaitEvent(op->stream, cp.done[c], 0));
  return LSMF_OK;
}

// identity rows on top of what dst holds: dst += src (mf_nh_operator.h:702-705)
static lsmf_status add_rows(const lsmf_op *op, void *dst, const void *src) {
  const Level &L = op->L();
  const int nc = (int)L.constrained.size();
  if (!nc) return LSMF_OK;
  const int g = (nc + 255) / 256 < 4 * num_sms() ? (nc + 255) / 256 : 4 * num_sms();
  if (op->precision == LSMF_FP64)
    constrained_add_kernel<double><<<g, 256, 0, op->stream>>>((double *)dst, (const double *)src, L.d_constrained.ptr, nc);
  else
    constrained_add_kernel<float><<<g, 256, 0, op->stream>>>((float *)dst, (const float *)src, L.d_constrained.ptr, nc);
  LSMF_CUDA(cudaGetLastError());
  return LSMF_OK;
}

lsmf_status launch_apply(const lsmf_op *op, void *dst, const void *src, unsigned mask, bool add) {
  const Level &L = op->L();
  const OpsTable *t = table_of(op);
  if (!t) return LSMF_ERR_UNSUPPORTED;
  const size_t n = (size_t)L.n_dofs();
  // (the node-sum path applies to full cell loops: gather and scatter, rows too)
  if (node_sum_path(op, mask)) return apply_node_sum(op, t, dst, src, mask, add || !(mask & LSMF_MASK_ZERO), true);
  if (chunkable(op, mask)) {
    const ChunkPlan *cp = nullptr;
    LSMF_TRY(chunk_plan(op, chunk_count(op), &cp));
    if (cp) return apply_chunked(op, t, *cp, dst, src, mask, !add && (mask & LSMF_MASK_ZERO));
  }
  const bool zero = !add && (mask & LSMF_MASK_ZERO), rows = mask & LSMF_MASK_RW;
  // the rows come first: the cell loop adds nothing to constrained dofs
  // (mf_nh_operator.h:702-705) and, as the dependent of the rows' launch,
  // hides its own start behind it (vmult_add of 8^3 Q2 tensor4 FP64 in a
  // graph: 6.09 us with the rows last, 5.56 us)
  bool dependent = rows && (zero || !L.constrained.empty());
  if (zero && rows) LSMF_TRY(identity_rows(op, dst, src, 0, n, op->stream));
  else if (zero) LSMF_CUDA(cudaMemsetAsync(dst, 0, n * op->elem(), op->stream));
  else if (rows) LSMF_TRY(add_rows(op, dst, src));
  return for_apply_ranges(op, mask, [&](CellRange r) {
    // the scatter of the first launch has to wait for the rows, that of
    // every further group of batches for the group before (small levels
    // are bound by the launches: 16^3 Q2 has 12 groups)
    r.dependent = r.dependent || dependent;
    dependent = false;
    return t->apply(op, dst, src, mask, r);
  });
}

// Cell loop of a partitioned FP64 vmult with the interface exchange fused
// in (range.peer_*: the ghost nodes' values are read from, and their
// contributions added to, the neighbour part's vectors), then the identity
// rows of the part's owned constrained dofs d_con[0 .. n_con).  dst is not
// zeroed here: the caller orders the zeroing of this part's and of the
// neighbour's dst before the launch.
lsmf_status launch_apply_peer(const lsmf_op *op, double *dst, const double *src, const CellRange &range,
                              const int *d_con, int n_con) {
  const OpsTable *t = table_of(op);
  if (!t) return LSMF_ERR_UNSUPPORTED;
  if (op->precision != LSMF_FP64 || op->basic || op->scatter != LSMF_SCATTER_ATOMIC || !range.peer_nodes) {
    set_error("the fused interface exchange needs an FP64 operator with the fast kernel and atomic scatter");
    return LSMF_ERR_INVALID_ARG;
  }
  LSMF_TRY(t->apply(op, dst, src, LSMF_MASK_RW | LSMF_MASK_SF | LSMF_MASK_QD, range));
  if (n_con) {
    const int g = (n_con + 255) / 256 < 4 * num_sms() ? (n_con + 255) / 256 : 4 * num_sms();
    constrained_add_kernel<double><<<g, 256, 0, op->stream>>>(dst, src, d_con, n_con);
    LSMF_CUDA(cudaGetLastError());
  }
  return LSMF_OK;
}

lsmf_status launch_apply_cells(const lsmf_op *op, void *dst, const void *src) {
  const OpsTable *t = table_of(op);
  if (!t) return LSMF_ERR_UNSUPPORTED;
  const unsigned mask = LSMF_MASK_RW | LSMF_MASK_SF | LSMF_MASK_QD;
  if (node_sum_path(op, mask)) return apply_node_sum(op, t, dst, src, mask, true, false);
  if (chunkable(op, mask)) {
    // the chunks' cell loops only, concurrent (nothing to zero)
    const ChunkPlan *cp = nullptr;
    LSMF_TRY(chunk_plan(op, chunk_count(op), &cp));
    if (cp) {
      LSMF_CUDA(cudaEventRecord(cp->fork, op->stream));
      for (int c = 0; c < cp->k; ++c) {
        LSMF_CUDA(cudaStreamWaitEvent(cp->stream[c], cp->fork, 0));
        CellRange r;
        r.first = cp->cell0[c];
        r.count = cp->cell0[c + 1] - cp->cell0[c];
        r.stream = cp->stream[c];
        LSMF_TRY(t->apply(op, dst, src, mask, r));
        LSMF_CUDA(cudaEventRecord(cp->done[c], cp->stream[c]));
      }
      for (int c = 0; c < cp->k; ++c) LSMF_CUDA(cudaStreamWaitEvent(op->stream, cp->done[c], 0));
      return LSMF_OK;
    }
  }
  return for_apply_ranges(op, mask, [&](CellRange r) { return t->apply(op, dst, src, mask, r); });
}

lsmf_status launch_coarse_cheb(const lsmf_op *op, const CoarsePlan &plan, void *x, const void *b, double theta,
                               double delta, int degree) {
  const OpsTable *t = table_of(op);
  return t ? t->coarse_cheb(op, plan, x, b, theta, delta, degree) : LSMF_ERR_UNSUPPORTED;
}

lsmf_status launch_coarse_eig(const lsmf_op *op, const CoarsePlan &plan, const CoarseEig &e) {
  const OpsTable *t = table_of(op);
  return t ? t->coarse_eig(op, plan, e) : LSMF_ERR_UNSUPPORTED;
}

// K g over the constrained columns: gather without zeroing, scatter skipping
// constrained rows (dst zeroed first, no identity rows)
lsmf_status launch_apply_inhomogeneous(const lsmf_op *op, void *dst, const void *g) {
  const Level &L = op->L();
  const OpsTable *t = table_of(op);
  if (!t) return LSMF_ERR_UNSUPPORTED;
  LSMF_CUDA(cudaMemsetAsync(dst, 0, (size_t)L.n_dofs() * op->elem(), op->stream));
  const unsigned mask = LSMF_MASK_RW | LSMF_MASK_SF | LSMF_MASK_QD | MASK_INHOM_BIT;
  return for_cell_ranges(L, op->scatter, [&](CellRange r) { return t->apply(op, dst, g, mask, r); });
}

lsmf_status launch_diagonal(lsmf_op *op) {
  const Level &L = op->L();
  const OpsTable *t = table_of(op);
  if (!t) return LSMF_ERR_UNSUPPORTED;
  const size_t n = (size_t)L.n_dofs();
  LSMF_CUDA(cudaMemsetAsync(op->d_diag.ptr, 0, n * op->elem(), op->stream));
  LSMF_TRY(for_cell_ranges(L, op->scatter, [&](CellRange r) { return t->diag(op, op->d_diag.ptr, r); }));
  const int nc = (int)L.constrained.size();
  const int g = 4 * num_sms();
  if (op->precision == LSMF_FP64) {
    if (nc) constrained_set_kernel<double><<<g, 256, 0, op->stream>>>((double *)op->d_diag.ptr, L.d_constrained.ptr, nc, 1.0);
    invert_kernel<double><<<g, 256, 0, op->stream>>>((double *)op->d_inv_diag.ptr, (const double *)op->d_diag.ptr, n);
  } else {
    if (nc) constrained_set_kernel<float><<<g, 256, 0, op->stream>>>((float *)op->d_diag.ptr, L.d_constrained.ptr, nc, 1.0f);
    invert_kernel<float><<<g, 256, 0, op->stream>>>((float *)op->d_inv_diag.ptr, (const float *)op->d_diag.ptr, n);
  }
  LSMF_CUDA(cudaGetLastError());
  return LSMF_OK;
}

lsmf_status launch_jacobi(const lsmf_op *op, void *dst, const void *src, double omega) {
  const size_t n = (size_t)op->L().n_dofs();
  const int g = 4 * num_sms();
  if (op->precision == LSMF_FP64)
    scaled_mul_kernel<double><<<g, 256, 0, op->stream>>>((double *)dst, (const double *)op->d_inv_diag.ptr,
                                                         (const double *)src, omega, n);
  else
    scaled_mul_kernel<float><<<g, 256, 0, op->stream>>>((float *)dst, (const float *)op->d_inv_diag.ptr,
                                                        (const float *)src, (float)omega, n);
  LSMF_CUDA(cudaGetLastError());
  return LSMF_OK;
}

}  // namespace lsmf
