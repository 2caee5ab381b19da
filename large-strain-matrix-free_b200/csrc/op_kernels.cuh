// sm_100a kernel templates of the matrix-free tangent operator, shared by
// the per-degree / per-precision instantiation units op_p<P>_<f64|f32>.cu:
//   cache_kernel       NeoHookOperator::cache + Eulerian MatrixFree metric
//   apply_kernel       NeoHookOperator::vmult_add cell loop, basic form with
//                      the MFMask stage switches
//   apply_line_kernel  the production vmult cell loop
//   diagonal_kernel    NeoHookOperator::compute_diagonal
// Every cell loop runs either over all cells with atomic scatter, or over
// one colour of the lattice (a list of cells no two of which share a node)
// with plain read-modify-write scatter; the host launches the 8 colours in
// order for a bit-reproducible result.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>

#include "cell_kernels.cuh"
#include "lsmf_internal.h"
#include "coarse_plan.h"
#include "op_dispatch.h"
#include "pair.cuh"

namespace lsmf {

namespace {

template <typename T>
struct KArgs {
  const int *cell_nodes;
  int n_cells;
  int slice_elems, batch_elems;  // record layout (RecLayout)
  int ring;              // slices of the bulk-copy ring
  int ref_per_cell;      // scalar caching: reference inverse Jacobian once per cell
  T *table;              // cache records (written by cache, read by apply/diag)
  const T *src;
  T *dst;
  const T *u;            // displacement (operator precision)
  const double *X;       // reference coordinates
  const double *mu;      // per cell
  double nu;
  int *flag;             // device error word
  unsigned mask;
  int wait_tries;        // try_wait calls before a bulk-copy wait gives up
  int prefetch;          // plain loads: L1 prefetch of the records (0 off, 1 this unit, 2 the next unit)
  const int *cells;      // cell list of one colour (nullptr: all n_cells cells)
  int n_batches;         // cells lists this many batches of the n_cells cells (production vmult)
  int plain;             // scatter with plain adds (colour launches) instead of atomics
  T *cellbuf;            // node-sum scatter: per-cell results [cell][local node][component]
  // fused interface exchange (SC_PEER): the neighbour part's vectors, read
  // and added to for the nodes with PEER_BIT in cell_nodes
  const T *psrc;
  T *pdst;
  const T *pu;
  int cell0;             // first cell of a contiguous chunk (cell list absent)
};

// cell of list entry i
template <typename T>
__device__ __forceinline__ int cell_of(const KArgs<T> &a, int i) { return a.cells ? __ldg(a.cells + i) : a.cell0 + i; }
template <typename T>
__device__ __forceinline__ void scatter_add(T *p, T v, bool plain) {
  if (plain) *p += v;
  else atomicAdd(p, v);
}

template <int P, int Q, typename T>
__device__ __forceinline__ void load_tables(const Tab<P, Q> &tab, T *sN, T *sD) {
  constexpr int N1 = P + 1;
  for (int i = threadIdx.x; i < Q * N1; i += blockDim.x) {
    sN[i] = T(tab.N[i / N1][i % N1]);
    sD[i] = T(tab.D[i / N1][i % N1]);
  }
  __syncthreads();
}

template <typename T>
__device__ __forceinline__ void material(double mu_d, double nu, T &mu, T &lambda, T &kappa) {
  // material.h:82-94
  mu = T(mu_d);
  lambda = T((2.0 * mu_d * nu) / (1.0 - 2.0 * nu));
  kappa = T((2.0 * mu_d * (1.0 + nu)) / (3.0 * (1.0 - 2.0 * nu)));
}

// gather a 3-component field of a cell into V[c*NN + a]
template <int NN, typename TS, typename TD>
__device__ __forceinline__ void gather(const int *__restrict__ cn, const TS *__restrict__ vec, bool zero_constr,
                                       TD *V, int lane) {
  for (int a = lane; a < NN; a += 32) {
    const int packed = __ldg(cn + a);
    const int node = packed & NODE_MASK;
    const int cm = zero_constr ? (packed >> NODE_BITS) : 0;
    const TS *v = vec + 3 * (size_t)node;
    V[a] = (cm & 1) ? TD(0) : TD(__ldg(v));
    V[NN + a] = (cm & 2) ? TD(0) : TD(__ldg(v + 1));
    V[2 * NN + a] = (cm & 4) ? TD(0) : TD(__ldg(v + 2));
  }
  __syncwarp();
}

template <typename T>
__device__ __forceinline__ void atomic_add(T *a, T v) { atomicAdd(a, v); }

// ------------------------------------------------ bulk-copy (TMA) helpers
// One-dimensional cp.async.bulk from this GPU's global memory into the
// issuing CTA's own shared memory with mbarrier completion (no tensor map):
// the records of a warp's cells are one contiguous, 16-byte aligned block.
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint64_t evict_first_policy() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar, uint64_t pol) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(pol)
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait: try_wait suspends for a hardware time slice per call, so
// 2^22 calls are seconds; a wait that runs out reports failure instead of
// spinning forever
constexpr int WAIT_TRIES_DEFAULT = 1 << 22;
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, int tries = WAIT_TRIES_DEFAULT) {
  for (int i = 0; i < tries; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// device error word bits: det F <= 0 at a point (cache), a bounded wait
// ran out, a kernel found less dynamic shared memory than its layout needs
// (it returned without touching memory)
constexpr int FLAG_DETF = 1, FLAG_TIMEOUT = 2, FLAG_SMEM = 4;
// Dynamic shared memory of a launch against what the kernel's layout needs
// (bytes, uniform over the grid).  The host computes the size of the kernels
// whose layout depends on run-time values; where it gives them less, they set
// the error word and touch no shared memory.
__device__ __forceinline__ bool smem_short(size_t need, int *flag) {
  uint32_t have;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(have));
  if (have >= need) return false;
  if (threadIdx.x == 0) atomicOr(flag, FLAG_SMEM);
  return true;
}
// internal stage bit: gather constrained entries instead of zeroing them
constexpr unsigned MASK_INHOM = MASK_INHOM_BIT;

// --------------------------------------------------- cells of a warp
// The number type of a kernel, the scalar it is made of and how many cells a
// lane carries: double and float one, f2 (packed FP32x2, pair.cuh) two.
template <typename T>
struct Num {
  using S = T;
  static constexpr int H = 1;
};
template <>
struct Num<f2> {
  using S = float;
  static constexpr int H = 2;
};
// cells per lane group in the table of a scalar type: FP32 tables interleave
// two cells, the halves of an f2
template <typename S>
__host__ __device__ constexpr int table_halves() { return sizeof(S) == 4 ? 2 : 1; }

// List entries of a warp's unit of work w: entry i0 (and i0 + 1 of an f2
// pair).  Contiguous loops follow the table: a double / f2 unit is one batch,
// a float unit (diagonal) one half of a batch; lists are taken in order.
// Entries past the end repeat the last one (pair) and are not stored.
template <int P, int Q, typename T, bool LIST>
struct UnitMap {
  using S = typename Num<T>::S;
  static constexpr int H = Num<T>::H, TH = table_halves<S>();
  static constexpr int CPW = 32 / (Q * Q);
  static constexpr bool HALF = !LIST && H == 1 && TH == 2;  // float over a paired table
  static __host__ __device__ __forceinline__ int units(int n) {
    return HALF ? 2 * ((n + 2 * CPW - 1) / (2 * CPW)) : (n + CPW * H - 1) / (CPW * H);
  }
  static __device__ __forceinline__ int entry(int w, int r) {
    return HALF ? ((w >> 1) * CPW + r) * 2 + (w & 1) : (w * CPW + r) * H;
  }
};

// ------------------------------------------------------------ cache kernel
// NeoHookOperator::cache and the Eulerian metric: gathers X and u, evaluates
// both gradients, and writes the cell records in FP64 arithmetic.  Lanes own
// lines of cells (SFC), so every store of a component is one contiguous
// access of the warp.  FP32 tables hold two cells per lane slot; their two
// halves are worked on one after the other.  AFFINE (box meshes): the
// reference Jacobian is one per cell, from four corners, instead of an
// evaluation of X at every point, which takes half of the gathers and
// sweeps and 12-42 registers off.  tensor4 FP64 at 60^3 Q2: 414 -> 329 us, with the
// 1.68 GB of the table alone 257 us at copy bandwidth.
template <int P, int Q, typename T, int VAR, bool AFFINE>
__global__ void __launch_bounds__(128) cache_kernel(KArgs<T> a, TabT<P, Q, double> tabt, Tab<P, Q> tab) {
  using S = SFC<P, Q, double>;
  constexpr int N1 = P + 1, NN = S::NN, L = S::L, CPW = S::CPW, TH = table_halves<T>();
  using RL = RecLayout<P, Q, TH>;
  const int WPB = blockDim.x >> 5;
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5;
  double *slab = (double *)smem + warp * S::SZ;
  const LanePos<Q> lp;
  const int gw = blockIdx.x * WPB + warp, nw = gridDim.x * WPB;
  const int n_units = TH * ((a.n_cells + RL::B - 1) / RL::B);
  int bad = 0;
  for (int w = gw; w < n_units; w += nw) {
    const int e = ((w / TH) * CPW + lp.r) * TH + w % TH;
    const bool valid = lp.act && e < a.n_cells;
    const int cell = e < a.n_cells ? e : a.n_cells - 1;
    const int *cn = a.cell_nodes + (size_t)cell * NN;
    double GX[AFFINE ? 1 : Q][3][3], GU[Q][3][3], UV[Q][3];
    {
      double vx[3][N1], vu[3][N1];
#pragma unroll
      for (int k = 0; k < N1; ++k) {
        const size_t d = 3 * (size_t)(__ldg(cn + k * L + lp.t) & NODE_MASK);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (!AFFINE) vx[c][k] = __ldg(a.X + d + c);
          vu[c][k] = (double)__ldg(a.u + d + c);
        }
      }
      if constexpr (AFFINE) affine_jacobian<P>(cn, a.X, GX[0]);
      else S::eval(tabt, vx, slab, lp, GX);
      S::eval(tabt, vu, slab, lp, GU, VAR == VAR_SCALAR_REF ? UV : nullptr);
    }
    const double mu = a.mu[cell];
    const double lambda = (2.0 * mu * a.nu) / (1.0 - 2.0 * a.nu);
    T *rec = a.table + RL::base(cell, a.batch_elems) + lp.t * RL::TS;
    constexpr int CS = RL::CS;
#pragma unroll(Q <= 3 ? Q : 1)
    for (int s = 0; s < Q; ++s) {
      const double w3 = tab.w[s] * tab.w[lp.b] * tab.w[lp.a];
      double Jr[3][3], Jc[3][3], Jri[3][3], Jci[3][3];
#pragma unroll
      for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int e2 = 0; e2 < 3; ++e2) {
          Jr[d][e2] = GX[AFFINE ? 0 : s][d][e2];
          Jc[d][e2] = Jr[d][e2] + GU[s][d][e2];
        }
      inv3(Jr, Jri);
      const double dc = inv3(Jc, Jci);
      T *r = rec + s * a.slice_elems;
      auto put = [&](int comp, double x) {
        if (valid) r[comp * CS] = T(x);
      };
      // scalar_referential / tensor4_ns integrate in the reference frame
      const double jxw = variant_referential(VAR) ? det3(Jr) * w3 : dc * w3;
#pragma unroll
      for (int i = 0; i < 9; ++i) put(C_JINV + i, variant_referential(VAR) ? Jri[i / 3][i % 3] : Jci[i / 3][i % 3]);
      // tensor4 / tensor2 / tensor4_ns store their coefficients times JxW
      constexpr int CV = variant_cvar(VAR);
      const double fw = variant_folds_jxw(VAR) ? jxw : 1.0;
      if (!variant_folds_jxw(VAR)) put(C_JXW, jxw);
      // F = I + Grad u (reference configuration, mf_nh_operator.h:462-476)
      double F[3][3];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int d = 0; d < 3; ++d)
          F[c][d] = GU[s][c][0] * Jri[0][d] + GU[s][c][1] * Jri[1][d] + GU[s][c][2] * Jri[2][d] + (c == d ? 1.0 : 0.0);
      const double det_F = det3(F);
      if (!(det_F > 0.0)) bad = 1;
      if (VAR == VAR_SCALAR_F0 || VAR == VAR_SCALAR_F1) {
        put(C_VAR, (VAR == VAR_SCALAR_F0) ? pow(det_F, -1.0 / 3.0) : mu - 2.0 * lambda * log(det_F));
        if (a.ref_per_cell) {
          // affine cell: the reference metric of the first point stands for all
          if (s == 0 && lp.t == 0 && valid) {
            T *ref = a.table + RL::ref(cell, a.batch_elems, a.slice_elems);
#pragma unroll
            for (int i = 0; i < 9; ++i) ref[i * RL::RS] = T(Jri[i / 3][i % 3]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 9; ++i) put(C_VAR + 1 + i, Jri[i / 3][i % 3]);
        }
        continue;
      }
      const double scalar = mu - 2.0 * lambda * log(det_F);
      if (VAR == VAR_SCALAR_REF) {
        // c and the displacement values at the point (phi_reference.begin_values())
        put(C_VAR, scalar);
#pragma unroll
        for (int c = 0; c < 3; ++c) put(C_VAR + 1 + c, UV[s][c]);
        continue;
      }
      if (VAR == VAR_TENSOR4_NS) {
        // 2 lambda F^-T (x) F^-T + (mu - 2 lambda ln J) F^-T_il F^-1_jk + mu I_ik I_jl
        double Fi[3][3];
        inv3(F, Fi);
#pragma unroll
        for (int m = 0; m < 9; ++m)
#pragma unroll
          for (int n = m; n < 9; ++n) {
            const int i = m / 3, j = m % 3, k = n / 3, l = n % 3;
            put(CV + tri_index(9, m, n), fw * (2.0 * lambda * Fi[j][i] * Fi[l][k] + scalar * Fi[l][i] * Fi[j][k] +
                                               (i == k && j == l ? mu : 0.0)));
          }
        continue;
      }
      const double idet = 1.0 / det_F;
      double tau[6];
#pragma unroll
      for (int I = 0; I < 6; ++I) {
        const int i = sym_i(I), j = sym_j(I);
        const double b = F[i][0] * F[j][0] + F[i][1] * F[j][1] + F[i][2] * F[j][2];
        tau[I] = mu * b - (i == j ? scalar : 0.0);
      }
      if (VAR == VAR_TENSOR2) {
        put(CV, fw * scalar * 2.0 * idet);
        put(CV + 1, fw * 2.0 * lambda * idet);
#pragma unroll
        for (int I = 0; I < 6; ++I) put(CV + 2 + I, fw * tau[I] * idet);
      } else {
#pragma unroll
        for (int I = 0; I < 6; ++I) put(CV + I, fw * tau[I] * idet);
        // C = (2c/J) S + (2 lambda/J) I (x) I  (mf_nh_operator.h:542-546)
        const double ca = scalar * 2.0 * idet, cb = lambda * 2.0 * idet;
#pragma unroll
        for (int I = 0; I < 6; ++I)
#pragma unroll
          for (int J = I; J < 6; ++J)
            put(CV + 6 + tri_index(6, I, J), fw * ((I == J ? ca : 0.0) + (I < 3 && J < 3 ? cb : 0.0)));
      }
    }
  }
  if (bad) atomicOr(a.flag, 1);
}

// ------------------------------------------------------------ apply kernel
// FULL: all MFMask stages (the production path); otherwise stage bits of
// a.mask switch RW / SF / QD on and off like vmult<mask> for breakdowns.
template <int P, int Q, typename T, int VAR, bool FULL>
__global__ void __launch_bounds__(256) apply_kernel(KArgs<T> a, Tab<P, Q> tab) {
  using S = SF<P, Q, T>;
  constexpr int NN = S::NN, NQ = S::NQ, QPL = S::QPL;
  const int WPB = blockDim.x >> 5;
  constexpr bool SCALAR = (VAR == VAR_SCALAR_F0 || VAR == VAR_SCALAR_F1);
  using RL = RecLayout<P, Q, table_halves<T>()>;
  constexpr int CS = RL::CS;
  extern __shared__ __align__(16) unsigned char smem[];
  T *sN = (T *)smem, *sD = sN + Q * (P + 1);
  load_tables<P, Q, T>(tab, sN, sD);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T *slab = sD + Q * (P + 1) + warp * S::SZ;
  T *V = slab, *A = slab + S::SZ1, *B = A + S::SZ2;
  const int gw = blockIdx.x * WPB + warp, nw = gridDim.x * WPB;
  const bool rw = FULL || (a.mask & LSMF_MASK_RW), sf = FULL || (a.mask & LSMF_MASK_SF),
             qd = FULL || (a.mask & LSMF_MASK_QD);
  for (int ic = gw; ic < a.n_cells; ic += nw) {
    const int cell = cell_of(a, ic);
    const int *cn = a.cell_nodes + (size_t)cell * NN;
    const T *rec = a.table + RL::base(cell, a.batch_elems);
    const T *ref = a.table + RL::ref(cell, a.batch_elems, a.slice_elems);
    T G[QPL][3][3], GU[QPL][3][3];
    if (SCALAR) {
      if (rw) gather<NN>(cn, a.u, false, V, lane);   // read_dof_values_plain(u)
      if (sf) S::eval(sN, sD, V, A, B, lane, GU);
    }
    if (rw) gather<NN>(cn, a.src, !(a.mask & MASK_INHOM), V, lane);  // read_dof_values(src)
    else {
      for (int i = lane; i < 3 * NN; i += 32) V[i] = T(0);
      __syncwarp();
    }
    if (sf) S::eval(sN, sD, V, A, B, lane, G);
    else {
#pragma unroll
      for (int l = 0; l < QPL; ++l)
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int e = 0; e < 3; ++e) G[l][c][e] = T(0);
    }
    T mu = 0, lambda = 0, kappa = 0;
    if (SCALAR || VAR == VAR_SCALAR_REF) material<T>(a.mu[cell], a.nu, mu, lambda, kappa);
    T H[QPL][3][3];
#pragma unroll
    for (int l = 0; l < QPL; ++l) {
      const int q = lane + 32 * l;
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int e = 0; e < 3; ++e) H[l][c][e] = T(0);
      if (q >= NQ || !qd) continue;
      const T *r = rec + RL::q_off(q, a.slice_elems);
      T Ji[3][3];
#pragma unroll
      for (int i = 0; i < 9; ++i) Ji[i / 3][i % 3] = r[(C_JINV + i) * CS];
      const T jxw = variant_folds_jxw(VAR) ? T(1) : T(r[C_JXW * CS]);
      T g[3][3];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int d = 0; d < 3; ++d) g[c][d] = G[l][c][0] * Ji[0][d] + G[l][c][1] * Ji[1][d] + G[l][c][2] * Ji[2][d];
      ScalarState<T> st;
      if (SCALAR) {
        T Jr[3][3];
#pragma unroll
        for (int i = 0; i < 9; ++i)
          Jr[i / 3][i % 3] = a.ref_per_cell ? ref[i * RL::RS] : r[(C_VAR + 1 + i) * CS];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int d = 0; d < 3; ++d)
            st.F[c][d] = GU[l][c][0] * Jr[0][d] + GU[l][c][1] * Jr[1][d] + GU[l][c][2] * Jr[2][d] + (c == d ? T(1) : T(0));
        st.det = det3(st.F);
      }
      if (VAR == VAR_SCALAR_REF) {
        T ux[3][Q];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int m = 0; m < Q; ++m) ux[c][m] = rec[m * a.slice_elems + (C_VAR + 1 + c) * CS + (q / Q) * RL::TS];
        collocation_F<Q, CS, RL::TS>(ux, rec + (q % Q) * a.slice_elems, q % Q, (q / Q) % Q, q / (Q * Q), tab.Dc, Ji, st.F);
        st.det = det3(st.F);
      }
      T Qm[3][3];
      physics<T, VAR, CS>(g, r, mu, lambda, kappa, st, Qm);
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          const T h = Qm[c][0] * Ji[e][0] + Qm[c][1] * Ji[e][1] + Qm[c][2] * Ji[e][2];
          H[l][c][e] = variant_folds_jxw(VAR) ? h : T(h * jxw);
        }
    }
    if (sf) {
      S::integrate(sN, sD, H, V, A, B, lane);
    } else {
      for (int i = lane; i < S::SZ2; i += 32) A[i] = T(0);
      __syncwarp();
    }
    if (rw) {
      for (int an = lane; an < NN; an += 32) {
        T o[3];
        S::integrate_node(sN, sD, A, an, o);
        const int packed = __ldg(cn + an);
        const int node = packed & NODE_MASK, cm = packed >> NODE_BITS;
        T *d = a.dst + 3 * (size_t)node;
        if (!(cm & 1)) scatter_add(d, o[0], a.plain);
        if (!(cm & 2)) scatter_add(d + 1, o[1], a.plain);
        if (!(cm & 4)) scatter_add(d + 2, o[2], a.plain);
      }
    }
    __syncwarp();
  }
}


// ---------------------------------------- apply kernel, production path
// The production vmult cell loop.  Q^2 lanes per cell, CPW cells per warp
// (SFC), for f2 two cells per lane; the gather of the next unit (node ids,
// src, and u for the scalar variants) is prefetched into registers while the
// current one is computed; with RING each warp streams the record slices of
// its units through a shared-memory ring of a.ring slices filled by
// cp.async.bulk (evict-first in L2): a slice's place is refilled as soon as
// the slice's points are done, so copies stay in flight through the whole
// unit; without it the records are read with plain coalesced loads.
// SC (scatter): SC_ATOMIC loops over all cells and adds with atomics;
// SC_COLOUR over the list of one group of batches (a.cells, a.n_batches
// entries; no two batches share a node) with plain adds, the cells of a batch
// one after the other; SC_CELLBUF over all
// cells, storing every cell's results to
// a.cellbuf[cell][local node][component] (constrained rows as zero) for the
// node sum that follows; SC_PEER as SC_ATOMIC, with the neighbour part's
// nodes (PEER_BIT in the index map) gathered from a.psrc / a.pu and added to
// a.pdst over peer memory: the partitioned vmult's ghost update and
// compress(add) done by the cell loop itself.
// Bound: HBM for the record-heavy variants (60^3 Q2 tensor4 FP64: 303 us for
// 1.79 GB, 0.90 of the measured copy bandwidth; tensor4_ns 406 us, 0.99),
// else shared-memory wavefronts and the latency of the sweeps (tensor2 229
// us, 0.60).  One cell per warp with row-per-lane sweeps, 51 / 90 values per
// point, took 397 / 654 / 274 us; 96^3 Q1 formulation 0 1167 -> 349 us, 36^3
// Q4 tensor4 504 -> 376 us.
constexpr int SC_ATOMIC = 0, SC_COLOUR = 1, SC_CELLBUF = 2, SC_PEER = 3;

// per-warp shared memory: the ring's slices and barriers, the slab, and for
// the scalar variants the displacement gradients of the unit's points
// (kept there while the source's sweeps run: two gradient sets in registers
// left 8 warps per SM and spilled from Q = 4 on)
template <int P, int Q, typename T, bool SCALAR>
__host__ __device__ __forceinline__ size_t line_warp_bytes(int ring, size_t slice_bytes) {
  using S = SFC<P, Q, T>;
  return (ring * slice_bytes + 16 * ((ring + 1) / 2) + (S::SZ + (SCALAR ? 9 * Q * S::LW : 0)) * sizeof(T) + 127) / 128 * 128;
}

// the cells' values as one number of the kernel's type
template <typename T>
__device__ __forceinline__ T join_of(const typename Num<T>::S *h, int stride) {
  if constexpr (Num<T>::H == 2) return pack2(h[0], h[stride]);
  else return h[0];
}

// One quadrature point of a lane's x line: G (reference gradient of the
// source) becomes H, what the transposed sweeps take.  slice: the cell's
// record at the point's slice and lane 0 (component stride CS, lane stride
// TS); ref: the cell's reference metric (entry stride RS) when ref_per_cell;
// park: the point's displacement gradient (scalar variants), entry stride
// LW; ux: displacement along the x line (scalar_referential).
template <int Q, typename T, int VAR, int CS, int TS, int LW, typename R, typename RF, typename DC>
__device__ __forceinline__ void line_point(T G[3][3], int s, const R &slice, const RF &ref, int RS, bool ref_per_cell,
                                           const T *park, const T ux[3][Q], const LanePos<Q> &lp, const DC &Dc, T mu,
                                           T lambda, T kappa) {
  constexpr bool SCALAR = (VAR == VAR_SCALAR_F0 || VAR == VAR_SCALAR_F1);
  const auto r = slice + lp.t * TS;
  T Ji[3][3];
#pragma unroll
  for (int i = 0; i < 9; ++i) Ji[i / 3][i % 3] = r[(C_JINV + i) * CS];
  const T jxw = variant_folds_jxw(VAR) ? T(1) : T(r[C_JXW * CS]);
  T g[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int d = 0; d < 3; ++d) g[i][d] = G[i][0] * Ji[0][d] + G[i][1] * Ji[1][d] + G[i][2] * Ji[2][d];
  ScalarState<T> st;
  if (SCALAR) {
    T Jr[3][3];
#pragma unroll
    for (int i = 0; i < 9; ++i) Jr[i / 3][i % 3] = ref_per_cell ? T(ref[i * RS]) : T(r[(C_VAR + 1 + i) * CS]);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const T u0 = park[(3 * i) * LW], u1 = park[(3 * i + 1) * LW], u2 = park[(3 * i + 2) * LW];
#pragma unroll
      for (int d = 0; d < 3; ++d) st.F[i][d] = u0 * Jr[0][d] + u1 * Jr[1][d] + u2 * Jr[2][d] + (i == d ? T(1) : T(0));
    }
    st.det = det3(st.F);
  }
  if (VAR == VAR_SCALAR_REF) {
    collocation_F<Q, CS, TS>(ux, slice, s, lp.b, lp.a, Dc, Ji, st.F);
    st.det = det3(st.F);
  }
  T Qm[3][3];
  physics<T, VAR, CS>(g, r, mu, lambda, kappa, st, Qm);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const T h0 = Qm[i][0] * Ji[e][0] + Qm[i][1] * Ji[e][1] + Qm[i][2] * Ji[e][2];
      G[i][e] = variant_folds_jxw(VAR) ? h0 : T(h0 * jxw);
    }
}

// Blocks of 128 threads the register allocation leaves room for: three (168
// registers, 12 warps per SM) up to degree 2 (60^3 Q2 FP64: tensor4 311 -> 303
// us, scalar 367 -> 348, scalar_referential 338 -> 329; 96^3 Q1 scalar 331 ->
// 315, formulation 0 387 -> 349; four blocks, 128 registers, spill: tensor4
// 363), and for tensor2 at degree 3 (167 -> 161); two from there on (255
// registers; 36^3 Q4 tensor4 376 against 438 us) and for the FP32
// scalar_referential Q2 kernel (194 against 210 us).  The Q2 kernels of the
// scalar types do not fit in 168 registers: they spill 116-220 bytes a thread
// in FP64, 184 (formulation 1) and 352 (formulation 0) in FP32, and three
// blocks are the better choice in spite of it, but for FP32 formulation 0: 60^3
// FP32 formulation 1 207 us against 213 with two blocks (no spills),
// formulation 0 249 against 244.
template <int P, int VAR, bool FP32>
constexpr int line_min_blocks() {
  if (P == 2 && VAR == VAR_SCALAR_REF && FP32) return 2;
  return P <= 2 || (P == 3 && VAR == VAR_TENSOR2) ? 3 : 2;
}

template <int P, int Q, typename T, int VAR, bool RING, int SC>
__global__ void __launch_bounds__(128, line_min_blocks<P, VAR, Num<T>::H == 2>()) apply_line_kernel(KArgs<typename Num<T>::S> a, TabT<P, Q, T> tab) {
  using E = typename Num<T>::S;
  constexpr int H = Num<T>::H, TH = table_halves<E>();
  constexpr bool COL = SC == SC_COLOUR;
  constexpr bool SCALAR = (VAR == VAR_SCALAR_F0 || VAR == VAR_SCALAR_F1);
  static_assert(H == TH, "one number holds the cells of a table entry");
  using S = SFC<P, Q, T>;
  using UM = UnitMap<P, Q, T, false>;
  using RL = RecLayout<P, Q, TH>;
  constexpr int N1 = P + 1, NN = S::NN, L = S::L, CPW = S::CPW, LW = S::LW;
  // record access in numbers of T
  constexpr int TS = 1, CS = LW, RS = CPW;
  const int SS = a.slice_elems / H;
  const int WPB = blockDim.x >> 5;
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const LanePos<Q> lp;
  const int D = RING ? a.ring : 0;
  const uint32_t slice_bytes = (uint32_t)(a.slice_elems * sizeof(E));
  const size_t warp_bytes = line_warp_bytes<P, Q, T, SCALAR>(D, slice_bytes);
  // too little shared memory: no unit is taken (a return here instead of this
  // cost small levels up to 0.3 us)
  const bool none = smem_short(WPB * warp_bytes, a.flag);
  // A colour group's successor waits for this whole launch before its first
  // scatter, so it may start, load and compute from here on (colour8 vmult
  // tensor4 FP64 at Q2: 8^3 53.9 -> 23.9 us, 60^3 452 -> 420 us)
  if (COL) asm volatile("griddepcontrol.launch_dependents;");
  unsigned char *wbase = smem + warp * warp_bytes;
  uint64_t *bar = (uint64_t *)(wbase + D * slice_bytes);
  T *slab = (T *)(wbase + D * slice_bytes + 16 * ((D + 1) / 2));
  T *park = slab + S::SZ + lp.ln;  // entry (s, c, e) at ((s * 3 + c) * 3 + e) * LW
  const int gw = blockIdx.x * WPB + warp, nw = gridDim.x * WPB;
  const int n_units = none ? 0 : COL ? a.n_batches : UM::units(a.n_cells);
  // batch of a unit, counted from a.cell0 (a multiple of the batch size)
  auto batch = [&](int w) -> int { return COL ? __ldg(a.cells + w) : w; };
  auto batch_ptr = [&](int w) -> const E * { return a.table + (size_t)(a.cell0 / RL::B + batch(w)) * a.batch_elems; };
  // cells of the lane: c[h]; ok[h]: stored by this lane
  auto cells_of = [&](int w, int c[H], bool ok[H]) {
    const int e0 = UM::entry(batch(w), lp.r);
    const int last = a.n_cells - 1;
    const int f = e0 < a.n_cells ? e0 : last - last % H;
    c[0] = a.cell0 + f;
    ok[0] = lp.act && e0 < a.n_cells;
    if (H == 2) {
      c[H - 1] = f + 1 < a.n_cells ? c[0] + 1 : c[0];
      ok[H - 1] = lp.act && e0 + 1 < a.n_cells;
    }
  };
  // gather registers of the lane's z line of nodes, and the cells' mu
  int pk[H][N1];
  E pv[H][3][N1], pu[H][3][N1];
  double pmu[H], cmu[H];
  auto prefetch_index = [&](int w) {
    int c[H];
    bool ok[H];
    cells_of(w, c, ok);
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int *cn = a.cell_nodes + (size_t)c[h] * NN + lp.t;
      if (SCALAR || VAR == VAR_SCALAR_REF) pmu[h] = __ldg(a.mu + c[h]);
#pragma unroll
      for (int k = 0; k < N1; ++k) pk[h][k] = __ldg(cn + k * L);
    }
  };
  auto prefetch_values = [&]() {
#pragma unroll
    for (int h = 0; h < H; ++h) {
#pragma unroll
      for (int k = 0; k < N1; ++k) {
        const int packed = pk[h][k];
        const bool pe = SC == SC_PEER && (packed & PEER_BIT);
        const size_t dof = 3 * (size_t)(packed & (SC == SC_PEER ? PEER_NODE_MASK : NODE_MASK));
        const E *sv = (pe ? a.psrc : a.src) + dof, *su = (pe ? a.pu : a.u) + dof;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          pv[h][i][k] = __ldg(sv + i);
          if (SCALAR) pu[h][i][k] = __ldg(su + i);
        }
      }
    }
  };
  // the first unit's index lists, the head of its chain of loads, are asked for
  // before the ring is set up (with the shared-memory check before the ring and
  // the lists behind it, CG with FP64 V-cycles 16^3 -> 32^3 80.9 ms, now 76.1)
  if (gw < n_units) prefetch_index(gw);
  uint64_t pol = 0;
  auto copy_slice = [&](int w, int s, int place) {
    mbar_expect_tx(&bar[place], slice_bytes);
    bulk_g2s(wbase + place * slice_bytes, batch_ptr(w) + (size_t)s * a.slice_elems, slice_bytes, &bar[place], pol);
  };
  if (RING) {
    pol = evict_first_policy();
    if (lane == 0 && gw < n_units) {
      for (int d = 0; d < D; ++d) mbar_init(&bar[d], 1);
      mbar_init_fence();
    }
    __syncwarp();
    if (lane == 0)
      for (int d = 0; d < D; ++d)
        if (gw + (d / Q) * nw < n_units) copy_slice(gw + (d / Q) * nw, d % Q, d);
  }
  int place = 0;        // ring place of the next slice, and the parity its
  uint32_t parity = 0;  // copy completes
  // the reference metric of a batch into L1, ahead of its use
  auto prefetch_ref = [&](int w) {
    if (SCALAR && a.ref_per_cell && lane * 128 < 9 * RL::B * (int)sizeof(E))
      asm volatile("prefetch.global.L1 [%0];" ::"l"((const char *)(batch_ptr(w) + (size_t)Q * a.slice_elems) + lane * 128));
  };
  if (gw < n_units) {
    prefetch_values();
    prefetch_ref(gw);
  } else {
    // a launch is not to end before the one whose dependent it is, also
    // where none of its warps has a unit
    asm volatile("griddepcontrol.wait;" ::: "memory");
  }
  for (int w = gw; w < n_units; w += nw) {
    int ck[H][N1];
    T G[Q][3][3];
    int c[H];
    bool ok[H];
    cells_of(w, c, ok);
    // the cell's record at lane 0 of the cell, and its reference metric
    const T *rec = (const T *)(a.table + RL::base(c[0], a.batch_elems));
    T ux[3][Q];  // scalar_referential: displacement along the x line
    if (VAR == VAR_SCALAR_REF) {
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int m = 0; m < Q; ++m) ux[i][m] = rec[m * SS + (C_VAR + 1 + i) * CS + lp.t * TS];
    }
    {
      T v[3][N1], vu[3][N1];
#pragma unroll
      for (int k = 0; k < N1; ++k) {
#pragma unroll
        for (int h = 0; h < H; ++h) ck[h][k] = pk[h][k];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          // read_dof_values(src): constrained entries read as zero
          E x[H];
#pragma unroll
          for (int h = 0; h < H; ++h) x[h] = ((pk[h][k] >> (NODE_BITS + i)) & 1) ? E(0) : pv[h][i][k];
          v[i][k] = join_of<T>(x, H - 1);
          if (SCALAR) {  // read_dof_values_plain(u)
#pragma unroll
            for (int h = 0; h < H; ++h) x[h] = pu[h][i][k];
            vu[i][k] = join_of<T>(x, H - 1);
          }
        }
      }
#pragma unroll
      for (int h = 0; h < H; ++h) cmu[h] = pmu[h];
      if (w + nw < n_units) {
        prefetch_index(w + nw);
        prefetch_values();
        prefetch_ref(w + nw);
      }
      if (!RING && a.prefetch) {
        // one 128-byte line of the records per lane into L1, issued before
        // the sweeps so that the point loop's loads find it there
        const int pw = a.prefetch == 2 ? w + nw : w;
        if (pw < n_units) {
          const char *base = (const char *)batch_ptr(pw);
          for (int off = lane * 128; off < Q * (int)slice_bytes; off += 32 * 128)
            asm volatile("prefetch.global.L1 [%0];" ::"l"(base + off));
        }
      }
      if (SCALAR) {
        S::eval(tab, vu, slab, lp, G);
#pragma unroll
        for (int s = 0; s < Q; ++s)
#pragma unroll
          for (int i = 0; i < 9; ++i) park[(s * 9 + i) * LW] = G[s][i / 3][i % 3];
      }
      S::eval(tab, v, slab, lp, G);
    }
    T mu = 0, lambda = 0, kappa = 0;
    if (SCALAR || VAR == VAR_SCALAR_REF) {
      E m[3][H];
#pragma unroll
      for (int h = 0; h < H; ++h) material<E>(cmu[h], a.nu, m[0][h], m[1][h], m[2][h]);
      mu = join_of<T>(m[0], H - 1);
      lambda = join_of<T>(m[1], H - 1);
      kappa = join_of<T>(m[2], H - 1);
    }
    const T *ref = (const T *)(a.table + RL::ref(c[0], a.batch_elems, a.slice_elems));
    auto point = [&](int s, auto slice) {
      line_point<Q, T, VAR, CS, TS, LW>(G[s], s, slice, ref, RS, a.ref_per_cell != 0, park + s * 9 * LW, ux, lp, tab.Dc, mu, lambda, kappa);
    };
#pragma unroll
    for (int s = 0; s < Q; ++s) {
      if constexpr (RING) {
        if (!mbar_wait_bounded(&bar[place], parity, a.wait_tries)) {
          if (lane == 0) atomicOr(a.flag, FLAG_TIMEOUT);
          // every copy this warp issued is still owed to a place of its
          // shared memory: the one given up on (k = 0) and those of the next
          // D - 1 slices.  Let each land (long bound) before the block
          // exits, so no copy writes shared memory that a later block owns.
          for (int k = 0; k < D; ++k) {
            if (w + ((s + k) / Q) * nw < n_units) mbar_wait_bounded(&bar[place], parity);
            if (++place == D) { place = 0; parity ^= 1; }
          }
          // the launch is not to end before the one whose dependent it is
          asm volatile("griddepcontrol.wait;" ::: "memory");
          return;
        }
        point(s, (const T *)(wbase + place * slice_bytes) + lp.r * L);
        __syncwarp();  // every lane is done reading the slice
        const int wn = w + ((s + D) / Q) * nw;
        if (lane == 0 && wn < n_units) {
          fence_proxy_async_smem();
          copy_slice(wn, (s + D) % Q, place);
        }
        if (++place == D) { place = 0; parity ^= 1; }
      } else {
        point(s, rec + s * SS);
      }
    }
    T out[3][N1];
    S::integrate(tab, G, slab, lp, out);
    // dst's rows are written by the kernel before (no effect in a launch that
    // is not its programmatic dependent)
    if (w == gw) asm volatile("griddepcontrol.wait;" ::: "memory");
    auto scatter = [&](int h) {
#pragma unroll
      for (int k = 0; k < N1; ++k) {
        const int packed = ck[h][k];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          E o;
          if constexpr (H == 2) o = h ? hi2(out[i][k]) : lo2(out[i][k]);
          else o = out[i][k];
          // distribute_local_to_global: constrained rows skipped
          const bool con = (packed >> (NODE_BITS + i)) & 1;
          if (SC == SC_CELLBUF) {
            a.cellbuf[((size_t)c[h] * NN + k * L + lp.t) * 3 + i] = con ? E(0) : o;
          } else if (SC == SC_PEER) {
            if (!con)
              atomic_add(((packed & PEER_BIT) ? a.pdst : a.dst) + 3 * (size_t)(packed & PEER_NODE_MASK) + i, o);
          } else if (!con) {
            atomic_add(a.dst + 3 * (size_t)(packed & NODE_MASK) + i, o);
          }
        }
      }
    };
    // plain adds of a line's values: all loads before the first store, as one
    // round trip (the compiler has to take nine in turn).  From L2: with the
    // launches of the groups overlapping, L1 may hold an earlier group's line.
    // 60^3 Q2 tensor4 FP64, launches in turn: 452 us, 707 with nine round trips; 747 us with one
    // cell per warp and a launch per lattice colour.
    auto add_line = [&](int h) {
      E old[N1][3];
#pragma unroll
      for (int k = 0; k < N1; ++k)
#pragma unroll
        for (int i = 0; i < 3; ++i) old[k][i] = __ldcg(a.dst + 3 * (size_t)(ck[h][k] & NODE_MASK) + i);
#pragma unroll
      for (int k = 0; k < N1; ++k)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          E o;
          if constexpr (H == 2) o = h ? hi2(out[i][k]) : lo2(out[i][k]);
          else o = out[i][k];
          if (!((ck[h][k] >> (NODE_BITS + i)) & 1)) a.dst[3 * (size_t)(ck[h][k] & NODE_MASK) + i] = old[k][i] + o;
        }
    };
    if constexpr (COL) {
      // neighbours within the batch add to the same nodes: in cell order
      for (int r = 0; r < CPW; ++r) {
#pragma unroll
        for (int h = 0; h < H; ++h) {
          if (lp.r == r && ok[h]) add_line(h);
          __syncwarp();
        }
      }
    } else {
#pragma unroll
      for (int h = 0; h < H; ++h)
        if (ok[h]) scatter(h);
    }
  }
}

// --------------------------------------------------------- diagonal kernel
// diag(a, c) = sum_q JxW n^T D_c n with n = grad_x N_a and
// D_c[d][l] = Q(e_c (x) e_l)[c][d]: identical to applying the cell operator
// to unit vectors (mf_nh_operator.h:881-899) and keeping the diagonal entry.
// Pulled back, M_c = J^-1 D_c J^-T JxW is a symmetric 3x3 matrix per point
// and n^T D_c n = sum_ef M_c[e][f] d_e N_a d_f N_a, whose factors are
// products of the 1D tables N N, N D and D D: six fields per component go
// through the three transposed sweeps, in place of a sum over all points
// for every node.
template <int P, int Q, typename T>
struct TabSq {
  T NN[Q][P + 1], ND[Q][P + 1], DD[Q][P + 1];
};

// D_c (symmetric) for row c of the tangent at a point; for the variants that
// fold JxW into their coefficients it comes out times JxW.  order of the six
// entries: 00, 11, 22, 01, 02, 12
template <typename T, int VAR, int CS, typename R>
__device__ __forceinline__ void diag_block(int c, const R &rec, T mu, T lambda, T kappa, const ScalarState<T> &st, T D[6]) {
  constexpr int CV = variant_cvar(VAR);
  if (VAR == VAR_TENSOR4_NS) {
#pragma unroll
    for (int I = 0; I < 6; ++I) D[I] = rec[(CV + tri_index(9, c * 3 + sym_i(I), c * 3 + sym_j(I))) * CS];
    return;
  }
  if (VAR == VAR_TENSOR4 || VAR == VAR_TENSOR2) {
    T c1 = 0, c2 = 0;
    if (VAR == VAR_TENSOR2) {
      c1 = rec[CV * CS];
      c2 = rec[(CV + 1) * CS];
    }
#pragma unroll
    for (int I = 0; I < 6; ++I) {
      const int d = sym_i(I), l = sym_j(I);
      T x = rec[(CV + (VAR == VAR_TENSOR2 ? 2 : 0) + I) * CS];
      if (VAR == VAR_TENSOR2) {
        x += c1 * (T(0.5) * T((d == l) + (d == c && l == c))) + (d == c && l == c ? c2 : T(0));
      } else {
        // entry (c, d), (c, l) of the 6x6 matrix acting on sym(e_c (x) e_l)
        const int Id = c == d ? c : (c + d) + 2, Il = c == l ? c : (c + l) + 2;  // (0,1) 3, (0,2) 4, (1,2) 5
        x += rec[(CV + 6 + tri_index(6, Id, Il)) * CS] * (c == l ? T(1) : T(0.5));
      }
      D[I] = x;
    }
    return;
  }
  T b[6];
#pragma unroll
  for (int I = 0; I < 6; ++I) {
    const int i = sym_i(I), j = sym_j(I);
    b[I] = st.F[i][0] * st.F[j][0] + st.F[i][1] * st.F[j][1] + st.F[i][2] * st.F[j][2];
  }
  const T x0 = rec[C_VAR * CS];
  if (VAR == VAR_SCALAR_F0) {
    // formulation 0 (mf_nh_operator.h:1001-1181), x0 = J^(-1/3)
    const T det = st.det, idet = T(1) / det;
    const T dPsi = (kappa / T(2)) * (det - idet), d2Psi = (kappa / T(2)) * (T(1) + idet * idet);
#pragma unroll
    for (int I = 0; I < 6; ++I) b[I] = b[I] * x0 * x0 * mu;  // tau_bar
    const T trb = b[0] + b[1] + b[2], trd = trb * T(1.0 / 3.0), two3 = T(2.0 / 3.0);
#pragma unroll
    for (int I = 0; I < 6; ++I) {
      const int d = sym_i(I), l = sym_j(I);
      auto iso = [&](int i, int j) -> T { return b[i == j ? i : i + j + 2] - (i == j ? trd : T(0)); };
      T v = (two3 * trb - T(2) * dPsi * det) * (T(0.5) * T((d == l) + (d == c && l == c)));
      if (d == c && l == c) v += det * (dPsi + det * d2Psi) - (two3 * trb) * T(1.0 / 3.0);
      if (l == c) v -= two3 * iso(c, d);
      if (d == c) v -= two3 * iso(c, l);
      v += b[I] + (d == l ? dPsi * det - trd : T(0));
      D[I] = v * idet;
    }
    return;
  }
  // formulation 1: W = c (I + e_c e_c^T) + 2 lambda e_c e_c^T + tau, over J
  // in the Eulerian frame
  const T f = VAR == VAR_SCALAR_F1 ? T(T(1) / st.det) : T(1);
#pragma unroll
  for (int I = 0; I < 6; ++I) {
    const int d = sym_i(I), l = sym_j(I);
    T v = mu * b[I];  // tau = mu b - x0 I cancels the x0 I of the first term
    if (d == c && l == c) v += x0 + T(2) * lambda;
    D[I] = v * f;
  }
}

template <int P, int Q, typename T, int VAR>
__global__ void __launch_bounds__(128) diagonal_kernel(KArgs<T> a, TabT<P, Q, T> tab, TabSq<P, Q, T> sq) {
  using S = SFC<P, Q, T>;
  constexpr int TH = table_halves<T>();
  using RL = RecLayout<P, Q, TH>;
  constexpr int N1 = P + 1, NN = S::NN, L = S::L, CPW = S::CPW, CS = RL::CS;
  constexpr int RA = S::RA, RB = S::RB, BA = S::BA, BB = S::BB;
  constexpr bool SCALAR = (VAR == VAR_SCALAR_F0 || VAR == VAR_SCALAR_F1);
  extern __shared__ __align__(16) unsigned char smem[];
  const int WPB = blockDim.x >> 5, warp = threadIdx.x >> 5;
  T *slab = (T *)smem + warp * S::SZ;
  const LanePos<Q> lp;
  const int gw = blockIdx.x * WPB + warp, nw = gridDim.x * WPB;
  const bool list = a.cells != nullptr;
  const int n_units = list ? UnitMap<P, Q, T, true>::units(a.n_cells) : UnitMap<P, Q, T, false>::units(a.n_cells);
  for (int w = gw; w < n_units; w += nw) {
    const int e = list ? UnitMap<P, Q, T, true>::entry(w, lp.r) : UnitMap<P, Q, T, false>::entry(w, lp.r);
    const bool valid = lp.act && e < a.n_cells;
    const int cell = cell_of(a, e < a.n_cells ? e : a.n_cells - 1);
    const int *cn = a.cell_nodes + (size_t)cell * NN + lp.t;
    const T *cr = a.table + RL::base(cell, a.batch_elems), *ref = a.table + RL::ref(cell, a.batch_elems, a.slice_elems);
    int ck[N1];
#pragma unroll
    for (int k = 0; k < N1; ++k) ck[k] = __ldg(cn + k * L);
    T GU[Q][3][3];
    if (SCALAR) {
      T vu[3][N1];
#pragma unroll
      for (int k = 0; k < N1; ++k)
#pragma unroll
        for (int i = 0; i < 3; ++i) vu[i][k] = __ldg(a.u + 3 * (size_t)(ck[k] & NODE_MASK) + i);
      S::eval(tab, vu, slab, lp, GU);
    }
    T mu = 0, lambda = 0, kappa = 0;
    if (SCALAR || VAR == VAR_SCALAR_REF) material<T>(a.mu[cell], a.nu, mu, lambda, kappa);
    T out[3][N1];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      T M[Q][6];
#pragma unroll
      for (int s = 0; s < Q; ++s) {
        const T *r = cr + s * a.slice_elems + lp.t * RL::TS;
        T Ji[3][3];
#pragma unroll
        for (int i = 0; i < 9; ++i) Ji[i / 3][i % 3] = r[(C_JINV + i) * CS];
        const T jxw = variant_folds_jxw(VAR) ? T(1) : T(r[C_JXW * CS]);
        ScalarState<T> st;
        if (SCALAR) {
          T Jr[3][3];
#pragma unroll
          for (int i = 0; i < 9; ++i) Jr[i / 3][i % 3] = a.ref_per_cell ? ref[i * RL::RS] : r[(C_VAR + 1 + i) * CS];
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int d = 0; d < 3; ++d)
              st.F[i][d] = GU[s][i][0] * Jr[0][d] + GU[s][i][1] * Jr[1][d] + GU[s][i][2] * Jr[2][d] + (i == d ? T(1) : T(0));
          st.det = det3(st.F);
        }
        if (VAR == VAR_SCALAR_REF) {
          T ux[3][Q];
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int m = 0; m < Q; ++m) ux[i][m] = cr[m * a.slice_elems + (C_VAR + 1 + i) * CS + lp.t * RL::TS];
          collocation_F<Q, CS, RL::TS>(ux, cr + s * a.slice_elems, s, lp.b, lp.a, tab.Dc, Ji, st.F);
          st.det = det3(st.F);
        }
        T D[6];
        diag_block<T, VAR, CS>(c, r, mu, lambda, kappa, st, D);
        if (VAR == VAR_SCALAR_REF) {
          // the block is W in the spatial frame: pull back with J^-1 F^-1
          T Fi[3][3], K[3][3];
          inv3(st.F, Fi);
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int d = 0; d < 3; ++d) K[i][d] = Ji[i][0] * Fi[0][d] + Ji[i][1] * Fi[1][d] + Ji[i][2] * Fi[2][d];
#pragma unroll
          for (int i = 0; i < 9; ++i) Ji[i / 3][i % 3] = K[i / 3][i % 3];
        }
        const T Df[3][3] = {{D[0], D[3], D[4]}, {D[3], D[1], D[5]}, {D[4], D[5], D[2]}};
        T DJ[3][3];  // D J^-T
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
          for (int f = 0; f < 3; ++f) DJ[d][f] = Df[d][0] * Ji[f][0] + Df[d][1] * Ji[f][1] + Df[d][2] * Ji[f][2];
#pragma unroll
        for (int I = 0; I < 6; ++I) {
          const int i = sym_i(I), f = sym_j(I);
          const T m = (Ji[i][0] * DJ[0][f] + Ji[i][1] * DJ[1][f] + Ji[i][2] * DJ[2][f]) * (I < 3 ? T(1) : T(2));
          M[s][I] = variant_folds_jxw(VAR) ? m : T(m * jxw);
        }
      }
      // x: fields xx, yy, zz, xy, xz, yz in lanes (qz, qy)
      __syncwarp();
#pragma unroll
      for (int i = 0; i < N1; ++i) {
        T f[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
#pragma unroll
        for (int s = 0; s < Q; ++s) {
          f[0] += sq.DD[s][i] * M[s][0];
          f[1] += sq.NN[s][i] * M[s][1];
          f[2] += sq.NN[s][i] * M[s][2];
          f[3] += sq.ND[s][i] * M[s][3];
          f[4] += sq.ND[s][i] * M[s][4];
          f[5] += sq.NN[s][i] * M[s][5];
        }
#pragma unroll
        for (int I = 0; I < 6; ++I) slab[I * BB + i * RB + lp.ln] = f[I];
      }
      __syncwarp();
      // y, lanes (qz, i): the fields that take N N, N D and D D along z
      T o[3][N1];
      {
        const T *Z = slab + lp.r * L + lp.a * Q + lp.b * RB;
        T z[6][Q];
#pragma unroll
        for (int I = 0; I < 6; ++I)
#pragma unroll
          for (int qy = 0; qy < Q; ++qy) z[I][qy] = Z[I * BB + qy];
#pragma unroll
        for (int j = 0; j < N1; ++j) {
          T s0 = 0, s1 = 0, s2 = 0;
#pragma unroll
          for (int qy = 0; qy < Q; ++qy) {
            s0 += sq.NN[qy][j] * z[0][qy];
            s0 += sq.DD[qy][j] * z[1][qy];
            s0 += sq.ND[qy][j] * z[3][qy];
            s1 += sq.NN[qy][j] * z[4][qy];
            s1 += sq.ND[qy][j] * z[5][qy];
            s2 += sq.NN[qy][j] * z[2][qy];
          }
          o[0][j] = s0;
          o[1][j] = s1;
          o[2][j] = s2;
        }
      }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < N1; ++j)
#pragma unroll
        for (int m = 0; m < 3; ++m) slab[m * BA + j * RA + lp.ln] = o[m][j];
      __syncwarp();
      // z, lanes (j, i)
      const T *Y = slab + lp.r * L + lp.b + lp.a * RA;
      T y[3][Q];
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int qz = 0; qz < Q; ++qz) y[m][qz] = Y[m * BA + qz * Q];
#pragma unroll
      for (int k = 0; k < N1; ++k) {
        T s = 0;
#pragma unroll
        for (int qz = 0; qz < Q; ++qz) {
          s += sq.NN[qz][k] * y[0][qz];
          s += sq.ND[qz][k] * y[1][qz];
          s += sq.DD[qz][k] * y[2][qz];
        }
        out[c][k] = s;
      }
    }
    if (valid && a.plain) {
      add_line_plain<N1>(a.dst, ck, out);
    } else if (valid) {
#pragma unroll
      for (int k = 0; k < N1; ++k)
#pragma unroll
        for (int i = 0; i < 3; ++i)
          if (!((ck[k] >> (NODE_BITS + i)) & 1)) atomic_add(a.dst + 3 * (size_t)(ck[k] & NODE_MASK) + i, out[i][k]);
    }
  }
}

// ------------------------------------------------ coarse-level solver
#include "coarse_kernels.cuh"

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

template <int P, int Q, typename T>
TabT<P, Q, T> make_tabt(const Basis &b) {
  TabT<P, Q, T> t;
  for (int k = 0; k < Q; ++k) {
    for (int i = 0; i <= P; ++i) {
      t.N[k][i] = T(b.N[k * (P + 1) + i]);
      t.D[k][i] = T(b.D[k * (P + 1) + i]);
    }
    for (int m = 0; m < Q; ++m) t.Dc[k][m] = T(b.Dc[k * Q + m]);
  }
  return t;
}

template <int P, int Q>
Tab<P, Q> make_tab(const Basis &b) {
  Tab<P, Q> t;
  for (int k = 0; k < Q; ++k) {
    for (int i = 0; i <= P; ++i) {
      t.N[k][i] = b.N[k * (P + 1) + i];
      t.D[k][i] = b.D[k * (P + 1) + i];
    }
    t.w[k] = b.qw[k];
    for (int m = 0; m < Q; ++m) t.Dc[k][m] = b.Dc[k * Q + m];
  }
  return t;
}

// grid for a persistent-style launch: a whole number of waves of the SMs
template <typename K>
int grid_for(K kernel, int threads, size_t smem, int n_items_per_block_total) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
  if (per_sm < 1) per_sm = 1;
  int g = num_sms() * per_sm;
  if (g > n_items_per_block_total) g = n_items_per_block_total;
  return g < 1 ? 1 : g;
}

// warps per block such that the per-warp slabs fit in ~200 KB of shared memory
inline int warps_for(size_t slab_bytes, int max_warps) {
  int w = max_warps;
  while (w > 1 && slab_bytes * w > 200 * 1024) w >>= 1;
  return w;
}
// largest warp count (<= max_warps) whose slabs fit in budget bytes
inline int warps_for_budget(size_t warp_bytes, int max_warps, size_t budget) {
  int w = max_warps;
  while (w > 0 && warp_bytes * w > budget) --w;
  return w;
}

int variant_of(const lsmf_op *op) {
  if (op->caching == LSMF_CACHE_TENSOR4) return VAR_TENSOR4;
  if (op->caching == LSMF_CACHE_TENSOR2) return VAR_TENSOR2;
  if (op->caching == LSMF_CACHE_SCALAR_REFERENTIAL) return VAR_SCALAR_REF;
  if (op->caching == LSMF_CACHE_TENSOR4_NS) return VAR_TENSOR4_NS;
  return op->formulation == 0 ? VAR_SCALAR_F0 : VAR_SCALAR_F1;
}

template <typename T>
KArgs<T> make_args(const lsmf_op *op) {
  const Level &L = op->L();
  KArgs<T> a;
  a.cell_nodes = L.d_cell_nodes.ptr;
  a.n_cells = L.n_cells;
  a.n_batches = 0;
  a.slice_elems = op->slice_elems;
  a.batch_elems = op->batch_elems;
  a.ring = 0;
  a.ref_per_cell = op->ref_per_cell ? 1 : 0;
  a.table = (T *)op->d_table.ptr;
  a.src = nullptr;
  a.dst = nullptr;
  a.u = (const T *)op->d_u;
  a.X = L.d_X.ptr;
  a.mu = op->d_mu.ptr;
  a.nu = op->nu;
  a.flag = op->d_flag.ptr;
  a.mask = LSMF_MASK_DEFAULT;
  a.wait_tries = op->wait_tries >= 0 ? op->wait_tries : WAIT_TRIES_DEFAULT;
  a.cells = nullptr;
  a.plain = 0;
  a.cellbuf = nullptr;
  a.prefetch = op->prefetch;
  a.psrc = nullptr;
  a.pdst = nullptr;
  a.pu = nullptr;
  a.cell0 = 0;
  return a;
}

template <typename T>
void set_range(KArgs<T> &a, const CellRange &r) {
  if (r.cells) {
    a.cells = r.cells;
    if (r.batches) a.n_batches = r.n_list;
    else a.n_cells = r.n_list;
  }
  a.plain = r.plain ? 1 : 0;
  a.cellbuf = (T *)r.cellbuf;
  if (r.count >= 0) {
    a.cell0 = r.first;
    a.n_cells = r.count;
  }
  if (r.peer_nodes) {
    a.cell_nodes = r.peer_nodes;
    a.psrc = (const T *)r.peer_src;
    a.pdst = (T *)r.peer_dst;
    a.pu = (const T *)r.peer_u;
  }
}

template <int P, int Q, typename T, int VAR>
lsmf_status run_cache(lsmf_op *op) {
  auto a = make_args<T>(op);
  const Tab<P, Q> tab = make_tab<P, Q>(op->mesh->basis);
  const TabT<P, Q, double> tabt = make_tabt<P, Q, double>(op->mesh->basis);
  using S = SFC<P, Q, double>;
  const int w = 4;
  const size_t smem = sizeof(double) * w * S::SZ;
  auto k = op->L().affine ? cache_kernel<P, Q, T, VAR, true> : cache_kernel<P, Q, T, VAR, false>;
  LSMF_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int units = (a.n_cells + S::CPW - 1) / S::CPW;
  const int g = grid_for(k, 32 * w, smem, (units + w - 1) / w);
  k<<<g, 32 * w, smem, op->stream>>>(a, tabt, tab);
  LSMF_CUDA(cudaGetLastError());
  return LSMF_OK;
}

// launch the production cell loop
template <int P, int Q, typename T, int VAR>
lsmf_status launch_line(const lsmf_op *op, KArgs<typename Num<T>::S> a, bool peer, bool dependent, int ring, int max_warps,
                        cudaStream_t stream) {
  using E = typename Num<T>::S;
  const TabT<P, Q, T> tab = make_tabt<P, Q, T>(op->mesh->basis);
  const bool col = a.cells != nullptr, cellbuf = a.cellbuf != nullptr;
  const size_t slice_bytes = a.slice_elems * sizeof(E);
  auto wbytes = [&](int d) { return line_warp_bytes<P, Q, T, VAR == VAR_SCALAR_F0 || VAR == VAR_SCALAR_F1>(d, slice_bytes); };
  // a smaller ring when it would leave fewer than 4 warps per SM
  while (ring > 0 && warps_for_budget(wbytes(ring), 8, 220 * 1024) < 4) --ring;
  a.ring = ring;
  // at most 4 warps per block (the kernel's launch bound is 128 threads);
  // smaller blocks let several blocks share an SM
  const int w = warps_for_budget(wbytes(ring), max_warps < 4 ? max_warps : 4, 220 * 1024);
  const size_t smem = w * wbytes(ring);
  const int units = col ? a.n_batches : UnitMap<P, Q, T, false>::units(a.n_cells);
  auto go = [&](auto k) -> lsmf_status {
    // small launches are bound by the host: shared memory up to 48 KB needs
    // no attribute, and a grid within the SMs no occupancy query
    if (smem > 48 * 1024) LSMF_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int blocks = (units + w - 1) / w;
    const int g = blocks <= num_sms() ? blocks : grid_for(k, 32 * w, smem, blocks);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(g);
    cfg.blockDim = dim3(32 * w);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = dependent ? 1 : 0;
    LSMF_CUDA(cudaLaunchKernelEx(&cfg, k, a, tab));
    return LSMF_OK;
  };
  if (col) return ring ? go(apply_line_kernel<P, Q, T, VAR, true, SC_COLOUR>) : go(apply_line_kernel<P, Q, T, VAR, false, SC_COLOUR>);
  if (cellbuf) return ring ? go(apply_line_kernel<P, Q, T, VAR, true, SC_CELLBUF>) : go(apply_line_kernel<P, Q, T, VAR, false, SC_CELLBUF>);
  if constexpr (sizeof(E) == 8)
    if (peer) return ring ? go(apply_line_kernel<P, Q, T, VAR, true, SC_PEER>) : go(apply_line_kernel<P, Q, T, VAR, false, SC_PEER>);
  return ring ? go(apply_line_kernel<P, Q, T, VAR, true, SC_ATOMIC>) : go(apply_line_kernel<P, Q, T, VAR, false, SC_ATOMIC>);
}

template <int P, int Q, typename T, int VAR>
lsmf_status run_apply(const lsmf_op *op, T *dst, const T *src, unsigned mask, CellRange range) {
  auto a = make_args<T>(op);
  cudaStream_t stream = range.stream ? range.stream : op->stream;
  a.src = src;
  a.dst = dst;
  a.mask = mask;
  set_range(a, range);
  if (a.n_cells == 0) return LSMF_OK;
  const bool full = (mask & (LSMF_MASK_RW | LSMF_MASK_SF | LSMF_MASK_QD)) ==
                        (LSMF_MASK_RW | LSMF_MASK_SF | LSMF_MASK_QD) &&
                    !(mask & MASK_INHOM);
  const bool col = a.cells != nullptr, cellbuf = a.cellbuf != nullptr, peer = range.peer_nodes != nullptr;
  if (cellbuf && !(full && !op->basic)) {
    set_error("the node-sum scatter serves the full vmult cell loop only");
    return LSMF_ERR_INVALID_ARG;
  }
  if (peer && (!full || op->basic || col || cellbuf || sizeof(T) != 8)) {
    set_error("the fused interface exchange serves the full FP64 vmult cell loop with atomic scatter only");
    return LSMF_ERR_INVALID_ARG;
  }
  if (full && !op->basic) {
    if (col && !range.batches) {
      set_error("the production vmult kernel takes a list of batches");
      return LSMF_ERR_INVALID_ARG;
    }
    if (a.cell0 % RecLayout<P, Q, table_halves<T>()>::B != 0) {
      set_error("a chunk of the cell loop must start at a whole batch of cells");
      return LSMF_ERR_INVALID_ARG;
    }
    // plain loads: L1 prefetch of the unit's records before its sweeps
    if (op->prefetch < 0) a.prefetch = 1;
    // Defaults measured on B200 over ring depth x warps per block x chunks at
    // 96^3 Q1, 60^3 Q2, 40^3 Q3 and 36^3 Q4, FP64 and FP32: a ring of two
    // slices almost everywhere (60^3 Q2 tensor4 FP64 303 us against 314 with
    // plain loads and 370 with three slices, which cost resident warps);
    // three slices for the small records of degree 4 (tensor2 308 against 318
    // us); plain loads for the scalar variants from degree 2 on (60^3 Q2 348
    // against 355 us: 11 values per point, and their parked gradients already
    // fill the shared memory).  2 warps per block; 1 for tensor4_ns up to
    // degree 2 (406 against 415 us) and 4 at degree 4 (tensor4 376 against
    // 381 us with 1).
    constexpr bool scalar = VAR == VAR_SCALAR_F0 || VAR == VAR_SCALAR_F1;
    constexpr int ring_auto = scalar && P >= 2 ? 0 : P == 4 && (VAR == VAR_TENSOR2 || VAR == VAR_SCALAR_REF) ? 3 : 2;
    constexpr int warps_auto = P == 4 ? 4 : VAR == VAR_TENSOR4_NS && P <= 2 ? 1 : 2;
    const int ring = op->stages >= 0 ? (op->stages ? op->stages + 1 : 0) : ring_auto;
    const int max_warps = op->max_warps > 0 ? op->max_warps : warps_auto;
    // FP32: two cells per lane, in packed registers
    using N = typename std::conditional<sizeof(T) == 8, double, f2>::type;
    LSMF_TRY((launch_line<P, Q, N, VAR>(op, a, peer, range.dependent, ring, max_warps, stream)));
  } else {
    const Tab<P, Q> tab = make_tab<P, Q>(op->mesh->basis);
    using S = SF<P, Q, T>;
    const int w = warps_for(sizeof(T) * S::SZ, 8);
    const size_t smem = sizeof(T) * (S::TAB + w * S::SZ);
    auto go = [&](auto k) -> lsmf_status {
      LSMF_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      const int g = grid_for(k, 32 * w, smem, (a.n_cells + w - 1) / w);
      k<<<g, 32 * w, smem, stream>>>(a, tab);
      return LSMF_OK;
    };
    if (full) LSMF_TRY(go(apply_kernel<P, Q, T, VAR, true>));
    else LSMF_TRY(go(apply_kernel<P, Q, T, VAR, false>));
  }
  LSMF_CUDA(cudaGetLastError());
  return LSMF_OK;
}

template <int P, int Q, typename T, int VAR>
lsmf_status run_diag(lsmf_op *op, T *diag, CellRange range) {
  auto a = make_args<T>(op);
  a.dst = diag;
  set_range(a, range);
  if (a.n_cells == 0) return LSMF_OK;
  const TabT<P, Q, T> tab = make_tabt<P, Q, T>(op->mesh->basis);
  TabSq<P, Q, T> sq;
  const Basis &b = op->mesh->basis;
  for (int k = 0; k < Q; ++k)
    for (int i = 0; i <= P; ++i) {
      const double n = b.N[k * (P + 1) + i], d = b.D[k * (P + 1) + i];
      sq.NN[k][i] = T(n * n);
      sq.ND[k][i] = T(n * d);
      sq.DD[k][i] = T(d * d);
    }
  using S = SFC<P, Q, T>;
  const int w = 4;
  const size_t smem = sizeof(T) * w * S::SZ;
  auto k = diagonal_kernel<P, Q, T, VAR>;
  LSMF_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int units = (a.n_cells + S::CPW - 1) / S::CPW + 1;
  const int g = grid_for(k, 32 * w, smem, (units + w - 1) / w);
  k<<<g, 32 * w, smem, op->stream>>>(a, tab, sq);
  LSMF_CUDA(cudaGetLastError());
  return LSMF_OK;
}

// Sizes of a CTA of the coarse-level solver with W working warps
template <int P, int Q, typename T, int VAR>
CoarseShape coarse_shape(const lsmf_op *op, int W) {
  CoarseShape s;
  s.batch = 32 / (Q * Q);
  s.cells = W * s.batch;
  s.unit_bytes = coarse_unit_bytes<P, Q, T, VAR>(op->slice_elems);
  s.out_offset = coarse_out_offset<P, Q, T, VAR>(op->slice_elems);
  return s;
}

// launch a coarse-level kernel: cooperative, one CTA per part of the plan
template <typename K, typename... A>
lsmf_status launch_coarse(const lsmf_op *op, const CoarsePlan &plan, K k, A &...args) {
  // every packet starts without a tag
  LSMF_CUDA(cudaMemsetAsync(plan.xbuf.ptr, 0, plan.xbuf.n * sizeof(ulonglong2), op->stream));
  LSMF_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)plan.smem));
  void *ptrs[] = {(void *)&args...};
  LSMF_CUDA(cudaLaunchCooperativeKernel((const void *)k, dim3(plan.n_cta), dim3(COARSE_THREADS), ptrs, plan.smem, op->stream));
  return LSMF_OK;
}
template <typename T>
CoarseArgs<T> coarse_level_args(const lsmf_op *op, const CoarsePlan &plan) {
  CoarseArgs<T> ca = coarse_args<T>(plan);
  ca.invd = (const T *)op->d_inv_diag.ptr;
  ca.cmask = op->L().d_cmask.ptr;
  return ca;
}

template <int P, int Q, typename T, int VAR>
lsmf_status run_coarse_cheb(const lsmf_op *op, const CoarsePlan &plan, void *x, const void *b, double theta, double delta,
                            int degree) {
  auto a = make_args<T>(op);
  const TabT<P, Q, T> tab = make_tabt<P, Q, T>(op->mesh->basis);
  CoarseArgs<T> ca = coarse_level_args<T>(op, plan);
  ca.b = (const T *)b;
  ca.x = (T *)x;
  ca.theta = theta;
  ca.delta = delta;
  ca.degree = degree;
  auto k = plan.max_nodes <= 2 * COARSE_THREADS ? coarse_cheb_kernel<P, Q, T, VAR, 2> : coarse_cheb_kernel<P, Q, T, VAR, 4>;
  return launch_coarse(op, plan, k, a, tab, ca);
}

template <int P, int Q, typename T, int VAR>
lsmf_status run_coarse_eig(const lsmf_op *op, const CoarsePlan &plan, const CoarseEig &e) {
  auto a = make_args<T>(op);
  const TabT<P, Q, T> tab = make_tabt<P, Q, T>(op->mesh->basis);
  CoarseArgs<T> ca = coarse_level_args<T>(op, plan);
  CoarseEigArgs ea;
  ea.mean = e.mean;
  ea.tol_abs = e.tol_abs;
  ea.tol_rel = e.tol_rel;
  ea.max_it = e.max_it;
  ea.alpha = e.alpha;
  ea.beta = e.beta;
  ea.res2 = e.res2;
  ea.its = e.its;
  auto k = plan.max_nodes <= 2 * COARSE_THREADS ? coarse_eig_kernel<P, Q, T, VAR, 2> : coarse_eig_kernel<P, Q, T, VAR, 4>;
  return launch_coarse(op, plan, k, a, tab, ca, ea);
}

#define LSMF_DISPATCH_VAR(v, ...)                                                     \
  [&]() -> lsmf_status {                                                              \
    switch (v) {                                                                      \
      case VAR_TENSOR4: { constexpr int V_ = VAR_TENSOR4; return __VA_ARGS__; }       \
      case VAR_TENSOR2: { constexpr int V_ = VAR_TENSOR2; return __VA_ARGS__; }       \
      case VAR_SCALAR_F1: { constexpr int V_ = VAR_SCALAR_F1; return __VA_ARGS__; }   \
      case VAR_SCALAR_REF: { constexpr int V_ = VAR_SCALAR_REF; return __VA_ARGS__; } \
      case VAR_TENSOR4_NS: { constexpr int V_ = VAR_TENSOR4_NS; return __VA_ARGS__; } \
      default: { constexpr int V_ = VAR_SCALAR_F0; return __VA_ARGS__; }             \
    }                                                                                 \
  }()

// the entry points of one (degree, precision) pair, Q = P + 1 Gauss points
template <int P, typename T>
struct DegreeOps {
  static constexpr int Q = P + 1;
  static lsmf_status cache(lsmf_op *op) {
    return LSMF_DISPATCH_VAR(variant_of(op), (run_cache<P, Q, T, V_>(op)));
  }
  static lsmf_status apply(const lsmf_op *op, void *dst, const void *src, unsigned mask, CellRange range) {
    return LSMF_DISPATCH_VAR(variant_of(op), (run_apply<P, Q, T, V_>(op, (T *)dst, (const T *)src, mask, range)));
  }
  static lsmf_status diag(lsmf_op *op, void *d, CellRange range) {
    return LSMF_DISPATCH_VAR(variant_of(op), (run_diag<P, Q, T, V_>(op, (T *)d, range)));
  }
  static CoarseShape shape(const lsmf_op *op, int W) {
    CoarseShape s;
    (void)LSMF_DISPATCH_VAR(variant_of(op), (s = coarse_shape<P, Q, T, V_>(op, W), LSMF_OK));
    return s;
  }
  static lsmf_status cheb(const lsmf_op *op, const CoarsePlan &plan, void *x, const void *b, double theta, double delta,
                          int degree) {
    return LSMF_DISPATCH_VAR(variant_of(op), (run_coarse_cheb<P, Q, T, V_>(op, plan, x, b, theta, delta, degree)));
  }
  static lsmf_status eig(const lsmf_op *op, const CoarsePlan &plan, const CoarseEig &e) {
    return LSMF_DISPATCH_VAR(variant_of(op), (run_coarse_eig<P, Q, T, V_>(op, plan, e)));
  }
  static const OpsTable &table() {
    static const OpsTable t = {&cache, &apply, &diag, &shape, &cheb, &eig};
    return t;
  }
};

}  // namespace
}  // namespace lsmf
