// Device building blocks of the cell kernels: warp-cooperative sum
// factorisation and the quadrature-point physics of the Neo-Hookean tangent.
//
// Execution model of the production kernels (SFC): a cell is worked on by
// Q^2 lanes of a warp, each holding whole lines of the cell (a z line of
// nodes, then a z line of points by x / y, finally an x line of quadrature
// points), so a warp carries 32 / Q^2 cells (8, 3, 2, 1 for Q = 2..5) and
// only the two transposes between the three sweeps go through a per-warp
// shared-memory slab.  The basic kernel (SF) keeps one cell per warp with
// lanes striding over the work items of each sweep.
#pragma once
#include <cuda_runtime.h>

#include "lsmf_internal.h"

namespace lsmf {

enum Variant {
  VAR_TENSOR4 = 0, VAR_TENSOR2 = 1, VAR_SCALAR_F1 = 2, VAR_SCALAR_F0 = 3,
  VAR_SCALAR_REF = 4,  // scalar_referential
  VAR_TENSOR4_NS = 5   // tensor4_ns (dP/dF)
};
__host__ __device__ constexpr bool variant_referential(int v) { return v == VAR_SCALAR_REF || v == VAR_TENSOR4_NS; }

// Components of the cell record.  The first 9 are the inverse Jacobian
// (row-major) of the frame the variant integrates in: Eulerian for tensor4 /
// tensor2 / scalar, reference for scalar_referential and tensor4_ns.  The
// point result of tensor4, tensor2 and tensor4_ns is linear in their cached
// coefficients, so those are stored multiplied by JxW and follow from
// component 9: tensor4 JxW tau/J (6) + JxW C (21: the 6x6 matrix acting on
// sym(g) is symmetric, its upper triangle is kept); tensor2 JxW c1, JxW c2,
// JxW tau/J (6); tensor4_ns JxW dP/dF (45: the 9x9 matrix of a hyperelastic
// material is symmetric, its upper triangle is kept).  The scalar variants
// keep JxW as component 9, then: scalar c + reference inverse Jacobian (9);
// scalar_referential c + u at the point (3).
// The records are interleaved over the cells a warp works on together, see
// RecLayout.
constexpr int C_JINV = 0, C_JXW = 9, C_VAR = 10;
__host__ __device__ constexpr bool variant_folds_jxw(int v) {
  return v == VAR_TENSOR4 || v == VAR_TENSOR2 || v == VAR_TENSOR4_NS;
}
// first coefficient component
__host__ __device__ constexpr int variant_cvar(int v) { return variant_folds_jxw(v) ? C_JXW : C_VAR; }
// components a point keeps (scalar on affine cells: 11, and the reference
// inverse Jacobian once per cell)
__host__ __device__ constexpr int variant_ncomp(int v) {
  return v == VAR_TENSOR4 ? 36 : v == VAR_TENSOR2 ? 17 : v == VAR_SCALAR_REF ? 14 : v == VAR_TENSOR4_NS ? 54 : 20;
}

// The cell records of the device table.  A batch of B consecutive cells (the
// cells one warp works on at a time: CPW groups of L = Q^2 lanes, and for
// FP32 tables TH = 2 cells per lane, the halves of a packed register) is
// stored as Q slices, one per point of the lanes' x lines, each
// [component][lane][half]: a component's load is one contiguous 256-byte
// (216 at Q = 3) access of the warp, and a slice is one contiguous block for
// the bulk-copy ring.  With [cell][comp][point] records the three cells of a
// Q2 warp would touch three 72-byte pieces per load.  A slice takes
// slice_elems values (its components, padded to 16 bytes), a batch
// batch_elems (Q slices, then for scalar caching on affine cells the
// reference inverse Jacobians of its cells, padded to 16 bytes).
template <int P, int Q, int TH>
struct RecLayout {
  static constexpr int L = Q * Q, CPW = 32 / L, LW = CPW * L, B = CPW * TH;
  static constexpr int TS = TH, CS = LW * TH;  // strides of lane, component
  static constexpr int RS = CPW * TH;          // stride of the entries of the reference inverse Jacobian
  // first value of a cell (slice 0, component 0, lane 0)
  static __host__ __device__ __forceinline__ size_t base(int cell, int batch_elems) {
    const int b = cell / B, e = cell - b * B;
    return (size_t)b * batch_elems + (e / TH) * (L * TH) + e % TH;
  }
  // offset of point q = (qz Q + qy) Q + qx
  static __host__ __device__ __forceinline__ int q_off(int q, int slice_elems) {
    return (q % Q) * slice_elems + (q / Q) * TS;
  }
  // first entry of a cell's reference inverse Jacobian
  static __host__ __device__ __forceinline__ size_t ref(int cell, int batch_elems, int slice_elems) {
    const int b = cell / B, e = cell - b * B;
    return (size_t)b * batch_elems + (size_t)Q * slice_elems + e;
  }
};

template <int P, int Q>
struct Tab {
  double N[Q][P + 1], D[Q][P + 1], w[Q];
  double Dc[Q][Q];  // collocation derivative on the Gauss points
};

// 1D tables in the arithmetic type, passed by value as a kernel parameter:
// with compile-time indices every entry is a constant-bank operand of the
// FMA, so the sweeps below load no shape values from memory.
template <int P, int Q, typename T>
struct TabT {
  T N[Q][P + 1], D[Q][P + 1];
  T Dc[Q][Q];  // collocation derivative on the Gauss points
};

// scalar_referential: F = I + Grad u at point (qx, qy, qz) from the
// displacement stored at the points of the cell record (collocation
// derivative, the FEEvaluationImplCollocation step of
// mf_nh_operator.h:1271-1300) and the reference inverse Jacobian.
// ux[c][m]: values along the point's x line; slice: the cell's record at the
// point's slice and lane 0 (a pointer, or an accessor with operator[] and
// + offset); CS, TS: its component and lane strides.
template <int Q, int CS, int TS, typename T, typename DC, typename R>
__device__ __forceinline__ void collocation_F(const T ux[3][Q], const R &slice, int qx, int qy, int qz, const DC &Dc,
                                              const T Ji[3][3], T F[3][3]) {
  T G[3][3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const auto u = slice + (C_VAR + 1 + c) * CS;
    T gx = 0, gy = 0, gz = 0;
#pragma unroll
    for (int m = 0; m < Q; ++m) {
      gx += T(Dc[qx][m]) * ux[c][m];
      gy += T(Dc[qy][m]) * u[(qz * Q + m) * TS];
      gz += T(Dc[qz][m]) * u[(m * Q + qy) * TS];
    }
    G[c][0] = gx; G[c][1] = gy; G[c][2] = gz;
  }
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int d = 0; d < 3; ++d)
      F[c][d] = G[c][0] * Ji[0][d] + G[c][1] * Ji[1][d] + G[c][2] * Ji[2][d] + (c == d ? T(1) : T(0));
}

// Place of a lane in its warp: cell slot r, line (a, b) of the cell, and the
// lane id clamped to the working lanes.  At Q = 3 / 5 the lanes 27..31 /
// 25..31 repeat the last working lane: they read and write the same
// shared-memory words with the same values, so the sweeps need no branches;
// only stores to global memory test `act`.
template <int Q>
struct LanePos {
  static constexpr int L = Q * Q, CPW = 32 / L, LW = CPW * L;
  int ln, r, t, a, b;
  bool act;
  __device__ __forceinline__ LanePos() {
    const int lane = threadIdx.x & 31;
    act = lane < LW;
    ln = act ? lane : LW - 1;
    r = ln / L;
    t = ln - r * L;
    a = t / Q;
    b = t - a * Q;
  }
};

// Jacobian of an affine cell from four of its corners (cn: the cell's nodes)
template <int P>
__device__ __forceinline__ void affine_jacobian(const int *__restrict__ cn, const double *__restrict__ X, double J[3][3]) {
  constexpr int N1 = P + 1;
  const double *x0 = X + 3 * (size_t)(__ldg(cn) & NODE_MASK);
  const int corner[3] = {P, P * N1, P * N1 * N1};
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const double *xe = X + 3 * (size_t)(__ldg(cn + corner[e]) & NODE_MASK);
#pragma unroll
    for (int d = 0; d < 3; ++d) J[d][e] = __ldg(xe + d) - __ldg(x0 + d);
  }
}

// Sum factorisation with whole lines per lane, Q^2 lanes per cell.
//   eval:      lane (j, i) holds the nodes k = 0..P of its z line; the z
//              sweep runs in registers, its two fields (value, derivative)
//              are transposed to lanes (qz, i) for the y sweep, and its
//              three fields to lanes (qz, qy) for the x sweep, which leaves
//              the reference gradients of an x line of points in registers.
//   integrate: the transpose, back to nodal values of z lines.
// Per cell and direction 2 * 3 + 3 * 3 words per lane go through shared
// memory each way; the row-per-lane form this replaces also moved the 9
// gradient components of every point (96 against 60 shared-memory accesses
// per lane and cell at Q = 3), and its kernels were bound by exactly that
// traffic.  The slab rows are 32 + Q (z / y transposes) and 33 (y / x)
// entries apart: = Q and = 1 modulo 16 and 32, which makes every access of
// both sides of a transpose conflict-free for 8- and 4-byte entries.
// NCG components go through the slab at a time (3, or 1 where shared memory
// is short: a third of the slab for three times the barriers).
template <int P, int Q, typename T, int NCG = 3>
struct SFC {
  static constexpr int N1 = P + 1, NN = N1 * N1 * N1, NQ = Q * Q * Q;
  static_assert(N1 == Q, "q = p + 1");
  static constexpr int L = Q * Q, CPW = 32 / L, LW = CPW * L;
  static constexpr int RA = 32 + Q, RB = 33;
  static constexpr int BA = Q * RA, BB = Q * RB;  // one component of one field
  static constexpr int SZ = NCG * (2 * BA > 3 * BB ? 2 * BA : 3 * BB);  // per-warp slab (elements of T)

  // v[c][k]: value of component c at node k of the lane's z line ->
  // G[s][c][e]: reference gradient at point s of the lane's x line, and with
  // Vq the values Vq[s][c] there
  static __device__ __forceinline__ void eval(const TabT<P, Q, T> &tb, const T v[3][N1], T *slab, const LanePos<Q> &lp,
                                              T G[Q][3][3], T (*Vq)[3] = nullptr) {
#pragma unroll
    for (int c0 = 0; c0 < 3; c0 += NCG) {
      __syncwarp();  // the slab's previous readers are done
#pragma unroll
      for (int g = 0; g < NCG; ++g)
#pragma unroll
        for (int qz = 0; qz < Q; ++qz) {
          T s0 = 0, s1 = 0;
#pragma unroll
          for (int k = 0; k < N1; ++k) {
            s0 += tb.N[qz][k] * v[c0 + g][k];
            s1 += tb.D[qz][k] * v[c0 + g][k];
          }
          slab[g * BA + qz * RA + lp.ln] = s0;
          slab[(NCG + g) * BA + qz * RA + lp.ln] = s1;
        }
      __syncwarp();
      // lane (qz, i) = (a, b)
      T a0[NCG][N1], a1[NCG][N1];
      {
        const T *A = slab + lp.r * L + lp.b + lp.a * RA;
#pragma unroll
        for (int g = 0; g < NCG; ++g)
#pragma unroll
          for (int j = 0; j < N1; ++j) {
            a0[g][j] = A[g * BA + j * Q];
            a1[g][j] = A[(NCG + g) * BA + j * Q];
          }
      }
      __syncwarp();
#pragma unroll
      for (int g = 0; g < NCG; ++g)
#pragma unroll
        for (int qy = 0; qy < Q; ++qy) {
          T s00 = 0, s01 = 0, s10 = 0;
#pragma unroll
          for (int j = 0; j < N1; ++j) {
            s00 += tb.N[qy][j] * a0[g][j];
            s01 += tb.D[qy][j] * a0[g][j];
            s10 += tb.N[qy][j] * a1[g][j];
          }
          slab[g * BB + qy * RB + lp.ln] = s00;
          slab[(NCG + g) * BB + qy * RB + lp.ln] = s01;
          slab[(2 * NCG + g) * BB + qy * RB + lp.ln] = s10;
        }
      __syncwarp();
      // lane (qz, qy) = (a, b)
      const T *B = slab + lp.r * L + lp.a * Q + lp.b * RB;
#pragma unroll
      for (int g = 0; g < NCG; ++g) {
        const int c = c0 + g;
        T b0[N1], by[N1], bz[N1];
#pragma unroll
        for (int i = 0; i < N1; ++i) {
          b0[i] = B[g * BB + i];
          by[i] = B[(NCG + g) * BB + i];
          bz[i] = B[(2 * NCG + g) * BB + i];
        }
#pragma unroll
        for (int s = 0; s < Q; ++s) {
          T gx = 0, gy = 0, gz = 0;
#pragma unroll
          for (int i = 0; i < N1; ++i) {
            gx += tb.D[s][i] * b0[i];
            gy += tb.N[s][i] * by[i];
            gz += tb.N[s][i] * bz[i];
          }
          G[s][c][0] = gx;
          G[s][c][1] = gy;
          G[s][c][2] = gz;
          if (Vq) {
            T x = 0;
#pragma unroll
            for (int i = 0; i < N1; ++i) x += tb.N[s][i] * b0[i];
            Vq[s][c] = x;
          }
        }
      }
    }
  }

  // H[s][c][e] at the points of the lane's x line -> out[c][k]: nodal value
  // of component c at node k of the lane's z line
  static __device__ __forceinline__ void integrate(const TabT<P, Q, T> &tb, const T H[Q][3][3], T *slab,
                                                   const LanePos<Q> &lp, T out[3][N1]) {
#pragma unroll
    for (int c0 = 0; c0 < 3; c0 += NCG) {
      __syncwarp();
#pragma unroll
      for (int g = 0; g < NCG; ++g)
#pragma unroll
        for (int i = 0; i < N1; ++i) {
          T zx = 0, zy = 0, zz = 0;
#pragma unroll
          for (int s = 0; s < Q; ++s) {
            zx += tb.D[s][i] * H[s][c0 + g][0];
            zy += tb.N[s][i] * H[s][c0 + g][1];
            zz += tb.N[s][i] * H[s][c0 + g][2];
          }
          slab[g * BB + i * RB + lp.ln] = zx;
          slab[(NCG + g) * BB + i * RB + lp.ln] = zy;
          slab[(2 * NCG + g) * BB + i * RB + lp.ln] = zz;
        }
      __syncwarp();
      // lane (qz, i) = (a, b)
      T o1[NCG][N1], o2[NCG][N1];
      {
        const T *Z = slab + lp.r * L + lp.a * Q + lp.b * RB;
#pragma unroll
        for (int g = 0; g < NCG; ++g) {
          T zx[Q], zy[Q], zz[Q];
#pragma unroll
          for (int qy = 0; qy < Q; ++qy) {
            zx[qy] = Z[g * BB + qy];
            zy[qy] = Z[(NCG + g) * BB + qy];
            zz[qy] = Z[(2 * NCG + g) * BB + qy];
          }
#pragma unroll
          for (int j = 0; j < N1; ++j) {
            T s1 = 0, s2 = 0;
#pragma unroll
            for (int qy = 0; qy < Q; ++qy) {
              s1 += tb.N[qy][j] * zx[qy];
              s1 += tb.D[qy][j] * zy[qy];
              s2 += tb.N[qy][j] * zz[qy];
            }
            o1[g][j] = s1;
            o2[g][j] = s2;
          }
        }
      }
      __syncwarp();
#pragma unroll
      for (int g = 0; g < NCG; ++g)
#pragma unroll
        for (int j = 0; j < N1; ++j) {
          slab[g * BA + j * RA + lp.ln] = o1[g][j];
          slab[(NCG + g) * BA + j * RA + lp.ln] = o2[g][j];
        }
      __syncwarp();
      // lane (j, i) = (a, b)
      const T *Y = slab + lp.r * L + lp.b + lp.a * RA;
#pragma unroll
      for (int g = 0; g < NCG; ++g) {
        T y1[Q], y2[Q];
#pragma unroll
        for (int qz = 0; qz < Q; ++qz) {
          y1[qz] = Y[g * BA + qz * Q];
          y2[qz] = Y[(NCG + g) * BA + qz * Q];
        }
#pragma unroll
        for (int k = 0; k < N1; ++k) {
          T s = 0;
#pragma unroll
          for (int qz = 0; qz < Q; ++qz) {
            s += tb.N[qz][k] * y1[qz];
            s += tb.D[qz][k] * y2[qz];
          }
          out[c0 + g][k] = s;
        }
      }
    }
  }
};

template <int P, int Q, typename T>
struct SF {
  static constexpr int N1 = P + 1, NN = N1 * N1 * N1, NQ = Q * Q * Q;
  static constexpr int QPL = (NQ + 31) / 32;   // quadrature points per lane
  static constexpr int NPL = (NN + 31) / 32;   // nodes per lane
  static constexpr int NA = 3 * N1 * N1 * Q;   // x-sweep outputs per field
  static constexpr int NB = 3 * N1 * Q * Q;    // y-sweep outputs per field
  static constexpr int SZ1 = (3 * NN > 9 * NQ) ? 3 * NN : 9 * NQ;
  static constexpr int SZ2 = 2 * NA;
  static constexpr int SZ3 = 3 * NB;
  static constexpr int SZ = SZ1 + SZ2 + SZ3;   // per-warp slab (elements of T)
  static constexpr int TAB = 2 * Q * N1;        // sN + sD

  // nodal values V[c][k][j][i] (c*NN + node) -> G[i][c][e] at the owned points
  static __device__ __forceinline__ void eval(const T *__restrict__ sN, const T *__restrict__ sD,
                                              const T *V, T *A, T *B, int lane, T G[QPL][3][3]) {
    for (int it = lane; it < NA; it += 32) {
      const int qx = it % Q, r = it / Q;
      const T *v = V + r * N1;
      T s0 = 0, s1 = 0;
#pragma unroll
      for (int i = 0; i < N1; ++i) {
        const T x = v[i];
        s0 += sN[qx * N1 + i] * x;
        s1 += sD[qx * N1 + i] * x;
      }
      A[it] = s0;
      A[NA + it] = s1;
    }
    __syncwarp();
    for (int it = lane; it < NB; it += 32) {
      const int qx = it % Q, qy = (it / Q) % Q, ck = it / (Q * Q);
      T s00 = 0, s01 = 0, s10 = 0;
#pragma unroll
      for (int j = 0; j < N1; ++j) {
        const T a0 = A[(ck * N1 + j) * Q + qx], a1 = A[NA + (ck * N1 + j) * Q + qx];
        const T nn = sN[qy * N1 + j], dd = sD[qy * N1 + j];
        s00 += nn * a0;
        s01 += dd * a0;
        s10 += nn * a1;
      }
      B[it] = s00;
      B[NB + it] = s01;
      B[2 * NB + it] = s10;
    }
    __syncwarp();
#pragma unroll
    for (int l = 0; l < QPL; ++l) {
      const int q = lane + 32 * l;
      if (q < NQ) {
        const int qx = q % Q, qy = (q / Q) % Q, qz = q / (Q * Q);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          T gx = 0, gy = 0, gz = 0;
#pragma unroll
          for (int k = 0; k < N1; ++k) {
            const int b = ((c * N1 + k) * Q + qy) * Q + qx;
            const T nn = sN[qz * N1 + k];
            gx += nn * B[2 * NB + b];
            gy += nn * B[NB + b];
            gz += sD[qz * N1 + k] * B[b];
          }
          G[l][c][0] = gx;
          G[l][c][1] = gy;
          G[l][c][2] = gz;
        }
      }
    }
    __syncwarp();
  }

  // H[i][c][e] at owned points -> nodal values out[c][node] in smem Yout
  // (= the V region), the transpose of eval().
  static __device__ __forceinline__ void integrate(const T *__restrict__ sN, const T *__restrict__ sD,
                                                   const T H[QPL][3][3], T *Hs, T *Y, T *Z, int lane) {
#pragma unroll
    for (int l = 0; l < QPL; ++l) {
      const int q = lane + 32 * l;
      if (q < NQ) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int e = 0; e < 3; ++e) Hs[(c * 3 + e) * NQ + q] = H[l][c][e];
      }
    }
    __syncwarp();
    // z: Z[c][k][qy][qx] for the three gradient directions
    for (int it = lane; it < NB; it += 32) {
      const int qx = it % Q, qy = (it / Q) % Q, ck = it / (Q * Q);
      const int c = ck / N1, k = ck % N1;
      T sx = 0, sy = 0, sz = 0;
#pragma unroll
      for (int qz = 0; qz < Q; ++qz) {
        const int q = (qz * Q + qy) * Q + qx;
        const T nn = sN[qz * N1 + k];
        sx += nn * Hs[(c * 3 + 0) * NQ + q];
        sy += nn * Hs[(c * 3 + 1) * NQ + q];
        sz += sD[qz * N1 + k] * Hs[(c * 3 + 2) * NQ + q];
      }
      Z[it] = sx;
      Z[NB + it] = sy;
      Z[2 * NB + it] = sz;
    }
    __syncwarp();
    // y: Yx[c][k][j][qx], Yo[c][k][j][qx]
    for (int it = lane; it < NA; it += 32) {
      const int qx = it % Q, j = (it / Q) % N1, ck = it / (Q * N1);
      T sx = 0, so = 0;
#pragma unroll
      for (int qy = 0; qy < Q; ++qy) {
        const int z = (ck * Q + qy) * Q + qx;
        const T nn = sN[qy * N1 + j];
        sx += nn * Z[z];
        so += sD[qy * N1 + j] * Z[NB + z] + nn * Z[2 * NB + z];
      }
      Y[it] = sx;
      Y[NA + it] = so;
    }
    __syncwarp();
  }

  // final x sweep for node a = (i, j, k): 3 component values
  static __device__ __forceinline__ void integrate_node(const T *__restrict__ sN, const T *__restrict__ sD,
                                                        const T *Y, int a, T out[3]) {
    const int i = a % N1, jk = a / N1;  // jk = k*N1 + j
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int base = ((c * N1 * N1) + jk) * Q;
      T s = 0;
#pragma unroll
      for (int qx = 0; qx < Q; ++qx) s += sD[qx * N1 + i] * Y[base + qx] + sN[qx * N1 + i] * Y[NA + base + qx];
      out[c] = s;
    }
  }
};

// dst += the values of a lane's line, without atomics (a colour of the lattice:
// no other lane of the launch has the line's nodes): all loads before the
// first store, one round trip where value-by-value adds take one after the
// other (the compiler may not move a load over a store to the same vector).
// Entries whose component is constrained in the packed node ids are skipped.
template <int N1, typename T>
__device__ __forceinline__ void add_line_plain(T *dst, const int ck[N1], const T out[3][N1]) {
  T old[N1][3];
#pragma unroll
  for (int k = 0; k < N1; ++k)
#pragma unroll
    for (int i = 0; i < 3; ++i) old[k][i] = dst[3 * (size_t)(ck[k] & NODE_MASK) + i];
#pragma unroll
  for (int k = 0; k < N1; ++k)
#pragma unroll
    for (int i = 0; i < 3; ++i)
      if (!((ck[k] >> (NODE_BITS + i)) & 1)) dst[3 * (size_t)(ck[k] & NODE_MASK) + i] = old[k][i] + out[i][k];
}

// --------------------------------------------------------------- physics
// symmetric storage (0,0),(1,1),(2,2),(0,1),(0,2),(1,2)
__device__ __forceinline__ int sym_i(int I) { return I < 3 ? I : (I == 5 ? 1 : 0); }
__device__ __forceinline__ int sym_j(int I) { return I < 3 ? I : (I == 3 ? 1 : 2); }

template <typename T>
__device__ __forceinline__ T det3(const T F[3][3]) {
  return F[0][0] * (F[1][1] * F[2][2] - F[1][2] * F[2][1]) - F[0][1] * (F[1][0] * F[2][2] - F[1][2] * F[2][0]) +
         F[0][2] * (F[1][0] * F[2][1] - F[1][1] * F[2][0]);
}
template <typename T>
__device__ __forceinline__ T inv3(const T J[3][3], T Ji[3][3]) {
  const T d = det3(J);
  const T id = T(1) / d;
  Ji[0][0] = (J[1][1] * J[2][2] - J[1][2] * J[2][1]) * id;
  Ji[0][1] = (J[0][2] * J[2][1] - J[0][1] * J[2][2]) * id;
  Ji[0][2] = (J[0][1] * J[1][2] - J[0][2] * J[1][1]) * id;
  Ji[1][0] = (J[1][2] * J[2][0] - J[1][0] * J[2][2]) * id;
  Ji[1][1] = (J[0][0] * J[2][2] - J[0][2] * J[2][0]) * id;
  Ji[1][2] = (J[0][2] * J[1][0] - J[0][0] * J[1][2]) * id;
  Ji[2][0] = (J[1][0] * J[2][1] - J[1][1] * J[2][0]) * id;
  Ji[2][1] = (J[0][1] * J[2][0] - J[0][0] * J[2][1]) * id;
  Ji[2][2] = (J[0][0] * J[1][1] - J[0][1] * J[1][0]) * id;
  return d;
}

// Per-point state of the scalar variants (computed from the displacement).
template <typename T>
struct ScalarState {
  T F[3][3];
  T det;
};

// upper triangle of a symmetric N x N matrix, row by row
__host__ __device__ constexpr int tri_index(int N, int i, int j) {
  return i <= j ? i * N - i * (i - 1) / 2 + (j - i) : j * N - j * (j - 1) / 2 + (i - j);
}

// Q(g) of do_operation_on_cell (mf_nh_operator.h:922-1499) for the point
// whose record is rec[comp * CS] (rec already offset to the point; a pointer, or an
// accessor with operator[] such as the record pair of two cells); for the
// variants that fold JxW into their coefficients Q(g) comes out times JxW.
template <typename T, int VAR, int CS, typename R>
__device__ __forceinline__ void physics(const T g[3][3], const R &rec, T mu, T lambda, T kappa,
                                        const ScalarState<T> &st, T Qm[3][3]) {
  constexpr int CV = variant_cvar(VAR);
  T s[6];
#pragma unroll
  for (int I = 0; I < 6; ++I) s[I] = T(0.5) * (g[sym_i(I)][sym_j(I)] + g[sym_j(I)][sym_i(I)]);
  const T tr = s[0] + s[1] + s[2];
  if (VAR == VAR_TENSOR4) {
    // g * (tau/J) + C : sym(g)     (mf_nh_operator.h:1425-1440)
    T Ts[6];
#pragma unroll
    for (int I = 0; I < 6; ++I) Ts[I] = rec[(CV + I) * CS];
    T cs[6];
#pragma unroll
    for (int I = 0; I < 6; ++I) {
      T a = 0;
#pragma unroll
      for (int J = 0; J < 6; ++J) a += rec[(CV + 6 + tri_index(6, I, J)) * CS] * s[J];
      cs[I] = a;
    }
    const T T00 = Ts[0], T11 = Ts[1], T22 = Ts[2], T01 = Ts[3], T02 = Ts[4], T12 = Ts[5];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      Qm[i][0] = g[i][0] * T00 + g[i][1] * T01 + g[i][2] * T02;
      Qm[i][1] = g[i][0] * T01 + g[i][1] * T11 + g[i][2] * T12;
      Qm[i][2] = g[i][0] * T02 + g[i][1] * T12 + g[i][2] * T22;
    }
    Qm[0][0] += cs[0]; Qm[1][1] += cs[1]; Qm[2][2] += cs[2];
    Qm[0][1] += cs[3]; Qm[1][0] += cs[3];
    Qm[0][2] += cs[4]; Qm[2][0] += cs[4];
    Qm[1][2] += cs[5]; Qm[2][1] += cs[5];
  } else if (VAR == VAR_TENSOR2) {
    // c1 sym(g) + c2 tr(g) I + g * (tau/J)   (mf_nh_operator.h:1401-1424)
    const T c1 = rec[CV * CS], c2 = rec[(CV + 1) * CS];
    const T T00 = rec[(CV + 2) * CS], T11 = rec[(CV + 3) * CS], T22 = rec[(CV + 4) * CS];
    const T T01 = rec[(CV + 5) * CS], T02 = rec[(CV + 6) * CS], T12 = rec[(CV + 7) * CS];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      Qm[i][0] = g[i][0] * T00 + g[i][1] * T01 + g[i][2] * T02;
      Qm[i][1] = g[i][0] * T01 + g[i][1] * T11 + g[i][2] * T12;
      Qm[i][2] = g[i][0] * T02 + g[i][1] * T12 + g[i][2] * T22;
    }
#pragma unroll
    for (int I = 0; I < 6; ++I) {
      const int i = sym_i(I), j = sym_j(I);
      const T v = c1 * s[I] + (I < 3 ? c2 * tr : T(0));
      Qm[i][j] += v;
      if (i != j) Qm[j][i] += v;
    }
  } else if (VAR == VAR_TENSOR4_NS) {
    // out_ij = A_ijkl Grad v_kl (double_contract<2,0,3,1>, mf_nh_operator.h:1441-1455)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        T a = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int l = 0; l < 3; ++l) a += rec[(CV + tri_index(9, i * 3 + j, k * 3 + l)) * CS] * g[k][l];
        Qm[i][j] = a;
      }
  } else if (VAR == VAR_SCALAR_REF) {
    // mf_nh_operator.h:1255-1400: g = Grad v; grad_x v = Grad v F^-1; the
    // scalar-variant physics; submitted as (jc + grad_x v tau) F^-T
    const T c = rec[C_VAR * CS];
    T Fi[3][3];
    inv3(st.F, Fi);
    T gx[3][3];
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int e = 0; e < 3; ++e) gx[d][e] = g[d][0] * Fi[0][e] + g[d][1] * Fi[1][e] + g[d][2] * Fi[2][e];
    T tau[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const T b = st.F[i][0] * st.F[j][0] + st.F[i][1] * st.F[j][1] + st.F[i][2] * st.F[j][2];
        tau[i][j] = mu * b - (i == j ? c : T(0));
      }
    const T trx = gx[0][0] + gx[1][1] + gx[2][2];
    T qd[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        T v = c * (gx[i][j] + gx[j][i]);
        if (i == j) v += T(2) * lambda * trx;
        v += gx[i][0] * tau[0][j] + gx[i][1] * tau[1][j] + gx[i][2] * tau[2][j];
        qd[i][j] = v;
      }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) Qm[i][j] = qd[i][0] * Fi[j][0] + qd[i][1] * Fi[j][1] + qd[i][2] * Fi[j][2];
  } else if (VAR == VAR_SCALAR_F1) {
    // mf_nh_operator.h:1182-1254: tau = mu b - c I, jc = 2c sym + 2 lambda tr I
    const T c = rec[C_VAR * CS];
    T jc[6];
#pragma unroll
    for (int I = 0; I < 6; ++I) jc[I] = T(2) * c * s[I] + (I < 3 ? T(2) * lambda * tr : T(0));
    T tau[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const T b = st.F[i][0] * st.F[j][0] + st.F[i][1] * st.F[j][1] + st.F[i][2] * st.F[j][2];
        tau[i][j] = mu * b - (i == j ? c : T(0));
      }
    const T idet = T(1) / st.det;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        T geo = g[i][0] * tau[0][j] + g[i][1] * tau[1][j] + g[i][2] * tau[2][j];
        Qm[i][j] = geo;
      }
#pragma unroll
    for (int I = 0; I < 6; ++I) {
      const int i = sym_i(I), j = sym_j(I);
      Qm[i][j] += jc[I];
      if (i != j) Qm[j][i] += jc[I];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) Qm[i][j] *= idet;
  } else {
    // formulation 0 (vol/iso split), mf_nh_operator.h:1001-1181
    const T Jm13 = rec[C_VAR * CS];
    const T det_F = st.det;
    T bbar[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        bbar[i][j] = (st.F[i][0] * st.F[j][0] + st.F[i][1] * st.F[j][1] + st.F[i][2] * st.F[j][2]) * Jm13 * Jm13;
    const T c_1 = T(0.5) * mu;
    T tau_bar[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) tau_bar[i][j] = bbar[i][j] * (T(2) * c_1);
    const T tr_tau_bar = tau_bar[0][0] + tau_bar[1][1] + tau_bar[2][2];
    const T trd = tr_tau_bar * T(1.0 / 3.0);
    const T dPsi = (kappa / T(2)) * (det_F - T(1) / det_F);
    const T dPsi_J = dPsi * det_F;
    const T d2Psi = (kappa / T(2)) * (T(1) + T(1) / (det_F * det_F));
    T sym[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) sym[i][j] = T(0.5) * (g[i][j] + g[j][i]);
    T tis = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) tis += (tau_bar[i][j] - (i == j ? trd : T(0))) * sym[i][j];
    const T volI = det_F * (dPsi + det_F * d2Psi) * tr;
    const T two3 = T(2.0 / 3.0);
    const T idet = T(1) / det_F;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const T tau_iso = tau_bar[i][j] - (i == j ? trd : T(0));
        T v = sym[i][j] * (-dPsi_J * T(2));
        if (i == j) v += volI;
        v += (two3 * tr_tau_bar) * (sym[i][j] - (i == j ? tr * T(1.0 / 3.0) : T(0)));
        v -= (two3 * tr) * tau_iso;
        if (i == j) v -= two3 * tis;
        Qm[i][j] = v;
      }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const T tau_0j = tau_bar[0][j] + (0 == j ? dPsi_J - trd : T(0));
        const T tau_1j = tau_bar[1][j] + (1 == j ? dPsi_J - trd : T(0));
        const T tau_2j = tau_bar[2][j] + (2 == j ? dPsi_J - trd : T(0));
        const T geo = g[i][0] * tau_0j + g[i][1] * tau_1j + g[i][2] * tau_2j;
        Qm[i][j] = (Qm[i][j] + geo) * idet;
      }
  }
}

}  // namespace lsmf
