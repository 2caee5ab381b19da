// Coarse-level solver kernel, included by op_kernels.cuh inside its
// namespace: the Chebyshev iteration of a level whose cells one CTA per SM
// takes (coarse_plan.h), as one cooperative launch.
//
// The coarse solve of the V-cycle takes hundreds of Chebyshev steps on a few
// thousand cells.  As two launches per step (cell loop, update) a step is
// bound by latency: launch and drain, index -> value -> record round trips
// to L2, atomics.  Here a CTA keeps its cells' records, index lists and its
// nodes' x in shared memory and the rest of their Chebyshev state in
// registers, so a step is
//   1. cell operator, from shared memory to shared memory (line sweeps)
//   2. a thread per node sums the cells' contributions; the sums of shared
//      nodes are stored to the exchange buffer
//   3. the other CTAs' sums are fetched, one per thread, into shared memory;
//      a node's thread adds them and its own in an order that is the same in
//      every CTA and updates its copy of the node.
// A sum travels as 16-byte packets that carry the step number beside the
// values and are stored and loaded as single 128-bit accesses, so data and
// flag arrive together: no barrier over the grid, no fence, one store and
// one load trip through L2 per step.  Two buffers alternate: a CTA stores
// step k + 2 only after it has seen step k + 1 of its neighbours, which they
// store after they have read step k.  Waits are bounded: a CTA that gives up
// stores NaN for its nodes, sets the operator's error word and returns, and
// so do the CTAs that wait for it (a CTA that owns no node matters only to
// those).
// A step at 15^3 Q2 cells (141 CTAs, tensor4) takes 3.7 us in FP32 and 5.4 us
// in FP64, where the two launches took 7.2 and 10.1 us.  Of the FP32 step the
// cell operator is 1.75 us (issue: two warps per scheduler), the exchange 1.2
// us (an L2 store and load trip), sums and update the rest; the FP64 operator
// is bound by shared-memory bandwidth (3.1 us: records and slabs of 24 cells).

template <int P, int Q, typename T, int VAR>
struct CoarseTraits {
  // tensor4 / tensor4_ns records in FP64 leave no room for the full slab
  static constexpr bool SMALL = sizeof(typename Num<T>::S) == 8 && (VAR == VAR_TENSOR4 || VAR == VAR_TENSOR4_NS);
  using S = SFC<P, Q, T, SMALL ? 1 : 3>;
  static constexpr bool SCALAR = VAR == VAR_SCALAR_F0 || VAR == VAR_SCALAR_F1;
};

// A node's three values in shared memory: padded to 16 bytes in FP32, one
// 128-bit access; packed in FP64, whose records leave no room
template <typename E>
__host__ __device__ constexpr int coarse_stride() { return sizeof(E) == 4 ? 4 : 3; }
__device__ __forceinline__ void ld3(const float *p, float v[3]) {
  const float4 t = *(const float4 *)p;
  v[0] = t.x;
  v[1] = t.y;
  v[2] = t.z;
}
__device__ __forceinline__ void ld3(const double *p, double v[3]) {
  v[0] = p[0];
  v[1] = p[1];
  v[2] = p[2];
}
__device__ __forceinline__ void st3(float *p, const float v[3]) { *(float4 *)p = make_float4(v[0], v[1], v[2], 0.f); }
__device__ __forceinline__ void st3(double *p, const double v[3]) {
  p[0] = v[0];
  p[1] = v[1];
  p[2] = v[2];
}

// shared memory of a working warp: record slices, reference metrics, slab
// (sweeps, then the cells' results), parked displacement gradients
template <int P, int Q, typename T, int VAR>
__host__ __device__ constexpr size_t coarse_slab_bytes() {
  using S = typename CoarseTraits<P, Q, T, VAR>::S;
  return (S::SZ * sizeof(T) + 15) / 16 * 16;
}
template <int P, int Q, typename T, int VAR>
__host__ __device__ inline size_t coarse_out_offset(int slice_elems) {
  constexpr int CPW = 32 / (Q * Q);
  const size_t rec = ((size_t)Q * (slice_elems / table_halves<typename Num<T>::S>()) * sizeof(T) + 15) / 16 * 16;
  const size_t ref = CoarseTraits<P, Q, T, VAR>::SCALAR ? ((size_t)9 * CPW * sizeof(T) + 15) / 16 * 16 : 0;
  return rec + ref;
}
template <int P, int Q, typename T, int VAR>
__host__ __device__ inline size_t coarse_unit_bytes(int slice_elems) {
  constexpr int LW = 32 / (Q * Q) * Q * Q;
  const size_t park = CoarseTraits<P, Q, T, VAR>::SCALAR ? (size_t)9 * Q * LW * sizeof(T) : 0;
  return (coarse_out_offset<P, Q, T, VAR>(slice_elems) + coarse_slab_bytes<P, Q, T, VAR>() + park + 15) / 16 * 16;
}

template <typename E>
struct CoarseArgs {
  int n_cta, warps, cells_per_cta, max_nodes, max_items, max_sums, n_slots;
  int unit_bytes;
  const int *counts, *cells, *send, *item_slot;
  const uint16_t *lid, *contrib, *item_place, *first;
  const unsigned *nodes;
  const uint8_t *sums;
  ulonglong2 *xbuf, *rbuf;
  const E *b, *invd;
  const uint8_t *cmask;
  E *x;
  double theta, delta;
  int degree;
};

// The units of a plan are as long as this kernel's, and the CTA has room for
// them and for what CoarseNodes keeps behind them
template <int P, int Q, typename T, int VAR, typename E>
__device__ __forceinline__ bool coarse_smem_short(const KArgs<E> &a, const CoarseArgs<E> &ca) {
  constexpr int XS = coarse_stride<E>();
  const size_t tail = ((size_t)((XS * ca.max_nodes + 3) / 4 * 4) + (size_t)XS * ca.max_sums) * sizeof(E);
  const bool unit = (size_t)ca.unit_bytes >= coarse_unit_bytes<P, Q, T, VAR>(a.slice_elems);
  return smem_short(unit ? (size_t)ca.warps * ca.unit_bytes + tail : ~(size_t)0, a.flag);
}

// NaN at the nodes a CTA stores: what x holds from an earlier call is not to
// be taken for a solution
template <typename E>
__device__ void coarse_no_solution(const CoarseArgs<E> &ca) {
  const unsigned *nodes = ca.nodes + (size_t)blockIdx.x * ca.max_nodes;
  for (int n = threadIdx.x; n < ca.counts[4 * blockIdx.x + 1]; n += blockDim.x)
    if (nodes[n] & 1)
      for (int i = 0; i < 3; ++i) ca.x[3 * (size_t)(nodes[n] >> 1) + i] = E(nan(""));
}

template <typename E>
CoarseArgs<E> coarse_args(const CoarsePlan &p) {
  CoarseArgs<E> c{};
  c.n_cta = p.n_cta;
  c.warps = p.warps;
  c.cells_per_cta = p.cells_per_cta;
  c.max_nodes = p.max_nodes;
  c.max_items = p.max_items;
  c.max_sums = p.max_sums;
  c.n_slots = p.n_slots;
  c.unit_bytes = (int)p.unit_bytes;
  c.counts = p.counts;
  c.cells = p.cells;
  c.send = p.send;
  c.item_slot = p.item_slot;
  c.lid = p.lid;
  c.contrib = p.contrib;
  c.item_place = p.item_place;
  c.first = p.first;
  c.nodes = p.nodes;
  c.sums = p.sums;
  c.xbuf = p.xbuf.ptr;
  c.rbuf = p.xbuf.ptr + (size_t)2 * p.n_slots * p.packets;
  return c;
}

// packets of a node's three values: the tag is the high word of the second
// half, so a packet is valid exactly when its tag is the step's
__device__ __forceinline__ void st_packet(ulonglong2 *p, unsigned long long x, unsigned long long y) {
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p), "l"(x), "l"(y)
               : "memory");
}
__device__ __forceinline__ ulonglong2 ld_packet(const ulonglong2 *p) {
  ulonglong2 v;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
               : "=l"(v.x), "=l"(v.y)
               : "l"(p)
               : "memory");
  return v;
}
// A load that comes before its packet is not only in vain: it leaves the old
// line in the reader's half of the L2, which the store has to invalidate
// first.  So a reader waits about as long as a store takes before it looks.
__device__ __forceinline__ void coarse_pause(int cycles) {
  const long long t0 = clock64();
  while (clock64() - t0 < cycles) {
  }
}
// measured at 15^3 / 8^3 Q2 cells (FP32, FP64): the reduction's lines have a
// reader in every CTA, an estimate's iteration takes 10.4 / 7.8 / 12.0 / 9.6
// us without a pause and 8.0 / 6.2 / 9.8 / 7.5 us with this one
constexpr int PAUSE_ALL_SUM = 800;
// exchange of shared nodes (one reader a line): FP32 15^3 Chebyshev step 3.75
// -> 3.63 us, estimate 7.67 -> 7.35 us; FP64 estimate 9.46 -> 9.4 us
template <typename E>
__host__ __device__ constexpr int pause_exchange() { return sizeof(E) == 4 ? 300 : 100; }
__device__ __forceinline__ unsigned packet_tag(const ulonglong2 &v) { return (unsigned)(v.y >> 32); }
template <typename E>
struct Packet;
template <>
struct Packet<float> {
  static constexpr int N = 1;
  static __device__ __forceinline__ void store(ulonglong2 *p, const float s[3], unsigned tag) {
    st_packet(p, ((unsigned long long)__float_as_uint(s[1]) << 32) | __float_as_uint(s[0]),
              ((unsigned long long)tag << 32) | __float_as_uint(s[2]));
  }
  static __device__ __forceinline__ void unpack(const ulonglong2 v[1], float *s) {
    s[0] = __uint_as_float((unsigned)v[0].x);
    s[1] = __uint_as_float((unsigned)(v[0].x >> 32));
    s[2] = __uint_as_float((unsigned)v[0].y);
  }
};
template <>
struct Packet<double> {
  static constexpr int N = 2;
  static __device__ __forceinline__ void store(ulonglong2 *p, const double s[3], unsigned tag) {
    const unsigned long long m = __double_as_longlong(s[1]), t = (unsigned long long)tag << 32;
    st_packet(p, __double_as_longlong(s[0]), t | (m & 0xffffffffull));
    st_packet(p + 1, __double_as_longlong(s[2]), t | (m >> 32));
  }
  static __device__ __forceinline__ void unpack(const ulonglong2 v[2], double *s) {
    s[0] = __longlong_as_double(v[0].x);
    s[1] = __longlong_as_double((v[1].y << 32) | (v[0].y & 0xffffffffull));
    s[2] = __longlong_as_double(v[1].x);
  }
};

// The cell operator of a CTA: one unit of CPW cells per working warp, one cell
// per lane in both precisions, records and index lists loaded once.
template <int P, int Q, typename T, int VAR>
struct CoarseCells {
  using E = typename Num<T>::S;
  static constexpr int TH = table_halves<E>();
  using TR = CoarseTraits<P, Q, T, VAR>;
  using S = typename TR::S;
  using RL = RecLayout<P, Q, TH>;
  static constexpr int N1 = P + 1, NN = S::NN, L = S::L, CPW = S::CPW, LW = S::LW;
  static constexpr int XS = coarse_stride<E>();
  static_assert(Num<T>::H == 1, "one cell per lane");
  static_assert(CPW * NN * XS <= S::SZ, "the cells' results fit in the slab");
  const TabT<P, Q, T> &tab;
  LanePos<Q> lp;
  T *rec, *ref, *slab, *park;
  int SS;
  bool ref_per_cell, active;
  int lid[N1];
  T mu, lambda, kappa;

  __device__ __forceinline__ CoarseCells(const KArgs<E> &a, const TabT<P, Q, T> &t, const CoarseArgs<E> &ca, unsigned char *smem)
      : tab(t) {
    const int warp = threadIdx.x >> 5, cta = blockIdx.x;
    const int n_cells = ca.counts[4 * cta];
    active = warp < ca.warps && warp * CPW < n_cells;
    ref_per_cell = a.ref_per_cell != 0;
    SS = a.slice_elems / TH;
    unsigned char *base = smem + (size_t)warp * ca.unit_bytes;
    rec = (T *)base;
    ref = (T *)(base + ((size_t)Q * SS * sizeof(T) + 15) / 16 * 16);
    slab = (T *)(base + coarse_out_offset<P, Q, T, VAR>(a.slice_elems));
    park = (T *)((unsigned char *)slab + coarse_slab_bytes<P, Q, T, VAR>()) + lp.ln;
    if (!active) return;
    const int slot = warp * CPW + lp.r;
    const int ce = ca.cells[(size_t)cta * ca.cells_per_cta + slot], cell = ce < 0 ? -1 - ce : ce;
    material<E>(a.mu[cell], a.nu, mu, lambda, kappa);
    const E *src = a.table + RL::base(cell, a.batch_elems) + lp.t * TH;
    const uint16_t *l = ca.lid + ((size_t)cta * ca.cells_per_cta + slot) * NN + lp.t;
#pragma unroll
    for (int k = 0; k < N1; ++k) lid[k] = XS * l[k * L];
    const int ncomp = TR::SCALAR && ref_per_cell ? C_VAR + 1 : variant_ncomp(VAR);
    for (int s = 0; s < Q; ++s)
      for (int c = 0; c < ncomp; ++c) rec[s * SS + c * LW + lp.ln] = src[(size_t)s * a.slice_elems + c * RL::CS];
    if constexpr (TR::SCALAR) {
      if (ref_per_cell && lp.t == 0) {
        const E *r = a.table + RL::ref(cell, a.batch_elems, a.slice_elems);
        for (int i = 0; i < 9; ++i) ref[i * CPW + lp.r] = r[i * RL::RS];
      }
      // the displacement gradients do not change during the solve
      T vu[3][N1], G[Q][3][3];
      const int *cn = a.cell_nodes + (size_t)cell * NN + lp.t;
#pragma unroll
      for (int k = 0; k < N1; ++k)
#pragma unroll
        for (int i = 0; i < 3; ++i) vu[i][k] = a.u[3 * (size_t)(cn[k * L] & NODE_MASK) + i];
      S::eval(tab, vu, slab, lp, G);
#pragma unroll
      for (int s = 0; s < Q; ++s)
#pragma unroll
        for (int i = 0; i < 9; ++i) park[(s * 9 + i) * LW] = G[s][i / 3][i % 3];
    }
    __syncwarp();
  }

  // results of the CTA's cells for the nodal values xg[XS * local node + c]
  // (constrained entries zero), into the warps' slabs
  __device__ __forceinline__ void apply(const E *xg) {
    if (!active) return;
    T v[3][N1], G[Q][3][3];
#pragma unroll
    for (int k = 0; k < N1; ++k) {
      E x[3];
      ld3(xg + lid[k], x);
#pragma unroll
      for (int i = 0; i < 3; ++i) v[i][k] = x[i];
    }
    S::eval(tab, v, slab, lp, G);
    T ux[3][Q];
    if (VAR == VAR_SCALAR_REF) {
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int m = 0; m < Q; ++m) ux[i][m] = rec[m * SS + (C_VAR + 1 + i) * LW + lp.ln];
    }
#pragma unroll
    for (int s = 0; s < Q; ++s)
      line_point<Q, T, VAR, LW, 1, LW>(G[s], s, (const T *)rec + s * SS + lp.r * L, (const T *)ref + lp.r, CPW, ref_per_cell,
                                       park + s * 9 * LW, ux, lp, tab.Dc, mu, lambda, kappa);
    T out[3][N1];
    S::integrate(tab, G, slab, lp, out);
    __syncwarp();
    E *ob = (E *)slab;
#pragma unroll
    for (int k = 0; k < N1; ++k) {
      const E o[3] = {out[0][k], out[1][k], out[2][k]};
      st3(ob + (lp.r * NN + k * L + lp.t) * XS, o);
    }
  }
};

// The nodes of a CTA: thread tid has the nodes tid + COARSE_THREADS * q.
// Shared nodes come first, so that their sums leave first.
template <typename E, int NPT>
struct CoarseNodes {
  static constexpr int PK = Packet<E>::N, XS = coarse_stride<E>();
  const E *units;  // shared memory, as elements
  E *xg, *recv;
  const int *item_slot;  // exchange slots of the items
  const uint16_t *item_place;  // ... and their places in recv
  ulonglong2 *xbuf;
  static constexpr int IB = 2;  // items of a thread that are fetched together
  int n_nodes, n_items, n_slots, my_slot[IB], my_place[IB];
  unsigned node[NPT];
  int send[NPT];
  unsigned meta[NPT];   // contributions | constrained components << 4 | sums << 8
  unsigned at[NPT][4];  // places of up to 8 contributions
  int first[NPT];       // the node's sums in recv, its own among them
  int own[NPT];
  E sum[NPT][3];

  __device__ __forceinline__ CoarseNodes(const CoarseArgs<E> &ca, unsigned char *smem) {
    const int cta = blockIdx.x, tid = threadIdx.x;
    units = (const E *)smem;
    xg = (E *)(smem + (size_t)ca.warps * ca.unit_bytes);
    recv = xg + (XS * ca.max_nodes + 3) / 4 * 4;
    n_nodes = ca.counts[4 * cta + 1];
    n_items = ca.counts[4 * cta + 2];
    n_slots = ca.n_slots;
    xbuf = ca.xbuf;
    item_slot = ca.item_slot + (size_t)cta * ca.max_items;
    item_place = ca.item_place + (size_t)cta * ca.max_items;
#pragma unroll
    for (int j = 0; j < IB; ++j) {
      const int i = tid + COARSE_THREADS * j;
      my_slot[j] = i < n_items ? item_slot[i] : 0;
      my_place[j] = i < n_items ? item_place[i] : 0;
    }
#pragma unroll
    for (int q = 0; q < NPT; ++q) {
      const int n = tid + COARSE_THREADS * q;
      node[q] = 0;
      send[q] = -1;
      meta[q] = 0;
      first[q] = own[q] = 0;
      if (n < n_nodes) {
        const size_t g = (size_t)cta * ca.max_nodes + n;
        node[q] = ca.nodes[g];
        send[q] = ca.send[g];
        const uint16_t *c = ca.contrib + 8 * g;
        int cnt = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          at[q][k] = (unsigned)c[2 * k] | ((unsigned)c[2 * k + 1] << 16);
          cnt += (c[2 * k] != 0xffff) + (c[2 * k + 1] != 0xffff);
        }
        const uint8_t *m = ca.cmask + 3 * (size_t)(node[q] >> 1);
        meta[q] = cnt | (m[0] ? 16u : 0u) | (m[1] ? 32u : 0u) | (m[2] ? 64u : 0u) | ((unsigned)(ca.sums[g] & 15) << 8);
        first[q] = ca.first[g];
        own[q] = first[q] + (ca.sums[g] >> 4);
      }
    }
  }
  __device__ __forceinline__ bool has(int q) const { return threadIdx.x + COARSE_THREADS * q < n_nodes; }
  __device__ __forceinline__ bool constrained(int q, int i) const { return (meta[q] >> (4 + i)) & 1; }
  // the node's values for the cells' gather: constrained entries read as zero
  __device__ __forceinline__ void put_x(int q, const double x[3]) {
    E v[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) v[i] = constrained(q, i) ? E(0) : E(x[i]);
    st3(xg + XS * (threadIdx.x + COARSE_THREADS * q), v);
  }

  // sum[q] = the CTA's contributions; the sums of shared nodes are sent
  __device__ __forceinline__ void sum_and_send(unsigned step) {
    ulonglong2 *buf = xbuf + (size_t)(step & 1) * n_slots * PK;
#pragma unroll
    for (int q = 0; q < NPT; ++q) {
      const int cnt = meta[q] & 15;
      E s[3] = {E(0), E(0), E(0)};
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (k < cnt) {
          E c[3];
          ld3(units + ((at[q][k / 2] >> (16 * (k & 1))) & 0xffff), c);
#pragma unroll
          for (int i = 0; i < 3; ++i) s[i] += c[i];
        }
      }
      if (send[q] >= 0) {
        Packet<E>::store(buf + (size_t)send[q] * PK, s, step);
        st3(recv + XS * own[q], s);
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) sum[q][i] = s[i];
    }
  }
  // the other CTAs' sums into recv.  false: a wait ran out
  __device__ __forceinline__ bool receive(unsigned step, int tries) {
    const ulonglong2 *buf = xbuf + (size_t)(step & 1) * n_slots * PK;
    coarse_pause(pause_exchange<E>());
    ulonglong2 v[IB][PK];
#pragma unroll
    for (int j = 0; j < IB; ++j)
      if (threadIdx.x + COARSE_THREADS * j < n_items)
#pragma unroll
        for (int k = 0; k < PK; ++k) v[j][k] = ld_packet(buf + (size_t)my_slot[j] * PK + k);
    bool ok = true;
#pragma unroll
    for (int j = 0; j < IB; ++j)
      if (threadIdx.x + COARSE_THREADS * j < n_items)
        ok = settle(buf + (size_t)my_slot[j] * PK, v[j], my_place[j], step, tries) && ok;
    for (int i = threadIdx.x + COARSE_THREADS * IB; i < n_items; i += COARSE_THREADS) {
      const ulonglong2 *p = buf + (size_t)__ldg(item_slot + i) * PK;
#pragma unroll
      for (int k = 0; k < PK; ++k) v[0][k] = ld_packet(p + k);
      ok = settle(p, v[0], __ldg(item_place + i), step, tries) && ok;
    }
    return ok;
  }
  __device__ __forceinline__ bool settle(const ulonglong2 *p, ulonglong2 v[PK], int place, unsigned step, int tries) {
    for (int t = 0;; ++t) {
      bool ok = true;
#pragma unroll
      for (int k = 0; k < PK; ++k) ok = ok && packet_tag(v[k]) == step;
      if (ok) break;
      if (t >= tries) return false;
#pragma unroll
      for (int k = 0; k < PK; ++k) v[k] = ld_packet(p + k);
    }
    E s[3];
    Packet<E>::unpack(v, s);
    st3(recv + XS * place, s);
    return true;
  }
  // A x at the thread's nodes without the identity rows, into sum: the CTAs'
  // sums in CTA order
  __device__ __forceinline__ void finish() {
#pragma unroll
    for (int q = 0; q < NPT; ++q) {
      const int m = meta[q] >> 8;
      if (m == 0) continue;
      E r[3] = {E(0), E(0), E(0)};
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (k < m) {
          E c[3];
          ld3(recv + XS * (first[q] + k), c);
#pragma unroll
          for (int i = 0; i < 3; ++i) r[i] += c[i];
        }
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) sum[q][i] = r[i];
    }
  }
};

// x = Chebyshev solution of A x = b after `degree` steps from zero
// (PreconditionChebyshev::vmult): the arithmetic of cheb_zero / cheb_step,
// in FP64 with x rounded to the level precision after every step.
template <int P, int Q, typename T, int VAR, int NPT>
__global__ void __launch_bounds__(COARSE_THREADS, 1)
    coarse_cheb_kernel(KArgs<T> a, TabT<P, Q, T> tab, CoarseArgs<T> ca) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int dead;
  if (coarse_smem_short<P, Q, T, VAR>(a, ca)) {
    coarse_no_solution(ca);
    return;
  }
  if (threadIdx.x == 0) dead = 0;
  CoarseCells<P, Q, T, VAR> cells(a, tab, ca, smem);
  CoarseNodes<T, NPT> nodes(ca, smem);
  double x[NPT][3], xo[NPT][3], b[NPT][3], iv[NPT][3];
#pragma unroll
  for (int q = 0; q < NPT; ++q) {
    if (!nodes.has(q)) continue;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const size_t d = 3 * (size_t)(nodes.node[q] >> 1) + i;
      b[q][i] = (double)ca.b[d];
      iv[q][i] = (double)ca.invd[d];
      x[q][i] = (double)T(iv[q][i] * b[q][i] * (1.0 / ca.theta));
      xo[q][i] = 0.0;
    }
    nodes.put_x(q, x[q]);
  }
  __syncthreads();
  double rhok = ca.delta / ca.theta;
  const double sigma = ca.theta / ca.delta;
  for (int k = 1; k < ca.degree; ++k) {
    cells.apply(nodes.xg);
    __syncthreads();
    nodes.sum_and_send((unsigned)k);
    // the step's coefficients, while the sums are on their way
    const double rhokp = 1. / (2. * sigma - rhok), f1 = rhokp * rhok, f2 = 2. * rhokp / ca.delta;
    rhok = rhokp;
    if (!nodes.receive((unsigned)k, a.wait_tries)) dead = 1;
    __syncthreads();
    if (dead) break;
    nodes.finish();
#pragma unroll
    for (int q = 0; q < NPT; ++q) {
      if (!nodes.has(q)) continue;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const double xi = x[q][i];
        const double ax = nodes.constrained(q, i) ? xi : (double)nodes.sum[q][i];
        const double xn = xi + f1 * (xi - xo[q][i]) + f2 * iv[q][i] * (b[q][i] - ax);
        xo[q][i] = xi;
        x[q][i] = (double)T(xn);
      }
      nodes.put_x(q, x[q]);
    }
    __syncthreads();
  }
  if (dead) {
    coarse_no_solution(ca);
    if (threadIdx.x == 0) atomicOr(a.flag, FLAG_TIMEOUT);
    return;
  }
#pragma unroll
  for (int q = 0; q < NPT; ++q) {
    if (!nodes.has(q) || !(nodes.node[q] & 1)) continue;
#pragma unroll
    for (int i = 0; i < 3; ++i) ca.x[3 * (size_t)(nodes.node[q] >> 1) + i] = T(x[q][i]);
  }
}

// Sums of v[0..NV) over all CTAs, the same bits in every thread of every CTA:
// each CTA's sums go out as tagged packets and every CTA adds all of them in
// CTA order.  Two buffers alternate (a CTA stores reduction r + 2 after it
// has seen every CTA's r + 1, which they store after reading r).
template <int NV>
__device__ __forceinline__ bool coarse_all_sum(double v[NV], ulonglong2 *rbuf, int n_cta, unsigned tag, int tries,
                                               double (*sh)[COARSE_MAX_WARPS][2]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto warp_sum = [&](double x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
  };
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const double s = warp_sum(v[j]);
    if (lane == 0) sh[0][warp][j] = s;
  }
  __syncthreads();
  // a line of its own for every writer
  constexpr int STRIDE = 8;
  ulonglong2 *buf = rbuf + (size_t)(tag & 1) * n_cta * STRIDE;
  if (threadIdx.x < NV) {
    double s = 0;
#pragma unroll
    for (int w = 0; w < COARSE_MAX_WARPS; ++w) s += sh[0][w][threadIdx.x];
    st_packet(buf + STRIDE * blockIdx.x + threadIdx.x, __double_as_longlong(s), (unsigned long long)tag << 32);
  }
  bool ok = true;
  double r[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) r[j] = 0;
  if (threadIdx.x < n_cta) {
    coarse_pause(PAUSE_ALL_SUM);
    const ulonglong2 *p = buf + STRIDE * threadIdx.x;
    for (int t = 0;; ++t) {
      bool all = true;
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        const ulonglong2 q = ld_packet(p + j);
        r[j] = __longlong_as_double(q.x);
        all = all && packet_tag(q) == tag;
      }
      if (all) break;
      if (t >= tries) {
        ok = false;
        break;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const double s = warp_sum(r[j]);
    if (lane == 0) sh[1][warp][j] = s;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    double s = 0;
#pragma unroll
    for (int w = 0; w < COARSE_MAX_WARPS; ++w) s += sh[1][w][j];
    v[j] = s;
  }
  return ok;
}

struct CoarseEigArgs {
  double mean;                          // of i mod 11 over the dofs
  double tol_abs, tol_rel;
  int max_it;
  double *alpha, *beta, *res2;          // history
  int *its;
};

// The eigenvalue estimate's CG (Jacobi, start vector (i mod 11) - mean) with
// its three dot products reduced over the CTAs: the arithmetic of eig_start /
// eig_dh / eig_update_precond / eig_dir_clear, stopped at the tolerance.  An
// iteration at 15^3 Q2 cells takes 7.4 us (FP32) / 9.4 us (FP64), of which the
// two reductions are about 3 us, where a cell loop and five vector and
// reduction launches took 18 / 20 us.
template <int P, int Q, typename T, int VAR, int NPT>
__global__ void __launch_bounds__(COARSE_THREADS, 1)
    coarse_eig_kernel(KArgs<T> a, TabT<P, Q, T> tab, CoarseArgs<T> ca, CoarseEigArgs ea) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ double sh[2][COARSE_MAX_WARPS][2];
  __shared__ int dead;
  if (coarse_smem_short<P, Q, T, VAR>(a, ca)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *ea.its = 0;
    return;
  }
  if (threadIdx.x == 0) dead = 0;
  CoarseCells<P, Q, T, VAR> cells(a, tab, ca, smem);
  CoarseNodes<T, NPT> nodes(ca, smem);
  T g[NPT][3], d[NPT][3], iv[NPT][3];
  double s[2] = {0, 0};
#pragma unroll
  for (int q = 0; q < NPT; ++q) {
    if (!nodes.has(q)) continue;
    const bool own = nodes.node[q] & 1;
    double dd[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const size_t dof = 3 * (size_t)(nodes.node[q] >> 1) + i;
      iv[q][i] = ca.invd[dof];
      g[q][i] = T(ea.mean - (double)(dof % 11));
      const T h = T(1) * iv[q][i] * g[q][i];
      d[q][i] = -h;
      dd[i] = (double)d[q][i];
      if (own) {
        s[0] += (double)g[q][i] * (double)g[q][i];
        s[1] += (double)g[q][i] * (double)h;
      }
    }
    nodes.put_x(q, dd);
  }
  __syncthreads();
  unsigned tag = 1;
  auto all_sum = [&](auto &v, auto nv) {
    if (!coarse_all_sum<decltype(nv)::value>(v, ca.rbuf, ca.n_cta, tag++, a.wait_tries, sh)) dead = 1;
  };
  all_sum(s, std::integral_constant<int, 2>{});
  double gh = s[1];
  const double res0 = sqrt(s[0]);
  const double tol = fmax(ea.tol_abs, ea.tol_rel * res0);
  int its = 0;
  bool done = !(res0 > tol) || ea.max_it < 1;
  while (!done) {
    const int k = its++;
    cells.apply(nodes.xg);
    __syncthreads();
    nodes.sum_and_send((unsigned)(k + 1));
    if (!nodes.receive((unsigned)(k + 1), a.wait_tries)) dead = 1;
    __syncthreads();
    if (dead) break;
    nodes.finish();
    double dh[1] = {0};
#pragma unroll
    for (int q = 0; q < NPT; ++q) {
      if (!nodes.has(q)) continue;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        if (nodes.constrained(q, i)) nodes.sum[q][i] = d[q][i];  // identity rows
        if (nodes.node[q] & 1) dh[0] += (double)d[q][i] * (double)nodes.sum[q][i];
      }
    }
    all_sum(dh, std::integral_constant<int, 1>{});
    const double alpha = gh / dh[0];
    s[0] = s[1] = 0;
    T h[NPT][3];
#pragma unroll
    for (int q = 0; q < NPT; ++q) {
      if (!nodes.has(q)) continue;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        g[q][i] = T((double)g[q][i] + alpha * (double)nodes.sum[q][i]);
        h[q][i] = T(1) * iv[q][i] * g[q][i];
        if (nodes.node[q] & 1) {
          s[0] += (double)g[q][i] * (double)g[q][i];
          s[1] += (double)g[q][i] * (double)h[q][i];
        }
      }
    }
    all_sum(s, std::integral_constant<int, 2>{});
    const double beta = s[1] / gh;
    gh = s[1];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      ea.alpha[k] = alpha;
      ea.beta[k] = beta;
      ea.res2[k] = s[0];
    }
    done = sqrt(s[0]) <= tol || its >= ea.max_it;
#pragma unroll
    for (int q = 0; q < NPT; ++q) {
      if (!nodes.has(q)) continue;
      double dd[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        d[q][i] = T(beta * (double)d[q][i] - (double)h[q][i]);
        dd[i] = (double)d[q][i];
      }
      nodes.put_x(q, dd);
    }
    __syncthreads();
    if (dead) break;
  }
  __syncthreads();  // the first reduction's outcome, where the loop was not entered
  if (threadIdx.x == 0) {
    if (dead) atomicOr(a.flag, FLAG_TIMEOUT);
    if (blockIdx.x == 0) *ea.its = its;
  }
}
