// Host side of the coarse-level solver's work distribution (coarse_plan.h).
#include "coarse_plan.h"

#include <algorithm>
#include <cmath>
#include <vector>

#include "op_dispatch.h"

namespace lsmf {

namespace {

// cells [first, last) into at most n parts of at most `cap` cells.  Cut
// along a whole layer of cells where both sides fit their share of the parts
// (the smaller the cut and the more even the sides the better): planar cuts
// keep the parts' surfaces, and so the sums to exchange, small (15^3 cells in
// parts of 24: 384 sums at most, 513 with cuts through layers).  Where no
// layer fits, cut through one.  The parts' ends are appended to `ends`.
void bisect(const Level &L, int *begin, int *first, int *last, int n, int cap, std::vector<int> &ends) {
  const int len = (int)(last - first);
  if (n == 1 || len <= cap) {
    std::sort(first, last);
    ends.push_back((int)(last - begin));
    return;
  }
  const int *ijk = L.cell_ijk.data();
  int lo[3] = {1 << 30, 1 << 30, 1 << 30}, hi[3] = {-1, -1, -1};
  for (int *it = first; it != last; ++it)
    for (int d = 0; d < 3; ++d) {
      lo[d] = std::min(lo[d], ijk[3 * (size_t)*it + d]);
      hi[d] = std::max(hi[d], ijk[3 * (size_t)*it + d]);
    }
  auto parts = [&](int cells) { return (cells + cap - 1) / cap; };
  const double scale = 1.0 / std::pow((double)len, 2.0 / 3.0);
  double best = 1e300;
  int ax = -1, at = 0, left = 0, nl = 0;
  for (int d = 0; d < 3; ++d) {
    std::vector<int> layer(hi[d] - lo[d] + 1, 0);
    for (int *it = first; it != last; ++it) ++layer[ijk[3 * (size_t)*it + d] - lo[d]];
    for (int cut = 1, l = 0; cut < (int)layer.size(); ++cut) {
      l += layer[cut - 1];
      if (l == 0 || l == len || parts(l) + parts(len - l) > n) continue;
      const double score = layer[cut - 1] * scale + 2.0 * std::abs(2 * l - len) / len;
      if (score < best) {
        best = score;
        ax = d;
        at = lo[d] + cut;
        left = l;
        nl = parts(l) + (int)((long long)(n - parts(l) - parts(len - l)) * l / len);
      }
    }
  }
  if (ax >= 0) {
    std::partition(first, last, [&](int c) { return ijk[3 * (size_t)c + ax] < at; });
  } else {
    ax = 0;
    for (int d = 1; d < 3; ++d)
      if (hi[d] - lo[d] > hi[ax] - lo[ax]) ax = d;
    nl = n / 2;
    left = (int)((long long)len * nl / n);
    left = std::max(left, len - (n - nl) * cap);  // both sides within their capacity
    left = std::min(left, nl * cap);
    const int o1 = (ax + 1) % 3, o2 = (ax + 2) % 3;
    std::nth_element(first, first + left, last, [&](int a, int b) {
      const int *p = ijk + 3 * (size_t)a, *q = ijk + 3 * (size_t)b;
      if (p[ax] != q[ax]) return p[ax] < q[ax];
      if (p[o2] != q[o2]) return p[o2] < q[o2];
      return p[o1] < q[o1];
    });
  }
  bisect(L, begin, first, first + left, nl, cap, ends);
  bisect(L, begin, first + left, last, n - nl, cap, ends);
}

}  // namespace

size_t coarse_tail_bytes(int max_nodes, int max_sums, size_t elem) {
  const int stride = elem == 4 ? 4 : 3;  // of a node's values (coarse_stride)
  return ((size_t)((stride * max_nodes + 3) / 4 * 4 + stride * max_sums) * elem + 15) / 16 * 16;
}

lsmf_status build_coarse_plan(const lsmf_op *op, int sms, size_t smem_limit, CoarsePlan &plan) {
  plan.usable = false;
  const Level &L = op->L();
  const OpsTable *t = L.q == L.p + 1 ? ops_for(L.p, op->precision == LSMF_FP32) : nullptr;
  if (!t || L.n_cells < 1) return LSMF_OK;
  const int nn = L.ncn();
  const size_t elem = op->elem(), stride = elem == 4 ? 4 : 3;
  CoarseShape sh;
  int W = 0;
  for (int w = 1; w <= COARSE_MAX_WARPS && !W; ++w) {
    sh = t->coarse_shape(op, w);
    if ((L.n_cells + sh.cells - 1) / sh.cells <= sms) W = w;
  }
  if (!W || W * sh.unit_bytes >= smem_limit) return LSMF_OK;
  if (((W - 1) * sh.unit_bytes + sh.out_offset) / elem + (size_t)sh.batch * nn * stride >= 65535) return LSMF_OK;
  std::vector<int> order(L.n_cells), ends;
  for (int c = 0; c < L.n_cells; ++c) order[c] = c;
  bisect(L, order.data(), order.data(), order.data() + L.n_cells, sms, sh.cells, ends);
  const int P = (int)ends.size();
  auto begin_of = [&](int p) { return p ? ends[p - 1] : 0; };
  // nodes of every part (in first-seen order), and the parts of every node in
  // part order (at most 8: a node has at most 8 cells)
  std::vector<int> part_nodes, node_off(P + 1, 0), seen(L.n_nodes, -1);
  std::vector<int> node_parts((size_t)L.n_nodes * 8);
  std::vector<uint8_t> n_parts(L.n_nodes, 0);
  part_nodes.reserve((size_t)L.n_nodes * 2);
  int max_nodes = 0;
  for (int p = 0; p < P; ++p) {
    for (int s = begin_of(p); s < ends[p]; ++s)
      for (int a = 0; a < nn; ++a) {
        const int n = L.cell_nodes[(size_t)order[s] * nn + a];
        if (seen[n] == p) continue;
        seen[n] = p;
        part_nodes.push_back(n);
        if (n_parts[n] == 8) return LSMF_OK;
        node_parts[8 * (size_t)n + n_parts[n]++] = p;
      }
    node_off[p + 1] = (int)part_nodes.size();
    max_nodes = std::max(max_nodes, node_off[p + 1] - node_off[p]);
  }
  // local order of a part's nodes: by falling number of sharing parts, nodes
  // shared with one part by that part, then by falling contributions; and the
  // exchange slots, consecutive in a part's local order, so that a line of
  // packets has one writer and mostly one reader (slots numbered by node, the
  // writers of a node side by side, cost 1.5 us a step)
  std::vector<int> count(L.n_nodes, 0), by(part_nodes.size()), node_slot((size_t)L.n_nodes * 8, -1);
  std::vector<uint64_t> keys;
  int n_slots = 0;
  for (int p = 0; p < P; ++p) {
    const int n0 = node_off[p], n1 = node_off[p + 1];
    for (int k = n0; k < n1; ++k) count[part_nodes[k]] = 0;
    for (int s = begin_of(p); s < ends[p]; ++s)
      for (int a = 0; a < nn; ++a) {
        int &c = count[L.cell_nodes[(size_t)order[s] * nn + a]];
        if (++c > 8) return LSMF_OK;
      }
    keys.resize(n1 - n0);
    for (int k = n0; k < n1; ++k) {
      const int n = part_nodes[k], m = n_parts[n];
      const int *np = &node_parts[8 * (size_t)n];
      const int other = m == 2 ? (np[0] == p ? np[1] : np[0]) : 0;
      keys[k - n0] = (uint64_t)(((8 - m) * 4096 + other) * 16 + (8 - count[n])) << 32 | (uint32_t)n;
    }
    std::sort(keys.begin(), keys.end());
    for (int k = n0; k < n1; ++k) by[k] = (int)(uint32_t)keys[k - n0];
    for (int k = n0; k < n1; ++k) {
      const int n = by[k];
      if (n_parts[n] < 2) break;
      int q = 0;
      while (node_parts[8 * (size_t)n + q] != p) ++q;
      node_slot[8 * (size_t)n + q] = n_slots++;
    }
    n_slots = (n_slots + 7) / 8 * 8;  // whole 128-byte lines
  }
  int max_items = 1, max_sums = 0;
  for (int p = 0; p < P; ++p) {
    int items = 0, sums = 0;
    for (int k = node_off[p]; k < node_off[p + 1]; ++k) {
      const int m = n_parts[part_nodes[k]];
      items += m - 1;
      sums += m > 1 ? m : 0;
    }
    max_items = std::max(max_items, items);
    max_sums = std::max(max_sums, sums);
  }
  const size_t smem = W * sh.unit_bytes + coarse_tail_bytes(max_nodes, max_sums, elem);
  if (smem > smem_limit || max_nodes > 4 * COARSE_THREADS || max_sums > 65535) return LSMF_OK;

  // one host image of the device lists: 4-byte, 2-byte, 1-byte arrays
  size_t bytes = 0;
  auto room = [&](size_t count, size_t size) {
    const size_t at = bytes;
    bytes = (bytes + count * size + 15) / 16 * 16;
    return at;
  };
  const size_t o_counts = room((size_t)4 * P, 4), o_cells = room((size_t)P * sh.cells, 4), o_nodes = room((size_t)P * max_nodes, 4),
               o_send = room((size_t)P * max_nodes, 4), o_slot = room((size_t)P * max_items, 4),
               o_lid = room((size_t)P * sh.cells * nn, 2), o_contrib = room((size_t)P * max_nodes * 8, 2),
               o_place = room((size_t)P * max_items, 2), o_first = room((size_t)P * max_nodes, 2),
               o_sums = room((size_t)P * max_nodes, 1);
  std::vector<uint8_t> img(bytes, 0);
  int *counts = (int *)&img[o_counts], *cells = (int *)&img[o_cells], *send = (int *)&img[o_send], *item_slot = (int *)&img[o_slot];
  unsigned *nodes = (unsigned *)&img[o_nodes];
  uint16_t *lid = (uint16_t *)&img[o_lid], *contrib = (uint16_t *)&img[o_contrib], *item_place = (uint16_t *)&img[o_place],
           *first = (uint16_t *)&img[o_first];
  uint8_t *sums = &img[o_sums];
  std::fill(send, send + (size_t)P * max_nodes, -1);
  std::fill(contrib, contrib + (size_t)P * max_nodes * 8, (uint16_t)0xffff);
  std::vector<int> local(L.n_nodes);
  for (int p = 0; p < P; ++p) {
    const int nc = ends[p] - begin_of(p), n_loc = node_off[p + 1] - node_off[p];
    const int *pn = &by[node_off[p]];
    for (int l = 0; l < n_loc; ++l) {
      local[pn[l]] = l;
      count[pn[l]] = 0;
    }
    for (int s = 0; s < sh.cells; ++s) {
      const int c = order[begin_of(p) + std::min(s, nc - 1)];
      cells[(size_t)p * sh.cells + s] = s < nc ? c : -1 - c;
      for (int a = 0; a < nn; ++a) {
        const int n = L.cell_nodes[(size_t)c * nn + a], l = local[n];
        lid[((size_t)p * sh.cells + s) * nn + a] = (uint16_t)l;
        if (s >= nc) continue;
        // results of unit s / batch: [cell][node][component]
        contrib[8 * ((size_t)p * max_nodes + l) + count[n]++] =
            (uint16_t)(((s / sh.batch) * sh.unit_bytes + sh.out_offset) / elem + ((size_t)(s % sh.batch) * nn + a) * stride);
      }
    }
    int it = 0, place = 0;
    for (int l = 0; l < n_loc; ++l) {
      const int n = pn[l], m = n_parts[n];
      const int *np = &node_parts[8 * (size_t)n];
      const size_t g = (size_t)p * max_nodes + l;
      nodes[g] = 2u * n + (np[0] == p ? 1u : 0u);
      if (m < 2) continue;
      first[g] = (uint16_t)place;
      for (int k = 0; k < m; ++k, ++place) {
        if (np[k] == p) {
          sums[g] = (uint8_t)(m | (k << 4));
          send[g] = node_slot[8 * (size_t)n + k];
        } else {
          item_slot[(size_t)p * max_items + it] = node_slot[8 * (size_t)n + k];
          item_place[(size_t)p * max_items + it++] = (uint16_t)place;
        }
      }
    }
    counts[4 * (size_t)p] = nc;
    counts[4 * (size_t)p + 1] = n_loc;
    counts[4 * (size_t)p + 2] = it;
  }
  plan.n_cta = P;
  plan.warps = W;
  plan.cells_per_cta = sh.cells;
  plan.max_nodes = max_nodes;
  plan.max_items = max_items;
  plan.max_sums = max_sums;
  plan.n_slots = n_slots;
  plan.packets = elem == 8 ? 2 : 1;
  plan.unit_bytes = sh.unit_bytes;
  plan.smem = smem;
  LSMF_TRY(plan.lists.upload(img.data(), img.size()));
  const uint8_t *d = plan.lists.ptr;
  plan.counts = (const int *)(d + o_counts);
  plan.cells = (const int *)(d + o_cells);
  plan.nodes = (const unsigned *)(d + o_nodes);
  plan.send = (const int *)(d + o_send);
  plan.item_slot = (const int *)(d + o_slot);
  plan.lid = (const uint16_t *)(d + o_lid);
  plan.contrib = (const uint16_t *)(d + o_contrib);
  plan.item_place = (const uint16_t *)(d + o_place);
  plan.first = (const uint16_t *)(d + o_first);
  plan.sums = d + o_sums;
  LSMF_TRY(plan.xbuf.alloc((size_t)2 * n_slots * plan.packets + (size_t)16 * P));
  plan.usable = true;
  return LSMF_OK;
}

}  // namespace lsmf
