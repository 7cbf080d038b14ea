// Host plan of the fused step: recursive coordinate bisection of the nodes
// into patches, the elements that touch each patch's owned nodes, and their
// local indices.  Deterministic for any number of threads.
#include "patch.h"

#include <algorithm>
#include <array>
#include <atomic>
#include <cmath>
#include <exception>
#include <thread>

namespace akb {
namespace {

struct Range {
  int64_t b, e;
  int inst;
};

int host_threads(int64_t work) {
  const int64_t t = std::min<int64_t>(std::max(1u, std::thread::hardware_concurrency()), 16);
  return (int)std::max<int64_t>(1, std::min<int64_t>(t, work / 16000));
}

// f(first, last, t) on contiguous chunks of [0, n), one per thread; a chunk
// whose thread cannot be started runs here, an exception is rethrown here
template <class F> void chunked(int64_t n, int threads, const F &f) {
  std::vector<std::exception_ptr> error(threads);
  auto part = [&](int t) {
    try {
      f(n * t / threads, n * (t + 1) / threads, t);
    } catch (...) {
      error[t] = std::current_exception();
    }
  };
  std::vector<std::thread> pool;
  pool.reserve(threads);
  for (int t = 1; t < threads; ++t) {
    try {
      pool.emplace_back(part, t);
    } catch (...) {
      part(t);
    }
  }
  part(0);
  for (auto &p : pool) p.join();
  for (auto &x : error)
    if (x) std::rethrow_exception(x);
}

// Node planes of a box of n nodes with extents ext, were it a regular grid:
// the spacing h solves prod(ext_a / h + 1) = n.
double grid_spacing(const double *ext, int D, double n) {
  double hi = 0.;
  for (int a = 0; a < D; ++a) hi = std::max(hi, ext[a]);
  if (hi <= 0.) return 1.;
  double lo = hi / n;
  for (int it = 0; it < 20; ++it) {
    const double h = std::sqrt(lo * hi);
    double p = 1.;
    for (int a = 0; a < D; ++a) p *= ext[a] / h + 1.;
    (p > n ? lo : hi) = h;
  }
  return std::sqrt(lo * hi);
}

// What each instance's coordinates are multiplied by before the bisection: one
// over the mean extent of its elements along each axis where these differ (from
// a sample of the elements), so that boxes of equal sides hold equal numbers of
// cells.  Cut by lengths, a mesh of stretched cells has patches of one or two
// cells along its coarse axis, which evaluate 2.2 times its elements (100 x 100 x
// 2 cells in a unit cube, mixed, us per step: cut by lengths 10.9, two kernels
// 9.3; cubic cells 5.8).
std::vector<std::array<double, 3>> cell_scales(const PatchMesh &m) {
  struct Extent {
    double sum[3] = {0., 0., 0.};
  };
  std::vector<Extent> ext(m.ninst);
  const int64_t samples = std::min<int64_t>(m.E, 4096 + 64 * (int64_t)m.ninst);
  for (int64_t k = 0; k < samples; ++k) {
    const int64_t e = m.E / samples * k + m.E % samples * k / samples;
    const int64_t inst = m.ninst <= 1 ? 0
                                      : std::upper_bound(m.inst_off, m.inst_off + m.ninst,
                                                         (int64_t)m.conn[e]) - m.inst_off - 1;
    for (int a = 0; a < m.D; ++a) {
      double lo = 0., hi = 0.;
      for (int c = 0; c < m.NN; ++c) {
        const double x = m.X[(int64_t)m.conn[(int64_t)c * m.E + e] * m.D + a];
        lo = c == 0 ? x : std::min(lo, x);
        hi = c == 0 ? x : std::max(hi, x);
      }
      ext[inst].sum[a] += hi - lo;
    }
  }
  std::vector<std::array<double, 3>> scale(m.ninst, {1., 1., 1.});
  for (int k = 0; k < m.ninst; ++k) {
    const double *h = ext[k].sum;
    const double lo = *std::min_element(h, h + m.D), hi = *std::max_element(h, h + m.D);
    if (!(lo > 0.) || !std::isfinite(hi) || hi <= 1.2 * lo) continue;
    for (int a = 0; a < m.D; ++a) scale[k][a] = hi / h[a];
  }
  return scale;
}

// a node and its coordinates, moved together (the bisection then streams
// through memory instead of looking every coordinate up)
struct Item {
  double x[3];
  int32_t node;
};
struct Box {
  double lo[3], hi[3];
};

// Splits it[b, e) into leaves of at most max_own nodes.  The axis split is the
// one with the most patch edges in its extent, at the fraction that leaves
// whole patch edges on both sides, moved to the nearest plane of equal
// coordinates: regular grids are cut between their planes, into boxes.  box:
// bounds of the nodes (the halves take the split coordinate as theirs).
void bisect(const PatchMesh &m, std::vector<Item> &it, int64_t b, int64_t e, const Box &box,
            int inst, int depth, std::vector<Range> &out) {
  const int64_t n = e - b;
  if (n <= m.max_own) {
    if (n > 0) out.push_back({b, e, inst});
    return;
  }
  double ext[3];
  for (int a = 0; a < m.D; ++a) ext[a] = box.hi[a] - box.lo[a];
  const double edge = std::floor(std::pow((double)m.max_own, 1. / m.D) + 1e-9);
  const double h = grid_spacing(ext, m.D, (double)n);
  int axis = 0;
  for (int a = 1; a < m.D; ++a)
    if (ext[a] > ext[axis]) axis = a;
  const int64_t parts =
      std::max<int64_t>(2, (int64_t)std::ceil((ext[axis] / h + 1.) / edge - 1e-3));
  int64_t at = b + n * (parts / 2) / parts;
  at = std::min(std::max(at, b + 1), e - 1);
  std::nth_element(it.begin() + b, it.begin() + at, it.begin() + e,
                   [axis](const Item &x, const Item &y) {
                     return x.x[axis] < y.x[axis] || (x.x[axis] == y.x[axis] && x.node < y.node);
                   });
  // the plane of equal coordinates around the split point is [p0, p1)
  const double c = it[at].x[axis];
  const int64_t p0 = std::partition(it.begin() + b, it.begin() + at,
                                    [=](const Item &i) { return i.x[axis] < c; }) - it.begin();
  const int64_t p1 = std::partition(it.begin() + at, it.begin() + e,
                                    [=](const Item &i) { return i.x[axis] == c; }) - it.begin();
  if (p0 > b || p1 < e) at = (p0 > b && (at - p0 <= p1 - at || p1 == e)) ? p0 : p1;
  // the nodes next to the cut bound the halves
  Box half[2] = {box, box};
  half[0].hi[axis] = box.lo[axis];
  for (int64_t k = b; k < at; ++k) half[0].hi[axis] = std::max(half[0].hi[axis], it[k].x[axis]);
  half[1].lo[axis] = at == p1 ? box.hi[axis] : c;
  if (at == p1)
    for (int64_t k = at; k < e; ++k) half[1].lo[axis] = std::min(half[1].lo[axis], it[k].x[axis]);
  if (depth > 0 && n > 50000) {
    std::vector<Range> list[2];
    chunked(2, 2, [&](int64_t, int64_t, int t) {
      bisect(m, it, t ? at : b, t ? e : at, half[t], inst, depth - 1, list[t]);
    });
    for (auto &x : list) out.insert(out.end(), x.begin(), x.end());
  } else {
    bisect(m, it, b, at, half[0], inst, 0, out);
    bisect(m, it, at, e, half[1], inst, 0, out);
  }
}

// the whole of one instance
void bisect_all(const PatchMesh &m, std::vector<Item> &it, int64_t b, int64_t e, int inst,
                int depth, std::vector<Range> &out) {
  if (b == e) return;
  Box box;
  for (int a = 0; a < 3; ++a) box.lo[a] = box.hi[a] = it[b].x[a];
  for (int64_t k = b; k < e; ++k)
    for (int a = 0; a < m.D; ++a) {
      box.lo[a] = std::min(box.lo[a], it[k].x[a]);
      box.hi[a] = std::max(box.hi[a], it[k].x[a]);
    }
  bisect(m, it, b, e, box, inst, depth, out);
}

}  // namespace

PatchCaps patch_caps(int D, int64_t N, int64_t E, int ninst, int max_own) {
  // compact patches of s nodes per edge touch about ((s + 1) / s)^D times
  // their share of the elements and hold ((s + 2) / s)^D times their nodes;
  // s is taken at 0.6 of the full patch's (cuts at node planes leave some
  // patches partly filled), plus a few small patches
  const double s = std::max(1., 0.6 * std::pow((double)max_own, 1. / D));
  PatchCaps c;
  const int64_t few = 64 + 2 * (int64_t)ninst;
  c.patches = (int64_t)((double)N / (max_own * std::pow(0.6, D))) + few;
  c.elems = (int64_t)((double)E * std::pow((s + 1.) / s, D)) + 16 * c.patches;
  c.nodes = (int64_t)((double)N * std::pow((s + 2.) / s, D)) + 8 * few;
  return c;
}

bool build_patches(const PatchMesh &m, const PatchCaps &caps, PatchPlan &plan) {
  const int NN = m.NN;
  const int64_t N = m.N, E = m.E;
  plan = PatchPlan();
  plan.NNP = NN <= 4 ? 4 : 8;
  const int NNP = plan.NNP;
  if (N == 0 || E == 0 || m.max_own < 1) return false;
  // ---- patches of nodes, instance by instance
  std::vector<int32_t> idx(N);
  std::vector<Range> leaves;
  const int nt = host_threads(N);
  {
    std::vector<Item> it(N);
    const std::vector<std::array<double, 3>> scale = cell_scales(m);
    chunked(N, nt, [&](int64_t i0, int64_t i1, int) {
      int64_t inst = 0;
      for (int64_t i = i0; i < i1; ++i) {
        while (inst + 1 < m.ninst && i >= m.inst_off[inst + 1]) ++inst;
        for (int a = 0; a < m.D; ++a) it[i].x[a] = m.X[i * m.D + a] * scale[inst][a];
        for (int a = m.D; a < 3; ++a) it[i].x[a] = 0.;
        it[i].node = (int32_t)i;
      }
    });
    if (m.ninst <= 1) {
      bisect_all(m, it, 0, N, 0, nt > 1 ? 4 : 0, leaves);
    } else {
      std::vector<std::vector<Range>> part(nt);
      chunked(m.ninst, nt, [&](int64_t k0, int64_t k1, int t) {
        for (int64_t k = k0; k < k1; ++k)
          bisect_all(m, it, m.inst_off[k], m.inst_off[k + 1], (int)k, 0, part[t]);
      });
      for (auto &p : part) leaves.insert(leaves.end(), p.begin(), p.end());
    }
    chunked(N, nt, [&](int64_t i0, int64_t i1, int) {
      for (int64_t i = i0; i < i1; ++i) idx[i] = it[i].node;
    });
  }
  const int64_t P = (int64_t)leaves.size();
  if (P > caps.patches) return false;
  std::vector<int32_t> owner(N);
  chunked(P, nt, [&](int64_t p0, int64_t p1, int) {
    for (int64_t p = p0; p < p1; ++p) {
      std::sort(idx.begin() + leaves[p].b, idx.begin() + leaves[p].e);
      for (int64_t k = leaves[p].b; k < leaves[p].e; ++k) owner[idx[k]] = (int32_t)p;
    }
  });
  // ---- elements of each patch: those with a node it owns, ascending
  const int et = host_threads(E);
  struct Pair {
    int32_t patch, element;
  };
  std::vector<std::vector<Pair>> pairs(et);
  std::vector<std::vector<int32_t>> count(et, std::vector<int32_t>(P + 1, 0));
  chunked(E, et, [&](int64_t e0, int64_t e1, int t) {
    std::vector<Pair> &list = pairs[t];
    std::vector<int32_t> &c = count[t];
    list.reserve((size_t)((e1 - e0) * 1.7) + 64);
    for (int64_t e = e0; e < e1; ++e) {
      int32_t of[8];
      int k = 0;
      for (int a = 0; a < NN; ++a) {
        const int32_t p = owner[m.conn[(int64_t)a * E + e]];
        int j = 0;
        while (j < k && of[j] != p) ++j;
        if (j == k) of[k++] = p;
      }
      for (int j = 0; j < k; ++j) {
        list.push_back({of[j], (int32_t)e});
        c[of[j]]++;
      }
    }
  });
  plan.head.resize(P);
  int64_t total = 0;
  for (int64_t p = 0; p < P; ++p) {
    int64_t n = 0;
    for (int t = 0; t < et; ++t) {
      const int32_t c = count[t][p];
      count[t][p] = (int32_t)(total + n);
      n += c;
    }
    PatchHead &h = plan.head[p];
    h.chunk0 = (int32_t)(total / 32);
    h.n_elem = (int32_t)n;
    h.n_own = (int32_t)(leaves[p].e - leaves[p].b);
    h.own0 = (int32_t)leaves[p].b;
    h.inst = leaves[p].inst;
    h.mat = -1;
    h.pad[0] = h.pad[1] = h.pad[2] = 0;
    total += (n + 31) / 32 * 32;
    if (total > caps.elems) return false;
  }
  plan.elems.assign(total, 0);
  chunked(et, et, [&](int64_t t0, int64_t t1, int) {
    for (int64_t t = t0; t < t1; ++t)
      for (const Pair &x : pairs[t]) plan.elems[count[t][x.patch]++] = x.element;
  });
  // ---- local indices
  plan.conn.assign((size_t)total * NNP, 0);
  plan.slot.assign((size_t)total * NNP, kNoSlot);
  std::vector<std::vector<int32_t>> local(P);
  plan.own.resize(N);
  std::atomic<bool> ok{true};
  chunked(P, et, [&](int64_t p0, int64_t p1, int) {
    // node -> 1 + its index in the patch, 0 outside; cleared after each patch
    std::vector<int32_t> where(N, 0);
    std::vector<int32_t> corner, mine;
    for (int64_t p = p0; p < p1 && ok; ++p) {
      PatchHead &h = plan.head[p];
      const int32_t *el = plan.elems.data() + (size_t)h.chunk0 * 32;
      const int32_t *mine0 = idx.data() + leaves[p].b;
      std::vector<int32_t> &nodes = local[p];
      nodes.reserve(2 * h.n_own + h.n_elem);
      nodes.assign(mine0, mine0 + h.n_own);
      int kmax = 0;
      for (const int32_t node : nodes) {
        where[node] = 1;
        kmax = std::max(kmax, m.ptr[node + 1] - m.ptr[node]);
      }
      corner.resize((size_t)h.n_elem * NN);
      for (int a = 0; a < NN; ++a) {
        const int32_t *c = m.conn + (int64_t)a * E;
        for (int k = 0; k < h.n_elem; ++k) {
          const int32_t node = c[el[k]];
          corner[(size_t)k * NN + a] = node;
          if (!where[node]) {
            where[node] = 1;
            nodes.push_back(node);
          }
        }
      }
      std::sort(nodes.begin() + h.n_own, nodes.end());
      std::inplace_merge(nodes.begin(), nodes.begin() + h.n_own, nodes.end());
      h.n_local = (int32_t)nodes.size();
      h.n_slot = kmax * h.n_own;
      if (h.n_local >= 65536 || (int64_t)kmax * h.n_own >= kNoSlot) {
        ok = false;
        break;
      }
      // local index, and the index among the owned nodes (-1: halo)
      mine.assign(h.n_local, -1);
      for (int k = 0, i = 0; k < h.n_local; ++k) {
        where[nodes[k]] = k + 1;
        if (i < h.n_own && mine0[i] == nodes[k]) {
          mine[k] = i;
          plan.own[leaves[p].b + i] = {nodes[k], (uint16_t)k,
                                       (uint16_t)(m.ptr[nodes[k] + 1] - m.ptr[nodes[k]])};
          ++i;
        }
      }
      if (m.mat && h.n_elem > 0) {
        h.mat = m.mat[el[0]];
        for (int k = 1; k < h.n_elem; ++k)
          if (m.mat[el[k]] != h.mat) h.mat = -1;
      }
      uint16_t *lc = plan.conn.data() + (size_t)h.chunk0 * 32 * NNP;
      uint16_t *sc = plan.slot.data() + (size_t)h.chunk0 * 32 * NNP;
      for (int a = 0; a < NN; ++a) {
        const int32_t *pos = m.pos + (int64_t)a * E;
        for (int k = 0; k < h.n_elem; ++k) {
          const int32_t node = corner[(size_t)k * NN + a], l = where[node] - 1;
          lc[(size_t)k * NNP + a] = (uint16_t)l;
          if (mine[l] >= 0)
            sc[(size_t)k * NNP + a] =
                (uint16_t)((pos[el[k]] - m.ptr[node]) * h.n_own + mine[l]);
        }
      }
      for (const int32_t node : nodes) where[node] = 0;
    }
  });
  if (!ok) return false;
  int64_t nodes = 0;
  for (int64_t p = 0; p < P; ++p) {
    PatchHead &h = plan.head[p];
    h.node0 = (int32_t)nodes;
    nodes += h.n_local;
    plan.max_local = std::max(plan.max_local, h.n_local);
    plan.max_slots = std::max(plan.max_slots, h.n_slot);
  }
  if (nodes > caps.nodes) return false;
  plan.nodes.resize(nodes);
  for (int64_t p = 0; p < P; ++p)
    std::copy(local[p].begin(), local[p].end(), plan.nodes.begin() + plan.head[p].node0);
  return true;
}

bool check_patches(const PatchMesh &m, const PatchPlan &plan) {
  std::vector<int> owned(m.N, 0);
  std::vector<int64_t> writer;
  for (const PatchHead &h : plan.head) {
    if (h.node0 < 0 || h.n_local < 0 || (size_t)h.node0 + h.n_local > plan.nodes.size() ||
        h.own0 < 0 || (size_t)h.own0 + h.n_own > plan.own.size() || h.n_local > plan.max_local ||
        h.n_slot > plan.max_slots || h.n_own > m.max_own ||
        ((size_t)h.chunk0 + (h.n_elem + 31) / 32) * 32 > plan.elems.size())
      return false;
    const PatchOwn *own = plan.own.data() + h.own0;
    int valence = 0;
    for (int i = 0; i < h.n_own; ++i) {
      const PatchOwn o = own[i];
      if (o.node < 0 || o.node >= m.N || o.local >= h.n_local ||
          plan.nodes[h.node0 + o.local] != o.node ||
          o.valence != m.ptr[o.node + 1] - m.ptr[o.node])
        return false;
      owned[o.node]++;
      valence = std::max<int>(valence, o.valence);
    }
    if (h.n_slot != valence * h.n_own) return false;
    writer.assign(h.n_slot, -1);
    for (int k = 0; k < (h.n_elem + 31) / 32 * 32; ++k)
      for (int a = 0; a < m.NN; ++a) {
        const size_t at = ((size_t)h.chunk0 * 32 + k) * plan.NNP + a;
        const int l = plan.conn[at], s = plan.slot[at];
        if (k >= h.n_elem) {
          if (s != kNoSlot) return false;
          continue;
        }
        const int64_t e = plan.elems[(size_t)h.chunk0 * 32 + k];
        if (e < 0 || e >= m.E || l >= h.n_local) return false;
        const int32_t node = m.conn[(int64_t)a * m.E + e];
        if (plan.nodes[h.node0 + l] != node) return false;
        if (s == kNoSlot) continue;
        if (s >= h.n_slot || own[s % h.n_own].node != node || writer[s] >= 0 ||
            m.ptr[node] + s / h.n_own != m.pos[(int64_t)a * m.E + e])
          return false;
        writer[s] = e;
      }
    for (int i = 0; i < h.n_own; ++i)
      for (int r = 0; r < own[i].valence; ++r)
        if (writer[(size_t)r * h.n_own + i] < 0) return false;
  }
  for (const int n : owned)
    if (n != 1) return false;
  return true;
}

}  // namespace akb
