// Host plan of the fused step: recursive coordinate bisection of the nodes
// into patches, the elements that touch each patch's owned nodes, and their
// local indices.  Deterministic for any number of threads.
#include "patch.h"

#include <algorithm>
#include <array>
#include <atomic>
#include <cmath>
#include <condition_variable>
#include <exception>
#include <functional>
#include <mutex>
#include <thread>
#include <utility>

namespace akb {
namespace {

using Range = PatchRange;

// Threads for the plan of a mesh: its initialisation goes on meanwhile, and
// others may be at theirs.
int host_threads(int64_t work) {
  const int64_t most = std::min<int64_t>(std::max(1u, std::thread::hardware_concurrency()), 8);
  return (int)std::min<int64_t>(most, 1 + work / 8000);
}

// The plan's threads, started once: its phases are too short to start threads
// for each.  Every phase is cut into parts() parts whatever number of threads
// could be started.
class Workers {
  using Part = std::function<void(int)>;

 public:
  explicit Workers(int parts) : parts_(parts), error_(parts) {
    pool_.reserve(parts - 1);
    for (int t = 1; t < parts; ++t) {
      try {
        pool_.emplace_back([this] { serve(); });
      } catch (const std::exception &) {
        break;  // the parts run on the threads there are
      }
    }
  }
  ~Workers() {
    {
      std::lock_guard<std::mutex> lock(mu_);
      stop_ = true;
    }
    wake_.notify_all();
    for (auto &p : pool_) p.join();
  }
  int parts() const { return parts_; }
  // f(first, last, part) on contiguous pieces of [0, n); an exception of one is
  // rethrown here
  template <class F> void chunked(int64_t n, const F &f) {
    run([&](int t) { f(n * t / parts_, n * (t + 1) / parts_, t); });
  }

 private:
  void run(const Part &part) {
    {
      std::lock_guard<std::mutex> lock(mu_);
      part_ = &part;
      next_ = 0;
      left_ = parts_;
    }
    if (!pool_.empty()) wake_.notify_all();
    std::unique_lock<std::mutex> lock(mu_);
    take_parts(lock);
    done_.wait(lock, [this] { return left_ == 0; });
    part_ = nullptr;
    for (auto &x : error_)
      if (x) std::rethrow_exception(std::exchange(x, nullptr));
  }
  void take_parts(std::unique_lock<std::mutex> &lock) {
    while (part_ && next_ < parts_) {
      const int t = next_++;
      const Part &part = *part_;
      lock.unlock();
      std::exception_ptr error;
      try {
        part(t);
      } catch (...) {
        error = std::current_exception();
      }
      lock.lock();
      error_[t] = error;
      if (--left_ == 0) done_.notify_one();
    }
  }
  void serve() {
    std::unique_lock<std::mutex> lock(mu_);
    while (!stop_) {
      wake_.wait(lock, [this] { return stop_ || (part_ && next_ < parts_); });
      take_parts(lock);
    }
  }
  const int parts_;
  std::vector<std::exception_ptr> error_;
  std::vector<std::thread> pool_;
  std::mutex mu_;
  std::condition_variable wake_, done_;
  const Part *part_ = nullptr;
  int next_ = 0, left_ = 0;
  bool stop_ = false;
};

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
                                                         (int64_t)m.elements[e * m.NN]) - m.inst_off - 1;
    for (int a = 0; a < m.D; ++a) {
      double lo = 0., hi = 0.;
      for (int c = 0; c < m.NN; ++c) {
        const double x = m.X[(int64_t)m.elements[e * m.NN + c] * m.D + a];
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
// nodes [b, e) of the bisection, ascending, and their bounds
struct Part {
  Range r;
  Box box;
};

// Splits a part of more than max_own nodes in two.  The axis split is the one
// with the most patch edges in its extent, at the fraction that leaves whole
// patch edges on both sides, moved to the nearest plane of equal coordinates:
// regular grids are cut between their planes, into boxes.  The half that the cut
// does not touch takes the split coordinate as its bound.  The coordinate of that
// rank is found from a histogram and the nodes of one of its bins, and the nodes
// are moved once, in order (through tmp): 5 passes of a few ns per node, where a
// selection by swaps took 27.
void split(const PatchMesh &m, Item *it, Item *tmp, const Part &p, Part half[2]) {
  constexpr int kBins = 256;
  const int64_t b = p.r.b, e = p.r.e, n = e - b;
  double ext[3] = {0., 0., 0.};
  for (int a = 0; a < m.D; ++a) ext[a] = p.box.hi[a] - p.box.lo[a];
  const double edge = std::floor(std::pow((double)m.max_own, 1. / m.D) + 1e-9);
  const double h = grid_spacing(ext, m.D, (double)n);
  int axis = 0;
  for (int a = 1; a < m.D; ++a)
    if (ext[a] > ext[axis]) axis = a;
  const int64_t parts =
      std::max<int64_t>(2, (int64_t)std::ceil(std::min((ext[axis] / h + 1.) / edge, (double)n) - 1e-3));
  int64_t at = n * (parts / 2) / parts;
  at = std::min(std::max<int64_t>(at, 1), n - 1);
  // bins of equal width
  const double lo = p.box.lo[axis], per = ext[axis] > 0. ? (kBins - 1) / ext[axis] : 0.;
  auto bin = [=](const Item &i) {
    const double k = (i.x[axis] - lo) * per;
    return k > 0. ? (int)std::min(k, (double)(kBins - 1)) : 0;
  };
  int64_t count[kBins] = {0};
  for (int64_t k = b; k < e; ++k) ++count[bin(it[k])];
  int at_bin = 0;
  int64_t below = 0;
  while (below + count[at_bin] <= at) below += count[at_bin++];
  std::vector<double> x;
  x.reserve(count[at_bin]);
  for (int64_t k = b; k < e; ++k)
    if (bin(it[k]) == at_bin) x.push_back(it[k].x[axis]);
  std::nth_element(x.begin(), x.begin() + (at - below), x.end());
  // the plane of equal coordinates around the split point is [p0, p1)
  const double c = x[at - below];
  int64_t p0 = below, p1 = below;
  for (const double v : x) {
    p0 += v < c;
    p1 += v <= c;
  }
  const bool cut = p0 > 0 || p1 < n;
  if (cut) at = (p0 > 0 && (at - p0 <= p1 - at || p1 == n)) ? p0 : p1;
  const bool with_plane = at == p1;  // the plane belongs to the first half
  Item *first = it + b, *second = tmp + b;
  double hi0 = p.box.lo[axis], lo1 = p.box.hi[axis];
  int64_t taken = 0;
  for (int64_t k = b; k < e; ++k) {
    const Item i = it[k];
    const double v = i.x[axis];
    const bool left = cut ? (with_plane ? v <= c : v < c) : taken < at;
    if (left) {
      hi0 = std::max(hi0, v);
      *first++ = i;
      ++taken;
    } else {
      lo1 = std::min(lo1, v);
      *second++ = i;
    }
  }
  std::copy(tmp + b, second, first);
  half[0] = half[1] = p;
  half[0].r.e = half[1].r.b = b + taken;
  half[0].box.hi[axis] = hi0;
  half[1].box.lo[axis] = with_plane ? lo1 : c;
}

// the leaves of a part, of at most max_own nodes, in order
void bisect(const PatchMesh &m, Item *it, Item *tmp, const Part &p, std::vector<Range> &out) {
  if (p.r.e - p.r.b <= m.max_own) {
    if (p.r.e > p.r.b) out.push_back(p.r);
    return;
  }
  Part half[2];
  split(m, it, tmp, p, half);
  bisect(m, it, tmp, half[0], out);
  bisect(m, it, tmp, half[1], out);
}

// the nodes' patches, instance by instance: every leaf's nodes in idx, ascending
std::vector<Range> leaves_of(const PatchMesh &m, Workers &w, int32_t *idx) {
  const int64_t N = m.N;
  std::unique_ptr<Item[]> it(new Item[N]), tmp(new Item[N]);
  const std::vector<std::array<double, 3>> scale = cell_scales(m);
  std::vector<std::vector<Part>> part(w.parts());
  std::vector<Part> all;
  w.chunked(N, [&](int64_t i0, int64_t i1, int) {
    int64_t inst = std::upper_bound(m.inst_off, m.inst_off + m.ninst, i0) - m.inst_off - 1;
    for (int64_t i = i0; i < i1; ++i) {
      while (inst + 1 < m.ninst && i >= m.inst_off[inst + 1]) ++inst;
      for (int a = 0; a < 3; ++a) {
        const double x = a < m.D ? m.X[i * m.D + a] * scale[inst][a] : 0.;
        // (what is no number has an order, and no difference overflows)
        it[i].x[a] = std::isnan(x) ? 0. : std::min(std::max(x, -1e150), 1e150);
      }
      it[i].node = (int32_t)i;
    }
  });
  auto join = [&] {
    all.clear();
    for (auto &p : part) {
      all.insert(all.end(), p.begin(), p.end());
      p.clear();
    }
  };
  w.chunked(m.ninst, [&](int64_t k0, int64_t k1, int t) {
    for (int64_t k = k0; k < k1; ++k) {
      const Range r = {m.inst_off[k], m.inst_off[k + 1], (int)k};
      if (r.b == r.e) continue;
      Box box;
      for (int a = 0; a < 3; ++a) box.lo[a] = box.hi[a] = it[r.b].x[a];
      for (int64_t i = r.b; i < r.e; ++i)
        for (int a = 0; a < m.D; ++a) {
          box.lo[a] = std::min(box.lo[a], it[i].x[a]);
          box.hi[a] = std::max(box.hi[a], it[i].x[a]);
        }
      part[t].push_back({r, box});
    }
  });
  join();
  // level by level until there is a part for every thread, then part by part
  for (size_t before = 0; w.parts() > 1 && all.size() != before &&
                          all.size() < 4 * (size_t)w.parts();) {
    before = all.size();
    w.chunked((int64_t)all.size(), [&](int64_t k0, int64_t k1, int t) {
      for (int64_t k = k0; k < k1; ++k) {
        if (all[k].r.e - all[k].r.b <= m.max_own) {
          part[t].push_back(all[k]);
          continue;
        }
        Part half[2];
        split(m, it.get(), tmp.get(), all[k], half);
        part[t].insert(part[t].end(), half, half + 2);
      }
    });
    join();
  }
  std::vector<std::vector<Range>> list(w.parts());
  w.chunked((int64_t)all.size(), [&](int64_t k0, int64_t k1, int t) {
    for (int64_t k = k0; k < k1; ++k) bisect(m, it.get(), tmp.get(), all[k], list[t]);
  });
  std::vector<Range> leaves;
  for (auto &x : list) leaves.insert(leaves.end(), x.begin(), x.end());
  w.chunked(N, [&](int64_t i0, int64_t i1, int) {
    for (int64_t i = i0; i < i1; ++i) idx[i] = it[i].node;
  });
  return leaves;
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

void cut_patches(const PatchMesh &m, PatchCut &cut) {
  Workers w(host_threads(std::max(m.N, m.E)));
  cut.nodes.resize(m.N);
  cut.owner.resize(m.N);
  cut.patch = leaves_of(m, w, cut.nodes.data());
  w.chunked((int64_t)cut.patch.size(), [&](int64_t p0, int64_t p1, int) {
    for (int64_t p = p0; p < p1; ++p)
      for (int64_t k = cut.patch[p].b; k < cut.patch[p].e; ++k)
        cut.owner[cut.nodes[k]] = (int32_t)p;
  });
}

bool build_patches(const PatchMesh &m, const PatchCut &cut, const PatchCaps &caps,
                   PatchPlan &plan) {
  const int NN = m.NN;
  const int64_t N = m.N, E = m.E;
  plan = PatchPlan();
  plan.NNP = NN <= 4 ? 4 : 8;
  const int NNP = plan.NNP;
  const std::vector<Range> &leaves = cut.patch;
  const std::vector<int32_t> &idx = cut.nodes, &owner = cut.owner;
  const int64_t P = (int64_t)leaves.size();
  if (P == 0 || P > caps.patches) return false;
  Workers w(host_threads(std::max(N, E)));
  // ---- elements of each patch: those with a node it owns, ascending
  const int et = w.parts();
  struct Pair {
    int32_t patch, element;
  };
  std::vector<std::vector<Pair>> pairs(et);
  std::vector<std::vector<int32_t>> count(et, std::vector<int32_t>(P + 1, 0));
  w.chunked(E, [&](int64_t e0, int64_t e1, int t) {
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
  plan.elems.resize(total);
  w.chunked(et, [&](int64_t t0, int64_t t1, int) {
    for (int64_t t = t0; t < t1; ++t)
      for (const Pair &x : pairs[t]) plan.elems[count[t][x.patch]++] = x.element;
  });
  // ---- local indices
  plan.conn.resize((size_t)total * NNP);
  plan.slot.resize((size_t)total * NNP);
  std::vector<std::vector<int32_t>> local(P);
  plan.own.resize(N);
  std::atomic<bool> ok{true};
  w.chunked(P, [&](int64_t p0, int64_t p1, int) {
    // node -> 1 + its index in the patch, 0 outside; cleared after each patch
    std::vector<int32_t> where(N, 0);
    std::vector<int32_t> corner, mine;
    for (int64_t p = p0; p < p1 && ok; ++p) {
      PatchHead &h = plan.head[p];
      int32_t *el = plan.elems.data() + (size_t)h.chunk0 * 32;
      std::fill(el + h.n_elem, el + (h.n_elem + 31) / 32 * 32, 0);
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
      const size_t padded = (size_t)(h.n_elem + 31) / 32 * 32 * NNP;
      std::fill(lc, lc + padded, (uint16_t)0);
      std::fill(sc, sc + padded, kNoSlot);
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
  w.chunked(P, [&](int64_t p0, int64_t p1, int) {
    for (int64_t p = p0; p < p1; ++p)
      std::copy(local[p].begin(), local[p].end(), plan.nodes.data() + plan.head[p].node0);
  });
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
