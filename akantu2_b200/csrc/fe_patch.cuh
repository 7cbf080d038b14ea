// Kernel of the fused step (patch.h): one thread block per patch of nodes.
//
// Why: the two-kernel step writes every elemental force to a slot array in
// HBM, one 128-byte line per lane, and reads it back in the node update; it
// gathers the displacements of every element by 8-byte loads through global
// indices.  Here a block copies its patch's displacements (owned nodes and
// halo) into shared memory once, evaluates every element that touches an
// owned node, keeps the forces in shared memory and updates its own nodes.
// Elements on the border of two patches are evaluated by both: redundant
// arithmetic instead of traffic, and one launch per step instead of two.
//
// The slot of the r-th element (in the reference's scatter order) of owned
// node i is r n_own + i: the update's lanes read consecutive slots, free of
// bank conflicts, and each node sums its slots in the same order as the CSR
// gather, so the results are those of the two-kernel step.
//
// Measured on B200, us per step, two kernels / fused: tetrahedra, mixed, 3 k
// 6.9 / 3.1, 48 k 7.7 / 4.5, 384 k 17.4 / 14.1, 912 k (neohookean) 45.9 / 32.0, a
// batch of 64 cubes (4.5 M) 201 / 138; FP64 3 k 7.6 / 2.8, 48 k 9.4 / 4.9, 1.3 M
// 95 / 73, the batch 308 / 224.  Which meshes gain is decided on the finished plan
// (patches_over_kernels).  What bounds the large ones (80^3 x 6 tetrahedra, mixed, ncu):
// 46 % of the issue slots, 60 % of the shared-memory pipe and 42 % of the DRAM
// bandwidth are busy; a block waits in turn for its node list, its displacements
// and its nodes' state, and three fit an SM.  Blocks that loop over patches and
// list the next one's nodes ahead were slower (5.0 against 3.3 us at 3 k
// tetrahedra, 166 against 165 for the batch), and so were 128, 160, 320 and 384
// threads (147 to 159 us).  Plastic triangles, one thread per point: 128
// triangles of 3 points, mixed, 7.5 / 3.7, 2 k of 6 points, FP64, 13.5 / 4.5 (9.3
// and 18.7 with one thread per element), 20 k of 3 points, mixed, 9.9 / 8.5.
#pragma once

#include "fe_kernels.cuh"
#include "patch.h"

namespace akb {

__device__ __forceinline__ void prefetch_l2_line(const void *p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(__cvta_generic_to_global(p)));
}

// Element tables of a patch in chunks of 32 elements, one lane each:
// [conn 32 x NNP x 2 bytes][slot, the same][rows x 32 values].  A warp reads
// a chunk in coalesced pieces of one contiguous block of memory.
template <int NN, int ROWS, class T> struct PatchChunk {
  static constexpr int NNP = NN <= 4 ? 4 : 8;
  static constexpr int kLocal = 32 * NNP * 2;                // bytes of conn (slot)
  static constexpr int kBytes = 2 * kLocal + ROWS * 32 * (int)sizeof(T);
  int cw[NNP / 2], sw[NNP / 2];  // conn and slot, two 16-bit entries per word
  T row[ROWS];
  __device__ __forceinline__ void load(const char *chunk, int lane) {
    if constexpr (NNP == 4) {
      const int2 c = reinterpret_cast<const int2 *>(chunk)[lane];
      const int2 s = reinterpret_cast<const int2 *>(chunk + kLocal)[lane];
      cw[0] = c.x, cw[1] = c.y;
      sw[0] = s.x, sw[1] = s.y;
    } else {
      const int4 c = reinterpret_cast<const int4 *>(chunk)[lane];
      const int4 s = reinterpret_cast<const int4 *>(chunk + kLocal)[lane];
      cw[0] = c.x, cw[1] = c.y, cw[2] = c.z, cw[3] = c.w;
      sw[0] = s.x, sw[1] = s.y, sw[2] = s.z, sw[3] = s.w;
    }
    const T *r = reinterpret_cast<const T *>(chunk + 2 * kLocal) + lane;
#pragma unroll
    for (int k = 0; k < ROWS; ++k) row[k] = r[k * 32];
  }
  __device__ __forceinline__ int node(int a) const { return (cw[a >> 1] >> (16 * (a & 1))) & 0xffff; }
  __device__ __forceinline__ int slot(int a) const { return (sw[a >> 1] >> (16 * (a & 1))) & 0xffff; }
};

// The next chunk is loaded into registers (tetrahedra) or, where those are
// needed for the arithmetic (kStaged), into a shared buffer of the warp, while
// the current one is evaluated: without it 184 against 168 us on the batch.

// r [NN][D] into the slots of the element whose chunk entry is ch
template <int D, int NN, class Chunk, class T>
__device__ __forceinline__ void store_slots(const Chunk &ch, const T *r, T *sl) {
#pragma unroll
  for (int a = 0; a < NN; ++a) {
    const int s = ch.slot(a);
    if (s != kNoSlot) {
#pragma unroll
      for (int i = 0; i < D; ++i) sl[s * D + i] = r[a * D + i];
    }
  }
}

// Element evaluators: the elemental force of the element whose chunk entry is
// ch (element le of its group), from the patch's displacements us, into its
// slots sl.

// linear tetrahedra: the arithmetic of element_pe; the chunk holds dN/dx
// (mixed: of nodes 1..3) and det J w
template <int LAW_, class T_> struct PatchTet4 {
  using T = T_;
  static constexpr int D = 3, NN = 4, LAW = LAW_;
  static constexpr bool REL = !std::is_same<T, double>::value;
  using Chunk = PatchChunk<NN, REL ? 10 : 13, T>;
  static constexpr bool kStaged = false;
  static constexpr int kPoints = 1;  // threads (and slot arrays) per element
  static constexpr int kIds = 2;  // nodes of a patch each thread lists ahead
  // the padding of the last chunk must not be evaluated (it writes state)
  static constexpr bool kActive = false;
  static constexpr bool kFetch = false;
  static __device__ __forceinline__ void forces(const PatchArgs &pa, const MatParams &mpe,
                                                const GroupArgs &ps, const double *us,
                                                const Chunk &ch, int64_t le, int, T *sl) {
    constexpr int ND = NN * D;
    T b[ND], ue[ND], r[ND];
#pragma unroll
    for (int c = REL ? 3 : 0; c < ND; ++c) b[c] = ch.row[REL ? c - 3 : c];
    const T w = ch.row[REL ? 9 : 12];
    double u0[D];
#pragma unroll
    for (int a = 0; a < NN; ++a) {
      const double *ua = us + ch.node(a) * D;
#pragma unroll
      for (int i = 0; i < D; ++i) {
        const double x = ua[i];
        if constexpr (REL) {
          if (a == 0) u0[i] = x;
          ue[a * D + i] = (T)(x - u0[i]);
        } else {
          ue[a * D + i] = x;
        }
      }
    }
    if constexpr (REL) {
#pragma unroll
      for (int j = 0; j < 3; ++j) b[j] = -((b[3 + j] + b[6 + j]) + b[9 + j]);
    }
    element_law<D, NN, LAW, T, REL>(ue, b, w, mpe, ps, pa.e_count, le, 0, r);
    store_slots<D, NN>(ch, r, sl);
  }
};

// mixed hexahedra of a mesh of parallelepipeds on packed FP32 pairs; the
// chunk holds the adjugate and 1/det.  PU pairs of points per unrolled
// iteration: 2, as the code of 4 does not stay in the instruction cache (no
// instruction ready 1.56 of 8.4 cycles per issue, 0.25 with 2)
template <int LAW_, int PU = 2> struct PatchHex8X2 {
  using T = float;
  static constexpr int D = 3, NN = 8, LAW = LAW_;
  using Chunk = PatchChunk<NN, 10, float>;
  static constexpr bool kStaged = true;
  static constexpr int kPoints = 1;
  static constexpr int kIds = 4;
  static constexpr bool kActive = false;
  static constexpr bool kFetch = false;
  static __device__ __forceinline__ void forces(const PatchArgs &pa, const MatParams &mpe,
                                                const GroupArgs &ps, const double *us,
                                                const Chunk &ch, int64_t le, int, float *sl) {
    constexpr int lex[8] = {0, 1, 3, 2, 4, 5, 7, 6};
    float wu[8][3], A[8][3];
    double u0[3];
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const double *ua = us + ch.node(a) * 3;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const double x = ua[i];
        if (a == 0) u0[i] = x;
        wu[lex[a]][i] = (float)(x - u0[i]);
      }
    }
    hex8sf_x2_forces<LAW, PU>(wu, ch.row, ch.row[9], mpe, ps, pa.e_count, le, A);
    float r[24];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
      for (int i = 0; i < 3; ++i) r[a * 3 + i] = A[lex[a]][i];
    store_slots<3, 8>(ch, r, sl);
  }
};

// plastic quadratic triangles, one thread per (element, point): the radial
// return is a long serial chain, and one thread going through an element's 3
// or 6 points makes the step of a small mesh as long as all of them.  The
// point's force goes to the point's own slot array; the update sums the
// points of a slot in increasing order.  The chunk holds the local indices,
// dN/dx and det J w are read where they are used from the rows behind them.
// An element is owned by the patch of its first node: that patch writes its
// new plastic state, the others evaluate it from the same previous state.
template <int NQ_, class T_> struct PatchTri6 {
  using T = T_;
  static constexpr int D = 2, NN = 6, NQ = NQ_, LAW = LAW_PLASTIC;
  static constexpr bool REL = !std::is_same<T, double>::value;
  static constexpr int ND = NN * D, kRows = NQ * (ND + 1);
  struct Chunk : PatchChunk<NN, 0, T> {
    static constexpr int kBytes = PatchChunk<NN, 0, T>::kBytes + kRows * 32 * (int)sizeof(T);
    const T *rows;  // [kRows][32]: dN_a/dx_j of point q at q ND + a D + j, then det J w
    __device__ __forceinline__ void load(const char *chunk, int lane) {
      PatchChunk<NN, 0, T>::load(chunk, lane);
      rows = reinterpret_cast<const T *>(chunk + 2 * PatchChunk<NN, 0, T>::kLocal) + lane;
    }
  };
  static constexpr bool kStaged = false;
  static constexpr int kPoints = NQ;
  static constexpr int kIds = 4;
  static constexpr bool kActive = true;
  static constexpr bool kFetch = true;  // its chunks prefetched into L2 at the start
  static __device__ __forceinline__ void forces(const PatchArgs &pa, const MatParams &mpe,
                                                const GroupArgs &ps, const double *us,
                                                const Chunk &ch, int64_t le, int q, T *sl) {
    const bool owner = ch.slot(0) != kNoSlot;
    const T *B = ch.rows + q * ND * 32;
    T ue[ND];
    double u0[D];
#pragma unroll
    for (int a = 0; a < NN; ++a) {
      const double *ua = us + ch.node(a) * D;
#pragma unroll
      for (int i = 0; i < D; ++i) {
        const double x = ua[i];
        if constexpr (REL) {
          if (a == 0) u0[i] = x;
          ue[a * D + i] = (T)(x - u0[i]);
        } else {
          ue[a * D + i] = x;
        }
      }
    }
    // the streamed law of element_pe_plastic_streamed, the same operations
    T g[D * D];
#pragma unroll
    for (int a = 0; a < NN; ++a) {
      T ba[D];
#pragma unroll
      for (int j = 0; j < D; ++j) ba[j] = B[(a * D + j) * 32];
#pragma unroll
      for (int j = 0; j < D; ++j)
#pragma unroll
        for (int i = 0; i < D; ++i)
          g[i + D * j] = (a == 0) ? ue[i] * ba[j] : g[i + D * j] + ue[a * D + i] * ba[j];
    }
    subtract_eigen<D, T>(ps, pa.e_count, le, q, g);
    T sig[D * D];
    {
      double gd[D * D], sd[D * D];
#pragma unroll
      for (int k = 0; k < D * D; ++k) gd[k] = (double)g[k];
      plastic_point<D, T, true>(mpe, ps, pa.e_count, le, q, gd, sd, owner);
#pragma unroll
      for (int k = 0; k < D * D; ++k) sig[k] = (T)sd[k];
    }
    const T w = ch.rows[(NQ * ND + q) * 32];
    if constexpr (REL) {
#pragma unroll
      for (int k = 0; k < D * D; ++k) sig[k] *= w;
    }
#pragma unroll
    for (int a = 0; a < NN; ++a) {
      const int s = ch.slot(a);
      if (s == kNoSlot) continue;
      T ba[D];
#pragma unroll
      for (int j = 0; j < D; ++j) ba[j] = ld_table(B + (a * D + j) * 32);
#pragma unroll
      for (int i = 0; i < D; ++i) {
        T x = sig[i] * ba[0];
#pragma unroll
        for (int j = 1; j < D; ++j) {
          if constexpr (REL) x += sig[i + D * j] * ba[j];
          else x = x + sig[i + D * j] * ba[j];
        }
        if constexpr (!REL) x = x * w;
        sl[s * D + i] = x;
      }
    }
  }
};

// AKB_BOUNDS_CHECK builds check every index of the plan before it is used: the
// ranges of a patch, the nodes it lists and owns, its elements' local indices
// and slots.  What has an index out of range sets status bit 2 and is skipped.
template <class EV>
__device__ __forceinline__ bool patch_head_ok(const PatchArgs &pa, const GroupArgs &ps,
                                              const PatchHead &h) {
#ifdef AKB_BOUNDS_CHECK
  const int64_t nod = ((int64_t)h.n_local * EV::D + 1) & ~(int64_t)1;
  if (h.node0 >= 0 && h.n_local >= 0 && (int64_t)h.node0 + h.n_local <= pa.list_nodes &&
      h.own0 >= 0 && h.n_own >= 0 && (int64_t)h.own0 + h.n_own <= ps.nb_nodes && h.chunk0 >= 0 &&
      h.n_elem >= 0 && ((int64_t)h.chunk0 + (h.n_elem + 31) / 32) * 32 <= pa.list_elems &&
      h.n_slot >= 0 && h.inst >= 0 && h.inst < pa.instances && h.mat < pa.materials &&
      8 * nod + (int64_t)sizeof(typename EV::T) * h.n_slot * EV::kPoints * EV::D <=
          (int64_t)pa.smem)
    return true;
  atomicOr(ps.status, ST_INDEX_RANGE);
  return false;
#else
  (void)pa, (void)ps, (void)h;
  return true;
#endif
}
__device__ __forceinline__ bool patch_node_ok(const GroupArgs &ps, int64_t node) {
#ifdef AKB_BOUNDS_CHECK
  if (node >= 0 && node < ps.nb_nodes) return true;
  atomicOr(ps.status, ST_INDEX_RANGE);
  return false;
#else
  (void)ps, (void)node;
  return true;
#endif
}
__device__ __forceinline__ bool patch_own_ok(const GroupArgs &ps, const PatchHead &h,
                                             const PatchOwn &o) {
#ifdef AKB_BOUNDS_CHECK
  if (o.node >= 0 && o.node < ps.nb_nodes && o.local < h.n_local &&
      (int64_t)o.valence * h.n_own <= h.n_slot)
    return true;
  atomicOr(ps.status, ST_INDEX_RANGE);
  return false;
#else
  (void)ps, (void)h, (void)o;
  return true;
#endif
}
template <int NN, class Chunk>
__device__ __forceinline__ bool patch_element_ok(const PatchArgs &pa, const GroupArgs &ps,
                                                 const PatchHead &h, const Chunk &ch,
                                                 int64_t le) {
#ifdef AKB_BOUNDS_CHECK
  bool ok = le >= 0 && le < pa.e_count;
#pragma unroll
  for (int a = 0; a < NN; ++a)
    ok = ok && ch.node(a) < h.n_local && (ch.slot(a) == kNoSlot || ch.slot(a) < h.n_slot);
  if (!ok) atomicOr(ps.status, ST_INDEX_RANGE);
  return ok;
#else
  (void)pa, (void)ps, (void)h, (void)ch, (void)le;
  return true;
#endif
}

// a chunk into the warp's shared buffer, 16 bytes per lane and pass
template <int BYTES> __device__ __forceinline__ void stage_chunk(char *dst, const char *src) {
  const int lane = threadIdx.x & 31;
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
#pragma unroll
  for (int k = 0; k < (BYTES + 511) / 512; ++k) {
    const int at = (k * 32 + lane) * 16;
    if (BYTES % 512 == 0 || at < BYTES)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + at), "l"(src + at)
                   : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// bytes of shared memory the element tables of a block are staged in
template <class EV, int THREADS> __host__ __device__ constexpr size_t patch_stage_bytes() {
  return EV::kStaged ? (size_t)(THREADS / 32) * 2 * EV::Chunk::kBytes : 0;
}

// One step of patch blockIdx.x.  KAHAN: compensated sum (mixed path); MULTI:
// a patch may hold several materials; EARLY: the thread's first owned node is
// read ahead, what no step changes before the preceding kernel has ended and
// its state before the elements (otherwise its lines are prefetched into L2);
// AHEAD: the next wave's tables are prefetched into L2.
// THREADS and MINB set how many warps
// share a patch's shared memory and what their registers are capped at.
template <class EV, bool KAHAN, bool MULTI, bool EARLY, bool AHEAD, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB)
    k_patch_step(const __grid_constant__ PatchArgs pa, const __grid_constant__ MatParams mp,
                 const __grid_constant__ GroupArgs ps) {
  using RT = typename EV::T;
  using Chunk = typename EV::Chunk;
  constexpr int D = EV::D, W = THREADS / 32, U = EV::kIds;
  extern __shared__ __align__(16) char patch_sm[];
  // one kernel a step: it lets the next one launch at once up to 8 patches per
  // SM (only where two steps' patches are resident together, 3 k tetrahedra
  // 3.15 against 3.68 us per step, 160 k 12.3 against 12.8)
  const bool trigger = gridDim.x <= 8 * kPatchSms;
  if (pa.presc.count && blockIdx.x == gridDim.x - 1) {
    pdl_begin(trigger);
    return prescribe_block(pa.presc, pa.u_next, true);
  }
  const PatchHead h = pa.head[blockIdx.x];
  if (!patch_head_ok<EV>(pa, ps, h)) return;
  const int32_t *nodes = pa.nodes + h.node0;
  const PatchOwn *own = pa.own + h.own0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  char *stage = patch_sm + warp * 2 * Chunk::kBytes;
  double *us = reinterpret_cast<double *>(patch_sm + patch_stage_bytes<EV, THREADS>());
  RT *sl = reinterpret_cast<RT *>(us + ((h.n_local * D + 1) & ~1));
  const int nchunk = (h.n_elem + 31) >> 5;
  const char *chunks = static_cast<const char *>(pa.tab) + (int64_t)h.chunk0 * Chunk::kBytes;
  // nothing a step changes is read before the preceding kernel has ended:
  // until then the first chunk of each warp and the node list
  Chunk ch;
  if constexpr (EV::kStaged) {
    if (warp < nchunk) stage_chunk<Chunk::kBytes>(stage, chunks + (int64_t)warp * Chunk::kBytes);
  } else {
    const int c = warp / EV::kPoints;
    if (c < nchunk) ch.load(chunks + (int64_t)c * Chunk::kBytes, lane);
  }
  if constexpr (EV::kFetch) {
    if (threadIdx.x == 0 && nchunk > 0)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(
                       __cvta_generic_to_global(chunks)),
                   "r"((unsigned)(nchunk * Chunk::kBytes))
                   : "memory");
  }
  int32_t id[U];
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const int i = threadIdx.x + k * THREADS;
    id[k] = i < h.n_local ? nodes[i] : 0;
  }
  PatchOwn o0;
  NodeState<D> st0;
  if constexpr (EARLY) {
    if (threadIdx.x < h.n_own) {
      o0 = own[threadIdx.x];
      if (patch_own_ok(ps, h, o0)) {
        st0.m = pa.mass[o0.node];
        st0.bl = pa.blocked[o0.node];
      }
    }
  }
  pdl_begin(trigger);
  // as in k_node_update_retire: a stopped instance keeps its state, and the
  // last step of an instance stores its internal force
  int flags = pa.flags;
  if (pa.inst_end) {
    const int64_t left = pa.inst_end[h.inst] - *pa.step;
    if (left <= 0) {
      copy_async_wait();
      if (flags & NU_PREDICT)
        for (int j = threadIdx.x; j < h.n_own * D; j += THREADS) {
          if (!patch_own_ok(ps, h, own[j / D])) continue;
          const int64_t k = (int64_t)own[j / D].node * D + j % D;
          pa.u[k] = pa.u_next[k];
        }
      return;
    }
    if (left == 1) flags |= NU_FINT;
  }
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const int i = threadIdx.x + k * THREADS;
    if (i < h.n_local && patch_node_ok(ps, id[k]))
#pragma unroll
      for (int c = 0; c < D; ++c) copy_async_8(us + i * D + c, pa.u + (int64_t)id[k] * D + c);
  }
  for (int i = threadIdx.x + U * THREADS; i < h.n_local; i += THREADS) {
    const int64_t n = nodes[i];
    if (!patch_node_ok(ps, n)) continue;
#pragma unroll
    for (int c = 0; c < D; ++c) copy_async_8(us + i * D + c, pa.u + n * D + c);
  }
  auto load_state = [&](int64_t node, NodeState<D> &st) {
#pragma unroll
    for (int c = 0; c < D; ++c) {
      const int64_t k = node * D + c;
      st.a[c] = pa.a[k];
      st.v[c] = pa.v[k];
      st.f[c] = (pa.flags & NU_FEXT_ZERO) ? 0. : pa.fext[k];
    }
  };
  if constexpr (EARLY) {
    if (threadIdx.x < h.n_own && patch_own_ok(ps, h, o0)) load_state(o0.node, st0);
  } else {
    // the owned nodes' state, which the update reads last, into L2 meanwhile
    for (int i = threadIdx.x; i < h.n_own; i += THREADS) {
      const int64_t node = own[i].node;
      if (!patch_node_ok(ps, node)) continue;
      prefetch_l2_line(pa.a + node * D);
      prefetch_l2_line(pa.v + node * D);
      prefetch_l2_line(pa.mass + node);
    }
  }
  // the lists and element tables of the block that follows this one on its
  // SM, from DRAM into L2
  constexpr int kWave = (int)kPatchSms * MINB;
  if (AHEAD && threadIdx.x == 32 && blockIdx.x + kWave < pa.npatch) {
    const PatchHead hn = pa.head[blockIdx.x + kWave];
    const bool next_ok = patch_head_ok<EV>(pa, ps, hn);
    auto fetch = [next_ok](const void *lo, const void *hi) {
      const uint64_t a = (uint64_t)__cvta_generic_to_global(lo) & ~(uint64_t)15;
      const uint64_t z = ((uint64_t)__cvta_generic_to_global(hi) + 15) & ~(uint64_t)15;
      if (z > a && next_ok)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((unsigned)(z - a))
                     : "memory");
    };
    fetch(pa.nodes + hn.node0, pa.nodes + hn.node0 + hn.n_local);
    fetch(pa.own + hn.own0, pa.own + hn.own0 + hn.n_own);
    const char *cn = static_cast<const char *>(pa.tab) + (int64_t)hn.chunk0 * Chunk::kBytes;
    fetch(cn, cn + (int64_t)((hn.n_elem + 31) >> 5) * Chunk::kBytes);
  }
  const MatParams mph = (ps.mtab && h.mat >= 0) ? ps.mtab[h.mat] : mp;
  const double dt = pa.inst_dt ? pa.inst_dt[h.inst] : pa.dt;
  copy_async_wait();
  __syncthreads();
  int buf = 0;
  // work items: chunk c of the elements, point q
  const int nitem = nchunk * EV::kPoints, plane = h.n_slot * D;
  for (int it = warp; it < nitem; it += W) {
    const int c = it / EV::kPoints, q = it - c * EV::kPoints;
    // the next chunk is on its way while this one is evaluated
    Chunk next;
    const bool more = it + W < nitem;
    const char *np = chunks + (int64_t)((it + W) / EV::kPoints) * Chunk::kBytes;
    if constexpr (EV::kStaged) {
      if (it != warp) copy_async_wait();
      __syncwarp();
      ch.load(stage + buf * Chunk::kBytes, lane);
      buf ^= 1;
      if (more) stage_chunk<Chunk::kBytes>(stage + buf * Chunk::kBytes, np);
    } else {
      if (more) next.load(np, lane);
    }
    int64_t le = 0;
    if (MULTI || pa.need_index) le = pa.elems[(int64_t)(h.chunk0 + c) * 32 + lane];
    const bool active = c * 32 + lane < h.n_elem;
    if ((!EV::kActive || active) && patch_element_ok<EV::NN>(pa, ps, h, ch, le)) {
      if constexpr (MULTI) {
        const MatParams mpe = ps.mtab[ps.mslot[le]];
        EV::forces(pa, mpe, ps, us, ch, le, q, sl + q * plane);
      } else {
        EV::forces(pa, mph, ps, us, ch, le, q, sl + q * plane);
      }
    }
    if constexpr (!EV::kStaged) ch = next;
  }
  __syncthreads();
  // the node update, one thread per owned node
  const int row = h.n_own * D;
  for (int i = threadIdx.x; i < h.n_own; i += THREADS) {
    PatchOwn o;
    NodeState<D> st;
    if (EARLY && i < THREADS) {
      o = o0;
      st = st0;
      if (!patch_own_ok(ps, h, o)) continue;
    } else {
      o = own[i];
      if (!patch_own_ok(ps, h, o)) continue;
      st.m = pa.mass[o.node];
      st.bl = pa.blocked[o.node];
      load_state(o.node, st);
    }
    const int64_t node = o.node;
#pragma unroll
    for (int c = 0; c < D; ++c) st.u[c] = us[o.local * D + c];
    double acc[D], comp[D];
#pragma unroll
    for (int c = 0; c < D; ++c) acc[c] = comp[c] = 0.;
    const RT *si = sl + i * D;
#pragma unroll 4
    for (int s = 0; s < o.valence; ++s) {
      double rv[D];
#pragma unroll
      for (int c = 0; c < D; ++c) {
        // integrate: sum over the points in increasing order
        RT x = si[s * row + c];
#pragma unroll
        for (int q = 1; q < EV::kPoints; ++q) x = x + si[q * plane + s * row + c];
        rv[c] = (double)x;
      }
      accumulate_slot<D, KAHAN>(rv, acc, comp);
    }
    node_apply_state<D, true>(node, acc, st, pa.fint, pa.a, pa.v, pa.u_next, dt, nullptr, nullptr,
                        flags, pa.status);
  }
}

}  // namespace akb
