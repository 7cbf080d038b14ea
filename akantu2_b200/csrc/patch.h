// The fused step: the mesh split into compact patches of nodes, one thread
// block per patch.  A block holds its patch's displacements and elemental
// forces in shared memory, so a step is one launch and the elemental forces
// never go through HBM.  Host-side plan (patch_build.cc) and launchers
// (kernels_patch.cu, kernels_patch64.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <memory>
#include <vector>

#include "presc.h"

namespace akb {

struct GroupArgs;
struct MatParams;

constexpr uint16_t kNoSlot = 0xffff;  // the node's force is not summed here

// one patch: its nodes (those it owns and the halo, the other nodes of the
// elements that touch an owned node), its owned nodes and its elements
struct alignas(16) PatchHead {
  int32_t node0, n_local;   // node list [node0, node0 + n_local), ascending
  int32_t own0, n_own;      // owned list [own0, own0 + n_own), ascending
  int32_t chunk0, n_elem;   // its elements are entries [32 chunk0, 32 chunk0 + n_elem)
  int32_t n_slot;           // slots: largest valence x n_own
  int32_t inst;             // instance of a batch (0 otherwise)
  int32_t mat;              // material of all its elements, or -1
  int32_t pad[3];
};
// an owned node: its local index in the patch's node list, its slot count
struct PatchOwn {
  int32_t node;
  uint16_t local, valence;
};

// What the builder reads, all in host memory.  cut_patches reads the first
// part only, build_patches all of it but elements.
struct PatchMesh {
  int D = 3, NN = 4;
  int64_t N = 0, E = 0;
  const double *X = nullptr;          // [N][D]
  const int32_t *elements = nullptr;  // [E][NN], in any order
  const int64_t *inst_off = nullptr;  // node offsets of the instances [ninst + 1]
  int ninst = 1;
  int max_own = 512;                  // owned nodes of a patch at most
  // in the internal element order
  const int32_t *conn = nullptr;     // [NN][E]
  const int32_t *ptr = nullptr;      // node -> slot CSR offsets [N + 1]
  const int32_t *pos = nullptr;      // [NN][E] CSR position of each slot
  const int32_t *mat = nullptr;      // material of each element [E], or null
};

// the patches' owned nodes: patch p has those of nodes [b, e), ascending
struct PatchRange {
  int64_t b, e;
  int inst;
};
struct PatchCut {
  std::vector<PatchRange> patch;
  std::vector<int32_t> nodes;  // [N]
  std::vector<int32_t> owner;  // [N] patch of each node
};
void cut_patches(const PatchMesh &m, PatchCut &cut);

// an array that is not written when it is made (its pages are then touched
// first by the threads that fill it)
template <class T> struct PlanArray {
  std::unique_ptr<T[]> p;
  size_t n = 0;
  void resize(size_t count) {
    p.reset(new T[count]);
    n = count;
  }
  size_t size() const { return n; }
  T *data() { return p.get(); }
  const T *data() const { return p.get(); }
  T &operator[](size_t k) { return p[k]; }
  const T &operator[](size_t k) const { return p[k]; }
};

// Every node is owned by one patch.  Patch element k has its nodes' local
// indices at conn[k NNP + a] and its slots at slot[k NNP + a]: slot
// r n_own + i for the r-th slot (in the reference's scatter order) of owned
// node i, or kNoSlot.  NNP is NN rounded up to 4 or 8.  The elements of a
// patch are padded to chunks of 32; the padding repeats element 0 with no
// slots.
struct PatchPlan {
  int NNP = 4;
  std::vector<PatchHead> head;
  PlanArray<int32_t> nodes;
  PlanArray<PatchOwn> own;  // N entries
  PlanArray<int32_t> elems;
  PlanArray<uint16_t> conn, slot;
  int max_local = 0;  // nodes of a patch at most
  int max_slots = 0;  // slots of a patch at most (largest valence x owned nodes)
};

// capacity of a plan's arrays (entries); a mesh that needs more is stepped
// without patches
struct PatchCaps {
  int64_t patches = 0, nodes = 0, elems = 0;
};
PatchCaps patch_caps(int D, int64_t N, int64_t E, int ninst, int max_own);

// false: the mesh does not fit (capacities, 16-bit local indices)
bool build_patches(const PatchMesh &m, const PatchCut &cut, const PatchCaps &caps,
                   PatchPlan &plan);

// every index of the plan is in range and names what it should: each node
// owned once, each slot of an owned node written by one element, in order
bool check_patches(const PatchMesh &m, const PatchPlan &plan);

// shared-memory bytes of the patch's displacements and slots
inline size_t patch_smem(int D, int max_local, int max_slots, size_t slot_value) {
  const size_t nod = ((size_t)max_local * D + 1) & ~(size_t)1;
  return sizeof(double) * nod + slot_value * (size_t)max_slots * D;
}
// 227 KB, the most one block can have, less the kernel's static variables
constexpr size_t kPatchMaxSmem = 232448 - 1024;
constexpr size_t kPatchStageSmem = 18432;  // staged element tables of the hexahedron kernel

constexpr int64_t kPatchSms = 148;

struct PatchArgs {
  int64_t npatch = 0;
  bool ahead = false;  // the plan is larger than L2
  int max_own = 0;  // owned nodes of a patch at most
  const PatchHead *head = nullptr;
  const int32_t *nodes = nullptr;
  const PatchOwn *own = nullptr;
  const int32_t *elems = nullptr;  // element of each chunk entry
  // per-element tables in chunks (PatchChunk): conn, slot and the rows dN/dx
  // and det J w (tetrahedra) or the adjugate and 1/det (hexahedra)
  const void *tab = nullptr;
  int64_t e_count = 0;  // elements of the (single) law group
  size_t smem = 0;      // of the largest patch, without the staged tables
  int nq = 1;           // quadrature points
  int multi = 0;        // some patch holds several materials
  int need_index = 0;   // element indices are read (per-element state or material)
  // nodal state: u read, u_next, v, a and (NU_FINT) fint written
  const double *fext = nullptr, *mass = nullptr;
  const uint8_t *blocked = nullptr;
  double *u = nullptr, *u_next = nullptr, *v = nullptr, *a = nullptr, *fint = nullptr;
  double dt = 0.;
  const double *inst_dt = nullptr;
  const int64_t *inst_end = nullptr, *step = nullptr;
  int flags = 0;
  unsigned int *status = nullptr;
  PrescArgs presc;  // prescribed motion, written by an extra block
#ifdef AKB_BOUNDS_CHECK
  int64_t list_nodes = 0, list_elems = 0;  // entries of nodes and elems
  int instances = 1, materials = 1;
#endif
};

// fills the chunks: conn and slot [entries][NNP], and rows value rows of
// every entry's element from in (the first rows_a of them, [.][E]) and inb
cudaError_t launch_patch_chunks(int NNP, int64_t entries, const int32_t *elems,
                                const uint16_t *conn, const uint16_t *slot, int64_t E, int rows_a,
                                const void *a, int rows_b, const void *b, size_t value, void *tab,
                                cudaStream_t s);

// one step of every patch (tetrahedra, and hexahedra of a mesh of
// parallelepipeds in mixed precision: elastic and neohookean laws; triangles:
// the plastic law); cudaErrorInvalidValue where no such kernel exists
cudaError_t launch_patch_step_mixed(int et, int law, const PatchArgs &pa, const MatParams &mp,
                                    const GroupArgs &ps, bool pdl, cudaStream_t s);
cudaError_t launch_patch_step_fp64(int et, int law, const PatchArgs &pa, const MatParams &mp,
                                   const GroupArgs &ps, bool pdl, cudaStream_t s);

}  // namespace akb
