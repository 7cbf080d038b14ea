// Fused step kernels of the mixed-precision path (contraction allowed, like
// the two-kernel forms of kernels_mixed.cu).
#include "patch_launch.cuh"

namespace akb {

namespace {
// one thread per chunk entry (PatchChunk's layout)
template <class T>
__global__ void k_patch_chunks(int NNP, int64_t n, const int32_t *__restrict__ elems,
                               const uint16_t *__restrict__ conn,
                               const uint16_t *__restrict__ slot, int64_t E, int rows_a,
                               const T *__restrict__ a, int rows_b, const T *__restrict__ b,
                               char *__restrict__ tab) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int lane = (int)(k & 31);
  const int64_t e = elems[k];
  const int64_t local = 64 * NNP, bytes = 2 * local + 32 * (int64_t)sizeof(T) * (rows_a + rows_b);
  char *chunk = tab + (k >> 5) * bytes;
  uint16_t *c = reinterpret_cast<uint16_t *>(chunk) + lane * NNP;
  uint16_t *s = reinterpret_cast<uint16_t *>(chunk + local) + lane * NNP;
  for (int i = 0; i < NNP; ++i) {
    c[i] = conn[k * NNP + i];
    s[i] = slot[k * NNP + i];
  }
  T *r = reinterpret_cast<T *>(chunk + 2 * local) + lane;
  for (int i = 0; i < rows_a; ++i) r[i * 32] = a[i * E + e];
  for (int i = 0; i < rows_b; ++i) r[(rows_a + i) * 32] = b[i * E + e];
}
}  // namespace

cudaError_t launch_patch_chunks(int NNP, int64_t entries, const int32_t *elems,
                                const uint16_t *conn, const uint16_t *slot, int64_t E, int rows_a,
                                const void *a, int rows_b, const void *b, size_t value, void *tab,
                                cudaStream_t s) {
  if (entries == 0) return cudaSuccess;
  if (value == sizeof(float))
    k_patch_chunks<float><<<grid_for(entries), kThreads, 0, s>>>(
        NNP, entries, elems, conn, slot, E, rows_a, (const float *)a, rows_b, (const float *)b,
        (char *)tab);
  else
    k_patch_chunks<double><<<grid_for(entries), kThreads, 0, s>>>(
        NNP, entries, elems, conn, slot, E, rows_a, (const double *)a, rows_b, (const double *)b,
        (char *)tab);
  return cudaGetLastError();
}

namespace {
// tetrahedra: small patches, one per SM, are bound by their chain of latencies
// (the state loaded first: 3 k tetrahedra 3.11 against 3.29 us per step);
// beyond, registers capped for three blocks per SM (the state held across the
// elements: batch of 64 cubes 161 against 145 us)
template <class EV>
cudaError_t launch_tet(const PatchArgs &pa, const MatParams &mp, const GroupArgs &ps, bool pdl,
                       cudaStream_t s) {
  if (pa.npatch <= kPatchSms && pa.max_own <= 27)
    return launch_patch<EV, true, true, 256, 1>(pa, mp, ps, pdl, s);
  if (pa.ahead) return launch_patch<EV, true, false, 256, 3, true>(pa, mp, ps, pdl, s);
  return launch_patch<EV, true, false, 256, 3>(pa, mp, ps, pdl, s);
}
// triangles: with one patch per SM the state first and all points of two
// chunks at once (24^2 x 2 of 3 points 6.12 against 6.70 us per step)
template <class EV>
cudaError_t launch_tri(const PatchArgs &pa, const MatParams &mp, const GroupArgs &ps, bool pdl,
                       cudaStream_t s) {
  if (pa.npatch <= kPatchSms) return launch_patch<EV, true, true, 256, 1>(pa, mp, ps, pdl, s);
  return launch_patch<EV, true, false, 192, 4>(pa, mp, ps, pdl, s);
}
}  // namespace

cudaError_t launch_patch_step_mixed(int et, int law, const PatchArgs &pa, const MatParams &mp,
                                    const GroupArgs &ps, bool pdl, cudaStream_t s) {
  if (et == ET_TET4 && law == LAW_ELASTIC)
    return launch_tet<PatchTet4<LAW_ELASTIC, float>>(pa, mp, ps, pdl, s);
  if (et == ET_TET4 && law == LAW_NEOHOOKEAN)
    return launch_tet<PatchTet4<LAW_NEOHOOKEAN, float>>(pa, mp, ps, pdl, s);
  if (et == ET_HEX8 && law == LAW_ELASTIC)
    return launch_patch<PatchHex8X2<LAW_ELASTIC>, true, true, 128, 2>(pa, mp, ps, pdl, s);
  if (et == ET_HEX8 && law == LAW_NEOHOOKEAN)
    return launch_patch<PatchHex8X2<LAW_NEOHOOKEAN>, true, true, 128, 2>(pa, mp, ps, pdl, s);
  if (et == ET_TRI6 && law == LAW_PLASTIC)
    return pa.nq == 3 ? launch_tri<PatchTri6<3, float>>(pa, mp, ps, pdl, s)
                      : launch_tri<PatchTri6<6, float>>(pa, mp, ps, pdl, s);
  return cudaErrorInvalidValue;
}

}  // namespace akb
