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

cudaError_t launch_patch_step_mixed(int et, int law, const PatchArgs &pa, const MatParams &mp,
                                    const GroupArgs &ps, bool pdl, cudaStream_t s) {
  if (et == ET_TET4 && law == LAW_ELASTIC)
    return launch_patch<PatchTet4<LAW_ELASTIC, float>, true, 256, 3>(pa, mp, ps, pdl, s);
  if (et == ET_TET4 && law == LAW_NEOHOOKEAN)
    return launch_patch<PatchTet4<LAW_NEOHOOKEAN, float>, true, 256, 3>(pa, mp, ps, pdl, s);
  if (et == ET_HEX8 && law == LAW_ELASTIC)
    return launch_patch<PatchHex8X2<LAW_ELASTIC>, true, 128, 4>(pa, mp, ps, pdl, s);
  if (et == ET_HEX8 && law == LAW_NEOHOOKEAN)
    return launch_patch<PatchHex8X2<LAW_NEOHOOKEAN>, true, 128, 4>(pa, mp, ps, pdl, s);
  if (et == ET_TRI6 && law == LAW_PLASTIC) {
    if (pa.nq == 3) return launch_patch<PatchTri6<3, float>, true, 192, 4>(pa, mp, ps, pdl, s);
    return launch_patch<PatchTri6<6, float>, true, 192, 4>(pa, mp, ps, pdl, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace akb
