// Fused step kernels of the plain FP64 path (built with --fmad=false: every
// product and sum rounded on its own, like the CPU path).
#include "patch_launch.cuh"

namespace akb {

cudaError_t launch_patch_step_fp64(int et, int law, const PatchArgs &pa, const MatParams &mp,
                                   const GroupArgs &ps, bool pdl, cudaStream_t s) {
  if (et == ET_TET4 && law == LAW_ELASTIC)
    return launch_patch<PatchTet4<LAW_ELASTIC, double>, false, 256, 2>(pa, mp, ps, pdl, s);
  if (et == ET_TET4 && law == LAW_NEOHOOKEAN)
    return launch_patch<PatchTet4<LAW_NEOHOOKEAN, double>, false, 256, 2>(pa, mp, ps, pdl, s);
  if (et == ET_TRI6 && law == LAW_PLASTIC) {
    if (pa.nq == 3) return launch_patch<PatchTri6<3, double>, false, 192, 3>(pa, mp, ps, pdl, s);
    return launch_patch<PatchTri6<6, double>, false, 192, 3>(pa, mp, ps, pdl, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace akb
