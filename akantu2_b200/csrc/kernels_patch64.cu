// Fused step kernels of the plain FP64 path (built with --fmad=false: every
// product and sum rounded on its own, like the CPU path).
#include "patch_launch.cuh"

namespace akb {

namespace {
// tetrahedra: the state first at every size (us per step, before / after: 48 k
// tetrahedra 5.20 / 4.86, 162 k 12.7 / 12.3, 1.3 M 74.7 / 73.1)
template <class EV>
cudaError_t launch_tet(const PatchArgs &pa, const MatParams &mp, const GroupArgs &ps, bool pdl,
                       cudaStream_t s) {
  if (pa.ahead) return launch_patch<EV, false, true, 256, 2, true>(pa, mp, ps, pdl, s);
  return launch_patch<EV, false, true, 256, 2>(pa, mp, ps, pdl, s);
}
// as in kernels_patch.cu
template <class EV>
cudaError_t launch_tri(const PatchArgs &pa, const MatParams &mp, const GroupArgs &ps, bool pdl,
                       cudaStream_t s) {
  if (pa.npatch <= kPatchSms) return launch_patch<EV, false, true, 256, 1>(pa, mp, ps, pdl, s);
  return launch_patch<EV, false, false, 192, 3>(pa, mp, ps, pdl, s);
}
}  // namespace

cudaError_t launch_patch_step_fp64(int et, int law, const PatchArgs &pa, const MatParams &mp,
                                   const GroupArgs &ps, bool pdl, cudaStream_t s) {
  if (et == ET_TET4 && law == LAW_ELASTIC)
    return launch_tet<PatchTet4<LAW_ELASTIC, double>>(pa, mp, ps, pdl, s);
  if (et == ET_TET4 && law == LAW_NEOHOOKEAN)
    return launch_tet<PatchTet4<LAW_NEOHOOKEAN, double>>(pa, mp, ps, pdl, s);
  if (et == ET_TRI6 && law == LAW_PLASTIC)
    return pa.nq == 3 ? launch_tri<PatchTri6<3, double>>(pa, mp, ps, pdl, s)
                      : launch_tri<PatchTri6<6, double>>(pa, mp, ps, pdl, s);
  return cudaErrorInvalidValue;
}

}  // namespace akb
