// Launch of one fused-step kernel, shared by its translation units.
#pragma once

#include <atomic>

#include "dispatch.cuh"
#include "fe_patch.cuh"

namespace akb {

template <class EV, bool KAHAN, bool MULTI, bool EARLY, bool AHEAD, int THREADS, int MINB>
cudaError_t launch_patch_kernel(const PatchArgs &pa, const MatParams &mp, const GroupArgs &ps, bool pdl,
                         cudaStream_t s) {
  auto kern = k_patch_step<EV, KAHAN, MULTI, EARLY, AHEAD, THREADS, MINB>;
  // shared memory above 48 KB is allowed once per kernel and device (a
  // host-side attribute of the current device, no stream work)
  static std::atomic<unsigned long long> opted{0ull};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (!(opted.load(std::memory_order_relaxed) & bit)) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kPatchMaxSmem);
    if (e != cudaSuccess) return e;
    opted.fetch_or(bit, std::memory_order_relaxed);
  }
  static_assert(patch_stage_bytes<EV, THREADS>() <= kPatchStageSmem, "staging");
  const size_t smem = pa.smem + patch_stage_bytes<EV, THREADS>();
  if (smem > kPatchMaxSmem) return cudaErrorInvalidConfiguration;
  return launch_step_smem(pdl, kern, (unsigned)pa.npatch + (pa.presc.count ? 1 : 0), THREADS,
                          smem, s, pa, mp, ps);
}

template <class EV, bool KAHAN, bool EARLY, int THREADS, int MINB, bool AHEAD = false>
cudaError_t launch_patch(const PatchArgs &pa, const MatParams &mp, const GroupArgs &ps, bool pdl,
                         cudaStream_t s) {
  return pa.multi
             ? launch_patch_kernel<EV, KAHAN, true, EARLY, AHEAD, THREADS, MINB>(pa, mp, ps, pdl, s)
             : launch_patch_kernel<EV, KAHAN, false, EARLY, AHEAD, THREADS, MINB>(pa, mp, ps, pdl,
                                                                                 s);
}

}  // namespace akb
