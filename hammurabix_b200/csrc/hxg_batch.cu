// hxg_batch.cu -- instantiations of the batch kernels that only a batch launches: the
// FP32C groups and persistent kernels (the FP64 groups are in hxg_batch64.cu).  Apart
// from the shell kernels, since the first launch of a kernel loads its whole file's
// code: with these among the shell kernels a process's first call took 41 ms in FP32C
// and 70 ms in FP64, 14 and 28 ms without.
#include "hxg_batch.cuh"
#include "hxg_dispatch.cuh"
#include "hxg_internal.h"

namespace hxg {

int shell_instance(bool fp32, const ShellLaunch &P) {
  return fp32 ? shell_key(P.ngroups, P.ext != nullptr, fast_models(P) && P.fast_ok)
              : shell64_instance(P);
}

cudaError_t launch_shell_group(cudaStream_t s, bool fp32, int nf, const ShellLaunch &P,
                               const void *g, unsigned blocks, unsigned threads) {
  if (!fp32) return launch_group64(s, nf, P, g, blocks, threads);
  const bool fast = fast_models(P) && P.fast_ok;
  return by_shape(P.ngroups, P.ext != nullptr, [&](auto ng, auto ext) {
    constexpr int NG = decltype(ng)::value;
    constexpr bool E = decltype(ext)::value;
    by_passes(nf, [&](auto f) {
      constexpr int NF = decltype(f)::value;
      const auto &G = *static_cast<const PlanGroup<NF> *>(g);
      if (fast)
        shell_fp32c_group_kernel<NG, false, NF, true><<<blocks, threads, 0, s>>>(G);
      else
        shell_fp32c_group_kernel<NG, E, NF, false><<<blocks, threads, 0, s>>>(G);
    });
  });
}

cudaError_t launch_batch_level(cudaStream_t s, int ngroups, bool ext, bool fast,
                               const BatchLevel &B, unsigned blocks) {
  return by_shape(ngroups, ext, [&](auto ng, auto ex) {
    constexpr int NG = decltype(ng)::value;
    constexpr bool E = decltype(ex)::value;
    if (fast)
      batch_fp32c_kernel<NG, false, true><<<blocks, 256, 0, s>>>(B);
    else
      batch_fp32c_kernel<NG, E, false><<<blocks, 256, 0, s>>>(B);
  });
}

cudaError_t launch_batch_level_multi(cudaStream_t s, int ngroups, bool ext, bool fast, int nf,
                                     const void *B, unsigned blocks) {
  return by_shape(ngroups, ext, [&](auto ng, auto ex) {
    constexpr int NG = decltype(ng)::value;
    constexpr bool E = decltype(ex)::value;
    const auto &B2 = *static_cast<const BatchLevelMulti<2> *>(B);
    const auto &B3 = *static_cast<const BatchLevelMulti<3> *>(B);
    if (fast && nf == 2)
      batch_fp32c_multi_kernel<NG, false, 2, true><<<blocks, HXG_BATCH_MULTI_THREADS, 0, s>>>(B2);
    else if (fast)
      batch_fp32c_multi_kernel<NG, false, 3, true><<<blocks, HXG_BATCH_MULTI_THREADS, 0, s>>>(B3);
    else if (nf == 2)
      batch_fp32c_multi_kernel<NG, E, 2, false><<<blocks, HXG_BATCH_MULTI_THREADS, 0, s>>>(B2);
    else
      batch_fp32c_multi_kernel<NG, E, 3, false><<<blocks, HXG_BATCH_MULTI_THREADS, 0, s>>>(B3);
  });
}

cudaError_t batch_multi_occupancy(int ngroups, bool ext, bool fast, int nf, int *blocks_per_sm) {
  const void *f = nullptr;
  by_shape(ngroups, ext, [&](auto ng, auto ex) {
    constexpr int NG = decltype(ng)::value;
    constexpr bool E = decltype(ex)::value;
    if (fast && nf == 2)
      f = (const void *)batch_fp32c_multi_kernel<NG, false, 2, true>;
    else if (fast)
      f = (const void *)batch_fp32c_multi_kernel<NG, false, 3, true>;
    else if (nf == 2)
      f = (const void *)batch_fp32c_multi_kernel<NG, E, 2, false>;
    else
      f = (const void *)batch_fp32c_multi_kernel<NG, E, 3, false>;
  });
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, f, HXG_BATCH_MULTI_THREADS, 0);
}

cudaError_t batch_level_occupancy(int ngroups, bool ext, bool fast, int *blocks_per_sm) {
  const void *f = nullptr;
  by_shape(ngroups, ext, [&](auto ng, auto ex) {
    constexpr int NG = decltype(ng)::value;
    constexpr bool E = decltype(ex)::value;
    if (fast)
      f = (const void *)batch_fp32c_kernel<NG, false, true>;
    else
      f = (const void *)batch_fp32c_kernel<NG, E, false>;
  });
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, f, 256, 0);
}

}  // namespace hxg
