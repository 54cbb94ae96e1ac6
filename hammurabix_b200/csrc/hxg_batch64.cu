// hxg_batch64.cu -- instantiations of the FP64 group kernels (see hxg_batch.cu).
#include "hxg_dispatch.cuh"
#include "hxg_fp64.cuh"
#include "hxg_internal.h"

namespace hxg {

int shell64_instance(const ShellLaunch &P) {
  return shell_key(shape64(P), P.ext != nullptr, fast_models(P) && P.fast_ok);
}

cudaError_t launch_group64(cudaStream_t s, int nf, const ShellLaunch &P, const void *g,
                           unsigned blocks, unsigned threads) {
  const bool fast = fast_models(P) && P.fast_ok;
  return by_shape(shape64(P), P.ext != nullptr, [&](auto ng, auto ext) {
    constexpr int NG = decltype(ng)::value;
    constexpr bool E = decltype(ext)::value;
    by_passes(nf, [&](auto f) {
      constexpr int NF = decltype(f)::value;
      const auto &G = *static_cast<const PlanGroup<NF> *>(g);
      if (fast)
        shell_fp64_group_kernel<NG, false, NF, true><<<blocks, threads, 0, s>>>(G);
      else
        shell_fp64_group_kernel<NG, E, NF, false><<<blocks, threads, 0, s>>>(G);
    });
  });
}

}  // namespace hxg
