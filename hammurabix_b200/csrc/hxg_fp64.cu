// hxg_fp64.cu -- instantiations of the FP64 shell kernels.
#include "hxg_dispatch.cuh"
#include "hxg_fp64.cuh"
#include "hxg_internal.h"

namespace hxg {

cudaError_t launch_shell64(cudaStream_t s, const ShellLaunch &P, unsigned blocks,
                           unsigned threads) {
  const bool fast = fast_models(P) && P.fast_ok;
  return by_shape(shape64(P), P.ext != nullptr, [&](auto ng, auto ext) {
    constexpr int NG = decltype(ng)::value;
    constexpr bool E = decltype(ext)::value;
    if (fast)
      shell_fp64_kernel<NG, false, true><<<blocks, threads, 0, s>>>(P);
    else
      shell_fp64_kernel<NG, E, false><<<blocks, threads, 0, s>>>(P);
  });
}

cudaError_t launch_shell64_multi(cudaStream_t s, const ShellLaunch &P, int nf, const void *fq,
                                 unsigned blocks, unsigned threads) {
  const bool fast = fast_models(P) && P.fast_ok;
  return by_shape(shape64(P), P.ext != nullptr, [&](auto ng, auto ext) {
    constexpr int NG = decltype(ng)::value;
    constexpr bool E = decltype(ext)::value;
    const FreqSet<2> &F2 = *static_cast<const FreqSet<2> *>(fq);
    const FreqSet<3> &F3 = *static_cast<const FreqSet<3> *>(fq);
    if (fast && nf == 2)
      shell_fp64_multi_kernel<NG, false, 2, true><<<blocks, threads, 0, s>>>(P, F2);
    else if (fast)
      shell_fp64_multi_kernel<NG, false, 3, true><<<blocks, threads, 0, s>>>(P, F3);
    else if (nf == 2)
      shell_fp64_multi_kernel<NG, E, 2, false><<<blocks, threads, 0, s>>>(P, F2);
    else
      shell_fp64_multi_kernel<NG, E, 3, false><<<blocks, threads, 0, s>>>(P, F3);
  });
}

}  // namespace hxg
