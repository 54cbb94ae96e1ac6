// hxg_adjoint.cu -- instantiations of the adjoint shell kernels.
#include "hxg_adjoint.cuh"
#include "hxg_adjoint32.cuh"
#include "hxg_internal.h"

namespace hxg {

cudaError_t launch_adjoint(cudaStream_t s, const AdjointLaunch &A,
                           unsigned blocks, unsigned threads) {
  const bool ext = A.F.ext != nullptr;
  const bool fast = fast_models(A.F) && A.F.fast_ok;
  if (A.F.ngroups == 0) {
    if (fast)
      shell_fp64_adjoint_kernel<0, false, true><<<blocks, threads, 0, s>>>(A);
    else if (ext)
      shell_fp64_adjoint_kernel<0, true, false><<<blocks, threads, 0, s>>>(A);
    else
      shell_fp64_adjoint_kernel<0, false, false><<<blocks, threads, 0, s>>>(A);
  } else {
    if (fast)
      shell_fp64_adjoint_kernel<1, false, true><<<blocks, threads, 0, s>>>(A);
    else if (ext)
      shell_fp64_adjoint_kernel<1, true, false><<<blocks, threads, 0, s>>>(A);
    else
      shell_fp64_adjoint_kernel<1, false, false><<<blocks, threads, 0, s>>>(A);
  }
  return cudaGetLastError();
}

cudaError_t launch_adjoint32(cudaStream_t s, const AdjointLaunch &A, unsigned blocks,
                             unsigned threads) {
  const bool fin = A.F.fast_ok;
  if (A.F.ngroups == 0 && fin)
    shell_fp32c_adjoint_kernel<0, true><<<blocks, threads, 0, s>>>(A);
  else if (A.F.ngroups == 0)
    shell_fp32c_adjoint_kernel<0, false><<<blocks, threads, 0, s>>>(A);
  else if (fin)
    shell_fp32c_adjoint_kernel<1, true><<<blocks, threads, 0, s>>>(A);
  else
    shell_fp32c_adjoint_kernel<1, false><<<blocks, threads, 0, s>>>(A);
  return cudaGetLastError();
}

}  // namespace hxg
