// hxg_dispatch.cuh -- choice of a kernel instantiation from a launch's shape.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

namespace hxg {

// The kernels are instantiated per grid-group count (0, 1, up to
// kMaxGroups) and per use of the Jaffe / JF12 / YMW16 blocks.
template <typename F>
inline cudaError_t by_shape(int ngroups, bool ext, F &&f) {
  const auto g = [&](auto ng) {
    if (ext)
      f(ng, std::true_type{});
    else
      f(ng, std::false_type{});
  };
  if (ngroups == 0)
    g(std::integral_constant<int, 0>{});
  else if (ngroups == 1)
    g(std::integral_constant<int, 1>{});
  else
    g(std::integral_constant<int, 4>{});
  return cudaGetLastError();
}

}  // namespace hxg
