// hxg_dispatch.cuh -- choice of a kernel instantiation from a launch's shape.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

namespace hxg {

// The grid-group count by whose instantiation an FP64 launch runs.  The one-grid
// kernels read a voxel record in one 32-byte load and index records with 32 bits;
// a caller's own records (hxg_write_grid_noalloc) need only 16-byte alignment and
// can be more than 2^32 - 1, so those take the kernel for several grids, whose
// loads are 16 bytes wide and whose indices have 64 bits.
inline int fp64_groups(int ngroups, const void *rec, int nx, int ny, int nz) {
  const bool one = (reinterpret_cast<uintptr_t>(rec) & 31) == 0 &&
                   (unsigned __int128)nx * ny * nz <= 0xFFFFFFFFu;
  return ngroups == 1 && !one ? 2 : ngroups;
}

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

// A number for the instantiation that by_shape and the kFast rule choose.
inline int shell_key(int ngroups, bool ext, bool fast) {
  return fast ? std::min(ngroups, 2) : 3 + 2 * std::min(ngroups, 2) + (ext ? 1 : 0);
}

// f with the pass count 1, 2 or 3 as a constant.
template <typename F>
inline void by_passes(int nf, F &&f) {
  if (nf == 1)
    f(std::integral_constant<int, 1>{});
  else if (nf == 2)
    f(std::integral_constant<int, 2>{});
  else
    f(std::integral_constant<int, 3>{});
}

}  // namespace hxg
