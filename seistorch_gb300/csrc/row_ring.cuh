// Row bookkeeping of nn_conv.cu's ring, apart from its barriers.
#pragma once

#ifndef __CUDACC__  // also compiled for the host, by the test of it
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace sgb {
namespace nn {

// Waits for the next `need` rows, wait(row) each; `rows` counts those that have
// arrived.  A row whose wait fails is not counted: its copy may still be in flight,
// and the kernel's drain waits for every row from `rows` on.
template <class Wait>
__host__ __device__ __forceinline__ bool take_rows(int need, int& rows, const Wait& wait) {
  for (int i = 0; i < need; ++i) {
    if (!wait(rows)) return false;
    ++rows;
  }
  return true;
}

}  // namespace nn
}  // namespace sgb
