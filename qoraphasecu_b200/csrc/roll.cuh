// Cyclic rolls between centre-origin and FFT order, walked row by row: one
// division per row instead of four per element.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "aux_kernels.cuh"

namespace qpb {

// Offset of each axis: out[i] = in[(i + off) mod n], off = n / 2 to FFT order
// and n - n / 2 to centre origin.
struct RollOffsets {
  int o0, o1, o2;
};
inline RollOffsets roll_offsets(Dims3 d, bool to_fft_order) {
  auto off = [&](int len) { return to_fft_order ? len / 2 : len - len / 2; };
  return {off(d.d0), off(d.d1), off(d.d2)};
}

inline constexpr int kRollThreads = 256;

// Threads of a block: as many along x as a row of d2 elements fills (32..256),
// the rest on further rows.
inline dim3 roll_block(Dims3 d) {
  int bx = 32;
  while (bx < kRollThreads && bx < d.d2) bx *= 2;
  return {static_cast<unsigned>(bx), static_cast<unsigned>(kRollThreads / bx), 1};
}
// Blocks for the rows of one array, at most `most`.
inline unsigned roll_blocks(Dims3 d, int most) {
  const long long rows = static_cast<long long>(d.d0) * d.d1;
  const int by = kRollThreads / static_cast<int>(roll_block(d).x);
  return static_cast<unsigned>(std::min<long long>((rows + by - 1) / by, most));
}

// f(i, source, row, x) for every element i = row d2 + x of the rolled array
// and its source element, the rows spread over the grid's x dimension.
template <class F>
__device__ __forceinline__ void for_rolled(Dims3 d, RollOffsets o, F&& f) {
  const int rows = d.d0 * d.d1;
  for (int row = blockIdx.x * blockDim.y + threadIdx.y; row < rows; row += gridDim.x * blockDim.y) {
    const int z = row / d.d1;
    int sy = row - z * d.d1 + o.o1;
    int sz = z + o.o0;
    if (sy >= d.d1) sy -= d.d1;
    if (sz >= d.d0) sz -= d.d0;
    const long long at = static_cast<long long>(row) * d.d2;
    const long long from = (static_cast<long long>(sz) * d.d1 + sy) * d.d2;
    for (int x = threadIdx.x; x < d.d2; x += blockDim.x) {
      int sx = x + o.o2;
      if (sx >= d.d2) sx -= d.d2;
      f(at + x, from + sx, row, x);
    }
  }
}

}  // namespace qpb
