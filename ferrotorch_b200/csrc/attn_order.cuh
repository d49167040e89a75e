// The order in which the CTAs of the attention kernels take their work.
#pragma once
#include <cuda_runtime.h>

namespace ft {

struct AttnBlock {
  int block, head, batch;
};

// Under a causal mask the blocks of rows differ in weight, and CTAs start in the order of their number.  All heads and sequences of the
// heaviest block go first, then those of the next (blocks count from the heaviest): what is left for the end is light, so the SMs finish
// together.  With the blocks of one head in a row, its heaviest block could start when the others were done (1 x 8192 tokens, 32 / 8 heads
// of 128, attention and its backward: 2869 us, 2577 now).  Without a mask all weigh the same, and the blocks
// of a head stay together for the sake of L2.
__device__ __forceinline__ AttnBlock attn_block(int blocks, int heads, bool by_weight) {
  const unsigned id = blockIdx.x, n = blocks;
  if (by_weight) {
    const unsigned all = gridDim.x / n, block = id / all, r = id - block * all;
    return {static_cast<int>(block), static_cast<int>(r % heads), static_cast<int>(r / heads)};
  }
  const unsigned r = id / n;
  return {static_cast<int>(id - r * n), static_cast<int>(r % heads), static_cast<int>(r / heads)};
}

inline dim3 attn_grid(int blocks, int heads, int batch) { return dim3(static_cast<unsigned>(blocks) * heads * batch); }

}  // namespace ft
