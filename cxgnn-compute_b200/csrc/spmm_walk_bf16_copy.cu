// Tiled walk, bf16 rows that the plan kernel has copied to whole 16-byte vectors.
#include "spmm_walk_impl.cuh"

namespace cxg {
bool walk_launch_bf16_copy(const WalkArgs &a, int valmode, bool share, cudaStream_t st, int *resident_tiles) {
  return walk::launch_copy<__nv_bfloat16>(a, valmode, share, st, resident_tiles);
}
}  // namespace cxg
