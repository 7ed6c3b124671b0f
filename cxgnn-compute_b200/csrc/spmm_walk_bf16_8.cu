// Tiled walk, bf16 rows read in vectors of 8 bytes.
#include "spmm_walk_impl.cuh"

namespace cxg {
bool walk_launch_bf16_8(const WalkArgs &a, int valmode, bool share, cudaStream_t st, int *resident_tiles) {
  return walk::launch<__nv_bfloat16, 8>(a, valmode, share, st, resident_tiles);
}
}  // namespace cxg
