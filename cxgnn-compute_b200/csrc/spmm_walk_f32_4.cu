// Tiled walk, fp32 rows read in vectors of 4 bytes.
#include "spmm_walk_impl.cuh"

namespace cxg {
bool walk_launch_f32_4(const WalkArgs &a, int valmode, bool share, cudaStream_t st, int *resident_tiles) {
  return walk::launch<float, 4>(a, valmode, share, st, resident_tiles);
}
}  // namespace cxg
