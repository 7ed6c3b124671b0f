// Interface between cxg_spmm_csr and its register-staged tiled walk (spmm_walk*.cu).
#pragma once
#include "common.cuh"

namespace cxg {

// Longer chains of partial rows are added in ordered blocks of this many partials.
constexpr int kWalkSeqPartials = 64;

// Word of the header that counts the tiles handed out behind the first round.
constexpr int kWalkHdrNext = 8;

// What the plan leaves per tile: its first row, its first edge and that row's range of edges (what the walk and the fix-up
// would otherwise fetch from ptr, one round trip behind the record). The entry behind the last tile ends the last one.
struct __align__(16) WalkTile {
  uint32_t row, begin, row_begin, row_end;
};
// The same of the fused GAT walks, which count in 64 bits.
struct __align__(16) WideTile {
  int64_t row, begin;
};
static_assert(sizeof(WalkTile) == sizeof(WideTile), "one layout holds either");

struct WalkArgs {
  const void *ptr;
  const void *idx;
  const void *x;
  void *y;
  const float *edge_val;
  const int32_t *edge_rel;
  int64_t n_dst;
  int64_t nnz;  // edges the caller declared: no kernel goes beyond
  int64_t rel_stride;
  int64_t max_tiles;
  int row_bytes, width, feat, heads, ptr_bytes, idx_bytes, reduce;
  int x_pitch;    // bytes from a row of x to the next (row_bytes, or those of the copied rows)
  int tile;       // edges per tile
  int accumulate; // 1: the output is added to
  int wide_tiles;
  int whole_rows; // 1: rows of up to `tile` edges are never cut (see spmm_walk_impl.cuh)
  uint64_t tile_magic;  // ceil(2^64 / tile), 0: divide
  int32_t *hdr;
  void *tiles;      // [tile + 1] WalkTile or (wide_tiles) WideTile
  int32_t *count;   // [tile] finished blocks of the long chain that starts in the tile
  float *partials;  // [tile][2][part_stride]: head partial, tail partial
  int part_stride;  // width in whole 16-byte vectors, or width
  // rows copied to whole 16-byte vectors by the plan kernel's blocks behind the first plan_blocks (x is that copy then)
  const void *x_rows;     // the caller's rows
  int64_t copy_vectors;   // 16-byte vectors of the copy, 0: none
  unsigned plan_blocks;
};

struct WalkLayout {
  size_t hdr, tiles, count, partials, total;
  int64_t max_tiles;
};

// part_stride: floats per partial, at least the width.
int walk_layout(int64_t nnz, int64_t part_stride, int tile, WalkLayout *L);
// Floats per partial where there is room: whole 16-byte vectors.
constexpr int64_t walk_part_stride(int64_t width) { return (width + 3) / 4 * 4; }
// True when the walk covers the descriptor: no edge mask, output rows in order and overwritten or (without edge values)
// added to, rows that fit its lane layouts.
bool walk_eligible(const cxg_spmm_desc *d);
// The plan kernel for a.ptr, a.tile, a.whole_rows: fills hdr, tiles, count (and sets a.tile_magic).
void walk_plan_run(WalkArgs &a, cudaStream_t st);
// The walk alone over the plan and the weights per (edge, head) in `a` (fp32 rows in vectors of vb bytes, heads a power of two),
// behind which walk_weights_slack bytes can be read. With resident_tiles set it only tells how many tiles are walked at the
// same time. False, too, for tiles of more than kWeightedTile edges.
constexpr int kWeightedTile = 256;   // most edges of a tile of that walk
constexpr int kWalkInFlight = 8;     // most edges that a lane has in flight
// The lane groups of a warp step together until the longest of their tiles ends, and read weights at every step: a last tile
// of one edge beside a full one is read on to where it would end if it were full, in whole steps.
constexpr size_t walk_weights_slack(int heads) { return static_cast<size_t>(kWeightedTile + kWalkInFlight) * heads * sizeof(float); }
bool walk_weighted(const WalkArgs &a, int vb, cudaStream_t st, int *resident_tiles);
// Edges per tile for that many.
int walk_tile_of_waves(int64_t nnz, int64_t resident);
// Edges per tile when `resident` tiles are walked at the same time: whole waves of up to 256 edges, or 512.
int walk_whole_waves(int64_t nnz, int64_t resident, int round);
// Edges per tile of cxg_spmm_csr_static, whose scratch has a fixed size: these decide which graphs it takes.
int walk_static_tile_edges(const cxg_spmm_desc *d);
// Edges per tile for this call (desc->split_edges when set).
int walk_tile_edges(const cxg_spmm_desc *d, bool copied);
// rows: scratch for a copy of the n_src rows of x, of the size that walk_copy_bytes gives, or null.
int walk_launch(const cxg_spmm_desc *d, bool whole_rows, int64_t n_src, void *rows, void *workspace, size_t workspace_bytes,
                cudaStream_t st);
// Bytes of a copy of x in rows of whole 16-byte vectors, where reading that copy is worth making it; otherwise 0.
size_t walk_copy_bytes(const cxg_spmm_desc *d, int64_t n_src);

// The aggregation of a.ptr, idx, x, y, edge_val as one launch of clusters (spmm_small.cu): rows of up to 64 vectors of 16
// bytes or 128 of fewer, up to small_most_rows() of them. False: no kernel for it.
bool small_launch(const WalkArgs &a, int dtype, int vb, cudaStream_t st);
int small_most_rows();

// One launcher per element type and vector width, each in a translation unit of its own. False: no kernel for it. With
// resident_tiles set nothing is launched: it receives the number of tiles that are walked at the same time.
bool walk_launch_f32_16(const WalkArgs &a, int valmode, bool share, cudaStream_t st, int *resident_tiles);
bool walk_launch_f32_8(const WalkArgs &a, int valmode, bool share, cudaStream_t st, int *resident_tiles);
bool walk_launch_f32_4(const WalkArgs &a, int valmode, bool share, cudaStream_t st, int *resident_tiles);
bool walk_launch_bf16_16(const WalkArgs &a, int valmode, bool share, cudaStream_t st, int *resident_tiles);
bool walk_launch_bf16_8(const WalkArgs &a, int valmode, bool share, cudaStream_t st, int *resident_tiles);
bool walk_launch_bf16_4(const WalkArgs &a, int valmode, bool share, cudaStream_t st, int *resident_tiles);
bool walk_launch_f32_copy(const WalkArgs &a, int valmode, bool share, cudaStream_t st, int *resident_tiles);
bool walk_launch_bf16_copy(const WalkArgs &a, int valmode, bool share, cudaStream_t st, int *resident_tiles);
bool walk_launch_bf16_2(const WalkArgs &a, int valmode, bool share, cudaStream_t st, int *resident_tiles);

#ifdef __CUDACC__
__device__ __forceinline__ WalkTile load_tile(const WalkArgs &a, int64_t t) {
  const uint4 v = reinterpret_cast<const uint4 *>(a.tiles)[t];
  return WalkTile{v.x, v.y, v.z, v.w};
}
// Edges the kernels walk: ptr[n_dst], but never more than the caller declared.
__device__ __forceinline__ int64_t edge_total(const WalkArgs &a) {
  const int64_t e = load_ptr(a.ptr, a.n_dst, a.ptr_bytes);
  return e > a.nnz ? a.nnz : e;
}
#endif

}  // namespace cxg
