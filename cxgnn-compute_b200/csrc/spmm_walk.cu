// Plan, fix-up and dispatch of the register-staged tiled walk (spmm_walk_impl.cuh).
#include "spmm_stream.cuh"
#include "spmm_walk.cuh"

namespace cxg {
namespace {

// Widest vector every row of x and y is aligned to; with several heads and edge values a vector stays inside one head.
int vector_bytes(const cxg_spmm_desc *d) {
  const int elem = d->dtype == CXG_F32 ? 4 : 2;
  const uint64_t row = static_cast<uint64_t>(d->feat) * d->heads * elem;
  const uint64_t bits = row | reinterpret_cast<uintptr_t>(d->x) | reinterpret_cast<uintptr_t>(d->y) |
                        ((d->heads > 1 && d->edge_val != nullptr) ? static_cast<uint64_t>(d->feat) * elem : 0);
  int vb = 16;
  while (bits % vb != 0) vb /= 2;
  return vb;
}

// e / tile
__device__ __forceinline__ int64_t tile_of(const WalkArgs &a, int64_t e) {
  const uint64_t v = static_cast<uint64_t>(e);
  return static_cast<int64_t>(a.tile_magic ? __umul64hi(v, a.tile_magic) : v / a.tile);
}

// Rows that own the first edge of a tile write the tile's record; a hub row that owns many is shared by its warp. One
// pass over ptr, so it costs what reading ptr costs (1 us for 170,000 rows, 17 us for 14 M), where a search per tile
// is a chain of 18 dependent loads (10 us). Also clears what the later kernels count in.
constexpr int kPlanRows = 4;  // rows per thread

__global__ void __launch_bounds__(256) walk_plan(const __grid_constant__ WalkArgs a) {
  const int64_t i0 = blockIdx.x * (256ll * kPlanRows) + threadIdx.x;
  int64_t raw_b[kPlanRows], raw_e[kPlanRows];
#pragma unroll
  for (int k = 0; k < kPlanRows; ++k) {
    const int64_t r = min(i0 + k * 256, a.n_dst - 1);
    raw_b[k] = load_ptr(a.ptr, r, a.ptr_bytes);
    raw_e[k] = load_ptr(a.ptr, r + 1, a.ptr_bytes);
  }
  const int64_t last = load_ptr(a.ptr, a.n_dst, a.ptr_bytes);
  const int64_t e_total = min(last, a.nnz);
  if (i0 < 64) a.hdr[i0] = (i0 == kSHdrError && last > a.nnz) ? kSErrEdgeCount : 0;
#pragma unroll
  for (int k = 0; k < kPlanRows; ++k)
    if (i0 + k * 256 < a.max_tiles) a.count[i0 + k * 256] = 0;
  if (i0 == 0) a.tiles[(e_total + a.tile - 1) / a.tile] = WalkTile{a.n_dst, e_total};
  auto record = [&](int64_t t, int64_t r, int64_t b, int64_t e) {
    const int64_t pos = t * a.tile;
    WalkTile w{r, pos};
    if (a.whole_rows && pos != b) {
      const int64_t at = b + tile_of(a, pos - b + a.tile - 1) * a.tile;
      if (e - b > a.tile && at < e)
        w.begin = at;
      else
        w = WalkTile{r + 1, e};
    }
    a.tiles[t] = w;
  };
#pragma unroll
  for (int k = 0; k < kPlanRows; ++k) {
    const int64_t i = i0 + k * 256;
    const int64_t rb = min(raw_b[k], e_total), re = i < a.n_dst ? min(raw_e[k], e_total) : rb;
    // tiles whose first edge lies in [rb, re)
    const int64_t t0 = tile_of(a, rb + a.tile - 1), t1 = re > rb ? tile_of(a, re + a.tile - 1) : t0;
    const bool many = t1 - t0 > 4;
    if (!many)
      for (int64_t t = t0; t < t1; ++t) record(t, i, rb, re);
    for (unsigned left = __ballot_sync(0xffffffffu, many); left != 0; left &= left - 1) {
      const int src = __ffs(left) - 1;
      const int64_t r = __shfl_sync(0xffffffffu, i, src), b = __shfl_sync(0xffffffffu, rb, src),
                    e = __shfl_sync(0xffffffffu, re, src), u0 = __shfl_sync(0xffffffffu, t0, src),
                    u1 = __shfl_sync(0xffffffffu, t1, src);
      for (int64_t t = u0 + (threadIdx.x & 31); t < u1; t += 32) record(t, r, b, e);
    }
  }
}

// Partial sums of the row's chain: element k > 0 is the head partial of tile ts + k, element 0 the tail partial of ts.
__device__ __forceinline__ float *chain_at(const WalkArgs &a, int64_t ts, int64_t k) {
  return a.partials + ((ts + k) * 2 + (k == 0 ? 1 : 0)) * a.width;
}

template <typename T, int VW>
__device__ __forceinline__ void finish_columns(const WalkArgs &a, T *dst, float (&s)[VW], int64_t deg) {
#pragma unroll
  for (int i = 0; i < VW; ++i) {
    float r = s[i];
    if (a.reduce == CXG_MEAN) r = __fdiv_rn(r, static_cast<float>(deg));
    if (a.accumulate) r += to_f32(dst[i]);
    dst[i] = from_f32<T>(r);
  }
}

// Adds n elements of the chain, step elements apart, from element k0 on, in order; `lanes` lanes of VW columns each. The
// result goes to `into` (fp32 scratch) or, when that is null, to the output row.
template <typename T, int VW>
__device__ __forceinline__ void chain_sum(const WalkArgs &a, int64_t ts, int64_t k0, int n, int step, float *into, int64_t row, int64_t deg,
                          int lane, int lanes) {
  constexpr int kDepth = 8;  // partials requested at once (16 halve the resident warps and cost more than they save)
  for (int c = lane * VW; c < a.width; c += lanes * VW) {
    float s[VW];
    auto load = [&](float (&v)[VW], const float *p) {
      if (VW == 4) {
        const float4 t = __ldcg(reinterpret_cast<const float4 *>(p));
        v[0] = t.x, v[1 % VW] = t.y, v[2 % VW] = t.z, v[3 % VW] = t.w;
      } else {
        v[0] = __ldcg(p);
      }
    };
    load(s, chain_at(a, ts, k0) + c);
    const int64_t stride = 2ll * step * a.width;
    const float *p = a.partials + (ts + k0) * 2 * a.width + c;
    for (int k = 1; k < n; k += kDepth) {
      float v[kDepth][VW];
#pragma unroll
      for (int u = 0; u < kDepth; ++u) {
        p += stride;
        if (k + u < n) load(v[u], p);
      }
#pragma unroll
      for (int u = 0; u < kDepth; ++u)
        if (k + u < n)
#pragma unroll
          for (int i = 0; i < VW; ++i) s[i] += v[u][i];
    }
    if (into != nullptr) {
#pragma unroll
      for (int i = 0; i < VW; ++i) into[c + i] = s[i];
    } else {
      finish_columns<T, VW>(a, static_cast<T *>(a.y) + row * a.width + c, s, deg);
    }
  }
}

// Adds the partials of the rows that tiles cut. A tile leads the first block of the chain that starts in it, and block
// k / 64 of the chain that runs through its start when it is that chain's element k, a multiple of 64. The leader that
// finishes a long chain's last block adds the block sums.
// A chain is a handful of loads that depend on one another, so latency is what counts: a warp looks `per` tiles over at
// once, a lane for each of a tile's two roles, and then adds as many chains side by side as there are `lanes`-wide groups
// in it (one tile after the other, a warp each: 72 us for 74,500 tiles of rows of 64 columns, now 33 us; 182,000 tiles of 128: 152 us).
template <typename T, int VW>
__global__ void __launch_bounds__(256, 3) walk_fix(const __grid_constant__ WalkArgs a, int per, int lanes) {
  dependency_wait();
  const int lane = threadIdx.x & 31;
  const int64_t e_total = edge_total(a);
  const int64_t t = (blockIdx.x * 8ll + (threadIdx.x >> 5)) * per + (lane & (per - 1));
  bool lead = false;
  int64_t row = 0, deg = 0;
  int ts = 0, k = 0, m = 0;
  if (lane < 2 * per && t < a.max_tiles && t * a.tile < e_total) {
    const WalkTile here = a.tiles[t], next = a.tiles[t + 1];  // not written behind the last tile, whose end is e_total
    const bool tail = lane < per;
    row = tail ? next.row : here.row;
    if (next.begin > here.begin && row < a.n_dst) {
      const int64_t rb = load_ptr(a.ptr, row, a.ptr_bytes);
      const int64_t re = min(load_ptr(a.ptr, row + 1, a.ptr_bytes), e_total);
      // cut by this tile's end, or by its start
      if (tail ? (rb < next.begin && rb >= here.begin) : rb < here.begin) {
        const int64_t first = tail ? t : tile_of(a, rb);
        ts = static_cast<int>(first), k = static_cast<int>(t - first);
        deg = re - rb;
        m = static_cast<int>(a.whole_rows ? tile_of(a, deg + a.tile - 1) : tile_of(a, re - 1) - first + 1);
        lead = k % kWalkSeqPartials == 0;
      }
    }
  }
  const int group = lane / lanes, groups = 32 / lanes, in_group = lane & (lanes - 1);
  const unsigned members = (lanes == 32 ? 0xffffffffu : ((1u << lanes) - 1) << (group * lanes));
  unsigned left = __ballot_sync(0xffffffffu, lead);
  while (left != 0) {
    unsigned mine = left;  // group g takes the g-th of the chains that are left
    for (int i = 0; i < group; ++i) mine &= mine - 1;
    for (int i = 0; i < groups; ++i) left &= left - 1;
    const int src = mine != 0 ? __ffs(mine) - 1 : 0;
    const int jts = __shfl_sync(0xffffffffu, ts, src), jk = __shfl_sync(0xffffffffu, k, src),
              jm = __shfl_sync(0xffffffffu, m, src);
    const int64_t jrow = __shfl_sync(0xffffffffu, row, src), jdeg = __shfl_sync(0xffffffffu, deg, src);
    if (mine != 0) {
      const int n_blocks = (jm + kWalkSeqPartials - 1) / kWalkSeqPartials;
      int k0 = jk, n = min(kWalkSeqPartials, jm - jk), step = 1;
      float *into = n_blocks == 1 ? nullptr : chain_at(a, jts, jk);
#pragma unroll 1
      while (true) {
        chain_sum<T, VW>(a, jts, k0, n, step, into, jrow, jdeg, in_group, lanes);
        if (into == nullptr) break;
        __threadfence();
        __syncwarp(members);
        int old = 0;
        if (in_group == 0) old = atomicAdd(a.count + jts, 1);
        old = __shfl_sync(members, old, group * lanes);
        if (old + 1 != n_blocks) break;
        __threadfence();
        k0 = 0, n = n_blocks, step = kWalkSeqPartials, into = nullptr;
      }
    }
    __syncwarp();
  }
}

bool dispatch(const cxg_spmm_desc *d, const WalkArgs &a, cudaStream_t st, int *resident_tiles) {
  const int valmode = d->flags & CXG_SPMM_ACCUMULATE ? 4
                      : d->edge_val == nullptr       ? (d->reduce == CXG_MEAN ? 3 : 0)
                                                     : (d->heads == 1 ? 1 : 2);
  const bool share = (d->flags & CXG_SPMM_SHARE_SMS) != 0;
  int vb = vector_bytes(d);
  // narrow rows take the vector that occupies eight lanes, the fewest a tile is given
  while (vb > 4 && a.row_bytes <= 4 * vb) vb /= 2;
  if (d->dtype == CXG_F32)
    return vb == 16  ? walk_launch_f32_16(a, valmode, share, st, resident_tiles)
           : vb == 8 ? walk_launch_f32_8(a, valmode, share, st, resident_tiles)
                     : walk_launch_f32_4(a, valmode, share, st, resident_tiles);
  return vb == 16  ? walk_launch_bf16_16(a, valmode, share, st, resident_tiles)
         : vb == 8 ? walk_launch_bf16_8(a, valmode, share, st, resident_tiles)
         : vb == 4 ? walk_launch_bf16_4(a, valmode, share, st, resident_tiles)
                   : walk_launch_bf16_2(a, valmode, share, st, resident_tiles);
}

}  // namespace

int walk_layout(int64_t nnz, int64_t width, int tile, WalkLayout *L) {
  const int64_t max_tiles = (nnz + tile - 1) / tile + 1;
  if (max_tiles > INT32_MAX) return CXG_ELIMIT;
  size_t off = 0;
  L->hdr = off;
  off += 64 * sizeof(int32_t);
  L->tiles = off;
  off = align_up(off + static_cast<size_t>(max_tiles + 1) * sizeof(WalkTile), 256);
  L->count = off;
  off = align_up(off + static_cast<size_t>(max_tiles) * sizeof(int32_t), 256);
  L->partials = off;
  off = align_up(off + static_cast<size_t>(max_tiles) * 2 * width * sizeof(float), 256);
  L->total = off;
  L->max_tiles = max_tiles;
  return CXG_OK;
}

bool walk_eligible(const cxg_spmm_desc *d) {
  if (d->edge_mask != nullptr || d->targets != nullptr) return false;
  if ((d->flags & CXG_SPMM_ACCUMULATE) && d->edge_val != nullptr) return false;
  const int elem = d->dtype == CXG_F32 ? 4 : 2;
  const int64_t row_bytes = static_cast<int64_t>(d->feat) * d->heads * elem;
  const int vb = vector_bytes(d);
  if (vb < elem) return false;
  return row_bytes <= (vb == 16 ? 128 : 256) * vb;
}

void walk_plan_run(WalkArgs &a, cudaStream_t st) {
  a.tile_magic = a.tile > 1 && a.tile < 30000 ? ~0ull / static_cast<uint64_t>(a.tile) + 1 : 0;  // exact up to 2^34 edges
  const int64_t threads = ((a.n_dst > a.max_tiles ? a.n_dst : a.max_tiles) + kPlanRows - 1) / kPlanRows;
  walk_plan<<<static_cast<unsigned>((threads + 255) / 256), 256, 0, st>>>(a);
}

int walk_whole_waves(int64_t nnz, int64_t resident) {
  // Whole waves: every resident group gets the same number of tiles, so many that a tile has at most 256 edges (2.3 M
  // edges, F = 128: 145 us with 3.1 waves of 160 edges, 131 us with 1.9 of 256). From four waves of 512 edges on the
  // last one no longer matters and the longer tile costs less (126 M edges: 5 % over 256). At least 64 edges, so that
  // small graphs do not become all borders.
  if (nnz >= 2048 * resident) return 512;
  const int64_t waves = (nnz + 256 * resident - 1) / (256 * resident);
  const int64_t t = waves > 0 ? (nnz + waves * resident - 1) / (waves * resident) : 0;
  return t < 64 ? 64 : static_cast<int>((t + 31) / 32 * 32);
}

int walk_tile_edges(const cxg_spmm_desc *d) {
  if (d->split_edges > 0) return d->split_edges;
  WalkArgs a;
  a.row_bytes = d->feat * d->heads * (d->dtype == CXG_F32 ? 4 : 2);
  int resident = kNumSM * 32;
  dispatch(d, a, nullptr, &resident);
  return walk_whole_waves(d->nnz, resident);
}

int walk_launch(const cxg_spmm_desc *d, bool whole_rows, void *workspace, size_t workspace_bytes, cudaStream_t st) {
  const int tile = walk_tile_edges(d);
  WalkArgs a;
  a.ptr = d->ptr, a.idx = d->idx, a.x = d->x, a.y = d->y;
  a.edge_val = d->edge_val, a.edge_rel = d->edge_rel;
  a.n_dst = d->n_dst, a.nnz = d->nnz, a.rel_stride = d->rel_stride;
  a.feat = d->feat, a.heads = d->heads, a.width = d->feat * d->heads;
  a.row_bytes = a.width * (d->dtype == CXG_F32 ? 4 : 2);
  a.ptr_bytes = d->ptr_bytes, a.idx_bytes = d->idx_bytes, a.reduce = d->reduce;
  a.accumulate = (d->flags & CXG_SPMM_ACCUMULATE) ? 1 : 0;
  a.tile = tile;
  a.whole_rows = whole_rows ? 1 : 0;
  WalkLayout L;
  const int rc = walk_layout(d->nnz, a.width, tile, &L);
  if (rc != CXG_OK) return set_error(rc, "cxg_spmm_csr: graph too large for 32-bit tile ids");
  if (workspace == nullptr || workspace_bytes < L.total)
    return set_error(CXG_EWORKSPACE, "cxg_spmm_csr: workspace %zu bytes, need %zu", workspace_bytes, L.total);
  char *ws = reinterpret_cast<char *>(workspace);
  a.hdr = reinterpret_cast<int32_t *>(ws + L.hdr);
  a.tiles = reinterpret_cast<WalkTile *>(ws + L.tiles);
  a.count = reinterpret_cast<int32_t *>(ws + L.count);
  a.partials = reinterpret_cast<float *>(ws + L.partials);
  a.max_tiles = L.max_tiles;
  walk_plan_run(a, st);
  if (!dispatch(d, a, st, nullptr)) return set_error(CXG_EUNSUPPORTED, "cxg_spmm_csr: rows of %d bytes", a.row_bytes);
  // tiles a warp looks over: one while the chip holds a warp for each, up to sixteen (two roles on 32 lanes)
  int per = 1;
  while (per < 16 && L.max_tiles > static_cast<int64_t>(per) * kNumSM * 24) per *= 2;
  const unsigned fg = static_cast<unsigned>((L.max_tiles + 8 * per - 1) / (8 * per));
  const bool v4 = a.width % 4 == 0;
  int lanes = 1;  // per chain
  while (lanes < 32 && lanes * (v4 ? 4 : 1) < a.width) lanes *= 2;
  cudaError_t e;
  if (d->dtype == CXG_F32)
    e = v4 ? launch_dependent(walk_fix<float, 4>, fg, 256, 0, st, a, per, lanes)
           : launch_dependent(walk_fix<float, 1>, fg, 256, 0, st, a, per, lanes);
  else
    e = v4 ? launch_dependent(walk_fix<__nv_bfloat16, 4>, fg, 256, 0, st, a, per, lanes)
           : launch_dependent(walk_fix<__nv_bfloat16, 1>, fg, 256, 0, st, a, per, lanes);
  if (e != cudaSuccess) return set_error(CXG_ECUDA, "cxg_spmm_csr: %s", cudaGetErrorString(e));
  count_launches(3);
  return check_launch("cxg_spmm_csr (walk)");
}

}  // namespace cxg
