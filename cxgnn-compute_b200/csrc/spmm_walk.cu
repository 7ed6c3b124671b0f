// Plan, fix-up and dispatch of the register-staged tiled walk (spmm_walk_impl.cuh).
#include <type_traits>

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

// Bytes from a copied row to the next: whole lines, so that eight lanes' vectors lie in one.
int64_t copy_pitch(int64_t row_bytes) { return (row_bytes + 127) / 128 * 128; }

// e / tile
__device__ __forceinline__ int64_t tile_of(const WalkArgs &a, int64_t e) {
  const uint64_t v = static_cast<uint64_t>(e);
  return static_cast<int64_t>(a.tile_magic ? __umul64hi(v, a.tile_magic) : v / a.tile);
}

// One 16-byte vector of the copy per thread, zeros behind a row's end. Words of the source are 4-byte aligned, its rows are not
// always (bf16): a vector is put together from the words around it.
template <typename T>
__device__ __forceinline__ void copy_vector(const WalkArgs &a, int64_t i) {
  constexpr int kElem = static_cast<int>(sizeof(T));
  const int per_row = (a.row_bytes + 15) / 16;
  const int64_t row = i / per_row;
  const int at = static_cast<int>(i - row * per_row) * 16;
  const int n = min(16, a.row_bytes - at) / kElem;  // values of the row in the vector
  const T *src = reinterpret_cast<const T *>(static_cast<const uint8_t *>(a.x_rows) + row * a.row_bytes + at);
  union {
    uint4 v;
    uint32_t w[4];
    uint16_t h[8];
  } out;
  out.v = make_uint4(0, 0, 0, 0);
  if (kElem == 4) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < n) out.w[k] = __ldg(reinterpret_cast<const uint32_t *>(src) + k);
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < n) out.h[k] = __ldg(reinterpret_cast<const uint16_t *>(src) + k);
  }
  *reinterpret_cast<uint4 *>(static_cast<uint8_t *>(const_cast<void *>(a.x)) + row * a.x_pitch + at) = out.v;
}

constexpr int kFixThreads = 64;  // of walk_fix
constexpr int kCopyVectors = 4;  // vectors of the copy per thread

// Rows that own the first edge of a tile write the tile's record; a hub row that owns many is shared by its warp. One pass
// over ptr costs what reading ptr costs (1 us for 170,000 rows, 17 us for 14 M) and the time that its code takes to arrive;
// a search per tile is a chain of 18 dependent loads (10 us). It is launched while the kernel in front of it in the stream
// still runs, which saves 2 us. Also clears what the later kernels count in.
template <int kPlanRows, typename Copy>
__global__ void __launch_bounds__(256) walk_plan(const __grid_constant__ WalkArgs a) {
  dependency_wait();
  if constexpr (!std::is_void_v<Copy>) {
    if (blockIdx.x >= a.plan_blocks) {
      const int64_t i0 = static_cast<int64_t>(blockIdx.x - a.plan_blocks) * (256ll * kCopyVectors) + threadIdx.x;
#pragma unroll
      for (int k = 0; k < kCopyVectors; ++k)
        if (i0 + k * 256 < a.copy_vectors) copy_vector<Copy>(a, i0 + k * 256);
      return;
    }
  }
  const int64_t i0 = blockIdx.x * (256ll * kPlanRows) + threadIdx.x;
  int64_t raw_b[kPlanRows], raw_e[kPlanRows], raw_n[kPlanRows];  // of the row, its end, that of the row behind it
#pragma unroll
  for (int k = 0; k < kPlanRows; ++k) {
    const int64_t r = min(i0 + k * 256, a.n_dst - 1);
    raw_b[k] = load_ptr(a.ptr, r, a.ptr_bytes);
    raw_e[k] = load_ptr(a.ptr, r + 1, a.ptr_bytes);
    raw_n[k] = a.whole_rows ? load_ptr(a.ptr, min(r + 2, a.n_dst), a.ptr_bytes) : 0;
  }
  const int64_t last = load_ptr(a.ptr, a.n_dst, a.ptr_bytes);
  const int64_t e_total = min(last, a.nnz);
  if (i0 < 64) a.hdr[i0] = (i0 == kSHdrError && last > a.nnz) ? kSErrEdgeCount : 0;
#pragma unroll
  for (int k = 0; k < kPlanRows; ++k)
    if (i0 + k * 256 < a.max_tiles) a.count[i0 + k * 256] = 0;
  auto put = [&](int64_t t, int64_t row, int64_t begin, int64_t row_begin, int64_t row_end) {
    if (a.wide_tiles)
      static_cast<WideTile *>(a.tiles)[t] = WideTile{row, begin};
    else
      static_cast<WalkTile *>(a.tiles)[t] = WalkTile{static_cast<uint32_t>(row), static_cast<uint32_t>(begin),
                                                     static_cast<uint32_t>(row_begin), static_cast<uint32_t>(row_end)};
  };
  if (i0 == 0) put((e_total + a.tile - 1) / a.tile, a.n_dst, e_total, e_total, e_total);
  auto record = [&](int64_t t, int64_t r, int64_t b, int64_t e, int64_t n) {
    const int64_t pos = t * a.tile;
    if (a.whole_rows && pos != b) {
      const int64_t at = b + tile_of(a, pos - b + a.tile - 1) * a.tile;
      if (e - b > a.tile && at < e)
        put(t, r, at, b, e);
      else
        put(t, r + 1, e, e, n);
    } else {
      put(t, r, pos, b, e);
    }
  };
#pragma unroll
  for (int k = 0; k < kPlanRows; ++k) {
    const int64_t i = i0 + k * 256;
    const int64_t rb = min(raw_b[k], e_total), re = i < a.n_dst ? min(raw_e[k], e_total) : rb;
    const int64_t rn = min(raw_n[k], e_total);
    // tiles whose first edge lies in [rb, re)
    const int64_t t0 = tile_of(a, rb + a.tile - 1), t1 = re > rb ? tile_of(a, re + a.tile - 1) : t0;
    const bool many = t1 - t0 > 4;
    if (!many)
      for (int64_t t = t0; t < t1; ++t) record(t, i, rb, re, rn);
    for (unsigned left = __ballot_sync(0xffffffffu, many); left != 0; left &= left - 1) {
      const int src = __ffs(left) - 1;
      const int64_t r = __shfl_sync(0xffffffffu, i, src), b = __shfl_sync(0xffffffffu, rb, src),
                    e = __shfl_sync(0xffffffffu, re, src), n = __shfl_sync(0xffffffffu, rn, src), u0 = __shfl_sync(0xffffffffu, t0, src),
                    u1 = __shfl_sync(0xffffffffu, t1, src);
      for (int64_t t = u0 + (threadIdx.x & 31); t < u1; t += 32) record(t, r, b, e, n);
    }
  }
}

// Partial sums of the row's chain: element k > 0 is the head partial of tile ts + k, element 0 the tail partial of ts.
__device__ __forceinline__ float *chain_at(const WalkArgs &a, int64_t ts, int64_t k) {
  return a.partials + ((ts + k) * 2 + (k == 0 ? 1 : 0)) * a.part_stride;
}

template <typename T, int VW>
__device__ __forceinline__ void finish_columns(const WalkArgs &a, T *dst, int left, float (&s)[VW], int64_t deg) {
#pragma unroll
  for (int i = 0; i < VW; ++i) {
    if (i >= left) break;
    float r = s[i];
    if (a.reduce == CXG_MEAN) r = __fdiv_rn(r, static_cast<float>(deg));
    if (a.accumulate) r += to_f32(dst[i]);
    dst[i] = from_f32<T>(r);
  }
}

template <int VW>
__device__ __forceinline__ void load_partial(float (&v)[VW], const float *p) {
  if constexpr (VW == 4) {
    const float4 t = __ldcg(reinterpret_cast<const float4 *>(p));
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
  } else {
    v[0] = __ldcg(p);
  }
}

// Adds n elements of the chain, step elements apart, from element k0 on, in order; `lanes` lanes of VW columns each. The
// result goes to `into` (fp32 scratch) or, when that is null, to the output row.
template <typename T, int VW>
__device__ __forceinline__ void chain_sum(const WalkArgs &a, int64_t ts, int64_t k0, int n, int step, float *into, int64_t row, int64_t deg,
                          int lane, int lanes) {
  constexpr int kDepth = 8;  // partials requested at once (16 take a third of the resident warps and cost more than they save)
  for (int c = lane * VW; c < a.width; c += lanes * VW) {
    float s[VW];
    const int64_t stride = 2ll * step * a.part_stride;
    const float *p = a.partials + (ts + k0) * 2 * a.part_stride + c;
    load_partial(s, chain_at(a, ts, k0) + c);
    for (int k = 1; k < n; k += kDepth) {
      float v[kDepth][VW];
#pragma unroll
      for (int u = 0; u < kDepth; ++u) {
        p += stride;
        if (k + u < n) load_partial(v[u], p);
      }
#pragma unroll
      for (int u = 0; u < kDepth; ++u)
        if (k + u < n)
#pragma unroll
          for (int i = 0; i < VW; ++i) s[i] += v[u][i];
    }
    if (into != nullptr) {
      if constexpr (VW == 4)
        *reinterpret_cast<float4 *>(into + c) = make_float4(s[0], s[1], s[2], s[3]);
      else
        into[c] = s[0];
    } else {
      finish_columns<T, VW>(a, static_cast<T *>(a.y) + row * a.width + c, a.width - c, s, deg);
    }
  }
}

// Adds the partials of the rows that tiles cut. A tile leads the first block of the chain that starts in it, and block
// k / 64 of the chain that runs through its start when it is that chain's element k, a multiple of 64. The leader that
// finishes a long chain's last block adds the block sums.
// A chain is a handful of loads that depend on one another, so latency is what counts: a warp looks `per` tiles over at
// once, a lane for each of a tile's two roles, and then adds as many chains side by side as there are `lanes`-wide groups
// in it (one tile after the other, a warp each: 72 us for 74,500 tiles of rows of 64 columns, now 33 us; 182,000 tiles of 128: 152 us).
// Nearly every chain has two elements, which lie next to each other: those go first, kPairs per group in flight (2.3 M edges,
// F = 128: 16.6 us, 20.7 without). Partials lie whole vectors apart, whatever the width. Small blocks, so that the warp with the
// longest chain does not keep the places of others.
template <typename T, int VW>
__global__ void __launch_bounds__(kFixThreads, 12) walk_fix(const __grid_constant__ WalkArgs a, int per, int lanes) {
  constexpr int kPairs = 4;
  dependency_wait();
  const int lane = threadIdx.x & 31;
  const int64_t e_total = edge_total(a);
  const int64_t t = (blockIdx.x * static_cast<int64_t>(kFixThreads / 32) + (threadIdx.x >> 5)) * per + (lane & (per - 1));
  bool lead = false;
  int64_t row = 0, deg = 0;
  int ts = 0, k = 0, m = 0;
  const WalkTile here = load_tile(a, min(t, a.max_tiles - 1)), next = load_tile(a, min(t, a.max_tiles - 1) + 1);
  if (lane < 2 * per && t < a.max_tiles && t * a.tile < e_total) {  // behind the last tile, whose end is e_total, nothing is written
    const bool tail = lane < per;
    row = tail ? next.row : here.row;
    if (next.begin > here.begin && row < a.n_dst) {
      const int64_t rb = tail ? next.row_begin : here.row_begin, re = tail ? next.row_end : here.row_end;
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
  // group g takes the g-th of the chains that are left, and so on; -1: none
  auto take = [&](unsigned &left) {
    unsigned mine = left;
    for (int i = 0; i < group; ++i) mine &= mine - 1;
    for (int i = 0; i < groups; ++i) left &= left - 1;
    return mine != 0 ? __ffs(mine) - 1 : -1;
  };
  unsigned left = __ballot_sync(0xffffffffu, lead && m == 2);
  while (left != 0) {
    int64_t jrow[kPairs], jdeg[kPairs];
    int jts[kPairs];
#pragma unroll
    for (int j = 0; j < kPairs; ++j) {
      const int src = take(left);
      jts[j] = __shfl_sync(0xffffffffu, ts, src & 31);
      jrow[j] = __shfl_sync(0xffffffffu, row, src & 31);
      jdeg[j] = __shfl_sync(0xffffffffu, deg, src & 31);
      if (src < 0) jts[j] = -1;
    }
    for (int c = in_group * VW; c < a.width; c += lanes * VW) {
      float s[kPairs][VW], v[kPairs][VW];
#pragma unroll
      for (int j = 0; j < kPairs; ++j)
        if (jts[j] >= 0) {
          const float *p = chain_at(a, jts[j], 0) + c;  // element 1 lies a row further on
          load_partial(s[j], p);
          load_partial(v[j], p + a.part_stride);
        }
#pragma unroll
      for (int j = 0; j < kPairs; ++j)
        if (jts[j] >= 0) {
#pragma unroll
          for (int i = 0; i < VW; ++i) s[j][i] += v[j][i];
          finish_columns<T, VW>(a, static_cast<T *>(a.y) + jrow[j] * a.width + c, a.width - c, s[j], jdeg[j]);
        }
    }
  }
  left = __ballot_sync(0xffffffffu, lead && m != 2);
  while (left != 0) {
    const int got = take(left), src = got & 31;
    const int jts = __shfl_sync(0xffffffffu, ts, src), jk = __shfl_sync(0xffffffffu, k, src),
              jm = __shfl_sync(0xffffffffu, m, src);
    const int64_t jrow = __shfl_sync(0xffffffffu, row, src), jdeg = __shfl_sync(0xffffffffu, deg, src);
    if (got >= 0) {
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

// Most bytes of a copy of x, a limit of memory and not of speed: the copy comes on top of x and y, and a caller that is short
// of memory has its allocator give everything back before it hears that there is none. 111 M rows of 47 fp32 values (20.9 GB)
// would be copied to 28.4. (x as it is / copied: 15 M rows of 201 bf16 values, 199 M edges, 7.7 GB 19.9 / 13.0 ms; 20 M rows,
// 10.2 GB 21.1 / 15.3, the first of them beyond the limit; 60 M rows of 47 bf16, 7.7 GB 17.1 / 14.4.)
constexpr int64_t kMostCopyBytes = int64_t{8} << 30;

// Bytes that a lane reads of a row: narrow rows take the vector that occupies eight lanes, the fewest a tile is given.
int walk_vector_bytes(const cxg_spmm_desc *d) {
  const int64_t row_bytes = static_cast<int64_t>(d->feat) * d->heads * (d->dtype == CXG_F32 ? 4 : 2);
  int vb = vector_bytes(d);
  while (vb > 4 && row_bytes <= 4 * vb) vb /= 2;
  return vb;
}

// One launch of clusters instead of plan, walk and fix-up. For rows of 512 bytes the two meet at 65,000 edges (17.7 / 18.5 us; 74,000
// 22.5 / 17.5), narrower ones gain up to 98,000 and beyond; there a graph whose edges all lie in one row, which one cluster
// then walks alone, takes about as long as three launches do. Its tiles have 64 edges, which is what walk_tile_of_waves gives
// graphs of this size.
bool small_graph(const cxg_spmm_desc *d) {
  const int64_t row_bytes = static_cast<int64_t>(d->feat) * d->heads * (d->dtype == CXG_F32 ? 4 : 2);
  return d->nnz <= 98304 && d->nnz * row_bytes <= (32 << 20) && d->n_dst <= small_most_rows() && d->edge_rel == nullptr &&
         !(d->flags & (CXG_SPMM_ACCUMULATE | CXG_SPMM_SHARE_SMS)) && (d->heads == 1 || d->edge_val == nullptr);
}

bool dispatch(const cxg_spmm_desc *d, const WalkArgs &a, bool copied, cudaStream_t st, int *resident_tiles) {
  const int valmode = d->flags & CXG_SPMM_ACCUMULATE ? 4
                      : d->edge_val == nullptr       ? (d->reduce == CXG_MEAN ? 3 : 0)
                                                     : (d->heads == 1 ? 1 : 2);
  const bool share = (d->flags & CXG_SPMM_SHARE_SMS) != 0;
  if (copied)
    return d->dtype == CXG_F32 ? walk_launch_f32_copy(a, valmode, share, st, resident_tiles)
                               : walk_launch_bf16_copy(a, valmode, share, st, resident_tiles);
  const int vb = walk_vector_bytes(d);
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

int walk_layout(int64_t nnz, int64_t part_stride, int tile, WalkLayout *L) {
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
  off = align_up(off + static_cast<size_t>(max_tiles) * 2 * part_stride * sizeof(float), 256);
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
  // the walk counts rows, edges and tiles in 32 bits (and a round of tiles beyond)
  if (d->n_dst > INT32_MAX - (1 << 20) || d->nnz > INT32_MAX - (1 << 20)) return false;
  return row_bytes <= (vb == 16 ? 128 : 256) * vb;
}

void walk_plan_run(WalkArgs &a, cudaStream_t st) {
  a.tile_magic = a.tile > 1 && a.tile < 30000 ? ~0ull / static_cast<uint64_t>(a.tile) + 1 : 0;  // exact up to 2^34 edges
  // a row per thread while the chip holds a thread for each (a quarter of the code: 5.2 -> 2.8 us for 20,000 rows), then four
  const int64_t rows = a.n_dst > a.max_tiles ? a.n_dst : a.max_tiles;
  const int per_thread = rows <= kNumSM * 2048 ? 1 : 4;
  a.plan_blocks = static_cast<unsigned>((rows + 256 * per_thread - 1) / (256 * per_thread));
  const unsigned grid = a.plan_blocks + static_cast<unsigned>((a.copy_vectors + 256 * kCopyVectors - 1) / (256 * kCopyVectors));
  auto go = [&](auto kernel) { launch_dependent(kernel, grid, 256, 0, st, a); };
  if (a.copy_vectors == 0)
    per_thread == 1 ? go(walk_plan<1, void>) : go(walk_plan<4, void>);
  else if (a.row_bytes == a.width * 4)
    per_thread == 1 ? go(walk_plan<1, float>) : go(walk_plan<4, float>);
  else
    per_thread == 1 ? go(walk_plan<1, __nv_bfloat16>) : go(walk_plan<4, __nv_bfloat16>);
}

int walk_whole_waves(int64_t nnz, int64_t resident, int round) {
  if (nnz >= 2048 * resident) return 512;
  const int64_t waves = (nnz + 256 * resident - 1) / (256 * resident);
  const int64_t t = waves > 0 ? (nnz + waves * resident - 1) / (waves * resident) : 0;
  return t < 64 ? 64 : static_cast<int>((t + round - 1) / round * round);
}

int walk_tile_of_waves(int64_t nnz, int64_t resident) {
  // One wave of tiles of up to 256 edges where that is enough (2.3 M edges, F = 64: 71 us, two waves of 128 edges 78), behind
  // that whole waves of up to 128, which even out what the groups get through (1.2 M edges, F = 201 bf16: 270 us with two
  // waves of 136, 250 with three of 88; 12.6 M, F = 47: 296 with six of 224, 290 with eleven of 128). From four waves of 512
  // edges on the longer tile costs less (126 M edges: 10 % less than 128). At least 64 edges, so that small graphs do not become
  // all borders. Several waves take multiples of 16 edges, whole lines of 64-bit ids (12.8 M edges, F = 16: 128 158 us, 120 172;
  // 176 156, 232 161); in one wave they would leave groups without a tile (140,000 edges, F = 11: 80 35.1 us, 72 34.1).
  if (nnz >= 2048 * resident) return 512;
  const int64_t most = nnz <= 256 * resident ? 256 : 128;
  const int64_t waves = (nnz + most * resident - 1) / (most * resident);
  const int64_t t = waves > 0 ? (nnz + waves * resident - 1) / (waves * resident) : 0;
  const int64_t round = waves > 1 ? 16 : 8;
  return t < 64 ? 64 : static_cast<int>((t + round - 1) / round * round);
}

bool walk_weighted(const WalkArgs &a, int vb, cudaStream_t st, int *resident_tiles) {
  if (resident_tiles == nullptr && a.tile > kWeightedTile) return false;
  const int valmode = a.heads == 1 ? 1 : vb != 16 || a.heads > 8 ? 2 : a.heads == 2 ? 5 : a.heads == 4 ? 6 : 7;
  return vb == 16  ? walk_launch_f32_16(a, valmode, false, st, resident_tiles)
         : vb == 8 ? walk_launch_f32_8(a, valmode, false, st, resident_tiles)
                   : walk_launch_f32_4(a, valmode, false, st, resident_tiles);
}

int walk_tile_edges(const cxg_spmm_desc *d, bool copied) {
  if (d->split_edges > 0) return d->split_edges;
  WalkArgs a;
  a.row_bytes = d->feat * d->heads * (d->dtype == CXG_F32 ? 4 : 2);
  int resident = kNumSM * 32;
  dispatch(d, a, copied, nullptr, &resident);
  return walk_tile_of_waves(d->nnz, resident);
}

int walk_static_tile_edges(const cxg_spmm_desc *d) {
  if (d->split_edges > 0) return d->split_edges;
  WalkArgs a;
  a.row_bytes = d->feat * d->heads * (d->dtype == CXG_F32 ? 4 : 2);
  int resident = kNumSM * 32;
  dispatch(d, a, false, nullptr, &resident);
  return walk_whole_waves(d->nnz, resident, 32);
}

size_t walk_copy_bytes(const cxg_spmm_desc *d, int64_t n_src) {
  const int elem = d->dtype == CXG_F32 ? 4 : 2;
  const int64_t row_bytes = static_cast<int64_t>(d->feat) * d->heads * elem;
  const uint64_t bits = static_cast<uint64_t>(row_bytes) | reinterpret_cast<uintptr_t>(d->x);
  if (!walk_eligible(d) || (d->flags & CXG_SPMM_ACCUMULATE) || (d->heads > 1 && d->edge_val != nullptr)) return 0;
  if (n_src <= 0 || n_src > UINT32_MAX || row_bytes <= 64 || bits % (row_bytes <= 128 ? 8 : 16) == 0) return 0;
  // The copy costs a row's bytes twice per source, an edge gains what its loads cost: 245,000 sources, fp32, x as it is / copied
  // (us): F = 19 (one line) 67 / 56 at 5 edges per source; F = 47 85 / 98 at 5, 123 / 125 at 11, 175 / 163 at 21, 337 / 290 at
  // 51; F = 101 148 / 158, 209 / 195, 305 / 255. Odd numbers of bf16 values: F = 47 83 / 88 at 5, 120 / 102 at 11, 400 / 236 at
  // 51; F = 201 225 / 250, 337 / 260. Small graphs do not repay the work behind the plan: 220,000 edges of 94 bytes 38 / 42, of
  // 404 bytes 46 / 43.
  const int64_t edges = row_bytes <= 128 ? 5 : bits % 4 != 0 ? 8 : 12;
  if (d->nnz < edges * n_src || d->nnz * row_bytes < (40 << 20) || n_src * copy_pitch(row_bytes) > kMostCopyBytes) return 0;
  return static_cast<size_t>(n_src) * copy_pitch(row_bytes);
}

int walk_launch(const cxg_spmm_desc *d, bool whole_rows, int64_t n_src, void *rows, void *workspace, size_t workspace_bytes,
                cudaStream_t st) {
  const bool copied = rows != nullptr;
  const int tile = walk_tile_edges(d, copied);
  WalkArgs a;
  a.ptr = d->ptr, a.idx = d->idx, a.x = d->x, a.y = d->y;
  a.edge_val = d->edge_val, a.edge_rel = d->edge_rel;
  a.n_dst = d->n_dst, a.nnz = d->nnz, a.rel_stride = d->rel_stride;
  a.feat = d->feat, a.heads = d->heads, a.width = d->feat * d->heads;
  a.row_bytes = a.width * (d->dtype == CXG_F32 ? 4 : 2);
  a.x_pitch = a.row_bytes;
  a.x_rows = nullptr;
  a.copy_vectors = 0;
  if (copied) {
    a.x_rows = d->x, a.x = rows;
    a.x_pitch = static_cast<int>(copy_pitch(a.row_bytes));
    a.copy_vectors = n_src * ((a.row_bytes + 15) / 16);
  }
  a.ptr_bytes = d->ptr_bytes, a.idx_bytes = d->idx_bytes, a.reduce = d->reduce;
  a.accumulate = (d->flags & CXG_SPMM_ACCUMULATE) ? 1 : 0;
  a.tile = tile;
  a.whole_rows = whole_rows ? 1 : 0;
  a.wide_tiles = 0;
  WalkLayout L;
  a.part_stride = static_cast<int>(walk_part_stride(a.width));
  int rc = walk_layout(d->nnz, a.part_stride, tile, &L);
  if (rc == CXG_OK && workspace_bytes < L.total && !copied) {  // scratch of a fixed size
    a.part_stride = a.width;
    rc = walk_layout(d->nnz, a.part_stride, tile, &L);
  }
  if (rc != CXG_OK) return set_error(rc, "cxg_spmm_csr: graph too large for 32-bit tile ids");
  if (workspace == nullptr || workspace_bytes < L.total)
    return set_error(CXG_EWORKSPACE, "cxg_spmm_csr: workspace %zu bytes, need %zu", workspace_bytes, L.total);
  char *ws = reinterpret_cast<char *>(workspace);
  a.hdr = reinterpret_cast<int32_t *>(ws + L.hdr);
  a.tiles = ws + L.tiles;
  a.count = reinterpret_cast<int32_t *>(ws + L.count);
  a.partials = reinterpret_cast<float *>(ws + L.partials);
  a.max_tiles = L.max_tiles;
  if (small_graph(d) && tile == 64 && (d->split_edges == 0 || !whole_rows) && small_launch(a, d->dtype, walk_vector_bytes(d), st)) {
    count_launches(1);
    return check_launch("cxg_spmm_csr (small)");
  }
  walk_plan_run(a, st);
  if (!dispatch(d, a, copied, st, nullptr)) return set_error(CXG_EUNSUPPORTED, "cxg_spmm_csr: rows of %d bytes", a.row_bytes);
  // tiles a warp looks over: one while the chip holds a warp for each, up to sixteen (two roles on 32 lanes)
  int per = 1;
  while (per < 16 && L.max_tiles > static_cast<int64_t>(per) * kNumSM * 24) per *= 2;
  const int per_block = kFixThreads / 32 * per;
  const unsigned fg = static_cast<unsigned>((L.max_tiles + per_block - 1) / per_block);
  const bool v4 = a.part_stride % 4 == 0;
  int lanes = 1;  // per chain
  while (lanes < 32 && lanes * (v4 ? 4 : 1) < a.width) lanes *= 2;
  cudaError_t e;
  if (d->dtype == CXG_F32)
    e = v4 ? launch_dependent(walk_fix<float, 4>, fg, kFixThreads, 0, st, a, per, lanes)
           : launch_dependent(walk_fix<float, 1>, fg, kFixThreads, 0, st, a, per, lanes);
  else
    e = v4 ? launch_dependent(walk_fix<__nv_bfloat16, 4>, fg, kFixThreads, 0, st, a, per, lanes)
           : launch_dependent(walk_fix<__nv_bfloat16, 1>, fg, kFixThreads, 0, st, a, per, lanes);
  if (e != cudaSuccess) return set_error(CXG_ECUDA, "cxg_spmm_csr: %s", cudaGetErrorString(e));
  count_launches(3);
  return check_launch("cxg_spmm_csr (walk)");
}

}  // namespace cxg
