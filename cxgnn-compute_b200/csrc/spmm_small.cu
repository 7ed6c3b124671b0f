// cxg_spmm_csr on small graphs as ONE launch: y[r,:] = red_{e in row r} v[e] * x[s(e),:] by clusters of thread blocks.
//
// The tiled walk takes three dependent launches (plan, walk, fix-up), each of which waits for the one in front and for its own
// code to arrive; with a few thousand edges that is all the time there is. Here the rows are dealt to clusters of kCtas blocks,
// by edges but in whole rows, and nothing leaves a cluster: every block looks up the cluster's rows in ptr (two rounds of one
// probe per thread), fetches their row pointers into shared memory, and its groups of lanes walk the tiles of kTile edges that
// the walk would have, but only the pieces of rows that start in a window of a tile each, so that what a group walks is as
// short as the rows allow. Pieces of rows that tiles cut go to the workspace, and behind the cluster's
// barrier the group in whose tile such a row begins adds them in tile order, chains of more than 64 in blocks of 64 first: the
// same sums, bit for bit, as those of plan, walk and fix-up where those do not keep rows whole.
//
// What bounds it: a chain of round trips to L2 (two probes, row pointers, ids, rows, per step of 8 or 16 edges, pieces) and the
// barrier. The code at a row's end exists once, not once per edge of a step as in the tiled walk: it has to arrive, too. Measured,
// three launches as they were -> one: 11,000 edges, 64 fp32 mean 20.5 -> 9.4 us, 47 columns 25.3 -> 9.5; 27,000, 128 fp32 18.8 -> 12.7,
// 256 bf16 21.0 -> 17.4; 56,000, 64 fp32 23.0 -> 16.4; 74,000, 31 fp32 27.1 -> 21.0, 64 bf16 25.1 -> 18.9.
#include <cooperative_groups.h>

#include <algorithm>

#include "spmm_walk_impl.cuh"

namespace cg = cooperative_groups;

namespace cxg {
namespace {

using walk::Acc;
using walk::kFar;
using walk::Words;

constexpr int kCtas = 8;
constexpr int kSmallThreads = 512;
constexpr int kWarps = kSmallThreads / 32;
constexpr int kTile = 64;         // edges per tile: that of walk_tile_of_waves for few edges
constexpr int kPitch = kTile;     // ids that a group stages: its pieces lie in one tile
constexpr int kSliceRows = 2560;  // row pointers that are kept in shared memory
constexpr int kClusters = 14;     // at most: what fits on the chip at once (of 16 two waited for the others: 12.5 -> 20 us)
constexpr int kRowsPerCluster = 2048;  // so that their pointers fit (200 rows of 400 edges and 28,000 of none: they may not)
static_assert(kClusters * kRowsPerCluster < kSmallThreads * (kSmallThreads - 1), "two rounds of probes find a row");

template <typename T, int VB, int G, int NV>
__global__ void __cluster_dims__(kCtas, 1, 1) __launch_bounds__(kSmallThreads) walk_small(const __grid_constant__ WalkArgs a, int clusters) {
  using A = Acc<T, VB>;
  constexpr int EL = A::EL, NG = 32 / G, kGroups = kCtas * kWarps * NG;
  constexpr int U = NV == 1 && EL <= 4 ? 16 : 8;  // edges in flight per lane
  __shared__ uint32_t slice[kSliceRows + 1];
  __shared__ __align__(16) uint32_t id_stage[kWarps][NG * kPitch];
  __shared__ __align__(16) float val_stage[kWarps][NG * kPitch];
  cg::cluster_group cluster = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, lg = lane & (G - 1), warp = tid >> 5;
  const int rank = static_cast<int>(cluster.block_rank()), me = static_cast<int>(blockIdx.x) / kCtas;
  const int n = static_cast<int>(a.n_dst), rb = a.row_bytes;
  auto ptr_at = [&](int r) { return walk::load_ptr_low(a.ptr, r, a.ptr_bytes); };
  dependency_wait();

  // rows [r_lo, r_hi) of this cluster: those whose first edge lies in its share of the edges
  const int64_t last = load_ptr(a.ptr, a.n_dst, a.ptr_bytes);
  const uint32_t e_total = static_cast<uint32_t>(min(last, a.nnz));
  if (blockIdx.x == 0 && tid < 64) a.hdr[tid] = (tid == kSHdrError && last > a.nnz) ? kSErrEdgeCount : 0;
  int r_lo = 0, r_hi = n;
  if (clusters > 1) {
    const uint32_t t_lo = static_cast<uint32_t>(static_cast<uint64_t>(e_total) * me / clusters);
    const uint32_t t_hi = static_cast<uint32_t>(static_cast<uint64_t>(e_total) * (me + 1) / clusters);
    const int stride = n / kSmallThreads + 1;
    const bool on = tid * stride <= n;
    const uint32_t probe = on ? ptr_at(tid * stride) : 0u;
    const int c_lo = __syncthreads_count(on && probe < t_lo), c_hi = __syncthreads_count(on && probe < t_hi);
    // behind probe c - 1, which is below the target, and up to probe c, which is not
    const int at_lo = max(c_lo - 1, 0) * stride + 1 + tid, at_hi = max(c_hi - 1, 0) * stride + 1 + tid;
    const bool in_lo = tid < stride - 1 && at_lo <= n, in_hi = tid < stride - 1 && at_hi <= n;
    const uint32_t v_lo = in_lo ? ptr_at(at_lo) : 0u, v_hi = in_hi ? ptr_at(at_hi) : 0u;
    const int m_lo = __syncthreads_count(in_lo && v_lo < t_lo), m_hi = __syncthreads_count(in_hi && v_hi < t_hi);
    if (me > 0) r_lo = c_lo == 0 ? 0 : (c_lo - 1) * stride + 1 + m_lo;
    if (me < clusters - 1) r_hi = c_hi == 0 ? 0 : (c_hi - 1) * stride + 1 + m_hi;
  }
  const int rows = r_hi - r_lo;
  const bool kept = rows <= kSliceRows;
  if (kept)
    for (int i = tid; i <= rows; i += kSmallThreads) slice[i] = ptr_at(r_lo + i);
  __syncthreads();
  auto start_of = [&](int i) { return kept ? slice[i] : ptr_at(r_lo + i); };  // first edge of the cluster's i-th row
  const uint32_t e0 = min(start_of(0), e_total), e1 = min(start_of(rows), e_total);
  const int first_tile = static_cast<int>(e0 / kTile), tiles = e1 > e0 ? static_cast<int>((e1 - 1) / kTile) - first_tile + 1 : 0;
  const int gid = (warp * NG + lane / G) * kCtas + rank;  // neighbouring windows in different blocks
  // the row that holds edge e, which lies in row `least` or behind it
  auto row_of = [&](uint32_t e, int least) {
    int lo = least + 1, hi = rows;  // the first row that starts behind e
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (start_of(mid) > e)
        hi = mid;
      else
        lo = mid + 1;
    }
    return lo - 1;
  };

  auto on = [&](int q) { return (lg + q * G) * VB < rb; };
  const uint8_t *xq[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) xq[q] = static_cast<const uint8_t *>(a.x) + (on(q) ? (lg + q * G) * VB : (rb - 1) / VB * VB);
  auto store = [&](int i, const float (&f)[NV][EL]) {
    uint8_t *dst = static_cast<uint8_t *>(a.y) + static_cast<uint64_t>(r_lo + i) * static_cast<uint32_t>(rb) + lg * VB;
#pragma unroll
    for (int q = 0; q < NV; ++q)
      if (on(q)) walk::store_row_bytes<T, VB>(dst + q * G * VB, f[q]);
  };
  auto zero_row = [&](int i) {
    const float z[NV][EL] = {};
    store(i, z);
  };
  auto finish = [&](int i, float (&f)[NV][EL], uint32_t edges) {
    if (a.reduce == CXG_MEAN)
#pragma unroll
      for (int q = 0; q < NV; ++q) walk::divide_by_count<EL>(f[q], static_cast<float>(edges));
    store(i, f);
  };
  // a piece: of the row that runs into the tile (part 0), of the one that runs out of it (part 1)
  auto piece_at = [&](int t, int part) { return a.partials + (static_cast<int64_t>(t) * 2 + part) * a.part_stride + lg * EL; };
  auto put_piece = [&](float *p, const float (&f)[NV][EL]) {
#pragma unroll
    for (int q = 0; q < NV; ++q)
      if (on(q)) {
#pragma unroll
        for (int i = 0; i < EL; ++i) p[q * G * EL + i] = f[q][i];
      }
  };

  for (int i = gid; i < rows && start_of(i + 1) <= e0; i += kGroups) zero_row(i);  // rows without edges in front

  // windows of 8 to kTile edges, as many as there are groups if that is enough
  int window = 8;
  while (window < kTile && static_cast<int64_t>(kGroups) * window < e1 - e0 + kTile) window *= 2;
  const int first_window = static_cast<int>(e0 / window), windows = e1 > e0 ? static_cast<int>((e1 - 1) / window) - first_window + 1 : 0;
  for (int i0 = 0; i0 < windows; i0 += kGroups) {
    // the pieces (a tile's part of a row) that start in the group's window
    const uint32_t w = first_window + i0 + gid, w_begin = max(e0, w * window), w_end = min(e1, (w + 1) * window);
    const int t = static_cast<int>(w * window / kTile);
    uint32_t begin = w_begin;
    int row = 0, len = 0;
    if (w_begin < w_end) {
      row = row_of(w_begin, 0);
      if (start_of(row) != w_begin && w_begin != max(e0, static_cast<uint32_t>(t) * kTile)) {  // runs in from an earlier window
        begin = start_of(++row);
        while (row < rows && start_of(row + 1) == begin) ++row;
      }
      if (begin < w_end)
        len = static_cast<int>(min(start_of(row_of(w_end - 1, row) + 1), min(e1, static_cast<uint32_t>(t + 1) * kTile)) - begin);
    }
    uint32_t *ids = id_stage[warp] + lane / G * kPitch;
    float *vals = val_stage[warp] + lane / G * kPitch;
    __syncwarp();
    {
      uint32_t id[kPitch / G];
      float val[kPitch / G];
#pragma unroll
      for (int j = 0; j < kPitch / G; ++j) {
        const int pos = j * G + lg;
        id[j] = 0u, val[j] = 1.f;  // times one is exact
        if (pos < len) {
          const uint32_t e = begin + pos;
          id[j] = walk::load_id_low(static_cast<const uint8_t *>(a.idx) + static_cast<uint64_t>(e) * static_cast<uint32_t>(a.idx_bytes));
          if (a.edge_val != nullptr) val[j] = __ldg(a.edge_val + e);
        }
      }
#pragma unroll
      for (int j = 0; j < kPitch / G; ++j) ids[j * G + lg] = id[j], vals[j * G + lg] = val[j];
    }
    A acc[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) acc[q].zero();
    int rend = kFar, rstart = 0, stop = kFar;
    if (len > 0) {
      rstart = start_of(row) < begin ? -1 : 0;
      rend = static_cast<int>(start_of(row + 1) - begin);
      stop = min(rend, len);
    }
    __syncwarp();
    const int longest = G == 32 ? len : __reduce_max_sync(0xffffffffu, len);
#pragma unroll 1
    for (int p = 0; p < longest; p += U) {
      Words<(VB + 3) / 4> v[U][NV];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint64_t off = static_cast<uint64_t>(ids[p + u]) * static_cast<uint32_t>(rb);
#pragma unroll
        for (int q = 0; q < NV; ++q) walk::load_row_bytes<VB>(v[u][q], xq[q] + off);
      }
      float weights[U];
#pragma unroll
      for (int u = 0; u < U; ++u) weights[u] = vals[p + u];
      // the edges of one row after another
      int q0 = 0;
#pragma unroll 1
      while (q0 < U && p + q0 < len) {
        const int q1 = min(stop - p, U);
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (u >= q0 && u < q1) {
            const float weight = weights[u];
#pragma unroll
            for (int q = 0; q < NV; ++q) acc[q].fma(v[u][q], weight);
          }
        q0 = q1;
        const int pos = p + q1;
        if (pos != stop) break;
        const bool row_done = pos == rend;
        float f[NV][EL];
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          acc[q].get(f[q]);
          acc[q].zero();
        }
        if (row_done && rstart >= 0)
          finish(row, f, static_cast<uint32_t>(rend - rstart));
        else
          put_piece(piece_at(t, rstart < 0 ? 0 : 1), f);
        if (row_done) {
          rstart = pos;
          for (;;) {
            ++row;
            rend = row < rows ? static_cast<int>(start_of(row + 1) - begin) : kFar;
            if (rend != pos) break;
            zero_row(row);
          }
        }
        stop = min(rend, len);
      }
    }
  }

  // Chains of pieces: element 0 is part 1 of the tile that the row begins in, element k part 0 of the k-th tile behind it.
  auto add_up = [&](int ts, int k0, int count, int step, float (&f)[NV][EL]) {
    constexpr int kDeep = EL * NV <= 4 ? 8 : EL * NV <= 8 ? 4 : 2;  // pieces asked for at once
#pragma unroll
    for (int q = 0; q < NV; ++q)
#pragma unroll
      for (int i = 0; i < EL; ++i) f[q][i] = on(q) ? __ldcg(piece_at(ts + k0, k0 == 0 ? 1 : 0) + q * G * EL + i) : 0.f;
#pragma unroll 1
    for (int k = 1; k < count; k += kDeep) {
      float piece[kDeep][NV][EL];
#pragma unroll
      for (int u = 0; u < kDeep; ++u) {
        const float *p = piece_at(ts + k0 + min(k + u, count - 1) * step, 0);
#pragma unroll
        for (int q = 0; q < NV; ++q)
#pragma unroll
          for (int i = 0; i < EL; ++i) piece[u][q][i] = on(q) ? __ldcg(p + q * G * EL + i) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < kDeep; ++u)
        if (k + u < count)
#pragma unroll
          for (int q = 0; q < NV; ++q)
#pragma unroll
            for (int i = 0; i < EL; ++i) f[q][i] += piece[u][q][i];
    }
  };
  cluster.sync();
  const bool long_chains = e1 - e0 > kWalkSeqPartials * kTile;
#pragma unroll 1
  for (int phase = long_chains ? 0 : 1; phase < 2; ++phase) {
#pragma unroll 1
    for (int i = gid; i < tiles; i += kGroups) {
      const int t = first_tile + i;
      const uint32_t begin = max(e0, static_cast<uint32_t>(t) * kTile), end = min(e1, static_cast<uint32_t>(t + 1) * kTile);
      // phase 0: blocks of 64 elements, by the tile of their first one; phase 1: rows that begin here and go on
#pragma unroll 1
      for (int part = phase; part < 2; ++part) {
        const int row = row_of(part == 0 ? begin : end - 1, 0);
        const uint32_t from = start_of(row), to = min(start_of(row + 1), e1);
        if (part == 0 ? from >= begin : to <= end || from < begin) continue;
        const int ts = static_cast<int>(from / kTile), count = static_cast<int>((to - 1) / kTile) - ts + 1, k = t - ts;
        float f[NV][EL];
        if (phase == 0) {
          if (count <= kWalkSeqPartials || k % kWalkSeqPartials != 0) continue;
          add_up(ts, k, min(kWalkSeqPartials, count - k), 1, f);
          put_piece(piece_at(t, part), f);
        } else {
          const int blocks = (count + kWalkSeqPartials - 1) / kWalkSeqPartials;
          add_up(ts, 0, blocks > 1 ? blocks : count, blocks > 1 ? kWalkSeqPartials : 1, f);
          finish(row, f, to - from);
        }
      }
    }
    if (phase == 0) cluster.sync();
  }
}

template <typename T, int VB>
bool launch_small(const WalkArgs &a, cudaStream_t st) {
  const int vectors = (a.row_bytes + VB - 1) / VB;
  auto go = [&](auto kernel, int g) {
    const int64_t groups = kCtas * kWarps * (32 / g);
    int64_t clusters = (a.nnz + 8 * groups - 1) / (8 * groups);
    clusters = std::max(clusters, (a.n_dst + kRowsPerCluster - 1) / kRowsPerCluster);
    clusters = clusters < 1 ? 1 : clusters > kClusters ? kClusters : clusters;
    return launch_dependent(kernel, static_cast<unsigned>(clusters * kCtas), kSmallThreads, 0, st, a, static_cast<int>(clusters)) == cudaSuccess;
  };
  if (vectors <= 8) return go(walk_small<T, VB, 8, 1>, 8);
  if (vectors <= 16) return go(walk_small<T, VB, 16, 1>, 16);
  if (vectors <= 32) return go(walk_small<T, VB, 32, 1>, 32);
  if (vectors <= 64) return go(walk_small<T, VB, 32, 2>, 32);
  if constexpr (VB < 16)
    if (vectors <= 128) return go(walk_small<T, VB, 32, 4>, 32);
  return false;
}

}  // namespace

bool small_launch(const WalkArgs &a, int dtype, int vb, cudaStream_t st) {
  while (vb > 4 && (a.row_bytes + vb - 1) / vb <= 8) vb /= 2;  // groups of four to a warp wait for each other's row ends
  if (dtype == CXG_F32) return vb == 16 ? launch_small<float, 16>(a, st) : vb == 8 ? launch_small<float, 8>(a, st) : launch_small<float, 4>(a, st);
  if (vb == 16 && a.row_bytes <= 512) vb = 8;  // eight columns per lane are too much work at a row's end: 22 us instead of 14
  return vb == 16  ? launch_small<__nv_bfloat16, 16>(a, st)
         : vb == 8 ? launch_small<__nv_bfloat16, 8>(a, st)
         : vb == 4 ? launch_small<__nv_bfloat16, 4>(a, st)
                   : launch_small<__nv_bfloat16, 2>(a, st);
}

int small_most_rows() { return kClusters * kRowsPerCluster; }

}  // namespace cxg
