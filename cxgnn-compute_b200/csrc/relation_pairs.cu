// The distinct (relation, source) pairs of a graph's edges, for the relational layer that transforms each of them once.
//
// A pair is a bit: one row of words per relation over the sources. Marking the bits, counting them per word and adding the
// counts up gives every pair its position, in order of relation and source, with every relation's positions padded to
// whole blocks of 128 (what the typed matmul takes); the position of an edge is then a bit count away, so there is no table
// of num_rel * n_src entries and no sort. Six launches with one read-back between them (the number of positions), where
// some twenty torch operators over num_rel * n_src entries with two synchronisations took 0.6 ms however small the graph
// was. A graph is met once in sampled training, so this is part of every step there.
#include "common.cuh"

namespace cxg {
namespace {

constexpr int kThreads = 256;
constexpr int kBlockWords = kThreads;  // words of one relation per block: 8,192 sources
constexpr int kScanThreads = 1024;

struct PairArgs {
  const void *idx;
  const void *rel;
  int idx_bytes, rel_bytes;
  int64_t nnz, n_src;
  int num_rel;
  int words, blocks;    // per relation
  uint32_t *bits;       // [num_rel][words]
  int32_t *before;      // [num_rel][words] pairs in front of a word, inside its block
  int32_t *src_before;  // [words] the same over all relations
  int32_t *sum;         // [num_rel][blocks] pairs of a block, then the position of its first one
  int32_t *src_sum;     // [blocks] the same over all relations, without padding
  int32_t *rel_first;   // [num_rel + 1] first position of a relation
  int32_t *rel_end;     // [num_rel] behind its last pair
  int64_t *sizes;       // positions, pairs, edges outside the ranges
};

__device__ __forceinline__ int64_t load_id(const void *p, int64_t i, int bytes) {
  return bytes == 8 ? static_cast<const int64_t *>(p)[i] : static_cast<const int32_t *>(p)[i];
}

__global__ void __launch_bounds__(kThreads) mark_pairs(PairArgs a) {
  for (int64_t e = blockIdx.x * static_cast<int64_t>(kThreads) + threadIdx.x; e < a.nnz; e += static_cast<int64_t>(gridDim.x) * kThreads) {
    const int64_t r = load_id(a.rel, e, a.rel_bytes), s = load_id(a.idx, e, a.idx_bytes);
    if (r < 0 || r >= a.num_rel || s < 0 || s >= a.n_src) {
      a.sizes[2] = 1;
      continue;
    }
    uint32_t *word = a.bits + r * a.words + (s >> 5);
    const uint32_t bit = 1u << (s & 31);
    if ((__ldcg(word) & bit) == 0) atomicOr(word, bit);  // hub sources are asked for again and again
  }
}

// Exclusive prefix of v over the block; *total: the sum.
template <int THREADS>
__device__ __forceinline__ int block_prefix(int v, int *total) {
  __shared__ int warp_sum[THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  __syncthreads();  // the sums of the call before have been read
  if (lane == 31) warp_sum[warp] = inc;
  __syncthreads();
  int front = 0, all = 0;
  for (int w = 0; w < THREADS / 32; ++w) {
    if (w == warp) front = all;
    all += warp_sum[w];
  }
  *total = all;
  return front + inc - v;
}

// blockIdx.y: a relation, or num_rel for all of them together
__global__ void __launch_bounds__(kThreads) count_pairs(PairArgs a) {
  const int w = blockIdx.x * kBlockWords + threadIdx.x, r = blockIdx.y;
  int n = 0;
  if (w < a.words) {
    if (r < a.num_rel)
      n = __popc(a.bits[static_cast<int64_t>(r) * a.words + w]);
    else
      for (int q = 0; q < a.num_rel; ++q) n += __popc(a.bits[static_cast<int64_t>(q) * a.words + w]);
  }
  int total;
  const int front = block_prefix<kThreads>(n, &total);
  if (r < a.num_rel) {
    if (w < a.words) a.before[static_cast<int64_t>(r) * a.words + w] = front;
    if (threadIdx.x == 0) a.sum[static_cast<int64_t>(r) * a.blocks + blockIdx.x] = total;
  } else {
    if (w < a.words) a.src_before[w] = front;
    if (threadIdx.x == 0) a.src_sum[blockIdx.x] = total;
  }
}

// Exclusive prefix of get(0 .. n) in order, put(i, prefix); returns the sum. One block.
template <typename Get, typename Put>
__device__ __forceinline__ int scan_in_order(int n, Get get, Put put) {
  const int per = (n + kScanThreads - 1) / kScanThreads, lo = min(n, static_cast<int>(threadIdx.x) * per), hi = min(n, lo + per);
  int mine = 0, total;
  for (int i = lo; i < hi; ++i) mine += get(i);
  int at = block_prefix<kScanThreads>(mine, &total);
  for (int i = lo; i < hi; ++i) {
    const int v = get(i);
    put(i, at);
    at += v;
  }
  __syncthreads();  // what was put is read by other threads
  return total;
}

__global__ void __launch_bounds__(kScanThreads) place_pairs(PairArgs a) {
  // pairs in front of every block, relation by relation
  const int pairs = scan_in_order(a.num_rel * a.blocks, [&](int i) { return a.sum[i]; }, [&](int i, int at) { a.sum[i] = at; });
  auto first = [&](int r) { return r < a.num_rel ? a.sum[r * a.blocks] : pairs; };
  // first positions with every relation rounded up to 128
  const int positions = scan_in_order(a.num_rel, [&](int r) { return (first(r + 1) - first(r) + 127) / 128 * 128; },
                                      [&](int r, int at) { a.rel_first[r] = at; });
  for (int r = threadIdx.x; r < a.num_rel; r += kScanThreads) a.rel_end[r] = a.rel_first[r] + first(r + 1) - first(r);
  __syncthreads();
  // `first` reads what is replaced here, so a relation's first block comes last
  for (int i = threadIdx.x; i < a.num_rel * a.blocks; i += kScanThreads)
    if (i % a.blocks != 0) a.sum[i] += a.rel_first[i / a.blocks] - first(i / a.blocks);
  __syncthreads();
  for (int r = threadIdx.x; r < a.num_rel; r += kScanThreads) a.sum[r * a.blocks] = a.rel_first[r];
  scan_in_order(a.blocks, [&](int b) { return a.src_sum[b]; }, [&](int b, int at) { a.src_sum[b] = at; });
  if (threadIdx.x == 0) {
    a.rel_first[a.num_rel] = positions;
    a.sizes[0] = positions;
    a.sizes[1] = pairs;
  }
}

struct PairOut {
  int64_t *rel, *src, *pos;  // per position
  int64_t *src_ptr;          // [n_src + 1]
  int32_t *src_pos;          // positions of every source, by relation
  int32_t *edge_pos;         // [nnz]
};

// position of the pair (r, s)
__device__ __forceinline__ int place_of(const PairArgs &a, int64_t r, int64_t s) {
  const int64_t at = r * a.words + (s >> 5);
  const uint32_t below = a.bits[at] & ((1u << (s & 31)) - 1);
  return a.sum[r * a.blocks + (s >> 5) / kBlockWords] + a.before[at] + __popc(below);
}

// A thread per source: its pairs' positions, and where its list of them starts.
__global__ void __launch_bounds__(kThreads) number_pairs(PairArgs a, PairOut o) {
  const int64_t s = blockIdx.x * static_cast<int64_t>(kThreads) + threadIdx.x;
  const int w = static_cast<int>(s >> 5), lane = threadIdx.x & 31;
  if (w >= a.words) return;  // the whole warp
  int own = 0;
  for (int r = 0; r < a.num_rel; ++r) own += (a.bits[static_cast<int64_t>(r) * a.words + w] >> lane) & 1u;
  int inc = own;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += t;
  }
  int at = a.src_sum[w / kBlockWords] + a.src_before[w] + inc - own;
  if (s <= a.n_src) o.src_ptr[s] = at;
  if (s + 1 == a.n_src && lane == 31) o.src_ptr[a.n_src] = at + own;  // no thread of this warp's words stands behind it
  for (int r = 0; r < a.num_rel; ++r) {
    if (((a.bits[static_cast<int64_t>(r) * a.words + w] >> lane) & 1u) == 0) continue;
    const int p = place_of(a, r, s);
    o.rel[p] = r, o.src[p] = s, o.pos[p] = p;
    o.src_pos[at++] = p;
  }
}

__global__ void __launch_bounds__(kThreads) place_edges(PairArgs a, PairOut o) {
  const int64_t i0 = blockIdx.x * static_cast<int64_t>(kThreads) + threadIdx.x, step = static_cast<int64_t>(gridDim.x) * kThreads;
  for (int64_t e = i0; e < a.nnz; e += step)
    o.edge_pos[e] = place_of(a, load_id(a.rel, e, a.rel_bytes), load_id(a.idx, e, a.idx_bytes));
  for (int64_t i = i0; i < a.num_rel * 128ll; i += step) {  // the padding behind a relation's pairs
    const int r = static_cast<int>(i >> 7), p = a.rel_end[r] + static_cast<int>(i & 127);
    if (p < a.rel_first[r + 1]) o.rel[p] = r, o.src[p] = -1, o.pos[p] = p;
  }
}

size_t layout(PairArgs &a, char *ws) {
  a.words = static_cast<int>((a.n_src + 31) / 32);
  a.blocks = (a.words + kBlockWords - 1) / kBlockWords;
  size_t off = 0;
  auto take = [&](auto *&p, int64_t n) {
    p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(ws + off);
    off = align_up(off + static_cast<size_t>(n) * sizeof(*p), 256);
  };
  take(a.bits, static_cast<int64_t>(a.num_rel) * a.words);
  take(a.before, static_cast<int64_t>(a.num_rel) * a.words);
  take(a.src_before, a.words);
  take(a.sum, static_cast<int64_t>(a.num_rel) * a.blocks);
  take(a.src_sum, a.blocks);
  take(a.rel_first, a.num_rel + 1);
  take(a.rel_end, a.num_rel);
  return off;
}

unsigned edge_grid(int64_t n) {
  const int64_t blocks = (n + kThreads - 1) / kThreads;
  return static_cast<unsigned>(blocks < 1 ? 1 : blocks > kNumSM * 32 ? kNumSM * 32 : blocks);
}

int prepare(PairArgs &a, const void *idx, int idx_bytes, const void *rel, int rel_bytes, int64_t nnz, int64_t n_src, int num_rel,
            void *workspace, size_t workspace_bytes, const char *who) {
  CXG_REQUIRE(nnz >= 0 && n_src > 0 && num_rel > 0, CXG_EINVAL, "%s: bad sizes", who);
  CXG_REQUIRE((idx_bytes == 4 || idx_bytes == 8) && (rel_bytes == 4 || rel_bytes == 8), CXG_EINVAL, "%s: index widths must be 4 or 8", who);
  CXG_REQUIRE(num_rel <= 65534 && (n_src + 255) * num_rel < (1ll << 31), CXG_ELIMIT, "%s: num_rel * n_src must be below 2^31", who);
  CXG_REQUIRE((idx && rel) || nnz == 0, CXG_ENULL, "%s: NULL argument", who);
  a.idx = idx, a.rel = rel, a.idx_bytes = idx_bytes, a.rel_bytes = rel_bytes;
  a.nnz = nnz, a.n_src = n_src, a.num_rel = num_rel;
  const size_t need = layout(a, static_cast<char *>(workspace));
  CXG_REQUIRE(workspace != nullptr && workspace_bytes >= need && reinterpret_cast<uintptr_t>(workspace) % 16 == 0, CXG_EWORKSPACE,
              "%s: workspace %zu bytes, need %zu", who, workspace_bytes, need);
  return CXG_OK;
}

}  // namespace
}  // namespace cxg

using namespace cxg;

extern "C" int cxg_relation_pairs_workspace_size(int64_t n_src, int num_rel, size_t *bytes) {
  CXG_REQUIRE(bytes != nullptr, CXG_ENULL, "cxg_relation_pairs_workspace_size: bytes is NULL");
  CXG_REQUIRE(n_src > 0 && num_rel > 0 && num_rel <= 65534 && (n_src + 255) * num_rel < (1ll << 31), CXG_ELIMIT,
              "cxg_relation_pairs_workspace_size: num_rel * n_src must be positive and below 2^31");
  PairArgs a;
  a.n_src = n_src, a.num_rel = num_rel;
  *bytes = layout(a, nullptr);
  return CXG_OK;
}

extern "C" int cxg_relation_pairs_count(const void *idx, int idx_bytes, const void *rel, int rel_bytes, int64_t nnz, int64_t n_src,
                                        int num_rel, int64_t *sizes, void *workspace, size_t workspace_bytes, void *stream) {
  PairArgs a;
  const int rc = prepare(a, idx, idx_bytes, rel, rel_bytes, nnz, n_src, num_rel, workspace, workspace_bytes, "cxg_relation_pairs_count");
  if (rc != CXG_OK) return rc;
  CXG_REQUIRE(sizes != nullptr, CXG_ENULL, "cxg_relation_pairs_count: sizes is NULL");
  a.sizes = sizes;
  cudaStream_t st = as_stream(stream);
  if (cudaMemsetAsync(a.bits, 0, static_cast<size_t>(num_rel) * a.words * sizeof(uint32_t), st) != cudaSuccess ||
      cudaMemsetAsync(sizes, 0, 3 * sizeof(int64_t), st) != cudaSuccess)
    return check_launch("cxg_relation_pairs_count: memset");
  mark_pairs<<<edge_grid(nnz), kThreads, 0, st>>>(a);
  count_pairs<<<dim3(static_cast<unsigned>(a.blocks), static_cast<unsigned>(num_rel + 1)), kThreads, 0, st>>>(a);
  place_pairs<<<1, kScanThreads, 0, st>>>(a);
  count_launches(3);
  return check_launch("cxg_relation_pairs_count");
}

extern "C" int cxg_relation_pairs_fill(const void *idx, int idx_bytes, const void *rel, int rel_bytes, int64_t nnz, int64_t n_src,
                                       int num_rel, int64_t *pos_rel, int64_t *pos_src, int64_t *pos, int64_t *src_ptr,
                                       int32_t *src_pos, int32_t *edge_pos, void *workspace, size_t workspace_bytes, void *stream) {
  PairArgs a;
  const int rc = prepare(a, idx, idx_bytes, rel, rel_bytes, nnz, n_src, num_rel, workspace, workspace_bytes, "cxg_relation_pairs_fill");
  if (rc != CXG_OK) return rc;
  CXG_REQUIRE(src_ptr && (nnz == 0 || (pos_rel && pos_src && pos && src_pos && edge_pos)), CXG_ENULL,
              "cxg_relation_pairs_fill: NULL argument");
  const PairOut o{pos_rel, pos_src, pos, src_ptr, src_pos, edge_pos};
  cudaStream_t st = as_stream(stream);
  number_pairs<<<static_cast<unsigned>((a.words * 32ll + kThreads - 1) / kThreads), kThreads, 0, st>>>(a, o);
  place_edges<<<edge_grid(nnz > num_rel * 128ll ? nnz : num_rel * 128ll), kThreads, 0, st>>>(a, o);
  count_launches(2);
  return check_launch("cxg_relation_pairs_fill");
}
