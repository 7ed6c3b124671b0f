// A whole mini-batch of layer-wise neighbour sampling without a host synchronisation between its hops.
//
// The draw is the one of cxg_sample_neighbors (sampler.cu): Floyd's subset algorithm over the positions of a node's CSR
// row with counter-based numbers from (seed, node), positions ascending. What differs is who waits for whom. Hop by hop
// from the host, every hop reads two counts back, sorts the ids it saw first (eight radix passes) and issues about 35
// launches: 0.9 ms for 1024 seeds and fanouts 15 / 10 / 5, almost all of it the host. Here the counts stay on the device,
// the grids are sized for the most a hop can reach, and new ids are numbered in ascending order from a bitmap over the
// nodes (mark, count, prefix) instead of a sort: four launches a hop.
//
//   count_front     sampled neighbours of every block of frontier nodes (and: neighbour ids of the hop before -> batch ids)
//   draw_front      block offsets by adding the blocks in front, row pointers, the draw; marks ids without a batch id
//   count_marks     new ids per block of the bitmap
//   number_marks    their batch ids in ascending order; clears the bitmap
//
// A group of lanes draws for one node: lane k holds draw k, the draws are settled in order (a draw that repeats an earlier
// one takes the position floor(k) instead), ranked by comparison and fetched side by side, where one thread per node ran
// 15 dependent insertions and loads.
//
// Small batches are a chain of launches and of loads that wait for one another, so the kernels' blocks become resident while
// the one in front drains, and small frontiers are spread over blocks of one node per group. 32 seeds, fanouts 15 / 10 / 5,
// 245 K nodes: the three draws 33 -> 18 us, inference of the sampled SAGE batch 292 -> 244 us. (A training step of 1,024 seeds
// and 2.4 M nodes, 1.25 to 1.4 ms, is bound by host work behind the batch, which varies by more than sampling gained.)
#include "common.cuh"

namespace cxg {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxFanout = 64;
constexpr int kMaxHops = 16;
constexpr int kMarkWords = 1024;  // bitmap words per block

__device__ __forceinline__ uint64_t splitmix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ int64_t bounded(uint64_t h, int64_t bound) {
  return static_cast<int64_t>(((h >> 32) * static_cast<uint64_t>(bound)) >> 32);
}

struct BatchArgs {
  const void *gptr;
  const void *gidx;
  int ptr_bytes, idx_bytes;
  int64_t n_nodes, n_words;
  int64_t *local_of;   // [n_nodes], -1 outside the batch
  uint32_t *bitmap;    // [n_words], zero at rest
  int64_t *nodes;      // batch id -> node
  int64_t *row_ptr;    // [rows + 1]
  int64_t *edges;      // neighbours, first as nodes, then as batch ids
  int64_t *known;      // [hops + 1] nodes of the batch before hop 0, after hop 0, ...
  int64_t *n_edges;    // [hops + 1]
  int32_t *front_sum;  // per block of frontier nodes
  int32_t *mark_sum;   // per block of bitmap words
  int per_block;       // frontier nodes per block
};

// Sum of v[0 .. n) by the whole block (kThreads threads).
__device__ __forceinline__ int64_t block_total(const int32_t *v, int64_t n, int64_t *shared) {
  int64_t s = 0;
  for (int64_t i = threadIdx.x; i < n; i += kThreads) s += v[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) shared[threadIdx.x >> 5] = s;
  __syncthreads();
  s = 0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) s += shared[w];
  __syncthreads();
  return s;
}

__global__ void __launch_bounds__(kThreads) start_batch(BatchArgs a, const int64_t *seeds, int64_t n_seeds) {
  dependency_wait();
  const int64_t i = blockIdx.x * static_cast<int64_t>(kThreads) + threadIdx.x;
  if (i == 0) {
    a.known[0] = n_seeds;
    a.n_edges[0] = 0;
    a.row_ptr[0] = 0;
  }
  if (i < n_seeds) {
    int64_t v = seeds[i];
    if (v >= 0 && v < a.n_nodes)
      a.local_of[v] = i;
    else
      v = -1;  // a row without neighbours; forget_nodes reports it
    a.nodes[i] = v;
  }
}

// First edge and number of edges of a node.
__device__ __forceinline__ int64_t degree(const BatchArgs &a, int64_t v, int64_t *first) {
  if (v < 0) {
    *first = 0;
    return 0;
  }
  *first = load_ptr(a.gptr, v, a.ptr_bytes);
  return load_ptr(a.gptr, v + 1, a.ptr_bytes) - *first;
}

__device__ __forceinline__ void translate(const BatchArgs &a, int64_t from, int64_t to, int64_t tid, int64_t threads) {
  for (int64_t e = from + tid; e < to; e += threads) a.edges[e] = a.local_of[a.edges[e]];
}

// hop: frontier = nodes[known[hop - 1] .. known[hop])
__global__ void __launch_bounds__(kThreads) count_front(BatchArgs a, int hop, int fanout) {
  dependency_wait();
  __shared__ int32_t sum;
  if (hop > 0)
    translate(a, a.n_edges[hop - 1], a.n_edges[hop], blockIdx.x * static_cast<int64_t>(kThreads) + threadIdx.x,
              static_cast<int64_t>(gridDim.x) * kThreads);
  const int64_t f0 = hop > 0 ? a.known[hop - 1] : 0, f1 = a.known[hop];
  const int64_t b0 = f0 + static_cast<int64_t>(blockIdx.x) * a.per_block;
  if (threadIdx.x == 0) sum = 0;
  __syncthreads();
  int32_t mine = 0;
  for (int64_t i = b0 + threadIdx.x; i < min(f1, b0 + a.per_block); i += kThreads) {
    int64_t lo;
    const int64_t deg = degree(a, a.nodes[i], &lo);
    mine += static_cast<int32_t>(deg < fanout ? deg : fanout);
  }
  for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  if ((threadIdx.x & 31) == 0 && mine != 0) atomicAdd(&sum, mine);
  __syncthreads();
  if (threadIdx.x == 0) a.front_sum[blockIdx.x] = sum;
}

// Lanes that draw for one node.
int draw_lanes(int fanout) { return fanout <= 8 ? 8 : fanout <= 16 ? 16 : 32; }

// GS lanes per node, GS >= fanout (or 32 with two draws per lane)
template <int GS, typename IdxT>
__global__ void __launch_bounds__(kThreads) draw_front(BatchArgs a, int hop, int fanout, uint64_t seed) {
  dependency_wait();
  constexpr int PER = GS == 32 ? 2 : 1;  // draws per lane
  __shared__ int64_t shared[kThreads / 32];
  __shared__ int64_t carry;
  const int64_t f0 = hop > 0 ? a.known[hop - 1] : 0, f1 = a.known[hop];
  const int64_t b0 = f0 + static_cast<int64_t>(blockIdx.x) * a.per_block;
  const int64_t b1 = min(f1, b0 + a.per_block);
  const int64_t blocks = (f1 - f0 + a.per_block - 1) / a.per_block;
  if (blockIdx.x == 0 && blocks == 0 && threadIdx.x == 0) a.n_edges[hop + 1] = a.n_edges[hop];
  if (b0 >= f1) return;
  const int64_t base = a.n_edges[hop] + block_total(a.front_sum, blockIdx.x, shared);
  if (blockIdx.x == blocks - 1) {
    const int64_t last = a.front_sum[blockIdx.x];
    if (threadIdx.x == 0) a.n_edges[hop + 1] = base + last;
  }
  if (threadIdx.x == 0) carry = base;
  __syncthreads();
  // row pointers: prefix of the counts, kThreads nodes at a time
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t c0 = b0; c0 < b1; c0 += kThreads) {
    const int64_t i = c0 + threadIdx.x;
    int64_t c = 0;
    if (i < b1) {
      int64_t lo;
      const int64_t deg = degree(a, a.nodes[i], &lo);
      c = deg < fanout ? deg : fanout;
    }
    int64_t inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) shared[warp] = inc;
    __syncthreads();
    int64_t before = carry;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w)
      if (w < warp) before += shared[w];
    if (i < b1) a.row_ptr[i + 1] = before + inc;
    __syncthreads();
    if (threadIdx.x == kThreads - 1) carry = before + inc;
    __syncthreads();
  }
  // the draw
  const int lg = threadIdx.x & (GS - 1);
  const unsigned gmask = GS == 32 ? 0xffffffffu : (((1u << GS) - 1u) << (lane & ~(GS - 1)));
  const IdxT *gidx = static_cast<const IdxT *>(a.gidx);
  for (int64_t i = b0 + threadIdx.x / GS; i < b1; i += kThreads / GS) {
    const int64_t v = a.nodes[i];
    int64_t lo;
    const int64_t deg = degree(a, v, &lo);
    const int n = static_cast<int>(deg < fanout ? deg : fanout);
    const int64_t out = a.row_ptr[i + 1] - n;
    int64_t pick[PER];
    int rank[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) pick[j] = lg + j * GS, rank[j] = lg + j * GS;
    if (deg > fanout) {
      const uint64_t h = splitmix64(seed ^ (static_cast<uint64_t>(v) * 0xD1B54A32D192ED03ull));
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        const int k = lg + j * GS;
        pick[j] = k < fanout ? bounded(splitmix64(h + static_cast<uint64_t>(k)), deg - fanout + k + 1) : -1;
      }
      for (int k = 1; k < fanout; ++k) {  // draw k against the settled draws in front of it
        const int64_t t = __shfl_sync(gmask, PER == 2 && k >= GS ? pick[PER - 1] : pick[0], k & (GS - 1), GS);
        bool seen = false;
#pragma unroll
        for (int j = 0; j < PER; ++j) seen |= lg + j * GS < k && pick[j] == t;
        if ((__ballot_sync(gmask, seen) & gmask) != 0) {
#pragma unroll
          for (int j = 0; j < PER; ++j)
            if (lg + j * GS == k) pick[j] = deg - fanout + k;
        }
      }
#pragma unroll
      for (int j = 0; j < PER; ++j) rank[j] = 0;
      for (int k = 0; k < fanout; ++k) {
        const int64_t t = __shfl_sync(gmask, PER == 2 && k >= GS ? pick[PER - 1] : pick[0], k & (GS - 1), GS);
#pragma unroll
        for (int j = 0; j < PER; ++j) rank[j] += t < pick[j] ? 1 : 0;
      }
    }
#pragma unroll
    for (int j = 0; j < PER; ++j)
      if (lg + j * GS < n) {
        const int64_t u = static_cast<int64_t>(gidx[lo + pick[j]]);
        a.edges[out + rank[j]] = u;
        if (a.local_of[u] < 0) atomicOr(a.bitmap + (u >> 5), 1u << (u & 31));
      }
  }
}

__global__ void __launch_bounds__(kThreads) count_marks(BatchArgs a) {
  dependency_wait();
  __shared__ int32_t sum;
  if (threadIdx.x == 0) sum = 0;
  __syncthreads();
  int32_t mine = 0;
#pragma unroll
  for (int k = 0; k < kMarkWords / kThreads; ++k) {
    const int64_t w = blockIdx.x * static_cast<int64_t>(kMarkWords) + k * kThreads + threadIdx.x;
    if (w < a.n_words) mine += __popc(a.bitmap[w]);
  }
  for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  if ((threadIdx.x & 31) == 0 && mine != 0) atomicAdd(&sum, mine);
  __syncthreads();
  if (threadIdx.x == 0) a.mark_sum[blockIdx.x] = sum;
}

__global__ void __launch_bounds__(kThreads) number_marks(BatchArgs a, int hop) {
  dependency_wait();
  __shared__ int64_t shared[kThreads / 32];
  __shared__ int32_t warp_sum[kThreads / 32];
  const bool last = blockIdx.x == gridDim.x - 1;
  const int32_t here = a.mark_sum[blockIdx.x];
  if (here == 0 && !last) return;
  const int64_t base = a.known[hop] + block_total(a.mark_sum, blockIdx.x, shared);
  if (last && threadIdx.x == 0) a.known[hop + 1] = base + here;
  if (here == 0) return;
  // consecutive words per thread, so that ids ascend with the thread
  constexpr int PER = kMarkWords / kThreads;
  const int64_t w0 = blockIdx.x * static_cast<int64_t>(kMarkWords) + threadIdx.x * PER;
  uint32_t word[PER];
  int32_t mine = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    word[k] = w0 + k < a.n_words ? a.bitmap[w0 + k] : 0u;
    mine += __popc(word[k]);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int32_t inc = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) warp_sum[warp] = inc;
  __syncthreads();
  int64_t at = base + inc - mine;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w)
    if (w < warp) at += warp_sum[w];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    if (word[k] != 0) a.bitmap[w0 + k] = 0u;
    for (uint32_t left = word[k]; left != 0; left &= left - 1) {
      const int64_t v = (w0 + k) * 32 + (__ffs(left) - 1);
      a.nodes[at] = v;
      a.local_of[v] = at;
      ++at;
    }
  }
}

__global__ void __launch_bounds__(kThreads) finish_edges(BatchArgs a, int hops) {
  dependency_wait();
  translate(a, a.n_edges[hops - 1], a.n_edges[hops], blockIdx.x * static_cast<int64_t>(kThreads) + threadIdx.x,
            static_cast<int64_t>(gridDim.x) * kThreads);
}
__global__ void __launch_bounds__(kThreads) forget_nodes(BatchArgs a, int hops) {
  dependency_wait();
  const int64_t n = a.known[hops];
  for (int64_t i = blockIdx.x * static_cast<int64_t>(kThreads) + threadIdx.x; i < n; i += static_cast<int64_t>(gridDim.x) * kThreads) {
    const int64_t v = a.nodes[i];
    if (v >= 0)
      a.local_of[v] = -1;
    else
      a.known[0] = -1;  // a seed outside the graph
  }
}

struct BatchBounds {
  int64_t front[kMaxHops + 1];  // frontier nodes of each hop, at most
  int64_t nodes, rows, edges;
  size_t front_sum, mark_sum, total;
  int64_t words, mark_blocks;
};

int batch_bounds(int64_t n_seeds, const int *fanouts, int hops, int64_t n_nodes, int64_t nnz, BatchBounds *b) {
  if (hops < 1 || hops > kMaxHops) return CXG_EUNSUPPORTED;
  b->front[0] = n_seeds;
  b->nodes = n_seeds;
  b->rows = 0;
  b->edges = 0;
  int64_t widest = 0;
  for (int h = 0; h < hops; ++h) {
    if (fanouts[h] < 1 || fanouts[h] > kMaxFanout) return CXG_EUNSUPPORTED;
    int64_t e = b->front[h] * fanouts[h];
    // the nodes of a later frontier are distinct, so all of them have nnz edges at most; seeds may repeat
    if (h > 0 && e > nnz) e = nnz;
    b->edges += e;
    b->rows += b->front[h];
    int64_t fresh = e < n_nodes ? e : n_nodes;
    b->front[h + 1] = fresh;
    b->nodes += fresh;
    if (b->front[h] > widest) widest = b->front[h];
  }
  if (b->nodes > n_nodes + n_seeds) b->nodes = n_nodes + n_seeds;
  if (b->rows > b->nodes) b->rows = b->nodes;
  b->words = (n_nodes + 31) / 32;
  b->mark_blocks = (b->words + kMarkWords - 1) / kMarkWords;
  b->front_sum = 0;
  b->mark_sum = align_up(static_cast<size_t>(widest / 64 + 2050) * sizeof(int32_t), 256);
  b->total = b->mark_sum + align_up(static_cast<size_t>(b->mark_blocks + 1) * sizeof(int32_t), 256);
  return CXG_OK;
}

}  // namespace
}  // namespace cxg

using namespace cxg;

extern "C" int cxg_sample_batch_bounds(int64_t n_seeds, const int *fanouts, int hops, int64_t n_nodes, int64_t nnz,
                                       int64_t *max_nodes, int64_t *max_rows, int64_t *max_edges, size_t *workspace_bytes) {
  CXG_REQUIRE(n_seeds >= 0 && n_nodes >= 0 && nnz >= 0, CXG_EINVAL, "cxg_sample_batch_bounds: negative size");
  CXG_REQUIRE(fanouts && max_nodes && max_rows && max_edges && workspace_bytes, CXG_ENULL, "cxg_sample_batch_bounds: NULL argument");
  BatchBounds b;
  const int rc = batch_bounds(n_seeds, fanouts, hops, n_nodes, nnz, &b);
  CXG_REQUIRE(rc == CXG_OK, rc, "cxg_sample_batch_bounds: 1 to %d hops of fanout 1 to %d", kMaxHops, kMaxFanout);
  *max_nodes = b.nodes, *max_rows = b.rows, *max_edges = b.edges, *workspace_bytes = b.total;
  return CXG_OK;
}

extern "C" int cxg_sample_batch(const void *graph_ptr, const void *graph_idx, int ptr_bytes, int idx_bytes, int64_t n_nodes,
                                int64_t nnz, const int64_t *seeds, int64_t n_seeds, const int *fanouts, int hops,
                                const uint64_t *hop_seeds, int64_t *local_of, uint32_t *bitmap, int64_t *nodes,
                                int64_t *row_ptr, int64_t *edges, int64_t *sizes, void *workspace, size_t workspace_bytes,
                                void *stream) {
  CXG_REQUIRE(n_seeds > 0 && n_nodes > 0 && nnz >= 0, CXG_EINVAL, "cxg_sample_batch: bad sizes");
  CXG_REQUIRE((ptr_bytes == 4 || ptr_bytes == 8) && (idx_bytes == 4 || idx_bytes == 8), CXG_EINVAL,
              "cxg_sample_batch: index widths must be 4 or 8");
  CXG_REQUIRE(graph_ptr && (graph_idx || nnz == 0) && seeds && fanouts && hop_seeds && local_of && bitmap && nodes && row_ptr &&
                  edges && sizes && workspace,
              CXG_ENULL, "cxg_sample_batch: NULL argument");
  BatchBounds b;
  const int rc = batch_bounds(n_seeds, fanouts, hops, n_nodes, nnz, &b);
  CXG_REQUIRE(rc == CXG_OK, rc, "cxg_sample_batch: 1 to %d hops of fanout 1 to %d", kMaxHops, kMaxFanout);
  CXG_REQUIRE(workspace_bytes >= b.total, CXG_EWORKSPACE, "cxg_sample_batch: workspace %zu bytes, need %zu", workspace_bytes, b.total);
  BatchArgs a;
  a.gptr = graph_ptr, a.gidx = graph_idx, a.ptr_bytes = ptr_bytes, a.idx_bytes = idx_bytes;
  a.n_nodes = n_nodes, a.n_words = b.words;
  a.local_of = local_of, a.bitmap = bitmap, a.nodes = nodes, a.row_ptr = row_ptr, a.edges = edges;
  a.known = sizes, a.n_edges = sizes + hops + 1;
  a.front_sum = reinterpret_cast<int32_t *>(static_cast<char *>(workspace) + b.front_sum);
  a.mark_sum = reinterpret_cast<int32_t *>(static_cast<char *>(workspace) + b.mark_sum);
  cudaStream_t st = as_stream(stream);
  launch_dependent(start_batch, static_cast<unsigned>((n_seeds + kThreads - 1) / kThreads), kThreads, 0, st, a, seeds, n_seeds);
  for (int h = 0; h < hops; ++h) {
    // A node costs a group of lanes four loads that wait for one another (its id, its row, the neighbour, that one's batch
    // id), so small frontiers take one node per group; a block adds the sums of all blocks in front, so from 2,048 blocks
    // on they are larger, up to 64 nodes, and again from 4,096 on.
    const int f = fanouts[h];
    a.per_block = kThreads / draw_lanes(f);
    while (a.per_block < 64 ? b.front[h] / a.per_block > 2048 : b.front[h] / a.per_block > 4096) a.per_block *= 2;
    int64_t blocks = (b.front[h] + a.per_block - 1) / a.per_block;
    if (blocks < 1) blocks = 1;
    const unsigned grid = static_cast<unsigned>(blocks);
    launch_dependent(count_front, grid, kThreads, 0, st, a, h, f);
    auto draw = [&](auto kernel) { launch_dependent(kernel, grid, kThreads, 0, st, a, h, f, hop_seeds[h]); };
    switch (draw_lanes(f)) {
      case 8: idx_bytes == 8 ? draw(draw_front<8, int64_t>) : draw(draw_front<8, int32_t>); break;
      case 16: idx_bytes == 8 ? draw(draw_front<16, int64_t>) : draw(draw_front<16, int32_t>); break;
      default: idx_bytes == 8 ? draw(draw_front<32, int64_t>) : draw(draw_front<32, int32_t>);
    }
    const unsigned marks = static_cast<unsigned>(b.mark_blocks);
    launch_dependent(count_marks, marks, kThreads, 0, st, a);
    launch_dependent(number_marks, marks, kThreads, 0, st, a, h);
  }
  const int64_t last_edges = b.front[hops - 1] * fanouts[hops - 1];
  int64_t tail = (last_edges + kThreads - 1) / kThreads;
  tail = tail < 1 ? 1 : (tail > kNumSM * 8 ? kNumSM * 8 : tail);
  launch_dependent(finish_edges, static_cast<unsigned>(tail), kThreads, 0, st, a, hops);
  int64_t all = (b.nodes + kThreads - 1) / kThreads;
  all = all > kNumSM * 8 ? kNumSM * 8 : all;
  launch_dependent(forget_nodes, static_cast<unsigned>(all), kThreads, 0, st, a, hops);
  count_launches(4 * hops + 3);
  return check_launch("cxg_sample_batch");
}
