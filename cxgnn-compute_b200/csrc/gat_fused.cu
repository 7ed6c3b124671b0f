// Fused GAT aggregation for sm_100a: attention score, LeakyReLU, edge softmax and the weighted
// neighbour sum in ONE walk over the edges, forward and backward.
//
// The reference runs this as five kernels with three [E, H] round trips through memory
// (cxgnncomp/graph_conv.py:458-496: two score reductions, edge_softmax_fwd with its mask,
// src/cpp/src/edge_softmax.cu:3-42, then gen_fwd_sum_edge_value_multi_head,
// src/cpp/src/aggr_kernel.cu:155-186; backward: aggr_kernel.cu:443-491 and edge_softmax.cu:44-95).
// Here no per-edge value crosses a call:
//
//   forward   y[r,h,:] = sum_e p[e,h] x[s(e),h,:],  p = softmax over the edges of row r of
//             t[e,h] = leaky(a_dst[r,h] + a_src[s(e),h]).  The walk is the register-staged tiled one
//             of the SpMM (spmm_walk_impl.cuh: tiles of consecutive edges, a group of lanes per tile,
//             rows of any width); per (row, head) it keeps a running maximum m and a running
//             sum s and rescales the fp32 accumulator when the maximum grows (online softmax):
//                 m' = max(m, t);  acc = acc * exp(m - m') + exp(t - m') * x;  s likewise.
//             Outputs y, row_max = m and row_sum = s per (row, head): [N, H] each instead of [E, H].
//             Larger ones first turn the scores of a tile's edges into weights ([nnz, H] in the workspace, a tile in shared
//             memory at a time) and then run the SpMM's weighted walk over the same tiles: a lane that holds four columns
//             of a head then loads its weight instead of computing two exponentials per edge (gat_weights).
//             A row that crosses tile borders leaves (acc, m, s) partials per tile; a second kernel
//             merges them in tile order with the same rescaling. No atomics: results are the same on
//             every run.
//   backward  on the TRANSPOSED graph (row = source s, entries = destinations r), with
//             D[r,h] = <dy[r,h,:], y[r,h,:]> precomputed per row (the softmax-gradient row sum
//             sum_e p dp equals it, so no second pass over the edges is needed):
//                 p  = exp(leaky(a_dst[r] + a_src[s]) - row_max[r]) / row_sum[r]      (recomputed)
//                 dp = <dy[r,h,:], x[s,h,:]>                                          (per-head SDDMM)
//                 dt = p (dp - D[r,h]) * (t > 0 ? 1 : slope)
//                 dx[s,h,:] += p dy[r,h,:];   d a_src[s,h] += dt      (registers, fixed order)
//                 d a_dst[r,h] += dt: with the forward position of every transposed edge at hand (t_eid of
//                 the transpose) dt is stored at that position of a [nnz, H] scratch array and every
//                 destination then adds its edges' values in a fixed order (same bits on every run); without
//                 it, one atomic add per edge and head (order not fixed, as the reference's grad_src atomics).
//
// Shapes covered: fp32 features, heads a power of two <= 16, a feature row (heads * c floats) of up to 2 KiB (c a
// multiple of 4), 1 KiB (c even) or 1.5 KiB (any c); backward with c a power of two, at most 128. Everything else stays on
// the separate kernels (cxg_gat_scores, cxg_edge_softmax_forward, cxg_spmm_csr).
//
// What bounds it: instructions per edge and per row end, with an IPC of 0.55 to 0.65 per scheduler; the gather stays in L2
// for graphs of this kind. 2.33 M edges, 4 heads x 32: backward 271 us, forward in one step 178 (46 instructions per edge),
// in two 34 + 104, of which the walk is bound by L2 like the sum over such rows (90).
#include "spmm_walk_impl.cuh"

namespace cxg {
namespace {

using walk::kFar;
using walk::kThreads;
using walk::load_id_stream;

constexpr float kNegBig = -1e30f;  // "no edge yet": exp(kNegBig - t) is 0 for every finite t
constexpr int kLongRowEdges = 256;  // ordered d a_dst: destinations with more edges are summed piecewise by CTAs
                                    // (a single warp on a longer row is the tail of the kernel)

struct GatArgs {
  WalkArgs w;            // graph that is walked (CSR forward, transposed CSR backward) and its plan; w.x = rows fetched per
                         // edge: x [n_src, H, C] (forward), dy [n_dst, H, C] (backward); w.y = y (forward), dx (backward)
  const float *g_small;  // small per-node record fetched per edge: a_src [n_src, H] (forward),
                         // stats [n_dst, H, 4] = {a_dst, row_max, 1 / row_sum, D} (backward)
  const float *r_small;  // per walked row: a_dst [n_dst, H] (forward), a_src [n_src, H] (backward)
  const float *r_feat;   // backward: x [n_src, H, C]
  float *row_max;        // forward [n_dst, H]
  float *row_sum;        // forward [n_dst, H]
  float *d_r_small;      // backward: d a_src [n_src, H]
  float *d_g_small;      // backward: d a_dst [n_dst, H], added into atomically (when d_edge is NULL)
  const void *eid;       // backward, ordered mode: forward edge of every transposed edge (width of idx)
  float *d_edge;         // backward, ordered mode: [nnz, H] score gradient of every edge at its forward position
  int heads, c;
  float slope;
  float *weights;        // forward by way of weights: [nnz, H]
  float *part_ms;        // [tile][2][heads][2]: forward (m, s); backward (unused, d a_src partial)
  float *block_ms;       // [tile][heads][2]: those of a block of a long chain
};

// exp(x) = 2^(x log2 e), with results below 2^-126 flushed to zero. The product and its constant are rounded once each, so
// the exponent is off by at most |x| * 1.45 * 1.5 * 2^-24; with the 2^-22 of ex2.approx the result is off by at most
// (1.5 |x| + 4) * 2^-24 of itself.
__device__ __forceinline__ float exp_flush(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x * 1.4426950408889634f));
  return r;
}

// Per-tile state of a walk: where the walk stands in the rows. Positions are relative to the tile's first edge.
struct TileWalk {
  const GatArgs &a;
  int64_t begin, row;
  int len, rend, rstart, stop;
  int64_t next_raw;  // end of the row behind the walked one, requested a row ahead
  __device__ __forceinline__ int64_t end_raw(int64_t r) const {
    return load_ptr(a.w.ptr, min(r + 1, a.w.n_dst), a.w.ptr_bytes);
  }
  __device__ __forceinline__ int end_rel(int64_t r, int64_t raw) const {
    const int64_t v = raw - begin;
    return r >= a.w.n_dst || v > kFar ? kFar : static_cast<int>(v);
  }
  __device__ __forceinline__ void start() {
    rend = end_rel(row, end_raw(row));
    next_raw = end_raw(row + 1);
    const int64_t s = load_ptr(a.w.ptr, row, a.w.ptr_bytes) - begin;
    rstart = s < -kFar ? -kFar : static_cast<int>(s);
    stop = min(rend, len);
  }
  __device__ __forceinline__ void next() {
    ++row;
    rend = end_rel(row, next_raw);
    next_raw = end_raw(row + 1);
  }
  __device__ __forceinline__ uint32_t load_id(int pos) const {
    if (pos >= len) return 0u;
    return a.w.idx_bytes == 8 ? static_cast<uint32_t>(load_id_stream(static_cast<const int64_t *>(a.w.idx) + begin + pos))
                              : static_cast<uint32_t>(load_id_stream(static_cast<const int32_t *>(a.w.idx) + begin + pos));
  }
  // backward: the score gradient of the edge at `pos`, whose destination is `dst`
  __device__ __forceinline__ void edge_gradient(int pos, uint32_t dst, int head, float dt) const {
    if (a.d_edge != nullptr) {
      const int64_t e = a.w.idx_bytes == 8 ? __ldg(static_cast<const int64_t *>(a.eid) + begin + pos)
                                           : __ldg(static_cast<const int32_t *>(a.eid) + begin + pos);
      a.d_edge[e * a.heads + head] = dt;
    } else {
      asm volatile("red.global.add.f32 [%0], %1;" ::"l"(a.d_g_small + static_cast<int64_t>(dst) * a.heads + head), "f"(dt)
                   : "memory");
    }
  }
};

// Tiles behind the first round go to whichever warp comes for them: SMs differ in what they get through. A warp asks while it
// walks and looks at the answer, which lane 0 holds, afterwards.
struct NextTile {
  int32_t *counter;
  int64_t n_tiles, first;
  __device__ __forceinline__ NextTile(const GatArgs &a, int64_t tiles, int64_t walked)
      : counter(a.w.hdr + kWalkHdrNext), n_tiles(tiles), first(walked) {}
  __device__ __forceinline__ int64_t ask(int count) const {
    return first < n_tiles && (threadIdx.x & 31) == 0 ? first + atomicAdd(counter, count) : n_tiles;
  }
  __device__ __forceinline__ int64_t get(int64_t asked) const { return __shfl_sync(0xffffffffu, asked, 0); }
};

template <int VB>
__device__ __forceinline__ void load_floats(float (&f)[VB / 4], const float *p) {
  if constexpr (VB == 16) {
    const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
    f[0] = v.x, f[1] = v.y, f[2] = v.z, f[3] = v.w;
  } else if constexpr (VB == 8) {
    const float2 v = __ldg(reinterpret_cast<const float2 *>(p));
    f[0] = v.x, f[1] = v.y;
  } else {
    f[0] = __ldg(p);
  }
}
template <int W>
__device__ __forceinline__ void store_floats(float *dst, const float (&f)[W]) {
  if constexpr (W == 4)
    __stcs(reinterpret_cast<float4 *>(dst), make_float4(f[0], f[1], f[2], f[3]));
  else if constexpr (W == 2)
    __stcs(reinterpret_cast<float2 *>(dst), make_float2(f[0], f[1]));
  else
    __stcs(dst, f[0]);
}

// acc = acc * keep + prob * f and acc += prob * f, two columns per instruction
template <int W>
__device__ __forceinline__ void scale_add(float (&acc)[W], float keep, const float (&f)[W], float prob) {
  if constexpr (W == 1) {
    acc[0] = fmaf(acc[0], keep, prob * f[0]);
  } else {
#pragma unroll
    for (int i = 0; i < W; i += 2)
      asm("{\n\t.reg .b64 a, k, v, p;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 k, {%2, %2};\n\tmov.b64 v, {%3, %4};\n\t"
          "mov.b64 p, {%5, %5};\n\tmul.rn.f32x2 v, v, p;\n\tfma.rn.f32x2 a, a, k, v;\n\tmov.b64 {%0, %1}, a;\n\t}"
          : "+f"(acc[i]), "+f"(acc[(i + 1) % W])
          : "f"(keep), "f"(f[i]), "f"(f[(i + 1) % W]), "f"(prob));
  }
}
template <int W>
__device__ __forceinline__ void scale_add(float (&acc)[W], const float (&f)[W], float prob) {
  if constexpr (W == 1) {
    acc[0] = fmaf(prob, f[0], acc[0]);
  } else {
#pragma unroll
    for (int i = 0; i < W; i += 2)
      asm("{\n\t.reg .b64 a, v, p;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 v, {%2, %3};\n\tmov.b64 p, {%4, %4};\n\t"
          "fma.rn.f32x2 a, v, p, a;\n\tmov.b64 {%0, %1}, a;\n\t}"
          : "+f"(acc[i]), "+f"(acc[(i + 1) % W])
          : "f"(f[i]), "f"(f[(i + 1) % W]), "f"(prob));
  }
}

// Rows of up to 32 vectors: a group of G lanes per tile, one vector of VB bytes per lane, U edges in flight; see
// spmm_walk. What a row needs besides its edges (its score, in the backward its features) is requested a row ahead.
template <int VB, int G, int U, bool BWD, int MINB>
__global__ void __launch_bounds__(kThreads, MINB) gat_walk(const __grid_constant__ GatArgs a) {
  constexpr int W = VB / 4;
  constexpr int NG = 32 / G;
  const int lane = threadIdx.x & 31;
  const int lg = lane & (G - 1);
  const int H = a.heads;
  dependency_wait();
  const int64_t e_total = edge_total(a.w);
  const int64_t n_tiles = (e_total + a.w.tile - 1) / a.w.tile;
  const int64_t wid = (static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x) >> 5;
  const int64_t n_warps = static_cast<int64_t>(gridDim.x) * (kThreads / 32);
  const int width = a.w.width;
  const int64_t n_rows = a.w.n_dst;
  // a lane behind the row reads column 0 again and is not stored
  const bool on = lg * W < width;
  const int col = on ? lg * W : 0;
  const int head = col / a.c;
  const bool lead = on && col == head * a.c;  // first lane of its head
  const int lanes_per_head = BWD ? a.c / W : 0;
  const float *x = static_cast<const float *>(a.w.x) + col;
  const float *small_of = a.g_small + head * (BWD ? 4 : 1);
  float *y = static_cast<float *>(a.w.y) + col;
  auto empty_row = [&](int64_t r) {
    float z[W];
#pragma unroll
    for (int i = 0; i < W; ++i) z[i] = 0.f;
    if (on) store_floats<W>(y + r * width, z);
    if (lead) {
      if (BWD) {
        a.d_r_small[r * H + head] = 0.f;
      } else {
        a.row_max[r * H + head] = kNegBig;
        a.row_sum[r * H + head] = 0.f;
      }
    }
  };
  if (e_total == 0) {
    for (int64_t r = wid * NG + lane / G; r < n_rows; r += n_warps * NG) empty_row(r);
    return;
  }

  int64_t next_row = 0, next_begin = 0, next_stop = 0;
  auto fetch = [&](int64_t t) {
    next_begin = next_stop = 0;
    if (t < n_tiles) {
      next_row = static_cast<const WideTile *>(a.w.tiles)[t].row;
      next_begin = static_cast<const WideTile *>(a.w.tiles)[t].begin;
      next_stop = static_cast<const WideTile *>(a.w.tiles)[t + 1].begin;
    }
  };
  fetch(wid * NG + lane / G);
  for (int64_t t0 = wid * NG; t0 < n_tiles; t0 += n_warps * NG) {
    const int64_t t = t0 + lane / G;
    TileWalk w{a};
    w.begin = next_begin;
    w.row = next_row;
    w.len = next_stop > next_begin ? static_cast<int>(next_stop - next_begin) : 0;
    fetch(t + n_warps * NG);
    constexpr int IB = 32 / G;
    uint32_t id_cur[IB], id_nxt[IB];
    auto load_batch = [&](int first) {
#pragma unroll
      for (int j = 0; j < IB; ++j) id_nxt[j] = w.load_id(first + j * G + lg);
    };
    w.rend = w.stop = kFar;
    w.rstart = 0;
    w.next_raw = 0;
    if (w.len > 0) {
      if (t == 0)
        for (int64_t r = 0; r < w.row; ++r) empty_row(r);  // leading rows without edges
      w.start();
    }
    float score, score_next;  // of the walked row and of the one after it
    float xr[W], xr_next[W];
    auto load_row = [&](int64_t r) {
      const int64_t k = min(r, n_rows - 1);
      score_next = __ldg(a.r_small + k * H + head);
      if constexpr (BWD) load_floats<VB>(xr_next, a.r_feat + k * width + col);
    };
    auto take_row = [&]() {
      score = score_next;
      if constexpr (BWD) {
#pragma unroll
        for (int i = 0; i < W; ++i) xr[i] = xr_next[i];
      }
    };
    load_row(w.row);
    take_row();
    load_row(w.row + 1);

    float *yr = y + w.row * width;
    // forward: acc = sum of exp(t - m) x, m = largest t so far, s = sum of exp(t - m); backward: acc = dx, s = d a_src
    float acc[W], m, s;
    auto reset = [&]() {
      m = kNegBig;
      s = 0.f;
#pragma unroll
      for (int i = 0; i < W; ++i) acc[i] = 0.f;
    };
    reset();
    auto event = [&](int pos) {
      const bool row_done = pos == w.rend;
      if (row_done && w.rstart >= 0) {
        if (!BWD) {
          const float inv = 1.f / s;
#pragma unroll
          for (int i = 0; i < W; ++i) acc[i] *= inv;
        }
        if (on) store_floats<W>(yr, acc);
        if (lead) {
          if (BWD) {
            a.d_r_small[w.row * H + head] = s;
          } else {
            a.row_max[w.row * H + head] = m;
            a.row_sum[w.row * H + head] = s;
          }
        }
      } else if (w.row < n_rows) {
        const int64_t slot = t * 2 + (w.rstart < 0 ? 0 : 1);
        if (on) {
          float *p = a.w.partials + slot * width + col;
#pragma unroll
          for (int i = 0; i < W; ++i) p[i] = acc[i];
        }
        if (lead) *reinterpret_cast<float2 *>(a.part_ms + (slot * H + head) * 2) = make_float2(m, s);
      }
      reset();
      if (row_done) {
        w.rstart = pos;
        for (;;) {
          w.next();
          yr += width;
          take_row();
          load_row(w.row + 1);
          if (w.rend != pos) break;
          empty_row(w.row);
        }
      }
      w.stop = pos == w.len ? kFar : min(w.rend, w.len);
    };

    const int longest = G == 32 ? w.len : __reduce_max_sync(0xffffffffu, w.len);
    load_batch(0);
    for (int p = 0; p < longest; p += U) {
      const int in_batch = p & 31;
      if (in_batch == 0) {
#pragma unroll
        for (int j = 0; j < IB; ++j) id_cur[j] = id_nxt[j];
        load_batch(p + 32);
      }
      uint32_t id = id_cur[0];
#pragma unroll
      for (int j = 1; j < IB; ++j) id = in_batch >= j * G ? id_cur[j] : id;
      const int lane0 = in_batch & (G - 1);
      float v[U][W], small[U][BWD ? 4 : 1];
      uint32_t from[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        from[u] = __shfl_sync(0xffffffffu, id, lane0 + u, G);
        load_floats<VB>(v[u], x + static_cast<uint64_t>(from[u]) * static_cast<uint32_t>(width));
        const float *gs = small_of + static_cast<uint64_t>(from[u]) * static_cast<uint32_t>(H * (BWD ? 4 : 1));
        if constexpr (BWD)
          load_floats<16>(small[u], gs);
        else
          small[u][0] = __ldg(gs);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int pos = p + u;
        const float z = score + small[u][0];
        const float tl = z > 0.f ? z : z * a.slope;
        if constexpr (BWD) {
          const float prob = exp_flush(tl - small[u][1]) * small[u][2];
          float dot = 0.f;
#pragma unroll
          for (int i = 0; i < W; ++i) dot = fmaf(v[u][i], xr[i], dot);
          if (!on) dot = 0.f;
          for (int o = lanes_per_head >> 1; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
          float dt = prob * (dot - small[u][3]);
          dt = z > 0.f ? dt : dt * a.slope;
          s += dt;
          scale_add<W>(acc, v[u], prob);
          if (lead && pos < w.len) w.edge_gradient(pos, from[u], head, dt);
        } else {
          const float mn = fmaxf(m, tl);
          const float keep = exp_flush(m - mn), prob = exp_flush(tl - mn);
          m = mn;
          s = fmaf(s, keep, prob);
          scale_add<W>(acc, keep, v[u], prob);
        }
        if (pos + 1 == w.stop) event(pos + 1);
      }
    }
  }
}

// Rows of 17 to 384 vectors: a whole warp per tile. Scores, maxima and exponentials are computed once per (edge, head), one
// of them per lane, instead of by every lane that holds columns of the head: with 4 heads of 32 the walk above would spend
// 53 warp instructions per edge on the forward and 99 on the backward. The U edges of a step are taken segment by segment:
// the edges of one row.
//
// Forward. Lane l scores the edges (l >> log2 H) + j * (32 >> log2 H) of a step for head l & (H - 1); P = scores per lane.
// ST: vectors that lie across two heads (C not a multiple of the vector, at least as large as one; the row is).
template <int VB, int NV, int U, int P, int MINB, bool ST = false>
__global__ void __launch_bounds__(kThreads, MINB) gat_wide_forward(const __grid_constant__ GatArgs a) {
  constexpr int W = VB / 4;
  __shared__ float probs[kThreads / 32][P * 32];
  const int lane = threadIdx.x & 31;
  const int H = a.heads, hs = __ffs(H) - 1;
  const int my_head = lane & (H - 1);
  float *prob = probs[threadIdx.x >> 5];
  dependency_wait();
  const int64_t e_total = edge_total(a.w);
  const int64_t n_tiles = (e_total + a.w.tile - 1) / a.w.tile;
  const int64_t wid = (static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x) >> 5;
  const int64_t n_warps = static_cast<int64_t>(gridDim.x) * (kThreads / 32);
  const int width = a.w.width;
  const int64_t n_rows = a.w.n_dst;
  int col[NV], head[NV];  // vectors behind the row read column 0 again and are not stored
  bool on[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    const int c = (lane + q * 32) * W;
    on[q] = c < width;
    col[q] = on[q] ? c : 0;
    head[q] = col[q] / a.c;
  }
  const float *prob_of[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) prob_of[q] = prob + head[q];
  int next_head[ST ? NV : 1], own[ST ? NV : 1];  // head of a vector's last value, and how many values the first head has
  if constexpr (ST)
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      next_head[q] = (col[q] + W - 1) / a.c;
      own[q] = (head[q] + 1) * a.c - col[q];
    }
  // a value per head, held by the lanes of the head's index, times the accumulators
  auto scale_heads = [&](float (&acc)[NV][W], float per_head) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      const float k = __shfl_sync(0xffffffffu, per_head, head[q]);
      float k2 = k;
      if constexpr (ST) k2 = __shfl_sync(0xffffffffu, per_head, next_head[q]);
#pragma unroll
      for (int i = 0; i < W; ++i) acc[q][i] *= ST && i >= own[q] ? k2 : k;
    }
  };
  const float *x = static_cast<const float *>(a.w.x);
  float *y = static_cast<float *>(a.w.y);
  auto empty_row = [&](int64_t r) {
    float z[W];
#pragma unroll
    for (int i = 0; i < W; ++i) z[i] = 0.f;
#pragma unroll
    for (int q = 0; q < NV; ++q)
      if (on[q]) store_floats<W>(y + r * width + col[q], z);
    if (lane < H) {
      a.row_max[r * H + lane] = kNegBig;
      a.row_sum[r * H + lane] = 0.f;
    }
  };
  if (e_total == 0) {
    for (int64_t r = wid; r < n_rows; r += n_warps) empty_row(r);
    return;
  }
  const NextTile next_tile(a, n_tiles, n_warps);
  for (int64_t t = wid, t_next; t < n_tiles; t = next_tile.get(t_next)) {
    t_next = next_tile.ask(1);
    TileWalk w{a};
    w.begin = static_cast<const WideTile *>(a.w.tiles)[t].begin;
    w.row = static_cast<const WideTile *>(a.w.tiles)[t].row;
    const int64_t end = static_cast<const WideTile *>(a.w.tiles)[t + 1].begin;
    if (end <= w.begin) continue;
    w.len = static_cast<int>(end - w.begin);
    if (t == 0)
      for (int64_t r = 0; r < w.row; ++r) empty_row(r);  // leading rows without edges
    uint32_t id_next = w.load_id(lane);
    w.start();
    auto row_score = [&](int64_t r) { return __ldg(a.r_small + min(r, n_rows - 1) * H + my_head); };
    float score = row_score(w.row), score_next = row_score(w.row + 1);
    // acc = sum of exp(t - m) x; m = largest t so far of the lane's scoring head, s = this lane's part of sum of exp(t - m)
    float acc[NV][W], m = kNegBig, s = 0.f;
#pragma unroll
    for (int q = 0; q < NV; ++q)
#pragma unroll
      for (int i = 0; i < W; ++i) acc[q][i] = 0.f;
    uint32_t id = 0u;
    for (int p = 0; p < w.len; p += U) {
      const int lane0 = p & 31;
      if (lane0 == 0) {
        id = id_next;
        id_next = w.load_id(p + 32 + lane);
      }
      float v[U][NV][W], small[P];
#pragma unroll
      for (int j = 0; j < P; ++j) {
        const int e = (lane >> hs) + j * (32 >> hs);
        const uint32_t nid = __shfl_sync(0xffffffffu, id, lane0 + (e & (U - 1)));
        small[j] = __ldg(a.g_small + static_cast<uint64_t>(nid) * static_cast<uint32_t>(H) + my_head);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t nid = __shfl_sync(0xffffffffu, id, lane0 + u);
        const float *xs = x + static_cast<uint64_t>(nid) * static_cast<uint32_t>(width);
#pragma unroll
        for (int q = 0; q < NV; ++q) load_floats<VB>(v[u][q], xs + col[q]);
      }
      int q0 = 0;
#pragma unroll 1
      do {
        const int q1 = min(w.stop - p, U);
        const unsigned edges = ((2u << (q1 - 1)) - 1u) & (~0u << q0);  // the segment's edges, a bit each
        float tl[P], mx = kNegBig;
        bool in[P];
#pragma unroll
        for (int j = 0; j < P; ++j) {
          const int e = (lane >> hs) + j * (32 >> hs);
          in[j] = (edges >> e) & 1u;
          const float z = score + small[j];
          tl[j] = z > 0.f ? z : z * a.slope;
          if (in[j]) mx = fmaxf(mx, tl[j]);
        }
        for (int o = H; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (__any_sync(0xffffffffu, mx > m)) {  // seldom after a row's first edges
          const float mn = fmaxf(m, mx);
          const float keep = exp_flush(m - mn);
          m = mn;
          s *= keep;
          scale_heads(acc, keep);
        }
#pragma unroll
        for (int j = 0; j < P; ++j) {
          const float pr = in[j] ? exp_flush(tl[j] - m) : 0.f;
          s += pr;
          prob[j * 32 + lane] = pr;
        }
        __syncwarp();
        auto add = [&](int u) {
#pragma unroll
          for (int q = 0; q < NV; ++q) {
            if constexpr (ST) {
              const float k = prob_of[q][u << hs], k2 = prob[(u << hs) + next_head[q]];
#pragma unroll
              for (int i = 0; i < W; ++i) acc[q][i] = fmaf(v[u][q][i], i >= own[q] ? k2 : k, acc[q][i]);
            } else {
              scale_add<W>(acc[q], v[u][q], prob_of[q][u << hs]);
            }
          }
        };
        if (edges == (1u << U) - 1u) {
#pragma unroll
          for (int u = 0; u < U; ++u) add(u);
        } else {
#pragma unroll
          for (int u = 0; u < U; ++u)
            if ((edges >> u) & 1u) add(u);
        }
        __syncwarp();
        q0 = q1;
        if (p + q1 != w.stop) break;
        // the end of a row, of the tile, or of both
        for (int o = H; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const bool row_done = p + q1 == w.rend;
        if (row_done && w.rstart >= 0) {
          scale_heads(acc, 1.f / s);
#pragma unroll
          for (int q = 0; q < NV; ++q) {
            if (on[q]) store_floats<W>(y + w.row * width + col[q], acc[q]);
          }
          if (lane < H) {
            a.row_max[w.row * H + lane] = m;
            a.row_sum[w.row * H + lane] = s;
          }
        } else if (w.row < n_rows) {
          const int64_t slot = t * 2 + (w.rstart < 0 ? 0 : 1);
#pragma unroll
          for (int q = 0; q < NV; ++q)
            if (on[q]) {
              float *pp = a.w.partials + slot * width + col[q];
#pragma unroll
              for (int i = 0; i < W; ++i) pp[i] = acc[q][i];
            }
          if (lane < H) *reinterpret_cast<float2 *>(a.part_ms + (slot * H + lane) * 2) = make_float2(m, s);
        }
#pragma unroll
        for (int q = 0; q < NV; ++q)
#pragma unroll
          for (int i = 0; i < W; ++i) acc[q][i] = 0.f;
        m = kNegBig;
        s = 0.f;
        if (row_done) {
          w.rstart = w.rend;
          for (;;) {
            w.next();
            score = score_next;
            score_next = row_score(w.row + 1);
            if (w.rend != w.rstart) break;
            empty_row(w.row);
          }
        }
        w.stop = p + q1 == w.len ? kFar : min(w.rend, w.len);
      } while (q0 < U);
    }
  }
}

// Backward. The dot products of U edges are reduced over a head's lanes and spread over them at the same time (at every
// step a lane keeps half of the edges and hands the other half to its partner): 7 exchanges for 8 edges where a reduction
// per edge takes 24. R = min(lanes per head, U); afterwards a lane holds E = U / R edges of its head, from first_edge on.
template <int U, int R>
__device__ __forceinline__ int first_edge(int lane) {
  int e = 0;
#pragma unroll
  for (int o = 1, n = U / 2; o < R; o <<= 1, n >>= 1) e += (lane & o) ? n : 0;
  return e;
}
template <int U, int R>
__device__ __forceinline__ constexpr int lane_of_edge(int u) {
  int l = 0;
  for (int o = 1, n = U / 2; o < R; o <<= 1, n >>= 1) l += (u & n) ? o : 0;
  return l;
}

template <int NV, int U, int R, int MINB>
__global__ void __launch_bounds__(kThreads, MINB) gat_wide_backward(const __grid_constant__ GatArgs a) {
  constexpr int W = 4;
  constexpr int E = U / R;
  const int lane = threadIdx.x & 31;
  const int H = a.heads;
  const int lph = a.c / W;  // lanes per head, a power of two >= R
  const int group = lane & ~(lph - 1) & 31;
  const bool own = (lane & (lph - 1)) < R;  // the head's other lanes hold copies
  const bool lead = (lane & (lph - 1)) == 0;
  const int e0 = first_edge<U, R>(lane);
  dependency_wait();
  const int64_t e_total = edge_total(a.w);
  const int64_t n_tiles = (e_total + a.w.tile - 1) / a.w.tile;
  const int64_t wid = (static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x) >> 5;
  const int64_t n_warps = static_cast<int64_t>(gridDim.x) * (kThreads / 32);
  const int width = a.w.width;
  const int64_t n_rows = a.w.n_dst;
  int col[NV], head[NV];
  bool on[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    const int c = (lane + q * 32) * W;
    on[q] = c < width;
    col[q] = on[q] ? c : 0;
    head[q] = col[q] / a.c;
  }
  const float *dy = static_cast<const float *>(a.w.x);
  float *dx = static_cast<float *>(a.w.y);
  auto empty_row = [&](int64_t r) {
    const float z[W] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < NV; ++q)
      if (on[q]) {
        store_floats<W>(dx + r * width + col[q], z);
        if (lead) a.d_r_small[r * H + head[q]] = 0.f;
      }
  };
  if (e_total == 0) {
    for (int64_t r = wid; r < n_rows; r += n_warps) empty_row(r);
    return;
  }
  const NextTile next_tile(a, n_tiles, n_warps);
  for (int64_t t = wid, t_next; t < n_tiles; t = next_tile.get(t_next)) {
    t_next = next_tile.ask(1);
    TileWalk w{a};
    w.begin = static_cast<const WideTile *>(a.w.tiles)[t].begin;
    w.row = static_cast<const WideTile *>(a.w.tiles)[t].row;
    const int64_t end = static_cast<const WideTile *>(a.w.tiles)[t + 1].begin;
    if (end <= w.begin) continue;
    w.len = static_cast<int>(end - w.begin);
    if (t == 0)
      for (int64_t r = 0; r < w.row; ++r) empty_row(r);
    uint32_t id_next = w.load_id(lane);
    w.start();
    float score[NV], score_next[NV], xr[NV][W], xr_next[NV][W];
    auto load_row = [&](int64_t r) {
      const int64_t k = min(r, n_rows - 1);
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        score_next[q] = __ldg(a.r_small + k * H + head[q]);
        load_floats<16>(xr_next[q], a.r_feat + k * width + col[q]);
        if (!on[q])
#pragma unroll
          for (int i = 0; i < W; ++i) xr_next[q][i] = 0.f;
      }
    };
    auto take_row = [&]() {
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        score[q] = score_next[q];
#pragma unroll
        for (int i = 0; i < W; ++i) xr[q][i] = xr_next[q][i];
      }
    };
    load_row(w.row);
    take_row();
    load_row(w.row + 1);
    float acc[NV][W], s[NV];  // dx and this lane's part of d a_src of the walked row
    auto reset = [&]() {
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        s[q] = 0.f;
#pragma unroll
        for (int i = 0; i < W; ++i) acc[q][i] = 0.f;
      }
    };
    reset();
    uint32_t id = 0u;
    for (int p = 0; p < w.len; p += U) {
      const int lane0 = p & 31;
      if (lane0 == 0) {
        id = id_next;
        id_next = w.load_id(p + 32 + lane);
      }
      float v[U][NV][W];
      float4 stat[E][NV];
      uint32_t mine[E];
#pragma unroll
      for (int i = 0; i < E; ++i) {
        mine[i] = __shfl_sync(0xffffffffu, id, lane0 + e0 + i);
#pragma unroll
        for (int q = 0; q < NV; ++q)
          stat[i][q] = __ldg(reinterpret_cast<const float4 *>(a.g_small) + static_cast<uint64_t>(mine[i]) * static_cast<uint32_t>(H) + head[q]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t nid = __shfl_sync(0xffffffffu, id, lane0 + u);
        const float *src = dy + static_cast<uint64_t>(nid) * static_cast<uint32_t>(width);
#pragma unroll
        for (int q = 0; q < NV; ++q) load_floats<16>(v[u][q], src + col[q]);
      }
      int q0 = 0;
#pragma unroll 1
      do {
        const int q1 = min(w.stop - p, U);
        const unsigned edges = ((2u << (q1 - 1)) - 1u) & (~0u << q0);  // the segment's edges, a bit each
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          float d[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            d[u] = v[u][q][0] * xr[q][0];
#pragma unroll
            for (int i = 1; i < W; ++i) d[u] = fmaf(v[u][q][i], xr[q][i], d[u]);
          }
#pragma unroll
          for (int o = 1, n = U / 2; o < R; o <<= 1, n >>= 1) {
            const bool upper = lane & o;
#pragma unroll
            for (int i = 0; i < n; ++i) {
              const float other = __shfl_xor_sync(0xffffffffu, upper ? d[i] : d[i + n], o);
              d[i] = (upper ? d[i + n] : d[i]) + other;
            }
          }
          for (int o = R; o < lph; o <<= 1) {
#pragma unroll
            for (int i = 0; i < E; ++i) d[i] += __shfl_xor_sync(0xffffffffu, d[i], o);
          }
          float prob[E];
#pragma unroll
          for (int i = 0; i < E; ++i) {
            const float4 r = stat[i][q];
            const float z = score[q] + r.x;
            const float tl = z > 0.f ? z : z * a.slope;
            prob[i] = exp_flush(tl - r.y) * r.z;
            float dt = prob[i] * (d[i] - r.w);
            dt = z > 0.f ? dt : dt * a.slope;
            const int e = e0 + i;
            if (own && on[q] && ((edges >> e) & 1u) && p + e < w.len) {
              s[q] += dt;
              w.edge_gradient(p + e, mine[i], head[q], dt);
            }
          }
          auto add = [&](int u) {
            scale_add<W>(acc[q], v[u][q], __shfl_sync(0xffffffffu, prob[u % E], group | lane_of_edge<U, R>(u)));
          };
          if (edges == (1u << U) - 1u) {
#pragma unroll
            for (int u = 0; u < U; ++u) add(u);
          } else {
#pragma unroll
            for (int u = 0; u < U; ++u)
              if ((edges >> u) & 1u) add(u);
          }
        }
        q0 = q1;
        if (p + q1 != w.stop) break;
#pragma unroll
        for (int q = 0; q < NV; ++q)
#pragma unroll
          for (int o = 1; o < R; o <<= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
        const bool row_done = p + q1 == w.rend;
        if (row_done && w.rstart >= 0) {
#pragma unroll
          for (int q = 0; q < NV; ++q)
            if (on[q]) {
              store_floats<W>(dx + w.row * width + col[q], acc[q]);
              if (lead) a.d_r_small[w.row * H + head[q]] = s[q];
            }
        } else if (w.row < n_rows) {
          const int64_t slot = t * 2 + (w.rstart < 0 ? 0 : 1);
#pragma unroll
          for (int q = 0; q < NV; ++q)
            if (on[q]) {
              *reinterpret_cast<float4 *>(a.w.partials + slot * width + col[q]) = make_float4(acc[q][0], acc[q][1], acc[q][2], acc[q][3]);
              if (lead) *reinterpret_cast<float2 *>(a.part_ms + (slot * H + head[q]) * 2) = make_float2(0.f, s[q]);
            }
        }
        reset();
        if (row_done) {
          w.rstart = w.rend;
          for (;;) {
            w.next();
            take_row();
            load_row(w.row + 1);
            if (w.rend != w.rstart) break;
            empty_row(w.row);
          }
        }
        w.stop = p + q1 == w.len ? kFar : min(w.rend, w.len);
      } while (q0 < U);
    }
  }
}

// Forward in two steps: the weights of a tile's edges, then the weighted walk of the SpMM over the same tiles. A warp per tile:
// a lane per edge fetches the scores of its source into shared memory, a lane per (row, head) turns those of its row into
// weights (rows of more than kKeep edges: the whole warp), and the tile's weights leave in one piece. Rows inside the
// tile get their final weights; a piece of a row that crosses tile borders has weights relative to its own maximum and
// leaves (m, s) for gat_fix, as the walks above do.
constexpr int kKeep = 8;  // values of a row that a lane keeps in registers

template <int H>
__global__ void __launch_bounds__(kThreads, 8) gat_weights(const __grid_constant__ GatArgs a) {
  extern __shared__ float score_stage[];
  constexpr int R = 32 / H;  // rows that are looked at together
  constexpr int HV = H < 4 ? H : 4;
  const int lane = threadIdx.x & 31, h = lane & (H - 1);
  float *p = score_stage + (threadIdx.x >> 5) * a.w.tile * H;
  dependency_wait();
  const uint32_t e_total = static_cast<uint32_t>(edge_total(a.w));
  const int n_tiles = static_cast<int>((e_total + static_cast<int64_t>(a.w.tile) - 1) / a.w.tile);
  const int n_rows = static_cast<int>(a.w.n_dst);
  const int warps = static_cast<int>(gridDim.x * (blockDim.x >> 5)), first = static_cast<int>(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
  auto end_of = [&](int r) {
    return __ldg(reinterpret_cast<const uint32_t *>(static_cast<const uint8_t *>(a.w.ptr) + static_cast<uint64_t>(static_cast<uint32_t>(min(r, n_rows))) * static_cast<uint32_t>(a.w.ptr_bytes)));
  };
  auto put = [&](int r, float m, float s) {
    a.row_max[static_cast<int64_t>(r) * H + h] = m;
    a.row_sum[static_cast<int64_t>(r) * H + h] = s;
  };
  if (e_total == 0) {
    for (int r = first * R + lane / H; r < n_rows; r += warps * R) put(r, kNegBig, 0.f);
    return;
  }
  for (int t = first; t < n_tiles; t += warps) {
    const WalkTile here = load_tile(a.w, t);
    const uint32_t begin = here.begin;
    const int len = static_cast<int>(load_tile(a.w, t + 1).begin - begin);
    if (t == 0)
      for (int r = lane / H; r < static_cast<int>(here.row); r += R) put(r, kNegBig, 0.f);
    int r = static_cast<int>(here.row) + lane / H;
    uint32_t raw_b = end_of(r), raw_e = end_of(r + 1);
    float add = __ldg(a.r_small + static_cast<int64_t>(min(r, n_rows - 1)) * H + h);
    for (int e0 = lane; e0 < len; e0 += 128) {
      uint32_t id[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        id[u] = e0 + u * 32 < len ? walk::load_id_low(static_cast<const uint8_t *>(a.w.idx) + static_cast<uint64_t>(begin + e0 + u * 32) * static_cast<uint32_t>(a.w.idx_bytes)) : 0u;
#pragma unroll
      for (int i = 0; i < H; i += HV) {
        float v[4][HV];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          load_floats<HV * 4>(v[u], a.g_small + static_cast<uint64_t>(id[u]) * H + i);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (e0 + u * 32 < len) {
#pragma unroll
            for (int k = 0; k < HV; ++k) p[(e0 + u * 32) * H + i + k] = v[u][k];
          }
      }
    }
    __syncwarp();
    for (;;) {
      // of the rows behind these
      const uint32_t next_b = end_of(r + R), next_e = end_of(r + R + 1);
      const float next_add = __ldg(a.r_small + static_cast<int64_t>(min(r + R, n_rows - 1)) * H + h);
      const int b = static_cast<int>(raw_b - begin), e = static_cast<int>(raw_e - begin);
      const bool mine = r < n_rows && (b < len || (b == len && e == len));  // rows without edges belong to the tile in front
      const int lo = max(b, 0), hi = min(e, len), n = mine ? hi - lo : 0;
      const bool whole = b >= 0 && e <= len;
      float m = kNegBig, s = 0.f;
      // `cnt` values of a row, `step` apart; KEEP of them are held in registers
      auto weigh = [&](float *q, int cnt, int step, float plus, bool final, auto &&join_max, auto &&join_sum, float &top, float &sum) {
        float t[kKeep];
        top = kNegBig, sum = 0.f;
#pragma unroll
        for (int i = 0; i < kKeep; ++i) {
          t[i] = kNegBig;
          if (i < cnt) {
            const float z = plus + q[i * step];
            t[i] = z > 0.f ? z : z * a.slope;
          }
          top = fmaxf(top, t[i]);
        }
        top = join_max(top);
#pragma unroll
        for (int i = 0; i < kKeep; ++i) {
          t[i] = exp_flush(t[i] - top);
          if (i < cnt) sum += t[i];
        }
        sum = join_sum(sum);
        const float inv = final ? 1.f / sum : 1.f;
#pragma unroll
        for (int i = 0; i < kKeep; ++i)
          if (i < cnt) q[i * step] = t[i] * inv;
      };
      if (n > 0 && n <= kKeep)
        weigh(p + lo * H + h, n, H, add, whole, [](float v) { return v; }, [](float v) { return v; }, m, s);
      for (unsigned left = __ballot_sync(0xffffffffu, n > kKeep && h == 0); left != 0; left &= left - 1) {
        const int src = __ffs(left) - 1;
        const int jlo = __shfl_sync(0xffffffffu, lo, src), jn = __shfl_sync(0xffffffffu, n, src);
        const bool jwhole = __shfl_sync(0xffffffffu, whole, src);
        const float jadd = __shfl_sync(0xffffffffu, add, src + h);
        float *q = p + (jlo + lane / H) * H + h;
        const int cnt = (jn - lane / H + R - 1) / R;  // of this lane: every R-th edge
        auto over_max = [](float v) {
#pragma unroll
          for (int o = H; o < 32; o <<= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
          return v;
        };
        auto over_sum = [](float v) {
#pragma unroll
          for (int o = H; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          return v;
        };
        float jm = kNegBig, js = 0.f;
        if (jn <= kKeep * R) {
          weigh(q, cnt, 32, jadd, jwhole, over_max, over_sum, jm, js);
        } else {
#pragma unroll 4
          for (int i = 0; i < cnt; ++i) {
            const float z = jadd + q[i * 32];
            jm = fmaxf(jm, z > 0.f ? z : z * a.slope);
          }
          jm = over_max(jm);
#pragma unroll 4
          for (int i = 0; i < cnt; ++i) {
            const float z = jadd + q[i * 32];
            const float pr = exp_flush((z > 0.f ? z : z * a.slope) - jm);
            q[i * 32] = pr;
            js += pr;
          }
          js = over_sum(js);
          if (jwhole) {
            const float inv = 1.f / js;
            for (int i = 0; i < cnt; ++i) q[i * 32] *= inv;
          }
        }
        if ((lane & ~(H - 1)) == src) m = jm, s = js;
      }
      if (mine) {
        if (whole)
          put(r, m, s);
        else
          *reinterpret_cast<float2 *>(a.part_ms + ((static_cast<int64_t>(t) * 2 + (b < 0 ? 0 : 1)) * H + h) * 2) = make_float2(m, s);
      }
      if (__any_sync(0xffffffffu, !mine)) break;
      r += R;
      raw_b = next_b, raw_e = next_e, add = next_add;
    }
    __syncwarp();
    float *out = a.weights + static_cast<int64_t>(begin) * H;
    for (int i = lane; i < len * H; i += 32) out[i] = p[i];
    __syncwarp();
  }
}

constexpr int kGatSeq = 16;  // a chain of more partials is joined in blocks of this many, then the blocks: the hub row of
                             // 2.3 M edges (420 partials) costs 2 + 4 round trips instead of 8 + 1 with blocks of 64

// Joins n elements of a chain of partials, step apart, from element k0 on, VW columns per lane, in SV pieces that lie in
// one head each. FROM_BLOCKS: the (m, s) of the elements are those of finished blocks. Result to the row, or to the
// block's element.
template <int VW, int SV, bool BWD, bool FROM_BLOCKS>
__device__ void gat_chain(const GatArgs &a, int64_t ts, int64_t k0, int64_t n, int64_t step, bool to_block, int64_t row, int lane) {
  const int width = a.w.width, H = a.heads;
  constexpr int PV = VW / SV;   // columns per piece
  constexpr int kDepth = 8 / SV;  // partials requested at once
  for (int c = lane * VW; c < width; c += 32 * VW) {
    int h[SV];
#pragma unroll
    for (int j = 0; j < SV; ++j) h[j] = (c + j * PV) / a.c;
    float acc[VW], m[SV], s[SV];
    auto at = [&](int64_t k, float (&v)[VW], float2 (&ms)[SV]) {
      const int64_t e = k0 + k * step, slot = (ts + e) * 2 + (e == 0 ? 1 : 0);
      const float *p = a.w.partials + slot * width + c;
      if constexpr (VW == 4) {
        const float4 t = __ldcg(reinterpret_cast<const float4 *>(p));
        v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
      } else {
        v[0] = __ldcg(p);
      }
#pragma unroll
      for (int j = 0; j < SV; ++j)
        ms[j] = __ldcg(reinterpret_cast<const float2 *>(FROM_BLOCKS ? a.block_ms + ((ts + e) * H + h[j]) * 2
                                                                    : a.part_ms + (slot * H + h[j]) * 2));
    };
    auto join = [&](const float (&v)[VW], const float2 (&ms)[SV]) {
#pragma unroll
      for (int j = 0; j < SV; ++j) {
        float mine = 1.f, theirs = 1.f;
        if (!BWD) {
          const float mn = fmaxf(m[j], ms[j].x);
          mine = exp_flush(m[j] - mn), theirs = exp_flush(ms[j].x - mn);
          m[j] = mn;
        }
        s[j] = s[j] * mine + ms[j].y * theirs;
#pragma unroll
        for (int i = j * PV; i < (j + 1) * PV; ++i) acc[i] = acc[i] * mine + v[i] * theirs;
      }
    };
    {
      float2 ms[SV];
      at(0, acc, ms);
#pragma unroll
      for (int j = 0; j < SV; ++j) m[j] = ms[j].x, s[j] = ms[j].y;
    }
    int64_t k = 1;
    for (; k + kDepth <= n; k += kDepth) {
      float v[kDepth][VW];
      float2 ms[kDepth][SV];
#pragma unroll
      for (int u = 0; u < kDepth; ++u) at(k + u, v[u], ms[u]);
#pragma unroll
      for (int u = 0; u < kDepth; ++u) join(v[u], ms[u]);
    }
    for (; k < n; ++k) {
      float v[VW];
      float2 ms[SV];
      at(k, v, ms);
      join(v, ms);
    }
    float *out = to_block ? a.w.partials + ((ts + k0) * 2 + (k0 == 0 ? 1 : 0)) * width + c
                          : static_cast<float *>(a.w.y) + row * width + c;
#pragma unroll
    for (int j = 0; j < SV; ++j) {
      const float inv = BWD || to_block ? 1.f : 1.f / s[j];
#pragma unroll
      for (int i = j * PV; i < (j + 1) * PV; ++i) out[i] = acc[i] * inv;
      if (c + j * PV != h[j] * a.c) continue;  // the first column of the head writes its (m, s)
      if (to_block) {
        *reinterpret_cast<float2 *>(a.block_ms + ((ts + k0) * H + h[j]) * 2) = make_float2(m[j], s[j]);
      } else if (BWD) {
        a.d_r_small[row * H + h[j]] = s[j];
      } else {
        a.row_max[row * H + h[j]] = m[j];
        a.row_sum[row * H + h[j]] = s[j];
      }
    }
  }
}

// Rows that tiles cut: one warp per tile, the roles of walk_fix (spmm_walk.cu).
template <int VW, int SV, bool BWD>
__global__ void __launch_bounds__(256, 3) gat_fix(const __grid_constant__ GatArgs a, int per) {
  dependency_wait();
  const int lane = threadIdx.x & 31;
  const WalkArgs &w = a.w;
  const int64_t e_total = edge_total(w);
  // as walk_fix: `per` tiles are looked over at once, a lane for each of a tile's two roles
  const int64_t t = (blockIdx.x * 8ll + (threadIdx.x >> 5)) * per + (lane & (per - 1));
  bool lead = false;
  int64_t row = 0;
  int ts = 0, k = 0, m = 0;
  if (lane < 2 * per && t < w.max_tiles && t * w.tile < e_total) {
    // not written behind the last tile, whose end is e_total
    WideTile here, next;
    if (w.wide_tiles) {
      here = static_cast<const WideTile *>(w.tiles)[t], next = static_cast<const WideTile *>(w.tiles)[t + 1];
    } else {
      const WalkTile h = load_tile(w, t), n = load_tile(w, t + 1);
      here = WideTile{h.row, h.begin}, next = WideTile{n.row, n.begin};
    }
    const bool tail = lane < per;
    row = tail ? next.row : here.row;
    if (next.begin > here.begin && row < w.n_dst) {
      const int64_t rb = load_ptr(w.ptr, row, w.ptr_bytes);
      const int64_t re = min(load_ptr(w.ptr, row + 1, w.ptr_bytes), e_total);
      if (tail ? (rb < next.begin && rb >= here.begin) : rb < here.begin) {
        const int64_t first = tail ? t : rb / w.tile;
        ts = static_cast<int>(first), k = static_cast<int>(t - first);
        m = static_cast<int>((re - 1) / w.tile - first + 1);
        lead = k % kGatSeq == 0;
      }
    }
  }
  for (unsigned left = __ballot_sync(0xffffffffu, lead); left != 0; left &= left - 1) {
    const int src = __ffs(left) - 1;
    const int jts = __shfl_sync(0xffffffffu, ts, src), jk = __shfl_sync(0xffffffffu, k, src), jm = __shfl_sync(0xffffffffu, m, src);
    const int64_t jrow = __shfl_sync(0xffffffffu, row, src);
    const int n_blocks = (jm + kGatSeq - 1) / kGatSeq;
    gat_chain<VW, SV, BWD, false>(a, jts, jk, min(kGatSeq, jm - jk), 1, n_blocks > 1, jrow, lane);
    if (n_blocks == 1) continue;
    __threadfence();
    __syncwarp();
    int old = 0;
    if (lane == 0) old = atomicAdd(w.count + jts, 1);
    old = __shfl_sync(0xffffffffu, old, 0);
    if (old + 1 != n_blocks) continue;
    __threadfence();
    gat_chain<VW, SV, BWD, true>(a, jts, 0, n_blocks, kGatSeq, false, jrow, lane);
  }
}

// Backward set-up, one warp per destination: stats[r, h] = {a_dst, row_max, 1 / row_sum, <dy[r,h,:], y[r,h,:]>}
// and d a_dst[r, h] = 0 (the walk adds into it). A head's columns lie with c / W neighbouring lanes. With col_part the block
// also leaves the sums of dy's columns over its rows [gridDim.x, width], the gradient of the layer's bias, which was a pass over
// dy of its own (169,343 rows of 128: 65 us for both, now 49 with the join).
template <int W, int kRounds>  // kRounds of 32 * W columns
__global__ void __launch_bounds__(256) gat_bwd_prepare(const float *dy, const float *y, const float *a_dst,
                                                       const float *row_max, const float *row_sum, float *stats,
                                                       float *d_a_dst, float *col_part, int64_t n_dst, int heads, int c) {
  __shared__ float sums[8][kRounds * 32 * W];
  const int lane = threadIdx.x & 31;
  const int lph = c / W, width = heads * c;
  const int64_t gwarp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  constexpr int kRows = kRounds == 4 ? 1 : 4 / kRounds;  // rows whose loads are in flight
  float total[kRounds][W] = {};
  int head[kRounds];
  bool on[kRounds], lead[kRounds];
#pragma unroll
  for (int j = 0; j < kRounds; ++j) {
    const int col = (j * 32 + lane) * W;
    on[j] = col < width;
    head[j] = on[j] ? col / c : 0;
    lead[j] = on[j] && col == head[j] * c;
  }
  for (int64_t r0 = gwarp; r0 < n_dst; r0 += kRows * nwarps) {
    float g[kRows][kRounds][W], v[kRows][kRounds][W], sum[kRows][kRounds], top[kRows][kRounds], add[kRows][kRounds];
#pragma unroll
    for (int u = 0; u < kRows; ++u)
#pragma unroll
      for (int j = 0; j < kRounds; ++j) {
        const int64_t r = min(r0 + u * nwarps, n_dst - 1);
        const int col = on[j] ? (j * 32 + lane) * W : 0;
        load_floats<W * 4>(g[u][j], dy + r * width + col);
        load_floats<W * 4>(v[u][j], y + r * width + col);
        if (lead[j]) sum[u][j] = __ldg(row_sum + r * heads + head[j]), top[u][j] = __ldg(row_max + r * heads + head[j]), add[u][j] = __ldg(a_dst + r * heads + head[j]);
      }
#pragma unroll
    for (int u = 0; u < kRows; ++u)
#pragma unroll
      for (int j = 0; j < kRounds; ++j) {
        const int64_t r = r0 + u * nwarps;
        float d = 0.f;
        if (on[j]) {
#pragma unroll
          for (int i = 0; i < W; ++i) d = fmaf(g[u][j][i], v[u][j][i], d);
          if (r < n_dst)
#pragma unroll
            for (int i = 0; i < W; ++i) total[j][i] += g[u][j][i];
        }
        for (int o = lph >> 1; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        if (r < n_dst && lead[j]) {
          *reinterpret_cast<float4 *>(stats + (r * heads + head[j]) * 4) =
              make_float4(add[u][j], top[u][j], sum[u][j] > 0.f ? 1.f / sum[u][j] : 0.f, d);
          d_a_dst[r * heads + head[j]] = 0.f;
        }
      }
  }
  if (col_part == nullptr) return;
#pragma unroll
  for (int j = 0; j < kRounds; ++j)
#pragma unroll
    for (int i = 0; i < W; ++i) sums[threadIdx.x >> 5][(j * 32 + lane) * W + i] = total[j][i];
  __syncthreads();
  for (int col = threadIdx.x; col < width; col += 256) {
    float s = sums[0][col];
#pragma unroll
    for (int w = 1; w < 8; ++w) s += sums[w][col];
    col_part[static_cast<int64_t>(blockIdx.x) * width + col] = s;
  }
}

// Ordered d a_dst. The backward walk has left the score gradient of every edge at the edge's forward position
// (d_edge [nnz, H]); a destination's gradient is the sum over its edges, added in an order that depends on the
// graph only: lane (slot, head) of a warp takes every (32 / H)-th edge of the row (four running sums, joined in
// a fixed order), then the slots are joined by a butterfly. Destinations with more than kLongRowEdges edges are
// listed for the two kernels below.
__device__ __forceinline__ float strided_sum(const float *v, int64_t lo, int64_t hi, int64_t step) {
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  int64_t e = lo;
  for (; e + 3 * step < hi; e += 4 * step) {
    s0 += __ldg(v + e);
    s1 += __ldg(v + e + step);
    s2 += __ldg(v + e + 2 * step);
    s3 += __ldg(v + e + 3 * step);
  }
  for (; e < hi; e += step) s0 += __ldg(v + e);
  return (s0 + s1) + (s2 + s3);
}

__global__ void __launch_bounds__(256) gat_dst_sum_rows(const void *ptr, int ptr_bytes, const float *d_edge, float *d_a_dst,
                                                        int64_t n_dst, int64_t nnz, int heads, int hshift, int32_t *hdr,
                                                        int64_t *long_rows, int max_long) {
  constexpr int kRows = 4;  // destinations per warp and round: their loads are in flight together
  const int lane = threadIdx.x & 31;
  const int head = lane & (heads - 1), slot = lane >> hshift, nslot = 32 >> hshift;
  const int64_t gwarp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t r0 = gwarp * kRows; r0 < n_dst; r0 += nwarps * kRows) {
    // ptr[r0 .. r0 + kRows] through the first lanes
    int64_t pe = 0;
    if (lane <= kRows && r0 + lane <= n_dst) pe = min(load_ptr(ptr, r0 + lane, ptr_bytes), nnz);
    int64_t e[kRows + 1];
#pragma unroll
    for (int j = 0; j <= kRows; ++j) e[j] = __shfl_sync(0xffffffffu, pe, j);
    // rows of at most 4 * nslot edges: all their values requested before any is used; a lane's (up to) four values
    // are added as (v0 + v1) + (v2 + v3), which is the order strided_sum gives the same values
    float v[kRows][4];
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
      const bool row_on = r0 + j < n_dst && e[j + 1] - e[j] <= 4 * nslot;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int64_t ed = e[j] + slot + k * nslot;
        v[j][k] = (row_on && ed < e[j + 1]) ? __ldg(d_edge + ed * heads + head) : 0.f;
      }
    }
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
      const int64_t r = r0 + j;
      if (r >= n_dst) break;
      const int64_t e0 = e[j], e1 = e[j + 1];
      if (e1 - e0 > kLongRowEdges) {
        if (lane == 0) {
          const int s = atomicAdd(hdr + 1, 1);  // the list's order does not enter any sum
          if (s < max_long) long_rows[s] = r;
        }
        continue;
      }
      float acc;
      if (e1 - e0 <= 4 * nslot)
        acc = (v[j][0] + v[j][1]) + (v[j][2] + v[j][3]);
      else  // value (e, head) sits at d_edge[e * heads + head]: this lane walks e = e0 + slot, e0 + slot + nslot, ...
        acc = strided_sum(d_edge + head, (e0 + slot) * heads, e1 * heads, 32);
      for (int o = heads; o < 32; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane < heads) d_a_dst[r * heads + head] = acc;
    }
  }
}

// Long destinations, first level: the edge array is cut into pieces of kPieceEdges consecutive edges; every piece of
// a listed row is summed by one CTA (thread (slot, head) takes every (256 / H)-th edge, then a fixed tree in shared
// memory) into piece_sums. A piece holds at most one listed row's first edges and at most one listed row's later
// edges, hence two slots per piece. The CTAs share a row's pieces round-robin; the rows' edge ranges are read 128
// rows at a time into shared memory.
constexpr int kPieceEdges = 1024;
__global__ void __launch_bounds__(256) gat_dst_sum_pieces(const void *ptr, int ptr_bytes, const float *d_edge,
                                                          float *piece_sums, int64_t nnz, int heads, int hshift,
                                                          const int32_t *hdr, const int64_t *long_rows, int max_long) {
  __shared__ float red[256];
  __shared__ int64_t range[2][128];
  const int tid = threadIdx.x;
  const int head = tid & (heads - 1), slot = tid >> hshift;
  const int n_long = min(hdr[1], max_long);
  const int G = gridDim.x;
  for (int i0 = 0; i0 < n_long; i0 += 128) {
    {
      const int i = i0 + (tid & 127);
      if (i < n_long) range[tid >> 7][tid & 127] = min(load_ptr(ptr, long_rows[i] + (tid >> 7), ptr_bytes), nnz);
    }
    __syncthreads();
    const int cnt = min(128, n_long - i0);
    for (int ii = 0; ii < cnt; ++ii) {
      const int i = i0 + ii;
      const int64_t e0 = range[0][ii], e1 = range[1][ii];
      const int64_t p0 = e0 / kPieceEdges, p1 = (e1 - 1) / kPieceEdges;
      const int first = (static_cast<int>(blockIdx.x) + G - (i % G)) % G;
      for (int64_t p = p0 + first; p <= p1; p += G) {
        const int64_t lo = max(e0, p * kPieceEdges), hi = min(e1, (p + 1) * kPieceEdges);
        red[tid] = strided_sum(d_edge + head, (lo + slot) * heads, hi * heads, 256);
        __syncthreads();
        for (int o = 128; o >= heads; o >>= 1) {
          if (tid < o) red[tid] += red[tid + o];
          __syncthreads();
        }
        if (tid < heads) piece_sums[(2 * p + (p == p0 ? 1 : 0)) * heads + tid] = red[tid];
        __syncthreads();
      }
    }
    __syncthreads();
  }
}

// Second level: one warp per listed destination adds the sums of its pieces, lane (slot, head) every (32 / H)-th
// piece in ascending order, then the butterfly.
__global__ void __launch_bounds__(256) gat_dst_sum_long(const void *ptr, int ptr_bytes, const float *piece_sums,
                                                        float *d_a_dst, int64_t nnz, int heads, int hshift,
                                                        const int32_t *hdr, const int64_t *long_rows, int max_long) {
  const int lane = threadIdx.x & 31;
  const int head = lane & (heads - 1), slot = lane >> hshift, nslot = 32 >> hshift;
  const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
  const int n_long = min(hdr[1], max_long);
  for (int i = gwarp; i < n_long; i += nwarps) {
    const int64_t r = long_rows[i];
    const int64_t e0 = min(load_ptr(ptr, r, ptr_bytes), nnz), e1 = min(load_ptr(ptr, r + 1, ptr_bytes), nnz);
    const int64_t p0 = e0 / kPieceEdges, p1 = (e1 - 1) / kPieceEdges;
    float acc = 0.f;
    for (int64_t p = p0 + slot; p <= p1; p += nslot) acc += piece_sums[(2 * p + (p == p0 ? 1 : 0)) * heads + head];
    for (int o = heads; o < 32; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane < heads) d_a_dst[r * heads + head] = acc;
  }
}

struct GatLayout {
  WalkLayout walk;
  size_t part_ms, block_ms, stats, col_part, long_rows, piece_sums, d_edge, total;
};

// Blocks of gat_bwd_prepare.
int64_t prepare_blocks(int64_t n_dst) { return n_dst / 8 + 1 < kNumSM * 8 ? n_dst / 8 + 1 : kNumSM * 8; }

int gat_layout(int64_t n_stats_rows, int64_t nnz, int heads, int c, GatLayout *L) {
  const int rc = walk_layout(nnz, static_cast<int64_t>(heads) * c, 64, &L->walk);  // 64 = smallest tile
  if (rc != CXG_OK) return rc;
  size_t off = L->walk.total;
  L->part_ms = off;
  off = align_up(off + static_cast<size_t>(L->walk.max_tiles) * 2 * heads * 2 * sizeof(float), 256);
  L->block_ms = off;
  off = align_up(off + static_cast<size_t>(L->walk.max_tiles) * heads * 2 * sizeof(float), 256);
  L->stats = off;
  off = align_up(off + static_cast<size_t>(n_stats_rows) * heads * 4 * sizeof(float), 256);
  L->col_part = off;
  off = align_up(off + static_cast<size_t>(prepare_blocks(n_stats_rows)) * heads * c * sizeof(float), 256);
  // ordered d a_dst of the backward: destinations of more than kLongRowEdges edges, and one value per edge and head
  L->long_rows = off;
  off = align_up(off + static_cast<size_t>(nnz / kLongRowEdges + 1) * sizeof(int64_t), 256);
  L->piece_sums = off;
  off = align_up(off + static_cast<size_t>(nnz / kPieceEdges + 1) * 2 * heads * sizeof(float), 256);
  L->d_edge = off;
  off = align_up(off + static_cast<size_t>(nnz) * heads * sizeof(float) + walk_weights_slack(heads), 256);
  L->total = off;
  return CXG_OK;
}

// Widest vector that stays inside a head, narrowed so that eight lanes, the fewest a tile is given, have one each.
int vector_of(int heads, int c) {
  int vb = 16;
  while ((c * 4) % vb != 0) vb /= 2;
  while (vb > 4 && heads * c * 4 <= 4 * vb) vb /= 2;
  return vb;
}

int check_shape(const char *who, int heads, int c, bool backward) {
  if (heads < 1 || heads > 16 || (heads & (heads - 1)) != 0 || c < 1)
    return set_error(CXG_EUNSUPPORTED, "%s: heads = %d must be a power of two <= 16", who, heads);
  const int vb = vector_of(heads, c), n = heads * c * 4 / vb;
  if (n > (vb == 4 ? 384 : 128))
    return set_error(CXG_EUNSUPPORTED, "%s: a feature row of heads * c = %d values is too wide", who, heads * c);
  if (backward && ((c & (c - 1)) != 0 || c * 4 / vb > 32))
    return set_error(CXG_EUNSUPPORTED, "%s: c = %d must be a power of two of at most 128 in the backward", who, c);
  return CXG_OK;
}

void fill_args(GatArgs &a, const GatLayout &L, void *workspace, int64_t nnz, int heads, int c, float slope) {
  char *ws = static_cast<char *>(workspace);
  WalkArgs &w = a.w;
  w.hdr = reinterpret_cast<int32_t *>(ws + L.walk.hdr);
  w.tiles = ws + L.walk.tiles;
  w.count = reinterpret_cast<int32_t *>(ws + L.walk.count);
  w.partials = reinterpret_cast<float *>(ws + L.walk.partials);
  w.nnz = nnz;
  w.width = heads * c, w.row_bytes = heads * c * 4, w.heads = heads, w.feat = c;
  w.whole_rows = 0;
  w.wide_tiles = 1;
  w.x_rows = nullptr, w.copy_vectors = 0;
  a.part_ms = reinterpret_cast<float *>(ws + L.part_ms);
  a.block_ms = reinterpret_cast<float *>(ws + L.block_ms);
  a.heads = heads;
  a.c = c;
  a.slope = slope;
}

// Rows of whole 16-byte vectors whose heads are not (class counts), from 65 values on: vectors that lie across two heads,
// in place of single values (16 heads of 15: 957 us, now 522; 4 of 17: 404, now 314; 4 of 47: 519, now 495) and of
// 8-byte ones from 16 values per head on (4 of 30: 357, now 327; 8 of 10 would take 376 instead of 344).
bool across_heads(const GatArgs &a, int vb) {
  return vb < 16 && (vb == 4 || a.c >= 16) && a.w.width % 4 == 0 && a.w.width > 64 && a.c >= 4 &&
         (reinterpret_cast<uintptr_t>(a.w.x) | reinterpret_cast<uintptr_t>(a.w.y)) % 16 == 0;
}

// Whether the forward goes by way of weights. Its second step is the SpMM's walk, which counts in 32 bits. It has a launch more
// than the single walk, which keeps rows of up to 32 16-byte vectors of small graphs (430,000 edges: 4 heads of 8 38 us in one
// step, 42 in two; 8 of 8 41 / 47; 4 of 32 51 / 47; 2.3 M edges: 99 / 98, 150 / 128, 198 / 157). Wider rows and other vectors
// gain everywhere: 27,000 edges 4 of 64 44 / 36, 2 of 33 47 / 35; 2.3 M 4 of 64 391 / 246, 1 of 47 301 / 115, 2 of 50 323 / 249.
bool by_weights(const GatArgs &a, int vb) {
  const bool one_step = vb == 16 && a.w.width <= 128 && a.w.nnz * a.w.row_bytes < (128 << 20);
  return !one_step && !across_heads(a, vb) && a.heads <= 8 && reinterpret_cast<uintptr_t>(a.g_small) % 16 == 0 && a.w.n_dst < INT32_MAX - (1 << 20) &&
         a.w.nnz < INT32_MAX - (1 << 20) && a.w.width * 4 <= (vb == 16 ? 128 * 16 : 256 * vb);
}

// Edges per tile of that form, 0: no lane layout for its rows.
int weighted_tile(const GatArgs &a, int vb) {
  int resident = 0;
  if (!walk_weighted(a.w, vb, nullptr, &resident)) return 0;
  const int tile = walk_whole_waves(a.w.nnz, resident, 16);
  return tile < kWeightedTile ? tile : kWeightedTile;
}

cudaError_t launch_by_weights(GatArgs &a, int vb, cudaStream_t st) {
  a.w.wide_tiles = 0;
  a.w.edge_val = a.weights;
  a.w.part_stride = a.w.width;
  a.w.tile = weighted_tile(a, vb);
  if (a.w.tile == 0) return cudaErrorInvalidValue;
  a.w.max_tiles = (a.w.nnz + a.w.tile - 1) / a.w.tile + 1;
  walk_plan_run(a.w, st);
  constexpr int warps = kThreads / 32;
  int64_t grid = (a.w.max_tiles + warps - 1) / warps;  // a tile per warp while that many blocks are worth launching
  if (grid > kNumSM * 64) grid = kNumSM * 64;
  cudaError_t err = cudaErrorInvalidValue;
  auto go = [&](auto kernel) {
    err = launch_dependent(kernel, static_cast<unsigned>(grid), 32 * warps, static_cast<size_t>(warps) * a.w.tile * a.heads * sizeof(float), st, a);
  };
  if (a.heads == 1) go(gat_weights<1>);
  if (a.heads == 2) go(gat_weights<2>);
  if (a.heads == 4) go(gat_weights<4>);
  if (a.heads == 8) go(gat_weights<8>);
  if (err != cudaSuccess) return err;
  return walk_weighted(a.w, vb, st, nullptr) ? cudaSuccess : cudaErrorInvalidValue;
}

// Lane layouts by bytes per vector and vectors per row; the last number is the resident CTAs per SM that the registers of
// that many edges in flight allow.
template <bool BWD>
cudaError_t launch_walk(GatArgs &a, cudaStream_t st) {
  const int vb = vector_of(a.heads, a.c), n = a.w.row_bytes / vb;
  cudaError_t err = cudaErrorInvalidValue;
  auto go = [&](auto kernel, int g, int ctas) {
    const int per_cta = kThreads / g;
    const int64_t resident = static_cast<int64_t>(kNumSM) * ctas;
    a.w.tile = walk_tile_of_waves(a.w.nnz, resident * per_cta);
    a.w.max_tiles = (a.w.nnz + a.w.tile - 1) / a.w.tile + 1;
    walk_plan_run(a.w, st);
    int64_t grid = (a.w.max_tiles + per_cta - 1) / per_cta;
    if (grid > resident) grid = resident;
    err = launch_dependent(kernel, static_cast<unsigned>(grid), kThreads, 0, st, a);
  };
#define CXG_GAT(VB, G, U, CTAS) \
  if (vb == VB && n <= G) go(gat_walk<VB, G, U, BWD, CTAS>, G, CTAS); else
#define CXG_GAT_FWD(VB, NV, U, P, CTAS) \
  if (vb == VB && n <= 32 * NV && U * a.heads <= 32 * P) go(gat_wide_forward<VB, NV, U, P, CTAS>, 32, CTAS); else
#define CXG_GAT_BWD(NV, U, R, CTAS) \
  if (vb == 16 && n <= 32 * NV && a.c / 4 >= R) go(gat_wide_backward<NV, U, R, CTAS>, 32, CTAS); else
  if constexpr (BWD) {
    CXG_GAT(16, 8, 4, 6)
    CXG_GAT(16, 16, 4, 6)
    CXG_GAT(8, 8, 4, 6)
    CXG_GAT(8, 16, 4, 6)
    CXG_GAT(4, 8, 4, 6)
    CXG_GAT(4, 16, 4, 6)
    CXG_GAT_BWD(1, 4, 4, 8)
    CXG_GAT_BWD(1, 4, 2, 7)
    CXG_GAT_BWD(2, 4, 4, 4)
    CXG_GAT_BWD(4, 2, 2, 3)
    return cudaErrorInvalidValue;
  } else {
    const bool across = across_heads(a, vb);
    if (by_weights(a, vb)) err = launch_by_weights(a, vb, st); else
#define CXG_GAT_ACROSS(NV, U, P, CTAS) \
  if (across && a.w.width <= 128 * NV && U * a.heads <= 32 * P) go(gat_wide_forward<16, NV, U, P, CTAS, true>, 32, CTAS); else
    CXG_GAT_ACROSS(1, 8, 1, 6)
    CXG_GAT_ACROSS(1, 8, 4, 6)
    CXG_GAT_ACROSS(2, 8, 1, 4)
    CXG_GAT_ACROSS(2, 4, 1, 5)
    CXG_GAT_ACROSS(2, 4, 2, 5)
    CXG_GAT_ACROSS(4, 4, 2, 3)
#undef CXG_GAT_ACROSS
    CXG_GAT(16, 8, 8, 6)
    CXG_GAT(16, 16, 8, 6)
    CXG_GAT(8, 8, 8, 6)
    CXG_GAT(8, 16, 8, 6)
    CXG_GAT(4, 8, 8, 6)
    CXG_GAT(4, 16, 8, 6)
    CXG_GAT(16, 32, 8, 6)
    CXG_GAT_FWD(16, 2, 4, 2, 6)
    CXG_GAT_FWD(16, 4, 2, 1, 5)
    CXG_GAT(8, 32, 8, 6)
    CXG_GAT_FWD(8, 2, 8, 4, 5)
    CXG_GAT_FWD(8, 4, 4, 2, 5)
    CXG_GAT(4, 32, 8, 6)
    CXG_GAT_FWD(4, 2, 8, 4, 6)
    CXG_GAT_FWD(4, 4, 8, 4, 5)
    CXG_GAT_FWD(4, 6, 4, 1, 5)
    CXG_GAT_FWD(4, 6, 4, 2, 5)
    CXG_GAT_FWD(4, 12, 2, 1, 5)
    return cudaErrorInvalidValue;
  }
#undef CXG_GAT
#undef CXG_GAT_FWD
#undef CXG_GAT_BWD
  if (err != cudaSuccess) return err;
  // tiles a warp looks over: one while the chip holds a warp for each, up to sixteen (two roles on 32 lanes)
  int per = 1;
  while (per < 16 && a.w.max_tiles > static_cast<int64_t>(per) * kNumSM * 24) per *= 2;
  const unsigned grid = static_cast<unsigned>((a.w.max_tiles + 8 * per - 1) / (8 * per));
  if (a.c % 4 == 0)
    err = launch_dependent(gat_fix<4, 1, BWD>, grid, 256, 0, st, a, per);
  else if (a.w.width % 4 == 0)  // vectors that lie across two heads
    err = launch_dependent(gat_fix<4, 4, BWD>, grid, 256, 0, st, a, per);
  else
    err = launch_dependent(gat_fix<1, 1, BWD>, grid, 256, 0, st, a, per);
  count_launches(3);
  return err;
}

}  // namespace
}  // namespace cxg

using namespace cxg;

extern "C" int cxg_gat_fused_workspace_size(int64_t n_dst, int64_t nnz, int heads, int c, size_t *bytes) {
  CXG_REQUIRE(bytes != nullptr, CXG_ENULL, "cxg_gat_fused_workspace_size: bytes is NULL");
  CXG_REQUIRE(n_dst >= 0 && nnz >= 0 && heads > 0 && c > 0, CXG_EINVAL, "cxg_gat_fused_workspace_size: bad sizes");
  GatLayout L;
  const int rc = gat_layout(n_dst, nnz, heads, c, &L);
  CXG_REQUIRE(rc == CXG_OK, rc, "cxg_gat_fused_workspace_size: graph too large for 32-bit tile ids");
  *bytes = L.total;
  return CXG_OK;
}

extern "C" int cxg_gat_fused_weights_room(int64_t n_dst, int64_t nnz, int heads, int c, int *tile, size_t *bytes) {
  CXG_REQUIRE(tile != nullptr && bytes != nullptr, CXG_ENULL, "cxg_gat_fused_weights_room: NULL argument");
  CXG_REQUIRE(n_dst >= 0 && nnz >= 0, CXG_EINVAL, "cxg_gat_fused_weights_room: negative size");
  int rc = check_shape("cxg_gat_fused_weights_room", heads, c, false);
  if (rc != CXG_OK) return rc;
  GatLayout L;
  rc = gat_layout(n_dst, nnz, heads, c, &L);
  CXG_REQUIRE(rc == CXG_OK, rc, "cxg_gat_fused_weights_room: graph too large for 32-bit tile ids");
  GatArgs a = {};
  a.w.n_dst = n_dst, a.w.nnz = nnz;
  a.w.width = heads * c, a.w.row_bytes = heads * c * 4, a.w.heads = a.heads = heads, a.w.feat = a.c = c;
  const int vb = vector_of(heads, c);
  *tile = by_weights(a, vb) ? weighted_tile(a, vb) : 0;
  *bytes = L.total - L.d_edge;
  return CXG_OK;
}

extern "C" int cxg_gat_fused_forward(const void *ptr, const void *idx, int ptr_bytes, int idx_bytes, const float *x,
                                     const float *a_src, const float *a_dst, float *y, float *row_max, float *row_sum,
                                     int64_t n_dst, int64_t nnz, int heads, int c, float slope, void *workspace,
                                     size_t workspace_bytes, void *stream) {
  CXG_REQUIRE(n_dst >= 0 && nnz >= 0, CXG_EINVAL, "cxg_gat_fused_forward: negative size");
  CXG_REQUIRE((ptr_bytes == 4 || ptr_bytes == 8) && (idx_bytes == 4 || idx_bytes == 8), CXG_EINVAL,
              "cxg_gat_fused_forward: index widths %d/%d", ptr_bytes, idx_bytes);
  int rc = check_shape("cxg_gat_fused_forward", heads, c, false);
  if (rc != CXG_OK) return rc;
  if (n_dst == 0) return CXG_OK;
  CXG_REQUIRE(ptr && a_dst && y && row_max && row_sum, CXG_ENULL, "cxg_gat_fused_forward: NULL argument");
  CXG_REQUIRE(nnz == 0 || (idx && x && a_src), CXG_ENULL, "cxg_gat_fused_forward: idx, x or a_src is NULL");
  CXG_REQUIRE(reinterpret_cast<uintptr_t>(x) % 16 == 0 && reinterpret_cast<uintptr_t>(y) % 16 == 0, CXG_EINVAL,
              "cxg_gat_fused_forward: x and y must be 16-byte aligned");
  GatLayout L;
  rc = gat_layout(n_dst, nnz, heads, c, &L);
  CXG_REQUIRE(rc == CXG_OK, rc, "cxg_gat_fused: graph too large for 32-bit tile ids");
  CXG_REQUIRE(workspace != nullptr && workspace_bytes >= L.total, CXG_EWORKSPACE,
              "cxg_gat_fused_forward: workspace %zu bytes, need %zu", workspace_bytes, L.total);
  CXG_REQUIRE(reinterpret_cast<uintptr_t>(workspace) % 16 == 0, CXG_EINVAL, "cxg_gat_fused_forward: workspace alignment");
  GatArgs a = {};
  fill_args(a, L, workspace, nnz, heads, c, slope);
  a.w.ptr = ptr, a.w.idx = idx, a.w.ptr_bytes = ptr_bytes, a.w.idx_bytes = idx_bytes;
  a.w.x = x, a.g_small = a_src, a.r_small = a_dst;
  a.w.y = y, a.row_max = row_max, a.row_sum = row_sum;
  a.w.n_dst = n_dst;
  a.weights = reinterpret_cast<float *>(static_cast<char *>(workspace) + L.d_edge);
  cudaError_t e = launch_walk<false>(a, as_stream(stream));
  if (e != cudaSuccess) return set_error(CXG_ECUDA, "cxg_gat_fused_forward: %s", cudaGetErrorString(e));
  return check_launch("cxg_gat_fused_forward");
}

extern "C" int cxg_gat_fused_backward_bias(const void *t_ptr, const void *t_idx, int ptr_bytes, int idx_bytes, const float *dy,
                                      const float *y, const float *x, const float *a_src, const float *a_dst,
                                      const float *row_max, const float *row_sum, float *dx, float *d_a_src,
                                      float *d_a_dst, int64_t n_src, int64_t n_dst, int64_t nnz, int heads, int c,
                                      float slope, const void *t_eid, const void *fwd_ptr, int fwd_ptr_bytes, float *d_bias,
                                      void *workspace, size_t workspace_bytes, void *stream) {
  CXG_REQUIRE(n_src >= 0 && n_dst >= 0 && nnz >= 0, CXG_EINVAL, "cxg_gat_fused_backward: negative size");
  CXG_REQUIRE((ptr_bytes == 4 || ptr_bytes == 8) && (idx_bytes == 4 || idx_bytes == 8), CXG_EINVAL,
              "cxg_gat_fused_backward: index widths %d/%d", ptr_bytes, idx_bytes);
  int rc = check_shape("cxg_gat_fused_backward", heads, c, true);
  if (rc != CXG_OK) return rc;
  if (n_src == 0) return CXG_OK;
  CXG_REQUIRE(t_ptr && x && a_src && dx && d_a_src && d_a_dst, CXG_ENULL, "cxg_gat_fused_backward: NULL argument");
  CXG_REQUIRE(n_dst == 0 || (dy && y && a_dst && row_max && row_sum), CXG_ENULL, "cxg_gat_fused_backward: NULL argument");
  CXG_REQUIRE(d_bias == nullptr || n_dst > 0, CXG_EINVAL, "cxg_gat_fused_backward_bias: no rows");
  CXG_REQUIRE(nnz == 0 || t_idx, CXG_ENULL, "cxg_gat_fused_backward: t_idx is NULL");
  CXG_REQUIRE((t_eid == nullptr) == (fwd_ptr == nullptr), CXG_EINVAL,
              "cxg_gat_fused_backward: t_eid and fwd_ptr select the ordered d_a_dst together");
  CXG_REQUIRE(fwd_ptr == nullptr || fwd_ptr_bytes == 4 || fwd_ptr_bytes == 8, CXG_EINVAL,
              "cxg_gat_fused_backward: fwd_ptr_bytes %d", fwd_ptr_bytes);
  CXG_REQUIRE(reinterpret_cast<uintptr_t>(x) % 16 == 0 && reinterpret_cast<uintptr_t>(dy) % 16 == 0 &&
                  reinterpret_cast<uintptr_t>(y) % 16 == 0 && reinterpret_cast<uintptr_t>(dx) % 16 == 0,
              CXG_EINVAL, "cxg_gat_fused_backward: feature matrices must be 16-byte aligned");
  GatLayout L;
  rc = gat_layout(n_dst, nnz, heads, c, &L);
  CXG_REQUIRE(rc == CXG_OK, rc, "cxg_gat_fused: graph too large for 32-bit tile ids");
  CXG_REQUIRE(workspace != nullptr && workspace_bytes >= L.total, CXG_EWORKSPACE,
              "cxg_gat_fused_backward: workspace %zu bytes, need %zu", workspace_bytes, L.total);
  CXG_REQUIRE(reinterpret_cast<uintptr_t>(workspace) % 16 == 0, CXG_EINVAL, "cxg_gat_fused_backward: workspace alignment");
  GatArgs a = {};
  fill_args(a, L, workspace, nnz, heads, c, slope);
  float *stats = reinterpret_cast<float *>(reinterpret_cast<char *>(workspace) + L.stats);
  a.w.ptr = t_ptr, a.w.idx = t_idx, a.w.ptr_bytes = ptr_bytes, a.w.idx_bytes = idx_bytes;
  a.w.x = dy, a.g_small = stats, a.r_small = a_src, a.r_feat = x;
  a.w.y = dx, a.d_r_small = d_a_src, a.d_g_small = d_a_dst;
  const bool ordered = t_eid != nullptr && nnz > 0 && n_dst > 0;
  a.eid = ordered ? t_eid : nullptr;
  a.d_edge = ordered ? reinterpret_cast<float *>(reinterpret_cast<char *>(workspace) + L.d_edge) : nullptr;
  a.w.n_dst = n_src;
  int hshift = 0;
  while ((1 << hshift) < heads) ++hshift;
  cudaStream_t st = as_stream(stream);
  if (n_dst > 0) {
    const unsigned pg = static_cast<unsigned>(prepare_blocks(n_dst));
    float *col_part = d_bias != nullptr ? reinterpret_cast<float *>(static_cast<char *>(workspace) + L.col_part) : nullptr;
    const int vb = vector_of(heads, c);
    if (vb == 4)
      gat_bwd_prepare<1, 1><<<pg, 256, 0, st>>>(dy, y, a_dst, row_max, row_sum, stats, d_a_dst, col_part, n_dst, heads, c);
    else if (vb == 8)
      gat_bwd_prepare<2, 1><<<pg, 256, 0, st>>>(dy, y, a_dst, row_max, row_sum, stats, d_a_dst, col_part, n_dst, heads, c);
    else
      (heads * c <= 128 ? gat_bwd_prepare<4, 1> : heads * c <= 256 ? gat_bwd_prepare<4, 2> : gat_bwd_prepare<4, 4>)<<<pg, 256, 0, st>>>(dy, y, a_dst, row_max, row_sum, stats, d_a_dst, col_part, n_dst, heads, c);
    count_launches(1);
    if (d_bias != nullptr) {
      column_sum_join(col_part, d_bias, static_cast<int>(pg), heads * c, st);
      count_launches(1);
    }
  }
  cudaError_t e = launch_walk<true>(a, st);
  if (e != cudaSuccess) return set_error(CXG_ECUDA, "cxg_gat_fused_backward: %s", cudaGetErrorString(e));
  if (ordered) {
    int64_t *long_rows = reinterpret_cast<int64_t *>(reinterpret_cast<char *>(workspace) + L.long_rows);
    const int max_long = static_cast<int>(nnz / kLongRowEdges + 1);
    // one warp per destination, all of them resident at once while they fit (a row costs two dependent loads)
    const unsigned pg = static_cast<unsigned>(n_dst / 8 + 1 < kNumSM * 64 ? n_dst / 8 + 1 : kNumSM * 64);
    gat_dst_sum_rows<<<pg, 256, 0, st>>>(fwd_ptr, fwd_ptr_bytes, a.d_edge, d_a_dst, n_dst, nnz, heads, hshift, a.w.hdr,
                                         long_rows, max_long);
    float *piece_sums = reinterpret_cast<float *>(reinterpret_cast<char *>(workspace) + L.piece_sums);
    gat_dst_sum_pieces<<<kNumSM * 2, 256, 0, st>>>(fwd_ptr, fwd_ptr_bytes, a.d_edge, piece_sums, nnz, heads, hshift,
                                                   a.w.hdr, long_rows, max_long);
    gat_dst_sum_long<<<kNumSM, 256, 0, st>>>(fwd_ptr, fwd_ptr_bytes, piece_sums, d_a_dst, nnz, heads, hshift, a.w.hdr,
                                             long_rows, max_long);
    count_launches(3);
  }
  return check_launch("cxg_gat_fused_backward");
}

extern "C" int cxg_gat_fused_backward(const void *t_ptr, const void *t_idx, int ptr_bytes, int idx_bytes, const float *dy,
                                      const float *y, const float *x, const float *a_src, const float *a_dst,
                                      const float *row_max, const float *row_sum, float *dx, float *d_a_src,
                                      float *d_a_dst, int64_t n_src, int64_t n_dst, int64_t nnz, int heads, int c,
                                      float slope, const void *t_eid, const void *fwd_ptr, int fwd_ptr_bytes,
                                      void *workspace, size_t workspace_bytes, void *stream) {
  return cxg_gat_fused_backward_bias(t_ptr, t_idx, ptr_bytes, idx_bytes, dy, y, x, a_src, a_dst, row_max, row_sum, dx, d_a_src,
                                     d_a_dst, n_src, n_dst, nnz, heads, c, slope, t_eid, fwd_ptr, fwd_ptr_bytes, nullptr, workspace,
                                     workspace_bytes, stream);
}
