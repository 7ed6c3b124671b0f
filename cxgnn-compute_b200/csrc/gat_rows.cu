// The passes of a GAT layer over the rows of its nodes, beside the walks over the edges (gat_fused.cu): the gradient that
// reaches the transformed features through the two attention scores, together with those of the attention vectors, and
// the bias (with the mean over the heads). All are bound by memory.
#include "common.cuh"

namespace cxg {
namespace {

constexpr int kRowThreads = 256;
constexpr int kRowCtas = kNumSM * 4;  // at most as many partial sums as cxg_gat_att_grad_workspace_size has room for

template <int V>
__device__ __forceinline__ void load_v(float (&v)[V], const float *p) {
  if constexpr (V == 4) {
    const float4 t = *reinterpret_cast<const float4 *>(p);
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
  } else {
    v[0] = *p;
  }
}
template <int V>
__device__ __forceinline__ void store_v(float *p, const float (&v)[V]) {
  if constexpr (V == 4)
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else
    *p = v[0];
}

// dx[n, h, :] += g_src[n, h] * att_src[h, :] + g_dst[n, h] * att_dst[h, :] (the second for n < n_dst), and the block's part
// of sum_n g_src[n, h] * feat[n, h, :] and sum_n g_dst[n, h] * feat[n, h, :]. A thread keeps V columns and goes down the
// rows of the block, two rows in flight. One pass over feat and dx where the gradient of the scores was written, added to
// dx, and feat was read again for the attention vectors: 169,343 rows of 128 took 175 us, now 41.
template <int V>
__global__ void __launch_bounds__(kRowThreads) scores_backward_add(const float *feat, const float *g_src, const float *g_dst,
                                                                   const float *att_src, const float *att_dst, float *dx,
                                                                   float *part, int64_t n_src, int64_t n_dst, int heads, int c) {
  dependency_wait();
  __shared__ float sh[2][kRowThreads * V];
  const int width = heads * c, per_row = width / V;  // threads per row
  const int subs = per_row <= kRowThreads ? kRowThreads / per_row : 1;
  const int64_t per = (n_src + gridDim.x - 1) / gridDim.x;
  const int64_t first = blockIdx.x * per, last = min(n_src, first + per);
  for (int t0 = 0; t0 < per_row; t0 += kRowThreads) {
    const int sub = per_row <= kRowThreads ? threadIdx.x / per_row : 0;
    const int col = (t0 + (per_row <= kRowThreads ? threadIdx.x % per_row : threadIdx.x)) * V;
    const bool on = col < width && sub < subs;
    const int h = on ? col / c : 0;
    float as[V] = {}, ad[V] = {};
    if (on) {
      float ws[V], wd[V];
      load_v<V>(ws, att_src + col);
      load_v<V>(wd, att_dst + col);
      auto row = [&](const float (&f)[V], float (&d)[V], float gs, float gd) {
#pragma unroll
        for (int i = 0; i < V; ++i) {
          d[i] += fmaf(gd, wd[i], gs * ws[i]);
          as[i] = fmaf(gs, f[i], as[i]);
          ad[i] = fmaf(gd, f[i], ad[i]);
        }
      };
      constexpr int U = 4;
      for (int64_t r = first + sub; r < last; r += U * subs) {
        float f[U][V], d[U][V], gs[U], gd[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int64_t ru = r + u * subs;
          if (ru >= last) break;
          load_v<V>(f[u], feat + ru * width + col);
          load_v<V>(d[u], dx + ru * width + col);
          gs[u] = __ldg(g_src + ru * heads + h);
          gd[u] = ru < n_dst ? __ldg(g_dst + ru * heads + h) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int64_t ru = r + u * subs;
          if (ru >= last) break;
          row(f[u], d[u], gs[u], gd[u]);
          store_v<V>(dx + ru * width + col, d[u]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < V; ++i) sh[0][threadIdx.x * V + i] = as[i], sh[1][threadIdx.x * V + i] = ad[i];
    __syncthreads();
    if (on && sub == 0) {
      for (int u = 1; u < subs; ++u)
#pragma unroll
        for (int i = 0; i < V; ++i) {
          as[i] += sh[0][u * width + threadIdx.x * V + i];
          ad[i] += sh[1][u * width + threadIdx.x * V + i];
        }
      store_v<V>(part + static_cast<int64_t>(blockIdx.x) * 2 * width + col, as);
      store_v<V>(part + (static_cast<int64_t>(blockIdx.x) * 2 + 1) * width + col, ad);
    }
    __syncthreads();
  }
}

// The blocks' parts in a fixed order: warp w of a block adds those of blocks w, w + 32, ... for 32 columns, the 32 sums
// are added in order. (A warp per column, 32 blocks a step, read 4 bytes per sector: 15 us for 1184 blocks of 128 columns.)
constexpr int kJoinThreads = 1024;
__global__ void __launch_bounds__(kJoinThreads) att_grad_join(const float *part, float *grad_src, float *grad_dst, int n_part,
                                                             int width) {
  dependency_wait();
  __shared__ float sh[kJoinThreads / 32][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + lane;  // of the 2 * width columns of a part
  float s = 0.f;
  if (col < 2 * width) {
    const float *p = part + col;
    const int64_t step = 2ll * width;
    int b = warp;
    for (; b + 96 < n_part; b += 128) {
      float v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = p[(b + 32 * u) * step];
#pragma unroll
      for (int u = 0; u < 4; ++u) s += v[u];
    }
    for (; b < n_part; b += 32) s += p[b * step];
  }
  sh[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && col < 2 * width) {
    for (int w = 1; w < kJoinThreads / 32; ++w) s += sh[w][lane];
    (col < width ? grad_src : grad_dst)[col < width ? col : col - width] = s;
  }
}

// out[n, :] = mean over the heads of x[n, h, :] + bias, V columns per thread. (torch: a reduction and a broadcast addition,
// 77 us for 169,343 rows of 4 x 47, now 49; the addition alone 60 us for rows of 128, now 26.)
template <int V, typename I>  // I: 32-bit positions wherever they suffice, the divisions are half of the work
__global__ void __launch_bounds__(kRowThreads, 6) head_mean_bias(const float *x, const float *bias, float *out, int64_t n, int heads,
                                                              int c) {
  dependency_wait();
  const I per_row = c / V, total = static_cast<I>(n) * per_row, step = static_cast<I>(gridDim.x) * kRowThreads;
  constexpr int U = V == 4 ? 2 : 4;
  for (int64_t i0 = blockIdx.x * static_cast<int64_t>(kRowThreads) + threadIdx.x; i0 < total; i0 += U * static_cast<int64_t>(step)) {
    float s[U][V];
    int64_t at[U];
    int col[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const I i = static_cast<I>(i0) + u * step, row = i / per_row;
      col[u] = static_cast<int>(i - row * per_row) * V;
      at[u] = i0 + u * static_cast<int64_t>(step) < total ? static_cast<int64_t>(row) * heads * c + col[u] : -1;
      if (at[u] >= 0) load_v<V>(s[u], x + at[u]);
    }
    for (int h = 1; h < heads; ++h) {
      float v[U][V];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (at[u] >= 0) load_v<V>(v[u], x + at[u] + static_cast<int64_t>(h) * c);
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int k = 0; k < V; ++k) s[u][k] += v[u][k];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (at[u] < 0) break;
      float b[V] = {};
      if (bias != nullptr) load_v<V>(b, bias + col[u]);
#pragma unroll
      for (int k = 0; k < V; ++k) s[u][k] = (heads > 1 ? s[u][k] * (1.f / heads) : s[u][k]) + b[k];
      store_v<V>(out + (i0 + u * static_cast<int64_t>(step)) * V, s[u]);
    }
  }
}

// Weights [heads * c, k] and attention vectors [heads, c] with the heads padded to cp columns of zeros, so that every head of
// the transformed features starts on a 16-byte boundary.
__global__ void __launch_bounds__(kRowThreads) pad_heads(const float *w, const float *att_src, const float *att_dst, float *wp,
                                                         float *src_p, float *dst_p, int heads, int c, int cp, int k) {
  dependency_wait();
  const int i = blockIdx.x * kRowThreads + threadIdx.x, rows = heads * cp;
  if (i >= rows * (k + 2)) return;
  const int row = i < rows * k ? i / k : (i - rows * k) % rows, at = row % cp, from = row / cp * c + at;
  if (i < rows * k)
    wp[i] = at < c ? w[static_cast<int64_t>(from) * k + (i - row * k)] : 0.f;
  else if (i < rows * (k + 1))
    src_p[row] = at < c ? att_src[from] : 0.f;
  else
    dst_p[row] = at < c ? att_dst[from] : 0.f;
}

// Rows of padded heads to the layer's output: the heads' mean [n, c], or the heads side by side [n, heads * c], plus the bias.
// A thread takes a vector of one column group: all its heads' loads are in flight.
template <bool JOIN>
__global__ void __launch_bounds__(kRowThreads) unpad_heads(const float *x, const float *bias, float *out, int64_t n, int heads, int c,
                                                           int cp) {
  dependency_wait();
  const int vecs = cp / 4, per_row = JOIN ? heads * vecs : vecs;
  const int64_t total = n * per_row, step = static_cast<int64_t>(gridDim.x) * kRowThreads;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(kRowThreads) + threadIdx.x; i < total; i += step) {
    const int64_t row = total < (1ll << 31) ? static_cast<int>(i) / per_row : i / per_row;
    const int rest = static_cast<int>(i - row * per_row), h = JOIN ? rest / vecs : 0, col = (rest - h * vecs) * 4;
    float s[4];
    load_v<4>(s, x + (row * heads + h) * cp + col);
    if (!JOIN) {
#pragma unroll 4
      for (int j = 1; j < heads; ++j) {
        float v[4];
        load_v<4>(v, x + (row * heads + j) * cp + col);
#pragma unroll
        for (int q = 0; q < 4; ++q) s[q] += v[q];
      }
    }
    float *o = out + (JOIN ? (row * heads + h) * c : row * c) + col;
    const float *b = bias != nullptr ? bias + (JOIN ? h * c : 0) + col : nullptr;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (col + q < c) o[q] = (JOIN || heads == 1 ? s[q] : s[q] * (1.f / heads)) + (b != nullptr ? b[q] : 0.f);
  }
}

bool vectors(int c, const void *a, const void *b, const void *d) {
  return c % 4 == 0 &&
         ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(d)) % 16) == 0;
}

}  // namespace
}  // namespace cxg

using namespace cxg;

extern "C" int cxg_gat_scores_backward_add(const float *feat, const float *g_src, const float *g_dst, const float *att_src,
                                           const float *att_dst, float *dx, float *grad_att_src, float *grad_att_dst,
                                           int64_t n_src, int64_t n_dst, int heads, int c, void *workspace,
                                           size_t workspace_bytes, void *stream) {
  CXG_REQUIRE(n_src >= 0 && n_dst >= 0 && n_dst <= n_src && heads > 0 && c > 0, CXG_EINVAL,
              "cxg_gat_scores_backward_add: bad sizes");
  CXG_REQUIRE(att_src && att_dst && grad_att_src && grad_att_dst, CXG_ENULL, "cxg_gat_scores_backward_add: NULL argument");
  CXG_REQUIRE(n_src == 0 || (feat && g_src && dx && (g_dst || n_dst == 0)), CXG_ENULL,
              "cxg_gat_scores_backward_add: NULL argument");
  const int width = heads * c;
  size_t need = 0;
  cxg_gat_att_grad_workspace_size(heads, c, &need);
  CXG_REQUIRE(workspace != nullptr && workspace_bytes >= need && need >= static_cast<size_t>(kRowCtas) * 2 * width * sizeof(float),
              CXG_EWORKSPACE, "cxg_gat_scores_backward_add: workspace %zu bytes, need %zu", workspace_bytes, need);
  cudaStream_t st = as_stream(stream);
  float *part = static_cast<float *>(workspace);
  // at least 32 rows per block, so that a small call does not add up more parts than rows
  int64_t ctas = (n_src + 31) / 32;
  if (ctas > kRowCtas) ctas = kRowCtas;
  if (ctas < 1) ctas = 1;
  const unsigned grid = static_cast<unsigned>(ctas);
  if (vectors(c, feat, dx, workspace) && vectors(c, att_src, att_dst, nullptr))
    launch_dependent(scores_backward_add<4>, grid, kRowThreads, 0, st, feat, g_src, g_dst, att_src, att_dst, dx, part, n_src, n_dst, heads, c);
  else
    launch_dependent(scores_backward_add<1>, grid, kRowThreads, 0, st, feat, g_src, g_dst, att_src, att_dst, dx, part, n_src, n_dst, heads, c);
  launch_dependent(att_grad_join, (2 * width + 31) / 32, kJoinThreads, 0, st, part, grad_att_src, grad_att_dst, static_cast<int>(grid), width);
  count_launches(2);
  return check_launch("cxg_gat_scores_backward_add");
}

extern "C" int cxg_head_mean_bias(const float *x, const float *bias, float *out, int64_t n, int heads, int c, void *stream) {
  CXG_REQUIRE(n >= 0 && heads > 0 && c > 0, CXG_EINVAL, "cxg_head_mean_bias: bad sizes");
  if (n == 0) return CXG_OK;
  CXG_REQUIRE(x && out, CXG_ENULL, "cxg_head_mean_bias: NULL argument");
  const bool v4 = vectors(c, x, out, bias);
  const int64_t each = (v4 ? 2 : 4) * kRowThreads, blocks = (n * (c / (v4 ? 4 : 1)) + each - 1) / each;
  const unsigned grid = static_cast<unsigned>(blocks < kNumSM * 32 ? blocks : kNumSM * 32);
  const bool narrow = n * c < (1ll << 30);
  cudaStream_t st = as_stream(stream);
  if (v4 && narrow)
    launch_dependent(head_mean_bias<4, int32_t>, grid, kRowThreads, 0, st, x, bias, out, n, heads, c);
  else if (v4)
    launch_dependent(head_mean_bias<4, int64_t>, grid, kRowThreads, 0, st, x, bias, out, n, heads, c);
  else if (narrow)
    launch_dependent(head_mean_bias<1, int32_t>, grid, kRowThreads, 0, st, x, bias, out, n, heads, c);
  else
    launch_dependent(head_mean_bias<1, int64_t>, grid, kRowThreads, 0, st, x, bias, out, n, heads, c);
  count_launches(1);
  return check_launch("cxg_head_mean_bias");
}

extern "C" int cxg_gat_pad_heads(const float *w, const float *att_src, const float *att_dst, float *w_padded, float *att_src_padded,
                                 float *att_dst_padded, int heads, int c, int c_padded, int k, void *stream) {
  CXG_REQUIRE(heads > 0 && c > 0 && c_padded >= c && k > 0 && static_cast<int64_t>(heads) * c_padded * (k + 2) < (1ll << 30),
              CXG_EINVAL, "cxg_gat_pad_heads: bad sizes");
  CXG_REQUIRE(w && att_src && att_dst && w_padded && att_src_padded && att_dst_padded, CXG_ENULL, "cxg_gat_pad_heads: NULL argument");
  const int total = heads * c_padded * (k + 2);
  launch_dependent(pad_heads, (total + kRowThreads - 1) / kRowThreads, kRowThreads, 0, as_stream(stream), w, att_src, att_dst, w_padded,
                   att_src_padded, att_dst_padded, heads, c, c_padded, k);
  count_launches(1);
  return check_launch("cxg_gat_pad_heads");
}

extern "C" int cxg_gat_unpad_heads(const float *x, const float *bias, float *out, int64_t n, int heads, int c, int c_padded, int join,
                                   void *stream) {
  CXG_REQUIRE(n >= 0 && heads > 0 && c > 0 && c_padded >= c && c_padded % 4 == 0, CXG_EINVAL, "cxg_gat_unpad_heads: bad sizes");
  if (n == 0) return CXG_OK;
  CXG_REQUIRE(x && out, CXG_ENULL, "cxg_gat_unpad_heads: NULL argument");
  CXG_REQUIRE(reinterpret_cast<uintptr_t>(x) % 16 == 0, CXG_EINVAL, "cxg_gat_unpad_heads: x must be 16-byte aligned");
  const int64_t blocks = (n * (join ? heads : 1) * (c_padded / 4) + kRowThreads - 1) / kRowThreads;
  const unsigned grid = static_cast<unsigned>(blocks < kNumSM * 64 ? blocks : kNumSM * 64);
  launch_dependent(join ? unpad_heads<true> : unpad_heads<false>, grid, kRowThreads, 0, as_stream(stream), x, bias, out, n, heads, c, c_padded);
  count_launches(1);
  return check_launch("cxg_gat_unpad_heads");
}
