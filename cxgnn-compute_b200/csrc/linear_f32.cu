// The linear transform of a layer in fp32 on the tensor cores: C[m, n] = A[m, :] . B[n, :] (+ bias[n]) (+ add[m, n]).
//
// Every fp32 operand is cut into three bf16 terms, v = h + m + l exactly (8 + 8 + 8 significant bits), and six of the nine
// products are summed: h.h into one accumulator, h.m, m.h, m.m, h.l, l.h (all below 2^-8 of it) into a second one; what is
// left out is below 2^-26. bf16 products are exact in the fp32 accumulator, so what remains is the tensor core's cut at
// every instruction, one per 16 columns of K into the large sum, and the result is as close to the exact one as that of an
// fp32 multiply-add chain (K = 128: 1.2e-7 of the result against 2.0e-7; two TF32 terms gave 3.2e-7, with twice as many
// instructions per K).
//
// A persistent CTA per SM owns NT columns of C (B's three terms for them stay in shared memory) and a range of row tiles of
// 128. The pipeline unit is 128 rows x 32 columns of A: the bulk tensor copy unit brings it in as fp32 (128-byte swizzle),
// eight converter warps write its three bf16 terms (64-byte swizzle), one thread issues the MMAs, four warps drain the
// accumulators. Raw and converted units have rings of their own, so the next unit lands while one is converted and one is
// multiplied. Two accumulator buffers of 2 * NT columns, so a tile is stored while the next one is summed.
//
// The five instructions per 16 columns of K read 20 KB of A and 24 KB of B from shared memory at NT = 128, 344 cycles at its
// 128 bytes a cycle, against 384 for the products: the operands bound the kernel as much as the tensor pipe, and memory
// traffic (173 MB for 169,343 rows of 128 -> 128, 26 us) less.
// Measured, cold, against the fp32 library GEMM: 169,343 rows 128 -> 128 49 us (132), 1.94 M rows 128 -> 64 293 us (734),
// 50,952 rows 256 -> 256 70 us (145).
//
// A call of few rows is a chain of latencies: the launch, B's terms, the units of one tile. So it takes blocks of as few as
// 16 columns (half as much of B to convert for each), the first units of A are requested before B is converted, and the
// blocks become resident while the kernel in front drains. The six products of a sampled SAGE batch of 32 seeds
// (100 -> 256 -> 256 -> 47, 32 to 4,800 rows) take 60 us instead of 75, the batch's inference 292 us instead of 306.
//
// Every wait is bounded, as in typed_mm.cu: a role that waits too long raises a CTA-wide flag and the status word, all roles
// leave their loops, the copies in flight are waited for (bounded as well), and the tensor memory is released.
#include "common.cuh"
#include "tensor_core.cuh"

namespace cxg {
namespace {

using namespace tc;

constexpr int kTileM = 128;
constexpr int kSpan = 32;                       // columns of A per unit
constexpr int kRawBytes = kTileM * kSpan * 4;   // a unit as it arrives
constexpr int kTermBytes = kTileM * kSpan * 2;  // one of its three terms
constexpr int kConvWarps = 8, kEpiWarps = 4;
constexpr int kMmaWarp = kEpiWarps, kLoadWarp = kMmaWarp + 1, kFirstConv = kLoadWarp + 1;
constexpr int kThreads = 32 * (kFirstConv + kConvWarps);
constexpr int kMaxStages = 4, kMinStages = 3;
constexpr int kSmemBudget = 225 * 1024;  // without the alignment of the first unit
constexpr float kMostF32 = 3.402823466e38f;   // the largest finite value
constexpr float kMostBf16 = 3.389531389e38f;  // and that of bf16

__device__ int32_t linear_status;  // set when a bounded wait ran out, cleared by cxg_linear_f32_status

struct LinArgs {
  const float *a, *b, *bias, *add;
  float *c;
  int64_t m;
  int k, n;
  int nt;         // columns of C per CTA
  int n_blocks;   // CTAs side by side for all columns
  int b_rows_k;   // B is [K][N] instead of [N][K]
  int stages;
  int acc_cols;   // tensor-memory columns of one accumulator buffer
  int test_stall; // test hook: the converters never hand over their first unit, so the waits for it run out
  long long wait_cycles;
};

struct LinBarriers {
  uint64_t raw_full[kMaxStages], raw_empty[kMaxStages];    // copy unit -> converters (bytes), converters -> loader
  uint64_t term_full[kMaxStages], term_empty[kMaxStages];  // converters -> MMA, MMA (commit) -> converters
  uint64_t acc_full[2], acc_empty[2];                      // MMA (commit) -> epilogue, epilogue -> MMA
};

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&t);
}

// Two values into their three bf16 terms, packed; every subtraction is exact.
__device__ __forceinline__ void split3(float a, float b, uint32_t &h, uint32_t &m, uint32_t &l) {
  h = pack_bf16(a, b);
  a -= __uint_as_float(h << 16), b -= __uint_as_float(h & 0xffff0000u);
  m = pack_bf16(a, b);
  a -= __uint_as_float(m << 16), b -= __uint_as_float(m & 0xffff0000u);
  l = pack_bf16(a, b);
}

// A[row, :] . B[col, :] as an fp32 multiply-add chain. The products of the terms cannot give an element that an infinity or
// a value above bf16's range takes part in: Inf - Inf is no second term, and an infinity times the other operand's lower
// terms, zeros or of either sign, is no third. Whatever comes out of the tensor core as an infinity or NaN is taken from
// here. A chain that has become NaN stays it, so a matrix full of them ends after four steps.
__device__ __noinline__ float exact_chain(const LinArgs &a, int64_t row, int col) {
  const float4 *x = reinterpret_cast<const float4 *>(a.a + row * a.k);
  const float *w = a.b + (a.b_rows_k ? col : static_cast<int64_t>(col) * a.k);
  const int64_t step = a.b_rows_k ? a.n : 1;
  float s = 0.f;
  for (int k = 0; k < a.k && s == s; k += 4, w += 4 * step) {
    const float4 v = x[k / 4];
    s = fmaf(v.x, w[0], s), s = fmaf(v.y, w[step], s), s = fmaf(v.z, w[2 * step], s), s = fmaf(v.w, w[3 * step], s);
  }
  return s;
}

// 8 bytes (four columns from 4 * c4 on) of a row of a tile of bf16 rows of 64 bytes, 64-byte swizzle
__device__ __forceinline__ uint32_t term_offset(int row, int c4) { return swizzled(row, c4 >> 1, 2, 0) + (c4 & 1) * 8; }

__global__ void __launch_bounds__(kThreads, 1) linear_tc(const __grid_constant__ LinArgs a,
                                                         const __grid_constant__ CUtensorMap tmap_a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) LinBarriers bars;
  __shared__ __align__(16) float s_bias[128];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_slot;
  volatile int *abort_flag = &abort_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int S = a.stages;
  const int spans = (a.k + kSpan - 1) / kSpan;
  uint8_t *raw = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
  uint8_t *terms = raw + S * kRawBytes;
  uint8_t *smem_b = terms + S * 3 * kTermBytes;
  const uint32_t term_b = a.nt * 64, span_b = 3 * term_b;  // bytes of one term of a span of B, and of all three

  const int n0 = static_cast<int>(blockIdx.x % a.n_blocks) * a.nt;
  const int64_t n_tiles = (a.m + kTileM - 1) / kTileM;
  const int64_t part = blockIdx.x / a.n_blocks, parts = gridDim.x / a.n_blocks;
  const int64_t tile_lo = n_tiles * part / parts, tile_hi = n_tiles * (part + 1) / parts;

  auto load_unit = [&](int s, int64_t tile, int sp) {
    const uint32_t bar = smem_addr(&bars.raw_full[s]);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kRawBytes) : "memory");
    tma_load_2d(smem_addr(raw + s * kRawBytes), &tmap_a, sp * kSpan, static_cast<int>(tile * kTileM), bar);
  };
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_slot)),
                 "r"(static_cast<uint32_t>(2 * a.acc_cols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  dependency_wait();  // A, B and what is added may come from the kernel in front, and C may be read by it
  if (warp == kLoadWarp && lane == 0) {
    abort_slot = 0;
    auto init = [&](uint64_t *bar, uint32_t count) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    };
    for (int s = 0; s < kMaxStages; ++s) {
      init(&bars.raw_full[s], 1);
      init(&bars.raw_empty[s], 32 * kConvWarps);
      init(&bars.term_full[s], 32 * kConvWarps);
      init(&bars.term_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      init(&bars.acc_full[b], 1);
      init(&bars.acc_empty[b], 32 * kEpiWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    // the first units are on their way while B is converted
    int64_t tile = tile_lo;
    for (int s = 0, sp = 0; s < S && tile < tile_hi; ++s) {
      load_unit(s, tile, sp);
      if (++sp == spans) sp = 0, ++tile;
    }
  }
  // the three terms of this CTA's rows of B; rows behind N and columns behind K are zeros
  bool b_infinite = false;  // B has a value that bf16 does not reach (or that the sum of four takes for one)
  {
    const int c4s = spans * (kSpan / 4), total = a.nt * c4s;
    constexpr int kAhead = 4;  // requested at once: this is what a call of few rows spends its time on
    for (int i0 = tid; i0 < total; i0 += kAhead * kThreads) {
      float4 v[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int i = i0 + u * kThreads;
        const int row = a.b_rows_k ? i % a.nt : i / c4s, c4 = a.b_rows_k ? i / a.nt : i % c4s;
        const int n = n0 + row, k = 4 * c4;
        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < total && n < a.n && k < a.k) {  // K is a multiple of four
          if (a.b_rows_k) {
            const float *p = a.b + static_cast<int64_t>(k) * a.n + n;
            v[u] = make_float4(p[0], p[a.n], p[2 * static_cast<int64_t>(a.n)], p[3 * static_cast<int64_t>(a.n)]);
          } else {
            v[u] = *reinterpret_cast<const float4 *>(a.b + static_cast<int64_t>(n) * a.k + k);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int i = i0 + u * kThreads;
        if (i >= total) break;
        const int row = a.b_rows_k ? i % a.nt : i / c4s, c4 = a.b_rows_k ? i / a.nt : i % c4s;
        uint2 h, m, l;
        b_infinite |= !((fabsf(v[u].x) + fabsf(v[u].y)) + (fabsf(v[u].z) + fabsf(v[u].w)) <= kMostBf16);
        split3(v[u].x, v[u].y, h.x, m.x, l.x);
        split3(v[u].z, v[u].w, h.y, m.y, l.y);
        uint8_t *d = smem_b + (c4 / (kSpan / 4)) * span_b + term_offset(row, c4 % (kSpan / 4));
        *reinterpret_cast<uint2 *>(d) = h;
        *reinterpret_cast<uint2 *>(d + term_b) = m;
        *reinterpret_cast<uint2 *>(d + 2 * term_b) = l;
      }
    }
    for (int i = tid; i < a.nt; i += kThreads) s_bias[i] = a.bias != nullptr && n0 + i < a.n ? a.bias[n0 + i] : 0.f;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor core reads B through the async proxy
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  b_infinite = __syncthreads_or(b_infinite) != 0;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_d = tmem_base_slot;
  auto wait = [&](uint64_t *bar, int64_t phase) {
    return wait_bar(bar, static_cast<uint32_t>(phase & 1), abort_flag, &linear_status, a.wait_cycles);
  };

  // the same for a whole warp that goes on together
  auto wait_all = [&](uint64_t *bar, int64_t phase) { return __all_sync(0xffffffffu, wait(bar, phase)) != 0; };

  if (warp == kLoadWarp) {
    if (lane == 0) {
      Ring ring(S);
      bool alive = true;
      for (int64_t tile = tile_lo; tile < tile_hi && alive; ++tile)
        for (int sp = 0; sp < spans; ++sp) {
          const int s = ring.stage;
          if (ring.reused()) {  // the first round has been requested in front of the loop
            if (!(alive = wait(&bars.raw_empty[s], ring.emptied()))) break;
            load_unit(s, tile, sp);
          }
          ring.next();
        }
      // the copies in flight land before the block ends, whatever became of their readers
      for (int j = 0; j < S; ++j) {
        uint32_t parity;
        if (!ring.last(j, &parity)) continue;
        const uint32_t bar = smem_addr(&bars.raw_full[j]);
        const long long t0 = clock64();
        while (!mbar_try_wait(bar, parity) && clock64() - t0 <= a.wait_cycles) {
        }
      }
    }
    __syncwarp();
  } else if (warp >= kFirstConv) {
    const int ct = tid - 32 * kFirstConv;
    constexpr int kPer = kTileM * 8 / (32 * kConvWarps);  // 16-byte chunks per thread
    Ring ring(S);
    bool alive = true;
    for (int64_t tile = tile_lo; tile < tile_hi && alive; ++tile)
      for (int sp = 0; sp < spans; ++sp, ring.next()) {
        const int s = ring.stage;
        if (!(alive = wait(&bars.raw_full[s], ring.filled()))) break;
        const float4 *src = reinterpret_cast<const float4 *>(raw + s * kRawBytes);
        float4 v[kPer];
#pragma unroll
        for (int u = 0; u < kPer; ++u) v[u] = src[ct + u * 32 * kConvWarps];
        if (ring.reused() && !(alive = wait(&bars.term_empty[s], ring.emptied()))) break;
        uint8_t *dst = terms + s * 3 * kTermBytes;
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
          const int i = ct + u * 32 * kConvWarps, row = i >> 3, c4 = (i & 7) ^ (row & 7);
          uint2 h, m, l;
          split3(v[u].x, v[u].y, h.x, m.x, l.x);
          split3(v[u].z, v[u].w, h.y, m.y, l.y);
          uint8_t *d = dst + term_offset(row, c4);
          *reinterpret_cast<uint2 *>(d) = h;
          *reinterpret_cast<uint2 *>(d + kTermBytes) = m;
          *reinterpret_cast<uint2 *>(d + 2 * kTermBytes) = l;
        }
        mbar_arrive(&bars.raw_empty[s]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (!(a.test_stall && tile == tile_lo && sp == 0)) mbar_arrive(&bars.term_full[s]);
      }
  } else if (warp == kMmaWarp) {
    const uint32_t idesc = make_idesc(1, kTileM, a.nt), idesc_wide = make_idesc(1, kTileM, 2 * a.nt);
    const uint64_t desc = desc_base(2);
    const uint32_t b0 = smem_addr(smem_b);
    Ring ring(S);
    int64_t tile_it = 0;
    bool alive = true;
    for (int64_t tile = tile_lo; tile < tile_hi && alive; ++tile, ++tile_it) {
      const int buf = static_cast<int>(tile_it & 1);
      const uint32_t d0 = tmem_d + buf * a.acc_cols, d1 = d0 + a.nt;  // h.h, and the small products
      if (tile_it >= 2 && !(alive = wait_all(&bars.acc_empty[buf], (tile_it >> 1) - 1))) break;
      for (int sp = 0; sp < spans; ++sp, ring.next()) {
        const int s = ring.stage;
        if (!(alive = wait_all(&bars.term_full[s], ring.filled()))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a0 = smem_addr(terms + s * 3 * kTermBytes), bs = b0 + sp * span_b;
        const int steps = a.k - sp * kSpan > 16 ? 2 : 1;  // 16 columns of K each
        for (int j = 0; j < steps; ++j) {
          const uint64_t ah = make_desc(desc, a0 + j * 32), am = make_desc(desc, a0 + kTermBytes + j * 32),
                         al = make_desc(desc, a0 + 2 * kTermBytes + j * 32);
          const uint64_t bh = make_desc(desc, bs + j * 32), bm = make_desc(desc, bs + term_b + j * 32),
                         bl = make_desc(desc, bs + 2 * term_b + j * 32);
          mma_ss<false>(d0, ah, bh, idesc_wide, sp > 0 || j > 0);  // h x [h | m]
          mma_ss<false>(d1, ah, bl, idesc, 1u);
          mma_ss<false>(d1, am, bh, idesc, 1u);
          mma_ss<false>(d1, am, bm, idesc, 1u);
          mma_ss<false>(d1, al, bh, idesc, 1u);
        }
        commit_to(&bars.term_empty[s]);
      }
      if (!alive) break;
      commit_to(&bars.acc_full[buf]);
    }
  } else {
    // epilogue: warp w owns the accumulator lanes 32 * w .. + 31 = rows of the tile
    const bool odd = lane & 1, quads = a.n % 4 == 0;
    const int cols = a.n - n0 < a.nt ? a.n - n0 : a.nt;
    int64_t tile_it = 0;
    bool alive = true;
    for (int64_t tile = tile_lo; tile < tile_hi && alive; ++tile, ++tile_it) {
      const int buf = static_cast<int>(tile_it & 1);
      if (!(alive = wait(&bars.acc_full[buf], tile_it >> 1))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t taddr = tmem_d + (static_cast<uint32_t>(warp * 32) << 16) + buf * a.acc_cols;
      const int64_t row = tile * kTileM + warp * 32 + lane;
      // two adjacent lanes trade 16-byte quads, so that one store of the pair writes a whole 32-byte sector
      const int64_t even = (row & ~1ll) * a.n + n0;
      const bool ok_a = (row & ~1ll) < a.m, ok_b = (row | 1) < a.m;
      // an infinity or NaN in a row of A shows in every column of the row, the first one included. (In the loop below the
      // calls cost the ordinary tiles 12 %, here one column read ahead.)
      uint32_t first[2];
      tmem_ld1(first, taddr);
      tmem_ld1(first + 1, taddr + a.nt);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (b_infinite || !__all_sync(0xffffffffu, fabsf(__uint_as_float(first[0]) + __uint_as_float(first[1])) <= kMostF32)) {
        for (int c0 = 0; c0 < a.nt; c0 += 16) {
          uint32_t v[16], sm[16];
          tmem_ld16(v, taddr + c0);
          tmem_ld16(sm, taddr + a.nt + c0);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (row < a.m) {
            const int64_t at = row * a.n + n0 + c0;
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (c0 + i < cols) {
                float f = __uint_as_float(v[i]) + __uint_as_float(sm[i]);
                if (!(fabsf(f) <= kMostF32)) f = exact_chain(a, row, n0 + c0 + i);
                f += s_bias[c0 + i];
                a.c[at + i] = a.add != nullptr ? f + a.add[at + i] : f;
              }
          }
          __syncwarp();
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        mbar_arrive(&bars.acc_empty[buf]);
        continue;
      }
      for (int c0 = 0; c0 < a.nt; c0 += 16) {
        // what is to be added: requested before the accumulator is read
        float4 pa[2], pb[2];
        if (quads && a.add != nullptr) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int col = c0 + 8 * h + (odd ? 4 : 0);
            if (col < cols && ok_a) pa[h] = *reinterpret_cast<const float4 *>(a.add + even + col);
            if (col < cols && ok_b) pb[h] = *reinterpret_cast<const float4 *>(a.add + even + a.n + col);
          }
        }
        uint32_t v[16], sm[16];
        tmem_ld16(v, taddr + c0);
        tmem_ld16(sm, taddr + a.nt + c0);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + 16 >= a.nt) {  // the accumulator buffer is in registers: give it back to the MMA thread
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          mbar_arrive(&bars.acc_empty[buf]);
        }
        float f[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) f[i] = (__uint_as_float(v[i]) + __uint_as_float(sm[i])) + s_bias[c0 + i];
        if (quads) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float4 q[2];
            q[0] = make_float4(f[8 * h], f[8 * h + 1], f[8 * h + 2], f[8 * h + 3]);
            q[1] = make_float4(f[8 * h + 4], f[8 * h + 5], f[8 * h + 6], f[8 * h + 7]);
            const float4 keep = odd ? q[1] : q[0], send = odd ? q[0] : q[1];
            float4 got;
            got.x = __shfl_xor_sync(0xffffffffu, send.x, 1);
            got.y = __shfl_xor_sync(0xffffffffu, send.y, 1);
            got.z = __shfl_xor_sync(0xffffffffu, send.z, 1);
            got.w = __shfl_xor_sync(0xffffffffu, send.w, 1);
            const int col = c0 + 8 * h + (odd ? 4 : 0);
            // quad `col` of the even lane's row, then of the odd lane's
            float4 va = odd ? got : keep, vb = odd ? keep : got;
            if (a.add != nullptr) {
              va.x += pa[h].x, va.y += pa[h].y, va.z += pa[h].z, va.w += pa[h].w;
              vb.x += pb[h].x, vb.y += pb[h].y, vb.z += pb[h].z, vb.w += pb[h].w;
            }
            if (col < cols) {
              if (ok_a) *reinterpret_cast<float4 *>(a.c + even + col) = va;
              if (ok_b) *reinterpret_cast<float4 *>(a.c + even + a.n + col) = vb;
            }
          }
        } else if (row < a.m) {
          const int64_t at = row * a.n + n0 + c0;
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (c0 + i < cols) a.c[at + i] = f[i] + (a.add != nullptr ? a.add[at + i] : 0.f);
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d),
                 "r"(static_cast<uint32_t>(2 * a.acc_cols))
                 : "memory");
  }
}

// Columns of C per CTA: as few blocks side by side as B's terms for a block fit next to three stages (every block converts
// all of A again), then more of them while all tiles together leave half of the SMs idle, down to the 16 columns of one
// instruction. 0: K is too large.
int columns_per_block(int64_t m, int k, int n) {
  const int spans = (k + kSpan - 1) / kSpan;
  const int room = (kSmemBudget - kMinStages * (kRawBytes + 3 * kTermBytes)) / (spans * 3 * 64);
  const int most = room >= 128 ? 128 : room / 16 * 16;
  if (most < 16) return 0;
  int64_t blocks = (n + most - 1) / most;
  const int64_t tiles = (m + kTileM - 1) / kTileM;
  while (tiles * blocks * 2 <= kNumSM && n > blocks * 16) blocks *= 2;
  return static_cast<int>(((n + blocks - 1) / blocks + 15) / 16 * 16);
}

}  // namespace
}  // namespace cxg

using namespace cxg;

extern "C" int cxg_linear_f32_supported(int64_t m, int k, int n) {
  return m > 0 && m < (1ll << 31) - 128 && k > 0 && k % 4 == 0 && n > 0 && n <= 128 * 64 && columns_per_block(m, k, n) > 0;
}

extern "C" int cxg_linear_f32(const float *a, const float *b, const float *bias, const float *add, float *c, int64_t m, int k,
                              int n, int b_rows_k, void *stream) {
  return cxg_linear_f32_ex(a, b, bias, add, c, m, k, n, b_rows_k ? CXG_LINEAR_B_ROWS_K : 0u, stream);
}

extern "C" int cxg_linear_f32_ex(const float *a, const float *b, const float *bias, const float *add, float *c, int64_t m, int k,
                                 int n, uint32_t flags, void *stream) {
  CXG_REQUIRE(m >= 0 && k > 0 && n > 0, CXG_EINVAL, "cxg_linear_f32: bad sizes");
  if (m == 0) return CXG_OK;
  CXG_REQUIRE(a && b && c, CXG_ENULL, "cxg_linear_f32: NULL argument");
  CXG_REQUIRE(cxg_linear_f32_supported(m, k, n), CXG_EUNSUPPORTED,
              "cxg_linear_f32: K = %d must be a multiple of 4 of which 16 rows fit in shared memory", k);
  CXG_REQUIRE((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
               reinterpret_cast<uintptr_t>(add)) % 16 == 0,
              CXG_EINVAL, "cxg_linear_f32: A, B, C and add must be 16-byte aligned");
  LinArgs t;
  t.a = a, t.b = b, t.bias = bias, t.add = add, t.c = c;
  t.m = m, t.k = k, t.n = n;
  t.nt = columns_per_block(m, k, n);
  t.n_blocks = (n + t.nt - 1) / t.nt;
  t.b_rows_k = (flags & CXG_LINEAR_B_ROWS_K) ? 1 : 0;
  t.test_stall = (flags & CXG_LINEAR_TEST_STALL) ? 1 : 0;
  t.acc_cols = 32;
  while (t.acc_cols < 2 * t.nt) t.acc_cols *= 2;
  t.wait_cycles = wait_limit_cycles();
  const int b_bytes = t.nt * ((k + kSpan - 1) / kSpan) * 3 * 64;
  const int unit = kRawBytes + 3 * kTermBytes;
  t.stages = (kSmemBudget - b_bytes) / unit;
  if (t.stages > kMaxStages) t.stages = kMaxStages;
  const int smem = 1024 + t.stages * unit + b_bytes;
  const int64_t tiles = (m + kTileM - 1) / kTileM;
  int64_t groups = t.n_blocks < kNumSM ? kNumSM / t.n_blocks : 1;
  if (groups > tiles) groups = tiles;
  const cudaError_t e = cudaFuncSetAttribute(linear_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return set_error(CXG_ECUDA, "cxg_linear_f32: %s", cudaGetErrorString(e));
  // behind a call of the runtime, which gives a thread that has not used the device yet its context
  CUtensorMap map;
  CXG_REQUIRE(encode_a_map(&map, a, m, k, 4, kTileM), CXG_ECUDA, "cxg_linear_f32: no tensor map for A");
  const unsigned grid = static_cast<unsigned>(groups * t.n_blocks);
  if (launch_dependent(linear_tc, grid, kThreads, static_cast<size_t>(smem), as_stream(stream), t, map) == cudaSuccess) count_launches(1);
  return check_launch("cxg_linear_f32");
}

extern "C" int cxg_linear_f32_status(void *stream) {
  void *word = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&word, linear_status);
  if (e != cudaSuccess) return set_error(CXG_ECUDA, "cxg_linear_f32_status: %s", cudaGetErrorString(e));
  return take_status_word(word, stream, "cxg_linear_f32");
}
