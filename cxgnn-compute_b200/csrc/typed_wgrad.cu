// Weight gradient of the typed (relation-bucketed) linear on the 5th-generation tensor cores:
//   dW[r] = sum over the positions m of relation r of  x[ix(m), :]^T (outer) g[ig(m), :]          [num_rel, K, N]
// with the positions sorted by relation and padded so that every aligned block of 128 positions holds one relation
// (TypedLinearE2EOP.preprocess, cxgnncomp/typed_linear.py:74-87). The reference computes it as one torch.mm per
// relation over row sets (typed_linear.py:115-137); here it is one launch: a contraction over POSITIONS.
//
// The contraction index is the row of both operands, so both are "MN-major" for the tensor core: a tile of 128
// positions of x ([128][K]) is the A operand A[m = column of x][k = position], a tile of g ([128][N]) the B operand.
// A tile is laid out in a 128-byte swizzle: per 128-byte span of a row one block of 128 rows x 128 bytes (row p at
// p * 128, its chunks permuted by the row number), the spans 16 KiB apart. The producers put it there themselves with
// 16-byte asynchronous copies (the rows are gathered by index).
//
// A persistent CTA per SM owns a contiguous range of tiles and accumulates consecutive tiles of one relation in
// tensor memory; when the relation changes (or the range ends) the epilogue warps flush the [K][N] accumulator to
// a partial slot of this CTA. A second kernel adds the slots of every relation in (CTA, slot) order: no atomics,
// the same bits on every run.
//
// An accumulator takes a bounded number of positions (its error grows with them), then the epilogue adds it to the sum in
// the slot. In rows of N columns every lane of that read-modify-write was in another line, and the four warps took longer
// for it than the tensor core for the next accumulator. Now four columns of all rows lie side by side, eight warps share
// the columns, and the old sums are asked for a step ahead: 169,343 positions, 128 x 128, 81 -> 54 us (a stream of both
// operands takes 26); 2.33 M positions, 128 x 64, gathered, 551 -> 503 us (1.79 GB, 270). What is left is spread thin: with
// no copies, conversion or epilogue the barriers and the 8 instructions of a tile alone take 354 us, without three quarters
// of the instructions 233, and shared memory is busy for two thirds of the time.
//
// fp32 inputs: plain TF32 products (precision 1) or, like the forward, error-compensated ones (precision 2): of both tiles
// of a stage, whose words the tensor core reads as hi = upper 19 bits, four converter warps write lo = v - hi rounded to 19
// bits (they wrote hi as well until it showed that nothing depends on it: same bits, 3 % of the kernel), and the tensor core
// accumulates A_hi.B_lo + A_lo.B_hi and A_hi.B_hi. (169,343 positions, 128 x 128, against float64: 3.8e-6 of the result with
// one accumulator and 512 positions in it, 0.9e-6 with two and 256; an fp32 GEMM 1.4e-6.)
//
// Every wait is bounded; a role that waits too long raises a CTA-wide abort flag and an error status.
#include "common.cuh"
#include "tensor_core.cuh"

namespace cxg {
namespace {

using namespace tc;

constexpr int kProdWarps = 8;
constexpr int kConvWarps = 4;
constexpr int kEpiWarps = 8;    // warps 0..7: tensor-memory lanes 32 * (warp % 4) .. + 31, every other 16 columns
constexpr int kMmaWarp = kEpiWarps;
constexpr int kFirstProd = kMmaWarp + 1;
constexpr int kFirstConv = kFirstProd + kProdWarps;
constexpr int kMaxStages = 4;
constexpr int kSmemBudget = 225 * 1024;
// Positions per tile of the compensated mode: a stage of 128 + 128 columns takes 64 KB, so three of them are in flight (with
// 64 positions it was one, and loading, splitting and multiplying took turns: 169,343 x 128 x 128 146 us, now 91).
constexpr int kPosX3 = 32;

struct WgArgs {
  const void *x;       // [*, k]
  const void *g;       // [*, n]
  const int64_t *rel;  // [m] relation of every position (constant per aligned block of 128)
  const int64_t *idx;    // [m] row of x of every position, or NULL (position = row)
  const int64_t *idx_g;  // [m] row of g of every position, or NULL (the row of x)
  int64_t m, x_rows, g_rows;  // positions; rows with an index in [0, x_rows) / [0, g_rows) exist, others count as zero rows
  int k, n, num_rel;
  int stages, slots;
  int dense;           // 0, or the column blocks of x: the whole matrices, one relation, a column block pair per blockIdx.y
  int chunk_tiles;     // tiles summed in one tensor-memory accumulator before the epilogue takes it over
  int test_stall;      // test hook: the producers never hand over their first tile, so the waits for it run out
  float *partial;      // [grid][slots][n / 4][k][4]; dense: [column block pair][blockIdx.x][128 / 4][128][4]
  int32_t *slot_rel;   // [grid][slots]: relation of a flushed slot, -1 when unused
  int32_t *status;
  long long wait_cycles;
};

// MN-major operand in a 128-byte swizzled layout: rows of 128 bytes (one per step of the contraction index), `lbo`
// bytes between 128-byte spans along M / N. 16-bit elements: groups of 8 rows 1024 bytes apart, the 16-byte chunks of
// a row permuted by row % 8 (layout type 2). 32-bit elements have their own form, the only one the tensor core takes
// for MN-major TF32 operands: groups of 4 rows 512 bytes apart, the 32-byte chunks of a row permuted by row % 4
// (layout type 1, "128-byte swizzle with a 32-byte base").
template <bool W32>
__device__ __forceinline__ uint64_t make_desc_mn_sw128(uint32_t addr, uint32_t lbo) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr >> 4) & 0x3fff);
  d |= static_cast<uint64_t>((lbo >> 4) & 0x3fff) << 16;
  d |= static_cast<uint64_t>((W32 ? 512 : 1024) >> 4) << 32;
  d |= 1ull << 46;  // descriptor version of sm_100
  d |= (W32 ? 1ull : 2ull) << 61;
  return d;
}

// Byte offset of 16-byte chunk c16 of row p inside a span of either layout.
template <bool W32>
__device__ __forceinline__ uint32_t swizzled_offset(int p, int c16) {
  if (W32) return p * 128 + ((((c16 >> 1) ^ (p & 3)) << 5) | ((c16 & 1) << 4));
  return p * 128 + ((c16 ^ (p & 7)) << 4);
}

// fp32 accumulate, A and B of format `fmt` (1 = bf16, 2 = tf32), both MN-major.
__device__ __forceinline__ uint32_t make_idesc_mn(int fmt, int m, int n) {
  uint32_t d = 0;
  d |= 1u << 4;
  d |= static_cast<uint32_t>(fmt) << 7;
  d |= static_cast<uint32_t>(fmt) << 10;
  d |= 1u << 15;  // A is MN-major
  d |= 1u << 16;  // B is MN-major
  d |= static_cast<uint32_t>(n >> 3) << 17;
  d |= static_cast<uint32_t>(m >> 4) << 24;
  return d;
}

struct Barriers {
  uint64_t full[kMaxStages];   // producers -> MMA (or converters): 256 arrivals
  uint64_t conv[kMaxStages];   // converters -> MMA: 128 arrivals
  uint64_t empty[kMaxStages];  // MMA -> producers: 1 commit
  uint64_t acc_full[2];        // MMA -> epilogue: the accumulator buffer holds a finished chunk (1 commit)
  uint64_t acc_empty[2];       // epilogue -> MMA: the buffer has been read (256 arrivals)
};

// X3: error-compensated fp32. T = float or __nv_bfloat16. kPos = positions per tile, the contraction length of one
// pipeline unit: 128, or 32 in the compensated mode, whose stages hold every tile twice.
template <typename T, bool X3>
__global__ void __launch_bounds__(32 * (kEpiWarps + 1 + kProdWarps + (X3 ? kConvWarps : 0)), 1) typed_wgrad_tc(WgArgs a) {
  constexpr bool TF32 = sizeof(T) == 4;
  constexpr int kPos = X3 ? kPosX3 : 128;
  constexpr int kSpan = 128 * kPos;  // bytes of one 128-byte span of a tile (kPos rows)
  constexpr int kInstrK = TF32 ? 8 : 16;  // positions per MMA
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ __align__(8) Barriers bars;
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_slot;
  volatile int *abort_flag = &abort_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // spans that hold the rows of x and of g. The tensor core reads 128 columns of x: those behind K lie in the memory
  // behind (g's spans, the next stage) and only reach rows of the result that are not stored.
  const int x_at = a.dense ? static_cast<int>(blockIdx.y % a.dense) * 128 : 0;  // first column of the block
  const int g_at = a.dense ? static_cast<int>(blockIdx.y / a.dense) * 128 : 0;
  const int k = a.dense ? min(128, a.k - x_at) : a.k, n = a.dense ? min(128, a.n - g_at) : a.n;
  const int xrow = k * static_cast<int>(sizeof(T)), grow = n * static_cast<int>(sizeof(T));
  const int spans_x = (xrow + 127) / 128, spans_g = (grow + 127) / 128;
  const int n_mma = spans_g * (128 / static_cast<int>(sizeof(T)));  // whole spans; columns behind N are zeros
  const uint32_t half_bytes = static_cast<uint32_t>(spans_x + spans_g) * kSpan;  // raw (or hi) tiles of x and g
  const uint32_t stage_bytes = X3 ? 2 * half_bytes : half_bytes;
  const int S = a.stages;
  uint8_t *smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);  // swizzled tiles: 1024-byte boundaries
  int tmem_cols = 32;
  while (tmem_cols < n_mma) tmem_cols <<= 1;
  // compensated mode: the small terms have an accumulator of their own where there is room (see typed_mm.cu)
  const uint32_t small_off = X3 && 4 * tmem_cols <= 512 ? n_mma : 0;
  if (small_off) tmem_cols *= 2;  // columns of one of the two buffers
  const uint32_t tmem_all = 2 * tmem_cols;

  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_slot)),
                 "r"(tmem_all)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    abort_slot = 0;
    for (int s = 0; s < kMaxStages; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&bars.full[s])), "r"(32 * kProdWarps) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&bars.conv[s])), "r"(32 * kConvWarps) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bars.empty[s])) : "memory");
    }
    for (int b = 0; b < 2; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bars.acc_full[b])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&bars.acc_empty[b])), "r"(32 * kEpiWarps) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  dependency_wait();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_d = tmem_base_slot;

  const int64_t n_tiles = (a.m + kPos - 1) / kPos;
  const int64_t tile_lo = n_tiles * blockIdx.x / gridDim.x, tile_hi = n_tiles * (blockIdx.x + 1) / gridDim.x;
  // Relation of a tile, for a role that walks the tiles in order: that of its aligned block of 128 positions, asked for a
  // block ahead (fetched when it is needed, it cost every role a round trip to memory per tile).
  struct RelCursor {
    const WgArgs &a;
    int64_t block, now, next;
    __device__ int64_t load(int64_t b) const { return b * 128 < a.m ? (a.dense ? 0 : a.rel[b * 128]) : -1; }
    __device__ RelCursor(const WgArgs &args, int64_t tile) : a(args), block(tile * kPos / 128) {
      now = load(block);
      next = load(block + 1);
    }
    __device__ int64_t at(int64_t tile) {
      if (tile * kPos / 128 != block) {
        ++block;
        now = next;
        next = load(block + 1);
      }
      return now;
    }
  };
  auto valid_rel = [&](int64_t r) { return r >= 0 && r < a.num_rel; };

  if (warp >= kFirstProd && warp < kFirstConv) {
    // ================= producers: gather the rows of x and g of a tile into the swizzled layout =================
    const int pt = tid - 32 * kFirstProd;  // 0 .. 255
    const int c16 = pt & 7;                // 16-byte chunk inside a 128-byte span
    const int prow = pt >> 3;              // row inside a pass of 32 rows
    const uint8_t *X = static_cast<const uint8_t *>(a.x) + x_at * sizeof(T), *G = static_cast<const uint8_t *>(a.g) + g_at * sizeof(T);
    const int64_t xpitch = a.k * static_cast<int64_t>(sizeof(T)), gpitch = a.n * static_cast<int64_t>(sizeof(T));
    constexpr int kPass = kPos / 32;  // passes of 32 rows per tile
    const uint32_t base = smem_addr(smem);
    const bool last_x = (spans_x - 1) * 128 + c16 * 16 < xrow, last_g = (spans_g - 1) * 128 + c16 * 16 < grow;
    auto copy = [](uint32_t dst, const uint8_t *src, bool in) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
    };
    // Row indices are fetched for 128 positions at once, 128 positions ahead: a tile ahead was not enough, a compensated
    // tile of 32 positions waited for its indices most of the time (2.33 M x 128 x 64: 776 us, now about 600).
    constexpr int kGroup = 128 / kPos, kAhead = kPass * kGroup;
    auto fetch = [&](int64_t tile, int64_t (&ia)[kAhead], int64_t (&ig)[kAhead]) {
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const int64_t pos = tile * kPos + q * 32 + prow;
        ia[q] = -1, ig[q] = -1;
        if (pos < tile_hi * kPos && pos < a.m) {
          ia[q] = a.idx != nullptr ? a.idx[pos] : pos;
          ig[q] = a.idx_g != nullptr ? a.idx_g[pos] : ia[q];
        }
      }
    };
    int64_t ia_next[kAhead], ig_next[kAhead];
    fetch(tile_lo, ia_next, ig_next);
    RelCursor rel(a, tile_lo);
    Ring ring(S);
    bool alive = true;
    for (int64_t tile0 = tile_lo; tile0 < tile_hi && alive; tile0 += kGroup) {
      int64_t ia[kAhead], ig[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; ++q) ia[q] = ia_next[q], ig[q] = ig_next[q];
      fetch(tile0 + kGroup, ia_next, ig_next);
#pragma unroll
      for (int t = 0; t < kGroup; ++t) {
        if (tile0 + t >= tile_hi || !alive || !valid_rel(rel.at(tile0 + t))) continue;  // invalid: a tile of padding only
        const int s = ring.stage;
        if (ring.reused()) {
          alive = wait_bar(&bars.empty[s], ring.emptied(), abort_flag, a.status, a.wait_cycles);
          if (!alive) continue;
        }
        const uint32_t st0 = base + static_cast<uint32_t>(s) * stage_bytes;
#pragma unroll
        for (int q = 0; q < kPass; ++q) {
          const int64_t xr = ia[t * kPass + q], gr = ig[t * kPass + q];
          // a position contributes only when both of its rows exist; size 0 writes zeros
          const bool ok = static_cast<uint64_t>(xr) < static_cast<uint64_t>(a.x_rows) &&
                          static_cast<uint64_t>(gr) < static_cast<uint64_t>(a.g_rows);
          const uint32_t d0 = st0 + swizzled_offset<TF32>(q * 32 + prow, c16);
          // a chunk behind the row's end (only the last span has them) is written as zeros
          auto row = [&](const uint8_t *src, int spans, bool last_in, uint32_t dst) {
            for (int j = 1; j < spans; ++j, dst += kSpan) {
              copy(dst, src, ok);
              if (ok) src += 128;
            }
            copy(dst, last_in ? src : X, ok && last_in);
          };
          row(ok ? X + xr * xpitch + c16 * 16 : X, spans_x, last_x, d0);
          row(ok ? G + gr * gpitch + c16 * 16 : G, spans_g, last_g, d0 + spans_x * kSpan);
        }
        if (!(a.test_stall && ring.round == 0 && ring.stage == 0))
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(&bars.full[s])) : "memory");
        ring.next();
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (X3 && warp >= kFirstConv) {
    // ================= converters: lo of the raw fp32 tiles, which are hi, into the second half of the stage =================
    const int ct = tid - 32 * kFirstConv;
    const int n16 = static_cast<int>(half_bytes / 16), x16 = spans_x * (kSpan / 16), g16 = n16 - x16;
    Ring ring(S);
    bool alive = true;
    RelCursor rel(a, tile_lo);
    for (int64_t tile = tile_lo; tile < tile_hi && alive; ++tile) {
      const int64_t r = rel.at(tile);
      if (!valid_rel(r)) continue;
      const int s = ring.stage;
      alive = wait_bar(&bars.full[s], ring.filled(), abort_flag, a.status, a.wait_cycles);
      if (!alive) break;
      const float4 *hi = reinterpret_cast<const float4 *>(smem + static_cast<size_t>(s) * stage_bytes);
      // the second half holds g's lo spans first, so that they follow g's hi spans, then those of x
      float4 *lo = reinterpret_cast<float4 *>(smem + static_cast<size_t>(s) * stage_bytes + half_bytes);
      constexpr int kStep = 32 * kConvWarps;
      for (int c0 = ct; c0 < n16; c0 += 4 * kStep) {  // four chunks requested at once
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (c0 + u * kStep < n16) v[u] = hi[c0 + u * kStep];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (c0 + u * kStep < n16) {
            const int c = c0 + u * kStep;
            lo[c < x16 ? g16 + c : c - x16] = make_float4(tf32_rest(v[u].x), tf32_rest(v[u].y), tf32_rest(v[u].z), tf32_rest(v[u].w));
          }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_arrive(&bars.conv[s]);
      ring.next();
    }
  } else if (warp == kMmaWarp) {
    // ================= MMA issuer =================
    // The tensor core's fp32 accumulation loses a little on every addition (the error grows linearly with the number
    // of positions summed in one accumulator), so an accumulator takes at most `chunk_tiles` tiles; the epilogue adds
    // the chunks of a relation with ordinary fp32 additions. Two accumulator buffers alternate.
    // the whole warp walks the tiles together; one lane issues (mma_ss)
    auto wait_all = [&](uint64_t *bar, uint32_t parity) {
      return __all_sync(0xffffffffu, wait_bar(bar, parity, abort_flag, a.status, a.wait_cycles)) != 0;
    };
    const uint32_t idesc = make_idesc_mn(TF32 ? 2 : 1, 128, n_mma);
    const uint32_t idesc_wide = make_idesc_mn(2, 128, small_off ? 2 * n_mma : n_mma);
    const uint32_t step_bytes = kInstrK * 128;  // the next kInstrK positions of a span
    Ring ring(S);
    int64_t chunk = 0;
    int in_chunk = 0;
    bool alive = true, open = false;  // open: the current accumulator holds tiles of relation `cur`
    int64_t cur = -1;
    RelCursor rel(a, tile_lo);
    for (int64_t tile = tile_lo; tile < tile_hi && alive; ++tile) {
      const int64_t r = rel.at(tile);
      if (!valid_rel(r)) continue;
      if (open && (r != cur || in_chunk == a.chunk_tiles)) {  // hand the chunk to the epilogue
        commit_to(&bars.acc_full[chunk & 1]);
        open = false;
        ++chunk;
      }
      const int buf = static_cast<int>(chunk & 1);
      if (!open) {
        if (chunk >= 2) {  // the epilogue has read the chunk that used this buffer before
          alive = wait_all(&bars.acc_empty[buf], static_cast<uint32_t>(((chunk >> 1) - 1) & 1));
          if (!alive) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        cur = r;
        in_chunk = 0;
      }
      const uint32_t d = tmem_d + buf * tmem_cols;
      const int s = ring.stage;
      alive = wait_all(X3 ? &bars.conv[s] : &bars.full[s], ring.filled());
      if (!alive) break;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t x0 = smem_addr(smem + static_cast<size_t>(s) * stage_bytes);
      const uint32_t g0 = x0 + spans_x * kSpan;
      for (int j = 0; j < kPos / kInstrK; ++j) {
        const uint32_t first = (open || j > 0) ? 1u : 0u;
        const uint32_t off = j * step_bytes;
        if (X3) {
          const uint64_t xa = make_desc_mn_sw128<TF32>(x0 + off, kSpan);
          const uint64_t xl = make_desc_mn_sw128<TF32>(x0 + half_bytes + spans_g * kSpan + off, kSpan);
          const uint64_t ga = make_desc_mn_sw128<TF32>(g0 + off, kSpan);
          if (small_off) {  // hi x [hi | lo] in one instruction
            mma_ss<TF32>(d, xa, ga, idesc_wide, first);
            mma_ss<TF32>(d + small_off, xl, ga, idesc, 1u);
          } else {
            mma_ss<TF32>(d, xa, make_desc_mn_sw128<TF32>(x0 + half_bytes + off, kSpan), idesc, first);
            mma_ss<TF32>(d, xl, ga, idesc, 1u);
            mma_ss<TF32>(d, xa, ga, idesc, 1u);
          }
        } else {
          mma_ss<TF32>(d, make_desc_mn_sw128<TF32>(x0 + off, kSpan), make_desc_mn_sw128<TF32>(g0 + off, kSpan), idesc, first);
        }
      }
      commit_to(&bars.empty[s]);
      open = true;
      ++in_chunk;
      ring.next();
    }
    if (alive && open) commit_to(&bars.acc_full[chunk & 1]);
  } else if (warp < kEpiWarps) {
    // ================= epilogue: add every chunk's accumulator into the relation segment's slot of this CTA =================
    // the chunks and segments are found by walking the same tile range as the MMA thread
    int64_t chunk = 0, seg = 0, cur = -1;
    int in_chunk = 0;
    bool alive = true, open = false, seg_started = false;
    const int row = (warp & 3) * 32 + lane;  // row of dW[r] = column of x
    const int c_first = (warp >> 2) * 16, rows = a.dense ? 128 : a.k;
    auto take_chunk = [&]() {
      const int buf = static_cast<int>(chunk & 1);
      // four columns of all rows side by side: a warp's access is 512 bytes in a row
      float *slot = a.dense ? a.partial + (static_cast<int64_t>(blockIdx.y) * gridDim.x + blockIdx.x) * (128 * 128)
                            : a.partial + (static_cast<int64_t>(blockIdx.x) * a.slots + seg) * a.k * a.n;
      float4 *out = reinterpret_cast<float4 *>(slot) + row;
      const bool more = seg_started && row < k;  // a later chunk of the segment: ordinary fp32 additions, in chunk order
      float4 old[2] = {}, next[2] = {};
      auto fetch = [&](int c) {
        if (more && c < n) next[0] = out[(c >> 2) * rows], next[1] = out[((c >> 2) + 1) * rows];
      };
      fetch(c_first);
      alive = wait_bar(&bars.acc_full[buf], static_cast<uint32_t>((chunk >> 1) & 1), abort_flag, a.status, a.wait_cycles);
      if (!alive) return;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t taddr = tmem_d + (static_cast<uint32_t>((warp & 3) * 32) << 16) + buf * tmem_cols;
      for (int c = c_first; c < n; c += (c & 8) ? 24 : 8) {  // 8 columns at a time, 16 of every 32
        old[0] = next[0], old[1] = next[1];
        fetch(c + ((c & 8) ? 24 : 8));
        uint32_t v[8];
        tmem_ld8(v, taddr + c);
        if (X3 && small_off) {
          uint32_t w[8];
          tmem_ld8(w, taddr + small_off + c);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(w[i]));
        } else {
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        }
        if (row < k) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            float4 acc = make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]), __uint_as_float(v[4 * q + 2]),
                                     __uint_as_float(v[4 * q + 3]));
            if (seg_started) acc.x += old[q].x, acc.y += old[q].y, acc.z += old[q].z, acc.w += old[q].w;
            out[((c >> 2) + q) * rows] = acc;
          }
        }
      }
      if (tid == 0 && !seg_started && !a.dense) a.slot_rel[static_cast<int64_t>(blockIdx.x) * a.slots + seg] = static_cast<int32_t>(cur);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive(&bars.acc_empty[buf]);
      seg_started = true;
      ++chunk;
    };
    RelCursor rel(a, tile_lo);
    for (int64_t tile = tile_lo; tile < tile_hi && alive; ++tile) {
      const int64_t r = rel.at(tile);
      if (!valid_rel(r)) continue;
      if (open && (r != cur || in_chunk == a.chunk_tiles)) {
        take_chunk();
        if (!alive) break;
        open = false;
        if (r != cur) {
          ++seg;
          seg_started = false;
        }
      }
      if (!open) in_chunk = 0;
      cur = r;
      open = true;
      ++in_chunk;
    }
    if (alive && open) take_chunk();
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(tmem_all)
                 : "memory");
  }
}

// dW[r][i] = sum of partial[cta][slot][i] over the slots whose relation is r, in (cta, slot) order. A block first lists the
// slots of its relation in order (8 slots a thread, a block scan), then adds them up with eight loads in flight. (Walking
// all 148 * (num_rel + 1) slots with one load after the other was bound by that chain: 65 us for eight relations of
// 128 x 64, now 5 us.) The small block spreads a small gradient over more SMs.
constexpr int kRedThreads = 128, kRedPer = 8, kRedChunk = kRedThreads * kRedPer;
__global__ void __launch_bounds__(kRedThreads) wgrad_reduce(const float *partial, const int32_t *slot_rel, float *dw,
                                                            int n_slots, int num_rel, int k, int n) {
  dependency_wait();
  __shared__ int list[kRedChunk];
  const int64_t kn = static_cast<int64_t>(k) * n;
  __shared__ int warp_sum[kRedThreads / 32];
  const int64_t i = blockIdx.x * static_cast<int64_t>(kRedThreads) + threadIdx.x;
  const int r = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool in = i < kn;
  const float *p = partial + (in ? i : 0);
  float s = 0.f;
  for (int base = 0; base < n_slots; base += kRedChunk) {
    const int q0 = base + static_cast<int>(threadIdx.x) * kRedPer;
    uint32_t hit = 0;
#pragma unroll
    for (int u = 0; u < kRedPer; ++u)
      if (q0 + u < n_slots && slot_rel[q0 + u] == r) hit |= 1u << u;
    const int own = __popc(hit);
    int at = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, at, d);
      if (lane >= d) at += o;
    }
    if (lane == 31) warp_sum[warp] = at;
    __syncthreads();
    int total = 0;
#pragma unroll
    for (int w = 0; w < kRedThreads / 32; ++w) {
      if (w == warp) at += total;
      total += warp_sum[w];
    }
    at -= own;
    for (; hit != 0; hit &= hit - 1) list[at++] = q0 + __ffs(hit) - 1;
    __syncthreads();
    int q = 0;
    for (; q + 8 <= total; q += 8) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = p[list[q + u] * kn];
#pragma unroll
      for (int u = 0; u < 8; ++u) s += v[u];
    }
    for (; q < total; ++q) s += p[list[q] * kn];
    __syncthreads();  // the list is free for the next chunk
  }
  if (in) {
    const int64_t q = i >> 2;  // four columns of all rows side by side
    dw[r * kn + q % k * n + (q / k * 4 + (i & 3))] = s;
  }
}

__global__ void wgrad_clear(int32_t *slot_rel, int n) {
  dependency_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) slot_rel[i] = -1;
}

// Dense mode: dW[i][j] = sum of the partials of its column block pair over the blocks, in order, eight loads in flight. An
// infinity times the other operand's lower term, a zero or of either sign, makes NaN of what an fp32 sum gives as an
// infinity, so an element that is not finite is summed again from x and g.
__global__ void __launch_bounds__(128) dense_reduce(const float *partial, const float *x, const float *g, int64_t m, float *dw,
                                                    int k, int n, int k_blocks, int parts) {
  dependency_wait();
  const int64_t i = blockIdx.x * 128ll + threadIdx.x;
  if (i >= static_cast<int64_t>(k) * n) return;
  // neighbouring threads in the order of the partials: four columns, then the rows
  const int r = static_cast<int>((i >> 2) % k), c = static_cast<int>((i >> 2) / k * 4 + (i & 3));
  const int64_t pair = r / 128 + static_cast<int64_t>(k_blocks) * (c / 128);
  const float *p = partial + pair * parts * (128 * 128) + (c % 128 / 4 * 128 + r % 128) * 4 + c % 4;
  float s = 0.f;
  int q = 0;
  for (; q + 8 <= parts; q += 8) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = p[static_cast<int64_t>(q + u) * (128 * 128)];
#pragma unroll
    for (int u = 0; u < 8; ++u) s += v[u];
  }
  for (; q < parts; ++q) s += p[static_cast<int64_t>(q) * (128 * 128)];
  if (!(fabsf(s) <= 3.402823466e38f)) {
    s = 0.f;
    for (int64_t t = 0; t < m && s == s; t += 8)  // a chain that has become NaN stays it
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (t + u < m) s = fmaf(__ldg(x + (t + u) * k + r), __ldg(g + (t + u) * n + c), s);
  }
  dw[static_cast<int64_t>(r) * n + c] = s;
}

__device__ int32_t dense_status;  // set when a bounded wait of the dense mode ran out, cleared by cxg_dense_wgrad_f32_status

// Blocks of positions of the dense mode: one block per SM over all column block pairs.
int dense_parts(int k, int n, int64_t m) {
  const int64_t pairs = static_cast<int64_t>((k + 127) / 128) * ((n + 127) / 128);
  const int64_t tiles = (m + kPosX3 - 1) / kPosX3, parts = pairs < kNumSM ? kNumSM / pairs : 1;
  return static_cast<int>(parts < tiles ? parts : tiles);
}

struct WgLayout {
  size_t status, slot_rel, partial, total;
  int grid, slots;
};

void wgrad_layout(int num_rel, int k, int n, WgLayout *L) {
  L->grid = kNumSM;
  L->slots = num_rel + 1;  // a contiguous range of sorted tiles meets every relation at most once, plus one
  size_t off = 0;
  L->status = off;
  off = align_up(off + 256, 256);
  L->slot_rel = off;
  off = align_up(off + static_cast<size_t>(L->grid) * L->slots * sizeof(int32_t), 256);
  L->partial = off;
  off = align_up(off + static_cast<size_t>(L->grid) * L->slots * k * n * sizeof(float), 256);
  L->total = off;
}

}  // namespace
}  // namespace cxg

using namespace cxg;

extern "C" int cxg_typed_wgrad_workspace_size(int num_rel, int k, int n, size_t *bytes) {
  CXG_REQUIRE(bytes != nullptr, CXG_ENULL, "cxg_typed_wgrad_workspace_size: bytes is NULL");
  CXG_REQUIRE(num_rel > 0 && k > 0 && n > 0, CXG_EINVAL, "cxg_typed_wgrad_workspace_size: bad sizes");
  WgLayout L;
  wgrad_layout(num_rel, k, n, &L);
  *bytes = L.total;
  return CXG_OK;
}

extern "C" int cxg_typed_wgrad(const void *x, const void *g, const int64_t *rel, const int64_t *idx, const int64_t *idx_g,
                               int64_t m, int64_t x_rows, int64_t g_rows, int k, int n, int num_rel, int dtype,
                               int precision, uint32_t flags, float *dw, void *workspace, size_t workspace_bytes,
                               void *stream) {
  CXG_REQUIRE(m >= 0 && x_rows >= 0 && g_rows >= 0 && k > 0 && n > 0 && num_rel > 0, CXG_EINVAL,
              "cxg_typed_wgrad: bad sizes");
  CXG_REQUIRE(dtype == CXG_F32 || dtype == CXG_BF16, CXG_EINVAL, "cxg_typed_wgrad: dtype %d", dtype);
  CXG_REQUIRE(precision == 1 || precision == 2, CXG_EINVAL, "cxg_typed_wgrad: precision %d (1 = plain, 2 = compensated)",
              precision);
  CXG_REQUIRE(dw != nullptr, CXG_ENULL, "cxg_typed_wgrad: dw is NULL");
  const int elem = dtype == CXG_F32 ? 4 : 2;
  CXG_REQUIRE(k <= 128 && (k * elem) % 16 == 0 && n % 16 == 0 && n <= 256, CXG_EUNSUPPORTED,
              "cxg_typed_wgrad: K = %d must be a multiple of %d up to 128 and N = %d one of 16 up to 256", k, 16 / elem, n);
  cudaStream_t st = as_stream(stream);
  const int64_t kn = static_cast<int64_t>(k) * n;
  if (m == 0) {
    if (cudaMemsetAsync(dw, 0, static_cast<size_t>(num_rel) * kn * sizeof(float), st) != cudaSuccess)
      return check_launch("cxg_typed_wgrad: memset");
    return CXG_OK;
  }
  CXG_REQUIRE(x && g && rel, CXG_ENULL, "cxg_typed_wgrad: NULL argument");
  CXG_REQUIRE(reinterpret_cast<uintptr_t>(x) % 16 == 0 && reinterpret_cast<uintptr_t>(g) % 16 == 0, CXG_EINVAL,
              "cxg_typed_wgrad: x and g must be 16-byte aligned");
  WgLayout L;
  wgrad_layout(num_rel, k, n, &L);
  CXG_REQUIRE(workspace != nullptr && workspace_bytes >= L.total, CXG_EWORKSPACE,
              "cxg_typed_wgrad: workspace %zu bytes, need %zu", workspace_bytes, L.total);
  CXG_REQUIRE(reinterpret_cast<uintptr_t>(workspace) % 16 == 0, CXG_EINVAL, "cxg_typed_wgrad: workspace alignment");
  const bool x3 = precision == 2 && dtype == CXG_F32;
  const int pos = x3 ? kPosX3 : 128;  // positions per tile, as in the kernel
  const int spans = (k * elem + 127) / 128 + (n * elem + 127) / 128;
  const size_t half = static_cast<size_t>(spans) * (128 * pos);
  const size_t stage = x3 ? 2 * half : half;
  // The tensor core reads elem spans of x (128 columns) from the start of its spans, which for narrow x goes beyond the tile:
  // room behind the last stage. In the compensated mode the last spans of a stage are x's lo spans.
  const int spans_x = (k * elem + 127) / 128, over = x3 ? elem - spans_x : elem - spans;
  const size_t behind = over > 0 ? static_cast<size_t>(over) * (128 * pos) : 0;
  int stages = static_cast<int>((kSmemBudget - 1024 - behind) / stage);
  if (stages > kMaxStages) stages = kMaxStages;
  CXG_REQUIRE(stages >= 1, CXG_EUNSUPPORTED, "cxg_typed_wgrad: one stage of %zu bytes exceeds shared memory", stage);
  const size_t smem = 1024 + stages * stage + behind;

  char *ws = static_cast<char *>(workspace);
  WgArgs a;
  a.x = x, a.g = g, a.rel = rel, a.idx = idx, a.idx_g = idx_g, a.m = m, a.x_rows = x_rows, a.g_rows = g_rows;
  a.k = k, a.n = n, a.num_rel = num_rel, a.stages = stages, a.slots = L.slots;
  a.test_stall = (flags & CXG_WGRAD_TEST_STALL) ? 1 : 0;
  a.dense = 0;
  a.chunk_tiles = x3 ? 256 / kPosX3 : 32;  // 256 / 4096 positions per accumulator: its error stays below that of an fp32 sum / below
                                // the rounding of the plain products
  a.partial = reinterpret_cast<float *>(ws + L.partial);
  a.slot_rel = reinterpret_cast<int32_t *>(ws + L.slot_rel);
  a.status = reinterpret_cast<int32_t *>(ws + L.status);
  a.wait_cycles = wait_limit_cycles();
  if (cudaMemsetAsync(a.status, 0, 256, st) != cudaSuccess) return check_launch("cxg_typed_wgrad: memset");
  const int n_slots = L.grid * L.slots;
  launch_dependent(wgrad_clear, (n_slots + 255) / 256, 256, 0, st, a.slot_rel, n_slots);
  const int64_t n_tiles = (m + pos - 1) / pos;  // a last partial tile holds positions past the padded buckets
  const unsigned grid = static_cast<unsigned>(n_tiles < L.grid ? n_tiles : L.grid);
  cudaError_t e = cudaSuccess;
  auto launch = [&](auto kernel, int warps) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e == cudaSuccess) launch_dependent(kernel, grid, 32 * warps, smem, st, a);
  };
  constexpr int kW = kEpiWarps + 1 + kProdWarps;
  if (dtype == CXG_F32) {
    if (x3)
      launch(typed_wgrad_tc<float, true>, kW + kConvWarps);
    else
      launch(typed_wgrad_tc<float, false>, kW);
  } else {
    launch(typed_wgrad_tc<__nv_bfloat16, false>, kW);
  }
  if (e != cudaSuccess) return set_error(CXG_ECUDA, "cxg_typed_wgrad: %s", cudaGetErrorString(e));
  dim3 rg(static_cast<unsigned>((kn + kRedThreads - 1) / kRedThreads), static_cast<unsigned>(num_rel));
  launch_dependent(wgrad_reduce, rg, kRedThreads, 0, st, a.partial, a.slot_rel, dw, n_slots, num_rel, k, n);
  count_launches(3);
  return check_launch("cxg_typed_wgrad");
}

extern "C" int cxg_dense_wgrad_f32_workspace_size(int64_t m, int k, int n, size_t *bytes) {
  CXG_REQUIRE(bytes != nullptr, CXG_ENULL, "cxg_dense_wgrad_f32_workspace_size: bytes is NULL");
  CXG_REQUIRE(m > 0 && k > 0 && n > 0, CXG_EINVAL, "cxg_dense_wgrad_f32_workspace_size: bad sizes");
  *bytes = static_cast<size_t>((k + 127) / 128) * ((n + 127) / 128) * dense_parts(k, n, m) * (128 * 128 * sizeof(float));
  return CXG_OK;
}

extern "C" int cxg_dense_wgrad_f32(const float *x, const float *g, int64_t m, int k, int n, float *dw, void *workspace,
                                   size_t workspace_bytes, void *stream) {
  return cxg_dense_wgrad_f32_ex(x, g, m, k, n, 0u, dw, workspace, workspace_bytes, stream);
}

extern "C" int cxg_dense_wgrad_f32_ex(const float *x, const float *g, int64_t m, int k, int n, uint32_t flags, float *dw,
                                      void *workspace, size_t workspace_bytes, void *stream) {
  CXG_REQUIRE(m > 0 && k > 0 && n > 0, CXG_EINVAL, "cxg_dense_wgrad_f32: bad sizes");
  CXG_REQUIRE(x && g && dw, CXG_ENULL, "cxg_dense_wgrad_f32: NULL argument");
  const int k_blocks = (k + 127) / 128, n_blocks = (n + 127) / 128;
  CXG_REQUIRE(k % 4 == 0 && n % 4 == 0 && k_blocks * n_blocks <= 65535, CXG_EUNSUPPORTED,
              "cxg_dense_wgrad_f32: K = %d and N = %d must be multiples of 4", k, n);
  CXG_REQUIRE((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(g)) % 16 == 0, CXG_EINVAL,
              "cxg_dense_wgrad_f32: x and g must be 16-byte aligned");
  size_t need = 0;
  cxg_dense_wgrad_f32_workspace_size(m, k, n, &need);
  CXG_REQUIRE(workspace != nullptr && workspace_bytes >= need && reinterpret_cast<uintptr_t>(workspace) % 16 == 0,
              CXG_EWORKSPACE, "cxg_dense_wgrad_f32: workspace %zu bytes, need %zu", workspace_bytes, need);
  cudaStream_t st = as_stream(stream);
  const int wk = k < 128 ? k : 128, wn = n < 128 ? n : 128;  // the widest column blocks
  const int spans = (wk + 31) / 32 + (wn + 31) / 32;
  const size_t stage = 2 * static_cast<size_t>(spans) * (128 * kPosX3);
  // the tensor core reads four spans of x from a tile's start (last block of columns included)
  const size_t behind = 4 * static_cast<size_t>(128 * kPosX3);
  int stages = static_cast<int>((kSmemBudget - 1024 - behind) / stage);
  if (stages > kMaxStages) stages = kMaxStages;
  WgArgs a;
  a.x = x, a.g = g, a.rel = nullptr, a.idx = nullptr, a.idx_g = nullptr, a.m = m, a.x_rows = m, a.g_rows = m;
  a.k = k, a.n = n, a.num_rel = 1, a.stages = stages, a.slots = 1, a.dense = k_blocks;
  a.test_stall = (flags & CXG_WGRAD_TEST_STALL) ? 1 : 0;
  a.chunk_tiles = 256 / kPosX3;
  a.partial = static_cast<float *>(workspace);
  a.slot_rel = nullptr;
  a.wait_cycles = wait_limit_cycles();
  void *word = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&word, dense_status);
  a.status = static_cast<int32_t *>(word);
  const int smem = static_cast<int>(1024 + stages * stage + behind);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(typed_wgrad_tc<float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return set_error(CXG_ECUDA, "cxg_dense_wgrad_f32: %s", cudaGetErrorString(e));
  const int parts = dense_parts(k, n, m);
  const dim3 grid(static_cast<unsigned>(parts), static_cast<unsigned>(k_blocks * n_blocks));
  launch_dependent(typed_wgrad_tc<float, true>, grid, 32 * (kEpiWarps + 1 + kProdWarps + kConvWarps), smem, st, a);
  launch_dependent(dense_reduce, static_cast<unsigned>((static_cast<int64_t>(k) * n + 127) / 128), 128, 0, st, a.partial, x, g, m, dw, k, n,
                                                                                            k_blocks, parts);
  count_launches(2);
  return check_launch("cxg_dense_wgrad_f32");
}

extern "C" int cxg_dense_wgrad_f32_status(void *stream) {
  void *word = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&word, dense_status);
  if (e != cudaSuccess) return set_error(CXG_ECUDA, "cxg_dense_wgrad_f32_status: %s", cudaGetErrorString(e));
  return take_status_word(word, stream, "cxg_dense_wgrad_f32");
}

extern "C" int cxg_typed_wgrad_status(const void *workspace, void *stream) {
  CXG_REQUIRE(workspace != nullptr, CXG_ENULL, "cxg_typed_wgrad_status: workspace is NULL");
  int32_t word = 0;
  cudaStream_t st = as_stream(stream);
  if (cudaMemcpyAsync(&word, workspace, sizeof(word), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return check_launch("cxg_typed_wgrad_status");
  if (word != 0) return set_error(CXG_ETIMEOUT, "cxg_typed_wgrad: a bounded wait ran out");
  return CXG_OK;
}
