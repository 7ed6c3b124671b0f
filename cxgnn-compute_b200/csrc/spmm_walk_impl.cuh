// The tiled walk of cxg_spmm_csr: y[t(r),:] (+)= red_{e in row r} v[e] * x[s(e),:].
//
// Work is cut by EDGES: tile t owns the edges [t*T, (t+1)*T) of the CSR edge array. A tile is walked by a GROUP of G
// lanes, 32 / G tiles side by side in a warp. A lane holds NV vectors of VB bytes of every row, so that narrow rows do
// not cost a whole warp instruction per load and rows of any width (F = 47, 100 ...) keep most of their lanes busy.
// Feature rows go global -> registers through L1 (where the hub rows of a power-law graph are found again: 32 to 43 % of the
// sectors), U edges in flight per lane, and are added strictly in edge order, one fp32 accumulator per column. When the walk
// passes the end of a row the accumulators are written and reset; rows without edges get zeros on the way.
//
// A row inside one tile is therefore summed like a sequential loop. A row that crosses tile borders leaves one fp32
// partial per tile; walk_fix adds the partials in tile order (sequentially up to 64; longer chains in blocks of 64
// consecutive partials, whose sums are then added in block order). No atomics touch feature data. (Letting the tile that
// arrives last add them inside this kernel measured 30 % slower: the fence and the counter cost every tile two round
// trips to L2 while the gather saturates it. The same holds for a search of the tile's first row in here: walk_plan
// leaves it. Neighbouring tiles walked as one piece, so that ids and row ends go on, measured 3 % slower below 3 M edges and no
// faster above: what a tile costs is its partials, not its start.)
// whole_rows: tile borders are moved so that only rows longer than T are cut, at multiples of T from their own start:
// tile t then owns the pieces that START in [t*T, (t+1)*T).
//
// Every edge of a step has its own copy of the code at a row's end, which therefore holds nothing that is not needed there:
// accumulating outputs have an instantiation of their own, scattered ones (targets) and those that accumulate sums of
// weighted rows take spmm_stream / spmm_rows.
//
// What bounds it: DRAM where x is far larger than L2 (126 M edges, F = 100: 90 % of copy bandwidth), L2 for wide rows, and in
// between the data stage of the load path, which takes one pass per line and eight lanes: 5.4 passes per edge of 12.6 M edges
// with F = 48 and edge values kept it 87 % busy. So lanes behind a row read what their neighbours read, ids and edge values
// come four at a time out of shared memory (a shuffle is a pass per edge), and 32-bit counters keep everything in 64
// registers (8 blocks per SM; the 64-bit ones spilled 100 to 200 bytes per lane, which are passes too). Tiles are handed
// out as warps come for them: SMs differ by 20 % in what they get through. Measured, whole call, before -> now: 12.6 M
// edges, F = 128 407 -> 357 us, with edge values 577 -> 386; F = 48 251 -> 223 and 374 -> 241; F = 47 389 -> 337 and 442 ->
// 356; 126 M edges, F = 100 mean 5.19 -> 4.78 ms; 200 M, F = 128 bf16 6.23 -> 5.69 ms; 2.3 M, F = 128 117 -> 109 us.
// Staging the rows in shared memory with 16-byte
// asynchronous copies was the form before: it needs a load, an address and a barrier more per edge, and rows that do not
// start at a multiple of 128 bytes land there at half the rate (F = 100: 12.9 ms for 126 M edges; here 4.9 ms).
#pragma once
#include "spmm_stream.cuh"
#include "spmm_walk.cuh"

namespace cxg {
namespace walk {

constexpr int kThreads = 128;
constexpr int kFar = 1 << 30;  // "no row end in sight" in tile-relative positions

template <int W>
struct Words {
  uint32_t w[W];
};
template <int VB>
__device__ __forceinline__ void load_row_bytes(Words<(VB + 3) / 4> &r, const uint8_t *p) {
  if constexpr (VB == 16) {
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p));
    r.w[0] = v.x, r.w[1] = v.y, r.w[2] = v.z, r.w[3] = v.w;
  } else if constexpr (VB == 8) {
    const uint2 v = __ldg(reinterpret_cast<const uint2 *>(p));
    r.w[0] = v.x, r.w[1] = v.y;
  } else if constexpr (VB == 4) {
    r.w[0] = __ldg(reinterpret_cast<const uint32_t *>(p));
  } else {
    r.w[0] = __ldg(reinterpret_cast<const uint16_t *>(p));
  }
}

__device__ __forceinline__ int64_t load_id_stream(const int64_t *p) {
  int64_t v;
  asm volatile("ld.global.nc.L1::no_allocate.s64 %0, [%1];" : "=l"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ int32_t load_id_stream(const int32_t *p) {
  int32_t v;
  asm volatile("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// The low 32 bits of an id (a row number below 2^32) and of a row pointer (an edge number below 2^32), of either width.
__device__ __forceinline__ uint32_t load_id_low(const uint8_t *p) {
  uint32_t v;
  asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t load_ptr_low(const void *ptr, int i, int ptr_bytes) {
  return __ldg(reinterpret_cast<const uint32_t *>(static_cast<const uint8_t *>(ptr) + static_cast<uint64_t>(static_cast<uint32_t>(i)) * static_cast<uint32_t>(ptr_bytes)));
}

// Two or four words of shared memory.
template <int N, typename V>
__device__ __forceinline__ void load_ids(V (&v)[N], const V *p) {
  static_assert(N == 2 || N == 4, "");
  if constexpr (N == 4) {
    const uint4 t = *reinterpret_cast<const uint4 *>(p);
    const uint32_t w[4] = {t.x, t.y, t.z, t.w};
    __builtin_memcpy(v, w, 16);
  } else {
    const uint2 t = *reinterpret_cast<const uint2 *>(p);
    const uint32_t w[2] = {t.x, t.y};
    __builtin_memcpy(v, w, 8);
  }
}

// EL = fp32 values in VB bytes of T
template <typename T, int VB>
struct Acc {
  static constexpr int EL = VB / static_cast<int>(sizeof(T));
  static constexpr int W = (VB + 3) / 4;
  static constexpr int P = EL / 2;
  unsigned long long p[P > 0 ? P : 1];  // packed pairs (add.rn.f32x2 rounds each half like the scalar add)
  float s;                              // EL == 1
  __device__ __forceinline__ static unsigned long long pair(uint32_t lo, uint32_t hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1,%2};" : "=l"(v) : "r"(lo), "r"(hi));
    return v;
  }
  __device__ __forceinline__ static unsigned long long operand(const Words<W> &r, int i) {
    if (sizeof(T) == 4) return pair(r.w[(2 * i) % W], r.w[(2 * i + 1) % W]);
    return pair(r.w[i % W] << 16, r.w[i % W] & 0xffff0000u);
  }
  __device__ __forceinline__ static float scalar(const Words<W> &r) {
    return __uint_as_float(sizeof(T) == 4 ? r.w[0] : r.w[0] << 16);
  }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < P; ++i) p[i] = 0ull;
    s = 0.f;
  }
  __device__ __forceinline__ void add(const Words<W> &r) {
    if (EL == 1) {
      s += scalar(r);
    } else if (sizeof(T) == 2) {
      // fp32 += bf16 in one instruction per value (the same rounding as widening first, which takes twice as many)
#pragma unroll
      for (int i = 0; i < P; ++i)
        asm("{\n\t.reg .b16 a0, a1;\n\t.reg .f32 f0, f1;\n\tmov.b32 {a0, a1}, %1;\n\tmov.b64 {f0, f1}, %0;\n\t"
            "add.rn.f32.bf16 f0, a0, f0;\n\tadd.rn.f32.bf16 f1, a1, f1;\n\tmov.b64 %0, {f0, f1};\n\t}"
            : "+l"(p[i])
            : "r"(r.w[i % W]));
    } else {
#pragma unroll
      for (int i = 0; i < P; ++i) asm("add.rn.f32x2 %0, %0, %1;" : "+l"(p[i]) : "l"(operand(r, i)));
    }
  }
  __device__ __forceinline__ void fma(const Words<W> &r, float v) {
    if (EL == 1) {
      s = fmaf(scalar(r), v, s);
    } else {
      const unsigned long long vv = pair(__float_as_uint(v), __float_as_uint(v));
#pragma unroll
      for (int i = 0; i < P; ++i) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(p[i]) : "l"(operand(r, i)), "l"(vv));
    }
  }
  __device__ __forceinline__ void get(float *f) const {
    if (EL == 1) {
      f[0] = s;
    } else {
#pragma unroll
      for (int i = 0; i < P; ++i) asm("mov.b64 {%0,%1}, %2;" : "=f"(f[2 * i]), "=f"(f[(2 * i + 1) % EL]) : "l"(p[i]));
    }
  }
};

// f[i] / d, rounded to nearest, for a whole number d >= 1. With r the correctly rounded reciprocal, q = f r and the
// residual f - q d taken exactly by an fma, q + r (f - q d) is the correctly rounded quotient as long as nothing
// underflows (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990); below
// 1e-28 the last bit can differ. One step of Newton's method makes r exact from the hardware's estimate for every
// mantissa (checked over all 2^23 of them). A full division per value is a dozen instructions and, in every copy of the
// row end, half of the kernel where eight lanes share a row.
template <int N>
__device__ __forceinline__ void divide_by_count(float (&f)[N], float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  r = fmaf(fmaf(-d, r, 1.f), r, r);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float q = f[i] * r;
    const float rest = fmaf(-q, d, f[i]);
    f[i] = rest == rest ? fmaf(rest, r, q) : q;  // infinities and NaN stay what they are
  }
}

template <typename T, int VB>
__device__ __forceinline__ void store_row_bytes(uint8_t *dst, const float *f) {
  constexpr int EL = VB / static_cast<int>(sizeof(T));
  if (sizeof(T) == 4) {
    if (VB == 16)
      __stcs(reinterpret_cast<float4 *>(dst), make_float4(f[0], f[1 % EL], f[2 % EL], f[3 % EL]));
    else if (VB == 8)
      __stcs(reinterpret_cast<float2 *>(dst), make_float2(f[0], f[1 % EL]));
    else
      __stcs(reinterpret_cast<float *>(dst), f[0]);
  } else if (EL == 1) {
    *reinterpret_cast<__nv_bfloat16 *>(dst) = __float2bfloat16_rn(f[0]);
  } else {
    constexpr int W = EL / 2 > 0 ? EL / 2 : 1;
    uint32_t w[W];
#pragma unroll
    for (int i = 0; i < EL / 2; ++i) {
      const __nv_bfloat162 t = __floats2bfloat162_rn(f[2 * i], f[(2 * i + 1) % EL]);
      w[i] = *reinterpret_cast<const uint32_t *>(&t);
    }
    if (W == 4)
      __stcs(reinterpret_cast<uint4 *>(dst), make_uint4(w[0], w[1 % W], w[2 % W], w[3 % W]));
    else if (W == 2)
      __stcs(reinterpret_cast<uint2 *>(dst), make_uint2(w[0], w[1 % W]));
    else
      __stcs(reinterpret_cast<unsigned int *>(dst), w[0]);
  }
}

// Bytes of an output row that is added to (not through the read-only path: the kernel writes them).
template <int VB>
__device__ __forceinline__ void load_output_bytes(Words<(VB + 3) / 4> &r, const uint8_t *p) {
  if constexpr (VB == 16) {
    const uint4 v = __ldcs(reinterpret_cast<const uint4 *>(p));
    r.w[0] = v.x, r.w[1] = v.y, r.w[2] = v.z, r.w[3] = v.w;
  } else if constexpr (VB == 8) {
    const uint2 v = __ldcs(reinterpret_cast<const uint2 *>(p));
    r.w[0] = v.x, r.w[1] = v.y;
  } else if constexpr (VB == 4) {
    r.w[0] = __ldcs(reinterpret_cast<const uint32_t *>(p));
  } else {
    r.w[0] = __ldcs(reinterpret_cast<const uint16_t *>(p));
  }
}
template <typename T, int VB>
__device__ __forceinline__ void add_words(float *f, const Words<(VB + 3) / 4> &r) {
#pragma unroll
  for (int i = 0; i < VB / static_cast<int>(sizeof(T)); ++i)
    f[i] += __uint_as_float(sizeof(T) == 4 ? r.w[i] : i % 2 == 0 ? r.w[i / 2] << 16 : r.w[i / 2] & 0xffff0000u);
}

// VB: bytes per load of a lane; NV loads per row, G lanes per tile, U edges in flight per lane. VALMODE: 0 no
// edge values, 1 one per edge, 2 one per (edge, head), 3 none and the mean of the row, 4 none and the sum (or the mean) is
// added to the output, 5 to 7 as 2 with 2, 4 or 8 heads and walk_weights_slack bytes behind the values: what lies behind a
// tile's end is read unasked and goes into sums that nobody reads.
// COPY: the rows of x are copies in whole vectors (walk_plan), those of y are not: a lane stores the values of its vector
// that lie inside the row one by one.
template <typename T, int VB, int G, int NV, int U, int VALMODE, int MINB, bool COPY>
__global__ void __launch_bounds__(kThreads, MINB) spmm_walk(const __grid_constant__ WalkArgs a) {
  using A = Acc<T, VB>;
  constexpr int W = (VB + 3) / 4;
  constexpr int EL = A::EL;
  constexpr int NG = 32 / G;
  static_assert(U <= kWalkInFlight, "walk_weights_slack covers a step");
  const int lane = threadIdx.x & 31;
  const int lg = lane & (G - 1);
  dependency_wait();
  const uint32_t e_total = static_cast<uint32_t>(edge_total(a));
  const int n_dst = static_cast<int>(a.n_dst);
  const int n_tiles = static_cast<int>((e_total + static_cast<int64_t>(a.tile) - 1) / a.tile);
  const int step = static_cast<int>(gridDim.x) * (kThreads / 32) * NG;  // tiles that are walked at the same time
  const int rb = a.row_bytes;
  const uint32_t pitch = static_cast<uint32_t>(COPY ? a.x_pitch : rb);
  // vector q of this lane covers bytes [(lg + q * G) * VB, +VB) of a row; one that lies behind the row reads the row's last
  // vector again (the line its neighbours read: a load takes a pass per line and eight lanes) and is not stored
  auto on = [&](int q) { return (lg + q * G) * VB < rb; };
  const uint8_t *xq[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q)
    xq[q] = static_cast<const uint8_t *>(a.x) + (on(q) ? (lg + q * G) * VB : (rb - 1) / VB * VB);
  auto row_of_y = [&](int r) { return static_cast<uint8_t *>(a.y) + static_cast<uint64_t>(r) * static_cast<uint32_t>(rb) + lg * VB; };
  constexpr int kHeads = VALMODE >= 5 ? 1 << (VALMODE - 4) : 0;
  constexpr bool kPerHead = VALMODE == 2 || kHeads > 0;
  int head[NV];
  if (kPerHead) {
#pragma unroll
    for (int q = 0; q < NV; ++q) head[q] = on(q) ? ((lg + q * G) * EL) / a.feat : 0;
  }

  auto store = [&](uint8_t *dst, float (&f)[NV][EL]) {
#pragma unroll
    for (int q = 0; q < NV; ++q)
      if constexpr (COPY) {
        const int left = (rb - (lg + q * G) * VB) / static_cast<int>(sizeof(T));
        T *out = reinterpret_cast<T *>(dst + q * G * VB);
#pragma unroll
        for (int i = 0; i < EL; ++i)
          if (i < left) out[i] = from_f32<T>(f[q][i]);
      } else if (on(q)) {
        store_row_bytes<T, VB>(dst + q * G * VB, f[q]);
      }
  };
  auto zero_row = [&](int r) {
    if (VALMODE == 4) return;
    float z[NV][EL];
#pragma unroll
    for (int q = 0; q < NV; ++q)
#pragma unroll
      for (int i = 0; i < EL; ++i) z[q][i] = 0.f;
    store(row_of_y(r), z);
  };
  const int t_first = static_cast<int>((blockIdx.x * static_cast<unsigned>(kThreads) + threadIdx.x) / G);
  if (e_total == 0) {  // no edge at all: every row is empty
    for (int r = t_first; r < n_dst; r += step) zero_row(r);
    return;
  }

  // Ids (and values) of a batch of 32 edges per group, read four at a time by all lanes of the group: a shuffle per edge
  // takes the load path's data stage as often as a quarter of a 512-byte row does. Groups lie 36 words apart: other banks.
  constexpr int kBatch = 36;
  __shared__ __align__(16) uint32_t id_stage[kThreads / 32][NG * kBatch];
  __shared__ __align__(16) float val_stage[VALMODE == 1 ? kThreads / 32 : 1][VALMODE == 1 ? NG * kBatch : 4];
  uint32_t *my_ids = id_stage[threadIdx.x >> 5] + lane / G * kBatch;
  float *my_vals = VALMODE == 1 ? val_stage[threadIdx.x >> 5] + lane / G * kBatch : nullptr;
  // the groups of a warp take neighbouring tiles: the first by the warp's number, then whichever are next
  int t_next = 0;
  for (int t = t_first; t - lane / G < n_tiles; t = t_next) {
    t_next = n_tiles;
    if (step < n_tiles) {
      if (lane == 0) t_next = step + atomicAdd(a.hdr + kWalkHdrNext, NG);
    }
    uint32_t begin = 0, row_begin = 0, row_end = 0;
    int row = 0, len = 0;
    if (t < n_tiles) {
      const WalkTile here = load_tile(a, t);
      begin = here.begin, row_begin = here.row_begin, row_end = here.row_end;
      row = static_cast<int>(here.row);
      len = static_cast<int>(load_tile(a, t + 1).begin - begin);
    }

    // Source ids (and edge values) are requested a whole batch of 32 edges ahead: lane lg holds edges j * G + lg.
    constexpr int IB = 32 / G;
    uint32_t id_nxt[IB];
    float val_nxt[IB];
    auto load_batch = [&](int first) {
#pragma unroll
      for (int j = 0; j < IB; ++j) {
        const int pos = first + j * G + lg;
        id_nxt[j] = 0u;
        val_nxt[j] = 0.f;
        if (pos < len) {
          const uint32_t e = begin + pos;
          id_nxt[j] = load_id_low(static_cast<const uint8_t *>(a.idx) + static_cast<uint64_t>(e) * static_cast<uint32_t>(a.idx_bytes));
          if (a.edge_rel != nullptr)
            id_nxt[j] += static_cast<uint32_t>(static_cast<int64_t>(__ldg(a.edge_rel + e)) * a.rel_stride);
          if (VALMODE == 1) val_nxt[j] = __ldg(a.edge_val + e);
        }
      }
    };

    // Row ends are positions relative to `begin`. The end of the row after the current one is requested a row ahead and
    // kept as it was loaded, so that nothing waits for it before it is used.
    auto end_raw = [&](int r) { return load_ptr_low(a.ptr, min(r + 1, n_dst), a.ptr_bytes); };
    auto end_rel = [&](int r, uint32_t raw) -> int {
      const uint32_t v = raw - begin;
      return r >= n_dst || v > static_cast<uint32_t>(kFar) ? kFar : static_cast<int>(v);
    };
    int rend = kFar, rstart = 0, stop = kFar;
    uint32_t next_raw = 0;
    if (len > 0) {
      if (t == 0)
        for (int r = 0; r < row; ++r) zero_row(r);  // leading rows without edges
      rstart = row_begin < begin ? -1 : 0;  // before the tile: how far does not matter
      next_raw = end_raw(row + 1);
      rend = end_rel(row, row_end);
      while (rend == 0) {  // empty rows that the previous tile's walk wrote
        ++row;
        rend = end_rel(row, next_raw);
        next_raw = end_raw(row + 1);
      }
      stop = min(rend, len);
    }
    // What rows hold that are added to is asked for a row ahead, so that it is in L2 when the walk comes to their end.
    // (2.3 M edges, F = 128 fp32: 157 us, 171 without it, 165 with the row held in registers from its start, which at
    // F = 256 spills: 265 / 300 / 402; overwriting 126 and 206. Through spmm_stream it took 240 and 675.)
    auto request_old = [&]() {
      if (VALMODE != 4 || row + 1 >= n_dst) return;
      const uint8_t *yr = row_of_y(row + 1);
#pragma unroll
      for (int q = 0; q < NV; ++q)
        if (on(q)) asm volatile("prefetch.global.L2 [%0];" ::"l"(yr + q * G * VB));
    };
    if (len > 0) request_old();
    A acc[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) acc[q].zero();

    // the walk stands at a row end, at the end of the tile, or at both
    auto event = [&](int pos) {
      const bool row_done = pos == rend;
      if (row_done && rstart >= 0) {
        const float d = static_cast<float>(rend - rstart);
        uint8_t *yr = row_of_y(row);
        float f[NV][EL];
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          acc[q].get(f[q]);
          if (VALMODE == 3 || (VALMODE == 4 && a.reduce == CXG_MEAN)) divide_by_count<EL>(f[q], d);
          if (VALMODE == 4 && on(q)) {
            Words<W> old;
            load_output_bytes<VB>(old, yr + q * G * VB);
            add_words<T, VB>(f[q], old);
          }
        }
        store(yr, f);
      } else if (row < n_dst) {
        // the row began in an earlier tile, or goes on in the next one
        float *p = a.partials + (static_cast<int64_t>(t) * 2 + (rstart < 0 ? 0 : 1)) * a.part_stride + lg * EL;
#pragma unroll
        for (int q = 0; q < NV; ++q)
          if (on(q)) {
            float f[EL];
            acc[q].get(f);
#pragma unroll
            for (int i = 0; i < EL; i += EL % 4 == 0 ? 4 : 1)
              if (COPY && (lg + q * G) * EL + i >= a.part_stride)
                break;
              else if constexpr (EL % 4 == 0)
                *reinterpret_cast<float4 *>(p + q * G * EL + i) = make_float4(f[i], f[i + 1], f[i + 2], f[i + 3]);
              else
                p[q * G * EL + i] = f[i];
          }
      }
#pragma unroll
      for (int q = 0; q < NV; ++q) acc[q].zero();
      if (row_done) {
        rstart = pos;
        for (;;) {
          ++row;
          rend = end_rel(row, next_raw);
          next_raw = end_raw(row + 1);
          if (rend != pos) break;
          zero_row(row);  // a row without edges
        }
        request_old();
      }
      stop = pos == len ? kFar : min(rend, len);
    };

    const int longest = G == 32 ? len : __reduce_max_sync(0xffffffffu, len);
    load_batch(0);
    for (int p = 0; p < longest; p += U) {
      const int in_batch = p & 31;
      if (in_batch == 0) {
        __syncwarp();
#pragma unroll
        for (int j = 0; j < IB; ++j) {
          my_ids[j * G + lg] = id_nxt[j];
          if (VALMODE == 1) my_vals[j * G + lg] = val_nxt[j];
        }
        __syncwarp();
        load_batch(p + 32);
      }
      // the rows of edges [p, p + U)
      Words<W> v[U][NV];
      constexpr int W4 = U < 4 ? U : 4;
      uint32_t ids[W4];
      float vals[W4];
      float ev[kPerHead ? U : 1][kPerHead ? NV : 1];
      const float *weights = kPerHead ? a.edge_val + static_cast<uint64_t>(begin + p) * static_cast<uint32_t>(kHeads > 0 ? kHeads : a.heads) : nullptr;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (u % W4 == 0) load_ids(ids, my_ids + in_batch + u);
        const uint64_t off = static_cast<uint64_t>(ids[u % W4]) * pitch;
#pragma unroll
        for (int q = 0; q < NV; ++q) load_row_bytes<VB>(v[u][q], xq[q] + off);
        if constexpr (kPerHead) {
#pragma unroll
          for (int q = 0; q < NV; ++q) {
            if constexpr (kHeads > 0)
              ev[u][q] = __ldg(weights + head[q] + u * kHeads);
            else
              ev[u][q] = p + u < len ? __ldg(weights + u * a.heads + head[q]) : 0.f;
          }
        }
      }
      // adds them; groups that have passed the end of their tile add into accumulators that nobody reads
      auto add = [&](int u) {
        if (VALMODE == 1 && u % W4 == 0) load_ids(vals, my_vals + in_batch + u);
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          if constexpr (VALMODE == 0 || VALMODE == 3 || VALMODE == 4)
            acc[q].add(v[u][q]);
          else if constexpr (VALMODE == 1)
            acc[q].fma(v[u][q], vals[u % W4]);
          else
            acc[q].fma(v[u][q], ev[u][q]);
        }
      };
      // no row ends among the U edges of any group (not worth asking with four groups: one of them nearly always has one)
      if (NG <= 2 && !__any_sync(0xffffffffu, stop - p <= U)) {
#pragma unroll
        for (int u = 0; u < U; ++u) add(u);
      } else {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          add(u);
          if (p + u + 1 == stop) event(p + u + 1);
        }
      }
    }
    t_next = __shfl_sync(0xffffffffu, t_next, 0) + lane / G;
  }
}

// Lane layouts: vectors per row -> (lanes per tile, loads per lane, edges in flight per lane, resident CTAs per SM).
// 512 bytes in flight per row and lane group and 32 warps per SM where 64 registers hold them: 7, 6 and 5 CTAs measured
// 3 to 25 % slower on 128- to 512-byte rows, twice the edges per step (128 registers) 40 %, and two steps in flight with
// half the edges each 30 %. Narrow fp32 rows read one word at a time (F = 47) want four edges per step, not eight.
// With resident_tiles set nothing is launched: it receives the tiles that are walked at the same time.
template <typename T, int VB, int VALMODE, bool COPY = false>
bool launch_width(const WalkArgs &a, bool share, cudaStream_t st, int *resident_tiles) {
  const int n = (a.row_bytes + VB - 1) / VB;
  auto go = [&](auto kernel, int g, int ctas) {
    const int per_cta = kThreads / g;
    if (resident_tiles != nullptr) {
      *resident_tiles = kNumSM * ctas * per_cta;
      return true;
    }
    int64_t grid = (a.max_tiles + per_cta - 1) / per_cta;
    const int64_t resident = kNumSM * (share ? ctas / 2 : ctas);
    if (grid > resident) grid = resident;
    return launch_dependent(kernel, static_cast<unsigned>(grid < 1 ? 1 : grid), kThreads, 0, st, a) == cudaSuccess;
  };
#define CXG_WALK(G, NV, U, CTAS) \
  if (n <= G * NV)               \
  return go(spmm_walk<T, VB, G, NV, U, VALMODE, CTAS, COPY>, G, CTAS)
  if constexpr (VB == 16) {
    CXG_WALK(8, 1, 8, 8);
    CXG_WALK(16, 1, 8, 8);
    CXG_WALK(32, 1, 8, 8);
    CXG_WALK(32, 2, 4, 8);
    CXG_WALK(32, 4, 2, 6);
  } else if constexpr (VB == 8) {
    CXG_WALK(8, 1, 8, 8);
    CXG_WALK(16, 1, 8, 8);
    CXG_WALK(16, 2, 4, 8);
    CXG_WALK(32, 2, 4, 8);
    CXG_WALK(32, 4, 4, 6);
    CXG_WALK(32, 8, 2, 5);
  } else {
    CXG_WALK(8, 1, 8, 8);
    CXG_WALK(8, 2, 8, 8);
    CXG_WALK(16, 2, 8, 8);
    CXG_WALK(16, 3, 4, 8);
    CXG_WALK(16, 4, 4, 8);
    CXG_WALK(32, 3, 4, 8);
    CXG_WALK(32, 4, 4, 7);
    CXG_WALK(32, 6, 4, 6);
    CXG_WALK(32, 8, 4, 5);
  }
#undef CXG_WALK
  return false;
}

template <typename T, int VB>
bool launch(const WalkArgs &a, int valmode, bool share, cudaStream_t st, int *resident_tiles) {
  if (valmode == 0) return launch_width<T, VB, 0>(a, share, st, resident_tiles);
  if (valmode == 1) return launch_width<T, VB, 1>(a, share, st, resident_tiles);
  if (valmode == 3) return launch_width<T, VB, 3>(a, share, st, resident_tiles);
  if (valmode == 4) return launch_width<T, VB, 4>(a, share, st, resident_tiles);
  if constexpr (sizeof(T) == 4 && VB == 16) {
    if (valmode == 5) return launch_width<T, VB, 5>(a, share, st, resident_tiles);
    if (valmode == 6) return launch_width<T, VB, 6>(a, share, st, resident_tiles);
    if (valmode == 7) return launch_width<T, VB, 7>(a, share, st, resident_tiles);
  }
  return launch_width<T, VB, 2>(a, share, st, resident_tiles);
}

// Rows copied to whole 16-byte vectors: sums, means and sums weighted by one value per edge.
template <typename T>
bool launch_copy(const WalkArgs &a, int valmode, bool share, cudaStream_t st, int *resident_tiles) {
  if (valmode == 0) return launch_width<T, 16, 0, true>(a, share, st, resident_tiles);
  if (valmode == 1) return launch_width<T, 16, 1, true>(a, share, st, resident_tiles);
  if (valmode == 3) return launch_width<T, 16, 3, true>(a, share, st, resident_tiles);
  return false;
}

}  // namespace walk
}  // namespace cxg
