// What the tensor-core kernels share: matrix descriptors, the instructions, mbarriers with bounded waits, tensor maps.
#pragma once
#include <cuda.h>  // CUtensorMap and its enums; the encoder is obtained through the runtime, nothing links libcuda

#include "common.cuh"

namespace cxg {
namespace tc {

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// Shared-memory matrix descriptors, K-major with a swizzle: a tile is cut along K into spans of 128, 64 or 32 bytes; a
// span holds its rows one behind the other, 8-row groups 8 * span bytes apart, and permutes the 16-byte chunks of a row by
// the row number, so that the tensor core reads 8 rows without bank conflicts. A span starts on a multiple of 8 * span
// bytes; K advances inside it by adding 32 bytes to the address. (As core matrices of 8 rows x 16 bytes without a swizzle,
// which is how the copies wrote A and W before, an instruction took some 230 cycles and the tensor core bounded the kernel:
// fp32, 2.33 M gathered rows, K = 128, N = 64 took 837 us, 564 us now; K = 64, N = 128: 495 us, now 364.)
// What is constant in a descriptor:
__device__ __forceinline__ uint64_t desc_base(int span_log) {
  uint64_t d = 0;
  d |= 1ull << 16;                                                  // leading offset: unused with a swizzle, canonical value 1
  d |= static_cast<uint64_t>((128u << span_log) >> 4) << 32;        // next 8-row group
  d |= 1ull << 46;                                                  // descriptor version of sm_100
  d |= static_cast<uint64_t>(span_log == 3 ? 2 : span_log == 2 ? 4 : 6) << 61;  // 128-, 64- or 32-byte swizzle
  return d;
}
__device__ __forceinline__ uint64_t make_desc(uint64_t base, uint32_t addr) { return base | ((addr >> 4) & 0x3fff); }
// byte offset of 16-byte chunk c of a row inside a tile whose spans are span_bytes apart
__device__ __forceinline__ uint32_t swizzled(int row, int c, int span_log, uint32_t span_bytes) {
  const uint32_t in = (c ^ (row >> (3 - span_log))) & ((1 << span_log) - 1);
  return (c >> span_log) * span_bytes + (static_cast<uint32_t>(row) << (span_log + 4)) + (in << 4);
}

// One tiled 2-D bulk tensor copy global -> shared (x = element column, y = row of the tensor map's matrix); its bytes
// are counted on `bar`. x * element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}

// v = hi + lo + what two bits of v cannot hold: hi the upper 19 bits of v, which the tensor core reads from v itself, as it
// ignores the other 13 of a word; lo = v - hi (exact, at most 13 significant bits) moved half a unit of its 19 bits up in
// magnitude, so that it is read rounded. Cut instead, every product would be short by 1e-7 of itself on the same side. (The
// addition turns a NaN, which lo is where v is infinite, into -0; hi carries infinities and NaN alone.)
__device__ __forceinline__ float tf32_rest(float v) {
  const float hi = __uint_as_float(__float_as_uint(v) & 0xffffe000u);
  return __uint_as_float(__float_as_uint(v - hi) + 0x1000u);
}

// Instruction descriptor: fp32 accumulate, A and B of format `fmt` (1 = bf16, 2 = tf32), both K-major.
__device__ __forceinline__ uint32_t make_idesc(int fmt, int m, int n) {
  uint32_t d = 0;
  d |= 1u << 4;                                 // D format: f32
  d |= static_cast<uint32_t>(fmt) << 7;         // A format
  d |= static_cast<uint32_t>(fmt) << 10;        // B format
  d |= static_cast<uint32_t>(n >> 3) << 17;     // N / 8
  d |= static_cast<uint32_t>(m >> 4) << 24;     // M / 16
  return d;
}

// One MMA of a warp: every lane comes here with the same operands and one of them issues it. (Behind `if (lane == 0)` the
// compiler cannot tell that the operands are the same in all active lanes and an instruction took 134 cycles whatever its
// size; issued this way 73, and 135 for 128 x 256, which is the tensor core's own time.)
template <bool TF32>
__device__ __forceinline__ void mma_ss(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  if (TF32)
    asm volatile(
        "{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait on phase `parity`; false after a time-out here or an abort raised by another role.
__device__ __forceinline__ bool wait_bar(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int32_t *status,
                                         long long limit) {
  const uint32_t b = smem_addr(bar);
  if (mbar_try_wait(b, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(b, parity)) {
    if (*abort_flag) return false;
    if (clock64() - t0 > limit) {
      *abort_flag = 1;
      atomicExch(status, 1);
      return false;
    }
  }
  return true;
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// Arrival on `bar` once the MMAs that this warp has issued are done (issued by the lane that issues the MMAs).
__device__ __forceinline__ void commit_to(uint64_t *bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_addr(bar))
      : "memory");
}

// Where a role stands in a ring of stages: the stage, and how often it has gone round. (Stage and round as remainder and
// quotient of a 64-bit unit counter cost every role two software divisions per unit, more than the unit's MMAs.)
struct Ring {
  int size, stage = 0;
  uint32_t round = 0;
  __device__ explicit Ring(int n) : size(n) {}
  __device__ void next() {
    if (++stage == size) stage = 0, ++round;
  }
  __device__ bool reused() const { return round > 0; }
  __device__ uint32_t filled() const { return round & 1; }        // parity of the phase that fills the stage this time
  __device__ uint32_t emptied() const { return (round & 1) ^ 1; }  // parity of the phase that emptied it after the last time
  // Parity of the last phase of stage i that this role has begun; false: none
  __device__ bool last(int i, uint32_t *parity) const {
    *parity = (i < stage ? round : round - 1) & 1;
    return i < stage || round > 0;
  }
};

// 16 consecutive 32-bit columns of this warp's 32 accumulator lanes; completion is awaited by the caller
__device__ __forceinline__ void tmem_ld16(uint32_t *v, uint32_t taddr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}

// 8 columns
__device__ __forceinline__ void tmem_ld8(uint32_t *v, uint32_t taddr) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}

// one column
__device__ __forceinline__ void tmem_ld1(uint32_t *v, uint32_t taddr) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v[0]) : "r"(taddr));
}

__device__ __forceinline__ void st_global_v4(void *p, uint4 v) {
  asm volatile("st.global.v4.b32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// Tensor map of a row-major [rows][k] matrix of bf16 or fp32 elements for boxes of box_rows rows x one 128-byte swizzle
// span of columns (64 / 32 elements). False when the driver's encoder is not available or refuses the arguments.
inline bool encode_a_map(CUtensorMap *map, const void *base, int64_t rows, int k, int elem, int box_rows) {
  typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                               const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const EncodeFn fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<EncodeFn>(p);
    (void)cudaGetLastError();
    return static_cast<EncodeFn>(nullptr);
  }();
  if (fn == nullptr) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k) * elem};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / elem), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t estr[2] = {1, 1};
  return fn(map, elem == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void *>(base),
            dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace tc
}  // namespace cxg
