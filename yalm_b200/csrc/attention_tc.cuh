// What the tcgen05 prefill attention kernels share (attention_tc.cu, attention_exact_tc.cu): tile sizes, TMA
// loads, operand descriptors, products issued by one lane of a whole warp, and loads and stores of
// tensor memory.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>

#include <type_traits>

#include "common.cuh"

namespace yalm {

constexpr int TA_BM = 128;     // query rows per tile; a block takes two tiles
constexpr int TA_BN = 64;      // keys per iteration
constexpr int TA_THREADS = 352;
constexpr int TA_MMA_B = 10;   // the warp that issues tile B's products (warp 1: tile A's)
constexpr int TA_KSTAGES = 3;
constexpr int TA_VSTAGES = 3;
constexpr float TA_RAISE = 8.f;   // a block's maximum may exceed the reference by this much (log2)

__device__ __forceinline__ void ta_tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y,
                                               uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// K-major operand tile: rows of 128 bytes (64 bf16), 128-byte swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t ta_desc_k(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// MN-major operand (V as TMA stores it: one row per key, 64 head elements = 128 bytes per
// row, the next 64 head elements `lbo` bytes further): 8-key groups 1024 B apart
__device__ __forceinline__ uint64_t ta_desc_mn(uint32_t addr, uint32_t lbo) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// A product issued from a whole warp: every lane runs the (uniform) descriptor arithmetic, so
// it can stay in uniform registers, and the instruction itself is issued by the lane whose
// `leader` is set.  (Inside a branch that one lane takes, every operand goes from a vector
// register to a uniform one, one transfer after the other: about 80 clocks per instruction.)
__device__ __forceinline__ void ta_umma_by(uint32_t leader, uint32_t tmem_d, uint64_t adesc,
                                           uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, q;\nsetp.ne.b32 p, %4, 0;\nsetp.ne.b32 q, %5, 0;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(leader)
      : "memory");
}
// ... with the A operand in tensor memory (row m in lane m, two 16-bit elements per column)
__device__ __forceinline__ void ta_umma_tmem_a_by(uint32_t leader, uint32_t tmem_d, uint32_t tmem_a,
                                                  uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, q;\nsetp.ne.b32 p, %4, 0;\nsetp.ne.b32 q, %5, 0;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(leader)
      : "memory");
}
__device__ __forceinline__ void ta_commit_by(uint32_t leader, uint32_t bar) {
  asm volatile(
      "{\n.reg .pred q;\nsetp.ne.b32 q, %1, 0;\n"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}"
      ::"r"(bar), "r"(leader) : "memory");
}
__device__ __forceinline__ void ta_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
// The same load without the wait: several can be in flight; ta_ld_wait32 then makes
// the registers of one of them (and, by the instruction's meaning, of all earlier
// ones) valid, and ta_ld_after32 ties the registers of another to that point.
__device__ __forceinline__ void ta_ld32_issue(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
#define YALM_R32(r)                                                                              \
  "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), \
  "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),       \
  "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),     \
  "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),     \
  "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
__device__ __forceinline__ void ta_ld_wait32(uint32_t* r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" : YALM_R32(r) : : "memory");
}
__device__ __forceinline__ void ta_ld_after32(uint32_t* r) {
  asm volatile("" : YALM_R32(r) : : "memory");
}
#undef YALM_R32
__device__ __forceinline__ void ta_st32(uint32_t taddr, const float* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])),
        "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])),
        "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
        "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])),
        "r"(__float_as_uint(v[11])), "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])),
        "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15])), "r"(__float_as_uint(v[16])),
        "r"(__float_as_uint(v[17])), "r"(__float_as_uint(v[18])), "r"(__float_as_uint(v[19])),
        "r"(__float_as_uint(v[20])), "r"(__float_as_uint(v[21])), "r"(__float_as_uint(v[22])),
        "r"(__float_as_uint(v[23])), "r"(__float_as_uint(v[24])), "r"(__float_as_uint(v[25])),
        "r"(__float_as_uint(v[26])), "r"(__float_as_uint(v[27])), "r"(__float_as_uint(v[28])),
        "r"(__float_as_uint(v[29])), "r"(__float_as_uint(v[30])), "r"(__float_as_uint(v[31]))
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ float ta_ex2(float x) {            // 2^x; 2^-inf = 0
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// V's rows of a key block that lie beyond what the sequence owns (another sequence's rows of the step, rows of
// the cache or of the pooled rows that this sequence has not written, the next block of rows where a capacity is
// no multiple of 64) come with a whole-block copy.  Their weights are zero, but zero times an infinity or a NaN
// is a NaN, so such a block is completed in two steps: its copy arrives on `landed`, and the producer warp clears
// the rows whose bit in `live` is not set before it completes `full`, which the product waits for.  (A row of
// 128 bytes keeps its place under the swizzle, which only permutes 16-byte pieces inside it.)  Called by a whole
// warp; false if a wait gave up.
template <int HD>
__device__ __forceinline__ bool ta_clear_foreign_rows(uint32_t v_block, uint64_t live, uint32_t landed, uint32_t parity,
                                                      uint32_t full, int lane, volatile int* abort_flag) {
  if (!__all_sync(0xffffffffu, mbar_wait(landed, parity, abort_flag))) return false;
#pragma unroll
  for (int sub = 0; sub < HD / 64; ++sub)
#pragma unroll 4
    for (int r = lane >> 3; r < TA_BN; r += 4)
      if (!((live >> r) & 1))
        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};"
                     ::"r"(v_block + (uint32_t)(sub * (TA_BN * 128) + r * 128 + (lane & 7) * 16)), "r"(0) : "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (lane == 0) mbar_arrive(full);
  return true;
}

typedef CUresult (*TaEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                               const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline TaEncodeFn ta_encode_fn() {
  static TaEncodeFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<TaEncodeFn>(p);
  }
  return fn;
}
// rows x cols of a 16-bit type, row-major; box = box_rows rows x 64 columns, 128-byte swizzle
inline int ta_make_map(CUtensorMap* map, const void* ptr, long long rows, long long cols,
                       int box_rows, bool half) {
  TaEncodeFn fn = ta_encode_fn();
  if (!fn) return -10;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, half ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                  const_cast<void*>(ptr), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -11;
}

}  // namespace yalm
