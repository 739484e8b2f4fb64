// tcgen05, tensor memory, TMA and mbarrier operations of gemm_f32.cu: operands of rows of 128 bytes, 128-byte swizzle.
#pragma once
#include "common.cuh"
#include <cuda.h>

#define TC_POLLS (1u << 24)

__device__ __forceinline__ unsigned tc_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tc_bar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_smem(bar)), "r"(count));
}
__device__ __forceinline__ void tc_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem(bar)) : "memory");
}
__device__ __forceinline__ void tc_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc_smem(bar)), "r"(bytes) : "memory");
}
// true when the phase with this parity has completed; false when the wait (or an earlier one of the CTA) ran out
__device__ __forceinline__ bool tc_wait(unsigned long long* bar, unsigned parity, volatile int* dead, unsigned backoff_ns = 0,
                                        unsigned polls = TC_POLLS) {
  return qd_mbar_wait_bounded(tc_smem(bar), parity, dead, polls, 2000000000ull, backoff_ns);
}
// the same without a call
__device__ __forceinline__ bool tc_wait_inline(unsigned long long* bar, unsigned parity, volatile int* dead, unsigned backoff_ns = 0) {
  return qd_mbar_wait_loop(tc_smem(bar), parity, dead, TC_POLLS, 2000000000ull, backoff_ns);
}
// x: innermost coordinate in elements (of whole 128 bytes here), y: row
__device__ __forceinline__ void tc_load_2d(void* dst, const CUtensorMap* map, int x, int y, unsigned long long* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(tc_smem(dst)), "l"(map), "r"(tc_smem(bar)), "r"(x), "r"(y) : "memory");
}
// A K-major tile of rows of 128 bytes with the 128-byte swizzle, groups of 8 rows 1024 bytes apart
__device__ __forceinline__ unsigned long long tc_desc_sw128(unsigned addr) {
  return (unsigned long long)((addr & 0x3FFFF) >> 4) | 1ull << 16 | (unsigned long long)(1024 >> 4) << 32 | 1ull << 46 | 2ull << 61;
}
// bfloat16 operands, both K-major, float32 accumulator, M x N
__device__ __forceinline__ unsigned tc_idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(m >> 4) << 24);
}
__device__ __forceinline__ void tc_mma_bf16(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, bool accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}\n"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(0u) : "memory");
}
// the same with A in tensor memory: 128 lanes, two neighbouring k a column
__device__ __forceinline__ void tc_mma_bf16_tmem(unsigned d, unsigned a, unsigned long long b, unsigned idesc, bool accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n}\n"
      ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(0u) : "memory");
}
// true for one lane of a whole warp
__device__ __forceinline__ bool tc_elect() {
  unsigned p;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
  return p;
}
__device__ __forceinline__ void tc_commit(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(bar)) : "memory");
}
// a whole warp; cols a power of two, 32 to 512
__device__ __forceinline__ void tc_alloc(unsigned* slot, unsigned cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(slot)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(unsigned tmem, unsigned cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_ld8(unsigned addr, unsigned (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(addr));
}
__device__ __forceinline__ void tc_st8(unsigned addr, const unsigned (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n"
               ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---- host: tensor maps
typedef CUresult (*TcEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static TcEncodeFn tc_encode_fn() {
  static TcEncodeFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = (TcEncodeFn)p;
  }
  return fn;
}
// rows x cols bfloat16 or float32, rows ``ld`` elements apart (0: contiguous); boxes of box_rows rows of 128 bytes, 128-byte
// swizzle, zeros outside
static bool tc_make_map(CUtensorMap* map, const void* base, bool bfloat16, long long rows, long long cols, int box_rows,
                        long long ld = 0) {
  TcEncodeFn fn = tc_encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(ld ? ld : cols) * (bfloat16 ? 2 : 4)};
  cuuint32_t box[2] = {bfloat16 ? 64u : 32u, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, bfloat16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims,
            strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
