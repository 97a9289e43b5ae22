// What the warm start's tensor-core kernels share (unet.cu, conv.cu): mbarriers with bounded waits, TMA tile loads,
// shared-memory descriptors and the instruction descriptor of tcgen05 kind::f16 with BF16 operands, the state of the
// producer / MMA / epilogue pipeline, and the driver's tensor-map encoder.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include "common.cuh"

namespace blml {

constexpr int NN_BM = 128, NN_BK = 64;

__device__ __forceinline__ uint32_t nn_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void nn_mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(nn_smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void nn_mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(nn_smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool nn_mbar_wait(uint64_t* bar, uint32_t parity) {
  for (long it = 0; it < (1L << 20); it++) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(nn_smem_u32(bar)), "r"(parity) : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void nn_tma_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               :: "r"(nn_smem_u32(dst)), "l"(map), "r"(c0), "r"(c1), "r"(nn_smem_u32(bar)) : "memory");
}
// K-major, 128-byte-swizzled operand tile: 8-row core groups 1024 bytes apart
__device__ __forceinline__ uint64_t nn_desc(const void* p) {
  const uint64_t addr = nn_smem_u32(p);
  uint64_t d = 0;
  d |= (addr >> 4) & 0x3FFFull;
  d |= (uint64_t)(16 >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// kind::f16 instruction descriptor: D f32, A and B bf16, both K-major, M = 128, N = n
__host__ __device__ constexpr uint32_t idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(NN_BM >> 4) << 24);
}

constexpr int NN_PIPE_THREADS = 192, NN_MAX_STAGES = 8;

struct NNPipeShared {
  uint64_t full[NN_MAX_STAGES], empty[NN_MAX_STAGES], tfull[2], tempty[2];
  uint32_t tslot;
  int abort;
  long long issued, consumed;           // K slices loaded by the producer / taken by the MMA issuer
};

__device__ __forceinline__ bool nn_wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort) {
  for (long it = 0; it < (1L << 20); it++) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(nn_smem_u32(bar)), "r"(parity) : "memory");
    if (done) return true;
    if ((it & 63) == 63 && abort && *abort) return false;
  }
  return false;
}

__device__ __forceinline__ void nn_fail(volatile int* abort, int* err) {
  *abort = 1;
  atomicExch(err, 1);
}

typedef CUresult (*NNEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                               const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline NNEncodeFn nn_encode() {
  static NNEncodeFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<NNEncodeFn>(p);
  }
  return fn;
}

}  // namespace blml
