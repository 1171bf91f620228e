// What the tcgen05 product kernels share: bounded waits on mbarriers, the shared-memory descriptor of a K-major tile, the
// driver's tensor-map encoder.
#pragma once
#include "common.cuh"
#include <cuda.h>
#include <cudaTypedefs.h>

namespace {

constexpr int G_WAIT_LIMIT = 1 << 20;   // tries of at most 2 microseconds each

__device__ __forceinline__ unsigned g_smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// false: the wait ran out, or (abort_flag given) another warp of the block gave up
__device__ __forceinline__ bool g_wait(unsigned bar, unsigned parity, const volatile int* abort_flag) {
  for (int i = 0; i < G_WAIT_LIMIT; ++i) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(bar), "r"(parity), "r"(2000u) : "memory");   // a try sleeps 2 microseconds at most
    if (ok) return true;
    if (abort_flag && (i & 255) == 255 && *abort_flag) return false;
  }
  return false;
}
__device__ __forceinline__ void g_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ unsigned long long g_desc(unsigned saddr) {      // K-major, 128-byte swizzle, 8-row groups of 1024 bytes
  unsigned long long d = 0;
  d |= (unsigned long long)((saddr & 0x3FFFF) >> 4);
  d |= (unsigned long long)(16 >> 4) << 16;
  d |= (unsigned long long)(1024 >> 4) << 32;
  d |= 1ull << 46;
  d |= 2ull << 61;
  return d;
}
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  }
  return fn;
}
}  // namespace
