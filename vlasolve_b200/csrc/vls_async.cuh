// vls_async.cuh -- shared-memory mbarriers and asynchronous (TMA / bulk)
// copies used by the step kernels.  No copy here multicasts across a
// cluster; every wait on an mbarrier is bounded.
#pragma once
#include <cstdint>

#include <cuda.h>
#include <cuda_runtime.h>

#include "vls_internal.h"

namespace vls {


__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_test_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// non-blocking polls with a short sleep between them, at most MBAR_SPIN_LIMIT
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity,
                                                  uint32_t limit = MBAR_SPIN_LIMIT) {
  for (uint32_t i = 0; i < limit; ++i) {
    if (mbar_test_wait(bar, parity)) return true;
    if (i >= 32) __nanosleep(20);
  }
  return false;
}
// the same for warps that wait for microseconds next to working ones, whose
// issue slots closer polls would take
__device__ __forceinline__ bool mbar_wait_idle(uint64_t *bar, uint32_t parity,
                                               uint32_t limit = MBAR_SPIN_LIMIT) {
  for (uint32_t i = 0; i < limit; ++i) {
    if (mbar_test_wait(bar, parity)) return true;
    __nanosleep(100);
  }
  return false;
}
// brings [src, src + bytes) into L2 (both multiples of 16)
__device__ __forceinline__ void bulk_prefetch_l2(const void *src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// 3D tiled TMA load (no multicast) of one box into shared memory
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *tm, int x, int y,
                                            int z, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}
// untiled bulk copy global -> shared (16-byte aligned addresses, size a
// multiple of 16), completing on an mbarrier's transaction count
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes,
                                          uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// untiled bulk copy shared -> global in the thread's bulk async-group
__device__ __forceinline__ void bulk_store(void *dst, const void *src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
               "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// the thread's committed bulk stores have finished reading shared memory
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

// ------------------------------------------------------- chained launches
// The kernels of a step follow one another in a stream.  A chained launch is
// set up while the previous kernel runs and starts its blocks when that
// kernel's blocks have left; chain_begin(), before a kernel's first access to
// global memory, waits until the previous kernel is complete and its writes
// are visible.  Every kernel launched this way does so first, so that what
// lies before the previous kernel is complete as well.  About 3 us less
// between two kernels: a step of 33 x 33 x 8 35 -> 25 us, 257 x 257 x 128
// FP32 124 -> 114, 513 x 513 x 256 617 -> 604.
//
// What the previous kernels of the stream wrote (f, G, C, shift, partial, the
// chains' rings, the adjoint's fields) is read by plain loads through pointers
// that are not __restrict__: the read-only path (__ldg, or what the compiler
// makes of a const __restrict__ argument) is for data that stays constant over
// the kernel's whole life, which here begins before those writes are visible,
// and such a load may be scheduled above the wait.  Tables that no kernel of a
// step writes may keep it.
//
// No kernel lets the next one's blocks in earlier (launch_dependents): they
// would run on SMs whose split of shared memory and L1 is still the previous
// kernel's (201 x 201 x 200 FP64 177 -> 233 us a step, 513 x 513 x 256 604 ->
// 666).
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
// Each argument converts to its parameter implicitly (the kernel alone names
// the parameter types), as in a <<<>>> launch: no pointer passes for another
// type's.  Returns the launch's error, and leaves none behind for the next
// cudaGetLastError of an unrelated call.
template <typename P>
struct ChainArg {
  using type = P;
};
template <typename... P>
inline cudaError_t chain_launch(void (*kern)(P...), dim3 grid, dim3 block, size_t smem,
                                cudaStream_t st, const typename ChainArg<P>::type &...args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&c, kern, args...);
  const cudaError_t last = cudaGetLastError();
  return e != cudaSuccess ? e : last;
}

}  // namespace vls
