// Thin inline-PTX helpers for TMA (cp.async.bulk.tensor) and mbarriers on
// sm_103a, plus host-side tensor-map encoding through the driver entry point
// (no link-time dependency on libcuda).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace mtr {

// ---- device ----------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// Invalidate an mbarrier with no pending operations before re-initialising it.
__device__ __forceinline__ void mbar_inval(uint64_t* bar) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: gives up after max_iter polls (each poll may suspend briefly
// in hardware) and reports failure instead of spinning forever.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint32_t max_iter) {
  for (uint32_t i = 0; i < max_iter; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// Programmatic dependent launch.  A kernel launched with launch_overlapped is
// set up and started while the kernel before it in the stream ends: up to
// stream_wait() it reads only its arguments and tables that were copied to the
// device and writes nothing in global memory; every thread that touches other
// data comes through the wait, which ends when the kernels before it have
// completed and what they wrote is visible.  It returns a zero that the
// compiler cannot see; the pointers of the read-only loads that follow take it
// as an offset, so that none of those loads moves above the wait.  The CTAs are
// not let in any earlier (griddepcontrol.launch_dependents): those of a small
// grid then crowd on the SMs that empty first (10 SIRT iterations at
// 128x128x32: 0.72 against 0.60 ms).  What it hides is the launch itself, 1-2 us
// of each: 256x256x64, 61 angles, 8 iterations 2.01 -> 1.94 ms; two leaning axes
// of 192x160x48 1.68 -> 1.65 ms.
__device__ __forceinline__ long long stream_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  long long zero = 0;
  asm volatile("" : "+l"(zero)::"memory");
  return zero;
}

template <typename... P, typename... Q>
inline void launch_overlapped(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Q&&... q) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kern, static_cast<P>(q)...);  // (a failure is the caller's cudaGetLastError, as with <<<>>>)
}

// Smallest e with 2^e >= w, for a finite w > 0.
__device__ __forceinline__ int log2_ceil(float w) {
  int e;
  const float m = frexpf(w, &e);  // w = m 2^e, m in [0.5, 1)
  return m == 0.5f ? e - 1 : e;
}

// 3-D tiled TMA load of one box into shared memory, completing on bar.
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

// 3-D tiled TMA reduce-add of a shared-memory box into global memory.
__device__ __forceinline__ void tma_reduce_add_3d(const CUtensorMap* map, const void* src, int x, int y, int z) {
  asm volatile(
      "cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2, %3}], [%4];"
      ::"l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(src))
      : "memory");
}

__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Generic-proxy shared-memory writes -> visible to the async (TMA) proxy.
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// Named barrier among `count` threads (count multiple of 32), id 1..15.
__device__ __forceinline__ void named_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// ---- host --------------------------------------------------------------------
// Encodes a 3-D tiled tensor map over [depth][height][width] elements with a
// row pitch of `pitch` elements; box = (bw, bh, 1); out-of-bounds reads fill 0.
// Returns false when the driver entry point is unavailable or the encoding is
// rejected (the caller then uses the non-TMA kernels).
bool encode_tensor_map_3d(CUtensorMap* map, const void* base, bool half, int width, int pitch, int height,
                          int depth, int bw, int bh);

}  // namespace mtr
