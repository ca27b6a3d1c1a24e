// Bulk copies (cp.async.bulk) with mbarrier completion and a bounded wait,
// and the lane-group reductions shared by the tiled bond loops.
#pragma once

#include <cstdint>

namespace pdgpu {
namespace {

constexpr unsigned kWaitTries = 1u << 22;  // bounded mbarrier wait

__device__ __forceinline__ uint32_t sa(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void bar_init(uint64_t *bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sa(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// orders this CTA's earlier shared-memory accesses before later bulk-copy writes
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void bar_arrive_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sa(bar)), "r"(bytes)
               : "memory");
}
// both addresses 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          sa(dst)),
      "l"(src), "r"(bytes), "r"(sa(bar))
      : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(sa(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// true once the phase of the given parity completed; false after kWaitTries attempts
__device__ __forceinline__ bool bar_wait(uint64_t *bar, uint32_t parity) {
  for (unsigned t = 0; t < kWaitTries; t++)
    if (bar_try(bar, parity)) return true;
  return false;
}

// Reductions over one node's group of LPN consecutive lanes.  All 32 lanes of
// the warp call them together (one full mask): with a mask per group the
// groups of a warp part company at the first vote or shuffle and run one
// after the other from there on (FP64 bond loop at 8 lanes per node, 2-D
// compression of 333 000 nodes: 363 us with a mask per group, 169 us with one;
// FP32 form in 3-D, pre-pass 100 and 85 us).
// LPN = 0: `lanes` of them, a power of two up to 32, known at run time.
constexpr unsigned kFullWarp = 0xffffffffu;

template <int LPN>
__device__ __forceinline__ double gsum(double v, int lanes = LPN) {
#pragma unroll
  for (int o = (LPN ? LPN : lanes) / 2; o > 0; o >>= 1) v += __shfl_xor_sync(kFullWarp, v, o);
  return v;
}
template <int LPN>
__device__ __forceinline__ float gmax(float v) {
#pragma unroll
  for (int o = LPN / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFullWarp, v, o));
  return v;
}

// does any bond of [b0, b1) (bit positions in a bitmap) start broken?
template <int LPN>
__device__ __forceinline__ bool any_broken(const uint32_t *bits, int b0, int b1, int lanes = LPN) {
  const int lpn = LPN ? LPN : lanes, lane = threadIdx.x & (lpn - 1);
  const int w0 = b0 >> 5, w1 = (b1 - 1) >> 5;
  bool hit = false;
  if (b1 > b0)
    for (int w = w0 + lane; w <= w1; w += lpn) {
      uint32_t m = bits[w];
      if (w == w0) m &= ~0u << (b0 & 31);
      if (w == w1) m &= ~0u >> (31 - ((b1 - 1) & 31));
      hit |= m != 0u;
    }
  if constexpr (LPN == 1) return hit;
  const unsigned all = __ballot_sync(kFullWarp, hit);
  // the group's lanes of the 32
  return ((all >> (threadIdx.x & 31u & ~(lpn - 1u))) & (kFullWarp >> (32 - lpn))) != 0u;
}

}  // namespace
}  // namespace pdgpu
