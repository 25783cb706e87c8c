// Launch accounting, programmatic dependent launch and CTA helpers shared by the
// kernel files.  Everything here is internal to each translation unit.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "ooc_internal.h"

namespace ooc {
namespace {

constexpr unsigned FULL = 0xffffffffu;

// Counts one launch and brackets it with the timing hooks of the calling
// thread's launch state, when one is installed.
struct KScope {
  const char* name;
  cudaStream_t st;
  LaunchState* ls;
  KScope(const char* n, cudaStream_t s) : name(n), st(s), ls(current_launch_state()) {
    if (!ls) return;
    ls->launches++;
    if (ls->hooks.begin) ls->hooks.begin(ls->hooks.user, name, st);
  }
  ~KScope() {
    if (ls && ls->hooks.end) ls->hooks.end(ls->hooks.user, name, st);
  }
};

// Programmatic dependent launch.  Every kernel here first waits until the
// grid before it on the stream has finished and its memory is visible, then
// lets the grid after it launch, so that grid's CTAs take the SMs this one's
// last CTAs free instead of waiting for the whole grid to drain.  Without the
// launch attribute (launch_k with ooc_tuning::pdl off) both are no-ops.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" :::);
}

// Launch `k` on `st`, with programmatic stream serialization when the calling
// thread's launch state asks for it.
template <typename... P, typename... A>
void launch_k(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  const LaunchState* ls = current_launch_state();
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = (ls && ls->pdl) ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k, std::forward<A>(args)...);
}

inline unsigned grid_for(uint64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

template <typename T>
__device__ __forceinline__ T warp_inclusive(T v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = __shfl_up_sync(FULL, v, o);
    if (lane >= o) v += y;
  }
  return v;
}

// Exclusive scan of one value per thread across the CTA; `total` gets the CTA sum.
template <typename T>
__device__ __forceinline__ T block_exclusive(T v, T& total) {
  __shared__ T warp_sums[33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const T inc = warp_inclusive(v);
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const T w = lane < nw ? warp_sums[lane] : T(0);
    const T wi = warp_inclusive(w);
    if (lane < nw) warp_sums[lane] = wi - w;
    if (lane == 31) warp_sums[32] = wi;
  }
  __syncthreads();
  const T r = inc - v + warp_sums[warp];
  total = warp_sums[32];
  __syncthreads();
  return r;
}

// Bit k set when byte k of w is non-zero.  The product moves the bytes' flags (bits 7, 15, 23,
// 31) to bits 28..31; its other terms fall on distinct lower bits or leave the word.
__device__ __forceinline__ uint32_t nonzero_bytes(uint32_t w) {
  const uint32_t t = (((w & 0x7f7f7f7fu) + 0x7f7f7f7fu) | w) & 0x80808080u;
  return (t * 0x00204081u) >> 28;
}

// The last index w < n of a non-decreasing array with at(w) <= r (at(0) <= r), by the whole
// warp: every step reads 32 entries at once, so 8,192 words take three dependent loads.
template <typename F>
__device__ __forceinline__ uint32_t warp_search(uint32_t n, uint32_t r, int lane, F at) {
  uint32_t lo = 0, step = 1;
  while (step * 32u < n) step *= 32u;
  for (;; step /= 32u) {
    const uint32_t i = lo + (uint32_t)lane * step;
    lo += (uint32_t)(__popc(__ballot_sync(FULL, i < n && at(i) <= r)) - 1) * step;
    if (step == 1) return lo;
  }
}

// ---- batched launches: a prefix of CTA counts maps each CTA to its stripe, whose
// job the CTA copies into shared memory ----
template <typename T>
__device__ __forceinline__ void stage(T& dst, const T& src) {
  static_assert(sizeof(T) % 4 == 0, "staged structs are word-sized");
  const uint32_t* s = reinterpret_cast<const uint32_t*>(&src);
  uint32_t* d = reinterpret_cast<uint32_t*>(&dst);
  for (uint32_t q = threadIdx.x; q < sizeof(T) / 4; q += blockDim.x) d[q] = s[q];
}

// CTA b belongs to the stripe s with cta_beg[s] <= b < cta_beg[s+1]; it is
// the stripe's CTA b - cta_beg[s] and covers the elements per CTA of its launch
// from there.  Every warp searches by itself, 32 stripes a probe: one thread's bisection
// held the CTA for up to ten loads in a row.
__device__ __forceinline__ uint32_t cta_stripe(const uint64_t* __restrict__ cta_beg, uint32_t n, uint64_t& cta) {
  const uint32_t s = warp_search(n, blockIdx.x, threadIdx.x & 31, [&](uint32_t i) { return cta_beg[i]; });
  cta = (uint64_t)(blockIdx.x - cta_beg[s]);  // the CTA's index within its stripe
  return s;
}

}  // namespace
}  // namespace ooc
