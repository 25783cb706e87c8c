// CUDA kernels of the partition -> voxelize -> SVO-build path (sm_103a).
//
// Compiled with -fmad=false; FP32 arithmetic additionally goes through the
// __f*_rn intrinsics so that each operation rounds once, as in the
// reference's x86-64 build.
#include <cuda_runtime.h>

#include <cstring>
#include <utility>

#include "ooc_device.cuh"
#include "ooc_internal.h"
#include "ooc_launch.cuh"

namespace ooc {

namespace {
thread_local LaunchState* t_launch = nullptr;  // the state of the call running on this thread
}  // namespace

LaunchState* current_launch_state() { return t_launch; }
LaunchScope::LaunchScope(LaunchState* s) : prev(t_launch) { t_launch = s; }
LaunchScope::~LaunchScope() { t_launch = prev; }

namespace {
constexpr int SCAN_THREADS = 256;

// ===========================================================================
// Exclusive scan (three phases: per-CTA reduce, scan of CTA sums, down-sweep)
// ===========================================================================
constexpr int SCAN_ITEMS = 16;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

template <typename T>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const T* __restrict__ in, uint64_t n,
                                                              T* __restrict__ partials) {
  pdl_enter();
  const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
  T v = 0;
#pragma unroll
  for (int q = 0; q < SCAN_ITEMS; q++) {
    const uint64_t i = base + (uint64_t)q * SCAN_THREADS + threadIdx.x;
    if (i < n) v += in[i];
  }
  T total;
  block_exclusive(v, total);
  if (threadIdx.x == 0) partials[blockIdx.x] = total;
}

// Also partials[np] = the grand total.
template <typename T>
__global__ void __launch_bounds__(1024) k_scan_partials(T* partials, uint64_t np) {
  pdl_enter();
  T carry = 0;
  for (uint64_t base = 0; base < np; base += blockDim.x) {
    const uint64_t i = base + threadIdx.x;
    const T v = i < np ? partials[i] : T(0);
    T total;
    const T ex = block_exclusive(v, total);
    if (i < np) partials[i] = ex + carry;
    carry += total;
  }
  if (threadIdx.x == 0) partials[np] = carry;
}

// Each thread scans SCAN_ITEMS consecutive elements staged through shared memory
// (`partials` NULL: a single tile, nothing before it).
template <typename T>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_down(T* data, uint64_t n, const T* __restrict__ partials) {
  pdl_enter();
  // the elements are counts: a zero total means all zero, which is already their scan
  if (partials && partials[gridDim.x] == T(0)) return;
  __shared__ T tile[SCAN_TILE + SCAN_TILE / 32];
  const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
#pragma unroll
  for (int q = 0; q < SCAN_ITEMS; q++) {
    const uint32_t li = q * SCAN_THREADS + threadIdx.x;
    const uint64_t i = base + li;
    tile[li + li / 32] = i < n ? data[i] : T(0);
  }
  __syncthreads();
  T v[SCAN_ITEMS];
  T sum = 0;
#pragma unroll
  for (int q = 0; q < SCAN_ITEMS; q++) {
    const uint32_t li = threadIdx.x * SCAN_ITEMS + q;
    v[q] = tile[li + li / 32];
    sum += v[q];
  }
  T total;
  T run = block_exclusive(sum, total) + (partials ? partials[blockIdx.x] : T(0));
#pragma unroll
  for (int q = 0; q < SCAN_ITEMS; q++) {
    const uint32_t li = threadIdx.x * SCAN_ITEMS + q;
    tile[li + li / 32] = run;
    run += v[q];
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < SCAN_ITEMS; q++) {
    const uint32_t li = q * SCAN_THREADS + threadIdx.x;
    const uint64_t i = base + li;
    if (i < n) data[i] = tile[li + li / 32];
  }
}

template <typename T>
void scan_exclusive(T* data, uint64_t n, T* partials, cudaStream_t st) {
  if (n == 0) return;
  const unsigned nb = (unsigned)((n + SCAN_TILE - 1) / SCAN_TILE);
  if (nb == 1) {  // one tile: one launch
    KScope k("scan_down", st);
    launch_k(k_scan_down<T>, dim3(1), dim3(SCAN_THREADS), 0, st, data, n, nullptr);
    return;
  }
  {
    KScope k("scan_reduce", st);
    launch_k(k_scan_reduce<T>, dim3(nb), dim3(SCAN_THREADS), 0, st, data, n, partials);
  }
  {
    KScope k("scan_partials", st);
    launch_k(k_scan_partials<T>, dim3(1), dim3(1024), 0, st, partials, nb);
  }
  {
    KScope k("scan_down", st);
    launch_k(k_scan_down<T>, dim3(nb), dim3(SCAN_THREADS), 0, st, data, n, partials);
  }
}

// ===========================================================================
// Partition binning (partitioner.cpp:101-149 with BBoxBuffer.h:70-84)
// ===========================================================================
struct WorldBox {
  float lo[3], hi[3];
};

__device__ __forceinline__ WorldBox tri_world_box(const float* __restrict__ tris, uint64_t t, int stride) {
  const TriVerts tv = load_verts(tris, t, stride);
  WorldBox b;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    b.lo[a] = smin(tv.v[0][a], smin(tv.v[1][a], tv.v[2][a]));
    b.hi[a] = smax(tv.v[0][a], smax(tv.v[1][a], tv.v[2][a]));
  }
  return b;
}

// Per axis, the partitions j whose world slab [lo_j, hi_j] passes the reference's inclusive test,
// !(hi < lo_j) && !(lo > hi_j), form one contiguous run [j0, j1]: the slabs' bounds grow with j, so what
// fails the second test comes first and what fails the first comes last.  (A NaN passes everywhere.)
__device__ __forceinline__ bool axis_run(float lo, float hi, const float* alo, const float* ahi, int PA, int& j0, int& j1) {
  j0 = 0;
  j1 = PA - 1;
  for (int j = 0; j < PA; j++) {
    j0 += lo > ahi[j] ? 1 : 0;
    j1 -= hi < alo[j] ? 1 : 0;
  }
  return j0 <= j1;
}

// The slabs' bounds of the three axes, lower and then upper, into shared memory.
__device__ __forceinline__ void stage_axes(float* dst, const float* __restrict__ axis_lo, const float* __restrict__ axis_hi,
                                           int PA) {
  for (int i = threadIdx.x; i < 3 * PA; i += blockDim.x) {
    dst[i] = axis_lo[i];
    dst[3 * PA + i] = axis_hi[i];
  }
}

// Per-axis partition runs of triangle t, packed 7 bits per bound with bit 63 set,
// or 0 when the triangle passes no partition's box test.
__device__ __forceinline__ uint64_t part_runs(const float* __restrict__ tris, int stride, uint64_t t, const float* axes,
                                              int PA) {
  const WorldBox b = tri_world_box(tris, t, stride);
  int x0, x1, y0, y1, z0, z1;
  const bool x = axis_run(b.lo[0], b.hi[0], axes, axes + 3 * PA, PA, x0, x1);
  const bool y = axis_run(b.lo[1], b.hi[1], axes + PA, axes + 4 * PA, PA, y0, y1);
  const bool z = axis_run(b.lo[2], b.hi[2], axes + 2 * PA, axes + 5 * PA, PA, z0, z1);
  if (!(x && y && z)) return 0ull;
  return (uint64_t)x0 | ((uint64_t)x1 << 7) | ((uint64_t)y0 << 14) | ((uint64_t)y1 << 21) | ((uint64_t)z0 << 28) |
         ((uint64_t)z1 << 35) | (1ull << 63);
}

__device__ __forceinline__ int run_bound(uint64_t r, int k) { return (int)((r >> (7 * k)) & 127u); }

template <typename F>
__device__ __forceinline__ void each_part(uint64_t r, F f) {
  if (!r) return;
  for (int jx = run_bound(r, 0); jx <= run_bound(r, 1); jx++)
    for (int jy = run_bound(r, 2); jy <= run_bound(r, 3); jy++)
      for (int jz = run_bound(r, 4); jz <= run_bound(r, 5); jz++) f(morton_local(jx, jy, jz));
}

// Bound by the additions to the partitions' counters (64 of them on the 20M-triangle soup), which finish
// about 3 ns apart each: a block adds a partition's triangles once, so it takes `per` times 256 of them.
// The two passes of that soup take 0.20 + 0.27 ms with 4,096 triangles a block and 0.40 + 0.42 with 256.
constexpr int kPartCta = 256, kPartMax = 16;  // 8 is the same

__global__ void __launch_bounds__(kPartCta) k_part_count(const float* __restrict__ tris, int stride, uint64_t n_tris,
                                                         const float* __restrict__ axis_lo,
                                                         const float* __restrict__ axis_hi, int pa_bits,
                                                         uint32_t n_parts, uint32_t* __restrict__ hist, int use_smem,
                                                         int per) {
  pdl_enter();
  extern __shared__ float axes[];
  const int PA = 1 << pa_bits;
  uint32_t* const sh = reinterpret_cast<uint32_t*>(axes + 6 * PA);
  stage_axes(axes, axis_lo, axis_hi, PA);
  if (use_smem)
    for (uint32_t i = threadIdx.x; i < n_parts; i += kPartCta) sh[i] = 0;
  __syncthreads();
  uint32_t* const to = use_smem ? sh : hist;
  for (int k = 0; k < per; k++) {
    const uint64_t t = ((uint64_t)blockIdx.x * per + k) * kPartCta + threadIdx.x;
    if (t < n_tris) each_part(part_runs(tris, stride, t, axes, PA), [&](uint32_t p) { atomicAdd(&to[p], 1u); });
  }
  if (use_smem) {
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n_parts; i += kPartCta)
      if (sh[i]) atomicAdd(&hist[i], sh[i]);
  }
}

__global__ void __launch_bounds__(kPartCta) k_part_emit(const float* __restrict__ tris, int stride, uint64_t n_tris,
                                                        const float* __restrict__ axis_lo,
                                                        const float* __restrict__ axis_hi, int pa_bits,
                                                        uint32_t n_parts, uint32_t* __restrict__ cursor,
                                                        uint32_t* __restrict__ items, int use_smem, int per) {
  pdl_enter();
  extern __shared__ uint64_t runs[];  // of the block's triangles
  const int PA = 1 << pa_bits;
  float* const axes = reinterpret_cast<float*>(runs + (use_smem ? per * kPartCta : 0));
  uint32_t* const cnt = reinterpret_cast<uint32_t*>(axes + 6 * PA);  // their number per partition, then where they go
  const uint64_t t0 = (uint64_t)blockIdx.x * per * kPartCta;
  stage_axes(axes, axis_lo, axis_hi, PA);
  if (use_smem)
    for (uint32_t i = threadIdx.x; i < n_parts; i += kPartCta) cnt[i] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < per * kPartCta; i += kPartCta) {
    const uint64_t r = t0 + i < n_tris ? part_runs(tris, stride, t0 + i, axes, PA) : 0ull;
    if (use_smem) {
      runs[i] = r;
      each_part(r, [&](uint32_t p) { atomicAdd(&cnt[p], 1u); });
    } else {
      each_part(r, [&](uint32_t p) { items[atomicAdd(&cursor[p], 1u)] = (uint32_t)(t0 + i); });
    }
  }
  if (!use_smem) return;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < n_parts; i += kPartCta)
    if (cnt[i]) cnt[i] = atomicAdd(&cursor[i], cnt[i]);
  __syncthreads();
  for (int i = threadIdx.x; i < per * kPartCta; i += kPartCta)
    each_part(runs[i], [&](uint32_t p) { items[atomicAdd(&cnt[p], 1u)] = (uint32_t)(t0 + i); });
}

// ---------------------------------------------------------------------------
// Out-of-core binning: the records of a group of consecutive partitions
// [p0, p0 + gp), gathered from one chunk of the triangle stream into the
// group's buffer, each partition's records contiguous and in stream order (the
// order of the reference's per-partition .tripdata files, partitioner.cpp:
// 101-149), so a smaller record index within a partition is an earlier
// triangle.  CTAs of kStreamCta triangles; mat[q * n_cta + cta] is CTA cta's
// count for group partition q, whose exclusive scan places every CTA's records.
// ---------------------------------------------------------------------------
constexpr int kStreamCta = (int)kStreamCtaTris;

__global__ void __launch_bounds__(kStreamCta) k_stream_count(const float* __restrict__ tris, int stride, uint64_t n,
                                                             const float* __restrict__ axis_lo,
                                                             const float* __restrict__ axis_hi, int pa_bits,
                                                             uint32_t p0, uint32_t gp, uint32_t* __restrict__ mat,
                                                             uint32_t n_cta) {
  pdl_enter();
  extern __shared__ float axes[];
  const int PA = 1 << pa_bits;
  uint32_t* const cnt = reinterpret_cast<uint32_t*>(axes + 6 * PA);
  stage_axes(axes, axis_lo, axis_hi, PA);
  for (uint32_t q = threadIdx.x; q < gp; q += kStreamCta) cnt[q] = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) mat[(uint64_t)gp * n_cta] = 0;  // the scan's total entry
  __syncthreads();
  const uint64_t t = (uint64_t)blockIdx.x * kStreamCta + threadIdx.x;
  if (t < n) {
    each_part(part_runs(tris, stride, t, axes, PA), [&](uint32_t p) {
      if (p - p0 < gp) atomicAdd(&cnt[p - p0], 1u);
    });
  }
  __syncthreads();
  for (uint32_t q = threadIdx.x; q < gp; q += kStreamCta) mat[(uint64_t)q * n_cta + blockIdx.x] = cnt[q];
}

// Each record goes to base[q] + (its CTA's place among the chunk's records of q) +
// (the CTA's earlier triangles that are in q).
__global__ void __launch_bounds__(kStreamCta) k_stream_emit(const float* __restrict__ tris, int stride, uint64_t n,
                                                            const float* __restrict__ axis_lo,
                                                            const float* __restrict__ axis_hi, int pa_bits,
                                                            uint32_t p0, uint32_t gp, const uint32_t* __restrict__ mat,
                                                            uint32_t n_cta, const uint64_t* __restrict__ base,
                                                            float* __restrict__ out) {
  pdl_enter();
  extern __shared__ float axes[];
  __shared__ uint64_t runs[kStreamCta];
  const int PA = 1 << pa_bits;
  stage_axes(axes, axis_lo, axis_hi, PA);
  __syncthreads();
  const uint64_t t = (uint64_t)blockIdx.x * kStreamCta + threadIdx.x;
  const uint64_t r = t < n ? part_runs(tris, stride, t, axes, PA) : 0ull;
  runs[threadIdx.x] = r;
  __syncthreads();
  if (!r) return;
  const float* src = tris + t * (uint64_t)stride;
  for (int jx = run_bound(r, 0); jx <= run_bound(r, 1); jx++)
    for (int jy = run_bound(r, 2); jy <= run_bound(r, 3); jy++)
      for (int jz = run_bound(r, 4); jz <= run_bound(r, 5); jz++) {
        const uint32_t q = morton_local(jx, jy, jz) - p0;
        if (q >= gp) continue;
        uint32_t rank = 0;
        for (uint32_t k = 0; k < threadIdx.x; k++) {
          const uint64_t o = runs[k];
          rank += (o >> 63) && run_bound(o, 0) <= jx && jx <= run_bound(o, 1) && run_bound(o, 2) <= jy &&
                  jy <= run_bound(o, 3) && run_bound(o, 4) <= jz && jz <= run_bound(o, 5);
        }
        const uint64_t row = (uint64_t)q * n_cta;
        const uint64_t dst = base[q] + (mat[row + blockIdx.x] - mat[row]) + rank;
        float* d = out + dst * (uint64_t)stride;
        for (int k = 0; k < stride; k++) d[k] = src[k];
      }
}

__global__ void k_stream_bases(const uint32_t* __restrict__ part_off, uint32_t p0, uint32_t gp,
                               uint64_t* __restrict__ base) {
  pdl_enter();
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < gp) base[q] = (uint64_t)(part_off[p0 + q] - part_off[p0]);
}

// After a chunk: every group partition's next record moves past the chunk's records of it.
__global__ void k_stream_advance(const uint32_t* __restrict__ mat, uint32_t n_cta, uint32_t gp,
                                 uint64_t* __restrict__ base) {
  pdl_enter();
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < gp) base[q] += mat[(uint64_t)(q + 1) * n_cta] - mat[(uint64_t)q * n_cta];
}

// ===========================================================================
// Voxelization (voxelizer.cpp:168-306)
//
// Pass 0 sets the Morton-ordered occupancy bits of the stripe; pass 1 (payload
// mode) keeps, per set voxel, the smallest passing triangle index, which is
// the reference's first-writer-wins rule (voxelizer.cpp:263, 293-299).  For a
// small item pass 0 also stores which of its (at most 64) candidates passed,
// so pass 1 only ranks those voxels instead of testing again.
// ===========================================================================
__device__ __forceinline__ bool item_box(const VoxJob& j, const TriVerts& tv, int lo[3], int hi[3]) {
  int gmin[3], gmax[3];
  grid_box(tv, j.unit_div, gmin, gmax);
#pragma unroll
  for (int a = 0; a < 3; a++) {
    // clamp to the partition (voxelizer.cpp:199-204), then keep the part in this stripe
    lo[a] = clampi(gmin[a], j.pa[a], j.pb[a]);
    hi[a] = clampi(gmax[a], j.pa[a], j.pb[a]);
    lo[a] = lo[a] < j.sa[a] ? j.sa[a] : lo[a];
    hi[a] = hi[a] > j.sb[a] ? j.sb[a] : hi[a];
  }
  return lo[0] <= hi[0] && lo[1] <= hi[1] && lo[2] <= hi[2];
}

// Sets `acc` in leaf word w and marks the word's 256-bit block, so every
// block with a set bit is marked.  The mark is a plain byte store: threads
// that mark the same block store the same value, and nothing reads the marks
// before the launch ends.
__device__ __forceinline__ void set_leaf(const VoxJob& j, uint32_t w, uint32_t acc) {
  atomicOr(&j.leafbits[w], acc);
  if (j.leaftouch) j.leaftouch[w >> 3] = 1;
}

// Rank of bit `b` among the set bits of the leaf level: the set bits before its
// 32-brick word, before its block within the word's bricks, before its leaf word
// within the block (all from the brick pass), and one popcount.
__device__ __forceinline__ uint32_t leaf_rank(const VoxJob& j, uint32_t b) {
  const uint32_t blk = b >> 8;
  const uint4 r = __ldg(reinterpret_cast<const uint4*>(j.blocks) + blk);
  const uint64_t woff = (uint64_t)r.x | ((uint64_t)r.y << 32);
  const uint32_t before = (uint32_t)(woff >> (8 * ((b >> 5) & 7u))) & 0xffu;
  return j.wpre[b >> 17].x + r.z + before + __popc(j.leafbits[b >> 5] & ((1u << (b & 31)) - 1u));
}

// Offers triangle t to voxel m: the smallest index wins, and the voxel's Morton code
// travels with it to the leaf payload pass, which then needs no search for it.
__device__ __forceinline__ void offer(const VoxJob& j, uint32_t m, uint32_t t) {
  atomicMin(&j.winners[leaf_rank(j, m)], ((unsigned long long)t << 32) | m);
}

__device__ __forceinline__ uint64_t item_triangle(const VoxJob& j, uint64_t i) {
  return j.item_tri ? (uint64_t)j.item_tri[j.ibeg + i] : j.ibeg + i;
}

// ---------------------------------------------------------------------------
// Large items walk lines along the axis of their largest normal component.  On
// every line the voxels that pass the plane test form one run (walk_line), so
// a line costs its run plus a few probes instead of its whole length; every
// voxel of the run still gets the complete test, so the result is the
// reference's candidate loop (voxelizer.cpp:257-305) voxel for voxel.
// ---------------------------------------------------------------------------

// Axis of the largest component of cross(e0, e1); the listing of the items and the
// walk call this same function, so they agree on the lines of every item.
__device__ __forceinline__ int walk_axis(const TriVerts& t) {
  const float e0x = t.v[1][0] - t.v[0][0], e0y = t.v[1][1] - t.v[0][1], e0z = t.v[1][2] - t.v[0][2];
  const float e1x = t.v[2][0] - t.v[1][0], e1y = t.v[2][1] - t.v[1][1], e1z = t.v[2][2] - t.v[1][2];
  const float ax = fabsf(e0y * e1z - e0z * e1y), ay = fabsf(e0z * e1x - e0x * e1z), az = fabsf(e0x * e1y - e0y * e1x);
  if (az >= ax && az >= ay) return 2;
  return ax >= ay ? 0 : 1;
}

// Lines of a large item: the box extents across the walk axis.
__device__ __forceinline__ uint64_t item_lines(int W, const int lo[3], const int hi[3]) {
  const uint64_t ex = (uint64_t)(hi[0] - lo[0] + 1), ey = (uint64_t)(hi[1] - lo[1] + 1),
                 ez = (uint64_t)(hi[2] - lo[2] + 1);
  return W == 0 ? ey * ez : (W == 1 ? ex * ez : ex * ey);
}

// The list of large items.  Pass 0 appends every large item once: to `large` when its
// lines make one task (at most `slice` lines), else to `big`, whose entries carry the number
// of their first task so that several warps share the item.  A full `big` (ctr[kCtrBig]'s
// count at its capacity) sends further items to `large`, where one warp walks them whole.
// The lists serve both passes; their order does not matter to the result.  Calls of the allocation-free
// pass that overlap share its lists and find each other's counts and items there, which may cost them
// voxels but no access out of range: additions past a list's end are dropped, and so are items that the
// job does not have.
//
// kCtrBig packs the entries (low kBigCountBits bits) and the tasks (the others) reserved so
// far, so one atomicAdd gives an entry and its first task in step.  A thread adds only after
// it has read a count below the capacity, so the count passes the capacity by at most the
// threads resident at once (below 2^19) and never reaches the tasks' bits.
constexpr int kBigCountBits = 20;
static_assert(kMaxBig + (1u << 19) < (1u << kBigCountBits), "the count stays in its bits");

// Item i of job j with more than `slice` lines: whether it went to `big`.
__device__ __forceinline__ bool append_big(const VoxJob& j, uint64_t i, uint32_t lines) {
  const unsigned long long now = *reinterpret_cast<volatile unsigned long long*>(j.ctr + kCtrBig);
  if ((now & ((1ull << kBigCountBits) - 1ull)) >= j.big_cap) return false;
  const uint32_t tasks = (lines + j.slice - 1u) / j.slice;
  const unsigned long long got = atomicAdd(j.ctr + kCtrBig, ((unsigned long long)tasks << kBigCountBits) | 1ull);
  const uint32_t slot = (uint32_t)got & ((1u << kBigCountBits) - 1u);
  if (slot >= j.big_cap) return false;
  j.big[slot] = make_uint4((uint32_t)(j.item0 + i), j.stripe, (uint32_t)(got >> kBigCountBits), tasks);
  return true;
}

// Every thread of a warp (CTA false) or of the CTA (of at most kChunk threads): item i of job j with
// `lines` lines, 0 for an item that is not large.  One atomic per CTA: additions to one address
// finish about 3 ns apart, and one per warp took all of the pass's time on the large soups (0.47 of
// 0.47 ms for 4M triangles).
template <bool CTA>
__device__ __forceinline__ void append_large(const VoxJob& j, uint64_t i, uint32_t lines) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool one = lines != 0 && !(lines > j.slice && append_big(j, i, lines));
  const uint32_t m = __ballot_sync(FULL, one);
  unsigned long long at = 0;
  if constexpr (CTA) {
    __shared__ uint32_t s_cnt[kChunk / 32];
    __shared__ unsigned long long s_at;
    if (lane == 0) s_cnt[warp] = __popc(m);
    const uint32_t total = (uint32_t)__syncthreads_count(one);
    if (total == 0) return;
    if (threadIdx.x == 0) s_at = atomicAdd(j.ctr + kCtrLarge, (unsigned long long)total);
    uint32_t before = 0;
    for (int k = 0; k < warp; k++) before += s_cnt[k];
    __syncthreads();
    at = s_at + before;
  } else {
    if (!m) return;
    if (lane == 0) at = atomicAdd(j.ctr + kCtrLarge, (unsigned long long)__popc(m));
    at = __shfl_sync(FULL, at, 0);
  }
  at += __popc(m & ((1u << lane) - 1u));
  if (one && at < j.large_cap) j.large[at] = (uint32_t)(j.item0 + i) | ((unsigned long long)j.stripe << 32);
}

// (x, y, z) -> (a, b, w): w the axis W, a and b the ones that follow it cyclically.
template <typename T>
__device__ __forceinline__ void turn(int W, T& x, T& y, T& z) {
  const T x0 = x, y0 = y, z0 = z;
  x = W == 2 ? x0 : (W == 0 ? y0 : z0);
  y = W == 2 ? y0 : (W == 0 ? z0 : x0);
  z = W == 2 ? z0 : (W == 0 ? x0 : y0);
}

// p[0..2] of the rotated axes (a, b, w), summed in the reference's order: w = z: a, b, w are
// x, y, z; w = x: y, z, x; w = y: z, x, y.
__device__ __forceinline__ float sum3(int W, float pa, float pb, float pw) {
  if (W == 2) return __fadd_rn(__fadd_rn(pa, pb), pw);
  return W == 0 ? __fadd_rn(__fadd_rn(pw, pa), pb) : __fadd_rn(__fadd_rn(pb, pw), pa);
}

// The constants of the test (voxelizer.cpp:207-254) with the coordinates rotated to (a, b, w).
__device__ __forceinline__ void tri_setup_rotated(const TriVerts& t, float u, int W, TriSetup& s) {
  float e[3][3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    e[0][a] = __fsub_rn(t.v[1][a], t.v[0][a]);
    e[1][a] = __fsub_rn(t.v[2][a], t.v[1][a]);
    e[2][a] = __fsub_rn(t.v[0][a], t.v[2][a]);
  }
  s.n[0] = __fsub_rn(__fmul_rn(e[0][1], e[1][2]), __fmul_rn(e[0][2], e[1][1]));
  s.n[1] = __fsub_rn(__fmul_rn(e[0][2], e[1][0]), __fmul_rn(e[0][0], e[1][2]));
  s.n[2] = __fsub_rn(__fmul_rn(e[0][0], e[1][1]), __fmul_rn(e[0][1], e[1][0]));
  const float r = __fdiv_rn(1.0f, __fsqrt_rn(sum3(W, __fmul_rn(s.n[0], s.n[0]), __fmul_rn(s.n[1], s.n[1]),
                                                  __fmul_rn(s.n[2], s.n[2]))));
#pragma unroll
  for (int a = 0; a < 3; a++) s.n[a] = __fmul_rn(s.n[a], r);
  float c1[3], c2[3];  // critical point and its opposite, minus the first vertex
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float c = s.n[a] > 0.0f ? u : 0.0f;
    c1[a] = __fmul_rn(s.n[a], __fsub_rn(c, t.v[0][a]));
    c2[a] = __fmul_rn(s.n[a], __fsub_rn(__fsub_rn(u, c), t.v[0][a]));
  }
  s.d1 = sum3(W, c1[0], c1[1], c1[2]);
  s.d2 = sum3(W, c2[0], c2[1], c2[2]);
  edge_setup(t, e, u, s);
}

// Two floats that go through one instruction, each with its own rounding.  A packed product whose only
// use is a packed sum is contracted to an FMA, whatever the compiler's flags and the .rn say (measured:
// the results differ), so a product that goes into a sum is an FMA itself, with -0 (which changes no
// product, signed zeros included) that the compiler cannot know: nz = minus_zero of a run-time value.
struct F2 {
  uint64_t v;
};
__device__ __forceinline__ F2 f2(float x, float y) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {  // never into a sum
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b, F2 nz) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(nz.v));
  return r;
}
__device__ __forceinline__ F2 minus_zero(uint32_t small) {  // any run-time value below 2^31
  const float z = __uint_as_float(0x80000000u | (small >> 31));
  return f2(z, z);
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ void split(F2 a, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
}

// A large item as the warp's lanes read it, in words of 16 bytes: the constants of the test with the
// coordinates turned so that the walk axis w comes last (the edge tests are cyclic in the axes, and sums
// of two products commutative, so that changes no rounding).  Of the three projections (a, b) is the
// line's own test, (a, w) and (b, w) go through the walk as pairs.
struct __align__(16) WalkItem {
  F2 ea, eb;                   // line test ea * a + eb * b + ed: of edges 0 and 1
  F2 ed;
  float ea2, eb2;              // and of edge 2
  float ed2, u;
  int alo, blo;                // clamped box
  uint32_t shape;              // lines along a (11 bits) | axis w << 11 | monotone << 13
  uint32_t magic;              // floor(c / ea) = (c * magic) >> 32 for line numbers c < 2^20; 0: one line along a
  uint32_t first;              // the first line of the task, less the lines of the items before it
  uint32_t tri;
  F2 w[3], f[3], d[3];         // edge k on (a, w) and (b, w): w * (w, w) + f * (a, b) + d
  F2 dd;                       // the plane's offsets d1, d2
  float nw, na, nb, inv_dir;   // normal
  int wlo, whi;
  uint32_t local;              // stripe-local alo, blo, wlo, 10 bits each
  uint32_t stripe;
};
static_assert(sizeof(WalkItem) == 44 * 4, "eight lanes that read 16 bytes of eight items in a row hit different banks");

__device__ __forceinline__ void walk_setup(const VoxJob& j, const TriVerts& tv, uint64_t t, uint32_t stripe, uint32_t first,
                                           int W, const int lo[3], const int hi[3], WalkItem& r) {
  TriVerts v = tv;
  int l[3] = {lo[0], lo[1], lo[2]}, h[3] = {hi[0], hi[1], hi[2]}, o[3] = {j.sa[0], j.sa[1], j.sa[2]};
#pragma unroll
  for (int k = 0; k < 3; k++) turn(W, v.v[k][0], v.v[k][1], v.v[k][2]);
  turn(W, l[0], l[1], l[2]);
  turn(W, h[0], h[1], h[2]);
  turn(W, o[0], o[1], o[2]);
  const float u = j.u;
  TriSetup s;
  tri_setup_rotated(v, u, W, s);
  r.ea = f2(s.xy[0][0], s.xy[1][0]), r.eb = f2(s.xy[0][1], s.xy[1][1]), r.ed = f2(s.dxy[0], s.dxy[1]);
  r.ea2 = s.xy[2][0], r.eb2 = s.xy[2][1], r.ed2 = s.dxy[2];
#pragma unroll
  for (int k = 0; k < 3; k++)
    r.w[k] = f2(s.zx[k][0], s.yz[k][1]), r.f[k] = f2(s.zx[k][1], s.yz[k][0]), r.d[k] = f2(s.dzx[k], s.dyz[k]);
  r.dd = f2(s.d1, s.d2);
  r.nw = s.n[2], r.na = s.n[0], r.nb = s.n[1];
  r.u = u;
  r.inv_dir = 1.0f / (s.n[2] * u);
  r.alo = l[0], r.blo = l[1], r.wlo = l[2], r.whi = h[2];
  r.local = (uint32_t)(l[0] - o[0]) | ((uint32_t)(l[1] - o[1]) << 10) | ((uint32_t)(l[2] - o[2]) << 20);
  const uint32_t ea = (uint32_t)(h[0] - l[0] + 1);
  const int top = max(hi[0], max(hi[1], hi[2]));
  const bool mono = monotone_setup(s, fabsf(__fmul_rn((float)(top + 1), u)));
  r.shape = ea | ((uint32_t)W << 11) | (mono ? 1u << 13 : 0u);
  // ceil(2^32 / ea): its excess adds less than c / 2^32 <= 2^-12 < 1 / ea to the quotient
  r.magic = ea > 1 ? (uint32_t)(0xffffffffu / ea) + 1u : 0u;
  r.first = first;
  r.tri = (uint32_t)t;
  r.stripe = stripe;
}

// spread3_10 of every coordinate, in shared memory: three lookups a line instead of three times eight
// instructions (4.2 and 4.0 ms on the 20M-triangle soup).  By all threads of a CTA.
__device__ __forceinline__ void fill_spread(uint32_t* spread) {
  for (uint32_t i = threadIdx.x; i < 1024u; i += blockDim.x) spread[i] = spread3_10(i);
  __syncthreads();
}

// Line (ra, rb) of a large item: pass 0 sets its bits, pass 1 offers the triangle to every
// voxel it passes.  The line's own projection has passed.
template <int PASS>
__device__ __forceinline__ void walk_line(const VoxJob& j, const WalkItem& r, uint32_t ra, uint32_t rb,
                                          const uint32_t* spread) {
  const float u = r.u, fa = __fmul_rn((float)(r.alo + (int)ra), u), fb = __fmul_rn((float)(r.blo + (int)rb), u);
  const uint32_t shape = r.shape;
  const int W = (int)(shape >> 11) & 3, w0 = r.wlo, w1 = r.whi;
  // n.p in the reference's order, (x + y) + z: with w = z a + b first, with w = x (w + a) + b, with w = y
  // (w + b) + a.  Adding the 0 changes only the sign of a zero, which no test sees.
  const float nw = r.nw, pa = __fmul_rn(r.na, fa), pb = __fmul_rn(r.nb, fb);
  const float q1 = W == 2 ? __fadd_rn(pa, pb) : (W == 0 ? pa : pb), q2 = W == 2 ? 0.0f : (W == 0 ? pb : pa);
  const F2 dd = r.dd, fab = f2(fa, fb), nz = minus_zero(r.shape);
  F2 cw[3], cf[3], cd[3];
#pragma unroll
  for (int k = 0; k < 3; k++) cw[k] = r.w[k], cf[k] = mul2(r.f[k], fab, nz), cd[k] = r.d[k];
  auto at = [&](int w) { return __fmul_rn((float)w, u); };
  auto rest = [&](float fw) {  // the two projections that depend on the walk coordinate; a NaN passes
    const F2 ww = f2(fw, fw);
    float m[6];
#pragma unroll
    for (int k = 0; k < 3; k++) split(add2(add2(mul2(cw[k], ww, nz), cf[k]), cd[k]), m[2 * k], m[2 * k + 1]);
    return !(fminf(fminf(fminf(m[0], m[1]), fminf(m[2], m[3])), fminf(m[4], m[5])) < 0.0f);
  };
  const bool up_side = nw * u > 0.0f;  // the plane value grows with w
  // Where the plane test of voxel w stands: 0 it passes, -1 the passing run lies at larger w, +1 at
  // smaller w.  Every operand of the test is a rounded sum or product of one monotone input, so along the
  // line the rounded plane value moves monotonically, the two offsets keep their order, and the passing
  // voxels form one run; outside it both factors have the sign that says which side it is on.
  auto side = [&](float fw) {
    const float v = __fadd_rn(__fadd_rn(__fmul_rn(nw, fw), q1), q2);
    float a, b;
    split(add2(f2(v, v), dd), a, b);
    if (!(__fmul_rn(a, b) > 0.0f)) return 0;
    return (a > 0.0f) == up_side ? 1 : -1;
  };
  // stripe-local Morton bits: the fixed coordinates, and the walk coordinate moving by carries
  const uint32_t la = (r.local & 1023u) + ra, lb = ((r.local >> 10) & 1023u) + rb, lw = r.local >> 20;
  const uint32_t mab = (spread[la] << (W == 2 ? 0 : W + 1)) | (spread[lb] << (W == 0 ? 2 : W - 1));
  const uint32_t wbits = 0x09249249u << W;
  auto emit = [&](uint32_t mw) {
    const uint32_t m = mab | mw;
    if (PASS == 0) set_leaf(j, m >> 5, 1u << (m & 31u));
    else offer(j, m, r.tri);  // pass 0 set this voxel's bit
  };
  if (!((shape >> 13) & 1u)) {  // every voxel of the line, complete test
    uint32_t mw = spread3_10(lw) << W;
    for (int w = w0; w <= w1; w++, mw = ((mw | ~wbits) + (1u << W)) & wbits) {
      const float fw = at(w);
      if (side(fw) == 0 && rest(fw)) emit(mw);
    }
    return;
  }
  // Start at the voxel nearest to the middle of the run, which is at least one voxel long: only a run
  // that the box cuts off, or rounding, leaves it outside (rounding down instead did for every fourth
  // line of random triangles).
  float d1, d2;
  split(dd, d1, d2);
  float west = -((pa + pb) + 0.5f * (d1 + d2)) * r.inv_dir;
  west = fminf(fmaxf(west, (float)w0), (float)w1);  // NaN becomes w0
  int start = (int)(west + 0.5f), walk = 0;                   // walk: +1 up only, -1 down only, 0 both ways
  const int g0 = side(at(start));
  if (g0 < 0) {  // the run lies above: first w with side >= 0
    int lo = start, hi = -1, step = 1;
    for (;;) {
      const int nx = min(lo + step, w1);
      if (side(at(nx)) >= 0) {
        hi = nx;
        break;
      }
      if (nx == w1) return;
      lo = nx;
      step <<= 1;
    }
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (side(at(mid)) >= 0) hi = mid;
      else lo = mid;
    }
    if (side(at(hi)) != 0) return;  // the run falls between two voxels
    start = hi;
    walk = 1;
  } else if (g0 > 0) {  // below: last w with side <= 0
    int hi = start, lo = -1, step = 1;
    for (;;) {
      const int nx = max(hi - step, w0);
      if (side(at(nx)) <= 0) {
        lo = nx;
        break;
      }
      if (nx == w0) return;
      hi = nx;
      step <<= 1;
    }
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (side(at(mid)) <= 0) lo = mid;
      else hi = mid;
    }
    if (side(at(lo)) != 0) return;
    start = lo;
    walk = -1;
  }
  // that voxel and its neighbours, whose plane tests go through as a pair
  const float fs = at(start);
  float fu, fd, pu, pd;
  const F2 f_ud = mul2(f2((float)(start + 1), (float)(start - 1)), f2(u, u));
  split(f_ud, fu, fd);
  {
    const F2 v = add2(add2(mul2(f2(nw, nw), f_ud, nz), f2(q1, q1)), f2(q2, q2));
    split(mul2(add2(v, f2(d1, d1)), add2(v, f2(d2, d2))), pu, pd);
  }
  const bool up = walk >= 0 && start < w1 && !(pu > 0.0f), down = walk <= 0 && start > w0 && !(pd > 0.0f);
  const uint32_t ms = spread[lw + (uint32_t)(start - w0)] << W;
  uint32_t mu = ((ms | ~wbits) + (1u << W)) & wbits, md = (ms - (1u << W)) & wbits;
  const bool on_s = rest(fs), on_u = up & rest(fu), on_d = down & rest(fd);
  if (PASS == 0) {  // one store per leaf word
    const uint32_t m0 = mab | ms, m1 = mab | mu, m2 = mab | md;
    uint32_t b0 = on_s ? 1u << (m0 & 31u) : 0u, b1 = on_u ? 1u << (m1 & 31u) : 0u, b2 = on_d ? 1u << (m2 & 31u) : 0u;
    if (((m0 ^ m1) >> 5) == 0) b0 |= b1, b1 = 0;
    if (((m0 ^ m2) >> 5) == 0) b0 |= b2, b2 = 0;
    if (b0) set_leaf(j, m0 >> 5, b0);
    if (b1) set_leaf(j, m1 >> 5, b1);
    if (b2) set_leaf(j, m2 >> 5, b2);
  } else {
    if (on_s) emit(ms);
    if (on_u) emit(mu);
    if (on_d) emit(md);
  }
  if (up)
    for (int w = start + 2; w <= w1; w++) {
      const float fw = at(w);
      if (side(fw) != 0) break;
      mu = ((mu | ~wbits) + (1u << W)) & wbits;
      if (rest(fw)) emit(mu);
    }
  if (down)
    for (int w = start - 2; w >= w0; w--) {
      const float fw = at(w);
      if (side(fw) != 0) break;
      md = (md - (1u << W)) & wbits;
      if (rest(fw)) emit(md);
    }
}

// ---------------------------------------------------------------------------
// Small items: the candidate tests by projection.  Of the seven tests of a
// candidate voxel (voxelizer.cpp:266-287) the three XY edge tests depend only
// on (x, y), the YZ tests only on (y, z), the ZX tests only on (z, x); only the
// plane test depends on all three.  Each is a pure function of its
// coordinates, so evaluating it once per distinct projection and reusing the
// result gives the reference's verdict for every candidate, bit for bit; the
// FP32 expressions are the reference's, operation by operation.  A candidate
// passes when all seven pass (the reference's order of early exits only saves
// work).
//
// Small are the boxes of at most small_vol voxels that are at most two wide along two
// axes; w is the third (the longest; z among equals), a and b are the ones that follow
// it cyclically.  The edge tests are cyclic in (x, y, z), so with the coordinates rotated
// to (a, b, w) they read the same for every w; the sums of three products keep the
// reference's order (x + y) + z.  The pass mask of an item has bit (ia * bb + ib) * bw + iw.
//
// Bound by ALU instructions.  One body for every orientation, its voxels' bits merged into
// one store per leaf word, took the pass from 86 to 90 us on a heightfield of 2M triangles,
// where almost every box was already 2 x 2 x w, and from 485 to 246 us on 4M random
// triangles and 282 to 173 us on 128 meshes (with append_large), where two boxes in three
// were not and ran a voxel at a time.
// ---------------------------------------------------------------------------

// A small box: w is walked in 2 x 2 x 2 bricks, every test of a brick evaluated without
// branches; slots outside the box are masked.  (In the rotated coordinates x, y, z below
// stand for a, b, w.)  The Morton bits of a coordinate + 1 come from the carry trick:
// setting every bit outside an axis' positions makes +1 carry across them.
__device__ __forceinline__ uint64_t vox_small_bricks(const VoxJob& j, const TriSetup& s, int W, const int lo[3],
                                                     const uint32_t local[3], uint32_t bx, uint32_t by, uint32_t bz) {
  const float px0 = __fmul_rn((float)lo[0], j.u), px1 = __fmul_rn((float)(lo[0] + 1), j.u);
  const float py0 = __fmul_rn((float)lo[1], j.u), py1 = __fmul_rn((float)(lo[1] + 1), j.u);
  // XY over the four columns (x_i, y_j)
  bool c00 = true, c01 = by > 1, c10 = bx > 1, c11 = bx > 1 && by > 1;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float a0 = __fmul_rn(s.xy[k][0], px0), a1 = __fmul_rn(s.xy[k][0], px1);
    const float b0 = __fmul_rn(s.xy[k][1], py0), b1 = __fmul_rn(s.xy[k][1], py1);
    c00 &= !(__fadd_rn(__fadd_rn(a0, b0), s.dxy[k]) < 0.0f);
    c01 &= !(__fadd_rn(__fadd_rn(a0, b1), s.dxy[k]) < 0.0f);
    c10 &= !(__fadd_rn(__fadd_rn(a1, b0), s.dxy[k]) < 0.0f);
    c11 &= !(__fadd_rn(__fadd_rn(a1, b1), s.dxy[k]) < 0.0f);
  }
  // the plane value's parts per column (see walk_line), and the halves of the YZ and ZX dot
  // products that do not depend on z; two sums go through one instruction (F2): the YZ and ZX
  // tests of a z as one pair, the plane values of two z as another
  const float n0x0 = __fmul_rn(s.n[0], px0), n0x1 = __fmul_rn(s.n[0], px1);
  const float n1y0 = __fmul_rn(s.n[1], py0), n1y1 = __fmul_rn(s.n[1], py1);
  // w = z: (x + y) + z, q the sum of the first two; otherwise (z + q) + r
  const bool z_last = W == 2;
  float q00, q01, q10, q11, r0 = 0.0f, r1 = 0.0f;
  if (z_last) {
    q00 = __fadd_rn(n0x0, n1y0), q01 = __fadd_rn(n0x0, n1y1), q10 = __fadd_rn(n0x1, n1y0), q11 = __fadd_rn(n0x1, n1y1);
  } else if (W == 0) {
    q00 = n0x0, q01 = n0x0, q10 = n0x1, q11 = n0x1;
    r0 = n1y0, r1 = n1y1;  // of y
  } else {
    q00 = n1y0, q01 = n1y1, q10 = n1y0, q11 = n1y1;
    r0 = n0x0, r1 = n0x1;  // of x
  }
  const F2 nz = minus_zero((uint32_t)j.stride);
  F2 cz[3], c0[3], c1[3], cd[3];  // ZX and YZ: of z, of (x_0, y_0), of (x_1, y_1), rest
#pragma unroll
  for (int k = 0; k < 3; k++) {
    cz[k] = f2(s.zx[k][0], s.yz[k][1]);
    c0[k] = f2(__fmul_rn(s.zx[k][1], px0), __fmul_rn(s.yz[k][0], py0));
    c1[k] = f2(__fmul_rn(s.zx[k][1], px1), __fmul_rn(s.yz[k][0], py1));
    cd[k] = f2(s.dzx[k], s.dyz[k]);
  }
  // Morton bits: the rotated axes' shifts are 0, 1, 2 turned by W
  const uint32_t xs = W == 2 ? 0u : (W == 0 ? 1u : 2u), ys = W == 2 ? 1u : (W == 0 ? 2u : 0u), zs = (uint32_t)W;
  const uint32_t XBITS = 0x09249249u << xs, YBITS = 0x09249249u << ys, ZBITS = 0x09249249u << zs;
  const uint32_t mx0 = spread3_10(local[0]) << xs, mx1 = ((mx0 | ~XBITS) + (1u << xs)) & XBITS;
  const uint32_t my0 = spread3_10(local[1]) << ys, my1 = ((my0 | ~YBITS) + (1u << ys)) & YBITS;
  const uint32_t z1 = 1u << zs;
  uint32_t mz = spread3_10(local[2]) << zs;
  // bits in their leaf words, and whether x, y + 1 lie in another word
  const uint32_t mxy = mx0 | my0;
  const bool sx = ((mx0 ^ mx1) >> 5) != 0, sy = ((my0 ^ my1) >> 5) != 0;
  uint64_t mask = 0;
  for (uint32_t zc = 0; zc < bz; zc += 2) {
    const bool z1ok = zc + 1 < bz;
    const float pz0 = __fmul_rn((float)(lo[2] + (int)zc), j.u), pz1 = __fmul_rn((float)(lo[2] + (int)zc + 1), j.u);
    bool y0z0, y0z1, y1z0, y1z1;  // YZ over (y_j, z_k)
    bool z0x0, z0x1, z1x0, z1x1;  // ZX over (z_k, x_i)
    {
      // dot((-e.x, e.z) * fy, (p.z, p.x)) + d and dot((-e.z, e.y) * fx, (p.y, p.z)) + d
      const F2 pzz0 = f2(pz0, pz0), pzz1 = f2(pz1, pz1);
      auto edges = [&](F2 pzz, const F2* c, bool& zx, bool& yz) {  // a NaN passes
        float a[3], b[3];
#pragma unroll
        for (int k = 0; k < 3; k++) split(add2(add2(mul2(cz[k], pzz, nz), c[k]), cd[k]), a[k], b[k]);
        zx = !(fminf(fminf(a[0], a[1]), a[2]) < 0.0f);
        yz = !(fminf(fminf(b[0], b[1]), b[2]) < 0.0f);
      };
      edges(pzz0, c0, z0x0, y0z0);
      edges(pzz0, c1, z0x1, y1z0);
      edges(pzz1, c0, z1x0, y0z1);
      edges(pzz1, c1, z1x1, y1z1);
      y0z1 &= z1ok, y1z1 &= z1ok;
    }
    // the plane test: (n.p + d1) (n.p + d2) > 0 fails
    const F2 g = mul2(f2(s.n[2], s.n[2]), f2(pz0, pz1), nz);
    auto plane = [&](float q, float r, bool& z0, bool& z1) {
      F2 v = add2(g, f2(q, q));
      if (!z_last) v = add2(v, f2(r, r));
      float a, b;
      split(mul2(add2(v, f2(s.d1, s.d1)), add2(v, f2(s.d2, s.d2))), a, b);
      z0 = !(a > 0.0f);
      z1 = !(b > 0.0f);
    };
    bool v000, v001, v010, v011, v100, v101, v110, v111;
    const bool of_y = W == 0;
    plane(q00, r0, v000, v001);
    plane(q01, of_y ? r1 : r0, v010, v011);
    plane(q10, of_y ? r0 : r1, v100, v101);
    plane(q11, r1, v110, v111);
    const bool p000 = c00 & y0z0 & z0x0 & v000, p001 = c00 & y0z1 & z1x0 & v001;
    const bool p010 = c01 & y1z0 & z0x0 & v010, p011 = c01 & y1z1 & z1x0 & v011;
    const bool p100 = c10 & y0z0 & z0x1 & v100, p101 = c10 & y0z1 & z1x1 & v101;
    const bool p110 = c11 & y1z0 & z0x1 & v110, p111 = c11 & y1z1 & z1x1 & v111;
    const uint32_t mz1 = ((mz | ~ZBITS) + z1) & ZBITS;
    if (j.item_mask) {  // payload: two bits per column
      const uint32_t c00b = (p000 ? 1u : 0u) | (p001 ? 2u : 0u), c01b = (p010 ? 1u : 0u) | (p011 ? 2u : 0u);
      const uint32_t c10b = (p100 ? 1u : 0u) | (p101 ? 2u : 0u), c11b = (p110 ? 1u : 0u) | (p111 ? 2u : 0u);
      uint64_t m = (uint64_t)c00b;
      if (by > 1) m |= (uint64_t)c01b << bz;
      if (bx > 1) m |= (uint64_t)c10b << (by * bz);
      if (bx > 1 && by > 1) m |= (uint64_t)c11b << ((by + 1) * bz);
      mask |= m << zc;
    }
    // The eight voxels' bits, merged along every axis whose + 1 stays in the word: one store per
    // leaf word the brick touches (one to eight), the same slot in every lane.
    const bool sz = ((mz ^ mz1) >> 5) != 0;
    auto bit = [&](bool p, uint32_t m) { return p ? 1u << (m & 31u) : 0u; };
    uint32_t b000 = bit(p000, mxy | mz), b001 = bit(p001, mxy | mz1);
    uint32_t b010 = bit(p010, mx0 | my1 | mz), b011 = bit(p011, mx0 | my1 | mz1);
    uint32_t b100 = bit(p100, mx1 | my0 | mz), b101 = bit(p101, mx1 | my0 | mz1);
    uint32_t b110 = bit(p110, mx1 | my1 | mz), b111 = bit(p111, mx1 | my1 | mz1);
    auto merge = [](bool apart, uint32_t& a, uint32_t& b) {
      if (!apart) {
        a |= b;
        b = 0;
      }
    };
    merge(sz, b000, b001), merge(sz, b010, b011), merge(sz, b100, b101), merge(sz, b110, b111);
    merge(sy, b000, b010), merge(sy, b001, b011), merge(sy, b100, b110), merge(sy, b101, b111);
    merge(sx, b000, b100), merge(sx, b001, b101), merge(sx, b010, b110), merge(sx, b011, b111);
    if (b000) set_leaf(j, (mxy | mz) >> 5, b000);
    if (b001) set_leaf(j, (mxy | mz1) >> 5, b001);
    if (b010) set_leaf(j, (mx0 | my1 | mz) >> 5, b010);
    if (b100) set_leaf(j, (mx1 | my0 | mz) >> 5, b100);
    if (b011 | b101 | b110 | b111) {
      if (b011) set_leaf(j, (mx0 | my1 | mz1) >> 5, b011);
      if (b101) set_leaf(j, (mx1 | my0 | mz1) >> 5, b101);
      if (b110) set_leaf(j, (mx1 | my1 | mz) >> 5, b110);
      if (b111) set_leaf(j, (mx1 | my1 | mz1) >> 5, b111);
    }
    mz = ((mz1 | ~ZBITS) + z1) & ZBITS;
  }
  return mask;
}

// The grid box of an item and what the pass does with it.
struct ItemBox {
  int lo[3];
  uint32_t b[3];  // extents
  int W;          // small: the walk axis
};
enum ItemKind { ITEM_NONE = 0, ITEM_SMALL = 1, ITEM_LARGE = 2 };

__device__ __forceinline__ ItemKind classify(const VoxJob& j, const TriVerts& tv, ItemBox& box, uint32_t& lines) {
  int hi[3];
  lines = 0;
  if (!item_box(j, tv, box.lo, hi)) return ITEM_NONE;
#pragma unroll
  for (int a = 0; a < 3; a++) box.b[a] = (uint32_t)(hi[a] - box.lo[a] + 1);
  const uint32_t b0 = box.b[0], b1 = box.b[1], b2 = box.b[2];
  box.W = b2 >= b0 && b2 >= b1 ? 2 : (b0 >= b1 ? 0 : 1);
  const uint32_t narrow = box.W == 2 ? max(b0, b1) : (box.W == 0 ? max(b1, b2) : max(b0, b2));
  // extents are at most a stripe's 1024: the product fits 32 bits
  if (narrow <= 2 && b0 * b1 * b2 <= j.small_vol) return ITEM_SMALL;
  lines = (uint32_t)item_lines(walk_axis(tv), box.lo, hi);
  return ITEM_LARGE;
}

// Voxelizes small item i; payload jobs get its pass mask and box.
__device__ __forceinline__ void vox_small_item(const VoxJob& j, uint64_t i, const TriVerts& tv, const ItemBox& box) {
  const int W = box.W;
  TriVerts t = tv;
  int lo[3] = {box.lo[0], box.lo[1], box.lo[2]};
  uint32_t b[3] = {box.b[0], box.b[1], box.b[2]};
  uint32_t local[3] = {(uint32_t)(lo[0] - j.sa[0]), (uint32_t)(lo[1] - j.sa[1]), (uint32_t)(lo[2] - j.sa[2])};
  if (W != 2) {
#pragma unroll
    for (int k = 0; k < 3; k++) turn(W, t.v[k][0], t.v[k][1], t.v[k][2]);
    turn(W, lo[0], lo[1], lo[2]);
    turn(W, b[0], b[1], b[2]);
    turn(W, local[0], local[1], local[2]);
  }
  TriSetup s;
  tri_setup_rotated(t, j.u, W, s);
  const uint64_t mask = vox_small_bricks(j, s, W, lo, local, b[0], b[1], b[2]);
  if (j.item_mask) {
    j.item_mask[i] = mask;
    // Morton code of the box origin, extents along b (1 or 2) and w, walk axis
    if (mask)
      j.item_box[i] = (uint64_t)morton_local((uint32_t)(box.lo[0] - j.sa[0]), (uint32_t)(box.lo[1] - j.sa[1]),
                                             (uint32_t)(box.lo[2] - j.sa[2])) |
                      ((uint64_t)b[1] << 32) | ((uint64_t)b[2] << 34) | ((uint64_t)W << 41);
  }
}

// Pass 0 for item i of job j (any i: past the last item nothing is done), one thread per item, by
// every thread of the warp or (CTA) of the CTA.
template <bool CTA>
__device__ __forceinline__ void vox_small_occ(const VoxJob& j, uint64_t i) {
  uint32_t lines = 0;
  ItemKind kind = ITEM_NONE;
  ItemBox box;
  TriVerts tv;
  if (i < j.n_items) {
    tv = load_verts(j.tris, item_triangle(j, i), j.stride);
    kind = classify(j, tv, box, lines);
    if (kind != ITEM_SMALL && j.item_mask) j.item_mask[i] = 0;
  }
  if (kind == ITEM_SMALL) vox_small_item(j, i, tv, box);
  append_large<CTA>(j, i, lines);  // last: its barrier then waits for little
}

// Pass 1 for small items: rank the voxels their pass mask names.
__device__ __forceinline__ void vox_small_win_item(const VoxJob& j, uint64_t i) {
  uint64_t mask = j.item_mask[i];
  if (!mask) return;
  const uint32_t t = (uint32_t)item_triangle(j, i);
  const uint64_t box = j.item_box[i];
  const uint32_t m0 = (uint32_t)box & 0x3fffffffu;  // Morton code of the box origin
  const uint32_t by = (uint32_t)(box >> 32) & 3u, bz = (uint32_t)(box >> 34) & 127u;
  const uint32_t W = (uint32_t)(box >> 41) & 3u;  // the axes are turned so that it comes last (z below)
  const uint32_t xs = W == 2 ? 0u : (W == 0 ? 1u : 2u), ys = W == 2 ? 1u : (W == 0 ? 2u : 0u);
  const uint32_t XB = 0x09249249u << xs, YB = 0x09249249u << ys, ZB = 0x09249249u << W;
  const uint32_t mx1 = ((m0 | ~XB) + (1u << xs)) & XB, my1 = ((m0 | ~YB) + (1u << ys)) & YB;
  while (mask) {
    const uint32_t q = (uint32_t)(__ffsll((long long)mask) - 1);
    mask &= mask - 1;
    const uint32_t col = (q >= bz ? 1u : 0u) + (q >= 2u * bz ? 1u : 0u) + (q >= 3u * bz ? 1u : 0u);
    uint32_t z = q - col * bz;  // below 64, its bits spread
    z = (z | (z << 8)) & 0x300fu;
    z = (z | (z << 4)) & 0x30c3u;
    z = (z | (z << 2)) & 0x9249u;
    const bool x = by == 2 ? col >= 2 : col != 0, y = by == 2 && (col & 1u);
    const uint32_t m = (x ? mx1 : m0 & XB) | (y ? my1 : m0 & YB) | (((m0 | ~ZB) + (z << W)) & ZB);
    offer(j, m, t);
  }
}


// ---------------------------------------------------------------------------
// Large items, several to a warp.  Up to kWalkItems lanes each set up one item (the set-up of
// one item by all lanes cost a third of the whole pass); then the lines of all of them stand in
// one row, 32 at a time are tested against their own projection, one per lane, and the ones that
// pass go onto a stack from which 32 at a time are walked, one per lane.  So the lanes stay full
// whatever the items' sizes.
//
// Bound by issue (no FMA), the walk three fifths of it, the lines' tests a quarter.  4.0 ms on the
// 20M-triangle soup at gridsize 4096 (8.8 with one item per warp at a time), 0.77 (1.51) ms on 4M triangles
// at 1024, 0.65 + 0.60 ms for the two passes of 128 meshes.  Of the rest a start at the voxel nearest the
// run's middle, the voxel's neighbours tested as a pair, two projections per instruction, setting up the
// turned triangle and finding a line's item with one reduction gave 5.3 -> 4.2, 1.01 -> 0.81 and 0.80 ->
// 0.63.  Eight items a warp are 2 to 4% slower; 32 are 2% faster on the soups and 5 to 15% slower on the
// smaller calls; 3 and 5 CTAs per SM 8% and 5% slower.
// ---------------------------------------------------------------------------
constexpr uint32_t kWalkBits = 4, kWalkItems = 1u << kWalkBits;
struct WalkScratch {
  WalkItem item[kWalkItems];
  uint32_t stack[64];  // item | ra << kWalkBits | rb << (kWalkBits + 10)
};

// The lanes with `has` (below kWalkItems): lines [first, first + most) of item `item` of stripe
// `stripe`, or, when `parts` is not 0, part `first` of `parts` of its lines.
template <int PASS, bool SINGLE>
__device__ __forceinline__ void walk_items(const VoxJob* __restrict__ jobs, const VoxJob& j0, bool has, uint32_t item,
                                           uint32_t stripe, uint32_t first, uint32_t most, uint32_t parts, int lane,
                                           WalkScratch& sm, const uint32_t* spread) {
  const uint32_t lt = (1u << lane) - 1u, le = (2u << lane) - 1u;
  uint32_t n = 0;
  uint64_t t = 0;
  TriVerts tv;
  int lo[3], hi[3], W = 0;
  if (has) {
    const VoxJob& j = SINGLE ? j0 : jobs[stripe];
    if (item < j.n_items && (PASS == 0 || j.winners)) {  // (a binary stripe in a mixed batch has no winner pass)
      t = item_triangle(j, item);
      tv = load_verts(j.tris, t, j.stride);
      if (item_box(j, tv, lo, hi)) {  // as when it was listed
        W = walk_axis(tv);
        const uint32_t lines = (uint32_t)item_lines(W, lo, hi);  // at most 1024^2 (a stripe's face)
        if (parts) {  // whole rounds of 32 lines
          most = (lines + 32u * parts - 1u) / (32u * parts) * 32u;
          first *= most;
        }
        if (first < lines) n = min(most, lines - first);
      }
    }
  }
  const uint32_t incl = warp_inclusive(n), excl = incl - n, total = __shfl_sync(FULL, incl, 31);
  const uint32_t with = __ballot_sync(FULL, n != 0);
  if (n) walk_setup(SINGLE ? j0 : jobs[stripe], tv, t, stripe, first - excl, W, lo, hi, sm.item[__popc(with & lt)]);
  __syncwarp();
  auto walk = [&](uint32_t e) {
    const WalkItem& r = sm.item[e & (kWalkItems - 1u)];
    walk_line<PASS>(SINGLE ? j0 : jobs[r.stripe], r, (e >> kWalkBits) & 1023u, e >> (kWalkBits + 10), spread);
  };
  uint32_t cnt = 0, begun = 0;  // lines on the stack; items that began in an earlier round
#pragma unroll 1
  for (uint32_t r0 = 0; r0 < total; r0 += 32u) {
    const uint32_t i = r0 + (uint32_t)lane;
    const uint32_t starts = __reduce_or_sync(FULL, n && excl - r0 < 32u ? 1u << (excl - r0) : 0u);
    const uint32_t o = begun + __popc(starts & le) - 1u;
    begun += __popc(starts);
    bool ok = i < total;
    uint32_t e = 0;
    if (ok) {
      const WalkItem& r = sm.item[o];
      const uint32_t c = i + r.first, ea = r.shape & 2047u;
      const uint32_t rb = r.magic ? __umulhi(c, r.magic) : c, ra = c - rb * ea;
      const float fa = __fmul_rn((float)(r.alo + (int)ra), r.u), fb = __fmul_rn((float)(r.blo + (int)rb), r.u);
      float t0, t1;
      const F2 nz = minus_zero(r.shape);
      split(add2(add2(mul2(r.ea, f2(fa, fa), nz), mul2(r.eb, f2(fb, fb), nz)), r.ed), t0, t1);
      const float t2 = __fadd_rn(__fadd_rn(__fmul_rn(r.ea2, fa), __fmul_rn(r.eb2, fb)), r.ed2);
      ok = !(fminf(fminf(t0, t1), t2) < 0.0f);  // a NaN passes
      e = o | (ra << kWalkBits) | (rb << (kWalkBits + 10));
    }
    const uint32_t vote = __ballot_sync(FULL, ok);
    if (ok) sm.stack[cnt + __popc(vote & lt)] = e;
    cnt += __popc(vote);
    __syncwarp();
    if (cnt >= 32u) {
      cnt -= 32u;
      walk(sm.stack[cnt + (uint32_t)lane]);
      __syncwarp();
    }
  }
  if ((uint32_t)lane < cnt) walk(sm.stack[lane]);
  __syncwarp();  // the items and the stack are free for the warp's next ones
}

// Persistent warps: first the tasks of the big items, one at a time (the longest work first),
// then the others, as many at a time as leave every warp two helpings.
template <int PASS, bool SINGLE>
__device__ __forceinline__ void walk_lists(const VoxJob* __restrict__ jobs, const VoxJob& j0, const LargeLists& L, int lane,
                                           WalkScratch& sm, const uint32_t* spread) {
  const unsigned long long n = min(__ldcg(L.ctr + kCtrLarge), (unsigned long long)L.large_cap), packed = __ldcg(L.ctr + kCtrBig);
  const uint32_t nb = min((uint32_t)(packed & ((1u << kBigCountBits) - 1u)), L.big_cap);
  uint64_t tasks = 0;
  if (nb) {
    const uint4 end = __ldcg(L.big + nb - 1);
    tasks = (uint64_t)end.z + end.w;
  }
  // Fewer items than warps: several warps share an item (up to 16, one per round of its 512 lines), so
  // a handful of triangles takes one round and not sixteen (80 triangles at gridsize 64: 21 -> 10 us).  A
  // warp's first helping is its number.
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const uint32_t parts = n ? (uint32_t)min(16ull, max(1ull, warps / n)) : 1u;
  const uint64_t total = n * parts;
  const uint32_t chunk = (uint32_t)min((unsigned long long)kWalkItems, n / (2 * warps) + 1);
  uint64_t t = (uint64_t)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * chunk;
  bool big = tasks != 0;
#pragma unroll 1
  for (;;) {
    bool has;
    uint32_t item, stripe, first, most = ~0u, ps = 0;
    if (big) {
      unsigned long long g = 0;
      if (lane == 0) g = atomicAdd(L.ctr + kCtrGrab + 32 * PASS, 1ull);
      g = __shfl_sync(FULL, g, 0);
      if (g >= tasks) {
        big = false;
        continue;
      }
      const uint4 e = __ldcg(L.big + warp_search(nb, (uint32_t)g, lane, [&](uint32_t i) { return __ldcg(&L.big[i].z); }));
      const uint32_t k = (uint32_t)g - e.z;
      has = lane == 0 && k < e.w;
      item = e.x, stripe = e.y, first = k * L.slice, most = L.slice;
    } else {
      if (t >= total) break;
      has = (uint32_t)lane < chunk && t + (uint32_t)lane < total;
      const uint64_t i = (t + (uint32_t)lane) / parts;
      const unsigned long long e = has ? __ldcg(L.large + i) : 0ull;
      item = (uint32_t)e, stripe = (uint32_t)(e >> 32), first = (uint32_t)(t + (uint32_t)lane - i * parts);
      if (parts > 1) ps = parts;
    }
    walk_items<PASS, SINGLE>(jobs, j0, has, item, stripe, first, most, ps, lane, sm, spread);
    if (!big) {
      if (lane == 0) t = (uint64_t)warps * chunk + atomicAdd(L.ctr + kCtrGrab + 16 + 32 * PASS, (unsigned long long)chunk);
      t = __shfl_sync(FULL, t, 0);
    }
  }
}

template <int PASS, bool SINGLE>
__global__ void __launch_bounds__(256, 4) kb_vox_large(const VoxJob* __restrict__ jobs, LargeLists lists, VoxJob j0) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char walk_smem[];
  __shared__ uint32_t s_spread[1024];
  fill_spread(s_spread);
  walk_lists<PASS, SINGLE>(jobs, j0, lists, threadIdx.x & 31, reinterpret_cast<WalkScratch*>(walk_smem)[threadIdx.x >> 5],
                           s_spread);
}

// n words into `dst` (mapped pinned host memory): small results the host waits for
// travel as the kernel's stores, not as copies queued on the copy engine.
__global__ void k_copy_words(const uint32_t* __restrict__ src, uint64_t n, uint32_t* __restrict__ dst) {
  pdl_enter();
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

// Records written on the host, at `src` device or mapped host memory (see launch_scatter_records).
__global__ void k_scatter_records(const uint64_t* __restrict__ src, uint64_t n_nodes, uint64_t n_data,
                                  uint64_t* __restrict__ nodes, uint64_t* __restrict__ data) {
  pdl_enter();
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_nodes + n_data) return;
  const bool node = i < n_nodes;
  const uint64_t* s = node ? src + i * 4 : src + n_nodes * 4 + (i - n_nodes) * 5;
  uint64_t* d = nodes ? (node ? nodes + s[0] * 3 : data + s[0] * 4) : reinterpret_cast<uint64_t*>(s[0]);
  for (int q = 0; q < (node ? 3 : 4); q++) d[q] = s[1 + q];
}

// ===========================================================================
// Batched forms: every stripe of a batch in one launch.  A chunk table gives
// each CTA one stripe and a run of at most kChunk elements; the CTA copies that
// stripe's job into shared memory and runs the per-element bodies above.
// ===========================================================================
// A one-stripe launch (SINGLE) takes the stripe's job as a kernel parameter
// and indexes elements directly; a batch launch finds its stripe first and
// stages the job in shared memory.
template <bool SINGLE>
__global__ void __launch_bounds__(kChunk, 3) kb_vox_occ(const VoxJob* __restrict__ jobs,
                                                       const uint64_t* __restrict__ cta_beg, uint32_t n, VoxJob j0) {
  pdl_enter();
  if constexpr (SINGLE) {
    vox_small_occ<true>(j0, (uint64_t)blockIdx.x * kChunk + threadIdx.x);
  } else {
    __shared__ VoxJob sj;
    uint64_t cta;
    const uint32_t s = cta_stripe(cta_beg, n, cta);
    stage(sj, jobs[s]);
    __syncthreads();
    vox_small_occ<true>(sj, cta * kChunk + threadIdx.x);
  }
}

template <bool SINGLE>
__global__ void __launch_bounds__(kChunk) kb_vox_win(const VoxJob* __restrict__ jobs, const uint64_t* __restrict__ cta_beg,
                                                     uint32_t n, VoxJob j0) {
  pdl_enter();
  if constexpr (SINGLE) {
    const uint64_t i = (uint64_t)blockIdx.x * kChunk + threadIdx.x;
    if (i < j0.n_items) vox_small_win_item(j0, i);
  } else {
    __shared__ VoxJob sj;
    uint64_t cta;
    const uint32_t s = cta_stripe(cta_beg, n, cta);
    stage(sj, jobs[s]);
    __syncthreads();
    const uint64_t i = cta * kChunk + threadIdx.x;
    if (i < sj.n_items) vox_small_win_item(sj, i);
  }
}

// ===========================================================================
// Persistent occupancy passes (ooc_tuning::persistent): the small pass and the
// large items of every stripe of a sub-batch in one launch.  Each warp takes
// 256-item chunks of the small pass from one counter, stripe by stripe; when none
// is left it waits until every chunk is done and joins the walk of the large
// items.  The wait is for chunks that running warps hold already, so it ends
// whether or not the whole grid is resident; it is still bounded: past
// kPersistWaitNs it records its code in the timeout counter and every warp stops.
// ===========================================================================
// Counters, each on its own 128-byte line so the polls of waiting warps do not
// queue behind the ticket atomics.
constexpr int kCtrTicket = 0, kCtrChunksDone = 16, kCtrTimeout = kPersistTimeoutWord;
static_assert(kPersistChunkItems == 32u * 8u, "a chunk is kPersistChunkRounds x 32 items");
constexpr uint64_t kPersistWaitNs = 4000000000ull;  // a wait gives up after four seconds
constexpr uint32_t kPersistChunkRounds = 8;          // a chunk is 8 x 32 items

__device__ __forceinline__ uint64_t ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Polling with a growing pause (64 ns to 4 us) and a bound in time.
struct Backoff {
  uint64_t t0 = 0;
  uint32_t ns = 64;
  // false once the bound has passed (recording `code`) or another warp has recorded one
  __device__ __forceinline__ bool pause(unsigned long long* ctr, uint32_t code) {
    if (ld_acquire(ctr + kCtrTimeout) != 0ull) return false;
    const uint64_t now = global_ns();
    if (t0 == 0) t0 = now;
    if (now - t0 > kPersistWaitNs) {
      atomicCAS(ctr + kCtrTimeout, 0ull, (unsigned long long)code);
      return false;
    }
    __nanosleep(ns);
    if (ns < 4096) ns <<= 1;
    return true;
  }
};

__device__ __forceinline__ uint32_t find_stripe(const uint64_t* __restrict__ beg, uint32_t n, uint64_t x) {
  uint32_t lo = 0, hi = n;  // beg[lo] <= x < beg[hi]
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (beg[mid] <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

template <typename T>
__device__ __forceinline__ void stage_warp(T& dst, const T& src, int lane) {
  static_assert(sizeof(T) % 4 == 0, "staged structs are word-sized");
  const uint32_t* s = reinterpret_cast<const uint32_t*>(&src);
  uint32_t* d = reinterpret_cast<uint32_t*>(&dst);
  for (uint32_t q = (uint32_t)lane; q < sizeof(T) / 4; q += 32u) d[q] = s[q];
  __syncwarp();
}

__global__ void __launch_bounds__(256, 4) kb_persist(PersistJob pj) {
  pdl_enter();
  __shared__ VoxJob s_job[8];
  __shared__ WalkScratch s_walk[8];
  __shared__ uint32_t s_spread[1024];
  fill_spread(s_spread);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint64_t C = pj.chunk_beg[pj.n];
  uint32_t job_s = ~0u;  // the stripe staged in s_job[w]
  for (;;) {
    unsigned long long t = 0;
    if (lane == 0)
      t = ld_acquire(pj.ctr + kCtrTimeout) != 0ull ? ~0ull : atomicAdd(pj.ctr + kCtrTicket, 1ull);
    t = __shfl_sync(FULL, t, 0);
    if (t == ~0ull) return;
    if (t >= C) break;
    const uint32_t s = find_stripe(pj.chunk_beg, pj.n, t);  // a chunk of kPersistChunkRounds x 32 items
    if (s != job_s) {
      __syncwarp();
      stage_warp(s_job[w], pj.jobs[s], lane);
      job_s = s;
    }
    const uint64_t c0 = (t - pj.chunk_beg[s]) * (32u * kPersistChunkRounds);
    for (uint32_t q = 0; q < kPersistChunkRounds; q++) {
      const uint64_t i0 = c0 + 32u * q;
      if (i0 >= s_job[w].n_items) break;
      vox_small_occ<false>(s_job[w], i0 + (uint64_t)lane);
    }
    // this chunk's listed items are visible before it counts as done
    __threadfence();
    __syncwarp();
    if (lane == 0) atomicAdd(pj.ctr + kCtrChunksDone, 1ull);
  }
  bool ok = true;
  if (lane == 0) {
    Backoff b;
    while (ld_acquire(pj.ctr + kCtrChunksDone) != C && ok) ok = b.pause(pj.ctr, 1u);
  }
  if (!__shfl_sync(FULL, ok, 0)) return;
  __syncwarp();
  walk_lists<0, false>(pj.jobs, s_job[w], pj.lists, lane, s_walk[w], s_spread);
}

}  // namespace

// ===========================================================================
// Launch wrappers
// ===========================================================================
uint64_t scan_partials_needed(uint64_t n) { return (n + SCAN_TILE - 1) / SCAN_TILE + 1; }

void launch_copy_words(const uint32_t* src, uint64_t n, uint32_t* dst, cudaStream_t st) {
  if (n == 0) return;
  KScope k("copy_words", st);
  const uint64_t g = std::min<uint64_t>((n + 255) / 256, 4096);
  launch_k(k_copy_words, dim3((unsigned)g), dim3(256), 0, st, src, n, dst);
}

// Rounds of kPartCta triangles a block takes: as many as leave eight blocks per SM, and runs that fit
// beside the counters in 48 KB.
static int part_rounds(uint64_t n_tris, size_t counters, int num_sms) {
  return (int)std::min<uint64_t>(std::min<uint64_t>(kPartMax, (49152 - counters) / (kPartCta * 8)),
                                 std::max<uint64_t>(1, n_tris / ((uint64_t)num_sms * 8 * kPartCta)));
}

void launch_part_count(const float* tris, int stride, uint64_t n_tris, const float* axis_lo, const float* axis_hi,
                       int pa_bits, uint64_t n_parts, uint32_t* hist, int num_sms, cudaStream_t st) {
  if (n_tris == 0) return;
  const int use_smem = n_parts <= 4096;
  const size_t smem = ((use_smem ? n_parts : 0) + 6ull * (1ull << pa_bits)) * sizeof(uint32_t);
  const int per = part_rounds(n_tris, smem, num_sms);
  KScope k("part_count", st);
  launch_k(k_part_count, dim3(grid_for(n_tris, kPartCta * per)), dim3(kPartCta), smem, st, tris, stride, n_tris, axis_lo,
           axis_hi, pa_bits, (uint32_t)n_parts, hist, use_smem, per);
}

void launch_part_emit(const float* tris, int stride, uint64_t n_tris, const float* axis_lo, const float* axis_hi,
                      int pa_bits, uint64_t n_parts, uint32_t* cursor, uint32_t* items, int num_sms, cudaStream_t st) {
  if (n_tris == 0) return;
  const int use_smem = n_parts <= 4096;
  size_t smem = ((use_smem ? n_parts : 0) + 6ull * (1ull << pa_bits)) * sizeof(uint32_t);
  const int per = part_rounds(n_tris, smem, num_sms);
  if (use_smem) smem += (size_t)per * kPartCta * 8;
  KScope k("part_emit", st);
  launch_k(k_part_emit, dim3(grid_for(n_tris, kPartCta * per)), dim3(kPartCta), smem, st, tris, stride, n_tris, axis_lo,
           axis_hi, pa_bits, (uint32_t)n_parts, cursor, items, use_smem, per);
}

uint32_t stream_ctas(uint64_t n) { return (uint32_t)((n + kStreamCta - 1) / kStreamCta); }

void launch_stream_bases(const uint32_t* part_off, uint32_t p0, uint32_t gp, uint64_t* base, cudaStream_t st) {
  if (gp == 0) return;
  KScope k("stream_bases", st);
  launch_k(k_stream_bases, dim3(grid_for(gp, 256)), dim3(256), 0, st, part_off, p0, gp, base);
}

void launch_stream_group_chunk(const float* tris, int stride, uint64_t n, const float* axis_lo, const float* axis_hi,
                               int pa_bits, uint32_t p0, uint32_t gp, uint32_t* mat, uint32_t* mat_partials,
                               uint64_t* base, float* out, cudaStream_t st) {
  if (n == 0 || gp == 0) return;
  const uint32_t n_cta = stream_ctas(n), axes = 6u << pa_bits;
  {
    KScope k("stream_count", st);
    launch_k(k_stream_count, dim3(n_cta), dim3(kStreamCta), (gp + axes) * sizeof(uint32_t), st, tris, stride, n, axis_lo,
             axis_hi, pa_bits, p0, gp, mat, n_cta);
  }
  scan_exclusive<uint32_t>(mat, (uint64_t)gp * n_cta + 1, mat_partials, st);
  {
    KScope k("stream_emit", st);
    launch_k(k_stream_emit, dim3(n_cta), dim3(kStreamCta), axes * sizeof(float), st, tris, stride, n, axis_lo, axis_hi, pa_bits,
             p0, gp, mat, n_cta, base, out);
  }
  KScope k("stream_advance", st);
  launch_k(k_stream_advance, dim3(grid_for(gp, 256)), dim3(256), 0, st, mat, n_cta, gp, base);
}

// One-stripe occupancy pass with the job as a kernel parameter (the
// allocation-free entry point uses these).  Launched with cudaLaunchKernel so
// that each returns the status of its own launch.
cudaError_t launch_vox_small_occupancy(const VoxJob& j, cudaStream_t st) {
  if (j.n_items == 0) return cudaSuccess;
  KScope k("vox_small_occupancy", st);
  const VoxJob* jobs = nullptr;
  const uint64_t* cta_beg = nullptr;
  uint32_t n = 1;
  VoxJob arg = j;
  void* args[] = {&jobs, &cta_beg, &n, &arg};
  return cudaLaunchKernel(reinterpret_cast<const void*>(&kb_vox_occ<true>), dim3(grid_for(j.n_items, kChunk)),
                          dim3(kChunk), args, 0, st);
}

cudaError_t launch_vox_large_occupancy(const VoxJob& j, cudaStream_t st, int num_sms) {
  if (j.n_items == 0) return cudaSuccess;
  KScope k("vox_large_occupancy", st);
  const VoxJob* jobs = nullptr;
  LargeLists lists = lists_of(j);
  VoxJob arg = j;
  void* args[] = {&jobs, &lists, &arg};
  return cudaLaunchKernel(reinterpret_cast<const void*>(&kb_vox_large<0, true>), dim3((unsigned)num_sms * 4), dim3(256),
                          args, 8 * sizeof(WalkScratch), st);
}

void launch_scatter_records(const uint64_t* src, uint64_t n_nodes, uint64_t n_data, uint64_t* nodes, uint64_t* data,
                            cudaStream_t st) {
  if (n_nodes + n_data == 0) return;
  KScope k("scatter_records", st);
  launch_k(k_scatter_records, dim3(grid_for(n_nodes + n_data, 128)), dim3(128), 0, st, src, n_nodes, n_data, nodes, data);
}

// ---- batched launch wrappers ----
void launch_b_vox_small(const VoxJob* jobs, const uint64_t* cta_beg, uint32_t n, uint64_t ctas, int pass,
                        const VoxJob* single, cudaStream_t st) {
  if (ctas == 0) return;
  KScope k(pass == 0 ? "vox_small_occupancy" : "vox_small_winner", st);
  VoxJob j0;
  std::memset(&j0, 0, sizeof(j0));
  if (single) j0 = *single;
  auto* kern = pass == 0 ? (single ? kb_vox_occ<true> : kb_vox_occ<false>) : (single ? kb_vox_win<true> : kb_vox_win<false>);
  launch_k(kern, dim3((unsigned)ctas), dim3(kChunk), 0, st, jobs, cta_beg, n, j0);
}

void launch_b_vox_large(const VoxJob* jobs, const LargeLists& lists, int pass, const VoxJob* single, cudaStream_t st,
                        int num_sms, int block, int ctas_per_sm) {
  KScope k(pass == 0 ? "vox_large_occupancy" : "vox_large_winner", st);
  VoxJob j0;
  std::memset(&j0, 0, sizeof(j0));
  if (single) j0 = *single;
  auto* kern = single ? (pass == 0 ? kb_vox_large<0, true> : kb_vox_large<1, true>)
                      : (pass == 0 ? kb_vox_large<0, false> : kb_vox_large<1, false>);
  launch_k(kern, dim3((unsigned)num_sms * (unsigned)ctas_per_sm), dim3(block), (size_t)(block / 32) * sizeof(WalkScratch), st,
           jobs, lists, j0);
}

int persist_ctas_per_sm() {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kb_persist, 256, 0) != cudaSuccess) return 0;
  return per_sm;
}

void launch_b_persist(const PersistJob& pj, int num_sms, int ctas_per_sm, cudaStream_t st) {
  KScope k("persistent_occupancy", st);
  launch_k(kb_persist, dim3((unsigned)(num_sms * ctas_per_sm)), dim3(256), 0, st, pj);
}

}  // namespace ooc
