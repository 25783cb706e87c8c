// Internal interfaces between the orchestration (ooc_api.cu) and the kernels
// (ooc_kernels.cu).  Not part of the public ABI.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "ooc_svo_gpu.h"

namespace ooc {

// Maximum stripe: 8^10 = 2^30 voxels, a 1024^3 Morton-aligned cube whose
// occupancy bitfield (128 MiB) is about the size of the GB300's 129 MB L2, so
// the voxelization atomics mostly stay on chip.
constexpr int kMaxStripeDepth = 10;

// A stripe's octree is cut into bricks: the nodes kBrickLevels levels above the
// leaves (16^3 voxels, 4,096 leaf bits; a stripe of depth 4 or less is one
// brick).  A brick's records are one contiguous run of the node file, so one
// warp lays out and writes a whole brick from its leaf bits, and nothing is
// stored per node.  Only the bricks and the few nodes above them (the upper
// levels 0..U, U = depth - K) have arrays:
//   * ubits: the occupancy bits of the upper levels;
//   * upre: per upper word, the set bits of its level before it;
//   * wpre: per level-U word (32 bricks), the leaves and the nodes strictly
//     between the leaves and the bricks before it;
//   * bpre: per brick, the same within the word; bunits: its child mask.
// Every position in the files follows from these by prefix sums: the nodes
// written before a brick's run are the leaves and inner nodes of earlier bricks
// and the upper nodes whose parents end before it.
constexpr int kBrickLevels = 4;
constexpr int kMaxUpper = kMaxStripeDepth - kBrickLevels;

// First word of upper level l in ubits / upre.  Every level has at least one
// spare word after its last, so the rank at its end can be read like any other.
__host__ __device__ inline uint32_t upper_off(int l) {
  return l < 3 ? 8u * (uint32_t)l : (l == 3 ? 24u : (l == 4 ? 48u : (l == 5 ? 184u : (l == 6 ? 1216u : 9416u))));
}
__host__ __device__ inline uint32_t upper_words(int l) { return l < 2 ? 1u : 1u << (3 * l - 5); }

// Words of the leaf level (whole 256-bit blocks) and its blocks.
__host__ __device__ inline uint64_t leaf_words(int depth) { return depth < 3 ? 8ull : 1ull << (3 * depth - 5); }
__host__ __device__ inline uint64_t leaf_blocks(int depth) { return leaf_words(depth) / 8; }

// What the rank of a leaf bit takes from its block of 256, in one load.
struct __align__(16) LeafBlock {
  uint64_t woff;   // byte k = set bits in the block's words 0..k-1
  uint32_t local;  // set bits before the block within its 32 bricks
  uint32_t inner;  // the leaves' parents and nodes of 64 leaf bits before the block within its brick
};

// The leaf levels and the marks live in buffers that are all zero between
// builds: the voxelization of a stripe of 512^3 voxels and more marks every
// 256-bit leaf block it sets a bit in (`touch`, one byte per block, written with
// plain stores), the passes over its leaf level read only marked blocks, and the
// emission zeroes what it has read.
struct Stripe {
  int depth;         // levels 0..depth, level `depth` = voxels of the stripe
  int K;             // levels below a brick: min(depth, kBrickLevels)
  int U;             // the bricks' level: depth - K
  uint32_t n_bricks; // 8^U
  uint32_t* leaf;    // leaf words
  uint8_t* touch;    // byte b non-zero: leaf block b has a set bit (NULL: every block is read)
  uint32_t* ubits;
  uint32_t* upre;
  uint2* wpre;       // .x leaves, .y inner nodes below the bricks (upper_words(U) + 1 entries)
  uint2* bpre;
  uint8_t* bunits;   // per brick: its child mask (1 for a brick of fewer levels); like bpre, whole words
  LeafBlock* blocks; // per leaf block of a payload stripe (else NULL; written for marked blocks)
  int block_inner;   // whether LeafBlock::inner is wanted (-levels)
};

// Mark bytes of a stripe's leaf level, padded to 16 bytes.
__host__ __device__ inline uint64_t touch_bytes(int depth) { return (leaf_blocks(depth) + 15) / 16 * 16; }

// Stripes of 512^3 voxels and more mark their leaf blocks; smaller leaf
// levels are read and zeroed whole (their marks would cost the voxelization
// more than they save).
constexpr int kMarkDepth = 9;

// Cell z of upper level l in the upper_cache.
__host__ __device__ inline uint64_t upper_cell(int l, uint64_t z) { return ((1ull << (3 * l)) - 1) / 7 + z; }

// Elements of a stripe's arrays in a sub-batch's buffers: what the engine allocates and what the
// serving loop admits a request for.
struct StripeSizes {
  uint64_t leaf;    // words
  uint64_t touch;   // bytes
  uint64_t blocks;  // the ranks of leaf bits: payload stripes only
  uint64_t upper;   // words of ubits, and as many of upre
  uint64_t words;   // wpre: one entry past the last word, in whole groups of eight
  uint64_t bricks;  // bpre and bunits: whole words
  uint64_t cells;   // with -levels: averages of the upper levels, the bricks and the bricks' children
};
inline StripeSizes stripe_sizes(int depth, bool payload, bool levels) {
  const int K = depth < kBrickLevels ? depth : kBrickLevels, U = depth - K;
  StripeSizes z;
  z.leaf = leaf_words(depth);
  z.touch = depth >= kMarkDepth ? touch_bytes(depth) : 0;
  z.blocks = payload ? leaf_blocks(depth) : 0;
  z.upper = upper_off(U + 1);
  z.words = (upper_words(U) + 8) / 8 * 8;
  z.bricks = U < 2 ? 32 : 1ull << (3 * U);
  z.cells = levels ? upper_cell(U + (K == kBrickLevels ? 2 : 1), 0) : 0;
  return z;
}
constexpr uint64_t kCellBytes = 24;
inline uint64_t stripe_bytes(const StripeSizes& z) {
  return z.leaf * 4 + z.touch + z.blocks * sizeof(LeafBlock) + z.upper * 8 + (z.words + z.bricks) * 8 + z.bricks +
         z.cells * kCellBytes;
}
constexpr uint64_t kItemBytes = 24;  // an item's place in the list of large items, its pass mask and its box

// Words of a stripe's counts as the host reads them.
// [0] leaves, [1] inner nodes below the bricks, [2 + l] nodes of upper level l, [kRootWord] the root's child mask
constexpr uint32_t kCountWords = 16, kRootWord = 15;

// Inputs of the voxelization kernels for one stripe.
struct VoxJob {
  const float* tris;
  int stride;               // 9 (binary) or 21 (payload)
  const uint32_t* item_tri; // triangle of each item (NULL: item i is triangle ibeg + i)
  uint64_t ibeg;
  uint64_t n_items;
  int pa[3], pb[3];         // partition box in grid coordinates (inclusive)
  int sa[3], sb[3];         // stripe box in grid coordinates (inclusive)
  float u, unit_div;
  uint32_t small_vol;       // small items have at most this many candidates (<= 64)
  uint32_t* leafbits;       // level-Ds words
  uint8_t* leaftouch;       // byte per 256-bit block of leafbits, set when a bit of the block is (may be NULL)
  // pass B (payload winners)
  const uint2* wpre;        // Stripe::wpre
  const LeafBlock* blocks;  // Stripe::blocks
  unsigned long long* winners;  // per leaf: min of triangle index << 32 | its local Morton code
  // the list of large items (shared by the stripes of a sub-batch)
  unsigned long long* large; // items of one task each: item | stripe << 32
  uint64_t large_cap;       // entries of `large`: at least the items
  uint4* big;               // the others: item, stripe, first task, tasks (big_cap entries)
  unsigned long long* ctr;  // kCtr* counters
  uint32_t big_cap;         // at most kMaxBig
  uint32_t slice;           // lines of a task: 32 x lines_per_lane
  uint32_t stripe;          // this job's index
  uint64_t item0;           // number of the job's first item in its stripe (a piece of an upload)
  uint64_t* item_mask;      // per small item: which of its candidates passed (pass 0 -> pass 1); may be NULL
  uint64_t* item_box;       // per small item with a non-zero mask: its packed stripe-local box
};

// The default of ooc_tuning::small_vol.  Occupancy passes, small + large, in us at 8, 12, 16 and 32
// candidates: heightfield of 2M triangles at gridsize 1024 113, 100, 94, 95 (its boxes of 2 x 2 x 3 fit
// 12 voxels: the line walk is no match for the one-thread pass there); 4M soup at 1024 1278, 1265, 1258,
// 1260; batch of 128 meshes 984, 970, 972, 978; 20k-triangle sphere at 256 26 to 27 for all.
constexpr uint32_t kSmallVol = 16;

// Counters of the large items' list, each on its own 128-byte line; all zero when pass 0 starts.
constexpr int kCtrLarge = 0;   // items in `large`
constexpr int kCtrBig = 16;    // entries and tasks of `big`
constexpr int kCtrGrab = 32;   // taken so far: big tasks of pass 0, large items of pass 0, and the same of pass 1
constexpr uint32_t kLargeCtrWords = 96;
constexpr uint32_t kMaxBig = 1u << 16;  // entries of `big`
struct LargeLists {
  const unsigned long long* large;
  const uint4* big;
  unsigned long long* ctr;
  uint64_t large_cap;
  uint32_t big_cap, slice;
};
inline LargeLists lists_of(const VoxJob& j) { return LargeLists{j.large, j.big, j.ctr, j.large_cap, j.big_cap, j.slice}; }

struct EmitJob {
  int binary;
  int levels;
  int color_mode;
  uint64_t gridsize;
  uint64_t stripe_base;     // global Morton code of the stripe's first voxel
  int origin[3];            // stripe origin in grid coordinates
  const float* tris;
  int stride;
  float unit_div;
  float* upper_cache;       // per cell of the upper levels and the bricks' children (upper_cell): its average; with -levels
  uint32_t* root_out;       // 6 words for the host: the stripe root's average; with -levels
  const unsigned long long* winners;  // per leaf: triangle << 32 | local Morton code
  uint64_t n_leaf;          // leaves of the stripe (payload)
  uint32_t bricks_per_warp; // of the emission
  uint64_t* node_win;       // node window (3 u64 per record)
  uint64_t node_win_base;   // global node index of node_win[0]
  unsigned char* data_win;  // data window (32 bytes per record)
  uint64_t data_win_base;
  uint64_t node_win_len;    // records the node window holds
  uint64_t data_win_len;    // records the data window holds
  uint64_t n_tris;          // triangles in `tris`
  uint32_t* flag;           // set non-zero by a kernel that finds an index out of range
  uint64_t node_base;       // file index of the stripe root's first written descendant
  uint64_t data_base;       // file index of the stripe's first data record
  uint64_t data_span;       // data records of the stripe
};

// CTAs of kTreeThreads threads over the cells above a stripe's bricks.
__host__ __device__ inline uint32_t upper_node_ctas(int U) { return (uint32_t)((upper_cell(U, 0) + 255u) / 256u); }

// Threads per CTA of the batched kernels; CTA b of a launch belongs to stripe s
// when cta_beg[s] <= b < cta_beg[s+1] and handles that stripe's elements from
// its CTA b - cta_beg[s] on.
constexpr uint32_t kChunk = 256;

// The message ooc_last_error returns for `c` (for failures found outside ooc_api.cu).
void set_ctx_error(ooc_ctx* c, const std::string& msg);
// ooc_build_files' out-of-core path: whether a mesh of n_tris records streams, and the
// build that reads them from the .tridata file partition group by partition group.
bool file_wants_stream(ooc_ctx* c, const ooc_build_params* prm, uint64_t n_tris);
int build_from_file_stream(ooc_ctx* c, const ooc_build_params* prm, const char* tridata, uint64_t n_tris,
                           ooc_sink_fn sink, void* user, ooc_build_info* info);
// ooc_file_times' values for `c` (set by ooc_build_files).
void set_ctx_file_times(ooc_ctx* c, float read_ms, float write_ms);

// ---- launches (ooc_kernels.cu); all asynchronous on `st` ----

// Optional callbacks around every kernel launch (per-kernel CUDA-event timing).
struct KernelHooks {
  void* user = nullptr;
  void (*begin)(void* user, const char* kernel, cudaStream_t st) = nullptr;
  void (*end)(void* user, const char* kernel, cudaStream_t st) = nullptr;
};

// Launch accounting of one build: its kernel count and its timing callbacks.
// Every launch wrapper reports to the state installed on the calling host
// thread (none installed: nothing is counted or timed).  A context owns one
// and installs it with LaunchScope for the length of each API call, so builds
// of different contexts on different threads never share a counter or hooks,
// and a call made from inside another call's callback restores the outer
// call's state when it returns.
struct LaunchState {
  unsigned long long launches = 0;
  KernelHooks hooks;
  bool pdl = false;  // launch with programmatic stream serialization (ooc_tuning::pdl)
};
LaunchState* current_launch_state();
struct LaunchScope {
  LaunchState* prev;
  explicit LaunchScope(LaunchState* s);
  ~LaunchScope();
  LaunchScope(const LaunchScope&) = delete;
  LaunchScope& operator=(const LaunchScope&) = delete;
};

// Scan partials of a scan over n elements.
uint64_t scan_partials_needed(uint64_t n);

// n words from device memory into `dst`, mapped pinned host memory, by a kernel.
void launch_copy_words(const uint32_t* src, uint64_t n, uint32_t* dst, cudaStream_t st);
void launch_part_count(const float* tris, int stride, uint64_t n_tris, const float* axis_lo, const float* axis_hi,
                       int pa_bits, uint64_t n_parts, uint32_t* hist, int num_sms, cudaStream_t st);
void launch_part_emit(const float* tris, int stride, uint64_t n_tris, const float* axis_lo, const float* axis_hi,
                      int pa_bits, uint64_t n_parts, uint32_t* cursor, uint32_t* items, int num_sms, cudaStream_t st);

// Out-of-core binning of one chunk of the triangle stream for the partition group
// [p0, p0 + gp) (gp <= kStreamMaxGroup): the chunk's records of each group partition q
// are copied, in stream order, to out[base[q]...] (record indices), and base[q] moves
// past them.  `mat` holds gp * stream_ctas(n) + 1 entries, `mat_partials`
// scan_partials_needed of that.
constexpr uint32_t kStreamMaxGroup = 4096;
constexpr uint64_t kStreamCtaTris = 64;  // triangles per CTA of the group binning
uint32_t stream_ctas(uint64_t n);
// base[q] = part_off[p0 + q] - part_off[p0] for q < gp: where each group partition's records start.
void launch_stream_bases(const uint32_t* part_off, uint32_t p0, uint32_t gp, uint64_t* base, cudaStream_t st);
void launch_stream_group_chunk(const float* tris, int stride, uint64_t n, const float* axis_lo, const float* axis_hi,
                               int pa_bits, uint32_t p0, uint32_t gp, uint32_t* mat, uint32_t* mat_partials,
                               uint64_t* base, float* out, cudaStream_t st);

// One-stripe occupancy pass with the job as a kernel parameter (the allocation-free
// entry point's launches); each returns the status of its own launch calls.
cudaError_t launch_vox_small_occupancy(const VoxJob& j, cudaStream_t st);
cudaError_t launch_vox_large_occupancy(const VoxJob& j, cudaStream_t st, int num_sms);

// Node records (n of 3 words) and then data records (of 4) at `src`, each after one word that says where
// it goes: its number in nodes or data or, without these, its address.
void launch_scatter_records(const uint64_t* src, uint64_t n_nodes, uint64_t n_data, uint64_t* nodes, uint64_t* data,
                            cudaStream_t st);

// ---- batched launches: per-stripe jobs in device arrays; `cta_beg` (n + 1 entries) maps CTAs to stripes ----
// `single` (may be NULL): the job of a one-stripe launch, passed as a kernel parameter.
void launch_b_vox_small(const VoxJob* jobs, const uint64_t* cta_beg, uint32_t n, uint64_t ctas, int pass,
                        const VoxJob* single, cudaStream_t st);
// The listed large items of every stripe (`single`: the job of a one-stripe launch).
void launch_b_vox_large(const VoxJob* jobs, const LargeLists& lists, int pass, const VoxJob* single, cudaStream_t st,
                        int num_sms, int block, int ctas_per_sm);
// The persistent occupancy kernel's inputs (ooc_tuning::persistent).
struct PersistJob {
  const VoxJob* jobs;
  uint32_t n;                 // stripes
  const uint64_t* chunk_beg;  // n + 1: prefix of 256-item chunks per stripe
  unsigned long long* ctr;    // kPersistCtrWords counters: tickets, chunks done, timeout code (kCtr* in the kernel),
                              // each on its own 128-byte line
  LargeLists lists;
};
// CTAs of the persistent kernel one SM holds (0 on an error).
int persist_ctas_per_sm();
void launch_b_persist(const PersistJob& pj, int num_sms, int ctas_per_sm, cudaStream_t st);
constexpr uint64_t kPersistChunkItems = 256;  // items of a chunk unit
constexpr uint32_t kPersistCtrWords = 64;     // counters of the persistent kernel
constexpr uint32_t kPersistTimeoutWord = 48;  // where it records the code of a wait that ran out

// ---- the octree (ooc_tree.cu) ----
// `single` / `sp`, `se` (may be NULL): the stripe (and emit job) of a one-stripe launch, passed
// as kernel parameters.

// Leaf and inner-node counts of every brick and word, and the level-U words: CTAs of kBrickCta warps,
// brick_ctas per stripe.
constexpr uint32_t kBrickCta = 4;
inline uint32_t brick_ctas(const Stripe& s) {
  return s.touch ? (upper_words(s.U) + kBrickCta - 1) / kBrickCta : upper_words(s.U);
}
void launch_b_bricks(const Stripe* stripes, const uint64_t* cta_beg, uint32_t n, uint64_t ctas, const Stripe* single,
                     cudaStream_t st);
// One CTA per stripe: the upper levels' words and prefixes, and every stripe's counts (kCountWords each)
// into `counts` (mapped pinned host memory), then the number of large items (`large_ctr`: kCtr*) and,
// when `code` is set, *code.
void launch_b_upper(const Stripe* stripes, uint32_t n, int max_upper, uint32_t* counts,
                    const unsigned long long* large_ctr, uint64_t* large_out, const uint64_t* code, uint64_t* code_out,
                    const Stripe* single, cudaStream_t st);
// The payloads of the stripes' leaves, into the data file: CTAs of kChunk threads, `ept` leaves each.
void launch_b_leaf_payload(const Stripe* stripes, const EmitJob* emits, const uint64_t* cta_beg, uint32_t n,
                           uint64_t ctas, uint32_t ept, const Stripe* sp, const EmitJob* se, cudaStream_t st);
// Every brick's run of records and its own record, and (with `levels`) its averages; zeroes the leaf
// levels and the marks.  CTAs of kTreeWarpsPerCta warps of EmitJob::bricks_per_warp non-empty bricks each.
constexpr uint32_t kTreeWarpsPerCta = 8;
void launch_b_emit(const Stripe* stripes, const EmitJob* emits, const uint64_t* cta_beg, uint32_t n, uint64_t ctas,
                   bool levels, int num_sms, unsigned long long* large_ctr, const Stripe* sp, const EmitJob* se,
                   cudaStream_t st);
// With -levels in the batch: the averages of the levels above the bricks, one launch per level of more than
// 4,096 cells and one for the rest, which also writes these levels' records and the roots' averages.
void launch_b_upper_levels(const Stripe* stripes, const EmitJob* emits, uint32_t n, int max_upper, const Stripe* sp,
                           const EmitJob* se, cudaStream_t st);

}  // namespace ooc
