// The octree of a stripe from its leaf bits: counts per brick, prefixes over the
// bricks and the levels above them, and the records of both files (sm_103a).
//
// Compiled with -fmad=false; FP32 arithmetic additionally goes through the
// __f*_rn intrinsics so that each operation rounds once, as in the
// reference's x86-64 build.
//
// Layout.  The reference writes a node's group of children when the Morton
// cursor leaves the node's region (groupNodes, OctreeBuilder.cpp:58-79; the loop
// of refineBuffers, 112-128), so the node file is the post-order of groups: the
// record of a node stands in its parent's group, after the groups of every inner
// node whose region ends earlier.  Positions are therefore counts, and counts are
// prefix sums of the occupancy bits:
//   * before a brick's run: the leaves and inner nodes of earlier bricks, and the
//     upper nodes whose parent's region ends before the brick;
//   * inside a brick, a node two levels above the leaves (64 leaf bits, one word)
//     owns a run of its leaves followed by their parents; the runs of eight such
//     words are followed by those words' own records, and the whole brick by the
//     records of its children.
// The data file (-levels) is ordered the same way, an inner node's average
// standing after its region's records.
#include <cuda_runtime.h>

#include <cstring>

#include "ooc_device.cuh"
#include "ooc_internal.h"
#include "ooc_launch.cuh"

namespace ooc {

namespace {

__device__ __forceinline__ uint32_t nonzero_bytes64(uint64_t v) {
  return nonzero_bytes((uint32_t)v) | (nonzero_bytes((uint32_t)(v >> 32)) << 4);
}


// Set bits of upper level l before bit `pos` (0 .. 8^l).
__device__ __forceinline__ uint32_t upper_rank(const Stripe& p, int l, uint32_t pos) {
  const uint32_t i = upper_off(l) + (pos >> 5);
  return p.upre[i] + __popc(p.ubits[i] & ((1u << (pos & 31u)) - 1u));
}

__device__ __forceinline__ uint32_t upper_byte(const Stripe& p, int l, uint32_t parent) {
  return (p.ubits[upper_off(l) + (parent >> 2)] >> (8u * (parent & 3u))) & 0xffu;
}

// Leaves (.x) and inner nodes below the bricks (.y) before brick `pos` (0 .. n_bricks).
__device__ __forceinline__ uint2 brick_prefix(const Stripe& p, uint32_t pos) {
  const uint32_t w = pos >> 5;
  uint2 v = p.wpre[w];
  if (pos & 31u) {
    const uint2 b = p.bpre[pos];
    v.x += b.x;
    v.y += b.y;
  }
  return v;
}

// A check of the layout failed: the host reads the flag and fails the build.
__device__ __forceinline__ void raise_flag(const EmitJob& e, uint32_t code) {
  *reinterpret_cast<volatile uint32_t*>(e.flag) = code;
}

// ===========================================================================
// Counts per brick and per level-U word (32 bricks).
//
// Bound by the latency of the leaf blocks' loads.  A marked leaf level is read
// only where it has bits: one warp per word, the marked blocks of the word's
// bricks handed out one per lane, so the lanes stay busy on sparse bricks.  An
// unmarked level (at most 4,096 bricks) is read whole, and its few words would
// leave most SMs idle for 16 rounds of loads: the CTA's four warps share a word,
// eight bricks each (18 -> 10 us at gridsize 256).
// ===========================================================================
// Bit position of the t-th (from 0) set bit of the 8-bit mask m.
__device__ __forceinline__ uint32_t select8(uint32_t m, uint32_t t) {
  uint32_t pos = 0, c = __popc(m & 15u);
  if (t >= c) {
    t -= c;
    pos = 4;
  }
  c = __popc((m >> pos) & 3u);
  if (t >= c) {
    t -= c;
    pos += 2;
  }
  return pos + (t >= ((m >> pos) & 1u) ? 1u : 0u);
}

struct WordCount {
  uint32_t l, i;  // leaves and inner nodes below the bricks
};

// Bricks [x0, x0 + 32), lane's brick x0 + lane (those at or past x1 have none): the counts
// before each brick and its units (bit q: the 512 leaf bits of child q are not all zero; for a
// brick of fewer levels bit 0: it has a bit); returns the totals.
__device__ __forceinline__ WordCount count_bricks(const Stripe& p, uint32_t x0, uint32_t x1, int lane, WordCount& before_x,
                                                  uint32_t& units) {
  const uint32_t x = x0 + (uint32_t)lane;
  uint32_t marked = 0;  // bit k: block k of brick x is to be read
  const uint32_t per = (uint32_t)min((uint64_t)16, leaf_blocks(p.depth));
  if (x < x1) {
    if (p.touch) {
      const uint4 m = reinterpret_cast<const uint4*>(p.touch)[x];
      marked = nonzero_bytes(m.x) | (nonzero_bytes(m.y) << 4) | (nonzero_bytes(m.z) << 8) | (nonzero_bytes(m.w) << 12);
    } else {
      marked = (1u << per) - 1u;
    }
  }
  const uint32_t cnt = __popc(marked);
  const uint32_t incl = warp_inclusive(cnt), excl = incl - cnt;
  const uint32_t total = __shfl_sync(FULL, incl, 31);
  uint32_t carry_l = 0, carry_i = 0;  // leaves, inner nodes of the blocks before this round
  uint32_t my_l = 0, my_i = 0;        // before brick x
  uint32_t seen = marked;             // blocks of brick x with a bit
  for (uint32_t round = 0; round < total; round += 32u) {
    const uint32_t j = round + (uint32_t)lane;  // this lane's block, in Morton order
    uint32_t o = 0;                             // its brick: the first lane with incl > j
#pragma unroll
    for (uint32_t st = 16; st; st >>= 1) {
      const uint32_t t = __shfl_sync(FULL, incl, (int)(o + st - 1));
      if (t <= j) o += st;
    }
    uint32_t m = __shfl_sync(FULL, marked, (int)o);
    const uint32_t before = __shfl_sync(FULL, excl, (int)o);
    uint32_t l = 0, in = 0;
    uint64_t blk = 0, wo = 0;
    if (j < total) {
      uint32_t k = j - before;
      if (p.touch) {  // the k-th marked block
        const uint32_t c = __popc(m & 0xffu);
        k = k < c ? select8(m & 0xffu, k) : 8u + select8(m >> 8, k - c);
      }
      blk = (uint64_t)(x0 + o) * 16u + k;
      const uint4* q = reinterpret_cast<const uint4*>(p.leaf) + 2 * blk;
      const uint4 q0 = q[0], q1 = q[1];
      const uint32_t wd[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
      for (int i = 0; i < 8; i++) {
        wo |= (uint64_t)l << (8 * i);  // at most 224
        l += __popc(wd[i]);
        if (p.K >= 2) in += __popc(nonzero_bytes(wd[i]));
      }
      if (p.K >= 3) {
#pragma unroll
        for (int i = 0; i < 8; i += 2) in += (wd[i] | wd[i + 1]) ? 1u : 0u;
      }
    }
    const uint32_t nonempty = __ballot_sync(FULL, l != 0);
    // both counts in one scan: at most 32 x 256 leaves and 32 x 36 nodes
    const uint32_t own = l | (in << 16), inc = warp_inclusive(own), before_own = inc - own;
    const uint32_t el = carry_l + (before_own & 0xffffu);
    const uint32_t src = excl - round;  // where this lane's brick starts, when it does in this round
    const uint32_t at_src = __shfl_sync(FULL, before_own, (int)(src & 31u));
    if (excl >= round && src < 32u) {
      my_l = carry_l + (at_src & 0xffffu);
      my_i = carry_i + (at_src >> 16);
      if (!p.touch) seen = (nonempty >> src) & marked;
    }
    if (p.blocks) {
      uint32_t inner = 0;  // after those before the block's brick
      if (p.block_inner) inner = carry_i + (before_own >> 16) - __shfl_sync(FULL, my_i, (int)o);
      if (j < total)
        reinterpret_cast<uint4*>(p.blocks)[blk] = make_uint4((uint32_t)wo, (uint32_t)(wo >> 32), el, inner);
    }
    const uint32_t all = __shfl_sync(FULL, inc, 31);
    carry_l += all & 0xffffu;
    carry_i += all >> 16;
  }
  if (excl >= total) {  // no block in this brick or after it
    my_l = carry_l;
    my_i = carry_i;
    seen = 0;
  }
  // units: pairs of blocks
  units = (seen | (seen >> 1)) & 0x5555u;
  units = (units | (units >> 1)) & 0x3333u;
  units = (units | (units >> 2)) & 0x0f0fu;
  units = (units | (units >> 4)) & 0xffu;
  if (p.K < kBrickLevels) units = units ? 1u : 0u;
  const uint32_t c3 = p.K == kBrickLevels ? __popc(units) : 0u;  // they are nodes
  const uint32_t i3 = warp_inclusive(c3);
  before_x = WordCount{my_l, my_i + i3 - c3};
  return WordCount{carry_l, carry_i + __shfl_sync(FULL, i3, 31)};
}

__device__ __forceinline__ void count_cta(const Stripe& p, uint32_t cta) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t off = upper_off(p.U);
  WordCount mine;
  uint32_t units;
  if (p.touch) {  // one word per warp
    const uint32_t w = cta * kBrickCta + (uint32_t)warp;
    if (w >= upper_words(p.U)) return;
    const WordCount t = count_bricks(p, w * 32u, p.n_bricks, lane, mine, units);
    const uint32_t bits = __ballot_sync(FULL, units != 0);
    p.bpre[w * 32u + (uint32_t)lane] = make_uint2(mine.l, mine.i);
    p.bunits[w * 32u + (uint32_t)lane] = (uint8_t)units;
    if (lane == 0) {
      p.ubits[off + w] = bits;
      p.wpre[w] = make_uint2(t.l, t.i);  // the word's own counts; kb_upper makes them prefixes
    }
    return;
  }
  // one word per CTA, a quarter of its bricks per warp
  static_assert(kBrickCta == 4, "a warp takes 8 of a word's 32 bricks");
  __shared__ WordCount s_t[kBrickCta];
  __shared__ uint32_t s_bits[kBrickCta];
  const uint32_t w = cta, x0 = w * 32u + 8u * (uint32_t)warp;
  const WordCount t = count_bricks(p, x0, min(p.n_bricks, x0 + 8u), lane, mine, units);
  const uint32_t bits = __ballot_sync(FULL, units != 0);
  if (lane == 0) {
    s_t[warp] = t;
    s_bits[warp] = bits;
  }
  __syncthreads();
  uint32_t l = 0, i = 0, all = 0;
#pragma unroll
  for (int k = 0; k < (int)kBrickCta; k++) {
    if (k < warp) {
      l += s_t[k].l;
      i += s_t[k].i;
    }
    all |= s_bits[k] << (8 * k);
  }
  if (p.blocks) {  // the blocks' ranks count from the word's start
    const uint32_t b0 = x0 * 16u, n = (uint32_t)min((uint64_t)128, leaf_blocks(p.depth) - min(leaf_blocks(p.depth), (uint64_t)b0));
    if (l)
      for (uint32_t k = (uint32_t)lane; k < n; k += 32u) p.blocks[b0 + k].local += l;
  }
  if (lane < 8) {
    p.bpre[x0 + (uint32_t)lane] = make_uint2(l + mine.l, i + mine.i);
    p.bunits[x0 + (uint32_t)lane] = (uint8_t)units;
  }
  if (warp == kBrickCta - 1 && lane == 0) {
    p.ubits[off + w] = all;
    p.wpre[w] = make_uint2(l + t.l, i + t.i);
  }
}

template <bool SINGLE>
__global__ void __launch_bounds__(32 * kBrickCta) kb_bricks(const Stripe* __restrict__ stripes,
                                                            const uint64_t* __restrict__ cta_beg, uint32_t n, Stripe p0) {
  pdl_enter();
  if constexpr (SINGLE) {
    count_cta(p0, blockIdx.x);
  } else {
    __shared__ Stripe sp;
    uint64_t cta;
    const uint32_t s = cta_stripe(cta_beg, n, cta);
    stage(sp, stripes[s]);
    __syncthreads();
    count_cta(sp, (uint32_t)cta);
  }
}

// Parent word of eight words of a level: bit i is set when byte i is non-zero.
__device__ __forceinline__ uint32_t parent_word(const uint32_t w[8]) {
  uint32_t p = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) p |= nonzero_bytes(w[k]) << (4 * k);
  return p;
}

// One CTA per stripe: the prefixes of level U, then the levels above it.  A warp takes
// 32 K consecutive words of level U, a lane words 32 apart, so loads and stores are whole
// lines (a thread on eight words in a row stored 4 bytes to a sector at a time: 20 us for
// 8,192 words, now 9).  Latency-bound; the levels above have at most 1,024 words and sit in
// shared memory, eight words to a thread, and those of 256 and fewer are left to the first
// warp, which needs no block barrier.
template <int T, int K>
__global__ void __launch_bounds__(T) kb_upper(const Stripe* __restrict__ stripes, uint32_t* __restrict__ counts,
                                              const unsigned long long* __restrict__ large_ctr,
                                              uint64_t* __restrict__ large_out, const uint64_t* __restrict__ code,
                                              uint64_t* __restrict__ code_out, const __grid_constant__ Stripe p0) {
  pdl_enter();
  __shared__ Stripe sp;
  __shared__ uint32_t s_words[2][1024];
  if (stripes) stage(sp, stripes[blockIdx.x]);
  else stage(sp, p0);
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *large_out = large_ctr[kCtrLarge] + large_ctr[kCtrBig];  // zero: none
    if (code) *code_out = *code;
  }
  uint32_t* out = counts + (uint64_t)blockIdx.x * kCountWords;
  const int U = sp.U, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t W = upper_words(U), off = upper_off(U);
  uint32_t carry_r = 0, carry_l = 0, carry_i = 0;
  for (uint32_t base = 0; base < W; base += T * K) {
    const uint32_t i0 = base + (uint32_t)warp * (32u * K) + (uint32_t)lane;
    uint32_t w[K], r[K];
    uint2 li[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t i = i0 + 32u * k;
      w[k] = i < W ? sp.ubits[off + i] : 0u;
      li[k] = i < W ? sp.wpre[i] : make_uint2(0u, 0u);
      r[k] = __popc(w[k]);
    }
    // exclusive within the warp's words: the 3 K scans side by side
#pragma unroll 1
    for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
      for (int k = 0; k < K; k++) {
        const uint32_t ur = __shfl_up_sync(FULL, r[k], d), ul = __shfl_up_sync(FULL, li[k].x, d),
                       ui = __shfl_up_sync(FULL, li[k].y, d);
        if (lane >= d) r[k] += ur, li[k].x += ul, li[k].y += ui;
      }
    }
    uint32_t sum_r = 0, sum_l = 0, sum_i = 0;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t tr = __shfl_sync(FULL, r[k], 31), tl = __shfl_sync(FULL, li[k].x, 31),
                     ti = __shfl_sync(FULL, li[k].y, 31);
      const uint32_t er = __shfl_up_sync(FULL, r[k], 1), el = __shfl_up_sync(FULL, li[k].x, 1),
                     ei = __shfl_up_sync(FULL, li[k].y, 1);
      r[k] = sum_r + (lane ? er : 0u);
      li[k] = make_uint2(sum_l + (lane ? el : 0u), sum_i + (lane ? ei : 0u));
      sum_r += tr;
      sum_l += tl;
      sum_i += ti;
    }
    // across the warps
    __shared__ uint32_t s_sum[3][33];
    if (lane == 0) s_sum[0][warp] = sum_r, s_sum[1][warp] = sum_l, s_sum[2][warp] = sum_i;
    __syncthreads();
    if (warp < 3) {
      const uint32_t v = lane < T / 32 ? s_sum[warp][lane] : 0u, inc = warp_inclusive(v);
      s_sum[warp][lane] = inc - v;
      if (lane == 31) s_sum[warp][32] = inc;
    }
    __syncthreads();
    const uint32_t br = carry_r + s_sum[0][warp], bl = carry_l + s_sum[1][warp], bi = carry_i + s_sum[2][warp];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t i = i0 + 32u * k;
      if (i < W) {
        sp.upre[off + i] = br + r[k];
        sp.wpre[i] = make_uint2(bl + li[k].x, bi + li[k].y);
      }
      if (U == 1 && i == 0) out[kRootWord] = w[k] & 0xffu;
      if (U > 0) {  // eight words' parent word: four bits each
        uint32_t pw = nonzero_bytes(w[k]) << (4 * (lane & 7));
        pw |= __shfl_xor_sync(FULL, pw, 1);
        pw |= __shfl_xor_sync(FULL, pw, 2);
        pw |= __shfl_xor_sync(FULL, pw, 4);
        if ((lane & 7) == 0 && i < W) {
          sp.ubits[upper_off(U - 1) + i / 8u] = pw;
          s_words[(U - 1) & 1][i / 8u] = pw;
        }
      }
    }
    carry_r += s_sum[0][32];
    carry_l += s_sum[1][32];
    carry_i += s_sum[2][32];
    __syncthreads();
  }
  if (threadIdx.x == 0) {  // the entries past the end
    sp.ubits[off + W] = 0u;
    sp.upre[off + W] = carry_r;
    sp.wpre[W] = make_uint2(carry_l, carry_i);
    out[0] = carry_l;
    out[1] = carry_i;
    out[2 + U] = carry_r;
    if (U == 0) {  // the root's children, straight from the brick
      uint32_t mask = 0;
      if (sp.K == kBrickLevels) mask = sp.bunits[0];
      else if (sp.K == 1) mask = sp.leaf[0] & 0xffu;
      else if (sp.K == 2) mask = nonzero_bytes(sp.leaf[0]) | (nonzero_bytes(sp.leaf[1]) << 4);
      else if (sp.K == 3)
        for (int k = 0; k < 8; k++) mask |= (sp.leaf[2 * k] | sp.leaf[2 * k + 1]) ? 1u << k : 0u;
      out[kRootWord] = mask;
    }
  }
  __syncthreads();
  for (int l = U - 1; l >= 0; l--) {
    W = upper_words(l);
    off = upper_off(l);
    const bool one_warp = W <= 256u;
    if (one_warp && threadIdx.x >= 32) return;  // every later level is smaller
    const uint32_t i0 = threadIdx.x * 8u;
    uint32_t w[8], r = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      w[k] = i0 + k < W ? s_words[l & 1][i0 + k] : 0u;
      r += __popc(w[k]);
    }
    uint32_t run, tot;
    if (one_warp) {
      const uint32_t inc = warp_inclusive(r);
      run = inc - r;
      tot = __shfl_sync(FULL, inc, 31);
    } else {
      run = block_exclusive<uint32_t>(r, tot);
    }
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (i0 + k < W) {
        sp.upre[off + i0 + k] = run;
        run += __popc(w[k]);
      }
    if (l == 1 && threadIdx.x == 0) out[kRootWord] = w[0] & 0xffu;
    if (l > 0 && i0 < W) {
      const uint32_t pw = parent_word(w);
      sp.ubits[upper_off(l - 1) + i0 / 8u] = pw;
      s_words[(l - 1) & 1][i0 / 8u] = pw;
    }
    if (threadIdx.x == 0) {
      sp.ubits[off + W] = 0u;
      sp.upre[off + W] = tot;
      out[2 + l] = tot;
    }
    if (one_warp) __syncwarp();
    else __syncthreads();
  }
}

// ===========================================================================
// Leaf payload (voxelizer.cpp:295-299, BarycentricCoords.h, main.cpp:373-382)
// ===========================================================================
__device__ void payload_color(const TriVerts& tv, const float n[3], int x, int y, int z, float unit_div,
                              const float* __restrict__ tr, float col[3]) {
  const float qx = __fdiv_rn((float)x, unit_div);
  const float qy = __fdiv_rn((float)y, unit_div);
  const float qz = __fdiv_rn((float)z, unit_div);
  const float coeffD = -dot3(tv.v[0][0], tv.v[0][1], tv.v[0][2], n[0], n[1], n[2]);
  const float nn = __fadd_rn(__fadd_rn(__fmul_rn(n[0], n[0]), __fmul_rn(n[1], n[1])), __fmul_rn(n[2], n[2]));
  const float k = __fdiv_rn(__fadd_rn(dot3(qx, qy, qz, n[0], n[1], n[2]), coeffD), nn);
  const float ptx = __fsub_rn(qx, __fmul_rn(k, n[0]));
  const float pty = __fsub_rn(qy, __fmul_rn(k, n[1]));
  const float ptz = __fsub_rn(qz, __fmul_rn(k, n[2]));
  // inverse(mat3(v0, v1, v2)) by adjugate over determinant
  const float a = tv.v[0][0], b = tv.v[1][0], c = tv.v[2][0];
  const float d = tv.v[0][1], e = tv.v[1][1], f = tv.v[2][1];
  const float g = tv.v[0][2], h = tv.v[1][2], i = tv.v[2][2];
  const float C00 = __fsub_rn(__fmul_rn(e, i), __fmul_rn(f, h));
  const float C01 = __fsub_rn(__fmul_rn(f, g), __fmul_rn(d, i));
  const float C02 = __fsub_rn(__fmul_rn(d, h), __fmul_rn(e, g));
  const float det = __fadd_rn(__fadd_rn(__fmul_rn(a, C00), __fmul_rn(b, C01)), __fmul_rn(c, C02));
  const float r = __fdiv_rn(1.0f, det);
  const float C10 = __fsub_rn(__fmul_rn(c, h), __fmul_rn(b, i));
  const float C11 = __fsub_rn(__fmul_rn(a, i), __fmul_rn(c, g));
  const float C12 = __fsub_rn(__fmul_rn(b, g), __fmul_rn(a, h));
  const float C20 = __fsub_rn(__fmul_rn(b, f), __fmul_rn(c, e));
  const float C21 = __fsub_rn(__fmul_rn(c, d), __fmul_rn(a, f));
  const float C22 = __fsub_rn(__fmul_rn(a, e), __fmul_rn(b, d));
  const float i00 = __fmul_rn(C00, r), i10 = __fmul_rn(C01, r), i20 = __fmul_rn(C02, r);
  const float i01 = __fmul_rn(C10, r), i11 = __fmul_rn(C11, r), i21 = __fmul_rn(C12, r);
  const float i02 = __fmul_rn(C20, r), i12 = __fmul_rn(C21, r), i22 = __fmul_rn(C22, r);
  const float bx = __fadd_rn(__fadd_rn(__fmul_rn(i00, ptx), __fmul_rn(i01, pty)), __fmul_rn(i02, ptz));
  const float by = __fadd_rn(__fadd_rn(__fmul_rn(i10, ptx), __fmul_rn(i11, pty)), __fmul_rn(i12, ptz));
  const float bz = __fadd_rn(__fadd_rn(__fmul_rn(i20, ptx), __fmul_rn(i21, pty)), __fmul_rn(i22, ptz));
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const float c0 = __ldg(tr + 12 + q), c1 = __ldg(tr + 15 + q), c2 = __ldg(tr + 18 + q);
    col[q] = __fadd_rn(__fadd_rn(__fmul_rn(bx, c0), __fmul_rn(by, c1)), __fmul_rn(bz, c2));
  }
}

// Colour and normal of the leaf whose winner (triangle << 32 | local Morton code) is `win`.
// Returns false (and flags) if the leaf has no winning triangle.
__device__ bool leaf_value(const EmitJob& e, unsigned long long win, float out[6]) {
  const uint32_t key = (uint32_t)win;
  uint32_t lx, ly, lz;
  morton_local_decode(key, lx, ly, lz);
  const int x = e.origin[0] + (int)lx, y = e.origin[1] + (int)ly, z = e.origin[2] + (int)lz;
  const uint64_t t = win >> 32;
  if (t >= e.n_tris) {  // every set voxel has a passing triangle; anything else is a bug
    raise_flag(e, 4u);
    return false;
  }
  const float* tr = e.tris + t * 21;
  const float nx = __ldg(tr + 9), ny = __ldg(tr + 10), nz = __ldg(tr + 11);
  if (e.color_mode == 1) {  // COLOR_FIXED
    out[0] = out[1] = out[2] = 1.0f;
  } else if (e.color_mode == 2) {  // COLOR_LINEAR: mortonToRGB (svo_builder_util.h:14-18)
    const float fn = (float)e.gridsize;
    out[0] = __fdiv_rn((float)z, fn);
    out[1] = __fdiv_rn((float)y, fn);
    out[2] = __fdiv_rn((float)x, fn);
  } else if (e.color_mode == 3) {  // COLOR_NORMAL
    float a = nx, b = ny, c = nz;
    normalize3(a, b, c);
    out[0] = __fdiv_rn(__fadd_rn(a, 1.0f), 2.0f);
    out[1] = __fdiv_rn(__fadd_rn(b, 1.0f), 2.0f);
    out[2] = __fdiv_rn(__fadd_rn(c, 1.0f), 2.0f);
  } else {  // COLOR_FROM_MODEL
    const TriVerts tv = load_verts(e.tris, t, 21);
    float n[3];
    tri_normal(tv, n);
    payload_color(tv, n, x, y, z, e.unit_div, tr, out);
  }
  out[3] = nx;
  out[4] = ny;
  out[5] = nz;
  return true;
}

__device__ __forceinline__ void store_data_record(const EmitJob& e, uint64_t idx, uint64_t morton, const float* v) {
  if (idx < e.data_win_base || idx - e.data_win_base >= e.data_win_len) {
    raise_flag(e, 2u);
    return;
  }
  uint4* dst = reinterpret_cast<uint4*>(e.data_win + (idx - e.data_win_base) * 32);
  dst[0] = make_uint4((uint32_t)morton, (uint32_t)(morton >> 32), __float_as_uint(v[0]), __float_as_uint(v[1]));
  dst[1] = make_uint4(__float_as_uint(v[2]), __float_as_uint(v[3]), __float_as_uint(v[4]), __float_as_uint(v[5]));
}

__device__ __forceinline__ void store_node_record(const EmitJob& e, uint64_t pos, uint64_t r0, uint64_t r1,
                                                  uint64_t r2) {
  if (pos < e.node_win_base || pos - e.node_win_base >= e.node_win_len) {
    raise_flag(e, 1u);
    return;
  }
  uint64_t* rec = e.node_win + (pos - e.node_win_base) * 3;
  rec[0] = r0;
  rec[1] = r1;
  rec[2] = r2;
}

__device__ __forceinline__ uint64_t child_offsets(uint32_t mask) {
  uint64_t off = 0;
  uint32_t r = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const uint64_t byte = ((mask >> k) & 1u) ? (uint64_t)(r++) : 0xffull;
    off |= byte << (8 * k);
  }
  return off;
}

constexpr uint32_t kTreeThreads = 256;
constexpr uint32_t kTreeWarps = kTreeThreads / 32;
static_assert(kTreeWarps == kTreeWarpsPerCta, "the host sizes the launches");

// ===========================================================================
// Leaf payloads, one thread per leaf: the winner pass left every leaf's triangle
// and Morton code.  The leaf goes straight into the data file: without -levels
// leaf i of the stripe is its data record i; with -levels the averages of the inner
// nodes whose regions end before the leaf stand before it too.
//
// Bound by the gathers of the winners' 84-byte triangle records.
// ===========================================================================
// Inner nodes of the stripe whose regions end before leaf bit `key`.
__device__ __forceinline__ uint32_t inner_before(const Stripe& p, uint32_t key) {
  const uint32_t x = p.K == kBrickLevels ? key >> 12 : 0u, blk = key >> 8;
  uint32_t s = p.wpre[x >> 5].y + p.bpre[x].y + p.blocks[blk].inner;
  if (p.K == kBrickLevels) s += __popc(p.bunits[x] & ((1u << ((key >> 9) & 7u)) - 1u));  // nodes of 512 leaf bits
  for (int l = 1; l <= p.U; l++) s += upper_rank(p, l, x >> (3 * (p.U - l)));
  const uint4* q = reinterpret_cast<const uint4*>(p.leaf) + 2 * (uint64_t)blk;
  const uint4 q0 = q[0], q1 = q[1];
  const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
  const uint32_t wi = (key >> 5) & 7u;
#pragma unroll
  for (uint32_t k = 0; k < 8; k++) {  // the block's words before the leaf's, and the bytes before the leaf's
    const uint32_t v = k < wi ? w[k] : (k == wi ? w[k] & ((1u << (key & 24u)) - 1u) : 0u);
    if (p.K >= 2) s += __popc(nonzero_bytes(v));
    if (p.K >= 3 && (k & 1u) && k < (wi & ~1u)) s += (w[k - 1] | w[k]) ? 1u : 0u;  // nodes of 64 leaf bits
  }
  return s;
}

// Leaves (cta * ept + k) * kTreeThreads + thread of the stripe; the next leaf's winner is loaded ahead.
__device__ __forceinline__ void leaf_payload(const Stripe& p, const EmitJob& e, uint64_t cta, uint32_t ept) {
  uint64_t i = cta * ept * kTreeThreads + threadIdx.x;
  unsigned long long next = i < e.n_leaf ? e.winners[i] : 0ull;
#pragma unroll 1
  for (uint32_t k = 0; k < ept && i < e.n_leaf; k++, i += kTreeThreads) {
    const unsigned long long win = next;
    if (k + 1 < ept && i + kTreeThreads < e.n_leaf) next = e.winners[i + kTreeThreads];
    float v[6];
    const uint32_t key = (uint32_t)win;
    if (leaf_value(e, win, v)) store_data_record(e, e.data_base + i + (e.levels ? inner_before(p, key) : 0u), e.stripe_base + key, v);
  }
}

template <bool SINGLE>
__global__ void __launch_bounds__(kTreeThreads) kb_leaf_payload(const Stripe* __restrict__ stripes,
                                                                const EmitJob* __restrict__ emits,
                                                                const uint64_t* __restrict__ cta_beg, uint32_t n,
                                                                uint32_t ept, Stripe p0, EmitJob e0) {
  pdl_enter();
  if constexpr (SINGLE) {
    leaf_payload(p0, e0, blockIdx.x, ept);
  } else {
    __shared__ Stripe sp;
    __shared__ EmitJob se;
    uint64_t cta;
    const uint32_t s = cta_stripe(cta_beg, n, cta);
    stage(sp, stripes[s]);
    stage(se, emits[s]);
    __syncthreads();
    leaf_payload(sp, se, cta, ept);
  }
}

// ===========================================================================
// Emission: the records of every brick's run and the brick's own.
//
// A warp takes consecutive non-empty bricks of the stripe, 32 at a time, and lays them out in
// steps of eight units (a unit: 512 leaf bits, a child of a brick), four lanes to
// a unit, whichever bricks the units belong to, so a step is full on sparse bricks
// too.  A lane holds 128 leaf bits: two nodes of 64 (a run of their leaves and
// those leaves' parents, and their own records in the unit's group).  One warp
// scan gives every position of a step.  The parents of leaves, whose number per
// lane varies most, are shared out over all lanes.  The records of a step are one
// run per brick: they are written to shared memory and leave as bulk copies, one
// per brick, so every sector of the node file is written whole and the copy costs
// the warp a few instructions (records stored by the lanes themselves took 2.2 times
// as long on the 20M-triangle soup at gridsize 4096).
//
// Bound by issue and latency on sparse bricks, by DRAM writes on dense ones.  The 20M-triangle soup at
// gridsize 4096 (651M records, 15.6 GB) takes 4.8 ms, 3.2 TB/s; 4M triangles at 1024 (2.9 GB) 0.49 ms, 5.9
// TB/s; the 1024^3 heightfield 33 us.  Taking the bricks word by word instead of 32 non-empty ones at a
// time, loading a step's leaf words in the step, filling the window with a pattern worked out per word and
// windows of 128 records on four CTAs per SM took 6.8, 0.73 and 0.043 ms; passes over arrays of every node
// (keys, subtree sizes bottom-up, positions top-down, leaf records) 19 ms for the first.
// ===========================================================================
// A window holds kWindow records and a gap of up to two slots between the records of eight bricks.
// Three CTAs per SM with windows of 288, and four with 160 (all that shared memory holds): 489 and 541 us
// on the 4M soup, 248 and 244 on 300k triangles with payload, 31 and 37 on the heightfield.
constexpr int kEmitCtas = 3;
constexpr uint32_t kWindow = 288;
constexpr uint32_t kSlots = kWindow + 16;

// A lane's words as the warp's lanes read them when they share out the step's parents of leaves.
struct __align__(16) LaneWords {
  uint64_t a, b;
  uint32_t m16_gap;  // non-zero bytes of a and b | slots before its brick's records << 16
  uint32_t c_pk;     // the lane's first record in the step | parents of leaves before it << 16
  uint32_t base;     // a record's number in the step + this = its position in the stripe
  uint32_t da;       // -levels: data records of the stripe before a's leaves
};
struct __align__(16) WarpScratch {
  uint64_t win[kSlots * 3];
  LaneWords words[32];
  uint32_t gaps[8];
  uint16_t units[256];  // of the 32 bricks in hand: brick | place in it << 5 | number in it << 8
};

// Bulk copies of shared memory to global memory (both 16-byte aligned, a multiple of 16
// bytes); a thread's copies since its last commit form a group.
__device__ __forceinline__ void bulk_store(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
               "r"((uint32_t)__cvta_generic_to_shared(src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// Shared memory written by this thread becomes visible to its warp's bulk copies.
__device__ __forceinline__ void bulk_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Running sum of a node's children (OctreeBuilder.cpp:81-99).  Adding a null slot's zero
// never changes a sum (no sum is -0), so null slots are skipped.
struct Sum {
  float v[6];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int q = 0; q < 6; q++) v[q] = 0.0f;
  }
  __device__ __forceinline__ void add(const float* c) {
#pragma unroll
    for (int q = 0; q < 6; q++) v[q] = __fadd_rn(v[q], c[q]);
  }
  // the colour and normal of a data record
  __device__ __forceinline__ void add(const uint4& r0, const uint4& r1) {
    const float c[6] = {__uint_as_float(r0.z), __uint_as_float(r0.w), __uint_as_float(r1.x),
                        __uint_as_float(r1.y), __uint_as_float(r1.z), __uint_as_float(r1.w)};
    add(c);
  }
  // divided by the children's number, the normal normalised
  __device__ __forceinline__ void average(uint32_t children) {
    const float n = (float)children;
#pragma unroll
    for (int q = 0; q < 6; q++) v[q] = __fdiv_rn(v[q], n);
    normalize3(v[3], v[4], v[5]);
  }
};

// -levels: the average of n <= 8 children from their data records, child k's at(k); four
// children's loads at a time.
template <typename F>
__device__ __forceinline__ void average_records(const EmitJob& e, uint32_t n, Sum& s, F at) {
  s.zero();
  for (uint32_t k0 = 0; k0 < n; k0 += 4) {
    uint4 r[4][2];
#pragma unroll
    for (uint32_t k = 0; k < 4; k++)
      if (k0 + k < n) {
        const uint64_t i = at(k0 + k) - e.data_win_base;
        if (i < e.data_win_len) {
          const uint4* src = reinterpret_cast<const uint4*>(e.data_win + i * 32);
          r[k][0] = src[0];
          r[k][1] = src[1];
        }
      }
#pragma unroll
    for (uint32_t k = 0; k < 4; k++)
      if (k0 + k < n) s.add(r[k][0], r[k][1]);
  }
  s.average(n);
}

// What the layout of up to 32 bricks, consecutive among the non-empty ones, needs from memory, lane =
// brick.  Loaded before the bricks ahead of them are laid out: the marks come from DRAM, and the
// first use of them would otherwise wait for several loads in a row.
struct BrickIn {
  uint32_t x;        // the brick (lanes below the number of bricks)
  uint32_t bits;     // the non-empty bricks from its parent's first child on
  uint2 pre;         // leaves and inner nodes before it
  uint2 end;         // the same of the first brick past the last lane's (lane 0) and past its parent's (lane 1)
  uint32_t units;
  uint4 marks;
  uint32_t up, upd;  // upper nodes recorded before the brick's parent's children; averaged before the brick (-levels)
};

template <bool LEVELS>
__device__ __forceinline__ BrickIn load_bricks(const Stripe& p, uint32_t x, uint32_t n, int lane) {
  BrickIn in;
  const int U = p.U;
  const uint32_t off = upper_off(U) + (x >> 5), last = __shfl_sync(FULL, x, (int)n - 1);
  const bool have = (uint32_t)lane < n;
  in.x = x;
  in.units = have ? p.bunits[x] : 0u;
  in.marks = make_uint4(~0u, ~0u, ~0u, ~0u);
  if (have && p.touch) in.marks = reinterpret_cast<const uint4*>(p.touch)[x];
  const uint32_t bits = p.ubits[off];
  const uint2 wp = p.wpre[x >> 5], bp = p.bpre[x];
  in.end = brick_prefix(p, lane == 0 ? last + 1u : (last | 7u) + 1u);
  in.bits = bits >> (x & 24u);
  in.pre = make_uint2(wp.x + bp.x, wp.y + bp.y);
  in.up = in.upd = 0;
  if (U) {
    const uint32_t pre = p.upre[off];
#pragma unroll
    for (int l = 1; l < kMaxUpper; l++)
      if (l < U) {
        const uint32_t anc = x >> (3 * (U - l));
        const uint32_t i = upper_off(l) + (anc >> 5), ub = p.ubits[i], ur = p.upre[i];
        in.up += ur + __popc(ub & ((1u << (anc & 24u)) - 1u));  // before its parent's children: whole bytes
        if (LEVELS) in.upd += ur + __popc(ub & ((1u << (anc & 31u)) - 1u));
      }
    in.up += pre + __popc(bits & ((1u << (x & 24u)) - 1u));
    if (LEVELS) in.upd += pre + __popc(bits & ((1u << (x & 31u)) - 1u));
  }
  return in;
}

// n bricks (1 to 32).
template <bool LEVELS>
__device__ __forceinline__ void emit_bricks(const Stripe& p, const EmitJob& e, uint32_t n, const BrickIn& in, int lane,
                                            WarpScratch& sm, const uint64_t* __restrict__ lut) {
  const uint32_t le = (2u << lane) - 1u, lt = le >> 1;
  const int K = p.K, U = p.U;
  const bool pay = !e.binary;
  uint64_t* const nodes = e.node_win - (int64_t)(e.node_win_base - e.node_base) * 3;  // the stripe's records
  const uint64_t dbase = e.data_base;
  // ---- lane = brick x ----
  const uint32_t x = in.x;
  bool mine = (uint32_t)lane < n;
  const uint32_t lpre = in.pre.x, ipre = in.pre.y;
  uint32_t units = mine && K ? in.units : 0u;
  // leaf blocks that may have a bit
  const uint32_t blocks = nonzero_bytes(in.marks.x) | (nonzero_bytes(in.marks.y) << 4) | (nonzero_bytes(in.marks.z) << 8) |
                          (nonzero_bytes(in.marks.w) << 12);
  const uint32_t up = in.up, upd = in.upd;
  const uint32_t sib = __popc(in.bits & ((1u << (x & 7u)) - 1u));
  const uint32_t start = up + lpre + ipre;  // stripe-relative, like all positions here
  // before the next brick: the next lane's, or past the last's
  uint32_t nl = __shfl_down_sync(FULL, lpre, 1), ni = __shfl_down_sync(FULL, ipre, 1);
  const uint32_t pend = (uint32_t)lane - sib + (uint32_t)__popc(in.bits & 0xffu);  // the lane past its parent's children
  uint32_t pl = __shfl_sync(FULL, lpre, (int)(pend & 31u)), pi = __shfl_sync(FULL, ipre, (int)(pend & 31u));
  {
    const uint32_t l0 = __shfl_sync(FULL, in.end.x, 0), i0 = __shfl_sync(FULL, in.end.y, 0);
    const uint32_t l1 = __shfl_sync(FULL, in.end.x, 1), i1 = __shfl_sync(FULL, in.end.y, 1);
    if ((uint32_t)lane + 1u >= n) nl = l0, ni = i0;
    if (pend >= n) pl = l1, pi = i1;
  }
  const uint32_t n3 = K == kBrickLevels ? __popc(units) : 0u;
  const uint32_t g3 = start + (nl - lpre) + (ni - ipre) - n3;  // where its children's group starts
  const uint32_t dpre = LEVELS ? (pay ? lpre : 0u) + ipre + upd : 0u;               // data records before its own
  const uint32_t dtop = LEVELS ? dpre + (pay ? nl - lpre : 0u) + (ni - ipre) : 0u;  // and before its average
  const uint32_t own_at = up + pl + pi + sib;                                       // its own record
  // every record of the brick lies in the window (the run from start to g3 + n3, then its own)
  if (mine && K &&
      (e.node_base + start < e.node_win_base ||
       e.node_base + max(g3 + n3, U ? own_at + 1u : 0u) - e.node_win_base > e.node_win_len)) {
    raise_flag(e, 1u);
    mine = false;
    units = 0;
  }
  if (U && mine) {  // its own record, in its parent's group
    uint64_t* t = nodes + (uint64_t)own_at * 3u;
    t[0] = LEVELS ? dbase + dtop : 0;
    t[1] = e.node_base + g3;
    t[2] = lut[units];
  }
  const uint32_t cnt = __popc(units);
  const uint32_t incl = warp_inclusive(cnt), excl = incl - cnt;
  const uint32_t total = __shfl_sync(FULL, incl, 31);
  for (uint32_t m = units, k = 0; m; m &= m - 1, k++)
    sm.units[excl + k] = (uint16_t)((uint32_t)lane | (((uint32_t)__ffs(m) - 1u) << 5) | (k << 8));
  __syncwarp();
  uint32_t carry = 0;          // records | leaves << 16 of the last step's last brick so far
  const uint32_t odd0 = (uint32_t)(reinterpret_cast<uintptr_t>(nodes) >> 3);
  // A step's words, loaded while the step before is laid out: the lane's unit's entry of
  // sm.units and its leaf words.
  uint32_t un_next = 0, x_next = 0;
  uint4 v_next = make_uint4(0u, 0u, 0u, 0u);
  auto unit_word = [&](uint32_t xo, uint32_t un) {
    return xo * 128u + ((un >> 5) & 7u) * 16u + (uint32_t)(lane & 3) * 4u;  // below 2^25
  };
  auto fetch = [&](uint32_t g) {
    const uint32_t u = g + (uint32_t)(lane >> 2);
    un_next = sm.units[min(u, total - 1u)];
    const uint32_t o_blocks = __shfl_sync(FULL, blocks, (int)(un_next & 31u));
    x_next = __shfl_sync(FULL, x, (int)(un_next & 31u));
    const uint32_t word = unit_word(x_next, un_next);
    v_next = make_uint4(0u, 0u, 0u, 0u);
    if (u < total && ((o_blocks >> (((un_next >> 4) & 14u) + (uint32_t)((lane >> 1) & 1))) & 1u) &&
        (K == kBrickLevels || word < leaf_words(p.depth)))
      v_next = *reinterpret_cast<const uint4*>(p.leaf + word);
  };
  if (total) fetch(0);
  for (uint32_t g = 0; g < total; g += 8u) {
    // ---- four lanes = unit u ----
    const uint32_t u = g + (uint32_t)(lane >> 2);
    const bool valid = u < total;
    const uint32_t un = un_next, xo = x_next;
    const uint32_t o = un & 31u, q = (un >> 5) & 7u, t3 = un >> 8;  // its brick, place and number in the brick
    const uint32_t o_first = u - t3;
    const uint32_t o_start = __shfl_sync(FULL, start, (int)o);
    const uint32_t o_g3 = __shfl_sync(FULL, g3, (int)o);
    uint32_t o_lpre = 0, o_dpre = 0;
    if (!LEVELS && pay) o_lpre = __shfl_sync(FULL, lpre, (int)o);
    if (LEVELS) o_dpre = __shfl_sync(FULL, dpre, (int)o);
    const uint64_t a = (uint64_t)v_next.x | ((uint64_t)v_next.y << 32), b = (uint64_t)v_next.z | ((uint64_t)v_next.w << 32);
    if (a | b) *reinterpret_cast<uint4*>(p.leaf + unit_word(xo, un)) = make_uint4(0u, 0u, 0u, 0u);  // zero for the next build
    if (g + 8u < total) fetch(g + 8u);
    const uint32_t ca = __popcll(a), cb = __popcll(b);
    const uint32_t ma = K >= 2 ? nonzero_bytes64(a) : 0u, mb = K >= 2 ? nonzero_bytes64(b) : 0u;
    const uint32_t ka = __popc(ma), kb = __popc(mb), kc = ka + kb;
    const uint32_t bal_a = __ballot_sync(FULL, ca != 0), bal_b = __ballot_sync(FULL, cb != 0);
    const uint32_t na4 = (bal_a >> (lane & 28)) & 15u, nb4 = (bal_b >> (lane & 28)) & 15u;
    // the unit's child mask: its lanes' a and b in turn
    const uint32_t m3 = ((na4 & 1u) | ((na4 & 2u) << 1) | ((na4 & 4u) << 2) | ((na4 & 8u) << 3)) |
                        (((nb4 & 1u) | ((nb4 & 2u) << 1) | ((nb4 & 4u) << 2) | ((nb4 & 8u) << 3)) << 1);
    const uint32_t k2 = K >= 3 ? __popc(m3) : 0u;
    const bool last = (lane & 3) == 3;
    // records | leaves << 16: of the lane, before it in the step, before it in its brick
    const uint32_t own = (ca + cb + kc + (last ? k2 : 0u)) | ((ca + cb) << 16);
    const uint32_t inc = warp_inclusive(own), before = inc - own;
    const uint32_t head = o_first > g ? o_first - g : 0u;  // the brick's first unit of this step
    const uint32_t in_brick = before - __shfl_sync(FULL, before, (int)((head * 4u) & 31u)) + (o_first < g ? carry : 0u);
    const uint32_t brick_end = in_brick + own;
    carry = __shfl_sync(FULL, brick_end, 31);
    const uint32_t S = __shfl_sync(FULL, inc, 31) & 0xffffu;  // records of the step
    const uint32_t c_at = before & 0xffffu;                   // the lane's first record in the step
    const uint32_t base = o_start + (in_brick & 0xffffu) - c_at;
    const uint32_t grp = o_start + (__shfl_sync(FULL, brick_end, lane | 3) & 0xffffu) - k2;  // the unit's children's group
    // the step's records stand brick by brick, brick s's starting at an even or odd word like in the
    // file: of the two slots before a brick's records one decides the parity
    const bool is_head = (lane & 3) == 0 && valid && (uint32_t)(lane >> 2) == head;
    const uint32_t heads = __ballot_sync(FULL, is_head);
    const uint32_t to_here = (2u << (lane & 28)) - 1u;
    const uint32_t later = heads & ~to_here;
    const uint32_t c_next = __shfl_sync(FULL, c_at, later ? __ffs(later) - 1 : 0);
    const uint32_t s = __popc(heads & to_here) - 1u;
    const uint32_t gap = 2u * s + ((odd0 + base) & 1u);
    if (is_head) sm.gaps[s & 7u] = gap;
    // parents of leaves: before the lane and in the step
    const uint32_t quad_lt = (1u << (lane & 28)) - 1u;
    const uint32_t own_recs = K >= 3 ? __popc(bal_a & quad_lt) + __popc(bal_b & quad_lt) : 0u;  // of earlier units' words
    const uint32_t pk = c_at - (before >> 16) - own_recs;
    const uint32_t n1 = __shfl_sync(FULL, pk + kc, 31);
    uint32_t da = 0, db = 0, d3 = 0;  // -levels: data records before a's, b's leaves and before the unit's average
    if (LEVELS) {
      const uint32_t in4 = (1u << (lane & 3)) - 1u;
      da = o_dpre + (in_brick & 0xffffu) - (pay ? 0u : in_brick >> 16) + t3;
      if (K >= 3) da += __popc(na4 & in4) + __popc(nb4 & in4);  // the words before it in the unit
      db = da + (pay ? ca : 0u) + ka + (K >= 3 && ca ? 1u : 0u);
      d3 = db + (pay ? cb : 0u) + kb + (K >= 3 && cb ? 1u : 0u);
    }
    const uint32_t has_k = __ballot_sync(FULL, kc != 0);
    if (kc) sm.words[__popc(has_k & lt)] = LaneWords{a, b, ma | (mb << 8) | (gap << 16), c_at | (pk << 16), base, da};
    __syncwarp();
    // item i0 + lane of the step's parents of leaves
    struct Parent {
      uint32_t mask, nc;  // its children
      uint32_t first;     // its first leaf's record in the step
      uint32_t r;         // its own
      uint32_t gap, base, d;  // d: -levels, data records before its leaves
    };
    auto parent = [&](uint32_t i0) {
      uint32_t h = 0;
      if (kc && pk - i0 < 32u) h = 1u << (pk - i0);
      h = __reduce_or_sync(FULL, h);
      const uint32_t slot = __popc(__ballot_sync(FULL, kc != 0 && pk < i0)) + __popc(h & le) - 1u;
      const LaneWords lw = sm.words[slot & 31u];
      const uint32_t m16 = lw.m16_gap & 0xffffu, ka1 = __popc(m16 & 0xffu);
      const uint32_t i = i0 + (uint32_t)lane - (lw.c_pk >> 16);  // its number among the owner's
      const bool in_b = i >= ka1;
      const uint32_t j = in_b ? i - ka1 : i;  // and among its word's
      const uint64_t v = in_b ? lw.b : lw.a;
      const uint32_t k = select8(in_b ? m16 >> 8 : m16 & 0xffu, j) & 7u;
      const uint32_t ca1 = __popcll(lw.a), l0 = __popcll(v & ((1ull << (8u * k)) - 1ull));
      const uint32_t word_at = (lw.c_pk & 0xffffu) + (in_b ? ca1 + ka1 : 0u);
      Parent t;
      t.mask = (uint32_t)(v >> (8u * k)) & 0xffu;
      t.nc = __popc(t.mask);
      t.first = word_at + l0;
      t.r = word_at + (uint32_t)__popcll(v) + j;
      t.gap = lw.m16_gap >> 16;
      t.base = lw.base;
      t.d = LEVELS ? lw.da + (in_b ? (pay ? ca1 : 0u) + ka1 + (K >= 3 && ca1 ? 1u : 0u) : 0u) + (pay ? l0 : 0u) + j : 0u;
      return t;
    };
    if (LEVELS) {  // the averages, each also a data record; the leaves' records are there already
      for (uint32_t i0 = 0; i0 < n1; i0 += 32u) {  // of leaves' parents
        const Parent t = parent(i0);
        if (i0 + (uint32_t)lane < n1) {
          Sum sum;
          if (pay) {
            average_records(e, t.nc, sum, [&](uint32_t k) { return dbase + t.d + k; });
          } else {
            sum.zero();
            sum.average(t.nc);
          }
          store_data_record(e, dbase + t.d + (pay ? t.nc : 0u), 0, sum.v);
        }
      }
      __syncwarp();
      Sum sa, sb;
      sa.zero();
      sb.zero();
      if (K >= 2) {  // of the lanes' words
        auto word_average = [&](uint64_t v, uint32_t m8, uint32_t d, Sum& sum) {
          uint32_t m = m8, at = d;
          average_records(e, __popc(m8), sum, [&](uint32_t) {
            at += pay ? __popc((uint32_t)(v >> (8u * ((uint32_t)__ffs(m) - 1u))) & 0xffu) : 0u;
            m &= m - 1;
            return dbase + at++;
          });
          if (K >= 3) store_data_record(e, dbase + at, 0, sum.v);
        };
        if (ka) word_average(a, ma, da, sa);
        if (kb) word_average(b, mb, db, sb);
      } else if (ca) {  // the leaves' parent is the stripe root
        if (pay) average_records(e, ca, sa, [&](uint32_t k) { return dbase + da + k; });
        else sa.average(ca);
      }
      if (K >= 3) {
        Sum s3;
        s3.zero();
#pragma unroll 1
        for (int k = 0; k < 8; k++) {
          float c[6];
#pragma unroll
          for (int i = 0; i < 6; i++) c[i] = __shfl_sync(FULL, (k & 1) ? sb.v[i] : sa.v[i], (lane & ~3) | (k >> 1));
          if ((m3 >> k) & 1u) s3.add(c);
        }
        sa = s3;
        if (last && valid) {
          sa.average(__popc(m3));
          if (K == kBrickLevels) store_data_record(e, dbase + d3, 0, sa.v);
        }
      }
      // for the brick's average: a child's, or (fewer levels) the brick's own
      if (K >= 3 ? (last && valid) : lane == 0) {
        float* c = e.upper_cache + (K == kBrickLevels ? upper_cell(U + 1, (uint64_t)xo * 8u + q) : upper_cell(U, xo)) * 6;
#pragma unroll
        for (int i = 0; i < 6; i++) c[i] = sa.v[i];
      }
    }
    if (K == kBrickLevels && last && valid) {  // the unit's own record
      uint64_t* t = nodes + (uint64_t)(o_g3 + t3) * 3u;
      t[0] = LEVELS ? dbase + d3 : 0;
      t[1] = e.node_base + grp;
      t[2] = lut[m3];
    }
    // ---- the records, window by window ----
    uint32_t next = 0, next_l = 0;  // the first parent whose record (whose last leaf's) is not yet written
    uint64_t leaf_data = 0;         // payload: the next leaf's data record
    if (!LEVELS && pay) leaf_data = dbase + __shfl_sync(FULL, o_lpre + (in_brick >> 16), 0);
    for (uint32_t w0 = 0; w0 < S; w0 += kWindow) {
      const uint32_t nrec = min(kWindow, S - w0);
      bulk_wait_read();  // the copies out of the window have read it
      __syncwarp();
      uint64_t* const rec = sm.win;
      {  // every slot a leaf's record, two words at a time
        const uint32_t n4 = ((nrec + 2u * __popc(heads)) * 3u + 1u) / 2u;
        ulonglong2* const q = reinterpret_cast<ulonglong2*>(rec);
        const uint64_t lead = pay ? 0ull : 1ull;
        // words 2 i and 2 i + 1 of the pattern lead, 0, ~0; 64 words on it is one word further
        const uint32_t f = (2u * (uint32_t)lane) % 3u;
        const ulonglong2 v0 = make_ulonglong2(f == 0 ? lead : (f == 1 ? 0ull : ~0ull), f == 0 ? 0ull : (f == 1 ? ~0ull : lead));
        const ulonglong2 v1 = make_ulonglong2(f == 2 ? lead : (f == 0 ? 0ull : ~0ull), f == 2 ? 0ull : (f == 0 ? ~0ull : lead));
        const ulonglong2 v2 = make_ulonglong2(f == 1 ? lead : (f == 2 ? 0ull : ~0ull), f == 1 ? 0ull : (f == 2 ? ~0ull : lead));
        for (uint32_t i = (uint32_t)lane; i < n4; i += 96u) {
          q[i] = v0;
          if (i + 32u < n4) q[i + 32u] = v1;
          if (i + 64u < n4) q[i + 64u] = v2;
        }
      }
      __syncwarp();
      auto put = [&](uint32_t slot, uint64_t d, uint32_t child, uint32_t mask) {
        uint64_t* t = rec + slot * 3u;
        t[0] = d;
        t[1] = e.node_base + child;
        t[2] = lut[mask];
      };
      while (next < n1) {  // the leaves' parents, in the order of their records
        const Parent t = parent(next);
        const bool in = next + (uint32_t)lane < n1 && t.r < w0 + kWindow;
        if (in) put(t.r - w0 + t.gap, LEVELS ? dbase + t.d + (pay ? t.nc : 0u) : 0, t.base + t.first, t.mask);
        const uint32_t done = __popc(__ballot_sync(FULL, in));
        next += done;
        if (done < 32u) break;
      }
      if (K >= 3) {  // the words' own records, in their units' groups
        const uint32_t gr = grp - base, below = 2u * (uint32_t)(lane & 3);
        const uint32_t r_a = gr + __popc(m3 & ((1u << below) - 1u)), r_b = gr + __popc(m3 & ((2u << below) - 1u));
        if (ca && r_a - w0 < kWindow) put(r_a - w0 + gap, LEVELS ? dbase + da + (pay ? ca : 0u) + ka : 0, base + c_at + ca, ma);
        if (cb && r_b - w0 < kWindow)
          put(r_b - w0 + gap, LEVELS ? dbase + db + (pay ? cb : 0u) + kb : 0, base + c_at + ca + ka + cb, mb);
      }
      if (pay && !LEVELS) {  // a leaf's data record: leaves stand in the order of their records
        __syncwarp();
        for (uint32_t i0 = 0; i0 < nrec; i0 += 32u) {
          const uint32_t r0 = w0 + i0;
          uint32_t h = 0;
          if (is_head && c_at - r0 < 32u) h = 1u << (c_at - r0);
          h = __reduce_or_sync(FULL, h);
          const uint32_t sg = __popc(__ballot_sync(FULL, is_head && c_at < r0)) + __popc(h & le) - 1u;
          uint64_t* t = rec + (i0 + (uint32_t)lane + sm.gaps[sg & 7u]) * 3u;
          const bool is_leaf = i0 + (uint32_t)lane < nrec && t[2] == ~0ull;
          const uint32_t bal = __ballot_sync(FULL, is_leaf);
          if (is_leaf) t[0] = leaf_data + __popc(bal & lt);
          leaf_data += __popc(bal);
        }
      }
      if (LEVELS && pay) {  // with the averages of the parents between them
        if (K < 2) {
          for (uint32_t t = 0; t < ca; t++) rec[(c_at + t + gap) * 3u] = dbase + da + t;  // (at most eight records)
        }
        while (next_l < n1) {
          const Parent t = parent(next_l);
          const bool have = next_l + (uint32_t)lane < n1;
          if (have)
            for (uint32_t k = 0; k < t.nc; k++)
              if (t.first + k - w0 < kWindow) rec[(t.first + k - w0 + t.gap) * 3u] = dbase + t.d + k;
          const uint32_t done = __popc(__ballot_sync(FULL, have && t.first + t.nc <= w0 + kWindow));
          next_l += done;
          if (done < 32u) break;
        }
      }
      bulk_fence();
      __syncwarp();
      if (is_head) {
        const uint32_t r0 = max(c_at, w0), r1 = min(later ? c_next : S, w0 + kWindow);
        if (r0 < r1) {
          uint64_t* dst = nodes + (uint64_t)(base + r0) * 3u;
          const uint64_t* src = rec + (r0 - w0 + gap) * 3u;
          uint32_t n = (r1 - r0) * 3u;
          if (reinterpret_cast<uintptr_t>(dst) & 8u) {
            *dst++ = *src++;
            n--;
          }
          if (n & 1u) dst[n - 1] = src[n - 1];
          if (n >= 2u) bulk_store(dst, src, (n & ~1u) * 8u);
        }
      }
      bulk_commit();
    }
    __syncwarp();  // the lanes' words are free for the next step
  }
  if (LEVELS && K) {
    __syncwarp();
    if (mine) {
      float* c = e.upper_cache + upper_cell(U, x) * 6;
      Sum s4;
      s4.zero();
      if (K == kBrickLevels) {  // from its children's averages
        for (uint32_t m = units; m; m &= m - 1)
          s4.add(e.upper_cache + upper_cell(U + 1, (uint64_t)x * 8u + (uint32_t)__ffs(m) - 1u) * 6);
        s4.average(__popc(units));
#pragma unroll
        for (int i = 0; i < 6; i++) c[i] = s4.v[i];
      } else {
#pragma unroll
        for (int i = 0; i < 6; i++) s4.v[i] = c[i];
      }
      store_data_record(e, dbase + dtop, 0, s4.v);
      if (U == 0)
        for (int i = 0; i < 6; i++) e.root_out[i] = __float_as_uint(s4.v[i]);
    }
  }
  if (mine && p.touch) reinterpret_cast<uint4*>(p.touch)[x] = make_uint4(0u, 0u, 0u, 0u);  // zero for the next build
  if (K == 0 && lane == 0) {  // one voxel
    p.leaf[0] = 0u;
    if (LEVELS && pay) {
      float c[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
      leaf_value(e, e.winners[0], c);
      for (int i = 0; i < 6; i++) e.root_out[i] = __float_as_uint(c[i]);
    }
  }
}

// The share of the stripe's warp i: bricks_per_warp consecutive ones of its non-empty bricks.
template <bool LEVELS>
__device__ __forceinline__ void emit_warp(const Stripe& p, const EmitJob& e, uint64_t i, int lane, WarpScratch& sm,
                                          const uint64_t* __restrict__ lut) {
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t W = upper_words(p.U), off = upper_off(p.U), all = p.upre[off + W];
  const uint64_t r0 = i * e.bricks_per_warp;
  if (r0 >= all) return;
  uint32_t left = (uint32_t)min((uint64_t)all - r0, (uint64_t)e.bricks_per_warp);
  // the word of the first, and the word's bricks from it on
  uint32_t w = warp_search(W, (uint32_t)r0, lane, [&](uint32_t i) { return p.upre[off + i]; });
  uint32_t first;
  {
    const uint32_t b = p.ubits[off + w], skip = (uint32_t)r0 - p.upre[off + w];
    first = __ballot_sync(FULL, ((b >> lane) & 1u) && __popc(b & lt) >= skip);
  }
  // Lane k's brick: the k-th of the n next; w and first move past them.
  uint32_t* const list = reinterpret_cast<uint32_t*>(sm.words);
  auto next_bricks = [&](uint32_t n) {
    uint32_t got = 0;
    while (got < n && w < W) {
      const uint32_t mine = w + (uint32_t)lane < W ? p.ubits[off + w + (uint32_t)lane] : 0u;
      uint32_t some = __ballot_sync(FULL, (lane == 0 ? mine & first : mine) != 0u);
      uint32_t to = w + 32u, to_first = ~0u;
      while (some) {
        const uint32_t k = (uint32_t)__ffs(some) - 1u;
        some &= some - 1u;
        const uint32_t b = __shfl_sync(FULL, mine, (int)k) & (k == 0 ? first : ~0u);
        const uint32_t pos = got + __popc(b & lt);
        const bool set = (b >> lane) & 1u;
        if (set && pos < n) list[pos] = (w + k) * 32u + (uint32_t)lane;
        got += __popc(b);
        if (got >= n) {
          to = w + k;
          to_first = __ballot_sync(FULL, set && pos >= n);
          break;
        }
      }
      w = to;
      first = to_first;
    }
    __syncwarp();
    const uint32_t x = list[min((uint32_t)lane, n - 1u)];
    __syncwarp();
    return x;
  };
  uint32_t n = min(left, 32u);
  BrickIn in = load_bricks<LEVELS>(p, next_bricks(n), n, lane);
  for (;;) {
    left -= n;
    const uint32_t n_next = min(left, 32u);
    BrickIn next = in;
    if (n_next) next = load_bricks<LEVELS>(p, next_bricks(n_next), n_next, lane);
    emit_bricks<LEVELS>(p, e, n, in, lane, sm, lut);
    if (!n_next) break;
    n = n_next;
    in = next;
  }
  bulk_wait_all();
}

// Nodes of the stripe written before the children of cell a of level m < U.
__device__ __forceinline__ uint32_t children_base(const Stripe& p, int m, uint32_t a) {
  uint32_t s = 0;
  for (int l = 1; l <= m + 1; l++) s += upper_rank(p, l, 8u * (a >> (3 * (m + 1 - l))));
  for (int l = m + 2; l <= p.U; l++) s += upper_rank(p, l, (a + 1u) << (3 * (l - m)));
  const uint2 v = brick_prefix(p, (a + 1u) << (3 * (p.U - m)));
  return s + v.x + v.y;
}

// Data records of the stripe (-levels) before the average of cell z of level m < U.
__device__ __forceinline__ uint32_t data_before(const Stripe& p, bool payload, int m, uint32_t z) {
  uint32_t s = 0;
  for (int l = 1; l <= m; l++) s += upper_rank(p, l, z >> (3 * (m - l)));
  for (int l = m + 1; l <= p.U; l++) s += upper_rank(p, l, (z + 1u) << (3 * (l - m)));
  const uint2 v = brick_prefix(p, (z + 1u) << (3 * (p.U - m)));
  return s + (payload ? v.x : 0u) + v.y;
}

// Cell i of levels 0 .. U-1.
__device__ __forceinline__ void upper_node(const Stripe& p, const EmitJob& e, uint64_t i) {
  int m = 0;
  while (i >= upper_cell(m + 1, 0)) m++;
  if (m >= p.U) return;
  const uint32_t z = (uint32_t)(i - upper_cell(m, 0));
  if (!((p.ubits[upper_off(m) + (z >> 5)] >> (z & 31u)) & 1u)) return;
  const uint32_t mask = upper_byte(p, m + 1, z);
  const float* v = e.levels ? e.upper_cache + i * 6 : nullptr;
  if (m == 0) {  // the stripe root, which the host writes
    if (v) {
      for (int k = 0; k < 6; k++) e.root_out[k] = __float_as_uint(v[k]);
      store_data_record(e, e.data_base + e.data_span - 1, 0, v);
    }
    return;
  }
  const uint32_t sib = upper_byte(p, m, z >> 3) & ((1u << (z & 7u)) - 1u);
  uint64_t di = 0;
  if (v) {
    di = e.data_base + data_before(p, !e.binary, m, z);
    store_data_record(e, di, 0, v);
  }
  store_node_record(e, e.node_base + children_base(p, m - 1, z >> 3) + __popc(sib), di,
                    e.node_base + children_base(p, m, z), child_offsets(mask));
}

// CTA `cta` of a stripe.  Without -levels the first ones write the records above the bricks (which wait
// for averages otherwise): a launch of their own took 7 us of a small call, and 0.1 of 12 ms on the
// 20M-triangle soup.
template <bool LEVELS>
__device__ __forceinline__ void emit_cta(const Stripe& p, const EmitJob& e, uint64_t cta, WarpScratch* ws,
                                         const uint64_t* lut) {
  if (!LEVELS) {
    const uint32_t upper = upper_node_ctas(p.U);
    if (cta < upper) {
      upper_node(p, e, cta * kTreeThreads + threadIdx.x);
      return;
    }
    cta -= upper;
  }
  const uint32_t warp = threadIdx.x >> 5;
  const uint64_t i = cta * kTreeWarps + warp;
  if (LEVELS && e.levels) emit_warp<true>(p, e, i, threadIdx.x & 31, ws[warp], lut);
  else emit_warp<false>(p, e, i, threadIdx.x & 31, ws[warp], lut);
}

template <bool SINGLE, bool LEVELS, int CTAS>
__global__ void __launch_bounds__(kTreeThreads, CTAS) kb_emit(const Stripe* __restrict__ stripes,
                                                              const EmitJob* __restrict__ emits,
                                                              const uint64_t* __restrict__ cta_beg, uint32_t n,
                                                              Stripe p0, EmitJob e0, unsigned long long* large_ctr) {
  __shared__ uint64_t lut[256];  // child_offsets of every mask
  __shared__ WarpScratch ws[kTreeWarps];
  static_assert(kTreeThreads == 256, "one table entry per thread, and upper_node_ctas");
  static_assert(kWindow % 2 == 0 && kSlots % 2 == 0, "windows start on 16 bytes, every window's parity is the same");
  lut[threadIdx.x] = child_offsets(threadIdx.x);
  pdl_enter();
  if (blockIdx.x == 0 && threadIdx.x < kLargeCtrWords) large_ctr[threadIdx.x] = 0ull;  // for the next build
  if constexpr (SINGLE) {
    __syncthreads();
    emit_cta<LEVELS>(p0, e0, blockIdx.x, ws, lut);
  } else {
    __shared__ Stripe sp;
    __shared__ EmitJob se;
    uint64_t cta;
    const uint32_t s = cta_stripe(cta_beg, n, cta);
    stage(sp, stripes[s]);
    stage(se, emits[s]);
    __syncthreads();
    emit_cta<LEVELS>(sp, se, cta, ws, lut);
  }
}

// ---- the levels above the bricks ----
// Average of cell z of level l from the cells of level l + 1.
__device__ __forceinline__ void average_cell(const Stripe& p, const EmitJob& e, int l, uint32_t z) {
  if (!((p.ubits[upper_off(l) + (z >> 5)] >> (z & 31u)) & 1u)) return;
  const uint32_t mask = upper_byte(p, l + 1, z);
  const float2* src = reinterpret_cast<const float2*>(e.upper_cache + upper_cell(l + 1, (uint64_t)z * 8u) * 6);
  float2 child[8][3];
#pragma unroll
  for (uint32_t k = 0; k < 8; k++)
    if ((mask >> k) & 1u)
      for (int q = 0; q < 3; q++) child[k][q] = src[k * 3 + q];
  Sum s;
  s.zero();
#pragma unroll
  for (uint32_t k = 0; k < 8; k++)
    if ((mask >> k) & 1u) {
      const float c[6] = {child[k][0].x, child[k][0].y, child[k][1].x, child[k][1].y, child[k][2].x, child[k][2].y};
      s.add(c);
    }
  s.average(__popc(mask));
  float2* out = reinterpret_cast<float2*>(e.upper_cache + upper_cell(l, z) * 6);
#pragma unroll
  for (int q = 0; q < 3; q++) out[q] = make_float2(s.v[2 * q], s.v[2 * q + 1]);
}

// Level l of the stripes that have it above their bricks, one thread per cell (grid.y: the stripes).
__global__ void __launch_bounds__(256) kb_upper_avg(const Stripe* __restrict__ stripes, const EmitJob* __restrict__ emits,
                                                    uint32_t n, int l, const __grid_constant__ Stripe p0,
                                                    const __grid_constant__ EmitJob e0) {
  pdl_enter();
  const uint32_t z = blockIdx.x * 256u + threadIdx.x;
  for (uint32_t s = blockIdx.y; s < n; s += gridDim.y) {
    const Stripe& p = stripes ? stripes[s] : p0;
    const EmitJob& e = stripes ? emits[s] : e0;
    if (e.levels && l < p.U && z < (1u << (3 * l)) && p.wpre[upper_words(p.U)].x) average_cell(p, e, l, z);
  }
}

// Levels min(l_hi, U - 1) .. 0 and then the records above the bricks, CTAS CTAs (a cluster) per stripe.
// Bound by latency, level after level.  One CTA took 29 us for the 4,681 cells above the bricks of a
// 512 stripe, most of it for the 4,096 of level 4, and another launch 8 us for their records.
constexpr uint32_t kTopThreads = 512;  // the cells of level 3
template <uint32_t CTAS>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(kTopThreads)
    kb_upper_top(const Stripe* __restrict__ stripes, const EmitJob* __restrict__ emits, int l_hi,
                 const __grid_constant__ Stripe p0, const __grid_constant__ EmitJob e0) {
  pdl_enter();
  const Stripe& p = stripes ? stripes[blockIdx.x / CTAS] : p0;
  const EmitJob& e = stripes ? emits[blockIdx.x / CTAS] : e0;
  if (p.U == 0 || p.wpre[upper_words(p.U)].x == 0) return;
  const uint32_t t = (blockIdx.x % CTAS) * kTopThreads + threadIdx.x;
  if (e.levels) {
    auto sync = [] {
      if (CTAS == 1) __syncthreads();
      else asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    };
    int l = min(l_hi, p.U - 1);
    for (; l > 3; l--) {
      for (uint32_t z = t; z < (1u << (3 * l)); z += CTAS * kTopThreads) average_cell(p, e, l, z);
      sync();
    }
    if (t < kTopThreads)  // the cluster's first CTA
      for (; l >= 0; l--) {
        if (t < (1u << (3 * l))) average_cell(p, e, l, t);
        __syncthreads();
      }
    sync();
  }
  for (uint64_t i = t; i < upper_cell(p.U, 0); i += CTAS * kTopThreads) upper_node(p, e, i);
}

}  // namespace

// ===========================================================================
// Launch wrappers
// ===========================================================================
namespace {
Stripe stripe_or_zero(const Stripe* s) {
  Stripe p;
  std::memset(&p, 0, sizeof(p));
  if (s) p = *s;
  return p;
}
EmitJob emit_or_zero(const EmitJob* s) {
  EmitJob e;
  std::memset(&e, 0, sizeof(e));
  if (s) e = *s;
  return e;
}
}  // namespace

void launch_b_bricks(const Stripe* stripes, const uint64_t* cta_beg, uint32_t n, uint64_t ctas, const Stripe* single,
                     cudaStream_t st) {
  if (ctas == 0) return;
  KScope k("bricks", st);
  const Stripe p0 = stripe_or_zero(single);
  launch_k(single ? kb_bricks<true> : kb_bricks<false>, dim3((unsigned)ctas), dim3(32 * kBrickCta), 0, st, stripes,
           cta_beg, n, p0);
}

void launch_b_upper(const Stripe* stripes, uint32_t n, int max_upper, uint32_t* counts,
                    const unsigned long long* large_ctr, uint64_t* large_out, const uint64_t* code, uint64_t* code_out,
                    const Stripe* single, cudaStream_t st) {
  if (n == 0) return;
  KScope k("upper", st);
  // level U has 8192, 1024, 128, ... words: one round of one word a thread, or eight
  auto* kern = max_upper >= 6 ? kb_upper<1024, 8> : (max_upper == 5 ? kb_upper<1024, 1> : kb_upper<128, 1>);
  launch_k(kern, dim3(n), dim3(max_upper >= 5 ? 1024 : 128), 0, st, single ? nullptr : stripes, counts, large_ctr,
           large_out, code, code_out, stripe_or_zero(single));
}

void launch_b_leaf_payload(const Stripe* stripes, const EmitJob* emits, const uint64_t* cta_beg, uint32_t n,
                           uint64_t ctas, uint32_t ept, const Stripe* sp, const EmitJob* se, cudaStream_t st) {
  if (ctas == 0) return;
  KScope k("leaf_payload", st);
  launch_k(se ? kb_leaf_payload<true> : kb_leaf_payload<false>, dim3((unsigned)ctas), dim3(kTreeThreads), 0, st, stripes,
           emits, cta_beg, n, ept, stripe_or_zero(sp), emit_or_zero(se));
}

void launch_b_emit(const Stripe* stripes, const EmitJob* emits, const uint64_t* cta_beg, uint32_t n, uint64_t ctas,
                   bool levels, int num_sms, unsigned long long* large_ctr, const Stripe* sp, const EmitJob* se,
                   cudaStream_t st) {
  if (ctas == 0) return;
  KScope k("emit", st);
  // With -levels two CTAs fit an SM only with 128 registers a thread, some of them spilled: where one CTA
  // per SM is all there is, the kernel that keeps everything (3,001 triangles at gridsize 128 45 and 35 us;
  // the heightfield at 512, more CTAs than SMs, 51 and 63).
  auto* kern = !levels ? (sp ? kb_emit<true, false, kEmitCtas> : kb_emit<false, false, kEmitCtas>)
               : !sp   ? kb_emit<false, true, 2>
                       : (ctas <= (uint64_t)num_sms ? kb_emit<true, true, 1> : kb_emit<true, true, 2>);
  launch_k(kern, dim3((unsigned)ctas), dim3(kTreeThreads), 0, st, stripes, emits, cta_beg, n, stripe_or_zero(sp),
           emit_or_zero(se), large_ctr);
}

void launch_b_upper_levels(const Stripe* stripes, const EmitJob* emits, uint32_t n, int max_upper, const Stripe* sp,
                           const EmitJob* se, cudaStream_t st) {
  if (n == 0 || max_upper == 0) return;
  constexpr int kTop = 4;  // 4,096 cells: one per thread of eight CTAs
  if (sp) stripes = nullptr;
  for (int l = max_upper - 1; l > kTop; l--) {
    KScope k("upper_average", st);
    launch_k(kb_upper_avg, dim3(1u << (3 * l - 8), n < 4096u ? n : 4096u), dim3(256), 0, st, stripes, emits, n, l,
             stripe_or_zero(sp), emit_or_zero(se));
  }
  KScope k("upper_top", st);
  // up to level 2 (64 cells, U = 3) one CTA; a cluster's barriers cost more there
  const bool one = max_upper <= 3;
  launch_k(one ? kb_upper_top<1> : kb_upper_top<8>, dim3(one ? n : n * 8u), dim3(kTopThreads), 0, st, stripes, emits, kTop,
           stripe_or_zero(sp), emit_or_zero(se));
}

}  // namespace ooc
