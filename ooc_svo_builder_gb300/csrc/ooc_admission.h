// The device memory a request of the serving loop is admitted for.  Header-only so that a host-side
// test can hold it against what the engine allocates.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "ooc_footprint.h"
#include "ooc_internal.h"
#include "ooc_svo_gpu.h"

namespace ooc {

// An upper bound on the partitions of `side`^3 voxels, `per_axis` along each axis, whose inclusive box test
// triangle v passes (partitioner.cpp:101-149).  A twentieth of a voxel covers the rounding of the
// slabs' bounds.
inline double partition_bound(const float* v, float unit_div, uint64_t side, uint64_t per_axis) {
  constexpr double slack = 0.05;
  double n = 1.0;
  for (int a = 0; a < 3; a++) {
    const double lo = (double)std::min(v[a], std::min(v[3 + a], v[6 + a])) * unit_div - slack;
    const double hi = (double)std::max(v[a], std::max(v[3 + a], v[6 + a])) * unit_div + slack;
    if (!std::isfinite(lo) || !std::isfinite(hi)) {
      n *= (double)per_axis;
      continue;
    }
    const double j0 = std::max(std::ceil(lo / (double)side) - 1.0, 0.0);
    const double j1 = std::min(std::floor(hi / (double)side), (double)per_axis - 1.0);
    n *= std::max(j1 - j0 + 1.0, 0.0);
  }
  return n;
}

// HBM a request may hold while it is in flight: its triangles; every stripe's arrays (stripe_bytes) and job
// tables; its (triangle, stripe) items; and for an upper bound on its nodes their records, the winners of its
// leaves, and, with several stripes, its records once more, parked until its sizes are known.  A tree with
// L leaves at depth D has at most min(8^l, L) nodes at level l.  The leaves are at most the summed
// per-triangle bounds on the voxels a triangle can set: the voxels of its grid box (voxelizer.cpp:189-204
// tests no other), and, for a triangle with a finite plane, the voxels that overlap it (voxel_bound).  (The
// quarter that the engines' buffers grow by beyond need is not in it.)
inline uint64_t footprint(const ooc_mesh& m) {
  const ooc_build_params& p = m.params;
  const uint64_t N = p.gridsize;
  const uint64_t stride = p.geometry_only ? 9 : 21;
  int D = 0;
  while ((1ull << D) < N) D++;
  const uint64_t P = ooc_estimate_partitions(N, p.memory_limit_mb);
  int kP = 0;
  while ((1ull << (3 * kP)) < P) kP++;
  const int Ds = std::min(D - kP, kMaxStripeDepth);
  const uint64_t stripes = (N * N * N) >> (3 * Ds);
  const float unit_div = 1.0f / ((p.bbox_max[0] - p.bbox_min[0]) / (float)N);
  const double cells = (double)N * (double)N * (double)N;
  double leaves = 0.0, pairs = P > 1 ? 0.0 : (double)m.n_tris;
  for (uint64_t t = 0; t < m.n_tris && (leaves < cells || P > 1); t++) {
    const float* v = m.tris + t * stride;
    if (leaves < cells) leaves += voxel_bound(v, unit_div, N);
    if (P > 1) pairs += partition_bound(v, unit_div, N >> kP, 1ull << kP);
  }
  leaves = std::min(leaves, cells);
  double nodes = 0.0;
  for (int l = 0; l <= D; l++) nodes += std::min(std::ldexp(1.0, 3 * l), leaves);
  constexpr double kTables = 2048.0;  // of a stripe: its jobs, its entries of the launches' tables
  const double items = pairs * (double)((stripes + P - 1) / P);
  const double data = 2.0 + (p.geometry_only ? 0.0 : leaves) + (p.generate_levels ? nodes : 0.0);
  const double records = (nodes + 1.0) * 24.0 + data * 32.0;
  double bytes = (double)((m.n_tris * stride * 4 + 255) / 256 * 256);
  bytes += (double)stripes * ((double)stripe_bytes(stripe_sizes(Ds, !p.geometry_only, p.generate_levels != 0)) + kTables);
  bytes += items * kItemBytes + std::min(items, (double)kMaxBig) * 16.0 + (P > 1 ? pairs * 4.0 : 0.0);
  bytes += records * (stripes > 1 ? 2.0 : 1.0) + (p.geometry_only ? 0.0 : leaves * 8.0);
  return (uint64_t)std::min(bytes, 1.8e19);
}

}  // namespace ooc
