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

// An upper bound on the (triangle, partition) pairs of n triangles whose clamped grid boxes hold `boxes` voxels
// together, with P partitions of `side`^3 voxels (the inclusive box test, partitioner.cpp:101-149).  A box of
// e voxels along an axis reaches at most e / side + 2 partitions along it, the slabs' rounded bounds included;
// the product over the axes is at most 8 + box (12 / side + 6 / side^2 + 1 / side^3), every extent being at
// least one.  It takes a sum from the pass over the triangles: requests wait behind that pass, and working
// each triangle's partitions out cost the serving loop 2 to 10% of its capacity.
inline double pair_bound(double n, double boxes, uint64_t side, uint64_t P) {
  const double r = 1.0 / (double)side;
  return std::min(n * (double)P, 8.0 * n + boxes * r * (12.0 + r * (6.0 + r)));
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
  double leaves = 0.0, boxes = 0.0;
  const double enough = P > 1 ? HUGE_VAL : cells;
  for (uint64_t t = 0; t < m.n_tris && leaves < enough; t++) {
    const float* v = m.tris + t * stride;
    const double box = box_voxels(v, unit_div, N);
    boxes += box;
    leaves += box_or_grown(v, unit_div, box);
  }
  const double pairs = P > 1 ? pair_bound((double)m.n_tris, boxes, N >> kP, P) : (double)m.n_tris;
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
