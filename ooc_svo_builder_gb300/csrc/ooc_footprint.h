// An upper bound on the voxels one triangle can set, used by the serving loop's
// admission footprint.  Header-only so that a host-side test can check it against
// the oracle's voxel counts.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>

namespace ooc {

// The volume that holds every voxel overlapping triangle v (9 floats; grid coordinates are v * unit_div): a
// voxel passing the overlap test has its centre within sqrt(3)/2 of the triangle, and all of it within
// sqrt(3), so it lies within the triangle grown by a ball of radius sqrt(3) voxels, whose volume is
// 2 r A + (pi / 2) r^2 L + (4 / 3) pi r^3 for area A and perimeter L (Steiner's formula for a flat convex
// body).  Infinite for a degenerate triangle, which has no plane test (its normal is NaN).
inline double grown_volume(const float* v, float unit_div) {
  // in voxel units
  double p[3][3];
  for (int k = 0; k < 3; k++)
    for (int a = 0; a < 3; a++) p[k][a] = (double)v[3 * k + a] * (double)unit_div;
  double e[3][3], len = 0.0;
  for (int k = 0; k < 3; k++) {
    double l2 = 0.0;
    for (int a = 0; a < 3; a++) {
      e[k][a] = p[(k + 1) % 3][a] - p[k][a];
      l2 += e[k][a] * e[k][a];
    }
    len += std::sqrt(l2);
  }
  const double cx = e[0][1] * e[1][2] - e[0][2] * e[1][1], cy = e[0][2] * e[1][0] - e[0][0] * e[1][2],
               cz = e[0][0] * e[1][1] - e[0][1] * e[1][0];
  const double area = 0.5 * std::sqrt(cx * cx + cy * cy + cz * cz);
  if (!(area > 1e-6) || !std::isfinite(area) || !std::isfinite(len)) return HUGE_VAL;
  const double r = std::sqrt(3.0), pi = 3.14159265358979323846;
  return 1.01 * (2.0 * r * area + 0.5 * pi * r * r * len + 4.0 / 3.0 * pi * r * r * r) + 1.0;
}

// Of two upper bounds, the voxels of a triangle's grid box (no other is tested) and the volume of those that
// overlap it, the smaller.  A small box (every small triangle of a fine mesh) is taken as it is, sparing
// the sizing thread the area bound's square roots.
inline double box_or_grown(const float* v, float unit_div, double box) {
  return box <= 64.0 ? box : std::min(box, grown_volume(v, unit_div));
}

// Voxels of the clamped grid box of triangle v in an N^3 grid.
inline double box_voxels(const float* v, float unit_div, uint64_t N) {
  double box = 1.0;
  for (int a = 0; a < 3; a++) {
    const float lo = std::min(v[a], std::min(v[3 + a], v[6 + a])) * unit_div;
    const float hi = std::max(v[a], std::max(v[3 + a], v[6 + a])) * unit_div;
    // NaN or out-of-range coordinates count as the whole axis
    const double l = (lo >= 0.0f) ? std::min((double)lo, (double)N - 1) : 0.0;
    const double h = (hi < (float)N) ? std::max((double)hi, 0.0) : (double)N - 1;
    box *= (h >= l) ? std::floor(h) - std::floor(l) + 1.0 : (double)N;
  }
  return box;
}

// Voxels of an N^3 grid that triangle v can set: at most those of its clamped grid box.
inline double voxel_bound(const float* v, float unit_div, uint64_t N) {
  return box_or_grown(v, unit_div, box_voxels(v, unit_div, N));
}

}  // namespace ooc
