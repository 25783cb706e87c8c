// Device helpers shared by the voxelization and octree kernels.
//
// Every FP32 expression here is evaluated in the reference's order
// (voxelizer.cpp:189-299, BarycentricCoords.h:4-33, OctreeBuilder.cpp:81-99)
// with one rounding per operation: the translation units that include this
// file are compiled with -fmad=false, and IEEE division and square root
// (nvcc's defaults -prec-div=true -prec-sqrt=true, no fast-math).
#pragma once

#include <stdint.h>

#include "ooc_morton.h"

namespace ooc {

// std::min / std::max argument semantics (intersection.h:9-18; voxelizer.cpp:228).
__device__ __forceinline__ float smin(float a, float b) { return (b < a) ? b : a; }
__device__ __forceinline__ float smax(float a, float b) { return (a < b) ? b : a; }
__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// glm-order dot products: (a.x*b.x + a.y*b.y) + a.z*b.z.
__device__ __forceinline__ float dot3(float ax, float ay, float az, float bx, float by, float bz) {
  const float px = __fmul_rn(ax, bx), py = __fmul_rn(ay, by), pz = __fmul_rn(az, bz);
  return __fadd_rn(__fadd_rn(px, py), pz);
}
__device__ __forceinline__ float dot2(float ax, float ay, float bx, float by) {
  return __fadd_rn(__fmul_rn(ax, bx), __fmul_rn(ay, by));
}

// Triangle vertices (the first nine floats of either record layout).
struct TriVerts {
  float v[3][3];
};

__device__ __forceinline__ TriVerts load_verts(const float* __restrict__ tris, uint64_t t, int stride) {
  TriVerts r;
  const float* p = tris + t * (uint64_t)stride;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    r.v[k][0] = __ldg(p + 3 * k);
    r.v[k][1] = __ldg(p + 3 * k + 1);
    r.v[k][2] = __ldg(p + 3 * k + 2);
  }
  return r;
}

// computeBoundingBox (intersection.h:9-18) followed by the grid-box truncation
// of voxelizer.cpp:189-196.
__device__ __forceinline__ void grid_box(const TriVerts& t, float unit_div, int gmin[3], int gmax[3]) {
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float lo = smin(t.v[0][a], smin(t.v[1][a], t.v[2][a]));
    const float hi = smax(t.v[0][a], smax(t.v[1][a], t.v[2][a]));
    gmin[a] = __float2int_rz(__fmul_rn(lo, unit_div));
    gmax[a] = __float2int_rz(__fmul_rn(hi, unit_div));
  }
}

// Per-triangle constants of the Schwarz-Seidel test (voxelizer.cpp:207-254).
struct TriSetup {
  float n[3];
  float d1, d2;
  float xy[3][2], dxy[3];
  float yz[3][2], dyz[3];
  float zx[3][2], dzx[3];
};

__device__ __forceinline__ void normalize3(float& x, float& y, float& z) {
  const float r = __fdiv_rn(1.0f, __fsqrt_rn(dot3(x, y, z, x, y, z)));
  x = __fmul_rn(x, r);
  y = __fmul_rn(y, r);
  z = __fmul_rn(z, r);
}

__device__ __forceinline__ void tri_normal(const TriVerts& t, float n[3]) {
  const float e0x = __fsub_rn(t.v[1][0], t.v[0][0]), e0y = __fsub_rn(t.v[1][1], t.v[0][1]),
              e0z = __fsub_rn(t.v[1][2], t.v[0][2]);
  const float e1x = __fsub_rn(t.v[2][0], t.v[1][0]), e1y = __fsub_rn(t.v[2][1], t.v[1][1]),
              e1z = __fsub_rn(t.v[2][2], t.v[1][2]);
  // cross(e0, e1)
  n[0] = __fsub_rn(__fmul_rn(e0y, e1z), __fmul_rn(e0z, e1y));
  n[1] = __fsub_rn(__fmul_rn(e0z, e1x), __fmul_rn(e0x, e1z));
  n[2] = __fsub_rn(__fmul_rn(e0x, e1y), __fmul_rn(e0y, e1x));
  normalize3(n[0], n[1], n[2]);
}

__device__ __forceinline__ float edge_offset(float a, float b, float va, float vb, float u) {
  // (-1 * dot(ne, v.proj)) + max(0, u*ne[0]) + max(0, u*ne[1])
  return __fadd_rn(__fadd_rn(-dot2(a, b, va, vb), smax(0.0f, __fmul_rn(u, a))), smax(0.0f, __fmul_rn(u, b)));
}

// The edge functions of the three projections from the edges `e` and the normal s.n.
__device__ __forceinline__ void edge_setup(const TriVerts& t, const float e[3][3], float u, TriSetup& s) {
  const float fz = (s.n[2] < 0.0f) ? -1.0f : 1.0f;
  const float fx = (s.n[0] < 0.0f) ? -1.0f : 1.0f;
  const float fy = (s.n[1] < 0.0f) ? -1.0f : 1.0f;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    // XY: (-e.y, e.x), YZ: (-e.z, e.y), ZX: (-e.x, e.z); sign-flipped by n.
    // Multiplying by +-1 is exact, like the reference's -1.0f * vec2.
    s.xy[k][0] = __fmul_rn(fz, -e[k][1]);
    s.xy[k][1] = __fmul_rn(fz, e[k][0]);
    s.yz[k][0] = __fmul_rn(fx, -e[k][2]);
    s.yz[k][1] = __fmul_rn(fx, e[k][1]);
    s.zx[k][0] = __fmul_rn(fy, -e[k][0]);
    s.zx[k][1] = __fmul_rn(fy, e[k][2]);
    s.dxy[k] = edge_offset(s.xy[k][0], s.xy[k][1], t.v[k][0], t.v[k][1], u);
    s.dyz[k] = edge_offset(s.yz[k][0], s.yz[k][1], t.v[k][1], t.v[k][2], u);
    s.dzx[k] = edge_offset(s.zx[k][0], s.zx[k][1], t.v[k][2], t.v[k][0], u);
  }
}

// True when the voxels of a line that pass the plane test form one run (walk_line):
// every constant of the test finite and small enough that no sum or product of the
// test overflows or turns into NaN (voxel coordinates are below 2^60 too).
__device__ __forceinline__ bool monotone_setup(const TriSetup& s, float coord_max) {
  const float lim = 1.0e18f;
  bool ok = fabsf(s.d1) < lim && fabsf(s.d2) < lim && coord_max < lim;
#pragma unroll
  for (int a = 0; a < 3; a++) ok = ok && fabsf(s.n[a]) < lim;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    ok = ok && fabsf(s.xy[k][0]) < lim && fabsf(s.xy[k][1]) < lim && fabsf(s.dxy[k]) < lim;
    ok = ok && fabsf(s.yz[k][0]) < lim && fabsf(s.yz[k][1]) < lim && fabsf(s.dyz[k]) < lim;
    ok = ok && fabsf(s.zx[k][0]) < lim && fabsf(s.zx[k][1]) < lim && fabsf(s.dzx[k]) < lim;
  }
  return ok;  // NaN fails every comparison
}

}  // namespace ooc
