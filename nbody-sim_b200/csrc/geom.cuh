// geom.cuh -- the root cube, the Morton key of a position and the rule for
// searches by cells, shared by the kernels that make keys and search them.
#pragma once
#include "common.cuh"
#include "kernels.cuh"

namespace nb {

// Root geometry from the encoded bbox, float arithmetic as the reference host
// code (BHTree.cu:440-446 then :481-485).
__device__ inline void compute_geom(const unsigned long long* enc, TreeGeom& g) {
  float bmin[3], bmax[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double lo = from_ordered_bits(enc[k]), hi = from_ordered_bits(enc[3 + k]);
    if (!(lo <= hi)) { lo = 0.0; hi = 0.0; }
    // round outward so the float box still holds every FP64 position
    float flo = __double2float_rd(lo), fhi = __double2float_ru(hi);
    float mid = __fmul_rn(__fadd_rn(flo, fhi), 0.5f);
    float half = __fmul_rn(__fmul_rn(__fsub_rn(fhi, flo), 0.5f), 1.001f);
    bmin[k] = __fsub_rn(mid, half);
    bmax[k] = __fadd_rn(mid, half);
    g.bmin[k] = bmin[k];
    g.bmax[k] = bmax[k];
    g.rc[k] = __fmul_rn(__fadd_rn(bmin[k], bmax[k]), 0.5f);
  }
  float ext = fmaxf(fmaxf(__fsub_rn(bmax[0], bmin[0]), __fsub_rn(bmax[1], bmin[1])),
                    __fsub_rn(bmax[2], bmin[2]));
  g.rhs = __fmul_rn(__fmul_rn(ext, 0.5f), 1.001f);
  double rhs = (double)g.rhs;
#pragma unroll
  for (int k = 0; k < 3; ++k) g.lo[k] = (double)g.rc[k] - rhs;
  g.scale = (rhs > 0.0) ? 512.0 / rhs : 0.0;
}

// 30-bit Morton key of a position in the root cube; a non-finite one raises
// kStatusNonFinite.
__device__ __forceinline__ uint32_t morton_key(const TreeGeom& g, double x, double y, double z,
                                               int* status) {
  const double p[3] = {x, y, z};
  uint32_t c[3];
  bool finite = true;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double q = (p[k] - g.lo[k]) * g.scale;
    finite &= (q == q);
    q = fmin(fmax(q, 0.0), 1023.0);
    c[k] = (q == q) ? (uint32_t)q : 0u;
  }
  if (!finite) atomicOr(status, kStatusNonFinite);
  return morton30(c[0], c[1], c[2]);
}

// How far along an axis a body within `radius` in FP32 can be, with a margin
// for float positions an ulp off the FP64 ones the keys were made from.
__device__ __forceinline__ float cell_reach(float x, float radius) {
  return radius * 1.00001f + 1e-6f * (fabsf(x) + radius) + 1e-30f;
}

// Whether a search of `radius` goes by the finest cells: a ball then meets at
// most two along each axis.
__device__ __forceinline__ bool by_cells(const TreeGeom& g, float radius) {
  float most = 0.f;
#pragma unroll
  for (int k = 0; k < 3; ++k) most = fmaxf(most, fmaxf(fabsf(g.bmin[k]), fabsf(g.bmax[k])));
  const float side = g.rhs * (1.f / 512.f);
  return radius > 0.f && 2.f * cell_reach(most, radius) <= side;
}

}  // namespace nb
