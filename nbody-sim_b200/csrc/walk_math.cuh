// walk_math.cuh -- the per-interaction arithmetic of the force walk, shared
// by the tree walk and the tape replays so that a replayed interaction
// rounds exactly as the recorded one did.
#pragma once
#include <cuda_runtime.h>

namespace nb {

// 1/sqrt(x) by the hardware approximation (rsqrt.approx, ~2^-22 relative),
// with subnormal inputs and results flushed to zero: r^2 >= eps^2 or a
// squared distance between distinct bodies is never subnormal here, and the
// flush spares the range fix-up the non-flushing form needs.
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// acc += m_s (s - p) / (|s - p|^2 + eps^2)^{3/2}  (s.w = m_s; FP32, FMA form)
template <bool kSoft>
__device__ __forceinline__ void interact(const float4 s, const float4 p, float eps2,
                                         float3& acc) {
  float dx = s.x - p.x, dy = s.y - p.y, dz = s.z - p.z;
  float r2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, eps2)));
  float inv = rsqrt_ftz(r2);
  if (!kSoft) inv = (r2 > 0.f) ? inv : 0.f;
  float f = s.w * (inv * inv * inv);
  acc.x = fmaf(f, dx, acc.x);
  acc.y = fmaf(f, dy, acc.y);
  acc.z = fmaf(f, dz, acc.z);
}

// A target's accelerations as pairs: .x sums the even-indexed sources of a
// list, .y the odd-indexed ones, added together once the walk is done.
struct PairAcc {
  float2 x, y, z;
};

// A target's negated coordinates, each in both halves of a pair.
struct PairTgt {
  float2 x, y, z;
};

// interact() on two sources at once in packed FP32 (f32x2, sm_100): the same
// operations in the same order on each half, so each interaction rounds as
// interact() rounds it (s + (-p) is s - p exactly).  sx .. sm hold the two
// sources' coordinates and masses.  Returns the two softened r^2.
template <bool kSoft>
__device__ __forceinline__ float2 interact2(const float2 sx, const float2 sy, const float2 sz,
                                            const float2 sm, const PairTgt& p, const float2 e2,
                                            PairAcc& acc) {
  const float2 dx = __fadd2_rn(sx, p.x), dy = __fadd2_rn(sy, p.y), dz = __fadd2_rn(sz, p.z);
  const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, e2)));
  float2 inv = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
  if (!kSoft) {
    inv.x = (r2.x > 0.f) ? inv.x : 0.f;
    inv.y = (r2.y > 0.f) ? inv.y : 0.f;
  }
  const float2 f = __fmul2_rn(sm, __fmul2_rn(__fmul2_rn(inv, inv), inv));
  acc.x = __ffma2_rn(f, dx, acc.x);
  acc.y = __ffma2_rn(f, dy, acc.y);
  acc.z = __ffma2_rn(f, dz, acc.z);
  return r2;
}

// Vector-Jacobian product of one interaction: with d = s - p and
// K(d) = d / (|d|^2 + eps^2)^{3/2}, returns g = m_s (dK/dd) lam
//   = m_s (lam r^-3 - 3 d (d . lam) r^-5),   r^2 = |d|^2 + eps^2.
// The target's position adjoint receives -g, the source's +g.
template <bool kSoft>
__device__ __forceinline__ float3 interact_vjp(const float4 s, const float4 p, float eps2,
                                               const float3 lam) {
  float dx = s.x - p.x, dy = s.y - p.y, dz = s.z - p.z;
  float r2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, eps2)));
  float inv = rsqrt_ftz(r2);
  if (!kSoft) inv = (r2 > 0.f) ? inv : 0.f;
  const float inv2 = inv * inv;
  const float f = s.w * (inv2 * inv);
  const float dl = fmaf(dx, lam.x, fmaf(dy, lam.y, dz * lam.z));
  const float t = 3.f * dl * inv2;
  return make_float3(f * fmaf(-t, dx, lam.x), f * fmaf(-t, dy, lam.y), f * fmaf(-t, dz, lam.z));
}

// interact_vjp() on two sources (or two targets) at once in packed FP32,
// added into acc: acc += m_s (lam r^-3 - 3 d (d . lam) r^-5), pair half by
// pair half.  p holds the negated target coordinates, sx .. sm the sources'
// coordinates and masses (a mass of 0 drops its half), lx .. lz the
// adjoints.
template <bool kSoft>
__device__ __forceinline__ void interact_vjp2(const float2 sx, const float2 sy, const float2 sz,
                                              const float2 sm, const PairTgt& p, const float2 e2,
                                              const float2 lx, const float2 ly, const float2 lz,
                                              PairAcc& acc) {
  const float2 dx = __fadd2_rn(sx, p.x), dy = __fadd2_rn(sy, p.y), dz = __fadd2_rn(sz, p.z);
  const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, e2)));
  float2 inv = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
  if (!kSoft) {
    inv.x = (r2.x > 0.f) ? inv.x : 0.f;
    inv.y = (r2.y > 0.f) ? inv.y : 0.f;
  }
  const float2 inv2 = __fmul2_rn(inv, inv);
  const float2 f = __fmul2_rn(sm, __fmul2_rn(inv2, inv));
  const float2 dl = __ffma2_rn(dx, lx, __ffma2_rn(dy, ly, __fmul2_rn(dz, lz)));
  const float2 nt = __fmul2_rn(__fmul2_rn(make_float2(-3.f, -3.f), dl), inv2);
  acc.x = __ffma2_rn(f, __ffma2_rn(nt, dx, lx), acc.x);
  acc.y = __ffma2_rn(f, __ffma2_rn(nt, dy, ly), acc.y);
  acc.z = __ffma2_rn(f, __ffma2_rn(nt, dz, lz), acc.z);
}

// Source lists in shared memory: one row per component (x, y, z, mass), so
// that four consecutive sources of a row are one 16-byte broadcast holding two
// register pairs.
template <typename L>
__device__ __forceinline__ void lst_put(L& w, int j, const float4 s) {
  w.lsrc[0][j] = s.x;
  w.lsrc[1][j] = s.y;
  w.lsrc[2][j] = s.z;
  w.lsrc[3][j] = s.w;
}

template <typename L>
__device__ __forceinline__ float4 lst_get(const L& w, int j) {
  return make_float4(w.lsrc[0][j], w.lsrc[1][j], w.lsrc[2][j], w.lsrc[3][j]);
}

template <typename L>
__device__ __forceinline__ float4 lst_row4(const L& w, int c, int j) {
  return *reinterpret_cast<const float4*>(&w.lsrc[c][j]);
}

// Sources j .. j+3 (j a multiple of 4) against the lane's kT targets: two
// packed interactions per target, sources j, j+2 in the .x halves of the
// accumulators and j+1, j+3 in the .y halves.  kRmin: also the least
// softened r^2 seen.
template <bool kSoft, int kT, bool kRmin, typename L>
__device__ __forceinline__ void eval_quad(const L& w, int j, const PairTgt (&pt)[kT],
                                          const float2 e2, PairAcc (&acc)[kT], float& rmin) {
  const float4 qx = lst_row4(w, 0, j), qy = lst_row4(w, 1, j);
  const float4 qz = lst_row4(w, 2, j), qm = lst_row4(w, 3, j);
#pragma unroll
  for (int t = 0; t < kT; ++t) {
    const float2 r0 = interact2<kSoft>(make_float2(qx.x, qx.y), make_float2(qy.x, qy.y),
                                       make_float2(qz.x, qz.y), make_float2(qm.x, qm.y), pt[t],
                                       e2, acc[t]);
    const float2 r1 = interact2<kSoft>(make_float2(qx.z, qx.w), make_float2(qy.z, qy.w),
                                       make_float2(qz.z, qz.w), make_float2(qm.z, qm.w), pt[t],
                                       e2, acc[t]);
    if (kRmin) rmin = fminf(rmin, fminf(fminf(r0.x, r0.y), fminf(r1.x, r1.y)));
  }
}

// One source in scalar FP32 into the .x halves.
template <bool kSoft, int kT, bool kRmin>
__device__ __forceinline__ void eval_one(const float4 s, const float4 (&me)[kT], float eps2,
                                         PairAcc (&acc)[kT], float& rmin) {
#pragma unroll
  for (int t = 0; t < kT; ++t) {
    if (kRmin) {
      const float dx = s.x - me[t].x, dy = s.y - me[t].y, dz = s.z - me[t].z;
      rmin = fminf(rmin, fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, eps2))));
    }
    float3 a3 = make_float3(acc[t].x.x, acc[t].y.x, acc[t].z.x);
    interact<kSoft>(s, me[t], eps2, a3);
    acc[t].x.x = a3.x;
    acc[t].y.x = a3.y;
    acc[t].z.x = a3.z;
  }
}

// Sources j, j + 1 (j even) into the .x halves in list order: the products
// packed, two sources an instruction, the sums one source after the other, so
// that each rounds as eval_one() twice.
template <bool kSoft, int kT, typename L>
__device__ __forceinline__ void eval_pair_seq(const L& w, int j, const PairTgt (&pt)[kT],
                                              const float2 e2, PairAcc (&acc)[kT]) {
  const float2 sx = *reinterpret_cast<const float2*>(&w.lsrc[0][j]);
  const float2 sy = *reinterpret_cast<const float2*>(&w.lsrc[1][j]);
  const float2 sz = *reinterpret_cast<const float2*>(&w.lsrc[2][j]);
  const float2 sm = *reinterpret_cast<const float2*>(&w.lsrc[3][j]);
#pragma unroll
  for (int t = 0; t < kT; ++t) {
    const float2 dx = __fadd2_rn(sx, pt[t].x), dy = __fadd2_rn(sy, pt[t].y);
    const float2 dz = __fadd2_rn(sz, pt[t].z);
    const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, e2)));
    float2 inv = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
    if (!kSoft) {
      inv.x = (r2.x > 0.f) ? inv.x : 0.f;
      inv.y = (r2.y > 0.f) ? inv.y : 0.f;
    }
    const float2 f = __fmul2_rn(sm, __fmul2_rn(__fmul2_rn(inv, inv), inv));
    acc[t].x.x = fmaf(f.y, dx.y, fmaf(f.x, dx.x, acc[t].x.x));
    acc[t].y.x = fmaf(f.y, dy.y, fmaf(f.x, dy.x, acc[t].y.x));
    acc[t].z.x = fmaf(f.y, dz.y, fmaf(f.x, dz.x, acc[t].z.x));
  }
}

// All lanes evaluate sources 0 .. cnt of the list for their kT targets
// (kCount > 0: exactly kCount, a multiple of 4): each quad of sources is four
// shared-memory broadcasts feeding 2 kT packed interaction chains; a tail of
// fewer than four goes through eval_one.  kSeq (recording walks and their
// replay): every source added in list order, as eval_one adds it.  Returns
// the least softened r^2 when kRmin.
template <bool kSoft, int kT, int kCount, bool kRmin = false, bool kSeq = false, typename L>
__device__ __forceinline__ float eval_list(const L& w, int cnt, const float4 (&me)[kT],
                                           const PairTgt (&pt)[kT], float eps2, const float2 e2,
                                           PairAcc (&acc)[kT]) {
  static_assert(kCount % 4 == 0, "full batches are whole quads");
  float rmin = INFINITY;
  if (kSeq) {
    const int c = (kCount > 0) ? kCount : cnt;
    int j = 0;
#pragma unroll 4
    for (; j + 2 <= c; j += 2) eval_pair_seq<kSoft, kT>(w, j, pt, e2, acc);
    for (; j < c; ++j) eval_one<kSoft, kT, kRmin>(lst_get(w, j), me, eps2, acc, rmin);
  } else if (kCount > 0) {
#pragma unroll
    for (int j = 0; j < kCount; j += 4) eval_quad<kSoft, kT, kRmin>(w, j, pt, e2, acc, rmin);
  } else {
    int j = 0;
    for (; j + 4 <= cnt; j += 4) eval_quad<kSoft, kT, kRmin>(w, j, pt, e2, acc, rmin);
    for (; j < cnt; ++j) eval_one<kSoft, kT, kRmin>(lst_get(w, j), me, eps2, acc, rmin);
  }
  return rmin;
}

}  // namespace nb
