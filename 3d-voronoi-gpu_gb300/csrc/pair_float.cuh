// Pairs of floats (h + l, 48 bits) for the robust-predicate option: vertices, and
// the signs that most near-zero tests need.  GB300 issues 64 FP32 operations for
// one in FP64.  On the device through the round-to-nearest intrinsics; host
// builds use -ffp-contract=off.
#pragma once

#include <cuda_runtime.h>

#include <cmath>

#include "exact_pred.cuh"

namespace vgb {

#ifdef __CUDA_ARCH__
#define VGB_FADD(a, b) __fadd_rn((a), (b))
#define VGB_FSUB(a, b) __fsub_rn((a), (b))
#define VGB_FMUL(a, b) __fmul_rn((a), (b))
#define VGB_FMA(a, b, c) __fmaf_rn((a), (b), (c))
#define VGB_FRCP(a) __frcp_rn(a)
#else
#define VGB_FADD(a, b) ((a) + (b))
#define VGB_FSUB(a, b) ((a) - (b))
#define VGB_FMUL(a, b) ((a) * (b))
#define VGB_FMA(a, b, c) std::fmaf((a), (b), (c))
#define VGB_FRCP(a) (1.f / (a))
#endif

// Products split by fma, sums by Knuth's
// TwoSum, every operation rounded on its own.
struct Pair {
  float h, l;
};
VGB_XHD inline Pair pair_fast(float h, float l) {  // |h| >= |l|
  const float s = VGB_FADD(h, l);
  return {s, VGB_FSUB(l, VGB_FSUB(s, h))};
}
VGB_XHD inline Pair pair_sum(float a, float b) {
  const float s = VGB_FADD(a, b), bv = VGB_FSUB(s, a);
  return {s, VGB_FADD(VGB_FSUB(a, VGB_FSUB(s, bv)), VGB_FSUB(b, bv))};
}
VGB_XHD inline Pair pair_add(Pair a, Pair b) {
  const Pair s = pair_sum(a.h, b.h);
  return pair_fast(s.h, VGB_FADD(s.l, VGB_FADD(a.l, b.l)));
}
VGB_XHD inline Pair pair_cross(float p, float q, float r, float t) {  // p q - r t
  const float a = VGB_FMUL(p, q), b = VGB_FMUL(r, t);
  const float ea = VGB_FMA(p, q, -a), eb = VGB_FMA(r, t, -b);
  const Pair s = pair_sum(a, -b);
  return pair_fast(s.h, VGB_FADD(s.l, VGB_FSUB(ea, eb)));
}
VGB_XHD inline Pair pair_mul(float a, Pair b) {
  const float p = VGB_FMUL(a, b.h);
  return pair_fast(p, VGB_FMA(a, b.l, VGB_FMA(a, b.h, -p)));
}
VGB_XHD inline Pair pair_dot(float a0, float a1, float a2, Pair b0, Pair b1, Pair b2) {
  return pair_add(pair_add(pair_mul(a0, b0), pair_mul(a1, b1)), pair_mul(a2, b2));
}
// -n / d, with r near 1 / d.h
VGB_XHD inline float pair_ratio(Pair n, Pair d, float r) {
  const float q = VGB_FMUL(n.h, r), p = VGB_FMUL(q, d.h);
  const float e = VGB_FMA(q, d.h, -p);
  const float rest = VGB_FADD(VGB_FSUB(VGB_FSUB(n.h, p), e), VGB_FMA(-q, d.l, n.l));
  return -VGB_FMA(rest, r, q);
}

// Sign of P at the vertex of A, B, C where pairs of floats tell it: with
// V = -num / det (Cramer), the sign of det (P.w det - P.n num), each factor's
// error below 2^-44 of the sum T of its terms' magnitudes; 0 when either is
// within 2^-40 of T.  (Sites from a lattice are cospherical up to the rounding
// of their positions, 2^-24: all but the exactly degenerate tests end here,
// for 450 FP32 operations instead of some thousands in FP64.)
VGB_XHD inline int pair_side(float4 a, float4 b, float4 c, float4 P) {
  const Pair bcx = pair_cross(b.y, c.z, b.z, c.y), bcy = pair_cross(b.z, c.x, b.x, c.z),
             bcz = pair_cross(b.x, c.y, b.y, c.x);
  const Pair cax = pair_cross(c.y, a.z, c.z, a.y), cay = pair_cross(c.z, a.x, c.x, a.z),
             caz = pair_cross(c.x, a.y, c.y, a.x);
  const Pair abx = pair_cross(a.y, b.z, a.z, b.y), aby = pair_cross(a.z, b.x, a.x, b.z),
             abz = pair_cross(a.x, b.y, a.y, b.x);
  auto m = [](float p, float q, float r, float t) { return fabsf(p * q) + fabsf(r * t); };
  const float mbx = m(b.y, c.z, b.z, c.y), mby = m(b.z, c.x, b.x, c.z), mbz = m(b.x, c.y, b.y, c.x);
  const float mcx = m(c.y, a.z, c.z, a.y), mcy = m(c.z, a.x, c.x, a.z), mcz = m(c.x, a.y, c.y, a.x);
  const float max_ = m(a.y, b.z, a.z, b.y), may = m(a.z, b.x, a.x, b.z), maz = m(a.x, b.y, a.y, b.x);
  const Pair det = pair_dot(a.x, a.y, a.z, bcx, bcy, bcz);
  const float md = fabsf(a.x) * mbx + fabsf(a.y) * mby + fabsf(a.z) * mbz;
  const Pair nx = pair_dot(a.w, b.w, c.w, bcx, cax, abx), ny = pair_dot(a.w, b.w, c.w, bcy, cay, aby),
             nz = pair_dot(a.w, b.w, c.w, bcz, caz, abz);
  const float aw = fabsf(a.w), bw = fabsf(b.w), cw = fabsf(c.w);
  const Pair pn = pair_dot(P.x, P.y, P.z, nx, ny, nz), pd = pair_mul(P.w, det);
  const Pair D = pair_add(pd, Pair{-pn.h, -pn.l});
  const float T = fabsf(P.w) * md + fabsf(P.x) * (aw * mbx + bw * mcx + cw * max_) +
                  fabsf(P.y) * (aw * mby + bw * mcy + cw * may) + fabsf(P.z) * (aw * mbz + bw * mcz + cw * maz);
  constexpr float eps = 1.f / (1048576.f * 1048576.f);  // 2^-40
  // (1e-20: the low parts must stay clear of underflow)
  if (!(fabsf(D.h) > eps * T && fabsf(det.h) > eps * md && fabsf(D.h) > 1e-20f && fabsf(det.h) > 1e-20f && T < 1e35f))
    return 0;
  return (D.h > 0.f) == (det.h > 0.f) ? 1 : -1;
}

// The vertex of three planes, if pairs of floats give it as double would: false
// where a coordinate needs more.  With V = -num / det (Cramer), each numerator
// and the determinant are good to about 2^-46 of the sum of their terms'
// magnitudes.  Where the determinant is more than 2^-13 of that sum and each
// numerator more than 2^-17, a coordinate is off by less than 2^-29 of itself
// (whatever its size against the others) before it is rounded to float.  About
// 400 FP32 operations instead of 65 in FP64.
VGB_XHD inline bool pair_vertex(float4 a, float4 b, float4 c, float3& x) {
  // (bounds on the sums of terms: each factor by its plane's sum)
  const float la = fabsf(a.x) + fabsf(a.y) + fabsf(a.z), lb = fabsf(b.x) + fabsf(b.y) + fabsf(b.z);
  const float lc = fabsf(c.x) + fabsf(c.y) + fabsf(c.z);
  const float least_det = la * lb * lc * (1.f / 8192.f);
  const float least = fmaxf((fabsf(a.w) * (lb * lc) + fabsf(b.w) * (lc * la) + fabsf(c.w) * (la * lb)) *
                            (1.f / 131072.f), 1e-20f);
  const Pair bcx = pair_cross(b.y, c.z, b.z, c.y), bcy = pair_cross(b.z, c.x, b.x, c.z),
             bcz = pair_cross(b.x, c.y, b.y, c.x);
  const Pair det = pair_dot(a.x, a.y, a.z, bcx, bcy, bcz);
  const float ad = fabsf(det.h);
  if (!(ad > least_det && ad > 1e-22f && ad < 1e30f)) return false;
  const float r = VGB_FRCP(det.h);
  const Pair nx = pair_dot(a.w, b.w, c.w, bcx, pair_cross(c.y, a.z, c.z, a.y), pair_cross(a.y, b.z, a.z, b.y));
  x.x = pair_ratio(nx, det, r);
  const Pair ny = pair_dot(a.w, b.w, c.w, bcy, pair_cross(c.z, a.x, c.x, a.z), pair_cross(a.z, b.x, a.x, b.z));
  x.y = pair_ratio(ny, det, r);
  const Pair nz = pair_dot(a.w, b.w, c.w, bcz, pair_cross(c.x, a.y, c.y, a.x), pair_cross(a.x, b.y, a.y, b.x));
  x.z = pair_ratio(nz, det, r);
  return fminf(fminf(fabsf(nx.h), fabsf(ny.h)), fabsf(nz.h)) > least;
}

}  // namespace vgb
