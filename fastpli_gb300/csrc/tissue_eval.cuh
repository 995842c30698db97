// Exact (FP64) and two-float evaluation of one (segment, voxel) candidate of
// the voxelizer.  Host+device: the kernels use it, and a host build checks
// the two-float decisions against the FP64 replay.
#pragma once

#include <cmath>

#include "ff.cuh"
#include "tissue.cuh"

namespace fpgb {

// Closest point of `pt` on segment S and its parameter t, in the reference's
// double operation order (generator.cpp:475-494).  -fmad=false keeps every
// product and sum separately rounded.
FPGB_HD void closest_point(const SegDev &S, const double pt[3],
                                              double cl[3], double &t) {
   const double w0 = pt[0] - S.p[0], w1 = pt[1] - S.p[1], w2 = pt[2] - S.p[2];
   double c1 = 0.0;
   c1 = c1 + w0 * S.v[0];
   c1 = c1 + w1 * S.v[1];
   c1 = c1 + w2 * S.v[2];
   if (c1 < 0) {
      cl[0] = S.p[0];
      cl[1] = S.p[1];
      cl[2] = S.p[2];
      t = 0.0;
   } else if (S.c2 <= c1) {
      cl[0] = S.q[0];
      cl[1] = S.q[1];
      cl[2] = S.q[2];
      t = 1.0;
   } else {
      const double b = c1 / S.c2;
      cl[0] = S.p[0] + S.v[0] * b;
      cl[1] = S.p[1] + S.v[1] * b;
      cl[2] = S.p[2] + S.v[2] * b;
      t = b;
   }
}

// FP32 estimate of a candidate's dist^2 from segment-local inputs (w = voxel
// centre - float(p - base), float(v), float(c2), float(1 / c2)), and a bound:
// the float that the reference's double arithmetic produces (exact_dist)
// lies in [d2f - margin, d2f + margin].
//
// The estimate is |w - t v|^2 = w.w - 2 t (w.v) + t^2 (v.v) at t = clamp(w.v /
// v.v, 0, 1) — the closest-point parameter, so no branch: for t = 0 it is
// |w|^2, for t = 1 |w - v|^2, in between |w|^2 - (w.v)^2 / v.v.  An error in
// t only raises the value by v.v (dt)^2 (the expression is the squared
// distance to a point of the segment, minimal at the exact t).  This form,
// with a bound of the candidate's own, is what voxel_marks filters by; the sweep
// takes the same estimate with the segment's bound (sweep_dist2).
// The bound covers the rounding of the float inputs, of every FP32 operation
// (fused multiply-adds: one rounding each, the same on the host and the
// device) and of the reference's own final rounding; a host build checks it
// over every voxel of random segment boxes (tests/test_voxel_fastpath.py).
FPGB_HD float dist2_yz_dot(float wy, float wz, float vy, float vz) {
   return fmaf(wz, vz, wy * vy);
}
FPGB_HD float dist2_yz_len(float wy, float wz) { return fmaf(wz, wz, wy * wy); }

FPGB_HD float approx_dist2_x(float wx, float a, float b, float vx, float c2f, float rc2,
                             float &margin) {
   const float c1 = fmaf(wx, vx, a);
   const float w2 = fmaf(wx, wx, b);
   const float t = fminf(fmaxf(c1 * rc2, 0.f), 1.f);
   const float m = fmaf(t, c2f, -2.f * c1);
   margin = fmaf(3.8e-6f, w2 + c2f, 1e-4f);
   return fmaf(t, m, w2);
}

FPGB_HD float approx_dist2(float wx, float wy, float wz, float vx, float vy, float vz,
                           float c2f, float rc2, float &margin) {
   return approx_dist2_x(wx, dist2_yz_dot(wy, wz, vy, vz), dist2_yz_len(wy, wz), vx, c2f, rc2,
                         margin);
}

// The same estimate as the sweep takes it, with the segment's own bound
// S.mg (seg_margin) already in the sum: c1n2 = -2 (w.v)'s y and z parts and
// b = wy^2 + wz^2 + mg come once per cell, vn2 = -2 vx, rch = -1/2 float(1 / c2).
// The value is an upper bound hi of the reference's float, hi - 2 mg a lower
// bound (mg covers the rounding of the two differences as well).
FPGB_HD float sweep_dist2(float wx, float a2, float b, float vn2, float c2f, float rch) {
   const float c1n = fmaf(wx, vn2, a2); // -2 w.v
#ifdef __CUDA_ARCH__
   const float t = __saturatef(c1n * rch);
#else
   const float t = fminf(fmaxf(c1n * rch, 0.f), 1.f);
#endif
   return fmaf(t, fmaf(t, c2f, c1n), fmaf(wx, wx, b));
}

// Bound on |estimate - reference float| of the sweep's FP32 dist^2
// (sweep_dist2) over a box of voxels, from the offsets `first` of its first
// voxel from the segment's start and its last one `steps` further, over the
// voxels that lie within or next to the segment's thickest end (thr): |w| <=
// |v| + r' for the voxel's offset w from the start.  With u = 2^-24, the
// rounding of the inputs (w: u (|w0| + |w| + 1) for the offset w0 of the
// sub-box's first cell, v, c2: u each), of the operations and of the sum of the
// margin itself stays below u (15 |w|^2 + 2 |w| |w0| + 12 c2 + 4) (the
// error of t enters squared: the value is the squared distance to some point
// of the segment); the reference's own double arithmetic adds 2^-50 pscale |w|
// and its final rounding u |w|^2.  18 u and 12 u are 1.08e-6 and 7.2e-7.  For a
// voxel farther away, d >= |w| - |v|, so that error is below 3.3e-6 d^2 + 4e-6
// c2 and the estimate stays past the thickest end as the distance does: r' has
// more than that on top.  Evaluated in float, whose own rounding (below 1e-5)
// the factor 1.001 covers.
FPGB_HD float sweep_margin(const float first[3], const float steps[3], float c2f, float pscale,
                           float thr) {
   float w2 = 0.f;
   for (int i = 0; i < 3; i++) {
      const float a = first[i], b = a + steps[i];
      w2 += fmaxf(a * a, b * b);
   }
   const float box = sqrtf(w2), v = sqrtf(c2f), ps = 1e-14f * pscale;
   const float near = v + sqrtf(thr * 1.0001f + 0.01f + 1e-4f * c2f +
                                10.f * ps * (v + sqrtf(thr) + 1.f));
   const float w = fminf(box, near);
   return 1.001f * (1.08e-6f * w * w + 1.5e-7f * w * box + 7.2e-7f * c2f + 2e-6f +
                    ps * (w + 1.f));
}

// float(|cl - pt|^2) and float(r(t)^2) exactly as generator.cpp:327-328.
FPGB_HD void exact_dist(const SegDev &S, const double pt[3],
                                           double cl[3], float &dist_squ,
                                           float &r_sqr) {
   double t;
   closest_point(S, pt, cl, t);
   const double d0 = cl[0] - pt[0], d1 = cl[1] - pt[1], d2 = cl[2] - pt[2];
   double l2 = 0.0;
   l2 = l2 + d0 * d0;
   l2 = l2 + d1 * d1;
   l2 = l2 + d2 * d2;
   dist_squ = (float)l2;
   const double r = S.r0 * (1.0 - t) + S.r1 * t; // fiber.cpp:115-120
   r_sqr = (float)(r * r);
}

// ----------------------------------------------------------------------
// Two-float fast path.  For one (segment, voxel) pair it evaluates the
// reference's double arithmetic in two-float precision (~2^-46 relative)
// with an explicit bound E on |two-float value - value the reference's
// double arithmetic produces| (rounding of the reference itself included,
// generously).  A float result is accepted only when every real in
// [value - E, value + E] rounds to the same float; branch decisions only
// when the compared quantities differ by more than their bound.  Anything
// else returns false and the caller replays the reference in FP64, so the
// outcome is always the reference's, bit for bit.
// ----------------------------------------------------------------------
//
// The pairs are kept unnormalised where the next operation does not need
// them normalised: products contribute their rounding error (one fused
// multiply-add) to a single low word.  The bounds count roundings at their
// worst, in units of u^2 = 2^-48 of the terms' magnitudes; wm and vm are the
// 1-norms of point - p and of v, b the parameter, d the offset, m = wm + vm b + 1.
//   ff_dot3    the low word holds three product and two sum errors and the cross
//              terms, five u |a| |b| in all (|a| |b| the sum of the products'
//              sizes): 32 for its ten roundings, 11 for the terms left out and
//              for a sum that cancels (none in |d|^2)
//   w . v      45 |w| |v| with the rounding of the inputs, and 5 vm from the low
//              part of p - base, which is not relative to |w|: branch_bound
//              has 64 and 8
//   b          that over v.v, and 25 b of the quotient
//   d          14 |v| b + 4 |w| + 4 across the segment (the products, three sums
//              and the inputs' low parts); along it |v| times b's error; 49 m
//              with both
//   |d|^2      an error of d along the segment counts squared only: 2 * 14 m |d| +
//              32 |d|^2 <= 60 m |d|
//   unit       49 m / |d| of d, and 37: half of |d|^2's 32, 16 of the Newton step
//              and its product, 5 of the components' products
// and the reference's double arithmetic, 2^-50.5 pscale in d, 2^-48.5 pscale |d|
// in |d|^2.
struct FastCand {
   float dist_squ, r_sqr;
   ff d[3];  // closest - point
   ff D;     // |d|^2
   float y0; // ~ 1 / |d| (0 for d = 0)
   float dn; // ~ |d|
   float m;  // magnitude scale of the terms that make up d (>= their 2-norm)
};

// 1 / sqrt(x) within a few units of 2^-23
FPGB_HD float rsqrt_est(float x) {
#ifdef __CUDA_ARCH__
   return rsqrtf(x);
#else
   return 1.0f / sqrtf(x);
#endif
}

FPGB_HD float branch_bound(float wm, float vm) {
   return 0x1p-42f * ((wm + 0.125f) * vm + 1.f); // 64, 8
}
FPGB_HD float dist_bound(const FastCand &c, float pscale) {
   return 0x1.ep-43f * c.m * (c.dn + 0x1p-20f * c.m) + // 60
          0x1.8p-50f * pscale * (2.f * c.dn + 1.f);
}
FPGB_HD float unit_bound(const FastCand &c, float pscale) {
   return (0x1.ap-43f * c.m + 0x1.2p-50f * pscale) * (1.001f * c.y0) + 0x1.4p-43f; // 52, 40
}

// closest - point of the candidate (generator.cpp:475-494) with its squared
// length, and r^2 where it needs no rounding decision (rsq0, rsq1, rsq_const;
// NaN: interior of a segment whose radius changes, b holds the parameter).
// False when the clamp of the closest-point parameter is undecided.
FPGB_HD bool fast_offset(const SegDev &S, const float pt[3], FastCand &c, ff &b) {
   ff w[3], v[3];
   float wm = 0.f, vm = 0.f; // 1-norms: bounds of the 2-norms
#pragma unroll
   for (int i = 0; i < 3; i++) { // point - p; pt is exact
      const ff s = two_sum(pt[i], -S.pf[i]);
      w[i] = ff{s.hi, s.lo - S.pl_lo[i]};
      v[i] = ff{S.vf[i], S.v_lo[i]};
      wm += fabsf(s.hi);
      vm += fabsf(S.vf[i]);
   }
   const ff c1 = ff_dot3(w, v);
   const float ec = branch_bound(wm, vm);
   const float dq = (c1.hi - S.c2f) + (c1.lo - S.c2_lo);
   b = ff{0.f, 0.f};
   if (c1.hi < -ec) { // c1 < 0: closest = s0, t = 0 (generator.cpp:483-484)
      c.r_sqr = S.rsq0;
   } else if (dq > ec) { // c2 <= c1: closest = s1, t = 1 (:487-488)
      b.hi = 1.f;
      c.r_sqr = S.rsq1;
   } else if (c1.hi > ec && dq < -ec) { // interior: b = c1 / c2 (:490-493)
      // one residual correction of the FP32 quotient: c1.hi - q c2 is exact
      const float q = c1.hi * S.c2_rcp;
      const ff p = two_prod(S.c2f, q);
      const float e = ((c1.hi - p.hi) - p.lo) + fmaf(-S.c2_lo, q, c1.lo);
      b = quick_two_sum(q, e * S.c2_rcp);
      c.r_sqr = S.rsq_const;
   } else {
      return false;
   }
#pragma unroll
   for (int i = 0; i < 3; i++) { // v b - w
      const ff p = two_prod(v[i].hi, b.hi);
      const ff s = two_sum(p.hi, -w[i].hi);
      const float lo = fmaf(v[i].hi, b.lo, fmaf(v[i].lo, b.hi, p.lo));
      c.d[i] = quick_two_sum(s.hi, (lo - w[i].lo) + s.lo);
   }
   c.D = ff_dot3(c.d, c.d);
   c.y0 = c.D.hi > 0.f ? rsqrt_est(c.D.hi) : 0.f;
   c.dn = c.D.hi * c.y0;
   c.m = wm + vm * b.hi + 1.f;
   return true;
}

FPGB_HD bool fast_candidate(const SegDev &S, const float pt[3], FastCand &c) {
   ff b;
   if (!fast_offset(S, pt, c, b))
      return false;
   if (!(c.r_sqr == c.r_sqr)) { // r = r0 (1 - t) + r1 t  (fiber.cpp:115-120)
      const ff R = ff_add(ff{S.r0_hi, S.r0_lo}, ff_mul(ff{S.dr_hi, S.dr_lo}, b));
      const ff R2 = ff_sqr(R);
      // b's error, at most 25 u^2 b + (45 |w| |v| + 5 vm) u^2 / c2, is below a
      // quarter of 2^-40 eb
      const float eb = c.m * c.m * S.c2_rcp + b.hi + 1.f;
      const float er = 0x1p-40f * (R2.hi + fabsf(R.hi) * fabsf(S.dr_hi) * eb);
      if (!ff_round_unique(R2, er, c.r_sqr))
         return false;
   }
   return ff_round_unique(c.D, dist_bound(c, S.pscale), c.dist_squ);
}

// float(unit(point - closest)) of the 'r' layer (generator.cpp:370-371)
FPGB_HD bool fast_radial(const SegDev &S, const FastCand &c, float out[3]) {
   if (!(c.dn > 0x1p-10f))
      return false;
   // 1 / |d| = y0 (1 + e/2 + 3 e^2/8 + ...), e = 1 - D y0^2 (|e| < 2^-20)
   const ff t = two_prod(c.y0, c.y0);
   const float e = fmaf(-c.D.lo, t.hi, fmaf(-c.D.hi, t.lo, fmaf(-c.D.hi, t.hi, 1.f)));
   const ff inv = quick_two_sum(c.y0, c.y0 * fmaf(0.375f * e, e, 0.5f * e));
   const float ex = unit_bound(c, S.pscale);
#pragma unroll
   for (int i = 0; i < 3; i++) { // nv = -d
      const ff p = two_prod(-c.d[i].hi, inv.hi);
      const float lo = fmaf(-c.d[i].hi, inv.lo, fmaf(-c.d[i].lo, inv.hi, p.lo));
      if (!ff_round_unique(quick_two_sum(p.hi, lo), ex, out[i]))
         return false;
   }
   return true;
}

} // namespace fpgb
