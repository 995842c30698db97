// Two-float ("double-float") arithmetic: a value is hi + lo with
// |lo| <= ulp(hi)/2, about 48 significant bits from FP32 instructions.
// Built on Knuth's error-free TwoSum and the FMA-based TwoProduct; these
// are the textbook error-free transformations, written out here.  GB300 runs
// FP64 at a small fraction of its FP32 rate, so the voxelizer evaluates its
// double-precision geometry this way and only drops to FP64 when a result
// lies too close to a float rounding boundary to be decided.
#pragma once

#include <cuda_runtime.h>

#include <cmath>

#ifndef FPGB_HD
#define FPGB_HD __host__ __device__ __forceinline__
#endif

namespace fpgb {

struct ff {
   float hi, lo;
};

// exact: a + b = s + e (Knuth TwoSum)
FPGB_HD ff two_sum(float a, float b) {
   const float s = a + b;
   const float bb = s - a;
   const float e = (a - (s - bb)) + (b - bb);
   return ff{s, e};
}

// exact when |a| >= |b| (Dekker FastTwoSum)
FPGB_HD ff quick_two_sum(float a, float b) {
   const float s = a + b;
   const float e = b - (s - a);
   return ff{s, e};
}

// exact: a * b = p + e, using one fused multiply-add
FPGB_HD ff two_prod(float a, float b) {
   const float p = a * b;
   const float e = fmaf(a, b, -p);
   return ff{p, e};
}

FPGB_HD ff ff_add(ff a, ff b) {
   ff s = two_sum(a.hi, b.hi);
   const ff t = two_sum(a.lo, b.lo);
   s.lo += t.hi;
   s = quick_two_sum(s.hi, s.lo);
   s.lo += t.lo;
   return quick_two_sum(s.hi, s.lo);
}

FPGB_HD ff ff_mul(ff a, ff b) {
   ff p = two_prod(a.hi, b.hi);
   p.lo += a.hi * b.lo + a.lo * b.hi;
   return quick_two_sum(p.hi, p.lo);
}

FPGB_HD ff ff_sqr(ff a) {
   ff p = two_prod(a.hi, a.hi);
   p.lo += 2.f * a.hi * a.lo;
   return quick_two_sum(p.hi, p.lo);
}

// a . b of two-float vectors: the products' rounding errors and the cross
// terms go to one low word (a few units of 2^-48 of |a| |b|)
FPGB_HD ff ff_dot3(const ff a[3], const ff b[3]) {
   const ff p0 = two_prod(a[0].hi, b[0].hi), p1 = two_prod(a[1].hi, b[1].hi),
            p2 = two_prod(a[2].hi, b[2].hi);
   const ff s = two_sum(p0.hi, p1.hi), r = two_sum(s.hi, p2.hi);
   float lo = ((p0.lo + p1.lo) + p2.lo) + (s.lo + r.lo);
#pragma unroll
   for (int i = 0; i < 3; i++)
      lo = fmaf(a[i].hi, b[i].lo, fmaf(a[i].lo, b[i].hi, lo));
   return quick_two_sum(r.hi, lo);
}

// The float nearest to every real in [x - e, x + e], or false when the
// interval straddles a rounding boundary.  x is normalised, so that float is
// x.hi or there is none.  The low word is widened by e and by the rounding of
// that sum; a float sum that gives back hi for both ends gives it for every
// real between (round-to-nearest is monotone).
FPGB_HD bool ff_round_unique(ff x, float e, float &out) {
   const float w = fmaf(0x1p-22f, fabsf(x.lo), 1.000001f * e);
   out = x.hi;
   return x.hi + (x.lo - w) == x.hi && x.hi + (x.lo + w) == x.hi;
}

} // namespace fpgb
