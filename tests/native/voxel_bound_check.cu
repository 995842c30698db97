// Host-side check of the error bounds that the two-float fast path states:
// over random segments and points, the largest |two-float value - value of the
// reference's double arithmetic| in units of dist_bound, and of the unit
// vector's components in units of unit_bound, with the estimate of 1 / |d| moved
// by a few units in the last place as the device's may be.  Prints both and
// fails above the given limit.  Runs on the CPU only.
//
//   nvcc -O2 -std=c++17 -fmad=false -Xcompiler -ffp-contract=off \
//        -I include tests/native/voxel_bound_check.cu -o check && ./check SEED LENGTH N LIMIT
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../fastpli_gb300/csrc/capi.cu"
#include "../../fastpli_gb300/csrc/tissue.cu"
#include "../../fastpli_gb300/csrc/voxel_bricks.cu"

using namespace fpgb;

int main(int argc, char **argv) {
   if (argc < 5)
      return 2;
   std::mt19937_64 rng(atoi(argv[1]));
   std::uniform_real_distribution<double> U(0.0, 1.0);
   const double length = atof(argv[2]), limit = atof(argv[4]);
   const long n = atol(argv[3]);
   const int64_t dim[3] = {300, 300, 300};
   double worst_d = 0, worst_u = 0;
   long used = 0, units = 0;
   for (long k = 0; k < n; k++) {
      double p[3], q[3], v[3], nv = 0;
      const int shape = (int)(U(rng) * 3); // any direction, near an axis, on one
      for (int i = 0; i < 3; i++) {
         v[i] = (U(rng) - 0.5) * (shape == 0 || i == (int)(k % 3) ? 1.0 : shape == 1 ? 1e-4 : 0.0);
         nv += v[i] * v[i];
      }
      const double scale = length * (0.2 + U(rng)) / std::sqrt(nv), t = U(rng);
      const double off = std::pow(10.0, -2 + 3.5 * U(rng));
      int x[3];
      for (int i = 0; i < 3; i++) {
         x[i] = (int)(U(rng) * 300);
         v[i] *= scale;
         p[i] = x[i] + 0.5 - t * v[i] + (U(rng) - 0.5) * off;
         q[i] = p[i] + v[i];
      }
      const double r0 = 1 + 5 * U(rng);
      SegDev S;
      fill_segment(p, q, r0, r0, 0, 1.f, 1.0, dim, S);
      if (!(S.pscale < 0x1p22f))
         continue;
      const float lpt[3] = {(float)(x[0] - S.base[0]) + 0.5f, (float)(x[1] - S.base[1]) + 0.5f,
                            (float)(x[2] - S.base[2]) + 0.5f};
      FastCand c;
      ff b;
      if (!fast_offset(S, lpt, c, b))
         continue;
      used++;
      // the reference's double |d|^2 and unit vector (generator.cpp:327, 370-371)
      const double pt[3] = {x[0] + 0.5, x[1] + 0.5, x[2] + 0.5};
      double cl[3], tt, l2 = 0.0, nvec[3], n2 = 0.0;
      closest_point(S, pt, cl, tt);
      for (int i = 0; i < 3; i++) {
         const double d = cl[i] - pt[i];
         l2 = l2 + d * d;
         nvec[i] = pt[i] - cl[i];
         n2 = n2 + nvec[i] * nvec[i];
      }
      const double err = std::fabs((double)((long double)c.D.hi + c.D.lo - (long double)l2));
      worst_d = std::max(worst_d, err / dist_bound(c, S.pscale));
      if (!(c.dn > 0x1p-10f))
         continue;
      units++;
      for (int ulps = -3; ulps <= 3; ulps += 3) {
         FastCand e = c;
         e.y0 = c.y0 * (1.f + ulps * 0x1p-23f);
         // fast_radial's arithmetic, before the rounding decision
         const ff sq = two_prod(e.y0, e.y0);
         const float res =
             fmaf(-e.D.lo, sq.hi, fmaf(-e.D.hi, sq.lo, fmaf(-e.D.hi, sq.hi, 1.f)));
         const ff inv = quick_two_sum(e.y0, e.y0 * fmaf(0.375f * res, res, 0.5f * res));
         const double in = 1.0 / std::sqrt(n2);
         for (int i = 0; i < 3; i++) {
            const ff pr = two_prod(-e.d[i].hi, inv.hi);
            const float lo = fmaf(-e.d[i].hi, inv.lo, fmaf(-e.d[i].lo, inv.hi, pr.lo));
            const ff z = quick_two_sum(pr.hi, lo);
            worst_u = std::max(worst_u, (double)std::fabs((long double)z.hi + z.lo -
                                                          (long double)(nvec[i] * in)) /
                                            unit_bound(e, S.pscale));
         }
      }
   }
   printf("candidates %ld dist %.4f units %ld unit %.4f\n", used, worst_d, units, worst_u);
   return !(used && worst_d <= limit && worst_u <= limit);
}
