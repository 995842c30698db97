// Host-side check of the voxelizer's sweep over every voxel of random segment
// boxes: the reference's dist^2 lies in [hi - 2 mg, hi] of the FP32 estimate
// (sweep_dist2, seg_margin) wherever that is not past the segment's thickest
// end, what is past it lies outside of the fiber, what is at or below acc_f
// inside; and the unit vector that fast_offset and fast_radial accept is the
// FP64 replay's.  Runs on the CPU only.
//
//   nvcc -O2 -std=c++17 -fmad=false -Xcompiler -ffp-contract=off \
//        -I include tests/native/voxel_sweep_check.cu -o check
//   ./check SEED VOXEL_SIZE LENGTH RADIUS FIBERS TAPER
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "../../fastpli_gb300/csrc/capi.cu"
#include "../../fastpli_gb300/csrc/tissue.cu"
#include "../../fastpli_gb300/csrc/voxel_bricks.cu"

using namespace fpgb;

int main(int argc, char **argv) {
   if (argc < 7)
      return 2;
   std::mt19937_64 rng(atoi(argv[1]));
   std::uniform_real_distribution<double> U(0.0, 1.0);
   const double vs = atof(argv[2]), len = atof(argv[3]), rad = atof(argv[4]);
   const int n_fibers = atoi(argv[5]);
   const bool taper = atoi(argv[6]) != 0;
   fpgb_volume vol{{96, 80, 64}, {0.37, -1.25, 0.5}, vs};
   std::vector<double> pts;
   std::vector<int64_t> foff{0};
   for (int f = 0; f < n_fibers; f++) {
      const double c[3] = {U(rng) * 96 * vs, U(rng) * 80 * vs, U(rng) * 64 * vs};
      double d[3], n = 0;
      for (double &x : d) {
         x = U(rng) - 0.5;
         n += x * x;
      }
      const double r = rad * (0.5 + U(rng));
      for (int k = -1; k < 2; k++) {
         const double at = k * len * (0.3 + U(rng)) / std::sqrt(n);
         for (int i = 0; i < 3; i++)
            pts.push_back(c[i] + d[i] * at);
         pts.push_back(taper ? r * (0.5 + U(rng)) : r);
      }
      foff.push_back(foff.back() + 3);
   }
   const int64_t boff[2] = {0, n_fibers}, loff[2] = {0, 1};
   const double sc[1] = {1.0}, dn[1] = {0.004}, mu[1] = {1};
   const char md[1] = {'r'};
   fpgb_fibers fb{1, boff, foff.data(), pts.data(), loff, sc, dn, mu, md};
   TissuePlan plan;
   if (plan_tissue(&vol, &fb, &plan) != FPGB_OK) {
      printf("plan failed: %s\n", fpgb_last_error());
      return 2;
   }
   const int brick[3] = {kBrickX, kBrickY, kBrickZ};
   long long n = 0, near = 0, bound_bad = 0, out_bad = 0, in_bad = 0, vec = 0, vec_bad = 0;
   for (const SegDev &S : plan.segs) {
      const float thr = fminf(fmaf(2.00001f, S.mg, S.thr_f), 3e38f);
      for (int64_t v = 0; v < (int64_t)S.ext[0] * S.ext[1] * S.ext[2]; v++) {
         const int64_t e[3] = {v / S.ext[2] / S.ext[1], v / S.ext[2] % S.ext[1], v % S.ext[2]};
         double pt[3], cl[3];
         float lpt[3], w[3], d, r;
         for (int i = 0; i < 3; i++) {
            const int64_t c = S.lo[i] + e[i];
            pt[i] = c + 0.5;
            lpt[i] = (float)(c - S.base[i]) + 0.5f;
            // the sub-box's first voxel, then steps of 4, 2 and 1 along x
            const int64_t x0 = std::max<int64_t>(S.lo[i], c / brick[i] * brick[i]);
            w[i] = ((float)(x0 - S.base[i]) + 0.5f) - S.pf[i];
            if (i == 0)
               for (int step = 4; step; step /= 2)
                  w[i] = (c - x0) & step ? w[i] + (float)step : w[i];
            else
               w[i] = w[i] + (float)(c - x0);
         }
         exact_dist(S, pt, cl, d, r);
         const float hi = sweep_dist2(
             w[0], fmaf(w[2], -2.f * S.vf[2], w[1] * (-2.f * S.vf[1])),
             fmaf(w[2], w[2], fmaf(w[1], w[1], S.mg)), -2.f * S.vf[0], S.c2f, -0.5f * S.c2_rcp);
         n++;
         if (!(hi > thr)) {
            near++;
            if (!((double)d <= hi && (double)d >= (double)hi - 2.0 * S.mg))
               bound_bad++;
         } else if (!(d > r)) {
            out_bad++;
         }
         if (hi <= S.acc_f && d > r)
            in_bad++;
         FastCand fc;
         ff t;
         float o[3];
         if (d <= r && S.pscale < 0x1p22f && fast_offset(S, lpt, fc, t) &&
             fast_radial(S, fc, o)) {
            vec++;
            double nv[3] = {pt[0] - cl[0], pt[1] - cl[1], pt[2] - cl[2]}, n2 = 0.0;
            for (double x : nv)
               n2 = n2 + x * x;
            const double inv = 1.0 / std::sqrt(n2);
            for (int i = 0; i < 3; i++)
               vec_bad += (float)(nv[i] * inv) != o[i];
         }
      }
   }
   printf("voxels %lld near %lld bound %lld outside %lld inside %lld vectors %lld wrong %lld\n", n,
          near, bound_bad, out_bad, in_bad, vec, vec_bad);
   return bound_bad || out_bad || in_bad || vec_bad || !near;
}
