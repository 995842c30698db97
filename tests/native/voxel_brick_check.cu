// Host-side replay of the voxelizer's bricks: binning, sweep records, keys and
// marks in list order, and the decode's decision, with the functions the
// kernel uses.  Every voxel that the replay leaves unmarked must have the
// segment and layer that the FP64 replay of all candidates gives it.  Prints
// how many voxels are marked, and how many bricks have more than fit a record.
// Runs on the CPU only.
//
//   nvcc -O2 -std=c++17 -fmad=false -Xcompiler -ffp-contract=off \
//        -I include tests/native/voxel_brick_check.cu -o check
//   ./check SEED X Y Z RADIUS FIBERS POINTS TAPER LENGTH
// (LENGTH 0: fibers through the volume along its longest side)
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "../../fastpli_gb300/csrc/capi.cu"
#include "../../fastpli_gb300/csrc/tissue.cu"
#include "../../fastpli_gb300/csrc/voxel_bricks.cu"

using namespace fpgb;

static SegSweep host_sweep(const SegDev &S) {
   SegSweep w;
   std::memcpy(&w, &S.pf[0], 80);
   w.mg = S.mg;
   return w;
}

int main(int argc, char **argv) {
   if (argc < 10)
      return 2;
   std::mt19937_64 rng(atoi(argv[1]));
   std::uniform_real_distribution<double> U(0.0, 1.0);
   const int64_t X = atoi(argv[2]), Y = atoi(argv[3]), Z = atoi(argv[4]);
   const double rad = atof(argv[5]);
   const int n_fibers = atoi(argv[6]), n_points = atoi(argv[7]);
   const double taper = atof(argv[8]), length = atof(argv[9]);
   const double size[3] = {(double)X, (double)Y, (double)Z};
   const int ax = (int)(std::max_element(size, size + 3) - size);
   fpgb_volume vol{{X, Y, Z}, {0, 0, 0}, 1.0};
   std::vector<double> pts;
   std::vector<int64_t> foff{0};
   for (int f = 0; f < n_fibers; f++) {
      double a[3], b[3];
      for (int i = 0; i < 3; i++) {
         a[i] = U(rng) * size[i];
         b[i] = U(rng) * size[i];
      }
      a[ax] = -5;
      b[ax] = size[ax] + 5;
      if (length > 0) { // through the middle of the two, as long as asked
         double n = 0;
         for (int i = 0; i < 3; i++)
            n += (b[i] - a[i]) * (b[i] - a[i]);
         n = std::sqrt(n);
         const double e = U(rng);
         for (int i = 0; i < 3; i++) {
            const double m = 0.5 * (a[i] + b[i]), d = (b[i] - a[i]) / n;
            a[i] = m - e * length * d;
            b[i] = m + (1 - e) * length * d;
         }
      }
      for (int k = 0; k < n_points; k++) {
         const double t = (double)k / (n_points - 1);
         for (int i = 0; i < 3; i++)
            pts.push_back(a[i] + t * (b[i] - a[i]));
         pts.push_back(rad * (1 + taper * (2 * U(rng) - 1)));
      }
      foff.push_back(foff.back() + n_points);
   }
   const int64_t boff[2] = {0, n_fibers}, loff[2] = {0, 2};
   const double sc[2] = {0.75, 1.0}, dn[2] = {-0.004, 0.004}, mu[2] = {10, 1};
   const char md[2] = {'p', 'r'};
   fpgb_fibers fb{1, boff, foff.data(), pts.data(), loff, sc, dn, mu, md};
   TissuePlan plan;
   if (plan_tissue(&vol, &fb, &plan) != FPGB_OK) {
      printf("plan failed: %s\n", fpgb_last_error());
      return 2;
   }
   int32_t nb[3];
   int64_t n_bricks;
   tile_bricks(X, Y, Z, nb, &n_bricks);
   std::vector<std::vector<unsigned>> lists(n_bricks);
   for (size_t s = 0; s < plan.segs.size(); s++) {
      const SegDev &S = plan.segs[s];
      int b0[3], n[3];
      const int kb[3] = {kBrickX, kBrickY, kBrickZ};
      for (int i = 0; i < 3; i++)
         n[i] = (int)brick_range(S.lo[i], S.ext[i], kb[i], b0[i]);
      for (int i = 0; i < n[0]; i++)
         for (int j = 0; j < n[1]; j++)
            for (int k = 0; k < n[2]; k++)
               lists[((int64_t)(b0[0] + i) * nb[1] + b0[1] + j) * nb[2] + b0[2] + k].push_back(
                   (unsigned)s);
   }
   const LayerDev &L = plan.layers[0];
   long long marked = 0, inside = 0, wrong = 0, over = 0, busy = 0;
#pragma omp parallel for schedule(dynamic, 8) reduction(+ : marked, inside, wrong, over, busy)
   for (int64_t brick = 0; brick < n_bricks; brick++) {
      const auto &list = lists[brick];
      if (list.empty())
         continue;
      busy++;
      const int ox = (int)(brick / nb[2] / nb[1]) * kBrickX, oy = (int)(brick / nb[2] % nb[1]) * kBrickY,
                oz = (int)(brick % nb[2]) * kBrickZ;
      const int nx = (int)std::min<int64_t>(kBrickX, X - ox), ny = (int)std::min<int64_t>(kBrickY, Y - oy),
                nz = (int)std::min<int64_t>(kBrickZ, Z - oz);
      std::vector<SweepRec> rec;
      float th = 0.f, mg = 0.f;
      for (unsigned s : list) {
         const SegDev &S = plan.segs[s];
         SegSweep w = host_sweep(S);
         SubBox b;
         if (!sub_box(w, ox, oy, oz, nx, ny, nz, b))
            std::abort(); // the list has it for this brick
         const SegPart g = seg_part<true>(S, w, b);
         rec.push_back(sweep_rec<true>(g, S.thr_f, b, true, ox, oy, oz));
         th = std::max(th, fmaf(2.0001f, g.mg, S.thr_f));
         mg = std::max(mg, g.mg);
      }
      const BrickScale k = brick_scale((unsigned)list.size(), th, mg);
      std::vector<unsigned> keys(kBrickVoxels, kNoKey);
      for (unsigned j = 0; j < list.size(); j++) {
         const SweepRec &g = rec[j];
         const int ncell = (int)(g.box & 511u), ex = (int)(g.box >> 15 & 15u), x0 = (int)(g.box >> 27);
         for (int c = 0; c < ncell; c++) {
            const Cell cell = cell_of(g, (float)(g.box >> 9 & 63u), (float)c);
            float wx = g.wx0;
            int left = ex;
            for (int i = 0; i < ex;) { // steps of 4, 2 and 1
               const int step = left >= 4 ? 4 : left >= 2 ? 2 : 1;
               for (int u = 0; u < step; u++) {
                  const float hi = sweep_dist2(u ? wx + (float)u : wx, cell.a2, cell.b, g.vn2x,
                                               g.c2f, g.rch);
                  const unsigned mine =
                      (unsigned)float_bits(fmaf(hi, k.scale, 8388608.f)) * k.mul + 2u * j;
                  unsigned &key = keys[(x0 + i + u) * kPlane + cell.yz];
                  if (hi > g.thr)
                     continue;
                  const unsigned old = key;
                  key = std::min(key, mine);
                  if (old - mine + k.win <= k.win2)
                     key |= 1u;
               }
               wx += (float)step;
               i += step;
               left -= step;
            }
         }
      }
      long long here = 0;
      for (int lx = 0; lx < nx; lx++)
         for (int ly = 0; ly < ny; ly++)
            for (int lz = 0; lz < nz; lz++) {
               const int x = ox + lx, y = oy + ly, z = oz + lz;
               const double pt[3] = {x + 0.5, y + 0.5, z + 0.5};
               unsigned best = ~0u;
               float bd = INFINITY, br = 0;
               for (unsigned s : list) { // ascending: ties go to the last
                  const SegDev &S = plan.segs[s];
                  const int v[3] = {x, y, z};
                  bool in = true;
                  for (int i = 0; i < 3; i++)
                     in = in && v[i] >= S.lo[i] && v[i] < S.lo[i] + S.ext[i];
                  if (!in)
                     continue;
                  double cl[3];
                  float d, r;
                  exact_dist(S, pt, cl, d, r);
                  if (d > L.f_ly_squ * r || !(bd >= d))
                     continue;
                  bd = d;
                  br = r;
                  best = s;
               }
               int layer = -1;
               if (best != ~0u) {
                  inside++;
                  layer = 0;
                  while (layer < L.n && bd / br > L.sq_fdown[layer])
                     layer++;
               }
               const unsigned key = keys[lx * kPlane + plane_place(ly, lz)];
               if (key == kNoKey) {
                  wrong += best != ~0u;
                  continue;
               }
               int w = -1;
               const unsigned seg = list[(key & (k.mul - 1u)) >> 1];
               if (!(key & 1u)) {
                  const SegDev &S = plan.segs[seg];
                  float rsq = S.dec_rsq;
                  const float up = key_bound(k, key);
                  float lo = up * (1.f - 4e-6f) - 2.f * k.quantum - k.mg2, hi = up;
                  if (!(rsq == rsq)) {
                     double cl[3];
                     exact_dist(S, pt, cl, lo, rsq);
                     hi = lo > L.f_ly_squ * rsq ? INFINITY : lo;
                  }
                  w = certain_layer(L.sq_fdown, L.n, lo, hi, rsq);
               }
               if (w < 0)
                  here++;
               else
                  wrong += seg != best || w != layer;
            }
      marked += here;
      over += here > (long long)kMarkList;
   }
   printf("segments %zu inside %lld wrong %lld marked %lld (%.5f) bricks %lld over %lld\n",
          plan.segs.size(), inside, wrong, marked, inside ? (double)marked / inside : 0.0, busy,
          over);
   return wrong != 0;
}
