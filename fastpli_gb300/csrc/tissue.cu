// Voxelizer: fiber polylines -> int32 label field + float32 orientation field.
//
// Replaces PliGenerator::RunTissueGeneration / FillVoxelsAroundFiberSegment
// (src/simulation/generator.cpp:163-383, 475-526).  The reference walks every
// segment in order and overwrites a voxel when `dist[ind] >= dist_squ`
// (generator.cpp:343), so the final owner of a voxel is the segment with the
// smallest float distance and, among equal distances, the LAST one in
// processing order.  Here every (segment, voxel) candidate is independent:
//
//   binning       every segment's clipped bounding box is binned to the
//                 8 x 8 x 32 voxel bricks it overlaps;
//   voxel_bricks  one CTA per brick sweeps the brick's candidates once with
//                 FP32 bounds of dist_squ that almost always name a voxel's
//                 winner; the voxels where two candidates are too close are
//                 marked and decided with the exact double->float distance
//                 of the reference; then every voxel's label and orientation
//                 are written (voxel_bricks.cu).
//
// This translation unit is compiled with -fmad=false: the label and vector
// decisions depend on separately rounded double products and sums
// (generator.cpp:324-349, vemath.hpp:342-344,390-402), which a fused
// multiply-add would change.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "ff.cuh"
#include "fpgb_common.cuh"
#include "tissue.cuh"
#include "tissue_eval.cuh"
#include "voxel_bricks.cuh"

namespace fpgb {

// ======================================================================
// the segment table (double precision, reference operation order)
// ======================================================================
// double -> (hi, lo) float pair; |d - hi - lo| <= 2^-48 |d|
FPGB_HD void split2(double d, float &hi, float &lo) {
   hi = (float)d;
   lo = (float)(d - (double)hi);
}

// The segment's own bound (sweep_margin) over its whole box.
FPGB_HD float seg_margin(const SegDev &S, float thr) {
   float first[3], steps[3];
   for (int i = 0; i < 3; i++) {
      first[i] = (float)((double)S.lo[i] + 0.5 - S.p[i]);
      steps[i] = (float)(S.ext[i] > 0 ? S.ext[i] - 1 : 0);
   }
   return sweep_margin(first, steps, S.c2f, S.pscale, thr);
}

// Host-side constants of the two-float path, all derived in double exactly
// as the reference derives the corresponding values.
FPGB_HD void fill_fast_fields(SegDev &S, const int64_t dim[3]) {
   double ps = 0;
   for (int i = 0; i < 3; i++) {
      split2(S.p[i] - (double)S.base[i], S.pf[i], S.pl_lo[i]);
      split2(S.v[i], S.vf[i], S.v_lo[i]);
      ps = fmax(ps, fmax(fabs(S.p[i]), fabs(S.q[i])));
      ps = fmax(ps, (double)dim[i]);
   }
   S.pscale = (float)(ps + 2.0);
   split2(S.c2, S.c2f, S.c2_lo);
   S.c2_rcp = S.c2 > 0 ? (float)(1.0 / S.c2) : 0.f;
   split2(S.r0, S.r0_hi, S.r0_lo);
   split2(S.r1 - S.r0, S.dr_hi, S.dr_lo);
   // Fiber::CalcRadius at t = 0 and t = 1 is exactly r0 and r1
   // (fiber.cpp:115-120): r0*(1-0) + r1*0 = r0, r0*0 + r1*1 = r1
   S.rsq0 = (float)(S.r0 * S.r0);
   S.rsq1 = (float)(S.r1 * S.r1);
   // r0 == r1: every interior r(t) is r0 within a few ulp, so float(r^2) is
   // fixed unless r0^2 sits next to a float rounding boundary
   S.rsq_const = NAN;
   if (S.r0 == S.r1) {
      const double r2 = S.r0 * S.r0;
      const double eps = 64.0 * 0x1p-53;
      const float a = (float)(r2 * (1.0 - eps)), b = (float)(r2 * (1.0 + eps));
      if (a == b)
         S.rsq_const = a;
   }
   S.dec_rsq = S.rsq_const == S.rsq0 && S.rsq_const == S.rsq1 ? S.rsq_const : NAN;
   // 'p' layer vector: vm::unit(q - p) (generator.cpp:372-373, vemath.hpp:390-402)
   double n2 = 0.0;
   n2 = n2 + S.v[0] * S.v[0];
   n2 = n2 + S.v[1] * S.v[1];
   n2 = n2 + S.v[2] * S.v[2];
   double u[3] = {S.v[0], S.v[1], S.v[2]};
   if (n2 > 0) {
      const double inv = 1.0 / sqrt(n2);
      for (int i = 0; i < 3; i++)
         u[i] = u[i] * inv;
   }
   for (int i = 0; i < 3; i++)
      S.vp[i] = (float)u[i];
}

// The segment's box clipped to the volume (generator.cpp:295-312): its voxel
// count, 0 when it is empty.
FPGB_HD int64_t segment_box(const double *P, const double *Q, double r0, double r1, double rsl,
                            const int64_t dim[3], int32_t lo_out[3], int32_t ext_out[3]) {
   const double rmax = (r0 < r1 ? r1 : r0) * rsl;
   int64_t count = 1;
   for (int i = 0; i < 3; i++) {
      double mn = P[i] < Q[i] ? P[i] : Q[i], mx = P[i] < Q[i] ? Q[i] : P[i];
      const double top = (double)dim[i];
      mn -= rmax;
      mx += rmax;
      if (0.0 > mn)
         mn = 0.0;
      if (top < mx)
         mx = top;
      if (!(mn <= mx)) { // empty or non-finite box
         lo_out[i] = 0;
         ext_out[i] = 0;
         count = 0;
         continue;
      }
      // (int64) truncation as generator.cpp:304-305; the clamp only
      // restates that the box already lies in [0, dim]
      int64_t lo = (int64_t)mn, hi = (int64_t)(mx + 0.5);
      lo = lo < 0 ? 0 : lo;
      hi = hi > dim[i] ? dim[i] : hi;
      lo_out[i] = (int32_t)lo;
      ext_out[i] = (int32_t)(hi > lo ? hi - lo : 0);
      count *= ext_out[i];
   }
   return count;
}

// One segment of the table from its ends and radii, in double exactly as the
// reference derives the corresponding values: host and device give the same
// bits (IEEE operations, no contraction).
FPGB_HD void fill_segment(const double *P, const double *Q, double r0, double r1, int32_t bundle,
                          float f_ly_squ, double sqrt_last, const int64_t dim[3], SegDev &S) {
   segment_box(P, Q, r0, r1, sqrt_last, dim, S.lo, S.ext);
   for (int i = 0; i < 3; i++) {
      S.p[i] = P[i];
      S.q[i] = Q[i];
      S.v[i] = Q[i] - P[i];
      const double base = floor(P[i]);
      S.base[i] = (int32_t)fmax(-2147483647.0, fmin(2147483647.0, base));
   }
   double c = 0.0;
   c = c + S.v[0] * S.v[0];
   c = c + S.v[1] * S.v[1];
   c = c + S.v[2] * S.v[2];
   S.c2 = c;
   S.r0 = r0;
   S.r1 = r1;
   fill_fast_fields(S, dim);
   const double rm = r0 < r1 ? r1 : r0;
   S.thr_f = (float)((double)f_ly_squ * rm * rm * (1.0 + 1e-5)) * (1.f + 0x1p-22f);
   S.mg = seg_margin(S, S.thr_f);
   const double rn = r0 < r1 ? r0 : r1;
   const double a = (double)f_ly_squ * rn * rn * (1.0 - 1e-5);
   float af = (float)a;
   if ((double)af > a)
      af = nextafterf(af, 0.f);
   S.acc_f = af > 0.f ? fminf(af, 3e38f) : -1.f; // (finite, as hi)
   // From 2^30 voxels on differences to base leave 32 bits, from 1e19 on the
   // estimate's squares overflow, and an infinite one is not a distance.
   if (!(S.pscale < 0x1p30f)) {
      S.mg = S.c2f = INFINITY;
      S.acc_f = -1.f;
   }
   S.bundle = bundle;
}

// ======================================================================
// host planning (double precision, reference operation order)
// ======================================================================
namespace {

struct Box {
   double mn[3], mx[3];
   void empty() {
      for (int i = 0; i < 3; i++) {
         mn[i] = INFINITY;
         mx[i] = -INFINITY;
      }
   }
   // aabb::AABB(p, q) unsorted constructor (aabb.hpp:54-71)
   void from_pq(const double *p, const double *q) {
      for (int i = 0; i < 3; i++) {
         if (p[i] < q[i]) {
            mn[i] = p[i];
            mx[i] = q[i];
         } else {
            mn[i] = q[i];
            mx[i] = p[i];
         }
      }
   }
   void unite(const Box &a) { // aabb.hpp:90-97
      for (int i = 0; i < 3; i++) {
         if (a.mn[i] < mn[i])
            mn[i] = a.mn[i];
         if (a.mx[i] > mx[i])
            mx[i] = a.mx[i];
      }
   }
};

bool overlap(const Box &a, const Box &b) { // aabb.hpp:128-137
   for (int i = 0; i < 3; i++)
      if (a.mn[i] >= b.mx[i] || a.mx[i] <= b.mn[i])
         return false;
   return true;
}

// Fiber::CalculateVoi (fiber.cpp:83-99) of already transformed points.
Box fiber_box(const double *xyz, const double *r, int64_t n) {
   Box b;
   b.empty();
   if (n == 0)
      return b;
   const double lo[3] = {xyz[0] - r[0], xyz[1] - r[0], xyz[2] - r[0]};
   const double hi[3] = {xyz[0] + r[0], xyz[1] + r[0], xyz[2] + r[0]};
   b.from_pq(lo, hi);
   for (int64_t s = 0; s + 1 < n; s++) {
      const double rm = r[s] < r[s + 1] ? r[s + 1] : r[s];
      Box t;
      t.from_pq(xyz + 3 * s, xyz + 3 * (s + 1));
      for (int i = 0; i < 3; i++) {
         t.mn[i] -= rm;
         t.mx[i] += rm;
      }
      b.unite(t);
   }
   return b;
}

} // namespace

// Up to this many points one thread plans faster than waking the others takes
// (320 points: 21 us against 42).
[[maybe_unused]] constexpr int64_t kSerialPoints = 1000;
// Segment tables up to this size are filled on the host and go up with the
// small tables: a copy from pageable memory costs the host about 8 us however
// small.  Larger ones are filled on the device from the points, a sixth of the
// bytes (94,451 segments: 325 us of 16 host threads and a copy of 165 us before;
// the kernel takes 36 us, and the whole call went from 2122 to 1501 us; 980,000 segments:
// 29.6 and 22.7 ms).
constexpr size_t kTogetherBytes = size_t(256) << 10;

int plan_tissue(const fpgb_volume *vol, const fpgb_fibers *fb, TissuePlan *plan, bool fill) {
   if (!vol || !fb) {
      set_error("generate_tissue: null volume or fibers");
      return FPGB_EINVAL;
   }
   // SetVolume (generator.cpp:49-53,115-117)
   if (vol->dim[0] <= 0 || vol->dim[1] <= 0 || vol->dim[2] <= 0) {
      set_error("dim.global[any] <= 0: [%lld,%lld,%lld]",
                (long long)vol->dim[0], (long long)vol->dim[1],
                (long long)vol->dim[2]);
      return FPGB_EINVAL;
   }
   if (!(vol->voxel_size > 0)) {
      set_error("voxel_size <= 0: %g", vol->voxel_size);
      return FPGB_EINVAL;
   }
   for (int i = 0; i < 3; i++)
      if (vol->dim[i] > (int64_t(1) << 30)) {
         set_error("dim[%d] = %lld exceeds 2^30", i, (long long)vol->dim[i]);
         return FPGB_EINVAL;
      }
   const int64_t nb = fb->n_bundles;
   if (nb < 0 || (nb > 0 && (!fb->bundle_fiber_off || !fb->fiber_point_off ||
                             !fb->bundle_layer_off))) {
      set_error("generate_tissue: malformed fiber bundle offsets");
      return FPGB_EINVAL;
   }
   plan->X = vol->dim[0];
   plan->Y = vol->dim[1];
   plan->Z = vol->dim[2];
   plan->n_bundles = nb;
   plan->long_segs = false;
   plan->segs.clear();
   plan->source.clear();
   plan->layers.assign(nb > 0 ? nb : 1, LayerDev{});
   plan->single_point = 0;

   // layers, sorted by scale (fiber_bundle.cpp:19-30,66,83-86)
   int max_layer = 0;
   for (int64_t b = 0; b < nb; b++) {
      const int64_t l0 = fb->bundle_layer_off[b], l1 = fb->bundle_layer_off[b + 1];
      const int n = int(l1 - l0);
      if (n < 0 || n > kMaxLayers) {
         set_error("bundle %lld has %d layers (1..%d supported)",
                   (long long)b, n, kMaxLayers);
         return FPGB_EINVAL;
      }
      std::vector<int> order(n);
      for (int i = 0; i < n; i++)
         order[i] = i;
      std::stable_sort(order.begin(), order.end(), [&](int a, int c) {
         return fb->layer_scale[l0 + a] < fb->layer_scale[l0 + c];
      });
      LayerDev &L = plan->layers[b];
      L.n = n;
      for (int i = 0; i < n; i++) {
         const int64_t l = l0 + order[i];
         const char m = fb->layer_model[l];
         if (m != 'b' && m != 'p' && m != 'r') {
            set_error("Orientation must be \"b\", \"p\", or \"r\"");
            return FPGB_EINVAL;
         }
         L.scale_sq[i] = fb->layer_scale[l] * fb->layer_scale[l];
         L.model[i] = m;
         L.models |= (uint32_t)(m == 'p' ? 1 : m == 'r' ? 2 : 0) << (2 * i);
         L.dn[i] = fb->layer_dn[l];
         L.mu[i] = fb->layer_mu[l];
      }
      for (int i = 0; i < n; i++) {
         float f = (float)L.scale_sq[i];
         if ((double)f > L.scale_sq[i])
            f = std::nextafter(f, -INFINITY);
         L.sq_fdown[i] = f;
      }
      if (n > 0) {
         L.f_ly_squ = (float)L.scale_sq[n - 1];
         L.sqrt_last = std::sqrt(L.scale_sq[n - 1]);
      }
      max_layer = std::max(max_layer, n);
   }
   plan->max_layer = max_layer;

   // property table (generator.cpp:496-526)
   plan->props.assign(2 * (nb * max_layer + 1), 0.0);
   for (int64_t b = 0; b < nb; b++)
      for (int l = 0; l < plan->layers[b].n; l++) {
         const int64_t id = 1 + l + b * max_layer;
         plan->props[2 * id + 1] = plan->layers[b].mu[l];
         plan->props[2 * id] =
             plan->layers[b].model[l] == 'b' ? 0.0 : plan->layers[b].dn[l];
      }

   // translate then resize (generator.cpp:185-197, fiber.cpp:128-150)
   const int64_t nf = nb > 0 ? fb->bundle_fiber_off[nb] : 0;
   const int64_t np = nf > 0 ? fb->fiber_point_off[nf] : 0;
   if (np > 0 && !fb->points) {
      set_error("generate_tissue: points == NULL");
      return FPGB_EINVAL;
   }
   // (a fiber of n points has fewer than n segments)
   plan->n_points = np;
   plan->source.reset((32 + sizeof(SegSrc)) * (size_t)np);
   double *xyz = reinterpret_cast<double *>(plan->source.data()), *rad = xyz + 3 * np;
   const bool translate =
       vol->origin[0] != 0 || vol->origin[1] != 0 || vol->origin[2] != 0;
   const double f = 1.0 / vol->voxel_size;
   // first non-finite coordinate (points are checked, translated and scaled
   // in parallel; the error names the lowest bad point as a serial scan would)
   int64_t bad = INT64_MAX;
#pragma omp parallel for schedule(static) reduction(min : bad) if (np > kSerialPoints)
   for (int64_t i = 0; i < np; i++) {
      const double *q = fb->points + 4 * i;
      if (!(std::isfinite(q[0]) && std::isfinite(q[1]) && std::isfinite(q[2]) &&
            std::isfinite(q[3]))) {
         bad = std::min(bad, i);
         continue;
      }
      for (int c = 0; c < 3; c++) {
         double v = q[c];
         if (translate)
            v = v + (-vol->origin[c]);
         xyz[3 * i + c] = v * f;
      }
      rad[i] = q[3] * f;
   }
   if (bad != INT64_MAX) {
      set_error("fiber point %lld is not finite", (long long)bad);
      return FPGB_EINVAL;
   }
   for (int64_t fi = 0; fi < nf; fi++) {
      const int64_t p0 = fb->fiber_point_off[fi], p1 = fb->fiber_point_off[fi + 1];
      if (p1 < p0 || p1 > np) {
         set_error("generate_tissue: malformed fiber_point_off");
         return FPGB_EINVAL;
      }
   }
   std::vector<Box> fbox(nf);
#pragma omp parallel for schedule(dynamic, 32) if (np > kSerialPoints)
   for (int64_t fi = 0; fi < nf; fi++) {
      const int64_t p0 = fb->fiber_point_off[fi], p1 = fb->fiber_point_off[fi + 1];
      fbox[fi] = fiber_box(xyz + 3 * p0, rad + p0, p1 - p0);
   }
   Box volbox;
   for (int i = 0; i < 3; i++) {
      volbox.mn[i] = 0.0;
      volbox.mx[i] = (double)vol->dim[i];
   }

   // segment table in the reference's processing order (generator.cpp:205-231):
   // which bundles overlap the volume is decided first, then the fibers are
   // planned in parallel into per-fiber lists that are concatenated in order
   std::vector<char> bundle_on(nb > 0 ? nb : 1, 0);
   std::vector<int32_t> fiber_bundle(nf);
   for (int64_t b = 0; b < nb; b++) {
      const int64_t f0 = fb->bundle_fiber_off[b], f1 = fb->bundle_fiber_off[b + 1];
      Box bb;
      bb.empty(); // fiber_bundle.cpp:147-154
      if (f1 > f0)
         bb = fbox[f0];
      for (int64_t fi = f0; fi < f1; fi++) {
         bb.unite(fbox[fi]);
         fiber_bundle[fi] = (int32_t)b;
      }
      bundle_on[b] = overlap(volbox, bb) ? 1 : 0;
   }
   // pass 1: segments each fiber keeps (its boxes only), their candidates and
   // bricks; pass 2 fills the table, or notes the segments' sources, in place at
   // the fibers' prefix offsets
   RawArray<char> kept;
   kept.reset((size_t)np);
   std::vector<int64_t> fiber_segs(nf + 1, 0);
   std::vector<char> single(nf, 0);
   auto fiber_used = [&](int64_t fi) -> bool {
      const int64_t b = fiber_bundle[fi];
      const int64_t p0 = fb->fiber_point_off[fi], p1 = fb->fiber_point_off[fi + 1];
      return bundle_on[b] && p1 - p0 > 1 && overlap(volbox, fbox[fi]) && plan->layers[b].n > 0;
   };
   int64_t cand = 0, pairs = 0;
   bool longer = false;
#pragma omp parallel for schedule(dynamic, 32) reduction(+ : cand, pairs) reduction(|| : longer) if (np > kSerialPoints)
   for (int64_t fi = 0; fi < nf; fi++) {
      const int64_t b = fiber_bundle[fi];
      const int64_t p0 = fb->fiber_point_off[fi], p1 = fb->fiber_point_off[fi + 1];
      if (bundle_on[b] && p1 - p0 <= 1)
         single[fi] = 1;
      if (!fiber_used(fi))
         continue;
      int64_t n = 0;
      SegDev S;
      double longest = 0.0; // squared
      for (int64_t s = p0; s + 1 < p1; s++) {
         const double *P = &xyz[3 * s], *Q = P + 3;
         const int64_t count = segment_box(P, Q, rad[s], rad[s + 1], plan->layers[b].sqrt_last,
                                           vol->dim, S.lo, S.ext);
         kept[s] = count > 0;
         if (count == 0)
            continue;
         n++;
         cand += count;
         pairs += segment_brick_pairs(S);
         const double c2 = (Q[0] - P[0]) * (Q[0] - P[0]) + (Q[1] - P[1]) * (Q[1] - P[1]) +
                           (Q[2] - P[2]) * (Q[2] - P[2]);
         longest = c2 > longest ? c2 : longest;
      }
      // (the fiber's box has its points: no coordinate is past it)
      for (int i = 0; i < 3; i++)
         longer = longer || !(fbox[fi].mn[i] > -0x1p29 && fbox[fi].mx[i] < 0x1p29);
      longer = longer || (float)longest > kLongSquared;
      fiber_segs[fi + 1] = n;
   }
   for (int64_t fi = 0; fi < nf; fi++) {
      fiber_segs[fi + 1] += fiber_segs[fi];
      plan->single_point += single[fi];
   }
   plan->n_segs = fiber_segs[nf];
   plan->candidates = cand;
   plan->brick_pairs = pairs;
   plan->long_segs = longer;
   if (plan->n_segs > 0xFFFFFFF0ll) {
      set_error("too many fiber segments: %lld", (long long)plan->n_segs);
      return FPGB_EINVAL;
   }
   fill = fill || sizeof(SegDev) * (size_t)plan->n_segs <= kTogetherBytes ||
          np > 0xFFFFFFFFll; // SegSrc::point
   if (fill)
      plan->segs.reset((size_t)plan->n_segs);
   SegDev *table = plan->segs.data();
   SegSrc *src = reinterpret_cast<SegSrc *>(rad + np);
#pragma omp parallel for schedule(dynamic, 32) if (np > kSerialPoints)
   for (int64_t fi = 0; fi < nf; fi++) {
      if (fiber_segs[fi + 1] == fiber_segs[fi])
         continue;
      const int64_t b = fiber_bundle[fi];
      const LayerDev &L = plan->layers[b];
      const int64_t p0 = fb->fiber_point_off[fi], p1 = fb->fiber_point_off[fi + 1];
      int64_t at = fiber_segs[fi];
      for (int64_t s = p0; s + 1 < p1; s++) {
         if (!kept[s])
            continue;
         if (fill)
            fill_segment(&xyz[3 * s], &xyz[3 * (s + 1)], rad[s], rad[s + 1], (int32_t)b,
                         L.f_ly_squ, L.sqrt_last, vol->dim, table[at]);
         else
            src[at] = SegSrc{(uint32_t)s, (int32_t)b};
         at++;
      }
   }
   if (fill)
      plan->source.clear();
   return FPGB_OK;
}

// ======================================================================
// device code
// ======================================================================
// The segment table from the points, a thread per segment.  Bound by its FP64
// arithmetic (the pipe 83% busy): 94,451 segments 36 us, 980,000 318 us.
__global__ void __launch_bounds__(128)
fill_segments(const double *__restrict__ xyz, const double *__restrict__ rad,
              const SegSrc *__restrict__ src, int64_t n, const LayerDev *__restrict__ layers,
              int64_t X, int64_t Y, int64_t Z, SegDev *__restrict__ segs) {
   const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
   if (i >= n)
      return;
   const int64_t dim[3] = {X, Y, Z};
   const int64_t s = src[i].point;
   const LayerDev &L = layers[src[i].bundle];
   SegDev S;
   fill_segment(xyz + 3 * s, xyz + 3 * (s + 1), rad[s], rad[s + 1], src[i].bundle, L.f_ly_squ,
                L.sqrt_last, dim, S);
   segs[i] = S;
}

// ======================================================================
// launch
// ======================================================================
// Device workspace of one voxelization: the tile header (one TileDev and the
// label / vector pointers), segment table, layers, counters, and the brick
// lists of the voxelizer.
static int64_t plan_bricks(const TissuePlan &p, int32_t nb[3]) {
   int64_t n = 0;
   tile_bricks(p.X, p.Y, p.Z, nb, &n);
   return n;
}

size_t tissue_workspace_bytes(const TissuePlan &p, bool most) {
   int32_t nb[3];
   const int64_t n_bricks = plan_bricks(p, nb);
   size_t b = align_up(sizeof(TileDev) + 2 * sizeof(void *), 256);
   b += align_up(sizeof(SegDev) * std::max<size_t>((size_t)p.n_segs, 1), 256);
   b += align_up(sizeof(LayerDev) * p.layers.size(), 256);
   b += align_up(sizeof(unsigned long long) * kCounterWords, 256);
   b += brick_workspace_bytes(n_bricks, p.brick_pairs, p.n_segs);
   return b + (most ? brick_workspace_more(n_bricks) : 0);
}

// Bricks of a slabbed launch, at least: 4 per SM (a wave of the 256-thread
// CTAs, half of one of the 128-thread ones).
constexpr int64_t kSlabBricks = 608;

int run_tissue(const TissuePlan &p, int only_label, int32_t *d_label,
               float *d_vector, void *d_ws, size_t ws_bytes,
               unsigned long long **d_counters_out, cudaStream_t st, int n_slabs,
               int (*after_slab)(void *ctx, int64_t x0, int64_t x1, cudaStream_t s), void *ctx,
               cudaStream_t alt) {
   const size_t need = tissue_workspace_bytes(p);
   if (ws_bytes < need) {
      set_error("generate_tissue: workspace %zu bytes < %zu needed", ws_bytes, need);
      return FPGB_ENOMEM;
   }
   if (reinterpret_cast<uintptr_t>(d_ws) % 256 != 0) {
      set_error("generate_tissue: workspace must be 256-byte aligned");
      return FPGB_EINVAL;
   }
   int32_t nb[3];
   const int64_t n_bricks = plan_bricks(p, nb);
   // head, layers and counters, then the segment table, then the brick lists
   const size_t layer_off = align_up(sizeof(TileDev) + 2 * sizeof(void *), 256);
   const size_t counter_off = layer_off + align_up(sizeof(LayerDev) * p.layers.size(), 256);
   const size_t seg_off =
       counter_off + align_up(sizeof(unsigned long long) * kCounterWords, 256);
   const size_t seg_bytes = sizeof(SegDev) * (size_t)p.n_segs;
   char *w = static_cast<char *>(d_ws);
   char *head = w;
   auto *layers = reinterpret_cast<LayerDev *>(w + layer_off);
   auto *counters = reinterpret_cast<unsigned long long *>(w + counter_off);
   auto *segs = reinterpret_cast<SegDev *>(w + seg_off);
   w += seg_off + align_up(sizeof(SegDev) * std::max<size_t>((size_t)p.n_segs, 1), 256);

   // the single volume as tile 0 of the brick voxelizer
   struct {
      TileDev t;
      void *label, *vector;
   } h{};
   h.t.vox_base = 0;
   h.t.n_vox = p.X * p.Y * p.Z;
   h.t.brick_base = 0;
   h.t.X = (int32_t)p.X;
   h.t.Y = (int32_t)p.Y;
   h.t.Z = (int32_t)p.Z;
   h.t.max_layer = p.max_layer;
   h.t.layer_base = 0;
   h.t.n_bundles = (int32_t)p.layers.size();
   for (int i = 0; i < 3; i++)
      h.t.nb[i] = nb[i];
   h.label = d_label;
   h.vector = only_label ? nullptr : d_vector;
   static_assert(sizeof(h) == sizeof(TileDev) + 2 * sizeof(void *), "tile header layout");

   // one upload of the small tables (counters 0), with the segments where they
   // are few
   const bool together = seg_bytes <= kTogetherBytes && !p.segs.empty();
   std::vector<char> stage(seg_off + (together ? seg_bytes : 0));
   std::memcpy(stage.data(), &h, sizeof h);
   std::memcpy(stage.data() + layer_off, p.layers.data(), sizeof(LayerDev) * p.layers.size());
   if (together && seg_bytes)
      std::memcpy(stage.data() + seg_off, p.segs.data(), seg_bytes);
   FPGB_CUDA_TRY(cudaMemcpyAsync(head, stage.data(), stage.size(), cudaMemcpyHostToDevice, st));
   if (!together && seg_bytes) {
      // the points go where the brick lists will be, when they fit
      const size_t bytes = p.source_bytes();
      if (p.segs.empty() && bytes <= ws_bytes - (size_t)(w - static_cast<char *>(d_ws))) {
         FPGB_CUDA_TRY(cudaMemcpyAsync(w, p.source.data(), bytes, cudaMemcpyHostToDevice, st));
         auto *xyz = reinterpret_cast<const double *>(w);
         fill_segments<<<(unsigned)((p.n_segs + 127) / 128), 128, 0, st>>>(
             xyz, xyz + 3 * p.n_points, reinterpret_cast<const SegSrc *>(xyz + 4 * p.n_points),
             p.n_segs, layers, p.X, p.Y, p.Z, segs);
         FPGB_CUDA_TRY(cudaGetLastError());
      } else {
         RawArray<SegDev> table; // (long fibers of which little is in the volume)
         const SegDev *from = p.segs.data();
         if (p.segs.empty()) {
            table.reset((size_t)p.n_segs);
            const int64_t dim[3] = {p.X, p.Y, p.Z};
            const double *xyz = reinterpret_cast<const double *>(p.source.data());
            const double *rad = xyz + 3 * p.n_points;
            auto *src = reinterpret_cast<const SegSrc *>(rad + p.n_points);
#pragma omp parallel for schedule(static)
            for (int64_t i = 0; i < p.n_segs; i++) {
               const LayerDev &L = p.layers[src[i].bundle];
               const int64_t a = src[i].point;
               fill_segment(xyz + 3 * a, xyz + 3 * (a + 1), rad[a], rad[a + 1], src[i].bundle,
                            L.f_ly_squ, L.sqrt_last, dim, table[i]);
            }
            from = table.data();
         }
         FPGB_CUDA_TRY(cudaMemcpyAsync(segs, from, seg_bytes, cudaMemcpyHostToDevice, st));
      }
   }
   auto *tile = reinterpret_cast<const TileDev *>(head);
   auto *lp = reinterpret_cast<int32_t *const *>(head + sizeof(TileDev));
   auto *vp = reinterpret_cast<float *const *>(head + sizeof(TileDev) + sizeof(void *));
   // x-slabs of whole brick columns: bricks are numbered x-major, so a range
   // of brick x indices is a contiguous brick range and a contiguous x range
   // of voxels
   struct Slabs {
      int64_t bx[65];
      int64_t X;
      int (*after)(void *, int64_t, int64_t, cudaStream_t);
      void *ctx;
      static int thunk(void *self, int c, cudaStream_t s) {
         const Slabs &S = *static_cast<const Slabs *>(self);
         const int64_t x0 = S.bx[c] * kBrickX, x1 = std::min(S.bx[c + 1] * kBrickX, S.X);
         return S.after ? S.after(S.ctx, x0, x1, s) : FPGB_OK;
      }
   } slabs;
   int64_t bound[65];
   BrickChunks chunks{};
   // (a launch of less than a wave of bricks takes as long as a whole one)
   const int n = (int)std::max<int64_t>(
       1, std::min<int64_t>({(int64_t)n_slabs, 64, nb[0], n_bricks / kSlabBricks}));
   if (n > 1) {
      slabs.X = p.X;
      slabs.after = after_slab;
      slabs.ctx = ctx;
      for (int c = 0; c <= n; c++) {
         slabs.bx[c] = nb[0] * c / n;
         bound[c] = slabs.bx[c] * nb[1] * nb[2];
      }
      chunks = BrickChunks{n, bound, &Slabs::thunk, &slabs, alt};
   }
   FPGB_TRY(launch_voxel_bricks(segs, nullptr, p.n_segs, tile, 1, n_bricks,
                                p.brick_pairs, layers, p.n_bundles > 1, p.long_segs, lp, vp, w,
                                ws_bytes - (size_t)(w - static_cast<char *>(d_ws)), counters, st,
                                n > 1 ? &chunks : nullptr));
   if (n == 1 && after_slab)
      FPGB_TRY(after_slab(ctx, 0, p.X, st));
   l2_end_state().store(1, std::memory_order_relaxed); // bricks run x-major: high x last
   if (d_counters_out)
      *d_counters_out = counters;
   return FPGB_OK;
}

// Copies of finished x-slabs of a host-buffer generation (page-locked
// outputs), queued on their own stream behind an event of the slab's launch.
// The slab launches alternate between two streams so that one slab's last
// bricks overlap the next slab's first; then thinner slabs pay: on the
// 512 x 512 x 120 bench volume a call took 4.24 ms with 8 slabs on one
// stream, 4.39 / 4.09 / 4.03 ms with 8 / 16 / 24 slabs on two (the copy
// alone is 2.62 ms).
constexpr int kCopySlabs = 24;

struct SlabCopy {
   int32_t *label;
   float *vector;
   const int32_t *d_label;
   const float *d_vector;
   int64_t row; // voxels per x
   cudaStream_t copy;
   std::vector<cudaEvent_t> events;

   static int after(void *self, int64_t x0, int64_t x1, cudaStream_t s) {
      SlabCopy &S = *static_cast<SlabCopy *>(self);
      cudaEvent_t ev;
      FPGB_CUDA_TRY(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
      S.events.push_back(ev);
      FPGB_CUDA_TRY(cudaEventRecord(ev, s));
      FPGB_CUDA_TRY(cudaStreamWaitEvent(S.copy, ev, 0));
      const int64_t v0 = x0 * S.row, nv = (x1 - x0) * S.row;
      FPGB_CUDA_TRY(cudaMemcpyAsync(S.label + v0, S.d_label + v0, sizeof(int32_t) * nv,
                                    cudaMemcpyDeviceToHost, S.copy));
      if (S.vector)
         FPGB_CUDA_TRY(cudaMemcpyAsync(S.vector + 3 * v0, S.d_vector + 3 * v0,
                                       sizeof(float) * 3 * nv, cudaMemcpyDeviceToHost, S.copy));
      return FPGB_OK;
   }
};

int finish_props(const TissuePlan &p, double *props, int64_t props_cap, int64_t *n_props) {
   const int64_t n = (int64_t)p.props.size() / 2;
   if (n_props)
      *n_props = n;
   if (props) {
      if (props_cap < n) {
         set_error("props_cap %lld < %lld rows", (long long)props_cap, (long long)n);
         return FPGB_EINVAL;
      }
      std::memcpy(props, p.props.data(), sizeof(double) * 2 * n);
   }
   return FPGB_OK;
}

int tissue_status_from_counters(const TissuePlan &p, const long long *h, fpgb_warnings *w) {
   if (h[6] & kStatusOverflow) { // the device binning disagreed with the host plan
      set_error("generate_tissue: internal error, segment-brick lists overflowed");
      return FPGB_ECUDA;
   }
   if (!w)
      return FPGB_OK;
   warnings_from_counters(h, w);
   w->overlap = w->overlap > 0 ? 1 : 0; // the reference warns once (generator.cpp:353-359)
   w->single_point = p.single_point;
   return FPGB_OK;
}

int read_tissue_warnings(const TissuePlan &p, unsigned long long *d_counters, fpgb_warnings *w,
                         cudaStream_t st) {
   if (!w)
      return FPGB_OK;
   long long h[kCounterWords];
   FPGB_CUDA_TRY(cudaMemcpyAsync(h, d_counters, sizeof h, cudaMemcpyDeviceToHost, st));
   FPGB_CUDA_TRY(cudaStreamSynchronize(st));
   return tissue_status_from_counters(p, h, w);
}

} // namespace fpgb

using namespace fpgb;

extern "C" {

size_t fpgb_generate_workspace_size(const fpgb_volume *vol, const fpgb_fibers *fibers) {
   TissuePlan p;
   if (plan_tissue(vol, fibers, &p, false) != FPGB_OK)
      return 0;
   return tissue_workspace_bytes(p);
}

int fpgb_generate_tissue_device(const fpgb_volume *vol, const fpgb_fibers *fibers,
                                int only_label, int32_t *d_label, float *d_vector,
                                double *props, int64_t props_cap, int64_t *n_props,
                                void *d_workspace, size_t workspace_bytes,
                                fpgb_warnings *warnings, void *stream) {
   TissuePlan p;
   FPGB_TRY(plan_tissue(vol, fibers, &p, false));
   if (!d_label || (!only_label && !d_vector)) {
      set_error("generate_tissue_device: null output buffer");
      return FPGB_EINVAL;
   }
   if (!d_workspace) {
      const size_t need = tissue_workspace_bytes(p, true);
      FPGB_TRY(pool_get(kSlotKeys, need, &d_workspace, as_stream(stream)));
      workspace_bytes = need;
   }
   unsigned long long *d_counters = nullptr;
   cudaStream_t st = as_stream(stream);
   FPGB_TRY(run_tissue(p, only_label, d_label, d_vector, d_workspace, workspace_bytes,
                       &d_counters, st));
   FPGB_TRY(finish_props(p, props, props_cap, n_props));
   return read_tissue_warnings(p, d_counters, warnings, st);
}

int fpgb_generate_tissue(const fpgb_volume *vol, const fpgb_fibers *fibers, int only_label,
                         int32_t *label, float *vector, double *props, int64_t props_cap,
                         int64_t *n_props, fpgb_warnings *warnings) {
   TissuePlan p;
   FPGB_TRY(plan_tissue(vol, fibers, &p, false));
   if (!label || (!only_label && !vector)) {
      set_error("generate_tissue: null output buffer");
      return FPGB_EINVAL;
   }
   const int64_t nvox = p.X * p.Y * p.Z;
   void *d_label = nullptr, *d_vec = nullptr, *d_ws = nullptr;
   FPGB_TRY(pool_get(kSlotLabel, sizeof(int32_t) * nvox, &d_label));
   if (!only_label)
      FPGB_TRY(pool_get(kSlotVector, sizeof(float) * 3 * nvox, &d_vec));
   const size_t need = tissue_workspace_bytes(p, true);
   FPGB_TRY(pool_get(kSlotKeys, need, &d_ws));
   cudaStream_t st = nullptr;
   unsigned long long *d_counters = nullptr;
   if (host_pinned(label) && (only_label || host_pinned(vector))) {
      // page-locked outputs: each x-slab's rows are copied on a second stream
      // while the next slabs are voxelized
      SlabCopy sc;
      sc.label = label;
      sc.vector = only_label ? nullptr : vector;
      sc.d_label = static_cast<const int32_t *>(d_label);
      sc.d_vector = static_cast<const float *>(d_vec);
      sc.row = p.Y * p.Z;
      cudaStream_t alt = nullptr;
      FPGB_CUDA_TRY(cudaStreamCreateWithFlags(&sc.copy, cudaStreamNonBlocking));
      cudaError_t e = cudaStreamCreateWithFlags(&alt, cudaStreamNonBlocking);
      int rc = e == cudaSuccess ? run_tissue(p, only_label, (int32_t *)d_label, (float *)d_vec,
                                             d_ws, need, &d_counters, st, kCopySlabs,
                                             &SlabCopy::after, &sc, alt)
                                : FPGB_ECUDA;
      if (e != cudaSuccess)
         set_error("generate_tissue: %s", cudaGetErrorString(e));
      e = cudaStreamSynchronize(sc.copy);
      for (cudaEvent_t ev : sc.events)
         cudaEventDestroy(ev);
      cudaStreamDestroy(sc.copy);
      if (alt) {
         cudaStreamSynchronize(alt);
         cudaStreamDestroy(alt);
      }
      FPGB_TRY(rc);
      if (e != cudaSuccess) {
         set_error("generate_tissue: %s", cudaGetErrorString(e));
         return FPGB_ECUDA;
      }
   } else {
      FPGB_TRY(run_tissue(p, only_label, (int32_t *)d_label, (float *)d_vec, d_ws, need,
                          &d_counters, st));
      // while the voxelizer runs
      prefault_host(label, sizeof(int32_t) * nvox);
      if (!only_label)
         prefault_host(vector, sizeof(float) * 3 * nvox);
      FPGB_CUDA_TRY(cudaMemcpyAsync(label, d_label, sizeof(int32_t) * nvox,
                                    cudaMemcpyDeviceToHost, st));
      if (!only_label)
         FPGB_CUDA_TRY(cudaMemcpyAsync(vector, d_vec, sizeof(float) * 3 * nvox,
                                       cudaMemcpyDeviceToHost, st));
   }
   FPGB_TRY(finish_props(p, props, props_cap, n_props));
   fpgb_warnings tmp;
   FPGB_TRY(read_tissue_warnings(p, d_counters, warnings ? warnings : &tmp, st));
   FPGB_CUDA_TRY(cudaStreamSynchronize(st));
   return FPGB_OK;
}

} // extern "C"
