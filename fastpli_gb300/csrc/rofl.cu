// ROFL tilt analysis (src/fastpli/analysis/rofl.py:16-63,
// _ROFL_with_jacobi.py:47-522; Schmitz et al., Front. Neuroanat. 2018,
// doi:10.3389/fnana.2018.00075) of every pixel of a 5-tilt image series,
// a few lanes of a warp per pixel, FP64.
//
// Per pixel, as the reference: the untilted direction (epa.direction) starts
// the fit; the measurements are centered (I / mean - 1) and weighted by
// 1 / sigma of the gain noise model; a 6 x 6 grid over inclination and t_rel
// picks the start point (first minimum); a Levenberg-Marquardt fit of
// (direction, inclination, t_rel) minimises the weighted residuals of the
// model sin(pi/2 t cos^2 alpha) sin(2 (rho - phi)) over all tilts; the result
// is folded into the PLI range and its standard deviations come from the
// reference's covariance formula.
//
// The fit is MINPACK's Levenberg-Marquardt as the reference calls it
// (scipy.optimize.leastsq: forward differences, or in grad_mode the
// reference's own Jacobian; the same tolerances, scaling and budget of 150
// evaluations), restated below; n_fev is MINPACK's evaluation count.
//
// FP64 is what bounds it, in two ways: an SM issues one FP64 warp instruction
// per 19 cycles whatever its warps, and a lone warp one per 64.  A thread per
// pixel keeps the instructions of a warp few but makes a map of some thousand
// pixels wait for the chain of its slowest fit (37 iterations of 13,000
// instructions: 17 ms); a warp per pixel repeats every per-pixel step (the
// 3 x 3 trust-region algebra, sums in a fixed order) in 32 lanes.  Four lanes
// share the measurements, the tilts and the Jacobian's columns of a pixel: the
// chain is a quarter as long, and the sums of the three columns, each in the
// order MINPACK (sequential) or numpy (pairwise) takes it, run side by side.
// Small maps, which wait for the longest chain, take 16 lanes, large ones 1
// (one_lane_pixels).
// Compiled with -fmad=false: products and sums round separately, as in the
// reference, except where a fused multiply-add is written out.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#include "fpgb_common.cuh"

namespace fpgb {

constexpr int kRoflMaxRot = 32;
constexpr int kRoflSmallRot = 10; // the usual 6 - 9 rotations: 50 measurements

struct RoflParams {
   int n_rot;
   int grad_mode;
   int inv_rot; // i / n_rot = i * inv_rot >> 16 for i < 5 n_rot
   double tau, gain, dir_offset, cos_tau;
   double rho[kRoflMaxRot];    // linspace(0, pi, R + 1)[:-1] + dir_offset
   double rho2s[kRoflMaxRot];  // sin / cos of 2 linspace(0, pi, R, False)
   double rho2c[kRoflMaxRot];  //   (epa.direction of the untilted series)
   double mat[4][9];           // tilt rotations, psi = 0, pi/2, pi, 3 pi/2
   double incl[6], trel[6];    // start grid
};

// numpy.remainder for b > 0: result in [0, b).  Within two periods of 0 the
// truncated remainder is the argument or one exact subtraction away (Sterbenz),
// which is what fmod's digit loop gives.
__device__ __forceinline__ double pymod(double a, double b) {
   const double x = fabs(a);
   double m;
   if (x < b)
      m = a;
   else if (x < 2.0 * b)
      m = a < 0.0 ? a + b : a - b;
   else
      m = fmod(a, b); // (NaN too)
   if (m != 0.0 && m < 0.0)
      m += b;
   return m == 0.0 ? 0.0 : m;
}

// Many quotients by one divisor, each rounded once: with y = 1 / b rounded,
// q = a y is within 2 ulps of a / b, one residual correction makes it faithful
// and a second one correct (Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990).  Outside of
// the range where every step is free of under- and overflow, and for zeros,
// the division itself.
struct Divisor {
   double b, y;
   bool safe;
   __device__ __forceinline__ explicit Divisor(double d) : b(d), y(1.0 / d) {
      const double m = fabs(d);
      safe = m > 0x1p-300 && m < 0x1p300;
   }
   __device__ __forceinline__ double quotient(double a) const {
      const double m = fabs(a);
      if (!(safe && m > 0x1p-300 && m < 0x1p300))
         return a / b;
      double q = a * y;
      q = fma(fma(-b, q, a), y, q);
      return fma(fma(-b, q, a), y, q);
   }
};

// CUDA's FP64 sin, cos, sincos, atan and asin called out of line: one copy
// of each in the kernel's code instead of one per call site (the fit is
// bound by instruction fetch while the threads of a warp are in different
// phases of their fits)
__device__ __noinline__ double ol_sin(double x) { return sin(x); }
__device__ __noinline__ double ol_cos(double x) { return cos(x); }
__device__ __noinline__ void ol_sincos(double x, double *s, double *c) { sincos(x, s, c); }
__device__ __noinline__ double ol_atan(double x) { return atan(x); }
__device__ __noinline__ double ol_asin(double x) { return asin(x); }

// _symmetrize_angles (_ROFL_with_jacobi.py:64-74)
__device__ __forceinline__ void symmetrize(double &dir, double &incl) {
   // floor(dir / pi) is 0 or -1 without the division, away from its steps
   double turns;
   if (dir >= 0.0 && dir < 3.14159265)
      turns = 0.0;
   else if (dir < -1e-300 && dir > -3.14159265)
      turns = -1.0;
   else
      turns = floor(dir / M_PI);
   const double s = -pymod(turns, 2.0) + 0.5; // +-0.5
   incl = (pymod(incl + M_PI / 2.0, M_PI) - M_PI / 2.0) * (s > 0.0 ? 1.0 : -1.0);
   dir = pymod(dir, M_PI);
}

// np.dot of a 3 x 3 matrix row and a 3-vector (_calculate_rotated_fiber_params,
// :179) as numpy 2.5 on x86-64 rounds it where the reference's results were
// recorded: fma(a2, v2, fma(a0, v0, a1 v1)), found by comparing np.dot with
// exact rational arithmetic (all of 6,000 random rows agreed with this form,
// at most 76% with any other order, fused or not)
__device__ __forceinline__ double np_dot3(const double *a, double v0, double v1, double v2) {
   return fma(a[2], v2, fma(a[0], v0, a[1] * v1));
}

// The G lanes of one pixel.
template <int G> struct Lanes {
   int g;         // this lane's place
   unsigned mask; // the lanes' bits in the warp
   __device__ __forceinline__ Lanes() {
      const int lane = threadIdx.x & 31;
      g = lane % G;
      mask = (G == 32 ? ~0u : (1u << (G & 31)) - 1u) << (lane - g);
   }
   __device__ __forceinline__ void sync() const {
      if (G > 1)
         __syncwarp(mask);
   }
   __device__ __forceinline__ double from(double v, int lane) const {
      return G > 1 ? __shfl_sync(mask, v, lane, G) : v;
   }
};

// Per-tilt values of the model at one point, next to the pixel's arrays.
struct TiltValues {
   double phi[5], alpha[5], amp[5];
};

// The model's factors at one point of the fit: wave[i] = sin 2 (rho - phi) of
// every measurement, i = tilt * R + rotation (the order of the reference's
// flattened intensity curves, :186-212), and cos^2 of each tilt's inclination.
// (direction, inclination) in the tilts: :150-183, folded as the model uses
// them.  t_rel enters neither, so the 6 start points of one inclination and the
// forward difference in t_rel share them.  base (or null): the waves of a
// point with the same phi, whose untilted ones are the same.  Out of line,
// like the Jacobian and the trust-region step below: one copy of each large
// body keeps the kernel's code in the instruction cache while the pixels of a
// warp are in different phases of their fits.
template <int G>
__device__ __noinline__ void px_waves(const RoflParams &P, double phi, double alpha,
                                      const double *base, double *wave, TiltValues &T,
                                      double cos2[5]) {
   const Lanes<G> L;
   double sp, cp, sa, ca;
   ol_sincos(phi, &sp, &cp);
   ol_sincos(alpha, &sa, &ca);
   const double v0 = ca * cp, v1 = ca * sp, v2 = sa;
   for (int t = L.g; t < 5; t += G) { // tilts 1 .. 4, then the untilted
      const int j = t < 4 ? t + 1 : 0;
      double ph = phi, al = alpha;
      if (t < 4) {
         const double *M = P.mat[t];
         const double w0 = np_dot3(M, v0, v1, v2);
         const double w1 = np_dot3(M + 3, v0, v1, v2);
         const double w2 = np_dot3(M + 6, v0, v1, v2);
         ph = ol_atan(w1 / w0);
         al = ol_asin(w2);
      }
      symmetrize(ph, al);
      const double c = ol_cos(al);
      T.phi[j] = ph;
      T.alpha[j] = al;
      cos2[j] = c * c;
   }
   L.sync();
   const int R = P.n_rot, M = 5 * R;
   for (int i = L.g + (base ? R : 0); i < M; i += G) {
      const int j = i * P.inv_rot >> 16;
      wave[i] = ol_sin(2.0 * (P.rho[i - j * R] - T.phi[j]));
   }
   if (base && base != wave)
      for (int k = L.g; k < R; k += G)
         wave[k] = base[k];
   L.sync();
}

// |t_rel| as the model uses it in tilt j
__device__ __forceinline__ double tilt_trel(const RoflParams &P, int j, double trel) {
   return fabs(j == 0 ? trel : trel / P.cos_tau);
}

// weighted residuals r[i] = w[i] (model_i - c[i]) (_residuum, :407-410)
template <int G>
__device__ __noinline__ void px_residuals(const RoflParams &P, const double *c, const double *w,
                                          const double *wave, const double cos2[5],
                                          TiltValues &T, double trel, double *r) {
   const Lanes<G> L;
   for (int j = L.g; j < 5; j += G)
      T.amp[j] = ol_sin(M_PI / 2.0 * tilt_trel(P, j, trel) * cos2[j]);
   L.sync();
   const int R = P.n_rot, M = 5 * R;
   for (int i = L.g; i < M; i += G)
      r[i] = w[i] * (T.amp[i * P.inv_rot >> 16] * wave[i] - c[i]);
   L.sync();
}

// the reference's Jacobian of the model with respect to each tilt's own
// angles (_calc_Jacobi, :215-258), weighted (_weighted_jacobi, :393-403), at
// the point that wave and T.alpha are of: columns J[0..2][i] at J + col[0..2];
// used by grad_mode and by the covariance
template <int G>
__device__ __noinline__ void px_jacobi(const RoflParams &P, const double *w, const double *wave,
                                       const TiltValues &T, double trel, double *J,
                                       const int col[3]) {
   const Lanes<G> L;
   const int R = P.n_rot;
#pragma unroll 1
   for (int j = 0; j < 5; j++) {
      const double tr = tilt_trel(P, j, trel);
      const double ca = ol_cos(T.alpha[j]), sa = ol_sin(T.alpha[j]);
      const double arg = M_PI / 2.0 * tr * (ca * ca);
      const double sarg = ol_sin(arg), carg = ol_cos(arg);
      const double dal = -M_PI * tr * ca * sa * carg; // times s2
      const double dtr = M_PI / 2.0 * (ca * ca);      // times s2, cos(arg)
      for (int k = L.g; k < R; k += G) {
         const int i = j * R + k;
         const double s2 = wave[i], c2 = ol_cos(2.0 * (P.rho[k] - T.phi[j]));
         const double wi = w[i];
         J[col[0] + i] = -2.0 * c2 * sarg * wi;
         J[col[1] + i] = dal * s2 * wi;
         J[col[2] + i] = dtr * s2 * carg * wi;
      }
   }
   L.sync();
}

// numpy's pairwise sum (np.sum of a contiguous float64 array, n <= 256):
// blocks of at most 128 values with 8 partial sums, longer arrays split once
// at a multiple of 8; get(i) gives the i-th value
template <class Get> __device__ __forceinline__ double np_sum_block(Get get, int b, int n) {
   if (n < 8) {
      double s = 0.0; // numpy adds from -0.0; same value for these data
      for (int i = 0; i < n; i++)
         s += get(b + i);
      return s;
   }
   double r[8];
#pragma unroll
   for (int i = 0; i < 8; i++)
      r[i] = get(b + i);
   int i = 8;
   for (; i + 8 <= n; i += 8)
#pragma unroll
      for (int t = 0; t < 8; t++)
         r[t] += get(b + i + t);
   double s = ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
   for (; i < n; i++)
      s += get(b + i);
   return s;
}

template <class Get> __device__ __forceinline__ double np_sum(Get get, int n) {
   if (n <= 128)
      return np_sum_block(get, 0, n);
   int n2 = n / 2;
   n2 -= n2 % 8;
   return np_sum_block(get, 0, n2) + np_sum_block(get, n2, n - n2);
}

// np.sum(np.square(r)) of n values, 8 <= n <= 256, by the pixel's lanes: numpy's
// 8 partial sums are spread over them.
template <int G> __device__ __forceinline__ double np_sumsq_block(const Lanes<G> &L,
                                                                  const double *r, int n) {
   constexpr int kOwn = G >= 8 ? 1 : 8 / G; // partial sums of a lane: g, g + G, ...
   double a[kOwn];
#pragma unroll
   for (int o = 0; o < kOwn; o++) {
      const double v = r[(L.g + o * G) & 7];
      a[o] = v * v;
   }
   int i = 8;
   for (; i + 8 <= n; i += 8)
#pragma unroll
      for (int o = 0; o < kOwn; o++) {
         const double v = r[i + ((L.g + o * G) & 7)];
         a[o] += v * v;
      }
   // ((r0 + r1) + (r2 + r3)) + ((r4 + r5) + (r6 + r7)): sums of two commute
#pragma unroll
   for (int o = 0; o < kOwn; o++) {
      a[o] = a[o] + __shfl_xor_sync(L.mask, a[o], 1);
      a[o] = a[o] + __shfl_xor_sync(L.mask, a[o], 2);
   }
   double s = kOwn == 2 ? a[0] + a[kOwn - 1] : a[0] + __shfl_xor_sync(L.mask, a[0], 4);
   for (; i < n; i++)
      s += r[i] * r[i];
   return s;
}

template <int G> __device__ __forceinline__ double np_sumsq(const Lanes<G> &L, const double *r,
                                                            int n) {
   static_assert(G == 1 || G == 4 || G >= 8, "the partial sums pair up within the lanes");
   if constexpr (G == 1)
      return np_sum([&](int i) { return r[i] * r[i]; }, n);
   if (n <= 128)
      return np_sumsq_block(L, r, n);
   int n2 = n / 2;
   n2 -= n2 % 8;
   return np_sumsq_block(L, r, n2) + np_sumsq_block(L, r + n2, n - n2);
}

// sum over i of a[i] b[i], sequential: MINPACK's enorm (a = b; every value of
// these fits lies in its unscaled range or is zero), qrfac's and qtf's column
// products.  By one lane; lanes may run different ones side by side.
__device__ __noinline__ double seq_dot(const double *a, const double *b, int n) {
   double s = 0.0;
   for (int i = 0; i < n; i++)
      s = s + a[i] * b[i];
   return s;
}

// The same of one pair of vectors by all lanes: the products first, into t.
template <int G>
__device__ __noinline__ double lanes_dot(const double *a, const double *b, int n, double *t) {
   if (G == 1)
      return seq_dot(a, b, n);
   const Lanes<G> L;
   for (int i = L.g; i < n; i += G)
      t[i] = a[i] * b[i];
   L.sync();
   double s = 0.0;
   for (int i = 0; i < n; i++)
      s = s + t[i];
   L.sync();
   return s;
}

// x^3 rounded once, as numpy's x**3 (pow) gives it: the exact cube as a
// double-double (Dekker's product through fma) rounded to the nearest double
__device__ __forceinline__ double cube_rn(double x) {
   const double p = x * x;
   const double pe = fma(x, x, -p); // x^2 = p + pe exactly
   const double h = p * x;
   const double he = fma(p, x, -h); // p x = h + he exactly
   return h + (he + pe * x);
}

// ----------------------------------------------------------------------------
// MINPACK's Levenberg-Marquardt (lmdif with a forward-difference Jacobian,
// lmder with the reference's own Jacobian in grad_mode), restated from the
// published algorithm (More, "The Levenberg-Marquardt algorithm:
// implementation and theory", 1978; MINPACK-1, 1980) as
// scipy.optimize.leastsq runs it for the reference (_ROFL_with_jacobi.py:
// 472-486): ftol = xtol = 1.49012e-8, gtol = 0, maxfev = 150, factor 100,
// automatic scaling, epsfcn = machine epsilon.  The m x 3 Jacobian and the
// residual vectors are the pixel's lanes'; the loops over the measurements
// run in MINPACK's order, so the iterates differ from the reference's only
// where CUDA's FP64 trigonometry rounds differently from the reference's
// numpy (a last-bit difference in some evaluations, which MINPACK's
// stopping tests can turn into a different last step).
// ----------------------------------------------------------------------------
constexpr double kMpEps = 2.220446049250313e-16;     // machine epsilon (dpmpar(1))
constexpr double kMpDwarf = 2.2250738585072014e-308; // smallest normal (dpmpar(2))
constexpr double kMpTol = 1.49012e-08;               // leastsq's ftol and xtol
constexpr int kMpMaxFev = 150;

__device__ __forceinline__ double mp_norm3(const double v[3]) {
   double s = 0.0;
   s = s + v[0] * v[0];
   s = s + v[1] * v[1];
   s = s + v[2] * v[2];
   return sqrt(s);
}

// qrsolv: solves (R; D) x = (qtb; 0) in the least-squares sense for the
// 3 x 3 upper triangular R of a pivoted QR (ipvt) and diagonal D; r's
// strict lower triangle receives S's, sdiag its diagonal
__device__ __noinline__ void mp_qrsolv(double r[3][3], const int ipvt[3], const double dg[3],
                          const double qtb[3], double x[3], double sdiag[3]) {
   double wa[3];
   for (int j = 0; j < 3; j++) {
      for (int i = j; i < 3; i++)
         r[i][j] = r[j][i];
      x[j] = r[j][j];
      wa[j] = qtb[j];
   }
   for (int j = 0; j < 3; j++) {
      const int l = ipvt[j];
      if (dg[l] != 0.0) {
         for (int k = j; k < 3; k++)
            sdiag[k] = 0.0;
         sdiag[j] = dg[l];
         double qtbpj = 0.0;
         for (int k = j; k < 3; k++) {
            if (sdiag[k] == 0.0)
               continue;
            double sn, cs;
            if (fabs(r[k][k]) < fabs(sdiag[k])) {
               const double cotan = r[k][k] / sdiag[k];
               sn = 0.5 / sqrt(0.25 + 0.25 * (cotan * cotan));
               cs = sn * cotan;
            } else {
               const double tn = sdiag[k] / r[k][k];
               cs = 0.5 / sqrt(0.25 + 0.25 * (tn * tn));
               sn = cs * tn;
            }
            r[k][k] = cs * r[k][k] + sn * sdiag[k];
            const double temp = cs * wa[k] + sn * qtbpj;
            qtbpj = -sn * wa[k] + cs * qtbpj;
            wa[k] = temp;
            for (int i = k + 1; i < 3; i++) {
               const double t2 = cs * r[i][k] + sn * sdiag[i];
               sdiag[i] = -sn * r[i][k] + cs * sdiag[i];
               r[i][k] = t2;
            }
         }
      }
      sdiag[j] = r[j][j];
      r[j][j] = x[j];
   }
   int nsing = 3;
   for (int j = 0; j < 3; j++) {
      if (sdiag[j] == 0.0 && nsing == 3)
         nsing = j;
      if (nsing < 3)
         wa[j] = 0.0;
   }
   for (int j = nsing - 1; j >= 0; j--) {
      double sum = 0.0;
      for (int i = j + 1; i < nsing; i++)
         sum = sum + r[i][j] * wa[i];
      wa[j] = (wa[j] - sum) / sdiag[j];
   }
   for (int j = 0; j < 3; j++)
      x[ipvt[j]] = wa[j];
}

// lmpar: the Levenberg-Marquardt parameter par and step x for trust radius
// delta (r: R in its upper triangle; its lower triangle is scratch)
__device__ __noinline__ void mp_lmpar(double r[3][3], const int ipvt[3], const double dg[3],
                         const double qtb[3], double delta, double &par, double x[3]) {
   double wa1[3], wa2[3], sdiag[3];
   int nsing = 3;
   for (int j = 0; j < 3; j++) {
      wa1[j] = qtb[j];
      if (r[j][j] == 0.0 && nsing == 3)
         nsing = j;
      if (nsing < 3)
         wa1[j] = 0.0;
   }
   for (int j = nsing - 1; j >= 0; j--) {
      wa1[j] = wa1[j] / r[j][j];
      const double temp = wa1[j];
      for (int i = 0; i < j; i++)
         wa1[i] = wa1[i] - r[i][j] * temp;
   }
   for (int j = 0; j < 3; j++)
      x[ipvt[j]] = wa1[j];
   int iter = 0;
   for (int j = 0; j < 3; j++)
      wa2[j] = dg[j] * x[j];
   double dxnorm = mp_norm3(wa2);
   double fp = dxnorm - delta;
   if (fp <= 0.1 * delta) {
      par = 0.0;
      return;
   }
   double parl = 0.0;
   if (nsing >= 3) {
      for (int j = 0; j < 3; j++) {
         const int l = ipvt[j];
         wa1[j] = dg[l] * (wa2[l] / dxnorm);
      }
      for (int j = 0; j < 3; j++) {
         double sum = 0.0;
         for (int i = 0; i < j; i++)
            sum = sum + r[i][j] * wa1[i];
         wa1[j] = (wa1[j] - sum) / r[j][j];
      }
      const double temp = mp_norm3(wa1);
      parl = ((fp / delta) / temp) / temp;
   }
   for (int j = 0; j < 3; j++) {
      double sum = 0.0;
      for (int i = 0; i <= j; i++)
         sum = sum + r[i][j] * qtb[i];
      wa1[j] = sum / dg[ipvt[j]];
   }
   const double gnorm = mp_norm3(wa1);
   double paru = gnorm / delta;
   if (paru == 0.0)
      paru = kMpDwarf / fmin(delta, 0.1);
   par = fmax(par, parl);
   par = fmin(par, paru);
   if (par == 0.0)
      par = gnorm / dxnorm;
   for (;;) {
      iter++;
      if (par == 0.0)
         par = fmax(kMpDwarf, 0.001 * paru);
      const double temp = sqrt(par);
      for (int j = 0; j < 3; j++)
         wa1[j] = temp * dg[j];
      mp_qrsolv(r, ipvt, wa1, qtb, x, sdiag);
      for (int j = 0; j < 3; j++)
         wa2[j] = dg[j] * x[j];
      dxnorm = mp_norm3(wa2);
      const double fp_old = fp;
      fp = dxnorm - delta;
      if (fabs(fp) <= 0.1 * delta || (parl == 0.0 && fp <= fp_old && fp_old < 0.0) ||
          iter == 10)
         break;
      for (int j = 0; j < 3; j++) {
         const int l = ipvt[j];
         wa1[j] = dg[l] * (wa2[l] / dxnorm);
      }
      for (int j = 0; j < 3; j++) {
         wa1[j] = wa1[j] / sdiag[j];
         const double t2 = wa1[j];
         for (int i = j + 1; i < 3; i++)
            wa1[i] = wa1[i] - r[i][j] * t2;
      }
      const double t3 = mp_norm3(wa1);
      const double parc = ((fp / delta) / t3) / t3;
      if (fp > 0.0)
         parl = fmax(parl, par);
      if (fp < 0.0)
         paru = fmin(paru, par);
      par = fmax(parl, par + parc);
   }
}

// A pixel's arrays in shared memory: measurements c, weights w, residuals F and
// waves S of two points, the Jacobian J (also a third wave's place) and
// products t.
template <int MAXM> struct PixelArrays {
   double c[MAXM], w[MAXM], F[2 * MAXM], S[2 * MAXM], J[3 * MAXM], t[MAXM];
   double cos2[3][5]; // of the points of S[0], S[1] and of a difference
   double trans[5];
   TiltValues T;
};

// The fit for one pixel (G lanes, which all hold the same scalars): x in: the
// start point, out: the last accepted point; A.F + cur * MAXM holds its
// residuals on return.  Returns MINPACK's info (5: evaluation budget spent);
// nfev counts as MINPACK counts (lmdif: 1 + 3 per Jacobian + 1 per trial step;
// lmder: 1 + 1 per trial step).
template <int MAXM, int G>
__device__ int mp_fit(const RoflParams &P, PixelArrays<MAXM> &A, int M, double x[3], int &cur,
                      int &nfev) {
   const Lanes<G> L;
   const double epsfd = sqrt(kMpEps); // sqrt(max(epsfcn, epsmch)), epsfcn = eps
   double *J = A.J;
   cur = 0;
   px_waves<G>(P, x[0], x[1], nullptr, A.S, A.T, A.cos2[0]);
   px_residuals<G>(P, A.c, A.w, A.S, A.cos2[0], A.T, x[2], A.F);
   nfev = 1;
   double fnorm = sqrt(lanes_dot<G>(A.F, A.F, M, A.t));
   double par = 0.0, delta = 0.0, xnorm = 0.0;
   double dg[3] = {1.0, 1.0, 1.0};
   int iter = 1;
   for (;;) {
      double *fv = A.F + cur * MAXM, *wa4 = A.F + (1 - cur) * MAXM;
      // the Jacobian's columns, J + col[j] after the pivoting swaps
      int col[3] = {0, MAXM, 2 * MAXM};
      if (P.grad_mode) { // (T is the accepted point's: the trial's, just evaluated)
         px_jacobi<G>(P, A.w, A.S + cur * MAXM, A.T, x[2], J, col);
      } else { // fdjac2
#pragma unroll 1
         for (int j = 0; j < 3; j++) {
            const double temp = x[j];
            double h = epsfd * fabs(temp);
            if (h == 0.0)
               h = epsfd;
            double *Jj = J + col[j];
            const double *Sc = A.S + cur * MAXM, *wave = Sc, *cc = A.cos2[cur];
            if (j < 2) { // (the waves take column 2's place, not yet filled)
               double *Sp = J + col[2];
               px_waves<G>(P, j == 0 ? temp + h : x[0], j == 1 ? temp + h : x[1],
                           j == 1 ? Sc : nullptr, Sp, A.T, A.cos2[2]);
               wave = Sp;
               cc = A.cos2[2];
            }
            px_residuals<G>(P, A.c, A.w, wave, cc, A.T, j == 2 ? temp + h : x[2], Jj);
            const Divisor by_h(h);
            for (int i = L.g; i < M; i += G)
               Jj[i] = by_h.quotient(Jj[i] - fv[i]);
         }
         L.sync();
         nfev += 3;
      }
      // qrfac with column pivoting; the columns' norms side by side
      double acnorm[3], rdiag[3], wa[3];
      int ipvt[3] = {0, 1, 2};
      {
         const double *a = J + min(L.g, 2) * MAXM;
         const double norm = sqrt(seq_dot(a, a, M));
#pragma unroll
         for (int j = 0; j < 3; j++) {
            acnorm[j] = L.from(norm, j);
            if (G == 1 && j)
               acnorm[j] = sqrt(seq_dot(J + j * MAXM, J + j * MAXM, M));
            rdiag[j] = wa[j] = acnorm[j];
         }
      }
#pragma unroll
      for (int j = 0; j < 3; j++) {
         int kmax = j;
#pragma unroll
         for (int k = j; k < 3; k++)
            if (rdiag[k] > rdiag[kmax])
               kmax = k;
#pragma unroll
         for (int k = j + 1; k < 3; k++)
            if (k == kmax) {
               const int tc = col[j];
               col[j] = col[k];
               col[k] = tc;
               rdiag[k] = rdiag[j];
               wa[k] = wa[j];
               const int t = ipvt[j];
               ipvt[j] = ipvt[k];
               ipvt[k] = t;
            }
         double *aj = J + col[j];
         // (the first column is as it was for acnorm)
         double ajnorm =
             j == 0 ? (ipvt[0] == 0 ? acnorm[0] : ipvt[0] == 1 ? acnorm[1] : acnorm[2])
                    : sqrt(lanes_dot<G>(aj + j, aj + j, M - j, A.t));
         if (ajnorm != 0.0) {
            if (aj[j] < 0.0)
               ajnorm = -ajnorm;
            L.sync(); // every lane has read aj[j]
            const Divisor by_norm(ajnorm);
            for (int i = j + L.g; i < M; i += G) {
               const double q = by_norm.quotient(aj[i]);
               aj[i] = i == j ? q + 1.0 : q;
            }
            L.sync();
            double sums[2] = {0.0, 0.0}; // of columns j + 1, j + 2
            if (j == 0) {
               const double sum = seq_dot(aj, J + ((L.g & 1) ? col[2] : col[1]), M);
               sums[0] = L.from(sum, 0);
               sums[1] = G == 1 ? seq_dot(aj, J + col[2], M) : L.from(sum, 1);
            } else if (j == 1) {
               sums[0] = lanes_dot<G>(aj + 1, J + col[2] + 1, M - 1, A.t);
            }
#pragma unroll
            for (int k = j + 1; k < 3; k++) {
               double *ak = J + col[k];
               const double temp = sums[k - j - 1] / aj[j];
               for (int i = j + L.g; i < M; i += G)
                  ak[i] = ak[i] - temp * aj[i];
            }
            L.sync();
#pragma unroll
            for (int k = j + 1; k < 3; k++)
               if (rdiag[k] != 0.0) {
                  const double *ak = J + col[k];
                  const double t2 = ak[j] / rdiag[k];
                  rdiag[k] = rdiag[k] * sqrt(fmax(0.0, 1.0 - t2 * t2));
                  const double q2 = rdiag[k] / wa[k];
                  if (0.05 * (q2 * q2) <= kMpEps) {
                     rdiag[k] = sqrt(seq_dot(ak + j + 1, ak + j + 1, M - j - 1));
                     wa[k] = rdiag[k];
                  }
               }
         }
         rdiag[j] = -ajnorm;
      }
      if (iter == 1) {
#pragma unroll
         for (int j = 0; j < 3; j++)
            dg[j] = acnorm[j] == 0.0 ? 1.0 : acnorm[j];
         const double w3[3] = {dg[0] * x[0], dg[1] * x[1], dg[2] * x[2]};
         xnorm = mp_norm3(w3);
         delta = 100.0 * xnorm;
         if (delta == 0.0)
            delta = 100.0;
      }
      // (Q^T fvec) in its first 3 rows (wa4 is the residual buffer's free
      // half), and R's diagonal restored
      double qtf[3];
      for (int i = L.g; i < M; i += G)
         wa4[i] = fv[i];
      L.sync();
#pragma unroll
      for (int j = 0; j < 3; j++) {
         double *aj = J + col[j];
         const double ajj = aj[j];
         if (ajj != 0.0) {
            const double sum = lanes_dot<G>(aj + j, wa4 + j, M - j, A.t);
            const double temp = -sum / ajj;
            for (int i = j + L.g; i < M; i += G)
               wa4[i] = wa4[i] + aj[i] * temp;
         }
         L.sync();
         if (L.g == 0)
            aj[j] = rdiag[j];
         qtf[j] = wa4[j];
      }
      L.sync();
      double R[3][3];
#pragma unroll
      for (int j = 0; j < 3; j++)
#pragma unroll
         for (int i = 0; i < 3; i++)
            R[i][j] = i <= j ? J[col[j] + i] : 0.0;
      double gnorm = 0.0;
      if (fnorm != 0.0) {
#pragma unroll
         for (int j = 0; j < 3; j++) {
            const int l = ipvt[j];
            const double an = l == 0 ? acnorm[0] : (l == 1 ? acnorm[1] : acnorm[2]);
            if (an != 0.0) {
               double sum = 0.0;
#pragma unroll
               for (int i = 0; i <= j; i++)
                  sum = sum + R[i][j] * (qtf[i] / fnorm);
               gnorm = fmax(gnorm, fabs(sum / an));
            }
         }
      }
      if (gnorm <= 0.0) // gtol = 0
         return 4;
#pragma unroll
      for (int j = 0; j < 3; j++)
         dg[j] = fmax(dg[j], acnorm[j]);
      // inner loop: trial steps until one is accepted
      for (;;) {
         double rr[3][3];
#pragma unroll
         for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++)
               rr[i][j] = R[i][j];
         double p[3];
         mp_lmpar(rr, ipvt, dg, qtf, delta, par, p);
         double w1[3], w2[3], w3[3];
#pragma unroll
         for (int j = 0; j < 3; j++) {
            w1[j] = -p[j];
            w2[j] = x[j] + w1[j];
            w3[j] = dg[j] * w1[j];
         }
         const double pnorm = mp_norm3(w3);
         if (iter == 1)
            delta = fmin(delta, pnorm);
         px_waves<G>(P, w2[0], w2[1], nullptr, A.S + (1 - cur) * MAXM, A.T, A.cos2[1 - cur]);
         px_residuals<G>(P, A.c, A.w, A.S + (1 - cur) * MAXM, A.cos2[1 - cur], A.T, w2[2], wa4);
         nfev++;
         const double fnorm1 = sqrt(lanes_dot<G>(wa4, wa4, M, A.t));
         double actred = -1.0;
         if (0.1 * fnorm1 < fnorm) {
            const double t = fnorm1 / fnorm;
            actred = 1.0 - t * t;
         }
#pragma unroll
         for (int j = 0; j < 3; j++) {
            w3[j] = 0.0;
            const int l = ipvt[j];
            const double temp = l == 0 ? w1[0] : (l == 1 ? w1[1] : w1[2]);
#pragma unroll
            for (int i = 0; i <= j; i++)
               w3[i] = w3[i] + R[i][j] * temp;
         }
         const double temp1 = mp_norm3(w3) / fnorm;
         const double temp2 = (sqrt(par) * pnorm) / fnorm;
         const double prered = temp1 * temp1 + (temp2 * temp2) / 0.5;
         const double dirder = -(temp1 * temp1 + temp2 * temp2);
         const double ratio = prered != 0.0 ? actred / prered : 0.0;
         if (ratio <= 0.25) {
            double temp = actred >= 0.0 ? 0.5 : 0.5 * dirder / (dirder + 0.5 * actred);
            if (0.1 * fnorm1 >= fnorm || temp < 0.1)
               temp = 0.1;
            delta = temp * fmin(delta, pnorm / 0.1);
            par = par / temp;
         } else if (par == 0.0 || ratio >= 0.75) {
            delta = pnorm / 0.5;
            par = 0.5 * par;
         }
         if (ratio >= 1e-4) { // accepted: the trial residuals become fvec
#pragma unroll
            for (int j = 0; j < 3; j++)
               x[j] = w2[j];
            const double w5[3] = {dg[0] * x[0], dg[1] * x[1], dg[2] * x[2]};
            xnorm = mp_norm3(w5);
            cur = 1 - cur;
            fnorm = fnorm1;
            iter++;
         }
         int info = 0;
         const bool fsmall = fabs(actred) <= kMpTol && prered <= kMpTol && 0.5 * ratio <= 1.0;
         if (fsmall)
            info = 1;
         if (delta <= kMpTol * xnorm)
            info = fsmall ? 3 : 2;
         if (info != 0)
            return info;
         if (nfev >= kMpMaxFev)
            info = 5;
         if (fabs(actred) <= kMpEps && prered <= kMpEps && 0.5 * ratio <= 1.0)
            info = 6; // tolerances too small (6, 7, 8)
         if (delta <= kMpEps * xnorm)
            info = 7;
         if (gnorm <= kMpEps)
            info = 8;
         if (info != 0)
            return info;
         if (ratio >= 1e-4)
            break; // a new Jacobian at the accepted point
         // rejected: wa4 (the free half) is scratch again
      }
   }
}

// One warp per CTA, 32 / G pixels at a time, taken from a counter by the warp
// (its pixels start together, so that their phases coincide).  MAXR bounds
// n_rot.  The arrays of the pixels (10 x 5 MAXR doubles each) live in shared
// memory, 33 KB per warp with G = 4 and 10 rotations, 26 KB with 16 and 32; with
// a lane per pixel in its local memory, interleaved across the warp and cached
// in L1 (held to 80 registers: 24 warps per SM).
// With a mask the pixels are those of rofl_select's list, whose length n the
// kernel finds in status[2]; it is one of those launched for several ranges of
// n, and the others return at once.
template <int MAXR, int G>
__global__ void __launch_bounds__(32, G == 1 ? 24 : 0)
rofl_fit(const double *__restrict__ data, int64_t n_pix, const int64_t *__restrict__ list,
         int64_t n_least, int64_t n_end, const RoflParams P, double *__restrict__ out,
         unsigned long long *__restrict__ status) {
   constexpr int MAXM = 5 * MAXR, kPixels = 32 / G;
   extern __shared__ __align__(16) unsigned char s_arrays[];
   PixelArrays<G == 1 ? MAXM : 1> own; // (local memory)
   const int lane = threadIdx.x & 31, R = P.n_rot, M = 5 * R;
   PixelArrays<MAXM> &A =
       G == 1 ? reinterpret_cast<PixelArrays<MAXM> &>(own)
              : reinterpret_cast<PixelArrays<MAXM> *>(s_arrays)[lane / G];
   const Lanes<G> L;
   const int64_t n = list ? (int64_t)status[2] : n_pix;
   if (n < n_least || n >= n_end)
      return;
   for (;;) {
      unsigned long long first = 0;
      if (lane == 0)
         first = atomicAdd(&status[1], (unsigned long long)kPixels);
      first = __shfl_sync(0xFFFFFFFFu, first, 0);
      if (first >= (unsigned long long)n)
         break;
      const int64_t q = (int64_t)first + lane / G;
      if (q < n) {
         const int64_t p = list ? list[q] : q;
         // tilt t, rotation k of pixel p: data[(t * n_pix + p) * R + k]
         for (int t = L.g; t < 5; t += G) {
            const double *d = data + (t * n_pix + p) * R;
            A.trans[t] = np_sum([&](int k) { return d[k]; }, R) / R; // np.mean
         }
         L.sync();
         // epa.direction of the untilted series (epa.py:48-77) + dir_offset
         double phi0;
         {
            const double *d0 = data + p * R, *wave = (L.g & 1) ? P.rho2c : P.rho2s;
            const double sum = np_sum([&](int k) { return d0[k] * wave[k]; }, R);
            const double cosine = G == 1 ? np_sum([&](int k) { return d0[k] * P.rho2c[k]; }, R)
                                         : L.from(sum, 1);
            const double a1 = 2.0 * L.from(sum, 0) / R, b1 = 2.0 * cosine / R;
            phi0 = pymod(0.5 * atan2(-b1, a1) + M_PI, M_PI) + P.dir_offset;
         }
         // _calc_centered_vals (:47-61)
#pragma unroll 1
         for (int t = 0; t < 5; t++) {
            const double *d = data + (t * n_pix + p) * R;
            const double tr = A.trans[t], tr2 = tr * tr, tr3r = cube_rn(tr) * R;
            for (int k = L.g; k < R; k += G) {
               const double v = d[k];
               A.c[t * R + k] = v / tr - 1.0;
               A.w[t * R + k] = 1.0 / sqrt(P.gain * (v / tr2 + v * v / tr3r));
            }
         }
         L.sync();
         // start grid (:261-328): inclination outer, t_rel inner, the first
         // minimum of the pairwise row sums (np.argmin: a NaN wins)
         double x[3] = {phi0, P.incl[0], P.trel[0]};
         {
            double best = INFINITY;
#pragma unroll 1
            for (int a = 0; a < 6; a++) {
               px_waves<G>(P, phi0, P.incl[a], a ? A.S : nullptr, A.S, A.T, A.cos2[0]);
#pragma unroll 1
               for (int t = 0; t < 6; t++) {
                  px_residuals<G>(P, A.c, A.w, A.S, A.cos2[0], A.T, P.trel[t], A.F);
                  const double cost = np_sumsq(L, A.F, M);
                  L.sync();
                  if (cost < best || (isnan(cost) && !isnan(best))) {
                     best = cost;
                     x[1] = P.incl[a];
                     x[2] = P.trel[t];
                  }
               }
            }
         }
         // MINPACK's fit, as scipy.optimize.leastsq runs it for the reference
         int n_fev = 0, cur = 0;
         const int info = mp_fit<MAXM, G>(P, A, M, x, cur, n_fev);
         if (info == 5 && L.g == 0)
            atomicAdd(&status[0], 1ull); // evaluation budget reached
         const double cost = np_sumsq(L, A.F + cur * MAXM, M); // np.sum(np.square)
         L.sync();
         // result (:488-520): fold, |t_rel|, covariance from the reference's
         // Jacobian at the folded point and its own 3x3 inverse
         double d = x[0], a = x[1];
         symmetrize(d, a);
         const double t = fabs(x[2]);
         const double sigma_sq = cost / (double)(M - 3);
         const int col[3] = {0, MAXM, 2 * MAXM};
         px_waves<G>(P, d, a, nullptr, A.S, A.T, A.cos2[0]);
         px_jacobi<G>(P, A.w, A.S, A.T, t, A.J, col);
         // the six sums of products, a lane each
         double s[6], own[(6 + G - 1) / G];
#pragma unroll
         for (int o = 0; o < (6 + G - 1) / G; o++) {
            const int e = min(L.g + o * G, 5); // (0 0) (0 1) (0 2) (1 1) (1 2) (2 2)
            const int i = e < 3 ? 0 : e < 5 ? 1 : 2, j = e < 3 ? e : e < 5 ? e - 2 : 2;
            own[o] = seq_dot(A.J + i * MAXM, A.J + j * MAXM, M);
         }
#pragma unroll
         for (int e = 0; e < 6; e++)
            s[e] = L.from(own[e / G], e % G);
         const double mm[9] = {s[0], s[1], s[2], s[1], s[3], s[4], s[2], s[4], s[5]};
         // _invertmatrix (:14-44) with the reference's determinant expression
         // (its fourth term is m20 * m12, without a third factor)
         const double det = mm[0] * mm[4] * mm[8] + mm[3] * mm[7] * mm[2] + mm[6] * mm[5] -
                            mm[0] * mm[7] * mm[5] - mm[6] * mm[4] * mm[2] - mm[3] * mm[1] * mm[8];
         const double i00 = (mm[4] * mm[8] - mm[5] * mm[7]) / det;
         const double i11 = (mm[0] * mm[8] - mm[2] * mm[6]) / det;
         const double i22 = (mm[0] * mm[4] - mm[1] * mm[3]) / det;
         if (L.g == 0) {
            double *o = out + 8 * p;
            o[0] = d;
            o[1] = a;
            o[2] = t;
            o[3] = sqrt(fabs(i00 * sigma_sq));
            o[4] = sqrt(fabs(i11 * sigma_sq));
            o[5] = sqrt(fabs(i22 * sigma_sq));
            o[6] = cost;
            o[7] = (double)n_fev;
         }
      }
      __syncwarp();
   }
}

// The unmasked pixels, in any order, and their number; NaN for the others.
__global__ void __launch_bounds__(256)
rofl_select(const unsigned char *__restrict__ mask, int64_t n_pix, int64_t *__restrict__ list,
            double *__restrict__ out, unsigned long long *__restrict__ status) {
   const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
   const bool on = p < n_pix && mask[p];
   const unsigned m = __ballot_sync(0xFFFFFFFFu, on);
   const int lane = threadIdx.x & 31;
   unsigned long long at = 0;
   if (lane == 0 && m)
      at = atomicAdd(&status[2], (unsigned long long)__popc(m));
   at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(m & ((1u << lane) - 1u));
   if (on)
      list[at] = p;
   else if (p < n_pix)
      for (int e = 0; e < 8; e++)
         out[8 * p + e] = nan("");
}

// Lanes per pixel.  Up to kRoflFewPixels 16: four warps per SM of two pixels
// each, which an SM's FP64 unit runs nearly as fast as one, so only the length
// of a pixel's chain counts.  From one_lane_pixels on 1: the map keeps every SM
// busy for many times the longest chain, so only the number of instructions
// counts.  Between them 4, up to 10 rotations (GB300, forward differences, 9
// rotations):
//   30 x 20     16: 1.70 ms   4:   2.72 ms   1:  6.3 ms
//   77 x 77     16: 4.94      4:   4.68      1:  9.8
//   160 x 150   16: 18.2      4:  13.8       1: 18.0
//   320 x 320                 4:  44.0       1: 35.7
//   512 x 512                 4: 109         1: 84.0
// With more rotations four lanes per pixel leave an SM two warps (105 KB of
// arrays each) and lose to 16 from 6,000 pixels on; and one lane wins sooner,
// the instructions that 16 lanes repeat being in proportion to the pixels, the
// longest chain to the rotations (ms, two maps of faster and slower fits; the
// thread per pixel before all of these 16.1 / 20.4, 23.6 / 26.0, 56.5 / 61.1 for
// 18 rotations and 6,000 / 12,100, 24,000, 79,000 pixels):
//   11 rotations   12,000: 16  9.7 / 10.9   1  7.3 / 14.1   24,000: 18.9 / 21.0    9.0 / 16.3
//   18             12,000:    10.8 / 11.8     11.5 / 15.4   24,000: 20.8 / 22.8   14.7 / 19.8
//   18             79,000:    67.4 / 72.8     33.7 / 43.8
//   32             24,000:    26.3 / 28.7     28.9 / 32.1   36,000: 38.8 / 41.8   33.8 / 38.2
// In grad_mode the chain is ten times as long: 16 and 1 lanes level at 79,000
// pixels of 11 rotations (219 and 222 ms), 16 ahead of 1 with more.
// Masked pixels do not count: a warp of one-lane pixels idles on those it meets
// (90% of 24,000 pixels masked, 18 rotations: 12.4 ms so, 4.2 with 16 lanes).
constexpr int64_t kRoflFewPixels = 1216, kRoflManyPixels = 80000;

static int64_t one_lane_pixels(const RoflParams &P) {
   return P.n_rot <= kRoflSmallRot || P.grad_mode ? kRoflManyPixels : 1000 * P.n_rot;
}

// As many warps as are resident (the pixels are taken from the counter), fewer
// for small maps; for n_least <= pixels < n_end.
template <int MAXR, int G>
static int launch_rofl(const double *d_data, int64_t n_pix, const int64_t *d_list, int64_t n_least,
                       int64_t n_end, const RoflParams &P, double *d_out,
                       unsigned long long *status, cudaStream_t st) {
   if (n_least >= n_end || n_pix < n_least || (!d_list && n_pix >= n_end))
      return FPGB_OK;
   constexpr int kPixels = 32 / G;
   constexpr int kBytes = G == 1 ? 0 : kPixels * (int)sizeof(PixelArrays<5 * MAXR>);
   int dev = 0, sms = 0, per_sm = 0;
   FPGB_CUDA_TRY(cudaGetDevice(&dev));
   FPGB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
   FPGB_CUDA_TRY(cudaFuncSetAttribute(rofl_fit<MAXR, G>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes));
   FPGB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, rofl_fit<MAXR, G>, 32,
                                                               kBytes));
   const int64_t most = std::min(n_pix, n_end - 1);
   const int64_t blocks = std::max<int64_t>(
       1, std::min<int64_t>((most + kPixels - 1) / kPixels, (int64_t)sms * std::max(per_sm, 1)));
   rofl_fit<MAXR, G><<<(unsigned)blocks, 32, kBytes, st>>>(d_data, n_pix, d_list, n_least, n_end,
                                                           P, d_out, status);
   FPGB_CUDA_TRY(cudaGetLastError());
   return FPGB_OK;
}

} // namespace fpgb

using namespace fpgb;

extern "C" {

int fpgb_rofl_device(const double *d_data, int64_t n_pix, int64_t n_rot, double tilt_angle,
                     double gain, double dir_offset, int grad_mode, const unsigned char *d_mask,
                     double *d_out, int64_t *n_unconverged, void *stream) {
   if (!d_data || !d_out || n_pix < 0 || n_rot <= 3 || n_rot > kRoflMaxRot) {
      set_error("rofl: null buffer, n_pix < 0, or n_rot outside 4..%d", kRoflMaxRot);
      return FPGB_EINVAL;
   }
   if (!(gain > 1.0)) {
      set_error("rofl gain <= 1");
      return FPGB_EINVAL;
   }
   RoflParams P;
   std::memset(&P, 0, sizeof P);
   P.n_rot = (int)n_rot;
   P.inv_rot = (1 << 16) / P.n_rot + 1;
   P.grad_mode = grad_mode ? 1 : 0;
   P.tau = tilt_angle;
   P.gain = gain;
   P.dir_offset = dir_offset;
   P.cos_tau = std::cos(tilt_angle);
   // numpy.linspace(start, stop, num): start + k * ((stop - start) / div)
   for (int k = 0; k < P.n_rot; k++) {
      P.rho[k] = (double)k * (M_PI / (double)n_rot) + dir_offset;
      const double r2 = 2.0 * ((double)k * (M_PI / (double)n_rot));
      P.rho2s[k] = std::sin(r2);
      P.rho2c[k] = std::cos(r2);
   }
   for (int t = 0; t < 4; t++) { // _create_rotation_matrix (:77-96)
      const double psi = (double)t * (2.0 * M_PI / 4.0);
      const double c = std::cos(psi), s = std::sin(psi), ct = std::cos(tilt_angle),
                   st = std::sin(tilt_angle);
      double *M = P.mat[t];
      M[0] = ct * c * c + s * s;
      M[1] = (ct - 1) * s * c;
      M[2] = c * st;
      M[3] = (ct - 1) * s * c;
      M[4] = ct * s * s + c * c;
      M[5] = s * st;
      M[6] = -c * st;
      M[7] = -s * st;
      M[8] = ct;
   }
   for (int k = 0; k < 6; k++) { // linspace(-pi/2, pi/2, 8)[1:-1], linspace(0, .9, 8)[1:-1]
      P.incl[k] = (double)(k + 1) * (M_PI / 7.0) + (-M_PI / 2.0);
      P.trel[k] = (double)(k + 1) * (0.9 / 7.0);
   }
   cudaStream_t st = as_stream(stream);
   void *w = nullptr;
   FPGB_TRY(pool_get(kSlotCounters, sizeof(unsigned long long) * kCounterWords, &w, st));
   auto *status = static_cast<unsigned long long *>(w);
   // status[0]: pixels at the evaluation limit, [1]: next pixel, [2]: unmasked ones
   FPGB_CUDA_TRY(cudaMemsetAsync(status, 0, 3 * sizeof(unsigned long long), st));
   if (n_pix > 0) {
      int64_t *list = nullptr;
      if (d_mask) {
         void *l = nullptr;
         FPGB_TRY(pool_get(kSlotStaging, sizeof(int64_t) * (size_t)n_pix, &l, st));
         list = static_cast<int64_t *>(l);
         rofl_select<<<(unsigned)((n_pix + 255) / 256), 256, 0, st>>>(d_mask, n_pix, list, d_out,
                                                                     status);
         FPGB_CUDA_TRY(cudaGetLastError());
      }
      const int64_t one = one_lane_pixels(P), none = INT64_MAX;
      if (P.n_rot <= kRoflSmallRot) {
         const int64_t few = kRoflFewPixels + 1;
         FPGB_TRY((launch_rofl<kRoflSmallRot, 16>(d_data, n_pix, list, 0, few, P, d_out, status,
                                                  st)));
         FPGB_TRY((launch_rofl<kRoflSmallRot, 4>(d_data, n_pix, list, few, one, P, d_out, status,
                                                 st)));
         FPGB_TRY((launch_rofl<kRoflSmallRot, 1>(d_data, n_pix, list, one, none, P, d_out, status,
                                                 st)));
      } else {
         FPGB_TRY((launch_rofl<kRoflMaxRot, 16>(d_data, n_pix, list, 0, one, P, d_out, status,
                                                st)));
         FPGB_TRY((launch_rofl<kRoflMaxRot, 1>(d_data, n_pix, list, one, none, P, d_out, status,
                                               st)));
      }
   }
   if (n_unconverged) {
      unsigned long long h = 0;
      FPGB_CUDA_TRY(cudaMemcpyAsync(&h, status, sizeof h, cudaMemcpyDeviceToHost, st));
      FPGB_CUDA_TRY(cudaStreamSynchronize(st));
      *n_unconverged = (int64_t)h;
   }
   return FPGB_OK;
}

} // extern "C"
