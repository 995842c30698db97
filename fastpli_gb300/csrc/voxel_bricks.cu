// Brick-tiled voxelizer (declarations and overview in voxel_bricks.cuh).
//
// Compiled with -fmad=false: the FP64 replay of the reference arithmetic
// (tissue_eval.cuh) must round every product and sum separately, and the
// roundings that the FP32 estimate's bound counts are the ones written out.
//
// The winner of a voxel is the segment with the smallest dist^2 (float, in
// the reference's arithmetic) among those it is inside of, ties going to the
// LAST segment: the reference's `>=` overwrite rule (generator.cpp:329-340).
// Most voxels need no exact distance to find it.  One sweep over the brick's
// segments gives every candidate an FP32 upper bound hi of its dist^2
// (sweep_dist2; hi - 2 mg is a lower bound).  A candidate whose lower bound is
// not past the thickest end of its segment lowers the voxel's 32-bit key (hi
// in quanta of 1 / scale, slot in the brick's list) with a shared-memory
// atomicMin that returns the old key.  When old and new lie within W = 2
// max(mg) of each other the order of the two may be the other way round: the
// voxel's key is marked (its lowest bit; a key that replaces it from farther
// below drops the mark, which only spoke of candidates that have lost).
//
// Every pair that could be out of order at the end marks the final key.  Let
// o hold it and c be another candidate with hi_c <= hi_o + W.  If c came
// after o, it met o's key.  If c came before o, o met some key between its
// own and c's.  So an unmarked key whose segment o the voxel is inside of
// names the winner: every other one is farther (ties are within W).
//
// Whether the voxel is inside of o, and in which of its layers, follows from
// the interval [hi - 2 mg, hi] unless that straddles a layer's boundary (the
// voxel is marked as well) or the radius changes along the segment; then o is
// evaluated with the reference's arithmetic (two-float fast path, FP64
// replay), and the voxel marked if it lies outside.
//
// voxel_bricks leaves kMarkedLabel in the marked voxels and lists them;
// voxel_marks resolves them with the reference's arithmetic: every candidate
// whose lower bound is at or below the smallest upper bound of the certain ones
// is evaluated, and the smallest float_bits(dist^2) << 32 | (0xFFFFFFFF -
// segment) wins.  A kernel of its own keeps its code and registers out of the
// sweep's.  Marked are, of the voxels inside a fiber, 0.3 to 1.4% at the joints of
// polylines, 0.01 to 0.1% otherwise, whatever a segment's length (long_part), but
// a sixth where radii change and all where fibers share their course.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "ff.cuh"
#include "fpgb_common.cuh"
#include "tissue.cuh"
#include "tissue_eval.cuh"
#include "voxel_bricks.cuh"

namespace fpgb {

// A brick's threads: small CTAs wait less at its barriers, but those of a
// volume of several bundles (31 KB of shared memory at 128 threads) then leave
// too little L1 (one bundle, 397 x 283 x 77: 202 us with 128 threads, 214 with
// 256; two, 512 x 512 x 120: 961 and 880).  As many sweep records at a time.
template <bool MULTI> constexpr int kBrickThreads = MULTI ? 256 : 128;
template <bool MULTI> constexpr unsigned kRecs = kBrickThreads<MULTI>;
static_assert(kBrickZ == 32, "the write phase maps one lane to one z of a brick row");

void tile_bricks(int64_t X, int64_t Y, int64_t Z, int32_t nb[3], int64_t *n_bricks) {
   nb[0] = (int32_t)((X + kBrickX - 1) / kBrickX);
   nb[1] = (int32_t)((Y + kBrickY - 1) / kBrickY);
   nb[2] = (int32_t)((Z + kBrickZ - 1) / kBrickZ);
   *n_bricks = (int64_t)nb[0] * nb[1] * nb[2];
}

FPGB_HD int64_t brick_range(int lo, int ext, int b, int &b0) {
   b0 = lo / b;
   return ext > 0 ? (lo + ext - 1) / b - b0 + 1 : 0;
}

int64_t segment_brick_pairs(const SegDev &S) {
   int b0;
   return brick_range(S.lo[0], S.ext[0], kBrickX, b0) * brick_range(S.lo[1], S.ext[1], kBrickY, b0) *
          brick_range(S.lo[2], S.ext[2], kBrickZ, b0);
}

// The marked voxels' records, a share of the space per launch: entries 0 and 1
// count {entries taken, records} and {full bricks}; a record is {brick, number}
// and the brick's marked voxels, four 16-bit places to an entry.  The launch's
// part of the bricks' count array becomes the directory: the records from its
// start, from its end the bricks with more marked voxels than a record takes.
// The space is what the workspace has left: the least has 32 bytes per segment,
// several times the marks of fibers of short segments; with 128 bytes per brick
// on top few long segments have room as well.
constexpr int kMarkHead = 2;

static size_t brick_list_bytes(int64_t n_bricks, int64_t n_pairs) {
   size_t w = 0;
   w += align_up(sizeof(unsigned) * (n_bricks + 1), 256); // offsets
   w += align_up(sizeof(unsigned) * std::max<int64_t>(n_bricks, 1), 256); // counts, then cursors
   w += align_up(sizeof(unsigned) * std::max<int64_t>(n_pairs, 1), 256);  // segment lists
   return w;
}

size_t brick_workspace_bytes(int64_t n_bricks, int64_t n_pairs, int64_t n_segs) {
   return brick_list_bytes(n_bricks, n_pairs) +
          align_up((size_t)std::max<int64_t>(0, 32 * n_segs - 256), 256);
}

size_t brick_workspace_more(int64_t n_bricks) { return (size_t(32) << 10) + 128 * n_bricks; }

// ---------------------------------------------------------------- binning ---
// Pair p of segment S in tile T (x slowest): its brick.
struct SegBricks {
   int bx0, by0, bz0;
   unsigned nx, ny, nz;
};

__device__ __forceinline__ SegBricks seg_bricks(const SegDev &S) {
   SegBricks r;
   r.nx = (unsigned)brick_range(S.lo[0], S.ext[0], kBrickX, r.bx0);
   r.ny = (unsigned)brick_range(S.lo[1], S.ext[1], kBrickY, r.by0);
   r.nz = (unsigned)brick_range(S.lo[2], S.ext[2], kBrickZ, r.bz0);
   return r;
}

__device__ __forceinline__ int64_t pair_brick(const SegBricks &r, const TileDev &T, unsigned p) {
   const unsigned i = p / (r.ny * r.nz), q = p - i * (r.ny * r.nz), j = q / r.nz, k = q - j * r.nz;
   return T.brick_base + ((int64_t)(r.bx0 + i) * T.nb[1] + (r.by0 + j)) * T.nb[2] + (r.bz0 + k);
}

// kBinLanes lanes share a segment's pairs: a pair is an atomic's latency, and
// a segment has about ten (15,013 segments: 21 us with one lane each).
constexpr int kBinLanes = 8;

template <bool FILL>
__global__ void brick_bin(const SegDev *__restrict__ segs, const int32_t *__restrict__ seg_tile,
                          int64_t n_segs, const TileDev *__restrict__ tiles,
                          unsigned *__restrict__ counts, const unsigned *__restrict__ offsets,
                          unsigned *__restrict__ list, int64_t n_pairs,
                          unsigned long long *__restrict__ counters) {
   for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_segs * kBinLanes;
        t += (int64_t)gridDim.x * blockDim.x) {
      const int64_t s = t / kBinLanes;
      const SegBricks r = seg_bricks(segs[s]);
      const TileDev &T = tiles[seg_tile ? seg_tile[s] : 0];
      const int64_t n = (int64_t)r.nx * r.ny * r.nz;
      for (int64_t p = t % kBinLanes; p < n; p += kBinLanes) {
         const int64_t b = pair_brick(r, T, (unsigned)p);
         const unsigned slot = atomicAdd(&counts[b], 1u);
         if (FILL) {
            const int64_t at = (int64_t)offsets[b] + slot;
            if (at < offsets[b + 1] && at < n_pairs)
               list[at] = (unsigned)s;
            else
               atomicOr(&counters[6], (unsigned long long)kStatusOverflow);
         }
      }
   }
}

// Count, scan and fill of a small volume by one CTA, its counts in shared
// memory: one launch for five (25 us on 280 segments and 30 bricks).
constexpr int64_t kSmallBricks = 4096, kSmallPairs = 16384;

__global__ void __launch_bounds__(1024)
brick_bin_small(const SegDev *__restrict__ segs, const int32_t *__restrict__ seg_tile,
                int n_segs, const TileDev *__restrict__ tiles, int n_bricks,
                unsigned *__restrict__ offsets, unsigned *__restrict__ list, int64_t n_pairs,
                uint2 *__restrict__ marks, int64_t mark_share, int n_shares,
                unsigned long long *__restrict__ counters) {
   __shared__ unsigned count[kSmallBricks], wsum[32];
   const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
   if (mark_share > 0 && t < n_shares) // the marked voxels' lists start empty
      marks[t * mark_share] = marks[t * mark_share + 1] = make_uint2(0u, 0u);
   for (int b = t; b < n_bricks; b += 1024)
      count[b] = 0;
   __syncthreads();
   auto pairs = [&](auto &&f) {
      for (int i = t; i < n_segs * kBinLanes; i += 1024) {
         const int s = i / kBinLanes;
         const SegBricks r = seg_bricks(segs[s]);
         const TileDev &T = tiles[seg_tile ? seg_tile[s] : 0];
         const unsigned n = r.nx * r.ny * r.nz; // at most n_bricks
         for (unsigned p = i % kBinLanes; p < n; p += kBinLanes)
            f(s, (int)pair_brick(r, T, p));
      }
   };
   pairs([&](int, int b) { atomicAdd(&count[b], 1u); });
   __syncthreads();
   // exclusive scan, 4 consecutive bricks per thread
   const int b0 = 4 * t;
   unsigned v[4], sum = 0;
#pragma unroll
   for (int i = 0; i < 4; i++) {
      v[i] = b0 + i < n_bricks ? count[b0 + i] : 0u;
      sum += v[i];
   }
   unsigned x = sum;
#pragma unroll
   for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o)
         x += y;
   }
   if (lane == 31)
      wsum[wid] = x;
   __syncthreads();
   if (wid == 0) {
      unsigned w = wsum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
         const unsigned y = __shfl_up_sync(0xffffffffu, w, o);
         if (lane >= o)
            w += y;
      }
      wsum[lane] = w;
   }
   __syncthreads();
   unsigned run = (wid ? wsum[wid - 1] : 0u) + (x - sum);
#pragma unroll
   for (int i = 0; i < 4; i++)
      if (b0 + i < n_bricks) {
         offsets[b0 + i] = count[b0 + i] = run; // the fill's cursor
         run += v[i];
      }
   if (t == 0)
      offsets[n_bricks] = wsum[31];
   __syncthreads();
   pairs([&](int s, int b) {
      const unsigned at = atomicAdd(&count[b], 1u);
      if ((int64_t)at < n_pairs)
         list[at] = (unsigned)s;
      else
         atomicOr(&counters[6], (unsigned long long)kStatusOverflow);
   });
}

// Exclusive scan of the per-brick counts, one CTA walking the counts in tiles
// of 1024 x 8: each thread loads 8 consecutive counts (two 16-byte loads when
// the tile is whole: the arrays start 256-byte aligned and a thread's first
// index is a multiple of 8), the thread sums are scanned across the block
// (warp shuffles, then the 32 warp sums) and the running total carries from
// tile to tile.  offsets[n] receives the total; a total of 2^32 - 1 or more
// is reported as an overflow of the 32-bit offsets.
constexpr int kScanPer = 8;

__global__ void __launch_bounds__(1024)
brick_scan(const unsigned *__restrict__ counts, int64_t n, unsigned *__restrict__ offsets,
           uint2 *__restrict__ marks, int64_t mark_share, int n_shares,
           unsigned long long *__restrict__ counters) {
   if (mark_share > 0 && (int)threadIdx.x < n_shares) // the marked voxels' lists start empty
      marks[threadIdx.x * mark_share] = marks[threadIdx.x * mark_share + 1] = make_uint2(0u, 0u);
   __shared__ unsigned long long wsum[32];
   const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
   // the callers' workspaces are 256-byte aligned; checked anyway before any
   // 16-byte access
   const bool vec = (((uintptr_t)counts | (uintptr_t)offsets) & 15) == 0;
   unsigned long long carry = 0; // total of the tiles before this one (the same in every thread)
   for (int64_t base = 0; base < n; base += (int64_t)blockDim.x * kScanPer) {
      const int64_t i0 = base + (int64_t)t * kScanPer;
      unsigned v[kScanPer];
      if (vec && i0 + kScanPer <= n) {
         const uint4 a = *reinterpret_cast<const uint4 *>(counts + i0);
         const uint4 b = *reinterpret_cast<const uint4 *>(counts + i0 + 4);
         v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
         v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
      } else {
#pragma unroll
         for (int k = 0; k < kScanPer; k++)
            v[k] = i0 + k < n ? counts[i0 + k] : 0u;
      }
      unsigned long long s = 0;
#pragma unroll
      for (int k = 0; k < kScanPer; k++)
         s += v[k];
      unsigned long long x = s; // inclusive scan over the warp
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
         const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
         if (lane >= o)
            x += y;
      }
      if (lane == 31)
         wsum[wid] = x;
      __syncthreads();
      if (wid == 0) { // inclusive scan of the warp sums
         unsigned long long w = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0ull;
#pragma unroll
         for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o)
               w += y;
         }
         wsum[lane] = w;
      }
      __syncthreads();
      unsigned long long run = carry + (wid ? wsum[wid - 1] : 0ull) + (x - s);
      unsigned o8[kScanPer];
#pragma unroll
      for (int k = 0; k < kScanPer; k++) {
         o8[k] = (unsigned)run;
         run += v[k];
      }
      if (vec && i0 + kScanPer <= n) {
         *reinterpret_cast<uint4 *>(offsets + i0) = make_uint4(o8[0], o8[1], o8[2], o8[3]);
         *reinterpret_cast<uint4 *>(offsets + i0 + 4) = make_uint4(o8[4], o8[5], o8[6], o8[7]);
      } else {
#pragma unroll
         for (int k = 0; k < kScanPer; k++)
            if (i0 + k < n)
               offsets[i0 + k] = o8[k];
      }
      carry += wsum[31];
      __syncthreads(); // wsum is rewritten by the next tile
   }
   if (t == 0) {
      offsets[n] = (unsigned)carry;
      if (carry >= 0xFFFFFFFFull)
         atomicOr(&counters[6], (unsigned long long)kStatusOverflow);
   }
}

// ----------------------------------------------------------------- sweep ---
constexpr int kPlane = kBrickY * kBrickZ; // distance of x neighbours in the shared arrays

// Place of (y, z) in a plane of the shared arrays.  A row y is rotated by 9 y:
// the lanes of a chunk cover several rows of a sub-box some 8 to 13 voxels
// high, which would else share that many of the 32 banks.
FPGB_HD int plane_place(int y, int z) {
   return y * kBrickZ + ((z + 9 * y) & (kBrickZ - 1));
}

// The inputs of the sweep of one segment (SegDev offsets 96..191: pf, vf,
// c2f, c2_rcp, thr_f, acc_f, base, lo, ext, bundle, mg) in 16-byte loads.
struct SegSweep {
   float4 a; // pf[0..2], vf[0]
   float4 b; // vf[1..2], c2f, c2_rcp
   float4 c; // thr_f, acc_f, base[0..1] (int bits)
   int4 d;   // base[2], lo[0..2]
   int4 e;   // ext[0..2], bundle
   float mg;
};

// a / b within 2 ulps, of the device's approximate division
FPGB_HD float quotient_est(float a, float b) {
#ifdef __CUDA_ARCH__
   return __fdividef(a, b);
#else
   return a / b;
#endif
}

FPGB_HD int int_min(int a, int b) { return a < b ? a : b; }
FPGB_HD int int_max(int a, int b) { return a > b ? a : b; }

FPGB_HD int leading_zeros(unsigned v) { // v > 0
#ifdef __CUDA_ARCH__
   return __clz((int)v);
#else
   return __builtin_clz(v);
#endif
}

FPGB_HD int float_bits(float f) {
#ifdef __CUDA_ARCH__
   return __float_as_int(f);
#else
   int i;
   std::memcpy(&i, &f, sizeof i);
   return i;
#endif
}

__device__ __forceinline__ SegSweep load_sweep(const SegDev &S) {
   const float4 *f = reinterpret_cast<const float4 *>(&S.pf[0]);
   const int4 *i = reinterpret_cast<const int4 *>(&S.pf[0]);
   return SegSweep{__ldg(f), __ldg(f + 1), __ldg(f + 2), __ldg(i + 3), __ldg(i + 4),
                   __ldg(&S.mg)};
}

// The part of segment S's clipped box inside the brick (origin o, extent n),
// swept as columns along x: its ey x ez (y, z) cells are numbered z fastest,
// lane l of chunk c owns cell 32 c + l and visits the ex voxels of that
// cell's x column.  The y and z parts of the estimate are computed once per
// cell; each voxel then costs five operations (sweep_dist2).
struct SubBox {
   int x0, y0, z0, ex, ey, ez, ncell;
   float inv_ez; // 1/ez for the division-free cell split
};

FPGB_HD bool sub_box(const SegSweep &w, int ox, int oy, int oz, int nx, int ny, int nz,
                     SubBox &b) {
   b.x0 = int_max(w.d.y, ox);
   b.y0 = int_max(w.d.z, oy);
   b.z0 = int_max(w.d.w, oz);
   b.ex = int_min(w.d.y + w.e.x, ox + nx) - b.x0;
   b.ey = int_min(w.d.z + w.e.y, oy + ny) - b.y0;
   b.ez = int_min(w.d.w + w.e.z, oz + nz) - b.z0;
   if (b.ex <= 0 || b.ey <= 0 || b.ez <= 0)
      return false;
   b.ncell = b.ey * b.ez;
   b.inv_ez = quotient_est(1.f, (float)b.ez);
   return true;
}

FPGB_HD int brick_index(int x, int y, int z, int ox, int oy, int oz) {
   return ((x - ox) * kBrickY + (y - oy)) * kBrickZ + (z - oz);
}

// The brick's quantisation of the keys: hi * scale rounds to an integer below
// 2^min(23, 32 - slot_bits) (added to 2^23 it sits in the float's mantissa),
// the slot takes the low slot_bits >= 8 bits but the last, the mark.  win: W
// in key units.
struct BrickScale {
   float scale, quantum; // quantum >= 1 / scale
   float mg2;            // 2 max(mg)
   int bits;             // slot_bits
   unsigned mul;         // 1 << slot_bits
   unsigned win, win2;   // W, 2 W (all ones: every two keys are close)
};

constexpr unsigned kNoKey = 0xFFFFFFFFu;

FPGB_HD BrickScale brick_scale(unsigned n_seg, float max_thr2, float max_mg) {
   BrickScale k;
   const int bits = n_seg <= 128u ? 8 : int_min(31, 33 - leading_zeros(n_seg - 1u));
   const int qbits = int_min(23, 32 - bits);
   k.bits = bits;
   k.mul = 1u << bits;
   const float top = qbits > 3 ? (float)((1u << qbits) - 4u) : 0.f;
   k.scale = 0.999999f * quotient_est(top, max_thr2);
   if (!(k.scale > 0.f && k.scale < 1e30f))
      k.scale = 0.f;
   k.quantum = k.scale > 0.f ? quotient_est(1.000001f, k.scale) : INFINITY;
   k.mg2 = 2.f * max_mg;
   const float w = fmaf(k.mg2, k.scale, 4.f) * (float)k.mul;
   if (w < 1e9f) {
      k.win = (unsigned)w;
      k.win2 = 2u * k.win;
   } else { // NaN too
      k.win = 0x7FFFFFFFu;
      k.win2 = 0xFFFFFFFFu;
   }
   return k;
}

// Upper bound of the hi that a voxel's key stands for.
FPGB_HD float key_bound(const BrickScale &k, unsigned key) {
   return ((float)(key >> k.bits) + 1.f) * k.quantum;
}

// A segment's inputs to the sweep of one brick, in shared memory: a thread
// prepares a segment (about 100 instructions), a warp then reads it with three
// 16-byte loads.
struct __align__(16) SweepRec {
   float wx0, wy0, wz0, mg;    // voxel centre - float(p - base) of the sub-box's first voxel
   float vn2x, vn2y, vn2z, c2f; // -2 v, v.v
   float rch, thr, inv_ez;     // -1/2 float(1 / c2), bound of hi
   unsigned box;               // ncell, ez << 9, ex << 15, first voxel's place << 19
};

// A segment as the sweep of one sub-box sees it: the first voxel's offset from
// its start, its direction, their FP32 invariants and the bound of the estimate.
struct SegPart {
   float w0[3], v[3], c2f, c2_rcp, mg;
};

// The estimate's error grows with the square of a segment's length, and the
// largest of a brick's margins decides which of its voxels are close calls.  So
// of a long segment the sweep takes the part that holds the closest point of
// every voxel of the sub-box: the distances are the same (the rounding of the
// part's start in double, below 2^-50 pscale, is a ninth of what sweep_margin
// has for that), the error that of a segment as long as the sub-box.
__host__ __device__ __noinline__ inline SegPart long_part(const SegDev &S, const SubBox &b) {
   SegPart r{};
   r.mg = INFINITY;
   if (!(S.mg < INFINITY)) // every voxel of the sub-box counts as inside, W marks it
      return r;
   const int first[3] = {b.x0, b.y0, b.z0}, ext[3] = {b.ex, b.ey, b.ez};
   // closest-point parameters of the sub-box: its centre's, give or take half its
   // extent along v and 1/16 voxel
   double mid = 0.0, reach = 0.0625 * sqrtf(S.c2f);
   for (int i = 0; i < 3; i++) {
      const double half = 0.5 * (ext[i] - 1);
      mid = mid + ((first[i] + 0.5 + half) - S.p[i]) * S.v[i];
      reach = reach + half * fabs(S.v[i]);
   }
   const double rc2 = 1.0 / S.c2;
   const double t0 = fmin(fmax((mid - reach) * rc2, 0.0), 1.0);
   const double part = fmin(fmax((mid + reach) * rc2, 0.0), 1.0) - t0;
   float steps[3];
   for (int i = 0; i < 3; i++) {
      r.w0[i] = (float)((first[i] + 0.5) - (S.p[i] + S.v[i] * t0));
      r.v[i] = (float)(S.v[i] * part);
      steps[i] = (float)(ext[i] - 1);
   }
   r.c2f = (float)(part * part * S.c2);
   r.c2_rcp = r.c2f > 0.f ? 1.f / r.c2f : 0.f;
   r.mg = sweep_margin(r.w0, steps, r.c2f, S.pscale, S.thr_f);
   return r;
}

template <bool LONG>
FPGB_HD SegPart seg_part(const SegDev &S, const SegSweep &w, const SubBox &b) {
   if (LONG && w.b.z > kLongSquared)
      return long_part(S, b);
   const int first[3] = {b.x0, b.y0, b.z0}, base[3] = {float_bits(w.c.z), float_bits(w.c.w), w.d.x};
   const float pf[3] = {w.a.x, w.a.y, w.a.z};
   SegPart r;
   for (int i = 0; i < 3; i++)
      r.w0[i] = ((float)(first[i] - base[i]) + 0.5f) - pf[i];
   r.v[0] = w.a.w;
   r.v[1] = w.b.x;
   r.v[2] = w.b.y;
   r.c2f = w.b.z;
   r.c2_rcp = w.b.w;
   r.mg = w.mg;
   return r;
}

template <bool LONG>
FPGB_HD SweepRec sweep_rec(const SegPart &g, float thr, const SubBox &b, bool any, int ox, int oy,
                           int oz) {
   SweepRec r;
   r.wx0 = g.w0[0];
   r.wy0 = g.w0[1];
   r.wz0 = g.w0[2];
   r.mg = !LONG || g.mg < INFINITY ? g.mg : 0.f;
   r.vn2x = -2.f * g.v[0];
   r.vn2y = -2.f * g.v[1];
   r.vn2z = -2.f * g.v[2];
   r.c2f = g.c2f;
   r.rch = -0.5f * g.c2_rcp;
   // (finite: a radius whose square is not)
   r.thr = fminf(fmaf(2.00001f, g.mg, thr), 3e38f);
   r.inv_ez = b.inv_ez;
   r.box = any ? (unsigned)b.ncell | (unsigned)b.ez << 9 | (unsigned)b.ex << 15 |
                     (unsigned)brick_index(b.x0, b.y0, b.z0, ox, oy, oz) << 19
               : 0u;
   return r;
}

// A lane's (y, z) cell of a chunk of 32, numbered z fastest, in float
// arithmetic (all integers below 2^24).  (c + 1/2) / ez lies at least
// 1/(2 ez) >= 2^-6 from an integer for c < 256 and ez <= 32, far beyond the
// error of the product with the approximate reciprocal, so the truncation is
// the exact quotient.
struct Cell {
   int yz;      // plane_place
   float a2, b; // the y / z parts of the estimate
};

FPGB_HD Cell cell_of(const SweepRec &g, float ezf, float c) {
   const float iy = truncf((c + 0.5f) * g.inv_ez);
   const float iz = fmaf(-iy, ezf, c);
   const float wy = g.wy0 + iy, wz = g.wz0 + iz;
   return Cell{plane_place((int)(g.box >> 24 & 7u) + (int)iy, (int)(g.box >> 19 & 31u) + (int)iz),
               fmaf(wz, g.vn2z, wy * g.vn2y),
               fmaf(wz, wz, fmaf(wy, wy, g.mg))};
}

constexpr int kSweepStep = 4; // candidates of a column at a time (2: 889 us, 8: 924)

// What a warp carries through the sweep of one segment.
struct SweepState {
   float thr;       // the lane's bound of hi (below every hi without a cell)
   float acc;       // hi at or below which the voxel is certainly inside
   unsigned bundle, slot2; // bundle, 2 slot
   unsigned *skey, *smark, *sminb;
};

// N candidates of the lane's x column, at wx, wx + 1, ... (their atomics are
// in flight together).  The atomic is predicated: it takes time per active
// lane (880 us; with kNoKey from the candidates outside 905).  multi: the
// smallest bundle whose fiber a voxel is certainly inside of is kept as well;
// voxels that are only possibly inside get a mark of their own, which stays.
template <bool MULTI, int N>
__device__ __forceinline__ void sweep_step(const SweepRec &g, const SweepState &w, const Cell &c,
                                           const BrickScale &k, bool multi, float wx,
                                           unsigned *key) {
   float hi[N];
   unsigned mine[N], old[N];
   bool close[N], any = false;
#pragma unroll
   for (int u = 0; u < N; u++) {
      hi[u] = sweep_dist2(u ? wx + (float)u : wx, c.a2, c.b, g.vn2x, g.c2f, g.rch);
      mine[u] = __float_as_uint(fmaf(hi[u], k.scale, 8388608.f)) * k.mul + w.slot2;
   }
   // (NaN, from an infinite bound, counts as inside)
   const unsigned a = (unsigned)__cvta_generic_to_shared(key);
#pragma unroll
   for (int u = 0; u < N; u++) {
      old[u] = 0;
      asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.f32 p, %3, %4;\n\t"
                   "@!p atom.shared.min.u32 %0, [%1], %2;\n\t}"
                   : "+r"(old[u])
                   : "r"(a + 4u * kPlane * u), "r"(mine[u]), "f"(hi[u]), "f"(w.thr)
                   : "memory");
   }
#pragma unroll
   for (int u = 0; u < N; u++) {
      close[u] = !(hi[u] > w.thr) && old[u] - mine[u] + k.win <= k.win2;
      any = any || close[u];
   }
   if (__any_sync(0xFFFFFFFFu, any)) {
#pragma unroll
      for (int u = 0; u < N; u++)
         if (close[u])
            atomicOr(key + u * kPlane, 1u);
   }
   if (MULTI && multi) {
#pragma unroll
      for (int u = 0; u < N; u++) {
         const int at = (int)(key - w.skey) + u * kPlane;
         if (hi[u] <= fminf(w.acc, w.thr)) {
            atomicMin(w.sminb + at, w.bundle);
         } else if (!(hi[u] > w.thr)) {
            const int yz = at & (kPlane - 1);
            atomicOr(&w.smark[yz >> 2], 1u << (8 * (yz & 3) + at / kPlane));
         }
      }
   }
}

// The sweep of one segment over its sub-box.  Every lane runs every step (the
// control flow of a warp stays uniform: diverging branches cost a quarter of
// the sweep's instructions); one without a cell of its own repeats the last
// with a bound that nothing meets (a NaN does, and marks a voxel too many).
template <bool MULTI>
__device__ __forceinline__ void brick_sweep(const SweepRec &rec, unsigned slot, float acc,
                                            unsigned bundle, const BrickScale &k, bool multi,
                                            unsigned *skey, unsigned *smark, unsigned *sminb,
                                            int lane) {
   const SweepRec g = rec;
   const float ezf = (float)(g.box >> 9 & 63u);
   const int ncell = (int)(g.box & 511u), ex = (int)(g.box >> 15 & 15u);
   unsigned *first = skey + (g.box >> 27) * kPlane;
   SweepState w{g.thr, acc, bundle, 2u * slot, skey, smark, sminb};
   for (int c0 = 0; c0 < ncell; c0 += 32) {
      const int at = c0 + lane;
      w.thr = at < ncell ? g.thr : -INFINITY;
      const Cell c = cell_of(g, ezf, (float)min(at, ncell - 1));
      unsigned *key = first + c.yz;
      float wx = g.wx0;
      int i = ex;
      for (; i >= kSweepStep; i -= kSweepStep, wx += (float)kSweepStep, key += kSweepStep * kPlane)
         sweep_step<MULTI, kSweepStep>(g, w, c, k, multi, wx, key);
#pragma unroll
      for (int n = kSweepStep / 2; n >= 1; n /= 2)
         if (i & n) {
            if (n == 2)
               sweep_step<MULTI, 2>(g, w, c, k, multi, wx, key);
            else
               sweep_step<MULTI, 1>(g, w, c, k, multi, wx, key);
            wx += (float)n;
            key += n * kPlane;
         }
   }
}

// Exact evaluation of one candidate: the two-float path, with the FP64
// replay of the reference arithmetic for the few it leaves undecided.  Out of
// line: one shared copy of these large bodies keeps the sweep loops that call
// them small in the instruction cache.
//
// float(|closest - point|^2) and float(r(t)^2) (generator.cpp:327-328) of
// (S, voxel x y z); returns true when the FP64 replay ran.
__device__ __noinline__ bool cand_dist(const SegDev &S, int x, int y, int z, float &dist_squ,
                                       float &r_sqr) {
   const float lpt[3] = {(float)(x - S.base[0]) + 0.5f, (float)(y - S.base[1]) + 0.5f,
                         (float)(z - S.base[2]) + 0.5f};
   FastCand fc;
   if (S.pscale < 0x1p22f && fast_candidate(S, lpt, fc)) {
      dist_squ = fc.dist_squ;
      r_sqr = fc.r_sqr;
      return false;
   }
   const double pt[3] = {(double)x + 0.5, (double)y + 0.5, (double)z + 0.5};
   double cl[3];
   exact_dist(S, pt, cl, dist_squ, r_sqr);
   return true;
}

// float(vm::unit(point - closest)) of the 'r' layer (generator.cpp:365-371);
// returns true when the FP64 replay ran.
__device__ __noinline__ bool cand_radial(const SegDev &S, int x, int y, int z, float o[3]) {
   const float lpt[3] = {(float)(x - S.base[0]) + 0.5f, (float)(y - S.base[1]) + 0.5f,
                         (float)(z - S.base[2]) + 0.5f};
   FastCand fc;
   ff t;
   if (S.pscale < 0x1p22f && fast_offset(S, lpt, fc, t) && fast_radial(S, fc, o))
      return false;
   const double pt[3] = {(double)x + 0.5, (double)y + 0.5, (double)z + 0.5};
   double cl[3];
   float d_chk, r_chk;
   exact_dist(S, pt, cl, d_chk, r_chk);
   // unit vector in the reference's double order
   double nv[3] = {pt[0] - cl[0], pt[1] - cl[1], pt[2] - cl[2]};
   double n2 = 0.0;
   n2 = n2 + nv[0] * nv[0];
   n2 = n2 + nv[1] * nv[1];
   n2 = n2 + nv[2] * nv[2];
   if (n2 > 0) {
      const double inv = 1.0 / sqrt(n2);
      nv[0] = nv[0] * inv;
      nv[1] = nv[1] * inv;
      nv[2] = nv[2] * inv;
   }
   o[0] = (float)nv[0];
   o[1] = (float)nv[1];
   o[2] = (float)nv[2];
   return true;
}

// Segments of a brick's list whose index, r^2 and bundle are kept in shared
// memory (the lists of the uneven tiles hold 30 on average, of a dense volume
// 180).
constexpr unsigned kSegCache = 512;
constexpr int32_t kMarkedLabel = INT32_MIN; // until voxel_marks has resolved it

// The layers of the tile's first bundles, in shared memory.
struct LayerLut {
   int n;
   unsigned models; // two bits per layer: 0 'b', 1 'p', 2 'r'
   float sq[kMaxLayers]; // sq_fdown
};
constexpr int kLayerCache = 4;

// Layer of a winner whose dist^2 lies in [lo, hi] with r^2 = r_sqr: the
// reference's lower_bound over scale^2 of the float dist^2 / r^2
// (generator.cpp:345-349).  2^-20 covers the rounding of the quotient and of
// the products here.  -1 when the interval straddles a boundary, the
// outermost one included.
FPGB_HD int certain_layer(const float *sq, int n, float lo, float hi, float r_sqr) {
   int w = 0;
   bool sure = true;
   for (int l = 0; l < n; l++) {
      const float b = sq[l] * r_sqr;
      const bool past = hi > b * (1.f - 0x1p-20f);
      w += past ? 1 : 0;
      sure = sure && (!past || lo > b * (1.f + 0x1p-20f));
   }
   return sure && w < n ? w : -1;
}

// The 'r' orientation of voxel (x, y, z) for winner S: unit(point - closest)
// (generator.cpp:365-371) by the two-float path, FP64 replay when undecided.
__device__ __forceinline__ void radial_vector(const SegDev &S, int x, int y, int z, float o[3],
                                              unsigned long long &n_slow) {
   if (cand_radial(S, x, y, z, o))
      n_slow++;
}

// A brick: its tile and place.
struct BrickPlace {
   const TileDev *T;
   int64_t tile;
   int ox, oy, oz, nx, ny, nz;
};

__device__ __forceinline__ BrickPlace brick_place(const TileDev *__restrict__ tiles,
                                                  int64_t n_tiles, int64_t brick) {
   // last tile whose brick_base <= brick
   int64_t lo = 0, hi = n_tiles - 1;
   while (lo < hi) {
      const int64_t mid = (lo + hi + 1) >> 1;
      if (tiles[mid].brick_base <= brick)
         lo = mid;
      else
         hi = mid - 1;
   }
   BrickPlace p;
   p.tile = lo;
   p.T = tiles + lo;
   const unsigned lb = (unsigned)(brick - p.T->brick_base); // below 2^32: the lists are 32-bit
   const unsigned rxy = lb / (unsigned)p.T->nb[2], bx = rxy / (unsigned)p.T->nb[1];
   p.ox = (int)bx * kBrickX;
   p.oy = (int)(rxy - bx * (unsigned)p.T->nb[1]) * kBrickY;
   p.oz = (int)(lb - rxy * (unsigned)p.T->nb[2]) * kBrickZ;
   p.nx = min(kBrickX, p.T->X - p.ox);
   p.ny = min(kBrickY, p.T->Y - p.oy);
   p.nz = min(kBrickZ, p.T->Z - p.oz);
   return p;
}

// --------------------------------------------------------- marked voxels ---
// Marked voxels of one brick that get a record; a brick with more is full.
constexpr unsigned kMarkList = 128;
constexpr int kMarkThreads = 128, kMarkQueue = 192;
constexpr unsigned kNoRecord = 0x80000000u; // directory entry of a brick whose record had no room

// What one warp of voxel_marks works on: up to 32 marked voxels of its brick,
// and the candidates found for them.
struct MarkWarp {
   unsigned long long exact[32]; // winner keys
   unsigned bound[32];           // float bits of the smallest certain upper bound
   unsigned minb[32];            // smallest bundle a voxel is inside of
   unsigned short voxel[32];     // place in the brick
   unsigned q_seg[kMarkQueue];
   float q_lo[kMarkQueue];
   unsigned char q_mark[kMarkQueue]; // voxel; bit 7: certainly inside
};

struct MarkCtx {
   BrickPlace p;
   unsigned n_seg;
   const unsigned *list;
   const SegDev *segs;
   const LayerDev *layers;
   int32_t *label;
   float *vec;
   bool multi; // the overlap warning is still open
};

// Label and orientation of a marked voxel from its winner's key
// (generator.cpp:343-372).
__device__ __forceinline__ void finish_voxel(const MarkCtx &C, unsigned long long key, int x,
                                             int y, int z, unsigned minb,
                                             unsigned long long &n_slow,
                                             unsigned long long &n_overlap,
                                             unsigned long long &n_overflow) {
   const int64_t i = ((int64_t)x * C.p.T->Y + y) * C.p.T->Z + z;
   int32_t lab = 0;
   float o[3] = {0.f, 0.f, 0.f};
   if (key != ~0ull) {
      const SegDev &S = C.segs[0xFFFFFFFFu - (unsigned)key];
      const LayerDev &L = C.layers[S.bundle];
      float dist_squ = __uint_as_float((unsigned)(key >> 32)), r_sqr = S.dec_rsq;
      if (!(r_sqr == r_sqr) && cand_dist(S, x, y, z, dist_squ, r_sqr))
         n_slow++;
      // std::lower_bound(scale^2, double(dist_squ / r_sqr)) (generator.cpp:345-349)
      const float qv = dist_squ / r_sqr;
      int w = 0;
      while (w < L.n && qv > L.sq_fdown[w])
         w++;
      if (w == L.n)
         n_overflow++;
      if (C.multi && minb < (unsigned)S.bundle)
         n_overlap++;
      lab = w + 1 + S.bundle * C.p.T->max_layer;
      const unsigned m = w < L.n ? L.models >> (2 * w) & 3u : 0u;
      if (m == 1u) {
         o[0] = S.vp[0];
         o[1] = S.vp[1];
         o[2] = S.vp[2];
      } else if (m == 2u && C.vec) {
         radial_vector(S, x, y, z, o, n_slow);
      }
   }
   C.label[i] = lab;
   if (C.vec) {
      C.vec[3 * i + 0] = o[0];
      C.vec[3 * i + 1] = o[1];
      C.vec[3 * i + 2] = o[2];
   }
}

// Evaluates the queued candidates that can still win, 32 at a time.
__device__ __forceinline__ void drain_marks(const MarkCtx &C, MarkWarp &W, int qn, int lane,
                                            unsigned long long &n_slow) {
   __syncwarp();
   int n = 0; // the ones kept, at the front of the queue
   for (int i = 0; i < qn; i += 32) {
      unsigned s = 0, m = 0;
      bool need = false;
      if (i + lane < qn) {
         s = W.q_seg[i + lane];
         m = W.q_mark[i + lane];
         need = !(W.q_lo[i + lane] > __uint_as_float(W.bound[m & 31u])) ||
                (C.multi && !(m & 128u) && (unsigned)C.segs[s].bundle < W.minb[m & 31u]);
      }
      const unsigned b = __ballot_sync(0xFFFFFFFFu, need);
      if (need) {
         const int at = n + __popc(b & ((1u << lane) - 1u));
         W.q_seg[at] = s;
         W.q_mark[at] = (unsigned char)m;
      }
      n += __popc(b);
      __syncwarp();
   }
   for (int i = lane; i < n; i += 32) {
      const unsigned s = W.q_seg[i], m = W.q_mark[i] & 31u;
      const SegDev &S = C.segs[s];
      const int v = W.voxel[m];
      float dist_squ, r_sqr;
      if (cand_dist(S, C.p.ox + (v >> 8), C.p.oy + (v >> 5 & 7), C.p.oz + (v & 31), dist_squ,
                    r_sqr))
         n_slow++;
      if (dist_squ > C.layers[S.bundle].f_ly_squ * r_sqr) // generator.cpp:329-331
         continue;
      atomicMin(&W.exact[m], ((unsigned long long)__float_as_uint(dist_squ) << 32) |
                                 (unsigned long long)(0xFFFFFFFFu - s));
      atomicMin(&W.bound[m], __float_as_uint(dist_squ));
      if (C.multi)
         atomicMin(&W.minb[m], (unsigned)S.bundle);
   }
   __syncwarp();
}

// The nm <= 32 marked voxels W.voxel: a segment of the list per lane, its
// inputs in registers while the voxels pass by.
__device__ __forceinline__ void resolve_marks(const MarkCtx &C, MarkWarp &W, int nm, int lane,
                                              unsigned long long &n_slow,
                                              unsigned long long &n_overlap,
                                              unsigned long long &n_overflow) {
   W.exact[lane] = ~0ull;
   W.bound[lane] = __float_as_uint(INFINITY);
   W.minb[lane] = ~0u;
   __syncwarp();
   int qn = 0;
   for (unsigned j = 0; j < C.n_seg; j += 32) {
      const bool have = j + lane < C.n_seg;
      const unsigned s = C.list[have ? j + lane : C.n_seg - 1];
      const SegSweep w = load_sweep(C.segs[s]);
      for (int m = 0; m < nm; m++) {
         const int v = W.voxel[m];
         const int x = C.p.ox + (v >> 8), y = C.p.oy + (v >> 5 & 7), z = C.p.oz + (v & 31);
         float lo = 0.f;
         bool in = have && x >= w.d.y && x < w.d.y + w.e.x && y >= w.d.z && y < w.d.z + w.e.y &&
                   z >= w.d.w && z < w.d.w + w.e.z;
         bool certain = false;
         if (in) {
            float mg;
            const float d2 = approx_dist2(((float)(x - __float_as_int(w.c.z)) + 0.5f) - w.a.x,
                                          ((float)(y - __float_as_int(w.c.w)) + 0.5f) - w.a.y,
                                          ((float)(z - w.d.x) + 0.5f) - w.a.z, w.a.w, w.b.x,
                                          w.b.y, w.b.z, w.b.w, mg);
            lo = w.mg < INFINITY ? __fsub_rd(d2, mg) : 0.f;
            const float hi = __fadd_ru(d2, mg);
            certain = hi <= w.c.y;
            in = !(lo > w.c.x);
            if (certain) {
               atomicMin(&W.bound[m], __float_as_uint(hi));
               if (C.multi)
                  atomicMin(&W.minb[m], (unsigned)w.e.w);
            }
         }
         const unsigned b = __ballot_sync(0xFFFFFFFFu, in);
         if (!b)
            continue;
         if (in) {
            const int at = qn + __popc(b & ((1u << lane) - 1u));
            W.q_seg[at] = s;
            W.q_lo[at] = lo;
            W.q_mark[at] = (unsigned char)(m | (certain ? 128 : 0));
         }
         qn += __popc(b);
         if (qn > kMarkQueue - 32) {
            drain_marks(C, W, qn, lane, n_slow);
            qn = 0;
         }
      }
   }
   drain_marks(C, W, qn, lane, n_slow);
   if (lane < nm) {
      const int v = W.voxel[lane];
      finish_voxel(C, W.exact[lane], C.p.ox + (v >> 8), C.p.oy + (v >> 5 & 7), C.p.oz + (v & 31),
                   W.minb[lane], n_slow, n_overlap, n_overflow);
   }
   __syncwarp();
}

// Full bricks: where fibers share their course, or a radius changes along a
// segment (then the shell between a segment's own and its thickest radius is
// undecided), a sixth to all of the voxels are marked.  A CTA takes half a
// brick: its warps sweep the segments over the marked voxels (a byte of marks
// per column lets the others pass) and queue the candidates whose lower bound is
// not past the smallest certain upper one, for 32 lanes at a time.  Bound by
// issue (46% of the slots at 14 warps per SM), most of it the exact
// evaluations.  A warp per brick that walked the list row by row before: 256 x
// 256 x 64, 58% of the voxels in two copies of a fiber 2,674 -> 444 us, two
// bundles of them 2,646 -> 459, tapered fibers 515 -> 205.
constexpr int kHalfX = kBrickX / 2, kFullRecs = 64;

struct FullSeg {
   float acc, mg2; // surely inside up to acc; hi - mg2 is a lower bound
   unsigned bundle, seg;
};

struct FullScratch {
   unsigned long long key[kHalfX * kPlane]; // winner's; until then {smallest certain hi, ~0}
   unsigned minb[kHalfX * kPlane];          // smallest bundle the voxel is inside of
   SweepRec rec[kFullRecs];
   FullSeg seg[kFullRecs];
   unsigned q_seg[kMarkThreads / 32][64];
   unsigned short q_voxel[kMarkThreads / 32][64];
   unsigned char mark[kPlane]; // a bit per x
   unsigned next;
};

// z of a place in the plane's row y (plane_place)
__device__ __forceinline__ int place_z(int place, int y) {
   return (place - 9 * y) & (kBrickZ - 1);
}

// Evaluates n <= 32 queued candidates, a lane each.
__device__ __forceinline__ void drain_full(const MarkCtx &C, FullScratch &F, int at, int n, int x0,
                                           int lane, int warp, unsigned long long &n_slow) {
   __syncwarp();
   if (lane < n) {
      const unsigned s = F.q_seg[warp][at + lane];
      const int li = F.q_voxel[warp][at + lane], y = li >> 5 & 7;
      const SegDev &S = C.segs[s];
      float dist_squ, r_sqr;
      if (cand_dist(S, C.p.ox + x0 + (li >> 8), C.p.oy + y, C.p.oz + place_z(li, y), dist_squ,
                    r_sqr))
         n_slow++;
      if (!(dist_squ > C.layers[S.bundle].f_ly_squ * r_sqr)) { // generator.cpp:329-331
         atomicMin(&F.key[li], ((unsigned long long)__float_as_uint(dist_squ) << 32) |
                                   (unsigned long long)(0xFFFFFFFFu - s));
         if (C.multi)
            atomicMin(&F.minb[li], (unsigned)S.bundle);
      }
   }
   __syncwarp();
}

// The marked voxels x0 <= x < x0 + nx <= x0 + kHalfX of a brick, by the CTA.
__device__ __forceinline__ void resolve_full(const MarkCtx &C, FullScratch &F, int x0, int nx,
                                             unsigned long long &n_slow,
                                             unsigned long long &n_overlap,
                                             unsigned long long &n_overflow) {
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   const int64_t plane = (int64_t)C.p.T->Y * C.p.T->Z;
   const int64_t corner =
       (C.p.ox + x0) * plane + (int64_t)C.p.oy * C.p.T->Z + C.p.oz; // of the half brick
   bool any = false;
   for (int yz = threadIdx.x; yz < kPlane; yz += kMarkThreads) {
      const int y = yz >> 5, z = yz & 31, at = plane_place(y, z);
      unsigned m = 0;
      for (int x = 0; x < kHalfX; x++) {
         if (x < nx && y < C.p.ny && z < C.p.nz &&
             C.label[corner + x * plane + (int64_t)y * C.p.T->Z + z] == kMarkedLabel)
            m |= 1u << x;
         F.key[x * kPlane + at] = ~0ull;
         F.minb[x * kPlane + at] = ~0u;
      }
      F.mark[at] = (unsigned char)m;
      any = any || m;
   }
   if (!__syncthreads_or(any))
      return;
   int qn = 0;
   for (unsigned base = 0; base < C.n_seg; base += kFullRecs) {
      const unsigned n = min(C.n_seg - base, (unsigned)kFullRecs);
      for (unsigned e = threadIdx.x; e < n; e += kMarkThreads) {
         const unsigned s = C.list[base + e];
         const SegSweep w = load_sweep(C.segs[s]);
         SubBox b;
         F.rec[e].box = 0u;
         if (sub_box(w, C.p.ox + x0, C.p.oy, C.p.oz, nx, C.p.ny, C.p.nz, b)) {
            const SegPart g = seg_part<true>(C.segs[s], w, b);
            F.rec[e] = sweep_rec<true>(g, w.c.x, b, true, C.p.ox + x0, C.p.oy, C.p.oz);
            F.seg[e] = FullSeg{w.c.y, 2.00001f * g.mg, (unsigned)w.e.w, s};
         }
      }
      if (threadIdx.x == 0)
         F.next = kMarkThreads / 32;
      __syncthreads();
      for (unsigned j = warp, next; j < n; j = __shfl_sync(0xFFFFFFFFu, next, 0)) {
         if (lane == 0)
            next = atomicAdd(&F.next, 1u);
         const SweepRec g = F.rec[j];
         const FullSeg f = F.seg[j];
         const float ezf = (float)(g.box >> 9 & 63u);
         const int ncell = (int)(g.box & 511u), ex = (int)(g.box >> 15 & 15u);
         const int first = (int)(g.box >> 27);
         for (int c0 = 0; c0 < ncell; c0 += 32) {
            const Cell c = cell_of(g, ezf, (float)min(c0 + lane, ncell - 1));
            const unsigned m =
                c0 + lane < ncell ? F.mark[c.yz] >> first & ((1u << ex) - 1u) : 0u;
            if (!__any_sync(0xFFFFFFFFu, m))
               continue;
            unsigned need = 0; // a bit per x
#pragma unroll
            for (int i = 0; i < kHalfX; i++) {
               const float hi = sweep_dist2(g.wx0 + (float)i, c.a2, c.b, g.vn2x, g.c2f, g.rch);
               if (!(m >> i & 1u) || hi > g.thr)
                  continue;
               // (keys only decrease: any value read bounds the last one; ~0 reads
               // as NaN, past which nothing is)
               const int li = (first + i) * kPlane + c.yz;
               volatile const unsigned *cur = reinterpret_cast<unsigned *>(&F.key[li]) + 1;
               const float best = __uint_as_float(*cur);
               bool mine = !(hi - f.mg2 > best);
               if (hi <= f.acc) {
                  if (!(hi >= best))
                     atomicMin(&F.key[li], ((unsigned long long)__float_as_uint(hi) << 32) |
                                               0xFFFFFFFFull);
                  if (C.multi)
                     atomicMin(&F.minb[li], f.bundle);
               } else if (C.multi) {
                  mine = mine || f.bundle < *reinterpret_cast<volatile unsigned *>(&F.minb[li]);
               }
               need |= mine ? 1u << i : 0u;
            }
            if (!__any_sync(0xFFFFFFFFu, need))
               continue;
            for (int i = 0; i < ex; i++) {
               const unsigned b = __ballot_sync(0xFFFFFFFFu, need >> i & 1u);
               if (need >> i & 1u) {
                  const int at = qn + __popc(b & ((1u << lane) - 1u));
                  F.q_seg[warp][at] = f.seg;
                  F.q_voxel[warp][at] = (unsigned short)((first + i) * kPlane + c.yz);
               }
               qn += __popc(b);
               if (qn >= 32) {
                  qn -= 32;
                  drain_full(C, F, qn, 32, x0, lane, warp, n_slow);
               }
            }
         }
      }
      __syncthreads(); // the records are rewritten
   }
   drain_full(C, F, 0, qn, x0, lane, warp, n_slow);
   __syncthreads();
   for (int yz = threadIdx.x; yz < C.p.ny * kBrickZ; yz += kMarkThreads) {
      const int y = yz >> 5, z = yz & 31, at = plane_place(y, z);
      const unsigned m = F.mark[at];
      for (int x = 0; x < nx; x++)
         if (m >> x & 1u)
            finish_voxel(C, F.key[x * kPlane + at], C.p.ox + x0 + x, C.p.oy + y, C.p.oz + z,
                         F.minb[x * kPlane + at], n_slow, n_overlap, n_overflow);
   }
   __syncthreads(); // the scratch is rewritten for the next
}

// Resolves the marked voxels of the bricks [brick_begin, brick_end): those of
// a record by a warp (bound by latency: 16 warps per SM, each a chain of list,
// segment and evaluation; a voxel per lane walking the list by itself took 260 us
// on the crossing volume instead of 153, 6 CTAs per SM at 80 registers 166),
// full bricks by halves, a CTA each, and so every brick when the launch has no
// space for records.  Units: 2^split parts of a brick, `part` marked voxels of
// one of them.
__global__ void __launch_bounds__(kMarkThreads)
voxel_marks(const SegDev *__restrict__ segs, const TileDev *__restrict__ tiles, int64_t n_tiles,
            int64_t brick_begin, int64_t brick_end, const unsigned *__restrict__ offsets,
            const unsigned *__restrict__ list, unsigned n_pairs,
            const unsigned *__restrict__ directory, const uint2 *__restrict__ marks,
            int64_t mark_share, int split, int part, const LayerDev *__restrict__ layers,
            int32_t *const *__restrict__ labels, float *const *__restrict__ vecs,
            unsigned long long *__restrict__ counters) {
   __shared__ union Scratch {
      MarkWarp warps[kMarkThreads / 32];
      FullScratch full;
      __device__ Scratch() {}
   } scratch;
   MarkWarp &W = scratch.warps[threadIdx.x >> 5];
   const int lane = threadIdx.x & 31;
   const int64_t warp = (blockIdx.x * (int64_t)kMarkThreads + threadIdx.x) >> 5;
   const int64_t n_warps = (int64_t)gridDim.x * (kMarkThreads / 32);
   unsigned long long n_slow = 0, n_overlap = 0, n_overflow = 0;
   const bool open = *reinterpret_cast<volatile unsigned long long *>(&counters[0]) == 0;
   const int64_t n_places = (brick_end - brick_begin) << split;
   const int64_t n = mark_share > 0 ? (int64_t)marks[0].y : 0;
   // the list of a place's brick; false when it is empty
   auto brick_of = [&](int64_t place, MarkCtx &C) -> bool {
      const int64_t brick = brick_begin + (place >> split);
      const unsigned j1 = min(offsets[brick + 1], n_pairs), j0 = min(offsets[brick], j1);
      if (j0 == j1)
         return false;
      C.p = brick_place(tiles, n_tiles, brick);
      C.n_seg = j1 - j0;
      C.list = list + j0;
      C.segs = segs;
      C.layers = layers + C.p.T->layer_base;
      C.label = labels[C.p.tile];
      C.vec = vecs[C.p.tile];
      C.multi = open && C.p.T->n_bundles > 1;
      return true;
   };
   const int parts = (int)kMarkList / part;
   for (int64_t u = warp; u < n * parts; u += n_warps) {
      const unsigned at = directory[u % n];
      const int g = (int)(u / n) * part;
      MarkCtx C;
      if ((at & kNoRecord) || !brick_of(marks[at].x, C))
         continue;
      const int total = min((int)marks[at].y, g + part);
      const unsigned short *voxel = reinterpret_cast<const unsigned short *>(marks + at + 1);
      for (int m = g; m < total; m += 32) {
         if (m + lane < total)
            W.voxel[lane] = voxel[m + lane];
         __syncwarp();
         resolve_marks(C, W, min(32, total - m), lane, n_slow, n_overlap, n_overflow);
      }
   }
   // full bricks, and where the records ran out of space those without one
   const int64_t n_full = mark_share > 0 ? (int64_t)marks[1].x : n_places;
   const int64_t n_more = mark_share > 0 && kMarkHead + (int64_t)marks[0].x > mark_share ? n : 0;
   const int halves = split ? 1 : 2;
   if (n_full + n_more > 0)
      __syncthreads();
   for (int64_t u = blockIdx.x; u < (n_full + n_more) * halves; u += gridDim.x) {
      const int64_t r = u / halves;
      int64_t place = r;
      if (r >= n_full) {
         const unsigned at = directory[r - n_full];
         if (!(at & kNoRecord))
            continue;
         place = at & ~kNoRecord;
      } else if (mark_share > 0) {
         place = directory[n_places - 1 - r];
      }
      MarkCtx C;
      if (!brick_of(place, C))
         continue;
      const int x0 = split ? (int)(place & ((1 << split) - 1)) * (kBrickX >> split)
                           : (int)(u - r * halves) * kHalfX;
      const int nx = min(C.p.nx - x0, split ? kBrickX >> split : kHalfX);
      if (nx > 0)
         resolve_full(C, scratch.full, x0, nx, n_slow, n_overlap, n_overflow);
   }
   if (n_overlap)
      atomicAdd(&counters[0], n_overlap);
   if (n_overflow)
      atomicAdd(&counters[5], n_overflow);
   if (n_slow)
      atomicAdd(&counters[9], n_slow);
}

// ------------------------------------------------------------- the brick ---
// Radial orientations a warp has still to compute.
struct RadialQueue {
   unsigned seg[64];
   unsigned short entry[64]; // voxel of the brick
};

// One CTA per brick (or 2^split, each a part of its x range): its warps share
// the brick's segments in the sweep, then its rows in the decode.  32 warps per
// SM (64 registers).  Bound by
// instruction issue (66-75% of the slots) and the shared-memory atomics: about
// a third of the time goes to the sweep, less than a third to the setup of
// bricks and segments, the rest to the decode, near half of it for the unit
// vectors of 'r' voxels.
// Segments prepared by a thread each and uniform control flow in the sweep
// against a warp's setup per segment and a branch per candidate: 397 x 283 x 77
// with 15,013 segments 218 -> 202 us, crossing 512 x 512 x 120 928 -> 880 us;
// work shared out by chunks of 32 cells instead of segments: 223 and 968 us.
// With the marked voxels in a kernel of their own (voxel_marks) against two
// sweeps with an exact evaluation of 0.9 candidates per voxel in this one:
// 523 -> 219 + 45 us and 2,216 -> 929 + 153 us; the marked voxels resolved here
// instead (a list, a queue and two barriers per brick): 330 and 1,290 us.
// LONG: the list may hold long segments (a kernel of its own: with long_part's
// call in it the kernel of the others took 888 us on the crossing volume
// instead of 866).
template <bool MULTI, bool LONG>
__global__ void __launch_bounds__(kBrickThreads<MULTI>, 1024 / kBrickThreads<MULTI>)
voxel_bricks(const SegDev *__restrict__ segs, const TileDev *__restrict__ tiles, int64_t n_tiles,
             int64_t brick_begin, int64_t brick_end, const unsigned *__restrict__ offsets,
             const unsigned *__restrict__ list, unsigned n_pairs, unsigned *__restrict__ directory,
             uint2 *__restrict__ marks, int64_t mark_share, int split,
             const LayerDev *__restrict__ layers, int32_t *const *__restrict__ labels,
             float *const *__restrict__ vecs, unsigned long long *__restrict__ counters) {
   constexpr int kThreads = kBrickThreads<MULTI>, kWarps = kThreads / 32;
   __shared__ __align__(16) unsigned skey[kBrickVoxels];
   __shared__ SweepRec s_rec[kRecs<MULTI>];
   __shared__ uint2 s_acc[MULTI ? kRecs<MULTI> : 1]; // acc_f, bundle
   __shared__ uint2 s_max[kWarps];
   __shared__ unsigned smark[MULTI ? kPlane / 4 : 1]; // a byte per (y, z), a bit per x
   // the first segments of the list: index, dec_rsq, bundle
   __shared__ unsigned s_seg[kSegCache];
   __shared__ float s_rsq[kSegCache];
   __shared__ int s_bundle[MULTI ? kSegCache : 1];
   __shared__ __align__(16) unsigned sminb[MULTI ? kBrickVoxels : 4];
   __shared__ LayerLut s_layers[MULTI ? kLayerCache : 1];
   __shared__ RadialQueue queues[kWarps];
   __shared__ unsigned short s_list[kMarkList];
   __shared__ unsigned s_next, s_marked;
   __shared__ bool s_multi;
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   unsigned long long n_slow = 0, n_overlap = 0;

   for (int64_t place = blockIdx.x; place < (brick_end - brick_begin) << split;
        place += gridDim.x) {
      const int64_t brick = brick_begin + (place >> split);
      const BrickPlace p = brick_place(tiles, n_tiles, brick);
      const int x0 = (int)(place & ((1 << split) - 1)) * (kBrickX >> split);
      const int nx = min(p.nx - x0, kBrickX >> split);
      if (nx <= 0)
         continue;
      const int ox = p.ox + x0, oy = p.oy, oz = p.oz, ny = p.ny, nz = p.nz;
      const int Y = p.T->Y, Z = p.T->Z, layer_base = p.T->layer_base;
      const int max_layer = p.T->max_layer, n_bundles = p.T->n_bundles;
      int32_t *label = labels[p.tile];
      float *vec = vecs[p.tile];
      // (clamped to the planned list size: every slot below it is written)
      const unsigned j1 = min(offsets[brick + 1], n_pairs), j0 = min(offsets[brick], j1);

      if (j0 == j1) { // no segment: background
         for (int ly = warp; ly < ny; ly += kWarps)
            for (int lx = 0; lx < nx; lx++) {
               const int64_t i0 = ((int64_t)(ox + lx) * Y + (oy + ly)) * Z + oz;
               if (lane < nz)
                  label[i0 + lane] = 0;
               if (vec)
                  for (int e = lane; e < 3 * nz; e += 32)
                     vec[3 * i0 + e] = 0.f;
            }
         continue;
      }

      const unsigned n_seg = j1 - j0;
      const uint4 none = make_uint4(kNoKey, kNoKey, kNoKey, kNoKey);
      for (int i = threadIdx.x; i < kBrickVoxels / 4; i += kThreads) {
         reinterpret_cast<uint4 *>(skey)[i] = none;
         if (MULTI)
            reinterpret_cast<uint4 *>(sminb)[i] = none;
      }
      if (MULTI && threadIdx.x < kPlane / 4)
         smark[threadIdx.x] = 0;
      {
         const int b = threadIdx.x / kMaxLayers, l = threadIdx.x % kMaxLayers;
         if (b < (MULTI ? min(kLayerCache, n_bundles) : 1)) {
            const LayerDev &L = layers[layer_base + b];
            s_layers[b].sq[l] = L.sq_fdown[l];
            if (l == 0) {
               s_layers[b].n = L.n;
               s_layers[b].models = L.models;
            }
         }
      }
      if (threadIdx.x == 0) {
         s_next = kWarps;
         s_marked = 0;
         // the overlap warning is one bit for the whole volume: once some
         // brick has raised it, the bundle minima are of no more use
         s_multi = MULTI && n_bundles > 1 &&
                   *reinterpret_cast<volatile unsigned long long *>(&counters[0]) == 0;
      }
      // the record of the list's segment j; the bound of its estimate
      auto prepare = [&](unsigned j, unsigned s) -> float {
         const SegSweep w = load_sweep(segs[s]);
         SubBox b;
         const bool any = sub_box(w, ox, oy, oz, nx, ny, nz, b); // (a brick's part may not)
         if (LONG && !any)
            b = SubBox{};
         const SegPart g = seg_part<LONG>(segs[s], w, b);
         s_rec[j % kRecs<MULTI>] = sweep_rec<LONG>(g, w.c.x, b, any, ox, oy, oz);
         if (MULTI)
            s_acc[j % kRecs<MULTI>] = make_uint2(__float_as_uint(w.c.y), (unsigned)w.e.w);
         return LONG && !any ? 0.f : g.mg;
      };
      { // the first records, and the largest bounds of the list's segments
        // (floats >= 0: bits order like values)
         unsigned th = 0, mg = 0;
         for (unsigned j = threadIdx.x; j < n_seg; j += kThreads) {
            const unsigned s = list[j0 + j];
            const SegDev &S = segs[s];
            float m = __ldg(&S.mg);
            if (j < kSegCache) {
               s_seg[j] = s;
               s_rsq[j] = __ldg(&S.dec_rsq);
               if (MULTI)
                  s_bundle[j] = __ldg(&S.bundle);
            }
            if (j < kRecs<MULTI>) {
               const float part = prepare(j, s);
               m = LONG ? part : m;
            } else if (LONG && __ldg(&S.c2f) > kLongSquared) {
               SubBox b;
               m = sub_box(load_sweep(S), ox, oy, oz, nx, ny, nz, b) ? long_part(S, b).mg : 0.f;
            }
            th = max(th, __float_as_uint(fmaf(2.0001f, m, __ldg(&S.thr_f))));
            mg = max(mg, __float_as_uint(m));
         }
         if (warp * 32 < n_seg) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
               th = max(th, __shfl_xor_sync(0xFFFFFFFFu, th, o));
               mg = max(mg, __shfl_xor_sync(0xFFFFFFFFu, mg, o));
            }
         }
         if (lane == 0)
            s_max[warp] = make_uint2(th, mg);
      }
      __syncthreads();
      unsigned th = 0, mg = 0;
#pragma unroll
      for (int i = 0; i < kWarps; i++) {
         th = max(th, s_max[i].x);
         mg = max(mg, s_max[i].y);
      }
      const BrickScale k = brick_scale(n_seg, __uint_as_float(th), __uint_as_float(mg));
      const bool multi = MULTI && s_multi;
      for (unsigned base = 0;;) {
         // sweep: warps take segments from a shared counter, the next one
         // while they are busy with one
         const unsigned n = min(n_seg - base, kRecs<MULTI>);
         for (unsigned j = warp, next; j < n; j = __shfl_sync(0xFFFFFFFFu, next, 0)) {
            if (lane == 0)
               next = atomicAdd(&s_next, 1u);
            const uint2 a = MULTI ? s_acc[j] : make_uint2(0u, 0u);
            brick_sweep<MULTI>(s_rec[j], base + j, __uint_as_float(a.x), a.y, k, multi, skey,
                               smark, sminb, lane);
         }
         base += kRecs<MULTI>;
         if (base >= n_seg)
            break;
         __syncthreads();
         if (threadIdx.x == 0)
            s_next = kWarps;
         for (unsigned e = threadIdx.x; e < min(kRecs<MULTI>, n_seg - base); e += kThreads)
            prepare(base + e, list[j0 + base + e]);
         __syncthreads();
      }
      __syncthreads();
      // decode: a warp per y, lane = z, along x: coalesced stores.  Radial
      // ('r') orientations go to the warp's queue and are computed 32 at a
      // time (a warp's row mixes 'b' and 'r' voxels: in place, half the lanes
      // would idle through the two-float unit vector).
      RadialQueue &rq = queues[warp];
      const LayerDev *tile_layers = layers + layer_base;
      int qn = 0;
      auto radial = [&](int at) {
         const int li = rq.entry[at];
         const int rx = ox + (li >> 8), ry = oy + ((li >> 5) & 7), rz = oz + (li & 31);
         float o[3];
         radial_vector(segs[rq.seg[at]], rx, ry, rz, o, n_slow);
         const int64_t i = ((int64_t)rx * Y + ry) * Z + rz;
         vec[3 * i + 0] = o[0];
         vec[3 * i + 1] = o[1];
         vec[3 * i + 2] = o[2];
      };
      for (int ly = warp; ly < ny; ly += kWarps) {
         const int yz = plane_place(ly, lane);
         const unsigned sticky = MULTI ? reinterpret_cast<const uint8_t *>(smark)[yz] : 0u;
         const int y = oy + ly, z = oz + lane;
         int64_t i = ((int64_t)ox * Y + y) * Z + z;
         for (int lx = 0; lx < nx; lx++, i += (int64_t)Y * Z) {
            const int li = lx * kPlane + yz;
            bool defer = false;
            unsigned seg = 0;
            int32_t lab = 0;
            if (lane < nz) {
               const unsigned key = skey[li];
               float o0 = 0.f, o1 = 0.f, o2 = 0.f;
               if (key != kNoKey || (MULTI && (sticky >> lx & 1u))) {
                  const unsigned slot = (key & (k.mul - 1u)) >> 1;
                  int w = -1, bundle = 0;
                  if (!(key & 1u) && !(MULTI && (sticky >> lx & 1u))) { // not marked
                     float rsq;
                     if (slot < kSegCache) {
                        seg = s_seg[slot];
                        rsq = s_rsq[slot];
                        bundle = MULTI ? s_bundle[slot] : 0;
                     } else {
                        seg = list[j0 + slot];
                        rsq = segs[seg].dec_rsq;
                        bundle = MULTI ? segs[seg].bundle : 0;
                     }
                     // 4e-6: the rounding of the quantum and of the product
                     const float up = key_bound(k, key);
                     float lo = up * (1.f - 4e-6f) - 2.f * k.quantum - k.mg2, hi = up;
                     if (!(rsq == rsq)) { // the radius changes: evaluate
                        float dist_squ;
                        if (cand_dist(segs[seg], ox + lx, y, z, dist_squ, rsq))
                           n_slow++;
                        lo = hi = dist_squ;
                        if (dist_squ > tile_layers[bundle].f_ly_squ * rsq)
                           hi = INFINITY; // outside (generator.cpp:329-331): no layer is certain
                     }
                     if (!MULTI || bundle < kLayerCache)
                        w = certain_layer(s_layers[MULTI ? bundle : 0].sq,
                                          s_layers[MULTI ? bundle : 0].n, lo, hi, rsq);
                     else
                        w = certain_layer(tile_layers[bundle].sq_fdown, tile_layers[bundle].n, lo,
                                          hi, rsq);
                  }
                  if (w >= 0) {
                     lab = w + 1 + bundle * max_layer;
                     if (MULTI && multi && sminb[li] < (unsigned)bundle)
                        n_overlap++;
                     const unsigned models = !MULTI || bundle < kLayerCache
                                                 ? s_layers[MULTI ? bundle : 0].models
                                                 : tile_layers[bundle].models;
                     const unsigned m = models >> (2 * w) & 3u;
                     if (m == 1u) {
                        o0 = segs[seg].vp[0];
                        o1 = segs[seg].vp[1];
                        o2 = segs[seg].vp[2];
                     }
                     defer = m == 2u && vec;
                  } else {
                     lab = kMarkedLabel;
                  }
               }
               label[i] = lab;
               if (vec && !defer) {
                  vec[3 * i + 0] = o0;
                  vec[3 * i + 1] = o1;
                  vec[3 * i + 2] = o2;
               }
            }
            if (lab == kMarkedLabel) {
               const unsigned at = atomicAdd(&s_marked, 1u);
               if (at < kMarkList)
                  s_list[at] = (unsigned short)((x0 + lx) * kPlane + ly * kBrickZ + lane);
            }
            const unsigned m = __ballot_sync(0xFFFFFFFFu, defer);
            if (defer) {
               const int at = qn + __popc(m & ((1u << lane) - 1u));
               rq.entry[at] = (unsigned short)(lx * kPlane + ly * kBrickZ + lane);
               rq.seg[at] = seg;
            }
            qn += __popc(m);
            if (qn >= 32) {
               __syncwarp();
               radial(qn - 32 + lane);
               qn -= 32;
               __syncwarp();
            }
         }
      }
      __syncwarp();
      if (lane < qn)
         radial(lane);
      __syncthreads();
      if (warp == 0 && s_marked && mark_share > 0) { // the brick's record
         const unsigned n = s_marked;
         const bool full = n > kMarkList;
         unsigned long long got = 0; // {entries taken, records}
         if (lane == 0) {
            if (full) {
               const int64_t last = ((brick_end - brick_begin) << split) - 1;
               directory[last - atomicAdd(&marks[1].x, 1u)] = (unsigned)place;
            } else {
               got = atomicAdd(reinterpret_cast<unsigned long long *>(marks),
                               (1ull << 32) | (1u + (n + 3u) / 4u));
            }
         }
         got = __shfl_sync(0xFFFFFFFFu, got, 0);
         const uint64_t at = (uint64_t)kMarkHead + (unsigned)got;
         const bool fits = !full && at + 1 + (n + 3) / 4 <= (uint64_t)mark_share;
         if (lane == 0 && !full) {
            directory[got >> 32] = fits ? (unsigned)at : kNoRecord | (unsigned)place;
            if (fits)
               marks[at] = make_uint2((unsigned)place, n);
         }
         if (fits)
            for (unsigned e = lane; e < n; e += 32)
               reinterpret_cast<unsigned short *>(marks + at + 1)[e] = s_list[e];
      }
      __syncthreads();
   }
   if (n_overlap)
      atomicAdd(&counters[0], n_overlap);
   if (n_slow)
      atomicAdd(&counters[9], n_slow);
}

// Small volumes are as long as their longest brick and its marks.  Up to two
// CTAs per SM a brick is swept by 2, 4 or 8 CTAs, each a part of its x range
// with the same list; up to 1,216 units (two waves of voxel_marks' CTAs if each
// held one) eight marked voxels go to a warp instead of a whole record.  Whole
// calls, two bundles, without either -> with both: 24 x 24 x 24 (9 bricks) 163 ->
// 118 us, 48 x 40 x 24 (30) 180 -> 156, 64 x 64 x 64 (128) 209 -> 177, with the
// marks alone 96 x 96 x 60 (288) 295 -> 252, 128 x 128 x 60 (512) 332 -> 284, 160 x
// 160 x 60 (800) 341 -> 313; 1,725 bricks 296 -> 301, and bricks split above 304
// units change nothing (288: 253, 512: 285) or cost (288 by four: 269).
constexpr int64_t kSplitBricks = 304, kSplitMarks = 1216;

int launch_voxel_bricks(const SegDev *segs, const int32_t *seg_tile, int64_t n_segs,
                        const TileDev *tiles, int64_t n_tiles, int64_t n_bricks, int64_t n_pairs,
                        const LayerDev *layers, bool multi_bundle, bool long_segs,
                        int32_t *const *labels, float *const *vecs, void *ws, size_t ws_bytes,
                        unsigned long long *counters,
                        cudaStream_t st, const BrickChunks *chunks) {
   if (n_tiles <= 0 || n_bricks <= 0)
      return FPGB_OK;
   if (chunks && (chunks->n < 1 || chunks->bound[0] != 0 || chunks->bound[chunks->n] != n_bricks)) {
      set_error("voxelizer: brick chunks do not cover the bricks");
      return FPGB_EINVAL;
   }
   if (n_pairs >= 0xFFFFFFFFll || n_segs >= 0xFFFFFFFFll) {
      set_error("voxelizer: %lld segment-brick pairs exceed the 32-bit lists",
                (long long)n_pairs);
      return FPGB_EINVAL;
   }
   const size_t lists = brick_list_bytes(n_bricks, n_pairs);
   if (ws_bytes < lists) {
      set_error("voxelizer: %zu bytes of scratch, %zu needed", ws_bytes, lists);
      return FPGB_ENOMEM;
   }
   char *w = static_cast<char *>(ws);
   auto *offsets = reinterpret_cast<unsigned *>(w);
   w += align_up(sizeof(unsigned) * (n_bricks + 1), 256);
   auto *counts = reinterpret_cast<unsigned *>(w);
   w += align_up(sizeof(unsigned) * std::max<int64_t>(n_bricks, 1), 256);
   auto *list = reinterpret_cast<unsigned *>(w);
   auto *marks = reinterpret_cast<uint2 *>(static_cast<char *>(ws) + lists);
   const int n_launch = chunks ? chunks->n : 1;
   // entries of one launch (kNoRecord is past every place among them)
   int64_t mark_share =
       n_launch <= 1024
           ? std::min<int64_t>((int64_t)((ws_bytes - lists) / sizeof(uint2)), 1 << 30) / n_launch
           : 0;
   if (mark_share < kMarkHead)
      mark_share = 0;

   if (n_bricks <= kSmallBricks && n_pairs <= kSmallPairs && n_segs <= kSmallPairs) {
      brick_bin_small<<<1, 1024, 0, st>>>(segs, seg_tile, (int)n_segs, tiles, (int)n_bricks,
                                          offsets, list, n_pairs, marks, mark_share, n_launch,
                                          counters);
      FPGB_CUDA_TRY(cudaGetLastError());
   } else {
      const unsigned g =
          (unsigned)std::min<int64_t>((n_segs * kBinLanes + 255) / 256, 1 << 20);
      FPGB_CUDA_TRY(cudaMemsetAsync(counts, 0, sizeof(unsigned) * n_bricks, st));
      if (n_segs > 0) {
         brick_bin<false><<<g, 256, 0, st>>>(segs, seg_tile, n_segs, tiles, counts, nullptr,
                                             nullptr, n_pairs, counters);
         FPGB_CUDA_TRY(cudaGetLastError());
      }
      brick_scan<<<1, 1024, 0, st>>>(counts, n_bricks, offsets, marks, mark_share, n_launch,
                                     counters);
      FPGB_CUDA_TRY(cudaGetLastError());
      if (n_segs > 0) {
         FPGB_CUDA_TRY(cudaMemsetAsync(counts, 0, sizeof(unsigned) * n_bricks, st));
         brick_bin<true><<<g, 256, 0, st>>>(segs, seg_tile, n_segs, tiles, counts, offsets, list,
                                            n_pairs, counters);
         FPGB_CUDA_TRY(cudaGetLastError());
      }
   }
   // (up to eight times as many places: their directory at the end of the
   // records' space)
   int split = 0;
   int64_t dir_entries = 0;
   while (n_launch == 1 && split < 3 && n_bricks << (split + 1) <= kSplitBricks &&
          mark_share > n_bricks << (split + 2)) {
      split++;
      dir_entries = ((n_bricks << split) + 1) / 2;
   }
   cudaStream_t alt = chunks && chunks->n > 1 ? chunks->alt : nullptr;
   cudaEvent_t joined[2] = {};
   auto launch_all = [&]() -> int {
      if (alt) { // alt starts after the binning
         FPGB_CUDA_TRY(cudaEventCreateWithFlags(&joined[0], cudaEventDisableTiming));
         FPGB_CUDA_TRY(cudaEventRecord(joined[0], st));
         FPGB_CUDA_TRY(cudaStreamWaitEvent(alt, joined[0], 0));
      }
      for (int c = 0; c < n_launch; c++) {
         const int64_t b0 = chunks ? chunks->bound[c] : 0;
         const int64_t b1 = chunks ? chunks->bound[c + 1] : n_bricks;
         cudaStream_t s = (alt && (c & 1)) ? alt : st;
         if (b1 > b0) {
            const int64_t n = (b1 - b0) << split;
            const unsigned grid = (unsigned)std::min<int64_t>(n, 0x7FFFFFFF);
            // a warp per record, or per part of it, a CTA per full brick, up to
            // about two waves
            const int part = n <= kSplitMarks ? 8 : (int)kMarkList;
            const unsigned mark_grid = (unsigned)std::min<int64_t>(
                n * std::max(1, (int)kMarkList / part / (kMarkThreads / 32)), 152 * 8);
            uint2 *share = marks + c * mark_share;
            const int64_t room = mark_share - dir_entries;
            unsigned *directory =
                split ? reinterpret_cast<unsigned *>(share + room) : counts + b0;
            auto kernel = multi_bundle ? long_segs ? voxel_bricks<true, true>
                                                   : voxel_bricks<true, false>
                          : long_segs  ? voxel_bricks<false, true>
                                       : voxel_bricks<false, false>;
            const int threads = multi_bundle ? kBrickThreads<true> : kBrickThreads<false>;
            kernel<<<grid, threads, 0, s>>>(segs, tiles, n_tiles, b0, b1, offsets, list,
                                            (unsigned)n_pairs, directory, share, room, split,
                                            layers, labels, vecs, counters);
            FPGB_CUDA_TRY(cudaGetLastError());
            // (unsplit, the fill's cursors have become the directory of the records)
            voxel_marks<<<mark_grid, kMarkThreads, 0, s>>>(
                segs, tiles, n_tiles, b0, b1, offsets, list, (unsigned)n_pairs, directory, share,
                room, split, part, layers, labels, vecs, counters);
            FPGB_CUDA_TRY(cudaGetLastError());
         }
         if (chunks && chunks->after)
            FPGB_TRY(chunks->after(chunks->ctx, c, s));
      }
      if (alt) { // st's later work sees every chunk
         FPGB_CUDA_TRY(cudaEventCreateWithFlags(&joined[1], cudaEventDisableTiming));
         FPGB_CUDA_TRY(cudaEventRecord(joined[1], alt));
         FPGB_CUDA_TRY(cudaStreamWaitEvent(st, joined[1], 0));
      }
      return FPGB_OK;
   };
   const int rc = launch_all();
   for (cudaEvent_t e : joined)
      if (e)
         cudaEventDestroy(e);
   return rc;
}

} // namespace fpgb
