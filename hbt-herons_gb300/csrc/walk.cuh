// walk.cuh - the tree walk (GravityTree_t::EvaluatePotential,
// src/gravity_tree.cpp:82-166) for 32 targets at a time.
//
// One warp takes 32 neighbouring targets (key order) of one subhalo.  Each
// target's interaction list is exactly the reference's: the cells its own
// opening test accepts and the leaves it reaches.  The warp finds the union
// of those lists in one traversal and evaluates it in a second phase:
//
//   traversal   A stack in shared memory holds ranges of sibling subtrees
//               (first slot, end slot, the targets still walking them).  Each
//               step pops up to 32 ranges, one per lane; a lane reads its
//               range's first node and classifies it against the bounding
//               box of the targets: every target accepts it, every target
//               opens it, or (near the opening distance) each target decides
//               with its own test.  The node becomes an entry of the
//               interaction list with the mask of the targets that accept it;
//               the rest of the range and, if some targets open the node, its
//               children (with the mask of those targets) go back on the stack.
//               Nodes of the third kind wait in a pending list; once it holds
//               32 (or the stack is empty) each lane takes one and runs every
//               target's own test on it, two targets per packed FP32x2
//               operation, which gives its entry mask and its children's.
//   evaluation  Entries go to one of three lists: "far" entries, which every
//               target sees beyond the softening length (box distance), split
//               into those that every target takes (no selection at all) and
//               the rest, and "near" ones.  Whenever a list fills, every lane reads each
//               entry (a shared-memory broadcast) and adds the term of the
//               entries its mask bit selects: -m / r for the far list with no
//               branch, and the cubic-spline softened kernel where r < h for
//               the near list.  Distances are formed two entries at a time in
//               packed FP32x2 arithmetic (each half an IEEE FP32 operation, so
//               the same values as scalar code).  Lists are padded to a multiple of
//               eight with massless entries; blocks of eight terms are summed
//               in FP32 and Kahan-added to the potential.
//
// Periodic wrap.  A wrapped separation is a - b, (a - box) - b or a -
// (b - box) (sep), and along each axis the box of 32 neighbouring targets
// nearly always takes one of the three for all of them.  Then the entry is
// stored as a or a - box, with a flag where the targets are to be taken as
// b - box, and it costs what an unwrapped one does; a cell's opening test by
// the box and the packed tests work on the same coordinates.  Only an entry
// that some targets wrap and others do not goes target by target.
//
// Opening test.  The reference opens a cell when len^2 > r^2 theta^2, with
// len^2 in float and r^2 in double from the float coordinates
// (src/gravity_tree.cpp:137-145).  Here r^2 is FP32; outside a band of 1e-6
// relative around the stored threshold len^2 / theta^2 (far wider than the
// FP32 error of r^2 and of the threshold) the FP32 comparison decides as the
// reference does, and inside the band the reference's double arithmetic
// decides.  The bounding-box classifications use the same band, and the box
// distances are computed with the same monotonic FP32 operations as each
// target's own r^2, so "every target accepts" and "every target opens" never
// disagree with a target's own test.
//
// Bounds.  Stack pushes happen only in steps that start with at most
// kWalkDrain = kWalkStack - 64 ranges (a step pops k <= 32 ranges and pushes
// at most 2k, or resolves pending nodes and pushes at most 32); above that
// the warp drains the stack one range at a time, each target walking that
// range on its own with the reference's stackless walk (no pushes).  A list
// holding more than its capacity - 40 entries after a step (at most 32 added
// per step) is evaluated, so with its padding (at most 7) it never exceeds
// its capacity.  Pending nodes are added only by steps that start with fewer
// than 32 (at most 32 added), so at most 63 wait.  Every loop advances a slot
// index strictly or shrinks the pending list.
// A node's second slot is read for leaves too: the tree array carries one
// padding slot after its last slot.
//
// Bound by instruction issue (79 % of the slots at 28 warps per SM), a little
// over half of it in the traversal.  So a step has one path for every lane
// (lanes without a range read the last one again), the three lists share one
// layout and one write, a warp's arrays lie together behind one base address,
// and the far terms use the PTX reciprocal square root that takes normal
// arguments only (rsqrt_normal).  Against a version with separate lists, per-kind
// branches and rsqrtf, on the 5e7-particle learned batch: 137.4 -> 123.7 ms a
// call; on a 5e6-particle plain batch with a halo across a box face 31.1 ->
// 29.0 ms (walk 20.9 -> 16.6 ms); a subsampled hydro call 23.5 -> 21.0 ms.
#pragma once

#include "kernels.cuh"

namespace hbtg
{
namespace
{

// List and stack capacities (per warp); the defaults are the measured best on
// GB300 (overridable at build time for sweeps).  HBTG_WALK_MIN_BLOCKS, when
// defined, adds a minimum of resident blocks to the launch bounds (a register
// cap); by default the compiler's own allocation (72 registers, 7 blocks of 4
// warps per SM, limited equally by registers and shared memory) is kept.
#ifndef HBTG_WALK_FULL
#define HBTG_WALK_FULL 96
#endif
#ifndef HBTG_WALK_STACK
#define HBTG_WALK_STACK 256
#endif
constexpr int kWalkWarps = 4;   // warps per block
constexpr int kWalkFull = HBTG_WALK_FULL; // far-list entries that every target takes, per warp
constexpr int kWalkFar = 64;    // other far-list entries per warp
constexpr int kWalkNear = 64;   // near-list entries per warp
constexpr int kWalkStack = HBTG_WALK_STACK; // traversal ranges per warp
constexpr int kWalkDrain = kWalkStack - 64; // a deeper stack is drained (a step pushes at most 2 per lane)
constexpr int kWalkPending = 64; // cells waiting for the targets' own opening tests
constexpr int kWalkWarp2 = 16;  // target pairs per warp
constexpr int kFlushMargin = 40; // a list is evaluated once it holds more than capacity - this
constexpr float kBandLo = 1.f - 1e-6f, kBandHi = 1.f + 1e-6f;

// Per-lane walk counters (counted calls): see kWalkCounters.
struct WalkCount
{
  unsigned long long v[kWalkCounters];
};

// Lane 0 adds the clock cycles since t to counter q (counted calls only).
template <bool Count>
__device__ __forceinline__ void tick(WalkCount &cnt, int q, long long &t, int lane)
{
  if (!Count)
    return;
  const long long now = clock64();
  if (lane == 0)
    cnt.v[q] += (unsigned long long)(now - t);
  t = now;
}

// Entry lists of one warp, in one array of pairs (a = (x0, x1, y0, y1),
// b = (z0, z1, -m0, -m1), two entries per packed operation): the far entries
// that every target takes, the other far entries, the near ones.  The last
// two have target masks; a wrapped walk, which lists every entry as near,
// keeps its wrap flags in the far list's words.
constexpr int kFarAt = kWalkFull, kNearAt = kWalkFull + kWalkFar, kWalkEntries = kNearAt + kWalkNear;

// Everything of a warp lies together, so one base address serves it all.
struct WalkWarp
{
  float4 a[kWalkEntries / 2];
  float4 b[kWalkEntries / 2];
  unsigned mask[kWalkFar + kWalkNear];
  int2 ie[kWalkStack];      // range: first slot, end slot
  unsigned im[kWalkStack];  //        targets still walking it
  int2 pend[kWalkPending];  // pending cell: slot, targets that reach it
  float4 txy[kWalkWarp2];   // targets, negated, in pairs: (x0, x1, y0, y1)
  float2 tz[kWalkWarp2];    //                             (z0, z1)
};

// a - b, with the periodic wrap of NEAREST (src/config_parser.h:218-219)
// formed without rounding the large intermediate a - b +- box: for a wrapped
// difference, a - box (or b - box) is exact (that operand is above half the
// box) and the result rounds once.
template <bool Wrap>
__device__ __forceinline__ float sep(float a, float b, const KParams &K)
{
  const float d = __fsub_rn(a, b);
  if (!Wrap)
    return d;
  return d > K.half ? __fsub_rn(__fsub_rn(a, K.box), b) : (d < -K.half ? __fsub_rn(a, __fsub_rn(b, K.box)) : d);
}

__device__ __forceinline__ float dist2(float dx, float dy, float dz)
{
  return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

// The reference's opening decision in its own arithmetic: float len^2
// against r^2 theta^2 in double, r^2 from the float coordinates.
__device__ __noinline__ bool opens_exact(float cx, float cy, float cz, float lenf, float tx, float ty, float tz,
                                         int periodic, float box, float half, float theta2)
{
  double d[3] = {(double)cx - (double)tx, (double)cy - (double)ty, (double)cz - (double)tz}; // exact
  if (periodic)
    for (int q = 0; q < 3; q++)
      d[q] = nearest_d(d[q], (double)half, (double)box);
  const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(d[0], d[0]), __dmul_rn(d[1], d[1])), __dmul_rn(d[2], d[2]));
  return (double)__fmul_rn(lenf, lenf) > __dmul_rn(r2, (double)theta2);
}

// One target's test of a cell (centre c, threshold crit = len^2/theta^2).
template <bool Wrap>
__device__ __forceinline__ bool target_opens(float cx, float cy, float cz, float crit, float lenf, float tx, float ty,
                                             float tz, const KParams &K)
{
  const float r2 = dist2(sep<Wrap>(cx, tx, K), sep<Wrap>(cy, ty, K), sep<Wrap>(cz, tz, K));
  if (r2 < __fmul_rn(crit, kBandLo))
    return true;
  if (r2 > __fmul_rn(crit, kBandHi))
    return false;
  return opens_exact(cx, cy, cz, lenf, tx, ty, tz, K.periodic, K.box, K.half, K.theta2);
}

// Target t of the warp from the negated pairs.
__device__ __forceinline__ void target_at(const float4 *txy, const float2 *tz, int t, float &x, float &y, float &z)
{
  const float4 P = txy[t >> 1];
  const float2 Z = tz[t >> 1];
  const bool h = (t & 1) != 0;
  x = -(h ? P.y : P.x);
  y = -(h ? P.w : P.z);
  z = -(h ? Z.y : Z.x);
}

// Every target's own decision on one cell (centre c, threshold crit, side
// lenf): bit t set when target t (of the mask m) opens it.  Two targets per
// packed operation; each half is the FP32 operation of target_opens (c + (-t)
// is c - t exactly), so the decisions are the same; the sign of r^2 minus the
// band's edge is the comparison, shifted into the mask (r^2 = NaN, from
// coordinates that are not finite, decides nothing of use either way).  With
// Wrap, c is the cell as all targets see it (wrap_cell) and a target's
// coordinate along the axes of `flags` is taken less one box.
template <bool Wrap>
__device__ __forceinline__ unsigned opens_mask(const float4 *txy, const float2 *tz, float cx, float cy, float cz,
                                               float crit, float lenf, unsigned m, unsigned flags, float ox, float oy,
                                               float oz, const KParams &K)
{
  const float lo = __fmul_rn(crit, kBandLo), hi = __fmul_rn(crit, kBandHi);
  const float2 c_x = make_float2(cx, cx), c_y = make_float2(cy, cy), c_z = make_float2(cz, cz);
  const float2 nlo = make_float2(-lo, -lo), nhi = make_float2(-hi, -hi);
  unsigned O = 0u, B = 0u; // nearer than the band; not beyond the band's far edge
#pragma unroll
  for (int q = kWalkWarp2 - 1; q >= 0; q--)
  {
    float4 P = txy[q];
    float2 Z = tz[q];
    if (Wrap && flags)
    { // -(t - box), rounded as t - box is
      if (flags & 1u)
      {
        P.x = __fadd_rn(P.x, K.box);
        P.y = __fadd_rn(P.y, K.box);
      }
      if (flags & 2u)
      {
        P.z = __fadd_rn(P.z, K.box);
        P.w = __fadd_rn(P.w, K.box);
      }
      if (flags & 4u)
      {
        Z.x = __fadd_rn(Z.x, K.box);
        Z.y = __fadd_rn(Z.y, K.box);
      }
    }
    const float2 dx = __fadd2_rn(c_x, make_float2(P.x, P.y));
    const float2 dy = __fadd2_rn(c_y, make_float2(P.z, P.w));
    const float2 dz = __fadd2_rn(c_z, Z);
    float2 r2 = __fmul2_rn(dx, dx);
    r2 = __ffma2_rn(dy, dy, r2);
    r2 = __ffma2_rn(dz, dz, r2);
    const float2 u = __fadd2_rn(r2, nlo), v = __fadd2_rn(nhi, r2);
    O = __funnelshift_l(__float_as_uint(u.y), O, 1); // (O << 1) | (r2.y < lo)
    O = __funnelshift_l(__float_as_uint(u.x), O, 1);
    B = __funnelshift_l(__float_as_uint(v.y), B, 1); // (B << 1) | (r2.y < hi)
    B = __funnelshift_l(__float_as_uint(v.x), B, 1);
  }
  O &= m;
  // inside the band: the reference's double arithmetic
  for (unsigned r = B & m & ~O; r; r &= r - 1u)
  {
    const int t = __ffs(r) - 1;
    float tx, ty, tzz;
    target_at(txy, tz, t, tx, ty, tzz);
    if (opens_exact(ox, oy, oz, lenf, tx, ty, tzz, K.periodic, K.box, K.half, K.theta2))
      O |= 1u << t;
  }
  return O;
}

// The same one target at a time, for a cell that some targets wrap and others
// do not.
__device__ __forceinline__ unsigned opens_mask_each(const float4 *txy, const float2 *tz, float cx, float cy, float cz,
                                                    float crit, float lenf, unsigned m, const KParams &K)
{
  unsigned O = 0u;
  for (unsigned r = m; r; r &= r - 1u)
  {
    const int t = __ffs(r) - 1;
    float tx, ty, tzz;
    target_at(txy, tz, t, tx, ty, tzz);
    if (target_opens<true>(cx, cy, cz, crit, lenf, tx, ty, tzz, K))
      O |= 1u << t;
  }
  return O;
}

// Axis by axis, how the targets' box [lo, hi] wraps against coordinate c
// (sep's comparisons at the box's ends; c - t is monotonic in t): returns the
// coordinate to store and adds to `flags` bit d where the targets are taken
// less one box, or kMixed where they differ.
constexpr unsigned kMixed = 8u;
__device__ __forceinline__ float wrap_axis(float c, float lo, float hi, int d, unsigned &flags, const KParams &K)
{
  const float dmin = __fsub_rn(c, hi), dmax = __fsub_rn(c, lo);
  if (dmin > K.half)
    return __fsub_rn(c, K.box);
  if (dmax < -K.half)
    flags |= 1u << d;
  else if (dmax > K.half || dmin < -K.half)
    flags |= kMixed;
  return c;
}

// Smallest and largest squared distance from a point to the targets' box.
__device__ __forceinline__ void box_dist2(const float *lo, const float *hi, float x, float y, float z, float &near2,
                                          float &far2)
{
  const float l[3] = {__fsub_rn(lo[0], x), __fsub_rn(lo[1], y), __fsub_rn(lo[2], z)};
  const float h[3] = {__fsub_rn(x, hi[0]), __fsub_rn(y, hi[1]), __fsub_rn(z, hi[2])};
  near2 = dist2(fmaxf(fmaxf(l[0], h[0]), 0.f), fmaxf(fmaxf(l[1], h[1]), 0.f), fmaxf(fmaxf(l[2], h[2]), 0.f));
  far2 = dist2(fmaxf(fabsf(l[0]), fabsf(h[0])), fmaxf(fabsf(l[1]), fabsf(h[1])), fmaxf(fabsf(l[2]), fabsf(h[2])));
}

// 1 / sqrt of a positive number that is not subnormal.  The PTX instruction is
// documented to be within 2^-22.9 (relative) over the positive floats, and with
// .ftz to take a subnormal argument for zero; the far entries lie beyond the
// softening length, so their squared distances are at least h2s, which is normal.
__device__ __forceinline__ float rsqrt_normal(float x)
{
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The potential term of one entry for one target at squared distance r2.
__device__ __forceinline__ float softened_term(float m, float r2, const KParams &K, float h2)
{
  return r2 >= h2 ? -m * rsqrtf(r2) : m * K.h_inv * spline_w(sqrtf(r2) * K.h_inv);
}

__device__ __forceinline__ void kahan_add(float &sum, float &comp, float v)
{
  const float y = v - comp;
  const float t = sum + y;
  comp = (t - sum) - y;
  sum = t;
}

// A massless entry far from every target (finite terms, so the evaluation
// loops need no guard).
constexpr float kFarAway = 3e18f;

// Writes entry k (pair layout).
__device__ __forceinline__ void entry_put(float4 *ea, float4 *eb, int k, float x, float y, float z, float nm)
{
  float *A = reinterpret_cast<float *>(ea + (k >> 1)) + (k & 1), *B = reinterpret_cast<float *>(eb + (k >> 1)) + (k & 1);
  A[0] = x;
  A[2] = y;
  B[0] = z;
  B[2] = nm;
}

// Pads the list that starts at entry `at` and holds n to a multiple of eight
// with massless entries; returns the padded length.  The caller leaves room
// for seven more entries.
__device__ __forceinline__ int pad8(float4 *ea, float4 *eb, unsigned *mask, int at, int n, int lane)
{
  const int padded = (n + 7) & ~7;
  if (n + lane < padded)
  {
    entry_put(ea, eb, at + n + lane, kFarAway, kFarAway, kFarAway, 0.f);
    if (at >= kFarAt)
      mask[at - kFarAt + n + lane] = 0u;
  }
  __syncwarp();
  return padded;
}

// Squared distances of entry pair (A, B) from a target (negated coordinates,
// entry + (-target) is exact as a subtraction).
__device__ __forceinline__ float2 pair_r2(const float4 &A, const float4 &B, float2 ntx, float2 nty, float2 ntz)
{
  const float2 dx = __fadd2_rn(make_float2(A.x, A.y), ntx);
  const float2 dy = __fadd2_rn(make_float2(A.z, A.w), nty);
  const float2 dz = __fadd2_rn(make_float2(B.x, B.y), ntz);
  float2 r2 = __fmul2_rn(dx, dx);
  r2 = __ffma2_rn(dy, dy, r2);
  return __ffma2_rn(dz, dz, r2);
}

// Far lists: every target is at least one softening length from every entry
// (never used for wrapped subhaloes).  Masked: only the targets of an entry's
// mask take it.
template <bool Masked>
__device__ __forceinline__ void eval_far(const float4 *ea, const float4 *eb, const unsigned *mask, int n,
                                         unsigned lanebit, float tx, float ty, float tz, float &sum, float &comp)
{
  const float2 ntx = make_float2(-tx, -tx), nty = make_float2(-ty, -ty), ntz = make_float2(-tz, -tz);
  const uint2 *fm = reinterpret_cast<const uint2 *>(mask);
  for (int i = 0; i < n; i += 8)
  {
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
      const int pp = (i >> 1) + q;
      const float4 A = ea[pp], B = eb[pp];
      const float2 r2 = pair_r2(A, B, ntx, nty, ntz);
      const float2 rs = make_float2(rsqrt_normal(r2.x), rsqrt_normal(r2.y));
      float2 nm = make_float2(B.z, B.w);
      if (Masked)
      {
        const uint2 mk = fm[pp];
        nm = make_float2((mk.x & lanebit) ? B.z : 0.f, (mk.y & lanebit) ? B.w : 0.f);
      }
      acc = __ffma2_rn(nm, rs, acc);
    }
    kahan_add(sum, comp, acc.x + acc.y);
  }
}

// One near entry's term: the softened form where the target is inside the
// softening length.  h2s >= h2 keeps subnormal r2 out of rsqrt_normal.
__device__ __forceinline__ float near_term(float nm, float r2, const KParams &K, float h2, float h2s)
{
  float v = __fmul_rn(nm, rsqrt_normal(r2));
  if (r2 < h2s)
    v = softened_term(-nm, r2, K, h2);
  return v;
}

// Squared distances of a pair of wrapped entries with flags f (wrap_axis).
__device__ __forceinline__ float2 pair_r2_wrapped(const float4 &A, const float4 &B, uint2 f, float tx, float ty, float tz,
                                                  const KParams &K)
{
  float r[2];
#pragma unroll
  for (int e = 0; e < 2; e++)
  {
    const unsigned fe = e ? f.y : f.x;
    const float ex = e ? A.y : A.x, ey = e ? A.w : A.z, ez = e ? B.y : B.x;
    if (fe & kMixed)
      r[e] = dist2(sep<true>(ex, tx, K), sep<true>(ey, ty, K), sep<true>(ez, tz, K));
    else
      r[e] = dist2(__fsub_rn(ex, (fe & 1u) ? __fsub_rn(tx, K.box) : tx),
                   __fsub_rn(ey, (fe & 2u) ? __fsub_rn(ty, K.box) : ty),
                   __fsub_rn(ez, (fe & 4u) ? __fsub_rn(tz, K.box) : tz));
  }
  return make_float2(r[0], r[1]);
}

// Near list: the softened kernel where r < h (src/gravity_tree.cpp:150-162).
// Near entries are those within h of the targets' box, so most eights of them
// lie beyond h of every target itself: one vote settles that for the eight,
// and their terms need no branch each (with a vote and a branch per entry a
// near entry took 280 cycles of its warp on a 5e6-particle plain batch, a
// masked far one 45; now 208, and 99 instead of 190 on a subsampled one).  A
// target that an entry's mask leaves out counts as infinitely far: often it is
// inside h of a cell that it opened, and its term is zero either way (5e7
// particles 110.1 -> 109.0 ms a call, the 5e6 batch 24.60 -> 24.37).
// With Wrap, `flags` holds how the targets take each entry (wrap_axis).
template <bool Wrap>
__device__ __forceinline__ void eval_near(const float4 *ea, const float4 *eb, const unsigned *mask,
                                          const unsigned *flags, int n, unsigned lanebit, float tx, float ty, float tz,
                                          const KParams &K, float h2, float h2s, float &sum, float &comp)
{
  const float2 ntx = make_float2(-tx, -tx), nty = make_float2(-ty, -ty), ntz = make_float2(-tz, -tz);
  const uint2 *nm2 = reinterpret_cast<const uint2 *>(mask), *nf2 = reinterpret_cast<const uint2 *>(flags);
  for (int i = 0; i < n; i += 8)
  {
    float r2[8], nm[8];
#pragma unroll
    for (int q = 0; q < 4; q++)
    {
      const int pp = (i >> 1) + q;
      const float4 A = ea[pp], B = eb[pp];
      const uint2 mk = nm2[pp];
      float2 r;
      if (Wrap)
      {
        const uint2 f = nf2[pp];
        r = (f.x | f.y) == 0u ? pair_r2(A, B, ntx, nty, ntz) : pair_r2_wrapped(A, B, f, tx, ty, tz, K);
      }
      else
        r = pair_r2(A, B, ntx, nty, ntz);
      const bool take0 = (mk.x & lanebit) != 0u, take1 = (mk.y & lanebit) != 0u;
      r2[2 * q] = take0 ? r.x : INFINITY;
      r2[2 * q + 1] = take1 ? r.y : INFINITY;
      nm[2 * q] = take0 ? B.z : 0.f;
      nm[2 * q + 1] = take1 ? B.w : 0.f;
    }
    const float least = fminf(fminf(fminf(r2[0], r2[1]), fminf(r2[2], r2[3])),
                              fminf(fminf(r2[4], r2[5]), fminf(r2[6], r2[7])));
    float part = 0.f;
    if (__any_sync(0xffffffffu, least < h2s))
    {
#pragma unroll
      for (int q = 0; q < 8; q++)
        part = __fadd_rn(part, near_term(nm[q], r2[q], K, h2, h2s));
    }
    else
    {
#pragma unroll
      for (int q = 0; q < 8; q++)
        part = __fadd_rn(part, __fmul_rn(nm[q], rsqrt_normal(r2[q])));
    }
    kahan_add(sum, comp, part);
  }
}

// A tree slot; Fresh: the tree may have been written by this kernel, or lie in
// shared memory, so not through the read-only path.
template <bool Fresh>
__device__ __forceinline__ float4 tree_slot(const float4 *p)
{
  return Fresh ? *p : __ldg(p);
}

// The reference's stackless walk of one range [a, e) of sibling subtrees for
// one target (open: next slot; accept: interact and skip the subtree).
template <bool Wrap, bool Fresh>
__device__ __forceinline__ void walk_range(const float4 *T, int a, int e, float tx, float ty, float tz,
                                           const KParams &K, float h2, float &sum, float &comp, WalkCount &cnt)
{
  int idx = a;
  while (idx < e)
  {
    const float4 n = tree_slot<Fresh>(&T[idx]);
    float m;
    int next;
    if (slot_is_cell(n.w))
    {
      const float4 b = tree_slot<Fresh>(&T[idx + 1]);
      const float crit = __uint_as_float(__float_as_uint(n.w) & 0x7fffffffu);
      if (target_opens<Wrap>(n.x, n.y, n.z, crit, b.z, tx, ty, tz, K))
      {
        idx += 2;
        continue;
      }
      m = b.x;
      next = __float_as_int(b.y);
    }
    else
    {
      m = n.w;
      next = idx + 1;
    }
    const float r2 = dist2(sep<Wrap>(n.x, tx, K), sep<Wrap>(n.y, ty, K), sep<Wrap>(n.z, tz, K));
    kahan_add(sum, comp, softened_term(m, r2, K, h2));
    cnt.v[0]++;
    idx = max(next, idx + 1);
  }
}

// Potentials of (up to) 32 targets in the tree T with the given root slot: the
// calling warp's lane holds target particle p at x (mass in w) with its self
// term; valid = false: no target.
template <bool Wrap, bool Count, bool Fresh>
__device__ __forceinline__ void walk_group(const float4 *T, float *pot, const KParams &K, int root, int lane, bool valid,
                                           int p, float4 x, float self, WalkWarp &sh, WalkCount &cnt)
{
  float4 *ea = sh.a, *eb = sh.b;
  unsigned *mask = sh.mask;
  int2 *ie = sh.ie, *pend = sh.pend;
  unsigned *im = sh.im;
  const unsigned full = 0xffffffffu, lanebit = 1u << lane, below = lanebit - 1u;
  const float h2 = K.h * K.h, h2s = fmaxf(h2, 1.17549435e-38f); // far entries: r^2 not subnormal
  long long t_all = Count ? clock64() : 0, t = t_all;
  const unsigned vmask = __ballot_sync(full, valid);
  // bounding box of the targets
  float lo[3] = {valid ? x.x : INFINITY, valid ? x.y : INFINITY, valid ? x.z : INFINITY};
  float hi[3] = {valid ? x.x : -INFINITY, valid ? x.y : -INFINITY, valid ? x.z : -INFINITY};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int d = 0; d < 3; d++)
    {
      lo[d] = fminf(lo[d], __shfl_xor_sync(full, lo[d], o));
      hi[d] = fmaxf(hi[d], __shfl_xor_sync(full, hi[d], o));
    }
  float sum = valid ? self / K.soft : 0.f, comp = 0.f;
  if (lane == 0)
  {
    ie[0] = make_int2(root, __float_as_int(tree_slot<Fresh>(&T[root + 1]).y));
    im[0] = vmask;
  }
  // the targets, negated, in pairs (the pending cells' tests read them)
  {
    float *X = reinterpret_cast<float *>(sh.txy), *Z = reinterpret_cast<float *>(sh.tz);
    const int q = lane >> 1, hh = lane & 1;
    X[4 * q + hh] = valid ? -x.x : 0.f;
    X[4 * q + 2 + hh] = valid ? -x.y : 0.f;
    Z[2 * q + hh] = valid ? -x.z : 0.f;
  }
  int sp = 1, np = 0, nf = 0, ng = 0, nn = 0;
  __syncwarp();
  tick<Count>(cnt, 8, t, lane);
  while (sp > 0 || np > 0)
  {
    if (sp > kWalkDrain)
    { // drain: each target walks the top range on its own
      sp--;
      const int2 r = ie[sp];
      const unsigned m = im[sp];
      __syncwarp();
      if (m & lanebit)
        walk_range<Wrap, Fresh>(T, r.x, r.y, x.x, x.y, x.z, K, h2, sum, comp, cnt);
      if (Count && lane == 0)
        cnt.v[7]++;
      tick<Count>(cnt, 14, t, lane);
      continue;
    }
    // Every lane reads a node (lanes past the last one read the last again,
    // with no targets), so the step has no branches but its two kinds.
    const bool resolve = np >= kWarp || sp == 0;
    const int k = min(resolve ? np : sp, kWarp);
    int a, e = 0;
    unsigned m;
    if (resolve)
    { // pending cells, one per lane, each against every target
      const int2 q = pend[np - k + min(lane, k - 1)];
      a = q.x;
      m = lane < k ? (unsigned)q.y : 0u;
      np -= k;
      if (Count && lane == 0)
        cnt.v[3]++;
    }
    else
    { // the first nodes of up to 32 ranges, one per lane
      sp -= k;
      const int at = sp + min(lane, k - 1);
      const int2 r = ie[at];
      a = r.x;
      e = r.y;
      m = lane < k ? im[at] : 0u;
      if (Count && lane == 0)
      {
        cnt.v[1]++;
        cnt.v[2] += k;
      }
    }
    __syncwarp();
    float4 na = tree_slot<Fresh>(&T[a]);
    const float4 nb = tree_slot<Fresh>(&T[a + 1]); // a cell's mass, skip and side length (the tree has a padding slot)
    const bool cell = slot_is_cell(na.w);
    const float crit = __uint_as_float(__float_as_uint(na.w) & 0x7fffffffu);
    const float ox = na.x, oy = na.y, oz = na.z; // the node's own centre
    bool near = true;
    unsigned A, O, flags = 0u;
    float near2 = 0.f, far2 = 0.f;
    if (Wrap)
    { // the node, and the box, as the targets see each other
      float wl[3] = {lo[0], lo[1], lo[2]}, wh[3] = {hi[0], hi[1], hi[2]};
      na.x = wrap_axis(na.x, lo[0], hi[0], 0, flags, K);
      na.y = wrap_axis(na.y, lo[1], hi[1], 1, flags, K);
      na.z = wrap_axis(na.z, lo[2], hi[2], 2, flags, K);
      if (flags & kMixed)
      {
        na.x = ox;
        na.y = oy;
        na.z = oz;
      }
      else
      {
#pragma unroll
        for (int d = 0; d < 3; d++)
          if (flags & (1u << d))
          {
            wl[d] = __fsub_rn(lo[d], K.box);
            wh[d] = __fsub_rn(hi[d], K.box);
          }
        if (resolve)
          box_dist2(wl, wh, na.x, na.y, na.z, near2, far2);
      }
    }
    else
    {
      box_dist2(lo, hi, na.x, na.y, na.z, near2, far2);
      near = near2 < h2s;
    }
    if (resolve)
    {
      e = __float_as_int(nb.y); // the cell's siblings are on the stack already
      if (Wrap)
      { // the box may decide for every target; else each does
        O = 0u;
        if (flags & kMixed)
          O = opens_mask_each(sh.txy, sh.tz, ox, oy, oz, crit, nb.z, m, K);
        else if (!(near2 > __fmul_rn(crit, kBandHi)))
          O = far2 < __fmul_rn(crit, kBandLo)
                ? m
                : opens_mask<true>(sh.txy, sh.tz, na.x, na.y, na.z, crit, nb.z, m, flags, ox, oy, oz, K);
      }
      else
        O = opens_mask<false>(sh.txy, sh.tz, na.x, na.y, na.z, crit, nb.z, m, 0u, ox, oy, oz, K);
      A = m & ~O;
      tick<Count>(cnt, 9, t, lane);
    }
    else
    {
      // every target accepts it (a leaf, or the box beyond the opening
      // distance), every target opens it, or each decides on its own: cells
      // near the targets' opening distance wait for a batch of their own
      const bool acc = !cell || (!Wrap && near2 > __fmul_rn(crit, kBandHi));
      const bool opn = !Wrap && far2 < __fmul_rn(crit, kBandLo);
      A = acc ? m : 0u;
      O = !acc && opn ? m : 0u;
      const bool wait = !acc && !opn && m != 0u;
      const unsigned bp = __ballot_sync(full, wait);
      if (wait)
        pend[np + __popc(bp & below)] = make_int2(a, (int)m);
      np += __popc(bp);
      tick<Count>(cnt, 8, t, lane);
    }
    const bool to_near = Wrap || near, every = A == vmask;
    const unsigned be = __ballot_sync(full, A != 0u);
    if (be)
    {
      const unsigned bn = be & (Wrap ? full : __ballot_sync(full, near)),
                     bg = Wrap ? 0u : be & ~bn & __ballot_sync(full, every), bf = be & ~bn & ~bg;
      if (A != 0u)
      {
        const int at = to_near ? kNearAt + nn + __popc(bn & below)
                               : (every ? ng + __popc(bg & below) : kFarAt + nf + __popc(bf & below));
        entry_put(ea, eb, at, na.x, na.y, na.z, -(cell ? nb.x : na.w));
        if (at >= kFarAt)
          mask[at - kFarAt] = A;
        if (Wrap)
          mask[at - kNearAt] = flags;
        if (Count)
          cnt.v[0] += __popc(A);
      }
      if (Count && lane == 0)
      {
        cnt.v[4] += __popc(bg);
        cnt.v[5] += __popc(bf);
        cnt.v[6] += __popc(bn);
      }
      ng += __popc(bg);
      nf += __popc(bf);
      nn += __popc(bn);
    }
    // the rest of each range, then the children of opened cells (popped first: depth first)
    const int next = cell ? __float_as_int(nb.y) : a + 1;
    const bool has_sib = m != 0u && next < e, has_kid = O != 0u;
    const unsigned bs = __ballot_sync(full, has_sib), bk = __ballot_sync(full, has_kid);
    if (has_sib)
    {
      const int at = sp + __popc(bs & below);
      ie[at] = make_int2(next, e);
      im[at] = m;
    }
    sp += __popc(bs);
    if (has_kid)
    {
      const int at = sp + __popc(bk & below);
      ie[at] = make_int2(a + 2, next);
      im[at] = O;
    }
    sp += __popc(bk);
    __syncwarp();
    tick<Count>(cnt, 10, t, lane);
    if (!Wrap && ng > kWalkFull - kFlushMargin)
    {
      eval_far<false>(ea, eb, nullptr, pad8(ea, eb, mask, 0, ng, lane), lanebit, x.x, x.y, x.z, sum, comp);
      ng = 0;
      __syncwarp();
      tick<Count>(cnt, 11, t, lane);
    }
    if (!Wrap && nf > kWalkFar - kFlushMargin)
    {
      eval_far<true>(ea + kFarAt / 2, eb + kFarAt / 2, mask, pad8(ea, eb, mask, kFarAt, nf, lane), lanebit, x.x, x.y,
                     x.z, sum, comp);
      nf = 0;
      __syncwarp();
      tick<Count>(cnt, 12, t, lane);
    }
    if (nn > kWalkNear - kFlushMargin)
    {
      eval_near<Wrap>(ea + kNearAt / 2, eb + kNearAt / 2, mask + kWalkFar, mask, pad8(ea, eb, mask, kNearAt, nn, lane),
                      lanebit, x.x, x.y, x.z, K, h2, h2s, sum, comp);
      nn = 0;
      __syncwarp();
      tick<Count>(cnt, 13, t, lane);
    }
  }
  if (!Wrap)
  {
    eval_far<false>(ea, eb, nullptr, pad8(ea, eb, mask, 0, ng, lane), lanebit, x.x, x.y, x.z, sum, comp);
    tick<Count>(cnt, 11, t, lane);
    eval_far<true>(ea + kFarAt / 2, eb + kFarAt / 2, mask, pad8(ea, eb, mask, kFarAt, nf, lane), lanebit, x.x, x.y, x.z,
                   sum, comp);
    tick<Count>(cnt, 12, t, lane);
  }
  eval_near<Wrap>(ea + kNearAt / 2, eb + kNearAt / 2, mask + kWalkFar, mask, pad8(ea, eb, mask, kNearAt, nn, lane),
                  lanebit, x.x, x.y, x.z, K, h2, h2s, sum, comp);
  __syncwarp();
  tick<Count>(cnt, 13, t, lane);
  t = t_all;
  tick<Count>(cnt, 15, t, lane);
  if (valid)
    pot[p] = (sum - comp) * K.G_over_a;
}

// One 32-target chunk: its subhalo, targets and self terms (as the
// reference: a target that is a tree source starts from +m/soft, cancelling
// its own leaf, src/gravity_tree.cpp:98-101).
template <bool Count>
__device__ __forceinline__ void walk_chunk(const DevState &D, const KParams &K, int c, int lane, WalkWarp &sh,
                                           WalkCount &cnt)
{
  const int s = find_segment_warp(D.chunk_off, D.S, c); // c is the same on every lane
  const int t = (c - D.chunk_off[s]) * kWarp + lane;
  const bool valid = t < D.tgt_cnt[s];
  const bool corr = D.corr[s] != 0;
  const int ngrav = D.ngrav[s];
  int p = 0;
  if (valid) // correction: key-ordered bound set; subsampled: every candidate; else the sources
    p = corr ? D.tgt[D.off[s] + t] : (ngrav ? D.ord[D.off[s] + t] : (int)D.val[D.src_off[s] + t]);
  const float4 x = valid ? D.pm[p] : make_float4(0.f, 0.f, 0.f, 0.f);
  const int nself = (corr && D.self_cnt) ? D.self_cnt[s] : 0;
  const float self =
    !valid ? 0.f : (corr ? (t < nself ? x.w : 0.f) : (ngrav ? (t < ngrav ? source_mass(D, s, p) : 0.f) : x.w));
  if (D.src_cnt[s] == 0)
  { // no sources this iteration: zero potential
    if (valid)
      D.pot[p] = 0.f;
    return;
  }
  const int root = D.src_off[s] + 2 * D.X[D.src_off[s]];
  if (D.wrap[s])
    walk_group<true, Count, false>(D.nodes, D.pot, K, root, lane, valid, p, x, self, sh, cnt);
  else
    walk_group<false, Count, false>(D.nodes, D.pot, K, root, lane, valid, p, x, self, sh, cnt);
}

// With walk counters, the chunks (key order) are split into `nranges`
// contiguous ranges of `per` chunks, one per SM (the host picks nranges so
// that every range holds a chunk): the warps resident on an SM take the
// chunks of their own range in order, so they walk neighbouring targets and
// share the tree slots in L1; a warp whose range is used up moves on to the
// next ranges (each tried once).  Without counters, a grid-stride loop.
template <bool Count>
#ifdef HBTG_WALK_MIN_BLOCKS
__global__ void __launch_bounds__(32 * kWalkWarps, HBTG_WALK_MIN_BLOCKS)
#else
__global__ void __launch_bounds__(32 * kWalkWarps)
#endif
  k_walk(DevState D, KParams K, int total_chunks, int nranges)
{
  __shared__ WalkWarp shared[kWalkWarps];
  const int lane = threadIdx.x & 31;
  WalkWarp &sh = shared[threadIdx.x >> 5];
  WalkCount cnt = {};
  if (D.walk_ctr)
  {
    unsigned smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    const int per = (total_chunks + nranges - 1) / nranges;
    int r = (int)(smid % (unsigned)nranges);
    for (int tries = 0; tries < nranges;)
    {
      int got = 0;
      if (lane == 0)
        got = (int)atomicAdd(&D.walk_ctr[r], 1u);
      got = __shfl_sync(0xffffffffu, got, 0);
      const long long c = (long long)r * per + got;
      if (got >= per || c >= total_chunks)
      {
        r = (r + 1 == nranges) ? 0 : r + 1;
        tries++;
        continue;
      }
      walk_chunk<Count>(D, K, (int)c, lane, sh, cnt);
    }
  }
  else
  {
    const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int c = warp_global; c < total_chunks; c += nwarps)
      walk_chunk<Count>(D, K, c, lane, sh, cnt);
  }
  if (Count)
    for (int q = 0; q < kWalkCounters; q++)
    {
      unsigned long long v = cnt.v[q];
      for (int o = 16; o > 0; o >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0)
        atomicAdd(D.interactions + q, v);
    }
}

} // namespace
} // namespace hbtg
