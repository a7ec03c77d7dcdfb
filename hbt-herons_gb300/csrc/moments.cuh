// moments.cuh - mass and centre of mass of a tree cell from its children, in
// exact integer arithmetic where that can be shown to round as the reference's
// double sums do.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace hbtg
{
namespace
{

// 64-bit integer <-> float conversions by exponent and mantissa arithmetic
// (the hardware's 64-bit conversions issue to the FP64 pipe, whose
// throughput is low on this GPU).

// v = hi + lo: hi is v rounded to float (to nearest even), lo the remainder
// rounded to float.  |v| < 2^63.
__device__ __forceinline__ void ll_to_float2(long long v, float &hi, float &lo)
{
  const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  float h, l = 0.f;
  if (a < (1ull << 24))
    h = __uint2float_rn((unsigned)a);
  else
  {
    const int e = 63 - __clzll((long long)a);
    const int sh = e - 23;
    unsigned long long mant = a >> sh;
    const unsigned long long rem = a & ((1ull << sh) - 1ull), half = 1ull << (sh - 1);
    long long r = (long long)rem;
    if (rem > half || (rem == half && (mant & 1ull)))
    {
      mant++;
      r -= (long long)(1ull << sh);
    }
    // a mantissa carried to 2^24 steps the exponent field by itself
    h = __uint_as_float((unsigned)((e + 127) << 23) + (unsigned)(mant - (1ull << 23)));
    const unsigned long long ar = r < 0 ? 0ull - (unsigned long long)r : (unsigned long long)r; // < 2^39
    l = __fmaf_rn(__uint2float_rn((unsigned)(ar >> 16)), 65536.f, __uint2float_rn((unsigned)(ar & 0xffffu)));
    if (r < 0)
      l = -l;
  }
  hi = v < 0 ? -h : h;
  lo = v < 0 ? -l : l;
}

// Mass and centre of mass of a cell from its children
// (GravityTree_t::UpdateInternalNodes / ProcessNode / FillNodeCenter,
// src/gravity_tree.cpp:18-80): children in octant order (their slot order),
// each child's float mass and float position (a leaf) or float centre (a
// cell) accumulated in double, then stored as float -- the reference's own
// rounding, so a cell's centre carries its children's roundings as in the
// reference.
__device__ __noinline__ void cell_moments_fp64(float4 *nodes, int slot)
{
  const int end = __float_as_int(nodes[slot + 1].y);
  double M = 0., X = 0., Y = 0., Z = 0.;
  float fx = 0.f, fy = 0.f, fz = 0.f; // first child's position (a massless cell)
  int ch = slot + 2;
  while (ch < end)
  {
    const float4 a = nodes[ch], b = nodes[ch + 1];
    const bool cell = slot_is_cell(a.w);
    if (ch == slot + 2)
    {
      fx = a.x;
      fy = a.y;
      fz = a.z;
    }
    const double md = (double)(cell ? b.x : a.w);
    M = __dadd_rn(M, md);
    X = __fma_rn((double)a.x, md, X); // the product is exact in double
    Y = __fma_rn((double)a.y, md, Y);
    Z = __fma_rn((double)a.z, md, Z);
    ch = max(cell ? __float_as_int(b.y) : ch + 1, ch + 1); // strictly increasing
  }
  float *cs = reinterpret_cast<float *>(&nodes[slot]);
  cs[0] = M > 0. ? __double2float_rn(__ddiv_rn(X, M)) : fx;
  cs[1] = M > 0. ? __double2float_rn(__ddiv_rn(Y, M)) : fy;
  cs[2] = M > 0. ? __double2float_rn(__ddiv_rn(Z, M)) : fz;
  reinterpret_cast<float *>(&nodes[slot + 1])[0] = __double2float_rn(M);
}

// The same results without FP64, whose throughput (two lanes a clock and SM)
// bound the per-level passes: a cell's coordinates along an axis differ by a
// few binades at most and its masses share a coarse unit, so the sums are
// exact in 64-bit integers.  At 5e6 particles a large level takes 34 us
// instead of 55; a 5e7-particle learned call 113.7 ms instead of 115.6.
constexpr int kMomentsWide = 11;    // bits beyond two 24-bit factors: the sums stay below 2^62
constexpr int kMomentsChildren = 8; // more (coincident particles) go to cell_moments_fp64

// Mantissa and exponent of a float: |x| = m 2^(e - 150); e = 0 for zero, ok
// cleared for a subnormal or non-finite x.
__device__ __forceinline__ unsigned float_parts(float x, int &e, bool &ok)
{
  const unsigned u = __float_as_uint(x) & 0x7fffffffu;
  e = (int)(u >> 23);
  ok = ok && e < 255 && (e > 0 || u == 0u);
  return u == 0u ? 0u : (u & 0x7fffffu) | 0x800000u;
}

// The float that the double quotient (double)X / (double)M rounds to, in the
// unit 2^(e - 150), for X exact, its terms of one sign (so no partial sum exceeds
// it, and it is zero only where all are) and M = Mh + Ml > 0 (an integer below 2^42):
// the quotient in a float pair (error < 2^-40 of it); where that leaves the
// rounding open, the exact sign of 2 X - 2 h M at the halfway point h
// decides.  Clears ok where the double arithmetic could differ from that: X
// beyond 2^53, or 2 X within 2^-49 of 2 h M but not on it (the double quotient
// may round onto the tie), or a quotient below 2^23 (a coordinate of zero among them).
__device__ __forceinline__ float quotient_float(long long X, long long M, float Mh, float Ml, float rM, int e,
                                                bool &ok)
{
  if (X == 0)
    return 0.f;
  const unsigned long long aX = X < 0 ? 0ull - (unsigned long long)X : (unsigned long long)X;
  float xh, xl;
  ll_to_float2((long long)aX, xh, xl);
  const float q1 = __fmul_rn(xh, rM);
  float r = __fmaf_rn(-q1, Mh, xh);
  r = __fmaf_rn(-q1, Ml, __fadd_rn(r, xl));
  const float q2 = __fmul_rn(r, rM);
  float c = __fadd_rn(q1, q2);
  const float d = __fsub_rn(q2, __fsub_rn(c, q1)), tol = __fmul_rn(c, 9.094947e-13f); // 2^-40
  ok = ok && c >= 8388608.f && c < 2147483648.f;
  if (__fadd_rn(c, __fadd_rn(d, tol)) != c || __fadd_rn(c, __fsub_rn(d, tol)) != c)
  {
    const unsigned mant = __float_as_uint(c) & 0x7fffffu;
    const int j = (int)(__float_as_uint(c) >> 23) - 150; // spacing of floats at c: 2^j, j >= 0
    const bool up = d > 0.f;
    ok = ok && j >= 0 && aX < (1ull << 53) && (mant != 0u || up);
    if (ok)
    {
      const unsigned step = 1u << j;
      const long long h2 = 2ll * (long long)__float2uint_rz(c) + (up ? (long long)step : -(long long)step);
      const long long D = 2ll * (long long)aX - h2 * M; // both terms near 2 X < 2^54
      const unsigned long long aD = D < 0 ? 0ull - (unsigned long long)D : (unsigned long long)D;
      ok = D == 0 || aD > (aX >> 48);
      if (D == 0 ? (mant & 1u) != 0u : (D > 0) == up)
        c = up ? __fadd_rn(c, (float)step) : __fsub_rn(c, (float)step);
    }
  }
  const int ce = (int)(__float_as_uint(c) >> 23) + e - 150;
  ok = ok && ce > 0 && ce < 255;
  return __uint_as_float((X < 0 ? 0x80000000u : 0u) | ((unsigned)ce << 23) | (__float_as_uint(c) & 0x7fffffu));
}

// The multipoles of the cell at `slot` from its children.
__device__ __forceinline__ void cell_moments(float4 *nodes, int slot)
{
  const int end = __float_as_int(nodes[slot + 1].y);
  float4 v[kMomentsChildren]; // position, mass
  int n = 0, ch = slot + 2;
#pragma unroll
  for (int k = 0; k < kMomentsChildren; k++)
  {
    v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (ch < end)
    { // both slots at once, needed or not (a padding slot follows the tree): one latency per child
      const float4 a = nodes[ch], b = nodes[ch + 1];
      const bool cell = slot_is_cell(a.w);
      v[k] = make_float4(a.x, a.y, a.z, cell ? b.x : a.w);
      ch = max(cell ? __float_as_int(b.y) : ch + 1, ch + 1); // strictly increasing
      n = k + 1;
    }
  }
  bool ok = ch >= end;
  // masses in units of the lowest bit set in any of them
  int low = 1 << 20;
#pragma unroll
  for (int k = 0; k < kMomentsChildren; k++)
  {
    int e;
    const unsigned m = float_parts(v[k].w, e, ok);
    if (m)
      low = min(low, e + __ffs((int)m) - 1);
  }
  long long a[kMomentsChildren], M = 0;
  int wide = 0; // bits that the masses, and below the coordinates, hold beyond 24
#pragma unroll
  for (int k = 0; k < kMomentsChildren; k++)
  {
    int e;
    const unsigned m = float_parts(v[k].w, e, ok);
    const int sh = m ? e - low : 0; // a right shift drops zeros only
    ok = ok && v[k].w >= 0.f;
    wide = max(wide, sh);
    a[k] = sh >= 0 ? (long long)m << min(sh, kMomentsWide) : (long long)(m >> min(-sh, 31));
    M += a[k];
  }
  ok = ok && M != 0 && wide <= kMomentsWide;
  float c[3] = {0.f, 0.f, 0.f};
  float Mf = 0.f;
  if (ok)
  {
    float Mh, Ml;
    ll_to_float2(M, Mh, Ml);
    const float rM = __frcp_rn(Mh);
    const int me = (int)(__float_as_uint(Mh) >> 23) + low - 150;
    ok = me > 0 && me < 255;
    Mf = __uint_as_float(((unsigned)me << 23) | (__float_as_uint(Mh) & 0x7fffffu));
#pragma unroll
    for (int d = 0; d < 3; d++)
    {
      int least = 255;
#pragma unroll
      for (int k = 0; k < kMomentsChildren; k++)
      {
        int e;
        if (float_parts(d == 0 ? v[k].x : d == 1 ? v[k].y : v[k].z, e, ok))
          least = min(least, e);
      }
      long long X = 0;
      unsigned signs = 0u; // bit 0: a positive coordinate, bit 1: a negative one
#pragma unroll
      for (int k = 0; k < kMomentsChildren; k++)
      {
        const float x = d == 0 ? v[k].x : d == 1 ? v[k].y : v[k].z;
        int e;
        const unsigned m = float_parts(x, e, ok);
        const int sh = m ? e - least : 0;
        ok = ok && sh + wide <= kMomentsWide && sh <= 6;
        const int q = (int)(m << min(sh, 6)); // < 2^30
        signs |= m ? (x < 0.f ? 2u : 1u) : 0u;
        X += (long long)(x < 0.f ? -q : q) * a[k]; // eight terms below 2^(48 + kMomentsWide)
      }
      // of both signs, the double chain may round partial sums that the total no longer shows
      ok = ok && signs != 3u;
      c[d] = quotient_float(X, M, Mh, Ml, rM, least, ok);
    }
  }
  if (!ok)
  {
    cell_moments_fp64(nodes, slot);
    return;
  }
  float *cs = reinterpret_cast<float *>(&nodes[slot]);
  cs[0] = c[0];
  cs[1] = c[1];
  cs[2] = c[2];
  reinterpret_cast<float *>(&nodes[slot + 1])[0] = Mf;
}

} // namespace
} // namespace hbtg
