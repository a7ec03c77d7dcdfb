// reassign.cuh - particle reassignment before unbinding
// (SubhaloSnapshot_t::ReassignParticles, src/subhalo_reassign_gas.cpp:65-197).
//
// Each FoF group's tracer particles form one geometric tree (the unbinding
// tree's build over the tracers, with cell bounding boxes; coordinates
// unwrapped about the group's first tracer, for the tree and its pruning
// only).  The non-tracer particles are put in the tree's spatial order, so
// that a warp's 32 searches visit the same cells; one thread per particle
// finds its k nearest tracers, with the distance of the k-th of its
// neighbours in key order as the first bound, by
// exact distance (double, from the float coordinates with the periodic wrap,
// as the reference's GeoTree_t::Search computes it) and then reads off what
// GeoTree_t::NearestNeighbours (src/geometric_tree.cpp:108-142) returns.
// That search widens its radius R_j (R_0 = SofteningHalo / 10 in float, each
// 1.26 times the last, rounded to float) until its collector holds
// min(tracers, k) entries; search j collects every tracer with
// |dx|, |dy|, |dz| <= R_j and r^2 < R_j * R_j (a float product), into the
// same collector, which keeps the k smallest r^2 it was given.  So a tracer
// first found by search jmin counts J - jmin + 1 times, J being the last
// search, and the list is the distinct tracers of those k entries, the
// nearest last.  Searches j < J collect fewer than k tracers, all among the
// k nearest, so the k nearest decide everything (up to ties in r^2, and to a
// tracer that the axis test rejects although r^2 < R_j * R_j: a rounding
// gap of one float ulp in R_j).
#pragma once

#include <cstdint>

#include "common.cuh"
#include "kernels.cuh"

namespace hbtg
{
namespace
{

constexpr int kMaxNeighbours = 32;

struct ReState
{
  int S;                     // subhaloes
  int G;                     // FoF groups
  const long long *off;      // [S+1] particles of each subhalo
  const int *sub_group;      // [S] FoF group of each subhalo
  const long long *gpart;    // [G+1] particles of each group (contiguous)
  const float *pos;          // [3N] raw positions
  const uint8_t *type;       // [N]
  long long *dest;           // [N] out
  int *flags, *rank;         // [N+1] tracer flags and their exclusive scan
  int *tg;                   // [T] particle of each packed tracer
  int *tsub;                 // [T] subhalo of each packed tracer
  float4 *raw;               // [T] tracers in the trees' leaf order: raw position, packed tracer (int bits)
  unsigned long long *qkey;  // [N - T] search order: group, then the top digits of the particle's tree key
  uint32_t *qval;            // [N - T] the non-tracers, in search order once sorted by qkey
  int tracer_mask;
  float box, half, r0, eps;
  int periodic, k;
};

constexpr int kReDigits = 10; // tree-key digits of the search order (3 bits each)

__device__ __forceinline__ bool re_tracer(const ReState &R, long long g)
{
  return ((1 << (int)R.type[g]) & R.tracer_mask) != 0;
}

__global__ void k_re_flags(ReState R, long long n)
{
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g > n)
    return;
  R.flags[g] = (g < n && re_tracer(R, g)) ? 1 : 0;
}

// Packs the tracers by group (the reference's order: subhalo, then particle)
// into the tree state D: unwrapped position, unit mass, identity order.
__global__ void k_re_pack(ReState R, DevState D, long long n)
{
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n || !R.flags[g])
    return;
  const int s = find_segment<long long>(R.off, R.S, g);
  const int t = R.rank[g];
  R.tg[t] = (int)g;
  R.tsub[t] = s;
  D.seg_of[t] = R.sub_group[s];
  D.ord[t] = t;
  D.ty[t] = 0;
}

// The group's first tracer as the unwrapping point (positions as the
// reference's NEAREST sees them from it).
__device__ __forceinline__ float unwrap(float x, float ref, const ReState &R)
{
  const float d = __fsub_rn(x, ref);
  return R.periodic ? __fadd_rn(ref, nearest_f(d, R.half, R.box)) : x;
}

__global__ void k_re_unwrap(ReState R, DevState D, int total)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total)
    return;
  const int h = D.seg_of[t];
  const float *ref = R.pos + 3 * (long long)R.tg[D.off[h]];
  const float *x = R.pos + 3 * (long long)R.tg[t];
  D.pm[t] = make_float4(unwrap(x[0], ref[0], R), unwrap(x[1], ref[1], R), unwrap(x[2], ref[2], R), 1.f);
}

// First packed tracer of each group.
__global__ void k_re_goff(ReState R, long long *goff)
{
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h <= R.G)
    goff[h] = R.rank[R.gpart[h]];
}

// Per group: the tracers are the sources when the group has non-tracers.
__global__ void k_re_plan(ReState R, DevState D)
{
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h > D.S)
    return;
  if (h == D.S)
  {
    D.src_cnt[h] = 0;
    return;
  }
  const int nt = (int)(D.off[h + 1] - D.off[h]);
  const long long np = R.gpart[h + 1] - R.gpart[h];
  D.state[h] = kActive;
  D.iter[h] = 1;
  D.corr[h] = 1; // no key-order record
  D.wrap[h] = 0;
  D.ngrav[h] = 0;
  D.src_begin[h] = 0;
  D.src_cnt[h] = (nt > 0 && np > nt) ? nt : 0;
  for (int q = 0; q < 6; q++)
    D.factor[6 * h + q] = 1.f;
  for (int d = 0; d < 3; d++)
  {
    D.bb_lo[3 * h + d] = 0xffffffffu;
    D.bb_hi[3 * h + d] = 0u;
  }
}

// Exact squared distance and largest axis offset, as GeoTree_t::Search.
__device__ __forceinline__ double re_d2(const float *a, const float *q, const ReState &R, double &dmax)
{
  double d2 = 0.;
  dmax = 0.;
#pragma unroll
  for (int k = 0; k < 3; k++)
  {
    double d = (double)a[k] - (double)q[k];
    if (R.periodic)
      d = nearest_d(d, (double)R.half, (double)R.box);
    dmax = fmax(dmax, fabs(d));
    d2 = __dadd_rn(d2, __dmul_rn(d, d));
  }
  return d2;
}

// The radii of the widening searches, R_j = 1.26 R_(j-1) rounded to float, up
// to the first that holds every float (and never more than kReRadii).
constexpr int kReRadii = 448; // 1.26^448 spans every float from 1e-6 up
struct ReRadii
{
  float r[kReRadii];
  int n;
  explicit ReRadii(float r0) : n(0)
  {
    for (float R = r0; n < kReRadii; R = (float)((double)R * 1.26))
    {
      r[n++] = R;
      if (R > 3.4e38f)
        break;
    }
  }
};

// The first search j < 4096 that collects a tracer at (d2, dmax): the radii
// do not decrease, so a binary search over the table finds it; past the
// table's end (an initial radius so small that it does not reach infinity
// there) the searches go on one by one.  dmax <= R and d2 < R * R (a float)
// are decided on the floats next to dmax (above) and d2 (below), which compare
// with a float as they do.
__device__ __forceinline__ int re_jmin(double d2, double dmax, const float *radii, int n)
{
  const float up = __double2float_ru(dmax), down = __double2float_rd(d2);
  auto takes = [&](float R) { return up <= R && down < __fmul_rn(R, R); };
  int lo = 0, hi = n;
  while (lo < hi)
  {
    const int mid = (lo + hi) >> 1;
    if (takes(radii[mid]))
      hi = mid;
    else
      lo = mid + 1;
  }
  if (lo < n)
    return lo;
  int j = n;
  for (float R = __double2float_rn((double)radii[n - 1] * 1.26); j < 4096; R = __double2float_rn((double)R * 1.26), j++)
    if (takes(R))
      break;
  return j;
}

// Tree key of a point in group h's root cube (k_root's constants): the slab
// indices of descent_key_fast, clamped into the cube.  Only a place to start
// and an order of work: a digit off costs time, not results.
__device__ __forceinline__ unsigned long long re_place(const float *x, const float *kp)
{
  unsigned long long key = 0;
#pragma unroll
  for (int d = 0; d < 3; d++)
  {
    const float t = __fmul_rn(__fsub_rn(__fsub_rn(x[d], kp[d]), kp[3 + d]), kp[6]);
    const float c = t > 0.f ? fminf(floorf(t), 2097151.f) : 0.f; // NaN: 0
    key |= spread3((unsigned long long)__float2uint_rz(c)) << d;
  }
  return key;
}

// The non-tracers with their search order (those of a group without a tree
// too: the search leaves them alone).
__global__ void k_re_queries(ReState R, DevState D, long long n)
{
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int s = find_segment_warp<long long>(R.off, R.S, min(g, n - 1));
  if (g >= n || R.flags[g])
    return;
  const int h = R.sub_group[s];
  unsigned long long key = 0;
  if (D.src_cnt[h] > 0)
  {
    const float *x = R.pos + 3 * g, *ref = R.pos + 3 * (long long)R.tg[D.off[h]];
    const float u[3] = {unwrap(x[0], ref[0], R), unwrap(x[1], ref[1], R), unwrap(x[2], ref[2], R)};
    key = re_place(u, D.keyp + 12 * h);
  }
  const long long i = g - R.rank[g];
  R.qkey[i] = ((unsigned long long)h << (3 * kReDigits)) | (key >> (63 - 3 * kReDigits));
  R.qval[i] = (uint32_t)g;
}

// Leaf order of the tracers: the leaf's w holds its place j among them, raw[j]
// the raw position and the packed tracer.
__global__ void k_re_leaves(ReState R, DevState D, int total)
{
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= total)
    return;
  const int t = (int)D.val[j];
  const float *x = R.pos + 3 * (long long)R.tg[t];
  R.raw[j] = make_float4(x[0], x[1], x[2], __int_as_float(t));
  reinterpret_cast<int *>(&D.nodes[j + 2 * D.X[j] + 2 * D.cnt[j]])[3] = j;
}

// One axis offset a - b with the periodic wrap of the exact distance, rounded
// once: the difference d and its own rounding error (two-sum) are exact, and so
// is d -+ box for d within [box / 2, 2 box].  (Taking the box off a or b first is
// exact only for coordinates inside the box.)
__device__ __forceinline__ float re_offset(float a, float b, const ReState &R)
{
  const float d = __fsub_rn(a, b);
  if (!R.periodic || !(fabsf(d) > R.half))
    return d;
  const float t = __fsub_rn(d, a), lost = __fsub_rn(__fsub_rn(a, __fsub_rn(d, t)), __fadd_rn(b, t));
  return __fadd_rn(d > 0.f ? __fsub_rn(d, R.box) : __fadd_rn(d, R.box), lost);
}

// Squared distance in FP32 from the raw positions: within kReLoose (relative)
// of the exact one.
constexpr float kReLoose = 2e-6f;
__device__ __forceinline__ float re_r2(const float4 &a, const float *q, const ReState &R)
{
  const float x = re_offset(a.x, q[0], R), y = re_offset(a.y, q[1], R), z = re_offset(a.z, q[2], R);
  return x * x + y * y + z * z;
}

// Squared reach of a search whose k-th squared distance is at most r2: a cell
// or leaf beyond it, by its unwrapped floats, is passed over (eps covers their
// rounding, the factor that of the arithmetic).
__device__ __forceinline__ float re_reach2(float r2, const ReState &R)
{
  const float r = __fsqrt_ru(r2) + R.eps;
  return r * r * (1.f + 4e-6f);
}

// Visits the leaves of group h's tree within reach of uq, in tree order, up to
// the root's end; take(j, reach) may shrink the reach.
template <typename Take>
__device__ __forceinline__ void re_walk(const float4 *T, int root, const float *uq, float reach, Take take)
{
  const int end = __float_as_int(T[root + 1].y);
  int idx = root;
  while (idx < end)
  {
    const float4 a = T[idx], b = T[idx + 1]; // both at once: one latency a node (a padding slot follows the tree)
    if (slot_is_cell(a.w))
    {
      const float gx = fmaxf(fmaxf(a.x - uq[0], uq[0] - b.x), 0.f);
      const float gy = fmaxf(fmaxf(a.y - uq[1], uq[1] - b.z), 0.f);
      const float gz = fmaxf(fmaxf(a.z - uq[2], uq[2] - b.w), 0.f);
      idx = gx * gx + gy * gy + gz * gz > reach ? max(__float_as_int(b.y), idx + 2) : idx + 2;
      continue;
    }
    idx++;
    const float fx = a.x - uq[0], fy = a.y - uq[1], fz = a.z - uq[2];
    if (!(fx * fx + fy * fy + fz * fz > reach))
      take(__float_as_int(a.w), reach);
  }
}

// One thread per non-tracer, in search order: dest = the subhalo it moves to
// (dest holds -1 before).  The k nearest are searched in FP32 (FP64, with its
// 16 cycles an SM and instruction, held a first version): a first bound from
// 2k neighbours in key order, then the k + 2 smallest FP32 distances; the
// exact distances of these decide, unless more tracers than that lie within
// the FP32 error of the k-th (coincident ones), when the search is repeated
// with exact distances.  Bound by the latency of the tree's slots.  From the
// tree's root without a bound, in the particles' list order, a call over 3e5
// particles in 40 groups (k = 10) took 45.2 ms; with exact distances
// throughout 3.26 ms, now 1.55 ms.
template <int kMax>
__global__ void __launch_bounds__(128)
  k_re_query(ReState R, DevState D, const __grid_constant__ ReRadii table, long long nq)
{
  constexpr int kKeep = kMax + 2;
  __shared__ float radii[kReRadii];
  const int n_radii = table.n;
  for (int j = threadIdx.x; j < n_radii; j += blockDim.x)
    radii[j] = table.r[j];
  __syncthreads();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq)
    return;
  const long long g = R.qval[i];
  const int h = (int)(R.qkey[i] >> (3 * kReDigits));
  const int nt = (int)(D.off[h + 1] - D.off[h]);
  if (nt == 0 || D.src_cnt[h] == 0)
    return;
  const int k = R.k;
  const float q[3] = {R.pos[3 * g], R.pos[3 * g + 1], R.pos[3 * g + 2]};
  const float *ref = R.pos + 3 * (long long)R.tg[D.off[h]];
  const float uq[3] = {unwrap(q[0], ref[0], R), unwrap(q[1], ref[1], R), unwrap(q[2], ref[2], R)};
  const int seg0 = D.src_off[h], seg1 = seg0 + nt;
  const int root = seg0 + 2 * D.X[seg0];
  float fd[kKeep]; // FP32 squared distances, ascending
  int fj[kKeep];   // their places in leaf order
  int cnt = 0;
  auto keep = [&](float r2, int j, int cap) {
    int at = cnt < cap ? cnt : cap - 1;
    while (at > 0 && fd[at - 1] > r2)
    {
      fd[at] = fd[at - 1];
      fj[at] = fj[at - 1];
      at--;
    }
    fd[at] = r2;
    fj[at] = j;
    cnt += cnt < cap;
  };
  // the k-th distance among 2k neighbours in key order bounds the k-th of all
  float bound = INFINITY;
  if (nt >= k)
  {
    const unsigned long long key = re_place(uq, D.keyp + 12 * h);
    int lo = seg0, hi = seg1;
    while (lo < hi)
    {
      const int mid = (lo + hi) >> 1;
      if (D.key[mid] < key)
        lo = mid + 1;
      else
        hi = mid;
    }
    const int j0 = max(seg0, min(lo - k, seg1 - 2 * k)), j1 = min(seg1, j0 + 2 * k);
    for (int j = j0; j < j1; j++)
    {
      const float r2 = re_r2(R.raw[j], q, R);
      if (cnt < k || r2 < fd[cnt - 1])
        keep(r2, j, k);
    }
    if (fd[k - 1] < bound) // not for a NaN
      bound = fd[k - 1] * (1.f + 2.f * kReLoose);
    cnt = 0;
  }
  const int cap = k + 2;
  re_walk(D.nodes, root, uq, re_reach2(bound, R), [&](int j, float &reach) {
    const float r2 = re_r2(R.raw[j], q, R);
    if (cnt < cap ? !(r2 > bound) : r2 < fd[cap - 1])
    {
      keep(r2, j, cap);
      if (cnt >= k && fd[k - 1] < bound)
      { // what lies within the error of the k-th stays in reach
        bound = fminf(bound, fd[k - 1] * (1.f + 2.f * kReLoose));
        reach = re_reach2(bound, R);
      }
    }
  });
  // their exact distances, ascending; equal ones in tree order
  double bd[kKeep], bm[kKeep];
  int bi[kKeep];
  auto exact_of = [&](int j, double &dmax) {
    const float4 a = R.raw[j];
    const float x[3] = {a.x, a.y, a.z};
    return re_d2(x, q, R, dmax);
  };
  int m = 0;
  // all that may belong to the k nearest are here unless the list is full of them
  const bool crowded = cnt == cap && !(fd[cap - 1] > fd[k - 1] * (1.f + 2.f * kReLoose));
  if (!crowded)
    for (int e = 0; e < cnt; e++)
    {
      double dmax;
      const double d2 = exact_of(fj[e], dmax);
      int at = m++;
      while (at > 0 && (bd[at - 1] > d2 || (bd[at - 1] == d2 && bi[at - 1] > fj[e])))
      {
        bd[at] = bd[at - 1];
        bm[at] = bm[at - 1];
        bi[at] = bi[at - 1];
        at--;
      }
      bd[at] = d2;
      bm[at] = dmax;
      bi[at] = fj[e];
    }
  else
    re_walk(D.nodes, root, uq, re_reach2(bound, R), [&](int j, float &) {
      double dmax;
      const double d2 = exact_of(j, dmax);
      if (m < k || d2 < bd[m - 1])
      { // the leaves come in tree order: equal distances keep the earlier
        int at = m < k ? m : k - 1;
        while (at > 0 && bd[at - 1] > d2)
        {
          bd[at] = bd[at - 1];
          bm[at] = bm[at - 1];
          bi[at] = bi[at - 1];
          at--;
        }
        bd[at] = d2;
        bm[at] = dmax;
        bi[at] = j;
        m += m < k;
      }
    });
  cnt = min(m, k);
  // the widening searches, from the k nearest
  int jm[kMax];
  int jmax = 0;
  for (int e = 0; e < cnt; e++)
  {
    jm[e] = re_jmin(bd[e], bm[e], radii, n_radii);
    jmax = max(jmax, jm[e]);
    bi[e] = __float_as_int(R.raw[bi[e]].w); // the packed tracer
  }
  const int to_find = min(nt, k);
  int J = jmax;
  long long cum = 0;
  for (int j = 0; j <= jmax; j++)
  {
    int nj = 0;
    for (int i = 0; i < cnt; i++)
      nj += jm[i] <= j;
    cum += nj;
    if (min(cum, (long long)k) >= to_find)
    {
      J = j;
      break;
    }
  }
  const int s = find_segment<long long>(R.off, R.S, g);
  long long taken = 0;
  int first = -1;
  bool found = false;
  for (int i = 0; i < cnt; i++)
  {
    if (jm[i] > J)
      continue;
    if (taken >= k)
      break;
    if (first < 0)
      first = bi[i];
    if (R.tsub[bi[i]] == s)
      found = true;
    taken += J - jm[i] + 1;
  }
  if (!found && first >= 0)
  {
    const int to = R.tsub[first];
    if (to >= 0 && to != s)
      R.dest[g] = to;
  }
}

} // namespace
} // namespace hbtg
