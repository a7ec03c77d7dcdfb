// settle.cuh - the unbinding loop of one subhalo by one team of threads, from
// wherever the lock-step iteration left it to its end.
//
// After the first few lock-step iterations only slowly converging subhaloes
// are left: tens of them, with a few thousand particles at most and a handful
// of tree sources each, for another ten to sixty iterations.  In lock step
// each of those costs its forty launches and three host reads (0.3-0.6 ms),
// whatever little they hold.  Here a team -- one block, a cluster of eight
// blocks for larger subhaloes, the whole grid for the largest -- keeps its
// subhalo until it converges, disrupts or no longer fits, with block, cluster
// or grid barriers between the steps.
//
// Every step is the lock-step one (kernels.cuh has the reference's lines):
// the same keys in the same stable order, the same tree, the same chunks of
// 32 targets walked by the same code, the same energies and partition.  The
// centre-of-mass sums are the one place where grouping could show: k_com adds
// single items in double once an iteration's bound sets hold at most kComSmall
// particles, some 1e-16 of the summed magnitudes off whatever its order, and
// teams (which add three-word FloatSums, then a double per warp) take over only
// from there on (IterationDriver::iterate).  So both round to the same float
// unless the sum lies within that of a halfway point: the results are the same
// bits in every case tried, and expected to be, but not by construction.
//
// Limits of a team: kSettleSrc tree sources (their keys and tree indices lie
// in shared memory), kSettleSlots tree slots, and no potential subsample.  A
// subhalo that does not fit at the top of an iteration goes back to lock step
// as it stands.
//
// Bound by latency: some 25 barriers and chains of dependent loads from L2 an
// iteration, and the longest walk of a chunk.  The 27 late iterations of a
// 1e6-particle subsampled call (334 subhaloes) take 1.0 ms, 37 us each, in
// place of 8 ms.  Teams alone took a call on one subhalo of 300 particles from
// 1.26 to 0.73 ms and one on 5e6 particles (plain) from 29.0 to 26.0 ms; small
// trees in shared memory then the first to 0.67 ms.
#pragma once

#include <cooperative_groups.h>

#include "kernels.cuh"
#include "walk.cuh"

namespace hbtg
{
namespace
{

// Threads of a block (C: blocks of its team).  The grid's blocks are one per
// SM, with enough warps for a chunk of 32 targets each.
constexpr int kGrid = 0; // team size standing for the whole (cooperative) grid
__host__ __device__ constexpr int settle_threads(int C) { return C == kGrid ? 512 : 256; }
constexpr int kSettleSrc = 2048;    // tree sources of a team
constexpr int kSettleSlots = 8192;  // tree slots of a block (each block of a cluster builds the tree for itself)
constexpr int kSettleCluster = 8;   // blocks of a cluster's team
// Targets up to which one block takes a subhalo (a chunk of 32 per warp, or
// four in the correction loop or when there are more of that size than
// clusters), and a cluster (one subhalo of 250 particles takes 0.58 ms with a block and 0.64 with a cluster, of 500
// 0.74 and 0.67; with kSettleOne at 512 or 2048 calls on 600 to 2,000 take the same time within 1 %; one of 7,000
// to 12,000 takes the same within 2 % with a cluster and with the grid); above kSettleMid, the grid, whose barriers cost most (some 3 us) and which takes one
// subhalo at a time.  One of 46,000 particles with 50 iterations left took 34 ms with a
// cluster's 64 warps, 31 ms in lock step and 15 ms with the grid.  Several of up to kSettleLarge go to clusters all
// the same, which take them side by side: six of 16,000 particles take a call of 10.4 ms one after the other, 3.5 ms
// with clusters and 3.8 ms in lock step; one alone 2.95, 2.99 and 3.03 ms.  Two of 30,000: 2.4 to 3.5 ms with the
// grid, 3.1 to 4.4 ms with clusters; three of 20,000: 3.1 to 4.0 and 3.3 to 4.1 (more do not fit into the 65,536).
constexpr int kSettleSmall = 256, kSettleOne = 1024, kSettleMid = 8192, kSettleLarge = 20480;
constexpr int kSettleTeams1 = 456, kSettleTeams8 = 38; // most teams of one launch (3 blocks fit an SM)
constexpr int kSettleMaxBlocks = 1024;                  // of a team (the grid's)
enum SettleClass : int
{
  kSettleA, kSettleB, kSettleC, kSettleD, kSettleE, // by the four limits above
  kSettleClasses
};

struct SettleArgs
{
  int *list;   // [kSettleClasses S]: the subhaloes of each class
  int *count;  // [kSettleClasses] their numbers
  float4 *nodes;  // kSettleSlots per block
  unsigned long long *skey; // kSettleSrc per team: sorted keys of a team of several blocks
  uint32_t *sval;           //                      and their particles
  double *xch;              // [2][blocks of the team][8] per team: sums in exchange between its blocks
  unsigned long long *cells; // tree cells built
  int *most;                 // most iterations that one subhalo took here
  int grid;                  // blocks of the grid's team (0: none)
};

// Arrays of a block that live between two walks (the walk's lists take their place).
struct SettleTree
{
  unsigned long long key[kSettleSrc], skey[kSettleSrc];
  uint32_t val[kSettleSrc], sval[kSettleSrc];
  int X[kSettleSrc];               // cells before each item
  unsigned short levels[kSettleSrc]; // first level of its cells | their number << 8
};
template <int C>
union SettleWork
{
  SettleTree t;
  WalkWarp walk[settle_threads(C) / kWarp];
  uint32_t tail[kSettleSrc];
};
// A block of a larger team has the shared memory of its SM to itself and keeps
// its tree there, for the multipoles and for the walk: with both in L2 they
// took 108 and 77 us of an iteration of the grid over 35,000 particles with
// 1,000 tree sources, and a call with 50 of those 41.5 ms instead of 35.0.
constexpr int kSettleOwn = 4096; // slots
template <int C>
struct SettleShared
{
  SettleWork<C> u;
  float4 nodes[C == 1 ? 1 : kSettleOwn];
};

// Subhaloes that a team can take over at the top of an iteration.
__global__ void k_settle_pick(DevState D, KParams K, SettleArgs A)
{
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= D.S || D.state[s] != kActive)
    return;
  const int n = D.nbound[s];
  const bool sampled = !D.corr[s] && K.max_sample > 0 && !(n < K.max_sample + D.nunsample[s]);
  if (sampled || (D.corr[s] ? D.nlast[s] - n : n) > kSettleSrc)
    return;
  // (the correction loop's trees are small: a block's barriers are cheaper there than a cluster's warps)
  const int c = n <= kSettleSmall || (n <= kSettleOne && D.corr[s]) ? kSettleA : n <= kSettleOne ? kSettleB : n <= kSettleMid ? kSettleC : n <= kSettleLarge ? kSettleD : kSettleE;
  A.list[(size_t)c * D.S + atomicAdd(&A.count[c], 1)] = s;
}

template <int C>
__device__ __forceinline__ void team_sync()
{
  if (C == 1)
    __syncthreads();
  else if (C == kGrid)
    cooperative_groups::this_grid().sync();
  else
  { // orders the cluster's global and shared accesses
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// Exclusive scan of one int per thread of the block; `par` alternates between
// two sets of partial sums, so one barrier is enough.
template <int Warps>
__device__ __forceinline__ int block_scan(int v, int (*part)[Warps], int &par, int &total)
{
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int incl = warp_inclusive_scan(v, lane);
  if (lane == 31)
    part[par][w] = incl;
  __syncthreads();
  int before = 0;
  total = 0;
#pragma unroll
  for (int k = 0; k < Warps; k++)
  {
    const int c = part[par][k];
    before += k < w ? c : 0;
    total += c;
  }
  par ^= 1;
  return before + incl - v;
}

// Rank of item i (value k) among n keys: those smaller, and equal ones before
// it (a stable sort).  i >> 5 is the same on the warp's lanes.
template <typename T>
__device__ __forceinline__ int stable_rank(const T *key, int n, int i, T k)
{
  const int tile = i & ~31;
  int r = 0;
#pragma unroll 4
  for (int j = 0; j < min(tile, n); j++)
    r += key[j] <= k;
  for (int j = tile; j < min(tile + 32, n); j++)
    r += key[j] < k || (key[j] == k && j < i);
#pragma unroll 4
  for (int j = tile + 32; j < n; j++)
    r += key[j] < k;
  return r;
}

// The same by a whole warp (every lane the same i and k, result on all).
template <typename T>
__device__ __forceinline__ int warp_rank(const T *key, int n, int i, T k)
{
  int r = 0;
  for (int j = threadIdx.x & 31; j < n; j += kWarp)
    r += key[j] < k || (key[j] == k && j < i);
  return __reduce_add_sync(0xffffffffu, r);
}

// Two counts of every block of a team, exchanged: their totals and the first
// one's sum over the blocks before this one.
template <int C>
__device__ __forceinline__ void team_counts(int &c0, int &c1, int &base, int blocks, int rank, double *xch, int &xpar)
{
  base = 0;
  if (C == 1)
    return;
  double *x = xch + (size_t)xpar * blocks * 8;
  if (threadIdx.x == 0)
  {
    x[8 * rank] = (double)c0;
    x[8 * rank + 1] = (double)c1;
  }
  team_sync<C>();
  int a = 0, b = 0;
  c0 = c1 = 0;
  for (int r = threadIdx.x & 31; r < blocks; r += kWarp)
  {
    const int c = (int)x[8 * r];
    a += r < rank ? c : 0;
    b += c;
    c1 += (int)x[8 * r + 1];
  }
  base = __reduce_add_sync(0xffffffffu, a);
  c0 = __reduce_add_sync(0xffffffffu, b);
  c1 = __reduce_add_sync(0xffffffffu, c1);
  xpar ^= 1;
}

// Tree of the m sources at ord[0..m), by way of the arrays t, in the slots T or
// (T changed) the block's own: false when it does not fit.  Returns its root cube's side and, in t.sval, the
// sources in key order.  Every block of a team builds the same tree; of
// several, each ranks a share of the sources and they exchange the order.
template <int C>
__device__ __forceinline__ bool settle_tree(const DevState &D, const KParams &K, const SettleArgs &A, const int *ord,
                                            int m, SettleTree &t, float4 *own, float4 *&T, int team, int rank, int blocks,
                                            double *root, float *kp, unsigned (*red)[6],
                                            int (*part)[settle_threads(C) / kWarp], int &par, unsigned *levels,
                                            int &cells)
{
  constexpr int kSettleThreads = settle_threads(C), kSettleWarps = kSettleThreads / kWarp;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  // bounding box (k_bbox)
  unsigned lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0u, 0u, 0u};
  for (int i = tid; i < m; i += kSettleThreads)
  {
    const int p = ord[i];
    t.val[i] = (uint32_t)p;
    const float4 x = D.pm[p];
    const unsigned v[3] = {float_to_ordered(x.x), float_to_ordered(x.y), float_to_ordered(x.z)};
#pragma unroll
    for (int d = 0; d < 3; d++)
    {
      lo[d] = min(lo[d], v[d]);
      hi[d] = max(hi[d], v[d]);
    }
  }
#pragma unroll
  for (int d = 0; d < 3; d++)
  {
    lo[d] = __reduce_min_sync(0xffffffffu, lo[d]);
    hi[d] = __reduce_max_sync(0xffffffffu, hi[d]);
  }
  if (lane == 0)
#pragma unroll
    for (int d = 0; d < 3; d++)
    {
      red[w][d] = lo[d];
      red[w][3 + d] = hi[d];
    }
  if (tid == 0)
    *levels = 0u;
  __syncthreads();
  // root cube (k_root), its parts on different warps
  if (lane == 0 && w < 6)
  {
    double l[3], h[3];
    for (int d = 0; d < 3; d++)
    {
      unsigned a = red[0][d], b = red[0][3 + d];
      for (int k = 1; k < kSettleWarps; k++)
      {
        a = min(a, red[k][d]);
        b = max(b, red[k][3 + d]);
      }
      l[d] = ordered_to_float(a);
      h[d] = ordered_to_float(b);
    }
    double len = h[0] - l[0];
    for (int d = 1; d < 3; d++)
      if (h[d] - l[d] > len)
        len = h[d] - l[d];
    if (w == 0)
    {
      for (int d = 0; d < 3; d++)
        root[d] = 0.5 * (h[d] + l[d]);
      root[3] = len;
    }
    else if (w == 1)
      root_levels(len, K, kp);
    else if (w == 2)
      root_sides(len, K, kp);
    else
      root_axis(l[w - 3], h[w - 3], len, kp, w - 3);
  }
  __syncthreads();
  for (int i = tid; i < m; i += kSettleThreads)
  {
    const float4 x = D.pm[t.val[i]];
    unsigned long long key;
    if (!descent_key_fast(x, kp, key))
      key = descent_key_exact(x, kp, root);
    t.key[i] = key;
  }
  __syncthreads();
  // key order
  if (C == 1)
  {
    for (int i = tid; i < m; i += kSettleThreads)
    {
      const unsigned long long k = t.key[i];
      const int r = stable_rank(t.key, m, i, k);
      t.skey[r] = k;
      t.sval[r] = t.val[i];
    }
    __syncthreads();
  }
  else
  {
    unsigned long long *gk = A.skey + (size_t)team * kSettleSrc;
    uint32_t *gv = A.sval + (size_t)team * kSettleSrc;
    for (int i = rank * kSettleWarps + w; i < m; i += blocks * kSettleWarps)
    {
      const unsigned long long k = t.key[i];
      const int r = warp_rank(t.key, m, i, k);
      if (lane == 0)
      {
        gk[r] = k;
        gv[r] = t.val[i];
      }
    }
    team_sync<C>();
    for (int i = tid; i < m; i += kSettleThreads)
    {
      t.skey[i] = gk[i];
      t.sval[i] = gv[i];
    }
    __syncthreads();
  }
  // cells that start at each item (k_tree_count), scanned
  cells = 0;
  unsigned mine = 0u;
  for (int i0 = 0; i0 < m; i0 += kSettleThreads)
  {
    const int i = i0 + tid;
    int c = 0, first = 0;
    if (i < m)
    {
      first = i == 0 ? 0 : lcp_levels(t.skey[i - 1], t.skey[i]) + 1;
      const int last = i == m - 1 ? (i == 0 ? 0 : -1) : lcp_levels(t.skey[i], t.skey[i + 1]);
      c = last >= first ? last - first + 1 : 0;
      t.levels[i] = (unsigned short)(first | (c << 8));
      if (c)
        mine |= ((1u << c) - 1u) << first;
    }
    int total;
    const int before = block_scan(c, part, par, total);
    if (i < m)
      t.X[i] = cells + before;
    cells += total;
  }
  if (m + 2 * cells + 1 > kSettleSlots) // one padding slot: the walk reads a node's second slot unconditionally
    return false;
  mine = __reduce_or_sync(0xffffffffu, mine);
  if (lane == 0 && mine)
    atomicOr(levels, mine);
  __syncthreads();
  // One block builds a small tree in shared memory, where the unsorted keys
  // were, and copies it out whole: its levels follow one another with shared
  // memory's latency instead of L2's (with the sums below kept in pairs: a
  // 1e6-particle subsampled call 11.5 -> 11.2 ms).  Of a larger team each block
  // keeps it (T) in its own shared memory where it fits.
  const int slots = m + 2 * cells; // and a padding slot
  float4 *const out = T;
  const bool small = C == 1 && slots < kSettleSrc * (int)sizeof(t.key[0]) / (int)sizeof(float4);
  if (small)
    T = reinterpret_cast<float4 *>(t.key);
  else if (C != 1 && slots < kSettleOwn)
    T = own;
  // slots in preorder (k_tree_emit)
  for (int i = tid; i < m; i += kSettleThreads)
  {
    const int first = t.levels[i] & 255, c = t.levels[i] >> 8, base = i + 2 * t.X[i];
    const float4 x = D.pm[t.sval[i]];
    T[base + 2 * c] = make_float4(x.x, x.y, x.z, fabsf(x.w));
    for (int q = 0; q < c; q++)
    { // the cell's last item: galloping forward over the keys
      const int L = first + q;
      int b = m - 1;
      if (L > 0)
      {
        const int shift = 63 - 3 * L;
        const unsigned long long pref = t.skey[i] >> shift;
        int a = i, e = m, step = 1;
        for (; a + step < m; step <<= 1)
        {
          if ((t.skey[a + step] >> shift) != pref)
          {
            e = a + step;
            break;
          }
          a += step;
        }
        while (e - a > 1)
        {
          const int mid = (a + e) >> 1;
          if ((t.skey[mid] >> shift) == pref)
            a = mid;
          else
            e = mid;
        }
        b = a;
      }
      put_cell(T + base + 2 * q, kp, L, b + 2 * t.X[b] + 2 * (t.levels[b] >> 8) + 1, K);
    }
  }
  __syncthreads();
  // multipoles, deepest level first (k_tree_moments)
  for (unsigned left = *levels; left;)
  {
    const int L = 31 - __clz((int)left);
    left ^= 1u << L;
    for (int i = tid; i < m; i += kSettleThreads)
    {
      const int first = t.levels[i] & 255, c = t.levels[i] >> 8;
      if (L >= first && L < first + c)
        cell_moments(T, i + 2 * t.X[i] + 2 * (L - first));
    }
    __syncthreads();
  }
  if (small)
  {
    for (int i = tid; i < slots; i += kSettleThreads)
      out[i] = T[i];
    T = out;
  }
  return true;
}

template <int C>
__global__ void __launch_bounds__(settle_threads(C), C == 1 ? 3 : 1) k_settle(DevState D, KParams K, SettleArgs A)
{
  constexpr int kSettleThreads = settle_threads(C), kSettleWarps = kSettleThreads / kWarp;
  extern __shared__ __align__(16) unsigned char settle_smem[];
  SettleShared<C> &SH = *reinterpret_cast<SettleShared<C> *>(settle_smem);
  SettleWork<C> &U = SH.u;
  __shared__ double root[4], dsum[kSettleWarps][7], dtot[7];
  __shared__ float kp[12], rp[3], rv[3], op[3], ov[3], s_mbound;
  __shared__ unsigned red[kSettleWarps][6], levels;
  __shared__ int part[2][kSettleWarps], wcnt[2][kSettleWarps][2], s_nuns;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int blocks = C == kGrid ? (int)gridDim.x : C; // of the team
  const int rank = (int)blockIdx.x % blocks, team = (int)blockIdx.x / blocks, teams = (int)gridDim.x / blocks;
  const int gtid = rank * kSettleThreads + tid, kTeam = blocks * kSettleThreads;
  // this kernel's subhaloes: up to three of the classes, one after the other
  const bool b_large = A.count[kSettleB] <= kSettleTeams8;               // class B to the clusters
  const bool d_alone = A.grid && A.count[kSettleD] + A.count[kSettleE] == 1; // class D to the grid
  const int c0 = C == 1 ? kSettleA : C == kGrid ? kSettleE : kSettleC;
  const int n0 = A.count[c0], n1 = C != kGrid && b_large == (C > 1) ? A.count[kSettleB] : 0,
            n2 = C != 1 && d_alone == (C == kGrid) ? A.count[kSettleD] : 0, count = n0 + n1 + n2;
  float4 *const slots = A.nodes + (size_t)blockIdx.x * kSettleSlots;
  double *xch = A.xch + (size_t)team * 2 * blocks * 8;
  int par = 0, xpar = 0; // alternating halves of `part` / wcnt and of xch
  for (int q = team; q < count; q += teams)
  {
    const int s = q < n0        ? A.list[(size_t)c0 * D.S + q]
                  : q < n0 + n1 ? A.list[(size_t)kSettleB * D.S + (q - n0)]
                                : A.list[(size_t)kSettleD * D.S + (q - n0 - n1)];
    const long long off = D.off[s];
    int *ord = D.ord + off, *ord_tmp = D.ord_tmp + off;
    int nbound = D.nbound[s], nlast = D.nlast[s], corr = D.corr[s], iter = D.iter[s], wrap = D.wrap[s];
    int nuns = D.nunsample[s], spn = D.sp_len[s], cur = 0, state = kActive, done = 0, tracers = 0;
    unsigned long long built = 0;
    if (tid < 3)
    {
      rp[tid] = D.ref_pos[3 * s + tid];
      rv[tid] = D.ref_vel[3 * s + tid];
      op[tid] = D.old_pos[3 * s + tid];
      ov[tid] = D.old_vel[3 * s + tid];
    }
    if (tid == 0)
      s_mbound = D.mbound[s];
    team_sync<C>();
    for (;;)
    {
      const int n = nbound;                             // targets, and items of the partition
      const int m = corr ? nlast - nbound : nbound;     // tree sources
      if (m > kSettleSrc || (!corr && K.max_sample > 0 && !(n < K.max_sample + nuns)))
        break; // lock step goes on with it
      int cells = 0;
      float4 *T = slots;
      if (m > 0 && !settle_tree<C>(D, K, A, ord + (corr ? n : 0), m, U.t, SH.nodes, T, team, rank, blocks, root, kp, red,
                                   part, par, &levels, cells))
        break;
      built += (unsigned long long)cells;
      iter++;
      done++;
      if (m > 0 && iter == 1 && !corr && !(D.warm && D.warm[s] == 1))
        wrap = K.periodic && root[3] > (double)K.half; // a first iteration decides it (k_root)
      // targets in key order: every source, or what is still bound of the last list
      if (!corr)
      {
        cur = 0;
        spn = n;
        if (rank == 0)
          for (int i = tid; i < m; i += kSettleThreads)
            D.sp[off + i] = (int)U.t.sval[i];
      }
      else
      {
        const int *from = (cur ? D.tgt : D.sp) + off;
        int *to = (cur ? D.sp : D.tgt) + off;
        const int per = (spn + blocks - 1) / blocks, a = min(spn, rank * per), b = min(spn, a + per);
        int base = 0;
        if (C != 1)
        { // how many the blocks before this one keep
          int keep = 0, none = 0, total;
          for (int i = a + tid; i < b; i += kSettleThreads)
            keep += D.bnd[from[i]];
          block_scan(keep, part, par, total);
          team_counts<C>(total, none, base, blocks, rank, xch, xpar);
        }
        for (int i0 = a; i0 < b; i0 += kSettleThreads)
        {
          const int i = i0 + tid;
          const int p = i < b ? from[i] : 0;
          const int f = i < b ? (int)D.bnd[p] : 0;
          int total;
          const int r = block_scan(f, part, par, total);
          if (f)
            to[base + r] = p;
          base += total;
        }
        cur ^= 1;
        spn = n;
      }
      team_sync<C>();
      { // the walk (walk_chunk)
        const int *tgt = (cur ? D.tgt : D.sp) + off;
        WalkCount none;
        for (int c = rank * kSettleWarps + w; c * kWarp < n; c += blocks * kSettleWarps)
        {
          const int t = c * kWarp + lane;
          const bool valid = t < n;
          const int p = valid ? tgt[t] : 0;
          if (m == 0)
          {
            if (valid)
              D.pot[p] = 0.f;
            continue;
          }
          const float4 x = valid ? D.pm[p] : make_float4(0.f, 0.f, 0.f, 0.f);
          const float self = valid && !corr ? x.w : 0.f;
          if (wrap)
            walk_group<true, false, true>(T, D.pot, K, 0, lane, valid, p, x, self, U.walk[w], none);
          else
            walk_group<false, false, true>(T, D.pot, K, 0, lane, valid, p, x, self, U.walk[w], none);
        }
      }
      team_sync<C>();
      // energies (k_energy), and how many stay bound
      const int per = (n + blocks - 1) / blocks, k0 = min(n, rank * per), k1 = min(n, k0 + per);
      int kept = 0, kept_tr = 0;
      for (int k = k0 + tid; k < k1; k += kSettleThreads)
      {
        const int p = ord[k];
        const float4 x = D.pm[p], v = D.vu[p];
        const float e = corr ? corrected_energy(D.Ep[p], x, v, D.pot[p], op, ov, rp, rv, K)
                             : binding_energy(x, v, D.pot[p], rp, rv, K);
        D.Ep[p] = e;
        kept += e < 0.f;
        kept_tr += e < 0.f && is_tracer_bits(D.ty[p]);
      }
      kept = __reduce_add_sync(0xffffffffu, kept);
      kept_tr = __reduce_add_sync(0xffffffffu, kept_tr);
      if (lane == 0)
      {
        wcnt[par][w][0] = kept;
        wcnt[par][w][1] = kept_tr;
      }
      __syncthreads();
      kept = kept_tr = 0;
#pragma unroll
      for (int k = 0; k < kSettleWarps; k++)
      {
        kept += wcnt[par][k][0];
        kept_tr += wcnt[par][k][1];
      }
      int nb = kept, base;
      tracers = kept_tr;
      team_counts<C>(nb, tracers, base, blocks, rank, xch, xpar);
      par ^= 1;
      // stable partition (k_part_scatter)
      for (int i0 = k0; i0 < k1; i0 += kSettleThreads)
      {
        const int k = i0 + tid;
        const int p = k < k1 ? ord[k] : 0;
        const int f = k < k1 && D.Ep[p] < 0.f;
        int total;
        const int rb = base + block_scan(f, part, par, total);
        if (k < k1)
        {
          ord_tmp[f ? rb : nb + (k - rb)] = p;
          D.bnd[p] = (uint8_t)f;
        }
        base += total;
      }
      team_sync<C>();
      for (int k = k0 + tid; k < k1; k += kSettleThreads)
        ord[k] = ord_tmp[k];
      if (iter == 1 && D.nb1 && gtid == 0)
        D.nb1[s] = nb;
      nlast = n;
      nbound = nb;
      if (nb < K.min_part || (K.dm_only ? nb : tracers) < K.min_tracer)
      { // disrupted (k_after_part)
        __syncthreads();
        if (tid < 3)
        {
          rp[tid] = D.mb_pos[3 * s + tid];
          rv[tid] = D.mb_vel[3 * s + tid];
        }
        if (tid == 0)
          s_mbound = 0.f;
        nbound = 0;
        state = kDisrupted;
        break;
      }
      team_sync<C>(); // ord is whole
      if (nuns > 0)
      { // CountUnsampledParticles
        if (tid == 0)
        {
          int k = 0;
          while (k < nuns && is_nosub_bits(D.ty[ord[k]]))
            k++;
          s_nuns = k;
        }
        __syncthreads();
        nuns = s_nuns;
      }
      const int ndiff = n - nb;
      if (ndiff < nb && (K.max_sample <= 0 || ndiff < K.max_sample))
      {
        corr = 1;
        if (tid < 3)
        { // read again only after the barriers below
          op[tid] = rp[tid];
          ov[tid] = rv[tid];
        }
      }
      // the removed particles by energy, stably (k_energy_keys and the tail sort)
      if (ndiff > 1)
      {
        // keys in shared memory, or (ndiff > kSettleSrc, never of one block) in global memory
        const bool fits = C == 1 || ndiff <= kSettleSrc;
        uint32_t *key = fits ? U.tail : D.k32 + off;
        for (int j = fits ? tid : gtid; j < ndiff; j += fits ? kSettleThreads : kTeam)
          key[j] = float_to_ordered(D.Ep[ord[nb + j]]);
        if (fits)
          __syncthreads();
        else
          team_sync<C>();
        if (C == 1)
          for (int j = tid; j < ndiff; j += kSettleThreads)
            ord_tmp[nb + stable_rank(key, ndiff, j, key[j])] = ord[nb + j];
        else
          for (int j = rank * kSettleWarps + w; j < ndiff; j += blocks * kSettleWarps)
          {
            const int r = warp_rank(key, ndiff, j, key[j]);
            if (lane == 0)
              ord_tmp[nb + r] = ord[nb + j];
          }
        team_sync<C>();
        for (int j = gtid; j < ndiff; j += kTeam)
          ord[nb + j] = ord_tmp[nb + j];
      }
      // centre-of-mass frame (k_com, frame_from_sums)
      {
        const float4 o = D.pm[ord[0]];
        FloatSum acc[8]; // the last one is padding
        for (int k = gtid; k < nb; k += kTeam)
        {
          const int p = ord[k];
          const float4 x = D.pm[p], v = D.vu[p];
          const float mass = x.w;
          acc[0].add(mass);
          const float xs[3] = {x.x, x.y, x.z}, os[3] = {o.x, o.y, o.z};
#pragma unroll
          for (int d = 0; d < 3; d++)
            acc[1 + d].add(com_offset(xs[d], os[d], mass, K));
          acc[4].add(__fmul_rn(v.x, mass));
          acc[5].add(__fmul_rn(v.y, mass));
          acc[6].add(__fmul_rn(v.z, mass));
        }
        const double sum = warp_sums(acc).value();
        if ((lane & 3) == 0 && lane < 28)
          dsum[w][lane >> 2] = sum;
        __syncthreads();
        if (tid < 7)
        {
          double v = 0.;
          for (int k = 0; k < kSettleWarps; k++)
            v += dsum[k][tid];
          dtot[tid] = v;
          if (C != 1)
            xch[((size_t)xpar * blocks + rank) * 8 + tid] = v;
        }
        if (C != 1)
        { // warp w adds quantity w over the blocks, in the same order everywhere
          team_sync<C>();
          double v = 0.;
          if (w < 7)
            for (int r = lane; r < blocks; r += kWarp)
              v += xch[((size_t)xpar * blocks + r) * 8 + w];
          for (int h = 16; h > 0; h >>= 1)
            v += __shfl_xor_sync(0xffffffffu, v, h);
          if (w < 7 && lane == 0)
            dtot[w] = v;
          xpar ^= 1;
        }
        __syncthreads();
        if (tid < 6)
        {
          const int d = tid % 3;
          const double org[3] = {o.x, o.y, o.z};
          double v = dtot[1 + tid] / dtot[0];
          if (tid < 3 && K.periodic)
            v += org[d];
          (tid < 3 ? rp : rv)[d] = (float)v;
        }
        if (tid == 6)
          s_mbound = (float)dtot[0];
      }
      if ((float)nb >= __fmul_rn((float)nlast, K.bmp))
        state = kConverged;
      else if (iter >= K.max_iter)
        state = kMaxIter;
      if (state != kActive)
        break;
      team_sync<C>();
    }
    __syncthreads();
    if (state == kActive && cur)
    { // lock step reads the list from sp
      for (int i = gtid; i < spn; i += kTeam)
        D.sp[off + i] = D.tgt[off + i];
    }
    if (rank == 0)
    {
      if (tid < 3)
      {
        D.ref_pos[3 * s + tid] = rp[tid];
        D.ref_vel[3 * s + tid] = rv[tid];
        D.old_pos[3 * s + tid] = op[tid];
        D.old_vel[3 * s + tid] = ov[tid];
      }
      if (tid == 0)
      {
        D.nbound[s] = nbound;
        D.nlast[s] = nlast;
        D.corr[s] = corr;
        D.iter[s] = iter;
        D.wrap[s] = wrap;
        D.nunsample[s] = nuns;
        D.sp_len[s] = spn;
        D.state[s] = state;
        D.mbound[s] = s_mbound;
        atomicAdd(A.cells, built);
        atomicMax(A.most, done);
      }
    }
    team_sync<C>(); // the next subhalo takes the shared arrays
  }
}

} // namespace
} // namespace hbtg
