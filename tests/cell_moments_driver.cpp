// csrc/moments.cuh on the host: cell_moments against cell_moments_fp64, bit for
// bit, over random cells of one kind.  Usage: driver <kind> <cells> <seed>.
// The device's intrinsics are the IEEE operations they name (compiled without
// contraction).
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <algorithm>
#include <random>

#include <cuda_runtime.h>

#ifndef __noinline__
#define __noinline__
#endif
using std::max;
using std::min;
template <typename To, typename From>
static To bits_as(From v)
{
  To t;
  std::memcpy(&t, &v, sizeof(t));
  return t;
}
static unsigned __float_as_uint(float v) { return bits_as<unsigned>(v); }
static float __uint_as_float(unsigned v) { return bits_as<float>(v); }
static int __float_as_int(float v) { return bits_as<int>(v); }
static float __fadd_rn(float a, float b) { return a + b; }
static float __fsub_rn(float a, float b) { return a - b; }
static float __fmul_rn(float a, float b) { return a * b; }
static float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
static float __frcp_rn(float a) { return 1.f / a; }
static double __dadd_rn(double a, double b) { return a + b; }
static double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static double __ddiv_rn(double a, double b) { return a / b; }
static float __double2float_rn(double a) { return (float)a; }
static float __uint2float_rn(unsigned a) { return (float)a; }
static unsigned __float2uint_rz(float a) { return (unsigned)a; }
static int __ffs(int v) { return __builtin_ffs(v); }
static int __clzll(long long v) { return v ? __builtin_clzll((unsigned long long)v) : 64; }
static int __popc(unsigned v) { return __builtin_popcount(v); }
static struct { int x; } threadIdx;
template <typename T> static T __ldg(const T *p) { return *p; }
static unsigned __ballot_sync(unsigned, bool v) { return v; }
template <typename T> static T __shfl_sync(unsigned, T v, int) { return v; }

#include "../hbt-herons_gb300/csrc/moments.cuh"

int main(int argc, char **argv)
{
  const int kind = std::atoi(argv[1]), cells = std::atoi(argv[2]);
  std::mt19937_64 rng(std::atoi(argv[3]));
  auto uni = [&](double a, double b) { return (float)std::uniform_real_distribution<double>(a, b)(rng); };
  auto integer = [&](int a, int b) { return (int)std::uniform_int_distribution<int>(a, b)(rng); };
  long long differ = 0;
  for (int c = 0; c < cells; c++)
  {
    const int n = kind == 5 ? integer(9, 12) : integer(1, 8);
    float x[12][3], m[12];
    for (int k = 0; k < n; k++)
    {
      m[k] = kind == 1 ? std::ldexp(uni(1, 2), integer(0, 11)) : kind == 2 ? (float)integer(1, 4) : uni(0.5, 2);
      for (int d = 0; d < 3; d++)
      {
        if (kind == 2) // a coarse grid and small whole masses: centres halfway between floats
          x[k][d] = 70.f + (float)integer(-3, 3) * std::ldexp(1.f, -17);
        else if (kind == 3 || kind == 4) // both signs
          x[k][d] = uni(-1, 1);
        else
          x[k][d] = 70.f + uni(-1, 1);
      }
    }
    if (kind == 4) // opposite pairs: every sum is zero, the partial sums are not representable
      for (int k = 0; k < n; k++)
      {
        if (k < n / 2)
        {
          const int o = k + n / 2;
          m[k] = m[o] = std::ldexp(uni(1, 2), integer(0, 9));
          for (int d = 0; d < 3; d++)
            x[o][d] = -x[k][d];
        }
        else if (n % 2 && k == n - 1)
          for (int d = 0; d < 3; d++)
            x[k][d] = 0.f;
      }
    float4 a[2 + 12 + 1], b[2 + 12 + 1];
    std::memset(a, 0, sizeof(a));
    a[0].w = -1.f; // a cell
    a[1].y = bits_as<float>(2 + n);
    for (int k = 0; k < n; k++)
      a[2 + k] = make_float4(x[k][0], x[k][1], x[k][2], m[k]);
    std::memcpy(b, a, sizeof(a));
    hbtg::cell_moments(a, 0);
    hbtg::cell_moments_fp64(b, 0);
    differ += std::memcmp(a, b, sizeof(a)) != 0;
  }
  std::printf("%lld\n", differ);
}
