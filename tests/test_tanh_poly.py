"""The polynomial of the pulsed force's tanh (wendy_gb300/csrc/wg_tanh.cuh) against
113-bit arithmetic, over every cell of its table: the header is compiled here as host
code, with the device intrinsics it uses spelled out.  Its narrow products are to be
no further off, at worst and on average, than full 64-bit products."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "wendy_gb300", "csrc")

PROGRAM = r"""
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#if __LDBL_MANT_DIG__ == 113
typedef long double Quad;
static Quad qtanh(Quad a) { return tanhl(a); }
#else
#include <quadmath.h>
typedef __float128 Quad;
static Quad qtanh(Quad a) { return tanhq(a); }
#endif
#define __host__
#define __device__
#define __forceinline__ inline
#define __noinline__
#define __align__(n) __attribute__((aligned(n)))
using std::min;
struct longlong2 { long long x, y; };
template <typename T> static T __ldg(const T* p) { return *p; }
static uint64_t __umul64hi(uint64_t a, uint64_t b) { return (uint64_t)((unsigned __int128)a * b >> 64); }
static long long __mul64hi(long long a, long long b) { return (long long)((__int128)a * b >> 64); }
static int __mulhi(int a, int b) { return (int)((long long)a * b >> 32); }
static uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)((uint64_t)a * b >> 32); }
static int __clz(int a) { return a ? __builtin_clz((unsigned)a) : 32; }
static int __clzll(long long a) { return a ? __builtin_clzll((unsigned long long)a) : 64; }
static uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, int s) {
  return (uint32_t)(((((uint64_t)hi << 32) | lo) << (s & 31)) >> 32);
}
static uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, int s) {
  return (uint32_t)((((uint64_t)hi << 32) | lo) >> (s & 31));
}
static long long __double_as_longlong(double d) { long long b; memcpy(&b, &d, 8); return b; }
static double __longlong_as_double(long long b) { double d; memcpy(&d, &b, 8); return d; }
static int __double2hiint(double d) { return (int)(__double_as_longlong(d) >> 32); }
static int __double2loint(double d) { return (int)__double_as_longlong(d); }
static long long __double2ll_rn(double d) { return llrint(d); }
static float __frcp_rn(float f) { return 1.f / f; }
static float __ull2float_rn(uint64_t u) { return (float)u; }
static uint64_t __float2ull_rn(float f) { return (uint64_t)llrintf(f); }
#include "wg_tanh.cuh"

int main() {
  const Quad one62 = (Quad)(1ull << 62);
  double worst[2] = {0, 0}, sum[2] = {0, 0};
  uint64_t rs = 88172645463325252ull;
  long count = 0;
  for (int i = 1; i < wg::kTanhCells; ++i) {
    const Quad a = (Quad)i / 1024, t = qtanh(a);
    Quad c[10] = {t};  // Taylor coefficients about a, from y' = 1 - y^2
    for (int n = 0; n < 9; ++n) {
      Quad q = n == 0 ? 1 : 0;
      for (int j = 0; j <= n; ++j) q -= c[j] * c[n - j];
      c[n + 1] = q / (n + 1);
    }
    // the row as the table has it, with tanh at the cell's start correctly rounded
    long long row[6];
    wg::tanh_table_row(i, row);
    row[0] = (long long)(t * one62 + (Quad)0.5);
    row[1] = (long long)((1ull << 62) - wg::tanh_fx::mul62(row[0], row[0]));
    for (int k = 0; k < 150; ++k) {
      rs ^= rs << 13; rs ^= rs >> 7; rs ^= rs << 17;
      const double y = (i + (double)(rs >> 11) * 0x1p-53) * 0x1p-10;
      if ((int)(y * 1024) != i) continue;
      const Quad dd = (Quad)y - a;
      const uint64_t D = (uint64_t)(dd * (Quad)0x1p64);
      Quad exact = 0;
      for (int n = 9; n >= 0; --n) exact = exact * dd + c[n];
      long long full = row[5];
      for (int n = 4; n >= 0; --n) full = row[n] + __mul64hi(full, (long long)D);
      const long long got = wg::tanh_poly({row[0], row[1]}, {row[2], row[3]}, {row[4], row[5]},
                                          (uint32_t)(D >> 32), (uint32_t)D);
      const double e[2] = {(double)((Quad)full - exact * one62),
                           (double)((Quad)got - exact * one62)};
      for (int q = 0; q < 2; ++q) {
        worst[q] = std::max(worst[q], std::fabs(e[q]));
        sum[q] += std::fabs(e[q]);
      }
      ++count;
    }
  }
  printf("%.4f %.4f %.4f %.4f\n", worst[0], worst[1], sum[0] / count, sum[1] / count);
  return 0;
}
"""


def test_narrow_products_are_no_less_accurate_than_full_ones(tmp_path):
    src, exe = tmp_path / "poly.cpp", tmp_path / "poly"
    src.write_text(PROGRAM)
    r = subprocess.run(["g++", "-std=gnu++17", "-O2", "-I", CSRC, str(src), "-o", str(exe),
                        "-lquadmath"], capture_output=True, text=True)
    if r.returncode != 0 and "quadmath" in r.stderr:
        r = subprocess.run(["g++", "-std=gnu++17", "-O2", "-I", CSRC, str(src), "-o", str(exe)],
                           capture_output=True, text=True)
        if r.returncode != 0 and "quadmath.h" in r.stderr:
            pytest.skip("no 113-bit arithmetic here")
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    worst_full, worst, mean_full, mean = map(float, out.split())
    assert worst <= worst_full and mean <= mean_full, out
    assert worst <= 2.  # 2^-61 absolute
