"""The noise's sine in integer arithmetic (kernels/noise_sin.cuh, se_sin_fast) against the one that
defines it (se_sin, binary64), compiled for the CPU: the same bits for every binary32 number of the
integer path's range, and for numbers around and beyond it."""
import ctypes
import os
import subprocess

CODE = r"""
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <thread>
#include <vector>
#define __device__
#define __forceinline__ inline
static inline double __dadd_rn(double a, double b) { return a + b; }
static inline double __dsub_rn(double a, double b) { return a - b; }
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline float __double2float_rn(double a) { return (float)a; }
static inline float __ull2float_rn(uint64_t a) { return (float)a; }
static inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
static inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) {
  return (uint32_t)((((uint64_t)hi << 32) | lo) >> (s & 31));
}
static inline uint32_t __float_as_uint(float f) {
  uint32_t u;
  memcpy(&u, &f, 4);
  return u;
}
static inline float __uint_as_float(uint32_t u) {
  float f;
  memcpy(&f, &u, 4);
  return f;
}
using std::fabs;
using std::floor;
#include "noise_sin.cuh"
static bool differ(uint32_t bits) {
  const float x = __uint_as_float(bits), a = se::rt::se_sin_fast(x), b = se::rt::se_sin(x);
  return __float_as_uint(a) != __float_as_uint(b) && !(std::isnan(a) && std::isnan(b));
}
// numbers whose bits lie in [lo, hi), every `step`-th, both signs
extern "C" unsigned long long differing(uint32_t lo, uint32_t hi, uint32_t step) {
  const unsigned n = std::max(1u, std::thread::hardware_concurrency());
  std::atomic<unsigned long long> bad{0};
  std::vector<std::thread> ts;
  for (unsigned t = 0; t < n; ++t)
    ts.emplace_back([&, t] {
      unsigned long long d = 0;
      for (uint64_t b = lo + (uint64_t)step * t; b < hi; b += (uint64_t)step * n)
        d += differ((uint32_t)b) + differ((uint32_t)b | 0x80000000u);
      bad += d;
    });
  for (auto& t : ts) t.join();
  return bad;
}
"""


def test_integer_sine_has_the_binary64_sines_bits(tmp_path):
    from sandengine_gb300 import build as B
    src, so = tmp_path / "sine.cpp", tmp_path / "sine.so"
    src.write_text(CODE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-ffp-contract=off", "-pthread",
                    f"-I{os.path.join(B.CSRC, 'kernels')}", str(src), "-o", str(so)], check=True)
    f = ctypes.CDLL(str(so)).differing
    f.restype, f.argtypes = ctypes.c_ulonglong, [ctypes.c_uint32] * 3
    lo, hi = (127 + 6) << 23, (127 + 26) << 23  # 2^6 <= |x| < 2^26
    assert f(lo, hi, 1) == 0
    assert f(lo - 65536, lo, 1) == 0 and f(hi, hi + 65536, 1) == 0
    assert f(0, 1 << 31, 65521) == 0  # NaN and infinities among them
