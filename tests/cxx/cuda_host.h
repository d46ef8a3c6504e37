// The CUDA qualifiers and integer intrinsics that the fixed-point device code
// (adg_fx.cuh) uses, for a host build of that header.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__

using std::max;
using std::min;

static inline int __clz(int x) { return x ? __builtin_clz((unsigned)x) : 32; }
static inline int __clzll(long long x) { return x ? __builtin_clzll((unsigned long long)x) : 64; }
static inline long long __double_as_longlong(double x) {
  long long v;
  std::memcpy(&v, &x, 8);
  return v;
}
static inline double __longlong_as_double(long long v) {
  double x;
  std::memcpy(&x, &v, 8);
  return x;
}
static inline int __double2hiint(double x) { return (int)(__double_as_longlong(x) >> 32); }
static inline int __double2loint(double x) { return (int)__double_as_longlong(x); }
static inline double __hiloint2double(int h, int l) {
  return __longlong_as_double((long long)(((unsigned long long)(unsigned)h << 32) | (unsigned)l));
}
static inline unsigned __funnelshift_l(unsigned lo, unsigned hi, int n) {
  n &= 31;
  return n ? (hi << n) | (lo >> (32 - n)) : hi;
}
static inline float __int_as_float(int i) {
  float f;
  std::memcpy(&f, &i, 4);
  return f;
}
static inline int __float_as_int(float f) {
  int i;
  std::memcpy(&i, &f, 4);
  return i;
}
static inline int __float2int_rn(float f) { return (int)std::lrintf(f); }
