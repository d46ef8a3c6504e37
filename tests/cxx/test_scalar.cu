// The kernels' own scalar functions (adg_device.cuh, adg_fx.cuh) against
// CUDA's operators and exact integer arithmetic, on the GPU.  Prints one count
// of differing arguments, with the first of them, per function.
#include <cstdio>

#include "adg_device.cuh"
#include "adg_fx.cuh"

using namespace adg;

struct Count {
  unsigned long long n, first;
};

__device__ unsigned long long mix(unsigned long long x) {  // splitmix64
  x += 0x9e3779b97f4a7c15ULL;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
  return x ^ (x >> 31);
}
__device__ void note(Count* c, bool bad, unsigned long long arg) {
  if (bad && atomicAdd(&c->n, 1ULL) == 0) c->first = arg;
}
__device__ bool differ(double a, double b) {
  return __double_as_longlong(a) != __double_as_longlong(b) && !(a != a && b != b);
}
__device__ bool differ(float a, float b) { return __float_as_int(a) != __float_as_int(b) && !(a != a && b != b); }

// Argument i: any bit pattern; a significand within 64 units of 1, sqrt(2) or
// 2 (and the borders of the fast ranges at 2^+-900); ties of the rounding to
// FP32 and their neighbours at its exponents, subnormal ones among them.
__device__ double argument(unsigned long long i) {
  const unsigned long long r = mix(i);
  unsigned long long b = r;
  if (i % 4 == 1) {
    const unsigned long long at[3] = {0, 0x6a09e667f3bcdULL, 0xfffffffffffffULL};
    b = (r & 0xfff0000000000000ULL) | ((at[i / 4 % 3] + mix(r) % 129 - 64) & 0xfffffffffffffULL);
  } else if (i % 4 == 2) {
    const unsigned long long e = i / 4 % 2 ? 121 + mix(r) % 5 : 1921 + mix(r) % 5;
    b = (r & 0x800fffffffffffffULL) | e << 52;
  } else if (i % 4 == 3) {
    const unsigned long long e = 870 + mix(r) % 310;
    const unsigned long long low[5] = {0x10000000, 0x0fffffff, 0x10000001, 0, 0x1fffffff};
    b = (r & 0x800fffffe0000000ULL) | e << 52 | low[i / 4 % 5];
  }
  return __longlong_as_double((long long)b);
}

__global__ void k_check(unsigned long long n, Count* c) {
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const double x = argument(i);
    const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
    note(c + 0, differ(fast_rcp(x), 1.0 / x), bits);
    note(c + 1, differ(fast_sqrt(x), sqrt(x)), bits);
    note(c + 2, differ(to_float(x), (float)x), bits);
    const float f = __int_as_float((int)(bits >> (i % 33)));
    note(c + 3, differ(to_double(f), (double)f), (unsigned)__float_as_int(f));
    // 2^(123 - z) / v in units of the result, exact in 128 bits
    const long long v = i % 5 ? (long long)(bits >> 4 | 1ULL << (40 + i % 20)) & ((1LL << (41 + i % 20)) - 1)
                              : i % 10 ? (1LL << (40 + i % 20)) + (long long)(bits % 65)
                                       : (1LL << (41 + i % 20)) - 1 - (long long)(bits % 65);
    const int z = __clzll(v);
    const long long r = fx_reciprocal(v, z);
    const __int128 d = (__int128)r * v - ((__int128)1 << (123 - z));
    // the estimate's error is below 2^-22, so the cut-off third order is 2^-6
    // units; three truncations of one unit each
    note(c + 4, (d < 0 ? -d : d) > (__int128)4 * v, (unsigned long long)v);
  }
}

int main() {
  Count* c;
  const char* name[5] = {"fast_rcp", "fast_sqrt", "to_float", "to_double", "fx_reciprocal"};
  if (cudaMallocManaged(&c, 5 * sizeof(Count)) != cudaSuccess) return 2;
  for (int i = 0; i < 5; ++i) c[i] = {0, 0};
  k_check<<<152 * 8, 256>>>(1ULL << 27, c);
  if (cudaDeviceSynchronize() != cudaSuccess) return 2;
  for (int i = 0; i < 5; ++i) std::printf("%s %llu %016llx\n", name[i], c[i].n, c[i].first);
  return 0;
}
