// Fixed-point columns: the linear operators of the FP64 path on the integer
// pipes.  GB300 issues 1.6 FP64 operations per clock and SM; beside them,
// without slowing them, it issues about 42 32 x 32 + 64 -> 64 multiply-adds
// and 64 to 128 shifts, adds and logic operations (measured).  The operators
// of an element are linear maps with constant coefficients, so they run on
// 64-bit integers with one exponent per (element, variable) column and leave
// the FP64 pipe to the flux evaluations.
//
// A column value is v 2^(E - 1082) with |v| <= 2^60; the bound of the column
// is 2^(E - 1022), so E compares with the exponent field of a double.  A
// coefficient is a 60-bit fraction C = ch 2^30 + cl (cl signed), an operand is
// split into v = h 2^30 + l, and c v = h ch + (h cl + l ch) / 2^30 takes three
// multiply-adds: the dropped product l cl is below one unit of the result, so
// a term's error is 2^-60 of the bound where the FP64 form's is 2^-53 of the
// partial sum.  Conversions are integer code too (a hardware conversion
// occupies the FP64 pipe).  NaN and infinities make a column's results NaN
// (fx_poison); columns beyond 2^1017 likewise, columns of subnormal numbers
// are zero.
#pragma once

#include <cstdint>

namespace adg {

constexpr int kFxLimb = 30;
constexpr int kFxLow = (1 << kFxLimb) - 1;
constexpr long long kFxHalf = 1LL << (kFxLimb - 1);  // half a unit of the sum of the middle products

__device__ __forceinline__ int fx_hi(long long v) { return (int)(v >> kFxLimb); }
__device__ __forceinline__ int fx_lo(long long v) { return (int)v & kFxLow; }

// Limbs of a coefficient's 60-bit fraction.
struct FxCoef {
  int h, l;
};

// Sum of products.  A product adds at most 1.5 2^60 to the middle sum B: it
// is folded after four.
struct FxSum {
  long long A = 0, B = kFxHalf;
  __device__ __forceinline__ void add(long long v) { A += v; }
  __device__ __forceinline__ void mul(int h, int l, int ch, int cl) {
    A = (long long)h * ch + A;
    B = (long long)h * cl + B;
    B = (long long)l * ch + B;
  }
  __device__ __forceinline__ void mul(long long v, const FxCoef& c) { mul(fx_hi(v), fx_lo(v), c.h, c.l); }
  // a compile-time coefficient: the dropped l cl made up for in the mean (l
  // is uniform), which costs one constant per sum
  __device__ __forceinline__ void mulc(int h, int l, int ch, int cl) {
    mul(h, l, ch, cl);
    B += cl >> 1;
  }
  __device__ __forceinline__ void fold() {
    A += B >> kFxLimb;
    B = 0;
  }
  __device__ __forceinline__ long long get() const { return A + (B >> kFxLimb); }
};

__device__ __forceinline__ int fx_exp_field(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// Quiet-NaN bits for every output of a column whose exponent is that of
// infinities and NaN or leaves the range of doubles.
constexpr int kFxMaxExp = 2039;
constexpr int kFxNanExp = 4096;
__device__ __forceinline__ int fx_poison(int E) { return E > kFxMaxExp ? 0x7ff80000 : 0; }

// x as a column value of exponent E >= the exponent field of x (exact down to
// 2^-7 of the bound, truncated toward zero below; a negative x one unit
// lower: its complement, not its negative); zero and subnormal numbers zero.
__device__ __forceinline__ long long fx_from_double(double x, int E) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
  const unsigned long long m = ((unsigned long long)mh << 39) | ((unsigned long long)(unsigned)lo << 7);
  const int f = (hi >> 20) & 0x7ff, r = E - f;
  const long long s = hi >> 31;  // 0 or -1
  return f ? (long long)(m >> (r < 63 ? r : 63)) ^ s : 0;
}

// Column value to the nearest double (a negative one from its complement);
// nan_bits: fx_poison of the column.  The common case has a bit set in the
// high word and a column exponent whose doubles are normal.
static __device__ __noinline__ double fx_to_double_small(long long v, int E, int nan_bits);
__device__ __forceinline__ double fx_to_double(long long v, int E, int nan_bits) {
  const int s = (int)(v >> 32) >> 31;
  const unsigned hi = (unsigned)((int)(v >> 32) ^ s), lo = (unsigned)((int)v ^ s);
  if (hi == 0 || E < 64) return fx_to_double_small(v, E, nan_bits);
  const int n = __clz((int)hi);
  const unsigned mh = __funnelshift_l(lo, hi, n), ml = lo << n;  // leading bit at 31
  // significand with its leading bit, rounded; the bit adds one to the field
  const unsigned long long d = ((((unsigned long long)mh << 32) | ml) >> 11) + ((ml >> 10) & 1u);
  const int field = (E + 3 - n) << 20;
  return __hiloint2double(((int)(d >> 32) + field) | (s & (int)0x80000000) | nan_bits, (int)d);
}
static __device__ __noinline__ double fx_to_double_small(long long v, int E, int nan_bits) {
  const long long s = v >> 63;
  const unsigned long long a = (unsigned long long)(v ^ s);
  const int n = __clzll((long long)a);
  const unsigned long long m = n < 64 ? a << n : 0;
  const int ef = E + 3 - n;
  const unsigned long long d = (m >> 11) + ((m >> 10) & 1) + ((unsigned long long)(unsigned)ef << 52);
  if (ef < 0 || (long long)m >= 0) return __hiloint2double(nan_bits, 0);
  return __hiloint2double((int)(d >> 32) | ((int)s & (int)0x80000000) | nan_bits, (int)d);
}

// v / 2, rounded.
__device__ __forceinline__ long long fx_half(long long v) { return (v + 1) >> 1; }

// v 2^-shift, truncated downward.
__device__ __forceinline__ long long fx_align(long long v, int shift) { return v >> (shift < 63 ? shift : 63); }
// the same for a shift of either sign
__device__ __forceinline__ long long fx_move(long long v, int shift) {
  if (shift <= 0) return v << -shift;
  return fx_align(v, shift);
}

// A positive double as a 60-bit fraction times 2^(ef - 1022).
struct FxFactor {
  FxCoef c;
  int ef;
};
__device__ __forceinline__ FxFactor fx_factor(double c) {
  const int hi = __double2hiint(c), lo = __double2loint(c);
  const unsigned long long m = ((unsigned long long)(((unsigned)hi & 0xfffffu) | 0x100000u) << 39) |
                               ((unsigned long long)(unsigned)lo << 7);
  return {{(int)(m >> kFxLimb), (int)m & kFxLow}, (hi >> 20) & 0x7ff};
}
__device__ __forceinline__ long long fx_scale(long long v, const FxFactor& f) {
  FxSum s;
  s.mul(v, f.c);
  return s.get();
}
// Exponent of fx_scale's result for operands of exponent e + growth (beyond
// every double's when the operands or the factor are not finite).
__device__ __forceinline__ int fx_scaled_exp(int e, int growth, const FxFactor& f) {
  return e > kFxMaxExp || f.ef == 2047 ? kFxNanExp : e + growth + f.ef - 1022;
}

// Product of two column values: exponents add, less 1022.
__device__ __forceinline__ long long fx_mul(int ah, int al, int bh, int bl) {
  FxSum s;
  s.mul(ah, al, bh, bl);
  return s.get();
}

__device__ __forceinline__ float fx_rcp_estimate(float x) {
#ifdef __CUDACC__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else  // a host build (tests)
  return 1.0f / x;
#endif
}

// Reciprocal of v, 2^40 <= v < 2^60, n = clz(v): 2^(123 - n) / v, in
// (2^59, 2^60].  The FP32 estimate r of the significand x in [1, 2) (24
// bits), e = 1 - x r exactly, one third-order Householder step r (1 + e + e^2).
__device__ __forceinline__ long long fx_reciprocal(long long v, int n) {
  const unsigned long long x = (unsigned long long)v << (n - 4);  // [2^59, 2^60)
  const float r = fx_rcp_estimate(__int_as_float(0x3f800000 | (((int)(x >> 36)) & 0x7fffff)));
  const unsigned r0 = (unsigned)__float2int_rn(r * 16777216.0f);  // 2^24 r, exact
  const long long e = -(long long)(x * r0);                       // 2^83 e: the product's 2^83 leaves 64 bits
  const int eh = (int)(e >> 32);
  const long long p = (e >> 23) + (((long long)eh * eh) >> 42);   // 2^60 (e + e^2)
  return ((long long)r0 << 36) + (((long long)r0 * p) >> 24);
}

// Exponent E with sum |x_n| <= 2^(E - 1022), x_n at stride s: the largest
// exponent field plus what the sum of the truncated significands (20 bits,
// rounded up) needs.  2047 (infinity or NaN) stays above kFxMaxExp.
template <int N>
__device__ __forceinline__ int fx_norm_exp(const double* x, int s) {
  int top = 0;
#pragma unroll 4
  for (int n = 0; n < N; ++n) top = max(top, fx_exp_field(x[n * s]));
  int sum = 0;
#pragma unroll 4
  for (int n = 0; n < N; ++n) {
    const int hi = __double2hiint(x[n * s]);
    const int r = top - ((hi >> 20) & 0x7ff);
    sum += (int)((((unsigned)hi & 0xfffffu) | 0x100000u) >> (r < 31 ? r : 31)) + 1;
  }
  const int bits = 32 - __clz(sum);  // sum < 2^bits, in units of 2^(top - 1023 - 20)
  return top + (bits > 21 ? bits - 21 : 0);
}

// ---------------------------------------------------------------------------
// The Euler fluxes of a point (Compressible_Euler.h:370-487, 562-589) on
// column values.  A 60-bit product is about 10 integer instructions, a third
// of what one FP64 operation keeps its pipe busy for; the exponents of all
// intermediate values are the element's, so a point does no normalisation
// but the density's.
// ---------------------------------------------------------------------------

// Smallest pressure the integer path takes, as a column value of exponent x:
// the model's floor, 10 2^-52 = 5 2^(1031 - 1082), which the FP64 evaluation
// applies, and 2^-40 of the bound.
__device__ __forceinline__ long long fx_min_pressure(int x) {
  const int s = 1031 - x;
  return s < 18 ? 1LL << 20 : 5LL << (s < 60 ? s : 60);
}

// Exponents: em momenta, ee energy, er density; n: the largest number of
// leading zeros of the element's densities, which bounds 1 / rho; gef: that
// of gamma - 1 (FxFactor::ef).  Pressure and enthalpy are bounded by the
// energy (a point has p >= 0 or goes to the FP64 evaluation), the kinetic
// terms m v by products of bounds: `lost` is by how much the largest of them
// exceeds the energy's bound.
template <int D>
struct FxFluxExp {
  int xv[D];  // velocities
  int xk[D];  // m_d v_d
  int xp, xe, xd[D];
  int lost;
  __device__ __forceinline__ FxFluxExp(const int* em, int ee, int er, int n, int gef) {
    xp = ee + gef - 1022;
    xe = max(ee, xp) + 1;
    lost = -kFxNanExp;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      xv[d] = em[d] + n - er + 1019;
      xk[d] = xv[d] + em[d] - 1022;
      lost = max(lost, xk[d] - ee);
      xd[d] = max(xk[d], xp) + 1;
    }
  }
  // exponent of flux d of variable q >= 1
  __device__ __forceinline__ int flux(int d, int q, const int* em) const {
    int x = xe + xv[0] - 1022, o = xd[0];
#pragma unroll
    for (int k = 0; k < D; ++k)
      if (k == d) {
        x = xe + xv[k] - 1022;
        o = xd[k];
      }
    if (q == D + 1) return x;
    if (q == d + 1) return o;
    int v = xv[0], m = em[0];
#pragma unroll
    for (int k = 0; k < D; ++k) {
      if (k == d) v = xv[k];
      if (k == q - 1) m = em[k];
    }
    return v + m - 1022;
  }
};

// Smallest density the integer path takes (2^-20 of its bound), and the most
// the densities of an element may lie apart and its kinetic terms exceed the
// energy's bound (as powers of two): the velocities' and the kinetic terms'
// bounds are that much larger than their values.  Error of the fluxes,
// relative to the element's largest, here / in FP64, over random elements of
// every (D, P): within these lines energy 3.6e-16 / 5.1e-16, momentum 4.1e-16
// / 4.8e-16 across and 5.2e-16 / 3.6e-15 along; densities 2^3 apart energy
// 5.1e-16 / 4.1e-16, 2^6 apart 2.4e-15 / 4.3e-16.
constexpr long long kFxMinRho = 1LL << 40;
constexpr int kFxRhoSpan = 2;
constexpr int kFxKineticSpan = 4;

// Fluxes F[d][q - 1], q >= 1, at exponents x.flux(d, q).  False where the
// density is out of range or the pressure below fx_min_pressure: such points
// are for the FP64 evaluation.
template <int D>
__device__ __forceinline__ bool fx_euler_flux(const long long* u, const FxFluxExp<D>& x, int ee, int n_max,
                                              const FxFactor& gm1, long long (&F)[D][D + 1]) {
  if (u[0] < kFxMinRho || u[0] >= (1LL << 60)) return false;
  const int n = __clz((int)(u[0] >> 32));
  if (n_max - n > kFxRhoSpan || x.lost > kFxKineticSpan) return false;
  const long long r = fx_reciprocal(u[0], n) >> (n_max - n);
  const int rh = fx_hi(r), rl = fx_lo(r);
  int mh[D], ml[D], vh[D], vl[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    mh[d] = fx_hi(u[d + 1]);
    ml[d] = fx_lo(u[d + 1]);
    const long long v = fx_mul(mh[d], ml[d], rh, rl);
    vh[d] = fx_hi(v);
    vl[d] = fx_lo(v);
  }
  // E - sum m v / 2 at the energy's exponent, or up to two bits above it so
  // that the kinetic terms (whose shift is -1 or more, then) stay in the word
  const int up = max(x.lost - 2, 0);
  long long p = u[D + 1] >> up;
  long long w[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    w[d] = fx_mul(mh[d], ml[d], vh[d], vl[d]);
    p -= fx_align(w[d] << 1, ee + up - x.xk[d] + 2);
  }
  p = fx_scale(p << up, gm1);
  if (p < fx_min_pressure(x.xp)) return false;
  const long long ep = fx_align(u[D + 1], x.xe - ee) + fx_align(p, x.xe - x.xp);
  const int eh = fx_hi(ep), el = fx_lo(ep);
#pragma unroll
  for (int d = 0; d < D; ++d) {
#pragma unroll
    for (int k = 0; k < D; ++k) {
      if (k < d)
        F[d][k] = F[k][d];  // m_k v_d = m_d v_k
      else if (k == d)
        F[d][k] = fx_align(w[d], x.xd[d] - x.xk[d]) + fx_align(p, x.xd[d] - x.xp);
      else
        F[d][k] = fx_mul(mh[k], ml[k], vh[d], vl[d]);
    }
    F[d][D] = fx_mul(eh, el, vh[d], vl[d]);
  }
  return true;
}

}  // namespace adg
