// Checks of the fixed-point columns (adg_fx.cuh) built for the host: one check
// per argument, "ok" or what failed on standard output.
#include "cuda_host.h"

#include <array>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <string>
#include <vector>

#include "adg_fx.cuh"

using namespace adg;

#define CHECK(c, ...)        \
  if (!(c)) {                \
    std::printf(__VA_ARGS__); \
    std::printf("\n");       \
    std::exit(1);            \
  }

static double field_value(long long v, int E) { return std::ldexp((double)v, E - 1082); }

// A point's fluxes from doubles, every column's exponent that of one more bit
// than the value (as fx_norm_exp gives a single mode).
template <int D>
static bool point_flux(const double* u, double gamma, double (&F)[D][D + 1]) {
  long long v[D + 2];
  int e[D + 2];
  for (int q = 0; q < D + 2; ++q) {
    e[q] = fx_norm_exp<1>(u + q, 1);
    v[q] = fx_from_double(u[q], e[q]);
  }
  const int n = __clz((int)(v[0] >> 32));
  const FxFactor gm1 = fx_factor(gamma - 1.0);
  const FxFluxExp<D> x(e + 1, e[D + 1], e[0], n, gm1.ef);
  long long f[D][D + 1];
  if (!fx_euler_flux<D>(v, x, e[D + 1], n, gm1, f)) return false;
  for (int d = 0; d < D; ++d)
    for (int q = 0; q <= D; ++q) F[d][q] = field_value(f[d][q], x.flux(d, q + 1, e + 1));
  return true;
}

// A pressure below the model's floor, 10 2^-52, is for the FP64 evaluation,
// which applies it, whatever the scale of the state; above the floor the
// momentum flux is the pressure.
template <int D>
static void pressure_floor() {
  const double floor = 10.0 * std::ldexp(1.0, -52);
  for (double rho : {1e-15, 1e-12, 1e-3, 1.0})
    for (double p = 1e-20; p < 1e-10; p *= 1.13)
      for (double m : {0.0, 1e-3 * std::sqrt(p * rho)}) {
        double u[D + 2] = {rho}, F[D][D + 1];
        u[1] = m;
        u[D + 1] = p / 0.4 + 0.5 * m * m / rho;
        const bool taken = point_flux<D>(u, 1.4, F);
        if (p < floor * (1 - 1e-9)) {
          CHECK(!taken, "D %d rho %g m %g: pressure %g below the floor taken", D, rho, m, p);
        } else if (p > floor * (1 + 1e-9)) {
          CHECK(taken, "D %d rho %g m %g: pressure %g above the floor refused", D, rho, m, p);
          CHECK(std::fabs(F[1][1] - p) < 1e-14 * p, "D %d rho %g: flux %g, pressure %g", D, rho, F[1][1], p);
        }
      }
}

// A column of zeros or subnormal numbers is zero, whatever its exponent and
// however its values are added up, and so is a zero in any column; a value is
// the double itself while its bits are above 2^-60 of the bound.
static void zero_columns() {
  for (double z : {0.0, -0.0, 4.9e-324, -2.2e-308}) {
    const double x[10] = {z, -z, z, z, z, z, -z, z, z, z};
    for (int E : {fx_norm_exp<10>(x, 1), 1, 60, 64, 1022, 2039}) {
      long long sum = 0;
      for (double y : x) {
        CHECK(fx_from_double(y, E) == 0, "%g in a column of exponent %d is %lld", y, E, fx_from_double(y, E));
        sum += fx_from_double(y, E);
      }
      const double back = fx_to_double(sum, E, 0);
      CHECK(back == 0.0 && !std::signbit(back), "the sum of a column of %g is %g", z, back);
      CHECK(fx_to_double(-1, 3, 0) == 0.0 && !std::signbit(fx_to_double(-1, 3, 0)), "-1 unit below the doubles");
    }
  }
  std::mt19937_64 rng(1);
  for (int i = 0; i < 1000000; ++i) {
    const int e = 8 + (int)(rng() % 2030);
    const double x = __longlong_as_double((long long)((rng() & 0x800fffffffffffffULL) | (unsigned long long)e << 52));
    for (int up = 0; up < 8 && e + up <= kFxMaxExp; ++up) {
      const double back = fx_to_double(fx_from_double(x, e + up), e + up, 0);
      CHECK(back == x, "%a in a column of exponent %d is %a", x, e + up, back);
    }
  }
}

// 113-bit arithmetic: the measure of both forms of the fluxes.
#ifdef __SIZEOF_FLOAT128__
typedef __float128 wide;
#else
typedef long double wide;
#endif
static wide wide_abs(wide x) { return x < 0 ? -x : x; }
static wide scaled(wide x, int e) {
  for (; e >= 60; e -= 60) x *= (wide)(1LL << 60);
  for (; e <= -60; e += 60) x /= (wide)(1LL << 60);
  return e >= 0 ? x * (wide)(1LL << e) : x / (wide)(1LL << -e);
}

static void legendre(int P, wide x, wide* v) {
  v[0] = 1;
  if (P > 0) v[1] = x;
  for (int n = 1; n < P; ++n) v[n + 1] = ((2 * n + 1) * x * v[n] - n * v[n - 1]) / (n + 1);
}
// Gauss points and weights, x and -x side by side.
static void gauss(int n, std::vector<double>& x, std::vector<double>& w) {
  auto deriv = [n](double z, double* p) {
    double a = 1.0, b = z;
    for (int k = 1; k < n; ++k) {
      const double c = ((2 * k + 1) * z * b - k * a) / (k + 1);
      a = b, b = c;
    }
    *p = b;
    return n * (z * b - a) / (z * z - 1.0);
  };
  for (int i = 1; i <= n / 2; ++i) {
    double z = std::cos(M_PI * (i - 0.25) / (n + 0.5)), p;
    for (int it = 0; it < 50; ++it) {
      const double d = deriv(z, &p);
      z -= p / d;
    }
    x.push_back(z), x.push_back(-z);
  }
  if (n % 2) x.push_back(0.0);
  for (double z : x) {
    double p;
    const double d = deriv(z, &p);
    w.push_back(2.0 / ((1.0 - z * z) * d * d));
  }
}

struct FluxErrors {  // along, across, energy; relative to the element's largest
  double fx[3] = {}, f64[3] = {};
  int taken = 0, elements = 0;
};

// Fluxes at the points of random elements: densities up to 60 apart, Mach
// numbers 0.08 to 12, pressures up to 100 apart, velocities smooth, constant
// or reversing, in fixed point and in the FP64 of euler_flux_all.
template <int D, int P>
static void flux_errors(int count, FluxErrors* out) {
  constexpr int Q = D + 2, N = P + 1, NP = D == 2 ? N * N : N * N * N;
  constexpr int NM = D == 2 ? N * (N + 1) / 2 : N * (N + 1) * (N + 2) / 6;
  std::mt19937_64 rng(100 * D + P);
  auto uniform = [&] { return 2.0 * ((double)(rng() >> 11) * 0x1p-53) - 1.0; };
  std::vector<double> x, w;
  gauss(N, x, w);
  wide L[N][N];
  for (int k = 0; k < N; ++k) legendre(P, x[k], L[k]);
  std::vector<std::array<int, 3>> modes;
  for (int a = 0; a <= P; ++a)
    for (int b = 0; a + b <= P; ++b)
      for (int c = 0; c <= (D == 3 ? P - a - b : 0); ++c) modes.push_back({a, b, c});
  const double gamma = 1.4, gm1 = gamma - 1.0;
  const FxFactor gm1x = fx_factor(gm1);
  for (int t = 0; t < count; ++t) {
    const double contrast = std::log(60.0) / 2 * std::fabs(uniform()), mach = std::exp(2.5 * uniform());
    const double speed = std::exp(3 * uniform()), scale = std::exp(2 * uniform());
    const double steep = 1 + 5 * std::fabs(uniform()), phase = uniform();
    const double pressures = rng() % 2 ? std::log(100.0) / 2 * std::fabs(uniform()) : 0.05;
    const int kind = (int)(rng() % 4);
    double dir[3], v0[3], norm = 0.0;
    for (int d = 0; d < 3; ++d) {
      dir[d] = d < D ? uniform() : 0.0;
      norm += std::fabs(dir[d]);
      v0[d] = uniform();
    }
    if (rng() % 4 == 0) v0[1] *= 0.01;
    double U[Q][NM] = {};
    for (int m = 0; m < NP; ++m) {
      const int k[3] = {m % N, m / N % N, m / N / N};
      double s = 0.0, ke = 0.0, u[Q];
      for (int d = 0; d < D; ++d) s += dir[d] / norm * x[k[d]];
      const double a = kind == 1 ? std::tanh(steep * (s + 0.3 * phase)) : s;
      u[0] = scale * std::exp(contrast * a);
      for (int d = 0; d < D; ++d) {
        double v = speed * (kind == 3 ? std::sin(3 * s + phase + d) : v0[d] + 0.2 * std::sin(2 * s + phase));
        if (kind == 2) v *= std::exp(-0.5 * contrast * a);
        u[d + 1] = u[0] * v;
        ke += 0.5 * u[0] * v * v;
      }
      u[D + 1] = scale * speed * speed / (mach * mach * 1.4) * std::exp(pressures * a) / gm1 + ke;
      for (int i = 0; i < NM; ++i) {
        double f = 1.0;
        for (int d = 0; d < D; ++d) f *= w[k[d]] * (double)L[k[d]][modes[i][d]] * (2 * modes[i][d] + 1) / 2;
        for (int q = 0; q < Q; ++q) U[q][i] += u[q] * f;
      }
    }
    int E[Q], n_max = 0;
    for (int q = 0; q < Q; ++q) E[q] = fx_norm_exp<NM>(U[q], 1);
    wide u[NP][Q];
    long long v[NP][Q];
    for (int m = 0; m < NP; ++m) {
      const int k[3] = {m % N, m / N % N, m / N / N};
      for (int q = 0; q < Q; ++q) {
        u[m][q] = 0;
        for (int i = 0; i < NM; ++i) {
          wide f = U[q][i];
          for (int d = 0; d < D; ++d) f *= L[k[d]][modes[i][d]];
          u[m][q] += f;
        }
        const wide f = scaled(u[m][q], 1082 - E[q]);
        v[m][q] = (long long)(f < 0 ? f - (wide)0.5 : f + (wide)0.5);
      }
      n_max = max(n_max, __clz((int)(v[m][0] >> 32)));
    }
    const FxFluxExp<D> X(E + 1, E[D + 1], E[0], n_max, gm1x.ef);
    long long F[NP][D][D + 1];
    bool taken = true;
    for (int m = 0; m < NP && taken; ++m) taken = fx_euler_flux<D>(v[m], X, E[D + 1], n_max, gm1x, F[m]);
    ++out->elements;
    if (!taken) continue;
    ++out->taken;
    for (int d = 0; d < D; ++d)
      for (int c = 0; c <= D; ++c) {
        wide largest = 0, efx = 0, e64 = 0;
        for (int m = 0; m < NP; ++m) {
          const wide r = 1 / u[m][0];
          wide ke = 0;
          for (int k = 0; k < D; ++k) ke += u[m][k + 1] * u[m][k + 1] * r;
          const wide p = (wide)gm1 * (u[m][D + 1] - ke / 2);
          const wide exact = c == D ? (u[m][D + 1] + p) * u[m][d + 1] * r : u[m][c + 1] * u[m][d + 1] * r + (c == d ? p : 0);
          double ud[Q], vd[D];
          for (int q = 0; q < Q; ++q) ud[q] = (double)u[m][q];
          const double rd = 1.0 / ud[0];
          for (int k = 0; k < D; ++k) vd[k] = ud[k + 1] * rd;
          double ked = ud[1] * vd[0];
          for (int k = 1; k < D; ++k) ked = std::fma(ud[k + 1], vd[k], ked);
          const double pd = gm1 * std::fma(-0.5, ked, ud[D + 1]);
          const double f64 = c == D ? (ud[D + 1] + pd) * vd[d] : c == d ? std::fma(ud[d + 1], vd[d], pd) : ud[c + 1] * vd[d];
          largest = max(largest, wide_abs(exact));
          e64 = max(e64, wide_abs(f64 - exact));
          efx = max(efx, wide_abs(scaled((wide)F[m][d][c], X.flux(d, c + 1, E + 1) - 1082) - exact));
        }
        const int cls = c == D ? 2 : c == d ? 0 : 1;
        out->fx[cls] = max(out->fx[cls], (double)(efx / largest));
        out->f64[cls] = max(out->f64[cls], (double)(e64 / largest));
      }
  }
}

// Where the integers evaluate an element's fluxes, their error is no larger
// than FP64's.
static void flux_accuracy() {
  FluxErrors e;
  flux_errors<2, 1>(1000, &e);
  flux_errors<2, 2>(2000, &e);
  flux_errors<2, 3>(4000, &e);
  flux_errors<2, 6>(1000, &e);
  flux_errors<3, 1>(1000, &e);
  flux_errors<3, 2>(2000, &e);
  flux_errors<3, 3>(500, &e);
  const char* name[3] = {"momentum along", "momentum across", "energy"};
  for (int i = 0; i < 3; ++i)
    CHECK(e.fx[i] <= e.f64[i], "%s: error %g, FP64 %g (%d of %d elements)", name[i], e.fx[i], e.f64[i], e.taken, e.elements);
  CHECK(3 * e.taken > e.elements, "only %d of %d elements in fixed point", e.taken, e.elements);
}

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  if (what == "pressure_floor") {
    pressure_floor<2>();
    pressure_floor<3>();
  } else if (what == "zero_columns") {
    zero_columns();
  } else if (what == "flux_accuracy") {
    flux_accuracy();
  } else {
    std::printf("unknown check %s\n", what.c_str());
    return 2;
  }
  std::printf("ok\n");
  return 0;
}
