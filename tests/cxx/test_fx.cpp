// Checks of the fixed-point columns (adg_fx.cuh) built for the host: one check
// per argument, "ok" or what failed on standard output.
#include "cuda_host.h"

#include <cstdio>
#include <cstdlib>
#include <random>
#include <string>

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

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  if (what == "pressure_floor") {
    pressure_floor<2>();
    pressure_floor<3>();
  } else {
    std::printf("unknown check %s\n", what.c_str());
    return 2;
  }
  std::printf("ok\n");
  return 0;
}
