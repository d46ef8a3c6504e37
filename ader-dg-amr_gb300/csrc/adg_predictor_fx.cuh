// Plain Picard predictor (AmrDG.tpp:495-537, 744-827) in fixed point
// (adg_fx.cuh); FP64 is left to the final stage's fluxes and the face physics.
//
// A block holds E elements, C = E Q columns, and gives every column
// N^(D-1) threads, one per line of points along x_0.  A sweep takes one time
// node at a time:
//   1  g(b) = sum_a P_a(t_k) h(b, a)                     (columns, over the modes b)
//   2  H on the thread's line of points                  (columns, lines)
//   3  fluxes F_d at the points                          (points)
//   4  each line of F_d projected along x_0, in place    (columns, lines)
//   5  the projections along the other dimensions, then  acc(b, a) += P_a(t_k) v(b)
// and after the last node H' = W U - sum_d (Dt/dx_d) C_d acc_d.  Points come
// in pairs x, -x, so a one-dimensional stage takes half the products.  The
// first sweep's initial guess does not depend on x_0 (AmrDG.tpp:520-533): its
// values on the (x_1 .., t) grid are those of U on the spatial grid, so it is
// one slice whose projections are spread over a_0 with the sums of P_a0.  The
// mass flux is the momentum, linear in H: its update K_d h comes from the
// modes, and phases 4 and 5 run over the columns of the other variables.
//
// Phase 3 evaluates the fluxes on the column values (fx_euler_flux); an
// element with a point whose density or pressure is out of that form's range
// (near vacuum, at the pressure floor, densities more than 2^2 apart, kinetic
// terms whose bound is more than 2^4 above the energy's) takes the FP64 fluxes
// for all of its points, and so do values that are not finite.
//
// Why this form: GB300 issues 1.6 FP64 operations per clock and SM.  The
// column-per-thread FP64 predictor kept that pipe 84 % busy; with the
// operators on the integer pipes it still set the time through the fluxes
// (D2P3, 256^2: 2330 -> 1169 us), and with integer fluxes in the sweeps the
// kernel issues 2.0 instructions per clock and SM (1169 -> 1010 us; a flux
// costs the integer pipes what its conversions cost before).  Now: dependent
// integer chains and the barriers between phases.  The stages are short loops
// over tables instead of unrolled code per (operator, time node):
// straight-line code starved on instruction fetch (57 k instructions per
// column, 16 % issue activity).
#pragma once

#include "adg_kernels.cuh"

namespace adg {

template <class O, int E>
struct FxShape {
  static constexpr int D = O::D, Q = O::Q, N = O::N, NP_S = O::NP_S, NP_ST = O::NP_ST, NS = O::NQ_S;
  static constexpr int C = E * Q;
  static constexpr int LD = C | 1;  // odd: the point phases read across columns
  static constexpr int LINES = NS / N;
  // threads per line: the columns, filled up to whole warps where that idles
  // few lanes (a warp then works on one line, its table reads are uniform)
  static constexpr int CP = C % 32 >= 28 ? (C + 31) / 32 * 32 : C;
  static constexpr int CF = E * (Q - 1);  // columns whose fluxes are projected in the sweeps
  static constexpr int NT = (CP * LINES + 31) / 32 * 32;
  static constexpr int ROWS = (NP_ST + LINES - 1) / LINES;            // rows of H_w per thread
  static constexpr int TASKS = (D * O::FX_NPRE + LINES - 1) / LINES;  // (direction, mode prefix) per thread
  static constexpr int PTS = (E * NS + NT - 1) / NT;                  // points per thread
  // warps per SM that the register limit allows: the phases wait at barriers,
  // so more blocks beat a few spills (the kernel at 16 / 24 / 32 warps: D2P3,
  // 256^2, 1163 / 1010 / 1068 us, 104 bytes spilled at 24; D3P2, 64^3, 13.3 /
  // 8.3 / 7.4 ms, 232 bytes at 32; D3P3, 20 x 14 x 18, 1007 / 691 / 652 us,
  // 392 bytes), except where a line is long (D2P4, 100^2, 625 / 691 / 822 us;
  // D2P6, 48^2, 851 / 1004 / 1022, 204 bytes at 16)
  static constexpr int WARPS = D == 3 ? 32 : N <= 4 ? 24 : 16;
  static constexpr int MIN_BLOCKS = WARPS * 32 / NT > 0 ? WARPS * 32 / NT : 1;
  // 64-bit slots: modes, U, g, fluxes, accumulators
  static constexpr int O_H = 0, O_U = O_H + NP_ST * LD, O_G = O_U + NP_S * LD, O_F = O_G + NP_S * LD,
                       O_A = O_F + D * NS * LD, SLOTS = O_A + D * NP_ST * LD;
  // 32-bit words after them, [i][column]: exponents of U, of H, NaN bits,
  // sum of H; in the mass columns the most leading zeros of the slice's
  // densities, and whether the element's fluxes are FP64; per direction the
  // exponent of the slice's fluxes, that of the largest so far, the
  // accumulators', what the slice raised it by, the largest change
  static constexpr int I_EU = 0, I_EH = C, I_NAN = 2 * C, I_SUM = 3 * C, I_N = 4 * C, I_F64 = 5 * C, I_X = 6 * C,
                       I_F = I_X + D * C, I_EA = I_F + D * C, I_UP = I_EA + D * C, I_Z = I_UP + D * C,
                       WORDS = I_Z + D * C;
  static constexpr size_t BYTES = (size_t)SLOTS * 8 + (size_t)WORDS * 4;
};

// Barrier of a block of NT threads.
template <int NT>
__device__ __forceinline__ void fx_sync() {
  if constexpr (NT == 32)
    __syncwarp();
  else
    __syncthreads();
}

// One-dimensional projection tables: P_a at the nodes, and the corrector's
// w P_a and w P_a'.
enum FxTab { FX_P, FX_W, FX_D };
template <class O, int TAB>
constexpr int fx_tab_shift() {
  return TAB == FX_P ? O::FX_SP : TAB == FX_W ? O::FX_SW : O::FX_SD;
}
template <class O, int TAB>
constexpr __host__ __device__ int fx_tab_h(int a, int k) {
  return TAB == FX_P ? O::fx_ph(a, k) : TAB == FX_W ? O::fx_wh(a, k) : O::fx_dh(a, k);
}
template <class O, int TAB>
constexpr __host__ __device__ int fx_tab_l(int a, int k) {
  return TAB == FX_P ? O::fx_pl(a, k) : TAB == FX_W ? O::fx_wl(a, k) : O::fx_dl(a, k);
}

// N line values (with one bit of room) as sums and differences of the pairs.
template <class O>
struct FxPairs {
  static constexpr int J = O::N / 2;
  long long s[J], d[J], mid;
  __device__ __forceinline__ explicit FxPairs(const long long* x) {
#pragma unroll
    for (int j = 0; j < J; ++j) {
      s[j] = x[2 * j] + x[2 * j + 1];
      d[j] = x[2 * j] - x[2 * j + 1];
    }
    mid = O::N % 2 ? x[O::N - 1] : 0;
  }
  // row a of the table (a compile-time constant after unrolling)
  template <int TAB>
  __device__ __forceinline__ long long row(int a) const {
    const bool odd = (a % 2 == 1) != (TAB == FX_D);
    if (TAB == FX_D && a == 0) return 0;
    if (TAB == FX_P && a == 0 && (O::N & (O::N - 1)) == 0) {  // the factor 2 / N is a shift
      long long t = J > 1 ? J / 2 : 0;
#pragma unroll
      for (int j = 0; j < J; ++j) t += s[j];
      return J == 1 ? t : J == 2 ? t >> 1 : t >> 2;
    }
    FxSum t;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const long long x = odd ? d[j] : s[j];
      t.mulc(fx_hi(x), fx_lo(x), fx_tab_h<O, TAB>(a, 2 * j), fx_tab_l<O, TAB>(a, 2 * j));
    }
    if (O::N % 2 && !odd) t.mulc(fx_hi(mid), fx_lo(mid), fx_tab_h<O, TAB>(a, O::N - 1), fx_tab_l<O, TAB>(a, O::N - 1));
    return t.get();
  }
};

// Modes along x_0 of a line: t(n0) = sum over the other modes of g with the
// line's values of their Legendre polynomials (c1, and c2 at D = 3; entry 0
// is one).  g at stride LD.
template <class O, int LD>
__device__ __forceinline__ void fx_line_modes(const long long* g, const FxCoef* c1, const FxCoef* c2, long long* t) {
  constexpr int P = O::P;
  int b = 0;
#pragma unroll
  for (int n0 = 0; n0 <= P; ++n0) {
    FxSum s;
#pragma unroll
    for (int n1 = 0; n1 <= P - n0; ++n1) {
      long long x;
      if constexpr (O::D == 2) {
        x = g[b++ * LD];
      } else {
        FxSum r;
        r.add(g[b++ * LD]);
#pragma unroll
        for (int n2 = 1; n2 <= P - n0 - n1; ++n2) r.mul(g[b++ * LD], c2[n2]);
        x = n0 + n1 < P ? r.get() : r.A;
      }
      if (n1 == 0) {
        s.add(x);
      } else {
        if (n1 == 5) s.fold();
        s.mul(x, c1[n1]);
      }
    }
    t[n0] = n0 < P ? s.get() : s.A;
  }
}

// Values at the N points of a line from its modes: out(k0, value).
template <class O, class Out>
__device__ __forceinline__ void fx_line_points(const long long* t, Out out) {
  constexpr int N = O::N, P = O::P;
  int h[N], l[N];
#pragma unroll
  for (int n = 1; n <= P; ++n) {
    h[n] = fx_hi(t[n]);
    l[n] = fx_lo(t[n]);
  }
#pragma unroll
  for (int j = 0; j < (N + 1) / 2; ++j) {
    FxSum ev, od;
    ev.add(t[0]);
#pragma unroll
    for (int n = 1; n <= P; ++n) (n % 2 ? od : ev).mulc(h[n], l[n], O::fx_vh(n, 2 * j), O::fx_vl(n, 2 * j));
    const long long a = P >= 2 ? ev.get() : ev.A;
    if (2 * j + 1 < N) {
      const long long b = od.get();
      out(2 * j, a + b);
      out(2 * j + 1, a - b);
    } else {
      out(2 * j, a);
    }
  }
}

// Values P_a(x_k) of a line's coordinate k as run-time coefficients.
template <class O>
__device__ __forceinline__ void fx_load_coefs(int k, FxCoef* c) {
#pragma unroll
  for (int a = 1; a < O::N; ++a) c[a] = O::fx_val(a, k);
}
template <class O>
__device__ __forceinline__ void fx_end_coefs(int side, FxCoef* c) {  // P_a(+-1)
#pragma unroll
  for (int a = 1; a < O::N; ++a) c[a] = {a % 2 && !side ? -(1 << kFxLimb) : 1 << kFxLimb, 0};
}

// The block: what every phase needs, and the thread's column and line, over
// all columns or over those of the sweeps' flux projections.
template <class O, int E>
struct FxBlock {
  using S = FxShape<O, E>;
  long long* m;  // shared slots
  int* w;        // shared words
  int line, col;
  bool act;      // the thread has a column
  __device__ __forceinline__ double* f() const { return reinterpret_cast<double*>(m + S::O_F); }
  __device__ __forceinline__ int& word(int base, int i = 0) const { return w[base + i * S::C + col]; }
};

constexpr int kFxNoExp = -30000;  // below every exponent

// The exponent of the largest magnitude on the thread's line of direction
// dir's fluxes into the column's: doubles, or column values of exponent x.
template <class O, int E>
__device__ __forceinline__ void fx_line_max(const FxBlock<O, E>& k, int dir, bool f64, int x) {
  using S = FxShape<O, E>;
  const int* f = reinterpret_cast<const int*>(k.f() + (dir * S::NS + k.line) * S::LD + k.col) + 1;
  int e = 0, bits = 0;
#pragma unroll
  for (int i = 0; i < O::N; ++i) {
    const int h = f[i * S::LINES * S::LD * 2];
    e = max(e, h & 0x7fffffff);
    bits |= h ^ (h >> 31);
  }
  atomicMax(&k.word(S::I_F, dir), f64 ? e >> 20 : x + 4 - __clz(bits));
}
// The exponent the column's fluxes are read at: one bit of room.
template <class O, int E>
__device__ __forceinline__ int fx_line_exp(const FxBlock<O, E>& k, int dir) {
  return k.word(FxShape<O, E>::I_F, dir) + 1;
}
// The line projected along x_0, in the place of its values.
template <class O, int E, int TAB>
__device__ __forceinline__ void fx_line_project(const FxBlock<O, E>& k, int dir, int e, bool f64, int x) {
  using S = FxShape<O, E>;
  constexpr int N = O::N;
  long long* t = k.m + S::O_F + (dir * S::NS + k.line) * S::LD + k.col;
  long long v[N];
  if (f64) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = fx_from_double(__longlong_as_double(t[i * S::LINES * S::LD]), e);
  } else {
    if (x >= e) {
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] = t[i * S::LINES * S::LD] << (x - e);
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] = fx_align(t[i * S::LINES * S::LD], e - x);
    }
  }
  const FxPairs<O> p(v);
#pragma unroll
  for (int a = 0; a < N; ++a) t[a * S::LINES * S::LD] = p.template row<TAB>(a);
}

// D = 3: projection along x_1 of the values (n0, k1, k2), in place, for the
// thread's (n0, k2).  Every further dimension halves its operands, one bit of
// room for the pairs.
template <class O, int E, int TAB>
__device__ __forceinline__ void fx_project_planes(const FxBlock<O, E>& k, int dir) {
  using S = FxShape<O, E>;
  constexpr int N = O::N, P = O::P;
  const int n0 = k.line / N, k2 = k.line % N;
  long long* t = k.m + S::O_F + (dir * S::NS + n0 * S::LINES + k2) * S::LD + k.col;
  long long v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = fx_half(t[i * N * S::LD]);
  const FxPairs<O> p(v);
#pragma unroll
  for (int a = 0; a < N; ++a)
    if (a <= P - n0) t[a * N * S::LD] = p.template row<TAB>(a);
}

// Operands of the last projection of (direction, prefix slot).
template <class O, int E>
__device__ __forceinline__ FxPairs<O> fx_last(const FxBlock<O, E>& k, int dir, int slot) {
  using S = FxShape<O, E>;
  const long long* t = k.m + S::O_F + (dir * S::NS + slot * O::N) * S::LD + k.col;
  long long v[O::N];
#pragma unroll
  for (int i = 0; i < O::N; ++i) v[i] = fx_half(t[i * S::LD]);
  return FxPairs<O>(v);
}

// (direction, prefix) of task j of the thread; false when there is none.
// Odd directions run through the prefixes backwards, so that a thread's
// tasks are of both sizes.
template <class O, int E>
__device__ __forceinline__ bool fx_task(int line, int j, int* dir, int* pre) {
  const int i = line + j * FxShape<O, E>::LINES;
  *dir = i / O::FX_NPRE;
  *pre = i % O::FX_NPRE;
  if (*dir & 1) *pre = O::FX_NPRE - 1 - *pre;
  return i < O::D * O::FX_NPRE;
}

// Phase 5: the last projection of the thread's tasks, v(b), and its products
// with the slice's P_a(t) / N added to the accumulators (FIRST: the sums of
// P_a0 / N, stored).
template <class O, int E, bool FIRST>
__device__ __forceinline__ void fx_accumulate(const FxBlock<O, E>& kf, int kt) {
  using S = FxShape<O, E>;
  constexpr int D = O::D, N = O::N, P = O::P, LD = S::LD;
  FxCoef ct[N];
#pragma unroll
  for (int a = 0; a < N; ++a) ct[a] = FIRST ? O::fx_ssum(a) : O::fx_valt(a, kt);
#pragma unroll 1
  for (int j = 0; j < S::TASKS; ++j) {
    int d, pre;
    if (!fx_task<O, E>(kf.line, j, &d, &pre)) continue;
    const FxPairs<O> p = fx_last<O, E>(kf, d, O::fx_pre_slot(pre));
    const int deg = O::fx_pre_deg(pre), b0 = O::fx_pre_base(pre);
    long long* acc = kf.m + S::O_A + d * O::NP_ST * LD + kf.col;
    long long* q = acc + O::fx_first(b0) * LD;
    if (!FIRST) {  // larger fluxes than in the slices before: what is there moves down
      const int up = kf.word(S::I_UP, d);
      if (up > 0) {
        const int cnt = (P - deg + 1) * (P - deg + 2) / 2;
#pragma unroll 1
        for (int i = 0; i < cnt; ++i) q[i * LD] = fx_align(q[i * LD], up);
      }
    }
#pragma unroll
    for (int n = 0; n < N; ++n) {
      if (n > P - deg) break;
      const long long v = p.template row<FX_P>(n);
      const int h = fx_hi(v), l = fx_lo(v);
#pragma unroll
      for (int a = 0; a < N - n; ++a) {
        if (a > P - deg - n) break;
        FxSum s;
        if (FIRST) {
          s.mul(h, l, ct[a].h, ct[a].l);
          acc[O::fx_init(b0 + n, a) * LD] = s.get();
        } else {
          s.add(q[a * LD]);
          s.mul(h, l, ct[a].h, ct[a].l);
          q[a * LD] = s.get();
        }
      }
      q += (P - deg - n + 1) * LD;  // the next mode's
    }
  }
}

// Phase 3: the fluxes of the slice's points in the place of their values;
// MASS: the momenta as the mass fluxes too.  An element with a point that is
// not for the integers (or with exponents near the range of doubles) has all
// of its points in FP64.  of_u: values of U, else of H.
template <class O, int E, bool MASS>
__device__ __forceinline__ void fx_point_fluxes(const FxBlock<O, E>& k, bool of_u, double gm1, const FxFactor& gm1x) {
  using S = FxShape<O, E>;
  constexpr int D = O::D, Q = O::Q, LD = S::LD;
  const int* wx = k.w + (of_u ? S::I_EU : S::I_EH);
  long long u[S::PTS][Q];
  bool bad = false;
#pragma unroll
  for (int r = 0; r < S::PTS; ++r) {
    const int it = threadIdx.x + r * S::NT;
    if (it < E * S::NS) {
      const int c0 = (it / S::NS) * Q, m = it % S::NS;
      long long* base = k.m + S::O_F + m * LD + c0;
#pragma unroll
      for (int v = 0; v < Q; ++v) u[r][v] = base[v];
      int em[D], range = max(abs(wx[c0] - 1022), abs(wx[c0 + D + 1] - 1022));
#pragma unroll
      for (int d = 0; d < D; ++d) {
        em[d] = wx[c0 + d + 1];
        range = max(range, em[d] - 1022);
      }
      const int n = k.w[S::I_N + c0];
      const FxFluxExp<D> x(em, wx[c0 + D + 1], wx[c0], n, gm1x.ef);
      long long F[D][D + 1];
      if (range < 480 && fx_euler_flux<D>(u[r], x, wx[c0 + D + 1], n, gm1x, F)) {
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
          for (int v = MASS ? 0 : 1; v < Q; ++v) base[d * S::NS * LD + v] = v ? F[d][v > 0 ? v - 1 : 0] : u[r][d + 1];
      } else {
        k.w[S::I_F64 + c0] = 1;
        bad = true;
      }
      if (m == 0) {
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
          for (int v = MASS ? 0 : 1; v < Q; ++v) k.w[S::I_X + d * S::C + c0 + v] = v ? x.flux(d, v, em) : em[d];
      }
    }
  }
  if (__syncthreads_or(bad)) {
#pragma unroll
    for (int r = 0; r < S::PTS; ++r) {
      const int it = threadIdx.x + r * S::NT;
      if (it < E * S::NS && k.w[S::I_F64 + (it / S::NS) * Q]) {
        const int c0 = (it / S::NS) * Q;
        double* base = k.f() + (it % S::NS) * LD + c0;
        double ud[Q], F[D * Q];
#pragma unroll
        for (int v = 0; v < Q; ++v)
          ud[v] = fx_to_double(u[r][v], wx[c0 + v], of_u ? fx_poison(wx[c0 + v]) : k.w[S::I_NAN + c0 + v]);
        euler_flux_all<D, double>(ud, gm1, F);
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
          for (int v = MASS ? 0 : 1; v < Q; ++v) base[d * S::NS * LD + v] = F[d * Q + v];
      }
    }
    fx_sync<S::NT>();
  }
}

// Phases 2 to 5 of one slice: H from the spatial modes g, fluxes, projections,
// accumulation.  kt < 0: the first sweep's slice (g = U).  k: all columns, kf:
// those projected.
template <class O, int E>
__device__ __forceinline__ void fx_sweep_slice(const FxBlock<O, E>& k, const FxBlock<O, E>& kf, const long long* g,
                                               const FxCoef* c1, const FxCoef* c2, int kt, double gm1,
                                               const FxFactor& gm1x) {
  using S = FxShape<O, E>;
  constexpr int D = O::D, Q = O::Q, N = O::N, P = O::P, LD = S::LD;
  if (k.act) {
    long long t[N];
    fx_line_modes<O, LD>(g + k.col, c1, c2, t);
    long long* h = k.m + S::O_F + k.line * LD + k.col;
    int n = 0;
    fx_line_points<O>(t, [&](int k0, long long v) {
      h[k0 * S::LINES * LD] = v;
      n = max(n, __clz((int)(v >> 32)));
    });
    if (k.col % Q == 0) atomicMax(&k.word(S::I_N), n);
  }
  fx_sync<S::NT>();
  fx_point_fluxes<O, E, false>(k, kt < 0, gm1, gm1x);
  const bool f64 = kf.act && k.w[S::I_F64 + kf.col / Q * Q];
  if (kf.act) {
#pragma unroll 1
    for (int d = 0; d < D; ++d) fx_line_max<O, E>(kf, d, f64, kf.word(S::I_X, d));
  }
  fx_sync<S::NT>();
  if (kf.act) {
#pragma unroll 1
    for (int d = 0; d < D; ++d) {
      const int e = fx_line_exp<O, E>(kf, d);
      if (kf.line == 0) {
        kf.word(S::I_UP, d) = kt > 0 ? e - kf.word(S::I_EA, d) : 0;
        kf.word(S::I_EA, d) = e;
      }
      fx_line_project<O, E, FX_P>(kf, d, e, f64, kf.word(S::I_X, d));
    }
  }
  fx_sync<S::NT>();
  if (k.act && k.line == 0 && k.col % Q == 0) k.word(S::I_N) = k.word(S::I_F64) = 0;
  if constexpr (D == 3) {
    if (kf.act) {
#pragma unroll 1
      for (int d = 0; d < D; ++d) fx_project_planes<O, E, FX_P>(kf, d);
    }
    fx_sync<S::NT>();
  }
  if (!kf.act) return;
  if (kt < 0)
    fx_accumulate<O, E, true>(kf, kt);
  else
    fx_accumulate<O, E, false>(kf, kt);
}

// z_d = Dt/dx_d C_d acc_d of the thread's rows; of the mass column K_d times
// the momentum's modes (first: of the first sweep's initial guess, whose only
// modes are U's).  One loop over the sparse rows of either.
template <class O, int E>
__device__ __forceinline__ void fx_changes(const FxBlock<O, E>& k, const FxFactor* cf, bool first,
                                           long long (&z)[FxShape<O, E>::ROWS][O::D]) {
  using S = FxShape<O, E>;
  constexpr int D = O::D;
  const bool mass = k.col % O::Q == 0;
  const int nv = mass && first ? O::NP_S : O::NP_ST;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const long long* v = k.m + k.col + (mass ? (first ? S::O_U : S::O_H) + d + 1 : S::O_A + d * O::NP_ST * S::LD);
    const int table = mass ? D + d : d;
    int bits = 0;
#pragma unroll
    for (int r = 0; r < S::ROWS; ++r) {
      const int n = k.line + r * S::LINES;
      z[r][d] = 0;
      if (n < O::NP_ST) {
        const int j1 = O::fx_row(table, n + 1);
        int j = O::fx_row(table, n), i = 0;
        if (j == j1) continue;
        FxSum s;
#pragma unroll 1
        for (; j < j1; ++j) {
          const int c = O::fx_col(j);
          if (c >= nv) break;
          s.mul(v[c * S::LD], O::fx_cval(j));
          if (O::NP_ST > 20 && (++i & 3) == 0) s.fold();
        }
        z[r][d] = fx_scale(s.get(), cf[d]);
        const int hi = (int)(z[r][d] >> 32);
        bits |= hi ^ (hi >> 31);
      }
    }
    atomicOr(&k.word(S::I_Z, d), bits);
  }
}

// H_w' = W U - sum_d z_d: the terms aligned to the largest of U's exponent
// and the changes' actual ones, then the column rescaled to its sum of
// magnitudes.
template <class O, int E>
__device__ __forceinline__ void fx_update(const FxBlock<O, E>& k, const FxFactor* cf, bool first) {
  using S = FxShape<O, E>;
  constexpr int D = O::D;
  long long z[S::ROWS][D];
  int ez[D], nan_bits = 0, top = 0;
  if (k.act) {
    fx_changes<O, E>(k, cf, first, z);
    const bool mass = k.col % O::Q == 0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      if (mass) {
        const int* w = k.w + k.col + d + 1;  // the momentum's column
        const int e = first ? w[S::I_EU] : w[S::I_EH];
        ez[d] = fx_scaled_exp(e, O::fx_sk(d), cf[d]);
        nan_bits |= first ? 0 : w[S::I_NAN];
      } else {
        ez[d] = fx_scaled_exp(k.word(S::I_EA, d), D - 1 + O::fx_sc(d), cf[d]);
      }
      nan_bits |= fx_poison(ez[d]);
    }
  }
  fx_sync<S::NT>();
  if (k.act) {
    const int eu = k.word(S::I_EU);
    top = eu;
    nan_bits |= fx_poison(eu);
#pragma unroll
    for (int d = 0; d < D; ++d) top = max(top, ez[d] + 4 - __clz(k.word(S::I_Z, d)));  // |z| < 2^(64 - clz)
    int sum = 0;
#pragma unroll
    for (int r = 0; r < S::ROWS; ++r) {
      const int n = k.line + r * S::LINES;
      if (n < O::NP_ST) {
        long long h = 0;
        if (O::fx_time(n) == 0) h = fx_align(k.m[S::O_U + O::fx_spatial(n) * S::LD + k.col], top - eu);
#pragma unroll
        for (int d = 0; d < D; ++d) h -= fx_move(z[r][d], top - ez[d]);
        z[r][0] = h;
        sum += (abs((int)(h >> 32)) >> 6) + 1;  // |h| < 2^38 of these
      }
    }
    atomicAdd(&k.word(S::I_SUM), sum);
  }
  fx_sync<S::NT>();
  if (k.act) {
    const int up = __clz(k.word(S::I_SUM)) - 10;  // sum |h| < 2^(70 - clz), to be below 2^60
#pragma unroll
    for (int r = 0; r < S::ROWS; ++r) {
      const int n = k.line + r * S::LINES;
      if (n < O::NP_ST) {
        k.m[S::O_H + n * S::LD + k.col] = fx_move(z[r][0], -up);
#pragma unroll
        for (int d = 0; d < D; ++d) k.m[S::O_A + (d * O::NP_ST + n) * S::LD + k.col] = 0;
      }
    }
    if (k.line == 0) {
      k.word(S::I_EH) = top - up;
      k.word(S::I_NAN) = nan_bits | fx_poison(top - up);
#pragma unroll
      for (int d = 0; d < D; ++d) {
        k.word(S::I_Z, d) = 0;
        k.word(S::I_F, d) = kFxNoExp;
      }
    }
  }
  fx_sync<S::NT>();
}

// The modes b whose g the thread computes: first(b) and degree.
template <class O, int E>
struct FxModes {
  static constexpr int NB = (O::NP_S + FxShape<O, E>::LINES - 1) / FxShape<O, E>::LINES;
  int first[NB], deg[NB];
  __device__ __forceinline__ explicit FxModes(const FxBlock<O, E>& k) {
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int b = k.line + i * FxShape<O, E>::LINES;
      first[i] = b < O::NP_S ? O::fx_first(b) : 0;
      deg[i] = b < O::NP_S ? O::fx_deg(b) : 0;
    }
  }
};
// g(b) = sum_a P_a(t_k) h(b, a) of time node kt.
template <class O, int E>
__device__ __forceinline__ void fx_time_slice(const FxBlock<O, E>& k, const FxModes<O, E>& md, int kt) {
  using S = FxShape<O, E>;
  constexpr int P = O::P;
  if (k.act) {
    FxCoef c[O::N];
    fx_load_coefs<O>(kt, c);
#pragma unroll
    for (int i = 0; i < FxModes<O, E>::NB; ++i) {
      const int b = k.line + i * S::LINES;
      if (b >= O::NP_S) break;
      const long long* h = k.m + S::O_H + md.first[i] * S::LD + k.col;
      FxSum s;
      s.add(h[0]);
#pragma unroll
      for (int a = 1; a <= P; ++a) {
        if (a > P - md.deg[i]) break;
        if (a == 5) s.fold();
        s.mul(h[a * S::LD], c[a]);
      }
      k.m[S::O_G + b * S::LD + k.col] = s.get();
    }
  }
  fx_sync<S::NT>();
}

// Face values of a slice: the two faces of x_0 from the line's modes, the
// others from lines that run along them (D = 2: the two sides of x_1; D = 3:
// side and x_2, x_1 and side): out(face 2d + side, point, value).
template <class O, int E, class Out>
__device__ __forceinline__ void fx_face_values(const FxBlock<O, E>& k, const long long* t, Out out) {
  long long lo = t[0], hi = t[0];
#pragma unroll
  for (int n = 1; n <= O::P; ++n) {
    hi += t[n];
    lo += n % 2 ? -t[n] : t[n];
  }
  out(0, k.line, lo);
  out(1, k.line, hi);
}

template <class O, int E, class Out>
__device__ __forceinline__ void fx_side_lines(const FxBlock<O, E>& k, const long long* g, Out out) {
  using S = FxShape<O, E>;
  constexpr int D = O::D, N = O::N, SIDES = D == 2 ? 2 : 4 * N;
#pragma unroll 1
  for (int i = k.line; i < SIDES; i += S::LINES) {
    FxCoef c1[N], c2[N];
    int face, x;  // point offset
    if constexpr (D == 2) {
      fx_end_coefs<O>(i, c1);
      face = 2 + i;
      x = 0;
    } else {
      const int side = (i / N) & 1, j = i % N;
      if (i < 2 * N) {
        fx_end_coefs<O>(side, c1);
        fx_load_coefs<O>(j, c2);
      } else {
        fx_load_coefs<O>(j, c1);
        fx_end_coefs<O>(side, c2);
      }
      face = (i < 2 * N ? 2 : 4) + side;
      x = j;
    }
    long long t[N];
    fx_line_modes<O, S::LD>(g + k.col, c1, c2, t);
    fx_line_points<O>(t, [&](int k0, long long v) { out(face, x + k0 * (D == 2 ? 1 : N), v); });
  }
}

// Corrector volume term of direction DIR from the time-integrated fluxes
// (AmrDG.tpp:696-709): projections with w P' along DIR and w P along the
// others; the modes' values as doubles into the accumulators' place.
template <class O, int E, int DIR>
__device__ __forceinline__ void fx_volume_last(const FxBlock<O, E>& k, int pre) {
  using S = FxShape<O, E>;
  constexpr int D = O::D, TAB = DIR == D - 1 ? FX_D : FX_W;
  const FxPairs<O> p = fx_last<O, E>(k, DIR, O::fx_pre_slot(pre));
  const int deg = O::fx_pre_deg(pre), ef = fx_line_exp<O, E>(k, DIR);
  const int e = ef + (D - 1) + O::FX_SD + (D - 1) * O::FX_SW, nan_bits = fx_poison(ef);
  double* out = reinterpret_cast<double*>(k.m + S::O_A) + (DIR * O::NP_S + O::fx_pre_base(pre)) * S::LD + k.col;
#pragma unroll
  for (int n = 0; n < O::N; ++n)
    if (n <= O::P - deg) out[n * S::LD] = fx_to_double(p.template row<TAB>(n), e, nan_bits);
}

// FX: the fluxes are those of fx_point_fluxes, else doubles.
template <class O, int E, bool FX>
__device__ __forceinline__ void fx_volume_term(const FxBlock<O, E>& k) {
  using S = FxShape<O, E>;
  constexpr int D = O::D;
  const bool f64 = !FX || (k.act && k.w[S::I_F64 + k.col / O::Q * O::Q]);
  auto exp = [&](int d) { return FX ? k.word(S::I_X, d) : 0; };
  if (k.act) {
#pragma unroll 1
    for (int d = 0; d < D; ++d) fx_line_max<O, E>(k, d, f64, exp(d));
  }
  fx_sync<S::NT>();
  if (k.act) {
    fx_line_project<O, E, FX_D>(k, 0, fx_line_exp<O, E>(k, 0), f64, exp(0));
#pragma unroll 1
    for (int d = 1; d < D; ++d) fx_line_project<O, E, FX_W>(k, d, fx_line_exp<O, E>(k, d), f64, exp(d));
  }
  fx_sync<S::NT>();
  if constexpr (D == 3) {
    if (k.act) {
      fx_project_planes<O, E, FX_W>(k, 0);
      fx_project_planes<O, E, FX_D>(k, 1);
      fx_project_planes<O, E, FX_W>(k, 2);
    }
    fx_sync<S::NT>();
  }
  if (k.act) {
#pragma unroll 1
    for (int j = 0; j < S::TASKS; ++j) {
      int d, pre;
      if (!fx_task<O, E>(k.line, j, &d, &pre)) continue;
      if (d == 0) fx_volume_last<O, E, 0>(k, pre);
      if (d == 1) fx_volume_last<O, E, 1>(k, pre);
      if constexpr (D == 3)
        if (d == 2) fx_volume_last<O, E, 2>(k, pre);
    }
  }
  fx_sync<S::NT>();
}

// U of the block's elements: coalesced loads, the column's exponent, fixed
// point; the words' initial values.
template <class O, int E, class Elem>
__device__ __forceinline__ void fx_load_state(const FxBlock<O, E>& k, const PredictorArgs& a, Elem element, bool live) {
  using S = FxShape<O, E>;
  constexpr int D = O::D, Q = O::Q, NP_S = O::NP_S, LD = S::LD, C = S::C, NT = S::NT;
  const int el = k.col / Q, q = k.col % Q;
  double* ud = reinterpret_cast<double*>(k.m + S::O_G);
  for (int i = threadIdx.x; i < C * NP_S; i += NT)
    ud[(i % NP_S) * LD + i / NP_S] = a.Uw[(size_t)element(i / (Q * NP_S)) * Q * NP_S + i % (Q * NP_S)];
  fx_sync<S::NT>();
  if (k.act && k.line == 0) {
    const int eu = fx_norm_exp<NP_S>(ud + k.col, LD);
    k.word(S::I_EU) = eu;
    k.word(S::I_SUM) = k.word(S::I_N) = k.word(S::I_F64) = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      k.word(S::I_Z, d) = 0;
      k.word(S::I_F, d) = kFxNoExp;
    }
    if (a.ubar_old && live) a.ubar_old[(size_t)element(el) * Q + q] = ud[k.col];
  }
  fx_sync<S::NT>();
  if (k.act)
    for (int b = k.line; b < NP_S; b += S::LINES)
      k.m[S::O_U + b * LD + k.col] = fx_from_double(ud[b * LD + k.col], k.word(S::I_EU));
  fx_sync<S::NT>();
}

// One group of E elements (positions chunk E .. of the range or list).
template <class O, int E>
__device__ __forceinline__ void fx_predictor_chunk(const PredictorArgs& a, char* smem, int chunk, int limit) {
  using S = FxShape<O, E>;
  constexpr int D = O::D, Q = O::Q, N = O::N, NP_S = O::NP_S, NP_ST = O::NP_ST, NS = S::NS, LD = S::LD, C = S::C;
  constexpr int NB = O::NQ_BD, NSB = NB / N, NF = 2 * D, TT = tr_tile<O>(), NT = S::NT;
  FxBlock<O, E> k;
  k.m = reinterpret_cast<long long*>(smem);
  k.w = reinterpret_cast<int*>(k.m + S::SLOTS);
  k.line = threadIdx.x / S::CP;
  k.act = k.line < S::LINES && (int)threadIdx.x % S::CP < C;
  k.col = k.act ? threadIdx.x % S::CP : 0;
  FxBlock<O, E> kf = k;  // the columns of the sweeps' flux projections: all but the mass
  kf.line = threadIdx.x / S::CF;
  kf.col = (threadIdx.x % S::CF) / (Q - 1) * Q + 1 + (threadIdx.x % S::CF) % (Q - 1);
  kf.act = kf.line < S::LINES;
  const int e0 = chunk * E;
  auto element = [&](int el) {  // past the end: the last one (its results are not written)
    const int i = e0 + el < limit ? e0 + el : limit - 1;
    return a.elem_list ? a.elem_list[i] : i;
  };
  const int el = k.col / Q, q = k.col % Q;
  const bool live = e0 + el < limit;
  const int e = element(el);
  const int lev = a.elem_level ? a.elem_level[e] : 0;
  double c[D];
  FxFactor cf[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    c[d] = a.dt[kScalDtDx + 3 * lev + d];
    cf[d] = fx_factor(c[d]);
  }
  const double gm1 = a.gamma - 1.0;
  const FxFactor gm1x = fx_factor(gm1);
  const FxModes<O, E> md(k);
  FxCoef c1[N], c2[N];
  fx_load_coefs<O>(D == 2 ? k.line % N : (k.line / N) % N, c1);
  if constexpr (D == 3) fx_load_coefs<O>(k.line % N, c2);

  fx_load_state<O, E>(k, a, element, live);

  // the first sweep on U, then the others (AmrDG.h:1103-1119)
  {
    fx_sweep_slice<O, E>(k, kf, k.m + S::O_U, c1, c2, -1, gm1, gm1x);
    fx_sync<S::NT>();
    fx_update<O, E>(k, cf, true);
  }
#pragma unroll 1
  for (int s = 1; s < a.sweeps; ++s) {
    if (k.act && k.line == 0) k.word(S::I_SUM) = 0;
#pragma unroll 1
    for (int kt = 0; kt < N; ++kt) {
      fx_time_slice<O, E>(k, md, kt);
      fx_sweep_slice<O, E>(k, kf, k.m + S::O_G, c1, c2, kt, gm1, gm1x);
    }
    fx_sync<S::NT>();
    fx_update<O, E>(k, cf, false);
  }
  const int eh = k.act ? k.word(S::I_EH) : 0, nan_bits = k.act ? k.word(S::I_NAN) : 0;
  if (a.Hw_out && k.act && live) {
    double* dst = a.Hw_out + ((size_t)e * Q + q) * NP_ST;
    for (int n = k.line; n < NP_ST; n += S::LINES) {
      bool same = true;
      for (int t = 0; t < D; ++t) same = same && O::fx_row(t, n) == O::fx_row(t, n + 1);
      dst[n] = fx_to_double(k.m[S::O_H + n * LD + k.col], eh, nan_bits);
      // a mode that no sweep changes is U's own
      if (same) dst[n] = O::fx_time(n) == 0 ? a.Uw[((size_t)e * Q + q) * NP_S + O::fx_spatial(n)] : 0.0;
    }
  }

  // final stage: per time node the face values and the volume fluxes, these
  // integrated over time by the threads of the points
  double fbar[S::PTS][D * Q];
#pragma unroll
  for (int r = 0; r < S::PTS; ++r)
#pragma unroll
    for (int v = 0; v < D * Q; ++v) fbar[r][v] = 0.0;
#pragma unroll 1
  for (int kt = 0; kt < N; ++kt) {
    fx_time_slice<O, E>(k, md, kt);
    if (k.act) {
      const long long* g = k.m + S::O_G;
      long long t[N];
      fx_line_modes<O, LD>(g + k.col, c1, c2, t);
      double* h = k.f() + k.line * LD + k.col;
      fx_line_points<O>(t, [&](int k0, long long v) { h[k0 * S::LINES * LD] = fx_to_double(v, eh, nan_bits); });
      if (live) {
        double* tr = a.Tr + (size_t)e * NF * TT + q * NB + kt * NSB;
        auto out = [&](int face, int x, long long v) { tr[face * TT + x] = fx_to_double(v, eh, nan_bits); };
        fx_face_values<O, E>(k, t, out);
        fx_side_lines<O, E>(k, g, out);
      }
    }
    fx_sync<S::NT>();
    const double w = O::weight(kt);
#pragma unroll
    for (int r = 0; r < S::PTS; ++r) {
      const int it = threadIdx.x + r * NT;
      if (it < E * NS) {
        const double* base = k.f() + (it % NS) * LD + (it / NS) * Q;
        double u[Q], F[D * Q];
#pragma unroll
        for (int v = 0; v < Q; ++v) u[v] = base[v];
        euler_flux_all<D, double>(u, gm1, F);
#pragma unroll
        for (int v = 0; v < D * Q; ++v) fbar[r][v] = fma(w, F[v], fbar[r][v]);
      }
    }
  }
  fx_sync<S::NT>();
#pragma unroll
  for (int r = 0; r < S::PTS; ++r) {
    const int it = threadIdx.x + r * NT;
    if (it < E * NS) {
      double* base = k.f() + (it % NS) * LD + (it / NS) * Q;
#pragma unroll
      for (int d = 0; d < D; ++d)
#pragma unroll
        for (int v = 0; v < Q; ++v) base[d * NS * LD + v] = fbar[r][d * Q + v];
    }
  }
  fx_sync<S::NT>();
  fx_volume_term<O, E, false>(k);
  // Rvol = M U + sum_d (Dt/dx_d) Sk_d F_d, coalesced
  const double* vt = reinterpret_cast<const double*>(k.m + S::O_A);
  for (int i = threadIdx.x; i < C * NP_S; i += NT) {
    const int b = i % NP_S, cc = i / NP_S;
    if (e0 + cc / Q >= limit) continue;
    const size_t o = (size_t)element(cc / Q) * Q * NP_S + i % (Q * NP_S);
    const int lv = a.elem_level ? a.elem_level[element(cc / Q)] : 0;
    double r = O::mdiag(b) * a.Uw[o];
#pragma unroll
    for (int d = 0; d < D; ++d) r = fma(a.dt[kScalDtDx + 3 * lv + d], vt[(d * NP_S + b) * LD + cc], r);
    a.Rvol[o] = r;
  }
  // face physics (AmrDG.h:1207-1251) on the values in the trace tiles
  for (int it = threadIdx.x; it < E * NF * NB; it += NT) {
    const int p = it % NB, face = (it / NB) % NF, ee = it / (NB * NF);
    if (e0 + ee >= limit) break;
    double* t = a.Tr + ((size_t)element(ee) * NF + face) * TT + p;
    double uu[Q], F[Q];
#pragma unroll
    for (int v = 0; v < Q; ++v) uu[v] = t[v * NB];
    const double df = euler_flux_normal<D>(face >> 1, uu, a.gamma, F);
#pragma unroll
    for (int v = 0; v < Q; ++v) t[(Q + v) * NB] = F[v];
    t[2 * Q * NB] = df;
  }
}

template <class O, int E>
__global__ void __launch_bounds__((FxShape<O, E>::NT), (FxShape<O, E>::MIN_BLOCKS)) k_predictor_fx(PredictorArgs a) {
  extern __shared__ __align__(16) char fx_smem[];
  fx_predictor_chunk<O, E>(a, fx_smem, blockIdx.x, a.n_elem);
}

// The time-independent part of a seeded step's final stage (split_epilogue of
// adg_kernels.cuh): the volume term of F(U) to Rvol, and U and its normal
// flux at the faces' spatial points to the split trace tiles.  In the FP64 of
// the seeded kernel this was 1850 of its 2050 FP64 operations an element and
// kept that pipe 65 % busy; one slice of the plain predictor's stages does it
// on the integer pipes.  D2P3, 15,600 elements: 27 us (blocks of 16 elements
// 30), the seeded kernel 45 us, where it was 90 us with both.
template <class O, int E>
struct FxBase {
  using S = FxShape<O, E>;
  static constexpr int NSB = O::NQ_BD / O::N, NF = 2 * O::D;
  // the face values lie in the accumulators' place and behind it
  static constexpr int SLOTS = S::O_A + NF * NSB * S::LD > S::SLOTS ? S::O_A + NF * NSB * S::LD : S::SLOTS;
  static constexpr size_t BYTES = (size_t)SLOTS * 8 + (size_t)S::WORDS * 4;
};

template <class O, int E>
__global__ void __launch_bounds__((FxShape<O, E>::NT), (FxShape<O, E>::MIN_BLOCKS)) k_split_base(PredictorArgs a) {
  using S = FxShape<O, E>;
  constexpr int D = O::D, Q = O::Q, N = O::N, NP_S = O::NP_S, LD = S::LD, C = S::C, NT = S::NT;
  constexpr int NSB = FxBase<O, E>::NSB, NF = 2 * D, TT = tr_tile<O>();
  extern __shared__ __align__(16) char fx_smem[];
  FxBlock<O, E> k;
  k.m = reinterpret_cast<long long*>(fx_smem);
  k.w = reinterpret_cast<int*>(k.m + FxBase<O, E>::SLOTS);
  k.line = threadIdx.x / S::CP;
  k.act = k.line < S::LINES && (int)threadIdx.x % S::CP < C;
  k.col = k.act ? threadIdx.x % S::CP : 0;
  const int e0 = blockIdx.x * E, limit = a.n_elem;
  auto element = [&](int el) {  // past the end: the last one (its results are not written)
    const int i = e0 + el < limit ? e0 + el : limit - 1;
    return a.elem_list ? a.elem_list[i] : i;
  };
  const double gm1 = a.gamma - 1.0;
  const FxFactor gm1x = fx_factor(gm1);
  FxCoef c1[N], c2[N];
  fx_load_coefs<O>(D == 2 ? k.line % N : (k.line / N) % N, c1);
  if constexpr (D == 3) fx_load_coefs<O>(k.line % N, c2);
  fx_load_state<O, E>(k, a, element, e0 + k.col / Q < limit);
  // U at the points and the faces' points
  const long long* g = k.m + S::O_U;
  long long* faces = k.m + S::O_A;
  if (k.act) {
    long long t[N];
    fx_line_modes<O, LD>(g + k.col, c1, c2, t);
    long long* h = k.m + S::O_F + k.line * LD + k.col;
    int n = 0;
    fx_line_points<O>(t, [&](int k0, long long v) {
      h[k0 * S::LINES * LD] = v;
      n = max(n, __clz((int)(v >> 32)));
    });
    auto out = [&](int face, int x, long long v) {
      faces[(face * NSB + x) * LD + k.col] = v;
      n = max(n, __clz((int)(v >> 32)));
    };
    fx_face_values<O, E>(k, t, out);
    fx_side_lines<O, E>(k, g, out);
    if (k.col % Q == 0) atomicMax(&k.word(S::I_N), n);
  }
  fx_sync<NT>();
  fx_point_fluxes<O, E, true>(k, true, gm1, gm1x);
  // the faces' spatial points: U and the normal flux
  const int* wx = k.w + S::I_EU;
#pragma unroll 1
  for (int it = threadIdx.x; it < E * NF * NSB; it += NT) {
    const int p = it % (NF * NSB), c0 = it / (NF * NSB) * Q, dir = p / (2 * NSB);
    if (e0 + c0 / Q >= limit) break;
    double* tile = a.Tr + ((size_t)element(c0 / Q) * NF + p / NSB) * TT + p % NSB;
    long long u[Q];
#pragma unroll
    for (int v = 0; v < Q; ++v) {
      u[v] = faces[p * LD + c0 + v];
      tile[v * NSB] = fx_to_double(u[v], wx[c0 + v], fx_poison(wx[c0 + v]));
    }
    int em[D], range = max(abs(wx[c0] - 1022), abs(wx[c0 + D + 1] - 1022));
#pragma unroll
    for (int d = 0; d < D; ++d) {
      em[d] = wx[c0 + d + 1];
      range = max(range, em[d] - 1022);
    }
    const int n = k.w[S::I_N + c0];
    const FxFluxExp<D> x(em, wx[c0 + D + 1], wx[c0], n, gm1x.ef);
    long long F[D][D + 1];
    double* f = tile + Q * NSB;
    if (range < 480 && fx_euler_flux<D>(u, x, wx[c0 + D + 1], n, gm1x, F)) {
#pragma unroll
      for (int v = 0; v < Q; ++v) {
        long long y = 0;
        int e = 0;
#pragma unroll
        for (int d = 0; d < D; ++d)
          if (d == dir) {
            y = v ? F[d][v > 0 ? v - 1 : 0] : u[d + 1];
            e = v ? x.flux(d, v, em) : em[d];
          }
        f[v * NSB] = fx_to_double(y, e, 0);
      }
    } else {
      double uu[Q], F64[Q];
#pragma unroll
      for (int v = 0; v < Q; ++v) uu[v] = fx_to_double(u[v], wx[c0 + v], fx_poison(wx[c0 + v]));
      (void)euler_flux_normal<D>(dir, uu, a.gamma, F64);
#pragma unroll
      for (int v = 0; v < Q; ++v) f[v * NSB] = F64[v];
    }
  }
  fx_sync<NT>();
  fx_volume_term<O, E, true>(k);
  // Rvol = M U + sum_d (Dt/dx_d) (sum_k w_k) Sk_d F_d(U), coalesced
  double* cw = reinterpret_cast<double*>(k.m + S::O_H);  // [element][d]
  for (int i = threadIdx.x; i < E * D; i += NT) {
    const int lev = a.elem_level ? a.elem_level[element(i / D)] : 0;
    cw[i] = a.dt[kScalDtDx + 3 * lev + i % D] * O::WEIGHT_SUM;
  }
  fx_sync<NT>();
  const double* vt = reinterpret_cast<const double*>(k.m + S::O_A);
  for (int i = threadIdx.x; i < C * NP_S; i += NT) {
    const int b = i % NP_S, cc = i / NP_S;
    if (e0 + cc / Q >= limit) continue;
    const size_t o = (size_t)element(cc / Q) * Q * NP_S + i % (Q * NP_S);
    double r = O::mdiag(b) * a.Uw[o];
#pragma unroll
    for (int d = 0; d < D; ++d) r = fma(cw[cc / Q * D + d], vt[(d * NP_S + b) * LD + cc], r);
    a.Rvol[o] = r;
  }
}

// The fallback pass: a short grid striding over a list counted on the device.
template <class O, int E>
__global__ void __launch_bounds__((FxShape<O, E>::NT)) k_predictor_fx_list(PredictorArgs a) {
  extern __shared__ __align__(16) char fx_smem[];
  const int limit = *a.list_count;
  if (a.count_total && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(a.count_total, (unsigned long long)limit);
#pragma unroll 1
  for (int chunk = blockIdx.x; chunk * E < limit; chunk += gridDim.x) {
    fx_predictor_chunk<O, E>(a, fx_smem, chunk, limit);
    fx_sync<FxShape<O, E>::NT>();
  }
}

}  // namespace adg
