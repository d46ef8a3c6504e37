// L2 projections between levels (L2ProjInterp, AmrDG_Interpolater.tpp:283-398):
// amr_scatter, one coarse element -> one of its children, and amr_gather, the
// 2^D children -> their coarse element, for the ghost fill, the regrid remap,
// the average down and a caller's batches.
//
// Per dimension the projections between a Legendre basis and that of the half
// intervals have exact dyadic coefficients,
//   P_n((x + s) / 2) = sum_j c_nj s^(n+j) P_j(x),        s = +-1,
// so both are chains of one-dimensional lines over the modes.
//
// k_gather.  Dense, a column is 4 x 40 FP64 operations at D2P3 and the batch
// was bound by the FP64 pipe (1.6 operations per clock and SM) and by column
// loads 80 bytes apart.  Here a block stages its children with asynchronous
// contiguous copies, the lines pair two children (sum and difference: half
// the products) and run in place in fixed point (adg_fx.cuh) with one-word
// coefficients: bound by integer issue for large batches, by latency below
// some 10,000 cells.
//   D2P3, 60001 cells 85 -> 38 us (the bytes alone: 14), 500 cells 8.1 -> 3.2;
//   D3P2, 30000 cells 85 -> 43 us; an average down of 2048 cells within a step
//   8.0 -> 5.2 us.
// Columns with infinities or NaN keep the dense FP64 operators, whose zeros
// decide which modes are affected, and so do columns near the ends of the
// range of doubles (xf_dense).
//
// k_scatter.  Dense, the four children's operators differ, so a warp with a
// batch's mixed children ran all of them, one after another on the FP64 pipe.
// The lines differ by a sign only: no divergence, 36 FP64 operations a column
// (29 dense, times the children met).
//   D2P3, 60001 cells 55 -> 17 us, 500 cells 6.5 -> 3.1; D3P2, 30000 cells
//   43 -> 11 us; a ghost fill of a few hundred elements 4.2 -> 3.9 us.
// In fixed point and staged as the gather it takes 14 us for the 60001 cells,
// but 5.6 within a step, where the few ghosts only meet its latency (three
// barriers and twice the code, fetched cold).
#pragma once

#include "adg_async.cuh"
#include "adg_kernels.cuh"

namespace adg {

// Work split of the gather: a thread takes a group of the lines of one column
// and pair of children, a warp's threads the same group, so a warp runs the
// code of its group only: a step's average downs meet cold instruction caches,
// where fetching the straight-line code of all lines took longer than running
// it (9.9 us, with 16 elements a block; 11.8 with run-time line lengths).
template <class O>
struct TransferShape {
  static constexpr int D = O::D, Q = O::Q, N = O::N, NP = O::NP_S, NOV = 1 << D, QN = Q * NP;
  static constexpr int LINES = D == 2 ? N : N * (N + 1) / 2;  // of a column
  static constexpr int GROUPS = D == 2 || N < 3 ? (N + 1) / 2 : 2;
  // coarse elements per block: about a warp of (column, pair) a group
  static constexpr int GATHER = D == 2 ? 4 : 3;
  static constexpr int threads(int n) { return (n + 31) / 32 * 32; }
  static constexpr int TG_G = threads(GATHER * Q * NOV / 2);  // of a group
  static constexpr int NT_G = GROUPS * TG_G, NT_S = 128;
  // k-th line of group g, long lines (small numbers) with short ones
  static constexpr int line(int g, int k) { return k % 2 ? (k + 1) * GROUPS - 1 - g : k * GROUPS + g; }
  static constexpr int PER_GROUP = (LINES + GROUPS - 1) / GROUPS;
};

// Lines along dimension d are numbered by the degrees (a, b) in the other
// dimensions (b = 0 in 2D), in the order of a + b.
template <class O, int d, int I>
struct XfLine {
  static constexpr int N = O::N;
  static constexpr int degree() {
    int t = 0;
    while (O::D == 3 && (t + 1) * (t + 2) / 2 <= I) ++t;
    return O::D == 2 ? I : t;
  }
  static constexpr int b = O::D == 2 ? 0 : I - degree() * (degree() + 1) / 2, a = degree() - b;
  static constexpr int LEN = N - degree();
  static constexpr int mode(int j) {
    if (O::D == 2) return O::fx_mode(d == 0 ? j * N + a : a * N + j);
    return O::fx_mode(d == 0 ? (j * N + a) * N + b : d == 1 ? (a * N + j) * N + b : (a * N + b) * N + j);
  }
};

// f(line) for the lines of group g (a run-time index) along d.
template <class O, int d, int G = 0, int K = 0, class F>
__device__ __forceinline__ void xf_each_line(int g, F&& f) {
  using S = TransferShape<O>;
  if constexpr (G < S::GROUPS) {
    if constexpr (K == 0) {
      if (g != G) return xf_each_line<O, d, G + 1>(g, f);
    }
    if constexpr (K < S::PER_GROUP) {
      if constexpr (S::line(G, K) < S::LINES) f(XfLine<O, d, S::line(G, K)>{});
      xf_each_line<O, d, G, K + 1>(g, f);
    }
  }
}

// One-word coefficients: no middle product of their low limb.
struct FxDyadic {
  long long A = 0, B = kFxHalf;
  __device__ __forceinline__ void mul(int h, int l, int c) {
    A = (long long)h * c + A;
    B = (long long)l * c + B;  // up to seven terms of 2^60
  }
  __device__ __forceinline__ long long get() const { return A + (B >> kFxLimb); }
};

// Columns that keep the FP64 operators: largest exponent field not in
// [128, 2030] (0: a column of zeros, whose result is zero).
__device__ __forceinline__ bool xf_dense(int e) { return e > 2030 || (e > 0 && e < 128); }

// Largest exponent field of the modes of group g in `parts` columns at stride
// ld (1 if all are subnormal, 0 if all are zero).
template <class O>
__device__ __forceinline__ int xf_exponent(int g, const double* x, int parts, int ld) {
  int e = 0, any = 0;
  xf_each_line<O, 0>(g, [&](auto line) {
#pragma unroll
    for (int j = 0; j < line.LEN; ++j)
      for (int c = 0; c < parts; ++c) {
        const double v = x[c * ld + line.mode(j)];
        e = max(e, __double2hiint(v) & 0x7fffffff);
        any |= __double2loint(v);
      }
  });
  return e >> 20 ? e >> 20 : (e | any) != 0;
}

// Operands of stage d: doubles, then (in the same words) column values.
template <int d>
__device__ __forceinline__ long long xf_value(double x, int e) {
  return d == 0 ? fx_from_double(x, e) : __double_as_longlong(x);
}

// Stage d of the gather: group g of the lines along x_d of children lo and hi,
// into lo.  A stage makes the column's exponent O::FX_XG_GROW larger.
template <class O, int d>
__device__ __forceinline__ void xf_gather_lines(int g, double* lo, const double* hi, int e) {
  xf_each_line<O, d>(g, [&](auto line) {
    constexpr int LEN = line.LEN;
    int sh[LEN], sl[LEN], dh[LEN], dl[LEN];
#pragma unroll
    for (int j = 0; j < LEN; ++j) {
      const long long x = xf_value<d>(lo[line.mode(j)], e), y = xf_value<d>(hi[line.mode(j)], e);
      const long long s = fx_half(y + x), t = fx_half(y - x);
      sh[j] = fx_hi(s);
      sl[j] = fx_lo(s);
      dh[j] = fx_hi(t);
      dl[j] = fx_lo(t);
    }
#pragma unroll
    for (int n = 0; n < LEN; ++n) {
      FxDyadic x;
#pragma unroll
      for (int j = 0; j <= n; ++j) {
        if (O::fx_xg(n, j) == 0) continue;
        (n + j) % 2 ? x.mul(dh[j], dl[j], O::fx_xg(n, j)) : x.mul(sh[j], sl[j], O::fx_xg(n, j));
      }
      lo[line.mode(n)] = __longlong_as_double(x.get());
    }
  });
}

template <class O>
__device__ __forceinline__ void pfc_rt(int l, const double* in, double* out) {
  switch (l) {
    case 0: O::template pfc<0>(RegIn{in}, RegOut{out}); break;
    case 1: O::template pfc<1>(RegIn{in}, RegOut{out}); break;
    case 2: O::template pfc<2>(RegIn{in}, RegOut{out}); break;
    case 3: O::template pfc<3>(RegIn{in}, RegOut{out}); break;
    default:
      if constexpr (O::D == 3) {
        switch (l) {
          case 4: O::template pfc<4>(RegIn{in}, RegOut{out}); break;
          case 5: O::template pfc<5>(RegIn{in}, RegOut{out}); break;
          case 6: O::template pfc<6>(RegIn{in}, RegOut{out}); break;
          default: O::template pfc<7>(RegIn{in}, RegOut{out}); break;
        }
      }
  }
}

// u_c = 2^-D Minv sum_l P_fc[l] u_f[l].  rec: coarse, fine_0 .. of every record
// in `fine` and `coarse` (the same array for the average down); nullptr: cell
// i of a batch.
template <class O>
__global__ void __launch_bounds__(TransferShape<O>::NT_G) k_gather(const double* fine, double* coarse, const int* rec,
                                                                 long long n) {
  using S = TransferShape<O>;
  constexpr int Q = S::Q, NP = S::NP, NOV = S::NOV, QN = S::QN, LD = (NOV * QN) | 1, NT = S::NT_G;
  constexpr int COLS = S::GATHER * Q;
  __shared__ double st[S::GATHER * LD];
  __shared__ int ex[S::GROUPS * NOV / 2][COLS];
  __shared__ int elem[S::GATHER * (NOV + 1)];
  const long long i0 = (long long)blockIdx.x * S::GATHER;
  const int items = (int)(n - i0 < S::GATHER ? n - i0 : S::GATHER);
  // the records first: a copy's address must not wait for memory
  if (rec) {
    for (int i = threadIdx.x; i < items * (NOV + 1); i += NT) elem[i] = rec[i0 * (NOV + 1) + i];
    __syncthreads();
  }
#pragma unroll 4
  for (int i = threadIdx.x; i < items * NOV * QN; i += NT) {
    const int it = i / (NOV * QN), w = i % (NOV * QN);
    const size_t src = rec ? (size_t)elem[it * (NOV + 1) + 1 + w / QN] * QN + w % QN : (size_t)i0 * (NOV * QN) + i;
    tc::cp_async8(st + it * LD + w, fine + src);
  }
  tc::cp_async_wait_all();
  __syncthreads();
  const int g = threadIdx.x / S::TG_G, l = threadIdx.x % S::TG_G / COLS;
  const int c = threadIdx.x % S::TG_G % COLS, it = c / Q, q = c % Q;
  double* u = st + it * LD + (l * Q + q) * NP;  // child l, later a sum of children
  auto column_exp = [&](int col) {
    int e = 0;
#pragma unroll
    for (int k = 0; k < S::GROUPS * NOV / 2; ++k) e = max(e, ex[k][col]);
    return e;
  };
  bool live = l < NOV / 2 && it < items;
  if (live) ex[g * NOV / 2 + l][c] = xf_exponent<O>(g, u, 2, NOV / 2 * QN);
  __syncthreads();
  const int e = live ? column_exp(c) : 0;
  if (live && xf_dense(e)) {
    live = false;
    if (g == 0 && l == 0) {
      double sum[NP], part[NP];
      for (int k = 0; k < NP; ++k) sum[k] = 0.0;
      for (int m = 0; m < NOV; ++m) {
        pfc_rt<O>(m, u + m * QN, part);
        for (int k = 0; k < NP; ++k) sum[k] += part[k];
      }
      for (int k = 0; k < NP; ++k) u[k] = (1.0 / NOV) * (O::minv(k) * sum[k]);
    }
  }
  if (live) xf_gather_lines<O, 0>(g, u, u + NOV / 2 * QN, e);
  __syncthreads();
  if (live && l < NOV / 4) xf_gather_lines<O, 1>(g, u, u + NOV / 4 * QN, e);
  __syncthreads();
  if constexpr (O::D == 3) {
    if (live && l == 0) xf_gather_lines<O, 2>(g, u, u + QN, e);
    __syncthreads();
  }
#pragma unroll 4
  for (int i = threadIdx.x; i < items * QN; i += NT) {
    const int r = i / QN, w = i % QN, ec = column_exp(r * Q + w / NP);
    const double v = st[r * LD + w];
    coarse[rec ? (size_t)elem[r * (NOV + 1)] * QN + w : (size_t)i0 * QN + i] =
        xf_dense(ec) ? v : ec ? fx_to_double(__double_as_longlong(v), ec + O::FX_XG_GROW * O::D, 0) : 0.0;
  }
}

// Stage d of the scatter, lines I and on along x_d; flip: the sign bit for the
// lower half, which changes the sign of every second product, else 0.
template <class O, int d, int I = 0>
__device__ __forceinline__ void xf_scatter_lines(double* v, int flip) {
  if constexpr (I < TransferShape<O>::LINES) {
    using L = XfLine<O, d, I>;
#pragma unroll
    for (int j = 0; j < L::LEN; ++j) {
      double x = O::xs(j, j) * v[L::mode(j)];
#pragma unroll
      for (int n = j + 1; n < L::LEN; ++n) {
        const double u = v[L::mode(n)];
        if (O::xs(n, j) == 0.0) continue;
        x = O::xs(n, j) * ((n + j) % 2 ? __hiloint2double(__double2hiint(u) ^ flip, __double2loint(u)) : u) + x;
      }
      v[L::mode(j)] = x;
    }
    xf_scatter_lines<O, d, I + 1>(v, flip);
  }
}

// Coarse -> fine projection (amr_scatter) into ghost elements, of the regrid
// remap (with src_old: valid data of the old layout where it existed), or of
// a batch (dst and parent nullptr: item i; a child out of range gives NaN).
struct ScatterArgs {
  double* fine;           // destination array
  const double* coarse;   // source array
  const double* old;      // optional: old layout's state
  const int* dst;         // [n] destination element
  const int* parent;      // [n] coarse parent element
  const int8_t* child;    // [n] child index
  const int* src_old;     // optional [n]: element in old, -1 = project
  long long n;
};

// A thread a column, loaded and stored directly: the latency of one round of
// index loads and one of a column's loads.
template <class O>
__global__ void __launch_bounds__(TransferShape<O>::NT_S) k_scatter(ScatterArgs a) {
  constexpr int D = O::D, Q = O::Q, NP = O::NP_S;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, i = t / Q;
  if (i >= a.n) return;
  const int q = (int)(t % Q), kid = a.child[i];
  double* out = a.fine + ((size_t)(a.dst ? a.dst[i] : i) * Q + q) * NP;
  const double* in = a.coarse + ((size_t)(a.parent ? a.parent[i] : i) * Q + q) * NP;
  const int old = a.src_old ? a.src_old[i] : -1;
  if (old >= 0) in = a.old + ((size_t)old * Q + q) * NP;
  double v[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) v[k] = in[k];
  if (old < 0) {
    auto half = [&](int d) { return (kid >> (D - 1 - d)) & 1 ? 0 : (int)0x80000000; };
    xf_scatter_lines<O, 0>(v, half(0));
    xf_scatter_lines<O, 1>(v, half(1));
    if constexpr (D == 3) xf_scatter_lines<O, 2>(v, half(2));
    if ((unsigned)kid >= 1u << D) {
#pragma unroll
      for (int k = 0; k < NP; ++k) v[k] = __longlong_as_double(0x7ff8000000000000LL);
    }
  }
#pragma unroll
  for (int k = 0; k < NP; ++k) out[k] = v[k];
}

}  // namespace adg
