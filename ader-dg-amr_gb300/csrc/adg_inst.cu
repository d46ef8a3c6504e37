// One (D, P) instantiation of the kernel set.  The build compiles this file
// once per configuration with -DADG_D, -DADG_HDR (generated operator header),
// -DADG_NS (its namespace) and -DADG_FACTORY (factory function name).
#include <atomic>
#include "adg_kernelset.hpp"
#include "adg_predictor_fx.cuh"
#include ADG_HDR

namespace adg {
namespace {

using O = ADG_NS::Ops;

// Dynamic shared memory of k_predictor per phase (ld = E Q + 1 slots per point):
//   FP64 sweeps             D NQ_ST ld doubles
//   FP32 sweeps (MODE 2)    D NQ_S ld floats     (one time slice at a time)
//   final volume slices     (1 + D) NQ_S ld doubles
//   face traces             2 NQ_BD ld doubles   (one direction at a time)
//   MODE 2, 3 final stage   split_epilogue_doubles (volume and face phases)
//   seed residual           2 E Q doubles
template <int E, int MODE>
constexpr size_t smem_bytes() {
  constexpr size_t ld = E * O::Q + 1;
  constexpr bool split = MODE == 2 || MODE == 3;
  constexpr size_t sweeps = MODE == 2 ? O::D * O::NQ_S * ld * sizeof(float) : O::D * O::NQ_ST * ld * sizeof(double);
  constexpr size_t fin = split ? split_epilogue_doubles<O>(ld, MODE == 3 || !base_apart<O>()) * sizeof(double)
                               : (1 + O::D) * O::NQ_S * ld * sizeof(double);
  constexpr size_t faces = split ? 0 : 2 * O::NQ_BD * ld * sizeof(double);
  constexpr size_t red = 2 * E * O::Q * sizeof(double);
  constexpr size_t m1 = sweeps > fin ? sweeps : fin;
  constexpr size_t m2 = faces > red ? faces : red;
  return m1 > m2 ? m1 : m2;
}

// The dynamic shared-memory limit of a kernel is an attribute of the current
// device's context: it is set once per device (bit d of mask; devices past 63
// set it on every launch), so a process that moves between GPUs sets it on
// each of them.
template <class F>
cudaError_t ensure_smem_attr(std::atomic<unsigned long long>& mask, F* func, size_t bytes) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = (dev >= 0 && dev < 64) ? (1ull << dev) : 0ull;
  if (bit && (mask.load(std::memory_order_acquire) & bit)) return cudaSuccess;
  e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess && bit) mask.fetch_or(bit, std::memory_order_acq_rel);
  return e;
}

// Grid of a fallback pass over a list of at most n elements counted on the
// device: two blocks per SM stride over it.
int list_grid(int n, int E) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
    sms = 152;
  const int grid = (n + E - 1) / E;
  return grid < 2 * sms ? grid : 2 * sms;
}

// Mode 0: the plain Picard path.
template <int E>
cudaError_t launch_plain(const PredictorArgs& a, cudaStream_t s) {
  constexpr size_t smem = FxShape<O, E>::BYTES;
  if (a.n_elem <= 0) return cudaSuccess;
  if (a.elem_list && a.list_count) {
    static std::atomic<unsigned long long> attr{0};
    cudaError_t e = ensure_smem_attr(attr, k_predictor_fx_list<O, E>, smem);
    if (e != cudaSuccess) return e;
    k_predictor_fx_list<O, E><<<list_grid(a.n_elem, E), FxShape<O, E>::NT, smem, s>>>(a);
  } else {
    static std::atomic<unsigned long long> attr{0};
    cudaError_t e = ensure_smem_attr(attr, k_predictor_fx<O, E>, smem);
    if (e != cudaSuccess) return e;
    k_predictor_fx<O, E><<<(a.n_elem + E - 1) / E, FxShape<O, E>::NT, smem, s>>>(a);
  }
  return cudaGetLastError();
}

// The time-independent part of mode 2's final stage.
template <int E>
cudaError_t launch_split_base(const PredictorArgs& a, cudaStream_t s) {
  constexpr size_t smem = FxBase<O, E>::BYTES;
  static std::atomic<unsigned long long> attr{0};
  if (a.n_elem <= 0) return cudaSuccess;
  cudaError_t e = ensure_smem_attr(attr, k_split_base<O, E>, smem);
  if (e != cudaSuccess) return e;
  k_split_base<O, E><<<(a.n_elem + E - 1) / E, FxShape<O, E>::NT, smem, s>>>(a);
  return cudaGetLastError();
}

// Modes 1 and 2 over the element range, mode 3 over a list counted on the
// device.
template <int E, int MODE>
cudaError_t launch_predictor_mode(const PredictorArgs& a, cudaStream_t s) {
  constexpr size_t smem = smem_bytes<E, MODE>();
  static std::atomic<unsigned long long> attr{0};
  if (a.n_elem <= 0) return cudaSuccess;
  if constexpr (MODE == 3) {
    if (!a.elem_list || !a.list_count) return cudaErrorInvalidValue;
    cudaError_t e = ensure_smem_attr(attr, k_predictor_list<O, E, MODE>, smem);
    if (e != cudaSuccess) return e;
    k_predictor_list<O, E, MODE><<<list_grid(a.n_elem, E), E * O::Q, smem, s>>>(a);
  } else {
    if (a.elem_list && a.list_count) return cudaErrorInvalidValue;
    cudaError_t e = ensure_smem_attr(attr, k_predictor<O, E, MODE>, smem);
    if (e != cudaSuccess) return e;
    k_predictor<O, E, MODE><<<(a.n_elem + E - 1) / E, E * O::Q, smem, s>>>(a);
  }
  return cudaGetLastError();
}

// The learned-seed path (predictor modes 1-3, the fused TF32 inference) is
// built for the elements whose network layers fit the fused kernel
// (seed_tc_fits: D = 2 with P <= 3, D = 3 with P <= 2).  Higher degrees run
// the plain FP64 path only, with one elements-per-block choice, which keeps
// their (large, generated) translation units quick to compile.
constexpr bool kSeedModes = seed_tc_fits(O::Q, O::NP_S, O::NP_ST);

template <int E>
cudaError_t launch_predictor(const PredictorArgs& a, cudaStream_t s, int mode) {
  if constexpr (kSeedModes) {
    if (mode == 1) return launch_predictor_mode<E, 1>(a, s);
    if (mode == 2) return launch_predictor_mode<E, 2>(a, s);
    if (mode == 3) return launch_predictor_mode<E, 3>(a, s);
  } else {
    if (mode != 0) return cudaErrorNotSupported;
  }
  return launch_plain<E>(a, s);
}

// Elements per block of the plain-only configurations: whole warps of columns
// at D = 2 (a block of 16 at P = 6 needs 214 KB of shared memory), at D = 3
// what leaves two blocks on an SM (P = 3, 20 x 14 x 18: 4 / 6 elements 641 /
// 656 us).
constexpr int lite_elems() { return O::D == 2 ? 8 : 4; }

struct Impl final : KernelSet {
  Impl() {
    D = O::D;
    P = O::P;
    Q = O::Q;
    Np_s = O::NP_S;
    Np_st = O::NP_ST;
    NQ_ST = O::NQ_ST;
    NQ_BD = O::NQ_BD;
    NQ_S = O::NQ_S;
    NM = O::NM;
    TR_TILE = tr_tile<O>();
    linear_fp64_per_column = O::LINEAR_FP64_PER_COLUMN;
  }
  bool seed_modes() const override { return kSeedModes; }
#if ADG_LITE
  std::vector<int> elems_per_block_choices() const override { return {lite_elems()}; }
  size_t predictor_smem(int) const override { return FxShape<O, lite_elems()>::BYTES; }
  cudaError_t predictor(const PredictorArgs& a, int, cudaStream_t s, int mode) const override {
    return launch_predictor<lite_elems()>(a, s, mode);
  }
#elif ADG_D == 2
  std::vector<int> elems_per_block_choices() const override { return {8, 16, 32}; }
  size_t predictor_smem(int E) const override {
    return E == 8 ? FxShape<O, 8>::BYTES : E == 16 ? FxShape<O, 16>::BYTES : FxShape<O, 32>::BYTES;
  }
  cudaError_t predictor(const PredictorArgs& a, int E, cudaStream_t s, int mode) const override {
    if (E == 8) return launch_predictor<8>(a, s, mode);
    if (E == 16) return launch_predictor<16>(a, s, mode);
    return launch_predictor<32>(a, s, mode);
  }
#else
  // (the plain path takes 6 elements for the choice 8: 30 columns fill a warp
  // and its table reads are uniform; the kernel with 8 / 6: P = 2, 64^3 7.54 /
  // 7.42 ms, 20^3 284 / 262 us; P = 1, 32^3 168 / 176 us)
  std::vector<int> elems_per_block_choices() const override { return {4, 8, 16}; }
  size_t predictor_smem(int E) const override {
    return E == 4 ? FxShape<O, 4>::BYTES : E == 8 ? FxShape<O, 6>::BYTES : FxShape<O, 16>::BYTES;
  }
  cudaError_t predictor(const PredictorArgs& a, int E, cudaStream_t s, int mode) const override {
    if (mode == 0 && E == 8) return launch_plain<6>(a, s);
    if (E == 4) return launch_predictor<4>(a, s, mode);
    if (E == 8) return launch_predictor<8>(a, s, mode);
    return launch_predictor<16>(a, s, mode);
  }
#endif
  cudaError_t split_base(const PredictorArgs& a, cudaStream_t s) const override {
    if constexpr (kSeedModes && base_apart<O>()) return launch_split_base<O::D == 2 ? 8 : 6>(a, s);
    return cudaErrorNotSupported;
  }
  bool split_base_apart() const override { return kSeedModes && base_apart<O>(); }
  cudaError_t numflux(const FaceArgs& a, long long nface, cudaStream_t s, bool split) const override {
    if (nface <= 0) return cudaSuccess;
    constexpr int FB = numflux_faces_per_block<O>();
    const unsigned grid = (unsigned)((nface + FB - 1) / FB);
    if (split)
      k_numflux_split<O><<<grid, FB * O::NQ_BD, 0, s>>>(a);
    else
      k_numflux<O><<<grid, FB * O::NQ_BD, 0, s>>>(a);
    return cudaGetLastError();
  }
  cudaError_t corrector(const CorrectorArgs& a, cudaStream_t s) const override {
    const long long n = ((long long)(a.elem_list ? a.n_list : a.n_valid) + (a.rec_of_elem ? a.nrec : 0)) * O::Q;
    // one-warp blocks: at its ~130 registers an SM holds 15 of them, so the
    // columns of ~16k elements run in one wave instead of 1.2
    const int bs = 32;
    k_corrector<O><<<(unsigned)((n + bs - 1) / bs), bs, 0, s>>>(a);
    return cudaGetLastError();
  }
  cudaError_t dt_reduce(const DtArgs& a, cudaStream_t s) const override {
    k_dt_reduce<O><<<(a.n_valid + kDtElems - 1) / kDtElems, 128, 0, s>>>(a);
    return cudaGetLastError();
  }
  cudaError_t average_down(double* Uw, const int* rec, int nrec, cudaStream_t s) const override {
    return gather(Uw, Uw, rec, nrec, s);
  }
  cudaError_t scatter(const ScatterArgs& a, cudaStream_t s) const override {
    if (a.n <= 0) return cudaSuccess;
    constexpr int NT = TransferShape<O>::NT_S;
    k_scatter<O><<<(unsigned)((a.n * O::Q + NT - 1) / NT), NT, 0, s>>>(a);
    return cudaGetLastError();
  }
  cudaError_t interp_scatter(const double* coarse, const int8_t* child, long long n, double* fine,
                             cudaStream_t s) const override {
    ScatterArgs a{};
    a.fine = fine;
    a.coarse = coarse;
    a.child = child;
    a.n = n;
    return scatter(a, s);
  }
  cudaError_t interp_gather(const double* fine, long long n, double* coarse, cudaStream_t s) const override {
    return gather(fine, coarse, nullptr, n, s);
  }
  static cudaError_t gather(const double* fine, double* coarse, const int* rec, long long n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    constexpr int B = TransferShape<O>::GATHER;
    k_gather<O><<<(unsigned)((n + B - 1) / B), TransferShape<O>::NT_G, 0, s>>>(fine, coarse, rec, n);
    return cudaGetLastError();
  }
  cudaError_t tag(const TagArgs& a, cudaStream_t s) const override {
    if (a.n == 0) return cudaSuccess;
    k_tag<O><<<(a.n + 127) / 128, 128, 0, s>>>(a);
    return cudaGetLastError();
  }
  cudaError_t seed_features(const SeedFeatArgs& a, cudaStream_t s) const override {
    const long long n = (long long)a.n * (O::Q * O::NP_S + 1);
    if (n == 0) return cudaSuccess;
    k_seed_features<O><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a);
    return cudaGetLastError();
  }
  cudaError_t seed_targets(const SeedFeatArgs& a, cudaStream_t s) const override {
    const long long n = (long long)a.n * O::Q;
    if (n == 0) return cudaSuccess;
    k_seed_targets<O><<<(unsigned)((n + 127) / 128), 128, 0, s>>>(a);
    return cudaGetLastError();
  }
  cudaError_t seed_assemble(const double* Uw, const float* Y, const float* y_mean, const float* y_std, int n,
                            const int8_t* elem_level, const LevelGeom& geom, const double* dt, double* Hseed,
                            cudaStream_t s) const override {
    const long long t = (long long)n * O::Q;
    if (t == 0) return cudaSuccess;
    k_seed_assemble<O><<<(unsigned)((t + 127) / 128), 128, 0, s>>>(Uw, Y, y_mean, y_std, n, elem_level, geom, dt,
                                                                    Hseed);
    return cudaGetLastError();
  }
  cudaError_t seed_infer_tc(const SeedTCArgs& a, cudaStream_t s) const override {
    if constexpr (!seed_tc_fits(O::Q, O::NP_S, O::NP_ST)) {
      return cudaErrorNotSupported;  // layers too wide for the fused kernel: the SIMT path serves
    } else {
      if (a.n <= 0) return cudaSuccess;
      static std::atomic<unsigned long long> attr{0};
      cudaError_t e = ensure_smem_attr(attr, k_seed_infer_tc<O>, kSeedTcSmem);
      if (e != cudaSuccess) return e;
      k_seed_infer_tc<O><<<(a.n + kSeedTcRows - 1) / kSeedTcRows, kSeedTcThreads, kSeedTcSmem, s>>>(a);
      return cudaGetLastError();
    }
  }
  cudaError_t limit_tvb(const LimiterArgs& a, cudaStream_t s) const override {
    if (a.n <= 0) return cudaSuccess;
    k_limit_tvb<O><<<(a.n + 127) / 128, 128, 0, s>>>(a);
    return cudaGetLastError();
  }
  cudaError_t lp_norm(const LpArgs& a, cudaStream_t s) const override {
    if (a.n_valid <= 0) return cudaSuccess;
    k_lp_norm<O><<<(a.n_valid + 127) / 128, 128, 0, s>>>(a);
    return cudaGetLastError();
  }
  cudaError_t init_ic(const ICArgs& a, cudaStream_t s) const override {
    const int bs = 64;
    k_init_ic<O><<<(a.n_elem + bs - 1) / bs, bs, 0, s>>>(a);
    return cudaGetLastError();
  }
};

}  // namespace

const KernelSet* ADG_FACTORY() {
  static Impl impl;
  return &impl;
}

}  // namespace adg
