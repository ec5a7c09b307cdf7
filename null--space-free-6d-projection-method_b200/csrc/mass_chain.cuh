// Host-side launch of one fused mass-operator chain (pass A -> B -> C) for a
// runtime axis length n = 2N, dispatching to the compile-time kernels.
#pragma once
#include "passb.cuh"

namespace fame {

inline int round32(int x) { return (x + 31) / 32 * 32; }

// Pass B over nfields tile-major fields with the tiled material Et (E/NF in the
// layout of k_tile_E for this n and T): a persistent grid of (resident CTAs per
// SM) x SMs, each CTA owning a contiguous range of (tile, field) units.
// poll_limit / arm_only: fault-path self-test (fame_selftest_bounded_wait).
template <int n, typename T, typename TE>
int launch_passB(C<T>* work, int nfields, const TE* Et, long long NF, cudaStream_t st, Gate gate,
                 unsigned poll_limit = kMbarPollLimit, int arm_only = 0) {
  using G = PassBGeom<n, T>;
  constexpr size_t smem = G::template smem_bytes<TE>();
  static DeviceOnce once;
  FAME_TRY(ensure_smem(k_passB<n, T, TE>, smem, once));
  static int per_sm = [] {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_passB<n, T, TE>, G::threads, smem) != cudaSuccess) b = 1;
    return b < 1 ? 1 : b;
  }();
  const int units = (G::n3 / G::TT) * nfields;
  const int grid = std::min(units, per_sm * num_sms());
  k_passB<n, T, TE><<<grid, G::threads, smem, st>>>(work, Et, nfields, NF, gate, fault_word(), poll_limit, arm_only);
  ::fame::count_launch();
  return FAME_OK;
}

// Threads of the general passes: one per (field, line) where the fields' lines are separate
// items (FP64, several fields), one per line otherwise.
template <int n, typename T, int F> int pass_threads(int G) {
  return std::min(512, std::max(32, round32(G * n * n * (FieldsInRegs<T, F>::value ? 1 : F))));
}

template <int n, typename T, int F, class Pro>
int launch_passA(const Pro& pro, C<T>* work, long long NF, cudaStream_t st, Gate gate) {
  using Q = Cube<n, T>;
  constexpr int G = PassACols<n, T>::value;
  const size_t smem = (size_t)G * F * Q::size * sizeof(C<T>);
  static DeviceOnce once;
  FAME_TRY(ensure_smem(k_passA<n, T, F, G, Pro>, smem, once));
  const int threads = pass_threads<n, T, F>(G);
  k_passA<n, T, F, G, Pro><<<Q::n3 / G, threads, smem, st>>>(pro, work, NF, gate);
  ::fame::count_launch();
  return FAME_OK;
}

template <int n, typename T, int F, class Epi>
int launch_passC(const Epi& epi, const C<T>* work, long long NF, cudaStream_t st, Gate gate) {
  using Q = Cube<n, T>;
  constexpr int G = PassACols<n, T>::value;
  const size_t smem = (size_t)G * F * Q::size * sizeof(C<T>);
  static DeviceOnce once;
  FAME_TRY(ensure_smem(k_passC<n, T, F, G, Epi>, smem, once));
  const int threads = pass_threads<n, T, F>(G);
  k_passC<n, T, F, G, Epi><<<Q::n3 / G, threads, smem, st>>>(epi, work, NF, gate);
  ::fame::count_launch();
  return FAME_OK;
}

// Number of CTAs pass C launches (size of the reduction partials it needs).
inline long long passC_blocks(int n) { return (long long)n * n * n; }

template <int n, typename T, int F, class Pro, class Epi, typename TE>
int chain_n(const Pro& pro, const Epi& epi, C<T>* work, const TE* Et, long long NF,
            cudaStream_t st, Gate gate) {
  FAME_TRY((launch_passA<n, T, F, Pro>(pro, work, NF, st, gate)));
  FAME_TRY((launch_passB<n, T, TE>(work, F, Et, NF, st, gate)));
  FAME_TRY((launch_passC<n, T, F, Epi>(epi, work, NF, st, gate)));
  FAME_CUDA_TRY(cudaGetLastError());
  return FAME_OK;
}

// y-chain for axis length n in {2,4,...,14}.  work holds F fields of NF.
template <typename T, int F, class Pro, class Epi, typename TE>
int run_chain(int n, const Pro& pro, const Epi& epi, C<T>* work, const TE* Et, long long NF, cudaStream_t st, Gate gate = Gate{nullptr}) {
  switch (n) {
    case 2: return chain_n<2, T, F>(pro, epi, work, Et, NF, st, gate);
    case 4: return chain_n<4, T, F>(pro, epi, work, Et, NF, st, gate);
    case 6: return chain_n<6, T, F>(pro, epi, work, Et, NF, st, gate);
    case 8: return chain_n<8, T, F>(pro, epi, work, Et, NF, st, gate);
    case 10: return chain_n<10, T, F>(pro, epi, work, Et, NF, st, gate);
    case 12: return chain_n<12, T, F>(pro, epi, work, Et, NF, st, gate);
    case 14: return chain_n<14, T, F>(pro, epi, work, Et, NF, st, gate);
    default: return fail(FAME_ERR_UNSUPPORTED, "mass operator supports 2N in {2,4,...,14}");
  }
}

// Columns per CTA of the linear-field passes (one line per thread).
// n >= 10: one column (100 lines and more) per CTA, several CTAs per SM (measured 1-3 % faster
// K_r^{-1} actions than two columns, in both precision forms).  Below, two, which only the
// one-field products still use (chain_par takes the others, one column per CTA): n^3 / 2 CTAs
// reach more SMs than the 512-thread CTAs that eight to sixteen columns make, and fill whole
// warps better than single columns.  FP64 products of 24 vectors, two / one / eight and more
// columns: N=3 35.3 / 38.8 / 36.3 us, N=4 154.5 / 175 / 168 us; single vectors within 2 us.
template <int n, typename T> struct LinCols {
  static constexpr int value = n >= 10 ? 1 : 2;
  static_assert((n * n * n) % value == 0 && value * n * n <= 512, "linear chain tiling");
};

template <int n, typename T, int F, int G, class Pro, class Epi, typename TE>
int chain_lin_g(const Pro& pro, const Epi& epi, C<T>* work, const TE* Et, long long NF,
                cudaStream_t st, Gate gate) {
  using Q = Cube<n, T>;
  const size_t smem = (size_t)G * Q::size * sizeof(C<T>);
  const int threads = round32(G * Q::n2);
  static DeviceOnce onceA;
  FAME_TRY(ensure_smem(k_passA_lin<n, T, F, G, Pro>, smem, onceA));
  static DeviceOnce onceC;
  FAME_TRY(ensure_smem(k_passC_lin<n, T, F, G, Epi>, smem, onceC));
  k_passA_lin<n, T, F, G, Pro><<<Q::n3 / G, threads, smem, st>>>(pro, work, NF, gate);
  ::fame::count_launch();
  FAME_TRY((launch_passB<n, T, TE>(work, F, Et, NF, st, gate)));
  k_passC_lin<n, T, F, G, Epi><<<Q::n3 / G, threads, smem, st>>>(epi, work, NF, gate);
  ::fame::count_launch();
  FAME_CUDA_TRY(cudaGetLastError());
  return FAME_OK;
}

// Linear chain with the fields side by side (k_passA_par).
template <int n, typename T, int F, class Pro, class Epi, typename TE>
int chain_par(const Pro& pro, const Epi& epi, C<T>* work, const TE* Et, long long NF, cudaStream_t st, Gate gate) {
  using Q = Cube<n, T>;
  constexpr int G = 1;
  const size_t smA = (size_t)G * (F + 1) * Q::size * sizeof(C<T>), smC = (size_t)G * F * Q::size * sizeof(C<T>);
  const int threads = round32(F * G * Q::n2);
  static DeviceOnce onceA;
  FAME_TRY(ensure_smem(k_passA_par<n, T, F, G, Pro>, smA, onceA));
  static DeviceOnce onceC;
  FAME_TRY(ensure_smem(k_passC_par<n, T, F, G, Epi>, smC, onceC));
  k_passA_par<n, T, F, G, Pro><<<Q::n3 / G, threads, smA, st>>>(pro, work, NF, gate);
  FAME_TRY((launch_passB<n, T, TE>(work, F, Et, NF, st, gate)));
  k_passC_par<n, T, F, G, Epi><<<Q::n3 / G, threads, smC, st>>>(epi, work, NF, gate);
  ::fame::count_launch(2);
  FAME_CUDA_TRY(cudaGetLastError());
  return FAME_OK;
}

// The linear chain of n: several fields side by side at n <= 8 (k_passA_par, one column per CTA),
// one after another with LinCols columns per CTA above and for one field.  `cols` selects one of
// the alternatives compiled for the Bloch-path sizes (n = 6, 8, 10): that many columns per CTA
// and, at n <= 8 too, the fields one after another; any other value is the default.  The choice
// changes the kernels and the order of the grid reductions, not the arithmetic of a mode.  Where
// many instances share the GPU the larger CTAs can win: eight concurrent solves at N=4 take 294
// against 312 ms (FP64) and 218 against 225 ms (mixed) with two columns; a solve alone, and
// batches at N=3 and N=5, are fastest with the default.
template <int n, typename T, int F, class Pro, class Epi, typename TE>
int chain_lin_n(const Pro& pro, const Epi& epi, C<T>* work, const TE* Et, long long NF, cudaStream_t st, Gate gate,
                int cols) {
  if constexpr (n == 10) {
    if (cols == 2) return chain_lin_g<n, T, F, 2>(pro, epi, work, Et, NF, st, gate);
    if (cols == 4) return chain_lin_g<n, T, F, 4>(pro, epi, work, Et, NF, st, gate);
  } else if constexpr (n == 8) {
    if (cols == 2) return chain_lin_g<n, T, F, 2>(pro, epi, work, Et, NF, st, gate);
    if (cols == 4) return chain_lin_g<n, T, F, 4>(pro, epi, work, Et, NF, st, gate);
  } else if constexpr (n == 6) {
    if (cols == 4) return chain_lin_g<n, T, F, 4>(pro, epi, work, Et, NF, st, gate);
    if (cols == 6) return chain_lin_g<n, T, F, 6>(pro, epi, work, Et, NF, st, gate);
  }
  if constexpr (n <= 8 && F > 1) return chain_par<n, T, F>(pro, epi, work, Et, NF, st, gate);
  else return chain_lin_g<n, T, F, LinCols<n, T>::value>(pro, epi, work, Et, NF, st, gate);
}

// Linear-field chain (see k_passA_lin) for axis length n in {2,4,...,14}.
template <typename T, int F, class Pro, class Epi, typename TE>
int run_chain_lin(int n, const Pro& pro, const Epi& epi, C<T>* work, const TE* Et, long long NF, cudaStream_t st,
                  Gate gate = Gate{nullptr}, int cols = 0) {
  switch (n) {
    case 2: return chain_lin_n<2, T, F>(pro, epi, work, Et, NF, st, gate, cols);
    case 4: return chain_lin_n<4, T, F>(pro, epi, work, Et, NF, st, gate, cols);
    case 6: return chain_lin_n<6, T, F>(pro, epi, work, Et, NF, st, gate, cols);
    case 8: return chain_lin_n<8, T, F>(pro, epi, work, Et, NF, st, gate, cols);
    case 10: return chain_lin_n<10, T, F>(pro, epi, work, Et, NF, st, gate, cols);
    case 12: return chain_lin_n<12, T, F>(pro, epi, work, Et, NF, st, gate, cols);
    case 14: return chain_lin_n<14, T, F>(pro, epi, work, Et, NF, st, gate, cols);
    default: return fail(FAME_ERR_UNSUPPORTED, "mass operator supports 2N in {2,4,...,14}");
  }
}

// ------------------------------------------------------------ functors
// Identity prologue/epilogue of the general chain (natural order): F columns.
template <typename T, int F> struct ProCols {
  static constexpr bool natural = true;
  const C<T>* x[F];
  __device__ __forceinline__ void load(long long, long long i, C<T>* v) const {
#pragma unroll
    for (int f = 0; f < F; ++f) v[f] = x[f][i];
  }
};
template <typename T, int F> struct EpiCols {
  using Acc = T;
  static constexpr int K = 0;
  static constexpr bool natural = true;
  C<T>* y[F];
  T* partials = nullptr;
  unsigned* counter = nullptr;
  __device__ __forceinline__ void store(long long, long long i, const C<T>* v, Red<T, 1>&) const {
#pragma unroll
    for (int f = 0; f < F; ++f) y[f][i] = v[f];
  }
  __device__ __forceinline__ void finalize(const Red<T, 1>&) const {}
};

// Identity prologue / epilogue of the one-field linear chain: vector blockIdx.y of a block of
// NF-vectors in natural order.
template <typename T> struct ProCol {
  static constexpr bool unit0 = true, staged = true;
  const C<T>* x;
  long long NF;
  __device__ __forceinline__ C<T> raw(long long in) const { return __ldg(x + blockIdx.y * NF + in); }
  __device__ __forceinline__ C<T> from(C<T> v, long long) const { return v; }
  __device__ __forceinline__ T coef(int, long long, long long) const { return (T)1; }
};
template <typename T> struct EpiCol {
  using Acc = T;
  static constexpr int K = 0;
  static constexpr bool unit0 = true, staged = true;
  C<T>* y;
  long long NF;
  T* partials = nullptr;
  unsigned* counter = nullptr;
  __device__ __forceinline__ T coef(int, long long, long long) const { return (T)1; }
  __device__ __forceinline__ C<T> to(C<T> s, long long) const { return s; }
  __device__ __forceinline__ void put(long long in, C<T> v) const { y[blockIdx.y * NF + in] = v; }
  __device__ __forceinline__ void finalize(const Red<T, 1>&) const {}
};

// Vectors one mass product takes through the passes together: enough to fill the GPU on small
// grids (launches, not bytes, bound those), three components otherwise.
inline int mass_fields(long long NF) { return (int)std::max<long long>(3, std::min<long long>(24, (1LL << 22) / NF)); }

// Pass A alone for nvec consecutive NF-vectors.
template <int n, typename T> int passA_cols_n(const C<T>* x, int nvec, C<T>* work, long long NF, cudaStream_t st) {
  using Q = Cube<n, T>;
  constexpr int G = LinCols<n, T>::value;
  const size_t smem = (size_t)G * Q::size * sizeof(C<T>);
  static DeviceOnce once;
  FAME_TRY(ensure_smem(k_passA_lin<n, T, 1, G, ProCol<T>>, smem, once));
  k_passA_lin<n, T, 1, G, ProCol<T>>
      <<<dim3(Q::n3 / G, nvec), round32(G * Q::n2), smem, st>>>(ProCol<T>{x, NF}, work, NF, Gate{nullptr});
  ::fame::count_launch();
  return FAME_OK;
}

// y = M x for nvec consecutive NF-vectors (x and y natural order, work nvec fields): three
// launches for all of them.
template <int n, typename T, typename TE>
int mass_cols_n(const C<T>* x, C<T>* y, int nvec, C<T>* work, const TE* Et, long long NF, cudaStream_t st) {
  using Q = Cube<n, T>;
  constexpr int G = LinCols<n, T>::value;
  const size_t smem = (size_t)G * Q::size * sizeof(C<T>);
  const int threads = round32(G * Q::n2);
  const dim3 grid(Q::n3 / G, nvec);
  static DeviceOnce onceC;
  FAME_TRY(ensure_smem(k_passC_lin<n, T, 1, G, EpiCol<T>>, smem, onceC));
  FAME_TRY((passA_cols_n<n, T>(x, nvec, work, NF, st)));
  FAME_TRY((launch_passB<n, T, TE>(work, nvec, Et, NF, st, Gate{nullptr})));
  k_passC_lin<n, T, 1, G, EpiCol<T>><<<grid, threads, smem, st>>>(EpiCol<T>{y, NF}, work, NF, Gate{nullptr});
  ::fame::count_launch();
  FAME_CUDA_TRY(cudaGetLastError());
  return FAME_OK;
}
template <typename T, typename TE>
int run_mass_cols(int n, const C<T>* x, C<T>* y, int nvec, C<T>* work, const TE* Et, long long NF, cudaStream_t st) {
  switch (n) {
    case 2: return mass_cols_n<2, T>(x, y, nvec, work, Et, NF, st);
    case 4: return mass_cols_n<4, T>(x, y, nvec, work, Et, NF, st);
    case 6: return mass_cols_n<6, T>(x, y, nvec, work, Et, NF, st);
    case 8: return mass_cols_n<8, T>(x, y, nvec, work, Et, NF, st);
    case 10: return mass_cols_n<10, T>(x, y, nvec, work, Et, NF, st);
    case 12: return mass_cols_n<12, T>(x, y, nvec, work, Et, NF, st);
    case 14: return mass_cols_n<14, T>(x, y, nvec, work, Et, NF, st);
    default: return fail(FAME_ERR_UNSUPPORTED, "mass operator supports 2N in {2,4,...,14}");
  }
}

// Coefficients of the orthogonalised inner operator
// (exp1/build_experiment1_q_system_C_compact.m:21-31).
template <typename T> struct MhatCoef {
  const T* invC;
  const T* W1;
  const T* W2;
};

}  // namespace fame
