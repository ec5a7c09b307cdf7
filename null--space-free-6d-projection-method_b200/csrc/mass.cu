// 6D Fourier mass operator: handle creation, the four mass modes of the
// reference (exp1/build_mass_backend_large_scalar.m:28-31), the raw
// applyMij_fft entry and the rank-1-lattice drop-in.
#include <algorithm>
#include <cstring>
#include <vector>
#include "internal.cuh"
#include "mass_chain.cuh"
#include "dmma.cuh"

namespace fame {

// Pass-B tile width of the chains in precision T for a runtime axis length n.
template <typename T> int work_tt(int n) {
  switch (n) {
    case 2: return WorkTile<2, T>::TT;
    case 4: return WorkTile<4, T>::TT;
    case 6: return WorkTile<6, T>::TT;
    case 8: return WorkTile<8, T>::TT;
    case 10: return WorkTile<10, T>::TT;
    case 12: return WorkTile<12, T>::TT;
    default: return WorkTile<14, T>::TT;
  }
}

// E*scale (and scale/E into outInv) in the pass-B tile order of the chains in precision T.
template <typename T> int tile_E(const double* E, int n, long long NF, double scale, T* out, cudaStream_t st,
                                  T* outInv = nullptr, MaterialRange* range = nullptr) {
  const int blocks = (int)std::min<long long>((NF + 255) / 256, 148 * 16);
  k_tile_E<T><<<blocks, 256, 0, st>>>(E, n, work_tt<T>(n), NF, scale, out, outInv, range);
  ::fame::count_launch();
  FAME_CUDA_TRY(cudaGetLastError());
  return FAME_OK;
}

// Verify that (inputIdx, targetIdx, M) is the radix rank-1 plan of
// exp1/build_radix_exact_rank1_plan_scalar.m:18-43 (1-based indices).
__global__ void k_check_rank1(const uint32_t* in, const uint32_t* tg, long long NF, int n,
                              long long B, long long M, long long shift, unsigned* bad) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < NF;
       i += (long long)gridDim.x * blockDim.x) {
    long long tmp = i, code = 0, z = 1;
    for (int j = 0; j < 6; ++j) {
      code += (tmp % n) * z;
      tmp /= n;
      z *= B;
    }
    const long long target = (code + shift) % M;
    if ((long long)in[i] != code + 1 || (long long)tg[i] != target + 1) atomicAdd(bad, 1u);
  }
}

// Scalar mass action on ncols consecutive columns, up to `fields` at a time.  work: that many
// NF-fields of scratch that must not alias x or y (pass C reads it tile-major while writing y
// by columns).  One chain over the three components of a product instead of three one-field
// chains whose passes read and wrote x and y by lines: FP64 product of 3 NF values at N=2
// 36.9 -> 15.2 us, N=5 118.6 -> 92.1 us, N=7 906 -> 706 us.
template <typename T>
int mass_scalar_cols(int n, long long NF, const C<T>* x, C<T>* y, int ncols, const T* Et, C<T>* work, int fields,
                     cudaStream_t st) {
  for (int j = 0; j < ncols; j += fields)
    FAME_TRY((run_mass_cols<T>(n, x + (long long)j * NF, y + (long long)j * NF, std::min(fields, ncols - j), work, Et, NF,
                               st)));
  return FAME_OK;
}

// out[j, t] = (1/NF) sum_y g_t(y) d_j(y), d_j = sum_c |w_c|^2 with w_c the unnormalised inverse
// DFT of component c of mode j, i.e. NF sum_y g_t(y) sum_c |ifftn(x_c)(y)|^2 = x^H (dM/dtheta_t) x.
// The product of 16 densities and 8 parameter fields as FP64 mma.m8n8k4 (rows modes, columns
// parameters, the contraction permuted so that a lane reads four consecutive y of one row): every
// field is read once for 16 modes, bound by HBM.  Per-mode sums read the parameter fields again
// for every mode (72 of 211 us per mode at N=6, seven parameters).
constexpr int kMaxAdjParams = 8;
struct AdjParams {
  const double* g[kMaxAdjParams];
};
template <bool VEC> __device__ __forceinline__ void load4(const double* p, double* v) {
  if (VEC) {
    const double2 a = __ldg(reinterpret_cast<const double2*>(p)), b = __ldg(reinterpret_cast<const double2*>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = __ldg(p + k);
  }
}
constexpr int kAdjWarps = 8;
// VEC: every parameter field is 16-byte aligned.  partials: [block][16][8]
template <bool VEC>
__global__ void __launch_bounds__(32 * kAdjWarps) k_adjoint_gemm(const double* __restrict__ dens, int modes, AdjParams gp,
                                                                int np, long long NF, double* partials,
                                                                unsigned* counter, double* out) {
  __shared__ double red[kAdjWarps][16][kMaxAdjParams];
  __shared__ bool am_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const bool r0 = g < modes, r1 = g + 8 < modes, cg = g < np;
  const double *d0 = dens + (r0 ? g : 0) * NF, *d1 = dens + (r1 ? g + 8 : 0) * NF, *gg = gp.g[cg ? g : 0];
  double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
  const long long step = 16LL * kAdjWarps * gridDim.x;
  for (long long y0 = 16LL * (blockIdx.x * kAdjWarps + warp); y0 < NF; y0 += step) {  // NF is a multiple of 64
    const long long y = y0 + 4 * t;
    double a[4] = {}, b[4] = {}, c[4] = {};
    if (r0) load4<true>(d0 + y, a);
    if (r1) load4<true>(d1 + y, b);
    if (cg) load4<VEC>(gg + y, c);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      dmma_8x8x4(acc[0][0], acc[0][1], a[k], c[k]);
      if (modes > 8) dmma_8x8x4(acc[1][0], acc[1][1], b[k], c[k]);
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int q = 0; q < 2; ++q) red[warp][8 * h + g][2 * t + q] = acc[h][q];
  __syncthreads();
  if (threadIdx.x < 128) {
    const int m = threadIdx.x / 8, q = threadIdx.x % 8;
    double s = 0.0;
    for (int w = 0; w < kAdjWarps; ++w) s += red[w][m][q];
    partials[(size_t)blockIdx.x * 128 + threadIdx.x] = s;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) am_last = atomicAdd(counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!am_last) return;
  __threadfence();
  // two threads of eight interleaved partial sums per value: short chains of loads and additions
  double s[8] = {};
  for (unsigned b = threadIdx.x / 128; b < gridDim.x; b += 16)
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (b + 2 * k < gridDim.x) s[k] += ((volatile double*)partials)[(size_t)(b + 2 * k) * 128 + threadIdx.x % 128];
  double* part = &red[0][0][0];
  part[threadIdx.x] = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
  __syncthreads();
  if (threadIdx.x < 128) out[threadIdx.x] = (part[threadIdx.x] + part[threadIdx.x + 128]) / (double)NF;
  if (threadIdx.x == 0) *counter = 0u;
}

// densities of `modes` consecutive modes (x: 3 NF each) through work (3 modes fields)
template <int n>
int launch_density(const double2* work, double* dens, int modes, long long NF, cudaStream_t st,
                   unsigned poll_limit = kMbarPollLimit, int arm_only = 0) {
  using G = PassBGeom<n, double>;
  constexpr size_t smem = 2 * (size_t)G::stage * sizeof(double2) + 2 * sizeof(uint64_t);
  static DeviceOnce once;
  FAME_TRY(ensure_smem(k_passB_density<n>, smem, once));
  static int per_sm = [] {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_passB_density<n>, G::threads, smem) != cudaSuccess) b = 1;
    return b < 1 ? 1 : b;
  }();
  const int grid = std::min((G::n3 / G::TT) * modes, per_sm * num_sms());
  k_passB_density<n><<<grid, G::threads, smem, st>>>(work, dens, modes, NF, fault_word(), poll_limit, arm_only);
  ::fame::count_launch();
  FAME_CUDA_TRY(cudaGetLastError());
  return FAME_OK;
}
template <int n>
int adjoint_density_n(const double2* x, double2* work, double* dens, int modes, long long NF, cudaStream_t st) {
  FAME_TRY((passA_cols_n<n, double>(x, 3 * modes, work, NF, st)));
  return launch_density<n>(work, dens, modes, NF, st);
}

int check_N(int N) {
  if (N < 1 || N > 7) return fail(FAME_ERR_UNSUPPORTED, "N must be in [1,7] (2N <= 14)");
  return FAME_OK;
}

long long grid_NF(int N) {
  long long n = 2 * N, NF = 1;
  for (int d = 0; d < 6; ++d) NF *= n;
  return NF;
}

// mode dispatch on a typed pointer pair
template <typename T> const T* et_of(fame_mass* m);
template <> const double* et_of<double>(fame_mass* m) { return m->Et64; }
template <> const float* et_of<float>(fame_mass* m) { return m->Et32; }

// mode dispatch on a typed pointer pair
template <typename T>
int mass_apply_typed(fame_mass* m, int mode, const C<T>* x, C<T>* y, int nrhs) {
  const long long NF = m->NF;
  cudaStream_t st = m->ctx->stream;
  const T* Et = et_of<T>(m);
  C<T>* work = reinterpret_cast<C<T>*>(m->work);
  const int nf = mass_fields(NF);
  switch (mode) {
    case FAME_MASS_SCALAR:
      return mass_scalar_cols<T>(m->n, NF, x, y, nrhs, Et, work, nf, st);
    case FAME_MASS_FULL3:
      // 3NF x nrhs, column-major: each column holds three components
      return mass_scalar_cols<T>(m->n, NF, x, y, 3 * nrhs, Et, work, nf, st);
    case FAME_MASS_COL3:
      for (int j = 0; j < nrhs; ++j) {
        C<T>* yj = y + 3LL * NF * j;
        FAME_CUDA_TRY(cudaMemsetAsync(yj, 0, 2 * NF * sizeof(C<T>), st));
        FAME_TRY(mass_scalar_cols<T>(m->n, NF, x + NF * j, yj + 2 * NF, 1, Et, work, nf, st));
      }
      return FAME_OK;
    case FAME_MASS_COLS12:
      for (int j = 0; j < nrhs; ++j) {
        C<T>* yj = y + 3LL * NF * j;
        FAME_TRY(mass_scalar_cols<T>(m->n, NF, x + 2 * NF * j, yj, 2, Et, work, nf, st));
        FAME_CUDA_TRY(cudaMemsetAsync(yj + 2 * NF, 0, NF * sizeof(C<T>), st));
      }
      return FAME_OK;
    default:
      return fail(FAME_ERR_INVALID, "unknown mass mode");
  }
}

// One-shot applyMij_fft with a caller's natural-order E: a temporary tiled E/NF.
template <typename T>
int apply_fft_raw(fame_ctx* ctx, int n, long long NF, const double* E, const C<T>* x, C<T>* y, int nrhs) {
  T* Et = nullptr;
  C<T>* work = nullptr;
  const int fields = std::max(1, std::min(nrhs, mass_fields(NF)));
  FAME_TRY(dalloc((void**)&Et, NF * sizeof(T)));
  int s = dalloc((void**)&work, fields * NF * sizeof(C<T>));
  if (s == FAME_OK) s = tile_E<T>(E, n, NF, 1.0 / (double)NF, Et, ctx->stream);
  if (s == FAME_OK) s = mass_scalar_cols<T>(n, NF, x, y, nrhs, Et, work, fields, ctx->stream);
  if (s == FAME_OK && cudaStreamSynchronize(ctx->stream) != cudaSuccess) s = fail(FAME_ERR_CUDA, "applyMij_fft");
  dfree(Et);
  dfree(work);
  return s;
}

bool exact_inverse_ok(const MaterialRange& r, double tol) {
  double lo, hi;
  static_assert(sizeof(lo) == sizeof(r.lo), "bit patterns");
  std::memcpy(&lo, &r.lo, sizeof(lo));
  const unsigned long long h = ~r.hiInv;
  std::memcpy(&hi, &h, sizeof(hi));
  return r.good != 0 && lo > 0.0 && hi < 1e300 && 16 * 2.220446049250313e-16 * (hi / lo) <= tol;
}

int read_range(fame_ctx* ctx, fame_mass* m, MaterialRange* r) {
  static_assert(sizeof(*r) == sizeof(m->rangeWords), "host copy of the range");
  FAME_CUDA_TRY(cudaStreamWaitEvent(ctx->stream, m->ready, 0));
  if (!m->rangeRead) FAME_TRY(read_back(ctx, m->range, m->rangeWords, sizeof(m->rangeWords)));
  m->rangeRead = true;
  std::memcpy(r, m->rangeWords, sizeof(*r));
  return FAME_OK;
}

}  // namespace fame

using namespace fame;

extern "C" {

int fame_applyMij_fft(fame_ctx* ctx, int N, const double* E, const void* x, void* y, int nrhs,
                      int prec) {
  if (!ctx || !E || !x || !y || nrhs < 0) return fail(FAME_ERR_INVALID, "applyMij_fft arguments");
  FAME_TRY(check_N(N));
  const long long NF = grid_NF(N);
  if (prec == FAME_F64) return apply_fft_raw<double>(ctx, 2 * N, NF, E, (const double2*)x, (double2*)y, nrhs);
  if (prec == FAME_F32) return apply_fft_raw<float>(ctx, 2 * N, NF, E, (const float2*)x, (float2*)y, nrhs);
  return fail(FAME_ERR_INVALID, "prec must be FAME_F64 or FAME_F32");
}

int fame_mass_create(fame_ctx* ctx, int N, const double* E, fame_mass** out) {
  if (!ctx || !E || !out) return fail(FAME_ERR_INVALID, "fame_mass_create arguments");
  *out = nullptr;
  FAME_TRY(check_N(N));
  fame_mass* m = new fame_mass();
  m->ctx = ctx;
  m->N = N;
  m->n = 2 * N;
  m->NF = grid_NF(N);
  // tables, scratch and range in one allocation: each one costs a host wait
  auto carve = [&](Carve& cv) {
    m->Et64 = cv.take<double>(m->NF);
    m->EtInv64 = cv.take<double>(m->NF);
    m->Et32 = cv.take<float>(m->NF);
    m->EtInv32 = cv.take<float>(m->NF);
    m->work = cv.take<double2>(mass_fields(m->NF) * m->NF);
    m->range = cv.take<MaterialRange>(1);
  };
  Carve cv;
  carve(cv);
  int s = dalloc(&m->store, cv.used);
  if (s == FAME_OK) {
    cv = Carve{};
    cv.base = static_cast<char*>(m->store);
    carve(cv);
    if (cudaMemsetAsync(m->range, 0xff, sizeof(MaterialRange), ctx->stream) != cudaSuccess)
      s = fail(FAME_ERR_CUDA, "fame_mass_create");
  }
  const double scale = 1.0 / (double)m->NF;
  if (s == FAME_OK) s = tile_E<double>(E, m->n, m->NF, scale, m->Et64, ctx->stream, m->EtInv64, m->range);
  if (s == FAME_OK) s = tile_E<float>(E, m->n, m->NF, scale, m->Et32, ctx->stream, m->EtInv32);
  if (s == FAME_OK && (cudaEventCreateWithFlags(&m->ready, cudaEventDisableTiming) != cudaSuccess ||
                       cudaEventRecord(m->ready, ctx->stream) != cudaSuccess))
    s = fail(FAME_ERR_CUDA, "fame_mass_create: event");
  if (s != FAME_OK) {
    if (m->ready) cudaEventDestroy(m->ready);
    dfree(m->store);
    delete m;
    return s;
  }
  *out = m;
  return FAME_OK;
}

int fame_mass_destroy(fame_mass* m) {
  if (!m) return FAME_OK;
  cudaStreamSynchronize(m->ctx->stream);
  if (m->ready) cudaEventDestroy(m->ready);
  dfree(m->store);
  delete m;
  return FAME_OK;
}

int fame_selftest_bounded_wait(fame_mass* m, unsigned poll_limit) {
  if (!m) return fail(FAME_ERR_INVALID, "fame_selftest_bounded_wait: mass is NULL");
  FAME_TRY(check_fault(m->ctx));  // start from a clear fault word
  FAME_TRY(fame_selftest_expired_wait(m, 0, poll_limit));
  return check_fault(m->ctx);  // FAME_ERR_CUDA: the timeout was detected and reported
}

int fame_selftest_expired_wait(fame_mass* m, int kernel, unsigned poll_limit) {
  if (!m || kernel < 0 || kernel > 2) return fail(FAME_ERR_INVALID, "fame_selftest_expired_wait arguments");
  if (poll_limit < 1 || poll_limit > (1u << 20)) return fail(FAME_ERR_INVALID, "poll_limit must be in [1, 2^20]");
  fame_ctx* ctx = m->ctx;
  if (kernel == 2) return selftest_gram_schmidt_wait(ctx, poll_limit);
  if (kernel == 1) {  // no CTA gets as far as the densities: the scratch field stands in for them
    const double2* w64 = static_cast<const double2*>(m->work);
    double* d = static_cast<double*>(m->work);
    switch (m->n) {
      case 2: return launch_density<2>(w64, d, 1, m->NF, ctx->stream, poll_limit, 1);
      case 4: return launch_density<4>(w64, d, 1, m->NF, ctx->stream, poll_limit, 1);
      case 6: return launch_density<6>(w64, d, 1, m->NF, ctx->stream, poll_limit, 1);
      case 8: return launch_density<8>(w64, d, 1, m->NF, ctx->stream, poll_limit, 1);
      case 10: return launch_density<10>(w64, d, 1, m->NF, ctx->stream, poll_limit, 1);
      case 12: return launch_density<12>(w64, d, 1, m->NF, ctx->stream, poll_limit, 1);
      default: return launch_density<14>(w64, d, 1, m->NF, ctx->stream, poll_limit, 1);
    }
  }
  // one FP32 field in the handle's scratch (8 NF bytes of its 16 NF); every stage barrier
  // expects bytes that no copy delivers, so each CTA's first wait runs out and returns
  float2* w = reinterpret_cast<float2*>(m->work);
  const Gate g{nullptr};
  int s = FAME_OK;
  switch (m->n) {
    case 2: s = launch_passB<2, float, float>(w, 1, m->Et32, m->NF, ctx->stream, g, poll_limit, 1); break;
    case 4: s = launch_passB<4, float, float>(w, 1, m->Et32, m->NF, ctx->stream, g, poll_limit, 1); break;
    case 6: s = launch_passB<6, float, float>(w, 1, m->Et32, m->NF, ctx->stream, g, poll_limit, 1); break;
    case 8: s = launch_passB<8, float, float>(w, 1, m->Et32, m->NF, ctx->stream, g, poll_limit, 1); break;
    case 10: s = launch_passB<10, float, float>(w, 1, m->Et32, m->NF, ctx->stream, g, poll_limit, 1); break;
    case 12: s = launch_passB<12, float, float>(w, 1, m->Et32, m->NF, ctx->stream, g, poll_limit, 1); break;
    default: s = launch_passB<14, float, float>(w, 1, m->Et32, m->NF, ctx->stream, g, poll_limit, 1); break;
  }
  FAME_TRY(s);
  FAME_CUDA_TRY(cudaGetLastError());
  return FAME_OK;
}

int fame_mass_apply(fame_mass* m, int mode, const void* x, void* y, int nrhs, int prec) {
  if (!m || !x || !y || nrhs < 0) return fail(FAME_ERR_INVALID, "fame_mass_apply arguments");
  if (prec == FAME_F64) return mass_apply_typed<double>(m, mode, (const double2*)x, (double2*)y, nrhs);
  if (prec == FAME_F32) return mass_apply_typed<float>(m, mode, (const float2*)x, (float2*)y, nrhs);
  return fail(FAME_ERR_INVALID, "prec must be FAME_F64 or FAME_F32");
}

int fame_mass_adjoint_fields(fame_mass* m, const void* X, int nmodes, const double* const* dEps, int nparams,
                             double* out) {
  if (!m || !X || !dEps || !out || nmodes < 0 || nparams < 1 || nparams > kMaxAdjParams)
    return fail(FAME_ERR_INVALID, "fame_mass_adjoint arguments (1 <= nparams <= 8)");
  AdjParams gp{};
  bool vec = true;
  for (int t = 0; t < nparams; ++t) {
    if (!dEps[t]) return fail(FAME_ERR_INVALID, "fame_mass_adjoint arguments (1 <= nparams <= 8)");
    gp.g[t] = dEps[t];
    vec = vec && reinterpret_cast<uintptr_t>(dEps[t]) % 16 == 0;
  }
  if (nmodes == 0) return FAME_OK;
  const long long NF = m->NF;
  cudaStream_t st = m->ctx->stream;
  // modes whose fields go through the passes together, and whose densities wait for one product
  const int batch = std::max(1, std::min(nmodes, mass_fields(NF) / 3)), group = std::min(nmodes, 16);
  const int groups = (nmodes + 15) / 16, blocks = (int)std::min<long long>(num_sms() * 4LL, (NF + 127) / 128);
  double2* work;
  double *dens, *partials, *res;
  unsigned* counter;
  auto carve = [&](Carve& cv) {
    work = cv.take<double2>(3LL * batch * NF);
    dens = cv.take<double>((size_t)group * NF);
    partials = cv.take<double>((size_t)blocks * 128);
    res = cv.take<double>((size_t)groups * 128);
    counter = cv.take<unsigned>(1);
  };
  Carve cv;
  carve(cv);
  void* ws = nullptr;
  FAME_TRY(dalloc(&ws, cv.used));
  cv = Carve{};
  cv.base = static_cast<char*>(ws);
  carve(cv);
  FaultWatch watch(m->ctx);
  int s = cudaMemsetAsync(counter, 0, sizeof(unsigned), st) == cudaSuccess ? FAME_OK : fail(FAME_ERR_CUDA, "adjoint");
  for (int j0 = 0; j0 < nmodes && s == FAME_OK; j0 += 16) {
    const int jn = std::min(16, nmodes - j0);
    for (int j = 0; j < jn && s == FAME_OK; j += batch) {
      const double2* x = (const double2*)X + 3 * NF * (j0 + j);
      double* d = dens + (size_t)j * NF;
      const int nb = std::min(batch, jn - j);
      switch (m->n) {
        case 2: s = adjoint_density_n<2>(x, work, d, nb, NF, st); break;
        case 4: s = adjoint_density_n<4>(x, work, d, nb, NF, st); break;
        case 6: s = adjoint_density_n<6>(x, work, d, nb, NF, st); break;
        case 8: s = adjoint_density_n<8>(x, work, d, nb, NF, st); break;
        case 10: s = adjoint_density_n<10>(x, work, d, nb, NF, st); break;
        case 12: s = adjoint_density_n<12>(x, work, d, nb, NF, st); break;
        case 14: s = adjoint_density_n<14>(x, work, d, nb, NF, st); break;
        default: s = fail(FAME_ERR_UNSUPPORTED, "adjoint: unsupported N");
      }
    }
    if (s != FAME_OK) break;
    double* o = res + (size_t)(j0 / 16) * 128;
    if (vec) k_adjoint_gemm<true><<<blocks, 32 * kAdjWarps, 0, st>>>(dens, jn, gp, nparams, NF, partials, counter, o);
    else k_adjoint_gemm<false><<<blocks, 32 * kAdjWarps, 0, st>>>(dens, jn, gp, nparams, NF, partials, counter, o);
    ::fame::count_launch();
    if (cudaGetLastError() != cudaSuccess) s = fail(FAME_ERR_CUDA, "adjoint launch");
  }
  std::vector<double> h((size_t)groups * 128);
  if (s == FAME_OK &&
      cudaMemcpyAsync(h.data(), res, h.size() * sizeof(double), cudaMemcpyDeviceToHost, st) != cudaSuccess)
    s = fail(FAME_ERR_CUDA, "adjoint");
  if (s == FAME_OK) s = watch.check();  // synchronises; a copy that never came leaves densities unwritten
  dfree(ws);
  FAME_TRY(s);
  for (int j = 0; j < nmodes; ++j)
    for (int t = 0; t < nparams; ++t) out[(size_t)j * nparams + t] = h[(size_t)(j / 16) * 128 + (j % 16) * 8 + t];
  return FAME_OK;
}

int fame_mass_adjoint(fame_mass* m, const void* X, int nmodes, const double* dEps, int nparams, double* out) {
  if (!m || !X || !dEps || !out || nmodes < 0 || nparams < 1 || nparams > kMaxAdjParams)
    return fail(FAME_ERR_INVALID, "fame_mass_adjoint arguments (1 <= nparams <= 8)");
  const double* g[kMaxAdjParams];
  for (int t = 0; t < nparams; ++t) g[t] = dEps + (long long)t * m->NF;
  return fame_mass_adjoint_fields(m, X, nmodes, g, nparams, out);
}

int fame_applyMij_rank1_exact(fame_mass* m, const uint32_t* inputIdx, const uint32_t* targetIdx,
                              long long M, const void* x, void* y, int nrhs) {
  if (!m || !inputIdx || !targetIdx || !x || !y || nrhs < 0)
    return fail(FAME_ERR_INVALID, "applyMij_rank1_exact arguments");
  const long long n = m->n, B = 2 * n - 1;
  long long Mexp = n;
  for (int j = 0; j < 5; ++j) Mexp *= B;
  if (M != Mexp) return fail(FAME_ERR_INVALID, "rank1_exact_fft_scatter:BadSize (plan.M mismatch)");
  long long sumz = 0, z = 1;
  for (int j = 0; j < 6; ++j) {
    sumz += z;
    z *= B;
  }
  const long long shift = ((n - 1) * sumz) % M;
  unsigned* bad = nullptr;
  FAME_TRY(dalloc((void**)&bad, sizeof(unsigned)));
  cudaStream_t st = m->ctx->stream;
  cudaMemsetAsync(bad, 0, sizeof(unsigned), st);
  const int blocks = (int)std::min<long long>((m->NF + 255) / 256, 148 * 16);
  k_check_rank1<<<blocks, 256, 0, st>>>(inputIdx, targetIdx, m->NF, m->n, B, M, shift, bad);
  ::fame::count_launch();
  unsigned hbad = 0;
  int s = read_back(m->ctx, bad, &hbad, sizeof(unsigned));
  dfree(bad);
  FAME_TRY(s);
  if (hbad != 0) return fail(FAME_ERR_INVALID, "rank-1 plan index vectors are not the radix plan");
  return mass_apply_typed<double>(m, FAME_MASS_SCALAR, (const double2*)x, (double2*)y, nrhs);
}

}  // extern "C"
