// Pass B of the 6D mass operator: inverse DFT along axes 4-6, multiply by the
// material E/NF, forward DFT along axes 4-6, for every tile of the
// tile-major work fields (WorkTile in fft6d.cuh).
//
// Persistent kernel: each CTA owns a contiguous range of units (tile k,
// field f) and streams them through two shared-memory stages.  One thread
// pulls a unit with n bulk copies (one per i6-plane, completed on the stage's
// mbarrier) plus, at the first unit of a tile, the material tile; the copy of
// unit i+2 is issued as soon as unit i has been read out of its stage, so
// global latency overlaps the transforms of the next unit.  In shared memory
// element (t, i4, i5, i6) of a unit sits at t + TT*i4 + P5*i5 + P6*i6 with
// P5 = TT*n and P6 = TT*n^2 + TT (one padding row per plane); each phase
// transforms one line per thread in place:
//   phase 1  axis 4, lanes (t, i6, i5) -- stride TT
//   phase 2  axis 6, lanes (t, i4, i5) -- stride P6
//   phase 3  axis 5, lanes (t, i4, i6) -- stride P5: inverse, *E/NF, forward
//   phase 4  axis 6 (forward)
//   phase 5  axis 4 (forward), then rows of TT elements stored to global.
// The lane orders and the padding row were chosen by counting shared-memory
// wavefronts of every phase (16-lane halves for 8-byte, 8-lane quarters for
// 16-byte elements); they reach the conflict-free count for n <= 8 and stay
// within 12% of it for the larger sizes.
#pragma once
#include "bulk.cuh"
#include "fft6d.cuh"


namespace fame {

// Range of a material grid, on the device: bit patterns of its smallest and largest value and
// whether every value is a positive finite number (good != 0).  Preset with 0xff bytes.
struct MaterialRange {
  unsigned long long lo, hiInv;  // hiInv: complement of the largest value's pattern
  unsigned good, pad;
};

template <int n, typename T> struct PassBGeom {
  static constexpr int TT = WorkTile<n, T>::TT;
  static constexpr int n2 = n * n, n3 = n * n * n;
  static constexpr int L = TT * n2;        // lines per phase (one per working thread)
  static constexpr int P5 = TT * n;        // i5 pitch (elements)
  static constexpr int P6 = TT * n2 + TT;  // i6 plane pitch
  static constexpr int stage = n * P6;     // elements per stage
  static constexpr int tile = TT * n3;     // elements per tile (global)
  static constexpr unsigned plane_bytes = (unsigned)(TT * n2 * sizeof(C<T>));
  static constexpr int threads = (L + 31) / 32 * 32;
  static_assert((P6 * sizeof(C<T>)) % 16 == 0 && (stage * sizeof(C<T>)) % 16 == 0, "bulk-copy alignment");
  static_assert(plane_bytes % 16 == 0, "bulk-copy size");
  // n >= 12: two stages of fields fill so much shared memory that staging the material too would
  // leave one CTA per SM; the threads read their material values from L2 / L1 instead, and the
  // register count is held to the CTAs that then fit (minBlocks).
  static constexpr bool stageE = n < 12;
  static constexpr int minBlocks = n == 12 ? 2 : n == 14 ? 1 : 0;
  static constexpr int maxThreads = n < 12 ? 512 : threads;
  template <typename TE> static constexpr size_t smem_bytes() {
    return 2 * stage * sizeof(C<T>) + (stageE ? 2 * (size_t)tile * sizeof(TE) : 0) + 2 * sizeof(uint64_t);
  }
};

template <int n, typename T, typename TE>
__global__ void __launch_bounds__(PassBGeom<n, T>::maxThreads, PassBGeom<n, T>::minBlocks) k_passB(C<T>* __restrict__ work, const TE* __restrict__ Et, int nfields,
                                              long long NF, Gate gate, unsigned* fault,
                                              unsigned poll_limit = kMbarPollLimit, int arm_only = 0) {
  if (gate.off()) return;
  using G = PassBGeom<n, T>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  C<T>* stg = reinterpret_cast<C<T>*>(smem_raw);
  TE* es = reinterpret_cast<TE*>(smem_raw + 2 * G::stage * sizeof(C<T>));
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + 2 * G::stage * sizeof(C<T>) +
                                              (G::stageE ? 2 * G::tile * sizeof(TE) : 0));
  constexpr int tiles = G::n3 / G::TT;
  const int U = tiles * nfields;
  const int u0 = (int)((long long)blockIdx.x * U / gridDim.x);
  const int u1 = (int)((long long)(blockIdx.x + 1) * U / gridDim.x);
  if (u0 >= u1) return;
  const int k0 = u0 / nfields;
  const int tid = threadIdx.x;

  auto issue = [&](int u, int s) {
    const int k = u / nfields, f = u - k * nfields;
    const bool needE = G::stageE && ((u == u0) || (f == 0));
    mbar_arrive_expect_tx(&bar[s], n * G::plane_bytes + (needE ? (unsigned)(G::tile * sizeof(TE)) : 0u));
    if (arm_only) return;  // fault-path self-test: the bytes never come, nothing is in flight
    const C<T>* src = work + (long long)f * NF + (long long)k * G::tile;
    C<T>* dst = stg + s * G::stage;
#pragma unroll 1
    for (int p = 0; p < n; ++p) bulk_g2s(dst + p * G::P6, src + p * G::TT * G::n2, G::plane_bytes, &bar[s]);
    if (needE)
      bulk_g2s(es + ((k - k0) & 1) * G::tile, Et + (long long)k * G::tile, (unsigned)(G::tile * sizeof(TE)), &bar[s]);
  };

  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init_fence();
    issue(u0, 0);
    if (u0 + 1 < u1) issue(u0 + 1, 1);
  }
  __syncthreads();

  const bool act = tid < G::L;
  const int t = tid % G::TT, r = tid / G::TT, ra = r % n, rb = r / n;
  const int b1 = t + G::P5 * rb + G::P6 * ra;  // axis-4 line (t, i6 = ra, i5 = rb)
  const int b2 = t + G::TT * ra + G::P5 * rb;  // axis-6 line (t, i4 = ra, i5 = rb)
  const int b3 = t + G::TT * ra + G::P6 * rb;  // axis-5 line (t, i4 = ra, i6 = rb)
  const int gout = G::TT * (n * rb + G::n2 * ra) + t;  // (t, i4 = 0, i5 = rb, i6 = ra) within a tile

#pragma unroll 1
  for (int u = u0, i = 0; u < u1; ++u, ++i) {
    const int s = i & 1;
    const bool landed = mbar_wait(&bar[s], (unsigned)((i >> 1) & 1), poll_limit);
    if (!__syncthreads_and(landed)) {  // bounded wait, agreed on by the whole CTA
      if (tid == 0) {
        // copies in flight still land in this CTA's shared memory: wait for them (bounded) before it exits
        mbar_wait(&bar[s], (unsigned)((i >> 1) & 1), poll_limit);
        if (u + 1 < u1) mbar_wait(&bar[s ^ 1], (unsigned)(((i + 1) >> 1) & 1), poll_limit);
        if (fault) atomicOr(fault, 1u);
      }
      return;
    }
    C<T>* S = stg + s * G::stage;
    const int k = u / nfields, f = u - k * nfields;
    const TE* E = es + ((k - k0) & 1) * G::tile;
    if (act) line_dft<n, +1, T>(S + b1, G::TT);
    __syncthreads();
    if (act) line_dft<n, +1, T>(S + b2, G::P6);
    TE ev[G::stageE ? 1 : n];  // unstaged material, on its way across the barrier
    if constexpr (!G::stageE) {
      if (act) {
#pragma unroll
        for (int j = 0; j < n; ++j) ev[j] = __ldg(Et + (long long)k * G::tile + j * G::L + tid);
      }
    }
    __syncthreads();
    if (act) {
      C<T>* p = S + b3;
      T re[n], im[n];
#pragma unroll
      for (int j = 0; j < n; ++j) {
        const C<T> v = p[j * G::P5];
        re[j] = v.x;
        im[j] = v.y;
      }
      Dft<n, +1, T>::run(re, im);
#pragma unroll
      for (int j = 0; j < n; ++j) {
        const T e = (T)(G::stageE ? E[j * G::L + tid] : ev[G::stageE ? 0 : j]);
        re[j] *= e;
        im[j] *= e;
      }
      Dft<n, -1, T>::run(re, im);
#pragma unroll
      for (int j = 0; j < n; ++j) p[j * G::P5] = mk<T>(re[j], im[j]);
    }
    __syncthreads();
    if (act) line_dft<n, -1, T>(S + b2, G::P6);
    __syncthreads();
    T re[n], im[n];
    if (act) {
#pragma unroll
      for (int j = 0; j < n; ++j) {
        const C<T> v = S[b1 + j * G::TT];
        re[j] = v.x;
        im[j] = v.y;
      }
      Dft<n, -1, T>::run(re, im);
    }
    __syncthreads();  // stage s has been read out: refill it
    if (tid == 0 && u + 2 < u1) {
      fence_proxy_async_smem();
      issue(u + 2, s);
    }
    if (act) {
      C<T>* dst = work + (long long)f * NF + (long long)k * G::tile + gout;
#pragma unroll
      for (int j = 0; j < n; ++j) dst[j * G::TT] = mk<T>(re[j], im[j]);
    }
  }
}

// Inverse-only pass B (axes 4-6, no material) for the mass adjoint: modes x 3 fields in, per
// mode the density sum_c |w_c|^2 in natural order out (the transformed fields are not needed
// and never written).  Persistent and fed like k_passB; a CTA takes whole (tile, mode) pairs,
// the three fields of a pair accumulate in the registers of the last axis' lines.
template <int n>
__global__ void __launch_bounds__((PassBGeom<n, double>::threads), n >= 10 && n < 14 ? 2 : 0)
k_passB_density(const double2* __restrict__ work, double* __restrict__ dens, int modes, long long NF, unsigned* fault,
                unsigned poll_limit = kMbarPollLimit, int arm_only = 0) {
  using G = PassBGeom<n, double>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  double2* stg = reinterpret_cast<double2*>(smem_raw);
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + 2 * G::stage * sizeof(double2));
  const int P = (G::n3 / G::TT) * modes;
  const int p0 = (int)((long long)blockIdx.x * P / gridDim.x), p1 = (int)((long long)(blockIdx.x + 1) * P / gridDim.x);
  if (p0 >= p1) return;
  const int units = 3 * (p1 - p0), tid = threadIdx.x;
  auto issue = [&](int i) {
    const int p = p0 + i / 3, k = p / modes, md = p - k * modes, s = i & 1;
    mbar_arrive_expect_tx(&bar[s], n * G::plane_bytes);
    if (arm_only) return;  // fault-path self-test, as in k_passB
    const double2* src = work + (3LL * md + i % 3) * NF + (long long)k * G::tile;
#pragma unroll 1
    for (int q = 0; q < n; ++q)
      bulk_g2s(stg + s * G::stage + q * G::P6, src + q * G::TT * G::n2, G::plane_bytes, &bar[s]);
  };
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init_fence();
    issue(0);
    issue(1);  // units >= 3
  }
  __syncthreads();
  const bool act = tid < G::L;
  const int t = tid % G::TT, r = tid / G::TT, ra = r % n, rb = r / n;
  double d[n];
#pragma unroll 1
  for (int i = 0; i < units; ++i) {
    const int s = i & 1, f = i % 3;
    const bool landed = mbar_wait(&bar[s], (unsigned)((i >> 1) & 1), poll_limit);
    if (!__syncthreads_and(landed)) {  // bounded wait, agreed on by the whole CTA
      if (tid == 0) {  // copies in flight land first, as in k_passB
        mbar_wait(&bar[s], (unsigned)((i >> 1) & 1), poll_limit);
        if (i + 1 < units) mbar_wait(&bar[s ^ 1], (unsigned)(((i + 1) >> 1) & 1), poll_limit);
        if (fault) atomicOr(fault, 1u);
      }
      return;
    }
    double2* S = stg + s * G::stage;
    if (act) line_dft<n, +1, double>(S + t + G::P5 * rb + G::P6 * ra, G::TT);  // axis 4
    __syncthreads();
    if (act) line_dft<n, +1, double>(S + t + G::TT * ra + G::P5 * rb, G::P6);  // axis 6
    __syncthreads();
    if (act) {  // axis 5
      const double2* p = S + t + G::TT * ra + G::P6 * rb;
      double re[n], im[n];
#pragma unroll
      for (int j = 0; j < n; ++j) {
        const double2 v = p[j * G::P5];
        re[j] = v.x;
        im[j] = v.y;
      }
      Dft<n, +1, double>::run(re, im);
#pragma unroll
      for (int j = 0; j < n; ++j) {
        const double a = re[j] * re[j] + im[j] * im[j];
        d[j] = f == 0 ? a : d[j] + a;
      }
    }
    __syncthreads();  // stage s has been read out: refill it
    if (tid == 0 && i + 2 < units) {
      fence_proxy_async_smem();
      issue(i + 2);
    }
    if (act && f == 2) {
      const int p = p0 + i / 3, k = p / modes, md = p - k * modes;
      double* o = dens + md * NF + (long long)k * G::TT + t + (long long)G::n3 * (ra + G::n2 * rb);
#pragma unroll
      for (int j = 0; j < n; ++j) o[(long long)G::n3 * n * j] = d[j];
    }
  }
}

// Material in the order pass B reads it: tile kt holds, for j = i5 and the
// phase-3 line index kk = t + TT*(i4 + n*i6), the value E(c123, c456)*scale at
// kt*TT*n^3 + j*TT*n^2 + kk, with c123 = kt*TT + t, c456 = i4 + n*j + n^2*i6.
// outInv (optional): scale / E in the same order (the material of the inverse mass operator).
// With range, the smallest and largest value of E and whether any is not a positive finite
// number (MaterialRange; every byte preset to 0xff by the caller).
template <typename TE>
__global__ void k_tile_E(const double* __restrict__ E, int n, int TT, long long NF, double scale, TE* __restrict__ out,
                         TE* __restrict__ outInv, MaterialRange* range) {
  unsigned long long lo = ~0ull, hi = 0ull;
  bool bad = false;
  const long long n3 = (long long)n * n * n, L = (long long)TT * n * n, tile = TT * n3;
  for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < NF; o += (long long)gridDim.x * blockDim.x) {
    const long long kt = o / tile, rem = o % tile;
    const long long j = rem / L, kk = rem % L;
    const long long t = kk % TT, rr = kk / TT, i4 = rr % n, i6 = rr / n;
    const long long c123 = kt * TT + t, c456 = i4 + n * j + (long long)n * n * i6;
    const double e = E[c123 + n3 * c456];
    out[o] = (TE)(e * scale);
    if (outInv) outInv[o] = (TE)(scale / e);
    if (range) {  // bit patterns of positive doubles are ordered like their values
      bad |= !(e > 0.0) || !isfinite(e);
      const unsigned long long b = (unsigned long long)__double_as_longlong(e);
      lo = b < lo ? b : lo;
      hi = b > hi ? b : hi;
    }
  }
  if (range) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long l2 = __shfl_xor_sync(0xffffffffu, lo, o), h2 = __shfl_xor_sync(0xffffffffu, hi, o);
      lo = l2 < lo ? l2 : lo;
      hi = h2 > hi ? h2 : hi;
    }
    const bool any_bad = __any_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&range->lo, lo);
      atomicMin(&range->hiInv, ~hi);
      if (any_bad) atomicAnd(&range->good, 0u);
    }
  }
}

}  // namespace fame
