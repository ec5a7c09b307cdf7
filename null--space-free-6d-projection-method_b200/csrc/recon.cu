// Yee-field reconstruction of a Fourier eigenvector component,
//   u(r) = sum_j c_j exp(i q_j . r)                (exp2/reconstruct_field_direct_blocked_exp3.m:8-15)
// and its multi-center Taylor approximation
//   u(r) ~ sum_{|a|<=p} gamma_a(r_c) (r - r_c)^a,
//   gamma_a(r_c) = i^|a|/a! sum_j c_j exp(i q_j . r_c) q_j^a   (exp2/taylor_on_blocks_exp3.m:1-79)
//
// Three device paths:
//  * k_direct_sum: the plain sum for any cut matrix (FP64 sincos per term);
//  * the factorised sum for an axis-block cut matrix P = [diag(d1); diag(d2)]
//    and points on a tensor grid: q_x depends only on (xi_1, xi_4), q_y on
//    (xi_2, xi_5), q_z on (xi_3, xi_6), so u = C x1 Ex x2 Ey x3 Ez is three
//    complex GEMMs against per-axis phase tables (exact in exact arithmetic);
//  * the Taylor moments (one CTA per mode chunk and center, one thread per
//    multi-index) and the per-block polynomial evaluation.
#include <algorithm>
#include <cmath>
#include <vector>
#include "internal.cuh"
#include "dmma.cuh"
#include "moment_slices.h"
#include "trig.cuh"

namespace fame {

static inline int rblocks(long long n, int t = 256) { return (int)std::min<long long>((n + t - 1) / t, 148 * 32); }

// ------------------------------------------------------------------ direct
constexpr int kDirectPts = 128;
constexpr int kDirectModes = 256;
__global__ void __launch_bounds__(kDirectPts) k_direct_sum(const double2* __restrict__ c, const double* __restrict__ Q,
                                                          long long NF, const double* __restrict__ R, long long M,
                                                          double2* __restrict__ u) {
  __shared__ double sq[3][kDirectModes];
  __shared__ double2 sc[kDirectModes];
  const long long i = (long long)blockIdx.x * kDirectPts + threadIdx.x;
  const bool act = i < M;
  const double rx = act ? R[i] : 0.0, ry = act ? R[M + i] : 0.0, rz = act ? R[2 * M + i] : 0.0;
  double ar = 0.0, ai = 0.0;
  for (long long j0 = 0; j0 < NF; j0 += kDirectModes) {
    const int nj = (int)std::min<long long>(kDirectModes, NF - j0);
    __syncthreads();
    for (int t = threadIdx.x; t < nj; t += blockDim.x) {
      sq[0][t] = Q[j0 + t];
      sq[1][t] = Q[NF + j0 + t];
      sq[2][t] = Q[2 * NF + j0 + t];
      sc[t] = c[j0 + t];
    }
    __syncthreads();
    if (act) {
      for (int t = 0; t < nj; ++t) {
        double s, co;
        sincos(sq[0][t] * rx + sq[1][t] * ry + sq[2][t] * rz, &s, &co);
        ar += sc[t].x * co - sc[t].y * s;
        ai += sc[t].x * s + sc[t].y * co;
      }
    }
  }
  if (act) u[i] = make_double2(ar, ai);
}

// -------------------------------------------------------------- factorised
// phase tables T[x + nx*a] = exp(i q(a) xs[x]),  a = j_lo + n j_hi,
// q(a) = d1 (xi(j_lo) + k_lo) + d2 (xi(j_hi) + k_hi); one job per axis (blockIdx.y) covers the
// ncomp components' points, xs and T component by component
struct PhaseJob {
  const double* xs;
  int nx;
  double d1, k1, d2, k2;
  double2* T;
};
struct PhaseJobs {
  PhaseJob j[3];
};
__global__ void __launch_bounds__(256) k_phase_tables(PhaseJobs jobs, int ncomp, int N) {
  const PhaseJob jb = jobs.j[blockIdx.y];
  const int n = 2 * N, n2 = n * n;
  const long long per = (long long)jb.nx * n2;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < ncomp * per;
       t += (long long)gridDim.x * blockDim.x) {
    const int comp = (int)(t / per), r = (int)(t - comp * per);
    const int x = r % jb.nx, a = r / jb.nx;
    const int jl = a % n, jh = a / n;
    const double xl = (jl < N ? jl : jl - n) + jb.k1, xh = (jh < N ? jh : jh - n) + jb.k2;
    double s, c;
    sincos_phase((jb.d1 * xl + jb.d2 * xh) * jb.xs[(long long)comp * jb.nx + x], &s, &c);
    jb.T[t] = make_double2(c, s);
  }
}

// Batched complex GEMM C(m,n) = sum_k A(m,k) B(k,n) with element strides, FP64 matrix
// instructions: Re and Im of an 8 x 8 block of C are two accumulators, four mma.m8n8k4 per
// block and four k.  A CTA (4 warps, three CTAs per SM) covers up to 48 x 48, each warp a quarter
// of 3 x 3 blocks: 36 matrix instructions for 6 16-byte loads.  The dimensions are cut into
// blocks of 8 and those shared out evenly over the tiles (83 = 11 blocks = 6 + 5), which leaves
// the padding of the last block of 8 only; which warp takes which quarter turns with the tile,
// so that the smaller quarters do not all fall to one scheduler (with 6 warps per CTA, and so
// two of four schedulers doing double work, the GEMMs ran at 62 % of the pipe).  k runs in tiles of 8 through four shared-memory buffers filled by 16-byte cp.async (zeros past the
// edges); rows are padded to 50 elements (a quarter warp's 16-byte loads hit all banks).  With
// gn > 0, B is gathered from the coefficients' natural 6D order (element (a, b + n^2 c), a = j1 + n j4,
// b = j2 + n j5, c = j3 + n j6) instead of a permuted copy.  Bound by the FP64 pipe: the three GEMMs of the direct sum at n = 40, N=5,
// three components (5.0 GFLOP) take 96 / 87 / 64 us (T1 / T2 / u), the pipe 69 % busy; 16 x 16
// threads with 32- and 64-wide register tiles took 144 / 138 / 94 us plus 37 us of permutation.
struct GemmArgs {
  const double2* A;
  const double2* B;
  double2* C;
  int M, N, K;
  long long sam, sak, sbk, sbn, scm, scn;
  long long bA, bB, bC;  // batch strides (blockIdx.z)
  int bdivB = 1;         // B advances by bB every bdivB batch entries
  int gn = 0;            // > 0: B gathered, k = j_a + gn j_(a+3), n = (b, c) pairs alike
};
constexpr int kGThreads = 128;
constexpr int kGKT = 8, kGStages = 4, kGBlk = 6, kGTile = 8 * kGBlk, kGPitch = kGTile + 2;
constexpr int kGElems = kGKT * kGTile / kGThreads;  // tile elements per thread and operand
constexpr int kGMaxK = 14 * 14;  // (2N)^2
constexpr size_t kGSmem = (size_t)kGStages * 2 * kGKT * kGPitch * sizeof(double2) + 2 * kGMaxK * sizeof(long long);

// One k tile of a quarter of IN x JN blocks (IN, JN <= 3; 0: the run-time counts in, jn)
template <int IN, int JN>
__device__ __forceinline__ void zgemm_quarter(const double2* As, const double2* Bs, int in, int jn, int t, int klen,
                                              double (&cr)[3][3][2], double (&ci)[3][3][2]) {
#pragma unroll
  for (int kk = 0; kk < kGKT; kk += 4) {
    if (kk < klen) {
      double2 a[3], b[3];
      double na[3];  // -Im a, by its sign bit: an FP64 instruction here would share the matrix pipe
#pragma unroll
      for (int i = 0; i < 3; ++i)
        if (i < (IN ? IN : in)) {
          a[i] = As[(kk + t) * kGPitch + 8 * i];
          na[i] = __hiloint2double(__double2hiint(a[i].y) ^ (int)0x80000000, __double2loint(a[i].y));
        }
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (j < (JN ? JN : jn)) b[j] = Bs[(kk + t) * kGPitch + 8 * j];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j)
            if (i < (IN ? IN : in) && j < (JN ? JN : jn)) {
              dmma_8x8x4(cr[i][j][0], cr[i][j][1], h ? na[i] : a[i].x, h ? b[j].y : b[j].x);
              dmma_8x8x4(ci[i][j][0], ci[i][j][1], h ? a[i].y : a[i].x, h ? b[j].x : b[j].y);
            }
    }
  }
}

__device__ __forceinline__ void cp_async16(double2* dst, const double2* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 16 : 0)
               : "memory");
}

__global__ void __launch_bounds__(kGThreads, 3) k_zgemm_mma(GemmArgs g) {
  extern __shared__ __align__(16) double2 zg_smem[];
  const double2* A = g.A + g.bA * blockIdx.z;
  const double2* B = g.B + g.bB * (blockIdx.z / g.bdivB);
  double2* Cm = g.C + g.bC * blockIdx.z;
  // this tile's blocks of 8 rows and 8 columns
  const int mb = (g.M + 7) / 8, nb = (g.N + 7) / 8;
  const int mb0 = (int)((long long)blockIdx.x * mb / gridDim.x), mi = (int)((long long)(blockIdx.x + 1) * mb / gridDim.x) - mb0;
  const int nb0 = (int)((long long)blockIdx.y * nb / gridDim.y), nj = (int)((long long)(blockIdx.y + 1) * nb / gridDim.y) - nb0;
  const int m0 = 8 * mb0, n0 = 8 * nb0;
  const int tid = threadIdx.x, lane = tid & 31, gq = lane >> 2, t = lane & 3;
  const bool bNfast = g.gn == 0 && g.sbn == 1;
  // three elements of each operand's 8 x 48 tile per thread: A and n-contiguous B along the 48,
  // k-contiguous B along k
  const double2* asrc[kGElems];
  const double2* bsrc[kGElems];
  int adst[kGElems], bdst[kGElems], akk[kGElems], bkk[kGElems];
  bool ain[kGElems], bin[kGElems];
#pragma unroll
  for (int e = 0; e < kGElems; ++e) {
    const int q = tid + kGThreads * e;
    const int mm = q % kGTile;
    akk[e] = q / kGTile;
    ain[e] = mm < 8 * mi && m0 + mm < g.M;
    asrc[e] = A + (ain[e] ? (m0 + mm) * g.sam : 0);
    adst[e] = akk[e] * kGPitch + mm;
    const int nn = bNfast ? q % kGTile : q / kGKT;
    bkk[e] = bNfast ? q / kGTile : q % kGKT;
    bin[e] = nn < 8 * nj && n0 + nn < g.N;
    long long off = 0;
    if (bin[e]) {
      if (g.gn > 0) {
        const long long n = g.gn, n2 = n * n, b = (n0 + nn) % n2, c = (n0 + nn) / n2;
        off = n * (b % n) + n2 * (c % n) + n2 * n2 * (b / n) + n2 * n2 * n * (c / n);
      } else {
        off = (n0 + nn) * g.sbn;
      }
    }
    bsrc[e] = B + off;
    bdst[e] = bkk[e] * kGPitch + nn;
  }
  // offsets of the k of either operand
  long long* aoff = reinterpret_cast<long long*>(zg_smem + kGStages * 2 * kGKT * kGPitch);
  long long* boff = aoff + kGMaxK;
  for (int k = tid; k < g.K; k += kGThreads) {
    aoff[k] = k * g.sak;
    boff[k] = g.gn > 0 ? k % g.gn + (long long)g.gn * g.gn * g.gn * (k / g.gn) : k * g.sbk;
  }
  __syncthreads();
  const int ns = (g.K + kGKT - 1) / kGKT;
  auto issue = [&](int s) {
    if (s < ns) {
      double2* As = zg_smem + (s % kGStages) * 2 * kGKT * kGPitch;
      double2* Bs = As + kGKT * kGPitch;
#pragma unroll
      for (int e = 0; e < kGElems; ++e) {
        const int ka = s * kGKT + akk[e], kb = s * kGKT + bkk[e];
        const bool ia = ain[e] && ka < g.K, ib = bin[e] && kb < g.K;
        cp_async16(As + adst[e], asrc[e] + (ia ? aoff[ka] : 0), ia);
        cp_async16(Bs + bdst[e], bsrc[e] + (ib ? boff[kb] : 0), ib);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // this warp's quarter: row blocks [ib, ib + in), column blocks [jb, jb + jn)
  constexpr int Q = kGBlk / 2;
  const int role = ((tid >> 5) + blockIdx.x + blockIdx.y + blockIdx.z) & 3;
  const int ib = (role & 1) ? (mi + 1) / 2 : 0, in = (role & 1) ? mi / 2 : (mi + 1) / 2;
  const int jb = (role & 2) ? (nj + 1) / 2 : 0, jn = (role & 2) ? nj / 2 : (nj + 1) / 2;
  double cr[Q][Q][2], ci[Q][Q][2];
#pragma unroll
  for (int i = 0; i < Q; ++i)
#pragma unroll
    for (int j = 0; j < Q; ++j) cr[i][j][0] = cr[i][j][1] = ci[i][j][0] = ci[i][j][1] = 0.0;
#pragma unroll
  for (int s = 0; s < kGStages - 1; ++s) issue(s);
  for (int s = 0; s < ns; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kGStages - 2) : "memory");
    __syncthreads();  // tile s has landed for every thread; tile s - 1 has been read out
    issue(s + kGStages - 1);
    const double2* As = zg_smem + (s % kGStages) * 2 * kGKT * kGPitch + 8 * ib + gq;
    const double2* Bs = zg_smem + ((s % kGStages) * 2 + 1) * kGKT * kGPitch + 8 * jb + gq;
    const int klen = g.K - s * kGKT;
    if (in == 3 && jn == 3) zgemm_quarter<3, 3>(As, Bs, in, jn, t, klen, cr, ci);
    else if (in == 3 && jn == 2) zgemm_quarter<3, 2>(As, Bs, in, jn, t, klen, cr, ci);
    else if (in == 2 && jn == 3) zgemm_quarter<2, 3>(As, Bs, in, jn, t, klen, cr, ci);
    else if (in == 2 && jn == 2) zgemm_quarter<2, 2>(As, Bs, in, jn, t, klen, cr, ci);
    else zgemm_quarter<0, 0>(As, Bs, in, jn, t, klen, cr, ci);
  }
#pragma unroll
  for (int i = 0; i < Q; ++i)
#pragma unroll
    for (int j = 0; j < Q; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m = m0 + 8 * (ib + i) + gq, n = n0 + 8 * (jb + j) + 2 * t + h;
        if (i < in && j < jn && m < g.M && n < g.N)
          Cm[m * g.scm + n * g.scn] = make_double2(cr[i][j][h], ci[i][j][h]);
      }
}

int zgemm(const GemmArgs& g, int batch, cudaStream_t s) {
  static DeviceOnce once;
  FAME_TRY(ensure_smem(k_zgemm_mma, kGSmem, once));
  if (g.K > kGMaxK) return fail(FAME_ERR_UNSUPPORTED, "zgemm: contraction too long");
  auto tiles = [](int d) { return ((d + 7) / 8 + kGBlk - 1) / kGBlk; };
  // 65535 tiles of columns per launch; only the last two GEMMs of long axes have more (a gathered
  // B has (2N)^4 columns)
  constexpr int kMaxN = 65535 * kGTile;
  for (long long n0 = 0; n0 < g.N; n0 += kMaxN) {
    GemmArgs part = g;
    part.N = (int)std::min<long long>(kMaxN, g.N - n0);
    part.B += n0 * g.sbn;
    part.C += n0 * g.scn;
    k_zgemm_mma<<<dim3(tiles(part.M), tiles(part.N), batch), kGThreads, kGSmem, s>>>(part);
    ::fame::count_launch();
  }
  FAME_CUDA_TRY(cudaGetLastError());
  return FAME_OK;
}

// ------------------------------------------------------------------ Taylor
// centers: per block the midpoint of the bounding box of its points, in two steps so that a
// few large blocks still fill the GPU: box[(b * chunks + x)] = {lo, hi} of every chunks-th
// run of 256 points of block b, then the boxes joined (one CTA per block needed 75 us at one
// block of 19,683 points, its loads being one dependent pair after the other).
constexpr int kBoxThreads = 256;
__global__ void __launch_bounds__(kBoxThreads) k_block_boxes(const double* __restrict__ R, long long M,
                                                            const long long* __restrict__ ptr,
                                                            const long long* __restrict__ ids, double* __restrict__ box) {
  __shared__ double red[kBoxThreads / 32][6];
  const int b = blockIdx.y;
  double v[6] = {1e300, 1e300, 1e300, -1e300, -1e300, -1e300};
  for (long long t = ptr[b] + (long long)blockIdx.x * kBoxThreads + threadIdx.x; t < ptr[b + 1];
       t += (long long)gridDim.x * kBoxThreads) {
    const long long i = ids[t];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double r = R[d * M + i];
      v[d] = fmin(v[d], r);
      v[3 + d] = fmax(v[3 + d], r);
    }
  }
#pragma unroll
  for (int d = 0; d < 6; ++d) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double w = __shfl_xor_sync(0xffffffffu, v[d], o);
      v[d] = d < 3 ? fmin(v[d], w) : fmax(v[d], w);
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][d] = v[d];
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    const int d = threadIdx.x;
    double w = red[0][d];
    for (int k = 1; k < kBoxThreads / 32; ++k) w = d < 3 ? fmin(w, red[k][d]) : fmax(w, red[k][d]);
    box[((long long)b * gridDim.x + blockIdx.x) * 6 + d] = w;
  }
}
__global__ void k_block_centers(const double* __restrict__ box, int chunks, int nB, const double* __restrict__ fixed,
                                double* __restrict__ centers) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 3 * nB) return;
  const int b = t / 3, d = t % 3;
  double lo = 1e300, hi = -1e300;
  for (int x = 0; x < chunks; ++x) {
    lo = fmin(lo, box[((long long)b * chunks + x) * 6 + d]);
    hi = fmax(hi, box[((long long)b * chunks + x) * 6 + 3 + d]);
  }
  centers[t] = fixed ? fixed[d] : 0.5 * (lo + hi);
}
// CTAs per block of points for kernels over (chunk, block): about two waves of the GPU in
// all, no more than the average block has runs of 256 points
static int block_chunks(long long M, int nB) {
  const long long runs = std::max<long long>(1, (M / nB + 255) / 256);
  const long long want = std::max<long long>(1, 16LL * num_sms() / nB);
  return (int)std::min<long long>(runs, want);
}

constexpr int kTaySub = 64;     // modes staged per sub-chunk
constexpr int kTayChunk = 4096; // modes per CTA at most
constexpr int kMaxP = 12;
// partial[(chunk * nB + b) * L + alpha] = sum_{j in chunk} c_j e^{i q_j.r_c} q_j^alpha
__global__ void __launch_bounds__(512) k_taylor_moments(const double2* __restrict__ c, const double* __restrict__ Q,
                                                       long long NF, const double* __restrict__ centers,
                                                       const int* __restrict__ alist, int L, int p, int nB,
                                                       long long per_chunk, double2* __restrict__ partial) {
  __shared__ double2 w[kTaySub];
  __shared__ double pw[3][kTaySub][kMaxP + 1];
  const int chunk = blockIdx.x, b = blockIdx.y;
  const double cx = centers[3 * b], cy = centers[3 * b + 1], cz = centers[3 * b + 2];
  const int al = threadIdx.x;
  const bool act = al < L;
  const int a1 = act ? alist[3 * al] : 0, a2 = act ? alist[3 * al + 1] : 0, a3 = act ? alist[3 * al + 2] : 0;
  double ar = 0.0, ai = 0.0;
  const long long j0c = chunk * per_chunk;
  const long long j1c = std::min<long long>(NF, j0c + per_chunk);
  for (long long j0 = j0c; j0 < j1c; j0 += kTaySub) {
    const int nj = (int)std::min<long long>(kTaySub, j1c - j0);
    __syncthreads();
    for (int t = threadIdx.x; t < nj; t += blockDim.x) {
      const long long j = j0 + t;
      const double qx = Q[j], qy = Q[NF + j], qz = Q[2 * NF + j];
      double s, co;
      sincos(qx * cx + qy * cy + qz * cz, &s, &co);
      const double2 cj = c[j];
      w[t] = make_double2(cj.x * co - cj.y * s, cj.x * s + cj.y * co);
      double px = 1.0, py = 1.0, pz = 1.0;
      for (int k = 0; k <= p; ++k) {
        pw[0][t][k] = px;
        pw[1][t][k] = py;
        pw[2][t][k] = pz;
        px *= qx;
        py *= qy;
        pz *= qz;
      }
    }
    __syncthreads();
    if (act) {
      for (int t = 0; t < nj; ++t) {
        const double mono = pw[0][t][a1] * pw[1][t][a2] * pw[2][t][a3];
        ar += w[t].x * mono;
        ai += w[t].y * mono;
      }
    }
  }
  if (act) partial[((long long)chunk * nB + b) * L + al] = make_double2(ar, ai);
}

// The same moments as FP64 matrix products: for a block of 8 WM centers the rows are Re and Im
// of c_j e^{i q_j.r_b}, the columns the monomials, the contraction the modes.  A CTA (16 warps,
// one CTA per SM) owns one slice of the modes, one block of centers and at most 128 / WM * NT
// columns.  Per stage of 32 modes all warps write both operands into shared memory (one sine
// and cosine per mode and center; the monomials in runs of four powers of qz, two products per
// mode and run and one per monomial, each made once per CTA), then all multiply them with FP64 mma.m8n8k4, WM warps along the rows and
// 16 / WM along the columns.  The two phases alternate on purpose: FP64 scalar and matrix
// instructions share the pipe and disturb each other, so generator warps working beside the
// multiplying ones (two stages handed over through barriers) took 4.3 ms per component where
// this takes 2.94 ms, evaluation included.  Operand rows are padded to 36 doubles (the fragment loads of a half warp hit 16
// different banks).  A slice is at most 4096 modes, so that the accumulation error stays that
// of k_taylor_moments' chunks.  Bound by the FP64 pipe: 2 * 64 * 286 * 10^6 FMA at N=5, p=10,
// 64 centers are 2.0 ms at the measured GEMM rate, the operands a quarter of that on top;
// k_taylor_moments, which rebuilds each monomial for every center, takes 16.0 ms.
constexpr int kMmaModes = 32;  // modes per stage
constexpr int kMmaPitch = kMmaModes + 4;
constexpr long long kMmaSlice = 4096;

// NT: column tiles of 8 per warp; blockIdx.z: column group of 128 / WM * NT
template <int NT, int WM>
__global__ void __launch_bounds__(512, 1)
k_taylor_moments_mma(const double2* __restrict__ c, const double* __restrict__ Q, long long NF,
                     const double* __restrict__ centers, const int* __restrict__ runs, int L, int nB,
                     long long per_slice, double2* __restrict__ partial) {
  extern __shared__ double mom_smem[];
  constexpr int kCen = 8 * WM, cols = 128 / WM * NT, kPow = 3 * (kMaxP + 1) * kMmaModes;
  constexpr int kPerWarp = (kCen + 15) / 16;  // centers per warp
  double* As = mom_smem;                      // [16 WM][kMmaPitch]
  double* Bs = As + 2 * kCen * kMmaPitch;     // [cols][kMmaPitch]
  double* pw = Bs + cols * kMmaPitch;         // two stages of [3][kMaxP + 1][32] powers
  int* dsc = reinterpret_cast<int*>(pw + 2 * kPow);  // [cols]: this column group's runs (moment_runs)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b0 = blockIdx.y * kCen, c0 = blockIdx.z * cols;
  const int nbl = min(kCen, nB - b0), nrun = runs[blockIdx.z + 1] - runs[blockIdx.z];
  const long long j0 = blockIdx.x * per_slice, j1 = min(NF, j0 + per_slice);
  const int nst = (int)((j1 - j0 + kMmaModes - 1) / kMmaModes);
  double cx[kPerWarp], cy[kPerWarp], cz[kPerWarp];  // centers warp, warp + 16
#pragma unroll
  for (int u = 0; u < kPerWarp; ++u) {
    const int b = b0 + min(warp + 16 * u, nbl - 1);
    cx[u] = centers[3 * b];
    cy[u] = centers[3 * b + 1];
    cz[u] = centers[3 * b + 2];
  }
  // rows past the last center and columns past L stay zero
  for (int i = threadIdx.x; i < (2 * kCen + cols) * kMmaPitch; i += 512) mom_smem[i] = 0.0;
  for (int i = threadIdx.x; i < nrun; i += 512) dsc[i] = runs[runs[blockIdx.z] + i];
  // powers of one wave-vector component of a stage's modes (warps 0..2: x, y, z)
  auto powers = [&](int it) {
    const long long j = j0 + (long long)it * kMmaModes + lane;
    double v[kMaxP + 1];
    v[0] = 1.0;
    v[1] = j < j1 ? Q[warp * NF + j] : 0.0;
#pragma unroll
    for (int k = 2; k <= kMaxP; ++k) v[k] = v[k / 2] * v[k - k / 2];
    double* row = pw + (it & 1) * kPow + warp * (kMaxP + 1) * kMmaModes + lane;
#pragma unroll
    for (int k = 0; k <= kMaxP; ++k) row[k * kMmaModes] = v[k];
  };
  double nqx = 0.0, nqy = 0.0, nqz = 0.0;  // this lane's mode of the next stage
  double2 ncj = make_double2(0.0, 0.0);
  auto fetch = [&](long long j) {
    const bool in = j < j1;
    nqx = in ? Q[j] : 0.0;
    nqy = in ? Q[NF + j] : 0.0;
    nqz = in ? Q[2 * NF + j] : 0.0;
    ncj = in ? c[j] : make_double2(0.0, 0.0);  // c = 0 past the slice: no contribution
  };
  const int wm = warp % WM, wn = warp / WM;  // this warp multiplies rows 16 wm, columns 8 NT wn
  const int g = lane >> 2, t = lane & 3;
  const double* ap = As + (16 * wm + g) * kMmaPitch + t;
  const double* bp = Bs + (8 * NT * wn + g) * kMmaPitch + t;
  double acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int h = 0; h < 4; ++h) acc[i][h] = 0.0;
  fetch(j0 + lane);
  if (warp < 3) powers(0);
  __syncthreads();
  for (int it = 0; it < nst; ++it) {
    const double qx = nqx, qy = nqy, qz = nqz;
    const double2 cj = ncj;
    fetch(j0 + (long long)(it + 1) * kMmaModes + lane);
#pragma unroll
    for (int u = 0; u < kPerWarp; ++u) {
      const int bl = warp + 16 * u;
      if (bl < nbl) {
        double s, co;
        sincos_phase(qx * cx[u] + qy * cy[u] + qz * cz[u], &s, &co);
        As[(2 * bl) * kMmaPitch + lane] = cj.x * co - cj.y * s;
        As[(2 * bl + 1) * kMmaPitch + lane] = cj.x * s + cj.y * co;
      }
    }
    const double* pt = pw + (it & 1) * kPow + lane;
    const double z2 = qz * qz, z3 = z2 * qz;
#pragma unroll 2
    for (int r = warp; r < nrun; r += 16) {
      const int d = dsc[r];
      const double m0 = pt[((d >> 10) & 15) * kMmaModes] * pt[(kMaxP + 1 + ((d >> 14) & 15)) * kMmaModes] *
                        pt[(2 * (kMaxP + 1) + 4 * ((d >> 18) & 3)) * kMmaModes];
      double* row = Bs + ((d & 1023) - 4) * kMmaPitch + lane;
      if (d & 1 << 20) row[0] = m0;
      if (d & 2 << 20) row[kMmaPitch] = m0 * qz;
      if (d & 4 << 20) row[2 * kMmaPitch] = m0 * z2;
      if (d & 8 << 20) row[3 * kMmaPitch] = m0 * z3;
    }
    if (warp < 3) powers(it + 1);  // into the other table; past the last stage unused
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kMmaModes; kk += 4) {
      const double a0 = ap[kk], a1 = ap[8 * kMmaPitch + kk];
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        const double b = bp[8 * i * kMmaPitch + kk];
        dmma_8x8x4(acc[i][0], acc[i][1], a0, b);
        dmma_8x8x4(acc[i][2], acc[i][3], a1, b);
      }
    }
    __syncthreads();
  }
  // accumulator rows 2 bl, 2 bl + 1 (Re, Im of center bl) sit in lanes g, g + 1 of the quads:
  // even quads write the pair
#pragma unroll
  for (int i = 0; i < NT; ++i) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const double im = __shfl_down_sync(0xffffffffu, acc[i][h], 4);
      const int bl = (16 * wm + g + (h >= 2 ? 8 : 0)) / 2, col = c0 + 8 * (NT * wn + i) + 2 * t + (h & 1);
      if ((g & 1) == 0 && bl < nbl && col < L)
        partial[((long long)blockIdx.x * nB + b0 + bl) * L + col] = make_double2(acc[i][h], im);
    }
  }
}

// 32 centers per CTA halve the monomial work per product against 16, and those against 8, while
// few enough rows stay empty
static int moments_mma_wm(int nB) { return nB <= 8 ? 1 : nB <= 16 ? 2 : 4; }
// Column groups: two where one CTA's columns would not fit its registers (WM = 4, p > 10)
static int moments_mma_groups(int L, int wm) { return wm == 4 && L > 288 ? 2 : 1; }

// The monomials of the column groups (columns [g cols, (g + 1) cols) of the list) as runs of up
// to four consecutive a3 at fixed (a1, a2), the first a multiple of four: column of that first
// one relative to the group + 4 (10 bits) | a1 (4) | a2 (4) | a3 / 4 (2) | which of the four
// belong to the group (4).  out: groups + 1 offsets into itself, then the runs.
static void moment_runs(const std::vector<int>& al, int L, int cols, int groups, std::vector<int>& out) {
  out.assign(groups + 1, groups + 1);
  for (int g = 0; g < groups; ++g) {
    for (int c = g * cols; c < std::min(L, (g + 1) * cols);) {
      const int a1 = al[3 * c], a2 = al[3 * c + 1], base = al[3 * c + 2] & ~3;
      int d = (c - g * cols - (al[3 * c + 2] - base) + 4) | a1 << 10 | a2 << 14 | (base / 4) << 18;
      for (; c < std::min(L, (g + 1) * cols) && al[3 * c] == a1 && al[3 * c + 1] == a2 && (al[3 * c + 2] & ~3) == base; ++c)
        d |= 1 << (20 + al[3 * c + 2] - base);
      out.push_back(d);
    }
    out[g + 1] = (int)out.size();
  }
}

template <int NT, int WM>
int launch_moments_mma(const double2* c, const double* Q, long long NF, const double* centers, const int* runs, int L,
                       int nB, int groups, int nslices, long long per_slice, double2* partial, cudaStream_t s) {
  constexpr size_t smem = (size_t)(16 * WM + 128 / WM * NT) * kMmaPitch * sizeof(double) +
                          6 * (kMaxP + 1) * kMmaModes * sizeof(double) + 128 / WM * NT * sizeof(int);
  static_assert(smem <= 227 * 1024, "operand stage");
  static DeviceOnce once;
  FAME_TRY(ensure_smem(k_taylor_moments_mma<NT, WM>, smem, once));
  k_taylor_moments_mma<NT, WM><<<dim3(nslices, (nB + 8 * WM - 1) / (8 * WM), groups), 512, smem, s>>>(
      c, Q, NF, centers, runs, L, nB, per_slice, partial);
  ::fame::count_launch();
  FAME_CUDA_TRY(cudaGetLastError());
  return FAME_OK;
}

// Slices of the modes: whole waves of one CTA per SM over (slice, center block, column group).
static void moments_mma_slices(long long NF, int nB, int L, int* nslices, long long* per_slice) {
  const int wm = moments_mma_wm(nB);
  const long long tiles = (long long)((nB + 8 * wm - 1) / (8 * wm)) * moments_mma_groups(L, wm);
  moment_slices(NF, tiles, num_sms(), kMmaModes, kMmaSlice, nslices, per_slice);
}

// Column tiles per warp: the smallest compiled count that holds the group's columns
static int moments_mma_nt(int L, int wm) {
  const int groups = moments_mma_groups(L, wm), tiles = ((L + 7) / 8 + groups - 1) / groups;
  const int nt = (tiles * wm + 15) / 16;
  if (wm == 1) return nt;              // <= 4
  if (wm == 2) return nt <= 5 ? nt : 8;
  return nt == 5 ? 6 : nt;             // <= 9
}

static int taylor_moments_mma(const double2* c, const double* Q, long long NF, const double* centers, const int* runs,
                              int L, int nB, int nslices, long long per_slice, double2* partial, cudaStream_t s) {
  const int wm = moments_mma_wm(nB), groups = moments_mma_groups(L, wm), nt = moments_mma_nt(L, wm);
#define FAME_MOM(NT, WM)       \
  if (nt == NT && wm == WM)    \
  return launch_moments_mma<NT, WM>(c, Q, NF, centers, runs, L, nB, groups, nslices, per_slice, partial, s)
  FAME_MOM(1, 1);
  FAME_MOM(2, 1);
  FAME_MOM(3, 1);
  FAME_MOM(4, 1);
  FAME_MOM(1, 2);
  FAME_MOM(2, 2);
  FAME_MOM(3, 2);
  FAME_MOM(4, 2);
  FAME_MOM(5, 2);
  FAME_MOM(8, 2);
  FAME_MOM(1, 4);
  FAME_MOM(2, 4);
  FAME_MOM(3, 4);
  FAME_MOM(4, 4);
  FAME_MOM(6, 4);
  FAME_MOM(7, 4);
  FAME_MOM(8, 4);
  FAME_MOM(9, 4);
#undef FAME_MOM
  return fail(FAME_ERR_UNSUPPORTED, "too many Taylor terms");
}

// gamma[b*L + a] = coef[a] * sum_chunks partial (fixed order): eight threads per value take
// every eighth chunk, so that few values do not leave the sum to one chain of loads
__global__ void __launch_bounds__(256) k_taylor_reduce(const double2* __restrict__ partial, int nChunks, int nB, int L,
                                                       const double2* __restrict__ coef, double2* __restrict__ gamma) {
  __shared__ double2 red[8][32];
  const long long total = (long long)nB * L, t = blockIdx.x * 32LL + threadIdx.x % 32;
  const int y = threadIdx.x / 32;
  double ar = 0.0, ai = 0.0;
  if (t < total)
    for (int ch = y; ch < nChunks; ch += 8) {
      const double2 v = partial[ch * total + t];
      ar += v.x;
      ai += v.y;
    }
  red[y][threadIdx.x % 32] = make_double2(ar, ai);
  __syncthreads();
  if (y != 0 || t >= total) return;
  for (int k = 1; k < 8; ++k) {
    ar += red[k][threadIdx.x].x;
    ai += red[k][threadIdx.x].y;
  }
  const double2 cf = coef[t % L];
  gamma[t] = make_double2(cf.x * ar - cf.y * ai, cf.x * ai + cf.y * ar);
}

// u(ids[t]) = sum_a gamma[b, a] (r - r_c)^a for the block's points, by Horner's rule along
// each axis (the list runs a1 outer, a3 inner, so it is walked backwards): two FMA per term
// and no power tables.  Bound by the FP64 pipe (571,787 points at p = 10: 0.42 GFMA, 23 us at
// its peak); per-thread tables of powers, whose run-time indices put them in local memory, took
// 212 us.
__global__ void __launch_bounds__(256) k_taylor_eval(const double* __restrict__ R, long long M,
                                                    const long long* __restrict__ ptr, const long long* __restrict__ ids,
                                                    const double* __restrict__ centers, const double2* __restrict__ gamma,
                                                    int L, int p, double2* __restrict__ u) {
  extern __shared__ double2 sg[];
  const int b = blockIdx.y;
  for (int t = threadIdx.x; t < L; t += blockDim.x) sg[t] = gamma[(long long)b * L + t];
  __syncthreads();
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long t = ptr[b] + (long long)blockIdx.x * blockDim.x + threadIdx.x; t < ptr[b + 1]; t += stride) {
    const long long i = ids[t];
    const double dx = R[i] - centers[3 * b], dy = R[M + i] - centers[3 * b + 1],
                 dz = R[2 * M + i] - centers[3 * b + 2];
    double ur = 0.0, ui = 0.0;
    int a = L - 1;
    for (int s1 = 0; s1 <= p; ++s1) {  // a1 = p - s1: a2 from s1 down
      double tr = 0.0, ti = 0.0;
      for (int s2 = 0; s2 <= s1; ++s2) {  // a2 = s1 - s2: a3 from s2 down
        double vr = 0.0, vi = 0.0;
        for (int s3 = 0; s3 <= s2; ++s3, --a) {
          const double2 gm = sg[a];
          vr = fma(vr, dz, gm.x);
          vi = fma(vi, dz, gm.y);
        }
        tr = fma(tr, dy, vr);
        ti = fma(ti, dy, vi);
      }
      ur = fma(ur, dx, tr);
      ui = fma(ui, dx, ti);
    }
    u[i] = make_double2(ur, ui);
  }
}

}  // namespace fame

using namespace fame;

extern "C" {

int fame_reconstruct_direct(fame_ctx* ctx, const void* coeff, const double* qModes, long long NF,
                            const double* rPoints, long long M, void* u) {
  if (!ctx || !coeff || !qModes || !rPoints || !u || NF <= 0 || M < 0)
    return fail(FAME_ERR_INVALID, "reconstruct_direct arguments");
  if (M == 0) return FAME_OK;
  k_direct_sum<<<(int)((M + kDirectPts - 1) / kDirectPts), kDirectPts, 0, ctx->stream>>>(
      (const double2*)coeff, qModes, NF, rPoints, M, (double2*)u);
  ::fame::count_launch();
  FAME_CUDA_TRY(cudaGetLastError());
  return FAME_OK;
}

// The factorised direct sum for ncomp components at once (component-stacked coeff, axes
// and u; equal grid sizes): each of the three GEMMs is one launch batched over the
// components (and, for the second, over its contraction slices), so the launches are
// ncomp times larger.  No host synchronisation: the results are ordered on the stream.
static int direct_grid_impl(fame_basis* bs, const void* coeff, int ncomp, const double* xs, int nx, const double* ys,
                            int ny, const double* zs, int nz, void* u, bool tc) {
  if (!bs || !coeff || !xs || !ys || !zs || !u || nx <= 0 || ny <= 0 || nz <= 0 || ncomp < 1 || ncomp > 3)
    return fail(FAME_ERR_INVALID, "reconstruct_direct_grid arguments");
  const double* P = bs->P;  // column-major 6 x 3
  for (int l = 0; l < 6; ++l)
    for (int c = 0; c < 3; ++c)
      if (l % 3 != c && P[c * 6 + l] != 0.0)
        return fail(FAME_ERR_UNSUPPORTED, "factorised reconstruction needs an axis-block cut matrix [diag; diag]");
  const int N = bs->N, n = 2 * N;
  const long long n2 = (long long)n * n, NF = bs->NF;
  if ((long long)ncomp * n2 > 65535) return fail(FAME_ERR_UNSUPPORTED, "reconstruct_direct_grid: too many slices");
  cudaStream_t s = bs->ctx->stream;
  // workspace pieces (per component, consecutive): phase tables, then the two GEMM
  // intermediates in FP64 or, on the tensor cores, the split operand panels (zgemm_tc.cu): Tx
  // (A of T1), coefficients (B of T1), Ty (B of T2), Tz (B of u), split together, and the
  // intermediates' own panels
  const int in2 = (int)n2;
  const ZChainSizes zc = zchain_sizes(nx, ny, in2, ncomp);
  ZPanelJob jTx{nullptr, 1, nx, (long long)nx * n2, nx, in2, ncomp, true, 0, nullptr};
  ZPanelJob jCp{nullptr, 0, 0, NF, (int)(n2 * n2), in2, ncomp, false, in2 * zc.cp, nullptr, in2 * zc.cp, n};
  ZPanelJob jTy{nullptr, 1, ny, (long long)ny * n2, ny, in2, ncomp, false, ny, nullptr};
  ZPanelJob jTz{nullptr, 1, nz, (long long)nz * n2, nz, in2, ncomp, false, nz, nullptr};
  auto carve = [&](Carve& cv, double2** Tx, double2** Ty, double2** Tz, double2** T1, double2** T2,
                   unsigned char** P1, unsigned char** P2) {
    *Tx = cv.take<double2>((size_t)ncomp * nx * n2);
    *Ty = cv.take<double2>((size_t)ncomp * ny * n2);
    *Tz = cv.take<double2>((size_t)ncomp * nz * n2);
    if (tc) {  // panel buffers start on 1024-byte boundaries of the actual addresses (sizes
               // are multiples of 1024); the sizing pass reserves the largest padding
      const uintptr_t at = reinterpret_cast<uintptr_t>(cv.base) + cv.used;
      cv.used += cv.base ? (1024 - (at & 1023)) & 1023 : 1024;
      for (ZPanelJob* j : {&jTx, &jCp, &jTy, &jTz}) {
        j->out = cv.take<unsigned char>((zpanel_bytes(*j) + 1023) / 1024 * 1024);
      }
      *P1 = cv.take<unsigned char>((size_t)ncomp * zc.bytes1);
      *P2 = cv.take<unsigned char>((size_t)ncomp * zc.bytes2);
      *T1 = *T2 = nullptr;
    } else {
      *T1 = cv.take<double2>((size_t)ncomp * nx * n2 * n2);
      *T2 = cv.take<double2>((size_t)ncomp * nx * ny * n2);
      *P1 = *P2 = nullptr;
    }
  };
  double2 *Tx, *Ty, *Tz, *T1, *T2;
  unsigned char *P1, *P2;
  Carve size_only;
  carve(size_only, &Tx, &Ty, &Tz, &T1, &T2, &P1, &P2);
  void* ws = nullptr;
  int st = ctx_workspace(bs->ctx, size_only.used, &ws);
  Carve cv;
  cv.base = static_cast<char*>(ws);
  carve(cv, &Tx, &Ty, &Tz, &T1, &T2, &P1, &P2);
  const double* k = bs->info.kLift;
  if (st == FAME_OK) {
    const PhaseJobs jobs{{{xs, nx, P[0], k[0], P[3], k[3], Tx},
                          {ys, ny, P[6 + 1], k[1], P[6 + 4], k[4], Ty},
                          {zs, nz, P[12 + 2], k[2], P[12 + 5], k[5], Tz}}};
    k_phase_tables<<<dim3(rblocks((long long)ncomp * std::max({nx, ny, nz}) * n2), 3), 256, 0, s>>>(jobs, ncomp, N);
    ::fame::count_launch();
    // T1[x, (b,c)] = sum_a Tx[x, a] Cp[a, (b,c)]                   (batched over components)
    GemmArgs g1{Tx, (const double2*)coeff, T1, nx, (int)(n2 * n2), (int)n2, 1, nx, 1, n2, 1, nx,
                (long long)nx * n2, NF, (long long)nx * n2 * n2, 1, n};
    // T2[x, y, c] = sum_b T1[x, b, c] Ty[y, b]   (batched over components x c; Ty per component)
    GemmArgs g2{T1, Ty, T2, nx, ny, (int)n2, 1, nx, ny, 1, 1, nx, (long long)nx * n2, (long long)ny * n2,
                (long long)nx * ny, (int)n2};
    // u[(x,y), z] = sum_c T2[(x,y), c] Tz[z, c]                    (batched over components)
    GemmArgs g3{T2, Tz, (double2*)u, nx * ny, nz, (int)n2, 1, (long long)nx * ny, nz, 1, 1, (long long)nx * ny,
                (long long)nx * ny * n2, (long long)nz * n2, (long long)nx * ny * nz};
    const GemmArgs* gs[3] = {&g1, &g2, &g3};
    const int batches[3] = {ncomp, (int)(ncomp * n2), ncomp};
    if (!tc) {
      for (int t = 0; t < 3 && st == FAME_OK; ++t) st = zgemm(*gs[t], batches[t], s);
    } else {
      jTx.src = Tx;
      jCp.src = (const double2*)coeff;
      jTy.src = Ty;
      jTz.src = Tz;
      const ZPanelJob first[4] = {jTx, jCp, jTy, jTz};
      st = zsplit_panels(first, 4, s);
      if (st == FAME_OK)
        st = zchain_3xtf32(jTx.out, jCp.out, jTy.out, jTz.out, P1, P2, (double2*)u, nx, ny, nz, in2, ncomp, s);
    }
  }
  return st;
}

int fame_reconstruct_direct_grid(fame_basis* bs, const void* coeff, const double* xs, int nx, const double* ys, int ny,
                                 const double* zs, int nz, void* u) {
  return direct_grid_impl(bs, coeff, 1, xs, nx, ys, ny, zs, nz, u, false);
}

int fame_reconstruct_direct_grid_3xtf32(fame_basis* bs, const void* coeff, const double* xs, int nx, const double* ys,
                                        int ny, const double* zs, int nz, void* u) {
  return direct_grid_impl(bs, coeff, 1, xs, nx, ys, ny, zs, nz, u, true);
}

int fame_reconstruct_direct_grid_fields(fame_basis* bs, const void* coeff, int ncomp, const double* xs, int nx,
                                        const double* ys, int ny, const double* zs, int nz, int tensor_cores,
                                        void* u) {
  return direct_grid_impl(bs, coeff, ncomp, xs, nx, ys, ny, zs, nz, u, tensor_cores != 0);
}

}  // extern "C"

namespace fame {

// Multi-center Taylor reconstruction (exp2/taylor_on_blocks_exp3.m:1-97); the block
// moments either in FP64 on the CUDA cores or as 3xTF32 products on the tensor cores
// (taylor_tc.cu).
// Whether the nB centers (x, y, z per block) form a tensor grid in block order
// b = i + m1 (j + m2 k) with axis values X[i], Y[j], Z[k] (exact equality); on success
// grid.m1..m3 are set and ax = [X, Y, Z].
static bool tensor_grid_of(const std::vector<double>& c, int nB, TaylorTcGrid& grid, std::vector<double>& ax) {
  int m1 = 1, m2 = 1;
  while (m1 < nB && c[3 * m1 + 1] == c[1] && c[3 * m1 + 2] == c[2]) ++m1;
  while (m1 * m2 < nB && c[3 * (m1 * m2) + 2] == c[2]) ++m2;
  if (nB % (m1 * m2) != 0) return false;
  const int m3 = nB / (m1 * m2);
  if (m1 + m2 + m3 > kTaylorTcMaxAxis) return false;
  for (int b = 0; b < nB; ++b) {
    const int i = b % m1, j = (b / m1) % m2, k = b / (m1 * m2);
    if (c[3 * b] != c[3 * i] || c[3 * b + 1] != c[3 * (m1 * j) + 1] || c[3 * b + 2] != c[3 * (m1 * m2 * k) + 2])
      return false;
  }
  ax.clear();
  for (int i = 0; i < m1; ++i) ax.push_back(c[3 * i]);
  for (int j = 0; j < m2; ++j) ax.push_back(c[3 * (m1 * j) + 1]);
  for (int k = 0; k < m3; ++k) ax.push_back(c[3 * (m1 * m2 * k) + 2]);
  grid.m1 = m1;
  grid.m2 = m2;
  grid.m3 = m3;
  return true;
}

static int taylor_impl(fame_ctx* ctx, const void* coeff, const double* qModes, long long NF, const double* rPoints,
                       long long M, int p, const long long* blockPtr, const long long* blockIds, int nBlocks,
                       const double* fixedCenter, void* u, bool tc) {
  if (!ctx || !coeff || !qModes || !rPoints || !u || !blockPtr || !blockIds || NF <= 0 || M < 0 ||
      nBlocks < 1)
    return fail(FAME_ERR_INVALID, "taylor_on_blocks arguments");
  if (p < 0 || p > kMaxP) return fail(FAME_ERR_UNSUPPORTED, "Taylor order must be in [0,12]");
  // multi-indices |a| <= p, a1 outer, a3 inner (exp2/build_multi_index_list_3d_exp3.m:3-14)
  double fact[kMaxP + 1] = {1.0};  // exact up to 12!
  for (int k = 1; k <= kMaxP; ++k) fact[k] = fact[k - 1] * k;
  std::vector<int> al;
  std::vector<double2> cf;
  for (int a1 = 0; a1 <= p; ++a1)
    for (int a2 = 0; a2 <= p - a1; ++a2)
      for (int a3 = 0; a3 <= p - a1 - a2; ++a3) {
        al.push_back(a1);
        al.push_back(a2);
        al.push_back(a3);
        const int s = a1 + a2 + a3;
        const double mag = 1.0 / (fact[a1] * fact[a2] * fact[a3]);
        const double re[4] = {1, 0, -1, 0}, im[4] = {0, 1, 0, -1};  // i^s
        cf.push_back(make_double2(mag * re[s % 4], mag * im[s % 4]));
      }
  const int L = (int)cf.size();
  if (L > 512) return fail(FAME_ERR_UNSUPPORTED, "too many Taylor terms");
  // FP64 moments: matrix products, except for one or two centers, which would use 2 or 4 of 16
  // accumulator rows (three components at N=5, p = 4 / 6 / 10, two centers: 0.93 / 1.08 / 2.14 ms
  // against 0.77 / 1.00 / 2.36 ms of k_taylor_moments; one center 2.07 against 1.43 ms at p = 10).
  // There the modes are cut so that a small grid still fills the GPU.
  const bool mma = !tc && nBlocks > 2;
  long long perSlice = std::min<long long>(
      kTayChunk, std::max<long long>(4 * kTaySub, (NF * nBlocks / (2 * num_sms()) + kTaySub - 1) / kTaySub * kTaySub));
  int nChunks = (int)((NF + perSlice - 1) / perSlice);
  if (mma) moments_mma_slices(NF, nBlocks, L, &nChunks, &perSlice);
  const TaylorTcPlan tp = tc ? taylor_tc_plan(NF, nBlocks, L, p) : TaylorTcPlan{};
  std::vector<int> packed, tcol;
  if (tc) {
    for (int a = 0; a < L; ++a) packed.push_back(al[3 * a] | al[3 * a + 1] << 8 | al[3 * a + 2] << 16);
    tcol.resize(tp.Npad);
    taylor_tc_columns(tp, al.data(), L, p, tcol.data());
  }
  const size_t nal = al.size();
  if (mma) {  // the column runs travel behind the multi-indices
    const int wm = moments_mma_wm(nBlocks);
    std::vector<int> runs;
    moment_runs(al, L, 128 / wm * moments_mma_nt(L, wm), moments_mma_groups(L, wm), runs);
    al.insert(al.end(), runs.begin(), runs.end());
  }
  cudaStream_t s = ctx->stream;
  int *dal, *dpk, *dcol;
  double2 *dcf, *partial, *gamma;
  double *centers, *dfix, *dax, *boxes;
  const int boxChunks = block_chunks(M, nBlocks);
  float* tout;
  auto carve = [&](Carve& cv) {
    dal = cv.take<int>(al.size());
    dpk = cv.take<int>(tc ? packed.size() : 1);
    dcol = cv.take<int>(tc ? tcol.size() : 1);
    dcf = cv.take<double2>(cf.size());
    partial = cv.take<double2>(tc ? 1 : (size_t)nChunks * nBlocks * L);
    gamma = cv.take<double2>((size_t)nBlocks * L);
    centers = cv.take<double>((size_t)nBlocks * 3);
    dfix = cv.take<double>(3);
    dax = cv.take<double>(kTaylorTcMaxAxis);
    boxes = cv.take<double>((size_t)nBlocks * boxChunks * 6);
    tout = cv.take<float>(tc ? tp.out_floats : 1);
  };
  Carve size_only;
  carve(size_only);
  void* ws = nullptr;
  int st = ctx_workspace(ctx, size_only.used, &ws);
  Carve cv;
  cv.base = static_cast<char*>(ws);
  carve(cv);
  if (!fixedCenter) dfix = nullptr;
  if (st == FAME_OK) {
    cudaMemcpyAsync(dal, al.data(), al.size() * sizeof(int), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(dcf, cf.data(), cf.size() * sizeof(double2), cudaMemcpyHostToDevice, s);
    if (fixedCenter) cudaMemcpyAsync(dfix, fixedCenter, 3 * sizeof(double), cudaMemcpyHostToDevice, s);
    if (!dfix) {
      k_block_boxes<<<dim3(boxChunks, nBlocks), kBoxThreads, 0, s>>>(rPoints, M, blockPtr, blockIds, boxes);
      ::fame::count_launch();
    }
    k_block_centers<<<(3 * nBlocks + 127) / 128, 128, 0, s>>>(boxes, dfix ? 0 : boxChunks, nBlocks, dfix, centers);
    ::fame::count_launch();
    if (mma) {
      st = taylor_moments_mma((const double2*)coeff, qModes, NF, centers, dal + nal, L, nBlocks, nChunks, perSlice,
                              partial, s);
      k_taylor_reduce<<<(nBlocks * L + 31) / 32, 256, 0, s>>>(partial, nChunks, nBlocks, L, dcf, gamma);
      ::fame::count_launch();
    } else if (!tc) {
      dim3 gm(nChunks, nBlocks);
      k_taylor_moments<<<gm, std::max(32, (L + 31) / 32 * 32), 0, s>>>((const double2*)coeff, qModes, NF, centers,
                                                                       dal, L, p, nBlocks, perSlice, partial);
      ::fame::count_launch();
      k_taylor_reduce<<<(nBlocks * L + 31) / 32, 256, 0, s>>>(partial, nChunks, nBlocks, L, dcf, gamma);
      ::fame::count_launch();
    } else {
      cudaMemcpyAsync(dpk, packed.data(), packed.size() * sizeof(int), cudaMemcpyHostToDevice, s);
      cudaMemcpyAsync(dcol, tcol.data(), tcol.size() * sizeof(int), cudaMemcpyHostToDevice, s);
      // centers on a tensor grid (the Yee block partition's are): the moment kernel then
      // factorises the phases per axis
      TaylorTcGrid grid;
      std::vector<double> hc((size_t)nBlocks * 3), hax;
      if (cudaMemcpyAsync(hc.data(), centers, hc.size() * sizeof(double), cudaMemcpyDeviceToHost, s) == cudaSuccess &&
          cudaStreamSynchronize(s) == cudaSuccess && tensor_grid_of(hc, nBlocks, grid, hax)) {
        cudaMemcpyAsync(dax, hax.data(), hax.size() * sizeof(double), cudaMemcpyHostToDevice, s);
        grid.ax = dax;
      }
      cudaGetLastError();
      st = taylor_moments_tc(tp, s, (const double2*)coeff, qModes, NF, centers, nBlocks, dpk, dcol, L, p, dcf, tout,
                             gamma, grid);
    }
    if (st == FAME_OK && M > 0) {
      k_taylor_eval<<<dim3(boxChunks, nBlocks), 256, L * sizeof(double2), s>>>(rPoints, M, blockPtr, blockIds, centers,
                                                                               gamma, L, p, (double2*)u);
      ::fame::count_launch();
    }
    if (st == FAME_OK && cudaGetLastError() != cudaSuccess) st = fail(FAME_ERR_CUDA, "taylor launch");
    if (st == FAME_OK && cudaStreamSynchronize(s) != cudaSuccess) st = fail(FAME_ERR_CUDA, "taylor sync");
  }
  return st;
}

}  // namespace fame

extern "C" {

int fame_taylor_on_blocks(fame_ctx* ctx, const void* coeff, const double* qModes, long long NF,
                          const double* rPoints, long long M, int p, const long long* blockPtr,
                          const long long* blockIds, int nBlocks, const double* fixedCenter, void* u) {
  return taylor_impl(ctx, coeff, qModes, NF, rPoints, M, p, blockPtr, blockIds, nBlocks, fixedCenter, u, false);
}

int fame_taylor_on_blocks_3xtf32(fame_ctx* ctx, const void* coeff, const double* qModes, long long NF,
                                 const double* rPoints, long long M, int p, const long long* blockPtr,
                                 const long long* blockIds, int nBlocks, const double* fixedCenter, void* u) {
  return taylor_impl(ctx, coeff, qModes, NF, rPoints, M, p, blockPtr, blockIds, nBlocks, fixedCenter, u, true);
}

}  // extern "C"
