// Batched complex GEMM C = A B (FP64 complex operands and result) on the tcgen05
// tensor cores in split FP32 (3xTF32): each operand value v = head + tail, both
// TF32, and the product is head*head + head*tail + tail*head.
//
// The complex product becomes one real GEMM over interleaved (re, im) pairs:
//   A' row 2m   = (Re A[m,k], -Im A[m,k]) for k = 0..K-1,
//   A' row 2m+1 = (Im A[m,k],  Re A[m,k]),
//   B' row n    = (Re B[k,n],  Im B[k,n]),
// so D[2m][n] = Re C[m,n] and D[2m+1][n] = Im C[m,n].
//
// Two kernels.  k_zsplit splits each operand once, in a bandwidth-bound pass, into
// panels already in the shared-memory form of the MMA: per (row tile, stage of 16
// complex k = 32 TF32 values of K', one 128-byte swizzle atom) a head part and a
// tail part, each rows x 128 bytes in the 128-byte swizzled K-major UMMA layout,
// one contiguous block per (tile, stage).  k_zgemm_3xtf32 then streams those blocks:
// one thread issues the A and B bulk copies of each stage (completed on the stage's
// mbarrier), one
// thread issues tcgen05.mma kind::tf32 -- head*head into one TMEM accumulator, the two
// cross products into a second (the tensor cores round the FP32 accumulation toward
// zero, and the cross products are 2^-11 smaller, so only the head*head sum carries
// that bias) -- and commits to the stage's release mbarrier; the epilogue (16 warps,
// four per 32 TMEM lanes) adds the two accumulators in FP64.  An A panel tile is 64
// complex rows (128 accumulator lanes); a B panel tile is Nt <= 256 columns.  Operands
// shared by several output tiles (the phase tables of the direct sum) are split once
// instead of once per tile, and the first two GEMMs of the direct sum write their results as
// the next one's panels (zchain_3xtf32).
//
// What bounds it, at N=5 on 243^3 points and three components: the panels on their way to
// shared memory.  A 64 x 256 tile reads 672 KB; the last GEMM's 2769 tiles take 322 us (1.9 GB
// of panels and 0.7 GB of results through L2, 7.9 TB/s), the second 198 us, the first 98 us, the
// split 35 us.
#include "internal.cuh"
#include "umma.cuh"

namespace fame {
namespace {

constexpr int kZM = 64;                     // complex rows per A tile (128 accumulator lanes)
constexpr int kZKC = 16;                    // complex k per stage
// producer (thread 0), MMA issuer (thread 32), epilogue (all 16 warps: a warp reads the 32 TMEM
// lanes of its number mod 4, so four warps share each lane group's columns).  One CTA per SM:
// nothing else hides the epilogue's conversions and stores; with four warps the three GEMMs of
// an N=5 field on 243^3 points, three components, took 72 us more.
constexpr int kZThreads = 512;
constexpr int kZColGroups = kZThreads / 128;
constexpr uint32_t kZABytes = 128u * 128u;  // one TF32 part of an A stage

__host__ __device__ constexpr uint32_t zb_bytes(int nt) { return (uint32_t)nt * 128u; }
__host__ __device__ constexpr uint32_t zstage_bytes(int nt) { return 2u * (kZABytes + zb_bytes(nt)); }
inline int zstages(int nt) { return zstage_bytes(nt) * 3u + 2048u <= 227u * 1024u ? 3 : 2; }
inline size_t zsmem(int nt) { return 1024 + (size_t)zstages(nt) * zstage_bytes(nt) + 128; }

// Operand panels: element (real row r, K' index kk) of stage ks of tile t of batch b sits at
// byte ((b * tiles + t) * stages + ks) * 2 * part + half * part + sw128_offset(r, kk),
// part = real rows per tile * 128 bytes (head: half 0, tail: half 1).
struct SplitArgs {
  const double2* src;
  long long s_row, s_k, s_batch;  // element strides of (complex row, k, batch)
  int rows, K, batches;
  int tile_rows;                   // complex rows per tile: 64 (A role) or Nt (B role)
  int a_role;                      // A: two real rows (Re, -Im), (Im, Re); B: one (Re, Im)
  unsigned char* out;
  int rows_pad;                    // rows of the panels (>= rows; zeros from rows on)
  int gn;                          // > 0: the source is one component's coefficients in natural 6D order
};

// Coefficient j1 + n j2 + ... + n^5 j6 as element (k = a, row = b + n^2 c) of the contraction
// over the axis pairs a = j1 + n j4, b = j2 + n j5, c = j3 + n j6.
__device__ __forceinline__ long long coeff_k(int n, int a) { return a % n + (long long)n * n * n * (a / n); }
__device__ __forceinline__ long long coeff_row(int n, int r) {
  const int n2 = n * n, b = r % n2, c = r / n2;
  const long long n3 = (long long)n2 * n;
  return (long long)n * (b % n) + n * n3 * (b / n) + (long long)n2 * (c % n) + n2 * n3 * (c / n);
}

// A CTA takes (a share of the rows of) one panel block (batch, tile, stage): the FP64 values
// are read along the operand's contiguous dimension into shared memory, then written as
// whole 128-byte rows, 16 bytes (four TF32 values of K' = two complex k) per thread.
constexpr int kSplitThreads = 256;
constexpr int kSplitMaxRows = 256;  // complex rows of a tile (B role, Nt <= 256)
// several operands in one launch: job j owns blocks [first[j], first[j + 1])
constexpr int kMaxSplitJobs = 4;
struct SplitJobs {
  SplitArgs job[kMaxSplitJobs];
  int first[kMaxSplitJobs + 1];
  int njobs;
  int pitch;  // shared tile row pitch: the largest per-CTA row share of the jobs, plus one
};
// A CTA covers at most kSplitRows complex rows of a panel block (B blocks of Nt = 256 rows
// take two CTAs: the rows of a block are independent), so its shared tile stays within 33 KB.
constexpr int kSplitRows = 128;
__device__ __forceinline__ int split_subs(const SplitArgs& a) { return (a.tile_rows + kSplitRows - 1) / kSplitRows; }
__global__ void __launch_bounds__(kSplitThreads) k_zsplit(SplitJobs jobs) {
  extern __shared__ double2 tile_raw[];  // [kZKC][pitch]: [k][complex row of this CTA's share]
  const int pitch = jobs.pitch;
  int j = 0;
  while (j + 1 < jobs.njobs && (int)blockIdx.x >= jobs.first[j + 1]) ++j;
  const SplitArgs& a = jobs.job[j];
  const int bid = (int)blockIdx.x - jobs.first[j];
  const int tiles = (a.rows_pad + a.tile_rows - 1) / a.tile_rows;
  const int stages = (a.K + kZKC - 1) / kZKC, subs = split_subs(a);
  const int ks = bid % stages, rest = bid / stages, h = rest % subs, t = (rest / subs) % tiles,
            b = rest / (subs * tiles);
  const int rr0 = h * kSplitRows, nr = a.tile_rows - rr0 < kSplitRows ? a.tile_rows - rr0 : kSplitRows;
  const int r0 = t * a.tile_rows + rr0, k0 = ks * kZKC;
  const bool rfast = a.s_row == 1;  // read along the contiguous dimension
  const double2* src = a.src + (long long)b * a.s_batch;
  for (int e = threadIdx.x; e < nr * kZKC; e += kSplitThreads) {
    const int rr = rfast ? e % nr : e / kZKC, kk = rfast ? e / nr : e % kZKC;
    const int r = r0 + rr, k = k0 + kk;
    double2 v = make_double2(0.0, 0.0);
    if (r < a.rows && k < a.K)
      v = __ldg(src + (a.gn > 0 ? coeff_row(a.gn, r) + coeff_k(a.gn, k) : (long long)r * a.s_row + (long long)k * a.s_k));
    tile_raw[kk * pitch + rr] = v;
  }
  __syncthreads();
  const int per = a.a_role ? 2 : 1;  // real rows per complex row
  const size_t part = (size_t)a.tile_rows * per * 128u;
  unsigned char* blk = a.out + ((size_t)((long long)b * tiles + t) * stages + ks) * 2 * part;
  // 16-byte chunk c of real row R holds K' = 4c .. 4c+3, i.e. complex k = 2c, 2c+1
  for (int e = threadIdx.x; e < nr * per * 8; e += kSplitThreads) {
    const int Rl = e / 8, c = e % 8, R = rr0 * per + Rl;  // Rl: real row within this CTA's share
    float hv[4], lv[4];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const double2 v = tile_raw[(2 * c + q) * pitch + Rl / per];
      float rh, rl, ih, il;
      umma::tf32_split_fast(v.x, rh, rl);
      umma::tf32_split_fast(v.y, ih, il);
      const bool second = a.a_role && (R & 1);  // A rows: (Re, -Im) then (Im, Re)
      hv[2 * q] = second ? ih : rh;
      hv[2 * q + 1] = second ? rh : (a.a_role ? -ih : ih);
      lv[2 * q] = second ? il : rl;
      lv[2 * q + 1] = second ? rl : (a.a_role ? -il : il);
    }
    const uint32_t off = umma::sw128_offset(R, 4 * c);
    *reinterpret_cast<float4*>(blk + off) = make_float4(hv[0], hv[1], hv[2], hv[3]);
    *reinterpret_cast<float4*>(blk + part + off) = make_float4(lv[0], lv[1], lv[2], lv[3]);
  }
}

// Destination panels of a chained GEMM (kToXC, kToXY): bytes per batch, output axis sizes.
struct ZChain {
  unsigned char* out;
  size_t batch;
  int nx, xs, x0, n2, cp;  // nx points, of which this launch has xs from x0 on
};

struct ZgArgs {
  const unsigned char* Ap;  // A panels (64-row tiles), per batch
  const unsigned char* Bp;  // B panels (Nt-row tiles), per B batch
  double2* C;
  int M, N, K, Nt, S;
  long long scm, scn, bC;
  int tilesA;  // A row tiles per batch (the launch may take a part of them)
  int tilesM, tilesN, batch;
  ZChain ch;
};

// Where the epilogue puts C.  kPlain: FP64 complex values at (m scm + n scn).  The other two
// write C as the next GEMM's A panels, already split: head and tail of the same FP64 sums that
// k_zsplit would read back, so the next GEMM's operand has the same bits, and the FP64
// intermediate is neither written nor read (at N=5, 243^3 points, three components the two
// passes of k_zsplit over the intermediates took 74 and 171 us; the GEMMs that write panels take
// 98 and 198 us where those that wrote FP64 took 68 and 154).  With x, y the output axes and (b, c) the two
// contracted axis pairs of n2 values each, c padded to cp, the next multiple of a stage:
//   kToXC: C(x, b + n2 c) -> row (x, c), k = b; a row tile is 4 x by 16 c, so that
//   kToXY: C((x, c), y) of that tile -> row x + nx y, k = c: the 16 complex rows of a warp's
//          lanes are the 16 k of one panel row, which it writes as whole 128-byte lines.
// Rows and columns of the padding are zero operands, so the padded k come out as zeros.
enum { kPlain = 0, kToXC = 1, kToXY = 2 };

// head and tail parts of (re, im) as A-role row pairs (Re, -Im), (Im, Re)
struct ZSplit {
  float rh, rl, ih, il;
  __device__ __forceinline__ explicit ZSplit(double2 v) {
    umma::tf32_split_fast(v.x, rh, rl);
    umma::tf32_split_fast(v.y, ih, il);
  }
};

// A warp's 16 rows by 32 columns of C on their way from lanes along rows to lanes along columns
// (kToXC), in the operand stages once every MMA is complete: columns 16.. start at 20 and the
// pitch is -1 mod 8, so the 16-byte writes meet no bank twice.  Written straight from the
// accumulator's lanes, 16 bytes to each of 32 lines per store, the first GEMM took 329 us, not 98.
constexpr int kTurnPitch = 39;
constexpr int kTurnElems = 16 * kTurnPitch;
constexpr bool turn_fits() {
  for (uint32_t nt = 32; nt <= 256; nt += 32) {
    const uint32_t stage = zstage_bytes((int)nt), S = stage * 3u + 2048u <= 227u * 1024u ? 3 : 2;
    if (S * stage < (nt / 32 * 4 < 16 ? nt / 32 * 4 : 16) * kTurnElems * 16u) return false;
  }
  return true;
}
static_assert(turn_fits(), "transposition buffers exceed the operand stages");

// The k < n2 of kToXC's panels are rounded up to whole stages by zeros: column b also zeroes
// b + n2, b + 2 n2, ... below cp.
__device__ __forceinline__ void put_xc(const ZChain& ch, unsigned char* pan, int x, int c, int b, double2 v0,
                                       double2 v1) {
  const ZSplit p(v0), q(v1);
  const int cst = ch.cp / kZKC;
  const int R = 2 * ((x & 3) * kZKC + (c & (kZKC - 1)));
  unsigned char* tile = pan + ((size_t)(x >> 2) * cst + c / kZKC) * cst * 2 * kZABytes;
  for (int k = b; k < ch.cp; k += ch.n2) {
    const bool in = k == b;
    unsigned char* blk = tile + (size_t)(k / kZKC) * 2 * kZABytes;
    const uint32_t o0 = umma::sw128_offset(R, 2 * (k & (kZKC - 1))), o1 = umma::sw128_offset(R + 1, 2 * (k & (kZKC - 1)));
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4*>(blk + o0) = in ? make_float4(p.rh, -p.ih, q.rh, -q.ih) : z;
    *reinterpret_cast<float4*>(blk + o1) = in ? make_float4(p.ih, p.rh, q.ih, q.rh) : z;
    *reinterpret_cast<float4*>(blk + kZABytes + o0) = in ? make_float4(p.rl, -p.il, q.rl, -q.il) : z;
    *reinterpret_cast<float4*>(blk + kZABytes + o1) = in ? make_float4(p.il, p.rl, q.il, q.rl) : z;
  }
}

__device__ __forceinline__ void put_xy(unsigned char* pan, int cst, int cs, int r, int k, double2 v) {
  const ZSplit p(v);
  unsigned char* blk = pan + ((size_t)(r / kZM) * cst + cs) * 2 * kZABytes;
  const int R = 2 * (r & (kZM - 1));
  const uint32_t o0 = umma::sw128_offset(R, 2 * k), o1 = umma::sw128_offset(R + 1, 2 * k);
  *reinterpret_cast<float2*>(blk + o0) = make_float2(p.rh, -p.ih);
  *reinterpret_cast<float2*>(blk + o1) = make_float2(p.ih, p.rh);
  *reinterpret_cast<float2*>(blk + kZABytes + o0) = make_float2(p.rl, -p.il);
  *reinterpret_cast<float2*>(blk + kZABytes + o1) = make_float2(p.il, p.rl);
}

template <int OUT>
__global__ void __launch_bounds__(kZThreads, 1) k_zgemm_3xtf32(ZgArgs g, unsigned* fault) {
  extern __shared__ unsigned char smraw[];
  unsigned char* sm = smraw + ((1024u - (smem_u32(smraw) & 1023u)) & 1023u);
  const int Nt = g.Nt, S = g.S;
  const uint32_t bB = zb_bytes(Nt), stB = zstage_bytes(Nt);
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + (size_t)S * stB);  // [S]: stage landed
  uint64_t* empty = full + S;                                          // [S]: stage read by the MMAs
  uint64_t* done = full + 2 * S;                                       // every MMA complete
  uint32_t* slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abortf = reinterpret_cast<volatile int*>(slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nch = (g.K + kZKC - 1) / kZKC;
  const size_t astride = 2 * (size_t)kZABytes, bstride = 2 * (size_t)bB;  // bytes per stage of a tile
  const ZChain& ch = g.ch;
  const int total = g.tilesM * g.tilesN * g.batch;
  const uint32_t ncols = 2 * Nt <= 32 ? 32u : 2 * Nt <= 64 ? 64u : 2 * Nt <= 128 ? 128u : 2 * Nt <= 256 ? 256u : 512u;

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(done, 1);
    *abortf = 0;
    mbar_init_fence();
  }
  if (warp == 0) {
    umma::tmem_alloc(slot, ncols);
    umma::tmem_relinquish();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *slot;  // columns [0, Nt): head*head; [Nt, 2 Nt): cross products

  // producer (thread 0): the stages of this CTA's tiles in turn, it = 0, 1, ..: into buffer it % S
  // once the MMAs of it - S are done
  int issued = 0;
  auto issue = [&](int t, int i) {
    const int s = issued % S;
    if (*abortf || (issued >= S && !mbar_wait(&empty[s], (unsigned)((issued / S - 1) & 1)))) {
      *abortf = 1;
      return false;
    }
    const int bx = t % g.tilesM, by = t / g.tilesM % g.tilesN, bz = t / (g.tilesM * g.tilesN);
    const unsigned char* Ap = g.Ap + (((size_t)bz * g.tilesA + bx) * nch + i) * astride;
    const unsigned char* Bp = g.Bp + (((size_t)bz * g.tilesN + by) * nch + i) * bstride;
    unsigned char* stg = sm + (size_t)s * stB;
    mbar_arrive_expect_tx(&full[s], (unsigned)(astride + bstride));
    bulk_g2s(stg, Ap, (unsigned)astride, &full[s]);
    bulk_g2s(stg + astride, Bp, (unsigned)bstride, &full[s]);
    ++issued;
    return true;
  };

  for (int t = blockIdx.x, it0 = 0, seq = 0; t < total; t += gridDim.x, it0 += nch, ++seq) {
    const int bx = t % g.tilesM, by = t / g.tilesM % g.tilesN, bz = t / (g.tilesM * g.tilesN);
    const int m0 = bx * kZM, n0 = by * Nt;
    double2* Cm = g.C + g.bC * bz;                    // kPlain
    unsigned char* pan = ch.out + (size_t)bz * ch.batch;  // kToXC, kToXY
    if (tid == 0) {
      for (int i = issued - it0; i < nch && issue(t, i); ++i) {
      }
    } else if (tid == 32) {
      const uint32_t id = umma::idesc_tf32(128, Nt);
      for (int i = 0; i < nch; ++i) {
        const int it = it0 + i, s = it % S;
        if (*abortf || !mbar_wait(&full[s], (unsigned)((it / S) & 1))) {
          *abortf = 1;
          break;
        }
        umma::fence_after_sync();
        const uint32_t sa = smem_u32(sm + (size_t)s * stB);
        for (int kk = 0; kk < 2 * kZKC / 8; ++kk) {
          const uint32_t o = kk * 32u, acc = (i | kk) != 0 ? 1u : 0u;
          const uint64_t ahi = umma::desc_kmajor_sw128(sa + o), alo = umma::desc_kmajor_sw128(sa + kZABytes + o);
          const uint64_t bhi = umma::desc_kmajor_sw128(sa + 2u * kZABytes + o);
          const uint64_t blo = umma::desc_kmajor_sw128(sa + 2u * kZABytes + bB + o);
          umma::mma_tf32(tmem, ahi, bhi, id, acc);
          umma::mma_tf32(tmem + (uint32_t)Nt, ahi, blo, id, acc);
          umma::mma_tf32(tmem + (uint32_t)Nt, alo, bhi, id, 1u);
        }
        umma::commit(&empty[s]);
      }
      umma::commit(done);  // arrives once every MMA issued above has completed
    }
    __syncwarp();
    const bool fin = mbar_wait(done, (unsigned)(seq & 1));
    const bool ok = __syncthreads_and(fin && !*abortf);
    if (!ok) {
      // copies issued for stages the MMAs never consumed still land in this CTA's shared
      // memory: wait for them (bounded) before the CTA may exit
      if (tid == 0) {
        for (int i = issued - S < 0 ? 0 : issued - S; i < issued; ++i) mbar_wait(&full[i % S], (unsigned)((i / S) & 1));
        if (fault) atomicOr(fault, 1u);
      }
      break;
    }
    // every MMA of the tile is complete, so the stages are free: the next tile's first S of them
    // land while this tile's sums are stored (the others overlap its MMAs)
    if (OUT != kToXC && tid == 0 && t + gridDim.x < total)
      for (int i = 0; i < S && i < nch && issue(t + gridDim.x, i); ++i) {
      }
    __syncwarp();
    umma::fence_after_sync();
    const int lg = warp & 3;
    const int m = m0 + (lg * 32 + lane) / 2;  // TMEM lane pair (2j, 2j+1) = (Re, Im) of row m
    const bool odd = lane & 1;
    double2* turn = reinterpret_cast<double2*>(sm) + (size_t)warp * kTurnElems;  // kToXC: the stages are free now
    for (int cc = warp >> 2; cc < Nt / 32; cc += kZColGroups) {
      uint32_t hh[32], xx[32];
      umma::ld_32x32b_x32(tmem + ((uint32_t)(lg * 32) << 16) + (uint32_t)(cc * 32), hh);
      umma::ld_32x32b_x32(tmem + ((uint32_t)(lg * 32) << 16) + (uint32_t)(Nt + cc * 32), xx);
      umma::wait_ld(hh);
      umma::wait_ld(xx);
      // the even lane stores columns 0..15 of the chunk, the odd lane 16..31
      const int nb = n0 + cc * 32 + (odd ? 16 : 0);
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const double lo = (double)__uint_as_float(hh[c]) + (double)__uint_as_float(xx[c]);
        const double hi = (double)__uint_as_float(hh[c + 16]) + (double)__uint_as_float(xx[c + 16]);
        const double other = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);
        const double2 v = odd ? make_double2(other, hi) : make_double2(lo, other);
        const int n = nb + c;
        if (OUT == kPlain) {
          if (m < g.M && n < g.N) Cm[(long long)m * g.scm + (long long)n * g.scn] = v;
        } else if (OUT == kToXC) {
          turn[(lane >> 1) * kTurnPitch + c + (odd ? 20 : 0)] = v;
        } else {
          const int cst = ch.cp / kZKC, x = bx / cst * 4 + lg;
          if (x < ch.xs && n < g.N) put_xy(pan, cst, bx % cst, ch.x0 + x + ch.nx * n, lane >> 1, v);
        }
      }
      if (OUT == kToXC) {  // eight lanes write the 16 columns of a row: n2 = (2N)^2 is even, so a pair shares c
        __syncwarp();
        for (int i = lane; i < 16 * 16; i += 32) {
          const int row = i >> 4, q = i & 15, n = n0 + cc * 32 + 2 * q, x = m0 + lg * 16 + row, c2 = n / ch.n2;
          const double2* t = turn + row * kTurnPitch + 2 * q + (q >= 8 ? 4 : 0);
          if (x < (ch.xs + 3) / 4 * 4 && n < g.N) put_xc(ch, pan, x, c2, n - c2 * ch.n2, t[0], t[1]);
        }
        __syncwarp();
      }
    }
    umma::fence_before_sync();
    __syncthreads();  // the accumulators have been read
    umma::fence_after_sync();
  }
  __syncthreads();
  if (warp == 0) {
    umma::fence_after_sync();
    umma::tmem_dealloc(tmem, ncols);
  }
}

inline int z_nt(int N) { return std::min(256, (N + 31) / 32 * 32); }
inline size_t panel_bytes(int rows, int K, int batches, int tile_rows, bool a_role) {
  const size_t tiles = (size_t)(rows + tile_rows - 1) / tile_rows, stages = (size_t)(K + kZKC - 1) / kZKC;
  return (size_t)batches * tiles * stages * 2 * (size_t)tile_rows * (a_role ? 2 : 1) * 128u;
}

}  // namespace

size_t zpanel_bytes(const ZPanelJob& j) {
  return panel_bytes(std::max(j.rows, j.rows_pad), j.K, j.batches, j.a_role ? kZM : z_nt(j.cols_for_b),
                     j.a_role);
}

int zsplit_panels(const ZPanelJob* jobs, int njobs, cudaStream_t s) {
  if (njobs < 1 || njobs > kMaxSplitJobs) return fail(FAME_ERR_INVALID, "zsplit_panels: job count");
  SplitJobs sj{};
  long long blocks = 0;
  int share = 1;
  for (int j = 0; j < njobs; ++j) {
    const ZPanelJob& z = jobs[j];
    const int tile_rows = z.a_role ? kZM : z_nt(z.cols_for_b);
    if (!z.src || !z.out || z.rows <= 0 || z.K <= 0 || z.batches <= 0 || tile_rows > kSplitMaxRows ||
        (reinterpret_cast<uintptr_t>(z.out) & 1023u) != 0)
      return fail(FAME_ERR_INVALID, "zsplit_panels: job");
    sj.job[j] = SplitArgs{z.src, z.s_row, z.s_k, z.s_batch, z.rows, z.K, z.batches, tile_rows, z.a_role ? 1 : 0, z.out,
                          std::max(z.rows, z.rows_pad), z.gather_n};
    sj.first[j] = (int)blocks;
    blocks += (long long)z.batches * ((sj.job[j].rows_pad + tile_rows - 1) / tile_rows) * ((z.K + kZKC - 1) / kZKC) *
              ((tile_rows + kSplitRows - 1) / kSplitRows);
    share = std::max(share, std::min(tile_rows, kSplitRows));
    if (blocks > 0x7fffffffLL) return fail(FAME_ERR_UNSUPPORTED, "zsplit_panels: too many panel blocks");
  }
  sj.first[njobs] = (int)blocks;
  sj.njobs = njobs;
  sj.pitch = share + 1;
  k_zsplit<<<(unsigned)blocks, kSplitThreads, (size_t)kZKC * sj.pitch * sizeof(double2), s>>>(sj);
  ::fame::count_launch();
  FAME_CUDA_TRY(cudaGetLastError());
  return FAME_OK;
}

namespace {

template <int OUT>
int launch_zgemm(ZgArgs g, int batch, cudaStream_t s) {
  if (g.M <= 0 || g.N <= 0 || g.K <= 0 || batch <= 0 || !g.Ap || !g.Bp || (OUT == kPlain ? !g.C : !g.ch.out))
    return fail(FAME_ERR_INVALID, "zgemm_3xtf32: arguments");
  if ((reinterpret_cast<uintptr_t>(g.Ap) & 1023u) != 0 || (reinterpret_cast<uintptr_t>(g.Bp) & 1023u) != 0 ||
      (reinterpret_cast<uintptr_t>(g.ch.out) & 1023u) != 0)
    return fail(FAME_ERR_INVALID, "zgemm_3xtf32: panels must be 1024-byte aligned");
  g.Nt = z_nt(g.N);
  g.S = zstages(g.Nt);
  static DeviceOnce once;
  FAME_TRY(ensure_smem(k_zgemm_3xtf32<OUT>, 227 * 1024, once));
  const long long gy = ((long long)g.N + g.Nt - 1) / g.Nt;
  if (gy > 65535 || batch > 65535) return fail(FAME_ERR_UNSUPPORTED, "zgemm_3xtf32: grid too large");
  g.tilesM = (g.M + kZM - 1) / kZM;
  g.tilesN = (int)gy;
  g.batch = batch;
  const long long total = (long long)g.tilesM * gy * batch;
  if (total > 0x3fffffffLL) return fail(FAME_ERR_UNSUPPORTED, "zgemm_3xtf32: grid too large");
  // one CTA per SM takes several tiles and loads ahead across them (one tile per CTA: the last two
  // GEMMs of the file's head 212 and 329 us, the call 701 against 664 us); kToXC's epilogue needs
  // the stages itself, so nothing could be loaded ahead and a CTA takes one tile
  const unsigned grid = (unsigned)(OUT == kToXC ? total : std::min<long long>(total, num_sms() > 0 ? num_sms() : 148));
  k_zgemm_3xtf32<OUT><<<grid, kZThreads, zsmem(g.Nt), s>>>(g, fault_word());
  ::fame::count_launch();
  FAME_CUDA_TRY(cudaGetLastError());
  return FAME_OK;
}

}  // namespace

// The x axis is taken in slabs so that the panels of T1 stay below 1 GB: no slab but on long thin
// grids, whose scratch would grow with the padding of c (four times at n2 = 4).
constexpr size_t kSlabBytes = (size_t)1 << 30;

ZChainSizes zchain_sizes(int nx, int ny, int n2, int ncomp) {
  ZChainSizes z;
  z.cp = (n2 + kZKC - 1) / kZKC * kZKC;
  const size_t per = panel_bytes(kZM * z.cp, n2, ncomp, kZM, true);  // kZM points of x
  z.xs = (int)std::min<long long>(((long long)nx + 3) / 4 * 4, kZM * (long long)std::max<size_t>(1, kSlabBytes / per));
  z.bytes1 = panel_bytes(z.xs * z.cp, n2, 1, kZM, true);
  z.bytes2 = panel_bytes(nx * ny, n2, 1, kZM, true);
  return z;
}

int zchain_3xtf32(const unsigned char* Tx, const unsigned char* Cp, const unsigned char* Ty, const unsigned char* Tz,
                  unsigned char* P1, unsigned char* P2, double2* u, int nx, int ny, int nz, int n2, int ncomp,
                  cudaStream_t s) {
  const ZChainSizes z = zchain_sizes(nx, ny, n2, ncomp);
  const int cst = z.cp / kZKC, tx = (nx + kZM - 1) / kZM;
  int st = FAME_OK;
  // T1(x, (b,c)) = sum_a Tx(x,a) Cp(a, (b,c)); T2((x,c), y) = sum_b T1 Ty; u((x,y), z) = sum_c T2 Tz
  for (int x0 = 0; x0 < nx && st == FAME_OK; x0 += z.xs) {
    const int xs = std::min(z.xs, nx - x0), t1 = (xs + 3) / 4 * cst;
    const ZChain c1{P1, z.bytes1, nx, xs, x0, n2, z.cp}, c2{P2, z.bytes2, nx, xs, x0, n2, z.cp};
    const unsigned char* Ax = Tx + (size_t)(x0 / kZM) * cst * 2 * kZABytes;
    st = launch_zgemm<kToXC>(ZgArgs{Ax, Cp, nullptr, xs, n2 * z.cp, n2, 0, 0, 0, 0, 0, tx, 0, 0, 0, c1}, ncomp, s);
    if (st == FAME_OK)
      st = launch_zgemm<kToXY>(ZgArgs{P1, Ty, nullptr, t1 * kZM, ny, n2, 0, 0, 0, 0, 0, z.xs / 4 * cst, 0, 0, 0, c2}, ncomp, s);
  }
  const int t2 = (nx * ny + kZM - 1) / kZM;
  if (st == FAME_OK)
    st = launch_zgemm<kPlain>(ZgArgs{P2, Tz, u, nx * ny, nz, n2, 0, 0, 1, (long long)nx * ny, (long long)nx * ny * nz,
                                     t2, 0, 0, 0, ZChain{}}, ncomp, s);
  return st;
}

}  // namespace fame
