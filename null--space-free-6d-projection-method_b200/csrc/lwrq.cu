// Physical validation of a reconstructed Yee field by the local weighted
// Rayleigh quotient (LWRQ), restating exp3/compute_yee_lwrq_metrics_exp4.m,
// exp3/compute_lwrq_exp4.m, exp3/apply_cropped_A_exp3.m,
// exp3/separable_conv3_same_exp4.m and exp3/sample_scalar_yee_material_exp4.m.
//
// Input: the three components on the plus-grid, m = 2n+3 points per axis,
// column-major with x fastest (the order of the Yee reconstruction).  All work
// is on the (2n+1)^3 interior, q = 2n+1:
//   k_lwrq_tables per-axis factors of the material (see YeeTab) and 1 / window mass;
//   k_lwrq_ab     curl-curl stencil Au, eps on the Yee edges, Bu = eps u,
//                 a = Re<u,Au>, b = Re<u,Bu> per point, written divided by the window's
//                 column normalisation, and the sums behind lambdaCrop and both residuals;
//   k_lwrq_xy     x and y axes of the zero-padded separable Gaussian window (radius 3
//                 cells, sigma 2h) for the a- and b-paths, one tile of a plane per CTA;
//   k_lwrq_z      z axis of the window, and every statistic of E, M and rho = E/M while
//                 they are in registers (neither is stored); the z = 0 / x = 0 slices of rho;
//   k_lwrq_dev    |rho - lambda3D| / |lambda3D| of the slices;
//   k_lwrq_resid  ||Au - lambda Bu||^2 with the stencil recomputed, only where the sums of
//                 k_lwrq_ab would lose digits to cancellation.
// The host reads once.  Reductions are the deterministic fixed-order grid sums used
// everywhere.  At n = 80 (4.2 M points) a call takes 353 us (127 / 62 / 39 us in ab / xy / z), against
// 1290 us with 36 cosines per point (668 us in the two stencil kernels), per-tap divisions in
// three window passes (235 us), three statistics passes (70 us) and five host reads.
#include <algorithm>
#include <cmath>
#include <vector>
#include "internal.cuh"

namespace fame {

constexpr int kLwrqR = 3;  // window radius in cells (exp3/make_config_experiment4.m:73)

struct YeeMat {
  int kind;          // 0: epsC exp(alpha/6 sum cos), 1: 1 + delta prod (1 + cos)/2
  double p0, p1;     // (epsC, alpha) or (delta, -)
  double P[18];      // cut matrix, column-major 6 x 3: P(l, c) = P[l + 6 c]
};

struct YeeGeom {
  const double2 *u1, *u2, *u3;
  int n, m, q;
  double h;
};

__device__ __forceinline__ double yee_eps(const YeeMat& mt, double x, double y, double z) {
  if (mt.kind == 0) {
    double s = 0.0;
#pragma unroll
    for (int l = 0; l < 6; ++l) s += cos(mt.P[l] * x + mt.P[l + 6] * y + mt.P[l + 12] * z);
    return mt.p0 * exp(mt.p1 / 6.0 * s);
  }
  double prod = 1.0;
#pragma unroll
  for (int l = 0; l < 6; ++l) prod *= 0.5 * (1.0 + cos(mt.P[l] * x + mt.P[l + 6] * y + mt.P[l + 12] * z));
  return 1.0 + mt.p0 * prod;
}

// Au and u (three components) at interior point (i, j, k) of the crop.
__device__ __forceinline__ void yee_curl(const YeeGeom& g, int i, int j, int k, double2* A, double2* U) {
  const long long m = g.m;
  const long long c0 = (i + 1) + m * (j + 1) + m * m * (k + 1);
  auto at = [&](const double2* u, int dx, int dy, int dz) { return u[c0 + dx + m * dy + m * m * dz]; };
  auto second = [&](const double2* u, int ax) {
    const int ex = ax == 0, ey = ax == 1, ez = ax == 2;
    const double2 c = at(u, 0, 0, 0), lo = at(u, -ex, -ey, -ez), hi = at(u, ex, ey, ez);
    return make_double2(2.0 * c.x - lo.x - hi.x, 2.0 * c.y - lo.y - hi.y);
  };
  // backward difference along `bk` of the forward difference along `fw`
  auto mixed = [&](const double2* u, int bk, int fw) {
    const int fx = fw == 0, fy = fw == 1, fz = fw == 2, bx = -(bk == 0), by = -(bk == 1), bz = -(bk == 2);
    const double2 a = at(u, fx + bx, fy + by, fz + bz), b = at(u, bx, by, bz), c = at(u, fx, fy, fz),
                  d = at(u, 0, 0, 0);
    return make_double2(a.x - b.x - c.x + d.x, a.y - b.y - c.y + d.y);
  };
  const double s = 1.0 / (g.h * g.h);
  double2 t1 = cadd<double>(second(g.u1, 1), second(g.u1, 2));
  t1 = csub<double>(csub<double>(t1, mixed(g.u2, 1, 0)), mixed(g.u3, 2, 0));
  double2 t2 = cadd<double>(second(g.u2, 0), second(g.u2, 2));
  t2 = csub<double>(csub<double>(t2, mixed(g.u1, 0, 1)), mixed(g.u3, 2, 1));
  double2 t3 = cadd<double>(second(g.u3, 0), second(g.u3, 1));
  t3 = csub<double>(csub<double>(t3, mixed(g.u1, 0, 2)), mixed(g.u2, 1, 2));
  A[0] = cscale<double>(t1, s);
  A[1] = cscale<double>(t2, s);
  A[2] = cscale<double>(t3, s);
  U[0] = at(g.u1, 0, 0, 0);
  U[1] = at(g.u2, 0, 0, 0);
  U[2] = at(g.u3, 0, 0, 0);
}

static inline int lblocks(long long n) { return (int)std::min<long long>((n + 255) / 256, 148 * 16); }

struct Window {
  double k[2 * kLwrqR + 1];
};

// sum of the window taps that fall inside [0, q) around index i (the
// normalisation of the zero-padded window along one axis)
__device__ __forceinline__ double window_mass(const Window& w, int i, int q) {
  double s = 0.0;
#pragma unroll
  for (int t = 0; t < 2 * kLwrqR + 1; ++t) {
    const int src = i - (t - kLwrqR);
    if (src >= 0 && src < q) s += w.k[t];
  }
  return s;
}

// Tables of length q per axis.  Where every row of the cut matrix has at most one nonzero entry
// (all axis-block matrices), eps(x, y, z) = c0 + p0 fx(x) fy(y) fz(z) for both materials, each
// factor the exp or product over the rows of its axis; f[2 axis + s] holds it at the grid points
// (s = 0) and half a cell further (s = 1).  f is null for other matrices, and the material is
// then evaluated per point (yee_eps).  rd[axis]: 1 / window mass.
struct YeeTab {
  double* f;   // [6][q] or nullptr
  double* rd;  // [q] (the axes are alike)
  double c0, p0;
};
__global__ void k_lwrq_tables(YeeMat mt, YeeTab tb, int n, int q, double h, Window w) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, i = t % q, as = t / q;
  if (as == 6) tb.rd[i] = 1.0 / window_mass(w, i, q);
  if (as >= 6 || !tb.f) return;
  const int ax = as / 2;
  const double x = (i - n) * h + ((as & 1) ? 0.5 * h : 0.0);
  double sum = 0.0, prod = 1.0;
  for (int l = 0; l < 6; ++l) {
    const double p = mt.P[l + 6 * ax];
    const bool none = mt.P[l] == 0.0 && mt.P[l + 6] == 0.0 && mt.P[l + 12] == 0.0;
    if (p != 0.0 || (none && ax == 0)) {  // a zero row is the constant cos 0 = 1
      const double c = cos(p * x);
      sum += c;
      prod *= 0.5 * (1.0 + c);
    }
  }
  tb.f[as * q + i] = mt.kind == 0 ? exp(mt.p1 / 6.0 * sum) : prod;
}
__device__ __forceinline__ void yee_eps3(const YeeGeom& g, const YeeMat& mt, const YeeTab& tb, int i, int j, int k,
                                         double* e) {
  if (tb.f) {
    const int q = g.q;
    const double x0 = tb.f[i], x1 = tb.f[q + i], y0 = tb.f[2 * q + j], y1 = tb.f[3 * q + j], z0 = tb.f[4 * q + k],
                 z1 = tb.f[5 * q + k];
    e[0] = tb.c0 + tb.p0 * (x1 * y0 * z0);
    e[1] = tb.c0 + tb.p0 * (x0 * y1 * z0);
    e[2] = tb.c0 + tb.p0 * (x0 * y0 * z1);
  } else {
    const double x = (i - g.n) * g.h, y = (j - g.n) * g.h, z = (k - g.n) * g.h, hh = 0.5 * g.h;
    e[0] = yee_eps(mt, x + hh, y, z);
    e[1] = yee_eps(mt, x, y + hh, z);
    e[2] = yee_eps(mt, x, y, z + hh);
  }
}

// out: [0] sum a, [1] sum b, [2] ||Au||^2, [3] ||Bu||^2, [4] ||R||^2, [5] Re<R, Bu> with
// R = Au - l6 Bu; a and b are written divided by the window's normalisation at their point.
// A CTA takes 16 x 16 columns, so that the y neighbours of one thread are the loads of another;
// a thread walks kAbRun planes of its column and keeps the values that the next plane needs
// again: 15 loads per point instead of 24.  Bound by the loads through L1 and L2.
// SEP: material from the tables (its per-point evaluation would take the registers of a second
// CTA per SM with it).
constexpr int kAbRun = 16, kAbTile = 16;
template <bool SEP>
__global__ void __launch_bounds__(256, SEP ? 2 : 1) k_lwrq_ab(YeeGeom g, YeeMat mt, YeeTab tb, double l6, double* a, double* b,
                                                 double* out, double* partials, unsigned* counter) {
  const int q = g.q;
  const long long m = g.m, mm = m * m;
  Red<double, 6> acc{};
  const int i = blockIdx.x * kAbTile + threadIdx.x % kAbTile, j = blockIdx.y * kAbTile + threadIdx.x / kAbTile;
  const int k0 = blockIdx.z * kAbRun, k1 = min(q, k0 + kAbRun);
  if (i < q && j < q) {
    const long long c0 = (i + 1) + m * (j + 1) + mm * (k0 + 1);
    const double2 *u1 = g.u1 + c0, *u2 = g.u2 + c0, *u3 = g.u3 + c0;
    const double rdij = tb.rd[i] * tb.rd[j], s = 1.0 / (g.h * g.h);
    double x0 = 0.0, x1 = 0.0, y0 = 0.0, y1 = 0.0;
    if (SEP) {
      x0 = tb.f[i];
      x1 = tb.f[q + i];
      y0 = tb.f[2 * q + j];
      y1 = tb.f[3 * q + j];
    }
    // of the plane below and this one: u1 and u2 at the point, u1 at x - 1, u2 at y - 1;
    // u3 at the point, x + 1 and y + 1
    double2 a0 = u1[-mm], a1 = u1[0], ax1 = u1[-1], b0 = u2[-mm], b1 = u2[0], by1 = u2[-m], d0 = u3[-mm],
            dx0 = u3[1 - mm], dy0 = u3[m - mm];
    for (int k = k0; k < k1; ++k, u1 += mm, u2 += mm, u3 += mm) {
      const double2 a2 = u1[mm], ax2 = u1[mm - 1], ayp = u1[m], aym = u1[-m], axyp = u1[m - 1];
      const double2 b2 = u2[mm], by2 = u2[mm - m], bxp = u2[1], bxm = u2[-1], bxpym = u2[1 - m];
      const double2 d1 = u3[0], dx1 = u3[1], dy1 = u3[m], dxm = u3[-1], dym = u3[-m];
      // backward difference (first index) of the forward difference (second) of u:
      // u(f - b) - u(-b) - u(f) + u(0)
      auto mix = [](double2 fb, double2 b_, double2 f, double2 o) {
        return make_double2(fb.x - b_.x - f.x + o.x, fb.y - b_.y - f.y + o.y);
      };
      auto sec = [](double2 c, double2 lo, double2 hi) {
        return make_double2(2.0 * c.x - lo.x - hi.x, 2.0 * c.y - lo.y - hi.y);
      };
      double2 A[3];
      const double2 U[3] = {a1, b1, d1};
      A[0] = csub<double>(csub<double>(cadd<double>(sec(a1, aym, ayp), sec(a1, a0, a2)), mix(bxpym, by1, bxp, b1)),
                          mix(dx0, d0, dx1, d1));
      A[1] = csub<double>(csub<double>(cadd<double>(sec(b1, bxm, bxp), sec(b1, b0, b2)), mix(axyp, ax1, ayp, a1)),
                          mix(dy0, d0, dy1, d1));
      A[2] = csub<double>(csub<double>(cadd<double>(sec(d1, dxm, dx1), sec(d1, dym, dy1)), mix(ax2, ax1, a2, a1)),
                          mix(by2, by1, b2, b1));
      double e[3];
      if (SEP) {
        const double z0 = tb.f[4 * q + k], z1 = tb.f[5 * q + k];
        e[0] = tb.c0 + tb.p0 * (x1 * y0 * z0);
        e[1] = tb.c0 + tb.p0 * (x0 * y1 * z0);
        e[2] = tb.c0 + tb.p0 * (x0 * y0 * z1);
      } else {
        yee_eps3(g, mt, tb, i, j, k, e);
      }
      double av = 0.0, bv = 0.0;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        A[c] = cscale<double>(A[c], s);
        const double2 B = cscale<double>(U[c], e[c]);
        const double2 R = csub<double>(A[c], cscale<double>(B, l6));
        av += U[c].x * A[c].x + U[c].y * A[c].y;  // Re(conj(u) Au)
        bv += U[c].x * B.x + U[c].y * B.y;
        acc.v[2] += cabs2<double>(A[c]);
        acc.v[3] += cabs2<double>(B);
        acc.v[4] += cabs2<double>(R);
        acc.v[5] += R.x * B.x + R.y * B.y;
      }
      const double rd = rdij * tb.rd[k];
      const size_t p = i + (size_t)q * (j + (size_t)q * k);
      a[p] = av * rd;
      b[p] = bv * rd;
      acc.v[0] += av;
      acc.v[1] += bv;
      a0 = a1;
      a1 = a2;
      ax1 = ax2;
      b0 = b1;
      b1 = b2;
      by1 = by2;
      d0 = d1;
      dx0 = dx1;
      dy0 = dy1;
    }
  }
  grid_sum_finalize<double, 6>(acc, partials, counter, [&](const Red<double, 6>& t) {
    for (int s2 = 0; s2 < 6; ++s2) out[s2] = t.v[s2];
  });
}

// x and y axes of the window for one kXyX x kXyY tile of plane blockIdx.z (zeros outside); in y
// each thread slides down four outputs of a column
constexpr int kXyX = 32, kXyY = 16;
__global__ void __launch_bounds__(256) k_lwrq_xy(const double* __restrict__ inA, const double* __restrict__ inB,
                                                 double* __restrict__ outA, double* __restrict__ outB, int q, Window w) {
  constexpr int R = kLwrqR, SX = kXyX + 2 * R, SY = kXyY + 2 * R;
  __shared__ double s[2][SY][SX];
  __shared__ double t[2][SY][kXyX];
  const int X0 = blockIdx.x * kXyX, Y0 = blockIdx.y * kXyY;
  const long long plane = (long long)blockIdx.z * q * q;
  const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
  for (int yy = wid; yy < SY; yy += 8) {
    const int y = Y0 + yy - R;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int xx = lane + 32 * h, x = X0 + xx - R;
      if (xx < SX) {
        const bool in = x >= 0 && x < q && y >= 0 && y < q;
        const long long p = plane + x + (long long)q * y;
        s[0][yy][xx] = in ? inA[p] : 0.0;
        s[1][yy][xx] = in ? inB[p] : 0.0;
      }
    }
  }
  __syncthreads();
  for (int e = wid; e < 2 * SY; e += 8) {
    const int f = e / SY, yy = e - f * SY;
    double v = 0.0;
#pragma unroll
    for (int d = 0; d < 2 * R + 1; ++d) v += w.k[d] * s[f][yy][lane + 2 * R - d];
    t[f][yy][lane] = v;
  }
  __syncthreads();
  const int f = wid / 4, yb = 4 * (wid % 4), x = X0 + lane;
  double col[4 + 2 * R];
#pragma unroll
  for (int r = 0; r < 4 + 2 * R; ++r) col[r] = t[f][yb + r][lane];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int y = Y0 + yb + r;
    double v = 0.0;
#pragma unroll
    for (int d = 0; d < 2 * R + 1; ++d) v += w.k[d] * col[r + 2 * R - d];
    if (x < q && y < q) (f ? outB : outA)[plane + x + (long long)q * y] = v;
  }
}

// z axis of the window, kZRun planes per thread (four at a time, their loads first), and the
// statistics of E and M with rho = E/M and l0 = sum a / sum b (out1, k_lwrq_ab): out [0] sum E,
// [1] sum M, [2] non-finite count, [3] sum M (rho - l0)^2, [4] sum M (rho - l0), [5] min M,
// [6] max M.  The window keeps the sums of a and b to rounding, so l0 is lambda3D to rounding
// and the sums about it lose nothing when the host moves them to lambda3D.  s0, s1: strides of
// the slices' two indices.
constexpr int kZRun = 24, kZStep = 4;
__global__ void __launch_bounds__(256) k_lwrq_z(const double* __restrict__ inA, const double* __restrict__ inB, int q,
                                                Window w, const double* __restrict__ out1, double* z0, double* x0, int s0,
                                                int s1, double* out, double* partials, unsigned* counter) {
  constexpr int R = kLwrqR, T = 2 * R + 1;
  __shared__ double red[8][7];
  __shared__ bool am_last;
  const int qq = q * q, col = blockIdx.x * 256 + threadIdx.x, c = (q - 1) / 2;
  const double l0 = out1[0] / out1[1];
  double v[7] = {0.0, 0.0, 0.0, 0.0, 0.0, INFINITY, -INFINITY};
  if (col < qq) {
    const int k0 = blockIdx.y * kZRun, k1 = min(q, k0 + kZRun), i = col % q, j = col / q;
    double wa[T - 1 + kZStep], wb[T - 1 + kZStep];  // planes k - R .. k + R + kZStep - 1
    auto load = [&](int d, int k) {
      const bool in = k >= 0 && k < q;
      wa[d] = in ? inA[(long long)k * qq + col] : 0.0;
      wb[d] = in ? inB[(long long)k * qq + col] : 0.0;
    };
#pragma unroll
    for (int d = 0; d < T - 1; ++d) load(d, k0 - R + d);
    for (int k = k0; k < k1; k += kZStep) {
#pragma unroll
      for (int u = 0; u < kZStep; ++u) load(T - 1 + u, k + R + u);
#pragma unroll
      for (int u = 0; u < kZStep; ++u) {
        if (k + u < k1) {
          double E = 0.0, M = 0.0;
#pragma unroll
          for (int d = 0; d < T; ++d) {  // tap d reads plane k + u + R - d
            E += w.k[d] * wa[u + T - 1 - d];
            M += w.k[d] * wb[u + T - 1 - d];
          }
          const double rho = E / M, dv = rho - l0;
          v[0] += E;
          v[1] += M;
          v[2] += (isfinite(E) && isfinite(M)) ? 0.0 : 1.0;
          v[3] += M * dv * dv;
          v[4] += M * dv;
          v[5] = fmin(v[5], M);
          v[6] = fmax(v[6], M);
          if (z0 && k + u == c) z0[i * s0 + j * s1] = rho;
          if (x0 && i == c) x0[j * s0 + (k + u) * s1] = rho;
        }
      }
#pragma unroll
      for (int d = 0; d < T - 1; ++d) {
        wa[d] = wa[d + kZStep];
        wb[d] = wb[d + kZStep];
      }
    }
  }
  // block, then grid, in a fixed order: five sums, a minimum and a maximum
  auto join = [](int s, double a, double b) { return s < 5 ? a + b : s == 5 ? fmin(a, b) : fmax(a, b); };
  auto block_join = [&](double* x) {  // result in x of threads 0..6 (value threadIdx.x in x[0])
#pragma unroll
    for (int s = 0; s < 7; ++s) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x[s] = join(s, x[s], __shfl_xor_sync(0xffffffffu, x[s], o));
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][s] = x[s];
    }
    __syncthreads();
    if (threadIdx.x < 7) {
      double r = red[0][threadIdx.x];
      for (int k = 1; k < 8; ++k) r = join(threadIdx.x, r, red[k][threadIdx.x]);
      x[0] = r;
    }
    __syncthreads();
  };
  block_join(v);
  const int nblk = gridDim.x * gridDim.y, blk = blockIdx.y * gridDim.x + blockIdx.x;
  if (threadIdx.x < 7) {
    partials[(size_t)blk * 7 + threadIdx.x] = v[0];
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) am_last = atomicAdd(counter, 1u) == (unsigned)nblk - 1;
  __syncthreads();
  if (!am_last) return;
  __threadfence();
  double u[7] = {0.0, 0.0, 0.0, 0.0, 0.0, INFINITY, -INFINITY};
  for (int i = threadIdx.x; i < nblk; i += 256)
#pragma unroll
    for (int s = 0; s < 7; ++s) u[s] = join(s, u[s], ((volatile double*)partials)[(size_t)i * 7 + s]);
  block_join(u);
  if (threadIdx.x < 7) out[threadIdx.x] = u[0];
  if (threadIdx.x == 0) *counter = 0u;
}

// relative deviation of the slices from lambda3D = sum E / sum M
// (exp3/compute_yee_lwrq_metrics_exp4.m:77-80)
__global__ void k_lwrq_dev(double* z0, double* x0, int n, const double* out) {
  const double lam = out[0] / out[1];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (z0) z0[i] = fabs(z0[i] - lam) / fabs(lam);
    if (x0) x0[i] = fabs(x0[i] - lam) / fabs(lam);
  }
}

// [0] ||Au - l3 Bu||^2, [1] ||Au - l6 Bu||^2
__global__ void __launch_bounds__(256) k_lwrq_resid(YeeGeom g, YeeMat mt, YeeTab tb, double l3, double l6, double* out,
                                                    double* partials, unsigned* counter) {
  const unsigned q = g.q, tot = q * q * q;
  Red<double, 2> acc{};
  for (unsigned p = blockIdx.x * blockDim.x + threadIdx.x; p < tot; p += gridDim.x * blockDim.x) {
    const unsigned r = p / q;
    const int i = (int)(p - r * q), k = (int)(r / q), j = (int)(r - k * q);
    double2 A[3], U[3];
    double e[3];
    yee_curl(g, i, j, k, A, U);
    yee_eps3(g, mt, tb, i, j, k, e);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double2 B = cscale<double>(U[c], e[c]);
      acc.v[0] += cabs2<double>(csub<double>(A[c], cscale<double>(B, l3)));
      acc.v[1] += cabs2<double>(csub<double>(A[c], cscale<double>(B, l6)));
    }
  }
  grid_sum_finalize<double, 2>(acc, partials, counter, [&](const Red<double, 2>& t) {
    out[0] = t.v[0];
    out[1] = t.v[1];
  });
}

}  // namespace fame

using namespace fame;

// rows: the slices row-major, the first index slowest (column-major otherwise)
static int lwrq_metrics(fame_ctx* ctx, const void* u1, const void* u2, const void* u3, int n, double h,
                        const double* P, int material_kind, double mp0, double mp1, double lambda6D, double* metrics,
                        double* slice_z0, double* slice_x0, bool rows) {
  if (!ctx || !u1 || !u2 || !u3 || !P || !metrics || n < 1 || !(h > 0.0) || (material_kind != 0 && material_kind != 1))
    return fail(FAME_ERR_INVALID, "fame_yee_lwrq_metrics arguments");
  if (!(std::fabs(lambda6D) > 0.0)) return fail(FAME_ERR_INVALID, "lambda6D must be nonzero");
  const int q = 2 * n + 1;
  const long long tot = (long long)q * q * q;
  cudaStream_t s = ctx->stream;
  YeeGeom g{(const double2*)u1, (const double2*)u2, (const double2*)u3, n, 2 * n + 3, q, h};
  YeeMat mt{};
  mt.kind = material_kind;
  mt.p0 = mp0;
  mt.p1 = mp1;
  for (int i = 0; i < 18; ++i) mt.P[i] = P[i];
  Window w{};
  const double sigma = 2.0 * h;
  for (int t = 0; t < 2 * kLwrqR + 1; ++t) {
    const double off = (t - kLwrqR) * h;
    w.k[t] = std::exp(-(off * off) / (sigma * sigma));
  }
  // 80 bytes of device memory per point: beyond any GPU's memory
  if (tot >= 0xF0000000LL) return fail(FAME_ERR_OOM, "fame_yee_lwrq_metrics: too many points");
  bool separable = true;
  for (int l = 0; l < 6; ++l) separable = separable && (P[l] != 0.0) + (P[l + 6] != 0.0) + (P[l + 12] != 0.0) <= 1;
  const int nb = lblocks(tot);
  const dim3 gab((q + kAbTile - 1) / kAbTile, (q + kAbTile - 1) / kAbTile, (q + kAbRun - 1) / kAbRun);
  const dim3 gxy((q + kXyX - 1) / kXyX, (q + kXyY - 1) / kXyY, q), gz((q * q + 255) / 256, (q + kZRun - 1) / kZRun);
  YeeTab tb{};
  double *a, *b, *T, *U, *sc, *part, *z0, *x0, *f;
  unsigned* counter;
  auto carve = [&](Carve& cv) {
    a = cv.take<double>(tot);
    b = cv.take<double>(tot);
    T = cv.take<double>(tot);
    U = cv.take<double>(tot);
    sc = cv.take<double>(16);
    part = cv.take<double>(std::max({(size_t)nb * 2, (size_t)gab.x * gab.y * gab.z * 6, (size_t)gz.x * gz.y * 7}));
    z0 = cv.take<double>((size_t)q * q);
    x0 = cv.take<double>((size_t)q * q);
    f = cv.take<double>((size_t)q * 6);
    tb.rd = cv.take<double>(q);
    counter = cv.take<unsigned>(1);
  };
  Carve cv;
  carve(cv);
  void* ws = nullptr;
  FAME_TRY(ctx_workspace(ctx, cv.used, &ws));
  cv = Carve{};
  cv.base = static_cast<char*>(ws);
  carve(cv);
  if (separable) tb.f = f;
  tb.c0 = material_kind == 0 ? 0.0 : 1.0;
  tb.p0 = mp0;
  FAME_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(unsigned), s));

  k_lwrq_tables<<<(7 * q + 63) / 64, 64, 0, s>>>(mt, tb, n, q, h, w);
  if (separable) k_lwrq_ab<true><<<gab, kAbTile * kAbTile, 0, s>>>(g, mt, tb, lambda6D, a, b, sc, part, counter);
  else k_lwrq_ab<false><<<gab, kAbTile * kAbTile, 0, s>>>(g, mt, tb, lambda6D, a, b, sc, part, counter);
  k_lwrq_xy<<<gxy, 256, 0, s>>>(a, b, T, U, q, w);
  k_lwrq_z<<<gz, 256, 0, s>>>(T, U, q, w, sc, slice_z0 ? z0 : nullptr, slice_x0 ? x0 : nullptr, rows ? q : 1,
                             rows ? 1 : q, sc + 6, part, counter);
  ::fame::count_launch(4);
  if (slice_z0 || slice_x0) {
    k_lwrq_dev<<<(q * q + 255) / 256, 256, 0, s>>>(slice_z0 ? z0 : nullptr, slice_x0 ? x0 : nullptr, q * q, sc + 6);
    ::fame::count_launch();
  }
  FAME_CUDA_TRY(cudaGetLastError());
  double hs[13];
  FAME_TRY(read_back(ctx, sc, hs, sizeof(hs)));
  const double sumA = hs[0], sumB = hs[1], nA = std::sqrt(hs[2]), nB = std::sqrt(hs[3]);
  if (!(sumB > 0.0)) return fail(FAME_ERR_INVALID, "Cropped Yee mass is not positive.");
  const double lamCrop = sumA / sumB, *st = hs + 6;
  if (st[2] != 0.0) return fail(FAME_ERR_NONFINITE, "Invalid LWRQ column-normalization or non-finite window sums.");
  const double sumE = st[0], sumM = st[1];
  const double lam = sumE / sumM;
  if (st[5] <= 1e-14 * st[6]) return fail(FAME_ERR_NONFINITE, "Nonpositive or numerically tiny local LWRQ mass encountered.");
  // sum M (rho - lam)^2 from the sums about lamCrop
  const double dl = lam - lamCrop;
  const double V = (st[3] - 2.0 * dl * st[4] + dl * dl * sumM) / (sumM * lam * lam);
  // ||Au - lam Bu||^2 = ||R - d Bu||^2 with R = Au - lambda6D Bu, d = lam - lambda6D: from the
  // sums while they do not cancel (at most two bits), else by a second pass over the field
  double h4[2] = {0.0, hs[4]};
  {
    const double d = lam - lambda6D;
    h4[0] = hs[4] - 2.0 * d * hs[5] + d * d * hs[3];
    if (!(h4[0] >= 0.25 * std::max(hs[4], d * d * hs[3]))) {
      k_lwrq_resid<<<nb, 256, 0, s>>>(g, mt, tb, lam, lambda6D, sc, part, counter);
      ::fame::count_launch();
      FAME_CUDA_TRY(cudaGetLastError());
      FAME_TRY(read_back(ctx, sc, h4, sizeof(h4)));
    }
  }
  const double tiny = 2.220446049250313e-16;
  const double partE = std::fabs(sumE - sumA) / std::max(std::fabs(sumA), tiny);
  const double partM = std::fabs(sumM - sumB) / std::max(std::fabs(sumB), tiny);
  metrics[0] = lamCrop;
  metrics[1] = lam;
  metrics[2] = std::sqrt(h4[0]) / (nA + std::fabs(lam) * nB);
  metrics[3] = std::sqrt(h4[1]) / (nA + std::fabs(lambda6D) * nB);
  metrics[4] = std::fabs(lam - lambda6D) / std::fabs(lambda6D);
  metrics[5] = V;
  metrics[6] = std::sqrt(std::max(V, 0.0));
  metrics[7] = std::max(partE, partM);
  metrics[8] = std::fabs(lam - lamCrop) / std::max(std::fabs(lamCrop), tiny);
  metrics[9] = sumB;
  // the slices into the caller's (pageable) arrays, on the stream
  if (slice_z0)
    FAME_CUDA_TRY(cudaMemcpyAsync(slice_z0, z0, (size_t)q * q * sizeof(double), cudaMemcpyDeviceToHost, s));
  if (slice_x0)
    FAME_CUDA_TRY(cudaMemcpyAsync(slice_x0, x0, (size_t)q * q * sizeof(double), cudaMemcpyDeviceToHost, s));
  if (slice_z0 || slice_x0) FAME_CUDA_TRY(cudaStreamSynchronize(s));
  return FAME_OK;
}

extern "C" {

int fame_yee_lwrq_metrics(fame_ctx* ctx, const void* u1, const void* u2, const void* u3, int n, double h,
                          const double* P, int material_kind, double mp0, double mp1, double lambda6D, double* metrics,
                          double* slice_z0, double* slice_x0) {
  return lwrq_metrics(ctx, u1, u2, u3, n, h, P, material_kind, mp0, mp1, lambda6D, metrics, slice_z0, slice_x0, false);
}

int fame_yee_lwrq_metrics_rows(fame_ctx* ctx, const void* u1, const void* u2, const void* u3, int n, double h,
                               const double* P, int material_kind, double mp0, double mp1, double lambda6D,
                               double* metrics, double* slice_z0, double* slice_x0) {
  return lwrq_metrics(ctx, u1, u2, u3, n, h, P, material_kind, mp0, mp1, lambda6D, metrics, slice_z0, slice_x0, true);
}

}  // extern "C"
