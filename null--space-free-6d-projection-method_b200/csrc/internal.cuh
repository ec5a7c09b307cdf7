// Internal handle layouts behind the opaque C ABI types.
#pragma once
#include <vector>
#include "fame_common.cuh"

struct fame_ctx {
  int device = 0;
  cudaStream_t own = nullptr;
  cudaStream_t stream = nullptr;
  cudaStream_t capture = nullptr;  // graph-capture stream when `stream` is the context's own
  cudaEvent_t ev = nullptr;
  void* pinned = nullptr;  // small host staging area (4 KB)
  void* ws = nullptr;      // grow-only device workspace (ctx_workspace)
  size_t ws_bytes = 0;
  std::vector<void*> allocs;
  unsigned faults_seen = 0;  // count of the device's reported faults at this context's last check
};

namespace fame {
struct MaterialRange;
}

struct fame_mass {
  fame_ctx* ctx = nullptr;
  int N = 0, n = 0;
  long long NF = 0;
  double* Et64 = nullptr;  // E / NF, FP64, pass-B tile order of the FP64 chains (k_tile_E)
  float* Et32 = nullptr;   // E / NF, FP32, pass-B tile order of the FP32 chains
  void* work = nullptr;    // mass_fields(NF) fields of complex128 scratch for the mass modes
  double* EtInv64 = nullptr;  // NF^-1 / E in the same tile order: the inverse mass operator
  float* EtInv32 = nullptr;
  fame::MaterialRange* range = nullptr;  // device: smallest and largest E, whether all E are positive and finite
  unsigned long long rangeWords[3] = {0, 0, 0};  // the same on the host once rangeRead (read_range)
  bool rangeRead = false;
  void* store = nullptr;                 // the one allocation behind the pointers above
  cudaEvent_t ready = nullptr;           // recorded behind the tables and range above
};

struct fame_basis {
  fame_ctx* ctx = nullptr;
  int N = 0, n = 0;
  long long NF = 0;
  // The cut matrix and the Bloch vector are real, so every diagonal of the basis is: they
  // are held as real arrays (half the bytes of the complex diagonals that fame_basis_get
  // hands out), and the passes scale by them instead of multiplying complex numbers:
  // FP32 Mhat action at N=7 531.5 -> 495.1 us, mixed N=5 solve 108.8 -> 105.3 ms.
  double* V[6] = {nullptr};  // V11,V21,V31,V12,V22,V32
  double *det = nullptr, *W1 = nullptr, *W2 = nullptr;
  double* D[4] = {nullptr};  // entries (r, c) of V1 / det V1 at 2 r + c (the pivoted V1 block)
  double *invC = nullptr, *Qq = nullptr, *q[3] = {nullptr};
  // line-order copies used inside solves (axis 1 slowest within each column)
  double *W1_l = nullptr, *W2_l = nullptr;
  double* invC_l = nullptr;
  float *W1f_l = nullptr, *W2f_l = nullptr;
  float* invCf_l = nullptr;
  void* store = nullptr;  // the one allocation behind the diagonals above
  void* work = nullptr;  // scratch of fame_apply_Mhat_C_scalar_compact (3 fields)
  size_t work_bytes = 0;
  double P[18] = {0};  // cut matrix, column-major 6 x 3
  int pivot = 2;       // physical component forming the V3 row of the explicit split
  fame_basis_info info{};
};

namespace fame {
// device allocation helpers recorded for cleanup by the owner
int dalloc(void** p, size_t bytes);
void dfree(void* p);
// While alive, dalloc/dfree of this host thread allocate from the library's memory
// pool in the order of stream s (all work on the blocks must be queued on s): frees
// then no longer synchronise the whole device.  Used by concurrent solves.
struct StreamOrderedAlloc {
  explicit StreamOrderedAlloc(cudaStream_t s);
  ~StreamOrderedAlloc();
  StreamOrderedAlloc(const StreamOrderedAlloc&) = delete;
  StreamOrderedAlloc& operator=(const StreamOrderedAlloc&) = delete;
  bool prev_on;
  cudaStream_t prev;
};
// copy a small device struct to host (synchronises the stream)
int read_back(fame_ctx* ctx, const void* dsrc, void* hdst, size_t bytes);
// FAME_ERR_CUDA if a bounded device-side wait gave up on ctx's device since the context's last
// check (or creation), also where another context's check found the device's fault word first
// and cleared it: the word does not say whose work was spoiled, so every context hears of it
// once.  Synchronises ctx's stream and clears the word.
int check_fault(fame_ctx* ctx);
// The same for one call whose own result rests on bounded waits: since the construction.
class FaultWatch {
  fame_ctx* ctx;
  unsigned seen;

 public:
  explicit FaultWatch(fame_ctx* ctx);
  int check();
};
// One block of the Gram-Schmidt tile kernel whose copies never come (lanczos.cu): the kernel
// sets the fault word and returns.
int selftest_gram_schmidt_wait(fame_ctx* ctx, unsigned poll_limit);
// At least `bytes` of device workspace owned by ctx, reused across calls (grown
// after a stream synchronisation); valid until the next call on the context.
int ctx_workspace(fame_ctx* ctx, size_t bytes, void** out);
// Whether M^{-1} is the same chain on 1/E to within a relative residual tol: every E positive
// and finite, and the chain's rounding (a few ulp of the largest field value, amplified by
// max E / min E when the residual is taken) below tol.  r: the handle's range, read back.
bool exact_inverse_ok(const MaterialRange& r, double tol);
// the handle's range on the host, with ctx's stream ordered behind the handle's set-up; the first
// call for a handle reads it from the device (the tables it describes never change)
int read_range(fame_ctx* ctx, fame_mass* m, MaterialRange* r);
// Taylor block moments on the tensor cores (taylor_tc.cu): launch shape and the
// FP32 partial-moment buffer (out_floats) it needs.
struct TaylorTcPlan {
  int Npad = 0, stages = 0, ntiles = 0, groups = 0;
  int nsplit = 1, Nc = 0;  // monomial columns split over nsplit CTAs of Nc columns each
  int Csep = 0;            // columns (of a CTA's Nc) whose cross products accumulate apart
  bool graded = false;     // the degree-p monomials take the last columns (taylor_tc_columns)
  long long Kc = 0, nslices = 0;
  size_t smem = 0, out_floats = 0;
};
TaylorTcPlan taylor_tc_plan(long long NF, int nB, int L, int p);
// col[a] (Npad entries): output column of monomial a (alist3: L triples a1, a2, a3).
void taylor_tc_columns(const TaylorTcPlan& plan, const int* alist3, int L, int p, int* col);
// Centers on a tensor grid: center b = (ax[b % m1], ax[m1 + (b / m1) % m2], ax[m1 + m2 + b / (m1 m2)]).
struct TaylorTcGrid {
  const double* ax = nullptr;  // device, m1 + m2 + m3 values (nullptr: centers are general)
  int m1 = 0, m2 = 0, m3 = 0;
};
constexpr int kTaylorTcMaxAxis = 24;  // m1 + m2 + m3 at most for the factorised phases
// gamma[b L + a] = coef[a] sum_j c_j e^{i q_j.r_b} q_j^a, with alistPacked[a] = a1 | a2 << 8 | a3 << 16.
int taylor_moments_tc(const TaylorTcPlan& plan, cudaStream_t s, const double2* c, const double* Q, long long NF,
                      const double* centers, int nB, const int* alistPacked, const int* col, int L, int p,
                      const double2* coef, float* out, double2* gamma, const TaylorTcGrid& grid);
// Batched complex GEMM C = A B (FP64 complex, element strides) as split-FP32
// (3xTF32) tcgen05 products (zgemm_tc.cu), in two steps: the operands are split into
// head/tail TF32 panels in the UMMA shared-memory layout (up to four operands per launch),
// then the GEMM streams the panels.  A panels: rows = M (complex rows m), batches = the
// GEMM's batch; B panels: rows = N (columns n), cols_for_b = N, batches = the distinct B
// operands (the GEMM uses B panel batch z / bdivB).  Strides are those of the FP64 operand:
// A (s_row, s_k) = (sam, sak), B = (sbn, sbk).  Panel buffers are 1024-byte aligned.
struct ZPanelJob {
  const double2* src;
  long long s_row, s_k, s_batch;
  int rows, K, batches;
  bool a_role;
  int cols_for_b;  // B role: the GEMM's N (sets the panel tile)
  unsigned char* out;
  int rows_pad = 0;  // panels of max(rows, rows_pad) rows, zeros from rows on
  int gather_n = 0;  // > 0: src is a coefficient vector of n^6 in natural order, element (k, row) gathered
};
size_t zpanel_bytes(const ZPanelJob& job);
int zsplit_panels(const ZPanelJob* jobs, int njobs, cudaStream_t s);
// The three contractions of the direct sum over split panels: u(x,y,z) of ncomp fields from the
// phase tables (Tx: A role, nx rows; Ty, Tz: B role) and the coefficients (B role, rows b + n2 c
// up to n2 cp); P1, P2 hold the intermediates' panels, bytes1 and bytes2 per field.
struct ZChainSizes {
  int cp, xs;  // n2 rounded up to whole stages; points of x per slab
  size_t bytes1, bytes2;
};
ZChainSizes zchain_sizes(int nx, int ny, int n2, int ncomp);
int zchain_3xtf32(const unsigned char* Tx, const unsigned char* Cp, const unsigned char* Ty, const unsigned char* Tz,
                  unsigned char* P1, unsigned char* P2, double2* u, int nx, int ny, int nz, int n2, int ncomp,
                  cudaStream_t s);
// A Hermitian operator on n-vectors of complex128 for the restarted Lanczos
// (lanczos.cu): y = A x on ctx's stream; *ws holds the reusable basis workspace.
struct LanczosOperator {
  fame_ctx* ctx;
  long long n;
  void** ws;
  int (*apply)(void* self, const double2* x, double2* y);
  void* self;
  // optional: reports an error of the last apply that was left for Lanczos to detect
  // (called when the step's Lanczos coefficients come back NaN/Inf)
  int (*check)(void* self) = nullptr;
};
int lanczos_run(const LanczosOperator& op, int nev, double tol, int maxiter, int p, const void* v0, double* theta,
                void* Y, fame_lanczos_info* info);
void lanczos_ws_release(void** ws);
// Consecutive 256-byte aligned pieces of one workspace.
struct Carve {
  size_t used = 0;
  char* base = nullptr;
  template <typename T> T* take(size_t count) {
    T* p = reinterpret_cast<T*>(base ? base + used : nullptr);
    used += (count * sizeof(T) + 255) / 256 * 256;
    return p;
  }
};
}  // namespace fame
