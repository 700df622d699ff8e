// h2g_noalloc.cu -- CalcRK! (src/NonUniform.jl:372-434) for callers that cannot allocate device
// memory.
//
// Who needs it: a caller whose device memory is owned by someone else -- a Julia program whose
// arrays live in CUDA.jl's pool, or a time-stepping loop that must not stall on
// cudaMalloc/cudaFree (both can synchronise the device).  Such a caller already holds the fields
// in device memory and only wants the residual r = b - A theta and its norm, without a solver
// handle (h2g_create allocates).  The call ends by copying ||r|| to the host and synchronising
// its stream, so it must not be issued while that stream is capturing a CUDA graph.
//
// The reduction of ||r|| needs scratch: one partial sum per row (j, k) of the interior, a ticket
// counter and the result.  They live in g_noalloc_scratch, a file-scope device array: every GPU
// that loads this library holds it (512 KiB) until the process exits.  Consequences:
//   * at most kNoAllocMaxRows = 65536 interior rows (NY * NZ) per call; larger grids are
//     rejected with H2G_BAD_ARG before any launch;
//   * all calls on a device share the array, the ticket (which each call counts round to zero) and the
//     result's place in the host page below, so the library runs them one after the other: a call holds its
//     device's lock from its launch until it has read the norm.  Work already in a call's stream must
//     therefore not wait for something that another thread does only after its own call here;
//   * the first call on a device looks up the array's device address (cudaGetSymbolAddress) with
//     that device current, and the first call of the process pins one page of the library's own host memory.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <mutex>

#include "../../include/h2g.h"

namespace h2gn {

constexpr int kNoAllocMaxRows = 65536;
constexpr int kSlots = kNoAllocMaxRows + 64;  // row partials, then ticket and result
constexpr int kTicket = kNoAllocMaxRows;      // unsigned int in a double slot
constexpr int kResult = kNoAllocMaxRows + 1;
constexpr int kThreads = 128;
constexpr int kMaxDevices = 64;

static __device__ __align__(256) double g_noalloc_scratch[kSlots];

// lambda_f (src/common.jl:35) and the stencil of CalcRK!, recomputed per cell in the reference's
// operation order (no FMA contraction: __dmul_rn / __dadd_rn / __ddiv_rn).
__device__ __forceinline__ double lam_f(double a, double b, double ma, double mb) {
  const double h = __ddiv_rn(__dmul_rn(__dmul_rn(2.0, a), b), __dadd_rn(a, b));
  return __dmul_rn(h, __dsub_rn(2.0, trunc(__dmul_rn(__dadd_rn(ma, mb), 0.5))));
}

struct Args {
  int MX, MY, MZ;
  const double *th, *b, *lam, *m, *rho, *cp, *ZC, *dZ;
  double dx, dy, dt, HC[6];
  int steady;
  double* r;
};

// Rows of one block: a thread walks up a column of them.
constexpr int kRows = 8;

// One block: kRows rows of a plane, 128 positions at a time.  What bounds it: theta, lambda, mask and b are
// read once and r written once (70 MB at 240x240x30, 11 us of HBM), but a cell's six conductances cost 14
// divisions, about 800 instructions.  Here 5 are left, side by side, and the next row's values are loaded
// while a row is computed:
//   * lambda_f(a, b) is symmetric to the last bit (2ab is exact up to its one rounding in either order), so a
//     cell takes its left face from the lane on its left and its lower face from the row before;
//   * the division by 2 is a product with 0.5 (exact), and the division by dz, the same for a whole plane,
//     two of Markstein's correction steps from 1/dz (div_by; the same quotient);
//   * a cell among six unmasked neighbours skips the convective terms, which are zero there.
// (Keeping a conductance while its two materials stay the same runs fewer divisions but one after another in
// a branch: slower.)
__device__ __forceinline__ double div_by(double a, double d, double y) {
  // P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
  // Dev. 34, 1990.  d and y = RN(1/d) are normal; a out of 2^+-400 (or d out of 2^+-100) takes the division.
  double q = __dmul_rn(a, y);
  double r = __fma_rn(d, q, -a);
  q = __fma_rn(-r, y, q);
  r = __fma_rn(d, q, -a);
  q = __fma_rn(-r, y, q);
  const double aa = fabs(a), ad = fabs(d);
  if (!(aa >= 0x1p-400 && aa <= 0x1p400 && ad >= 0x1p-100 && ad <= 0x1p100)) q = __ddiv_rn(a, d);
  return q;
}

// What a cell reads besides itself and the row before.
struct Row {
  double lxp, lyp, lzm, lzp, mxm, mxp, myp, mzm, mzp, txm, txp, typ, tzm, tzp, b;
};
__device__ __forceinline__ Row load_row(const Args& a, long long c, int MX, long long pl) {
  Row q;
  q.lxp = __ldg(a.lam + c + 1);
  q.lyp = __ldg(a.lam + c + MX);
  q.lzm = __ldg(a.lam + c - pl);
  q.lzp = __ldg(a.lam + c + pl);
  q.mxm = __ldg(a.m + c - 1);
  q.mxp = __ldg(a.m + c + 1);
  q.myp = __ldg(a.m + c + MX);
  q.mzm = __ldg(a.m + c - pl);
  q.mzp = __ldg(a.m + c + pl);
  q.txm = __ldg(a.th + c - 1);
  q.txp = __ldg(a.th + c + 1);
  q.typ = __ldg(a.th + c + MX);
  q.tzm = __ldg(a.th + c - pl);
  q.tzp = __ldg(a.th + c + pl);
  q.b = a.b[c];
  return q;
}

__global__ void __launch_bounds__(kThreads, 4) k_calcrk_rows(Args a, double* scratch,
                                                             double* __restrict__ out) {
  const int MX = a.MX, MY = a.MY, NX = MX - 2, NY = MY - 2, NZ = a.MZ - 2;
  const int groups = (NY + kRows - 1) / kRows;
  const int j0 = 1 + (int)(blockIdx.x % groups) * kRows, k = 1 + (int)(blockIdx.x / groups);
  const int rows = min(kRows, NY - j0 + 1);
  const long long pl = (long long)MX * MY;
  const double dx0 = a.dx, dy0 = a.dy, ddx = 1.0 / dx0, ddy = 1.0 / dy0, ddt = 1.0 / a.dt;
  const double dz_k = a.dZ[k];
  const double dzm = __dsub_rn(a.ZC[k], a.ZC[k - 1]), dzp = __dsub_rn(a.ZC[k + 1], a.ZC[k]);
  const double yzm = __ddiv_rn(1.0, dzm), yzp = __ddiv_rn(1.0, dzp);
  // convective factors of the six faces; with all of them finite a face to an unmasked cell adds a zero
  __shared__ double conv[6];
  __shared__ double acc[kRows][kThreads];
  if (threadIdx.x < 6) {
    const int f = threadIdx.x;
    conv[f] = __dmul_rn(__dmul_rn(a.HC[f], f < 2 ? dy0 : dx0), f < 4 ? dz_k : dy0);
  }
#pragma unroll
  for (int r = 0; r < kRows; ++r) acc[r][threadIdx.x] = 0.0;
  __syncthreads();
  const bool plain = isfinite(conv[0]) && isfinite(conv[1]) && isfinite(conv[2]) && isfinite(conv[3]) &&
                     isfinite(conv[4]) && isfinite(conv[5]);
  const double *L = a.lam, *M = a.m, *th = a.th;
  for (int i0 = 1; i0 <= NX; i0 += kThreads) {
    const int i = i0 + threadIdx.x;
    const bool on = i <= NX, first = (threadIdx.x & 31) == 0;
    const unsigned warp_on = __ballot_sync(0xffffffffu, on);
    if (!on) continue;
    long long c = (long long)i + (long long)MX * ((long long)j0 + (long long)MY * k);
    double l0 = L[c], m0 = M[c], t0 = th[c], tm = th[c - MX], mm = M[c - MX];
    double cym = __dmul_rn(__dmul_rn(__dmul_rn(lam_f(L[c - MX], l0, mm, m0), dx0), dz_k), ddy);
    Row n = load_row(a, c, MX, pl);
#pragma unroll 1
    for (int r = 0; r < rows; ++r) {
      const Row q = n;
      if (r + 1 < rows) n = load_row(a, c + MX, MX, pl);
      const double cxp = __dmul_rn(__dmul_rn(__dmul_rn(lam_f(q.lxp, l0, q.mxp, m0), dy0), dz_k), ddx);
      const double cyp = __dmul_rn(__dmul_rn(__dmul_rn(lam_f(q.lyp, l0, q.myp, m0), dx0), dz_k), ddy);
      const double czm = div_by(__dmul_rn(__dmul_rn(lam_f(q.lzm, l0, q.mzm, m0), dx0), dy0), dzm, yzm);
      const double czp = div_by(__dmul_rn(__dmul_rn(lam_f(q.lzp, l0, q.mzp, m0), dx0), dy0), dzp, yzp);
      double cxm = __shfl_up_sync(warp_on, cxp, 1);
      if (first) cxm = __dmul_rn(__dmul_rn(__dmul_rn(lam_f(L[c - 1], l0, q.mxm, m0), dy0), dz_k), ddx);
      double s = __dadd_rn(cxp, cxm);
      s = __dadd_rn(s, cyp);
      s = __dadd_rn(s, cym);
      s = __dadd_rn(s, czp);
      s = __dadd_rn(s, czm);
      const bool inner = plain && m0 == 1.0 && mm == 1.0 && q.mxm == 1.0 && q.mxp == 1.0 && q.myp == 1.0 &&
                         q.mzm == 1.0 && q.mzp == 1.0;
      if (!inner) {
        s = __dadd_rn(s, __dmul_rn(conv[1], __dsub_rn(1.0, q.mxp)));
        s = __dadd_rn(s, __dmul_rn(conv[0], __dsub_rn(1.0, q.mxm)));
        s = __dadd_rn(s, __dmul_rn(conv[3], __dsub_rn(1.0, q.myp)));
        s = __dadd_rn(s, __dmul_rn(conv[2], __dsub_rn(1.0, mm)));
        s = __dadd_rn(s, __dmul_rn(conv[5], __dsub_rn(1.0, q.mzp)));
        s = __dadd_rn(s, __dmul_rn(conv[4], __dsub_rn(1.0, q.mzm)));
      }
      double ap = 0.0;
      if (!a.steady)
        ap = __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(a.rho[c], a.cp[c]), dx0), dy0), dz_k), ddt);
      s = __dadd_rn(s, ap);
      const double dd = __dadd_rn(__dsub_rn(1.0, m0), __dmul_rn(s, m0));
      double ss = __dmul_rn(cxp, q.txp);
      ss = __dadd_rn(ss, __dmul_rn(cxm, q.txm));
      ss = __dadd_rn(ss, __dmul_rn(cyp, q.typ));
      ss = __dadd_rn(ss, __dmul_rn(cym, tm));
      ss = __dadd_rn(ss, __dmul_rn(czp, q.tzp));
      ss = __dadd_rn(ss, __dmul_rn(czm, q.tzm));
      const double rs = __dmul_rn(__dsub_rn(q.b, __dsub_rn(ss, __dmul_rn(dd, t0))), m0);
      a.r[c] = rs;
      acc[r][threadIdx.x] = __fma_rn(rs, rs, acc[r][threadIdx.x]);
      // on to the next row: the cell above becomes the cell
      tm = t0;
      mm = m0;
      cym = cyp;
      t0 = q.typ;
      l0 = q.lyp;
      m0 = q.myp;
      c += MX;
    }
  }
  // fixed-order sum of each row (row number: j fastest), then the last block adds the row partials in order
  __shared__ double sm[kRows][kThreads / 32];
  __shared__ int last;
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    double v = acc[r][threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sm[r][threadIdx.x >> 5] = v;
  }
  __syncthreads();
  if (threadIdx.x < rows) {
    double t = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) t += sm[threadIdx.x][w];
    scratch[(j0 - 1 + threadIdx.x) + NY * (k - 1)] = t;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0)
    last = atomicInc(reinterpret_cast<unsigned*>(scratch + kTicket), gridDim.x - 1) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  double t = 0.0;
  const int n = NY * NZ;
  for (int q0 = threadIdx.x; q0 < n; q0 += 16 * kThreads) {
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) v[u] = q0 + u * kThreads < n ? __ldcg(scratch + q0 + u * kThreads) : 0.0;
#pragma unroll
    for (int u = 0; u < 16; ++u) t += v[u];
  }
  for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) sm[0][threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    double tot = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) tot += sm[0][w];
    *out = sqrt(tot);
  }
}

// ||r|| is written straight into this page of host memory, pinned on first use (the copy of 8 bytes to
// pageable memory and the clearing of the ticket cost 25 us of a 48 us call on a small grid).
static __attribute__((aligned(4096))) volatile double g_result[512];
static double* g_result_dev[64] = {nullptr};

static std::mutex g_mu;
static std::mutex g_call_mu[kMaxDevices];  // one call at a time on a device
static double* g_scratch_ptr[kMaxDevices] = {nullptr};

// Device addresses of the scratch array and of the result page on the current device (looked up once per
// device; *result is null where the page cannot be pinned).
static int scratch_address(int dev, double** out, double** result) {
  std::lock_guard<std::mutex> lk(g_mu);
  if (dev < 0 || dev >= kMaxDevices) return H2G_UNSUPPORTED;
  if (!g_scratch_ptr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return H2G_CUDA_ERROR;
    g_scratch_ptr[dev] = static_cast<double*>(p);
  }
  *out = g_scratch_ptr[dev];
  if (!g_result_dev[dev]) {
    static bool pinned = false;
    void* host = const_cast<double*>(g_result);
    if (!pinned)
      pinned = cudaHostRegister(host, sizeof g_result, cudaHostRegisterMapped | cudaHostRegisterPortable) == cudaSuccess;
    void* p = nullptr;
    if (pinned && cudaHostGetDevicePointer(&p, host, 0) == cudaSuccess) g_result_dev[dev] = static_cast<double*>(p);
    cudaGetLastError();
  }
  *result = g_result_dev[dev];
  return H2G_OK;
}

}  // namespace h2gn

extern "C" int h2g_calcrk_noalloc(int MX, int MY, int MZ, const double* theta, const double* b, const double* lambda,
                                  const double* mask, const double* rho, const double* cp, const double* ZC,
                                  const double* dZ, double dx, double dy, double dt, const double* HC, int is_steady,
                                  double* r, double* res, void* stream) {
  using namespace h2gn;
  if (MX < 3 || MY < 3 || MZ < 3) return H2G_BAD_ARG;
  const long long rows = (long long)(MY - 2) * (MZ - 2);
  if (rows > kNoAllocMaxRows) {
    fprintf(stderr, "h2g_calcrk_noalloc: %lld interior rows (NY*NZ) exceed the scratch limit of %d\n", rows,
            kNoAllocMaxRows);
    return H2G_BAD_ARG;
  }
  if (!theta || !b || !lambda || !mask || !ZC || !dZ || !HC || !r || !res) return H2G_BAD_ARG;
  if (!is_steady && (!rho || !cp || !(dt > 0))) return H2G_BAD_ARG;
  if (!(dx > 0) || !(dy > 0)) return H2G_BAD_ARG;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return H2G_CUDA_ERROR;
  double* scratch = nullptr;
  double* result = nullptr;
  int rc = scratch_address(dev, &scratch, &result);
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  Args a;
  a.MX = MX; a.MY = MY; a.MZ = MZ;
  a.th = theta; a.b = b; a.lam = lambda; a.m = mask; a.rho = rho; a.cp = cp; a.ZC = ZC; a.dZ = dZ;
  a.dx = dx; a.dy = dy; a.dt = is_steady ? 1.0 : dt;
  for (int f = 0; f < 6; ++f) a.HC[f] = HC[f];
  a.steady = is_steady ? 1 : 0;
  a.r = r;
  std::lock_guard<std::mutex> one(g_call_mu[dev]);
  const unsigned blocks = (unsigned)(((MY - 2 + kRows - 1) / kRows) * (MZ - 2));
  k_calcrk_rows<<<blocks, kThreads, 0, st>>>(a, scratch, result ? result + dev : scratch + kResult);
  if (cudaGetLastError() != cudaSuccess) return H2G_CUDA_ERROR;
  if (!result && cudaMemcpyAsync(res, scratch + kResult, sizeof(double), cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return H2G_CUDA_ERROR;
  if (cudaStreamSynchronize(st) != cudaSuccess) return H2G_CUDA_ERROR;
  if (result) *res = g_result[dev];
  return H2G_OK;
}
