// h2g_device.cuh -- what every kernel file shares: the block shape of the stencil kernels, warp
// constants, relaxed loads and the scalar logic of the solver stages.
#pragma once
#include "h2g_internal.cuh"

namespace h2g {

// Rows per block of the stencil kernels with a reduction: fixes the order of the partial sums of the
// dot products, and with it the iteration count.
#ifndef H2G_BY
#define H2G_BY 8
#endif

constexpr int kBX = 32;       // threads along the half-row
constexpr int kBY = H2G_BY;   // rows per block
constexpr int kThreads = kBX * kBY;

constexpr unsigned kFull = 0xffffffffu;
constexpr unsigned kNoClass = 0xffffu;  // class index of a cell that is never updated

__device__ __forceinline__ unsigned int ld_relaxed_u32(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int ld_relaxed_s32(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void set_cond(cudaGraphConditionalHandle h, int use_cond, int value) {
  if (use_cond) cudaGraphSetConditional(h, value ? 1u : 0u);
}

// Scalar logic of each stage (runs on one thread).  Mirrors the control flow of PBiCGSTAB!
// (NonUniform.jl:262-349) and CG! (NonUniform.jl:131-225).
static __device__ void finish_stage(int stage, SolverState* st, double s1, double s2) {
  switch (stage) {
    case kStageInit:  // NonUniform.jl:263-294: res0, early return, rho of iteration 1
    case kStageInitCg: {
      const double res0 = sqrt(s1);
      st->res0 = res0;
      st->res = 1.0;
      st->rho = s1;
      st->rho_old = 1.0;
      st->alpha = 0.0;
      st->omega = 1.0;
      st->beta = 0.0;
      st->itr = 1;
      st->first = 1;
      st->stop = 0;
      st->converged = 0;
      st->reason = kRunning;
      if (res0 == 0.0) {
        st->stop = 1; st->converged = 1; st->itr = 0; st->res = 0.0; st->reason = kConverged;
      } else if (!isfinite(res0)) {
        st->stop = 1; st->itr = 0; st->reason = kNonFinite;
      } else if (stage == kStageInit && fabs(s1) < kFloatMin) {
        st->stop = 1; st->reason = kBreakdown;
      }
      break;
    }
    case kStageAlpha:  // NonUniform.jl:309
      st->alpha = __ddiv_rn(st->rho, s1);
      break;
    case kStageOmega:  // NonUniform.jl:320-326
      if (fabs(s1) < kFloatMin) { st->stop = 1; st->reason = kBreakdown; }
      else st->omega = __ddiv_rn(s2, s1);
      break;
    case kStageUpdate: {  // NonUniform.jl:331-346 and the top of the next iteration 289-299
      const double res = __ddiv_rn(sqrt(s1), st->res0);
      if (st->hist && st->itr >= 1 && st->itr <= st->hist_len) st->hist[st->itr - 1] = res;
      st->res = res;
      st->first = 0;
      if (res < st->tol) { st->stop = 1; st->converged = 1; st->reason = kConverged; break; }
      if (!isfinite(res) || (st->div_limit > 0.0 && res > st->div_limit)) {
        st->stop = 1; st->reason = kNonFinite; break;
      }
      if (st->itr >= st->maxItr) { st->stop = 1; st->reason = kMaxItr; break; }
      st->rho_old = st->rho;
      st->rho = s2;
      st->itr += 1;
      if (fabs(s2) < kFloatMin) { st->stop = 1; st->reason = kBreakdown; break; }
      st->beta = __ddiv_rn(__dmul_rn(__ddiv_rn(st->rho, st->rho_old), st->alpha), st->omega);
      break;
    }
    case kStageResid:
      st->scale = sqrt(s1);
      break;
    case kStageCgInit:  // NonUniform.jl:155
      st->rho_old = s1;
      st->itr = 1;
      break;
    case kStageCgAlpha:  // NonUniform.jl:168-176
      if (fabs(s1) < kFloatMin) { st->stop = 1; st->reason = kBreakdown; }
      else st->alpha = __ddiv_rn(st->rho_old, s1);
      break;
    case kStageCgRes: {  // NonUniform.jl:185-198
      const double res = __ddiv_rn(sqrt(s1), st->res0);
      if (st->hist && st->itr >= 1 && st->itr <= st->hist_len) st->hist[st->itr - 1] = res;
      st->res = res;
      if (res < st->tol) { st->stop = 1; st->converged = 1; st->reason = kConverged; break; }
      if (!isfinite(res) || (st->div_limit > 0.0 && res > st->div_limit)) { st->stop = 1; st->reason = kNonFinite; }
      break;
    }
    case kStageCgBeta:  // NonUniform.jl:206-222, then the loop bound
      if (fabs(s1) < kFloatMin) { st->stop = 1; st->reason = kBreakdown; break; }
      st->beta = __ddiv_rn(s1, st->rho_old);
      st->rho_old = s1;
      if (st->itr >= st->maxItr) { st->stop = 1; st->reason = kMaxItr; break; }
      st->itr += 1;
      break;
    case kStageDot:
      st->dot1 = s1;
      st->dot2 = s2;
      break;
    case kStageSorInit: {  // solveSOR! NonUniform.jl:1031-1035: res0 (1 if zero)
      double res0 = sqrt(s1);
      if (res0 == 0.0) res0 = 1.0;
      st->res0 = res0;
      st->res = 1.0;
      st->itr = 0;
      st->stop = 0;
      st->converged = 0;
      st->reason = kRunning;
      if (!isfinite(res0)) { st->stop = 1; st->reason = kNonFinite; }
      break;
    }
    case kStageSorHalf:  // colour 0 of rbsor! (NonUniform.jl:952-955)
      st->dot1 = s1;
      break;
    case kStageSorIter: {  // colour 1, then the test of solveSOR! (NonUniform.jl:1038-1048)
      const double res = __ddiv_rn(sqrt(__dadd_rn(st->dot1, s1)), st->res0);
      st->itr += 1;
      if (st->hist && st->itr <= st->hist_len) st->hist[st->itr - 1] = res;
      st->res = res;
      if (res < st->tol) { st->stop = 1; st->converged = 1; st->reason = kConverged; break; }
      if (!isfinite(res)) { st->stop = 1; st->reason = kNonFinite; break; }
      if (st->itr >= st->maxItr) { st->stop = 1; st->reason = kMaxItr; break; }
      break;
    }
    default:
      break;
  }
}

// a/d correctly rounded from y = RN(1/d), by two of Markstein's correction steps (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34,
// 1990): q + (a - d q) y with a fused remainder.  The first step makes q one of the two neighbours of
// a/d, the second rounds it correctly.  The remainder is formed negated, so that a zero keeps its
// sign.  Valid while neither the remainder nor the quotient leaves the normal range: d within
// 2^+-100 (checked when the class table is made) and a within 2^+-400 or zero; anything else takes the
// division (div_fix).
__device__ __forceinline__ double div_by(double a, double d, double y) {
  double q = __dmul_rn(a, y);
  double r = __fma_rn(d, q, -a);
  q = __fma_rn(-r, y, q);
  r = __fma_rn(d, q, -a);
  q = __fma_rn(-r, y, q);
  return q;
}
// Whether a is outside that range: its exponent is, and it is not zero (the residual far from a heat source,
// the lanes beyond the grid: a branch taken for those would be taken all the time).
__device__ __forceinline__ bool div_bad(double a) {
  const unsigned hi = (unsigned)__double2hiint(a), lo = (unsigned)__double2loint(a);
  return 2u * hi - 2u * ((1023u - 400u) << 20) > 2u * (800u << 20) && ((hi & 0x7fffffffu) | lo) != 0u;
}

}  // namespace h2g
