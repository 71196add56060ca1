// k_reduce.cuh -- block reductions, the Krylov scalars' control logic, and the
// last-block pattern: a reduction kernel's last block to finish sums the
// partials and runs the control step, instead of a single-block kernel after
// it.
#pragma once
#include <cfloat>

#include "gbims_internal.cuh"
#include "k_krylov.cuh"

namespace gb {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The entry of largest magnitude of a warp, the smallest row among equals (as
// maxloc_merge; {0, -1} when all are zero), in every lane.  Three integer
// warp reductions and a shuffle: merging pairs over five shuffle steps took
// some 400 instructions a warp, a good part of an update kernel on the sizes
// where a thread has one or two rows.
__device__ __forceinline__ MaxLoc warp_maxloc(MaxLoc m) {
  const unsigned all = 0xffffffffu;
  const unsigned hi = (unsigned)__double2hiint(m.val) & 0x7fffffffu, lo = (unsigned)__double2loint(m.val);
  const unsigned mh = __reduce_max_sync(all, hi);
  const unsigned ml = __reduce_max_sync(all, hi == mh ? lo : 0u);
  const bool best = hi == mh && lo == ml && (mh | ml) != 0u;
  const unsigned row = best ? (unsigned)m.idx : all;
  const unsigned mr = __reduce_min_sync(all, row);
  const unsigned who = __ballot_sync(all, best && row == mr);
  const int sh = __shfl_sync(all, __double2hiint(m.val), who ? __ffs((int)who) - 1 : 0);
  MaxLoc r;
  r.val = who ? __hiloint2double(sh, (int)ml) : 0.0;
  r.idx = mr == all ? -1 : (long long)mr;
  return r;
}

// Sum NV values over the block; thread 0 gets the results (fixed order).
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV]) {
  __shared__ double sh[NV][kRedBlock / 32];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double s = warp_sum(v[k]);
    if (lane == 0) sh[k][wid] = s;
  }
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double s = (lane < (int)(blockDim.x >> 5)) ? sh[k][lane] : 0.0;
      v[k] = warp_sum(s);
    }
  }
  __syncthreads();
}

template <int NM>
__device__ __forceinline__ void block_maxloc(MaxLoc (&m)[NM]) {
  __shared__ double shv[NM][kRedBlock / 32];
  __shared__ long long shi[NM][kRedBlock / 32];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NM; ++k) {
    MaxLoc r = warp_maxloc(m[k]);
    if (lane == 0) {
      shv[k][wid] = r.val;
      shi[k][wid] = r.idx;
    }
  }
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int k = 0; k < NM; ++k) {
      MaxLoc r;
      r.val = 0.0;
      r.idx = -1;
      if (lane < (int)(blockDim.x >> 5)) {
        r.val = shv[k][lane];
        r.idx = shi[k][lane];
      }
      m[k] = warp_maxloc(r);
    }
  }
  __syncthreads();
}

// 1 if v is Inf or NaN, tested on the exponent bits with integer
// instructions: on GB300 every FP64 instruction (a compare included) goes
// through the narrow FP64 pipe, which bounds the vector updates otherwise.
__device__ __forceinline__ unsigned nonfinite(double v) {
  return ((unsigned)__double2hiint(v) & 0x7ff00000u) == 0x7ff00000u;
}
__device__ __forceinline__ unsigned nonfinite(float v) {
  return (__float_as_uint(v) & 0x7f800000u) == 0x7f800000u;
}

// Sums of FP32 products with FP64-like accuracy and no FP64 instruction per
// element (on GB300 those run on a narrow pipe): each product is split
// exactly into p + e (p = x*y rounded, e = fma(x, y, -p)), and the p are
// added with Neumaier's compensated summation, their rounding errors and
// the e collected in c.  The pair enters the FP64 reductions as
// (double)s + (double)c.  Explicit _rn operations keep the compiler from
// contracting the splitting steps.
struct CSum {
  float s, c;
};
__device__ __forceinline__ void csum_add(CSum &a, float p) {
  const float t = __fadd_rn(a.s, p);
  const float bp = __fsub_rn(t, a.s);
  a.c = __fadd_rn(a.c, __fadd_rn(__fsub_rn(a.s, __fsub_rn(t, bp)), __fsub_rn(p, bp)));
  a.s = t;
}
__device__ __forceinline__ void csum_prod(CSum &a, float x, float y) {
  const float p = __fmul_rn(x, y);
  const float e = __fmaf_rn(x, y, -p);
  csum_add(a, p);
  a.c = __fadd_rn(a.c, e);
}
__device__ __forceinline__ double csum_value(const CSum &a) { return (double)a.s + (double)a.c; }

// ---------------------------------------------------------------------------
// partial-sum finalisation: by one block, after all partials are written (read
// past L1: the block may be one of the grid that wrote them)
// ---------------------------------------------------------------------------
static __device__ __forceinline__ double ctl_reduce_sum(const double *part, int G) {
  double v[1] = {0.0};
  for (int i = threadIdx.x; i < G; i += blockDim.x) v[0] += __ldcg(part + i);
  block_sum<1>(v);
  return v[0];  // valid in thread 0
}

static __device__ __forceinline__ MaxLoc ctl_reduce_maxloc(const double *pv, const double *pi, int G) {
  MaxLoc m[1];
  m[0].val = 0.0;
  m[0].idx = -1;
  for (int i = threadIdx.x; i < G; i += blockDim.x) {
    MaxLoc b;
    b.val = __ldcg(pv + i);
    b.idx = (long long)__ldcg(pi + i);
    maxloc_merge(m[0], b);
  }
  block_maxloc<1>(m);
  return m[0];
}

__device__ __forceinline__ bool d_is_close(double a, double b) {
  if (a == b) return true;
  double tol = 100.0 * DBL_EPSILON * fmax(fabs(a), fabs(b));
  if (tol < 0.0) tol = 0.0;
  return fabs(a - b) <= tol;
}

__device__ __forceinline__ void d_testcnvg(int icnvgopt, int &icnvg, int iiter, double dvmax,
                                           double rmax, double rmax0, double epfact,
                                           double dvclose, double rclose) {
  if (icnvgopt == 0) {
    if (fabs(dvmax) <= dvclose && fabs(rmax) <= rclose) icnvg = 1;
  } else if (icnvgopt == 1) {
    if (fabs(dvmax) <= dvclose && fabs(rmax) <= rclose) icnvg = (iiter == 1) ? 1 : -1;
  } else if (icnvgopt == 2) {
    if (fabs(dvmax) <= dvclose || rmax <= rclose) icnvg = 1;
    else if (rmax <= rmax0 * epfact) icnvg = -1;
  } else if (icnvgopt == 3) {
    if (fabs(dvmax) <= dvclose) icnvg = 1;
    else if (rmax <= rmax0 * rclose) icnvg = -1;
  } else if (icnvgopt == 4) {
    if (fabs(dvmax) <= dvclose && rmax <= rclose) icnvg = 1;
    else if (rmax <= rmax0 * epfact) icnvg = -1;
  }
}

__device__ __forceinline__ double sign_dprec(double den) { return copysign(DBL_EPSILON, den); }

// Sets the WHILE condition of the graph.  Independently of the IMS exit logic,
// the loop is cut after 2*itmax + 16 bodies, so no input can keep the device
// looping.
__device__ __forceinline__ void set_loop(Ctl *ctl, unsigned long long cond, int use_cond) {
  ctl->bodies += 1;
  if (ctl->bodies > 2 * ctl->itmax + 16 && !ctl->done) {
    ctl->done = 1;
    ctl->guard_tripped = 1;
  }
  if (use_cond) cudaGraphSetConditional((cudaGraphConditionalHandle)cond, ctl->done ? 0u : 1u);
}

static __device__ __forceinline__ void ctl_cg_rho(Ctl *ctl, const double *part, int G) {
  if (ctl->done) return;
  double s = ctl_reduce_sum(part, G);
  if (threadIdx.x == 0) {
    ctl->rho = s;
    ctl->beta = ctl->first ? 0.0 : s / ctl->rho0;
  }
}
static __device__ __forceinline__ void ctl_alpha(Ctl *ctl, const double *part, int G) {
  if (ctl->done) return;
  double s = ctl_reduce_sum(part, G);
  if (threadIdx.x == 0) {
    double den = s + sign_dprec(s);
    ctl->alpha = ctl->rho / den;
  }
}
static __device__ __forceinline__ void ctl_bcgs_rho(Ctl *ctl, const double *part, int G) {
  if (ctl->done) return;
  double s = ctl_reduce_sum(part, G);
  if (threadIdx.x == 0) {
    ctl->rho = s;
    if (!ctl->first) ctl->beta = (s / ctl->rho0) * (ctl->alpha0 / ctl->omega0);
  }
}
static __device__ __forceinline__ void ctl_omega(Ctl *ctl, const double *part, int G) {
  if (ctl->done) return;
  double num = ctl_reduce_sum(part, G);
  double den = ctl_reduce_sum(part + G, G);
  if (threadIdx.x == 0) {
    den = den + sign_dprec(den);
    ctl->omega = num / den;
  }
}
// True in the one block of a launch (of the nblocks that share the counter)
// that comes here last; what the others wrote before is visible to it.  The
// counter wraps to zero for the next launch.  Thread 0 writes a block's
// partials.  The partials are summed by the same code in the same order as in
// a kernel of its own, so the scalars do not depend on which block it is.
__device__ __forceinline__ bool last_block(unsigned *counter, unsigned nblocks) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicInc(counter, nblocks - 1) == nblocks - 1;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

template <int FIN>
__device__ __forceinline__ void finish_dot(Ctl *ctl, const double *part, int G) {
  if (FIN == kFinCgRho) ctl_cg_rho(ctl, part, G);
  if (FIN == kFinAlpha) ctl_alpha(ctl, part, G);
  if (FIN == kFinBcgsRho) ctl_bcgs_rho(ctl, part, G);
  if (FIN == kFinOmega) ctl_omega(ctl, part, G);
}

}  // namespace gb
