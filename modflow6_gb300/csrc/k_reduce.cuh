// k_reduce.cuh -- block reductions, the Krylov scalars' control logic, and the
// last-block pattern: a reduction kernel's last block to finish sums the
// partials and runs the control step, instead of a single-block kernel after
// it.
#pragma once
#include <cfloat>

#include "gbims_internal.cuh"
#include "k_krylov.cuh"

namespace gb {

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

// Sum NV values over a block of kRedBlock threads, for its thread 0 (fixed
// order: within a warp lanes 16, 8, 4, 2, 1 apart, then warps 4, 2, 1 apart).
// One warp adds all of them, eight values a lane from shared memory: an FP64
// instruction holds its sub-partition's pipe about 75 cycles however many
// lanes take part, and this tree is 12 full instructions where every warp's own
// shuffle tree made 45, which with eight blocks an SM was a third of a dot
// product: on 400,000 rows 8.2 -> 6.2 us, on 3.6 million 14.3 -> 11.9.
// The warp that adds differs between the blocks of an SM, which are a
// multiple of the SM count apart, or next to one another: its number sets the
// sub-partition.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV]) {
  constexpr int kWarps = kRedBlock / 32, kPitch = 36;  // pitch: no bank conflicts
  static_assert(kWarps == 8, "the tree below is written for eight warps");
  __shared__ double sh[NV][kWarps * kPitch];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k) sh[k][wid * kPitch + lane] = v[k];
  __syncthreads();
  if (wid == (int)((blockIdx.x + blockIdx.x / kNumSM) % kWarps)) {
    double t[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const double *s = sh[k] + (lane >> 2) * kPitch + (lane & 3);  // four lanes a warp's values
      double a[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = s[4 * j];
#pragma unroll
      for (int j = 0; j < 4; ++j) a[j] = a[j] + a[j + 4];
      t[k] = (a[0] + a[2]) + (a[1] + a[3]);
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      t[k] += __shfl_xor_sync(0xffffffffu, t[k], 2);
      t[k] += __shfl_xor_sync(0xffffffffu, t[k], 1);
      t[k] += __shfl_xor_sync(0xffffffffu, t[k], 16);
      t[k] += __shfl_xor_sync(0xffffffffu, t[k], 8);
      t[k] += __shfl_xor_sync(0xffffffffu, t[k], 4);
      if (lane == 0) sh[k][0] = t[k];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {  // which also is the one to write here next
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = sh[k][0];
  }
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
// (double)f with integer instructions: the conversion runs on the FP64 pipe,
// like an addition.  With the sums and the maxima's partials as integers, the
// mixed form's update went from 12.3 to 8.2 us on 400,000 rows and from 24.7
// to 15.6 on 3.6 million.
__device__ __forceinline__ double widen(float f) {
  const unsigned u = __float_as_uint(f), sign = u & 0x80000000u, e = u & 0x7f800000u;
  unsigned m = u & 0x7fffffffu;
  unsigned up = 0x38000000u;  // exponent bias 1023 for 127
  if (e == 0x7f800000u) up = 0x70000000u;
  if (e == 0u) {
    if (m == 0u) return __hiloint2double((int)sign, 0);
    const unsigned shift = (unsigned)__clz((int)m) - 8u;  // subnormal
    m = m << shift;  // its leading one adds one to the exponent
    up = 0x38000000u - (shift << 20);
  }
  return __hiloint2double((int)(sign | ((m >> 3) + up)), (int)(m << 29));
}
__device__ __forceinline__ double csum_value(const CSum &a) { return widen(a.s) + widen(a.c); }

// ---------------------------------------------------------------------------
// partial-sum finalisation: by one block, after all partials are written (read
// past L1: the block may be one of the grid that wrote them)
// ---------------------------------------------------------------------------
constexpr int kPartTrips = (kMaxRedBlocks + kRedBlock - 1) / kRedBlock;  // all of a grid's partials

static __device__ __forceinline__ double ctl_reduce_sum(const double *part, int G) {
  double v[1] = {0.0};
  for (int i0 = threadIdx.x; i0 < G; i0 += kPartTrips * kRedBlock) {
    double p[kPartTrips];
#pragma unroll
    for (int t = 0; t < kPartTrips; ++t)
      if (i0 + t * kRedBlock < G) p[t] = __ldcg(part + i0 + t * kRedBlock);
#pragma unroll
    for (int t = 0; t < kPartTrips; ++t)
      if (i0 + t * kRedBlock < G) v[0] += p[t];
  }
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
