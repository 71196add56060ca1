// k_krylov.cu -- fused vector updates, deterministic reductions and the
// device-side control logic of the IMS Krylov accelerators.
//
// PCG: ims_base_cg (src/Solution/LinearMethods/ImsLinearBase.f90:30-240).
// BiCGSTAB: ims_base_bcgs (:249-549).  Convergence: ims_base_testcnvg
// (:1101-1146) and is_close (src/Utilities/MathUtil.f90:45-86).
//
// Each reduction kernel writes one partial per block; its last block to finish
// sums the partials in a fixed order (so results are reproducible run to
// run), then runs the scalar logic of the reference on the device: beta,
// alpha, omega with the +SIGN(DPREC, denominator) guard, the closure test,
// the stagnation exits and the NORTH residual schedule.  It sets Ctl::done,
// which every kernel of the loop checks first, and the WHILE condition of the
// CUDA graph, so the whole inner loop runs without a host round trip.
#include "gbims_internal.cuh"
#include "k_krylov.cuh"
#include "k_reduce.cuh"

namespace gb {

__device__ __forceinline__ double to_d(double v) { return v; }
__device__ __forceinline__ double to_d(float v) { return (double)v; }

// ---------------------------------------------------------------------------
// dot products: partial[b] (and partial[G+b])
// ---------------------------------------------------------------------------
template <typename TA, typename TB, int FIN>
__global__ void __launch_bounds__(kRedBlock) k_dot(int n, const TA *__restrict__ a,
                                                    const TB *__restrict__ b, double *part,
                                                    Ctl *ctl) {
  if (ctl->done) return;
  double v[1] = {0.0};
  // four rows per trip, loads first: the same summation order as one row
  // per trip, with four times the loads in flight
  constexpr int R = 4;
  const int stride = gridDim.x * blockDim.x;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + (R - 1) * stride < n; i += R * stride) {
    double ar[R], br[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      ar[r] = to_d(a[i + r * stride]);
      br[r] = to_d(b[i + r * stride]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) v[0] = fma(ar[r], br[r], v[0]);
  }
  for (; i < n; i += stride) v[0] = fma(to_d(a[i]), to_d(b[i]), v[0]);
  block_sum<1>(v);
  if (threadIdx.x == 0) part[blockIdx.x] = v[0];
  if (FIN && last_block(&ctl->fin, gridDim.x)) finish_dot<FIN>(ctl, part, gridDim.x);
}

// The mixed form's FP32 dot products, summed as above.
template <int FIN>
__global__ void __launch_bounds__(kRedBlock) k_dot32c(int n, const float *__restrict__ a,
                                                       const float *__restrict__ b, double *part,
                                                       Ctl *ctl) {
  if (ctl->done) return;
  CSum acc{0.f, 0.f};
  const int stride = gridDim.x * blockDim.x;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + stride < n; i += 2 * stride) {
    const float a0 = a[i], b0 = b[i], a1 = a[i + stride], b1 = b[i + stride];
    csum_prod(acc, a0, b0);
    csum_prod(acc, a1, b1);
  }
  if (i < n) csum_prod(acc, a[i], b[i]);
  double v[1] = {csum_value(acc)};
  block_sum<1>(v);
  if (threadIdx.x == 0) part[blockIdx.x] = v[0];
  if (FIN && last_block(&ctl->fin, gridDim.x)) finish_dot<FIN>(ctl, part, gridDim.x);
}

__global__ void __launch_bounds__(kRedBlock) k_dot_tq_tt32c(int n, const float *__restrict__ t,
                                                             const float *__restrict__ q,
                                                             double *part, Ctl *ctl) {
  if (ctl->done) return;
  CSum tq{0.f, 0.f}, tt{0.f, 0.f};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float ti = t[i];
    csum_prod(tq, ti, q[i]);
    csum_prod(tt, ti, ti);
  }
  double v[2] = {csum_value(tq), csum_value(tt)};
  block_sum<2>(v);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = v[0];
    part[gridDim.x + blockIdx.x] = v[1];
  }
  if (last_block(&ctl->fin, gridDim.x)) finish_dot<kFinOmega>(ctl, part, gridDim.x);
}

// t.q and t.t in one pass (BiCGSTAB omega)
template <typename T>
__global__ void __launch_bounds__(kRedBlock) k_dot_tq_tt(int n, const T *__restrict__ t,
                                                          const T *__restrict__ q, double *part,
                                                          Ctl *ctl) {
  if (ctl->done) return;
  double v[2] = {0.0, 0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double ti = to_d(t[i]);
    v[0] = fma(ti, to_d(q[i]), v[0]);
    v[1] = fma(ti, ti, v[1]);
  }
  block_sum<2>(v);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = v[0];
    part[gridDim.x + blockIdx.x] = v[1];
  }
  if (last_block(&ctl->fin, gridDim.x)) finish_dot<kFinOmega>(ctl, part, gridDim.x);
}

// sum of squares (L2NORM0)
template <typename T>
__global__ void __launch_bounds__(kRedBlock) k_sumsq(int n, const T *__restrict__ a,
                                                      double *__restrict__ part) {
  double v[1] = {0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double ai = to_d(a[i]);
    v[0] = fma(ai, ai, v[0]);
  }
  block_sum<1>(v);
  if (threadIdx.x == 0) part[blockIdx.x] = v[0];
}

// ---------------------------------------------------------------------------
// PCG
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_cg_pupdate64(int n, const double *__restrict__ z,
                                                      double *__restrict__ p,
                                                      const Ctl *__restrict__ ctl) {
  if (ctl->done) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  p[i] = ctl->first ? z[i] : fma(ctl->beta, p[i], z[i]);
}


__global__ void __launch_bounds__(256) k_cg_pupdate32(int n, const float *__restrict__ z,
                                                      float *__restrict__ p,
                                                      const Ctl *__restrict__ ctl) {
  if (ctl->done) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  p[i] = ctl->first ? z[i] : fmaf((float)ctl->beta, p[i], z[i]);
}

// The element of largest magnitude a thread has seen, kept as its bits: for
// finite doubles the order of the magnitudes' bit patterns is the order of the
// magnitudes, Inf and NaN come above all of them.  Integer instructions and
// selects only, in inline PTX: from the plain comparison the compiler made a
// branch per row, behind which the rows' FP64 instructions waited for one
// another (the update of 3.6 million rows took 68 us, without the maxima 35).
struct MaxBits {
  unsigned long long s = 0;
  int i = -1;
  __device__ __forceinline__ void take(double v, int row) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v);
    asm("{\n .reg .pred p;\n .reg .b64 a, b;\n"
        " and.b64 a, %2, 0x7fffffffffffffff;\n and.b64 b, %0, 0x7fffffffffffffff;\n"
        " setp.gt.u64 p, a, b;\n selp.b64 %0, %2, %0, p;\n selp.b32 %1, %3, %1, p;\n}"
        : "+l"(s), "+r"(i)
        : "l"(u), "r"(row));
  }
  __device__ __forceinline__ unsigned nonfinite() const { return ((unsigned)(s >> 32) & 0x7ff00000u) == 0x7ff00000u; }
  __device__ __forceinline__ double value() const { return __longlong_as_double((long long)s); }
  // of the block's partials, in any order of their rows
  __device__ __forceinline__ void merge(double v, int row) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v);
    const unsigned long long a = u & 0x7fffffffffffffffull, b = s & 0x7fffffffffffffffull;
    if (a > b || (a == b && (unsigned)row < (unsigned)i)) {
      s = u;
      i = row;
    }
  }
  // the largest of the warp, the smallest row among equals, in every lane
  __device__ __forceinline__ void warp() {
    const MaxLoc m = warp_maxloc(MaxLoc{value(), (long long)i});
    s = (unsigned long long)__double_as_longlong(m.val);
    i = (int)m.idx;
  }
};

struct MaxBits32 {
  unsigned s = 0;
  int i = -1;
  __device__ __forceinline__ void take(float v, int row) {
    asm("{\n .reg .pred p;\n .reg .b32 a, b;\n"
        " and.b32 a, %2, 0x7fffffff;\n and.b32 b, %0, 0x7fffffff;\n"
        " setp.gt.u32 p, a, b;\n selp.b32 %0, %2, %0, p;\n selp.b32 %1, %3, %1, p;\n}"
        : "+r"(s), "+r"(i)
        : "r"(__float_as_uint(v)), "r"(row));
  }
  __device__ __forceinline__ unsigned nonfinite() const { return (s & 0x7f800000u) == 0x7f800000u; }
  __device__ __forceinline__ double value() const { return widen(__uint_as_float(s)); }
  __device__ __forceinline__ void warp() {
    const unsigned all = 0xffffffffu, a = s & 0x7fffffffu;
    const unsigned top = __reduce_max_sync(all, a);
    const unsigned row = a == top ? (unsigned)i : all;  // -1 while nothing is above zero
    const unsigned first = __reduce_min_sync(all, row);
    const unsigned who = __ballot_sync(all, a == top && row == first);
    s = __shfl_sync(all, s, __ffs((int)who) - 1);
    i = (int)first;
  }
};

// A block's share of an update into its partial slots: [0]=l2 (when taken),
// [1]=dx val, [2]=dx idx, [3]=r val, [4]=r idx, [5]=nonfinite; the rows and
// the flag as integers.
template <bool L2, class M>
__device__ __forceinline__ void update_partials(double l2, unsigned nf, M mx, M mr, double *part, int G, int b) {
  __shared__ decltype(M::s) sv[2][kRedBlock / 32];
  __shared__ int si[2][kRedBlock / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  mx.warp();
  mr.warp();
  if (lane == 0) {
    sv[0][wid] = mx.s;
    si[0][wid] = mx.i;
    sv[1][wid] = mr.s;
    si[1][wid] = mr.i;
  }
  const int any = __syncthreads_or((int)nf);
  if (wid == 0) {
    mx = M();
    mr = M();
    if (lane < kRedBlock / 32) {
      mx.s = sv[0][lane];
      mx.i = si[0][lane];
      mr.s = sv[1][lane];
      mr.i = si[1][lane];
    }
    mx.warp();
    mr.warp();
  }
  double v[1] = {l2};
  if (L2) block_sum<1>(v);
  if (threadIdx.x == 0) {
    part[b] = L2 ? v[0] : 0.0;
    part[G + b] = mx.value();
    part[2 * G + b] = __longlong_as_double(mx.i);
    part[3 * G + b] = mr.value();
    part[4 * G + b] = __longlong_as_double(mr.i);
    part[5 * G + b] = __longlong_as_double(any ? 1 : 0);
  }
}

// Finalise an update reduction into ctl (deltax, rmax, l2norm, nonfinite).
template <bool L2>
__device__ __forceinline__ void ctl_finish_update(Ctl *ctl, const double *part, int G) {
  double l2[1] = {0.0};
  MaxBits mx, mr;
  int nf = 0;
  for (int i0 = threadIdx.x; i0 < G; i0 += kPartTrips * kRedBlock) {
    double l[kPartTrips], xv[kPartTrips], rv[kPartTrips];
    int xi[kPartTrips], ri[kPartTrips];
#pragma unroll
    for (int t = 0; t < kPartTrips; ++t) {
      const int i = i0 + t * kRedBlock;
      if (i < G) {
        if (L2) l[t] = __ldcg(part + i);
        xv[t] = __ldcg(part + G + i);
        xi[t] = __double2loint(__ldcg(part + 2 * G + i));
        rv[t] = __ldcg(part + 3 * G + i);
        ri[t] = __double2loint(__ldcg(part + 4 * G + i));
        nf |= __double2loint(__ldcg(part + 5 * G + i));
      }
    }
#pragma unroll
    for (int t = 0; t < kPartTrips; ++t)
      if (i0 + t * kRedBlock < G) {
        if (L2) l2[0] += l[t];
        mx.merge(xv[t], xi[t]);
        mr.merge(rv[t], ri[t]);
      }
  }
  nf = __syncthreads_or(nf);
  if (L2) block_sum<1>(l2);
  MaxLoc m[2] = {{mx.value(), mx.i}, {mr.value(), mr.i}};
  block_maxloc<2>(m);
  if (threadIdx.x == 0) {
    ctl->l2norm = L2 ? sqrt(l2[0]) : 0.0;
    ctl->deltax = m[0].val;
    ctl->xloc = m[0].idx;
    ctl->rmax = m[1].val;
    ctl->rloc = m[1].idx;
    if (nf) ctl->nonfinite = 1;
  }
}

// Writes this iteration's record (called by every thread of the control
// block after ctl_finish_update, before the iteration count advances):
// ITINNER, the CACCEL values (alpha; BiCGSTAB also omega) and per model
// dvmax, locdv, rmax, locr.  With one model these are the update's own
// maxima.  The reference resets the per-model locations every PCG iteration
// but not every BiCGSTAB iteration (ImsLinearBase.f90:141-146 against
// :432-435), so a BiCGSTAB model whose maxima stay zero keeps its last rows.
__device__ void ctl_record(Ctl *ctl, bool bcgs) {
  const int nm = ctl->rec_nmod, G = ctl->rec_G;
  const int row = ctl->iter - 1;
  const bool keep = row >= 0 && row < ctl->rec_cap;
  double *r = ctl->rec + (size_t)(keep ? row : 0) * (3 + 4 * nm);
  for (int im = 0; im < nm; ++im) {
    MaxLoc dx, rm;
    if (nm == 1) {
      dx.val = ctl->deltax; dx.idx = ctl->xloc;
      rm.val = ctl->rmax; rm.idx = ctl->rloc;
    } else {
      const double *pp = ctl->rec_part;
      dx = ctl_reduce_maxloc(pp + (4 * im) * G, pp + (4 * im + 1) * G, G);
      rm = ctl_reduce_maxloc(pp + (4 * im + 2) * G, pp + (4 * im + 3) * G, G);
    }
    if (threadIdx.x == 0) {
      long long ldv = dx.idx, lr = rm.idx;
      if (bcgs) {
        if (ldv < 0) ldv = ctl->rec_loc[2 * im];
        if (lr < 0) lr = ctl->rec_loc[2 * im + 1];
      }
      ctl->rec_loc[2 * im] = ldv;
      ctl->rec_loc[2 * im + 1] = lr;
      if (keep) {
        r[3 + 4 * im] = dx.val;
        r[4 + 4 * im] = (double)ldv;
        r[5 + 4 * im] = rm.val;
        r[6 + 4 * im] = (double)lr;
      }
    }
  }
  if (threadIdx.x == 0 && keep) {
    r[0] = (double)ctl->iter;
    r[1] = ctl->alpha;
    r[2] = bcgs ? ctl->omega : 0.0;
    ctl->rec_count = row + 1;
  }
}

// End of a PCG iteration: closure test and loop control (ImsLinearBase.f90:196-236).
template <bool L2>
__device__ __forceinline__ void ctl_cg_cnvg(Ctl *ctl, const double *part, int G, unsigned long long cond,
                              int use_cond) {
  if (ctl->done) {
    if (threadIdx.x == 0) set_loop(ctl, cond, use_cond);
    return;
  }
  ctl_finish_update<L2>(ctl, part, G);
  if (ctl->rec) ctl_record(ctl, false);
  if (threadIdx.x != 0) return;
  double rcnvg = (ctl->icnvgopt == 2 || ctl->icnvgopt == 3 || ctl->icnvgopt == 4) ? ctl->l2norm
                                                                                : ctl->rmax;
  int icnvg = ctl->icnvg;
  d_testcnvg(ctl->icnvgopt, icnvg, ctl->iter, ctl->deltax, rcnvg, ctl->l2norm0, ctl->epfact,
             ctl->dvclose, ctl->rclose);
  if (rcnvg == 0.0) icnvg = 1;
  ctl->icnvg = icnvg;
  ctl->north_due = 0;
  if (ctl->nonfinite) {
    ctl->done = 1;
  } else if (icnvg != 0) {
    ctl->done = 1;
    ctl->exit_reason = (rcnvg == 0.0) ? kExitExact : kExitClosure;
  } else if (d_is_close(ctl->rho, ctl->rho0)) {
    ctl->done = 1;
    ctl->exit_reason = kExitStagnation;
  } else {
    if (ctl->north > 0 && ((ctl->iter + 1) % ctl->north) == 0) ctl->north_due = 1;
    if (ctl->rho == 0.0) {
      ctl->done = 1;
      ctl->exit_reason = kExitZeroRho;
    } else {
      ctl->rho0 = ctl->rho;
      if (ctl->iter >= ctl->itmax) {
        ctl->done = 1;
        ctl->exit_reason = kExitItmax;
      } else {
        ctl->iter += 1;
        ctl->first = 0;
      }
    }
  }
  if (ctl->done && ctl->icnvg < 0) ctl->icnvg = 0;
  set_loop(ctl, cond, use_cond);
}
// End of a BiCGSTAB iteration (ImsLinearBase.f90:498-545).
template <bool L2>
__device__ __forceinline__ void ctl_bcgs_cnvg(Ctl *ctl, const double *part, int G, unsigned long long cond,
                                int use_cond) {
  if (ctl->done) {
    if (threadIdx.x == 0) set_loop(ctl, cond, use_cond);
    return;
  }
  ctl_finish_update<L2>(ctl, part, G);
  if (ctl->rec) ctl_record(ctl, true);
  if (threadIdx.x != 0) return;
  double rcnvg = (ctl->icnvgopt == 2 || ctl->icnvgopt == 3 || ctl->icnvgopt == 4) ? ctl->l2norm
                                                                                : ctl->rmax;
  int icnvg = ctl->icnvg;
  d_testcnvg(ctl->icnvgopt, icnvg, ctl->iter, ctl->deltax, rcnvg, ctl->l2norm0, ctl->epfact,
             ctl->dvclose, ctl->rclose);
  if (rcnvg == 0.0) icnvg = 1;
  ctl->icnvg = icnvg;
  ctl->north_due = 0;
  if (ctl->nonfinite) {
    ctl->done = 1;
  } else if (icnvg != 0) {
    ctl->done = 1;
    ctl->exit_reason = (rcnvg == 0.0) ? kExitExact : kExitClosure;
  } else if (d_is_close(ctl->rho, ctl->rho0) || d_is_close(ctl->alpha, ctl->alpha0) ||
             d_is_close(ctl->omega, ctl->omega0)) {
    ctl->done = 1;
    ctl->exit_reason = kExitStagnation;
  } else {
    if (ctl->north > 0 && ((ctl->iter + 1) % ctl->north) == 0) ctl->north_due = 1;
    if (ctl->rho * ctl->omega == 0.0) {
      ctl->done = 1;
      ctl->exit_reason = kExitZeroRho;
    } else {
      ctl->rho0 = ctl->rho;
      ctl->alpha0 = ctl->alpha;
      ctl->omega0 = ctl->omega;
      if (ctl->iter >= ctl->itmax) {
        ctl->done = 1;
        ctl->exit_reason = kExitItmax;
      } else {
        ctl->iter += 1;
        ctl->first = 0;
      }
    }
  }
  if (ctl->done && ctl->icnvg < 0) ctl->icnvg = 0;
  set_loop(ctl, cond, use_cond);
}
// End of a mixed inner iteration.  The IMS test runs on the recursive FP32
// residual; when it passes, or the recursive residual has dropped by
// refine_factor since the last refinement, the next true-residual check is
// requested (Ctl::north_due = 2) instead of stopping.
__device__ __forceinline__ void ctl_mixed_inner(Ctl *ctl, const double *part, int G, int bcgs,
                                  double refine_factor) {
  if (ctl->done) return;
  ctl_finish_update<true>(ctl, part, G);
  if (threadIdx.x != 0) return;
  double rcnvg = (ctl->icnvgopt == 2 || ctl->icnvgopt == 3 || ctl->icnvgopt == 4) ? ctl->l2norm
                                                                                : ctl->rmax;
  int icnvg = 0;
  d_testcnvg(ctl->icnvgopt, icnvg, ctl->iter, ctl->deltax, rcnvg, ctl->l2norm0, ctl->epfact,
             ctl->dvclose, ctl->rclose);
  if (rcnvg == 0.0) icnvg = 1;
  ctl->north_due = 0;
  // scratch[0]: L2 norm of the residual at the start of this refinement
  bool stag = d_is_close(ctl->rho, ctl->rho0);
  if (bcgs) stag = stag || d_is_close(ctl->alpha, ctl->alpha0) || d_is_close(ctl->omega, ctl->omega0);
  bool zero = bcgs ? (ctl->rho * ctl->omega == 0.0) : (ctl->rho == 0.0);
  if (ctl->nonfinite) {
    ctl->done = 1;
    return;
  }
  if (icnvg != 0 || ctl->l2norm <= refine_factor * ctl->scratch[0] || stag || zero) {
    ctl->north_due = 2;  // request the FP64 true residual
    // Every refinement restarts the recurrence from the true residual: with
    // FP32 search directions, continuing after a residual replacement costs
    // more iterations than a restart (measured on the 10M-cell case)
    (void)bcgs;
    ctl->restart_due = 1;
    ctl->scratch[1] = ctl->deltax;
    ctl->scratch[2] = (double)ctl->xloc;
  }
  ctl->rho0 = ctl->rho;
  ctl->alpha0 = ctl->alpha;
  ctl->omega0 = ctl->omega;
  if (ctl->north_due != 2) {
    if (ctl->iter >= ctl->itmax) {
      ctl->north_due = 2;  // final true-residual check at the iteration limit
      ctl->restart_due = 0;
      ctl->scratch[1] = ctl->deltax;
      ctl->scratch[2] = (double)ctl->xloc;
    } else {
      ctl->iter += 1;
      ctl->first = 0;
    }
  }
}
// Closure test on the FP64 true residual; restart the inner loop if needed.
__device__ __forceinline__ void ctl_refine(Ctl *ctl, const double *part, int G, unsigned long long cond,
                             int use_cond) {
  if (ctl->done || ctl->north_due != 2) {
    if (threadIdx.x == 0) set_loop(ctl, cond, use_cond);
    return;
  }
  double dsave = ctl->scratch[1];
  long long lsave = (long long)ctl->scratch[2];
  ctl_finish_update<true>(ctl, part, G);
  if (threadIdx.x != 0) return;
  ctl->deltax = dsave;
  ctl->xloc = lsave;
  double rcnvg = (ctl->icnvgopt == 2 || ctl->icnvgopt == 3 || ctl->icnvgopt == 4) ? ctl->l2norm
                                                                                : ctl->rmax;
  int icnvg = 0;
  d_testcnvg(ctl->icnvgopt, icnvg, ctl->iter, ctl->deltax, rcnvg, ctl->l2norm0, ctl->epfact,
             ctl->dvclose, ctl->rclose);
  if (rcnvg == 0.0) icnvg = 1;
  ctl->north_due = 0;
  if (ctl->nonfinite) {
    ctl->done = 1;
  } else if (icnvg > 0) {
    ctl->icnvg = 1;
    ctl->done = 1;
    ctl->exit_reason = (rcnvg == 0.0) ? kExitExact : kExitClosure;
  } else if (ctl->iter >= ctl->itmax) {
    ctl->icnvg = 0;
    ctl->done = 1;
    ctl->exit_reason = kExitItmax;
  } else {
    // The FP32 recurrence residual is replaced by the FP64 true residual and
    // the recurrence restarts from it (restart_due); a recurrence that
    // carried on instead, like the reference's NORTH residual refresh
    // (ImsLinearBase.f90:221-227), would keep its search direction.
    ctl->scratch[0] = ctl->l2norm;
    ctl->scratch[3] += 1.0;  // refinement count
    if (ctl->restart_due) {
      ctl->first = 1;
      ctl->rho0 = 0.0;
      ctl->alpha0 = 0.0;
      ctl->omega0 = 0.0;
    } else {
      ctl->first = 0;
    }
    ctl->iter += 1;
  }
  set_loop(ctl, cond, use_cond);
}
// The closure tests as kernels of their own, behind the per-model records.
template <bool L2>
__global__ void k_ctl_cg_cnvg(Ctl *ctl, const double *part, int G, unsigned long long cond,
                              int use_cond) {
  ctl_cg_cnvg<L2>(ctl, part, G, cond, use_cond);
}

template <bool L2>
__global__ void k_ctl_bcgs_cnvg(Ctl *ctl, const double *part, int G, unsigned long long cond,
                                int use_cond) {
  ctl_bcgs_cnvg<L2>(ctl, part, G, cond, use_cond);
}

// x += alpha*p ; d -= alpha*q ; max|alpha p|, max|d|, sum d^2 (FP64 path).
// partial slots: [0]=l2, [1]=dx val, [2]=dx idx, [3]=r val, [4]=r idx, [5]=nonfinite
// The sum of squares is taken only when the closure test reads it (L2 =
// true: RCLOSE options L2NORM_RCLOSE and RELATIVE_RCLOSE, ICNVGOPT 2-4); with
// the infinity-norm tests the reference computes it but never reads it
// inside the loop, and on GB300 it is a quarter of the kernel's FP64 work.
// p1: P alternates between p (even iterations) and p1 (odd ones), or null.
// FIN: the last block runs the closure test.
template <bool L2, bool FIN>
__global__ void __launch_bounds__(kRedBlock) k_cg_update64(int n, double *__restrict__ x,
                                                            double *__restrict__ d, const double *p,
                                                            const double *p1,
                                                            const double *__restrict__ q,
                                                            double *part, Ctl *ctl,
                                                            unsigned long long cond, int use_cond) {
  if (ctl->done) {
    if (FIN && blockIdx.x == 0 && threadIdx.x == 0) set_loop(ctl, cond, use_cond);
    return;
  }
  const double alpha = ctl->alpha;
  if (p1 && (ctl->iter & 1)) p = p1;
  double v[1] = {0.0};
  MaxBits mx, mr;
  // four rows per trip, their 16 loads issued before any row is used (the
  // same order of rows per thread as one row per trip, so the same sums and
  // maxima): the loads of a trip cover the latency of the FP64 work of the
  // trip before
  constexpr int R = 4;
  const int stride = gridDim.x * blockDim.x;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + (R - 1) * stride < n; i += R * stride) {
    double pr[R], xr[R], qr[R], dr[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = i + r * stride;
      pr[r] = __ldcs(p + j);
      xr[r] = __ldcs(x + j);
      qr[r] = __ldcs(q + j);
      dr[r] = __ldcs(d + j);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = i + r * stride;
      pr[r] = alpha * pr[r];
      x[j] = xr[r] + pr[r];
      dr[r] = fma(-alpha, qr[r], dr[r]);
      d[j] = dr[r];
      if (L2) v[0] = fma(dr[r], dr[r], v[0]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      mx.take(pr[r], i + r * stride);
      mr.take(dr[r], i + r * stride);
    }
  }
  for (; i < n; i += stride) {
    const double tv = alpha * p[i], di = fma(-alpha, q[i], d[i]);
    x[i] = x[i] + tv;
    d[i] = di;
    if (L2) v[0] = fma(di, di, v[0]);
    mx.take(tv, i);
    mr.take(di, i);
  }
  update_partials<L2>(v[0], mx.nonfinite() | mr.nonfinite(), mx, mr, part, gridDim.x, blockIdx.x);
  if (FIN && last_block(&ctl->fin, gridDim.x)) ctl_cg_cnvg<L2>(ctl, part, gridDim.x, cond, use_cond);
}


// Mixed inner update: the step alpha*p in FP32, added to the FP64 heads;
// d32 -= alpha*q32; the maxima on FP32 magnitudes (integer compares of the
// bit patterns) and the L2 sum compensated in FP32, so that the only FP64
// instructions per row are the conversion of the step and the head update.
template <bool FIN>
__global__ void __launch_bounds__(kRedBlock) k_cg_update_mixed(int n, double *__restrict__ x,
                                                                float *__restrict__ d, const float *p,
                                                                const float *p1,
                                                                const float *__restrict__ q,
                                                                double *part, Ctl *ctl,
                                                                double refine_factor) {
  if (ctl->done) return;
  const float alphaf = (float)ctl->alpha;
  if (p1 && (ctl->iter & 1)) p = p1;
  CSum l2{0.f, 0.f};
  MaxBits32 mx, mr;
  // four rows per trip, as in k_cg_update64
  constexpr int R = 4;
  const int stride = gridDim.x * blockDim.x;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + (R - 1) * stride < n; i += R * stride) {
    float pr[R], qr[R], dr[R];
    double xr[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = i + r * stride;
      pr[r] = p[j];
      xr[r] = x[j];
      qr[r] = q[j];
      dr[r] = d[j];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int j = i + r * stride;
      pr[r] = __fmul_rn(alphaf, pr[r]);
      x[j] = xr[r] + widen(pr[r]);
      dr[r] = __fmaf_rn(-alphaf, qr[r], dr[r]);
      d[j] = dr[r];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      mx.take(pr[r], i + r * stride);
      mr.take(dr[r], i + r * stride);
      csum_prod(l2, dr[r], dr[r]);
    }
  }
  for (; i < n; i += stride) {
    const float tv = __fmul_rn(alphaf, p[i]), di = __fmaf_rn(-alphaf, q[i], d[i]);
    x[i] = x[i] + widen(tv);
    d[i] = di;
    mx.take(tv, i);
    mr.take(di, i);
    csum_prod(l2, di, di);
  }
  update_partials<true>(csum_value(l2), mx.nonfinite() | mr.nonfinite(), mx, mr, part, gridDim.x, blockIdx.x);
  if (FIN && last_block(&ctl->fin, gridDim.x)) ctl_mixed_inner(ctl, part, gridDim.x, 0, refine_factor);
}

// Per-model maxima of one iteration for the inner records, when the solution
// has more than one model (CONVNMOD > 1; ImsLinearBase.f90:141-182 for PCG,
// :431-480 for BiCGSTAB): for each model's rows, the largest head change
// (the step the update kernel added: PCG alpha*p, BiCGSTAB alpha*phat +
// omega*qhat, times DSCALE when scaled) and the largest residual (divided by
// DSCALE when scaled), signed, with its row.  The step is recomputed with the
// update kernel's own expression, so the values are the ones the update
// compared.  Partial slots per model im: [4im] dx value, [4im+1] its row,
// [4im+2] r value, [4im+3] its row (G blocks each).
template <bool BCGS>
__global__ void __launch_bounds__(kRedBlock) k_rec_models(int nm, const int *__restrict__ modstart,
                                                          const double *__restrict__ p,
                                                          const double *__restrict__ q,
                                                          const double *__restrict__ d,
                                                          const double *__restrict__ dscale,
                                                          double *__restrict__ part,
                                                          const Ctl *__restrict__ ctl) {
  if (ctl->done) return;
  const double alpha = ctl->alpha, omega = ctl->omega;
  const int G = gridDim.x, b = blockIdx.x;
  for (int im = 0; im < nm; ++im) {
    MaxLoc m[2];
    m[0].val = 0.0; m[0].idx = -1; m[1].val = 0.0; m[1].idx = -1;
    const int r0 = modstart[im], r1 = modstart[im + 1];
    for (int i = r0 + b * blockDim.x + threadIdx.x; i < r1; i += G * blockDim.x) {
      double tv;
      if (BCGS) tv = fma(alpha, p[i], omega * q[i]);
      else tv = alpha * p[i];
      double rv = d[i];
      if (BCGS && dscale) {
        tv = tv * dscale[i];
        rv = rv / dscale[i];
      }
      if (absgt(tv, m[0].val)) { m[0].val = tv; m[0].idx = i; }
      if (absgt(rv, m[1].val)) { m[1].val = rv; m[1].idx = i; }
    }
    block_maxloc<2>(m);
    if (threadIdx.x == 0) {
      part[(4 * im) * G + b] = m[0].val;
      part[(4 * im + 1) * G + b] = (double)m[0].idx;
      part[(4 * im + 2) * G + b] = m[1].val;
      part[(4 * im + 3) * G + b] = (double)m[1].idx;
    }
  }
}

// ---------------------------------------------------------------------------
// BiCGSTAB
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) k_bcgs_p(int n, const T *__restrict__ d, T *__restrict__ p,
                                                const T *__restrict__ v,
                                                const Ctl *__restrict__ ctl) {
  if (ctl->done) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (ctl->first) {
    p[i] = d[i];
  } else {
    T beta = (T)ctl->beta, om = (T)ctl->omega0;
    T inner = fma(-om, v[i], p[i]);
    p[i] = fma(beta, inner, d[i]);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) k_bcgs_q(int n, const T *__restrict__ d, const T *__restrict__ v,
                                                T *__restrict__ q, const Ctl *__restrict__ ctl) {
  if (ctl->done) return;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  q[i] = fma(-(T)ctl->alpha, v[i], d[i]);
}

// x += alpha*phat + omega*qhat ; d = q - omega*t (ImsLinearBase.f90:428-480).
// L2 as in k_cg_update64.
// FIN 1: the last block runs the closure test; 2: the end of a mixed inner
// iteration.
template <typename T, bool L2, int FIN>
__global__ void __launch_bounds__(kRedBlock) k_bcgs_update(int n, double *__restrict__ x,
                                                            T *__restrict__ d,
                                                            const T *__restrict__ phat,
                                                            const T *__restrict__ qhat,
                                                            const T *__restrict__ q,
                                                            const T *__restrict__ t,
                                                            const double *__restrict__ dscale,
                                                            double *part, Ctl *ctl,
                                                            unsigned long long cond, int use_cond,
                                                            double refine_factor) {
  if (ctl->done) {
    if (FIN == 1 && blockIdx.x == 0 && threadIdx.x == 0) set_loop(ctl, cond, use_cond);
    return;
  }
  const double alpha = ctl->alpha, omega = ctl->omega;
  const T omegat = (T)omega;
  double v[1] = {0.0};
  MaxBits mx, mr;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double tv = fma(alpha, to_d(phat[i]), omega * to_d(qhat[i]));
    x[i] = x[i] + tv;
    if (dscale) tv = tv * dscale[i];
    mx.take(tv, i);
    T di = fma(-omegat, t[i], q[i]);
    d[i] = di;
    double rv = to_d(di);
    if (dscale) rv = rv / dscale[i];
    mr.take(rv, i);
    if (L2) v[0] = fma(rv, rv, v[0]);
  }
  update_partials<L2>(v[0], mx.nonfinite() | mr.nonfinite(), mx, mr, part, gridDim.x, blockIdx.x);
  if (FIN && last_block(&ctl->fin, gridDim.x)) {
    if (FIN == 1) ctl_bcgs_cnvg<L2>(ctl, part, gridDim.x, cond, use_cond);
    else ctl_mixed_inner(ctl, part, gridDim.x, 1, refine_factor);
  }
}

// ---------------------------------------------------------------------------
// Mixed precision: FP64 iterative refinement around the FP32 inner loop
// ---------------------------------------------------------------------------

// True residual r = b - A x in FP64 with its max|r| and L2, only when
// requested; the FP32 residual is reset from it.
__global__ void __launch_bounds__(kRedBlock) k_true_resid_stats(int n, const double *__restrict__ r,
                                                                 float *__restrict__ d32,
                                                                 float *__restrict__ dhat32,
                                                                 double *__restrict__ dhat64,
                                                                 const double *__restrict__ dscale,
                                                                 double *part, Ctl *ctl,
                                                                 unsigned long long cond,
                                                                 int use_cond) {
  if (ctl->done || ctl->north_due != 2) {
    if (blockIdx.x == 0 && threadIdx.x == 0) set_loop(ctl, cond, use_cond);
    return;
  }
  double v[1] = {0.0};
  unsigned nf = 0;
  MaxBits none, mr;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double ri = r[i];
    if (d32) d32[i] = (float)ri;
    if (ctl->restart_due) {  // BiCGSTAB shadow residual, on a restart
      if (dhat32) dhat32[i] = (float)ri;
      if (dhat64) dhat64[i] = ri;
    }
    if (dscale) ri = ri / dscale[i];    // BiCGSTAB reports the unscaled residual
    mr.take(ri, i);
    v[0] = fma(ri, ri, v[0]);
    nf |= nonfinite(ri);
  }
  update_partials<true>(v[0], nf, none, mr, part, gridDim.x, blockIdx.x);
  if (last_block(&ctl->fin, gridDim.x)) ctl_refine(ctl, part, gridDim.x, cond, use_cond);
}

// ---------------------------------------------------------------------------
// misc elementwise kernels
// ---------------------------------------------------------------------------
template <typename TD, typename TS>
__global__ void k_convert(int n, const TS *__restrict__ s, TD *__restrict__ d) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) d[i] = (TD)s[i];
}

__device__ void ctl_set_l2norm0(Ctl *ctl, const double *part, int G) {
  double s = ctl_reduce_sum(part, G);
  if (threadIdx.x == 0) {
    ctl->l2norm0 = sqrt(s);
    ctl->scratch[0] = ctl->l2norm0;
    if (ctl->l2norm0 == 0.0 || ctl->itmax <= 0) {
      ctl->done = 1;
      if (ctl->l2norm0 == 0.0) {
        ctl->icnvg = 1;
        ctl->exit_reason = kExitExact;
      }
    }
    if (!isfinite(s)) {
      ctl->nonfinite = 1;
      ctl->done = 1;
    }
  }
}
__global__ void k_ctl_set_l2norm0(Ctl *ctl, const double *part, int G) {
  ctl_set_l2norm0(ctl, part, G);
}
// The L2 norm of the final residual, for a loop that did not take it.
__global__ void k_ctl_set_l2norm(Ctl *ctl, const double *part, int G) {
  double s = ctl_reduce_sum(part, G);
  if (threadIdx.x == 0 && ctl->l2norm0 != 0.0) ctl->l2norm = sqrt(s);
}

// ---------------------------------------------------------------------------
// Batched ensemble: independent systems ("members") concatenated into one
// block-diagonal system and iterated in lockstep.  Rows are cut into chunks
// that never straddle two members; one chunk is one block of the vector
// kernels and owns one reduction partial per slot.  Member m's partials are
// laid out like a single solve's (slot k of its b-th chunk at
// part[8*mc[m] + k*Gm + b], Gm = its chunk count), so the per-member control
// logic is exactly the single-solve code above, run by block m.  A member
// whose Ctl is done skips all of its chunks; the loop ends when every member
// is done.
// ---------------------------------------------------------------------------
struct ChunkRef {
  int m, b, G, r0, r1;
};

__device__ __forceinline__ ChunkRef chunk_of(const BatchDev &B, int c) {
  ChunkRef r;
  r.m = B.cm[c];
  const int c0 = B.mc[r.m];
  r.b = c - c0;
  r.G = B.mc[r.m + 1] - c0;
  r.r0 = B.cr[c];
  r.r1 = B.cr[c + 1];
  return r;
}

__device__ __forceinline__ double *member_part(double *part, const BatchDev &B, int m) {
  return part + 8LL * B.mc[m];
}

// Rows a thread of a chunk's block handles: its loads are issued before any
// row is used.
constexpr int kChunkTrips = kChunkRows / kRedBlock;

template <int FIN>
__global__ void __launch_bounds__(kRedBlock) k_b_dot(BatchDev B, const double *__restrict__ a,
                                                     const double *__restrict__ b, double *part) {
  const ChunkRef c = chunk_of(B, blockIdx.x);
  Ctl *ctl = B.ctls + c.m;
  if (ctl->done) return;
  double v[1] = {0.0};
  double ar[kChunkTrips], br[kChunkTrips];
  const int i0 = c.r0 + threadIdx.x;
#pragma unroll
  for (int t = 0; t < kChunkTrips; ++t)
    if (i0 + t * kRedBlock < c.r1) {
      ar[t] = a[i0 + t * kRedBlock];
      br[t] = b[i0 + t * kRedBlock];
    }
#pragma unroll
  for (int t = 0; t < kChunkTrips; ++t)
    if (i0 + t * kRedBlock < c.r1) v[0] = fma(ar[t], br[t], v[0]);
  block_sum<1>(v);
  double *pm = member_part(part, B, c.m);
  if (threadIdx.x == 0) pm[c.b] = v[0];
  if (last_block(&ctl->fin, c.G)) finish_dot<FIN>(ctl, pm, c.G);
}

__global__ void __launch_bounds__(kRedBlock) k_b_sumsq(BatchDev B, const double *__restrict__ a,
                                                       double *__restrict__ part) {
  const ChunkRef c = chunk_of(B, blockIdx.x);
  double v[1] = {0.0};
  for (int i = c.r0 + threadIdx.x; i < c.r1; i += blockDim.x) v[0] = fma(a[i], a[i], v[0]);
  block_sum<1>(v);
  if (threadIdx.x == 0) member_part(part, B, c.m)[c.b] = v[0];
}

template <typename T>
__global__ void __launch_bounds__(kRedBlock) k_b_cg_pupdate(BatchDev B, const T *__restrict__ z,
                                                            T *__restrict__ p) {
  const ChunkRef c = chunk_of(B, blockIdx.x);
  const Ctl &ctl = B.ctls[c.m];
  if (ctl.done) return;
  const bool first = ctl.first;
  const double beta = ctl.beta;
  T zr[kChunkTrips], pr[kChunkTrips];
  const int i0 = c.r0 + threadIdx.x;
#pragma unroll
  for (int t = 0; t < kChunkTrips; ++t)
    if (i0 + t * kRedBlock < c.r1) {
      zr[t] = z[i0 + t * kRedBlock];
      pr[t] = p[i0 + t * kRedBlock];
    }
#pragma unroll
  for (int t = 0; t < kChunkTrips; ++t)
    if (i0 + t * kRedBlock < c.r1)
      p[i0 + t * kRedBlock] = first ? zr[t] : (T)fma((double)(T)beta, (double)pr[t], (double)zr[t]);
}

// The batch's own control block gets done = every member done; it gates the
// shared kernels (SpMV, preconditioner) and drives the WHILE condition.  By
// one block, after every member's control step.
__device__ __forceinline__ void batch_all_done(const BatchDev &B, Ctl *gctl, unsigned long long cond,
                                               int use_cond, int count_body) {
  int any = 0;
  for (int m = threadIdx.x; m < B.nm; m += blockDim.x) any |= !((volatile Ctl *)B.ctls)[m].done;
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) {
    if (!any) gctl->done = 1;
    if (count_body) set_loop(gctl, cond, use_cond);
  }
}

// x += alpha*p ; d -= alpha*q with the same partial slots as k_cg_update64
// (L2 as there); a member's last block runs its closure test, the launch's
// last block decides whether the batch goes on.  With a thread's eight rows
// one at a time the loads' latency and the FP64 work took turns (61 us on 1.7
// million rows).
template <bool L2>
__global__ void __launch_bounds__(kRedBlock) k_b_cg_update64(BatchDev B, double *__restrict__ x,
                                                             double *__restrict__ d,
                                                             const double *__restrict__ p,
                                                             const double *__restrict__ q,
                                                             double *part, Ctl *gctl,
                                                             unsigned long long cond, int use_cond) {
  const ChunkRef c = chunk_of(B, blockIdx.x);
  Ctl *ctl = B.ctls + c.m;
  if (!ctl->done) {
    const double alpha = ctl->alpha;
    double v[1] = {0.0};
    MaxBits mx, mr;
    const int row0 = B.mr[c.m];  // member-local row numbers for the maxima
    constexpr int R = 4;
#pragma unroll
    for (int h = 0; h < kChunkTrips / R; ++h) {
      double pr[R], xr[R], qr[R], dr[R];
      const int i0 = c.r0 + threadIdx.x + h * R * kRedBlock;
#pragma unroll
      for (int t = 0; t < R; ++t) {
        const int i = i0 + t * kRedBlock;
        if (i < c.r1) {
          pr[t] = p[i];
          xr[t] = x[i];
          qr[t] = q[i];
          dr[t] = d[i];
        }
      }
#pragma unroll
      for (int t = 0; t < R; ++t) {
        const int i = i0 + t * kRedBlock;
        if (i < c.r1) {
          pr[t] = alpha * pr[t];
          x[i] = xr[t] + pr[t];
          dr[t] = fma(-alpha, qr[t], dr[t]);
          d[i] = dr[t];
          if (L2) v[0] = fma(dr[t], dr[t], v[0]);
        }
      }
#pragma unroll
      for (int t = 0; t < R; ++t) {
        const int i = i0 + t * kRedBlock;
        if (i < c.r1) {
          mx.take(pr[t], i - row0);
          mr.take(dr[t], i - row0);
        }
      }
    }
    double *pm = member_part(part, B, c.m);
    update_partials<L2>(v[0], mx.nonfinite() | mr.nonfinite(), mx, mr, pm, c.G, c.b);
    if (last_block(&ctl->fin, c.G)) ctl_cg_cnvg<L2>(ctl, pm, c.G, 0ULL, 0);
  }
  __syncthreads();
  if (last_block(&gctl->fin, gridDim.x)) batch_all_done(B, gctl, cond, use_cond, 1);
}

__global__ void k_b_ctl_set_l2norm0(BatchDev B, const double *part) {
  const int m = blockIdx.x;
  ctl_set_l2norm0(B.ctls + m, part + 8LL * B.mc[m], B.mc[m + 1] - B.mc[m]);
}
// The L2 norm of a member's final residual, for a loop that did not take it.
__global__ void k_b_ctl_set_l2norm(BatchDev B, const double *part) {
  const int m = blockIdx.x;
  Ctl *ctl = B.ctls + m;
  const double s = ctl_reduce_sum(part + 8LL * B.mc[m], B.mc[m + 1] - B.mc[m]);
  if (threadIdx.x == 0 && ctl->l2norm0 != 0.0) ctl->l2norm = sqrt(s);
}

__global__ void k_b_all_done(BatchDev B, Ctl *gctl) { batch_all_done(B, gctl, 0ULL, 0, 0); }

// ---------------------------------------------------------------------------
// Batched mixed form: the single solve's FP32 inner loop and FP64
// refinement (k_dot32c, k_cg_pupdate32, k_cg_update_mixed,
// ctl_mixed_inner, k_true_resid_stats, ctl_refine) per member.
// ---------------------------------------------------------------------------
template <int FIN>
__global__ void __launch_bounds__(kRedBlock) k_b_dot32c(BatchDev B, const float *__restrict__ a,
                                                         const float *__restrict__ b, double *part) {
  const ChunkRef c = chunk_of(B, blockIdx.x);
  Ctl *ctl = B.ctls + c.m;
  if (ctl->done) return;
  CSum acc{0.f, 0.f};
  for (int i = c.r0 + threadIdx.x; i < c.r1; i += blockDim.x) csum_prod(acc, a[i], b[i]);
  double v[1] = {csum_value(acc)};
  block_sum<1>(v);
  double *pm = member_part(part, B, c.m);
  if (threadIdx.x == 0) pm[c.b] = v[0];
  if (last_block(&ctl->fin, c.G)) finish_dot<FIN>(ctl, pm, c.G);
}

__global__ void __launch_bounds__(kRedBlock) k_b_cg_pupdate32(BatchDev B, const float *__restrict__ z,
                                                               float *__restrict__ p) {
  const ChunkRef c = chunk_of(B, blockIdx.x);
  const Ctl &ctl = B.ctls[c.m];
  if (ctl.done) return;
  const bool first = ctl.first;
  const float beta = (float)ctl.beta;
  for (int i = c.r0 + threadIdx.x; i < c.r1; i += blockDim.x) p[i] = first ? z[i] : fmaf(beta, p[i], z[i]);
}

__global__ void __launch_bounds__(kRedBlock) k_b_cg_update_mixed(BatchDev B, double *__restrict__ x,
                                                                  float *__restrict__ d,
                                                                  const float *__restrict__ p,
                                                                  const float *__restrict__ q,
                                                                  double *part, double refine_factor) {
  const ChunkRef c = chunk_of(B, blockIdx.x);
  Ctl *ctl = B.ctls + c.m;
  if (ctl->done) return;
  const float alphaf = (float)ctl->alpha;
  const int row0 = B.mr[c.m];  // member-local row numbers for the maxima
  CSum l2{0.f, 0.f};
  MaxBits32 mx, mr;
  for (int i = c.r0 + threadIdx.x; i < c.r1; i += blockDim.x) {
    const float tv = __fmul_rn(alphaf, p[i]), di = __fmaf_rn(-alphaf, q[i], d[i]);
    x[i] = x[i] + widen(tv);
    d[i] = di;
    mx.take(tv, i - row0);
    mr.take(di, i - row0);
    csum_prod(l2, di, di);
  }
  double *pm = member_part(part, B, c.m);
  update_partials<true>(csum_value(l2), mx.nonfinite() | mr.nonfinite(), mx, mr, pm, c.G, c.b);
  if (last_block(&ctl->fin, c.G)) ctl_mixed_inner(ctl, pm, c.G, 0, refine_factor);
}

// The batch's own block asks for the FP64 true residual when any member
// does (the residual kernel is gated on it; members that are not due
// ignore it).
__global__ void k_b_any_due(BatchDev B, Ctl *gctl) {
  __shared__ int s_any;
  if (threadIdx.x == 0) s_any = 0;
  __syncthreads();
  for (int m = threadIdx.x; m < B.nm; m += blockDim.x)
    if (!B.ctls[m].done && B.ctls[m].north_due == 2) atomicOr(&s_any, 1);
  __syncthreads();
  if (threadIdx.x == 0) gctl->north_due = s_any ? 2 : 0;
}

__global__ void __launch_bounds__(kRedBlock) k_b_true_resid_stats(BatchDev B,
                                                                   const double *__restrict__ r,
                                                                   float *__restrict__ d32,
                                                                   double *part, Ctl *gctl,
                                                                   unsigned long long cond,
                                                                   int use_cond) {
  const ChunkRef c = chunk_of(B, blockIdx.x);
  Ctl *ctl = B.ctls + c.m;
  if (!ctl->done && ctl->north_due == 2) {
    const int row0 = B.mr[c.m];
    double v[1] = {0.0};
    unsigned nf = 0;
    MaxBits none, mr;
    for (int i = c.r0 + threadIdx.x; i < c.r1; i += blockDim.x) {
      const double ri = r[i];
      d32[i] = (float)ri;
      mr.take(ri, i - row0);
      v[0] = fma(ri, ri, v[0]);
      nf |= nonfinite(ri);
    }
    double *pm = member_part(part, B, c.m);
    update_partials<true>(v[0], nf, none, mr, pm, c.G, c.b);
    if (last_block(&ctl->fin, c.G)) ctl_refine(ctl, pm, c.G, 0ULL, 0);
  }
  __syncthreads();
  if (last_block(&gctl->fin, gridDim.x)) batch_all_done(B, gctl, cond, use_cond, 1);
}

// ---------------------------------------------------------------------------
// residual d = b - A x with its L2 norm and signed max|d| from CSR device
// arrays, one row per thread (ims_base_residual + dnrm2, ImsLinearBase.f90:
// 1291-1312; the row sum in amux order with FMA).  With one 256-row block per
// partial, the sum of squares rounds exactly like k_sumsq + k_ctl_set_l2norm0
// on a vector of at most kMaxRedBlocks * 256 rows.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kRedBlock) k_resid_rows(int n, const int *__restrict__ ia,
                                                           const int *__restrict__ ja, int base,
                                                           const double *__restrict__ amat,
                                                           const double *__restrict__ x,
                                                           const double *__restrict__ b,
                                                           double *__restrict__ resid,
                                                           double *__restrict__ part) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double v[1] = {0.0};
  MaxLoc m[1];
  m[0].val = 0.0;
  m[0].idx = -1;
  if (i < n) {
    double t = 0.0;
    const int k1 = ia[i + 1] - base;
    for (int k = ia[i] - base; k < k1; ++k) t = fma(amat[k], x[ja[k] - base], t);
    const double d = b[i] - t;
    if (resid) resid[i] = d;
    v[0] = fma(d, d, v[0]);
    if (absgt(d, m[0].val)) { m[0].val = d; m[0].idx = i; }
  }
  block_sum<1>(v);
  block_maxloc<1>(m);
  if (threadIdx.x == 0) {
    const int G = gridDim.x;
    part[blockIdx.x] = v[0];
    part[G + blockIdx.x] = m[0].val;
    part[2 * G + blockIdx.x] = (double)m[0].idx;
  }
}

// out[0] = L2 norm, out[1] = signed max|d|, out[2] = its row.
__global__ void k_resid_final(const double *__restrict__ part, int G, double *__restrict__ out) {
  const double s = ctl_reduce_sum(part, G);
  const MaxLoc m = ctl_reduce_maxloc(part + G, part + 2 * G, G);
  if (threadIdx.x == 0) {
    out[0] = sqrt(s);
    out[1] = m.val;
    out[2] = (double)m.idx;
  }
}

// ---------------------------------------------------------------------------
// host launch wrappers
// ---------------------------------------------------------------------------
void kr_residual_rows(int n, const int *ia, const int *ja, int base, const double *amat,
                      const double *x, const double *b, double *resid, double *part,
                      double *out, cudaStream_t st) {
  const int G = (n + kRedBlock - 1) / kRedBlock;
  k_resid_rows<<<G, kRedBlock, 0, st>>>(n, ia, ja, base, amat, x, b, resid, part);
  k_resid_final<<<1, kRedBlock, 0, st>>>(part, G, out);
}
static inline int egrid(int n) { return std::max(1, (n + 255) / 256); }

void kr_dot64(int n, const double *a, const double *b, double *part, int G, Ctl *ctl, Fin fin, cudaStream_t st) {
  auto *k = fin == kFinCgRho ? k_dot<double, double, kFinCgRho>
            : fin == kFinAlpha ? k_dot<double, double, kFinAlpha>
            : fin == kFinBcgsRho ? k_dot<double, double, kFinBcgsRho> : k_dot<double, double, kFinNone>;
  k<<<G, kRedBlock, 0, st>>>(n, a, b, part, ctl);
}
void kr_dot_tq_tt64(int n, const double *t, const double *q, double *part, int G, Ctl *ctl, cudaStream_t st) {
  k_dot_tq_tt<double><<<G, kRedBlock, 0, st>>>(n, t, q, part, ctl);
}
void kr_dot32(int n, const float *a, const float *b, double *part, int G, Ctl *ctl, Fin fin, cudaStream_t st) {
  auto *k = fin == kFinCgRho ? k_dot32c<kFinCgRho>
            : fin == kFinAlpha ? k_dot32c<kFinAlpha>
            : fin == kFinBcgsRho ? k_dot32c<kFinBcgsRho> : k_dot32c<kFinNone>;
  k<<<G, kRedBlock, 0, st>>>(n, a, b, part, ctl);
}
void kr_dot_tq_tt32(int n, const float *t, const float *q, double *part, int G, Ctl *ctl, cudaStream_t st) {
  k_dot_tq_tt32c<<<G, kRedBlock, 0, st>>>(n, t, q, part, ctl);
}
void kr_sumsq64(int n, const double *a, double *part, int G, cudaStream_t st) {
  k_sumsq<double><<<G, kRedBlock, 0, st>>>(n, a, part);
}
void kr_ctl_set_l2norm0(Ctl *ctl, const double *part, int G, cudaStream_t st) {
  k_ctl_set_l2norm0<<<1, kRedBlock, 0, st>>>(ctl, part, G);
}
void kr_ctl_set_l2norm(Ctl *ctl, const double *part, int G, cudaStream_t st) {
  k_ctl_set_l2norm<<<1, kRedBlock, 0, st>>>(ctl, part, G);
}
void kr_cg_pupdate64(int n, const double *z, double *p, const Ctl *ctl, cudaStream_t st) {
  k_cg_pupdate64<<<egrid(n), 256, 0, st>>>(n, z, p, ctl);
}
// Blocks of an update that only takes maxima, which come out the same from any
// grid: what is resident at once.
constexpr int kUpdateBlocks = 4 * kNumSM;

void kr_cg_update64(int n, double *x, double *d, const double *p, const double *p1, const double *q,
                    double *part, int G, Ctl *ctl, bool fin, unsigned long long cond, int use_cond,
                    cudaStream_t st, bool l2) {
  auto *k = l2 ? (fin ? k_cg_update64<true, true> : k_cg_update64<true, false>)
               : (fin ? k_cg_update64<false, true> : k_cg_update64<false, false>);
  if (!l2) G = std::min(G, kUpdateBlocks);
  k<<<G, kRedBlock, 0, st>>>(n, x, d, p, p1, q, part, ctl, cond, use_cond);
}
void kr_rec_models(bool bcgs, int nm, const int *modstart, const double *p, const double *q,
                   const double *d, const double *dscale, double *part, int G, const Ctl *ctl,
                   cudaStream_t st) {
  if (bcgs) k_rec_models<true><<<G, kRedBlock, 0, st>>>(nm, modstart, p, q, d, dscale, part, ctl);
  else k_rec_models<false><<<G, kRedBlock, 0, st>>>(nm, modstart, p, q, d, dscale, part, ctl);
}
void kr_cg_pupdate32(int n, const float *z, float *p, const Ctl *ctl, cudaStream_t st) {
  k_cg_pupdate32<<<egrid(n), 256, 0, st>>>(n, z, p, ctl);
}
void kr_cg_update_mixed(int n, double *x, float *d, const float *p, const float *p1, const float *q,
                        double *part, int G, Ctl *ctl, bool fin, double refine_factor, cudaStream_t st) {
  auto *k = fin ? k_cg_update_mixed<true> : k_cg_update_mixed<false>;
  k<<<G, kRedBlock, 0, st>>>(n, x, d, p, p1, q, part, ctl, refine_factor);
}
void kr_ctl_cg_cnvg(Ctl *ctl, const double *part, int G, unsigned long long cond, int use_cond,
                    cudaStream_t st, bool l2) {
  if (!l2) G = std::min(G, kUpdateBlocks);
  auto *k = l2 ? k_ctl_cg_cnvg<true> : k_ctl_cg_cnvg<false>;
  k<<<1, kRedBlock, 0, st>>>(ctl, part, G, cond, use_cond);
}
void kr_bcgs_p64(int n, const double *d, double *p, const double *v, const Ctl *ctl, cudaStream_t st) {
  k_bcgs_p<double><<<egrid(n), 256, 0, st>>>(n, d, p, v, ctl);
}
void kr_bcgs_q64(int n, const double *d, const double *v, double *q, const Ctl *ctl, cudaStream_t st) {
  k_bcgs_q<double><<<egrid(n), 256, 0, st>>>(n, d, v, q, ctl);
}
void kr_bcgs_p32(int n, const float *d, float *p, const float *v, const Ctl *ctl, cudaStream_t st) {
  k_bcgs_p<float><<<egrid(n), 256, 0, st>>>(n, d, p, v, ctl);
}
void kr_bcgs_q32(int n, const float *d, const float *v, float *q, const Ctl *ctl, cudaStream_t st) {
  k_bcgs_q<float><<<egrid(n), 256, 0, st>>>(n, d, v, q, ctl);
}
void kr_bcgs_update64(int n, double *x, double *d, const double *phat, const double *qhat,
                      const double *q, const double *t, const double *dscale, double *part, int G,
                      Ctl *ctl, bool fin, unsigned long long cond, int use_cond, cudaStream_t st, bool l2) {
  auto *k = l2 ? (fin ? k_bcgs_update<double, true, 1> : k_bcgs_update<double, true, 0>)
               : (fin ? k_bcgs_update<double, false, 1> : k_bcgs_update<double, false, 0>);
  if (!l2) G = std::min(G, kUpdateBlocks);
  k<<<G, kRedBlock, 0, st>>>(n, x, d, phat, qhat, q, t, dscale, part, ctl, cond, use_cond, 0.0);
}
void kr_bcgs_update32(int n, double *x, float *d, const float *phat, const float *qhat,
                      const float *q, const float *t, const double *dscale, double *part, int G,
                      Ctl *ctl, double refine_factor, cudaStream_t st) {
  k_bcgs_update<float, true, 2><<<G, kRedBlock, 0, st>>>(n, x, d, phat, qhat, q, t, dscale, part, ctl,
                                                         0ULL, 0, refine_factor);
}
void kr_ctl_bcgs_cnvg(Ctl *ctl, const double *part, int G, unsigned long long cond, int use_cond,
                      cudaStream_t st, bool l2) {
  if (!l2) G = std::min(G, kUpdateBlocks);
  auto *k = l2 ? k_ctl_bcgs_cnvg<true> : k_ctl_bcgs_cnvg<false>;
  k<<<1, kRedBlock, 0, st>>>(ctl, part, G, cond, use_cond);
}
void kr_true_resid_stats(int n, const double *r, float *d32, float *dhat32, double *dhat64,
                         const double *dscale, double *part, int G, Ctl *ctl,
                         unsigned long long cond, int use_cond, cudaStream_t st) {
  k_true_resid_stats<<<G, kRedBlock, 0, st>>>(n, r, d32, dhat32, dhat64, dscale, part, ctl, cond,
                                              use_cond);
}
void kr_f64_to_f32(int n, const double *s, float *d, cudaStream_t st) {
  k_convert<float, double><<<std::min(egrid(n), 4 * kNumSM), 256, 0, st>>>(n, s, d);
}
void kr_f32_to_f64(int n, const float *s, double *d, cudaStream_t st) {
  k_convert<double, float><<<std::min(egrid(n), 4 * kNumSM), 256, 0, st>>>(n, s, d);
}


// batched ensemble launchers
void kb_dot64(const BatchDev &B, const double *a, const double *b, double *part, Fin fin, cudaStream_t st) {
  auto *k = fin == kFinCgRho ? k_b_dot<kFinCgRho> : k_b_dot<kFinAlpha>;
  k<<<B.nchunks, kRedBlock, 0, st>>>(B, a, b, part);
}
void kb_sumsq64(const BatchDev &B, const double *a, double *part, cudaStream_t st) {
  k_b_sumsq<<<B.nchunks, kRedBlock, 0, st>>>(B, a, part);
}
void kb_cg_pupdate64(const BatchDev &B, const double *z, double *p, cudaStream_t st) {
  k_b_cg_pupdate<double><<<B.nchunks, kRedBlock, 0, st>>>(B, z, p);
}
void kb_cg_update64(const BatchDev &B, double *x, double *d, const double *p, const double *q,
                    double *part, Ctl *gctl, unsigned long long cond, int use_cond, cudaStream_t st,
                    bool l2) {
  auto *k = l2 ? k_b_cg_update64<true> : k_b_cg_update64<false>;
  k<<<B.nchunks, kRedBlock, 0, st>>>(B, x, d, p, q, part, gctl, cond, use_cond);
}
void kb_ctl_set_l2norm0(const BatchDev &B, const double *part, cudaStream_t st) {
  k_b_ctl_set_l2norm0<<<B.nm, kRedBlock, 0, st>>>(B, part);
}
void kb_ctl_set_l2norm(const BatchDev &B, const double *part, cudaStream_t st) {
  k_b_ctl_set_l2norm<<<B.nm, kRedBlock, 0, st>>>(B, part);
}
void kb_all_done(const BatchDev &B, Ctl *gctl, cudaStream_t st) {
  k_b_all_done<<<1, kRedBlock, 0, st>>>(B, gctl);
}
void kb_dot32(const BatchDev &B, const float *a, const float *b, double *part, Fin fin, cudaStream_t st) {
  auto *k = fin == kFinCgRho ? k_b_dot32c<kFinCgRho> : k_b_dot32c<kFinAlpha>;
  k<<<B.nchunks, kRedBlock, 0, st>>>(B, a, b, part);
}
void kb_cg_pupdate32(const BatchDev &B, const float *z, float *p, cudaStream_t st) {
  k_b_cg_pupdate32<<<B.nchunks, kRedBlock, 0, st>>>(B, z, p);
}
void kb_cg_update_mixed(const BatchDev &B, double *x, float *d, const float *p, const float *q,
                        double *part, double refine_factor, cudaStream_t st) {
  k_b_cg_update_mixed<<<B.nchunks, kRedBlock, 0, st>>>(B, x, d, p, q, part, refine_factor);
}
void kb_any_due(const BatchDev &B, Ctl *gctl, cudaStream_t st) {
  k_b_any_due<<<1, kRedBlock, 0, st>>>(B, gctl);
}
void kb_true_resid_stats(const BatchDev &B, const double *r, float *d32, double *part, Ctl *gctl,
                         unsigned long long cond, int use_cond, cudaStream_t st) {
  k_b_true_resid_stats<<<B.nchunks, kRedBlock, 0, st>>>(B, r, d32, part, gctl, cond, use_cond);
}

}  // namespace gb
