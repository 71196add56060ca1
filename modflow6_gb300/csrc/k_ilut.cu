// k_ilut.cu -- ILUT / MILUT factorisation on the GPU.
//
// ilut (src/Utilities/Libraries/sparskit2/ilut.f90:48-462, Saad's dual
// threshold ILU with MODFLOW's relaxation of the dropped sum and its pivot
// guard) restated for one warp per row.  Row ii depends only on the U rows
// of the earlier rows it eliminates, and those are known only once its own
// elimination reaches them (fill brings new ones), so rows are not levelled
// ahead of time: every warp claims the next row from a counter and, before
// it eliminates row jrow, waits for jrow's completion word.  Rows are claimed
// in increasing order, so the lowest unfinished claimed row never waits on an
// unclaimed one and every wait ends; each wait is still bounded (kWaitCycles) and
// gives up when the attempt is void (a pivot failed, an error was raised).
//
// The working row follows the reference's bookkeeping where it decides the
// result: the elimination takes the smallest remaining column each time; the
// multipliers are kept in elimination order, the U candidates in the order
// they entered the row (the row's own upper entries in JA order, then the
// fill as it appears); dropped terms are summed in the reference's order; the
// lfil largest multipliers and the lfil - 1 largest U entries are chosen by
// the same partial quick-sort (qsplit, :519-581), whose output order is the
// storage order and so the summation order of the triangular solves.  Every
// operation is rounded on its own (no FMA), as in the CPU code.
//
// Output: per row, in padded slots (lfil L entries, lfil - 1 U entries), the
// kept columns and values, their counts and the inverse pivot.  The host
// turns the counts into the IAPC/JAPC layout of the ILU0 preconditioner and
// k_ilut_scatter moves the values there, so the general patterns' sweeps apply
// ILUT unchanged (lusol, :465-516, is the ilu0a pair of sweeps).
#include "gbims_internal.cuh"
#include "k_llword.cuh"
#include <algorithm>
#include <climits>

namespace gb {
namespace {

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_release_u32(unsigned *p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ bool attempt_void(const IlutStatus *s) {
  const volatile IlutStatus *vs = s;
  return vs->pivot_fail != INT_MAX || vs->err != 0;
}

__device__ __forceinline__ void raise_error(IlutStatus *s, int code, int row) {
  if (atomicCAS(&s->err, 0, code) == 0) atomicExch(&s->err_row, row);
}

// Waits until row r of this factorisation is complete; every lane acquires.
// False (in all lanes) when the attempt became void or the wait ran out (then
// an error is raised).
__device__ __forceinline__ bool wait_row(const IlutDev &I, int r) {
  unsigned turns = 0;
  while (!__all_sync(0xffffffffu, ld_acquire_u32(I.rdone + r) == I.epoch)) {
    if ((++turns & 63u) != 0) continue;
    if (!__all_sync(0xffffffffu, !attempt_void(I.stat))) return false;
    if (turns > (1u << 22)) {  // L2 round trips: seconds
      raise_error(I.stat, kIlutErrWait, r);
      return false;
    }
  }
  return true;
}

__device__ __forceinline__ unsigned long long magnitude(double v) {
  return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffULL;
}

// Partial quick-sort by decreasing magnitude around the ncut-th entry
// (1-based): the arrangement qsplit leaves, entry for entry.  One lane works,
// in shared memory.  Magnitudes are compared as integers (an FP64 comparison
// takes 77 cycles); NaN, which the reference's > never selects, counts as
// zero.
__device__ __forceinline__ unsigned long long split_key(double v) {
  const unsigned long long m = magnitude(v);
  return m > 0x7ff0000000000000ULL ? 0ULL : m;
}
__device__ void split_by_magnitude(int n, double *a, int *ind, int ncut) {
  int first = 0, last = n - 1;
  const int cut = ncut - 1;
  if (cut < first || cut > last) return;
  for (;;) {
    int mid = first;
    const double kv = a[mid];
    const bool knan = magnitude(kv) > 0x7ff0000000000000ULL;
    const unsigned long long key = magnitude(kv);
    for (int j = first + 1; j <= last; ++j) {
      const double v = a[j];
      if (!knan && split_key(v) > key) {
        ++mid;
        const double t = a[mid];
        a[mid] = v;
        a[j] = t;
        const int it = ind[mid];
        ind[mid] = ind[j];
        ind[j] = it;
      }
    }
    const double t = a[mid];
    a[mid] = a[first];
    a[first] = t;
    const int it = ind[mid];
    ind[mid] = ind[first];
    ind[first] = it;
    if (mid == cut) return;
    if (mid > cut) last = mid - 1;
    else first = mid + 1;
  }
}

// The working row of a warp: L candidates (kGone once eliminated), the
// multipliers kept so far in elimination order, and the U candidates in the
// order they entered.
constexpr int kGone = INT_MAX;
struct alignas(16) IlutRow {
  int lc[kIlutCap], mc[kIlutCap], uc[kIlutCap];
  double lv[kIlutCap], mv[kIlutCap], uv[kIlutCap];
};
constexpr int kIlutWarps = 4;

// Position of column c among the first `count` of a list, or -1: each lane
// its own c, four entries a load.  Entries past `count` are never equal to a
// column (the lists are filled with -1 ahead).
__device__ __forceinline__ int find_column(const int *list, int count, int c) {
  int p = -1;
  for (int t = 0; t < count; t += 4) {
    const int4 v = *reinterpret_cast<const int4 *>(list + t);
    if (v.x == c) p = t;
    if (v.y == c) p = t + 1;
    if (v.z == c) p = t + 2;
    if (v.w == c) p = t + 3;
  }
  return p;
}

// A warp per row.  Bound by the chain of rows (with fill, row (i, j) of a grid
// waits for (i-1, j+1), so a level is j + 2i and more): what a row does after
// its last wait counts.  The smallest remaining column comes from a warp
// minimum, the U entries of an eliminated row are taken by a lane each, and
// the working row lies in shared memory; with a thread per row, searching its
// lists in local memory and waiting for the thread beside it, a row took some
// 150 us of the chain (39 ms for ILUT(5, 1e-4) on 6 x 60 x 60 cells).
__global__ void __launch_bounds__(32 * kIlutWarps) k_ilut_factor(
    IlutDev I, const int *__restrict__ ia, const int *__restrict__ ja, const double *__restrict__ a,
    double droptol, double relax, double delta, int izero) {
  extern __shared__ __align__(16) unsigned char smem_ilut[];
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  IlutRow &W = reinterpret_cast<IlutRow *>(smem_ilut)[threadIdx.x >> 5];
  const int lfil = I.lfil;
  for (;;) {
    if (!__all_sync(all, !attempt_void(I.stat))) return;
    unsigned long long claim = 0;
    if (lane == 0) claim = atomicAdd(&I.stat->next, 1ULL);
    claim = __shfl_sync(all, claim, 0);
    if (claim >= (unsigned long long)I.n) return;
    const int row = (int)claim;
    const int j1 = ia[row], j2 = ia[row + 1];
    for (int k = lane; k < kIlutCap; k += 32) W.lc[k] = W.uc[k] = -1;
    double tnorm = 0.0;
    for (int k = j1; k < j2; ++k) tnorm = __dadd_rn(tnorm, fabs(a[k]));
    if (tnorm == 0.0) {
      raise_error(I.stat, kIlutErrZeroRow, row);
      return;
    }
    tnorm = __ddiv_rn(tnorm, (double)(j2 - j1));
    __syncwarp();
    // (a matrix row has at most kMaxRowLen entries: no list overflows here)
    int lenl = 0, nu = 0;
    double wd = 0.0;
    for (int j = j1; j < j2; ++j) {
      const int c = ja[j];
      const double t = a[j];
      if (c < row) {
        if (lane == 0) {
          W.lc[lenl] = c;
          W.lv[lenl] = t;
        }
        ++lenl;
      } else if (c == row) {
        wd = t;
      } else {
        if (lane == 0) {
          W.uc[nu] = c;
          W.uv[nu] = t;
        }
        ++nu;
      }
    }
    __syncwarp();
    // the sum of the dropped entries, in order; without relaxation it only
    // matters when it is not finite (0 * inf), so it is taken only once an
    // entry is so large that up to 512 of them might overflow (the sum so far
    // was finite, and any finite value will do for it)
    double dropsum = 0.0;
    auto drop = [&](double v) {
      if (relax != 0.0 || magnitude(v) >= 0x7e80000000000000ULL || !isfinite(dropsum))
        dropsum = __dadd_rn(dropsum, v);
    };
    int ilen = 0;
    for (int left = lenl; left > 0; --left) {
      // the smallest remaining column
      int best = kGone, at = 0;
      for (int k = lane; k < lenl; k += 32) {
        const int c = W.lc[k];
        if (c < best) {
          best = c;
          at = k;
        }
      }
      const int jrow = (int)__reduce_min_sync(all, (unsigned)best);
      const unsigned who = __ballot_sync(all, best == jrow);
      at = __shfl_sync(all, at, __ffs((int)who) - 1);
      const double wj = W.lv[at];
      __syncwarp();
      if (lane == 0) W.lc[at] = kGone;
      if (!wait_row(I, jrow)) return;
      // the row's count, pivot and first 32 U slots in one round trip
      const size_t ub = (size_t)jrow * I.su;
      const int nuj = __ldcg(I.nu + jrow);
      const double dj = __ldcg(I.dinv + jrow);
      int cq = -2;
      double vq = 0.0;
      if (lane < I.su) {
        cq = __ldcg(I.ucol + ub + lane);
        vq = __ldcg(I.uval + ub + lane);
      }
      const double fact = __dmul_rn(wj, dj);
      if (fabs(fact) <= droptol) {
        drop(wj);
        __syncwarp();
        continue;
      }
      for (int q0 = 0; q0 < nuj; q0 += 32) {
        const int q = q0 + lane;
        int c = -2;
        double sv = 0.0;
        if (q < nuj) {
          c = q0 == 0 ? cq : __ldcg(I.ucol + ub + q);
          sv = __dmul_rn(fact, q0 == 0 ? vq : __ldcg(I.uval + ub + q));
        }
        __syncwarp();
        // columns between jrow and row go to L, those above row to U, row
        // itself is the diagonal; a U row's columns are distinct, so no two
        // lanes share a target
        const bool lower = c > jrow && c < row, upper = c > row;
        int p = -1;
        if (__any_sync(all, upper)) {
          const int r = find_column(W.uc, nu, c);
          if (upper) p = r;
        }
        if (__any_sync(all, lower)) {
          const int r = find_column(W.lc, lenl, c);
          if (lower) p = r;
        }
        const unsigned newu = __ballot_sync(all, upper && p < 0), newl = __ballot_sync(all, lower && p < 0);
        const unsigned dg = __ballot_sync(all, c == row);
        if (nu + __popc(newu) > kIlutCap || lenl + __popc(newl) > kIlutCap) {
          raise_error(I.stat, kIlutErrCap, row);
          return;
        }
        if (upper || lower) {
          const unsigned below = (1u << lane) - 1u;
          double *list = upper ? W.uv : W.lv;
          if (p >= 0) {
            list[p] = __dsub_rn(list[p], sv);
          } else if (upper) {
            p = nu + __popc(newu & below);
            W.uc[p] = c;
            W.uv[p] = -sv;
          } else {
            p = lenl + __popc(newl & below);
            W.lc[p] = c;
            W.lv[p] = -sv;
          }
        }
        if (dg) wd = __dsub_rn(wd, __shfl_sync(all, sv, __ffs((int)dg) - 1));
        nu += __popc(newu);
        lenl += __popc(newl);
        left += __popc(newl);
        __syncwarp();
      }
      if (lane == 0) {
        W.mv[ilen] = fact;
        W.mc[ilen] = jrow;
      }
      ++ilen;
      __syncwarp();
    }
    // L: the lfil largest multipliers
    const int nkeep = min(ilen, lfil);
    // U: drop below droptol x tnorm, in order, then the lfil - 1 largest
    const double tol = __dmul_rn(droptol, tnorm);
    int m = 0;
    for (int k0 = 0; k0 < nu; k0 += 32) {
      const int k = k0 + lane;
      const double v = k < nu ? W.uv[k] : 0.0;
      const int c = k < nu ? W.uc[k] : 0;
      const bool keep = k < nu && fabs(v) > tol;
      // (one at a time only where the sum matters)
      unsigned gone = __ballot_sync(all, k < nu && !keep &&
                                             (relax != 0.0 || magnitude(v) >= 0x7e80000000000000ULL));
      const unsigned kept = __ballot_sync(all, keep);
      while (gone) {
        const int l = __ffs((int)gone) - 1;
        drop(__shfl_sync(all, v, l));
        gone &= gone - 1u;
      }
      __syncwarp();
      if (keep) {
        const int p = m + __popc(kept & ((1u << lane) - 1u));
        W.uv[p] = v;
        W.uc[p] = c;
      }
      m += __popc(kept);
      __syncwarp();
    }
    const int ulen = min(m + 1, lfil);
    const int ukeep = ulen > 0 ? ulen - 1 : 0;
    // the pivot, guarded against a sign change or zero
    double dw = __dadd_rn(__dmul_rn(__dadd_rn(1.0, delta), wd), __dmul_rn(relax, dropsum));
    bool bad = false;
    if (copysign(fabs(wd), dw) != wd) {
      if (izero > 1) dw = __dmul_rn(__dmul_rn(copysign(1.0, wd), __dadd_rn(1.0e-4, droptol)), tnorm);
      else bad = true;
    }
    if (!bad && fabs(dw) == 0.0) {
      if (izero > 1) dw = __dmul_rn(__dmul_rn(copysign(1.0, wd), __dadd_rn(1.0e-4, droptol)), tnorm);
      else bad = true;
    }
    if (bad) {
      if (lane == 0) atomicMin(&I.stat->pivot_fail, row);
      return;
    }
    if (lane == 0) {
      I.dinv[row] = __drcp_rn(dw);
      I.nu[row] = ukeep;
      split_by_magnitude(m, W.uv, W.uc, ulen);
    }
    __syncwarp();
    const size_t ubr = (size_t)row * I.su, lb = (size_t)row * I.sl;
    for (int k = lane; k < ukeep; k += 32) {
      I.ucol[ubr + k] = W.uc[k];
      I.uval[ubr + k] = W.uv[k];
    }
    // the rows that wait for this one need its pivot and U entries only: the
    // release (which covers what the warp's other lanes wrote before the
    // barrier) comes before the choice of the L entries
    __syncwarp();
    if (lane == 0) st_release_u32(I.rdone + row, I.epoch);
    if (lane == 0) split_by_magnitude(ilen, W.mv, W.mc, nkeep);
    __syncwarp();
    for (int k = lane; k < nkeep; k += 32) {
      I.lcol[lb + k] = W.mc[k];
      I.lval[lb + k] = W.mv[k];
    }
    if (lane == 0) I.nl[row] = nkeep;
    __syncwarp();
  }
}

// Values from the padded rows into the IAPC/JAPC/APC layout.
__global__ void k_ilut_scatter(IlutDev I, const int *__restrict__ iapc,
                               const int *__restrict__ japc, double *__restrict__ apc) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= I.n) return;
  apc[row] = I.dinv[row];
  const int l0 = iapc[row], u0 = japc[row];
  const int nl = I.nl[row], nu = I.nu[row];
  const size_t lb = (size_t)row * I.sl, ub = (size_t)row * I.su;
  for (int k = 0; k < nl; ++k) apc[l0 + k] = I.lval[lb + k];
  for (int k = 0; k < nu; ++k) apc[u0 + k] = I.uval[ub + k];
}

}  // namespace

static_assert(kIlutWarps * sizeof(IlutRow) <= 48 * 1024, "no opt-in needed");
static int ilut_grid() {
  static const int per_sm = [] {  // every device is a GB300
    int occ = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_ilut_factor, 32 * kIlutWarps,
                                                  kIlutWarps * sizeof(IlutRow));
    return std::max(1, occ);
  }();
  return per_sm * kNumSM;
}

void launch_ilut_factor(const IlutDev &I, const int *d_ia, const int *d_ja, const double *d_amat,
                        double droptol, double relax, double delta, int izero, cudaStream_t st) {
  const int grid = std::max(1, std::min(ilut_grid(), (I.n + kIlutWarps - 1) / kIlutWarps));
  k_ilut_factor<<<grid, 32 * kIlutWarps, kIlutWarps * sizeof(IlutRow), st>>>(
      I, d_ia, d_ja, d_amat, droptol, relax, delta, izero);
}

void launch_ilut_scatter(const IlutDev &I, const int *d_iapc, const int *d_japc, double *d_apc,
                         cudaStream_t st) {
  k_ilut_scatter<<<(I.n + 255) / 256, 256, 0, st>>>(I, d_iapc, d_japc, d_apc);
}

}  // namespace gb
