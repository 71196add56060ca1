// k_ilu.cu -- ILU0 / MILU0 factorisation of general patterns and the triangular
// sweeps a level at a time.
//
// Factorisation: ims_base_pcilu0 (src/Solution/LinearMethods/ImsLinearBase.f90:928-1042)
// restated per row in one launch, a lane a row, the lanes of a warp through
// their lower entries together (see k_ilu0_factor).
// The row's work vector W is indexed by the row's sorted pattern (IAPC/JAPC
// from ims_base_pccrs); every update to a W slot and to the dropped-fill sum
// rs happens in the reference's order, and every operation is rounded
// separately (no FMA), so APC is bit-for-bit the reference's.
//
// Apply: ims_base_ilu0a (:1049-1092).  Forward sweep D = R - L*D (unit lower),
// backward sweep D = (D - U*D) * APC(n).  Rows of a level are independent: one
// launch per level, or one sync-free launch per sweep for patterns of few levels
// (k_range.cu has the others').  Entries are summed in JAPC order with FMA.
#include "gbims_internal.cuh"
#include "k_llword.cuh"
#include <algorithm>
#include <climits>

namespace gb {

void levels_build_host(int n, const std::vector<int> &iapc, const std::vector<int> &japc,
                       bool forward, Levels &L, cudaStream_t st) {
  std::vector<int> lev(n, 0);
  int nlev = 0;
  if (forward) {
    for (int r = 0; r < n; ++r) {
      int l = 0;
      for (int j = iapc[r]; j < japc[r]; ++j) l = std::max(l, lev[japc[j]] + 1);
      lev[r] = l;
      nlev = std::max(nlev, l + 1);
    }
  } else {
    for (int r = n - 1; r >= 0; --r) {
      int l = 0;
      for (int j = japc[r]; j < iapc[r + 1]; ++j) l = std::max(l, lev[japc[j]] + 1);
      lev[r] = l;
      nlev = std::max(nlev, l + 1);
    }
  }
  L.nlev = nlev;
  L.ptr.assign(nlev + 1, 0);
  for (int r = 0; r < n; ++r) L.ptr[lev[r] + 1]++;
  for (int l = 0; l < nlev; ++l) L.ptr[l + 1] += L.ptr[l];
  std::vector<int> rows(n), fill(L.ptr.begin(), L.ptr.end() - 1);
  for (int r = 0; r < n; ++r) rows[fill[lev[r]]++] = r;
  L.maxwidth = 0;
  for (int l = 0; l < nlev; ++l) L.maxwidth = std::max(L.maxwidth, L.ptr[l + 1] - L.ptr[l]);
  // slices: up to 32 rows of one level
  std::vector<int2> sl;
  for (int l = 0; l < nlev; ++l)
    for (int q = L.ptr[l]; q < L.ptr[l + 1]; q += 32)
      sl.push_back(make_int2(q, std::min(32, L.ptr[l + 1] - q)));
  L.nslices = (int)sl.size();
  if (L.d_rows) cudaFree(L.d_rows);
  if (L.d_slices) cudaFree(L.d_slices);
  L.d_rows = nullptr;
  L.d_slices = nullptr;
  if (n > 0) {
    cudaMalloc(&L.d_rows, sizeof(int) * n);
    cudaMemcpyAsync(L.d_rows, rows.data(), sizeof(int) * n, cudaMemcpyHostToDevice, st);
    cudaMalloc(&L.d_slices, sizeof(int2) * sl.size());
    cudaMemcpyAsync(L.d_slices, sl.data(), sizeof(int2) * sl.size(), cudaMemcpyHostToDevice, st);
    cudaStreamSynchronize(st);
  }
}

// Position of column c in the sorted off-diagonal pattern japc[i0:i1), or -1.
__device__ __forceinline__ int find_sorted(const int *__restrict__ japc, int i0, int i1, int c) {
  int lo = i0, hi = i1 - 1;
  while (lo <= hi) {
    int mid = (lo + hi) >> 1;
    int v = japc[mid];
    if (v == c) return mid - i0;
    if (v < c) lo = mid + 1;
    else hi = mid - 1;
  }
  return -1;
}

// Where an elimination product goes: an off-diagonal slot of the row (its
// position), the diagonal, or the dropped-fill sum.
constexpr int kToDiag = 14, kDropped = 15;
constexpr int kShort = 6;  // lower and upper entries of a row of the short form (a target fits 4 bits)

// The whole factorisation in one launch.  Bound by its chain: a level hands
// its inverse pivots and upper entries to the next through L2 (0.7 us) and a
// row has about 25 dependent FP64 instructions of 64 cycles.  A launch per
// level added a launch, its ten dependent index loads and the gap between
// kernels to each: a factorisation of 1 x 100 x 100 cells (199 levels) took 2.1
// ms and takes 0.55, of 10 x 200 x 200 (408) 8.5 and 2.0, of 10 x 400 x 400
// (808) 18.4 and 4.1.
//
// Warps claim slices (up to 32 rows of one level) in level order.  A warp
// waits for the row a lane eliminates next by polling the words that row's
// owner writes: its inverse pivot and upper entries, each tagged with the
// epoch of the launch (k_llword.cuh), so that no fence stands between them.
// All lanes of a warp take their e-th lower entry together: an FP64
// instruction costs the same for one lane as for 32.  Slices are claimed in
// order, so the lowest unfinished one can always proceed, however many warps
// are resident; every wait is bounded.
//
// Where a pivot fails, the attempt is void, and the last attempt's rows before
// the first failure are the factor's (ImsLinearBase.f90:1010-1042).  So the
// rows after a failed one are left out as soon as it is known, the rows before
// it are all made, and the values go to APC from the words, by
// k_ilu0_commit, up to the first failure.
//
// SHORT: rows of at most kShort lower and upper entries; their index work is
// done before the waits.  MILU: the dropped-fill sum is needed (relax > 0);
// without it only products that might overflow are summed, because then
// 0 * rs is not zero.
template <bool SHORT, bool MILU>
__global__ void __launch_bounds__(128) k_ilu0_factor(
    int nslices, const int2 *__restrict__ slices, const int *__restrict__ rows,
    const int *__restrict__ ia, const int *__restrict__ ja, const double *__restrict__ amat,
    const int *__restrict__ iapc, const int *__restrict__ japc, LLWord<double> *words, unsigned ep, int *claim, double relax, double delta, int ipcflag, Ctl *ctl) {
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  volatile int *failed = &ctl->pivot_fail;
  while (true) {
    int s = 0;
    if (lane == 0) s = atomicAdd(claim, 1);
    s = __shfl_sync(all, s, 0);
    if (s >= nslices) return;
    const int2 sl = slices[s];
    const int n = rows[sl.x + min(lane, sl.y - 1)];
    bool mine = lane < sl.y && n < *failed;  // not behind a row that failed
    if (!__any_sync(all, mine)) continue;
    // false when a wait runs out
    unsigned turns = 0;
    auto keep_waiting = [&]() -> bool {
      if ((++turns & 63u) != 0) return true;
      if (turns > (1u << 23)) {  // L2 round trips: seconds
        if (lane == 0) atomicExch(&ctl->scratch_err, 1);
        return false;
      }
      mine = mine && n < *failed;
      return __all_sync(all, *(volatile int *)&ctl->scratch_err == 0);
    };
    const int ic0 = iapc[n], ic1 = iapc[n + 1], iu = japc[n];
    const int len = ic1 - ic0, nlow = iu - ic0;
    // w[0..len): off-diagonal slots in JAPC order; wd: the diagonal slot
    double w[SHORT ? 2 * kShort : kMaxRowLen];
    if (!SHORT) {
#pragma unroll 8
      for (int k = 0; k < kMaxRowLen; ++k)
        if (k < len) w[k] = 0.0;
    } else {
#pragma unroll
      for (int k = 0; k < 2 * kShort; ++k) w[k] = 0.0;
    }
    double wd = 0.0;
    // W(jcol) = W(jcol) + AMAT(j) over the CSR row (ImsLinearBase.f90:985-989)
    for (int j = ia[n]; j < ia[n + 1]; ++j) {
      const int c = ja[j];
      if (c == n) {
        wd = __dadd_rn(wd, amat[j]);
      } else {
        const int k = find_sorted(japc, ic0, ic1, c);
        if (k >= 0) w[k] = __dadd_rn(w[k], amat[j]);
      }
    }
    // the index work of a short row: per lower entry its row, where that
    // row's upper entries start, how many there are, and their targets
    int col[kShort], u0[kShort], nu[kShort];
    unsigned tgt[kShort];
    if (SHORT) {
#pragma unroll
      for (int e = 0; e < kShort; ++e) {
        col[e] = u0[e] = nu[e] = 0;
        tgt[e] = 0;
        if (e < nlow) {
          col[e] = japc[ic0 + e];
          u0[e] = japc[col[e]];
          nu[e] = iapc[col[e] + 1] - u0[e];
#pragma unroll
          for (int u = 0; u < kShort; ++u)
            if (u < nu[e]) {
              const int c = japc[u0[e] + u];
              int t = kToDiag;
              if (c != n) {
                t = find_sorted(japc, ic0, ic1, c);
                if (t < 0) t = kDropped;
              }
              tgt[e] |= (unsigned)t << (4 * u);
            }
        }
      }
    }
    double nrs = 0.0;  // minus the dropped-fill sum
    // LOWER loop (:993-1007): one product into its target
    auto eliminate = [&](double tl, double uval, int t) {
      if (t == kDropped && !MILU && !may_overflow(tl, uval)) return;
      const double prod = __dmul_rn(tl, uval);
      double x = t == kToDiag ? wd : t == kDropped ? nrs : w[t];
      x = __dsub_rn(x, prod);
      if (t == kToDiag) wd = x;
      else if (t == kDropped) nrs = x;
      else w[t] = x;
    };
    const int maxlow = __reduce_max_sync(all, mine ? nlow : 0);
    if (SHORT) {
#pragma unroll
      for (int e = 0; e < kShort; ++e) {
        if (e >= maxlow) break;
        bool act;
        LLRaw rd, ru[kShort];
        while (true) {
          bool ok = true;
          act = mine && e < nlow;
          if (act) {
            ll_issue(words + col[e], rd);
#pragma unroll
            for (int u = 0; u < kShort; ++u)
              if (u < nu[e]) ll_issue(words + u0[e] + u, ru[u]);
            ok = ll_ready<double>(rd, ep);
#pragma unroll
            for (int u = 0; u < kShort; ++u)
              if (u < nu[e]) ok = ok && ll_ready<double>(ru[u], ep);
          }
          if (__all_sync(all, ok)) break;
          if (!keep_waiting()) return;
        }
        if (act) {
          double dv;
          ll_take(rd, dv);
          const double tl = __dmul_rn(w[e], dv);
          w[e] = tl;
#pragma unroll
          for (int u = 0; u < kShort; ++u)
            if (u < nu[e]) {
              double uv;
              ll_take(ru[u], uv);
              eliminate(tl, uv, (int)((tgt[e] >> (4 * u)) & 15u));
            }
        }
      }
    } else {
      for (int e = 0; e < maxlow; ++e) {
        int jcol = 0, uu0 = 0, uu1 = 0;
        if (mine && e < nlow) {
          jcol = japc[ic0 + e];
          uu0 = japc[jcol];
          uu1 = iapc[jcol + 1];
        }
        double tl = 0.0;
        const int most = __reduce_max_sync(all, uu1 - uu0);
        for (int ub = 0; ub == 0 || ub < most; ub += 4) {
          // the inverse pivot with the first four upper entries
          bool act;
          LLRaw rd, ru[4];
          while (true) {
            bool ok = true;
            act = mine && e < nlow;
            if (act) {
              if (ub == 0) ll_issue(words + jcol, rd);
#pragma unroll
              for (int u = 0; u < 4; ++u)
                if (uu0 + ub + u < uu1) ll_issue(words + uu0 + ub + u, ru[u]);
              if (ub == 0) ok = ll_ready<double>(rd, ep);
#pragma unroll
              for (int u = 0; u < 4; ++u)
                if (uu0 + ub + u < uu1) ok = ok && ll_ready<double>(ru[u], ep);
            }
            if (__all_sync(all, ok)) break;
            if (!keep_waiting()) return;
          }
          if (act) {
            if (ub == 0) {
              double dv;
              ll_take(rd, dv);
              tl = __dmul_rn(w[e], dv);
              w[e] = tl;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (uu0 + ub + u < uu1) {
                const int c = japc[uu0 + ub + u];
                double uv;
                ll_take(ru[u], uv);
                const int k = c == n ? -2 : find_sorted(japc, ic0, ic1, c);
                if (k == -1 && !MILU && !may_overflow(tl, uv)) continue;
                const double prod = __dmul_rn(tl, uv);
                const double x = __dsub_rn(k == -2 ? wd : k == -1 ? nrs : w[k], prod);
                if (k == -2) wd = x;
                else if (k == -1) nrs = x;
                else w[k] = x;
              }
          }
        }
      }
    }
    if (!mine) continue;
    // the upper entries are final (the lower ones go to APC from their words)
    for (int k = nlow; k < len; ++k) ll_put(words + ic0 + k, w[k], ep);
    for (int k = 0; k < nlow; ++k) ll_put(words + ic0 + k, w[k], ep);
    // DIAGONAL (:1010-1037)
    const double d = wd;
    double tl = __dsub_rn(__dmul_rn(__dadd_rn(1.0, delta), d), __dmul_rn(relax, -nrs));
    const double sd1 = copysign(fabs(d), tl);
    bool bad = false;
    if (sd1 != d) {
      if (ipcflag > 1) tl = copysign(1.0e-6, d);
      else bad = true;
    }
    if (!bad && fabs(tl) == 0.0) {
      if (ipcflag > 1) tl = copysign(1.0e-6, d);
      else bad = true;
    }
    if (bad) {
      atomicMin(&ctl->pivot_fail, n);
      continue;
    }
    ll_put(words + n, __drcp_rn(tl), ep);
  }
}

// The rows before the first failure into APC; the others keep what they held.
__global__ void __launch_bounds__(256) k_ilu0_commit(int n, const int *__restrict__ iapc,
                                                     const LLWord<double> *__restrict__ words,
                                                     double *__restrict__ apc, const Ctl *ctl) {
  if (ctl->scratch_err) return;
  const int rows = min(n, ctl->pivot_fail), end = iapc[rows];
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < end; p += gridDim.x * blockDim.x)
    if (p < rows || p >= n) apc[p] = ll_val(words[p]);
}

// True when every row has at most kShort lower and upper entries.
bool ilu_short_rows(int n, const std::vector<int> &iapc, const std::vector<int> &japc) {
  for (int r = 0; r < n; ++r)
    if (japc[r] - iapc[r] > kShort || iapc[r + 1] - japc[r] > kShort) return false;
  return true;
}

// A new epoch for the words of the next launch, and its claims from zero.
int factor_words_next(FactorWords &W, cudaStream_t st) {
  W.epoch += 1;
  if (W.epoch == 0) {  // the epochs wrapped: clear the words
    if (cudaMemsetAsync(W.words, 0, 16 * W.count, st) != cudaSuccess) return -1;
    W.epoch = 1;
  }
  return cudaMemsetAsync(W.claim, 0, sizeof(int), st) == cudaSuccess ? 0 : -1;
}

// Warps at work: enough that those ahead of the front have their rows' index
// work done when it arrives, few enough that their polls do not slow it
// (kFactorAhead 2, 4, 8, 16 and 64 on 10 x 400 x 400 cells: 5.3, 4.4, 4.8, 6.1
// and 50 ms).
int launch_ilu_factor(int n, const int *d_ia, const int *d_ja, const double *d_amat,
                      const int *d_iapc, const int *d_japc, double *d_apc, const Levels &L,
                      FactorWords &W, double relax, double delta, int ipcflag, Ctl *ctl,
                      cudaStream_t st) {
  if (factor_words_next(W, st) != 0) return -1;
  const long long warps = std::min<long long>((long long)(L.maxwidth + 31) / 32 * kFactorAhead, L.nslices);
  const int grid = (int)std::max<long long>(1, std::min<long long>((warps + 3) / 4, 8LL * kNumSM));
  auto *k = W.short_rows ? (relax > 0.0 ? k_ilu0_factor<true, true> : k_ilu0_factor<true, false>)
                         : (relax > 0.0 ? k_ilu0_factor<false, true> : k_ilu0_factor<false, false>);
  LLWord<double> *words = static_cast<LLWord<double> *>(W.words);
  k<<<grid, 128, 0, st>>>(L.nslices, L.d_slices, L.d_rows, d_ia, d_ja, d_amat, d_iapc, d_japc, words, W.epoch,
                          W.claim, relax, delta, ipcflag, ctl);
  k_ilu0_commit<<<std::min<int>((int)((W.count + 255) / 256), 8 * kNumSM), 256, 0, st>>>(n, d_iapc, words, d_apc,
                                                                                        ctl);
  return 0;
}

template <typename T>
__device__ __forceinline__ T fms(T a, T b, T c);  // c - a*b with one rounding
template <>
__device__ __forceinline__ double fms<double>(double a, double b, double c) { return fma(-a, b, c); }
template <>
__device__ __forceinline__ float fms<float>(float a, float b, float c) { return fmaf(-a, b, c); }

template <typename T>
__global__ void k_ilu_fwd_level(const int *__restrict__ rows, int nrows,
                                const int *__restrict__ iapc, const int *__restrict__ japc,
                                const T *__restrict__ apc, const T *__restrict__ r, T *d,
                                const Ctl *__restrict__ ctl) {
  if (ctl && ctl->done) return;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nrows) return;
  int n = rows[t];
  T tv = r[n];
  for (int j = iapc[n]; j < japc[n]; ++j) tv = fms<T>(apc[j], d[japc[j]], tv);
  d[n] = tv;
}

template <typename T>
__global__ void k_ilu_bwd_level(const int *__restrict__ rows, int nrows,
                                const int *__restrict__ iapc, const int *__restrict__ japc,
                                const T *__restrict__ apc, T *d,
                                const Ctl *__restrict__ ctl) {
  if (ctl && ctl->done) return;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nrows) return;
  int n = rows[t];
  T tv = d[n];
  for (int j = japc[n]; j < iapc[n + 1]; ++j) tv = fms<T>(apc[j], d[japc[j]], tv);
  d[n] = tv * apc[n];
}

template <typename T>
static void apply_levels(const int *d_iapc, const int *d_japc, const T *d_apc,
                         const Levels &F, const Levels &B, const T *r, T *d, const Ctl *ctl,
                         cudaStream_t st) {
  for (int l = 0; l < F.nlev; ++l) {
    int nr = F.ptr[l + 1] - F.ptr[l];
    k_ilu_fwd_level<T><<<(nr + 127) / 128, 128, 0, st>>>(F.d_rows + F.ptr[l], nr, d_iapc,
                                                          d_japc, d_apc, r, d, ctl);
  }
  for (int l = 0; l < B.nlev; ++l) {
    int nr = B.ptr[l + 1] - B.ptr[l];
    k_ilu_bwd_level<T><<<(nr + 127) / 128, 128, 0, st>>>(B.d_rows + B.ptr[l], nr, d_iapc,
                                                          d_japc, d_apc, d, ctl);
  }
}

// The sync-free sweeps: one launch per sweep, a thread a row, the rows in level
// order, every value handed over through L2 as a word tagged with the launch's
// epoch.  Polling is warp-synchronous: in each round every unfinished lane loads
// all its dependencies' words (up to kDeps in flight at once), and a lane whose
// words are all of this epoch finishes its row; a lane may wait for one of its own
// warp, which is seen in the next round.  Rows depend only on rows of lower levels,
// earlier in the list, and a CTA takes the 256 rows of its ticket, in the order in
// which CTAs start: the lowest unfinished row is always a running CTA's, however
// many are resident, also beside another handle's sweeps.  Every wait is bounded
// besides.
//
// Bound by the levels, 1.6 us each (more where the rows far ahead of the front are
// many: their polls slow it), where a range sweep pays for its setup, for its
// halo's way through three warps (5 ns an entry) and for its crossings between
// ranges: both sweeps of a red-black ordered 500 x 500 grid (2 levels) take 16 us
// against 54 in ranges, of 300 x 300 cells in random order (16) 64 against 132, of
// a random graph of 200,000 rows (22) 142 against 224; of 1000 separate 10 x 10
// grids (19) 76 against 37.  With fixed strides over a grid of resident CTAs the
// first three took 15, 61 and 128 and 1500 x 1500 red-black 91 against 108 now, but
// all CTAs had to be resident: beside another handle's sweeps a warp could wait for
// a CTA that waited for its place.  Claims by warp took 24, 65, -, 137.
template <typename T, int DIR>
__global__ void __launch_bounds__(256) k_ilu_sweep_sf(int n, const int *__restrict__ rows,
                                                      const int *__restrict__ iapc,
                                                      const int *__restrict__ japc,
                                                      const T *__restrict__ apc,
                                                      const T *__restrict__ r,
                                                      const LLWord<T> *__restrict__ yin,
                                                      LLWord<T> *out, T *d,
                                                      unsigned long long *ticket, int *err,
                                                      Ctl *ctl) {
  __shared__ unsigned s_ep;
  __shared__ int s_t;
  if (threadIdx.x == 0) {
    // every CTA takes a ticket, so launch e owns tickets [e*grid, (e+1)*grid)
    const unsigned long long tk = atomicAdd(ticket, 1ULL), launch = tk / gridDim.x;
    s_ep = (unsigned)launch + 1u;
    s_t = (int)(tk - launch * gridDim.x);
  }
  __syncthreads();
  if (ctl && ctl->done) return;
  const unsigned ep = s_ep;
  const int lane = threadIdx.x & 31;
  volatile int *vdone = ctl ? &ctl->done : nullptr;
  constexpr int kDeps = 8;
  const int q = s_t * 256 + (int)threadIdx.x;
  bool done = q >= n;
  int row = 0, j0 = 0, j1 = 0;
  T tv0 = T(0);
  if (!done) {
    row = rows[q];
    if (DIR > 0) {
      tv0 = r[row];
      j0 = iapc[row];
      j1 = japc[row];
    } else {
      tv0 = ll_val(yin[row]);
      j0 = japc[row];
      j1 = iapc[row + 1];
    }
  }
  const unsigned long long t0 = wclock();
  while (true) {
    if (!done) {
      T tv = tv0;
      bool ok = true;
      for (int jb = j0; ok && jb < j1; jb += kDeps) {
        LLRaw w[kDeps];
        const int nd = min(kDeps, j1 - jb);
#pragma unroll
        for (int q2 = 0; q2 < kDeps; ++q2)
          if (q2 < nd) ll_issue(out + japc[jb + q2], w[q2]);
#pragma unroll
        for (int q2 = 0; q2 < kDeps; ++q2) {
          if (q2 >= nd || !ok) break;
          if (!ll_ready<T>(w[q2], ep)) {
            ok = false;
          } else {
            T v;
            ll_take(w[q2], v);
            tv = fms<T>(apc[jb + q2], v, tv);
          }
        }
      }
      if (ok) {
        if (DIR < 0) {
          tv = tv * apc[row];
          d[row] = tv;
        }
        ll_put(out + row, tv, ep);
        done = true;
      }
    }
    if (!__any_sync(0xffffffffu, !done)) break;
    if (__any_sync(0xffffffffu, (vdone && *vdone) || wclock() - t0 > kWaitCycles)) {
      if (lane == 0) {
        atomicExch(err, 1);
        if (ctl) ctl->done = 1;
      }
      return;
    }
  }
}

template <typename T>
static void apply_sf(int n, const int *d_iapc, const int *d_japc, const T *d_apc, const Levels &F,
                     const Levels &B, const LevelWords &W, const T *r, T *d, Ctl *ctl, cudaStream_t st) {
  LLWord<T> *yf = static_cast<LLWord<T> *>(W.fwd);
  LLWord<T> *zb = static_cast<LLWord<T> *>(W.bwd);
  const int grid = (int)(((long long)n + 255) / 256);
  k_ilu_sweep_sf<T, 1><<<grid, 256, 0, st>>>(n, F.d_rows, d_iapc, d_japc, d_apc, r, nullptr, yf, nullptr, W.ticket,
                                             W.err, ctl);
  k_ilu_sweep_sf<T, -1><<<grid, 256, 0, st>>>(n, B.d_rows, d_iapc, d_japc, d_apc, nullptr, yf, zb, d, W.ticket + 16,
                                              W.err, ctl);
}

void launch_ilu_apply_sf(int n, const int *d_iapc, const int *d_japc, const double *d_apc, const Levels &F,
                         const Levels &B, const LevelWords &W, const double *r, double *d, Ctl *ctl,
                         cudaStream_t st) {
  apply_sf<double>(n, d_iapc, d_japc, d_apc, F, B, W, r, d, ctl, st);
}
void launch_ilu_apply_sf32(int n, const int *d_iapc, const int *d_japc, const float *d_apc32, const Levels &F,
                           const Levels &B, const LevelWords &W, const float *r, float *d, Ctl *ctl,
                           cudaStream_t st) {
  apply_sf<float>(n, d_iapc, d_japc, d_apc32, F, B, W, r, d, ctl, st);
}

void launch_ilu_apply_levels(int n, const int *d_iapc, const int *d_japc, const double *d_apc,
                             const Levels &F, const Levels &B, const double *r, double *d,
                             const Ctl *ctl, cudaStream_t st) {
  (void)n;
  apply_levels<double>(d_iapc, d_japc, d_apc, F, B, r, d, ctl, st);
}

void launch_ilu_apply_levels32(int n, const int *d_iapc, const int *d_japc,
                               const float *d_apc32, const Levels &F, const Levels &B,
                               const float *r, float *d, const Ctl *ctl, cudaStream_t st) {
  (void)n;
  apply_levels<float>(d_iapc, d_japc, d_apc32, F, B, r, d, ctl, st);
}

}  // namespace gb
