// k_dia7_factor.cu -- ILU0 / MILU0 factorisation of full DIS grids along the
// sweeps' wavefront.
//
// A row of a 7-point grid eliminates the row above (k-1), behind (i-1) and to
// its left (j-1), in that order. No two of a row's neighbours are neighbours,
// so nothing fills in: the upper entries stay the matrix's, a lower entry is
// the matrix's times the neighbour's inverse pivot, and all that rows hand to
// one another is the inverse pivot.  Operations, their order and rounding are
// those of k_ilu0_factor (one product and one difference each, no FMA), so APC
// is the same bit for bit.
#include "gbims_internal.cuh"
#include "k_llword.cuh"
#include <algorithm>
#include <climits>

namespace gb {

namespace {

constexpr int kLines = 32;  // the sweeps' W, lane skew 1

// 0.0 + a, which turns -0 into +0, off the FP64 pipe.
__device__ __forceinline__ double plus_zero(double a) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(a);
  return (u << 1) == 0ULL ? 0.0 : a;
}

// A normal number with a normal reciprocal.
__device__ __forceinline__ bool ordinary(double x) {
  return (((unsigned)__double2hiint(x) >> 20) & 0x7ffu) - 1u < 2044u;
}
// 1/x of such a number, rounded to nearest, by integer arithmetic: Newton's iteration
// y += y (1 - x y) on the mantissa in 64-bit fixed point, twice from an FP32
// estimate (23, then 45, then 61 bits), and the exact remainder 2^105 - q m
// decides the last place.  1.1 us a step with CUDA's reciprocal and its FP64
// instructions, 0.8 with this.
__device__ __forceinline__ double reciprocal(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned mh = (hi & 0xfffffu) | 0x100000u;
  const unsigned long long m = ((unsigned long long)mh << 32) | lo;
  const unsigned long long M = m << 11;  // x's mantissa, 2^63 for 1
  float f = __uint_as_float(0x3f800000u | ((unsigned)(M >> 40) & 0x7fffffu));
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(f));
  const unsigned y0 = max(0x3f000000u, min(__float_as_uint(f), 0x3f7fffffu));
  unsigned long long y = (unsigned long long)((y0 & 0x7fffffu) | 0x800000u) << 39;  // 2^63 for 1
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const long long e = (long long)(0x4000000000000000ull - __umul64hi(M, y));
    y += (unsigned long long)__mul64hi((long long)y, e * 4);
  }
  unsigned long long q = (y + 512u) >> 10;
  const long long r = (long long)(0ull - q * m);
  if (2 * r > (long long)m) q += 1;
  else if (2 * r < -(long long)m) q -= 1;
  if (m == 0x10000000000000ull) q = 0x20000000000000ull;  // a power of two
  const unsigned ex = (hi >> 20) & 0x7ffu;
  return __hiloint2double((int)((((2044u - ex) << 20) + (unsigned)(q >> 32)) | (hi & 0x80000000u)), (int)q);
}

// A lower entry and the upper entry of a row it eliminates, one of them so
// large that the entry's product with another upper entry, or a sum of a row's
// such products, could overflow.  Every upper entry meets one row.
__device__ __forceinline__ bool large(double tl, double u) {
  return ((__double2hiint(tl) >> 20) & 0x7ff) > 1023 + 600 || ((__double2hiint(u) >> 20) & 0x7ff) > 1023 + 300;
}

// 1 / the pivot of the diagonal d with dropped-fill sum -nrs (the reference's
// test of the pivot, ImsLinearBase.f90:1010-1037), the tests on the bits.
__device__ __forceinline__ double invert_pivot(double d, double nrs, double relax, double delta, int ipcflag,
                                               bool plain, bool &bad) {
  double tl = plain ? d : __dsub_rn(__dmul_rn(__dadd_rn(1.0, delta), d), __dmul_rn(relax, -nrs));
  const unsigned long long ud = (unsigned long long)__double_as_longlong(d);
  const unsigned long long ut = (unsigned long long)__double_as_longlong(tl);
  const bool nan = (ud << 1) > 0xffe0000000000000ULL, zero = (ud << 1) == 0ULL;
  bad = false;
  if (nan || (!zero && (long long)(ud ^ ut) < 0) || (ut << 1) == 0ULL) {
    if (ipcflag > 1) tl = copysign(1.0e-6, d);
    else bad = true;
  }
  return __drcp_rn(tl);
}

// DROP: with the dropped-fill sum.  Without it (relax 0) large entries are
// reported: the attempt is then to be made again with the sum, because 0 * rs is
// not zero when rs overflows.
//
// What a row needs of the matrix: its diagonal and lower entries and, of each
// lower neighbour, the upper entries that meet this row (u) or are dropped (f).
// The order: d, then per neighbour w, u and the two f.
template <bool DROP>
struct Row {
  static constexpr int kPer = DROP ? 4 : 2, kCount = 1 + 3 * kPer;
  double a[kCount];
};

__device__ __forceinline__ void copy_async(double *dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// One warp a block of 32 lines of one layer; lane l holds line l and is at
// column g - l in step g.  The inverse pivots come from the lane's own last
// step (left), from lane l-1 (behind; lane 0: the block before) and from the
// layer above, the latter two as words tagged with the launch's epoch; blocks
// take tickets in an order in which what they wait for came first.
//
// Bound by a step's chain in one warp: the left neighbour's pivot is multiplied
// twice, subtracted and inverted, 0.8 us a step with some 400 instructions; a
// level of the general kernel takes 4.3 (its rows meet through L2).  Cold
// caches: 5 x 90 x 90 cells 793 -> 213 us, 10 x 200 x 200 1808 -> 478, 1 x 100 x
// 100 211.
template <bool DROP>
__global__ void __launch_bounds__(kLines) k_dia7_factor(const Dia7Geo *__restrict__ geos, int nm, int n,
                                                        const double *__restrict__ v,
                                                        LLWord<double> *words, unsigned ep, int *claim,
                                                        double relax, double delta, int ipcflag, Ctl *ctl) {
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x;
  int id = 0;
  if (lane == 0) id = atomicAdd(claim, 1);
  id = __shfl_sync(all, id, 0);
  int lo = 0, hi = nm - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (geos[mid].ticket0 <= id) lo = mid;
    else hi = mid - 1;
  }
  const Dia7Geo geo = geos[lo];
  const int lid = id - geo.ticket0, nlay = geo.nlay, ncol = geo.ncol, nrc = geo.nrow * ncol;
  const int k = lid % nlay, b = lid / nlay, i = b * kLines + lane;
  const bool line = i < geo.nrow, hz = line && k > 0, hy = line && i > 0;
  const bool below = k < nlay - 1, front = i < geo.nrow - 1;
  const int row0 = (int)geo.row0 + k * nrc + i * ncol;
  auto tile = [&](int kk, int bb) { return geo.slot0 + ((long long)kk * geo.nb + bb) * geo.G * kLines; };
  LLWord<double> *mine = words + tile(k, b) + lane;
  const LLWord<double> *zsrc = hz ? words + tile(k - 1, b) + lane : nullptr;
  // lane 0: column j of the line before is the last lane's at its step j + 31
  const LLWord<double> *ysrc =
      lane == 0 && hy ? words + tile(k, b - 1) + (long long)(kLines - 1) * kLines + (kLines - 1) : nullptr;
  const bool plain = !DROP && delta == 0.0;
  const size_t N = (size_t)n;

  // Matrix values come through shared memory, kAhead steps ahead, copied and
  // read by the lane that uses them: a warp has too few scoreboards to tell the
  // loads of that many steps apart in registers, and waits for the last ones.
  // The words are loaded PF steps ahead.
  constexpr int kAhead = 8, PF = 2, kCount = Row<DROP>::kCount, kPer = Row<DROP>::kPer;
  __shared__ double ring[kAhead][kCount][kLines];
  const int steps = ncol + kLines - 1;
  const double *from[kCount];
  {
    const double *at = v + ((long long)row0 - lane);  // of step 0
    const size_t slot[3] = {1, 2, 3}, meets[3] = {6, 5, 4}, f0[3] = {4, 4, 5}, f1[3] = {5, 6, 6};
    const long long back[3] = {nrc, ncol, 1};
    from[0] = at;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      from[1 + e * kPer] = at + slot[e] * N;
      from[2 + e * kPer] = at + meets[e] * N - back[e];
      if (DROP) {
        from[DROP ? 3 + e * kPer : 0] = at + f0[e] * N - back[e];
        from[DROP ? 4 + e * kPer : 0] = at + f1[e] * N - back[e];
      }
    }
  }
  auto copy = [&](int g) {
    const int j = g - lane;
    double (*to)[kLines] = ring[g % kAhead];
    if (line && j >= 0 && j < ncol) {
#pragma unroll
      for (int e = 0; e < kCount; ++e)
        if (e == 0 || (e <= kPer ? hz : e <= 2 * kPer ? hy : j > 0)) copy_async(&to[e][lane], from[e] + g);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  LLRaw zr[PF], yr[PF];
  auto issue = [&](int g, LLRaw &z, LLRaw &y) {
    const int j = g - lane;
    if (!line || j < 0 || j >= ncol) return;
    if (hz) ll_issue(zsrc + (long long)g * kLines, z);
    if (ysrc) ll_issue(ysrc + (long long)g * kLines, y);
  };
  for (int g = 0; g < kAhead; ++g) copy(g);
#pragma unroll
  for (int t = 0; t < PF; ++t) issue(t, zr[t], yr[t]);
  double inv = 0.0;
  unsigned turns = 0;
  for (int g0 = 0; g0 < steps; g0 += PF) {
#pragma unroll
    for (int t = 0; t < PF; ++t) {
      const int g = g0 + t;
      if (g >= steps) break;
      const int j = g - lane;
      const bool act = line && j >= 0 && j < ncol;
      asm volatile("cp.async.wait_group %0;" ::"n"(kAhead - 1) : "memory");
      Row<DROP> q;
#pragma unroll
      for (int e = 0; e < kCount; ++e) q.a[e] = ring[g % kAhead][e][lane];
      const double behind = __shfl_up_sync(all, inv, 1);
      // the words that were not there when their loads were issued
      while (true) {
        bool ok = true;
        if (act && hz) ok = ll_ready<double>(zr[t], ep);
        if (act && ysrc) ok = ok && ll_ready<double>(yr[t], ep);
        if (__all_sync(all, ok)) break;
        if ((++turns & 63u) == 0) {
          if (turns > (1u << 23)) {  // L2 round trips: seconds
            if (lane == 0) atomicOr(&ctl->scratch_err, 1);
            return;
          }
          if (__any_sync(all, *(volatile int *)&ctl->scratch_err != 0)) return;
        }
        if (act && hz) ll_issue(zsrc + (long long)g * kLines, zr[t]);
        if (act && ysrc) ll_issue(ysrc + (long long)g * kLines, yr[t]);
      }
      // of a zero's sign only the diagonal's can matter (a retry's copysign)
      double d = plus_zero(q.a[0]), nrs = 0.0, dz = 0.0, dy = behind;
      if (act && hz) ll_take(zr[t], dz);
      if (act && ysrc) ll_take(yr[t], dy);
      bool big = false;
      auto drop = [&](double tl, double f) { nrs = __dsub_rn(nrs, __dmul_rn(tl, f)); };
      if (act && hz) {
        const double tl = __dmul_rn(q.a[1], dz);
        big = big || large(tl, q.a[2]);
        if (DROP) {
          if (j < ncol - 1) drop(tl, q.a[DROP ? 3 : 0]);
          if (front) drop(tl, q.a[DROP ? 4 : 0]);
        }
        d = __dsub_rn(d, __dmul_rn(tl, q.a[2]));
      }
      if (act && hy) {
        const double tl = __dmul_rn(q.a[1 + kPer], dy);
        big = big || large(tl, q.a[2 + kPer]);
        if (DROP && j < ncol - 1) drop(tl, q.a[DROP ? 3 + kPer : 0]);
        d = __dsub_rn(d, __dmul_rn(tl, q.a[2 + kPer]));
        if (DROP && below) drop(tl, q.a[DROP ? 4 + kPer : 0]);
      }
      if (act && j > 0) {
        const double tl = __dmul_rn(q.a[1 + 2 * kPer], inv);
        big = big || large(tl, q.a[2 + 2 * kPer]);
        d = __dsub_rn(d, __dmul_rn(tl, q.a[2 + 2 * kPer]));
        if (DROP) {
          if (front) drop(tl, q.a[DROP ? 3 + 2 * kPer : 0]);
          if (below) drop(tl, q.a[DROP ? 4 + 2 * kPer : 0]);
        }
      }
      if (!DROP && big) atomicOr(&ctl->scratch_err, 2);
      bool bad = false;
      double x = 0.0;
      if (plain && ordinary(d)) x = reciprocal(d);  // of the diagonal's sign and not zero
      else if (act) x = invert_pivot(d, nrs, relax, delta, ipcflag, plain, bad);
      // a failed pivot voids the attempt; the rows that wait for it go on
      if (bad) atomicMin(&ctl->pivot_fail, row0 + j);
      inv = x;
      if (act) ll_put(mine + (long long)g * kLines, inv, ep);
      issue(g + PF, zr[t], yr[t]);
      copy(g + kAhead);
    }
  }
}

// The factor's rows from the inverse pivots.  From the first row whose pivot
// failed on, the rows keep what they held, as in the reference.
__global__ void __launch_bounds__(256) k_dia7_factor_rows(const Dia7Geo *__restrict__ geos, int nm, int n,
                                                          const double *__restrict__ v,
                                                          const LLWord<double> *__restrict__ words,
                                                          const int *__restrict__ iapc,
                                                          double *__restrict__ apc, const Ctl *ctl) {
  if (ctl->scratch_err) return;
  const size_t N = (size_t)n;
  const int rows = min(n, ctl->pivot_fail);
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
    int lo = 0, hi = nm - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (geos[mid].row0 <= r) lo = mid;
      else hi = mid - 1;
    }
    const Dia7Geo g = geos[lo];
    const int ncol = g.ncol, nrc = g.nrow * ncol, lr = r - (int)g.row0;
    const int k = lr / nrc, rem = lr - k * nrc, i = rem / ncol, j = rem - i * ncol;
    auto pivot = [&](int kk, int ii, int jj) {
      const int bb = ii / kLines, l = ii - bb * kLines;
      return ll_val(words[g.slot0 + (((long long)kk * g.nb + bb) * g.G + jj + l) * kLines + l]);
    };
    const bool up[3] = {j < ncol - 1, i < g.nrow - 1, k < g.nlay - 1};
    const bool low[3] = {k > 0, i > 0, j > 0};
    apc[r] = pivot(k, i, j);
    int p = iapc[r];
#pragma unroll
    for (int e = 0; e < 3; ++e)
      if (low[e])
        apc[p++] = __dmul_rn(__dadd_rn(0.0, v[(1 + e) * N + r]),
                             pivot(k - (e == 0), i - (e == 1), j - (e == 2)));
#pragma unroll
    for (int s = 0; s < 3; ++s)
      if (up[s]) apc[p++] = __dadd_rn(0.0, v[(4 + s) * N + r]);
  }
}

}  // namespace

int launch_dia7_factor(const Dia7 &D, int n, const int *d_iapc, double *d_apc, FactorWords &W, double relax,
                       double delta, int ipcflag, bool dropped, Ctl *ctl, cudaStream_t st) {
  if (factor_words_next(W, st) != 0) return -1;
  LLWord<double> *words = static_cast<LLWord<double> *>(W.words);
  const int grid = std::min((n + 255) / 256, 8 * kNumSM);
  auto *k = dropped ? k_dia7_factor<true> : k_dia7_factor<false>;
  k<<<D.ntickets, kLines, 0, st>>>(D.d_geo, D.nm, n, D.d_sv, words, W.epoch, W.claim, relax, delta, ipcflag, ctl);
  k_dia7_factor_rows<<<grid, 256, 0, st>>>(D.d_geo, D.nm, n, D.d_sv, words, d_iapc, d_apc, ctl);
  return 0;
}

}  // namespace gb
