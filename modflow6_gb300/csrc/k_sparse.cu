// k_sparse.cu -- SELL-32 sparse matrix-vector products.
//
// Replaces amux (src/Utilities/Libraries/sparsekit/sparsekit.f90:1-59) and
// ims_base_residual (src/Solution/LinearMethods/ImsLinearBase.f90:1291-1312).
// One thread per row, one warp per 32-row slice; the k-th entry of every row
// of a slice is contiguous, so each entry column of a slice is one coalesced
// 256-byte value load and one 128-byte index load.  Entries are summed in CSR
// (JA) order with fused multiply-adds, t = fma(a, x, t) from t = 0, the order
// of amux with FMA contraction.
#include "gbims_internal.cuh"
#include "k_krylov.cuh"
#include "k_reduce.cuh"

namespace gb {

void sell_build_host(int n, const std::vector<int> &ia, const std::vector<int> &ja,
                     std::vector<int> &ptr, std::vector<int> &col, std::vector<int> &src) {
  int nslices = (n + kSell - 1) / kSell;
  ptr.assign(nslices + 1, 0);
  long long total = 0;
  for (int s = 0; s < nslices; ++s) {
    int w = 0;
    for (int r = s * kSell; r < std::min(n, (s + 1) * kSell); ++r) w = std::max(w, ia[r + 1] - ia[r]);
    ptr[s] = (int)total;
    total += (long long)w * kSell;
  }
  ptr[nslices] = (int)total;
  col.assign(total, 0);
  src.assign(total, -1);
  for (int s = 0; s < nslices; ++s) {
    int w = (ptr[s + 1] - ptr[s]) / kSell;
    for (int l = 0; l < kSell; ++l) {
      int r = s * kSell + l;
      for (int k = 0; k < w; ++k) {
        long long p = ptr[s] + (long long)k * kSell + l;
        if (r < n && k < ia[r + 1] - ia[r]) {
          col[p] = ja[ia[r] + k];
          src[p] = ia[r] + k;
        } else {
          col[p] = (r < n) ? r : 0;  // padding: zero value times x[row]
          src[p] = -1;
        }
      }
    }
  }
}

__global__ void k_sell_fill(long long nstored, const int *__restrict__ src,
                            const double *__restrict__ amat, double *__restrict__ val,
                            float *__restrict__ val32) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < nstored;
       p += (long long)gridDim.x * blockDim.x) {
    int s = src[p];
    double v = (s >= 0) ? amat[s] : 0.0;
    val[p] = v;
    if (val32) val32[p] = (float)v;
  }
}

void launch_sell_fill(const Sell &S, const double *d_amat, cudaStream_t st) {
  if (S.nstored == 0) return;
  int grid = (int)std::min<long long>((S.nstored + 255) / 256, 8LL * kNumSM);
  k_sell_fill<<<grid, 256, 0, st>>>(S.nstored, S.d_src, d_amat, S.d_val, S.d_val32);
}

// Streaming loads for matrix data (read once per product) keep the L2 for
// the gathered vector.
template <typename T>
__device__ __forceinline__ T ld_stream(const T *p) { return __ldcs(p); }

template <typename T>
__device__ __forceinline__ T mac(T a, T x, T t);
template <>
__device__ __forceinline__ double mac<double>(double a, double x, double t) { return fma(a, x, t); }
template <>
__device__ __forceinline__ float mac<float>(float a, float x, float t) { return fmaf(a, x, t); }

// y = A*x (MODE 0), or d = b - A*x (MODE 1).
template <typename T, int MODE, typename TM = T>
__global__ void __launch_bounds__(256) k_sell_spmv(int n, const int *__restrict__ ptr,
                                                    const int *__restrict__ col,
                                                    const TM *__restrict__ val,
                                                    const T *__restrict__ x,
                                                    const T *__restrict__ b, T *__restrict__ y,
                                                    const Ctl *__restrict__ ctl,
                                                    int only_if_north_due,
                                                    const int *__restrict__ slm,
                                                    const int *__restrict__ mrow, int nm,
                                                    const Ctl *__restrict__ mctl) {
  if (ctl) {
    if (ctl->done) return;
    if (only_if_north_due && !ctl->north_due) return;
  }
  int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= n) return;
  int s = row / kSell, lane = row % kSell;
  if (mctl) {  // batched ensemble: rows of a member that is done are skipped
    int m = slm[s];
    if (m < 0) {
      int lo = 0, hi = nm - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (mrow[mid] <= row) lo = mid;
        else hi = mid - 1;
      }
      m = lo;
    }
    if (mctl[m].done) return;
  }
  int p0 = ptr[s];
  int w = (ptr[s + 1] - p0) / kSell;
  const int *c = col + p0 + lane;
  const TM *v = val + p0 + lane;
  T t = T(0);
  if (w <= 8) {
    // the common 5/7-point case: issue all loads first, then the gathers
    int cc[8];
    TM vv[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k < w) {
        cc[k] = ld_stream(c + k * kSell);
        vv[k] = ld_stream(v + k * kSell);
      }
    }
    T xx[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < w) xx[k] = __ldg(x + cc[k]);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < w) t = mac<T>((T)vv[k], xx[k], t);
  } else {
    for (int k = 0; k < w; ++k)
      t = mac<T>((T)ld_stream(v + k * kSell), __ldg(x + ld_stream(c + k * kSell)), t);
  }
  if (MODE == 0) y[row] = t;
  else y[row] = b[row] - t;
}

static inline int rows_grid(int n) { return (n + 255) / 256; }

// ---------------------------------------------------------------------------
// Full DIS grids (7-point, natural order): the same products without index
// arrays.  Value slot s of row r sits at v[s*n + r], slots in CSR (JA) order
// (diagonal, k-1, i-1, j-1, j+1, i+1, k+1); absent neighbours hold zero and
// are skipped, so every row sums exactly the entries of its CSR row in JA
// order, like the SELL kernel.
// ---------------------------------------------------------------------------
// Which of the slots row r (counted within its grid) has.
struct Dia7Has {
  bool has[7];
  __device__ __forceinline__ Dia7Has(int r, int nlay, int nrow, int ncol) {
    const int nrc = nrow * ncol, k = r / nrc, rem = r - k * nrc, i = rem / ncol, j = rem - i * ncol;
    has[0] = true;
    has[1] = k > 0;
    has[2] = i > 0;
    has[3] = j > 0;
    has[4] = j < ncol - 1;
    has[5] = i < nrow - 1;
    has[6] = k < nlay - 1;
  }
};

__device__ __forceinline__ void dia7_vfill(const Dia7Has &h, long long n, long long r, int p,
                                           const double *__restrict__ amat, double *__restrict__ v,
                                           float *__restrict__ v32) {
#pragma unroll
  for (int s = 0; s < 7; ++s) {
    const double a = h.has[s] ? amat[p++] : 0.0;
    if (v) v[s * n + r] = a;
    if (v32) v32[s * n + r] = (float)a;
  }
}

__global__ void k_dia7_vfill(int nlay, int nrow, int ncol, const int *__restrict__ ia,
                             const double *__restrict__ amat, double *__restrict__ v,
                             float *__restrict__ v32) {
  const long long nrc = (long long)nrow * ncol, n = nrc * nlay;
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < n;
       r += (long long)gridDim.x * blockDim.x)
    dia7_vfill(Dia7Has((int)r, nlay, nrow, ncol), n, r, ia[r], amat, v, v32);
}

// A batch: member grids end to end, kBlocksPerChunk blocks a chunk of rows, so
// that the chain of loads to a member's shape is walked once for several rows:
// a solve of 24 members took 108.8 ms with eight, 108.0 with four, 108.4 with
// two, 110.3 with one.
constexpr int kBlocksPerChunk = 4;
struct BatchRows {
  int m, r, end;
  __device__ __forceinline__ explicit BatchRows(const Dia7Rows &B) {
    const int c = blockIdx.x / kBlocksPerChunk, part = blockIdx.x % kBlocksPerChunk;
    const int first = B.cr[c] + part * (kChunkRows / kBlocksPerChunk);
    m = B.cm[c];
    r = first + threadIdx.x;
    end = min(B.cr[c + 1], first + kChunkRows / kBlocksPerChunk);
  }
};

__global__ void __launch_bounds__(256) k_b_dia7_vfill(Dia7Rows B, const int *__restrict__ ia,
                                                      const double *__restrict__ amat,
                                                      double *__restrict__ v, float *__restrict__ v32) {
  const BatchRows R(B);
  const Dia7Geo g = B.geo[R.m];
  for (int r = R.r; r < R.end; r += 256)
    dia7_vfill(Dia7Has(r - (int)g.row0, g.nlay, g.nrow, g.ncol), B.n, r, ia[r], amat, v, v32);
}

// Row r's product (loads first): its neighbours lie the same distances away in
// a batch, whose members are whole grids.
template <typename T, int MODE, typename TM>
__device__ __forceinline__ void dia7_product(const Dia7Has &h, int nrow, int ncol, int n, int r,
                                             const TM *__restrict__ v, const T *__restrict__ x,
                                             const T *__restrict__ b, T *__restrict__ y) {
  const int nrc = nrow * ncol;
  const int off[7] = {0, -nrc, -ncol, -1, 1, ncol, nrc};
  TM vv[7];
  T xx[7];
#pragma unroll
  for (int s = 0; s < 7; ++s)
    if (h.has[s]) vv[s] = ld_stream(v + (size_t)s * n + r);
#pragma unroll
  for (int s = 0; s < 7; ++s)
    if (h.has[s]) xx[s] = __ldg(x + r + off[s]);
  T t = T(0);
#pragma unroll
  for (int s = 0; s < 7; ++s)
    if (h.has[s]) t = mac<T>((T)vv[s], xx[s], t);
  if (MODE == 0) y[r] = t;
  else y[r] = b[r] - t;
}

template <typename T, int MODE, typename TM = T>
__global__ void __launch_bounds__(256) k_dia7_spmv(int nlay, int nrow, int ncol,
                                                   const TM *__restrict__ v,
                                                   const T *__restrict__ x,
                                                   const T *__restrict__ b, T *__restrict__ y,
                                                   const Ctl *__restrict__ ctl,
                                                   int only_if_north_due) {
  if (ctl) {
    if (ctl->done) return;
    if (only_if_north_due && !ctl->north_due) return;
  }
  const int n = nrow * ncol * nlay;
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  dia7_product<T, MODE>(Dia7Has(r, nlay, nrow, ncol), nrow, ncol, n, r, v, x, b, y);
}

// The same for a batch of full grids; rows of members that are done are
// skipped.  24 members, 1.7 million rows, FP64, cold caches: 52 us a product
// with SELL's index arrays, 37 without (the FP64 pipe's share is 20, the
// bytes' 18), a solve 107.8 -> 102.3 ms.
template <typename T, int MODE>
__global__ void __launch_bounds__(256) k_b_dia7_spmv(Dia7Rows B, const T *__restrict__ v,
                                                     const T *__restrict__ x, const T *__restrict__ b,
                                                     T *__restrict__ y, const Ctl *__restrict__ ctl,
                                                     int only_if_north_due) {
  if (ctl) {
    if (ctl->done) return;
    if (only_if_north_due && !ctl->north_due) return;
  }
  const BatchRows R(B);
  if (B.mctl[R.m].done) return;
  const Dia7Geo g = B.geo[R.m];
  for (int r = R.r; r < R.end; r += 256)
    dia7_product<T, MODE>(Dia7Has(r - (int)g.row0, g.nlay, g.nrow, g.ncol), g.nrow, g.ncol, B.n, r, v,
                          x, b, y);
}

void launch_dia7_vfill(const Dia7 &D, const int *d_ia, const double *d_amat, cudaStream_t st) {
  if (D.rows.nchunks > 0) {
    k_b_dia7_vfill<<<D.rows.nchunks * kBlocksPerChunk, 256, 0, st>>>(D.rows, d_ia, d_amat, D.d_sv, D.f_sv);
    return;
  }
  const long long n = (long long)D.nlay * D.nrow * D.ncol;
  const int grid = (int)std::min<long long>((n + 255) / 256, 8LL * kNumSM);
  k_dia7_vfill<<<grid, 256, 0, st>>>(D.nlay, D.nrow, D.ncol, d_ia, d_amat, D.d_sv, D.f_sv);
}

template <typename T, int MODE>
static void dia7_spmv(const Dia7 &D, const T *v, const T *x, const T *b, T *y, const Ctl *ctl,
                      int only_if_north_due, cudaStream_t st) {
  if (D.rows.nchunks > 0)
    k_b_dia7_spmv<T, MODE><<<D.rows.nchunks * kBlocksPerChunk, 256, 0, st>>>(D.rows, v, x, b, y, ctl,
                                                                            only_if_north_due);
  else
    k_dia7_spmv<T, MODE><<<rows_grid(D.nlay * D.nrow * D.ncol), 256, 0, st>>>(
        D.nlay, D.nrow, D.ncol, v, x, b, y, ctl, only_if_north_due);
}

void launch_dia7_spmv64(const Dia7 &D, const double *x, double *y, const Ctl *ctl,
                        cudaStream_t st) {
  dia7_spmv<double, 0>(D, D.d_sv, x, nullptr, y, ctl, 0, st);
}

void launch_dia7_spmv32(const Dia7 &D, const float *x, float *y, const Ctl *ctl,
                        cudaStream_t st) {
  dia7_spmv<float, 0>(D, D.f_sv, x, nullptr, y, ctl, 0, st);
}

void launch_dia7_residual64(const Dia7 &D, const double *x, const double *b, double *d,
                            const Ctl *ctl, int only_if_north_due, cudaStream_t st) {
  dia7_spmv<double, 1>(D, D.d_sv, x, b, d, ctl, only_if_north_due, st);
}

void launch_spmv64(const Sell &S, const double *x, double *y, const Ctl *ctl, cudaStream_t st) {
  if (S.n == 0) return;
  k_sell_spmv<double, 0><<<rows_grid(S.n), 256, 0, st>>>(S.n, S.d_ptr, S.d_col, S.d_val, x,
                                                          nullptr, y, ctl, 0, S.d_slm, S.d_mrow,
                                                          S.nm, S.mctl);
}

void launch_spmv32(const Sell &S, const float *x, float *y, const Ctl *ctl, cudaStream_t st) {
  if (S.n == 0) return;
  k_sell_spmv<float, 0><<<rows_grid(S.n), 256, 0, st>>>(S.n, S.d_ptr, S.d_col, S.d_val32, x,
                                                         nullptr, y, ctl, 0, S.d_slm, S.d_mrow,
                                                         S.nm, S.mctl);
}

void launch_residual64(const Sell &S, const double *x, const double *b, double *d,
                       const Ctl *ctl, int only_if_north_due, cudaStream_t st) {
  if (S.n == 0) return;
  k_sell_spmv<double, 1><<<rows_grid(S.n), 256, 0, st>>>(S.n, S.d_ptr, S.d_col, S.d_val, x, b,
                                                          d, ctl, only_if_north_due, S.d_slm,
                                                          S.d_mrow, S.nm, S.mctl);
}

// ---------------------------------------------------------------------------
// Products fused with the Krylov steps around them (SpmvFin), for systems
// where launches and the gaps between them are what an iteration costs: the
// search direction's update, the product, its dot product and the scalar are
// one kernel instead of four.  PCG's direction is recomputed at each row's
// neighbours, which doubles the product's FP64 instructions: on large systems,
// where those bound it, the kernels stay apart (kFuseRows, kFuseEntries, with
// both sides measured).  One row a thread, 256 rows a block: the rows, and so
// the partial sums, of k_dot's blocks.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double prod_sum(double a, double b) { return fma(a, b, 0.0); }
__device__ __forceinline__ double prod_sum(float a, float b) {
  CSum s{0.f, 0.f};
  csum_prod(s, a, b);
  return csum_value(s);
}

template <typename T>
struct FinArgs {
  const T *x, *w;
  T *p0, *p1, *y;
  double *part;
  Ctl *ctl;
};

// The vector a product multiplies: x, or P of this iteration from z = x and
// the last P.
template <typename T, int OP>
struct Operand {
  const T *x, *old = nullptr;
  T *now = nullptr;
  T beta = T(0);
  bool first = false;
  __device__ __forceinline__ explicit Operand(const FinArgs<T> &a) : x(a.x) {
    if (OP == 0) {
      const bool odd = a.ctl->iter & 1;
      now = odd ? a.p1 : a.p0;
      old = odd ? a.p0 : a.p1;
      beta = (T)a.ctl->beta;
      first = a.ctl->first != 0;
    }
  }
  struct Raw {
    T a, b;
  };
  __device__ __forceinline__ void load(int i, Raw &r) const {
    r.a = __ldg(x + i);
    if (OP == 0 && !first) r.b = old[i];
  }
  __device__ __forceinline__ T value(const Raw &r) const {
    if (OP == 0) return first ? r.a : mac<T>(beta, r.b, r.a);
    return r.a;
  }
};

// What a block does with its rows' products.
template <typename T, int OP>
__device__ __forceinline__ void finish_rows(const FinArgs<T> &a, int row, bool ok, T own, T t,
                                            const Operand<T, OP> &x) {
  constexpr int NV = OP == 2 ? 2 : 1;
  double v[NV] = {};
  if (ok) {
    a.y[row] = t;
    if (OP == 0) {
      x.now[row] = own;
      v[0] = prod_sum(own, t);
    } else {
      v[0] = OP == 1 ? prod_sum(a.w[row], t) : prod_sum(t, a.w[row]);
      if (OP == 2) v[NV - 1] = prod_sum(t, t);
    }
  }
  block_sum<NV>(v);
  if (threadIdx.x == 0) {
    a.part[blockIdx.x] = v[0];
    if (OP == 2) a.part[gridDim.x + blockIdx.x] = v[NV - 1];
  }
  if (last_block(&a.ctl->fin, gridDim.x))
    finish_dot<OP == 2 ? kFinOmega : kFinAlpha>(a.ctl, a.part, gridDim.x);
}

template <typename T, int OP>
__global__ void __launch_bounds__(kRedBlock) k_dia7_spmv_fin(int nlay, int nrow, int ncol,
                                                             const T *__restrict__ v, FinArgs<T> a) {
  if (a.ctl->done) return;
  const int nrc = nrow * ncol, n = nrc * nlay;
  const int r = blockIdx.x * kRedBlock + threadIdx.x;
  const Operand<T, OP> x(a);
  T t = T(0), own = T(0);
  if (r < n) {
    const int k = r / nrc;
    const int rem = r - k * nrc;
    const int i = rem / ncol, j = rem - i * ncol;
    const bool has[7] = {true, k > 0, i > 0, j > 0, j < ncol - 1, i < nrow - 1, k < nlay - 1};
    const int off[7] = {0, -nrc, -ncol, -1, 1, ncol, nrc};
    T vv[7];
    typename Operand<T, OP>::Raw xx[7];
#pragma unroll
    for (int s = 0; s < 7; ++s)
      if (has[s]) {
        vv[s] = v[(size_t)s * n + r];
        x.load(r + off[s], xx[s]);
      }
    own = x.value(xx[0]);
    t = mac<T>(vv[0], own, t);
#pragma unroll
    for (int s = 1; s < 7; ++s)
      if (has[s]) t = mac<T>(vv[s], x.value(xx[s]), t);
  }
  finish_rows<T, OP>(a, r, r < n, own, t, x);
}

template <typename T, int OP>
__global__ void __launch_bounds__(kRedBlock) k_sell_spmv_fin(int n, const int *__restrict__ ptr,
                                                             const int *__restrict__ col,
                                                             const T *__restrict__ val, FinArgs<T> a) {
  if (a.ctl->done) return;
  const int r = blockIdx.x * kRedBlock + threadIdx.x;
  const Operand<T, OP> x(a);
  T t = T(0), own = T(0);
  if (r < n) {
    const int s = r / kSell, lane = r % kSell;
    const int p0 = ptr[s], w = (ptr[s + 1] - p0) / kSell;
    const int *c = col + p0 + lane;
    const T *v = val + p0 + lane;
    for (int b = 0; b < w; b += 8) {
      int cc[8];
      T vv[8];
      typename Operand<T, OP>::Raw xx[8];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (b + k < w) {
          cc[k] = c[(b + k) * kSell];
          vv[k] = v[(b + k) * kSell];
        }
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (b + k < w) x.load(cc[k], xx[k]);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (b + k < w) {
          const T xv = x.value(xx[k]);
          if (b + k == 0) own = xv;  // the diagonal comes first
          t = mac<T>(vv[k], xv, t);
        }
    }
  }
  finish_rows<T, OP>(a, r, r < n, own, t, x);
}

template <typename T, int OP>
static void spmv_fin_t(const Dia7 *D, const Sell *S, const T *val, const SpmvFin &f, cudaStream_t st) {
  FinArgs<T> a;
  a.x = static_cast<const T *>(f.x);
  a.w = static_cast<const T *>(f.w);
  a.p0 = static_cast<T *>(f.p0);
  a.p1 = static_cast<T *>(f.p1);
  a.y = static_cast<T *>(f.y);
  a.part = f.part;
  a.ctl = f.ctl;
  if (D)
    k_dia7_spmv_fin<T, OP><<<rows_grid(D->nlay * D->nrow * D->ncol), kRedBlock, 0, st>>>(
        D->nlay, D->nrow, D->ncol, val, a);
  else
    k_sell_spmv_fin<T, OP><<<rows_grid(S->n), kRedBlock, 0, st>>>(S->n, S->d_ptr, S->d_col, val, a);
}

void launch_spmv_fin(const Dia7 *D, const Sell *S, bool fp32, const SpmvFin &f, cudaStream_t st) {
  if (!fp32) {
    const double *val = D ? D->d_sv : S->d_val;
    if (f.op == 0) spmv_fin_t<double, 0>(D, S, val, f, st);
    else if (f.op == 1) spmv_fin_t<double, 1>(D, S, val, f, st);
    else spmv_fin_t<double, 2>(D, S, val, f, st);
  } else {
    const float *val = D ? D->f_sv : S->d_val32;
    if (f.op == 0) spmv_fin_t<float, 0>(D, S, val, f, st);
    else if (f.op == 1) spmv_fin_t<float, 1>(D, S, val, f, st);
    else spmv_fin_t<float, 2>(D, S, val, f, st);
  }
}

}  // namespace gb
