// k_range.cu -- triangular sweeps of general patterns, one launch per sweep.
//
// Replaces the level-by-level sweeps of ims_base_ilu0a
// (src/Solution/LinearMethods/ImsLinearBase.f90:1049-1092) and lusol
// (sparskit2/ilut.f90:465-516) on patterns without the wavefront layout:
// DISV and DISU grids, XT3D's wide rows, ILUT factors.
//
// What bounds such a sweep is its chain of dependent rows, not bytes: a
// hexagon grid of 150 x 150 x 4 cells has 450 levels, and a hand-over from
// row to row through L2 takes about 2 us, while the factor is read in a few
// microseconds.  Most dependencies of a grid's rows are near, though: the
// neighbour before, the row of cells before, the layer above.  So the rows
// are cut into contiguous ranges, one CTA each, and a CTA keeps its range's
// results in shared memory: a hand-over inside a range is a shared-memory
// store and load, and only values that cross into a range travel through L2.
//
// * Results wait in shared memory as slots that hold a quiet NaN of a fixed
//   payload until they are written; the value is its own flag (one 8-byte
//   store), so no fence and no barrier stand between producer and consumer.
//   A NaN result with just this payload is stored as the default NaN.
// * The first slots are the range's own rows, in the order of its slices: the
//   rows of one level, which a warp stores and the next level reads together,
//   lie side by side (in row order a grid's wavefront put all lanes of an
//   access into the same banks, which doubled the time of a sweep).  The
//   following slots are the range's halo: the rows of other ranges it reads.  Fetch warps poll the halo's
//   epoch-tagged words (k_llword.cuh) in the order in which the rows need
//   them and drop each value into its slot, so that a compute warp never
//   waits for an L2 round trip on behalf of one lane.
// * Compute warps take slices of up to 32 rows of one level, a lane a row, the
//   slices of a range in level order and dealt out in turn.  A GB300 FP64
//   instruction holds its sub-partition's pipe for 64 cycles however many
//   lanes it has, so the rows of a slice go through their entries together:
//   entry e of all rows is awaited, then one FMA takes it.  The entries that
//   arrive early are consumed while the warp waits for the last one, which
//   then costs a shared-memory load, a vote, one FMA and a store.  Four
//   compute warps, one a sub-partition: more would share the FP64 pipes
//   (with 8 a sweep took 1.7 times as long).  Each row sums its entries in
//   JAPC order with FMA, as the per-level kernels do: bit-identical results.
// * A slice's operands are one packed block in global memory (its rows, slot
//   numbers, factor values and inverse pivots), which a loader thread brings
//   into a ring of shared-memory buffers with one bulk copy, many slices
//   ahead: the compute warps spend no instructions on addresses and no time
//   on the latency of global loads.
//
// Rows of a level do not depend on one another, slices come in level order,
// and ranges depend only on ranges with smaller tickets (forward: lower
// rows, backward: higher rows), which are resident or finished: the lowest
// unfinished slice can always proceed, and every wait is bounded besides.
//
// Both sweeps, FP64 (before: one launch per sweep, every row's values handed
// over through L2): DISV hexagons 4 x 150 x 150 1885 -> 288 us, XT3D 3 x 70 x 70
// 1668 -> 283 us, ILUT (5, 1e-4) on 6 x 60 x 60 cells 1538 -> 242 us.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cstring>
#include <memory>
#include <new>
#include <thread>

#include "gbims_internal.cuh"
#include "k_llword.cuh"

namespace gb {

namespace {

constexpr int kComputeWarps = 4;  // one per SM sub-partition: each has its own FP64 pipe
constexpr int kFetchWarps = 3;
constexpr int kRangeThreads = 32 * (kComputeWarps + kFetchWarps + 1);  // and the loader's warp
// Shared memory: the ring (kMinStages to kMaxStages buffers of the plan's
// largest block, about kRingBytes) and the range's slots.  A compute warp
// looks kComputeWarps slices ahead, so the ring must hold more than that.
constexpr int kMinStages = 6, kMaxStages = 16;
constexpr size_t kRingBytes = 48 * 1024, kSmemBytes = 216 * 1024;
// Largest block of a plan whose full slices' ring does not fit, which starts
// at about 107 FP64 entries for 32 rows: wide levels of long rows are then cut
// into slices of fewer rows (6 of 256 entries).
constexpr int kNarrowBlock = 16 * 1024;

// A slice's block: a 16-byte header (SliceHead), the row numbers (~row when
// another range reads it), the slot numbers (entry e of row l at e*rows + l),
// the factor values in the same order, the inverse pivots; every part starts
// on 16 bytes.  Shorter rows are padded with zero
// values and the slot that always holds zero: fma(-0, 0, t) is t.
struct BlockLayout {
  int rows, slots, vals, dinv, bytes;
  __host__ __device__ BlockLayout(int nl, int w, int tsize) {
    rows = 16;
    slots = rows + ((4 * nl + 15) & ~15);
    vals = slots + ((2 * w * nl + 15) & ~15);
    dinv = vals + ((tsize * w * nl + 15) & ~15);
    bytes = dinv + ((tsize * nl + 15) & ~15);
  }
};

// The header: rows and the first row's slot, the start of the slot numbers and
// the entries of the longest row (ILUT keeps up to kIlutCap of them, one more
// than eight bits hold), the starts of the values and the pivots.
struct SliceHead {
  int x, y, vals, dinv;
  static SliceHead pack(int nl, int entries, int first, const BlockLayout &L) {
    return {(int)((unsigned)nl | (unsigned)first << 16), (int)((unsigned)L.slots | (unsigned)entries << 16),
            L.vals, L.dinv};
  }
  __host__ __device__ int rows() const { return x & 0xffff; }
  __host__ __device__ unsigned first() const { return (unsigned)x >> 16; }
  __host__ __device__ int entries() const { return (int)((unsigned)y >> 16); }
  __host__ __device__ int slots() const { return y & 0xffff; }
};
static_assert(sizeof(SliceHead) == 16 && kIlutCap < 65536 && kMaxRowLen < 65536,
              "a slice's header is 16 bytes and counts a row's entries in 16 bits");

__device__ __forceinline__ unsigned smem_addr(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void bar_init(unsigned long long *b) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned long long *b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ bool bar_test(unsigned long long *b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// A block into its buffer: bytes a multiple of 16, both ends 16-byte aligned.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes,
                                          unsigned long long *b) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(b))
      : "memory");
}

template <typename T>
struct Slot;
template <>
struct Slot<double> {
  using U = unsigned long long;
  static constexpr U kEmpty = 0x7ff8c0de00000000ULL;
  static __device__ __forceinline__ bool ready(U u) { return (unsigned)(u >> 32) != 0x7ff8c0deu; }
  static __device__ __forceinline__ U bits(double v) { return (U)__double_as_longlong(v); }
  static __device__ __forceinline__ double value(U u) { return __longlong_as_double((long long)u); }
  static __device__ __forceinline__ double fms(double a, double b, double c) { return fma(-a, b, c); }
  static __device__ __forceinline__ U load(unsigned a) {
    U v;
    asm volatile("ld.volatile.shared.b64 %0, [%1];" : "=l"(v) : "r"(a));
    return v;
  }
  static __device__ __forceinline__ void store(unsigned a, double v) {
    const U u = ready(bits(v)) ? bits(v) : 0x7ff8000000000000ULL;
    asm volatile("st.volatile.shared.b64 [%0], %1;" ::"r"(a), "l"(u));
  }
};
template <>
struct Slot<float> {
  using U = unsigned;
  static constexpr U kEmpty = 0x7fc0de01u;
  static __device__ __forceinline__ bool ready(U u) { return u != kEmpty; }
  static __device__ __forceinline__ U bits(float v) { return __float_as_uint(v); }
  static __device__ __forceinline__ float value(U u) { return __uint_as_float(u); }
  static __device__ __forceinline__ float fms(float a, float b, float c) { return fmaf(-a, b, c); }
  static __device__ __forceinline__ U load(unsigned a) {
    U v;
    asm volatile("ld.volatile.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
  }
  static __device__ __forceinline__ void store(unsigned a, float v) {
    const U u = ready(bits(v)) ? bits(v) : 0x7fc00000u;
    asm volatile("st.volatile.shared.b32 [%0], %1;" ::"r"(a), "r"(u));
  }
};

// Waits are bounded by their turns (64 cycles each at the least, so 2 s or
// more; the fetch warps' turns are L2 round trips): a clock, an abort flag or
// a call in the wait loops made a sweep 15 % longer.  A warp whose wait runs
// out sets the error flag and Ctl::done and ends; so do the warps that wait
// for it, when their own waits run out, and the CTAs to come return at once.
constexpr int kWaitTurns = 1 << 26, kFetchTurns = 1 << 23;

template <typename T>
struct RangeArgs {
  int n, R, nr;
  int stages, stage_bytes;     // ring buffers and their size
  const unsigned char *blk;        // the slices' blocks
  const int *off;                  // slice -> its block's start (nslices+1), in 16 bytes
  const int *rslice;               // range -> first slice
  const int *hptr, *halo;          // range -> its halo rows, in order of need
  const T *rhs;                    // forward: r; backward: the forward result
  T *d;
  LLWord<T> *words;
  unsigned long long *ticket;
  unsigned long long recip;  // floor((2^64 - 1) / grid)
  int *err;
  Ctl *ctl;
};

// W entries of a slice's rows, all lanes together: their slots' values are
// read ahead, and each is awaited and taken in turn.  The values are checked
// in registers, and a turn of the wait reads all the entries left again, so
// that those that came with the awaited one are at hand when it is taken.
// False when a wait ran out.
template <typename T, int W>
__device__ __forceinline__ bool take_entries(unsigned slots, const unsigned short *sls,
                                             const T *vals, int nl, T &tv) {
  using S = Slot<T>;
  unsigned at[W];
  T a[W];
  typename S::U v[W];
#pragma unroll
  for (int e = 0; e < W; ++e) at[e] = slots + (unsigned)sizeof(T) * sls[e * nl];
#pragma unroll
  for (int e = 0; e < W; ++e) v[e] = S::load(at[e]);
#pragma unroll
  for (int e = 0; e < W; ++e) a[e] = vals[e * nl];
#pragma unroll
  for (int e = 0; e < W; ++e) {
    int turns = kWaitTurns;
    while (!__all_sync(0xffffffffu, S::ready(v[e]))) {
      if (--turns == 0) return false;
#pragma unroll
      for (int f = e; f < W; ++f) v[f] = S::load(at[f]);
    }
    tv = S::fms(a[e], S::value(v[e]), tv);
  }
  return true;
}

template <typename T, int DIR>
__global__ void __launch_bounds__(kRangeThreads, 1) k_range_sweep(RangeArgs<T> p) {
  using S = Slot<T>;
  using U = typename S::U;
  extern __shared__ __align__(128) unsigned char smem_range[];
  unsigned char *ring = smem_range;
  U *slots = reinterpret_cast<U *>(smem_range + (size_t)p.stages * p.stage_bytes);
  __shared__ unsigned long long full[kMaxStages], empty[kMaxStages];
  __shared__ unsigned s_ep;
  __shared__ int s_t;
  if (threadIdx.x == 0) {
    // every CTA takes a ticket, so launch e owns tickets [e*grid, (e+1)*grid)
    const unsigned long long tk = atomicAdd(p.ticket, 1ULL);
    // (the quotient by the grid's reciprocal, corrected: a 64-bit division is
    // a call, and its calling convention costs the whole kernel registers)
    unsigned long long launch = __umul64hi(tk, p.recip);
    unsigned long long t = tk - launch * gridDim.x;
    while (t >= gridDim.x) {
      t -= gridDim.x;
      ++launch;
    }
    s_t = (int)t;
    s_ep = (unsigned)launch + 1u;
    for (int s = 0; s < p.stages; ++s) {
      bar_init(full + s);
      bar_init(empty + s);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (p.ctl && p.ctl->done) return;
  const int b = (DIR > 0) ? s_t : p.nr - 1 - s_t;
  const unsigned ep = s_ep;
  const int r0 = b * p.R, nloc = min(p.R, p.n - r0);
  const int s0 = p.rslice[b], ns = p.rslice[b + 1] - s0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto give_up = [&] {
    atomicExch(p.err, 1);
    if (p.ctl) p.ctl->done = 1;
  };

  if (warp == kComputeWarps + kFetchWarps) {
    // ---------------- loader ----------------
    // It needs no slot, so it starts before they are initialised; the other
    // warps' barrier below counts its lanes too.
    const int ahead = min(ns, p.stages);
    if (lane == 0)
      for (int s = 0; s < ahead; ++s)
        bulk_load(ring + (size_t)s * p.stage_bytes, p.blk + 16ULL * p.off[s0 + s],
                  16u * (unsigned)(p.off[s0 + s + 1] - p.off[s0 + s]), full + s);
    __syncthreads();
    if (lane != 0) return;
    int issued = ahead, q = 0;
    unsigned parity = 0;
    int o0 = ahead < ns ? p.off[s0 + ahead] : 0, o1 = ahead < ns ? p.off[s0 + ahead + 1] : 0;
    for (int s = ahead; s < ns; ++s) {
      const int o2 = s + 1 < ns ? p.off[s0 + s + 2] : 0;
      int turns = kWaitTurns;
      while (!bar_test(empty + q, parity) && --turns != 0) {
      }
      if (turns == 0) {
        give_up();
        break;
      }
      bulk_load(ring + (size_t)q * p.stage_bytes, p.blk + 16ULL * o0, 16u * (unsigned)(o1 - o0),
                full + q);
      issued = s + 1;
      o0 = o1;
      o1 = o2;
      if (++q == p.stages) {
        q = 0;
        parity ^= 1u;
      }
    }
    // every copy issued has landed before this thread, and so the CTA, ends
    for (int s = max(0, issued - p.stages); s < issued; ++s) {
      int turns = kWaitTurns;
      while (!bar_test(full + s % p.stages, (s / p.stages) & 1) && --turns != 0) {
      }
    }
    return;
  }

  const int h0 = p.hptr[b], nh = p.hptr[b + 1] - h0;
  for (int i = threadIdx.x; i < nloc + nh; i += 32 * (kComputeWarps + kFetchWarps)) slots[i] = S::kEmpty;
  if (threadIdx.x == 0) slots[nloc + nh] = 0;  // the padding entries' slot
  const unsigned slots_at = smem_addr(slots);
  __syncthreads();

  if (warp >= kComputeWarps) {
    // ---------------- fetch warps ----------------
    // Each lane walks two queues of halo entries; a turn issues both loads
    // before it looks at either.
    constexpr int Q = 2, kStep = 32 * Q * kFetchWarps;
    int turns = kFetchTurns;
    int idx[Q], row[Q], nxt[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      idx[q] = ((warp - kComputeWarps) * Q + q) * 32 + lane;
      row[q] = idx[q] < nh ? p.halo[h0 + idx[q]] : -1;
      nxt[q] = idx[q] + kStep < nh ? p.halo[h0 + idx[q] + kStep] : -1;
    }
    while (true) {
      LLRaw w[Q];
      bool more = false;
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (row[q] >= 0) ll_issue(p.words + row[q], w[q]);
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (row[q] >= 0) {
          if (ll_ready<T>(w[q], ep)) {
            T v;
            ll_take(w[q], v);
            S::store(slots_at + (unsigned)sizeof(T) * (nloc + idx[q]), v);
            idx[q] += kStep;
            row[q] = nxt[q];
            nxt[q] = idx[q] + kStep < nh ? p.halo[h0 + idx[q] + kStep] : -1;
          }
          more = more || row[q] >= 0;
        }
      if (!__any_sync(0xffffffffu, more)) return;
      if (--turns == 0) {
        give_up();
        return;
      }
    }
  }

  // ---------------- compute warps ----------------
  // A slice's rows are read, and its right-hand side requested, while the
  // warp works on the one before.  Lanes past a slice's rows follow its last
  // row and store nothing, so that no step of the chain is conditional.
  int n_code = 0;
  T n_rhs = T(0);
  SliceHead n_head = {0, 0, 0, 0};
  int q = warp < ns ? warp : 0, nq = q;  // ring buffers of this slice and the next
  unsigned parity = 0;                   // of the next slice's
  auto ahead = [&]() -> bool {
    int turns = kWaitTurns;
    while (!__all_sync(0xffffffffu, bar_test(full + nq, parity)))
      if (--turns == 0) return false;
    const unsigned char *bl = ring + (unsigned)nq * (unsigned)p.stage_bytes;
    const int4 word = *reinterpret_cast<const int4 *>(bl);
    n_head = {word.x, word.y, word.z, word.w};
    const int l = min(lane, n_head.rows() - 1);
    n_code = reinterpret_cast<const int *>(bl + 16)[l];
    n_rhs = p.rhs[n_code < 0 ? ~n_code : n_code];
    return true;
  };
  bool ok = warp >= ns || ahead();
  for (int s = warp; ok && s < ns; s += kComputeWarps) {
    const unsigned char *bl = ring + (unsigned)q * (unsigned)p.stage_bytes;
    const SliceHead head = n_head;
    const int nl = head.rows(), w = head.entries(), l = min(lane, nl - 1);
    const unsigned own = slots_at + (unsigned)sizeof(T) * (head.first() + lane);
    const int code = n_code, row = code < 0 ? ~code : code;
    T tv = n_rhs;
    nq = q + kComputeWarps;
    if (nq >= p.stages) {
      nq -= p.stages;
      parity ^= 1u;
    }
    ok = s + kComputeWarps >= ns || ahead();
    const unsigned short *sls = reinterpret_cast<const unsigned short *>(bl + head.slots()) + l;
    const T *vals = reinterpret_cast<const T *>(bl + head.vals) + l;
    const T dinv = (DIR < 0) ? reinterpret_cast<const T *>(bl + head.dinv)[l] : T(0);
    int left = w;
    for (; ok && left > 8; left -= 8) {
      ok = take_entries<T, 8>(slots_at, sls, vals, nl, tv);
      sls += 8 * nl;
      vals += 8 * nl;
    }
    if (ok) {
      switch (left) {
        case 1: ok = take_entries<T, 1>(slots_at, sls, vals, nl, tv); break;
        case 2: ok = take_entries<T, 2>(slots_at, sls, vals, nl, tv); break;
        case 3: ok = take_entries<T, 3>(slots_at, sls, vals, nl, tv); break;
        case 4: ok = take_entries<T, 4>(slots_at, sls, vals, nl, tv); break;
        case 5: ok = take_entries<T, 5>(slots_at, sls, vals, nl, tv); break;
        case 6: ok = take_entries<T, 6>(slots_at, sls, vals, nl, tv); break;
        case 7: ok = take_entries<T, 7>(slots_at, sls, vals, nl, tv); break;
        case 8: ok = take_entries<T, 8>(slots_at, sls, vals, nl, tv); break;
        default: break;
      }
    }
    if (!ok) break;
    if (DIR < 0) tv = tv * dinv;
    if (lane < nl) {
      S::store(own, tv);
      if (code < 0) ll_put(p.words + row, tv, ep);
      p.d[row] = tv;
    }
    __syncwarp();
    if (lane == 0) bar_arrive(empty + q);  // the buffer goes back to the loader
    q = nq;
  }
  if (!ok) give_up();
}

// Factor values and inverse pivots into the blocks.
template <typename T>
__global__ void k_range_fill(int nent, const int *__restrict__ src, const int *__restrict__ dst,
                             const T *__restrict__ apc, T *__restrict__ blk) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nent; q += gridDim.x * blockDim.x)
    blk[dst[q]] = apc[src[q]];
}

// On the stream of the kernels that read it: work on a non-blocking stream does
// not wait for copies on the legacy stream.  spare: room for the next pattern.
template <class H, typename V>
bool upload(const H &h, V **d, size_t *cap, bool spare, cudaStream_t st) {
  const size_t n = h.size();
  if (n > *cap || !*d) {
    if (*d) cudaFree(*d);
    *d = nullptr;
    *cap = 0;
    const size_t want = std::max<size_t>(1, n + (spare ? n / 8 : 0));
    if (cudaMalloc((void **)d, sizeof(V) * want) != cudaSuccess) return false;
    *cap = want;
  }
  return n == 0 || cudaMemcpyAsync(*d, h.data(), sizeof(V) * n, cudaMemcpyHostToDevice, st) == cudaSuccess;
}

// Up to `most` threads that do several jobs together, the calling one among them:
// started once (a thread costs some 50 us, an entry of a plan some 10 ns) and
// yielding between jobs, of which there are a few in each millisecond.
constexpr int kPlanThreads = 8;
class Team {
  std::vector<std::thread> others;
  std::atomic<int> job{0}, left{0}, next{0}, count{0};
  std::atomic<bool> ok{true}, end{false};
  bool (*call)(void *, int, int) = nullptr;
  void *what = nullptr;

  void take(int thread) {
    try {
      for (int i; ok.load(std::memory_order_relaxed) && (i = next.fetch_add(1)) < count.load();)
        if (!call(what, i, thread)) ok = false;
    } catch (...) {
      ok = false;
    }
  }

 public:
  Team(long long work, int most) {
    const int want = (int)std::min<long long>({(long long)most, 1 + work / 50000,
                                               (long long)std::max(1u, std::thread::hardware_concurrency())});
    try {
      for (int t = 1; t < want; ++t)
        others.emplace_back([this, t] {
          for (int seen = 0;;) {
            while (job.load(std::memory_order_acquire) == seen && !end) std::this_thread::yield();
            if (end) return;
            ++seen;
            take(t);
            left.fetch_sub(1, std::memory_order_release);
          }
        });
    } catch (...) {  // fewer threads, then
    }
  }
  ~Team() {
    end = true;
    for (std::thread &t : others) t.join();
  }
  Team(const Team &) = delete;
  // f(i, thread) for i < n; false when one returned false or threw.
  template <class F>
  bool run(int n, F f) {
    call = [](void *w, int i, int thread) { return (*static_cast<F *>(w))(i, thread); };
    what = &f;
    next = 0;
    count = n;
    left = (int)others.size();
    job.fetch_add(1, std::memory_order_release);
    take(0);
    while (left.load(std::memory_order_acquire) > 0) std::this_thread::yield();
    return ok;
  }
};

}  // namespace

// The plan of one sweep for ranges of R rows, its slices' blocks of at most
// `block` bytes where they have more than one row; false when a range's slots
// and the ring exceed the shared memory.  `lev`: the rows' levels.  The ranges
// are laid out side by side: one thread took 8 ms for the 930,000 entries of an
// ILUT factor of 100,000 rows, at every factorisation, and most of a first solve.
static bool range_layout(int n, const std::vector<int> &iapc, const std::vector<int> &japc,
                         bool forward, const std::vector<int> &lev, int R, int block, size_t tsize,
                         RangeHost &P) {
  const int nr = (n + R - 1) / R;
  const long long work = (long long)iapc[n] - iapc[0] + n;
  P.R = R;
  P.nr = nr;
  auto first = [&](int r) { return forward ? iapc[r] : japc[r]; };
  auto last = [&](int r) { return forward ? japc[r] : iapc[r + 1]; };
  struct Slice {
    int q, nl, w;
  };
  struct Range {
    std::vector<Slice> slices;
    std::vector<int> halo;
    long long bytes = 0, entries = 0;
    int maxblock = 0;
  };
  std::vector<Range> ranges(nr);
  P.rows.resize(n);
  std::vector<int> place(n);  // row -> its slot, when it is its range's own
  // which rows other ranges read is only known when all blocks are done
  std::unique_ptr<std::atomic<unsigned char>[]> read(new std::atomic<unsigned char>[(size_t)n]);
  struct Scratch {
    std::vector<int> mark, hidx;
    std::vector<size_t> pads;
  };
  // (two words a row and thread: at most 800 MB, or one thread's)
  std::vector<Scratch> scratch((size_t)std::max(1LL, std::min({(long long)kPlanThreads, 100000000LL / n, (long long)nr})));
  Team team(work, (int)scratch.size());
  // the rows of each range in level order, cut into slices of up to 32 rows of
  // one level
  const bool cut = team.run(nr, [&](int b, int) {
    Range &G = ranges[b];
    const int r0 = b * R, nloc = std::min(R, n - r0);
    int lo = INT_MAX, hi = 0;
    for (int r = r0; r < r0 + nloc; ++r) {
      lo = std::min(lo, lev[r]);
      hi = std::max(hi, lev[r]);
      read[r].store(0, std::memory_order_relaxed);
    }
    int *rows = &P.rows[r0];
    if (hi - lo < 4 * nloc) {
      std::vector<int> at(hi - lo + 2, 0);
      for (int r = r0; r < r0 + nloc; ++r) at[lev[r] - lo + 1]++;
      for (size_t l = 1; l < at.size(); ++l) at[l] += at[l - 1];
      for (int r = r0; r < r0 + nloc; ++r) rows[at[lev[r] - lo]++] = r;
    } else {
      for (int q = 0; q < nloc; ++q) rows[q] = r0 + q;
      std::stable_sort(rows, rows + nloc, [&](int a, int c) { return lev[a] < lev[c]; });
    }
    for (int q = 0; q < nloc; ++q) place[rows[q]] = q;
    for (int q0 = 0; q0 < nloc;) {
      int q1 = q0, w = 0;
      const int l0 = lev[rows[q0]];
      for (; q1 < nloc && q1 < q0 + 32 && lev[rows[q1]] == l0; ++q1) {
        const int wide = std::max(w, last(rows[q1]) - first(rows[q1]));
        if (q1 > q0 && BlockLayout(q1 + 1 - q0, wide, (int)tsize).bytes > block) break;
        w = wide;
      }
      if (w > 65535) return false;
      const int bytes = BlockLayout(q1 - q0, w, (int)tsize).bytes;
      G.slices.push_back(Slice{q0, q1 - q0, w});
      G.bytes += bytes;
      G.maxblock = std::max(G.maxblock, bytes);
      q0 = q1;
    }
    for (int r = r0; r < r0 + nloc; ++r) G.entries += last(r) - first(r);
    if (!forward) G.entries += nloc;
    return true;
  });
  if (!cut) return false;
  // where each range's parts start
  std::vector<long long> byte0(nr + 1, 0), entry0(nr + 1, 0);
  P.rslice.assign(nr + 1, 0);
  P.maxblock = 0;
  for (int b = 0; b < nr; ++b) {
    byte0[b + 1] = byte0[b] + ranges[b].bytes;
    entry0[b + 1] = entry0[b] + ranges[b].entries;
    P.rslice[b + 1] = P.rslice[b] + (int)ranges[b].slices.size();
    P.maxblock = std::max(P.maxblock, ranges[b].maxblock);
  }
  if (byte0[nr] / 16 > INT_MAX || byte0[nr] / (long long)tsize > INT_MAX || entry0[nr] > INT_MAX) return false;
  P.stages = (int)std::min<size_t>(kMaxStages, std::max<size_t>(kMinStages, kRingBytes / P.maxblock));
  P.blk.need((size_t)byte0[nr]);
  P.src.need((size_t)entry0[nr]);
  P.dst.need((size_t)entry0[nr]);
  P.off.resize((size_t)P.rslice[nr] + 1);
  P.off[P.rslice[nr]] = (int)(byte0[nr] / 16);
  const bool filled = team.run(nr, [&](int b, int thread) {
    Range &G = ranges[b];
    Scratch &S = scratch[thread];
    if (S.mark.empty()) {
      S.mark.assign(n, -1);
      S.hidx.resize(n);
    }
    S.pads.clear();
    const int r0 = b * R, nloc = std::min(R, n - r0);
    size_t at = (size_t)byte0[b], en = (size_t)entry0[b];
    int s = P.rslice[b];
    unsigned char *blk = P.blk.data();
    int *src = P.src.data(), *dst = P.dst.data();
    for (const Slice &sl : G.slices) {
      const int nl = sl.nl, w = sl.w, *rows = &P.rows[r0 + sl.q];
      const BlockLayout L(nl, w, (int)tsize);
      memset(blk + at, 0, L.bytes);
      const SliceHead head = SliceHead::pack(nl, w, sl.q, L);
      memcpy(blk + at, &head, sizeof(head));
      memcpy(blk + at + L.rows, rows, sizeof(int) * nl);
      unsigned short *slots = reinterpret_cast<unsigned short *>(blk + at + L.slots);
      const int val0 = (int)((at + L.vals) / tsize), dinv0 = (int)((at + L.dinv) / tsize);
      for (int l = 0; l < nl; ++l) {
        const int r = rows[l], j0 = first(r), j1 = last(r);
        for (int j = j0, e = 0; j < j1; ++j, ++e) {
          const int dep = japc[j];
          int slot;
          if (dep >= r0 && dep - r0 < nloc) {
            slot = place[dep];
          } else {
            if (S.mark[dep] != b) {
              S.mark[dep] = b;
              S.hidx[dep] = (int)G.halo.size();
              G.halo.push_back(dep);
              read[dep].store(1, std::memory_order_relaxed);
            }
            slot = nloc + S.hidx[dep];
          }
          if (slot > 65534) return false;
          slots[e * nl + l] = (unsigned short)slot;
          src[en] = j;
          dst[en++] = val0 + e * nl + l;
        }
        for (int e = j1 - j0; e < w; ++e) S.pads.push_back(at + L.slots + 2 * ((size_t)e * nl + l));
        if (!forward) {
          src[en] = r;
          dst[en++] = dinv0 + l;
        }
      }
      P.off[s++] = (int)(at / 16);
      at += L.bytes;
    }
    const int zero = nloc + (int)G.halo.size();  // the slot after the halo
    if (zero > 65535) return false;
    for (size_t sp : S.pads) *reinterpret_cast<unsigned short *>(blk + sp) = (unsigned short)zero;
    return true;
  });
  if (!filled) return false;
  P.hptr.assign(nr + 1, 0);
  P.halo.clear();
  P.maxslots = 0;
  for (int b = 0; b < nr; ++b) {
    const Range &G = ranges[b];
    P.halo.insert(P.halo.end(), G.halo.begin(), G.halo.end());
    P.hptr[b + 1] = (int)P.halo.size();
    P.maxslots = std::max(P.maxslots, std::min(R, n - b * R) + (int)G.halo.size() + 1);
  }
  if ((size_t)P.stages * P.maxblock + tsize * (size_t)P.maxslots > kSmemBytes) return false;
  return team.run(nr, [&](int b, int) {
    for (int s = P.rslice[b]; s < P.rslice[b + 1]; ++s) {
      unsigned char *bl = P.blk.data() + 16 * (size_t)P.off[s];
      SliceHead head;
      memcpy(&head, bl, sizeof(head));
      int *rows = reinterpret_cast<int *>(bl + sizeof(SliceHead));
      for (int l = 0; l < head.rows(); ++l)
        if (read[rows[l]].load(std::memory_order_relaxed)) rows[l] = ~rows[l];
    }
    return true;
  });
}

// The rows' levels in one sweep.
static void sweep_levels(int n, const std::vector<int> &iapc, const std::vector<int> &japc,
                         bool forward, std::vector<int> &lev) {
  lev.assign(n, 0);
  for (int q = 0; q < n; ++q) {
    const int r = forward ? q : n - 1 - q;
    const int j0 = forward ? iapc[r] : japc[r], j1 = forward ? japc[r] : iapc[r + 1];
    int l = 0;
    for (int j = j0; j < j1; ++j) l = std::max(l, lev[japc[j]] + 1);
    lev[r] = l;
  }
}

bool range_build(RangePlan &P, int n, const std::vector<int> &iapc, const std::vector<int> &japc,
                 bool forward, int rows, bool fp32, bool spare, const std::vector<int> *levels,
                 cudaStream_t st) try {
  RangeHost &H = P.host;
  std::vector<int> found;
  if (!levels) sweep_levels(n, iapc, japc, forward, found);
  const std::vector<int> &lev = levels ? *levels : found;
  // full slices in ranges of at least 256 rows, else narrow ones in any
  const int R0 = std::max(32, (rows + 31) / 32 * 32);
  bool fits = false;
  for (int block : {INT_MAX, kNarrowBlock}) {
    const int least = block == INT_MAX ? 256 : 32;
    for (int R = R0; !fits; R = std::max(least, R / 2)) {
      fits = range_layout(n, iapc, japc, forward, lev, R, block, fp32 ? 4 : 8, H);
      if (R <= least) break;
    }
  }
  if (!fits) {
    H = RangeHost();
    return false;
  }
  P.n = n;
  P.R = H.R;
  P.nr = H.nr;
  P.maxslots = H.maxslots;
  P.stages = H.stages;
  P.maxblock = H.maxblock;
  P.nent = (int)H.src.size();
  const bool sent =
      upload(H.blk, &P.d_blk, &P.c_blk, spare, st) && upload(H.off, &P.d_off, &P.c_off, spare, st) &&
      upload(H.rslice, &P.d_rslice, &P.c_rslice, spare, st) && upload(H.src, &P.d_src, &P.c_src, spare, st) &&
      upload(H.dst, &P.d_dst, &P.c_dst, spare, st) && upload(H.hptr, &P.d_hptr, &P.c_hptr, spare, st) &&
      upload(H.halo, &P.d_halo, &P.c_halo, spare, st);
  // the host arrays may go when this returns
  return cudaStreamSynchronize(st) == cudaSuccess && sent;
} catch (const std::bad_alloc &) {
  P.host = RangeHost();
  return false;
}

// Both forms' times from the pattern alone, us a sweep.  Sync-free: 4.5 and 1.6 a
// level.  Over ranges: 5.5, 5 ns for each row and halo entry of the largest
// range, and the longest chain of dependent rows at 0.2 a link inside a range
// and 1.5 across.  Estimated / measured, both sweeps: 60 x 60 x 60 cells 579 / 1323
// sync-free and 298 / 372 in ranges, 1000 x 1000 6406 / 10463 and 2110 / 1956, 1000
// grids of 10 x 10 70 / 76 and 42 / 37, 300 x 300 in random order 60 / 64 and 148 /
// 132, a random graph of 200,000 rows 79 / 142 and 215 / 224, red-black 500 x 500
// 15 / 16 and 62 / 54, 3000 rows without entries 12 / 8 and 32 / 33, a chain of 7
// rows 31 / 19 and 14 / 12.
bool ranges_faster(int n, const std::vector<int> &iapc, const std::vector<int> &japc, int rows,
                   std::vector<int> (&levels)[2]) {
  const int R = std::max(32, (rows + 31) / 32 * 32);
  double free[2], ranges[2];
  Team team((long long)iapc[n] - iapc[0] + n, 2);
  const bool ok = team.run(2, [&](int dir, int) {
    const bool forward = dir == 0;
    std::vector<int> &lev = levels[dir], mark(n, -1);
    std::vector<float> t(n);
    lev.resize(n);
    int nlev = 0, halo = 0, most = 0, last = -1;
    float longest = 0.f;
    for (int q = 0; q < n; ++q) {
      const int r = forward ? q : n - 1 - q, b = r / R;
      const int j0 = forward ? iapc[r] : japc[r], j1 = forward ? japc[r] : iapc[r + 1];
      if (b != last) {
        last = b;
        halo = 0;
      }
      const int r0 = b * R;
      int l = 0;
      float x = 0.f;
      for (int j = j0; j < j1; ++j) {
        const int dep = japc[j];
        const bool own = dep >= r0 && dep - r0 < R;
        l = std::max(l, lev[dep] + 1);
        x = std::max(x, t[dep] + (own ? 0.2f : 1.5f));
        if (!own && mark[dep] != b) {
          mark[dep] = b;
          ++halo;
        }
      }
      lev[r] = l;
      t[r] = x;
      nlev = std::max(nlev, l + 1);
      longest = std::max(longest, x);
      most = std::max(most, halo);
    }
    free[dir] = 4.5 + 1.6 * nlev;
    ranges[dir] = 5.5 + 0.0052 * (std::min(n, R) + most) + longest;
    return true;
  });
  return ok && ranges[0] + ranges[1] <= free[0] + free[1];
}

void range_free(RangePlan &P) {
  void *ptrs[] = {P.d_blk, P.d_off, P.d_rslice, P.d_src, P.d_dst, P.d_hptr, P.d_halo};
  for (void *q : ptrs)
    if (q) cudaFree(q);
  P = RangePlan();
}

template <typename T>
static void fill_t(const RangePlan &P, const T *apc, cudaStream_t st) {
  const int grid = std::max(1, std::min((P.nent + 255) / 256, 8 * kNumSM));
  k_range_fill<T><<<grid, 256, 0, st>>>(P.nent, P.d_src, P.d_dst, apc, reinterpret_cast<T *>(P.d_blk));
}
void launch_range_fill(const RangePlan &F, const RangePlan &B, const double *apc, cudaStream_t st) {
  fill_t<double>(F, apc, st);
  fill_t<double>(B, apc, st);
}
void launch_range_fill32(const RangePlan &F, const RangePlan &B, const float *apc, cudaStream_t st) {
  fill_t<float>(F, apc, st);
  fill_t<float>(B, apc, st);
}

template <typename T, int DIR>
static void sweep_t(const RangePlan &P, const T *rhs, T *d, void *words, unsigned long long *ticket,
                    int *err, Ctl *ctl, cudaStream_t st) {
  RangeArgs<T> a;
  a.n = P.n;
  a.R = P.R;
  a.nr = P.nr;
  a.stages = P.stages;
  a.stage_bytes = P.maxblock;
  a.blk = P.d_blk;
  a.off = P.d_off;
  a.rslice = P.d_rslice;
  a.hptr = P.d_hptr;
  a.halo = P.d_halo;
  a.rhs = rhs;
  a.d = d;
  a.words = static_cast<LLWord<T> *>(words);
  a.ticket = ticket;
  a.recip = ~0ULL / (unsigned long long)P.nr;
  a.err = err;
  a.ctl = ctl;
  static SharedOptIn opt_in;
  opt_in(k_range_sweep<T, DIR>, kSmemBytes);
  const size_t sm = (size_t)P.stages * P.maxblock + ((sizeof(T) * (size_t)P.maxslots + 15) & ~(size_t)15);
  k_range_sweep<T, DIR><<<P.nr, kRangeThreads, sm, st>>>(a);
}

template <typename T>
static void apply_t(const RangePlan &F, const RangePlan &B, const LevelWords &W, const T *r, T *d,
                    Ctl *ctl, cudaStream_t st) {
  sweep_t<T, 1>(F, r, d, W.fwd, W.ticket, W.err, ctl, st);
  sweep_t<T, -1>(B, d, d, W.bwd, W.ticket + 16, W.err, ctl, st);
}
void launch_range_apply(const RangePlan &F, const RangePlan &B, const LevelWords &W, const double *r,
                        double *d, Ctl *ctl, cudaStream_t st) {
  apply_t<double>(F, B, W, r, d, ctl, st);
}
void launch_range_apply32(const RangePlan &F, const RangePlan &B, const LevelWords &W, const float *r,
                          float *d, Ctl *ctl, cudaStream_t st) {
  apply_t<float>(F, B, W, r, d, ctl, st);
}

}  // namespace gb
