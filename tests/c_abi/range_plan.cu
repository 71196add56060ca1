// range_plan.cu -- the plans of the range sweeps (k_range.cu) walked on the
// host: built with the kernel file itself and a stand-in for the CUDA runtime
// (host_cudart.cpp), so that no GPU is needed.
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "k_range.cu"

extern "C" void host_largest(long long bytes);  // host_cudart.cpp

namespace {

// What is wrong with a plan: 0 nothing.
enum { kOk = 0, kNoPlan = 1, kSmem = 2, kSlotEmpty = 3, kSlotTwice = 4, kWordMissing = 5, kBlock = 6, kSpare = 7 };

template <typename T>
int walk(const gb::RangePlan &P, bool forward, const T *apc, const T *rhs, T *out) {
  const size_t smem = (size_t)P.stages * P.maxblock + sizeof(T) * (size_t)P.maxslots;
  const gb::RangeHost &H = P.host;
  const size_t entries = std::max<size_t>(1, H.src.size());
  if (P.c_blk != H.blk.size() || P.c_src != entries || P.c_dst != entries) return kSpare;
  if (P.stages < gb::kMinStages || P.stages > gb::kMaxStages || smem > gb::kSmemBytes) return kSmem;
  T *vals = reinterpret_cast<T *>(P.d_blk);
  for (int q = 0; q < P.nent; ++q) vals[P.d_dst[q]] = apc[P.d_src[q]];
  std::vector<T> word(P.n);
  std::vector<char> there(P.n, 0);
  for (int t = 0; t < P.nr; ++t) {
    const int b = forward ? t : P.nr - 1 - t;
    const int r0 = b * P.R, nloc = std::min(P.R, P.n - r0);
    const int h0 = P.d_hptr[b], nh = P.d_hptr[b + 1] - h0;
    if (nloc + nh + 1 > P.maxslots) return kSmem;
    std::vector<T> slot(nloc + nh + 1, T(0));
    std::vector<char> full(nloc + nh + 1, 0);
    full[nloc + nh] = 1;
    for (int i = 0; i < nh; ++i) {
      const int row = P.d_halo[h0 + i];
      if (!there[row]) return kWordMissing;
      slot[nloc + i] = word[row];
      full[nloc + i] = 1;
    }
    for (int s = P.d_rslice[b]; s < P.d_rslice[b + 1]; ++s) {
      const unsigned char *bl = P.d_blk + 16ULL * P.d_off[s];
      if (16LL * (P.d_off[s + 1] - P.d_off[s]) > P.maxblock) return kBlock;
      gb::SliceHead head;
      std::memcpy(&head, bl, sizeof(head));
      const int nl = head.rows(), w = head.entries();
      if (nl < 1 || nl > 32) return kBlock;
      for (int l = 0; l < nl; ++l) {
        int code;
        std::memcpy(&code, bl + 16 + 4 * l, 4);
        const int row = code < 0 ? ~code : code;
        T tv = rhs[row];
        for (int e = 0; e < w; ++e) {
          unsigned short at;
          T a;
          std::memcpy(&at, bl + head.slots() + 2 * ((size_t)e * nl + l), 2);
          std::memcpy(&a, bl + head.vals + sizeof(T) * ((size_t)e * nl + l), sizeof(T));
          if (at >= slot.size() || !full[at]) return kSlotEmpty;
          tv = std::fma(-a, slot[at], tv);
        }
        if (!forward) {
          T dinv;
          std::memcpy(&dinv, bl + head.dinv + sizeof(T) * l, sizeof(T));
          tv = tv * dinv;
        }
        const size_t own = head.first() + l;
        if (own >= (size_t)nloc || full[own]) return kSlotTwice;
        slot[own] = tv;
        full[own] = 1;
        if (code < 0) {
          word[row] = tv;
          there[row] = 1;
        }
        out[row] = tv;
      }
    }
  }
  return kOk;
}

}  // namespace

// Builds the plan of one sweep in ranges of about `rows` rows and walks it on
// rhs; info: R, ranges, ring buffers, largest block, slices.
extern "C" int range_walk64(int n, const int *iapc, const int *japc, int njapc, const double *apc,
                            int forward, int rows, const double *rhs, double *out, int *info) {
  gb::RangePlan P;
  std::vector<int> ia(iapc, iapc + n + 1), ja(japc, japc + njapc);
  if (!gb::range_build(P, n, ia, ja, forward != 0, rows, false, false, nullptr, nullptr)) return kNoPlan;
  const int v[5] = {P.R, P.nr, P.stages, P.maxblock, (int)P.host.off.size() - 1};
  std::memcpy(info, v, sizeof(v));
  const int rc = walk<double>(P, forward != 0, apc, rhs, out);
  gb::range_free(P);
  return rc;
}

extern "C" int range_walk32(int n, const int *iapc, const int *japc, int njapc, const float *apc,
                            int forward, int rows, const float *rhs, float *out, int *info) {
  gb::RangePlan P;
  std::vector<int> ia(iapc, iapc + n + 1), ja(japc, japc + njapc);
  if (!gb::range_build(P, n, ia, ja, forward != 0, rows, true, false, nullptr, nullptr)) return kNoPlan;
  const int v[5] = {P.R, P.nr, P.stages, P.maxblock, (int)P.host.off.size() - 1};
  std::memcpy(info, v, sizeof(v));
  const int rc = walk<float>(P, forward != 0, apc, rhs, out);
  gb::range_free(P);
  return rc;
}

// A plan where no allocation of more than `bytes` succeeds: kOk or kNoPlan, -1 when
// an exception gets out.
extern "C" int range_starved(int n, const int *iapc, const int *japc, int njapc, int forward, int rows,
                             long long bytes) {
  gb::RangePlan P;
  std::vector<int> ia(iapc, iapc + n + 1), ja(japc, japc + njapc);
  int rc = -1;
  host_largest(bytes);
  try {
    rc = gb::range_build(P, n, ia, ja, forward != 0, rows, false, false, nullptr, nullptr) ? kOk : kNoPlan;
  } catch (const std::bad_alloc &) {
  }
  host_largest(LLONG_MAX);
  gb::range_free(P);
  return rc;
}
