// k_mpnn.cu -- learned warm start: a message-passing network over the IMS
// matrix graph that predicts a time step's head change, trained and run on
// the GPU by the kernels below (no counterpart in the reference, which
// starts every time step from the previous heads).
//
// Network (hidden width H = 64, L = 8 message-passing layers):
//   H0   = relu(X W0 + b0)                        X: N x 16 node features
//   A_l  = S H_{l-1}                               S: normalised conductances
//   Z_l  = [H_{l-1}, A_l] W_l + b_l                (N x 128) (128 x 64)
//   H_l  = H_{l-1} + relu(Z_l)                     l = 1..L
//   y    = H_L w_out + b_out                       predicted scaled head change
// S_ij = c_ij / sqrt(d_i d_j), c_ij = -a_ij the off-diagonal conductance of
// the assembled matrix and d_i = sum_j c_ij, so S is symmetric and the same
// kernel serves the forward and the backward pass.
//
// GEMM operands are BF16, accumulation FP32, on the tensor cores
// (mma.sync m16n8k16 BF16 -> FP32); the residual stream, the loss, the
// gradients and the Adam state are FP32.
#include <algorithm>

#include "k_mpnn.cuh"

namespace gb {

namespace {

constexpr int kH = kMpnnHidden;
constexpr int kIn = kMpnnFeatures;
constexpr int kL = kMpnnLayers;
constexpr int kCat = 2 * kH;

__device__ __forceinline__ void mma_bf16(float (&d)[4], const unsigned (&a)[4],
                                         const unsigned (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}


// Rows of [X | X] operands and weights in shared memory are padded by 8
// elements, so that the 8 rows of a fragment load fall into different banks.
constexpr int kPad = 8;
constexpr int kTile = 64;           // nodes per tile of the layer kernels
constexpr int kLayerThreads = 256;  // 8 warps: 4 row groups of 16 x 2 column halves
constexpr int kHs = kH + 8;         // padded row of the tile's FP32 residual stream

// acc[NT][4] += rows r0..r0+15 of xs (row-major, K wide) times the NT*8
// columns from c0 on of the weights ws (column-major: row c holds column c's
// K entries), k in steps of 16 as one chain per element.
template <int K, int NT>
__device__ __forceinline__ void tile_mma(const __nv_bfloat16 *xs, const __nv_bfloat16 *ws, int r0,
                                         int c0, float (&acc)[NT][4]) {
  constexpr int KP = K + kPad;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int ks = 0; ks < K / 16; ++ks) {
    const int k0 = ks * 16 + 2 * t;
    unsigned a[4];
    a[0] = *reinterpret_cast<const unsigned *>(xs + (r0 + g) * KP + k0);
    a[1] = *reinterpret_cast<const unsigned *>(xs + (r0 + g + 8) * KP + k0);
    a[2] = *reinterpret_cast<const unsigned *>(xs + (r0 + g) * KP + k0 + 8);
    a[3] = *reinterpret_cast<const unsigned *>(xs + (r0 + g + 8) * KP + k0 + 8);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      unsigned b[2];
      b[0] = *reinterpret_cast<const unsigned *>(ws + (c0 + nt * 8 + g) * KP + k0);
      b[1] = *reinterpret_cast<const unsigned *>(ws + (c0 + nt * 8 + g) * KP + k0 + 8);
      mma_bf16(acc[nt], a, b);
    }
  }
}

// Weights (N rows of K, BF16) into padded shared memory, 16 bytes a load.
template <int K, int N>
__device__ __forceinline__ void load_weights(const __nv_bfloat16 *__restrict__ W, __nv_bfloat16 *ws) {
  for (int e = threadIdx.x; e < N * K / 8; e += kLayerThreads) {
    const int r = e / (K / 8), c = e % (K / 8) * 8;
    *reinterpret_cast<uint4 *>(ws + r * (K + kPad) + c) =
        *reinterpret_cast<const uint4 *>(W + (size_t)r * K + c);
  }
}

// Epilogue of a 64-column tile: z = acc + bias, y = max(z, 0) + hold (hold in
// shared memory, or none).  FP32 y; for training also its BF16 copy and the
// mask z > 0 as two 32-bit words a node (bit = column).
template <bool HOLD, bool TRAIN>
__device__ __forceinline__ void layer_epilogue(int n, int row0, int r0, int half,
                                               const float (&acc)[4][4],
                                               const float *__restrict__ bias, const float *hs,
                                               float *__restrict__ Y,
                                               __nv_bfloat16 *__restrict__ Ybf,
                                               unsigned *__restrict__ mask) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int lr = r0 + g + 8 * h, r = row0 + lr;
    unsigned m = 0;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int c = half * 32 + nt * 8 + 2 * t;
      const float z0 = acc[nt][2 * h] + bias[c], z1 = acc[nt][2 * h + 1] + bias[c + 1];
      float y0 = z0 > 0.f ? z0 : 0.f, y1 = z1 > 0.f ? z1 : 0.f;
      if (HOLD) {
        const float2 o = *reinterpret_cast<const float2 *>(hs + lr * kHs + c);
        y0 += o.x;
        y1 += o.y;
      }
      if (TRAIN) m |= (z0 > 0.f ? 1u : 0u) << (nt * 8 + 2 * t) | (z1 > 0.f ? 2u : 0u) << (nt * 8 + 2 * t);
      if (r < n) {
        const size_t o = (size_t)r * kH + c;
        *reinterpret_cast<float2 *>(Y + o) = make_float2(y0, y1);
        if (TRAIN) *reinterpret_cast<__nv_bfloat162 *>(Ybf + o) = __floats2bfloat162_rn(y0, y1);
      }
    }
    if (TRAIN) {
      m |= __shfl_xor_sync(0xffffffffu, m, 1);
      m |= __shfl_xor_sync(0xffffffffu, m, 2);
      if (t == 0 && r < n) mask[(size_t)r * 2 + half] = m;
    }
  }
}

// H0 = relu(X W0 + b0).
template <bool TRAIN>
__global__ void __launch_bounds__(kLayerThreads) k_layer0(int n, const __nv_bfloat16 *__restrict__ X,
                                                          const __nv_bfloat16 *__restrict__ Bt,
                                                          const float *__restrict__ bias,
                                                          float *__restrict__ Y,
                                                          __nv_bfloat16 *__restrict__ Ybf,
                                                          unsigned *__restrict__ mask) {
  __shared__ __align__(16) __nv_bfloat16 xs[kTile * (kIn + kPad)];
  __shared__ __align__(16) __nv_bfloat16 ws[kH * (kIn + kPad)];
  load_weights<kIn, kH>(Bt, ws);
  const int warp = threadIdx.x >> 5, r0 = (warp & 3) * 16, half = warp >> 2;
  const int ntile = (n + kTile - 1) / kTile;
  for (int tl = blockIdx.x; tl < ntile; tl += gridDim.x) {
    const int row0 = tl * kTile;
    __syncthreads();
    if (threadIdx.x < kTile * kIn / 8) {
      const int r = threadIdx.x / (kIn / 8), c = threadIdx.x % (kIn / 8) * 8;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (row0 + r < n) v = *reinterpret_cast<const uint4 *>(X + (size_t)(row0 + r) * kIn + c);
      *reinterpret_cast<uint4 *>(xs + r * (kIn + kPad) + c) = v;
    }
    __syncthreads();
    float acc[4][4] = {};
    tile_mma<kIn, 4>(xs, ws, r0, half * 32, acc);
    layer_epilogue<false, TRAIN>(n, row0, r0, half, acc, bias, nullptr, Y, Ybf, mask);
  }
}

// Sums over the off-diagonal entries of kQ nodes of w * row (FP32, entry
// order): a half-warp a node, a lane 4 of the 64 features.  The nodes' row
// pointers are loaded together, then their first 8 entries, then each node's
// 8 rows at once: the latencies of a tile's nodes overlap.
constexpr int kQ = kTile / 16;  // nodes of a half-warp in a tile
struct Gather {
  int p0[kQ], p1[kQ], j[kQ];
  float w[kQ];
  __device__ __forceinline__ void load(int row0, int n, const int *__restrict__ ia,
                                       const int *__restrict__ ja, const float *__restrict__ wt) {
    const int hw = threadIdx.x >> 4, l16 = threadIdx.x & 15;
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
      const int node = row0 + q * 16 + hw;
      p0[q] = p1[q] = 0;
      if (node < n) {
        p0[q] = ia[node] + 1;
        p1[q] = ia[node + 1];
      }
    }
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
      j[q] = 0;
      w[q] = 0.f;
      if (l16 < 8 && p0[q] + l16 < p1[q]) {
        j[q] = ja[p0[q] + l16];
        w[q] = wt[p0[q] + l16];
      }
    }
  }
  __device__ __forceinline__ float4 sum(int q, const int *__restrict__ ja,
                                        const float *__restrict__ wt, const float *__restrict__ X) {
    const int l16 = threadIdx.x & 15;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    int p = p0[q], jv = j[q];
    float wv = w[q];
    while (true) {
      const int m = p1[q] - p;
      float4 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int jk = __shfl_sync(0xffffffffu, jv, k, 16);
        if (k < m) v[k] = reinterpret_cast<const float4 *>(X + (size_t)jk * kH)[l16];
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float wk = __shfl_sync(0xffffffffu, wv, k, 16);
        if (k < m) {
          a.x = fmaf(wk, v[k].x, a.x);
          a.y = fmaf(wk, v[k].y, a.y);
          a.z = fmaf(wk, v[k].z, a.z);
          a.w = fmaf(wk, v[k].w, a.w);
        }
      }
      p += 8;
      if (!__any_sync(0xffffffffu, p < p1[q])) return a;
      // a node with more than 8 neighbours
      jv = 0;
      wv = 0.f;
      if (l16 < 8 && p + l16 < p1[q]) {
        jv = ja[p + l16];
        wv = wt[p + l16];
      }
    }
  }
};

__device__ __forceinline__ uint2 pack_bf16(float4 v) {
  union {
    __nv_bfloat162 b[2];
    uint2 u;
  } x;
  x.b[0] = __floats2bfloat162_rn(v.x, v.y);
  x.b[1] = __floats2bfloat162_rn(v.z, v.w);
  return x.u;
}

// One message-passing layer, H_l = H_{l-1} + relu([H_{l-1}, S H_{l-1}] W + b),
// in one pass over the nodes.  Bound by memory: 512 bytes a node to and from
// HBM and seven gathered rows of 256 bytes from L2, against 16 kFLOP a node
// of products.  So a tile's aggregation, both halves of its BF16 operand and
// its residual rows stay in shared memory (they used to pass through global
// memory between two kernels), the weights stay there for all of a block's
// tiles, and every access is 8 or 16 bytes.  196,608 nodes of a 7-point graph:
// 251 us a layer as an aggregation and a product kernel, 93 us now (80 us
// without the copies for training); the gathers alone move 350 MB from L2.
template <bool TRAIN>
__global__ void __launch_bounds__(kLayerThreads, 4)
    k_layer(int n, const int *__restrict__ ia, const int *__restrict__ ja, const float *__restrict__ w,
            const float *__restrict__ H, const __nv_bfloat16 *__restrict__ Bt,
            const float *__restrict__ bias, float *__restrict__ Y, __nv_bfloat16 *__restrict__ Abf,
            __nv_bfloat16 *__restrict__ Ybf, unsigned *__restrict__ mask) {
  constexpr int KP = kCat + kPad;
  extern __shared__ __align__(16) unsigned char smem_layer[];
  __nv_bfloat16 *ws = reinterpret_cast<__nv_bfloat16 *>(smem_layer);
  __nv_bfloat16 *xs = ws + kH * KP;
  float *hs = reinterpret_cast<float *>(xs + kTile * KP);
  load_weights<kCat, kH>(Bt, ws);
  const int warp = threadIdx.x >> 5, r0 = (warp & 3) * 16, half = warp >> 2;
  const int hw = threadIdx.x >> 4, l16 = threadIdx.x & 15;
  const int ntile = (n + kTile - 1) / kTile;
  for (int tl = blockIdx.x; tl < ntile; tl += gridDim.x) {
    const int row0 = tl * kTile;
    __syncthreads();  // the last tile's operands are read
    Gather gt;
    gt.load(row0, n, ia, ja, w);
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
      const int r = q * 16 + hw, node = row0 + r;
      float4 own = make_float4(0.f, 0.f, 0.f, 0.f);
      if (node < n) own = reinterpret_cast<const float4 *>(H + (size_t)node * kH)[l16];
      const uint2 a = pack_bf16(gt.sum(q, ja, w, H));
      *reinterpret_cast<float4 *>(hs + r * kHs + 4 * l16) = own;
      *reinterpret_cast<uint2 *>(xs + r * KP + 4 * l16) = pack_bf16(own);
      *reinterpret_cast<uint2 *>(xs + r * KP + kH + 4 * l16) = a;
      if (TRAIN && node < n) *reinterpret_cast<uint2 *>(Abf + (size_t)node * kH + 4 * l16) = a;
    }
    __syncthreads();
    float acc[4][4] = {};
    tile_mma<kCat, 4>(xs, ws, r0, half * 32, acc);
    layer_epilogue<true, TRAIN>(n, row0, r0, half, acc, bias, hs, Y, Ybf, mask);
  }
}

// Four 8x8 BF16 matrices from shared memory, transposed.
__device__ __forceinline__ void ldsm_t4(unsigned (&r)[4], const __nv_bfloat16 *p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}

// The gradient that reaches a layer's output, of the tile's nodes: T + S D
// (T the residual and own-row part, D the aggregated part of the layer
// above, both from its kernel), or dy wout^T below the read-out.  Masked by
// the layer's relu it goes into zs as BF16; the bias gradient's sums are kept
// in db; the unmasked gradient in hs if given.
template <bool TOP>
__device__ __forceinline__ void tile_dz(int n, int row0, const int *__restrict__ ia,
                                        const int *__restrict__ ja, const float *__restrict__ w,
                                        const float *__restrict__ T, const float *__restrict__ D,
                                        const float *__restrict__ dy, const float *__restrict__ wout,
                                        const unsigned *__restrict__ mask, __nv_bfloat16 *zs,
                                        float *hs, float4 &db) {
  const int hw = threadIdx.x >> 4, l16 = threadIdx.x & 15;
  Gather gt;
  if (!TOP) gt.load(row0, n, ia, ja, w);
#pragma unroll
  for (int q = 0; q < kQ; ++q) {
    const int r = q * 16 + hw, node = row0 + r;
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
    unsigned m = 0;
    if (node < n) {
      m = mask[(size_t)node * 2 + (l16 >> 3)] >> (4 * (l16 & 7));
      if (TOP) {
        const float e = dy[node];
        d = make_float4(e * wout[4 * l16], e * wout[4 * l16 + 1], e * wout[4 * l16 + 2],
                        e * wout[4 * l16 + 3]);
      } else {
        d = reinterpret_cast<const float4 *>(T + (size_t)node * kH)[l16];
      }
    }
    if (!TOP) {
      const float4 a = gt.sum(q, ja, w, D);
      d = make_float4(d.x + a.x, d.y + a.y, d.z + a.z, d.w + a.w);
    }
    if (hs) *reinterpret_cast<float4 *>(hs + r * kHs + 4 * l16) = d;
    const float4 z = make_float4(m & 1u ? d.x : 0.f, m & 2u ? d.y : 0.f, m & 4u ? d.z : 0.f,
                                 m & 8u ? d.w : 0.f);
    *reinterpret_cast<uint2 *>(zs + r * (kH + kPad) + 4 * l16) = pack_bf16(z);
    db.x += z.x;
    db.y += z.y;
    db.z += z.z;
    db.w += z.w;
  }
}

// The block's bias-gradient sums into the gradient.
__device__ __forceinline__ void flush_db(float *sb, float4 db, float *__restrict__ g) {
  const int l16 = threadIdx.x & 15;
  __syncthreads();
  if (threadIdx.x < kH) sb[threadIdx.x] = 0.f;
  __syncthreads();
  atomicAdd(sb + 4 * l16, db.x);
  atomicAdd(sb + 4 * l16 + 1, db.y);
  atomicAdd(sb + 4 * l16 + 2, db.z);
  atomicAdd(sb + 4 * l16 + 3, db.w);
  __syncthreads();
  if (threadIdx.x < kH) atomicAdd(g + threadIdx.x, sb[threadIdx.x]);
}

// Backward of one message-passing layer, in one pass over the nodes:
//   dH = T + S D (or dy wout^T), dZ = mask * dH, dW += [H, A]^T dZ, db += dZ,
//   [dX1, dX2] = dZ W^T, Tout = dH + dX1, Dout = dX2
// where the layer below then takes Tout + S Dout as its dH.  Bound by memory
// like the forward layer (1.3 kB a node and seven gathered rows): dZ and dH
// stay in shared memory, and dW is summed in the tensor cores' FP32
// accumulators over all of a block's tiles, a block's sums going out once
// (a reduction per 64 nodes, 8192 atomics each, took 240 of 390 us).
// 196,608 nodes: 392 us a layer in four kernels before, 161 us now.
constexpr int kBwdSmem = (kCat * (kH + kPad) + kTile * (kH + kPad) + kTile * (kCat + kPad)) * 2 +
                         kTile * kHs * 4;
template <bool TOP>
__global__ void __launch_bounds__(kLayerThreads, 2)
    k_layer_bwd(int n, const int *__restrict__ ia, const int *__restrict__ ja,
                const float *__restrict__ w, const float *__restrict__ T, const float *__restrict__ D,
                const float *__restrict__ dy, const float *__restrict__ wout,
                const unsigned *__restrict__ mask, const __nv_bfloat16 *__restrict__ Hbf,
                const __nv_bfloat16 *__restrict__ Abf, const __nv_bfloat16 *__restrict__ W,
                float *__restrict__ Tout, float *__restrict__ Dout, float *__restrict__ gW,
                float *__restrict__ gb) {
  constexpr int KP = kH + kPad, XP = kCat + kPad;
  extern __shared__ __align__(16) unsigned char smem_layer[];
  __shared__ float sb[kH];
  __nv_bfloat16 *ws = reinterpret_cast<__nv_bfloat16 *>(smem_layer);
  __nv_bfloat16 *zs = ws + kCat * KP;
  __nv_bfloat16 *xs = zs + kTile * KP;
  float *hs = reinterpret_cast<float *>(xs + kTile * XP);
  load_weights<kH, kCat>(W, ws);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int r0 = (warp & 3) * 16, half = warp >> 2;
  const int ntile = (n + kTile - 1) / kTile;
  float4 db = make_float4(0.f, 0.f, 0.f, 0.f);
  float dw[8][4] = {};  // rows 16*warp.. of dW, all 64 columns
  for (int tl = blockIdx.x; tl < ntile; tl += gridDim.x) {
    const int row0 = tl * kTile;
    __syncthreads();  // the last tile's operands are read
    for (int e = threadIdx.x; e < kTile * kCat / 8; e += kLayerThreads) {
      const int r = e / (kCat / 8), c = e % (kCat / 8) * 8, node = row0 + r;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (node < n)
        v = *reinterpret_cast<const uint4 *>(c < kH ? Hbf + (size_t)node * kH + c
                                                    : Abf + (size_t)node * kH + (c - kH));
      *reinterpret_cast<uint4 *>(xs + r * XP + c) = v;
    }
    tile_dz<TOP>(n, row0, ia, ja, w, T, D, dy, wout, mask, zs, hs, db);
    __syncthreads();
    // dW += X^T dZ
#pragma unroll
    for (int ks = 0; ks < kTile / 16; ++ks) {
      unsigned a[4];
      ldsm_t4(a, xs + (ks * 16 + (lane & 7) + (lane >> 4) * 8) * XP + warp * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        unsigned b[4];
        ldsm_t4(b, zs + (ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * KP + np * 16 + (lane >> 4) * 8);
        const unsigned b0[2] = {b[0], b[1]}, b1[2] = {b[2], b[3]};
        mma_bf16(dw[2 * np], a, b0);
        mma_bf16(dw[2 * np + 1], a, b1);
      }
    }
    // dX = dZ W^T: warps 0-3 the own-row half, 4-7 the aggregated half
    float acc[8][4] = {};
    tile_mma<kH, 8>(zs, ws, r0, half * kH, acc);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int lr = r0 + g + 8 * h, r = row0 + lr;
      if (r >= n) continue;
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        const int c = nt * 8 + 2 * t;
        float2 v = make_float2(acc[nt][2 * h], acc[nt][2 * h + 1]);
        if (half == 0) {
          const float2 o = *reinterpret_cast<const float2 *>(hs + lr * kHs + c);
          v = make_float2(o.x + v.x, o.y + v.y);
          *reinterpret_cast<float2 *>(Tout + (size_t)r * kH + c) = v;
        } else {
          *reinterpret_cast<float2 *>(Dout + (size_t)r * kH + c) = v;
        }
      }
    }
  }
#pragma unroll
  for (int nt = 0; nt < 8; ++nt)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float *o = gW + (warp * 16 + g + 8 * h) * kH + nt * 8 + 2 * t;
      atomicAdd(o, dw[nt][2 * h]);
      atomicAdd(o + 1, dw[nt][2 * h + 1]);
    }
  flush_db(sb, db, gb);
}

// Backward of the input layer: dZ as above, dW0 += X^T dZ, db0 += dZ.
__global__ void __launch_bounds__(kLayerThreads, 4)
    k_layer0_bwd(int n, const int *__restrict__ ia, const int *__restrict__ ja,
                 const float *__restrict__ w, const float *__restrict__ T, const float *__restrict__ D,
                 const unsigned *__restrict__ mask, const __nv_bfloat16 *__restrict__ X,
                 float *__restrict__ gW, float *__restrict__ gb) {
  constexpr int KP = kH + kPad, XP = kIn + kPad;
  __shared__ __align__(16) __nv_bfloat16 zs[kTile * KP];
  __shared__ __align__(16) __nv_bfloat16 xs[kTile * XP];
  __shared__ float sb[kH];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ntile = (n + kTile - 1) / kTile;
  float4 db = make_float4(0.f, 0.f, 0.f, 0.f);
  float dw[4] = {};  // the 16 rows of dW0, columns 8*warp..
  for (int tl = blockIdx.x; tl < ntile; tl += gridDim.x) {
    const int row0 = tl * kTile;
    __syncthreads();
    if (threadIdx.x < kTile * kIn / 8) {
      const int r = threadIdx.x / (kIn / 8), c = threadIdx.x % (kIn / 8) * 8;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (row0 + r < n) v = *reinterpret_cast<const uint4 *>(X + (size_t)(row0 + r) * kIn + c);
      *reinterpret_cast<uint4 *>(xs + r * XP + c) = v;
    }
    tile_dz<false>(n, row0, ia, ja, w, T, D, nullptr, nullptr, mask, zs, nullptr, db);
    __syncthreads();
#pragma unroll
    for (int kp = 0; kp < kTile / 32; ++kp) {
      // the B fragments of two k-steps of this warp's 8 columns
      unsigned b[4];
      ldsm_t4(b, zs + (kp * 32 + lane) * KP + warp * 8);
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        unsigned a[4];
        ldsm_t4(a, xs + (kp * 32 + s * 16 + (lane & 7) + (lane >> 4) * 8) * XP + ((lane >> 3) & 1) * 8);
        const unsigned bb[2] = {b[2 * s], b[2 * s + 1]};
        mma_bf16(dw, a, bb);
      }
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float *o = gW + (g + 8 * h) * kH + warp * 8 + 2 * t;
    atomicAdd(o, dw[2 * h]);
    atomicAdd(o + 1, dw[2 * h + 1]);
  }
  flush_db(sb, db, gb);
}

// Edge weights S_ij = c_ij / sqrt(d_i d_j) from the assembled matrix.
__global__ void k_edge_deg(int n, const int *__restrict__ ia, const double *__restrict__ amat,
                           float *__restrict__ deg) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double d = 0.0;
    for (int p = ia[i] + 1; p < ia[i + 1]; ++p) d += fmax(-amat[p], 0.0);
    deg[i] = (float)d;
  }
}
__global__ void k_edge_w(int n, const int *__restrict__ ia, const int *__restrict__ ja,
                         const double *__restrict__ amat, const float *__restrict__ deg,
                         float *__restrict__ w) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    w[ia[i]] = 0.f;
    for (int p = ia[i] + 1; p < ia[i + 1]; ++p) {
      const float c = (float)fmax(-amat[p], 0.0);
      const float dd = deg[i] * deg[ja[p]];
      w[p] = dd > 0.f ? c * rsqrtf(dd) : 0.f;
    }
  }
}

__global__ void k_f32_to_bf16(long long n, const float *__restrict__ s, __nv_bfloat16 *__restrict__ d) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    d[i] = __float2bfloat16(s[i]);
}

// y = H wout + bout (one warp per node at a time); with a target also dy.
__global__ void __launch_bounds__(256) k_readout(int n, const float *__restrict__ H,
                                                 const float *__restrict__ wout,
                                                 const float *__restrict__ bout,
                                                 float *__restrict__ y,
                                                 const float *__restrict__ target,
                                                 const float *__restrict__ mask, float inv_count,
                                                 float *__restrict__ dy) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const float w0 = wout[2 * lane], w1 = wout[2 * lane + 1], b = bout[0];
  for (int node = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; node < n; node += warps) {
    const float2 h = reinterpret_cast<const float2 *>(H + (size_t)node * kH)[lane];
    float s = h.x * w0 + h.y * w1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
      const float yv = s + b;
      y[node] = yv;
      if (target) dy[node] = 2.f * ((yv - target[node]) * mask[node]) * inv_count;
    }
  }
}

// loss += sum of the masked squared errors, one FP32 addition a node in node
// order (so that the loss is the same from run to run): 4 cycles a node on
// one thread, 0.4 ms at 200,000 nodes, while the backward pass runs on the
// main stream.  One atomic a node, in any order, took 0.31 ms of the forward
// pass.  The other threads prepare the next 2048 terms meanwhile.
__global__ void __launch_bounds__(256) k_loss(int n, const float *__restrict__ y,
                                              const float *__restrict__ target,
                                              const float *__restrict__ mask, float inv_count,
                                              float *__restrict__ loss) {
  constexpr int kChunk = 2048;
  __shared__ __align__(16) float term[2][kChunk];
  const int nch = (n + kChunk - 1) / kChunk;
  float sum = 0.f;
  for (int c = 0; c <= nch; ++c) {
    if (c < nch && threadIdx.x >= 32)
      for (int k = threadIdx.x - 32; k < kChunk; k += 224) {
        const int i = c * kChunk + k;
        float v = 0.f;
        if (i < n) {
          const float e = (y[i] - target[i]) * mask[i];
          v = e * e * inv_count;
        }
        term[c & 1][k] = v;
      }
    if (c > 0 && threadIdx.x == 0) {
      const float4 *t = reinterpret_cast<const float4 *>(term[(c - 1) & 1]);
#pragma unroll 8
      for (int k = 0; k < kChunk / 4; ++k) {
        const float4 v = t[k];
        sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, v.x), v.y), v.z), v.w);
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(loss, sum);
}

// Read-out backward: dwout += H^T dy, dbout += sum dy.
__global__ void k_readout_bwd(int n, const float *__restrict__ H, const float *__restrict__ dy,
                              float *__restrict__ dwout, float *__restrict__ dbout) {
  __shared__ float sw[kH];
  __shared__ float sb;
  if (threadIdx.x < kH) sw[threadIdx.x] = 0.f;
  if (threadIdx.x == 0) sb = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  float g0 = 0.f, g1 = 0.f, gb = 0.f;
  for (int node = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; node < n; node += warps) {
    const float d = dy[node];
    const float2 h = reinterpret_cast<const float2 *>(H + (size_t)node * kH)[lane];
    g0 = fmaf(d, h.x, g0);
    g1 = fmaf(d, h.y, g1);
    if (lane == 0) gb += d;
  }
  atomicAdd(&sw[2 * lane], g0);
  atomicAdd(&sw[2 * lane + 1], g1);
  if (lane == 0) atomicAdd(&sb, gb);
  __syncthreads();
  if (threadIdx.x < kH) atomicAdd(&dwout[threadIdx.x], sw[threadIdx.x]);
  if (threadIdx.x == 0) atomicAdd(dbout, sb);
}

// Adam (bias-corrected), FP32 master weights.
__global__ void k_adam(int n, float *__restrict__ p, const float *__restrict__ g,
                       float *__restrict__ m, float *__restrict__ v, float lr, float b1, float b2,
                       float c1, float c2, float eps) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// W (K x N, FP32 master) -> Bt (N x K, BF16) for the forward GEMM and
// Wbf (K x N, BF16) for the backward one.
__global__ void k_weights_bf16(int K, int N, const float *__restrict__ W, __nv_bfloat16 *__restrict__ Bt,
                               __nv_bfloat16 *__restrict__ Wbf) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < K * N; e += gridDim.x * blockDim.x) {
    const int k = e / N, c = e % N;
    const __nv_bfloat16 v = __float2bfloat16(W[e]);
    Bt[c * K + k] = v;
    Wbf[e] = v;
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// Parameter layout (FP32): W0 (kIn x kH), b0 (kH), then per layer
// W_l (kCat x kH), b_l (kH), then wout (kH), bout (1).
struct MpnnLayout {
  static constexpr long long w0 = 0, b0 = w0 + kIn * kH;
  static constexpr long long layer0 = b0 + kH, layer_sz = kCat * kH + kH;
  static constexpr long long wout = layer0 + kL * layer_sz, bout = wout + kH;
  static constexpr long long total = bout + 1;
  static constexpr long long W(int l) { return layer0 + (l - 1) * layer_sz; }
  static constexpr long long B(int l) { return W(l) + kCat * kH; }
};

long long mpnn_param_count() { return MpnnLayout::total; }

static int ngrid(long long work, int block) {
  return (int)std::max<long long>(1, std::min<long long>((work + block - 1) / block, 16LL * gb::kNumSM));
}

void mpnn_set_graph(MpnnDev &D, const double *d_amat, cudaStream_t st) {
  k_edge_deg<<<ngrid(D.n, 256), 256, 0, st>>>(D.n, D.ia, d_amat, D.deg);
  k_edge_w<<<ngrid(D.n, 256), 256, 0, st>>>(D.n, D.ia, D.ja, d_amat, D.deg, D.w);
  if (D.amat) cudaMemcpyAsync(D.amat, d_amat, sizeof(double) * D.nja, cudaMemcpyDeviceToDevice, st);
}

// ---- energy loss (mode 1) ----
// e = mask*(dh(y) - dh(t)), tt = mask*dh(t) in head units, dh(u) = soft*sinh(u*scale).
__global__ void k_energy_err(int n, const float *__restrict__ y, const float *__restrict__ t,
                             const float *__restrict__ mask, double soft, double scale,
                             double *__restrict__ ee, double *__restrict__ tt) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double m = mask[i] > 0.f ? 1.0 : 0.0;
    const double dt = soft * sinh((double)t[i] * scale);
    const double dy = soft * sinh((double)y[i] * scale);
    ee[i] = m * (dy - dt);
    tt[i] = m * dt;
  }
}

// we = -A e over the active rows, and per-block partials of e'(-A e) and
// t'(-A t) (epart[2b], epart[2b+1]).
__global__ void k_energy_dots(int n, const int *__restrict__ ia, const int *__restrict__ ja,
                              const double *__restrict__ amat, const float *__restrict__ mask,
                              const double *__restrict__ ee, const double *__restrict__ tt,
                              double *__restrict__ we, double *__restrict__ epart) {
  double s1 = 0.0, s2 = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double ae = 0.0, at = 0.0;
    if (mask[i] > 0.f) {
      for (int k = ia[i]; k < ia[i + 1]; ++k) {
        const int j = ja[k];
        ae = fma(-amat[k], ee[j], ae);
        at = fma(-amat[k], tt[j], at);
      }
    }
    we[i] = ae;
    s1 = fma(ee[i], ae, s1);
    s2 = fma(tt[i], at, s2);
  }
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  __shared__ double sh[2][32];
  if ((threadIdx.x & 31) == 0) {
    sh[0][threadIdx.x >> 5] = s1;
    sh[1][threadIdx.x >> 5] = s2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      a += sh[0][w];
      b += sh[1][w];
    }
    epart[2 * blockIdx.x] = a;
    epart[2 * blockIdx.x + 1] = b;
  }
}

// dy += 2 (W e)_i / t'Wt * dh'(y_i) on active cells and loss += e'We / t'Wt,
// the partials summed in block order by every block.
__global__ void k_energy_grad(int n, int G, const double *__restrict__ epart,
                              const double *__restrict__ we, const float *__restrict__ y,
                              const float *__restrict__ mask, double soft, double scale,
                              float *__restrict__ dy, float *__restrict__ loss) {
  __shared__ double s_inv;
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int q = 0; q < G; ++q) {
      a += epart[2 * q];
      b += epart[2 * q + 1];
    }
    s_inv = (b > 0.0) ? 1.0 / b : 0.0;
    if (blockIdx.x == 0) atomicAdd(loss, (float)(a * s_inv));
  }
  __syncthreads();
  const double inv = s_inv;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (!(mask[i] > 0.f)) continue;
    const double d = soft * scale * cosh((double)y[i] * scale);
    dy[i] += (float)(2.0 * we[i] * inv * d);
  }
}

void mpnn_refresh_bf16(MpnnDev &D, cudaStream_t st) {
  using P = MpnnLayout;
  k_weights_bf16<<<ngrid(kIn * kH, 256), 256, 0, st>>>(kIn, kH, D.p + P::w0, D.bt0, D.wbf0);
  for (int l = 1; l <= kL; ++l)
    k_weights_bf16<<<ngrid(kCat * kH, 256), 256, 0, st>>>(kCat, kH, D.p + P::W(l), D.bt[l - 1],
                                                          D.wbf[l - 1]);
}

// The network's input for a warm-start guess, written as BF16: the static
// columns of `stat` (n x kIn: standardised ln K, well rate, CHD mask, layer
// position, bias), column 1 the previous heads (x - head_ref) / head_scale,
// column 6 the previous step's head change in network units
// asinh(dh / dh_soft) / dh_scale (zero on the first step and on inactive
// cells).
__global__ void k_guess_features(int n, const float *__restrict__ stat, const double *__restrict__ x,
                                 const double *__restrict__ xold, int first,
                                 const int *__restrict__ ibound, GuessScaling sc,
                                 __nv_bfloat16 *__restrict__ xbf) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < (long long)n * kIn;
       q += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(q / kIn), f = (int)(q % kIn);
    float v;
    if (f == 1) {
      v = (float)((x[i] - sc.head_ref) / sc.head_scale);
    } else if (f == 6) {
      const double dh = (first || ibound[i] <= 0) ? 0.0 : x[i] - xold[i];
      v = (float)(asinh(dh / sc.dh_soft) / sc.dh_scale);
    } else {
      v = stat[q];
    }
    xbf[q] = __float2bfloat16(v);
  }
}

// guess = x + sinh(clamp(y) * dh_scale) * dh_soft on active cells, x elsewhere
__global__ void k_guess_out(int n, const float *__restrict__ y, const double *__restrict__ x,
                            const int *__restrict__ ibound, GuessScaling sc,
                            double *__restrict__ guess) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double u = (double)y[i];
    if (sc.unit_max > 0.0) u = fmin(fmax(u, -sc.unit_max), sc.unit_max);
    const double dh = sinh(u * sc.dh_scale) * sc.dh_soft;
    guess[i] = (ibound[i] > 0) ? x[i] + dh : x[i];
  }
}

static void forward_from_xbf(MpnnDev &D, const float *target, const float *mask, float inv_count,
                             cudaStream_t st);

void mpnn_guess(MpnnDev &D, const float *d_static, const double *x, const double *xold,
                int first, const int *ibound, const GuessScaling &sc, double *guess,
                cudaStream_t st) {
  const int n = D.n;
  k_guess_features<<<ngrid((long long)n * kIn, 256), 256, 0, st>>>(n, d_static, x, xold, first,
                                                                    ibound, sc, D.xbf);
  forward_from_xbf(D, nullptr, nullptr, 0.f, st);
  k_guess_out<<<ngrid(n, 256), 256, 0, st>>>(n, D.y, x, ibound, sc, guess);
}

// Forward pass from features (N x kIn FP32); y (N) written.  With a target,
// the loss and dy are produced too.
void mpnn_forward(MpnnDev &D, const float *d_x, const float *target, const float *mask,
                  float inv_count, cudaStream_t st) {
  const int n = D.n;
  k_f32_to_bf16<<<ngrid((long long)n * kIn, 256), 256, 0, st>>>((long long)n * kIn, d_x, D.xbf);
  forward_from_xbf(D, target, mask, inv_count, st);
}

// Blocks of the layer kernel: as many as are resident, each with the weights
// in shared memory and a stride of tiles.
constexpr size_t kLayerSmem = (kH + kTile) * (kCat + kPad) * 2 + kTile * kHs * 4;
template <bool TRAIN>
static int layer_grid(int tiles) {
  static SharedOptIn opt_in;
  opt_in(k_layer<TRAIN>, kLayerSmem);
  static const int per_sm = [] {  // every device is a GB300
    int occ = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_layer<TRAIN>, kLayerThreads, kLayerSmem);
    return std::max(1, occ);
  }();
  return std::min(per_sm * kNumSM, tiles);
}

// The layers, H[0] to H[kL].  Without a target nothing is kept for a backward
// pass: no BF16 copies, no masks, and the residual stream alternates between
// two buffers (100 MB at 200,000 nodes, which stay in L2).
template <bool TRAIN>
static void forward_layers(MpnnDev &D, cudaStream_t st) {
  using P = MpnnLayout;
  const int n = D.n;
  const int tiles = (n + kTile - 1) / kTile;
  k_layer0<TRAIN><<<std::min(tiles, 8 * kNumSM), kLayerThreads, 0, st>>>(
      n, D.xbf, D.bt0, D.p + P::b0, D.H[0], D.Hbf[0], D.mask[0]);
  const int grid = layer_grid<TRAIN>(tiles);
  for (int l = 1; l <= kL; ++l) {
    float *in = D.H[TRAIN ? l - 1 : (l - 1) & 1], *out = D.H[TRAIN ? l : l & 1];
    k_layer<TRAIN><<<grid, kLayerThreads, kLayerSmem, st>>>(n, D.ia, D.ja, D.w, in, D.bt[l - 1],
                                                      D.p + P::B(l), out, D.Abf[l], D.Hbf[l],
                                                      D.mask[l]);
  }
}

static void forward_from_xbf(MpnnDev &D, const float *target, const float *mask, float inv_count,
                             cudaStream_t st) {
  using P = MpnnLayout;
  const int n = D.n;
  static_assert(kL % 2 == 0, "the last layer's output in H[0] without a target");
  const float *top = target ? D.H[kL] : D.H[0];
  if (target) forward_layers<true>(D, st);
  else forward_layers<false>(D, st);
  if (target) cudaMemsetAsync(D.loss, 0, sizeof(float), st);
  const bool energy = target && D.energy;
  const float inv_loss = energy ? inv_count * D.mse_w : inv_count;
  k_readout<<<ngrid((long long)n * 32, 256), 256, 0, st>>>(
      n, top, D.p + P::wout, D.p + P::bout, D.y, target, mask, inv_loss, D.dy);
  if (target) {
    // on a stream of its own beside what follows; mpnn_backward waits for it
    cudaEventRecord(D.fork, st);
    cudaStreamWaitEvent(D.side, D.fork, 0);
    k_loss<<<1, 256, 0, D.side>>>(n, D.y, target, mask, inv_loss, D.loss);
    cudaEventRecord(D.join, D.side);
  }
  if (energy) {
    const int G = std::min(kMpnnRedBlocks, (n + 255) / 256);
    k_energy_err<<<ngrid(n, 256), 256, 0, st>>>(n, D.y, target, mask, D.dh_soft, D.dh_scale, D.ee, D.tt);
    k_energy_dots<<<G, 256, 0, st>>>(n, D.ia, D.ja, D.amat, mask, D.ee, D.tt, D.we, D.epart);
    k_energy_grad<<<ngrid(n, 256), 256, 0, st>>>(n, G, D.epart, D.we, D.y, mask, D.dh_soft,
                                                 D.dh_scale, D.dy, D.loss);
  }
}

// Backward pass after mpnn_forward with a target: gradients into D.g.
void mpnn_backward(MpnnDev &D, cudaStream_t st) {
  using P = MpnnLayout;
  const int n = D.n;
  cudaMemsetAsync(D.g, 0, sizeof(float) * P::total, st);
  k_readout_bwd<<<ngrid((long long)n * 32, 256), 256, 0, st>>>(n, D.H[kL], D.dy, D.g + P::wout,
                                                               D.g + P::bout);
  const int tiles = (n + kTile - 1) / kTile;
  static SharedOptIn opt_in[2];
  opt_in[0](k_layer_bwd<true>, kBwdSmem);
  opt_in[1](k_layer_bwd<false>, kBwdSmem);
  // two blocks an SM fill the register files; one place is left for the loss
  // kernel beside them (a block without a place would run after all others
  // and double the layer's time)
  const int grid = std::min(tiles, 2 * kNumSM - 1);
  for (int l = kL; l >= 1; --l) {
    const int in = l & 1, out = in ^ 1;
    if (l == kL)
      k_layer_bwd<true><<<grid, kLayerThreads, kBwdSmem, st>>>(
          n, D.ia, D.ja, D.w, nullptr, nullptr, D.dy, D.p + P::wout, D.mask[l], D.Hbf[l - 1],
          D.Abf[l], D.wbf[l - 1], D.T[out], D.A[out], D.g + P::W(l), D.g + P::B(l));
    else
      k_layer_bwd<false><<<grid, kLayerThreads, kBwdSmem, st>>>(
          n, D.ia, D.ja, D.w, D.T[in], D.A[in], nullptr, nullptr, D.mask[l], D.Hbf[l - 1],
          D.Abf[l], D.wbf[l - 1], D.T[out], D.A[out], D.g + P::W(l), D.g + P::B(l));
  }
  k_layer0_bwd<<<std::min(tiles, 4 * kNumSM - 1), kLayerThreads, 0, st>>>(
      n, D.ia, D.ja, D.w, D.T[0], D.A[0], D.mask[0], D.xbf, D.g + P::w0, D.g + P::b0);
  cudaStreamWaitEvent(st, D.join, 0);  // the loss of the forward pass
}

void mpnn_adam(MpnnDev &D, float lr, cudaStream_t st) {
  const float b1 = 0.9f, b2 = 0.999f;
  D.steps += 1;
  const float c1 = 1.f - powf(b1, (float)D.steps), c2 = 1.f - powf(b2, (float)D.steps);
  k_adam<<<ngrid(MpnnLayout::total, 256), 256, 0, st>>>((int)MpnnLayout::total, D.p, D.g, D.m, D.v,
                                                        lr, b1, b2, c1, c2, 1e-8f);
  mpnn_refresh_bf16(D, st);
}

}  // namespace gb
