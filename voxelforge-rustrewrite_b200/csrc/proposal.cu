// Learned wake proposal: a 32 -> 64 -> 64 -> 1 MLP (ReLU, ReLU, sigmoid) over per-brick
// features, with hand-written fp16 tensor-core forward and backward kernels (mma.sync m16n8k16,
// f16 operands, f32 accumulation), a BCE loss and an Adam step. fp32 master weights; the fp16
// operand copies are refreshed after every step.
//
// The network only proposes which bricks to stage ahead of the exact scheduler; it never decides
// what the fluid computes.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/vf_fluid.h"

namespace vfm {

constexpr int IN = 32, H = 64;
// flat fp32 parameter layout: W1[IN][H] (input-major), b1[H], W2[H][H] (input-major), b2[H],
// w3[H], b3[1]
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + IN * H, OFF_W2 = OFF_B1 + H, OFF_B2 = OFF_W2 + H * H, OFF_W3 = OFF_B2 + H,
              OFF_B3 = OFF_W3 + H, NPARAM = OFF_B3 + 1;
constexpr int WARPS = 4;  // 16-row tiles per CTA = WARPS

struct Dev {
  float* p;       // parameters (fp32 master)
  float* g;       // gradients (fp32)
  float* m;       // Adam first moment
  float* v;       // Adam second moment
  __half* w1t;    // [H][IN]  output-major: B operand of X.W1
  __half* w2t;    // [H][H]   output-major: B operand of H1.W2
  __half* w2n;    // [H][H]   input-major: B operand of dH2.W2^T
  float* loss;    // scratch scalar
  unsigned* ticket;  // CTAs that have added their gradients
};

__device__ __forceinline__ void mma16816(float* c, const unsigned* a, const unsigned* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ unsigned pack2(float lo, float hi) {
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<unsigned*>(&h);
}
__device__ __forceinline__ unsigned ld2(const __half* p) { return *reinterpret_cast<const unsigned*>(p); }

// Four 8x8 blocks of a row-major half matrix in shared memory: lane 8m + r gives the address of row r of
// block m; lane (g, t) gets elements (g, 2t), (g, 2t + 1) of every block, of its transpose with ldsm_t.
__device__ __forceinline__ void ldsm(unsigned (&r)[4], const __half* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((unsigned)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm_t(unsigned (&r)[4], const __half* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((unsigned)__cvta_generic_to_shared(p)));
}

// The network in shared memory, all of it fetched at once: a kernel here is one chain of latencies, and
// the 96 fragment loads of a 16-row tile from L2 were most of it.
constexpr int LDX = IN + 8, LDH = H + 8;  // row strides in halves: eight rows fall into different banks
struct __align__(16) Net {
  __half w1t[H][LDX], w2t[H][LDH];
  float b1[H], b2[H], w3[H], b3;
};
template <int COLS, int LD, int NT>
__device__ __forceinline__ void load_matrix(__half (*dst)[LD], const __half* src) {
#pragma unroll
  for (int k = 0; k < H * COLS / 8 / NT; ++k) {
    const int e = (threadIdx.x + k * NT) * 8;
    *reinterpret_cast<uint4*>(&dst[e / COLS][e % COLS]) = *reinterpret_cast<const uint4*>(src + e);
  }
}
template <int NT>
__device__ __forceinline__ void load_net(const Dev& d, Net& s) {
  static_assert(H * IN / 8 % NT == 0, "whole 16-byte pieces for every thread");
  load_matrix<IN, LDX, NT>(s.w1t, d.w1t);
  load_matrix<H, LDH, NT>(s.w2t, d.w2t);
  if (threadIdx.x < H) {
    s.b1[threadIdx.x] = d.p[OFF_B1 + threadIdx.x];
    s.b2[threadIdx.x] = d.p[OFF_B2 + threadIdx.x];
    s.w3[threadIdx.x] = d.p[OFF_W3 + threadIdx.x];
    if (threadIdx.x == 0) s.b3 = d.p[OFF_B3];
  }
}

// Per-warp forward of 16 rows. Fragment conventions of m16n8k16: g = lane/4, t = lane%4; an A
// fragment holds (row g | g+8) x (cols 2t,2t+1 | 2t+8,2t+9) of a 16x16 tile; an accumulator tile
// (16x8) holds rows g, g+8 x cols 2t, 2t+1; a B fragment holds k = 2t,2t+1 (+8) of column g.
struct Fwd {
  float h1[8][4];  // relu(X W1 + b1): 8 n-tiles of 8 columns
  float h2[8][4];  // relu(H1 W2 + b2)
  float z[2];      // logits of rows g and g+8
};

// The A fragments of a warp's 16 rows of X (16 x 32: two k-steps), rows past the end zero.
__device__ __forceinline__ void load_rows(const __half* X, int row0, int n, unsigned (&a)[2][4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int r0 = row0 + g, r1 = row0 + g + 8;
#pragma unroll
  for (int kk = 0; kk < 2; ++kk) {
    const int c = kk * 16 + 2 * t;
    a[kk][0] = r0 < n ? ld2(X + (size_t)r0 * IN + c) : 0u;
    a[kk][1] = r1 < n ? ld2(X + (size_t)r1 * IN + c) : 0u;
    a[kk][2] = r0 < n ? ld2(X + (size_t)r0 * IN + c + 8) : 0u;
    a[kk][3] = r1 < n ? ld2(X + (size_t)r1 * IN + c + 8) : 0u;
  }
}

__device__ __forceinline__ void forward_tile(const Net& s, const unsigned (&a)[2][4], Fwd& f) {
  const int lane = threadIdx.x & 31, t = lane & 3, m = lane >> 3, l8 = lane & 7;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float c[4] = {0.f, 0.f, 0.f, 0.f};
    unsigned b[4];  // k = 0..31 of columns 8j..8j+7
    ldsm(b, &s.w1t[8 * j + l8][8 * m]);
    mma16816(c, a[0], b);
    mma16816(c, a[1], b + 2);
    const float bb0 = s.b1[8 * j + 2 * t], bb1 = s.b1[8 * j + 2 * t + 1];
    f.h1[j][0] = fmaxf(c[0] + bb0, 0.f);
    f.h1[j][1] = fmaxf(c[1] + bb1, 0.f);
    f.h1[j][2] = fmaxf(c[2] + bb0, 0.f);
    f.h1[j][3] = fmaxf(c[3] + bb1, 0.f);
  }
  // layer 2: A fragments straight from the layer-1 accumulators (k-step kk = tiles 2kk, 2kk+1)
  unsigned a2[4][4];
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    a2[kk][0] = pack2(f.h1[2 * kk][0], f.h1[2 * kk][1]);
    a2[kk][1] = pack2(f.h1[2 * kk][2], f.h1[2 * kk][3]);
    a2[kk][2] = pack2(f.h1[2 * kk + 1][0], f.h1[2 * kk + 1][1]);
    a2[kk][3] = pack2(f.h1[2 * kk + 1][2], f.h1[2 * kk + 1][3]);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      unsigned b[4];
      ldsm(b, &s.w2t[8 * j + l8][32 * kk + 8 * m]);
      mma16816(c, a2[2 * kk], b);
      mma16816(c, a2[2 * kk + 1], b + 2);
    }
    const float bb0 = s.b2[8 * j + 2 * t], bb1 = s.b2[8 * j + 2 * t + 1];
    f.h2[j][0] = fmaxf(c[0] + bb0, 0.f);
    f.h2[j][1] = fmaxf(c[1] + bb1, 0.f);
    f.h2[j][2] = fmaxf(c[2] + bb0, 0.f);
    f.h2[j][3] = fmaxf(c[3] + bb1, 0.f);
  }
  // layer 3: 64 -> 1 dot products, reduced over the 4 threads of a row group
  float z0 = 0.f, z1 = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float w0 = s.w3[8 * j + 2 * t], w1 = s.w3[8 * j + 2 * t + 1];
    z0 += f.h2[j][0] * w0 + f.h2[j][1] * w1;
    z1 += f.h2[j][2] * w0 + f.h2[j][3] * w1;
  }
  z0 += __shfl_xor_sync(0xFFFFFFFFu, z0, 1);
  z0 += __shfl_xor_sync(0xFFFFFFFFu, z0, 2);
  z1 += __shfl_xor_sync(0xFFFFFFFFu, z1, 1);
  z1 += __shfl_xor_sync(0xFFFFFFFFu, z1, 2);
  f.z[0] = z0 + s.b3;
  f.z[1] = z1 + s.b3;
}

__device__ __forceinline__ float sigmoidf_(float z) { return 1.0f / (1.0f + expf(-z)); }

// Probabilities of n rows, 16 a warp. 23,137 rows: 5.0 us, 7.8 with the weights read from L2 (their bytes
// and products take 0.3 us; the rest is launch and one round of latencies).
__global__ void __launch_bounds__(32 * WARPS) k_forward(Dev d, const __half* X, int n, float* prob) {
  __shared__ Net s;
  const int row0 = (blockIdx.x * WARPS + (threadIdx.x >> 5)) * 16;
  unsigned a[2][4];
  load_rows(X, row0, n, a);
  load_net<32 * WARPS>(d, s);
  __syncthreads();
  if (row0 >= n) return;
  Fwd f;
  forward_tile(s, a, f);
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  if (t == 0) {
    if (row0 + g < n) prob[row0 + g] = sigmoidf_(f.z[0]);
    if (row0 + g + 8 < n) prob[row0 + g + 8] = sigmoidf_(f.z[1]);
  }
}

// Sums of v[8j'..] over the eight row groups g: on return lane (g, t) holds those of v[2g], v[2g + 1], that
// is of columns 8g + 2t, 8g + 2t + 1 (each step hands half of the values to the other half of the groups:
// 14 shuffles instead of 48).
__device__ __forceinline__ void column_sums(float (&v)[16], int lane) {
#pragma unroll
  for (int h = 8; h >= 2; h >>= 1) {
    const int o = 2 * h;  // lanes 16, 8, 4 apart
    const bool hi = lane & o;
#pragma unroll
    for (int q = 0; q < h; ++q) {
      const float keep = hi ? v[q + h] : v[q], give = hi ? v[q] : v[q + h];
      v[q] = keep + __shfl_xor_sync(0xFFFFFFFFu, give, o);
    }
  }
}

// Backward of mean BCE-with-logits over n rows; gradients accumulate into d.g (fp32). With `host` (mapped
// host memory) the last CTA to finish moves the sums there and leaves d.g empty.
//
// What bounds it: latency; a training batch of 4096 rows is 64 CTAs and 0.2 GFLOP. A call took 77 us with a
// kernel per 16 rows a warp, two memsets, a copy and two waits; 40 us in this form with the weights read
// from L2 fragment by fragment (kernel 24 us); 26 us with them in shared memory (kernel 11.5 us, of which
// about 3 are the last CTA's). A CTA takes 64 rows a time. Each warp runs the chain of 16 rows forward and back in registers and leaves H1, dZ2, dZ1 and X
// in shared memory; then the warps share out the two weight gradients, which are contractions over the
// 64 rows, so that every sum has one owner and stays in its accumulators until the CTA's rows are done: no
// atomics in shared memory (6,144 per warp when each warp made the products of its own 16 rows), and
// half as many to global memory (pairs).
struct __align__(16) BackSmem {
  static constexpr int ROWS = 16 * WARPS, NSUM = 3 * H + 1;
  Net net;
  __half w2n[H][LDH];
  __half x[ROWS][LDX], h1[ROWS][LDH], d2[ROWS][LDH], d1[ROWS][LDH];
  float sum[WARPS][NSUM + 1];  // column sums of a warp's rows: dw3, db2, db1, db3
  bool last;
};
__global__ void __launch_bounds__(32 * WARPS) k_backward(Dev d, const __half* X, const float* y, int n, float inv_n, float* host) {
  constexpr int ROWS = BackSmem::ROWS, NT = 32 * WARPS, NSUM = BackSmem::NSUM;
  static_assert(WARPS == 4, "the weight gradients are shared out over four warps");
  extern __shared__ __align__(16) unsigned char smem[];
  BackSmem& S = *reinterpret_cast<BackSmem*>(smem);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, m = lane >> 3, l8 = lane & 7;
  float a2[8][4] = {}, a1[4][4] = {}, as[2] = {0.f, 0.f};  // rows 16w of dW2; 16(w & 1) x 32(w >> 1) of dW1; sums
  for (int tile = blockIdx.x; tile * ROWS < n; tile += gridDim.x) {
    const int row0 = tile * ROWS + 16 * w;
    unsigned ax[2][4];
    load_rows(X, row0, n, ax);
    if (tile == (int)blockIdx.x) {
      load_net<NT>(d, S.net);
      load_matrix<H, LDH, NT>(S.w2n, d.w2n);
      __syncthreads();
    }
#pragma unroll
    for (int kk = 0; kk < 2; ++kk)
#pragma unroll
      for (int q = 0; q < 4; ++q) *reinterpret_cast<unsigned*>(&S.x[16 * w + g + 8 * (q & 1)][16 * kk + 2 * t + 8 * (q >> 1)]) = ax[kk][q];
    {
      Fwd f;
      forward_tile(S.net, ax, f);
      const int r0 = row0 + g, r1 = row0 + g + 8;
      const float dz0 = r0 < n ? (sigmoidf_(f.z[0]) - y[r0]) * inv_n : 0.f;
      const float dz1 = r1 < n ? (sigmoidf_(f.z[1]) - y[r1]) * inv_n : 0.f;
      float sz = dz0 + dz1;
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) sz += __shfl_xor_sync(0xFFFFFFFFu, sz, o);
      if (lane == 0) S.sum[w][3 * H] = sz;
      // dw3, dZ2 = dz w3 (relu')
      float d2[8][4], v[16];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c0 = 8 * j + 2 * t;
        const float w0 = S.net.w3[c0], w1 = S.net.w3[c0 + 1];
        v[2 * j] = f.h2[j][0] * dz0 + f.h2[j][2] * dz1;
        v[2 * j + 1] = f.h2[j][1] * dz0 + f.h2[j][3] * dz1;
        d2[j][0] = f.h2[j][0] > 0.f ? dz0 * w0 : 0.f;
        d2[j][1] = f.h2[j][1] > 0.f ? dz0 * w1 : 0.f;
        d2[j][2] = f.h2[j][2] > 0.f ? dz1 * w0 : 0.f;
        d2[j][3] = f.h2[j][3] > 0.f ? dz1 * w1 : 0.f;
        *reinterpret_cast<unsigned*>(&S.h1[16 * w + g][c0]) = pack2(f.h1[j][0], f.h1[j][1]);
        *reinterpret_cast<unsigned*>(&S.h1[16 * w + g + 8][c0]) = pack2(f.h1[j][2], f.h1[j][3]);
        *reinterpret_cast<unsigned*>(&S.d2[16 * w + g][c0]) = pack2(d2[j][0], d2[j][1]);
        *reinterpret_cast<unsigned*>(&S.d2[16 * w + g + 8][c0]) = pack2(d2[j][2], d2[j][3]);
      }
      column_sums(v, lane);
      *reinterpret_cast<float2*>(&S.sum[w][8 * g + 2 * t]) = make_float2(v[0], v[1]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[2 * j] = d2[j][0] + d2[j][2];
        v[2 * j + 1] = d2[j][1] + d2[j][3];
      }
      column_sums(v, lane);
      *reinterpret_cast<float2*>(&S.sum[w][H + 8 * g + 2 * t]) = make_float2(v[0], v[1]);
      // dH1 = dZ2 W2^T (relu'): M = 16, N = 64 (i), K = 64 (j); A from the dZ2 accumulators
      unsigned ad[4][4];
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        ad[kk][0] = pack2(d2[2 * kk][0], d2[2 * kk][1]);
        ad[kk][1] = pack2(d2[2 * kk][2], d2[2 * kk][3]);
        ad[kk][2] = pack2(d2[2 * kk + 1][0], d2[2 * kk + 1][1]);
        ad[kk][3] = pack2(d2[2 * kk + 1][2], d2[2 * kk + 1][3]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
          unsigned b[4];  // B[k=j'][n=i] = W2[i][j'] (input-major copy), columns i = 8j..8j+7
          ldsm(b, &S.w2n[8 * j + l8][32 * kk + 8 * m]);
          mma16816(c, ad[2 * kk], b);
          mma16816(c, ad[2 * kk + 1], b + 2);
        }
        const int c0 = 8 * j + 2 * t;
#pragma unroll
        for (int q = 0; q < 4; ++q) c[q] = f.h1[j][q] > 0.f ? c[q] : 0.f;
        v[2 * j] = c[0] + c[2];
        v[2 * j + 1] = c[1] + c[3];
        *reinterpret_cast<unsigned*>(&S.d1[16 * w + g][c0]) = pack2(c[0], c[1]);
        *reinterpret_cast<unsigned*>(&S.d1[16 * w + g + 8][c0]) = pack2(c[2], c[3]);
      }
      column_sums(v, lane);
      *reinterpret_cast<float2*>(&S.sum[w][2 * H + 8 * g + 2 * t]) = make_float2(v[0], v[1]);
    }
    __syncthreads();
    // dW2[i][j] = sum_r H1[r][i] dZ2[r][j], dW1[i][j] = sum_r X[r][i] dZ1[r][j]; K = 64 (r)
#pragma unroll
    for (int ks = 0; ks < WARPS; ++ks) {
      const int ra = 16 * ks + 8 * (m >> 1) + l8, rb = 16 * ks + 8 * (m & 1) + l8;
      unsigned a[4], b[4];
      ldsm_t(a, &S.h1[ra][16 * w + 8 * (m & 1)]);
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        ldsm_t(b, &S.d2[rb][16 * np + 8 * (m >> 1)]);
        mma16816(a2[2 * np], a, b);
        mma16816(a2[2 * np + 1], a, b + 2);
      }
      ldsm_t(a, &S.x[ra][16 * (w & 1) + 8 * (m & 1)]);
#pragma unroll
      for (int np = 0; np < 2; ++np) {
        ldsm_t(b, &S.d1[rb][32 * (w >> 1) + 16 * np + 8 * (m >> 1)]);
        mma16816(a1[2 * np], a, b);
        mma16816(a1[2 * np + 1], a, b + 2);
      }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int c = (int)threadIdx.x + k * NT;
      if (c < NSUM) as[k] += (S.sum[0][c] + S.sum[1][c]) + (S.sum[2][c] + S.sum[3][c]);
    }
    __syncthreads();
  }
  // ---- the CTA's sums to d.g
  auto add2 = [&](int at, float x, float z) { atomicAdd(reinterpret_cast<float2*>(d.g + at), make_float2(x, z)); };
#pragma unroll
  for (int nj = 0; nj < 8; ++nj) {
    const int at = OFF_W2 + (16 * w + g) * H + 8 * nj + 2 * t;
    add2(at, a2[nj][0], a2[nj][1]);
    add2(at + 8 * H, a2[nj][2], a2[nj][3]);
  }
#pragma unroll
  for (int nj = 0; nj < 4; ++nj) {
    const int at = OFF_W1 + (16 * (w & 1) + g) * H + 32 * (w >> 1) + 8 * nj + 2 * t;
    add2(at, a1[nj][0], a1[nj][1]);
    add2(at + 8 * H, a1[nj][2], a1[nj][3]);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int c = (int)threadIdx.x + k * NT;
    const int at = c < H ? OFF_W3 + c : c < 2 * H ? OFF_B2 + c - H : c < 3 * H ? OFF_B1 + c - 2 * H : OFF_B3;
    if (c < NSUM) atomicAdd(d.g + at, as[k]);
  }
  if (!host) return;
  // ---- the last CTA hands the sums over
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) S.last = atomicAdd(d.ticket, 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!S.last) return;
  __threadfence();
  constexpr int QUADS = NPARAM / 4;
  float4* g4 = reinterpret_cast<float4*>(d.g);
  float4* h4 = reinterpret_cast<float4*>(host);
  float4 q[(QUADS + NT - 1) / NT];  // all under way at once
#pragma unroll
  for (int k = 0; k < (QUADS + NT - 1) / NT; ++k) q[k] = __ldcg(g4 + min((int)threadIdx.x + k * NT, QUADS - 1));
  static_assert(NPARAM == 4 * QUADS + 1, "one parameter past the quads");
  if (threadIdx.x == 0) {
    host[NPARAM - 1] = __ldcg(d.g + NPARAM - 1);
    d.g[NPARAM - 1] = 0.f;
    *d.ticket = 0u;
  }
#pragma unroll
  for (int k = 0; k < (QUADS + NT - 1) / NT; ++k) {
    const int i = (int)threadIdx.x + k * NT;
    if (i >= QUADS) continue;
    h4[i] = q[k];
    g4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// mean BCE-with-logits over n rows (for monitoring)
__global__ void __launch_bounds__(32 * WARPS) k_loss(Dev d, const __half* X, const float* y, int n, float inv_n) {
  __shared__ Net s;
  const int row0 = (blockIdx.x * WARPS + (threadIdx.x >> 5)) * 16;
  unsigned a[2][4];
  load_rows(X, row0, n, a);
  load_net<32 * WARPS>(d, s);
  __syncthreads();
  if (row0 >= n) return;
  Fwd f;
  forward_tile(s, a, f);
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  float l = 0.f;
  if (t == 0) {
    for (int k = 0; k < 2; ++k) {
      int r = row0 + g + 8 * k;
      if (r < n) {
        float z = f.z[k];
        l += fmaxf(z, 0.f) - z * y[r] + log1pf(expf(-fabsf(z)));
      }
    }
  }
  for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xFFFFFFFFu, l, o);
  if (lane == 0) atomicAdd(d.loss, l * inv_n);
}

// Adam on the fp32 master weights, then refresh the fp16 operand copies.
__global__ void k_adam(Dev d, float lr, float b1, float b2, float eps, float c1, float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NPARAM; i += gridDim.x * blockDim.x) {
    float gi = d.g[i];
    float m = b1 * d.m[i] + (1.f - b1) * gi;
    float v = b2 * d.v[i] + (1.f - b2) * gi * gi;
    d.m[i] = m;
    d.v[i] = v;
    d.p[i] -= lr * (m / c1) / (sqrtf(v / c2) + eps);
    d.g[i] = 0.f;
  }
}

__global__ void k_refresh(Dev d) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < H * H + IN * H; i += gridDim.x * blockDim.x) {
    if (i < IN * H) {  // W1[in][out] -> w1t[out][in]
      int in = i / H, out = i % H;
      d.w1t[out * IN + in] = __float2half_rn(d.p[OFF_W1 + i]);
    } else {
      int k = i - IN * H, in = k / H, out = k % H;
      d.w2t[out * H + in] = __float2half_rn(d.p[OFF_W2 + k]);
      d.w2n[in * H + out] = __float2half_rn(d.p[OFF_W2 + k]);
    }
  }
}

}  // namespace vfm

using namespace vfm;

struct vf_mlp {
  int device = 0;
  Dev d{};
  int step = 0;
  int ctas = 1;           // resident CTAs of k_backward
  float* hgrad = nullptr; // mapped host memory the gradients come back in
  float* dgrad = nullptr; // its device address
  std::vector<void*> allocs;
};

namespace {
template <class T>
bool alloc(vf_mlp* h, T** p, size_t n) {
  if (cudaMalloc((void**)p, sizeof(T) * n) != cudaSuccess) return false;
  h->allocs.push_back(*p);
  cudaMemset(*p, 0, sizeof(T) * n);
  return true;
}
void release(vf_mlp* h) {
  for (void* p : h->allocs) cudaFree(p);
  if (h->hgrad) cudaFreeHost(h->hgrad);
  delete h;
}
// The sums' reader empties them; where a call failed it may not have run, so the call that says so does it, and
// takes its error with it (the next call asks for errors of its own).
int failed(vf_mlp* h, cudaStream_t st) {
  cudaMemsetAsync(h->d.g, 0, NPARAM * 4, st);
  cudaMemsetAsync(h->d.ticket, 0, 4, st);
  cudaGetLastError();
  return VF_ERR_CUDA;
}
unsigned blocks_for(uint64_t n) { return (unsigned)((n + 16 * WARPS - 1) / (16 * WARPS)); }
}  // namespace

extern "C" {

int vf_mlp_create(int32_t device, uint64_t seed, vf_mlp** out) {
  if (!out) return VF_ERR_INVALID;
  if (cudaSetDevice(device) != cudaSuccess) return VF_ERR_NO_DEVICE;
  auto* h = new vf_mlp();
  h->device = device;
  if (!alloc(h, &h->d.p, NPARAM) || !alloc(h, &h->d.g, NPARAM) || !alloc(h, &h->d.m, NPARAM) || !alloc(h, &h->d.v, NPARAM) ||
      !alloc(h, &h->d.w1t, H * IN) || !alloc(h, &h->d.w2t, H * H) || !alloc(h, &h->d.w2n, H * H) || !alloc(h, &h->d.loss, 1) || !alloc(h, &h->d.ticket, 1) ||
      cudaHostAlloc((void**)&h->hgrad, NPARAM * 4, cudaHostAllocMapped) != cudaSuccess ||
      cudaHostGetDevicePointer((void**)&h->dgrad, h->hgrad, 0) != cudaSuccess) {
    release(h);
    return VF_ERR_OOM;
  }
  if (cudaFuncSetAttribute(k_backward, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(BackSmem)) != cudaSuccess) {
    release(h);
    return VF_ERR_CUDA;
  }
  int sms = 1;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  h->ctas = 2 * sms;
  // He-uniform init from a splitmix64 stream (host), biases 0
  std::vector<float> p(NPARAM, 0.f);
  uint64_t s = seed * 0x9E3779B97F4A7C15ULL + 1;
  auto rnd = [&]() {
    uint64_t z = (s += 0x9E3779B97F4A7C15ULL);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    z ^= z >> 31;
    return (float)((z >> 11) * (1.0 / 9007199254740992.0)) * 2.f - 1.f;
  };
  const float a1 = std::sqrt(6.f / IN), a2 = std::sqrt(6.f / H), a3 = std::sqrt(3.f / H);
  for (int i = 0; i < IN * H; ++i) p[OFF_W1 + i] = a1 * rnd();
  for (int i = 0; i < H * H; ++i) p[OFF_W2 + i] = a2 * rnd();
  for (int i = 0; i < H; ++i) p[OFF_W3 + i] = a3 * rnd();
  cudaMemcpy(h->d.p, p.data(), NPARAM * 4, cudaMemcpyHostToDevice);
  k_refresh<<<32, 256>>>(h->d);
  if (cudaDeviceSynchronize() != cudaSuccess) {
    release(h);
    return VF_ERR_CUDA;
  }
  *out = h;
  return VF_OK;
}

void vf_mlp_destroy(vf_mlp* h) {
  if (!h) return;
  release(h);
}

int vf_mlp_nparams(void) { return NPARAM; }

int vf_mlp_get_params(vf_mlp* h, float* out) {
  if (!h || !out) return VF_ERR_INVALID;
  return cudaMemcpy(out, h->d.p, NPARAM * 4, cudaMemcpyDeviceToHost) == cudaSuccess ? VF_OK : VF_ERR_CUDA;
}

int vf_mlp_set_params(vf_mlp* h, const float* in) {
  if (!h || !in) return VF_ERR_INVALID;
  if (cudaMemcpy(h->d.p, in, NPARAM * 4, cudaMemcpyHostToDevice) != cudaSuccess) return VF_ERR_CUDA;
  k_refresh<<<32, 256>>>(h->d);
  return cudaDeviceSynchronize() == cudaSuccess ? VF_OK : VF_ERR_CUDA;
}

// probabilities for n feature rows (x: n x 32 fp16, device), out: n fp32 (device)
int vf_mlp_forward(vf_mlp* h, const void* dev_x, uint64_t n, float* dev_prob, void* stream) {
  if (!h || (!dev_x && n)) return VF_ERR_INVALID;
  if (!n) return VF_OK;
  k_forward<<<blocks_for(n), 32 * WARPS, 0, (cudaStream_t)stream>>>(h->d, (const __half*)dev_x, (int)n, dev_prob);
  return cudaGetLastError() == cudaSuccess ? VF_OK : VF_ERR_CUDA;
}

// gradients of the mean BCE over n rows into the flat fp32 host array grads (NPARAM), no update
int vf_mlp_grads(vf_mlp* h, const void* dev_x, const float* dev_y, uint64_t n, float* grads, void* stream) {
  if (!h || !dev_x || !dev_y || !n || !grads) return VF_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  // (d.g is empty between calls: its reader empties it)
  k_backward<<<std::min(blocks_for(n), (unsigned)h->ctas), 32 * WARPS, sizeof(BackSmem), st>>>(h->d, (const __half*)dev_x, dev_y, (int)n, 1.0f / (float)n, h->dgrad);
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) return failed(h, st);
  std::memcpy(grads, h->hgrad, NPARAM * 4);
  return VF_OK;
}

// one Adam step on a minibatch (device arrays); *loss (host, optional) = the batch's mean BCE
// before the step
int vf_mlp_train_step(vf_mlp* h, const void* dev_x, const float* dev_y, uint64_t n, float lr, float* loss, void* stream) {
  if (!h || !dev_x || !dev_y || !n) return VF_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  if (loss) {
    cudaMemsetAsync(h->d.loss, 0, 4, st);
    k_loss<<<blocks_for(n), 32 * WARPS, 0, st>>>(h->d, (const __half*)dev_x, dev_y, (int)n, 1.0f / (float)n);
  }
  k_backward<<<std::min(blocks_for(n), (unsigned)h->ctas), 32 * WARPS, sizeof(BackSmem), st>>>(h->d, (const __half*)dev_x, dev_y, (int)n, 1.0f / (float)n, nullptr);
  h->step += 1;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - std::pow(b1, (float)h->step), c2 = 1.f - std::pow(b2, (float)h->step);
  k_adam<<<(NPARAM + 255) / 256, 256, 0, st>>>(h->d, lr, b1, b2, 1e-8f, c1, c2);
  k_refresh<<<32, 256, 0, st>>>(h->d);
  if (loss) {
    if (cudaMemcpyAsync(loss, h->d.loss, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess) return failed(h, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return failed(h, st);
  }
  return cudaGetLastError() == cudaSuccess ? VF_OK : failed(h, st);
}

}  // extern "C"
