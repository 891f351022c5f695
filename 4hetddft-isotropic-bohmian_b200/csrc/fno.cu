// fno.cu -- forward and backward kernels of the Fourier neural operator used
// as the coarse propagator of the parareal driver, plus the grid transfers
// between the solver grid and the FNO grid.  BF16 weights, FP32 activations
// and FP32 accumulation; every reduction runs in a fixed order, so training
// is run-to-run reproducible.
//
// A Fourier layer is  v' = act(W v + b + K v),  K v = F^-1 (R . F v)|modes,
// where F keeps mx x my x mz modes (kx in [0, mx), ky, kz in the lowest
// |k|).  The truncated transforms are dense contractions with small DFT
// matrices (he4_fno_contract), applied axis by axis; their adjoints are the
// same contractions with the conjugate-transposed matrices and the real /
// complex flags swapped, which is how the backward pass runs them.
#include <cuda_bf16.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/he4_fno.h"
#include "common.cuh"
#include "reduce.cuh"

namespace he4 {
namespace fno {

constexpr int kThreads = 256;

// 32-bit element indices, with room for a grid-stride step past the end
static inline bool fits32(int64_t n) { return n < (1ll << 31); }

static inline unsigned blocks_for(int64_t n, int t = kThreads) {
  return (unsigned)std::min<int64_t>((n + t - 1) / t, (int64_t)148 * 32);
}
static inline unsigned mix_blocks(int64_t n) { return blocks_for(n, 32); }

__device__ __forceinline__ float bf(uint16_t u) { return __uint_as_float((uint32_t)u << 16); }

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
  return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

// packed FP32 pairs (sm_100 f32x2 arithmetic, round to nearest as the scalar form)
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2,%3};\n\tmov.b64 rb, {%4,%5};\n\tmov.b64 rc, {%6,%7};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0,%1}, rd;}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}

// ---------------------------------------------------------------------------
// axis contraction  y[o][k][r] = sum_j A[k][j] x[o][j][r]
// ---------------------------------------------------------------------------
// A CTA owns kCols columns (o, r) and every output mode; lanes are columns, so
// the KT entries A[k0..][j] of a step are one broadcast read.  JS = 1: warps take
// groups of KT outputs.  JS > 1 (KT covers every output): warps take slices of
// j, whose sums are added in order through shared memory, so that each input is
// loaded by one thread.  The kernels are bound by load latency, not by bytes or
// products: kJ loads per thread are in flight while A is staged, eight slices
// leave a 64-point axis one such round, and the index arithmetic is 32-bit.
// 64^3, width 32, one sample: 64 -> 12 modes along y / z 16.8 -> 6.5 us a pass, 12 -> 64 14.5 -> 7.8 us.
constexpr int kCols = 32;
template <bool IN_REAL, bool OUT_REAL, int KT, int JS>
__global__ void __launch_bounds__(512) k_contract(const void *__restrict__ xv, void *__restrict__ yv,
                                                  const float2 *__restrict__ A, unsigned ncol, int J, int K,
                                                  unsigned inner, int accumulate) {
  extern __shared__ __align__(16) float2 sA[];  // [J][Kp], Kp = K rounded up to KT, zero-padded; [JS][KT][kCols]
  constexpr int kJ = JS > 1 ? 8 : 16;
  const int Kp = (K + KT - 1) / KT * KT;
  const int lane = threadIdx.x % kCols, wp = threadIdx.x / kCols, groups = blockDim.x / kCols;
  const int jl = (J + JS - 1) / JS, jb = JS > 1 ? min(wp * jl, J) : 0, je = min(jb + jl, J);
  float2 x[kJ];
  auto load = [&](int64_t base, int j0) {
#pragma unroll
    for (int u = 0; u < kJ; u++) {
      const int64_t e = base + (int64_t)min(j0 + u, J - 1) * inner;
      if (IN_REAL)
        x[u] = make_float2(__ldg(reinterpret_cast<const float *>(xv) + e), 0.f);
      else
        x[u] = __ldg(reinterpret_cast<const float2 *>(xv) + e);
    }
  };
  bool first = true;
  for (unsigned c0 = blockIdx.x * kCols; c0 < ncol; c0 += gridDim.x * kCols) {
    const unsigned col = c0 + lane;
    const bool in = col < ncol;
    const unsigned o = (in ? col : 0) / inner, r = (in ? col : 0) - o * inner;
    const int64_t base = (int64_t)o * J * inner + r;
    bool have = true;
    load(base, jb);
    if (first) {
      first = false;
      for (int t0 = threadIdx.x; t0 < J * K; t0 += 4 * blockDim.x) {
        float2 v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = __ldg(A + min(t0 + u * (int)blockDim.x, J * K - 1));
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int t = t0 + u * blockDim.x, k = t / J;
          if (t < J * K) sA[(t - k * J) * Kp + k] = v[u];
        }
      }
      if (Kp > K)
        for (int j = threadIdx.x; j < J; j += blockDim.x)
          for (int k = K; k < Kp; k++) sA[j * Kp + k] = make_float2(0.f, 0.f);
      __syncthreads();
    }
    auto put = [&](int64_t oi, float2 v) {
      if (OUT_REAL) {
        float *y = reinterpret_cast<float *>(yv);
        y[oi] = accumulate ? y[oi] + v.x : v.x;
      } else {
        float2 *y = reinterpret_cast<float2 *>(yv);
        if (accumulate) {
          const float2 p = y[oi];
          v = make_float2(p.x + v.x, p.y + v.y);
        }
        y[oi] = v;
      }
    };
    const int64_t ob = (int64_t)o * K * inner + r;
    for (int k0 = JS > 1 ? 0 : wp * KT; k0 < Kp; k0 += groups * KT) {
      float2 acc[KT];
#pragma unroll
      for (int q = 0; q < KT; q++) acc[q] = make_float2(0.f, 0.f);
      for (int j0 = jb; j0 < je; j0 += kJ) {
        if (!have) load(base, j0);
        have = false;
#pragma unroll
        for (int u = 0; u < kJ; u++) {
          if (j0 + u >= je) break;
          const float2 *a = sA + (j0 + u) * Kp + k0;
          const float2 xx = make_float2(x[u].x, x[u].x), xy = make_float2(-x[u].y, x[u].y);
#pragma unroll
          for (int q = 0; q < KT; q += 2) {
            const float4 w = *reinterpret_cast<const float4 *>(a + q);
            acc[q] = fma2(make_float2(w.x, w.y), xx, acc[q]);
            acc[q + 1] = fma2(make_float2(w.z, w.w), xx, acc[q + 1]);
            if (!IN_REAL) {
              acc[q] = fma2(make_float2(w.y, w.x), xy, acc[q]);
              acc[q + 1] = fma2(make_float2(w.w, w.z), xy, acc[q + 1]);
            }
          }
        }
      }
      if (JS > 1) {
        float2 *red = sA + J * Kp;
#pragma unroll
        for (int q = 0; q < KT; q++) red[(wp * KT + q) * kCols + lane] = acc[q];
        __syncthreads();
        for (int k = wp; k < K; k += JS) {  // lanes keep their column
          float2 v = red[k * kCols + lane];
#pragma unroll
          for (int t = 1; t < JS; t++) {
            const float2 p = red[(t * KT + k) * kCols + lane];
            v = make_float2(v.x + p.x, v.y + p.y);
          }
          if (in) put(ob + (int64_t)k * inner, v);
        }
        __syncthreads();
        break;
      }
      if (!in) continue;
#pragma unroll
      for (int q = 0; q < KT; q++)
        if (k0 + q < K) put(ob + (int64_t)(k0 + q) * inner, acc[q]);
    }
  }
}

// Along the contiguous axis (inner = 1), real <-> complex: a real GEMM
// C[row][n] (+)= sum_k X[row][k] B[k][n] over the rows of the activations.
//  - real in, complex out (Fx and the adjoint GxH): X = x [outer][J],
//    B[j][2k + c] = (Re, Im) of entry (k, j);
//  - complex in, real out (Gx and FxH): X = x [outer][J] complex as 2J floats,
//    B[2j + c][k] = (Re, -Im) of entry (k, j).
// 64 k-steps and 24 columns are too little work per row to pay for splitting
// FP32 into three BF16 pieces on the tensor cores (the conversions and their
// 16-bit stores were most of the time): in FP32 the products are 5 us of FMA
// at 64^3, width 32, against 7 us of bytes.  A CTA stages kXRows rows; a thread
// takes two rows and NO columns, its B entries one broadcast read per four
// (16 FMA of two rows), its rows 16 bytes at a time (pitch + 4: conflict-free).
// One sample: x forward 28.8 -> 17.6 us, inverse 25.6 -> 17.9 us.
constexpr int kXRows = 128;
// (mk, mn: ceil(2^32 / (kreal / 4)) and the same of nreal, for the row of an
// element index below 2^16 as a high product)
// U: loads per thread and round, 4 where they cover the rows (the clamped rest of 16
// would only take registers: inverse 42 -> 35 us, batch 2)
template <int NO, int U>
__global__ void __launch_bounds__(256) k_contract_x(const float *__restrict__ x, float *__restrict__ y,
                                                    const float2 *__restrict__ Am, int rows, int J, int K,
                                                    int in_real, int acc, unsigned mk, unsigned mn) {
  constexpr int UB = U > 4 ? 8 : 4;
  extern __shared__ __align__(16) float sm[];
  const int kreal = in_real ? J : 2 * J, nreal = in_real ? 2 * K : K;  // multiples of 4 and of NO
  const int pitch = kreal + 4;
  float *B = sm, *X = sm + kreal * nreal;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int r0 = blockIdx.x * kXRows, nr = min(kXRows, rows - r0);
  const int k4 = kreal / 4, n4 = nreal / 4;
  // the rows and B in flight together: U + UB loads per thread and round
  const float4 *src = reinterpret_cast<const float4 *>(x + (int64_t)r0 * kreal);
  for (int e0 = tid; e0 == tid || e0 < nr * k4; e0 += U * nt) {  // every thread stages its part of B
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; u++) v[u] = __ldg(src + min(e0 + u * nt, nr * k4 - 1));
    if (e0 == tid) {
      for (int t0 = tid; t0 < J * K; t0 += UB * nt) {
        float2 a[UB];
#pragma unroll
        for (int u = 0; u < UB; u++) a[u] = __ldg(Am + min(t0 + u * nt, J * K - 1));
#pragma unroll
        for (int u = 0; u < UB; u++) {
          const int t = t0 + u * nt, k = t / J, j = t - k * J;  // entry (k, j)
          if (t >= J * K) break;
          if (in_real) {
            *reinterpret_cast<float2 *>(B + j * nreal + 2 * k) = a[u];
          } else {
            B[2 * j * nreal + k] = a[u].x;
            B[(2 * j + 1) * nreal + k] = -a[u].y;
          }
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int e = e0 + u * nt;
      if (e < nr * k4) {
        const int r = __umulhi(e, mk);
        *reinterpret_cast<float4 *>(X + r * pitch + 4 * (e - r * k4)) = v[u];
      }
    }
  }
  __syncthreads();
  const int rp = tid % (kXRows / 2), n0 = tid / (kXRows / 2) * NO;  // warps share n0
  float2 c[2][NO / 2];
#pragma unroll
  for (int q = 0; q < NO / 2; q++) c[0][q] = c[1][q] = make_float2(0.f, 0.f);
  const float *xa = X + rp * pitch, *xb = X + (rp + kXRows / 2) * pitch;
  for (int k = 0; k < kreal; k += 4) {
    const float4 a4 = *reinterpret_cast<const float4 *>(xa + k), b4 = *reinterpret_cast<const float4 *>(xb + k);
    const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const float *bk = B + (k + u) * nreal + n0;
      const float2 aa = make_float2(av[u], av[u]), bb = make_float2(bv[u], bv[u]);
#pragma unroll
      for (int q = 0; q < NO / 2; q += 2) {
        const float4 w = *reinterpret_cast<const float4 *>(bk + 2 * q);
        c[0][q] = fma2(make_float2(w.x, w.y), aa, c[0][q]);
        c[1][q] = fma2(make_float2(w.x, w.y), bb, c[1][q]);
        c[0][q + 1] = fma2(make_float2(w.z, w.w), aa, c[0][q + 1]);
        c[1][q + 1] = fma2(make_float2(w.z, w.w), bb, c[1][q + 1]);
      }
    }
  }
  // through shared memory, so that the stores are whole rows in order
  __syncthreads();
  const int op = nreal + 4;
#pragma unroll
  for (int q = 0; q < NO / 2; q += 2) {
    *reinterpret_cast<float4 *>(X + rp * op + n0 + 2 * q) = make_float4(c[0][q].x, c[0][q].y, c[0][q + 1].x, c[0][q + 1].y);
    *reinterpret_cast<float4 *>(X + (rp + kXRows / 2) * op + n0 + 2 * q) =
        make_float4(c[1][q].x, c[1][q].y, c[1][q + 1].x, c[1][q + 1].y);
  }
  __syncthreads();
  float4 *dst = reinterpret_cast<float4 *>(y + (int64_t)r0 * nreal);
  for (int e0 = tid; e0 < nr * n4; e0 += 8 * nt) {
    float4 p[8];
    if (acc) {
#pragma unroll
      for (int u = 0; u < 8; u++) p[u] = dst[min(e0 + u * nt, nr * n4 - 1)];
    }
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int e = e0 + u * nt;
      if (e >= nr * n4) break;
      const int r = __umulhi(e, mn);
      float4 v = *reinterpret_cast<const float4 *>(X + r * op + 4 * (e - r * n4));
      if (acc) v = make_float4(v.x + p[u].x, v.y + p[u].y, v.z + p[u].z, v.w + p[u].w);
      dst[e] = v;
    }
  }
}

// ---------------------------------------------------------------------------
// spectral channel mixing
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 load_bf2(const uint16_t *R, int64_t e) {
  const uint32_t u = reinterpret_cast<const uint32_t *>(R)[e];
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}

// A CTA takes 32 outputs; its eight warps take every eighth channel and add
// their sums, in order, through shared memory: bound by load latency (R is 7 MB
// at width 32 and 12^3 modes), a thread then has two rounds of few loads where
// one thread per output had 32.  BWD: gx = sum_o gy conj(R), else y = sum_i x R.
// I: 32-bit indices where they suffice.  64^3, width 32, 12^3 modes: forward 15.4
// -> 7.8 us.
template <typename I, bool BWD>
__global__ void __launch_bounds__(kThreads) k_mix(const float2 *x, const uint16_t *__restrict__ R, float2 *y, I total,
                                                  int ci, int co, I M) {
  constexpr int S = kThreads / 32, U = 4;
  __shared__ float2 red[S][32];
  const int lane = threadIdx.x % 32, wp = threadIdx.x / 32;
  const int nsum = BWD ? co : ci, nout = BWD ? ci : co;
  for (I i0 = blockIdx.x * (I)32; i0 < total; i0 += gridDim.x * (I)32) {
    const I idx = i0 + lane, ic = idx < total ? idx : total - 1;
    const I q = ic / M, m = ic - q * M, b = q / nout, o = q - b * nout;
    const float2 *xb = x + (size_t)b * nsum * M + m;
    const size_t w0 = (BWD ? (size_t)o * co : (size_t)o) * M + m, ws = BWD ? M : (size_t)co * M;
    float re = 0.f, im = 0.f;
    for (int c0 = wp; c0 < nsum; c0 += S * U) {
      float2 v[U], w[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int c = min(c0 + S * u, nsum - 1);
        v[u] = xb[(size_t)c * M];
        w[u] = load_bf2(R, w0 + c * ws);
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (c0 + S * u >= nsum) break;
        if (BWD) {  // g * conj(w)
          re += v[u].x * w[u].x + v[u].y * w[u].y;
          im += v[u].y * w[u].x - v[u].x * w[u].y;
        } else {
          re += v[u].x * w[u].x - v[u].y * w[u].y;
          im += v[u].x * w[u].y + v[u].y * w[u].x;
        }
      }
    }
    red[wp][lane] = make_float2(re, im);
    __syncthreads();
    if (wp == 0) {
      float2 v = red[0][lane];
#pragma unroll
      for (int t = 1; t < S; t++) v = make_float2(v.x + red[t][lane].x, v.y + red[t][lane].y);
      if (idx < total) y[idx] = v;
    }
    __syncthreads();
  }
}

template <typename I>
__global__ void __launch_bounds__(kThreads) k_mix_gR(const float2 *__restrict__ gy, const float2 *__restrict__ x,
                                                     float2 *__restrict__ gR, int B, I total, int ci, int co, I M) {
  for (I idx = blockIdx.x * (I)blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * (I)blockDim.x) {
    const I q = idx / M, m = idx - q * M, i = q / co, o = q - i * co;
    float re = 0.f, im = 0.f;
    for (int b = 0; b < B; b++) {
      const float2 v = x[((size_t)b * ci + i) * M + m];
      const float2 g = gy[((size_t)b * co + o) * M + m];
      // conj(v) * g
      re += v.x * g.x + v.y * g.y;
      im += v.x * g.y - v.y * g.x;
    }
    gR[idx] = make_float2(re, im);
  }
}

// ---------------------------------------------------------------------------
// pointwise layers
// ---------------------------------------------------------------------------
constexpr int kMaxCh = 64;

template <int CI>
__global__ void k_pointwise(const float *__restrict__ x, const uint16_t *__restrict__ W,
                            const float *__restrict__ bias, const float *__restrict__ add, float *__restrict__ pre,
                            float *__restrict__ y, int B, int co, int64_t P, int act) {
  __shared__ float sW[kMaxCh * kMaxCh];
  __shared__ float sb[kMaxCh];
  for (int t = threadIdx.x; t < co * CI; t += blockDim.x) sW[t] = bf(W[t]);
  for (int t = threadIdx.x; t < co; t += blockDim.x) sb[t] = bias ? bias[t] : 0.f;
  __syncthreads();
  const int64_t total = (int64_t)B * P;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = idx / P, p = idx - b * P;
    float xv[CI];
#pragma unroll
    for (int i = 0; i < CI; i++) xv[i] = x[(b * CI + i) * P + p];
    for (int o = 0; o < co; o++) {
      float s = sb[o];
#pragma unroll
      for (int i = 0; i < CI; i++) s += sW[o * CI + i] * xv[i];
      const int64_t oi = (b * co + o) * P + p;
      if (add) s += add[oi];
      if (pre) pre[oi] = s;
      y[oi] = act ? gelu(s) : s;
    }
  }
}

// ---------------------------------------------------------------------------
// pointwise layers of 16 or 32 channels: y = W x (+ bias, + add, act), or the
// input gradient y = W^T g with g = gy act'(pre) formed on load and written back.
// A CTA stages 64 point pairs of every input channel in shared memory; a thread
// then takes one pair and 16 outputs, its weight row four broadcast 16-byte
// reads, the products packed FP32 pairs of outputs.  Everything a thread reads
// from memory (its share of the tile, pre, add) is one round of loads, since the
// kernel is bound by their latency: 1024 products per point are 7 us of FMA at
// 64^3 against 20 us of bytes, less than the three-piece BF16 conversion that the
// tensor cores needed for FP32 accuracy.  Layer 37 -> 33 us (one sample),
// gradient with act' 47 + 46 -> 64 us (batch 2).
// ---------------------------------------------------------------------------
constexpr int kPwPairs = 64;
template <int KC, int MC, bool TRANS, bool ACTB>
__global__ void __launch_bounds__(kPwPairs *MC / 16) k_pointwise_ch(float *x, const uint16_t *__restrict__ W,
                                                                    const float *__restrict__ bias,
                                                                    const float *__restrict__ add, float *pre,
                                                                    float *__restrict__ y, int64_t P, unsigned npair,
                                                                    int act) {
  constexpr int G = MC / 16, NT = kPwPairs * G, U = KC / G;  // thread groups; channels a thread stages
  __shared__ __align__(16) float sW[KC][MC];
  __shared__ __align__(16) float2 sx[KC][kPwPairs];
  const int pl = threadIdx.x % kPwPairs, grp = threadIdx.x / kPwPairs;
  const unsigned half = (unsigned)(P / 2), idx = blockIdx.x * kPwPairs + pl, ic = idx < npair ? idx : npair - 1;
  const unsigned b = ic / half, p = 2 * (ic - b * half);
  float2 v[U], hv[ACTB ? U : 1], d[16];
  float *xb = x + (int64_t)b * KC * P + p;
#pragma unroll
  for (int u = 0; u < U; u++) v[u] = *reinterpret_cast<const float2 *>(xb + (int64_t)(grp + G * u) * P);
  if (ACTB) {
    const float *pb = pre + (int64_t)b * KC * P + p;
#pragma unroll
    for (int u = 0; u < U; u++) hv[u] = *reinterpret_cast<const float2 *>(pb + (int64_t)(grp + G * u) * P);
  }
  const int64_t ob = ((int64_t)b * MC + 16 * grp) * P + p;  // this thread's outputs 16 grp ..
  if (add) {
#pragma unroll
    for (int u = 0; u < 16; u++) d[u] = *reinterpret_cast<const float2 *>(add + ob + (int64_t)u * P);
  }
  {
    constexpr int NW = KC * MC / NT;
    uint16_t w[NW];
#pragma unroll
    for (int u = 0; u < NW; u++) w[u] = __ldg(W + threadIdx.x + u * NT);
#pragma unroll
    for (int u = 0; u < NW; u++) {
      const int t = threadIdx.x + u * NT;
      if (TRANS)
        sW[t / MC][t % MC] = bf(w[u]);  // W is [KC][MC]
      else
        sW[t % KC][t / KC] = bf(w[u]);  // W is [MC][KC]
    }
  }
#pragma unroll
  for (int u = 0; u < U; u++) {
    if (ACTB) {
      v[u] = make_float2(v[u].x * gelu_grad(hv[u].x), v[u].y * gelu_grad(hv[u].y));
      if (idx < npair) *reinterpret_cast<float2 *>(xb + (int64_t)(grp + G * u) * P) = v[u];
    }
    sx[grp + G * u][pl] = v[u];
  }
  __syncthreads();
  float2 c0[8], c1[8];  // outputs (2q, 2q + 1) of the two points
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const int o = 16 * grp + 2 * q;
    c0[q] = c1[q] = bias ? make_float2(__ldg(bias + o), __ldg(bias + o + 1)) : make_float2(0.f, 0.f);
  }
#pragma unroll 8
  for (int k = 0; k < KC; k++) {
    const float2 xv = sx[k][pl];
    const float2 a0 = make_float2(xv.x, xv.x), a1 = make_float2(xv.y, xv.y);
#pragma unroll
    for (int q = 0; q < 8; q += 2) {
      const float4 w = *reinterpret_cast<const float4 *>(&sW[k][16 * grp + 2 * q]);
      c0[q] = fma2(make_float2(w.x, w.y), a0, c0[q]);
      c1[q] = fma2(make_float2(w.x, w.y), a1, c1[q]);
      c0[q + 1] = fma2(make_float2(w.z, w.w), a0, c0[q + 1]);
      c1[q + 1] = fma2(make_float2(w.z, w.w), a1, c1[q + 1]);
    }
  }
  if (idx >= npair) return;
#pragma unroll
  for (int u = 0; u < 16; u++) {
    float2 r = (u & 1) ? make_float2(c0[u / 2].y, c1[u / 2].y) : make_float2(c0[u / 2].x, c1[u / 2].x);
    if (add) r = make_float2(r.x + d[u].x, r.y + d[u].y);
    const int64_t oi = ob + (int64_t)u * P;
    if (!ACTB && pre) *reinterpret_cast<float2 *>(pre + oi) = r;
    *reinterpret_cast<float2 *>(y + oi) = act ? make_float2(gelu(r.x), gelu(r.y)) : r;
  }
}

// Weight and bias gradients gW = g x^T summed over the points, CI and CO of 16
// or 32.  A CTA stages 64 points of both, [channel][point]; a thread keeps the
// outer products of CO / 8 rows o = ot + 8 q and CI / 8 columns i = it + 8 q and
// reads them four points at a time (row pitch 68 floats: the eight rows of a
// read lie in distinct banks): 8 reads of 16 bytes for 64 FMA.  The four point
// groups of a CTA are added in order at the end.  Each CTA sums a fixed chunk of
// whole tiles and writes its partials in k_pointwise_wgrad's layout (pair o *
// (CI + 1) + i, the bias at i = CI), which k_wgrad_finish completes.  batch 2:
// 85 -> 59 us (three-piece BF16 products on the tensor cores before).
constexpr int kWgPts = 64;
template <int CI, int CO>
__global__ void __launch_bounds__(256) k_wgrad_ch(const float *__restrict__ g, const float *__restrict__ x,
                                                  float *__restrict__ part, int64_t P, int ntiles) {
  constexpr int PT = kWgPts + 4, QO = CO / 8, QI = CI / 8;
  __shared__ __align__(16) float sg[CO][PT];
  __shared__ __align__(16) float sx[CI][PT];
  __shared__ float sb[CO][17];
  const int tid = threadIdx.x, grp = tid / 64, ot = tid % 64 / 8, it = tid % 8;
  float acc[QO][QI];
#pragma unroll
  for (int q = 0; q < QO; q++)
#pragma unroll
    for (int r = 0; r < QI; r++) acc[q][r] = 0.f;
  // staging: 16 threads per channel, 4 points each, channels c0 + 16 i
  const int c0 = tid / 16, p4 = tid % 16 * 4;
  constexpr int GO = CO / 16, GI = CI / 16;
  float bp[GO];
#pragma unroll
  for (int i = 0; i < GO; i++) bp[i] = 0.f;
  const int per = (ntiles + gridDim.x - 1) / gridDim.x;
  const int t0 = blockIdx.x * per, t1 = min(t0 + per, ntiles);
  const int tiles_per_b = (int)(P / kWgPts);
  float4 gv[GO], xv[GI];
  auto load = [&](int tile) {
    const int b = tile / tiles_per_b;
    const int64_t p = (int64_t)(tile - b * tiles_per_b) * kWgPts + p4;
#pragma unroll
    for (int i = 0; i < GO; i++)
      gv[i] = *reinterpret_cast<const float4 *>(g + ((int64_t)b * CO + c0 + 16 * i) * P + p);
#pragma unroll
    for (int i = 0; i < GI; i++)
      xv[i] = *reinterpret_cast<const float4 *>(x + ((int64_t)b * CI + c0 + 16 * i) * P + p);
  };
  if (t0 < t1) load(t0);
  for (int tile = t0; tile < t1; tile++) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < GO; i++) {
      *reinterpret_cast<float4 *>(&sg[c0 + 16 * i][p4]) = gv[i];
      bp[i] += (gv[i].x + gv[i].y) + (gv[i].z + gv[i].w);
    }
#pragma unroll
    for (int i = 0; i < GI; i++) *reinterpret_cast<float4 *>(&sx[c0 + 16 * i][p4]) = xv[i];
    __syncthreads();
    if (tile + 1 < t1) load(tile + 1);  // in flight during the products
#pragma unroll
    for (int p = 0; p < kWgPts / 4; p += 4) {
      const int pp = grp * (kWgPts / 4) + p;
      float4 a[QO], w[QI];
#pragma unroll
      for (int q = 0; q < QO; q++) a[q] = *reinterpret_cast<const float4 *>(&sg[ot + 8 * q][pp]);
#pragma unroll
      for (int r = 0; r < QI; r++) w[r] = *reinterpret_cast<const float4 *>(&sx[it + 8 * r][pp]);
#pragma unroll
      for (int q = 0; q < QO; q++)
#pragma unroll
        for (int r = 0; r < QI; r++)
          acc[q][r] = fmaf(a[q].w, w[r].w, fmaf(a[q].z, w[r].z, fmaf(a[q].y, w[r].y, fmaf(a[q].x, w[r].x, acc[q][r]))));
    }
  }
  // the four point groups, in order, through shared memory
  constexpr int npair = CO * (CI + 1);
  float *out = part + (int64_t)blockIdx.x * npair;
  float *red = &sg[0][0];  // CO * CI floats fit
  for (int s = 1; s < 4; s++) {
    __syncthreads();
    if (grp == s)
#pragma unroll
      for (int q = 0; q < QO; q++)
#pragma unroll
        for (int r = 0; r < QI; r++) red[(ot + 8 * q) * CI + it + 8 * r] = acc[q][r];
    __syncthreads();
    if (grp == 0)
#pragma unroll
      for (int q = 0; q < QO; q++)
#pragma unroll
        for (int r = 0; r < QI; r++) acc[q][r] += red[(ot + 8 * q) * CI + it + 8 * r];
  }
  if (grp == 0)
#pragma unroll
    for (int q = 0; q < QO; q++)
#pragma unroll
      for (int r = 0; r < QI; r++) out[(ot + 8 * q) * (CI + 1) + it + 8 * r] = acc[q][r];
#pragma unroll
  for (int i = 0; i < GO; i++) sb[c0 + 16 * i][tid % 16] = bp[i];
  __syncthreads();
  if (tid < CO) {
    float s = 0.f;
    for (int q = 0; q < 16; q++) s += sb[tid][q];
    out[tid * (CI + 1) + CI] = s;
  }
}

static int launched();

static bool aligned(const void *p, size_t n) { return ((uintptr_t)p & (n - 1)) == 0; }

// the two-points-per-thread form applies: 16 or 32 channels, an even number of
// points per sample and 8-byte aligned arrays (null: absent)
static bool pointwise_ch_ok(int kc, int mc, int batch, int64_t P, const void *a, const void *b, const void *c,
                            const void *d) {
  return (kc == 16 || kc == 32) && (mc == 16 || mc == 32) && P % 2 == 0 && fits32(batch * (P / 2)) &&
         aligned(a, 8) && aligned(b, 8) && aligned(c, 8) && aligned(d, 8);
}

template <bool TRANS, bool ACTB>
static int launch_pointwise_ch(float *x, const uint16_t *W, const float *bias, const float *add, float *pre, float *y,
                               int batch, int kc, int mc, int64_t P, int act, cudaStream_t s) {
  const unsigned npair = (unsigned)(batch * (P / 2));
  const unsigned grid = (npair + kPwPairs - 1) / kPwPairs;
  auto run = [&](auto kern) {
    kern<<<grid, kPwPairs * (mc / 16), 0, s>>>(x, W, bias, add, pre, y, P, npair, act);
    return launched();
  };
  if (kc == 16) return mc == 16 ? run(k_pointwise_ch<16, 16, TRANS, ACTB>) : run(k_pointwise_ch<16, 32, TRANS, ACTB>);
  return mc == 16 ? run(k_pointwise_ch<32, 16, TRANS, ACTB>) : run(k_pointwise_ch<32, 32, TRANS, ACTB>);
}

__global__ void k_act_bwd(float *__restrict__ g, const float *__restrict__ pre, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    g[i] *= gelu_grad(pre[i]);
}

template <int CO>
__global__ void k_pointwise_gx(const float *__restrict__ g, const uint16_t *__restrict__ W, float *__restrict__ gx,
                               int B, int ci, int64_t P) {
  __shared__ float sW[kMaxCh * kMaxCh];
  for (int t = threadIdx.x; t < CO * ci; t += blockDim.x) sW[t] = bf(W[t]);
  __syncthreads();
  const int64_t total = (int64_t)B * P;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = idx / P, p = idx - b * P;
    float gv[CO];
#pragma unroll
    for (int o = 0; o < CO; o++) gv[o] = g[(b * CO + o) * P + p];
    for (int i = 0; i < ci; i++) {
      float s = 0.f;
#pragma unroll
      for (int o = 0; o < CO; o++) s += sW[o * ci + i] * gv[o];
      gx[(b * ci + i) * P + p] = s;
    }
  }
}

// weight and bias gradients: block partials over fixed point ranges, then a
// fixed-order sum over the blocks
constexpr int kWgBlocks = 296;  // two CTAs per SM
constexpr int kWgTile = 64;

// Any channel counts up to 64.  Pairs (o, i) over the threads; with few pairs
// several thread groups share a tile's points (added in order at the end), four
// points per 16-byte read.  Lifting (3 -> 32) and projection (32 -> 2), batch 2:
// 103 -> 48 us each.
__global__ void __launch_bounds__(kThreads) k_pointwise_wgrad(const float *__restrict__ g, const float *__restrict__ x,
                                                              float *__restrict__ part, int B, int ci, int co,
                                                              int64_t P) {
  constexpr int PT = kWgTile + 4;
  extern __shared__ __align__(16) float sw[];  // [ci][PT], [co][PT]; the group sums at the end
  float *sx = sw, *sg = sw + ci * PT;
  const int npair = co * (ci + 1);
  const int groups = npair < kThreads ? kThreads / npair : 1;
  const int64_t total = (int64_t)B * P;
  const int64_t chunk = (total + gridDim.x - 1) / gridDim.x;
  const int64_t t0 = blockIdx.x * chunk, t1 = (t0 + chunk < total) ? t0 + chunk : total;
  // a thread owns pairs pr, pr + blockDim.x, ... (one when there are groups)
  constexpr int kMaxPairs = (kMaxCh * (kMaxCh + 1) + kThreads - 1) / kThreads;
  const int grp = groups > 1 ? threadIdx.x / npair : 0, pr0 = threadIdx.x - grp * (groups > 1 ? npair : 0);
  float acc[kMaxPairs];
#pragma unroll
  for (int q = 0; q < kMaxPairs; q++) acc[q] = 0.f;
  // a thread stages one point of every fourth channel; the next tile's first kPre
  // channels load while this one's products run
  constexpr int kPre = 10, kStep = kThreads / kWgTile;
  const int u0 = threadIdx.x % kWgTile, cf = threadIdx.x / kWgTile, nch = ci + co;
  float pre[kPre];
  auto at = [&](int64_t tt, int c) -> float {  // (a point past the chunk: the tile's first, unused)
    const int64_t t = tt + u0 < t1 ? tt + u0 : tt, b = t / P, p = t - b * P;
    return c < ci ? x[(b * ci + c) * P + p] : g[(b * co + (c - ci)) * P + p];
  };
  auto fetch = [&](int64_t tt) {
#pragma unroll
    for (int q = 0; q < kPre; q++) pre[q] = at(tt, min(cf + q * kStep, nch - 1));
  };
  if (t0 < t1) fetch(t0);
  for (int64_t tt = t0; tt < t1; tt += kWgTile) {
    const bool have = tt + u0 < t1;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kPre; q++)
      if (cf + q * kStep < nch) sw[(cf + q * kStep) * PT + u0] = have ? pre[q] : 0.f;
    for (int c0 = cf + kPre * kStep; c0 < nch; c0 += 8 * kStep) {
      float v[8];
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] = at(tt, min(c0 + q * kStep, nch - 1));
#pragma unroll
      for (int q = 0; q < 8; q++)
        if (c0 + q * kStep < nch) sw[(c0 + q * kStep) * PT + u0] = have ? v[q] : 0.f;
    }
    if (tt + kWgTile < t1) fetch(tt + kWgTile);
    __syncthreads();
    if (grp < groups) {
#pragma unroll
      for (int q = 0; q < kMaxPairs; q++) {
        const int pr = pr0 + q * kThreads;
        if (pr >= npair) break;
        const int o = pr / (ci + 1), i = pr - o * (ci + 1);
        float s = 0.f;
        for (int u = 4 * grp; u < kWgTile; u += 4 * groups) {
          const float4 a = *reinterpret_cast<const float4 *>(sg + o * PT + u);
          const float4 w =
              i < ci ? *reinterpret_cast<const float4 *>(sx + i * PT + u) : make_float4(1.f, 1.f, 1.f, 1.f);
          s = fmaf(a.w, w.w, fmaf(a.z, w.z, fmaf(a.y, w.y, fmaf(a.x, w.x, s))));
        }
        acc[q] += s;
      }
    }
  }
  if (groups > 1) {
    __syncthreads();
    if (grp < groups) sw[threadIdx.x] = acc[0];
    __syncthreads();
    if (grp == 0)
      for (int s = 1; s < groups; s++) acc[0] += sw[s * npair + pr0];
    if (grp != 0) return;
  }
#pragma unroll
  for (int q = 0; q < kMaxPairs; q++) {
    const int pr = pr0 + q * kThreads;
    if (pr < npair) part[(int64_t)blockIdx.x * npair + pr] = acc[q];
  }
}

// one warp per (output, input or bias) pair: lane l sums the partials of
// blocks l, l + 32, ... in FP64, then a fixed shuffle tree adds the lanes,
// so the order (and the result) is the same on every run
__global__ void k_wgrad_finish(const float *__restrict__ part, float *__restrict__ gW, float *__restrict__ gb,
                               int nblk, int ci, int co) {
  const int npair = co * (ci + 1);
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (int pr = blockIdx.x * wpb + (threadIdx.x >> 5); pr < npair; pr += gridDim.x * wpb) {
    double s = 0.0;
    for (int b = lane; b < nblk; b += 32) s += (double)part[(int64_t)b * npair + pr];
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if (lane != 0) continue;
    const int o = pr / (ci + 1), i = pr % (ci + 1);
    if (i < ci) {
      if (gW) gW[o * ci + i] = (float)s;
    } else if (gb) {
      gb[o] = (float)s;
    }
  }
}

// ---------------------------------------------------------------------------
// loss, optimizer
// ---------------------------------------------------------------------------
constexpr int kLossBlocks = 296;

__global__ void k_loss_part(const float *__restrict__ pred, const float *__restrict__ tgt, double *part, int64_t n) {
  __shared__ double sh[32];
  double e = 0.0, t2 = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double d = (double)pred[i] - (double)tgt[i];
    e += d * d;
    t2 += (double)tgt[i] * tgt[i];
  }
  e = block_sum(e, sh);
  t2 = block_sum(t2, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = e;
    part[gridDim.x + blockIdx.x] = t2;
  }
}

// one warp: lane sums in index order, then a fixed shuffle tree (one thread
// over the 296 partials took 15 us)
__device__ __forceinline__ void warp_sum2(const double *part, int nb, double &a, double &b) {
  a = b = 0.0;
  for (int i = threadIdx.x; i < nb; i += 32) {
    a += part[i];
    b += part[nb + i];
  }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, d);
    b += __shfl_xor_sync(0xffffffffu, b, d);
  }
}

__global__ void k_loss_finish(const double *part, int nb, double *out) {
  double e, t2;
  warp_sum2(part, nb, e, t2);
  if (threadIdx.x == 0) {
    out[0] = e / (t2 > 0 ? t2 : 1.0);
    out[1] = t2;
  }
}

__global__ void k_loss_grad(const float *__restrict__ pred, const float *__restrict__ tgt, float *grad,
                            const double *out, int64_t n) {
  const double t2 = out[1] > 0 ? out[1] : 1.0;
  const float c = (float)(2.0 / t2);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    grad[i] = c * (pred[i] - tgt[i]);
}

__device__ __forceinline__ uint16_t to_bf16(float f) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(f));
}

struct AdamC {
  float lr, b1, b2, eps, c1, c2;
};
__device__ __forceinline__ void adam1(float &p, float g, float &m, float &v, const AdamC &a) {
  m = a.b1 * m + (1.f - a.b1) * g;
  v = a.b2 * v + (1.f - a.b2) * g * g;
  p = p - a.lr * (m / a.c1) / (sqrtf(v / a.c2) + a.eps);
}

// V4: 16-byte accesses, n4 = n / 4 groups (88 -> 64 us for the 14 M parameters
// of width 32, 12^3 modes: 425 MB); else, and for the remainder from n4 * 4 on,
// one value per thread
template <bool V4>
__global__ void __launch_bounds__(kThreads) k_adam(float *p, const float *__restrict__ g, float *m, float *v,
                                                   uint16_t *pb, int64_t n, AdamC a) {
  const int64_t n4 = V4 ? n / 4 : 0, step = (int64_t)gridDim.x * blockDim.x;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  for (int64_t i = t; i < n4; i += step) {
    float4 P = reinterpret_cast<float4 *>(p)[i], M = reinterpret_cast<float4 *>(m)[i],
           V = reinterpret_cast<float4 *>(v)[i];
    const float4 G = reinterpret_cast<const float4 *>(g)[i];
    adam1(P.x, G.x, M.x, V.x, a);
    adam1(P.y, G.y, M.y, V.y, a);
    adam1(P.z, G.z, M.z, V.z, a);
    adam1(P.w, G.w, M.w, V.w, a);
    reinterpret_cast<float4 *>(p)[i] = P;
    reinterpret_cast<float4 *>(m)[i] = M;
    reinterpret_cast<float4 *>(v)[i] = V;
    if (pb)
      reinterpret_cast<uint2 *>(pb)[i] =
          make_uint2(to_bf16(P.x) | ((uint32_t)to_bf16(P.y) << 16), to_bf16(P.z) | ((uint32_t)to_bf16(P.w) << 16));
  }
  for (int64_t i = 4 * n4 + t; i < n; i += step) {
    float P = p[i], M = m[i], V = v[i];
    adam1(P, g[i], M, V, a);
    p[i] = P;
    m[i] = M;
    v[i] = V;
    if (pb) pb[i] = to_bf16(P);
  }
}

__global__ void k_to_bf16(const float *__restrict__ x, uint16_t *y, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    y[i] = to_bf16(x[i]);
}

// ---------------------------------------------------------------------------
// grid transfer
// ---------------------------------------------------------------------------
__global__ void k_restrict(const double *__restrict__ src, float *__restrict__ dst, int nf, int f, int cplx,
                           float scale) {
  const int nc = nf / f;
  const int64_t nc3 = (int64_t)nc * nc * nc;
  const float inv = scale / (float)(f * f * f);
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < nc3; c += (int64_t)gridDim.x * blockDim.x) {
    const int cx = (int)(c % nc), cy = (int)((c / nc) % nc), cz = (int)(c / ((int64_t)nc * nc));
    double re = 0.0, im = 0.0;
    for (int dz = 0; dz < f; dz++)
      for (int dy = 0; dy < f; dy++)
        for (int dx = 0; dx < f; dx++) {
          const int64_t fi = ((int64_t)(cz * f + dz) * nf + (cy * f + dy)) * nf + (cx * f + dx);
          if (cplx) {
            re += src[2 * fi];
            im += src[2 * fi + 1];
          } else {
            re += src[fi];
          }
        }
    dst[c] = (float)re * inv;
    if (cplx) dst[nc3 + c] = (float)im * inv;
  }
}

__global__ void k_prolong_add(const float *__restrict__ src, double2 *dst, int nf, int f, float scale) {
  const int nc = nf / f;
  const int64_t nc3 = (int64_t)nc * nc * nc;
  const int64_t nf3 = (int64_t)nf * nf * nf;
  const float off = 0.5f * (float)(f - 1);
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nf3; q += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(q % nf), y = (int)((q / nf) % nf), z = (int)(q / ((int64_t)nf * nf));
    const float ux = (x - off) / f, uy = (y - off) / f, uz = (z - off) / f;
    const int x0 = (int)floorf(ux), y0 = (int)floorf(uy), z0 = (int)floorf(uz);
    const float wx = ux - x0, wy = uy - y0, wz = uz - z0;
    float re = 0.f, im = 0.f;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const int ix = ((x0 + (c & 1)) % nc + nc) % nc;
      const int iy = ((y0 + ((c >> 1) & 1)) % nc + nc) % nc;
      const int iz = ((z0 + (c >> 2)) % nc + nc) % nc;
      const float w = ((c & 1) ? wx : 1.f - wx) * (((c >> 1) & 1) ? wy : 1.f - wy) * ((c >> 2) ? wz : 1.f - wz);
      const int64_t ci = ((int64_t)iz * nc + iy) * nc + ix;
      re += w * src[ci];
      im += w * src[nc3 + ci];
    }
    double2 d = dst[q];
    d.x += (double)(scale * re);
    d.y += (double)(scale * im);
    dst[q] = d;
  }
}

__global__ void k_deposit_coarse(const double *__restrict__ r, int npar, float *dst, int nc, double xmax) {
  const double hc = 2.0 * xmax / nc;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npar; p += gridDim.x * blockDim.x) {
    const double a = (r[p] + xmax) / hc, b = (r[npar + p] + xmax) / hc, c = (r[2 * npar + p] + xmax) / hc;
    if (!(a >= 0 && a < nc && b >= 0 && b < nc && c >= 0 && c < nc)) continue;
    const int ix = (int)a, iy = (int)b, iz = (int)c;
    // counts stay below 2^24, so FP32 additions of 1 are exact and order-free
    atomicAdd(&dst[((int64_t)iz * nc + iy) * nc + ix], 1.0f);
  }
}

__global__ void k_scale(float *x, int64_t n, float s) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] *= s;
}

// parareal correction: u_new = s (g_new + fine - g_old), written over u
// (the previous iterate).  Pass 1 sums |g_new + fine - g_old|^2 and
// |fine|^2 per block; s = sqrt(sum |fine|^2 / sum |u_new|^2) when the norm
// projection is on (the fine propagator conserves the norm), else 1.  Pass 2
// writes u and sums |u_new - u|^2 and |u|^2 per block.
__global__ void k_parareal_norms(const double *__restrict__ gnew, const double *__restrict__ fine,
                                 const double *__restrict__ gold, int64_t n, double *part) {
  __shared__ double sh[32];
  double nn = 0.0, ff = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double v = (gnew[i] + fine[i]) - gold[i];
    nn += v * v;
    ff += fine[i] * fine[i];
  }
  nn = block_sum(nn, sh);
  ff = block_sum(ff, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = nn;
    part[gridDim.x + blockIdx.x] = ff;
  }
}

__global__ void k_parareal(const double *__restrict__ gnew, const double *__restrict__ fine,
                           const double *__restrict__ gold, double *u, int64_t n, const double *scale,
                           double *part) {
  __shared__ double sh[32];
  double sc = 1.0;
  if (scale) sc = (scale[0] > 0.0) ? sqrt(scale[1] / scale[0]) : 1.0;
  double dd = 0.0, uu = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double old = u[i];
    const double v = sc * ((gnew[i] + fine[i]) - gold[i]);
    u[i] = v;
    dd += (v - old) * (v - old);
    uu += old * old;
  }
  dd = block_sum(dd, sh);
  uu = block_sum(uu, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = dd;
    part[gridDim.x + blockIdx.x] = uu;
  }
}

__global__ void k_sum2(const double *part, int nb, double *out) {
  double a, b;
  warp_sum2(part, nb, a, b);
  if (threadIdx.x == 0) {
    out[0] = a;
    out[1] = b;
  }
}

static int launched() {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("FNO kernel launch: %s", cudaGetErrorString(e));
    return HE4_E_CUDA;
  }
  return HE4_OK;
}

#define FNO_CI_SWITCH(ci, KER, ...)                            \
  switch (ci) {                                                 \
    case 1: KER<1><<<__VA_ARGS__; break;                        \
    case 2: KER<2><<<__VA_ARGS__; break;                        \
    case 3: KER<3><<<__VA_ARGS__; break;                        \
    case 4: KER<4><<<__VA_ARGS__; break;                        \
    case 8: KER<8><<<__VA_ARGS__; break;                        \
    case 16: KER<16><<<__VA_ARGS__; break;                      \
    case 32: KER<32><<<__VA_ARGS__; break;                      \
    case 64: KER<64><<<__VA_ARGS__; break;                      \
    default:                                                    \
      set_error("FNO: %d channels are not supported", (int)ci); \
      return HE4_E_UNSUPPORTED;                                 \
  }

}  // namespace fno
}  // namespace he4

using namespace he4;
using namespace he4::fno;

namespace {
// Dynamic shared memory limit of the k_contract kernels, one value for every size: a
// limit of each call's own need can be lowered by another thread's call before this
// one's launch, which then fails.  J K <= 6144 entries and the dispatch below need
// 96 KB at most (J = 6144, K = 1: two entries per j).
constexpr int kContractSmem = 96 * 1024;
template <int KT, int JS>
int launch_contract(const void *x, void *y, const float2 *A, unsigned ncol, int J, int K, unsigned inner, int in_real,
                    int out_real, int accumulate, cudaStream_t s) {
  const int Kp = (K + KT - 1) / KT * KT, warps = JS > 1 ? JS : std::min(Kp / KT, 512 / kCols);
  const unsigned grid = std::min((ncol + kCols - 1) / kCols, 148u * 32);
  const size_t sm = sizeof(float2) * ((size_t)J * Kp + (JS > 1 ? (size_t)JS * KT * kCols : 0));
  auto run = [&](auto kern) {
    // J K has 6144 entries at most (48 KB); the rounded-up rows and the partial sums may need more
    if (sm > 48 * 1024 &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kContractSmem) != cudaSuccess)
      return launched();
    kern<<<grid, warps * kCols, sm, s>>>(x, y, A, ncol, J, K, inner, accumulate);
    return launched();
  };
  if (in_real) return out_real ? run(k_contract<true, true, KT, JS>) : run(k_contract<true, false, KT, JS>);
  return out_real ? run(k_contract<false, true, KT, JS>) : run(k_contract<false, false, KT, JS>);
}
template <int NO>
int launch_contract_x(const float *x, float *y, const float2 *A, int rows, int J, int K, int in_real, int acc,
                      cudaStream_t s) {
  const int kreal = in_real ? J : 2 * J, nreal = in_real ? 2 * K : K;
  const size_t sm = sizeof(float) * ((size_t)kreal * nreal + (size_t)kXRows * (std::max(kreal, nreal) + 4));
  const int threads = kXRows / 2 * (nreal / NO);
  auto magic = [](int d) { return (unsigned)(((1ull << 32) + d - 1) / d); };
  auto run = [&](auto kern) {
    if (sm > 48 * 1024 &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024) != cudaSuccess)
      return launched();
    kern<<<(rows + kXRows - 1) / kXRows, threads, sm, s>>>(x, y, A, rows, J, K, in_real, acc, magic(kreal / 4),
                                                          magic(nreal / 4));
    return launched();
  };
  return kXRows * (kreal / 4) <= 4 * threads ? run(k_contract_x<NO, 4>) : run(k_contract_x<NO, 16>);
}
}  // namespace

extern "C" {

int he4_fno_contract(const void *x, void *y, const float *A, int32_t outer, int32_t J, int32_t K, int32_t inner,
                     int32_t in_real, int32_t out_real, int32_t accumulate, void *stream) {
  if (!x || !y || !A || outer < 1 || J < 1 || K < 1 || inner < 1 || (int64_t)J * K * 8 > 48 * 1024) {
    set_error("he4_fno_contract: invalid arguments");
    return HE4_E_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  if (!fits32((int64_t)outer * inner)) {  // (outer > 1: inner alone fits) in two halves
    const int32_t half = outer / 2;
    const size_t xs = in_real ? 4 : 8, ys = out_real ? 4 : 8;
    HE4_TRY(he4_fno_contract(x, y, A, half, J, K, inner, in_real, out_real, accumulate, stream));
    return he4_fno_contract(static_cast<const char *>(x) + xs * half * J * (size_t)inner,
                            static_cast<char *>(y) + ys * half * K * (size_t)inner, A, outer - half, J, K, inner,
                            in_real, out_real, accumulate, stream);
  }
  const float2 *A2 = reinterpret_cast<const float2 *>(A);
  // along the contiguous axis, real <-> complex, rows of whole 16-byte units (two at least)
  // and output columns that 64-row-pair CTAs of at most 256 threads cover
  if (inner == 1 && in_real != out_real && aligned(x, 16) && aligned(y, 16)) {
    const int kreal = in_real ? J : 2 * J, nreal = in_real ? 2 * K : K;
    const float *xf = reinterpret_cast<const float *>(x);
    float *yf = reinterpret_cast<float *>(y);
    if (kreal % 4 == 0 && kreal >= 8 && kreal <= 64 && nreal <= 64) {
      if (nreal % 16 == 0 && nreal > 16)
        return launch_contract_x<16>(xf, yf, A2, outer, J, K, in_real, accumulate, s);
      if (nreal % 12 == 0 && nreal <= 48) return launch_contract_x<12>(xf, yf, A2, outer, J, K, in_real, accumulate, s);
      if (nreal == 20) return launch_contract_x<20>(xf, yf, A2, outer, J, K, in_real, accumulate, s);
      if (nreal % 8 == 0 && nreal <= 32)
        return launch_contract_x<8>(xf, yf, A2, outer, J, K, in_real, accumulate, s);
    }
  }
  // onto few modes from a long axis: all outputs in one thread, eight slices of
  // j; else (back to the full axis, or a short one) groups of eight outputs
  const unsigned ncol = (unsigned)outer * (unsigned)inner;
  if (J > 512 && K < 8)  // long and thin: the rounded-up A of the others may not fit
    return launch_contract<2, 1>(x, y, A2, ncol, J, K, inner, in_real, out_real, accumulate, s);
  if (K <= 16 && J >= 32) {
    if (K <= 8) return launch_contract<8, 8>(x, y, A2, ncol, J, K, inner, in_real, out_real, accumulate, s);
    if (K <= 12) return launch_contract<12, 8>(x, y, A2, ncol, J, K, inner, in_real, out_real, accumulate, s);
    return launch_contract<16, 8>(x, y, A2, ncol, J, K, inner, in_real, out_real, accumulate, s);
  }
  return launch_contract<8, 1>(x, y, A2, ncol, J, K, inner, in_real, out_real, accumulate, s);
}

int he4_fno_mix(const float *x, const uint16_t *R, float *y, int32_t batch, int32_t cin, int32_t cout,
                int32_t modes, void *stream) {
  if (!x || !R || !y || batch < 1 || cin < 1 || cout < 1 || modes < 1) {
    set_error("he4_fno_mix: invalid arguments");
    return HE4_E_ARG;
  }
  const int64_t total = (int64_t)batch * cout * modes;
  const float2 *x2 = reinterpret_cast<const float2 *>(x);
  float2 *y2 = reinterpret_cast<float2 *>(y);
  cudaStream_t s = (cudaStream_t)stream;
  if (fits32(total))
    k_mix<uint32_t, false><<<mix_blocks(total), kThreads, 0, s>>>(x2, R, y2, (uint32_t)total, cin, cout, modes);
  else
    k_mix<uint64_t, false><<<mix_blocks(total), kThreads, 0, s>>>(x2, R, y2, total, cin, cout, modes);
  return launched();
}

int he4_fno_mix_bwd(const float *gy, const float *x, const uint16_t *R, float *gx, float *gR, int32_t batch,
                    int32_t cin, int32_t cout, int32_t modes, void *stream) {
  if (!gy || !x || !R || batch < 1 || cin < 1 || cout < 1 || modes < 1) {
    set_error("he4_fno_mix_bwd: invalid arguments");
    return HE4_E_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const float2 *g2 = reinterpret_cast<const float2 *>(gy), *x2 = reinterpret_cast<const float2 *>(x);
  const int64_t nR = (int64_t)cin * cout * modes, nx = (int64_t)batch * cin * modes;
  float2 *gR2 = reinterpret_cast<float2 *>(gR), *gx2 = reinterpret_cast<float2 *>(gx);
  // gR first: gx may overwrite x
  if (gR) {
    if (fits32(nR))
      k_mix_gR<uint32_t><<<blocks_for(nR), kThreads, 0, s>>>(g2, x2, gR2, batch, (uint32_t)nR, cin, cout, modes);
    else
      k_mix_gR<uint64_t><<<blocks_for(nR), kThreads, 0, s>>>(g2, x2, gR2, batch, nR, cin, cout, modes);
    HE4_TRY(launched());
  }
  if (gx) {
    if (fits32(nx))
      k_mix<uint32_t, true><<<mix_blocks(nx), kThreads, 0, s>>>(g2, R, gx2, (uint32_t)nx, cin, cout, modes);
    else
      k_mix<uint64_t, true><<<mix_blocks(nx), kThreads, 0, s>>>(g2, R, gx2, nx, cin, cout, modes);
    HE4_TRY(launched());
  }
  return HE4_OK;
}

int he4_fno_pointwise(const float *x, const uint16_t *W, const float *bias, const float *add, float *pre, float *y,
                      int32_t batch, int32_t cin, int32_t cout, int64_t npts, int32_t act, void *stream) {
  if (!x || !W || !y || batch < 1 || cin < 1 || cout < 1 || cout > kMaxCh || npts < 1) {
    set_error("he4_fno_pointwise: invalid arguments");
    return HE4_E_ARG;
  }
  if (pointwise_ch_ok(cin, cout, batch, npts, x, add, pre, y))
    return launch_pointwise_ch<false, false>(const_cast<float *>(x), W, bias, add, pre, y, batch, cin, cout, npts, act,
                                             (cudaStream_t)stream);
  const int64_t total = (int64_t)batch * npts;
  FNO_CI_SWITCH(cin, k_pointwise, blocks_for(total), kThreads, 0, (cudaStream_t)stream >>>(x, W, bias, add, pre, y,
                                                                                         batch, cout, npts, act));
  return launched();
}

int64_t he4_fno_pointwise_work(int32_t batch, int32_t cin, int32_t cout, int64_t npts) {
  (void)batch;
  (void)npts;
  return (int64_t)kWgBlocks * cout * (cin + 1);
}

int he4_fno_pointwise_bwd(float *gy, const float *pre, const float *x, const uint16_t *W, float *gx, float *gW,
                          float *gbias, float *work, int32_t batch, int32_t cin, int32_t cout, int64_t npts,
                          int32_t act, void *stream) {
  if (!gy || !x || !W || batch < 1 || cin < 1 || cout < 1 || cin > kMaxCh || cout > kMaxCh || npts < 1 ||
      (act && !pre) || ((gW || gbias) && !work)) {
    set_error("he4_fno_pointwise_bwd: invalid arguments");
    return HE4_E_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t total = (int64_t)batch * npts;
  const bool ch = gx && pointwise_ch_ok(cout, cin, batch, npts, gy, pre, gx, nullptr);
  if (act && !ch) {
    k_act_bwd<<<blocks_for(total * cout), kThreads, 0, s>>>(gy, pre, total * cout);
    HE4_TRY(launched());
  }
  if (ch && act) {  // act' applied and gy written on the way
    HE4_TRY((launch_pointwise_ch<true, true>(gy, W, nullptr, nullptr, const_cast<float *>(pre), gx, batch, cout, cin,
                                             npts, 0, s)));
  } else if (ch) {
    HE4_TRY((launch_pointwise_ch<true, false>(gy, W, nullptr, nullptr, nullptr, gx, batch, cout, cin, npts, 0, s)));
  } else if (gx) {
    FNO_CI_SWITCH(cout, k_pointwise_gx, blocks_for(total), kThreads, 0, s >>>(gy, W, gx, batch, cin, npts));
    HE4_TRY(launched());
  }
  if (gW || gbias) {
    const int64_t ntiles = batch * (npts / kWgPts);
    const bool tiles = npts % kWgPts == 0 && ntiles < (1ll << 31) && aligned(gy, 16) && aligned(x, 16);
    if (tiles && cin == 32 && cout == 32)
      k_wgrad_ch<32, 32><<<kWgBlocks, 256, 0, s>>>(gy, x, work, npts, (int)ntiles);
    else if (tiles && cin == 16 && cout == 16)
      k_wgrad_ch<16, 16><<<kWgBlocks, 256, 0, s>>>(gy, x, work, npts, (int)ntiles);
    else
      k_pointwise_wgrad<<<kWgBlocks, kThreads,
                          sizeof(float) * std::max((cin + cout) * (kWgTile + 4), (int)kThreads), s>>>(
          gy, x, work, batch, cin, cout, npts);
    HE4_TRY(launched());
    const int wpb = kThreads / 32;  // one warp per pair
    k_wgrad_finish<<<(cout * (cin + 1) + wpb - 1) / wpb, kThreads, 0, s>>>(work, gW, gbias, kWgBlocks, cin, cout);
    HE4_TRY(launched());
  }
  return HE4_OK;
}

int he4_fno_loss(const float *pred, const float *target, float *grad, double *out, int64_t n, double *work,
                 void *stream) {
  if (!pred || !target || !out || !work || n < 1) {
    set_error("he4_fno_loss: invalid arguments");
    return HE4_E_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  k_loss_part<<<kLossBlocks, kThreads, 0, s>>>(pred, target, work, n);
  HE4_TRY(launched());
  k_loss_finish<<<1, 32, 0, s>>>(work, kLossBlocks, out);
  HE4_TRY(launched());
  if (grad) {
    k_loss_grad<<<blocks_for(n), kThreads, 0, s>>>(pred, target, grad, out, n);
    HE4_TRY(launched());
  }
  return HE4_OK;
}

int he4_fno_adam(float *p, const float *g, float *m, float *v, uint16_t *pb, int64_t n, float lr, float beta1,
                 float beta2, float eps, int32_t step, void *stream) {
  if (!p || !g || !m || !v || n < 1 || step < 1) {
    set_error("he4_fno_adam: invalid arguments");
    return HE4_E_ARG;
  }
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  const AdamC a{lr, beta1, beta2, eps, c1, c2};
  if (n >= 4 && aligned(p, 16) && aligned(g, 16) && aligned(m, 16) && aligned(v, 16) && aligned(pb, 8))
    k_adam<true><<<blocks_for(n / 4), kThreads, 0, (cudaStream_t)stream>>>(p, g, m, v, pb, n, a);
  else
    k_adam<false><<<blocks_for(n), kThreads, 0, (cudaStream_t)stream>>>(p, g, m, v, pb, n, a);
  return launched();
}

int he4_fno_to_bf16(const float *x, uint16_t *y, int64_t n, void *stream) {
  if (!x || !y || n < 1) {
    set_error("he4_fno_to_bf16: invalid arguments");
    return HE4_E_ARG;
  }
  k_to_bf16<<<blocks_for(n), kThreads, 0, (cudaStream_t)stream>>>(x, y, n);
  return launched();
}

int he4_fno_restrict(const double *src, float *dst, int32_t nf, int32_t f, int32_t complex_src, float scale,
                     void *stream) {
  if (!src || !dst || f < 1 || nf < f || nf % f != 0) {
    set_error("he4_fno_restrict: invalid arguments");
    return HE4_E_ARG;
  }
  const int64_t nc = nf / f;
  k_restrict<<<blocks_for(nc * nc * nc), kThreads, 0, (cudaStream_t)stream>>>(src, dst, nf, f, complex_src, scale);
  return launched();
}

int he4_fno_prolong_add(const float *src, double *dst, int32_t nf, int32_t f, float scale, void *stream) {
  if (!src || !dst || f < 1 || nf < f || nf % f != 0) {
    set_error("he4_fno_prolong_add: invalid arguments");
    return HE4_E_ARG;
  }
  k_prolong_add<<<blocks_for((int64_t)nf * nf * nf), kThreads, 0, (cudaStream_t)stream>>>(
      src, reinterpret_cast<double2 *>(dst), nf, f, scale);
  return launched();
}

int he4_fno_deposit(const double *r, int32_t npar, float *dst, int32_t nc, double xmax, float scale, void *stream) {
  if (!r || !dst || npar < 1 || nc < 1 || !(xmax > 0)) {
    set_error("he4_fno_deposit: invalid arguments");
    return HE4_E_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t n3 = (int64_t)nc * nc * nc;
  if (cudaMemsetAsync(dst, 0, sizeof(float) * n3, s) != cudaSuccess) {
    set_error("he4_fno_deposit: memset failed");
    return HE4_E_CUDA;
  }
  k_deposit_coarse<<<blocks_for(npar), kThreads, 0, s>>>(r, npar, dst, nc, xmax);
  HE4_TRY(launched());
  const double hc = 2.0 * xmax / nc;
  k_scale<<<blocks_for(n3), kThreads, 0, s>>>(dst, n3, (float)(scale / (npar * hc * hc * hc)));
  return launched();
}

int he4_parareal_correct(const double *gnew, const double *fine, const double *gold, double *u, int64_t n,
                         int32_t renorm, double *out, double *work, void *stream) {
  if (!gnew || !fine || !gold || !u || !out || !work || n < 1) {
    set_error("he4_parareal_correct: invalid arguments");
    return HE4_E_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  if (renorm) {
    k_parareal_norms<<<kLossBlocks, kThreads, 0, s>>>(gnew, fine, gold, n, work);
    HE4_TRY(launched());
    k_sum2<<<1, 32, 0, s>>>(work, kLossBlocks, out + 2);
    HE4_TRY(launched());
  }
  k_parareal<<<kLossBlocks, kThreads, 0, s>>>(gnew, fine, gold, u, n, renorm ? out + 2 : nullptr, work);
  HE4_TRY(launched());
  k_sum2<<<1, 32, 0, s>>>(work, kLossBlocks, out);
  return launched();
}

}  // extern "C"
