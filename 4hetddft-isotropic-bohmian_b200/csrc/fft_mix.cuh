// fft_mix.cuh -- two-step register FFT passes for axis lengths N = N1 N2
// (powers of two from 16 to 256, and 36..250 with factors 3 and 5), in FP64
// and, for powers of two, FP32.
//
// With j = j1 + N1 j2 and k = k2 + N2 k1 a pencil's forward transform is
//   thread j1: the N2-point DFT of x[j1 + N1 j2], loaded straight from global
//     memory, times w_N^(j1 k2), into shared memory at (k2, j1);
//   barrier;
//   thread t: the N1-point DFTs of its rows k2, leaving X[k2 + N2 k1].
// The inverse runs backwards from that register layout.  max(N1, N2) threads
// serve a pencil, some of them idle in one of the two steps (the factors are
// chosen nearly equal), or N1 threads with several rows each (Mix::CR).  A
// transform has one shared-memory exchange and one barrier: a thread reads in
// the inverse the column it wrote in the forward and writes the rows it read,
// so no barrier separates the two.
//
// Bound by memory latency and, in FP64, by instruction issue; small CTAs (64
// to 128 threads, one working set of registers) keep their load, transform
// and store phases overlapped on an SM.  Measured per launch (one to three
// fields), against shared-memory Stockham passes: 96^3 FP64 y pass 13.5 -> 5.9
// us, z convolution 29 -> 10, x C2R 12.7 -> 6.0; 192 x 192 x 240 y pass 105 ->
// 51, x R2C 116 -> 49; against one-tile-per-SM register passes with two
// barriers per exchange: 64^3 FP64 y pass 6.1 -> 3.4, z sum 16 -> 11; 128^3
// FP64 y 15 -> 11, z sum 55 -> 41, FP32 y 12.5 -> 6.1, z sum 31 -> 20; 256^3
// FP64 x C2R 105 -> 80, z sum 287 -> 235, FP32 z sum 151 -> 103.  PC step:
// 96^3 1.30 -> 0.60 ms, 64^3 0.44 -> 0.34, 128^3 FP64 1.28 -> 1.13 and FP32
// 0.98 -> 0.76, 256^3 FP64 7.28 -> 6.63 and FP32 4.55 -> 4.05.
//
// Shared memory: a pencil's element (k2, j1) at k2 RP + j1, RP = N1 | 1, and
// pencils PP apart, PP odd: with the pencil index varying fastest over the
// lanes (y and z passes) every access is conflict-free, and with the
// in-pencil index fastest (x passes) the odd row pitch keeps rows apart.
// Offsets inside a pencil are compile-time constants.
#pragma once
#include <algorithm>

#include "common.cuh"
#include "fft_codelets.cuh"
#include "fft_passes.cuh"
#include "reduce.cuh"

namespace he4 {

// factors of a length: N1 for the second step, N2 for the first
template <int N>
struct MixFactors;
#define HE4_MIX_F(n, a, b)                  \
  template <>                               \
  struct MixFactors<n> {                    \
    static constexpr int N1 = a, N2 = b;    \
  };
HE4_MIX_F(16, 4, 4)
HE4_MIX_F(32, 4, 8)
HE4_MIX_F(64, 8, 8)
HE4_MIX_F(128, 8, 16)
HE4_MIX_F(256, 16, 16)
HE4_MIX_F(36, 6, 6)
HE4_MIX_F(40, 5, 8)
HE4_MIX_F(45, 5, 9)
HE4_MIX_F(48, 6, 8)
HE4_MIX_F(50, 5, 10)
HE4_MIX_F(54, 6, 9)
HE4_MIX_F(60, 6, 10)
HE4_MIX_F(72, 8, 9)
HE4_MIX_F(75, 5, 15)
HE4_MIX_F(80, 8, 10)
HE4_MIX_F(81, 9, 9)
HE4_MIX_F(90, 9, 10)
HE4_MIX_F(96, 8, 12)
HE4_MIX_F(100, 10, 10)
HE4_MIX_F(108, 9, 12)
HE4_MIX_F(120, 10, 12)
HE4_MIX_F(125, 5, 25)
HE4_MIX_F(135, 9, 15)
HE4_MIX_F(144, 12, 12)
HE4_MIX_F(150, 10, 15)
HE4_MIX_F(160, 10, 16)
HE4_MIX_F(162, 9, 18)
HE4_MIX_F(180, 12, 15)
HE4_MIX_F(192, 12, 16)
HE4_MIX_F(200, 10, 20)
HE4_MIX_F(216, 12, 18)
HE4_MIX_F(225, 15, 15)
HE4_MIX_F(240, 15, 16)
HE4_MIX_F(243, 9, 27)
HE4_MIX_F(250, 10, 25)
#undef HE4_MIX_F

// F1: another first factor (the autotuner's alternatives), 0 = the default.
// ROWS: where N1 divides N2, N1 threads with N2 / N1 rows each serve a pencil.
template <int N, int F1 = 0, bool ROWS = false>
struct Mix {
  static constexpr int N1 = F1 ? F1 : MixFactors<N>::N1, N2 = N / N1;
  static constexpr int CR = ROWS && N2 % N1 == 0 ? N2 / N1 : 1;        // rows per thread
  static constexpr int T = CR > 1 ? N1 : (N1 > N2 ? N1 : N2);          // threads of a pencil
  static constexpr int TR = N2 / CR;                                   // threads with rows
  static constexpr int E = CR * N1;                                    // row elements of a thread
  static constexpr int R = E > N2 ? E : N2;                            // register elements
  static constexpr int RP = N1 | 1, PP = (N2 * RP) | 1;
  // pencils per CTA are capped to this; codelets past 16 points need more
  // than the 128 registers that 512 threads leave
  static constexpr int kMaxThreads = R > 16 ? 256 : 512;
  // element e of thread t in the second step's layout: wave number
  static __device__ __forceinline__ int k(int t, int e) { return t + TR * (e / N1) + N2 * (e % N1); }
};

// The pipelined kernels: pencils per CTA (at least a 128-byte segment per row
// and 64 threads) and the resident CTAs they are compiled for, with KREGS
// registers beside two register tiles of a thread
template <typename M, typename C2, int KREGS>
struct MixPipe {
  static constexpr int Wseg = 128 / sizeof(C2), Wthr = (64 / M::T + 7) / 8 * 8;
  static constexpr int W = Wseg > Wthr ? Wseg : Wthr, threads = W * M::T;
  static constexpr int regs = (int)sizeof(C2) / 4 * M::R * 2 + KREGS;
  static constexpr int fit = 65536 / (threads * regs);
  static constexpr int ctas = fit < 1 ? 1 : fit;
};
constexpr int kPipeYRegs = 44;  // addresses, twiddle and codelet temporaries
// the z passes also hold a kernel value per element
template <typename M, typename C2>
constexpr int pipe_z_regs() { return 52 + (int)sizeof(C2) / 8 * M::E; }

// twiddles w_N^(j1 k2) in both lane orders: ta[k2 N1 + j1], tb[j1 N2 + k2]
// (AxisPlan::mix: ta, then tb), read through the cache with consecutive lanes on
// consecutive entries (x passes) or on one entry (y and z passes)

// forward, first step: a[j2] = x[t + N1 j2] -> shared memory
template <typename M, bool INV, typename C2>
__device__ __forceinline__ void mix_fwd1(C2 (&a)[M::R], C2 *S, int t, const C2 *__restrict__ ta) {
  regfft::Dft<M::N2, INV, C2>::run(a);
#pragma unroll
  for (int k2 = 0; k2 < M::N2; k2++) {
    if (k2 > 0) {
      C2 w = __ldg(ta + k2 * M::N1 + t);
      if (INV) w.y = -w.y;
      a[k2] = regfft::mul(a[k2], w);
    }
    S[k2 * M::RP + t] = a[k2];
  }
}
// forward, second step: rows t + TR c -> a[e] = X[M::k(t, e)]
template <typename M, bool INV, typename C2>
__device__ __forceinline__ void mix_fwd2(C2 (&a)[M::R], const C2 *S, int t) {
#pragma unroll
  for (int c = 0; c < M::CR; c++) {
#pragma unroll
    for (int j = 0; j < M::N1; j++) a[c * M::N1 + j] = S[(t + M::TR * c) * M::RP + j];
    regfft::Dft<M::N1, INV, C2>::run(a + c * M::N1);
  }
}
// inverse, first step: a[e] = X[M::k(t, e)] -> rows of shared memory
template <typename M, bool INV, typename C2>
__device__ __forceinline__ void mix_bwd1(C2 (&a)[M::R], C2 *S, int t, const C2 *__restrict__ tb) {
#pragma unroll
  for (int c = 0; c < M::CR; c++) {
    regfft::Dft<M::N1, INV, C2>::run(a + c * M::N1);
#pragma unroll
    for (int j = 0; j < M::N1; j++) {
      C2 &x = a[c * M::N1 + j];
      if (j > 0) {
        C2 w = __ldg(tb + j * M::N2 + t + M::TR * c);
        if (INV) w.y = -w.y;
        x = regfft::mul(x, w);
      }
      S[(t + M::TR * c) * M::RP + j] = x;
    }
  }
}
// inverse, second step: column t -> a[n2] = x[t + N1 n2]
template <typename M, bool INV, typename C2>
__device__ __forceinline__ void mix_bwd2(C2 (&a)[M::R], const C2 *S, int t) {
#pragma unroll
  for (int k2 = 0; k2 < M::N2; k2++) a[k2] = S[k2 * M::RP + t];
  regfft::Dft<M::N2, INV, C2>::run(a);
}

// ---------------------------------------------------------------------------
// y pass (and z without a multiply): strided pencils in place.  Pencil pid is
// column kx = pid mod nxh of plane o = pid / nxh; the z pass's pencils are
// then consecutive elements.
// ---------------------------------------------------------------------------
template <typename C2>
struct MixYArgs {
  int nxh, nother;
  long so, sf;         // strides of o and of the transformed axis
  const C2 *ta;
  const BoxPair *box;  // non-null: only planes o inside the force box
  int nz;
  C2 *buf[kRegBatch];
};

template <typename M, bool INV, typename C2>
__global__ void __launch_bounds__(M::kMaxThreads) k_mix_y(MixYArgs<C2> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  after_previous();
  const int W = blockDim.x / M::T;
  const int w = threadIdx.x % W, t = threadIdx.x / W;
  C2 *S = reinterpret_cast<C2 *>(smem_raw) + w * M::PP;
  int lo = 0, hi = a.nother - 1;
  if (a.box) force_range(a.box, 2, a.nz, &lo, &hi);
  const int npid = (hi - lo + 1) * a.nxh;
  C2 *data = a.buf[blockIdx.y];
  for (int p0 = blockIdx.x * W; p0 < npid; p0 += gridDim.x * W) {
    const int pid = p0 + w, o = pid / a.nxh;
    const bool in = pid < npid;
    C2 *d = data + (long)(lo + o) * a.so + (pid - o * a.nxh);
    C2 v[M::R];
    if (in && t < M::N1) {
      C2 *s = d + t * a.sf;
#pragma unroll
      for (int j = 0; j < M::N2; j++) v[j] = s[(long)(M::N1 * j) * a.sf];
      mix_fwd1<M, INV>(v, S, t, a.ta);
    }
    __syncthreads();
    if (in && t < M::TR) {
      mix_fwd2<M, INV>(v, S, t);
      C2 *s = d + t * a.sf;
#pragma unroll
      for (int e = 0; e < M::E; e++) s[(long)M::k(0, e) * a.sf] = v[e];
    }
    if (p0 + gridDim.x * W < npid) __syncthreads();  // the next tile overwrites the rows
  }
}

// The same, persistent and software-pipelined: a CTA strides over the tiles
// and loads the next tile into registers before it transforms this one.
template <typename M, bool INV, typename C2>
__global__ void __launch_bounds__(MixPipe<M, C2, kPipeYRegs>::threads, MixPipe<M, C2, kPipeYRegs>::ctas)
    k_mix_y_pipe(MixYArgs<C2> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  after_previous();
  constexpr int W = MixPipe<M, C2, kPipeYRegs>::W;
  const int w = threadIdx.x % W, t = threadIdx.x / W;
  C2 *S = reinterpret_cast<C2 *>(smem_raw) + w * M::PP;
  const int npid = a.nother * a.nxh;
  C2 *data = a.buf[blockIdx.y];
  auto base = [&](int pid) -> C2 * {
    const int o = pid / a.nxh;
    return data + (long)o * a.so + (pid - o * a.nxh) + t * a.sf;
  };
  int pid = blockIdx.x * W + w;
  C2 *d = base(pid);
  C2 v[M::R];
  if (pid < npid && t < M::N1) {
#pragma unroll
    for (int j = 0; j < M::N2; j++) v[j] = d[(long)(M::N1 * j) * a.sf];
  }
  for (int p0 = blockIdx.x * W; p0 < npid; p0 += gridDim.x * W) {
    const int pidn = pid + gridDim.x * W;
    C2 *dn = base(pidn);
    C2 vn[M::R];
    if (pidn < npid && t < M::N1) {
#pragma unroll
      for (int j = 0; j < M::N2; j++) vn[j] = dn[(long)(M::N1 * j) * a.sf];
    }
    if (pid < npid && t < M::N1) mix_fwd1<M, INV>(v, S, t, a.ta);
    __syncthreads();
    if (pid < npid && t < M::TR) {
      mix_fwd2<M, INV>(v, S, t);
#pragma unroll
      for (int e = 0; e < M::E; e++) d[(long)M::k(0, e) * a.sf] = v[e];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < M::N2; j++) v[j] = vn[j];
    pid = pidn;
    d = dn;
  }
}

// ---------------------------------------------------------------------------
// z pass: IFFT_z(coef K [i D] FFT_z(in)), one job per output.  Outputs of one
// input each transform it again: the extra forward transform (its input from
// L2: jobs of a tile are adjacent CTAs; a job's output may be its own input,
// not another job's) costs less than keeping the forward
// result, which halves the CTAs per SM (256^3: density convolutions and force
// 375 -> 262 us per
// evaluation in FP64, 160 -> 147 in FP32).
// ---------------------------------------------------------------------------
template <typename C2>
struct MixZJob {
  const C2 *in;
  C2 *out;
  C2 *out2;  // non-null: out = i D_x and out2 = i D_y times the result (both
             // constant along z)
  const typename regfft::Re<C2>::type *kern;
  double coef;
  int dsym_axis;  // derivative symbol (2: along z) inside the transform, or -1
  int boxz;       // store only the z planes of the force box
};
constexpr int kMixJobs = 8;
template <typename C2>
struct MixZArgs {
  int npid, nxh, nx, ny, nz, njob;
  long sf;
  const typename regfft::Re<C2>::type *dsym;
  const C2 *ta, *tb;
  const BoxPair *box;
  MixZJob<C2> job[kMixJobs];
};

// DS: the jobs may carry derivative symbols and the box
template <typename M, bool DS, typename C2>
__global__ void __launch_bounds__(M::kMaxThreads) k_mix_zconv(MixZArgs<C2> a) {
  using T = typename regfft::Re<C2>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  after_previous();
  const int W = blockDim.x / M::T;
  const int w = threadIdx.x % W, t = threadIdx.x / W;
  C2 *S = reinterpret_cast<C2 *>(smem_raw) + w * M::PP;
  const int tile = blockIdx.x / a.njob;
  const MixZJob<C2> &J = a.job[blockIdx.x - tile * a.njob];
  const int pid = tile * W + w;
  const bool in = pid < a.npid, s1 = in && t < M::N1, s2 = in && t < M::TR;
  C2 v[M::R];
  if (s1) {
    const C2 *s = J.in + pid + t * a.sf;
#pragma unroll
    for (int j = 0; j < M::N2; j++) v[j] = s[(long)(M::N1 * j) * a.sf];
    mix_fwd1<M, false>(v, S, t, a.ta);
  }
  T K[M::E];
  if (s2) {
    const T coef = (T)J.coef;
    const T *kern = J.kern ? J.kern + pid + t * a.sf : nullptr;
#pragma unroll
    for (int e = 0; e < M::E; e++) K[e] = kern ? coef * __ldg(kern + (long)M::k(0, e) * a.sf) : coef;
  }
  __syncthreads();
  if (s2) {
    mix_fwd2<M, false>(v, S, t);
    T ds = 0;
    if (DS && J.dsym_axis >= 0 && J.dsym_axis < 2) {
      const int ky = pid / a.nxh;
      ds = J.dsym_axis == 0 ? a.dsym[pid - ky * a.nxh] : a.dsym[a.nx + ky];
    }
#pragma unroll
    for (int e = 0; e < M::E; e++) {
      v[e] = regfft::scale(v[e], K[e]);
      if (DS && J.dsym_axis >= 0) {
        if (J.dsym_axis == 2) ds = a.dsym[a.nx + a.ny + M::k(t, e)];
        v[e] = regfft::mk<C2>(-v[e].y * ds, v[e].x * ds);
      }
    }
    mix_bwd1<M, true>(v, S, t, a.tb);
  }
  __syncthreads();
  if (!s1) return;
  mix_bwd2<M, true>(v, S, t);
  C2 *d = J.out + pid + t * a.sf;
  if (!DS) {
#pragma unroll
    for (int n = 0; n < M::N2; n++) d[(long)(M::N1 * n) * a.sf] = v[n];
    return;
  }
  int zlo = 0, zhi = a.nz - 1;
  if (J.boxz) force_range(a.box, 2, a.nz, &zlo, &zhi);
  if (J.out2) {
    C2 *e = J.out2 + pid + t * a.sf;
    const int ky = pid / a.nxh;
    const T dx = a.dsym[pid - ky * a.nxh], dy = a.dsym[a.nx + ky];
#pragma unroll
    for (int n = 0; n < M::N2; n++) {
      const int z = t + M::N1 * n;
      if (z >= zlo && z <= zhi) {
        d[(long)(M::N1 * n) * a.sf] = regfft::mk<C2>(-v[n].y * dx, v[n].x * dx);
        e[(long)(M::N1 * n) * a.sf] = regfft::mk<C2>(-v[n].y * dy, v[n].x * dy);
      }
    }
  } else {
#pragma unroll
    for (int n = 0; n < M::N2; n++) {
      const int z = t + M::N1 * n;
      if (z >= zlo && z <= zhi) d[(long)(M::N1 * n) * a.sf] = v[n];
    }
  }
}

// z pass of a sum of convolutions.  The sum waits in shared memory at cells
// only its own thread uses (V), which keeps a thread's registers at one
// working set.
template <typename C2>
struct MixZSumArgs {
  int npid;
  long sf;
  const C2 *ta, *tb;
  const BoxPair *box;  // the z planes outside which a boxed term is zero
  int nz;
  int nterm;           // the first term is not boxed
  ZTermT<C2> t[kMaxTerms];
  C2 *out;
};
// z planes of the impurity box (lo > hi: none)
__device__ __forceinline__ void term_range(const BoxPair *bp, int nz, int *lo, int *hi) {
  const Box b = bp->cur;
  *lo = b.full ? 0 : b.empty ? 1 : b.lo[2];
  *hi = b.full ? nz - 1 : b.empty ? 0 : b.hi[2];
}

template <typename M, typename C2>
__global__ void __launch_bounds__(M::kMaxThreads) k_mix_zsum(MixZSumArgs<C2> a) {
  using T = typename regfft::Re<C2>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  after_previous();
  const int W = blockDim.x / M::T;
  const int w = threadIdx.x % W, t = threadIdx.x / W;
  C2 *S0 = reinterpret_cast<C2 *>(smem_raw), *S = S0 + w * M::PP;
  C2 *V = S0 + W * M::PP + threadIdx.x;
  const int pid = blockIdx.x * W + w;
  const bool in = pid < a.npid, s1 = in && t < M::N1, s2 = in && t < M::TR;
  C2 v[M::R];
  for (int j = 0; j < a.nterm; j++) {
    if (s1) {
      const C2 *s = a.t[j].in + pid + t * a.sf;
      if (a.t[j].boxed) {
        int lo, hi;
        term_range(a.box, a.nz, &lo, &hi);
#pragma unroll
        for (int q = 0; q < M::N2; q++) {
          const int z = t + M::N1 * q;
          v[q] = z >= lo && z <= hi ? s[(long)(M::N1 * q) * a.sf] : regfft::mk<C2>(0, 0);
        }
      } else {
#pragma unroll
        for (int q = 0; q < M::N2; q++) v[q] = s[(long)(M::N1 * q) * a.sf];
      }
    }
    if (j > 0) __syncthreads();  // every thread has read term j-1's rows
    if (s1) mix_fwd1<M, false>(v, S, t, a.ta);
    T K[M::E];
    if (s2) {
      const T coef = (T)a.t[j].coef;
#pragma unroll
      for (int e = 0; e < M::E; e++) K[e] = coef * __ldg(a.t[j].kern + pid + (long)M::k(t, e) * a.sf);
    }
    __syncthreads();
    if (s2) {
      mix_fwd2<M, false>(v, S, t);
#pragma unroll
      for (int k = 0; k < M::E; k++) {
        v[k] = regfft::scale(v[k], K[k]);
        if (j > 0) v[k] = regfft::add(V[k * blockDim.x], v[k]);
        if (j + 1 < a.nterm) V[k * blockDim.x] = v[k];
      }
    }
  }
  if (s2) mix_bwd1<M, true>(v, S, t, a.tb);
  __syncthreads();
  if (s1) {
    mix_bwd2<M, true>(v, S, t);
    C2 *d = a.out + pid + t * a.sf;
#pragma unroll
    for (int n = 0; n < M::N2; n++) d[(long)(M::N1 * n) * a.sf] = v[n];
  }
}

// The same, persistent and software-pipelined over (tile, term)
template <typename M, typename C2>
__global__ void __launch_bounds__(MixPipe<M, C2, pipe_z_regs<M, C2>()>::threads,
                                  MixPipe<M, C2, pipe_z_regs<M, C2>()>::ctas) k_mix_zsum_pipe(MixZSumArgs<C2> a) {
  using T = typename regfft::Re<C2>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  after_previous();
  constexpr int W = MixPipe<M, C2, pipe_z_regs<M, C2>()>::W;
  const int w = threadIdx.x % W, t = threadIdx.x / W;
  C2 *S0 = reinterpret_cast<C2 *>(smem_raw), *S = S0 + w * M::PP;
  C2 *V = S0 + W * M::PP + threadIdx.x;
  int pid = blockIdx.x * W + w;
  C2 v[M::R];
  if (pid < a.npid && t < M::N1) {
    const C2 *s = a.t[0].in + pid + t * a.sf;
#pragma unroll
    for (int q = 0; q < M::N2; q++) v[q] = s[(long)(M::N1 * q) * a.sf];
  }
  for (int p0 = blockIdx.x * W; p0 < a.npid; p0 += gridDim.x * W) {
    const bool in = pid < a.npid, s1 = in && t < M::N1, s2 = in && t < M::TR;
    for (int j = 0; j < a.nterm; j++) {
      const bool last = j + 1 == a.nterm;
      const int pidn = last ? pid + gridDim.x * W : pid;
      C2 vn[M::R];
      if (pidn < a.npid && t < M::N1) {
        const int jn = last ? 0 : j + 1;
        const C2 *s = a.t[jn].in + pidn + t * a.sf;
        if (a.t[jn].boxed) {
          int lo, hi;
          term_range(a.box, a.nz, &lo, &hi);
#pragma unroll
          for (int q = 0; q < M::N2; q++) {
            const int z = t + M::N1 * q;
            vn[q] = z >= lo && z <= hi ? s[(long)(M::N1 * q) * a.sf] : regfft::mk<C2>(0, 0);
          }
        } else {
#pragma unroll
          for (int q = 0; q < M::N2; q++) vn[q] = s[(long)(M::N1 * q) * a.sf];
        }
      }
      if (s1) mix_fwd1<M, false>(v, S, t, a.ta);
      T K[M::E];
      if (s2) {
        const T coef = (T)a.t[j].coef;
#pragma unroll
        for (int e = 0; e < M::E; e++) K[e] = coef * __ldg(a.t[j].kern + pid + (long)M::k(t, e) * a.sf);
      }
      __syncthreads();
      if (s2) {
        mix_fwd2<M, false>(v, S, t);
#pragma unroll
        for (int k = 0; k < M::E; k++) {
          v[k] = regfft::scale(v[k], K[k]);
          if (j > 0) v[k] = regfft::add(V[k * blockDim.x], v[k]);
          if (!last) V[k * blockDim.x] = v[k];
        }
      }
      if (last) {
        if (s2) mix_bwd1<M, true>(v, S, t, a.tb);
        __syncthreads();
        if (s1) {
          mix_bwd2<M, true>(v, S, t);
          C2 *d = a.out + pid + t * a.sf;
#pragma unroll
          for (int n = 0; n < M::N2; n++) d[(long)(M::N1 * n) * a.sf] = v[n];
        }
      } else {
        __syncthreads();  // every thread has read this term's rows
      }
#pragma unroll
      for (int q = 0; q < M::N2; q++) v[q] = vn[q];
    }
    pid += gridDim.x * W;
  }
}

// ---------------------------------------------------------------------------
// z pass of the energies: sums over k of |F|^2 K1 and Re(conj(F) G) K2, F and G
// the transforms of den and denx, which are the convolution energies
// sum_x den IFFT(F K1) and sum_x den IFFT(G K2) without their inverse
// transforms (Parseval; kx = 0 and nx / 2 count once, the others twice).  One
// read of the two x/y spectra that an evaluation keeps.  FP64 throughout: FP32
// spectra (CI = float2) are widened on load, since with an FP32 z transform the
// energies' rounding was 1.3 to 1.8 times that of the summed fields.
// ---------------------------------------------------------------------------
struct MixZEnergyArgs {
  int npid, nxh, nx, nz, w;  // w: pencils per CTA
  long sf;
  const double2 *ta;
  const BoxPair *box;
  const void *den, *denx;  // double2 or float2
  const double *k1, *k2;
  double *part;  // [2][gridDim.x]
};

template <typename M, typename CI>
__global__ void __launch_bounds__(M::kMaxThreads) k_mix_zenergy(MixZEnergyArgs a) {
  using C2 = double2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  after_previous();
  __shared__ double sh[32];
  // the CTA is rounded up to whole warps (block_sum); the threads past W T, whose
  // t is T or more, take neither step and add zeros
  const int W = a.w, VP = W * M::T;
  const int w = threadIdx.x % W, t = threadIdx.x / W;
  C2 *S0 = reinterpret_cast<C2 *>(smem_raw), *S = S0 + w * M::PP;
  C2 *V = S0 + W * M::PP + threadIdx.x;  // F at cells of this thread only
  const int pid = blockIdx.x * W + w;
  const bool in = pid < a.npid, s1 = in && t < M::N1, s2 = in && t < M::TR;
  const int kx = pid % a.nxh;
  const double wt = kx == 0 || 2 * kx == a.nx ? 1.0 : 2.0;
  double e1 = 0.0, e2 = 0.0;
  C2 v[M::R];
  if (s1) {
    const CI *s = static_cast<const CI *>(a.den) + pid + t * a.sf;
#pragma unroll
    for (int j = 0; j < M::N2; j++) {
      const CI x = s[(long)(M::N1 * j) * a.sf];
      v[j] = make_double2(x.x, x.y);
    }
    mix_fwd1<M, false>(v, S, t, a.ta);
  }
  __syncthreads();
  if (s2) {
    mix_fwd2<M, false>(v, S, t);
#pragma unroll
    for (int e = 0; e < M::E; e++) {
      const double x = v[e].x, y = v[e].y;
      e1 += (x * x + y * y) * __ldg(a.k1 + pid + (long)M::k(t, e) * a.sf);
      V[e * VP] = v[e];
    }
  }
  __syncthreads();
  if (s1) {
    int lo, hi;
    term_range(a.box, a.nz, &lo, &hi);
    const CI *s = static_cast<const CI *>(a.denx) + pid + t * a.sf;
#pragma unroll
    for (int j = 0; j < M::N2; j++) {
      const int z = t + M::N1 * j;
      v[j] = make_double2(0.0, 0.0);
      if (z >= lo && z <= hi) {
        const CI x = s[(long)(M::N1 * j) * a.sf];
        v[j] = make_double2(x.x, x.y);
      }
    }
    mix_fwd1<M, false>(v, S, t, a.ta);
  }
  __syncthreads();
  if (s2) {
    mix_fwd2<M, false>(v, S, t);
#pragma unroll
    for (int e = 0; e < M::E; e++) {
      const C2 F = V[e * VP];
      e2 += (F.x * v[e].x + F.y * v[e].y) * __ldg(a.k2 + pid + (long)M::k(t, e) * a.sf);
    }
  }
  e1 = block_sum(wt * e1, sh);
  e2 = block_sum(wt * e2, sh);
  if (threadIdx.x == 0) {
    a.part[blockIdx.x] = e1;
    a.part[gridDim.x + blockIdx.x] = e2;
  }
}

// ---------------------------------------------------------------------------
// x passes: two real rows per complex pencil (XRegArgs of fft_passes.cuh;
// tw holds ta, tw2 holds tb)
// ---------------------------------------------------------------------------
template <typename M, typename C2, int OP, typename TI>
__global__ void __launch_bounds__(M::kMaxThreads) k_mix_xr2c(XRegArgs<C2> a) {
  using T = typename regfft::Re<C2>::type;
  constexpr int N = M::N1 * M::N2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  after_previous();
  const int P = blockDim.x / M::T;
  const int p = threadIdx.x / M::T, t = threadIdx.x - p * M::T;
  C2 *S = reinterpret_cast<C2 *>(smem_raw) + p * M::PP;
  // fields that share an operand (ALFA) are neighbouring CTAs, which find it in
  // L2: 3 x 256^3 in FP64 212 -> 195 us
  const unsigned rt = OP == XLOAD_ALFA ? blockIdx.x / a.nb : blockIdx.x;
  const unsigned fld = OP == XLOAD_ALFA ? blockIdx.x - rt * a.nb : blockIdx.y;
  const long ra = ((long)rt * P + p) * 2, rb = ra + 1;
  const TI *in = static_cast<const TI *>(a.rin[fld]);
  C2 *out = a.cout[fld];
  bool ina = ra < a.nrow, inb = rb < a.nrow;
  if (a.boxp) {
    // an input that is zero outside the box's z planes: rows of planes of the
    // previous box are transformed or zeroed again, the others hold zeros
    auto within = [&](const Box &b, long row) {
      const int z = (int)(row / a.ny);
      return b.full || (!b.empty && z >= b.lo[2] && z <= b.hi[2]);
    };
    const Box cur = a.boxp->cur, prev = a.boxp->prev;
    const bool work = (ina && within(cur, ra)) || (inb && within(cur, rb));
    const bool stale = !work && ((ina && within(prev, ra)) || (inb && within(prev, rb)));
    if (stale)
      for (int k = t; k < a.nxh; k += M::T) {
        out[ra * a.nxh + k] = regfft::mk<C2>(0, 0);
        if (inb) out[rb * a.nxh + k] = regfft::mk<C2>(0, 0);
      }
    if (!__syncthreads_or(work)) return;
    ina = ina && work;
    inb = inb && work;
  }
  C2 v[M::R];
  if (ina && t < M::N1) {
    const long rbc = inb ? rb : ra;  // both rows' loads without a branch
    const float c0f = (float)a.ld.c0, c1f = (float)a.ld.c1;
#pragma unroll
    for (int j = 0; j < M::N2; j++) {
      const int x = t + M::N1 * j;
      v[j].x = xload_t<OP, TI, T>(a.ld, in, ra * N + x, c0f, c1f);
      v[j].y = xload_t<OP, TI, T>(a.ld, in, rbc * N + x, c0f, c1f);
    }
    if (!inb) {
#pragma unroll
      for (int j = 0; j < M::N2; j++) v[j].y = 0;
    }
    mix_fwd1<M, false>(v, S, t, a.tw);
  }
  __syncthreads();
  if (ina && t < M::TR) mix_fwd2<M, false>(v, S, t);
  __syncthreads();
  if (ina && t < M::TR) {  // the spectrum in natural order
#pragma unroll
    for (int e = 0; e < M::E; e++) S[M::k(t, e)] = v[e];
  }
  __syncthreads();
  if (!ina) return;
  for (int k = t; k <= N / 2; k += M::T) {
    const C2 zk = S[k], zm = S[k ? N - k : 0];
    // rows a, b: (Z(k) + conj Z(-k)) / 2 and -i (Z(k) - conj Z(-k)) / 2
    out[ra * a.nxh + k] = regfft::mk<C2>(T(0.5) * (zk.x + zm.x), T(0.5) * (zk.y - zm.y));
    if (inb) out[rb * a.nxh + k] = regfft::mk<C2>(T(0.5) * (zk.y + zm.y), T(-0.5) * (zk.x - zm.x));
  }
}

// the second step's threads load Z = X + i Y of their k straight from the two
// half spectra (k > N/2: the conjugates of N - k, which the cache holds from
// the lower half's loads), so the only shared-memory traffic is the exchange
template <typename M, typename C2, typename TO>
__global__ void __launch_bounds__(M::kMaxThreads) k_mix_xc2r(XRegArgs<C2> a) {
  using T = typename regfft::Re<C2>::type;
  constexpr int N = M::N1 * M::N2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  after_previous();
  const int P = blockDim.x / M::T;
  const int p = threadIdx.x / M::T, t = threadIdx.x - p * M::T;
  C2 *S = reinterpret_cast<C2 *>(smem_raw) + p * M::PP;
  const long ra = ((long)blockIdx.x * P + p) * 2, rb = ra + 1;
  bool ina = ra < a.nrow, inb = rb < a.nrow;
  if (a.box) {
    int ylo, yhi, zlo, zhi;
    force_range(a.box, 1, a.ny, &ylo, &yhi);
    force_range(a.box, 2, a.nz, &zlo, &zhi);
    const int za = (int)(ra / a.ny), ya = (int)(ra - (long)za * a.ny);
    const int zb = ya + 1 < a.ny ? za : za + 1, yb = ya + 1 < a.ny ? ya + 1 : 0;
    ina = ina && ya >= ylo && ya <= yhi && za >= zlo && za <= zhi;
    inb = inb && yb >= ylo && yb <= yhi && zb >= zlo && zb <= zhi;
    if (!__syncthreads_or(ina || inb)) return;
  }
  const C2 *in = a.cin[blockIdx.y];
  TO *out = static_cast<TO *>(a.rout[blockIdx.y]);
  C2 v[M::R];
  if ((ina || inb) && t < M::TR) {
    const C2 *A = in + (ina ? ra : rb) * a.nxh, *B = in + (inb ? rb : ra) * a.nxh;
#pragma unroll
    for (int i = 0; i < M::E; i++) {
      const int k = M::k(t, i);
      const bool up = 2 * k > N;
      const int q = up ? N - k : k;
      C2 X = A[q], Y = B[q];
      if (q == 0 || 2 * q == N) {  // DC / Nyquist of a real transform: drop Im
        X.y = 0;
        Y.y = 0;
      }
      if (up) {
        X.y = -X.y;
        Y.y = -Y.y;
      }
      v[i] = regfft::mk<C2>(X.x - Y.y, X.y + Y.x);
    }
    mix_bwd1<M, true>(v, S, t, a.tw2);
  }
  __syncthreads();
  if ((ina || inb) && t < M::N1) {
    mix_bwd2<M, true>(v, S, t);
    const T sc = (T)a.scale;
#pragma unroll
    for (int n = 0; n < M::N2; n++) {
      const int x = t + M::N1 * n;
      if (ina) out[ra * N + x] = (TO)(v[n].x * sc);
      if (inb) out[rb * N + x] = (TO)(v[n].y * sc);
    }
  }
}

// ---------------------------------------------------------------------------
// launches of one length
// ---------------------------------------------------------------------------
template <typename C2>
struct MixOps {
  int n, n1;   // n1: the second step's transform length
  int t, tx;   // threads of a pencil in the y and z passes, in the x passes
  // dynamic shared memory limits of the length's kernels on the current device
  int (*attrs)();
  int (*y)(Handle *h, MixYArgs<C2> &a, int nb, bool inverse, int w);
  int (*zconv)(Handle *h, MixZArgs<C2> &a, bool derivatives, int w);
  int (*zsum)(Handle *h, MixZSumArgs<C2> &a, int w);
  // (FP64 entries only) f32: the spectra are FP32
  int (*zenergy)(Handle *h, MixZEnergyArgs &a, bool f32, int w, int *ctas);
  int (*x)(Handle *h, XRegArgs<C2> &a, int nb, bool inverse, int p, bool out32);
};
// nullptr when the length has no such kernels; n1 = 0: the default factors
template <typename C2>
const MixOps<C2> *mix_ops(int n, int n1 = 0);

template <int N, typename C2, int F1 = 0>
struct MixLaunch {
  // Several rows per thread in the FP32 y and z passes only (128^3: y pass 7.0
  // -> 6.1 us, z sum 25 -> 20 us): FP64's second working set and the x passes'
  // shorter lane runs lose more than the busy threads gain (128^3: FP64 z sum
  // 40 -> 56 us, FP32 x C2R 7.2 -> 11.2 us)
  using M = Mix<N, F1, sizeof(C2) == 8>;
  using MX = Mix<N, F1, false>;
  using PY = MixPipe<M, C2, kPipeYRegs>;
  using PZ = MixPipe<M, C2, pipe_z_regs<M, C2>()>;
  static constexpr bool kPow2 = (N & (N - 1)) == 0;  // lengths of the FP32-convolution form
  // pencils per CTA: the tile width, capped by the kernels' thread limit
  template <typename Q = M>
  static int cap(int w) {
    return std::max(8, std::min(w, Q::kMaxThreads / Q::T / 8 * 8));
  }
  // the kernels with a second buffer: at least two CTAs per SM
  static int capv(int w) {
    w = cap(w);
    while (w > 8 && smem_v(w) > 110 * 1024) w -= 8;
    return w;
  }
  static size_t smem(int w) { return sizeof(C2) * (size_t)w * M::PP; }  // M and MX share the layout
  static size_t smem_v(int w) { return sizeof(C2) * (size_t)w * (M::PP + (size_t)M::T * M::E); }

  template <typename K>
  static int limit(K kern, size_t bytes) {
    HE4_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return HE4_OK;
  }
  template <typename TI>
  static int attrs_x() {
    const size_t s = smem(cap<MX>(32));
    HE4_TRY(limit(k_mix_xr2c<MX, C2, XLOAD_PLAIN, TI>, s));
    HE4_TRY(limit(k_mix_xr2c<MX, C2, XLOAD_ALFA, TI>, s));
    HE4_TRY(limit(k_mix_xr2c<MX, C2, XLOAD_CORR, TI>, s));
    return limit(k_mix_xc2r<MX, C2, TI>, s);
  }
  static int attrs() {
    const size_t s = smem(cap(32)), sv = smem_v(capv(32));
    HE4_TRY(limit(k_mix_y<M, false, C2>, s));
    HE4_TRY(limit(k_mix_y<M, true, C2>, s));
    HE4_TRY(limit(k_mix_y_pipe<M, false, C2>, s));
    HE4_TRY(limit(k_mix_y_pipe<M, true, C2>, s));
    HE4_TRY(limit(k_mix_zconv<M, false, C2>, s));
    HE4_TRY(limit(k_mix_zconv<M, true, C2>, s));
    if constexpr (kZSumPipe) HE4_TRY(limit(k_mix_zsum_pipe<M, C2>, sv));
    HE4_TRY(limit(k_mix_zsum<M, C2>, sv));
    if constexpr (sizeof(C2) == 16) {
      HE4_TRY(limit(k_mix_zenergy<M, double2>, sv));
      if constexpr (kPow2) HE4_TRY(limit(k_mix_zenergy<M, float2>, sv));
    }
    HE4_TRY(attrs_x<double>());
    if constexpr (sizeof(C2) == 8) HE4_TRY(attrs_x<float>());
    return HE4_OK;
  }
  static int y(Handle *h, MixYArgs<C2> &a, int nb, bool inverse, int w) {
    w = cap(w);
    long tiles = ((long)a.nxh * a.nother + w - 1) / w;
    const long ptiles = ((long)a.nxh * a.nother + PY::W - 1) / PY::W, resident = 148L * PY::ctas / nb;
    if (!a.box && ptiles > resident) {
      const dim3 grid((unsigned)resident, nb);
      if (inverse)
        HE4_TRY(launch_after(h, grid, PY::threads, smem(PY::W), k_mix_y_pipe<M, true, C2>, a));
      else
        HE4_TRY(launch_after(h, grid, PY::threads, smem(PY::W), k_mix_y_pipe<M, false, C2>, a));
      HE4_LAUNCHED(h);
      return HE4_OK;
    }
    // a box-restricted pass has few planes: a small grid strides over them
    if (a.box) tiles = std::min<long>(tiles, 148 * 4);
    const dim3 grid((unsigned)tiles, nb);
    if (inverse)
      HE4_TRY(launch_after(h, grid, w * M::T, smem(w), k_mix_y<M, true, C2>, a));
    else
      HE4_TRY(launch_after(h, grid, w * M::T, smem(w), k_mix_y<M, false, C2>, a));
    HE4_LAUNCHED(h);
    return HE4_OK;
  }
  static int zconv(Handle *h, MixZArgs<C2> &a, bool derivatives, int w) {
    w = cap(w);
    const unsigned grid = (unsigned)((a.npid + w - 1) / w) * a.njob;
    if (derivatives)
      HE4_TRY(launch_after(h, grid, w * M::T, smem(w), k_mix_zconv<M, true, C2>, a));
    else
      HE4_TRY(launch_after(h, grid, w * M::T, smem(w), k_mix_zconv<M, false, C2>, a));
    HE4_LAUNCHED(h);
    return HE4_OK;
  }
  // FP64 with 256 points: two register tiles of 255-register threads beat three
  // CTAs of one (343 -> 235 us at 256^3); at 240 points they measured equal (141
  // and 139 us) and below, and in FP32, slower (256^3: 103 and 147 us)
  static constexpr bool kZSumPipe = sizeof(C2) == 16 && N == 256;
  static int zsum(Handle *h, MixZSumArgs<C2> &a, int w) {
    const long resident = 148L * PZ::ctas;
    if constexpr (kZSumPipe) {
      if ((a.npid + PZ::W - 1) / PZ::W > resident) {
        HE4_TRY(launch_after(h, (unsigned)resident, PZ::threads, smem_v(PZ::W), k_mix_zsum_pipe<M, C2>, a));
        HE4_LAUNCHED(h);
        return HE4_OK;
      }
    }
    w = capv(w);
    HE4_TRY(launch_after(h, (unsigned)((a.npid + w - 1) / w), w * M::T, smem_v(w), k_mix_zsum<M, C2>, a));
    HE4_LAUNCHED(h);
    return HE4_OK;
  }
  static int zenergy(Handle *h, MixZEnergyArgs &a, bool f32, int w, int *ctas) {
    if constexpr (sizeof(C2) == 16) {
      a.w = w = capv(w);
      *ctas = (a.npid + w - 1) / w;
      const int threads = (w * M::T + 31) / 32 * 32;  // at most kMaxThreads, as w T is
      if (!f32) {
        HE4_TRY(launch_after(h, *ctas, threads, smem_v(w), k_mix_zenergy<M, double2>, a));
      } else if constexpr (kPow2) {
        HE4_TRY(launch_after(h, *ctas, threads, smem_v(w), k_mix_zenergy<M, float2>, a));
      }
      HE4_LAUNCHED(h);
      return HE4_OK;
    }
    set_error("the energies' z pass runs in FP64");
    return HE4_E_ARG;
  }
  template <typename TI>
  static int r2c(Handle *h, XRegArgs<C2> &a, dim3 grid, int threads, size_t sm) {
    a.nb = (int)grid.y;
    if (a.ld.op == XLOAD_ALFA)
      HE4_TRY(launch_after(h, dim3(grid.x * grid.y), threads, sm, k_mix_xr2c<MX, C2, XLOAD_ALFA, TI>, a));
    else if (a.ld.op == XLOAD_CORR)
      HE4_TRY(launch_after(h, grid, threads, sm, k_mix_xr2c<MX, C2, XLOAD_CORR, TI>, a));
    else
      HE4_TRY(launch_after(h, grid, threads, sm, k_mix_xr2c<MX, C2, XLOAD_PLAIN, TI>, a));
    return HE4_OK;
  }
  // out32, a.ld.real32: float real grids (FP32-convolution form only)
  static int x(Handle *h, XRegArgs<C2> &a, int nb, bool inverse, int p, bool out32) {
    p = cap<MX>(p);
    const dim3 grid((unsigned)((a.nrow + 2 * p - 1) / (2 * p)), nb);
    const size_t sm = smem(p);
    const int threads = p * MX::T;
    if constexpr (sizeof(C2) == 8) {
      if (inverse && out32)
        HE4_TRY(launch_after(h, grid, threads, sm, k_mix_xc2r<MX, C2, float>, a));
      else if (!inverse && a.ld.real32)
        HE4_TRY(r2c<float>(h, a, grid, threads, sm));
      else if (inverse)
        HE4_TRY(launch_after(h, grid, threads, sm, k_mix_xc2r<MX, C2, double>, a));
      else
        HE4_TRY(r2c<double>(h, a, grid, threads, sm));
    } else {
      if (out32 || a.ld.real32) {
        set_error("float real grids need the FP32-convolution form");
        return HE4_E_ARG;
      }
      if (inverse)
        HE4_TRY(launch_after(h, grid, threads, sm, k_mix_xc2r<MX, C2, double>, a));
      else
        HE4_TRY(r2c<double>(h, a, grid, threads, sm));
    }
    HE4_LAUNCHED(h);
    return HE4_OK;
  }
  static constexpr MixOps<C2> ops() { return MixOps<C2>{N, M::N1, M::T, MX::T, &attrs, &y, &zconv, &zsum, &zenergy, &x}; }
};

// one translation unit per group of lengths (they compile in parallel)
#define HE4_MIX_TABLE(name, C2, ...)                                 \
  const MixOps<C2> *name(int n, int n1) {                            \
    static const MixOps<C2> t[] = {__VA_ARGS__};                     \
    for (const MixOps<C2> &o : t)                                    \
      if (o.n == n && (n1 == 0 || o.n1 == n1)) return &o;            \
    return nullptr;                                                  \
  }

}  // namespace he4
