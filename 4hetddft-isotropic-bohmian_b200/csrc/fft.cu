// fft.cu -- batched 3D real FFTs for the convolutions of the mean field.
//
// Replaces the FFTW plans and their executions (fft.f90:43-65, 79-207).
// Layout: real grids [nz][ny][nx]; half spectra [nz][ny][nx/2+1] (the FFTW
// r2c layout of the reference).  Forward transforms are unnormalised; the
// reference's backward scaling by renor = 1/N (fft.f90:130,138,...) is folded
// into the coefficient of the k-space multiply of the z pass.
//
// A 3D transform is three passes over HBM:
//   x pass  (R2C / C2R): two real rows packed into one complex pencil,
//   y pass  (complex), and
//   z pass  (complex) fused with the k-space kernel multiply and the inverse
//           z transform: FFT_z -> coef*K(k) (*i*D(k)) -> IFFT_z in one launch.
// Axis lengths 36..250 with factors 2, 3 and 5 and the powers of two from 16 to 256
// run as the two-step register passes of fft_mix.cuh (FP32 spectra: the powers of two
// only), chosen per axis; this file holds their tables and launches.  The other
// lengths (8..30) run the generic kernels below: each CTA stages a tile of pencils
// in shared memory and runs a mixed-radix (2/3/4/5) Stockham transform between two
// shared buffers; pencils of one tile are contiguous in x, so every global access is
// a coalesced segment.
#include <math.h>
#include <stdlib.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <set>
#include <utility>
#include <vector>

#include <cuda_pipeline.h>

#include "common.cuh"
#include "fft_mix.cuh"
#include "fft_passes.cuh"

namespace he4 {

static constexpr double kC3S = 0.86602540378443864676372317075293618;   // sin(2pi/3)
static constexpr double kC5C1 = 0.30901699437494742410229341718281906;  // cos(2pi/5)
static constexpr double kC5C2 = -0.80901699437494742410229341718281906; // cos(4pi/5)
static constexpr double kC5S1 = 0.95105651629515357211643933337938214;  // sin(2pi/5)
static constexpr double kC5S2 = 0.58778525229247312916870595463907277;  // sin(4pi/5)

constexpr int kThreads = 256;

// ---------------------------------------------------------------------------
// small DFTs (forward: exp(-2 pi i jk/R); inverse: conjugate roots)
// ---------------------------------------------------------------------------
template <int R, bool INV>
struct Dft;

template <bool INV>
struct Dft<2, INV> {
  static __device__ __forceinline__ void run(double2 *u) {
    double2 t = u[0];
    u[0] = cadd(t, u[1]);
    u[1] = csub(t, u[1]);
  }
};

template <bool INV>
struct Dft<4, INV> {
  static __device__ __forceinline__ void run(double2 *u) {
    double2 a = cadd(u[0], u[2]), b = csub(u[0], u[2]);
    double2 c = cadd(u[1], u[3]), d = cmuli<INV>(csub(u[1], u[3]));
    u[0] = cadd(a, c);
    u[2] = csub(a, c);
    u[1] = cadd(b, d);
    u[3] = csub(b, d);
  }
};

template <bool INV>
struct Dft<3, INV> {
  static __device__ __forceinline__ void run(double2 *u) {
    double2 t1 = cadd(u[1], u[2]);
    double2 t2 = csub(u[0], cscale(t1, 0.5));
    double2 t3 = cscale(cmuli<INV>(csub(u[1], u[2])), kC3S);
    u[0] = cadd(u[0], t1);
    u[1] = cadd(t2, t3);
    u[2] = csub(t2, t3);
  }
};

template <bool INV>
struct Dft<5, INV> {
  static __device__ __forceinline__ void run(double2 *u) {
    double2 a1 = cadd(u[1], u[4]), b1 = csub(u[1], u[4]);
    double2 a2 = cadd(u[2], u[3]), b2 = csub(u[2], u[3]);
    double2 r1 = cadd(u[0], cadd(cscale(a1, kC5C1), cscale(a2, kC5C2)));
    double2 r2 = cadd(u[0], cadd(cscale(a1, kC5C2), cscale(a2, kC5C1)));
    double2 s1 = cmuli<INV>(cadd(cscale(b1, kC5S1), cscale(b2, kC5S2)));
    double2 s2 = cmuli<INV>(csub(cscale(b1, kC5S2), cscale(b2, kC5S1)));
    u[0] = cadd(u[0], cadd(a1, a2));
    u[1] = cadd(r1, s1);
    u[4] = csub(r1, s1);
    u[2] = cadd(r2, s2);
    u[3] = csub(r2, s2);
  }
};

// One Stockham stage on W pencils stored [n][ld] (pencil w at column w):
// butterfly i of pencil w reads x[i + j n/R], applies w_{pR}^{jk}
// (k = i mod p), runs the R-point DFT and writes y[(i/p) p R + k + j p].
template <int R, bool INV>
__device__ __forceinline__ void stage(const double2 *__restrict__ src, double2 *__restrict__ dst, int n,
                                      int p, int W, int ld, const double2 *__restrict__ tw) {
  const int m = n / R, tstep = n / (p * R);
  const int nb = m * W;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    const int w = b % W, i = b / W, k = i % p;
    double2 u[R];
#pragma unroll
    for (int j = 0; j < R; j++) u[j] = src[(i + j * m) * ld + w];
    if (k) {
#pragma unroll
      for (int j = 1; j < R; j++) {
        double2 t = tw[j * k * tstep];
        if (INV) t.y = -t.y;
        u[j] = cmul(u[j], t);
      }
    }
    Dft<R, INV>::run(u);
    const int j0 = (i / p) * p * R + k;
#pragma unroll
    for (int j = 0; j < R; j++) dst[(j0 + j * p) * ld + w] = u[j];
  }
}

// Full transform of W pencils; a holds the input, b is scratch.  Returns the
// buffer holding the natural-order result.
template <bool INV>
__device__ double2 *fft_smem(double2 *a, double2 *b, const AxisPlan &P, int W, int ld,
                             const double2 *__restrict__ tw) {
  int p = 1;
  for (int s = 0; s < P.nst; s++) {
    const int R = P.radix[s];
    switch (R) {
      case 4: stage<4, INV>(a, b, P.n, p, W, ld, tw); break;
      case 2: stage<2, INV>(a, b, P.n, p, W, ld, tw); break;
      case 3: stage<3, INV>(a, b, P.n, p, W, ld, tw); break;
      default: stage<5, INV>(a, b, P.n, p, W, ld, tw); break;
    }
    __syncthreads();
    double2 *t = a;
    a = b;
    b = t;
    p *= R;
  }
  return a;
}

__device__ __forceinline__ void load_tw(double2 *s_tw, const AxisPlan &P) {
  for (int t = threadIdx.x; t < P.n; t += blockDim.x) s_tw[t] = P.tw[t];
}

// ---------------------------------------------------------------------------
// x pass
// ---------------------------------------------------------------------------
constexpr int kMaxBatch = 8;

struct XArgs {
  AxisPlan ax;
  int nxh, P;
  long nrow;
  double scale;
  const double *rin[kMaxBatch];
  double2 *cout[kMaxBatch];
  const double2 *cin[kMaxBatch];
  double *rout[kMaxBatch];
};

__global__ void __launch_bounds__(kThreads) k_fft_x_r2c(XArgs a) {
  extern __shared__ double2 smem[];
  const int n = a.ax.n, P = a.P, ld = P + 1, nxh = a.nxh;
  double2 *b0 = smem, *b1 = smem + n * ld, *tw = smem + 2 * n * ld;
  load_tw(tw, a.ax);
  const double *in = a.rin[blockIdx.y];
  double2 *out = a.cout[blockIdx.y];
  const long row0 = (long)blockIdx.x * 2 * P;
  for (int e = threadIdx.x; e < n * P; e += blockDim.x) {
    const int q = e / n, x = e - q * n;
    const long ra = row0 + 2 * q, rb = ra + 1;
    double va = (ra < a.nrow) ? in[ra * n + x] : 0.0;
    double vb = (rb < a.nrow) ? in[rb * n + x] : 0.0;
    b0[x * ld + q] = make_double2(va, vb);
  }
  __syncthreads();
  double2 *res = fft_smem<false>(b0, b1, a.ax, P, ld, tw);
  for (int e = threadIdx.x; e < nxh * P; e += blockDim.x) {
    const int q = e / nxh, k = e - q * nxh;
    const long ra = row0 + 2 * q, rb = ra + 1;
    const double2 zk = res[k * ld + q];
    const double2 zm = cconj(res[((n - k) % n) * ld + q]);
    const double2 A = cscale(cadd(zk, zm), 0.5);
    const double2 d = cscale(csub(zk, zm), 0.5);
    if (ra < a.nrow) out[ra * nxh + k] = A;
    if (rb < a.nrow) out[rb * nxh + k] = make_double2(d.y, -d.x);
  }
}

__global__ void __launch_bounds__(kThreads) k_fft_x_c2r(XArgs a) {
  extern __shared__ double2 smem[];
  const int n = a.ax.n, P = a.P, ld = P + 1, nxh = a.nxh;
  double2 *b0 = smem, *b1 = smem + n * ld, *tw = smem + 2 * n * ld;
  load_tw(tw, a.ax);
  const double2 *in = a.cin[blockIdx.y];
  double *out = a.rout[blockIdx.y];
  const long row0 = (long)blockIdx.x * 2 * P;
  for (int e = threadIdx.x; e < nxh * P; e += blockDim.x) {
    const int q = e / nxh, k = e - q * nxh;
    const long ra = row0 + 2 * q, rb = ra + 1;
    double2 X = (ra < a.nrow) ? in[ra * nxh + k] : make_double2(0.0, 0.0);
    double2 Y = (rb < a.nrow) ? in[rb * nxh + k] : make_double2(0.0, 0.0);
    if (k == 0 || 2 * k == n) {  // DC / Nyquist of a real transform: drop Im
      X.y = 0.0;
      Y.y = 0.0;
    }
    b0[k * ld + q] = make_double2(X.x - Y.y, X.y + Y.x);  // X + iY
    if (k > 0 && n - k >= nxh) b0[(n - k) * ld + q] = make_double2(X.x + Y.y, Y.x - X.y);  // conj(X) + i conj(Y)
  }
  __syncthreads();
  double2 *res = fft_smem<true>(b0, b1, a.ax, P, ld, tw);
  const double sc = a.scale;
  for (int e = threadIdx.x; e < n * P; e += blockDim.x) {
    const int q = e / n, x = e - q * n;
    const long ra = row0 + 2 * q, rb = ra + 1;
    const double2 v = res[x * ld + q];
    if (ra < a.nrow) out[ra * n + x] = v.x * sc;
    if (rb < a.nrow) out[rb * n + x] = v.y * sc;
  }
}

struct YArgs {
  AxisPlan ay;
  PencilMap map;
  long sf;  // element stride along the transformed axis
  double2 *buf[kMaxBatch];
};

template <bool INV>
__global__ void __launch_bounds__(kThreads) k_fft_y(YArgs a) {
  extern __shared__ double2 smem[];
  const int n = a.ay.n, W = a.map.W;
  double2 *b0 = smem, *b1 = smem + n * W, *tw = smem + 2 * n * W;
  long *offs = reinterpret_cast<long *>(tw + n);
  load_tw(tw, a.ay);
  for (int w = threadIdx.x; w < W; w += blockDim.x) {
    int kx, o;
    offs[w] = pencil_offset(a.map, (long)blockIdx.x * W + w, &kx, &o);
  }
  __syncthreads();
  double2 *data = a.buf[blockIdx.y];
  for (int e = threadIdx.x; e < n * W; e += blockDim.x) {
    const int w = e % W, j = e / W;
    const long off = offs[w];
    b0[j * W + w] = (off >= 0) ? data[off + j * a.sf] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  double2 *res = fft_smem<INV>(b0, b1, a.ay, W, W, tw);
  for (int e = threadIdx.x; e < n * W; e += blockDim.x) {
    const int w = e % W, j = e / W;
    const long off = offs[w];
    if (off >= 0) data[off + j * a.sf] = res[j * W + w];
  }
}

struct ZArgs {
  AxisPlan az;
  PencilMap map;
  long sf;
  int nx, ny, nz;
  const double *dsym;  // [nx | ny | nz]
  ZOp ops[kMaxBatch];
};

__global__ void __launch_bounds__(kThreads) k_fft_z_conv(ZArgs a) {
  extern __shared__ double2 smem[];
  const int n = a.az.n, W = a.map.W;
  double2 *b0 = smem, *b1 = smem + n * W, *tw = smem + 2 * n * W;
  long *offs = reinterpret_cast<long *>(tw + n);
  int *kxs = reinterpret_cast<int *>(offs + W);
  int *kys = kxs + W;
  load_tw(tw, a.az);
  for (int w = threadIdx.x; w < W; w += blockDim.x) {
    int kx = 0, o = 0;
    offs[w] = pencil_offset(a.map, (long)blockIdx.y * W + w, &kx, &o);
    kxs[w] = kx;
    kys[w] = o;
  }
  __syncthreads();
  const ZOp op = a.ops[blockIdx.x];
  for (int e = threadIdx.x; e < n * W; e += blockDim.x) {
    const int w = e % W, j = e / W;
    const long off = offs[w];
    b0[j * W + w] = (off >= 0) ? op.in[off + j * a.sf] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  if (op.mode != 0) {  // plain forward or inverse transform along z
    double2 *r = (op.mode == 1) ? fft_smem<false>(b0, b1, a.az, W, W, tw) : fft_smem<true>(b0, b1, a.az, W, W, tw);
    for (int e = threadIdx.x; e < n * W; e += blockDim.x) {
      const int w = e % W, j = e / W;
      const long off = offs[w];
      if (off >= 0) op.out[off + j * a.sf] = r[j * W + w];
    }
    return;
  }
  double2 *res = fft_smem<false>(b0, b1, a.az, W, W, tw);
  double2 *wk = (res == b0) ? b1 : b0;
  for (int e = threadIdx.x; e < n * W; e += blockDim.x) {
    const int w = e % W, j = e / W;
    const long off = offs[w];
    double c = op.coef;
    if (off >= 0 && op.kern) c *= op.kern[off + j * a.sf];
    double2 v = cscale(res[j * W + w], c);
    if (op.dsym_axis >= 0) {
      double ds;
      if (op.dsym_axis == 0) ds = a.dsym[kxs[w]];
      else if (op.dsym_axis == 1) ds = a.dsym[a.nx + kys[w]];
      else ds = a.dsym[a.nx + a.ny + j];
      v = make_double2(-v.y * ds, v.x * ds);  // times i*ds
    }
    wk[j * W + w] = v;
  }
  __syncthreads();
  double2 *out = (wk == b0) ? fft_smem<true>(b0, b1, a.az, W, W, tw) : fft_smem<true>(b1, b0, a.az, W, W, tw);
  for (int e = threadIdx.x; e < n * W; e += blockDim.x) {
    const int w = e % W, j = e / W;
    const long off = offs[w];
    if (off >= 0) op.out[off + j * a.sf] = out[j * W + w];
  }
}


// ---------------------------------------------------------------------------
// two-step register kernels (fft_mix.cuh): the tables of the translation units
// ---------------------------------------------------------------------------
const MixOps<double2> *mix_table0(int n, int n1);
const MixOps<double2> *mix_table1(int n, int n1);
const MixOps<double2> *mix_table2(int n, int n1);
const MixOps<double2> *mix_table3(int n, int n1);
const MixOps<double2> *mix_table4(int n, int n1);
const MixOps<double2> *mix_table5(int n, int n1);
const MixOps<double2> *mix_table6(int n, int n1);
const MixOps<float2> *mix_table7(int n, int n1);

template <>
const MixOps<double2> *mix_ops<double2>(int n, int n1) {
  const MixOps<double2> *(*const tables[])(int, int) = {mix_table6, mix_table0, mix_table1, mix_table2,
                                                        mix_table3, mix_table4, mix_table5};
  for (auto *t : tables)
    if (const MixOps<double2> *o = t(n, n1)) return o;
  return nullptr;
}
template <>
const MixOps<float2> *mix_ops<float2>(int n, int n1) {
  return mix_table7(n, n1);
}

// axis lengths whose first factor n1 the tile autotuner may choose
static bool pow2_axis(int n) { return n >= 16 && n <= 256 && (n & (n - 1)) == 0; }
static bool n1_ok(int n, int n1) { return pow2_axis(n) && n1 > 0 && mix_ops<double2>(n, n1) != nullptr; }

// ---------------------------------------------------------------------------
// twiddle tables
// ---------------------------------------------------------------------------
static int axis_init(AxisPlan &A, int n) {
  A.n = n;
  A.nst = 0;
  int r = n;
  while (r % 4 == 0) { A.radix[A.nst++] = 4; r /= 4; }
  while (r % 2 == 0) { A.radix[A.nst++] = 2; r /= 2; }
  while (r % 3 == 0) { A.radix[A.nst++] = 3; r /= 3; }
  while (r % 5 == 0) { A.radix[A.nst++] = 5; r /= 5; }
  if (r != 1 || A.nst > kMaxStages) {
    set_error("FFT length %d is not of the form 2^a 3^b 5^c", n);
    return HE4_E_UNSUPPORTED;
  }
  // one allocation and one upload for all of an axis's tables (each costs the
  // driver a fraction of a millisecond): w_n^t, then per choice of the first
  // factor n1 of the two-step kernels w_n^(j k) by (k, j) and by (j, k), and
  // the same rounded to FP32
  std::vector<double2> tab(n);
  std::vector<float2> w32(n);
  for (int t = 0; t < n; t++) {
    long double ang = -2.0L * 3.14159265358979323846264338327950288L * (long double)t / (long double)n;
    const long double c = cosl(ang), s = sinl(ang);
    tab[t] = make_double2((double)c, (double)s);
    w32[t] = make_float2((float)c, (float)s);
  }
  int nv = 0;
  for (int n1 = 2; n1 <= n && nv < AxisPlan::kSplits; n1++)
    if (mix_ops<double2>(n, n1)) A.split[nv++] = n1;
  // FP32 tables after the FP64 ones: 2 n float2 take the room of n double2
  tab.resize(n + 3 * (size_t)n * nv);
  for (int v = 0; v < nv; v++) {
    const int n1 = A.split[v], n2 = n / n1;
    double2 *m = &tab[n + 2 * (size_t)n * v];
    float2 *mf = reinterpret_cast<float2 *>(&tab[n + 2 * (size_t)n * nv + (size_t)n * v]);
    for (int j = 0; j < n1; j++)
      for (int k = 0; k < n2; k++) {  // j k < n
        m[k * n1 + j] = m[n + j * n2 + k] = tab[j * k];
        mf[k * n1 + j] = mf[n + j * n2 + k] = w32[j * k];
      }
  }
  cudaError_t e = cudaMalloc(&A.tw, sizeof(double2) * tab.size());
  if (e == cudaSuccess) e = cudaMemcpy(A.tw, tab.data(), sizeof(double2) * tab.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    set_error("twiddle upload: %s", cudaGetErrorString(e));
    return HE4_E_CUDA;
  }
  for (int v = 0; v < nv; v++) {
    A.mix[v] = A.tw + n + 2 * (size_t)n * v;
    A.mix32[v] = reinterpret_cast<float2 *>(A.tw + n + 2 * (size_t)n * nv + (size_t)n * v);
  }
  return HE4_OK;
}

// kernels and tables of an axis with first factor n1 (0: the default) in the
// spectrum type C2; ops is null when the length has none
template <typename C2>
struct AxisMix {
  const MixOps<C2> *ops;
  const C2 *ta, *tb;
};
template <typename C2>
static const C2 *mix_tab(const AxisPlan &A, int v);
template <>
const double2 *mix_tab<double2>(const AxisPlan &A, int v) { return A.mix[v]; }
template <>
const float2 *mix_tab<float2>(const AxisPlan &A, int v) { return A.mix32[v]; }
template <typename C2>
static AxisMix<C2> axis_mix(const AxisPlan &A, int n1) {
  AxisMix<C2> m{mix_ops<C2>(A.n, n1), nullptr, nullptr};
  if (!m.ops) return m;
  for (int v = 0; v < AxisPlan::kSplits; v++)
    if (A.split[v] == m.ops->n1) m.ta = mix_tab<C2>(A, v);
  m.tb = m.ta + A.n;
  return m;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static int tile_width(int n) {
  int w = 2048 / n;
  w = (w / 8) * 8;
  return std::max(8, std::min(32, w));
}

static size_t smem_x(const FftPlan &P) { return sizeof(double2) * (2 * (size_t)P.nx * (P.px + 1) + P.nx); }
static size_t smem_yz(int n, int W) {
  return sizeof(double2) * (2 * (size_t)n * W + n) + sizeof(long) * W + 2 * sizeof(int) * W;
}

// The dynamic shared memory limits of the generic-path kernels are set per
// device (a cudaFuncSetAttribute call applies to the current device only);
// per device they only ever grow, to the widest tiles any plan there uses.
// A maximum is recorded only after the attribute call succeeded, so a failed
// call is retried by the next plan.
static int generic_attrs(const FftPlan &P) {
  static std::mutex mu;
  static size_t max_x[kMaxDevices] = {0}, max_y[kMaxDevices] = {0}, max_z[kMaxDevices] = {0};
  int dev = 0;
  HE4_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) {
    set_error("device ordinal %d beyond the %d this library supports", dev, kMaxDevices);
    return HE4_E_ARG;
  }
  std::lock_guard<std::mutex> lock(mu);
  const size_t sx = smem_x(P), sy = smem_yz(P.ny, P.wy), sz = smem_yz(P.nz, P.wz);
  if (sx > max_x[dev]) {
    HE4_CUDA_TRY(cudaFuncSetAttribute(k_fft_x_r2c, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sx));
    HE4_CUDA_TRY(cudaFuncSetAttribute(k_fft_x_c2r, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sx));
    max_x[dev] = sx;
  }
  if (sy > max_y[dev]) {
    HE4_CUDA_TRY(cudaFuncSetAttribute(k_fft_y<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sy));
    HE4_CUDA_TRY(cudaFuncSetAttribute(k_fft_y<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sy));
    max_y[dev] = sy;
  }
  if (sz > max_z[dev]) {
    HE4_CUDA_TRY(cudaFuncSetAttribute(k_fft_z_conv, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sz));
    max_z[dev] = sz;
  }
  return HE4_OK;
}

// dynamic shared memory limits of a length's two-step kernels, set once per
// device (they do not depend on the plan)
template <typename C2>
static int mix_attrs(const MixOps<C2> *mo) {
  static std::mutex mu;
  static std::set<std::pair<const void *, int>> done;
  int dev = 0;
  HE4_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (done.count({mo, dev})) return HE4_OK;
  HE4_TRY(mo->attrs());
  done.insert({mo, dev});
  return HE4_OK;
}

int fft_plan_init(FftPlan &P, int nx, int ny, int nz) {
  P.nx = nx;
  P.ny = ny;
  P.nz = nz;
  P.nxh = nx / 2 + 1;
  HE4_TRY(axis_init(P.ax, nx));
  HE4_TRY(axis_init(P.ay, ny));
  HE4_TRY(axis_init(P.az, nz));
  // axes with factors 3 and 5: 8 pencils per CTA, the most CTAs and (FP64)
  // 128-byte segments; 16 and 24 measured 1-5 % and 8-16 % slower steps at
  // 96^3, 90 x 100 x 120, 144 x 150 x 160 and 192 x 192 x 240
  auto width = [](int n) { return mix_ops<double2>(n) && !pow2_axis(n) ? 8 : tile_width(n); };
  P.px = width(nx);
  P.wy = width(ny);
  P.wz = width(nz);
  HE4_TRY(generic_attrs(P));
  const int ns[3] = {nx, ny, nz};
  for (int a = 0; a < 3; a++) {
    const int n = ns[a];
    P.n1[a] = pow2_axis(n) ? mix_ops<double2>(n)->n1 : 0;
    const AxisPlan &A = a == 0 ? P.ax : a == 1 ? P.ay : P.az;
    for (int v = 0; v < AxisPlan::kSplits && A.split[v]; v++) {
      if (const auto *mo = mix_ops<double2>(n, A.split[v])) HE4_TRY(mix_attrs(mo));
      if (const auto *mo = mix_ops<float2>(n, A.split[v])) HE4_TRY(mix_attrs(mo));
    }
  }
  return HE4_OK;
}

// Tile shapes: t = {n1 x, n1 y, n1 z, px, wy, wz}.  n1 applies to the axes of 16 to
// 256 points that are powers of two (0 = default split), px / wy / wz (pencils per
// CTA, multiples of 8 in [8, 32]) to all others; an axis ignores the other entry.
int fft_set_tiles(FftPlan &P, const int *t) {
  const int ns[3] = {P.nx, P.ny, P.nz};
  int n1[3];
  for (int a = 0; a < 3; a++) {
    n1[a] = 0;
    if (!pow2_axis(ns[a])) continue;
    n1[a] = t[a] ? t[a] : mix_ops<double2>(ns[a])->n1;
    if (!n1_ok(ns[a], n1[a])) {
      set_error("axis %d: no register FFT split %d x %d", a, n1[a], ns[a] / n1[a]);
      return HE4_E_ARG;
    }
  }
  FftPlan Q = P;
  Q.px = pow2_axis(P.nx) ? P.px : t[3];
  Q.wy = pow2_axis(P.ny) ? P.wy : t[4];
  Q.wz = pow2_axis(P.nz) ? P.wz : t[5];
  const int ws[3] = {Q.px, Q.wy, Q.wz};
  for (int a = 0; a < 3; a++)
    if (ws[a] < 8 || ws[a] > 32 || ws[a] % 8) {
      set_error("tile width %d is not a multiple of 8 in [8, 32]", ws[a]);
      return HE4_E_ARG;
    }
  const size_t lim = 200 * 1024;
  if (smem_x(Q) > lim || smem_yz(Q.ny, Q.wy) > lim || smem_yz(Q.nz, Q.wz) > lim) {
    set_error("tile widths need more than %zu bytes of shared memory", lim);
    return HE4_E_ARG;
  }
  HE4_TRY(generic_attrs(Q));
  for (int a = 0; a < 3; a++) Q.n1[a] = n1[a];
  P = Q;
  return HE4_OK;
}

void fft_get_tiles(const FftPlan &P, int *t) {
  for (int a = 0; a < 3; a++) t[a] = P.n1[a];
  t[3] = P.px;
  t[4] = P.wy;
  t[5] = P.wz;
}

void fft_plan_free(FftPlan &P) {
  AxisPlan *axes[3] = {&P.ax, &P.ay, &P.az};
  for (AxisPlan *A : axes) {
    cudaFree(A->tw);
    for (int v = 0; v < AxisPlan::kSplits; v++) {
      A->mix[v] = nullptr;
      A->mix32[v] = nullptr;
    }
    A->tw = nullptr;
  }
}

// the handle's spectrum type has two-step register kernels of length n
static bool mix_any(const Handle *h, int n) {
  return h->fp32 ? mix_ops<float2>(n) != nullptr : mix_ops<double2>(n) != nullptr;
}

// pencils per CTA of the two-step kernels, t threads each.  Axes with factors
// 3 and 5 take the plan's tile width w; powers of two a 128-byte segment per
// row (x passes: 8 row pairs) and at least 64 threads (wider tiles and CTAs
// measured slower, see fft_mix.cuh)
static int mix_width(int n, int t, int seg, int w) {
  return pow2_axis(n) ? std::max(seg, (64 / t + 7) / 8 * 8) : w;
}

// two-step x pass in the spectrum type C2; real grids FP64, or float
// (ld.real32 / out32) in the merged evaluation of the FP32-convolution form
template <typename C2>
static int x_pass_mix(Handle *h, int nb, const void *const *rin, double2 *const *cout, double2 *const *cin,
                      void *const *rout, bool inverse, const BoxPair *box, const XLoad &ld, bool out32) {
  const FftPlan &P = h->fft;
  const AxisMix<C2> m = axis_mix<C2>(P.ax, P.n1[0]);
  XRegArgs<C2> a{};
  a.nxh = P.nxh;
  a.nrow = (long)P.ny * P.nz;
  a.scale = 1.0;
  a.tw = m.ta;
  a.tw2 = m.tb;
  a.box = inverse ? box : nullptr;
  a.boxp = inverse ? nullptr : box;
  a.ny = P.ny;
  a.nz = P.nz;
  a.ld = ld;
  for (int i = 0; i < nb; i++) {
    if (inverse) {
      a.cin[i] = reinterpret_cast<const C2 *>(cin[i]);
      a.rout[i] = rout[i];
    } else {
      a.rin[i] = rin[i];
      a.cout[i] = reinterpret_cast<C2 *>(cout[i]);
    }
  }
  return m.ops->x(h, a, nb, inverse, mix_width(P.nx, m.ops->tx, 8, P.px), out32);
}

// box (two-step kernels): C2R restricted to the rows of the force box, R2C of
// rows that are zero outside the impurity box
// rin / rout: double grids, or float grids when ld.real32 (R2C) / out32 (C2R)
static int x_pass_v(Handle *h, int n, const void *const *rin, double2 *const *cout, double2 *const *cin,
                    void *const *rout, bool inverse, const BoxPair *box, const XLoad &ld, bool out32) {
  const FftPlan &P = h->fft;
  const long nrow = (long)P.ny * P.nz;
  for (int b0 = 0; b0 < n; b0 += kMaxBatch) {
    const int nb = std::min(kMaxBatch, n - b0);
    const void *const *ri = rin ? rin + b0 : nullptr;
    double2 *const *co = cout ? cout + b0 : nullptr;
    double2 *const *ci = cin ? cin + b0 : nullptr;
    void *const *ro = rout ? rout + b0 : nullptr;
    if (mix_any(h, P.nx)) {
      if (h->fp32)
        HE4_TRY(x_pass_mix<float2>(h, nb, ri, co, ci, ro, inverse, box, ld, out32));
      else
        HE4_TRY(x_pass_mix<double2>(h, nb, ri, co, ci, ro, inverse, box, ld, out32));
      continue;
    }
    if (ld.op != XLOAD_PLAIN || ld.real32 || out32) {
      set_error("formed-on-load x pass needs a register-path axis length");
      return HE4_E_UNSUPPORTED;
    }
    if (h->fp32) {
      set_error("FP32 spectra need register-path axis lengths");
      return HE4_E_UNSUPPORTED;
    }
    XArgs a{};
    a.ax = P.ax;
    a.nxh = P.nxh;
    a.P = P.px;
    a.nrow = nrow;
    a.scale = 1.0;
    for (int i = 0; i < nb; i++) {
      if (inverse) {
        a.cin[i] = cin[b0 + i];
        a.rout[i] = static_cast<double *>(rout[b0 + i]);
      } else {
        a.rin[i] = static_cast<const double *>(rin[b0 + i]);
        a.cout[i] = cout[b0 + i];
      }
    }
    dim3 grid((unsigned)((nrow + 2 * P.px - 1) / (2 * P.px)), nb);
    if (inverse)
      k_fft_x_c2r<<<grid, kThreads, smem_x(P), h->stream>>>(a);
    else
      k_fft_x_r2c<<<grid, kThreads, smem_x(P), h->stream>>>(a);
    HE4_LAUNCHED(h);
  }
  return HE4_OK;
}

static int x_pass(Handle *h, int n, const double *const *rin, double2 *const *cout, double2 *const *cin,
                  double *const *rout, bool inverse, const BoxPair *box = nullptr) {
  const void *ri[64];
  void *ro[64];
  if (n > 64) {
    set_error("x pass of more than 64 fields");
    return HE4_E_ARG;
  }
  for (int i = 0; i < n; i++) {
    ri[i] = rin ? rin[i] : nullptr;
    ro[i] = rout ? rout[i] : nullptr;
  }
  return x_pass_v(h, n, rin ? ri : nullptr, cout, cin, rout ? ro : nullptr, inverse, box, XLoad(), false);
}

// two-step transform of strided pencils in the spectrum type C2
template <typename C2>
static int yz_mix(Handle *h, int nb, double2 *const *buf, int axis, bool inverse, const BoxPair *box) {
  const FftPlan &P = h->fft;
  const AxisMix<C2> m = axis_mix<C2>((axis == 1) ? P.ay : P.az, P.n1[axis]);
  MixYArgs<C2> a{};
  a.nxh = P.nxh;
  a.nother = (axis == 1) ? P.nz : P.ny;
  a.so = (axis == 1) ? (long)P.ny * P.nxh : P.nxh;
  a.sf = (axis == 1) ? (long)P.nxh : (long)P.ny * P.nxh;
  a.ta = m.ta;
  a.box = (axis == 1) ? box : nullptr;
  a.nz = P.nz;
  for (int i = 0; i < nb; i++) a.buf[i] = reinterpret_cast<C2 *>(buf[i]);
  const int w = mix_width((axis == 1) ? P.ny : P.nz, m.ops->t, 128 / sizeof(C2), (axis == 1) ? P.wy : P.wz);
  return m.ops->y(h, a, nb, inverse, w);
}

// in-place complex transform of every pencil along y (axis 1) or z (axis 2);
// box (y pass, two-step lengths): only pencils whose z lies in the force box
static int strided_pass(Handle *h, int n, double2 *const *buf, int axis, bool inverse,
                        const BoxPair *box = nullptr) {
  const FftPlan &P = h->fft;
  const int len = (axis == 1) ? P.ny : P.nz;
  for (int b0 = 0; b0 < n; b0 += kMaxBatch) {
    const int nb = std::min(kMaxBatch, n - b0);
    if (mix_any(h, len)) {
      if (h->fp32)
        HE4_TRY(yz_mix<float2>(h, nb, buf + b0, axis, inverse, box));
      else
        HE4_TRY(yz_mix<double2>(h, nb, buf + b0, axis, inverse, box));
      continue;
    }
    if (h->fp32) {
      set_error("FP32 spectra need register-path axis lengths");
      return HE4_E_UNSUPPORTED;
    }
    PencilMap map;
    map.nxh = P.nxh;
    map.nother = (axis == 1) ? P.nz : P.ny;
    map.so = (axis == 1) ? (long)P.ny * P.nxh : P.nxh;
    const long sf = (axis == 1) ? (long)P.nxh : (long)P.ny * P.nxh;
    const long total = (long)P.nxh * map.nother;
    if (axis == 1) {
      YArgs a{};
      a.ay = P.ay;
      map.W = P.wy;
      a.map = map;
      a.sf = sf;
      for (int i = 0; i < nb; i++) a.buf[i] = buf[b0 + i];
      dim3 grid((unsigned)((total + P.wy - 1) / P.wy), nb);
      if (inverse)
        k_fft_y<true><<<grid, kThreads, smem_yz(P.ny, P.wy), h->stream>>>(a);
      else
        k_fft_y<false><<<grid, kThreads, smem_yz(P.ny, P.wy), h->stream>>>(a);
      HE4_LAUNCHED(h);
    } else {
      for (int i = 0; i < nb; i++) {
        ZOp op{buf[b0 + i], buf[b0 + i], nullptr, 1.0, -1, inverse ? 2 : 1};
        HE4_TRY(fft_z_conv(h, 1, &op));
      }
    }
  }
  return HE4_OK;
}

int fft_y(Handle *h, int n, double2 *const *buf, bool inverse) { return strided_pass(h, n, buf, 1, inverse); }

int fft_r2c(Handle *h, int n, const double *const *in, double2 *const *out) {
  HE4_TRY(x_pass(h, n, in, out, nullptr, nullptr, false));
  HE4_TRY(fft_y(h, n, out, false));
  return HE4_OK;
}

// The x pass writes the row pairs that touch the impurity box's planes, the y pass
// transforms the planes of the force box, one more on either side.  Those two stay
// exact zeros through any number of in-place transforms: with odd ny the row that a
// pair shares with a plane beyond the box is the first or last of its plane, the
// row beside it in the pair is the last or first of the box's plane, and both are
// zero in `in`, since a box that comes within 2 m cells of a face in y is the whole
// grid (k_box_find).  A pair of zero rows transforms to zeros.
int fft_r2c_box(Handle *h, const double *in, double2 *out) {
  const FftPlan &P = h->fft;
  const double *ri[1] = {in};
  double2 *co[1] = {out};
  if (!mix_any(h, P.nx) || !mix_any(h, P.ny)) return fft_r2c(h, 1, ri, co);
  HE4_TRY(x_pass(h, 1, ri, co, nullptr, nullptr, false, h->box));
  return strided_pass(h, 1, co, 1, false, h->box);
}

int fft_r2c_load(Handle *h, int n, const void *const *in, double2 *const *out, const XLoad &ld) {
  HE4_TRY(x_pass_v(h, n, in, out, nullptr, nullptr, false, nullptr, ld, false));
  HE4_TRY(fft_y(h, n, out, false));
  return HE4_OK;
}

int fft_c2r_f32(Handle *h, int n, double2 *const *in, float *const *out) {
  void *ro[64];
  if (n > 64) {
    set_error("x pass of more than 64 fields");
    return HE4_E_ARG;
  }
  for (int i = 0; i < n; i++) ro[i] = out[i];
  HE4_TRY(fft_y(h, n, in, true));
  HE4_TRY(x_pass_v(h, n, nullptr, nullptr, in, ro, true, nullptr, XLoad(), true));
  return HE4_OK;
}

int fft_c2r(Handle *h, int n, double2 *const *in, double *const *out) {
  HE4_TRY(fft_y(h, n, in, true));
  HE4_TRY(x_pass(h, n, nullptr, nullptr, in, out, true));
  return HE4_OK;
}

int fft_c2r_box(Handle *h, int n, double2 *const *in, double *const *out) {
  HE4_TRY(strided_pass(h, n, in, 1, true, h->box));
  HE4_TRY(x_pass(h, n, nullptr, nullptr, in, out, true, h->box));
  return HE4_OK;
}

// kernel array of an operation in the spectrum type's real type
template <typename C2>
static const typename regfft::Re<C2>::type *kern_of(const Handle *h, const double *k);
template <>
const double *kern_of<double2>(const Handle *, const double *k) { return k; }
template <>
const float *kern_of<float2>(const Handle *h, const double *k) { return h->kern32(k); }

template <typename C2>
static const typename regfft::Re<C2>::type *dsym_of(const Handle *h);
template <>
const double *dsym_of<double2>(const Handle *h) { return h->dsym; }
template <>
const float *dsym_of<float2>(const Handle *h) { return h->dsym32; }

// two-step fused z pass: one job per output
template <typename C2>
static int zconv_mix(Handle *h, int n, const ZOp *ops) {
  const FftPlan &P = h->fft;
  const AxisMix<C2> m = axis_mix<C2>(P.az, P.n1[2]);
  MixZArgs<C2> a{};
  a.nxh = P.nxh;
  a.npid = P.nxh * P.ny;
  a.nx = P.nx;
  a.ny = P.ny;
  a.nz = P.nz;
  a.sf = (long)P.ny * P.nxh;
  a.dsym = dsym_of<C2>(h);
  a.ta = m.ta;
  a.tb = m.tb;
  a.box = h->box;
  auto job = [&](const ZOp &op) {
    return MixZJob<C2>{reinterpret_cast<const C2 *>(op.in), reinterpret_cast<C2 *>(op.out), nullptr,
                       kern_of<C2>(h, op.kern), op.coef, op.dsym_axis, op.boxz};
  };
  // the three derivatives of one convolution (the force field): D_x(kx) and
  // D_y(ky) are constant along a z pencil, so the x and y outputs are i D
  // times one shared transform
  auto gradient = [&](int i) {
    if (!h->zconv_share_xy || i + 3 > n) return false;
    for (int o = 0; o < 3; o++)
      if (ops[i + o].in != ops[i].in || ops[i + o].kern != ops[i].kern || ops[i + o].coef != ops[i].coef ||
          ops[i + o].boxz != ops[i].boxz || ops[i + o].dsym_axis != o)
        return false;
    return true;
  };
  auto launch = [&]() -> int {
    if (a.njob == 0) return HE4_OK;
    bool der = false;
    for (int i = 0; i < a.njob; i++) der = der || a.job[i].dsym_axis >= 0 || a.job[i].out2 || a.job[i].boxz;
    HE4_TRY(m.ops->zconv(h, a, der, mix_width(P.nz, m.ops->t, 128 / sizeof(C2), P.wz)));
    a.njob = 0;
    return HE4_OK;
  };
  for (int i = 0; i < n; i++) {
    if (ops[i].kern && !kern_of<C2>(h, ops[i].kern)) {
      set_error("no FP32 copy of a z-pass kernel");
      return HE4_E_ARG;
    }
    if (a.njob + 2 > kMixJobs) HE4_TRY(launch());
    if (gradient(i)) {
      MixZJob<C2> &xy = a.job[a.njob++] = job(ops[i]);
      xy.dsym_axis = -1;
      xy.out2 = reinterpret_cast<C2 *>(ops[i + 1].out);
      a.job[a.njob++] = job(ops[i + 2]);
      i += 2;
    } else {
      a.job[a.njob++] = job(ops[i]);
    }
  }
  return launch();
}

int fft_z_conv(Handle *h, int n, const ZOp *ops) {
  const FftPlan &P = h->fft;
  if (n <= 0) return HE4_OK;
  const bool plain = ops[0].mode != 0;
  const bool mo = mix_any(h, P.nz);
  if (mo && !plain) return h->fp32 ? zconv_mix<float2>(h, n, ops) : zconv_mix<double2>(h, n, ops);
  if (mo) {
    for (int i = 0; i < n; i++) {
      double2 *b[1] = {ops[i].out};
      if (ops[i].out != ops[i].in) {
        set_error("plain z transforms are in place");
        return HE4_E_ARG;
      }
      HE4_TRY(strided_pass(h, 1, b, 2, ops[i].mode == 2));
    }
    return HE4_OK;
  }
  if (h->fp32) {
    set_error("FP32 spectra need register-path axis lengths");
    return HE4_E_UNSUPPORTED;
  }
  for (int b0 = 0; b0 < n; b0 += kMaxBatch) {
    int nb = std::min(kMaxBatch, n - b0);
    ZArgs a{};
    a.az = P.az;
    a.map.nxh = P.nxh;
    a.map.nother = P.ny;
    a.map.W = P.wz;
    a.map.so = P.nxh;
    a.sf = (long)P.ny * P.nxh;
    a.nx = P.nx;
    a.ny = P.ny;
    a.nz = P.nz;
    a.dsym = h->dsym;
    for (int i = 0; i < nb; i++) a.ops[i] = ops[b0 + i];
    long total = (long)P.nxh * P.ny;
    dim3 grid(nb, (unsigned)((total + P.wz - 1) / P.wz));
    k_fft_z_conv<<<grid, kThreads, smem_yz(P.nz, P.wz), h->stream>>>(a);
    HE4_LAUNCHED(h);
  }
  return HE4_OK;
}

template <typename C2>
static int zsum_mix(Handle *h, int nterm, const ZTerm *terms, double2 *out) {
  const FftPlan &P = h->fft;
  const AxisMix<C2> m = axis_mix<C2>(P.az, P.n1[2]);
  MixZSumArgs<C2> a{};
  a.npid = P.nxh * P.ny;
  a.sf = (long)P.ny * P.nxh;
  a.ta = m.ta;
  a.tb = m.tb;
  a.box = h->box;
  a.nz = P.nz;
  a.nterm = nterm;
  for (int j = 0; j < nterm; j++) {
    a.t[j] = ZTermT<C2>{reinterpret_cast<const C2 *>(terms[j].in), kern_of<C2>(h, terms[j].kern), terms[j].coef,
                        terms[j].boxed};
    if (!a.t[j].kern) {
      set_error("z-pass sum term without a kernel");
      return HE4_E_ARG;
    }
  }
  a.out = reinterpret_cast<C2 *>(out);
  return m.ops->zsum(h, a, mix_width(P.nz, m.ops->t, 128 / sizeof(C2), P.wz));
}

bool fft_energy_ok(const Handle *h) { return mix_ops<double2>(h->fft.nz) != nullptr; }
int fft_energy(Handle *h, double *part, int *ctas) {
  const FftPlan &P = h->fft;
  const AxisMix<double2> m = axis_mix<double2>(P.az, P.n1[2]);
  MixZEnergyArgs a{};
  a.nxh = P.nxh;
  a.npid = P.nxh * P.ny;
  a.nx = P.nx;
  a.nz = P.nz;
  a.sf = (long)P.ny * P.nxh;
  a.ta = m.ta;
  a.box = h->box;
  a.den = h->spec[0];
  a.denx = h->spec[4];
  a.k1 = h->fvlj4;
  a.k2 = h->vq;
  a.part = part;
  return m.ops->zenergy(h, a, h->fp32 != 0, mix_width(P.nz, m.ops->t, 8, P.wz), ctas);
}

// the merged evaluation: a z pass that sums convolutions, and x passes that
// form their sources on load
bool fft_z_sum_ok(const Handle *h) {
  const FftPlan &P = h->fft;
  return mix_any(h, P.nz) && mix_any(h, P.nx);
}

int fft_z_sum(Handle *h, int nterm, const ZTerm *terms, double2 *out) {
  if (nterm < 1 || nterm > kMaxTerms || !fft_z_sum_ok(h)) {
    set_error("fft_z_sum: %d terms, z length %d", nterm, h->fft.nz);
    return HE4_E_ARG;
  }
  return h->fp32 ? zsum_mix<float2>(h, nterm, terms, out) : zsum_mix<double2>(h, nterm, terms, out);
}

int fft_z_only(Handle *h, double2 *buf, bool inverse) {
  ZOp op{buf, buf, nullptr, 1.0, -1, inverse ? 2 : 1};
  return fft_z_conv(h, 1, &op);
}

// the inverse x pass alone with float output rows (FP32-convolution form)
int fft_x_c2r_f32_only(Handle *h, const double2 *cin, float *rout) {
  double2 *ci[1] = {const_cast<double2 *>(cin)};
  void *ro[1] = {rout};
  return x_pass_v(h, 1, nullptr, nullptr, ci, ro, true, nullptr, XLoad(), true);
}

int fft_x_only(Handle *h, const double *rin, double2 *cout, const double2 *cin, double *rout, bool inverse) {
  const double *ri[1] = {rin};
  double2 *co[1] = {cout};
  double2 *ci[1] = {const_cast<double2 *>(cin)};
  double *ro[1] = {rout};
  return x_pass(h, 1, ri, co, ci, ro, inverse);
}

}  // namespace he4
