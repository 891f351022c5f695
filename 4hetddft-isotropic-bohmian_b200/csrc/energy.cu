// energy.cu -- energy() (energy.f90:12-129).
//
// The convolution energies of delj4 and uimp (energy.f90's elj4 and eHeX) are
// summed in k space from the x/y spectra that every evaluation keeps
// (k_mix_zenergy), so a merged evaluation's missing delj4 and uimp are not
// computed for them; k_energy evaluates the first derivatives of psi and the
// other grid sums per CTA.  Up to 32 CTAs then add the per-CTA partials in a fixed
// order, and the host combines the sums with the formulas of energy.f90:374-407.
// The gradients and alpha_s integrals of ealphas are FP64 grids in both forms
// (field_alpha_fp64).  256^3, per call: split evaluation and one sum kernel 4.9 ms
// (FP64) and 3.8 ms (FP32 form) before, 1.0 and 1.7 here (0.7 of the latter for
// those grids).
#include <algorithm>

#include "common.cuh"
#include "reduce.cuh"
#include "stencil.cuh"

namespace he4 {

struct EArgs {
  double aux1, aux2, beta, den_m, den0s;
  int otc;
};

constexpr int kESums = 7;  // ekin4, ecor4, ealphas, esolid, ekinqx, elj4, eHeX

// T: the type of the evaluation's dencg and denalf (float: results of FP32
// transforms, which a wider grid would hold unchanged).  CONV: elj4 and eHeX from
// delj4 and uimp (z lengths without the k-space form).
template <typename T, bool CONV>
__global__ void k_energy(const double2 *__restrict__ psi, const double *__restrict__ den, const T *__restrict__ dencg,
                         const T *__restrict__ denalf, const double *__restrict__ dx, const double *__restrict__ dy,
                         const double *__restrict__ dz, const double *__restrict__ i0, const double *__restrict__ i1,
                         const double *__restrict__ i2, const double *__restrict__ psix,
                         const double *__restrict__ hpsix, const double *__restrict__ delj4,
                         const double *__restrict__ uimp, const BoxPair *__restrict__ bp, double *part, size_t stride,
                         Stencil st, Geo g, EArgs a) {
  __shared__ double sh[32];
  const int i = blockIdx.x * 32 + threadIdx.x;
  const int j = blockIdx.y * 8 + threadIdx.y;
  const int k = blockIdx.z;
  double v[kESums] = {0, 0, 0, 0, 0, 0, 0};
  if (i < g.nx && j < g.ny) {
    const size_t t = ((size_t)k * g.ny + j) * g.nx + i;
    const double2 d1 = stencil_axis_c(psi, st, 1, g, i, j, k, 0);
    const double2 d2 = stencil_axis_c(psi, st, 1, g, i, j, k, 1);
    const double2 d3 = stencil_axis_c(psi, st, 1, g, i, j, k, 2);
    v[0] = (d1.x * d1.x + d1.y * d1.y) + (d2.x * d2.x + d2.y * d2.y) + (d3.x * d3.x + d3.y * d3.y);
    const double dn = den[t], dc = (double)dencg[t];
    v[1] = dn * dc * dc * (a.aux1 + a.aux2 * dc);
    if (a.otc) v[2] = (1.0 - (double)denalf[t] / a.den0s) * (dx[t] * i0[t] + dy[t] * i1[t] + dz[t] * i2[t]);
    v[3] = dn * (1.0 + tanh(a.beta * (dn - a.den_m)));
    const Box b = bp->cur;  // psix is zero outside the particle box
    if (b.full || (!b.empty && k >= b.lo[2] && k <= b.hi[2] && j >= b.lo[1] && j <= b.hi[1] && i >= b.lo[0] &&
                   i <= b.hi[0]))
      v[4] = psix[t] * hpsix[t];
    if (CONV) {
      v[5] = delj4[t] * dn;
      v[6] = uimp[t] * dn;
    }
  }
  const size_t b = ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
#pragma unroll
  for (int q = 0; q < (CONV ? kESums : 5); q++) {
    const double s = block_sum(v[q], sh);
    if (threadIdx.x == 0 && threadIdx.y == 0) part[q * stride + b] = s;
  }
}

__global__ void __launch_bounds__(kPartThreads) k_sumsq(const double *__restrict__ x, int n, GridRed *gr, double *out) {
  __shared__ double sh[kPartThreads / 32 + 1];
  double acc[1] = {0.0}, tot[1];
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) acc[0] += x[t] * x[t];
  if (grid_sums_last<1>(acc, gr->part, &gr->count[3], sh, tot) && threadIdx.x == 0) *out = tot[0];
}

int compute_energy(Handle *h, he4_energies *E) {
  const Geo g{h->nx, h->ny, h->nz, zpad_of(h->p.icon)};
  const he4_params &p = h->p;
  EArgs a;
  a.aux1 = 0.5 * p.cp4;
  a.aux2 = (1.0 / 3.0) * p.cpp4;
  a.beta = p.beta_solid;
  a.den_m = p.den_m;
  a.den0s = p.den0s;
  a.otc = (p.core4 == HE4_CORE_OTC);
  dim3 gr = grid3(g);
  const size_t nb = (size_t)gr.x * gr.y * gr.z;
  // the red workspace holds 8 nb: kESums sums of nb CTAs, or five and the two
  // of the k-space pass ((nx/2 + 1) ny / 8 CTAs at most, under nb)
  const bool kspace = fft_energy_ok(h);
  int zb = 0;
  double *zpart = h->red + 5 * nb;
  if (kESums * nb > h->red_len || (kspace && 2 * (((size_t)h->nxh * h->ny + 7) / 8) > 3 * nb)) {
    set_error("reduction workspace too small");
    return HE4_E_STATE;
  }
  auto grids = [&](auto kern, auto *dencg, auto *denalf) {
    kern<<<gr, block3(), 0, h->stream>>>(h->psi, h->den, dencg, denalf, h->dxden, h->dyden, h->dzden, h->intx, h->inty,
                                         h->intz, h->psix, h->hpsix, h->delj4, h->uimp, h->box, h->red, nb, h->st, g,
                                         a);
  };
  if (!kspace) {
    grids(k_energy<double, true>, h->dencg, h->denalf);
  } else if (h->real32 && !h->split_valid) {  // the float grids of the merged evaluation
    if (a.otc) HE4_TRY(field_alpha_fp64(h));
    grids(k_energy<float, false>, h->g32[0], h->g32[1]);
  } else {
    grids(k_energy<double, false>, h->dencg, h->denalf);
  }
  HE4_LAUNCHED(h);
  if (kspace) {
    HE4_TRY(finalize_sums<5>(h, h->red, nb, (int)nb, 1.0, 1.0, h->scal + 16));
    HE4_TRY(fft_energy(h, zpart, &zb));
    HE4_TRY(finalize_sums<2>(h, zpart, zb, zb, h->renor, 1.0, h->scal + 16 + 5));
  } else {
    HE4_TRY(finalize_sums<kESums>(h, h->red, nb, (int)nb, 1.0, 1.0, h->scal + 16));
  }
  const int n3 = 3 * h->npar;
  k_sumsq<<<std::max(1, std::min(kPartMaxCta, (n3 + kPartThreads - 1) / kPartThreads)), kPartThreads, 0, h->stream>>>(
      h->vimp, n3, h->gred, h->scal + 16 + kESums);
  HE4_LAUNCHED(h);
  HE4_CUDA_TRY(cudaMemcpyAsync(h->hscal + 16, h->scal + 16, sizeof(double) * (kESums + 1), cudaMemcpyDeviceToHost,
                               h->stream));
  HE4_CUDA_TRY(cudaStreamSynchronize(h->stream));
  const double *s = h->hscal + 16;
  const double dxyz = h->dxyz;
  double ekin4 = p.h2o2m4 * s[0] * dxyz;
  double elj4 = 0.5 * s[5] * dxyz;
  double ecor4 = s[1] * dxyz;
  double ealphas = 0.0;
  if (a.otc) ealphas = -p.h2o2m4 * 0.5 * p.alphas * s[2] * dxyz;
  double esolid = p.c_solid * s[3] * dxyz;
  double etot4 = ekin4 + elj4 + ecor4 + esolid;
  if (a.otc) etot4 += ealphas;
  double ekinx = 0.5 * h->mAg_u * s[7] / h->npar;
  double ekinqx = s[4] * dxyz;
  double eHeX = s[6] * dxyz;
  double eimpu = ekinx + eHeX + ekinqx;
  E->etot = etot4 + eimpu;
  E->etot4 = etot4;
  E->ekin4 = ekin4;
  E->elj4 = elj4;
  E->ecor4 = ecor4;
  E->ealphas = ealphas;
  E->esolid = esolid;
  E->ekinx = ekinx;
  E->ekinqx = ekinqx;
  E->eHeX = eHeX;
  E->eimpu = eimpu;
  return HE4_OK;
}

}  // namespace he4
