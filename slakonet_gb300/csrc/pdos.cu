// Atom-type projected DOS from eigenvectors with Gaussian broadening.
//
// Replaces compute_atom_projected_dos (slakonet/predict_slakonet.py:119-210),
// which loops over (k, band) in Python.  Two launches:
//   k_pdos_weights  thread per (k, band): w[k][b][g] = sum_{i in group g} |c_ib|^2
//                   (rows i of the eigenvector matrix are read across
//                   consecutive bands, so warps load contiguous memory);
//   k_pdos          sum over (k, band) of
//                   w * exp(-0.5 ((E - e_kb) / sigma)^2) / (sigma sqrt(2 pi)),
//                   divided by nk, on the torch.linspace grid shifted by E_F.
#include "gauss_sum.cuh"
#include "skn_common.cuh"

namespace {

constexpr int PT = 128;

__global__ void __launch_bounds__(PT) k_pdos_weights(int nk, int nb, int n_orb, const double2* __restrict__ vec,
                                                     const int32_t* __restrict__ group, int n_group,
                                                     double* __restrict__ w) {
  const int64_t t = (int64_t)blockIdx.x * PT + threadIdx.x;
  if (t >= (int64_t)nk * nb) return;
  const int k = (int)(t / nb), b = (int)(t % nb);
  const double2* v = vec + (int64_t)k * n_orb * nb + b;
  for (int g = 0; g < n_group; ++g) {
    double s = 0.0;
    for (int i = 0; i < n_orb; ++i) {
      if (group[i] != g) continue;
      const double2 c = v[(int64_t)i * nb];
      s = __dadd_rn(s, __dadd_rn(__dmul_rn(c.x, c.x), __dmul_rn(c.y, c.y)));
    }
    w[t * n_group + g] = s;
  }
}

// PDOS of one atom type on PTS grid points per cluster (gauss_sum.cuh); slices as in the DOS.  The bands need
// no order.  64 k-points x 54 bands on 1000 points, 2 types: 4.3 ms with one thread per point.
__global__ void __cluster_dims__(1, 1, skn_gauss::Z) __launch_bounds__(skn_gauss::THREADS)
    k_pdos(int nk, int nb, const double* __restrict__ eig, const double* __restrict__ w, int n_group, double fermi_ev,
           double e_lo, double e_hi, int npts, double sigma, double h2e, double* __restrict__ grid,
           double* __restrict__ pdos) {
  namespace sg = skn_gauss;
  __shared__ double part[sg::SL * sg::PTS], xg[sg::PTS];
  const int g = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int p0 = blockIdx.x * sg::PTS, i0 = p0 + lane * sg::DG;
  sg::Lane L;
  sg::cta_points(xg, p0, e_lo, e_hi, npts, fermi_ev);
  sg::lane_init(L, xg + lane * sg::DG, 0.0, e_lo, e_hi, npts, sigma, h2e, INFINITY);
  const int slice = blockIdx.z * sg::SL + warp;
  const int parts = max(1, sg::SLICES / nk);
  if (i0 < npts) {
    for (int k = slice / parts; k < nk; k += sg::SLICES) {
      const int64_t kb = (int64_t)k * nb;
      for (int b = slice % parts; b < nb; b += parts) sg::add_band<false>(L, eig[kb + b], w[(kb + b) * n_group + g]);
    }
  }
  double v = sg::cluster_total(L, part);
  if (blockIdx.z == 0) v = sg::at_grid(L, xg, v, e_lo, e_hi, npts, part);
  if (blockIdx.z == 0 && p0 + tid < npts) {
    if (g == 0) grid[p0 + tid] = sg::lin_grid(e_lo, e_hi, npts, p0 + tid);
    const double norm = 1.0 / (sigma * sqrt(2.0 * 3.141592653589793));
    pdos[(int64_t)g * npts + p0 + tid] = v * norm / (double)nk;
  }
}

}  // namespace

extern "C" int skn_atom_pdos(int nk, int nb, int n_orb, const double* eig, const double* vec,
                             const int32_t* orb_group, int n_group, double fermi_ev, double e_lo, double e_hi,
                             int npts, double sigma, double h2e, double* weights, double* grid, double* pdos,
                             cudaStream_t stream) {
  if (nk < 0 || nb < 0 || n_orb < 0 || n_group < 1 || npts < 1 || !(sigma > 0.0)) return SKN_ERR_ARG;
  if (!eig || !vec || !orb_group || !weights || !grid || !pdos) return SKN_ERR_ARG;
  if (n_group > 65535) return SKN_ERR_CAPACITY;
  const int64_t nkb = (int64_t)nk * nb;
  if (nkb > 0) {
    k_pdos_weights<<<(unsigned)((nkb + PT - 1) / PT), PT, 0, stream>>>(nk, nb, n_orb, (const double2*)vec,
                                                                      orb_group, n_group, weights);
    if (cudaPeekAtLastError() != cudaSuccess) return SKN_ERR_CUDA;
  }
  const dim3 pg((npts + skn_gauss::PTS - 1) / skn_gauss::PTS, n_group, skn_gauss::Z);
  k_pdos<<<pg, skn_gauss::THREADS, 0, stream>>>(nk > 0 ? nk : 1, nkb > 0 ? nb : 0, eig, weights, n_group, fermi_ev,
                                                e_lo, e_hi, npts, sigma, h2e, grid, pdos);
  return cudaPeekAtLastError() == cudaSuccess ? SKN_OK : SKN_ERR_CUDA;
}
