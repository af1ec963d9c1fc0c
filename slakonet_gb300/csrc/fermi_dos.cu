// Fermi level, band-gap statistics and Gaussian DOS, one cluster per structure.
//
// Fermi level.  The reference iterates mu <- mu - L / (dL/dmu + 1e-12) on
// L = (2 sum_k w_k sum_b f(e_kb; mu, kT) - Ne)^2 from mu0 = mean(e), with
// f = 1/(exp((e - mu)/kT) + 1) and dL/dmu taken by autograd, stopping once
// |dL/dmu| < tol or after max_iter updates (slakonet/fermi.py:139-215).
// Autograd's derivative of that expression is
//   dL/dmu = 2 (N - Ne) * 2 sum w f^2 exp(x) / kT,
// which is NaN as soon as one exp(x) overflows (0 * inf); the kernel keeps
// that product so divergent cases end in NaN exactly where the reference's do.
//
// Gap statistics follow calculate_band_gap (slakonet/main.py:637-707),
// calculate_band_structure_properties (slakonet/main.py:1539-1642) and the
// get_fermi extras (slakonet/optim.py:1011-1060); H2E = 27.211 eV/Ha
// (slakonet/main.py:34).
//
// DOS.  dos(E) = sum_k w_k sum_b exp(-((E - (e_kb - mu) H2E)/sigma)^2 / 2)
// / (sigma sqrt(2 pi)) on the torch.linspace grid (slakonet/main.py:709-797).
// A window keeps, for each grid point, the bands within `window_sigmas` sigma.
#include "exact_round.cuh"
#include "gauss_sum.cuh"
#include "skn_common.cuh"

namespace {

constexpr double H2E = 27.211;
constexpr int NT = 256;

// stats layout (SKN_NSTAT doubles per structure)
enum {
  ST_MU_HA = 0, ST_FERMI_EV = 1, ST_GAP_EV = 2, ST_VBM_EV = 3, ST_CBM_EV = 4, ST_DIRECT = 5,
  ST_VBM_K = 6, ST_CBM_K = 7, ST_VWIDTH = 8, ST_CWIDTH = 9, ST_MIN_DGAP = 10, ST_DIRECT_SEMI = 11,
  ST_EFERMI_EV = 12, ST_BANDGAP_EV = 13, ST_CONVERGED = 14, ST_ITERS = 15, ST_DOS_FERMI = 16,
  ST_DOS_GAPC = 17, ST_DOS_TOTAL = 18, ST_METAL = 19, ST_FALLBACK = 20, ST_VBM_FLAT = 21, ST_CBM_FLAT = 22,
  ST_BAND_ENERGY = 23
};

__device__ __forceinline__ double qnan() { return __longlong_as_double(0x7ff8000000000000LL); }

// block reductions for 2 sums
__device__ __forceinline__ void block_sum2(double& a, double& b, double* red) {
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) { red[w] = a; red[nw + w] = b; }
  __syncthreads();
  a = 0.0; b = 0.0;
  for (int i = 0; i < nw; ++i) { a += red[i]; b += red[nw + i]; }
}

// block max/min with first flat index of the extreme (ties: smallest index)
__device__ __forceinline__ void block_argext(double& v, int& idx, bool is_max, double* redv, int* redi) {
  for (int o = 16; o > 0; o >>= 1) {
    double ov = __shfl_xor_sync(0xffffffffu, v, o);
    int oi = __shfl_xor_sync(0xffffffffu, idx, o);
    bool take = is_max ? (ov > v || (ov == v && oi < idx)) : (ov < v || (ov == v && oi < idx));
    if (take) { v = ov; idx = oi; }
  }
  const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) { redv[w] = v; redi[w] = idx; }
  __syncthreads();
  v = redv[0]; idx = redi[0];
  for (int i = 1; i < nw; ++i) {
    bool take = is_max ? (redv[i] > v || (redv[i] == v && redi[i] < idx)) : (redv[i] < v || (redv[i] == v && redi[i] < idx));
    if (take) { v = redv[i]; idx = redi[i]; }
  }
}

// Extremes and sums of one CTA's share of a structure, combined over the cluster in rank order.
struct GapPart {
  double be, vbm, cbm, vmax, vmin, cmax, cmin, dgap, gv, gc;
  int vbi, cbi, metal, nocc, nunocc;
};

SKN_DEVINL void take_max(double& v, int& i, double ov, int oi) {
  if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}
SKN_DEVINL void take_min(double& v, int& i, double ov, int oi) {
  if (ov < v || (ov == v && oi < i)) { v = ov; i = oi; }
}
SKN_DEVINL void combine(GapPart& a, const GapPart& o) {
  a.be += o.be;
  take_max(a.vbm, a.vbi, o.vbm, o.vbi);
  take_min(a.cbm, a.cbi, o.cbm, o.cbi);
  a.vmax = fmax(a.vmax, o.vmax);
  a.vmin = fmin(a.vmin, o.vmin);
  a.cmax = fmax(a.cmax, o.cmax);
  a.cmin = fmin(a.cmin, o.cmin);
  a.dgap = fmin(a.dgap, o.dgap);
  a.gv = fmax(a.gv, o.gv);
  a.gc = fmin(a.gc, o.gc);
  a.metal |= o.metal;
  a.nocc |= o.nocc;
  a.nunocc |= o.nunocc;
}
SKN_DEVINL GapPart shfl_part(const GapPart& a, int o) {
  GapPart r;
  r.be = __shfl_down_sync(0xffffffffu, a.be, o);
  r.vbm = __shfl_down_sync(0xffffffffu, a.vbm, o);
  r.cbm = __shfl_down_sync(0xffffffffu, a.cbm, o);
  r.vmax = __shfl_down_sync(0xffffffffu, a.vmax, o);
  r.vmin = __shfl_down_sync(0xffffffffu, a.vmin, o);
  r.cmax = __shfl_down_sync(0xffffffffu, a.cmax, o);
  r.cmin = __shfl_down_sync(0xffffffffu, a.cmin, o);
  r.dgap = __shfl_down_sync(0xffffffffu, a.dgap, o);
  r.gv = __shfl_down_sync(0xffffffffu, a.gv, o);
  r.gc = __shfl_down_sync(0xffffffffu, a.gc, o);
  r.vbi = __shfl_down_sync(0xffffffffu, a.vbi, o);
  r.cbi = __shfl_down_sync(0xffffffffu, a.cbi, o);
  r.metal = __shfl_down_sync(0xffffffffu, a.metal, o);
  r.nocc = __shfl_down_sync(0xffffffffu, a.nocc, o);
  r.nunocc = __shfl_down_sync(0xffffffffu, a.nunocc, o);
  return r;
}

// One cluster of FCL CTAs per structure.  The search is a chain of up to max_iter full sums, and an occupation
// costs ~30 FP64 instructions (two per clock and SM), so one CTA's SM bounded it: 512 k-points x 18 bands took
// 1.4 ms, 48 primitive cells of ~500 k-points 11 ms.  The eigenvalues are dealt to as many CTAs as there are
// blocks of 256 (a rule on the structure alone); every CTA leaves its two sums in the others' shared memory,
// alternating between two slots, so an iteration has one cluster barrier, and every CTA adds the slots in
// the same tree and takes the same step.  States more than FULL_X kT below or above mu are full or empty to the last
// bit; integer compares tell them, and only the states near mu, packed by the CTA in a fixed order, take an
// exponential.  Sums and the step are one warp's work.  The two cases: 0.42 and 3.1 ms with every state evaluated,
// 0.33 and 2.1 ms now.  Quotients by kT and the step's keep the rounding of a division (plain products with a rounded
// reciprocal were 6% faster, and 2% further from extended precision).  Registers for four CTAs an SM: at three the many
// structures of a batch take 15% longer.
constexpr int FCL = 16;
constexpr int F_BLOCK = 256;
constexpr int NEAR = 4 * NT;               // states a CTA looks at between two barriers
constexpr double FULL_X = 64.0;            // exp(-64) = 1.6e-28: 1 / (1 + exp(-x)) is 1 and exp(-x) nothing beside it

// Orders doubles by their high words; equal keys say nothing. -inf has KEY_MINUS_INF, negative NaNs lie below it and
// positive ones above every threshold.
constexpr int KEY_MINUS_INF = INT_MIN + 0x000fffff;
SKN_DEVINL int order_key(double v) {
  const int h = __double2hiint(v);
  return h ^ ((h >> 31) & 0x7fffffff);
}

__global__ void __launch_bounds__(NT, 4)
    k_fermi_gap(const int64_t* __restrict__ eig_off, const int32_t* __restrict__ nkv, const int32_t* __restrict__ nbv,
                const int64_t* __restrict__ kw_off, const double* __restrict__ kweights, const double* __restrict__ nelec,
                const double* __restrict__ eigall, double kT, double tol, int max_iter, double* __restrict__ mu_out,
                double* __restrict__ stats, int32_t* __restrict__ status) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ double red[2][NT / 32];
  __shared__ double slots[2][FCL][2];
  __shared__ double s_mu, near_e[NEAR], near_w[NEAR];
  __shared__ int s_edge[3], s_near[NT / 32], s_stop;
  __shared__ GapPart wpart[NT / 32];
  __shared__ GapPart cpart;
  const int s = blockIdx.x / FCL, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = (int)cl.block_rank();
  const int nk = nkv[s], nb = nbv[s];
  const int tot = nk * nb;
  const int ranks = min(FCL, max(1, (tot + F_BLOCK - 1) / F_BLOCK));
  if (rank >= ranks) return;           // its shared memory is never addressed, and barriers do not wait for it
  const double* E = eigall + eig_off[s];
  const double* w = kweights + kw_off[s];
  const double ne = nelec[s];
  const int stride = NT * ranks, e0 = rank * NT + tid;
  const int dk = nb > 0 ? stride / nb : 0, db = nb > 0 ? stride - dk * nb : 0;
  const int k0 = nb > 0 ? e0 / nb : 0, b0 = nb > 0 ? e0 - k0 * nb : 0;
  int turn = 0;

  // sums of a and b over the structure, the same bits in every CTA; in warp 0 alone
  auto total2 = [&](double& a, double& b) {
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane == 0) {
      red[0][warp] = a;
      red[1][warp] = b;
    }
    __syncthreads();
    if (warp == 0) {
      a = red[0][lane & (NT / 32 - 1)];
      b = red[1][lane & (NT / 32 - 1)];
      for (int o = NT / 64; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
      }
    }
    if (ranks > 1) {
      if (tid < ranks) {
        double* to = cl.map_shared_rank(&slots[turn][0][0], tid) + 2 * rank;
        to[0] = a;
        to[1] = b;
      }
      cl.sync();
      if (warp == 0) {
        a = lane < ranks ? slots[turn][lane][0] : 0.0;
        b = lane < ranks ? slots[turn][lane][1] : 0.0;
        for (int o = FCL / 2; o > 0; o >>= 1) {
          a += __shfl_xor_sync(0xffffffffu, a, o);
          b += __shfl_xor_sync(0xffffffffu, b, o);
        }
      }
      turn ^= 1;
    }
  };
  const bool plain_kT = kT > 1e-290 && kT < 1e290;      // in the range of its reciprocal
  // the next mu and the energies beyond which a state is full or empty to the last bit, for all threads
  auto publish = [&](double m, int stop) {
    if (tid == 0) {
      s_mu = m;
      s_stop = stop;
      const bool usable = fabs(m) < 1e300 && plain_kT;
      s_edge[0] = usable ? order_key(m - FULL_X * kT) : INT_MIN;
      s_edge[1] = usable ? order_key(m + FULL_X * kT) : INT_MAX;
      s_edge[2] = usable ? order_key(m + 700.0 * kT) : INT_MIN;
    }
    __syncthreads();
  };
  if (ranks > 1) cl.sync();            // every CTA's shared memory is there before the first remote store

  // mu0 = mean(e)
  double a = 0.0, b = 0.0;
  for (int e = e0; e < tot; e += stride) a += E[e];
  total2(a, b);
  publish(a / (double)tot, 0);
  const SknRecip by_kT = skn_recip(kT);
  int iters = max_iter, conv = 0;
  // this thread's states of one trip, kept over the iterations when one trip takes them all
  double ev[NEAR / NT], wv[NEAR / NT];
  const bool single = tot <= (int64_t)(NEAR / NT) * stride;
  for (int it = 0; it < max_iter; ++it) {
    const double mu = s_mu;
    const int below = s_edge[0], above = s_edge[1], top = s_edge[2];
    const bool usable = top != INT_MIN;          // no diverged search: mu is finite
    double sumo = 0.0, sumg = 0.0;
    int k = k0, bb = b0;
    for (int64_t base = rank * NT; base < tot; base += (int64_t)(NEAR / NT) * stride) {      // the same trips for every thread
      unsigned near[NEAR / NT];
      int mine = 0;
#pragma unroll
      for (int u = 0; u < NEAR / NT; ++u) {
        const int64_t e = base + tid + (int64_t)u * stride;
        bool slow = false;
        if (e < tot) {
          if (it == 0 || !single) {
            ev[u] = E[e];
            wv[u] = w[k];
          }
          const int key = order_key(ev[u]);
          if (key < below && key >= KEY_MINUS_INF) sumo += wv[u];
          else slow = !(key > above && key < top);
        }
        near[u] = __ballot_sync(0xffffffffu, slow);
        mine += __popc(near[u]);
        k += dk;
        bb += db;
        if (bb >= nb) { bb -= nb; ++k; }
      }
      if (lane == 0) s_near[warp] = mine;
      __syncthreads();
      int at = 0, count = 0;
      for (int q = 0; q < NT / 32; ++q) {
        if (q < warp) at += s_near[q];
        count += s_near[q];
      }
#pragma unroll
      for (int u = 0; u < NEAR / NT; ++u) {
        if (near[u] >> lane & 1) {
          const int to = at + __popc(near[u] & ((1u << lane) - 1));
          near_e[to] = ev[u];
          near_w[to] = wv[u];
        }
        at += __popc(near[u]);
      }
      __syncthreads();
      for (int q = tid; q < count; q += NT) {
        const double wk = near_w[q];
        const double d = near_e[q] - mu;
        const double t3 = exp(usable ? skn_over(d, by_kT) : plain_kT ? skn_quotient(d, kT, by_kT.hi) : d / kT);
        const double occ = 1.0 / (t3 + 1.0);
        sumo = fma(occ, wk, sumo);
        sumg += ((wk * occ) * occ) * t3;
      }
    }
    total2(sumo, sumg);
    const double total = 2.0 * sumo;
    const double diff = total - ne;
    const double loss = diff * diff;
    const double slope = (2.0 * (2.0 * diff)) * sumg;
    const double grad = usable ? skn_over(slope, by_kT) : slope / kT;
    const bool done = fabs(grad) < tol;
    const double y = grad + 1e-12;
    publish(done ? mu : mu - skn_quotient(loss, y, 1.0 / y), done);
    if (s_stop) { iters = it; conv = 1; break; }
  }
  const double mu = s_mu;

  GapPart P;
  P.be = 0.0;
  P.vbm = P.vmax = P.cmax = P.gv = -INFINITY;
  P.cbm = P.vmin = P.cmin = P.dgap = P.gc = INFINITY;
  P.vbi = P.cbi = 0x7fffffff;
  P.metal = P.nocc = P.nunocc = 0;
  const double kT_e = 0.025 / H2E, inv_kT_e = 1.0 / kT_e;
  const double f_ev = mu * H2E;
  for (int e = e0, k = k0, bb = b0; e < tot; e += stride) {
    const double Ee = E[e];
    // Fermi-smeared band energy, SimpleDftb._calculate_electronic_energy (slakonet/main.py:1430-1448):
    // sum_k w_k sum_b f(e_kb; mu, 0.025 eV) e_kb, with f = 0 where e_kb is exactly zero (fermi_smearing,
    // slakonet/fermi.py:54-96)
    const double occ = (Ee == 0.0) ? 0.0 : 1.0 / (1.0 + exp(skn_quotient(Ee - mu, kT_e, inv_kT_e)));
    P.be += (occ * Ee) * w[k];
    // calculate_band_gap
    const double ev = Ee * H2E;
    if (fabs(ev - f_ev) < 1e-3) P.metal = 1;
    if (ev < f_ev) { P.nocc = 1; take_max(P.vbm, P.vbi, ev, e); }
    if (ev >= f_ev) { P.nunocc = 1; take_min(P.cbm, P.cbi, ev, e); }
    // calculate_band_structure_properties on (e - mu) H2E
    const double rel = (Ee - mu) * H2E;
    if (rel < 0.0) { P.vmax = fmax(P.vmax, rel); P.vmin = fmin(P.vmin, rel); }
    if (rel >= 0.0) { P.cmax = fmax(P.cmax, rel); P.cmin = fmin(P.cmin, rel); }
    // get_fermi extras: occ = e <= mu, unocc = e > mu
    if (Ee <= mu) P.gv = fmax(P.gv, Ee);
    if (Ee > mu) P.gc = fmin(P.gc, Ee);
    k += dk;
    bb += db;
    if (bb >= nb) { bb -= nb; ++k; }
  }
  // smallest direct gap: a warp per k-point
  for (int k = rank * (NT / 32) + (tid >> 5); k < nk; k += ranks * (NT / 32)) {
    double kv = -INFINITY, kc = INFINITY;
    for (int bb = lane; bb < nb; bb += 32) {
      const double rel = (E[(int64_t)k * nb + bb] - mu) * H2E;
      if (rel < 0.0) kv = fmax(kv, rel);
      if (rel > 0.0) kc = fmin(kc, rel);
    }
    for (int o = 16; o > 0; o >>= 1) {
      kv = fmax(kv, __shfl_xor_sync(0xffffffffu, kv, o));
      kc = fmin(kc, __shfl_xor_sync(0xffffffffu, kc, o));
    }
    if (kv != -INFINITY && kc != INFINITY) P.dgap = fmin(P.dgap, kc - kv);
  }
  for (int o = 16; o > 0; o >>= 1) combine(P, shfl_part(P, o));
  if (lane == 0) wpart[tid >> 5] = P;
  __syncthreads();
  if (tid == 0) {
    for (int q = 1; q < NT / 32; ++q) combine(P, wpart[q]);
    cpart = P;
  }
  if (ranks > 1) cl.sync();
  if (rank == 0 && tid == 0) {
    for (int r = 1; r < ranks; ++r) combine(P, *cl.map_shared_rank(&cpart, r));
    double* st = stats + (int64_t)SKN_NSTAT * s;
    st[ST_BAND_ENERGY] = P.be;
    mu_out[s] = mu;
    const bool vfound = P.vmax != -INFINITY, cfound = P.cmin != INFINITY;
    const double bs_gap = (vfound && cfound) ? (P.cmin - P.vmax) : 0.0;
    st[ST_VWIDTH] = vfound ? (P.vmax - P.vmin) : 0.0;
    st[ST_CWIDTH] = cfound ? (P.cmax - P.cmin) : 0.0;
    const bool dfound = P.dgap != INFINITY;
    st[ST_MIN_DGAP] = dfound ? P.dgap : qnan();
    st[ST_DIRECT_SEMI] = dfound ? (fabs(bs_gap - P.dgap) < 0.01 ? 1.0 : 0.0) : 0.0;
    st[ST_CONVERGED] = conv;
    st[ST_ITERS] = iters;
    st[ST_METAL] = P.metal;
    const bool none = P.nocc == 0 || P.nunocc == 0;
    if (P.metal) {
      st[ST_MU_HA] = mu; st[ST_FERMI_EV] = mu * H2E; st[ST_GAP_EV] = 0.0;
      st[ST_VBM_EV] = f_ev; st[ST_CBM_EV] = f_ev; st[ST_DIRECT] = 0.0;
      st[ST_VBM_K] = 0; st[ST_CBM_K] = 0; st[ST_FALLBACK] = 0.0;
    } else if (none) {
      // the reference's empty max/min raises; get_properties_dict falls back to zeros
      st[ST_MU_HA] = 0.0; st[ST_FERMI_EV] = 0.0; st[ST_GAP_EV] = 0.0;
      st[ST_VBM_EV] = 0.0; st[ST_CBM_EV] = 0.0; st[ST_DIRECT] = 1.0;
      st[ST_VBM_K] = 0; st[ST_CBM_K] = 0; st[ST_FALLBACK] = 1.0;
    } else {
      st[ST_MU_HA] = mu; st[ST_FERMI_EV] = mu * H2E; st[ST_GAP_EV] = P.cbm - P.vbm;
      st[ST_VBM_EV] = P.vbm; st[ST_CBM_EV] = P.cbm;
      const int vk = P.vbi / nb, ck = P.cbi / nb;
      st[ST_DIRECT] = (vk == ck) ? 1.0 : 0.0;
      st[ST_VBM_K] = vk; st[ST_CBM_K] = ck; st[ST_FALLBACK] = 0.0;
    }
    st[ST_VBM_FLAT] = (P.metal || none) ? -1.0 : (double)P.vbi;
    st[ST_CBM_FLAT] = (P.metal || none) ? -1.0 : (double)P.cbi;
    st[ST_EFERMI_EV] = mu * H2E;
    const double bg = P.gc - P.gv;
    st[ST_BANDGAP_EV] = (bg > 0.0 ? bg : (bg == bg ? 0.0 : bg)) * H2E;
    status[s] = conv ? SKN_OK : SKN_ERR_NO_CONVERGE;
  }
  if (ranks > 1) cl.sync();            // rank 0 has read every part before its owner exits
}

// DOS of one structure on PTS grid points per cluster (gauss_sum.cuh).  A slice takes every 64th k-point, or,
// with fewer k-points than slices, every parts-th band of one k-point.  With a window the bands in reach of a
// tile are found by binary search (they ascend per k); without one every band is visited, and a lane whose
// points all lie beyond the underflow of the exponential skips it.
// 512 k-points x 18 bands on the 5000-point grid: 16.4 ms with one thread per grid point over all bands and
// one exponential per pair.
template <bool WINDOWED>
__global__ void __cluster_dims__(1, 1, skn_gauss::Z) __launch_bounds__(skn_gauss::THREADS)
    k_dos(const int64_t* __restrict__ eig_off, const int32_t* __restrict__ nkv, const int32_t* __restrict__ nbv,
          const int64_t* __restrict__ kw_off, const double* __restrict__ kweights, const double* __restrict__ eigall,
          const double* __restrict__ muv, double e_lo, double e_hi, int npts, double sigma, double window,
          double* __restrict__ grid, double* __restrict__ dos) {
  namespace sg = skn_gauss;
  __shared__ double part[sg::SL * sg::PTS], xg[sg::PTS];
  const int s = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int p0 = blockIdx.x * sg::PTS;
  const int nk = nkv[s], nb = nbv[s];
  const double* E = eigall + eig_off[s];
  const double* w = kweights + kw_off[s];
  const double mu = muv[s];
  const double inv_norm = 1.0 / (sigma * sqrt(2.0 * 3.141592653589793));
  sg::Lane L;
  const int i0 = p0 + lane * sg::DG;
  sg::cta_points(xg, p0, e_lo, e_hi, npts, 0.0);
  sg::lane_init(L, xg + lane * sg::DG, mu, e_lo, e_hi, npts, sigma, H2E, WINDOWED ? window : INFINITY);
  const int slice = blockIdx.z * sg::SL + warp;
  const int parts = max(1, sg::SLICES / max(nk, 1));
  const int part_id = slice % parts;
  if (i0 < npts && mu == mu) {
    // energies in reach of this tile, widened by far more than the rounding of the test
    const int t0 = p0 + (lane / sg::SUB) * sg::TP;
    const double reach = window * sigma * (1.0 + 1e-9);
    const double x0 = sg::lin_grid(e_lo, e_hi, npts, min(t0, npts - 1));
    const double x1 = sg::lin_grid(e_lo, e_hi, npts, min(t0 + sg::TP - 1, npts - 1));
    const double a_lo = mu + (fmin(x0, x1) - reach) / H2E, a_hi = mu + (fmax(x0, x1) + reach) / H2E;
    const double m_lo = a_lo - 1e-9 * (1.0 + fabs(a_lo)), m_hi = a_hi + 1e-9 * (1.0 + fabs(a_hi));
    for (int k = slice / parts; k < nk; k += sg::SLICES) {      // parts > 1: at most one k-point per slice
      const double* Ek = E + (int64_t)k * nb;
      const double wk = w[k] * inv_norm;
      int b = 0;
      if (WINDOWED) {
        int hi = nb;
        while (b < hi) {
          const int m = (b + hi) >> 1;
          if (Ek[m] < m_lo) b = m + 1; else hi = m;
        }
        if (parts > 1) b += (part_id - b % parts + parts) % parts;
      } else {
        b = part_id;
      }
      for (; b < nb; b += parts) {
        const double e = Ek[b];
        if (WINDOWED && e > m_hi) break;
        sg::add_band<WINDOWED>(L, e, wk);
      }
    }
  }
  double v = sg::cluster_total(L, part);
  if (blockIdx.z == 0) v = sg::at_grid(L, xg, v, e_lo, e_hi, npts, part);
  if (blockIdx.z == 0 && p0 + tid < npts) {
    if (s == 0) grid[p0 + tid] = xg[tid];
    dos[(int64_t)s * npts + p0 + tid] = mu == mu ? v : qnan();
  }
}

// dos_at_fermi (grid point closest to 0), gap centre (DOS minimum within |E| < 2 eV)
// and trapezoid integral, as get_properties_dict (slakonet/main.py:1766-1782).
constexpr int DS_NT = 512;

//
// In the middle of a gap of more than about 75 sigma the unwindowed DOS runs through the subnormal numbers to zero, and
// the minimum's place, the first point that is zero, hangs on the rounding of each term there. Those points (a sigma's
// width at each edge, and the zeros next to it) are therefore summed again term by term, exponential first, as the
// reference's expression is written; every other point keeps k_dos's value. A warp takes a point, a lane a k-point.
constexpr double SUBNORMAL_BELOW = 1e-307, GONE_T = 39.0;      // exp(-t^2 / 2) is zero past t = 38.7

__global__ void __launch_bounds__(DS_NT) k_dos_stats(const int64_t* __restrict__ eig_off, const int32_t* __restrict__ nkv,
                                                     const int32_t* __restrict__ nbv, const int64_t* __restrict__ kw_off,
                                                     const double* __restrict__ kweights, const double* __restrict__ eigall,
                                                     const double* __restrict__ muv, double sigma, int windowed,
                                                     const double* __restrict__ grid, double* dos, int npts,
                                                     double* __restrict__ stats) {
  __shared__ double red[2 * DS_NT / 32];
  __shared__ int redi[DS_NT / 32];
  __shared__ int again[DS_NT], n_again;
  const int s = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double* D = dos + (int64_t)s * npts;
  double av = INFINITY, mv = INFINITY, tr = 0.0, dummy = 0.0;
  int ai = 0x7fffffff, mi = 0x7fffffff;
  for (int i = tid; i < npts; i += DS_NT) {
    const double g = grid[i];
    const double ag = fabs(g);
    if (ag < av || (ag == av && i < ai)) { av = ag; ai = i; }
    if (ag < 2.0 && (D[i] < mv || (D[i] == mv && i < mi))) { mv = D[i]; mi = i; }
    if (i + 1 < npts) tr += (grid[i + 1] - g) * (D[i] + D[i + 1]) * 0.5;
  }
  block_argext(av, ai, false, red, redi);
  block_argext(mv, mi, false, red, redi);
  block_sum2(tr, dummy, red);
  if (mv < SUBNORMAL_BELOW && !windowed && npts > 1) {
    const int nk = nkv[s], nb = nbv[s];
    const double* E = eigall + eig_off[s];
    const double* w = kweights + kw_off[s];
    const double mu = muv[s], inv_sigma = 1.0 / sigma;
    const double inv_norm = 1.0 / (sigma * sqrt(2.0 * 3.141592653589793));
    const double step = fabs(grid[1] - grid[0]);
    const int reach = step > 0.0 && 0.2 * sigma < 64.0 * step ? 1 + (int)(0.2 * sigma / step) : 64;
    for (int base = 0; base < npts; base += DS_NT) {
      const int i = base + tid;
      if (tid == 0) n_again = 0;
      __syncthreads();
      if (i < npts && fabs(grid[i]) < 2.0 && D[i] < SUBNORMAL_BELOW) {
        bool take = D[i] != 0.0;
        for (int q = max(0, i - reach); q <= min(npts - 1, i + reach) && !take; ++q) take = D[q] != 0.0;
        if (take) again[atomicAdd(&n_again, 1)] = i;       // their order does not matter
      }
      __syncthreads();
      for (int c = warp; c < n_again; c += DS_NT / 32) {
        const int i0 = again[c];
        const double x = grid[i0];
        double acc = 0.0;
        for (int k0 = 0; k0 < nk; k0 += 32) {
          double sk = 0.0;
          const double wk = k0 + lane < nk ? w[k0 + lane] : 0.0;
          if (k0 + lane < nk) {
            const double* Ek = E + (int64_t)(k0 + lane) * nb;
            for (int b = 0; b < nb; ++b) {
              const double t = (x - (Ek[b] - mu) * H2E) * inv_sigma;
              if (fabs(t) < GONE_T) sk += exp(-0.5 * (t * t)) * inv_norm;
            }
          }
          for (unsigned any = __ballot_sync(0xffffffffu, sk != 0.0); any; any &= any - 1) {
            const int l = __ffs(any) - 1;
            acc = fma(__shfl_sync(0xffffffffu, wk, l), __shfl_sync(0xffffffffu, sk, l), acc);
          }
        }
        if (lane == 0) D[i0] = acc;
      }
      __syncthreads();
    }
    mv = INFINITY;
    mi = 0x7fffffff;
    for (int i = tid; i < npts; i += DS_NT)
      if (fabs(grid[i]) < 2.0 && (D[i] < mv || (D[i] == mv && i < mi))) { mv = D[i]; mi = i; }
    block_argext(mv, mi, false, red, redi);
  }
  if (tid == 0) {
    double* st = stats + (int64_t)SKN_NSTAT * s;
    st[ST_DOS_FERMI] = D[ai];
    st[ST_DOS_GAPC] = (mi < npts) ? grid[mi] : qnan();
    st[ST_DOS_TOTAL] = tr;
  }
}

}  // namespace

extern "C" int skn_fermi_gap(int n_struct, const int64_t* eig_off, const int32_t* nk, const int32_t* nb,
                             const int64_t* kw_off, const double* kweights, const double* nelec, const double* eig,
                             double kT, double tol, int max_iter, double* mu, double* stats, int32_t* status,
                             cudaStream_t stream) {
  if (n_struct < 0 || max_iter < 0 || !(kT > 0.0)) return SKN_ERR_ARG;
  if (n_struct == 0) return SKN_OK;
  if (!eig_off || !nk || !nb || !kw_off || !kweights || !nelec || !eig || !mu || !stats || !status)
    return SKN_ERR_ARG;
  if (n_struct > INT32_MAX / FCL) return SKN_ERR_CAPACITY;
  if (cudaFuncSetAttribute(k_fermi_gap, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return SKN_ERR_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)n_struct * FCL);
  cfg.blockDim = dim3(NT);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = FCL;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, k_fermi_gap, eig_off, nk, nb, kw_off, kweights, nelec, eig, kT, tol, max_iter, mu,
                         stats, status) != cudaSuccess)
    return SKN_ERR_CUDA;
  return cudaPeekAtLastError() == cudaSuccess ? SKN_OK : SKN_ERR_CUDA;
}

extern "C" int skn_dos(int n_struct, const int64_t* eig_off, const int32_t* nk, const int32_t* nb,
                       const int64_t* kw_off, const double* kweights, const double* eig, const double* mu,
                       double e_lo, double e_hi, int npts, double sigma, double window_sigmas, double* grid,
                       double* dos, double* stats, cudaStream_t stream) {
  if (n_struct < 0 || npts <= 0 || !(sigma > 0.0) || window_sigmas < 0.0) return SKN_ERR_ARG;
  if (n_struct == 0) return SKN_OK;
  if (!eig_off || !nk || !nb || !kw_off || !kweights || !eig || !mu || !grid || !dos || !stats) return SKN_ERR_ARG;
  if (n_struct > 65535) return SKN_ERR_CAPACITY;
  const dim3 g((npts + skn_gauss::PTS - 1) / skn_gauss::PTS, n_struct, skn_gauss::Z);
  if (window_sigmas > 0.0)
    k_dos<true><<<g, skn_gauss::THREADS, 0, stream>>>(eig_off, nk, nb, kw_off, kweights, eig, mu, e_lo, e_hi, npts,
                                                      sigma, window_sigmas, grid, dos);
  else
    k_dos<false><<<g, skn_gauss::THREADS, 0, stream>>>(eig_off, nk, nb, kw_off, kweights, eig, mu, e_lo, e_hi, npts,
                                                       sigma, 0.0, grid, dos);
  if (cudaPeekAtLastError() != cudaSuccess) return SKN_ERR_CUDA;
  k_dos_stats<<<n_struct, DS_NT, 0, stream>>>(eig_off, nk, nb, kw_off, kweights, eig, mu, sigma, window_sigmas > 0.0,
                                              grid, dos, npts, stats);
  return cudaPeekAtLastError() == cudaSuccess ? SKN_OK : SKN_ERR_CUDA;
}

extern "C" int skn_abi_version(void) { return 100; }
