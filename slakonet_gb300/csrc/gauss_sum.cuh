// Sums of Gaussians on a uniform energy grid: sum_b w_b exp(-((x_i - e_b) / sigma)^2 / 2), shared by the DOS
// and the atom-projected DOS.
//
// FP64 issue is the bound (two FMAs per clock and SM), so the work is counted in FP64 instructions.  Eight
// lanes hold 8 consecutive grid points each (one 64-point tile) and walk over bands: with t = (x_0 - e) / sigma
// at a lane's first point and d = step / sigma, the Gaussian at its point j is
//   exp(-t^2 / 2) exp(-t d)^j exp(-(j d)^2 / 2),
// so a band costs a lane two exponentials and two operations per point (a power and a fused add with the
// constant last factor) instead of one exponential (~20 FP64 instructions) per point.  Every term of the
// product is positive and the power's exponent is at most 7, so the result keeps its relative accuracy.
// Grids so coarse that the last factor would leave the normal range take one exponential per point.
//
// The powers stand at x_0 + j step; the grid's own points are rounded, up to 1e-15 eV away, which a Gaussian of width
// sigma answers with |t| times that over sigma: more than all other rounding.  At the end each point's sum is moved to
// the grid's point along its slope (at_grid).  Energies count from the Fermi level before they are scaled, as a sum with the
// level's own size would round.  Both together: 5000 points over 512 x 18 bands 0.47 to 0.49 ms, and errors below those of
// one exponential per point and band.
//
// A warp's four tiles are adjacent and read the same bands.  The bands of a structure are cut into 64 slices,
// eight per CTA and eight CTAs in a cluster; slice sums are added in slice order (shared memory, then
// distributed shared memory), so the result depends on the structure alone: not on the batch, and not on
// the order in which CTAs run.  One structure of the default 5000-point grid is 160 CTAs.
#pragma once
#include <cooperative_groups.h>

#include "skn_common.cuh"

namespace skn_gauss {
namespace {

constexpr int DG = 8;                       // grid points per lane
constexpr int SUB = 8;                      // lanes per tile
constexpr int TP = DG * SUB;                // points per tile
constexpr int CT = 32 / SUB;                // tiles per warp (and CTA)
constexpr int SL = 8;                       // slices (warps) per CTA
constexpr int Z = 8;                        // CTAs per cluster
constexpr int SLICES = SL * Z;
constexpr int THREADS = 32 * SL;
constexpr int PTS = TP * CT;                // points per CTA
static_assert(PTS == THREADS, "one thread per point in the final sums");
constexpr double FAR_T = 36.0;              // exp(-t^2/2) and its powers stay normal up to here
constexpr double ZERO_T = 38.8;             // beyond: exp(-t^2/2) is exactly zero
constexpr double MAX_T = 41.0;              // exp(-t^2/2) 2^230 and its powers stay normal up to here
constexpr int HI_INF = 0x7ff00000;          // high word of an infinity; a NaN's is no smaller

// torch.linspace grid: fma(step, i, lo) for the first half, fma(-step, n-1-i, hi) after.
SKN_DEVINL double lin_grid(double lo, double hi, int n, int i) {
  if (n == 1) return lo;
  const double step = (hi - lo) / (double)(n - 1);
  return (i < n / 2) ? fma(step, (double)i, lo) : fma(-step, (double)(n - 1 - i), hi);
}

// High word of |v|: orders magnitudes to 2^-20 relative without the FP64 pipe.
SKN_DEVINL int hi_abs(double v) { return __double2hiint(v) & 0x7fffffff; }

// Nearest integer of |v| < 2^31 by the magic-number addition (one FP64 instruction).
SKN_DEVINL int near_int(double v) { return __double2loint(v + 6755399441055744.0); }

struct Lane {
  double x0, e0;      // first point, eV, plus the shift; level that the energies count from
  const double* x;    // its points, as x0
  double d, inv_d;    // step / sigma, sigma / step
  double inv_sigma, scale;
  double window;      // in sigma; infinity: none
  double cl, ch;      // offsets of the first and last point index inside the window
  int hi_far, hi_zero, hi_max;
  bool fast, masked;
  double C[DG];       // exp(-(j d)^2 / 2)
  double acc[DG];
};

// The CTA's points from p0 on, plus an energy shift, into xg: all threads, ends in step.
SKN_DEVINL void cta_points(double* xg, int p0, double e_lo, double e_hi, int npts, double shift) {
  xg[threadIdx.x] = lin_grid(e_lo, e_hi, npts, min(p0 + (int)threadIdx.x, npts - 1)) + shift;
  __syncthreads();
}

// A lane's points x[0] .. x[DG - 1]; a band of energy E stands at (E - e0) scale.
SKN_DEVINL void lane_init(Lane& L, const double* x, double e0, double e_lo, double e_hi, int npts, double sigma,
                          double scale, double window) {
  L.x = x;
  L.x0 = x[0];
  L.e0 = e0;
  L.inv_sigma = 1.0 / sigma;
  L.scale = scale;
  L.d = npts > 1 ? (e_hi - e_lo) / (double)(npts - 1) * L.inv_sigma : 0.0;
  L.inv_d = L.d > 0.0 ? 1.0 / L.d : 0.0;
  L.window = window;
  L.hi_far = __double2hiint(FAR_T);
  L.hi_zero = __double2hiint(ZERO_T);
  L.hi_max = __double2hiint(MAX_T);
  // 1e-6 < d: the window's edge indices stay far inside 32 bits; 7 d <= 8: exp(-(7 d)^2 / 2) >= e^-32
  L.fast = L.d > 1e-6 && (DG - 1) * L.d <= 8.0;
  L.masked = L.fast && window + (DG - 1) * L.d <= FAR_T;
  // ceil and floor as nearest integers of the half-shifted index; 1e-9 of a step keeps a point on the edge in
  L.cl = -window * L.inv_d + (0.5 - 1e-9);
  L.ch = window * L.inv_d - (0.5 - 1e-9);
#pragma unroll
  for (int j = 0; j < DG; ++j) {
    const double u = (double)j * L.d;
    L.C[j] = L.fast ? exp(-0.5 * (u * u)) : 1.0;
    L.acc[j] = 0.0;
  }
}

// Adds one band of energy E (before scaling) and weight w to the lane's points.
template <bool WINDOWED>
SKN_DEVINL void add_band(Lane& L, double E, double w) {
  const double t = fma(L.e0 - E, L.scale, L.x0) * L.inv_sigma;
  const int ht = hi_abs(t);
  if (WINDOWED && L.masked) {
    if (ht >= HI_INF) return;                  // a NaN is outside every window
    const int jl = near_int(fma(t, -L.inv_d, L.cl)), jh = near_int(fma(t, -L.inv_d, L.ch));
    if (jl > DG - 1 || jh < 0) return;
    double g = exp(-0.5 * (t * t)) * w;
    const double q = exp(-t * L.d);
#pragma unroll
    for (int j = 0; j < DG; ++j) {
      if (j >= jl && j <= jh) L.acc[j] = fma(g, L.C[j], L.acc[j]);
      g *= q;
    }
    return;
  }
  const double te = fma((double)(DG - 1), L.d, t);
  // all points on one side of the band and beyond the underflow; an infinity or a NaN, also of the weight, is no zero:
  // its terms are formed
  const int he = hi_abs(te);
  if ((__double2hiint(t) ^ __double2hiint(te)) >= 0 && min(ht, he) > L.hi_zero && max(max(ht, he), hi_abs(w)) < HI_INF)
    return;
  if (L.fast && max(ht, he) < L.hi_max && (!WINDOWED || (fabs(t) <= L.window && fabs(te) <= L.window))) {
    // where the first factor would leave the normal range it is carried times 2^230, which leaves each term
    // as its last rounding
    const bool far = max(ht, he) >= L.hi_far;
    double g = exp(fma(-0.5 * t, t, far ? 230.0 * 0.6931471805599453 : 0.0)) * w;
    const double q = exp(-t * L.d);
    if (!far) {
#pragma unroll
      for (int j = 0; j < DG; ++j) {
        L.acc[j] = fma(g, L.C[j], L.acc[j]);
        g *= q;
      }
    } else {
#pragma unroll
      for (int j = 0; j < DG; ++j) {
        L.acc[j] = fma(g * 0x1p-230, L.C[j], L.acc[j]);
        g *= q;
      }
    }
    return;
  }
#pragma unroll 1
  for (int j = 0; j < DG; ++j) {
    // where no power is taken, the grid's own point
    const double tj = L.fast ? fma((double)j, L.d, t) : fma(L.e0 - E, L.scale, L.x[j]) * L.inv_sigma;
    const double g = (!WINDOWED || fabs(tj) <= L.window) ? exp(-0.5 * (tj * tj)) * w : 0.0;
#pragma unroll
    for (int i = 0; i < DG; ++i)
      if (i == j) L.acc[i] += g;
  }
}

// log2 of a positive normal number; far below it otherwise
SKN_DEVINL float log2_of(double v) {
  const int h = __double2hiint(v);
  if (h < 0x01000000 || h >= HI_INF) return -1e9f;
  const double m = __hiloint2double((h & 0xfffff) | 0x3ff00000, __double2loint(v));
  return (float)((h >> 20) - 1023) + log2f((float)m);
}
// The sum v of the CTA's point tid, formed at its lane's first point plus whole steps, at the grid's point: along the slope
// of its logarithm, from the points beside it (of one Gaussian that is a parabola, whose central difference is exact).
// All threads of the CTA; `part` is free.
SKN_DEVINL double at_grid(const Lane& L, const double* xg, double v, double e_lo, double e_hi, int npts, double* part) {
  const int tid = threadIdx.x, j = tid & (DG - 1);
  float* lg = reinterpret_cast<float*>(part);
  lg[tid] = log2_of(v);
  __syncthreads();
  if (!L.fast) return v;
  const int c = min(max(tid, 1), PTS - 2), side = tid - c;        // side: -1, 0 or 1 from the middle of three points
  const float a = lg[c - 1], m = lg[c], b = lg[c + 1];
  if (fminf(fminf(a, m), b) < -1e8f) return v;
  const float slope = 0.5f * (b - a) + (float)side * (a - 2.0f * m + b);          // per step
  const double step = (e_hi - e_lo) / (double)(npts - 1);
  const float off = (float)fma(-(double)j, step, xg[tid] - xg[tid - j]) / (float)step;
  return fma(v, (double)(0.6931472f * slope * off), v);
}

// Sum over the CTA's slices, then over the cluster's CTAs in rank order; the thread of point `tid` of rank 0
// gets the total (other ranks: unspecified).  `part` holds SL x PTS doubles.  Ends with the cluster in step.
SKN_DEVINL double cluster_total(const Lane& L, double* part) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll
  for (int j = 0; j < DG; ++j) part[warp * PTS + lane * DG + j] = L.acc[j];
  __syncthreads();
  double v = part[tid];
#pragma unroll
  for (int q = 1; q < SL; ++q) v += part[q * PTS + tid];
  __syncthreads();
  part[tid] = v;
  cl.sync();
  if (cl.block_rank() == 0) {
#pragma unroll
    for (int r = 1; r < Z; ++r) v += cl.map_shared_rank(part, r)[tid];
  }
  cl.sync();
  return v;
}

}  // namespace
}  // namespace skn_gauss
