// Eigenvectors of H x = e S x for problems whose values kernel kept the reflectors (lower triangle of H), tau, the
// tridiagonal (d, e) and L (lower triangle of S):
//   1. k_inverse: inverse iteration on T - e_j I (Gaussian elimination with partial pivoting on the tridiagonal, two
//      solves from a pseudo-random start), one thread per eigenvalue; vectors of eigenvalues closer than 1e-9 of the
//      spectrum's scale are re-orthogonalised (modified Gram-Schmidt, twice);
//   2. k_back: y = Q z with Q = H_0 H_1 ... H_{n-2} (reflectors applied last first), then x = L^-H y, so that
//      x^H S x = 1.
// Vectors are written row-major per problem: vec[i*n + j] is component i of eigenvector j (the reference's eigh
// column convention).
#include "eigvec.cuh"
#include "skn_common.cuh"

namespace {

constexpr int MAX_N = 2048;
using skn_vec::VNT;
constexpr int VNW = VNT / 32;

__device__ __forceinline__ double hash_unit(unsigned a, unsigned b) {
  unsigned h = a * 0x9E3779B1u ^ (b + 0x7F4A7C15u) * 0x85EBCA77u;
  h ^= h >> 15; h *= 0x2C1B3C6Du; h ^= h >> 12; h *= 0x297A2D39u; h ^= h >> 15;
  return (double)((int)(h & 0xFFFFFF) - 0x800000) * (1.0 / 8388608.0);   // [-1, 1)
}

__device__ double vblock_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int i = 0; i < VNW; ++i) t += red[i];
  return t;
}

__global__ void __launch_bounds__(VNT) k_inverse(int n_prob, const int32_t* __restrict__ nvec,
                                                const int64_t* __restrict__ hs_off, const int64_t* __restrict__ eig_off,
                                                const int32_t* __restrict__ order, const double* __restrict__ eig,
                                                const double* __restrict__ tri_all, const int32_t* __restrict__ status,
                                                double2* __restrict__ vec, double* __restrict__ scratch,
                                                int32_t* __restrict__ counter, int max_n) {
  extern __shared__ double smem[];
  double* red = smem;                                      // 2*VNW
  double* d = smem + 2 * VNW;                              // max_n
  double* e = d + max_n;                                   // max_n
  __shared__ int s_idx;
  const int tid = threadIdx.x;
  const int64_t sstride = (int64_t)max_n * VNT;
  double* su = scratch + (int64_t)blockIdx.x * 5 * sstride;   // rows i: [i*VNT + tid]
  double* s_ru1 = su;                 // 1 / u1
  double* s_u2 = su + sstride;
  double* s_u3 = su + 2 * sstride;
  double* s_m = su + 3 * sstride;
  double* s_pv = su + 4 * sstride;    // 1.0 where rows were swapped
  for (;;) {
    if (tid == 0) s_idx = atomicAdd(counter, 1);
    __syncthreads();
    const int idx = s_idx;
    __syncthreads();
    if (idx >= n_prob) break;
    const int p = order[idx];
    const int n = nvec[p];
    if (n > max_n) continue;                         // refused by the values kernel
    double2* Y = vec + hs_off[p];
    if (status[p] != SKN_OK) {
      // a problem the values kernel refused for its size keeps its buffers untouched
      if (status[p] != SKN_ERR_CAPACITY)
        for (int q = tid; q < n * n; q += VNT) Y[q] = make_double2(__longlong_as_double(0x7ff8000000000000LL), 0.0);
      __syncthreads();
      continue;
    }
    const double* tri = tri_all + 4 * eig_off[p];
    const double* w = eig + eig_off[p];
    for (int i = tid; i < n; i += VNT) {
      d[i] = tri[i];
      e[i] = tri[n + i];
    }
    __syncthreads();
    double scale = 0.0;
    for (int i = tid; i < n; i += VNT) scale = fmax(scale, fabs(w[i]));
    for (int o = 16; o > 0; o >>= 1) scale = fmax(scale, __shfl_xor_sync(0xffffffffu, scale, o));
    __syncthreads();
    if ((tid & 31) == 0) red[tid >> 5] = scale;
    __syncthreads();
    scale = red[0];
    for (int q = 1; q < VNW; ++q) scale = fmax(scale, red[q]);
    scale = fmax(scale, 1e-300);
    const double pivmin = 1e-300 * fmax(1.0, scale);

    // ---- 1. inverse iteration, one eigenvalue per thread
    for (int j0 = 0; j0 < n; j0 += VNT) {
      const int j = j0 + tid;
      if (j < n) {
        const double lam = w[j];
        double u1 = d[0] - lam, u2 = (n > 1) ? e[0] : 0.0;
        double rmax = 0.0;                 // largest |1 / pivot|
        for (int i = 0; i < n - 1; ++i) {
          const double c = e[i];
          const double a1 = d[i + 1] - lam;
          const double b1 = (i + 1 < n - 1) ? e[i + 1] : 0.0;
          double m, r1, r2, r3, pv;
          if (fabs(u1) >= fabs(c)) {
            if (fabs(u1) < pivmin) u1 = (u1 < 0.0) ? -pivmin : pivmin;
            m = c / u1;
            r1 = u1; r2 = u2; r3 = 0.0; pv = 0.0;
            u1 = a1 - m * u2;
            u2 = b1;
          } else {
            m = u1 / c;
            r1 = c; r2 = a1; r3 = b1; pv = 1.0;
            u1 = u2 - m * a1;
            u2 = -m * b1;
          }
          s_ru1[i * VNT + tid] = 1.0 / r1;
          rmax = fmax(rmax, fabs(1.0 / r1));
          s_u2[i * VNT + tid] = r2;
          s_u3[i * VNT + tid] = r3;
          s_m[i * VNT + tid] = m;
          s_pv[i * VNT + tid] = pv;
        }
        if (fabs(u1) < pivmin) u1 = (u1 < 0.0) ? -pivmin : pivmin;
        s_ru1[(n - 1) * VNT + tid] = 1.0 / u1;
        s_u2[(n - 1) * VNT + tid] = 0.0;   // the last row has no columns to its right: the back substitution
        s_u3[(n - 1) * VNT + tid] = 0.0;   // multiplies these by zero, and scratch may hold a NaN
        rmax = fmax(rmax, fabs(1.0 / u1));
        // A lam exact to the last bit (the secant step can land on the eigenvalue) leaves a pivot at the
        // 1e-300 floor, and a solve then grows the vector by up to 1 / pivot: its sum of squares overflowed
        // and the eigenvector came out NaN.  Every solve's right-hand side is therefore scaled by
        // ysc = 2^-e with 2^e >= rmax, which keeps the solution near unit size; a power of two scales
        // exactly, so without a tiny pivot the normalised vectors are bitwise what they were unscaled.
        int rex = 0;
        frexp(rmax, &rex);
        const double ysc = rex > 0 ? ldexp(1.0, -rex) : 1.0;
        // y lives in the real parts of column j of Y
        for (int i = 0; i < n; ++i) Y[(int64_t)i * n + j] = make_double2(hash_unit(j, i) * ysc, 0.0);
        for (int it = 0; it < 2; ++it) {
          for (int i = 0; i < n - 1; ++i) {
            const double m = s_m[i * VNT + tid];
            const double yi = Y[(int64_t)i * n + j].x, yn = Y[(int64_t)(i + 1) * n + j].x;
            if (s_pv[i * VNT + tid] != 0.0) {
              Y[(int64_t)i * n + j].x = yn;
              Y[(int64_t)(i + 1) * n + j].x = yi - m * yn;
            } else {
              Y[(int64_t)(i + 1) * n + j].x = yn - m * yi;
            }
          }
          double x2 = 0.0, x1 = 0.0, nrm = 0.0;
          for (int i = n - 1; i >= 0; --i) {
            const double xi = (Y[(int64_t)i * n + j].x - s_u2[i * VNT + tid] * x1 - s_u3[i * VNT + tid] * x2) *
                              s_ru1[i * VNT + tid];
            Y[(int64_t)i * n + j].x = xi;
            nrm = fma(xi, xi, nrm);
            x2 = x1;
            x1 = xi;
          }
          if (!(nrm > 0.0 && nrm <= 1.7976931348623157e308)) {   // vanished, overflowed or NaN: restart from e_j
            for (int i = 0; i < n; ++i) Y[(int64_t)i * n + j].x = (i == j) ? ysc : 0.0;
            nrm = ysc * ysc;
          }
          // normalised, and scaled by ysc again when it is the next solve's right-hand side
          const double inv = (it == 0 ? ysc : 1.0) / sqrt(nrm);
          for (int i = 0; i < n; ++i) Y[(int64_t)i * n + j].x *= inv;
        }
      }
    }
    __syncthreads();
    // ---- clusters: modified Gram-Schmidt (twice) within runs of close eigenvalues
    {
      const double ctol = 1e-9 * scale;
      int j = 1;
      while (j < n) {
        if (w[j] - w[j - 1] > ctol) { ++j; continue; }
        int j0 = j - 1, j1 = j + 1;
        while (j1 < n && w[j1] - w[j1 - 1] <= ctol) ++j1;
        for (int pass = 0; pass < 2; ++pass) {
          for (int q = j0; q < j1; ++q) {
            for (int r = j0; r < q; ++r) {
              double dp = 0.0;
              for (int i = tid; i < n; i += VNT) dp = fma(Y[(int64_t)i * n + r].x, Y[(int64_t)i * n + q].x, dp);
              dp = vblock_sum(dp, red);
              for (int i = tid; i < n; i += VNT) Y[(int64_t)i * n + q].x -= dp * Y[(int64_t)i * n + r].x;
              __syncthreads();
            }
            double nn = 0.0;
            for (int i = tid; i < n; i += VNT) nn = fma(Y[(int64_t)i * n + q].x, Y[(int64_t)i * n + q].x, nn);
            nn = vblock_sum(nn, red);
            const double inv = 1.0 / sqrt(nn);
            for (int i = tid; i < n; i += VNT) Y[(int64_t)i * n + q].x *= inv;
            __syncthreads();
          }
        }
        j = j1;
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ back-transformation
// What bounds it: FP64 issue, 12 n^3 flops a complex problem.  A column of Y needs no other column, so a CTA takes BT
// columns of one problem, one per lane, and its four warps (one per scheduler: FP64 issues at one warp instruction
// per 64 clocks on each) every fourth row; a reflector's dot products meet in shared memory in a fixed order and
// nowhere else.  Y stays in shared memory as long as n allows.  The problems' CTAs used to hold all n columns, one
// per thread, in global memory: the 484 problems of 30 to 116 orbitals of a training step took 11.0 ms with their inverse
// iteration, 7.4 now (2.2 of FP64 at its rate, half of each lane's work on ragged column tiles and short reflectors).
constexpr int BT = 32;                   // columns per CTA
constexpr int BW = 4;                    // warps
constexpr int SMEM_MAX = 232448 - 1024;

inline size_t back_smem(int n, bool tile) {
  return sizeof(double2) * (3 * (size_t)n + 2 * BW * BT + (tile ? (size_t)n * BT : 0));
}
constexpr int TILE_MAX_N = (int)((SMEM_MAX / sizeof(double2) - 2 * BW * BT) / (BT + 3));

template <bool R>
SKN_DEVINL double2 fma_cj(double2 a, double2 b, double2 c) {        // c + conj(a) b
  c.x = fma(a.x, b.x, c.x);
  if constexpr (!R) {
    c.x = fma(a.y, b.y, c.x);
    c.y = fma(a.x, b.y, c.y);
    c.y = fma(-a.y, b.x, c.y);
  }
  return c;
}

template <bool R>
SKN_DEVINL double2 add2(double2 a, double2 b) { return make_double2(a.x + b.x, R ? 0.0 : a.y + b.y); }

// Rows lo.. of the vectors: Y[(i) * ld + lane].  SM: the tile is in shared memory.
template <bool R, bool SM>
SKN_DEVINL void back(int n, int j0, const double2* __restrict__ A, const double2* __restrict__ L,
                     const double* __restrict__ tri, double2* __restrict__ Yg, double2* sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // col: 3 x n, the columns of this step, the next and the one after.  A step has one barrier, after its dot products:
  // what is fetched behind it is read behind the next step's, and replaces what was last read before it.
  double2* col = sm;
  double2* part = sm + 3 * n;                      // 2 x BW x BT
  double2* Y = SM ? part + 2 * BW * BT + lane : Yg + j0 + lane;
  const int ld = SM ? BT : n;
  const bool live = j0 + lane < n;
  auto value = [](double2 v) { return R ? make_double2(v.x, 0.0) : v; };
  if (SM)
    for (int i = warp; i < n; i += BW) Y[(int64_t)i * ld] = live ? Yg[(int64_t)i * n + j0 + lane] : make_double2(0.0, 0.0);
  // the sum of the warps' parts of one step
  auto meet = [&](int buf, double2 s) {
    part[(buf * BW + warp) * BT + lane] = s;
    __syncthreads();
    const double2* q = part + buf * BW * BT + lane;
    return add2<R>(add2<R>(q[0], q[BT]), add2<R>(q[2 * BT], q[3 * BT]));
  };
  // conj(c) . Y over this warp's rows from `from`; c[r] belongs to row from + r
  auto dot = [&](const double2* c, int from) {
    double2 s0 = make_double2(0.0, 0.0), s1 = s0;
    int i = from + ((warp - from) & (BW - 1));
    if (SM || live) {
      for (; i + BW < n; i += 2 * BW) {
        s0 = fma_cj<R>(c[i - from], Y[(int64_t)i * ld], s0);
        s1 = fma_cj<R>(c[i + BW - from], Y[(int64_t)(i + BW) * ld], s1);
      }
      if (i < n) s0 = fma_cj<R>(c[i - from], Y[(int64_t)i * ld], s0);
    }
    return add2<R>(s0, s1);
  };
  auto fetch = [&](const double2* M, int k, int buf, bool reflector) {       // column k below the diagonal
    if (k < 0) return;
    for (int r = tid; r < n - k - 1; r += BT * BW)
      col[buf * n + r] = reflector && r == 0 ? make_double2(1.0, 0.0) : value(M[(k + 1 + r) + (int64_t)k * n]);
  };
  // y = Q z
  fetch(A, n - 2, 0, true);
  fetch(A, n - 3, 1, true);
  __syncthreads();
  int buf = 0;
  for (int k = n - 2; k >= 0; --k) {
    const double2 tau = make_double2(tri[2 * n + 2 * k], R ? 0.0 : tri[2 * n + 2 * k + 1]);
    const double2* c = col + buf * n;
    const bool none = tau.x == 0.0 && tau.y == 0.0;
    const double2 s = meet(k & 1, none ? make_double2(0.0, 0.0) : dot(c, k + 1));
    fetch(A, k - 2, buf == 0 ? 2 : buf - 1, true);
    buf = buf == 2 ? 0 : buf + 1;
    if (none) continue;
    double2 ts = make_double2(-tau.x * s.x, 0.0);                            // y -= tau v (v^H y)
    if constexpr (!R) ts = make_double2(fma(tau.y, s.y, -tau.x * s.x), -fma(tau.x, s.y, tau.y * s.x));
    if (SM || live)
      for (int i = k + 1 + ((warp - k - 1) & (BW - 1)); i < n; i += BW) {
        const double2 v = c[i - k - 1];
        double2 y = Y[(int64_t)i * ld];
        y.x = fma(v.x, ts.x, y.x);
        if constexpr (!R) {
          y.x = fma(-v.y, ts.y, y.x);
          y.y = fma(v.x, ts.y, y.y);
          y.y = fma(v.y, ts.x, y.y);
        }
        Y[(int64_t)i * ld] = y;
      }
  }
  // x = L^-H y
  __syncthreads();
  fetch(L, n - 1, 0, false);
  fetch(L, n - 2, 1, false);
  __syncthreads();
  buf = 0;
  for (int i = n - 1; i >= 0; --i) {
    const double2 s = meet(i & 1, dot(col + buf * n, i + 1));
    fetch(L, i - 2, buf == 0 ? 2 : buf - 1, false);
    buf = buf == 2 ? 0 : buf + 1;
    if (warp == (i & (BW - 1)) && (SM || live)) {
      const double rl = 1.0 / L[i + (int64_t)i * n].x;
      const double2 y = Y[(int64_t)i * ld];
      Y[(int64_t)i * ld] = make_double2((y.x - s.x) * rl, R ? 0.0 : (y.y - s.y) * rl);
    }
  }
  if (SM && live)
    for (int i = warp; i < n; i += BW) Yg[(int64_t)i * n + j0 + lane] = Y[(int64_t)i * ld];
}

template <bool SM>
__global__ void __launch_bounds__(BT * BW) k_back(const int32_t* __restrict__ nvec, const int64_t* __restrict__ hs_off,
                                                  const int64_t* __restrict__ eig_off, const int32_t* __restrict__ order,
                                                  const int32_t* __restrict__ real, const double2* __restrict__ H,
                                                  const double2* __restrict__ S, const double* __restrict__ tri_all,
                                                  const int32_t* __restrict__ status, double2* __restrict__ vec, int n_prob,
                                                  int tiles, int most) {
  extern __shared__ double2 back_sm[];
  for (int64_t t = blockIdx.x; t < (int64_t)n_prob * tiles; t += gridDim.x) {
    const int p = order[t / tiles], n = nvec[p], j0 = (int)(t % tiles) * BT;
    if (n > most || j0 >= n || status[p] != SKN_OK) continue;
    const double2 *A = H + hs_off[p], *L = S + hs_off[p];
    const double* tri = tri_all + 4 * eig_off[p];
    if (real && real[p])
      back<true, SM>(n, j0, A, L, tri, vec + hs_off[p], back_sm);
    else
      back<false, SM>(n, j0, A, L, tri, vec + hs_off[p], back_sm);
    __syncthreads();
  }
}

size_t inverse_smem(int mn) { return sizeof(double) * (2 * VNW + 2 * (size_t)mn); }

cudaError_t limits() {
  cudaError_t e = cudaFuncSetAttribute(k_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)inverse_smem(MAX_N));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_back<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_back<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)back_smem(MAX_N, false));
  return e;
}

constexpr int64_t SCRATCH_BUDGET = (int64_t)2 << 30;

}  // namespace

namespace skn_vec {

int64_t cta_bytes(int max_n) { return (int64_t)5 * (max_n < 1 ? 1 : max_n) * VNT * (int64_t)sizeof(double); }

int grid(int n_prob, int max_n) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms < 1) sms = 1;
  const int mn = max_n < 1 ? 1 : max_n;
  if (limits() != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_inverse, VNT, inverse_smem(mn)) != cudaSuccess ||
      per_sm < 1)
    per_sm = 2;
  int64_t g = (int64_t)sms * per_sm;
  const int64_t cap = SCRATCH_BUDGET / cta_bytes(mn);
  if (g > cap) g = cap;
  if (g < sms) g = sms < n_prob ? sms : n_prob;      // never fewer than one CTA per SM (or per problem)
  if (g > n_prob) g = n_prob;
  return g > 0 ? (int)g : 1;
}

cudaError_t launch(int n_prob, const int32_t* n, const int64_t* hs_off, const int64_t* eig_off, const int32_t* order,
                   const int32_t* real, const double* H, const double* S, const double* eig, const double* tri,
                   const int32_t* status, double* vec, double* scratch, int n_cta, int32_t* counter, int most,
                   cudaStream_t stream) {
  cudaError_t e = limits();
  if (e != cudaSuccess) return e;
  const int mn = most < 1 ? 1 : most;
  k_inverse<<<n_cta, VNT, inverse_smem(mn), stream>>>(n_prob, n, hs_off, eig_off, order, eig, tri, status,
                                                      (double2*)vec, scratch, counter, mn);
  if ((e = cudaPeekAtLastError()) != cudaSuccess) return e;
  const bool tile = mn <= TILE_MAX_N;
  const int tiles = (mn + BT - 1) / BT;
  const int64_t all = (int64_t)n_prob * tiles;
  const unsigned g = (unsigned)(all < (1 << 20) ? all : (1 << 20));
  auto go = [&](auto kernel) {
    kernel<<<g, BT * BW, back_smem(mn, tile), stream>>>(n, hs_off, eig_off, order, real, (const double2*)H,
                                                        (const double2*)S, tri, status, (double2*)vec, n_prob, tiles, mn);
  };
  tile ? go(k_back<true>) : go(k_back<false>);
  return cudaPeekAtLastError();
}

}  // namespace skn_vec

extern "C" int skn_eigvec_scratch_bytes(int n_prob, int max_n, int64_t* bytes) {
  if (!bytes || max_n < 0 || n_prob < 0) return SKN_ERR_ARG;
  *bytes = skn_vec::grid(n_prob, max_n) * skn_vec::cta_bytes(max_n);
  return SKN_OK;
}

extern "C" int skn_eigvec(int n_prob, int max_n, const int32_t* prob, const int32_t* n, const int32_t* real,
                          const int64_t* hs_off, const int64_t* eig_off, const double* H, const double* S,
                          const double* eig, const double* tri, const int32_t* status, double* vec, double* scratch,
                          int64_t scratch_bytes, int32_t* counter, cudaStream_t stream) {
  if (n_prob < 0 || max_n < 0) return SKN_ERR_ARG;
  if (n_prob == 0) return SKN_OK;
  if (!prob || !n || !hs_off || !eig_off || !H || !S || !eig || !tri || !status || !vec || !scratch || !counter)
    return SKN_ERR_ARG;
  if (max_n > MAX_N) return SKN_ERR_CAPACITY;
  int64_t ctas = scratch_bytes / skn_vec::cta_bytes(max_n);
  const int most = skn_vec::grid(n_prob, max_n);
  if (ctas > most) ctas = most;
  if (ctas < 1) return SKN_ERR_CAPACITY;
  if (cudaMemsetAsync(counter, 0, sizeof(int32_t), stream) != cudaSuccess) return SKN_ERR_CUDA;
  return skn_vec::launch(n_prob, n, hs_off, eig_off, prob, real, H, S, eig, tri, status, vec, scratch, (int)ctas,
                         counter, max_n, stream) == cudaSuccess ? SKN_OK : SKN_ERR_CUDA;
}
