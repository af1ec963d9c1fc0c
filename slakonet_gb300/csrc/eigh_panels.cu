// Generalized Hermitian eigenvalues of problems of about 100 orbitals and more, blocked, with every O(n^3)
// step but the Hermitian matrix-vector products on the tcgen05 tensor cores.
//
// The problems of one call go through one sequence of launches together, largest first; every launch covers all that
// still have columns at its panel:
//   1. set-up: zero rows (eighb's aux option, slakonet/utils.py:741-747), the upper triangle of H;
//   2. per panel: Cholesky of the diagonal block of S; triangular solves of the panel's rows and of the block
//      row of B = L^-1 H; one update S22 -= L21 L21^H and H_below -= L21 B_panel on the tensor cores;
//   3. per panel: the column block of C = B L^-H by row solves; one update of the trailing lower triangle
//      C22 -= C_panel L21^H on the tensor cores;
//   4. per 16 columns: the trailing tiles in 56-bit fixed point (k_fixed), Householder reflectors and the W vectors of
//      LAPACK's zlatrd (k_tri_panel, a team of CTAs per problem), then A22 -= V W^H + W V^H on the tensor cores;
//   5. eigenvalues of the tridiagonal (sturm.cuh).
// The reference calls torch.linalg.cholesky / solve / eigh per k (slakonet/utils.py:749-783,
// slakonet/main.py:174).
//
// GB300 notes.  An SM does two FP64 multiply-adds per clock, so what stays on that unit bounds everything.  The updates
// are sums of integer slice products on the tensor cores, the leading ones added exactly and rounded once per panel; the
// matrix-vector products of the tridiagonalisation are sums of 28-bit limb products on the integer units, rounded once per
// tile (what each leaves out stands below); FP64 keeps the reflectors, the O(n) work of a column and the diagonal blocks.  Every sum that crosses warps or CTAs goes to its own
// slot and is added in a fixed order, or is an integer, so a problem's results depend neither on the other problems nor
// on the number of CTAs it is given.
// Measured (random pencils): 492 orbitals x 300 problems 393 ms with one CTA per problem, 208 with the products in FP64,
// 97 now (tridiagonalisation 48, updates 32, solves 8, eigenvalues 4); 432 x 8 190, 18.8, 9.8 ms (5.8 of them the
// tridiagonalisation, 13 us a column); 1152 x 2 47, 31.3 ms.
#include <algorithm>
#include <array>
#include <map>
#include <mutex>
#include <utility>

#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "exact_round.cuh"
#include "skn_common.cuh"
#include "sturm.cuh"

namespace {

namespace cg = cooperative_groups;

constexpr int NB = 32;               // panel width of the factorisations
constexpr int NT = 16;               // columns per tridiagonalisation panel
constexpr int TS = 32;               // tile edge of the matrix-vector products
constexpr int SLICES = 8;
constexpr int KP = 64;               // inner dimension of the sliced products (32 complex columns)
constexpr int BM = 128, BN = 16;     // output tile of the tensor-core update
constexpr int PANELS_MAX_N = 2048;

SKN_DEVINL int cdiv_d(int a, int b) { return (a + b - 1) / b; }
inline int cdiv(int a, int b) { return (a + b - 1) / b; }

// ------------------------------------------------------------------ arithmetic (R: real parts only)
template <bool R> SKN_DEVINL double2 ld(const double2* p) {
  if constexpr (R) return make_double2(p->x, 0.0); else return *p;
}
template <bool R> SKN_DEVINL double2 ldc(const double2* p) {      // written by another CTA of this launch
  if constexpr (R) return make_double2(__ldcg(&p->x), 0.0); else return __ldcg(p);
}
template <bool R> SKN_DEVINL void st(double2* p, double2 v) {
  if constexpr (R) p->x = v.x; else *p = v;
}
template <bool R> SKN_DEVINL double2 fma_(double2 a, double2 b, double2 c) {        // c + a b
  if constexpr (R) { c.x = fma(a.x, b.x, c.x); return c; } else return cfma(a, b, c);
}
template <bool R> SKN_DEVINL double2 fma_cja(double2 a, double2 b, double2 c) {     // c + conj(a) b
  if constexpr (R) { c.x = fma(a.x, b.x, c.x); return c; } else return cfma_conj(a, b, c);
}
template <bool R> SKN_DEVINL double2 fms(double2 a, double2 b, double2 c) {         // c - a b
  c.x = fma(-a.x, b.x, c.x);
  if constexpr (!R) {
    c.x = fma(a.y, b.y, c.x);
    c.y = fma(-a.x, b.y, c.y);
    c.y = fma(-a.y, b.x, c.y);
  }
  return c;
}
template <bool R> SKN_DEVINL double2 fms_cj(double2 a, double2 b, double2 c) {      // c - a conj(b)
  if constexpr (R) { c.x = fma(-a.x, b.x, c.x); return c; } else return cfms_conj(a, b, c);
}
template <bool R> SKN_DEVINL double2 mul(double2 a, double2 b) {
  if constexpr (R) return make_double2(a.x * b.x, 0.0); else return cmul(a, b);
}
template <bool R> SKN_DEVINL double2 add(double2 a, double2 b) {
  return make_double2(a.x + b.x, R ? 0.0 : a.y + b.y);
}
template <bool R> SKN_DEVINL double2 warp_sum(double2 s) {                          // fixed butterfly
  for (int o = 16; o > 0; o >>= 1) {
    s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
    if constexpr (!R) s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
  }
  return s;
}
SKN_DEVINL double2 zero2() { return make_double2(0.0, 0.0); }

// ------------------------------------------------------------------ scratch (per problem slot)
struct Lay {
  int64_t W, VW, xc, Yp, sN, sT, sD, li, d, e2, d32, e232, bnd, flg, bar, sa, sb, sc, ea, eb, ec, fx, fe, vf, ve, stride;   // bytes
};
__host__ __device__ inline int64_t take(int64_t& o, int64_t bytes) {
  const int64_t r = o;
  o += (bytes + 255) / 256 * 256;
  return r;
}
// Rows of a slice array: a 128-row tile may start at any multiple of 16 up to n.
__host__ __device__ inline int64_t slice_rows(int n) { return ((int64_t)n + 127) / 128 * 128 + 128; }
__host__ __device__ inline Lay layout(int n) {
  const int64_t nt = (n + TS - 1) / TS, nr = slice_rows(n);
  Lay L;
  int64_t o = 0;
  L.W = take(o, 16 * (int64_t)NT * n);         // W panel, column q at W + q n (row index of the matrix)
  L.VW = take(o, 16 * (int64_t)2 * NT * n);    // rows of [W V]: row r at VW + 2 NT r
  L.xc = take(o, 16 * (int64_t)n);             // the current column before its scaling
  L.Yp = take(o, 16 * nt * n);                 // matrix-vector partial sums: slot s at Yp + s n
  L.sN = take(o, 8 * nt);                      // column norm, per 32-row chunk
  L.sT = take(o, 8 * nt * (nt + 1) / 2);       // v^H A v, per tile
  L.sD = take(o, 16 * nt * 2 * NT);            // [W V]^H v, per 32-row chunk
  L.li = take(o, 16 * (int64_t)NB * NB * ((n + NB - 1) / NB));   // inverses of the diagonal blocks, row-major
  L.d = take(o, 8 * (int64_t)n);
  L.e2 = take(o, 8 * (int64_t)n);
  L.d32 = take(o, 4 * (int64_t)n);
  L.e232 = take(o, 4 * (int64_t)n);
  L.bnd = take(o, 64);
  L.flg = take(o, 4 * 2 * (int64_t)n);
  L.bar = take(o, 4 * ((int64_t)n / NT + 1));  // arrivals at a grid team's barriers, per tridiagonalisation panel
  L.sa = take(o, 2 * SLICES * nr * KP);        // row operand
  L.sb = take(o, 2 * 2 * SLICES * nr * KP);    // column operand from rows: form B, then B'
  L.sc = take(o, 2 * 2 * SLICES * nr * KP);    // column operand from the block row of B
  L.ea = take(o, 4 * nr);                      // row exponents of sa, sb, sc
  L.eb = take(o, 4 * nr);
  L.ec = take(o, 4 * nr);
  L.fx = take(o, 16 * (int64_t)TS * TS * (nt * (nt + 1) / 2));   // the trailing block's tiles in 56-bit fixed point
  L.fe = take(o, 4 * (nt * (nt + 1) / 2));                       // their exponents
  L.vf = take(o, 16 * (int64_t)TS * 2 * NT * nt);                // chunks of [W V] in fixed point, column by column
  L.ve = take(o, 4 * (int64_t)2 * NT * nt);                      // the exponent of each of their columns
  L.stride = o;
  return L;
}

// Polls after which the waits of a kernel give up: the solves' and the updates' on their products and copies, a grid
// team's barriers (a poll of the last takes about half a microsecond).
struct Limits {
  int solve, update, team;
};
constexpr Limits LIMITS{1 << 26, 1 << 26, 1 << 22};

struct Grp {
  int nmax, n_prob;
  Limits limits;
  const int32_t* prob;       // [n_prob] problem of each slot, sizes descending
  const int64_t* ws_off;     // [n_prob] byte offset of each slot's scratch
  const int32_t* nvec;
  const int32_t* real;       // [*] 1 where H and S are exactly real; may be null
  const int64_t* hs_off;
  const int64_t* eig_off;
  double2* H;
  double2* S;
  double* eig;
  int32_t* status;
  double* tri;               // d, e, tau per problem at 4 eig_off (for eigenvectors); may be null
  char* scratch;
  int64_t scratch_bytes;
};

struct WS {
  double2 *W, *VW, *xc, *Yp, *sD, *li;
  double *sN, *sT, *d, *e2, *bnd;
  float *d32, *e232;
  int *flg, *ea, *eb, *ec;
  unsigned* bar;
  uint16_t *sa, *sb, *sc;
  int4 *fx, *vf;
  int *fe, *ve;
  int64_t nr;                // rows of a slice array
};
SKN_DEVINL WS ws_of(const Grp& G, int g) {
  const int n = G.nvec[G.prob[g]];
  const Lay L = layout(n);
  char* b = G.scratch + G.ws_off[g];
  WS w;
  w.W = (double2*)(b + L.W); w.VW = (double2*)(b + L.VW); w.xc = (double2*)(b + L.xc); w.Yp = (double2*)(b + L.Yp);
  w.sD = (double2*)(b + L.sD); w.sN = (double*)(b + L.sN); w.sT = (double*)(b + L.sT); w.li = (double2*)(b + L.li);
  w.d = (double*)(b + L.d); w.e2 = (double*)(b + L.e2); w.bnd = (double*)(b + L.bnd);
  w.d32 = (float*)(b + L.d32); w.e232 = (float*)(b + L.e232); w.flg = (int*)(b + L.flg);
  w.bar = (unsigned*)(b + L.bar);
  w.ea = (int*)(b + L.ea); w.eb = (int*)(b + L.eb); w.ec = (int*)(b + L.ec);
  w.sa = (uint16_t*)(b + L.sa); w.sb = (uint16_t*)(b + L.sb); w.sc = (uint16_t*)(b + L.sc);
  w.fx = (int4*)(b + L.fx); w.fe = (int*)(b + L.fe);
  w.vf = (int4*)(b + L.vf); w.ve = (int*)(b + L.ve);
  w.nr = slice_rows(n);
  return w;
}
SKN_DEVINL bool live(const Grp& G, int p) { return G.status[p] == SKN_OK; }
SKN_DEVINL bool is_real(const Grp& G, int p) { return G.real != nullptr && G.real[p] != 0; }

// ------------------------------------------------------------------ integer slices
// Error-free splitting (Ozaki, Ogita and Oishi, Numer. Algorithms 59, 2012).  A row of 32 complex values is
// scaled by its exponent ex and cut into SLICES digits of 7 bits, x = 2^ex sum_s d_s 2^(-7 (s + 1)) with
// |d_0| <= 128 and -64 <= d_s < 64 after it, each exact in bf16; what is cut off is at most 2^-57 2^ex, 2^-56 of
// the row's largest entry.  A slice product is an integer of at most 14 bits and a 64-term sum of the at most
// 8 slice pairs of one level s + t < 8 stays below 2^23, exact in an FP32 accumulator.  The pairs of higher levels are left
// out: 2^-49 of the two rows' scales if all their digits were extreme and of one sign, 2^-55 for digits without a pattern
// (each FP64 product would be off by 2^-53 of itself).  The complex product P Q^H takes A = [Pr Pi], B = [Qr Qi] for the real part and B' = [-Qi Qr] for the imaginary part.
// The digits are taken with integer operations: the FP64 pipe would cost more than the solves.
constexpr int EXP_NAN = INT32_MIN;       // a row with a non-finite entry: its products become NaN

// Element index in a slice array, in the tensor cores' K-major core-matrix order (8-row groups of KP x 8
// elements, each a run of 8 x 8 core matrices along K), so rows starting at a multiple of 8 are one run.
SKN_DEVINL int64_t tc_idx(int r, int k) { return (int64_t)(r >> 3) * (8 * KP) + (k >> 3) * 64 + (r & 7) * 8 + (k & 7); }

SKN_DEVINL long long fixed56(double x, int emax) {       // round(x 2^(56 - ex)), ex = emax - 1022
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7ff), d = emax - e;
  const unsigned long long m = (b & 0xfffffffffffffull) | 0x10000000000000ull;
  // m 2^3 is the value at d = 0; one bit more is kept for the rounding
  unsigned long long f = d <= 59 ? (m << 4) >> d : 0;
  f = (f + 1) >> 1;
  const long long sg = (long long)b >> 63;
  return e == 0 ? 0 : ((long long)f ^ sg) - sg;
}
// 64 at each of the seven low digits: the digits of f + DIGIT_BIAS are its bit fields, each 64 too large
constexpr long long DIGIT_BIAS = 64LL * (1 + (1LL << 7) + (1LL << 14) + (1LL << 21) + (1LL << 28) + (1LL << 35) + (1LL << 42));
// Digit s of a biased value as a float, exact in its upper 16 bits (bf16).
SKN_DEVINL uint32_t digit_bf16(long long fb, int s) {
  if (s == 0)                                             // the leading digit, unbiased, |d| <= 128
    return __float_as_uint(__int_as_float(0x4B400000 + (int)(fb >> 49)) - 12582912.0f);
  const int sh = 7 * (SLICES - 1 - s);
  const uint32_t v = sh + 7 <= 32 ? (uint32_t)fb >> sh
                     : sh >= 32   ? (uint32_t)(fb >> 32) >> (sh - 32)
                                  : __funnelshift_r((uint32_t)fb, (uint32_t)(fb >> 32), sh);
  return __float_as_uint(__uint_as_float(0x4B400000u | (v & 127u)) - 12582976.0f);
}
SKN_DEVINL uint4 neg4(uint4 v) {
  return make_uint4(v.x ^ 0x80008000u, v.y ^ 0x80008000u, v.z ^ 0x80008000u, v.w ^ 0x80008000u);
}

// The digits of 8 entries of one part of a row: kb < 4 the real parts of z_(8 kb) .., then the imaginary ones.
template <class Get>
SKN_DEVINL void slice_block(Get get, int kb, int emax, uint4* out) {
  uint32_t w[SLICES][4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const double2 z0 = get((kb & 3) * 8 + 2 * u), z1 = get((kb & 3) * 8 + 2 * u + 1);
    const long long f0 = fixed56(kb < 4 ? z0.x : z0.y, emax) + DIGIT_BIAS;
    const long long f1 = fixed56(kb < 4 ? z1.x : z1.y, emax) + DIGIT_BIAS;
#pragma unroll
    for (int s = 0; s < SLICES; ++s) w[s][u] = __byte_perm(digit_bf16(f0, s), digit_bf16(f1, s), 0x7632);
  }
#pragma unroll
  for (int s = 0; s < SLICES; ++s) out[s] = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
}

constexpr int SE = 8;                     // entries of a row a thread slices: one block of digits per part
SKN_DEVINL int high_word8(const double2* z) {
  int hm = 0;
#pragma unroll
  for (int q = 0; q < SE; ++q)
    hm = max(hm, max(__double2hiint(z[q].x) & 0x7fffffff, __double2hiint(z[q].y) & 0x7fffffff));
  return hm;
}
// Slices of 8 of a row's 32 entries, part `part` of row r.  A form to sa (null: none) with exponent ea[r]; B and B' forms
// to sb, of the row with its halves swapped when `swap` (z' = [z_16.. z_31, z_0.. z_15]).
SKN_DEVINL void slice_part(const double2* z, int part, int emax, int r, int64_t nr, uint16_t* sa, int* ea, uint16_t* sb,
                           int* eb, bool swap) {
  const int ex = emax == 0x7ff ? EXP_NAN : emax - 1022;
  if (part == 0) {
    if (sa) ea[r] = ex;
    if (sb) eb[r] = ex;
  }
#pragma unroll
  for (int im = 0; im < 2; ++im) {
    uint4 out[SLICES];
    slice_block([&](int k) { return z[k & (SE - 1)]; }, 4 * im, emax, out);
    const int kb = part + 4 * im, pb = swap ? 4 * im + ((part + 2) & 3) : kb;      // place of these entries in A, in B
#pragma unroll
    for (int s = 0; s < SLICES; ++s) {
      const uint4 v = out[s];
      if (sa) *reinterpret_cast<uint4*>(sa + (int64_t)s * nr * KP + tc_idx(r, kb * 8)) = v;
      if (sb) {
        *reinterpret_cast<uint4*>(sb + (int64_t)s * nr * KP + tc_idx(r, pb * 8)) = v;
        // B' = [-Qi Qr]: the real part of Q goes to the second half, minus the imaginary part to the first
        *reinterpret_cast<uint4*>(sb + (int64_t)(SLICES + s) * nr * KP + tc_idx(r, (pb ^ 4) * 8)) = im ? neg4(v) : v;
      }
    }
  }
}

// ------------------------------------------------------------------ set-up
__global__ void __launch_bounds__(256) k_init(Grp G) {
  const int g = blockIdx.y, p = G.prob[g], n = G.nvec[p];
  const bool ok = n >= 1 && n <= G.nmax && G.hs_off[p] >= 0 && G.eig_off[p] >= 0 && G.ws_off[g] >= 0 &&
                  G.ws_off[g] % 256 == 0 && G.ws_off[g] + layout(n).stride <= G.scratch_bytes;
  if (blockIdx.x == 0 && threadIdx.x == 0) G.status[p] = ok ? SKN_OK : SKN_ERR_CAPACITY;
  if (!ok) return;
  const WS w = ws_of(G, g);
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < 2 * n) w.flg[i] = 0;
  if (i <= n / NT) w.bar[i] = 0;
}

// Rows with a nonzero entry, from 32 x 32 tiles of the lower triangles (entry (i, j) marks rows i and j), and
// the upper triangle of H from the lower one.  One warp per tile; blockIdx.z: 0 H, 1 S.
__global__ void __launch_bounds__(256) k_scan(Grp G) {
  const int g = blockIdx.y, which = blockIdx.z, p = G.prob[g];
  if (!live(G, p)) return;
  const int n = G.nvec[p], nt = cdiv_d(n, TS), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ double2 tiles[8][TS * (TS / 8 + 1)];
  const int t = blockIdx.x * 8 + warp;
  if (t >= nt * nt) return;
  const int I = t / nt, J = t % nt;
  if (J > I) return;
  double2* A = (which ? G.S : G.H) + G.hs_off[p];
  int* flg = ws_of(G, g).flg + which * n;
  const int i = I * TS + lane;
  bool row = false;
  double2* T = tiles[warp];
  for (int c0 = 0; c0 < TS; c0 += 4) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = J * TS + c0 + c;
      double2 a = zero2();
      bool nz = false;
      if (i < n && j <= i) {
        a = A[i + (int64_t)j * n];
        nz = !(is_zero_bits(a.x) && is_zero_bits(a.y));
      }
      row |= nz;
      if (__any_sync(0xffffffffu, nz) && lane == 0) flg[j] = 1;
      T[lane * 5 + c] = a;
    }
    __syncwarp();
    if (which == 0) {                       // column j of the lower tile is row j of the upper one
      const int c = lane & 3, j = J * TS + c0 + c;
      for (int r = lane >> 2; r < TS; r += 8) {
        const int gi = I * TS + r;
        if (gi < n && j < gi) {
          const double2 a = T[r * 5 + c];
          A[j + (int64_t)gi * n] = make_double2(a.x, flip_sign(a.y));
        }
      }
    }
    __syncwarp();
  }
  if (row) flg[i] = 1;
}

__global__ void __launch_bounds__(256) k_fix(Grp G) {
  const int g = blockIdx.y, p = G.prob[g];
  if (!live(G, p)) return;
  const int n = G.nvec[p], i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const int* flg = ws_of(G, g).flg;
  double2* H = G.H + G.hs_off[p] + (int64_t)i * (n + 1);
  double2* S = G.S + G.hs_off[p] + (int64_t)i * (n + 1);
  const double h = H->x + (flg[i] ? 0.0 : 1.0);
  *H = make_double2(h, 0.0);
  if (!flg[n + i]) S->x += 1.0;
}

// ------------------------------------------------------------------ Cholesky of a diagonal block
// One CTA of 8 warps; warp q holds columns q, q + 8, q + 16, q + 24 of the block and of its inverse (lane = row), so
// column k is one warp's registers: that warp takes the root and scales it, all apply it to both.  The inverse X
// starts as the unit matrix: step k scales its row k and subtracts l_i times it from the rows below.
__global__ void __launch_bounds__(256) k_potrf(Grp G, int c0) {
  const int g = blockIdx.x, p = G.prob[g];
  if (!live(G, p)) return;
  const int n = G.nvec[p], w = min(NB, n - c0), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (w <= 0) return;
  __shared__ double2 col[2][NB];
  __shared__ double s_rd[2];
  __shared__ int s_bad;
  double2* A11 = G.S + G.hs_off[p] + c0 + (int64_t)c0 * n;
  double2 a[4], x[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int j = warp + 8 * u;
    a[u] = (lane < w && j <= lane) ? A11[lane + (int64_t)j * n] : zero2();
    x[u] = make_double2(lane == j ? 1.0 : 0.0, 0.0);
  }
  if (threadIdx.x == 0) s_bad = 0;
  __syncthreads();
#pragma unroll
  for (int kb = 0; kb < 4; ++kb) {          // columns 8 kb .. 8 kb + 7: static register indices
#pragma unroll 1
    for (int kq = 0; kq < 8; ++kq) {
      const int k = kb * 8 + kq;
      if (k >= w) break;
      if (warp == kq) {
        // root and reciprocal as in the small eigensolver: a reciprocal root and one Newton step on the root
        const double akk = __shfl_sync(0xffffffffu, a[kb].x, k);
        const bool ok = akk > 0.0 && is_finite_bits(akk);
        const double q = ok ? akk : 1.0, r = rsqrt(q), r0 = q * r;
        const double dk = fma(fma(-r0, r0, q), 0.5 * r, r0);
        double2 l = make_double2(a[kb].x * r, a[kb].y * r);
        if (lane == k) l = make_double2(dk, 0.0);
        if (lane < k) l = zero2();
        col[k & 1][lane] = l;
        a[kb] = l;
        if (lane == 0) {
          s_rd[k & 1] = r;
          if (!ok) s_bad = 1;
        }
      }
      __syncthreads();
      const double2 li = col[k & 1][lane];
      const double r = s_rd[k & 1];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = warp + 8 * u;
        if (u >= kb && j > k && j < w) a[u] = cfms_conj(li, col[k & 1][j], a[u]);
        if (u <= kb && j <= k) {
          if (lane == k) x[u] = make_double2(x[u].x * r, x[u].y * r);
          double2 xk;
          xk.x = __shfl_sync(0xffffffffu, x[u].x, k);
          xk.y = __shfl_sync(0xffffffffu, x[u].y, k);
          if (lane > k) x[u] = fms<false>(li, xk, x[u]);
        }
      }
    }
  }
  double2* li = ws_of(G, g).li + (int64_t)(c0 / NB) * NB * NB;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int j = warp + 8 * u;
    if (lane < w && j <= lane && j < w) A11[lane + (int64_t)j * n] = a[u];
    li[lane * NB + j] = (lane < w && j <= lane) ? x[u] : zero2();
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_bad) G.status[p] = SKN_ERR_NOT_SPD;
}

// ------------------------------------------------------------------ tensor-core building blocks
SKN_DEVINL uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// Shared-memory matrix descriptor: no swizzle, K-major core matrices (8 rows x 16 bytes), 128 bytes between core
// matrices along K, KP * 16 bytes between 8-row groups.
SKN_DEVINL uint64_t tc_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)((128u >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)(((KP * 16u) >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}
// kind::f16: D F32, A and B BF16, both K-major, M = 128, N columns
SKN_DEVINL uint32_t tc_idesc(int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}
SKN_DEVINL void tc_mma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}
SKN_DEVINL void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar));
}
SKN_DEVINL void tmem_ld4(uint32_t a, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(a));
}
// Exact sums of UC columns over the levels: hi counts units of 2^28 of lo.  The level sums are integers below 2^22:
// the FP32 addition of 1.5 2^23 leaves them in the low bits, and two levels fit 32 bits.
constexpr int UC = 4;                                // columns a thread takes at once
SKN_DEVINL void level_sums(uint32_t base, int level_cols, long long* hi, long long* lo) {
  auto quad = [&](int L, long long* out) {
    uint32_t t[4][UC];
#pragma unroll
    for (int l = 0; l < 4; ++l) tmem_ld4(base + (uint32_t)((L + l) * level_cols), t[l]);
    asm volatile("tcgen05.wait::ld.sync.aligned;");
    auto whole = [](uint32_t x) { return __float_as_int(__uint_as_float(x) + 12582912.0f) - 0x4B400000; };
#pragma unroll
    for (int q = 0; q < UC; ++q)
      out[q] = (long long)(whole(t[0][q]) * 128 + whole(t[1][q])) * 16384 + (whole(t[2][q]) * 128 + whole(t[3][q]));
  };
  quad(0, hi);
  quad(4, lo);
}

// Wait for a phase of a barrier; gives up after `limit` polls or once the CTA has failed.
SKN_DEVINL bool upd_wait(uint32_t bar, uint32_t parity, volatile int* fail, int limit) {
  for (int it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 1023) == 1023 && *fail) return false;
  }
  return false;
}
SKN_DEVINL void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
SKN_DEVINL void bar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

constexpr int A_BYTES = BM * KP * 2;                 // 16 KB: one slice of 128 rows

// ------------------------------------------------------------------ triangular solves
// Rows x of x L11^H = a and columns of L11 x = a, through the inverse X of the diagonal block: x = a X^H, and for a
// column conj(x) = conj(a) X^H, on the tensor cores (a substitution in FP64 kept one warp per 32 rows busy for 85 us
// a panel, and was a quarter of the FP64 work at n = 400).  MODE 1 (Cholesky sweep): blocks [0, nrow): rows below
// the panel of S, sliced as both operands of the update; the others: columns of the block row of H, sliced as column
// operand.  MODE 2 (second sweep): blocks [0, nrow): rows from the panel's own down of H, sliced as row operand; the
// others: rows of L21, sliced as column operand without a solve.
// One CTA per 128 rows, four threads a row with 8 of its 32 entries each: they slice them into shared memory (four more
// warps the rows of X), one thread issues the products, each rounds its 8 sums and slices them for the update.  The row's
// exponent is the only thing the four share.  Bound by the latency of that chain: with one thread a row a CTA took 53 us
// (MODE 1) and 42 (MODE 2), 25 and 21 now.
constexpr int SV_PARTS = 4, SV_ROW_WARPS = 4 * SV_PARTS, SV_THREADS = 32 * (SV_ROW_WARPS + SV_PARTS);
constexpr int X_BYTES = 2 * NB * KP * 2;             // 8 KB: one slice of X, both forms
constexpr int SV_SMEM = SLICES * (A_BYTES + X_BYTES);              // 192 KB
constexpr uint32_t SV_COLS = SLICES * 2 * NB;        // 512 TMEM columns
static_assert(NB / SV_PARTS == SE, "four threads slice a row");

template <int MODE>
__global__ void __launch_bounds__(SV_THREADS, 1) k_solve(Grp G, int c0, int nrow) {
  const int g = blockIdx.y, p = G.prob[g];
  if (!live(G, p)) return;
  const int n = G.nvec[p], w = min(NB, n - c0);
  const bool rows = blockIdx.x < nrow;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int first = rows ? (MODE == 1 ? c0 + NB : c0) : (MODE == 1 ? 0 : c0 + NB);
  const int base = first + (rows ? blockIdx.x : blockIdx.x - nrow) * BM;
  if (c0 >= n || base >= n) return;
  const WS ws = ws_of(G, g);
  double2* S = G.S + G.hs_off[p];
  double2* H = G.H + G.hs_off[p];
  const bool xwarp = warp >= SV_ROW_WARPS;
  const int part = xwarp ? warp - SV_ROW_WARPS : warp >> 2;
  const int row = xwarp ? lane : (warp & 3) * 32 + lane;
  const int r = base + row;                          // row, or column of the block row (not the warps of X)
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ int s_hm[SV_PARTS][BM + NB];
  const int slot = xwarp ? BM + row : row;
  // the exponent field of the four threads' entries
  auto together = [&](const double2* z) {
    s_hm[part][slot] = high_word8(z);
    __syncthreads();
    return max(max(s_hm[0][slot], s_hm[1][slot]), max(s_hm[2][slot], s_hm[3][slot])) >> 20;
  };
  double2 z[SE];
  if (MODE == 2 && !rows) {
#pragma unroll
    for (int q = 0; q < SE; ++q) z[q] = !xwarp && r < n ? S[r + (int64_t)(c0 + part * SE + q) * n] : zero2();
    const int emax = together(z);
    if (!xwarp && r < n) slice_part(z, part, emax, r, ws.nr, nullptr, nullptr, ws.sb, ws.eb, false);
    return;
  }
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_ex[NB];
  __shared__ volatile int s_fail;
  const uint32_t a0 = smem_u32(smem), x0 = a0 + SLICES * A_BYTES, bar = smem_u32(&s_bar);
  if (tid == 0) {
    s_fail = 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  if (warp == SV_ROW_WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(SV_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  // entry k of this thread's row; a column's entries are taken conjugate
  const bool conj_in = !rows;
  double2* src = rows ? (MODE == 1 ? S : H) + r + (int64_t)c0 * n : H + c0 + (int64_t)r * n;
  const int64_t step = rows ? n : 1;
  const double2* X = ws.li + (int64_t)(c0 / NB) * NB * NB + lane * NB;
#pragma unroll
  for (int q = 0; q < SE; ++q) {
    const int k = part * SE + q;
    z[q] = zero2();
    if (xwarp) {
      z[q] = X[k];
    } else if (r < n && k < w && !(MODE == 2 && k > r - c0)) {      // above the diagonal: not updated, not needed
      z[q] = src[k * step];
      if (conj_in) z[q].y = flip_sign(z[q].y);
    }
  }
  int er;
  {
    const int emax = together(z);
    er = emax == 0x7ff ? EXP_NAN : emax - 1022;
    if (xwarp && part == 0) s_ex[row] = er;
    // slice s of X: rows 0 .. 31 form B, rows 32 .. 63 form B'
    uint16_t* dst = reinterpret_cast<uint16_t*>(smem + (xwarp ? SLICES * A_BYTES : 0));
    const int slice_el = (xwarp ? X_BYTES : A_BYTES) / 2;
#pragma unroll
    for (int im = 0; im < 2; ++im) {
      uint4 v[SLICES];
      slice_block([&](int k) { return z[k & (SE - 1)]; }, 4 * im, emax, v);
      const int kb = part + 4 * im;
#pragma unroll
      for (int s = 0; s < SLICES; ++s) {
        uint16_t* D = dst + (int64_t)s * slice_el;
        *reinterpret_cast<uint4*>(D + tc_idx(row, kb * 8)) = v[s];
        if (xwarp) *reinterpret_cast<uint4*>(D + tc_idx(row + NB, (kb ^ 4) * 8)) = im ? neg4(v[s]) : v[s];
      }
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");    // the products read what the threads wrote
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_slot;
  if (tid == 32 * SV_ROW_WARPS) {
    for (int s = 0; s < SLICES; ++s) {
      // column slices 0 .. SLICES - 1 - s side by side give levels s .. SLICES - 1; at most 256 columns a product
      for (int t0 = 0; t0 < SLICES - s; t0 += 4) {
        const int cnt = min(4, SLICES - s - t0);
        const uint32_t id = tc_idesc(cnt * 2 * NB);
#pragma unroll
        for (int kk = 0; kk < KP / 16; ++kk)
          tc_mma(tmem + (uint32_t)((s + t0) * 2 * NB), tc_desc(a0 + (uint32_t)(s * A_BYTES) + kk * 256),
                 tc_desc(x0 + (uint32_t)(t0 * X_BYTES) + kk * 256), id, (s > 0 || kk > 0) ? 1u : 0u);
      }
    }
    tc_commit(bar);
  }
  if (!upd_wait(bar, 0, &s_fail, G.limits.solve)) s_fail = 1;
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (s_fail && tid == 0) {            // the products must have completed before the CTA frees its TMEM and exits
    volatile int never = 0;
    upd_wait(bar, 0, &never, LIMITS.solve);
  }
#pragma unroll
  for (int q = 0; q < SE; ++q) z[q] = zero2();
  if (!s_fail && !xwarp) {
    const uint32_t tb = tmem + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
    for (int h = 0; h < SE; h += 4) {
      const int cb = part * SE + h;
      long long hr[4], lr[4], hi[4], li[4];
      level_sums(tb + cb, 2 * NB, hr, lr);
      level_sums(tb + NB + cb, 2 * NB, hi, li);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int k = cb + q, ex = s_ex[k];
        if (r < n && k < w) {
          double2 v;
          if (er == EXP_NAN || ex == EXP_NAN) {
            v = make_double2(__longlong_as_double(0x7ff8000000000000LL), __longlong_as_double(0x7ff8000000000000LL));
          } else {
            v = make_double2(round_sum28(hr[q], lr[q], er + ex - 63), round_sum28(hi[q], li[q], er + ex - 63));
          }
          z[h + q] = v;
          if (conj_in) v.y = flip_sign(v.y);
          src[k * step] = v;
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  const int emax = together(z);                      // its barrier: the accumulators have been read
  if (!s_fail && !xwarp && r < n) {
    if (rows && r >= c0 + NB)
      slice_part(z, part, emax, r, ws.nr, ws.sa, ws.ea, MODE == 1 ? ws.sb : nullptr, ws.eb, false);
    if (!rows && c0 + NB < n) slice_part(z, part, emax, r, ws.nr, nullptr, nullptr, ws.sc, ws.ec, false);
  }
  if (tid == 0 && s_fail) G.status[p] = SKN_ERR_CUDA;
  if (warp == SV_ROW_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(SV_COLS));
}

// ------------------------------------------------------------------ tensor-core update
constexpr int BH_BYTES = BN * KP * 2;                // 2 KB: one slice of a tile's columns, one form
constexpr int B_BYTES = SLICES * 2 * BH_BYTES;       // 32 KB
constexpr int UPD_SMEM = SLICES * A_BYTES + 2 * B_BYTES;       // 192 KB
constexpr uint32_t BUF_COLS = SLICES * 2 * BN;       // TMEM columns of one tile
constexpr uint32_t TMEM_COLS = 2 * BUF_COLS;
constexpr int UPD_WARPS = 16, UPD_THREADS = 32 * (UPD_WARPS + 1);

// C -= A B^T over BM x BN tiles.  SWEEP 1: blocks [0, nlow) of S22 (lower triangle, columns from sb), the rest
// of H below the panel over all columns (sc); SWEEP 2 and 3: the trailing lower triangle of H (sb).
// c1: first row and column of the trailing matrix.  A CTA has one 128-row block I and up to jc column tiles: its
// 8 row slices stay in shared memory (128 KB), the column slices and the accumulators are double-buffered.
// One thread copies and issues the products of every slice pair of level < SLICES; warps 0-3 and 8-11 take the halves of
// the even tiles, the others those of the odd: a thread has a row, fetches its entries of C while the products run, adds
// the levels exactly in int64 and rounds once.  Bound by the latency of that chain, so the warps count: at n = 492 x 300
// problems a tile takes 39k clocks of an SM with one tile per CTA, 16k with eight warps, 12.9k with sixteen.
// All waits are bounded; one that runs out marks the problem SKN_ERR_CUDA and leaves the tile, and the
// copies and products that were issued are still waited for (bounded).
template <int SWEEP>
__global__ void __launch_bounds__(UPD_THREADS, 1) k_update(Grp G, int c1, int nlow, int chunks_low, int chunks_all,
                                                           int jc) {
  const int g = blockIdx.y, p = G.prob[g];
  if (!live(G, p)) return;
  const int n = G.nvec[p], m = n - c1;
  if (m <= 0 || (SWEEP == 3 && m == 1)) return;      // the panel kernel has finished a lone last entry
  const bool low = SWEEP != 1 || blockIdx.x < nlow;
  const int bx = low ? blockIdx.x : blockIdx.x - nlow;
  const int I = bx / (low ? chunks_low : chunks_all), ch = bx % (low ? chunks_low : chunks_all);
  const int r0 = I * BM;
  if (r0 >= m) return;
  // tile columns of the block: the lower triangle ends with the block's last row
  const int nj = low ? cdiv_d(min(m, r0 + BM), BN) : cdiv_d(n, BN);
  const int j0 = ch * jc, ntile = min(jc, nj - j0);
  if (ntile <= 0) return;
  const WS w = ws_of(G, g);
  const uint16_t* sB = low ? w.sb : w.sc;
  const int* eB = low ? w.eb : w.ec;
  const int boff = low ? c1 : 0;                     // matrix column (and slice row) of tile column 0
  const int arow = c1 + r0;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t a0 = smem_u32(smem), b0 = a0 + SLICES * A_BYTES;
  __shared__ __align__(8) uint64_t bars[SLICES + 6];  // row slices landed; columns landed; products done; drained
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int s_fail;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto bar = [&](int b) { return smem_u32(&bars[b]); };
  constexpr int B_FULL = SLICES, T_FULL = SLICES + 2, T_EMPTY = SLICES + 4;
  if (tid == 0) {
    s_fail = 0;
    for (int b = 0; b < T_EMPTY; ++b) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar(b)));
    for (int b = T_EMPTY; b < T_EMPTY + 2; ++b) asm volatile("mbarrier.init.shared::cta.b64 [%0], 8;" ::"r"(bar(b)));
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  if (warp == UPD_WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_slot;
  if (warp == UPD_WARPS) {
    if (lane == 0) {
      auto load_b = [&](int i) {
        const uint32_t bb = bar(B_FULL + (i & 1)), dst = b0 + (uint32_t)((i & 1) * B_BYTES);
        bar_expect(bb, B_BYTES);
        const int64_t row = boff + (j0 + i) * BN;
        for (int t = 0; t < SLICES; ++t)
          for (int f = 0; f < 2; ++f)
            bulk_g2s(dst + (uint32_t)((2 * t + f) * BH_BYTES), sB + ((int64_t)(f * SLICES + t) * w.nr + row) * KP, BH_BYTES,
                     bb);
      };
      for (int s = 0; s < SLICES; ++s) {
        bar_expect(bar(s), A_BYTES);
        bulk_g2s(a0 + (uint32_t)(s * A_BYTES), w.sa + ((int64_t)s * w.nr + arow) * KP, A_BYTES, bar(s));
        if (s == 0) load_b(0);
      }
      int loaded = 1, issued = 0, landed = 0, a_landed = 0, finished = 0;   // tiles (or row slices) so far
      if (ntile > 1) {
        load_b(1);
        loaded = 2;
      }
      bool ok = true;
      for (int i = 0; ok && i < ntile; ++i) {
        const int b = i & 1;
        ok = upd_wait(bar(B_FULL + b), (uint32_t)((i >> 1) & 1), &s_fail, G.limits.update);
        if (!ok) break;
        ++landed;
        if (i >= 2) ok = upd_wait(bar(T_EMPTY + b), (uint32_t)(((i >> 1) - 1) & 1), &s_fail, G.limits.update);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t bs = b0 + (uint32_t)(b * B_BYTES), td = tmem + (uint32_t)b * BUF_COLS;
        for (int s = 0; s < SLICES; ++s) {
          if (i == 0) {
            ok = upd_wait(bar(s), 0, &s_fail, G.limits.update);
            if (!ok) break;
            ++a_landed;
            asm volatile("tcgen05.fence::after_thread_sync;");
          }
          // row slice s by the column slices 0 .. SLICES - 1 - s side by side: levels s .. SLICES - 1 in one product
          const uint32_t id = tc_idesc((SLICES - s) * 2 * BN);
#pragma unroll
          for (int kk = 0; kk < KP / 16; ++kk)
            tc_mma(td + (uint32_t)(s * 2 * BN), tc_desc(a0 + (uint32_t)(s * A_BYTES) + kk * 256), tc_desc(bs + kk * 256),
                   id, (s > 0 || kk > 0) ? 1u : 0u);
        }
        tc_commit(bar(T_FULL + b));
        ++issued;
        if (!ok) break;
        if (i >= 1 && i + 1 < ntile) {                // the other column buffer, once tile i - 1 has been multiplied
          ok = upd_wait(bar(T_FULL + (b ^ 1)), (uint32_t)(((i - 1) >> 1) & 1), &s_fail, G.limits.update);
          if (!ok) break;
          finished = i;
          load_b(i + 1);
          ++loaded;
        }
      }
      // whatever was issued must have completed before the CTA frees its TMEM and exits
      if (!ok) s_fail = 1;
      volatile int never = 0;
      for (; a_landed < SLICES; ++a_landed)
        if (!upd_wait(bar(a_landed), 0, &never, LIMITS.update)) ok = false;
      for (; landed < loaded; ++landed)
        if (!upd_wait(bar(B_FULL + (landed & 1)), (uint32_t)((landed >> 1) & 1), &never, LIMITS.update)) ok = false;
      for (; finished < issued; ++finished)
        if (!upd_wait(bar(T_FULL + (finished & 1)), (uint32_t)((finished >> 1) & 1), &never, LIMITS.update)) ok = false;
      if (!ok) s_fail = 1;
    }
  } else {
    const int grp = (warp >> 2) & 1, wq = warp & 3, c0 = (warp >> 3) * (BN / 2);        // a warp reads TMEM lanes 32 (warp mod 4) .. + 31
    const int i = r0 + wq * 32 + lane;               // trailing row
    const bool rok = i < m;
    const int er = rok ? w.ea[c1 + i] : 0;
    double2* C = (SWEEP == 1 && low ? G.S : G.H) + G.hs_off[p] + c1 + i;
    const uint32_t base = tmem + (uint32_t)grp * BUF_COLS + ((uint32_t)(wq * 32) << 16);
    for (int it = grp; it < ntile; it += 2) {
      const int q0 = (j0 + it) * BN;                 // tile's first column, counted from boff
      double2 cv[BN / 2];
#pragma unroll
      for (int q = 0; q < BN / 2; ++q) {
        const int gc = boff + q0 + c0 + q;
        cv[q] = zero2();
        if (rok && gc < n && (!low || i >= q0 + c0 + q)) cv[q] = C[(int64_t)gc * n];
      }
      const bool ok = upd_wait(bar(T_FULL + grp), (uint32_t)((it >> 1) & 1), &s_fail, G.limits.update);
      if (!ok || s_fail) {
        s_fail = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
      for (int h = 0; h < BN / 2; h += UC) {
        const int cb = c0 + h;
        long long hr[UC], lr[UC], hi[UC], li[UC];
        level_sums(base + cb, 2 * BN, hr, lr);
        level_sums(base + BN + cb, 2 * BN, hi, li);
        if (h + UC == BN / 2) {                      // the accumulators have been read: the next tile may start
          asm volatile("tcgen05.fence::before_thread_sync;");
          if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar(T_EMPTY + grp)) : "memory");
        }
#pragma unroll
        for (int q = 0; q < UC; ++q) {
          const int j = q0 + cb + q, gc = boff + j;
          if (rok && gc < n && (!low || i >= j)) {
            double2 v = cv[h + q];
            const int ec = eB[gc];
            if (er == EXP_NAN || ec == EXP_NAN) {
              v = make_double2(__longlong_as_double(0x7ff8000000000000LL), __longlong_as_double(0x7ff8000000000000LL));
            } else {
              const int e = er + ec - 63;            // the sums count units of 2^(er + ec - 63)
              v.x -= round_sum28(hr[q], lr[q], e);
              v.y = (low && i == j) ? 0.0 : v.y - round_sum28(hi[q], li[q], e);
            }
            C[(int64_t)gc * n] = v;
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (tid == 0 && s_fail) G.status[p] = SKN_ERR_CUDA;
  if (warp == UPD_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
}

// ------------------------------------------------------------------ tridiagonalisation panel
// Columns c0 .. c0 + w - 1 by one cluster of CTAs per problem, in zlatrd order.  Rows are counted from c0;
// 32-row chunk c belongs to CTA c mod C (a warp per chunk, lane = row); the 32 x 32 tiles of the lower triangle
// are dealt to the cluster's warps.  A column takes two cluster barriers:
//   after the column's update: its norm (per chunk);
//   after the products: y = A22 v (a slot per tile row and column), [W V]^H v (per chunk), v^H A22 v (per tile).
// Then w = tau (y - V (W^H v) - W (V^H v)) + alpha v with alpha = -|tau|^2 / 2 (v^H A22 v - 2 Re (W^H v)^H (V^H v)),
// which needs no further reduction, and the next column's update runs on the same rows in the same pass.
// Every CTA computes W's entry of the next pivot row itself, with the same operations.
// A tile is read once for both products: lane = row (A v), then lane = column (A^H v); both, and the products with [W V],
// in fixed point (below).  The FP64 unit belongs to one of the SM's four partitions: a warp issues one FP64 instruction
// per 64 clocks, however independent its instructions are, so the FP64 work of a phase is spread over the warps.
// RES: a CTA's tiles and its rows of [W V] fit its shared memory and stay there for the panel's 16 columns; eight warps
// take a tile each, and two a chunk's row.  The form for few problems, bound by the latency of a column: 25,600 clocks at
// 432 orbitals on clusters of 12, 5,500 of them the products (20,000 in FP64), the rest two barriers, the reflector, the
// sums and the row's update.  Else a warp takes whole tiles, streamed, and the CTAs of other problems fill the partitions:
// the form for many, bound by latency too (at 320 x 152 a scheduler issues on 23% of its cycles, its waits split between
// barriers, loads and fixed latencies; the integer pipe is busy 23%, FP64 14%), so residency and even rounds count.  Integer
// sums do not depend on their order and FP64 sums keep theirs, so both forms give the same bits.
constexpr int PW = 4;                            // warps per CTA when streamed, one per partition
constexpr int PWR = 8;                           // and when resident: two per partition hide each other's latency
constexpr int PT = 32 * PW, PTR = 32 * PWR;
static_assert(PWR * 32 * sizeof(double2) <= 2 * PW * 32 * sizeof(int4), "W's entries fit the multipliers");
constexpr int TILE_LD = TS + 1;
constexpr int TILE_EL = TS * TILE_LD;            // a resident tile, or a chunk's 32 columns of [W V]
constexpr int QT = TS / PW;                      // columns or rows of a quarter; columns staged when streamed
constexpr int VMAX = 8;                          // column entries a thread fetches ahead (1024 rows)
struct PanelSm {
  double2 rowV[NT], rowW[NT];                    // V and W at the next pivot row
  double2 part[PW][2 * NT];                      // [W V]^H v by quarters of the chunks
  int4 tf[PW][2 * NT], qf[PW][2 * NT];           // multipliers of [W V]'s columns for a warp's chunk
  double2 tau, scl, yrow, wrow;
  double vav, alpha;
  int triv, dead;
};

SKN_DEVINL void tile_ij(int t, int& I, int& J) {     // lower-triangle tile index, I >= J
  int i = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
  while (i > 0 && i * (i + 1) / 2 > t) --i;
  while ((i + 1) * (i + 2) / 2 <= t) ++i;
  I = i;
  J = t - i * (i + 1) / 2;
}
constexpr int EPS = TS * PW * (16 + 64);         // a chunk's partial sums: four of y's slots, four of the two integer sums
template <bool R> SKN_DEVINL double2 sum4(double2 a, double2 b, double2 c, double2 d) {
  return add<R>(add<R>(a, b), add<R>(c, d));
}

// ------------------------------------------------------------------ fixed-point products
// A tile and a chunk of v are held as integers of 56 bits under one exponent, each in two limbs of 28 (balanced, so the
// low one has a sign).  Of a product's four partial products the lowest, 2^-58 of the largest, is left out; the others are
// exact in 64-bit accumulators over the 32 terms of a tile, and a tile's sum is rounded once.  The error per term is that
// of the operands' last bit, at most 2^-56 of the largest, against 2^-53 of each product for FP64: it stays below FP64's own
// as long as the entries of a tile are within 2^3 of each other, and relative to the matrix's norm always.  Entries further
// below their tile's largest keep fewer bits than in FP64.  Measured against extended precision, eigenvalues are no further
// off for it: physical pencils of 65 to 400 orbitals 0.3-0.5 eps of the scale (one CTA in FP64 0.9), random ones 0.16-0.23
// (0.31-0.38), graded and block-scaled ones over 3 to 9 decades within 2% of the FP64 kernel's error or below it.
// A partition issues a multiply-add of two 32-bit integers into 64 bits every 4.8 clocks and an FP64 instruction every 64:
// three of the one replace one of the other.
struct alignas(8) Limb { int h, l; };
SKN_DEVINL Limb limbs(long long f) {
  const long long h = (f + (1LL << 27)) >> 28;
  return {(int)h, (int)(f - (h << 28))};
}
template <bool R> SKN_DEVINL int4 fixed_point(double2 a, int emax) {
  const Limb x = limbs(fixed56(a.x, emax));
  if constexpr (R) return make_int4(x.h, x.l, 0, 0);
  const Limb y = limbs(fixed56(a.y, emax));
  return make_int4(x.h, x.l, y.h, y.l);
}
template <bool R> SKN_DEVINL int high_word(double2 a) {         // orders magnitudes; its upper bits are the exponent
  const int x = __double2hiint(a.x) & 0x7fffffff;
  if constexpr (R) return x;
  return max(x, __double2hiint(a.y) & 0x7fffffff);
}
constexpr int EXP_BAD = 1 << 20;                                // an infinity or a NaN among the operands
SKN_DEVINL int exp_sum(int a, int b) { return a == 0x7ff || b == 0x7ff ? EXP_BAD : a + b; }
SKN_DEVINL long long wide(int a, int b, long long c) { return c + (long long)a * b; }
// sums of a v (or conj(a) v): real and imaginary parts, high (2^56) and middle (2^28) weights
template <bool R> struct Dot {
  long long rh = 0, rm = 0, ih = 0, im = 0, qh = 0, qm = 0;
  SKN_DEVINL void add(int4 a, int4 v) {                         // a v
    rh = wide(a.x, v.x, rh);
    rm = wide(a.x, v.y, wide(a.y, v.x, rm));
    if constexpr (!R) {
      qh = wide(a.z, v.z, qh);
      qm = wide(a.z, v.w, wide(a.w, v.z, qm));
      ih = wide(a.x, v.z, wide(a.z, v.x, ih));
      im = wide(a.x, v.w, wide(a.y, v.z, wide(a.z, v.y, wide(a.w, v.x, im))));
    }
  }
  SKN_DEVINL void add_conj(int4 a, int4 v) {                    // conj(a) v
    rh = wide(a.x, v.x, rh);
    rm = wide(a.x, v.y, wide(a.y, v.x, rm));
    if constexpr (!R) {
      rh = wide(a.z, v.z, rh);
      rm = wide(a.z, v.w, wide(a.w, v.z, rm));
      ih = wide(a.x, v.z, ih);
      im = wide(a.x, v.w, wide(a.y, v.z, im));
      qh = wide(a.z, v.x, qh);
      qm = wide(a.z, v.y, wide(a.w, v.x, qm));
    }
  }
  SKN_DEVINL void close(bool conj) {                            // then (rh, rm) + i (ih, im)
    if constexpr (!R) {
      if (conj) { ih -= qh; im -= qm; } else { rh -= qh; rm -= qm; }
    }
  }
  SKN_DEVINL void sum_lanes(int o) {
    rh += __shfl_xor_sync(0xffffffffu, rh, o);
    rm += __shfl_xor_sync(0xffffffffu, rm, o);
    if constexpr (!R) {
      ih += __shfl_xor_sync(0xffffffffu, ih, o);
      im += __shfl_xor_sync(0xffffffffu, im, o);
    }
  }
  SKN_DEVINL void put(long long* p, int stride) const {
    p[0] = rh;
    p[stride] = rm;
    if constexpr (!R) {
      p[2 * stride] = ih;
      p[3 * stride] = im;
    }
  }
  SKN_DEVINL void take(const long long* p, int stride) {
    rh += p[0];
    rm += p[stride];
    if constexpr (!R) {
      ih += p[2 * stride];
      im += p[3 * stride];
    }
  }
  // the rounded sum; ke: the sum of the operands' exponent fields
  SKN_DEVINL double2 value(int ke) const {
    if (ke == EXP_BAD) {
      const double q = __longlong_as_double(0x7ff8000000000000LL);
      return make_double2(q, R ? 0.0 : q);
    }
    const int k = ke - 2 * (1022 + 56);
    return make_double2(round_wide28(rh, rm, k + 28), R ? 0.0 : round_wide28(ih, im, k + 28));
  }
};

// entry (i, j) of the Hermitian block of M rows at A, from its lower triangle
template <bool R> SKN_DEVINL double2 trailing_entry(const double2* A, int n, int M, int i, int j) {
  if (i >= M || j >= M) return zero2();
  double2 a = ld<R>(i >= j ? A + i + (int64_t)j * n : A + j + (int64_t)i * n);
  if constexpr (!R) a.y = i == j ? 0.0 : cond_flip(a.y, i < j);
  return a;
}

// The tiles of the trailing block at c0 in fixed point, for the 16 columns of a panel: a CTA per tile, a warp per 8
// columns.  Bound by its reads and writes, 32 bytes an entry.
template <bool R>
SKN_DEVINL void fixed_body(const Grp& G, int g, int p, int c0, int* red) {
  const int n = G.nvec[p], M = n - c0, nt = cdiv_d(M, TS), t = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (t >= nt * (nt + 1) / 2) return;
  int I, J;
  tile_ij(t, I, J);
  const WS ws = ws_of(G, g);
  const double2* A = G.H + G.hs_off[p] + c0 + (int64_t)c0 * n;
  double2 a[QT];
  int hm = 0;
#pragma unroll
  for (int u = 0; u < QT; ++u) {
    a[u] = trailing_entry<R>(A, n, M, I * TS + lane, J * TS + warp * QT + u);
    hm = max(hm, high_word<R>(a[u]));
  }
  hm = __reduce_max_sync(0xffffffffu, hm);
  if (lane == 0) red[warp] = hm;
  __syncthreads();
  const int emax = max(max(red[0], red[1]), max(red[2], red[3])) >> 20;
  if (threadIdx.x == 0) ws.fe[t] = emax;
  int4* T = ws.fx + (int64_t)t * TS * TS + warp * QT * TS + lane;
#pragma unroll
  for (int u = 0; u < QT; ++u) {
    const int4 f = fixed_point<R>(a[u], emax);
    if constexpr (R) reinterpret_cast<int2*>(T + u * TS)[0] = make_int2(f.x, f.y);
    else T[u * TS] = f;
  }
}
__global__ void __launch_bounds__(PT) k_fixed(Grp G, int c0) {
  __shared__ int red[PW];
  const int g = blockIdx.y, p = G.prob[g];
  if (!live(G, p) || c0 >= G.nvec[p] - 1) return;
  if (is_real(G, p)) fixed_body<true>(G, g, p, c0, red);
  else fixed_body<false>(G, g, p, c0, red);
}
template <bool R> SKN_DEVINL int4 ld_fixed(const int4* p) {
  if constexpr (R) {
    const int2 v = *reinterpret_cast<const int2*>(p);
    return make_int4(v.x, v.y, 0, 0);
  } else {
    return *p;
  }
}

// The CTAs of one problem: a cluster, or (more than 16) CTAs of a cooperative launch that meet at a counter.  A
// wait is bounded; once one has run out the problem is marked SKN_ERR_CUDA and its CTAs no longer wait.
struct Team {
  int rank, C, limit;
  bool grid;
  unsigned* count;
  unsigned target;
  int32_t* status;
  int* dead;                                     // shared: a wait has run out
  SKN_DEVINL void sync() {
    if (C == 1) {
      __syncthreads();
    } else if (!grid) {
      cg::this_cluster().sync();
    } else {
      target += (unsigned)C;
      __syncthreads();
      if (threadIdx.x == 0 && !*dead) {
        __threadfence();
        atomicAdd(count, 1u);
        int it = 0;
        for (; it < limit; ++it) {
          unsigned v;
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
          if (v >= target) break;
        }
        if (it == limit) {
          *dead = 1;
          *status = SKN_ERR_CUDA;
        }
        __threadfence();
      }
      __syncthreads();
    }
  }
};

// v 2^k for the two operands below, which meet near the root of the matrix's scale: no overflow; what falls below the normal
// range is far below the row's largest entry and counts as zero.
SKN_DEVINL double halfway(double v, int k) {
  const int h = __double2hiint(v), e = (h >> 20) & 0x7ff;
  if (e == 0x7ff) return v;
  return e == 0 || e + k <= 0 ? 0.0 : __hiloint2double(h + (int)((unsigned)k << 20), __double2loint(v));
}

// sv: the Householder vector, svf: the same in fixed point, sve: its exponents by 32 rows; big: streamed, a quarter of a
// tile per warp; RES, tiles (rt), chunks of [W V] (cpc) and their partial sums (2 x cpc x PW x 32).
template <bool R, bool RES>
SKN_DEVINL void panel_body(const Grp& G, int g, int p, int c0, Team& team, int rt, int cpc, PanelSm& sm, double2* sv,
                           int4* svf, int* sve, double2* big) {
  constexpr int NWP = RES ? PWR : PW, NTH = 32 * NWP;
  const int rank = team.rank, C = team.C;
  const int n = G.nvec[p], M = n - c0, w = min(NT, n - 1 - c0);
  const int nt = cdiv_d(M, TS), ntile = nt * (nt + 1) / 2;
  const WS ws = ws_of(G, g);
  double2* A = G.H + G.hs_off[p] + c0 + (int64_t)c0 * n;      // entry (r, c) of the trailing block at r + c n
  double2* W = ws.W;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double* tri = G.tri ? G.tri + 4 * G.eig_off[p] : nullptr;
  int4* wvs = reinterpret_cast<int4*>(big + (int64_t)rt * TILE_EL);      // chunk lc, column q, row r at lc TILE_EL + q TILE_LD + r
  char* eps = reinterpret_cast<char*>(wvs + (int64_t)cpc * TILE_EL);     // chunk lc at lc EPS: y by quarters, then the integer sums
  int* wve = reinterpret_cast<int*>(eps + (int64_t)cpc * EPS);      // chunk lc: 32 exponents, then the sums' two
  auto sync = [&]() { team.sync(); };
  // column q of chunk ch of [W V] in fixed point, lane = row
  auto put_fixed = [&](int ch, int q, int4 f, int emax) {
    if constexpr (RES) {
      wvs[(ch / C) * TILE_EL + q * TILE_LD + lane] = f;
      if (lane == 0) wve[(ch / C) * (2 * NT + 2) + q] = emax;
    } else {
      int4* d = ws.vf + ((int64_t)ch * 2 * NT + q) * TS + lane;
      if constexpr (R) *reinterpret_cast<int2*>(d) = make_int2(f.x, f.y);
      else *d = f;
      if (lane == 0) ws.ve[ch * 2 * NT + q] = emax;
    }
  };
  auto fixed_exp = [&](int ch, int q) { return RES ? wve[(ch / C) * (2 * NT + 2) + q] : ws.ve[ch * 2 * NT + q]; };
  // chunks and tiles of this CTA are rank, rank + C, ...; streamed, a warp takes every PW-th of them
  const int first = rank + C * warp, stride = C * NWP;
  if constexpr (RES) {
    for (int t = rank, i = 0; t < ntile; t += C, ++i) {
      int4* T = reinterpret_cast<int4*>(big) + (int64_t)i * TILE_EL;
      const int4* src = ws.fx + (int64_t)t * TS * TS;
#pragma unroll
      for (int c = warp; c < TS; c += NWP) T[c * TILE_LD + lane] = ld_fixed<R>(src + c * TS + lane);
    }
  }
  // first column as it stands
  for (int ch = first; ch < nt; ch += stride) {
    const int r = ch * 32 + lane;
    double2 a = zero2();
    if (r < M) {
      a = ld<R>(A + r);
      if (r == 0) a.y = 0.0;
      st<R>(ws.xc + r, a);
      if (r == 0) ws.d[c0] = a.x;
    }
    double s = r >= 2 && r < M ? (R ? a.x * a.x : fma(a.x, a.x, a.y * a.y)) : 0.0;
    s = warp_sum<true>(make_double2(s, 0.0)).x;
    if (lane == 0) ws.sN[ch] = s;
  }
  for (int j = 0; j < w; ++j) {
    const int k = c0 + j;
    sync();
    // ---- the reflector: two warps take the norm, one the quotient by beta, one the scale of v; meanwhile the column arrives
    double2 xv[VMAX];
#pragma unroll
    for (int u = 0; u < VMAX; ++u) {
      const int r = tid + u * NTH;
      if (u * NTH < nt * 32) xv[u] = (r > j + 1 && r < M) ? ldc<R>(ws.xc + r) : zero2();
    }
    if (warp < 2) {
      const double2 al = ldc<R>(ws.xc + j + 1);
      double s = 0.0;
      for (int c = lane; c < nt; c += 32) s += __ldcg(ws.sN + c);
      const double xnorm2 = warp_sum<true>(make_double2(s, 0.0)).x;
      const bool triv = xnorm2 == 0.0 && al.y == 0.0;
      const double q = triv ? 1.0 : fma(al.x, al.x, fma(al.y, al.y, xnorm2));
      const double inv = rsqrt(q), r0 = q * inv;                 // a root (one Newton step) and its reciprocal from one chain
      const double nrm = fma(fma(-r0, r0, q), 0.5 * inv, r0);
      const bool up = al.x >= 0.0;
      const double beta = triv ? al.x : (up ? -nrm : nrm), ib = up ? -inv : inv;
      if (warp == 0) {
        const double taur = triv ? 0.0 : (beta - al.x) * ib;
        const double taui = (R || triv) ? 0.0 : -al.y * ib;
        if (lane == 0) {
          sm.tau = make_double2(taur, taui);
          sm.triv = triv;
          if (rank == 0) {
            ws.e2[k] = beta * beta;
            if (tri) {
              tri[n + k] = beta;
              tri[2 * n + 2 * k] = taur;
              tri[2 * n + 2 * k + 1] = taui;
            }
          }
        }
      } else if (warp == 1) {
        const double dr = al.x - beta, di = al.y;
        const double den = triv ? 0.0 : 1.0 / fma(dr, dr, di * di);
        if (lane == 0) sm.scl = make_double2(dr * den, -di * den);
      }
    }
    __syncthreads();
    const int triv = sm.triv;
    const double2 tau = sm.tau, scl = sm.scl;
    auto put_v = [&](int r, double2 v) {
      if (r > j && r < M && (r >> 5) % C == rank) {
        st<R>(A + r + (int64_t)j * n, v);
        st<R>(ws.VW + (int64_t)r * 2 * NT + NT + j, v);
      }
    };
    auto fix_v = [&](int r, double2 v) {                     // a warp's rows are a chunk
      const int emax = __reduce_max_sync(0xffffffffu, high_word<R>(v)) >> 20;
      const int4 f = fixed_point<R>(v, emax);
      svf[r] = f;
      if (lane == 0) sve[r >> 5] = emax;
      if ((r >> 5) % C == rank) put_fixed(r >> 5, NT + j, f, emax);
    };
#pragma unroll
    for (int u = 0; u < VMAX; ++u) {
      const int r = tid + u * NTH;
      if (u * NTH < nt * 32 && r < nt * 32) {
        double2 v = xv[u];
        if (r == j + 1) v = make_double2(1.0, 0.0);
        else if (!triv) v = mul<R>(v, scl);
        sv[r] = v;
        put_v(r, v);
        fix_v(r, v);
      }
    }
    for (int r = tid + VMAX * NTH; r < nt * 32; r += NTH) {
      double2 v = r < M ? ldc<R>(ws.xc + r) : zero2();      // r > j + 1: past the entries above
      if (!triv) v = mul<R>(v, scl);
      sv[r] = v;
      put_v(r, v);
      fix_v(r, v);
    }
    __syncthreads();
    // ---- products with v
    // y of tile t's rows (lane = row); a diagonal tile is whole, another one stands for its transpose too
    auto put_tile = [&](int t, int I, int J, double2 y) {
      const int gi = I * TS + lane;
      const bool diag = I == J;
      if (gi < M) st<R>(ws.Yp + (int64_t)J * n + gi, y);
      const double2 vi = sv[gi];
      double s = R ? vi.x * y.x : fma(vi.x, y.x, vi.y * y.y);   // Re conj(v) y
      s = warp_sum<true>(make_double2(s, 0.0)).x;
      if (lane == 0) ws.sT[t] = diag ? s : 2.0 * s;
    };
    if (!triv) {
      if constexpr (RES) {
        for (int t = first, i = warp; t < ntile; t += stride, i += NWP) {
          int I, J;
          tile_ij(t, I, J);
          const int4* T = reinterpret_cast<const int4*>(big) + (int64_t)i * TILE_EL;
          const int4 *vI = svf + I * TS, *vJ = svf + J * TS;
          const int ea = ws.fe[t];
          Dot<R> y;
#pragma unroll 8
          for (int c = 0; c < TS; ++c) y.add(T[c * TILE_LD + lane], vJ[c]);
          y.close(false);
          if (I != J) {
            Dot<R> z;
#pragma unroll 8
            for (int r = 0; r < TS; ++r) z.add_conj(T[lane * TILE_LD + r], vI[r]);
            z.close(true);
            st<R>(ws.Yp + (int64_t)I * n + J * TS + lane, z.value(exp_sum(ea, sve[I])));      // J TS + 31 < I TS < M
          }
          put_tile(t, I, J, y.value(exp_sum(ea, sve[J])));
        }
      } else {
        int4* T = reinterpret_cast<int4*>(big) + (int64_t)warp * QT * TILE_LD;
        const int qc = lane & (QT - 1), qr = lane / QT;
        for (int t = first; t < ntile; t += stride) {
          int I, J;
          tile_ij(t, I, J);
          const bool diag = I == J;
          const int4 *vI = svf + I * TS + qr * QT, *vJ = svf + J * TS;
          const int4* src = ws.fx + (int64_t)t * TS * TS + lane;
          const int ea = ws.fe[t];
          Dot<R> y, z;
#pragma unroll
          for (int q = 0; q < PW; ++q) {
            int4 a[QT];
#pragma unroll
            for (int u = 0; u < QT; ++u) a[u] = ld_fixed<R>(src + (q * QT + u) * TS);
            __syncwarp();
#pragma unroll
            for (int u = 0; u < QT; ++u) {
              y.add(a[u], vJ[q * QT + u]);
              if (!diag) T[u * TILE_LD + lane] = a[u];
            }
            if (diag) continue;
            __syncwarp();
            Dot<R> zq;
            const int4* Tc = T + qc * TILE_LD + qr * QT;
#pragma unroll
            for (int u = 0; u < QT; ++u) zq.add_conj(Tc[u], vI[u]);
            zq.close(true);
            zq.sum_lanes(QT);
            zq.sum_lanes(2 * QT);
            if (qr == q) z = zq;
          }
          y.close(false);
          if (!diag) st<R>(ws.Yp + (int64_t)I * n + J * TS + lane, z.value(exp_sum(ea, sve[I])));
          put_tile(t, I, J, y.value(exp_sum(ea, sve[J])));
        }
      }
      if (j > 0) {
        // lane = column of [W V]: W columns 0..j-1 and V columns NT..NT+j-1; a sum per chunk
        const bool on = lane < NT ? lane < j : lane - NT < j;
        if constexpr (RES) {
          const int mine = (ntile - rank + C - 1) / C;         // the chunks go on where the tiles' deal to the warps ended
          for (int ch = rank, i = 0; ch < nt; ch += C, ++i) {
            if ((mine + i) % NWP != warp) continue;
            const int4 *src = wvs + (int64_t)i * TILE_EL + lane * TILE_LD, *v = svf + ch * TS;
            Dot<R> z;
#pragma unroll 8
            for (int r = 0; r < TS; ++r) z.add_conj(src[r], v[r]);
            z.close(true);
            if (on) st<R>(ws.sD + ch * 2 * NT + lane, z.value(exp_sum(fixed_exp(ch, lane), sve[ch])));
          }
        } else {
          int4* T = reinterpret_cast<int4*>(big) + (int64_t)warp * QT * TILE_LD;
          const int qc = lane & (QT - 1), qr = lane / QT;
          for (int ch = first; ch < nt; ch += stride) {
            const int4 *src = ws.vf + (int64_t)ch * 2 * NT * TS + lane, *v = svf + ch * TS + qr * QT;
            Dot<R> z;
#pragma unroll
            for (int q = 0; q < PW; ++q) {
              if ((q & 1) * QT >= j) continue;                 // none of its columns is there yet
              int4 a[QT];
#pragma unroll
              for (int u = 0; u < QT; ++u) a[u] = ld_fixed<R>(src + (q * QT + u) * TS);
              __syncwarp();
#pragma unroll
              for (int u = 0; u < QT; ++u) T[u * TILE_LD + lane] = a[u];
              __syncwarp();
              Dot<R> zq;
              const int4* Tc = T + qc * TILE_LD + qr * QT;
#pragma unroll
              for (int u = 0; u < QT; ++u) zq.add_conj(Tc[u], v[u]);
              zq.close(true);
              zq.sum_lanes(QT);
              zq.sum_lanes(2 * QT);
              if (qr == q) z = zq;
            }
            if (on) st<R>(ws.sD + ch * 2 * NT + lane, z.value(exp_sum(fixed_exp(ch, lane), sve[ch])));
          }
        }
      }
    }
    // the next column of the panel, or (last panel) the one remaining entry, the last diagonal element
    const bool next = j + 1 < w || j + 2 == M;
    sync();
    // ---- W's column j; the next column
    {
      const bool on = lane < NT ? lane < j : lane - NT < j;
      double2 s = zero2();
      if (!triv && on && warp < PW) {
#pragma unroll 4
        for (int c = warp; c < nt; c += PW) s = add<R>(s, ldc<R>(ws.sD + c * 2 * NT + lane));
      }
      if (warp < PW) sm.part[warp][lane] = s;
      constexpr int W0 = RES ? PW : 1;                       // the warps past those of the sums, if there are any
      if (!triv && warp == W0) {
        double q = 0.0;
#pragma unroll 8
        for (int t = lane; t < ntile; t += 32) q += __ldcg(ws.sT + t);
        q = warp_sum<true>(make_double2(q, 0.0)).x;
        if (lane == 0) sm.vav = q;
      } else if (!triv && warp == W0 + 1) {
        double2 q = zero2();
        for (int t = lane; t < nt; t += 32) q = add<R>(q, ldc<R>(ws.Yp + (int64_t)t * n + j + 1));
        q = warp_sum<R>(q);
        if (lane == 0) sm.yrow = q;
      } else if (warp == W0 + 2 && lane < j) {
        sm.rowV[lane] = ldc<R>(A + (j + 1) + (int64_t)lane * n);
        sm.rowW[lane] = ldc<R>(W + (int64_t)lane * n + c0 + j + 1);
      }
    }
    __syncthreads();
    double2 tm, qm;                 // multipliers of [W V]'s column `lane` in y and in the next column
    {
      const double2 s = sum4<R>(sm.part[0][lane], sm.part[1][lane], sm.part[2][lane], sm.part[3][lane]);
      // lane q < NT has t1_q, lane NT + q has t2_q; W's columns take t2, V's take t1
      const double2 o = make_double2(__shfl_xor_sync(0xffffffffu, s.x, NT),
                                     R ? 0.0 : __shfl_xor_sync(0xffffffffu, s.y, NT));
      const int c = lane & (NT - 1);
      const bool on = c < j;
      tm = on && !triv ? o : zero2();
      qm = on && next ? (lane < NT ? sm.rowV[c] : sm.rowW[c]) : zero2();
      if constexpr (!R) qm.y = -qm.y;
      // resident, by the warps that have no corrections to sum
      if (!triv && warp == (RES ? PWR - 1 : 0)) {          // the pivot row's tau (y - V t1 - W t2)
        double2 c = zero2();
        if (lane < j) {
          c = mul<R>(sm.rowV[lane], s);
          c = fma_<R>(sm.rowW[lane], o, c);
        }
        for (int q = 8; q > 0; q >>= 1) {
          c.x += __shfl_xor_sync(0xffffffffu, c.x, q);
          if constexpr (!R) c.y += __shfl_xor_sync(0xffffffffu, c.y, q);
        }
        if (lane == 0) sm.wrow = mul<R>(tau, make_double2(sm.yrow.x - c.x, R ? 0.0 : sm.yrow.y - c.y));
      } else if (!triv && warp == (RES ? PWR - 2 : 1)) {   // alpha, with Re sum_q conj(t1_q) t2_q
        double dot = lane < j ? (R ? s.x * o.x : fma(s.x, o.x, s.y * o.y)) : 0.0;
        for (int q = 8; q > 0; q >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, q);
        const double t2 = R ? tau.x * tau.x : fma(tau.x, tau.x, tau.y * tau.y);
        if (lane == 0) sm.alpha = -0.5 * t2 * (sm.vav - 2.0 * dot);
      }
    }
    // the multipliers in fixed point against chunk ch, whose columns have exponents of their own: kt and kq are the
    // largest products' exponents
    auto multipliers = [&](int ch, int& kt, int& kq) {
      const bool on = (lane & (NT - 1)) < j;
      const int ev = on ? fixed_exp(ch, lane) : 0;
      const int et = high_word<R>(tm) >> 20, eq = high_word<R>(qm) >> 20;
      kt = __reduce_max_sync(0xffffffffu, on ? et + ev : 0);
      kq = __reduce_max_sync(0xffffffffu, on ? eq + ev : 0);
      sm.tf[warp][lane] = fixed_point<R>(tm, kt - ev);
      sm.qf[warp][lane] = fixed_point<R>(qm, kq - ev);
      if (__any_sync(0xffffffffu, on && (ev == 0x7ff || et == 0x7ff))) kt = EXP_BAD;
      if (__any_sync(0xffffffffu, on && (ev == 0x7ff || eq == 0x7ff))) kq = EXP_BAD;
      __syncwarp();
    };
    // columns c0, c0 + step, ... of W and V into a row's two sums
    auto corrections = [&](int ch, int from, int step, Dot<R>& dy, Dot<R>& da) {
      const int4* src = RES ? wvs + (int64_t)(ch / C) * TILE_EL + lane : ws.vf + (int64_t)ch * 2 * NT * TS + lane;
      constexpr int LD = RES ? TILE_LD : TS;
#pragma unroll 2
      for (int c = from; c < j; c += step) {
        const int4 wq = RES ? src[c * LD] : ld_fixed<R>(src + c * LD);
        const int4 vq = RES ? src[(NT + c) * LD] : ld_fixed<R>(src + (NT + c) * LD);
        dy.add(wq, sm.tf[warp][c]);
        dy.add(vq, sm.tf[warp][NT + c]);
        if (next) {
          da.add(wq, sm.qf[warp][c]);
          da.add(vq, sm.qf[warp][NT + c]);
        }
      }
      dy.close(false);
      da.close(false);
    };
    // slots q, q + 4, ... of a row's y
    auto slots = [&](int ch, int q) {
      const int r = ch * 32 + lane;
      double2 y = zero2();
      if (!triv && r > j && r < M) {
#pragma unroll 4
        for (int s = q; s < nt; s += PW) y = add<R>(y, ldc<R>(ws.Yp + (int64_t)s * n + r));
      }
      return y;
    };
    // the row's entry of W's column j, from the sums
    auto w_entry = [&](int ch, double2 y, const Dot<R>& dy, int kt) {
      const int r = ch * 32 + lane;
      const double al = triv ? 0.0 : sm.alpha;
      double2 wv = zero2();
      if (r > j && r < M && !triv) {
        const double2 v = sv[r], d = dy.value(kt);
        y = make_double2(y.x - d.x, R ? 0.0 : y.y - d.y);
        wv = mul<R>(tau, y);
        wv.x = fma(al, v.x, wv.x);
        if constexpr (!R) wv.y = fma(al, v.y, wv.y);
      }
      return wv;
    };
    auto put_w = [&](int ch, double2 wv) {
      const int r = ch * 32 + lane;
      if (r > j && r < M) {
        st<R>(W + (int64_t)j * n + c0 + r, wv);
        st<R>(ws.VW + (int64_t)r * 2 * NT + j, wv);
      }
      const int emax = __reduce_max_sync(0xffffffffu, high_word<R>(wv)) >> 20;
      put_fixed(ch, j, fixed_point<R>(wv, emax), emax);
    };
    // the next column's entry but for W's column j, and with it
    auto a_entry = [&](int ch, const Dot<R>& da, int kq) {
      const int r = ch * 32 + lane;
      const double al = triv ? 0.0 : sm.alpha;
      const double2 wrow = triv ? zero2() : make_double2(sm.wrow.x + al, sm.wrow.y);
      double2 a = zero2();
      if (r > j && r < M && next) {
        const double2 d = da.value(kq);
        a = ld<R>(A + r + (int64_t)(j + 1) * n);
        a = make_double2(a.x - d.x, R ? 0.0 : a.y - d.y);
        a = fms_cj<R>(sv[r], wrow, a);
      }
      return a;
    };
    auto put_a = [&](int ch, double2 a, double2 wv) {
      const int r = ch * 32 + lane;
      if (!next) return;
      if (r > j && r < M) {
        a.x -= wv.x;                                       // V at the pivot row is 1
        if constexpr (!R) a.y -= wv.y;
        if (r == j + 1) {
          a.y = 0.0;
          ws.d[k + 1] = a.x;
        }
        st<R>(ws.xc + r, a);
      }
      double s = r >= j + 3 && r < M ? (R ? a.x * a.x : fma(a.x, a.x, a.y * a.y)) : 0.0;
      s = warp_sum<true>(make_double2(s, 0.0)).x;
      if (lane == 0) ws.sN[ch] = s;
    };
    if constexpr (RES) {
      for (int ch = rank, i = 0; ch < nt; ch += C, ++i) {
        char* e = eps + (int64_t)i * EPS;
        if (warp >= PW) {                                    // half of the warps sum the slots, half the corrections
          reinterpret_cast<double2*>(e)[(warp - PW) * TS + lane] = slots(ch, warp - PW);
        } else {
          int kt, kq;
          Dot<R> dy, da;
          multipliers(ch, kt, kq);
          corrections(ch, warp, PW, dy, da);
          long long* d = reinterpret_cast<long long*>(e + PW * 16 * TS) + warp * 8 * TS + lane;
          dy.put(d, TS);
          da.put(d + 4 * TS, TS);
          if (warp == 0 && lane < 2) wve[i * (2 * NT + 2) + 2 * NT + lane] = lane ? kq : kt;
          __syncwarp();
        }
      }
      __syncthreads();
      // two warps a chunk: W's column, and the next column
      for (int i0 = 0; rank + C * i0 < nt; i0 += NWP / 2) {
        const int i = i0 + (warp >> 1), ch = rank + C * i;
        const bool have = ch < nt;
        // W's entries for the other warp, in turn, where the multipliers were
        double2* wx = reinterpret_cast<double2*>(sm.tf) + ((i0 / (NWP / 2) & 1) * (NWP / 2) + (warp >> 1)) * 32;
        const char* e = eps + (int64_t)i * EPS;
        const int* ke = wve + i * (2 * NT + 2) + 2 * NT;
        const long long* d = reinterpret_cast<const long long*>(e + PW * 16 * TS) + (warp & 1) * 4 * TS + lane;
        double2 x = zero2();
        if (have) {
          Dot<R> z;
#pragma unroll
          for (int q = 0; q < PW; ++q) z.take(d + q * 8 * TS, TS);
          if ((warp & 1) == 0) {
            const double2* y = reinterpret_cast<const double2*>(e) + lane;
            x = w_entry(ch, sum4<R>(y[0], y[TS], y[2 * TS], y[3 * TS]), z, ke[0]);
            wx[lane] = x;
          } else {
            x = a_entry(ch, z, ke[1]);
          }
        }
        __syncthreads();
        if (have) {
          if ((warp & 1) == 0) put_w(ch, x);
          else put_a(ch, x, wx[lane]);
        }
      }
    } else {
      __syncthreads();
      for (int ch = first; ch < nt; ch += stride) {
        int kt, kq;
        Dot<R> dy, da;
        multipliers(ch, kt, kq);
        corrections(ch, 0, 1, dy, da);
        const double2 y = sum4<R>(slots(ch, 0), slots(ch, 1), slots(ch, 2), slots(ch, 3));
        const double2 wv = w_entry(ch, y, dy, kt), a = a_entry(ch, da, kq);
        put_w(ch, wv);
        put_a(ch, a, wv);
        __syncwarp();
      }
    }
    __syncthreads();
  }
  // slices of the rows below the panel: z = [V W], both operands; four warps a chunk.  A row has one exponent, and V's
  // entries are at most 1 while W's have the matrix's scale: V 2^k and W 2^-k meet halfway, and V W^H is the same.
  if (M - w > 1) {
    const int part = warp & 3;
    int em = 0;
    for (int t = lane; t < ntile; t += 32) em = max(em, ws.fe[t]);
    em = __reduce_max_sync(0xffffffffu, em);
    const int half = em == 0x7ff ? 0 : (em - 1022) / 2;
    int* hms = reinterpret_cast<int*>(sm.part);             // a warp's 32 high words
    for (int i = 0; rank + C * i < nt; i += NWP / 4) {
      const int ch = rank + C * (i + (warp >> 2)), r = ch * 32 + lane;
      const bool mine = ch < nt && r >= w && r < M;
      const double2* vw = ws.VW + (int64_t)r * 2 * NT;
      double2 z[SE];
#pragma unroll
      for (int e = 0; e < SE; ++e) {
        const int q = part * SE + e;
        const int k = q < NT ? half : -half;
        z[e] = mine && (q & (NT - 1)) < w ? vw[q ^ NT] : zero2();
        z[e] = make_double2(halfway(z[e].x, k), R ? 0.0 : halfway(z[e].y, k));
      }
      hms[warp * 32 + lane] = high_word8(z);
      __syncthreads();
      const int* hm = hms + (warp & ~3) * 32 + lane;
      const int emax = max(max(hm[0], hm[32]), max(hm[64], hm[96])) >> 20;
      if (mine) slice_part(z, part, emax, c0 + r, ws.nr, ws.sa, ws.ea, ws.sb, ws.eb, true);
      __syncthreads();
    }
  }
}

template <bool RES>
__global__ void __launch_bounds__(RES ? PTR : PT, RES ? 1 : 4) k_tri_panel(Grp G, int c0, int C, int rt, int cpc, int grid,
                                                                  unsigned sve_off) {
  const int g = blockIdx.x / C, p = G.prob[g];
  if (!live(G, p)) return;
  if (c0 >= G.nvec[p] - 1) return;
  extern __shared__ __align__(16) char smem_raw[];
  PanelSm& sm = *reinterpret_cast<PanelSm*>(smem_raw);
  double2* sv = reinterpret_cast<double2*>(smem_raw + sizeof(PanelSm));
  const int rows = cdiv_d(G.nmax - c0, TS) * TS;
  int4* svf = reinterpret_cast<int4*>(sv + rows);
  double2* big = reinterpret_cast<double2*>(svf + rows);
  int* sve = reinterpret_cast<int*>(smem_raw + sve_off);
  if (threadIdx.x == 0) sm.dead = 0;
  // grid teams are resident (plan_panel)
  Team team{(int)(blockIdx.x % C), C, G.limits.team, RES && grid != 0, ws_of(G, g).bar + c0 / NT, 0u, G.status + p, &sm.dead};
  if (is_real(G, p))
    panel_body<true, RES>(G, g, p, c0, team, rt, cpc, sm, sv, svf, sve, big);
  else
    panel_body<false, RES>(G, g, p, c0, team, rt, cpc, sm, sv, svf, sve, big);
}

// ------------------------------------------------------------------ eigenvalues
__global__ void __launch_bounds__(256) k_bounds(Grp G) {
  const int g = blockIdx.x, p = G.prob[g];
  if (!live(G, p)) return;
  const int n = G.nvec[p], tid = threadIdx.x;
  const WS w = ws_of(G, g);
  __shared__ double red[3 * 8];
  if (n == 1 && tid == 0) w.d[0] = (G.H + G.hs_off[p])->x;     // no column, no panel
  __syncthreads();
  double lo = 1e300, hi = -1e300, emax = 0.0;
  for (int i = tid; i < n; i += 256) {
    const double ea = (i > 0) ? sqrt(w.e2[i - 1]) : 0.0;
    const double eb = (i < n - 1) ? sqrt(w.e2[i]) : 0.0;
    lo = fmin(lo, w.d[i] - ea - eb);
    hi = fmax(hi, w.d[i] + ea + eb);
    emax = fmax(emax, skn_sturm::row_max(w.d[i], i < n - 1 ? w.e2[i] : 0.0));
    w.d32[i] = (float)w.d[i];
    w.e232[i] = (i < n - 1) ? (float)w.e2[i] : 0.0f;
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, o));
  }
  if ((tid & 31) == 0) {
    red[tid >> 5] = lo;
    red[8 + (tid >> 5)] = hi;
    red[16 + (tid >> 5)] = emax;
  }
  __syncthreads();
  if (tid == 0) {
    for (int q = 1; q < 8; ++q) {
      red[0] = fmin(red[0], red[q]);
      red[8] = fmax(red[8], red[8 + q]);
      red[16] = fmax(red[16], red[16 + q]);
    }
    w.bnd[0] = red[0];
    w.bnd[1] = red[8];
    w.bnd[2] = red[16];
  }
  if (G.tri) {
    double* tri = G.tri + 4 * G.eig_off[p];
    for (int i = tid; i < n; i += 256) tri[i] = w.d[i];
    if (tid == 0) {
      tri[2 * n - 1] = 0.0;
      tri[4 * n - 2] = 0.0;
      tri[4 * n - 1] = 0.0;
    }
  }
}

// Bound by FP64 issue when a GPU is full of them; 16 CTAs per SM, so that 1000 problems of 128 orbitals are one round.
__global__ void __launch_bounds__(64, 16) k_eig(Grp G) {
  const int g = blockIdx.y, p = G.prob[g];
  const int n = G.nvec[p], j = blockIdx.x * 64 + threadIdx.x;
  const int st = G.status[p];
  if (st == SKN_ERR_CAPACITY || j >= n) return;
  double* out = G.eig + G.eig_off[p];
  if (st != SKN_OK) {                        // S not positive definite, or a wait that ran out
    out[j] = __longlong_as_double(0x7ff8000000000000LL);
    return;
  }
  const WS w = ws_of(G, g);
  const skn_sturm::Bounds B = skn_sturm::make_bounds(w.bnd[0], w.bnd[1], w.bnd[2], n);
  out[j] = skn_sturm::eigenvalue(w.d, w.e2, w.d32, w.e232, n, j, B);
}

// ------------------------------------------------------------------ host sequence
constexpr size_t SMEM_MAX = 227 * 1024;

// Shared memory of a panel over m rows: streamed, or (rt > 0) resident with rt tiles and cpc chunks per CTA; the exponents
// of v are its last part.
size_t panel_smem(int m, int rt, int cpc) {
  const size_t head = sizeof(PanelSm) + (size_t)cdiv(m, TS) * (TS * (sizeof(double2) + sizeof(int4)) + sizeof(int));
  if (rt == 0) return head + (size_t)PW * QT * TILE_LD * sizeof(int4);
  return head + (size_t)(rt + cpc) * TILE_EL * sizeof(int4) + (size_t)cpc * (EPS + (2 * NT + 2) * sizeof(int));
}

inline int pow2_below(int v, int most) {
  int c = 1;
  while (c < most && 2 * c <= v) c *= 2;
  return c;
}

// Clusters of C CTAs of either form that the GPU holds at once, per_sm CTAs to an SM: a cluster stays within one of its
// processor clusters, which are not all of 16 SMs or more (GB300, resident: 7 of 16, 8 of 12, 15 of 8).
int clusters_at_once(bool resident, int C, int per_sm, int sms) {
  static std::mutex lock;
  static std::map<std::array<int, 4>, int> known;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> hold(lock);
  int& n = known[{dev, (int)resident, C, per_sm}];
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)C * sms);
    cfg.blockDim = dim3(resident ? PTR : PT);
    cfg.dynamicSmemBytes = SMEM_MAX / per_sm - 2048;
    if (!resident) cfg.dynamicSmemBytes = std::min(cfg.dynamicSmemBytes, panel_smem(PANELS_MAX_N, 0, 0));    // its limit
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e = resident ? cudaOccupancyMaxActiveClusters(&n, k_tri_panel<true>, &cfg)
                                   : cudaOccupancyMaxActiveClusters(&n, k_tri_panel<false>, &cfg);
    if (e != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = std::max(1, sms * per_sm / (2 * C));
    }
  }
  return n;
}

// CTAs per problem over m rows, and the tiles of each when they are resident (0: streamed).  Resident: one CTA per SM,
// up to one per tile, if shared memory holds its part and all problems run at once.  A cluster's barrier takes about 1200
// clocks, a counter's 5000, so a grid team only from GRID_FROM CTAs: where a cluster holds the tiles too it is 1 to 4% faster
// (200 to 432 orbitals x 3 to 6 problems), and where it does not the grid team is 13% faster than streaming (640 x 3 to 6;
// with the line at 17 also 640 x 7 and 8, by 8 to 12%, and 432 x 7 and 8 2 to 4% slower).  Streamed, with the GPU to itself: the size whose
// rounds are the shortest, as a problem's time falls with its CTAs and a round that is nearly empty costs as much as a full
// one (492 orbitals x 300 problems 98 ms, with 10 CTAs for each SM 111; 320 x 456 54 and 56).  Beside other calls there are
// no rounds, and STREAM_PER_SM CTAs for each SM of its part (four are resident; the rest wait) even the calls out.  At 5, 10
// and 20 four mixed batches take 112.8, 111.1, 112.9; 21.7, 21.9, 21.8; 25.9, 25.5, 25.6; 28.1, 28.0, 28.5 ms: a flat
// optimum.  The terms of `cost` are estimates of what a wider cluster's barriers add, not fitted to anything.
constexpr int GRID_FROM = 24, STREAM_PER_SM = 10;
void plan_panel(int m, int n_prob, int sms, int all, int& C, int& rt) {
  const int nt = cdiv(m, TS), tiles = nt * (nt + 1) / 2;
  const int most = std::min(tiles, std::max(1, sms / n_prob));
  C = most;
  if (most < GRID_FROM)
    for (C = std::min(most, 16); C > 1 && clusters_at_once(true, C, 1, all) < n_prob;) --C;
  rt = cdiv(tiles, C);
  if ((int64_t)n_prob * C <= all && panel_smem(m, rt, cdiv(nt, C)) <= SMEM_MAX) return;
  rt = 0;
  if (sms < all) {
    C = pow2_below(std::min(std::max(1, STREAM_PER_SM * sms / n_prob), std::max(1, tiles / (2 * PW))), 16);
    return;
  }
  const int per_sm = std::max(1, std::min(4, (int)(SMEM_MAX / (panel_smem(m, 0, 0) + 1024))));
  double best = 0.0;
  for (int c = 1; c <= 16 && c <= std::max(1, tiles / (2 * PW)); c *= 2) {
    const int rounds = cdiv(n_prob, clusters_at_once(false, c, per_sm, all));
    const double cost = (double)rounds / c * (1.0 + 0.05 * (c > 1) + 0.03 * (c > 2) + 0.03 * (c > 4) + 0.03 * (c > 8));
    if (c == 1 || cost < best) {
      best = cost;
      C = c;
    }
  }
}

cudaError_t launch_panel(const Grp& G, int count, int c0, int sms, int all, cudaStream_t stream) {
  const int m = G.nmax - c0;
  int C, rt;
  plan_panel(m, count, sms, all, C, rt);
  const int cpc = cdiv(cdiv(m, TS), C);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)count * C);
  cfg.blockDim = dim3(rt ? PTR : PT);
  cfg.dynamicSmemBytes = panel_smem(m, rt, cpc);
  cfg.stream = stream;
  const int grid = C > 16;
  cudaLaunchAttribute at[1];
  if (grid) {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  } else {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  }
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const unsigned sve_off = (unsigned)(cfg.dynamicSmemBytes - sizeof(int) * cdiv(m, TS));
  const int nt = cdiv(m, TS);
  k_fixed<<<dim3((unsigned)(nt * (nt + 1) / 2), (unsigned)count), PT, 0, stream>>>(G, c0);
  return rt ? cudaLaunchKernelEx(&cfg, k_tri_panel<true>, G, c0, C, rt, cpc, grid, sve_off)
            : cudaLaunchKernelEx(&cfg, k_tri_panel<false>, G, c0, C, rt, cpc, grid, sve_off);
}

// One update of the first `count` problems: jc column tiles per CTA, so that the GPU gets about two CTAs per SM at
// least.
template <int SWEEP>
void launch_update(const Grp& G, int count, int c1, int sms, cudaStream_t stream) {
  const int m = G.nmax - c1, nI = cdiv(m, BM);
  const int jl = cdiv(m, BN), ja = SWEEP == 1 ? cdiv(G.nmax, BN) : 0;
  const int64_t tiles = (int64_t)count * nI * ((jl + BM / BN + 1) / 2 + ja);
  int jc = (int)(tiles / (2 * (int64_t)sms));
  jc = jc < 2 ? 2 : (jc > 32 ? 32 : jc);
  const int cl = cdiv(jl, jc), ca = ja ? cdiv(ja, jc) : 1;
  const int nlow = nI * cl;
  k_update<SWEEP><<<dim3((unsigned)(nlow + (ja ? nI * ca : 0)), (unsigned)count), UPD_THREADS, UPD_SMEM, stream>>>(
      G, c1, nlow, cl, ca, jc);
}

// sizes: the slots' n, descending.  A launch covers the slots that have columns at its panel.
cudaError_t run(const Grp& G, const int32_t* sizes, int budget, cudaStream_t stream) {
  const int n = G.nmax, T = cdiv(n, NB);
  const unsigned P = (unsigned)G.n_prob;
  int dev = 0, all = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&all, cudaDevAttrMultiProcessorCount, dev);
  const int sms = budget > 0 && budget < all ? budget : all;
  auto above = [&](int m) {                    // slots with more than m orbitals
    return (int)(std::lower_bound(sizes, sizes + G.n_prob, m, [](int a, int b) { return a > b; }) - sizes);
  };
  const int nt = cdiv(n, TS);
  k_init<<<dim3(cdiv(2 * n, 256), P), 256, 0, stream>>>(G);
  k_scan<<<dim3(cdiv(nt * nt, 8), P, 2), 256, 0, stream>>>(G);
  k_fix<<<dim3(cdiv(n, 256), P), 256, 0, stream>>>(G);
  for (int t = 0; t < T; ++t) {
    const int c0 = t * NB, m = n - c0 - NB;
    const int nrow = m > 0 ? cdiv(m, BM) : 0;
    const unsigned A = (unsigned)above(c0);
    k_potrf<<<A, 256, 0, stream>>>(G, c0);
    k_solve<1><<<dim3(nrow + cdiv(n, BM), A), SV_THREADS, SV_SMEM, stream>>>(G, c0, nrow);
    if (m > 0) launch_update<1>(G, above(c0 + NB), c0 + NB, sms, stream);
  }
  for (int t = 0; t < T; ++t) {
    const int c0 = t * NB, m = n - c0 - NB;
    const int nrow = cdiv(n - c0, BM), nl = m > 0 ? cdiv(m, BM) : 0;
    k_solve<2><<<dim3(nrow + nl, (unsigned)above(c0)), SV_THREADS, SV_SMEM, stream>>>(G, c0, nrow);
    if (m > 0) launch_update<2>(G, above(c0 + NB), c0 + NB, sms, stream);
  }
  for (int c0 = 0; c0 < n - 1; c0 += NT) {
    const cudaError_t e = launch_panel(G, above(c0 + 1), c0, sms, all, stream);
    if (e != cudaSuccess) return e;
    if (n - c0 - NT > 1) launch_update<3>(G, above(c0 + NT + 1), c0 + NT, sms, stream);
  }
  k_bounds<<<P, 256, 0, stream>>>(G);
  k_eig<<<dim3(cdiv(n, 64), P), 64, 0, stream>>>(G);
  return cudaPeekAtLastError();
}

cudaError_t set_attrs() {
  cudaError_t e = cudaFuncSetAttribute(k_tri_panel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_tri_panel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)panel_smem(PANELS_MAX_N, 0, 0));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_tri_panel<true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_tri_panel<false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_solve<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, SV_SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_solve<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, SV_SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_update<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, UPD_SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_update<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, UPD_SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_update<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, UPD_SMEM);
  return e;
}

}  // namespace

extern "C" int skn_eigh_panels_scratch_bytes(int n, int64_t* bytes) {
  if (!bytes || n < 1) return SKN_ERR_ARG;
  if (n > PANELS_MAX_N) return SKN_ERR_CAPACITY;
  *bytes = layout(n).stride;
  return SKN_OK;
}

static int panels_entry(int n_prob, const int32_t* sizes, const int32_t* prob, const int64_t* ws_off, const int32_t* nvec,
                        const int32_t* real, const int64_t* hs_off, const int64_t* eig_off, double* H, double* S,
                        double* eig, int32_t* status, double* tri, double* scratch, int64_t scratch_bytes, int sms,
                        Limits limits, cudaStream_t stream) {
  if (n_prob < 0 || sms < 0) return SKN_ERR_ARG;
  if (n_prob == 0) return SKN_OK;
  if (!sizes || !prob || !ws_off || !nvec || !hs_off || !eig_off || !H || !S || !eig || !status || !scratch)
    return SKN_ERR_ARG;
  if (sizes[0] < 1 || !std::is_sorted(sizes, sizes + n_prob, [](int a, int b) { return a > b; })) return SKN_ERR_ARG;
  if (sizes[0] > PANELS_MAX_N || n_prob > 65535 || scratch_bytes < layout(sizes[0]).stride) return SKN_ERR_CAPACITY;
  if ((reinterpret_cast<uintptr_t>(scratch) & 15) || (reinterpret_cast<uintptr_t>(H) & 15) ||
      (reinterpret_cast<uintptr_t>(S) & 15))
    return SKN_ERR_ARG;
  if (set_attrs() != cudaSuccess) return SKN_ERR_CUDA;
  Grp G{sizes[0], n_prob, limits, prob, ws_off, nvec, real, hs_off, eig_off, (double2*)H, (double2*)S, eig, status, tri,
        (char*)scratch, scratch_bytes};
  try {                                      // the occupancy table and its lock may throw
    return run(G, sizes, sms, stream) == cudaSuccess ? SKN_OK : SKN_ERR_CUDA;
  } catch (...) {
    return SKN_ERR_CUDA;
  }
}

extern "C" int skn_eigh_gen_panels(int n_prob, const int32_t* sizes, const int32_t* prob, const int64_t* ws_off,
                                   const int32_t* nvec, const int32_t* real, const int64_t* hs_off,
                                   const int64_t* eig_off, double* H, double* S, double* eig, int32_t* status,
                                   double* tri, double* scratch, int64_t scratch_bytes, int sms, cudaStream_t stream) {
  return panels_entry(n_prob, sizes, prob, ws_off, nvec, real, hs_off, eig_off, H, S, eig, status, tri, scratch,
                      scratch_bytes, sms, LIMITS, stream);
}

extern "C" int skn_eigh_gen_panels_limits(int n_prob, const int32_t* sizes, const int32_t* prob, const int64_t* ws_off,
                                          const int32_t* nvec, const int32_t* real, const int64_t* hs_off,
                                          const int64_t* eig_off, double* H, double* S, double* eig, int32_t* status,
                                          double* tri, double* scratch, int64_t scratch_bytes, int sms,
                                          const int32_t* polls, cudaStream_t stream) {
  if (!polls || polls[0] < 0 || polls[1] < 0 || polls[2] < 0) return SKN_ERR_ARG;
  const Limits limits{std::min(polls[0], LIMITS.solve), std::min(polls[1], LIMITS.update), std::min(polls[2], LIMITS.team)};
  return panels_entry(n_prob, sizes, prob, ws_off, nvec, real, hs_off, eig_off, H, S, eig, status, tri, scratch,
                      scratch_bytes, sms, limits, stream);
}
