// Generalized Hermitian eigenvalues of problems of up to 96 orbitals, one CTA per problem, all in shared memory.
//
//   1. B = L^-1 H beside the Cholesky factorisation S = L L^H: step k scales column k of S and row k of H and
//      updates the trailing triangle of S and all rows of H below;
//   2. C = B L^-H on the lower triangle, column by column;
//   3. Householder tridiagonalisation of C (LAPACK zhetd2 order);
//   4. eigenvalues of the tridiagonal (sturm.cuh), one thread each.
// The reference runs torch.linalg.cholesky / solve / matmul / eigh per k (slakonet/utils.py:741-783).
//
// GB300 notes.  An SM partition issues one FP64 warp instruction per 64 clocks (77 with all four busy), so a step
// lasts as long as its busiest warp, and lanes without an element cost as much as lanes with one.  Every O(n^2)
// loop therefore deals elements of a packed range over all threads, the product with the Householder vector
// deals (row, column range) pairs, and scalar chains (a root is 830 clocks, a quotient 1440, a reciprocal 550) run
// in one warp: the pivot of the next Cholesky step beside the others' update, by a warp that has that much less of
// it.  A call's problems are of one size class, so that as many CTAs as possible share an SM; which class and
// thread count a problem takes depends on its size alone, and so do its results.
// n = 40 x 164 problems took 1.35 ms with the column-by-column kernel (skn_eigh_gen_batched).
#include "skn_common.cuh"
#include "sturm.cuh"

namespace {

constexpr int SMALL_MAX_N = 96;

// ------------------------------------------------------------------ arithmetic (R: real parts only)
template <bool R> SKN_DEVINL double2 fma_(double2 a, double2 b, double2 c) {        // c + a b
  if constexpr (R) { c.x = fma(a.x, b.x, c.x); return c; } else return cfma(a, b, c);
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
template <bool R> SKN_DEVINL double2 scl(double2 a, double s) { return make_double2(a.x * s, R ? 0.0 : a.y * s); }
template <bool R> SKN_DEVINL double norm2(double2 a, double s) {                    // s + |a|^2
  return R ? fma(a.x, a.x, s) : fma(a.x, a.x, fma(a.y, a.y, s));
}

// Column j of a packed lower triangle of order n starts (at its diagonal) at tri_off(j, n).
SKN_DEVINL int tri_off(int j, int n) { return j * n - (j * (j - 1)) / 2; }

template <int T>
struct Shared {
  double2 *H, *S, *v, *w, *part;   // n x lda; packed lower triangle; vectors; (row, column range) sums
  double *rd, *d, *e2;
  double* red;                     // T / 32 + 8
  uint8_t* ranges;                 // n + 1: column ranges of the product with a vector of that length
  int lda;
};
// Bytes of dynamic shared memory for problems of up to n orbitals.  The partial sums of the tridiagonalisation lie
// on the triangle of S, which is done with by then (written back first where it is wanted).
inline size_t small_smem(int n) {
  const int lda = n | 1;
  const size_t tri = (size_t)n * (n + 1) / 2, part = 8 * (size_t)n;
  return 16 * ((size_t)n * lda + (tri > part ? tri : part) + 2 * (size_t)n) + 8 * (3 * (size_t)n + 16) + (size_t)n + 1;
}

template <int T> SKN_DEVINL void barrier() {
  if constexpr (T == 32) __syncwarp(); else __syncthreads();
}

// Unit diagonal for rows that are entirely zero (eighb's aux option, slakonet/utils.py:741-747).
template <int T>
SKN_DEVINL void aux_zero_rows(const Shared<T>& m, int n) {
  for (int r = threadIdx.x; r < 2 * n; r += T) {
    const bool h = r < n;
    const int i = h ? r : r - n;
    bool zero = true;
    for (int j = 0; j < n && zero; ++j) {
      const double2 a = h ? m.H[i + j * m.lda]
                          : m.S[j <= i ? tri_off(j, n) + i - j : tri_off(i, n) + j - i];
      zero = is_zero_bits(a.x) && is_zero_bits(a.y);
    }
    if (zero) {
      if (h) m.H[i + i * m.lda].x = 1.0; else m.S[tri_off(i, n)].x = 1.0;
    }
  }
}

// sqrt(a) and 1 / sqrt(a) from one reciprocal root (600 clocks; a root and a quotient are 830 + 550): inv is off by its own
// last place, the root a inv takes one Newton step on r^2 = a, r + (a - r^2) inv / 2, which squares that error, so the root
// is the rounded one or its neighbour.  A column is scaled by inv: within two last places of the quotient by the root.
SKN_DEVINL void roots(double a, double& root, double& inv) {
  inv = rsqrt(a);
  const double r = a * inv;
  root = fma(fma(-r, r, a), 0.5 * inv, r);
}
SKN_DEVINL void pivot(double a, double& dk, double& rd, bool& ok) {
  ok = (a > 0.0) && is_finite_bits(a);
  roots(ok ? a : 1.0, dk, rd);
}

// Elements e = start, start + step, ... of a packed range dealt without divisions: (r, c) with e = c w + r.
struct Deal {
  int r, c, dr, dc, w;
  SKN_DEVINL Deal(int start, int step, int width) : w(width) {
    c = start / w;
    r = start - c * w;
    dc = step / w;
    dr = step - dc * w;
  }
  SKN_DEVINL void next() {
    r += dr;
    c += dc;
    if (r >= w) {
      r -= w;
      ++c;
    }
  }
};
// The lower triangle of order m as a rectangle: column c and column m - 1 - c (m even, width m + 1), or column c and
// column m - c (m odd, width m) make one line.  (r, c) of it -> (i, j), i >= j.
SKN_DEVINL int fold_width(int m) { return m + 1 - (m & 1); }
SKN_DEVINL void fold(int m, int r, int c, int& i, int& j) {
  const int len = m - c;                     // of column c
  const bool tail = r >= len;
  j = tail ? m - 1 + (m & 1) - c : c;
  i = tail ? j + r - len : c + r;
}

// L (packed in S) and B = L^-1 H in place of H.  False (every thread) when S is not positive definite.
template <int T, bool R>
SKN_DEVINL bool factor(const Shared<T>& m, int n) {
  constexpr int W = T / 32;
  // FP64 instructions of a pivot's root and quotient, in units of a 32-element update (4 or 1 instructions each)
  constexpr int AHEAD = R ? 36 : 9;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int* bad = reinterpret_cast<int*>(m.red + W);
  if (tid == 0) {
    double dk, rd;
    bool ok;
    pivot(m.S[0].x, dk, rd, ok);
    m.S[0] = make_double2(dk, 0.0);
    m.rd[0] = rd;
    *bad = ok ? 0 : 1;
  }
  barrier<T>();
  for (int k = 0; k < n; ++k) {
    if (*bad) return false;
    const double rd = m.rd[k];
    const int mr = n - k - 1;
    double2* col = m.S + tri_off(k, n) + 1;
    for (int e = tid; e < mr + n; e += T) {
      if (e < mr) {
        const double2 l = scl<R>(col[e], rd);
        col[e] = l;
        m.v[e] = l;
      } else {
        double2* h = m.H + k + (e - mr) * m.lda;
        const double2 b = scl<R>(*h, rd);
        *h = b;
        m.w[e - mr] = b;
      }
    }
    barrier<T>();
    if (mr == 0) break;
    // chunks of 32 elements: the trailing triangle of S without its first entry, then mr x n of H
    const int tri = mr * (mr + 1) / 2, nel = tri - 1 + mr * n, nch = (nel + 31) >> 5;
    const int ahead = (k + 1) % W;                     // the warp that takes the next pivot
    if (warp == ahead) {
      double2* dg = m.S + tri_off(k + 1, n);
      if (lane == 0) {
        const double2 l = m.v[0];
        const double a = R ? fma(-l.x, l.x, dg->x) : fma(-l.y, l.y, fma(-l.x, l.x, dg->x));
        double dk, rdn;
        bool ok;
        pivot(a, dk, rdn, ok);
        *dg = make_double2(dk, 0.0);
        m.rd[k + 1] = rdn;
        if (!ok) *bad = 1;
      }
    }
    // that warp starts AHEAD chunks late
    int c0 = warp, step = W;
    int lo = 0;
    if constexpr (W > 1) {
      const int share = (nch + AHEAD + W - 1) / W;      // chunks per warp, the pivot counted as AHEAD of them
      const int mine = max(0, share - AHEAD);
      const int q = (warp - ahead + W) % W;             // 0: the pivot's warp
      lo = q == 0 ? 0 : mine + (q - 1) * share;
      c0 = lo;
      step = 1;
      const int hi = min(nch, q == 0 ? mine : lo + share);
      lo = hi;                                          // end of this warp's chunks
    } else {
      lo = nch;
    }
    double2* T22 = m.S + tri_off(k + 1, n);
    // elements [32 c0, 32 lo), the triangle first: its own numbering in memory order needs row and column
    const int e1 = min(lo * 32, nel), es = step * 32;
    int e = c0 * 32 + lane;
    for (; e < min(e1, tri - 1); e += es) {
      int i, j;
      tri_index(e + 1, mr, i, j);                       // packed order of the trailing triangle is memory order
      T22[e + 1] = fms_cj<R>(m.v[i], m.v[j], T22[e + 1]);
    }
    if (e < e1) {
      Deal q(e - (tri - 1), es, mr);
#pragma unroll 2
      for (; e < e1; e += es, q.next()) {
        double2* h = m.H + k + 1 + q.r + q.c * m.lda;
        *h = fms<R>(m.v[q.r], m.w[q.c], *h);
      }
    }
    barrier<T>();
  }
  return true;
}

// C = B L^-H on the lower triangle of H.
template <int T, bool R>
SKN_DEVINL void second(const Shared<T>& m, int n) {
  const int tid = threadIdx.x;
  for (int i = tid; i < n; i += T) m.H[i] = scl<R>(m.H[i], m.rd[0]);
  barrier<T>();
  for (int k = 0; k + 1 < n; ++k) {
    const int mr = n - k - 1, tri = mr * (mr + 1) / 2;
    const double2* L = m.S + tri_off(k, n) + 1;         // L[j, k], j > k
    const double2* C = m.H + k + 1 + k * m.lda;
    const double rdn = m.rd[k + 1];
    Deal q(tid, T, fold_width(mr));
#pragma unroll 2
    for (int e = tid; e < tri; e += T, q.next()) {
      int i, j;
      fold(mr, q.r, q.c, i, j);
      double2* h = m.H + k + 1 + i + (k + 1 + j) * m.lda;
      double2 a = fms_cj<R>(C[i], L[j], *h);
      if (j == 0) a = scl<R>(a, rdn);                   // column k + 1 is complete
      if (i == j) a.y = 0.0;
      *h = a;
    }
    barrier<T>();
  }
}

// Column ranges per row for the product with the Householder vector: the count, up to 8, that leaves the fewest
// lanes of the T threads without a (row, range) pair.
SKN_DEVINL int ranges(int m, int T) {
  int best = 1;
  float eff = 0.0f;
  for (int p = 1; p <= 8; ++p) {
    const int cols = (m + p - 1) / p, rounds = (m * p + T - 1) / T;
    const float f = (float)m / (float)(cols * rounds + p);      // work per thread, with the later sum of p parts
    if (f > eff) {
      eff = f;
      best = p;
    }
  }
  return best;
}

// One warp takes the norm and the reflector (one reciprocal root, one reciprocal), alternating between the
// partitions; sums over rows run in the warps that have rows.
template <int T, bool R>
SKN_DEVINL void tridiag(const Shared<T>& m, int n, double* tri) {
  constexpr int W = T / 32;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double* sc = m.red + W + 1;                           // tau (2), 1 / (alpha - beta) (2), trivial
  for (int k = 0; k < n - 1; ++k) {
    const int mr = n - k - 1, rw = (mr + 31) >> 5;      // rows, warps with rows
    double2* x = m.H + k + 1 + k * m.lda;
    if (warp == k % W) {
      double s = 0.0;
      for (int i = 1 + lane; i < mr; i += 32) s = norm2<R>(x[i], s);
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const double2 al = x[0];
      const bool triv = s == 0.0 && (R || al.y == 0.0);
      double nrm, inv;
      roots(triv ? 1.0 : norm2<R>(al, s), nrm, inv);
      const bool up = al.x >= 0.0;                      // beta = -nrm
      const double beta = triv ? al.x : (up ? -nrm : nrm), ib = up ? -inv : inv;
      const double dr = al.x - beta, di = R ? 0.0 : al.y;
      const double den = triv ? 0.0 : 1.0 / (R ? dr * dr : fma(dr, dr, di * di));
      if (lane == 0) {
        const double taur = triv ? 0.0 : -dr * ib, taui = (R || triv) ? 0.0 : -di * ib;
        sc[0] = taur;
        sc[1] = taui;
        sc[2] = dr * den;
        sc[3] = -di * den;
        sc[4] = triv ? 1.0 : 0.0;
        m.d[k] = m.H[k + k * m.lda].x;
        m.e2[k] = beta * beta;
        if (tri) {
          tri[n + k] = beta;
          tri[2 * n + 2 * k] = taur;
          tri[2 * n + 2 * k + 1] = taui;
        }
      }
    }
    barrier<T>();
    if (sc[4] != 0.0) {
      barrier<T>();                                     // everyone has read it
      if (tid == 0) m.H[(k + 1) * (m.lda + 1)].y = 0.0;
      continue;
    }
    for (int i = tid; i < mr; i += T) {
      const double2 v = i == 0 ? make_double2(1.0, 0.0) : mul<R>(x[i], make_double2(sc[2], sc[3]));
      m.v[i] = v;
      x[i] = v;
    }
    barrier<T>();
    // y = A22 v from the lower triangle: thread (row, range of columns)
    const double2* A = m.H + (k + 1) * (m.lda + 1);
    const int P = m.ranges[mr], cols = (mr + P - 1) / P;
    Deal q(tid, T, mr);
    for (int u = tid; u < mr * P; u += T, q.next()) {
      const int i = q.r, j0 = q.c * cols, j1 = min(mr, j0 + cols);
      double2 y = make_double2(0.0, 0.0);
#pragma unroll 4
      for (int j = j0; j < j1; ++j) {
        const bool up = j > i;
        double2 a = up ? A[j + i * m.lda] : A[i + j * m.lda];
        if constexpr (!R) a.y = cond_flip(a.y, up);
        y = fma_<R>(a, m.v[j], y);
      }
      m.part[u] = y;
    }
    barrier<T>();
    const double2 tau = make_double2(sc[0], sc[1]);
    if (warp < rw) {                                    // v^H A22 v, real; a thread has one row (n <= T)
      double pr = 0.0;
      if (tid < mr) {
        double2 y = m.part[tid];
        for (int u = 1; u < P; ++u) {
          y.x += m.part[u * mr + tid].x;
          if constexpr (!R) y.y += m.part[u * mr + tid].y;
        }
        const double2 v = m.v[tid];
        pr = R ? v.x * y.x : fma(v.x, y.x, v.y * y.y);
        m.w[tid] = mul<R>(tau, y);
      }
      for (int o = 16; o > 0; o >>= 1) pr += __shfl_xor_sync(0xffffffffu, pr, o);
      if (lane == 0) m.red[warp] = pr;
    }
    barrier<T>();
    if (tid < mr) {                                     // w = tau y - tau/2 (w^H v) v
      double pr = m.red[0];
      for (int u = 1; u < rw; ++u) pr += m.red[u];
      const double t2 = R ? tau.x * tau.x : fma(tau.x, tau.x, tau.y * tau.y);
      const double alpha = -0.5 * t2 * pr;
      double2 w = m.w[tid];
      const double2 v = m.v[tid];
      w.x = fma(alpha, v.x, w.x);
      if constexpr (!R) w.y = fma(alpha, v.y, w.y);
      m.w[tid] = w;
    }
    barrier<T>();
    const int tr = mr * (mr + 1) / 2;
    Deal f(tid, T, fold_width(mr));
#pragma unroll 2
    for (int e = tid; e < tr; e += T, f.next()) {
      int i, j;
      fold(mr, f.r, f.c, i, j);
      double2* a = m.H + k + 1 + i + (k + 1 + j) * m.lda;
      double2 t = fms_cj<R>(m.v[i], m.w[j], *a);
      t = fms_cj<R>(m.w[i], m.v[j], t);
      if (i == j) t.y = 0.0;
      *a = t;
    }
    barrier<T>();
  }
  if (tid == 0) m.d[n - 1] = m.H[(n - 1) * (m.lda + 1)].x;
  barrier<T>();
  if (tri) {
    for (int i = tid; i < n; i += T) tri[i] = m.d[i];
    if (tid == 0) {
      tri[2 * n - 1] = 0.0;
      tri[4 * n - 2] = 0.0;
      tri[4 * n - 1] = 0.0;
    }
  }
}

template <int T>
SKN_DEVINL void eigenvalues(const Shared<T>& m, int n, double* out) {
  const int tid = threadIdx.x;
  float* d32 = reinterpret_cast<float*>(m.part);        // the matrices are done with
  float* e232 = d32 + n;
  double* ext = reinterpret_cast<double*>(m.part + n);
  double lo = 1e300, hi = -1e300, emax = 0.0;
  barrier<T>();
  for (int i = tid; i < n; i += T) {
    const double ea = (i > 0) ? sqrt(m.e2[i - 1]) : 0.0;
    const double eb = (i < n - 1) ? sqrt(m.e2[i]) : 0.0;
    lo = fmin(lo, m.d[i] - ea - eb);
    hi = fmax(hi, m.d[i] + ea + eb);
    emax = fmax(emax, skn_sturm::row_max(m.d[i], i < n - 1 ? m.e2[i] : 0.0));
    d32[i] = (float)m.d[i];
    e232[i] = i < n - 1 ? (float)m.e2[i] : 0.0f;
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, o));
  }
  if ((tid & 31) == 0) {
    ext[3 * (tid >> 5)] = lo;
    ext[3 * (tid >> 5) + 1] = hi;
    ext[3 * (tid >> 5) + 2] = emax;
  }
  barrier<T>();
  for (int q = 0; q < T / 32; ++q) {
    lo = fmin(lo, ext[3 * q]);
    hi = fmax(hi, ext[3 * q + 1]);
    emax = fmax(emax, ext[3 * q + 2]);
  }
  const skn_sturm::Bounds B = skn_sturm::make_bounds(lo, hi, emax, n);
  for (int j = tid; j < n; j += T) out[j] = skn_sturm::eigenvalue(m.d, m.e2, d32, e232, n, j, B);
}

template <int T, bool R>
SKN_DEVINL void solve(const Shared<T>& m, int n, double2* Hg, double2* Sg, double* eig, int32_t* status, double* tri) {
  const int tid = threadIdx.x;
  for (int e = tid; e < n * n; e += T) {
    const int j = e / n, i = e - j * n;
    if (i >= j) {
      double2 h = Hg[e];
      const double2 s = Sg[e];
      if (R || i == j) h.y = 0.0;
      m.H[i + j * m.lda] = h;
      if (i > j) m.H[j + i * m.lda] = make_double2(h.x, flip_sign(h.y));
      m.S[tri_off(j, n) + i - j] = make_double2(s.x, R ? 0.0 : s.y);
    }
  }
  if (tid < n) m.ranges[tid + 1] = (uint8_t)ranges(tid + 1, T);      // n <= T
  barrier<T>();
  aux_zero_rows<T>(m, n);
  barrier<T>();
  if (!factor<T, R>(m, n)) {
    for (int j = tid; j < n; j += T) eig[j] = __longlong_as_double(0x7ff8000000000000LL);
    if (tid == 0) *status = SKN_ERR_NOT_SPD;
    return;
  }
  second<T, R>(m, n);
  if (tri) {
    for (int e = tid; e < n * n; e += T) {
      const int j = e / n, i = e - j * n;
      if (i >= j) Sg[e] = m.S[tri_off(j, n) + i - j];
    }
    barrier<T>();
  }
  tridiag<T, R>(m, n, tri);
  if (tri) {
    for (int e = tid; e < n * n; e += T) {
      const int j = e / n, i = e - j * n;
      if (i >= j) Hg[e] = m.H[i + j * m.lda];
    }
  }
  eigenvalues<T>(m, n, eig);
  if (tid == 0) *status = SKN_OK;
}

template <int T>
__global__ void __launch_bounds__(T) k_eigh_small(int max_n, const int32_t* __restrict__ prob,
                                                  const int32_t* __restrict__ nvec, const int32_t* __restrict__ real,
                                                  const int64_t* __restrict__ hs_off,
                                                  const int64_t* __restrict__ eig_off, double2* H, double2* S,
                                                  double* eig, int32_t* status, double* tri_all) {
  extern __shared__ __align__(16) char smem[];
  const int p = prob[blockIdx.x], n = nvec[p];
  if (n < 1 || n > max_n || hs_off[p] < 0 || eig_off[p] < 0) {
    if (threadIdx.x == 0) status[p] = n == 0 ? SKN_OK : SKN_ERR_CAPACITY;
    return;
  }
  Shared<T> m;
  m.lda = n | 1;
  const int tri = n * (n + 1) / 2;
  m.H = reinterpret_cast<double2*>(smem);
  m.S = m.H + n * m.lda;
  m.part = m.S;
  m.v = m.S + max(tri, 8 * n);
  m.w = m.v + n;
  m.rd = reinterpret_cast<double*>(m.w + n);
  m.d = m.rd + n;
  m.e2 = m.d + n;
  m.red = m.e2 + n;
  m.ranges = reinterpret_cast<uint8_t*>(m.red + 16);
  double* tr = tri_all ? tri_all + 4 * eig_off[p] : nullptr;
  double2 *Hg = H + hs_off[p], *Sg = S + hs_off[p];
  if (real != nullptr && real[p])
    solve<T, true>(m, n, Hg, Sg, eig + eig_off[p], status + p, tr);
  else
    solve<T, false>(m, n, Hg, Sg, eig + eig_off[p], status + p, tr);
}

template <int T>
cudaError_t launch(int n_prob, int max_n, const int32_t* prob, const int32_t* nvec, const int32_t* real,
                   const int64_t* hs_off, const int64_t* eig_off, double* H, double* S, double* eig, int32_t* status,
                   double* tri, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(k_eigh_small<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)small_smem(T == 32 ? 16 : T == 64 ? 32 : SMALL_MAX_N));
  if (e != cudaSuccess) return e;
  k_eigh_small<T><<<n_prob, T, small_smem(max_n), stream>>>(max_n, prob, nvec, real, hs_off, eig_off, (double2*)H,
                                                            (double2*)S, eig, status, tri);
  return cudaPeekAtLastError();
}

}  // namespace

extern "C" int skn_eigh_gen_small(int n_prob, int max_n, const int32_t* prob, const int32_t* nvec, const int32_t* real,
                                  const int64_t* hs_off, const int64_t* eig_off, double* H, double* S, double* eig,
                                  int32_t* status, double* tri, cudaStream_t stream) {
  if (n_prob < 0 || max_n < 1) return SKN_ERR_ARG;
  if (n_prob == 0) return SKN_OK;
  if (!prob || !nvec || !hs_off || !eig_off || !H || !S || !eig || !status) return SKN_ERR_ARG;
  if (max_n > SMALL_MAX_N) return SKN_ERR_CAPACITY;
  const cudaError_t e =
      max_n <= 16   ? launch<32>(n_prob, max_n, prob, nvec, real, hs_off, eig_off, H, S, eig, status, tri, stream)
      : max_n <= 32 ? launch<64>(n_prob, max_n, prob, nvec, real, hs_off, eig_off, H, S, eig, status, tri, stream)
                    : launch<128>(n_prob, max_n, prob, nvec, real, hs_off, eig_off, H, S, eig, status, tri, stream);
  return e == cudaSuccess ? SKN_OK : SKN_ERR_CUDA;
}
