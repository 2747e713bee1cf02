// Batched symmetric eigensolver for the small projected matrices of the
// Lanczos iteration, up to 384 rows one thread-block cluster per matrix
// (sym_eig_cluster_kernel), above that one CTA:
//   1. Householder reduction to tridiagonal form (Golub & Van Loan, Alg. 8.3.1),
//   2. multisection on Sturm sequence counts for the wanted eigenvalues
//      (Barth, Martin & Wilkinson 1967), several lanes per eigenvalue, with a
//      division-free count,
//   3. inverse iteration on the tridiagonal with partial pivoting (Peters &
//      Wilkinson 1971), all eigenvalues at once with the LU factors reused
//      across sweeps, and modified Gram-Schmidt inside clusters of
//      (near-)equal eigenvalues after every sweep,
//   4. back-transformation by the stored Householder reflectors.
// FP64 throughput is low on this GPU, so the sequential parts (counts,
// triangular solves) are arranged to issue as few FP64 instructions as
// possible and to keep every warp of the CTA busy.
#include <cfloat>
#include <cmath>
#include "cluster.cuh"
#include "dense.cuh"
#include "dfloat.cuh"

namespace lapy {

constexpr int kEigThreads = 256;

size_t sym_eig_work_doubles(int lda, int want) {
  return (size_t)lda * 4 + (size_t)want * 2 + (size_t)want * 5 * lda + 64;
}

__device__ __forceinline__ int exponent_field(double x) {
  return (__double2hiint(x) >> 20) & 0x7ff;
}

// Number of eigenvalues of the tridiagonal (d, e2 = e^2) below x, from the
// signs of its leading principal minors p_i = (d_i - x) p_{i-1} -
// e2_{i-1} p_{i-2} (the Sturm sequence; Wilkinson, The Algebraic Eigenvalue
// Problem, 1965, ch. 5): a sign change from p_{i-1} to p_i is a negative
// pivot of T - xI = LDL'.  The recurrence needs no division (the FP64 pipe is
// the bottleneck here).  The pair of latest minors is rescaled by a power of
// two whenever its larger exponent leaves [2^-400, 2^400], and a minor that
// comes out exactly zero is replaced, with its predecessor, by the pair
// (s, -2^-600 s), s = sign of the predecessor: a negative pivot of magnitude
// 2^-600, as the ratio form replaces a zero pivot by -pivmin.
__device__ __forceinline__ int sturm_count(const double* d, const double* e2, int n, double x) {
  double a = 1.0, b = d[0] - x;
  if (b == 0.0) b = -0x1p-600;
  int cnt = signbit(b) ? 1 : 0;
  for (int i = 1; i < n; ++i) {
    double c = fma(d[i] - x, b, -e2[i - 1] * a);
    if ((__double_as_longlong(c) << 1) == 0) {
      a = copysign(1.0, b);
      c = -0x1p-600 * a;
    } else {
      a = b;
    }
    cnt += (signbit(c) != signbit(a)) ? 1 : 0;
    b = c;
    const int em = max(exponent_field(a), exponent_field(b));
    if (em > 1023 + 400 || em < 1023 - 400) {
      const double s = __hiloint2double((2046 - em) << 20, 0);  // 2^(1023 - em)
      a *= s;
      b *= s;
    }
  }
  return cnt;
}

// LU with partial pivoting of the tridiagonal (d, e) minus theta*I (Peters &
// Wilkinson 1971).  Factors are stored with stride ld (one column per
// eigenvalue): the reciprocal pivots U0i, the two superdiagonals U1, U2 of U,
// the multipliers L and the row-swap flags P.  Pivots below `tiny` in
// magnitude are replaced by +-tiny.
__device__ void tri_factor(const double* d, const double* e, int n, double theta, double* U0i,
                           double* U1, double* U2, double* L, double* P, int ld, double tiny) {
  double x0 = d[0] - theta, x1 = (n > 1) ? e[0] : 0.0, x2 = 0.0;
  for (int k = 0; k < n - 1; ++k) {
    const double y0 = e[k], y1 = d[k + 1] - theta, y2 = (k + 2 < n) ? e[k + 1] : 0.0;
    const bool sw = fabs(x0) < fabs(y0);
    double p0 = sw ? y0 : x0;
    const double p1 = sw ? y1 : x1, p2 = sw ? y2 : x2;
    const double o0 = sw ? x0 : y0, o1 = sw ? x1 : y1, o2 = sw ? x2 : y2;
    if (fabs(p0) < tiny) p0 = (p0 < 0 ? -tiny : tiny);
    const double r = 1.0 / p0;
    const double l = o0 * r;
    const int64_t o = (int64_t)k * ld;
    P[o] = sw ? 1.0 : 0.0;
    L[o] = l;
    U0i[o] = r;
    U1[o] = p1;
    U2[o] = p2;
    x0 = o1 - l * p1;
    x1 = o2 - l * p2;
    x2 = 0.0;
  }
  if (fabs(x0) < tiny) x0 = (x0 < 0 ? -tiny : tiny);
  const int64_t o = (int64_t)(n - 1) * ld;
  U0i[o] = 1.0 / x0;
  U1[o] = 0.0;
  U2[o] = 0.0;
}

// Solve with the factors of tri_factor in place on y (stride ld).
__device__ void tri_solve(const double* U0i, const double* U1, const double* U2, const double* L,
                          const double* P, int n, int ld, double* y) {
  double yk = y[0];
  for (int k = 0; k < n - 1; ++k) {
    const int64_t o = (int64_t)k * ld;
    double yn = y[o + ld];
    if (P[o] != 0.0) { const double t = yk; yk = yn; yn = t; }
    y[o] = yk;
    yk = yn - L[o] * yk;
  }
  const int64_t ol = (int64_t)(n - 1) * ld;
  double z1 = yk * U0i[ol], z2 = 0.0;  // z_{k+1}, z_{k+2}
  y[ol] = z1;
  for (int k = n - 2; k >= 0; --k) {
    const int64_t o = (int64_t)k * ld;
    const double z = (y[o] - U1[o] * z1 - U2[o] * z2) * U0i[o];
    y[o] = z;
    z2 = z1;
    z1 = z;
  }
}

__global__ void __launch_bounds__(kEigThreads, 4) sym_eig_kernel(double* Aall, int lda,
                                                              const int32_t* nsize, int want,
                                                              double* theta_all, double* S_all,
                                                              double* work_all, size_t wstride,
                                                              const int32_t* active) {
  extern __shared__ double svec[];  // v and w of the current reflector, FP64 and double-float (4 lda)
  __shared__ double sh[32];
  __shared__ double s_tau, s_beta, s_K;
  __shared__ int s_skip;
  const int b = blockIdx.x;
  if (active && !active[b]) return;
  const int n = nsize[b];
  const int t = threadIdx.x;
  const int lane_e = t & 31, warp_e = t >> 5, nwarp_e = kEigThreads / 32;
  double* A = Aall + (int64_t)b * lda * lda;
  double* W = work_all + (int64_t)b * wstride;
  double* d = W;
  double* e = W + lda;
  double* tau = W + 2 * lda;
  double* e2 = W + 3 * lda;
  double* th = W + 4 * lda;                // want
  int* clus = (int*)(W + 4 * lda + want);  // 2 want ints: leader flags, cluster starts
  double* vecw = W + 4 * lda + 2 * want;   // 5 want lda: LU factors per eigenvalue
  double* theta = theta_all + (int64_t)b * want;
  double* S = S_all + (int64_t)b * lda * want;
  const int nw = min(want, n);

  // ---- 1. Householder tridiagonalisation (lower), A[i*lda + j].  The
  // trailing block A22 is held in double-float (the 8 bytes of an entry as
  // an FP32 pair): its product with the reflector and its rank-2 update, the
  // O(n^3) part, run on the FP32 pipe, 64x the FP64 rate here; scalars,
  // reflectors (written back as FP64 into row and column k) and the
  // tridiagonal stay FP64.
  float2* Af = reinterpret_cast<float2*>(A);
  for (int64_t q = t; q < (int64_t)n * n; q += kEigThreads) {
    const int64_t r = q / n, c = q - r * n;
    Af[r * lda + c] = df_split(A[r * lda + c]);
  }
  __syncthreads();
  for (int k = 0; k < n - 2; ++k) {
    // column k below the subdiagonal
    double s2 = 0.0;
    for (int i = k + 2 + t; i < n; i += kEigThreads) {
      const double x = df_to_double(Af[(int64_t)i * lda + k]);
      s2 += x * x;
    }
    s2 = block_sum(s2, sh);
    if (t == 0) {
      const double alpha = df_to_double(Af[(int64_t)(k + 1) * lda + k]);
      if (s2 == 0.0) {
        s_skip = 1;
        s_tau = 0.0;
        e[k] = alpha;
      } else {
        s_skip = 0;
        const double beta = -copysign(sqrt(alpha * alpha + s2), alpha);
        s_tau = (beta - alpha) / beta;
        s_beta = 1.0 / (alpha - beta);
        e[k] = beta;
      }
      tau[k] = s_tau;
      d[k] = df_to_double(Af[(int64_t)k * lda + k]);
    }
    __syncthreads();
    if (s_skip) continue;
    // v: v[k+1] = 1, v[i] = A[i][k] * s_beta, stored (FP64) in column k and,
    // for a contiguous copy read by the back-transformation, in row k (row
    // and column k are not touched by the later steps)
    const int m0 = k + 1;
    double* vs = svec;
    double* ws = svec + lda;
    float2* vsf = reinterpret_cast<float2*>(svec + 2 * lda);
    float2* wsf = reinterpret_cast<float2*>(svec + 3 * lda);
    for (int i = m0 + t; i < n; i += kEigThreads) {
      double vi;
      if (i == m0) vi = 1.0;
      else {
        vi = df_to_double(Af[(int64_t)i * lda + k]) * s_beta;
        A[(int64_t)i * lda + k] = vi;
      }
      A[(int64_t)k * lda + i] = vi;
      vs[i] = vi;
      vsf[i] = df_split(vi);
    }
    __syncthreads();
    // p = tau * A22 v: warp per row (A22 is kept symmetric, so row i is
    // column i), lanes along the row, two rows in flight per warp; the row
    // sums in double-float, reduced over the warp with the two-sum
    double pdot = 0.0;
    for (int i = m0 + warp_e; i < n; i += 2 * nwarp_e) {
      const int i2 = i + nwarp_e;
      const float2* Ai = Af + (int64_t)i * lda;
      const float2* Ai2 = Af + (int64_t)(i2 < n ? i2 : i) * lda;
      float h1 = 0.f, l1 = 0.f, h2 = 0.f, l2 = 0.f;
      for (int j = m0 + lane_e; j < n; j += 32) {
        const float2 vj = vsf[j];
        df_fma(Ai[j], vj, h1, l1);
        df_fma(Ai2[j], vj, h2, l2);
      }
      {
        float h = __fadd_rn(h1, l1), l = __fsub_rn(l1, __fsub_rn(h, h1));
        float g = __fadd_rn(h2, l2), m = __fsub_rn(l2, __fsub_rn(g, h2));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const float bh = __shfl_xor_sync(0xffffffffu, h, o), bl = __shfl_xor_sync(0xffffffffu, l, o);
          const float ch = __shfl_xor_sync(0xffffffffu, g, o), cl = __shfl_xor_sync(0xffffffffu, m, o);
          df_add(h, l, bh, bl);
          df_add(g, m, ch, cl);
        }
        h1 = h; l1 = l; h2 = g; l2 = m;
      }
      const double a1 = ((double)h1 + (double)l1) * s_tau;
      const double a2 = ((double)h2 + (double)l2) * s_tau;
      if (lane_e == 0) {
        ws[i] = a1;
        pdot += a1 * vs[i];
        if (i2 < n) {
          ws[i2] = a2;
          pdot += a2 * vs[i2];
        }
      }
    }
    pdot = block_sum(pdot, sh);
    if (t == 0) s_K = -0.5 * s_tau * pdot;
    __syncthreads();
    for (int i = m0 + t; i < n; i += kEigThreads) {  // w
      const double wi = ws[i] + s_K * vs[i];
      ws[i] = wi;
      wsf[i] = df_split(wi);
    }
    __syncthreads();
    // A22 -= v w' + w v' in double-float: warp per row, lanes along the row
    for (int i = m0 + warp_e; i < n; i += nwarp_e) {
      float2* Ai = Af + (int64_t)i * lda;
      const float2 vi = vsf[i], wi = wsf[i];
      for (int j = m0 + lane_e; j < n; j += 32) {
        float uh = 0.f, ul = 0.f;
        df_fma(vsf[j], wi, uh, ul);
        df_fma(wsf[j], vi, uh, ul);
        float2 a = Ai[j];
        df_add(a.x, a.y, -uh, -ul);
        Ai[j] = a;
      }
    }
    __syncthreads();
  }
  if (t == 0) {
    if (n >= 2) {
      d[n - 2] = df_to_double(Af[(int64_t)(n - 2) * lda + (n - 2)]);
      e[n - 2] = df_to_double(Af[(int64_t)(n - 1) * lda + (n - 2)]);
      tau[n - 2] = 0.0;
    }
    d[n - 1] = df_to_double(Af[(int64_t)(n - 1) * lda + (n - 1)]);
    if (n >= 1) e[n - 1] = 0.0;
  }
  __syncthreads();
  for (int i = t; i < n; i += kEigThreads) e2[i] = e[i] * e[i];
  __syncthreads();

  // ---- 2. bisection for the nw largest eigenvalues
  double gl = 0.0, gu = 0.0, emax2 = 0.0;
  {
    double lo = DBL_MAX, hi = -DBL_MAX, em = 0.0;
    for (int i = t; i < n; i += kEigThreads) {
      const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0);
      lo = fmin(lo, d[i] - r);
      hi = fmax(hi, d[i] + r);
      if (i < n - 1) em = fmax(em, e2[i]);
    }
    // block min/max via shared scratch
    __syncthreads();
    if (t < 32) sh[t] = DBL_MAX;
    __syncthreads();
    for (int o = 16; o > 0; o >>= 1) lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    if ((t & 31) == 0) sh[t >> 5] = lo;
    __syncthreads();
    if (t == 0) {
      double m = DBL_MAX;
      for (int w = 0; w < kEigThreads / 32; ++w) m = fmin(m, sh[w]);
      s_tau = m;
    }
    __syncthreads();
    gl = s_tau;
    __syncthreads();
    for (int o = 16; o > 0; o >>= 1) hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    if ((t & 31) == 0) sh[t >> 5] = hi;
    __syncthreads();
    if (t == 0) {
      double m = -DBL_MAX;
      for (int w = 0; w < kEigThreads / 32; ++w) m = fmax(m, sh[w]);
      s_tau = m;
    }
    __syncthreads();
    gu = s_tau;
    __syncthreads();
    for (int o = 16; o > 0; o >>= 1) em = fmax(em, __shfl_xor_sync(0xffffffffu, em, o));
    if ((t & 31) == 0) sh[t >> 5] = em;
    __syncthreads();
    if (t == 0) {
      double m = 0.0;
      for (int w = 0; w < kEigThreads / 32; ++w) m = fmax(m, sh[w]);
      s_tau = m;
    }
    __syncthreads();
    emax2 = s_tau;
    __syncthreads();
  }
  const double tnorm = fmax(fabs(gl), fabs(gu));
  const double pivmin = DBL_MIN * fmax(1.0, emax2) * 4.0;
  gl -= 4.0 * DBL_EPSILON * tnorm + 2 * pivmin;
  gu += 4.0 * DBL_EPSILON * tnorm + 2 * pivmin;
  // multisection: a group of G lanes per eigenvalue probes G interior points
  // of its interval and keeps the sub-interval where the count passes the
  // eigenvalue's index
  {
    int G = 1;
    while (G < 32 && 2 * G * nw <= kEigThreads) G *= 2;
    const int ngroup = kEigThreads / G, sub = t % G, gl0 = (t & 31) - sub;
    const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << gl0);
    const double frac = 1.0 / (double)(G + 1);
    for (int j = t / G; j < nw; j += ngroup) {
      const int idx = n - 1 - j;  // index from the bottom
      double lo = gl, hi = gu;
      for (int itb = 0; itb < 200; ++itb) {
        const double w = hi - lo;
        if (w <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + pivmin) break;
        const double x = lo + (double)(sub + 1) * (w * frac);
        const bool le = sturm_count(d, e2, n, x) <= idx;
        const unsigned m = (__ballot_sync(gmask, le) & gmask) >> gl0;
        // the probe just above the highest one at or below the eigenvalue
        const int kk = (m == 0u) ? 0 : 32 - __clz(m);
        const double nlo = (kk == 0) ? lo : lo + (double)kk * (w * frac);
        const double nhi = (kk == G) ? hi : lo + (double)(kk + 1) * (w * frac);
        if (nlo == lo && nhi == hi) break;
        lo = nlo;
        hi = nhi;
      }
      if (sub == 0) th[j] = 0.5 * (lo + hi);
    }
  }
  __syncthreads();

  // ---- 3. inverse iteration for all wanted eigenvalues at once (thread q
  // owns eigenvalue q); the vectors live in S (row-major, stride want) and
  // after each sweep the members of every cluster of close eigenvalues are
  // orthonormalised by modified Gram-Schmidt, one warp per cluster
  const int lane = t & 31, warp = t >> 5;
  const double ctol = 1e-7 * fmax(tnorm, DBL_MIN);
  const double tiny = DBL_EPSILON * fmax(tnorm, DBL_MIN);
  int* lead = clus + want;  // first member of every cluster
  for (int j = t; j < nw; j += kEigThreads) clus[j] = (j == 0) || (th[j - 1] - th[j] > ctol);
  __syncthreads();
  if (t == 0) {
    int c = 0;
    for (int j = 0; j < nw; ++j)
      if (clus[j]) lead[c++] = j;
    s_skip = c;  // number of clusters
  }
  double* Y = S;
  double* U0i = vecw;
  double* U1 = U0i + (int64_t)lda * want;
  double* U2 = U1 + (int64_t)lda * want;
  double* Lm = U2 + (int64_t)lda * want;
  double* Pv = Lm + (int64_t)lda * want;
  for (int q = t; q < nw; q += kEigThreads) {
    int j = q;
    while (j > 0 && !clus[j]) --j;
    // members of a cluster get shifts a few ulps apart (as LAPACK dstein)
    const double shift = th[q] - (double)(q - j) * 10.0 * DBL_EPSILON * fmax(fabs(th[j]), tnorm);
    tri_factor(d, e, n, shift, U0i + q, U1 + q, U2 + q, Lm + q, Pv + q, want, tiny);
    for (int i = 0; i < n; ++i) {  // deterministic start vector
      unsigned h = (unsigned)(i * 2654435761u) ^ (unsigned)(q * 40503u + 0x9e3779b9u);
      h ^= h >> 15; h *= 2246822519u; h ^= h >> 13;
      Y[(int64_t)i * want + q] = ((double)(h & 0xffffff) / 16777216.0) - 0.5;
    }
  }
  __syncthreads();
  const int ncl = s_skip;
  for (int itr = 0; itr < 4; ++itr) {
    for (int q = t; q < nw; q += kEigThreads) tri_solve(U0i + q, U1 + q, U2 + q, Lm + q, Pv + q, n, want, Y + q);
    __syncthreads();
    for (int c = warp; c < ncl; c += kEigThreads / 32) {
      const int j0 = lead[c], j1 = (c + 1 < ncl) ? lead[c + 1] : nw;
      for (int m = j0; m < j1; ++m) {
        for (int r = j0; r < m; ++r) {
          double dp = 0.0;
          for (int i = lane; i < n; i += 32) dp += Y[(int64_t)i * want + r] * Y[(int64_t)i * want + m];
          dp = warp_sum(dp);
          for (int i = lane; i < n; i += 32) Y[(int64_t)i * want + m] -= dp * Y[(int64_t)i * want + r];
        }
        double nrm = 0.0;
        for (int i = lane; i < n; i += 32) nrm += Y[(int64_t)i * want + m] * Y[(int64_t)i * want + m];
        nrm = warp_sum(nrm);
        const double inv = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
        for (int i = lane; i < n; i += 32) Y[(int64_t)i * want + m] *= inv;
      }
    }
    __syncthreads();
  }

  // ---- 4. back-transformation Y <- H_0 ... H_{n-3} Y, one reflector at a
  // time for all vectors (the reflector is read from its copy in row k):
  // column dots by (row part, vector) threads, then the rank-1 update.  Y is
  // held in double-float meanwhile (its O(n^2 nw) products run on the FP32
  // pipe); each reflector is split once into shared memory.
  constexpr int kBtCols = 64, kBtRows = kEigThreads / kBtCols;
  const int tx = t % kBtCols, ty = t / kBtCols;
  float2* part = reinterpret_cast<float2*>(svec);                 // kBtRows x want partial dots
  double* dps = svec + (int64_t)kBtRows * want;                   // want scaled dots
  float2* dpsf = reinterpret_cast<float2*>(dps + want);           // the same, double-float
  float2* vkf = reinterpret_cast<float2*>(dps + 2 * (int64_t)want);  // the reflector, double-float (lda)
  float2* Yf = reinterpret_cast<float2*>(Y);
  for (int i = ty; i < n; i += kBtRows)
    for (int q = tx; q < nw; q += kBtCols) Yf[(int64_t)i * want + q] = df_split(Y[(int64_t)i * want + q]);
  __syncthreads();
  for (int k = n - 3; k >= 0; --k) {
    const double tk = tau[k];
    if (tk == 0.0) continue;  // uniform: tau is in global memory, read by all
    const double* vk = A + (int64_t)k * lda;  // vk[k+1] = 1
    for (int i = k + 1 + t; i < n; i += kEigThreads) vkf[i] = df_split(vk[i]);
    __syncthreads();
    for (int q = tx; q < nw; q += kBtCols) {
      float h = 0.f, l = 0.f;
      for (int i = k + 1 + ty; i < n; i += kBtRows) df_fma(vkf[i], Yf[(int64_t)i * want + q], h, l);
      const float hh = __fadd_rn(h, l);
      part[ty * want + q] = make_float2(hh, __fsub_rn(l, __fsub_rn(hh, h)));
    }
    __syncthreads();
    for (int q = t; q < nw; q += kEigThreads) {
      float h = 0.f, l = 0.f;
      for (int r = 0; r < kBtRows; ++r) df_add(h, l, part[r * want + q].x, part[r * want + q].y);
      const double d = tk * ((double)h + (double)l);
      dps[q] = d;
      dpsf[q] = df_split(d);
    }
    __syncthreads();
    for (int i = k + 1 + ty; i < n; i += kBtRows) {
      const float2 vi = vkf[i];
      for (int q = tx; q < nw; q += kBtCols) {
        float uh = 0.f, ul = 0.f;
        df_fma(dpsf[q], vi, uh, ul);
        float2 y = Yf[(int64_t)i * want + q];
        df_add(y.x, y.y, -uh, -ul);
        Yf[(int64_t)i * want + q] = y;
      }
    }
    __syncthreads();
  }
  for (int i = ty; i < n; i += kBtRows)
    for (int q = tx; q < nw; q += kBtCols) Y[(int64_t)i * want + q] = df_to_double(Yf[(int64_t)i * want + q]);
  __syncthreads();
  // rows beyond n and columns beyond nw (if want > n) are zero
  for (int i = ty; i < lda; i += kBtRows)
    for (int q = tx; q < want; q += kBtCols)
      if (i >= n || q >= nw) Y[(int64_t)i * want + q] = 0.0;
  for (int q = t; q < want; q += kEigThreads) theta[q] = (q < nw) ? th[q] : 0.0;
}

// ---- the same eigensolver, one thread-block cluster per matrix -----------------
// The one-CTA kernel above keeps its matrix in global memory: a step of the
// Householder reduction is several passes over L2 with one CTA's loads in
// flight, and FP64 (two results per clock and SM) of all its eigenvalues runs
// on one SM.  Here the rows (double-float) are dealt round-robin to the CTAs
// of a cluster and stay in shared memory.  A step has two cluster barriers: the
// warp that owns row k forms the reflector and stores it in every CTA; every
// warp multiplies its rows with it and stores the results w in every CTA; every
// warp then updates its rows (w + K v formed in registers on the way), the one
// that owns row k + 1 first, so that the next reflector is formed while the
// other warps still update.  Eigenvalues, their inverse iteration (factors in
// shared memory) and the back-transformation (one warp per vector, held in
// registers) are split over the CTAs, clusters of close eigenvalues together.
constexpr int kSymWarps = 16;

__device__ __forceinline__ float2 df_mul(float2 a, float2 b) {
  float h = 0.f, l = 0.f;
  df_fma(a, b, h, l);
  const float s = __fadd_rn(h, l);
  return make_float2(s, __fsub_rn(l, __fsub_rn(s, h)));
}
// Sum of (h, l) over the warp's lanes, in every lane.
__device__ __forceinline__ float2 df_warp_sum(float h, float l) {
  const float s = __fadd_rn(h, l);
  l = __fsub_rn(l, __fsub_rn(s, h));
  h = s;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float bh = __shfl_xor_sync(0xffffffffu, h, o), bl = __shfl_xor_sync(0xffffffffu, l, o);
    df_add(h, l, bh, bl);
  }
  return make_float2(h, l);
}

// Sturm counts on the tridiagonal scaled to norm 1 (d, e2 = e^2 as pairs): in
// FP32 from the leading parts, and in double-float (x = xh + xl).  Both count
// the eigenvalues below x of a matrix within their rounding of this one; the
// minors are rescaled as in sturm_count.
__device__ __forceinline__ int sturm_count_f32(const float2* d, const float2* e2, int n, float x) {
  float a = 1.f, b = d[0].x - x;
  if (b == 0.f) b = -0x1p-60f;
  int cnt = b < 0.f;
  for (int i = 1; i < n; ++i) {
    float c = fmaf(d[i].x - x, b, -e2[i - 1].x * a);
    a = b;
    if (c == 0.f) {
      a = copysignf(1.f, b);
      c = -0x1p-60f * a;
    }
    cnt += (__float_as_int(c) ^ __float_as_int(a)) < 0;
    b = c;
    const int em = max((__float_as_int(a) >> 23) & 0xff, (__float_as_int(b) >> 23) & 0xff);
    if (em > 127 + 40 || em < 127 - 40) {
      const float s = __int_as_float((254 - em) << 23);
      a *= s;
      b *= s;
    }
  }
  return cnt;
}
__device__ __forceinline__ int sturm_count_df(const float2* d, const float2* e2, int n, float xh, float xl) {
  float2 a = make_float2(1.f, 0.f), b = d[0];
  df_add(b.x, b.y, -xh, -xl);
  if (b.x == 0.f) b = make_float2(-0x1p-80f, 0.f);
  int cnt = b.x < 0.f;
  for (int i = 1; i < n; ++i) {
    float2 t = d[i];
    df_add(t.x, t.y, -xh, -xl);
    float h = 0.f, l = 0.f;
    df_fma(t, b, h, l);
    df_fma(make_float2(-e2[i - 1].x, -e2[i - 1].y), a, h, l);
    const float s0 = __fadd_rn(h, l);
    float2 c = make_float2(s0, __fsub_rn(l, __fsub_rn(s0, h)));
    a = b;
    if (c.x == 0.f) {
      a = make_float2(copysignf(1.f, b.x), 0.f);
      c = make_float2(-0x1p-80f * a.x, 0.f);
    }
    cnt += (__float_as_int(c.x) ^ __float_as_int(a.x)) < 0;
    b = c;
    const int em = max((__float_as_int(a.x) >> 23) & 0xff, (__float_as_int(b.x) >> 23) & 0xff);
    if (em > 127 + 24 || em < 127 - 24) {
      const float s = __int_as_float((254 - em) << 23);
      a.x *= s; a.y *= s;
      b.x *= s; b.y *= s;
    }
  }
  return cnt;
}

// As tri_factor and tri_solve with the swap flags as bytes and without the
// second superdiagonal of U, which is e[k + 1] after a swap and zero otherwise
// (33 instead of 48 bytes per entry: the factors fit into shared memory).
__device__ void tri_factor_compact(const double* d, const double* e, int n, double theta, double* U0i, double* U1,
                                   double* L, unsigned char* P, int ld, double tiny) {
  double x0 = d[0] - theta, x1 = (n > 1) ? e[0] : 0.0;
  for (int k = 0; k < n - 1; ++k) {
    const double y0 = e[k], y1 = d[k + 1] - theta, y2 = (k + 2 < n) ? e[k + 1] : 0.0;
    const bool sw = fabs(x0) < fabs(y0);
    double p0 = sw ? y0 : x0;
    const double p1 = sw ? y1 : x1;
    if (fabs(p0) < tiny) p0 = (p0 < 0 ? -tiny : tiny);
    const double r = 1.0 / p0;
    const double l = (sw ? x0 : y0) * r;
    const int o = k * ld;
    P[o] = sw;
    L[o] = l;
    U0i[o] = r;
    U1[o] = p1;
    x0 = (sw ? x1 : y1) - l * p1;
    x1 = sw ? -l * y2 : y2;
  }
  if (fabs(x0) < tiny) x0 = (x0 < 0 ? -tiny : tiny);
  U0i[(n - 1) * ld] = 1.0 / x0;
}
__device__ void tri_solve_compact(const double* e, const double* U0i, const double* U1, const double* L,
                                  const unsigned char* P, int n, int ld, double* y) {
  double yk = y[0];
  for (int k = 0; k < n - 1; ++k) {
    const int o = k * ld;
    double yn = y[o + ld];
    if (P[o]) { const double t = yk; yk = yn; yn = t; }
    y[o] = yk;
    yk = yn - L[o] * yk;
  }
  double z1 = yk * U0i[(n - 1) * ld], z2 = 0.0;  // z_{k+1}, z_{k+2}
  y[(n - 1) * ld] = z1;
  for (int k = n - 2; k >= 0; --k) {
    const int o = k * ld;
    const double u2 = P[o] ? e[k + 1] : 0.0;  // (z2 = 0 at k = n - 2)
    const double z = (y[o] - U1[o] * z1 - u2 * z2) * U0i[o];
    y[o] = z;
    z2 = z1;
    z1 = z;
  }
}

struct SymLayout {  // shared memory, byte offsets (rows: also the inverse iteration's factors)
  int o_v, o_w, o_mail, o_d, o_e, o_e2, o_ds, o_es, o_tau, o_th, o_flag, o_rows;
  int rows_bytes;
};

template <int NC>  // 32 NC >= n
__global__ void __launch_bounds__(32 * kSymWarps, 1) sym_eig_cluster_kernel(double* Aall, int lda, const int32_t* nsize,
                                                                            int want, double* theta_all, double* S_all,
                                                                            double* work_all, size_t wstride,
                                                                            const int32_t* active, int exact, SymLayout lay) {
  extern __shared__ __align__(16) unsigned char smx[];
  __shared__ double s_bound[3];
  __shared__ float2 s_tau[2];
  __shared__ int s_range[2];
  const unsigned rank = cl_rank(), cs = cl_size();
  const int b = blockIdx.x / cs;
  if (active && !active[b]) return;  // every CTA of the cluster
  const int n = nsize[b];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  double* A = Aall + (int64_t)b * lda * lda;
  float2* Av = reinterpret_cast<float2*>(A);  // reflector k: row k, double-float
  double* W = work_all + (int64_t)b * wstride;
  double* theta = theta_all + (int64_t)b * want;
  double* S = S_all + (int64_t)b * lda * want;
  const int nw = min(want, n);
  float2* vb = reinterpret_cast<float2*>(smx + lay.o_v);      // two reflectors (alternating)
  float2* wb = reinterpret_cast<float2*>(smx + lay.o_w);      // tau A v
  float2* mail = reinterpret_cast<float2*>(smx + lay.o_mail); // every warp's part of w'v
  double* d = reinterpret_cast<double*>(smx + lay.o_d);
  double* e = reinterpret_cast<double*>(smx + lay.o_e);
  double* e2 = reinterpret_cast<double*>(smx + lay.o_e2);
  float2* ds = reinterpret_cast<float2*>(smx + lay.o_ds);    // d and e^2 scaled to norm 1, double-float
  float2* es = reinterpret_cast<float2*>(smx + lay.o_es);
  float2* tau = reinterpret_cast<float2*>(smx + lay.o_tau);
  double* th = reinterpret_cast<double*>(smx + lay.o_th);
  int* flag = reinterpret_cast<int*>(smx + lay.o_flag);       // want: first of a cluster of eigenvalues
  float2* Ar = reinterpret_cast<float2*>(smx + lay.o_rows);   // local row li: row li cs + rank

  const int nloc = (n + (int)cs - 1 - (int)rank) / (int)cs;
  for (int li = warp; li < nloc; li += kSymWarps) {
    const double* src = A + (int64_t)(li * (int)cs + (int)rank) * lda;
    for (int j = lane; j < n; j += 32) Ar[li * n + j] = df_split(src[j]);
  }
  cl_sync(cs);  // every CTA has read A (its rows are overwritten by reflectors) and runs

  // reflector of row k (its owner's warp): d, e, tau and v to global memory, v
  // and tau to every CTA
  auto reflector = [&](int k) {
    const float2* Ak = Ar + (k / (int)cs) * n;
    const int ck = (k + 1) >> 5;
    // all in double-float (an FP64 square root and division here were most of
    // a step's time), the column scaled by a power of two to entries of at
    // most 2: squares of entries at rounding level would leave FP32's range
    float2 x[NC];
    float big = 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int j = lane + 32 * c;
      x[c] = (c >= ck && j > k && j < n) ? Ak[j] : make_float2(0.f, 0.f);
      big = fmaxf(big, fabsf(x[c].x));
    }
    big = warp_max(big);
    const int ex = (__float_as_int(big) >> 23) & 0xff;  // 0: the column is zero (or far below rounding)
    const bool scale = ex > 0 && ex < 253;
    const float sc = __int_as_float((scale ? 254 - ex : 127) << 23);
    float h = 0.f, l = 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      x[c].x *= sc;
      x[c].y *= sc;
      if (c >= ck && lane + 32 * c > k + 1) df_fma(x[c], x[c], h, l);
    }
    const float2 sum = df_warp_sum(h, l);
    const float2 alpha = make_float2(Ak[k + 1].x * sc, Ak[k + 1].y * sc);
    float2 beta = alpha, tk = make_float2(0.f, 0.f), inv = make_float2(0.f, 0.f);
    if (scale && sum.x > 0.f) {
      // square root and reciprocals from their FP32 values by Newton steps on
      // the double-float residual
      float2 tt = sum;
      df_fma(alpha, alpha, tt.x, tt.y);
      const float y0 = rsqrtf(tt.x);
      float2 root = make_float2(tt.x * y0, 0.f);
#pragma unroll
      for (int it = 0; it < 2; ++it) {
        float2 res = tt;
        df_fma(make_float2(-root.x, -root.y), root, res.x, res.y);
        df_add(root.x, root.y, 0.5f * y0 * (res.x + res.y), 0.f);
      }
      auto recip = [](float2 x) {
        const float q = 1.f / x.x;
        float2 e1 = make_float2(1.f, 0.f);
        df_fma(make_float2(-q, 0.f), x, e1.x, e1.y);
        float2 r = make_float2(q, 0.f);
        df_add(r.x, r.y, q * (e1.x + e1.y), 0.f);
        return r;
      };
      const bool neg = alpha.x < 0.f;
      const float2 aa = neg ? make_float2(-alpha.x, -alpha.y) : alpha;
      float2 den = aa;
      df_add(den.x, den.y, root.x, root.y);
      inv = recip(den);
      if (neg) inv = make_float2(-inv.x, -inv.y);
      beta = neg ? root : make_float2(-root.x, -root.y);
      tk = df_mul(den, recip(root));  // (beta - alpha) / beta
    }
    const float rs = __int_as_float((scale ? ex : 127) << 23);  // 1 / sc
    if (lane == 0) {
      W[k] = df_to_double(Ak[k]);
      W[lda + k] = df_to_double(make_float2(beta.x * rs, beta.y * rs));
      reinterpret_cast<float2*>(W)[2 * lda + k] = tk;
    }
    float2* vk = vb + (k & 1) * n;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int j = lane + 32 * c;
      if (j > k && j < n) {
        const float2 v = j == k + 1 ? make_float2(1.f, 0.f) : df_mul(x[c], inv);
        Av[(int64_t)k * lda + j] = v;
        for (unsigned r = 0; r < cs; ++r)
          if (r == rank) vk[j] = v;
          else cl_store2(cl_map(smem_u32(vk + j), r), v.x, v.y);
      }
    }
    if (lane < (int)cs) {
      if (lane == (int)rank) s_tau[k & 1] = tk;
      else cl_store2(cl_map(smem_u32(&s_tau[k & 1]), lane), tk.x, tk.y);
    }
  };

  // ---- 1. Householder tridiagonalisation
  if (rank == 0 && warp == 0 && n > 2) reflector(0);
  for (int k = 0; k + 2 < n; ++k) {
    cl_sync(cs);
    const int m0 = k + 1, c0 = m0 >> 5;
    const float2* vk = vb + (k & 1) * n;
    const float2 tk = s_tau[k & 1];
    float2 v[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int j = lane + 32 * c;
      v[c] = (j >= m0 && j < n) ? vk[j] : make_float2(0.f, 0.f);
    }
    // this warp's rows at or after m0 (local index = warp mod kSymWarps)
    int l0 = m0 > (int)rank ? (m0 - (int)rank + (int)cs - 1) / (int)cs : 0;
    l0 += (warp - l0) & (kSymWarps - 1);
    // w = tau A v (two rows in flight) and w'v
    float ph = 0.f, pl = 0.f;
    for (int li = l0; li < nloc; li += 2 * kSymWarps) {
      const bool two = li + kSymWarps < nloc;
      const float2* A1 = Ar + li * n;
      const float2* A2 = two ? A1 + kSymWarps * n : A1;
      float h1 = 0.f, l1 = 0.f, h2 = 0.f, l2 = 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        if (c >= c0) {
          const int j = min(lane + 32 * c, n - 1);
          df_fma(A1[j], v[c], h1, l1);
          df_fma(A2[j], v[c], h2, l2);
        }
      }
      const float2 w1 = df_mul(tk, df_warp_sum(h1, l1)), w2 = df_mul(tk, df_warp_sum(h2, l2));
      const int i1 = li * (int)cs + (int)rank, i2 = i1 + kSymWarps * (int)cs;
      df_fma(w1, vk[i1], ph, pl);
      if (two) df_fma(w2, vk[i2], ph, pl);
      if (lane < (int)cs) {
        if (lane == (int)rank) {
          wb[i1] = w1;
          if (two) wb[i2] = w2;
        } else {
          cl_store2(cl_map(smem_u32(wb + i1), lane), w1.x, w1.y);
          if (two) cl_store2(cl_map(smem_u32(wb + i2), lane), w2.x, w2.y);
        }
      }
    }
    if (lane < (int)cs) {
      float2* at = mail + rank * kSymWarps + warp;
      if (lane == (int)rank) *at = make_float2(ph, pl);
      else cl_store2(cl_map(smem_u32(at), lane), ph, pl);
    }
    cl_sync(cs);
    float kh = 0.f, kl = 0.f;
    for (int i = lane; i < kSymWarps * (int)cs; i += 32) df_add(kh, kl, mail[i].x, mail[i].y);
    const float2 K = df_mul(make_float2(-0.5f * tk.x, -0.5f * tk.y), df_warp_sum(kh, kl));
    float2 w[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int j = lane + 32 * c;
      w[c] = (j >= m0 && j < n) ? wb[j] : make_float2(0.f, 0.f);
      df_fma(K, v[c], w[c].x, w[c].y);
    }
    // A22 -= v w' + w v'
    for (int li = l0; li < nloc; li += kSymWarps) {
      const int i = li * (int)cs + (int)rank;
      float2* Ai = Ar + li * n;
      const float2 vi = vk[i];
      float2 wi = wb[i];
      df_fma(K, vi, wi.x, wi.y);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int j = lane + 32 * c;
        if (c >= c0 && j < n) {
          float uh = 0.f, ul = 0.f;
          df_fma(v[c], wi, uh, ul);
          df_fma(w[c], vi, uh, ul);
          float2 a = Ai[j];
          df_add(a.x, a.y, -uh, -ul);
          Ai[j] = a;
        }
      }
      __syncwarp();
      if (i == m0 && m0 + 2 < n) reflector(m0);
    }
  }
  if (lane == 0) {  // the last two rows
    for (int i = max(0, n - 2); i < n; ++i) {
      if (i % (int)cs != (int)rank || (i / (int)cs) % kSymWarps != warp) continue;
      const float2* Ai = Ar + (i / (int)cs) * n;
      W[i] = df_to_double(Ai[i]);
      W[lda + i] = i + 1 < n ? df_to_double(Ai[i + 1]) : 0.0;
      W[2 * lda + i] = 0.0;
    }
  }
  cl_sync(cs);
  for (int i = t; i < n; i += blockDim.x) {
    const double x = __ldcg(W + lda + i);
    d[i] = __ldcg(W + i);
    e[i] = x;
    e2[i] = x * x;
    tau[i] = __ldcg(reinterpret_cast<const float2*>(W) + 2 * lda + i);
  }
  __syncthreads();

  // ---- 2. multisection for the nw largest eigenvalues, split over the CTAs
  if (warp == 0) {
    double lo = DBL_MAX, hi = -DBL_MAX, em = 0.0;
    for (int i = lane; i < n; i += 32) {
      const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0);
      lo = fmin(lo, d[i] - r);
      hi = fmax(hi, d[i] + r);
      if (i < n - 1) em = fmax(em, e2[i]);
    }
    for (int o = 16; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      em = fmax(em, __shfl_xor_sync(0xffffffffu, em, o));
    }
    if (lane == 0) {
      s_bound[0] = lo;
      s_bound[1] = hi;
      s_bound[2] = em;
    }
  }
  __syncthreads();
  double gl = s_bound[0], gu = s_bound[1];
  const double tnorm = fmax(fabs(gl), fabs(gu));
  const double pivmin = DBL_MIN * fmax(1.0, s_bound[2]) * 4.0;
  gl -= 4.0 * DBL_EPSILON * tnorm + 2 * pivmin;
  gu += 4.0 * DBL_EPSILON * tnorm + 2 * pivmin;
  const double rn = tnorm > 0.0 ? 1.0 / tnorm : 0.0;
  for (int i = t; i < n; i += blockDim.x) {
    ds[i] = df_split(d[i] * rn);
    es[i] = df_split(e2[i] * rn * rn);
  }
  __syncthreads();
  const int j0 = nw * (int)rank / (int)cs, j1 = nw * ((int)rank + 1) / (int)cs;
  {
    // A group of G lanes per eigenvalue probes G interior points a round: in
    // FP32 down to 2^-20 of the norm, from there, widened by the FP32 counts'
    // error (8 eps; twice that is taken), in double-float to 2^-42.  FP64
    // counts, which cost 20 times as much a round (270 ns a row of T), finish
    // only where the eigenvalues are a result (`exact`), from a verified bracket.
    int G = 2;
    while (G < 32 && 2 * G * (j1 - j0) <= 256) G *= 2;
    const int ngroup = (int)blockDim.x / G, sub = t % G, gl0 = lane - sub;
    const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << gl0);
    const float frac = 1.f / (float)(G + 1);
    for (int j = j0 + t / G; j < j1; j += ngroup) {
      const int idx = n - 1 - j;  // index from the bottom
      // probes at or below the eigenvalue, from each lane's count
      auto below = [&](bool le) {
        const unsigned m = (__ballot_sync(gmask, le) & gmask) >> gl0;
        return (m == 0u) ? 0 : 32 - __clz(m);
      };
      float fl = -1.0001f, fw = 2.0002f;
      while (fw > 0x1p-20f) {
        const int kk = below(sturm_count_f32(ds, es, n, fl + (float)(sub + 1) * (fw * frac)) <= idx);
        fl += (float)kk * (fw * frac);
        fw *= frac;
      }
      fl -= 0x1p-19f;
      fw += 0x1p-18f;
      float2 l2 = make_float2(fl, 0.f);
      // the bracket holds: no more than idx below its lower end, more below its upper
      const bool at_lo = sub == 0 ? sturm_count_df(ds, es, n, fl, 0.f) <= idx
                                  : sub == 1 ? sturm_count_df(ds, es, n, fl + fw, 0.f) > idx : true;
      const bool good = (__ballot_sync(gmask, at_lo) & gmask) == gmask;
      double lo = gl, hi = gu;
      if (good) {
        while (fw > 0x1p-42f) {
          float2 x = l2;
          df_add(x.x, x.y, (float)(sub + 1) * (fw * frac), 0.f);
          const int kk = below(sturm_count_df(ds, es, n, x.x, x.y) <= idx);
          df_add(l2.x, l2.y, (float)kk * (fw * frac), 0.f);
          fw *= frac;
        }
        lo = df_to_double(l2) * tnorm;
        hi = lo + (double)fw * tnorm;
      }
      if (exact || !good) {
        if (good) {  // widened by the double-float counts' error, then checked
          const double wide = 0x1p-41 * tnorm;
          const bool ok = sub == 0 ? sturm_count(d, e2, n, lo - wide) <= idx
                                   : sub == 1 ? sturm_count(d, e2, n, hi + wide) > idx : true;
          if ((__ballot_sync(gmask, ok) & gmask) == gmask) {
            lo -= wide;
            hi += wide;
          } else {
            lo = gl;
            hi = gu;
          }
        }
        for (int itb = 0; itb < 200; ++itb) {
          const double wd = hi - lo;
          if (wd <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + pivmin) break;
          const double step = wd / (double)(G + 1);
          const int kk = below(sturm_count(d, e2, n, lo + (double)(sub + 1) * step) <= idx);
          const double nlo = (kk == 0) ? lo : lo + (double)kk * step;
          const double nhi = (kk == G) ? hi : lo + (double)(kk + 1) * step;
          if (nlo == lo && nhi == hi) break;
          lo = nlo;
          hi = nhi;
        }
      }
      if (sub == 0) {
        const double v = 0.5 * (lo + hi);
        for (unsigned r = 0; r < cs; ++r)
          if (r == rank) th[j] = v;
          else cl_store(cl_map(smem_u32(th + j), r), v);
      }
    }
  }
  __syncwarp();
  cl_sync(cs);

  // ---- 3. inverse iteration; a cluster of close eigenvalues belongs to the CTA
  // whose share holds its first member
  const double ctol = 1e-7 * fmax(tnorm, DBL_MIN);
  const double tiny = DBL_EPSILON * fmax(tnorm, DBL_MIN);
  for (int j = t; j < nw; j += blockDim.x) flag[j] = (j == 0) || (th[j - 1] - th[j] > ctol);
  __syncthreads();
  if (t < 2) {
    int j = t == 0 ? j0 : j1;
    while (j < nw && !flag[j]) ++j;
    s_range[t] = j;
  }
  __syncthreads();
  const int qa = s_range[0], qb = s_range[1], cnt = qb - qa;
  const bool on_chip = (int64_t)33 * (cnt | 1) * n <= lay.rows_bytes;
  const int ldq = on_chip ? cnt | 1 : want;
  double* vecw = W + 4 * lda + 2 * want;
  double* fac = on_chip ? reinterpret_cast<double*>(Ar) : vecw + qa;
  const int64_t fs = on_chip ? (int64_t)ldq * n : (int64_t)lda * want;
  double *U0i = fac, *U1 = fac + fs, *Lm = fac + 2 * fs;
  double* Y = on_chip ? fac + 3 * fs : S + qa;
  unsigned char* Pv = reinterpret_cast<unsigned char*>(on_chip ? fac + 4 * fs : vecw + 3 * fs) + (on_chip ? 0 : qa);
  for (int ql = t; ql < cnt; ql += blockDim.x) {
    const int q = qa + ql;
    int j = q;
    while (j > 0 && !flag[j]) --j;
    // members of a cluster get shifts a few ulps apart (as LAPACK dstein)
    const double shift = th[q] - (double)(q - j) * 10.0 * DBL_EPSILON * fmax(fabs(th[j]), tnorm);
    tri_factor_compact(d, e, n, shift, U0i + ql, U1 + ql, Lm + ql, Pv + ql, ldq, tiny);
    for (int i = 0; i < n; ++i) {  // deterministic start vector
      unsigned h = (unsigned)(i * 2654435761u) ^ (unsigned)(q * 40503u + 0x9e3779b9u);
      h ^= h >> 15; h *= 2246822519u; h ^= h >> 13;
      Y[(int64_t)i * ldq + ql] = ((double)(h & 0xffffff) / 16777216.0) - 0.5;
    }
  }
  __syncthreads();
  for (int itr = 0; itr < 4; ++itr) {
    for (int ql = t; ql < cnt; ql += blockDim.x)
      tri_solve_compact(e, U0i + ql, U1 + ql, Lm + ql, Pv + ql, n, ldq, Y + ql);
    __syncthreads();
    int c = 0;  // number of the cluster, dealt round-robin to the warps
    for (int a0 = qa; a0 < qb; ++c) {
      int a1 = a0 + 1;
      while (a1 < qb && !flag[a1]) ++a1;
      if (c % kSymWarps == warp) {
        for (int m = a0 - qa; m < a1 - qa; ++m) {
          for (int r = a0 - qa; r < m; ++r) {
            double dp = 0.0;
            for (int i = lane; i < n; i += 32) dp += Y[(int64_t)i * ldq + r] * Y[(int64_t)i * ldq + m];
            dp = warp_sum(dp);
            for (int i = lane; i < n; i += 32) Y[(int64_t)i * ldq + m] -= dp * Y[(int64_t)i * ldq + r];
          }
          double nrm = 0.0;
          for (int i = lane; i < n; i += 32) nrm += Y[(int64_t)i * ldq + m] * Y[(int64_t)i * ldq + m];
          nrm = warp_sum(nrm);
          const double inv = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
          for (int i = lane; i < n; i += 32) Y[(int64_t)i * ldq + m] *= inv;
        }
      }
      a0 = a1;
    }
    __syncthreads();
  }

  // ---- 4. back-transformation Y <- H_0 ... H_{n-3} Y, a warp per vector in
  // double-float registers, the next reflector's loads in flight
  for (int ql = warp; ql < cnt; ql += kSymWarps) {
    float2 y[NC], v[NC], vn[NC];
    auto load = [&](int k, float2 (&x)[NC]) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int j = lane + 32 * c;
        x[c] = (k >= 0 && j > k && j < n) ? __ldcg(Av + (int64_t)k * lda + j) : make_float2(0.f, 0.f);
      }
    };
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int j = lane + 32 * c;
      y[c] = j < n ? df_split(Y[(int64_t)j * ldq + ql]) : make_float2(0.f, 0.f);
    }
    load(n - 3, v);
    for (int k = n - 3; k >= 0; --k) {
      load(k - 1, vn);
      float h = 0.f, l = 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) df_fma(v[c], y[c], h, l);
      const float2 s = df_mul(tau[k], df_warp_sum(h, l));
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        float uh = 0.f, ul = 0.f;
        df_fma(s, v[c], uh, ul);
        df_add(y[c].x, y[c].y, -uh, -ul);
        v[c] = vn[c];
      }
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int j = lane + 32 * c;
      if (j < n) S[(int64_t)j * want + qa + ql] = df_to_double(y[c]);
    }
  }
  // rows beyond n and columns beyond nw (if want > n) are zero
  for (int64_t i = (int64_t)rank * blockDim.x + t; i < (int64_t)lda * want; i += (int64_t)cs * blockDim.x)
    if (i / want >= n || i % want >= nw) S[i] = 0.0;
  if (rank == 0)
    for (int q = t; q < want; q += blockDim.x) theta[q] = (q < nw) ? th[q] : 0.0;
}

// Shared memory of the cluster kernel for matrices of up to n rows.
static size_t sym_layout(int n, int cs, int want, SymLayout* lay) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += (bytes + 15) & ~size_t(15);
    return (int)o;
  };
  lay->o_v = take(16 * (size_t)n);
  lay->o_w = take(8 * (size_t)n);
  lay->o_mail = take(8 * (size_t)kSymWarps * cs);
  lay->o_d = take(8 * (size_t)n);
  lay->o_e = take(8 * (size_t)n);
  lay->o_e2 = take(8 * (size_t)n);
  lay->o_ds = take(8 * (size_t)n);
  lay->o_es = take(8 * (size_t)n);
  lay->o_tau = take(8 * (size_t)n);
  lay->o_th = take(8 * (size_t)want);
  lay->o_flag = take(4 * (size_t)want);
  lay->rows_bytes = (int)(8 * (size_t)((n + cs - 1) / cs) * n);
  lay->o_rows = take((size_t)lay->rows_bytes);
  return off;
}

static int launch_sym_cluster(int nmat, int cs, int n, double* A, int lda, const int32_t* nsize, int want,
                              double* theta, double* S, double* work, const int32_t* active, bool exact, cudaStream_t stream,
                              bool* launched) {
  *launched = false;
  constexpr size_t kMax = 226 * 1024;
  SymLayout lay;
  size_t smem = sym_layout(n, cs, want, &lay);
  if (smem > kMax) return LAPY_OK;
  // what is free goes to the inverse iteration's factors
  lay.rows_bytes += (int)((kMax - smem) & ~size_t(15));
  lay.rows_bytes = std::min<int64_t>(lay.rows_bytes, std::max<int64_t>(8 * (int64_t)((n + cs - 1) / cs) * n,
                                                                      (int64_t)33 * ((want + cs - 1) / cs | 1) * n));
  smem = (size_t)lay.o_rows + (size_t)lay.rows_bytes;
  auto kern = n <= 128 ? sym_eig_cluster_kernel<4> : n <= 256 ? sym_eig_cluster_kernel<8> : sym_eig_cluster_kernel<12>;
  LAPY_CUDA_TRY(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMax));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(nmat * cs));
  cfg.blockDim = dim3(32 * kSymWarps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)cs;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int resident = 0;
  if (cudaOccupancyMaxActiveClusters(&resident, (const void*)kern, &cfg) != cudaSuccess || resident < 1) {
    cudaGetLastError();
    return LAPY_OK;
  }
  LAPY_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, A, lda, nsize, want, theta, S, work, sym_eig_work_doubles(lda, want),
                                   active, exact ? 1 : 0, lay));
  *launched = true;
  return lapy_check_launch("sym_eig_cluster_kernel");
}

int sym_eig_top(int nmat, double* A, int lda, const int32_t* nsize, int nmax, int want, double* theta,
                double* S, double* work, const int32_t* active, bool exact, cudaStream_t stream) {
  if (nmat <= 0) return LAPY_OK;
  if (nmax > 0 && nmax <= 384 && nmax <= lda) {
    // the smallest cluster whose CTAs hold the rows, doubled while CTAs keep
    // 24 rows or more and all matrices still run at once
    int cs = 1;
    SymLayout lay;
    while (cs < 8 && sym_layout(nmax, cs, want, &lay) > 226 * 1024) cs *= 2;
    while (cs < 8 && nmat * cs * 2 <= 120 && nmax >= 48 * cs) cs *= 2;
    bool launched = false;
    LAPY_TRY(launch_sym_cluster(nmat, cs, nmax, A, lda, nsize, want, theta, S, work, active, exact, stream, &launched));
    if (launched) return LAPY_OK;
  }
  // v and w of a reflector in FP64 and double-float (4 lda); partial dots,
  // scaled dots and the double-float reflector of the back-transformation
  // (6 want + lda)
  const size_t smem = sizeof(double) * std::max<size_t>(4 * (size_t)lda, 6 * (size_t)want + (size_t)lda);
  if (smem > 48 * 1024) {
    LAPY_CUDA_TRY(cudaFuncSetAttribute(sym_eig_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  }
  sym_eig_kernel<<<nmat, kEigThreads, smem, stream>>>(A, lda, nsize, want, theta, S, work,
                                                     sym_eig_work_doubles(lda, want), active);
  return lapy_check_launch("sym_eig_kernel");
}

}  // namespace lapy
