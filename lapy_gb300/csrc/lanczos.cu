// Block shift-invert Lanczos for A x = lambda M x on a batch of meshes.
//
// The operator OP = (A - sigma M)^-1 M is self-adjoint in the M inner product.
// Each block step applies OP to the newest basis block (inner solves: FP32
// PCG inside FP64 iterative refinement), orthogonalises the result against
// the whole basis twice (classical Gram-Schmidt, FP64), stores the projection
// coefficients as a block column of T = Q' M OP M Q, and M-orthonormalises
// the block with two Cholesky-QR passes.  No restarts: the basis is kept
// (HBM holds it easily), so the projected matrix is the Rayleigh quotient of
// OP on the whole Krylov space.  At check points the top eigenpairs of T
// (FP64, dense.cu) give residual estimates ||B_m S_last,i|| / |theta_i|.  A
// converged segment is frozen; when all are, the Ritz vectors X = Q S enter a
// final FP64 Rayleigh-Ritz step with the exact A and M, which returns the
// eigenvalues (ascending) and M-orthonormal eigenvectors.
//
// This is the method of lapy/solver.py:667-716 (eigsh in shift-invert mode
// with OPinv = splu(A - sigma M).solve): same operator, same sigma, same
// output convention; ARPACK's implicit restarts are replaced by a full basis
// and the sparse LU by iterative inner solves.
#include <cmath>
#include <vector>
#include "blas.cuh"
#include "dfloat.cuh"
#include "dense.cuh"
#include "solve.cuh"
#include "coarse.cuh"
#include "spmv.cuh"

namespace lapy {

static size_t a256(size_t x) { return (x + 255) & ~size_t(255); }

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
__global__ void rand_fill_kernel(int64_t n, uint64_t seed, double* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint64_t h = (uint64_t)i * 0x9E3779B97F4A7C15ull + seed * 0xD1B54A32D192ED03ull + 0x632BE59BD9B4E019ull;
  h ^= h >> 31; h *= 0xBF58476D1CE4E5B9ull; h ^= h >> 27; h *= 0x94D049BB133111EBull; h ^= h >> 31;
  out[i] = ((double)(h >> 11) * (1.0 / 9007199254740992.0)) - 0.5;
}

// Zero rows of segments that are not active (block per chunk).
__global__ void zero_inactive_kernel(double* __restrict__ X, int ncol, const int32_t* __restrict__ chunk_row,
                                     const int32_t* __restrict__ chunk_seg, const int32_t* __restrict__ active) {
  const int c = blockIdx.x;
  if (active[chunk_seg[c]]) return;
  const int64_t r0 = chunk_row[c], r1 = chunk_row[c + 1];
  for (int64_t i = r0 * ncol + threadIdx.x; i < r1 * ncol; i += blockDim.x) X[i] = 0.0;
}

// Block-strided addressing: element (row, a) of a matrix stored as blocks of
// `bs` columns, block stride `bst` elements: base[(a/bs)*bst + row*bs + a%bs].
struct BMat {
  const double* base;
  int bs;
  int64_t bst;
  __device__ __forceinline__ double at(int64_t row, int a) const {
    return base[(int64_t)(a / bs) * bst + row * bs + (a % bs)];
  }
};

constexpr int kTile = 16;
constexpr int kGemmChunkRows = 16384;

// partial[c][a][b] = sum over the chunk's rows of X(row, a) * Y(row, b)
__global__ void __launch_bounds__(256) gemm_tn_partial_kernel(BMat X, int na, BMat Y, int nb,
                                                              const int32_t* __restrict__ chunk_row,
                                                              const int32_t* __restrict__ chunk_seg,
                                                              const int32_t* __restrict__ active,
                                                              double* __restrict__ partial) {
  const int c = blockIdx.x;
  const int a = blockIdx.y * kTile + threadIdx.x / kTile;
  const int b = blockIdx.z * kTile + threadIdx.x % kTile;
  const bool act = !active || active[chunk_seg[c]];
  double acc = 0.0;
  if (act && a < na && b < nb) {
    const int64_t r0 = chunk_row[c], r1 = chunk_row[c + 1];
    for (int64_t r = r0; r < r1; ++r) acc += X.at(r, a) * Y.at(r, b);
  }
  if (a < na && b < nb) partial[((int64_t)c * na + a) * nb + b] = acc;
}

// out[s][a][b] (leading dim ldo) = sum over chunks of segment s: eight lanes
// per entry, lane k adding chunks k, k + 8, ... (four neighbouring entries per
// warp read a chunk's partials together), then three exchanges.  One thread
// per entry took 40 us for the 161 chunks of a 10,242-row mesh.
__global__ void gemm_tn_reduce_kernel(const double* __restrict__ partial, int na, int nb,
                                      const int32_t* __restrict__ seg_chunk, double* __restrict__ out,
                                      int64_t out_seg_stride, int ldo) {
  const int s = blockIdx.x;
  const int c0 = seg_chunk[s], c1 = seg_chunk[s + 1];
  const int lane = threadIdx.x & 31, k = lane >> 2;
  const int64_t m = (int64_t)na * nb;
  for (int64_t e0 = ((int64_t)blockIdx.y * blockDim.x + threadIdx.x) / 32 * 4; e0 < m;
       e0 += (int64_t)gridDim.y * blockDim.x / 8) {
    const int64_t e = e0 + (lane & 3);
    double acc = 0.0;
    if (e < m)
      for (int c = c0 + k; c < c1; c += 8) acc += partial[(int64_t)c * m + e];
    for (int o = 16; o >= 4; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (k == 0 && e < m) out[(int64_t)s * out_seg_stride + e / nb * ldo + e % nb] = acc;
  }
}

// Y(row, b) = beta*Y(row, b) + alpha * sum_a X(row, a) * H_s[a*ldh + b]
__global__ void __launch_bounds__(256) gemm_nn_kernel(BMat X, int na, const double* __restrict__ H,
                                                      int64_t h_seg_stride, int ldh, double* __restrict__ Y,
                                                      int ldy, int nb, double alpha, double beta,
                                                      const int32_t* __restrict__ chunk_row,
                                                      const int32_t* __restrict__ chunk_seg,
                                                      const int32_t* __restrict__ active) {
  const int c = blockIdx.x;
  const int s = chunk_seg[c];
  if (active && !active[s]) return;
  const double* Hs = H + (int64_t)s * h_seg_stride;
  const int64_t r0 = chunk_row[c], r1 = chunk_row[c + 1];
  for (int64_t e = r0 * nb + threadIdx.x; e < r1 * nb; e += blockDim.x) {
    const int64_t row = e / nb;
    const int b = (int)(e - row * nb);
    double acc = 0.0;
    for (int a = 0; a < na; ++a) acc += X.at(row, a) * Hs[(int64_t)a * ldh + b];
    const int64_t o = row * ldy + b;
    Y[o] = (beta == 0.0) ? alpha * acc : beta * Y[o] + alpha * acc;
  }
}

// Block-row forms of the two basis products for a basis stored as blocks of P
// columns (block j: n x P row-major at X + j * bst), one thread per row.
//
// NN: Y(row, b) = beta Y(row, b) + alpha sum_j sum_a X_j(row, a) H_s[j*P + a][b]
// with the segment's H (nblk*P x P) staged in shared memory.
template <int P>
__global__ void __launch_bounds__(256) gemm_nn_blk_kernel(const double* __restrict__ X, int64_t bst, int nblk,
                                                          const double* __restrict__ H, int64_t h_seg_stride,
                                                          int ldh, double* __restrict__ Y, double alpha, double beta,
                                                          const int32_t* __restrict__ chunk_row,
                                                          const int32_t* __restrict__ chunk_seg,
                                                          const int32_t* __restrict__ active) {
  extern __shared__ double hsm[];
  const int c = blockIdx.x;
  const int s = chunk_seg[c];
  if (active && !active[s]) return;
  const double* Hs = H + (int64_t)s * h_seg_stride;
  for (int i = threadIdx.x; i < nblk * P * P; i += blockDim.x) hsm[i] = Hs[(int64_t)(i / P) * ldh + (i % P)];
  __syncthreads();
  const int64_t r1 = chunk_row[c + 1];
  for (int64_t r = chunk_row[c] + threadIdx.x; r < r1; r += blockDim.x) {
    double acc[P];
#pragma unroll
    for (int b = 0; b < P; ++b) acc[b] = 0.0;
    for (int j = 0; j < nblk; ++j) {
      const double* xr = X + (int64_t)j * bst + r * P;
      const double* hj = hsm + j * P * P;
#pragma unroll
      for (int a = 0; a < P; ++a) {
        const double x = __ldg(xr + a);
#pragma unroll
        for (int b = 0; b < P; ++b) acc[b] = fma(x, hj[a * P + b], acc[b]);
      }
    }
    double* yr = Y + r * P;
#pragma unroll
    for (int b = 0; b < P; ++b) yr[b] = (beta == 0.0) ? alpha * acc[b] : beta * yr[b] + alpha * acc[b];
  }
}

// ---- double-float basis products --------------------------------------------
// A double x is held as the float pair (hi, lo), hi = fl32(x), lo = fl32(x - hi)
// (about 48 significant bits).  A product x*y is formed with the FP32
// error-free transformations: p = fl(xh*yh) and its exact error by fmaf, plus
// the cross terms xh*yl + xl*yh; the running sum (sh, sl) takes p by an exact
// two-sum and the error terms in sl.  Relative error about 2^-44 per product,
// on FP32 instructions, of which this part issues about 64x more per clock
// than FP64 ones.  The round-to-nearest intrinsics keep the compiler from
// contracting the steps into FMAs (which would break the exactness).
__global__ void to_df_kernel(int64_t m, const double* __restrict__ x, float2* __restrict__ y) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const double v = x[i];
  const float h = __double2float_rn(v);
  y[i] = make_float2(h, __double2float_rn(v - (double)h));
}

// In place: the 8-byte double becomes its 8-byte float pair.
__global__ void to_df_inplace_kernel(int64_t m, double* x) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const double v = x[i];
  const float h = __double2float_rn(v);
  reinterpret_cast<float2*>(x)[i] = make_float2(h, __double2float_rn(v - (double)h));
}

// Sums of NV double-float values over the warp's lanes l, l + TPR, l + 2 TPR,
// ... (the 32 / TPR lanes of one residue mod TPR) by halving exchanges: NV - 1
// exchanges or fewer instead of NV log2(32 / TPR).  Afterwards the lane holds
// the sums of the values first .. first + left - 1 in its leading entries.
template <int NV, int TPR>
__device__ __forceinline__ int df_lane_totals(float (&h)[NV], float (&l)[NV], int& left) {
  const int lane = threadIdx.x & 31;
  int first = 0;
  constexpr int LOG = (TPR == 1 ? 5 : TPR == 2 ? 4 : TPR == 4 ? 3 : 2);
  left = NV;
#pragma unroll
  for (int st = 0; st < LOG; ++st) {
    const int mask = 16 >> st;
    const int half = NV >> (st + 1);
    if (half > 0) {
      const bool up = lane & mask;
#pragma unroll
      for (int i = 0; i < (NV >> (st + 1)); ++i) {
        const float kh = up ? h[i + half] : h[i], kl = up ? l[i + half] : l[i];
        const float sh = up ? h[i] : h[i + half], sl = up ? l[i] : l[i + half];
        h[i] = kh;
        l[i] = kl;
        df_add(h[i], l[i], __shfl_xor_sync(0xffffffffu, sh, mask), __shfl_xor_sync(0xffffffffu, sl, mask));
      }
      first += up ? half : 0;
      left = half;
    } else {
      df_add(h[0], l[0], __shfl_xor_sync(0xffffffffu, h[0], mask), __shfl_xor_sync(0xffffffffu, l[0], mask));
    }
  }
  return first;
}
// The same in FP64.
template <int NV, int TPR>
__device__ __forceinline__ int f64_lane_totals(double (&v)[NV], int& left) {
  const int lane = threadIdx.x & 31;
  int first = 0;
  constexpr int LOG = (TPR == 1 ? 5 : TPR == 2 ? 4 : TPR == 4 ? 3 : 2);
  left = NV;
#pragma unroll
  for (int st = 0; st < LOG; ++st) {
    const int mask = 16 >> st;
    const int half = NV >> (st + 1);
    if (half > 0) {
      const bool up = lane & mask;
#pragma unroll
      for (int i = 0; i < (NV >> (st + 1)); ++i) {
        const double keep = up ? v[i + half] : v[i], send = up ? v[i] : v[i + half];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
      }
      first += up ? half : 0;
      left = half;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], mask);
    }
  }
  return first;
}

// TN with the basis in double-float form: TPR lanes share a row, each taking
// P / TPR of the block's columns (16 accumulators per lane at P = 8, so that
// the sums over lanes cost 14 exchanges; one lane per row had 64 accumulators
// and 320).  A warp's lanes read consecutive 16-byte pieces of X.  Bound by
// the FP32 pipe (about 10 instructions per product) on large batches, by
// latency on one mesh; per product 300 -> 15 us at 10,242 rows, 8 columns,
// 128 basis vectors.
template <int P, int TPR, int JB>
__global__ void __launch_bounds__(256) gemm_tn_df_kernel(const float2* __restrict__ X, int64_t bst, int nblk,
                                                         const float2* __restrict__ Y,
                                                         const int32_t* __restrict__ chunk_row,
                                                         const int32_t* __restrict__ chunk_seg,
                                                         const int32_t* __restrict__ active,
                                                         double* __restrict__ partial) {
  constexpr int PA = P / TPR;        // columns of X per lane
  constexpr int NV = JB * PA * P;    // accumulators: [jj][a][b]
  __shared__ double red[8][TPR][NV];
  const int c = blockIdx.x, j0 = blockIdx.y * JB;
  const int warp = threadIdx.x >> 5, sub = threadIdx.x % TPR;
  float sh[NV], sl[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) { sh[v] = 0.f; sl[v] = 0.f; }
  if (!active || active[chunk_seg[c]]) {
    const int64_t r1 = chunk_row[c + 1];
    for (int64_t r = chunk_row[c] + threadIdx.x / TPR; r < r1; r += blockDim.x / TPR) {
      float2 y[P];
#pragma unroll
      for (int b = 0; b < P; ++b) y[b] = __ldg(Y + r * P + b);
#pragma unroll
      for (int jj = 0; jj < JB; ++jj) {
        if (j0 + jj < nblk) {
          const float2* xr = X + (int64_t)(j0 + jj) * bst + r * P + sub * PA;
#pragma unroll
          for (int a = 0; a < PA; ++a) {
            const float2 x = xr[a];
#pragma unroll
            for (int b = 0; b < P; ++b) df_fma(x, y[b], sh[(jj * PA + a) * P + b], sl[(jj * PA + a) * P + b]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) {  // normalise before the two-sums
    const float h = __fadd_rn(sh[v], sl[v]);
    sl[v] = __fsub_rn(sl[v], __fsub_rn(h, sh[v]));
    sh[v] = h;
  }
  int left;
  const int first = df_lane_totals<NV, TPR>(sh, sl, left);
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (i < left) red[warp][sub][first + i] = (double)sh[i] + (double)sl[i];  // (equal sums from several lanes)
  __syncthreads();
  const int na = nblk * P;
  for (int e = threadIdx.x; e < TPR * NV; e += blockDim.x) {
    const int s = e / NV, v = e % NV;
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += red[w][s][v];
    const int jj = v / (PA * P), a = s * PA + (v / P) % PA, b = v % P;
    if (j0 + jj < nblk) partial[((int64_t)c * na + (j0 + jj) * P + a) * P + b] = t;
  }
}

// P x P Gram matrices X' Y in FP64 (X, Y: n x P), split as gemm_tn_df_kernel.
template <int P, int TPR>
__global__ void __launch_bounds__(256) gram_f64_kernel(const double* __restrict__ X, const double* __restrict__ Y,
                                                       const int32_t* __restrict__ chunk_row,
                                                       const int32_t* __restrict__ chunk_seg,
                                                       const int32_t* __restrict__ active,
                                                       double* __restrict__ partial) {
  constexpr int PA = P / TPR, NV = PA * P;
  __shared__ double red[8][TPR][NV];
  const int c = blockIdx.x;
  const int warp = threadIdx.x >> 5, sub = threadIdx.x % TPR;
  double acc[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) acc[v] = 0.0;
  if (!active || active[chunk_seg[c]]) {
    const int64_t r1 = chunk_row[c + 1];
    for (int64_t r = chunk_row[c] + threadIdx.x / TPR; r < r1; r += blockDim.x / TPR) {
      double y[P];
#pragma unroll
      for (int b = 0; b < P; ++b) y[b] = __ldg(Y + r * P + b);
#pragma unroll
      for (int a = 0; a < PA; ++a) {
        const double x = __ldg(X + r * P + sub * PA + a);
#pragma unroll
        for (int b = 0; b < P; ++b) acc[a * P + b] = fma(x, y[b], acc[a * P + b]);
      }
    }
  }
  int left;
  const int first = f64_lane_totals<NV, TPR>(acc, left);
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (i < left) red[warp][sub][first + i] = acc[i];
  __syncthreads();
  for (int e = threadIdx.x; e < TPR * NV; e += blockDim.x) {
    const int s = e / NV, v = e % NV;
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += red[w][s][v];
    partial[((int64_t)c * P + s * PA + v / P) * P + v % P] = t;
  }
}

// NN with the basis in double-float form: Y(row, b) = beta Y + alpha sum X_j(row, a) H[j*P+a][b].
template <int P>
__global__ void __launch_bounds__(256) gemm_nn_df_kernel(const float2* __restrict__ X, int64_t bst, int nblk,
                                                         const double* __restrict__ H, int64_t h_seg_stride,
                                                         int ldh, double* __restrict__ Y, double alpha, double beta,
                                                         const int32_t* __restrict__ chunk_row,
                                                         const int32_t* __restrict__ chunk_seg,
                                                         const int32_t* __restrict__ active) {
  extern __shared__ float2 hdf[];
  const int c = blockIdx.x;
  const int s = chunk_seg[c];
  if (active && !active[s]) return;
  const double* Hs = H + (int64_t)s * h_seg_stride;
  for (int i = threadIdx.x; i < nblk * P * P; i += blockDim.x) hdf[i] = df_split(Hs[(int64_t)(i / P) * ldh + (i % P)]);
  __syncthreads();
  const int64_t r1 = chunk_row[c + 1];
  for (int64_t r = chunk_row[c] + threadIdx.x; r < r1; r += blockDim.x) {
    float sh[P], sl[P];
#pragma unroll
    for (int b = 0; b < P; ++b) { sh[b] = 0.f; sl[b] = 0.f; }
#pragma unroll 2
    for (int j = 0; j < nblk; ++j) {  // two blocks' loads in flight
      const float2* xr = X + (int64_t)j * bst + r * P;
      const float2* hj = hdf + j * P * P;
#pragma unroll
      for (int a = 0; a < P; ++a) {
        const float2 x = xr[a];
#pragma unroll
        for (int b = 0; b < P; ++b) df_fma(x, hj[a * P + b], sh[b], sl[b]);
      }
    }
    double* yr = Y + r * P;
#pragma unroll
    for (int b = 0; b < P; ++b) {
      const double acc = (double)sh[b] + (double)sl[b];
      yr[b] = (beta == 0.0) ? alpha * acc : beta * yr[b] + alpha * acc;
    }
  }
}

// Y(row, b) = sum_a Q(row, a) H_s[a][b] in double-float, one thread per
// output entry (Q: double-float, blocks of p columns; H_s pre-split): the
// fallback of the register-tiled form below when H's column tile does not fit
// in shared memory.
__global__ void __launch_bounds__(256) gemm_nn_dfany_kernel(const float2* __restrict__ X, int p, int64_t bst,
                                                            int na, const float2* __restrict__ H,
                                                            int64_t h_seg_stride, int ldh, double* __restrict__ Y,
                                                            int ldy, int nb, const int32_t* __restrict__ chunk_row,
                                                            const int32_t* __restrict__ chunk_seg) {
  const int c = blockIdx.x;
  const float2* Hs = H + (int64_t)chunk_seg[c] * h_seg_stride;
  const int64_t r0 = chunk_row[c], r1 = chunk_row[c + 1];
  const int nblk = na / p;
  for (int64_t e = r0 * nb + threadIdx.x; e < r1 * nb; e += blockDim.x) {
    const int64_t row = e / nb;
    const int b = (int)(e - row * nb);
    float sh = 0.f, sl = 0.f;
    for (int j = 0; j < nblk; ++j) {
      const float2* xr = X + (int64_t)j * bst + row * p;
      for (int q = 0; q < p; ++q) df_fma(xr[q], Hs[(int64_t)(j * p + q) * ldh + b], sh, sl);
    }
    Y[row * ldy + b] = (double)sh + (double)sl;
  }
}


// Register-tiled forms of the final Rayleigh-Ritz products.
//
// NN: Y(row, b0 + t) = sum_a X(row, a) H_s[a][b0 + t], t < TB, for a
// double-float X stored as blocks of bs columns (block stride bst float2;
// bs = na for a row-major matrix) and a double-float H whose TB columns the
// CTA stages in shared memory (na x TB).  One thread per row holds TB
// accumulators, so every X value is read once per column tile instead of once
// per output.
constexpr int kNnTile = 16;
template <int TB>
__global__ void __launch_bounds__(256) gemm_nn_df_tile_kernel(const float2* __restrict__ X, int bs, int64_t bst,
                                                              int na, const float2* __restrict__ H,
                                                              int64_t h_seg_stride, int ldh, double* __restrict__ Y,
                                                              int ldy, int nb, const int32_t* __restrict__ chunk_row,
                                                              const int32_t* __restrict__ chunk_seg) {
  extern __shared__ float2 hs[];  // na x TB
  const int c = blockIdx.x, b0 = blockIdx.y * TB;
  const float2* Hs = H + (int64_t)chunk_seg[c] * h_seg_stride;
  for (int i = threadIdx.x; i < na * TB; i += blockDim.x) {
    const int a = i / TB, b = b0 + i % TB;
    hs[i] = b < nb ? Hs[(int64_t)a * ldh + b] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  const int64_t r1 = chunk_row[c + 1];
  for (int64_t row = chunk_row[c] + threadIdx.x; row < r1; row += blockDim.x) {
    float sh[TB], sl[TB];
#pragma unroll
    for (int t = 0; t < TB; ++t) { sh[t] = 0.f; sl[t] = 0.f; }
    for (int a0 = 0; a0 < na; a0 += bs) {
      const float2* xr = X + (int64_t)(a0 / bs) * bst + row * bs;
      const int w = min(bs, na - a0);
      for (int q = 0; q < w; ++q) {
        const float2 x = xr[q];
        const float2* h = hs + (a0 + q) * TB;
#pragma unroll
        for (int t = 0; t < TB; ++t) df_fma(x, h[t], sh[t], sl[t]);
      }
    }
    double* yr = Y + row * ldy + b0;
#pragma unroll
    for (int t = 0; t < TB; ++t)
      if (b0 + t < nb) yr[t] = (double)sh[t] + (double)sl[t];
  }
}

// TN: partial[c][a][b] = sum over chunk c's rows of X(row, a) Y(row, b) for
// row-major double-float X (n x na) and Y (n x nb).  A CTA computes a 64 x 64
// output tile (grid.y, grid.z), each thread 4 x 4 of it; rows pass through
// shared memory 16 at a time.
constexpr int kTnRows = 16;
__global__ void __launch_bounds__(256) gemm_tn_df_tile_kernel(const float2* __restrict__ X, int na,
                                                              const float2* __restrict__ Y, int nb,
                                                              const int32_t* __restrict__ chunk_row,
                                                              double* __restrict__ partial) {
  __shared__ float2 sx[kTnRows][64];
  __shared__ float2 sy[kTnRows][64];
  const int c = blockIdx.x, a0 = blockIdx.y * 64, b0 = blockIdx.z * 64;
  const int ta = (threadIdx.x >> 4) * 4, tb = (threadIdx.x & 15) * 4;
  float sh[4][4], sl[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) { sh[i][j] = 0.f; sl[i][j] = 0.f; }
  const int64_t r0 = chunk_row[c], r1 = chunk_row[c + 1];
  for (int64_t rt = r0; rt < r1; rt += kTnRows) {
    __syncthreads();  // the previous tile is consumed
    for (int i = threadIdx.x; i < kTnRows * 64; i += blockDim.x) {
      const int r = i >> 6, col = i & 63;
      const int64_t row = rt + r;
      const bool ok = row < r1;
      sx[r][col] = (ok && a0 + col < na) ? X[row * na + a0 + col] : make_float2(0.f, 0.f);
      sy[r][col] = (ok && b0 + col < nb) ? Y[row * nb + b0 + col] : make_float2(0.f, 0.f);
    }
    __syncthreads();
#pragma unroll 4
    for (int r = 0; r < kTnRows; ++r) {
      float2 xa[4], yb[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { xa[i] = sx[r][ta + i]; yb[i] = sy[r][tb + i]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) df_fma(xa[i], yb[j], sh[i][j], sl[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int a = a0 + ta + i, b = b0 + tb + j;
      if (a < na && b < nb) partial[((int64_t)c * na + a) * nb + b] = (double)sh[i][j] + (double)sl[i][j];
    }
}

// Selective second CGS pass: segment s repeats the projection when the first
// pass cancelled more than a factor 1/eta of some column's M-norm
// (||W'||^2 < eta^2 ||W||^2, NaN included); otherwise one FP64 pass already
// leaves W orthogonal to the basis to about eps / eta relative.
// cnt[0] += active segments, cnt[1] += segments that repeat.
__global__ void reorth_mask_kernel(int nseg, int p, const double* __restrict__ n0, const double* __restrict__ n1,
                                   double eta2, const int32_t* __restrict__ active, int32_t* __restrict__ active2,
                                   unsigned long long* __restrict__ cnt) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  const int a = active[s] != 0;
  int need = 0;
  if (a)
    for (int q = 0; q < p; ++q) need |= !(n1[(int64_t)s * p + q] >= eta2 * n0[(int64_t)s * p + q]);
  active2[s] = a && need;
  if (a) atomicAdd(&cnt[0], 1ull);
  if (a && need) atomicAdd(&cnt[1], 1ull);
}

// Cholesky of the p x p Gram matrix of every segment: G = R' R (R upper), one
// warp per segment, lane i holding column i of R (p <= 16): a pivot's square
// root and reciprocal are the chain, one of each per column (one thread did a
// division per entry: 25 us at p = 8).  Inactive segments get R = I.  A column
// that depends on those before it to rounding is dropped: its row of R is zero,
// and so are its columns of Q and of the projected matrix from there on (the
// basis keeps the directions that are there, its Ritz values those of the rest).
// fail[s] = 1 when no column is left: the basis holds an invariant space.
__global__ void chol_small_kernel(int nseg, int p, const double* __restrict__ G, double* __restrict__ R,
                                  const int32_t* __restrict__ active, int32_t* __restrict__ fail) {
  const int s = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (s >= nseg) return;
  const double* g = G + (int64_t)s * p * p;
  double* r = R + (int64_t)s * p * p;
  if (!active[s]) {
    for (int e = lane; e < p * p; e += 32) r[e] = (e / p == e % p) ? 1.0 : 0.0;
    return;
  }
  const int i = min(lane, p - 1);
  double gmax = fabs(g[i * p + i]);
  for (int o = 16; o > 0; o >>= 1) gmax = fmax(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
  double col[16];  // rows j of column i, what is left of (G + G') / 2, then R
#pragma unroll
  for (int j = 0; j < 16; ++j) col[j] = j < p ? 0.5 * (g[j * p + i] + g[i * p + j]) : 0.0;
  int left = 0;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (j < p) {
      const double d = __shfl_sync(0xffffffffu, col[j], j);
      const bool keep = d > 1e-28 * gmax && isfinite(d);
      const double rjj = keep ? sqrt(d) : 0.0, inv = keep ? 1.0 / rjj : 0.0;
      left += keep;
      col[j] = i == j ? rjj : i > j && keep ? col[j] * inv : 0.0;
#pragma unroll
      for (int k = j + 1; k < 16; ++k)
        if (k < p) col[k] -= __shfl_sync(0xffffffffu, col[j], k) * col[j];
    }
  }
  if (lane < p) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (j < p) r[j * p + i] = col[j];
  }
  if (lane == 0) fail[s] = left == 0;
}

// W(row, :) = W(row, :) * R_s^-1  (R upper triangular, p x p): R and the
// reciprocals of its diagonal staged in shared memory once per chunk, so a
// row costs p(p+1)/2 FMAs and no division (FP64 division is slow here).
// Columns whose diagonal entry is zero become zero.
template <int PT>
__global__ void trsm_right_kernel(double* __restrict__ W, const double* __restrict__ R,
                                  const int32_t* __restrict__ chunk_row, const int32_t* __restrict__ chunk_seg) {
  __shared__ double sr[PT * PT];
  __shared__ double sinv[PT];
  const int c = blockIdx.x;
  const int s = chunk_seg[c];
  const double* r = R + (int64_t)s * PT * PT;
  for (int e = threadIdx.x; e < PT * PT; e += blockDim.x) sr[e] = r[e];
  if (threadIdx.x < PT) {
    const double d = r[threadIdx.x * PT + threadIdx.x];
    sinv[threadIdx.x] = d == 0.0 ? 0.0 : 1.0 / d;
  }
  __syncthreads();
  const int64_t r0 = chunk_row[c], r1 = chunk_row[c + 1];
  for (int64_t row = r0 + threadIdx.x; row < r1; row += blockDim.x) {
    double x[PT];
    double* w = W + row * PT;
#pragma unroll
    for (int j = 0; j < PT; ++j) x[j] = w[j];
#pragma unroll
    for (int j = 0; j < PT; ++j) {
      double v = x[j];
#pragma unroll
      for (int i = 0; i < j; ++i) v -= x[i] * sr[i * PT + j];
      x[j] = v * sinv[j];
    }
#pragma unroll
    for (int j = 0; j < PT; ++j) w[j] = x[j];
  }
}

static int launch_trsm_right(double* W, int p, const double* R, const ChunkTable& gt, cudaStream_t st) {
  switch (p) {
    case 1: trsm_right_kernel<1><<<gt.nchunk, 128, 0, st>>>(W, R, gt.chunk_row, gt.chunk_seg); break;
    case 2: trsm_right_kernel<2><<<gt.nchunk, 128, 0, st>>>(W, R, gt.chunk_row, gt.chunk_seg); break;
    case 4: trsm_right_kernel<4><<<gt.nchunk, 128, 0, st>>>(W, R, gt.chunk_row, gt.chunk_seg); break;
    case 8: trsm_right_kernel<8><<<gt.nchunk, 128, 0, st>>>(W, R, gt.chunk_row, gt.chunk_seg); break;
    case 16: trsm_right_kernel<16><<<gt.nchunk, 128, 0, st>>>(W, R, gt.chunk_row, gt.chunk_seg); break;
    default:
      lapy_set_last_message("eigs: block width %d not in {1,2,4,8,16}", p);
      return LAPY_ERR_INVALID;
  }
  return lapy_check_launch("trsm_right_kernel");
}

// C_s = A_s * B_s for p x p (used for B_j = R2 R1)
__global__ void small_matmul_kernel(int nseg, int p, const double* __restrict__ A, const double* __restrict__ B,
                                    double* __restrict__ C) {
  const int s = blockIdx.x;
  const double* a = A + (int64_t)s * p * p;
  const double* b = B + (int64_t)s * p * p;
  for (int e = threadIdx.x; e < p * p; e += blockDim.x) {
    const int i = e / p, j = e % p;
    double acc = 0.0;
    for (int k = 0; k < p; ++k) acc += a[i * p + k] * b[k * p + j];
    C[(int64_t)s * p * p + e] = acc;
  }
}

// T_s[r][jp + c] = T_s[jp + c][r] = H_s[r][c] for r < (j+1)p (diagonal block symmetrised)
__global__ void store_T_kernel(int p, int j, const double* __restrict__ H, int64_t h_seg_stride,
                               double* __restrict__ T, int lda, const int32_t* __restrict__ active) {
  const int s = blockIdx.x;
  if (!active[s]) return;
  const double* h = H + (int64_t)s * h_seg_stride;
  double* t = T + (int64_t)s * lda * lda;
  const int rows = (j + 1) * p;
  for (int e = threadIdx.x; e < rows * p; e += blockDim.x) {
    const int r = e / p, c = e % p;
    double v = h[(int64_t)r * p + c];
    if (r >= j * p) {
      const int a = r - j * p;
      v = 0.5 * (v + h[(int64_t)(j * p + c) * p + a]);
    }
    t[(int64_t)r * lda + j * p + c] = v;
    t[(int64_t)(j * p + c) * lda + r] = v;
  }
}

__global__ void copy_T_kernel(const double* __restrict__ T, double* __restrict__ Tc, int lda, int m,
                              const int32_t* __restrict__ active) {
  const int s = blockIdx.x;
  if (!active[s]) return;
  const double* t = T + (int64_t)s * lda * lda;
  double* tc = Tc + (int64_t)s * lda * lda;
  for (int e = threadIdx.x; e < m * m; e += blockDim.x) {
    const int r = e / m, c = e % m;
    tc[(int64_t)r * lda + c] = t[(int64_t)r * lda + c];
  }
}

// Residual estimates of the k wanted Ritz pairs; freeze converged segments, and
// those whose rows the next block would not fit into: what it held beyond them
// would be rounding noise, which Cholesky does not always flag.  nconv: pairs
// that meet the tolerance, or -1 in a segment frozen without meeting it.
__global__ void conv_check_kernel(int nseg, int p, int m, int lda, int keff, int k, double tol,
                                  const int32_t* __restrict__ seg_row, const double* __restrict__ theta,
                                  const double* __restrict__ S, const double* __restrict__ Bm,
                                  int32_t* __restrict__ nconv, int32_t* __restrict__ active,
                                  double* __restrict__ Sfinal, double* __restrict__ theta_final,
                                  double* __restrict__ resid_out) {
  __shared__ double sh[32];
  __shared__ int s_stop;
  const int s = blockIdx.x;
  if (!active[s]) return;
  const double* th = theta + (int64_t)s * keff;
  const double* Ss = S + (int64_t)s * lda * keff;
  const double* B = Bm + (int64_t)s * p * p;
  double worst = 0.0;
  int cnt = 0;
  for (int i = threadIdx.x; i < k; i += blockDim.x) {
    double r2 = 0.0;
    for (int a = 0; a < p; ++a) {
      double v = 0.0;
      for (int b = 0; b < p; ++b) v += B[a * p + b] * Ss[(int64_t)(m - p + b) * keff + i];
      r2 += v * v;
    }
    const double res = sqrt(r2) / fmax(fabs(th[i]), 1e-300);
    const bool finite = isfinite(res) && isfinite(th[i]);
    worst = fmax(worst, finite ? res : 1e300);
    cnt += (finite && res <= tol) ? 1 : 0;
  }
  cnt = block_sum(cnt, (int*)sh);
  // block max
  for (int o = 16; o > 0; o >>= 1) worst = fmax(worst, __shfl_xor_sync(0xffffffffu, worst, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = worst;
  __syncthreads();
  if (threadIdx.x == 0) {
    double w = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) w = fmax(w, sh[i]);
    const bool ok = w <= tol, full = m + p > seg_row[s + 1] - seg_row[s];
    resid_out[s] = w;
    nconv[s] = ok || !full ? cnt : -1;
    s_stop = ok || full;
  }
  __syncthreads();
  if (!s_stop) return;
  for (int64_t e = threadIdx.x; e < (int64_t)lda * keff; e += blockDim.x)
    Sfinal[(int64_t)s * lda * keff + e] = Ss[e];
  for (int i = threadIdx.x; i < keff; i += blockDim.x) theta_final[(int64_t)s * keff + i] = th[i];
  __syncthreads();
  if (threadIdx.x == 0) active[s] = 0;
}

// Final Rayleigh-Ritz, dense part (one CTA per segment):
//   Mk = L L', C = L^-1 Ak L^-T, stored negated (so the top eigenpairs of -C
//   are the smallest of C).
__global__ void rr_prepare_kernel(int keff, double* __restrict__ Ak, double* __restrict__ Mk,
                                  double* __restrict__ Cneg, int32_t* __restrict__ fail) {
  const int s = blockIdx.x;
  double* A = Ak + (int64_t)s * keff * keff;
  double* L = Mk + (int64_t)s * keff * keff;
  double* C = Cneg + (int64_t)s * keff * keff;
  __shared__ int bad;
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  // symmetrise both
  for (int e = threadIdx.x; e < keff * keff; e += blockDim.x) {
    const int i = e / keff, j = e % keff;
    if (i < j) {
      const double a = 0.5 * (A[i * keff + j] + A[j * keff + i]);
      A[i * keff + j] = a; A[j * keff + i] = a;
      const double m = 0.5 * (L[i * keff + j] + L[j * keff + i]);
      L[i * keff + j] = m; L[j * keff + i] = m;
    }
  }
  __syncthreads();
  // Cholesky (lower, left-looking), L overwrites Mk's lower triangle
  for (int j = 0; j < keff; ++j) {
    if (threadIdx.x == 0) {
      double d = L[j * keff + j];
      for (int k = 0; k < j; ++k) d -= L[j * keff + k] * L[j * keff + k];
      if (!(d > 0) || !isfinite(d)) { bad = 1; d = 1e-300; }
      L[j * keff + j] = sqrt(d);
    }
    __syncthreads();
    const double ljj = L[j * keff + j];
    for (int i = j + 1 + threadIdx.x; i < keff; i += blockDim.x) {
      double v = L[i * keff + j];
      for (int k = 0; k < j; ++k) v -= L[i * keff + k] * L[j * keff + k];
      L[i * keff + j] = v / ljj;
    }
    __syncthreads();
  }
  // Z = L^-1 A  (column per thread), stored in C
  for (int col = threadIdx.x; col < keff; col += blockDim.x) {
    for (int i = 0; i < keff; ++i) {
      double v = A[i * keff + col];
      for (int k = 0; k < i; ++k) v -= L[i * keff + k] * C[k * keff + col];
      C[i * keff + col] = v / L[i * keff + i];
    }
  }
  __syncthreads();
  // C = L^-1 Z'  : transpose Z into A (scratch), then forward-substitute
  for (int e = threadIdx.x; e < keff * keff; e += blockDim.x) {
    const int i = e / keff, j = e % keff;
    A[j * keff + i] = C[i * keff + j];
  }
  __syncthreads();
  for (int col = threadIdx.x; col < keff; col += blockDim.x) {
    for (int i = 0; i < keff; ++i) {
      double v = A[i * keff + col];
      for (int k = 0; k < i; ++k) v -= L[i * keff + k] * C[k * keff + col];
      C[i * keff + col] = v / L[i * keff + i];
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < keff * keff; e += blockDim.x) C[e] = -C[e];
  if (threadIdx.x == 0) fail[s] = bad;
}

// Yv = L^-T V  (V: keff x k eigenvectors of -C), written over V; lambda = -theta.
__global__ void rr_finish_kernel(int keff, int k, const double* __restrict__ Lm, double* __restrict__ V,
                                 const double* __restrict__ theta, double* __restrict__ evals) {
  const int s = blockIdx.x;
  const double* L = Lm + (int64_t)s * keff * keff;
  double* v = V + (int64_t)s * keff * k;
  for (int col = threadIdx.x; col < k; col += blockDim.x) {
    for (int i = keff - 1; i >= 0; --i) {
      double x = v[(int64_t)i * k + col];
      for (int j = i + 1; j < keff; ++j) x -= L[j * keff + i] * v[(int64_t)j * k + col];
      v[(int64_t)i * k + col] = x / L[i * keff + i];
    }
    evals[(int64_t)s * k + col] = -theta[(int64_t)s * k + col];
  }
}

// ---- aggregate-contiguous row order (two-level eigensolves) ---------------
// New row i is old row perm[i]; its entries are those of the old row with
// columns renumbered by iperm and sorted ascending (insertion sort on the
// row's own output range); pos[k] = old position of new entry k.
__global__ void permute_pattern_kernel(int64_t n, const int32_t* __restrict__ indptr,
                                       const int32_t* __restrict__ indices, const int32_t* __restrict__ perm,
                                       const int32_t* __restrict__ iperm, const int32_t* __restrict__ pindptr,
                                       int32_t* __restrict__ pindices, int32_t* __restrict__ pos) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t o = perm[i];
  const int32_t kb = indptr[o], len = indptr[o + 1] - kb, out = pindptr[i];
  for (int32_t t = 0; t < len; ++t) {
    const int32_t c = iperm[indices[kb + t]], k = kb + t;
    int32_t j = t;
    while (j > 0 && pindices[out + j - 1] > c) {
      pindices[out + j] = pindices[out + j - 1];
      pos[out + j] = pos[out + j - 1];
      --j;
    }
    pindices[out + j] = c;
    pos[out + j] = k;
  }
}

__global__ void inverse_perm_kernel(int64_t n, const int32_t* __restrict__ perm, int32_t* __restrict__ iperm) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) iperm[perm[i]] = (int32_t)i;
}

// out[k] = in[idx[k]]
__global__ void gather_f64_kernel(int64_t m, const int32_t* __restrict__ idx, const double* __restrict__ in,
                                  double* __restrict__ out) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < m) out[k] = in[idx[k]];
}

// Rows back to the caller's order: out[perm[i]][c] = in[i][c] (ncol columns).
__global__ void unpermute_rows_kernel(int64_t n, int ncol, const int32_t* __restrict__ perm,
                                      const double* __restrict__ in, double* __restrict__ out) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * ncol) return;
  const int64_t i = t / ncol;
  const int c = (int)(t - i * ncol);
  out[(int64_t)perm[i] * ncol + c] = in[t];
}

// ---------------------------------------------------------------------------
// host driver
// ---------------------------------------------------------------------------
struct EigPlan {
  int64_t n, nnz;
  int nseg, p, k, keff, mb, lda;
  int precond = kPrecJacobi;  // inner PCG: Jacobi or two-level
  int agg_target = kAggTarget;  // rows per aggregate (two-level)
  PcgTuning pcg;                // launch knobs of the inner PCG
  int64_t nagg_max = 0;
  ChunkTable ct;   // PCG chunks
  ChunkTable gt;   // GEMM chunks (larger)
  ChunkTable tt;   // chunks of the Gram-Schmidt TN products (at least 512 rows where the mesh has them)
};

struct EigPtrs {
  void* ct_mem; void* gt_mem; void* tt_mem;
  int32_t* diag_pos; double* k64; float* k32; double* dinv64; float* dinv32;
  double* basis; float2* basis_df; double* Y; double* W; double* MW; float2* MW_df; float2* S_df; float2* X_df;
  void* ir_ws; size_t ir_bytes;
  void* sell_mem; size_t sell_bytes;
  void* sell64_mem; void* sellm_mem; size_t sell64_bytes;
  void* tl_mem; size_t tl_bytes;
  double* partial;
  double* H; double* Hsum; double* G; double* R1; double* R2; double* Bm;
  double* T; double* Tc; double* theta; double* S; double* eigw;
  double* Sfinal; double* theta_final;
  double* X; double* AX; double* MX;
  double* Ak; double* Mk; double* Cneg; double* theta2; double* V; double* eigw2;
  int32_t* active; int32_t* nsize; int32_t* fail; int32_t* nconv; double* resid;
  double* wn0; double* wn1; int32_t* active2; unsigned long long* rcnt;
  // aggregate-contiguous copy of the system (two-level only)
  int32_t* perm; int32_t* iperm; int32_t* pindptr; int32_t* pindices; int32_t* ppos; double* pa; double* pm;
};

static void plan_eig(int64_t n, int64_t nnz, int nseg, const int32_t* seg_row, int k, int p, int max_vectors,
                     int precond, EigPlan* P) {
  P->n = n; P->nnz = nnz; P->nseg = nseg; P->p = p; P->k = k;
  P->precond = precond;
  P->nagg_max = precond == kPrecTwoLevel ? two_level_max_aggs(seg_row, nseg) : 0;
  P->keff = k + p;
  P->mb = std::max((max_vectors + p - 1) / p, (P->keff + 2 * p + p - 1) / p + 1);
  P->lda = P->mb * p;
  std::vector<int32_t> srow(seg_row, seg_row + nseg + 1);
  plan_chunks(srow.data(), nseg, 4 * lapy_num_sms(), &P->ct);
  // basis products: long chunks, so a CTA's register tiles sum many rows
  // before their one reduction
  plan_chunks(srow.data(), nseg, 2 * lapy_num_sms(), &P->gt, kGemmChunkRows);
  // the TN products split over basis blocks too: a CTA sums at least 512 rows
  // before its one reduction over the warp, which costs as much as eight rows
  plan_chunks(srow.data(), nseg, (int)std::min<int64_t>(2 * lapy_num_sms(), std::max<int64_t>(1, n / 512)), &P->tt,
              kGemmChunkRows);
}

static size_t layout_eig(const EigPlan& P, char* base, EigPtrs* q) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* r = base ? base + off : nullptr;
    off += a256(bytes);
    return r;
  };
  const int64_t n = P.n, nnz = P.nnz;
  const int ns = P.nseg, p = P.p, keff = P.keff, lda = P.lda, k = P.k;
  EigPtrs e;
  e.ct_mem = take(chunk_table_bytes(P.ct));
  e.gt_mem = take(chunk_table_bytes(P.gt));
  e.tt_mem = take(chunk_table_bytes(P.tt));
  e.diag_pos = (int32_t*)take(4 * n);
  e.k64 = (double*)take(8 * nnz);
  e.k32 = (float*)take(4 * nnz);
  e.dinv64 = (double*)take(8 * n);
  e.dinv32 = (float*)take(4 * n);
  e.basis = (double*)take(8 * (size_t)(P.mb + 1) * n * p);
  e.basis_df = (float2*)take(8 * (size_t)(P.mb + 1) * n * p);
  e.Y = (double*)take(8 * n * p);
  e.W = (double*)take(8 * n * p);
  e.MW = (double*)take(8 * n * p);
  e.MW_df = (float2*)take(8 * n * p);
  e.ir_bytes = ir_workspace_bytes(n, p, P.ct, 1, P.precond, P.nagg_max);
  e.ir_ws = take(e.ir_bytes);
  e.tl_bytes = P.precond == kPrecTwoLevel ? two_level_bytes(n, P.ct.h_seg_row.data(), ns, P.ct.nvc) : 0;
  e.tl_mem = take(e.tl_bytes);
  e.sell_bytes = sell_bytes_bound(nnz, P.ct, sizeof(float));
  e.sell_mem = take(e.sell_bytes);
  e.sell64_bytes = sell_bytes_bound(nnz, P.ct, sizeof(double));
  e.sell64_mem = take(e.sell64_bytes);
  e.sellm_mem = take(e.sell64_bytes);
  const size_t part_elems = (size_t)std::max(P.gt.nchunk, P.tt.nchunk) * std::max((size_t)lda * p, (size_t)keff * keff);
  e.partial = (double*)take(8 * part_elems);
  e.H = (double*)take(8 * (size_t)ns * lda * p);
  e.Hsum = (double*)take(8 * (size_t)ns * lda * p);
  e.G = (double*)take(8 * (size_t)ns * p * p);
  e.R1 = (double*)take(8 * (size_t)ns * p * p);
  e.R2 = (double*)take(8 * (size_t)ns * p * p);
  e.Bm = (double*)take(8 * (size_t)ns * p * p);
  e.T = (double*)take(8 * (size_t)ns * lda * lda);
  e.Tc = (double*)take(8 * (size_t)ns * lda * lda);
  e.theta = (double*)take(8 * (size_t)ns * keff);
  e.S = (double*)take(8 * (size_t)ns * lda * keff);
  e.eigw = (double*)take(8 * (size_t)ns * sym_eig_work_doubles(lda, keff));
  e.Sfinal = (double*)take(8 * (size_t)ns * lda * keff);
  e.theta_final = (double*)take(8 * (size_t)ns * keff);
  e.X = (double*)take(8 * n * keff);
  e.X_df = (float2*)take(8 * n * keff);
  e.S_df = (float2*)take(8 * (size_t)ns * lda * keff);
  e.AX = (double*)take(8 * n * keff);
  e.MX = (double*)take(8 * n * keff);
  e.Ak = (double*)take(8 * (size_t)ns * keff * keff);
  e.Mk = (double*)take(8 * (size_t)ns * keff * keff);
  e.Cneg = (double*)take(8 * (size_t)ns * keff * keff);
  e.theta2 = (double*)take(8 * (size_t)ns * k);
  e.V = (double*)take(8 * (size_t)ns * keff * k);
  e.eigw2 = (double*)take(8 * (size_t)ns * sym_eig_work_doubles(keff, k));
  e.active = (int32_t*)take(4 * ns);
  e.nsize = (int32_t*)take(4 * ns);
  e.fail = (int32_t*)take(4 * ns);
  e.nconv = (int32_t*)take(4 * ns);
  e.resid = (double*)take(8 * ns);
  e.wn0 = (double*)take(8 * (size_t)ns * p);
  e.wn1 = (double*)take(8 * (size_t)ns * p);
  e.active2 = (int32_t*)take(4 * ns);
  e.rcnt = (unsigned long long*)take(32);  // two counters, then the StepStatus of a block step
  const bool reorder = P.precond == kPrecTwoLevel;
  e.perm = (int32_t*)take(reorder ? 4 * n : 0);
  e.iperm = (int32_t*)take(reorder ? 4 * n : 0);
  e.pindptr = (int32_t*)take(reorder ? 4 * (n + 1) : 0);
  e.pindices = (int32_t*)take(reorder ? 4 * nnz : 0);
  e.ppos = (int32_t*)take(reorder ? 4 * nnz : 0);
  e.pa = (double*)take(reorder ? 8 * nnz : 0);
  e.pm = (double*)take(reorder ? 8 * std::max<int64_t>(nnz, n) : 0);
  if (q) *q = e;
  return off + 256;
}

struct EigOps {
  const EigPlan& P;
  const EigPtrs& e;
  const int32_t* indptr;
  const int32_t* indices;
  const double* a_vals;
  const double* m_vals;
  int m_is_diag;
  int G;
  cudaStream_t st;
  SellMatrix<double> sellM;  // SELL copy of a consistent M (val == nullptr: CSR)

  int apply_M(const double* X, double* Y, int ncol) const {
    if (m_is_diag) {
      return lapy_diag_mm_f64(P.n, m_vals, ncol, X, Y, 1.0, 0.0, st);
    }
    if (sellM.val && sell_spmm<double>(sellM, P.ct.nunit, P.ct.unit_row, ncol, X, Y, 1.0, 0.0, st) == LAPY_OK)
      return LAPY_OK;
    return csr_spmm<double>(P.n, indptr, indices, m_vals, ncol, X, Y, 1.0, 0.0, G, st);
  }
  dim3 reduce_grid(int na, int nb) const {  // 32 entries per CTA of gemm_tn_reduce_kernel
    return dim3(P.nseg, std::max(1u, std::min(256u, lapy_ceil_div((int64_t)na * nb, 32))));
  }
  // out_s (na x nb, ldo) = X' Y per segment
  int gemm_tn(BMat X, int na, BMat Y, int nb, double* out, int64_t out_stride, int ldo, const int32_t* act) const {
    if (X.bs == nb && Y.bs == nb && Y.bst == 0 && na == nb && (nb == 1 || nb == 2 || nb == 4 || nb == 8)) {
      auto kern = nb == 1 ? gram_f64_kernel<1, 1> : nb == 2 ? gram_f64_kernel<2, 1>
                          : nb == 4 ? gram_f64_kernel<4, 2> : gram_f64_kernel<8, 4>;
      kern<<<P.gt.nchunk, 256, 0, st>>>(X.base, Y.base, P.gt.chunk_row, P.gt.chunk_seg, act, e.partial);
      LAPY_TRY(lapy_check_launch("gram_f64_kernel"));
    } else {
      dim3 grid(P.gt.nchunk, lapy_ceil_div(na, kTile), lapy_ceil_div(nb, kTile));
      gemm_tn_partial_kernel<<<grid, 256, 0, st>>>(X, na, Y, nb, P.gt.chunk_row, P.gt.chunk_seg, act, e.partial);
      LAPY_TRY(lapy_check_launch("gemm_tn_partial_kernel"));
    }
    gemm_tn_reduce_kernel<<<reduce_grid(na, nb), 256, 0, st>>>(e.partial, na, nb, P.gt.seg_chunk, out, out_stride, ldo);
    return lapy_check_launch("gemm_tn_reduce_kernel");
  }
  // CGS products against basis blocks 0..nbasis/p-1 from the double-float copy
  template <int PB, int TPR, int JB>
  int gemm_tn_df_p(int nbasis, const double* Y, const int32_t* act) const {
    const int nblk = nbasis / PB;
    // Y split into (hi, lo) pairs once, not once per basis-block CTA (the
    // split is FP64 work, the slow pipe here)
    const int64_t m = P.n * PB;
    to_df_kernel<<<lapy_ceil_div(m, 256), 256, 0, st>>>(m, Y, e.MW_df);
    LAPY_TRY(lapy_check_launch("to_df_kernel"));
    dim3 grid(P.tt.nchunk, lapy_ceil_div(nblk, JB));
    gemm_tn_df_kernel<PB, TPR, JB><<<grid, 256, 0, st>>>(e.basis_df, P.n * PB, nblk, e.MW_df, P.tt.chunk_row,
                                                         P.tt.chunk_seg, act, e.partial);
    return lapy_check_launch("gemm_tn_df_kernel");
  }
  int cgs_tn(int nbasis, const double* MW, double* out, int64_t out_stride, int ldo, const int32_t* act) const {
    const int p = P.p;
    int st_ = LAPY_ERR_INVALID;
    if (p == 1) st_ = gemm_tn_df_p<1, 1, 16>(nbasis, MW, act);
    else if (p == 2) st_ = gemm_tn_df_p<2, 1, 4>(nbasis, MW, act);
    else if (p == 4) st_ = gemm_tn_df_p<4, 1, 1>(nbasis, MW, act);
    else if (p == 8) st_ = gemm_tn_df_p<8, 4, 1>(nbasis, MW, act);
    else return gemm_tn(BMat{e.basis, p, P.n * p}, nbasis, BMat{MW, p, 0}, p, out, out_stride, ldo, act);
    LAPY_TRY(st_);
    gemm_tn_reduce_kernel<<<reduce_grid(nbasis, p), 256, 0, st>>>(e.partial, nbasis, p, P.tt.seg_chunk, out,
                                                                  out_stride, ldo);
    return lapy_check_launch("gemm_tn_reduce_kernel");
  }
  // (on the PCG's short chunks: the NN product has no per-chunk reduction,
  // and the long basis-product chunks left half the SMs' warp slots empty)
  template <int PB>
  int gemm_nn_df_p(int nbasis, const double* H, int64_t hs, int ldh, double* W, const int32_t* act) const {
    const int nblk = nbasis / PB;
    const size_t smem = sizeof(float2) * (size_t)nblk * PB * PB;
    gemm_nn_df_kernel<PB><<<P.ct.nchunk, 256, smem, st>>>(e.basis_df, P.n * PB, nblk, H, hs, ldh, W, -1.0, 1.0,
                                                          P.ct.chunk_row, P.ct.chunk_seg, act);
    return lapy_check_launch("gemm_nn_df_kernel");
  }
  // W -= Q H per segment
  int cgs_nn(int nbasis, const double* H, int64_t hs, int ldh, double* W, const int32_t* act) const {
    const int p = P.p;
    const bool fits = sizeof(float2) * (size_t)nbasis * p <= 48 * 1024;
    if (fits && p == 1) return gemm_nn_df_p<1>(nbasis, H, hs, ldh, W, act);
    if (fits && p == 2) return gemm_nn_df_p<2>(nbasis, H, hs, ldh, W, act);
    if (fits && p == 4) return gemm_nn_df_p<4>(nbasis, H, hs, ldh, W, act);
    if (fits && p == 8) return gemm_nn_df_p<8>(nbasis, H, hs, ldh, W, act);
    return gemm_nn(BMat{e.basis, p, P.n * p}, nbasis, H, hs, ldh, W, p, p, -1.0, 1.0, act);
  }
  int basis_to_df(int j) const {
    const int64_t m = P.n * P.p;
    to_df_kernel<<<lapy_ceil_div(m, 256), 256, 0, st>>>(m, e.basis + (size_t)j * m, e.basis_df + (size_t)j * m);
    return lapy_check_launch("to_df_kernel");
  }
  template <int PB>
  int gemm_nn_blk(BMat X, int na, const double* H, int64_t hs, int ldh, double* Y, double alpha, double beta,
                  const int32_t* act) const {
    const int nblk = na / PB;
    const size_t smem = sizeof(double) * (size_t)nblk * PB * PB;
    gemm_nn_blk_kernel<PB><<<P.gt.nchunk, 256, smem, st>>>(X.base, X.bst, nblk, H, hs, ldh, Y, alpha, beta,
                                                            P.gt.chunk_row, P.gt.chunk_seg, act);
    return lapy_check_launch("gemm_nn_blk_kernel");
  }
  int gemm_nn(BMat X, int na, const double* H, int64_t hs, int ldh, double* Y, int ldy, int nb, double alpha,
              double beta, const int32_t* act) const {
    const bool blk = X.bs == nb && ldy == nb && na % nb == 0 && sizeof(double) * (size_t)na * nb <= 48 * 1024;
    if (blk && nb == 1) return gemm_nn_blk<1>(X, na, H, hs, ldh, Y, alpha, beta, act);
    if (blk && nb == 2) return gemm_nn_blk<2>(X, na, H, hs, ldh, Y, alpha, beta, act);
    if (blk && nb == 4) return gemm_nn_blk<4>(X, na, H, hs, ldh, Y, alpha, beta, act);
    if (blk && nb == 8) return gemm_nn_blk<8>(X, na, H, hs, ldh, Y, alpha, beta, act);
    gemm_nn_kernel<<<P.gt.nchunk, 256, 0, st>>>(X, na, H, hs, ldh, Y, ldy, nb, alpha, beta, P.gt.chunk_row,
                                               P.gt.chunk_seg, act);
    return lapy_check_launch("gemm_nn_kernel");
  }
  // M-orthonormalise W (n x p) in place with two Cholesky-QR passes; Bm = R2 R1.
  int chol_qr2(double* W) const {
    const int p = P.p;
    BMat Wm{W, p, 0};
    for (int pass = 0; pass < 2; ++pass) {
      LAPY_TRY(apply_M(W, e.MW, p));
      BMat MWm{e.MW, p, 0};
      LAPY_TRY(gemm_tn(Wm, p, MWm, p, e.G, (int64_t)p * p, p, e.active));
      double* R = pass == 0 ? e.R1 : e.R2;
      chol_small_kernel<<<lapy_ceil_div(P.nseg, 2), 64, 0, st>>>(P.nseg, p, e.G, R, e.active, e.fail);
      LAPY_TRY(lapy_check_launch("chol_small_kernel"));
      LAPY_TRY(launch_trsm_right(W, p, R, P.gt, st));
    }
    small_matmul_kernel<<<P.nseg, 64, 0, st>>>(P.nseg, p, e.R2, e.R1, e.Bm);
    return lapy_check_launch("small_matmul_kernel");
  }
};

// Cost model of the convergence-check stride (seconds on this part): a check of
// m x m projected matrices (1.0 ms at m = 128, 2.1 ms at 224 for one mesh, 3.1
// ms at 160 for 128 meshes); a block step's fixed cost plus its inner
// iterations, on chip (0.8 ms at 10,242 rows and 110 iterations, 2.3 ms at
// 244,228, 10 ms at 1,251,846, before 5 to 15 % went to plain CG) or as
// grid-wide launches.
constexpr double kCheckSecPerDim = 1.0e-5;
constexpr double kCheckMeshes = 64.0;  // meshes that double a check's time
constexpr double kChipStepSec = 3.5e-4, kChipIterSec = 4.0e-6, kChipIterSecPerRow = 6.0e-11;
constexpr double kGridStepSec = 1.0e-3, kGridIterSec = 2.0e-5, kGridIterSecPerRow = 9.0e-11;
// Pairs that converge per basis vector once the first check is made: 0.33 to
// 0.37 measured for 50 pairs (10,242-vertex sphere, batches of 24 and 128
// meshes), 0.16 for 10 pairs.
constexpr double kPairsPerVector = 0.35;

// Threshold of the selective second Gram-Schmidt pass (reorth_mask_kernel):
// the classical 1/sqrt(2).  On the batched ShapeDNA workload about 98 % of the
// (mesh, block step) pairs still repeat the pass; a threshold of 1e-2 skipped
// 98 % of them but slowed Lanczos convergence (more steps, unconverged meshes).
constexpr double kReorthEta = 0.7071067811865476;

// What the host needs to know of a block step, in one small copy: the first
// status that is not LAPY_OK among the inner solve's columns, its iterations,
// and whether a Cholesky of an active segment failed.
struct StepStatus {
  long long iters;
  int32_t status, fail;
};

__global__ void step_status_kernel(int nsp, const int32_t* __restrict__ state,
                                   const unsigned long long* __restrict__ ctl, int ns,
                                   const int32_t* __restrict__ fail, const int32_t* __restrict__ active,
                                   StepStatus* __restrict__ out) {
  __shared__ int first, any;
  if (threadIdx.x == 0) {
    first = INT_MAX;
    any = 0;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nsp; i += blockDim.x)
    if (state[i] != LAPY_OK) {
      atomicMin(&first, i);
      break;
    }
  for (int s = threadIdx.x; s < ns; s += blockDim.x)
    if (active[s] && fail[s]) any = 1;
  __syncthreads();
  if (threadIdx.x == 0) {
    out->iters = (long long)ctl[0];
    out->status = first < INT_MAX ? state[first] : LAPY_OK;
    out->fail = any;
  }
}

struct EigResult {
  std::vector<int32_t> status;
  std::vector<int32_t> nbasis;
  int64_t inner_iters = 0;
  int blocks = 0;
};

// Two-level eigensolves run on an aggregate-contiguous row order of the
// system (plan_aggregate_order): the copies (pattern, A, M) go to the
// workspace, *indptr etc. are redirected to them, and lab_out receives the
// aggregate labels in that order.
static int reorder_system(const EigPlan& P, const EigPtrs& e, const int32_t** indptr, const int32_t** indices,
                          const double** a_vals, const double** m_vals, int m_is_diag, std::vector<int32_t>* lab_out,
                          cudaStream_t st) {
  const int64_t n = P.n, nnz = P.nnz;
  // host copies of the pattern and the permutation, kept per host thread
  // across calls (grown, never shrunk): a repeated solve does not allocate,
  // zero and fault in these hundreds of megabytes again
  thread_local std::vector<int32_t> hptr, hidx, perm, nptr;
  if ((int64_t)hptr.size() < n + 1) hptr.resize(n + 1);
  if ((int64_t)hidx.size() < nnz) hidx.resize(nnz);
  if ((int64_t)perm.size() < n) perm.resize(n);
  if ((int64_t)nptr.size() < n + 1) nptr.resize(n + 1);
  LAPY_CUDA_TRY(cudaMemcpyAsync(hptr.data(), *indptr, 4 * (size_t)(n + 1), cudaMemcpyDeviceToHost, st));
  LAPY_CUDA_TRY(cudaMemcpyAsync(hidx.data(), *indices, 4 * (size_t)nnz, cudaMemcpyDeviceToHost, st));
  LAPY_CUDA_TRY(cudaStreamSynchronize(st));
  nptr[0] = 0;
  lab_out->assign(n, -1);
  LAPY_TRY(plan_aggregate_order(n, hptr.data(), hidx.data(), P.ct.h_seg_row.data(), P.nseg, perm.data(),
                                lab_out->data(), P.agg_target));
  for (int64_t i = 0; i < n; ++i) nptr[i + 1] = nptr[i] + (hptr[perm[i] + 1] - hptr[perm[i]]);
  LAPY_CUDA_TRY(cudaMemcpyAsync(e.perm, perm.data(), 4 * (size_t)n, cudaMemcpyHostToDevice, st));
  LAPY_CUDA_TRY(cudaMemcpyAsync(e.pindptr, nptr.data(), 4 * (size_t)(n + 1), cudaMemcpyHostToDevice, st));
  const unsigned nb = lapy_ceil_div(n, 256), zb = lapy_ceil_div(nnz, 256);
  inverse_perm_kernel<<<nb, 256, 0, st>>>(n, e.perm, e.iperm);
  LAPY_TRY(lapy_check_launch("inverse_perm_kernel"));
  permute_pattern_kernel<<<nb, 256, 0, st>>>(n, *indptr, *indices, e.perm, e.iperm, e.pindptr, e.pindices, e.ppos);
  LAPY_TRY(lapy_check_launch("permute_pattern_kernel"));
  gather_f64_kernel<<<zb, 256, 0, st>>>(nnz, e.ppos, *a_vals, e.pa);
  LAPY_TRY(lapy_check_launch("gather_f64_kernel"));
  if (m_is_diag)
    gather_f64_kernel<<<nb, 256, 0, st>>>(n, e.perm, *m_vals, e.pm);
  else
    gather_f64_kernel<<<zb, 256, 0, st>>>(nnz, e.ppos, *m_vals, e.pm);
  LAPY_TRY(lapy_check_launch("gather_f64_kernel"));
  // the host vectors are pageable: the copies complete before they go away
  LAPY_CUDA_TRY(cudaStreamSynchronize(st));
  *indptr = e.pindptr;
  *indices = e.pindices;
  *a_vals = e.pa;
  *m_vals = e.pm;
  return LAPY_OK;
}

static int eigs_run(const EigPlan& P, const EigPtrs& e, const int32_t* indptr, const int32_t* indices,
                    const double* a_vals, const double* m_vals, int m_is_diag, double sigma, double tol,
                    double inner_rtol, double round_rtol, int inner_maxiter, uint64_t seed, double* evals,
                    double* evecs, cudaStream_t st, EigResult* res) {
  const int64_t n = P.n;
  const int p = P.p, ns = P.nseg, keff = P.keff, lda = P.lda, k = P.k;
  const int G = spmm_pick_group(n, P.nnz);
  const bool reorder = P.precond == kPrecTwoLevel;
  std::vector<int32_t> lab;
  if (reorder) LAPY_TRY(reorder_system(P, e, &indptr, &indices, &a_vals, &m_vals, m_is_diag, &lab, st));
  EigOps ops{P, e, indptr, indices, a_vals, m_vals, m_is_diag, G, st, SellMatrix<double>()};
  ChunkTable ct = P.ct, gt = P.gt, tt = P.tt;
  LAPY_TRY(upload_chunk_table(&ct, e.ct_mem, st));
  LAPY_TRY(upload_chunk_table(&gt, e.gt_mem, st));
  LAPY_TRY(upload_chunk_table(&tt, e.tt_mem, st));
  const_cast<EigPlan&>(P).ct = ct;
  const_cast<EigPlan&>(P).gt = gt;
  const_cast<EigPlan&>(P).tt = tt;

  // K = A - sigma M (f64 and f32), Jacobi diagonal
  LAPY_TRY(lapy_csr_diag_index(n, indptr, indices, e.diag_pos, st));
  if (m_is_diag) {
    LAPY_CUDA_TRY(cudaMemcpyAsync(e.k64, a_vals, 8 * P.nnz, cudaMemcpyDeviceToDevice, st));
    LAPY_TRY(add_diag(n, e.diag_pos, -sigma, m_vals, e.k64, st));
  } else {
    LAPY_TRY(vec_axpby(P.nnz, 1.0, a_vals, -sigma, m_vals, e.k64, st));
  }
  LAPY_TRY(cast_f64_f32(P.nnz, e.k64, e.k32, st));
  LAPY_TRY(jacobi_inverse(n, e.diag_pos, e.k64, e.dinv64, e.dinv32, st));
  SysMatrix K;
  K.tuning = P.pcg;
  K.n = n; K.nnz = P.nnz; K.indptr = indptr; K.indices = indices;
  K.k64 = e.k64; K.k32 = e.k32; K.dinv64 = e.dinv64; K.dinv32 = e.dinv32;
  // inner solves: on chip when every mesh fits, else the persistent PCG on
  // SELL copies of K
  std::vector<int32_t> h_seg_agg, h_agg_rows;
  if (P.precond == kPrecTwoLevel)
    LAPY_TRY(build_two_level(n, indptr, indices, e.k64, P.ct.h_seg_row.data(), ns, P.ct.nvc, e.tl_mem,
                             e.tl_bytes, &K.pc32, st, reorder ? lab.data() : nullptr, P.agg_target, &h_seg_agg,
                             &h_agg_rows));
  ClusterPlan cluster;
  if (P.precond != kPrecTwoLevel || h_agg_rows.size() == 2 * (size_t)h_seg_agg[ns])
    LAPY_TRY(cluster_plan(n, P.nnz, indptr, indices, e.k32, ns, P.ct.h_seg_row.data(),
                          P.precond == kPrecTwoLevel ? h_seg_agg.data() : nullptr, h_agg_rows.data(), p, e.sell_mem,
                          e.sell_bytes, &cluster, st));
  if (cluster.ok) {
    K.cluster = &cluster;
  } else {
    bool fits = false;
    LAPY_TRY(build_sell<float>(n, indptr, indices, e.k32, P.ct, e.sell_mem, e.sell_bytes, &K.sell32, &fits, st));
    if (!fits) K.sell32 = SellMatrix<float>();
    LAPY_TRY(build_sell<double>(n, indptr, indices, e.k64, P.ct, e.sell64_mem, e.sell64_bytes, &K.sell64, &fits, st));
    if (!fits) K.sell64 = SellMatrix<double>();
  }
  if (!m_is_diag) {
    bool fits = false;
    LAPY_TRY(build_sell<double>(n, indptr, indices, m_vals, P.ct, e.sellm_mem, e.sell64_bytes, &ops.sellM, &fits,
                                st));
    if (!fits) ops.sellM = SellMatrix<double>();
  }

  LAPY_CUDA_TRY(cudaMemsetAsync(e.rcnt, 0, 16, st));
  std::vector<int32_t> hact(ns, 1), hnsize(ns, 0);
  LAPY_CUDA_TRY(cudaMemcpyAsync(e.active, hact.data(), 4 * ns, cudaMemcpyHostToDevice, st));
  LAPY_CUDA_TRY(cudaMemsetAsync(e.T, 0, 8 * (size_t)ns * lda * lda, st));
  LAPY_CUDA_TRY(cudaMemsetAsync(e.Sfinal, 0, 8 * (size_t)ns * lda * keff, st));
  LAPY_CUDA_TRY(cudaMemsetAsync(e.fail, 0, 4 * ns, st));

  // Q_0: random, M-orthonormal
  double* Q0 = e.basis;
  rand_fill_kernel<<<lapy_ceil_div(n * p, 256), 256, 0, st>>>(n * p, seed, Q0);
  LAPY_TRY(lapy_check_launch("rand_fill_kernel"));
  LAPY_TRY(ops.chol_qr2(Q0));
  LAPY_TRY(ops.basis_to_df(0));

  std::vector<int32_t> hfail(ns);
  res->status.assign(ns, LAPY_ERR_NOCONV);
  res->nbasis.assign(ns, 0);
  // First check once the basis holds ~2.5 k vectors (shift-invert Lanczos
  // needs 3-5 k), or the next block does not fit into the rows of the smallest
  // mesh; afterwards the stride is the larger of (a) the block steps that the
  // missing pairs take, on the mean over the unconverged meshes, and (b) the
  // stride that balances the cost of a check c against that of a block step s:
  // checking every m steps costs c/m per step and overshoots convergence by
  // (m-1)/2 steps on average, least at m = sqrt(2 c / s).  c and s come from a
  // cost model of this GPU, not from timers, so the stopping step - and with it
  // every result - is the same on every run.  (With half of the missing pairs'
  // blocks as (a), 10 checks instead of 5 for 642 vertices and 11 instead of 6
  // for 128 meshes.)  No more pairs than a block has columns are checked at
  // every step: where an eigenvalue has more copies than that, rounding brings
  // the others into the basis later, and the first ones look unconverged while
  // they mix.
  const int first_check = std::max((keff + p + p - 1) / p, (int)std::ceil(2.5 * k / p));
  int next_check = first_check;
  int64_t rows_min = INT64_MAX;  // of the meshes that have not stopped
  for (int s = 0; s < ns; ++s) rows_min = std::min<int64_t>(rows_min, P.ct.h_seg_row[s + 1] - P.ct.h_seg_row[s]);
  int64_t step_pcg_iters = 0;
  std::vector<int32_t> hnconv(ns);
  auto inner_done = [&](int status, int64_t iters) -> int {
    res->inner_iters += iters;
    step_pcg_iters = iters;
    if (status != LAPY_ERR_NAN && status != LAPY_ERR_BREAKDOWN) return LAPY_OK;
    lapy_set_last_message("eigs: inner solve failed (%s)", lapy_status_string(status));
    return status;
  };
  StepStatus* dstat = (StepStatus*)(e.rcnt + 2);
  int j = 0;
  bool all_done = false;
  std::vector<int32_t> seg_conv_blocks(ns, 0);
  for (j = 0; j < P.mb && !all_done; ++j) {
    double* Qj = e.basis + (size_t)j * n * p;
    double* Qn = e.basis + (size_t)(j + 1) * n * p;
    // Y = M Q_j ; W = K^-1 Y
    LAPY_TRY(ops.apply_M(Qj, e.Y, p));
    zero_inactive_kernel<<<P.ct.nchunk, 256, 0, st>>>(e.Y, p, P.ct.chunk_row, P.ct.chunk_seg, e.active);
    LAPY_TRY(lapy_check_launch("zero_inactive_kernel"));
    // the solve's status is read with the step's at its end: a wait here left
    // the GPU idle for the launches of the rest of the step
    IrDeferred def;
    LAPY_TRY(ir_solve_deferred(K, P.ct, p, e.Y, e.W, inner_rtol, inner_maxiter, round_rtol, 16, e.ir_ws, e.ir_bytes,
                               st, &def));
    if (!def.taken) {
      IrStats irs;
      LAPY_TRY(ir_solve(K, P.ct, p, e.Y, e.W, inner_rtol, inner_maxiter, 1, round_rtol, 16, e.ir_ws, e.ir_bytes, st,
                        &irs, nullptr, nullptr));
      LAPY_TRY(inner_done(irs.status, irs.pcg_iters));
    }
    // classical Gram-Schmidt against the basis blocks 0..j in the M inner
    // product: a first pass, then a second one where the first cancelled
    // much of a column (the mask leaves H = 0 for the other segments)
    const int nbasis = (j + 1) * p;
    LAPY_TRY(ops.apply_M(e.W, e.MW, p));
    LAPY_TRY(seg_col_dot(e.W, e.MW, p, P.ct, e.wn0, st));
    LAPY_TRY(ops.cgs_tn(nbasis, e.MW, e.Hsum, (int64_t)lda * p, p, e.active));
    LAPY_TRY(ops.cgs_nn(nbasis, e.Hsum, (int64_t)lda * p, p, e.W, e.active));
    LAPY_TRY(ops.apply_M(e.W, e.MW, p));
    LAPY_TRY(seg_col_dot(e.W, e.MW, p, P.ct, e.wn1, st));
    reorth_mask_kernel<<<lapy_ceil_div(ns, 128), 128, 0, st>>>(ns, p, e.wn0, e.wn1, kReorthEta * kReorthEta,
                                                               e.active, e.active2, e.rcnt);
    LAPY_TRY(lapy_check_launch("reorth_mask_kernel"));
    LAPY_TRY(ops.cgs_tn(nbasis, e.MW, e.H, (int64_t)lda * p, p, e.active2));
    LAPY_TRY(ops.cgs_nn(nbasis, e.H, (int64_t)lda * p, p, e.W, e.active2));
    // Hsum += H
    LAPY_TRY(vec_axpby((int64_t)ns * lda * p, 1.0, e.Hsum, 1.0, e.H, e.Hsum, st));
    store_T_kernel<<<ns, 256, 0, st>>>(p, j, e.Hsum, (int64_t)lda * p, e.T, lda, e.active);
    LAPY_TRY(lapy_check_launch("store_T_kernel"));
    // new block
    LAPY_CUDA_TRY(cudaMemcpyAsync(Qn, e.W, 8 * n * p, cudaMemcpyDeviceToDevice, st));
    LAPY_TRY(ops.chol_qr2(Qn));
    LAPY_TRY(ops.basis_to_df(j + 1));
    const int m = (j + 1) * p;
    const bool check = (j + 1 >= next_check) || j + 1 == P.mb || rows_min < (int64_t)(j + 2) * p;
    bool any_fail = false;
    if (def.taken) {
      StepStatus hs;
      step_status_kernel<<<1, 256, 0, st>>>(ns * p, def.state, def.ctl, ns, e.fail, e.active, dstat);
      LAPY_TRY(lapy_check_launch("step_status_kernel"));
      LAPY_CUDA_TRY(cudaMemcpyAsync(&hs, dstat, sizeof(hs), cudaMemcpyDeviceToHost, st));
      LAPY_CUDA_TRY(cudaStreamSynchronize(st));
      LAPY_TRY(inner_done(hs.status, hs.iters));
      any_fail = hs.fail != 0;
    } else {
      LAPY_CUDA_TRY(cudaMemcpyAsync(hfail.data(), e.fail, 4 * ns, cudaMemcpyDeviceToHost, st));
      LAPY_CUDA_TRY(cudaStreamSynchronize(st));
      for (int s = 0; s < ns; ++s) any_fail |= (hact[s] && hfail[s]);
    }
    if (check || any_fail) {
      for (int s = 0; s < ns; ++s) hnsize[s] = m;
      LAPY_CUDA_TRY(cudaMemcpyAsync(e.nsize, hnsize.data(), 4 * ns, cudaMemcpyHostToDevice, st));
      copy_T_kernel<<<ns, 256, 0, st>>>(e.T, e.Tc, lda, m, e.active);
      LAPY_TRY(lapy_check_launch("copy_T_kernel"));
      LAPY_TRY(sym_eig_top(ns, e.Tc, lda, e.nsize, m, keff, e.theta, e.S, e.eigw, e.active, false, st));
      conv_check_kernel<<<ns, 128, 0, st>>>(ns, p, m, lda, keff, k, tol, P.ct.seg_row, e.theta, e.S, e.Bm, e.nconv,
                                            e.active, e.Sfinal, e.theta_final, e.resid);
      LAPY_TRY(lapy_check_launch("conv_check_kernel"));
      std::vector<int32_t> hact2(ns);
      LAPY_CUDA_TRY(cudaMemcpyAsync(hact2.data(), e.active, 4 * ns, cudaMemcpyDeviceToHost, st));
      LAPY_CUDA_TRY(cudaMemcpyAsync(hnconv.data(), e.nconv, 4 * ns, cudaMemcpyDeviceToHost, st));
      LAPY_CUDA_TRY(cudaStreamSynchronize(st));
      all_done = true;
      int64_t missing = 0;
      int worst = 0;
      rows_min = INT64_MAX;
      for (int s = 0; s < ns; ++s) {
        if (hact[s] && !hact2[s]) {
          res->status[s] = hnconv[s] < 0 ? LAPY_ERR_BREAKDOWN : LAPY_OK;
          res->nbasis[s] = m;
        }
        if (hact2[s]) {
          missing += k - hnconv[s];
          worst = std::max(worst, k - hnconv[s]);
          rows_min = std::min<int64_t>(rows_min, P.ct.h_seg_row[s + 1] - P.ct.h_seg_row[s]);
        }
        hact[s] = hact2[s];
        all_done &= !hact[s];
      }
      int nact = 0;
      for (int s = 0; s < ns; ++s) nact += hact[s] != 0;
      const double check_cost = kCheckSecPerDim * (double)(m + p) * (1.0 + (double)nact / kCheckMeshes);
      const double it = (double)step_pcg_iters;
      // (by what solves: the profile's timers keep the solve from being deferred)
      const double step_cost = cluster.ok ? kChipStepSec + it * (kChipIterSec + kChipIterSecPerRow * (double)n)
                                          : kGridStepSec + it * (kGridIterSec + kGridIterSecPerRow * (double)n);
      const int balanced = (int)std::lround(std::sqrt(2.0 * check_cost / step_cost));
      const int steps = (int)std::lround((double)missing / std::max(1, nact) / (kPairsPerVector * p));
      int stride = k <= p ? 1 : std::max({1, steps, balanced});
      // a basis that nears the rows of a mesh: short strides
      if (rows_min < 2 * (int64_t)(j + 1 + stride) * p) stride = std::max(1, (worst + 2 * p - 1) / (2 * p));
      next_check = j + 1 + stride;
    }
  }
  res->blocks = j;
  if (lapy_profile_enabled()) {
    unsigned long long hc[2] = {0, 0};
    LAPY_CUDA_TRY(cudaMemcpyAsync(hc, e.rcnt, 16, cudaMemcpyDeviceToHost, st));
    LAPY_CUDA_TRY(cudaStreamSynchronize(st));
    lapy_profile_add_reorth((long long)hc[0], (long long)hc[1]);
  }
  // segments that never converged: use their last Ritz vectors anyway (status NOCONV)
  {
    std::vector<int32_t> ones(ns, 1);
    bool any = false;
    for (int s = 0; s < ns; ++s) any |= (hact[s] != 0);
    if (any) {
      // copy current S/theta into the final store for still-active segments
      for (int s = 0; s < ns; ++s) {
        if (!hact[s]) continue;
        LAPY_CUDA_TRY(cudaMemcpyAsync(e.Sfinal + (size_t)s * lda * keff, e.S + (size_t)s * lda * keff,
                                      8 * (size_t)lda * keff, cudaMemcpyDeviceToDevice, st));
        res->nbasis[s] = j * p;
      }
    }
    LAPY_CUDA_TRY(cudaMemcpyAsync(e.active, ones.data(), 4 * ns, cudaMemcpyHostToDevice, st));
    LAPY_CUDA_TRY(cudaStreamSynchronize(st));
  }
  // X = Q S_final (n x keff): basis blocks 0..j-1 (S rows beyond a segment's m are zero)
  const int nb_used = j * p;
  auto to_df = [&](const double* x, float2* y, int64_t m) {
    to_df_kernel<<<lapy_ceil_div(m, 256), 256, 0, st>>>(m, x, y);
    return lapy_check_launch("to_df_kernel");
  };
  // Y = X H per segment in double-float, register-tiled (H's columns staged in
  // shared memory); the one-thread-per-entry form when H is too tall for it
  auto gemm_nn_df_tiled = [&](const float2* X, int bs, int64_t bst, int na, const float2* H, int64_t hstride,
                              int ldh, double* Y, int ldy, int nb) -> int {
    constexpr size_t kSmemMax = 96 * 1024;
    const size_t smem = sizeof(float2) * (size_t)na * kNnTile;
    if (smem > kSmemMax) {
      gemm_nn_dfany_kernel<<<P.gt.nchunk, 256, 0, st>>>(X, bs, bst, na, H, hstride, ldh, Y, ldy, nb, P.gt.chunk_row,
                                                        P.gt.chunk_seg);
      return lapy_check_launch("gemm_nn_dfany_kernel");
    }
    LAPY_CUDA_TRY(cudaFuncSetAttribute(gemm_nn_df_tile_kernel<kNnTile>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kSmemMax));
    dim3 grid(P.gt.nchunk, lapy_ceil_div(nb, kNnTile));
    gemm_nn_df_tile_kernel<kNnTile><<<grid, 256, smem, st>>>(X, bs, bst, na, H, hstride, ldh, Y, ldy, nb,
                                                             P.gt.chunk_row, P.gt.chunk_seg);
    return lapy_check_launch("gemm_nn_df_tile_kernel");
  };
  LAPY_TRY(to_df(e.Sfinal, e.S_df, (int64_t)ns * lda * keff));
  LAPY_TRY(gemm_nn_df_tiled(e.basis_df, p, n * p, nb_used, e.S_df, (int64_t)lda * keff, keff, e.X, keff, keff));
  // final Rayleigh-Ritz with the exact A and M (projections in double-float;
  // AX and MX are only read by them, so they are split in place)
  LAPY_TRY(csr_spmm<double>(n, indptr, indices, a_vals, keff, e.X, e.AX, 1.0, 0.0, G, st));
  LAPY_TRY(ops.apply_M(e.X, e.MX, keff));
  LAPY_TRY(to_df(e.X, e.X_df, n * keff));
  for (double* buf : {e.AX, e.MX}) {
    to_df_inplace_kernel<<<lapy_ceil_div(n * keff, 256), 256, 0, st>>>(n * keff, buf);
    LAPY_TRY(lapy_check_launch("to_df_inplace_kernel"));
  }
  {
    dim3 grid(P.gt.nchunk, lapy_ceil_div(keff, 64), lapy_ceil_div(keff, 64));
    const dim3 g2 = ops.reduce_grid(keff, keff);
    gemm_tn_df_tile_kernel<<<grid, 256, 0, st>>>(e.X_df, keff, reinterpret_cast<const float2*>(e.AX), keff,
                                                 P.gt.chunk_row, e.partial);
    LAPY_TRY(lapy_check_launch("gemm_tn_df_tile_kernel"));
    gemm_tn_reduce_kernel<<<g2, 256, 0, st>>>(e.partial, keff, keff, P.gt.seg_chunk, e.Ak, (int64_t)keff * keff,
                                              keff);
    LAPY_TRY(lapy_check_launch("gemm_tn_reduce_kernel"));
    gemm_tn_df_tile_kernel<<<grid, 256, 0, st>>>(e.X_df, keff, reinterpret_cast<const float2*>(e.MX), keff,
                                                 P.gt.chunk_row, e.partial);
    LAPY_TRY(lapy_check_launch("gemm_tn_df_tile_kernel"));
    gemm_tn_reduce_kernel<<<g2, 256, 0, st>>>(e.partial, keff, keff, P.gt.seg_chunk, e.Mk, (int64_t)keff * keff,
                                              keff);
    LAPY_TRY(lapy_check_launch("gemm_tn_reduce_kernel"));
  }
  rr_prepare_kernel<<<ns, 128, 0, st>>>(keff, e.Ak, e.Mk, e.Cneg, e.fail);
  LAPY_TRY(lapy_check_launch("rr_prepare_kernel"));
  std::vector<int32_t> hk(ns, keff);
  LAPY_CUDA_TRY(cudaMemcpyAsync(e.nsize, hk.data(), 4 * ns, cudaMemcpyHostToDevice, st));
  LAPY_TRY(sym_eig_top(ns, e.Cneg, keff, e.nsize, keff, k, e.theta2, e.V, e.eigw2, nullptr, true, st));
  rr_finish_kernel<<<ns, 128, 0, st>>>(keff, k, e.Mk, e.V, e.theta2, evals);
  LAPY_TRY(lapy_check_launch("rr_finish_kernel"));
  // eigenvectors X V in double-float (X_df holds X; V split into S_df, which
  // is free now)
  LAPY_TRY(to_df(e.V, e.S_df, (int64_t)ns * keff * k));
  if (reorder) {  // eigenvectors in the system's order, then back to the caller's (AX is free here)
    LAPY_TRY(gemm_nn_df_tiled(e.X_df, keff, 0, keff, e.S_df, (int64_t)keff * k, k, e.AX, k, k));
    unpermute_rows_kernel<<<lapy_ceil_div(n * k, 256), 256, 0, st>>>(n, k, e.perm, e.AX, evecs);
    LAPY_TRY(lapy_check_launch("unpermute_rows_kernel"));
  } else {
    LAPY_TRY(gemm_nn_df_tiled(e.X_df, keff, 0, keff, e.S_df, (int64_t)keff * k, k, evecs, k, k));
  }
  LAPY_CUDA_TRY(cudaMemcpyAsync(hfail.data(), e.fail, 4 * ns, cudaMemcpyDeviceToHost, st));
  LAPY_CUDA_TRY(cudaStreamSynchronize(st));
  for (int s = 0; s < ns; ++s)
    if (hfail[s] && res->status[s] == LAPY_OK) res->status[s] = LAPY_ERR_BREAKDOWN;
  return LAPY_OK;
}

}  // namespace lapy

using namespace lapy;

static int eig_block_ok(int p) { return p == 1 || p == 2 || p == 4 || p == 8 || p == 16; }

static int eig_precond_ok(int pc) { return pc == kPrecJacobi || pc == kPrecTwoLevel; }

extern "C" size_t lapy_eigs_workspace_bytes(int64_t n, int64_t nnz, int nseg, const int32_t* seg_row, int k,
                                            int block, int max_vectors, int precond) {
  if (n <= 0 || nnz <= 0 || nseg <= 0 || !seg_row || k <= 0 || !eig_block_ok(block) || !eig_precond_ok(precond))
    return 0;
  EigPlan P;
  plan_eig(n, nnz, nseg, seg_row, k, block, max_vectors, precond, &P);
  return layout_eig(P, nullptr, nullptr);
}

extern "C" int lapy_eigs_shift_invert(int64_t n, const int32_t* indptr, const int32_t* indices,
                                      const double* a_vals, const double* m_vals, int m_is_diag, int64_t nnz,
                                      int nseg, const int32_t* seg_row, double sigma, int k, int block,
                                      int max_vectors, double tol, double inner_rtol, int inner_maxiter,
                                      int precond, uint64_t seed, double* evals, double* evecs, int32_t* status_out,
                                      int32_t* nbasis_out, int64_t* inner_iters_out, void* ws, size_t ws_bytes,
                                      void* stream) {
  return lapy_eigs_shift_invert_tuned(n, indptr, indices, a_vals, m_vals, m_is_diag, nnz, nseg, seg_row, sigma, k,
                                      block, max_vectors, tol, inner_rtol, inner_maxiter, precond, seed, evals, evecs,
                                      status_out, nbasis_out, inner_iters_out, ws, ws_bytes, stream, nullptr);
}

extern "C" int lapy_eigs_shift_invert_tuned(int64_t n, const int32_t* indptr, const int32_t* indices,
                                            const double* a_vals, const double* m_vals, int m_is_diag, int64_t nnz,
                                            int nseg, const int32_t* seg_row, double sigma, int k, int block,
                                            int max_vectors, double tol, double inner_rtol, int inner_maxiter,
                                            int precond, uint64_t seed, double* evals, double* evecs,
                                            int32_t* status_out, int32_t* nbasis_out, int64_t* inner_iters_out,
                                            void* ws, size_t ws_bytes, void* stream,
                                            const lapy_eigs_tuning* tuning) {
  lapy_eigs_tuning tn{0, 0.0, 0, 0, 0};
  if (tuning) tn = *tuning;
  if (tn.agg_target != 0 && (tn.agg_target < kAggTarget || tn.agg_target > 1024)) {
    lapy_set_last_message("eigs: agg_target must be 0 (default) or in [%d, 1024]", kAggTarget);
    return LAPY_ERR_INVALID;
  }
  if (tn.round_rtol != 0.0 && !(tn.round_rtol > 0.0 && tn.round_rtol < 1.0)) {
    lapy_set_last_message("eigs: round_rtol must be 0 (default) or in (0, 1)");
    return LAPY_ERR_INVALID;
  }
  if (tn.fold_pieces < 0 || tn.fold_aggs < 0 || tn.ctas_per_sm < 0 || tn.ctas_per_sm > 5) {
    lapy_set_last_message("eigs: fold thresholds must be >= 0 and ctas_per_sm in [0, 5]");
    return LAPY_ERR_INVALID;
  }
  if (n <= 0 || !indptr || !indices || !a_vals || !m_vals || nnz <= 0 || nseg <= 0 || !seg_row || k <= 0 ||
      !eig_block_ok(block) || !evals || !evecs || !ws || !(tol > 0) || !(inner_rtol > 0) || inner_maxiter <= 0 ||
      !eig_precond_ok(precond)) {
    lapy_set_last_message("eigs_shift_invert: invalid arguments");
    return LAPY_ERR_INVALID;
  }
  if (seg_row[0] != 0 || seg_row[nseg] != n) {
    lapy_set_last_message("eigs_shift_invert: segment rows must span [0, n)");
    return LAPY_ERR_INVALID;
  }
  for (int s = 0; s < nseg; ++s) {
    const int ns = seg_row[s + 1] - seg_row[s];
    if (ns < k + 2 * block + 1) {
      lapy_set_last_message("eigs_shift_invert: segment %d has %d rows; need >= k + 2*block + 1 = %d", s, ns,
                            k + 2 * block + 1);
      return LAPY_ERR_INVALID;
    }
  }
  EigPlan P;
  plan_eig(n, nnz, nseg, seg_row, k, block, max_vectors, precond, &P);
  if (tn.agg_target) P.agg_target = tn.agg_target;
  if (tn.fold_pieces) P.pcg.fold_pieces = tn.fold_pieces;
  if (tn.fold_aggs) P.pcg.fold_aggs = tn.fold_aggs;
  if (tn.ctas_per_sm) P.pcg.ctas_per_sm = tn.ctas_per_sm;
  if (ws_bytes < layout_eig(P, nullptr, nullptr)) return LAPY_ERR_WORKSPACE;
  EigPtrs e;
  layout_eig(P, (char*)(((uintptr_t)ws + 255) & ~uintptr_t(255)), &e);
  EigResult r;
  // FP32 refinement rounds of 1e-3 (on chip, 128 meshes of 642 to 40,962
  // vertices: 1e-2 / 3e-3 / 2e-3 / 1e-3 / 3e-4 / 1e-4 / 1e-5 per round took 597 /
  // 579 / 580 / 547 / 563 / 563 / 572 ms; tighter rounds spend iterations where
  // FP32 CG stalls, looser ones restart more often)
  const double round_rtol = tn.round_rtol > 0.0 ? tn.round_rtol : 1e-3;
  LAPY_TRY(eigs_run(P, e, indptr, indices, a_vals, m_vals, m_is_diag, sigma, tol, inner_rtol, round_rtol,
                    inner_maxiter, seed, evals, evecs, (cudaStream_t)stream, &r));
  for (int s = 0; s < nseg; ++s) {
    if (status_out) status_out[s] = r.status[s];
    if (nbasis_out) nbasis_out[s] = r.nbasis[s];
  }
  if (inner_iters_out) *inner_iters_out = r.inner_iters;
  return LAPY_OK;
}
