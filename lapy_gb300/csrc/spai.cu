// Learned factorised sparse approximate inverse (per-edge MLP).
//
// For an SPD system K on a symmetric mesh pattern, G is lower triangular on
// the pattern's lower part.  A per-edge network (6 -> 64 -> 64 -> 1, tanh,
// BF16 weights, FP32 accumulation; the forward pass's 64 x 64 layer on the
// tensor pipe) emits w_ij for every strictly lower entry;
// row i then gets
//   q_i = (e_i - w_i)' K (e_i - w_i),  G_ii = q_i^-1/2,  G_ij = -w_ij G_ii,
// so diag(G K G') = 1 and G'G is SPD for every w (w = 0 is Jacobi).  The
// training loss sum_i log q_i is the Kaporin functional of G K G' (its exact
// minimiser is FSAI); dL/dw_ij = (-2 K_ij + 2 sum_k w_ik K_jk) / q_i.
//
// Lower pattern: rows' entries with col <= row in CSR order (diagonal last);
// upper pattern: col >= row (diagonal first), with umap[u] the lower index of
// the transposed entry, so G' values are a gather of G's.
#include <cmath>
#include <cuda_bf16.h>
#include "common.cuh"
#include "scan.cuh"

namespace lapy {

constexpr int kNF = 6, kHid = 64;
constexpr int kOW1 = 0, kOB1 = kOW1 + kHid * kNF, kOW2 = kOB1 + kHid, kOB2 = kOW2 + kHid * kHid,
              kOW3 = kOB2 + kHid, kOB3 = kOW3 + kHid, kNParam = kOB3 + 1;
static_assert(kNParam == 4673, "parameter layout");

static size_t a256(size_t x) { return (x + 255) & ~size_t(255); }

// ---- pattern ---------------------------------------------------------------
__global__ void spai_count_kernel(int64_t n, const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                                  int32_t* __restrict__ lcnt, int32_t* __restrict__ ucnt) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int32_t l = 0, u = 0;
  for (int32_t k = indptr[i]; k < indptr[i + 1]; ++k) {
    const int32_t c = indices[k];
    l += c <= i;
    u += c >= i;
  }
  lcnt[i] = l;
  ucnt[i] = u;
}

__global__ void spai_fill_kernel(int64_t n, const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                                 const int32_t* __restrict__ lptr, const int32_t* __restrict__ uptr,
                                 int32_t* __restrict__ lcol, int32_t* __restrict__ lpos, int32_t* __restrict__ ucol) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int32_t l = lptr[i], u = uptr[i];
  for (int32_t k = indptr[i]; k < indptr[i + 1]; ++k) {
    const int32_t c = indices[k];
    if (c <= i) { lcol[l] = c; lpos[l] = k; ++l; }
    if (c >= i) { ucol[u] = c; ++u; }
  }
}

__global__ void spai_umap_kernel(int64_t n, const int32_t* __restrict__ uptr, const int32_t* __restrict__ ucol,
                                 const int32_t* __restrict__ lptr, const int32_t* __restrict__ lcol,
                                 int32_t* __restrict__ umap, int* __restrict__ missing) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  for (int32_t u = uptr[j]; u < uptr[j + 1]; ++u) {
    const int32_t i = ucol[u];  // entry (j, i), i >= j: the lower entry (i, j)
    int32_t lo = lptr[i], hi = lptr[i + 1] - 1, found = -1;
    while (lo <= hi) {
      const int32_t mid = (lo + hi) >> 1;
      const int32_t c = lcol[mid];
      if (c == (int32_t)j) { found = mid; break; }
      if (c < (int32_t)j) lo = mid + 1; else hi = mid - 1;
    }
    umap[u] = found;
    if (found < 0) atomicExch(missing, 1);
  }
}

// ---- features --------------------------------------------------------------
__global__ void spai_mass_kernel(int64_t n, const int32_t* __restrict__ indptr, const double* __restrict__ m_vals,
                                 int m_is_diag, double* __restrict__ mass) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (m_is_diag) {
    mass[i] = m_vals[i];
  } else {
    double s = 0.0;
    for (int32_t k = indptr[i]; k < indptr[i + 1]; ++k) s += m_vals[k];
    mass[i] = s;
  }
}

__device__ __forceinline__ int seg_of_row(const int32_t* __restrict__ seg_row, int nseg, int64_t i) {
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (seg_row[mid] <= i) lo = mid; else hi = mid - 1;
  }
  return lo;
}

template <typename T>
__global__ void spai_features_kernel(int64_t n, int nseg, const int32_t* __restrict__ seg_row, const T* __restrict__ v,
                                     const double* __restrict__ a_vals, const double* __restrict__ mass,
                                     const int32_t* __restrict__ lptr, const int32_t* __restrict__ lcol,
                                     const int32_t* __restrict__ lpos, const double* __restrict__ t_seg,
                                     const double* __restrict__ sigma_seg, const double* __restrict__ h_seg,
                                     float* __restrict__ feat) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int s = seg_of_row(seg_row, nseg, i);
  const double h = h_seg[s], h2 = h * h;
  const float f4 = (float)log(t_seg[s] / h2), f5 = (float)sigma_seg[s];
  const double mi = mass[i] / h2;
  const double xi = (double)v[3 * i], yi = (double)v[3 * i + 1], zi = (double)v[3 * i + 2];
  for (int32_t e = lptr[i]; e < lptr[i + 1]; ++e) {
    const int32_t j = lcol[e];
    const double dx = xi - (double)v[3 * (int64_t)j], dy = yi - (double)v[3 * (int64_t)j + 1],
                 dz = zi - (double)v[3 * (int64_t)j + 2];
    float* f = feat + (int64_t)e * kNF;
    f[0] = (float)(-a_vals[lpos[e]]);
    f[1] = (float)(sqrt(dx * dx + dy * dy + dz * dz) / h);
    f[2] = (float)mi;
    f[3] = (float)(mass[j] / h2);
    f[4] = f4;
    f[5] = f5;
  }
}

// ---- network on the tensor pipe ---------------------------------------------
// Forward pass with warp-level BF16 matrix instructions
// (mma.sync.m16n8k16, FP32 accumulate): a warp takes 16 edges at a time.
// Layer 1 (6 -> 64) runs on the FP32 pipe, each lane computing exactly the
// hidden units its A fragments hold (rows lane/4 and lane/4 + 8, units
// 16t + 2(lane%4) + {0,1} and + 8 of every 16-unit step t), so no shuffles
// are needed.  Layer 2 (64 x 64, 90 % of the work) is 32 tiles of 16 x 8 x 16
// per 16 edges; its input is split into three BF16 terms (hi + mid + lo,
// about 24 bits) so that the product with the BF16 weights keeps the FP32
// path's accuracy.  Layer 3 (64 -> 1) is folded into the epilogue of each
// 8-unit output tile, and the four lanes of a row sum their parts.
constexpr int kMmaWarps = 4;
constexpr int kW2Ld = kHid + 8;  // padded row of the staged W2 (BF16): conflict-free B-fragment loads

struct SpaiMmaSmem {
  __nv_bfloat16 W2[kHid * kW2Ld];
  float W1[kHid * kNF], b1[kHid], b2[kHid], W3[kHid], b3;
};

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  const uint32_t l = __bfloat16_as_ushort(__float2bfloat16_rn(lo));
  const uint32_t h = __bfloat16_as_ushort(__float2bfloat16_rn(hi));
  return l | (h << 16);
}

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__global__ void __launch_bounds__(32 * kMmaWarps) spai_forward_mma_kernel(int64_t ne, const float* __restrict__ feat,
                                                                          const __nv_bfloat16* __restrict__ wb,
                                                                          float* __restrict__ out) {
  __shared__ __align__(16) SpaiMmaSmem s;
  for (int p = threadIdx.x; p < kHid * kHid; p += blockDim.x) s.W2[(p / kHid) * kW2Ld + p % kHid] = wb[kOW2 + p];
  for (int p = threadIdx.x; p < kHid * kNF; p += blockDim.x) s.W1[p] = __bfloat162float(wb[kOW1 + p]);
  for (int p = threadIdx.x; p < kHid; p += blockDim.x) {
    s.b1[p] = __bfloat162float(wb[kOB1 + p]);
    s.b2[p] = __bfloat162float(wb[kOB2 + p]);
    s.W3[p] = __bfloat162float(wb[kOW3 + p]);
  }
  if (threadIdx.x == 0) s.b3 = __bfloat162float(wb[kOB3]);
  __syncthreads();
  const int lane = threadIdx.x & 31, grp = lane >> 2, tig = lane & 3;
  const int64_t warp0 = (int64_t)blockIdx.x * kMmaWarps + (threadIdx.x >> 5);
  const int64_t nwarp = (int64_t)gridDim.x * kMmaWarps;
  const uint32_t* W2w = reinterpret_cast<const uint32_t*>(s.W2);  // two BF16 per word
  for (int64_t tile = warp0; tile * 16 < ne; tile += nwarp) {
    const int64_t e0 = tile * 16 + grp, e1 = e0 + 8;
    float f0[kNF], f1[kNF];
#pragma unroll
    for (int k = 0; k < kNF; ++k) {
      f0[k] = e0 < ne ? feat[e0 * kNF + k] : 0.f;
      f1[k] = e1 < ne ? feat[e1 * kNF + k] : 0.f;
    }
    // layer 1 for this lane's fragment units; A fragments of layer 2 in
    // three BF16 terms
    uint32_t ahi[4][4], amid[4][4], alo[4][4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
#pragma unroll
      for (int half = 0; half < 2; ++half) {  // units 16t + 8 half + 2 tig + {0, 1}
        const int u = 16 * t + 8 * half + 2 * tig;
        float h[2][2];  // [row 0/8][unit u/u+1]
#pragma unroll
        for (int du = 0; du < 2; ++du) {
          float a0 = s.b1[u + du], a1 = s.b1[u + du];
#pragma unroll
          for (int k = 0; k < kNF; ++k) {
            a0 = fmaf(s.W1[(u + du) * kNF + k], f0[k], a0);
            a1 = fmaf(s.W1[(u + du) * kNF + k], f1[k], a1);
          }
          h[0][du] = tanhf(a0);
          h[1][du] = tanhf(a1);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int reg = 2 * half + r;  // a0: (row, k), a1: (row + 8, k), a2: (row, k + 8), a3: (row + 8, k + 8)
          float x0 = h[r][0], x1 = h[r][1];
          const float hi0 = __bfloat162float(__float2bfloat16_rn(x0)), hi1 = __bfloat162float(__float2bfloat16_rn(x1));
          ahi[t][reg] = pack_bf16x2(x0, x1);
          x0 -= hi0;
          x1 -= hi1;
          const float mi0 = __bfloat162float(__float2bfloat16_rn(x0)), mi1 = __bfloat162float(__float2bfloat16_rn(x1));
          amid[t][reg] = pack_bf16x2(x0, x1);
          alo[t][reg] = pack_bf16x2(x0 - mi0, x1 - mi1);
        }
      }
    }
    float part0 = 0.f, part1 = 0.f;  // layer-3 partial sums of rows grp and grp + 8
#pragma unroll 2
    for (int j = 0; j < kHid / 8; ++j) {  // output units 8j .. 8j + 7
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      const int n = 8 * j + grp;  // B column = W2 row
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint32_t b0 = W2w[(n * kW2Ld + 16 * t + 2 * tig) >> 1];
        const uint32_t b1 = W2w[(n * kW2Ld + 16 * t + 8 + 2 * tig) >> 1];
        mma_bf16_16816(acc, alo[t], b0, b1);
        mma_bf16_16816(acc, amid[t], b0, b1);
        mma_bf16_16816(acc, ahi[t], b0, b1);
      }
      const int o = 8 * j + 2 * tig;
      part0 = fmaf(s.W3[o], tanhf(acc[0] + s.b2[o]), part0);
      part0 = fmaf(s.W3[o + 1], tanhf(acc[1] + s.b2[o + 1]), part0);
      part1 = fmaf(s.W3[o], tanhf(acc[2] + s.b2[o]), part1);
      part1 = fmaf(s.W3[o + 1], tanhf(acc[3] + s.b2[o + 1]), part1);
    }
    part0 += __shfl_xor_sync(0xffffffffu, part0, 1);
    part0 += __shfl_xor_sync(0xffffffffu, part0, 2);
    part1 += __shfl_xor_sync(0xffffffffu, part1, 1);
    part1 += __shfl_xor_sync(0xffffffffu, part1, 2);
    if (tig == 0) {
      if (e0 < ne) out[e0] = s.b3 + part0;
      if (e1 < ne) out[e1] = s.b3 + part1;
    }
  }
}

// ---- factor, loss and dL/dw ------------------------------------------------
__device__ __forceinline__ double k_at(const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                                       const double* __restrict__ kv, int32_t row, int32_t col) {
  int32_t lo = indptr[row], hi = indptr[row + 1] - 1;
  while (lo <= hi) {
    const int32_t mid = (lo + hi) >> 1;
    const int32_t c = indices[mid];
    if (c == col) return kv[mid];
    if (c < col) lo = mid + 1; else hi = mid - 1;
  }
  return 0.0;
}

__global__ void spai_factor_kernel(int64_t n, const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                                   const double* __restrict__ kv, const int32_t* __restrict__ lptr,
                                   const int32_t* __restrict__ lcol, const int32_t* __restrict__ lpos,
                                   const float* __restrict__ w, float* __restrict__ g, double* __restrict__ logq,
                                   float* __restrict__ dldw) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t e0 = lptr[i], ed = lptr[i + 1] - 1;  // ed: the diagonal entry
  const double kii = kv[lpos[ed]];
  double q = kii;
  for (int32_t e = e0; e < ed; ++e) {
    const double we = w[e];
    q -= 2.0 * we * kv[lpos[e]];
    for (int32_t f = e0; f < ed; ++f) q += we * (double)w[f] * k_at(indptr, indices, kv, lcol[e], lcol[f]);
  }
  const bool ok = q > 0.0 && isfinite(q);
  if (!ok) q = kii;  // the Jacobi row
  const double gd = 1.0 / sqrt(q);
  g[ed] = (float)gd;
  if (logq) logq[i] = log(q);
  if (dldw) dldw[ed] = 0.f;
  for (int32_t e = e0; e < ed; ++e) {
    g[e] = ok ? (float)(-(double)w[e] * gd) : 0.f;
    if (dldw) {
      double dq = -2.0 * kv[lpos[e]];
      for (int32_t f = e0; f < ed; ++f) dq += 2.0 * (double)w[f] * k_at(indptr, indices, kv, lcol[e], lcol[f]);
      dldw[e] = ok ? (float)(dq / q) : 0.f;
    }
  }
}

__global__ void spai_gather_kernel(int64_t m, const int32_t* __restrict__ umap, const float* __restrict__ gl,
                                   float* __restrict__ gu) {
  const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (u < m) gu[u] = gl[umap[u]];
}

// ---- backward --------------------------------------------------------------
// Gradient of sum_e dw_e w_e on the tensor pipe (mma.sync.m16n8k16 BF16, FP32
// accumulate), four warps per CTA, 16 edges per warp and tile.  A warp
// recomputes its edges' activations as the forward kernel does, forms
// dz2 = d3 W3 (1 - h2^2) and dh1 = dz2 W2 with the accumulator fragments of
// one product as the A fragments of the next, and leaves h1, dz2 and dz1 in
// shared memory; then every warp accumulates 16 rows of dW2 = dz2' h1 and of
// [dW1 | db1] = dz1' [f | 1] over the CTA's 64 edges in registers.  Activations
// and gradients are split into three BF16 terms (about 24 bits), products of
// two split factors keep the six terms above 2^-24, and the 16-wide products
// of a sum are added in FP32 (the tensor pipe rounds its running sums towards
// zero).  Against 64 bits on the same FP32 inputs the gradient is off by 7.4e-8
// (geometric mean over 24 batches of 46,000 to 912,000 entries), 2.8e-7 for the
// FP32 path it replaces (one thread per edge, one thread per group of
// parameters), which took 1,054 us for 462,000 entries, 11 TFLOP/s.  Whole
// gradient pass there: 1,192 -> 364 us, off by 6.40e-6, before 6.42e-6.
constexpr int kBwdWarps = 4;
constexpr int kBwdThreads = 32 * kBwdWarps;
constexpr int kBwdEdges = 16 * kBwdWarps;

struct SpaiBwdSmem {
  SpaiMmaSmem w;
  alignas(16) __nv_bfloat16 W2T[kHid * kW2Ld];                 // W2T[k][o] = W2[o][k]
  alignas(16) __nv_bfloat16 h1[3][kBwdEdges][kW2Ld];           // split activations, gradients
  alignas(16) __nv_bfloat16 dz2[3][kBwdEdges][kW2Ld];
  alignas(16) __nv_bfloat16 dz1[3][kBwdEdges][kW2Ld];
  alignas(16) __nv_bfloat16 f[3][kBwdEdges][8];                // features, a one, a zero
  float g3[kBwdWarps][kHid], d3[kBwdWarps];
};

// x0, x1 as three packed BF16 pairs whose sums are the values to about 24 bits.
__device__ __forceinline__ void split3(float x0, float x1, uint32_t (&p)[3]) {
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const __nv_bfloat16 h0 = __float2bfloat16_rn(x0), h1 = __float2bfloat16_rn(x1);
    p[t] = (uint32_t)__bfloat16_as_ushort(h0) | ((uint32_t)__bfloat16_as_ushort(h1) << 16);
    x0 -= __bfloat162float(h0);
    x1 -= __bfloat162float(h1);
  }
}

__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const void* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void ldsm2t(uint32_t& r0, uint32_t& r1, const void* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
               : "=r"(r0), "=r"(r1)
               : "r"(a)
               : "memory");
}

__global__ void __launch_bounds__(kBwdThreads, 2) spai_backward_kernel(int64_t ne, const float* __restrict__ feat,
                                                                       const __nv_bfloat16* __restrict__ wb,
                                                                       const float* __restrict__ dw,
                                                                       float* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char smem[];
  SpaiBwdSmem& s = *reinterpret_cast<SpaiBwdSmem*>(smem);
  for (int p = threadIdx.x; p < kHid * kHid; p += blockDim.x) {
    const __nv_bfloat16 v = wb[kOW2 + p];
    s.w.W2[(p / kHid) * kW2Ld + p % kHid] = v;
    s.W2T[(p % kHid) * kW2Ld + p / kHid] = v;
  }
  for (int p = threadIdx.x; p < kHid * kNF; p += blockDim.x) s.w.W1[p] = __bfloat162float(wb[kOW1 + p]);
  for (int p = threadIdx.x; p < kHid; p += blockDim.x) {
    s.w.b1[p] = __bfloat162float(wb[kOB1 + p]);
    s.w.b2[p] = __bfloat162float(wb[kOB2 + p]);
    s.w.W3[p] = __bfloat162float(wb[kOW3 + p]);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = lane >> 2, tig = lane & 3;
  const uint32_t* W2w = reinterpret_cast<const uint32_t*>(s.w.W2);
  const uint32_t* W2Tw = reinterpret_cast<const uint32_t*>(s.W2T);
  float gW2[8][4], gW1[4] = {0.f, 0.f, 0.f, 0.f}, gb2[4] = {0.f, 0.f, 0.f, 0.f};
  float gW3[8][2], gb3 = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
#pragma unroll
    for (int c = 0; c < 4; ++c) gW2[j][c] = 0.f;
    gW3[j][0] = gW3[j][1] = 0.f;
  }
  const uint32_t ones = grp == 0 ? 0x3f803f80u : 0u;  // B fragment whose column 0 is all ones
  const int r0 = 16 * warp + grp;                     // this lane's rows of the tile: r0, r0 + 8
  for (int64_t base = (int64_t)blockIdx.x * kBwdEdges; base < ne; base += (int64_t)gridDim.x * kBwdEdges) {
    const int64_t e0 = base + r0, e1 = e0 + 8;
    float f0[kNF], f1[kNF];
#pragma unroll
    for (int k = 0; k < kNF; ++k) {
      f0[k] = e0 < ne ? feat[e0 * kNF + k] : 0.f;
      f1[k] = e1 < ne ? feat[e1 * kNF + k] : 0.f;
    }
    const float d0 = e0 < ne ? dw[e0] : 0.f, d1 = e1 < ne ? dw[e1] : 0.f;
    // ---- layer 1: units 16 t + 8 half + 2 tig + {0, 1} of both rows
    float h[8][4];         // [8-unit tile][row0 u, row0 u + 1, row1 u, row1 u + 1]
    uint32_t a1[3][4][4];  // their A fragments, split
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int u = 8 * j + 2 * tig;
#pragma unroll
      for (int du = 0; du < 2; ++du) {
        float x0 = s.w.b1[u + du], x1 = s.w.b1[u + du];
#pragma unroll
        for (int k = 0; k < kNF; ++k) {
          x0 = fmaf(s.w.W1[(u + du) * kNF + k], f0[k], x0);
          x1 = fmaf(s.w.W1[(u + du) * kNF + k], f1[k], x1);
        }
        h[j][du] = tanhf(x0);
        h[j][2 + du] = tanhf(x1);
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        uint32_t p[3];
        split3(h[j][2 * r], h[j][2 * r + 1], p);
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          a1[t][j >> 1][2 * (j & 1) + r] = p[t];
          *reinterpret_cast<uint32_t*>(&s.h1[t][r0 + 8 * r][u]) = p[t];
        }
      }
    }
    // ---- layer 2, dz2 and its A fragments
    uint32_t a2[3][4][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      const int n = 8 * j + grp;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint32_t b0 = W2w[(n * kW2Ld + 16 * t + 2 * tig) >> 1];
        const uint32_t b1 = W2w[(n * kW2Ld + 16 * t + 8 + 2 * tig) >> 1];
        float hi[4] = {0.f, 0.f, 0.f, 0.f};
        mma_bf16_16816(hi, a1[2][t], b0, b1);
        mma_bf16_16816(hi, a1[1][t], b0, b1);
        mma_bf16_16816(hi, a1[0][t], b0, b1);
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] += hi[c];
      }
      const int u = 8 * j + 2 * tig;
      float z[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int o = u + (c & 1);
        const float d = c < 2 ? d0 : d1;
        const float h2 = tanhf(acc[c] + s.w.b2[o]);
        z[c] = d * s.w.W3[o] * (1.f - h2 * h2);
        gW3[j][c & 1] = fmaf(d, h2, gW3[j][c & 1]);
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        uint32_t p[3];
        split3(z[2 * r], z[2 * r + 1], p);
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          a2[t][j >> 1][2 * (j & 1) + r] = p[t];
          *reinterpret_cast<uint32_t*>(&s.dz2[t][r0 + 8 * r][u]) = p[t];
        }
      }
    }
    gb3 += tig == 0 ? d0 + d1 : 0.f;
    // ---- dz1 = (dz2 W2) (1 - h1^2)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      const int n = 8 * j + grp;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint32_t b0 = W2Tw[(n * kW2Ld + 16 * t + 2 * tig) >> 1];
        const uint32_t b1 = W2Tw[(n * kW2Ld + 16 * t + 8 + 2 * tig) >> 1];
        float hi[4] = {0.f, 0.f, 0.f, 0.f};
        mma_bf16_16816(hi, a2[2][t], b0, b1);
        mma_bf16_16816(hi, a2[1][t], b0, b1);
        mma_bf16_16816(hi, a2[0][t], b0, b1);
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] += hi[c];
      }
      const int u = 8 * j + 2 * tig;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        uint32_t p[3];
        const float g0 = h[j][2 * r], g1 = h[j][2 * r + 1];
        split3(acc[2 * r] * (1.f - g0 * g0), acc[2 * r + 1] * (1.f - g1 * g1), p);
#pragma unroll
        for (int t = 0; t < 3; ++t) *reinterpret_cast<uint32_t*>(&s.dz1[t][r0 + 8 * r][u]) = p[t];
      }
    }
    if (tig < 2) {  // the rows' features, a one behind them
#pragma unroll
      for (int q = 0; q < 4; q += 2) {
        const int k = 4 * tig + q;
        uint32_t p[3];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          float x0, x1;
          if (tig == 0) {
            x0 = r ? f1[q] : f0[q];
            x1 = r ? f1[q + 1] : f0[q + 1];
          } else {
            x0 = q == 0 ? (r ? f1[4] : f0[4]) : 1.f;
            x1 = q == 0 ? (r ? f1[5] : f0[5]) : 0.f;
          }
          split3(x0, x1, p);
#pragma unroll
          for (int t = 0; t < 3; ++t) *reinterpret_cast<uint32_t*>(&s.f[t][r0 + 8 * r][k]) = p[t];
        }
      }
    }
    __syncthreads();
    // ---- parameter gradients: rows 16 warp .. 16 warp + 15 of dW2, dW1, db
    const int o0 = 16 * warp;
    const int ar = ((lane >> 4) << 3) + (lane & 7), ac = o0 + (((lane >> 3) & 1) << 3);  // ldmatrix rows of A
    const int br = (((lane >> 3) & 1) << 3) + (lane & 7), bc = (lane >> 4) << 3;          // of two B tiles
    // (each tile summed on its own and added in FP32: the tensor pipe rounds
    // its running sums towards zero)
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      float t0[4] = {0.f, 0.f, 0.f, 0.f}, t1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
      for (int kt = 0; kt < kBwdEdges / 16; ++kt) {
        uint32_t az[3][4], bh[3][4];
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          ldsm4t(az[t], &s.dz2[t][16 * kt + ar][ac]);
          ldsm4t(bh[t], &s.h1[t][16 * kt + br][8 * j + bc]);
        }
        // smallest products first
        constexpr int ta[6] = {2, 0, 1, 1, 0, 0}, tb[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          mma_bf16_16816(t0, az[ta[q]], bh[tb[q]][0], bh[tb[q]][1]);
          mma_bf16_16816(t1, az[ta[q]], bh[tb[q]][2], bh[tb[q]][3]);
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        gW2[j][c] += t0[c];
        gW2[j + 1][c] += t1[c];
      }
    }
    {
      float t0[4] = {0.f, 0.f, 0.f, 0.f}, t1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
      for (int kt = 0; kt < kBwdEdges / 16; ++kt) {
        uint32_t az[3][4], bf[3][2];
#pragma unroll
        for (int t = 0; t < 3; ++t) ldsm4t(az[t], &s.dz2[t][16 * kt + ar][ac]);
#pragma unroll
        for (int t = 2; t >= 0; --t) mma_bf16_16816(t1, az[t], ones, ones);
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          ldsm4t(az[t], &s.dz1[t][16 * kt + ar][ac]);
          ldsm2t(bf[t][0], bf[t][1], &s.f[t][16 * kt + (lane & 15)][0]);
        }
        constexpr int ta[6] = {2, 0, 1, 1, 0, 0}, tb[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
        for (int q = 0; q < 6; ++q) mma_bf16_16816(t0, az[ta[q]], bf[tb[q]][0], bf[tb[q]][1]);
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        gW1[c] += t0[c];
        gb2[c] += t1[c];
      }
    }
    __syncthreads();
  }
  float* out = partial + (int64_t)blockIdx.x * kNParam;
  const int oa = 16 * warp + grp, ob = oa + 8;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int k = 8 * j + 2 * tig;
    out[kOW2 + oa * kHid + k] = gW2[j][0];
    out[kOW2 + oa * kHid + k + 1] = gW2[j][1];
    out[kOW2 + ob * kHid + k] = gW2[j][2];
    out[kOW2 + ob * kHid + k + 1] = gW2[j][3];
  }
  if (tig < 3) {  // columns 0 .. 5: W1
    out[kOW1 + oa * kNF + 2 * tig] = gW1[0];
    out[kOW1 + oa * kNF + 2 * tig + 1] = gW1[1];
    out[kOW1 + ob * kNF + 2 * tig] = gW1[2];
    out[kOW1 + ob * kNF + 2 * tig + 1] = gW1[3];
  } else {  // column 6: the one
    out[kOB1 + oa] = gW1[0];
    out[kOB1 + ob] = gW1[2];
  }
  if (tig == 0) {
    out[kOB2 + oa] = gb2[0];
    out[kOB2 + ob] = gb2[2];
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int du = 0; du < 2; ++du) {
      float v = gW3[j][du];
      v += __shfl_xor_sync(0xffffffffu, v, 4);
      v += __shfl_xor_sync(0xffffffffu, v, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 16);
      if (grp == 0) s.g3[warp][8 * j + 2 * tig + du] = v;
    }
  gb3 = warp_sum(gb3);
  if (lane == 0) s.d3[warp] = gb3;
  __syncthreads();
  for (int u = threadIdx.x; u < kHid; u += blockDim.x) {
    float v = s.g3[0][u];
    for (int w = 1; w < kBwdWarps; ++w) v += s.g3[w][u];
    out[kOW3 + u] = v;
  }
  if (threadIdx.x == 0) {
    float v = s.d3[0];
    for (int w = 1; w < kBwdWarps; ++w) v += s.d3[w];
    out[kOB3] = v;
  }
}

// Eight lanes per parameter (four neighbouring parameters per warp), lane k
// adding blocks k, k + 8, ...
__global__ void spai_grad_reduce_kernel(int nblk, const float* __restrict__ partial, float scale,
                                        float* __restrict__ grad) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  const int p = t / 32 * 4 + (lane & 3);
  float a = 0.f;
  if (p < kNParam)
    for (int b = lane >> 2; b < nblk; b += 8) a += partial[(int64_t)b * kNParam + p];
  for (int o = 16; o >= 4; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if (lane < 4 && p < kNParam) grad[p] = a * scale;
}

__global__ void spai_adam_kernel(int np, float* __restrict__ theta, const float* __restrict__ grad,
                                 float* __restrict__ m, float* __restrict__ v, __nv_bfloat16* __restrict__ wb,
                                 float lr, float b1, float b2, float eps, float c1, float c2) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  const float g = grad[p];
  const float mp = b1 * m[p] + (1.f - b1) * g;
  const float vp = b2 * v[p] + (1.f - b2) * g * g;
  m[p] = mp;
  v[p] = vp;
  const float th = theta[p] - lr * (mp / c1) / (sqrtf(vp / c2) + eps);
  theta[p] = th;
  wb[p] = __float2bfloat16_rn(th);
}

__global__ void spai_to_bf16_kernel(int np, const float* __restrict__ theta, __nv_bfloat16* __restrict__ wb) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < np) wb[p] = __float2bfloat16_rn(theta[p]);
}

static size_t bwd_smem() { return sizeof(SpaiBwdSmem); }

}  // namespace lapy

using namespace lapy;

extern "C" int lapy_spai_param_count(void) { return kNParam; }

extern "C" size_t lapy_spai_pattern_workspace_bytes(int64_t n) {
  return a256(4 * (size_t)(n + 1)) * 2 + a256(4 * (size_t)scan_scratch_elems(n + 1)) + 512;
}

extern "C" int lapy_spai_pattern(int64_t n, const int32_t* indptr, const int32_t* indices, int64_t nnz,
                                 int32_t* lptr, int32_t* lcol, int32_t* lpos, int32_t* uptr, int32_t* ucol,
                                 int32_t* umap, void* work, size_t ws_bytes, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (n <= 0 || !indptr || !indices || nnz < n || !lptr || !lcol || !lpos || !uptr || !ucol || !umap || !work)
    return LAPY_ERR_INVALID;
  if ((nnz + n) % 2 != 0) {
    lapy_set_last_message("spai_pattern: the pattern is not symmetric with a full diagonal");
    return LAPY_ERR_PATTERN;
  }
  if (ws_bytes < lapy_spai_pattern_workspace_bytes(n)) return LAPY_ERR_WORKSPACE;
  char* w = (char*)(((uintptr_t)work + 255) & ~uintptr_t(255));
  int32_t* lcnt = (int32_t*)w; w += a256(4 * (size_t)(n + 1));
  int32_t* ucnt = (int32_t*)w; w += a256(4 * (size_t)(n + 1));
  int32_t* scratch = (int32_t*)w; w += a256(4 * (size_t)scan_scratch_elems(n + 1));
  int* missing = (int*)w;
  const unsigned nb = lapy_ceil_div(n, 256);
  spai_count_kernel<<<nb, 256, 0, stream>>>(n, indptr, indices, lcnt, ucnt);
  LAPY_TRY(lapy_check_launch("spai_count_kernel"));
  LAPY_TRY(exclusive_scan_i32(lcnt, lptr, n, scratch, stream));
  LAPY_TRY(exclusive_scan_i32(ucnt, uptr, n, scratch, stream));
  int32_t tot[2] = {0, 0};
  LAPY_CUDA_TRY(cudaMemcpyAsync(&tot[0], lptr + n, 4, cudaMemcpyDeviceToHost, stream));
  LAPY_CUDA_TRY(cudaMemcpyAsync(&tot[1], uptr + n, 4, cudaMemcpyDeviceToHost, stream));
  LAPY_CUDA_TRY(cudaStreamSynchronize(stream));
  if ((int64_t)tot[0] != (nnz + n) / 2 || tot[1] != tot[0]) {
    lapy_set_last_message("spai_pattern: the pattern is not symmetric with a full diagonal");
    return LAPY_ERR_PATTERN;
  }
  spai_fill_kernel<<<nb, 256, 0, stream>>>(n, indptr, indices, lptr, uptr, lcol, lpos, ucol);
  LAPY_TRY(lapy_check_launch("spai_fill_kernel"));
  LAPY_CUDA_TRY(cudaMemsetAsync(missing, 0, sizeof(int), stream));
  spai_umap_kernel<<<nb, 256, 0, stream>>>(n, uptr, ucol, lptr, lcol, umap, missing);
  LAPY_TRY(lapy_check_launch("spai_umap_kernel"));
  int miss = 0;
  LAPY_CUDA_TRY(cudaMemcpyAsync(&miss, missing, sizeof(int), cudaMemcpyDeviceToHost, stream));
  LAPY_CUDA_TRY(cudaStreamSynchronize(stream));
  if (miss) {
    lapy_set_last_message("spai_pattern: the pattern is not symmetric");
    return LAPY_ERR_PATTERN;
  }
  return LAPY_OK;
}

extern "C" int lapy_spai_features(int64_t n, int nseg, const int32_t* seg_row, const void* v, int coords_f32,
                                  const int32_t* indptr, const double* a_vals, const double* m_vals, int m_is_diag,
                                  const int32_t* lptr, const int32_t* lcol, const int32_t* lpos, const double* t_seg,
                                  const double* sigma_seg, const double* h_seg, double* mass_work, float* feat,
                                  void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (n <= 0 || nseg <= 0 || !seg_row || !v || !indptr || !a_vals || !m_vals || !lptr || !lcol || !lpos || !t_seg ||
      !sigma_seg || !h_seg || !mass_work || !feat)
    return LAPY_ERR_INVALID;
  const unsigned nb = lapy_ceil_div(n, 256);
  spai_mass_kernel<<<nb, 256, 0, stream>>>(n, indptr, m_vals, m_is_diag, mass_work);
  LAPY_TRY(lapy_check_launch("spai_mass_kernel"));
  if (coords_f32)
    spai_features_kernel<float><<<nb, 256, 0, stream>>>(n, nseg, seg_row, (const float*)v, a_vals, mass_work, lptr,
                                                       lcol, lpos, t_seg, sigma_seg, h_seg, feat);
  else
    spai_features_kernel<double><<<nb, 256, 0, stream>>>(n, nseg, seg_row, (const double*)v, a_vals, mass_work, lptr,
                                                        lcol, lpos, t_seg, sigma_seg, h_seg, feat);
  return lapy_check_launch("spai_features_kernel");
}

extern "C" int lapy_spai_forward(int64_t ne, const float* feat, const void* weights_bf16, float* w_out,
                                 void* stream_) {
  if (ne <= 0 || !feat || !weights_bf16 || !w_out) return LAPY_ERR_INVALID;
  const unsigned grid = std::min<unsigned>(lapy_ceil_div(ne, 16 * kMmaWarps), 16u * lapy_num_sms());
  spai_forward_mma_kernel<<<grid, 32 * kMmaWarps, 0, (cudaStream_t)stream_>>>(
      ne, feat, (const __nv_bfloat16*)weights_bf16, w_out);
  return lapy_check_launch("spai_forward_mma_kernel");
}

extern "C" int lapy_spai_factor(int64_t n, const int32_t* indptr, const int32_t* indices, const double* k_vals,
                                const int32_t* lptr, const int32_t* lcol, const int32_t* lpos, const float* w,
                                float* g_lower, double* logq, float* dldw, void* stream_) {
  if (n <= 0 || !indptr || !indices || !k_vals || !lptr || !lcol || !lpos || !w || !g_lower) return LAPY_ERR_INVALID;
  spai_factor_kernel<<<lapy_ceil_div(n, 128), 128, 0, (cudaStream_t)stream_>>>(n, indptr, indices, k_vals, lptr,
                                                                             lcol, lpos, w, g_lower, logq, dldw);
  return lapy_check_launch("spai_factor_kernel");
}

extern "C" int lapy_spai_transpose_values(int64_t m, const int32_t* umap, const float* g_lower, float* g_upper,
                                          void* stream_) {
  if (m <= 0 || !umap || !g_lower || !g_upper) return LAPY_ERR_INVALID;
  spai_gather_kernel<<<lapy_ceil_div(m, 256), 256, 0, (cudaStream_t)stream_>>>(m, umap, g_lower, g_upper);
  return lapy_check_launch("spai_gather_kernel");
}

static int bwd_blocks(int64_t ne) {
  return std::max(1, std::min<int>((int)std::min<int64_t>(lapy_ceil_div(ne, kBwdEdges), 1 << 20),
                                   2 * lapy_num_sms()));
}

extern "C" size_t lapy_spai_backward_workspace_bytes(int64_t ne) {
  return a256(4 * (size_t)kNParam * bwd_blocks(std::max<int64_t>(ne, 1))) + 256;
}

extern "C" int lapy_spai_backward(int64_t ne, const float* feat, const void* weights_bf16, const float* dldw,
                                  float scale, float* grad, void* work, size_t ws_bytes, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (ne <= 0 || !feat || !weights_bf16 || !dldw || !grad || !work) return LAPY_ERR_INVALID;
  const int nblk = bwd_blocks(ne);
  if (ws_bytes < a256(4 * (size_t)kNParam * nblk) + 256) return LAPY_ERR_WORKSPACE;
  float* partial = (float*)(((uintptr_t)work + 255) & ~uintptr_t(255));
  const size_t smem = bwd_smem();
  LAPY_CUDA_TRY(cudaFuncSetAttribute(spai_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  spai_backward_kernel<<<nblk, kBwdThreads, smem, stream>>>(ne, feat, (const __nv_bfloat16*)weights_bf16, dldw,
                                                            partial);
  LAPY_TRY(lapy_check_launch("spai_backward_kernel"));
  spai_grad_reduce_kernel<<<lapy_ceil_div(kNParam, 32), 256, 0, stream>>>(nblk, partial, scale, grad);
  return lapy_check_launch("spai_grad_reduce_kernel");
}

extern "C" int lapy_spai_adam(int nparam, float* theta, const float* grad, float* m, float* v, void* weights_bf16,
                              float lr, float beta1, float beta2, float eps, int step, void* stream_) {
  if (nparam <= 0 || !theta || !grad || !m || !v || !weights_bf16 || step <= 0) return LAPY_ERR_INVALID;
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  spai_adam_kernel<<<lapy_ceil_div(nparam, 256), 256, 0, (cudaStream_t)stream_>>>(
      nparam, theta, grad, m, v, (__nv_bfloat16*)weights_bf16, lr, beta1, beta2, eps, c1, c2);
  return lapy_check_launch("spai_adam_kernel");
}

extern "C" int lapy_spai_weights_to_bf16(int nparam, const float* theta, void* weights_bf16, void* stream_) {
  if (nparam <= 0 || !theta || !weights_bf16) return LAPY_ERR_INVALID;
  spai_to_bf16_kernel<<<lapy_ceil_div(nparam, 256), 256, 0, (cudaStream_t)stream_>>>(nparam, theta,
                                                                                   (__nv_bfloat16*)weights_bf16);
  return lapy_check_launch("spai_to_bf16_kernel");
}
