// On-chip refined PCG: one thread-block cluster per (segment, column group).
//
// The persistent PCG of pcg.cu streams every vector and the matrix from HBM
// or L2 in each iteration and passes three or four grid barriers; on meshes of
// a few thousand rows it is bound by those barriers and by dependent L2 round
// trips (25 to 40 us per iteration for one 642- to 10,242-row mesh).  Here a
// mesh lives on the SMs of one cluster: the residual, the solution and (where
// registers allow) the search direction in registers, one row per lane; the
// direction in shared memory too, where neighbouring rows are read; copies of the
// rows that other CTAs of the cluster own; the FP32 matrix with 16-bit column
// codes in shared memory.  Copies of directions are updated where they are read
// (p = z + beta p; their owners store z through distributed shared memory), so
// that r'z is reduced by the barrier that publishes z, and q = K p, p'q are
// computed as plain CG has them: three cluster barriers per iteration with the
// two-level preconditioner, two with Jacobi (one more where the copies are
// many).  (The Chronopoulos-Gear form, q by recurrence and p'q = z'K z - beta r'z
// / alpha_old, needs no more barriers either, but the difference cancels where K
// is close to singular in FP32: spheres of radius 0.02 and 0.03 at sigma = -0.01
// took up to 25 times the iterations or failed.)  Every CTA adds the partial sums
// of all CTAs in one order, so each takes the same decisions and a solve is
// reproducible to the bit.
//
// The FP64 refinement (true residual B - K X in FP64, FP32 correction solves)
// runs in the same kernel: a solve is one launch per cluster size.
//
// Measured per PCG iteration (persistent PCG -> here): one 642-vertex surface,
// 8 columns, two-level 35 -> 2.8 us; 10,242 vertices 45 -> 5.0 us; 11,466-vertex
// solid 47 -> 6.0 us; 40,962 vertices, one column, Jacobi 17 -> 3.9 us; 24
// meshes of 642 to 40,962 vertices, 4 columns 60 -> 14 us, 128 of them 106 ->
// 62 us.  What bounds it now: for small meshes the chain of reductions and
// barriers; for full CTAs (counters of eight meshes, clusters of 16 CTAs)
// instruction issue and shared-memory wavefronts, 42 % each of the active
// cycles, between those barriers: waits for shared memory are first among the
// stalls, for the CTA's and the cluster's barriers next.
#include <algorithm>
#include <cmath>
#include <vector>
#include "cluster.cuh"
#include "fork_join.h"
#include "pcg_cluster.cuh"
#include "scan.cuh"
#include "slice_starts.h"

namespace lapy {

static size_t a256(size_t x) { return (x + 255) & ~size_t(255); }

constexpr int kClMaxWarps = 16;
constexpr int kClMaxRows = 4096;  // rows per CTA a 12-bit code can name
constexpr size_t kClSmemMax = 226 * 1024;  // dynamic; the rest of the 227 KB is static
constexpr int32_t kClActive = INT32_MAX;
// Most halo rows whose directions a CTA updates itself, from copies of z.  More
// of them, or copies that do not fit, are sent as directions, after one more
// barrier: 390 and 2,023 rows a CTA are 9 and 3 % slower that way (geodesics of
// 40,962 vertices, eigs of 11,466), 15,348 rows 17 % faster (Poisson on 40,962
// vertices in the order of refinement: 11.9 -> 9.9 ms).
constexpr int kZHalo = 5000;

struct ClArgs {
  int p;
  const double* B;
  double* X;
  const int32_t* indptr;
  const int32_t* indices;
  const double* k64;
  const float* dinv;
  const ClusterCta* cta;
  const int32_t* unit_row;
  const int32_t* unit_agg;
  const int32_t* agg_unit;
  const int32_t* slice_ptr;
  const uint16_t* code;
  const float* val;
  const float* diag;
  const int32_t* push_ptr;
  const uint32_t* push;
  const int32_t* seg_agg;
  const int64_t* kinv_off;
  const uint16_t* kinv;
  const float* kvec;
  const float* kscale;
  double rtol, inner_rtol;
  int max_rounds, maxiter;
  int32_t* state;
  double* relres2;
  unsigned long long* ctl;
  int mat_smem, coarse_smem, z_halo;
  // shared memory layout (byte offsets, the same in every CTA of a launch) and
  // rows reserved for the halo's z and for p (own rows and halo)
  int o_z, o_p, o_rc, o_yc, o_up, o_wp, o_mail, o_tab, o_push, o_val, o_code, o_coarse;
  int zrows, prows;
};

// Row `slot` of a z / p array of this CTA.
// NP = 8 keeps two planes of four columns, so that 16-byte reads of
// consecutive rows touch consecutive words.
template <int NP>
__device__ __forceinline__ void cl_load(const float* base, int plane_f, int slot, float (&x)[NP]) {
  if constexpr (NP == 1) {
    x[0] = base[slot];
  } else if constexpr (NP == 2) {
    const float2 v = reinterpret_cast<const float2*>(base)[slot];
    x[0] = v.x; x[1] = v.y;
  } else {
#pragma unroll
    for (int h = 0; h < NP / 4; ++h) {
      const float4 v = reinterpret_cast<const float4*>(base + h * plane_f)[slot];
      x[4 * h] = v.x; x[4 * h + 1] = v.y; x[4 * h + 2] = v.z; x[4 * h + 3] = v.w;
    }
  }
}
template <int NP>
__device__ __forceinline__ void cl_save(float* base, int plane_f, int slot, const float (&x)[NP]) {
  if constexpr (NP == 1) {
    base[slot] = x[0];
  } else if constexpr (NP == 2) {
    reinterpret_cast<float2*>(base)[slot] = make_float2(x[0], x[1]);
  } else {
#pragma unroll
    for (int h = 0; h < NP / 4; ++h)
      reinterpret_cast<float4*>(base + h * plane_f)[slot] =
          make_float4(x[4 * h], x[4 * h + 1], x[4 * h + 2], x[4 * h + 3]);
  }
}

// Warp sums of V per-lane values by halving exchanges (V + 4 - log2 V
// shuffles instead of 5 V): lane l ends with the total of value
// l >> (5 - log2 V) in its return value.
constexpr int ilog2(int v) { return v <= 1 ? 0 : 1 + ilog2(v / 2); }
template <int V, typename T>
__device__ __forceinline__ T lane_totals(T (&v)[V]) {
  static_assert((V & (V - 1)) == 0 && V <= 32, "power of two");
  const int lane = threadIdx.x & 31;
  int mask = 16;
#pragma unroll
  for (int h = V / 2; h >= 1; h /= 2) {
    const bool up = lane & mask;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const T keep = up ? v[i + h] : v[i], send = up ? v[i] : v[i + h];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
    }
    mask >>= 1;
  }
#pragma unroll
  for (int m = 16 >> ilog2(V); m >= 1; m >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], m);
  return v[0];
}

// Sum of 16 values `stride` apart (slots of absent warps and CTAs stay zero):
// independent loads, one round trip to shared memory instead of 16.
template <typename T>
__device__ __forceinline__ T sum16(const T* p, int stride) {
  T v[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = p[k * stride];
#pragma unroll
  for (int k = 1; k < 16; ++k) v[0] += v[k];
  return v[0];
}

// NP consecutive values of a global row (aligned to NP * sizeof(T) or 16 bytes).
template <int NP>
__device__ __forceinline__ void ldg_row(const double* p, double (&x)[NP]) {
  if constexpr (NP == 1) {
    x[0] = __ldcg(p);
  } else {
#pragma unroll
    for (int h = 0; h < NP / 2; ++h) {
      const double2 v = __ldcg(reinterpret_cast<const double2*>(p) + h);
      x[2 * h] = v.x; x[2 * h + 1] = v.y;
    }
  }
}
template <int NP>
__device__ __forceinline__ void stg_row(double* p, const double (&x)[NP]) {
  if constexpr (NP == 1) {
    *p = x[0];
  } else {
#pragma unroll
    for (int h = 0; h < NP / 2; ++h) reinterpret_cast<double2*>(p)[h] = make_double2(x[2 * h], x[2 * h + 1]);
  }
}

// BF16 element e (0..3) of four packed in a uint2.
__device__ __forceinline__ float cl_bf16(const uint2& w, int e) {
  const unsigned word = (e < 2) ? w.x : w.y;
  return __uint_as_float((e & 1) ? (word & 0xffff0000u) : (word << 16));
}

// Coarse product, two-level preconditioner: yc[i] = sum_j R[i][j] rc[j] for
// the CTA's own aggregates; lanes stream four entries of R each, RW rows of a
// warp at a time, rc read from shared memory in the swizzled order it was
// written in (entry j at (j % 4) * ld / 4 + j / 4: lanes read consecutive rows).
template <int NP>
__device__ __forceinline__ void cl_coarse(const uint16_t* kseg, int nc, int nrow, const float* rc, float* yc) {
  constexpr int RW = NP >= 8 ? 1 : NP == 4 ? 2 : 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int ld = (nc + 7) & ~7, l4 = ld >> 2;
  // as few rows per warp as one pass needs; the last warp has the scalars to do
  const int cw = max(nwarp - 1, 1);
  const int rw = min(RW, (nrow + cw - 1) / cw);
  for (int r0 = warp * rw; warp < cw && r0 < nrow; r0 += cw * rw) {
    const int nr = min(rw, nrow - r0);
    float acc[RW * NP];
#pragma unroll
    for (int v = 0; v < RW * NP; ++v) acc[v] = 0.f;
    const uint2* kq = reinterpret_cast<const uint2*>(kseg + (int64_t)r0 * ld);
#pragma unroll 2
    for (int j4 = lane; j4 < l4; j4 += 32) {
      uint2 w[RW];
#pragma unroll
      for (int r = 0; r < RW; ++r) w[r] = r < nr ? kq[r * l4 + j4] : make_uint2(0u, 0u);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float x[NP];
        const int pos = e * l4 + j4;
        if constexpr (NP == 1) {
          x[0] = rc[pos];
        } else if constexpr (NP == 2) {
          const float2 v = reinterpret_cast<const float2*>(rc)[pos];
          x[0] = v.x; x[1] = v.y;
        } else {
#pragma unroll
          for (int h = 0; h < NP / 4; ++h) {
            const float4 v = reinterpret_cast<const float4*>(rc)[pos * (NP / 4) + h];
            x[4 * h] = v.x; x[4 * h + 1] = v.y; x[4 * h + 2] = v.z; x[4 * h + 3] = v.w;
          }
        }
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          const float kv = cl_bf16(w[r], e);
#pragma unroll
          for (int q = 0; q < NP; ++q) acc[r * NP + q] = fmaf(kv, x[q], acc[r * NP + q]);
        }
      }
    }
    constexpr int V = RW * NP;
    const float tot = lane_totals<V>(acc);
    constexpr int per = 32 / V;
    const int idx = lane / per;  // row idx / NP, column idx % NP
    if (lane % per == 0 && idx / NP < nr) yc[(r0 + idx / NP) * NP + idx % NP] = tot;
  }
}

template <int N>
struct Count {
  static constexpr int value = N;
};

// One cluster solves one segment's columns [col0, col0 + NP).  UPW: most
// 32-row units a warp holds.  A CTA keeps its rows in slots of 32 per unit
// (lanes past a unit's last row hold zero residuals and matrix entries, so the
// iteration needs no masks), followed by the halo: copies of the neighbouring
// rows of other CTAs, whose z their owners store after every preconditioning.
template <int NP, int UPW, bool TL>
__global__ void __launch_bounds__(32 * kClMaxWarps, 1) ir_cluster_kernel(const ClArgs a, int cta_base) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ float s_vrc[NP];
  __shared__ double s_rtol;
  __shared__ int s_own[16];  // rows of every CTA's own slots
  __shared__ int s_act, s_rdone, s_mask;
  const ClusterCta c = a.cta[cta_base + blockIdx.x];
  const unsigned rank = cl_rank(), cs = cl_size();
  const int lcs = 31 - __clz((int)cs);  // (a power of two)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int nrow = c.row1 - c.row0, nunit = c.unit1 - c.unit0;
  const int nagg = TL ? c.agg1 - c.agg0 : 0;
  const bool boss = warp == nwarp - 1;  // the warp that keeps the columns' scalars
  const int u0 = nunit * warp / nwarp, nu = nunit * (warp + 1) / nwarp - u0;
  const int slot0 = 32 * u0 + lane;  // slot of unit i of this warp: slot0 + 32 i
  float* Z = reinterpret_cast<float*>(sm + a.o_z);  // halo rows only
  float* P = reinterpret_cast<float*>(sm + a.o_p);
  float* rc = reinterpret_cast<float*>(sm + a.o_rc);
  float* yc = reinterpret_cast<float*>(sm + a.o_yc);
  float* up = reinterpret_cast<float*>(sm + a.o_up);
  // per-warp partial sums and, from every CTA, their sums over its warps: an
  // area for each of the three reductions (restriction, r'z, p'q), written again
  // only after another barrier (the first: doubles in the residual stage)
  float* wp = reinterpret_cast<float*>(sm + a.o_wp);
  float* wp2 = wp + 16 * 2 * NP;
  float* wp3 = wp2 + 16 * 2 * NP;
  float* mail = reinterpret_cast<float*>(sm + a.o_mail);
  float* mail2 = mail + 16 * 2 * NP;
  float* mail3 = mail2 + 16 * 2 * NP;
  double* mail64 = reinterpret_cast<double*>(mail3 + 16 * NP);
  int32_t* ubase = reinterpret_cast<int32_t*>(sm + a.o_tab);   // slice start of every unit, relative
  int32_t* urow = ubase + nunit + 1;                           // first row, relative
  int32_t* uagg = urow + nunit + 1;                            // aggregate, relative to the CTA (0: none, with kv = 0)
  float* ukv = reinterpret_cast<float*>(uagg + nunit);         // its entry of the dominant coarse vector
  int32_t* upush = reinterpret_cast<int32_t*>(ukv + nunit);    // first push entry of every unit, relative
  int32_t* aunit = upush + nunit + 1;                          // first unit of every aggregate, relative, and number << 16
  unsigned* push = reinterpret_cast<unsigned*>(sm + a.o_push); // halo rows other CTAs hold copies of
  const int zplane = a.zrows * 4, pplane = a.prows * 4;        // NP = 8: floats per plane of four columns
  int segbase = 0, nc = 0, ld = 0;
  float cscale = 0.f;
  const uint16_t* kseg = nullptr;
  if constexpr (TL) {
    segbase = a.seg_agg[c.seg];
    nc = a.seg_agg[c.seg + 1] - segbase;
    ld = (nc + 7) & ~7;
    cscale = nc > 0 ? a.kscale[c.seg] : 0.f;  // (a segment without aggregates has no coarse space)
    kseg = a.kinv + a.kinv_off[c.seg] + (int64_t)(c.agg0 - segbase) * ld;  // this CTA's rows of the coarse inverse
  }

  // ---- set-up: tables, matrix, zeroed arrays
  const int32_t e0 = a.slice_ptr[c.unit0], e1 = a.slice_ptr[c.unit1];
  const int32_t h0 = a.push_ptr[c.unit0], h1 = a.push_ptr[c.unit1];
  for (int u = threadIdx.x; u <= nunit; u += blockDim.x) {
    ubase[u] = a.slice_ptr[c.unit0 + u] - e0;
    urow[u] = a.unit_row[c.unit0 + u] - c.row0;
    upush[u] = a.push_ptr[c.unit0 + u] - h0;
    if (u < nunit) {
      const int g = TL ? a.unit_agg[c.unit0 + u] : -1;
      uagg[u] = g >= 0 ? g - c.agg0 : 0;
      ukv[u] = (TL && g >= 0) ? a.kvec[g] : 0.f;
    }
  }
  if constexpr (TL)
    for (int g = threadIdx.x; g < nagg; g += blockDim.x) {
      const int ua = a.agg_unit[2 * (c.agg0 + g)], ub = a.agg_unit[2 * (c.agg0 + g) + 1];
      aunit[g] = (ua - c.unit0) | ((ub - ua) << 16);
    }
  for (int i = threadIdx.x; i < h1 - h0; i += blockDim.x) push[i] = a.push[h0 + i];
  if (threadIdx.x < cs) {
    const ClusterCta* o = a.cta + cta_base + blockIdx.x - rank + threadIdx.x;
    s_own[threadIdx.x] = 32 * (o->unit1 - o->unit0);
  }
  for (int i = threadIdx.x; i < 16 * 5 * NP; i += blockDim.x) wp[i] = 0.f;    // all three areas
  for (int i = threadIdx.x; i < 16 * 7 * NP; i += blockDim.x) mail[i] = 0.f;  // all four areas
  const float* val = a.val + e0;
  const uint16_t* code = a.code + e0;
  if (a.mat_smem) {
    float4* dv = reinterpret_cast<float4*>(sm + a.o_val);
    uint4* dc = reinterpret_cast<uint4*>(sm + a.o_code);
    for (int i = threadIdx.x; i < (e1 - e0) / 4; i += blockDim.x) dv[i] = __ldg(reinterpret_cast<const float4*>(val) + i);
    for (int i = threadIdx.x; i < (e1 - e0) / 8; i += blockDim.x) dc[i] = __ldg(reinterpret_cast<const uint4*>(code) + i);
    val = reinterpret_cast<const float*>(dv);
    code = reinterpret_cast<const uint16_t*>(dc);
  }
  if constexpr (TL) {
    if (a.coarse_smem) {
      uint4* dk = reinterpret_cast<uint4*>(sm + a.o_coarse);
      for (int i = threadIdx.x; i < nagg * (ld >> 3); i += blockDim.x) dk[i] = __ldg(reinterpret_cast<const uint4*>(kseg) + i);
    }
    for (int i = threadIdx.x; i < ld * NP; i += blockDim.x) rc[i] = 0.f;
    for (int i = threadIdx.x; i < nunit * NP; i += blockDim.x) up[i] = 0.f;
    for (int i = threadIdx.x; i < max(nagg, 1) * NP; i += blockDim.x) yc[i] = 0.f;
  }
  __syncthreads();

  // residual, solution, and the direction where its registers are few (geodesics
  // of 40,962 vertices 9.2 -> 8.5 ms; with 12 a lane the matrix product has fewer
  // loads in flight: 128 spectra 531 -> 557 ms)
  constexpr bool kDirRegs = UPW * NP <= 8;
  float R[UPW][NP], X[UPW][NP], D[kDirRegs ? UPW : 1][NP], dv[UPW], dg[UPW];
  // the direction in unit i of this warp
  auto direction = [&](int i, float (&x)[NP]) {
    if constexpr (kDirRegs) {
#pragma unroll
      for (int q = 0; q < NP; ++q) x[q] = D[i][q];
    } else {
      cl_load<NP>(P, pplane, slot0 + 32 * i, x);
    }
  };
  // global row of unit i of this warp and lane, or -1 past the unit's last row
  auto row_of = [&](int i) -> int64_t {
    if (i >= nu) return -1;
    const int r0 = urow[u0 + i];
    return lane < urow[u0 + i + 1] - r0 ? (int64_t)c.row0 + r0 + lane : -1;
  };
  // NV per-warp values of `part` summed over the CTA's warps and stored in every
  // CTA's area `area`; the caller passes a cluster barrier before it sums them
  // with total() (one CTA: total() reads `part` itself)
  auto exchange = [&](const float* part, float* area, int nv) {
    __syncthreads();
    if (cs == 1) return;
    // (destination-major: the lanes of a store go to one CTA)
    for (int e = threadIdx.x; e < nv * (int)cs; e += blockDim.x) {
      const int dst = e / nv, v = e % nv;
      const float s = sum16(part + v, nv);
      if (dst == (int)rank) area[rank * nv + v] = s;
      else cl_store(cl_map(smem_u32(area + rank * nv + v), dst), s);
    }
  };
  // this warp's rows into the neighbours' copies of them: rows of `arr` there,
  // behind its own slots (own = 1) or by themselves (0)
  auto push_rows = [&](const float (&v)[UPW][NP], float* arr, int plane, int own) {
#pragma unroll
    for (int i = 0; i < UPW; ++i) {
      if (i < nu) {
        const int e1 = upush[u0 + i + 1];
        for (int e0 = upush[u0 + i]; e0 < e1; e0 += 32) {
          const unsigned w = push[min(e0 + lane, e1 - 1)];  // slot (12 bits), rank (4), halo row (16)
          const unsigned rk = (w >> 12) & 15u, dst = (w >> 16) + (unsigned)(own * s_own[rk]);
          float x[NP];
#pragma unroll
          for (int q = 0; q < NP; ++q) x[q] = __shfl_sync(0xffffffffu, v[i][q], (int)(w & 31u));
          if (e0 + lane < e1) {
            const unsigned ra = cl_map(smem_u32(arr), rk);
            if constexpr (NP >= 4) {
#pragma unroll
              for (int h = 0; h < NP / 4; ++h)
                cl_store4(ra + 4u * (unsigned)(h * plane) + 16u * dst, x[4 * h], x[4 * h + 1], x[4 * h + 2],
                          x[4 * h + 3]);
            } else if constexpr (NP == 2) {
              cl_store2(ra + 8u * dst, x[0], x[1]);
            } else {
              cl_store(ra + 4u * dst, x[0]);
            }
          }
        }
      }
    }
  };
  // value lane mod nv of the totals; nv = 1, 2, 4, 8 or 16, in every warp: all
  // lanes read (16 reads by nv lanes of each warp took 512 of an iteration's
  // shared-memory wavefronts)
  auto total = [&](const float* part, const float* area, auto nvc) -> float {
    constexpr int nv = decltype(nvc)::value;
    const float* src = (cs == 1 ? part : area) + lane;
    float v = 0.f;
#pragma unroll
    for (int j = 0; j < 16 * nv; j += 32)
      if (16 * nv >= 32 || lane < 16 * nv) v += src[j];
#pragma unroll
    for (int m = 16; m >= nv; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
    return v;
  };
  // column sums over the cluster in FP64, on lanes 0..NP-1 of the boss warp
  auto reduce64 = [&](double (&acc)[NP]) -> double {
    double* wd = reinterpret_cast<double*>(wp);
    const double t = lane_totals<NP>(acc);
    constexpr int per = 32 / NP;
    if (warp == 0)  // slots of absent warps
      for (int e = lane; e < 16 * NP; e += 32)
        if (e / NP >= nwarp) wd[e] = 0.0;
    if (lane % per == 0) wd[warp * NP + lane / per] = t;
    __syncthreads();
    for (int e = threadIdx.x; e < (int)cs * NP; e += blockDim.x) {
      const int dst = e / NP, q = e % NP;
      const double s = sum16(wd + q, NP);
      if (dst == (int)rank) mail64[rank * NP + q] = s;
      else cl_store(cl_map(smem_u32(mail64 + rank * NP + q), dst), s);
    }
    cl_sync(cs);
    const double s = (boss && lane < NP) ? sum16(mail64 + lane, NP) : 0.0;
    for (int e = threadIdx.x; e < 16 * 2 * NP; e += blockDim.x) wp[e] = 0.f;  // read above before the barrier
    return s;
  };

  // ---- R = B, ||B||^2
  double hb = 0.0, hr = 0.0;  // of column `lane` (boss warp)
  {
    double acc[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) acc[q] = 0.0;
#pragma unroll
    for (int i = 0; i < UPW; ++i) {
#pragma unroll
      for (int q = 0; q < NP; ++q) R[i][q] = 0.f;
      dv[i] = 0.f;
      dg[i] = i < nu ? a.diag[32 * (int64_t)(c.unit0 + u0 + i) + lane] : 0.f;
      const int64_t row = row_of(i);
      if (row >= 0) {
        double b[NP];
        ldg_row<NP>(a.B + row * a.p + c.col0, b);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          acc[q] += b[q] * b[q];
          R[i][q] = (float)b[q];
        }
        dv[i] = a.dinv[row];
      }
    }
    if (cs > 1) cl_sync(cs);  // every CTA of the cluster runs before its memory is written
    hb = reduce64(acc);
  }

  // columns that are done, zeroed in R: solved, failed, or never begun (a zero
  // right-hand side is solved by zero; NaN or Inf in it is an error, and its
  // solution is left zero)
  auto clear = [&](int mk) {
#pragma unroll
    for (int i = 0; i < UPW; ++i)
#pragma unroll
      for (int q = 0; q < NP; ++q)
        if ((mk >> q) & 1) R[i][q] = 0.f;
  };
  int fst = isfinite(hb) ? LAPY_OK : LAPY_ERR_NAN;  // column `lane` (boss warp)
  bool masked = !(hb > 0.0) || !isfinite(hb);
  if (boss) {
    const unsigned mk = __ballot_sync(0xffffffffu, lane >= NP || masked);
    if (lane == 0) s_mask = (int)mk;
  }
  __syncthreads();
  clear(s_mask);
  double round_rtol = a.inner_rtol;
  int iters = 0, rounds = 0;
  for (int round = 0; round < a.max_rounds; ++round) {
    ++rounds;
    const float rtol2 = (float)(round_rtol * round_rtol);
    // ---- FP32 PCG from zero on R
#pragma unroll
    for (int i = 0; i < UPW; ++i) {
      float zero[NP];
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        X[i][q] = 0.f;
        zero[q] = 0.f;
        if constexpr (kDirRegs) D[i][q] = 0.f;
      }
      if (!kDirRegs && i < nu) cl_save<NP>(P, pplane, slot0 + 32 * i, zero);
    }
    for (int h = threadIdx.x; h < c.nhalo; h += blockDim.x) {
      float zero[NP];
#pragma unroll
      for (int q = 0; q < NP; ++q) zero[q] = 0.f;
      cl_save<NP>(P, pplane, 32 * nunit + h, zero);
    }
    __syncthreads();
    // of column `lane`: its state and ||r0||^2 (two-level: in the boss warp),
    // and the last r'z (0: none yet), the same in every warp
    int32_t st = kClActive;
    float bb = 0.f, rzold = 0.f;
    int it = 0;
    // convergence of column `lane` from its squared residual
    auto judge = [&](float rr) {
      if (it == 0) {
        bb = rr;
        if (!isfinite(rr)) st = LAPY_ERR_NAN;
        else if (rr == 0.f) st = 0;
      } else if (st == kClActive) {
        if (!isfinite(rr)) st = LAPY_ERR_NAN;
        else if (rr <= rtol2 * bb) st = it;
      }
    };
    for (;; ++it) {
      if constexpr (TL) {
        // ---- ||r||^2, v'W'r and the restriction W'r
        // (the warp's unit sums, ||r||^2 and v'W'r in one halving reduction)
        constexpr int NS = UPW * NP + 2 * NP;
        constexpr int NR = NS <= 4 ? 4 : NS <= 8 ? 8 : NS <= 16 ? 16 : 32;
        static_assert(NS <= 32, "one value per lane");
        float red[NR];
#pragma unroll
        for (int v = UPW * NP; v < NR; ++v) red[v] = 0.f;
#pragma unroll
        for (int i = 0; i < UPW; ++i) {
          const float kv = i < nu ? ukv[u0 + i] : 0.f;
#pragma unroll
          for (int q = 0; q < NP; ++q) {
            red[i * NP + q] = R[i][q];
            red[UPW * NP + q] = fmaf(R[i][q], R[i][q], red[UPW * NP + q]);
            red[UPW * NP + NP + q] = fmaf(kv, R[i][q], red[UPW * NP + NP + q]);
          }
        }
        {
          const float t = lane_totals<NR>(red);
          constexpr int per = 32 / NR;
          const int v = lane / per;
          if (lane % per == 0) {
            if (v < nu * NP) up[u0 * NP + v] = t;
            else if (v >= UPW * NP && v < NS) wp[warp * 2 * NP + v - UPW * NP] = t;
          }
        }
        exchange(wp, mail, 2 * NP);
        if (nc > 0) {
          // (a warp per destination CTA; one CTA: all warps share it)
          const int step = 32 * (nwarp >> lcs > 0 ? nwarp >> lcs : 1);
          for (int dst = warp & ((int)cs - 1); dst < (int)cs; dst += nwarp)
            for (int g = 32 * (warp >> lcs) + lane; g < nagg; g += step) {
              const int ua = aunit[g] & 0xffff, na = aunit[g] >> 16;
              float s[NP];
#pragma unroll
              for (int q = 0; q < NP; ++q) s[q] = up[ua * NP + q];
              for (int u = 1; u < na; ++u)
#pragma unroll
                for (int q = 0; q < NP; ++q) s[q] += up[(ua + u) * NP + q];
              const int j = c.agg0 + g - segbase;
              float* at = rc + ((j & 3) * (ld >> 2) + (j >> 2)) * NP;
              if (dst == (int)rank) {
#pragma unroll
                for (int q = 0; q < NP; ++q) at[q] = s[q];
                continue;
              }
              const unsigned ra = cl_map(smem_u32(at), dst);
              if constexpr (NP >= 4) {
#pragma unroll
                for (int h = 0; h < NP / 4; ++h)
                  cl_store4(ra + 16u * h, s[4 * h], s[4 * h + 1], s[4 * h + 2], s[4 * h + 3]);
              } else if constexpr (NP == 2) {
                cl_store2(ra, s[0], s[1]);
              } else {
                cl_store(ra, s[0]);
              }
            }
        }
        cl_sync(cs);
        if (boss) {
          const float s = total(wp, mail, Count<2 * NP>());
          if (lane >= NP && lane < 2 * NP) s_vrc[lane - NP] = cscale * s;
          if (lane < NP) judge(s);
          const unsigned m = __ballot_sync(0xffffffffu, lane < NP && st == kClActive);
          if (lane == 0) s_act = it < a.maxiter ? (int)m : 0;
        }
        if (nc > 0) {  // (two calls, so that the compiler knows the address space)
          if (a.coarse_smem) cl_coarse<NP>(reinterpret_cast<const uint16_t*>(sm + a.o_coarse), nc, nagg, rc, yc);
          else cl_coarse<NP>(kseg, nc, nagg, rc, yc);
        }
        __syncthreads();
        if (s_act == 0) break;
      }
      // ---- z = D^-1 r (+ the coarse correction), r'z (and ||r||^2 for Jacobi)
      constexpr int NV = TL ? NP : 2 * NP;  // partial sums per warp
      float z[UPW][NP];
      {
        float red[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) red[v] = 0.f;
#pragma unroll
        for (int i = 0; i < UPW; ++i) {
          if (i < nu) {
#pragma unroll
            for (int q = 0; q < NP; ++q) z[i][q] = dv[i] * R[i][q];
            if constexpr (TL) {
              const float* y = yc + uagg[u0 + i] * NP;
              const float kv = ukv[u0 + i];
#pragma unroll
              for (int q = 0; q < NP; ++q) z[i][q] += y[q] + kv * s_vrc[q];
            }
#pragma unroll
            for (int q = 0; q < NP; ++q) {
              red[q] = fmaf(R[i][q], z[i][q], red[q]);
              if constexpr (!TL) red[NP + q] = fmaf(R[i][q], R[i][q], red[NP + q]);
            }
          }
        }
        constexpr int per = 32 / NV;
        const float t = lane_totals<NV>(red);
        if (lane % per == 0) wp2[warp * NV + lane / per] = t;
      }
      if (a.z_halo) push_rows(z, Z, zplane, 0);
      exchange(wp2, mail2, NV);
      if (cs > 1) cl_sync(cs);
      // ---- beta, p = z + beta p in the CTA's rows and its copies (scalars of
      // column `lane` in every warp)
      float gam = total(wp2, mail2, Count<NV>());
      bool act;
      if constexpr (TL) {
        act = (s_act >> lane) & 1;
      } else {
        const float rr = __shfl_sync(0xffffffffu, gam, (lane + NP) & 31);
        if (lane < NP) judge(rr);
        act = lane < NP && st == kClActive && it < a.maxiter;
        if (!__any_sync(0xffffffffu, act)) break;
      }
      if (act && !(gam > 0.f && isfinite(gam))) {
        st = isfinite(gam) ? LAPY_ERR_BREAKDOWN : LAPY_ERR_NAN;
        act = false;
      }
      {
        const float b = act && rzold > 0.f ? gam / rzold : 0.f;
        rzold = gam;
        float be[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) be[q] = __shfl_sync(0xffffffffu, b, q);
#pragma unroll
        for (int i = 0; i < UPW; ++i) {
          if (i < nu) {
            float pv[NP];
            direction(i, pv);
#pragma unroll
            for (int q = 0; q < NP; ++q) {
              z[i][q] = fmaf(be[q], pv[q], z[i][q]);
              if constexpr (kDirRegs) D[i][q] = z[i][q];
            }
            cl_save<NP>(P, pplane, slot0 + 32 * i, z[i]);
          }
        }
        if (a.z_halo) {
          for (int h = threadIdx.x; h < c.nhalo; h += blockDim.x) {
            float zv[NP], pv[NP];
            cl_load<NP>(Z, zplane, h, zv);
            cl_load<NP>(P, pplane, 32 * nunit + h, pv);
#pragma unroll
            for (int q = 0; q < NP; ++q) pv[q] = fmaf(be[q], pv[q], zv[q]);
            cl_save<NP>(P, pplane, 32 * nunit + h, pv);
          }
          __syncthreads();
        } else {
          if (cs > 1) push_rows(z, P, pplane, 1);
          cl_sync(cs);
        }
      }
      // ---- q = K p, p'q
      float Q[UPW][NP];
      {
        float red[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) red[q] = 0.f;
#pragma unroll
        for (int i = 0; i < UPW; ++i) {
#pragma unroll
          for (int q = 0; q < NP; ++q) Q[i][q] = 0.f;
          if (i < nu) {
            const int b0 = ubase[u0 + i], b1 = ubase[u0 + i + 1];
            const float2* vp = reinterpret_cast<const float2*>(val + b0) + lane;
            const uint32_t* cp = reinterpret_cast<const uint32_t*>(code + b0) + lane;
            // pairs of entries of the lane's row, two pairs at a time
            int k = (b1 - b0) >> 6;
#pragma unroll 1
            for (; k >= 2; k -= 2, vp += 64, cp += 64) {
              const uint32_t ca = cp[0], cb = cp[32];
              const float2 va = vp[0], vb = vp[32];
              float x0[NP], x1[NP], x2[NP], x3[NP];
              cl_load<NP>(P, pplane, ca & 0xffff, x0);
              cl_load<NP>(P, pplane, ca >> 16, x1);
              cl_load<NP>(P, pplane, cb & 0xffff, x2);
              cl_load<NP>(P, pplane, cb >> 16, x3);
#pragma unroll
              for (int q = 0; q < NP; ++q) {
                Q[i][q] = fmaf(va.x, x0[q], Q[i][q]);
                Q[i][q] = fmaf(va.y, x1[q], Q[i][q]);
                Q[i][q] = fmaf(vb.x, x2[q], Q[i][q]);
                Q[i][q] = fmaf(vb.y, x3[q], Q[i][q]);
              }
            }
            if (k) {
              const uint32_t ca = cp[0];
              const float2 va = vp[0];
              float x0[NP], x1[NP];
              cl_load<NP>(P, pplane, ca & 0xffff, x0);
              cl_load<NP>(P, pplane, ca >> 16, x1);
#pragma unroll
              for (int q = 0; q < NP; ++q) {
                Q[i][q] = fmaf(va.x, x0[q], Q[i][q]);
                Q[i][q] = fmaf(va.y, x1[q], Q[i][q]);
              }
            }
            float pv[NP];
            direction(i, pv);
#pragma unroll
            for (int q = 0; q < NP; ++q) {
              Q[i][q] = fmaf(dg[i], pv[q], Q[i][q]);
              red[q] = fmaf(pv[q], Q[i][q], red[q]);
            }
          }
        }
        constexpr int per = 32 / NP;
        const float t = lane_totals<NP>(red);
        if (lane % per == 0) wp3[warp * NP + lane / per] = t;
      }
      exchange(wp3, mail3, NP);
      if (cs > 1) cl_sync(cs);
      // ---- x += alpha p, r -= alpha q
      {
        const float pq = total(wp3, mail3, Count<NP>());
        float alpha = 0.f;
        if (act) {
          if (!(pq > 0.f) || !isfinite(pq)) {
            st = LAPY_ERR_BREAKDOWN;
          } else {
            alpha = gam / pq;
            if (!isfinite(alpha)) {
              alpha = 0.f;
              st = LAPY_ERR_NAN;
            }
          }
        }
        float al[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) al[q] = __shfl_sync(0xffffffffu, alpha, q);
#pragma unroll
        for (int i = 0; i < UPW; ++i) {
          if (i < nu) {
            float pv[NP];
            direction(i, pv);
#pragma unroll
            for (int q = 0; q < NP; ++q) {
              X[i][q] = fmaf(al[q], pv[q], X[i][q]);
              R[i][q] = fmaf(-al[q], Q[i][q], R[i][q]);
            }
          }
        }
      }
    }
    iters += it;

    // ---- X64 += x, R = B - K X64 in FP64
#pragma unroll
    for (int i = 0; i < UPW; ++i) {
      const int64_t row = row_of(i);
      if (row >= 0) {
        double* xp = a.X + row * a.p + c.col0;
        double x[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) x[q] = 0.0;
        if (round > 0) ldg_row<NP>(xp, x);
#pragma unroll
        for (int q = 0; q < NP; ++q) x[q] += (double)X[i][q];
        stg_row<NP>(xp, x);
      }
    }
    cl_sync(cs);
    {
      double acc[NP];
#pragma unroll
      for (int q = 0; q < NP; ++q) acc[q] = 0.0;
#pragma unroll
      for (int i = 0; i < UPW; ++i) {
        const int64_t row = row_of(i);
        if (row >= 0) {
          double y[NP], b[NP];
#pragma unroll
          for (int q = 0; q < NP; ++q) y[q] = 0.0;
          const int32_t kb = a.indptr[row], ke = a.indptr[row + 1];
#pragma unroll 2
          for (int32_t k = kb; k < ke; ++k) {
            double x[NP];
            const double v = __ldg(a.k64 + k);
            ldg_row<NP>(a.X + (int64_t)__ldg(a.indices + k) * a.p + c.col0, x);
#pragma unroll
            for (int q = 0; q < NP; ++q) y[q] = fma(v, x[q], y[q]);
          }
          ldg_row<NP>(a.B + row * a.p + c.col0, b);
#pragma unroll
          for (int q = 0; q < NP; ++q) {
            const double r = b[q] - y[q];
            acc[q] += r * r;
            R[i][q] = (float)r;
          }
        }
      }
      hr = reduce64(acc);
    }
    if (boss) {
      if (lane < NP && !masked) {
        if (st == LAPY_ERR_NAN || st == LAPY_ERR_BREAKDOWN || !isfinite(hr)) {
          fst = (st < 0) ? st : LAPY_ERR_NAN;
          masked = true;
        } else if (hr <= a.rtol * a.rtol * hb) {
          masked = true;
        }
      }
      // largest reduction still missing over the active columns (factor 4 margin)
      double need = 1.0;
      if (lane < NP && !masked && hr > 0.0) need = fmin(1.0, 0.25 * a.rtol * sqrt(hb / hr));
      for (int o = 16; o > 0; o >>= 1) need = fmin(need, __shfl_xor_sync(0xffffffffu, need, o));
      const unsigned mk = __ballot_sync(0xffffffffu, lane >= NP || masked);
      if (lane == 0) {
        s_rtol = fmax(a.inner_rtol, fmin(0.5, need));
        s_mask = (int)mk;
        s_rdone = mk == 0xffffffffu;
      }
    }
    __syncthreads();
    round_rtol = s_rtol;
    if (s_rdone) break;
    clear(s_mask);
  }
  if (rank == 0 && boss) {
    if (lane < NP) {
      const int64_t o = (int64_t)c.seg * a.p + c.col0 + lane;
      if (fst == LAPY_OK && hb > 0.0 && !(hr <= a.rtol * a.rtol * hb)) fst = LAPY_ERR_NOCONV;
      a.state[o] = fst;
      a.relres2[o] = !isfinite(hb) ? nan("") : hb > 0.0 ? hr / hb : 0.0;
    }
    if (lane == 0) {
      atomicMax(a.ctl + 0, (unsigned long long)iters);
      atomicMax(a.ctl + 1, (unsigned long long)rounds);
    }
  }
  if (threadIdx.x == 0) {  // rows, entries and coarse bytes the iterations went over
    atomicAdd(a.ctl + 2, (unsigned long long)iters * (unsigned long long)nrow);
    atomicAdd(a.ctl + 3, (unsigned long long)iters * (unsigned long long)(a.indptr[c.row1] - a.indptr[c.row0]));
    if (TL) atomicAdd(a.ctl + 4, 2ull * (unsigned long long)iters * (unsigned long long)nagg * (unsigned long long)ld);
  }
  if (cs > 1) cl_sync(cs);  // no CTA leaves while another may still write its memory
}

// ---- packed matrix -------------------------------------------------------------
// The diagonal is kept apart (one value per slot).  Slices hold the other
// entries of 32 rows, two of a row side by side: per pair 32 x 2 values and
// 32 x 2 codes, rows padded to an even number (regular triangle meshes have 6:
// no padding); a code is the slot of the column's row in the CTA that owns the
// slice: its own row or a halo copy.
__global__ void cl_width_kernel(int nunit, const int32_t* __restrict__ unit_row, const int32_t* __restrict__ unit_cta,
                                const int32_t* __restrict__ cta_unit0, const int32_t* __restrict__ indptr,
                                const int32_t* __restrict__ indices, int32_t* __restrict__ elems, int32_t* __restrict__ row_slot) {
  const int u = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (u >= nunit) return;
  const int r = unit_row[u] + lane;
  const bool valid = r < unit_row[u + 1];
  int len = 0, diag = 0;
  if (valid)
    for (int k = indptr[r]; k < indptr[r + 1]; ++k) {
      ++len;
      diag |= indices[k] == r;
    }
  const int w = warp_max(len - diag);
  if (lane == 0) elems[u] = 32 * ((w + 1) & ~1);
  const int k = unit_cta[u];
  if (valid) row_slot[r] = (k << 12) | (32 * (u - cta_unit0[k]) + lane);
}

// One block per CTA of the split: the rows of other CTAs its rows refer to
// (a bitmap over the segment's rows, and the rank of every word's first bit),
// counted per unit of the owner.  A column outside the segment sets *bad.
struct ClSplitCta {
  int32_t row0, row1, seg0, seg1, first;  // rows, the segment's rows, the segment's first split CTA
  int64_t word0;                          // first bitmap word
};
__global__ void cl_halo_kernel(const ClSplitCta* __restrict__ split, const int32_t* __restrict__ indptr,
                               const int32_t* __restrict__ indices, const int32_t* __restrict__ row_slot,
                               const int32_t* __restrict__ cta_unit0, uint32_t* __restrict__ bits,
                               int32_t* __restrict__ rank, int32_t* __restrict__ halo, int32_t* __restrict__ push_cnt,
                               int* __restrict__ bad) {
  __shared__ uint32_t map[kClMaxRows * 16 / 32];
  __shared__ int32_t sums[32];
  const ClSplitCta c = split[blockIdx.x];
  const int nw = (c.seg1 - c.seg0 + 31) >> 5;
  for (int i = threadIdx.x; i < nw; i += blockDim.x) map[i] = 0u;
  __syncthreads();
  const int k0 = indptr[c.row0], k1 = indptr[c.row1];
  for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
    const int col = indices[k];
    if (col < c.seg0 || col >= c.seg1) *bad = 1;
    else if (col < c.row0 || col >= c.row1) atomicOr(&map[(col - c.seg0) >> 5], 1u << ((col - c.seg0) & 31));
  }
  __syncthreads();
  // exclusive ranks of the words: one thread sums a stretch, then the stretches
  const int per = (nw + blockDim.x - 1) / blockDim.x;
  const int a = min(nw, (int)threadIdx.x * per), b = min(nw, a + per);
  int mine = 0;
  for (int i = a; i < b; ++i) mine += __popc(map[i]);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane == 31) sums[warp] = inc;
  __syncthreads();
  int before = inc - mine;
  for (int w = 0; w < warp; ++w) before += sums[w];
  for (int i = a; i < b; ++i) {
    bits[c.word0 + i] = map[i];
    rank[c.word0 + i] = before;
    before += __popc(map[i]);
    for (uint32_t m = map[i]; m; m &= m - 1) {
      const int rs = row_slot[c.seg0 + 32 * i + __ffs(m) - 1];
      atomicAdd(&push_cnt[cta_unit0[rs >> 12] + ((rs & 4095) >> 5)], 1);
    }
  }
  if (threadIdx.x == blockDim.x - 1) halo[blockIdx.x] = before;
}

// Push lists of the owners (the order within a unit's list does not matter).
__global__ void cl_push_kernel(const ClSplitCta* __restrict__ split, const int32_t* __restrict__ row_slot,
                               const int32_t* __restrict__ cta_unit0, const uint32_t* __restrict__ bits, const int32_t* __restrict__ rank,
                               const int32_t* __restrict__ push_ptr, int32_t* __restrict__ push_fill,
                               uint32_t* __restrict__ push) {
  const ClSplitCta c = split[blockIdx.x];
  const int nw = (c.seg1 - c.seg0 + 31) >> 5;
  const uint32_t me = (uint32_t)(blockIdx.x - c.first);
  for (int i = threadIdx.x; i < nw; i += blockDim.x) {
    int at = rank[c.word0 + i];
    for (uint32_t m = bits[c.word0 + i]; m; m &= m - 1, ++at) {
      const int rs = row_slot[c.seg0 + 32 * i + __ffs(m) - 1];
      const int u = cta_unit0[rs >> 12] + ((rs & 4095) >> 5);
      push[push_ptr[u] + atomicAdd(&push_fill[u], 1)] = (uint32_t)(rs & 4095) | (me << 12) | ((uint32_t)at << 16);
    }
  }
}

__global__ void cl_fill_kernel(int nunit, const int32_t* __restrict__ unit_row, const int32_t* __restrict__ unit_cta,
                               const int32_t* __restrict__ cta_unit0, const int32_t* __restrict__ cta_units,
                               const ClSplitCta* __restrict__ split, const int32_t* __restrict__ row_slot,
                               const uint32_t* __restrict__ bits, const int32_t* __restrict__ rank,
                               const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                               const float* __restrict__ vals, const int32_t* __restrict__ slice_ptr,
                               uint16_t* __restrict__ code, float* __restrict__ val,
                               float* __restrict__ diag) {
  const int u = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (u >= nunit) return;
  const int k = unit_cta[u];
  const ClSplitCta c = split[k];
  const int own = 32 * cta_units[k];
  const int r = unit_row[u] + lane;
  const bool valid = r < unit_row[u + 1];
  const int32_t kb = valid ? indptr[r] : 0, len = valid ? indptr[r + 1] - kb : 0;
  const int32_t base = slice_ptr[u];
  const int w = (slice_ptr[u + 1] - base) >> 5;
  const uint16_t self = (uint16_t)(32 * (u - cta_unit0[k]) + lane);
  float dg = 0.f;
  bool have = false;  // the first diagonal entry is the diagonal
  int32_t k0 = kb;
  for (int e = 0; e < w; ++e) {
    uint16_t cd = self;
    float v = 0.f;
    if (!have && k0 < kb + len && indices[k0] == r) {
      dg = vals[k0++];
      have = true;
    }
    if (k0 < kb + len) {
      const int col = indices[k0];
      if (col >= c.row0 && col < c.row1) {
        cd = (uint16_t)(row_slot[col] & 4095);
        v = vals[k0];
      } else if (col >= c.seg0 && col < c.seg1) {
        const int i = col - c.seg0;
        cd = (uint16_t)(own + rank[c.word0 + (i >> 5)] + __popc(bits[c.word0 + (i >> 5)] & ((1u << (i & 31)) - 1u)));
        v = vals[k0];
      }
      ++k0;
    }
    const int64_t o = base + 64 * (e >> 1) + 2 * lane + (e & 1);
    code[o] = cd;
    val[o] = v;
  }
  if (!have && k0 < kb + len) dg = vals[k0];  // the diagonal is the row's last entry
  diag[32 * (int64_t)u + lane] = dg;
}

// ---- kernel variants -------------------------------------------------------------
using ClKernel = void (*)(const ClArgs, int);

// Units a warp holds, by columns: four NP-wide register rows per unit (r, x, z or
// q, and p where they are few), 36 registers at most, so that 16 warps fit
// without spilling.
struct ClVariant {
  int np, upw;
  ClKernel tl, jacobi;
};
#define CL_VARIANT(NP, U) {NP, U, ir_cluster_kernel<NP, U, true>, ir_cluster_kernel<NP, U, false>}
static const ClVariant kVariants[] = {
    CL_VARIANT(1, 2), CL_VARIANT(1, 4), CL_VARIANT(1, 8), CL_VARIANT(2, 2), CL_VARIANT(2, 4), CL_VARIANT(2, 6),
    CL_VARIANT(4, 1), CL_VARIANT(4, 2), CL_VARIANT(4, 3), CL_VARIANT(8, 1),
};
// The first variant that holds `units` units of a CTA.
static const ClVariant* variant(int np, int units) {
  for (const ClVariant& v : kVariants)
    if (v.np == np && units <= kClMaxWarps * v.upw) return &v;
  return nullptr;
}
static int max_units(int np) {
  int m = 0;
  for (const ClVariant& v : kVariants)
    if (v.np == np) m = std::max(m, kClMaxWarps * v.upw);
  return m;
}

// Shared memory of a class; the byte offsets when `a` is given.
static size_t class_layout(const ClusterClass& k, int np, bool tl, bool mat, bool coarse, bool z_halo, ClArgs* a) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += (bytes + 15) & ~size_t(15);
    return (int)o;
  };
  const size_t row = 4 * (size_t)np;
  const int zrows = z_halo ? k.halo : 0, prows = k.slots;
  const int oz = take(row * zrows), op = take(row * prows);
  const int orc = take(tl ? row * k.ld : 0), oyc = take(tl ? row * std::max(k.aggs, 1) : 0);
  const int oup = take(tl ? row * k.units : 0);
  const int owp = take(320 * (size_t)np);               // 16 warps x (2 NP + 2 NP + NP floats; NP doubles)
  const int omail = take(448 * (size_t)np);             // 16 CTAs x (2 NP + 2 NP + NP floats, NP doubles)
  const int otab = take(4 * (5 * (size_t)k.units + 3 + (size_t)(tl ? k.aggs : 0)));
  const int opush = take(4 * (size_t)k.push);
  const int oval = take(mat ? 4 * (size_t)k.elems : 0), ocode = take(mat ? 2 * (size_t)k.elems : 0);
  const int oco = take(tl && coarse ? 2 * (size_t)k.aggs * k.ld : 0);
  if (a) {
    a->o_z = oz; a->o_p = op; a->o_rc = orc; a->o_yc = oyc; a->o_up = oup; a->o_wp = owp; a->o_mail = omail;
    a->o_tab = otab; a->o_push = opush; a->o_val = oval; a->o_code = ocode; a->o_coarse = oco;
    a->zrows = zrows;
    a->prows = prows;
  }
  return off;
}

static void launch_config(const ClusterClass& k, cudaStream_t stream, cudaLaunchConfig_t* cfg,
                          cudaLaunchAttribute* attr) {
  cfg->gridDim = dim3((unsigned)k.ncta);
  cfg->blockDim = dim3((unsigned)(32 * k.warps));
  cfg->dynamicSmemBytes = k.smem;
  cfg->stream = stream;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = (unsigned)k.cs;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 1;
}

ClusterPlan::~ClusterPlan() {
  for (cudaEvent_t e : events) cudaEventDestroy(e);
  for (cudaStream_t t : streams) cudaStreamDestroy(t);
}

// Streams of a plan with several classes: the larger clusters, which need a
// whole GPC's worth of free SMs, ahead of the smaller ones that fill the rest.
static int make_streams(ClusterPlan* plan) {
  const size_t want = plan->cls.size() > 1 ? plan->cls.size() : 0;
  int least = 0, greatest = 0;
  LAPY_CUDA_TRY(cudaDeviceGetStreamPriorityRange(&least, &greatest));
  while (plan->streams.size() < want) {
    const int prio = std::min(least, greatest + (int)plan->streams.size());
    cudaStream_t t = nullptr;
    LAPY_CUDA_TRY(cudaStreamCreateWithPriority(&t, cudaStreamNonBlocking, prio));
    plan->streams.push_back(t);
  }
  while (want > 0 && plan->events.size() < want + 1) {
    cudaEvent_t e = nullptr;
    LAPY_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    plan->events.push_back(e);
  }
  return LAPY_OK;
}

// ---- planning ----------------------------------------------------------------------
int cluster_plan(int64_t n, int64_t nnz, const int32_t* indptr, const int32_t* indices, const float* k32, int nseg,
                 const int32_t* seg_row, const int32_t* seg_agg, const int32_t* agg_rows, int p, void* mem,
                 size_t bytes, ClusterPlan* out, cudaStream_t stream) {
  out->ok = false;
  const bool tl = seg_agg != nullptr;
  const int nagg = tl ? seg_agg[nseg] : 0;
  // units of all segments, in row order (inside aggregates where there are any)
  std::vector<int32_t> unit_row, unit_agg, seg_unit(nseg + 1, 0), agg_unit(2 * (size_t)nagg, 0);
  unit_row.reserve(n / 24 + nseg + 1);
  unit_agg.reserve(n / 24 + nseg + 1);
  for (int s = 0; s < nseg; ++s) {
    seg_unit[s] = (int32_t)unit_row.size();
    if (seg_row[s + 1] - seg_row[s] > 16 * kClMaxRows) return LAPY_OK;
    const bool has = tl && seg_agg[s + 1] > seg_agg[s];
    const int g0 = has ? seg_agg[s] : 0, g1 = has ? seg_agg[s + 1] : 1;
    int32_t next = seg_row[s];  // the units of a segment cover its rows
    for (int g = g0; g < g1; ++g) {
      const int32_t r0 = has ? agg_rows[2 * g] : seg_row[s], r1 = has ? agg_rows[2 * g + 1] : seg_row[s + 1];
      if (r0 != next || r1 < r0) return LAPY_OK;
      next = r1;
      if (has) agg_unit[2 * g] = (int32_t)unit_row.size();
      for (int32_t r = r0; r < r1; r += 32) {
        unit_row.push_back(r);
        unit_agg.push_back(has ? g : -1);
      }
      if (has) agg_unit[2 * g + 1] = (int32_t)unit_row.size();
    }
    if (next != seg_row[s + 1]) return LAPY_OK;
  }
  const int nunit = (int)unit_row.size();
  seg_unit[nseg] = nunit;
  unit_row.push_back((int32_t)n);
  if (nunit == 0) return LAPY_OK;

  // Columns per cluster and units per CTA: the combination with the least
  // modelled time per iteration (microseconds).  A CTA's iteration costs its
  // barriers and reductions plus its units' products: measured with two-level
  // clusters of 1 / 8 / 4 CTAs at 21 / 43 / 86 units of 7 entries a row, one
  // column: 2.4 / 4.5 / 5.7 us, two columns: 2.7 / 5.2 / 6.8 us, and 14
  // entries a row, two columns: 7.5 / 12.5 us at 46 / 92 units (with q by
  // recurrence; 5 to 15 % more since, on all of them).  One mesh is
  // therefore spread over more, narrower clusters until the GPU is full, a
  // batch over as few CTAs as hold it.  Clusters do not cross GPCs: those of
  // 16 CTAs fill 112 of the 152 SMs, of 8 120, of 4 144.
  int best_np = 0, best_u = 0;
  double best = 1e300;
  int largest = 0;
  for (int s = 0; s < nseg; ++s) largest = std::max(largest, seg_unit[s + 1] - seg_unit[s]);
  const double width = (double)nnz / (double)n;
  for (int np = std::min(p, 8); np >= 1; np /= 2) {
    for (int u = max_units(np); u >= 8; u /= 2) {
      if ((int64_t)largest > (int64_t)u * 16) continue;
      double sum = 0.0, worst[5] = {0, 0, 0, 0, 0};
      int64_t count[5] = {0, 0, 0, 0, 0};
      for (int s = 0; s < nseg; ++s) {
        const int us = seg_unit[s + 1] - seg_unit[s];
        int lc = 0;
        while ((u << lc) < us) ++lc;
        const double base = (lc > 0 ? 2.6 + 0.1 * lc : 1.7) * (tl ? 1.0 : 0.75);
        const double t = base + (0.006 + (0.0028 + 0.0017 * np) * width) * (double)us / (1 << lc);
        worst[lc] = std::max(worst[lc], t);
        count[lc] += p / np;
        sum += t * (double)((p / np) << lc);
      }
      static const int fits[5] = {152, 76, 36, 15, 7};  // clusters resident at once
      double t = sum / 145.0;
      for (int lc = 0; lc < 5; ++lc) t = std::max(t, worst[lc] * (double)((count[lc] + fits[lc] - 1) / fits[lc]));
      if (t < best) {
        best = t;
        best_np = np;
        best_u = u;
      }
    }
  }
  if (best_np == 0) return LAPY_OK;
  const int np = best_np, groups = p / np, cap = max_units(np);

  // row split of every segment over its CTAs (at aggregate boundaries)
  std::vector<int32_t> split_cs(nseg), split0(nseg), cta_unit0, cta_units, unit_cta(nunit);
  std::vector<ClSplitCta> split;
  int64_t words = 0;
  for (int s = 0; s < nseg; ++s) {
    const int ua = seg_unit[s], ub = seg_unit[s + 1], us = ub - ua;
    int cs = 1;
    while (cs * best_u < us) cs *= 2;
    std::vector<int32_t> cut;
    for (;; cs *= 2) {
      if (cs > 16) return LAPY_OK;
      cut.assign(1, ua);
      for (int k = 1; k < cs; ++k) {
        int u = ua + (int)((int64_t)us * k / cs);
        if (u > ua && u < ub && unit_agg[u] >= 0) {  // the nearest aggregate boundary
          int lo = u, hi = u;
          while (lo > ua && unit_agg[lo] == unit_agg[lo - 1]) --lo;
          while (hi < ub && unit_agg[hi] == unit_agg[hi - 1]) ++hi;
          u = (u - lo <= hi - u) ? lo : hi;
        }
        cut.push_back(std::max(u, cut.back()));
      }
      cut.push_back(ub);
      bool fits = true;
      for (int k = 0; k < cs; ++k) fits &= cut[k + 1] - cut[k] <= cap;
      if (fits) break;
    }
    split_cs[s] = cs;
    split0[s] = (int32_t)split.size();
    for (int k = 0; k < cs; ++k) {
      ClSplitCta c;
      c.row0 = cut[k] < ub ? unit_row[cut[k]] : seg_row[s + 1];
      c.row1 = cut[k + 1] < ub ? unit_row[cut[k + 1]] : seg_row[s + 1];
      c.seg0 = seg_row[s];
      c.seg1 = seg_row[s + 1];
      c.first = split0[s];
      c.word0 = words;
      words += (c.seg1 - c.seg0 + 31) >> 5;
      for (int u = cut[k]; u < cut[k + 1]; ++u) unit_cta[u] = (int32_t)split.size();
      cta_unit0.push_back(cut[k]);
      cta_units.push_back(cut[k + 1] - cut[k]);
      split.push_back(c);
    }
  }
  const int nsplit = (int)split.size();
  if (nsplit >= (1 << 19)) return LAPY_OK;  // row_slot keeps the CTA in 19 bits

  // device memory: tables, then codes and values
  char* w = (char*)(((uintptr_t)mem + 255) & ~uintptr_t(255));
  char* const end = (char*)mem + bytes;
  auto take = [&](size_t b) {
    char* r = w;
    w += a256(b);
    return r;
  };
  int max_cta = 0;
  for (int s = 0; s < nseg; ++s) max_cta += split_cs[s] * groups;
  auto* d_row = (int32_t*)take(4 * (size_t)(nunit + 1));
  auto* d_agg = (int32_t*)take(4 * (size_t)nunit);
  auto* d_aun = (int32_t*)take(8 * (size_t)nagg);
  auto* d_uct = (int32_t*)take(4 * (size_t)nunit);
  auto* d_cu0 = (int32_t*)take(4 * (size_t)nsplit);
  auto* d_cun = (int32_t*)take(4 * (size_t)nsplit);
  auto* d_spl = (ClSplitCta*)take(sizeof(ClSplitCta) * (size_t)nsplit);
  auto* d_cta = (ClusterCta*)take(sizeof(ClusterCta) * (size_t)max_cta);
  auto* d_slot = (int32_t*)take(4 * (size_t)n);
  auto* d_bits = (uint32_t*)take(4 * (size_t)words);
  auto* d_rank = (int32_t*)take(4 * (size_t)words);
  auto* d_scr = (int32_t*)take(4 * (size_t)scan_scratch_elems(nunit + 1));
  auto* d_cnt = (int32_t*)take(4 * (size_t)(nunit + 1));
  // read back together: slice sizes (summed there), push lists, halo sizes, flag
  auto* d_ptr = (int32_t*)take(4 * (size_t)(nunit + 1));
  auto* d_pp = (int32_t*)take(4 * (size_t)(nunit + 1));
  auto* d_halo = (int32_t*)take(4 * (size_t)nsplit);
  auto* d_bad = (int*)take(4);
  const size_t back = (size_t)(w - (char*)d_ptr);
  if (w > end) return LAPY_OK;
  auto put = [&](void* dst, const void* src, size_t b) -> int {
    if (b) LAPY_CUDA_TRY(cudaMemcpyAsync(dst, src, b, cudaMemcpyHostToDevice, stream));
    return LAPY_OK;
  };
  LAPY_TRY(put(d_row, unit_row.data(), 4 * (size_t)(nunit + 1)));
  LAPY_TRY(put(d_uct, unit_cta.data(), 4 * (size_t)nunit));
  LAPY_TRY(put(d_cu0, cta_unit0.data(), 4 * (size_t)nsplit));
  LAPY_TRY(put(d_cun, cta_units.data(), 4 * (size_t)nsplit));
  LAPY_TRY(put(d_spl, split.data(), sizeof(ClSplitCta) * (size_t)nsplit));
  LAPY_TRY(put(d_agg, unit_agg.data(), 4 * (size_t)nunit));
  LAPY_TRY(put(d_aun, agg_unit.data(), 8 * (size_t)nagg));
  LAPY_CUDA_TRY(cudaMemsetAsync(d_bad, 0, 4, stream));
  const unsigned blocks = lapy_ceil_div((int64_t)nunit * 32, 256);
  cl_width_kernel<<<blocks, 256, 0, stream>>>(nunit, d_row, d_uct, d_cu0, indptr, indices, d_ptr, d_slot);
  LAPY_TRY(lapy_check_launch("cl_width_kernel"));
  LAPY_CUDA_TRY(cudaMemsetAsync(d_cnt, 0, 4 * (size_t)(nunit + 1), stream));
  cl_halo_kernel<<<nsplit, 256, 0, stream>>>(d_spl, indptr, indices, d_slot, d_cu0, d_bits, d_rank, d_halo, d_cnt,
                                             d_bad);
  LAPY_TRY(lapy_check_launch("cl_halo_kernel"));
  LAPY_TRY(exclusive_scan_i32(d_cnt, d_pp, nunit, d_scr, stream));
  std::vector<char> hback(back);
  LAPY_CUDA_TRY(cudaMemcpyAsync(hback.data(), d_ptr, back, cudaMemcpyDeviceToHost, stream));
  LAPY_CUDA_TRY(cudaStreamSynchronize(stream));
  std::vector<int32_t> slice;
  const int64_t total = slice_starts((const int32_t*)hback.data(), nunit, &slice);
  const int32_t* pptr = (const int32_t*)(hback.data() + ((char*)d_pp - (char*)d_ptr));
  const int32_t* halo = (const int32_t*)(hback.data() + ((char*)d_halo - (char*)d_ptr));
  if (*(const int*)(hback.data() + ((char*)d_bad - (char*)d_ptr))) return LAPY_OK;
  const int64_t npush = pptr[nunit];  // (no more than the matrix has entries)
  if (total < 0) return LAPY_OK;
  auto* d_push = (uint32_t*)take(4 * (size_t)npush);
  auto* d_code = (uint16_t*)take(2 * (size_t)total);
  auto* d_val = (float*)take(4 * (size_t)total);
  auto* d_diag = (float*)take(128 * (size_t)nunit);
  if (w > end) return LAPY_OK;
  LAPY_TRY(put(d_ptr, slice.data(), 4 * slice.size()));

  // launches: clusters of one size together, the larger meshes first
  std::vector<int32_t> items(nseg);
  for (int s = 0; s < nseg; ++s) items[s] = s;
  std::stable_sort(items.begin(), items.end(), [&](int32_t x, int32_t y) {
    if (split_cs[x] != split_cs[y]) return split_cs[x] > split_cs[y];
    return seg_unit[x + 1] - seg_unit[x] > seg_unit[y + 1] - seg_unit[y];
  });
  std::vector<ClusterCta> cta;
  cta.reserve(max_cta);
  out->cls.clear();
  for (const int32_t s : items) {
    if (seg_row[s + 1] == seg_row[s]) continue;
    const int cs = split_cs[s];
    if (out->cls.empty() || out->cls.back().cs != cs) {
      ClusterClass k;
      k.cs = cs;
      k.cta0 = (int)cta.size();
      out->cls.push_back(k);
    }
    ClusterClass& k = out->cls.back();
    for (int g = 0; g < groups; ++g)
      for (int r = 0; r < cs; ++r) {
        const int q = split0[s] + r, ua = cta_unit0[q], ub = ua + cta_units[q];
        if (32 * cta_units[q] + halo[q] > 65535) return LAPY_OK;
        ClusterCta c;
        c.row0 = split[q].row0;
        c.row1 = split[q].row1;
        c.unit0 = ua;
        c.unit1 = ub;
        c.agg0 = c.agg1 = 0;
        if (tl && seg_agg[s + 1] > seg_agg[s]) {
          c.agg0 = ua < seg_unit[s + 1] ? unit_agg[ua] : seg_agg[s + 1];
          c.agg1 = ub < seg_unit[s + 1] ? unit_agg[ub] : seg_agg[s + 1];
          k.ld = std::max(k.ld, (seg_agg[s + 1] - seg_agg[s] + 7) & ~7);
        }
        c.seg = s;
        c.col0 = g * np;
        k.units = std::max(k.units, ub - ua);
        c.nhalo = halo[q];
        k.halo = std::max(k.halo, halo[q]);
        k.slots = std::max(k.slots, 32 * (ub - ua) + halo[q]);
        k.aggs = std::max(k.aggs, c.agg1 - c.agg0);
        k.push = std::max(k.push, pptr[ub] - pptr[ua]);
        k.elems = std::max<int64_t>(k.elems, slice[ub] - slice[ua]);
        cta.push_back(c);
      }
    k.ncta = (int)cta.size() - k.cta0;
  }
  for (ClusterClass& k : out->cls) {
    const ClVariant* var = variant(np, k.units);
    if (!var) return LAPY_OK;
    k.kernel = (const void*)(tl ? var->tl : var->jacobi);
    k.warps = std::max(1, std::min(kClMaxWarps, k.units));
    k.z_halo = k.halo <= kZHalo && class_layout(k, np, tl, false, false, true, nullptr) <= kClSmemMax;
    k.mat_smem = class_layout(k, np, tl, true, false, k.z_halo, nullptr) <= kClSmemMax;
    k.coarse_smem = class_layout(k, np, tl, k.mat_smem, true, k.z_halo, nullptr) <= kClSmemMax;
    k.smem = class_layout(k, np, tl, k.mat_smem, k.coarse_smem, k.z_halo, nullptr);
    if (k.smem > kClSmemMax) return LAPY_OK;
    LAPY_CUDA_TRY(cudaFuncSetAttribute(k.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClSmemMax));
    LAPY_CUDA_TRY(cudaFuncSetAttribute(k.kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr;
    launch_config(k, stream, &cfg, &attr);
    int resident = 0;
    if (cudaOccupancyMaxActiveClusters(&resident, k.kernel, &cfg) != cudaSuccess || resident < 1) {
      cudaGetLastError();  // a device (or a part of one) without room for this cluster size
      return LAPY_OK;
    }
  }
  LAPY_TRY(put(d_cta, cta.data(), sizeof(ClusterCta) * cta.size()));
  if (npush > 0) {
    LAPY_CUDA_TRY(cudaMemsetAsync(d_cnt, 0, 4 * (size_t)(nunit + 1), stream));
    cl_push_kernel<<<nsplit, 256, 0, stream>>>(d_spl, d_slot, d_cu0, d_bits, d_rank, d_pp, d_cnt, d_push);
    LAPY_TRY(lapy_check_launch("cl_push_kernel"));
  }
  cl_fill_kernel<<<blocks, 256, 0, stream>>>(nunit, d_row, d_uct, d_cu0, d_cun, d_spl, d_slot, d_bits, d_rank, indptr,
                                             indices, k32, d_ptr, d_code, d_val, d_diag);
  LAPY_TRY(lapy_check_launch("cl_fill_kernel"));
  LAPY_CUDA_TRY(cudaStreamSynchronize(stream));  // the host vectors are pageable
  LAPY_TRY(make_streams(out));
  out->p = p;
  out->np = np;
  out->cta = d_cta;
  out->unit_row = d_row;
  out->unit_agg = d_agg;
  out->agg_unit = d_aun;
  out->slice_ptr = d_ptr;
  out->code = d_code;
  out->val = d_val;
  out->diag = d_diag;
  out->push_ptr = d_pp;
  out->push = d_push;
  out->ok = true;
  return LAPY_OK;
}

int cluster_solve(const ClusterPlan& plan, const ClusterSolve& s, cudaStream_t stream) {
  const bool tl = s.pc->kind == kPrecTwoLevel;
  ClArgs a{};
  a.p = plan.p;
  a.B = s.B;
  a.X = s.X;
  a.indptr = s.indptr;
  a.indices = s.indices;
  a.k64 = s.k64;
  a.dinv = s.dinv;
  a.cta = plan.cta;
  a.unit_row = plan.unit_row;
  a.unit_agg = plan.unit_agg;
  a.agg_unit = plan.agg_unit;
  a.slice_ptr = plan.slice_ptr;
  a.code = plan.code;
  a.val = plan.val;
  a.diag = plan.diag;
  a.push_ptr = plan.push_ptr;
  a.push = plan.push;
  a.seg_agg = s.pc->seg_agg;
  a.kinv_off = s.pc->kinv_off;
  a.kinv = s.pc->kinv;
  a.kvec = s.pc->kvec;
  a.kscale = s.pc->kscale;
  a.rtol = s.rtol;
  a.inner_rtol = s.inner_rtol;
  a.max_rounds = s.max_rounds;
  a.maxiter = s.maxiter;
  a.state = s.state;
  a.relres2 = s.relres2;
  a.ctl = s.ctl;
  const int ncls = (int)plan.cls.size();
  const bool fork = ncls > 1;
  if (fork) LAPY_CUDA_TRY(cudaEventRecord(plan.events.back(), stream));
  auto begin = [&](int i) -> int {
    const ClusterClass& k = plan.cls[i];
    cudaStream_t on = fork ? plan.streams[i] : stream;
    if (fork) LAPY_CUDA_TRY(cudaStreamWaitEvent(on, plan.events.back(), 0));
    class_layout(k, plan.np, tl, k.mat_smem, k.coarse_smem, k.z_halo, &a);
    a.z_halo = k.z_halo ? 1 : 0;
    a.mat_smem = k.mat_smem ? 1 : 0;
    a.coarse_smem = k.coarse_smem ? 1 : 0;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr;
    launch_config(k, on, &cfg, &attr);
    LAPY_CUDA_TRY(cudaLaunchKernelEx(&cfg, (ClKernel)k.kernel, (const ClArgs)a, k.cta0));
    return lapy_check_launch("ir_cluster_kernel");
  };
  // the caller's stream waits for the class; where that fails, the host does
  auto join = [&](int i) -> int {
    if (!fork) return LAPY_OK;
    if (cudaEventRecord(plan.events[i], plan.streams[i]) == cudaSuccess &&
        cudaStreamWaitEvent(stream, plan.events[i], 0) == cudaSuccess)
      return LAPY_OK;
    cudaGetLastError();
    LAPY_CUDA_TRY(cudaStreamSynchronize(plan.streams[i]));
    return LAPY_OK;
  };
  return fork_join(ncls, begin, join);
}

}  // namespace lapy
