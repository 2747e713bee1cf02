// FEM assembly for triangle and tetrahedral meshes: deterministic CSR build
// (segmented sort-and-reduce) and per-element cotangent stiffness / mass.
//
// This translation unit is compiled with --fmad=false so that the element
// arithmetic rounds every product separately, as NumPy does in
// lapy/solver.py:_fem_tria / _fem_tria_aniso / _fem_tetra.
#include "common.cuh"
#include "scan.cuh"

namespace lapy {

// COO slot of the local entry (i, j), four bits each, in the reference's order
// Triangles: solver.py:174-175  (t1,t2,t2,t3,t3,t1,t1,t2,t3) x (t2,t1,t3,t2,t1,t3,t1,t2,t3)
// Tetrahedra: solver.py:492-497.
template <int NPE>
__device__ __forceinline__ int coo_slot(int i, int j) {
  constexpr uint64_t kSlots = NPE == 3 ? 0x834271506ull : 0xfb97ae3482d1650cull;
  return (int)(kSlots >> (4 * (i * NPE + j))) & 15;
}

// ---------------------------------------------------------------------------
// Symbolic phase
// ---------------------------------------------------------------------------
// Every corner of an element adds npe entries to the row of its vertex, so
// rows are bucketed by corners (element * npe + corner, 4 bytes each) and the
// npe (column, position) keys of a corner are formed where they are sorted.
struct SymbolicWs {
  int32_t* row_count;   // n      corners per row, later fill cursor
  int32_t* corner_ptr;  // n + 1  exclusive scan of row_count
  int32_t* row_nnz;     // n      distinct columns per row
  int32_t* corners;     // m*npe  corners, bucketed by row
  uint64_t* sorted;     // m*L    keys (col << 32 | pos) sorted inside each row, bit 31: first of its column
  int32_t* scan_scratch;
  int* bad;             // set if an index lies outside [0, n)
};

static size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

static size_t symbolic_layout(int64_t n, int64_t m, int npe, char* base, SymbolicWs* ws) {
  const int64_t coo = m * npe * npe;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* p = base ? base + off : nullptr;
    off += align256(bytes);
    return p;
  };
  char* p0 = take(sizeof(int32_t) * (size_t)n);
  char* p1 = take(sizeof(int32_t) * (size_t)(n + 1));
  char* p2 = take(sizeof(int32_t) * (size_t)n);
  char* p3 = take(sizeof(int32_t) * (size_t)(m * npe));
  char* p4 = take(sizeof(uint64_t) * (size_t)coo);
  char* p5 = take(sizeof(int32_t) * (size_t)scan_scratch_elems(n + 1));
  char* p6 = take(sizeof(int));
  if (ws) {
    ws->row_count = (int32_t*)p0;
    ws->corner_ptr = (int32_t*)p1;
    ws->row_nnz = (int32_t*)p2;
    ws->corners = (int32_t*)p3;
    ws->sorted = (uint64_t*)p4;
    ws->scan_scratch = (int32_t*)p5;
    ws->bad = (int*)p6;
  }
  return off;
}

__global__ void corner_count_kernel(const int32_t* __restrict__ elems, int64_t ncorner,
                                    int32_t* __restrict__ row_count, int64_t n, int* bad) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncorner) return;
  const int32_t r = elems[c];
  if (r < 0 || r >= n) {
    atomicExch(bad, 1);
    return;
  }
  atomicAdd(&row_count[r], 1);
}

__global__ void corner_bucket_kernel(const int32_t* __restrict__ elems, int64_t ncorner,
                                     const int32_t* __restrict__ corner_ptr, int32_t* __restrict__ cursor,
                                     int32_t* __restrict__ corners, int64_t n) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncorner) return;
  const int32_t r = elems[c];
  if (r < 0 || r >= n) return;
  corners[corner_ptr[r] + atomicAdd(&cursor[r], 1)] = (int32_t)c;
}

constexpr int kSortChunk = 128;  // keys of a row held per warp
constexpr int kSortWarps = 8;

// Key of entry a of a row whose corners start at `cs`.
template <int NPE>
__device__ __forceinline__ uint64_t coo_key(const int32_t* __restrict__ elems, const int32_t* __restrict__ cs, int a) {
  const int32_t c = cs[a / NPE];
  const int j = a % NPE, e = c / NPE, i = c - e * NPE;
  const int l = coo_slot<NPE>(i, j);
  return ((uint64_t)(uint32_t)elems[(int64_t)e * NPE + j] << 32) | (uint32_t)(e * (NPE * NPE) + l);
}

// Ranks of the NQ keys a lane holds (keys [a0, a0 + 32 NQ) of a row of k).
template <int NPE, int NQ>
__device__ __forceinline__ void rank_chunk(const int32_t* __restrict__ elems, const int32_t* __restrict__ cs, int k,
                                           int a0, int lane, uint64_t* sm, uint64_t* __restrict__ sorted) {
  uint64_t ka[NQ];
  int rank[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int a = a0 + lane + 32 * q;
    ka[q] = a < k ? coo_key<NPE>(elems, cs, a) : ~uint64_t(0);
    rank[q] = 0;
  }
  for (int b0 = 0; b0 < k; b0 += kSortChunk) {
    const int nb = min(kSortChunk, k - b0);
    __syncwarp();
    if (b0 == a0) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) sm[lane + 32 * q] = ka[q];
    } else {
      for (int t = lane; t < nb; t += 32) sm[t] = coo_key<NPE>(elems, cs, b0 + t);
    }
    __syncwarp();
#pragma unroll 4
    for (int t = 0; t < nb; ++t) {
      const uint64_t kb = sm[t];
#pragma unroll
      for (int q = 0; q < NQ; ++q) rank[q] += kb < ka[q] ? 1 : 0;
    }
  }
  if (k <= kSortChunk) {  // back through shared memory: the caller reads it, stores coalesced
    __syncwarp();
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (lane + 32 * q < k) sm[rank[q]] = ka[q];
  } else {
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (a0 + lane + 32 * q < k) sorted[rank[q]] = ka[q];
  }
  __syncwarp();
}

constexpr uint32_t kFirst = 0x80000000u;  // positions are below 2^31

// One warp sorts a row of k keys by rank (the keys are unique, so the rank of
// a key is the number of smaller keys), marks the first key of every column
// and returns the number of columns.
template <int NPE>
__device__ __forceinline__ int warp_sort_row(const int32_t* __restrict__ elems, const int32_t* __restrict__ cs, int k,
                                             uint64_t* sm, uint64_t* __restrict__ out, int lane) {
  for (int a0 = 0; a0 < k; a0 += kSortChunk) {
    const int na = k - a0;
    if (na <= 32) rank_chunk<NPE, 1>(elems, cs, k, a0, lane, sm, out);
    else if (na <= 64) rank_chunk<NPE, 2>(elems, cs, k, a0, lane, sm, out);
    else rank_chunk<NPE, 4>(elems, cs, k, a0, lane, sm, out);
  }
  int cnt = 0;
  if (k <= kSortChunk) {
    for (int a = lane; a < k; a += 32) {
      const uint64_t key = sm[a];
      const bool first = a == 0 || (uint32_t)(sm[a - 1] >> 32) != (uint32_t)(key >> 32);
      out[a] = first ? key | kFirst : key;
      cnt += first ? 1 : 0;
    }
  } else {
    uint32_t* half = reinterpret_cast<uint32_t*>(out);  // column at 2a + 1, position at 2a
    for (int a = lane; a < k; a += 32) {
      const bool first = a == 0 || half[2 * (int64_t)a - 1] != half[2 * (int64_t)a + 1];
      if (first) half[2 * (int64_t)a] |= kFirst;
      cnt += first ? 1 : 0;
    }
  }
  __syncwarp();
  return warp_sum(cnt);
}

// Tetrahedra: one warp per row (about 24 corners, 96 keys).
__global__ void __launch_bounds__(32 * kSortWarps) row_sort_tet_kernel(int64_t n, const int32_t* __restrict__ elems,
                                                                       const int32_t* __restrict__ corner_ptr,
                                                                       const int32_t* __restrict__ corners,
                                                                       uint64_t* __restrict__ sorted,
                                                                       int32_t* __restrict__ row_nnz) {
  __shared__ uint64_t keys[kSortWarps][kSortChunk];
  const int lane = threadIdx.x & 31;
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= n) return;
  const int32_t c0 = corner_ptr[row];
  const int cnt = warp_sort_row<4>(elems, corners + c0, (corner_ptr[row + 1] - c0) * 4, keys[threadIdx.x >> 5],
                                   sorted + (int64_t)c0 * 4, lane);
  if (lane == 0) row_nnz[row] = cnt;
}

// Triangles: one thread per row of up to kNarrow corners, wider rows (and rows
// of elements that name a vertex twice) by the warp afterwards.  A thread sorts
// its corners and the two off-diagonal keys of each by networks in registers;
// the diagonal entries follow from the corners' order.  A warp's rows are
// neighbours in memory, so the keys leave through shared memory in whole
// lines.  A warp per row was bound by instruction issue (about 400 slots for 18
// keys): 374 us for 1.25 million rows with the keys from memory, 72 us now.
constexpr int kNarrow = 8;
constexpr int kTriaSortWarps = 4;

template <typename K, int N>
__device__ __forceinline__ void sort_network(K (&x)[N]) {  // Batcher's odd-even merge sort, N a power of two
#pragma unroll
  for (int p = 1; p < N; p *= 2)
#pragma unroll
    for (int k = p; k >= 1; k /= 2)
#pragma unroll
      for (int j = 0; j + k < N; ++j)
        if (j >= k % p && (j - k % p) % (2 * k) < k && j / (2 * p) == (j + k) / (2 * p)) {
          const K lo = min(x[j], x[j + k]), hi = max(x[j], x[j + k]);
          x[j] = lo;
          x[j + k] = hi;
        }
}

__global__ void __launch_bounds__(32 * kTriaSortWarps) row_sort_tria_kernel(int64_t n,
                                                                            const int32_t* __restrict__ elems,
                                                                            const int32_t* __restrict__ corner_ptr,
                                                                            const int32_t* __restrict__ corners,
                                                                            uint64_t* __restrict__ sorted,
                                                                            int32_t* __restrict__ row_nnz) {
  __shared__ uint64_t stage[kTriaSortWarps][32 * kNarrow * 3];  // also the warp's kSortChunk keys
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, row0 = row - lane;
  if (row0 >= n) return;
  uint64_t* sm = stage[threadIdx.x >> 5];
  const int32_t c0 = row < n ? corner_ptr[row] : 0;
  const int val = row < n ? corner_ptr[row + 1] - c0 : 0;
  bool wide = val > kNarrow;
  uint32_t c[kNarrow];
  uint64_t key[2 * kNarrow];
  if (!wide) {
#pragma unroll
    for (int d = 0; d < kNarrow; ++d) c[d] = d < val ? (uint32_t)corners[c0 + d] : 0xffffffffu;
    sort_network(c);
#pragma unroll
    for (int d = 0; d < kNarrow; ++d) {
      const uint32_t e = c[d] / 3, i = c[d] - 3 * e;
#pragma unroll
      for (uint32_t o = 0; o < 2; ++o) {
        const uint32_t j = (i + 1 + o) % 3;
        uint64_t x = ~uint64_t(0);
        if (d < val) {
          const uint32_t col = (uint32_t)elems[3 * (int64_t)e + j];
          wide |= col == (uint32_t)row;
          x = ((uint64_t)col << 32) | (9 * e + coo_slot<3>(i, j));
        }
        key[2 * d + o] = x;
      }
    }
    sort_network(key);
  }
  const bool staged = !__any_sync(0xffffffffu, wide);
  const int32_t w0 = __shfl_sync(0xffffffffu, c0, 0);
  if (!wide && val > 0) {
    uint64_t* out = staged ? sm + 3 * (c0 - w0) : sorted + 3 * (int64_t)c0;
    int cnt = 1, less = 0;
#pragma unroll
    for (int q = 0; q < 2 * kNarrow; ++q)
      if (q < 2 * val) {
        const uint32_t col = (uint32_t)(key[q] >> 32);
        const bool first = q == 0 || col != (uint32_t)(key[q - (q > 0)] >> 32), before = col < (uint32_t)row;
        out[before ? q : q + val] = first ? key[q] | kFirst : key[q];
        cnt += first ? 1 : 0;
        less += before ? 1 : 0;
      }
#pragma unroll
    for (int d = 0; d < kNarrow; ++d)
      if (d < val) {
        const uint32_t e = c[d] / 3, pos = 9 * e + 6 + (c[d] - 3 * e);
        out[less + d] = ((uint64_t)(uint32_t)row << 32) | (d == 0 ? pos | kFirst : pos);
      }
    row_nnz[row] = cnt;
  } else if (row < n && val == 0) {
    row_nnz[row] = 0;
  }
  __syncwarp();
  if (staged) {
    const int total = 3 * (corner_ptr[min(row0 + 32, n)] - w0);
    for (int t = lane; t < total; t += 32) sorted[3 * (int64_t)w0 + t] = sm[t];
    return;
  }
  for (unsigned todo = __ballot_sync(0xffffffffu, wide); todo; todo &= todo - 1) {
    const int src = __ffs(todo) - 1;
    const int32_t r0 = __shfl_sync(0xffffffffu, c0, src);
    const int k = 3 * __shfl_sync(0xffffffffu, val, src);
    const int cnt = warp_sort_row<3>(elems, corners + r0, k, sm, sorted + 3 * (int64_t)r0, lane);
    if (lane == 0) row_nnz[row0 + src] = cnt;
  }
}

// Column indices, run starts and source positions: a CTA takes kFillRows rows,
// whose entries and runs are contiguous, and compacts the marked keys.  Bound
// by memory: 1.25 million rows 185 us with a warp per row, 51 us now.
constexpr int kFillRows = 256;
constexpr int kFillWarps = 8;
constexpr int kFillItems = 4;

__global__ void __launch_bounds__(32 * kFillWarps) row_fill_kernel(int64_t n, int npe, int64_t nnz,
                                                                   const int32_t* __restrict__ corner_ptr,
                                                                   const uint64_t* __restrict__ sorted,
                                                                   const int32_t* __restrict__ indptr,
                                                                   int32_t* __restrict__ indices,
                                                                   int32_t* __restrict__ seg_ptr,
                                                                   int32_t* __restrict__ seg_src) {
  __shared__ int wsum[2][kFillWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t r0 = (int64_t)blockIdx.x * kFillRows, r1 = min(r0 + kFillRows, n);
  const int64_t b0 = (int64_t)npe * corner_ptr[r0], b1 = (int64_t)npe * corner_ptr[r1];
  if (r1 == n && threadIdx.x == 0) seg_ptr[nnz] = (int32_t)b1;
  int32_t out = indptr[r0];
  int buf = 0;
  for (int64_t base = b0; base < b1; base += 32 * kFillWarps * kFillItems, buf ^= 1) {
    const int64_t a0 = base + (warp * kFillItems) * 32 + lane;
    uint64_t key[kFillItems];
    unsigned mask[kFillItems];
    int cnt = 0;
#pragma unroll
    for (int q = 0; q < kFillItems; ++q) key[q] = a0 + 32 * q < b1 ? sorted[a0 + 32 * q] : 0;
#pragma unroll
    for (int q = 0; q < kFillItems; ++q) {
      mask[q] = __ballot_sync(0xffffffffu, ((uint32_t)key[q] & kFirst) != 0);
      cnt += __popc(mask[q]);
    }
    if (lane == 0) wsum[buf][warp] = cnt;
    __syncthreads();  // the other buffer's readers are past the next iteration's barrier
    int32_t at = out;
#pragma unroll
    for (int w = 0; w < kFillWarps; ++w) {
      const int x = wsum[buf][w];
      at += w < warp ? x : 0;
      out += x;
    }
#pragma unroll
    for (int q = 0; q < kFillItems; ++q) {
      const int64_t a = a0 + 32 * q;
      if (a < b1) seg_src[a] = (int32_t)((uint32_t)key[q] & ~kFirst);
      if ((uint32_t)key[q] & kFirst) {
        const int32_t o = at + __popc(mask[q] & ((1u << lane) - 1u));
        indices[o] = (int32_t)(key[q] >> 32);
        seg_ptr[o] = (int32_t)a;
      }
      at += __popc(mask[q]);
    }
  }
}

// ---------------------------------------------------------------------------
// Numeric phase
// ---------------------------------------------------------------------------
// Distinct local values of an element, one 16-byte aligned record each:
// triangles a12 a23 a31 a11 a22 a33 | bii bij, tetrahedra a12 a23 a13 a14 a24
// a34 a11 .. a44 | bii bij.
template <int NPE>
struct Rec {
  static constexpr int kSize = NPE == 3 ? 8 : 12;
  static constexpr int kOff = NPE * (NPE - 1);       // COO slots off the diagonal, in equal pairs
  static constexpr int kBii = kSize - 2, kBij = kSize - 1;
};

struct NumericWs {
  double* vol;       // m      (element measure in the coordinate type, widened)
  double* partials;  // kVolBlocks
  double* clamp;     // max(nseg, 1): max(1e-4 * mean(vol), eps) per mesh
  char* local;       // m*Rec  local values (output type)
  int* low;          // set if an element's measure is below eps
};
constexpr int kVolBlocks = 1024;
constexpr int kVolThreads = 256;

static size_t numeric_layout(int64_t m, int npe, int nseg, char* base, NumericWs* ws) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* p = base ? base + off : nullptr;
    off += align256(bytes);
    return p;
  };
  char* p0 = take(sizeof(double) * (size_t)m);
  char* p1 = take(sizeof(double) * kVolBlocks);
  char* p2 = take(sizeof(double) * (size_t)std::max(nseg, 2));
  char* p3 = take(sizeof(double) * (size_t)(m * (npe == 3 ? Rec<3>::kSize : Rec<4>::kSize)));
  char* p4 = take(sizeof(int));
  if (ws) {
    ws->vol = (double*)p0;
    ws->partials = (double*)p1;
    ws->clamp = (double*)p2;
    ws->local = p3;
    ws->low = (int*)p4;
  }
  return off;
}

template <typename T>
struct V3 {
  T x, y, z;
};
template <typename T>
__device__ __forceinline__ V3<T> load_v(const T* v, int32_t i) {
  return V3<T>{v[3 * (int64_t)i], v[3 * (int64_t)i + 1], v[3 * (int64_t)i + 2]};
}
template <typename T>
__device__ __forceinline__ V3<T> sub(V3<T> a, V3<T> b) {
  return V3<T>{a.x - b.x, a.y - b.y, a.z - b.z};
}
// NumPy order: np.sum(a * b, axis=1) over 3 columns = (a0*b0 + a1*b1) + a2*b2
template <typename T>
__device__ __forceinline__ T dot3(V3<T> a, V3<T> b) {
  T s = a.x * b.x;
  s = s + a.y * b.y;
  s = s + a.z * b.z;
  return s;
}
// np.cross: (a1*b2 - a2*b1, a2*b0 - a0*b2, a0*b1 - a1*b0)
template <typename T>
__device__ __forceinline__ V3<T> cross3(V3<T> a, V3<T> b) {
  return V3<T>{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

template <typename T>
__device__ __forceinline__ T tria_vol(const T* v, const int32_t* t, int64_t e) {
  const V3<T> v1 = load_v(v, t[3 * e]), v2 = load_v(v, t[3 * e + 1]), v3 = load_v(v, t[3 * e + 2]);
  const V3<T> v3mv2 = sub(v3, v2), v1mv3 = sub(v1, v3);
  const V3<T> cr = cross3(v3mv2, v1mv3);
  return T(2) * sqrt(dot3(cr, cr));  // solver.py:155-156  (= 4 * area)
}

template <typename T>
__device__ __forceinline__ T tet_vol(const T* v, const int32_t* t, int64_t e) {
  const V3<T> v1 = load_v(v, t[4 * e]), v2 = load_v(v, t[4 * e + 1]), v3 = load_v(v, t[4 * e + 2]),
              v4 = load_v(v, t[4 * e + 3]);
  const V3<T> e1 = sub(v2, v1), e3 = sub(v1, v3), e4 = sub(v4, v1);
  const V3<T> cr = cross3(e1, e3);
  return abs(dot3(e4, cr));  // solver.py:433-434  (= 6 * volume)
}

// The numeric phase computes all elements at once; only if one of them has a
// measure below eps (degenerate, `low` set) do the three kernels after it run:
// element measures, mean and clamp per mesh, and those elements again.
//
// Element measures and per-block partial sums (for the global mean).
template <typename T, int NPE>
__global__ void elem_vol_kernel(const T* __restrict__ v, const int32_t* __restrict__ t, int64_t m,
                                const int* __restrict__ low, double* __restrict__ vol,
                                double* __restrict__ partials) {
  __shared__ double sh[32];
  if (*low == 0) return;
  double acc = 0.0;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m;
       e += (int64_t)gridDim.x * blockDim.x) {
    const T w = (NPE == 3) ? tria_vol<T>(v, t, e) : tet_vol<T>(v, t, e);
    vol[e] = (double)w;
    acc += (double)w;
  }
  acc = block_sum(acc, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = acc;
}

// clamp = max(1e-4 * mean(vol), DBL_EPSILON)  (solver.py:158, :272, :436)
template <typename T>
__global__ void vol_clamp_kernel(const double* __restrict__ partials, int nparts, int64_t m,
                                 const int* __restrict__ low, double* __restrict__ clamp) {
  __shared__ double sh[32];
  if (*low == 0) return;
  double acc = 0.0;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) acc += partials[i];
  acc = block_sum(acc, sh);
  if (threadIdx.x == 0) {
    const T mean = (T)(acc / (double)m);
    const T c = T(0.0001) * mean;
    const double eps = 2.220446049250313e-16;
    clamp[0] = ((double)c > eps) ? (double)c : eps;
  }
}

// Per-mesh clamps of a batch: one block per mesh sums the measures of its
// element range [seg_elem[s], seg_elem[s+1]) in a fixed order, so that each
// mesh is clamped with its own mean exactly as a single-mesh assembly does.
template <typename T>
__global__ void seg_vol_clamp_kernel(const double* __restrict__ vol, const int32_t* __restrict__ seg_elem,
                                     const int* __restrict__ low, double* __restrict__ clamp) {
  __shared__ double sh[32];
  if (*low == 0) return;
  const int s = blockIdx.x;
  const int32_t e0 = seg_elem[s], e1 = seg_elem[s + 1];
  double acc = 0.0;
  for (int32_t e = e0 + (int32_t)threadIdx.x; e < e1; e += blockDim.x) acc += vol[e];
  acc = block_sum(acc, sh);
  if (threadIdx.x == 0) {
    const T mean = (e1 > e0) ? (T)(acc / (double)(e1 - e0)) : T(0);
    const T c = T(0.0001) * mean;
    const double eps = 2.220446049250313e-16;
    clamp[s] = ((double)c > eps) ? (double)c : eps;
  }
}

// Where the clamp of element e comes from: clamp[0] for a single mesh, else
// the clamp of the mesh whose element range holds e.
struct ClampDesc {
  const double* clamp;
  const int32_t* seg_elem;  // nseg + 1 element offsets (batches), or null
  int nseg;
  int* low;                 // set by the first pass if an element needs the second
  int fix;                  // second pass: only elements below eps, with their clamp
};

// Whether this pass computes element e (`vol` replaced by the clamp if so).
template <typename T>
__device__ __forceinline__ bool clamp_vol(T& vol, const ClampDesc& cd, int64_t e) {
  const T eps = (T)2.220446049250313e-16;
  if (!(vol < eps)) return !cd.fix;
  if (!cd.fix) {
    *cd.low = 1;
    return false;
  }
  int s = 0;
  if (cd.seg_elem) {  // largest s with seg_elem[s] <= e
    int lo = 0, hi = cd.nseg - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if ((int64_t)cd.seg_elem[mid] <= e) lo = mid; else hi = mid - 1;
    }
    s = lo;
  }
  vol = (T)cd.clamp[s];
  return true;
}

// Record of element e, stored as 16-byte vectors.
template <int NPE, typename O>
__device__ __forceinline__ void store_rec(O* __restrict__ loc, int64_t e, const O (&q)[Rec<NPE>::kSize]) {
  constexpr int kPer = 16 / (int)sizeof(O);
  O* p = loc + Rec<NPE>::kSize * e;
#pragma unroll
  for (int i = 0; i < Rec<NPE>::kSize; i += kPer) {
    if constexpr (kPer == 2)
      *reinterpret_cast<double2*>(p + i) = make_double2(q[i], q[i + 1]);
    else
      *reinterpret_cast<float4*>(p + i) = make_float4(q[i], q[i + 1], q[i + 2], q[i + 3]);
  }
}

// The local values are bound by the FP64 rate (about 100 operations per
// triangle, two per clock and SM); the sums by the gathers, hence one record of
// 64 (96) bytes per element instead of two of 72 (128).  At 2.5 million
// triangles: measures, clamps and values 737 -> 410 us, sums 235 -> 205 us.
//
// Local values (triangles): local stiffness (cotangent) and mass values.
template <typename T, typename O>
__global__ void tria_local_kernel(const T* __restrict__ v, const int32_t* __restrict__ t, int64_t m,
                                  const ClampDesc clamp, int lump, O* __restrict__ loc) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m || (clamp.fix && *clamp.low == 0)) return;
  const V3<T> v1 = load_v(v, t[3 * e]), v2 = load_v(v, t[3 * e + 1]), v3 = load_v(v, t[3 * e + 2]);
  const V3<T> v2mv1 = sub(v2, v1), v3mv2 = sub(v3, v2), v1mv3 = sub(v1, v3);
  const V3<T> cr = cross3(v3mv2, v1mv3);
  T vol = T(2) * sqrt(dot3(cr, cr));
  if (!clamp_vol(vol, clamp, e)) return;
  // solver.py:163-169
  const T a12 = dot3(v3mv2, v1mv3) / vol;
  const T a23 = dot3(v1mv3, v2mv1) / vol;
  const T a31 = dot3(v2mv1, v3mv2) / vol;
  const T a11 = -a12 - a31;
  const T a22 = -a12 - a23;
  const T a33 = -a31 - a23;
  const O bii = (O)(vol / T(lump ? 12 : 24));  // solver.py:182-190
  const O q[8] = {(O)a12, (O)a23, (O)a31, (O)a11, (O)a22, (O)a33, bii, (O)(bii * O(0.5))};  // bij = vol / 48
  store_rec<3, O>(loc, e, q);
}

// Local values (anisotropic triangles, solver.py:254-307).  Edge vectors and the
// element measure are in the coordinate type; the curvature frame u1, u2 and
// aniso_mat are float64 as curvature_tria produces them, so the projections
// and quotients run in float64 exactly as NumPy's type promotion does.
template <typename T, typename O>
__global__ void tria_aniso_local_kernel(const T* __restrict__ v, const int32_t* __restrict__ t,
                                        int64_t m, const double* __restrict__ u1,
                                        const double* __restrict__ u2,
                                        const double* __restrict__ an,
                                        const ClampDesc clamp, int lump, O* __restrict__ loc) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m || (clamp.fix && *clamp.low == 0)) return;
  const V3<T> v1 = load_v(v, t[3 * e]), v2 = load_v(v, t[3 * e + 1]), v3 = load_v(v, t[3 * e + 2]);
  const V3<T> v2mv1 = sub(v2, v1), v3mv2 = sub(v3, v2), v1mv3 = sub(v1, v3);
  const V3<double> U1{u1[3 * e], u1[3 * e + 1], u1[3 * e + 2]};
  const V3<double> U2{u2[3 * e], u2[3 * e + 1], u2[3 * e + 2]};
  auto widen = [](V3<T> a) { return V3<double>{(double)a.x, (double)a.y, (double)a.z}; };
  const V3<double> d21 = widen(v2mv1), d32 = widen(v3mv2), d13 = widen(v1mv3);
  const double p21[2] = {dot3(U1, d21), dot3(U2, d21)};
  const double p32[2] = {dot3(U1, d32), dot3(U2, d32)};
  const double p13[2] = {dot3(U1, d13), dot3(U2, d13)};
  const V3<T> cr = cross3(v3mv2, v1mv3);
  T vol = T(2) * sqrt(dot3(cr, cr));
  if (!clamp_vol(vol, clamp, e)) return;
  const double a0 = an[2 * e], a1 = an[2 * e + 1];
  const double dv = (double)vol;
  // np.sum(x * aniso_mat * y, axis=1) = (x0*a0)*y0 + (x1*a1)*y1
  const double a12 = ((p32[0] * a0) * p13[0] + (p32[1] * a1) * p13[1]) / dv;
  const double a23 = ((p13[0] * a0) * p21[0] + (p13[1] * a1) * p21[1]) / dv;
  const double a31 = ((p21[0] * a0) * p32[0] + (p21[1] * a1) * p32[1]) / dv;
  const double a11 = -a12 - a31;
  const double a22 = -a12 - a23;
  const double a33 = -a31 - a23;
  const O bii = (O)(vol / T(lump ? 12 : 24));  // solver.py:182-190
  const O q[8] = {(O)a12, (O)a23, (O)a31, (O)a11, (O)a22, (O)a33, bii, (O)(bii * O(0.5))};  // bij = vol / 48
  store_rec<3, O>(loc, e, q);
}

// Local values (tetrahedra, solver.py:426-532).
template <typename T, typename O>
__global__ void tet_local_kernel(const T* __restrict__ v, const int32_t* __restrict__ t, int64_t m,
                                 const ClampDesc clamp, int lump, O* __restrict__ loc) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m || (clamp.fix && *clamp.low == 0)) return;
  const V3<T> v1 = load_v(v, t[4 * e]), v2 = load_v(v, t[4 * e + 1]), v3 = load_v(v, t[4 * e + 2]),
              v4 = load_v(v, t[4 * e + 3]);
  const V3<T> e1 = sub(v2, v1), e2 = sub(v3, v2), e3 = sub(v1, v3), e4 = sub(v4, v1),
              e5 = sub(v4, v2), e6 = sub(v4, v3);
  const V3<T> cr = cross3(e1, e3);
  T vol = abs(dot3(e4, cr));
  if (!clamp_vol(vol, clamp, e)) return;
  const T e11 = dot3(e1, e1), e22 = dot3(e2, e2), e33 = dot3(e3, e3), e44 = dot3(e4, e4),
          e55 = dot3(e5, e5), e66 = dot3(e6, e6);
  const T e12 = dot3(e1, e2), e13 = dot3(e1, e3), e14 = dot3(e1, e4), e15 = dot3(e1, e5),
          e23 = dot3(e2, e3), e25 = dot3(e2, e5), e26 = dot3(e2, e6), e34 = dot3(e3, e4),
          e36 = dot3(e3, e6);
  (void)e11; (void)e22; (void)e33; (void)e44; (void)e55;
  // solver.py:460-465
  const T a12 = ((-e36) * e26 + e23 * e66) / vol;
  const T a13 = ((-e15) * e25 + e12 * e55) / vol;
  const T a14 = (e23 * e26 - e36 * e22) / vol;
  const T a23 = ((-e14) * e34 + e13 * e44) / vol;
  const T a24 = (e13 * e34 - e14 * e33) / vol;
  const T a34 = ((-e14) * e13 + e11 * e34) / vol;
  // solver.py:467-470
  const T a11 = (-a12 - a13) - a14;
  const T a22 = (-a12 - a23) - a24;
  const T a33 = (-a13 - a23) - a34;
  const T a44 = (-a14 - a24) - a34;
  const T six = T(6);
  const O bii = (O)(vol / T(lump ? 24 : 60));  // solver.py:504-529, stiffness / 6 as solver.py:472-498
  const O q[12] = {(O)(a12 / six), (O)(a23 / six), (O)(a13 / six), (O)(a14 / six), (O)(a24 / six), (O)(a34 / six),
                   (O)(a11 / six), (O)(a22 / six), (O)(a33 / six), (O)(a44 / six), bii, (O)(bii * O(0.5))};
  store_rec<4, O>(loc, e, q);
}

// Per nonzero, sum its run of local values in (element, slot) order.  Lumped
// mass: every diagonal run holds a diagonal slot, whose corner names the row;
// the run's other slots (elements that name a vertex twice) add nothing.  (A
// pass of its own over the rows took 103 us at 2.5 million rows.)
template <typename O, int NPE, bool LUMP>
__global__ void segmented_reduce_kernel(int64_t nnz, const int32_t* __restrict__ seg_ptr,
                                        const int32_t* __restrict__ seg_src, const int32_t* __restrict__ elems,
                                        const O* __restrict__ loc, O* __restrict__ a, O* __restrict__ mvals) {
  constexpr int L = NPE * NPE, kOff = Rec<NPE>::kOff;
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nnz) return;
  const int32_t s0 = seg_ptr[k], s1 = seg_ptr[k + 1];
  O sa = O(0), sm = O(0);
  int32_t corner = -1;
  for (int32_t s = s0; s < s1; ++s) {
    const int32_t src = seg_src[s], e = src / L, l = src - e * L;
    const bool off = l < kOff;
    const O* rec = loc + (int64_t)e * Rec<NPE>::kSize;
    const O va = rec[off ? l >> 1 : l - kOff / 2];
    sa = s == s0 ? va : sa + va;
    if (LUMP) {
      if (!off) {
        sm += rec[Rec<NPE>::kBii];
        corner = e * NPE + l - kOff;
      }
    } else {
      const O vm = rec[off ? Rec<NPE>::kBij : Rec<NPE>::kBii];
      sm = s == s0 ? vm : sm + vm;
    }
  }
  a[k] = sa;
  if (!LUMP) mvals[k] = sm;
  else if (corner >= 0) mvals[elems[corner]] = sm;
}

}  // namespace lapy

using namespace lapy;

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
extern "C" size_t lapy_csr_symbolic_workspace_bytes(int64_t n, int64_t m, int npe) {
  if (n < 0 || m < 0 || (npe != 3 && npe != 4)) return 0;
  return symbolic_layout(n, m, npe, nullptr, nullptr) + 256;
}

extern "C" int lapy_csr_symbolic_count(const int32_t* elems, int64_t m, int npe, int64_t n,
                                       int32_t* indptr, int64_t* nnz_out, void* workspace,
                                       size_t ws_bytes, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if ((npe != 3 && npe != 4) || n <= 0 || m <= 0 || !elems || !indptr || !nnz_out) {
    lapy_set_last_message("csr_symbolic_count: invalid arguments (npe=%d n=%lld m=%lld)", npe,
                          (long long)n, (long long)m);
    return LAPY_ERR_INVALID;
  }
  const int64_t L = (int64_t)npe * npe;
  if (m * L >= (int64_t)INT32_MAX || n >= (int64_t)INT32_MAX) {
    lapy_set_last_message("csr_symbolic_count: %lld local entries exceed int32", (long long)(m * L));
    return LAPY_ERR_INVALID;
  }
  if (ws_bytes < lapy_csr_symbolic_workspace_bytes(n, m, npe)) return LAPY_ERR_WORKSPACE;
  SymbolicWs ws;
  char* base = (char*)(((uintptr_t)workspace + 255) & ~uintptr_t(255));
  symbolic_layout(n, m, npe, base, &ws);
  LAPY_CUDA_TRY(cudaMemsetAsync(ws.row_count, 0, sizeof(int32_t) * n, stream));
  LAPY_CUDA_TRY(cudaMemsetAsync(ws.bad, 0, sizeof(int), stream));
  const int64_t nc = m * npe;
  corner_count_kernel<<<lapy_ceil_div(nc, 256), 256, 0, stream>>>(elems, nc, ws.row_count, n, ws.bad);
  LAPY_TRY(lapy_check_launch("corner_count_kernel"));
  LAPY_TRY(exclusive_scan_i32(ws.row_count, ws.corner_ptr, n, ws.scan_scratch, stream));
  LAPY_CUDA_TRY(cudaMemsetAsync(ws.row_count, 0, sizeof(int32_t) * n, stream));
  corner_bucket_kernel<<<lapy_ceil_div(nc, 256), 256, 0, stream>>>(elems, nc, ws.corner_ptr, ws.row_count,
                                                                   ws.corners, n);
  LAPY_TRY(lapy_check_launch("corner_bucket_kernel"));
  if (npe == 3)
    row_sort_tria_kernel<<<lapy_ceil_div(n, 32 * kTriaSortWarps), 32 * kTriaSortWarps, 0, stream>>>(
        n, elems, ws.corner_ptr, ws.corners, ws.sorted, ws.row_nnz);
  else
    row_sort_tet_kernel<<<lapy_ceil_div(n, kSortWarps), 32 * kSortWarps, 0, stream>>>(
        n, elems, ws.corner_ptr, ws.corners, ws.sorted, ws.row_nnz);
  LAPY_TRY(lapy_check_launch("row_sort_kernel"));
  LAPY_TRY(exclusive_scan_i32(ws.row_nnz, indptr, n, ws.scan_scratch, stream));
  // one wait for both results (a bad index is left out of the buckets above)
  int32_t nnz = 0;
  int hbad = 0;
  LAPY_CUDA_TRY(cudaMemcpyAsync(&hbad, ws.bad, sizeof(int), cudaMemcpyDeviceToHost, stream));
  LAPY_CUDA_TRY(cudaMemcpyAsync(&nnz, indptr + n, sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
  LAPY_CUDA_TRY(cudaStreamSynchronize(stream));
  if (hbad) {
    lapy_set_last_message("csr_symbolic_count: element index outside [0, %lld)", (long long)n);
    return LAPY_ERR_INVALID;
  }
  *nnz_out = nnz;
  return LAPY_OK;
}

extern "C" int lapy_csr_symbolic_fill(const int32_t* elems, int64_t m, int npe, int64_t n,
                                      const int32_t* indptr, int64_t nnz, int32_t* indices,
                                      int32_t* seg_ptr, int32_t* seg_src, void* workspace,
                                      size_t ws_bytes, void* stream_) {
  (void)elems;
  cudaStream_t stream = (cudaStream_t)stream_;
  if ((npe != 3 && npe != 4) || n <= 0 || m <= 0 || !indptr || !indices || !seg_ptr || !seg_src)
    return LAPY_ERR_INVALID;
  if (ws_bytes < lapy_csr_symbolic_workspace_bytes(n, m, npe)) return LAPY_ERR_WORKSPACE;
  SymbolicWs ws;
  char* base = (char*)(((uintptr_t)workspace + 255) & ~uintptr_t(255));
  symbolic_layout(n, m, npe, base, &ws);
  row_fill_kernel<<<lapy_ceil_div(n, kFillRows), 32 * kFillWarps, 0, stream>>>(n, npe, nnz, ws.corner_ptr, ws.sorted, indptr,
                                                                  indices, seg_ptr, seg_src);
  return lapy_check_launch("row_fill_kernel");
}

extern "C" size_t lapy_fem_numeric_workspace_bytes(int64_t m, int npe) {
  if (m < 0 || (npe != 3 && npe != 4)) return 0;
  return numeric_layout(m, npe, 1, nullptr, nullptr) + 256;
}

extern "C" size_t lapy_fem_batch_numeric_workspace_bytes(int64_t m, int npe, int nseg) {
  if (m < 0 || (npe != 3 && npe != 4) || nseg < 1) return 0;
  return numeric_layout(m, npe, nseg, nullptr, nullptr) + 256;
}

namespace {

enum class ElemKind { Tria, TriaAniso, Tet };

template <typename T, typename O>
int fem_numeric_impl(ElemKind kind, const T* v, const int32_t* t, int64_t m, const double* u1,
                     const double* u2, const double* an, int64_t n, const int32_t* indptr,
                     const int32_t* indices, const int32_t* seg_ptr, const int32_t* seg_src,
                     int64_t nnz, int lump, O* a_vals, O* m_vals, const NumericWs& ws,
                     int nseg, const int32_t* seg_elem, cudaStream_t stream) {
  const int npe = (kind == ElemKind::Tet) ? 4 : 3;
  O* loc = (O*)ws.local;
  const unsigned eb = lapy_ceil_div(m, 128);
  auto elements = [&](int fix) {
    const ClampDesc cd{ws.clamp, seg_elem, nseg, ws.low, fix};
    if (kind == ElemKind::Tria)
      tria_local_kernel<T, O><<<eb, 128, 0, stream>>>(v, t, m, cd, lump, loc);
    else if (kind == ElemKind::TriaAniso)
      tria_aniso_local_kernel<T, O><<<eb, 128, 0, stream>>>(v, t, m, u1, u2, an, cd, lump, loc);
    else
      tet_local_kernel<T, O><<<eb, 128, 0, stream>>>(v, t, m, cd, lump, loc);
    return lapy_check_launch("elem_local_kernel");
  };
  LAPY_CUDA_TRY(cudaMemsetAsync(ws.low, 0, sizeof(int), stream));
  LAPY_TRY(elements(0));
  const unsigned vb = (unsigned)std::min<int64_t>(kVolBlocks, std::max<int64_t>(1, lapy_ceil_div(m, kVolThreads)));
  if (npe == 3)
    elem_vol_kernel<T, 3><<<vb, kVolThreads, 0, stream>>>(v, t, m, ws.low, ws.vol, ws.partials);
  else
    elem_vol_kernel<T, 4><<<vb, kVolThreads, 0, stream>>>(v, t, m, ws.low, ws.vol, ws.partials);
  LAPY_TRY(lapy_check_launch("elem_vol_kernel"));
  if (seg_elem) {
    seg_vol_clamp_kernel<T><<<nseg, 256, 0, stream>>>(ws.vol, seg_elem, ws.low, ws.clamp);
    LAPY_TRY(lapy_check_launch("seg_vol_clamp_kernel"));
  } else {
    vol_clamp_kernel<T><<<1, 256, 0, stream>>>(ws.partials, (int)vb, m, ws.low, ws.clamp);
    LAPY_TRY(lapy_check_launch("vol_clamp_kernel"));
  }
  LAPY_TRY(elements(1));
  const unsigned nb = lapy_ceil_div(nnz, 256);
  if (lump) LAPY_CUDA_TRY(cudaMemsetAsync(m_vals, 0, sizeof(O) * (size_t)n, stream));  // rows of no element
  if (npe == 3 && lump)
    segmented_reduce_kernel<O, 3, true><<<nb, 256, 0, stream>>>(nnz, seg_ptr, seg_src, t, loc, a_vals, m_vals);
  else if (npe == 3)
    segmented_reduce_kernel<O, 3, false><<<nb, 256, 0, stream>>>(nnz, seg_ptr, seg_src, t, loc, a_vals, m_vals);
  else if (lump)
    segmented_reduce_kernel<O, 4, true><<<nb, 256, 0, stream>>>(nnz, seg_ptr, seg_src, t, loc, a_vals, m_vals);
  else
    segmented_reduce_kernel<O, 4, false><<<nb, 256, 0, stream>>>(nnz, seg_ptr, seg_src, t, loc, a_vals, m_vals);
  LAPY_TRY(lapy_check_launch("segmented_reduce_kernel"));
  return LAPY_OK;
}

int fem_numeric_dispatch(ElemKind kind, const void* v, int coords_f32, const int32_t* t, int64_t m,
                         const void* u1, const void* u2, const void* an, int64_t n,
                         const int32_t* indptr, const int32_t* indices, const int32_t* seg_ptr,
                         const int32_t* seg_src, int64_t nnz, int lump, int out_f32, void* a_vals,
                         void* m_vals, void* work, size_t ws_bytes, void* stream_, int nseg = 1,
                         const int32_t* seg_elem = nullptr) {
  cudaStream_t stream = (cudaStream_t)stream_;
  const int npe = (kind == ElemKind::Tet) ? 4 : 3;
  if (!v || !t || m <= 0 || n <= 0 || nnz <= 0 || !indptr || !indices || !seg_ptr || !seg_src ||
      !a_vals || !m_vals || !work) {
    lapy_set_last_message("fem_numeric: invalid arguments");
    return LAPY_ERR_INVALID;
  }
  if (kind == ElemKind::TriaAniso && (!u1 || !u2 || !an)) {
    lapy_set_last_message("fem_tria_aniso_numeric: u1, u2 and aniso_mat are required");
    return LAPY_ERR_INVALID;
  }
  if (nseg < 1 || (seg_elem == nullptr && nseg != 1)) {
    lapy_set_last_message("fem_numeric: nseg must be >= 1, with seg_elem for nseg > 1");
    return LAPY_ERR_INVALID;
  }
  if (ws_bytes < lapy_fem_batch_numeric_workspace_bytes(m, npe, nseg)) return LAPY_ERR_WORKSPACE;
  NumericWs ws;
  char* base = (char*)(((uintptr_t)work + 255) & ~uintptr_t(255));
  numeric_layout(m, npe, nseg, base, &ws);
  const double* U1 = (const double*)u1;
  const double* U2 = (const double*)u2;
  const double* AN = (const double*)an;
  if (coords_f32) {
    if (out_f32)
      return fem_numeric_impl<float, float>(kind, (const float*)v, t, m, U1, U2, AN, n, indptr,
                                            indices, seg_ptr, seg_src, nnz, lump, (float*)a_vals,
                                            (float*)m_vals, ws, nseg, seg_elem, stream);
    return fem_numeric_impl<float, double>(kind, (const float*)v, t, m, U1, U2, AN, n, indptr,
                                           indices, seg_ptr, seg_src, nnz, lump, (double*)a_vals,
                                           (double*)m_vals, ws, nseg, seg_elem, stream);
  }
  if (out_f32)
    return fem_numeric_impl<double, float>(kind, (const double*)v, t, m, U1, U2, AN, n, indptr,
                                           indices, seg_ptr, seg_src, nnz, lump, (float*)a_vals,
                                           (float*)m_vals, ws, nseg, seg_elem, stream);
  return fem_numeric_impl<double, double>(kind, (const double*)v, t, m, U1, U2, AN, n, indptr,
                                          indices, seg_ptr, seg_src, nnz, lump, (double*)a_vals,
                                          (double*)m_vals, ws, nseg, seg_elem, stream);
}

}  // namespace

extern "C" int lapy_fem_tria_numeric(const void* v, int coords_f32, const int32_t* t, int64_t m,
                                     int64_t n, const int32_t* indptr, const int32_t* indices,
                                     const int32_t* seg_ptr, const int32_t* seg_src, int64_t nnz,
                                     int lump, int out_f32, void* a_vals, void* m_vals, void* work,
                                     size_t ws_bytes, void* stream) {
  return fem_numeric_dispatch(ElemKind::Tria, v, coords_f32, t, m, nullptr, nullptr, nullptr, n,
                              indptr, indices, seg_ptr, seg_src, nnz, lump, out_f32, a_vals, m_vals,
                              work, ws_bytes, stream);
}

extern "C" int lapy_fem_tria_aniso_numeric(const void* v, int coords_f32, const int32_t* t,
                                           int64_t m, const double* u1, const double* u2,
                                           const double* aniso_mat, int64_t n,
                                           const int32_t* indptr, const int32_t* indices,
                                           const int32_t* seg_ptr, const int32_t* seg_src,
                                           int64_t nnz, int lump, int out_f32, void* a_vals,
                                           void* m_vals, void* work, size_t ws_bytes, void* stream) {
  return fem_numeric_dispatch(ElemKind::TriaAniso, v, coords_f32, t, m, u1, u2, aniso_mat, n,
                              indptr, indices, seg_ptr, seg_src, nnz, lump, out_f32, a_vals, m_vals,
                              work, ws_bytes, stream);
}

extern "C" int lapy_fem_tet_numeric(const void* v, int coords_f32, const int32_t* t, int64_t m,
                                    int64_t n, const int32_t* indptr, const int32_t* indices,
                                    const int32_t* seg_ptr, const int32_t* seg_src, int64_t nnz,
                                    int lump, int out_f32, void* a_vals, void* m_vals, void* work,
                                    size_t ws_bytes, void* stream) {
  return fem_numeric_dispatch(ElemKind::Tet, v, coords_f32, t, m, nullptr, nullptr, nullptr, n,
                              indptr, indices, seg_ptr, seg_src, nnz, lump, out_f32, a_vals, m_vals,
                              work, ws_bytes, stream);
}

extern "C" int lapy_fem_batch_numeric(int npe, const void* v, int coords_f32, const int32_t* t, int64_t m,
                                      int nseg, const int32_t* seg_elem, int64_t n, const int32_t* indptr,
                                      const int32_t* indices, const int32_t* seg_ptr, const int32_t* seg_src,
                                      int64_t nnz, int lump, int out_f32, void* a_vals, void* m_vals, void* work,
                                      size_t ws_bytes, void* stream) {
  if ((npe != 3 && npe != 4) || nseg < 1 || !seg_elem) {
    lapy_set_last_message("fem_batch_numeric: npe must be 3 or 4, nseg >= 1 and seg_elem given");
    return LAPY_ERR_INVALID;
  }
  return fem_numeric_dispatch(npe == 4 ? ElemKind::Tet : ElemKind::Tria, v, coords_f32, t, m, nullptr, nullptr,
                              nullptr, n, indptr, indices, seg_ptr, seg_src, nnz, lump, out_f32, a_vals, m_vals,
                              work, ws_bytes, stream, nseg, seg_elem);
}
