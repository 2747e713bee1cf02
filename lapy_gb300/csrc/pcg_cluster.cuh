// On-chip refined PCG: one thread-block cluster per (segment, column group).
//
// A segment whose vectors and matrix fit into the shared memory and registers
// of at most 16 SMs is solved by one cluster from the FP64 right-hand side to
// the FP64 solution (FP32 iterations inside FP64 refinement) without a grid
// barrier, a host round trip or a pass over HBM per iteration.
#pragma once
#include "pcg.cuh"

namespace lapy {

// One CTA of a cluster: its rows, its 32-row units, its aggregates (two-level),
// the first of the columns its cluster solves and its copies of other CTAs' rows.
struct ClusterCta {
  int32_t row0, row1;
  int32_t unit0, unit1;
  int32_t agg0, agg1;
  int32_t seg, col0;
  int32_t nhalo;
};

// Clusters of one size: a launch.
struct ClusterClass {
  int cs = 1;        // CTAs per cluster
  int warps = 16;    // warps per CTA
  const void* kernel = nullptr;
  int cta0 = 0, ncta = 0;
  int slots = 0, halo = 0, units = 0, aggs = 0, ld = 0, push = 0;  // largest of the class
  int64_t elems = 0;
  bool z_halo = true;    // owners store z into the halo (else p, after one more barrier)
  bool mat_smem = true;  // matrix in shared memory (else read through L2)
  bool coarse_smem = true;  // rows of the coarse inverse likewise
  size_t smem = 0;
};

struct ClusterPlan {
  ClusterPlan() = default;
  ClusterPlan(const ClusterPlan&) = delete;
  ClusterPlan& operator=(const ClusterPlan&) = delete;
  ~ClusterPlan();
  // Plans of several cluster sizes launch them side by side: one stream and
  // one event each (owned by the plan), forked from and joined to the caller's
  // stream.
  std::vector<cudaStream_t> streams;
  std::vector<cudaEvent_t> events;
  bool ok = false;
  int p = 0;      // columns of the solve this plan was made for
  int np = 0;     // columns per cluster
  std::vector<ClusterClass> cls;
  const ClusterCta* cta = nullptr;      // device, ncta
  const int32_t* unit_row = nullptr;    // device, nunit + 1
  const int32_t* unit_agg = nullptr;    // device, nunit (global aggregate or -1)
  const int32_t* agg_unit = nullptr;    // device, 2 nagg: first unit and end of every aggregate
  const int32_t* slice_ptr = nullptr;   // device, nunit + 1
  const uint16_t* code = nullptr;       // device: slot of the column's row in the CTA (its own or a halo copy)
  const float* val = nullptr;           // device
  const float* diag = nullptr;          // device, 32 nunit
  const int32_t* push_ptr = nullptr;    // device, nunit + 1: halo copies to store, per unit of the owner
  const uint32_t* push = nullptr;       // device: slot | CTA of the cluster << 12 | halo row there << 16
};

// Plan the clusters for p columns and build the packed FP32 matrix into
// `mem`.  seg_agg / agg_rows (host; null: Jacobi): aggregates per segment, and
// the first row and the end of each.
// out->ok = false (and nothing else) when a segment does not fit on chip, its
// aggregates do not cover its rows one after the other, the copy does not fit
// into `bytes`, or a column lies outside its segment.
int cluster_plan(int64_t n, int64_t nnz, const int32_t* indptr, const int32_t* indices, const float* k32, int nseg,
                 const int32_t* seg_row, const int32_t* seg_agg, const int32_t* agg_rows, int p, void* mem,
                 size_t bytes, ClusterPlan* out, cudaStream_t stream);

struct ClusterSolve {
  int64_t n = 0;
  const int32_t* indptr = nullptr;
  const int32_t* indices = nullptr;
  const double* k64 = nullptr;
  const float* dinv = nullptr;
  const PcgPrecondDesc<float>* pc = nullptr;  // kind: Jacobi or two-level
  const double* B = nullptr;   // n x p
  double* X = nullptr;         // n x p
  double rtol = 0, inner_rtol = 0;
  int max_rounds = 0, maxiter = 0;
  int32_t* state = nullptr;    // nseg * p: LAPY_OK or a negative status
  double* relres2 = nullptr;   // nseg * p
  unsigned long long* ctl = nullptr;  // 8 words, cleared by the caller: iterations, rounds, row / entry / coarse-byte counts
};
int cluster_solve(const ClusterPlan& plan, const ClusterSolve& s, cudaStream_t stream);

}  // namespace lapy
