// Host interface of the resident PCG (resident.cu): a whole solve -- block
// Jacobi, every iteration, the reliable updates and the stopping rule -- in
// one cooperative launch, for operators that stay in L2 or shared memory.
#pragma once

#include "pcg_types.cuh"
#include "rowops.cuh"
#include "../../include/gfea.h"

namespace gfea {

struct ResidentOut {
  gfea_pcg_result res;
  int32_t timed_out;  // a wait ran out in some CTA: x holds the updates so far, 'res' is void
  int32_t pad;
};

// One solve.  The scratch is the multi-kernel PCG's workspace.
template <typename T>
struct ResidentProblem {
  SysT<T> S;
  const double* vals64;
  const double* b;
  double* x;          // known values and initial guess in, solution out
  T* p;               // packets of the search direction (2 Nn dof_n values)
  CoarseDev C;        // aggregation, A_c^-1 (Ac), accumulators (rcp: 3 nc doubles)
  T* ec;              // packets of the coarse correction (2 nc values)
  int coarse;         // two-level preconditioner
  double* box;        // packets of the partial sums (zero at launch)
  ResidentOut* out;   // zero at launch
  double rtol, delta2;
  int max_iters, max_upd;
};

// Two sets of four values' packets from every CTA to every CTA.
constexpr size_t kResidentBox = (size_t)2 * 4 * 152 * 152 * 16;

// Grid and shared memory of a solve.
struct ResidentGeom {
  int grid;        // CTAs (one per SM at most)
  int npc;         // nodes per CTA
  int lanes;       // lanes per node of the FP32 SpMV
  size_t smem;
};

// Geometry for an operator of dof_n components per node, with at most
// 'sms' CTAs; false when the CTAs' vectors do not fit in shared memory.
template <typename T>
bool resident_geom(int D, int64_t Nn, int64_t n_pairs, int nc, int n_agg, int sms, ResidentGeom* g);

// GFEA_OK, an error, or kResidentRefused: the grid does not fit on the SMs this
// context has (nothing was launched).
constexpr int kResidentRefused = -1;
template <typename T>
int resident_launch(int D, const ResidentProblem<T>& P, const ResidentGeom& g, cudaStream_t st);

}  // namespace gfea
