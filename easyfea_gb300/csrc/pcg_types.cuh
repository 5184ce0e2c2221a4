// Records shared by the PCG's translation units: the coarse level of the
// two-level preconditioner and its warp-level restriction.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace gfea {

// Regularisation of a coarse matrix R^T K R, relative to its largest diagonal
// entry: one at most zero_tol is replaced by the largest (empty or fully
// constrained unknowns), the others are shifted (rotations of degenerate
// aggregates).  FP32 values: their rounding reaches the 1e-6 level in nearly
// degenerate modes.  FP64: 1e-8 keeps those modes well above the float-float
// rounding of the inversion (~1e-12 of the largest entry, times the growth
// over the pivot blocks); at 1e-10 the inverse of a 64-aggregate HEXA8 bar
// comes out indefinite, also with its pivot blocks in FP64.  Iterations are
// the same with either.
struct CoarseReg {
  double zero_tol, shift;
};
inline CoarseReg coarse_reg(bool f32) { return f32 ? CoarseReg{1e-6, 1e-6} : CoarseReg{1e-14, 1e-8}; }

inline int coarse_nr(int D) { return D == 1 ? 1 : (D == 2 ? 3 : 6); }

// Aggregation kept at the start of the coarse workspace, so that a later
// solve on the same mesh can reuse it.
struct CoarseHdr {
  int32_t n_agg, nc, nr, valid;
  int64_t Nn;
};

// The restriction's FP64 atomics go to kRcCopies copies of the coarse vector
// (block b adds into copy b % kRcCopies): one copy held them all on a few L2
// slices, where they serialised.  Below kRcCopyMinNodes nodes the atomics
// are few and an iteration is launch-latency bound: one copy (rc itself,
// cleared by the coarse solve) and no summing launch.
constexpr int kRcCopies = 16;
constexpr int64_t kRcCopyMinNodes = 100000;

struct CoarseDev {
  int nr = 0, n_agg = 0, nc = 0;
  int ncopies = 1;         // 1: restriction into rc; kRcCopies: into rcp, summed by rc_sum_kernel
  CoarseHdr* hdr = nullptr;
  int32_t* agg = nullptr;  // node -> aggregate
  float4* off = nullptr;   // node offset from its cell centre / largest cell size
  double* Ac = nullptr;    // nc x nc, inverted in place
  // working storage of the inversion: float-float pairs (hi, lo)
  float* Ahi = nullptr;    // nc x nc (batched inversion)
  float* Alo = nullptr;
  float* rowph = nullptr;  // kGJB x nc: row panel of the pivot block
  float* rowpl = nullptr;
  float* colph = nullptr;  // nc x kGJB: column panel of the pivot block
  float* colpl = nullptr;
  float* pinvh = nullptr;  // kGJB x kGJB: inverse of the pivot block
  float* pinvl = nullptr;
  double* rc = nullptr;    // nc: restriction R^T r (summed from the copies)
  double* rcp = nullptr;   // kRcCopies x nc: restriction accumulators, one per group of blocks
  double* ec = nullptr;    // nc: coarse correction
  float* ecf = nullptr;    // nc: its FP32 copy (read by the FP32 prolongation)
};

// rc += the values v of the warp's nodes (lane = node, aggregate g, -1: no
// node): lanes of a run of equal aggregates are summed by a segmented scan,
// one FP64 atomic per run and mode.
template <int nr, typename T>
__device__ __forceinline__ void restrict_add(double* rc, int g, T (&v)[nr]) {
  const int lane = threadIdx.x & 31;
  const int gp = __shfl_up_sync(0xffffffffu, g, 1);
  const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || g != gp);
  const int start = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));  // first lane of this lane's run
  const int gn = __shfl_down_sync(0xffffffffu, g, 1);
  const bool tail = lane == 31 || gn != g;
#pragma unroll
  for (int m = 0; m < nr; ++m) {
    T s = v[m];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const T t = __shfl_up_sync(0xffffffffu, s, d);
      if (lane - d >= start) s += t;
    }
    if (tail && g >= 0 && s != 0) atomicAdd(&rc[g * nr + m], (double)s);
  }
}

}  // namespace gfea
