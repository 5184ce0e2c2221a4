// Inverse of the two-level preconditioner's SPD coarse matrix in one
// cooperative launch.
//
// In-place blocked Gauss-Jordan (no pivoting: every pivot block of an SPD
// matrix is SPD) on float-float pairs.  For the pivot block K of B =
// [[B_KK, B_KJ], [B_IK, B_IJ]], with P = B_KK^-1:
//   B_KK <- P,  B_KJ <- P B_KJ,  B_IK <- -B_IK P,  B_IJ <- B_IJ - B_IK P B_KJ.
// Every CTA keeps one tile of B in shared memory for the whole inversion.  A
// step reads only the raw rows B_K* (16 x n, published by the tiles that own
// them at the end of the step before): the columns B_*K are the same numbers,
// B_iK = B_Ki^T for rows not yet eliminated and -B_Ki^T for those that are.
// So a step is one barrier, the pivot block's inverse (by every CTA), P B_KJ
// for the tile's columns and the rank-16 update of the tile.
//
// The trailing updates run on pairs; P and P B_KJ are FP64, as in the two
// launches per pivot block this replaces (pairs there lost up to two decades
// against an inverse in extended precision where aggregates have one or two
// nodes: 384 unknowns of HEXA8, relative error 2.2e-2 instead of 8e-5).
//
// Bound: latency -- per step a barrier (~2 us), the panel's trip through L2,
// the 16 dependent pivots -- and for n > 1000 the FP32 pipe (13 operations a
// product).  The two launches took ~40 us a pair, most of it the pivot block's
// inverse, which every block repeated on the FP64 pipe.  Before -> now:
// n = 33 0.10 -> 0.06 ms, 192 0.45 -> 0.13, 612 1.80 -> 0.75, 1152 3.76 -> 2.50.
#include <math.h>

#include <algorithm>

#include "common.cuh"
#include "ff.cuh"
#include "inverse.cuh"
#include "stage.cuh"

namespace gfea {
namespace {

constexpr int kB = 16;        // pivot block
constexpr int kIT = 256;      // threads per CTA
constexpr int kTileMax = 128; // rows and columns of a tile
constexpr double kIllResidual = 1e-8;  // of a pivot block inverted in pairs

struct Tile {
  int rows, cols;  // tile size (multiples of kB)
  int gc;          // tiles per row of tiles
};

// Shared memory: tile (hi, lo), raw rows for the tile's columns and rows,
// pivot block (two states), P B_KJ.
__host__ __device__ inline size_t tile_smem(const Tile& t) {
  static_assert(sizeof(float2) == sizeof(double), "a pair and a double take the same room");
  return sizeof(float2) * ((size_t)t.rows * t.cols + (size_t)kB * (t.cols + t.rows) + 2 * kB * (kB + 1) +
                           (size_t)kB * t.cols);
}

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// All CTAs have arrived (bounded wait); their earlier writes are visible
// through ld.cg.
__device__ bool grid_barrier(uint32_t* bar, uint32_t target, int* ok) {
  if (gridDim.x == 1) {
    __syncthreads();
    return true;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    const uint64_t t0 = global_ns();
    bool good = true;
    for (uint32_t i = 1; (int32_t)(ld_acquire(bar) - target) < 0; ++i)
      if ((i & 255u) == 0 && global_ns() - t0 > kWaitLimitNs) {
        good = false;
        break;
      }
    *ok = good;
  }
  __syncthreads();
  return *ok != 0;
}

__global__ void __launch_bounds__(kIT, 1) coarse_inverse_kernel(double* __restrict__ A, int n, Tile T, float* h0,
                                                                float* l0, float* h1, float* l1, uint32_t* bar,
                                                                double zero_tol, double shift) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned long long s_max[kIT / 32];
  __shared__ int s_ok;
  __shared__ double D[2][kB][kB + 1];
  float2* B = reinterpret_cast<float2*>(smem);              // rows x cols
  double* RJ = reinterpret_cast<double*>(B + T.rows * T.cols);  // kB x cols: raw rows at the tile's columns
  float2* RI = reinterpret_cast<float2*>(RJ + kB * T.cols);     // rows x kB: at the tile's rows (transposed, signed)
  float2(*M)[kB][kB + 1] = reinterpret_cast<float2(*)[kB][kB + 1]>(RI + kB * T.rows);
  float2* PR = RI + kB * T.rows + 2 * kB * (kB + 1);        // kB x cols
  const int tid = threadIdx.x, lane = tid & 31;
  const int i0 = (blockIdx.x / T.gc) * T.rows, j0 = (blockIdx.x % T.gc) * T.cols;
  float *ph[2] = {h0, h1}, *pl[2] = {l0, l1};
  if (tid == 0) s_ok = 1;

  // largest diagonal entry: a unit diagonal for empty or fully constrained
  // coarse unknowns, a relative shift elsewhere (rotations of degenerate
  // aggregates)
  unsigned long long m = 0;  // non-negative doubles order like their bits
  for (int i = tid; i < n; i += kIT)
    m = max(m, (unsigned long long)__double_as_longlong(fabs(__ldcg(A + (int64_t)i * n + i))));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) s_max[tid / 32] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kIT / 32; ++w) m = max(m, s_max[w]);
  const double dmax = m > 0 ? __longlong_as_double((long long)m) : 1.0;

  // the tile; beyond n the identity
  for (int e = tid; e < T.rows * T.cols; e += kIT) {
    const int i = i0 + e / T.cols, j = j0 + e % T.cols;
    double v = i == j ? 1.0 : 0.0;
    if (i < n && j < n) {
      v = __ldcg(A + (int64_t)i * n + j);
      if (i == j) v = v > zero_tol * dmax ? v + shift * dmax : dmax;
    }
    ff_split(v, B[e].x, B[e].y);
  }
  __syncthreads();
  // raw rows of block k at the tile's columns, for every tile that holds them
  auto publish = [&](int k) {
    const int k0 = k * kB;
    if (k0 < i0 || k0 >= i0 + T.rows) return;
    for (int e = tid; e < kB * T.cols; e += kIT) {
      const int l = e / T.cols, j = j0 + e % T.cols;
      if (j < n) {
        const float2 v = B[(k0 - i0 + l) * T.cols + e % T.cols];
        __stcg(ph[k & 1] + (int64_t)l * n + j, v.x);
        __stcg(pl[k & 1] + (int64_t)l * n + j, v.y);
      }
    }
  };
  publish(0);
  const int steps = (n + kB - 1) / kB;
  uint32_t target = gridDim.x;
  bool ok = grid_barrier(bar, target, &s_ok);
  for (int k = 0; k < steps && ok; ++k) {
    const int k0 = k * kB;
    const float *rh = ph[k & 1], *rl = pl[k & 1];
    auto raw = [&](int l, int j) {  // B[k0 + l][j]
      return j < n ? make_float2(__ldcg(rh + (int64_t)l * n + j), __ldcg(rl + (int64_t)l * n + j))
                   : make_float2(k0 + l == j ? 1.f : 0.f, 0.f);
    };
    {
      const int l = tid / kB, c = tid % kB;
      M[0][l][c] = raw(l, k0 + c);
    }
    for (int e = tid; e < kB * T.cols; e += kIT) {
      const float2 v = raw(e / T.cols, j0 + e % T.cols);
      RJ[e] = (double)v.x + (double)v.y;
    }
    for (int e = tid; e < kB * T.rows; e += kIT) {
      const int l = e / T.rows, i = i0 + e % T.rows;
      float2 v = raw(l, i);
      if (i < k0) v = make_float2(-v.x, -v.y);
      RI[(e % T.rows) * kB + l] = v;
    }
    __syncthreads();
    // P: Gauss-Jordan of the pivot block, one element per thread
    {
      const int i = tid / kB, j = tid % kB;
#pragma unroll 1
      for (int p = 0; p < kB; ++p) {
        const float2(*S)[kB + 1] = M[p & 1];
        const float2 r = ff_recip(S[p][p]);
        const float2 pj = j == p ? r : ff_mul(S[p][j], r);  // row p of the new state
        float2 v = pj;
        if (i != p) {
          const float2 c = ff_mul(S[i][p], pj);
          const float2 b = j == p ? make_float2(0.f, 0.f) : S[i][j];
          ff_sub(b.x, b.y, c.x, c.y, v.x, v.y);
        }
        M[(p + 1) & 1][i][j] = v;
        __syncthreads();
      }
    }
    static_assert(kB % 2 == 0 && kIT == kB * kB, "P ends in M[0], one element per thread");
    // the pairs lose the block's condition number; one step
    // P <- P + P (I - B_KK P) with the residual in FP64 restores it to FP64
    // (its product with P needs few digits while the residual is below 1e-8,
    // whose square and whose 2^-24 are lost on P).  A block too
    // ill-conditioned for that (rotations of one- or two-node aggregates leave
    // pivots at the level of the shift) is inverted in FP64, ~15 us slower.
    // P stays in FP64 for P B_KJ.
    {
      const int i = tid / kB, j = tid % kB;
      const float2 b = raw(i, k0 + j), p0 = M[0][i][j];
      D[0][i][j] = (double)b.x + (double)b.y;
      const double p64 = (double)p0.x + (double)p0.y;
      D[1][i][j] = p64;
      __syncthreads();
      double e = i == j ? 1.0 : 0.0;
#pragma unroll
      for (int q = 0; q < kB; ++q) e -= D[0][i][q] * D[1][q][j];
      M[1][i][j].x = (float)e;
      if (!__syncthreads_or(!(fabs(e) <= kIllResidual))) {
        float c = 0.f;
#pragma unroll
        for (int q = 0; q < kB; ++q) c += M[0][i][q].x * M[1][q][j].x;
        D[0][i][j] = p64 + (double)c;
      } else {
#pragma unroll 1
        for (int p = 0; p < kB; ++p) {
          const double(*S)[kB + 1] = D[p & 1];
          const double r = 1.0 / S[p][p];
          const double pj = j == p ? r : S[p][j] * r;
          D[(p + 1) & 1][i][j] = i == p ? pj : (j == p ? 0.0 : S[i][j]) - S[i][p] * pj;
          __syncthreads();
        }
      }
      __syncthreads();
    }
    const double(*P)[kB + 1] = D[0];
    // P B_KJ (columns of the pivot block itself: P)
    for (int e = tid; e < kB * T.cols; e += kIT) {
      const int l = e / T.cols, c = e % T.cols, j = j0 + c;
      double t = 0;
      if (j >= k0 && j < k0 + kB) {
        t = P[l][j - k0];
      } else {
#pragma unroll
        for (int q = 0; q < kB; ++q) t += P[l][q] * RJ[q * T.cols + c];
      }
      ff_split(t, PR[e].x, PR[e].y);
    }
    __syncthreads();
    // the tile: a thread owns one column for a share of the rows
    {
      const int groups = kIT / T.cols, c = tid % T.cols, g = tid / T.cols;
      if (g < groups) {
        const bool jk = j0 + c >= k0 && j0 + c < k0 + kB;
        float2 pr[kB];
#pragma unroll
        for (int l = 0; l < kB; ++l) pr[l] = PR[l * T.cols + c];
        for (int r = g; r < T.rows; r += groups) {
          const int i = i0 + r;
          float2 v;
          if (i >= k0 && i < k0 + kB) {
            v = PR[(i - k0) * T.cols + c];
          } else {
            const float4* ci = reinterpret_cast<const float4*>(RI + r * kB);
            float sh = 0.f, sl = 0.f;
#pragma unroll
            for (int l = 0; l < kB; l += 2) {
              const float4 q = ci[l / 2];
              ff_fma_acc(sh, sl, q.x, q.y, pr[l].x, pr[l].y);
              ff_fma_acc(sh, sl, q.z, q.w, pr[l + 1].x, pr[l + 1].y);
            }
            const float2 b = jk ? make_float2(0.f, 0.f) : B[r * T.cols + c];
            ff_sub(b.x, b.y, sh, sl, v.x, v.y);
          }
          B[r * T.cols + c] = v;
        }
      }
    }
    if (k + 1 < steps) {
      __syncthreads();
      publish(k + 1);
      target += gridDim.x;
      ok = grid_barrier(bar, target, &s_ok);
    }
  }
  __syncthreads();
  for (int e = tid; e < T.rows * T.cols; e += kIT) {
    const int i = i0 + e / T.cols, j = j0 + e % T.cols;
    // a wait that ran out must not leave a plausible inverse
    if (i < n && j < n) A[(int64_t)i * n + j] = ok ? (double)B[e].x + (double)B[e].y : (double)NAN;
  }
}

}  // namespace

// The smallest tiles (most CTAs) whose grid fits on the SMs, one CTA each.
// Up to 48 unknowns one CTA saves the barriers.
int coarse_inverse(const CoarseDev& C, double zero_tol, double shift, cudaStream_t st) {
  const int n = C.nc, panels = (int)ceil_div(n, kB);
  Tile best{0, 0, 0};
  int grid = 0;
  if (panels <= 3) {
    best = Tile{panels * kB, panels * kB, 1};
    grid = 1;
  } else {
    int area = 1 << 30;
    for (int a = 1; a * kB <= kTileMax; ++a)
      for (int b = 1; b * kB <= kTileMax; ++b) {
        const int gr = (int)ceil_div(panels, a), gc = (int)ceil_div(panels, b);
        if (gr * gc > kSMs) continue;
        // equal areas: the squarer tile (shorter panels to load)
        if (a * b < area || (a * b == area && a + b < (best.rows + best.cols) / kB)) {
          area = a * b;
          best = Tile{a * kB, b * kB, gc};
          grid = gr * gc;
        }
      }
    if (grid == 0) return GFEA_ERR_ARG;
  }
  const size_t smem = tile_smem(best);
  GFEA_CUDA_TRY(allow_smem(coarse_inverse_kernel, tile_smem(Tile{kTileMax, kTileMax, 1})));
  uint32_t* bar = reinterpret_cast<uint32_t*>(C.pinvh);
  GFEA_CUDA_TRY(cudaMemsetAsync(bar, 0, sizeof(uint32_t), st));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kIT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = grid > 1 ? 1 : 0;
  GFEA_CUDA_TRY(cudaLaunchKernelEx(&cfg, coarse_inverse_kernel, C.Ac, n, best, C.rowph, C.rowpl, C.colph, C.colpl,
                                   bar, zero_tol, shift));
  GFEA_LAUNCH_CHECK();
  return GFEA_OK;
}

}  // namespace gfea
