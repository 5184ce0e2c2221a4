// Inverse of the two-level preconditioner's SPD coarse matrix, a launch per
// pivot block.
//
// In-place blocked Gauss-Jordan (no pivoting: every pivot block of an SPD
// matrix is SPD) on float-float pairs.  For the pivot block K of B =
// [[B_KK, B_KJ], [B_IK, B_IJ]], with P = B_KK^-1:
//   B_KK <- P,  B_KJ <- P B_KJ,  B_IK <- -B_IK P,  B_IJ <- B_IJ - B_IK P B_KJ.
// A CTA owns one tile of B.  A step reads only the raw rows B_K* (16 x n,
// published by the tiles that own them at the end of the step before): the
// columns B_*K are the same numbers, B_iK = B_Ki^T for rows not yet eliminated
// and -B_Ki^T for those that are.  So a step is one launch: the pivot block's
// inverse (by every CTA), P B_KJ for the tile's columns and the rank-16 update
// of the tile.  Nothing waits on another CTA: any number of SMs does, and no
// wait can run out.  Each launch is a programmatic dependent of the one before,
// which hides part of the gap between them.
//
// The trailing updates run on pairs; P and P B_KJ are FP64 (pairs there lost up
// to two decades against an inverse in extended precision where aggregates
// have one or two nodes: 384 unknowns of HEXA8, relative error 2.2e-2 instead
// of 8e-5).
//
// Bound: latency -- per step the launch (~2 us), the panel's and the tile's
// trips through L2, the 16 dependent pivots -- and for n > 1000 the FP32 pipe
// (13 operations a product).  Two launches per pivot block with the block's
// inverse in FP64 by every block -> this (all steps in one cooperative launch
// with the tiles kept in shared memory): n = 33 0.10 -> 0.06 ms (0.06), 192
// 0.45 -> 0.15 (0.14), 612 1.80 -> 0.75 (0.62), 1152 3.76 -> 2.32 (1.79).
#include <math.h>

#include <algorithm>

#include "common.cuh"
#include "ff.cuh"
#include "inverse.cuh"

namespace gfea {
namespace {

constexpr int kB = 16;        // pivot block
constexpr int kIT = 256;      // threads per CTA
constexpr size_t kSmemMax = 216 * 1024;  // dynamic shared memory
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

// The largest diagonal entry (non-negative doubles order like their bits).
__device__ double largest_diagonal(const double* __restrict__ A, int n) {
  __shared__ unsigned long long s_max[kIT / 32];
  unsigned long long m = 0;
  for (int i = threadIdx.x; i < n; i += kIT)
    m = max(m, (unsigned long long)__double_as_longlong(fabs(A[(int64_t)i * n + i])));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (threadIdx.x % 32 == 0) s_max[threadIdx.x / 32] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kIT / 32; ++w) m = max(m, s_max[w]);
  return m > 0 ? __longlong_as_double((long long)m) : 1.0;
}

// Entry (i, j) of the regularised matrix, beyond n the identity: a unit
// diagonal (the largest entry) for empty or fully constrained coarse unknowns,
// a relative shift elsewhere (rotations of degenerate aggregates).
__device__ __forceinline__ double regularised(const double* __restrict__ A, int n, int i, int j, double dmax,
                                              double zero_tol, double shift) {
  if (i >= n || j >= n) return i == j ? 1.0 : 0.0;
  const double v = A[(int64_t)i * n + j];
  return i != j ? v : (v > zero_tol * dmax ? v + shift * dmax : dmax);
}

// Ahead of the steps: the largest diagonal entry and the raw rows of the first
// pivot block.
__global__ void __launch_bounds__(kIT) coarse_inverse_start_kernel(const double* __restrict__ A, int n,
                                                                   float2* rows, double* scale, double zero_tol,
                                                                   double shift) {
  const double dmax = largest_diagonal(A, n);
  if (blockIdx.x == 0 && threadIdx.x == 0) *scale = dmax;
  const int j = blockIdx.x * kIT + threadIdx.x;
  if (j < n)
#pragma unroll
    for (int l = 0; l < kB; ++l)
      if (l < n) rows[(int64_t)l * n + j] = ff_pair(regularised(A, n, l, j, dmax, zero_tol, shift));
}

// Steps [first, last) of the inversion.  Between two launches A holds the
// tile's pairs in the place of its doubles.
__global__ void __launch_bounds__(kIT) coarse_inverse_kernel(double* A, int n, Tile T, float2* rows0,
                                                             float2* rows1, const double* scale, int first, int last,
                                                             double zero_tol, double shift) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double D[2][kB][kB + 1];
  float2* B = reinterpret_cast<float2*>(smem);                  // rows x cols
  double* RJ = reinterpret_cast<double*>(B + T.rows * T.cols);  // kB x cols: raw rows at the tile's columns
  float2* RI = reinterpret_cast<float2*>(RJ + kB * T.cols);     // rows x kB: at the tile's rows (transposed, signed)
  float2(*M)[kB][kB + 1] = reinterpret_cast<float2(*)[kB][kB + 1]>(RI + kB * T.rows);
  float2* PR = RI + kB * T.rows + 2 * kB * (kB + 1);            // kB x cols
  float2* A2 = reinterpret_cast<float2*>(A);
  cudaGridDependencySynchronize();            // the step before is complete
  cudaTriggerProgrammaticLaunchCompletion();  // the next one may take its place on the SMs
  const int tid = threadIdx.x;
  const int i0 = (int)(blockIdx.x / T.gc) * T.rows, j0 = (int)(blockIdx.x % T.gc) * T.cols;
  float2* rows[2] = {rows0, rows1};  // of an even and an odd block
  const double dmax = first > 0 ? 0.0 : (scale ? *scale : largest_diagonal(A, n));
  for (int e = tid; e < T.rows * T.cols; e += kIT) {
    const int i = i0 + e / T.cols, j = j0 + e % T.cols;
    if (first == 0)
      B[e] = ff_pair(regularised(A, n, i, j, dmax, zero_tol, shift));
    else
      B[e] = i < n && j < n ? A2[(int64_t)i * n + j] : make_float2(i == j ? 1.f : 0.f, 0.f);
  }
  // raw rows of block k at the tile's columns, for every tile that holds them
  auto publish = [&](int k) {
    const int k0 = k * kB;
    if (k0 < i0 || k0 >= i0 + T.rows) return;
    for (int e = tid; e < kB * T.cols; e += kIT) {
      const int l = e / T.cols, j = j0 + e % T.cols;
      if (j < n) rows[k & 1][(int64_t)l * n + j] = B[(k0 - i0 + l) * T.cols + e % T.cols];
    }
  };
  const int steps = (n + kB - 1) / kB;
  __syncthreads();
  if (first == 0 && !scale) publish(0);
  __syncthreads();
  for (int k = first; k < last; ++k) {
    const int k0 = k * kB;
    const float2* rk = rows[k & 1];
    auto raw = [&](int l, int j) {  // B[k0 + l][j]
      return j < n && k0 + l < n ? __ldcg(rk + (int64_t)l * n + j) : make_float2(k0 + l == j ? 1.f : 0.f, 0.f);
    };
    const int pi = tid / kB, pj = tid % kB;  // the thread's element of the pivot block
    const float2 own = raw(pi, k0 + pj);
    M[0][pi][pj] = own;
    for (int e = tid; e < kB * T.cols; e += kIT) {
      const float2 v = raw(e / T.cols, j0 + e % T.cols);
      RJ[e] = (double)v.x + (double)v.y;
    }
    for (int r0 = 0; r0 < T.rows; r0 += 64) {  // 64 rows, a quarter of the block's columns a thread
      const int r = r0 + tid % 64, i = i0 + r, l0 = tid / 64 * 4;
      if (r >= T.rows) continue;
      float2 v[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) v[l] = raw(l0 + l, i);
      const float sg = i < k0 ? -1.f : 1.f;
      float4* q = reinterpret_cast<float4*>(RI + r * kB + l0);
      q[0] = make_float4(sg * v[0].x, sg * v[0].y, sg * v[1].x, sg * v[1].y);
      q[1] = make_float4(sg * v[2].x, sg * v[2].y, sg * v[3].x, sg * v[3].y);
    }
    __syncthreads();
    // P: Gauss-Jordan of the pivot block, one element per thread
#pragma unroll 1
    for (int p = 0; p < kB; ++p) {
      const float2(*S)[kB + 1] = M[p & 1];
      const float2 r = ff_recip(S[p][p]);
      const float2 row = pj == p ? r : ff_mul(S[p][pj], r);  // row p of the new state
      float2 v = row;
      if (pi != p) {
        const float2 c = ff_mul(S[pi][p], row);
        const float2 b = pj == p ? make_float2(0.f, 0.f) : S[pi][pj];
        ff_sub(b.x, b.y, c.x, c.y, v.x, v.y);
      }
      M[(p + 1) & 1][pi][pj] = v;
      __syncthreads();
    }
    static_assert(kB % 2 == 0 && kIT == kB * kB, "P ends in M[0], one element per thread");
    // the pairs lose the block's condition number; one step
    // P <- P + P (I - B_KK P) with the residual in FP64 restores it to FP64
    // (its product with P needs few digits while the residual is below 1e-8,
    // whose square and whose 2^-24 are lost on P).  A block too
    // ill-conditioned for that (rotations of one- or two-node aggregates leave
    // pivots at the level of the shift) is inverted in FP64, ~15 us slower.
    // P stays in FP64 for P B_KJ.
    const float2 pp = M[0][pi][pj];
    const double p64 = (double)pp.x + (double)pp.y;
    D[0][pi][pj] = (double)own.x + (double)own.y;
    D[1][pi][pj] = p64;
    __syncthreads();
    double e = pi == pj ? 1.0 : 0.0;
#pragma unroll
    for (int q = 0; q < kB; ++q) e -= D[0][pi][q] * D[1][q][pj];
    M[1][pi][pj].x = (float)e;
    if (!__syncthreads_or(!(fabs(e) <= kIllResidual))) {
      float c = 0.f;
#pragma unroll
      for (int q = 0; q < kB; ++q) c += M[0][pi][q].x * M[1][q][pj].x;
      D[0][pi][pj] = p64 + (double)c;
    } else {
#pragma unroll 1
      for (int p = 0; p < kB; ++p) {
        const double(*S)[kB + 1] = D[p & 1];
        const double r = 1.0 / S[p][p];
        const double row = pj == p ? r : S[p][pj] * r;
        D[(p + 1) & 1][pi][pj] = pi == p ? row : (pj == p ? 0.0 : S[pi][pj]) - S[pi][p] * row;
        __syncthreads();
      }
    }
    __syncthreads();
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
        constexpr int R = 2;  // rows at once: each row is one chain of additions
        for (int r0 = g; r0 < T.rows; r0 += R * groups) {
          float sh[R], sl[R];
          int r[R];
#pragma unroll
          for (int m = 0; m < R; ++m) {
            r[m] = r0 + m * groups < T.rows ? r0 + m * groups : r0;
            sh[m] = sl[m] = 0.f;
          }
#pragma unroll
          for (int l = 0; l < kB; l += 2)
#pragma unroll
            for (int m = 0; m < R; ++m) {
              const float4 q = reinterpret_cast<const float4*>(RI + r[m] * kB)[l / 2];
              ff_fma_acc(sh[m], sl[m], q.x, q.y, pr[l].x, pr[l].y);
              ff_fma_acc(sh[m], sl[m], q.z, q.w, pr[l + 1].x, pr[l + 1].y);
            }
          float2 v[R];
#pragma unroll
          for (int m = 0; m < R; ++m) {
            const int i = i0 + r[m];
            const float2 b = jk ? make_float2(0.f, 0.f) : B[r[m] * T.cols + c];
            ff_sub(b.x, b.y, sh[m], sl[m], v[m].x, v[m].y);
            if (i >= k0 && i < k0 + kB) v[m] = PR[(i - k0) * T.cols + c];
          }
#pragma unroll
          for (int m = 0; m < R; ++m) B[r[m] * T.cols + c] = v[m];
        }
      }
    }
    __syncthreads();
    if (k + 1 < steps) publish(k + 1);
    __syncthreads();  // a launch of several steps has one CTA: it reads its own rows
  }
  for (int e = tid; e < T.rows * T.cols; e += kIT) {
    const int i = i0 + e / T.cols, j = j0 + e % T.cols;
    if (i >= n || j >= n) continue;
    if (last == steps)
      A[(int64_t)i * n + j] = (double)B[e].x + (double)B[e].y;
    else
      A2[(int64_t)i * n + j] = B[e];
  }
}

}  // namespace

// Tile of an inversion of 'panels' pivot blocks on 'sms' SMs, one CTA each:
// the least work per step (cycles: 1.6 an entry of the tile, 128 a column for
// P B_KJ at two FP64 products a cycle, 6 a row or column loaded, 6000 for the
// rest).  Narrow tiles save FP64 work: 612 unknowns in 64 x 64 tiles took 0.90
// ms, in 208 x 16 ones 0.82.  Up to 48 unknowns one CTA does all steps in one
// launch.
static Tile pick_tile(int panels, int sms) {
  Tile best{panels * kB, panels * kB, 1};
  if (panels <= 3) return best;
  double cost = 1e300;
  for (int a = 1; a <= panels; ++a)
    for (int b = 1; b <= panels; ++b) {
      const Tile t{a * kB, b * kB, (int)ceil_div(panels, b)};
      if (t.cols > kIT || tile_smem(t) > kSmemMax) continue;
      const double waves = (double)ceil_div(ceil_div(panels, a) * t.gc, sms);
      const double c = waves * (1.6 * t.rows * t.cols + 128.0 * t.cols + 6.0 * (t.rows + t.cols) + 6000);
      if (c < cost) {
        cost = c;
        best = t;
      }
    }
  return best;
}

int coarse_inverse(const CoarseDev& C, double zero_tol, double shift, cudaStream_t st) {
  const int n = C.nc, panels = (int)ceil_div(n, kB);
  const Tile t = pick_tile(panels, kSMs);
  const int grid = (int)ceil_div(panels * kB, t.rows) * t.gc;
  const size_t smem = tile_smem(t);
  GFEA_CUDA_TRY(allow_smem(coarse_inverse_kernel, kSmemMax));
  // the published rows: pairs over (rowph, rowpl) for even blocks, (colph, colpl) for odd ones
  float2 *rows0 = reinterpret_cast<float2*>(C.rowph), *rows1 = reinterpret_cast<float2*>(C.colph);
  double* scale = grid > 1 ? reinterpret_cast<double*>(C.pinvh) : nullptr;
  if (scale) {
    coarse_inverse_start_kernel<<<(int)ceil_div(n, kIT), kIT, 0, st>>>(C.Ac, n, rows0, scale, zero_tol, shift);
    GFEA_LAUNCH_CHECK();
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kIT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = scale ? 1 : 0;
  const int each = scale ? 1 : panels;  // one CTA takes every step in one launch
  for (int k = 0; k < panels; k += each) {
    GFEA_CUDA_TRY(cudaLaunchKernelEx(&cfg, coarse_inverse_kernel, C.Ac, n, t, rows0, rows1, (const double*)scale, k,
                                     k + each, zero_tol, shift));
    GFEA_LAUNCH_CHECK();
  }
  return GFEA_OK;
}

}  // namespace gfea
