// Cluster-resident batched PCG: many independent systems in one persistent launch.
//
// Each thread-block cluster (kCL CTAs) takes one system at a time from a work
// counter and runs its whole solve without returning to the host: the node
// loops are spread over the cluster's CTAs, every reduction is a block
// reduction followed by one hardware cluster barrier and a fixed-order sum of
// the kCL block partials read through distributed shared memory (so every
// thread of the cluster obtains the same value, control flow stays uniform,
// and a system's result does not depend on which other systems share the
// launch).  Iterations are FP32 (values, vectors, block-Jacobi) with FP64 dot
// products, scalars and reliable-update residuals, or FP64 throughout.
//
// The phases of an iteration are bound by chains of L2 round trips (8 or 16
// warps per SM), so each batches the loads of several rows, nodes or
// neighbour passes before it uses the first.  32 random-material cantilevers
// of 2000 to 50000 unknowns, mixed precision, assembly included: 26.8 ms with
// one neighbour pass and one node at a time and 256 threads throughout, 23.9
// with the batched loads, 16.8 with the wide clusters; 64 of 3000 unknowns
// 9.2 -> 7.3 ms, 256 of 2000 to 200000 (10.9 million in all) 276 -> 228 ms, the
// 256 random-material cantilevers of the benchmark (13.3 million) 351 -> 285.
//
// Cross-CTA reads of vectors written inside the launch use L2-only loads
// (ld.global.cg), so no stale L1 line is ever consulted; the cluster barrier
// orders the writes (release/acquire at cluster scope).

#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>
#include <vector>

#include "coarse.cuh"
#include "common.cuh"
#include "rowops.cuh"

namespace cg = cooperative_groups;

namespace gfea {
namespace {

constexpr int kCL = 8;    // CTAs per cluster (portable cluster size)

// Threads per CTA: 256 (two CTAs per SM), or 512 (one) for systems of at least
// kWideValues stored values where they are the tail of their batch.  A
// cluster's passes over its rows are bound by L2 latency at either width, so
// twice the warps shorten a solve (24021 QUAD4 nodes: 19.0 -> 14.4 ms, 5425:
// 5.4 -> 4.8 ms), but 8 whole SMs a cluster leave SMs unused and small systems
// wait on barriers.  2000 to 50000 unknowns, 32 systems: 22.0 ms narrow, 16.2
// wide; to 60000, 40 systems: 29.7 and 20.3, 100 systems: 40.0 and 43.2; 64 of
// 3000: 7.3 and 13.3; 256 of 2000 to 200000 (10.9 million): 228 and 280.  So:
// wide where the largest system is over twice its share of the batch (the time
// of the batch on all narrow clusters).
//
// Both widths divide a system among the same kCL * 512 virtual threads, of
// which a thread of the narrow one is two (VT, kWide / VT apart), and sum
// their partials in the same order: a system's result is the same to the bit
// at either width, so it does not depend on the others in the launch.
constexpr int kNarrow = 256, kWide = 512;
constexpr int64_t kWideValues = 400000;

__host__ __device__ inline int64_t stored_values(const gfea_batch_instance& I) { return I.n_pairs * I.dof_n * I.dof_n; }

size_t a256(size_t b) { return (b + 255) & ~size_t(255); }

template <typename T>
struct BatchBuf {
  T *r, *z, *pa, *pb, *Ap, *dinv, *dx;
  double* r64;
};

template <typename T>
__host__ __device__ size_t batch_layout(int64_t Nn, int D, BatchBuf<T>* w, char* base) {
  const size_t N = (size_t)Nn * D;
  size_t off = 0;
  auto take = [&](size_t bytes) -> char* {
    char* p = base ? base + off : nullptr;
    off += (bytes + 255) & ~size_t(255);
    return p;
  };
  BatchBuf<T> t;
  if (!w) w = &t;
  w->r = (T*)take(sizeof(T) * N);
  w->z = (T*)take(sizeof(T) * N);
  w->pa = (T*)take(sizeof(T) * N);
  w->pb = (T*)take(sizeof(T) * N);
  w->Ap = (T*)take(sizeof(T) * N);
  w->dinv = (T*)take(sizeof(T) * N * D);
  w->dx = (T*)take(sizeof(T) * N);
  w->r64 = (double*)take(sizeof(double) * N);
  return off;
}

template <typename T>
__device__ __forceinline__ T ldcg(const T* p) {
  return __ldcg(p);
}

struct Ctx {
  cg::cluster_group cl;
  unsigned rank;
  double* slots;  // this CTA's 2 x 4 reduction slots
  double* sh;     // warp partials, 4 values
  int phase;
};

// Cluster-wide sum of NV values (one per virtual thread); every thread of every
// CTA gets the same result.
// (c.sh is free again once the cluster barrier has been passed.)
template <int NV, int VT>
__device__ void csum(Ctx& c, const double (&v)[VT][NV], double (&out)[NV]) {
  constexpr int kWarps = kWide / 32;
  double* slot = c.slots + (c.phase & 1) * 4;
  const int wp = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int q = 0; q < VT; ++q) {
      double t = v[q][k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (l == 0) c.sh[k * kWarps + q * (kWarps / VT) + wp] = t;
    }
  __syncthreads();
  if (wp == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double t = l < kWarps ? c.sh[k * kWarps + l] : 0.0;
#pragma unroll
      for (int o = kWarps / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (l == 0) slot[k] = t;
    }
  }
  c.cl.sync();
#pragma unroll
  for (int k = 0; k < NV; ++k) out[k] = 0;
#pragma unroll
  for (unsigned r = 0; r < (unsigned)kCL; ++r) {
    const double* rs = c.cl.map_shared_rank(slot, r);
#pragma unroll
    for (int k = 0; k < NV; ++k) out[k] += rs[k];
  }
  ++c.phase;
}

// FP64 residual r64 = P(b - A64 x) over the cluster; partials r.r, ||P(b - A x_c)||^2,
// ||P(|A||x| + |b|)||^2 accumulated into v[0..2].
//
// The three products share one pass over the row, two rows at a time with the
// loads of kPasses neighbour passes in flight (bound by the chain of L2 round
// trips, as node_rows_multi below).
constexpr int kPasses = 3;

template <int D, int G, int VT>
__device__ __noinline__ void resid64(const SysT<double>& S, const double* b, const double* x, double* r64, int64_t grp,
                                     int64_t ngrp, int lane, double (&v)[VT][4]) {
  constexpr int LA = G - G % D;
  constexpr int NPP = LA / D;
  constexpr int R = D < 3 || VT == 2 ? 2 : 1;
  const int64_t Nn = S.Nn;
  const int64_t sub = grp % (32 / G);
  const int j = lane % D;
  for (int64_t a0 = grp - sub; a0 < Nn; a0 += (R / VT) * ngrp) {
    int64_t an[R];
    int32_t p0[R], nb[R];
    double all[R][D], kn[R][D], ab[R][D];
    int32_t maxnb = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      an[r] = a0 + sub + (r % VT) * (kWide / VT / G) + (r / VT) * ngrp;
      const int64_t ac = an[r] < Nn ? an[r] : Nn - 1;
      p0[r] = S.node_ptr[ac];
      nb[r] = S.node_ptr[ac + 1] - p0[r];
      maxnb = nb[r] > maxnb ? nb[r] : maxnb;
#pragma unroll
      for (int i = 0; i < D; ++i) all[r][i] = kn[r][i] = ab[r][i] = 0;
    }
    if (lane < LA) {
      for (int32_t k0 = lane / D, t0 = lane; k0 < maxnb; k0 += kPasses * NPP, t0 += kPasses * LA) {
        int32_t c[kPasses][R];
        double val[kPasses][R][D], xv[kPasses][R];
        bool known[kPasses][R];
#pragma unroll
        for (int u = 0; u < kPasses; ++u)
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int32_t k = k0 + u * NPP;
            const bool in = k < nb[r];
            c[u][r] = in ? __ldg(S.nbr + p0[r] + k) : -1;
#pragma unroll
            for (int i = 0; i < D; ++i)
              val[u][r][i] =
                  in ? __ldg(S.vals + (int64_t)D * D * p0[r] + (int64_t)i * D * nb[r] + t0 + u * LA) : 0.0;
          }
#pragma unroll
        for (int u = 0; u < kPasses; ++u)
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int64_t col = (int64_t)c[u][r] * D + j;
            xv[u][r] = c[u][r] >= 0 ? ldcg(x + col) : 0.0;
            known[u][r] = c[u][r] >= 0 ? S.known[col] : false;
          }
#pragma unroll
        for (int u = 0; u < kPasses; ++u)
#pragma unroll
          for (int r = 0; r < R; ++r)
#pragma unroll
            for (int i = 0; i < D; ++i) {
              all[r][i] += val[u][r][i] * xv[u][r];
              kn[r][i] += val[u][r][i] * (known[u][r] ? xv[u][r] : 0.0);
              ab[r][i] += fabs(val[u][r][i]) * fabs(xv[u][r]);
            }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int i = 0; i < D; ++i) {
        all[r][i] = group_sum<G, double>(all[r][i]);
        kn[r][i] = group_sum<G, double>(kn[r][i]);
        ab[r][i] = group_sum<G, double>(ab[r][i]);
      }
      if (an[r] < Nn && lane == 0) {
#pragma unroll
        for (int i = 0; i < D; ++i) {
          const int64_t dof = an[r] * D + i;
          const bool unk = !S.known[dof];
          const double bi = __ldg(b + dof);
          const double ri = unk ? bi - all[r][i] : 0.0;
          const double rci = unk ? bi - kn[r][i] : 0.0;
          const double ai = unk ? ab[r][i] + fabs(bi) : 0.0;
          r64[dof] = ri;
          v[r % VT][0] += ri * ri;
          v[r % VT][1] += rci * rci;
          v[r % VT][2] += ai * ai;
        }
      }
    }
  }
}

// r = (T) r64, z = D^-1 r (masked) for the nodes of this thread; partials r.z, r.r.
template <int D, typename T, int VT>
__device__ void restart_rz(const gfea_batch_instance& I, const BatchBuf<T>& w, int64_t gtid, int64_t nthr,
                           double (&v)[VT][2]) {
#pragma unroll
  for (int q = 0; q < VT; ++q)
    for (int64_t a = gtid + q * (kWide / VT); a < I.n_nodes; a += nthr) {
      T rl[D];
#pragma unroll
      for (int i = 0; i < D; ++i) {
        const int64_t dof = a * D + i;
        rl[i] = (T)ldcg(w.r64 + dof);
        w.r[dof] = rl[i];
      }
#pragma unroll
      for (int i = 0; i < D; ++i) {
        T zi = 0;
#pragma unroll
        for (int j = 0; j < D; ++j) zi += ldcg(w.dinv + a * D * D + i * D + j) * rl[j];
        if (I.known[a * D + i]) zi = 0;
        w.z[a * D + i] = zi;
        v[q][0] += (double)rl[i] * (double)zi;
        v[q][1] += (double)rl[i] * (double)rl[i];
      }
    }
}

// node_rows for R nodes at once (one G-lane group): the index, value and
// gathered-vector loads of the R rows in kPasses neighbour passes are
// independent and issued together.  A cluster runs 16 warps per SM, too few to
// hide the three dependent L2 round trips of a row (row pointer, neighbour
// index, gather) one row at a time; a QUAD4 or HEXA8 interior row has three
// passes, so it takes the three round trips once.  self: xf at the lane's own
// component of each row.
template <int D, int G, typename T, bool DIFF, int R, typename XF>
__device__ __forceinline__ void node_rows_multi(const int64_t (&a)[R], const int32_t (&p0)[R], const int32_t (&nb)[R],
                                                int lane, const SysT<T>& S, XF xf, T (&acc)[R][D], T (&self)[R]) {
  constexpr int LA = G - G % D;
  constexpr int NPP = LA / D;
  const int j = lane % D;
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int i = 0; i < D; ++i) acc[r][i] = 0;
  if (lane < LA) {
#pragma unroll
    for (int r = 0; r < R; ++r) self[r] = xf(a[r] * D + j);
    int32_t maxnb = nb[0];
#pragma unroll
    for (int r = 1; r < R; ++r) maxnb = nb[r] > maxnb ? nb[r] : maxnb;
    for (int32_t k0 = lane / D, t0 = lane; k0 < maxnb; k0 += kPasses * NPP, t0 += kPasses * LA) {
      int32_t c[kPasses][R];
      T v[kPasses][R][D], xv[kPasses][R];
#pragma unroll
      for (int u = 0; u < kPasses; ++u)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int32_t k = k0 + u * NPP;
          const bool in = k < nb[r];
          c[u][r] = in ? __ldg(S.nbr + p0[r] + k) : -1;
#pragma unroll
          for (int i = 0; i < D; ++i)
            v[u][r][i] =
                in ? __ldg(S.vals + (int64_t)D * D * p0[r] + (int64_t)i * D * nb[r] + t0 + u * LA) : (T)0;
        }
#pragma unroll
      for (int u = 0; u < kPasses; ++u)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const T x = c[u][r] >= 0 ? xf((int64_t)c[u][r] * D + j) : (T)0;
          xv[u][r] = DIFF && c[u][r] >= 0 ? x - self[r] : x;
        }
#pragma unroll
      for (int u = 0; u < kPasses; ++u)
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int i = 0; i < D; ++i) acc[r][i] += v[u][r][i] * xv[u][r];
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int i = 0; i < D; ++i) acc[r][i] = group_sum<G, T>(acc[r][i]);
}

// Coarse correction of the two-level preconditioner, cluster-wide:
// rc = R^T r (one warp per aggregate, its nodes in ascending order, fixed
// butterfly), ec = A_c^-1 rc (one warp per row; FP32 inverse for the FP32
// iteration).  Every thread of the cluster calls it; r must be written.
template <int D, typename T>
__device__ __noinline__ void coarse_correct(Ctx& c, const gfea_batch_instance& I, const T* r, int64_t gtid, int64_t nthr) {
  constexpr int nr = Modes<D>::nr;
  const gfea_coarse_level& L = I.coarse;
  const int lane = threadIdx.x & 31;
  const int64_t gw = gtid >> 5, nw = nthr >> 5;
  const float4* off = reinterpret_cast<const float4*>(L.off);
  c.cl.sync();  // r of every node written
  for (int64_t g = gw; g < L.n_agg; g += nw) {
    T v[nr];
#pragma unroll
    for (int m = 0; m < nr; ++m) v[m] = 0;
    const int32_t k1 = L.agg_ptr[g + 1];
    constexpr int B = D < 3 ? 4 : 2;  // nodes per lane with their loads in flight
    for (int32_t k = L.agg_ptr[g] + lane; k < k1; k += B * 32) {
      int64_t a[B];
      T ri[B][D];
      float4 o[B];
      uint8_t kn[B][D];
#pragma unroll
      for (int q = 0; q < B; ++q) a[q] = k + q * 32 < k1 ? L.agg_nodes[k + q * 32] : -1;
#pragma unroll
      for (int q = 0; q < B; ++q) {
        if (a[q] < 0) continue;
        o[q] = off[a[q]];
#pragma unroll
        for (int i = 0; i < D; ++i) {
          kn[q][i] = I.known[a[q] * D + i];
          ri[q][i] = ldcg(r + a[q] * D + i);
        }
      }
#pragma unroll
      for (int q = 0; q < B; ++q) {
        if (a[q] < 0) continue;
        T R[D][nr];
        node_modes<D, T>(o[q], kn[q], R);
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
          for (int m = 0; m < nr; ++m) v[m] += R[i][m] * ri[q][i];
      }
    }
#pragma unroll
    for (int m = 0; m < nr; ++m) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[m] += __shfl_xor_sync(0xffffffffu, v[m], o);
      if (lane == 0) L.rc[g * nr + m] = (double)v[m];
    }
  }
  c.cl.sync();  // rc complete
  const int nc = L.nc;
  constexpr int RG = 4;  // rows per warp with their loads in flight
  for (int64_t i0 = gw; i0 < nc; i0 += RG * nw) {
    int64_t row[RG];
    T acc[RG];
#pragma unroll
    for (int q = 0; q < RG; ++q) {
      row[q] = i0 + q * nw < nc ? i0 + q * nw : i0;
      acc[q] = 0;
    }
    constexpr int U = sizeof(T) == 4 ? 6 : 3;
    for (int j0 = lane; j0 < nc; j0 += 32 * U) {
      T rj[U], ij[U][RG];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int j = j0 + 32 * u;
        rj[u] = j < nc ? (T)ldcg(L.rc + j) : (T)0;
#pragma unroll
        for (int q = 0; q < RG; ++q)
          ij[u][q] = j >= nc ? (T)0
                             : (sizeof(T) == 4 ? (T)__ldg(L.inv32 + row[q] * nc + j) : (T)__ldg(L.inv + row[q] * nc + j));
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int q = 0; q < RG; ++q) acc[q] += ij[u][q] * rj[u];
    }
#pragma unroll
    for (int q = 0; q < RG; ++q) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
      if (lane == 0 && i0 + q * nw < nc) L.ec[i0 + q * nw] = (double)acc[q];
    }
  }
  c.cl.sync();  // ec complete
}

// z = D^-1 r + R ec[agg] (masked) for the nodes of this thread; partials r.z, r.r.
template <int D, typename T, int VT>
__device__ __noinline__ void z_two_level(const gfea_batch_instance& I, const BatchBuf<T>& w, int64_t gtid, int64_t nthr,
                                         double (&out)[VT][2]) {
  constexpr int nr = Modes<D>::nr;
  const gfea_coarse_level& L = I.coarse;
  const float4* off = reinterpret_cast<const float4*>(L.off);
  constexpr int B = D * sizeof(T) <= 8 ? 4 : (D * sizeof(T) <= 12 ? 2 : VT);  // nodes per thread with their loads in flight
  DotAcc<T> rz[VT], rr[VT];
  for (int64_t a0 = gtid; a0 < I.n_nodes; a0 += (B / VT) * nthr) {
    auto node = [&](int q) { return a0 + (q % VT) * (kWide / VT) + (q / VT) * nthr; };
    T rl[B][D], di[B][D][D], e[B][nr];
    float4 o[B];
    uint8_t kn[B][D];
    int g[B];
#pragma unroll
    for (int q = 0; q < B; ++q) {
      const int64_t a = node(q) < I.n_nodes ? node(q) : a0;
      g[q] = L.agg[a];
      o[q] = off[a];
#pragma unroll
      for (int i = 0; i < D; ++i) {
        rl[q][i] = ldcg(w.r + a * D + i);
        kn[q][i] = I.known[a * D + i];
#pragma unroll
        for (int j = 0; j < D; ++j) di[q][i][j] = ldcg(w.dinv + a * D * D + i * D + j);
      }
    }
#pragma unroll
    for (int q = 0; q < B; ++q)
#pragma unroll
      for (int m = 0; m < nr; ++m) e[q][m] = (T)ldcg(L.ec + g[q] * nr + m);
#pragma unroll
    for (int q = 0; q < B; ++q) {
      const int64_t a = node(q);
      if (a >= I.n_nodes) continue;
      T R[D][nr];
      node_modes<D, T>(o[q], kn[q], R);
#pragma unroll
      for (int i = 0; i < D; ++i) {
        T zi = 0;
#pragma unroll
        for (int j = 0; j < D; ++j) zi += di[q][i][j] * rl[q][j];
#pragma unroll
        for (int m = 0; m < nr; ++m) zi += R[i][m] * e[q][m];
        if (kn[q][i]) zi = 0;
        w.z[a * D + i] = zi;
        rz[q % VT].add_prod(rl[q][i], zi);
        rr[q % VT].add_prod(rl[q][i], rl[q][i]);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < VT; ++q) {
    out[q][0] = rz[q].value();
    out[q][1] = rr[q].value();
  }
}

// restart_rz with the coarse level: r = (T) r64, coarse correction, z.
template <int D, typename T, int VT>
__device__ void restart_rz_two_level(Ctx& c, const gfea_batch_instance& I, const BatchBuf<T>& w, int64_t gtid,
                                     int64_t nthr, double (&v)[VT][2]) {
  const int64_t rtid = (int64_t)c.rank * blockDim.x + threadIdx.x, rthr = (int64_t)kCL * blockDim.x;
  for (int64_t a = rtid; a < I.n_nodes; a += rthr)
#pragma unroll
    for (int i = 0; i < D; ++i) w.r[a * D + i] = (T)ldcg(w.r64 + a * D + i);
  coarse_correct<D, T>(c, I, w.r, rtid, rthr);
  z_two_level<D, T, VT>(I, w, gtid, nthr, v);
}

// Direction pb = z + beta pa and Ap = A pb (masked SpMV); the partials of
// pb.Ap.
template <int D, int G, typename T, bool DIFF, int VT>
__device__ __noinline__ void direction_apply(const SysT<T>& S, const T* z, const T* pa, T* pb, T* Ap, T beta,
                                             int64_t grp, int64_t ngrp, int lane, double (&out)[VT][1]) {
  const int64_t Nn = S.Nn;
  const int64_t sub = grp % (32 / G);
  DotAcc<T> pap[VT];
  constexpr int R = D * sizeof(T) <= 12 ? 4 : 2;  // rows per group per round
  // the row pointers of the next round are fetched during this one
  int32_t q0[R], q1[R];
  auto row = [&](int64_t a0, int r) { return a0 + sub + (r % VT) * (kWide / VT / G) + (r / VT) * ngrp; };
  auto fetch = [&](int64_t a0) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int64_t a = row(a0, r);
      const int64_t ac = a < Nn ? a : Nn - 1;
      q0[r] = __ldg(S.node_ptr + ac);
      q1[r] = __ldg(S.node_ptr + ac + 1);
    }
  };
  fetch(grp - sub);
  for (int64_t a0 = grp - sub; a0 < Nn; a0 += (R / VT) * ngrp) {
    int64_t an[R], ac[R];
    int32_t p0[R], nb[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      an[r] = row(a0, r);
      ac[r] = an[r] < Nn ? an[r] : Nn - 1;
      p0[r] = q0[r];
      nb[r] = q1[r] - q0[r];
    }
    fetch(a0 + (R / VT) * ngrp);
    uint8_t kn[R];
#pragma unroll
    for (int r = 0; r < R; ++r) kn[r] = S.known[ac[r] * D + lane % D];
    T acc[R][D], self[R];
    auto dir = [&](int64_t cc) { return ldcg(z + cc) + beta * ldcg(pa + cc); };
    node_rows_multi<D, G, T, DIFF, R>(ac, p0, nb, lane, S, dir, acc, self);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (an[r] < Nn && lane < D) {
        T av = acc[r][0];
#pragma unroll
        for (int i = 1; i < D; ++i)
          if (lane == i) av = acc[r][i];
        const int64_t dof = an[r] * D + lane;
        if (kn[r]) av = 0;
        pb[dof] = self[r];
        Ap[dof] = av;
        pap[r % VT].add_prod(self[r], av);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < VT; ++q) out[q][0] = pap[q].value();
}

template <int D, int G, typename T, int VT>
__device__ void solve_instance(Ctx& c, const gfea_batch_instance& I, double delta2) {
  const int64_t Nn = I.n_nodes;
  BatchBuf<T> w;
  batch_layout<T>(Nn, D, &w, static_cast<char*>(I.work));
  const T* vals = sizeof(T) == 4 ? reinterpret_cast<const T*>(I.vals32) : reinterpret_cast<const T*>(I.vals64);
  const SysT<T> S{Nn, I.node_ptr, I.nbr, vals, I.known, I.translation_invariant};
  const SysT<double> S64{Nn, I.node_ptr, I.nbr, I.vals64, I.known, 0};
  const int tid = threadIdx.x;
  // this thread's first virtual thread, and its real index (loops without sums)
  const int64_t gtid = (int64_t)c.rank * kWide + tid;
  const int64_t nthr = (int64_t)kCL * kWide;
  const int64_t rtid = (int64_t)c.rank * (kWide / VT) + tid;
  const int64_t rthr = (int64_t)kCL * (kWide / VT);
  const int lane = tid % G;
  const int64_t grp = gtid / G, ngrp = nthr / G;
  const double eps64 = 2.220446049250313e-16;
  const bool two_level = I.coarse.n_agg > 0;

  // block-Jacobi inverses (thread per node)
  double bad = 0;
  for (int64_t a = rtid; a < Nn; a += rthr) {
    const int32_t p0 = S.node_ptr[a], p1 = S.node_ptr[a + 1];
    int lo = p0, hi = p1;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (S.nbr[mid] < a) lo = mid + 1; else hi = mid;
    }
    const bool has = lo < p1 && S.nbr[lo] == a;
    const int32_t W = D * (p1 - p0);
    double M[D][D], iM[D][D];
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int j = 0; j < D; ++j) {
        double v = has ? (double)vals[(int64_t)D * D * p0 + (int64_t)i * W + D * (lo - p0) + j] : 0.0;
        if (S.known[a * D + i] || S.known[a * D + j]) v = (i == j) ? 1.0 : 0.0;
        M[i][j] = v;
      }
    const double det = det_inv<D>(M, iM);
    if (!(fabs(det) > 0) || !isfinite(det)) {
      bad += 1;
#pragma unroll
      for (int i = 0; i < D; ++i)
#pragma unroll
        for (int j = 0; j < D; ++j) iM[i][j] = (i == j) ? 1.0 : 0.0;
    }
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int j = 0; j < D; ++j) w.dinv[a * D * D + i * D + j] = (T)iM[i][j];
  }

  // FP64 residual of the start
  double v4[VT][4] = {}, o4[4];
  v4[0][3] = bad;
  resid64<D, G, VT>(S64, I.b, I.x, w.r64, grp, ngrp, lane, v4);
  csum<4, VT>(c, v4, o4);
  double rr_true = o4[0];
  const double bb = o4[1];
  double floor2 = (32 * eps64) * (32 * eps64) * o4[2];
  double tol2 = fmax(I.rtol * I.rtol * bb, floor2);
  int status = GFEA_ERR_NOT_CONVERGED, iters = 0, updates = 0;
  bool finished = false;
  if (o4[3] > 0) {
    status = GFEA_ERR_SINGULAR;
    finished = true;
  } else if (!isfinite(rr_true) || !(bb == bb)) {
    status = GFEA_ERR_NAN;
    finished = true;
  } else if (bb == 0) {  // b_i - A_ic x_c = 0: the unknowns are zero
    for (int64_t a = rtid; a < Nn; a += rthr)
#pragma unroll
      for (int i = 0; i < D; ++i)
        if (!I.known[a * D + i]) I.x[a * D + i] = 0.0;
    status = GFEA_OK;
    finished = true;
  } else if (rr_true <= tol2) {
    status = GFEA_OK;
    finished = true;
  }

  if (!finished) {
    // start: r = r64, dx = 0, p = 0, z = D^-1 r
    for (int64_t a = rtid; a < Nn; a += rthr)
#pragma unroll
      for (int i = 0; i < D; ++i) {
        w.dx[a * D + i] = 0;
        w.pa[a * D + i] = 0;
      }
    double v2[VT][2] = {}, o2[2];
    if (two_level)
      restart_rz_two_level<D, T, VT>(c, I, w, gtid, nthr, v2);
    else
      restart_rz<D, T, VT>(I, w, gtid, nthr, v2);
    csum<2, VT>(c, v2, o2);
    double rz = o2[0];
    double beta = 0;
    double trigger = fmax(delta2 * rr_true, 0.25 * tol2);
    double rr_best = rr_true;
    int stall = 0;
    T* pa = w.pa;
    T* pb = w.pb;
    const bool diff = sizeof(T) == 4 && S.diff;
    for (;;) {
      double va[VT][1], oa[1];
      if (diff)
        direction_apply<D, G, T, true, VT>(S, w.z, pa, pb, w.Ap, (T)beta, grp, ngrp, lane, va);
      else
        direction_apply<D, G, T, false, VT>(S, w.z, pa, pb, w.Ap, (T)beta, grp, ngrp, lane, va);
      csum<1, VT>(c, va, oa);
      const double pap = oa[0];
      if (!(pap > 0) || !isfinite(pap)) {
        status = isfinite(pap) ? GFEA_ERR_BREAKDOWN : GFEA_ERR_NAN;
        break;
      }
      const double alpha = rz / pap;
      // x, r, z update; partials r.z, r.r
      double vb[VT][2], ob[2];
      const T al = (T)alpha;
      if (two_level) {  // x, r; then the coarse correction; then z
        constexpr int B = 4;  // unknowns per thread with their loads in flight
        const int64_t N = Nn * D;
        for (int64_t d0 = rtid; d0 < N; d0 += B * rthr) {
          T xo[B], po[B], ro[B], ao[B];
#pragma unroll
          for (int q = 0; q < B; ++q) {
            const int64_t dof = d0 + q * rthr < N ? d0 + q * rthr : d0;
            xo[q] = ldcg(w.dx + dof);
            po[q] = ldcg(pb + dof);
            ro[q] = ldcg(w.r + dof);
            ao[q] = ldcg(w.Ap + dof);
          }
#pragma unroll
          for (int q = 0; q < B; ++q) {
            const int64_t dof = d0 + q * rthr;
            if (dof < N) {
              w.dx[dof] = xo[q] + al * po[q];
              w.r[dof] = ro[q] - al * ao[q];
            }
          }
        }
        coarse_correct<D, T>(c, I, w.r, rtid, rthr);
        z_two_level<D, T, VT>(I, w, gtid, nthr, vb);
      } else {
#pragma unroll
        for (int q = 0; q < VT; ++q) {
          DotAcc<T> rz_acc, rr_acc;
          for (int64_t a = gtid + q * (kWide / VT); a < Nn; a += nthr) {
            T rl[D];
#pragma unroll
            for (int i = 0; i < D; ++i) {
              const int64_t dof = a * D + i;
              w.dx[dof] = ldcg(w.dx + dof) + al * ldcg(pb + dof);
              rl[i] = ldcg(w.r + dof) - al * ldcg(w.Ap + dof);
              w.r[dof] = rl[i];
            }
#pragma unroll
            for (int i = 0; i < D; ++i) {
              T zi = 0;
#pragma unroll
              for (int j = 0; j < D; ++j) zi += ldcg(w.dinv + a * D * D + i * D + j) * rl[j];
              if (I.known[a * D + i]) zi = 0;
              w.z[a * D + i] = zi;
              rz_acc.add_prod(rl[i], zi);
              rr_acc.add_prod(rl[i], rl[i]);
            }
          }
          vb[q][0] = rz_acc.value();
          vb[q][1] = rr_acc.value();
        }
      }
      csum<2, VT>(c, vb, ob);
      beta = ob[0] / rz;
      rz = ob[0];
      const double rr_it = ob[1];
      ++iters;
      T* t = pa;
      pa = pb;
      pb = t;
      if (!isfinite(rr_it)) {
        status = GFEA_ERR_NAN;
        break;
      }
      if (rr_it > trigger && iters < I.max_iters) continue;
      // reliable update: x += dx in FP64, then the FP64 residual replaces r
      for (int64_t a = rtid; a < Nn; a += rthr)
#pragma unroll
        for (int i = 0; i < D; ++i) {
          const int64_t dof = a * D + i;
          if (!I.known[dof]) I.x[dof] = ldcg(I.x + dof) + (double)ldcg(w.dx + dof);
          w.dx[dof] = 0;
        }
      c.cl.sync();  // the updated x of every node is visible before the residual reads neighbours
      double vr[VT][4] = {}, orr[4];
      resid64<D, G, VT>(S64, I.b, I.x, w.r64, grp, ngrp, lane, vr);
      csum<4, VT>(c, vr, orr);
      rr_true = orr[0];
      ++updates;
      floor2 = (32 * eps64) * (32 * eps64) * orr[2];
      tol2 = fmax(I.rtol * I.rtol * bb, floor2);
      if (!isfinite(rr_true)) {
        status = GFEA_ERR_NAN;
        break;
      }
      if (rr_true <= tol2) {
        status = GFEA_OK;
        break;
      }
      if (iters >= I.max_iters) break;
      stall = rr_true > 0.9 * rr_best ? stall + 1 : 0;
      rr_best = fmin(rr_best, rr_true);
      if (stall >= 8) break;
      double vz[VT][2] = {}, oz[2];
      if (two_level)
        restart_rz_two_level<D, T, VT>(c, I, w, gtid, nthr, vz);
      else
        restart_rz<D, T, VT>(I, w, gtid, nthr, vz);
      csum<2, VT>(c, vz, oz);
      beta = next_beta(2, oz[0], rz, beta);
      rz = oz[0];
      trigger = fmax(delta2 * rr_true, 0.25 * tol2);
    }
  }
  if (c.rank == 0 && tid == 0) {
    gfea_pcg_result* R = I.result;
    R->status = status;
    R->iterations = iters;
    R->refinements = updates;
    R->pad = 0;
    R->rel_residual = bb > 0 ? sqrt(rr_true / bb) : 0.0;
    R->floor_rel = bb > 0 ? sqrt(floor2 / bb) : 0.0;
  }
}

template <typename T, int VT>
__device__ void dispatch(Ctx& c, const gfea_batch_instance& I, double delta2) {
  switch (I.dof_n) {
    case 1: solve_instance<1, 8, T, VT>(c, I, delta2); break;
    case 2: solve_instance<2, 8, T, VT>(c, I, delta2); break;
    default: solve_instance<3, 32, T, VT>(c, I, delta2); break;
  }
}

// One launch per width; the systems are sorted by stored values, the wide ones
// first.  The narrow launch is a programmatic dependent of the wide one: it
// starts when the wide clusters hold their SMs, takes the SMs they leave, and
// completes after them.
template <typename T, int BT>
__global__ void __cluster_dims__(kCL, 1, 1) __launch_bounds__(BT, 2 * kNarrow / BT)
    batch_pcg_kernel(const gfea_batch_instance* __restrict__ insts, int n, int* next, double delta2) {
  __shared__ double slots[8];
  __shared__ double sh[4 * (kWide / 32)];
  __shared__ int s_idx;
  if (BT == kWide) cudaTriggerProgrammaticLaunchCompletion();
  Ctx c{cg::this_cluster(), 0, slots, sh, 0};
  c.rank = c.cl.block_rank();
  // the wide systems are [0, split): none where the batch fills the narrow
  // clusters for longer than its largest system takes
  int split = 0;
  double total = 0;
  for (int i = threadIdx.x; i < n; i += BT) total += (double)stored_values(insts[i]);
  total = block_sum(total, sh);
  if (threadIdx.x == 0) s_idx = (double)stored_values(insts[0]) * (2 * kSMs / kCL) > 2 * total;
  __syncthreads();
  if (s_idx) {
    int hi = n;
    while (split < hi) {
      const int mid = (split + hi) >> 1;
      if (stored_values(insts[mid]) >= kWideValues) split = mid + 1; else hi = mid;
    }
  }
  __syncthreads();
  const int first = BT == kWide ? 0 : split, last = BT == kWide ? split : n;
  for (;;) {
    if (c.rank == 0 && threadIdx.x == 0) s_idx = first + atomicAdd(next + (BT == kWide ? 0 : 1), 1);
    c.cl.sync();
    const int idx = *c.cl.map_shared_rank(&s_idx, 0);
    c.cl.sync();  // rank 0's slot is read by all before it changes
    if (idx >= last) break;
    const gfea_batch_instance I = insts[idx];
    dispatch<T, kWide / BT>(c, I, delta2);
  }
  if (BT == kNarrow) cudaGridDependencySynchronize();
}

// Persistent clusters: enough to fill the GPU, never more than the systems.
// The wide launch takes no more than can be resident at once, so that the
// narrow one does not wait for a wide solve to end.
template <typename T>
int launch_widths(const gfea_batch_instance* desc, int n, int* next, double delta2, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.stream = s;
  cfg.blockDim = dim3(kWide);
  cfg.gridDim = dim3(kCL);
  int resident = 0;
  GFEA_CUDA_TRY(cudaOccupancyMaxActiveClusters(&resident, batch_pcg_kernel<T, kWide>, &cfg));
  cfg.gridDim = dim3(kCL * std::max(1, std::min(n, resident)));
  GFEA_CUDA_TRY(cudaLaunchKernelEx(&cfg, batch_pcg_kernel<T, kWide>, desc, n, next, delta2));
  GFEA_LAUNCH_CHECK();
  cudaLaunchAttribute overlap = {};
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &overlap;
  cfg.numAttrs = 1;
  cfg.blockDim = dim3(kNarrow);
  cfg.gridDim = dim3(kCL * std::max(1, std::min(n, 2 * kSMs / kCL)));
  GFEA_CUDA_TRY(cudaLaunchKernelEx(&cfg, batch_pcg_kernel<T, kNarrow>, desc, n, next, delta2));
  GFEA_LAUNCH_CHECK();
  return GFEA_OK;
}

}  // namespace
}  // namespace gfea

using namespace gfea;

extern "C" size_t gfea_batch_workspace_size(int64_t n_nodes, int dof_n, int precision) {
  if (n_nodes <= 0 || dof_n < 1 || dof_n > 3) return 0;
  return precision == GFEA_F64 ? batch_layout<double>(n_nodes, dof_n, nullptr, nullptr)
                               : batch_layout<float>(n_nodes, dof_n, nullptr, nullptr);
}

extern "C" size_t gfea_batch_scratch_size(int n_instances) {
  if (n_instances < 0) return 0;
  return a256(sizeof(int)) + a256(sizeof(gfea_batch_instance) * (size_t)n_instances);
}

extern "C" int gfea_batch_prepare(const gfea_batch_instance* inst_host, int n, void* scratch, size_t scratch_bytes,
                                  const gfea_pcg_opts* opts_host, void* stream) {
  if (!inst_host || n < 0 || !scratch || !opts_host || opts_host->version != GFEA_ABI_VERSION) return GFEA_ERR_ARG;
  if (scratch_bytes < gfea_batch_scratch_size(n)) return GFEA_ERR_WORKSPACE;
  const int prec = opts_host->precision;
  if (prec != GFEA_F64 && prec != GFEA_F32) return GFEA_ERR_ARG;
  for (int i = 0; i < n; ++i) {
    const gfea_batch_instance& I = inst_host[i];
    if (I.version != GFEA_ABI_VERSION || I.dof_n < 1 || I.dof_n > 3 || I.n_nodes <= 0 || !I.node_ptr || !I.nbr ||
        !I.vals64 || !I.known || !I.b || !I.x || !I.work || !I.result || I.max_iters < 1 || !(I.rtol > 0))
      return GFEA_ERR_ARG;
    if (prec == GFEA_F32 && !I.vals32) return GFEA_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(I.work) & 255) != 0) return GFEA_ERR_ARG;
    const gfea_coarse_level& L = I.coarse;
    if (L.n_agg < 0) return GFEA_ERR_ARG;
    if (L.n_agg > 0) {
      const int nr = I.dof_n == 1 ? 1 : (I.dof_n == 2 ? 3 : 6);
      if (L.nr != nr || L.nc != nr * L.n_agg || L.nc > 512 || !L.agg || !L.off || !L.agg_ptr || !L.agg_nodes ||
          !L.inv || !L.inv32 || !L.rc || !L.ec)
        return GFEA_ERR_ARG;
    }
  }
  if (n == 0) return GFEA_OK;
  // largest systems first (longest-processing-time order over the clusters)
  std::vector<gfea_batch_instance> order(inst_host, inst_host + n);
  std::stable_sort(order.begin(), order.end(), [](const gfea_batch_instance& a, const gfea_batch_instance& b) {
    return stored_values(a) > stored_values(b);
  });
  auto* desc = reinterpret_cast<gfea_batch_instance*>(static_cast<char*>(scratch) + a256(sizeof(int)));
  GFEA_CUDA_TRY(cudaMemcpyAsync(desc, order.data(), sizeof(gfea_batch_instance) * (size_t)n, cudaMemcpyHostToDevice,
                                static_cast<cudaStream_t>(stream)));
  // (a copy from pageable host memory has been staged when cudaMemcpyAsync
  // returns, so the local descriptor array may go out of scope)
  return GFEA_OK;
}

extern "C" int gfea_batch_launch(void* scratch, int n, const gfea_pcg_opts* opts_host, void* stream) {
  if (!scratch || n < 0 || !opts_host || opts_host->version != GFEA_ABI_VERSION) return GFEA_ERR_ARG;
  const int prec = opts_host->precision;
  if (prec != GFEA_F64 && prec != GFEA_F32) return GFEA_ERR_ARG;
  if (n == 0) return GFEA_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int* next = static_cast<int*>(scratch);
  auto* desc = reinterpret_cast<gfea_batch_instance*>(static_cast<char*>(scratch) + a256(sizeof(int)));
  GFEA_CUDA_TRY(cudaMemsetAsync(next, 0, 2 * sizeof(int), s));
  const double d = (opts_host->inner_rtol > 0 && opts_host->inner_rtol < 1) ? opts_host->inner_rtol : 0.1;
  return prec == GFEA_F64 ? launch_widths<double>(desc, n, next, 1e-6, s) : launch_widths<float>(desc, n, next, d * d, s);
}

extern "C" int gfea_batch_pcg(const gfea_batch_instance* inst_host, int n, void* scratch, size_t scratch_bytes,
                              const gfea_pcg_opts* opts_host, void* stream) {
  int e = gfea_batch_prepare(inst_host, n, scratch, scratch_bytes, opts_host, stream);
  if (e) return e;
  return gfea_batch_launch(scratch, n, opts_host, stream);
}
