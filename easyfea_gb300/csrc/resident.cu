// Resident PCG: a whole solve in one cooperative launch.
//
// An operator that fits in L2 is not bound by HBM: the multi-kernel iteration
// (four dependent launches, each ending in a last-block reduction) took ~31 us
// for 1e4 to 1e5 unknowns where its bytes need ~1 us.  Here every CTA owns a
// contiguous range of nodes for the whole solve: r, the correction, p, D^-1
// and as many of its rows of the operator as fit stay in shared memory, with
// its neighbours' part of p (the halo, read once per iteration).  Per
// iteration:
//
//   halo of p; q = A p; s += R^T q (atomics); partial p.q              -> (1)
//   x += alpha p, r -= alpha q, y = D^-1 r; rc -= alpha s (every CTA keeps the
//   coarse residual); own rows of ec = A_c^-1 rc; partials r.r and
//   r.z = r.y + rc.ec                                                  -> (2)
//   p = y + R ec + beta p                                              -> (3)
//
// Restricting q instead of r lets the restriction end at the point where
// alpha needs a global sum anyway; rc follows r by the same recurrence and is
// recomputed from the FP64 residual at every reliable update.
//
// Exchange between CTAs.  A counter barrier costs four dependent trips to L2
// (fence, arrival, poll, then the data), ~2 us across the two dies.  Partial
// sums, ec and p travel instead as packets -- a value and the number of its
// exchange in one 8- or 16-byte word, stored and loaded as one access -- and
// a consumer reads the packets it needs until their number is the current
// one: one trip.  A packet is overwritten only after an exchange that its
// readers enter once they have read it (partial sums, read and published at
// the same exchanges, alternate between two sets).  Only what is not in
// packets (the sums s, x after an update) is ordered by fences around the
// exchange of the partial sums (1).  Every CTA adds the partials in the same
// order, so all take the same decisions (convergence, updates, stopping)
// without the host.  The launch is cooperative (the CTAs are co-resident);
// every poll is bounded: after 2 s (a context suspended that long) the launch
// ends and reports it, and the host goes on with the multi-kernel iteration,
// which waits for nothing.
//
// Bound: latency (three exchanges of ~2 us, the halo, the serial chains
// between them); in FP64 3D also the FP64 pipe (27 x 9 products per node: 5 us
// of the 25 us iteration at 13,104 nodes).  Whole solves, multi-kernel ->
// resident: 208 unknowns FP64 1.82 -> 0.99 ms, QUAD4 240x26 FP64 4.61 -> 2.16,
// HEXA8 77x13x11 FP64 8.07 -> 3.44, QUAD9 461x50 mixed 15.6 -> 9.5, load step
// of the 80,000-triangle plate 12.7 -> 6.7 (counters: barrier stalls of the
// warps that wait for the polling one, 20 to 27 per issue; QUAD9 5.8 and 40 MB
// an iteration from L2).
//
// FP64 instructions retire at a sixteenth of a warp per cycle and SM, so the
// scalar recurrences run in one thread, the sums of the partials in one warp
// per value, and the restriction sums each aggregate's nodes directly (in
// float pairs in the FP32 solve: a CTA's share of an aggregate may be hundreds
// of nodes).
#include <math.h>
#include <stdlib.h>

#include <algorithm>

#include "coarse.cuh"
#include "common.cuh"
#include "resident.cuh"
#include "rowops.cuh"
#include "stage.cuh"

namespace gfea {
namespace {

constexpr int kRT = 512;  // threads per CTA
constexpr int kRW = kRT / 32;
constexpr size_t kRSmemMax = 216 * 1024;  // dynamic shared memory
constexpr int kAggWords = 48;             // 32-bit words of the aggregates' bitmap (1536 aggregates)

// ---- packets: a value and the number of its exchange -----------------------
template <typename T>
struct Packet;
template <>
struct Packet<float> {
  static __device__ __forceinline__ void store(float* p, float v, uint32_t tag) {
    const uint64_t w = (uint64_t)tag << 32 | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
  }
  static __device__ __forceinline__ float load(const float* p, uint32_t* tag) {
    uint64_t w;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    *tag = (uint32_t)(w >> 32);
    return __uint_as_float((uint32_t)w);
  }
};
template <>
struct Packet<double> {
  static __device__ __forceinline__ void store(double* p, double v, uint32_t tag) {
    asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"((uint64_t)tag)
                 : "memory");
  }
  static __device__ __forceinline__ double load(const double* p, uint32_t* tag) {
    long long v;
    uint64_t t;
    asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
                 : "=l"(v), "=l"(t)
                 : "l"(p)
                 : "memory");
    *tag = (uint32_t)t;
    return __longlong_as_double(v);
  }
};

// Bounded polling: expired() is true once the limit has passed or another
// thread of the CTA gave up.
struct Deadline {
  uint64_t t0 = 0;
  uint32_t n = 0;
  __device__ __forceinline__ bool expired(volatile int* abort, uint64_t limit_ns) {
    if ((++n & 255u) != 0) return false;
    const uint64_t t = global_ns();
    if (t0 == 0) t0 = t;
    if (*abort || t - t0 > limit_ns) {
      *abort = 1;
      return true;
    }
    return false;
  }
};

// The value of packet p once it carries 'tag' (0 when the wait ran out).
template <typename T>
__device__ __forceinline__ T await_packet(const T* p, uint32_t tag, volatile int* abort, uint64_t limit_ns) {
  uint32_t t;
  T v = Packet<T>::load(p, &t);
  Deadline d;
  while (t != tag) {
    if (d.expired(abort, limit_ns)) return 0;
    v = Packet<T>::load(p, &t);
  }
  return v;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The CTAs of one solve.
struct Team {
  double* box;         // packets of the partial sums, [parity][value][reader][writer]
  uint32_t number;     // exchanges so far
  double (*shw)[kRW];  // warp sums
  double* res;         // reduced values
  volatile int* abort; // a wait of this CTA ran out
  int* ok;             // its verdict at the last exchange, the same for every thread
  uint64_t limit_ns;
};

// Exchange of NV sums (w: warp sums, valid in lane 0).  Value k belongs to
// warp k, which publishes the CTA's sum and adds all CTAs' in a fixed order;
// the other warps run meanwhile(thread, threads); thread 0 then runs
// f(totals), whose shared-memory results every thread sees.  FENCE: writes
// before the exchange (any CTA) are visible after it (through ld.cg).  False,
// for every thread of the CTA, when a wait ran out before.
template <int NV, bool FENCE, typename M, typename F>
__device__ __forceinline__ bool exchange(Team& t, const double (&w)[NV], M meanwhile, F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool solo = gridDim.x == 1;
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) t.shw[k][warp] = w[k];
  __syncthreads();
  const uint32_t tag = ++t.number;
  if (warp < NV) {
    double s = lane < kRW ? t.shw[warp][lane] : 0.0;
#pragma unroll
    for (int o = kRW / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    s = __shfl_sync(0xffffffffu, s, 0);
    if (!solo) {
      // a packet of its own for every reader: one set read by all would sit
      // on a few L2 slices, and the CTAs' polls there cost ~5 us an exchange
      const int grid = gridDim.x;
      // two sets in turn: a CTA may publish the next exchange while a reader
      // still polls this one, but not the one after it
      double* box = t.box + 2 * (size_t)((tag & 1u) * 4 + warp) * grid * grid;
      if (FENCE) __threadfence();
      for (int i = lane; i < grid; i += 32) Packet<double>::store(box + 2 * ((size_t)i * grid + blockIdx.x), s, tag);
      const double* slot = box + 2 * (size_t)blockIdx.x * grid;
      // all of the lane's packets in flight at once
      constexpr int U = (kSMs + 31) / 32;
      double v[U];
      bool wait = false;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        v[u] = 0;
        const int i = lane + 32 * u;
        if (i < (int)gridDim.x) {
          uint32_t got;
          v[u] = Packet<double>::load(slot + 2 * i, &got);
          wait |= got != tag;
        }
      }
      Deadline d;
      while (wait && !d.expired(t.abort, t.limit_ns)) {
        wait = false;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = lane + 32 * u;
          if (i < (int)gridDim.x) {
            uint32_t got;
            v[u] = Packet<double>::load(slot + 2 * i, &got);
            wait |= got != tag;
          }
        }
      }
      __syncwarp();
      if (FENCE) __threadfence();
      s = v[0];
#pragma unroll
      for (int u = 1; u < U; ++u)
        if (32 * u < (int)gridDim.x) s += v[u];
      s = warp_sum(s);
    }
    if (lane == 0) t.res[warp] = s;
  } else {
    meanwhile((int)threadIdx.x - NV * 32, kRT - NV * 32);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    f(t.res);
    *t.ok = *t.abort == 0;  // one reading for all: a thread ahead may give up while another reads
  }
  __syncthreads();
  return *t.ok != 0;
}

template <bool FENCE>
__device__ __forceinline__ bool exchange_nothing(Team& t) {
  const double w[1] = {0};
  return exchange<1, FENCE>(t, w, [](int, int) {}, [](const double*) {});
}

enum Mode { kIter, kStart, kUpdate, kEnd };

// Scalars of the solve.  Thread 0 of every CTA computes them from the same
// sums, so they agree everywhere.
struct Ctl {
  double alpha, beta;
  double rz, rr, bb, rr_true, rr_best, tol2, floor2, trigger;
  int mode, status, st_inner, iters, updates, stall;
};

// Shared memory of one CTA's fixed arrays; the halo, the operator's rows and
// rows of A_c^-1 take the rest in this order, as far as they fit.
template <typename T>
struct Layout {
  size_t q, r, p, dx, dinv, off, rc, sv, ecl, nptr, seg_ptr, seg_agg, order, la, kn, total;
  __host__ __device__ Layout(int D, int npc, int nc, int n_agg, bool solo) {
    size_t o = 0;
    auto take = [&](size_t bytes) {
      const size_t at = o;
      o += (bytes + 15) & ~size_t(15);
      return at;
    };
    const size_t rows = (size_t)npc * D;
    const size_t segs = n_agg < npc ? n_agg : npc;
    const int nr = n_agg > 0 ? nc / n_agg : 0;
    q = take(sizeof(T) * rows);
    r = take(sizeof(T) * rows);
    p = take(sizeof(T) * rows);
    dx = take(sizeof(T) * rows);
    dinv = take(sizeof(T) * rows * D);
    off = take(nc && D > 1 ? sizeof(T) * rows : 0);
    rc = take(sizeof(double) * nc);
    sv = take(solo ? sizeof(double) * nc : 0);
    ecl = take(sizeof(T) * segs * nr);
    nptr = take(sizeof(int32_t) * (npc + 1));
    seg_ptr = take(sizeof(int32_t) * (segs + 1));
    seg_agg = take(sizeof(int32_t) * segs);
    order = take(nc ? sizeof(uint16_t) * npc : 0);
    la = take(nc ? sizeof(uint16_t) * npc : 0);
    kn = take(rows);
    total = o;
  }
};

// Exclusive prefix sum of one int per thread over the CTA (total in *sum).
__device__ __forceinline__ int block_scan(int v, int* scratch, int* sum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int s = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += u;
  }
  __syncthreads();
  if (lane == 31) scratch[warp] = s;
  __syncthreads();
  int base = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kRW; ++w) {
    const int u = scratch[w];
    base += w < warp ? u : 0;
    total += u;
  }
  *sum = total;
  return base + s - v;
}

// The D entries of a packed block's component j.
template <int D, typename T>
__device__ __forceinline__ void load_block(const T* b, T (&v)[D]) {
  if constexpr (D == 2 && sizeof(T) == 4) {
    const float2 u = *reinterpret_cast<const float2*>(b);
    v[0] = u.x;
    v[1] = u.y;
  } else if constexpr (D == 2) {
    const double2 u = *reinterpret_cast<const double2*>(b);
    v[0] = u.x;
    v[1] = u.y;
  } else {
#pragma unroll
    for (int d = 0; d < D; ++d) v[d] = b[d];
  }
}

// Component k of R e at offset o (e: the modes' coefficients).
template <int D, typename T>
__device__ __forceinline__ T prolong(int k, const T* o, const T* e) {
  if constexpr (D == 1) {
    return e[0];
  } else if constexpr (D == 2) {
    return k == 0 ? e[0] - o[1] * e[2] : e[1] + o[0] * e[2];
  } else {
    const int b = k == 2 ? 0 : k + 1, c = k == 0 ? 2 : k - 1;
    return e[k] + (o[c] * e[3 + b] - o[b] * e[3 + c]);
  }
}

// G: lanes per node of the FP32 SpMV (values read along the row); the FP64
// one gives each lane one component of one node (it is bound by the FP64
// pipe, and a lane then spends no FP64 additions on lane sums).
template <int D, int G, typename T>
__global__ void __launch_bounds__(kRT, 1) resident_kernel(ResidentProblem<T> P, ResidentGeom geom) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double s_w[4][kRW];
  __shared__ double s_res[4];
  __shared__ int s_abort, s_ok, s_scan[kRW], s_range[2], s_nseg;
  __shared__ uint32_t s_bits[kAggWords];
  __shared__ int s_base[kAggWords];
  __shared__ Ctl ctl;
  constexpr int nr = Modes<D>::nr;
  constexpr int NPW = 32 / D;  // nodes per warp in the component-per-lane loops
  using Pk = Packet<T>;
  const SysT<T>& S = P.S;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool solo = gridDim.x == 1;
  const int nc = P.coarse ? P.C.nc : 0;
  const int n_agg = P.coarse ? P.C.n_agg : 0;
  const Layout<T> L(D, geom.npc, nc, n_agg, solo);
  T* q_s = reinterpret_cast<T*>(smem + L.q);
  T* r_s = reinterpret_cast<T*>(smem + L.r);
  T* p_s = reinterpret_cast<T*>(smem + L.p);
  T* dx_s = reinterpret_cast<T*>(smem + L.dx);
  T* dinv_s = reinterpret_cast<T*>(smem + L.dinv);
  T* off_s = reinterpret_cast<T*>(smem + L.off);
  double* rc_s = reinterpret_cast<double*>(smem + L.rc);
  double* sv_s = reinterpret_cast<double*>(smem + L.sv);
  T* ecl_s = reinterpret_cast<T*>(smem + L.ecl);
  int32_t* nptr_s = reinterpret_cast<int32_t*>(smem + L.nptr);
  int32_t* seg_ptr = reinterpret_cast<int32_t*>(smem + L.seg_ptr);
  int32_t* seg_agg = reinterpret_cast<int32_t*>(smem + L.seg_agg);
  uint16_t* order_s = reinterpret_cast<uint16_t*>(smem + L.order);
  uint16_t* la_s = reinterpret_cast<uint16_t*>(smem + L.la);
  uint8_t* kn_s = smem + L.kn;
  size_t used = L.total;
  if (tid == 0) {
    s_abort = 0;
    ctl = Ctl{};
    ctl.mode = kStart;
    ctl.status = GFEA_ERR_NOT_CONVERGED;
    ctl.st_inner = GFEA_OK;
    s_range[0] = INT32_MAX;
    s_range[1] = -1;
    s_nseg = 0;
  }
  Team team{P.box, 0, s_w, s_res, &s_abort, &s_ok, kWaitLimitNs};

  // ---- own nodes a0 .. a0 + n ---------------------------------------------
  const int64_t a0 = min((int64_t)blockIdx.x * geom.npc, S.Nn);
  const int n = (int)(min(a0 + geom.npc, S.Nn) - a0);
  const int rows = n * D;
  const int32_t pair0 = S.node_ptr[a0];
  const int n_slots = S.node_ptr[a0 + n] - pair0;
  const int32_t* NBg = S.nbr + pair0;
  const T* Vg = S.vals + (int64_t)D * D * pair0;
  for (int i = tid; i <= n; i += kRT) nptr_s[i] = S.node_ptr[a0 + i] - pair0;
  for (int i = tid; i < rows; i += kRT) {
    kn_s[i] = S.known[a0 * D + i];
    dx_s[i] = p_s[i] = 0;
    if (!solo) Pk::store(P.p + 2 * (a0 * D + i), 0, 0);  // packets of an earlier solve may carry any number
  }

  // ---- the own nodes of each aggregate ------------------------------------
  if (nc) {
    for (int i = tid; i < kAggWords; i += kRT) s_bits[i] = 0;
    __syncthreads();
    for (int i = tid; i < n; i += kRT) {
      const int g = P.C.agg[a0 + i];
      atomicOr(&s_bits[g >> 5], 1u << (g & 31));
      if constexpr (D > 1) {
        const float4 o = P.C.off[a0 + i];
        off_s[i * D] = o.x;
        off_s[i * D + 1] = o.y;
        if constexpr (D == 3) off_s[i * D + 2] = o.z;
      }
    }
    __syncthreads();
    if (tid == 0) {
      int s = 0;
      for (int w = 0; w < kAggWords; ++w) {
        s_base[w] = s;
        s += __popc(s_bits[w]);
      }
      s_nseg = s;
    }
    __syncthreads();
    for (int i = tid; i <= s_nseg; i += kRT) seg_ptr[i] = 0;
    __syncthreads();
    for (int i = tid; i < n; i += kRT) {
      const int g = P.C.agg[a0 + i];
      const int l = s_base[g >> 5] + __popc(s_bits[g >> 5] & ((1u << (g & 31)) - 1u));
      la_s[i] = (uint16_t)l;
      seg_agg[l] = g;
      atomicAdd(&seg_ptr[l], 1);
    }
    __syncthreads();
    if (tid == 0) {  // end positions; the fill below counts them down to the starts
      int s = 0;
      for (int l = 0; l < s_nseg; ++l) seg_ptr[l] = s += seg_ptr[l];
      seg_ptr[s_nseg] = s;
    }
    __syncthreads();
    for (int i = tid; i < n; i += kRT) order_s[atomicSub(&seg_ptr[la_s[i]], 1) - 1] = (uint16_t)i;
    // coarse corrections: packets, and the accumulators of s
    double* rcp = P.C.rcp;
    if (solo) {
      for (int i = tid; i < nc; i += kRT) sv_s[i] = 0;
    } else if (blockIdx.x == 0) {
      for (int i = tid; i < 3 * nc; i += kRT) rcp[i] = 0;
    }
    if (!solo)
      for (int i = blockIdx.x + tid * gridDim.x; i < nc; i += kRT * gridDim.x) Pk::store(P.ec + 2 * i, 0, 0);
  }
  __syncthreads();

  // ---- halo: the distinct neighbours of the own nodes, ascending -----------
  // A bitmap over their range and its prefix counts give each neighbour its
  // place; they live where the operator's rows go afterwards.
  int32_t* halo_s = nullptr;  // node ids
  uint16_t* lidx_s = nullptr; // place in the halo of each neighbour slot
  T* pl_s = nullptr;          // their part of p
  int halo = 0;
  {
    int lo = INT32_MAX, hi = -1;
    for (int i = tid; i < n_slots; i += kRT) {
      const int b = __ldg(NBg + i);
      lo = min(lo, b);
      hi = max(hi, b);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0 && hi >= 0) {
      atomicMin(&s_range[0], lo);
      atomicMax(&s_range[1], hi);
    }
    __syncthreads();
    lo = s_range[0];
    hi = s_range[1];
    const int words = hi >= 0 ? (hi - lo) / 32 + 1 : 0;
    const size_t idx_bytes = (sizeof(uint16_t) * (size_t)n_slots + 15) & ~size_t(15);
    if (words > 0 && used + idx_bytes + 8 * (size_t)words + 64 <= geom.smem) {
      lidx_s = reinterpret_cast<uint16_t*>(smem + used);
      uint32_t* bits = reinterpret_cast<uint32_t*>(smem + used + idx_bytes);
      int* base = reinterpret_cast<int*>(bits + words);
      for (int i = tid; i < words; i += kRT) bits[i] = 0;
      __syncthreads();
      for (int i = tid; i < n_slots; i += kRT) {
        const int b = __ldg(NBg + i) - lo;
        atomicOr(&bits[b >> 5], 1u << (b & 31));
      }
      __syncthreads();
      const int per = (words + kRT - 1) / kRT, w0 = min(tid * per, words), w1 = min(w0 + per, words);
      int c = 0;
      for (int w = w0; w < w1; ++w) c += __popc(bits[w]);
      int at = block_scan(c, s_scan, &halo);
      for (int w = w0; w < w1; ++w) {
        base[w] = at;
        at += __popc(bits[w]);
      }
      __syncthreads();
      const size_t ids = (sizeof(int32_t) * (size_t)halo + 15) & ~size_t(15);
      const size_t pl = (sizeof(T) * D * (size_t)halo + 15) & ~size_t(15);
      if (halo <= 65535 && used + idx_bytes + ids + pl <= geom.smem) {
        for (int i = tid; i < n_slots; i += kRT) {
          const int b = __ldg(NBg + i) - lo;
          lidx_s[i] = (uint16_t)(base[b >> 5] + __popc(bits[b >> 5] & ((1u << (b & 31)) - 1u)));
        }
        __syncthreads();  // the bitmap is read no more
        halo_s = reinterpret_cast<int32_t*>(smem + used + idx_bytes);
        for (int i = tid; i < n_slots; i += kRT) halo_s[lidx_s[i]] = __ldg(NBg + i);
        pl_s = reinterpret_cast<T*>(smem + used + idx_bytes + ids);
        used += idx_bytes + ids + pl;
      } else {
        lidx_s = nullptr;
      }
    }
  }
  __syncthreads();

  // ---- the operator's rows: the first n_res own nodes' in shared memory ----
  T* v_s = reinterpret_cast<T*>(smem + used);
  int n_res = 0;
  {
    const size_t room = (geom.smem - used) / (sizeof(T) * D * D);  // slots
    int lo = 0, hi = n;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if ((size_t)nptr_s[mid] <= room) lo = mid; else hi = mid - 1;
    }
    n_res = lo;
    const int nv = nptr_s[n_res] * D * D;
    // block (i, k) as [j][d]: a lane of component j reads the D rows' entries
    // as one word; rows of known DOFs are zero
    for (int i = warp; i < n_res; i += kRW) {
      const int32_t s0 = nptr_s[i], W = D * (nptr_s[i + 1] - s0);
      for (int e = lane; e < D * W; e += 32) {
        const int d = e / W, t = e - d * W;
        const T v = __ldcs(Vg + D * D * s0 + e);
        v_s[D * D * (s0 + t / D) + (t % D) * D + d] = kn_s[i * D + d] ? (T)0 : v;
      }
    }
    used += (sizeof(T) * (size_t)nv + 15) & ~size_t(15);
  }
  // rows blockIdx.x, blockIdx.x + grid, ... of A_c^-1 when there is room left
  const int my_rows = nc > (int)blockIdx.x ? (nc - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  const double* A = P.C.Ac + (int64_t)blockIdx.x * nc;
  int64_t a_stride = (int64_t)gridDim.x * nc;
  if (nc && n_res == n && used + sizeof(double) * (size_t)my_rows * nc <= geom.smem) {
    double* A_s = reinterpret_cast<double*>(smem + used);
    for (int k = warp; k < my_rows; k += kRW)
      for (int i = lane; i < nc; i += 32) A_s[k * nc + i] = __ldcs(A + k * a_stride + i);
    A = A_s;
    a_stride = nc;
  }
  __syncthreads();

  // ---- block-Jacobi inverses of the own nodes ------------------------------
  double bad = 0;
  for (int i = tid; i < n; i += kRT) {
    const int64_t a = a0 + i;
    const int32_t s0 = nptr_s[i], nb = nptr_s[i + 1] - s0;
    int lo = 0, hi = nb;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (NBg[s0 + mid] < a) lo = mid + 1; else hi = mid;
    }
    const bool has = lo < nb && NBg[s0 + lo] == a;
    const int W = D * nb;
    double M[D][D], iM[D][D];
#pragma unroll
    for (int k = 0; k < D; ++k)
#pragma unroll
      for (int j = 0; j < D; ++j) {
        double v = has ? (double)Vg[D * D * s0 + k * W + D * lo + j] : 0.0;
        if (kn_s[i * D + k] || kn_s[i * D + j]) v = (k == j) ? 1.0 : 0.0;
        M[k][j] = v;
      }
    const double det = det_inv<D>(M, iM);
    if (!(fabs(det) > 0) || !isfinite(det)) {
      bad += 1;
#pragma unroll
      for (int k = 0; k < D; ++k)
#pragma unroll
        for (int j = 0; j < D; ++j) iM[k][j] = (k == j) ? 1.0 : 0.0;
    }
#pragma unroll
    for (int k = 0; k < D; ++k)
#pragma unroll
      for (int j = 0; j < D; ++j) dinv_s[(i * D + k) * D + j] = (T)iM[k][j];
  }
  bool ok = exchange_nothing<true>(team);  // cleared packets and accumulators precede their first use

  // accumulators of s in turn: in use, cleared, cleared during this iteration
  // (an index, not three pointers: the product's loads need the registers; 2D
  // FP32 128 -> 112, the 80,000-triangle load step 7.15 -> 6.68 ms, QUAD9
  // 461x50 10.15 -> 9.53)
  int turn = 0;
  auto s_of = [&](int ahead) { return P.C.rcp + (turn + ahead < 3 ? turn + ahead : turn + ahead - 3) * nc; };
  // lanes per (aggregate, mode) sum of the restriction
  int H = 1;
  while (H < 32 && 2 * H * s_nseg * nr <= kRT) H *= 2;
  // s += R^T v for the own nodes' v (zero on known DOFs)
  auto restrict_rows = [&](const T* v_s) {
    const int tasks = s_nseg * nr, h = tid % H;
    for (int t0 = 0; t0 < tasks; t0 += kRT / H) {
      const int t = t0 + tid / H;
      DotAcc<T> v;
      int g = 0, m = 0;
      if (t < tasks) {
        const int l = t / nr;
        m = t - l * nr;
        g = seg_agg[l];
        const int k1 = seg_ptr[l + 1];
        for (int k = seg_ptr[l] + h; k < k1; k += H) {
          const int i = order_s[k];
          add_mode<D, T>(v, m, off_s + i * D, v_s + i * D);
        }
      }
      const double sum = warp_sum_acc(v, H);
      if (t < tasks && h == 0) {
        if (solo)
          sv_s[g * nr + m] = sum;
        else
          atomicAdd(s_of(0) + g * nr + m, sum);
      }
    }
  };
  const bool diff = sizeof(T) == 4 && S.diff;
  uint32_t p_number = 0;  // number of the last published p

  while (ok) {
    const int mode = ctl.mode;
    if (mode == kEnd) break;
    if (mode == kIter) {
      // ---- halo of p --------------------------------------------------------
      if (pl_s) {
        const int cnt = halo * D;
        if (solo) {
          for (int i = tid; i < cnt; i += kRT) pl_s[i] = p_s[halo_s[i / D] * D + i % D];
        } else {
          constexpr int U = 4;
          for (int i0 = tid; i0 < cnt; i0 += U * kRT) {
            T v[U];
            uint32_t tag[U];
            const T* src[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const int i = i0 + u * kRT;
              tag[u] = p_number;
              if (i < cnt) {
                src[u] = P.p + 2 * ((int64_t)halo_s[i / D] * D + i % D);
                v[u] = Pk::load(src[u], &tag[u]);
              }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const int i = i0 + u * kRT;
              if (i < cnt) {
                if (tag[u] != p_number) v[u] = await_packet<T>(src[u], p_number, &s_abort, kWaitLimitNs);
                pl_s[i] = v[u];
              }
            }
          }
        }
        __syncthreads();
      }
      // ---- q = A p (masked) ------------------------------------------------
      auto p_at = [&](int slot, int j) -> T {
        if (pl_s) return pl_s[lidx_s[slot] * D + j];
        const int64_t c = (int64_t)__ldg(NBg + slot) * D + j;
        return solo ? p_s[c] : await_packet<T>(P.p + 2 * c, p_number, &s_abort, kWaitLimitNs);
      };
      if constexpr (sizeof(T) == 4) {
        constexpr int LA = G - G % D, NPP = LA / D;
        constexpr int R = 4;             // nodes of a lane group at once: their loads overlap
        constexpr int step = kRW * (32 / G);
        const int l = lane % G, j = l % D, k0 = l / D;
        for (int i0 = warp * (32 / G); i0 < n; i0 += R * step) {
          T acc[R][D], self[R];
          int32_t s0[R], nb[R];
          int most = 0;
          bool res = pl_s != nullptr;  // uniform over the lane group's nodes: everything in shared memory
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int i = i0 + r * step + lane / G;
            const bool in = i < n && l < LA;
            s0[r] = in ? nptr_s[i] : 0;
            nb[r] = in ? nptr_s[i + 1] - s0[r] : 0;
            self[r] = diff && in ? p_s[i * D + j] : (T)0;
            most = max(most, nb[r]);
            res = res && (i >= n || i < n_res);
#pragma unroll
            for (int d = 0; d < D; ++d) acc[r][d] = 0;
          }
          if (res) {
            for (int k = k0; k < most; k += NPP) {
              T xv[R], v[R][D];
#pragma unroll
              for (int r = 0; r < R; ++r) {
                xv[r] = 0;
#pragma unroll
                for (int d = 0; d < D; ++d) v[r][d] = 0;
                if (k < nb[r]) {
                  xv[r] = pl_s[lidx_s[s0[r] + k] * D + j] - self[r];
                  load_block<D, T>(v_s + (D * (s0[r] + k) + j) * D, v[r]);
                }
              }
#pragma unroll
              for (int r = 0; r < R; ++r)
#pragma unroll
                for (int d = 0; d < D; ++d) acc[r][d] += v[r][d] * xv[r];
            }
          } else {
            for (int k = k0, t = l; k < most; k += NPP, t += LA) {
              T v[R][D];
#pragma unroll
              for (int r = 0; r < R; ++r)
#pragma unroll
                for (int d = 0; d < D; ++d) v[r][d] = k < nb[r] ? __ldg(Vg + D * D * s0[r] + d * D * nb[r] + t) : (T)0;
#pragma unroll
              for (int r = 0; r < R; ++r) {
                const T xv = k < nb[r] ? p_at(s0[r] + k, j) - self[r] : (T)0;
#pragma unroll
                for (int d = 0; d < D; ++d) acc[r][d] += v[r][d] * xv;
              }
            }
          }
          __syncwarp();
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int i = i0 + r * step + lane / G;
            const T av = group_sum_rows<D, G, T>(acc[r], l);
#pragma unroll
            for (int d = 0; d < D; ++d)
              if (i < n && l == row_lane<D, G>(d)) q_s[i * D + d] = !res && kn_s[i * D + d] ? (T)0 : av;
          }
        }
      } else {
        for (int base = warp * NPW; base < n; base += kRW * NPW) {
          const int i = base + lane / D;
          const bool live = lane < NPW * D && i < n;
          const int j = live ? lane % D : 0;
          T acc[D];
#pragma unroll
          for (int k = 0; k < D; ++k) acc[k] = 0;
          if (live) {
            const int32_t s0 = nptr_s[i], nb = nptr_s[i + 1] - s0;
            const int W = D * nb;
            if (pl_s && i < n_res) {
#pragma unroll 3
              for (int k = 0; k < nb; ++k) {
                const T xv = pl_s[lidx_s[s0 + k] * D + j];
                T v[D];
                load_block<D, T>(v_s + (D * (s0 + k) + j) * D, v);
#pragma unroll
                for (int d = 0; d < D; ++d) acc[d] += v[d] * xv;
              }
            } else {
              // the lane's trips to L2 are one chain: U neighbours' at once
              // (three, and one packet of p at a time without a halo: 9,225
              // PRISM18 nodes 10.05 ms, four 8.39, the multi-kernel iteration 9.69)
              constexpr int U = 4;
              const T* vr = Vg + D * D * s0 + j;
              for (int k0 = 0; k0 < nb; k0 += U) {
                T v[U][D], xv[U];
                const T* src[U];
                uint32_t tag[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                  const int k = k0 + u;
                  const bool in = k < nb;
                  tag[u] = p_number;
                  xv[u] = 0;
                  src[u] = P.p;
                  if (in && pl_s) {
                    xv[u] = pl_s[lidx_s[s0 + k] * D + j];
                  } else if (in) {
                    const int64_t c = (int64_t)__ldg(NBg + s0 + k) * D + j;
                    src[u] = P.p + 2 * c;
                    xv[u] = solo ? p_s[c] : Pk::load(src[u], &tag[u]);
                  }
#pragma unroll
                  for (int d = 0; d < D; ++d) v[u][d] = in ? __ldg(vr + d * W + D * k) : (T)0;
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                  if (tag[u] != p_number) xv[u] = await_packet<T>(src[u], p_number, &s_abort, kWaitLimitNs);
#pragma unroll
                  for (int d = 0; d < D; ++d) acc[d] += v[u][d] * xv[u];
                }
              }
            }
          }
          const T av = node_rows_exchange<D, T>(acc, j, live ? lane : lane - lane % D);
          if (live) q_s[i * D + j] = kn_s[i * D + j] ? (T)0 : av;
        }
      }
      __syncthreads();
      if (nc) restrict_rows(q_s);
      DotAcc<T> pap;
      for (int i = tid; i < rows; i += kRT) pap.add_prod(p_s[i], q_s[i]);
      const double w[1] = {warp * 32 < rows ? warp_sum_acc(pap) : 0.0};
      ok = exchange<1, true>(team, w, [](int, int) {}, [&](const double* o) {
        if (!(o[0] > 0) || !isfinite(o[0])) {
          ctl.st_inner = isfinite(o[0]) ? GFEA_ERR_BREAKDOWN : GFEA_ERR_NAN;
          ctl.mode = kUpdate;
        } else {
          ctl.alpha = ctl.rz / o[0];
        }
      });
      if (!ok) break;
      if (ctl.mode == kUpdate) {  // s was not consumed: clear it
        if (blockIdx.x == 0 && !solo)
          for (int i = tid; i < nc; i += kRT) s_of(0)[i] = 0;
        continue;
      }
    } else {
      if (mode == kUpdate) {  // x += dx
        for (int i = tid; i < rows; i += kRT) {
          const int64_t dof = a0 * D + i;
          if (!kn_s[i]) __stcg(P.x + dof, __ldcg(P.x + dof) + (double)dx_s[i]);
          dx_s[i] = 0;
        }
        if (!(ok = exchange_nothing<true>(team))) break;
      }
      // ---- r = P (b - A x) in FP64; ||P(b - A x_c)||^2 at the start;
      // ||P(|A||x| + |b|)||^2 (from the FP32 values in the FP32 solve) --------
      const bool kn = mode == kStart;
      double w[4] = {0, 0, 0, bad};
      const double* V64 = P.vals64 + (int64_t)D * D * pair0;
      for (int base = warp * NPW; base < n; base += kRW * NPW) {
        const int i = base + lane / D;
        const bool live = lane < NPW * D && i < n;
        const int j = live ? lane % D : 0;
        double all[D], xk[D];
        T ab[D];
#pragma unroll
        for (int d = 0; d < D; ++d) {
          all[d] = xk[d] = 0;
          ab[d] = 0;
        }
        if (live) {
          const int32_t s0 = nptr_s[i], nb = nptr_s[i + 1] - s0;
          const int W = D * nb;
          const bool res = i < n_res;
          const T* vr = res ? (const T*)(v_s + D * D * s0 + j * D) : Vg + D * D * s0 + j;
          const int dk = res ? D * D : D, dd = res ? 1 : W;  // strides of a neighbour and of a row
          const double* vr64 = V64 + D * D * s0;
#pragma unroll 3
          for (int k = 0; k < nb; ++k) {
            const uint32_t c = (uint32_t)__ldg(NBg + s0 + k) * D + j;
            const double xv = __ldcg(P.x + c);
            const T xa = (T)fabs(xv);
            const bool isk = kn && S.known[c];
#pragma unroll
            for (int d = 0; d < D; ++d) {
              const T v = vr[d * dd + dk * k];
              const double v64 = sizeof(T) == 8 ? (double)v : __ldg(vr64 + d * W + D * k + j);
              all[d] += v64 * xv;
              if (isk) xk[d] += v64 * xv;
              ab[d] += (v < 0 ? -v : v) * xa;
            }
          }
        }
        const int el = live ? lane : lane - lane % D;
        const double s_all = node_rows_exchange<D, double>(all, j, el);
        const double s_kn = kn ? node_rows_exchange<D, double>(xk, j, el) : 0.0;
        const double s_ab = (double)node_rows_exchange<D, T>(ab, j, el);
        if (live) {
          const bool unk = !kn_s[i * D + j];
          const double bv = P.b[(a0 + i) * D + j];
          const double ri = unk ? bv - s_all : 0.0;
          const double rci = unk ? bv - s_kn : 0.0;
          const double ai = unk ? s_ab + fabs(bv) : 0.0;
          r_s[i * D + j] = (T)ri;
          w[0] += ri * ri;
          w[1] += rci * rci;
          w[2] += ai * ai;
        }
      }
      if (nc) {
        __syncthreads();
        restrict_rows(r_s);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) w[k] = warp_sum(w[k]);
      ok = exchange<4, true>(team, w, [](int, int) {}, [&](const double* o) {
        constexpr double eps64 = 2.220446049250313e-16;
        ctl.rr_true = o[0];
        ctl.floor2 = (32 * eps64) * (32 * eps64) * o[2];
        int end = -1;  // status of a solve that ends here
        if (mode == kStart) {
          ctl.bb = o[1];
          ctl.rr_best = o[0];
          if (o[3] > 0)
            end = GFEA_ERR_SINGULAR;
          else if (!(o[1] == o[1]) || !isfinite(o[0]))
            end = GFEA_ERR_NAN;
          else if (o[1] == 0)
            end = GFEA_OK;
        } else {
          ++ctl.updates;
        }
        ctl.tol2 = fmax(P.rtol * P.rtol * ctl.bb, ctl.floor2);
        if (end < 0 && !isfinite(o[0])) end = GFEA_ERR_NAN;
        if (end < 0 && o[0] <= ctl.tol2) end = GFEA_OK;
        if (end < 0 && mode == kUpdate) {
          if (ctl.st_inner != GFEA_OK) {
            end = ctl.st_inner;
          } else {
            ctl.stall = o[0] > 0.9 * ctl.rr_best ? ctl.stall + 1 : 0;
            if (o[0] < ctl.rr_best) ctl.rr_best = o[0];
            if (ctl.stall >= 8 || ctl.updates >= P.max_upd) end = GFEA_ERR_NOT_CONVERGED;
          }
        }
        if (end >= 0) {
          ctl.status = end;
          ctl.mode = kEnd;
        }
      });
      if (!ok) break;
      if (ctl.mode == kEnd) {
        if (mode == kStart && ctl.status == GFEA_OK && ctl.bb == 0)  // b_i - A_ic x_c = 0: the unknowns are zero
          for (int i = tid; i < rows; i += kRT)
            if (!kn_s[i]) P.x[a0 * D + i] = 0.0;
        break;
      }
    }

    // ---- x, r update and coarse residual -----------------------------------
    const double alpha = ctl.alpha;
    for (int i = tid; i < nc; i += kRT) {
      const double v = solo ? sv_s[i] : __ldcg(s_of(0) + i);
      rc_s[i] = mode == kIter ? rc_s[i] - alpha * v : v;
      // cleared for the iteration after the next: its last readers have
      // entered exchange (1) since, and the next one publishes this
      if (blockIdx.x == 0 && !solo) s_of(2)[i] = 0;
    }
    if (mode == kIter) {
      const T al = (T)alpha;
      for (int i = tid; i < rows; i += kRT) {
        dx_s[i] += al * p_s[i];
        r_s[i] -= al * q_s[i];
      }
    }
    __syncthreads();
    // ---- y = D^-1 r (into q_s); own rows of ec = A_c^-1 rc -----------------
    DotAcc<T> rz_acc, rr_acc;
    for (int i = tid; i < rows; i += kRT) {
      const int a = i / D;
      T y = 0;
#pragma unroll
      for (int j = 0; j < D; ++j) y += dinv_s[i * D + j] * r_s[a * D + j];
      if (kn_s[i]) y = 0;
      q_s[i] = y;
      const T ri = r_s[i];
      rz_acc.add_prod(ri, y);
      rr_acc.add_prod(ri, ri);
    }
    double w[2] = {0, 0};
    if (warp * 32 < rows) {
      w[0] = warp_sum_acc(rz_acc);
      w[1] = warp_sum_acc(rr_acc);
    }
    const uint32_t ec_number = team.number + 1;  // of the exchange that follows
    // rows from the last warp down: the first ones hold the vector rows
    for (int k = kRW - 1 - warp; k < my_rows; k += kRW) {
      const double* row = A + k * a_stride;
      double v = 0;
      for (int j = lane; j < nc; j += 32) v += row[j] * rc_s[j];
      v = warp_sum(v);
      if (lane == 0) {
        const int i = blockIdx.x + k * gridDim.x;
        if (solo) {
          const int g = i / nr;
          if (s_bits[g >> 5] >> (g & 31) & 1u)
            ecl_s[(s_base[g >> 5] + __popc(s_bits[g >> 5] & ((1u << (g & 31)) - 1u))) * nr + i % nr] = (T)v;
        } else {
          Pk::store(P.ec + 2 * i, (T)v, ec_number);
        }
        w[0] += (double)(T)v * rc_s[i];  // r.z of the z that takes ec rounded to T
      }
    }
    ok = exchange<2, false>(
        team, w,
        [&](int t, int nt) {  // the own aggregates' corrections
          if (!solo)
            for (int i = t; i < s_nseg * nr; i += nt)
              ecl_s[i] = await_packet<T>(P.ec + 2 * (seg_agg[i / nr] * nr + i % nr), ec_number, &s_abort, kWaitLimitNs);
        },
        [&](const double* o) {
          const double rz = o[0], rr = o[1];
          ctl.beta = next_beta(mode == kIter ? 0 : (mode == kStart ? 1 : 2), rz, ctl.rz, ctl.beta);
          ctl.rz = rz;
          ctl.rr = rr;
          if (mode == kIter) {
            ++ctl.iters;
          } else {
            ctl.trigger = fmax(P.delta2 * ctl.rr_true, 0.25 * ctl.tol2);
            ctl.mode = kIter;
          }
          if (!isfinite(rr) || !isfinite(rz)) {
            ctl.st_inner = GFEA_ERR_NAN;
            ctl.mode = kUpdate;
          } else if (mode == kIter && rr <= ctl.trigger) {
            ctl.mode = kUpdate;
          } else if (ctl.iters >= P.max_iters) {
            ctl.st_inner = GFEA_ERR_NOT_CONVERGED;
            ctl.mode = kUpdate;
          } else if (rr <= ctl.trigger) {
            ctl.mode = kUpdate;
          }
        });
    if (!ok) break;
    turn = turn < 2 ? turn + 1 : 0;
    if (ctl.mode == kUpdate) continue;  // p is formed after the update

    // ---- p = z + beta p, z = y + R ec --------------------------------------
    const T bt = (T)ctl.beta;
    ++p_number;
    for (int i = tid; i < rows; i += kRT) {
      const int a = i / D;
      T z = q_s[i];
      if (nc && !kn_s[i]) z += prolong<D, T>(i - a * D, off_s + a * D, ecl_s + la_s[a] * nr);
      const T pn = z + bt * p_s[i];
      p_s[i] = pn;
      if (!solo) Pk::store(P.p + 2 * (a0 * D + i), pn, p_number);
    }
    if (solo || !pl_s) __syncthreads();
  }
  if (!ok && tid == 0) P.out->timed_out = 1;
  if (blockIdx.x == 0 && tid == 0) {
    gfea_pcg_result res{};
    res.status = ctl.status;
    res.iterations = ctl.iters;
    res.refinements = ctl.updates;
    const bool rel = ctl.bb > 0 && ctl.status != GFEA_ERR_SINGULAR;
    res.rel_residual = rel ? sqrt(ctl.rr_true / ctl.bb) : 0.0;
    res.floor_rel = rel ? sqrt(ctl.floor2 / ctl.bb) : 0.0;
    P.out->res = res;
  }
}

// Two CTAs, of which the second takes part in an exchange and publishes a
// packet, or leaves at once: the first one's waits end or run out.
__device__ __align__(16) double selftest_box[2 * 4 * 2 * 2 * 2 + 2];
__device__ int32_t selftest_exchanged;

__global__ void __launch_bounds__(kRT) exchange_selftest_kernel(uint64_t limit_ns, int present) {
  __shared__ double s_w[4][kRW];
  __shared__ double s_res[4];
  __shared__ int s_abort, s_ok;
  if (blockIdx.x == 1 && !present) return;
  if (threadIdx.x == 0) s_abort = 0;
  __syncthreads();
  Team team{selftest_box, 0, s_w, s_res, &s_abort, &s_ok, limit_ns};
  float* packet = reinterpret_cast<float*>(selftest_box + 2 * 4 * 2 * 2 * 2);
  const double w[1] = {1.0};
  double total = 0;
  bool ok = exchange<1, true>(team, w, [](int, int) {}, [&](const double* o) { total = o[0]; });
  if (blockIdx.x == 1) {
    if (threadIdx.x == 0) Packet<float>::store(packet, 3.f, 7);
    return;
  }
  const float v = await_packet<float>(packet, 7, &s_abort, limit_ns);
  __syncthreads();
  ok = ok && s_abort == 0;
  if (threadIdx.x == 0) selftest_exchanged = ok && total == 2.0 * kRW && v == 3.f ? GFEA_OK : GFEA_ERR_TIMEOUT;
}

template <int D, int G, typename T>
int launch(const ResidentProblem<T>& P, const ResidentGeom& g, cudaStream_t st) {
  auto kern = resident_kernel<D, G, T>;
  GFEA_CUDA_TRY(allow_smem(kern, kRSmemMax));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(g.grid);
  cfg.blockDim = dim3(kRT);
  cfg.dynamicSmemBytes = g.smem;
  cfg.stream = st;
  cudaLaunchAttribute a[1];
  a[0].id = cudaLaunchAttributeCooperative;
  a[0].val.cooperative = 1;
  cfg.attrs = a;
  cfg.numAttrs = g.grid > 1 ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, P, g);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();  // not sticky: taken back
    return kResidentRefused;
  }
  GFEA_CUDA_TRY(e);
  GFEA_LAUNCH_CHECK();
  return GFEA_OK;
}

}  // namespace

// Rows per CTA: enough to keep its threads busy, few enough to use many SMs; in
// 3D no more than 10,240 values (of HEXA8 139 rows, of HEXA27 65), by which a
// CTA's time goes there.  (In 2D more CTAs cost more in exchanges than they
// save: 12,261 TRI15 nodes, FP32, 96 CTAs 4.9 ms, 111 5.2, 152 5.4.)  Shared
// memory: room for rows of two (2D) and three times the average length.
// Numberings that take the corner nodes first (every quadratic mesh) give the
// first CTAs the long rows, which room for the average left to L2; all of it for
// every solve is 0.5 % slower.  In FP64, average room and 128 rows -> this, beside
// the multi-kernel iteration's: 425 HEXA27 nodes 4.75 -> 2.42 ms (3.22), 2,025
// 8.42 -> 3.97 (6.31), 600 HEXA20 6.21 -> 3.20 (4.79), 2,025 PRISM18 7.68 -> 3.82
// (5.60), 2,025 TETRA10 6.71 -> 3.61 (6.11).
template <typename T>
bool resident_geom(int D, int64_t Nn, int64_t n_pairs, int nc, int n_agg, int sms, ResidentGeom* g) {
  const double nb = (double)n_pairs / (double)Nn;
  int64_t rows = sizeof(T) == 8 ? 128 : 256;
  if (D == 3) rows = std::min<int64_t>(rows, std::max<int64_t>(32, (int64_t)(10240 / (nb * D))));
  if (const char* e = getenv("GFEA_RESIDENT_CTAS"))  // fewer, larger CTAs
    if (atoi(e) > 0) sms = std::min(sms, atoi(e));
  int64_t grid = ceil_div(Nn * D, rows);
  grid = std::min<int64_t>(std::max<int64_t>(grid, 1), std::min(sms, kSMs));
  const int64_t npc = ceil_div(Nn, grid);
  if (npc > 65535 / D) return false;
  g->npc = (int)npc;
  g->grid = (int)ceil_div(Nn, npc);
  if (n_agg > kAggWords * 32) return false;
  const size_t fixed = Layout<T>(D, g->npc, nc, n_agg, g->grid == 1).total;
  if (fixed > kRSmemMax / 2) return false;
  const double want = (double)fixed + (D == 3 ? 3.0 : 2.0) * npc * nb * (sizeof(T) * D * D + 2) +
                      (4 + sizeof(T) * D) * std::min<double>((double)Nn, npc * nb) + 8.0 * nc * (nc / g->grid + 1) + 4096;
  g->smem = (size_t)std::min<double>(want, (double)kRSmemMax);
  // lanes per node by the row length, as in the multi-kernel SpMV
  const double W = D * nb;
  g->lanes = D == 1 ? (W <= 10 ? 4 : 8) : (D == 2 ? (W <= 24 ? 8 : 16) : (W <= 56 ? 16 : 32));
  return true;
}

template <typename T>
int resident_launch(int D, const ResidentProblem<T>& P, const ResidentGeom& g, cudaStream_t st) {
  if constexpr (sizeof(T) == 8) {
    switch (D) {
      case 1: return launch<1, 8, T>(P, g, st);
      case 2: return launch<2, 8, T>(P, g, st);
      case 3: return launch<3, 16, T>(P, g, st);
    }
  } else {
    switch (D * 100 + g.lanes) {
      case 104: return launch<1, 4, T>(P, g, st);
      case 108: return launch<1, 8, T>(P, g, st);
      case 208: return launch<2, 8, T>(P, g, st);
      case 216: return launch<2, 16, T>(P, g, st);
      case 316: return launch<3, 16, T>(P, g, st);
      case 332: return launch<3, 32, T>(P, g, st);
    }
  }
  return GFEA_ERR_ARG;
}

template bool resident_geom<float>(int, int64_t, int64_t, int, int, int, ResidentGeom*);
template bool resident_geom<double>(int, int64_t, int64_t, int, int, int, ResidentGeom*);
template int resident_launch<float>(int, const ResidentProblem<float>&, const ResidentGeom&, cudaStream_t);
template int resident_launch<double>(int, const ResidentProblem<double>&, const ResidentGeom&, cudaStream_t);

}  // namespace gfea

using namespace gfea;

extern "C" int gfea_selftest_exchange(int32_t limit_us, int32_t present, int32_t* status_host, void* stream) {
  if (!status_host || limit_us < 1 || limit_us > 1000000) return GFEA_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int32_t unset = -1;
  void* box = nullptr;
  GFEA_CUDA_TRY(cudaGetSymbolAddress(&box, selftest_box));
  GFEA_CUDA_TRY(cudaMemsetAsync(box, 0, sizeof(selftest_box), st));
  GFEA_CUDA_TRY(cudaMemcpyToSymbolAsync(selftest_exchanged, &unset, sizeof(int32_t), 0, cudaMemcpyHostToDevice, st));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(2);
  cfg.blockDim = dim3(kRT);
  cfg.stream = st;
  cudaLaunchAttribute a[1];
  a[0].id = cudaLaunchAttributeCooperative;
  a[0].val.cooperative = 1;
  cfg.attrs = a;
  cfg.numAttrs = 1;
  GFEA_CUDA_TRY(cudaLaunchKernelEx(&cfg, exchange_selftest_kernel, (uint64_t)limit_us * 1000ull, (int)(present != 0)));
  GFEA_LAUNCH_CHECK();
  GFEA_CUDA_TRY(cudaMemcpyFromSymbolAsync(status_host, selftest_exchanged, sizeof(int32_t), 0, cudaMemcpyDeviceToHost,
                                          st));
  GFEA_CUDA_TRY(cudaStreamSynchronize(st));
  return GFEA_OK;
}
