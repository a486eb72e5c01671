// Betweenness centrality: the bc application (bc_np_consolidate_gpu,
// apps/bc/src/gpu/bc_wrapper.cu:678-741) with the results of its CPU version
// bc_cpu (apps/bc/src/cpu/bc.cpp:152-186, bc_kernel.cpp:3-106), bit for bit.
//
// Brandes' algorithm, one source per CTA.  The reference launches grid-wide
// kernels per BFS level of one source at a time, with a host round trip per
// level; here each source's levels run inside one CTA separated by
// __syncthreads (no grid barrier and no host round trip), and the grid works on
// many sources at once.
//
// Per source s (CTA-private scratch: level, sigma, the vertices in BFS order and
// the level bounds in that order; the source's delta row of a block buffer):
//   forward   level-synchronous BFS.  For an edge u -> v from the frontier
//             (level L), an unvisited v (level = MAX_LEVEL) takes level L + 1 by
//             atomicCAS and is appended to the order; if v is at level L + 1,
//             sigma[v] += sigma[u] (int, wrapping like the reference's
//             __sync_fetch_and_add; integer sums do not depend on order).
//             Rows of 32 edges or more are walked by a whole warp.
//   backward  deepest level first, one thread per vertex u of level L, its
//             edges in CSR order: for v at level L + 1,
//             delta[u] = (float)((double)delta[u] + (double)sigma[u] / sigma[v]
//                                 * (1.0f + delta[v]))
//             with the rounding of every step made explicit (no fused
//             multiply-add), as the reference's x86 code rounds it.
//   sum       bc[v] += delta_s[v] for every reached v other than s, in float, in
//             source order: a second kernel folds the block's delta rows into
//             bc in order, so the result equals the reference's sequential loop
//             over sources exactly.
//
// MAX_LEVEL = 9999 marks unvisited vertices as in the reference
// (common/global.h:17).  A vertex on level 9999 therefore still counts as unvisited there:
// every edge from level 9998 takes it into the order again, and so do edges from later
// levels, which move it behind themselves.  bc_sources_kernel<true> keeps that, with room
// for the repeated visits; the other kernels stop when a source gets that far, and the
// call starts again with it.  Path counts wrap as the reference's int sums do; where
// that gives 0 / 0 the result is NaN on both sides, but with different payloads
// (x86 writes 0xFFC00000, the GPU 0x7FFFFFFF), so NaNs match as NaNs only.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "nps.h"
#include "nps_internal.h"

namespace {

// 256-thread CTAs: 87.9 ms for every source of R-MAT scale 14, against 106 ms with
// 512 (fewer threads per source, more sources in flight; 128 gave 87.5 ms)
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int32_t kMaxLevel = 9999;
// Order entries beyond n for vertices taken more than once (only in graphs of more than
// kMaxLevel vertices); when they run out the call ends with NPS_ERR_CAPACITY.
constexpr size_t kDeepSlack = 4096;
__host__ __device__ constexpr size_t bc_order_entries(size_t n) { return n + (n > (size_t)kMaxLevel ? kDeepSlack : 0); }
constexpr int32_t kWarpRow = 32;  // rows of at least this many edges are walked by a warp (forward)

struct BcArgs {
  const int32_t* row;
  const int32_t* col;
  int32_t n;
  int64_t m;
  const int32_t* sources;  // null: source k is vertex k
  int32_t src_base;        // this block's sources are entries [src_base, src_base + count)
  int32_t count;
  int32_t* level;          // per CTA: n entries each
  int32_t* sigma;
  int32_t* order;          // per CTA: bc_order_entries(n) each
  int32_t* lb;             // per CTA: bc_order_entries(n) + 2 level bounds
  float* delta;            // count rows of n
  uint32_t* status;        // an error; [1]: the call starts again with another kernel (2: for level
                           // kMaxLevel), [2]: sources found narrow
  int32_t narrow;          // a source with fewer vertices than this up to level kLookLevel is narrow (0: none)
};

__device__ __forceinline__ void flag_format(uint32_t* status) { atomicCAS(status, 0u, (uint32_t)NPS_ERR_FORMAT); }

__device__ __forceinline__ bool row_ok(const BcArgs& a, int32_t u, int32_t& s, int32_t& e) {
  s = a.row[u];
  e = a.row[u + 1];
  if (s < 0 || e < s || (int64_t)e > a.m) {
    flag_format(a.status);
    s = e = 0;
    return false;
  }
  return true;
}

// Forward relaxation of edge k from a vertex of level L with path count su.  Below level
// kMaxLevel a vertex enters the order once, so it has room; else (DEEP) `cap` entries.
template <bool DEEP>
__device__ __forceinline__ void forward_edge(const BcArgs& a, int32_t* level, int32_t* sigma, int32_t* order,
                                             int32_t cap, int* s_tail, int64_t k, int32_t L, int32_t su) {
  const int32_t v = __ldg(a.col + k);
  if ((uint32_t)v >= (uint32_t)a.n) {
    flag_format(a.status);
    return;
  }
  int32_t lv = __ldcg(level + v);
  if (lv == kMaxLevel) {
    lv = atomicCAS(level + v, kMaxLevel, L + 1);
    if (lv == kMaxLevel) {
      lv = L + 1;
      const int32_t i = atomicAdd(s_tail, 1);
      if (!DEEP || i < cap) order[i] = v;
      else atomicCAS(a.status, 0u, (uint32_t)NPS_ERR_CAPACITY);
    }
  }
  if (lv == L + 1) atomicAdd(sigma + v, su);  // wraps as the reference's int sum does
}

template <bool DEEP>
__global__ void __launch_bounds__(kThreads) bc_sources_kernel(BcArgs a) {
  __shared__ int s_tail;
  __shared__ int s_nbig[2];  // per sweep parity: a count is reset one sweep after its last read
  __shared__ int32_t s_big[kThreads];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t n = (size_t)a.n;
  int32_t* level = a.level + blockIdx.x * n;
  int32_t* sigma = a.sigma + blockIdx.x * n;
  const int32_t cap = (int32_t)bc_order_entries(n);
  int32_t* order = a.order + blockIdx.x * (size_t)cap;
  int32_t* lb = a.lb + blockIdx.x * ((size_t)cap + 2);
  int sweep = 0;  // the same count in every thread
  if (tid == 0) s_nbig[0] = s_nbig[1] = 0;
  for (int j = blockIdx.x; j < a.count; j += gridDim.x) {
    const int32_t s = a.sources ? a.sources[a.src_base + j] : a.src_base + j;
    float* delta = a.delta + (size_t)j * n;
    for (size_t v = tid; v < n; v += kThreads) delta[v] = 0.0f;
    if (tid == 0) {
      level[s] = 0;
      sigma[s] = 1;
      order[0] = s;
      lb[0] = 0;
      lb[1] = DEEP || a.n < kMaxLevel || __ldcg(a.status + 1) == 0u;  // no frontier when the call starts again
      s_tail = 1;
    }
    __syncthreads();
    // ---- forward: the frontier is order[lb[L], lb[L + 1])
    int32_t L = 0;
    for (;;) {
      const int32_t lo = __ldcg(lb + L), hi = __ldcg(lb + L + 1);
      if (lo >= hi) break;
      for (int32_t base = lo; base < hi; base += kThreads, ++sweep) {  // the same sweeps for every thread
        const int par = sweep & 1;
        const int32_t i = base + tid;
        if (i < hi) {
          const int32_t u = __ldcg(order + i);
          int32_t rs, re;
          if (row_ok(a, u, rs, re)) {
            if (re - rs >= kWarpRow) {
              s_big[atomicAdd(&s_nbig[par], 1)] = u;  // at most one per thread per sweep
            } else {
              const int32_t su = __ldcg(sigma + u);
              for (int64_t k = rs; k < re; ++k) forward_edge<DEEP>(a, level, sigma, order, cap, &s_tail, k, L, su);
            }
          }
        }
        __syncthreads();
        const int nbig = s_nbig[par];
        if (tid == 0) s_nbig[par ^ 1] = 0;  // last read in the previous sweep, before the barrier above
        for (int b = warp; b < nbig; b += kWarps) {
          const int32_t u = s_big[b];
          const int32_t rs = a.row[u], re = a.row[u + 1];  // checked when listed
          const int32_t su = __ldcg(sigma + u);
          for (int64_t k = (int64_t)rs + lane; k < re; k += 32) forward_edge<DEEP>(a, level, sigma, order, cap, &s_tail, k, L, su);
        }
        __syncthreads();
      }
      __syncthreads();
      if (tid == 0) {
        int32_t end = DEEP ? min(s_tail, cap) : s_tail;
        if (!DEEP && L + 2 == kMaxLevel && end > hi) {  // level kMaxLevel may follow: an empty frontier instead
          atomicExch(a.status + 1, 2u);
          end = hi;
        }
        lb[L + 2] = end;
      }
      __syncthreads();
      ++L;
    }
    // here L = deepest level + 1.  ---- backward: levels L - 2 down to 1 (level 0 is
    // the source alone, whose delta is never summed; the deepest level's delta is 0)
    for (int32_t d = L - 2; d >= 1; --d) {
      const int32_t lo = __ldcg(lb + d), hi = __ldcg(lb + d + 1);
      for (int32_t i = lo + tid; i < hi; i += kThreads) {
        const int32_t u = __ldcg(order + i);
        const int32_t rs = a.row[u], re = a.row[u + 1];  // checked in the forward pass (else empty)
        if (rs < 0 || re < rs || (int64_t)re > a.m) continue;
        const double su = (double)__ldcg(sigma + u);
        float du = 0.0f;
        for (int64_t k = rs; k < re; ++k) {
          const int32_t v = __ldg(a.col + k);
          if ((uint32_t)v >= (uint32_t)a.n) continue;  // reported in the forward pass
          if (__ldcg(level + v) == d + 1) {
            const double q = __ddiv_rn(su, (double)__ldcg(sigma + v));
            const double t = __dmul_rn(q, (double)__fadd_rn(1.0f, __ldcg(delta + v)));
            du = __double2float_rn(__dadd_rn((double)du, t));
          }
        }
        delta[u] = du;
      }
      __syncthreads();
    }
    // ---- leave the scratch as found: every reached vertex back to unvisited
    const int32_t reached = DEEP ? min(s_tail, cap) : s_tail;
    for (int32_t i = tid; i < reached; i += kThreads) {
      const int32_t v = __ldcg(order + i);
      level[v] = kMaxLevel;
      sigma[v] = 0;
    }
    __syncthreads();
  }
}

// ---- the whole source in shared memory
//
// Level, path count, dependency and order of every vertex of a small graph fit an SM's
// shared memory (12 1/8 bytes per vertex).  The random accesses that bound the kernel
// above -- an L2 sector per edge and array -- then stay on the SM, and only the edges
// come from L2, in order.  A warp takes up to 32 vertices of the level (fewer when the
// level is small against the CTA), a stride apart: a level's long rows come first in the
// order, as most edges lead to them, and so spread over the items (R-MAT 14, every source:
// 57 ms with consecutive vertices).  It walks their rows flat, so a row's length does not
// hold a lane.  In the backward pass the lanes compute the terms of consecutive edges
// side by side; the float sum of a row, whose order and roundings are the reference's,
// is then formed by the lane that owns the row, from the terms in shared memory.
//
// What bounds it: instruction issue (ncu, R-MAT 14: 56 % of issue slots, ALU the busiest
// pipe) and the level barriers; shared memory and L2 are below half.  Measured against the
// kernel above: R-MAT 14, every source, 88 -> 34.4 ms; R-MAT 12 6.6 -> 2.2; uniform 6,209 x
// 23,666 4.5 -> 3.1; 380 sources of R-MAT 12 at edge factor 4 0.72 -> 0.14.  Of that: flat
// rows in shared memory 57 ms, items a stride apart 52, long rows without the owner search
// 44, their sums by ordered_sum 42, heads gathered before their terms are formed 34.
constexpr int kFwdEdges = 4;      // edges per lane and step, forward
constexpr int kBwdEdges = 2;      // ... and backward
constexpr int kSmemBounds = 256;  // level bounds kept in shared memory; deeper ones in a.lb
constexpr uint16_t kUnseen = 0xffff;
constexpr int32_t kLookLevel = 11;      // levels between looks whether the call goes on
static_assert(kMaxLevel % kLookLevel == 0, "a source looks before level kMaxLevel");
constexpr int32_t kLongRow = 32;        // rows of at least this many edges are walked one at a time

// Shared memory of a CTA of `threads` for a graph of n vertices.
__host__ __device__ constexpr size_t bc_smem_bytes(size_t n, int threads) {
  return (size_t)(threads / 32) * 32 * kBwdEdges * sizeof(double) + n * (4 + 4) + ((n + 31) / 32) * 4 +
         ((n + 1) & ~(size_t)1) * 4;
}

// Flat walk of one row per lane: the exclusive prefix and the total of their lengths.
__device__ __forceinline__ uint32_t flat_prefix(uint32_t d, int lane, uint32_t& excl) {
  uint32_t incl = d;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  excl = incl - d;
  return __shfl_sync(0xffffffffu, incl, 31);
}

// The lane whose row holds flat position k: the last one whose prefix is <= k.
__device__ __forceinline__ int flat_owner(uint32_t excl, uint32_t k) {
  int o = 0;
#pragma unroll
  for (int step = 16; step >= 1; step >>= 1) {
    const uint32_t x = __shfl_sync(0xffffffffu, excl, o + step);
    if (x <= k) o += step;
  }
  return o;
}

// du plus the terms t of lanes 0 .. n - 1 as the reference adds them: one after the other,
// each sum rounded to double and then to float.  One term at a time that is a chain of 51 cycles
// per term.  While the running sum stays in one binade [2^E, 2^(E+1)) it is a multiple m u
// of u = 2^(E-23), and adding t >= 0 gives (m + r) u: the first rounding, to multiples of
// 2^(E-52), and the second, to multiples of u, round t itself, whatever m is, unless t
// then lies halfway between two multiples of u (the one case that depends on m's parity).
// So the lanes round their terms at once (adding and subtracting 1.5 2^E and 1.5 2^(E+29)
// rounds to those multiples), a warp scan of the exact r u gives every running sum, and
// only a term that leaves the binade, is a tie, or is not small against the sum is added
// by itself.  Every lane returns the sum.
__device__ __forceinline__ float ordered_sum(float du, double t, uint32_t n, int lane) {
  constexpr unsigned kAll = 0xffffffffu;
  uint32_t pos = 0;
  for (int stops = 0; pos < n; ++stops) {
    const int eb = (int)(__float_as_uint(du) >> 23);  // biased exponent; 256 or more: negative
    if (eb < 64 || eb > 190 || stops == 8) {
      for (uint32_t c = pos; c < n; ++c) du = __double2float_rn(__dadd_rn((double)du, __shfl_sync(kAll, t, c)));
      break;
    }
    const int E = eb - 127 + 1023;  // as a double's biased exponent
    const double k1 = __hiloint2double(E << 20 | 0x80000, 0), k2 = __hiloint2double((E + 29) << 20 | 0x80000, 0);
    const double half = __hiloint2double((E - 24) << 20, 0), small = __hiloint2double((E - 1) << 20, 0);
    const double top = __hiloint2double((E + 1) << 20, 0);
    const bool in = (uint32_t)lane >= pos && (uint32_t)lane < n;
    const double z = __dadd_rn(__dadd_rn(t, k1), -k1), r = __dadd_rn(__dadd_rn(z, k2), -k2);
    const bool alone = in && (!(t >= 0.0 && t < small) || fabs(__dadd_rn(z, -r)) == half);
    double p = in && !alone ? r : 0.0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double q = __shfl_up_sync(kAll, p, o);
      if (lane >= o) p = __dadd_rn(p, q);
    }
    const double x = __dadd_rn((double)du, p);
    const uint32_t b = __ballot_sync(kAll, in && (alone || !(x < top)));
    const uint32_t f = b ? (uint32_t)__ffs(b) - 1u : n;  // terms before f are in
    if (f > pos) du = __double2float_rn(__shfl_sync(kAll, x, f - 1));
    if (f < n) du = __double2float_rn(__dadd_rn((double)du, __shfl_sync(kAll, t, f)));
    pos = f + 1;
  }
  return du;
}

// (512 threads: 40 registers, so that three CTAs fit an SM; R-MAT 12 takes 2.6 ms with 62 and
// two CTAs, 2.3 with three)
template <int NT>
__global__ void __launch_bounds__(NT, NT == 1024 ? 1 : (NT == 512 ? 3 : 4)) bc_smem_kernel(BcArgs a) {
  constexpr int NW = NT / 32;
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ double s_dyn[];
  __shared__ int s_tail, s_stop, s_item[2];
  __shared__ int32_t s_lb[kSmemBounds];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const int n = a.n, words = (n + 31) / 32;
  double* const term = s_dyn + warp * 32 * kBwdEdges;    // this warp's terms of short rows,
  int32_t* const head = reinterpret_cast<int32_t*>(term);  // or up to 95 heads of a long row
  int32_t* const sigma = reinterpret_cast<int32_t*>(s_dyn + NW * 32 * kBwdEdges);
  float* const delta = reinterpret_cast<float*>(sigma + n);
  uint32_t* const seen = reinterpret_cast<uint32_t*>(delta + n);
  uint16_t* const level = reinterpret_cast<uint16_t*>(seen + words);
  uint16_t* const order = level + ((n + 1) & ~1);
  int32_t* const lb = a.lb + (size_t)blockIdx.x * ((size_t)n + 2);
  auto bound = [&](int32_t L) { return L < kSmemBounds ? s_lb[L] : __ldcg(lb + L); };
  auto set_bound = [&](int32_t L, int32_t v) {
    if (L < kSmemBounds) s_lb[L] = v;
    else lb[L] = v;
  };
  // Thread 0, after level L of source j, at multiples of kLookLevel: whether the source ends
  // here, because the call takes the other kernel.  That is so when the next level, kMaxLevel,
  // has vertices (`more`), or a quarter of the first sources is narrow.  Sources end and begin
  // with an empty frontier then: an exit from the loops would cost each level 4 %.
  auto leave = [&](int32_t L, int j, bool more) {
    const bool vote = L + 1 == kLookLevel && j == (int)blockIdx.x && a.src_base == 0 && s_tail < a.narrow &&
                        4 * (atomicAdd(a.status + 2, 1u) + 1) >= gridDim.x;
    if (vote) atomicMax(a.status + 1, 1u);
    if (L + 1 == kMaxLevel && more) atomicMax(a.status + 1, 2u);
    s_stop = (n > kMaxLevel || a.narrow) && __ldcg(a.status + 1) != 0u;
    return s_stop != 0;
  };
  // Forward edge to v from a vertex of level L with path count su (lanes with `on`).
  auto reach = [&](int32_t v, int32_t su, bool on, int32_t L) {
    if (on && (uint32_t)v >= (uint32_t)n) {
      flag_format(a.status);
      on = false;
    }
    if (!on) return;
    uint32_t lv = level[v];
    if (lv == kUnseen) {
      const uint32_t bit = 1u << (v & 31);
      if ((atomicOr(&seen[v >> 5], bit) & bit) == 0u) {  // the first edge to reach v
        level[v] = (uint16_t)(L + 1);
        order[atomicAdd(&s_tail, 1)] = (uint16_t)v;
      }
      lv = (uint32_t)L + 1u;  // whoever was first was so in this level
    }
    if (lv == (uint32_t)L + 1u) atomicAdd(&sigma[v], su);  // wraps as the reference's int sum does
  };
  // Backward: the term of edge u -> v for u of level d with path count su, stored at the
  // lane's rank behind `base` when v is on level d + 1.  Returns who stored one.
  auto terms = [&](int32_t v, int32_t su, int32_t d, uint32_t base) {
    const bool on = (uint32_t)v < (uint32_t)n && level[v] == (uint32_t)d + 1u;
    const uint32_t b = __ballot_sync(kAll, on);
    if (on) {
      const double r = __ddiv_rn((double)su, (double)sigma[v]);
      term[base + __popc(b & lt)] = __dmul_rn(r, (double)__fadd_rn(1.0f, delta[v]));
    }
    return b;
  };
  for (int j = blockIdx.x; j < a.count; j += gridDim.x) {
    const int32_t src = a.sources ? a.sources[a.src_base + j] : a.src_base + j;
    for (int v = tid; v < n; v += NT) {
      sigma[v] = v == src;
      delta[v] = 0.0f;
      level[v] = v == src ? 0 : kUnseen;
    }
    for (int i = tid; i < words; i += NT) seen[i] = i == src / 32 ? 1u << (src % 32) : 0u;
    if (tid == 0) {
      order[0] = (uint16_t)src;
      s_stop = (n > kMaxLevel || a.narrow) && __ldcg(a.status + 1) != 0u;
      set_bound(0, 0);
      set_bound(1, s_stop ? 0 : 1);
      s_tail = 1;
      s_item[0] = s_item[1] = 0;
    }
    __syncthreads();
    int sweep = 0;  // levels walked: the item counter of a level is reset in the next one
    // ---- forward: the frontier is order[bound(L), bound(L + 1))
    int32_t L = 0;
    for (;; ++L, ++sweep) {
      const int32_t lo = bound(L), hi = bound(L + 1);
      if (lo >= hi) break;
      if (tid == 0) s_item[(sweep + 1) & 1] = 0;
      const int per = min(32, (hi - lo + NW - 1) / NW), items = (hi - lo + per - 1) / per;
      for (;;) {
        int it = 0;
        if (lane == 0) it = atomicAdd(&s_item[sweep & 1], 1);
        it = __shfl_sync(kAll, it, 0);
        if (it >= items) break;
        const int32_t i = lo + it + lane * items;
        int32_t rs = 0, re = 0, su = 0;
        if (lane < per && i < hi) {
          const int32_t u = order[i];
          row_ok(a, u, rs, re);
          su = sigma[u];
        }
        uint32_t lng = __ballot_sync(kAll, re - rs >= kLongRow), excl;
        const uint32_t total = flat_prefix(re - rs < kLongRow ? (uint32_t)(re - rs) : 0u, lane, excl);
        for (uint32_t k0 = 0; k0 < total; k0 += 32 * kFwdEdges) {
          int32_t v[kFwdEdges], s[kFwdEdges];
#pragma unroll
          for (int q = 0; q < kFwdEdges; ++q) {
            v[q] = -1;
            s[q] = 0;
            if (k0 + 32 * q >= total) continue;  // the whole warp
            const uint32_t k = k0 + 32 * q + lane;
            const int o = flat_owner(excl, k);
            const int32_t so = __shfl_sync(kAll, rs, o);
            const uint32_t eo = __shfl_sync(kAll, excl, o);
            s[q] = __shfl_sync(kAll, su, o);
            if (k < total) v[q] = __ldg(a.col + so + (int32_t)(k - eo));
          }
#pragma unroll
          for (int q = 0; q < kFwdEdges; ++q)
            if (k0 + 32 * q < total) reach(v[q], s[q], k0 + 32 * q + lane < total, L);
        }
        // long rows, one at a time: no search for an edge's owner
        while (lng) {
          const int o = __ffs(lng) - 1;
          lng &= lng - 1;
          const int32_t so = __shfl_sync(kAll, rs, o), eo = __shfl_sync(kAll, re, o);
          const int32_t s = __shfl_sync(kAll, su, o);
          const int32_t* c = a.col + so + lane;
          int32_t rest = eo - so;
          for (; rest >= 32 * kFwdEdges; rest -= 32 * kFwdEdges, c += 32 * kFwdEdges) {
            int32_t v[kFwdEdges];
#pragma unroll
            for (int q = 0; q < kFwdEdges; ++q) v[q] = __ldg(c + 32 * q);
#pragma unroll
            for (int q = 0; q < kFwdEdges; ++q) reach(v[q], s, true, L);
          }
          for (; rest > 0; rest -= 32, c += 32) reach(lane < rest ? __ldg(c) : 0, s, lane < rest, L);
        }
      }
      __syncthreads();
      if (tid == 0) {
        int32_t end = s_tail;
        if ((L + 1) % kLookLevel == 0 && leave(L, j, end > hi)) end = hi;  // an empty frontier
        set_bound(L + 2, end);
      }
      __syncthreads();
    }
    // ---- backward: levels L - 2 down to 1 (as in bc_sources_kernel)
    for (int32_t d = s_stop ? 0 : L - 2; d >= 1; --d, ++sweep) {
      const int32_t lo = bound(d), hi = bound(d + 1);
      if (tid == 0) s_item[(sweep + 1) & 1] = 0;
      const int per = min(32, (hi - lo + NW - 1) / NW), items = (hi - lo + per - 1) / per;
      for (;;) {
        int it = 0;
        if (lane == 0) it = atomicAdd(&s_item[sweep & 1], 1);
        it = __shfl_sync(kAll, it, 0);
        if (it >= items) break;
        const int32_t i = lo + it + lane * items;
        int32_t u = 0, rs = 0, re = 0, su = 0;
        const bool own = lane < per && i < hi;
        if (own) {
          u = order[i];
          rs = a.row[u];
          re = a.row[u + 1];
          if (rs < 0 || re < rs || (int64_t)re > a.m) rs = re = 0;  // reported in the forward pass
          su = sigma[u];
        }
        uint32_t lng = __ballot_sync(kAll, re - rs >= kLongRow), excl;
        const uint32_t deg = re - rs < kLongRow ? (uint32_t)(re - rs) : 0u;
        const uint32_t total = flat_prefix(deg, lane, excl);
        float du = 0.0f;
        for (uint32_t k0 = 0; k0 < total; k0 += 32 * kBwdEdges) {
          uint32_t b[kBwdEdges];
          int32_t v[kBwdEdges], s[kBwdEdges];
#pragma unroll
          for (int q = 0; q < kBwdEdges; ++q) {
            const uint32_t k = k0 + 32 * q + lane;
            const int o = flat_owner(excl, k);
            const int32_t so = __shfl_sync(kAll, rs, o);
            const uint32_t eo = __shfl_sync(kAll, excl, o);
            s[q] = __shfl_sync(kAll, su, o);
            v[q] = k < total ? __ldg(a.col + so + (int32_t)(k - eo)) : -1;
          }
          b[0] = terms(v[0], s[0], d, 0);
          b[1] = terms(v[1], s[1], d, __popc(b[0]));
          __syncwarp();
          // this lane's row: the terms of its edges in [k0, k0 + 64), in order
          if (deg && excl < k0 + 32 * kBwdEdges && excl + deg > k0) {
            const uint64_t on = (uint64_t)b[1] << 32 | b[0];
            const uint32_t p0 = max(excl, k0) - k0, p1 = min(excl + deg, k0 + 32 * kBwdEdges) - k0;
            const uint32_t c0 = __popcll(on & (((uint64_t)1 << p0) - 1));
            const uint32_t c1 = p1 >= 64 ? __popcll(on) : __popcll(on & (((uint64_t)1 << p1) - 1));
            for (uint32_t c = c0; c < c1; ++c) du = __double2float_rn(__dadd_rn((double)du, term[c]));
          }
          __syncwarp();
        }
        // long rows, one at a time; every lane forms the sum
        while (lng) {
          const int o = __ffs(lng) - 1;
          lng &= lng - 1;
          const int32_t so = __shfl_sync(kAll, rs, o), eo = __shfl_sync(kAll, re, o);
          const int32_t s = __shfl_sync(kAll, su, o);
          // heads on level d + 1 gather in order; 32 at a time the lanes form their terms
          float dl = 0.0f;
          uint32_t have = 0;
          auto flush = [&](uint32_t from, uint32_t cnt) {
            double t = 0.0;
            if ((uint32_t)lane < cnt) {
              const int32_t v = head[from + lane];
              t = __dmul_rn(__ddiv_rn((double)s, (double)sigma[v]), (double)__fadd_rn(1.0f, delta[v]));
            }
            dl = ordered_sum(dl, t, cnt, lane);
          };
          const int32_t* c = a.col + so + lane;
          int32_t rest = eo - so;
          int32_t v0 = lane < rest ? __ldg(c) : -1, v1 = 32 + lane < rest ? __ldg(c + 32) : -1;
          for (; rest > 0; rest -= 64) {
            const bool on0 = (uint32_t)v0 < (uint32_t)n && level[v0] == (uint32_t)d + 1u;
            const bool on1 = (uint32_t)v1 < (uint32_t)n && level[v1] == (uint32_t)d + 1u;
            const uint32_t b0 = __ballot_sync(kAll, on0), b1 = __ballot_sync(kAll, on1);
            if (on0) head[have + __popc(b0 & lt)] = v0;
            have += __popc(b0);
            if (on1) head[have + __popc(b1 & lt)] = v1;
            have += __popc(b1);
            c += 64;  // the next heads load while these are summed
            v0 = 64 + lane < rest ? __ldg(c) : -1;
            v1 = 96 + lane < rest ? __ldg(c + 32) : -1;
            if (have >= 32) {
              __syncwarp();
              flush(0, 32);
              if (have >= 64) flush(32, 32);
              // those left move down: no store beyond them, where the next step's heads go, and
              // a barrier before other lanes store those (a ballot alone orders no memory)
              const uint32_t done = have & ~31u;
              have -= done;
              const int32_t y = (uint32_t)lane < have ? head[done + lane] : 0;
              __syncwarp();
              if ((uint32_t)lane < have) head[lane] = y;
              __syncwarp();
            }
          }
          __syncwarp();
          if (have) flush(0, have);
          __syncwarp();
          if (lane == o) du = dl;
        }
        if (own) delta[u] = du;
      }
      __syncthreads();
    }
    float* const out = a.delta + (size_t)j * n;
    for (int v = tid; v < n; v += NT) out[v] = delta[v];
    __syncthreads();
  }
}
static_assert(kBwdEdges == 2, "two ballots make the mask of a backward step, and 128 words hold 95 heads");

// bc[v] += delta_j[v] for the block's sources j in order (float, one rounding per add).
__global__ void bc_fold_kernel(float* bc, const float* delta, int32_t n, int32_t count) {
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    float acc = bc[v];
    for (int32_t j = 0; j < count; ++j) acc = __fadd_rn(acc, __ldcs(delta + (size_t)j * n + v));
    bc[v] = acc;
  }
}

__global__ void bc_fill_kernel(int32_t* level, int32_t* sigma, size_t total) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    level[i] = kMaxLevel;
    sigma[i] = 0;
  }
}

__global__ void bc_check_sources_kernel(const int32_t* sources, int32_t nsrc, int32_t n, uint32_t* status) {
  for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nsrc; i += gridDim.x * blockDim.x)
    if ((uint32_t)sources[i] >= (uint32_t)n) atomicCAS(status, 0u, (uint32_t)NPS_ERR_INVALID_ARG);
}


using BcKernel = void (*)(BcArgs);

// The shared-memory kernel for n vertices, or null when they do not fit.  Threads per CTA
// follow from how many CTAs an SM then holds: one fills it with 1,024, two or more take
// 512 each, small graphs 256.
BcKernel bc_pick_smem(size_t n, int device, int* threads) {
  int limit = 0;
  if (cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) return nullptr;
  const size_t fixed = 2048;  // static shared memory
  if (bc_smem_bytes(n, 1024) + fixed > (size_t)limit) return nullptr;
  if (2 * (bc_smem_bytes(n, 512) + fixed) > (size_t)limit) {
    *threads = 1024;
    return bc_smem_kernel<1024>;
  }
  if (8 * (bc_smem_bytes(n, 256) + fixed) > (size_t)limit) {
    *threads = 512;
    return bc_smem_kernel<512>;
  }
  *threads = 256;
  return bc_smem_kernel<256>;
}

// The vertices below which a source counts as narrow (BcArgs::narrow) in a call of `count`
// sources, of which the shared-memory kernel holds `here` at once on `per_sm` CTAs per SM and
// bc_sources_kernel `there`.  A narrow source (a grid, a chain) costs its levels' latency, not
// its edges, so what counts is how many run at once, and state in shared memory leaves fewer:
// the other kernel takes the call when it needs so many rounds of sources less that its
// slower levels pay.  Its levels take 2.2 times as long on grids with one CTA per SM here, less
// with more CTAs, more with longer rows, which it walks by a thread each (lattices of degree 4
// / 8 / 32: 2.2 / 2.8 / 6), 3 to 6 times on random graphs just connected (degree below 2, the
// levels of which are not as small), and as long on paths.  ms of bc_sources_kernel / shared-memory
// kernel: 128 x 128 grid, 200 sources 2.31 / 1.92, 300 2.39 / 2.61, 2,000 5.1 / 11.6; 64 x 64
// grid, 600 sources 1.07 / 1.00, every source 3.7 / 5.4; 5,000-vertex path, 2,000 sources 23 /
// 52; 16,000-vertex ring, degree 32, 2,000 sources 30.6 / 32.4.  R-MAT and uniform graphs
// have a handful of levels and never ask.
int32_t bc_narrow_limit(int64_t n, int64_t m, int64_t count, int64_t here, int64_t there, int per_sm) {
  auto rounds = [&](int64_t at_once) {  // between whole rounds and their share
    const double r = (double)count / (double)at_once;
    return r <= 1.0 ? 1.0 : 0.5 * (r + std::ceil(r));
  };
  const double gain = rounds(here) / rounds(there), degree = (double)m / (double)n;
  const double slower = std::max(1.0, 2.45 - 0.25 * per_sm) * (degree < 2.0 ? 2.0 : std::max(1.0, 0.25 * degree));
  if (gain > slower) return 32 * kLookLevel;
  return gain > 1.0 ? 4 * kLookLevel : 0;
}

struct BcWork {
  unsigned long long ctx_id = 0;  // context the cached buffers live in (nps_context_id)
  std::mutex mu;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev[4] = {};
  int sms = 0;
  uint32_t* status = nullptr;
  int32_t* scratch = nullptr;  // level, sigma, order, lb for every CTA
  size_t scratch_n = 0;
  float* delta = nullptr;
  size_t delta_n = 0;
  int32_t* row = nullptr;
  size_t row_n = 0;
  int32_t* col = nullptr;
  size_t col_n = 0;
  int32_t* src = nullptr;
  size_t src_n = 0;
  float* bc = nullptr;
  size_t bc_n = 0;
};

std::mutex g_bc_mu;
std::vector<BcWork*> g_bc;


}  // namespace

extern "C" nps_status nps_bc(const int32_t* row_ptr, const int32_t* col, int32_t n, int64_t m,
                             const int32_t* sources, int32_t nsrc, const nps_params* pin, float* bc_out,
                             nps_stats* st) {
  nps_clear_error();
  nps_params p;
  if (pin) p = *pin;
  else nps_params_default(&p);
  if (n <= 0) return nps_fail(NPS_ERR_INVALID_ARG, "n must be positive");
  if (m < 0 || m >= (int64_t)INT32_MAX) return nps_fail(NPS_ERR_INVALID_ARG, "m must be in [0, 2^31-1)");
  if (!row_ptr || !bc_out || (m > 0 && !col)) return nps_fail(NPS_ERR_INVALID_ARG, "null array");
  if (sources && nsrc < 0) return nps_fail(NPS_ERR_INVALID_ARG, "nsrc must be >= 0");
  if (!p.device_ptrs && (row_ptr[0] != 0 || row_ptr[n] != (int32_t)m))
    return nps_fail(NPS_ERR_FORMAT, "malformed CSR: row_ptr[0] must be 0 and row_ptr[n] must be m");
  if (!p.device_ptrs && sources)
    for (int32_t i = 0; i < nsrc; ++i)
      if (sources[i] < 0 || sources[i] >= n) return nps_fail(NPS_ERR_INVALID_ARG, "bc: source out of range");
  const int32_t count_all = sources ? nsrc : n;
  int dcount = 0;
  if (cudaGetDeviceCount(&dcount) != cudaSuccess || dcount == 0) {
    cudaGetLastError();
    return nps_fail(NPS_ERR_NO_DEVICE, "no CUDA device");
  }
  if (p.device < 0 || p.device >= dcount) return nps_fail(NPS_ERR_INVALID_ARG, "device ordinal out of range");
  NPS_CUDA_RETURN(cudaSetDevice(p.device));
  BcWork* W;
  {
    std::lock_guard<std::mutex> lk(g_bc_mu);
    if ((int)g_bc.size() <= p.device) g_bc.resize(p.device + 1, nullptr);
    {
    const unsigned long long id = nps_context_id(p.device);
    if (g_bc[p.device] && id != 0 && g_bc[p.device]->ctx_id != id) g_bc[p.device] = nullptr;  // device reset: abandoned
    if (!g_bc[p.device]) {
      g_bc[p.device] = new BcWork();
      g_bc[p.device]->ctx_id = id;
    }
  }
    W = g_bc[p.device];
  }
  std::lock_guard<std::mutex> lk(W->mu);
  if (!W->stream) NPS_CUDA_RETURN(cudaStreamCreateWithFlags(&W->stream, cudaStreamNonBlocking));
  if (!W->ev[0])
    for (auto& ev : W->ev) NPS_CUDA_RETURN(cudaEventCreate(&ev));
  if (!W->status) NPS_CUDA_RETURN(cudaMalloc((void**)&W->status, 3 * sizeof(uint32_t)));
  if (!W->sms) NPS_CUDA_RETURN(cudaDeviceGetAttribute(&W->sms, cudaDevAttrMultiProcessorCount, p.device));
  cudaStream_t s = p.stream ? (cudaStream_t)p.stream : W->stream;
  if (st) memset(st, 0, sizeof(*st));
  nps_status e;
  NPS_CUDA_RETURN(cudaEventRecord(W->ev[0], s));
  const int32_t* drow = row_ptr;
  const int32_t* dcol = col;
  const int32_t* dsrc = sources;
  float* dbc = bc_out;
  if (!p.device_ptrs) {
    if ((e = nps_ensure(&W->row, &W->row_n, (size_t)n + 1, s, "bc")) || (e = nps_ensure(&W->col, &W->col_n, (size_t)m, s, "bc")) ||
        (e = nps_ensure(&W->bc, &W->bc_n, (size_t)n, s, "bc")))
      return e;
    NPS_CUDA_RETURN(cudaMemcpyAsync(W->row, row_ptr, sizeof(int32_t) * ((size_t)n + 1), cudaMemcpyHostToDevice, s));
    if (m > 0) NPS_CUDA_RETURN(cudaMemcpyAsync(W->col, col, sizeof(int32_t) * (size_t)m, cudaMemcpyHostToDevice, s));
    if (sources && nsrc > 0) {
      if ((e = nps_ensure(&W->src, &W->src_n, (size_t)nsrc, s, "bc"))) return e;
      NPS_CUDA_RETURN(cudaMemcpyAsync(W->src, sources, sizeof(int32_t) * (size_t)nsrc, cudaMemcpyHostToDevice, s));
      dsrc = W->src;
    }
    drow = W->row;
    dcol = W->col;
    dbc = W->bc;
  }
  if (dsrc && nsrc > 0 && p.device_ptrs) {  // a bad device-side source list stops the call before any kernel reads it
    uint32_t bad = 0;
    NPS_CUDA_RETURN(cudaMemsetAsync(W->status, 0, 3 * sizeof(uint32_t), s));
    bc_check_sources_kernel<<<(int)std::min<int64_t>(1024, ((int64_t)nsrc + 255) / 256), 256, 0, s>>>(dsrc, nsrc, n,
                                                                                               W->status);
    NPS_CUDA_RETURN(cudaGetLastError());
    NPS_CUDA_RETURN(cudaMemcpyAsync(&bad, W->status, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    NPS_CUDA_RETURN(cudaStreamSynchronize(s));
    if (bad) return nps_fail(NPS_ERR_INVALID_ARG, "bc: source out of range");
  }
  BcArgs a;
  a.row = drow;
  a.col = dcol;
  a.n = n;
  a.m = m;
  a.sources = dsrc;
  a.status = W->status;
  // one CTA per source at a time, as many CTAs as are resident; a block of
  // sources shares one delta buffer
  int smem_threads = 0;
  BcKernel smem_kernel = bc_pick_smem((size_t)n, p.device, &smem_threads);
  uint32_t h_status[3];
  bool deep = false;
  int grid = 0;
  for (bool first = true;; first = false) {
    const BcKernel kernel = smem_kernel ? smem_kernel : (deep ? bc_sources_kernel<true> : bc_sources_kernel<false>);
    const int threads = smem_kernel ? smem_threads : kThreads;
    const size_t dyn = smem_kernel ? bc_smem_bytes((size_t)n, threads) : 0;
    if (smem_kernel)
      NPS_CUDA_RETURN(cudaFuncSetAttribute((const void*)smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
    int per_sm = 0;
    NPS_CUDA_RETURN(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)kernel, threads, dyn));
    const size_t ordered = bc_order_entries((size_t)n);
    const size_t per_cta = smem_kernel ? (size_t)n + 2 : 2 * (size_t)n + 2 * ordered + 2;
    // at most 8 GB of CTA scratch (16 n bytes each): large graphs run fewer sources at once
    const int64_t by_memory = std::max<int64_t>(W->sms, (int64_t)((8ull << 30) / (per_cta * sizeof(int32_t))));
    grid = (int)std::max<int64_t>(
        1, std::min<int64_t>(std::min<int64_t>((int64_t)W->sms * std::max(1, per_sm), by_memory), count_all));
    a.narrow = 0;
    if (smem_kernel) {
      int other = 0;  // CTAs of bc_sources_kernel per SM
      NPS_CUDA_RETURN(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&other, (const void*)bc_sources_kernel<false>, kThreads, 0));
      a.narrow = bc_narrow_limit(n, m, count_all, grid, (int64_t)W->sms * std::max(1, other), per_sm);
    }
    if ((e = nps_ensure(&W->scratch, &W->scratch_n, per_cta * (size_t)grid, s, "bc"))) return e;
    const size_t budget = (size_t)1 << 31;  // bytes of delta rows per block
    int64_t cap = std::max<int64_t>(grid, budget / (4 * (size_t)n));
    if (p.reserved[1] > 0) cap = p.reserved[1];
    const int32_t block = (int32_t)std::max<int64_t>(1, std::min<int64_t>(count_all, cap));
    if ((e = nps_ensure(&W->delta, &W->delta_n, (size_t)block * (size_t)n, s, "bc"))) return e;
    NPS_CUDA_RETURN(cudaMemsetAsync(W->status, 0, 3 * sizeof(uint32_t), s));
    NPS_CUDA_RETURN(cudaMemsetAsync(dbc, 0, sizeof(float) * (size_t)n, s));
    if (smem_kernel) {
      a.level = a.sigma = a.order = nullptr;
      a.lb = W->scratch;
    } else {
      a.level = W->scratch;
      a.sigma = a.level + (size_t)n * grid;
      a.order = a.sigma + (size_t)n * grid;
      a.lb = a.order + ordered * grid;
      bc_fill_kernel<<<W->sms * 4, 256, 0, s>>>(a.level, a.sigma, (size_t)n * grid);
      NPS_CUDA_RETURN(cudaGetLastError());
    }
    a.delta = W->delta;
    if (first) NPS_CUDA_RETURN(cudaEventRecord(W->ev[1], s));
    const int fold_grid = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)n + 255) / 256, (int64_t)W->sms * 8));
    for (int32_t base = 0; base < count_all; base += block) {
      a.src_base = base;
      a.count = std::min<int32_t>(block, count_all - base);
      kernel<<<grid, threads, dyn, s>>>(a);
      NPS_CUDA_RETURN(cudaGetLastError());
      bc_fold_kernel<<<fold_grid, 256, 0, s>>>(dbc, W->delta, n, a.count);
      NPS_CUDA_RETURN(cudaGetLastError());
    }
    NPS_CUDA_RETURN(cudaEventRecord(W->ev[2], s));
    if (!p.device_ptrs) NPS_CUDA_RETURN(cudaMemcpyAsync(bc_out, dbc, sizeof(float) * (size_t)n, cudaMemcpyDeviceToHost, s));
    NPS_CUDA_RETURN(cudaMemcpyAsync(h_status, W->status, sizeof(h_status), cudaMemcpyDeviceToHost, s));
    NPS_CUDA_RETURN(cudaEventRecord(W->ev[3], s));
    NPS_CUDA_RETURN(cudaStreamSynchronize(s));
    if (!h_status[1]) break;
    deep = h_status[1] == 2;
    smem_kernel = nullptr;
  }
  if (st) {
    st->status = (int32_t)h_status[0];
    st->grid_ctas = grid;
    st->vertices_processed = (uint64_t)count_all;
    cudaEventElapsedTime(&st->kernel_ms, W->ev[1], W->ev[2]);
    cudaEventElapsedTime(&st->total_ms, W->ev[0], W->ev[3]);
  }
  if (h_status[0] == NPS_ERR_FORMAT)
    return nps_fail(NPS_ERR_FORMAT, "malformed CSR: a row range or column index is out of bounds");
  if (h_status[0] == NPS_ERR_CAPACITY)
    return nps_fail(NPS_ERR_CAPACITY, "bc: no room for the repeated visits of vertices on level 9999");
  return NPS_OK;
}
