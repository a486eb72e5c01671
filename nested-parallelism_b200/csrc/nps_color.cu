// Graph coloring: the graph-color application (gclr_np_consolidate_gpu,
// apps/graph-color/src/gpu/graph_color_wrapper.cu:368-412, kernels
// graph_color_kernel.cu:14-35 and :541-723).
//
// The reference colors in iterations c = 1, 2, ...: an uncolored vertex v takes
// color c when none of its out-neighbours u < v is uncolored or colored c
// (graph_color_kernel.cu:19-32); it stops when every vertex is colored.  A
// neighbour that takes color c in the same iteration blocks v whether v sees it
// before or after, so the result does not depend on scheduling:
//     color(v) = 1 + max { color(u) : u in the row of v, u < v }
// (1 when v has no smaller out-neighbour), and the iteration count is the
// largest color.  The reference tests every uncolored vertex in every iteration.
//
// Here every edge is read once, by one kernel without barriers.  The vertices are cut, in
// id order, into units for a warp: a run of up to 32 consecutive rows below kLong edges,
// or a chunk of kChunk edges of a longer row (the warp and grid consolidation of long
// rows).  Warps claim units from a ticket counter, in that order, walk their edges and
// look up the colors of the smaller neighbours.  Neighbours still without a color (0) go
// to the warp's list in shared memory, which it polls until each of them has one; a
// vertex whose smaller neighbours all have colors takes its own at once (the last chunk
// of a long row does it).  A vertex waits only for smaller ids, whose units have smaller
// tickets, each claimed by a warp that is running: the first unit not finished never
// waits, so every wait ends, whatever is resident.  A color is one word, written once, so
// no ordering between words is needed.  Each wait is bounded: it ends the call when for
// timeout_s neither its list shrinks nor any warp claims a unit, which each does when it
// finishes one.
//
// What bounds it: the chain of dependent colors, each link a store and the poll that sees
// it (R-MAT scale 22: 1,295 links, 1.6 us each), beside 33 M random 4-byte lookups, of
// which the hubs' hit in L1.  Measured, kernel time, against rounds over reverse lists
// with two grid barriers per color: R-MAT 22 42.8 -> 2.03 ms, R-MAT 20 19.1 -> 1.09, R-MAT
// 12 1.12 -> 0.08, 2048 x 2048 grid 38.7 -> 10.7, a 5,000-color chain 30.6 -> 1.2, a
// 300,000-edge row 6.5 -> 0.04, uniform 1 M x 8 M 1.06 -> 0.12.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "nps.h"
#include "nps_internal.h"

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kScanItems = 1024;  // elements per CTA of the scan (4 per thread)
constexpr int kEdges = 4;         // edges per lane and step of a run
constexpr int kChunkEdges = 8;    // ... and of a chunk
// Chunks of 1,024 and rows from 64 edges on: a long row is a unit of its own, so it is not
// walked after, or polled with, 31 others, and most long rows are one chunk.  R-MAT scale
// 22 (kernel ms at kChunk / kLong, 2 CTAs per SM): 1024/64 2.03, 1024/128 2.03, 1024/256
// 2.14, 512/64 2.20, 512/32 2.24, 256/64 2.67; 1024/1024, before chunk sums shared a word, 4.1.
constexpr int32_t kChunk = 1024;  // edges per chunk
constexpr int32_t kLong = 64;     // rows of at least this many edges are cut into chunks
// CTAs per SM: more vertices in flight find more neighbours without a color, and poll for
// them; fewer leave too few rows in flight where colors are few.  Kernel ms at 1 / 2 / 3 / 5:
// R-MAT 22 2.09 / 2.03 / 2.10 / 2.45, R-MAT 20 1.00 / 1.09 / 1.21 / 1.58, 2048 x 2048 grid
// 12.9 / 10.7 / 9.4 / 8.4, uniform 1 M x 8 M 0.19 / 0.12 / 0.10 / 0.10.
constexpr int kCtasPerSm = 2;
constexpr int kList = 384;        // neighbours without a color a run can hold; a step adds at most 128
constexpr int kPoll = 2;          // list entries per lane looked up together
constexpr unsigned kFull = 0xffffffffu;
static_assert(kChunk * sizeof(int32_t) <= 4096 && kList * sizeof(int2) <= 4096, "list memory of a warp");

struct ColorCtr {
  uint32_t next;    // ticket: units claimed
  uint32_t status;
  uint32_t abort;   // a wait ran out: every warp stops
  int32_t max_color;
  unsigned long long edges;  // edges to smaller vertices
  unsigned long long total;  // edges of all rows: more than m when the row offsets are malformed
};

struct ColorArgs {
  const int32_t* row;
  const int32_t* col;
  int32_t n;
  int64_t m;
  int32_t* color;   // zeroed before the launch
  int32_t* ucount;  // units per group of 32 vertices, then their exclusive scan within a scan CTA
  int32_t* ubase;   // per scan CTA: the units before it; the last entry: all units
  int32_t nscan;    // scan CTAs
  int4* unit;       // run {first vertex, vertices, 0, 0}; chunk {vertex, edge begin, edge end, chunks of the row}
  unsigned long long* lrow;  // long rows: (chunks not finished << 32) | the largest color among the
                             // smaller neighbours in the finished ones
  unsigned long long timeout_ns;
  uint32_t inject;  // test hook: the first group waits for a color that never comes
  ColorCtr* c;
};

__device__ __forceinline__ void flag_format(ColorCtr* c) { atomicCAS(&c->status, 0u, (uint32_t)NPS_ERR_FORMAT); }

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t ld_relaxed_u32(const void* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_relaxed(int32_t* p, int32_t v) {
  asm volatile("st.relaxed.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Columns are read once: no L1 allocation, so that L1 keeps the colors.
__device__ __forceinline__ int32_t ld_col(const int32_t* p) {
  int32_t v;
  asm volatile("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// First lookup of a color, through L1: an old copy can only show 0 for a color that is
// there by now, and then the poll, which reads past L1, finds it.
__device__ __forceinline__ int32_t ld_color(const int32_t* p) {
  int32_t v;
  asm volatile("ld.global.ca.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Row of vertex v; malformed bounds are reported and taken as an empty row.
__device__ __forceinline__ void row_bounds(const ColorArgs& a, int64_t v, int32_t& s, int32_t& e) {
  s = e = 0;
  if (v >= a.n) return;
  s = a.row[v];
  e = a.row[v + 1];
  if (s < 0 || e < s || (int64_t)e > a.m) {
    flag_format(a.c);
    s = e = 0;
  }
}

// Units of a group of 32 vertices, of which this lane's row has `d` edges: runs between
// its long rows, and their chunks.  Every lane gets the group's total and its own unit
// offset; the lane of a run's first vertex or of a long row has units to write.
__device__ __forceinline__ uint32_t group_units(int32_t d, int64_t v, int32_t n, int lane, uint32_t& first,
                                                uint32_t& count, uint32_t& run) {
  const bool in = v < n, lng = in && d >= kLong;
  const uint32_t lm = __ballot_sync(kFull, lng), im = __ballot_sync(kFull, in);
  // a run starts at a row that is not long and is lane 0's or follows a long one
  const bool start = in && !lng && (lane == 0 || ((lm >> (lane - 1)) & 1u));
  const uint32_t after = (lm | ~im) & ~((1u << lane) - 1u);
  run = start ? (after ? (uint32_t)__ffs(after) - 1u : 32u) - lane : 0u;
  count = lng ? (uint32_t)((d + kChunk - 1) / kChunk) : start;
  uint32_t incl = count;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  first = incl - count;
  return __shfl_sync(kFull, incl, 31);
}

__global__ void __launch_bounds__(kThreads) color_count_kernel(ColorArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t groups = ((int64_t)a.n + 31) / 32, warps = (int64_t)gridDim.x * kWarps;
  unsigned long long sum = 0;
  for (int64_t g = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5); g < groups; g += warps) {
    int32_t s, e;
    row_bounds(a, g * 32 + lane, s, e);
    sum += (unsigned long long)(e - s);
    uint32_t first, count, run;
    const uint32_t total = group_units(e - s, g * 32 + lane, a.n, lane, first, count, run);
    if (lane == 0) a.ucount[g] = (int32_t)total;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
  if (lane == 0 && sum) atomicAdd(&a.c->total, sum);
}

// Rows that overlap hold more than m edges, and more units than the table: nothing is
// colored then, the call reports the format error.
__device__ __forceinline__ bool overlapping(const ColorArgs& a) {
  if (a.c->total <= (unsigned long long)a.m) return false;
  if (threadIdx.x == 0) flag_format(a.c);
  return true;
}

// Exclusive scan of the units per group: per-CTA scans of kScanItems and a single CTA over
// the CTA totals; the unit kernel adds the two.
__global__ void __launch_bounds__(kThreads) scan_blocks_kernel(int32_t* x, int32_t n, int32_t* bsum) {
  __shared__ int32_t s_warp[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = (int64_t)blockIdx.x * kScanItems + threadIdx.x * 4;
  int32_t v[4], t = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[i] = base + i < n ? x[base + i] : 0;
    t += v[i];
  }
  int32_t incl = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  int32_t woff = 0;
  for (int w = 0; w < warp; ++w) woff += s_warp[w];
  int32_t run = woff + incl - t;  // exclusive prefix of this thread's first element within the CTA
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (base + i < n) x[base + i] = run;
    run += v[i];
  }
  if (threadIdx.x == kThreads - 1) bsum[blockIdx.x] = woff + incl;
}

__global__ void __launch_bounds__(kThreads) scan_totals_kernel(int32_t* bsum, int32_t nb, int32_t* total) {
  __shared__ int32_t s_carry;
  __shared__ int32_t s_warp[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (int32_t base = 0; base < nb; base += kThreads) {
    const int32_t i = base + threadIdx.x;
    const int32_t t = i < nb ? bsum[i] : 0;
    int32_t incl = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    int32_t woff = 0;
    for (int w = 0; w < warp; ++w) woff += s_warp[w];
    if (i < nb) bsum[i] = s_carry + woff + incl - t;
    __syncthreads();
    if (threadIdx.x == kThreads - 1) s_carry += woff + incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = s_carry;
}

// The unit table, and the state of the long rows.
__global__ void __launch_bounds__(kThreads) color_units_kernel(ColorArgs a) {
  if (overlapping(a)) return;
  const int lane = threadIdx.x & 31;
  const int64_t groups = ((int64_t)a.n + 31) / 32, warps = (int64_t)gridDim.x * kWarps;
  for (int64_t g = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5); g < groups; g += warps) {
    const int64_t v = g * 32 + lane;
    int32_t s, e;
    row_bounds(a, v, s, e);
    uint32_t first, count, run;
    group_units(e - s, v, a.n, lane, first, count, run);
    const uint32_t base = (uint32_t)a.ucount[g] + (uint32_t)a.ubase[g / kScanItems];
    if (run) a.unit[base + first] = make_int4((int32_t)v, (int32_t)run, 0, 0);
    else if (count) a.lrow[v] = (unsigned long long)count << 32;
    uint32_t todo = __ballot_sync(kFull, count > 0 && run == 0);
    while (todo) {  // the chunks of one long row at a time
      const int j = __ffs(todo) - 1;
      todo &= todo - 1;
      const int32_t js = __shfl_sync(kFull, s, j), je = __shfl_sync(kFull, e, j);
      const uint32_t jb = base + __shfl_sync(kFull, first, j), jn = __shfl_sync(kFull, count, j);
      for (uint32_t i = lane; i < jn; i += 32) {
        const int64_t cs = (int64_t)js + (int64_t)i * kChunk;
        a.unit[jb + i] = make_int4((int32_t)(g * 32 + j), (int32_t)cs, (int32_t)min((int64_t)je, cs + kChunk),
                                   (int32_t)jn);
      }
    }
  }
}

// A warp's wait: counted from the last time an entry left its list or the ticket moved.
// (The last of a window of vertices waits for the colors of all others: 18 ms on a path,
// however short the timeout.)
struct Wait {
  unsigned long long since;
  uint32_t spins, next;
};

// After a poll that changed nothing: true when the warp must stop, because this wait or
// another one ran out.
__device__ __forceinline__ bool wait_more(const ColorArgs& a, Wait& w, int lane) {
  if ((++w.spins & 63u) == 0) {
    uint32_t quit = 0;
    if (lane == 0) {
      const unsigned long long now = globaltimer_ns();
      const uint32_t next = ld_relaxed_u32(&a.c->next);
      if (w.since == 0 || next != w.next) w.since = now;
      w.next = next;
      quit = ld_relaxed_u32(&a.c->abort) != 0;
      if (!quit && now - w.since > a.timeout_ns) {
        atomicCAS(&a.c->status, 0u, (uint32_t)NPS_ERR_TIMEOUT);
        atomicExch(&a.c->abort, 1u);
        quit = 1;
      }
    }
    if (__shfl_sync(kFull, quit, 0)) return true;
  }
  __nanosleep(20);
  return false;
}

struct Warp {
  int4* mem;      // list memory, 4 KB
  int32_t* best;  // runs, per lane: the largest color among the smaller neighbours so far
  int32_t* wait;  // runs, per lane: neighbours in the list, plus one until the row is walked
  int32_t* mine;  // runs, per lane: the vertex's color, 0 while it has none
};

// A run: vertices base + lane for lane < count, their rows walked flat.  A run's own
// vertices pass their colors through shared memory.  Returns false when stopped.
__device__ __forceinline__ bool color_run(const ColorArgs& a, const Warp& W, int32_t base, int32_t count,
                                          uint32_t inject, int lane, int32_t& most, unsigned long long& edges) {
  int2* const list = reinterpret_cast<int2*>(W.mem);  // {neighbour without a color, lane that waits for it}
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t len = 0;
  bool done = lane >= count, walked = done;
  int32_t s, e;
  row_bounds(a, done ? (int64_t)a.n : (int64_t)base + lane, s, e);
  W.best[lane] = 0;
  W.wait[lane] = 1 + (lane == 0 ? (int32_t)inject : 0);
  W.mine[lane] = 0;
  const uint32_t d = (uint32_t)(e - s);
  uint32_t incl = d;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  const uint32_t excl = incl - d, total = __shfl_sync(kFull, incl, 31);
  __syncwarp();
  Wait w = {0ull, 0u, 0u};
  for (uint32_t k0 = 0;;) {
    if (!walked && incl <= k0) {  // this lane's row is walked
      atomicSub(&W.wait[lane], 1);
      walked = true;
    }
    __syncwarp();
    if (!done && W.wait[lane] == 0) {
      const int32_t c = W.best[lane] + 1;
      st_relaxed(a.color + base + lane, c);
      W.mine[lane] = c;
      most = max(most, c);
      done = true;
    }
    __syncwarp();
    if (__all_sync(kFull, done)) return true;
    if (k0 < total && len <= (uint32_t)(kList - 32 * kEdges)) {
      int32_t u[kEdges], c[kEdges];
      int own[kEdges];
#pragma unroll
      for (int j = 0; j < kEdges; ++j) {
        const uint32_t k = k0 + 32 * j + lane;
        int o = 0;  // the last lane whose prefix is <= k
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
          const uint32_t x = __shfl_sync(kFull, excl, o + step);
          if (x <= k) o += step;
        }
        const int32_t so = __shfl_sync(kFull, s, o);
        const uint32_t eo = __shfl_sync(kFull, excl, o);
        own[j] = k < total ? o : -1;
        u[j] = k < total ? ld_col(a.col + so + (int32_t)(k - eo)) : 0;
      }
#pragma unroll
      for (int j = 0; j < kEdges; ++j) {
        if ((uint32_t)u[j] >= (uint32_t)a.n) {  // neighbour id outside [0, n): reported and skipped
          flag_format(a.c);
          own[j] = -1;
        } else if (u[j] >= base + own[j]) {
          own[j] = -1;  // not a smaller vertex
        }
        c[j] = own[j] >= 0 && u[j] < base ? ld_color(a.color + u[j]) : 0;
      }
#pragma unroll
      for (int j = 0; j < kEdges; ++j) {
        const bool open = own[j] >= 0 && c[j] == 0;
        if (own[j] >= 0) {
          edges += 1;
          if (open) atomicAdd(&W.wait[own[j]], 1);
          else if (c[j] > W.best[own[j]]) atomicMax(&W.best[own[j]], c[j]);
        }
        const uint32_t b = __ballot_sync(kFull, open);
        if (open) list[len + __popc(b & lt)] = make_int2(u[j], own[j]);
        len += __popc(b);
      }
      k0 += 32 * kEdges;
      continue;
    }
    if (k0 >= total && len <= 64) {
      // the rows are walked and the list fits two entries per lane: poll it from registers
      int2 x[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) x[j] = 32 * j + lane < len ? list[32 * j + lane] : make_int2(0, -1);
      for (;;) {
        bool got = false;
        int32_t c[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          c[j] = 0;
          if (x[j].y >= 0)
            c[j] = x[j].x >= base ? W.mine[x[j].x - base] : (int32_t)ld_relaxed_u32(a.color + x[j].x);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
          if (c[j] > 0) {
            atomicMax(&W.best[x[j].y], c[j]);
            atomicSub(&W.wait[x[j].y], 1);
            x[j].y = -1;
            got = true;
          }
        __syncwarp();
        if (__any_sync(kFull, got)) {
          w.since = 0;
          if (!done && W.wait[lane] == 0) {
            const int32_t cv = W.best[lane] + 1;
            W.mine[lane] = cv;
            st_relaxed(a.color + base + lane, cv);
            most = max(most, cv);
            done = true;
          }
          __syncwarp();
          if (__all_sync(kFull, done)) return true;
        } else if (wait_more(a, w, lane)) {
          return false;
        }
      }
    }
    // poll the list
    uint32_t kept = 0;
    for (uint32_t i0 = 0; i0 < len; i0 += 32 * kPoll) {
      int2 x[kPoll];
      int32_t c[kPoll];
#pragma unroll
      for (int j = 0; j < kPoll; ++j) {
        const uint32_t i = i0 + 32 * j + lane;
        x[j] = i < len ? list[i] : make_int2(0, -1);
        c[j] = 0;
        if (x[j].y >= 0) c[j] = x[j].x >= base ? W.mine[x[j].x - base] : (int32_t)ld_relaxed_u32(a.color + x[j].x);
      }
      __syncwarp();  // read before entries move down
#pragma unroll
      for (int j = 0; j < kPoll; ++j) {
        if (c[j] > 0) {
          if (c[j] > W.best[x[j].y]) atomicMax(&W.best[x[j].y], c[j]);
          atomicSub(&W.wait[x[j].y], 1);
        }
        const bool keep = x[j].y >= 0 && c[j] == 0;
        const uint32_t b = __ballot_sync(kFull, keep);
        if (keep) list[kept + __popc(b & lt)] = x[j];
        kept += __popc(b);
      }
      __syncwarp();
    }
    if (kept < len) w.since = 0;
    else if (wait_more(a, w, lane)) return false;
    len = kept;
  }
}

// A chunk [s, e) of the row of v, one of nch.  Returns false when stopped.
__device__ __forceinline__ bool color_chunk(const ColorArgs& a, const Warp& W, int32_t v, int32_t s, int32_t e,
                                            int32_t nch, uint32_t inject, int lane, int32_t& most,
                                            unsigned long long& edges) {
  int32_t* const list = reinterpret_cast<int32_t*>(W.mem);
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t len = 0;
  int32_t best = 0;
  __syncwarp();
  for (int64_t k0 = s; k0 < e; k0 += 32 * kChunkEdges) {
    int32_t u[kChunkEdges], c[kChunkEdges];
#pragma unroll
    for (int j = 0; j < kChunkEdges; ++j) u[j] = k0 + 32 * j + lane < e ? ld_col(a.col + k0 + 32 * j + lane) : v;
#pragma unroll
    for (int j = 0; j < kChunkEdges; ++j) {
      if ((uint32_t)u[j] >= (uint32_t)a.n) {  // neighbour id outside [0, n): reported and skipped
        flag_format(a.c);
        u[j] = v;
      }
      c[j] = u[j] < v ? ld_color(a.color + u[j]) : 1;
    }
#pragma unroll
    for (int j = 0; j < kChunkEdges; ++j) {
      if (u[j] < v) {
        edges += 1;
        best = max(best, c[j]);
      }
      const uint32_t b = __ballot_sync(kFull, c[j] == 0);
      if (c[j] == 0) list[len + __popc(b & lt)] = u[j];
      len += __popc(b);
    }
  }
  __syncwarp();
  // all of them must have colors, in whatever order they get them: wait for kPoll entries
  // per lane at a time, so that a poll never goes over the whole list
  Wait w = {0ull, 0u, 0u};
  while (inject)
    if (wait_more(a, w, lane)) return false;
  for (uint32_t i0 = 0; i0 < len; i0 += 32 * kPoll) {
    int32_t x[kPoll];
    bool open[kPoll];
#pragma unroll
    for (int j = 0; j < kPoll; ++j) {
      const uint32_t i = i0 + 32 * j + lane;
      open[j] = i < len;
      x[j] = open[j] ? list[i] : 0;
    }
    for (uint32_t left = 0, now = 1; now; left = now) {
      int32_t c[kPoll];
#pragma unroll
      for (int j = 0; j < kPoll; ++j) c[j] = open[j] ? (int32_t)ld_relaxed_u32(a.color + x[j]) : 0;
      now = 0;
#pragma unroll
      for (int j = 0; j < kPoll; ++j) {
        best = max(best, c[j]);
        open[j] = open[j] && c[j] == 0;
        now += __popc(__ballot_sync(kFull, open[j]));
      }
      if (now != left) w.since = 0;
      else if (now && wait_more(a, w, lane)) return false;
    }
  }
  best = __reduce_max_sync(kFull, best);
  if (lane == 0) {
    // one word holds both: a maximum and a count of their own would need a fence between
    bool last = nch == 1;
    if (!last) {
      unsigned long long old = __ldcg(a.lrow + v), now;
      for (;;) {
        now = ((old >> 32) - 1) << 32 | (uint32_t)max((int32_t)(uint32_t)old, best);
        const unsigned long long got = atomicCAS(a.lrow + v, old, now);
        if (got == old) break;
        old = got;
      }
      last = (now >> 32) == 0;
      best = (int32_t)(uint32_t)now;
    }
    if (last) {
      st_relaxed(a.color + v, best + 1);
      most = max(most, best + 1);
    }
  }
  return true;
}

__global__ void __launch_bounds__(kThreads) color_kernel(ColorArgs a) {
  __shared__ int4 s_mem[kWarps][256];
  __shared__ int32_t s_best[kWarps][32], s_wait[kWarps][32], s_mine[kWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Warp W = {s_mem[warp], s_best[warp], s_wait[warp], s_mine[warp]};
  if (overlapping(a)) return;
  const uint32_t units = (uint32_t)a.ubase[a.nscan];
  int32_t most = 0;
  unsigned long long edges = 0;
  for (bool go = true; go;) {
    uint32_t t = 0;
    if (lane == 0) t = atomicAdd(&a.c->next, 1u);
    t = __shfl_sync(kFull, t, 0);
    if (t >= units) break;
    const int4 u = a.unit[t];
    const uint32_t inject = t == 0 ? a.inject : 0u;
    go = u.w ? color_chunk(a, W, u.x, u.y, u.z, u.w, inject, lane, most, edges)
             : color_run(a, W, u.x, u.y, inject, lane, most, edges);
  }
  most = __reduce_max_sync(kFull, most);
#pragma unroll
  for (int o = 16; o; o >>= 1) edges += __shfl_xor_sync(kFull, edges, o);
  if (lane == 0) {
    if (edges) atomicAdd(&a.c->edges, edges);
    if (most) atomicMax(&a.c->max_color, most);
  }
}

struct ColorWork {
  unsigned long long ctx_id = 0;  // context the cached buffers live in (nps_context_id)
  std::mutex mu;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev[4] = {};
  int sms = 0;
  ColorCtr* ctr = nullptr;
  ColorCtr* snap = nullptr;  // pinned copy of the counters
  int32_t* state = nullptr;  // units per group, scan totals
  size_t state_n = 0;
  unsigned long long* lrow = nullptr;
  size_t lrow_n = 0;
  int4* unit = nullptr;
  size_t unit_n = 0;
  int32_t* row = nullptr;
  size_t row_n = 0;
  int32_t* col = nullptr;
  size_t col_n = 0;
  int32_t* color = nullptr;
  size_t color_n = 0;
};

std::mutex g_color_mu;
std::vector<ColorWork*> g_color;


}  // namespace

extern "C" nps_status nps_color(const int32_t* row_ptr, const int32_t* col, int32_t n, int64_t m,
                                const nps_params* pin, int32_t* color_out, nps_stats* st) {
  nps_clear_error();
  nps_params p;
  if (pin) p = *pin;
  else nps_params_default(&p);
  if (p.threshold < 1) return nps_fail(NPS_ERR_INVALID_ARG, "threshold must be >= 1");
  if (!(p.timeout_s > 0) || p.timeout_s > 3600) return nps_fail(NPS_ERR_INVALID_ARG, "timeout_s must be in (0, 3600]");
  if (n <= 0) return nps_fail(NPS_ERR_INVALID_ARG, "n must be positive");
  if (m < 0 || m >= (int64_t)INT32_MAX) return nps_fail(NPS_ERR_INVALID_ARG, "m must be in [0, 2^31-1)");
  if (!row_ptr || !color_out || (m > 0 && !col)) return nps_fail(NPS_ERR_INVALID_ARG, "null array");
  if (!p.device_ptrs && (row_ptr[0] != 0 || row_ptr[n] != (int32_t)m))
    return nps_fail(NPS_ERR_FORMAT, "malformed CSR: row_ptr[0] must be 0 and row_ptr[n] must be m");
  int dcount = 0;
  if (cudaGetDeviceCount(&dcount) != cudaSuccess || dcount == 0) {
    cudaGetLastError();
    return nps_fail(NPS_ERR_NO_DEVICE, "no CUDA device");
  }
  if (p.device < 0 || p.device >= dcount) return nps_fail(NPS_ERR_INVALID_ARG, "device ordinal out of range");
  NPS_CUDA_RETURN(cudaSetDevice(p.device));
  ColorWork* W;
  {
    std::lock_guard<std::mutex> lk(g_color_mu);
    if ((int)g_color.size() <= p.device) g_color.resize(p.device + 1, nullptr);
    {
    const unsigned long long id = nps_context_id(p.device);
    if (g_color[p.device] && id != 0 && g_color[p.device]->ctx_id != id) g_color[p.device] = nullptr;  // device reset: abandoned
    if (!g_color[p.device]) {
      g_color[p.device] = new ColorWork();
      g_color[p.device]->ctx_id = id;
    }
  }
    W = g_color[p.device];
  }
  std::lock_guard<std::mutex> lk(W->mu);
  if (!W->stream) NPS_CUDA_RETURN(cudaStreamCreateWithFlags(&W->stream, cudaStreamNonBlocking));
  if (!W->ev[0]) {
    for (auto& ev : W->ev) NPS_CUDA_RETURN(cudaEventCreate(&ev));
  }
  if (!W->ctr) NPS_CUDA_RETURN(cudaMalloc((void**)&W->ctr, sizeof(ColorCtr)));
  if (!W->snap) NPS_CUDA_RETURN(cudaMallocHost((void**)&W->snap, sizeof(ColorCtr)));
  if (!W->sms) NPS_CUDA_RETURN(cudaDeviceGetAttribute(&W->sms, cudaDevAttrMultiProcessorCount, p.device));
  cudaStream_t s = p.stream ? (cudaStream_t)p.stream : W->stream;
  if (st) memset(st, 0, sizeof(*st));
  nps_status e;
  NPS_CUDA_RETURN(cudaEventRecord(W->ev[0], s));
  ColorArgs a;
  a.row = row_ptr;
  a.col = col;
  a.color = color_out;
  if (!p.device_ptrs) {
    if ((e = nps_ensure(&W->row, &W->row_n, (size_t)n + 1, s, "color")) || (e = nps_ensure(&W->col, &W->col_n, (size_t)m, s, "color")) ||
        (e = nps_ensure(&W->color, &W->color_n, (size_t)n, s, "color")))
      return e;
    NPS_CUDA_RETURN(cudaMemcpyAsync(W->row, row_ptr, sizeof(int32_t) * ((size_t)n + 1), cudaMemcpyHostToDevice, s));
    if (m > 0) NPS_CUDA_RETURN(cudaMemcpyAsync(W->col, col, sizeof(int32_t) * (size_t)m, cudaMemcpyHostToDevice, s));
    a.row = W->row;
    a.col = W->col;
    a.color = W->color;
  }
  const size_t nn = (size_t)n, groups = (nn + 31) / 32;
  a.nscan = (int32_t)((groups + kScanItems - 1) / kScanItems);
  // a long row adds its chunks, at most m / kChunk + 1 a row, and splits one run
  const size_t nunits = groups + (size_t)m / kChunk + 2 * ((size_t)m / kLong) + 1;
  if ((e = nps_ensure(&W->state, &W->state_n, groups + (size_t)a.nscan + 1, s, "color")) ||
      (e = nps_ensure(&W->unit, &W->unit_n, nunits, s, "color")) || (e = nps_ensure(&W->lrow, &W->lrow_n, nn, s, "color")))
    return e;
  a.n = n;
  a.m = m;
  a.c = W->ctr;
  a.ucount = W->state;
  a.ubase = W->state + groups;
  a.lrow = W->lrow;
  a.unit = W->unit;
  a.timeout_ns = (unsigned long long)(p.timeout_s * 1e9);
  a.inject = p.reserved[0] == 1 ? 1u : 0u;  // test hook: the first wait cannot end
  int per_sm = 0;
  NPS_CUDA_RETURN(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, color_kernel, kThreads, 0));
  const int use = std::min(p.ctas_per_sm > 0 ? p.ctas_per_sm : kCtasPerSm, std::max(1, per_sm));
  const int grid = (int)std::max<int64_t>(
      1, std::min<int64_t>(((int64_t)n + kThreads - 1) / kThreads, (int64_t)W->sms * use));
  NPS_CUDA_RETURN(cudaMemsetAsync(W->ctr, 0, sizeof(ColorCtr), s));
  NPS_CUDA_RETURN(cudaMemsetAsync(a.color, 0, sizeof(int32_t) * (size_t)n, s));
  NPS_CUDA_RETURN(cudaEventRecord(W->ev[1], s));
  const int ugrid = (int)std::min<int64_t>(((int64_t)groups + kWarps - 1) / kWarps, (int64_t)W->sms * 8);
  color_count_kernel<<<ugrid, kThreads, 0, s>>>(a);
  scan_blocks_kernel<<<a.nscan, kThreads, 0, s>>>(a.ucount, (int32_t)groups, a.ubase);
  scan_totals_kernel<<<1, kThreads, 0, s>>>(a.ubase, a.nscan, a.ubase + a.nscan);
  color_units_kernel<<<ugrid, kThreads, 0, s>>>(a);
  color_kernel<<<grid, kThreads, 0, s>>>(a);
  NPS_CUDA_RETURN(cudaGetLastError());
  NPS_CUDA_RETURN(cudaEventRecord(W->ev[2], s));
  if (!p.device_ptrs)
    NPS_CUDA_RETURN(cudaMemcpyAsync(color_out, a.color, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToHost, s));
  NPS_CUDA_RETURN(cudaMemcpyAsync(W->snap, W->ctr, sizeof(ColorCtr), cudaMemcpyDeviceToHost, s));
  NPS_CUDA_RETURN(cudaEventRecord(W->ev[3], s));
  NPS_CUDA_RETURN(cudaStreamSynchronize(s));
  const ColorCtr& f = *W->snap;
  if (st) {
    st->status = (int32_t)f.status;
    st->iterations = (uint32_t)f.max_color;  // the reference's iteration count: one color per iteration
    st->buckets = (uint32_t)f.max_color;     // the levels of the dependency order, one per color
    st->edges_scanned = f.edges;
    st->grid_ctas = grid;
    cudaEventElapsedTime(&st->kernel_ms, W->ev[1], W->ev[2]);
    cudaEventElapsedTime(&st->total_ms, W->ev[0], W->ev[3]);
  }
  if (f.status == NPS_ERR_FORMAT)
    return nps_fail(NPS_ERR_FORMAT, "malformed CSR: a row range or column index is out of bounds");
  if (f.status == NPS_ERR_TIMEOUT) return nps_fail(NPS_ERR_TIMEOUT, "color: a wait exceeded timeout_s");
  return NPS_OK;
}
