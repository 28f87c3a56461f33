// Orientation: degree order or degeneracy (k-core peeling) order, then the
// DAG CSR relabelled by rank.
//
// Reference behaviour kept:
//   * degree orientation keeps u->v iff deg u < deg v, or equal and u < v
//     (include/main_support.cuh:54-87 with node degrees, src/main.cu:181);
//   * degeneracy orientation keeps u->v iff prio u < prio v, or equal and
//     u < v (include/main_support.cuh:89-128), where prio is the peel
//     sub-round of SingleGPU_Kcore::findKcoreIncremental_async
//     (kcore/kcore.cuh:442-584): level L peels every vertex of current degree
//     L in sub-rounds, each sub-round's vertices get the running sub-round
//     counter (kcore.cuh:192 and :564) and the batch that empties the graph
//     keeps the initial value 2m (kcore.cuh:471-472, break at :496-498).
//
// B200 design: the whole peel runs in ONE cooperative persistent kernel with
// grid-wide barriers between phases (the reference launches kernels and
// synchronises the host per sub-round). The bucket of candidate vertices is
// compacted every level so a level scans only live low-degree vertices.
//
// The DAG is stored in rank labels: a vertex's label is its position in the
// orientation's total order, so every out-list holds larger labels only and
// the induced-subgraph bitmaps of the counting stage are upper-triangular.
#include <algorithm>

#include "bits.cuh"
#include "dev_common.cuh"
#include "engine.h"
#include "prims.cuh"

namespace kc {

namespace {

int bits_for(uint64_t x) {  // bits needed to hold values in [0, x]
  int b = 0;
  while (b < 64 && (x >> b) != 0) ++b;
  return b;
}

uint32_t grid_for(uint64_t work, int sms, int per_sm = 16) {
  return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((work + 255) / 256, (uint64_t)sms * per_sm));
}

// Sort keys (graph, major, v): the graph field (batches only) is the most
// significant so each graph's vertices get a contiguous range of ranks; it
// never changes the order of two vertices of the same graph.
__global__ void k_degree_keys(const uint32_t* __restrict__ rp, uint32_t n, int vbits, const uint32_t* __restrict__ vg,
                              int gshift, unsigned long long* keys) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    unsigned long long k = ((unsigned long long)(rp[v + 1] - rp[v]) << vbits) | v;
    if (vg) k |= (unsigned long long)vg[v] << gshift;
    keys[v] = k;
  }
}

__global__ void k_prio_keys(const uint32_t* __restrict__ prio, uint32_t n, int vbits, uint32_t cap,
                            const uint32_t* __restrict__ vg, int gshift, unsigned long long* keys) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    unsigned long long k = ((unsigned long long)min(prio[v], cap) << vbits) | v;
    if (vg) k |= (unsigned long long)vg[v] << gshift;
    keys[v] = k;
  }
}

__global__ void k_rank_from_sorted(const unsigned long long* __restrict__ keys, uint32_t n,
                                   unsigned long long vmask, uint32_t* rank, uint32_t* inv) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t v = (uint32_t)(keys[i] & vmask);
    inv[i] = v;
    rank[v] = i;
  }
}

// The ranks of the next 32 kRowsInFlight neighbours of a row, kRowsInFlight per
// lane, all loads in flight together: a hub's row is walked by one warp, and
// one neighbour per lane at a time cost it two memory latencies per 32 entries
// (R-MAT 18: k_fill_dag 602 us, k_out_degree 136 us; 127 and 103 us now).
// Entries past the end get rank 0.
constexpr uint32_t kRowsInFlight = 8;

__device__ __forceinline__ void row_ranks(const uint32_t* __restrict__ col, const uint32_t* __restrict__ rank,
                                          uint32_t i0, uint32_t e, uint32_t (&rw)[kRowsInFlight]) {
  uint32_t x[kRowsInFlight];
#pragma unroll
  for (uint32_t q = 0; q < kRowsInFlight; ++q) {
    const uint32_t i = i0 + q * 32u + lane_id();
    x[q] = i < e ? col[i] : 0xffffffffu;
  }
#pragma unroll
  for (uint32_t q = 0; q < kRowsInFlight; ++q) rw[q] = x[q] != 0xffffffffu ? rank[x[q]] : 0u;
}

// Warp per vertex: out-degree in rank order (neighbours of larger rank).
__global__ void k_out_degree(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ col, uint32_t n,
                             const uint32_t* __restrict__ rank, uint32_t* odeg) {
  const uint32_t lane = lane_id();
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t v = gw; v < n; v += nw) {
    const uint32_t rv = rank[v], b = rp[v], e = rp[v + 1];
    uint32_t c = 0, i0 = b;
    for (; i0 + 64u < e; i0 += 32u * kRowsInFlight) {
      uint32_t rw[kRowsInFlight];
      row_ranks(col, rank, i0, e, rw);
#pragma unroll
      for (uint32_t q = 0; q < kRowsInFlight; ++q) c += rw[q] > rv;
    }
    for (uint32_t i = i0 + lane; i < e; i += 32) c += rank[col[i]] > rv;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) odeg[rv] = c;
  }
}

__global__ void k_fill_dag(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ col, uint32_t n,
                           const uint32_t* __restrict__ rank, const uint32_t* __restrict__ drp, uint32_t* dcol) {
  const uint32_t lane = lane_id();
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t v = gw; v < n; v += nw) {
    const uint32_t rv = rank[v], b = rp[v], e = rp[v + 1];
    uint32_t pos = drp[rv], i0 = b;
    for (; i0 + 64u < e; i0 += 32u * kRowsInFlight) {
      uint32_t rw[kRowsInFlight];
      row_ranks(col, rank, i0, e, rw);
#pragma unroll
      for (uint32_t q = 0; q < kRowsInFlight; ++q) {
        const bool keep = rw[q] > rv;
        const uint32_t bal = __ballot_sync(0xffffffffu, keep);
        if (keep) dcol[pos + __popc(bal & lanemask_lt())] = rw[q];
        pos += __popc(bal);
      }
    }
    for (; i0 < e; i0 += 32) {
      uint32_t i = i0 + lane;
      uint32_t rw = i < e ? rank[col[i]] : 0;
      bool keep = i < e && rw > rv;
      uint32_t bal = __ballot_sync(0xffffffffu, keep);
      if (keep) dcol[pos + __popc(bal & lanemask_lt())] = rw;
      pos += __popc(bal);
    }
  }
}

__global__ void k_edge_rows(const uint32_t* __restrict__ drp, uint32_t n, uint32_t* erow) {
  const uint32_t lane = lane_id();
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t r = gw; r < n; r += nw)
    for (uint32_t i = drp[r] + lane; i < drp[r + 1]; i += 32) erow[i] = r;
}

__global__ void k_max_row_len(const uint32_t* __restrict__ off, uint32_t n, uint32_t* out) {
  uint32_t mx = 0;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    mx = max(mx, off[v + 1] - off[v]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane_id() == 0 && mx) atomicMax(out, mx);
}

// Original-id export of the DAG (the reference's layout): row of original u =
// original ids of the out-neighbours of rank[u].
__global__ void k_export_deg(const uint32_t* __restrict__ drp, const uint32_t* __restrict__ rank, uint32_t n,
                             uint32_t* deg) {
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x)
    deg[u] = drp[rank[u] + 1] - drp[rank[u]];
}

__global__ void k_export_fill(const uint32_t* __restrict__ drp, const uint32_t* __restrict__ dcol,
                              const uint32_t* __restrict__ rank, const uint32_t* __restrict__ inv, uint32_t n,
                              const uint32_t* __restrict__ orp, uint32_t* ocol) {
  const uint32_t lane = lane_id();
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t u = gw; u < n; u += nw) {
    const uint32_t r = rank[u], b = drp[r], e = drp[r + 1], o = orp[u];
    for (uint32_t i = b + lane; i < e; i += 32) ocol[o + (i - b)] = inv[dcol[i]];
  }
}

// ---- degeneracy peel: one cooperative persistent kernel -----------------------
//
// What bounds it is not bytes but the chain of sub-rounds (420 for R-MAT scale
// 18, over 1,000 for a batch of 200 graphs), each a few dependent memory
// latencies and a barrier; most hold a few vertices. So:
//   * one barrier per sub-round: the vertices of a front are not marked as
//     peeled before their neighbours are decremented. A peeled vertex's degree
//     never exceeds the level, so a further decrement of it never yields
//     level + 1 (the next front) or the end of the bucket's window, and a
//     vertex below the level is a peeled one: no flags are kept;
//   * one CTA of 1024 threads per SM, since a barrier costs by the CTA;
//   * runs of small fronts (and short bucket scans) are done by one CTA alone
//     with block barriers, the others waiting at the next grid barrier. Its
//     edges are dealt out singly (a search in the front's length prefix). After
//     kSoloSteps steps it comes to the barrier and starts again, so that no wait
//     there is longer than that many steps;
//   * a front is a list of row pieces of at most kPiece entries, so a hub's
//     row (15,000 entries) is spread over many warps;
//   * levels without vertices are skipped through the smallest degree seen.
// R-MAT scale 18 (3.8M edges): 9.6 ms with two barriers per sub-round, flags
// and four CTAs per SM, 2.6 ms now; scale 11 (16k edges) 0.78 ms, 0.27 ms now.

constexpr uint32_t PEEL_WINDOW = 64;     // degree window of the candidate bucket
constexpr uint32_t kPeelThreads = 1024;
constexpr uint32_t kPiece = 128;         // row entries per front piece (four per lane of a warp)
// One CTA takes a front of up to kSoloFront pieces with up to kSoloEdges row
// entries, and bucket or vertex scans of up to kSoloScan entries: one SM makes
// about one random access per cycle, so 4,096 of them cost what a grid step's
// barrier does.
constexpr uint32_t kSoloFront = 1024, kSoloEdges = 4096, kSoloScan = 4096;
// Steps of one stretch of the solo CTA: 2 us each on a path (1M vertices are
// 500,000 sub-rounds), so a stretch is some 10 ms, and its barrier 0.1% of it.
constexpr uint32_t kSoloSteps = 4096;

struct PeelArgs {
  const uint32_t* rp;
  const uint32_t* col;
  uint32_t n;
  int* deg;             // current degree (below the level: peeled)
  uint32_t* prio;
  uint32_t* level;
  uint32_t* bucket_a;   // candidate bucket (ping-pong, capacity n)
  uint32_t* bucket_b;
  uint2* front_a;       // frontier (ping-pong): [begin, end) in col of every row piece
  uint2* front_b;
  uint32_t* ctr;        // 4 phase slots x 4 counters, zeroed; then two slots for the solo CTA's state
  uint32_t init_prio;   // 2m: the priority the final batch keeps
  uint32_t* bar;        // grid barrier: arrivals so far, zeroed
  uint32_t* out;        // [0] last level, [1] sub-rounds, [2] error
};
// ctr: kPeelStateWords words left by the solo CTA. Two slots taken in turn: a
// stretch may follow another at once, and its state is written while the other
// CTAs may still be reading that of the one before.
constexpr uint32_t kPeelSolo = 32, kPeelSoloSlot = 16;
constexpr uint32_t kPeelStateWords = 9;

__global__ void k_peel_init(const uint32_t* __restrict__ rp, uint32_t n, int* deg) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    deg[v] = (int)(rp[v + 1] - rp[v]);
}

// Appends x to list (for the lanes with pred) with one atomic per warp.
__device__ __forceinline__ void warp_append(bool pred, uint32_t x, uint32_t* list, uint32_t* cnt) {
  const uint32_t m = __ballot_sync(0xffffffffu, pred);
  if (!m) return;
  const uint32_t leader = __ffs(m) - 1;
  uint32_t base = 0;
  if (lane_id() == leader) base = atomicAdd(cnt, (uint32_t)__popc(m));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (pred) list[base + __popc(m & lanemask_lt())] = x;
}

// The lanes with pred put their vertex v into the front that sub-round
// `priority` of level L will peel: level and priority are written now, the
// row's pieces appended to `front` (the first kSoloFront of them to `sfront`
// too, where there is one: in the solo CTA). cnt[0] counts pieces, cnt[1]
// vertices; in global memory with one atomic, since what the warps of a large scan
// wait for is the counter (G(4M, 32M edges): 11.4 ms with an atomic each, 8.1 ms so).
__device__ __forceinline__ void front_append(const PeelArgs& a, bool pred, uint32_t v, uint32_t L, uint32_t priority,
                                             uint2* front, uint2* sfront, uint32_t* cnt) {
  const uint32_t m = __ballot_sync(0xffffffffu, pred);
  if (!m) return;
  uint32_t b = 0, e = 0, pieces = 0;
  if (pred) {
    b = a.rp[v];
    e = a.rp[v + 1];
    pieces = max(1u, (e - b + kPiece - 1u) / kPiece);  // (an isolated vertex is one empty piece)
    a.level[v] = L;
    a.prio[v] = priority;
  }
  uint32_t incl = pieces;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane_id() >= (uint32_t)o) incl += y;
  }
  uint32_t base = 0;
  if (lane_id() == 31u) {
    if (sfront != nullptr) {  // (counters in shared memory: a 64-bit add there is a loop of exchanges)
      base = atomicAdd(&cnt[0], incl);
      atomicAdd(&cnt[1], (uint32_t)__popc(m));
    } else {
      base = (uint32_t)atomicAdd(reinterpret_cast<unsigned long long*>(cnt),
                                 (unsigned long long)__popc(m) << 32 | incl);
    }
  }
  base = __shfl_sync(0xffffffffu, base, 31) + incl - pieces;
  for (uint32_t i = 0; i < pieces; ++i) {
    const uint2 pc = make_uint2(b + i * kPiece, min(e, b + (i + 1u) * kPiece));
    front[base + i] = pc;
    if (sfront != nullptr && base + i < kSoloFront) sfront[base + i] = pc;
  }
}

// The control state. Every thread keeps an identical copy, derived from
// counters read after a grid barrier (or from the state the solo CTA left), so
// all threads take the same branches and reach the same barriers.
struct PeelState {
  uint32_t todo;        // vertices not yet peeled
  uint32_t L;           // level
  uint32_t bucket_end;  // the bucket holds the live vertices of degree in [L, bucket_end)
  uint32_t bsize, fsize;  // bucket entries; vertices of the front
  uint32_t pieces;        // row pieces of the front
  uint32_t priority;    // sub-rounds done
  uint32_t flips;       // bit 0: the bucket is in bucket_b, bit 1: the front is in front_b
  uint32_t too_big;     // the front holds more edges than one CTA should take
};

__device__ __forceinline__ bool solo_takes(const PeelState& st, uint32_t n) {
  if (st.fsize) return st.pieces <= kSoloFront && !st.too_big;
  return (st.L < st.bucket_end ? st.bsize : n) <= kSoloScan;
}

// Block-wide exclusive scan of one value per thread; the total goes to *total.
__device__ __forceinline__ uint32_t peel_scan(uint32_t v, uint32_t* wsum, uint32_t* total) {
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += y;
  }
  if (lane == 31) wsum[w] = incl;
  __syncthreads();
  const uint32_t s = lane < kPeelThreads / 32 ? wsum[lane] : 0u;
  uint32_t si = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, si, o);
    if (lane >= (uint32_t)o) si += y;
  }
  *total = __shfl_sync(0xffffffffu, si, 31);
  return incl - v + __shfl_sync(0xffffffffu, si - s, w);
}

// One CTA peels alone for as long as the next step is small, kSoloSteps steps
// at most (it takes at least one). Counters live in shared memory; lists in
// global memory.
__device__ void peel_solo(const PeelArgs& a, PeelState& st) {
  __shared__ uint32_t pre[kSoloFront], beg[kSoloFront], wsum[kPeelThreads / 32];
  __shared__ uint2 sfront[kSoloFront];
  __shared__ uint32_t cn[2], cb, cmin;  // next front (pieces, vertices), bucket, smallest degree above the level (complemented)
  const uint32_t tid = threadIdx.x;
  bool in_shared = false;  // the front is in sfront
  for (uint32_t steps = 0; steps < kSoloSteps && st.todo > 0 && solo_takes(st, a.n); ++steps) {
    uint32_t* bucket = (st.flips & 1u) ? a.bucket_b : a.bucket_a;
    uint32_t* bucket2 = (st.flips & 1u) ? a.bucket_a : a.bucket_b;
    uint2* front = (st.flips & 2u) ? a.front_b : a.front_a;
    uint2* next = (st.flips & 2u) ? a.front_a : a.front_b;
    if (tid == 0) { cn[0] = cn[1] = 0; cb = st.fsize ? st.bsize : 0u; cmin = 0; }
    if (st.fsize) {  // a sub-round
      if (st.fsize == st.todo) {  // the final batch
        st.todo = 0;
        break;
      }
      uint32_t len = 0, total = 0;
      if (tid < st.pieces) {
        const uint2 pc = in_shared ? sfront[tid] : front[tid];
        beg[tid] = pc.x;
        len = pc.y - pc.x;
      }
      const uint32_t ex = peel_scan(len, wsum, &total);
      if (tid < st.pieces) pre[tid] = ex;
      if (total > kSoloEdges) {
        st.too_big = 1u;
        __syncthreads();
        return;
      }
      st.todo -= st.fsize;
      __syncthreads();
      uint32_t top = 1;
      while (top < st.pieces) top <<= 1;
      constexpr uint32_t kU = kSoloEdges / kPeelThreads;  // edges per thread, all in flight
      for (uint32_t i0 = 0; i0 < total; i0 += kU * kPeelThreads) {
        uint32_t u[kU];
        int cur[kU];
#pragma unroll
        for (uint32_t q = 0; q < kU; ++q) {
          const uint32_t i = i0 + q * kPeelThreads + tid;
          u[q] = 0xffffffffu;
          if (i < total) {
            uint32_t j = 0;  // the last piece with pre[j] <= i
            for (uint32_t s = top >> 1; s; s >>= 1)
              if (j + s < st.pieces && pre[j + s] <= i) j += s;
            u[q] = a.col[beg[j] + (i - pre[j])];
          }
        }
#pragma unroll
        for (uint32_t q = 0; q < kU; ++q) cur[q] = u[q] != 0xffffffffu ? atomicSub(&a.deg[u[q]], 1) : -1;
#pragma unroll
        for (uint32_t q = 0; q < kU; ++q) {
          if (i0 + q * kPeelThreads >= total) break;
          const bool to_next = cur[q] == (int)st.L + 1;
          front_append(a, to_next, u[q], st.L, st.priority + 1u, next, sfront, cn);
          warp_append(!to_next && cur[q] == (int)st.bucket_end, u[q], bucket, &cb);
        }
      }
      __syncthreads();
      st.fsize = min(cn[1], a.n);
      st.pieces = cn[0];
      st.bsize = min(cb, a.n);
      st.flips ^= 2u;
      ++st.priority;
      in_shared = true;
      if (st.fsize == 0) ++st.L;
    } else if (st.L < st.bucket_end) {  // the bucket's vertices at this level
      in_shared = true;
      __syncthreads();
      uint32_t mn = 0;
      for (uint32_t i0 = 0; i0 < st.bsize; i0 += kPeelThreads) {
        const uint32_t i = i0 + tid;
        const uint32_t v = i < st.bsize ? bucket[i] : 0u;
        const int d = i < st.bsize ? __ldcg(a.deg + v) : -1;
        front_append(a, d == (int)st.L, v, st.L, st.priority, front, sfront, cn);
        warp_append(d > (int)st.L, v, bucket2, &cb);
        if (d > (int)st.L) mn = max(mn, ~(uint32_t)d);
      }
      mn = __reduce_max_sync(0xffffffffu, mn);
      if (lane_id() == 0 && mn) atomicMax(&cmin, mn);
      __syncthreads();
      st.fsize = min(cn[1], a.n);
      st.pieces = cn[0];
      st.bsize = min(cb, a.n);
      st.flips ^= 1u;
      if (st.fsize == 0) st.L = cmin ? min(~cmin, st.bucket_end) : st.bucket_end;
    } else {  // a new window
      __syncthreads();
      uint32_t mn = 0;
      for (uint32_t v0 = 0; v0 < a.n; v0 += kPeelThreads) {
        const uint32_t v = v0 + tid;
        const int d = v < a.n ? __ldcg(a.deg + v) : -1;
        warp_append(d >= (int)st.L && d < (int)(st.L + PEEL_WINDOW), v, bucket, &cb);
        if (d >= (int)st.L) mn = max(mn, ~(uint32_t)d);
      }
      mn = __reduce_max_sync(0xffffffffu, mn);
      if (lane_id() == 0 && mn) atomicMax(&cmin, mn);
      __syncthreads();
      st.bsize = min(cb, a.n);
      if (cmin == 0u) {  // no live vertex left, todo > 0: cannot happen for a valid CSR
        if (tid == 0) a.out[2] = DEV_ERR_INPUT;
        st.todo = 0;
        break;
      }
      if (st.bsize == 0) st.L = ~cmin;  // every live vertex lies above the window
      else st.bucket_end = st.L + PEEL_WINDOW;
      if (st.bsize == 0) st.bucket_end = st.L;
    }
    st.too_big = 0;
    __syncthreads();  // the counters are read before they are set again
  }
}

// Barrier over the cooperative grid (a release-add and an acquire spin per
// CTA, 2.4k cycles), after which thread 0 of every CTA reads `words` words at
// src for its CTA: with every warp of 148 CTAs reading the counters itself,
// one L2 line served 40,000 requests, which took 15k cycles. The spin is
// bounded: a CTA whose polls (an L2 round trip each) run out records a timeout,
// and every CTA leaves the kernel at its next barrier; the whole CTA returns
// false then. The longest wait by design is one solo stretch or one grid step.
// (The checked build gives up 256 times sooner, so that its tests see a wait
// that grows with the graph.)
#ifdef KC_CHECKED
constexpr uint32_t kPeelSpins = 1u << 18;
#else
constexpr uint32_t kPeelSpins = 1u << 26;
#endif

__device__ __forceinline__ bool grid_barrier(const PeelArgs& a, uint32_t& target, const uint32_t* src, uint32_t words,
                                             uint32_t* got) {
  target += gridDim.x;
  int ok = 1;
  __syncthreads();
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
      uint32_t seen = 0, spins = 0;
      do {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.bar) : "memory");
      } while ((int32_t)(seen - target) < 0 && ++spins < kPeelSpins);  // (the count may wrap)
      ok = (int32_t)(seen - target) >= 0;
      if (!ok) set_error(a.out + 2, DEV_ERR_TIMEOUT);
    }
    __syncwarp();
    if (threadIdx.x < words) got[threadIdx.x] = __ldcg(src + threadIdx.x);
  }
  return __syncthreads_and(ok) != 0;
}

__global__ void __launch_bounds__(kPeelThreads, 1) k_peel(PeelArgs a) {
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t lane = lane_id();
  const uint32_t gw = tid >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  PeelState st = {a.n, 0, 0, 0, 0, 0, 0, 0, 0};
  uint32_t bar = 0;
  __shared__ uint32_t got[kPeelStateWords];  // what the last barrier brought
  // Counters live in four phase slots; a phase zeroes the slot two phases
  // ahead, which every thread has finished reading by then.
  uint32_t phase = 0;
  uint32_t stretch = 0;  // of the solo CTA
  auto slot = [&](uint32_t ph) { return a.ctr + (ph & 3u) * 4u; };
  while (st.todo > 0) {
    if (solo_takes(st, a.n)) {
      uint32_t* o = a.ctr + kPeelSolo + (stretch++ & 1u) * kPeelSoloSlot;
      if (blockIdx.x == 0) {
        peel_solo(a, st);
        if (tid == 0) {
          o[0] = st.todo; o[1] = st.L; o[2] = st.bucket_end; o[3] = st.bsize;
          o[4] = st.fsize; o[5] = st.pieces; o[6] = st.priority; o[7] = st.flips; o[8] = st.too_big;
        }
      }
      if (!grid_barrier(a, bar, o, kPeelStateWords, got)) return;
      st = {got[0], got[1], got[2], got[3], got[4], got[5], got[6], got[7], got[8]};
      continue;
    }
    uint32_t* bucket = (st.flips & 1u) ? a.bucket_b : a.bucket_a;
    uint32_t* bucket2 = (st.flips & 1u) ? a.bucket_a : a.bucket_b;
    uint2* front = (st.flips & 2u) ? a.front_b : a.front_a;
    uint2* next = (st.flips & 2u) ? a.front_a : a.front_b;
    if (tid == 0) {
      uint32_t* z = slot(phase + 2);
      z[0] = z[1] = z[2] = z[3] = 0;
    }
    uint32_t* c = slot(phase++);  // front pieces, front vertices, bucket, smallest degree (complemented)
    st.too_big = 0;
    if (st.fsize) {  // a sub-round
      const bool last = st.fsize == st.todo;  // the final batch
      st.todo -= st.fsize;
      if (last) break;
      for (uint32_t i = gw; i < st.pieces; i += nw) {
        const uint2 pc = front[i];
        uint32_t u[kPiece / 32u];
        int cur[kPiece / 32u];
#pragma unroll
        for (uint32_t q = 0; q < kPiece / 32u; ++q) {
          const uint32_t j = pc.x + q * 32u + lane;
          u[q] = j < pc.y ? a.col[j] : 0xffffffffu;
        }
#pragma unroll
        for (uint32_t q = 0; q < kPiece / 32u; ++q) cur[q] = u[q] != 0xffffffffu ? atomicSub(&a.deg[u[q]], 1) : -1;
#pragma unroll
        for (uint32_t q = 0; q < kPiece / 32u; ++q) {
          if (pc.x + q * 32u >= pc.y) break;  // (most rows are short)
          const bool to_next = cur[q] == (int)st.L + 1;
          front_append(a, to_next, u[q], st.L, st.priority + 1u, next, nullptr, c);
          warp_append(!to_next && cur[q] == (int)st.bucket_end, u[q], bucket + st.bsize, &c[2]);
        }
      }
      if (!grid_barrier(a, bar, c, 4, got)) return;
      st.pieces = got[0];
      st.fsize = min(got[1], a.n);
      st.bsize = min(st.bsize + got[2], a.n);
      st.flips ^= 2u;
      ++st.priority;
      if (st.fsize == 0) ++st.L;
    } else if (st.L < st.bucket_end) {  // the bucket's vertices at this level, and the bucket compacted
      uint32_t mn = 0;
      for (uint32_t i0 = gw * 32; i0 < st.bsize; i0 += nw * 32) {
        const uint32_t i = i0 + lane;
        const uint32_t v = i < st.bsize ? bucket[i] : 0u;
        const int d = i < st.bsize ? __ldcg(a.deg + v) : -1;
        front_append(a, d == (int)st.L, v, st.L, st.priority, front, nullptr, c);
        warp_append(d > (int)st.L, v, bucket2, &c[2]);
        if (d > (int)st.L) mn = max(mn, ~(uint32_t)d);
      }
      mn = __reduce_max_sync(0xffffffffu, mn);
      if (lane == 0 && mn) atomicMax(&c[3], mn);
      if (!grid_barrier(a, bar, c, 4, got)) return;
      st.pieces = got[0];
      st.fsize = min(got[1], a.n);
      st.bsize = min(got[2], a.n);
      st.flips ^= 1u;
      const uint32_t m = got[3];
      if (st.fsize == 0) st.L = m ? min(~m, st.bucket_end) : st.bucket_end;
    } else {  // a new window
      uint32_t mn = 0;
      for (uint32_t v0 = gw * 32; v0 < a.n; v0 += nw * 32) {
        const uint32_t v = v0 + lane;
        const int d = v < a.n ? __ldcg(a.deg + v) : -1;
        warp_append(d >= (int)st.L && d < (int)(st.L + PEEL_WINDOW), v, bucket, &c[2]);
        if (d >= (int)st.L) mn = max(mn, ~(uint32_t)d);
      }
      mn = __reduce_max_sync(0xffffffffu, mn);
      if (lane == 0 && mn) atomicMax(&c[3], mn);
      if (!grid_barrier(a, bar, c, 4, got)) return;
      st.bsize = min(got[2], a.n);
      const uint32_t m = got[3];
      if (m == 0u) {  // no live vertex left, todo > 0: cannot happen for a valid CSR; never spin
        if (tid == 0) a.out[2] = DEV_ERR_INPUT;
        break;
      }
      if (st.bsize == 0) st.L = ~m;  // every live vertex lies above the window
      st.bucket_end = st.bsize == 0 ? st.L : st.L + PEEL_WINDOW;
    }
  }
  if (tid == 0) {
    a.out[0] = st.L;
    a.out[1] = st.priority;
  }
  // the final batch keeps its initial priority (every vertex has been put in
  // a front, and what any CTA wrote there was ordered by the last barrier)
  if (!grid_barrier(a, bar, a.ctr, 0, got)) return;
  for (uint32_t v = tid; v < a.n; v += nw * 32u)
    if (__ldcg(a.prio + v) == st.priority) a.prio[v] = a.init_prio;
}

}  // namespace

namespace {

// The peel into prio / level (n >= 1); temporaries freed on every path.
kc_status run_peel(kc_graph* g, uint32_t* prio, uint32_t* level) {
  kc_ctx* ctx = g->ctx;
  cudaStream_t s = ctx->stream;
  const uint32_t n = g->n;
  DevTemps t(s);
  int* deg = nullptr;
  uint32_t *ba = nullptr, *bb = nullptr, *ctr = nullptr;
  uint2 *fa = nullptr, *fb = nullptr;
  // a front holds at most every vertex: n pieces and one more per kPiece entries
  const size_t front_cap = (size_t)n + 2 * g->m / kPiece;
  KC_CUDA(t.alloc(&deg, sizeof(int) * n));
  KC_CUDA(t.alloc(&ba, sizeof(uint32_t) * n));
  KC_CUDA(t.alloc(&bb, sizeof(uint32_t) * n));
  KC_CUDA(t.alloc(&fa, sizeof(uint2) * front_cap));
  KC_CUDA(t.alloc(&fb, sizeof(uint2) * front_cap));
  static_assert(kPeelSolo + 2 * kPeelSoloSlot <= 128 && kPeelStateWords <= kPeelSoloSlot, "state slots overlap");
  constexpr uint32_t kCtrWords = 128 + 1;  // the barrier's counter on a line of its own
  KC_CUDA(t.alloc(&ctr, sizeof(uint32_t) * kCtrWords));
  KC_CUDA(cudaMemsetAsync(ctr, 0, sizeof(uint32_t) * kCtrWords, s));
  const uint32_t init_prio = (uint32_t)std::min<uint64_t>(2 * g->m, 0xffffffffull);
  k_peel_init<<<grid_for(n, ctx->sms), 256, 0, s>>>(g->rp, n, deg);
  KC_CUDA(cudaGetLastError());

  PeelArgs a;
  a.rp = g->rp; a.col = g->col; a.n = n; a.deg = deg; a.prio = prio; a.level = level;
  a.bucket_a = ba; a.bucket_b = bb; a.front_a = fa; a.front_b = fb; a.ctr = ctr; a.out = ctr + 16;
  a.init_prio = init_prio;
  a.bar = ctr + 128;
  // At most one CTA per SM, each with enough row entries or pieces of a front (a
  // warp takes a piece at a time: 20 hubs over 16,384 vertices 322 us with a CTA
  // per 4,096 vertices, 268 us per 1,024, 248 us per 256) to be worth a barrier's
  // arrival. A small graph is peeled by one CTA alone.
  const uint64_t want = std::max<uint64_t>(n <= kSoloScan ? 1 : ceil_div<uint64_t>(n, kPeelThreads / 4),
                                           ceil_div<uint64_t>(2 * g->m, 4 * kSoloEdges));
  dim3 grid((uint32_t)std::min<uint64_t>((uint64_t)ctx->sms, std::max<uint64_t>(1, want))), block(kPeelThreads);
  void* args[] = {&a};
  KC_CUDA(cudaLaunchCooperativeKernel((void*)k_peel, grid, block, args, 0, s));
  uint32_t out[3] = {0, 0, 0};
  KC_CUDA(cudaMemcpyAsync(out, ctr + 16, sizeof(out), cudaMemcpyDeviceToHost, s));
  KC_CUDA(cudaStreamSynchronize(s));
  if (out[2]) return fail(KC_ERR_INTERNAL, "peel did not converge (device error %u)", out[2]);
  g->max_core = out[0];
  g->peel_rounds = out[1];
  return KC_OK;
}

}  // namespace

// Peel priorities and core numbers of the graph; the graph keeps them only
// when the whole peel succeeded.
kc_status peel_graph(kc_graph* g) {
  if (g->prio) return KC_OK;
  const uint32_t n = g->n;
  uint32_t *prio = nullptr, *level = nullptr;
  KC_TRY(dev_alloc(g, (void**)&prio, sizeof(uint32_t) * std::max<size_t>(1, n)));
  kc_status st = dev_alloc(g, (void**)&level, sizeof(uint32_t) * std::max<size_t>(1, n));
  if (st == KC_OK && n == 0) g->max_core = 0;
  else if (st == KC_OK) st = run_peel(g, prio, level);
  if (st != KC_OK) {
    dev_free(g, prio);
    dev_free(g, level);
    return st;
  }
  g->prio = prio;
  g->level = level;
  return KC_OK;
}

kc_status orient_graph(kc_graph* g, uint32_t orientation) {
  if (orientation > KC_ORIENT_DEGEN) return fail(KC_ERR_INVALID_ARG, "unknown orientation %u", orientation);
  kc_ctx* ctx = g->ctx;
  cudaStream_t s = ctx->stream;
  const uint32_t n = g->n;
  if (g->oriented == (int)orientation) return KC_OK;
  // drop a previous orientation
  dev_free(g, g->rank); dev_free(g, g->inv); dev_free(g, g->drp); dev_free(g, g->dcol); dev_free(g, g->erow);
  g->rank = g->inv = g->drp = g->dcol = g->erow = nullptr;
  g->oriented = -1;
  if (orientation == KC_ORIENT_DEGEN) KC_TRY(peel_graph(g));

  KC_TRY(dev_alloc(g, (void**)&g->rank, sizeof(uint32_t) * std::max<size_t>(1, n)));
  KC_TRY(dev_alloc(g, (void**)&g->inv, sizeof(uint32_t) * std::max<size_t>(1, n)));
  KC_TRY(dev_alloc(g, (void**)&g->drp, sizeof(uint32_t) * ((size_t)n + 1)));
  const bool bits = g->bits.words != nullptr;
  if (!bits) KC_TRY(dev_alloc(g, (void**)&g->dcol, sizeof(uint32_t) * std::max<uint64_t>(1, g->m)));
  const int vbits = bits_for(n ? n - 1 : 0);
  DevTemps t(s);
  unsigned long long *keys = nullptr, *tmp = nullptr;
  uint32_t *odeg = nullptr, *ucnt = nullptr, *mx = nullptr;
  KC_CUDA(t.alloc(&keys, sizeof(unsigned long long) * std::max<size_t>(1, n)));
  KC_CUDA(t.alloc(&tmp, sizeof(unsigned long long) * std::max<size_t>(1, n)));
  KC_CUDA(t.alloc(&odeg, sizeof(uint32_t) * ((size_t)n + 1)));
  KC_CUDA(t.alloc(&ucnt, sizeof(uint32_t) * ((size_t)n + 1)));
  KC_CUDA(t.alloc(&mx, sizeof(uint32_t)));
  KC_CUDA(cudaMemsetAsync(mx, 0, sizeof(uint32_t), s));
  int major_bits;
  const int graph_bits = g->vgraph_orig ? bits_for(g->n_graphs ? g->n_graphs - 1 : 0) : 0;
  if (orientation == KC_ORIENT_DEGREE) {
    major_bits = bits_for(g->max_deg);
    k_degree_keys<<<grid_for(n, ctx->sms), 256, 0, s>>>(g->rp, n, vbits, g->vgraph_orig, vbits + major_bits, keys);
  } else {
    // Peel priorities are sub-round indices below peel_rounds, except the
    // final batch's 2m; capping that one at peel_rounds keeps every order and
    // keeps the key narrow.
    const uint32_t cap = (uint32_t)std::min<uint64_t>(std::min<uint64_t>(2 * g->m, 0xffffffffull), g->peel_rounds);
    major_bits = bits_for(cap);
    k_prio_keys<<<grid_for(n, ctx->sms), 256, 0, s>>>(g->prio, n, vbits, cap, g->vgraph_orig, vbits + major_bits,
                                                    keys);
  }
  KC_CUDA(cudaGetLastError());
  if (vbits + major_bits + graph_bits > 64) return fail(KC_ERR_INTERNAL, "orientation key exceeds 64 bits");
  KC_CUDA(prim::radix_sort_u64(keys, tmp, n, vbits + major_bits + graph_bits, s));
  k_rank_from_sorted<<<grid_for(n, ctx->sms), 256, 0, s>>>(keys, n, (vbits >= 64) ? ~0ull : ((1ull << vbits) - 1),
                                                          g->rank, g->inv);
  const uint32_t gw = grid_for((uint64_t)n * 32, ctx->sms, 32);
  if (bits) KC_TRY(bits_dag(g, odeg));
  else k_out_degree<<<gw, 256, 0, s>>>(g->rp, g->col, n, g->rank, odeg);
  KC_CUDA(prim::scan_exclusive_u32(odeg, g->drp, n, s));
  if (!bits) k_fill_dag<<<gw, 256, 0, s>>>(g->rp, g->col, n, g->rank, g->drp, g->dcol);
  if (n) k_max_row_len<<<grid_for(n, ctx->sms), 256, 0, s>>>(g->drp, n, mx);
  uint32_t max_out = 0;
  KC_CUDA(cudaMemcpyAsync(&max_out, mx, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  KC_CUDA(cudaStreamSynchronize(s));
  // Units above 1024 vertices take lists: a batch that holds one drops its
  // oriented bit rows.
  if (bits && max_out > 1024u) {
    KC_TRY(dev_alloc(g, (void**)&g->dcol, sizeof(uint32_t) * std::max<uint64_t>(1, g->m)));
    KC_TRY(bits_dag_lists(g));
    g->dbits = BitRows();
  }
  // out-lists in rank order (values are distinct, so dedup keeps them all)
  if (g->dcol) KC_CUDA(prim::segmented_sort_unique(g->drp, g->dcol, ucnt, n, max_out, n, s));
  KC_CUDA(cudaGetLastError());
  KC_CUDA(cudaStreamSynchronize(s));
  g->max_out = max_out;
  g->oriented = (int)orientation;
  return KC_OK;
}

kc_status ensure_edge_rows(kc_graph* g) {
  if (g->erow) return KC_OK;
  KC_TRY(dev_alloc(g, (void**)&g->erow, sizeof(uint32_t) * std::max<uint64_t>(1, g->m)));
  k_edge_rows<<<grid_for((uint64_t)g->n * 32, g->ctx->sms, 32), 256, 0, g->ctx->stream>>>(g->drp, g->n, g->erow);
  KC_CUDA(cudaGetLastError());
  return KC_OK;
}

// Exports the DAG in original ids with rows sorted by id (host buffers).
kc_status export_dag(kc_graph* g, uint32_t* h_rp, uint32_t* h_col) {
  kc_ctx* ctx = g->ctx;
  cudaStream_t s = ctx->stream;
  const uint32_t n = g->n;
  DevTemps t(s);
  uint32_t *deg = nullptr, *orp = nullptr, *ocol = nullptr, *ucnt = nullptr;
  KC_CUDA(t.alloc(&deg, sizeof(uint32_t) * ((size_t)n + 1)));
  KC_CUDA(t.alloc(&orp, sizeof(uint32_t) * ((size_t)n + 1)));
  KC_CUDA(t.alloc(&ocol, sizeof(uint32_t) * std::max<uint64_t>(1, g->m)));
  KC_CUDA(t.alloc(&ucnt, sizeof(uint32_t) * ((size_t)n + 1)));
  k_export_deg<<<grid_for(n, ctx->sms), 256, 0, s>>>(g->drp, g->rank, n, deg);
  KC_CUDA(prim::scan_exclusive_u32(deg, orp, n, s));
  k_export_fill<<<grid_for((uint64_t)n * 32, ctx->sms, 32), 256, 0, s>>>(g->drp, g->dcol, g->rank, g->inv, n, orp, ocol);
  KC_CUDA(prim::segmented_sort_unique(orp, ocol, ucnt, n, g->max_out, n, s));
  KC_CUDA(cudaMemcpyAsync(h_rp, orp, sizeof(uint32_t) * ((size_t)n + 1), cudaMemcpyDeviceToHost, s));
  if (g->m) KC_CUDA(cudaMemcpyAsync(h_col, ocol, sizeof(uint32_t) * g->m, cudaMemcpyDeviceToHost, s));
  KC_CUDA(cudaStreamSynchronize(s));
  return KC_OK;
}

}  // namespace kc
