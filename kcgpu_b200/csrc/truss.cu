// k-truss support: sup(u,v) = |N(u) ∩ N(v)| for every undirected edge.
//
// The reference parses `-m ktruss` (include/Config.h:66-67) but never
// dispatches it; its only truss code is peeling helpers (truss/kernels.cuh).
// This kernel defines the operation the engine exports: one support value
// per edge u < v, in the row-major order of the symmetric CSR's upper
// triangle.
//
// Every edge is counted at its longer end u (more neighbours; ties: the larger
// id): the shorter row is streamed and each entry tested for membership in
// N(u) with one read, of a bitmap of all vertices in shared memory (a CTA per
// vertex of more than kSupportSmall or kSupportMid neighbours) or by a search of
// the row in shared memory (a warp per smaller vertex). Eight lanes read a row
// together. One warp per edge with a search for the edge's row and a binary search
// per entry, both chains of dependent L2 reads, took 2.03 ms on R-MAT scale 17
// (1.26M edges); this takes 0.72 ms. That form is still the one for graphs above
// kSupportBitmap vertices, whose bitmap does not fit, and for graphs of few edges.
// Where it loses to that form is a star: 300k leaves take 0.50 ms, 0.40 ms there.
#include <algorithm>

#include "dev_common.cuh"
#include "engine.h"
#include "prims.cuh"

namespace kc {

namespace {

// Number of neighbours of u that are larger than u.
__global__ void k_upper_count(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ col, uint32_t n,
                              uint32_t* cnt) {
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
    const uint32_t b = rp[u], e = rp[u + 1];
    cnt[u] = e - b - lower_bound_u32(col + b, e - b, u + 1);
  }
}

constexpr uint32_t kSupportBitmap = 1u << 20;  // 128 KB of bits
// Below this many edges the extra launches and the longest task cost more than
// the searches (R-MAT of 16k and 40k edges: 66 and 107 us with a warp per edge, 82
// and 120 us with bitmaps; G(1000, 50k edges): 113 and 100; G(20000, 100k edges):
// 157 and 129).
constexpr uint64_t kSupportEdges = 49'152;
// Most neighbours of a vertex that is a warp's: where a bitmap leaves room for one
// CTA only, a task for 33 to 128 neighbours is mostly waiting (G(1M, 20M edges):
// 38.5 ms with 32 there, 22.4 with 128; with a warp per edge 28.6).
constexpr uint32_t kSupportSmall = 32, kSupportMid = 128;
constexpr uint32_t kRowLanes = 8;

// Neighbours of one task of a vertex of du. Every task pays for setting the
// vertex's bits; as one task a hub of 15,000 neighbours was the launch's tail. So
// a task has `least` of them, 1024 (R-MAT 19: 5.5 ms, 6.2 with 256) or, in a graph
// of few edges, whose tail is most of it, 256 (R-MAT 14: 336 us, 399 with 1024);
// but no vertex has more than kSupportTasks (a star of 1M leaves as 977 tasks
// took 4.7 ms, as 64 it takes 1.3 ms).
constexpr uint32_t kSupportTasks = 64, kSupportChunk = 1024, kSupportChunkFew = 256;
constexpr uint64_t kSupportFewEdges = 1u << 20;

__device__ __forceinline__ uint32_t support_chunk(uint32_t du, uint32_t least) {
  return max(least, (du + kSupportTasks - 1u) / kSupportTasks);
}

// The tasks of the vertices of more than `small` neighbours, in any order:
// (vertex, first neighbour).
__global__ void k_support_list(const uint32_t* __restrict__ rp, uint32_t n, uint32_t small, uint32_t least,
                               uint2* list, uint32_t* count) {
  for (uint32_t u0 = blockIdx.x * blockDim.x; u0 < n; u0 += gridDim.x * blockDim.x) {
    const uint32_t u = u0 + threadIdx.x;
    const uint32_t du = u < n ? rp[u + 1] - rp[u] : 0u;
    const uint32_t chunk = support_chunk(du, least);
    const uint32_t tasks = du > small ? (du + chunk - 1u) / chunk : 0u;
    if (!__any_sync(0xffffffffu, tasks != 0u)) continue;
    uint32_t incl = tasks;
#pragma unroll
    for (uint32_t o = 1; o < 32u; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane_id() >= o) incl += y;
    }
    uint32_t base = 0;
    if (lane_id() == 31u) base = atomicAdd(count, incl);
    base = __shfl_sync(0xffffffffu, base, 31) + incl - tasks;
    for (uint32_t i = 0; i < tasks; ++i) list[base + i] = make_uint2(u, i * chunk);
  }
}

// Where the support of edge {u, v} goes: ju is v's position in row u, iv u's
// position in row v.
__device__ __forceinline__ uint32_t support_index(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ ubase,
                                                  uint32_t u, uint32_t v, uint32_t ju, uint32_t iv) {
  const uint32_t w = min(u, v), j = u < v ? ju : iv;
  return ubase[w] + j - ((rp[w + 1] - rp[w]) - (ubase[w + 1] - ubase[w]));
}

// The neighbours v of u (row [ub, ub + du)) whose rows are not longer, number
// `first`, first + step, .. below `end`: the lanes of a group of kRowLanes stream row v and
// count its members of N(u).
template <class Member>
__device__ __forceinline__ void support_of_rows(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ col,
                                                const uint32_t* __restrict__ ubase, uint32_t u, uint32_t ub, uint32_t du,
                                                uint32_t first, uint32_t end, uint32_t step, uint32_t* sup,
                                                Member member) {
  const uint32_t l = lane_id() % kRowLanes;
  const uint32_t mask = 0xffu << (lane_id() / kRowLanes * kRowLanes);
  for (uint32_t j = first; j < end; j += step) {
    const uint32_t v = col[ub + j], b = rp[v], e = rp[v + 1];
    if (e - b > du || (e - b == du && v > u)) continue;
    uint32_t hits = 0, at = 0;  // at: u's position in row v
    for (uint32_t i0 = b; i0 < e; i0 += 4u * kRowLanes) {
      uint32_t x[4];
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q) {
        const uint32_t i = i0 + q * kRowLanes + l;
        x[q] = i < e ? col[i] : 0xffffffffu;
      }
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q) {
        if (x[q] == u) at = i0 + q * kRowLanes + l - b;
        if (x[q] != 0xffffffffu && member(x[q])) ++hits;
      }
    }
#pragma unroll
    for (uint32_t o = 1; o < kRowLanes; o <<= 1) {
      hits += __shfl_xor_sync(mask, hits, o);
      at = max(at, __shfl_xor_sync(mask, at, o));
    }
    if (l == 0) sup[support_index(rp, ubase, u, v, j, at)] = hits;
  }
}

template <uint32_t CAP>
__global__ void __launch_bounds__(256) k_support_small(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ col,
                                                       uint32_t n, const uint32_t* __restrict__ ubase, uint32_t* sup) {
  __shared__ uint32_t rows[8][CAP];
  uint32_t* su = rows[threadIdx.x >> 5];
  const uint32_t lane = lane_id();
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t u = gw; u < n; u += nw) {
    const uint32_t ub = rp[u], du = rp[u + 1] - ub;
    if (du == 0u || du > CAP) continue;
    const uint32_t cap = du <= 32u ? 32u : CAP;
    __syncwarp();
    for (uint32_t i = lane; i < cap; i += 32u) su[i] = i < du ? col[ub + i] : 0xffffffffu;
    __syncwarp();
    support_of_rows(rp, col, ubase, u, ub, du, lane / kRowLanes, du, 32u / kRowLanes, sup, [&](uint32_t x) {
      uint32_t j = 0;  // the last entry <= x, or the first
      for (uint32_t s = cap / 2u; s; s >>= 1)
        if (su[j + s] <= x) j += s;
      return su[j] == x;
    });
  }
}

template <int BT>
__global__ void __launch_bounds__(BT) k_support_big(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ col,
                                                    uint32_t n, const uint32_t* __restrict__ ubase,
                                                    const uint2* __restrict__ list, const uint32_t* count,
                                                    uint32_t max_tasks, uint32_t least, uint32_t* ticket,
                                                    uint32_t* sup) {
  extern __shared__ __align__(16) uint32_t bits[];
  __shared__ uint32_t next;
  const uint32_t words = (n + 31u) / 32u, cnt = min(*count, max_tasks);
  for (uint32_t i = threadIdx.x; i < words; i += BT) bits[i] = 0u;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) next = atomicAdd(ticket, 1u);
    __syncthreads();
    if (next >= cnt) break;
    const uint2 task = list[next];
    const uint32_t u = task.x, ub = rp[u], du = rp[u + 1] - ub;
    for (uint32_t i = threadIdx.x; i < du; i += BT) {
      const uint32_t x = col[ub + i];
      atomicOr(&bits[x >> 5], 1u << (x & 31u));
    }
    __syncthreads();
    support_of_rows(rp, col, ubase, u, ub, du, task.y + threadIdx.x / kRowLanes, min(du, task.y + support_chunk(du, least)),
                    BT / kRowLanes, sup,
                    [&](uint32_t x) { return (bits[x >> 5] >> (x & 31u)) & 1u; });
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < du; i += BT) bits[col[ub + i] >> 5] = 0u;
  }
}

// One warp per edge, for graphs whose bitmap does not fit.
__global__ void k_support(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ col, uint32_t n,
                          const uint32_t* __restrict__ ubase, uint32_t m, uint32_t* sup) {
  const uint32_t lane = lane_id();
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t e = gw; e < m; e += nw) {
    // row of edge e: last u with ubase[u] <= e
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (ubase[mid] <= e) lo = mid; else hi = mid;
    }
    const uint32_t u = lo;
    const uint32_t ub = rp[u], ue = rp[u + 1];
    const uint32_t first_upper = ue - (ubase[u + 1] - ubase[u]);
    const uint32_t v = col[first_upper + (e - ubase[u])];
    const uint32_t vb = rp[v], ve = rp[v + 1];
    const uint32_t *A, *L;
    uint32_t la, ll;
    if (ue - ub <= ve - vb) { A = col + ub; la = ue - ub; L = col + vb; ll = ve - vb; }
    else { A = col + vb; la = ve - vb; L = col + ub; ll = ue - ub; }
    uint32_t c = 0;
    for (uint32_t i0 = 0; i0 < la; i0 += 32) {
      const uint32_t i = i0 + lane;
      bool hit = false;
      if (i < la) {
        const uint32_t x = A[i];
        const uint32_t pos = lower_bound_u32(L, ll, x);
        hit = pos < ll && L[pos] == x;
      }
      c += __popc(__ballot_sync(0xffffffffu, hit));
    }
    if (lane == 0) sup[e] = c;
  }
}

}  // namespace

kc_status truss_support(kc_graph* g, uint32_t* d_support) {
  kc_ctx* ctx = g->ctx;
  cudaStream_t s = ctx->stream;
  const uint32_t n = g->n;
  if (g->m == 0) return KC_OK;
  DevTemps t(s);
  uint32_t *cnt = nullptr, *ubase = nullptr;
  KC_CUDA(t.alloc(&cnt, sizeof(uint32_t) * ((size_t)n + 1)));
  KC_CUDA(t.alloc(&ubase, sizeof(uint32_t) * ((size_t)n + 1)));
  const uint32_t g1 = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, (uint64_t)ctx->sms * 16));
  k_upper_count<<<g1, 256, 0, s>>>(g->rp, g->col, n, cnt);
  KC_CUDA(prim::scan_exclusive_u32(cnt, ubase, n, s));
  if (n <= kSupportBitmap && g->m >= kSupportEdges) {
    // four CTAs of 512 threads per SM while their bitmaps fit, else one of 1024,
    // for which only longer rows are worth a task
    const uint32_t bytes = (n + 31u) / 32u * 4u;
    const bool four = bytes <= 48u * 1024u;
    const uint32_t small = four ? kSupportSmall : kSupportMid;
    uint32_t* ctl = nullptr;  // [0] tasks of the large vertices, [1] ticket
    uint2* tasks = nullptr;
    const uint32_t least = g->m < kSupportFewEdges ? kSupportChunkFew : kSupportChunk;
    const uint32_t max_tasks = (uint32_t)(2 * g->m / kSupportSmall + 2 * g->m / least + 1);
    KC_CUDA(t.alloc(&ctl, 2 * sizeof(uint32_t)));
    KC_CUDA(t.alloc(&tasks, sizeof(uint2) * max_tasks));
    KC_CUDA(cudaMemsetAsync(ctl, 0, 2 * sizeof(uint32_t), s));
    k_support_list<<<g1, 256, 0, s>>>(g->rp, n, small, least, tasks, ctl);
    const uint32_t gs = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(((uint64_t)n * 32 + 255) / 256, (uint64_t)ctx->sms * 16));
    if (four) k_support_small<kSupportSmall><<<gs, 256, 0, s>>>(g->rp, g->col, n, ubase, d_support);
    else k_support_small<kSupportMid><<<gs, 256, 0, s>>>(g->rp, g->col, n, ubase, d_support);
    if (g->max_deg > small) {
      // (the limit is raised for both: the 48 KB a launch may take without that
      // hold the kernel's static shared memory too)
      if (four) {
        KC_CUDA(cudaFuncSetAttribute(k_support_big<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, 48 * 1024));
        k_support_big<512><<<ctx->sms * 4, 512, bytes, s>>>(g->rp, g->col, n, ubase, tasks, ctl, max_tasks, least, ctl + 1, d_support);
      } else {
        KC_CUDA(cudaFuncSetAttribute(k_support_big<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(kSupportBitmap / 8u)));
        k_support_big<1024><<<ctx->sms, 1024, bytes, s>>>(g->rp, g->col, n, ubase, tasks, ctl, max_tasks, least, ctl + 1, d_support);
      }
    }
  } else {
    const uint32_t g2 = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((g->m * 32 + 255) / 256, (uint64_t)ctx->sms * 32));
    k_support<<<g2, 256, 0, s>>>(g->rp, g->col, n, ubase, (uint32_t)g->m, d_support);
  }
  KC_CUDA(cudaGetLastError());
  return KC_OK;
}

}  // namespace kc
