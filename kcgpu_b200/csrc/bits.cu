// Offsets and oriented bit rows of a batch of small graphs.
//
// The bit rows stand in for four passes of the general build (making ids
// global, degrees, scatter, row sort with dedup), its compaction, and the fill
// and sort of the DAG: setting a bit is idempotent, so duplicates and both
// directions cost nothing more, and a row holds its neighbours in order. The
// counting kernels then AND a unit's own row with the rows of its members
// (count_kernels.cu). What bounds the build is the L2's rate of 64 random
// atomics a cycle, two per edge; the rows are n^2 / 8 bytes per graph (0.34 MB
// on average for graphs of 50 to 5,000 vertices), written once and read twice.
// Batch of 2,500 mixed graphs (84M input edges): build and orientation 8.3 ms
// the general way, 4.1 ms here.
#include <algorithm>

#include "bits.cuh"
#include "dev_common.cuh"
#include "prims.cuh"

namespace kc {

namespace {

constexpr uint32_t kChunk = 4096;  // edges per CTA step of k_set_bits

__global__ void __launch_bounds__(256) k_set_bits(const uint32_t* __restrict__ src, const uint32_t* __restrict__ dst,
                                                  unsigned long long E, const unsigned long long* __restrict__ eoff,
                                                  uint32_t G, BitRows b, uint32_t* words, uint32_t* err) {
  for (unsigned long long c0 = (unsigned long long)blockIdx.x * kChunk; c0 < E;
       c0 += (unsigned long long)gridDim.x * kChunk) {
    // graph of the chunk's first edge: the last g with eoff[g] <= c0
    uint32_t g = 0, hi = G;
    while (hi - g > 1u) {
      const uint32_t mid = (g + hi) >> 1;
      if (eoff[mid] <= c0) g = mid;
      else hi = mid;
    }
    const unsigned long long end = min(E, c0 + (unsigned long long)kChunk);
    uint32_t cur = 0xffffffffu, n = 0, rw = 0;
    uint32_t* base = nullptr;
    for (unsigned long long i0 = c0 + threadIdx.x; i0 < end; i0 += 4u * 256u) {
      uint32_t u[4], v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const unsigned long long i = i0 + 256u * q;
        u[q] = i < end ? src[i] : 0u;
        v[q] = i < end ? dst[i] : 0u;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const unsigned long long i = i0 + 256u * q;
        if (i >= end) break;
        while (i >= eoff[g + 1]) ++g;  // (eoff[G] = E > i)
        if (g != cur) {
          cur = g;
          n = b.voff[g + 1] - b.voff[g];
          rw = bit_row_words(n);
          base = words + b.off[g];
        }
        if (u[q] >= n || v[q] >= n) {
          atomicCAS(err, 0u, g + 1u);
          continue;
        }
        if (u[q] == v[q]) continue;
        atomicOr(base + (size_t)u[q] * rw + (v[q] >> 5), 1u << (v[q] & 31u));
        atomicOr(base + (size_t)v[q] * rw + (u[q] >> 5), 1u << (u[q] & 31u));
      }
    }
  }
}

// Warp per vertex.
__global__ void k_bits_degree(BitRows b, const uint32_t* __restrict__ vg, uint32_t n, uint32_t* deg, uint32_t* max_deg) {
  const uint32_t lane = lane_id();
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  uint32_t mx = 0;
  for (uint32_t v = gw; v < n; v += nw) {
    const BitRow r = bit_row(b, vg[v], v);
    uint32_t c = 0;
    for (uint32_t w = lane * 4u; w < r.words; w += 128u) {
      const uint4 x = *reinterpret_cast<const uint4*>(r.row + w);
      c += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) deg[v] = c;
    mx = max(mx, c);
  }
  if (lane == 0 && mx) atomicMax(max_deg, mx);
}

// The neighbours of a vertex, from its row: the warp lists the set bits of 32
// words at a time (at most 1,024, in shared memory), then the lanes take the
// listed neighbours in turn, so their loads (of ranks) are in flight together.
// f(u, valid) is called by whole warps, u local to the graph.
constexpr uint32_t kListed = 1024;

template <class F>
__device__ __forceinline__ void visit_row(const BitRow& r, uint16_t* list, F f) {
  const uint32_t lane = lane_id();
  for (uint32_t w0 = 0; w0 < r.words; w0 += 32u) {
    const uint32_t w = w0 + lane;
    const uint32_t x = w < r.words ? r.row[w] : 0u;
    const uint32_t c = __popc(x);
    uint32_t incl = c;
#pragma unroll
    for (uint32_t o = 1; o < 32u; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    uint32_t at = incl - c;
    for (uint32_t y = x; y; y &= y - 1u) list[at++] = (uint16_t)(w * 32u + (uint32_t)__ffs(y) - 1u);
    __syncwarp();
    for (uint32_t i0 = 0; i0 < total; i0 += 32u) {
      const bool valid = i0 + lane < total;
      f(valid ? (uint32_t)list[i0 + lane] : 0u, valid);
    }
    __syncwarp();
  }
}

__global__ void __launch_bounds__(256) k_bits_columns(BitRows b, const uint32_t* __restrict__ vg, uint32_t n,
                                                      const uint32_t* __restrict__ rp, uint32_t* col) {
  __shared__ uint16_t lists[8][kListed];
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t v = gw; v < n; v += nw) {
    const uint32_t g = vg[v], v0 = b.voff[g];
    uint32_t at = rp[v];
    visit_row(bit_row(b, g, v), lists[threadIdx.x >> 5], [&](uint32_t u, bool valid) {
      if (valid) col[at + lane_id()] = v0 + u;
      at += __popc(__ballot_sync(0xffffffffu, valid));
    });
  }
}

// Row rank[v] of `out` from row v: the ranks above it, set in shared memory and
// written from its first word on; and the out-degree.
__global__ void __launch_bounds__(256) k_bits_dag(BitRows b, const uint32_t* __restrict__ vg, uint32_t n,
                                                  const uint32_t* __restrict__ rank, uint32_t* out, uint32_t* odeg) {
  __shared__ uint16_t lists[8][kListed];
  __shared__ __align__(16) uint32_t rows[8][kBitsMaxVertices / 32u];
  const uint32_t lane = lane_id();
  uint32_t* row = rows[threadIdx.x >> 5];
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t v = gw; v < n; v += nw) {
    const uint32_t g = vg[v], v0 = b.voff[g], rv = rank[v] - v0;
    const BitRow r = bit_row(b, g, v);
    const uint32_t first = bit_row_first(rv);
    for (uint32_t w = first + lane; w < r.words; w += 32u) row[w] = 0u;
    __syncwarp();
    uint32_t c = 0;
    visit_row(r, lists[threadIdx.x >> 5], [&](uint32_t u, bool valid) {
      const uint32_t ru = valid ? rank[v0 + u] - v0 : 0u;
      if (ru > rv) {
        atomicOr(&row[ru >> 5], 1u << (ru & 31u));
        ++c;
      }
    });
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) odeg[rv + v0] = c;
    uint32_t* to = out + b.off[g] + (size_t)rv * r.words;
    for (uint32_t w = first + lane; w < r.words; w += 32u) to[w] = row[w];
    __syncwarp();
  }
}

__global__ void __launch_bounds__(256) k_bits_dag_lists(BitRows b, const uint32_t* __restrict__ vg, uint32_t n,
                                                        const uint32_t* __restrict__ rank,
                                                        const uint32_t* __restrict__ drp, uint32_t* dcol) {
  __shared__ uint16_t lists[8][kListed];
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t v = gw; v < n; v += nw) {
    const uint32_t g = vg[v], v0 = b.voff[g], rv = rank[v];
    uint32_t at = drp[rv];
    visit_row(bit_row(b, g, v), lists[threadIdx.x >> 5], [&](uint32_t u, bool valid) {
      const uint32_t ru = valid ? rank[v0 + u] : 0u;
      const bool keep = ru > rv;
      const uint32_t m = __ballot_sync(0xffffffffu, keep);
      if (keep) dcol[at + __popc(m & lanemask_lt())] = ru;
      at += __popc(m);
    });
  }
}

uint32_t warp_grid(uint64_t n, int sms) {
  return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((n * 32 + 255) / 256, (uint64_t)sms * 32));
}

}  // namespace

kc_status build_bits(kc_graph* g, const uint32_t* d_src, const uint32_t* d_dst, uint64_t E,
                     const unsigned long long* d_eoff, uint32_t n_graphs, uint32_t n, bool columns, uint32_t* d_err,
                     uint32_t* h_err) {
  cudaStream_t s = g->ctx->stream;
  const int sms = g->ctx->sms;
  g->n = n;
  DevTemps t(s);
  uint32_t *deg = nullptr, *mx = nullptr;
  KC_CUDA(t.alloc(&deg, sizeof(uint32_t) * ((size_t)n + 1)));
  KC_CUDA(t.alloc(&mx, sizeof(uint32_t)));
  KC_CUDA(cudaMemsetAsync(mx, 0, sizeof(uint32_t), s));
  KC_CUDA(cudaMemsetAsync(g->bit_words, 0, sizeof(uint32_t) * g->n_bit_words, s));
  const uint32_t ge = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((E + kChunk - 1) / kChunk, (uint64_t)sms * 8));
  if (E) k_set_bits<<<ge, 256, 0, s>>>(d_src, d_dst, E, d_eoff, n_graphs, g->bits, g->bit_words, d_err);
  if (n) k_bits_degree<<<warp_grid(n, sms), 256, 0, s>>>(g->bits, g->vgraph_orig, n, deg, mx);
  KC_TRY(dev_alloc(g, (void**)&g->rp, sizeof(uint32_t) * ((size_t)n + 1)));
  KC_CUDA(prim::scan_exclusive_u32(deg, g->rp, n, s));
  uint32_t m2 = 0;
  KC_CUDA(cudaMemcpyAsync(h_err, d_err, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  KC_CUDA(cudaMemcpyAsync(&m2, g->rp + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  KC_CUDA(cudaMemcpyAsync(&g->max_deg, mx, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  KC_CUDA(cudaStreamSynchronize(s));
  if (*h_err) return KC_OK;  // (the caller reports it)
  g->m = m2 / 2;
  if (columns) {
    KC_TRY(dev_alloc(g, (void**)&g->col, sizeof(uint32_t) * std::max<size_t>(1, m2)));
    if (n) k_bits_columns<<<warp_grid(n, sms), 256, 0, s>>>(g->bits, g->vgraph_orig, n, g->rp, g->col);
  }
  KC_CUDA(cudaGetLastError());
  return KC_OK;
}

kc_status bits_dag(kc_graph* g, uint32_t* odeg) {
  KC_TRY(dev_alloc(g, (void**)&g->dbit_words, sizeof(uint32_t) * std::max<uint64_t>(1, g->n_bit_words)));
  g->dbits = g->bits;
  g->dbits.words = g->dbit_words;
  if (g->n)
    k_bits_dag<<<warp_grid(g->n, g->ctx->sms), 256, 0, g->ctx->stream>>>(g->bits, g->vgraph_orig, g->n, g->rank,
                                                                      g->dbit_words, odeg);
  KC_CUDA(cudaGetLastError());
  return KC_OK;
}

kc_status bits_dag_lists(kc_graph* g) {
  if (g->n)
    k_bits_dag_lists<<<warp_grid(g->n, g->ctx->sms), 256, 0, g->ctx->stream>>>(g->bits, g->vgraph_orig, g->n, g->rank,
                                                                            g->drp, g->dcol);
  KC_CUDA(cudaGetLastError());
  return KC_OK;
}

}  // namespace kc
