// Bit rows of a batch of small graphs (bits.cu).
//
// Graph g's n_g vertices have n_g rows of bit_row_words(n_g) words at off[g] of
// `words`. Vertices are the batch's: graph g owns [voff[g], voff[g + 1]), as
// vertex ids and as rank labels. Two sets of rows exist: kc_graph::bits, by
// vertex id, both directions of every edge; and kc_graph::dbits, by rank label,
// row r holding the labels above r that r is adjacent to (its out-list). Of a
// row of dbits only the words from bit_row_first(r) on are written and read.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "engine.h"

namespace kc {

struct BitRow {
  const uint32_t* row;
  uint32_t words;
};

// (a multiple of four: rows are read 16 bytes at a time)
__host__ __device__ __forceinline__ uint32_t bit_row_words(uint32_t n) { return ((n + 127u) >> 7) << 2; }
__device__ __forceinline__ uint32_t bit_row_first(uint32_t r) { return (r >> 7) << 2; }

// Row of the batch's vertex v, which belongs to graph gph.
__device__ __forceinline__ BitRow bit_row(const BitRows& b, uint32_t gph, uint32_t v) {
  const uint32_t v0 = b.voff[gph], words = bit_row_words(b.voff[gph + 1] - v0);
  return {b.words + b.off[gph] + (size_t)(v - v0) * words, words};
}

// Sets the bits of a batch's edges (ids local to their graphs) in the zeroed
// rows and fills g->rp (row offsets of the symmetric CSR), g->n, g->m and
// g->max_deg; with `columns` also g->col (sorted rows). An endpoint that is
// not below its graph's vertex count sets *err to 1 + the graph. `err` is
// read back by the call.
kc_status build_bits(kc_graph* g, const uint32_t* d_src, const uint32_t* d_dst, uint64_t E,
                     const unsigned long long* d_eoff, uint32_t n_graphs, uint32_t n, bool columns, uint32_t* d_err,
                     uint32_t* h_err);
// The rows of dbits and the out-degrees, both in rank order (needs the ranks).
kc_status bits_dag(kc_graph* g, uint32_t* odeg);
// The DAG rows as lists of rank labels, in no order (needs the row pointer).
kc_status bits_dag_lists(kc_graph* g);

}  // namespace kc
