// Bitmap-encoded counting kernels (orientation and pivoting) and the launch
// planner shared with the list-encoded kernels.
//
// One kernel body serves node and edge units; the unit only changes how the
// vertex set S is formed:
//   node unit u:     S = N+(u)                 (kckernels_orientation.cuh:357-377)
//   edge unit u->v:  S = N+(u) ∩ N+(v)         (kckernels_orientation.cuh:518-555)
// Orientation traversal (kckernels_orientation.cuh:380-470): every t-clique
// (t = k-1 for node units, k-2 for edge units) of the DAG on S is counted
// once from its lowest vertex; the last level is counted by popcount.
// Pivot traversal (kckernels_pivoting.cuh:124-338): the succinct clique tree
// with the max-neighbourhood pivot, ties to the smallest index; a leaf adds
// C(drop, k - held) from an exact table (the reference parses doubles,
// kclique/kclique.cuh:1694-1717). Where this differs from the reference in
// how, not what:
//   * a whole warp walks one tree node (the reference walks one node per
//     block with __syncthreads between steps); the launch's partition size
//     bounds the lanes that score one pivot candidate, as the reference's
//     partitions split the candidates of the block's node (:250-308);
//   * nodes with r = k - held <= 2 are closed: 1, |C| + drop, or
//     edges(G[C]) + drop |C| + C(drop, 2), instead of expanding their leaves;
//   * the pivot's own branch is taken last and reuses its parent's frame, so
//     the stack holds at most k - held0 + 1 frames;
//   * a unit's tree is cut at depth 1, 2 or 3 and the nodes at the cut go to
//     the unit's warps by ticket (a dense unit's root has few branches);
//   * edge units are grouped by source when N+(u) fits a shared-memory bitmap:
//     the unit u builds G[N+(u)] once and its out-edges are the root branches.
#include <algorithm>
#include <type_traits>

#include "bits.cuh"
#include "count_kernels.cuh"
#include "dev_common.cuh"

namespace kc {

namespace {

struct Part {
  uint32_t P, plane, pmask, pbase;
};

// First set bit of set[w0, W) (all lanes of the partition agree); -1 if none.
__device__ __forceinline__ int part_next_bit(const uint32_t* set, uint32_t w0, uint32_t W, const Part& pt,
                                             uint32_t* wi) {
  for (uint32_t base = w0; base < W; base += pt.P) {
    const uint32_t w = base + pt.plane;
    const uint32_t x = w < W ? set[w] : 0u;
    const uint32_t bal = (__ballot_sync(pt.pmask, x != 0u) & pt.pmask) >> pt.pbase;
    if (bal) {
      const uint32_t f = __ffs(bal) - 1;
      const uint32_t xv = __shfl_sync(pt.pmask, x, pt.pbase + f);
      *wi = base + f;
      return (int)((base + f) * 32u + (uint32_t)__ffs(xv) - 1u);
    }
  }
  return -1;
}

__device__ __forceinline__ uint32_t low_mask(uint32_t v, uint32_t w) {  // bits < v inside word w
  const uint32_t vw = v >> 5;
  return w < vw ? 0xffffffffu : (w == vw ? ((1u << (v & 31u)) - 1u) : 0u);
}

__device__ __forceinline__ uint32_t valid_mask(uint32_t d, uint32_t w) {  // bits < d inside word w
  return low_mask(d, w);
}

// Gather tables (shared memory, needed until the bitmap stands): the member
// map of up to kSpanWords * 32 rank labels with its prefix, or, for a wider S,
// a hash (hT keys, 16-bit local indices) behind a filter of one bit per hash
// value; then the row table (start and length of every row).
constexpr uint32_t kSpanWords = 256;
__host__ __device__ constexpr uint32_t filter_words(uint32_t G) { return G == 32u ? 256u : 1024u; }
__host__ __device__ constexpr uint32_t gather_rows_at(uint32_t hT, uint32_t G) {
  return hT + hT / 2u + filter_words(G) > 2u * kSpanWords ? hT + hT / 2u + filter_words(G) : 2u * kSpanWords;
}
constexpr uint32_t kRowLanes = 8;  // gather: lanes that read one row together

template <int NW>
__device__ __forceinline__ void load_row(const uint32_t* B, uint32_t v, uint32_t (&r)[NW]) {
  if constexpr (NW == 4) {
    const uint4 q = *reinterpret_cast<const uint4*>(B + v * 4u);
    r[0] = q.x; r[1] = q.y; r[2] = q.z; r[3] = q.w;
  } else if constexpr (NW == 2) {
    const uint2 q = *reinterpret_cast<const uint2*>(B + v * 2u);
    r[0] = q.x; r[1] = q.y;
  } else {
    r[0] = B[v];
  }
}

// Position of the r-th (0-based) set bit of x (x has more than r set bits).
__device__ __forceinline__ uint32_t select_bit(uint32_t x, uint32_t r) {
  uint32_t pos = 0;
#pragma unroll
  for (uint32_t w = 16; w; w >>= 1) {
    const uint32_t lowc = __popc(x & ((1u << w) - 1u));
    if (r >= lowc) {
      r -= lowc;
      x >>= w;
      pos += w;
    }
  }
  return pos;
}

// Orientation traversal with one lane per subtree: the candidate set (NW
// words) lives in registers, rows come from shared memory with one vector
// load, and a lane's stack holds only the sets of the levels above it.
// Counts the t-cliques of the unit whose bitmap B has rows of stride NW.
// Lanes take subtrees by ticket: second-level vertices j (row j), or, when
// pre holds the exclusive prefix of the row popcounts (pre[d] = edges of
// G[S]), the third-level pairs (j, i), i in row j, with candidates
// row j ∩ row i: a unit's first rows are its largest, and splitting them
// keeps one lane from holding a warp's whole tail.
// Returns false when the unit ran over its budget (its count is then void).
template <int NW>
__device__ bool lane_dfs(const uint32_t* B, uint32_t d, uint32_t t, const uint32_t* pre, uint32_t* hdr,
                         uint32_t budget, unsigned __int128& uacc, unsigned long long& st_nodes,
                         unsigned long long& st_words KC_ERR_PARAM) {
  uint32_t stk[kLaneStack][NW];
  unsigned long long cnt = 0;
  uint32_t since = 0;
  bool ok = true;
  const bool pairs = pre != nullptr;
  const uint32_t total = pairs ? pre[d] : d;
  t = pairs ? t - 1u : t;  // a pair's candidates complete (t-1)-cliques the same way a row's complete t-cliques
  for (;;) {
    if (budget && *(volatile uint32_t*)&hdr[5]) { ok = false; break; }
    const uint32_t tk = atomicAdd(&hdr[1], 1u);
    if (tk >= total) break;
    uint32_t cur[NW];
    if (pairs) {
      uint32_t lo = 0, hi = d;  // pre[lo] <= tk < pre[hi]
      while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (pre[mid] <= tk) lo = mid;
        else hi = mid;
      }
      uint32_t rj[NW], ri[NW];
      load_row<NW>(B, lo, rj);
      uint32_t r = tk - pre[lo], i = 0;
      bool found = false;
#pragma unroll
      for (int q = 0; q < NW; ++q) {
        const uint32_t pc = __popc(rj[q]);
        if (!found && r < pc) {
          i = (uint32_t)q * 32u + select_bit(rj[q], r);
          found = true;
        } else if (!found) {
          r -= pc;
        }
      }
      load_row<NW>(B, i, ri);
#pragma unroll
      for (int q = 0; q < NW; ++q) cur[q] = rj[q] & ri[q];
    } else {
      load_row<NW>(B, tk, cur);
    }
    uint32_t c = 0;
#pragma unroll
    for (int q = 0; q < NW; ++q) c += __popc(cur[q]);
    st_nodes++;
    st_words += NW;
    if (t == 2u) { cnt += c; continue; }
    if (c < t - 1u) continue;
    int lv = 0;
    for (;;) {
      int w = -1;
#pragma unroll
      for (int q = NW - 1; q >= 0; --q)
        if (cur[q]) w = q;
      if (w < 0) {
        if (lv == 0) break;
        --lv;
#pragma unroll
        for (int q = 0; q < NW; ++q) cur[q] = stk[lv][q];
        continue;
      }
      uint32_t word = 0;
#pragma unroll
      for (int q = 0; q < NW; ++q)
        if (q == w) { word = cur[q]; cur[q] = word & (word - 1u); }
      const uint32_t v = (uint32_t)w * 32u + (uint32_t)__ffs(word) - 1u;
      uint32_t row[NW], child[NW];
      load_row<NW>(B, v, row);
      uint32_t n = 0;
#pragma unroll
      for (int q = 0; q < NW; ++q) {
        child[q] = cur[q] & row[q];
        n += __popc(child[q]);
      }
      st_nodes++;
      st_words += NW;
      const uint32_t rem = t - (uint32_t)(lv + 2);
      if (rem == 1u) {
        cnt += n;
      } else if (n >= rem && KC_IN_BOUNDS(lv, kLaneStack, err)) {
#pragma unroll
        for (int q = 0; q < NW; ++q) {
          stk[lv][q] = cur[q];
          cur[q] = child[q];
        }
        ++lv;
      }
      if (budget && ++since >= 64u) {
        since = 0;
        if (atomicAdd(&hdr[4], 64u) + 64u > budget) hdr[5] = 1u;
        if (*(volatile uint32_t*)&hdr[5]) { ok = false; break; }
      }
    }
    if (!ok) break;
  }
  uacc += cnt;
  return ok;
}

// ---- small clique-tree nodes, closed in one step ------------------------------
//
// A pivoting node (candidate set F of nc vertices, `drop` pivots, r = k - held)
// contributes sum_j C(drop, j) cliques(G[F], r - j). Walked node by node that
// costs a warp about 1.5 us of latency per tree node (frame, candidate list,
// scores, reductions) with most lanes idle, and almost all nodes of a tree are
// small and near its leaves. Two kinds are therefore counted whole: r = 3 with
// at most 128 candidates (the triangles of G[F]) and r up to 19 with at most 32
// candidates (a lane per subproblem).
// Both first copy G[F] into a compact bitmap of nc rows and ceil(nc / 32)
// words. Larger nodes are worth splitting further: their branches are what
// the walkers share. R-MAT scale 17, k = 5 (edge units): 37.8M tree nodes,
// 37.1 ms before; 1.4M, 6.3 ms now. Chung-Lu 1M + planted cliques, k = 6
// (node units): 76.7M, 145 ms before; 3.7M, 48 ms now (r = 4 closed the same
// way, a triangle count per vertex, took 42 ms where this had come to 30).
// R-MAT of 21k edges, k = 8, built, oriented and counted: 3.5 ms before, 1.6 ms.

// Words of the compact bitmap of up to `n` candidates.
__host__ __device__ constexpr uint32_t compact_words(uint32_t n) {
  return n <= 32u ? 36u : (n <= 64u ? 64u * 2u : 128u * 4u);
}

// The compact bitmap of the candidates cand[0, nc) (ascending): bit i of row j
// is set when cand[i] and cand[j] are adjacent (UPPER: and i > j). The lanes
// test a row's nc bits side by side, and a ballot makes 32 of them a word: the
// lanes read one row of B at a time, so there are no bank conflicts, and there
// is no dependence between rows. Rows have ST words in out (ST = 1, 2 or 4).
template <int NW, int ST, bool UPPER>
__device__ __forceinline__ void compact_rows(const uint32_t* B, uint32_t Ws, const uint32_t* cand, uint32_t nc,
                                             uint32_t* out KC_ERR_PARAM) {
  const uint32_t lane = lane_id();
  uint32_t cw[NW], cb[NW];
#pragma unroll
  for (int t = 0; t < NW; ++t) {
    const uint32_t i = (uint32_t)t * 32u + lane;
    const uint32_t c = cand[i < nc ? i : 0u];
    cw[t] = c >> 5;
    cb[t] = i < nc ? (1u << (c & 31u)) : 0u;
  }
#pragma unroll
  for (int jb = 0; jb < NW; ++jb) {  // rows 32 jb .. 32 jb + 31
    const uint32_t je = min(nc, (uint32_t)jb * 32u + 32u);
#pragma unroll 4
    for (uint32_t j = (uint32_t)jb * 32u; j < je; ++j) {
      const uint32_t* row = B + cand[j] * Ws;
      uint32_t m[ST];
#pragma unroll
      for (int t = 0; t < ST; ++t) {
        m[t] = 0u;
        if (t < NW && (!UPPER || t >= jb)) {
          m[t] = __ballot_sync(0xffffffffu, (row[cw[t < NW ? t : 0]] & cb[t < NW ? t : 0]) != 0u);
          if (UPPER && t == jb) m[t] &= 0xfffffffeu << (j & 31u);
        }
      }
      if (lane == 0 && KC_IN_BOUNDS(j * ST + ST - 1u, compact_words(32u * NW), err)) {
        if constexpr (ST == 4) *reinterpret_cast<uint4*>(out + j * 4u) = make_uint4(m[0], m[1], m[2], m[3]);
        else if constexpr (ST == 2) *reinterpret_cast<uint2*>(out + j * 2u) = make_uint2(m[0], m[1]);
        else out[j] = m[0];
      }
    }
  }
  __syncwarp();
}

// Carry-save counter of set bits: POPC runs at an eighth of the logic rate, so
// four words are added into `ones` / `twos` with six LOP3 and one POPC.
struct BitCount {
  uint32_t ones = 0, twos = 0, fours = 0;  // fours: already popcounted
  __device__ __forceinline__ void add4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    const uint32_t t1 = (ones & a) | (ones & b) | (a & b);
    ones = ones ^ a ^ b;
    const uint32_t t2 = (ones & c) | (ones & d) | (c & d);
    ones = ones ^ c ^ d;
    const uint32_t f = (twos & t1) | (twos & t2) | (t1 & t2);
    twos = twos ^ t1 ^ t2;
    fours += __popc(f);
  }
  __device__ __forceinline__ uint32_t total() const { return 4u * fours + 2u * __popc(twos) + __popc(ones); }
};

// The upper rows i, i + 32, .. (ST words each) of lane i, from up; returns the
// lane's share of the edges.
template <int NW, int ST>
__device__ __forceinline__ uint32_t own_rows(const uint32_t* up, uint32_t nc, uint32_t (&P)[NW][ST]) {
  uint32_t edges = 0;
#pragma unroll
  for (int g = 0; g < NW; ++g) {
    const uint32_t i = (uint32_t)g * 32u + lane_id();
#pragma unroll
    for (int w = 0; w < ST; ++w) P[g][w] = 0u;
    if (i < nc) load_row<ST>(up, i, P[g]);
#pragma unroll
    for (int w = g; w < NW; ++w) edges += __popc(P[g][w]);
  }
  return edges;
}

// Four upper rows j0 .. j0 + 3 of block jb, the same for every lane.
template <int ST>
__device__ __forceinline__ void four_rows(const uint32_t* up, uint32_t j0, uint32_t (&U)[4][ST]) {
  if constexpr (ST == 1) {
    load_row<4>(up + j0, 0u, *reinterpret_cast<uint32_t(*)[4]>(&U[0][0]));
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) load_row<ST>(up, j0 + (uint32_t)q, U[q]);
  }
}

// Common upper neighbours of the lane's row P (words from jb on) and of those
// of the four rows U that it holds (bits j0 .. j0 + 3 of block jb).
template <int NW, int ST>
__device__ __forceinline__ void add_common(BitCount& bc, const uint32_t (&P)[ST], const uint32_t (&U)[4][ST], int jb,
                                           uint32_t j0) {
  uint32_t has[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) has[q] = (uint32_t)((int32_t)(P[jb] << (31u - ((j0 + (uint32_t)q) & 31u))) >> 31);
#pragma unroll
  for (int w = 0; w < NW; ++w)
    if (w >= jb)
      bc.add4(P[w] & U[0][w] & has[0], P[w] & U[1][w] & has[1], P[w] & U[2][w] & has[2], P[w] & U[3][w] & has[3]);
}

// Triangles of a graph of nc <= 32 NW vertices whose upper rows (zero rows up
// to a multiple of four) are in up: every row j is broadcast to all lanes, and
// a lane whose rows hold j adds the common upper neighbours. No divergence and
// no bank conflicts, about nc^2 / 64 words per lane whatever the density.
// Returns the lane's share of the triangles and, in edges, of the edges.
template <int NW, int ST>
__device__ __forceinline__ uint32_t count_triangles(const uint32_t* up, uint32_t nc, uint32_t& edges) {
  uint32_t P[NW][ST];
  edges = own_rows<NW, ST>(up, nc, P);
  BitCount bc;
#pragma unroll
  for (int jb = 0; jb < NW; ++jb) {  // rows 32 jb .. 32 jb + 31
    const uint32_t je = min(nc, (uint32_t)jb * 32u + 32u);
    for (uint32_t j0 = (uint32_t)jb * 32u; j0 < je; j0 += 4u) {
      uint32_t U[4][ST];
      four_rows<ST>(up, j0, U);
#pragma unroll
      for (int g = 0; g < NW; ++g)
        if (g <= jb) add_common<NW, ST>(bc, P[g], U, jb, j0);
    }
  }
  return bc.total();
}

constexpr uint32_t kPairPrefix = 36;   // close_small: exclusive prefix of the row lengths
constexpr uint32_t kWideMax = 128;     // most candidates of an r = 3 node closed whole
constexpr uint32_t kSmallMax = 32;     // most candidates of any other node closed whole
constexpr int kSmallStack = 16;        // close_small: a lane's own frames (r - 3 at most)
constexpr uint32_t kSmallMaxR = 19;
constexpr uint32_t kQueueCap = 236;    // close_small: nodes on its shared stack
// several k: the largest r closed whole, and the words of its histogram. No more
// vertices than the node has can be held, so a node of nc candidates is closed
// as one of r = nc where r is larger (multi_r): k = 3..33 over blocks of 100
// vertices (p = 0.4) took 1.62 ms with r alone deciding, 0.40 ms so.
constexpr uint32_t kSmallMaxRMulti = 15;
__device__ __forceinline__ uint32_t multi_r(uint32_t r, uint32_t nc) { return min(r, max(nc, 3u)); }
constexpr uint32_t kHistWords = (kSmallMaxRMulti + 1u) * (kSmallMax + 1u);

// r = 3: triangles + drop edges + C(drop, 2) vertices + C(drop, 3). Every lane
// returns its share.
template <int NW, int ST>
__device__ __forceinline__ unsigned long long close_wide(const uint32_t* B, uint32_t Ws, const uint32_t* cand,
                                                         uint32_t nc, uint32_t* up, uint32_t drop KC_ERR_PARAM) {
  const uint32_t pad = (nc + 3u) & ~3u;
  if (lane_id() < (pad - nc) * ST && KC_IN_BOUNDS(pad * ST - 1u, compact_words(32u * NW), err)) up[nc * ST + lane_id()] = 0u;  // (nc is at most 32 NW, a multiple of four)
  compact_rows<NW, ST, true>(B, Ws, cand, nc, up KC_ERR_ARG(err));
  uint32_t edges = 0;
  const unsigned long long d1 = drop, d2 = drop >= 2u ? d1 * (d1 - 1ull) / 2ull : 0ull;
  unsigned long long t = count_triangles<NW, ST>(up, nc, edges);
  t += d1 * edges;
  if (lane_id() == 0) t += d2 * nc + (drop >= 3u ? d2 * (d1 - 2ull) / 3ull : 0ull);
  return t;
}

__device__ __forceinline__ unsigned __int128 binom_at(const unsigned long long* binom, uint32_t cols, uint32_t nn,
                                                      uint32_t r) {
  if (r > nn) return 0;
  const unsigned long long* e = binom + 2ull * ((size_t)nn * (cols + 1u) + r);
  return ((unsigned __int128)e[1] << 64) | e[0];
}

// r >= 3 with at most 32 candidates: adj holds their rows (one word each,
// symmetric). The lanes count subproblems (set, vertices to go, pivots) side by
// side, with sets in registers, the last three levels by listing:
//   * r <= 4: a task is a pair i < j of adjacent candidates, with the common
//     neighbours above j as its set and r - 2 vertices to go (pairs, not
//     vertices: a dense node's first vertices hold most of its cliques);
//   * r > 4: the tasks are clique-tree nodes on a stack in shared memory. Up to
//     32 of them are taken at a time; a lane closes its node or pushes its
//     branches. Splitting by pivots keeps a near-clique's tree small, where
//     pairs would walk it once per pair (R-MAT of 21k edges, k = 8: 1.1 ms for
//     the units of up to 32 vertices by pairs, 0.06 ms). Lanes whose branches no
//     longer fit walk their nodes to the end on stacks of their own.
// Vertices adjacent to the whole set are moved to the pivots at once (their
// branches are empty). Returns the lane's share; pre[32] receives the steps
// (rows visited, the most of any lane per round).
//
// MK (several k in one walk): nothing is known of the smaller k, so instead of
// binomials of one k the lanes count, in hist[h (kSmallMax + 1) + x], the
// cliques of F by the h vertices they hold and the x pivots of F that may join
// them: each stands for C(drop + x, k - held - h) cliques of every k. r belongs
// to the largest k; the closed forms for r <= 3 hold for every smaller k too.
// R-MAT of 55k edges, k = 3..15 in one walk: 11.5 ms with every node walked,
// 4.2 ms by pairs, 1.5 ms now.
template <bool MK>
__device__ __forceinline__ unsigned __int128 close_small(const uint32_t* adj, uint32_t* pre, uint32_t nc, uint32_t r,
                                                         uint32_t drop, const unsigned long long* binom, uint32_t cols,
                                                         uint2* queue, uint32_t* hist KC_ERR_PARAM) {
  const uint32_t lane = lane_id();
  const uint32_t mine = lane < nc ? adj[lane] : 0u;
  unsigned __int128 acc = 0;
  uint32_t it = 0, steps = 0;
  auto put = [&](uint32_t held, uint32_t dd, uint32_t times) {
    if (times && KC_IN_BOUNDS(held * (kSmallMax + 1u) + (dd - drop), kHistWords, err))
      atomicAdd(&hist[held * (kSmallMax + 1u) + (dd - drop)], times);
  };
  // a node (P, rr vertices to go, dd pivots) without candidates, or with rr <= 3
  auto leaf = [&](uint32_t rr, uint32_t dd) {
    if (MK) put(r - rr, dd, 1u);
    else acc += binom_at(binom, cols, dd, rr);
  };
  auto listed = [&](uint32_t P, uint32_t rr, uint32_t dd) {
    const uint32_t n = __popc(P);
    uint32_t e = 0, tri = 0;
    if (rr >= 2u)
      for (uint32_t x = P; x; x &= x - 1u) {
        const uint32_t u = (uint32_t)__ffs(x) - 1u;
        const uint32_t X = (x & (x - 1u)) & adj[u];
        e += __popc(X);
        ++it;
        if (rr == 3u)
          for (uint32_t y = X; y; y &= y - 1u) {
            tri += __popc((y & (y - 1u)) & adj[__ffs(y) - 1]);
            ++it;
          }
      }
    if (MK) {
      put(r - rr, dd, 1u);
      put(r - rr + 1u, dd, n);
      if (rr >= 2u) put(r - rr + 2u, dd, e);
      if (rr == 3u) put(r, dd, tri);
    } else {
      const unsigned long long d1 = dd, d2 = dd >= 2u ? d1 * (d1 - 1ull) / 2ull : 0ull;
      if (rr == 1u) acc += n + d1;
      else if (rr == 2u) acc += e + d1 * n + d2;
      else acc += tri + d1 * e + d2 * n + (dd >= 3u ? d2 * (d1 - 2ull) / 3ull : 0ull);
    }
  };
  if (MK) {
    for (uint32_t i = lane; i < (r + 1u) * (kSmallMax + 1u) && KC_IN_BOUNDS(i, kHistWords, err); i += 32u) hist[i] = 0u;
    __syncwarp();
  }
  if (r <= 4u) {
    const uint32_t up = mine & (0xfffffffeu << lane);
    const uint32_t c = __popc(up);
    uint32_t incl = c;
#pragma unroll
    for (uint32_t o = 1; o < 32u; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    pre[lane] = incl - c;
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    if (lane == 0) {  // the empty set and the single candidates
      if (MK) {
        put(0u, drop, 1u);
        put(1u, drop, nc);
      } else {
        acc = binom_at(binom, cols, drop, r);
        if (drop + 1u >= r) acc += (unsigned __int128)nc * binom_at(binom, cols, drop, r - 1u);
      }
    }
    __syncwarp();
    for (uint32_t t = lane; t < total; t += 32u) {
      uint32_t i = 0;  // pre[i] <= t < pre[i + 1]
#pragma unroll
      for (uint32_t s = 16; s; s >>= 1)
        if (pre[i + s] <= t) i += s;
      const uint32_t ui = adj[i] & (0xfffffffeu << i);
      const uint32_t j = select_bit(ui, t - pre[i]);
      if (!KC_IN_BOUNDS(j, nc, err)) break;
      listed(ui & adj[j] & (0xfffffffeu << j), r - 2u, drop);
    }
    steps = __reduce_max_sync(0xffffffffu, it);
  } else {
    // the root: its scores are the row lengths
    const uint32_t s0 = __popc(mine);
    const uint32_t uni0 = __ballot_sync(0xffffffffu, lane < nc && s0 + 1u == nc);
    const uint32_t P0 = (nc < 32u ? (1u << nc) - 1u : 0xffffffffu) & ~uni0;
    const uint32_t d0 = drop + (uint32_t)__popc(uni0);
    uint32_t top = 0;
    if (!MK && __reduce_max_sync(0xffffffffu, s0) + 1u + drop < r) {
      // no clique of F is large enough
    } else if (P0 == 0u) {
      if (lane == 0) leaf(r, d0);
    } else {
      const bool in = (P0 >> lane) & 1u;
      const uint32_t piv = __reduce_max_sync(0xffffffffu, in ? (s0 << 8) | lane : 0u) & 31u;
      const uint32_t R = P0 & ~__shfl_sync(0xffffffffu, mine, piv) & ~(1u << piv);
      const uint32_t below = R & lanemask_lt();
      if ((R >> lane) & 1u) queue[__popc(below)] = make_uint2(P0 & ~below & mine, ((r - 1u) << 16) | d0);
      if (lane == piv) queue[__popc(R)] = make_uint2(P0 & ~R & mine, (r << 16) | (d0 + 1u));
      top = (uint32_t)__popc(R) + 1u;
    }
    __syncwarp();
    uint32_t sP[kSmallStack], sR[kSmallStack], sX[kSmallStack];  // set, branches left, (rr, pivot, dd)
    while (top) {
      const uint32_t cnt = min(top, 32u);
      top -= cnt;
      uint32_t P = 0, rr = 0, dd = 0, R = 0, piv = 0;
      bool work = lane < cnt;
      if (work) {
        const uint2 q = queue[top + lane];
        P = q.x;
        rr = q.y >> 16;
        dd = q.y & 0xffffu;
      }
      int lv = 0;
      for (bool own = false;; own = true) {  // own: on the lane's own stack
        uint32_t kids = 0;
        bool fresh = !own;
        while (work) {
          bool open = false;
          if (fresh) {
            const uint32_t n = __popc(P);
            if (MK || n + dd >= rr) {
              if (n == 0u) {
                leaf(rr, dd);
              } else if (rr <= 3u) {
                listed(P, rr, dd);
              } else {
                uint32_t best = 0, uni = 0;  // best: 1 + score, in the high half, of a non-universal candidate
                for (uint32_t x = P; x; x &= x - 1u) {
                  const uint32_t u = (uint32_t)__ffs(x) - 1u;
                  const uint32_t s = __popc(P & adj[u]);
                  if (s + 1u == n) uni |= 1u << u;
                  else best = max(best, ((s + 1u) << 16) | u);
                  ++it;
                }
                const uint32_t most = uni ? n : best >> 16;  // no clique of P has more vertices
                const bool enough = MK || most + dd >= rr;
                dd += __popc(uni);
                P &= ~uni;
                if (P == 0u) {
                  leaf(rr, dd);
                } else if (enough) {
                  open = true;
                  piv = best & 31u;
                  R = P & ~adj[piv] & ~(1u << piv);
                }
              }
            }
          }
          if (open && !own) {
            kids = (uint32_t)__popc(R) + 1u;
            break;
          }
          if (open && KC_IN_BOUNDS(lv, kSmallStack, err)) {
            sP[lv] = P;
            sR[lv] = R;
            sX[lv] = (rr << 24) | (piv << 16) | dd;
            ++lv;
          }
          if (lv == 0) break;
          // the next branch: the candidates outside the pivot's neighbourhood,
          // then the pivot's own branch in its parent's frame
          const uint32_t x = sX[lv - 1];
          R = sR[lv - 1];
          P = sP[lv - 1];
          rr = x >> 24;
          dd = x & 0xffffu;
          if (R) {
            const uint32_t u = (uint32_t)__ffs(R) - 1u;
            sR[lv - 1] = R & (R - 1u);
            sP[lv - 1] = P & ~(1u << u);
            P &= adj[u];
            --rr;
          } else {
            --lv;
            P &= adj[(x >> 16) & 31u];
            ++dd;
          }
          fresh = true;
        }
        __syncwarp();  // every node of the round has been read
        steps += __reduce_max_sync(0xffffffffu, it) + 2u;
        it = 0;
        if (own || !__any_sync(0xffffffffu, kids != 0u)) break;
        // the branches that fit go on the stack, in lane order
        uint32_t incl = kids;
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += y;
        }
        const bool fits = top + incl <= kQueueCap;
        if (kids && fits && KC_IN_BOUNDS(top + incl - 1u, kQueueCap, err)) {
          uint2* q = queue + top + (incl - kids);
          *q++ = make_uint2(P & ~R & adj[piv], (rr << 16) | (dd + 1u));
          for (uint32_t x = R; x; x &= x - 1u) {
            const uint32_t u = (uint32_t)__ffs(x) - 1u;
            *q++ = make_uint2(P & adj[u], ((rr - 1u) << 16) | dd);
            P &= ~(1u << u);
          }
        }
        top += __reduce_max_sync(0xffffffffu, fits ? incl : 0u);
        work = kids != 0u && !fits;
        if (work) {
          sP[0] = P;
          sR[0] = R;
          sX[0] = (rr << 24) | (piv << 16) | dd;
          lv = 1;
        }
        __syncwarp();
        if (!__any_sync(0xffffffffu, work)) break;
      }
    }
  }
  if (lane == 0) pre[32] = steps;
  return acc;
}

// A node counted whole (see above): its candidates are cand[0, nc), or, with
// cand null (r > 3, nc <= 32), its symmetric rows of one word are B itself. One copy of this
// code serves every call site. The lane's share is returned and cmp[0] holds
// the node's cost, in tree nodes of the work budget.
__device__ __noinline__ unsigned __int128 close_node(const uint32_t* B, uint32_t Ws, const uint32_t* cand, uint32_t nc,
                                                     uint32_t* cmp, uint32_t r, uint32_t drop,
                                                     const unsigned long long* binom, uint32_t cols KC_ERR_PARAM) {
  unsigned __int128 t;
  uint32_t cost = 1u + (nc >> 5);
  if (r > 3u && nc <= kSmallMax) {
    if (cand) compact_rows<1, 1, false>(B, Ws, cand, nc, cmp KC_ERR_ARG(err));
    t = close_small<false>(cand ? cmp : B, cmp + kPairPrefix, nc, r, drop, binom, cols,
                           reinterpret_cast<uint2*>(cmp + 2u * kPairPrefix), nullptr KC_ERR_ARG(err));
    __syncwarp();
    cost = 1u + (cmp[kPairPrefix + 32u] >> 4);
  } else if (nc <= 32u) {
    t = close_wide<1, 1>(B, Ws, cand, nc, cmp, drop KC_ERR_ARG(err));
  } else if (nc <= 64u) {
    t = close_wide<2, 2>(B, Ws, cand, nc, cmp, drop KC_ERR_ARG(err));
  } else if (nc <= 96u) {
    t = close_wide<3, 4>(B, Ws, cand, nc, cmp, drop KC_ERR_ARG(err));
  } else {
    t = close_wide<4, 4>(B, Ws, cand, nc, cmp, drop KC_ERR_ARG(err));
  }
  __syncwarp();
  if (lane_id() == 0) cmp[0] = cost;
  __syncwarp();
  return t;
}

// close_node for several k at once (nc <= 32; r of the largest k, or multi_r of
// it, at most kSmallMaxRMulti): the lane's own k has kr = k - held vertices to go (`open`: it is
// still to be counted), and its whole count below the node is returned.
__device__ __noinline__ unsigned __int128 close_node_multi(const uint32_t* B, uint32_t Ws, const uint32_t* cand,
                                                           uint32_t nc, uint32_t* cmp, uint32_t r, uint32_t drop,
                                                           const unsigned long long* binom, uint32_t cols,
                                                           uint32_t kr, bool open KC_ERR_PARAM) {
  const uint32_t lane = lane_id();
  uint32_t* hist = cmp + 2u * kPairPrefix + 2u * kQueueCap;
  if (cand) compact_rows<1, 1, false>(B, Ws, cand, nc, cmp KC_ERR_ARG(err));
  close_small<true>(cand ? cmp : B, cmp + kPairPrefix, nc, r, drop, binom, cols,
                    reinterpret_cast<uint2*>(cmp + 2u * kPairPrefix), hist KC_ERR_ARG(err));
  __syncwarp();
  unsigned __int128 t = 0;
  const uint32_t words = (r + 1u) * (kSmallMax + 1u);
  for (uint32_t i0 = 0; i0 < words; i0 += 32u) {
    const uint32_t mine = i0 + lane < words ? hist[i0 + lane] : 0u;
    for (uint32_t m = __ballot_sync(0xffffffffu, mine != 0u); m; m &= m - 1u) {
      const uint32_t b = (uint32_t)__ffs(m) - 1u;
      const uint32_t times = __shfl_sync(0xffffffffu, mine, b);
      const uint32_t h = (i0 + b) / (kSmallMax + 1u), x = (i0 + b) - h * (kSmallMax + 1u);
      if (open && kr >= h) t += (unsigned __int128)times * binom_at(binom, cols, drop + x, kr - h);
    }
  }
  if (lane == 0) cmp[0] = 1u + (cmp[kPairPrefix + 32u] >> 4);
  __syncwarp();
  return t;
}

// Register budgets: orientation fits 64 registers without spills (four
// 256-thread CTAs per SM). Pivoting is held to 80 (three): local counts fit them,
// the walk for one k spills (384 bytes stored, 640 loaded), the walk for several
// a little (52 and 88). Two CTAs without spills: a batch 29.0 to 31.1 ms, Chung-Lu
// 1M no faster.
// MK: several k in one walk (pivoting, one graph). GATHER: out-lists, a batch's
// bit rows, or either. Listing has a kernel for each: with the code of both in
// one, its traversal was slower (k = 5, partition 32: Chung-Lu 1M 217 ms, 192 ms
// so; R-MAT 16 73 and 68). The walk for one k has one kernel for both, which
// compiles to the faster walk (R-MAT 17, k = 5, node units: 10.0 ms, 10.9 ms
// with a kernel for each; the batch 13.0 ms either way).
enum Gather { kLists, kBitRows, kEither };

template <int MODE, bool LOCAL, bool MK, Gather GATHER>
__global__ void __launch_bounds__(256, MODE == 0 ? 4 : 3) k_count_bitmap(CountParams p) {
  extern __shared__ __align__(16) uint32_t smem[];
  const uint32_t G = p.G;
  const uint32_t gpb = blockDim.x / G;
  const uint32_t gib = threadIdx.x / G;
  const uint32_t gt = threadIdx.x - gib * G;
  const uint32_t lane = lane_id();
  const uint32_t wig = gt >> 5, nwg = G >> 5;
  Part pt;
  pt.P = p.P;
  pt.plane = gt % p.P;
  pt.pbase = (lane / p.P) * p.P;
  pt.pmask = p.P >= 32 ? 0xffffffffu : (((1u << p.P) - 1u) << pt.pbase);
  const uint32_t part = gt / p.P;
  // Several k in one walk (MK, p.nk of them): the walk goes to
  // the largest k, and lane `plane` of every partition keeps the count of
  // kset[plane]. A clique-tree node with `hold` held vertices, `drop` pivots
  // and candidate set C adds sum_j C(drop, j) cliques(G[C], k - hold - j);
  // for a given k that sum is closed once k - hold <= 2, so k is taken
  // (closed) at the first node on a path where k - hold <= 2, and the node
  // below a non-pivot step from a parent with k - hold = 3 is where k - hold
  // first reaches 2. A k that is still open at a leaf (no candidates) adds
  // C(drop, k - hold) there.
  constexpr bool mk = MK;
  const bool kon = mk && pt.plane < p.nk;
  const uint32_t kl = kon ? p.kset[pt.plane] : 0u;

  uint32_t* sb = smem + (size_t)gib * p.group_words;
  uint32_t* gb = p.gbuf ? p.gbuf + (size_t)(blockIdx.x * gpb + gib) * p.gbuf_words : nullptr;
  uint32_t* hdr = sb;
  uint32_t* S = sb + 16;
  uint32_t* B = p.bitmap_global ? gb : sb + p.off_B;
  uint32_t* R0 = sb + p.off_R0;
  uint32_t* frames = (p.frames_global ? gb + p.goff_fr : sb + p.off_fr) + (size_t)part * p.pstride;
  uint32_t* cand = frames + p.off_cand;  // pivoting: the candidates of the node being entered
  // pivoting: the compact bitmap of a node counted whole (then its prefix table)
  const bool compact = MODE == 1 && !LOCAL && p.compact != 0u;
  uint32_t* cmp = cand + ((p.dcap + 3u) & ~3u);
  // open-addressing hash of S: vertex -> local index (linear probing, load <= 1/2)
  const uint32_t hT = p.hash_T;
  uint32_t* hkey = sb + p.off_H;
  uint16_t* hval = reinterpret_cast<uint16_t*>(hkey + hT);

  // class bounds come from device memory: clamp them so no unit index can leave the queue
  const uint32_t ubeg = min(p.bounds[2 * p.cls], p.n_units_max);
  const uint32_t ucnt = min(p.bounds[2 * p.cls + 1], (p.n_units_max - ubeg + p.qstride - 1) / p.qstride);
  unsigned __int128 acc = 0;
  uint32_t acc_graph = 0xffffffffu;
  unsigned long long st_nodes = 0, st_words = 0, st_bytes = 0;
  // With statistics, each group leader times its units' phases with the SM
  // clock: [0] forming S and its hash, [1] gathering the induced subgraph,
  // [2] traversing. Sums go to a per-block shared array, then to global.
  __shared__ unsigned long long blk_cy[3];
  const bool timing = p.stats != nullptr && gt == 0;
  if (p.stats != nullptr) {
    if (threadIdx.x < 3) blk_cy[threadIdx.x] = 0ull;
    __syncthreads();
  }
  uint32_t tc = 0;
  auto clk32 = []() -> uint32_t {
    uint32_t t;
    asm volatile("mov.u32 %0, %%clock;" : "=r"(t));
    return t;
  };
  auto lap = [&](int phase) {
    if (timing) {
      const uint32_t t = clk32();
      atomicAdd(&blk_cy[phase], (unsigned long long)(t - tc));  // a phase over 2^32 cycles (~2 s) wraps
      tc = t;
    }
  };

  auto gsync = [&]() {
    if (G == 32) __syncwarp(); else __syncthreads();
  };
  auto flush = [&]() {
    if (mk) {
      if (kon && acc != 0 && acc_graph != 0xffffffffu)
        atomic_add_u128(p.out + 2ull * ((size_t)acc_graph * p.nk + pt.plane), acc);
    } else if (pt.plane == 0 && acc != 0 && acc_graph != 0xffffffffu) {
      atomic_add_u128(p.out + 2ull * acc_graph, acc);
    }
    acc = 0;
  };

  // Work budget: a unit whose traversal exceeds p.budget nodes stops, drops
  // its partial count and is appended to the heavy list, which a CTA-wide
  // pass counts afterwards. Nodes are charged to hdr[4] in steps of 64 and
  // hdr[5] flags the stop; each partition (pivoting: its lanes' sum) keeps the
  // unit's count in uacc until the unit is known to have finished.
  const bool budgeted = p.budget != 0;
  unsigned __int128 uacc = 0;
  uint32_t since_charge = 0;
  auto over_budget = [&]() -> bool {  // partition-uniform
    uint32_t stop = 0;
    if (pt.plane == 0) {
      stop = *(volatile uint32_t*)&hdr[5];
      if (!stop && ++since_charge >= 64) {
        const uint32_t add = since_charge;
        since_charge = 0;
        if (atomicAdd(&hdr[4], add) + add > p.budget) {
          hdr[5] = 1u;
          stop = 1u;
        }
      }
    }
    return __shfl_sync(pt.pmask, stop, pt.pbase) != 0u;
  };

  // Local (per-vertex) counts, orientation mode: every vertex of S keeps a
  // u64 counter in shared memory for the unit, the unit's own vertices (u,
  // and v for an edge unit) get the unit's total; both are added to the
  // global (lo, hi) counters when the unit commits.
  unsigned long long* loc = reinterpret_cast<unsigned long long*>(smem + (size_t)gib * p.group_words + p.off_loc);
  auto local_add_bits = [&](uint32_t w, uint32_t x) {  // +1 for every vertex of word w of a set
    for (; x; x &= x - 1u) atomicAdd(&loc[w * 32u + (uint32_t)__ffs(x) - 1u], 1ull);
  };
  // pivoting keeps a (lo, hi) pair per vertex of S (counts of large cliques pass 2^64)
  auto loc2_add = [&](uint32_t i, unsigned __int128 v) { atomic_add_u128(loc + 2ull * i, v); };

  // Tail helping: once the queue is empty, a CTA joins a unit that another
  // CTA is still walking. Every walker of a unit (its owner's partitions and
  // the helpers') walks the clique tree above the cut the same way and takes
  // the nodes at the cut by a global ticket; only the owner's partition 0
  // adds what lies above the cut. A walker that has been through all of the
  // unit's cut nodes holds a ticket past the last one, so every cut node is
  // taken: it sets bit 31 of the ticket, and no helper joins after that.
  const bool help = MODE == 1 && !LOCAL && p.help_ticket != nullptr;
  // In the heavy pass, which starts with more CTAs than units, a CTA without a
  // unit would look before the owners have a unit to show: an owner announces
  // itself before it takes its ticket, and whoever finds only announcements
  // looks again (kHelpPolls times at most, then it leaves).
  const bool announce = help && p.class_exit == nullptr;
  bool drained = false;
  const bool pairs = GATHER == kEither ? p.bits.words != nullptr : GATHER == kBitRows;  // out-lists are bit rows
  for (;;) {
    if (gt == 0) {
      if (announce && !drained) {
        *(volatile uint32_t*)&p.help_active[blockIdx.x] = kHelpSetUp;
        __threadfence();
      }
      uint32_t tk = atomicAdd(p.ticket, 1u);
      if (tk < ucnt && past_limit(p.time_limit_ns, p.t0)) {  // out of time: take no more units
        set_error(p.err, DEV_ERR_TIMEOUT);
        tk = 0xffffffffu;
      }
      // (no unit: the announcement comes down, or the idle CTAs would look on for it)
      if (announce && !drained && tk >= ucnt) *(volatile uint32_t*)&p.help_active[blockIdx.x] = 0u;
      hdr[0] = tk;
      hdr[1] = 0;  // subtree ticket of this unit
      hdr[4] = 0;  // nodes charged to this unit
      hdr[5] = 0;  // unit over budget
      hdr[6] = 0;  // helping: 1 + the queue position of the unit joined
    }
    gsync();
    const uint32_t ui = hdr[0];
    size_t pos = ubeg + (size_t)ui * p.qstride;
    bool helper = false;
    if (ui >= ucnt) {
      if (!help || ui == 0xffffffffu) break;
      drained = true;
      // A CTA of a class launch helps only once the plan's other class
      // launches have finished (all their CTAs exited): while they run, its
      // slot serves them better than a share of another CTA's unit. The
      // heavy pass runs alone and always helps.
      if (p.class_exit != nullptr) {
        uint32_t busy = 0;
        if (gt == 0)
          for (int c = 0; c < kNumClasses; ++c)
            if (c != (int)p.cls && p.class_grid[c] != 0u &&
                *(volatile const uint32_t*)&p.class_exit[c] < p.class_grid[c])
              busy = 1;
        if (gt == 0) hdr[7] = busy;
        gsync();
        if (hdr[7]) break;
      }
      if (wig == 0) {  // the first warp looks for a unit still being walked
        const uint32_t nb = gridDim.x;
        uint32_t pick = 0;
        for (uint32_t poll = 0; poll < kHelpPolls; ++poll) {
          uint32_t soon = 0;
          for (uint32_t i0 = 0; i0 < nb && pick == 0u; i0 += 32u) {
            uint32_t c = 0;
            if (i0 + lane < nb) {
              const uint32_t b = (blockIdx.x + 1u + i0 + lane) % nb;
              const uint32_t a = *(volatile const uint32_t*)&p.help_active[b];
              if (a == kHelpSetUp) soon = 1u;
              else if (a != 0u && !(*(volatile const uint32_t*)&p.help_ticket[a - 1u] & 0x80000000u)) c = a;
            }
            const uint32_t m = __ballot_sync(0xffffffffu, c != 0u);
            if (m) pick = __shfl_sync(0xffffffffu, c, __ffs(m) - 1);
          }
          if (pick != 0u || !announce || !__any_sync(0xffffffffu, soon)) break;
          __nanosleep(500);
        }
        if (lane == 0) hdr[6] = pick;
      }
      gsync();
      const uint32_t a = hdr[6];
      if (a == 0u) break;
      helper = true;
      pos = a - 1u;
    }
    if (timing) tc = clk32();
    const uint32_t unit = p.queue[pos];
    uacc = 0;
    since_charge = 0;
    uint32_t src, d;
    if (!p.edge_units) {
      src = unit;
      const uint32_t b = p.rp[src];
      d = p.rp[src + 1] - b;
      if (d <= p.dcap && !pairs)
        for (uint32_t j = gt; j < d; j += G) S[j] = p.col[b + j];
    } else {
      src = p.erow[unit];
      const uint32_t v = p.col[unit];
      if (wig == 0) {
        // S = N+(u) ∩ N+(v): stream the shorter list, search the longer
        const uint32_t ub = p.rp[src], ue = p.rp[src + 1], vb = p.rp[v], ve = p.rp[v + 1];
        const uint32_t *A, *L;
        uint32_t la, ll;
        if (ue - ub <= ve - vb) { A = p.col + ub; la = ue - ub; L = p.col + vb; ll = ve - vb; }
        else { A = p.col + vb; la = ve - vb; L = p.col + ub; ll = ue - ub; }
        uint32_t cnt = 0;
        for (uint32_t i0 = 0; i0 < la; i0 += 32) {
          const uint32_t i = i0 + lane;
          bool found = false;
          uint32_t x = 0;
          if (i < la) {
            x = A[i];
            const uint32_t pos = lower_bound_u32(L, ll, x);
            found = pos < ll && L[pos] == x;
          }
          const uint32_t bal = __ballot_sync(0xffffffffu, found);
          if (found && cnt + __popc(bal & lanemask_lt()) < p.dcap) S[cnt + __popc(bal & lanemask_lt())] = x;
          cnt += __popc(bal);
        }
        if (lane == 0) hdr[2] = cnt;
        st_bytes += 4ull * (la + la * 8ull);
      }
      gsync();
      d = hdr[2];
    }
    const uint32_t gph = p.vgraph ? p.vgraph[src] : 0u;
    const uint32_t k = p.gk ? p.gk[gph] : p.k0;
    gsync();
    if (gph != acc_graph) {
      flush();
      acc_graph = gph;
    }
    if (d > p.dcap) {
      if (gt == 0) set_error(p.err, DEV_ERR_CAPACITY);
      gsync();
      continue;
    }
    // row stride in words: the unit's own width, or the launch's fixed 1/2/4
    // words when rows are read with one vector load by the lane traversal
    const uint32_t W = p.lane_dfs ? p.W : (d + 31u) >> 5;
    const bool sym = MODE == 1;
    // pivoting reads 32 rows at once (one candidate per lane): an odd row
    // stride puts them in distinct shared-memory banks
    const uint32_t Ws = sym ? (W | 1u) : W;

    if (MODE == 0) {
      const uint32_t t = p.edge_units ? k - 2u : k - 1u;
      if (t <= 1u || d < t) {
        if (part == 0 && d >= t) acc += (t == 0u) ? 1u : d;
        if (LOCAL && d >= t && d <= p.dcap) {
          if (t == 1u)
            for (uint32_t i = gt; i < d; i += G) atomic_add_u128(p.local + 2ull * S[i], 1u);
          if (gt == 0) {
            const unsigned long long tot = (t == 0u) ? 1ull : d;
            atomic_add_u128(p.local + 2ull * src, tot);
            if (p.edge_units) atomic_add_u128(p.local + 2ull * p.col[unit], tot);
          }
        }
        gsync();
        continue;
      }
    } else if (mk) {
      // several k: every k with k - hold0 <= 1 is closed at the unit (the
      // unit is the clique, or one more vertex of S); the others need G[S]
      const uint32_t hold0 = p.edge_units ? 2u : 1u;
      // (into uacc: a unit that outruns its budget drops it with its walk,
      // and the heavy pass counts the whole unit again)
      const uint32_t r0 = kl - hold0;  // (wraps for kl < hold0: no contribution)
      if (part == 0 && !helper && kon && r0 <= 1u) uacc += (r0 == 0u) ? 1u : d;
      if (d == 0u || k < hold0 + 2u || hold0 + d < max(p.kset[0], hold0 + 2u)) {
        acc += uacc;
        gsync();
        continue;
      }
    } else {
      // k - hold0 <= 1: the unit's count is 1 (the unit is the clique) or d
      const uint32_t hold0 = p.edge_units ? 2u : 1u;
      if (d == 0u || hold0 + d < k || k <= hold0 + 1u) {
        if (part == 0 && !helper && k >= hold0 && hold0 + d >= k) acc += (k == hold0) ? 1u : d;
        if (LOCAL && k >= hold0 && hold0 + d >= k && d <= p.dcap) {
          if (k == hold0 + 1u)
            for (uint32_t i = gt; i < d; i += G) atomic_add_u128(p.local + 2ull * S[i], 1u);
          if (gt == 0) {
            const unsigned long long tot = (k == hold0) ? 1ull : d;
            atomic_add_u128(p.local + 2ull * src, tot);
            if (p.edge_units) atomic_add_u128(p.local + 2ull * p.col[unit], tot);
          }
        }
        gsync();
        continue;
      }
    }

    // ---- induced subgraph on S as a bitmap (row j, bit i: S[i] in N+(S[j]))
    for (uint32_t i = gt; i < d * Ws; i += G) B[i] = 0u;
    if (LOCAL)
      for (uint32_t i = gt; i < (MODE == 0 ? d : 2u * d); i += G) loc[i] = 0ull;
    const uint32_t hshift = hT ? 33u - (uint32_t)__ffs(hT) : 0u;  // 32 - log2(hT)
    // An S that spans at most kSpanWords * 32 rank labels (every graph of up to
    // 8,192 vertices) has a member map of that span: bit x - S[0] is set for
    // every x of S, and mpre[w] counts the members in the words below w, so
    // x's local index is mpre[w] + popc(map[w] & bits below x). A wider S has a
    // hash behind a filter: almost every gathered word is not in S, and the
    // filter (one bit per hash value, at most 3% of them set) turns those away
    // with one read, where a probe of the half-full hash takes two to five.
    const uint32_t s0 = pairs ? 0u : S[0], last = pairs ? 0u : S[d - 1];
    const bool wmap = !pairs && hT != 0u && last - s0 < kSpanWords * 32u;
    uint32_t* map = hkey;
    uint32_t* mpre = hkey + kSpanWords;
    const uint32_t fw = filter_words(G);
    const uint32_t fshift = G == 32u ? 19u : 17u;  // 32 - log2(32 fw)
    uint32_t* filter = hkey + hT + hT / 2u;
    uint32_t* rbase = hkey + gather_rows_at(hT, G);
    uint32_t* rlen = rbase + p.dcap;
    if (hT && !pairs) {
      const uint32_t nmw = ((last - s0) >> 5) + 1u;
      if (wmap) {
        for (uint32_t w = gt; w < nmw; w += G) map[w] = 0u;
      } else {
        for (uint32_t i = gt; i < hT; i += G) hkey[i] = 0xffffffffu;
        for (uint32_t i = gt; i < fw; i += G) filter[i] = 0u;
      }
      for (uint32_t j = gt; j < d; j += G) {
        const uint32_t x = S[j], b = p.rp[x];
        rbase[j] = b;
        rlen[j] = p.rp[x + 1] - b;
      }
      gsync();
      for (uint32_t i = gt; i < d; i += G) {
        const uint32_t x = S[i];
        if (wmap) {
          const uint32_t o = x - s0;
          if (KC_IN_BOUNDS(o >> 5, kSpanWords, p.err)) atomicOr(&map[o >> 5], 1u << (o & 31u));
        } else {
          const uint32_t hx = x * 0x9e3779b1u;
          atomicOr(&filter[hx >> (fshift + 5u)], 1u << ((hx >> fshift) & 31u));
          uint32_t h = hx >> hshift;
          while (atomicCAS(&hkey[h], 0xffffffffu, x) != 0xffffffffu) h = (h + 1u) & (hT - 1u);
          hval[h] = (uint16_t)i;
        }
      }
      if (wmap) {
        gsync();
        if (wig == 0) {
          uint32_t carry = 0;
          for (uint32_t w0 = 0; w0 < nmw; w0 += 32u) {
            const uint32_t w = w0 + lane;
            const uint32_t c = w < nmw ? (uint32_t)__popc(map[w]) : 0u;
            uint32_t incl = c;
#pragma unroll
            for (uint32_t o = 1; o < 32u; o <<= 1) {
              const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
              if (lane >= o) incl += y;
            }
            if (w < nmw) mpre[w] = carry + incl - c;
            carry += __shfl_sync(0xffffffffu, incl, 31);
          }
        }
      }
    }
    // Bit rows: the member map is the unit's own row, from its first word on,
    // and S the labels of its bits (local to the graph).
    uint32_t rw = 0, first = 0;
    const uint32_t* rows = nullptr;
    if (pairs) {
      const uint32_t v0 = p.bits.voff[gph];
      rw = bit_row_words(p.bits.voff[gph + 1] - v0);
      rows = p.bits.words + p.bits.off[gph];
      first = bit_row_first(unit - v0);
      if (wig == 0) {
        const uint32_t* own = rows + (size_t)(unit - v0) * rw;
        uint32_t carry = 0;
        for (uint32_t w0 = first; w0 < rw; w0 += 128u) {
          const uint32_t w = w0 + lane * 4u;
          uint4 x = make_uint4(0u, 0u, 0u, 0u);
          if (w < rw) x = __ldg(reinterpret_cast<const uint4*>(own + w));
          const uint32_t c0 = __popc(x.x), c1 = __popc(x.y), c2 = __popc(x.z), c = c0 + c1 + c2 + __popc(x.w);
          uint32_t incl = c;
#pragma unroll
          for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
          }
          uint32_t at = carry + incl - c;
          if (w < rw && KC_IN_BOUNDS(w - first + 3u, kSpanWords, p.err)) {
            *reinterpret_cast<uint4*>(map + (w - first)) = x;
            *reinterpret_cast<uint4*>(mpre + (w - first)) = make_uint4(at, at + c0, at + c0 + c1, at + c0 + c1 + c2);
          }
#pragma unroll
          for (uint32_t q = 0; q < 4; ++q)
            for (uint32_t y = q == 0 ? x.x : q == 1 ? x.y : q == 2 ? x.z : x.w; y; y &= y - 1u)
              if (KC_IN_BOUNDS(at, d, p.err)) S[at++] = (w + q) * 32u + (uint32_t)__ffs(y) - 1u;
          carry += __shfl_sync(0xffffffffu, incl, 31);
        }
      }
    }
    gsync();
    lap(0);
    if (pairs) {
      // kRowLanes lanes take a row of a member, from the member's own word on
      // (an out-list lies above it), 16 bytes per lane and step, and AND it
      // with the member map: 128 labels in six instructions, where a list costs
      // a test per entry, nine in ten of them not in S. Only common labels pay
      // for their local index and the bitmap's atomic. Batch of 2,500 mixed
      // graphs: counting 17.6 ms from lists, 15.4 ms from bit rows. (Testing all
      // pairs of S in rows by vertex id took 18.5 ms: a load per pair, each of a
      // sector of its own.)
      const uint32_t sub = lane / kRowLanes, ll = lane % kRowLanes;
      for (uint32_t j0 = wig * (32u / kRowLanes); j0 < d; j0 += nwg * (32u / kRowLanes)) {
        const uint32_t j = j0 + sub;
        const uint32_t r = j < d ? S[j] : 0u;
        const uint32_t* row = rows + (size_t)r * rw;
        const uint32_t wb = j < d ? bit_row_first(r) : rw;
        if (p.stats) st_bytes += 4ull * __reduce_add_sync(0xffffffffu, ll == 0u && j < d ? rw - wb + 1u : 0u);
        for (uint32_t w0 = __reduce_min_sync(0xffffffffu, wb); w0 < rw; w0 += 4u * kRowLanes * 2u) {
          // (two steps of loads in flight)
          uint4 x[2];
#pragma unroll
          for (uint32_t q = 0; q < 2; ++q) {
            const uint32_t w = w0 + (q * kRowLanes + ll) * 4u;
            x[q] = make_uint4(0u, 0u, 0u, 0u);
            if (w >= wb && w < rw) x[q] = __ldg(reinterpret_cast<const uint4*>(row + w));
          }
#pragma unroll
          for (uint32_t q = 0; q < 2; ++q) {
            const uint32_t w = w0 + (q * kRowLanes + ll) * 4u;
            if (w >= wb && w < rw) {
              const uint4 m = *reinterpret_cast<const uint4*>(map + (w - first));
              x[q].x &= m.x; x[q].y &= m.y; x[q].z &= m.z; x[q].w &= m.w;
              while (x[q].x | x[q].y | x[q].z | x[q].w) {
                uint32_t y, k4;
                if (x[q].x) { y = x[q].x; k4 = 0u; x[q].x &= y - 1u; }
                else if (x[q].y) { y = x[q].y; k4 = 1u; x[q].y &= y - 1u; }
                else if (x[q].z) { y = x[q].z; k4 = 2u; x[q].z &= y - 1u; }
                else { y = x[q].w; k4 = 3u; x[q].w &= y - 1u; }
                const uint32_t mi = w - first + k4;
                const uint32_t lo = mpre[mi] + (uint32_t)__popc(map[mi] & ((y & (0u - y)) - 1u));
                if (KC_IN_BOUNDS(j * Ws + (lo >> 5), d * Ws, p.err)) atomicOr(&B[j * Ws + (lo >> 5)], 1u << (lo & 31u));
                if (sym && KC_IN_BOUNDS(lo * Ws + (j >> 5), d * Ws, p.err))
                  atomicOr(&B[lo * Ws + (j >> 5)], 1u << (j & 31u));
              }
            }
          }
        }
      }
    } else if (hT) {
      // The out-lists of S's rows: kRowLanes lanes read a row, so a warp has
      // four rows in hand, and every lane tests U words of its row per step
      // (8, or 4 when no row of the four is longer than 32). What a step costs
      // is issue, so the test is one table read per word, and only the words
      // found to be members, one or two of a lane's U, pay for the local index
      // and the bitmap's atomic. Before, a lane's words were eight consecutive
      // ones of all rows joined, with a search for the row of every word: about
      // 47 lane instructions a word. Batch of 2,500 mixed graphs (3.5e9 words):
      // counting 26.8 ms before, 21.0 ms now; its gather's share of the unit
      // groups' cycles fell from 8.8e10 to 6.0e10.
      const uint32_t sub = lane / kRowLanes, ll = lane % kRowLanes, span = last - s0;
      auto step = [&](auto ucount, const uint32_t* row, uint32_t len, uint32_t off, uint32_t j) {
        constexpr uint32_t U = decltype(ucount)::value;
        uint32_t xs[U], hit = 0;
#pragma unroll
        for (uint32_t q = 0; q < U; ++q) {
          const uint32_t i = off + q * kRowLanes + ll;
          xs[q] = i < len ? __ldg(row + i) : 0xffffffffu;
        }
        if (wmap) {
#pragma unroll
          for (uint32_t q = 0; q < U; ++q) {
            const uint32_t o = xs[q] - s0;
            if (o <= span) hit |= ((map[o >> 5] >> (o & 31u)) & 1u) << q;
          }
        } else {
#pragma unroll
          for (uint32_t q = 0; q < U; ++q) {
            const uint32_t hx = xs[q] * 0x9e3779b1u;
            if (xs[q] <= last) hit |= ((filter[hx >> (fshift + 5u)] >> ((hx >> fshift) & 31u)) & 1u) << q;
          }
        }
        for (; hit; hit &= hit - 1u) {
          const uint32_t x = __ldg(row + off + ((uint32_t)__ffs(hit) - 1u) * kRowLanes + ll);
          uint32_t lo = 0xffffffffu;
          if (wmap) {
            const uint32_t o = x - s0;
            lo = mpre[o >> 5] + (uint32_t)__popc(map[o >> 5] & ((1u << (o & 31u)) - 1u));
          } else {
            uint32_t h = (x * 0x9e3779b1u) >> hshift;
            for (uint32_t hk; (hk = hkey[h]) != 0xffffffffu; h = (h + 1u) & (hT - 1u))
              if (hk == x) {
                lo = hval[h];
                break;
              }
            if (lo == 0xffffffffu) continue;
          }
          if (KC_IN_BOUNDS(j * Ws + (lo >> 5), d * Ws, p.err)) atomicOr(&B[j * Ws + (lo >> 5)], 1u << (lo & 31u));
          if (sym && KC_IN_BOUNDS(lo * Ws + (j >> 5), d * Ws, p.err))
            atomicOr(&B[lo * Ws + (j >> 5)], 1u << (j & 31u));
        }
      };
      for (uint32_t j0 = wig * (32u / kRowLanes); j0 < d; j0 += nwg * (32u / kRowLanes)) {
        const uint32_t j = j0 + sub;
        const uint32_t len = j < d ? rlen[j] : 0u;
        const uint32_t* row = p.col + (j < d ? rbase[j] : 0u);
        const uint32_t most = __reduce_max_sync(0xffffffffu, len);
        if (p.stats) st_bytes += 4ull * __reduce_add_sync(0xffffffffu, ll == 0u && j < d ? len + 1u : 0u);
        if (most <= 4u * kRowLanes) {
          step(std::integral_constant<uint32_t, 4>{}, row, len, 0u, j);
        } else {
          for (uint32_t off = 0; off < most; off += 8u * kRowLanes)
            step(std::integral_constant<uint32_t, 8>{}, row, len, off, j);
        }
      }
    } else {
      for (uint32_t j = wig; j < d; j += nwg) {
        const uint32_t x0 = S[j];
        const uint32_t b = p.rp[x0], e = p.rp[x0 + 1];
        for (uint32_t i0 = b; i0 < e; i0 += 32) {
          const uint32_t i = i0 + lane;
          const uint32_t x = i < e ? __ldg(p.col + i) : 0xffffffffu;
          const bool inr = x <= last;
          if (!__any_sync(0xffffffffu, inr)) break;
          if (inr) {
            const uint32_t lo = j + 1u + lower_bound_u32(S + j + 1u, d - j - 1u, x);
            if (lo < d && S[lo] == x && KC_IN_BOUNDS(lo, d, p.err)) {
              atomicOr(&B[j * Ws + (lo >> 5)], 1u << (lo & 31u));
              if (sym) atomicOr(&B[lo * Ws + (j >> 5)], 1u << (j & 31u));
            }
          }
        }
        st_bytes += 4ull * (e - b + 1u);  // the row and its vertex of S (warp-uniform)
      }
    }
    gsync();
    lap(1);

    if (mk) {
      // several k: the k with k - hold0 = 2 is the number of edges of G[S]
      const uint32_t hold0 = p.edge_units ? 2u : 1u;
      if (part == 0 && !helper) {
        unsigned long long e2 = 0;  // twice the edges: the bitmap is symmetric
        for (uint32_t j = pt.plane; j < d; j += pt.P)
          for (uint32_t w = 0; w < W; ++w) e2 += __popc(B[j * Ws + w]);
        for (uint32_t o = 1; o < pt.P; o <<= 1) e2 += __shfl_xor_sync(pt.pmask, e2, o);
        if (kon && kl == hold0 + 2u) uacc += e2 / 2u;
      }
      if (k <= hold0 + 2u) {
        acc += uacc;
        gsync();
        continue;
      }
    } else if (MODE == 1 && k == (p.edge_units ? 4u : 3u)) {
      // k - hold0 = 2: the unit's count is the number of edges of G[S]; a
      // vertex of S is in as many of those cliques as it has neighbours in S
      if (part == 0 && !helper) {
        unsigned long long e2 = 0;  // twice the edges: the bitmap is symmetric
        for (uint32_t j = pt.plane; j < d; j += pt.P) {
          uint32_t dj = 0;
          for (uint32_t w = 0; w < W; ++w) dj += __popc(B[j * Ws + w]);
          e2 += dj;
          if (LOCAL && dj) atomic_add_u128(p.local + 2ull * S[j], dj);
        }
        for (uint32_t o = 1; o < pt.P; o <<= 1) e2 += __shfl_xor_sync(pt.pmask, e2, o);
        acc += e2 / 2u;
        if (LOCAL && pt.plane == 0 && e2) {
          atomic_add_u128(p.local + 2ull * src, e2 / 2u);
          if (p.edge_units) atomic_add_u128(p.local + 2ull * p.col[unit], e2 / 2u);
        }
      }
      gsync();
      continue;
    }

    if (MODE == 0 && p.lane_dfs) {
      // ---- orientation traversal, one lane per subtree
      const uint32_t t = p.edge_units ? k - 2u : k - 1u;
      const uint32_t bud = budgeted ? p.budget : 0u;
      // for t >= 4, the exclusive prefix of the row popcounts, in the hash
      // region (free once the bitmap is built; 2 hT >= 8 dcap words)
      const uint32_t* pre = nullptr;
      if (hT != 0u && t >= 4u) {
        uint32_t carry = 0;
        for (uint32_t j0 = 0; j0 < d; j0 += 32u) {
          const uint32_t j = j0 + lane;
          uint32_t c = 0;
          if (j < d)
            for (uint32_t q = 0; q < W; ++q) c += __popc(B[j * W + q]);
          uint32_t incl = c;
          for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
          }
          if (j < d) hkey[j] = carry + incl - c;
          carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) hkey[d] = carry;
        __syncwarp();
        pre = hkey;
      }
      if (W == 1u) lane_dfs<1>(B, d, t, pre, hdr, bud, uacc, st_nodes, st_words KC_ERR_ARG(p.err));
      else if (W == 2u) lane_dfs<2>(B, d, t, pre, hdr, bud, uacc, st_nodes, st_words KC_ERR_ARG(p.err));
      else lane_dfs<4>(B, d, t, pre, hdr, bud, uacc, st_nodes, st_words KC_ERR_ARG(p.err));
    } else if (MODE == 0) {
      // ---- orientation traversal
      const uint32_t t = p.edge_units ? k - 2u : k - 1u;
      for (;;) {
        if (budgeted && over_budget()) break;
        uint32_t j = 0;
        if (pt.plane == 0) j = atomicAdd(&hdr[1], 1u);
        j = __shfl_sync(pt.pmask, j, pt.pbase);
        if (j >= d) break;
        uint32_t* F0 = frames;
        const uint32_t ws = j >> 5;
        uint32_t c = 0;
        for (uint32_t w = ws + pt.plane; w < W; w += pt.P) {
          const uint32_t x = B[j * W + w];
          F0[w] = x;
          c += __popc(x);
        }
        c = __reduce_add_sync(pt.pmask, c);
        st_nodes++;
        st_words += W - ws;
        if (t == 2u) {
          uacc += c;
          if (LOCAL) {  // the edges (j, x), x in row j
            if (pt.plane == 0 && c) atomicAdd(&loc[j], (unsigned long long)c);
            for (uint32_t w = ws + pt.plane; w < W; w += pt.P) local_add_bits(w, F0[w]);
          }
          continue;
        }
        if (c < t - 1u) continue;
        if (pt.plane == 0) {
          F0[W] = ws;
          if (LOCAL) { F0[W + 1] = j; F0[W + 2] = F0[W + 3] = 0u; }
        }
        __syncwarp(pt.pmask);
        int lv = 0;
        while (lv >= 0) {
          if (budgeted && over_budget()) break;
          uint32_t* F = frames + (size_t)lv * p.fw;
          uint32_t wi = 0;
          const int vb = part_next_bit(F, F[W], W, pt, &wi);
          if (vb < 0) {
            if (LOCAL && pt.plane == 0) {
              // the frame's subtree total belongs to its vertex and to every ancestor
              const unsigned long long tot = ((unsigned long long)F[W + 3] << 32) | F[W + 2];
              if (tot) {
                atomicAdd(&loc[F[W + 1]], tot);
                if (lv > 0) {
                  uint32_t* Fp = F - p.fw;
                  const unsigned long long pt2 = (((unsigned long long)Fp[W + 3] << 32) | Fp[W + 2]) + tot;
                  Fp[W + 2] = (uint32_t)pt2;
                  Fp[W + 3] = (uint32_t)(pt2 >> 32);
                }
              }
            }
            __syncwarp(pt.pmask);
            --lv;
            continue;
          }
          const uint32_t v = (uint32_t)vb;
          __syncwarp(pt.pmask);
          if (pt.plane == 0) { F[wi] &= ~(1u << (v & 31u)); F[W] = wi; }
          __syncwarp(pt.pmask);
          const uint32_t rem = t - (uint32_t)(lv + 2);
          uint32_t* Fc = F + p.fw;
          const bool store = rem > 1u && (uint32_t)(lv + 1) < p.depth;
          uint32_t cc = 0;
          for (uint32_t w = wi + pt.plane; w < W; w += pt.P) {
            const uint32_t x = F[w] & B[v * W + w];
            if (store) Fc[w] = x;
            cc += __popc(x);
          }
          cc = __reduce_add_sync(pt.pmask, cc);
          st_nodes++;
          st_words += W - wi;
          if (rem == 1u) {
            uacc += cc;
            if (LOCAL && cc) {
              // the cliques path + v + x: v gets cc now, the path's frames
              // their totals on the way up, each x of the child one
              for (uint32_t w = wi + pt.plane; w < W; w += pt.P) local_add_bits(w, F[w] & B[v * W + w]);
              if (pt.plane == 0) {
                atomicAdd(&loc[v], (unsigned long long)cc);
                const unsigned long long t2 = (((unsigned long long)F[W + 3] << 32) | F[W + 2]) + cc;
                F[W + 2] = (uint32_t)t2;
                F[W + 3] = (uint32_t)(t2 >> 32);
              }
              __syncwarp(pt.pmask);
            }
          } else if (cc >= rem) {
            if (!store) {
              if (pt.plane == 0) set_error(p.err, DEV_ERR_STACK);
            } else {
              if (pt.plane == 0) {
                Fc[W] = wi;
                if (LOCAL) { Fc[W + 1] = v; Fc[W + 2] = Fc[W + 3] = 0u; }
              }
              __syncwarp(pt.pmask);
              ++lv;
            }
          }
        }
      }
    } else if (MODE == 1 && compact && (d <= kSmallMax || (!mk && d <= kWideMax && k == (p.edge_units ? 5u : 4u))) &&
               (mk ? multi_r(k - (p.edge_units ? 2u : 1u), d) <= kSmallMaxRMulti : k <= kSmallMaxR)) {
      // ---- a unit counted whole (edge roots: their sum is the unit's count)
      const uint32_t r = k - (p.edge_units ? 2u : 1u);  // >= 3 here
      if (part == 0 && !helper) {
        st_nodes++;
        for (uint32_t i = pt.plane; i < d; i += 32u) cand[i] = i;
        __syncwarp();
        if constexpr (MK)  // the k with k - hold0 <= 2 are closed already
          uacc += close_node_multi(B, Ws, nullptr, d, cmp, multi_r(r, d), 0u, p.binom, p.binom_cols, kl - (k - r),
                                   kon && kl + r >= k + 3u KC_ERR_ARG(p.err));
        else
          uacc += close_node(B, Ws, r > 3u && d <= kSmallMax ? nullptr : cand, d, cmp, r, 0u, p.binom,
                             p.binom_cols KC_ERR_ARG(p.err));
        st_words += 32u * cmp[0];
      }
    } else {
      // ---- pivot traversal (succinct clique tree)
      // Root: a pivot p0 of G[S] and its branches R0 = S \ N(p0). With edge
      // roots the root has no pivot: every v in S is a branch, the edge
      // (u, S[v]) whose subproblem is N+(u) ∩ N+(S[v]), the bits above v of
      // row v.
      const uint32_t hold0 = p.edge_units ? 2u : 1u;
      if (p.edge_roots) {
        if (gt == 0) hdr[3] = 0xffffffffu;
        for (uint32_t w = gt; w < W; w += G) R0[w] = valid_mask(d, w);
      } else {
        uint32_t key = 0;
        for (uint32_t v = gt; v < d; v += G) {
          uint32_t c = 0;
          for (uint32_t w = 0; w < W; ++w) c += __popc(B[v * Ws + w]);
          key = max(key, (c << 16) | (0xffffu - v));
        }
        key = __reduce_max_sync(0xffffffffu, key);
        if (lane == 0) hdr[8 + wig] = key;
        gsync();
        if (gt == 0) {
          uint32_t m = 0;
          for (uint32_t q = 0; q < nwg; ++q) m = max(m, hdr[8 + q]);
          hdr[3] = 0xffffu - (m & 0xffffu);
        }
        gsync();
        const uint32_t q0 = hdr[3];
        for (uint32_t w = gt; w < W; w += G) R0[w] = ~B[q0 * Ws + w] & valid_mask(d, w);
      }
      gsync();
      const uint32_t p0 = hdr[3];

      auto binom = [&](uint32_t nn, uint32_t r) -> unsigned __int128 {
        if (r > nn) return 0;
        const unsigned long long* e = p.binom + 2ull * ((size_t)nn * (p.binom_cols + 1u) + r);
        return ((unsigned __int128)e[1] << 64) | e[0];
      };
      // Work split inside the unit: the clique tree (root at depth 0) is cut
      // at depth L and the nodes at depth L go out by ticket (hdr[1]) to the
      // group's partitions. Every partition walks the levels above the cut
      // itself, re-deriving the same pivots, so no frame crosses partitions;
      // partition 0 alone adds what the nodes above the cut contribute.
      // L grows when the root has few branches (dense units, whose pivot
      // neighbours nearly everything).
      // The cut is sized for the CTA's own partitions (helpers take what is
      // left of it): a deeper cut would make every walker, helpers included,
      // walk more levels above it, and on bushy trees that costs more than
      // the finer split gains.
      const uint32_t nparts = G / pt.P;
      uint32_t nr0 = 0;
      for (uint32_t w = pt.plane; w < W; w += pt.P) nr0 += __popc(R0[w]);
      nr0 = __reduce_add_sync(pt.pmask, nr0);
      const uint32_t L = (nparts == 1u || nr0 >= 4u * nparts) ? 1u : (nr0 <= 2u ? 3u : 2u);
      const bool top_owner = part == 0u && !helper;
      uint32_t* cut_ticket = help ? p.help_ticket + pos : &hdr[1];
      if (help && !helper && gt == 0) {  // the unit can take helpers from now on
        __threadfence();
        *(volatile uint32_t*)&p.help_active[blockIdx.x] = (uint32_t)pos + 1u;
      }
      auto ticket = [&]() -> uint32_t {
        uint32_t t = 0;
        if (pt.plane == 0) t = atomicAdd(cut_ticket, 1u);
        return __shfl_sync(pt.pmask, t, pt.pbase);
      };
      uint32_t seen = 0, mine = ticket();
      auto claim = [&]() -> bool {  // at a depth-L node: does this partition take it?
        const bool take = seen == mine;
        ++seen;
        if (take) mine = ticket();
        return take;
      };

      // A clique-tree node with `hold` held vertices, `drop` pivots and the
      // candidate set F[0, W) contributes sum_j C(drop, j) * cliques(G[F], r - j)
      // with r = k - hold. For r <= 2 that sum is closed (cliques of size 0,
      // 1, 2 are 1, |F| and the edges of G[F]), so the subtree is not walked.
      // Otherwise the node's pivot and branch set are stored and it is pushed.
      // Frame: F [0, W), branches R [W, 2W), then hold, drop, pivot, cursor.
      // The pivot's branch goes last and reuses its parent's slot (nothing of
      // the parent is needed after it), so only non-pivot branches, which
      // each hold one more vertex, deepen the stack: at most k - hold0 + 1
      // levels, whatever the length of the drop chains.
      // With a full-warp walker and rows of at most 32 words (every launch
      // but the one for units above 1024 vertices) lane w holds word w of a
      // candidate set, and a ballot gives the words that hold candidates:
      // the listing and the scoring below visit only those.
      const bool narrow = pt.P == 32u && W <= 32u;
      const bool lc = LOCAL;  // local (per-vertex) counts
      unsigned __int128 leaf_cnt = 0, leaf_pinc = 0;
      // pchild: the node is its parent's pivot branch (same held vertices);
      // otherwise it holds one vertex more than its parent
      // above: a node above the cut, which every walker of the unit enters; a
      // node counted whole there goes to the walker that holds its ticket
      auto enter = [&](uint32_t* F, uint32_t hold, uint32_t drop, bool own, bool pchild, bool above) -> bool {
        uint32_t nc = 0, nzm = 0;
        if (narrow) {
          const uint32_t x = pt.plane < W ? F[pt.plane] : 0u;
          nc = __reduce_add_sync(pt.pmask, (uint32_t)__popc(x));
          nzm = __ballot_sync(pt.pmask, x != 0u);
        } else {
          for (uint32_t w = pt.plane; w < W; w += pt.P) nc += __popc(F[w]);
          nc = __reduce_add_sync(pt.pmask, nc);
        }
        const uint32_t r = k - hold;  // callers keep hold <= k
        // a node that ends here leaves (for local counts) leaf_cnt, its
        // cliques (each holds the node's held vertices), and leaf_pinc, the
        // cliques that hold any one of its pivots
        leaf_cnt = 0;
        leaf_pinc = 0;
        // several k: this lane's k is still open here if its k - hold was
        // at least 3 at the parent
        // the walker's own adds: every lane its k, else (one k) lane 0 alone, as
        // nodes counted whole add each lane's share
        const bool adds = mk || LOCAL || pt.plane == 0u;
        bool kopen = kon && kl + (pchild ? 0u : 1u) >= hold + 3u;
        if (nc == 0u) {
          leaf_cnt = binom(drop, r);
          if (r >= 1u && drop >= 1u) leaf_pinc = binom(drop - 1u, r - 1u);
          if (own && adds) uacc += mk ? (kopen ? binom(drop, kl - hold) : (unsigned __int128)0u) : leaf_cnt;
          return false;
        }
        if (hold + drop + nc < (mk ? p.kset[0] : k)) return false;
        if (r <= 1u) {  // (never with several k: an open k has k - hold >= 2 here)
          leaf_cnt = (r == 0u) ? (unsigned __int128)1u : (unsigned __int128)(nc + drop);
          leaf_pinc = (r == 1u && drop >= 1u) ? 1u : 0u;
          if (own && adds && !mk) uacc += leaf_cnt;
          if (lc && own && r == 1u)  // each candidate c completes one clique
            for (uint32_t w = pt.plane; w < W; w += pt.P)
              for (uint32_t x = F[w]; x; x &= x - 1u) loc2_add(w * 32u + (uint32_t)__ffs(x) - 1u, 1u);
          return false;
        }
        // a small node is counted whole: the walker that owns it copies G[F]
        // and counts it (see close_node)
        auto small = [&](uint32_t n) {
          return compact && r >= 3u && n <= (!mk && r == 3u ? kWideMax : kSmallMax) &&
                 (mk ? multi_r(r, n) <= kSmallMaxRMulti : r <= kSmallMaxR);
        };
        bool whole = small(nc);
        if (whole && !(above ? claim() : own)) return false;
        uint32_t best = 0, nw = 0;
        unsigned long long esum = 0;
      relist:
        // the candidates are listed in order first (one pass over the words,
        // a bit per lane)
        if (narrow) {
          uint32_t base = 0;
          for (uint32_t m = nzm; m; m &= m - 1u) {
            const uint32_t q = (uint32_t)__ffs(m) - 1u;
            const uint32_t x = F[q];
            const uint32_t ci = base + __popc(x & ((1u << pt.plane) - 1u));
            if (((x >> pt.plane) & 1u) && KC_IN_BOUNDS(ci, p.dcap, p.err)) cand[ci] = q * 32u + pt.plane;
            base += __popc(x);
          }
        } else {
          uint32_t base = 0;
          for (uint32_t q = 0; q < W; ++q) {
            const uint32_t x = F[q];
            if (x == 0u) continue;
            for (uint32_t b = pt.plane; b < 32u; b += pt.P)
              if (((x >> b) & 1u) && KC_IN_BOUNDS(base + __popc(x & ((1u << b) - 1u)), p.dcap, p.err))
                cand[base + __popc(x & ((1u << b) - 1u))] = q * 32u + b;
            base += __popc(x);
          }
        }
        __syncwarp(pt.pmask);
        nw = narrow ? (uint32_t)__popc(nzm) : W;
        if (whole) {
          if constexpr (MK)
            uacc += close_node_multi(B, Ws, cand, nc, cmp, multi_r(r, nc), drop, p.binom, p.binom_cols, kl - hold,
                                     kopen KC_ERR_ARG(p.err));
          else
            uacc += close_node(B, Ws, cand, nc, cmp, r, drop, p.binom, p.binom_cols KC_ERR_ARG(p.err));
          const uint32_t cost = cmp[0];
          since_charge += cost;
          st_words += 32u * cost;
          return false;
        }
        // score every candidate u by |F ∩ N(u)|; the lanes take the listed
        // candidates in turn, so each lane scores ceil(nc / P) of them.
        // Q lanes score one candidate, each over every Q-th word: as many as
        // leave no lane idle (one per candidate once there are 32 of them),
        // at most the launch's partition size
        uint32_t Q = 1u;
        while ((Q << 1) * nc <= pt.P && Q < nw) Q <<= 1;
        if (p.Q != 0u && Q > p.Q) Q = p.Q;
        const uint32_t qs = (uint32_t)__ffs(Q) - 1u;  // Q is a power of two
        const uint32_t ng = pt.P >> qs, gq = pt.plane >> qs, lq = pt.plane & (Q - 1u);
        // Universal candidates (adjacent to every other one): their branch
        // sets are empty, so all of them become pivots in this one step.
        const bool univ = !LOCAL && nc <= 32u * ng;  // (a bit of `um` per candidate of this lane)
        uint32_t um = 0, ub = 1u;
        for (uint32_t i0 = 0; i0 < nc; i0 += ng, ub <<= 1) {
          const uint32_t i = i0 + gq;
          uint32_t c = 0, u = 0;
          if (i < nc) {
            u = cand[i];
            const uint32_t* Bu = B + u * Ws;
            if (narrow) {
              uint32_t j = 0;
              for (uint32_t m = nzm; m; m &= m - 1u, ++j)
                if ((j & (Q - 1u)) == lq) {
                  const uint32_t q = (uint32_t)__ffs(m) - 1u;
                  c += __popc(F[q] & Bu[q]);
                }
            } else {
              for (uint32_t q = lq; q < W; q += Q) c += __popc(F[q] & Bu[q]);
            }
          }
          for (uint32_t o = 1; o < Q; o <<= 1) c += __shfl_xor_sync(pt.pmask, c, o);
          if (i < nc && lq == 0u) {
            esum += c;
            if (univ && c + 1u == nc) um |= ub;
            else best = max(best, (c << 16) | (0xffffu - u));
            // r = 2: candidate u is in a clique with each neighbour in F and each pivot
            if (lc && own && r == 2u && c + drop) loc2_add(u, c + drop);
          }
        }
        if (own) st_words += (unsigned long long)nc * nw / pt.P;
        for (uint32_t o = 1; o < pt.P; o <<= 1) esum += __shfl_xor_sync(pt.pmask, esum, o);
        if (r == 2u) {  // edges of G[F] + drop * |F| + C(drop, 2)
          leaf_cnt = (unsigned __int128)(esum / 2u) + (unsigned __int128)drop * nc + binom(drop, 2u);
          leaf_pinc = drop >= 1u ? (unsigned __int128)(nc + drop - 1u) : 0u;
          if (own && adds) uacc += mk ? ((kopen && kl == hold + 2u) ? leaf_cnt : (unsigned __int128)0u) : leaf_cnt;
          return false;
        }
        // several k: a smaller k that reaches k - hold = 2 here is closed here
        if (mk && kopen && kl == hold + 2u) {
          if (own) uacc += (unsigned __int128)(esum / 2u) + (unsigned __int128)drop * nc + binom(drop, 2u);
          kopen = false;
        }
        // no clique of G[F] has more vertices than the best score + 1 (one k: a
        // node whose cliques and pivots together cannot reach k counts nothing)
        if (!mk && !LOCAL) {
          const uint32_t top = um != 0u ? nc - 1u : best >> 16;
          if (__reduce_max_sync(pt.pmask, top) + 1u + drop < r) return false;
        }
        if (univ && __any_sync(pt.pmask, um != 0u)) {
          const uint32_t nu = __reduce_add_sync(pt.pmask, (uint32_t)__popc(um));
          for (uint32_t x = um; x; x &= x - 1u) {
            const uint32_t u = cand[((uint32_t)__ffs(x) - 1u) * ng + gq];
            atomicAnd(&F[u >> 5], ~(1u << (u & 31u)));
          }
          __syncwarp(pt.pmask);
          drop += nu;
          nc -= nu;
          if (nc == 0u) {  // F was a clique: a leaf with all of it as pivots
            leaf_cnt = binom(drop, r);
            if (own && adds) uacc += mk ? (kopen ? binom(drop, kl - hold) : (unsigned __int128)0u) : leaf_cnt;
            return false;
          }
          if (narrow) nzm = __ballot_sync(pt.pmask, pt.plane < W && F[pt.plane] != 0u);
          if (small(nc)) {  // what is left is small
            whole = true;
            if (!(above ? claim() : own)) return false;
            goto relist;
          }
        }
        best = __reduce_max_sync(pt.pmask, best);
        const uint32_t piv = 0xffffu - (best & 0xffffu);
        // branch set: candidates outside N(piv), less the pivot itself, whose
        // branch is taken last in this frame's own slot
        for (uint32_t w = pt.plane; w < W; w += pt.P) {
          uint32_t rw = F[w] & ~B[piv * Ws + w];
          if (w == (piv >> 5)) rw &= ~(1u << (piv & 31u));
          F[W + w] = rw;
        }
        __syncwarp(pt.pmask);
        if (pt.plane == 0) {
          F[2 * W] = hold;
          F[2 * W + 1] = drop;
          F[2 * W + 2] = piv;
          F[2 * W + 3] = 0;
        }
        __syncwarp(pt.pmask);
        return true;
      };

      // Local counts: a frame also keeps its held vertex (the branch that
      // pushed it; none for the root pivot's branch), where its pivots start
      // in the walker's drop list, and the totals of the cliques ended below
      // it: T_H (each holds the frame's held vertices) and T_P (cliques that
      // hold any one of the frame's pivots). A pivot joins the list with
      // minus the T_P reached so far and gets the final T_P when its frame
      // pops; totals then move up to the parent frame.
      uint32_t* dl = cand + ((p.dcap + 3u) & ~3u);
      uint32_t ndl = 0;
      auto fr_get = [&](const uint32_t* F, uint32_t off) -> unsigned __int128 {
        const uint32_t* q = F + 2u * W + off;
        return ((unsigned __int128)q[3] << 96) | ((unsigned __int128)q[2] << 64) |
               ((unsigned __int128)q[1] << 32) | q[0];
      };
      auto fr_set = [&](uint32_t* F, uint32_t off, unsigned __int128 v) {
        uint32_t* q = F + 2u * W + off;
        q[0] = (uint32_t)v;
        q[1] = (uint32_t)(v >> 32);
        q[2] = (uint32_t)(v >> 64);
        q[3] = (uint32_t)(v >> 96);
      };
      auto fr_open = [&](uint32_t* F, uint32_t held) {  // plane 0
        F[2 * W + 4] = held;
        F[2 * W + 5] = ndl;
        fr_set(F, 6, 0);
        fr_set(F, 10, 0);
      };
      auto fr_take = [&](uint32_t* F) {  // a node that ended in this frame's slot (plane 0)
        fr_set(F, 6, fr_get(F, 6) + leaf_cnt);
        fr_set(F, 10, fr_get(F, 10) + leaf_pinc);
      };
      auto fr_close = [&](uint32_t* F, int level) {  // the frame pops (plane 0)
        const unsigned __int128 th = fr_get(F, 6), tp = fr_get(F, 10);
        const uint32_t hv = F[2 * W + 4], st = F[2 * W + 5];
        if (hv != 0xffffffffu && th) loc2_add(hv, th);
        if (tp)
          for (uint32_t i = st; i < ndl; ++i) loc2_add(dl[i], tp);
        if (level > 0) {
          uint32_t* Fp = F - p.fw;
          fr_set(Fp, 6, fr_get(Fp, 6) + th);
          fr_set(Fp, 10, fr_get(Fp, 10) + tp);
        }
      };

      // One loop and one call site of `enter` (its code is large, and three
      // copies of it kept the warps waiting for instructions, the top stall of
      // dense units): a step forms the candidate set of the next node (a root
      // branch, a branch of the top frame, or the top frame's pivot branch in
      // that frame's own slot), enters it, and pushes or drops its frame.
      enum Step { kRoot, kBranch, kPivot };
      const bool direct = L == 1u && narrow;
      uint32_t r0cnt = 0, r0incl = 0;  // lane w: branches in R0[w], and in R0[0, w]
      if (direct) {
        r0cnt = pt.plane < W ? (uint32_t)__popc(R0[pt.plane]) : 0u;
        r0incl = r0cnt;
        for (uint32_t o = 1; o < 32u; o <<= 1) {
          const uint32_t y = __shfl_up_sync(pt.pmask, r0incl, o);
          if (pt.plane >= o) r0incl += y;
        }
      }
      int lv = -1;  // top frame
      uint32_t v = 0;  // root branches below v are done
      for (;;) {
        if (budgeted && over_budget()) break;
        Step step;
        uint32_t* F;
        uint32_t hold, drop, held;  // held: the vertex that the node's branch holds
        bool own, above;
        if (lv < 0) {
          // the next root branch: with the cut at depth 1 and a bitmap row in a
          // warp's lanes, a ticket is a branch number and its branch is found
          // by the branches' prefix (stepping over the others' branches, 140 of
          // them in a sparse unit, took a third of the walk); else in order
          if (direct) {
            const uint32_t t = mine;
            if (t >= nr0) break;
            mine = ticket();
            const uint32_t w = (uint32_t)__popc(__ballot_sync(pt.pmask, r0incl <= t));
            const uint32_t before = __shfl_sync(pt.pmask, r0incl - r0cnt, w);
            held = w * 32u + select_bit(R0[w], t - before);
          } else {
            while (v < d) {
              const uint32_t x = R0[v >> 5] >> (v & 31u);
              if (x) {
                v += (uint32_t)__ffs(x) - 1u;
                break;
              }
              v = (v | 31u) + 1u;
            }
            if (v >= d) break;
            held = v++;
            if (L == 1u && !claim()) continue;
          }
          step = kRoot;
          own = L == 1u || top_owner;
          above = L > 1u;
          hold = hold0 + (held != p0 ? 1u : 0u);
          drop = (held == p0) ? 1u : 0u;
          if (own) st_nodes++;
          if (hold > k) continue;
          F = frames;
          for (uint32_t w = pt.plane; w < W; w += pt.P) F[w] = B[held * Ws + w] & ~(R0[w] & low_mask(held, w));
          __syncwarp(pt.pmask);
        } else {
          F = frames + (size_t)lv * p.fw;
          uint32_t wi = 0;
          const int vb = part_next_bit(F + W, F[2 * W + 3], W, pt, &wi);
          hold = F[2 * W];
          drop = F[2 * W + 1];
          held = F[2 * W + 2];
          if (vb < 0) {
            // every other branch is done: the pivot's branch replaces the frame
            step = kPivot;
            own = (uint32_t)lv + 1u >= L || top_owner;
            above = (uint32_t)lv + 1u < L;
            if (own) st_nodes++;
            __syncwarp(pt.pmask);
            if (lc) {  // the pivot joins this frame's pivots
              if (pt.plane == 0) {
                dl[ndl] = held;
                const unsigned __int128 tp = fr_get(F, 10);
                if (tp) loc2_add(held, (unsigned __int128)0 - tp);
              }
              ++ndl;
            }
            ++drop;
            for (uint32_t w = pt.plane; w < W; w += pt.P) F[w] &= B[held * Ws + w];
            __syncwarp(pt.pmask);
          } else {
            step = kBranch;
            held = (uint32_t)vb;
            __syncwarp(pt.pmask);
            if (pt.plane == 0) {
              F[W + wi] &= ~(1u << (held & 31u));
              F[2 * W + 3] = wi;
            }
            ++hold;  // the branch is not the pivot's
            bool descend = hold <= k;
            if (descend && (uint32_t)(lv + 1) >= p.depth) {
              if (pt.plane == 0) set_error(p.err, DEV_ERR_STACK);
              descend = false;
            }
            own = (uint32_t)lv + 2u > L || top_owner;
            above = (uint32_t)lv + 2u < L;
            if (descend && (uint32_t)lv + 2u == L) own = descend = claim();
            if (own) st_nodes++;
            uint32_t* Fc = F + p.fw;
            if (descend)
              for (uint32_t w = pt.plane; w < W; w += pt.P) Fc[w] = F[w] & B[held * Ws + w];
            __syncwarp(pt.pmask);
            if (pt.plane == 0) F[held >> 5] &= ~(1u << (held & 31u));  // later siblings exclude it
            __syncwarp(pt.pmask);
            if (!descend) continue;
            F = Fc;
          }
        }
        const bool pushed = enter(F, hold, drop, own, step == kRoot ? held == p0 : step == kPivot, above);
        if (!lc) {
          if (step == kPivot) lv -= pushed ? 0 : 1;
          else lv += pushed ? 1 : 0;
        } else if (step == kRoot) {
          if (pushed) {
            if (pt.plane == 0) {
              ndl = 0;
              fr_open(F, held != p0 ? held : 0xffffffffu);
              if (held == p0) dl[0] = p0;  // the root pivot is a pivot of this whole subtree
            }
            ndl = (held == p0) ? 1u : 0u;
            lv = 0;
          } else if (own && pt.plane == 0) {
            const unsigned __int128 x = (held != p0) ? leaf_cnt : leaf_pinc;
            if (x) loc2_add(held, x);
          }
          __syncwarp(pt.pmask);
        } else if (step == kPivot) {
          if (!pushed) {
            if (pt.plane == 0) {
              if (own) fr_take(F);
              fr_close(F, lv);
            }
            __syncwarp(pt.pmask);
            ndl = F[2 * W + 5];
            __syncwarp(pt.pmask);
            --lv;
          }
        } else {
          if (pushed) {
            if (pt.plane == 0) fr_open(F, held);
            ++lv;
          } else if (own && pt.plane == 0) {
            // the child ended at once: it holds its cliques, the parent's frame takes them too
            if (leaf_cnt) loc2_add(held, leaf_cnt);
            fr_take(F - p.fw);
          }
          __syncwarp(pt.pmask);
        }
      }
      // this walker has been through every cut node: all of them are taken
      if (help && pt.plane == 0) atomicOr(cut_ticket, 0x80000000u);
    }
    gsync();
    lap(2);
    if (help && !helper && gt == 0) *(volatile uint32_t*)&p.help_active[blockIdx.x] = 0u;
    // commit the unit, or hand it to the heavy pass when it ran over budget
    if (budgeted && hdr[5]) {
      if (gt == 0) p.heavy[atomicAdd(p.heavy_count, 1u)] = unit;
    } else {
      if (MODE == 1 && !LOCAL && !MK && __any_sync(pt.pmask, uacc != 0)) {  // the lanes' shares, summed in every lane
        for (uint32_t o = 1; o < pt.P; o <<= 1) {
          const unsigned long long lo = __shfl_xor_sync(pt.pmask, (unsigned long long)uacc, o);
          const unsigned long long hi = __shfl_xor_sync(pt.pmask, (unsigned long long)(uacc >> 64), o);
          uacc += ((unsigned __int128)hi << 64) | lo;
        }
      }
      acc += uacc;
      if (LOCAL) {
        // the unit's total (its own vertices are in every one of its cliques)
        // in hdr[8..11], free once the root pivot is known
        unsigned long long* ut = reinterpret_cast<unsigned long long*>(&hdr[8]);
        if (gt == 0) ut[0] = ut[1] = 0ull;
        gsync();
        if (pt.plane == 0 && uacc != 0) atomic_add_u128(ut, uacc);
        gsync();
        for (uint32_t i = gt; i < d; i += G) {
          const unsigned __int128 v = MODE == 0 ? (unsigned __int128)loc[i]
                                                : (((unsigned __int128)loc[2 * i + 1] << 64) | loc[2 * i]);
          if (v) atomic_add_u128(p.local + 2ull * S[i], v);
        }
        if (gt == 0) {
          const unsigned __int128 tot = ((unsigned __int128)ut[1] << 64) | ut[0];
          if (tot) {
            atomic_add_u128(p.local + 2ull * src, tot);
            if (p.edge_units) atomic_add_u128(p.local + 2ull * p.col[unit], tot);
          }
        }
      }
    }
    gsync();
  }
  flush();
  if (p.class_exit != nullptr) {  // this CTA is done: count it out of its class launch
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(&p.class_exit[p.cls], 1u);
    }
  }
  if (p.stats && pt.plane == 0) {
    atomicAdd(p.stats + 0, st_nodes);
    atomicAdd(p.stats + 1, st_words);
  }
  // gather bytes are counted warp-uniformly, once per warp
  if (p.stats && lane == 0 && st_bytes) atomicAdd(p.stats + 2, st_bytes);
  if (p.stats != nullptr) {
    __syncthreads();
    if (threadIdx.x < 3) atomicAdd(p.stats + 3 + threadIdx.x, blk_cy[threadIdx.x]);
  }
}

}  // namespace

kc_status prepare_launch(kc_ctx* ctx, const LaunchPlan& lp, const CountParams& p0, cudaStream_t s,
                         PreparedLaunch* out) {
  if (lp.encoding == KC_ENC_LIST) return prepare_launch_list(ctx, lp, p0, s, out);
  CountParams p = p0;
  uint32_t P = lp.part;
  if (P == 0 || P > 32 || (P & (P - 1)) != 0)
    return fail(KC_ERR_INVALID_ARG, "partition size %u is not one of 1,2,4,8,16,32", P);
  const uint32_t G = lp.G, block = lp.block;
  const uint32_t dcap = std::max<uint32_t>(1, lp.dcap);
  uint32_t W = (dcap + 31) / 32;
  const uint32_t t_max = lp.edge ? (lp.k_max >= 2 ? lp.k_max - 2 : 0) : lp.k_max - 1;
  // Warp units in orientation mode run the lane-per-subtree traversal: one
  // lane is one partition, rows have 1, 2 or 4 words, no frames in shared memory.
  const bool lane = lp.mode == KC_MODE_ORIENT && G == 32 && dcap <= 128 && t_max <= (uint32_t)kLaneStack + 2 &&
                    !lp.local;
  if (lane) {
    P = 1;
    W = W <= 1 ? 1 : (W <= 2 ? 2 : 4);
  }
  // Pivoting walks each clique-tree node with a whole warp (partitions of one
  // warp would walk different nodes one after another); the partition size
  // bounds the number of lanes that score one pivot candidate.
  if (lp.mode != KC_MODE_ORIENT) {
    p.Q = lp.q;
    P = 32;
  }
  const uint32_t nparts = G / P;
  const uint32_t gpb = block / G;
  uint32_t depth, fw;
  if (lp.mode == KC_MODE_ORIENT) {
    depth = std::max<uint32_t>(1, t_max >= 2 ? t_max - 2 : 1);
    fw = lp.local ? W + 4 : W + 1;  // local counts: + the frame's vertex and its subtree total
  } else {
    // a pushed frame holds one more vertex than its parent (pivot branches
    // reuse the parent's slot), so k - hold0 + 1 levels always suffice
    const uint32_t hold0 = lp.edge ? 2u : 1u;
    depth = std::min<uint32_t>(dcap + 2, std::max<uint32_t>(2, lp.k_max + 2 - std::min(lp.k_max, hold0)));
    fw = 2 * W + (lp.local ? 14 : 4);  // local counts: held vertex, drop-list start, two u128 totals
  }
  auto al4 = [](size_t x) { return (x + 3) & ~(size_t)3; };
  const size_t hdr = 16, sS = al4(dcap), sR0 = al4(W);
  const bool pivot = lp.mode != KC_MODE_ORIENT;
  const size_t sB = (size_t)dcap * (pivot ? (W | 1u) : W);  // pivot rows use an odd stride
  // per walker: the frames, then (pivoting) the candidate list and, for local
  // counts, the drop list, else the compact bitmap of a node counted whole
  const bool mk = pivot && p.nk != 0;
  bool compact = pivot && !lp.local;
  // (rows and prefix, then the stack of small nodes; triangles use the same words for wider rows)
  const size_t sCmp = std::max<size_t>(2 * kPairPrefix + 2 * kQueueCap + (mk ? kHistWords : 0), compact_words(dcap));
  const size_t frame_words = al4((size_t)depth * fw);
  auto pstride_of = [&]() {
    return frame_words + (pivot ? al4(dcap) * (lp.local ? 2 : 1) : 0) + (compact ? al4(sCmp) : 0);
  };
  size_t pstride = pstride_of();
  size_t sFr = lane ? 0 : al4((size_t)nparts * pstride);
  const size_t limit_words = ((size_t)ctx->max_smem_optin - kStaticSmemBytes) / 4;
  // hash of S for the bitmap build: hT the power of two >= 2 dcap (load at
  // most 1/2)
  uint32_t hT = 0;
  if (dcap <= 2048) {
    hT = 64;
    while (hT < 2u * dcap) hT <<= 1;
  }
  // the gather's row table (start and length of each row) follows its tables
  const size_t sRow = al4(2 * (size_t)dcap);
  bool bitmap_global = lp.force_global_bitmap;
  bool frames_global = false;
  // The hash is needed only while the bitmap is built and the frames only
  // after it, so in shared memory they share one region.
  // local counts: a u64 (orientation) or a (lo, hi) pair (pivoting) per vertex of S
  const size_t sLoc = lp.local ? al4((pivot ? 4 : 2) * (size_t)dcap) : 0;
  auto group_words = [&]() {
    return hdr + sS + sR0 + (bitmap_global ? 0 : al4(sB)) + sLoc +
           std::max<size_t>(frames_global ? 0 : sFr,
                            // (bit rows need the member map and, after it, the listing's prefix)
                            p.bits.words ? 2 * kSpanWords : !hT ? 0 : gather_rows_at(hT, G) + sRow);
  };
  if (compact && (size_t)gpb * group_words() > limit_words) {  // the frames come before the compact bitmaps
    compact = false;
    pstride = pstride_of();
    sFr = al4((size_t)nparts * pstride);
  }
  if ((size_t)gpb * group_words() > limit_words) frames_global = true;
  if ((size_t)gpb * group_words() > limit_words) bitmap_global = true;
  if ((size_t)gpb * group_words() > limit_words) hT = 0;
  if ((size_t)gpb * group_words() > limit_words)
    return fail(KC_ERR_INVALID_ARG, "unit size %u does not fit the shared-memory plan", dcap);
  p.dcap = dcap;
  p.W = W;
  p.P = P;
  p.G = G;
  p.depth = depth;
  p.fw = fw;
  p.pstride = (uint32_t)pstride;
  p.off_cand = (uint32_t)frame_words;
  p.compact = compact ? 1u : 0u;
  p.group_words = (uint32_t)group_words();
  p.off_R0 = (uint32_t)(hdr + sS);
  p.hash_T = hT;
  p.lane_dfs = lane ? 1u : 0u;
  p.off_B = (uint32_t)(hdr + sS + sR0);
  p.off_loc = (uint32_t)(p.off_B + (bitmap_global ? 0 : al4(sB)));
  p.off_fr = (uint32_t)(p.off_loc + sLoc);
  p.off_H = p.off_fr;
  p.bitmap_global = bitmap_global;
  p.frames_global = frames_global;
  p.gbuf_words = (bitmap_global ? al4(sB) : 0) + (frames_global ? sFr : 0);
  p.goff_fr = bitmap_global ? al4(sB) : 0;
  p.gbuf = nullptr;

  const size_t smem_bytes = (size_t)gpb * p.group_words * 4;
  const bool bits = p.bits.words != nullptr;
  if (bits && (lp.local || mk)) return fail(KC_ERR_INTERNAL, "bit rows are a batch's");
  auto kern = !pivot ? (lp.local ? k_count_bitmap<0, true, false, kLists>
                        : bits   ? k_count_bitmap<0, false, false, kBitRows>
                                 : k_count_bitmap<0, false, false, kLists>)
              : lp.local ? k_count_bitmap<1, true, false, kLists>
              : mk       ? k_count_bitmap<1, false, true, kLists>
                         : k_count_bitmap<1, false, false, kEither>;
  // Several classes launch the same kernel with different shared-memory sizes;
  // the attribute is per function, so it is set to the device maximum, once per
  // context (and the occupancy is looked up once per launch shape).
  // (the kernel's static shared memory counts against the same per-block limit)
  if (ctx->kernel_static_smem.find((const void*)kern) == ctx->kernel_static_smem.end()) {
    cudaFuncAttributes fa;
    KC_CUDA(cudaFuncGetAttributes(&fa, kern));
    if (fa.sharedSizeBytes > kStaticSmemBytes)
      return fail(KC_ERR_INTERNAL, "counting kernel uses %zu bytes of static shared memory, planned for %zu",
                  fa.sharedSizeBytes, kStaticSmemBytes);
    KC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 ctx->max_smem_optin - (int)fa.sharedSizeBytes));
    ctx->kernel_static_smem[(const void*)kern] = (int)fa.sharedSizeBytes;
  }
  int& per_sm = ctx->occupancy[std::make_tuple((const void*)kern, block, smem_bytes)];
  if (per_sm == 0) {
    int found = 0;
    KC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&found, kern, block, smem_bytes));
    per_sm = std::max(1, found);
  }
  uint64_t grid = std::min<uint64_t>((uint64_t)ctx->sms * per_sm, ((uint64_t)p.n_units_max + gpb - 1) / gpb);
  grid = std::max<uint64_t>(1, grid);
  if (p.gbuf_words) {
    // keep the global scratch of the whole grid within 24 GiB
    const uint64_t per_block = (uint64_t)gpb * p.gbuf_words * 4;
    const uint64_t cap = std::max<uint64_t>(1, (24ull << 30) / std::max<uint64_t>(1, per_block));
    grid = std::min(grid, cap);
    KC_CUDA(dmalloc(&out->gbuf, grid * per_block, s));
    p.gbuf = out->gbuf;
  }
  out->p = p;
  out->grid = (uint32_t)grid;
  out->block = block;
  out->smem = smem_bytes;
  out->kernel = (void*)kern;
  out->list = false;
  return KC_OK;
}

kc_status enqueue_launch(const PreparedLaunch& pl, cudaStream_t s) {
  CountParams p = pl.p;
  size_t cap = pl.cap_edges;
  void* args_bitmap[] = {&p};
  void* args_list[] = {&p, &cap};
  KC_CUDA(cudaLaunchKernel(pl.kernel, dim3(pl.grid), dim3(pl.block), pl.list ? args_list : args_bitmap, pl.smem, s));
  return KC_OK;
}

void release_launch(PreparedLaunch& pl, cudaStream_t s) {
  if (pl.gbuf) dfree(pl.gbuf, s);
  pl.gbuf = nullptr;
}

}  // namespace kc
