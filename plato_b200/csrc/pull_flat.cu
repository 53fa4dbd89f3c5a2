// Builds the edge streams of the flat pull (pull_flat.cuh) on the device.
#include <algorithm>
#include <vector>

#include <cub/device/device_scan.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include "graph.cuh"
#include "plato_b200/dualmode.cuh"
#include "pull_flat.cuh"

namespace plato_b200 {
namespace {

// Which edges are hot.  Rows above kFlatRowDeg0 in-edges take part in block 0,
// rows above kFlatRowDeg1 in the further blocks: a segment costs a store and a
// load of its sum, so it has to hold a few edges (RMAT s24, epoch: further
// blocks above 32 / 48 / 64 / 96 / 128 in-edges 562 / 539 / 532 / 537 / 577 us;
// block 0 above 4 / 8 / 16 / 32: 580 / 577 / 583 / 589).  What a block holds is
// counted over the rows that take part.  A further block is used where that is
// kFlatMore edges and one more for each such row: its copies and segments cost
// something too (us an epoch with 1 / 4 / 10 / 16 / 24 blocks, and how many are
// chosen: RMAT s21 84.9 / 72.8 / 74.8 / 76.8 / 83.4, 7; s22 168 / 142 / 134 / 133
// / 138, 11; s23 342 / 290 / 260 / 251 / 251, 16; s24 with 10 / 16 / 20 / 22 / 24
// 537 / 521 / 503 / 497 / 507, 22; s22 with 6 edges a vertex 85.7 / 76.9 / 80.8 /
// 81.1 / 87.3, 5).  There are hot streams where all of them together hold
// kFlatFirst: below, one more launch costs what the gathers save (edges that
// would be hot, epoch without / with them: RMAT s19 6.5M 26.4 / 27.5, s20 with 10
// a vertex 8.3M 36.1 / 37.7, s19 with 20 8.6M 31.6 / 33.1, s21 with 6 8.9M 57.5 /
// 48.1, s20 13.9M 51.0 / 45.3).  A count that took in the rows below the limits gave
// uniform edges with one long row streams that were all but empty: 16M over 1M
// vertices 162 us instead of 80, 64M over 4M 378 instead of 288.
constexpr uint32_t kFlatRowDeg0 = 8;
constexpr uint32_t kFlatRowDeg1 = 64;
// Up to this many edges all epochs run in one launch (k_flat_run).  The line lies
// between graphs with hubs, whose separate kernels gather from a larger L1, and
// graphs without (epoch in one launch / in separate ones: RMAT s16 1.0M edges 9.0
// / 10.0 us, s17 1.9M 12.2 / 12.7, s18 2.0M 13.3 / 12.8, 2.5M 16.4 / 13.3, 3.9M
// 21.5 / 15.6; uniform over 200K rows 2M 14.3 / 15.3, 3M 17.8 / 18.8, 4M 21.0 /
// 22.1, over 500K 3M 23.2 / 22.4).
constexpr uint64_t kFlatRunEdges = 3500000;
// ... and rows: its warps also update every 32-row word (uniform edges, 0.1 a row:
// 4M rows 21.5 / 30.1, 8M 56.8 / 51.7, 16M 118 / 98).
constexpr uint32_t kFlatRunRows = 6000000;
constexpr unsigned long long kFlatFirst = 8500000, kFlatMore = 250000;
// Where the blocks cover all sources, every row can take part in every stream
// and no cold pass is left.  That pays from 1.5 edges a segment, unless block 0
// has most of the gathers, which then come from L1 anyway (without / with it:
// uniform edges over 1M vertices, 16M 80 / 91.5, 24M 108 / 105, 32M 143 / 116, 64M
// 256 / 135; 8M over 300K 38 / 28; RMAT s19 26.2 / 28.1, s20 43.9 / 47.4).
bool flat_all_hot(uint64_t rows, uint64_t edges, uint64_t first_block, uint32_t blocks) {
  return static_cast<uint64_t>(blocks) * kFlatBlock >= rows && 2 * edges >= 3 * rows * blocks &&
         2 * first_block < edges;
}

// Which graphs pull by the degree bins instead (pull_binned.cuh).  A row costs
// a flat plan a segment's store, load and meta, the bins only its offsets; what
// it saves is gathers, and the launch of a kernel a bin (about 6 us each).  One
// epoch, flat / bins, one B200:
//   no row above kShortMax (4) edges, one bin: rings of 10K / 100K / 1M / 4M
//   vertices 4.7 / 4.4, 5.3 / 4.4, 12.0 / 10.1, 35.9 / 29.2 us, grids 5.1 / 4.4,
//   5.7 / 4.9, 14.6 / 10.6, 46 / 32, 4 random in-edges a row 5.3 / 4.4, 6.7 / 6.5,
//   25.5 / 22.6, 95 / 76; up to kFlatClusterSteps words one cluster runs all
//   epochs (5K vertices 3.7-4.4 / 4.4).  With an early exit each of their epochs
//   has its decision in a kernel of its own, and the one-launch epochs are the
//   faster (30 epochs: grids of 90K / 250K / 1M vertices 220 / 318, 263 / 380, 443 /
//   502 us): where there are such, the graph has both plans;
//   rows up to 16 (two bins), uniform: 600K rows with 3.5 edges 19.9 / 20.9, 1M
//   with 1.5 / 2.5 / 3.5 19.3 / 21.0, 26.1 / 23.0, 31.5 / 29.1, 4M with 0.5 / 1 /
//   2.5 35.0 / 37.4, 51.0 / 42.2, 82.0 / 63.9, 8M with 0.1 / 1 51.7 / 45.0, 99 /
//   73, 16M with 2.5 / 3.5 302 / 300, 365 / 491;
//   longer ones too: 2M with 5 66.1 / 69.4, 4M with 5 / 6 121 / 118, 133 / 136, 8M
//   with 5 234 / 221; RMAT s22 with 4.4 29.9 / 92.5 (half of the edges in them).
// With weights the bins' rows above 4 edges fall behind sooner (40 epochs: 1M rows
// with 2.5 / 3.6 edges 1.32 / 1.36, 1.57 / 1.77 ms, 2M with 2.5 2.37 / 2.11, 4M with
// 2.5 / 5 4.24 / 3.85, 5.89 / 7.31).
struct flat_census {
  uint64_t rows, few, some;      // all rows, rows of 1..4 and of 5..16 edges
  uint64_t edges, long_edges;    // all edges, those in rows above 16
  bool weighted;
};
enum class flat_use { always, early_exit, never };
flat_use flat_suits(const flat_census& c, bool run) {
  if (c.some == 0 && c.long_edges == 0)
    return c.rows <= 32ull * kFlatClusterSteps ? flat_use::always : run ? flat_use::early_exit : flat_use::never;
  bool bins;
  if (c.rows > 10000000 && 2 * c.edges > 5 * c.rows)
    bins = false;
  else if (c.long_edges == 0)
    bins = (c.few + c.some >= (c.weighted ? 1500000 : 900000) && c.edges >= 2500000) || c.rows >= 6000000;
  else
    bins = !c.weighted && 20 * c.long_edges <= c.edges && c.edges <= 6 * c.rows && c.few + c.some >= 2500000;
  return bins ? flat_use::never : flat_use::always;
}

// out[0]: one past the last row above kFlatRowDeg1 edges, out[1]: how many there
// are, out[2..4]: few, some and long_edges of the census, out[5]: gathers of the
// sources of block 0 (`uses` by source), out[kFlatSurvey + k]: k_flat_uses.
constexpr uint32_t kFlatSurvey = 6;
__global__ void __launch_bounds__(256) k_flat_survey(const uint64_t* __restrict__ off,
                                                     const uint32_t* __restrict__ uses, uint32_t V,
                                                     unsigned long long* out) {
  __shared__ unsigned long long s_red[32];
  unsigned long long last = 0, n = 0, few = 0, some = 0, longs = 0;
  for (uint64_t v = blockIdx.x * 256ull + threadIdx.x; v < V; v += gridDim.x * 256ull) {
    const uint64_t d = off[v + 1] - off[v];
    if (d > kFlatRowDeg1) {
      last = v + 1;
      ++n;
    }
    few += d > 0 && d <= 4;
    some += d > 4 && d <= 16;
    longs += d > 16 ? d : 0;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
  if ((threadIdx.x & 31) == 0 && last) atomicMax(out, last);
  n = block_sum_u64<256>(n, s_red);
  if (threadIdx.x == 0 && n) atomicAdd(out + 1, n);
  few = block_sum_u64<256>(few, s_red);
  some = block_sum_u64<256>(some, s_red);
  longs = block_sum_u64<256>(longs, s_red);
  if (threadIdx.x == 0) {
    if (few) atomicAdd(out + 2, few);
    if (some) atomicAdd(out + 3, some);
    if (longs) atomicAdd(out + 4, longs);
  }
  n = 0;
  for (uint64_t v = blockIdx.x * 256ull + threadIdx.x; v < min(V, kFlatBlock); v += gridDim.x * 256ull) n += uses[v];
  n = block_sum_u64<256>(n, s_red);
  if (threadIdx.x == 0 && n) atomicAdd(out + 5, n);
}

__device__ __forceinline__ uint64_t flat_lower_bound(const uint32_t* __restrict__ adj, uint64_t lo, uint64_t hi,
                                                     uint32_t bound) {
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (adj[mid] < bound) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// out[k]: edges of block k in the rows that take part in its stream.  A warp
// takes 32 rows; the rows of block 0 alone a lane each, the others one after
// another with a block a lane.
__global__ void __launch_bounds__(256) k_flat_uses(const uint64_t* __restrict__ off, const uint32_t* __restrict__ adj,
                                                   uint32_t V, uint32_t nblocks, unsigned long long* out) {
  static_assert(kFlatMaxBlocks <= 32, "a block a lane");
  const unsigned lane = threadIdx.x & 31;
  const uint64_t nwarps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  unsigned long long first = 0, mine = 0;
  for (uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; w < (V + 31ull) / 32; w += nwarps) {
    const uint64_t v = w * 32 + lane;
    const uint64_t b = v < V ? off[v] : 0, e = v < V ? off[v + 1] : 0;
    const bool all = e - b > kFlatRowDeg1;
    if (!all && e - b > kFlatRowDeg0) first += flat_lower_bound(adj, b, e, kFlatBlock) - b;
    for (unsigned todo = __ballot_sync(0xffffffffu, all); todo; todo &= todo - 1) {
      const int l = __ffs(todo) - 1;
      const uint64_t rb = __shfl_sync(0xffffffffu, b, l), re = __shfl_sync(0xffffffffu, e, l);
      const uint64_t end = lane < nblocks ? flat_lower_bound(adj, rb, re, (lane + 1) * kFlatBlock) : re;
      const uint64_t begin = __shfl_up_sync(0xffffffffu, end, 1);
      if (lane < nblocks) mine += end - (lane ? begin : rb);
    }
  }
  first = warp_sum(first);
  if (lane == 0) mine += first;
  if (lane < nblocks && mine) atomicAdd(out + lane, mine);
}

struct flat_rows {
  const uint64_t* off;
  const uint32_t* adj;
  uint32_t V, nb, rows1;  // rows1: the rows of the middle streams, in whole 32-row words
  uint32_t deg0, deg1;           // kFlatRowDeg0, kFlatRowDeg1, or 0 where no source is cold
  // hot streams that row v takes part in
  __device__ __forceinline__ uint32_t streams(uint32_t v) const {
    const uint64_t d = off[v + 1] - off[v];
    return d > deg1 ? nb : d > deg0 ? min(nb, 1u) : 0u;
  }
  __device__ __forceinline__ uint64_t cell(uint32_t k, uint32_t v) const { return flat_place(k, V, rows1) + v; }
};

// cnt[cell(k, v)] = edges of row v in stream k.
__global__ void k_flat_split(flat_rows f, uint32_t* cnt) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < f.V;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = static_cast<uint32_t>(i);
    uint64_t pos = f.off[v];
    const uint64_t end = f.off[v + 1];
    const uint32_t ns = f.streams(v);
    for (uint32_t k = 0; k < f.nb; ++k) {
      if (k > 0 && v >= f.rows1) break;
      uint64_t lo = pos;
      if (k < ns) lo = flat_lower_bound(f.adj, pos, end, (k + 1) * kFlatBlock);
      cnt[f.cell(k, v)] = static_cast<uint32_t>(lo - pos);
      pos = lo;
    }
    cnt[f.cell(f.nb, v)] = static_cast<uint32_t>(end - pos);
  }
}

struct flat_starts {
  uint64_t edge[kFlatMaxBlocks + 1];  // first edge of each stream (padded numbering)
  uint64_t sum[kFlatMaxBlocks + 1];   // edges of the streams before it (unpadded)
};

// Copies every edge (and its weight) to its stream and flags segment ends.  A
// warp takes a merge tile of the CSC; a lane finds its edge's row in the tile.
__global__ void __launch_bounds__(256) k_flat_fill(flat_rows f, const uint32_t* __restrict__ trow,
                                                   const uint64_t* __restrict__ tedge, uint32_t tiles,
                                                   const uint32_t* __restrict__ cnt,
                                                   const uint64_t* __restrict__ pos, flat_starts st,
                                                   const float* __restrict__ w, uint16_t* hid, uint32_t* cid,
                                                   float* hw, float* cw, uint32_t* hflags, uint32_t* cflags) {
  const unsigned lane = threadIdx.x & 31;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const uint64_t cold0 = st.edge[f.nb];
  for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < tiles; t += nwarps) {
    const uint32_t ra = trow[t], rb = min(trow[t + 1], f.V - 1);
    const uint64_t je = tedge[t + 1];
    for (uint64_t e = tedge[t] + lane; e < je; e += 32) {
      uint32_t lo = ra, hi = rb;  // the last row of the tile that starts at or before e
      while (lo < hi) {
        const uint32_t mid = lo + (hi - lo + 1) / 2;
        if (f.off[mid] <= e) lo = mid; else hi = mid - 1;
      }
      const uint32_t v = lo;
      const uint32_t id = f.adj[e];
      const uint32_t ns = f.streams(v);
      uint32_t k = id / kFlatBlock;
      if (k >= ns) k = f.nb;
      uint32_t before = 0;
      for (uint32_t j = 0; j < min(k, ns); ++j) before += cnt[f.cell(j, v)];
      const size_t at = f.cell(k, v);
      const uint32_t i = static_cast<uint32_t>(e - f.off[v]) - before;
      uint64_t to = st.edge[k] + (pos[at] - st.sum[k]) + i;
      uint32_t* flags = hflags;
      if (k < f.nb) {
        hid[to] = static_cast<uint16_t>(id - k * kFlatBlock);
        if (w) hw[to] = w[e];
      } else {
        to -= cold0;
        flags = cflags;
        cid[to] = id;
        if (w) cw[to] = w[e];
      }
      if (i + 1 == cnt[at]) atomicOr(flags + (to >> 5), 1u << (to & 31));
    }
  }
}

// The stream of place i in arrays by stream and 32-row word.
__device__ __forceinline__ uint32_t flat_stream_of(uint64_t i, uint32_t nb, uint32_t words, uint32_t words1) {
  if (i < words) return 0;
  return words1 ? static_cast<uint32_t>(min(static_cast<uint64_t>(nb), 1 + (i - words) / words1)) : nb;
}

// Rows with a segment, 32 at a time, and the ordinal of the first.
__global__ void k_flat_meta(flat_rows f, const uint32_t* __restrict__ cnt, const uint32_t* __restrict__ ord,
                            uint32_t words, uint64_t total, uint4* meta) {
  const unsigned lane = threadIdx.x & 31;
  const uint32_t words1 = (f.rows1 + 31) / 32;
  const uint64_t nwarps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t i = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; i < total; i += nwarps) {
    const uint32_t k = flat_stream_of(i, f.nb, words, words1);
    const uint32_t w = static_cast<uint32_t>(i - flat_place(k, words, words1));
    const uint32_t v = w * 32 + lane;
    const bool has = v < f.V && cnt[f.cell(k, v)] != 0;
    const unsigned m = __ballot_sync(0xffffffffu, has);
    if (lane == 0) meta[i] = make_uint4(m, ord[f.cell(k, w * 32)], 0u, 0u);
  }
}

struct flat_has {
  __host__ __device__ uint32_t operator()(uint32_t c) const { return c != 0 ? 1u : 0u; }
};

// The marks of each step from its flag bits, and the number of segments that
// end in it; a warp per step, N edges a lane.
template <int N, typename T>
__global__ void k_flat_marks(const uint32_t* __restrict__ flags, uint32_t steps, T* marks, uint32_t* ends) {
  const unsigned lane = threadIdx.x & 31;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < steps; s += nwarps) {
    const uint64_t e = static_cast<uint64_t>(s) * 32 * N + lane * N;
    const uint32_t fl = (flags[e / 32] >> (e % 32)) & ((1u << N) - 1u);
    const uint32_t n = __popc(fl);
    uint32_t c = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t o = __shfl_up_sync(0xffffffffu, c, d);
      if (static_cast<int>(lane) >= d) c += o;
    }
    marks[static_cast<size_t>(s) * 32 + lane] = static_cast<T>((c - n) << N | fl);
    if (lane == 31) ends[s] = c;
  }
}

struct flat_crossing {
  const uint4* meta;
  __device__ uint32_t operator()(uint32_t i) const { return __popc(meta[i].z); }
};

// Piece p continues a segment of an earlier piece; *j is its ordinal.
__device__ __forceinline__ bool flat_continues(const flat_view& f, uint32_t p, uint32_t* j) {
  const uint2 pc = f.pieces[p];
  if ((pc.x & kPieceFirst) || pc.x >= pc.y) return false;
  const size_t before = static_cast<size_t>(pc.x) * 32 - 1;
  if (p < f.cold_piece0) {
    if (f.hmark[before] >> (kFlatHotLane - 1) & 1u) return false;
    *j = f.hseg[pc.x];
  } else {
    if (f.cmark[before] >> (kFlatColdLane - 1) & 1u) return false;
    *j = f.cseg[pc.x];
  }
  return true;
}

// Segments cut by piece boundaries, one thread per piece; the first piece
// that continues a segment records it.  fill = false marks the rows in
// meta.z and finds the last word with a wide span, fill = true writes the spans
// (meta.w scanned in between).
template <bool kFill>
__global__ void k_flat_spans(flat_view f, uint32_t npieces, uint32_t hot_steps, uint32_t cold_steps,
                             uint32_t segments, uint4* meta, uint2* spans, uint32_t* wide_words) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t j = 0;
  if (p >= npieces || !flat_continues(f, p, &j) || j >= segments) return;
  uint32_t q = p - 1;  // the piece before that is not empty
  while (f.pieces[q].x >= f.pieces[q].y && !(f.pieces[q].x & kPieceFirst)) --q;
  uint32_t jq = 0;
  if (flat_continues(f, q, &jq) && jq == j) return;
  // j ends in the last step before which at most j segments have ended, and in
  // the last piece that starts no later: an empty piece starts no later than the
  // next one.  (A hub row crosses thousands of pieces: both by search.)
  const bool hot = p < f.cold_piece0;
  const uint32_t* ended = hot ? f.hseg : f.cseg;
  uint32_t s_end = f.pieces[p].x, s_hi = (hot ? hot_steps : cold_steps) - 1;
  while (s_end < s_hi) {
    const uint32_t mid = s_end + (s_hi - s_end + 1) / 2;
    if (ended[mid] <= j) s_end = mid; else s_hi = mid - 1;
  }
  uint32_t last = p, p_hi = (hot ? f.cold_piece0 : npieces) - 1;
  while (last < p_hi) {
    const uint32_t mid = last + (p_hi - last + 1) / 2;
    if ((f.pieces[mid].x & ~kPieceFirst) <= s_end) last = mid; else p_hi = mid - 1;
  }
  // the row: the last word whose first ordinal is at most j
  const uint64_t total = flat_place(f.nb, f.words, f.words1) + f.words;
  uint64_t lo = 0, hi = total - 1;
  while (lo < hi) {
    const uint64_t mid = lo + (hi - lo + 1) / 2;
    if (f.meta[mid].y <= j) lo = mid; else hi = mid - 1;
  }
  // the bit of the (j - first)-th segment of the word
  uint32_t bits = f.meta[lo].x;
  for (uint32_t n = j - f.meta[lo].y; n > 0; --n) bits &= bits - 1;
  const uint32_t bit = bits & (0u - bits);
  if (!kFill) {
    atomicOr(&meta[lo].z, bit);
    if (last - q > kFlatWideSpan) {
      const uint64_t word = lo - flat_place(flat_stream_of(lo, f.nb, f.words, f.words1), f.words, f.words1);
      atomicMax(wide_words, static_cast<uint32_t>(word) + 1u);
    }
  } else {
    spans[meta[lo].w + __popc(meta[lo].z & (bit - 1u))] = make_uint2(q, last);
  }
}

__global__ void k_flat_span_base(const uint32_t* __restrict__ scan, uint64_t n, uint4* meta) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    meta[i].w = scan[i];
}

// Scratch of a plan's construction, from the engine's stream-ordered pool: no
// cudaMalloc, and no cudaFree that waits for the device.
template <typename T>
struct scratch {
  T* p = nullptr;
  cudaStream_t st;
  explicit scratch(cudaStream_t s) : st(s) {}
  scratch(const scratch&) = delete;
  scratch& operator=(const scratch&) = delete;
  ~scratch() { release(); }
  void release() {
    if (p) cudaFreeAsync(p, st);
    p = nullptr;
  }
  int alloc(cudaMemPool_t pool, size_t n) {
    release();
    const cudaError_t e =
        cudaMallocFromPoolAsync(reinterpret_cast<void**>(&p), std::max<size_t>(n, 1) * sizeof(T), pool, st);
    if (e == cudaSuccess) return PLATO_OK;
    p = nullptr;
    cudaGetLastError();
    return set_error(e == cudaErrorMemoryAllocation ? PLATO_ENOMEM : PLATO_ECUDA,
                     std::string("flat plan: scratch allocation failed: ") + cudaGetErrorString(e));
  }
};

template <class It, typename T>
int scan(It in, T* out, uint64_t n, cudaMemPool_t pool, cudaStream_t st) {
  size_t bytes = 0;
  const auto plus = [] __device__(T a, T b) -> T { return a + b; };  // sums in T, whatever the input's type
  PLATO_CUDA_TRY(cub::DeviceScan::ExclusiveScan(nullptr, bytes, in, out, plus, T(0), static_cast<int64_t>(n), st));
  scratch<uint8_t> tmp(st);
  PLATO_TRY(tmp.alloc(pool, bytes));
  PLATO_CUDA_TRY(cub::DeviceScan::ExclusiveScan(tmp.p, bytes, in, out, plus, T(0), static_cast<int64_t>(n), st));
  count_launch();
  return PLATO_OK;
}

// Lays arrays out one after another, each on a 256-byte boundary.
struct layout {
  size_t bytes = 0;
  size_t add(size_t n) {
    const size_t at = bytes;
    bytes += (n + 255) / 256 * 256;
    return at;
  }
};

template <typename T>
int put(T* d, const std::vector<T>& h, cudaStream_t st) {
  if (!h.empty())
    PLATO_CUDA_TRY(cudaMemcpyAsync(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, st));
  return PLATO_OK;
}

}  // namespace

int build_flat_plan(plato_graph* g, flat_plan& pl, cudaStream_t st) {
  const uint32_t V = g->info.vertices;
  const uint64_t E = g->stored_edges;
  pl.valid = false;
  if (!g->relabeled || !g->own_sources || E == 0) return PLATO_OK;
  const uint64_t* off = g->in_off.p;
  const bool weighted = g->weighted;
  const uint32_t nblocks = std::min<uint32_t>((V + kFlatBlock - 1) / kFlatBlock, kFlatMaxBlocks);
  cudaMemPool_t pool{};
  try {
    pool = engine_pool();
  } catch (const std::exception& e) {
    return set_error(PLATO_ECUDA, e.what());
  }
  scratch<unsigned long long> d_survey(st);
  PLATO_TRY(d_survey.alloc(pool, kFlatSurvey + kFlatMaxBlocks));
  PLATO_CUDA_TRY(cudaMemsetAsync(d_survey.p, 0, (kFlatSurvey + kFlatMaxBlocks) * sizeof(unsigned long long), st));
  k_flat_survey<<<grid_for(V, 256, 148 * 4), 256, 0, st>>>(off, g->out_deg.p, V, d_survey.p);
  PLATO_LAUNCHED("k_flat_survey");
  const bool run = E <= kFlatRunEdges && V <= kFlatRunRows;
  if (!run) {
    k_flat_uses<<<grid_for(V, 256, 148 * 8), 256, 0, st>>>(off, g->in_adj.p, V, nblocks, d_survey.p + kFlatSurvey);
    PLATO_LAUNCHED("k_flat_uses");
  }
  unsigned long long h[kFlatSurvey + kFlatMaxBlocks];
  PLATO_CUDA_TRY(cudaMemcpyAsync(h, d_survey.p, sizeof(h), cudaMemcpyDeviceToHost, st));
  PLATO_CUDA_TRY(cudaStreamSynchronize(st));
  const flat_use use = flat_suits(flat_census{V, h[2], h[3], E, h[4], weighted}, run);
  if (use == flat_use::never) return PLATO_OK;
  pl.early_only = use == flat_use::early_exit;
  flat_rows rows{off, g->in_adj.p, V, 0, 0, kFlatRowDeg0, kFlatRowDeg1};
  uint32_t nb = 0;
  const bool all_hot = !run && flat_all_hot(V, E, h[5], nblocks);
  if (all_hot) {
    nb = nblocks;
    rows.deg0 = rows.deg1 = 0;
  } else if (!run) {
    const unsigned long long* uses = h + kFlatSurvey;
    unsigned long long hot = uses[0];
    for (nb = 1; nb < nblocks && uses[nb] >= kFlatMore + h[1]; ++nb) hot += uses[nb];
    if (hot < kFlatFirst) nb = 0;
  }
  rows.nb = nb;
  // whole words; the last may be short
  rows.rows1 = nb <= 1 ? 0 : all_hot ? V : std::min((static_cast<uint32_t>(h[0]) + 31) / 32 * 32, V);
  const uint32_t streams = nb + 1, words = (V + 31) / 32, words1 = (rows.rows1 + 31) / 32;
  const uint64_t cells = flat_place(nb, V, rows.rows1) + V;

  scratch<uint32_t> cnt(st), ord(st);
  scratch<uint64_t> pos(st);
  PLATO_TRY(cnt.alloc(pool, cells));
  PLATO_TRY(pos.alloc(pool, cells));
  PLATO_TRY(ord.alloc(pool, cells));
  k_flat_split<<<grid_for(V, 256), 256, 0, st>>>(rows, cnt.p);
  PLATO_LAUNCHED("k_flat_split");
  PLATO_TRY(scan(cnt.p, pos.p, cells, pool, st));
  PLATO_TRY(scan(thrust::make_transform_iterator(cnt.p, flat_has()), ord.p, cells, pool, st));
  // edges before each stream, and the last cells for the number of segments
  std::vector<uint64_t> sum(streams + 1, 0);
  uint32_t last_cnt = 0, segments = 0;
  for (uint32_t k = 0; k < streams; ++k)
    PLATO_CUDA_TRY(cudaMemcpyAsync(&sum[k], pos.p + flat_place(k, V, rows.rows1), 8, cudaMemcpyDeviceToHost, st));
  PLATO_CUDA_TRY(cudaMemcpyAsync(&last_cnt, cnt.p + cells - 1, 4, cudaMemcpyDeviceToHost, st));
  PLATO_CUDA_TRY(cudaMemcpyAsync(&segments, ord.p + cells - 1, 4, cudaMemcpyDeviceToHost, st));
  PLATO_CUDA_TRY(cudaStreamSynchronize(st));
  segments += last_cnt != 0;
  sum[streams] = E;
  flat_starts fs{};
  uint64_t edges = 0;
  for (uint32_t k = 0; k < streams; ++k) {
    const uint32_t step = k < nb ? kFlatHotStep : kFlatColdStep;
    fs.edge[k] = edges;
    fs.sum[k] = sum[k];
    edges += (sum[k + 1] - sum[k] + step - 1) / step * step;
  }
  const uint64_t hot_edges = fs.edge[nb], cold_edges = edges - hot_edges;
  const uint32_t hot_steps = static_cast<uint32_t>(hot_edges / kFlatHotStep);
  const uint32_t cold_steps = static_cast<uint32_t>(cold_edges / kFlatColdStep);
  // grids, and bounds on the pieces
  int sms = 0;
  PLATO_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device));
  const uint32_t per_block = kFlatColdThreads / 32;
  pl.hot_ctas = std::min<uint32_t>(sms, (hot_steps + kFlatHotWarps - 1) / kFlatHotWarps);
  pl.run_ctas = pl.run_warps = pl.cold_blocks = 0;
  pl.run_cluster = false;
  if (run) {
    const uint32_t work = std::max(cold_steps, words);  // a warp each, as far as they go
    if (work <= 4) {
      pl.run_ctas = 1;
      pl.run_warps = 4;
    } else if (work <= kFlatClusterSteps) {
      pl.run_cluster = true;
      pl.run_ctas = kFlatCluster;
      pl.run_warps = std::min<uint32_t>(32, std::max<uint32_t>(4, (work + kFlatCluster - 1) / kFlatCluster));
    } else {
      pl.run_ctas = std::min<uint32_t>(sms, (work + 7) / 8);
      pl.run_warps = std::min<uint32_t>(32, (work + pl.run_ctas - 1) / pl.run_ctas);
    }
  } else if (cold_steps) {
    // a wave of resident CTAs, and more (up to about five waves, so that the
    // last one is short) while a warp keeps 8 steps
    const uint32_t wave = sms * kFlatColdCtas, fill = cold_steps / (8 * per_block);
    pl.cold_blocks = std::min<uint32_t>((cold_steps + per_block - 1) / per_block,
                                        std::min<uint32_t>(sms * 24u, std::max(wave, fill)));
  }
  const uint32_t cold_pieces = run ? pl.run_ctas * pl.run_warps : pl.cold_blocks * per_block;
  const uint32_t max_subs = pl.hot_ctas + nb, max_pieces = max_subs * kFlatHotWarps + cold_pieces;
  const uint64_t nmeta = flat_place(nb, words, words1) + words;
  layout lay;
  const size_t o_hid = lay.add(hot_edges * 2ull), o_cid = lay.add(cold_edges * 4ull);
  const size_t o_hw = lay.add(weighted ? hot_edges * 4ull : 0), o_cw = lay.add(weighted ? cold_edges * 4ull : 0);
  const size_t o_hmark = lay.add(hot_steps * 128ull), o_cmark = lay.add(cold_steps * 64ull);
  const size_t o_seg = lay.add((static_cast<uint64_t>(hot_steps) + cold_steps) * 4);
  const size_t o_meta = lay.add(nmeta * sizeof(uint4));
  const size_t o_spans = lay.add(max_pieces * sizeof(uint2)), o_pieces = lay.add(max_pieces * sizeof(uint2));
  const size_t o_subs = lay.add(max_subs * sizeof(flat_sub)), o_cta = lay.add((pl.hot_ctas + 1) * 4ull);
  const size_t o_part = lay.add(segments * sizeof(float)), o_head = lay.add(max_pieces * sizeof(float));
  const size_t o_carry = lay.add(max_pieces * sizeof(float));
  PLATO_TRY(pl.mem.alloc(lay.bytes));
  unsigned char* mem = pl.mem.p;
  uint16_t* hid = reinterpret_cast<uint16_t*>(mem + o_hid);
  uint32_t* cid = reinterpret_cast<uint32_t*>(mem + o_cid);
  float* hw = weighted ? reinterpret_cast<float*>(mem + o_hw) : nullptr;
  float* cw = weighted ? reinterpret_cast<float*>(mem + o_cw) : nullptr;
  uint32_t* hmark = reinterpret_cast<uint32_t*>(mem + o_hmark);
  uint16_t* cmark = reinterpret_cast<uint16_t*>(mem + o_cmark);
  uint32_t* seg = reinterpret_cast<uint32_t*>(mem + o_seg);
  uint4* meta = reinterpret_cast<uint4*>(mem + o_meta);
  uint2* spans = reinterpret_cast<uint2*>(mem + o_spans);
  uint2* d_pieces = reinterpret_cast<uint2*>(mem + o_pieces);
  flat_sub* d_subs = reinterpret_cast<flat_sub*>(mem + o_subs);
  uint32_t* d_cta = reinterpret_cast<uint32_t*>(mem + o_cta);
  scratch<uint32_t> hflags(st), cflags(st);
  PLATO_TRY(hflags.alloc(pool, hot_edges / 32));
  PLATO_TRY(cflags.alloc(pool, cold_edges / 32));
  PLATO_CUDA_TRY(cudaMemsetAsync(hflags.p, 0, hot_edges / 8, st));
  PLATO_CUDA_TRY(cudaMemsetAsync(cflags.p, 0, cold_edges / 8, st));
  // the padding of a stream's last step: source 0, weight 0, no flag
  for (uint32_t k = 0; k < streams; ++k) {
    const uint64_t end = k + 1 < streams ? fs.edge[k + 1] : edges;
    if (end == fs.edge[k]) continue;
    if (k < nb) {
      PLATO_CUDA_TRY(cudaMemsetAsync(hid + (end - kFlatHotStep), 0, kFlatHotStep * 2, st));
      if (weighted) PLATO_CUDA_TRY(cudaMemsetAsync(hw + (end - kFlatHotStep), 0, kFlatHotStep * 4, st));
    } else {
      const uint64_t b = cold_edges - kFlatColdStep;
      PLATO_CUDA_TRY(cudaMemsetAsync(cid + b, 0, kFlatColdStep * 4, st));
      if (weighted) PLATO_CUDA_TRY(cudaMemsetAsync(cw + b, 0, kFlatColdStep * 4, st));
    }
  }
  // merge tiles of the direction's rows and edges, 224 of both a tile
  const uint32_t tiles = static_cast<uint32_t>((V + E + 223) / 224);
  scratch<uint32_t> trow(st);
  scratch<uint64_t> tedge(st);
  PLATO_TRY(trow.alloc(pool, tiles + 1));
  PLATO_TRY(tedge.alloc(pool, tiles + 1));
  PLATO_TRY(merge_tile_starts(off, V, E, 224, tiles, trow.p, tedge.p, st));
  k_flat_fill<<<grid_for(static_cast<uint64_t>(tiles) * 32, 256), 256, 0, st>>>(
      rows, trow.p, tedge.p, tiles, cnt.p, pos.p, fs, weighted ? g->in_w.p : nullptr, hid, cid, hw,
      cw, hflags.p, cflags.p);
  PLATO_LAUNCHED("k_flat_fill");
  // marks, and segments that end before each step (numbered through all streams)
  scratch<uint32_t> ends(st);
  PLATO_TRY(ends.alloc(pool, hot_steps + cold_steps));
  if (hot_steps) {
    k_flat_marks<kFlatHotLane, uint32_t><<<grid_for(hot_steps * 32ull, 256), 256, 0, st>>>(hflags.p, hot_steps,
                                                                                           hmark, ends.p);
    PLATO_LAUNCHED("k_flat_marks");
  }
  if (cold_steps) {
    k_flat_marks<kFlatColdLane, uint16_t><<<grid_for(cold_steps * 32ull, 256), 256, 0, st>>>(
        cflags.p, cold_steps, cmark, ends.p + hot_steps);
    PLATO_LAUNCHED("k_flat_marks");
  }
  PLATO_TRY(scan(ends.p, seg, hot_steps + cold_steps, pool, st));
  k_flat_meta<<<grid_for(nmeta * 32, 256), 256, 0, st>>>(rows, cnt.p, ord.p, words, nmeta, meta);
  PLATO_LAUNCHED("k_flat_meta");

  // Pieces: the hot steps split evenly over one CTA per SM, cut at block
  // ends, each part split over the CTA's warps; the cold steps over all warps
  // of the cold grid.
  // Cost of the hot steps before each one: a step with segment ends costs
  // about half as much again, and every end is a store.  (RMAT s24, k_flat_hot
  // with the steps split evenly 291 us, by this cost 182.)
  const uint32_t all_steps = hot_steps + cold_steps;
  std::vector<uint32_t> h_seg(hot_steps + 1, segments);
  if (hot_steps) {
    PLATO_CUDA_TRY(cudaMemcpyAsync(h_seg.data(), seg, std::min(hot_steps + 1, all_steps) * 4ull,
                                   cudaMemcpyDeviceToHost, st));
    PLATO_CUDA_TRY(cudaStreamSynchronize(st));
  }
  std::vector<float> cost(hot_steps + 1);
  {
    double c = 0.0;
    for (uint32_t s = 0; s < hot_steps; ++s) {
      cost[s] = static_cast<float>(c);
      const uint32_t n = h_seg[s + 1] - h_seg[s];
      c += 1.0 + (n ? 0.5 : 0.0) + 0.01 * n;
    }
    cost[hot_steps] = static_cast<float>(c);
  }
  std::vector<uint2> pieces;
  std::vector<flat_sub> subs;
  std::vector<uint32_t> cta_sub;
  auto add = [&pieces](uint32_t first, uint32_t a, uint32_t b) {
    pieces.push_back(make_uint2(a == first ? a | kPieceFirst : a, b));
  };
  // first step in [lo, hi] whose cost is at least c
  auto at_cost = [&cost](uint32_t lo, uint32_t hi, double c) {
    return static_cast<uint32_t>(std::lower_bound(cost.begin() + lo, cost.begin() + hi, static_cast<float>(c)) -
                                 cost.begin());
  };
  uint32_t a = 0;
  for (uint32_t c = 0; c < pl.hot_ctas; ++c) {
    cta_sub.push_back(static_cast<uint32_t>(subs.size()));
    const double end = static_cast<double>(cost[hot_steps]) * (c + 1) / pl.hot_ctas;
    const uint32_t b = c + 1 == pl.hot_ctas ? hot_steps : at_cost(a, hot_steps, end);
    for (uint32_t k = 0; k < nb; ++k) {
      const uint32_t k0 = static_cast<uint32_t>(fs.edge[k] / kFlatHotStep);
      const uint32_t k1 = static_cast<uint32_t>(fs.edge[k + 1] / kFlatHotStep);
      const uint32_t lo = std::max(a, k0), hi = std::min(b, k1);
      if (lo >= hi) continue;
      subs.push_back(flat_sub{k, static_cast<uint32_t>(pieces.size())});
      uint32_t p0 = lo;
      for (uint32_t w = 0; w < kFlatHotWarps; ++w) {
        const double c1 = cost[lo] + (static_cast<double>(cost[hi]) - cost[lo]) * (w + 1) / kFlatHotWarps;
        const uint32_t p1 = w + 1 == kFlatHotWarps ? hi : at_cost(p0, hi, c1);
        add(k0, p0, p1);
        p0 = p1;
      }
    }
    a = b;
  }
  cta_sub.push_back(static_cast<uint32_t>(subs.size()));
  const uint32_t cold_piece0 = static_cast<uint32_t>(pieces.size());
  for (uint32_t w = 0; w < cold_pieces; ++w)
    add(0, static_cast<uint32_t>(static_cast<uint64_t>(cold_steps) * w / cold_pieces),
        static_cast<uint32_t>(static_cast<uint64_t>(cold_steps) * (w + 1) / cold_pieces));
  const uint32_t npieces = static_cast<uint32_t>(pieces.size());
  PLATO_TRY(put(d_pieces, pieces, st));
  PLATO_TRY(put(d_subs, subs, st));
  PLATO_TRY(put(d_cta, cta_sub, st));
  flat_view& f = pl.v;
  f = flat_view{};
  f.V = V;
  f.nb = nb;
  f.words = words;
  f.words1 = words1;
  f.cold_piece0 = cold_piece0;
  f.cold_pieces = npieces - cold_piece0;
  f.cold_back = pl.cold_blocks > sms * kFlatColdCtas;
  f.hid = hid;
  f.cid = cid;
  f.hw = hw;
  f.cw = cw;
  f.hmark = hmark;
  f.cmark = cmark;
  f.hseg = seg;
  f.cseg = seg + hot_steps;
  f.pieces = d_pieces;
  f.cta_sub = d_cta;
  f.subs = d_subs;
  f.meta = meta;
  f.spans = spans;
  f.part = reinterpret_cast<float*>(mem + o_part);
  f.head = reinterpret_cast<float*>(mem + o_head);
  f.carry = reinterpret_cast<float*>(mem + o_carry);
  const unsigned span_grid = (npieces + 127) / 128;
  scratch<uint32_t> wide(st);
  PLATO_TRY(wide.alloc(pool, 1));
  PLATO_CUDA_TRY(cudaMemsetAsync(wide.p, 0, 4, st));
  k_flat_spans<false><<<span_grid, 128, 0, st>>>(pl.v, npieces, hot_steps, cold_steps, segments, meta, nullptr,
                                                wide.p);
  PLATO_LAUNCHED("k_flat_spans");
  scratch<uint32_t> base(st);
  PLATO_TRY(base.alloc(pool, nmeta));
  PLATO_TRY(scan(thrust::make_transform_iterator(thrust::counting_iterator<uint32_t>(0), flat_crossing{meta}),
                     base.p, nmeta, pool, st));
  k_flat_span_base<<<grid_for(nmeta, 256), 256, 0, st>>>(base.p, nmeta, meta);
  PLATO_LAUNCHED("k_flat_span_base");
  k_flat_spans<true><<<span_grid, 128, 0, st>>>(pl.v, npieces, hot_steps, cold_steps, segments, meta, spans,
                                               nullptr);
  PLATO_LAUNCHED("k_flat_spans");
  PLATO_CUDA_TRY(cudaMemcpyAsync(&f.wide_words, wide.p, 4, cudaMemcpyDeviceToHost, st));
  PLATO_CUDA_TRY(cudaStreamSynchronize(st));  // the temporaries and the host vectors go
  pl.update_blocks = f.wide_words + std::min<uint32_t>(sms * 4, (words - f.wide_words + 15) / 16);
  if (pl.hot_ctas) {
    PLATO_CUDA_TRY(cudaFuncSetAttribute(k_flat_hot<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        kFlatBlockBytes));
    PLATO_CUDA_TRY(cudaFuncSetAttribute(k_flat_hot<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        kFlatBlockBytes));
  }
  pl.valid = true;
  return PLATO_OK;
}

}  // namespace plato_b200
