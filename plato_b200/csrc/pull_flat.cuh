// Flat pull: the pull gather as segmented sums over blocked edge streams.
//
// The sources [0, nb * kFlatBlock) of a relabelled graph are the most
// gathered ones (descending in-degree; out-degree goes with it).  The in-edges
// of a plan are split by source into nb hot streams, stream k holding the
// edges whose source lies in block k = [k * kFlatBlock, (k+1) * kFlatBlock),
// and one cold stream with the rest.  A stream is in row order; a row's edges
// of one stream are a segment.  k_flat_hot copies a block's ranks to shared
// memory (224 KB, one CTA of 32 warps per SM) and gathers there, with 16-bit
// ids; k_flat_cold gathers from global memory with 32-bit ids;
// k_flat_update adds each row's segment sums in stream order and applies the
// rank update.
//
// A stream is cut into steps of 512 (hot) or 256 (cold) edges, 16 or 8 per
// lane, and a warp walks a contiguous run of steps (a piece), so the work per
// warp does not depend on the row lengths.  One flag bit per edge marks the last edge of a segment.
// A step without a flag only adds to the lane's running sum; a step with
// flags joins the lanes with a segmented scan and stores each finished
// segment's sum at its ordinal in part[] (segments are numbered in stream
// order, so the stores of a warp are consecutive).  A segment cut by a piece
// boundary leaves its sums in carry[] and head[] of the pieces it crosses; the
// update adds those in piece order.  Every sum has a fixed order: results are
// the same from run to run.
//
// Why.  A gather of 4 random bytes costs an L2 request, and the chip answers
// 276 G of them a second whatever the array's size (64 warps per SM, 4 to 16 in
// flight a lane); L1 hits go at 560-790 G/s, shared memory at 1700 G/s.  RMAT
// s24's 263M gathers are 0.95 ms of L2 requests; its hottest 57344 sources are
// 46% of them, 24 blocks 90%.  RMAT s24, one PageRank epoch on one B200: 826 us
// with degree bins (pull_binned.cuh), 495 us here: k_flat_hot 211 us (210M
// edges), k_flat_cold 226 (53M), k_flat_update 82.  RMAT s22 219 -> 130 us, s20
// 98 -> 45, 16M uniform edges over 1M vertices 107 -> 80, 64M over 1M 300 -> 132.
#pragma once

#include <utility>

#include "common.cuh"
#include "profile.cuh"
#include "pull_merge.cuh"

struct plato_graph;

namespace plato_b200 {

constexpr int kFlatHotLane = 16;          // edges of a lane in a hot step
constexpr int kFlatColdLane = 8;          // and in a cold step
constexpr uint32_t kFlatHotStep = 32 * kFlatHotLane;
constexpr uint32_t kFlatColdStep = 32 * kFlatColdLane;
constexpr uint32_t kFlatBlock = 57344;    // sources of a hot block
constexpr uint32_t kFlatBlockBytes = kFlatBlock * sizeof(float);
constexpr uint32_t kFlatMaxBlocks = 24;
// Up to this many steps (64K edges) and words k_flat_run's CTAs are one cluster of 8 (epoch
// over a cooperative grid / over the cluster, one B200: RMAT s10 5.5 / 4.4 us,
// s11 6.3 / 4.9, s12 6.5 / 6.3, s13 6.3 / 7.6).
constexpr uint32_t kFlatCluster = 8, kFlatClusterSteps = 256;
constexpr uint32_t kFlatHotWarps = 32;
constexpr uint32_t kFlatColdThreads = 256;
constexpr uint32_t kFlatColdCtas = 5;      // resident per SM
constexpr uint32_t kPieceFirst = 0x80000000u;  // a piece at the start of its stream

// A part of one hot block that a CTA walks, its steps shared by its 32 warps.
struct flat_sub {
  uint32_t block, piece0;
};

struct flat_view {
  uint32_t V, nb, words;            // words = ceil(V / 32)
  uint32_t words1;                  // 32-row words that take part in the hot streams after the first
  uint32_t wide_words;              // the first words, which hold every segment across more than kFlatWideSpan pieces
  uint32_t cold_piece0, cold_pieces;
  uint32_t cold_back;               // k_flat_cold's CTAs take the pieces from the end
  const uint16_t* hid;              // hot ids, relative to their block
  const uint32_t* cid;              // cold ids
  const float* hw;                  // weights of the same edges, or null
  const float* cw;
  // a mark per lane and step: a bit per edge, set on the last of a segment,
  // and above it the number of such bits in the step's lanes before
  const uint32_t* hmark;            // 16 + 16 bits
  const uint16_t* cmark;            // 8 + 8 bits
  const uint32_t* hseg;             // segments that end before each step
  const uint32_t* cseg;
  const uint2* pieces;              // [pieces] first step | kPieceFirst, end step
  const uint32_t* cta_sub;          // [hot CTAs + 1]
  const flat_sub* subs;
  // per stream and 32 rows (flat_place): rows with a segment, ordinal of the
  // first, rows whose segment crosses pieces, index of the first of those in spans
  const uint4* meta;
  const uint2* spans;               // first and last piece of a crossing segment
  float* part;                          // [segments]
  float* head;                          // [pieces]
  float* carry;                         // [pieces]
};

// Place of stream k in arrays by stream and row (or 32-row word): every row
// for the first and the last stream, `rows1` for those between.
__host__ __device__ inline uint64_t flat_place(uint32_t k, uint64_t rows, uint64_t rows1) {
  return k == 0 ? 0 : rows + (k - 1) * rows1;
}

struct flat_plan {
  bool valid = false;
  bool early_only = false;               // epochs without an early exit are the bins'
  uint32_t hot_ctas = 0, cold_blocks = 0, update_blocks = 0;
  uint32_t run_ctas = 0, run_warps = 0;  // not 0: k_flat_run's grid, the plan's only kernel
  bool run_cluster = false;              // its CTAs are one cluster
  flat_view v{};
  dbuf<unsigned char> mem;  // every array of v
};

// Builds the plan of g's pull on `st` (pull_flat.cu): rows gather their
// in-neighbours.  plan.valid stays false where there is nothing to gather, the
// sources are not g's vertices (a partition), the rows are short (the degree
// bins are the faster), or the graph keeps its caller's order (its pull sums in
// the merge path's order, as plato_pagerank_csc_noalloc).
int build_flat_plan(plato_graph* g, flat_plan& plan, cudaStream_t st);

__device__ __forceinline__ void flat_prefetch(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// 32 consecutive bytes in one load, so that a warp's ids are read once.  The
// streams are read once an epoch and pass L1 and L2 by.
struct flat_words {
  uint32_t w[8];
};
template <bool kOnce>
__device__ __forceinline__ void flat_load(const void* p, flat_words& r) {
  if constexpr (kOnce)
    asm volatile("ld.global.nc.L1::no_allocate.L2::evict_first.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]), "=r"(r.w[6]),
                   "=r"(r.w[7])
                 : "l"(p));
  else
    asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]), "=r"(r.w[6]),
                   "=r"(r.w[7])
                 : "l"(p));
}

// A lane's weights of one step, multiplied into its values.
template <bool kOnce, int N>
__device__ __forceinline__ void flat_weigh(const float* w, float (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 8) {
    flat_words t;
    flat_load<kOnce>(w + i, t);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[i + k] *= __uint_as_float(t.w[k]);
  }
}

// The edges of a lane in one step, hot: 16-bit ids into shared memory.
template <bool kW>
struct flat_hot_gather {
  static constexpr int kLane = kFlatHotLane;
  static constexpr uint32_t kStep = kFlatHotStep;
  static constexpr uint32_t kAhead = 6;  // steps whose ids are on their way to L2
  const uint16_t* ids;
  const float* w;
  const uint32_t* marks;
  const uint32_t* seg;
  const float* xs;
  using regs = flat_words;
  __device__ __forceinline__ void ahead(uint32_t step, unsigned lane) const {
    const size_t e = static_cast<size_t>(step) * kStep;
    if (lane < kStep / 64) flat_prefetch(ids + e + lane * 64);
    if (lane == 8) flat_prefetch(marks + static_cast<size_t>(step) * 32);
    if (kW && lane >= 16) flat_prefetch(w + e + (lane - 16) * 32);
  }
  __device__ __forceinline__ void load(uint32_t step, unsigned lane, regs& r) const {
    flat_load<true>(ids + static_cast<size_t>(step) * kStep + lane * kLane, r);
  }
  __device__ __forceinline__ uint32_t mark(uint32_t step, unsigned lane) const {
    return __ldcs(marks + static_cast<size_t>(step) * 32 + lane);
  }
  __device__ __forceinline__ void values(uint32_t step, unsigned lane, const regs& r, float (&v)[kLane]) const {
#pragma unroll
    for (int i = 0; i < kLane / 2; ++i) {
      v[2 * i] = xs[r.w[i] & 0xFFFFu];
      v[2 * i + 1] = xs[r.w[i] >> 16];
    }
    if constexpr (kW) flat_weigh<true>(w + static_cast<size_t>(step) * kStep + lane * kLane, v);
  }
};

// Cold: 32-bit ids into global memory.  kRun: in a kernel that runs many
// epochs the state is written by other SMs between epochs: plain loads, which
// the barrier's acquire orders.
template <bool kW, bool kRun>
struct flat_cold_gather {
  static constexpr int kLane = kFlatColdLane;
  static constexpr uint32_t kAhead = kRun ? 0 : 4;
  const uint32_t* ids;
  const float* w;
  const uint16_t* marks;
  const uint32_t* seg;
  const float* x;
  using regs = flat_words;
  __device__ __forceinline__ void ahead(uint32_t step, unsigned lane) const {
    const size_t e = static_cast<size_t>(step) * kFlatColdStep;
    if (lane < 8) flat_prefetch(ids + e + lane * 32);
    if (lane == 8) flat_prefetch(marks + static_cast<size_t>(step) * 32);
    if (kW && lane >= 16 && lane < 24) flat_prefetch(w + e + (lane - 16) * 32);
  }
  __device__ __forceinline__ void load(uint32_t step, unsigned lane, regs& r) const {
    flat_load<!kRun>(ids + static_cast<size_t>(step) * kFlatColdStep + lane * kLane, r);
  }
  __device__ __forceinline__ uint32_t mark(uint32_t step, unsigned lane) const {
    const uint16_t* p = marks + static_cast<size_t>(step) * 32 + lane;
    return kRun ? __ldg(p) : __ldcs(p);
  }
  __device__ __forceinline__ void values(uint32_t step, unsigned lane, const regs& r, float (&v)[kLane]) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = kRun ? x[r.w[i]] : __ldg(x + r.w[i]);
    if constexpr (kW) flat_weigh<!kRun>(w + static_cast<size_t>(step) * kFlatColdStep + lane * kLane, v);
  }
};

// A store that a lane skips without leaving its warp.
__device__ __forceinline__ void flat_store_if(uint32_t on, float* p, float v) {
  asm volatile("{ .reg .pred q; setp.ne.u32 q, %0, 0; @q st.global.f32 [%1], %2; }" ::"r"(on), "l"(p), "f"(v)
               : "memory");
}

// An addition of its own, not one that the compiler keeps from an earlier use.
__device__ __forceinline__ float flat_add(float a, float b) {
  float c;
  asm("add.f32 %0, %1, %2;" : "=f"(c) : "f"(a), "f"(b));
  return c;
}
// A sum and what its additions rounded away, which is no number once the sum
// is infinite.
__device__ __forceinline__ float flat_mend(float sum, float lost) { return lost == lost ? sum + lost : sum; }

// One warp's walk over the steps of piece p.
//
// Rounding.  A lane adds its edges in pairs, so a row of n edges meets about
// n / 2 running sums; and the steps without an end, of which a hub row has
// thousands, keep what each addition rounds away (a few large terms are common
// there: a hub's own edge beside its leaves').  Largest relative error of a
// rank, edges one by one / so / by the degree bins: RMAT s18 5.2 / 4.2 / 3.6e-7,
// s24 4.9 / 4.2 / 3.8e-7, 18M uniform edges 4.4 / 3.9 / 3.3e-7; 64M edges into
// one vertex with its own 64 among them 1.7e-6 / 6e-8 / 3.6e-7.  Epoch one by
// one / so: RMAT s16 8.9 / 8.6 us, s20 44.3 / 45.1, s22 133.8 / 133.8, 64M uniform
// edges over 1M vertices 135 / 132, RMAT s21 with weights 105 / 106.  A hot step's
// second loop forms its pair sums again (flat_add): kept across the scan, eight
// more registers spill (s22 139 us); a cold step's four do not.
template <class Gather>
__device__ __forceinline__ void flat_piece(const flat_view& f, uint32_t p, const Gather& g) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int N = Gather::kLane;
  constexpr uint32_t kEnds = (1u << N) - 1u;
  const unsigned lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const uint2 pc = f.pieces[p];
  const uint32_t s0 = pc.x & ~kPieceFirst, s1 = pc.y;
  if (s0 >= s1) {
    if (lane == 0) f.carry[p] = 0.f;
    return;
  }
  typename Gather::regs cur;
  g.load(s0, lane, cur);
  uint32_t mark = g.mark(s0, lane);
  uint32_t base = __ldg(g.seg + s0);
  if constexpr (Gather::kAhead > 0)
    for (uint32_t s = s0 + 1; s < min(s1, s0 + Gather::kAhead); ++s) g.ahead(s, lane);
  const bool open =
      !(pc.x & kPieceFirst) && !(__ldg(g.marks + static_cast<size_t>(s0) * 32 - 1) & (1u << (N - 1)));
  const uint32_t j0 = open ? base : 0xffffffffu;  // the segment that began in an earlier piece
  float acc = 0.f;       // this lane's part of the open segment, from steps without an end
  float lost = 0.f;      // and what its additions have rounded away
  float carry = 0.f;     // the open segment's sum before those, the same in every lane
  for (uint32_t s = s0; s < s1; ++s) {
    float v[N];
    g.values(s, lane, cur, v);
    uint32_t mark_n = 0, base_n = 0;
    if (s + 1 < s1) {
      g.load(s + 1, lane, cur);
      mark_n = g.mark(s + 1, lane);
      base_n = __ldg(g.seg + s + 1);
    }
    if constexpr (Gather::kAhead > 0)
      if (s + Gather::kAhead < s1) g.ahead(s + Gather::kAhead, lane);
    const uint32_t fl = mark & kEnds;
    const unsigned ends = __ballot_sync(kAll, fl != 0);
    if (ends == 0) {
      float a = 0.f;
#pragma unroll
      for (int i = 0; i < N; i += 8)
        a += ((v[i] + v[i + 1]) + (v[i + 2] + v[i + 3])) + ((v[i + 4] + v[i + 5]) + (v[i + 6] + v[i + 7]));
      const float b = acc + a, d = b - acc;  // the sum, and its exact error (Knuth's two-sum)
      lost += (acc - (b - d)) + (a - d);
      acc = b;
    } else {
      // this lane's sum after its last segment end, joined over the lanes
      float t = 0.f;
#pragma unroll
      for (int i = 0; i < N; i += 2) {
        t = (fl >> i) & 1u ? v[i + 1] : t + (v[i] + v[i + 1]);
        t = (fl >> (i + 1)) & 1u ? 0.f : t;
      }
      const unsigned le = ends & (kAll >> (31 - lane));
      const int lo = le ? 31 - __clz(le) : 0;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const float o = __shfl_up_sync(kAll, t, d);
        if (static_cast<int>(lane) - d >= lo) t += o;
      }
      carry += warp_sum(flat_mend(acc, lost));
      acc = lost = 0.f;
      float run = __shfl_up_sync(kAll, t, 1);
      if (lane == 0) run = 0.f;
      if (!(ends & below)) run += carry;
      carry = __shfl_sync(kAll, t, 31);
      // the segments that end here; a step of several pieces' segment goes to head
      const uint32_t ord = base + (mark >> N);
      float* to = f.part + ord;
      if (ord == j0 && fl) {
        // its first end closes a segment of an earlier piece
        const int e = __ffs(fl) - 1;
        float h = 0.f;
#pragma unroll
        for (int i = 0; i < N; i += 2) h += (i <= e ? v[i] : 0.f) + (i < e ? v[i + 1] : 0.f);
        f.head[p] = run + h;
      }
#pragma unroll
      for (int i = 0; i < N; i += 2) {
        const uint32_t on0 = fl & (1u << i), on1 = fl & (2u << i);
        flat_store_if(on0, to, run + v[i]);
        to += on0 ? 1 : 0;
        run = on0 ? v[i + 1] : run + (N == 8 ? v[i] + v[i + 1] : flat_add(v[i], v[i + 1]));
        flat_store_if(on1, to, run);
        to += on1 ? 1 : 0;
        run = on1 ? 0.f : run;
      }
    }
    mark = mark_n;
    base = base_n;
  }
  acc = warp_sum(flat_mend(acc, lost));
  if (lane == 0) f.carry[p] = carry + acc;
}

// The kernels of an epoch are launched behind one another with programmatic
// serialisation: the next one's CTAs take the SMs that the last CTAs of the one
// before leave idle, and wait here until it has ended.  (Nothing before this
// reads what an earlier kernel wrote.)  Not so k_flat_cold behind k_flat_hot: a
// CTA that comes to an SM before it is idle finds it with 224 KB of shared memory
// and the rest as its L1 (RMAT s22 146 -> 197 us).  Epochs without / with it:
// RMAT s18 19.4 / 16.6 us, s19 31.8 / 26.6, 16M uniform edges 85 / 81.
__device__ __forceinline__ void flat_after() {
  asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
}

// Hot streams (bound by the L1/shared pipe, 78% busy at RMAT s22: 3.4-way bank
// conflicts and the segments' stores; about 300 instructions a step of 512 edges): CTA c walks its parts [cta_sub[c], cta_sub[c+1]), each within
// one block whose ranks it first copies to shared memory.
template <bool kW>
__global__ void __launch_bounds__(kFlatHotWarps * 32, 1) k_flat_hot(flat_view f, const float* __restrict__ x,
                                                                   const int* mode) {
  extern __shared__ float4 s_x4[];
  flat_after();
  if (mode && *mode == 2) return;
  const uint32_t sub1 = f.cta_sub[blockIdx.x + 1];
  for (uint32_t sub = f.cta_sub[blockIdx.x]; sub < sub1; ++sub) {
    const flat_sub sb = f.subs[sub];
    const uint32_t src0 = sb.block * kFlatBlock;
    const uint32_t n = min(kFlatBlock, f.V - src0), n4 = n / 4;
    __syncthreads();
    const float4* x4 = reinterpret_cast<const float4*>(x + src0);
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < n4; i += kFlatHotWarps * 32) s_x4[i] = __ldg(x4 + i);
    if (threadIdx.x < n % 4)
      reinterpret_cast<float*>(s_x4)[n4 * 4 + threadIdx.x] = __ldg(x + src0 + n4 * 4 + threadIdx.x);
    __syncthreads();
    const flat_hot_gather<kW> g{f.hid, f.hw, f.hmark, f.hseg, reinterpret_cast<const float*>(s_x4)};
    flat_piece(f, sb.piece0 + (threadIdx.x >> 5), g);
  }
}

// The cold stream, bound by L2 requests.  Its last pieces hold the short rows, a
// segment every few edges, and take longest.  A grid of more than one wave
// starts with them (epoch in order / from the end: RMAT s22 140 / 132 us, s23 257
// / 250, s24 503 / 497); within a wave all run at once, and the update's CTAs
// follow better in order (s18 16.7 / 18.0, s19 27.3 / 32.2, s21 72.4 / 73.0).
template <bool kW>
__global__ void __launch_bounds__(kFlatColdThreads, kFlatColdCtas)
    k_flat_cold(flat_view f, const float* __restrict__ x, const int* mode) {
  flat_after();
  if (mode && *mode == 2) return;
  const uint32_t cta = f.cold_back ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
  const uint32_t w = (cta * blockDim.x + threadIdx.x) >> 5;
  if (w >= f.cold_pieces) return;
  const flat_cold_gather<kW, false> g{f.cid, f.cw, f.cmark, f.cseg, x};
  flat_piece(f, f.cold_piece0 + w, g);
}

// The sums of one 32-row word's segments of a stream: lane l gets row l's.
// They were written by other SMs, in the same kernel when it runs many epochs.
// A lane adds the pieces of its row's segment four at a time.
__device__ __forceinline__ float flat_segment(const flat_view& f, const uint4& m, unsigned lane) {
  const unsigned below = (1u << lane) - 1u;
  if (!((m.x >> lane) & 1u)) return 0.f;
  if (!((m.z >> lane) & 1u)) return __ldcg(f.part + m.y + __popc(m.x & below));
  const uint2 sp = __ldg(f.spans + m.w + __popc(m.z & below));
  float y = 0.f;
  for (uint32_t p = sp.x; p < sp.y; p += 4) {  // 4 loads in flight
    float t[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = p + i < sp.y ? __ldcg(f.carry + p + i) : 0.f;
    y += (t[0] + t[1]) + (t[2] + t[3]);
  }
  return y + __ldcg(f.head + sp.y);
}

// The same where a segment may cross many pieces (a hub row crosses all pieces
// of a stream): the warp adds those longer than kFlatWideSpan one after another,
// 256 pieces in flight each.  Lanes alone wait for L2 every four pieces, but all
// rows of the word at once.  One epoch with all segments added by their lanes /
// the warp from 32, 16, 8 pieces up, one B200: 1M edges into one vertex 77 /
// 13.8, 13.8, 13.9 us; RMAT s16 8.8 / 8.9, 9.0, 14.2; s14 6.3 / 6.3, 6.3, 6.6.
constexpr uint32_t kFlatWideSpan = 32;
__device__ __forceinline__ float flat_wide_segment(const flat_view& f, const uint4& m, unsigned lane) {
  const unsigned below = (1u << lane) - 1u;
  float y = 0.f, h = 0.f;
  if (((m.x & ~m.z) >> lane) & 1u) y = __ldcg(f.part + m.y + __popc(m.x & below));
  if (m.z == 0) return y;  // the same in every lane
  uint2 sp = make_uint2(0u, 0u);
  if ((m.z >> lane) & 1u) {
    sp = __ldg(f.spans + m.w + __popc(m.z & below));
    h = __ldcg(f.head + sp.y);
  }
  const bool wide = sp.y - sp.x > kFlatWideSpan;
  if (!wide)
    for (uint32_t p = sp.x; p < sp.y; p += 4) {
      float t[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) t[i] = p + i < sp.y ? __ldcg(f.carry + p + i) : 0.f;
      y += (t[0] + t[1]) + (t[2] + t[3]);
    }
  for (unsigned todo = __ballot_sync(0xffffffffu, wide); todo; todo &= todo - 1) {  // in 64 bits: up to 28K pieces
    const int l = __ffs(todo) - 1;
    const uint32_t p0 = __shfl_sync(0xffffffffu, sp.x, l), p1 = __shfl_sync(0xffffffffu, sp.y, l);
    double a = 0.0;
    for (uint32_t p = p0 + lane; p < p1; p += 256) {
      float t[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) t[i] = p + 32 * i < p1 ? __ldcg(f.carry + p + 32 * i) : 0.f;
      a += static_cast<double>(((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7])));
    }
    a = warp_sum(a);
    if (lane == static_cast<unsigned>(l)) y = static_cast<float>(a);
  }
  return y + h;
}

__device__ __forceinline__ uint4 flat_shfl(const uint4& m, int l) {
  return make_uint4(__shfl_sync(0xffffffffu, m.x, l), __shfl_sync(0xffffffffu, m.y, l),
                    __shfl_sync(0xffffffffu, m.z, l), __shfl_sync(0xffffffffu, m.w, l));
}

// The metas of word w in the hot streams between the first and the cold one:
// lane k holds stream k + 1's.
__device__ __forceinline__ uint4 flat_middle_meta(const flat_view& f, uint32_t w, unsigned lane) {
  if (w >= f.words1 || lane + 1 >= f.nb) return make_uint4(0, 0, 0, 0);
  return __ldg(f.meta + f.words + static_cast<size_t>(lane) * f.words1 + w);
}

// The sums of those streams for the word's 32 rows, 8 streams' loads in flight
// (a chain of 23 streams at RMAT s24; epoch with 4 / 8: s24 518 / 503 us, s22
// 140.5 / 139.5, 64M uniform edges over 1M vertices 137.5 / 135).
__device__ __forceinline__ float flat_middle(const flat_view& f, const uint4& mk, unsigned lane) {
  float y = 0.f;
  for (uint32_t k = 0; k + 1 < f.nb; k += 8) {
    float t[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) t[i] = flat_segment(f, flat_shfl(mk, k + i), lane);  // streams past nb: empty
    y += ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
  }
  return y;
}

// Adds each row's segment sums, in stream order, and applies the update.  A
// warp takes two words of 32 rows at a time, nwarps apart, and loads the metas
// of its next two one round ahead, as the sums' loads wait for the metas.  RMAT
// s24: 82 us (about 170 instructions a word, issue 42% busy, the rest latency);
// 1 / 3 / 4 words at a time with 6 / 3 / 2 CTAs per SM 113 / 94 / 118.
// The first wide_words words have a CTA each, whose warps share the streams
// (epoch with the lanes' sums only / so: 5M edges into one vertex of 1M 220 /
// 15.4 us, 16M 303 / 27.4, 64M 275 / 55; flat_wide_segment in the main loop
// spills).
// With c.ctrl the last CTA to finish sums the partials in a fixed order and
// takes the epoch decision (epoch_decide).
struct flat_control {
  int* ctrl;       // [0] mode of the next epoch, [1] epochs run, [2] CTAs that finished
  double* delta;
  double scale, eps;
  uint32_t iteration;
  uint32_t polls;  // of a grid barrier of k_flat_run, before it gives up
  unsigned long long* seen = nullptr;  // the decision on the host, as it falls (epoch_decide)
};

template <class Update>
__global__ void __launch_bounds__(256, 4) k_flat_update(flat_view f, Update upd,
                                                        double* partials, flat_control c) {
  constexpr int R = 2;
  __shared__ double s_red[32];
  __shared__ bool s_last;
  __shared__ double s_wide[8][32];
  flat_after();
  if (upd.skip()) return;
  const unsigned lane = threadIdx.x & 31;
  const uint32_t nwarps = ((gridDim.x - f.wide_words) * blockDim.x) >> 5;
  const uint4* cold = f.meta + flat_place(f.nb, f.words, f.words1);
  double dl = 0.0;
  uint32_t w = f.words;
  if (blockIdx.x < f.wide_words) {
    const uint32_t warp = threadIdx.x >> 5;
    double y = 0.0;
    for (uint32_t k = warp; k <= f.nb; k += 8)
      if (k == 0 || k == f.nb || blockIdx.x < f.words1)
        y += flat_wide_segment(f, __ldg(f.meta + flat_place(k, f.words, f.words1) + blockIdx.x), lane);
    s_wide[warp][lane] = y;
    __syncthreads();
    if (warp == 0) {
      y = 0.0;
#pragma unroll
      for (int i = 0; i < 8; ++i) y += s_wide[i][lane];
      const uint32_t v = blockIdx.x * 32 + lane;
      if (v < f.V) dl = upd.apply(v, static_cast<float>(y), upd.load(v));
    }
  } else {
    w = f.wide_words + (((blockIdx.x - f.wide_words) * blockDim.x + threadIdx.x) >> 5);
  }
  uint4 m0[R], m1[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t wr = w + r * nwarps;
    m0[r] = f.nb && wr < f.words ? __ldg(f.meta + wr) : make_uint4(0, 0, 0, 0);
    m1[r] = wr < f.words ? __ldg(cold + wr) : make_uint4(0, 0, 0, 0);
  }
  for (; w < f.words; w += R * nwarps) {
    typename Update::operands ops[R];
    float y[R], z[R];
    uint4 n0[R], n1[R], mk[R];
#pragma unroll
    for (int r = 0; r < R; ++r) mk[r] = flat_middle_meta(f, w + r * nwarps, lane);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t v = (w + r * nwarps) * 32 + lane;
      ops[r] = upd.load(v < f.V ? v : 0u);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t wr = w + (R + r) * nwarps;
      n0[r] = f.nb && wr < f.words ? __ldg(f.meta + wr) : make_uint4(0, 0, 0, 0);
      n1[r] = wr < f.words ? __ldg(cold + wr) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      y[r] = flat_segment(f, m0[r], lane);
      z[r] = flat_segment(f, m1[r], lane);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t wr = w + r * nwarps, v = wr * 32 + lane;
      if (wr < f.words1) y[r] += flat_middle(f, mk[r], lane);
      y[r] += z[r];
      if (wr < f.words && v < f.V) dl += upd.apply(v, y[r], ops[r]);
      m0[r] = n0[r];
      m1[r] = n1[r];
    }
  }
  dl = block_sum<256>(dl, s_red);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = dl;
    if (c.ctrl) {
      __threadfence();
      s_last = atomicAdd(c.ctrl + 2, 1) == static_cast<int>(gridDim.x) - 1;
    }
  }
  if (!c.ctrl) return;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double t = 0.0;
  for (uint32_t i = threadIdx.x; i < gridDim.x; i += 256) t += __ldcg(partials + i);
  t = block_sum<256>(t, s_red);
  if (threadIdx.x == 0) {
    c.ctrl[2] = 0;
    epoch_decide(c.ctrl, c.delta, t * c.scale, c.eps, c.iteration, c.seen);
  }
}

// All arrivals of a barrier are in.  The count goes round after 2^32 arrivals
// (14.5M epochs on 148 CTAs); no two CTAs are more than a barrier apart.
constexpr __host__ __device__ bool flat_arrived(uint32_t seen, uint32_t target) {
  return static_cast<int32_t>(seen - target) >= 0;
}
static_assert(flat_arrived(148, 148) && !flat_arrived(147, 148) && flat_arrived(4, 0xFFFFFFF0u) &&
              !flat_arrived(0xFFFFFFF0u, 4), "also where the count has gone round");

// Barrier over the CTAs of k_flat_run.  One cluster: the hardware's barrier,
// which orders global memory over the cluster.  A cooperative launch: sync[0]
// counts arrivals over the whole launch (`target` of them release this
// barrier), sync[1] is set when a CTA gives up waiting after `polls` reads
// (kBarrierPolls: many seconds), and then every CTA returns.
__device__ __forceinline__ bool flat_barrier(uint32_t* sync, uint32_t target, bool cluster, uint32_t polls) {
  __shared__ int s_ok;
  if (cluster) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    return true;
  }
  __syncthreads();
  if (gridDim.x == 1) return true;
  if (threadIdx.x == 0) {
    int ok = 0;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(sync) : "memory");
    for (uint32_t n = 0; n < polls; ++n) {
      uint32_t seen, failed;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(sync) : "memory");
      if (flat_arrived(seen, target)) {
        ok = 1;
        break;
      }
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(failed) : "l"(sync + 1) : "memory");
      if (failed) break;
    }
    if (!ok) asm volatile("st.relaxed.gpu.global.u32 [%0], 1;" ::"l"(sync + 1) : "memory");
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

template <class Update>
__device__ __noinline__ void flat_poison(const flat_view& f, const Update& upd, uint32_t w0,
                                         uint32_t nwarps) {
  for (uint32_t w = w0; w < f.words; w += nwarps) {
    const uint32_t v = w * 32 + (threadIdx.x & 31);
    if (v < f.V) upd.poison(v);
  }
}

// Every epoch of a small graph in one launch, cooperative over gridDim.x <= SMs
// CTAs or, up to 256 steps, one cluster of 8 (one CTA alone is bound by issue,
// and a barrier through L2 costs more than 64K edges' gathers): gather, barrier,
// update, barrier.  The grid has a warp for every step and every 32-row word, as
// far as they go (by the steps alone, 1000 edges over 1M vertices 3.0 ms an epoch).
// The epoch kinds and the eps exit follow epoch_decide;
// ctrl[1] = epochs run, counted from `start`.  Launches bound these graphs: one
// epoch with a launch per degree bin / here, RMAT s10 52 / 4.4 us, s12 54 / 6.3, s16
// 70 / 9.4, 48K uniform edges 28 / 5.8.  A CTA that gives up waiting leaves NaN
// in its rows; the host finds the give-up word with the results.
template <class Update, bool kW>
__global__ void __launch_bounds__(kFlatHotWarps * 32, 1) k_flat_run(flat_view f,
                                                                   Update upd, uint32_t start, uint32_t iteration,
                                                                   double scale, double eps, int* ctrl, double* delta,
                                                                   double* partials, uint32_t* sync, bool cluster,
                                                                   uint32_t polls) {
  __shared__ double s_red[32];
  __shared__ double s_delta;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t cta_warps = blockDim.x >> 5;
  const uint32_t w0 = blockIdx.x * cta_warps + warp, nwarps = gridDim.x * cta_warps;
  const bool deltas = !(eps <= 0.0);  // as run_pull_epochs: an eps that is no number never ends the epochs
  uint32_t barriers = 0, ran = start;
  bool last = start + 1 >= iteration;
  for (;;) {
    upd.final_epoch = last ? 1 : 0;
    flat_piece(f, w0, flat_cold_gather<kW, true>{f.cid, f.cw, f.cmark, f.cseg, upd.gathered()});
    if (!flat_barrier(sync, ++barriers * gridDim.x, cluster, polls)) return flat_poison(f, upd, w0, nwarps);
    double dl = 0.0;
    for (uint32_t w = w0; w < f.words; w += nwarps) {
      const uint32_t v = w * 32 + lane;
      const bool mine = v < f.V;
      const typename Update::operands ops = upd.load_l2(mine ? v : w * 32);
      const float y = flat_wide_segment(f, __ldg(f.meta + w), lane);
      if (mine) dl += upd.apply(v, y, ops);
    }
    ++ran;
    if (last) break;
    double* sums = partials + (ran & 1u) * gridDim.x;
    if (deltas) {
      dl = warp_sum(dl);
      if (lane == 0) s_red[warp] = dl;
      __syncthreads();
      dl = warp_sum(lane < cta_warps ? s_red[lane] : 0.0);
      if (threadIdx.x == 0) __stcg(sums + blockIdx.x, dl);
    }
    if (!flat_barrier(sync, ++barriers * gridDim.x, cluster, polls)) return flat_poison(f, upd, w0, nwarps);
    last = ran + 1 >= iteration;
    if (deltas) {  // every CTA sums the partials in the same order
      if (warp == 0) {
        double t = 0.0;
        for (uint32_t i = lane; i < gridDim.x; i += 32) t += __ldcg(sums + i);
        t = warp_sum(t) * scale;
        if (lane == 0) s_delta = t;
      }
      __syncthreads();
      if (s_delta < eps) last = true;
    }
    upd.flip();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctrl[0] = 2;
    ctrl[1] = static_cast<int>(ran);
    if (deltas && ran > start + 1) *delta = s_delta;
  }
}

template <class... P, class... A>
cudaError_t flat_launch(bool behind, void (*kernel)(P...), uint32_t grid, uint32_t block, size_t smem, cudaStream_t st,
                        A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = behind ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// The kernels of one epoch of a plan without run_ctas: sums of x into upd.
template <class Upd, bool kW>
int launch_flat_epoch(const flat_plan& p, const float* x, const Upd& upd, double* partials, const flat_control& c,
                      cudaStream_t st) {
  if (p.hot_ctas) {
    prof_scope ps("k_flat_hot", st);
    PLATO_CUDA_TRY(flat_launch(true, k_flat_hot<kW>, p.hot_ctas, kFlatHotWarps * 32, kFlatBlockBytes, st, p.v,
                               x, c.ctrl));
    PLATO_LAUNCHED("k_flat_hot");
  }
  if (p.cold_blocks) {
    prof_scope ps("k_flat_cold", st);
    PLATO_CUDA_TRY(flat_launch(p.hot_ctas == 0, k_flat_cold<kW>, p.cold_blocks, kFlatColdThreads, 0, st, p.v, x,
                               c.ctrl));
    PLATO_LAUNCHED("k_flat_cold");
  }
  prof_scope ps("k_flat_update", st);
  PLATO_CUDA_TRY(flat_launch(true, k_flat_update<Upd>, p.update_blocks, 256, 0, st, p.v, upd, partials, c));
  PLATO_LAUNCHED("k_flat_update");
  return PLATO_OK;
}

// All epochs of a plan with run_ctas.  c.ctrl [4]: [1] becomes the epochs run,
// [2] and [3] are the barrier's; cleared here.
template <class Upd, bool kW>
int launch_flat_run(const flat_plan& p, const Upd& upd, uint32_t start, double* partials,
                    const flat_control& c, cudaStream_t st) {
  PLATO_CUDA_TRY(cudaMemsetAsync(c.ctrl, 0, 4 * sizeof(int), st));
  prof_scope ps("k_flat_run", st);
  uint32_t* sync = reinterpret_cast<uint32_t*>(c.ctrl + 2);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(p.run_ctas);
  cfg.blockDim = dim3(p.run_warps * 32);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  if (p.run_cluster) {
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = p.run_ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
  } else {
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
  }
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  PLATO_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_flat_run<Upd, kW>, p.v, upd, start, c.iteration, c.scale, c.eps, c.ctrl,
                                    c.delta, partials, sync, p.run_cluster, c.polls));
  PLATO_LAUNCHED("k_flat_run");
  return PLATO_OK;
}

}  // namespace plato_b200
