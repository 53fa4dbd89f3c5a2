// TrustRank: good-seed selection, then seed-set personalized PageRank.
//
// Mirrors plato/algo/trustrank/trustrank.hpp:
//   select (select_good_seeds, :88-146)
//     V <= seed_num       every good vertex is a seed;
//     method 0 / 1        the seed_num vertices of highest inverse PageRank
//                         (PageRank of the transposed graph, generate_rank_pairs
//                         over the out-edges, :52-71) or PageRank, ordered by
//                         rank descending then id ascending, that are good;
//     method 2            seed_num distinct vertices drawn uniformly, the good
//                         ones kept (the reference seeds its generator from
//                         std::random_device; here the caller's seed is used,
//                         so a run can be repeated).
//   trust (trustrank, :163-259)  seed-set PPR with those seeds: init 1/|S|
//                         (divided by the out-degree) on seeds, teleport
//                         (1-d)/|S| on seeds, eps early exit into a final
//                         epoch -- plato_seedset_ppr on the binned pull.
// The selection PageRank is the reference's default run (pagerank_opts_t:
// 100 epochs, damping 0.85, eps 0.001; pagerank.hpp:39-46, 81-146) in double
// precision on the flat pull (pull_flat.cuh; over the out-edges for the
// transposed graph), so the order of the ranks is the reference's up to FP64
// rounding, and the same from run to run.
#include <algorithm>
#include <exception>
#include <mutex>
#include <random>
#include <unordered_set>
#include <vector>

#include <cub/device/device_radix_sort.cuh>

#include "graph.cuh"
#include "plato_b200/dualmode.cuh"
#include "pull_flat.cuh"

namespace plato_b200 {
namespace {

__global__ void k_tr_init(double* x, const uint32_t* __restrict__ deg, uint32_t V) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V;
       v += (uint64_t)gridDim.x * blockDim.x)
    x[v] = deg[v] > 0 ? 1.0 / deg[v] : 1.0;  // pagerank.hpp:90-98
}

__global__ void k_tr_fill(double* x, uint32_t V, double value) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V;
       v += (uint64_t)gridDim.x * blockDim.x)
    x[v] = value;
}

// pagerank.hpp:118-135: r = (1-d) + d*y; non-final epochs divide by the degree
// and sum |x' - x| * deg.
struct selection_update {
  using value = double;
  const double* x;  // current state
  double* xn;       // next state
  const uint32_t* __restrict__ deg;
  double d;
  int final_epoch;
  const int* mode = nullptr;  // epoch kind on the device, as in rank_update

  __device__ __forceinline__ bool skip() const { return mode && *mode == 2; }
  __device__ __forceinline__ bool storing_rank() const { return mode ? (*mode == 1) : (final_epoch != 0); }

  struct operands {
    uint32_t dg;
    double xo;
  };
  __device__ __forceinline__ operands load(uint32_t v) const { return {__ldcs(deg + v), __ldcs(x + v)}; }
  // load() inside a kernel that runs many epochs (the state is other SMs' work)
  __device__ __forceinline__ operands load_l2(uint32_t v) const { return {__ldg(deg + v), __ldcg(x + v)}; }
  __device__ __forceinline__ const double* gathered() const { return x; }
  __device__ __forceinline__ void flip() {
    const double* t = x;
    x = xn;
    xn = const_cast<double*>(t);
  }
  __device__ __forceinline__ void poison(uint32_t v) const {
    xn[v] = const_cast<double*>(x)[v] = __longlong_as_double(0x7fffffffffffffffll);
  }
  __device__ __forceinline__ double apply(uint32_t v, double y, operands o) const {
    double r = (1.0 - d) + d * y, dl = 0.0;
    if (!storing_rank()) {
      if (o.dg > 0) {
        r /= o.dg;
        dl = fabs(r - o.xo) * o.dg;
      } else {
        dl = fabs(r - o.xo);
      }
    }
    xn[v] = r;
    return dl;
  }
};

// Selection ranks laid out by caller id, with the caller ids beside them.
__global__ void k_tr_keys(const double* __restrict__ r, const uint32_t* __restrict__ to_ext, uint32_t V,
                          double* keys, uint32_t* ids) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V;
       v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t e = to_ext ? to_ext[v] : static_cast<uint32_t>(v);
    keys[e] = r[v];
    ids[e] = e;
  }
}

// The k caller ids of highest rank, ties by smaller id (trustrank.hpp:108-112),
// chosen on the device: a stable descending radix sort of (rank, id) pairs
// laid out by ascending id keeps equal ranks in id order.  Ranks are
// positive and finite, where the radix order of doubles is their numeric
// order.
std::vector<uint32_t> top_ids(const double* r, const uint32_t* to_ext, uint32_t V, uint32_t k) {
  double *ka = nullptr, *kb = nullptr;
  uint32_t *ia = nullptr, *ib = nullptr;
  void* tmp = nullptr;
  size_t bytes = 0;
  std::vector<uint32_t> out(k);
  check_cuda(cub::DeviceRadixSort::SortPairsDescending(nullptr, bytes, ka, kb, ia, ib, static_cast<int64_t>(V)),
             "top ids");
  try {
    dev_alloc(&ka, 8ull * V, "top ids");
    dev_alloc(&kb, 8ull * V, "top ids");
    dev_alloc(&ia, 4ull * V, "top ids");
    dev_alloc(&ib, 4ull * V, "top ids");
    dev_alloc(&tmp, bytes, "top ids");
    k_tr_keys<<<grid_for(V, 256), 256>>>(r, to_ext, V, ka, ia);
    check_cuda(cudaGetLastError(), "k_tr_keys");
    count_launch();
    check_cuda(cub::DeviceRadixSort::SortPairsDescending(tmp, bytes, ka, kb, ia, ib, static_cast<int64_t>(V)),
               "top ids");
    if (k) check_cuda(cudaMemcpy(out.data(), ib, 4ull * k, cudaMemcpyDeviceToHost), "top ids");
  } catch (...) {
    dev_free(ka);
    dev_free(kb);
    dev_free(ia);
    dev_free(ib);
    dev_free(tmp);
    throw;
  }
  dev_free(ka);
  dev_free(kb);
  dev_free(ia);
  dev_free(ib);
  dev_free(tmp);
  return out;
}

}  // namespace

// The selection's plans (pulls over the in-edges and, transposed, over the
// out-edges), kept with the graph, and its epoch control.
struct trust_workspace {
  flat_plan<double> plan[2];
  bool built[2] = {false, false};
  dbuf<double> x[2], partials, delta;
  dbuf<int> ctrl;
  int* h_ctrl = nullptr;  // pinned [8]: two control words
  cudaEvent_t polled[2] = {nullptr, nullptr};
  ~trust_workspace() {
    if (h_ctrl) cudaFreeHost(h_ctrl);
    for (cudaEvent_t e : polled)
      if (e) cudaEventDestroy(e);
  }
};

void destroy_trust_workspace(trust_workspace* w) { delete w; }

namespace {

constexpr uint32_t kSelectIterations = 100;
constexpr double kSelectDamping = 0.85, kSelectEps = 0.001;

// The selection PageRank on the flat pull (pull_flat.cuh) in 64 bits, its exit
// decided on the device; *ranks = the state that holds them.
int selection_ranks(plato_graph* g, bool inverse, cudaStream_t st, const double** ranks) {
  if (!g->trust_ws) {
    g->trust_ws = new (std::nothrow) trust_workspace();
    if (!g->trust_ws) return set_error(PLATO_ENOMEM, "trustrank: host allocation failed");
  }
  trust_workspace* ws = g->trust_ws;
  const int side = inverse ? 1 : 0;
  const uint32_t V = g->info.vertices;
  flat_plan<double>& pl = ws->plan[side];
  if (!ws->built[side]) {
    PLATO_TRY(build_flat_plan<double>(g, inverse, pl, st));
    ws->built[side] = true;
  }
  *ranks = nullptr;
  if (!pl.valid) return PLATO_OK;
  for (auto& x : ws->x) PLATO_TRY(x.alloc(V));
  PLATO_TRY(ws->partials.alloc(std::max<size_t>(pl.update_blocks, 2ull * pl.run_ctas)));
  PLATO_TRY(ws->delta.alloc(1));
  PLATO_TRY(ws->ctrl.alloc(4));
  if (!ws->h_ctrl) PLATO_CUDA_TRY(cudaMallocHost(reinterpret_cast<void**>(&ws->h_ctrl), 8 * sizeof(int)));
  for (cudaEvent_t& e : ws->polled)
    if (!e) PLATO_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  // out-degrees of the structure the pull walks: in-degrees when transposed
  const uint32_t* deg = inverse ? g->in_deg.p : g->out_deg.p;
  k_tr_init<<<grid_for(V, 256), 256, 0, st>>>(ws->x[0].p, deg, V);
  PLATO_LAUNCHED("k_tr_init");
  const flat_control c{ws->ctrl.p, ws->delta.p, 1.0, kSelectEps, kSelectIterations};
  const auto update = [&](uint32_t epoch, const int* mode) {
    return selection_update{ws->x[epoch & 1].p, ws->x[(epoch & 1) ^ 1].p, deg, kSelectDamping, 0, mode};
  };
  int ran = 0;
  if (pl.run_ctas) {
    PLATO_TRY((launch_flat_run<selection_update, false>(pl, update(0, nullptr), 0, ws->partials.p, c, st)));
    PLATO_CUDA_TRY(cudaMemcpyAsync(ws->h_ctrl, ws->ctrl.p, 4 * sizeof(int), cudaMemcpyDeviceToHost, st));
    PLATO_CUDA_TRY(cudaStreamSynchronize(st));
    if (ws->h_ctrl[3]) return set_error(PLATO_ETIMEDOUT, "k_flat_run: a grid barrier ran out");
    ran = ws->h_ctrl[1];
  } else {
    PLATO_CUDA_TRY(cudaMemsetAsync(ws->ctrl.p, 0, 4 * sizeof(int), st));
    // a few epochs at a time, one batch ahead of the control word read
    constexpr uint32_t kBatch = 6;
    uint32_t epoch = 0, batches = 0;
    while (epoch < kSelectIterations) {
      for (uint32_t k = 0; k < kBatch && epoch < kSelectIterations; ++k, ++epoch)
        PLATO_TRY((launch_flat_epoch<selection_update, false>(pl, ws->x[epoch & 1].p, update(epoch, ws->ctrl.p),
                                                              ws->partials.p, c, st)));
      const uint32_t slot = batches++ & 1u;
      PLATO_CUDA_TRY(cudaMemcpyAsync(ws->h_ctrl + 4 * slot, ws->ctrl.p, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
      PLATO_CUDA_TRY(cudaEventRecord(ws->polled[slot], st));
      if (batches == 1) continue;
      PLATO_CUDA_TRY(cudaEventSynchronize(ws->polled[slot ^ 1]));
      if (ws->h_ctrl[4 * (slot ^ 1)] == 2) break;
    }
    PLATO_CUDA_TRY(cudaStreamSynchronize(st));
    ran = ws->h_ctrl[4 * ((batches - 1) & 1u) + 1];
  }
  *ranks = ws->x[ran & 1].p;
  return PLATO_OK;
}

int select_seeds(plato_graph* g, const plato_trustrank_opts* o, const uint8_t* good,
                 std::vector<plato_vid_t>* seeds) {
  const uint32_t V = g->info.vertices;
  auto is_good = [good](uint32_t v) { return good == nullptr || good[v] != 0; };
  seeds->clear();
  if (static_cast<uint64_t>(g->info.max_v_i) + 1 <= o->seed_num) {  // trustrank.hpp:98-102
    for (uint32_t v = 0; v < V; ++v)
      if (is_good(v)) seeds->push_back(v);
    return PLATO_OK;
  }
  if (o->select_method == 2) {  // trustrank.hpp:124-143
    std::mt19937_64 gen(o->random_seed);
    std::uniform_int_distribution<uint32_t> dist(0, g->info.max_v_i);
    std::unordered_set<uint32_t> picked;
    while (picked.size() < o->seed_num) {
      const uint32_t v = dist(gen);
      if (picked.insert(v).second && is_good(v)) seeds->push_back(v);
    }
    std::sort(seeds->begin(), seeds->end());
    return PLATO_OK;
  }
  const uint32_t k = std::min<uint32_t>(o->seed_num, V);
  const double* ranks = nullptr;
  PLATO_TRY(selection_ranks(g, o->select_method == 0, 0, &ranks));
  dbuf<double> flat_ranks;
  if (!ranks) {  // no edge: every vertex keeps the teleport
    PLATO_TRY(flat_ranks.alloc(V));
    k_tr_fill<<<grid_for(V, 256), 256>>>(flat_ranks.p, V, 1.0 - kSelectDamping);
    PLATO_LAUNCHED("k_tr_fill");
    ranks = flat_ranks.p;
  }
  const std::vector<uint32_t> order = top_ids(ranks, g->relabeled ? g->to_ext.p : nullptr, V, k);
  for (uint32_t i = 0; i < k; ++i)
    if (is_good(order[i])) seeds->push_back(order[i]);
  std::sort(seeds->begin(), seeds->end());
  return PLATO_OK;
}

}  // namespace
}  // namespace plato_b200

using namespace plato_b200;

extern "C" int plato_trustrank(plato_graph* g, const plato_trustrank_opts* opts,
                               const uint8_t* good_vertices, float* ranks, plato_vid_t* seeds_out,
                               uint32_t* n_seeds, plato_run_stats* stats) {
  if (!g || !opts) return set_error(PLATO_EINVAL, "plato_trustrank: null argument");
  if (opts->select_method > 2) return set_error(PLATO_EINVAL, "plato_trustrank: select_method must be 0, 1 or 2");
  if (opts->seed_num == 0) return set_error(PLATO_EINVAL, "plato_trustrank: seed_num must be >= 1");
  std::vector<plato_vid_t> seeds;
  {
    std::lock_guard<std::mutex> lock(g->mu);
    PLATO_CUDA_TRY(cudaSetDevice(g->device));
    PLATO_CUDA_TRY(cudaStreamSynchronize(g->stream));  // the selection runs on the default stream
    try {
      PLATO_TRY(select_seeds(g, opts, good_vertices, &seeds));
    } catch (const std::exception& e) {
      return set_error(PLATO_ECUDA, std::string("plato_trustrank: ") + e.what());
    }
  }
  if (n_seeds) *n_seeds = static_cast<uint32_t>(seeds.size());
  if (seeds_out) std::copy(seeds.begin(), seeds.end(), seeds_out);
  if (seeds.empty())
    return set_error(PLATO_EINVAL, "plato_trustrank: no good vertex among the selected seeds");
  const plato_ppr_opts po{opts->iteration, opts->damping, 0, opts->eps};
  return plato_seedset_ppr(g, seeds.data(), static_cast<uint32_t>(seeds.size()), &po, ranks, stats);
}
