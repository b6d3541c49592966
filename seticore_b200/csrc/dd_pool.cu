// sc_dd_pool: many searches of different shapes in one pass over the GPU.
//
// A pool owns a device scratch arena of a stated budget.  A call takes a list of search
// requests (each with its own timesteps, channels, frequency resolution, drift range,
// threshold and precision), admits them into sub-batches whose scratch fits the arena,
// and for each sub-batch queues one fixed sequence of launches through exec_queue: every
// kernel runs once for up to 64 searches, and the tree kernel's persistent CTAs pull work
// items (tile x drift-block chunk) from all searches of the same row count.
//
// Autotuning: the first time a tree launch of a given class (rows, element type, and the
// power-of-two buckets of its largest drift-block count and total channels) is seen, it is
// timed with each candidate launch shape -- tile width (1056 or 352 channels) and
// shared-memory budget (which sets how many drift blocks share a staged trapezoid and how
// many CTAs share an SM) -- and the fastest is kept.  Timing reruns are harmless: the tree
// kernel only raises per-channel maxima, so repeating it is idempotent.
//
// CUDA graphs: a sub-batch seen before (same requests, same arena layout) is replayed
// from a captured graph, whose last kernels write the results to pinned host memory.
#include <algorithm>
#include <cstddef>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <unordered_map>
#include <vector>

#include "dd_common.cuh"
#include "dd_internal.h"

namespace {

thread_local std::string g_pool_error;

int pfail(int code, const std::string& m) {
  g_pool_error = m;
  return code;
}
int pcuda(cudaError_t e, const char* what) { return pfail(SC_DD_ECUDA, std::string(what) + ": " + cudaGetErrorString(e)); }

constexpr int kHostCands = 256;
constexpr int kMaxGraphs = 16;

uint64_t fnv(uint64_t h, const void* p, size_t n) {
  const unsigned char* c = static_cast<const unsigned char*>(p);
  for (size_t i = 0; i < n; ++i) h = (h ^ c[i]) * 1099511628211ull;
  return h;
}

int round_up_pow2(int n) {
  int r = 1;
  while (r < n) r *= 2;
  return r;
}

struct Planned {
  scb::ExecSearch es;
  double res;
  double min_drift;
  int beam, coarse;
  size_t bytes;
};

}  // namespace

struct sc_dd_pool {
  int device = 0, num_sms = 148;
  size_t budget = 0;
  char* arena = nullptr;
  size_t arena_bytes = 0;
  float* lvl_a = nullptr;
  float* lvl_b = nullptr;
  size_t lvl_floats = 0;
  size_t lvl_tried = 0;  // the largest size asked for so far
  scb::LevelSide side;  // side stream i's buffers: lvl_a + 2 + 2i and 3 + 2i lvl_floats
  char* host = nullptr;  // pinned: headers + candidate heads of the largest sub-batch
  size_t host_bytes = 0;
  cudaStream_t cap_stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, evj = nullptr, t0 = nullptr, t1 = nullptr;
  struct Graph {
    uint64_t key;
    cudaGraphExec_t exec;
    uint64_t last_use;
  };
  std::vector<Graph> graphs;
  std::unordered_map<uint64_t, int> seen;  // sub-batch key -> times seen
  std::unordered_map<uint64_t, scb::TreeLaunch> tuned_launch;
  uint64_t clock = 0;
  int tuning = 1, use_graphs = 1;
  bool tuning_now = false;
  sc_dd_pool_stats st{};
};

namespace {

// Power-of-two bucket of a positive count (tuning keys describe a launch's class, not
// its exact composition, so a mix of shapes is tuned a few times rather than per batch).
int bucket(long long v) {
  int b = 0;
  while ((1ll << b) < v) ++b;
  return b;
}

scb::TreeLaunch pool_tree_launch(void* ctx, const scb::TreeBatch& tb, int R, int elem) {
  sc_dd_pool* p = static_cast<sc_dd_pool*>(ctx);
  // The launch shape decides how many drift blocks share a staged tile, how wide the tile is
  // and how many CTAs fit an SM: the key is the rows, the element type, the largest
  // drift-block count and the launch's total channels, each bucketed.
  int max_jobs = 1;
  long long channels = 0;
  for (int k = 0; k < tb.count; ++k) {
    max_jobs = std::max(max_jobs, tb.g[k].n_jobs);
    channels += tb.g[k].N;
  }
  const int v[5] = {R, elem, bucket(max_jobs), bucket(channels), tb.pair16};
  const uint64_t key = fnv(1469598103934665603ull, v, sizeof(v));
  auto it = p->tuned_launch.find(key);
  if (it != p->tuned_launch.end()) return it->second;
  if (!p->tuning || !p->tuning_now) return scb::TreeLaunch{};
  // Time each candidate on the stream the search runs on (idempotent reruns): shared-memory
  // budgets with 1056-channel tiles, and 352-channel tiles.  The 32-row tree runs one CTA per
  // SM with long strips only: its candidates are the budgets from 200 KB up.
  cudaStream_t s = p->cap_stream;
  const scb::TreeLaunch cands16[5] = {{110, 1056}, {160, 1056}, {200, 1056}, {110, 352}, {48, 352}};
  const scb::TreeLaunch cands32[2] = {{200, 1056}, {226, 1056}};
  const scb::TreeLaunch* cands = R == 32 ? cands32 : cands16;
  const int n_cands = R == 32 ? 2 : 5;
  scb::TreeLaunch best{};
  float best_ms = 1e30f;
  for (int ci = 0; ci < n_cands; ++ci) {
    const scb::TreeLaunch& c = cands[ci];
    scb::TreeBatch copy = tb;
    cudaEventRecord(p->t0, s);
    if (scb::tree_max_batch(copy, R, p->num_sms, s, elem, c) != cudaSuccess) continue;
    cudaEventRecord(p->t1, s);
    cudaEventSynchronize(p->t1);
    float ms = 0;
    cudaEventElapsedTime(&ms, p->t0, p->t1);
    if (ms < best_ms) {
      best_ms = ms;
      best = c;
    }
  }
  p->tuned_launch[key] = best;
  p->st.tuned_launches++;
  return best;
}

// Grows the arena and the level buffers in stream order on `stream` (cudaFreeAsync /
// cudaMallocAsync): every earlier call of this pool has finished with them (a call
// synchronises its stream before it returns), and work of other streams -- another pool's,
// another server worker's -- is not waited for, as a device-wide synchronisation or a plain
// cudaFree would.  Graphs captured over the old buffers are dropped.  lvl_min: floats per level
// buffer that the searches need; lvl_want: that they can use, given where the memory is there.
int ensure_device(sc_dd_pool* p, size_t arena, size_t lvl_min, size_t lvl_want, cudaStream_t stream) {
  cudaError_t e;
  const bool levels = lvl_min > p->lvl_floats || lvl_want > std::max(p->lvl_floats, p->lvl_tried);
  if (arena > p->arena_bytes || levels) {
    for (auto& g : p->graphs) cudaGraphExecDestroy(g.exec);
    p->graphs.clear();
    p->seen.clear();
  }
  if (arena > p->arena_bytes) {
    if (p->arena) cudaFreeAsync(p->arena, stream);
    p->arena = nullptr;
    p->arena_bytes = 0;
    if ((e = cudaMallocAsync(reinterpret_cast<void**>(&p->arena), arena, stream)) != cudaSuccess)
      return pfail(SC_DD_ENOMEM, std::string("pool arena: ") + cudaGetErrorString(e));
    if ((e = cudaMemsetAsync(p->arena, 0, arena, stream)) != cudaSuccess) return pcuda(e, "pool arena memset");
    p->arena_bytes = arena;
  }
  if (levels) {
    const size_t least = std::max(lvl_min, p->lvl_floats);
    p->lvl_tried = std::max(p->lvl_tried, lvl_want);
    if (p->lvl_a) cudaFreeAsync(p->lvl_a, stream);
    p->lvl_a = p->lvl_b = nullptr;
    for (int i = 0; i < scb::kLevelSides; ++i) p->side.lvl_a[i] = p->side.lvl_b[i] = nullptr;
    p->lvl_floats = 0;
    // All pairs of level buffers in one allocation: the emitting level addresses a pair as
    // one array; pair 0 serves the pool's stream, pair 1 + i side stream i.
    const size_t pairs = 1 + (size_t)p->side.n;
    size_t lvl = std::max(least, lvl_want);
    e = cudaMallocAsync(reinterpret_cast<void**>(&p->lvl_a), 2 * pairs * lvl * sizeof(float), stream);
    if (e != cudaSuccess && lvl > least) {
      cudaGetLastError();
      lvl = least;
      e = cudaMallocAsync(reinterpret_cast<void**>(&p->lvl_a), 2 * pairs * lvl * sizeof(float), stream);
    }
    if (e != cudaSuccess) return pfail(SC_DD_ENOMEM, std::string("pool level buffers: ") + cudaGetErrorString(e));
    p->lvl_b = p->lvl_a + lvl;
    for (int i = 0; i < p->side.n; ++i) {
      p->side.lvl_a[i] = p->lvl_a + (2 + 2 * i) * lvl;
      p->side.lvl_b[i] = p->lvl_a + (3 + 2 * i) * lvl;
    }
    p->lvl_floats = lvl;
  }
  return SC_DD_OK;
}

// Queues one sub-batch; its results land in p->host.
cudaError_t queue_sub(sc_dd_pool* p, std::vector<Planned>& sub, cudaStream_t s) {
  std::vector<scb::ExecSearch> es(sub.size());
  char* h = p->host;
  for (size_t k = 0; k < sub.size(); ++k) {  // the last kernel of each search writes its results there
    es[k] = sub[k].es;
    es[k].report.hdr = reinterpret_cast<scb::SearchHeader*>(h);
    es[k].report.cands = reinterpret_cast<scb::Candidate*>(h + sizeof(scb::SearchHeader));
    es[k].report.head = std::min(kHostCands, es[k].cand_cap);
    h += sizeof(scb::SearchHeader) + sizeof(scb::Candidate) * kHostCands;
  }
  scb::ExecHooks hooks;
  hooks.ctx = p;
  hooks.tree_launch = pool_tree_launch;
  cudaError_t e = scb::exec_queue(es.data(), (int)es.size(), p->lvl_a, p->lvl_b, p->num_sms, s, hooks,
                                  p->side.n == 0 ? nullptr : &p->side);
  return e;
}

}  // namespace

extern "C" {

const char* sc_dd_pool_last_error(void) { return g_pool_error.c_str(); }

int sc_dd_pool_create(size_t scratch_budget_bytes, sc_dd_pool** out) {
  g_pool_error.clear();
  if (!out) return pfail(SC_DD_EINVAL, "sc_dd_pool_create: out is null");
  *out = nullptr;
  sc_dd_pool* p = new (std::nothrow) sc_dd_pool();
  if (!p) return pfail(SC_DD_ENOMEM, "sc_dd_pool_create: host allocation");
  cudaError_t e = cudaGetDevice(&p->device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&p->num_sms, cudaDevAttrMultiProcessorCount, p->device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&p->cap_stream, cudaStreamNonBlocking);
  if (e == cudaSuccess && scb::level_sides(false) > 0) e = cudaEventCreateWithFlags(&p->side.fork, cudaEventDisableTiming);
  for (int i = 0; i < scb::level_sides(false) && e == cudaSuccess; ++i) {
    if ((e = cudaStreamCreateWithFlags(&p->side.stream[i], cudaStreamNonBlocking)) == cudaSuccess &&
        (e = cudaEventCreateWithFlags(&p->side.join[i], cudaEventDisableTiming)) == cudaSuccess)
      p->side.n = i + 1;
  }
  for (cudaEvent_t* ev : {&p->ev0, &p->ev1, &p->evj, &p->t0, &p->t1})
    if (e == cudaSuccess) e = cudaEventCreate(ev);
  // The host buffer of the largest possible sub-batch, allocated once: pinned allocations
  // synchronise the device, which a pool serving beside other streams must not do per call.
  p->host_bytes = (size_t)4 * scb::kMaxBatch * (sizeof(scb::SearchHeader) + sizeof(scb::Candidate) * kHostCands);
  if (e == cudaSuccess) e = cudaMallocHost(&p->host, p->host_bytes);
  if (e != cudaSuccess) {
    if (p->host) cudaFreeHost(p->host);
    for (cudaEvent_t ev : {p->ev0, p->ev1, p->evj, p->t0, p->t1, p->side.fork})
      if (ev) cudaEventDestroy(ev);
    if (p->cap_stream) cudaStreamDestroy(p->cap_stream);
    for (int i = 0; i < scb::kLevelSides; ++i) {
      if (p->side.stream[i]) cudaStreamDestroy(p->side.stream[i]);
      if (p->side.join[i]) cudaEventDestroy(p->side.join[i]);
    }
    delete p;
    return pcuda(e, "sc_dd_pool_create");
  }
  p->budget = scratch_budget_bytes;
  *out = p;
  return SC_DD_OK;
}

int sc_dd_pool_destroy(sc_dd_pool* p) {
  if (!p) return SC_DD_OK;
  cudaDeviceSynchronize();
  for (auto& g : p->graphs) cudaGraphExecDestroy(g.exec);
  if (p->arena) cudaFreeAsync(p->arena, nullptr);
  if (p->lvl_a) cudaFreeAsync(p->lvl_a, nullptr);
  cudaDeviceSynchronize();
  if (p->host) cudaFreeHost(p->host);
  for (cudaEvent_t ev : {p->ev0, p->ev1, p->evj, p->t0, p->t1})
    if (ev) cudaEventDestroy(ev);
  if (p->cap_stream) cudaStreamDestroy(p->cap_stream);
  for (int i = 0; i < scb::kLevelSides; ++i) {
    if (p->side.stream[i]) cudaStreamDestroy(p->side.stream[i]);
    if (p->side.join[i]) cudaEventDestroy(p->side.join[i]);
  }
  if (p->side.fork) cudaEventDestroy(p->side.fork);
  delete p;
  return SC_DD_OK;
}

int sc_dd_pool_configure(sc_dd_pool* p, int autotune, int cuda_graphs) {
  if (!p) return pfail(SC_DD_EINVAL, "sc_dd_pool_configure: null pool");
  p->tuning = autotune ? 1 : 0;
  p->use_graphs = cuda_graphs ? 1 : 0;
  return SC_DD_OK;
}

int sc_dd_pool_stats_get(const sc_dd_pool* p, sc_dd_pool_stats* out) {
  if (!p || !out) return pfail(SC_DD_EINVAL, "sc_dd_pool_stats_get: null argument");
  *out = p->st;
  return SC_DD_OK;
}

size_t sc_dd_request_scratch_bytes(const sc_dd_request* r) {
  if (!r || r->num_timesteps < 2 || r->num_channels < 64) return 0;
  const int Tr = round_up_pow2(r->num_timesteps);
  const double res = 1e6 * r->foff_mhz / ((Tr - 1) * r->tsamp_s);
  const double nmax = r->max_drift / std::fabs(res * (Tr - 1));
  const int w = (int)(2 * std::ceil(nmax * (Tr - 1)));
  if (w < 1) return 0;
  const long long nwin = ((long long)r->num_channels + w - 1) / w;
  const int cap = (int)std::min<long long>(nwin + 1, r->num_channels / 2 + 2);
  const int elem = r->precision == SC_DD_PRECISION_BF16 ? scb::kElemBF16
                   : r->precision == SC_DD_PRECISION_FP16 ? scb::kElemF16 : scb::kElemF32;
  return scb::ExecSearch::scratch_bytes(Tr, r->num_channels, cap, elem);
}

int sc_dd_pool_search(sc_dd_pool* p, const sc_dd_request* reqs, int count, sc_dd_hit* out, int capacity,
                      int* num_hits, void* stream_ptr) {
  g_pool_error.clear();
  if (!p || count < 0 || (count > 0 && (!reqs || !num_hits)) || (capacity > 0 && !out))
    return pfail(SC_DD_EINVAL, "sc_dd_pool_search: null argument");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  // Plan every request.
  std::vector<Planned> plans(count);
  for (int i = 0; i < count; ++i) {
    const sc_dd_request& r = reqs[i];
    if (!r.dev_input || r.num_timesteps < 2 || r.num_timesteps > 2048 || r.num_channels < 64 ||
        r.row_stride < r.num_channels || !(r.tsamp_s > 0) || !(r.foff_mhz != 0))
      return pfail(SC_DD_EINVAL, "sc_dd_pool_search: bad request " + std::to_string(i));
    Planned& pl = plans[i];
    scb::ExecSearch& q = pl.es;
    q = scb::ExecSearch{};
    q.input = r.dev_input;
    q.row_stride = r.row_stride;
    q.T = r.num_timesteps;
    q.Tr = round_up_pow2(r.num_timesteps);
    q.N = r.num_channels;
    // dedoppler.cu:84-87, 194-198, 274
    const int dt = q.Tr - 1;
    pl.res = 1e6 * r.foff_mhz / (dt * r.tsamp_s);
    const double nmax = r.max_drift / std::fabs(pl.res * dt);
    q.dmin = (int)std::floor(-nmax);
    q.dmax = (int)std::floor(nmax);
    q.window_size = (int)(2 * std::ceil(nmax * dt));
    if (!(q.window_size >= 1) || q.dmax < q.dmin)
      return pfail(SC_DD_EINVAL, "sc_dd_pool_search: request " + std::to_string(i) + " has no drift range");
    q.snr_threshold = r.snr_threshold;
    q.elem = r.precision == SC_DD_PRECISION_BF16 ? scb::kElemBF16
             : r.precision == SC_DD_PRECISION_FP16 ? scb::kElemF16 : scb::kElemF32;
    const long long nwin = ((long long)q.N + q.window_size - 1) / q.window_size;
    q.cand_cap = (int)std::min<long long>(nwin + 1, q.N / 2 + 2);
    pl.min_drift = r.min_drift;
    pl.beam = r.beam;
    pl.coarse = r.coarse_channel;
    pl.bytes = scb::ExecSearch::scratch_bytes(q.Tr, q.N, q.cand_cap, q.elem);
  }
  // Admission: consecutive requests while their scratch fits the budget (at least one).
  size_t arena_need = 0, lvl_min = 0, lvl_want = 0;
  std::vector<std::pair<int, int>> subs;
  {
    int i = 0;
    while (i < count) {
      size_t used = 0;
      int j = i;
      while (j < count && (j == i || used + plans[j].bytes <= p->budget) && j - i < 4 * scb::kMaxBatch) {
        used += plans[j].bytes;
        ++j;
      }
      subs.push_back({i, j});
      arena_need = std::max(arena_need, used);
      i = j;
    }
    for (const Planned& pl : plans)
      if (pl.es.Tr > 32) {
        lvl_min = std::max(lvl_min, scb::level_buffer_floats(pl.es.Tr, pl.es.N));
        lvl_want = std::max(lvl_want, scb::level_buffer_want(pl.es.Tr, pl.es.N, pl.es.dmax - pl.es.dmin + 1));
      }
  }
  int rc = ensure_device(p, arena_need, lvl_min, lvl_want, stream);
  if (rc != SC_DD_OK) return rc;

  cudaError_t e;
  int total = 0;
  p->st.calls++;
  cudaEventRecord(p->ev0, stream);
  for (auto& sb : subs) {
    std::vector<Planned> sub(plans.begin() + sb.first, plans.begin() + sb.second);
    size_t off = 0;
    uint64_t key = 1469598103934665603ull;
    for (Planned& pl : sub) {
      pl.es.carve(p->arena + off);
      off += pl.bytes;
      const sc_dd_request& r = reqs[sb.first + (&pl - sub.data())];
      key = fnv(key, &r, sizeof(r));
    }
    // and the process-wide settings that change the launches
    const long long settings[4] = {scb::exact_statistics_always() ? 1 : 0, scb::stage_wait_tries(),
                                   scb::paired_fp16() ? 1 : 0, scb::level_stripe_bytes()};
    key = fnv(key, settings, sizeof(settings));
    p->st.sub_batches++;
    auto git = std::find_if(p->graphs.begin(), p->graphs.end(), [&](const sc_dd_pool::Graph& g) { return g.key == key; });
    if (p->use_graphs && git != p->graphs.end()) {
      git->last_use = ++p->clock;
      if ((e = cudaGraphLaunch(git->exec, stream)) != cudaSuccess) return pcuda(e, "graph launch");
      p->st.graph_replays++;
    } else {
      const int seen = ++p->seen[key];
      if (p->use_graphs && seen >= 2) {
        // Capture on the pool's stream, ordered after the caller's stream.
        cudaEventRecord(p->evj, stream);
        cudaStreamWaitEvent(p->cap_stream, p->evj, 0);
        cudaGraph_t g = nullptr;
        if ((e = cudaStreamBeginCapture(p->cap_stream, cudaStreamCaptureModeThreadLocal)) != cudaSuccess)
          return pcuda(e, "begin capture");
        p->tuning_now = false;
        cudaError_t qe = queue_sub(p, sub, p->cap_stream);
        e = cudaStreamEndCapture(p->cap_stream, &g);
        if (qe != cudaSuccess) return pcuda(qe, "capture");
        if (e != cudaSuccess) return pcuda(e, "end capture");
        cudaGraphExec_t ex = nullptr;
        e = cudaGraphInstantiate(&ex, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) return pcuda(e, "instantiate");
        if ((int)p->graphs.size() >= kMaxGraphs) {
          auto lru = std::min_element(p->graphs.begin(), p->graphs.end(),
                                      [](const sc_dd_pool::Graph& a, const sc_dd_pool::Graph& b) {
                                        return a.last_use < b.last_use;
                                      });
          cudaGraphExecDestroy(lru->exec);
          p->graphs.erase(lru);
        }
        p->graphs.push_back({key, ex, ++p->clock});
        p->st.graph_captures++;
        if ((e = cudaGraphLaunch(ex, stream)) != cudaSuccess) return pcuda(e, "graph launch");
      } else {
        // First sight: run directly; tree launches not seen before are tuned.
        p->tuning_now = true;
        std::swap(p->cap_stream, stream);  // the tuning hooks time on p->cap_stream
        e = queue_sub(p, sub, p->cap_stream);
        std::swap(p->cap_stream, stream);
        p->tuning_now = false;
        if (e != cudaSuccess) return pcuda(e, "search kernels");
      }
    }
    if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) return pcuda(e, "synchronise");
    // Results.
    const char* h = p->host;
    for (size_t k = 0; k < sub.size(); ++k, h += sizeof(scb::SearchHeader) + sizeof(scb::Candidate) * kHostCands) {
      const Planned& pl = sub[k];
      const scb::SearchHeader hd = *reinterpret_cast<const scb::SearchHeader*>(h);
      if (hd.error) return pfail(SC_DD_EINTERNAL, "a tree kernel gave up waiting for its staged rows");
      const int ncand = std::min(hd.num_candidates, pl.es.cand_cap);
      const int head = std::min(kHostCands, pl.es.cand_cap);
      std::vector<scb::Candidate> cands(ncand);
      const scb::Candidate* hc = reinterpret_cast<const scb::Candidate*>(h + sizeof(scb::SearchHeader));
      std::copy(hc, hc + std::min(ncand, head), cands.begin());
      if (ncand > head) {
        if ((e = cudaMemcpyAsync(cands.data() + head, pl.es.cands + head, sizeof(scb::Candidate) * (ncand - head),
                                 cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
            (e = cudaStreamSynchronize(stream)) != cudaSuccess)
          return pcuda(e, "candidate copy");
      }
      std::sort(cands.begin(), cands.end(),
                [](const scb::Candidate& a, const scb::Candidate& b) { return a.index < b.index; });
      int nk = 0;
      for (const scb::Candidate& c : cands) {
        int drift_bins = 0;
        if (!scb::decode_candidate(c, pl.es.dmin, pl.es.Tr, &drift_bins))
          return pfail(SC_DD_EINTERNAL, "drift recovery did not reproduce a top sum");
        const double drift_rate = drift_bins * pl.res;  // dedoppler.cu:305-317
        const float snr = (c.power - hd.median) / hd.std_dev;
        if (std::fabs(drift_rate) >= pl.min_drift) {
          if (total < capacity) {
            sc_dd_hit& o = out[total];
            o.index = c.index;
            o.drift_steps = drift_bins;
            o.drift_rate = drift_rate;
            o.snr = snr;
            o.power = c.power;
            o.incoherent_power = 0.0f;
            o.coarse_channel = pl.coarse;
            o.beam = pl.beam;
            o.num_timesteps = pl.es.T;
          }
          ++total;
          ++nk;
        }
      }
      num_hits[sb.first + k] = nk;
    }
  }
  cudaEventRecord(p->ev1, stream);
  cudaEventSynchronize(p->ev1);
  cudaEventElapsedTime(&p->st.last_call_ms, p->ev0, p->ev1);
  if (total > capacity) return pfail(SC_DD_ETRUNC, "more hits than capacity");
  return SC_DD_OK;
}

}  // extern "C"
