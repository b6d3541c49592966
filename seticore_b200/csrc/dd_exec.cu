// Queues the kernels of a list of searches of any shapes, drift ranges and precisions.
//
// Used by the engine (dd_api.cu, one shape) and by the pool (dd_pool.cu, mixed shapes).
// The searches travel in batches of up to kMaxBatch as kernel parameters, so a call is a
// fixed sequence of launches (capturable in a CUDA graph) whatever the mix:
//   clear -> [normalise] -> [one or two searches: column sums, statistics beside what follows] ->
//   tree launches grouped by (rows, element type), the float32 ones
//   adding the column sums -> levels for more than 32 rows, one search at a time -> column
//   sums (searches whose trees did not compute them) -> statistics -> exact statistics ->
//   [flag + FP32 recompute of the flagged channels] -> hits
#include <algorithm>
#include <cstddef>
#include <cstdlib>

#include "dd_common.cuh"
#include "dd_internal.h"

namespace scb {

namespace {

// Zeroes, per search of the batch: top (and the 16-bit tops), the result header and the
// flagged-channel count.
__global__ void clear_kernel(const __grid_constant__ SearchBatch b, const __grid_constant__ PrecisionBatch pb) {
  const SearchDesc& d = b.s[blockIdx.y];
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < d.N; c += gridDim.x * blockDim.x) d.top[c] = 0.0f;
  if (blockIdx.x == 0 && threadIdx.x < (int)(sizeof(SearchHeader) / 4))
    reinterpret_cast<int*>(d.hdr)[threadIdx.x] = 0;
  if (pb.count > 0 && blockIdx.y < (unsigned)pb.count && pb.s[blockIdx.y].flag_count) {
    const PrecisionDesc& q = pb.s[blockIdx.y];
    float* t16 = const_cast<float*>(q.top16);
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < q.N; c += gridDim.x * blockDim.x) t16[c] = 0.0f;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      *q.flag_count = 0;
      *q.ticket = 0;
    }
  }
}

SearchDesc to_desc(const ExecSearch& e) {
  SearchDesc s{};
  s.input = e.input;
  s.row_stride = e.row_stride;
  s.Tr = e.Tr;
  s.N = e.N;
  s.dmin = e.dmin;
  s.dmax = e.dmax;
  s.window_size = e.window_size;
  s.first = (int)ceil(0.05 * e.N);  // dedoppler.cu:247
  s.mid = e.N / 2;                   // dedoppler.cu:211
  s.last = (int)floor(0.95 * e.N);  // dedoppler.cu:248
  s.snr_threshold = e.snr_threshold;
  s.top = e.top;
  s.colsum = e.colsum;
  s.work = e.work;
  s.lists = e.lists;
  s.hdr = e.hdr;
  s.cands = e.cands;
  s.cand_cap = e.cand_cap;
  s.report = e.report;
  s.report.flag_count = e.flag_count;
  s.report.norm = e.norm_moments ? e.norm_moments + 2 * kVarChunks : nullptr;
  return s;
}

// 16-bit 16- and 32-row searches take the paired-FP16 tree when it is on (the flag bound must
// know).
bool pair16_search(const ExecSearch& e, bool on) { return on && e.elem != kElemF32 && pair_rows(e.Tr); }

PrecisionDesc to_pdesc(const ExecSearch& e, const SearchHeader* hdr, bool pair_on) {
  PrecisionDesc q{};
  q.input = e.input;
  q.row_stride = e.row_stride;
  q.T = e.T;
  q.Tr = e.Tr;
  q.N = e.N;
  q.norm = e.norm16;
  q.colsum = e.colsum;
  q.moments = e.norm_moments;
  q.ticket = e.norm_ticket;
  q.top16 = e.top16;
  q.hdr = hdr;
  q.snr_threshold = e.snr_threshold;
  q.dmin = e.dmin;
  q.dmax = e.dmax;
  q.top = e.top;
  q.flag_list = e.flags;
  q.flag_count = e.flag_count;
  q.pair16 = pair16_search(e, pair_on) ? 1 : 0;
  return q;
}

// Searches whose column sums come with another pass over the input: the float32 tree of up
// to 32 rows (its drift range always holds drift block 0: dmin <= 0 <= dmax), and the
// 16-bit forms' normalising pass.
bool tree_colsum(const ExecSearch& e) { return e.elem == kElemF32 && e.Tr <= 32 && e.dmin <= 0 && e.dmax >= 0; }
bool fused_colsum(const ExecSearch& e) { return tree_colsum(e) || e.elem != kElemF32; }

// Whether the first level of a search of more than 32 float rows forms the column sums on the way.
// They cost it its spread: a tile's row groups then run one after another on one CTA.  That pays
// where tiles are many -- a dozen per SM for a search alone, two per SM beside others, whose launches
// fill the gaps.  32 beams of 256 x 131072: 5.13 -> 4.95 ms (0.60 ms of their own launch before, 0.43
// ms more in the levels); 4 of 64 x 2^20: 0.16 of 3.65 ms saved; but one by one, 256 x 131072 with 4
// drift blocks 2.00 -> 2.27 ms of levels for 0.17 ms of sums.
bool levels_sum_columns(const ExecSearch& q, bool alone, int num_sms) {
  return q.N / 352 >= (alone ? 12ll : 2ll) * num_sms;
}

// Whether a batch is one or two searches so long that the whole GPU forms their statistics (after the
// tree) faster than a cluster each: from 2^22 channels on (one of 2^24, whose statistics a cluster forms in
// 0.82 ms and the GPU in 0.18; at 3 * 2^20 the two are even).
bool long_searches(const ExecSearch* s, int m) {
  if (m > kWideStatsSearches) return false;
  for (int k = 0; k < m; ++k)
    if (s[k].N < kWideStatsChannels) return false;
  return true;
}

// Whether the trees of long searches of up to 32 rows take long enough to hide a cluster's statistics beside
// them: their work per channel, about Tr (log2 Tr + 3/4) for each drift block, against 50 us per 2^20
// channels. One of 2^22 channels, statistics beside the tree and by the GPU after it: 16 x 6 drift
// blocks 387 and 350 us, 16 x 10 393 and 436, 8 x 12 353 and 345, 8 x 26 404 and 451, 4 x 54 336 and 374.
// The 32-row tree, one CTA per SM, gives up more for the cluster's SMs: 32 x 26 1745 and 1649, 54 3212
// and 3186, two searches of 54 6143 and 6252.
bool tree_hides_statistics(const ExecSearch* s, int m) {
  long long work = 0;
  for (int k = 0; k < m; ++k) work += (long long)(s[k].dmax - s[k].dmin + 1) * s[k].Tr * (4 * (31 - __builtin_clz(s[k].Tr)) + 3);
  return work >= (s[0].Tr == 32 ? 73600 : 2360);  // 100 drift blocks of 32 rows; 7.8 of 16
}

// Whether the column sums and the statistics of a batch run before its tree, which then starts while
// the statistics are under way.  The statistics of a search are a chain of barriers on 16 SMs (25 us
// at 32768 channels, 70 at 2^20) that leaves the others idle; beside the tree they cost it those SMs
// for that long, and one more read of the input for the sums (12 us at 16 x 2^20, which the tree then
// finds in L2).  Device time, after and before the tree: 16 x 2^20, 54 drift blocks 310 -> 268 us,
// 14 drift blocks 167 -> 130; 16 x 32768 71 -> 52; 16 x 4096 63 -> 49; 32 x 2^20 546 -> 503; 64 x
// 100003 272 -> 248; 256 x 131072, 2 drift blocks 702 -> 670.  Two searches gain as much (2 of
// 16 x 2^20 555 -> 526); four, whose statistics take 64 SMs, no more than 2 % and lose as much at
// some sizes (4 of 16 x 32768, 14 drift blocks 74 -> 75).  Not where the levels form the sums on the
// way.  The 16-bit forms, whose sums the normalising pass forms before the tree, have not been measured
// this way.
bool statistics_first(const ExecSearch* s, int m, int num_sms) {
  if (m > 2) return false;
  if (long_searches(s, m) && !tree_hides_statistics(s, m)) return false;
  if (s[0].Tr > 32)
    return m == 1 && s[0].elem == kElemF32 && s[0].Tr <= 256 && !levels_sum_columns(s[0], true, num_sms);
  for (int k = 0; k < m; ++k)
    if (!tree_colsum(s[k]) || s[k].Tr != s[0].Tr) return false;
  return true;
}

// The search's header word that a kernel sets when it gives up a wait.
int* header_status(const ExecSearch& e) {
  return reinterpret_cast<int*>(reinterpret_cast<char*>(e.hdr) + offsetof(SearchHeader, error));
}

TreeGroup tree_group(const ExecSearch& e, const void* rows, long long row_stride, float* top) {
  TreeGroup g{};
  g.rows = rows;
  g.row_stride = row_stride;
  g.job_row_stride = 0;
  g.N = e.N;
  g.d_first = e.dmin;
  g.d_step = 1;
  g.n_jobs = e.dmax - e.dmin + 1;
  g.db_first = e.dmin;
  g.db_step = 1;
  g.off_base = 0;
  g.off_step = 0;
  g.elig_T1 = e.Tr - 1;
  g.top = top;
  g.status = header_status(e);
  return g;
}

}  // namespace

int level_sides(bool engine) {
  static const long v = [] {
    const char* e = getenv("SETICORE_B200_LEVEL_SIDES");
    return e ? strtol(e, nullptr, 10) : -1L;
  }();
  // An engine holds one search shape, so its extra buffer pairs are small: three sides
  // (beams 194.5 -> 197.4 Gsamples/s).  A pool sizes its pairs for its largest search and
  // serves beside others: one.
  const long x = v >= 0 ? v : (engine ? 3 : 1);
  return (int)std::min<long>(kLevelSides, std::max<long>(0, x));
}

cudaError_t exec_queue(const ExecSearch* s, int n, float* lvl_a, float* lvl_b, int num_sms, cudaStream_t stream,
                       const ExecHooks& hooks, const LevelSide* side) {
  cudaError_t e = cudaSuccess;
  const bool pair_on = paired_fp16();  // read once: the trees and the flag bounds agree
  for (int k0 = 0; k0 < n && e == cudaSuccess; k0 += kMaxBatch) {
    const int m = std::min(kMaxBatch, n - k0);
    const ExecSearch* ss = s + k0;
    SearchBatch b;
    b.count = m;
    b.maxN = 0;
    for (int k = 0; k < m; ++k) {
      b.s[k] = to_desc(ss[k]);
      b.maxN = std::max(b.maxN, ss[k].N);
    }
    // Clear (one launch).
    PrecisionBatch clear_pb;
    clear_pb.count = m;
    clear_pb.maxN = b.maxN;
    clear_pb.elem = kElemBF16;
    for (int k = 0; k < m; ++k) {
      clear_pb.s[k] = PrecisionDesc{};
      if (ss[k].elem != kElemF32) clear_pb.s[k] = to_pdesc(ss[k], b.s[k].hdr, pair_on);
    }
    {
      int gx = (b.maxN + 1023) / 1024;
      if (gx > 64) gx = 64;
      clear_kernel<<<dim3(gx, m), 256, 0, stream>>>(b, clear_pb);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    // Normalisation of the 16-bit searches (one launch per element type).
    for (int elem : {kElemBF16, kElemF16}) {
      PrecisionBatch q;
      q.count = 0;
      q.maxN = 0;
      q.elem = elem;
      for (int k = 0; k < m; ++k)
        if (ss[k].elem == elem) {
          q.s[q.count++] = to_pdesc(ss[k], b.s[k].hdr, pair_on);
          q.maxN = std::max(q.maxN, ss[k].N);
        }
      if (q.count && (e = normalize_batch(q, num_sms, stream)) != cudaSuccess) return e;
    }
    const bool stats_first = statistics_first(ss, m, num_sms);
    const int min_ties = exact_statistics_ties();
    if (stats_first && (e = column_sums_batch(b, stream)) != cudaSuccess) return e;
    if (hooks.before_tree) hooks.before_tree(hooks.ctx, stream);
    if (stats_first && (e = search_stats_emulated(b, num_sms, min_ties, stream)) != cudaSuccess) return e;
    // Trees over up to 32 rows: one launch per (rows, element type).
    for (int R : {2, 4, 8, 16, 32}) {
      for (int elem : {kElemF32, kElemBF16, kElemF16}) {
        TreeBatch tb;
        tb.count = 0;
        tb.n_items = 0;
        tb.pair16 = (elem != kElemF32 && pair_rows(R) && pair_on) ? 1 : 0;
        SearchHeader* first = nullptr;
        tb.beside_previous = stats_first ? 1 : 0;
        for (int k = 0; k < m; ++k) {
          if (ss[k].Tr != R || ss[k].elem != elem) continue;
          if (!tb.count) first = b.s[k].hdr;
          if (elem == kElemF32) {
            TreeGroup g = tree_group(ss[k], ss[k].input, ss[k].row_stride, ss[k].top);
            if (tree_colsum(ss[k]) && !stats_first) {
              g.colsum = ss[k].colsum;
              g.colsum_job = -ss[k].dmin;
            }
            tb.g[tb.count++] = g;
          } else if (tb.pair16) {
            // the paired copy: channel 0 of row 0 sits kPairPad words into the buffer
            TreeGroup g = tree_group(ss[k], static_cast<const uint32_t*>(ss[k].norm16) + kPairPad,
                                     pair_row_words(ss[k].N), ss[k].top16);
            g.pad = kPairPad;
            tb.g[tb.count++] = g;
          } else {
            tb.g[tb.count++] = tree_group(ss[k], ss[k].norm16, ss[k].N, ss[k].top16);
          }
        }
        if (tb.count && R <= 16) tb.next_item = &first->next_item;
        if (tb.count && (e = tree_max_batch(tb, R, num_sms, stream, elem, hooks.tree_launch(hooks.ctx, tb, R, elem))) !=
                            cudaSuccess)
          return e;
      }
    }
    // More than 32 rows: the level path, one search at a time per level-buffer pair.  FP32
    // searches are dealt round-robin over the main stream and the side streams, when there are
    // any (two concurrent 16-bit level searches measured slower than one after the other: their
    // first level is bound by L1 throughput, not by latency); the 16-bit searches run it on
    // their normalised copy, with the default split, on the main stream, before the side streams
    // start: beside the float searches there they were never faster (pools of 2 to 16 searches of 64
    // to 2048 rows: -0.5 to 6 % slower).  A search that is alone,
    // or wide (below), runs on the main stream with every pair, which lie side by side: a search
    // of many drift blocks then needs a pass per eight of them, not per two (60 x 100003, 36
    // drift blocks: levels 0.68 -> 0.46 ms).
    const long long half = lvl_b - lvl_a;
    const int pairs = side && side->n > 0 ? 1 + side->n : 1;
    // Wide: its drift blocks do not fit one pass of its own pair, and a pass of all pairs fills
    // the GPU for long enough (128 MB of planes) that the launches' ends do not matter.  Eight
    // searches each: 256 x 131072, 4 drift blocks 2195 -> 2007 us; 128 x 131072, 10 drift blocks
    // 2628 -> 2317; 4 of 64 x 2^20, 8 drift blocks 3948 -> 3482.  But 16 of 64 x 32768, 8 drift
    // blocks: 573 side by side and 618 one by one; 256 x 131072, 2 drift blocks: 1112 and 1202.
    // More than 256 rows take one drift block at a time whatever the buffers hold, so there the
    // planes of one drift block decide: from 48 MB on, the planes of searches side by side push one
    // another's out of L2 between the levels.  Eight searches, 10 drift blocks, side by side and one by
    // one: 2048 x 1024 (10 MB) 1.69 and 2.52 ms; 1024 x 8192 (35 MB) 3.99 and 4.30; 512 x 20480
    // (43 MB) 5.06 and 4.86; 512 x 24576 (52 MB) 5.99 and 5.59; 512 x 131072 (277 MB) 31.2 and 25.8.  Not
    // with two drift blocks: 1024 x 12288 1.30 and 1.35.
    auto wide = [&](const ExecSearch& q) {
      const long long np = level_row_length(q.N), per_db = q.Tr * (np + kLevelRowSlack), ndb = q.dmax - q.dmin + 1;
      if (pairs == 1) return false;
      if (q.Tr > 256) return ndb > 2 && q.Tr * np * (long long)sizeof(float) >= (48ll << 20);
      return ndb * per_db > 2 * half &&
             std::min<long long>(ndb, 2 * half * pairs / per_db) * per_db * (long long)sizeof(float) >= (128ll << 20);
    };
    bool summed[kMaxBatch];
    for (int k = 0; k < m; ++k) summed[k] = stats_first || fused_colsum(ss[k]);
    auto level = [&](int k, bool alone, float* la, float* lb, cudaStream_t st) {
      const ExecSearch& q = ss[k];
      float* colsum = levels_sum_columns(q, alone, num_sms) ? q.colsum : nullptr;
      return levels_search(q.input, q.row_stride, q.Tr, q.N, q.dmin, q.dmax, la, lb, q.top, num_sms, st, colsum, &summed[k],
                           kElemF32, header_status(q), &b.s[k].hdr->next_item, stats_first);
    };
    int n_level = 0;
    for (int k = 0; k < m; ++k) n_level += ss[k].Tr > 32 && ss[k].elem == kElemF32 && !wide(ss[k]);
    const int lanes = pairs > 1 && n_level >= 2 ? std::min(pairs, n_level) : 1;
    for (int k = 0; k < m; ++k) {  // the main stream's searches, before the side streams start
      const ExecSearch& q = ss[k];
      if (q.Tr <= 32) continue;
      if (q.elem != kElemF32)
        e = levels_search(q.norm16, q.N, q.Tr, q.N, q.dmin, q.dmax, lvl_a, lvl_b, q.top16, num_sms, stream, nullptr,
                          nullptr, q.elem, header_status(q));
      else if (lanes == 1 || wide(q))
        e = level(k, true, lvl_a, lvl_a + half * pairs, stream);
      if (e != cudaSuccess) return e;
    }
    if (lanes > 1) {
      if ((e = cudaEventRecord(side->fork, stream)) != cudaSuccess) return e;
      for (int i = 0; i + 1 < lanes; ++i)
        if ((e = cudaStreamWaitEvent(side->stream[i], side->fork, 0)) != cudaSuccess) return e;
      int j = 0;
      for (int k = 0; k < m; ++k) {
        if (ss[k].Tr <= 32 || ss[k].elem != kElemF32 || wide(ss[k])) continue;
        const int lane = j++ % lanes;  // 0: the main stream
        if ((e = lane ? level(k, false, side->lvl_a[lane - 1], side->lvl_b[lane - 1], side->stream[lane - 1])
                      : level(k, false, lvl_a, lvl_b, stream)) != cudaSuccess)
          return e;
      }
    }
    for (int i = 0; i + 1 < lanes; ++i) {
      if ((e = cudaEventRecord(side->join[i], side->stream[i])) != cudaSuccess ||
          (e = cudaStreamWaitEvent(stream, side->join[i], 0)) != cudaSuccess)
        return e;
    }
    if (hooks.after_tree) hooks.after_tree(hooks.ctx, stream);
    // Column sums where the statistics did not come first: the float32 trees over up to 32 rows compute
    // their own from the staged rows, the 16-bit forms in their normalising pass and the levels where
    // they can; the rest read the input once more here.
    {
      SearchBatch cb;
      cb.count = 0;
      cb.maxN = 0;
      for (int k = 0; k < m; ++k)
        if (!summed[k]) {
          cb.s[cb.count++] = b.s[k];
          cb.maxN = std::max(cb.maxN, ss[k].N);
        }
      if ((e = column_sums_batch(cb, stream)) != cudaSuccess) return e;
    }
    if (!stats_first && (e = long_searches(ss, m) ? search_stats_wide(b, num_sms, min_ties, stream)
                                                   : search_stats_emulated(b, num_sms, min_ties, stream)) != cudaSuccess)
      return e;
    if ((e = search_stats_exact(b, min_ties, stream)) != cudaSuccess) return e;
    // The 16-bit searches: list the channels near the threshold, recompute them exactly
    // in FP32 from the original power.
    {
      PrecisionBatch q;
      q.count = 0;
      q.maxN = 0;
      q.elem = kElemBF16;
      for (int k = 0; k < m; ++k)
        if (ss[k].elem != kElemF32) {
          q.s[q.count++] = to_pdesc(ss[k], b.s[k].hdr, pair_on);
          q.maxN = std::max(q.maxN, ss[k].N);
        }
      if (q.count) {
        if ((e = flag_channels_batch(q, num_sms, stream)) != cudaSuccess) return e;
        if ((e = recompute_batch(q, num_sms, stream)) != cudaSuccess) return e;
      }
    }
    if ((e = search_hits_batch(b, num_sms, stream)) != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

size_t ExecSearch::scratch_bytes(int Tr, int N, int cand_cap, int elem) {
  auto a = [](size_t x) { return (x + 255) & ~size_t(255); };
  size_t b = a(sizeof(float) * N) * 2 + a(sizeof(float) * order_work_floats(N)) +
             a(sizeof(int) * order_list_entries(N)) + a(sizeof(SearchHeader)) + a(sizeof(Candidate) * cand_cap);
  if (elem != kElemF32) {
    b += a(norm_buffer_bytes(Tr, N)) + a(sizeof(float) * N) + a(sizeof(int) * N) + a(sizeof(int)) +
         a(sizeof(double) * kNormMomentsDoubles) + a(sizeof(unsigned));
  }
  return b;
}

void ExecSearch::carve(char* base) {
  auto a = [](size_t x) { return (x + 255) & ~size_t(255); };
  char* p = base;
  top = reinterpret_cast<float*>(p);
  p += a(sizeof(float) * N);
  colsum = reinterpret_cast<float*>(p);
  p += a(sizeof(float) * N);
  work = reinterpret_cast<float*>(p);
  p += a(sizeof(float) * order_work_floats(N));
  lists = reinterpret_cast<int*>(p);
  p += a(sizeof(int) * order_list_entries(N));
  hdr = reinterpret_cast<SearchHeader*>(p);
  p += a(sizeof(SearchHeader));
  cands = reinterpret_cast<Candidate*>(p);
  p += a(sizeof(Candidate) * cand_cap);
  if (elem != kElemF32) {
    norm16 = p;
    p += a(norm_buffer_bytes(Tr, N));
    top16 = reinterpret_cast<float*>(p);
    p += a(sizeof(float) * N);
    flags = reinterpret_cast<int*>(p);
    p += a(sizeof(int) * N);
    flag_count = reinterpret_cast<int*>(p);
    p += a(sizeof(int));
    norm_moments = reinterpret_cast<double*>(p);
    p += a(sizeof(double) * kNormMomentsDoubles);
    norm_ticket = reinterpret_cast<unsigned*>(p);
  }
}

}  // namespace scb
