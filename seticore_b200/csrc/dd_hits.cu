// Hit selection on the GPU.
//
// window_kernel: the reference's window de-duplication (dedoppler.cu:264-303).  Channels
//   are cut into non-overlapping windows of window_size; a window's candidate is the
//   first channel holding its largest top sum, if that sum is strictly above the
//   threshold; it survives if no channel in [c - window_size + 1, c + window_size) has a
//   strictly larger top sum.  One warp or block per window.
// resolve_kernel: recovers the drift of each survivor.  The reference keeps, per channel,
//   the first (drift block, offset) in scan order whose sum beat the running maximum
//   (dedoppler.cu:49-53); that is the first eligible path, in (drift block, offset)
//   order, whose sum equals the final top sum.  The fused tree kernel keeps only the top
//   value, so the few survivors recompute their paths here, bit-identically (the tree's
//   pairing): one thread per (survivor, drift block) up to 16 rows (resolve_direct_kernel),
//   one thread per (survivor, path) beyond; the host decodes the packed best and checks its
//   sum against the stored top sum.
// path_values_kernel: addIncoherentPower (dedoppler.cu:139-176): the path sum along a
//   hit's path; the drift block is floor((float)drift_steps / (Tr-1)) in float, as there.
#include <algorithm>

#include "dd_common.cuh"
#include "dd_internal.h"

namespace scb {

namespace {

// The first channel of [start, end) with the largest value above `best`, over GROUP threads
// (a warp or the block), each of which holds its own first best on return.  Eight loads in
// flight per thread: a window's time is its loads' latency.
template <int GROUP>
__device__ __forceinline__ void window_best(const float* __restrict__ top, int start, int end, int t, float& best,
                                            int& bidx) {
  constexpr int K = 8;
  const float floor_v = best;
  const float* __restrict__ p = top + start;
  const int n = end - start;
  for (int f0 = t; f0 < n; f0 += GROUP * K) {
    float v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = f0 + GROUP * k < n ? __ldg(p + f0 + GROUP * k) : floor_v;  // floor_v: not above best
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (v[k] > best) {
        best = v[k];
        bidx = start + f0 + GROUP * k;
      }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bidx, o);
    if (oi >= 0 && (bidx < 0 || ov > best || (ov == best && oi < bidx))) {
      best = ov;
      bidx = oi;
    }
  }
}

// Whether a value above `best` lies in [lo, hi) among this thread's share.
template <int GROUP>
__device__ __forceinline__ bool window_larger(const float* __restrict__ top, int lo, int hi, int t, float best) {
  constexpr int K = 8;
  const float* __restrict__ p = top + lo;
  const int n = hi - lo;
  bool larger = false;
  for (int f0 = t; f0 < n && !larger; f0 += GROUP * K) {
    float v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = f0 + GROUP * k < n ? __ldg(p + f0 + GROUP * k) : best;
#pragma unroll
    for (int k = 0; k < K; ++k) larger = larger || v[k] > best;
  }
  return larger;
}

constexpr int kWindowThreads = 256;

// A search whose windows are no more than its blocks takes a block for each: one warp for 2194
// channels with one load in flight needed 31 us on 46 windows (eight in flight 17 us, a block
// 8 us).  With more windows than blocks a warp each is the faster (64 searches of 1338 windows
// of 784 channels: 80 us, and 239 us by blocks, most of whose threads idle).
__global__ void __launch_bounds__(kWindowThreads) window_kernel(const __grid_constant__ SearchBatch b) {
  const SearchDesc& sd = b.s[blockIdx.y];
  const float* __restrict__ top = sd.top;
  const int N = sd.N, w = sd.window_size, cap = sd.cand_cap;
  SearchHeader* hdr = sd.hdr;
  Candidate* cands = sd.cands;
  const float thr = hdr->threshold;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long nwin = ((long long)N + w - 1) / w;
  auto keep = [&](int idx, float best) {
    const int slot = atomicAdd(&hdr->num_candidates, 1);
    if (slot < cap) cands[slot] = Candidate{idx, 0, best, 0, 0ull};
  };
  if (nwin > gridDim.x) {
    const long long nw = (long long)gridDim.x * (kWindowThreads / 32);
    for (long long i = (long long)blockIdx.x * (kWindowThreads / 32) + warp; i < nwin; i += nw) {
      float best = thr;
      int bidx = -1;
      window_best<32>(top, (int)(i * w), (int)min((long long)N, (i + 1) * w), lane, best, bidx);
      if (bidx < 0) continue;
      const bool larger = window_larger<32>(top, max(0, bidx - w + 1), (int)min((long long)N, (long long)bidx + w), lane, best);
      if (__any_sync(0xffffffffu, larger)) continue;
      if (lane == 0) keep(bidx, best);
    }
    return;
  }
  __shared__ float s_best[kWindowThreads / 32];
  __shared__ int s_idx[kWindowThreads / 32];
  for (long long i = blockIdx.x; i < nwin; i += gridDim.x) {
    float best = thr;
    int bidx = -1;
    window_best<kWindowThreads>(top, (int)(i * w), (int)min((long long)N, (i + 1) * w), threadIdx.x, best, bidx);
    if (lane == 0) {
      s_best[warp] = best;
      s_idx[warp] = bidx;
    }
    __syncthreads();
    best = s_best[0];
    bidx = s_idx[0];
    for (int k = 1; k < kWindowThreads / 32; ++k) {
      const float ov = s_best[k];
      const int oi = s_idx[k];
      if (oi >= 0 && (bidx < 0 || ov > best || (ov == best && oi < bidx))) {
        best = ov;
        bidx = oi;
      }
    }
    if (bidx < 0) {
      __syncthreads();  // before the next window's writes
      continue;
    }
    const bool larger = window_larger<kWindowThreads>(top, max(0, bidx - w + 1), (int)min((long long)N, (long long)bidx + w),
                                                      threadIdx.x, best);
    if (!__syncthreads_or(larger) && threadIdx.x == 0) keep(bidx, best);
  }
}

// The end of a search's drift recovery: the last of its CTAs to arrive writes the header and
// the first candidates to host memory, a few hundred bytes: two copies of every search's whole
// candidate window stood after the launches before (6 KB per search, at a large pitch).
__device__ void report_results(const SearchDesc& sd) {
  const HostReport& r = sd.report;
  if (!r.hdr) return;
  __shared__ bool last_block;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last_block = atomicAdd(&sd.hdr->ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last_block) return;
  __threadfence();
  const int n = min(min(sd.hdr->num_candidates, sd.cand_cap), r.head);
  const unsigned long long* src = reinterpret_cast<const unsigned long long*>(sd.cands);
  unsigned long long* dst = reinterpret_cast<unsigned long long*>(r.cands);
  static_assert(sizeof(Candidate) == 24 && sizeof(SearchHeader) % 8 == 0, "records of whole 8-byte words");
  for (int i = threadIdx.x; i < 3 * n; i += blockDim.x) dst[i] = __ldcg(src + i);
  const unsigned long long* hs = reinterpret_cast<const unsigned long long*>(sd.hdr);
  if (threadIdx.x < (int)(sizeof(SearchHeader) / 8))
    reinterpret_cast<unsigned long long*>(r.hdr)[threadIdx.x] = __ldcg(hs + threadIdx.x);
  if (threadIdx.x == 0 && r.flag_out) *r.flag_out = *r.flag_count;
  if (threadIdx.x < 2 && r.norm_out) r.norm_out[threadIdx.x] = r.norm[threadIdx.x];
}

// One thread per (candidate, path): every eligible path of every surviving channel is
// summed in tree order and folded into the candidate's packed best with atomicMax.
__global__ void resolve_kernel(const __grid_constant__ SearchBatch b) {
  const SearchDesc& sd = b.s[blockIdx.y];
  const float* __restrict__ in = sd.input;
  const long long stride = sd.row_stride;
  const int Tr = sd.Tr, N = sd.N, dmin = sd.dmin, dmax = sd.dmax, cap = sd.cand_cap;
  const SearchHeader* hdr = sd.hdr;
  Candidate* cands = sd.cands;
  const long long n = min(hdr->num_candidates, cap);
  const long long npaths = (long long)(dmax - dmin + 1) * Tr;
  const long long total = n * npaths;
  const int levels = 31 - __clz(Tr);  // Tr is a power of two
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long i = idx / npaths;
    const int p = (int)(idx - i * npaths);
    const long long c = cands[i].index;
    const int db = dmin + p / Tr;
    const int off = p - (p / Tr) * Tr;
    const long long e = (long long)(Tr - 1) * db;
    if (c + e < 0 || c + e + off >= N) continue;
    const float v = path_sum_by16(levels, off, [&](int t, int pos) {
      return __ldg(in + (long long)t * stride + c + (long long)db * t + pos);
    });
    if (v > 0.0f) {  // the reference's top sums start at zero and update on strict >
      const unsigned long long key = ((unsigned long long)float_key(v) << 32) | (unsigned long long)(~(uint32_t)p);
      atomicMax(&cands[i].best, key);
    }
  }
  report_results(sd);
}

__global__ void path_values_kernel(const float* __restrict__ in, long long stride, int Tr, int N,
                                   const int* index, const int* drift_steps, float* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int shift = Tr - 1;
  const int ds = drift_steps[i];
  const int db = (int)floorf((float)ds / (float)shift);
  const int off = ds - db * shift;
  const long long c = index[i];
  const long long first = c, last = c + (long long)db * shift + off;
  if (off < 0 || off >= Tr || first < 0 || first >= N || last < 0 || last >= N) {
    out[i] = __int_as_float(0x7fc00000);
    return;
  }
  out[i] = path_sum_by16(31 - __clz(Tr), off, [&](int t, int pos) {  // Tr is a power of two
    return __ldg(in + (long long)t * stride + c + (long long)db * t + pos);
  });
}

#include "generated/taylor_direct_gen.cuh"

// Up to 16 rows: one thread per (survivor, drift block) computes all Tr offsets of the
// block from the subtree's leaves (taylor_direct_M, the tree's pairing; leaves outside
// [0, N) read as zero, which only ineligible paths touch) and merges its best packed key.
template <int M>
__global__ void resolve_direct_kernel(const __grid_constant__ SearchBatch b) {
  const SearchDesc& sd = b.s[blockIdx.y];
  const float* __restrict__ in = sd.input;
  const long long stride = sd.row_stride;
  const int N = sd.N, dmin = sd.dmin, ndb = sd.dmax - sd.dmin + 1, cap = sd.cand_cap;
  Candidate* cands = sd.cands;
  const long long n = min(sd.hdr->num_candidates, cap);
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n * ndb;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long i = idx / ndb;
    const int j = (int)(idx - i * ndb);
    const int db = dmin + j;
    const long long c = cands[i].index;
    const long long e = (long long)(M - 1) * db;
    if (c + e < 0) continue;  // no offset of this drift block is eligible
    auto ld = [&](int t, int pos) {
      const long long x = c + (long long)db * t + pos;
      return (x >= 0 && x < N) ? __ldg(in + t * stride + x) : 0.0f;
    };
    float out[M];
    if constexpr (M == 16) taylor_direct_16(ld, out);
    else if constexpr (M == 8) taylor_direct_8(ld, out);
    else if constexpr (M == 4) taylor_direct_4(ld, out);
    else taylor_direct_2(ld, out);
    unsigned long long best = 0;
#pragma unroll
    for (int off = 0; off < M; ++off) {
      if (c + e + off >= N || !(out[off] > 0.0f)) continue;  // eligible, and above the zero start
      const uint32_t p = (uint32_t)(j * M + off);
      const unsigned long long key = ((unsigned long long)float_key(out[off]) << 32) | (unsigned long long)(~p);
      best = key > best ? key : best;
    }
    if (best) atomicMax(&cands[i].best, best);
  }
  report_results(sd);
}

}  // namespace

cudaError_t search_hits_batch(const SearchBatch& b, int num_sms, cudaStream_t stream) {
  if (b.count <= 0) return cudaSuccess;
  long long nwin = 1;
  for (int k = 0; k < b.count; ++k) {
    const long long w = b.s[k].window_size;
    long long n = ((long long)b.s[k].N + w - 1) / w;
    if (n > nwin) nwin = n;
  }
  long long wblocks = nwin;
  const long long wcap = (8ll * num_sms + b.count - 1) / b.count;
  if (wblocks > wcap) wblocks = wcap;
  if (wblocks < 1) wblocks = 1;
  window_kernel<<<dim3((unsigned)wblocks, b.count), kWindowThreads, 0, stream>>>(b);
  int rblocks = (4 * num_sms + b.count - 1) / b.count;
  if (rblocks < 4) rblocks = 4;
  // Drift recovery, one launch per row count: the direct form up to 16 rows, one path per
  // thread beyond.
  for (int R : {2, 4, 8, 16, 0}) {
    SearchBatch q;
    q.count = 0;
    q.maxN = 0;
    for (int k = 0; k < b.count; ++k)
      if (R ? b.s[k].Tr == R : b.s[k].Tr > 16) {
        q.s[q.count++] = b.s[k];
        q.maxN = std::max(q.maxN, b.s[k].N);
      }
    if (!q.count) continue;
    const dim3 grid(rblocks, q.count);
    switch (R) {
      case 2: resolve_direct_kernel<2><<<grid, 128, 0, stream>>>(q); break;
      case 4: resolve_direct_kernel<4><<<grid, 128, 0, stream>>>(q); break;
      case 8: resolve_direct_kernel<8><<<grid, 128, 0, stream>>>(q); break;
      case 16: resolve_direct_kernel<16><<<grid, 128, 0, stream>>>(q); break;
      default: resolve_kernel<<<grid, 256, 0, stream>>>(q); break;
    }
  }
  return cudaGetLastError();
}

cudaError_t path_values(const float* input, long long row_stride, int Tr, int N, const int* index,
                        const int* drift_steps, float* out, int n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  path_values_kernel<<<(n + 127) / 128, 128, 0, stream>>>(input, row_stride, Tr, N, index, drift_steps,
                                                          out, n);
  return cudaGetLastError();
}

}  // namespace scb
