// Column sums and the noise statistics of a search, on the GPU.
//
// The reference copies the column sums to the host and uses std::nth_element for the
// median and the 5% / 95% order statistics, then a mean and standard deviation over the
// sorted positions [ceil(0.05 N), floor(0.95 N)] (dedoppler.cu:242-262).  Here:
//   * colsum_kernel: sumColumns (dedoppler.cu:63-72), same sequential float order.
//   * stats_kernel: everything else, one cluster of CTAs per search, which meet at the cluster's
//     hardware barrier and read one another's shared memory:
//       - the key range [kmin, kmax] of the column sums, cut into 4096 bins; the bin holding
//         each target rank becomes that target's range, and further passes cut it again until
//         the range is one key or holds at most 4096 values, which are then collected and
//         picked from in shared memory.  Exact, and typically two reads of the column sums
//         after the range: one histogram and the collection.  The collection also sums (FP64,
//         as the reference's std::accumulate with a double start) the values between the two
//         percentiles' ranges; the boundary candidates and ties are added exactly and the mean
//         formed with the reference's roundings (float sum, float division);
//       - the variance (searches whose order statistics sit on repeated values are done
//         exactly in the reference's order by dd_order.cu instead).  The reference accumulates
//         (f - m)^2 in FLOAT, one term at a time (dedoppler.cu:257-261).  Once the accumulator
//         is large, every term is rounded to the accumulator's ulp and terms under half an ulp
//         vanish, which biases the sum low (about 4e-4 relative at 2^20 channels, nearly
//         independent of the order).  An exact FP64 variance would therefore differ from the
//         reference's by more than the SNR tolerance.  The float accumulation is reproduced in
//         parallel: an exact prefix sum gives the accumulator A_i each term meets (in channel
//         order), and the term contributes rint(t_i / ulp(float(A_i))) * ulp(float(A_i)).  The
//         result tracks a sequential float sum to about 1e-5 relative; the remaining
//         difference comes from the order (the reference's order is whatever std::nth_element
//         leaves).
// One launch, because what bounds the statistics of one search is not its four reads of 4 MB
// but the launches and last-block hand-overs between them: nine kernels took 92 us at 2^20
// channels and 54 us at 32768, besides the gaps between them; the one takes 70 and 25 us (16
// SMs; at 2^20 channels it is bound by instruction issue and by the cluster's 24 bytes per
// clock and SM from L2).  64 searches of 2^20: 624 -> 395 us, the later reads served by L2.
#include <cooperative_groups.h>

#include <algorithm>
#include <climits>
#include <type_traits>

#include "dd_common.cuh"
#include "dd_internal.h"

namespace scb {

namespace {

namespace cg = cooperative_groups;

constexpr int kSelBins = 4096;     // histogram bins per order-statistic pass
constexpr int kSelCands = 4096;    // candidates collected per order statistic
constexpr int kSelThreads = 512;
constexpr int kSelWarps = kSelThreads / 32;
constexpr int kMaxCluster = 16;

// Column sums of search blockIdx.y (dedoppler.cu:63-72: a float sum in row order).
__global__ void colsum_kernel(const __grid_constant__ SearchBatch b) {
  const SearchDesc& d = b.s[blockIdx.y];
  const float* in = d.input;
  const long long row_stride = d.row_stride;
  const int N = d.N, Tr = d.Tr;
  const bool vec = ((reinterpret_cast<uintptr_t>(in) & 15) == 0) && ((row_stride & 3) == 0) && ((N & 3) == 0);
  if (vec) {
    const int c4 = blockIdx.x * blockDim.x + threadIdx.x;
    if (c4 * 4 >= N) return;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int t = 0; t < Tr; ++t) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(in + (long long)t * row_stride) + c4);
      acc.x += v.x;
      acc.y += v.y;
      acc.z += v.z;
      acc.w += v.w;
    }
    reinterpret_cast<float4*>(d.colsum)[c4] = acc;
  } else {
    const int c_end = min(N, (blockIdx.x + 1) * blockDim.x * 4);
    for (int c = blockIdx.x * blockDim.x * 4 + threadIdx.x; c < c_end; c += blockDim.x) {
      float acc = 0.0f;
      for (int t = 0; t < Tr; ++t) acc += __ldg(in + (long long)t * row_stride + c);
      d.colsum[c] = acc;
    }
  }
}

// Number of bits that hold v (0 for 0).
__device__ __forceinline__ uint32_t bit_width(uint32_t v) { return 32u - (uint32_t)__clz((int)v); }

// Visits x[i0, i1) (i0 a multiple of 8), four at a time where the array allows: fn(values, valid
// mask), with every lane of a warp running the same trip count (for warp-wide
// votes inside fn).  Eight 16-byte loads in flight per thread: with four, a pass over 2^20
// channels took 7.5 us on 16 SMs, all of it waiting for L2.
template <typename Fn>
__device__ __forceinline__ void for_each_value(const float* __restrict__ x, int i0, int i1, Fn fn) {
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const int n4 = vec ? (i1 - i0) / 4 : 0;
  const float4* __restrict__ x4 = reinterpret_cast<const float4*>(x + i0);
  constexpr int K = 8;
  const int whole = n4 / (K * kSelThreads) * (K * kSelThreads);
  for (int i = threadIdx.x; i < whole; i += K * kSelThreads) {
    float4 v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = __ldg(x4 + i + k * kSelThreads);
#pragma unroll
    for (int k = 0; k < K; ++k) fn(v[k], 0xfu);
  }
  for (int i = whole + threadIdx.x; i < (n4 + kSelThreads - 1) / kSelThreads * kSelThreads; i += kSelThreads) {
    const bool in = i < n4;
    fn(in ? __ldg(x4 + i) : make_float4(0.f, 0.f, 0.f, 0.f), in ? 0xfu : 0u);
  }
  const int rest = i1 - i0 - 4 * n4;
  for (int i = 4 * threadIdx.x; i < (rest + 4 * kSelThreads - 1) / (4 * kSelThreads) * (4 * kSelThreads); i += 4 * kSelThreads) {
    float f[4];
    unsigned in = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      f[k] = i + k < rest ? x[i0 + 4 * n4 + i + k] : 0.0f;
      in |= (i + k < rest ? 1u : 0u) << k;
    }
    fn(make_float4(f[0], f[1], f[2], f[3]), in);
  }
}

// sel_key, without the tests of the sign and of -0 where every value is positive.
__device__ __forceinline__ uint32_t key_of(float f, std::true_type) { return __float_as_uint(f) | 0x80000000u; }
__device__ __forceinline__ uint32_t key_of(float f, std::false_type) { return sel_key(f); }

// The ulp of the float that accumulator value a >= 0 rounds to is 2^(exponent - 150), with the
// exponent of the smallest subnormal for 0 (the first add is exact).
__device__ __forceinline__ uint32_t acc_exponent(double a) {
  return max((__float_as_uint(__double2float_rn(a)) >> 23) & 0xffu, 1u);
}
// That ulp and its reciprocal.
__device__ __forceinline__ void float_ulp(double a, double* u, double* inv) {
  const uint32_t e = acc_exponent(a);
  const long long k = (long long)e - 150;  // ulp = 2^k
  *u = e == 255u ? __longlong_as_double(0x7ff8000000000000ll) : __longlong_as_double((1023 + k) << 52);
  *inv = __longlong_as_double((1023 - k) << 52);
}

// The squared deviation the reference adds: (f - m) * (f - m) in float.
__device__ __forceinline__ float var_term(float f, float m) {
  const float d = f - m;
  return __fmul_rn(d, d);
}

__device__ __forceinline__ bool var_inside(float f, float lo, float hi) { return f > lo && f < hi; }

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Exclusive block scan of one unsigned per thread; *total gets the sum (every thread).
__device__ __forceinline__ unsigned block_exclusive(unsigned v, unsigned* warp_tot, unsigned* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  __syncthreads();
  if (lane == 31) warp_tot[warp] = inc;
  __syncthreads();
  unsigned before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kSelWarps; ++w) {
    const unsigned t = warp_tot[w];
    if (w < warp) before += t;
    all += t;
  }
  *total = all;
  return before + inc - v;
}

// One order-statistic target: its range [lo, lo + 2^wshift), its rank inside the range and how
// many values the range holds; mode 0: narrow further, 1: pick from the candidates, 2: one key.
struct SelectTarget {
  uint32_t lo, wshift, rank, count, mode;
};

struct StatsShared {
  unsigned bins[3][kSelBins];  // histograms; then region j holds this CTA's candidates of target j
  uint32_t cand[kSelCands];    // CTA j: target j's candidates of the whole cluster
  SelectTarget target[3], next[3];
  int found[3];
  unsigned ncand[3];           // this CTA's candidates
  uint32_t kmin[kMaxCluster], kmax[kMaxCluster];  // every CTA's range
  unsigned slice[3][kMaxCluster];                 // every CTA's histogram slice total
  uint32_t key[3];
  long long lt[3], eq[3];
  double part[kMaxCluster];                // every CTA's share of the inner sum
  double wsum[kMaxCluster * kSelWarps];    // every warp's sum of squared deviations
  double emu[kMaxCluster];                 // CTA 0: every CTA's emulated share
  unsigned warp_tot[kSelWarps];
  uint32_t warp_min[kSelWarps], warp_max[kSelWarps];
  double red[kSelWarps];
  double inner;
};

// Narrows target j's range to one key with its n candidates in shared memory (CTA j): twelve bits
// per pass over at most kSelCands keys.
__device__ void pick_candidate(StatsShared& S, int j, int n, long long target_rank) {
  SelectTarget t = S.target[j];
  const long long below = target_rank - t.rank;  // values under the target's range
  const uint32_t rank0 = t.rank;
  __shared__ uint32_t s_lo, s_rank, s_count;
  if (t.mode == 1) {
    const uint32_t* keys = S.cand;
    unsigned* h = S.bins[0];  // every CTA has read its candidates from here
    t.rank = min(t.rank, (uint32_t)max(n - 1, 0));  // the rank is below the count; keeps the pick inside
    while (t.wshift > 0) {
      const uint32_t shift = t.wshift > 12u ? t.wshift - 12u : 0u;
      for (int i = threadIdx.x; i < kSelBins; i += kSelThreads) h[i] = 0;
      __syncthreads();
      for (int i = threadIdx.x; i < n; i += kSelThreads) {
        const uint32_t d = keys[i] - t.lo;
        if (keys[i] >= t.lo && (unsigned long long)d < (1ull << t.wshift)) atomicAdd(&h[d >> shift], 1u);
      }
      __syncthreads();
      constexpr int per = kSelBins / kSelThreads;
      unsigned c[per], tot = 0, all;
#pragma unroll
      for (int q = 0; q < per; ++q) tot += c[q] = h[threadIdx.x * per + q];
      unsigned acc = block_exclusive(tot, S.warp_tot, &all);
      if (t.rank >= acc && t.rank < acc + tot) {
#pragma unroll
        for (int q = 0; q < per; ++q) {
          if (t.rank >= acc && t.rank < acc + c[q]) {
            s_lo = t.lo + ((uint32_t)(threadIdx.x * per + q) << shift);
            s_rank = t.rank - acc;
            s_count = c[q];
          }
          acc += c[q];
        }
      }
      __syncthreads();
      t.lo = s_lo;
      t.rank = s_rank;
      t.count = s_count;
      t.wshift = shift;
    }
  }
  cg::cluster_group cl = cg::this_cluster();
  if (threadIdx.x < cl.num_blocks()) {
    StatsShared* o = cl.map_shared_rank(&S, threadIdx.x);
    o->key[j] = t.lo;
    o->lt[j] = below + (rank0 - t.rank);
    o->eq[j] = t.count;
  }
}

// The noise statistics of search blockIdx.y by one cluster: CTA r of C takes the channels
// [r, r + 1) * 16 * wl, its warp w the wl channels from (16 r + w) * wl.  C is at least 4 (the
// three targets' candidates live in CTAs 0 to 2).  min_ties: a search whose most repeated order
// statistic value has at least that many copies leaves the deviation to dd_order.cu.
// MINB: CTAs per SM at least.  A few searches run fastest with all the registers (one CTA per SM:
// 2^20 channels 91 us at 64 registers and 76 with all when the two were compared); more hide one
// another's barriers (64 searches 402 us with two CTAs per SM, 451 with one; 8 of 999424 channels 107 and 131).
template <int MINB>
__global__ void __launch_bounds__(kSelThreads, MINB) stats_kernel(const __grid_constant__ SearchBatch b, int min_ties) {
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  StatsShared& S = *reinterpret_cast<StatsShared*>(dyn_smem);
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), r = (int)cl.block_rank();
  const SearchDesc& sd = b.s[blockIdx.y];
  const float* __restrict__ x = sd.colsum;
  const int N = sd.N;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wl = (int)((((long long)N + C * kSelWarps - 1) / (C * kSelWarps) + 7) & ~7ll);
  const int c0 = (int)min((long long)N, (long long)r * kSelWarps * wl);
  const int c1 = (int)min((long long)N, (long long)(r + 1) * kSelWarps * wl);
  // The tree of a search whose column sums came first may run beside this (dd_exec.cu).
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  cl.sync();  // every CTA of the cluster runs: its shared memory may be written from here on

  // The key range.
  uint32_t kmn = 0xffffffffu, kmx = 0u;
  for_each_value(x, c0, c1, [&](const float4& v, unsigned in) {
    const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint32_t k = sel_key(f[c]);
      if ((in >> c) & 1u) {
        kmn = min(kmn, k);
        kmx = max(kmx, k);
      }
    }
  });
  kmn = __reduce_min_sync(0xffffffffu, kmn);
  kmx = __reduce_max_sync(0xffffffffu, kmx);
  if (lane == 0) {
    S.warp_min[warp] = kmn;
    S.warp_max[warp] = kmx;
  }
  if (tid < 3) S.ncand[tid] = 0;
  for (int i = tid; i < kSelBins; i += kSelThreads) S.bins[0][i] = 0;
  __syncthreads();
  if (tid < C) {
    for (int w = 0; w < kSelWarps; ++w) {
      kmn = min(kmn, S.warp_min[w]);
      kmx = max(kmx, S.warp_max[w]);
    }
    StatsShared* o = cl.map_shared_rank(&S, tid);
    o->kmin[r] = kmn;
    o->kmax[r] = kmx;
  }
  cl.sync();
  kmn = 0xffffffffu;
  kmx = 0u;
  for (int q = 0; q < C; ++q) {
    kmn = min(kmn, S.kmin[q]);
    kmx = max(kmx, S.kmax[q]);
  }
  const bool positive = kmn > 0x80000000u;  // what power is: every column sum above 0
  // Histogram passes.  The first bins the whole range once for the three targets; later ones
  // bin the range that each target still in mode 0 was left with.  Exact: the ranges nest,
  // and a range of width one is the target's key.
  SelectTarget t[3];
#pragma unroll
  for (int j = 0; j < 3; ++j)
    t[j] = SelectTarget{kmn, bit_width(kmx - kmn), (uint32_t)(j == 0 ? sd.first : (j == 1 ? sd.mid : sd.last)), (uint32_t)N, 0u};
  const int per_cta = kSelBins / C;  // bins of this CTA's slice (C divides kSelBins)
  for (bool first = true; t[0].mode == 0 || t[1].mode == 0 || t[2].mode == 0; first = false) {
    // Targets with the same range share a histogram.
    int slot[3], slots = 0;
    uint32_t slo[3] = {0u, 0u, 0u}, sbs[3] = {0u, 0u, 0u};
    unsigned long long swidth[3] = {0ull, 0ull, 0ull};  // 0: nothing is binned there
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      slot[j] = -1;
      if (t[j].mode != 0) continue;
#pragma unroll
      for (int i = 0; i < j; ++i)
        if (slot[i] >= 0 && t[i].lo == t[j].lo && t[i].wshift == t[j].wshift) slot[j] = slot[i];
      if (slot[j] < 0) {
        slot[j] = slots++;
#pragma unroll
        for (int q = 0; q < 3; ++q)
          if (q == slot[j]) {
            slo[q] = t[j].lo;
            sbs[q] = t[j].wshift > 12u ? t[j].wshift - 12u : 0u;  // 2^sbs keys per bin
            swidth[q] = 1ull << t[j].wshift;
          }
      }
    }
    if (!first) {  // the first pass's single histogram was cleared before the range's barrier
      for (int i = tid; i < 3 * kSelBins; i += kSelThreads) (&S.bins[0][0])[i] = 0;
      __syncthreads();
    }
    auto bin = [&](const float4& v, unsigned in, auto n_slots, auto plain) {
      const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t k = key_of(f[c], plain);
#pragma unroll
        for (int q = 0; q < decltype(n_slots)::value; ++q)
          if (((in >> c) & 1u) && k >= slo[q] && (unsigned long long)(k - slo[q]) < swidth[q])
            atomicAdd(&S.bins[q][(k - slo[q]) >> sbs[q]], 1u);
      }
    };
    // The first pass's range holds every value: no range test.
    auto bin_all = [&](const float4& v, unsigned in, auto plain) {
      const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if ((in >> c) & 1u) atomicAdd(&S.bins[0][(key_of(f[c], plain) - slo[0]) >> sbs[0]], 1u);
    };
    if (first && positive)
      for_each_value(x, c0, c1, [&](const float4& v, unsigned in) { bin_all(v, in, std::true_type{}); });
    else if (first)
      for_each_value(x, c0, c1, [&](const float4& v, unsigned in) { bin_all(v, in, std::false_type{}); });
    else
      for_each_value(x, c0, c1, [&](const float4& v, unsigned in) {
        bin(v, in, std::integral_constant<int, 3>{}, std::false_type{});
      });
    cl.sync();
    // This CTA's slice of the bins, summed over the cluster; thread i holds `per` of them.
    const int per = (per_cta + kSelThreads - 1) / kSelThreads;  // 1 or 2 (C >= 4)
    unsigned c[3][2], tot[3], before[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      c[q][0] = c[q][1] = tot[q] = before[q] = 0;
      if (q >= slots) continue;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int bin = tid * per + k;
        if (k < per && bin < per_cta)
          for (int g = 0; g < C; ++g) c[q][k] += cl.map_shared_rank(&S, (r + g) % C)->bins[q][r * per_cta + bin];
      }
      tot[q] = c[q][0] + c[q][1];
      unsigned all;
      before[q] = block_exclusive(tot[q], S.warp_tot, &all);
      if (tid < C) cl.map_shared_rank(&S, tid)->slice[q][r] = all;
    }
    cl.sync();
    // The thread whose bin holds a target's rank sets the target's next range; its CTA tells all.
    if (tid < 3) S.found[tid] = 0;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      if (t[j].mode != 0) continue;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        if (slot[j] != q) continue;
        unsigned at = before[q];
        for (int g = 0; g < r; ++g) at += S.slice[q][g];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const unsigned n = c[q][k];
          if (t[j].rank >= at && t[j].rank < at + n) {
            const uint32_t bin = (uint32_t)(r * per_cta + tid * per + k);
            const SelectTarget u{t[j].lo + (bin << sbs[q]), sbs[q], t[j].rank - at, n,
                                 sbs[q] == 0 ? 2u : (n <= (unsigned)kSelCands ? 1u : 0u)};
            S.next[j] = u;
            S.found[j] = 1;
          }
          at += n;
        }
      }
    }
    __syncthreads();
    if (tid < C) {
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (S.found[j]) cl.map_shared_rank(&S, tid)->target[j] = S.next[j];
    }
    cl.sync();
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (t[j].mode == 0) t[j] = S.target[j];
  }

  // The values of each mode-1 target's range (at most kSelCands each) are listed, each CTA's in
  // its own shared memory and then together in CTA j's, and the values strictly between the
  // first and the last target's ranges are summed in FP64.  The ranges of two targets are
  // equal or disjoint (they refine the same bins).  After the first histogram a range is at
  // most 2^20 keys wide, so each test is one 32-bit unsigned compare.
  const bool disjoint = t[0].lo != t[2].lo;
  const uint32_t in_lo = t[0].lo + (uint32_t)(1ull << t[0].wshift);
  const uint32_t in_len = disjoint ? t[2].lo - in_lo : 0u;
  uint32_t w[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) w[j] = t[j].mode == 1 ? (uint32_t)(1ull << t[j].wshift) : 0u;  // 0: lists nothing
  double acc = 0.0, acc4[4] = {0.0, 0.0, 0.0, 0.0};
  // Targets with the same range share a list.  Nearly every warp read of 128 values holds a
  // candidate (about one value in a hundred is one), so the listing is branch-free: a predicated
  // atomic per value whose result is waited for only by the predicated store, where branches
  // around the atomics would wait for each in turn.
  const int list_of[3] = {0, t[1].lo == t[0].lo ? 0 : 1, t[2].lo == t[0].lo ? 0 : (t[2].lo == t[1].lo ? 1 : 2)};
  const uint32_t w1 = list_of[1] == 1 ? w[1] : 0u, w2 = list_of[2] == 2 ? w[2] : 0u;
  const unsigned count_a = static_cast<unsigned>(__cvta_generic_to_shared(&S.ncand[0]));
  auto list = [&](const float4& v, unsigned in, auto plain) {
    const float f[4] = {v.x, v.y, v.z, v.w};
    uint32_t k[4];
    unsigned at[4];
    int j[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      k[c] = key_of(f[c], plain);
      const bool ok = (in >> c) & 1u;
      acc4[c] += (double)(ok && k[c] - in_lo < in_len ? f[c] : 0.0f);
      const bool p0 = k[c] - t[0].lo < w[0], p1 = k[c] - t[1].lo < w1, p2 = k[c] - t[2].lo < w2;
      j[c] = p1 ? 1 : (p2 ? 2 : 0);
      const unsigned take = ok && (p0 || p1 || p2) ? 1u : 0u;
      at[c] = kSelCands;
      asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p atom.shared.add.u32 %0, [%1], 1;\n}\n"
                   : "+r"(at[c])
                   : "r"(count_a + 4u * (unsigned)j[c]), "r"(take)
                   : "memory");
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (at[c] < (unsigned)kSelCands) S.bins[j[c]][at[c]] = k[c];
  };
  if (positive)
    for_each_value(x, c0, c1, [&](const float4& v, unsigned in) { list(v, in, std::true_type{}); });
  else
    for_each_value(x, c0, c1, [&](const float4& v, unsigned in) { list(v, in, std::false_type{}); });
  acc = (acc4[0] + acc4[1]) + (acc4[2] + acc4[3]);
  acc = warp_sum(acc);
  if (lane == 0) S.red[warp] = acc;
  cl.sync();
  int n_cand = 0;  // of target r, in CTA r
  if (r < 3) {
    // Warp g copies CTA g's list behind the lists of the CTAs before it.
    const int l = r == 0 ? 0 : (r == 1 ? list_of[1] : list_of[2]);
    const int mine = lane < C ? (int)min(cl.map_shared_rank(&S, lane)->ncand[l], (unsigned)kSelCands) : 0;
    int inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    n_cand = min(__shfl_sync(0xffffffffu, inc, 31), kSelCands);  // the range's count
    if (warp < C) {
      const uint32_t* src = cl.map_shared_rank(&S, warp)->bins[l];
      const int m = __shfl_sync(0xffffffffu, mine, warp), to = __shfl_sync(0xffffffffu, inc, warp) - m;
      for (int i = lane; i < m && to + i < kSelCands; i += 32) S.cand[to + i] = src[i];
    }
  }
  cl.sync();
  if (r < 3) pick_candidate(S, r, n_cand, r == 0 ? sd.first : (r == 1 ? sd.mid : sd.last));
  cl.sync();
  const float v_first = key_float(S.key[0]), v_mid = key_float(S.key[1]), v_last = key_float(S.key[2]);
  // The boundary candidates between the percentiles (once when both ends share a range).
  acc = 0.0;
  if ((r == 0 || (r == 2 && disjoint)) && S.target[r].mode == 1) {
    for (int i = tid; i < n_cand; i += kSelThreads) {
      const float f = key_float(S.cand[i]);
      if (f > v_first && f < v_last) acc += (double)f;
    }
  }
  acc = warp_sum(acc);
  if (lane == 0) S.red[warp] += acc;
  __syncthreads();
  if (tid < C) {
    double p = 0.0;
    for (int i = 0; i < kSelWarps; ++i) p += S.red[i];
    cl.map_shared_rank(&S, tid)->part[r] = p;
  }
  cl.sync();
  // The mean over the sorted positions [first, last] as the reference forms it
  // (dedoppler.cu:255-256): a double sum of the floats, rounded to float, divided by the count
  // in float.  Every thread forms it alike.
  const long long n = (long long)sd.last - sd.first + 1;
  double s1;
  long long n_lo, n_hi;
  if (v_first == v_last) {
    s1 = (double)n * v_first;
    n_lo = n;
    n_hi = 0;
  } else {
    // Sorted positions holding v_first are [lt_first, lt_first + eq_first - 1], those
    // holding v_last are [lt_last, lt_last + eq_last - 1]; count the ones in [first, last].
    n_lo = min(S.lt[0] + S.eq[0] - 1, (long long)sd.last) - sd.first + 1;
    n_hi = (long long)sd.last - max(S.lt[2], (long long)sd.first) + 1;
    double inner = 0.0;
    for (int q = 0; q < C; ++q) inner += S.part[q];
    s1 = inner + (double)n_lo * v_first + (double)n_hi * v_last;
  }
  const float sum_f = (float)s1;
  const float m = sum_f / (float)n;
  // How often the most repeated of the three order-statistic values occurs: column sums with
  // many equal values (integer-valued power) are where the order of the float variance sum
  // matters, and those searches take the exact statistics of dd_order.cu.
  const int ties = (int)min(max(S.eq[0], max(S.eq[1], S.eq[2])), (long long)INT_MAX);
  if (r == 0 && tid == 0) {
    SearchHeader* hdr = sd.hdr;
    hdr->median = v_mid;
    hdr->mean = m;
    hdr->ties = ties;
    hdr->order_exact = 0;
  }
  if (ties >= min_ties) return;  // every CTA alike; nothing of another CTA is read after this

  // Exact sums of the terms of the channels strictly between the percentiles, per warp.
  const int b0 = (int)min((long long)N, (long long)(r * kSelWarps + warp) * wl), b1 = min(N, b0 + wl);
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  constexpr int K = 8;  // consecutive channels per lane and step of 256 channels
  constexpr int G = 4;  // steps loaded together
  auto load8 = [&](int i0, float (&v)[K]) {
    if (vec && i0 + K <= b1) {
      const float4 p = __ldg(reinterpret_cast<const float4*>(x + i0));
      const float4 q = __ldg(reinterpret_cast<const float4*>(x + i0) + 1);
      v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w;
      v[4] = q.x; v[5] = q.y; v[6] = q.z; v[7] = q.w;
    } else {
#pragma unroll
      for (int k = 0; k < K; ++k) v[k] = (i0 + k < b1) ? x[i0 + k] : v_first;  // v_first: not inside
    }
  };
#pragma unroll
  for (int g = 0; g < G; ++g) acc4[g] = 0.0;
  for (int i0 = b0 + lane * K; i0 < b1; i0 += G * 32 * K) {
    float v[G][K];
#pragma unroll
    for (int g = 0; g < G; ++g) load8(i0 + g * 32 * K, v[g]);
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int k = 0; k < K; ++k)
        acc4[g] += (double)(var_inside(v[g][k], v_first, v_last) ? var_term(v[g][k], m) : 0.0f);
  }
  acc = (acc4[0] + acc4[1]) + (acc4[2] + acc4[3]);
  acc = warp_sum(acc);
  acc = __shfl_sync(0xffffffffu, acc, 0);
  if (lane < C) cl.map_shared_rank(&S, lane)->wsum[r * kSelWarps + warp] = acc;
  cl.sync();
  // The exact accumulator before this warp's channels, then the emulation, in channel order: a
  // warp scan per 256 channels, each lane walking its 8.
  double base = 0.0;
  for (int i = lane; i < r * kSelWarps + warp; i += 32) base += S.wsum[i];
  base = warp_sum(base);
  base = __shfl_sync(0xffffffffu, base, 0);
  double contrib = 0.0;
  for (int t0 = b0; t0 < b1; t0 += G * 32 * K) {
    float v[G][K];
#pragma unroll
    for (int g = 0; g < G; ++g) load8(t0 + (g * 32 + lane) * K, v[g]);
    // The G steps' sums and scans side by side (they do not depend on the accumulator).
    double tsums[G], incs[G];
    float tmaxs[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      tsums[g] = 0.0;
      tmaxs[g] = 0.0f;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        v[g][k] = var_inside(v[g][k], v_first, v_last) ? var_term(v[g][k], m) : 0.0f;
        tsums[g] += (double)v[g][k];
        tmaxs[g] = fmaxf(tmaxs[g], v[g][k]);
      }
      incs[g] = tsums[g];
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const double y = __shfl_up_sync(0xffffffffu, incs[g], o);
        if (lane >= o) incs[g] += y;
      }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const double tsum = tsums[g], inc = incs[g];
      const float tmax = tmaxs[g];
      double a = base + (inc - tsum);
      const uint32_t e = acc_exponent(a), e_end = acc_exponent(a + tsum);
      // One binade holds the lane's eight sums and every term is below 2^20 of its steps (the
      // float 2^(e - 130)): adding and taking away 1.5 * 2^23 steps rounds a term to whole steps
      // as rint does (ties to even), and the eight roundings add up exactly in float.
      if (e == e_end && e > 23u && e < 250u && tmax < __uint_as_float((e - 3u) << 23)) {
        const float big = __uint_as_float((e << 23) | 0x400000u);
        float c = 0.0f;
#pragma unroll
        for (int k = 0; k < K; ++k) c += __fsub_rn(__fadd_rn(v[g][k], big), big);
        contrib += (double)c;
      } else {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          if (v[g][k] != 0.0f) {
            const double term = (double)v[g][k];
            double u, inv;
            float_ulp(a, &u, &inv);
            contrib += rint(term * inv) * u;
            a += term;
          }
        }
      }
      base += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
  contrib = warp_sum(contrib);
  if (lane == 0) S.red[warp] = contrib;
  __syncthreads();
  if (tid == 0) {
    double p = 0.0;
    for (int i = 0; i < kSelWarps; ++i) p += S.red[i];
    cl.map_shared_rank(&S, 0)->emu[r] = p;
  }
  cl.sync();  // the last use of another CTA's memory
  if (r != 0 || warp != 0) return;
  double exact = 0.0;
  for (int i = lane; i < C * kSelWarps; i += 32) exact += S.wsum[i];
  exact = warp_sum(exact);
  double sum = warp_sum(lane < C ? S.emu[lane] : 0.0);
  if (lane != 0) return;
  // The percentile values themselves (ties at the boundaries), added after the rest.
  const double tlo = (double)var_term(v_first, m), thi = (double)var_term(v_last, m);
  for (long long k = 0; k < n_lo + n_hi; ++k) {
    const double term = (k < n_lo) ? tlo : thi;
    if (term != 0.0) {
      double u, inv;
      float_ulp(exact, &u, &inv);
      sum += rint(term * inv) * u;
    }
    exact += term;
  }
  const float std_dev = sqrtf((float)sum / (float)n);  // dedoppler.cu:262
  sd.hdr->std_dev = std_dev;
  sd.hdr->threshold = (float)(sd.snr_threshold * (double)std_dev + (double)v_mid);  // dedoppler.cu:273
}

}  // namespace

cudaError_t column_sums_batch(const SearchBatch& b, cudaStream_t stream) {
  if (b.count <= 0) return cudaSuccess;
  dim3 cgrid((b.maxN + 4 * 256 - 1) / (4 * 256), b.count);
  colsum_kernel<<<cgrid, 256, 0, stream>>>(b);
  return cudaGetLastError();
}

cudaError_t search_stats_emulated(const SearchBatch& b, int num_sms, int min_ties, cudaStream_t stream) {
  if (b.count <= 0) return cudaSuccess;
  const int smem = (int)sizeof(StatsShared);
  auto kern = b.count <= 4 ? stats_kernel<1> : stats_kernel<2>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  // Sixteen CTAs per search while they fit the SMs side by side, eight for larger batches, and
  // fewer for short rows, whose time is the barriers.  33 clusters of eight run at once (two CTAs per
  // SM): more take four CTAs each instead of a second round, up to 65536 channels (37 searches of 16384
  // 121 -> 88 us, 64 of 65536 256 -> 218, the tree included).  Beyond, a search of many equal values,
  // whose histogram adds queue, holds the others up (one among 48 of 524288: 1.81 ms, with four 1.92).
  int c = b.count * 16 <= num_sms ? 16 : (b.count <= 33 || b.maxN > 65536 ? 8 : 4);
  while (c > 4 && b.maxN <= c * 1024) c /= 2;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(kSelThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  for (;; c /= 2) {
    at[0].val.clusterDim.x = c;
    cfg.gridDim = dim3(c, b.count);
    int clusters = 0;
    if (c <= 8 || (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters > 0)) break;
    cudaGetLastError();  // sixteen CTAs do not fit one cluster here
  }
  return cudaLaunchKernelEx(&cfg, kern, b, min_ties);
}

}  // namespace scb
