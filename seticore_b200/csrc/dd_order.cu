// The noise statistics of a search, bit-identical to the reference's, for the searches whose
// column sums hold repeated values.
//
// The reference copies the column sums to the host and runs (dedoppler.cu:242-262):
//   nth_element(a, a + mid, a + N);  nth_element(a, a + first, a + mid - 1);
//   nth_element(a + mid + 1, a + last, a + N);
//   median = a[mid];  sum = accumulate(a + first, a + last + 1, 0.0)  (double, in order);
//   m = float(sum) / n;  accum (float) += (f - m) * (f - m) over a[first..last] in order;
//   std_dev = sqrt(accum / n),  n = last + 1 - first.
// The float accumulation depends on the order of its terms, which is the permutation that
// std::nth_element leaves; with many equal column sums (integer-valued power) that order
// moves the deviation by a few 1e-4, beyond what the channel-order emulation of dd_stats.cu
// (about 1e-5 on distinct values) can absorb.  For every search whose order statistics sit
// on values held by kExactStatsTies or more column sums, the kernels below reproduce the
// permutation and then both sequential sums exactly, and overwrite the statistics:
//
// * nth_element is libstdc++'s introselect: while the range holds more than 3 values, a
//   median-of-three pivot (__move_median_to_first of positions first+1, mid, last-1) and an
//   unguarded Hoare partition of [first+1, last) against it, then a final insertion sort;
//   at the depth limit 2*floor(log2 n) a heap selection instead (one thread).  The partition swaps the k-th value >= pivot counted from
//   the left with the k-th value <= pivot counted from the right, for as long as the left one
//   lies before the right one.  With cL(x) values >= pivot left of x and cR(x) values <= pivot
//   at or right of x, the number of swapped pairs is K = max_x min(cL(x), cR(x)), and the cut
//   it returns is L[0] for K = 0, else min(L[K], R[K-1]) (L ascending positions of values >=
//   pivot, R descending positions of values <= pivot).  A step is therefore: count both kinds
//   per segment, locate K and the cut, list the K pairs with their values, write them
//   swapped.  Ranges of up to kSmemRange values run in shared memory.
// * A sequential sum: an accumulator A of p significand bits lies on the grid of its binade
//   (multiples of u = ulp(A)).  While the sum stays in that binade, adding a term t moves A by
//   k = q + round(r) grid steps (q + r = |t| / u, sign of t), and only an exact tie (r = 1/2)
//   depends on A itself: round half to even makes the new A even.  So over a chunk of terms
//   the parity of A before each term is a scan of the maps p -> p ^ (k & 1) and p -> 0, and A
//   before each term is a prefix sum of the k.  The first term whose sum would leave the
//   binade is added with a real floating-point add and the scan restarts from the new
//   binade.  The result is the sequential sum, bit for bit.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <type_traits>

#include "dd_common.cuh"
#include "dd_internal.h"

namespace scb {

namespace {

namespace cg = cooperative_groups;

constexpr int kOrdThreads = 1024;
constexpr int kOrdWarps = kOrdThreads / 32;
constexpr int kV4 = 8;                   // float4 groups per lane in one warp step
constexpr int kStep = 32 * 4 * kV4;      // positions per warp step
constexpr int kMaxSegs = kOrderMaxSegs;  // counting segments per partition step
constexpr int kSmemRange = 16384;        // ranges of at most this many values run in shared memory
constexpr int kSmemPairs = kSmemRange / 2 + 1;
constexpr int kSerialRange = 256;        // ranges of at most this many values are finished by one thread
constexpr int kOrderCluster = 16;        // CTAs per search, at most
constexpr int kSideBySide16 = 7, kSideBySide8 = 15, kSideBySide4 = 33;  // clusters that run at once, by CTAs
constexpr int kSumSeg = 4096;            // terms per speculative piece of the float sum
constexpr int kSeqPrefix = 2048;         // leading terms of a sum added one by one (thread 0)
constexpr int kTermsPerThreadF = 16;     // terms per thread in one scan chunk of a float sum
constexpr int kTermsPerThreadD = 8;      // ... of a double sum (two registers per term)
constexpr int kSumChunk = kOrdThreads * kTermsPerThreadF;
constexpr int kSumBuf = kSumChunk + kSumChunk / 16;  // one pad word per 16 terms: conflict-free

// A piece of kSumSeg terms of the float sum, evaluated before the accumulator that meets it is known:
// on the grid of the binade that an approximate prefix sum predicts, the steps it adds and the
// parity it leaves for either parity of the accumulator before it.  Both compose along the terms.
struct SumPiece {
  int eb;       // biased exponent of the predicted accumulator (0: not evaluated)
  int k[2];     // grid steps added for accumulator parity 0 and 1 (saturated: 2^25 is too many)
  int map;      // parity after, as map_then takes it
};
// Shared memory of the kernel beyond the dynamic shared-memory range buffer.
struct OrdShared {
  double warp_d[kOrdWarps], warp_d2[kOrdWarps];
  int seg_ge[kMaxSegs + 1];  // per segment: values >= pivot; then their exclusive prefix
  int seg_le[kMaxSegs + 1];  // per segment: values <= pivot; then their exclusive prefix
  float pivot;
  int total_ge, total_le;
  int cross, K, lk, rk;
  int warp_i[kOrdWarps];
  long long warp_ll[kOrdWarps];
  unsigned warp_map[kOrdWarps];
  long long warp_ll2[kOrdWarps];
  unsigned warp_map2[kOrdWarps];
  // sequential-sum state
  int s_eu;
  long long s_a;
  long long s_cross;
  long long s_a_at_cross;
  int s_slow;
};

// ---------------------------------------------------------------------------------------
// introselect (libstdc++ bits/stl_algo.h), on a range of `a` (global or shared memory)
// ---------------------------------------------------------------------------------------

// __move_median_to_first(result, a, b, c) with comp = operator<.
__device__ void move_median_to_first(float* v, int result, int x, int y, int z) {
  int m;
  if (v[x] < v[y]) {
    if (v[y] < v[z]) m = y;
    else if (v[x] < v[z]) m = z;
    else m = x;
  } else if (v[x] < v[z]) {
    m = x;
  } else if (v[y] < v[z]) {
    m = z;
  } else {
    m = y;
  }
  const float t = v[result];
  v[result] = v[m];
  v[m] = t;
}

// __insertion_sort(first, last): stable, one thread.
__device__ void insertion_sort(float* v, int first, int last) {
  if (first == last) return;
  for (int i = first + 1; i < last; ++i) {
    const float val = v[i];
    if (val < v[first]) {
      for (int j = i; j > first; --j) v[j] = v[j - 1];
      v[first] = val;
    } else {
      int j = i;
      while (val < v[j - 1]) {
        v[j] = v[j - 1];
        --j;
      }
      v[j] = val;
    }
  }
}

// The heap selection libstdc++ falls back to when introselect reaches its depth limit
// (bits/stl_heap.h __push_heap, __adjust_heap, __make_heap; bits/stl_algo.h __heap_select),
// one thread, on f[0..) with comp = operator<.
__device__ void push_heap_(float* f, int hole, int top, float value) {
  int parent = (hole - 1) / 2;
  while (hole > top && f[parent] < value) {
    f[hole] = f[parent];
    hole = parent;
    parent = (hole - 1) / 2;
  }
  f[hole] = value;
}
__device__ void adjust_heap_(float* f, int hole, int len, float value) {
  const int top = hole;
  int second = hole;
  while (second < (len - 1) / 2) {
    second = 2 * (second + 1);
    if (f[second] < f[second - 1]) second--;
    f[hole] = f[second];
    hole = second;
  }
  if ((len & 1) == 0 && second == (len - 2) / 2) {
    second = 2 * (second + 1);
    f[hole] = f[second - 1];
    hole = second - 1;
  }
  push_heap_(f, hole, top, value);
}
__device__ void heap_select_(float* f, int middle, int last) {
  if (middle >= 2) {
    for (int parent = (middle - 2) / 2;; --parent) {
      adjust_heap_(f, parent, middle, f[parent]);
      if (parent == 0) break;
    }
  }
  for (int i = middle; i < last; ++i) {
    if (f[i] < f[0]) {  // __pop_heap(first, middle, i)
      const float value = f[i];
      f[i] = f[0];
      adjust_heap_(f, 0, middle, value);
    }
  }
}

// Exclusive prefix sums of arr[0..n) in place (n <= kMaxSegs), by a block of NT threads;
// arr[n] = the total.  warp_tmp: NT / 32 ints of shared memory.
template <int NT>
__device__ void block_exclusive_scan(int* arr, int n, int* warp_tmp) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int per = (kMaxSegs + NT - 1) / NT;
  constexpr int nw = NT / 32;
  int v[per];
  int tot = 0;
#pragma unroll
  for (int q = 0; q < per; ++q) {
    const int i = tid * per + q;
    v[q] = i < n ? arr[i] : 0;
    tot += v[q];
  }
  int inc = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) warp_tmp[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const int w = lane < nw ? warp_tmp[lane] : 0;
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += y;
    }
    if (lane < nw) warp_tmp[lane] = wi - w;
    if (lane == nw - 1) arr[n] = wi;
  }
  __syncthreads();
  int run = warp_tmp[warp] + inc - tot;
#pragma unroll
  for (int q = 0; q < per; ++q) {
    const int i = tid * per + q;
    if (i < n) arr[i] = run;
    run += v[q];
  }
  __syncthreads();
}

__device__ __forceinline__ int warp_incl_scan(int x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// One warp step: the float4 groups at a0 + 128 q + 4 lane (q < kV4, a0 a multiple of 4)
// that overlap [x0, x1), loaded together (an element's position order is (q, lane, c)).
// The buffers are padded so that a group overlapping the end of a range stays inside them.
// GLOBAL: from the work array, which the cluster's other CTAs write too (read in L2); else shared.
template <bool GLOBAL>
struct VChunk {
  float4 v[kV4];
  __device__ __forceinline__ void load(const float* a, int a0, int x0, int x1) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < kV4; ++q) {
      const int p = a0 + 128 * q + 4 * lane;
      v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p + 3 >= x0 && p < x1) {
        if constexpr (GLOBAL) v[q] = __ldcg(reinterpret_cast<const float4*>(a + p));
        else v[q] = *reinterpret_cast<const float4*>(a + p);
      }
    }
  }
  __device__ __forceinline__ float at(int q, int c) const {
    return c == 0 ? v[q].x : (c == 1 ? v[q].y : (c == 2 ? v[q].z : v[q].w));
  }
  // 4-bit masks of this lane's group q: values >= p (ge) and <= p (le) inside [x0, x1).
  __device__ __forceinline__ void masks(int q, int a0, int x0, int x1, float p, unsigned& mg, unsigned& ml) const {
    if (a0 >= x0 && a0 + kStep <= x1) {  // a whole step inside: no position tests
      mg = ml = 0u;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float f = at(q, c);
        mg |= (!(f < p) ? 1u : 0u) << c;
        ml |= (!(p < f) ? 1u : 0u) << c;
      }
      return;
    }
    const int base = a0 + 128 * q + 4 * (int)(threadIdx.x & 31);
    mg = ml = 0u;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const bool in = base + c >= x0 && base + c < x1;
      const float f = at(q, c);
      mg |= (in && !(f < p) ? 1u : 0u) << c;
      ml |= (in && !(p < f) ? 1u : 0u) << c;
    }
  }
};

// Segments of a partition step over [s, e): aligned windows of seglen positions from
// A0 = s rounded down to a multiple of 4, clipped to [s, e).
struct Segs {
  int s, e, A0, seglen, nseg;
  __device__ __forceinline__ Segs(int s_, int e_) : s(s_), e(e_), A0(s_ & ~3) {
    const int span = e - A0;
    const int steps = (span + kStep - 1) / kStep;
    seglen = ((steps + kMaxSegs - 1) / kMaxSegs) * kStep;
    nseg = (span + seglen - 1) / seglen;
  }
  __device__ __forceinline__ int start(int g) const { return A0 + g * seglen; }  // aligned
  __device__ __forceinline__ int x0(int g) const { return max(s, start(g)); }
  __device__ __forceinline__ int x1(int g) const { return min(e, start(g) + seglen); }
};

// Position of the value of rank r (0-based, in position order) among the values of one kind
// in segment g; every lane gets it.  The caller guarantees the segment holds it.
template <bool GLOBAL>
__device__ int find_rank(const float* a, const Segs& sg, int g, float p, bool kind_ge, int r) {
  const int lane = threadIdx.x & 31;
  const int x0 = sg.x0(g), x1 = sg.x1(g);
  for (int a0 = sg.start(g); a0 < x1; a0 += kStep) {
    VChunk<GLOBAL> w;
    w.load(a, a0, x0, x1);
#pragma unroll
    for (int q = 0; q < kV4; ++q) {
      unsigned mg, ml;
      w.masks(q, a0, x0, x1, p, mg, ml);
      const unsigned m = kind_ge ? mg : ml;
      const int cnt = __popc(m);
      const int inc = warp_incl_scan(cnt);
      const int tot = __shfl_sync(0xffffffffu, inc, 31);
      if (r < tot) {
        const int ex = inc - cnt;
        const bool mine = r >= ex && r < inc;
        int pos = 0;
        if (mine) {
          unsigned mm = m;
          for (int t = 0; t < r - ex; ++t) mm &= mm - 1u;
          pos = a0 + 128 * q + 4 * lane + __ffs((int)mm) - 1;
        }
        const int src = __ffs((int)__ballot_sync(0xffffffffu, mine)) - 1;
        return __shfl_sync(0xffffffffu, pos, src);
      }
      r -= tot;
    }
  }
  return INT_MAX;  // not reached when the caller's rank is inside the segment
}

// The parts of __unguarded_partition_pivot(first, last) over a[first, last), pivot p already moved to
// `first`.  A step in shared memory runs them by one block; a step over more values shares parts
// 1, 3 and 4 among the CTAs of the cluster.
//
// 1. Per segment, the values >= p and <= p; warp w of nw takes segments w, w + nw, ...
template <bool GLOBAL>
__device__ void count_segments(const float* a, const Segs& sg, float p, int w0, int nw, int* seg_ge, int* seg_le) {
  const int lane = threadIdx.x & 31;
  for (int g = w0; g < sg.nseg; g += nw) {
    const int x0 = sg.x0(g), x1 = sg.x1(g);
    int cge = 0, cle = 0;
    for (int a0 = sg.start(g); a0 < x1; a0 += kStep) {
      VChunk<GLOBAL> w;
      w.load(a, a0, x0, x1);
      if (a0 >= x0 && a0 + kStep <= x1) {
#pragma unroll
        for (int q = 0; q < kV4; ++q)
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            cge += w.at(q, c) < p ? 0 : 1;
            cle += p < w.at(q, c) ? 0 : 1;
          }
        continue;
      }
#pragma unroll
      for (int q = 0; q < kV4; ++q) {
        unsigned mg, ml;
        w.masks(q, a0, x0, x1, p, mg, ml);
        cge += __popc(mg);
        cle += __popc(ml);
      }
    }
    cge = __reduce_add_sync(0xffffffffu, cge);
    cle = __reduce_add_sync(0xffffffffu, cle);
    if (lane == 0) {
      seg_ge[g] = cge;
      seg_le[g] = cle;
    }
  }
}

// 2. One block, the counts in S.seg_ge and S.seg_le: their exclusive prefixes in place, S.K pairs, and
// the cut (returned).
template <bool GLOBAL>
__device__ int scan_and_cut(const float* a, const Segs& sg, float p, OrdShared& S) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nseg = sg.nseg;
  if (tid == 0) S.cross = 0;
  block_exclusive_scan<kOrdThreads>(S.seg_ge, nseg, S.warp_i);
  block_exclusive_scan<kOrdThreads>(S.seg_le, nseg, S.warp_i);
  const int total_ge = S.seg_ge[nseg], total_le = S.seg_le[nseg];
  // The segment where cL stops being <= cR: the last segment g whose start has
  // cL = seg_ge[g] <= cR = total_le - seg_le[g] (segment 0 always qualifies).
  for (int g = tid; g < nseg; g += kOrdThreads)
    if (S.seg_ge[g] <= total_le - S.seg_le[g]) atomicMax(&S.cross, g);
  __syncthreads();
  // K = max over positions x of the crossing segment of min(cL(x), cR(x)) (warp 0).
  if (warp == 0) {
    const int g = S.cross;
    const int x0 = sg.x0(g), x1 = sg.x1(g);
    int cl = S.seg_ge[g], cr = total_le - S.seg_le[g];
    int best = 0;
    for (int a0 = sg.start(g); a0 < x1; a0 += kStep) {
      VChunk<GLOBAL> w;
      w.load(a, a0, x0, x1);
#pragma unroll
      for (int q = 0; q < kV4; ++q) {
        unsigned mg, ml;
        w.masks(q, a0, x0, x1, p, mg, ml);
        const int packed = __popc(mg) | (__popc(ml) << 16);
        const int inc = warp_incl_scan(packed);
        const int ex = inc - packed;
        const int base = a0 + 128 * q + 4 * lane;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const unsigned below = (1u << c) - 1u;
          if (base + c >= x0 && base + c < x1)
            best = max(best, min(cl + (ex & 0xffff) + __popc(mg & below), cr - (ex >> 16) - __popc(ml & below)));
        }
        const int tot = __shfl_sync(0xffffffffu, inc, 31);
        cl += tot & 0xffff;
        cr -= tot >> 16;
      }
    }
    best = max(best, min(cl, cr));  // the position after the segment
    best = __reduce_max_sync(0xffffffffu, best);
    if (lane == 0) S.K = best;
  }
  __syncthreads();
  const int K = S.K;
  // L[K] (warp 0) and R[K-1] (warp 1): the segment holding the rank, then a scan of it.
  if (warp < 2) {
    const bool kind_ge = warp == 0;
    const int* pre = kind_ge ? S.seg_ge : S.seg_le;
    const int rank = kind_ge ? K : total_le - K;  // ascending rank among values of that kind
    const bool exists = kind_ge ? K < total_ge : K >= 1;
    int pos = INT_MAX;
    if (exists) {
      int lo = 0, hi = nseg - 1;  // the last segment g with pre[g] <= rank
      while (lo < hi) {
        const int m = (lo + hi + 1) >> 1;
        if (pre[m] <= rank) lo = m;
        else hi = m - 1;
      }
      pos = find_rank<GLOBAL>(a, sg, lo, p, kind_ge, rank - pre[lo]);
    }
    if (lane == 0) {
      if (kind_ge) S.lk = pos;
      else S.rk = pos;
    }
  }
  __syncthreads();
  return K == 0 ? S.lk : min(S.lk, S.rk);
}

// 3. The K pairs: positions and values, listed by rank.  seg_ge, seg_le: the prefixes.  A warp takes
// 32 consecutive positions at a time, so the ranks come from two ballots and neighbouring lanes
// store to neighbouring places (four positions per lane, with scans and scattered stores, took
// 2.4 times as long on 2^20 values).
template <bool GLOBAL>
__device__ void list_pairs(const float* a, const Segs& sg, float p, int K, int total_le, const int* seg_ge,
                           const int* seg_le, int w0, int nw, int* lpos, float* lval, int* rpos, float* rval) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  auto pre = [](const int* s, int g) {
    if constexpr (GLOBAL) return __ldcg(s + g);
    else return s[g];
  };
  constexpr int B = 16;  // loads in flight per lane
  for (int g = w0; g < sg.nseg; g += nw) {
    int rge = pre(seg_ge, g), rle = total_le - 1 - pre(seg_le, g);  // the next ranks (from the right for rle)
    if (rge >= K && total_le - pre(seg_le, g + 1) >= K) continue;  // no pair has a value in this segment
    const int x0 = sg.x0(g), x1 = sg.x1(g);
    for (int b0 = x0; b0 < x1; b0 += 32 * B) {
      float v[B];
#pragma unroll
      for (int k = 0; k < B; ++k) {
        const int i = b0 + 32 * k + lane;
        v[k] = 0.0f;
        if (i < x1) {
          if constexpr (GLOBAL) v[k] = __ldcg(a + i);
          else v[k] = a[i];
        }
      }
#pragma unroll
      for (int k = 0; k < B; ++k) {
        const int i = b0 + 32 * k + lane;
        const bool in = i < x1, ge = in && !(v[k] < p), le = in && !(p < v[k]);
        const unsigned mg = __ballot_sync(0xffffffffu, ge), ml = __ballot_sync(0xffffffffu, le);
        const int r = rge + __popc(mg & below), rd = rle - __popc(ml & below);
        if (ge && r < K) {
          lpos[r] = i;
          lval[r] = v[k];
        }
        if (le && rd < K) {
          rpos[rd] = i;
          rval[rd] = v[k];
        }
        rge += __popc(mg);
        rle -= __popc(ml);
      }
    }
  }
}

// 4. The swaps: the k-th value >= p goes where the k-th value <= p was, and back; thread t of nt.
template <bool GLOBAL>
__device__ void swap_pairs(float* a, int K, int t, int nt, const int* lpos, const float* lval, const int* rpos,
                           const float* rval) {
  auto at = [](const auto* p) {
    if constexpr (GLOBAL) return __ldcg(p);
    else return *p;
  };
  for (int k0 = t; k0 < K; k0 += 4 * nt) {
    int i[4], j[4];
    float vi[4], vj[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = k0 + u * nt;
      if (k < K) {
        i[u] = at(lpos + k);
        j[u] = at(rpos + k);
        vi[u] = at(lval + k);
        vj[u] = at(rval + k);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (k0 + u * nt < K) {
        a[i[u]] = vj[u];
        a[j[u]] = vi[u];
      }
    }
  }
}

// __unguarded_partition_pivot(first, last) over a[first, last) in shared memory, block-wide:
// returns the cut.  The lists hold at least (last - first) / 2 + 1 entries.
__device__ int partition_step(float* a, int first, int last, int* lpos, float* lval, int* rpos, float* rval, OrdShared& S) {
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    move_median_to_first(a, first, first + 1, first + (last - first) / 2, last - 1);
    S.pivot = a[first];
  }
  __syncthreads();
  const float p = S.pivot;
  const Segs sg(first + 1, last);
  count_segments<false>(a, sg, p, warp, kOrdWarps, S.seg_ge, S.seg_le);
  __syncthreads();
  const int cut = scan_and_cut<false>(a, sg, p, S);
  const int K = S.K;
  if (K == 0) return cut;
  list_pairs<false>(a, sg, p, K, S.seg_le[sg.nseg], S.seg_ge, S.seg_le, warp, kOrdWarps, lpos, lval, rpos, rval);
  __syncthreads();
  swap_pairs<false>(a, K, tid, kOrdThreads, lpos, lval, rpos, rval);
  __syncthreads();
  return cut;
}

// Introselect's partition steps on [fr, lr) by one thread, in shared memory, until the range holds at
// most 3 values, the depth budget is spent or the range is bad (the caller's cut check).
__device__ void small_steps(float* v, int& fr, int& lr, int nr, int& depth, bool* bad) {
  while (lr - fr > 3 && depth > 0) {
    --depth;
    move_median_to_first(v, fr, fr + 1, fr + (lr - fr) / 2, lr - 1);
    const float p = v[fr];
    // __unguarded_partition(fr + 1, lr, pivot): the pivot bounds both scans.
    int i = fr + 1, j = lr;
    for (;;) {
      while (i < lr && v[i] < p) ++i;
      --j;
      while (j > fr && p < v[j]) --j;
      if (!(i < j)) break;
      const float t = v[i];
      v[i] = v[j];
      v[j] = t;
      ++i;
    }
    if (i <= fr || i >= lr) {
      *bad = true;
      return;
    }
    if (i <= nr) fr = i;
    else lr = i;
  }
}

// The rest of std::nth_element(a + first, a + nth, a + last) as libstdc++ runs it, one block, from the
// range and depth budget that the cluster's steps left: at most kSmemRange values, which move
// to shared memory (sdata, slists), or a spent budget.  Partition steps while the range holds
// more than 3 values; at the depth limit a heap selection of [first, nth] and a swap of
// a[first] with a[nth]; else a final insertion sort.  A cut outside (first, last) -- impossible
// for a correct partition -- stops the selection and sets *bad, so that no later access
// leaves the range.
__device__ void introselect_from(float* a, int first, int nth, int last, int depth, float* sdata, int* slists, OrdShared& S,
                                 bool* bad) {
  if (first == last || nth == last) return;
  const int f0 = first, n = last - first;
  if (n > kSmemRange) {  // the depth budget is spent
    if (threadIdx.x == 0) {
      heap_select_(a + first, nth + 1 - first, last - first);
      const float t = a[first];
      a[first] = a[nth];
      a[nth] = t;
    }
    __syncthreads();
    return;
  }
  for (int i = threadIdx.x; i < n; i += kOrdThreads) sdata[i] = __ldcg(a + f0 + i);
  __syncthreads();
  int fr = 0, lr = n;
  const int nr = nth - f0;
  while (lr - fr > kSerialRange && depth > 0) {
    --depth;
    const int cut = partition_step(sdata, fr, lr, slists, reinterpret_cast<float*>(slists + kSmemPairs),
                                   slists + 2 * kSmemPairs, reinterpret_cast<float*>(slists + 3 * kSmemPairs), S);
    if (cut <= fr || cut >= lr) {
      *bad = true;
      break;
    }
    if (cut <= nr) fr = cut;
    else lr = cut;
  }
  if (threadIdx.x == 0 && !*bad) {
    small_steps(sdata, fr, lr, nr, depth, bad);
    if (*bad) {
      S.K = -1;
    } else {
      if (lr - fr > 3) {  // the depth budget is spent
        heap_select_(sdata + fr, nr + 1 - fr, lr - fr);
        const float t = sdata[fr];
        sdata[fr] = sdata[nr];
        sdata[nr] = t;
      } else {
        insertion_sort(sdata, fr, lr);
      }
      S.K = 0;
    }
  }
  __syncthreads();
  if (!*bad && S.K < 0) *bad = true;
  for (int i = threadIdx.x; i < n; i += kOrdThreads) a[f0 + i] = sdata[i];
  __syncthreads();
}

// ---------------------------------------------------------------------------------------
// Exact sequential sums
// ---------------------------------------------------------------------------------------

template <typename Acc>
struct AccTraits;
template <>
struct AccTraits<float> {
  static constexpr int P = 24;       // significand bits
  static constexpr int EMIN = -149;  // exponent of the grid of the subnormals
};
template <>
struct AccTraits<double> {
  static constexpr int P = 53;
  static constexpr int EMIN = -1074;
};

// S = A * 2^eu with A on the grid of S's binade (|A| < 2^P).
template <typename Acc>
__device__ void acc_split(Acc S, int* eu, long long* A) {
  using T = AccTraits<Acc>;
  int ex = 0;
  if (S != Acc(0)) frexp(S, &ex);
  int e = ex - T::P;  // floor(log2|S|) - (P - 1)
  if (S == Acc(0) || e < T::EMIN) e = T::EMIN;
  *eu = e;
  *A = (long long)ldexp(S, -e);
}

// A term (a float value, exactly) against the grid 2^eu of an accumulator of P significand
// bits, packed into one word: q (grid steps of |t|, below 2^(P+2)) in the low P + 2 bits,
// then the rounding class of the remainder (0: none or below half, 1: exactly half, 2:
// above half), the sign, "big" (2^(P+1) steps or more, or not finite: the sum always
// leaves the binade) and "nonzero".
template <int P>
struct Packed {
  using W = typename std::conditional<(P <= 24), uint32_t, uint64_t>::type;
  static constexpr int QB = P + 2;
  static constexpr W QMASK = (W(1) << QB) - 1;
  __device__ static __forceinline__ W make(float t, int eu) {
    const uint32_t b = __float_as_uint(t);
    const W neg = (W)(b >> 31) << (QB + 2);
    const int ex = (b >> 23) & 0xff;
    constexpr W kBig = W(1) << (QB + 3), kNz = W(1) << (QB + 4);
    if (ex == 0xff) return neg | kBig | kNz;
    const uint32_t man = b & 0x7fffffu;
    const uint32_t M = ex ? (man | 0x800000u) : man;
    if (M == 0) return neg;
    const int et = ex ? ex - 150 : -149;
    if (et >= eu) {
      const int sh = et - eu;
      if (sh > P - 22) return neg | kBig | kNz;  // M * 2^sh >= 2^(P+1)
      const W q = (W)M << sh;
      return q > (W(1) << (P + 1)) ? (neg | kBig | kNz) : (q | neg | kNz);
    }
    const int s = eu - et;
    if (s > 25) return neg | kNz;  // below a quarter step: rounds to nothing
    const uint32_t rem = M & ((1u << s) - 1u), half = 1u << (s - 1);
    const W cls = rem < half ? 0 : (rem == half ? 1 : 2);
    return (W)(M >> s) | (cls << QB) | neg | kNz;
  }
  __device__ static __forceinline__ long long q(W w) { return (long long)(w & QMASK); }
  __device__ static __forceinline__ int cls(W w) { return (int)((w >> QB) & 3); }
  __device__ static __forceinline__ bool neg(W w) { return (w >> (QB + 2)) & 1; }
  __device__ static __forceinline__ bool big(W w) { return (w >> (QB + 3)) & 1; }
  __device__ static __forceinline__ bool nz(W w) { return (w >> (QB + 4)) & 1; }
  // Grid steps the term adds to an accumulator of parity `par`.
  __device__ static __forceinline__ long long steps(W w, int par) {
    const long long qq = q(w);
    const int c = cls(w);
    const long long k = qq + (c == 2 ? 1 : (c == 1 ? ((par ^ (int)(qq & 1)) & 1) : 0));
    return neg(w) ? -k : k;
  }
  // The parity map of the term: p -> p ^ (k & 1), or p -> 0 for a tie (round half to even).
  __device__ static __forceinline__ unsigned pmap(W w) {
    const int c = cls(w);
    if (c == 1) return 0u;
    return ((c == 2) ^ (int)(q(w) & 1)) ? 1u : 2u;
  }
};

// Parity maps p -> (m >> p) & 1, two bits; composition "first f, then g".
__device__ __forceinline__ unsigned map_then(unsigned f, unsigned g) {
  return ((g >> (f & 1)) & 1) | (((g >> ((f >> 1) & 1)) & 1) << 1);
}

// The terms of v[pos, end) (at most kOrdThreads * TPT of them), staged in shared memory:
// term i - pos at sbuf[r + (r >> 4)], r = i - pos (a pad word per 16 keeps a thread's run of
// consecutive terms free of bank conflicts).  Loads are coalesced and all in flight at once.
template <int TPT, typename TermFn>
__device__ __forceinline__ void stage_terms(const float* __restrict__ v, long long pos, long long end, TermFn term,
                                            float* sbuf) {
  float tv[TPT];
#pragma unroll
  for (int k = 0; k < TPT; ++k) {
    const long long i = pos + threadIdx.x + (long long)k * kOrdThreads;
    tv[k] = i < end ? __ldcg(v + i) : 0.0f;
  }
#pragma unroll
  for (int k = 0; k < TPT; ++k) {
    const int r = threadIdx.x + k * kOrdThreads;
    if (pos + r < end) sbuf[r + (r >> 4)] = term(tv[k]);
  }
}

// The first terms of a sum, [lo, min(hi + 1, lo + kSeqPrefix)), added one by one into s_sum (shared)
// from 0; returns the position after them.
template <typename Acc, typename TermFn>
__device__ long long sequential_start(const float* __restrict__ v, long long lo, long long hi, TermFn term, float* sbuf,
                                      Acc& s_sum) {
  const long long pre_end = min(hi + 1, lo + kSeqPrefix);
  stage_terms<kSeqPrefix / kOrdThreads>(v, lo, pre_end, term, sbuf);
  __syncthreads();
  if (threadIdx.x == 0) {
    Acc acc = Acc(0);
    const int n = (int)(pre_end - lo);
    int r = 0;
    for (; r + 16 <= n; r += 16) {  // one padded run at a time, its loads ahead of its adds
      float t[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) t[k] = sbuf[r + (r >> 4) + k];
#pragma unroll
      for (int k = 0; k < 16; ++k) acc = acc + (Acc)t[k];
    }
    for (; r < n; ++r) acc = acc + (Acc)sbuf[r + (r >> 4)];
    s_sum = acc;
  }
  __syncthreads();
  return pre_end;
}

// Adds term(v[i]) for i in [pos, hi] to s_sum (shared) in index order, rounded after every add as an Acc
// accumulator does.  Block-wide, TPT terms per thread at a time.  sbuf: kSumBuf floats of
// shared memory.
template <typename Acc, int TPT, typename TermFn>
__device__ void sequential_range(const float* __restrict__ v, long long pos, long long hi, TermFn term, float* sbuf,
                                 OrdShared& S, Acc& s_sum) {
  using Tr = AccTraits<Acc>;
  using PK = Packed<Tr::P>;
  using W = typename PK::W;
  constexpr long long CH = (long long)kOrdThreads * TPT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr long long kTop = (1ll << Tr::P) - 1;
  constexpr long long kLow = 1ll << (Tr::P - 1);
  if (tid == 0) S.s_slow = 0;
  __syncthreads();
  while (pos <= hi) {
    const long long chunk_end = min(hi + 1, pos + CH);
    stage_terms<TPT>(v, pos, chunk_end, term, sbuf);
    if (tid == 0) {
      const Acc cur = s_sum;
      if (!isfinite(cur)) {
        S.s_slow = 1;
      } else {
        int eu;
        long long A;
        acc_split(cur, &eu, &A);
        S.s_eu = eu;
        S.s_a = A;
      }
      S.s_cross = LLONG_MAX;
    }
    __syncthreads();
    if (S.s_slow) break;
    const int eu = S.s_eu;
    const long long A0 = S.s_a;
    const long long lowb = eu == Tr::EMIN ? 0 : kLow;
    // This thread's run of consecutive terms, classified once.
    const int r0 = tid * TPT;
    W tm[TPT];
    unsigned fmap = 2u;  // identity: 0 -> 0, 1 -> 1
    bool careful = false;
    // The steps of this thread's terms when no tie needs a parity, saturated at kSat (a
    // double grid step count reaches 2^54 per term; the sum only has to tell whether it
    // stays below 2^P).
    constexpr long long kSat = 1ll << 61;
    long long tfast = 0;
#pragma unroll
    for (int j = 0; j < TPT; ++j) {
      const int r = r0 + j;
      tm[j] = pos + r < chunk_end ? PK::make(sbuf[r + (r >> 4)], eu) : W(0);
      fmap = map_then(fmap, PK::pmap(tm[j]));
      careful |= PK::cls(tm[j]) == 1 || PK::neg(tm[j]) || PK::big(tm[j]);
      tfast = min(tfast + PK::steps(tm[j], 0), kSat);
    }
    // The common chunk: no tie (every step count is fixed), no negative term (the sum only
    // grows) and a total that keeps the sum inside its binade: add the total and move on.
    if (!__syncthreads_or(careful)) {
      long long t = tfast;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t = min(t + __shfl_down_sync(0xffffffffu, t, o), kSat);
      if (lane == 0) S.warp_ll[warp] = t;
      __syncthreads();
      long long total = 0;
#pragma unroll 8
      for (int w = 0; w < kOrdWarps; ++w) total = min(total + S.warp_ll[w], kSat);
      if (A0 + total <= kTop) {
        if (tid == 0) s_sum = (Acc)ldexp((Acc)(A0 + total), eu);
        pos = chunk_end;
        __syncthreads();
        continue;
      }
      __syncthreads();  // a crossing inside the chunk: the full scan below finds it
    }
    // Exclusive scan of the parity maps: the parity before this thread's first term.
    unsigned inc = fmap;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc = map_then(y, inc);
    }
    const unsigned yl = __shfl_up_sync(0xffffffffu, inc, 1);
    const unsigned excl_lane = lane ? yl : 2u;
    if (lane == 31) S.warp_map[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      unsigned wi = S.warp_map[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane >= o) wi = map_then(y, wi);
      }
      const unsigned y = __shfl_up_sync(0xffffffffu, wi, 1);
      S.warp_map2[lane] = lane ? y : 2u;
    }
    __syncthreads();
    const unsigned before = map_then(S.warp_map2[warp], excl_lane);
    const int par0 = (int)((before >> (int)(A0 & 1)) & 1);
    // Steps of this thread's terms, then their exclusive prefix over the block.
    long long tsum = 0;
    {
      int pp = par0;
#pragma unroll
      for (int j = 0; j < TPT; ++j) {
        const long long k = PK::steps(tm[j], pp);
        tsum += k;
        pp = PK::cls(tm[j]) == 1 ? 0 : (pp ^ (int)(k & 1));
      }
    }
    long long incs = tsum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, incs, o);
      if (lane >= o) incs += y;
    }
    if (lane == 31) S.warp_ll[warp] = incs;
    __syncthreads();
    if (warp == 0) {
      long long wi = S.warp_ll[lane];
      const long long w0 = wi;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane >= o) wi += y;
      }
      S.warp_ll2[lane] = wi - w0;
    }
    __syncthreads();
    long long A = A0 + S.warp_ll2[warp] + incs - tsum;
    // The first term whose sum leaves the binade.  A term toward zero may end below it, on a
    // finer grid: it must keep 2^(P-1) steps with a whole step to spare (unless the grid is
    // already the finest); a term away from zero must stay below 2^P steps.
    long long cross = LLONG_MAX, a_at = 0;
    int par = par0;
#pragma unroll
    for (int j = 0; j < TPT; ++j) {
      const long long i = pos + r0 + j;
      if (i >= chunk_end || cross != LLONG_MAX) continue;
      const W w = tm[j];
      const long long k = PK::steps(w, par);
      const long long nA = A + k;
      const long long mag = nA < 0 ? -nA : nA;
      const long long absA = A < 0 ? -A : A;
      const bool toward = PK::nz(w) && A != 0 && (PK::neg(w) != (A < 0));
      if (PK::big(w) || mag > kTop || (toward && absA - PK::q(w) - 1 < lowb)) {
        cross = i;
        a_at = A;
      } else {
        A = nA;
        par = PK::cls(w) == 1 ? 0 : (par ^ (int)(k & 1));
      }
    }
    if (cross != LLONG_MAX) atomicMin(&S.s_cross, cross);
    __syncthreads();
    const long long c = S.s_cross;
    if (c == LLONG_MAX) {
      // the last thread with terms holds the final accumulator
      if (tid == (int)((chunk_end - 1 - pos) / TPT)) s_sum = (Acc)ldexp((Acc)A, eu);
      pos = chunk_end;
    } else {
      if (cross == c) {
        const int r = (int)(c - pos);
        s_sum = (Acc)ldexp((Acc)a_at, eu) + (Acc)sbuf[r + (r >> 4)];
      }
      pos = c + 1;
    }
    __syncthreads();
  }
  if (S.s_slow && tid == 0) {  // a non-finite accumulator: finish one term at a time
    Acc acc = s_sum;
    for (long long i = pos; i <= hi; ++i) acc = acc + (Acc)term(__ldcg(v + i));
    s_sum = acc;
  }
  __syncthreads();
}

// A CTA's share of the double sum of v[lo..hi] in any order: the sum, the sum of magnitudes and the
// lowest set bit of any term (INT_MAX: all zero, INT_MIN: a term is not finite).
struct PlainSum {
  double abs, sum;
  int g, pad;
};
__device__ PlainSum plain_sum(const float* v, long long lo, long long hi, int cta, int ctas, OrdShared& S) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double sa = 0.0, ss = 0.0;
  int g = INT_MAX;
  const long long b0 = lo & ~3ll;  // whole float4 groups from an aligned start
  const long long nt = (long long)ctas * kOrdThreads;
  for (long long i0 = b0 + 4ll * (cta * kOrdThreads + tid); i0 <= hi; i0 += 4ll * 4 * nt) {
    float4 q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long i = i0 + 4ll * u * nt;
      q[u] = i <= hi ? __ldcg(reinterpret_cast<const float4*>(v + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long i = i0 + 4ll * u * nt;
      const float f4[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (i + c < lo || i + c > hi) continue;
        const float f = f4[c];
        const uint32_t b = __float_as_uint(f);
        const int ex = (b >> 23) & 0xff;
        const uint32_t man = b & 0x7fffffu;
        const uint32_t M = ex ? (man | 0x800000u) : man;
        if (ex == 0xff) g = INT_MIN;  // not finite: take the sequential path
        else if (M && g != INT_MIN) g = min(g, (ex ? ex - 150 : -149) + __ffs((int)M) - 1);
        sa += fabs((double)f);
        ss += (double)f;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    sa += __shfl_down_sync(0xffffffffu, sa, o);
    ss += __shfl_down_sync(0xffffffffu, ss, o);
    g = min(g, __shfl_down_sync(0xffffffffu, g, o));
  }
  __syncthreads();
  if (lane == 0) {
    S.warp_d[warp] = sa;
    S.warp_d2[warp] = ss;
    S.warp_i[warp] = g;
  }
  __syncthreads();
  PlainSum r{0.0, 0.0, INT_MAX, 0};
  for (int w = 0; w < kOrdWarps; ++w) {
    r.abs += S.warp_d[w];
    r.sum += S.warp_d2[w];
    r.g = min(r.g, S.warp_i[w]);
  }
  __syncthreads();
  return r;
}
// Every partial sum is a multiple of 2^g, g the lowest set bit of any term, and at most
// sum |v| in magnitude; when that bound is below 2^(52+g) every partial sum is a double, so every
// order of adding gives the exact sum, and a parallel reduction equals the sequential one.
__device__ __forceinline__ bool any_order_is_exact(const PlainSum& p) {
  return p.g == INT_MAX || (p.g != INT_MIN && p.g > -1000 && p.abs < ldexp(1.0, 52 + p.g));
}

constexpr int kPieceSat = 1 << 25;
__device__ __forceinline__ SumPiece then(const SumPiece& f, const SumPiece& g) {
  SumPiece r;
  r.eb = f.eb;
  r.k[0] = min(f.k[0] + ((f.map & 1) ? g.k[1] : g.k[0]), kPieceSat);
  r.k[1] = min(f.k[1] + ((f.map & 2) ? g.k[1] : g.k[0]), kPieceSat);
  r.map = (int)map_then((unsigned)f.map, (unsigned)g.map);
  return r;
}
// One warp: the piece v[pos, end), end - pos <= kSumSeg, on the grid of an accumulator of biased
// exponent eb, each lane a run of consecutive terms.  Lane 0 gets it.  A term that no such
// accumulator keeps in its binade saturates the piece.
template <typename TermFn>
__device__ SumPiece sum_piece(const float* v, long long pos, long long end, int eb, TermFn term) {
  constexpr int kRun = kSumSeg / 32, kU = 16;
  const int lane = threadIdx.x & 31;
  const int n = (int)(end - pos);
  const float scale = __uint_as_float((uint32_t)(277 - eb) << 23);  // 2^(150 - eb): a term in grid steps, exactly
  SumPiece p{eb, {0, 0}, 2};
  for (int r0 = lane * kRun; r0 < (lane + 1) * kRun; r0 += kU) {
    float4 f[kU / 4];
#pragma unroll
    for (int j = 0; j < kU / 4; ++j)  // pos is a multiple of 4; the array is padded to whole groups
      f[j] = r0 + 4 * j < n ? __ldcg(reinterpret_cast<const float4*>(v + pos + r0 + 4 * j)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < kU; ++j) {
      const float4 q4 = f[j / 4];
      const float t = r0 + j < n ? term(j % 4 == 0 ? q4.x : (j % 4 == 1 ? q4.y : (j % 4 == 2 ? q4.z : q4.w))) : 0.0f;
      // Whole steps and the rest, exactly (a term too small to scale exactly is far below half a
      // step); a tie goes to the even sum.  Not a number, or 2^25 steps or more: saturated.
      const float x = t * scale;
      const float w = floorf(x), rest = x - w;
      const int q = x < (float)kPieceSat ? (int)w : kPieceSat;
      const int up = rest > 0.5f ? 1 : 0;
      const bool tie = rest == 0.5f;
      SumPiece s;
      s.k[0] = q + (tie ? (q & 1) : up);
      s.k[1] = q + (tie ? ((q & 1) ^ 1) : up);
      s.map = tie ? 0 : ((s.k[0] & 1) ? 1 : 2);
      p = then(p, s);
    }
  }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {  // neighbouring runs, left then right
    SumPiece y;
    y.k[0] = __shfl_down_sync(0xffffffffu, p.k[0], o);
    y.k[1] = __shfl_down_sync(0xffffffffu, p.k[1], o);
    y.map = __shfl_down_sync(0xffffffffu, p.map, o);
    if ((lane & (2 * o - 1)) == 0) p = then(p, y);
  }
  return p;
}

// ---------------------------------------------------------------------------------------
// One cluster per search
// ---------------------------------------------------------------------------------------
//
// While the range of an nth_element call is larger than kSmemRange, the CTAs of the cluster share
// its partition steps, meeting at the cluster's hardware barrier; the rest of the call is one
// CTA's, in shared memory.  The two calls of the ends touch disjoint ranges and run side by side
// on the cluster's halves.

__device__ __forceinline__ OrderTask* order_tasks(const SearchDesc& sd) {
  return reinterpret_cast<OrderTask*>(sd.lists + order_pair_entries(sd.N));
}

// The pair lists of call t (0: the middle, 1 and 2: the ends): four lists of *big entries.
__device__ __forceinline__ int* task_lists(const SearchDesc& sd, int t, int* big) {
  const int N = sd.N;
  if (t == 0) {
    *big = N / 2 + 1;
    return sd.lists;
  }
  *big = N / 4 + 2;
  return sd.lists + (t == 1 ? 0 : 4 * (N / 4 + 2));
}

// The start of call t's first step or the next one (one thread): if its range is still
// larger than kSmemRange and the depth budget allows, the median of three moves to `first`
// as __unguarded_partition_pivot does, and the step's range is recorded.
__device__ void task_next_step(float* a, OrderTask& T) {
  if (T.error || T.last - T.first <= kSmemRange || T.depth == 0) {
    T.active = 0;
    return;
  }
  --T.depth;
  T.sfirst = T.first;
  T.slast = T.last;
  move_median_to_first(a, T.first, T.first + 1, T.first + (T.last - T.first) / 2, T.last - 1);
  T.pivot = a[T.first];
  T.active = 1;
}

// Call t of a search starts on [first, last) with target nth (std::nth_element returns at
// once when first == last or nth == last).
__device__ void task_init(float* a, OrderTask& T, int first, int nth, int last) {
  T.first = first;
  T.last = last;
  T.nth = nth;
  T.depth = last > first ? 2 * (31 - __clz(last - first)) : 0;
  T.sfirst = T.slast = first;
  T.error = 0;
  T.active = 0;
  if (first == last || nth == last) {
    T.first = T.last;  // nothing to do
    return;
  }
  task_next_step(a, T);
}

// The partition steps of one call by CTAs cta of `ctas` (the first leads), until its range fits
// shared memory.  Every CTA of the cluster runs the same number of barriers: `other` is the call
// that the rest of the cluster works on (or the same one).
__device__ void cluster_steps(cg::cluster_group& cl, const SearchDesc& sd, OrderTask* tasks, int t, int other, int cta,
                              int ctas, OrdShared& S) {
  OrderTask& T = tasks[t];
  OrderTask& O = tasks[other];
  float* a = sd.work;
  int big;
  int* lists = task_lists(sd, t, &big);
  int* lpos = lists;
  float* lval = reinterpret_cast<float*>(lists + big);
  int* rpos = lists + 2 * big;
  float* rval = reinterpret_cast<float*>(lists + 3 * big);
  const int tid = threadIdx.x, w0 = cta * kOrdWarps + (tid >> 5), nw = ctas * kOrdWarps;
  // At most the depth budget of the larger call: each of its steps spends one.
  while (__ldcg(&T.active) || __ldcg(&O.active)) {
    const bool mine = __ldcg(&T.active) != 0;
    const float p = __ldcg(&T.pivot);
    const Segs sg(__ldcg(&T.sfirst) + 1, mine ? __ldcg(&T.slast) : __ldcg(&T.sfirst) + 2);
    if (mine) count_segments<true>(a, sg, p, w0, nw, T.seg_ge, T.seg_le);
    cl.sync();
    if (mine && cta == 0) {
      for (int g = tid; g < sg.nseg; g += kOrdThreads) {
        S.seg_ge[g] = __ldcg(&T.seg_ge[g]);
        S.seg_le[g] = __ldcg(&T.seg_le[g]);
      }
      __syncthreads();
      const int cut = scan_and_cut<true>(a, sg, p, S);
      for (int g = tid; g <= sg.nseg; g += kOrdThreads) {
        T.seg_ge[g] = S.seg_ge[g];
        T.seg_le[g] = S.seg_le[g];
      }
      if (tid == 0) {
        T.K = S.K;
        T.cut = cut;
        if (cut <= T.sfirst || cut >= T.slast) {  // impossible for a correct partition
          T.error = 1;
          T.K = 0;
        } else if (cut <= T.nth) {
          T.first = cut;
        } else {
          T.last = cut;
        }
      }
    }
    cl.sync();
    const int K = mine ? __ldcg(&T.K) : 0;
    if (K > 0)
      list_pairs<true>(a, sg, p, K, __ldcg(&T.seg_le[sg.nseg]), T.seg_ge, T.seg_le, w0, nw, lpos, lval, rpos, rval);
    cl.sync();
    if (K > 0) swap_pairs<true>(a, K, cta * kOrdThreads + tid, ctas * kOrdThreads, lpos, lval, rpos, rval);
    cl.sync();
    if (mine && cta == 0 && tid == 0) {
      __threadfence();
      task_next_step(a, T);
    }
    cl.sync();
  }
}

// One cluster per search whose order statistics sit on repeated values (min_ties copies or more; the
// others leave at once): the column sums permuted as the reference's three nth_element calls
// leave them, then the median, the mean and the deviation exactly as the reference forms them.
//
// As 51 launches (three per partition step, whether a search needed them or not) these cost every
// call 67 to 165 us and a search of 2^20 whole-number column sums 2.0 ms; the one launch costs
// 2 to 5 us and 1.1 ms (partition steps 0.6 ms, bound by their barriers, the lists' scattered
// stores and the leader's scans; the selections' last steps in shared memory 0.25 ms; the sums
// 0.2 ms).
__device__ __forceinline__ void order_search(const SearchDesc& sd) {
  const int N = sd.N;
  __shared__ OrdShared S;
  extern __shared__ __align__(16) float dyn[];
  cg::cluster_group cl = cg::this_cluster();
  const int r = (int)cl.block_rank(), C = (int)cl.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float* sdata = dyn;                                      // kSmemRange values
  int* slists = reinterpret_cast<int*>(dyn + kSmemRange);  // 4 * kSmemPairs entries
  OrderTask* tasks = order_tasks(sd);
  float* a = sd.work;
  // The column sums copied to the work array (16-byte words: both start 16-byte aligned).
  const int n4 = N / 4;
  for (int i = r * kOrdThreads + tid; i < n4; i += C * kOrdThreads)
    reinterpret_cast<float4*>(a)[i] = __ldcg(reinterpret_cast<const float4*>(sd.colsum) + i);
  if (r == 0)
    for (int i = 4 * n4 + tid; i < N; i += kOrdThreads) a[i] = __ldcg(sd.colsum + i);
  cl.sync();
  if (r == 0 && tid == 0) {
    __threadfence();
    task_init(a, tasks[0], 0, sd.mid, N);
  }
  cl.sync();
  cluster_steps(cl, sd, tasks, 0, 0, r, C, S);
  bool bad = false;
  if (r == 0) {
    __threadfence();
    bad = tasks[0].error != 0;
    if (!bad) introselect_from(a, tasks[0].first, sd.mid, tasks[0].last, tasks[0].depth, sdata, slists, S, &bad);
    if (tid == 0) {
      if (bad) {
        atomicExch(&sd.hdr->error, 2);  // the results of this search are invalid
        for (int t = 1; t < 3; ++t) {
          tasks[t].first = tasks[t].last = tasks[t].nth = tasks[t].sfirst = 0;
          tasks[t].active = tasks[t].error = 0;
        }
      } else {
        __threadfence();
        task_init(a, tasks[1], 0, sd.first, sd.mid - 1);
        task_init(a, tasks[2], sd.mid + 1, sd.last, N);
      }
    }
  }
  cl.sync();
  const int half = C / 2, t = r < half ? 1 : 2, cta = r % half;
  cluster_steps(cl, sd, tasks, t, 3 - t, cta, half, S);
  if (cta == 0) {
    __threadfence();
    const OrderTask& T = tasks[t];
    bad = T.error != 0;
    if (!bad) introselect_from(a, T.first, T.nth, T.last, T.depth, sdata, slists, S, &bad);
    if (bad && tid == 0) atomicExch(&sd.hdr->error, 2);
  }
  cl.sync();
  if (*(volatile int*)&sd.hdr->error) return;  // set before the barrier, if at all: every CTA alike

  // float sum = std::accumulate(a + first, a + last + 1, 0.0): a double sum in order.
  const int first = sd.first, last = sd.last, n = last + 1 - first;
  __shared__ PlainSum s_plain[kOrderCluster];
  __shared__ double s_dsum;
  float* sbuf = dyn;  // kSumBuf floats
  {
    const PlainSum p = plain_sum(a, first, last, r, C, S);
    if (tid < C) cl.map_shared_rank(s_plain, tid)[r] = p;
  }
  cl.sync();
  PlainSum tot = s_plain[0];
  for (int q = 1; q < C; ++q) {
    tot.abs += s_plain[q].abs;
    tot.sum += s_plain[q].sum;
    tot.g = min(tot.g, s_plain[q].g);
  }
  if (!any_order_is_exact(tot)) {
    if (r == 0) {
      auto same = [](float f) { return f; };
      const long long pos = sequential_start(a, (long long)first, (long long)last, same, sbuf, s_dsum);
      sequential_range<double, kTermsPerThreadD>(a, pos, (long long)last, same, sbuf, S, s_dsum);
      if (tid < C) *cl.map_shared_rank(&s_dsum, tid) = s_dsum;
    }
    cl.sync();
    tot.sum = s_dsum;
  }
  const float m = __fdiv_rn((float)(tot.g == INT_MAX ? 0.0 : tot.sum), (float)n);
  // accum += (f - m) * (f - m), float, in order: an approximate prefix sum predicts the binade of
  // the accumulator before every piece, the cluster evaluates the pieces on those grids, and
  // one CTA strings them together, taking the pieces that leave their binade term by term.
  auto term = [m](float f) {
    const float d = __fsub_rn(f, m);
    return __fmul_rn(d, d);
  };
  const int base = first & ~3;  // pieces start at multiples of 4, so that they take 16-byte loads
  const int np = (last + 1 - base + kSumSeg - 1) / kSumSeg;
  // In the pair lists' memory (8 bytes per channel): the pieces, then the prefix sums.
  SumPiece* pieces = reinterpret_cast<SumPiece*>(sd.lists);
  double* prefix = reinterpret_cast<double*>(pieces + np);
  for (int c = r * kOrdWarps + warp; c < np; c += C * kOrdWarps) {
    const int c1 = (int)min((long long)last + 1, (long long)base + (c + 1ll) * kSumSeg);
    double acc = 0.0;
    for (int i = max(first, base + c * kSumSeg) + lane; i < c1; i += 32) acc += (double)term(__ldcg(a + i));
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) prefix[c] = acc;
  }
  cl.sync();
  if (r == 0 && warp == 0) {  // exclusive prefix, 32 pieces at a time
    double run = 0.0;
    for (int c0 = 0; c0 < np; c0 += 32) {
      const double v = c0 + lane < np ? __ldcg(prefix + c0 + lane) : 0.0;
      double inc = v;
      for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
      }
      if (c0 + lane < np) prefix[c0 + lane] = run + inc - v;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
  cl.sync();
  for (int c = 1 + r * kOrdWarps + warp; c < np; c += C * kOrdWarps) {  // piece 0 starts from zero: term by term
    const int eb = (int)((__float_as_uint((float)__ldcg(prefix + c)) >> 23) & 0xffu);
    SumPiece p{0, {0, 0}, 2};
    if (eb > 24 && eb < 255)
      p = sum_piece(a, (long long)base + (long long)c * kSumSeg, min((long long)last + 1, (long long)base + (c + 1ll) * kSumSeg),
                    eb, term);
    if (lane == 0) pieces[c] = p;
  }
  cl.sync();
  if (r != 0) return;
  __shared__ float s_sum;
  __shared__ int s_at;
  SumPiece* sp = reinterpret_cast<SumPiece*>(dyn + kSumBuf);  // behind sbuf
  constexpr int kTile = 1024;
  long long pos = sequential_start(a, (long long)first, (long long)last, term, sbuf, s_sum);
  sequential_range<float, kSumSeg / kOrdThreads>(a, pos, min((long long)last, (long long)base + kSumSeg - 1), term, sbuf, S,
                                                 s_sum);
  for (int c0 = 1; c0 < np;) {
    const int cn = min(np, c0 + kTile);
    for (int i = tid; i < cn - c0; i += kOrdThreads) {
      const int4 w = __ldcg(reinterpret_cast<const int4*>(pieces + c0 + i));
      sp[i] = SumPiece{w.x, {w.y, w.z}, w.w};
    }
    __syncthreads();
    for (int c = c0; c < cn;) {
      if (tid == 0) {
        uint32_t u = __float_as_uint(s_sum);
        int at = c;
        for (; at < cn; ++at) {
          const SumPiece& p = sp[at - c0];
          if (p.eb == 0 || p.eb != (int)(u >> 23)) break;  // not evaluated, or another binade
          const int A = (int)((u & 0x7fffffu) | 0x800000u) + p.k[u & 1u];
          if (A > 0xffffff) break;  // leaves the binade
          u = (u & 0x7f800000u) | ((uint32_t)A & 0x7fffffu);
        }
        s_sum = __uint_as_float(u);
        s_at = at;
      }
      __syncthreads();
      c = s_at;
      __syncthreads();
      if (c < cn) {
        const long long p0 = (long long)base + (long long)c * kSumSeg;
        sequential_range<float, kSumSeg / kOrdThreads>(a, p0, min((long long)last, p0 + kSumSeg - 1), term, sbuf, S, s_sum);
        ++c;
      }
    }
    c0 = cn;
  }
  if (tid == 0) {
    const float median = __ldcg(a + sd.mid);
    const float std_dev = sqrtf(__fdiv_rn(s_sum, (float)n));
    SearchHeader* hdr = sd.hdr;
    hdr->median = median;
    hdr->mean = m;
    hdr->std_dev = std_dev;
    hdr->threshold = (float)(sd.snr_threshold * (double)std_dev + (double)median);  // dedoppler.cu:273
    hdr->order_exact = 1;
  }
}

// CHOSEN: the launch acts only where min_tied to max_tied searches of the batch take the reference's
// order.  A second launch, which acts where the first does not, may start beside it and ends after it
// (its first CTA waits; the others leave the SMs to the first launch and to other streams).
template <bool CHOSEN>
__global__ void __launch_bounds__(kOrdThreads, 1)
    order_kernel(const __grid_constant__ SearchBatch b, int min_ties, int min_tied, int max_tied) {
  const SearchDesc& sd = b.s[blockIdx.y];
  if constexpr (CHOSEN) asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  if (sd.N > 0 && sd.hdr->ties >= min_ties && !*(volatile int*)&sd.hdr->error) {  // every CTA of the cluster alike
    bool act = true;
    if constexpr (CHOSEN) {
      const int k = min((int)threadIdx.x, b.count - 1);
      const int tied = __syncthreads_count((int)threadIdx.x < b.count && b.s[k].hdr->ties >= min_ties);
      act = tied >= min_tied && tied <= max_tied;
    }
    if (act) order_search(sd);
  }
  if constexpr (CHOSEN) {
    if (blockIdx.x == 0 && blockIdx.y == 0) asm volatile("griddepcontrol.wait;\n" ::: "memory");
  }
}

}  // namespace

cudaError_t search_stats_exact(const SearchBatch& b, int min_ties, cudaStream_t stream) {
  if (b.count <= 0) return cudaSuccess;
  const int smem = (int)(sizeof(float) * kSmemRange + sizeof(int) * 4 * kSmemPairs);
  static_assert(sizeof(float) * kSumBuf + 1024 * sizeof(SumPiece) <= sizeof(float) * kSmemRange + sizeof(int) * 4 * kSmemPairs,
                "the sum's buffers fit the selection's");
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(kOrdThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  // A CTA fills an SM: 7 clusters of sixteen, 15 of eight, 33 of four and 74 of two run side by side.
  // Sixteen CTAs per search while the batch fits so, and eight while it runs in two turns (64 searches
  // that all leave at once: 8.6 and 5.0 us).  More searches of eight run in turns, most of whose SMs
  // idle in the steps that one CTA does alone, so they take four or two CTAs each (64 searches of
  // whole-number sums: N = 16384 1279 -> 439 us, 131072 2784 -> 1170, 2^20 7363 -> 5906; 33: 773 ->
  // 379, 1680 -> 906, 4091 -> 3288).  Where only a few of a large batch take the order, eight are the
  // faster from 131072 channels on (one of 64 searches of 2^20: 3.4 ms, with two 4.4): two launches then,
  // of which the number that take it picks one; the other costs 1 to 3 us.
  const bool all = min_ties == INT_MIN;  // every search takes the order
  const int small = b.count <= kSideBySide4 ? 4 : 2;
  int c = b.count <= kSideBySide16 ? 16 : 8, wide = kMaxBatch;
  if (b.count > (all ? 1 : 2) * kSideBySide8) {
    if (all || b.maxN <= 65536) c = small;
    else wide = b.maxN >= (1 << 19) && small == 2 ? 2 * kSideBySide8 : kSideBySide8;
  }
  auto kern = wide == kMaxBatch ? order_kernel<false> : order_kernel<true>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  for (;; c /= 2) {
    at[0].val.clusterDim.x = c;
    cfg.gridDim = dim3(c, b.count);
    int clusters = 0;
    if (c <= 8 || (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters > 0)) break;
    cudaGetLastError();
  }
  e = cudaLaunchKernelEx(&cfg, kern, b, min_ties, 1, wide);
  if (e != cudaSuccess || wide == kMaxBatch) return e;
  cfg.numAttrs = 2;
  at[0].val.clusterDim.x = small;
  cfg.gridDim = dim3(small, b.count);
  return cudaLaunchKernelEx(&cfg, kern, b, min_ties, wide + 1, kMaxBatch);
}

namespace {
std::atomic<bool> g_exact_always{false};
}
void set_exact_statistics_always(bool always) { g_exact_always.store(always); }
bool exact_statistics_always() { return g_exact_always.load(); }

int exact_statistics_ties() { return exact_statistics_always() ? INT_MIN : kExactStatsTies; }

cudaError_t search_stats_batch(const SearchBatch& b, int num_sms, cudaStream_t stream) {
  const int min_ties = exact_statistics_ties();
  cudaError_t e = search_stats_emulated(b, num_sms, min_ties, stream);
  if (e == cudaSuccess) e = search_stats_exact(b, min_ties, stream);
  return e;
}

}  // namespace scb
