// Fused Taylor tree + per-channel top path sum (sm_100a).
//
// Replaces, for one search, the reference's per-drift-block loop of optimizedTaylorTree
// (taylor.cu:333-350, tiledTaylorKernel taylor.cu:218-254) followed by findTopPathSums
// (dedoppler.cu:32-55).  One work item is a tile of W = 32*S output channels and a
// chunk of drift blocks ("jobs"):
//
//   1. The CTA stages, once, the union of the tile's sheared windows over all drift
//      blocks of the chunk: row t covers channels [x0 + d0*t, x0 + d1*t + W + R - 1).
//      This trapezoid lives in shared memory; each input value is read from HBM/L2 once
//      per chunk instead of once per drift block.  Float rows arrive by one bulk async copy
//      per row (the TMA engine's cp.async.bulk, completing on an mbarrier; each row from its own
//      16-byte phase) with the ragged edges filled by the threads; 16-bit rows arrive raw the same way, in the second half
//      of the tile, and are converted to float in place.
//   2. Each warp takes (drift block, offset part) units: all offsets of the block for up
//      to 16 rows, one of two halves for 32 rows, and halves in the short-strip form.
//      Lane l streams the channels
//      [x0 + S*l, x0 + S*l + S) through the register-resident Taylor tree generated by
//      gen_taylor_stream.py (a loop of U channels per iteration) and folds every output
//      into a per-channel maximum (root offsets in pairs through their shared left
//      operand, exact by monotonic rounding).  The lane stride S is odd, so the 32 lanes of a warp
//      hit 32 distinct shared-memory banks (for 4- and 2-byte elements).
//   3. The maxima meet in shared memory (atomicMax on the float bits, valid because only
//      positive sums can beat the reference's zero start) and then in the global top
//      array.
//
// The top value per channel equals the reference's: the maximum over eligible paths,
// floored at 0.  A path (db, off) is eligible for start channel c when
// c + (Tr-1)*db >= 0 and c + (Tr-1)*db + off < N: findTopPathSums returns at the first
// offset whose last channel leaves [0, N) (dedoppler.cu:40-46), which for negative
// drift blocks near the low edge skips every offset.  Lanes whose whole strip is
// eligible run the generated code; edge strips run it too but fold only their fully eligible
// channels, and sum the paths of the few partially eligible ones with the lanes of the warp (edge_unit).
//
// The element type E of the input is float (the plain form) or a 16-bit type (the
// precision form's normalised spectra, converted to float as they are staged); sums are
// accumulated in float, in the tree's own pairing -- except in the paired-FP16 form (PAIR) of
// the 16-bit forms' 16-row searches, which stages the paired copy (32-bit words holding the
// FP16 leaves of two drift blocks) and adds both drift blocks with one __hadd2.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "dd_common.cuh"
#include "dd_internal.h"

namespace scb {

// Bulk (TMA) row copies for float rows: one cp.async.bulk per staged row, completing on a
// shared-memory mbarrier.  Both addresses must be 16-byte aligned and the size a multiple
// of 16 bytes.
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(bar));
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(a) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, unsigned bytes) {
  const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(bar));
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(a), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy_row(float* smem_dst, const float* gsrc, unsigned bytes, uint64_t* bar) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  const unsigned b = static_cast<unsigned>(__cvta_generic_to_shared(bar));
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(d),
               "l"(gsrc), "r"(bytes), "r"(b)
               : "memory");
}
// The same with an L2 eviction-priority hint (a createpolicy value).
__device__ __forceinline__ void bulk_copy_row_hint(float* smem_dst, const float* gsrc, unsigned bytes, uint64_t* bar,
                                                   uint64_t policy) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  const unsigned b = static_cast<unsigned>(__cvta_generic_to_shared(bar));
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;\n" ::"r"(d),
      "l"(gsrc), "r"(bytes), "r"(b), "l"(policy)
      : "memory");
}
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}
// Waits for the mbarrier phase with the given parity; false after `tries` polls (the default,
// 2^22, is about a second).
constexpr int kStageWaitTries = 1 << 22;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity, int tries = kStageWaitTries) {
  const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(bar));
  for (int i = 0; i < tries; ++i) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// Merges a non-negative maximum into a CTA-wide per-channel maximum in shared memory.
// Non-negative floats order like their bit patterns as signed integers, so an integer
// atomicMax is a float max here (the values are clamped at 0 by the callers).
__device__ __forceinline__ void fold_max(float* slot, float v) {
  atomicMax(reinterpret_cast<int*>(slot), __float_as_int(v));
}

__device__ __forceinline__ float to_float(float v) { return v; }
__device__ __forceinline__ float to_float(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float to_float(__half v) { return __half2float(v); }

// Element accessor handed to the generated code: row[j] is float j of one staged row, by its
// 32-bit shared-memory address (a register per row where a generic pointer takes two).  The
// load is not volatile, so the compiler may schedule and merge these loads freely; they
// cannot move above the barrier that ends staging because every address depends on the
// row layout read from shared memory after it, and their values feed the atomics on the
// CTA maxima before the next barrier.
struct SharedRow {
  unsigned a;
  __device__ __forceinline__ float operator[](int j) const {
    float v;
    asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a + 4u * (unsigned)j));
    return v;
  }
};

// Paired-FP16 tile: word j of a staged row holds (row value j, row value j + d_step*t) as a
// __half2, the leaves of two consecutive drift blocks at the same strip position.
struct SharedRowPair {
  unsigned a;
  __device__ __forceinline__ __half2 operator[](int j) const {
    unsigned v;
    asm("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a + 4u * (unsigned)j));
    __half2 h;
    memcpy(&h, &v, sizeof(h));
    return h;
  }
};
// One half of a paired tile as floats: the leaves of the low (H = 0) or high (H = 1) drift
// block, for the float code of the band's edges.
template <int H>
struct SharedRowHalf {
  unsigned a;
  __device__ __forceinline__ float operator[](int j) const {
    unsigned v;
    asm("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a + 4u * (unsigned)j));
    __half2 h;
    memcpy(&h, &v, sizeof(h));
    return H ? __high2float(h) : __low2float(h);
  }
};

#include "generated/taylor_stream_gen.cuh"

namespace {

constexpr int kU = 11;      // channels per loop iteration of the generated strip code
constexpr int kIters = 3;   // iterations per strip
constexpr int kStrip = kU * kIters;  // 33 float words per strip: 32 distinct banks


// Collects the root offsets [LO, LO + PART) of one lane's strip in its warp's buffer of
// PART rows of W channels (shared memory); the warp then stores each buffered row to its
// plane as one bulk copy.  The lane's strip starts S words into each row and S is odd, so
// the 32 lanes' stores of one (offset, position) fall in 32 distinct banks.
template <int W>
struct BufferSink {
  unsigned a;  // shared address of row 0 at this lane's first channel
  __device__ __forceinline__ void put(int i, int s, float v) const {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(a + 4u * (unsigned)(i * W + s)), "f"(v) : "memory");
  }
};

// Bulk shared->global stores of whole buffered rows (the async proxy), tracked per issuing
// thread as bulk groups.  Both addresses are 16-byte aligned and the size a multiple of 16.
__device__ __forceinline__ void bulk_store_row(float* gdst, const float* smem_src, unsigned bytes) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem_src));
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(gdst), "r"(s), "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void bulk_store_row_hint(float* gdst, const float* smem_src, unsigned bytes, uint64_t policy) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem_src));
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group.L2::cache_hint [%0], [%1], %2, %3;\n" ::"l"(gdst), "r"(s),
               "r"(bytes), "l"(policy)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
}
// The issuing thread's bulk stores have read their shared source (the buffer may be reused).
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory"); }
// The issuing thread's bulk stores are complete.
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }

// Folds of a strip's per-channel maxima (channel s of the lane's strip at mrow[s]): every
// channel (interior strips), or the channels [lo, hi] whose paths are all eligible (strips at
// the band's edges; the others are finished per path or have no eligible path).
struct FoldAll {
  __device__ __forceinline__ void operator()(float* mrow, int s, float v) const { fold_max(mrow + s, v); }
};
struct FoldRange {
  int lo, hi;
  __device__ __forceinline__ void operator()(float* mrow, int s, float v) const {
    if (s >= lo && s <= hi) fold_max(mrow + s, v);
  }
};
// Paired-FP16 strips: both drift blocks' maxima, or the low one's alone when the high
// drift block lies past the chunk's last (an odd count).  Both halves start at +0 and
// __hmax2 never returns NaN against a number, so the value is >= 0 (or -0, which loses).
struct FoldPair {
  bool hi;
  __device__ __forceinline__ void operator()(float* mrow, int s, __half2 v) const {
    float x = __low2float(v);
    if (hi) x = fmaxf(x, __high2float(v));
    fold_max(mrow + s, x);
  }
};

// Runs the generated strip code of offset part `part` (PART offsets each); the parts are
// unrolled at compile time so that each call site names one generated function.
constexpr int kPacked = -1;  // as RELOAD: the packed form (both halves of the tree in float2 adds)
template <int R, int PART, int U, int ITERS, int RELOAD, int P = 0, typename Row, typename Fold>
__device__ __forceinline__ void strip_part(int part, const Row (&row)[R], float* mrow, const Fold& fold) {
  if constexpr (P * PART < R) {
    if (part == P) {
      if constexpr (RELOAD == kPacked) taylor_strip_x2<R, P * PART, P * PART + PART, U, ITERS>(row, mrow, fold);
      else taylor_strip_loop<R, P * PART, P * PART + PART, U, ITERS, RELOAD>(row, mrow, fold);
    } else strip_part<R, PART, U, ITERS, RELOAD, P + 1>(part, row, mrow, fold);
  }
}

// The sum of one path of R staged rows, in the tree's pairing: row(t) is the row's shared address
// at the path's start channel.
template <int R, typename Row, typename RowAt>
__device__ __forceinline__ float staged_path_sum(int off, RowAt row_at) {
  constexpr int LEVELS = (R >= 32) ? 5 : (R >= 16) ? 4 : (R >= 8) ? 3 : (R >= 4) ? 2 : 1;
  static_assert((1 << LEVELS) == R, "rows are a power of two");
  float v[R];
#pragma unroll
  for (int t = 0; t < R; ++t) {
    // path_pos(off, R, t), unrolled: the bits of t are constants here
    int pos = 0;
#pragma unroll
    for (int m = 0; m < LEVELS; ++m)
      if (t & (1 << m)) pos += ((off >> (LEVELS - 1 - m)) + 1) >> 1;
    v[t] = Row{row_at(t)}[pos];
  }
#pragma unroll
  for (int h = 1; h < R; h *= 2)
#pragma unroll
    for (int t = 0; t + h < R; t += 2 * h) v[t] = v[t] + v[t + h];
  return v[0];
}

// A warp's unit at the band's edges (some lane's strip has paths that leave [0, N);
// dedoppler.cu:40-46: path (db, off) counts for channel c iff c + e >= 0 and c + e + off < N,
// e = (Tr-1)*db).  Channels whose offsets [lo, hi) are all eligible take the generated code with
// a range fold (its other channels read staged zeros or neighbours and are not folded).  The
// fewer than hi - lo channels with some offsets eligible lie side by side in the tile, and the
// warp's lanes share their paths, one path sum at a time each: one lane alone needed 16-row
// sums for up to 120 paths, which whole rounds of CTAs waited for (16 rows, 54 drift blocks:
// 32768 channels 45 -> 27 us, 2^20 channels 258 -> 244 us, eight of them 1887 -> 1785 us).  Channels with no eligible path are skipped.  Out of line, so that its second
// instance of the generated code does not raise the register needs of the interior path.
// tbase: the tile's shared address; Row: the staged element (float, or one half of a pair).
template <typename Row, int R, int PART, int U, int ITERS, int RELOAD>
__device__ __noinline__ void edge_unit(int part, int lo, int hi, unsigned tbase, const int* win, int ks, float* top,
                                       long long x0, long long e, long long base_off, long long N) {
  constexpr int S = U * ITERS;
  const int lane = threadIdx.x & 31;
  // all offsets of channel c eligible iff first <= c <= last_all
  const long long first = -e;
  const long long last_all = N - 1 - e - base_off - (hi - 1);
  const long long cs = x0 + (long long)lane * S;
  const int f_lo = (int)min(max(0ll, first - cs), (long long)S), f_hi = (int)max(min((long long)S - 1, last_all - cs), -1ll);
  if (f_lo <= f_hi) {
    Row row[R];
#pragma unroll
    for (int t = 0; t < R; ++t) row[t].a = tbase + 4u * (unsigned)(lane * S + win[t] + ks * t);
    strip_part<R, PART, U, ITERS, RELOAD>(part, row, top + lane * S, FoldRange{f_lo, f_hi});
  }
  // partially eligible: offsets [lo, lim) with lim = N - c - e - base_off in (lo, hi)
  const long long p_lo = max(max(x0, first), last_all + 1);
  const long long p_hi = min(min(x0 + kWarp * S - 1, N - 1), N - 1 - e - base_off - lo);
  const int n = p_hi >= p_lo ? (int)(p_hi - p_lo + 1) * PART : 0;
  for (int i = lane; i < n; i += kWarp) {
    const int c = (int)(p_lo - x0) + i / PART;  // channel of the tile
    const int r = lo + i % PART;
    if (x0 + c + e + base_off + r >= N) continue;
    const float v = staged_path_sum<R, Row>(r, [&](int t) { return tbase + 4u * (unsigned)(c + win[t] + ks * t); });
    fold_max(top + c, fmaxf(v, 0.0f));
  }
}

// strip_part for the paired-FP16 code.
template <int R, int PART, int U, int ITERS, int RELOAD, int P = 0, typename Row, typename Fold>
__device__ __forceinline__ void strip_part_h2(int part, const Row (&row)[R], float* mrow, const Fold& fold) {
  if constexpr (P * PART < R) {
    if (part == P) taylor_strip_loop_h2<R, P * PART, P * PART + PART, U, ITERS, RELOAD>(row, mrow, fold);
    else strip_part_h2<R, PART, U, ITERS, RELOAD, P + 1>(part, row, mrow, fold);
  }
}

// A launch that started beside the kernel before it (TreeBatch::beside_previous) ends after it.
__device__ __forceinline__ void wait_previous_kernel() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// MAXW: warps per CTA at most; 8 / MAXW CTAs share an SM.
// PAIR: the paired-FP16 tree over the paired copy (the rows are 32-bit words, staged like
// float rows: word j of row t holds the FP16 pair (y[t][j], y[t][j + t]), the leaves of drift
// blocks k and k + 1 side by side), so each warp unit runs two drift blocks with one __hadd2
// per pair of float adds (the taylor_strip_loop_h2 code).
template <typename E, int R, int NPARTS, int S, bool EMIT, int MAXW, int MINB, int RELOAD, bool PAIR = false>
__global__ void __launch_bounds__(MAXW * 32, MINB) tree_max_kernel(const __grid_constant__ TreeBatch tb) {
  static_assert(!PAIR || (std::is_same<E, float>::value && (R == 16 || R == 32) && NPARTS == R / 16 && !EMIT),
                "the paired tree stages 32-bit pair words, 16 or 32 rows in parts of sixteen offsets");
  static_assert(S % kU == 0, "strip length must be a whole number of generated iterations");
  constexpr int ITERS = S / kU;
  constexpr int W = kWarp * S;
  constexpr int LEAD = R - 1;
  constexpr int PART = R / NPARTS;
  constexpr int V = 16 / sizeof(E);  // elements per 16-byte copy
  extern __shared__ __align__(16) float smem[];
  // Per (segment, row) geometry of the staged windows.  Jobs that share their rows
  // (job_row_stride == 0) share one trapezoid segment; otherwise each job has its own.
  __shared__ int geo_base[kMaxSeg][R], geo_win[kMaxSeg][R], geo_wid[kMaxSeg][R];
  __shared__ long long geo_start[kMaxSeg][R];
  __shared__ int item_group, item_tile, item_next;
  // Bulk-copied part of each staged row, as offsets [blo, bhi) from the row's start (float
  // rows only); the threads fill the rest.
  __shared__ int geo_blo[kMaxSeg][R], geo_bhi[kMaxSeg][R];
  __shared__ __align__(8) uint64_t stage_bar;
  __shared__ unsigned item_tx;
  __shared__ int item_floats;  // floats of the item's staged rows (F)
  __shared__ int stage_failed;
  if (threadIdx.x == 0) {
    mbar_init(&stage_bar);
    stage_failed = 0;
  }
  unsigned stage_phase = 0;
  // Maximum form: topS [W] holds the per-channel maxima of the CTA's units (bits as int,
  // >= 0).  Emitting form: the warps' output buffers (MAXW x PART rows of W floats) instead.
  float* topS = smem;
  // The staged rows are float whatever the input type: 16-bit inputs are converted once
  // while staging, so the tree (which reads every staged value about 2 x ndb times) runs
  // the float code.
  float* tile = smem + (EMIT ? MAXW * PART * W : ((W + 3) & ~3));
  if constexpr (!EMIT)
    for (int i = threadIdx.x; i < W; i += blockDim.x) topS[i] = 0.0f;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int nwarps = blockDim.x >> 5;
  // Emitting form: lanes 0..PART-1 of each warp issue the bulk stores of its buffer.
  float* const ebuf = smem + warp * PART * W;
  bool stores_pending = false;
  __shared__ float csum[EMIT ? W : 1];  // tile-major launches: the tile's column sums so far
  const int run = EMIT && tb.tile_major ? tb.count : 1;  // consecutive items a CTA takes
  // Items are taken as CTAs finish: the SMs of a long launch drift apart by a few per cent (64
  // searches of 16 x 2^20: 14.29 -> 13.69 ms; in the BF16 form, 32 of them, 4.89 -> 4.56).  Not for 32 rows, one
  // CTA per SM (8 x 32 x 2^20: 3410 and 3425 us), nor for short strips, whose items are too short.
  constexpr bool kTakes = EMIT || (R <= 16 && S == kStrip);
  int item = blockIdx.x * run;
  while (item < tb.n_items) {
    __syncthreads();  // the previous item is finished with the tile, the layout and item_group
    // The item after this one, asked for by the last warp while warp 0 lays this one out.
    if (kTakes && tb.next_item && threadIdx.x == blockDim.x - 1) {
      const unsigned taken = atomicAdd(tb.next_item, 1u);
      item_next = (int)(gridDim.x + taken);
      if (taken == (unsigned)(tb.n_items - 1)) *tb.next_item = 0;  // one request an item: this is the launch's last
    }
    // Warp 0 decodes the item and lays out the staged rows, one row per lane.
    if (warp == 0) {
      constexpr unsigned kAll = 0xffffffffu;
      int gi = 0;  // the last group whose first item is <= item
      if (run > 1) gi = item % run;
      for (int base = 0; base < (run > 1 ? 0 : tb.count); base += 32) {
        const int i = base + lane;
        const unsigned m = __ballot_sync(kAll, i < tb.count && tb.g[i].item_begin <= item);
        if (m) gi = base + 31 - __clz(m);
      }
      const TreeGroup& pg = tb.g[gi];
      const int local = run > 1 ? item / run : item - pg.item_begin;
      const int lt = local / pg.n_chunks;
      const int tile_i = lt + pg.tile_first;
      if (lane == 0) {
        item_group = gi;
        item_tile = tile_i;
      }
      {
        // Row layout: row t of segment g holds global channels [as, as + wpad), where as is the
        // window's start moved down to the row's last 16-byte boundary: V elements apart, and
        // each row has its own phase, so that rows of any stride and base take the bulk copies
        // (with one phase for all, a row stride that is not a multiple of four floats sent every
        // row through per-thread loads, a memory latency per row: 60 x 100003 with such rows,
        // 1163 -> 900 us a search).  The sheared window of job k (in a
        // shared trapezoid) starts k*t further.  Rows are packed in (segment, row) order:
        // offsets by a warp scan.
        const int k0w = (local - lt * pg.n_chunks) * pg.jobs_per_chunk;
        const int njw = min(pg.jobs_per_chunk, pg.n_jobs - k0w);
        const bool shared_w = (pg.job_row_stride == 0);
        const int nsegw = shared_w ? 1 : njw;
        const int extra = shared_w ? (njw - 1) * pg.d_step : 0;
        const long long x0w = (long long)tile_i * W;
        // The in-range 16-byte chunks of a row take bulk copies; 16-bit rows land raw in the
        // second half of the tile and are converted in place.
        unsigned tx = 0;
        int off = 0;
        for (int e0 = 0; e0 < nsegw * R; e0 += 32) {
          const int e = e0 + lane;
          const bool valid = e < nsegw * R;
          const int gg = valid ? e / R : 0;
          const int t = valid ? e - gg * R : 0;
          int wpad = 0, a = 0;
          long long as = 0;
          if (valid) {
            const long long dg = (long long)pg.d_first + (long long)(k0w + gg) * pg.d_step;
            const long long gs = x0w + dg * t;
            const long long at = (long long)(reinterpret_cast<uintptr_t>(pg.rows) / sizeof(E)) +
                                 (long long)(k0w + gg) * pg.job_row_stride + (long long)t * pg.row_stride;
            const int m = (int)(at & (V - 1));  // channel 0's place in its 16-byte chunk
            as = floor_div(gs + m, V) * V - m;
            a = (int)(gs - as);
            wpad = (a + W + LEAD + extra * t + V - 1) / V * V;
          }
          int incl = wpad;
#pragma unroll
          for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(kAll, incl, d);
            if (lane >= d) incl += y;
          }
          if (valid) {
            const int at = off + incl - wpad;
            geo_base[gg][t] = at;
            geo_win[gg][t] = at + a;
            geo_wid[gg][t] = wpad;
            geo_start[gg][t] = as;
            // whole chunks inside [-pad, N) (rows hold data from -pad on)
            const long long b_lo = as >= -pg.pad ? as : as + (-pg.pad - as + V - 1) / V * V;
            const long long end = as + wpad < pg.N ? as + wpad : pg.N;
            const long long b_hi = end > as ? as + (end - as) / V * V : as;
            const bool bulk = b_hi > b_lo;
            geo_blo[gg][t] = bulk ? (int)(b_lo - as) : 0;
            geo_bhi[gg][t] = bulk ? (int)(b_hi - as) : 0;
            if (bulk) tx += (unsigned)(b_hi - b_lo) * (unsigned)sizeof(E);
          }
          off += __shfl_sync(kAll, incl, 31);
        }
        tx = __reduce_add_sync(kAll, tx);
        if (lane == 0) item_floats = off;
        if (tx) {
          // The tile was last read through ordinary loads; order those before the bulk writes.
          asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
          if (lane == 0) mbar_arrive_expect_tx(&stage_bar, tx);
          __syncwarp();
          for (int e = lane; e < nsegw * R; e += 32) {
            const int gg = e / R, t = e - gg * R;
            const int blo = geo_blo[gg][t], bhi = geo_bhi[gg][t];
            if (bhi > blo) {
              const E* src = static_cast<const E*>(pg.rows) + (long long)(k0w + gg) * pg.job_row_stride +
                             (long long)t * pg.row_stride + geo_start[gg][t] + blo;
              if constexpr (std::is_same<E, float>::value) {
                if (tb.cache_mode == 1)  // stripe passes: the input is read once, do not keep it
                  bulk_copy_row_hint(tile + geo_base[gg][t] + blo, src, (unsigned)(bhi - blo) * 4u, &stage_bar,
                                     policy_evict_first());
                else
                  bulk_copy_row(tile + geo_base[gg][t] + blo, src, (unsigned)(bhi - blo) * 4u, &stage_bar);
              } else {
                // raw element i of the tile (the same index as its float) at byte 2*F + 2*i
                char* dst = reinterpret_cast<char*>(tile) + 2ll * off + 2ll * (geo_base[gg][t] + blo);
                bulk_copy_row(reinterpret_cast<float*>(dst), reinterpret_cast<const float*>(src),
                              (unsigned)(bhi - blo) * (unsigned)sizeof(E), &stage_bar);
              }
            }
          }
        }
        if (lane == 0) item_tx = tx;
      }
    }
    __syncthreads();
    const TreeGroup& p = tb.g[item_group];
    const E* rows = static_cast<const E*>(p.rows);
    const int local = run > 1 ? item / run : item - p.item_begin;
    const int tile_idx = item_tile;
    const int chunk = local - (local / p.n_chunks) * p.n_chunks;
    const long long x0 = (long long)tile_idx * W;
    const int k0 = chunk * p.jobs_per_chunk;
    const int nj = min(p.jobs_per_chunk, p.n_jobs - k0);
    const bool shared_rows = (p.job_row_stride == 0);
    const int nseg = shared_rows ? 1 : nj;
    bool stage_waited = false;  // the 16-bit bulk path waits before its conversion
    if constexpr (std::is_same<E, float>::value) {
      for (int g = 0; g < nseg; ++g) {
        for (int t = 0; t < R; ++t) {
          const int wp = geo_wid[g][t];
          const long long as = geo_start[g][t];
          const E* src = rows + (long long)(k0 + g) * p.job_row_stride + (long long)t * p.row_stride;
          float* dst = tile + geo_base[g][t];
          // the chunks outside the bulk-copied [blo, bhi): left of it, then right of it
          const int blo = geo_blo[g][t], bhi = geo_bhi[g][t];
          const int n_left = blo / V, n_edge = n_left + (wp - bhi) / V;
          for (int q = threadIdx.x; q < n_edge; q += blockDim.x) {
            const int j = q < n_left ? q * V : bhi + (q - n_left) * V;
            const long long c = as + j;
            float* d = dst + j;
            for (int i = 0; i < V; ++i) d[i] = (c + i >= -p.pad && c + i < p.N) ? src[c + i] : 0.0f;
          }
        }
      }
    } else if (item_tx) {
      // 16-bit rows, bulk-copied raw into the second half of the tile (element i at byte
      // 2F + 2i, F the item's floats), then converted in place.  Converting [a, b) writes bytes
      // [4a, 4b) while the raw elements not yet read lie in [2F + 2a, 4F), so b = (F + a) / 2 is
      // the largest safe step: ranges of halving length, a barrier after each, and the last
      // few values (at most four per thread) through registers.
      if (!mbar_wait(&stage_bar, stage_phase, tb.stage_wait_tries >= 0 ? tb.stage_wait_tries : kStageWaitTries))
        stage_failed = 1;
      stage_phase ^= 1u;
      stage_waited = true;
      __syncthreads();
      if (!stage_failed) {
        const int F = item_floats;
        const E* raw = reinterpret_cast<const E*>(reinterpret_cast<const char*>(tile) + 2ll * F);
        int a = 0;
        const int nt = blockDim.x;
        while (F - a > 4 * nt) {
          const int b = a + (F - a) / 2;
          for (int i = a + (int)threadIdx.x; i < b; i += nt) tile[i] = to_float(raw[i]);
          __syncthreads();
          a = b;
        }
        float rv[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int i = a + (int)threadIdx.x + k * nt;
          rv[k] = i < F ? to_float(raw[i]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int i = a + (int)threadIdx.x + k * nt;
          if (i < F) tile[i] = rv[k];
        }
        // the chunks outside each row's bulk-copied [blo, bhi), from global memory
        for (int g = 0; g < nseg; ++g) {
          for (int t = 0; t < R; ++t) {
            const int wp = geo_wid[g][t];
            const long long as = geo_start[g][t];
            const E* src = rows + (long long)(k0 + g) * p.job_row_stride + (long long)t * p.row_stride;
            float* dst = tile + geo_base[g][t];
            const int blo = geo_blo[g][t], bhi = geo_bhi[g][t];
            const int n_left = blo / V, n_edge = n_left + (wp - bhi) / V;
            for (int q = threadIdx.x; q < n_edge; q += blockDim.x) {
              const int j = q < n_left ? q * V : bhi + (q - n_left) * V;
              const long long c = as + j;
              float* d = dst + j;
              for (int i = 0; i < V; ++i) d[i] = (c + i >= 0 && c + i < p.N) ? to_float(src[c + i]) : 0.0f;
            }
          }
        }
      }
    } else {
      // 16-bit rows without a whole chunk in range: zeros and a few ragged values.
      for (int e = warp; e < nseg * R; e += nwarps) {
        const int g = e / R, t = e - g * R;
        const E* src = rows + (long long)(k0 + g) * p.job_row_stride + (long long)t * p.row_stride;
        for (int i = lane; i < geo_wid[g][t]; i += kWarp) {
          const long long c = geo_start[g][t] + i;
          tile[geo_base[g][t] + i] = (c >= 0 && c < p.N) ? to_float(src[c]) : 0.0f;
        }
      }
    }
    if (item_tx && !stage_waited) {
      if (!mbar_wait(&stage_bar, stage_phase, tb.stage_wait_tries >= 0 ? tb.stage_wait_tries : kStageWaitTries))
        stage_failed = 1;
      stage_phase ^= 1u;
    }
    __syncthreads();
    if (stage_failed) {  // every thread leaves together; the results of this launch are invalid
      if (threadIdx.x == 0 && p.status) atomicExch(p.status, 1);
      if (item_tx) mbar_wait(&stage_bar, stage_phase ^ 1u);  // the copies may still be landing (full limit)
      if (EMIT && stores_pending) bulk_wait_all();
      wait_previous_kernel();
      return;
    }

    if constexpr (EMIT) {
      // Column sums across the groups of the tile, in row order: the zero-shear job's window of row
      // t starts at channel x0.
      if (run > 1 && p.colsum) {
        const int gi = item_group;
        for (int i = threadIdx.x; i < W; i += blockDim.x) {
          float acc = gi == 0 ? 0.0f : csum[i];
#pragma unroll
          for (int t = 0; t < R; ++t) acc += tile[geo_win[0][t] + p.colsum_job * p.d_step * t + i];
          csum[i] = acc;
          if (gi == run - 1 && x0 + i < p.N) p.colsum[x0 + i] = acc;
        }
      }
    }
    if constexpr (!EMIT && !PAIR) {
      // Column sums from the staged rows, in row order (bit-identical to sumColumns).
      // The zero-shear job's window of row t starts at channel x0, kz*d_step*t past the
      // chunk's first window (shared rows: one segment).
      const int kz = p.colsum_job - k0;
      if (p.colsum && kz >= 0 && kz < nj) {
        for (int i = threadIdx.x; i < W && x0 + i < p.N; i += blockDim.x) {
          float acc = 0.0f;
#pragma unroll
          for (int t = 0; t < R; ++t) acc += tile[geo_win[0][t] + kz * p.d_step * t + i];
          p.colsum[x0 + i] = acc;
        }
      }
    }
    float* mrow = topS + lane * S;  // this lane's channels
    const long long cs = x0 + (long long)lane * S;  // first channel of this lane's strip
    if constexpr (PAIR) {
      // Units of two drift blocks (k, k + 1) and an offset part, part-major; an odd chunk's
      // last pair folds only its first drift block.
      const unsigned tile_a = static_cast<unsigned>(__cvta_generic_to_shared(tile));
      const unsigned tb0 = tile_a + 4u * (unsigned)(lane * S);
      const int np = (nj + 1) / 2;
      for (int u = warp; u < np * NPARTS; u += nwarps) {
        const int part = u / np;
        const int k = 2 * (u - part * np);
        const int lo = part * PART, hi = lo + PART;
        const bool hi_ok = k + 1 < nj;
        const int ks = k * p.d_step;
        SharedRowPair row[R];
#pragma unroll
        for (int t = 0; t < R; ++t) row[t].a = tb0 + 4u * (unsigned)(geo_win[0][t] + ks * t);
        const long long e0 = (long long)p.elig_T1 * (p.db_first + (long long)(k0 + k) * p.db_step);
        const long long e1 = e0 + (long long)p.elig_T1 * p.db_step;
        const long long b0 = p.off_base + (long long)(k0 + k) * p.off_step;
        const long long b1 = b0 + p.off_step;
        const bool in0 = (cs + e0 >= 0) && (cs + S - 1 + e0 + b0 + hi - 1 <= p.N - 1);
        const bool in1 = !hi_ok || ((cs + e1 >= 0) && (cs + S - 1 + e1 + b1 + hi - 1 <= p.N - 1));
        // One lane at the edge sends the warp's whole unit down the edge path, whose float sums
        // of the FP16 leaves are within the paired tree's bound (closer to the exact sums).
        if (__all_sync(0xffffffffu, in0 && in1)) {
          strip_part_h2<R, PART, kU, ITERS, RELOAD>(part, row, mrow, FoldPair{hi_ok});
        } else {
          constexpr int FR = R == 16 ? 12 : 0;  // the float code's reread threshold
          edge_unit<SharedRowHalf<0>, R, PART, kU, ITERS, FR>(part, lo, hi, tile_a, &geo_win[0][0], ks, topS, x0, e0, b0, p.N);
          if (hi_ok)
            edge_unit<SharedRowHalf<1>, R, PART, kU, ITERS, FR>(part, lo, hi, tile_a, &geo_win[0][0], ks, topS, x0, e1, b1,
                                                                p.N);
        }
      }
    }
    // Part-major order: the CTA's warps run the same offset part (the same generated code)
    // for consecutive drift blocks, so the instruction cache holds one part at a time.
    for (int u = warp; u < (PAIR ? 0 : nj * NPARTS); u += nwarps) {
      const int part = u / nj;
      const int k = u - part * nj;
      const int lo = part * PART;
      const int hi = lo + PART;
      const int g = shared_rows ? 0 : k;
      const int ks = shared_rows ? k * p.d_step : 0;  // extra shear inside a shared trapezoid
      SharedRow row[R];
      {
        const unsigned tb = static_cast<unsigned>(__cvta_generic_to_shared(tile)) + 4u * (unsigned)(lane * S);
#pragma unroll
        for (int t = 0; t < R; ++t) row[t].a = tb + 4u * (unsigned)(geo_win[g][t] + ks * t);
      }

      if constexpr (EMIT) {
        static_assert(R == 16 && S == kU, "the emitting form is generated for 16 rows and short strips");
        // The buffer's previous rows have been read by their bulk stores.
        if (stores_pending) bulk_wait_read();
        __syncwarp();
        BufferSink<W> sink{static_cast<unsigned>(__cvta_generic_to_shared(ebuf)) + 4u * (unsigned)(lane * S)};
        if constexpr (NPARTS == 1) {
          taylor_strip_emit<R, 0, R, kU, ITERS>(row, sink);
        } else {  // two halves: the packed form
          if (part == 0) taylor_strip_emit_x2<R, 0, PART, kU, ITERS>(row, sink);
          else taylor_strip_emit_x2<R, PART, R, kU, ITERS>(row, sink);
        }
        // Order the buffer's generic-proxy writes before the async-proxy reads of the stores.
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
        if (lane < PART) {
          // Plane rows are padded to whole tiles, so every row stores whole.
          float* dst = p.emit_out + (long long)(k0 + k) * p.emit_job_stride +
                       (long long)(lo + lane) * p.emit_plane_stride + x0;
          if (tb.cache_mode == 1)  // stripe passes: keep the planes for the last level
            bulk_store_row_hint(dst, ebuf + lane * W, (unsigned)(W * sizeof(float)), policy_evict_last());
          else
            bulk_store_row(dst, ebuf + lane * W, (unsigned)(W * sizeof(float)));
          stores_pending = true;
        }
        continue;
      }
      const long long e = (long long)p.elig_T1 * (p.db_first + (long long)(k0 + k) * p.db_step);
      const long long base_off = p.off_base + (long long)(k0 + k) * p.off_step;
      const bool interior = (cs + e >= 0) && (cs + S - 1 + e + base_off + hi - 1 <= p.N - 1);
      if (__all_sync(0xffffffffu, interior)) {
        strip_part<R, PART, kU, ITERS, RELOAD>(part, row, mrow, FoldAll{});
      } else {
        edge_unit<SharedRow, R, PART, kU, ITERS, RELOAD>(part, lo, hi,
                                                         static_cast<unsigned>(__cvta_generic_to_shared(tile)),
                                                         &geo_win[g][0], ks, topS, x0, e, base_off, p.N);
      }
    }

    if constexpr (!EMIT) {
      __syncthreads();
      for (int i = threadIdx.x; i < W; i += blockDim.x) {
        const float v = topS[i];
        if (v > 0.0f && x0 + i < p.N) atomicMax(reinterpret_cast<int*>(p.top) + x0 + i, __float_as_int(v));
        topS[i] = 0.0f;
      }
    }
    if (kTakes && tb.next_item) item = item_next;
    else item += item % run == run - 1 ? (int)(gridDim.x - 1) * run + 1 : 1;
  }
  if (EMIT && stores_pending) bulk_wait_all();  // the buffers stay valid until read
  wait_previous_kernel();
}

template <typename E, int R, int NPARTS, int S, bool EMIT = false, int MAXW = 8>
size_t tree_smem_bytes(int nj, int d_step, bool shared_rows) {
  constexpr int W = kWarp * S;
  constexpr int V = 16 / sizeof(E);
  size_t bytes = sizeof(float) * (EMIT ? (size_t)MAXW * (R / NPARTS) * W : (size_t)((W + 3) & ~3));
  const int nseg = shared_rows ? 1 : nj;
  const int extra = shared_rows ? (nj - 1) * d_step : 0;
  for (int g = 0; g < nseg; ++g)
    for (int t = 0; t < R; ++t) bytes += sizeof(float) * (size_t)((V - 1 + W + (R - 1) + extra * t + V - 1) / V * V);
  return bytes;
}

template <typename E, int R, int NPARTS, int S, bool EMIT = false, int MAXW = 8, int MINB = 1, int RELOAD = 0,
          bool PAIR = false>
cudaError_t launch_tree(TreeBatch& b, int num_sms, size_t smem_budget, cudaStream_t stream) {
  constexpr int W = kWarp * S;
  auto kern = tree_max_kernel<E, R, NPARTS, S, EMIT, MAXW, MINB, RELOAD, PAIR>;
  // The dynamic shared memory a CTA can have: the device's opt-in limit less the kernel's
  // static arrays.  Budgets above it (a tuned launch of a larger shape class) are clamped, so
  // the chunk of jobs chosen below always fits.
  int dev = 0, optin = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err == cudaSuccess) err = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (err != cudaSuccess) return err;
  cudaFuncAttributes fa;
  if ((err = cudaFuncGetAttributes(&fa, kern)) != cudaSuccess) return err;
  const int max_dyn = optin - (int)fa.sharedSizeBytes;  // static + dynamic must fit the opt-in limit
  if (smem_budget > (size_t)max_dyn) smem_budget = (size_t)max_dyn;
  // The attribute is raised to the device's opt-in maximum, the same value from every
  // caller: host threads launching with different budgets cannot lower it under each other.
  err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn);
  if (err != cudaSuccess) return err;
  // The items that take longest first, so that the last ones to be taken are short.
  if (b.next_item) std::stable_sort(b.g, b.g + b.count, [](const TreeGroup& x, const TreeGroup& y) { return x.n_jobs > y.n_jobs; });
  size_t smem = 0;
  int max_warps = 1;
  long long n_items = 0;
  // Lays the groups' items out in order, group k in chunks of jobs_per_chunk jobs.
  auto lay_out = [&]() {
    smem = 0;
    max_warps = 1;
    n_items = 0;
    for (int k = 0; k < b.count; ++k) {
      TreeGroup& p = b.g[k];
      const bool shared_rows = (p.job_row_stride == 0);
      const int jpc = p.jobs_per_chunk;
      p.n_chunks = (p.n_jobs + jpc - 1) / jpc;
      const long long x_end = p.x_end > 0 ? p.x_end : (p.x_end < 0 ? p.x_begin : p.N);
      p.tile_first = p.x_begin / W;
      p.n_tiles = (int)std::max<long long>(0, (x_end + W - 1) / W - p.tile_first);
      p.item_begin = (int)n_items;
      n_items += (long long)p.n_tiles * p.n_chunks;
      const size_t sm = tree_smem_bytes<E, R, NPARTS, S, EMIT, MAXW>(jpc, p.d_step, shared_rows);
      if (sm > smem) smem = sm;
      const int w = (PAIR ? (jpc + 1) / 2 : jpc) * NPARTS;  // warp units of a chunk
      if (w > max_warps) max_warps = w;
    }
  };
  for (int k = 0; k < b.count; ++k) {
    TreeGroup& p = b.g[k];
    if (p.x_begin < 0 || p.x_begin % W != 0) return cudaErrorInvalidValue;
    const bool shared_rows = (p.job_row_stride == 0);
    // Largest chunk of jobs whose staged windows fit the shared-memory budget.
    int jpc = shared_rows ? p.n_jobs : (p.n_jobs < kMaxSeg ? p.n_jobs : kMaxSeg);
    while (jpc > 1 && tree_smem_bytes<E, R, NPARTS, S, EMIT, MAXW>(jpc, p.d_step, shared_rows) > smem_budget)
      jpc = shared_rows ? (jpc + 1) / 2 : jpc - 1;
    p.jobs_per_chunk = jpc;
  }
  lay_out();
  if (smem > (size_t)max_dyn) return cudaErrorInvalidValue;  // one job alone does not fit
  // CTAs that run at once, with the largest chunks.
  auto resident = [&]() {
    const int warps = max_warps > MAXW ? MAXW : max_warps;
    int per_sm = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, warps * kWarp, smem) != cudaSuccess || per_sm < 1)
      per_sm = 1;
    return (long long)per_sm * num_sms;
  };
  long long slots = resident();
  // The items that do not fill a whole round of resident CTAs -- all of them for a small search,
  // the last round of a larger one -- are cut into smaller chunks of jobs, so that the idle SMs
  // share their drift blocks.  A chunk's time is its staging, about 0.4 of a 16-row unit's strip
  // (kStage, in strips of this row count), and one strip per round of its units over the CTA's
  // warps; the cut with the smallest estimate is taken.  16 rows, 54 drift blocks: 32768
  // channels (32 tiles) 148 -> 45 us, 2^20 channels (993 tiles on 296 slots) 324 -> 258 us;
  // a launch of a dozen rounds or more whose CTAs take their items as they finish cuts its last round
  // into quarters instead, so that it ends within a short item: 8 searches of 15 x 1033216, 27
  // rounds, 2740 -> 2701 us a call.  With fixed shares whole chunks stage least.
  if constexpr (!EMIT) {
    const bool many = n_items >= 12 * slots;
    bool shared = n_items > 0 && (!many || (b.next_item && R <= 16 && S == kStrip));  // kTakes
    for (int k = 0; k < b.count; ++k) shared = shared && b.g[k].job_row_stride == 0;
    if (shared) {
      constexpr int kLevels = R >= 32 ? 5 : R >= 16 ? 4 : R >= 8 ? 3 : R >= 4 ? 2 : 1;
      constexpr double kStage = 0.4 * 64.0 / (R * kLevels / NPARTS);
      const long long rem = many ? slots : n_items % slots;
      // Tail groups: whole groups inside the last round, and the split rest of the one that
      // reaches into it.
      int first_tail = b.count;
      long long left = rem;
      while (left > 0 && first_tail > 0) {
        TreeGroup& p = b.g[first_tail - 1];
        const long long items = (long long)p.n_tiles * p.n_chunks;
        if (items <= left) {
          left -= items;
          --first_tail;
          continue;
        }
        const int tiles = (int)(left / p.n_chunks);  // its last tiles lie in the last round
        if (tiles > 0 && b.count < kMaxBatch) {
          for (int k = b.count; k > first_tail; --k) b.g[k] = b.g[k - 1];
          ++b.count;
          TreeGroup& q = b.g[first_tail];
          q = b.g[first_tail - 1];
          const int cut = (p.tile_first + p.n_tiles - tiles) * W;
          b.g[first_tail - 1].x_end = cut;
          q.x_begin = cut;
          if (q.x_end == 0) q.x_end = q.N;
          q.n_tiles = tiles;
        }
        left = 0;
      }
      int best = 0, max_jobs = 0;
      double best_time = 0.0;
      for (int k = first_tail; k < b.count; ++k) max_jobs = std::max(max_jobs, b.g[k].jobs_per_chunk);
      for (int j = many ? 0 : max_jobs; j >= 1; --j) {
        long long items = 0;
        for (int k = first_tail; k < b.count; ++k) {
          const int jk = std::min(j, b.g[k].jobs_per_chunk);
          items += (long long)b.g[k].n_tiles * ((b.g[k].n_jobs + jk - 1) / jk);
        }
        const int units = (PAIR ? (j + 1) / 2 : j) * NPARTS;
        const double t = (double)((items + slots - 1) / slots) * (kStage + (units + MAXW - 1) / MAXW);
        if (best == 0 || t < best_time) {
          best = j;
          best_time = t;
        }
      }
      if (many) best = std::max(1, (max_jobs / 4 + MAXW - 1) / MAXW * MAXW);
      for (int k = first_tail; k < b.count; ++k)
        b.g[k].jobs_per_chunk = std::min(best, b.g[k].jobs_per_chunk);
      lay_out();
      slots = resident();
    }
  }
  if (n_items == 0) return cudaSuccess;
  if (n_items > (1ll << 30)) return cudaErrorInvalidValue;
  b.n_items = (int)n_items;
  b.stage_wait_tries = stage_wait_tries();
  // Enough warps for every (job, offset part) unit of a chunk, at most MAXW.
  const int warps = max_warps > MAXW ? MAXW : max_warps;
  long long runs = n_items;
  if constexpr (EMIT) {
    if (b.tile_major) {
      for (int k = 0; k < b.count; ++k)  // the same tiles, whole chunks
        if (b.g[k].n_tiles != b.g[0].n_tiles || b.g[k].tile_first != b.g[0].tile_first || b.g[k].n_chunks != 1)
          return cudaErrorInvalidValue;
      runs = n_items / b.count;
    }
  }
  const int grid = (int)(runs < slots ? runs : slots);
  if (b.beside_previous) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(warps * kWarp);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, b);
  }
  kern<<<grid, warps * kWarp, smem, stream>>>(b);
  return cudaGetLastError();
}

// Shared memory per CTA (KB): 110 lets two CTAs share an SM; SETICORE_B200_TREE_SMEM_KB
// overrides it (tuning).
size_t tree_smem_budget() {
  static const size_t kb = [] {  // initialised once, thread-safely
    const char* e = getenv("SETICORE_B200_TREE_SMEM_KB");
    const long v = e ? strtol(e, nullptr, 10) : 0;
    return (v >= 48 && v <= 226) ? (size_t)v : (size_t)110;
  }();
  return kb * 1024;
}

int pair_reload() {
  static const int v = [] {
    const char* e = getenv("SETICORE_B200_PAIR_RELOAD");
    return (e && strtol(e, nullptr, 10) == 10) ? 10 : 12;
  }();
  return v;
}

template <typename E, int S>
cudaError_t launch_rows(TreeBatch& b, int R, int num_sms, size_t budget, cudaStream_t stream) {
  switch (R) {
    case 2: return launch_tree<E, 2, 1, S>(b, num_sms, budget, stream);
    case 4: return launch_tree<E, 4, 1, S>(b, num_sms, budget, stream);
    case 8:
      return launch_tree<E, 8, 1, S, false, 8, 1, (S == kU && std::is_same<E, float>::value ? kPacked : 0)>(
          b, num_sms, budget, stream);
    case 16:
      // Long strips: all 16 offsets in one warp, which loads most leaves once per drift block
      // (two offset halves load every leaf twice; shared-memory bandwidth bounded that form).
      // Carrying every leaf window takes ~213 registers, room for 8 warps per SM; the leaves
      // whose windows span 12 or more channels (8 for 16-bit inputs, whose staging needs more
      // registers) are read again at each use instead, which fits 128 registers and so two
      // CTAs of eight warps per SM (+5 % over two CTAs of four; for float, thresholds 8 and 10
      // reread more leaves and measured 1-2 % slower, and 12 spilled the 16-bit forms 5 %).
      if constexpr (S == kStrip)
        return launch_tree<E, 16, 1, S, false, 8, 2, (std::is_same<E, float>::value ? 12 : 8)>(b, num_sms, budget, stream);
      // Short strips (the last level of a tree of more than 32 rows, one job of two offset
      // halves per CTA): capped at 128 registers, eight such CTAs share an SM (six at the
      // 134 registers the compiler picks unbounded; 5 % slower on 256-row beams).  Float planes
      // take the packed form, and so does the first level: fewer instructions per channel where
      // neither the adds' pipes nor the loads are the limit (32 beams of 256 rows, both levels:
      // 4.56 -> 4.36 ms; ten or twelve CTAs per SM at 96 or 80 registers: 4.41, 4.45).  The long
      // strips keep the single-float form: packed, their 16-row tree issues 21 % fewer
      // instructions but needs 168 registers, so twelve warps per SM (16 searches of 2^20
      // channels: 3.55 against 3.50 ms; at 128 registers it spills, 3.69).
      else if constexpr (std::is_same<E, float>::value)
        return launch_tree<E, 16, 2, S, false, 2, 8, kPacked>(b, num_sms, budget, stream);
      else return launch_tree<E, 16, 2, S, false, 2, 8>(b, num_sms, budget, stream);
    default: return cudaErrorInvalidValue;
  }
}

// 32 rows: two parts of sixteen offsets, long strips only.  Each part loads all 32 leaves of
// a channel, so fewer parts mean fewer shared loads per path sum (eight parts of four took 1.7x
// as long).  A part carries ~230 registers of node windows; capped at 168 (a few spilled) one
// CTA of twelve warps fills an SM (9 % faster than eight warps at 230), and it stages as many
// drift blocks per tile as 200 KB or more of shared memory holds.
template <typename E>
cudaError_t launch_rows32(TreeBatch& b, int num_sms, size_t budget, cudaStream_t stream) {
  const size_t min_budget = (size_t)200 * 1024;
  if (budget < min_budget) budget = min_budget;
  // the paired-FP16 tree of 16-bit searches: the same shape over the paired copy
  if (b.pair16) return launch_tree<float, 32, 2, kStrip, false, 12, 1, 0, true>(b, num_sms, budget, stream);
  return launch_tree<E, 32, 2, kStrip, false, 12, 1>(b, num_sms, budget, stream);
}

template <typename E>
cudaError_t tree_dispatch(TreeBatch& b, int R, int num_sms, cudaStream_t stream, TreeLaunch how) {
  // Jobs that each stage their own rows (the last level of a tree of more than 32 rows)
  // default to short strips and one job per CTA: a 352-channel tile needs a third of the
  // shared memory per job, so three times as many warps fit an SM and the small CTAs overlap
  // one another's staging (each staged value serves a single drift block there) with their
  // tree work, at the price of more window fills per channel.
  bool own_rows = b.count > 0;
  for (int k = 0; k < b.count; ++k) own_rows = own_rows && b.g[k].job_row_stride != 0;
  int tile = how.tile ? how.tile : (own_rows ? kWarp * kU : kWarp * kStrip);
  size_t budget = how.smem_kb > 0 ? (size_t)how.smem_kb * 1024 : tree_smem_budget();
  if (b.pair16) {
    // The paired-FP16 tree: long strips, two CTAs of eight warps per SM; the leaves whose
    // windows span 12 channels or more (10 with SETICORE_B200_PAIR_RELOAD=10) are reread.
    // Node, BF16: 75.3 Gsamples/s at 12, 73.6 at 10; seven-warp CTAs (a whole number of
    // rounds for 27 units) measured 62.2 and 68.0: they spill more at the same 128 registers;
    // six-warp CTAs (168 registers) 72.7 and 72.3.  32 rows: launch_rows32's shape.
    if (own_rows || (R != 16 && R != 32)) return cudaErrorInvalidValue;
    if (R == 32) return launch_rows32<float>(b, num_sms, budget, stream);
    if (pair_reload() == 10) return launch_tree<float, 16, 1, kStrip, false, 8, 2, 10, true>(b, num_sms, budget, stream);
    return launch_tree<float, 16, 1, kStrip, false, 8, 2, 12, true>(b, num_sms, budget, stream);
  }
  if (own_rows && how.smem_kb <= 0) budget = (size_t)24 * 1024;
  // Last levels of 4 rows or fewer have little tree work per staged row: long strips and up
  // to four jobs per CTA spread each item's fixed cost (layout, barriers, top updates) over
  // three times the channels (14 % faster on 64-row searches; 5 % slower at 8 rows).
  if (own_rows && R <= 4 && how.smem_kb <= 0 && how.tile == 0) {
    tile = kWarp * kStrip;
    budget = (size_t)72 * 1024;
  }
  if (R == 32) return own_rows ? cudaErrorInvalidValue : launch_rows32<E>(b, num_sms, budget, stream);  // pairs too
  if (tile == kWarp * kU) return launch_rows<E, kU>(b, R, num_sms, budget, stream);
  if (tile == kWarp * kStrip) return launch_rows<E, kStrip>(b, R, num_sms, budget, stream);
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t tree_max_batch(TreeBatch& b, int R, int num_sms, cudaStream_t stream, int elem, TreeLaunch how) {
  if (how.smem_kb > 226) how.smem_kb = 226;
  switch (elem) {
    case kElemF32: return tree_dispatch<float>(b, R, num_sms, stream, how);
    case kElemBF16: return tree_dispatch<__nv_bfloat16>(b, R, num_sms, stream, how);
    case kElemF16: return tree_dispatch<__half>(b, R, num_sms, stream, how);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t tree_emit_batch(TreeBatch& b, int num_sms, cudaStream_t stream, int smem_budget_kb, int nparts) {
  if (smem_budget_kb > 226) smem_budget_kb = 226;
  const size_t budget = smem_budget_kb > 0 ? (size_t)smem_budget_kb * 1024 : (size_t)80 * 1024;
  // Short strips; two halves of eight offsets (four warps, 45 KB of buffers) or all sixteen
  // offsets in one warp (loads each leaf once per drift block; two warps, 45 KB).
  if (nparts == 1) return launch_tree<float, 16, 1, kU, true, 2, 1>(b, num_sms, budget, stream);
  return launch_tree<float, 16, 2, kU, true, 4, 1>(b, num_sms, budget, stream);
}

int tree_tile_width() { return kWarp * kStrip; }

namespace {
std::atomic<int> g_stage_wait_tries{-1};
std::atomic<bool> g_paired_fp16{true};
}
void set_paired_fp16(bool on) { g_paired_fp16.store(on); }
bool paired_fp16() { return g_paired_fp16.load(); }
void set_stage_wait_tries(int tries) { g_stage_wait_tries.store(tries < 0 ? -1 : tries); }
int stage_wait_tries() { return g_stage_wait_tries.load(); }

}  // namespace scb
