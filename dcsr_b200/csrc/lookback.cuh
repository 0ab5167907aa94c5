// lookback.cuh -- device side of the single-pass kernels (decoupled
// look-back) and the scan over a row or entry function that the load, export,
// schedule and update kernels are built from.
#pragma once
#include <type_traits>

#include "common.cuh"

namespace dcsr {

// ------------------------------------------------- decoupled look-back
//
// Single-pass kernels: every block takes the next tile number from a device
// counter (so all tiles before it are running or finished), publishes its
// tile's aggregate, adds the aggregates of the tiles before it back to the
// nearest published inclusive prefix, and publishes its own inclusive prefix.
// A wait is only ever on an earlier tile, which therefore always finishes;
// every wait still has an iteration limit, after which it counts a fault and
// stops waiting.

__device__ __forceinline__ unsigned long long ld_vol(const unsigned long long *p) {
  return *(const volatile unsigned long long *)p;
}

// Look-back words are packed: a tag (the epoch's low 30 bits, a 2-bit kind)
// above a 32-bit value, so a word is published with one store and read with
// one load -- no fences, no second load.  A sort's word per (tile, digit)
// holds a count (kind 1: the tile's aggregate, 2: its inclusive prefix); a
// scan has one 128-bit word per tile, tag and kind above 96 bits of
// sums, stored and loaded whole.  The two kinds have areas of their own: the
// lower half of a scan's word has no tag, and read as a sort's word its sums
// could be taken for a current count.  A word is current when its tag is the
// kernel's; the tag repeats every 2^30 kernels on one area, so the kernel
// whose last block advances the epoch to such a multiple clears both areas
// (lb_advance) and a stale word never matches.
constexpr unsigned long long LB_EMASK = (1ull << 30) - 1;
__host__ __device__ __forceinline__ unsigned long long lb_pack(unsigned long long e, int kind, unsigned v) {
  return ((e & LB_EMASK) << 34) | ((unsigned long long)kind << 32) | v;
}

// A wait that gave up: count it, mark the area's fault word with this
// kernel's epoch (its other waits then give up early) and report
// DCSR_TIMEOUT in the operation's status word.
__device__ __forceinline__ void lb_give_up(const Lookback &lb, unsigned long long e) {
  atomicAdd(&lb.g->faults, 1ull);
  *(volatile unsigned long long *)lb.fault = (e & LB_EMASK) + 1;
  __threadfence();  // before the block counts as finished
  if (lb.status) atomicCAS(reinterpret_cast<unsigned long long *>(lb.status), 0ull, (unsigned long long)DCSR_TIMEOUT);
}
// True when another wait of this kernel (epoch e) gave up already.
__device__ __forceinline__ bool lb_faulted(const Lookback &lb, unsigned long long e) {
  return ld_vol(lb.fault) == (e & LB_EMASK) + 1;
}

// Thread 0 of every block: the block's tile and the kernel's epoch.
__device__ __forceinline__ void lb_begin(const Lookback &lb, unsigned *tile, unsigned long long *ep) {
  if (threadIdx.x == 0) {
    *tile = atomicAdd(lb.tiles, 1u);
    *ep = ld_vol(lb.epoch);
  }
}

// End of every block (all threads): true in the last block to finish.
__device__ __forceinline__ bool lb_end(const Lookback &lb) {
  __shared__ int last;
  __syncthreads();
  // (no fence: this block's results reach later kernels at the launch boundary)
  if (threadIdx.x == 0) last = atomicAdd(lb.done, 1u) == gridDim.x - 1;
  __syncthreads();
  return last;
}

// The last block (all its threads): reset the counters and advance the
// epoch; at a multiple of 2^30 clear the words first (their tags come round).
__device__ __forceinline__ void lb_advance(const Lookback &lb) {
  __shared__ unsigned long long next;
  if (threadIdx.x == 0) next = ld_vol(lb.epoch) + 1;
  __syncthreads();
  if ((next & LB_EMASK) == 0)
    for (unsigned long long i = threadIdx.x; i < lb.slots; i += blockDim.x) lb.flag[i] = lb.scan[i] = 0;
  __syncthreads();
  if (threadIdx.x == 0) {
    *(volatile unsigned *)lb.tiles = 0;
    *(volatile unsigned *)lb.done = 0;
    __threadfence();
    *(volatile unsigned long long *)lb.epoch = next;
  }
}

// A scan's 128-bit look-back word (16-byte aligned), written and read as one
// relaxed access: hi = tag | kind | 32 bits, lo = 64 bits; the 96 bits hold
// one sum of 64 bits, one of 64 and one of 32, or three of 32 (the 32-bit ones
// modulo 2^32).  Of two sums the first is the one that may be large: layout
// capacities, whose options allow 2^31 entries a row.
struct LbWord {
  unsigned long long lo, hi;
};
__device__ __forceinline__ LbWord lb_load(const unsigned long long *p) {
  LbWord w;
  asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
               : "=l"(w.lo), "=l"(w.hi)
               : "l"(p)
               : "memory");
  return w;
}
__device__ __forceinline__ void lb_store(unsigned long long *p, const LbWord &w) {
  asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%0, %1};\n\tst.relaxed.gpu.global.b128 [%2], q;\n\t}" ::"l"(w.lo),
               "l"(w.hi), "l"(p)
               : "memory");
}
template <int NS>
__host__ __device__ __forceinline__ LbWord lb_word(unsigned long long e, int kind, const long long (&v)[NS]) {
  static_assert(NS >= 1 && NS <= 3, "one to three sums");
  LbWord w;
  w.lo = (unsigned long long)v[0];
  w.hi = lb_pack(e, kind, 0);
  if constexpr (NS == 3) {
    w.lo = (w.lo & 0xffffffffull) | ((unsigned long long)v[1] << 32);
    w.hi |= (unsigned long long)v[2] & 0xffffffffull;
  }
  if constexpr (NS == 2) w.hi |= (unsigned long long)v[1] & 0xffffffffull;
  return w;
}
template <int NS>
__host__ __device__ __forceinline__ long long lb_sum(const LbWord &w, int q) {
  if constexpr (NS == 1) return (long long)w.lo;
  if constexpr (NS == 3) return (long long)(unsigned)(q == 0 ? w.lo : q == 1 ? w.lo >> 32 : w.hi);
  return q == 0 ? (long long)w.lo : (long long)(unsigned)w.hi;
}
// Look-back words (8 bytes) that a scan of `tiles` tiles needs.
constexpr int LB_SCAN_WORDS = 2;

// Warp 0 of tile t (the first tile of its sequence is t0): publish the NS
// aggregates agg (in every lane), look back over the earlier tiles, publish
// the inclusive prefixes; excl receives the sums of the tiles before t (in
// every lane).  A step loads 32 * LB_U tiles' words together: when all tiles
// of a scan run at once (up to about 2^20 items) the look-back is a chain of
// such round trips, and the 512 tiles of a 2^20-row scan took 10 of its 16 us
// with 32 tiles and four 64-bit words each a step.
constexpr int LB_U = 4;
template <int NS>
__device__ __forceinline__ void lb_lookback(const Lookback &lb, unsigned long long e, int64_t t, int64_t t0,
                                            const long long (&agg)[NS], long long (&excl)[NS]) {
  const int lane = lane_id();
  const unsigned tag2 = (unsigned)(e & LB_EMASK) << 2;  // a current word's upper 32 bits, less its kind
  unsigned long long *w = lb.scan;
#pragma unroll
  for (int q = 0; q < NS; q++) excl[q] = 0;
  if (t == t0) {
    if (lane == 0 && !(lb.g->stall && t == 0)) lb_store(w + 2 * t, lb_word<NS>(e, 2, agg));
    return;
  }
  if (lane == 0) lb_store(w + 2 * t, lb_word<NS>(e, 1, agg));
  int idle = 0;
  const int limit = lb.g->spin_limit;
  bool done = false;
  for (int64_t j = t - 1; !done;) {
    LbWord x[LB_U];
#pragma unroll
    for (int u = 0; u < LB_U; u++) {
      const int64_t r = j - 32 * u - lane;  // u = 0, lane 0: the nearest earlier tile
      if (r >= t0) x[u] = lb_load(w + 2 * r);
      else x[u] = LbWord{0, lb_pack(e, 2, 0)};  // before the first tile: an inclusive prefix of 0
    }
    int used = 0;
    bool live = true;
#pragma unroll
    for (int u = 0; u < LB_U; u++) {
      if (!live) continue;
      const unsigned kind = (unsigned)(x[u].hi >> 32) - tag2;  // 1, 2, or not published in this epoch
      const unsigned rm = __ballot_sync(FULL, kind - 1u < 2u), im = __ballot_sync(FULL, kind == 2u);
      const int first = im ? __ffs(im) - 1 : 32;  // nearest inclusive prefix among these 32
      const unsigned need = first >= 31 ? FULL : ((2u << first) - 1u);
      live = (rm & need) == need;  // everything up to it published
      if (live) {
#pragma unroll
        for (int q = 0; q < NS; q++) excl[q] += warp_sum(lane <= first ? lb_sum<NS>(x[u], q) : 0ll);
        used = u + 1;
        done = first < 32;
        live = !done;
      }
    }
    j -= 32 * used;
    if (used) {
      idle = 0;
      continue;
    }
    if (++idle >= limit || ((idle & 1023) == 1023 && __any_sync(FULL, lb_faulted(lb, e)))) {
      if (lane == 0) lb_give_up(lb, e);
      break;
    }
    if (idle >= 32) __nanosleep(64);
  }
  long long inclv[NS];
#pragma unroll
  for (int q = 0; q < NS; q++) inclv[q] = excl[q] + agg[q];
  if (lane == 0) lb_store(w + 2 * t, lb_word<NS>(e, 2, inclv));
}

// ------------------------------------------------------- scan over a function
//
// One kernel computes a value (NS of them) per item i in [0, n), scans it
// exclusively and hands every item its prefix, so an operator needs no array
// of flags, no scan of it and no pass over the result.  F supplies
//   static constexpr int NS, IT;     sums; items per thread
//   struct State;                    what load leaves for emit (registers)
//   load(i, ok, st, v[NS])           value of item i (ok false: past the end, v must be 0),
//                                    or, with a member LOAD_ALL, load_all(base, n, st[], v[][NS])
//                                    for the thread's items base + 32*j at once
//   emit(i, ok, st, excl[NS], v[NS]) item i's prefix; called by whole warps (with a member
//                                    EMIT_ALL after emit_all(base, n, st[], v[][NS]))
//   total(tot[NS])                   one thread, the totals
//   fault()                          (if there) one thread, last of all, when a look-back wait gave up:
//                                    marks the result so that kernels behind it do not use it
// A warp takes 32*IT consecutive items, item j*32 + lane in lane's j-th step
// (coalesced, and every step's prefix by a warp scan in registers -- no
// staging through shared memory), a block SM_THREADS*IT.  Light functions
// (IT = 8) of up to SM_ONE items run in one block without look-back, with as
// few items a thread as its 1024 threads allow (a few rows of many tiles each
// are then marked by as many warps as can be: 500 rows of 78 tiles 8.8 us,
// 46 with eight rows a lane in two warps); heavy ones (IT = 4: searches, plans)
// spread over blocks from 1024 items on.
constexpr int SM_LIGHT = 8, SM_HEAVY = 4;
constexpr int SM_THREADS = 256;
constexpr int SM_ONE_THREADS = 1024;
constexpr int64_t SM_ONE = SM_ONE_THREADS * SM_LIGHT;
// Light functions of up to SM_FEW items take SM_THIN a thread: at 8 a thread a
// scan of 131072 rows runs in 64 blocks, most SMs idle and each thread's eight
// loads and stores one after the other (placing rows 20 -> 13 us at 131072 rows,
// 18 -> 8 at 20011).  SM_FEW is 512 blocks of that size (148
// SMs hold 592 at once; 1024 words of look-back area, which every area has);
// above it the wide form fills the SMs as well.
constexpr int SM_THIN = 2;
constexpr int64_t SM_FEW = 512 * SM_THREADS * SM_THIN;

template <class F, class = void>
struct ScanHasEmitAll : std::false_type {};
template <class F>
struct ScanHasEmitAll<F, std::void_t<decltype(F::EMIT_ALL)>> : std::bool_constant<F::EMIT_ALL> {};
template <class F, class = void>
struct ScanHasLoadAll : std::false_type {};
template <class F>
struct ScanHasLoadAll<F, std::void_t<decltype(F::LOAD_ALL)>> : std::true_type {};

template <class F, class = void>
struct ScanHasFault : std::false_type {};
template <class F>
struct ScanHasFault<F, std::void_t<decltype(&F::fault)>> : std::true_type {};

template <int TH, class F, int SM_ITEMS = F::IT>
__global__ void __launch_bounds__(TH, TH > SM_THREADS ? 1 : F::IT == SM_HEAVY || ScanHasLoadAll<F>::value ? 3 : 4) k_scan_map(F f, int64_t n, Lookback lb) {
  constexpr int NS = F::NS, NW = TH / 32;
  __shared__ long long wsum[NS][NW];
  __shared__ long long sh_prefix[NS];
  __shared__ unsigned sh_tile;
  __shared__ unsigned long long sh_ep;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool single = gridDim.x == 1;
  int64_t t = 0;
  unsigned long long e = 0;
  if (!single) {
    lb_begin(lb, &sh_tile, &sh_ep);
    __syncthreads();
    t = sh_tile;
    e = sh_ep;
    if (t >= gridDim.x) {  // a tile counter left non-zero (a bug): report it, touch nothing
      if (threadIdx.x == 0) lb_give_up(lb, e);
      if (lb_end(lb)) lb_advance(lb);
      return;
    }
  }
  const int64_t base = t * (TH * SM_ITEMS) + (int64_t)w * (32 * SM_ITEMS) + lane;
  typename F::State st[SM_ITEMS];
  typename F::T v[SM_ITEMS][NS], ex[SM_ITEMS][NS];
  long long run[NS];
#pragma unroll
  for (int q = 0; q < NS; q++) run[q] = 0;
  if constexpr (ScanHasLoadAll<F>::value) {
    f.load_all(base, n, st, v);
  } else {
#pragma unroll
    for (int j = 0; j < SM_ITEMS; j++) {
      const int64_t i = base + 32 * j;
      f.load(i, i < n, st[j], v[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < SM_ITEMS; j++)
#pragma unroll
    for (int q = 0; q < NS; q++) {
      const typename F::T inc = warp_incl_scan(v[j][q]);
      ex[j][q] = (typename F::T)run[q] + inc - v[j][q];
      run[q] += __shfl_sync(FULL, inc, 31);
    }
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NS; q++) wsum[q][w] = run[q];
  __syncthreads();
  long long before[NS], agg[NS];
#pragma unroll
  for (int q = 0; q < NS; q++) {
    long long x = lane < NW ? wsum[q][lane] : 0;  // NW <= 32 warps
    agg[q] = warp_sum(x);
    before[q] = warp_sum(lane < w ? x : 0ll);
  }
  if (!single) {
    if (w == 0) {
      long long excl[NS];
      lb_lookback<NS>(lb, e, t, 0, agg, excl);
      if (lane == 0)
#pragma unroll
        for (int q = 0; q < NS; q++) sh_prefix[q] = excl[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NS; q++) before[q] += sh_prefix[q];
  }
  if constexpr (ScanHasEmitAll<F>::value) f.emit_all(base, n, st, v);
#pragma unroll
  for (int j = 0; j < SM_ITEMS; j++) {
    const int64_t i = base + 32 * j;
    long long p[NS];
#pragma unroll
    for (int q = 0; q < NS; q++) p[q] = before[q] + (long long)ex[j][q];
    f.emit(i, i < n, st[j], p, v[j]);
  }
  if (threadIdx.x == 0 && t == (int64_t)gridDim.x - 1) {
    long long tot[NS];
#pragma unroll
    for (int q = 0; q < NS; q++) tot[q] = (single ? 0 : sh_prefix[q]) + agg[q];
    f.total(tot);
    if constexpr (ScanHasFault<F>::value)
      if (!single) __threadfence();  // (fault() may write over it from another block)
  }
  if (!single && lb_end(lb)) {
    if constexpr (ScanHasFault<F>::value)
      if (threadIdx.x == 0 && lb_faulted(lb, e)) f.fault();
    lb_advance(lb);
  }
}

// n >= 1 items.  Needs LB_SCAN_WORDS look-back slots per SM_THREADS*IT items.
template <class F>
static int scan_map(const F &f, int64_t n, Arena &ar, cudaStream_t s) {
  Lookback lb;
  std::memset(&lb, 0, sizeof(lb));
  const int64_t nt = div_up(n, SM_THREADS * F::IT);
  constexpr bool ANY = F::IT == SM_LIGHT && !ScanHasLoadAll<F>::value && !ScanHasEmitAll<F>::value;  // items a thread
  if constexpr (ANY) {
    if (n <= SM_ONE_THREADS) {
      DCSR_LAUNCH((k_scan_map<SM_ONE_THREADS, F, 1>), 1, SM_ONE_THREADS, 0, s, f, n, lb);
      return DCSR_OK;
    }
    if (n <= 2 * SM_ONE_THREADS) {
      DCSR_LAUNCH((k_scan_map<SM_ONE_THREADS, F, 2>), 1, SM_ONE_THREADS, 0, s, f, n, lb);
      return DCSR_OK;
    }
    if (n <= 4 * SM_ONE_THREADS) {
      DCSR_LAUNCH((k_scan_map<SM_ONE_THREADS, F, 4>), 1, SM_ONE_THREADS, 0, s, f, n, lb);
      return DCSR_OK;
    }
  }
  if (nt == 1) {
    DCSR_LAUNCH((k_scan_map<SM_THREADS, F>), 1, SM_THREADS, 0, s, f, n, lb);
    return DCSR_OK;
  }
  if constexpr (F::IT == SM_LIGHT) {
    if (n <= SM_ONE) {
      DCSR_LAUNCH((k_scan_map<SM_ONE_THREADS, F>), 1, SM_ONE_THREADS, 0, s, f, n, lb);
      return DCSR_OK;
    }
  }
  if constexpr (ANY) {
    if (n <= SM_FEW) {
      const int64_t few = div_up(n, SM_THREADS * SM_THIN);
      DCSR_TRY(ar.lookback((size_t)(LB_SCAN_WORDS * few), s, &lb));
      DCSR_LAUNCH((k_scan_map<SM_THREADS, F, SM_THIN>), (unsigned)few, SM_THREADS, 0, s, f, n, lb);
      return DCSR_OK;
    }
  }
  DCSR_TRY(ar.lookback((size_t)(LB_SCAN_WORDS * nt), s, &lb));
  DCSR_LAUNCH((k_scan_map<SM_THREADS, F>), (unsigned)nt, SM_THREADS, 0, s, f, n, lb);
  return DCSR_OK;
}

}  // namespace dcsr
