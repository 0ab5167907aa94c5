// prims.cu -- device-wide primitives: exclusive scan, stable LSD radix sort of
// (key, value) pairs, and the public segmented primitives
// (count_sorted_indices, reduce_by_key).  All hand-written for sm_100a.
#include <algorithm>
#include <cstddef>
#include <mutex>
#include <utility>

#include "lookback.cuh"

namespace dcsr {

std::atomic<uint64_t> g_launches{0};

bool debug_sync() {
  static const bool on = [] {
    const char *e = getenv("DCSR_DEBUG_SYNC");
    return e && e[0] == '1';
  }();
  return on;
}

void debug_check(cudaStream_t s, const char *kernel, const char *file, int line) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return;
  const cudaError_t e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) fprintf(stderr, "dcsr: kernel %s (%s:%d) failed: %s\n", kernel, file, line, cudaGetErrorString(e));
}

int sm_count() {
  // function-local statics are initialised once, thread-safely (the server
  // launches from several threads)
  static const int n = [] {
    int dev = 0, c = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev);
    return c > 0 ? c : 148;
  }();
  return n;
}

int persistent_grid(const void *kernel, int block, size_t smem) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  return per_sm * sm_count();
}

// ------------------------------------------------------------------ scan

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

// Block-wide exclusive scan of one value per thread; returns the block total.
template <typename T>
__device__ __forceinline__ T block_excl_scan(T v, T *total) {
  __shared__ T wsum[33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  T inc = warp_incl_scan(v);
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    T w = lane < nw ? wsum[lane] : T(0);
    T wi = warp_incl_scan(w);
    if (lane < nw) wsum[lane] = wi - w;
    if (lane == nw - 1) wsum[32] = wi;
  }
  __syncthreads();
  T out = inc - v + wsum[warp];
  *total = wsum[32];
  __syncthreads();
  return out;
}

constexpr int SPIN_LIMIT = 1 << 22;
// Wait limit of the look-back kernels (SPIN_LIMIT unless a test lowered it),
// the test switch that keeps the first tile of every single-pass kernel
// from publishing so the waits on it run out (dcsr_debug_lookback), and the
// count of waits that did.  Kernels of every file reach it through Lookback.
__device__ LookbackGlobals g_lookback = {0ull, SPIN_LIMIT, 0};
#ifndef DCSR_LB_W
#define DCSR_LB_W 8
#endif
constexpr int LB_W = DCSR_LB_W;  // earlier tiles whose flags one radix look-back step loads together

int lookback_globals(LookbackGlobals **out) {
  static std::mutex mu;
  static std::atomic<LookbackGlobals *> ptr[128] = {};
  int dev = 0;
  DCSR_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 128) return DCSR_NOT_SUPPORTED;
  LookbackGlobals *g = ptr[dev].load();
  if (!g) {
    std::lock_guard<std::mutex> lock(mu);
    void *p = nullptr;
    DCSR_CUDA(cudaGetSymbolAddress(&p, g_lookback));
    g = (LookbackGlobals *)p;
    ptr[dev].store(g);
  }
  *out = g;
  return DCSR_OK;
}

long long spin_faults() {
  LookbackGlobals v;
  if (cudaMemcpyFromSymbol(&v, g_lookback, sizeof(v)) != cudaSuccess) return -1;
  return (long long)v.faults;
}

int debug_lookback(int spin_limit, int stall) {
  const int lim = spin_limit > 0 ? spin_limit : SPIN_LIMIT;
  DCSR_CUDA(cudaMemcpyToSymbol(g_lookback, &lim, sizeof(int), offsetof(LookbackGlobals, spin_limit)));
  DCSR_CUDA(cudaMemcpyToSymbol(g_lookback, &stall, sizeof(int), offsetof(LookbackGlobals, stall)));
  DCSR_CUDA(cudaDeviceSynchronize());
  return DCSR_OK;
}

struct ScanArgs {
  const long long *in;
  long long *out;
  long long *total;
  int64_t n, nt;
};

// Exclusive scan, one pass: tiles of SCAN_TILE values; warp 0 looks back over
// the earlier tiles (lb_lookback).  In place (in == out) is allowed.
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_1p(ScanArgs a, Lookback lb) {
  __shared__ long long tile[SCAN_TILE];
  __shared__ unsigned sh_tile;
  __shared__ unsigned long long sh_ep;
  __shared__ long long sh_prefix;
  lb_begin(lb, &sh_tile, &sh_ep);
  __syncthreads();
  const int64_t t = sh_tile;
  const unsigned long long e = sh_ep;
  if (t >= gridDim.x) {  // a tile counter left non-zero (a bug): report it, touch nothing
    if (threadIdx.x == 0) lb_give_up(lb, e);
    if (lb_end(lb)) lb_advance(lb);
    return;
  }
  const long long *__restrict__ in = a.in;
  long long *out = a.out;
  const int64_t n = a.n;
  const int64_t base = t * SCAN_TILE;
#pragma unroll
  for (int j = 0; j < SCAN_ITEMS; j++) {
    const int64_t i = base + j * SCAN_THREADS + threadIdx.x;
    tile[j * SCAN_THREADS + threadIdx.x] = i < n ? in[i] : 0;
  }
  __syncthreads();
  long long loc[SCAN_ITEMS];
  long long sum = 0;
#pragma unroll
  for (int j = 0; j < SCAN_ITEMS; j++) {
    loc[j] = tile[threadIdx.x * SCAN_ITEMS + j];
    sum += loc[j];
  }
  long long bt;
  long long ex = block_excl_scan(sum, &bt);
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const long long agg[1] = {bt};
    long long before[1];
    lb_lookback<1>(lb, e, t, 0, agg, before);
    const long long excl = before[0];
    if (lane == 0) sh_prefix = excl;
  }
  __syncthreads();
  ex += sh_prefix;
#pragma unroll
  for (int j = 0; j < SCAN_ITEMS; j++) {
    tile[threadIdx.x * SCAN_ITEMS + j] = ex;
    ex += loc[j];
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < SCAN_ITEMS; j++) {
    const int64_t i = base + j * SCAN_THREADS + threadIdx.x;
    if (i < n) out[i] = tile[j * SCAN_THREADS + threadIdx.x];
  }
  if (threadIdx.x == 0 && a.total && base + SCAN_TILE >= n) *a.total = sh_prefix + bt;
  if (lb_end(lb)) lb_advance(lb);
}

// Small inputs: one block; coalesced loads into shared memory, each thread
// scans 4 consecutive values, one block scan, coalesced stores.
constexpr int SCAN_SMALL = 1024 * 4;
__global__ void __launch_bounds__(1024) k_scan_small(ScanArgs a) {
  const long long *__restrict__ in = a.in;
  long long *out = a.out;
  long long *total = a.total;
  const int64_t n = a.n;
  __shared__ long long tile[SCAN_SMALL];
  for (int i = threadIdx.x; i < SCAN_SMALL; i += 1024) tile[i] = i < n ? in[i] : 0;
  __syncthreads();
  long long loc[4], sum = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    loc[j] = tile[threadIdx.x * 4 + j];
    sum += loc[j];
  }
  long long bt;
  long long ex = block_excl_scan(sum, &bt);
#pragma unroll
  for (int j = 0; j < 4; j++) {
    tile[threadIdx.x * 4 + j] = ex;
    ex += loc[j];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += 1024) out[i] = tile[i];
  if (threadIdx.x == 0 && total) *total = bt;
}

size_t scan_scratch_bytes(int64_t n) { return arena_bytes(div_up(n, SCAN_TILE) + 1, 8); }

int scan_i64(const long long *in, long long *out, int64_t n, long long *total, Arena &ar, cudaStream_t s) {
  if (n <= 0) {
    if (total) DCSR_CUDA(cudaMemsetAsync(total, 0, sizeof(long long), s));
    return DCSR_OK;
  }
  const ScanArgs a{in, out, total, n, div_up(n, SCAN_TILE)};
  if (n <= SCAN_SMALL) {
    DCSR_LAUNCH(k_scan_small, 1, 1024, 0, s, a);
    return DCSR_OK;
  }
  Lookback lb;
  DCSR_TRY(ar.lookback((size_t)(LB_SCAN_WORDS * a.nt), s, &lb));
  DCSR_LAUNCH(k_scan_1p, (unsigned)a.nt, SCAN_THREADS, 0, s, a, lb);
  return DCSR_OK;
}

// ------------------------------------------------------------ radix sort
//
// Stable LSD radix sort of (key, input index) by 8-bit digits.  Where key and
// index fit in 64 bits together (every update and load whose
// row, column and triple count do: 40-bit keys of a 2^20 x 2^20 matrix with up
// to 2^24 triples) the sort moves one packed word per item -- the first pass
// packs, the last one unpacks -- else a key and an index.
//   up to RS_SMALL items  one CTA, the words in registers, every pass a rank
//                         and a scatter through shared memory;
//   up to RS_BIG          one histogram kernel for all digits (its last block
//                         scans them), then per pass one scatter kernel: a
//                         block takes the next tile, ranks its items per warp
//                         through lane masks (ties keep input order), publishes
//                         its digit counts, orders the tile in shared memory,
//                         finds the items of each digit in the tiles before
//                         it by decoupled look-back (one thread per digit,
//                         LB_W earlier tiles per step) and writes whole digit
//                         runs;
//   larger                three kernels per pass (tile histograms, the scan of
//                         the digit-major table, a scatter), which bounds the
//                         look-back area.
// Measured, 40-bit keys (five passes): 1.05M items 15.5 us a pass and 14 us
// the histograms (35 and 11 us with key-index pairs, match_any and a scatter
// straight from registers in tiles of 2048), 16.8M items 142-156 us a pass and
// 57 us (350 and 67 us).  A pass moves 16 bytes an item (a floor of 40 us at
// 16.8M); it is bound by the rank chains through shared memory at 24 warps
// per SM.  Tiles of 2048, 3072 and 8192 items, 8 or 16 look-back words a step
// and four blocks per SM (spills) were within 3% or slower.

constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_BINS = 256;
#ifndef DCSR_RS_MID_LOG2
#define DCSR_RS_MID_LOG2 22
#endif
// Sorts above RS_MID may take the three-kernel passes inside a stream capture
// (when the look-back area, one word per tile and digit, was not sized before
// it), sorts above RS_BIG always do.  Either tier gives the same order.
constexpr int64_t RS_MID = int64_t(1) << DCSR_RS_MID_LOG2;
constexpr int64_t RS_BIG = int64_t(1) << 25;

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

template <int RS_ITEMS>
__global__ void __launch_bounds__(RS_THREADS) k_radix_hist(const unsigned long long *keys, int64_t n, int shift,
                                                            long long *ghist, int64_t ntiles) {
  constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
  __shared__ unsigned h[RS_BINS];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = (int64_t)blockIdx.x * RS_TILE + (int64_t)warp * (32 * RS_ITEMS);
#pragma unroll 4
  for (int j = 0; j < RS_ITEMS; j++) {
    int64_t i = base + j * 32 + lane;
    unsigned d = i < n ? (unsigned)((keys[i] >> shift) & 0xff) : 0x100u;
    unsigned peers = __match_any_sync(FULL, d);
    if (d < 0x100u && (__ffs(peers) - 1) == lane) atomicAdd(&h[d], (unsigned)__popc(peers));
  }
  __syncthreads();
  ghist[(int64_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

template <int RS_ITEMS>
__global__ void __launch_bounds__(RS_THREADS) k_radix_scatter(const unsigned long long *keys, const unsigned *vals,
                                                               unsigned long long *keys_out, unsigned *vals_out,
                                                               int64_t n, int shift, const long long *goff,
                                                               int64_t ntiles) {
  constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
  __shared__ unsigned wcnt[RS_WARPS][RS_BINS];
  __shared__ long long boff[RS_BINS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int w = 0; w < RS_WARPS; w++) wcnt[w][threadIdx.x] = 0;
  boff[threadIdx.x] = goff[(int64_t)threadIdx.x * ntiles + blockIdx.x];
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * RS_TILE + (int64_t)warp * (32 * RS_ITEMS);
  unsigned long long k[RS_ITEMS];
  unsigned rank[RS_ITEMS];
  const unsigned lt = lanemask_lt();
#pragma unroll
  for (int j = 0; j < RS_ITEMS; j++) {
    int64_t i = base + j * 32 + lane;
    k[j] = i < n ? keys[i] : ~0ull;
    unsigned d = i < n ? (unsigned)((k[j] >> shift) & 0xff) : 0x100u;
    unsigned peers = __match_any_sync(FULL, d);
    unsigned pre = d < 0x100u ? wcnt[warp][d] : 0u;
    rank[j] = pre + __popc(peers & lt);
    __syncwarp();
    if (d < 0x100u && (__ffs(peers) - 1) == lane) wcnt[warp][d] = pre + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  {  // exclusive prefix across warps per digit
    unsigned run = 0;
    for (int w = 0; w < RS_WARPS; w++) {
      unsigned t = wcnt[w][threadIdx.x];
      wcnt[w][threadIdx.x] = run;
      run += t;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < RS_ITEMS; j++) {
    int64_t i = base + j * 32 + lane;
    if (i < n) {
      unsigned d = (unsigned)((k[j] >> shift) & 0xff);
      int64_t pos = boff[d] + wcnt[warp][d] + rank[j];
      keys_out[pos] = k[j];
      vals_out[pos] = vals[i];
    }
  }
}

// Digit histograms of every pass (keys read once), into the look-back
// area's histogram table (zero on entry: the previous sort's last pass left
// it cleared); the last block turns each pass's counts into the digits' first
// positions.
__global__ void __launch_bounds__(RS_THREADS) k_radix_hist_all(const unsigned long long *keys, int64_t n,
                                                                int passes, Lookback lb) {
  __shared__ unsigned h[8 * RS_BINS];
  for (int i = threadIdx.x; i < 8 * RS_BINS; i += RS_THREADS) h[i] = 0;
  __syncthreads();
  constexpr int U = 4;  // keys in flight per thread
  const int64_t stride = (int64_t)gridDim.x * RS_THREADS;
  for (int64_t i = (int64_t)blockIdx.x * RS_THREADS + threadIdx.x; i < n; i += U * stride) {
    unsigned long long k[U];
#pragma unroll
    for (int u = 0; u < U; u++) k[u] = i + u * stride < n ? __ldg(keys + i + u * stride) : 0ull;
#pragma unroll
    for (int u = 0; u < U; u++)
      if (i + u * stride < n) {
#pragma unroll
        for (int p = 0; p < 8; p++)
          if (p < passes) atomicAdd(&h[p * RS_BINS + (unsigned)((k[u] >> (8 * p)) & 0xff)], 1u);
      }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * RS_BINS; i += RS_THREADS)
    if (h[i]) atomicAdd(lb.hist + i, h[i]);
  __threadfence();
  if (lb_end(lb)) {
    static_assert(RS_THREADS == RS_BINS, "a thread per digit");
    __threadfence();
    for (int p = 0; p < passes; p++) {
      int all;
      const int c = (int)__ldcg(lb.hist + p * RS_BINS + threadIdx.x);
      lb.hist[p * RS_BINS + threadIdx.x] = (unsigned)block_excl_scan(c, &all);
    }
    if (threadIdx.x == 0) *(volatile unsigned *)lb.done = 0;
  }
}

// Ranks of a warp's IT items (digit dg(j) of item j*32 + lane, for ok(j))
// among the warp's items of the same digit, in input order; cnt (RS_BINS
// counters, zero on entry) receives the warp's digit counts.  The lanes with
// the same digit are found through a table of lane masks in shared memory
// (RS_BINS words of the warp's own, zero on entry and on return): about ten
// instructions, against forty for a ballot per bit; match_any ran at half the
// ballots' speed.
template <int IT, typename C, typename D, typename O>
__device__ __forceinline__ void warp_digit_ranks(D &&dg, O &&ok, unsigned (&rank)[IT], C *cnt, unsigned *mask) {
  const unsigned lt = lanemask_lt(), me = 1u << lane_id();
#pragma unroll
  for (int j = 0; j < IT; j++) {
    const bool v = ok(j);
    const unsigned d = dg(j);
    if (v) atomicOr(&mask[d], me);
    __syncwarp();
    const unsigned peers = v ? mask[d] : 0u, pre = v ? cnt[d] : 0u;
    const unsigned below = peers & lt;
    rank[j] = pre + __popc(below);
    __syncwarp();
    if (v && below == 0) {
      cnt[d] = (C)(pre + __popc(peers));
      mask[d] = 0;
    }
    __syncwarp();
  }
}

#ifndef DCSR_OS_MINB
#define DCSR_OS_MINB 3
#endif
// One pass of the mid tier (a thread owns a digit in the middle).  PACK: keys_in holds key << ib | index words, or (FIRST) the bare
// keys, packed here with their input positions; LAST unpacks to keys_out and
// vals_out.  Not PACK: keys and indices side by side.
template <int TH, int IT, bool PACK, bool FIRST, bool LAST>
__global__ void __launch_bounds__(TH, DCSR_OS_MINB) k_radix_onesweep(const unsigned long long *__restrict__ keys,
                                                           const unsigned *__restrict__ vals,
                                                           unsigned long long *__restrict__ keys_out,
                                                           unsigned *__restrict__ vals_out, int64_t n, int pass,
                                                           int ib, int last_pass, Lookback lb) {
  constexpr int TILE = TH * IT, WARPS = TH / 32;
  static_assert(TH == RS_BINS, "a thread per digit");
  static_assert(TILE >= 2 * WARPS * RS_BINS * 4 / 8, "rank tables fit the tile's room");
  extern __shared__ __align__(16) unsigned char os_sm[];
  unsigned long long *sw = reinterpret_cast<unsigned long long *>(os_sm);  // the tile in digit order
  unsigned *sv = reinterpret_cast<unsigned *>(sw + TILE);                   // (not PACK) its indices
  unsigned(*mask)[RS_BINS] = reinterpret_cast<unsigned(*)[RS_BINS]>(os_sm);  // lane masks, before the tile is there
  __shared__ unsigned wcnt[WARPS][RS_BINS];
  __shared__ unsigned dstart[RS_BINS];  // a digit's first position in the ordered tile
  __shared__ int goff[RS_BINS];         // its output position less that
  __shared__ unsigned sh_tile;
  __shared__ unsigned long long sh_ep;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, d = threadIdx.x;
  lb_begin(lb, &sh_tile, &sh_ep);
  for (int i = lane; i < RS_BINS; i += 32) {
    wcnt[warp][i] = 0;
    mask[warp][i] = 0;
  }
  const unsigned gbase = __ldcg(lb.hist + pass * RS_BINS + d);
  __syncthreads();
  const int64_t t = sh_tile;
  const unsigned long long e = sh_ep;
  if (t >= gridDim.x) {  // a tile counter left non-zero (a bug): report it, touch nothing
    if (threadIdx.x == 0) lb_give_up(lb, e);
    if (lb_end(lb)) lb_advance(lb);
    return;
  }
  const int64_t t0 = t * TILE;
  const int cnt = n - t0 < TILE ? (int)(n - t0) : TILE;
  const int wbase = warp * (32 * IT) + lane;
  const int shift = 8 * pass + (PACK ? ib : 0);
  unsigned long long k[IT];
  unsigned val[PACK ? 1 : IT];
#pragma unroll
  for (int j = 0; j < IT; j++) {
    const int p = wbase + 32 * j;
    k[j] = 0;
    if constexpr (!PACK) val[j] = 0;
    if (p < cnt) {
      k[j] = __ldcs(keys + t0 + p);
      if constexpr (!PACK) val[j] = __ldcs(vals + t0 + p);
      if constexpr (PACK && FIRST) k[j] = (k[j] << ib) | (unsigned long long)(t0 + p);
    }
  }
  auto digit = [&](int j) { return (unsigned)(k[j] >> shift) & 0xffu; };
  auto valid = [&](int j) { return wbase + 32 * j < cnt; };
  unsigned rank[IT];
  warp_digit_ranks<IT>(digit, valid, rank, wcnt[warp], mask[warp]);
  __syncthreads();
  unsigned run = 0;  // exclusive prefix across warps per digit; run = the tile's count of digit d
  const int64_t slot = t * RS_BINS + d;
  const unsigned tag2 = (unsigned)(e & LB_EMASK) << 2;  // a current look-back word's upper half, less its kind
  auto publish = [&](unsigned kind, unsigned v) {
    *(volatile unsigned long long *)(lb.flag + slot) = ((unsigned long long)(tag2 | kind) << 32) | v;
  };
#pragma unroll
  for (int w = 0; w < WARPS; w++) {
    const unsigned c = wcnt[w][d];
    wcnt[w][d] = run;
    run += c;
  }
  // published before the tile is put in order: later tiles can look back
  if (t > 0) publish(1, run);
  else if (!lb.g->stall) publish(2, run);
  unsigned all;
  const unsigned ds = block_excl_scan(run, &all);
  dstart[d] = ds;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < IT; j++) {
    if (valid(j)) {
      const unsigned dg = digit(j);
      const unsigned lp = dstart[dg] + wcnt[warp][dg] + rank[j];
      sw[lp] = k[j];
      if constexpr (!PACK) sv[lp] = val[j];
    }
  }
  // items of digit d in the tiles before this one: look back over windows of
  // LB_W earlier tiles (their flags loaded together), consuming published
  // aggregates up to the nearest published inclusive prefix
  {
    unsigned excl = 0;
    if (t > 0) {
      const int limit = lb.g->spin_limit;
      int q = (int)t - 1, idle = 0;
      bool done = false;
      while (!done) {
        const unsigned long long *f0 = lb.flag + (int64_t)q * RS_BINS + d;
        unsigned long long f[LB_W];
#pragma unroll
        for (int j = 0; j < LB_W; j++)  // before tile 0: an inclusive prefix of 0
          f[j] = q >= j ? ld_vol(f0 - j * RS_BINS) : (unsigned long long)(tag2 | 2u) << 32;
        int used = 0;
        bool live = true;
#pragma unroll
        for (int j = 0; j < LB_W; j++) {
          const unsigned kind = (unsigned)(f[j] >> 32) - tag2;  // 1, 2, or not published in this epoch
          live = live && kind - 1u < 2u;
          if (live) {
            excl += (unsigned)f[j];
            used = j + 1;
            done = kind == 2u;
            live = !done;
          }
        }
        q -= used;
        if (used == 0) {  // the nearest tile has not published yet
          if (++idle >= limit || ((idle & 1023) == 1023 && lb_faulted(lb, e))) {
            lb_give_up(lb, e);
            break;
          }
          if (idle >= 32) __nanosleep(64);
        }
      }
      publish(2, excl + run);
    }
    goff[d] = (int)(gbase + excl - ds);
  }
  __syncthreads();
  const unsigned long long imask = (1ull << ib) - 1;
#pragma unroll
  for (int j = 0; j < IT; j++) {
    const int lp = j * TH + threadIdx.x;
    if (lp < cnt) {
      const unsigned long long w = sw[lp];
      const unsigned pos = (unsigned)(goff[(unsigned)(w >> shift) & 0xffu] + lp);
      if constexpr (PACK && LAST) {
        keys_out[pos] = w >> ib;
        vals_out[pos] = (unsigned)(w & imask);
      } else {
        keys_out[pos] = w;
        if constexpr (!PACK) vals_out[pos] = sv[lp];
      }
    }
  }
  if (lb_end(lb)) {
    if (last_pass)  // leave the histogram table cleared for the next sort
      for (int i = threadIdx.x; i < 8 * RS_BINS; i += TH) lb.hist[i] = 0;
    __syncthreads();
    lb_advance(lb);
  }
}

// Small inputs (n <= RS_SMALL, key and a 13-bit index within 64 bits): one
// 1024-thread block keeps IT packed words per thread in registers and runs
// every pass as rank (per-warp digit counters), prefix over warps and digits,
// scatter to and reload from shared memory.  8192 keys of 24 bits: 56 us with
// eight rounds of 1024 items per pass before.
constexpr int RS_SMALL = 8192;
constexpr int RS_SMALL_BITS = 13;
constexpr int RS_SMALL_T = 1024;

template <int IT>
__global__ void __launch_bounds__(RS_SMALL_T) k_radix_small(const unsigned long long *__restrict__ keys,
                                                            unsigned long long *__restrict__ keys_out,
                                                            unsigned *__restrict__ vals_out, int n, int bits) {
  constexpr int WARPS = RS_SMALL_T / 32, TILE = RS_SMALL_T * IT;
  extern __shared__ __align__(16) unsigned char rs_sm[];
  unsigned long long *sw = reinterpret_cast<unsigned long long *>(rs_sm);
  unsigned *mask = reinterpret_cast<unsigned *>(sw + TILE);                      // [WARPS][RS_BINS] lane masks
  unsigned short *wc = reinterpret_cast<unsigned short *>(mask + WARPS * RS_BINS);  // [WARPS][RS_BINS] counts
  __shared__ unsigned quad[4][RS_BINS];  // digit counts of each quarter of the warps
  __shared__ unsigned dstart[RS_BINS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wbase = warp * (32 * IT) + lane;
  const unsigned long long imask = (1ull << RS_SMALL_BITS) - 1;
  unsigned long long k[IT];
#pragma unroll
  for (int j = 0; j < IT; j++) {
    const int p = wbase + 32 * j;
    k[j] = p < n ? (keys[p] << RS_SMALL_BITS) | (unsigned long long)p : ~0ull;
  }
  for (int i = tid; i < WARPS * RS_BINS; i += RS_SMALL_T) mask[i] = 0;
  for (int shift = RS_SMALL_BITS; shift < bits + RS_SMALL_BITS; shift += 8) {
    unsigned *wz = reinterpret_cast<unsigned *>(wc);
    for (int i = tid; i < WARPS * RS_BINS / 2; i += RS_SMALL_T) wz[i] = 0;
    __syncthreads();
    auto digit = [&](int j) { return (unsigned)(k[j] >> shift) & 0xffu; };
    auto valid = [&](int j) { return wbase + 32 * j < n; };
    unsigned rank[IT];
    warp_digit_ranks<IT>(digit, valid, rank, wc + warp * RS_BINS, mask + warp * RS_BINS);
    __syncthreads();
    // prefix over the warps: a thread per digit and quarter of the warps
    const int dd = tid & (RS_BINS - 1), q = tid >> 8;
    unsigned run = 0;
#pragma unroll
    for (int w = 0; w < WARPS / 4; w++) {
      unsigned short *c = wc + (q * (WARPS / 4) + w) * RS_BINS + dd;
      const unsigned x = *c;
      *c = (unsigned short)run;
      run += x;
    }
    quad[q][dd] = run;
    __syncthreads();
    if (warp == 0) {  // digit totals (8 per lane) -> first positions; quarters -> their offsets
      unsigned tot[8], sum = 0;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        unsigned c[4], o = 0;
#pragma unroll
        for (int x = 0; x < 4; x++) {
          c[x] = quad[x][lane * 8 + j];
          quad[x][lane * 8 + j] = o;
          o += c[x];
        }
        tot[j] = o;
        sum += o;
      }
      unsigned ex = warp_incl_scan(sum) - sum;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        dstart[lane * 8 + j] = ex;
        ex += tot[j];
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < IT; j++)
      if (valid(j)) {
        const unsigned dg = digit(j);
        sw[dstart[dg] + quad[warp / (WARPS / 4)][dg] + wc[warp * RS_BINS + dg] + rank[j]] = k[j];
      }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < IT; j++) k[j] = wbase + 32 * j < n ? sw[wbase + 32 * j] : ~0ull;
    // (the next pass syncs before it writes the shared words)
  }
#pragma unroll
  for (int j = 0; j < IT; j++) {
    const int p = wbase + 32 * j;
    if (p < n) {
      keys_out[p] = k[j] >> RS_SMALL_BITS;
      vals_out[p] = (unsigned)(k[j] & imask);
    }
  }
}

size_t radix_scratch_bytes(int64_t n) {
  if (n <= RS_MID) return 0;
  return arena_bytes(div_up(n, RS_THREADS * 16) * RS_BINS, 8);
}

// Items per thread of the single-pass scatter's tiles.
#ifndef DCSR_OS_I
#define DCSR_OS_I 16
#endif
constexpr int OS_I = DCSR_OS_I, OS_T = RS_BINS;
constexpr int OS_TILE = OS_T * OS_I;

size_t lookback_slots(int64_t n) {
  // single-pass sorts: one slot per (tile, digit); larger ones: the scan of
  // their histogram table; scans: a two-slot word per (smallest) tile
  const int64_t sort = n <= RS_BIG ? div_up(n, OS_TILE) * RS_BINS
                                   : LB_SCAN_WORDS * div_up(div_up(n, RS_THREADS * 16) * RS_BINS, SCAN_TILE);
  return (size_t)(std::max<int64_t>(sort, LB_SCAN_WORDS * div_up(n, SM_THREADS * SM_HEAVY)) + 1);
}

// Large inputs: three kernels per pass (tile histograms, table scan, scatter).
static int radix_passes_table(unsigned long long **keys, unsigned **vals, unsigned long long **keys_tmp,
                              unsigned **vals_tmp, int64_t n, int bits, Arena &ar, cudaStream_t s) {
  constexpr int ITEMS = 16;
  const int64_t nt = div_up(n, RS_THREADS * ITEMS);
  size_t mark = ar.used;
  long long *hist = ar.take<long long>(nt * RS_BINS);
  if (ar.overflow) return DCSR_OOM;  // scratch sizing bug: no kernel sees a null pointer
  for (int shift = 0; shift < bits; shift += 8) {
    DCSR_LAUNCH(k_radix_hist<ITEMS>, (unsigned)nt, RS_THREADS, 0, s, *keys, n, shift, hist, nt);
    DCSR_TRY(scan_i64(hist, hist, nt * RS_BINS, nullptr, ar, s));
    DCSR_LAUNCH(k_radix_scatter<ITEMS>, (unsigned)nt, RS_THREADS, 0, s, *keys, *vals, *keys_tmp, *vals_tmp, n,
                shift, hist, nt);
    unsigned long long *tk = *keys;
    *keys = *keys_tmp;
    *keys_tmp = tk;
    unsigned *tv = *vals;
    *vals = *vals_tmp;
    *vals_tmp = tv;
  }
  ar.used = mark;
  return DCSR_OK;
}

template <bool PACK, bool FIRST, bool LAST>
static int launch_onesweep(const unsigned long long *ki, const unsigned *vi, unsigned long long *ko, unsigned *vo,
                           int64_t n, int pass, int ib, bool last, const Lookback &lb, cudaStream_t s) {
  constexpr size_t smem = (size_t)OS_TILE * (PACK ? 8 : 12);
  static const cudaError_t attr = cudaFuncSetAttribute(k_radix_onesweep<OS_T, OS_I, PACK, FIRST, LAST>,
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  DCSR_CUDA(attr);
  DCSR_LAUNCH((k_radix_onesweep<OS_T, OS_I, PACK, FIRST, LAST>), (unsigned)div_up(n, OS_TILE), OS_T, smem, s, ki, vi, ko,
              vo, n, pass, ib, last ? 1 : 0, lb);
  return DCSR_OK;
}

// Mid-size inputs: one histogram kernel, then one single-pass scatter per pass.
static int radix_passes_onesweep(unsigned long long **keys, unsigned **vals, unsigned long long **keys_tmp,
                                 unsigned **vals_tmp, int64_t n, int bits, Arena &ar, cudaStream_t s) {
  const int passes = (int)div_up(bits, 8), ib = bits_for(n);
  if (passes <= 0) return DCSR_OK;
  const bool pack = bits + ib <= 64;
  Lookback lb;
  DCSR_TRY(ar.lookback((size_t)(div_up(n, OS_TILE) * RS_BINS), s, &lb));
  const int gh = (int)std::min<int64_t>(div_up(n, RS_THREADS * 8), 6 * sm_count());
  DCSR_LAUNCH(k_radix_hist_all, gh, RS_THREADS, 0, s, *keys, n, passes, lb);
  for (int p = 0; p < passes; p++) {
    const bool first = p == 0, last = p == passes - 1;
    if (!pack)
      DCSR_TRY((launch_onesweep<false, false, false>(*keys, *vals, *keys_tmp, *vals_tmp, n, p, 0, last, lb, s)));
    else if (first && last)
      DCSR_TRY((launch_onesweep<true, true, true>(*keys, *vals, *keys_tmp, *vals_tmp, n, p, ib, last, lb, s)));
    else if (first)
      DCSR_TRY((launch_onesweep<true, true, false>(*keys, *vals, *keys_tmp, *vals_tmp, n, p, ib, last, lb, s)));
    else if (last)
      DCSR_TRY((launch_onesweep<true, false, true>(*keys, *vals, *keys_tmp, *vals_tmp, n, p, ib, last, lb, s)));
    else
      DCSR_TRY((launch_onesweep<true, false, false>(*keys, *vals, *keys_tmp, *vals_tmp, n, p, ib, last, lb, s)));
    std::swap(*keys, *keys_tmp);
    if (!pack || last) std::swap(*vals, *vals_tmp);
  }
  return DCSR_OK;
}

template <int IT>
static int launch_small(const unsigned long long *ki, unsigned long long *ko, unsigned *vo, int64_t n, int bits,
                        cudaStream_t s) {
  constexpr size_t smem = (size_t)RS_SMALL_T * IT * 8 + RS_SMALL_T / 32 * RS_BINS * 6;
  static const cudaError_t attr =
      cudaFuncSetAttribute(k_radix_small<IT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  DCSR_CUDA(attr);
  DCSR_LAUNCH(k_radix_small<IT>, 1, RS_SMALL_T, smem, s, ki, ko, vo, (int)n, bits);
  return DCSR_OK;
}

int radix_sort_pairs(unsigned long long **keys, unsigned **vals, unsigned long long **keys_tmp,
                     unsigned **vals_tmp, int64_t n, int bits, Arena &ar, cudaStream_t s) {
  if (n <= 1) return DCSR_OK;
  if (n <= RS_SMALL && bits + RS_SMALL_BITS <= 64) {
    if (n <= RS_SMALL_T) DCSR_TRY(launch_small<1>(*keys, *keys_tmp, *vals_tmp, n, bits, s));
    else if (n <= 2 * RS_SMALL_T) DCSR_TRY(launch_small<2>(*keys, *keys_tmp, *vals_tmp, n, bits, s));
    else if (n <= 4 * RS_SMALL_T) DCSR_TRY(launch_small<4>(*keys, *keys_tmp, *vals_tmp, n, bits, s));
    else DCSR_TRY(launch_small<8>(*keys, *keys_tmp, *vals_tmp, n, bits, s));
    std::swap(*keys, *keys_tmp);
    std::swap(*vals, *vals_tmp);
    return DCSR_OK;
  }
  if (n <= RS_MID) return radix_passes_onesweep(keys, vals, keys_tmp, vals_tmp, n, bits, ar, s);
  if (n <= RS_BIG) {
    bool fits = ar.lb && ar.lb_slots >= (size_t)(div_up(n, OS_TILE) * RS_BINS);
    if (!fits) {  // the area is grown on demand, but not inside a capture
      cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
      DCSR_CUDA(cudaStreamIsCapturing(s, &cs));
      fits = cs == cudaStreamCaptureStatusNone;
    }
    if (fits) return radix_passes_onesweep(keys, vals, keys_tmp, vals_tmp, n, bits, ar, s);
  }
  return radix_passes_table(keys, vals, keys_tmp, vals_tmp, n, bits, ar, s);
}

// ------------------------------------------------- public segmented ops

// X[I[n]] += run length, one atomic per run (runs found with warp ballots).
__global__ void k_count_sorted(const int32_t *I, int64_t n, int32_t *X) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < n; base += stride) {
    int64_t i = base + threadIdx.x;
    int32_t key = i < n ? I[i] : INT32_MIN;
    int32_t prev = __shfl_up_sync(FULL, key, 1);
    const int lane = threadIdx.x & 31;
    if (lane == 0) prev = (i > 0 && i < n) ? I[i - 1] : INT32_MIN;
    bool head = i < n && (key != prev || lane == 0);
    unsigned hm = __ballot_sync(FULL, head);
    unsigned valid = __ballot_sync(FULL, i < n);
    if (head) {
      unsigned later = hm & ~((2u << lane) - 1u);
      int end = later ? (__ffs(later) - 1) : (32 - __clz(valid));
      atomicAdd(&X[key], end - lane);
    }
  }
}

// Reduce-by-key: heads flagged, head positions compacted by scan.  A run is
// summed in pieces of at most RBK_PIECE keys (a piece starts at the run's
// head or at a multiple of RBK_PIECE inside the run), each piece left to
// right by one thread; the thread at the head writes its piece's sum and the
// pieces that continue a run leave theirs in cpart; a second kernel adds a
// run's continuation pieces to its head piece in order.  The order of the
// additions is fixed by the input alone, so results are deterministic, and no
// thread sums more than RBK_PIECE values (a run of 2^20 equal keys is summed
// by 4096 threads, then 4096 partials by one).
constexpr int64_t RBK_PIECE = 256;
__global__ void k_rbk_flags(const int32_t *keys, int64_t n, long long *flag) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) flag[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1 : 0;
}
template <typename V>
__global__ void k_rbk_emit(const int32_t *keys, const V *vals, int64_t n, const long long *pos,
                           int32_t *keys_out, V *vals_out, V *cpart) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const bool head = i == 0 || keys[i] != keys[i - 1];
  if (!head && i % RBK_PIECE != 0) return;
  const int64_t end = (i / RBK_PIECE + 1) * RBK_PIECE < n ? (i / RBK_PIECE + 1) * RBK_PIECE : n;
  V acc = vals[i];
  for (int64_t j = i + 1; j < end && keys[j] == keys[i]; j++) acc = acc + vals[j];
  if (head) {
    keys_out[pos[i]] = keys[i];
    vals_out[pos[i]] = acc;
  } else {
    cpart[i / RBK_PIECE] = acc;
  }
}
// One thread per piece boundary b = s * RBK_PIECE (s >= 1): the owner of a
// run that crosses b is the boundary whose previous piece holds the run's
// head; it adds the run's continuation pieces s, s+1, ... to the head piece.
template <typename V>
__global__ void k_rbk_fix(const int32_t *keys, int64_t n, const long long *pos, V *vals_out, const V *cpart) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int64_t b = s * RBK_PIECE;
  if (b >= n || keys[b] != keys[b - 1]) return;       // no run crosses b
  if (pos[b] == pos[b - RBK_PIECE]) return;  // no head in [b - RBK_PIECE, b): an earlier boundary owns the run
  const int64_t out = pos[b] - 1;  // the run's output slot (heads before b, minus one)
  V acc = vals_out[out];
  const int32_t key = keys[b];
  for (int64_t t = s; t * RBK_PIECE < n; t++) {
    if (keys[t * RBK_PIECE] != key) break;  // the run ended before this piece (keys are sorted)
    acc = acc + cpart[t];
  }
  vals_out[out] = acc;
}

template <typename V>
static int rbk_launch(const int32_t *keys, const V *vals, int64_t n, long long *pos, long long *n_out, int32_t *keys_out,
                      V *vals_out, V *cpart, Arena &ar, cudaStream_t s) {
  const unsigned g = (unsigned)div_up(n, 256);
  DCSR_LAUNCH(k_rbk_flags, g, 256, 0, s, keys, n, pos);
  DCSR_TRY(scan_i64(pos, pos, n, n_out, ar, s));
  DCSR_LAUNCH(k_rbk_emit<V>, g, 256, 0, s, keys, vals, n, pos, keys_out, vals_out, cpart);
  const int64_t nb = (n - 1) / RBK_PIECE;  // piece boundaries inside [1, n)
  if (nb > 0) DCSR_LAUNCH(k_rbk_fix<V>, (unsigned)div_up(nb, 256), 256, 0, s, keys, n, pos, vals_out, cpart);
  return DCSR_OK;
}

// ------------------------------------------- allocation-free reduce-by-key
//
// Scratch for dcsr_reduce_by_key_noalloc: head positions (one int64 per key),
// the continuation-piece partials and the scan's look-back area, in one
// static device array (zero at module
// load, as the look-back protocol needs).  Every GPU that loads the library
// holds it until exit.  Host code must not pass the symbol itself to a
// kernel (in host code it names a host-side stand-in); the device address is
// looked up once per device.
constexpr size_t NOALLOC_POS_BYTES = (size_t)DCSR_NOALLOC_MAX_KEYS * sizeof(long long);
constexpr size_t NOALLOC_PART_BYTES = (size_t)(DCSR_NOALLOC_MAX_KEYS / RBK_PIECE + 1) * sizeof(double);
constexpr size_t NOALLOC_LB_SLOTS = LB_SCAN_WORDS * ((DCSR_NOALLOC_MAX_KEYS + SCAN_TILE - 1) / SCAN_TILE) + 4;
// (a multiple of 256: the look-back area behind it holds 16-byte words)
constexpr size_t NOALLOC_ARENA_BYTES = (NOALLOC_POS_BYTES + 256 + NOALLOC_PART_BYTES + 256 + 255) / 256 * 256;
static_assert(NOALLOC_LB_SLOTS % 2 == 0, "the scans' words start on 16 bytes");
constexpr size_t NOALLOC_BYTES = NOALLOC_ARENA_BYTES + lb_bytes(NOALLOC_LB_SLOTS);
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_BYTES];

static int noalloc_scratch(void **out) {
  static std::mutex mu;
  static void *ptr[128] = {};
  int dev = 0;
  DCSR_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 128) return DCSR_NOT_SUPPORTED;
  std::lock_guard<std::mutex> lock(mu);
  if (!ptr[dev]) {
    void *p = nullptr;
    DCSR_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    ptr[dev] = p;
  }
  *out = ptr[dev];
  return DCSR_OK;
}

}  // namespace dcsr

using namespace dcsr;

extern "C" int dcsr_reduce_by_key_noalloc(const int32_t *keys, const void *vals, int64_t n, int32_t dtype,
                                          int32_t *keys_out, void *vals_out, int64_t *n_out, void *stream) {
  if (n < 0 || n > DCSR_NOALLOC_MAX_KEYS || (dtype != DCSR_F32 && dtype != DCSR_F64) || !n_out ||
      (n > 0 && (!keys || !vals || !keys_out || !vals_out)))
    return DCSR_BAD_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (n == 0) {
    DCSR_CUDA(cudaMemsetAsync(n_out, 0, sizeof(int64_t), s));
    return DCSR_OK;
  }
  void *base = nullptr;
  DCSR_TRY(noalloc_scratch(&base));
  Arena ar;  // a view over the static array: take() and lookback() only, never reserve()/release()
  ar.base = (char *)base;
  ar.cap = NOALLOC_ARENA_BYTES;
  ar.used = 0;
  ar.lb = (unsigned char *)base + NOALLOC_ARENA_BYTES;
  ar.lb_slots = NOALLOC_LB_SLOTS;
  // every word below is written before it is read in each call: positions
  // by the flag kernel, a partial by the piece that owns it
  long long *pos = ar.take<long long>(n);
  double *cpart = ar.take<double>(n / RBK_PIECE + 1);
  if (ar.overflow) return DCSR_OOM;  // scratch sizing bug: no kernel sees a null pointer
  if (dtype == DCSR_F32)
    return rbk_launch<float>(keys, (const float *)vals, n, pos, (long long *)n_out, keys_out, (float *)vals_out,
                             (float *)cpart, ar, s);
  return rbk_launch<double>(keys, (const double *)vals, n, pos, (long long *)n_out, keys_out, (double *)vals_out,
                            cpart, ar, s);
}

extern "C" int dcsr_count_sorted_indices(const int32_t *I, int64_t n, int32_t *X, void *stream) {
  if (n < 0 || (n > 0 && (!I || !X))) return DCSR_BAD_ARG;
  if (n == 0) return DCSR_OK;
  cudaStream_t s = (cudaStream_t)stream;
  int grid = (int)std::min<int64_t>(div_up(n, 256), (int64_t)sm_count() * 8);
  DCSR_LAUNCH(k_count_sorted, grid, 256, 0, s, I, n, X);
  return DCSR_OK;
}

extern "C" int dcsr_reduce_by_key(const int32_t *keys, const void *vals, int64_t n, int32_t dtype, int32_t *keys_out,
                                  void *vals_out, int64_t *n_out, void *stream) {
  if (n < 0 || (dtype != DCSR_F32 && dtype != DCSR_F64)) return DCSR_BAD_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (n == 0) {
    if (n_out) DCSR_CUDA(cudaMemsetAsync(n_out, 0, sizeof(int64_t), s));
    return DCSR_OK;
  }
  Arena ar;
  DCSR_TRY(ar.reserve(arena_bytes(n, 8) + arena_bytes(n / RBK_PIECE + 1, 8) + scan_scratch_bytes(n), s));
  long long *pos = ar.take<long long>(n);
  double *cpart = ar.take<double>(n / RBK_PIECE + 1);
  if (ar.overflow) return DCSR_OOM;  // scratch sizing bug: no kernel sees a null pointer
  const int rc = dtype == DCSR_F32 ? rbk_launch<float>(keys, (const float *)vals, n, pos, (long long *)n_out, keys_out,
                                                       (float *)vals_out, (float *)cpart, ar, s)
                                   : rbk_launch<double>(keys, (const double *)vals, n, pos, (long long *)n_out,
                                                        keys_out, (double *)vals_out, cpart, ar, s);
  ar.release(s);
  return rc;
}
