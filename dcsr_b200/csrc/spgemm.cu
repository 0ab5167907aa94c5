// spgemm.cu -- C = A*B for DCSR matrices (expand - sort - reduce).
//
// 1. count   products per row P_i = sum_{k in A_i} |B_k|, rows per size class
//            (reference CalcSortSizes_SPMM / SetBins_SPMM include/spmm.inl:951-1061)
// 2. stage   one scan: per-row staging offsets, C's pool bound
// 3. numeric per row: expand products a_ik*b_kj tagged with their product
//            index p, sort by (column, p), sum equal columns left to right,
//            write unique columns to the staging area:
//              P_i <= 256   warp per row, bitonic sort in registers
//              P_i <= 1024  the same, 16 or 32 keys a lane, where column and p
//                           fit 32 bits (columns of up to 22 bits)
//              P_i <= 4096  CTA per row, bitonic sort in shared memory
//              P_i >  4096  all such rows together: global stable radix sort
//                           of (row, column) keys (no row is skipped; the
//                           reference left rows > 2048 products uncomputed,
//                           include/spmm.h:368-389)
//            The warp classes take the rows in row order and pass over those
//            of other classes; the upper two have lists, built only where
//            there are such rows (a sort of all rows by class and its
//            searches cost 42 us of a product of 131072 rows).
// 4. layout  C's rows placed straight from the staging area into C's pool
//            with C's slack policy; the pool is allocated at an upper bound
//            (the policy capacity of P_i per row) so nothing waits for the
//            unique counts.  Two synchronisations (three with rows of the upper
//            two classes, whose lists are checked): the product counts (to size
//            the staging area) and C's pool top.
// Sorting by (column, p) makes every sum run in product order, so values are
// reproducible and match the CPU oracle bit for bit; explicit zeros are kept
// (reference include/spmm.inl:215-218).
#include <algorithm>

#include "internal.cuh"
#include "lookback.cuh"

namespace dcsr {

constexpr int SG_THREADS = 256;
constexpr int SG_WARP_MAX = 256;   // products per warp-row
constexpr int SG_WARP4_MAX = 1024; // products per warp-row of the class above (columns of up to 22 bits)
constexpr int SG_CTA_MAX = 4096;   // products per CTA-row
enum { SG_EMPTY = 0, SG_WARP = 1, SG_WARP4 = 2, SG_CTA = 3, SG_GLOBAL = 4, SG_CLASSES = 5 };
// Result words: the rows of each class, then
enum { SG_R_GPROD = SG_CLASSES, SG_R_PROD, SG_R_CAPS, SG_R_STATUS, SG_R_NEXT, SG_R_NEXT4, SG_R_WORDS = 16 };

__host__ __device__ __forceinline__ int sg_class(int64_t p, int warp_max) {
  return p == 0 ? SG_EMPTY : p <= SG_WARP_MAX ? SG_WARP : p <= warp_max ? SG_WARP4 : p <= SG_CTA_MAX ? SG_CTA : SG_GLOBAL;
}

// Per row its product count P_i; per class the number of rows, and the
// products of the global class's.
template <typename V>
__global__ void __launch_bounds__(SG_THREADS) k_sg_count(Mat<V> A, Mat<V> B, int warp_max, long long *cnt,
                                                         long long *res) {
  constexpr int G = 8;  // lanes per row: a warp has four rows' loads in flight
  __shared__ unsigned rows[SG_CLASSES];
  __shared__ unsigned long long gprod;
  if (threadIdx.x < SG_CLASSES) rows[threadIdx.x] = 0;
  if (threadIdx.x == 0) gprod = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, j = lane & (G - 1);
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (32 / G); i0 < A.n_rows;
       i0 += nw * (32 / G)) {
    const int64_t i = i0 + lane / G;
    long long s = 0;
    if (i < A.n_rows) {
      const Chain ch = load_chain(A, (int32_t)i);
      const int64_t L = A.row_sizes[i];
      for (int64_t p = j; p < L; p += G) s += B.row_sizes[A.cols[ch.phys(p)]];
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
    if (j == 0 && i < A.n_rows) {
      cnt[i] = s;
      const int c = sg_class(s, warp_max);
      atomicAdd(&rows[c], 1u);
      if (c == SG_GLOBAL) atomicAdd(&gprod, (unsigned long long)s);
    }
  }
  __syncthreads();
  if (threadIdx.x < SG_CLASSES && rows[threadIdx.x])
    atomicAdd((unsigned long long *)&res[threadIdx.x], (unsigned long long)rows[threadIdx.x]);
  if (threadIdx.x == 0 && gprod) atomicAdd((unsigned long long *)&res[SG_R_GPROD], gprod);
}

// The capacities that C's layout policy gives rows of P_i entries added up (an
// upper bound of the pool, whatever the rows' unique columns), and the staging
// offsets ub (n + 1) from the product counts; no unique columns yet.  The
// products may pass the 32 bits of a second sum only where the capacities, at
// least as many, pass the pool's range: the call then ends before they are used.
struct StageScan {
  static constexpr int NS = 2, IT = SM_LIGHT;
  using T = long long;
  struct State {};
  const long long *cnt;
  dcsr_opts o;
  long long *ub, *ucnt, *res;
  int32_t n;
  __device__ __forceinline__ void load(int64_t i, bool ok, State &, T (&v)[2]) const {
    v[1] = ok ? cnt[i] : 0;
    v[0] = ok ? policy_cap(o, v[1]) : 0;
  }
  __device__ __forceinline__ void emit(int64_t i, bool ok, const State &, const long long (&p)[2],
                                       const T (&)[2]) const {
    if (ok) {
      ub[i] = p[1];
      ucnt[i] = 0;
    }
  }
  __device__ __forceinline__ void total(const long long (&t)[2]) const {
    ub[n] = t[1];
    res[SG_R_PROD] = t[1];
    res[SG_R_CAPS] = t[0];
  }
};

// The rows of the CTA class and of the global class, in row order.
struct ListScan {
  static constexpr int NS = 2, IT = SM_LIGHT;
  using T = long long;
  struct State {};
  const long long *ub;
  int warp_max;
  unsigned *cta, *global;
  __device__ __forceinline__ void load(int64_t i, bool ok, State &, T (&v)[2]) const {
    const int c = ok ? sg_class(ub[i + 1] - ub[i], warp_max) : SG_EMPTY;
    v[0] = c == SG_CTA;
    v[1] = c == SG_GLOBAL;
  }
  __device__ __forceinline__ void emit(int64_t i, bool, const State &, const long long (&p)[2],
                                       const T (&v)[2]) const {
    if (v[0]) cta[p[0]] = (unsigned)i;
    if (v[1]) global[p[1]] = (unsigned)i;
  }
  __device__ __forceinline__ void total(const long long (&)[2]) const {}
};

// Sort keys of the warp classes: (column, product index p < MAXP) packed into
// 32 bits when the column bits and p's fit, else (256 products) into 64.
template <typename K, int MAXP>
struct SgKey {
  static constexpr int S = sizeof(K) == 8 ? 32 : MAXP == 256 ? 8 : 10;
  static_assert((1 << (S < 31 ? S : 30)) >= MAXP, "p fits below the column");
  __device__ __forceinline__ static K make(int32_t col, int p) { return ((K)(uint32_t)col << S) | (K)p; }
  __device__ __forceinline__ static int32_t col(K k) { return (int32_t)(k >> S); }
  __device__ __forceinline__ static uint32_t idx(K k) { return (uint32_t)(k & ((K(1) << S) - 1)); }
};

// The warp classes' expand (P_i <= MAXP): row i's A entries are taken 32 at
// a time, one per lane, each lane loading its entry's column k and value,
// then B row k's length and segments, side by side (no load waits on another
// entry's); the B-row lengths are scanned into product offsets, and lane l
// produces products q = l, l + 32, ... of the group.  The entry owning q: when
// no B row of the group is empty, the starts within 32 products are a bit mask
// (one warp OR) and the owner is the number of starts up to q, minus one (6
// instructions against 20 of a search); else a binary search over the lanes'
// offsets.  H x 32 products' B loads are issued before the first is used.
// Product p = the row's p-th product in A-entry-major order.
template <typename V, typename K, int MAXP>
__device__ __forceinline__ int sg_expand_warp(const Mat<V> &A, const Mat<V> &B, int64_t i, int lane, K *key,
                                              V *prod) {
  constexpr int H = MAXP == SG_WARP_MAX ? 2 : 4;
  const int32_t LA = A.row_sizes[i];
  const Chain ca = load_chain_used(A, (int32_t)i, LA);
  int base = 0;
  for (int32_t e0 = 0; e0 < LA; e0 += 32) {
    const int nE = LA - e0 < 32 ? LA - e0 : 32;
    int32_t kb = 0, lb = 0;
    V a = V(0);
    if (lane < nE) {
      const int64_t qa = ca.phys(e0 + lane);
      kb = A.cols[qa];
      a = A.vals[qa];
      lb = B.row_sizes[kb];
    }
    const Chain cb = load_chain_used(B, kb, lb);
    const bool flat = __all_sync(FULL, cb.ns <= 1);  // every B row in its first segment (the common case)
    const bool dense = __all_sync(FULL, lane >= nE || lb > 0);  // no empty B row among the entries
    const int incl = warp_incl_scan(lb);
    const int pos = incl - lb;
    const int tot = __shfl_sync(FULL, incl, 31);  // base + tot <= P_i <= MAXP
    int started = 0;  // entries that start before the current 32 products (dense)
    // products in groups of H per lane: every B load of a group in flight at once
    for (int t0 = 0; t0 * 32 < tot; t0 += H) {
      int own[H];
      int32_t bc[H];
      V bv[H];
#pragma unroll
      for (int h = 0; h < H; h++) {
        const int q = (t0 + h) * 32 + lane;
        own[h] = 0;
        bc[h] = 0;
        bv[h] = V(0);
        if ((t0 + h) * 32 < tot) {  // warp-uniform
          int lo = 0;  // the last entry (< nE) whose offset is <= q: it owns q
          if (dense) {
            const unsigned sm =
                __reduce_or_sync(FULL, lane < nE && (pos >> 5) == t0 + h ? 1u << (pos & 31) : 0u);
            lo = started + __popc(sm & (0xffffffffu >> (31 - lane))) - 1;  // product 0 is a start: lo >= 0
            started += __popc(sm);
          } else {
#pragma unroll
            for (int st = 16; st > 0; st >>= 1) {
              const int c = lo + st;  // <= 31
              const int pc = __shfl_sync(FULL, pos, c);
              if (c < nE && pc <= q) lo = c;
            }
          }
          own[h] = lo;
          const int pj = __shfl_sync(FULL, pos, lo);
          int64_t qb;
          if (flat) {
            qb = (int64_t)__shfl_sync(FULL, cb.st[0], lo) + (q - pj);
          } else {
            const Chain co = shfl_chain(cb, lo);
            qb = co.phys(q - pj);
          }
          if (q < tot) {
            bc[h] = B.cols[qb];
            bv[h] = B.vals[qb];
          }
        }
      }
#pragma unroll
      for (int h = 0; h < H; h++) {
        const int q = (t0 + h) * 32 + lane;
        if ((t0 + h) * 32 < tot) {
          const V ao = __shfl_sync(FULL, a, own[h]);
          if (q < tot) {
            key[base + q] = SgKey<K, MAXP>::make(bc[h], base + q);
            V pr;
            if constexpr (sizeof(V) == 4) pr = __fmul_rn(ao, bv[h]);
            else pr = __dmul_rn(ao, bv[h]);
            prod[base + q] = pr;
          }
        }
      }
    }
    base += tot;
  }
  return base;
}

__device__ __forceinline__ int next_pow2(int x) {
  int p = 32;
  while (p < x) p <<= 1;
  return p;
}

// Bitonic sort of n2 (power of two) keys by `nthr` threads; sync() between steps.
template <typename K, typename Sync>
__device__ __forceinline__ void bitonic(K *key, int n2, int tid, int nthr, Sync sync) {
  for (int k = 2; k <= n2; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = tid; t < (n2 >> 1); t += nthr) {
        const int i = ((t & ~(j - 1)) << 1) | (t & (j - 1));
        const int l = i + j;
        const bool up = (i & k) == 0;
        const K a = key[i], b = key[l];
        if ((a > b) == up) {
          key[i] = b;
          key[l] = a;
        }
      }
      sync();
    }
}

// Bitonic sort of the 32*E keys held by a warp, E per lane: key i = lane*E + t
// in v[t].  The network whose comparators all ascend: a merge of two sorted
// halves starts with the mirror image (i against i ^ (k - 1)), so no step
// needs the direction of its block.  Steps with both keys in a lane are a min
// and a max of registers; the others take the partner's key by shuffle and
// one select (the lower lane keeps the smaller key).  Nothing goes through
// shared memory.
template <int E, typename K>
__device__ __forceinline__ void warp_bitonic(K (&v)[E], int lane) {
  constexpr int N = 32 * E;
#pragma unroll
  for (int k = 2; k <= N; k <<= 1) {
    if (k <= E) {
#pragma unroll
      for (int t = 0; t < E; t++) {
        const int q = t ^ (k - 1);
        if (q > t) {
          const K a = v[t], b = v[q];
          v[t] = a < b ? a : b;
          v[q] = a < b ? b : a;
        }
      }
    } else {
      const bool low = (lane & (k / E / 2)) == 0;
      K o[E];
#pragma unroll
      for (int t = 0; t < E; t++) o[t] = __shfl_xor_sync(FULL, v[E - 1 - t], k / E - 1);
#pragma unroll
      for (int t = 0; t < E; t++) v[t] = (o[t] < v[t]) == low ? o[t] : v[t];
    }
#pragma unroll
    for (int j = k >> 2; j > 0; j >>= 1) {
      if (j >= E) {
        const bool low = (lane & (j / E)) == 0;
#pragma unroll
        for (int t = 0; t < E; t++) {
          const K o = __shfl_xor_sync(FULL, v[t], j / E);
          v[t] = (o < v[t]) == low ? o : v[t];
        }
      } else {
#pragma unroll
        for (int t = 0; t < E; t++) {
          const int q = t ^ j;
          if (q > t) {
            const K a = v[t], b = v[q];
            v[t] = a < b ? a : b;
            v[q] = a < b ? b : a;
          }
        }
      }
    }
  }
}

// Where sorted key i lies in shared memory: one word of padding per 32, so
// that lanes writing their E consecutive keys hit different banks.
__device__ __forceinline__ int sg_slot(int i) { return i + (i >> 5); }

// A warp-row's P keys (in key[0, P), P <= 32*E) sorted through registers into
// key[sg_slot(i)]; slots past P take the largest key and end up past P.
template <int E, typename K>
__device__ __forceinline__ void sort_row_keys(K *key, int P, int lane) {
  K v[E];
#pragma unroll
  for (int t = 0; t < E; t++) v[t] = t * 32 + lane < P ? key[t * 32 + lane] : ~K(0);
  warp_bitonic<E>(v, lane);
  __syncwarp();  // every key read before the first is overwritten
#pragma unroll
  for (int t = 0; t < E; t++) key[sg_slot(lane * E + t)] = v[t];
}

// A warp's keys and products in shared memory.
template <typename V, typename K, int MAXP>
struct SgWarp {
  V prod[MAXP];
  K key[MAXP + MAXP / 32];
};

// Warp per row: P_i <= 256 (CLS SG_WARP), 256 < P_i <= 1024 (CLS SG_WARP4).
// Instruction issue bounds it (77% of the slots, DRAM 14%): expand, sort and
// emit take about 1800 instructions of a 169-product row, 6700 of an
// 841-product one, so what counts is few instructions and many warps.  The
// lower class at 6 blocks of 256 threads per SM with 2 x 32 products' loads at
// a time (a few spilled registers included): 286 us of 131072 rows of 169 FP64
// products; 3 blocks and 4 x 32: 333 us; the whole call 647 us at 4 blocks and
// 4 x 32, 623 at 4 and 2 x 32, 610 at 6.
// The upper class ends at 1024 products: 32 keys a lane and 8 or 12 KB of
// shared memory per warp still leave 3 or 2 blocks per SM; twice that would
// leave one.  Rows of 841 FP32 products in a CTA each, sorted as 64-bit keys in
// shared memory, took 1022 us for 20011 rows; in a warp each 215 us.  Rows come
// from a counter: a stride over the rows would give some warps only long rows
// where lengths repeat with its period.
template <typename V, typename K, int CLS>
__global__ void __launch_bounds__(SG_THREADS, CLS == SG_WARP ? (sizeof(K) == 4 ? 6 : 4) : sizeof(V) == 4 ? 3 : 2)
    k_sg_warp(Mat<V> A, Mat<V> B, const long long *ub, int warp_max, int G, unsigned long long *next, int32_t *tcol,
              V *tval, long long *ucnt) {
  constexpr int MAXP = CLS == SG_WARP ? SG_WARP_MAX : SG_WARP4_MAX;
  using KO = SgKey<K, MAXP>;
  extern __shared__ unsigned long long sg_smem[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  SgWarp<V, K, MAXP> &sh = reinterpret_cast<SgWarp<V, K, MAXP> *>(sg_smem)[w];
  const unsigned lt = (1u << lane) - 1u;
  K *key = sh.key;
  V *prod = sh.prod;
  // rows in row order, G <= 32 at a time from one counter; the next G are asked
  // for before these are worked on
  unsigned long long r0 = 0;
  if (lane == 0) r0 = atomicAdd(next, (unsigned long long)G);
  r0 = __shfl_sync(FULL, r0, 0);
  while (r0 < (unsigned long long)A.n_rows) {
    const int64_t g0 = (int64_t)r0;
    unsigned long long r1 = 0;
    if (lane == 0) r1 = atomicAdd(next, (unsigned long long)G);
    const bool mine = lane < G && g0 + lane < A.n_rows;
    const long long u = mine ? ub[g0 + lane] : 0, u1 = mine ? ub[g0 + lane + 1] : 0;
    unsigned todo = __ballot_sync(FULL, sg_class(u1 - u, warp_max) == CLS);
    for (; todo; todo &= todo - 1) {
      const int at = __ffs(todo) - 1;
      const int64_t i = g0 + at;
      const int64_t base = __shfl_sync(FULL, u, at);
      const int P = sg_expand_warp<V, K, MAXP>(A, B, i, lane, key, prod);
      __syncwarp();
      if constexpr (CLS == SG_WARP) {
        if (P <= 32) sort_row_keys<1>(key, P, lane);
        else if (P <= 64) sort_row_keys<2>(key, P, lane);
        else if (P <= 128) sort_row_keys<4>(key, P, lane);
        else sort_row_keys<8>(key, P, lane);
      } else {
        if (P <= 512) sort_row_keys<16>(key, P, lane);
        else sort_row_keys<32>(key, P, lane);
      }
      __syncwarp();
      int heads = 0;
      int32_t last = -1;  // the column before the current 32 keys
      for (int c0 = 0; c0 < P; c0 += 32) {
        const int idx = c0 + lane;
        const bool valid = idx < P;
        const K k = valid ? key[sg_slot(idx)] : ~K(0);
        const int32_t c = KO::col(k);
        int32_t before = __shfl_up_sync(FULL, c, 1);
        if (lane == 0) before = last;
        last = __shfl_sync(FULL, c, 31);
        const bool head = valid && before != c;
        const unsigned hm = __ballot_sync(FULL, head);
        if (head) {
          V v = prod[KO::idx(k)];
          for (int j = idx + 1; j < P; j++) {
            const K kj = key[sg_slot(j)];
            if (KO::col(kj) != c) break;
            v = v + prod[KO::idx(kj)];
          }
          const int64_t o = base + heads + __popc(hm & lt);
          tcol[o] = c;
          tval[o] = v;
        }
        heads += __popc(hm);
      }
      if (lane == 0) ucnt[i] = heads;
      __syncwarp();
    }
    r0 = __shfl_sync(FULL, r1, 0);
  }
}

// The CTA class's expand (the class above): row i's A entries are taken
// 256 at a time, one per thread (column, value, B row length and first
// segment loaded side by side), the lengths scanned across the block into
// product offsets, then each thread produces products q = tid, tid + 256,
// ... of the group -- the owning entry found by a binary search over the
// offsets in shared memory, four products' B loads in flight at a time.  A
// B row that does not lie in its first segment is read through its chain.
// Same keys and products as the warp class (product p = the row's p-th
// product in A-entry-major order).
template <typename V>
__device__ __forceinline__ int sg_expand_cta(const Mat<V> &A, const Mat<V> &B, int64_t i, int tid,
                                             unsigned long long *key, V *prod, int *soff, int32_t *sk, V *sa,
                                             int32_t *sst, int *wsum) {
  constexpr int H = 4;
  const int32_t LA = A.row_sizes[i];
  const Chain ca = load_chain_used(A, (int32_t)i, LA);
  int base = 0;
  for (int32_t e0 = 0; e0 < LA; e0 += SG_THREADS) {
    const int nE = LA - e0 < SG_THREADS ? LA - e0 : SG_THREADS;
    int32_t kb = 0, lb = 0, st0 = -1;
    V a = V(0);
    if (tid < nE) {
      const int64_t qa = ca.phys(e0 + tid);
      kb = A.cols[qa];
      a = A.vals[qa];
      lb = B.row_sizes[kb];
      const int2 s0 = __ldg(reinterpret_cast<const int2 *>(B.seg + 2 * (int64_t)kb));
      st0 = s0.x >= 0 && s0.y - s0.x >= lb ? s0.x : -1;  // all of the row in its first segment
    }
    const int incl = warp_incl_scan(lb);
    if ((tid & 31) == 31) wsum[tid >> 5] = incl;
    __syncthreads();
    int pre = 0, tot = 0;
#pragma unroll
    for (int q = 0; q < SG_THREADS / 32; q++) {
      if (q < (tid >> 5)) pre += wsum[q];
      tot += wsum[q];
    }
    soff[tid] = pre + incl - lb;
    sk[tid] = kb;
    sa[tid] = a;
    sst[tid] = st0;
    __syncthreads();
    for (int q0 = tid; q0 < tot; q0 += H * SG_THREADS) {
      int own[H];
      int32_t bc[H];
      V bv[H];
#pragma unroll
      for (int h = 0; h < H; h++) {
        const int q = q0 + h * SG_THREADS;
        own[h] = 0;
        bc[h] = 0;
        bv[h] = V(0);
        if (q < tot) {
          int lo = 0, hi = nE - 1;  // the last entry whose offset is <= q owns q
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (soff[mid] <= q) lo = mid;
            else hi = mid - 1;
          }
          own[h] = lo;
          const int32_t j = q - soff[lo];
          const int64_t qb = sst[lo] >= 0 ? (int64_t)sst[lo] + j : load_chain(B, sk[lo]).phys(j);
          bc[h] = B.cols[qb];
          bv[h] = B.vals[qb];
        }
      }
#pragma unroll
      for (int h = 0; h < H; h++) {
        const int q = q0 + h * SG_THREADS;
        if (q < tot) {
          key[base + q] = ((unsigned long long)(uint32_t)bc[h] << 32) | (unsigned long long)(base + q);
          V pr;
          if constexpr (sizeof(V) == 4) pr = __fmul_rn(sa[own[h]], bv[h]);
          else pr = __dmul_rn(sa[own[h]], bv[h]);
          prod[base + q] = pr;
        }
      }
    }
    base += tot;
    __syncthreads();  // the group's tables are reused by the next group
  }
  return base;
}

// CTA per row, up to 4096 products (dynamic shared memory).
template <typename V>
__global__ void __launch_bounds__(SG_THREADS) k_sg_cta(Mat<V> A, Mat<V> B, const unsigned *rows,
                                                       int64_t n_rows, const long long *ub, int32_t *tcol, V *tval,
                                                       long long *ucnt) {
  extern __shared__ unsigned long long sg_smem[];
  unsigned long long *key = sg_smem;
  V *prod = reinterpret_cast<V *>(sg_smem + SG_CTA_MAX);
  __shared__ int wheads[SG_THREADS / 32 + 1];
  __shared__ int soff[SG_THREADS], wsum[SG_THREADS / 32];
  __shared__ int32_t sk[SG_THREADS], sst[SG_THREADS];
  __shared__ V sa[SG_THREADS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int64_t it = blockIdx.x; it < n_rows; it += gridDim.x) {
    const int64_t i = rows[it];
    const int P = sg_expand_cta(A, B, i, threadIdx.x, key, prod, soff, sk, sa, sst, wsum);
    const int n2 = next_pow2(P);
    for (int t = P + threadIdx.x; t < n2; t += SG_THREADS) key[t] = ~0ull;
    __syncthreads();
    bitonic(key, n2, threadIdx.x, SG_THREADS, []() { __syncthreads(); });
    const int64_t base = ub[i];
    int heads = 0;  // running total (uniform across the block)
    for (int c0 = 0; c0 < P; c0 += SG_THREADS) {
      const int idx = c0 + threadIdx.x;
      const bool valid = idx < P;
      const unsigned long long k = valid ? key[idx] : 0;
      const bool head = valid && (idx == 0 || (key[idx - 1] >> 32) != (k >> 32));
      const unsigned hm = __ballot_sync(FULL, head);
      if (lane == 0) wheads[w] = __popc(hm);
      __syncthreads();
      int before = 0, total = 0;
      for (int q = 0; q < SG_THREADS / 32; q++) {
        if (q < w) before += wheads[q];
        total += wheads[q];
      }
      if (head) {
        V v = prod[(uint32_t)k];
        for (int j = idx + 1; j < P && (key[j] >> 32) == (k >> 32); j++) v = v + prod[(uint32_t)key[j]];
        const int64_t o = base + heads + before + __popc(hm & ((1u << lane) - 1u));
        tcol[o] = (int32_t)(k >> 32);
        tval[o] = v;
      }
      heads += total;
      __syncthreads();
    }
    if (threadIdx.x == 0) ucnt[i] = heads;
    __syncthreads();
  }
}

// Global path: expand rows with P_i > 4096 into (key = slot<<cb | col, value = global product index).
template <typename V>
__global__ void k_sg_global_expand(Mat<V> A, Mat<V> B, const unsigned *rows, int64_t n_rows,
                                   const long long *goff, int cb, unsigned long long *gkey, unsigned *gidx,
                                   V *gprod) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t slot = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; slot < n_rows; slot += nw) {
    const int64_t i = rows[slot];
    const int64_t o = goff[slot];
    const Chain ca = load_chain(A, (int32_t)i);
    const int64_t LA = A.row_sizes[i];
    int64_t pos = 0;
    for (int64_t ea = 0; ea < LA; ea++) {
      const int64_t qa = ca.phys(ea);
      const int32_t k = A.cols[qa];
      const V a = A.vals[qa];
      const Chain ck = load_chain(B, k);
      const int64_t LB = B.row_sizes[k];
      for (int64_t j = lane; j < LB; j += 32) {
        const int64_t qb = ck.phys(j);
        gkey[o + pos + j] = ((unsigned long long)slot << cb) | (unsigned long long)(uint32_t)B.cols[qb];
        gidx[o + pos + j] = (unsigned)(o + pos + j);
        V pr;
        if constexpr (sizeof(V) == 4) pr = __fmul_rn(a, B.vals[qb]);
        else pr = __dmul_rn(a, B.vals[qb]);
        gprod[o + pos + j] = pr;
      }
      pos += LB;
    }
  }
}

// Heads of equal keys after the sort.
__global__ void k_sg_global_flags(const unsigned long long *gkey, int64_t n, long long *flag) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += stride)
    flag[q] = (q == 0 || gkey[q] != gkey[q - 1]) ? 1 : 0;
}

template <typename V>
__global__ void k_sg_global_emit(const unsigned long long *gkey, const unsigned *gidx, const V *gprod, int64_t n,
                                 const long long *hpos, const unsigned *rows, const long long *goff,
                                 const long long *ub, int cb, int32_t *tcol, V *tval,
                                 long long *ucnt) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const unsigned long long cmask = (1ull << cb) - 1;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += stride) {
    const unsigned long long k = gkey[q];
    if (q > 0 && gkey[q - 1] == k) continue;
    const int64_t slot = (int64_t)(k >> cb);
    const int64_t i = rows[slot];
    V v = gprod[gidx[q]];
    for (int64_t j = q + 1; j < n && gkey[j] == k; j++) v = v + gprod[gidx[j]];
    const int64_t first = hpos[goff[slot]];  // head rank of the row's first product
    const int64_t o = ub[i] + (hpos[q] - first);
    tcol[o] = (int32_t)(k & cmask);
    tval[o] = v;
    atomicAdd((unsigned long long *)&ucnt[i], 1ull);
  }
}

// slot products for the global class: goff[slot] = ub-like offsets of the
// large rows in a dense staging array
__global__ void k_sg_global_sizes(const unsigned *rows, int64_t n_rows, const long long *ub, long long *gsz) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t it = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; it <= n_rows; it += stride)
    gsz[it] = it < n_rows ? ub[rows[it] + 1] - ub[rows[it]] : 0;
}

static int grid_for(int64_t n, int block) {
  int64_t g = div_up(n, block);
  int64_t cap = (int64_t)sm_count() * 16;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

// A warp class's launch: warps that stay and take rows from a counter.
template <typename V, typename K, int CLS>
static int sg_warp_rows(const Mat<V> &A, const Mat<V> &B, int64_t n_rows, const long long *ub, int warp_max,
                        long long *next, int32_t *tcol, V *tval, long long *ucnt, cudaStream_t s) {
  constexpr int W = SG_THREADS / 32;
  constexpr size_t smem = sizeof(SgWarp<V, K, CLS == SG_WARP ? SG_WARP_MAX : SG_WARP4_MAX>) * W;
  static const int g = [] {  // once, thread-safely: the kernel's shared-memory limit, then its grid
    cudaFuncSetAttribute(k_sg_warp<V, K, CLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return persistent_grid((const void *)k_sg_warp<V, K, CLS>, SG_THREADS, smem);
  }();
  // a warp asks for about GR rows of the class at a time
  constexpr int64_t GR = CLS == SG_WARP ? 2 : 1;
  const int64_t G = std::min<int64_t>(32, GR * A.n_rows / n_rows);
  DCSR_LAUNCH((k_sg_warp<V, K, CLS>), (int)std::min<int64_t>(g, div_up(A.n_rows, G * W)), SG_THREADS, smem, s, A, B,
              ub, warp_max, (int)G, (unsigned long long *)next, tcol, tval, ucnt);
  return DCSR_OK;
}

template <typename V>
static int spgemm_impl(dcsr_handle hA, dcsr_handle hB, dcsr_handle hC, cudaStream_t s) {
  const int32_t n = hA->n_rows;
  Mat<V> A = hA->view<V>(), B = hB->view<V>();
  Arena ar;
  DCSR_TRY(ar.reserve(arena_bytes(n + 2, 8) * 3 + arena_bytes(n + 2, 4) * 2 + arena_bytes(SG_R_WORDS, 8) +
                          scan_scratch_bytes(n + 2),
                      s));
  long long *cnt = ar.take<long long>(n + 2), *ub = ar.take<long long>(n + 2), *ucnt = ar.take<long long>(n + 2);
  unsigned *r_cta = ar.take<unsigned>(n + 2), *r_glob = ar.take<unsigned>(n + 2);
  long long *res = ar.take<long long>(SG_R_WORDS);
  if (ar.overflow) return DCSR_OOM;  // scratch sizing bug: no kernel sees a null pointer
  ar.status = res + SG_R_STATUS;  // look-back timeouts of the scans here
  DCSR_CUDA(cudaMemsetAsync(res, 0, sizeof(long long) * SG_R_WORDS, s));
  // rows of 257 to 1024 products: 32-bit keys (column, p) where the columns leave p its 10 bits
  const int warp_max = hB->n_cols <= (1 << 22) ? SG_WARP4_MAX : SG_WARP_MAX;
  if (n > 0) {
    DCSR_LAUNCH(k_sg_count<V>, grid_for((int64_t)n * 8, SG_THREADS), SG_THREADS, 0, s, A, B, warp_max, cnt, res);
    DCSR_TRY(scan_map(StageScan{cnt, hC->o, ub, ucnt, res, n}, n, ar, s));
  }
  // the one read before the numeric pass: staging and C's pool are sized here
  long long host[SG_R_WORDS];
  DCSR_CUDA(cudaMemcpyAsync(host, res, sizeof(host), cudaMemcpyDeviceToHost, s));
  DCSR_CUDA(cudaStreamSynchronize(s));
  if (host[SG_R_STATUS] == DCSR_TIMEOUT) {
    ar.release(s);
    return DCSR_TIMEOUT;
  }
  const int64_t Pg = host[SG_R_GPROD], P = host[SG_R_PROD], cap_bound = pool_capacity(hC->o, host[SG_R_CAPS]);
  const int64_t n_cta = host[SG_CTA], n_global = host[SG_GLOBAL];
  // C's pool is allocated for cap_bound entries: out of its index range, no
  // staging either
  const int refused = Pg > 0xffffffffLL ? DCSR_NOT_SUPPORTED
                      : host[SG_R_CAPS] > 0x7fffffffLL || cap_bound > 0x7fffffffLL ? DCSR_OOM : DCSR_OK;
  if (refused != DCSR_OK) {
    ar.release(s);
    return refused;
  }
  if (n_cta + n_global > 0) {
    // (read back before the lists are used: a list that a timed-out look-back
    // left unfinished must not reach a kernel)
    DCSR_TRY(scan_map(ListScan{ub, warp_max, r_cta, r_glob}, n, ar, s));
    DCSR_CUDA(cudaMemcpyAsync(host + SG_R_STATUS, res + SG_R_STATUS, sizeof(long long), cudaMemcpyDeviceToHost, s));
    DCSR_CUDA(cudaStreamSynchronize(s));
    if (host[SG_R_STATUS] == DCSR_TIMEOUT) {
      ar.release(s);
      return DCSR_TIMEOUT;
    }
  }
  // staging: row i's unique columns at ub[i]
  int32_t *tcol = nullptr;
  V *tval = nullptr;
  DCSR_CUDA(dcsr::dev_alloc((void **)&tcol, sizeof(int32_t) * (P + 1), s));
  DCSR_CUDA(dcsr::dev_alloc((void **)&tval, sizeof(V) * (P + 1), s));
  const size_t cta_smem = SG_CTA_MAX * (sizeof(unsigned long long) + sizeof(V));
  static const int g_cta = [] {  // once, thread-safely: the CTA kernels' shared-memory limit, then their grid
    cudaFuncSetAttribute(k_sg_cta<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(SG_CTA_MAX * (sizeof(unsigned long long) + sizeof(float))));
    cudaFuncSetAttribute(k_sg_cta<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(SG_CTA_MAX * (sizeof(unsigned long long) + sizeof(double))));
    return persistent_grid((const void *)k_sg_cta<double>, SG_THREADS,
                           SG_CTA_MAX * (sizeof(unsigned long long) + sizeof(double)));
  }();
  if (host[SG_WARP] > 0) {
    const bool narrow = hB->n_cols <= (1 << 24);  // (column, p) in 32-bit keys
    DCSR_TRY((narrow ? sg_warp_rows<V, unsigned, SG_WARP> : sg_warp_rows<V, unsigned long long, SG_WARP>)(
        A, B, host[SG_WARP], ub, warp_max, res + SG_R_NEXT, tcol, tval, ucnt, s));
  }
  if (host[SG_WARP4] > 0)
    DCSR_TRY((sg_warp_rows<V, unsigned, SG_WARP4>(A, B, host[SG_WARP4], ub, warp_max, res + SG_R_NEXT4, tcol, tval,
                                                  ucnt, s)));
  if (n_cta > 0)
    DCSR_LAUNCH(k_sg_cta<V>, g_cta, SG_THREADS, cta_smem, s, A, B, r_cta, n_cta, ub, tcol, tval, ucnt);
  Arena gg;
  if (n_global > 0) {
    // products of all large rows, laid out densely by slot, then one stable
    // radix sort by (slot, column) keeps every column's products in p order
    gg.status = hC->stat + ST_STATUS;  // look-back timeouts reach C's status
    DCSR_TRY(gg.reserve(arena_bytes(n_global + 2, 8) + 2 * arena_bytes(Pg, 8) + 2 * arena_bytes(Pg, 4) +
                            arena_bytes(Pg, sizeof(V)) + arena_bytes(Pg + 1, 8) + radix_scratch_bytes(Pg) +
                            scan_scratch_bytes(Pg + 1) + scan_scratch_bytes(n_global + 2), s));
    long long *goff = gg.take<long long>(n_global + 2);
    unsigned long long *gk0 = gg.take<unsigned long long>(Pg), *gk1 = gg.take<unsigned long long>(Pg);
    unsigned *gi0 = gg.take<unsigned>(Pg), *gi1 = gg.take<unsigned>(Pg);
    V *gprod = (V *)gg.take<double>(Pg);
    long long *hpos = gg.take<long long>(Pg + 1);
    if (gg.overflow) return DCSR_OOM;  // scratch sizing bug: no kernel sees a null pointer
    DCSR_LAUNCH(k_sg_global_sizes, grid_for(n_global + 1, 256), 256, 0, s, r_glob, n_global, ub, goff);
    DCSR_TRY(scan_i64(goff, goff, n_global + 1, nullptr, gg, s));
    const int cb = bits_for(hB->n_cols);
    DCSR_LAUNCH(k_sg_global_expand<V>, grid_for(n_global * 32, 256), 256, 0, s, A, B, r_glob, n_global, goff, cb,
                gk0, gi0, gprod);
    DCSR_TRY(radix_sort_pairs(&gk0, &gi0, &gk1, &gi1, Pg, bits_for(n_global) + cb, gg, s));
    DCSR_LAUNCH(k_sg_global_flags, grid_for(Pg, 256), 256, 0, s, gk0, Pg, hpos);
    DCSR_TRY(scan_i64(hpos, hpos, Pg, nullptr, gg, s));
    DCSR_LAUNCH(k_sg_global_emit<V>, grid_for(Pg, 256), 256, 0, s, gk0, gi0, gprod, Pg, hpos, r_glob, goff, ub, cb,
                tcol, tval, ucnt);
  }
  // C's rows go straight from the staging area into C's pool (policy
  // capacities); the last synchronisation reads C's pool top
  const int st = load_from_rows(hC, ub, ucnt, tcol, tval, P, cap_bound, s);
  gg.release(s);
  ar.release(s);
  dcsr::dev_free(tcol, s);
  dcsr::dev_free(tval, s);
  return st;
}

}  // namespace dcsr

using namespace dcsr;

extern "C" int dcsr_spgemm(dcsr_handle A, dcsr_handle B, dcsr_handle C, void *stream) {
  if (!A || !B || !C) return DCSR_BAD_ARG;
  if (A->n_cols != B->n_rows || C->n_rows != A->n_rows || C->n_cols != B->n_cols || A->dtype != B->dtype ||
      C->dtype != A->dtype || C == A || C == B)
    return DCSR_BAD_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (A->dtype == DCSR_F32) return spgemm_impl<float>(A, B, C, s);
  return spgemm_impl<double>(A, B, C, s);
}
