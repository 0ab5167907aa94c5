// update.cu -- in-place batch updates of one DCSR matrix or of a set of
// matrices at once, and COO grouping for loads.
//
// Pipeline (all on the caller's stream, no host synchronisation); every
// kernel runs over the union of all matrices' triples / touched rows:
//   keys     (matrix, row, col) keys with an index check        k_make_keys
//   sort     stable LSD radix sort of (key, global triple index) radix_sort_pairs
//   group    one scan kernel (scan_map): MERGE: each (row, col) group head
//            searches its column in the row; row heads list the touched
//            rows, new columns are written out in order         GroupScan
//   plan     one scan kernel over the touched rows: new length, capacity,
//            layer, relocation, the row-ordered allocation of new segments
//            (offsets per matrix, relative to its first touched row), the
//            lists of rows to shift and the relocation tiles    PlanScan
//            APPEND: the reference's segment walk per touched row
//   check    per matrix: pool / layer / index status -> go flag   k_check
//            (one matrix, MERGE: by the plan kernel)
//   apply    existing columns in place (thread per group), then one kernel
//            for the relocation tiles (rows whose in-place shift would
//            exceed reloc_min, or that outgrow a chain already max_segs
//            long, merged out of place into a fresh segment), the larger
//            shifts (a warp per row) and the small ones (8 lanes per row)
//   finish   chain reset of relocated rows, new pool tops          k_finish
// A rejected matrix (status != OK) is left untouched; the others proceed.
//
// Reference: device::UpdateMatrix include/load.h:258-325 and UpdateMatrix_dcsr
// include/sparse_update.inl:16-130 (segment walk, bump allocation, layer
// linking).  The reference appends without merging and allocates with
// atomicAdd; here MERGE mode keeps rows sorted and unique (duplicates summed
// in batch order) and the allocation is a row-ordered scan, so layouts are
// reproducible bit for bit, alone or in a batch.
#include <algorithm>
#include <cstring>

#include "internal.cuh"
#include "lookback.cuh"

namespace dcsr {

constexpr int UPD_THREADS = 256;
constexpr int RT_TILE = 256;  // relocation: positions per tile (a warp's, 8 per lane)
constexpr int SMALL_AFF = 32;  // apply: rows whose last <= 32 positions change use 8 lanes (one step), others a warp

enum { AUX_BAD_INDEX = 1, AUX_LAYER_OVF = 2 };

// Key layout: [matrix | row | col] (MERGE) or [matrix | row] (APPEND).
struct KeyFmt {
  int cb, rb, merge;
  __device__ __forceinline__ int32_t row(unsigned long long k) const {
    const unsigned long long rk = merge ? (k >> cb) : k;
    return (int32_t)(rk & ((1ull << rb) - 1));
  }
  __device__ __forceinline__ int item(unsigned long long k) const { return (int)(k >> (rb + (merge ? cb : 0))); }
  __device__ __forceinline__ unsigned long long rowkey(unsigned long long k) const { return merge ? (k >> cb) : k; }
  __device__ __forceinline__ int32_t col(unsigned long long k) const { return (int32_t)(k & ((1ull << cb) - 1)); }
};

// ------------------------------------------------------------ matrix sources

// One matrix, passed by value.
template <typename V>
struct UpdOne {
  Mat<V> m;
  const int32_t *rows, *cols;
  const V *vals;
  __device__ __forceinline__ const Mat<V> &mat(int) const { return m; }
  __device__ __forceinline__ long long *st(int) const { return m.stat; }
  __device__ __forceinline__ int item_of_g(int64_t) const { return 0; }
  __device__ __forceinline__ int64_t local(int, int64_t g) const { return g; }
  __device__ __forceinline__ const int32_t *urows(int) const { return rows; }
  __device__ __forceinline__ const int32_t *ucols(int) const { return cols; }
  __device__ __forceinline__ const V *uvals(int) const { return vals; }
};

// A set of matrices: device array of batch items.
template <typename V>
struct UpdMany {
  const BatchItem<V> *it;
  int count;
  __device__ __forceinline__ const Mat<V> &mat(int i) const { return it[i].m; }
  __device__ __forceinline__ long long *st(int i) const { return it[i].m.stat; }
  __device__ __forceinline__ int item_of_g(int64_t g) const {
    int lo = 0, hi = count;  // largest i with toff <= g
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (it[mid].toff <= g) lo = mid;
      else hi = mid;
    }
    return lo;
  }
  __device__ __forceinline__ int64_t local(int i, int64_t g) const { return g - it[i].toff; }
  __device__ __forceinline__ const int32_t *urows(int i) const { return it[i].rows; }
  __device__ __forceinline__ const int32_t *ucols(int i) const { return it[i].cols; }
  __device__ __forceinline__ const V *uvals(int i) const { return (const V *)it[i].vals; }
};

// ------------------------------------------------------------------ keys

template <typename V, typename Src>
__global__ void k_item_init(Src src, int count, long long *gstat) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (tid == 0) gstat[ST_LISTS] = gstat[ST_RELOC] = 0;
  for (int i = tid; i < count; i += gridDim.x * blockDim.x) {
    long long *st = src.st(i);
    st[ST_AUX] = 0;
    st[ST_A0] = 0;
    st[ST_A1] = 0;
    st[ST_GO] = 0;
  }
}

template <typename V, typename Src>
__global__ void k_make_keys(Src src, int64_t n, KeyFmt f, unsigned long long *keys, unsigned *perm) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < n; g += stride) {
    const int i = src.item_of_g(g);
    const int64_t l = src.local(i, g);
    const Mat<V> &m = src.mat(i);
    int32_t r = src.urows(i)[l], c = src.ucols(i)[l];
    if (r < 0 || r >= m.n_rows || c < 0 || c >= m.n_cols) {
      atomicOr((unsigned long long *)&src.st(i)[ST_AUX], (unsigned long long)AUX_BAD_INDEX);
      r = 0;
      c = 0;
    }
    const unsigned long long it = (unsigned long long)i << (f.rb + (f.merge ? f.cb : 0));
    keys[g] = f.merge ? (it | ((unsigned long long)r << f.cb) | (unsigned long long)c) : (it | (unsigned long long)r);
    perm[g] = (unsigned)g;
  }
}

// Sub-warp of S lanes (S divides 32): lane-local mask, ballot and helpers.
template <int S>
struct Sub {
  int sl, sw;
  unsigned mask;
  __device__ __forceinline__ Sub() {
    const int lane = lane_id();
    sl = lane & (S - 1);
    sw = lane / S;
    mask = S == 32 ? FULL : (((1u << S) - 1u) << (sw * S));
  }
  __device__ __forceinline__ unsigned ballot(bool p) const {
    const unsigned b = __ballot_sync(mask, p);
    return S == 32 ? b : (b >> (sw * S)) & ((1u << S) - 1u);
  }
  __device__ __forceinline__ unsigned full() const { return S == 32 ? FULL : (1u << S) - 1u; }
  __device__ __forceinline__ void sync() const { __syncwarp(mask); }
  __device__ __forceinline__ int incl_scan(int v) const {
#pragma unroll
    for (int o = 1; o < S; o <<= 1) {
      const int w = __shfl_up_sync(mask, v, o, S);
      if (sl >= o) v += w;
    }
    return v;
  }
  // consecutive set bits of a lane-local ballot starting at bit 0
  __device__ __forceinline__ int leading(unsigned bm) const { return bm == full() ? S : __ffs(~bm) - 1; }
};

// --------------------------------------------------------------- grouping

// A touched row as the plan leaves it for the apply kernels: what they need
// to start on its entries at once, without the row's own tables.
struct __align__(16) RowDesc {
  int32_t row, item;  // matrix
  int32_t n0, mnew;   // its new entries n0 .. n0+mnew-1 (MERGE: of the new columns; APPEND: of the sorted batch)
  int32_t len;        // its length before the update
  int32_t start;      // its first pool slot when the row, grown, stays in its only segment; else -1
  int32_t lo;         // MERGE: first insertion point
  int32_t info;       // bits 0..7: the new segment's layer (int8, -1 none); bit 8: relocated
  int32_t cap;        // capacity of a new segment (0: none)
  int32_t tile0;      // relocation tiles of the rows before it (relocated: its first tile)
  long long addr;     // the new segment's offset in the batch's allocation order
};

// Scratch of one update (T triples).
template <typename V>
struct UpdWork {
  const unsigned long long *keys;  // sorted
  const unsigned *perm;            // batch position of each
  int64_t T;
  KeyFmt f;
  long long *gstat;
  int32_t *bslot;               // [T] pool slot of an existing column's group head, else -1
  int32_t *trow, *tmat, *tn0;   // [T+2] touched rows: row, matrix, first new entry (tn0[touched] = their number)
  int32_t *ncol, *nins;         // [T] new columns in (row, column) order: column, insertion point in the row
  V *nval;                      // [T] their values (batch-order sums)
  RowDesc *desc;                // [T] per touched row
  int32_t *small, *big;         // [T] touched rows to shift (or append to) in place
  int32_t *reloc;               // [T] touched rows relocated
};

// x plus the triples from j on that have the lane's key, in batch order (called
// by whole warps; lanes that are not active have none).  A lane walks its first
// GROUP_LANE triples itself, as far as almost every group goes; a longer group
// is taken by the whole warp, 128 triples' keys, indices and values in flight
// together, so that it is a chain of additions, not of loads: a pair that comes
// 100,000 times in one update takes 1.6 ms (16.3 when its thread walked it
// alone, 11.5 with the values put in order before).
constexpr int GROUP_LANE = 4;
template <typename V, typename Src>
__device__ __forceinline__ V group_sum(const Src &src, const UpdWork<V> &w, bool active, int item,
                                       unsigned long long key, int64_t j, V x) {
  constexpr int U = 4;
  const int lane = lane_id();
  bool more = active;
  for (int n = 0; more; n++) {
    more = j < w.T && w.keys[j] == key;
    if (!more || n == GROUP_LANE) break;
    x = x + src.uvals(item)[src.local(item, w.perm[j])];
    j++;
  }
  unsigned longs = __ballot_sync(FULL, more);
  while (longs) {
    const int s = __ffs(longs) - 1;
    longs &= longs - 1;
    const unsigned long long k = __shfl_sync(FULL, key, s);
    const int it = __shfl_sync(FULL, item, s);
    V y = __shfl_sync(FULL, x, s);
    int64_t at = __shfl_sync(FULL, j, s) + lane;
    for (bool on = true; on;) {
      V o[U];
      int cnt[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int64_t p = at + 32 * u;
        const bool in = p < w.T && w.keys[p] == k;
        const unsigned b = __ballot_sync(FULL, in);
        cnt[u] = ~b ? __ffs(~b) - 1 : 32;
        o[u] = in ? src.uvals(it)[src.local(it, w.perm[p])] : V(0);
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (!on) continue;
        if (cnt[u] == 32) {
#pragma unroll
          for (int q = 0; q < 32; q++) y = y + __shfl_sync(FULL, o[u], q);
        } else {
          for (int q = 0; q < cnt[u]; q++) y = y + __shfl_sync(FULL, o[u], q);
          on = false;
        }
      }
      at += 32 * U;
    }
    if (lane == s) x = y;
  }
  return x;
}

// MERGE: scans (row heads, new columns) over the sorted batch.  A thread's
// group heads search their rows in step: the loads of one step of all of
// them are in flight together.
template <typename V, typename Src>
struct GroupScan {
  static constexpr int NS = 2, IT = SM_HEAVY;
  static constexpr bool LOAD_ALL = true;
  using T = int32_t;
  struct State {
    unsigned long long key;
    int32_t pos;  // group heads: pool slot of an existing column, ~insertion point of a new one
    bool head;    // of a (row, column) group
  };
  Src src;
  UpdWork<V> w;
  __device__ __forceinline__ void load_all(int64_t base, int64_t n, State (&st)[IT], T (&v)[IT][2]) const {
    const KeyFmt f = w.f;
    int32_t lo[IT], hi[IT], s0[IT], len[IT];
    bool flat[IT];
#pragma unroll
    for (int j = 0; j < IT; j++) {
      const int64_t g = base + 32 * j;
      st[j].key = g < n ? w.keys[g] : 0;
      st[j].pos = -1;
      const unsigned long long prev = g > 0 && g < n ? w.keys[g - 1] : 0;
      st[j].head = g < n && (g == 0 || prev != st[j].key);
      v[j][0] = g < n && (g == 0 || f.rowkey(prev) != f.rowkey(st[j].key)) ? 1 : 0;
      v[j][1] = 0;
    }
#pragma unroll
    for (int j = 0; j < IT; j++) {
      lo[j] = hi[j] = s0[j] = len[j] = 0;
      flat[j] = true;
      if (st[j].head) {
        const Mat<V> &m = src.mat(f.item(st[j].key));
        const int64_t r = f.row(st[j].key);
        const int2 sg = *reinterpret_cast<const int2 *>(m.seg + 2 * r);
        len[j] = m.row_sizes[r];
        s0[j] = sg.x;
        flat[j] = len[j] == 0 || (sg.x >= 0 && len[j] <= sg.y - sg.x);
        hi[j] = flat[j] ? len[j] : 0;
      }
    }
    // lower bounds, three probes a step (a quarter of the range is left)
    bool more = true;
    while (more) {
      more = false;
      int32_t c[IT][3];
#pragma unroll
      for (int j = 0; j < IT; j++)
        if (lo[j] < hi[j]) {
          const int32_t *p = src.mat(f.item(st[j].key)).cols + (int64_t)s0[j] + lo[j];
          const unsigned d = hi[j] - lo[j];
          c[j][0] = p[d >> 2];
          c[j][1] = p[d >> 1];
          c[j][2] = p[d - 1 - (d >> 2)];
        }
#pragma unroll
      for (int j = 0; j < IT; j++)
        if (lo[j] < hi[j]) {
          const int32_t x = f.col(st[j].key), l = lo[j];
          const unsigned d = hi[j] - l;
          if (c[j][1] < x) {
            lo[j] = l + (d >> 1) + 1;
            if (lo[j] < hi[j]) {
              const int32_t m3 = l + d - 1 - (d >> 2);
              if (m3 >= lo[j]) {
                if (c[j][2] < x) lo[j] = m3 + 1;
                else hi[j] = m3;
              }
            }
          } else {
            hi[j] = l + (d >> 1);
            if (lo[j] < hi[j]) {
              if (c[j][0] < x) lo[j] = l + (d >> 2) + 1;
              else hi[j] = l + (d >> 2);
            }
          }
          more |= lo[j] < hi[j];
        }
    }
#pragma unroll
    for (int j = 0; j < IT; j++) {
      if (!st[j].head) continue;
      const Mat<V> &m = src.mat(f.item(st[j].key));
      const int32_t col = f.col(st[j].key);
      if (flat[j]) {
        const bool found = lo[j] < len[j] && m.cols[(int64_t)s0[j] + lo[j]] == col;
        st[j].pos = found ? s0[j] + lo[j] : ~lo[j];
      } else {  // a row in several segments
        const Chain ch = load_chain(m, f.row(st[j].key));
        int32_t a = 0, b = len[j];
        while (a < b) {
          const int32_t mid = (a + b) >> 1;
          if (m.cols[ch.phys(mid)] < col) a = mid + 1;
          else b = mid;
        }
        const int64_t q = a < len[j] ? ch.phys(a) : 0;
        st[j].pos = a < len[j] && m.cols[q] == col ? (int32_t)q : ~a;
      }
      v[j][1] = st[j].pos < 0 ? 1 : 0;
    }
  }
  __device__ __forceinline__ void emit(int64_t g, bool ok, const State &st, const long long (&p)[2],
                                       const T (&v)[2]) const {
    const KeyFmt f = w.f;
    const int i = f.item(st.key);
    const bool add = ok && v[1] && p[1] >= 0 && p[1] < w.T;
    V x = add ? src.uvals(i)[src.local(i, w.perm[g])] : V(0);
    x = group_sum(src, w, add, i, st.key, g + 1, x);
    if (!ok) return;
    w.bslot[g] = st.head && st.pos >= 0 ? st.pos : -1;
    if (v[0] && p[0] >= 0 && p[0] < w.T) {
      w.trow[p[0]] = f.row(st.key);
      w.tmat[p[0]] = i;
      w.tn0[p[0]] = (int32_t)p[1];
    }
    if (add) {
      w.ncol[p[1]] = f.col(st.key);
      w.nins[p[1]] = ~st.pos;
      w.nval[p[1]] = x;
    }
  }
  __device__ __forceinline__ void total(const long long (&t)[2]) const {
    w.gstat[ST_TOUCHED] = t[0];
    if (t[0] >= 0 && t[0] <= w.T) w.tn0[t[0]] = (int32_t)t[1];
  }
};

// APPEND: touched rows with their first triple in the sorted batch.
template <typename V, typename Src>
struct RowHeadScan {
  static constexpr int NS = 1, IT = SM_LIGHT;
  using T = int32_t;
  struct State {
    unsigned long long key;
  };
  Src src;
  UpdWork<V> w;
  __device__ __forceinline__ void load(int64_t g, bool ok, State &st, T (&v)[1]) const {
    st.key = ok ? w.keys[g] : 0;
    v[0] = ok && (g == 0 || w.f.rowkey(w.keys[g - 1]) != w.f.rowkey(st.key)) ? 1 : 0;
  }
  __device__ __forceinline__ void emit(int64_t g, bool ok, const State &st, const long long (&p)[1],
                                       const T (&v)[1]) const {
    if (!ok || !v[0] || p[0] < 0 || p[0] >= w.T) return;
    w.trow[p[0]] = w.f.row(st.key);
    w.tmat[p[0]] = w.f.item(st.key);
    w.tn0[p[0]] = (int32_t)g;
  }
  __device__ __forceinline__ void total(const long long (&t)[1]) const {
    w.gstat[ST_TOUCHED] = t[0];
    if (t[0] >= 0 && t[0] <= w.T) w.tn0[t[0]] = (int32_t)w.T;
  }
};

// --------------------------------------------------------------- planning

// Per matrix: requirement from its new segments, status and go flag.
template <typename V>
__device__ __forceinline__ void check_item(const Mat<V> &m, long long *st) {
  const long long aux = st[ST_AUX];
  const long long top = m.row_sizes[m.n_rows];
  const long long need = top + (st[ST_A1] - st[ST_A0]);
  st[ST_TOP] = top;
  st[ST_NEED] = need;
  int s = DCSR_OK;
  if (aux & AUX_BAD_INDEX) s = DCSR_BAD_INDEX;
  else if (aux & AUX_LAYER_OVF) s = DCSR_LAYER_OVERFLOW;
  else if (need > m.pool_cap || need > 0x7fffffffLL) s = DCSR_POOL_EXHAUSTED;
  st[ST_GO] = s == DCSR_OK ? 1 : 0;
  if (s != DCSR_OK && st[ST_STATUS] == 0) st[ST_STATUS] = s;
  st[ST_AUX] = 0;
}

template <typename V, typename Src>
__global__ void k_check(Src src, int count) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
    check_item(src.mat(i), src.st(i));
}

// Scans (new-segment capacities, relocation tiles) over the touched rows.
// MERGE: new length, capacity, layer, relocation; APPEND: the reference's
// segment walk and allocation size.  ONE: a single matrix (its check is done
// here in MERGE mode).
template <typename V, typename Src, bool MERGE, bool ONE>
struct PlanScan {
  static constexpr int NS = 2, IT = SM_HEAVY;
  using T = long long;
  struct State {
    int32_t row, item, n0, mnew, len, start, lo, info, list;  // list: 0 none, 1 small, 2 big
  };
  Src src;
  UpdWork<V> w;
  __device__ __forceinline__ void load(int64_t t, bool ok, State &st, T (&v)[2]) const {
    v[0] = v[1] = 0;
    st.row = -1;
    st.list = 0;
    if (!ok || t >= w.gstat[ST_TOUCHED]) return;
    const int i = w.tmat[t];
    const Mat<V> &m = src.mat(i);
    const int32_t r = w.trow[t];
    const int32_t n0 = w.tn0[t], mnew = w.tn0[t + 1] - n0;
    st.row = r;
    st.item = i;
    st.n0 = n0;
    st.mnew = mnew;
    int64_t cap = 0;
    int layer = -1, reloc = 0;
    st.len = m.row_sizes[r];
    st.start = -1;
    st.lo = 0;
    if constexpr (MERGE) {
      if (mnew > 0) {
        const int64_t L = st.len;
        const Chain ch = load_chain(m, r);
        const int64_t ins0 = w.nins[n0], nl = L + mnew;
        st.lo = (int32_t)ins0;
        if (ch.ns == 1 && nl <= ch.total) st.start = ch.st[0];
        if (L - ins0 > m.o.reloc_min) {
          reloc = 1;
        } else if (nl > ch.total) {
          layer = ch.total == 0 ? 0 : ch.ns;
          if (layer >= m.max_segs) reloc = 1;  // every layer in use: merged out of place, chain reset
          else cap = (policy_cap(m.o, nl) - ch.total + m.o.align - 1) & ~(int64_t)(m.o.align - 1);
        }
        if (reloc) {
          layer = 0;
          cap = policy_cap(m.o, nl);
          v[1] = (nl + RT_TILE - 1) / RT_TILE;
        } else {
          st.list = nl - ins0 > SMALL_AFF ? 2 : 1;
        }
      }
    } else {
      const int64_t rlB = mnew, rlA = st.len;
      const int2 l0 = *reinterpret_cast<const int2 *>(m.seg + 2 * (int64_t)r);
      if (rlA == 0 && l0.x == l0.y) {
        cap = rlB + m.o.alpha;
        layer = 0;
      } else {
        // segment holding position rlA (reference walk :77-88): the first
        // whose cumulative capacity reaches rlA; free = that capacity - rlA
        const Chain ch = load_chain(m, r);
        int off = 0;
        int64_t before = 0, after = 0;
        bool found = false;
#pragma unroll
        for (int q = 0; q < MAX_SEGS; q++) {
          if (!found && q < ch.ns) {
            after = before + ch.cp[q];
            off = q;
            if (after >= rlA || q + 1 >= ch.ns) found = true;
            else before = after;
          }
        }
        const int64_t fr = after - rlA;
        if (fr < rlB) {
          cap = rlB - fr + m.o.alpha;
          layer = off + 1;
          if (layer >= m.max_segs)
            atomicOr((unsigned long long *)&src.st(i)[ST_AUX], (unsigned long long)AUX_LAYER_OVF);
        }
      }
    }
    v[0] = cap;
    st.info = (layer & 0xff) | (reloc << 8);
  }
  // Lists of the rows to shift, and of the relocated ones: a warp's rows of
  // each take consecutive places, one atomic per warp for the first two (an
  // atomic per list and step queued up on the two words), one for the third.
  static constexpr bool EMIT_ALL = true;
  __device__ __forceinline__ void emit_all(int64_t base, int64_t, const State (&st)[IT], const T (&)[IT][2]) const {
    if (!MERGE) return;
    unsigned ms[IT], mb[IT], mr[IT], ns = 0, nb = 0, nr = 0;
#pragma unroll
    for (int j = 0; j < IT; j++) {
      ms[j] = __ballot_sync(FULL, st[j].list == 1);
      mb[j] = __ballot_sync(FULL, st[j].list == 2);
      mr[j] = __ballot_sync(FULL, st[j].row >= 0 && (st[j].info & 0x100));
      ns += __popc(ms[j]);
      nb += __popc(mb[j]);
      nr += __popc(mr[j]);
    }
    const unsigned lt = (1u << lane_id()) - 1u;
    if (nr) {  // the same in every lane
      unsigned long long at = 0;
      if (lane_id() == 0) at = atomicAdd((unsigned long long *)&w.gstat[ST_RELOC], (unsigned long long)nr);
      at = __shfl_sync(FULL, at, 0);
#pragma unroll
      for (int j = 0; j < IT; j++) {
        if (mr[j] >> lane_id() & 1u) w.reloc[at + __popc(mr[j] & lt)] = (int32_t)(base + 32 * j);
        at += __popc(mr[j]);
      }
    }
    if (ns + nb == 0) return;
    unsigned long long at = 0;
    if (lane_id() == 0)
      at = atomicAdd((unsigned long long *)&w.gstat[ST_LISTS], ((unsigned long long)nb << 32) | ns);
    at = __shfl_sync(FULL, at, 0);
    unsigned as = (unsigned)at, ab = (unsigned)(at >> 32);
#pragma unroll
    for (int j = 0; j < IT; j++) {
      const int32_t t = (int32_t)(base + 32 * j);
      if (st[j].list == 1) w.small[as + __popc(ms[j] & lt)] = t;
      if (st[j].list == 2) w.big[ab + __popc(mb[j] & lt)] = t;
      as += __popc(ms[j]);
      ab += __popc(mb[j]);
    }
  }
  __device__ __forceinline__ void emit(int64_t t, bool ok, const State &st, const long long (&p)[2],
                                       const T (&v)[2]) const {
    if (st.row < 0) return;
    RowDesc d;
    d.row = st.row;
    d.item = st.item;
    d.n0 = st.n0;
    d.mnew = st.mnew;
    d.len = st.len;
    d.start = st.start;
    d.lo = st.lo;
    d.info = st.info;
    d.cap = (int32_t)v[0];
    d.tile0 = (int32_t)p[1];
    d.addr = p[0];
    w.desc[t] = d;
    if (!ONE && (t == 0 || w.tmat[t - 1] != st.item)) {  // the first touched row of a matrix
      src.st(st.item)[ST_A0] = p[0];
      if (t > 0) src.st(w.tmat[t - 1])[ST_A1] = p[0];
    }
  }
  __device__ __forceinline__ void total(const long long (&t)[2]) const {
    w.gstat[ST_TOTAL] = t[0];
    w.gstat[ST_TILES] = t[1];
    if (ONE) {
      src.st(0)[ST_A1] = t[0];
      // MERGE: every input of the check is known (bad indices were flagged
      // by the key kernel); APPEND's layer overflows are still being flagged
      if (MERGE) check_item(src.mat(0), src.st(0));
    } else {
      const long long nt = w.gstat[ST_TOUCHED];
      if (nt > 0 && nt <= w.T) src.st(w.tmat[nt - 1])[ST_A1] = t[0];
    }
  }
};

// --------------------------------------------------------------- applying

// Apply, step 1 (thread per batch group): existing columns take their batch
// values in batch order, in place, before any shift or relocation reads them.
template <typename V, typename Src>
__global__ void k_apply_existing(Src src, UpdWork<V> w) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t g0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane_id(); g0 < w.T; g0 += stride) {  // (warps)
    const int64_t g = g0 + lane_id();
    const int32_t q = g < w.T ? w.bslot[g] : -1;
    const unsigned long long k = q >= 0 ? w.keys[g] : 0;
    const int i = w.f.item(k);
    const bool on = q >= 0 && src.st(i)[ST_GO];
    const V v = group_sum(src, w, on, i, k, g, on ? src.mat(i).vals[q] : V(0));
    if (on) src.mat(i).vals[q] = v;
  }
}

// The pool slot of a relocated or linked new segment.
template <typename V, typename Src>
__device__ __forceinline__ int32_t new_segment(const Src &src, const RowDesc &d) {
  const long long *st = src.st(d.item);
  return (int32_t)(st[ST_TOP] + (d.addr - st[ST_A0]));
}

// The segments of a row that is not in a single one, with its new one linked.
template <typename V, typename Src>
__device__ __forceinline__ Chain row_chain(const Src &src, const RowDesc &d, const Mat<V> &m, bool link) {
  Chain ch = load_chain(m, d.row);
  if (d.cap > 0) {
    const int32_t s = new_segment<V>(src, d);
    const int layer = (int8_t)(d.info & 0xff);
    ch.append(s, d.cap, layer == 0);
    if (link)
      *reinterpret_cast<int2 *>(m.seg + (int64_t)layer * m.pitch + 2 * (int64_t)d.row) = make_int2(s, s + d.cap);
  }
  return ch;
}

// A stretch of a row in its new order: positions d0 .. d0+n-1, n <= S*E.  New
// column k lands at ins[k] + k (strictly increasing), so a bit mask of those
// positions gives every position its source: a set bit takes the next new
// column, the others the old entry as many places before as bits are set up
// to there -- loads and stores both run along the row.  k0: new columns
// before d0, k1: before d0+n.  Every load comes before the first store (the
// row may be moved in place, last stretch first: a stretch writes only where
// entries have already been read).  8 lanes: the mask is one word in
// registers; a warp: E words of shared memory.
template <int S, int E, typename V, typename From, typename To>
__device__ __forceinline__ void move_stretch(const Sub<S> &sub, unsigned *mask, const Mat<V> &m, From &&from, To &&to,
                                             int32_t d0, int n, int32_t k0, int32_t k1, const int32_t *ins,
                                             const int32_t *ncol, const V *nval) {
  constexpr bool WIDE = S == 32;
  static_assert(WIDE || S * E == 32, "one mask word");
  unsigned word = 0;
  if constexpr (WIDE) {
    if (sub.sl < E) mask[sub.sl] = 0;
    sub.sync();
    for (int32_t k = k0 + sub.sl; k < k1; k += S) {
      const int p = ins[k] + k - d0;
      atomicOr(&mask[p >> 5], 1u << (p & 31));
    }
    sub.sync();
  } else {
    for (int32_t k = k0 + sub.sl; k < k1; k += S) word |= 1u << (ins[k] + k - d0);
#pragma unroll
    for (int o = S / 2; o > 0; o >>= 1) word |= __shfl_xor_sync(sub.mask, word, o, S);
  }
  int32_t col[E], base = k0;
  V val[E];
#pragma unroll
  for (int i = 0; i < E; i++) {
    const int p = i * S + sub.sl;
    const unsigned b = WIDE ? mask[i] : word;
    const int bit = WIDE ? sub.sl : p;
    const int32_t r = base + __popc(b & ((2u << bit) - 1u));  // new columns at or before p
    if (p < n) {
      if ((b >> bit) & 1) {
        col[i] = ncol[r - 1];
        val[i] = nval[r - 1];
      } else {
        const int64_t q = from(d0 + p - r);
        col[i] = m.cols[q];
        val[i] = m.vals[q];
      }
    }
    if (WIDE) base += __popc(b);
  }
  sub.sync();
#pragma unroll
  for (int i = 0; i < E; i++) {
    const int p = i * S + sub.sl;
    if (p < n) {
      const int64_t q = to(d0 + p);
      m.cols[q] = col[i];
      m.vals[q] = val[i];
    }
  }
  sub.sync();
}

// In-place insertion into one row by S lanes: the positions from the first
// insertion point on, in stretches from the row's new end.  Measured on the
// R-MAT 2^20 stream's update by 1M triples (190k rows, 8.6M entries moved, 217
// rows relocated): 118 us for all of k_apply_rows; an entry per lane and step,
// its place by a histogram of the insertion points, in three launches that
// each walked all touched rows, took 256 us for the rows shifting more than
// 96 entries, 107 us for the others and 43 us for the relocations.  Bound by
// each row's chain of round trips (descriptor, insertion points, entries) at
// 24 warps per SM.
template <int S, int E, typename V, typename At>
__device__ __forceinline__ void insert_row(const Sub<S> &sub, unsigned *mask, const Mat<V> &m, At &&at, int32_t L,
                                           int32_t lo, int32_t mnew, const int32_t *ins, const int32_t *ncol,
                                           const V *nval) {
  int32_t k1 = mnew;
  for (int32_t d1 = L + mnew; d1 > lo;) {
    const int32_t d0 = d1 - S * E > lo ? d1 - S * E : lo;
    int32_t k0 = 0;
    if (d0 > lo) {  // new columns before d0
      k0 = k1;
      for (;;) {
        const int32_t k = k0 - 1 - sub.sl;
        const int c = sub.leading(sub.ballot(k >= 0 && ins[k] + k >= d0));
        k0 -= c;
        if (c < S) break;
      }
    }
    move_stretch<S, E>(sub, mask, m, at, at, d0, d1 - d0, k0, k1, ins, ncol, nval);
    d1 = d0;
    k1 = k0;
  }
}

// The rows of one list, S lanes each.  The next row's descriptor and the
// number of the one after are loaded while a row is worked on.
template <int S, int E, typename V, typename Src>
__device__ __forceinline__ void apply_list(const Src &src, const UpdWork<V> &w, unsigned *mask, const int32_t *list,
                                           int64_t n) {
  const Sub<S> sub;
  const int64_t step = (int64_t)gridDim.x * blockDim.x / S;
  int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / S;
  if (i >= n) return;
  RowDesc d = w.desc[list[i]];
  int32_t t = i + step < n ? list[i + step] : -1;
  while (i < n) {
    RowDesc next = d;
    if (t >= 0) next = w.desc[t];
    i += step;
    t = i + step < n ? list[i + step] : -1;
    if (src.st(d.item)[ST_GO]) {
      const Mat<V> &m = src.mat(d.item);
      const int32_t *ins = w.nins + d.n0, *ncol = w.ncol + d.n0;
      const V *nval = w.nval + d.n0;
      if (d.start >= 0) {
        const int64_t s0 = d.start;
        insert_row<S, E>(sub, mask, m, [&](int32_t p) { return s0 + p; }, d.len, d.lo, d.mnew, ins, ncol, nval);
      } else {
        const Chain ch = row_chain(src, d, m, sub.sl == 0);
        insert_row<S, E>(sub, mask, m, [&](int32_t p) { return ch.phys(p); }, d.len, d.lo, d.mnew, ins, ncol, nval);
      }
      if (sub.sl == 0) m.row_sizes[d.row] = d.len + d.mnew;
    }
    sub.sync();
    d = next;
  }
}

// Relocation of rows into fresh segments, a warp per RT_TILE positions.  A
// tile's row is the last touched row with no more tiles before it than the
// tile's number (rows without tiles share theirs with the next row's): the
// relocated rows need no order of their own, and no count in the plan's scan.
template <typename V, typename Src>
__device__ __forceinline__ void relocate_tiles(const Src &src, const UpdWork<V> &w, unsigned *mask) {
  const Sub<32> sub;
  const int64_t ntiles = w.gstat[ST_TILES], nt = w.gstat[ST_TOUCHED];
  const int lane = lane_id();
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x / 32);
  // the number of leading i in [0, n) for which f(i) holds: 32 probes a step
  auto leading = [&](int64_t n, auto &&f) -> int64_t {
    int64_t lo = 0, hi = n + 1;  // the answer is in [lo, hi)
    while (hi - lo > 1) {
      const int64_t span = hi - lo;
      auto probe = [&](int q) { return lo + (span * q + 32) / 33; };  // q = 1 .. 32, growing, > lo
      const int64_t p = probe(lane + 1);
      const int c = __popc(__ballot_sync(FULL, p < hi && f(p - 1)));  // the first c probes hold
      const int64_t nhi = c < 32 ? probe(c + 1) : hi, nlo = c ? probe(c) : lo;
      hi = nhi < hi ? nhi : hi;
      lo = nlo;
    }
    return lo;
  };
  for (int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32; q < ntiles; q += nw) {
    const int64_t at = leading(nt, [&](int64_t i) { return w.desc[i].tile0 <= q; }) - 1;
    const RowDesc d = w.desc[at];
    if (!src.st(d.item)[ST_GO]) continue;
    const Mat<V> &m = src.mat(d.item);
    const Chain ch = load_chain(m, d.row);
    const int64_t to = new_segment<V>(src, d);
    const int32_t *ins = w.nins + d.n0;
    const int32_t d0 = (int32_t)(q - d.tile0) * RT_TILE, d1 = min(d.len + d.mnew, d0 + RT_TILE);
    const int32_t k0 = (int32_t)leading(d.mnew, [&](int64_t k) { return ins[k] + k < d0; });
    int32_t k1 = k0;
    for (;;) {
      const int32_t k = k1 + lane;
      const int c = sub.leading(sub.ballot(k < d.mnew && ins[k] + k < d1));
      k1 += c;
      if (c < 32) break;
    }
    move_stretch<32, RT_TILE / 32>(sub, mask, m, [&](int32_t p) { return ch.phys(p); },
                                   [&](int32_t p) { return to + p; }, d0, d1 - d0, k0, k1, ins, w.ncol + d.n0,
                                   w.nval + d.n0);
  }
}

// Apply, step 2: relocation tiles, larger shifts, small shifts, whichever
// warp is free for them -- different rows, so in any order.
template <typename V, typename Src>
__global__ void __launch_bounds__(UPD_THREADS, 3) k_apply_rows(Src src, UpdWork<V> w) {
  __shared__ __align__(16) unsigned masks[UPD_THREADS / 32][8];
  unsigned *mask = masks[threadIdx.x >> 5];
  relocate_tiles(src, w, mask);
  apply_list<32, 8>(src, w, mask, w.big, (unsigned long long)w.gstat[ST_LISTS] >> 32);
  apply_list<8, 4>(src, w, mask, w.small, w.gstat[ST_LISTS] & 0xffffffff);
}

template <typename V, typename Src>
__global__ void k_finish(Src src, UpdWork<V> w, int count, int merge) {
  const int64_t nr = w.gstat[ST_RELOC];
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (merge)
    for (int64_t r = tid; r < nr; r += stride) {
      const RowDesc d = w.desc[w.reloc[r]];
      if (!src.st(d.item)[ST_GO]) continue;
      const Mat<V> &m = src.mat(d.item);
      const int32_t s = new_segment<V>(src, d);
      for (int l = 1; l < m.max_segs; l++)
        *reinterpret_cast<int2 *>(m.seg + (int64_t)l * m.pitch + 2 * (int64_t)d.row) = make_int2(-1, -1);
      *reinterpret_cast<int2 *>(m.seg + 2 * (int64_t)d.row) = make_int2(s, s + d.cap);
      m.row_sizes[d.row] = d.len + d.mnew;
    }
  for (int64_t i = tid; i < count; i += stride) {
    const long long *st = src.st((int)i);
    if (st[ST_GO]) {
      const Mat<V> &m = src.mat((int)i);
      m.row_sizes[m.n_rows] = (int32_t)st[ST_NEED];
    }
  }
}

// APPEND: every touched row's triples after its last entry, 8 lanes per row;
// what a row has past its first 64 by the whole warp, 128 in flight (100,000
// triples of one row: 0.76 ms, 6.1 with one at a time in each of the 8 lanes).
template <typename V, typename Src>
__global__ void __launch_bounds__(UPD_THREADS) k_apply_append(Src src, UpdWork<V> w) {
  constexpr int S = 8, FIRST = 64;
  const Sub<S> sub;
  const int lane = lane_id();
  const int64_t nt = w.gstat[ST_TOUCHED];
  const int64_t step = (int64_t)gridDim.x * blockDim.x / S;
  // triples j0, j0 + lanes, ... below j1 of a row of len entries before, U in flight
  auto put = [&](auto u_, int item, int32_t n0, int32_t len, const Chain &ch, int32_t j0, int32_t j1, int lanes) {
    constexpr int U = decltype(u_)::value;
    const Mat<V> &m = src.mat(item);
    for (; j0 < j1; j0 += U * lanes) {
      int64_t p[U];
      int32_t c[U];
      V v[U];
#pragma unroll
      for (int u = 0; u < U; u++) p[u] = j0 + u * lanes < j1 ? src.local(item, w.perm[n0 + j0 + u * lanes]) : -1;
#pragma unroll
      for (int u = 0; u < U; u++) {
        c[u] = p[u] >= 0 ? src.ucols(item)[p[u]] : 0;
        v[u] = p[u] >= 0 ? src.uvals(item)[p[u]] : V(0);
      }
#pragma unroll
      for (int u = 0; u < U; u++)
        if (p[u] >= 0) {
          const int64_t q = ch.phys(len + j0 + u * lanes);
          m.cols[q] = c[u];
          m.vals[q] = v[u];
        }
    }
  };
  for (int64_t t0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ll) / S; t0 < nt; t0 += step) {  // (warps)
    const int64_t t = t0 + sub.sw;
    RowDesc d = w.desc[t < nt ? t : t0];
    const bool on = t < nt && src.st(d.item)[ST_GO];
    Chain ch;
#pragma unroll
    for (int l = 0; l < MAX_SEGS; l++) ch.st[l] = ch.cp[l] = 0;
    ch.ns = 0;
    ch.total = 0;
    if (on) {
      const Mat<V> &m = src.mat(d.item);
      ch = row_chain(src, d, m, sub.sl == 0);
      put(std::integral_constant<int, 1>(), d.item, d.n0, d.len, ch, sub.sl, d.mnew < FIRST ? d.mnew : FIRST, S);
      if (sub.sl == 0) m.row_sizes[d.row] = d.len + d.mnew;
    }
    unsigned longs = __ballot_sync(FULL, on && sub.sl == 0 && d.mnew > FIRST);
    while (longs) {
      const int s = __ffs(longs) - 1;
      longs &= longs - 1;
      put(std::integral_constant<int, 4>(), __shfl_sync(FULL, d.item, s), __shfl_sync(FULL, d.n0, s),
          __shfl_sync(FULL, d.len, s), shfl_chain(ch, s), FIRST + lane, __shfl_sync(FULL, d.mnew, s), 32);
    }
  }
}

// ------------------------------------------------------------ host driver

static int grid_for(int64_t n, int block) {
  int64_t g = div_up(n, block);
  int64_t cap = (int64_t)sm_count() * 16;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

size_t update_scratch_bytes(int64_t T, size_t vsize) {
  return 2 * arena_bytes(T, 8) + 2 * arena_bytes(T, 4) + 7 * arena_bytes(T + 2, 4) + arena_bytes(T, vsize) +
         arena_bytes(T, sizeof(RowDesc)) + radix_scratch_bytes(T) + scan_scratch_bytes(T + 2);
}

template <typename V, bool MERGE, bool ONE, typename Src>
static int update_plan(const Src &src, const UpdWork<V> &w, Arena &ar, cudaStream_t s) {
  return scan_map(PlanScan<V, Src, MERGE, ONE>{src, w}, w.T, ar, s);
}

// The update of `count` matrices (one Src) with T triples in total.
// gstat: batch-global status words (ST_TOUCHED, ST_TILES, ST_RELOC, ST_TOTAL, ST_LISTS).
// pool: pool entries of all matrices, an upper bound of what relocations move.
template <typename V, bool ONE, typename Src>
static int update_pipeline(const Src &src, int count, int64_t T, int64_t pool, bool merge, int rb, int cb,
                           long long *gstat, Arena &ar, cudaStream_t s) {
  const int ib = count > 1 ? bits_for(count) : 0;
  const KeyFmt f{cb, rb, merge ? 1 : 0};
  const int bits = ib + rb + (merge ? cb : 0);
  if (bits > 63) return DCSR_NOT_SUPPORTED;
  DCSR_TRY(ar.reserve(update_scratch_bytes(T, sizeof(V)), s));
  unsigned long long *k0 = ar.take<unsigned long long>(T), *k1 = ar.take<unsigned long long>(T);
  unsigned *p0 = ar.take<unsigned>(T), *p1 = ar.take<unsigned>(T);
  UpdWork<V> w;
  std::memset(&w, 0, sizeof(w));
  w.T = T;
  w.f = f;
  w.gstat = gstat;
  w.bslot = ar.take<int32_t>(T + 2);
  w.trow = ar.take<int32_t>(T + 2);
  w.tmat = ar.take<int32_t>(T + 2);
  w.tn0 = ar.take<int32_t>(T + 2);
  w.reloc = ar.take<int32_t>(T + 2);
  w.small = ar.take<int32_t>(T + 2);
  w.big = ar.take<int32_t>(T + 2);
  w.nval = ar.take<V>(T);
  w.desc = ar.take<RowDesc>(T);
  if (ar.overflow) return DCSR_OOM;  // scratch sizing bug: no kernel sees a null pointer
  const int gT = grid_for(T + 1, 256);
  const int gI = grid_for(count, 256);

  DCSR_LAUNCH((k_item_init<V, Src>), gI, 256, 0, s, src, count, gstat);
  DCSR_LAUNCH((k_make_keys<V, Src>), gT, 256, 0, s, src, T, f, k0, p0);
  DCSR_TRY(radix_sort_pairs(&k0, &p0, &k1, &p1, T, bits, ar, s));
  // k1 is free after the sort: the new columns and their insertion points
  w.keys = k0;
  w.perm = p0;
  w.ncol = (int32_t *)k1;
  w.nins = w.ncol + T;
  if (merge) {
    DCSR_TRY(scan_map(GroupScan<V, Src>{src, w}, T, ar, s));
    DCSR_TRY((update_plan<V, true, ONE>(src, w, ar, s)));
  } else {
    DCSR_TRY(scan_map(RowHeadScan<V, Src>{src, w}, T, ar, s));
    DCSR_TRY((update_plan<V, false, ONE>(src, w, ar, s)));
  }
  if (!merge || !ONE) DCSR_LAUNCH((k_check<V, Src>), gI, 256, 0, s, src, count);
  if (merge) {
    static const int g_apply = persistent_grid((const void *)k_apply_rows<V, Src>, UPD_THREADS, 0);
    DCSR_LAUNCH((k_apply_existing<V, Src>), gT, 256, 0, s, src, w);
    // warps for the triples' rows, and for the tiles of the rows they may
    // relocate: one triple can move a row of millions (20 triples into rows of 1M
    // and 2M entries: 205 us, 1170 with warps for the triples alone)
    const int64_t warps = std::max(T, div_up(pool, RT_TILE));
    DCSR_LAUNCH((k_apply_rows<V, Src>), (int)std::min<int64_t>(g_apply, div_up(warps, UPD_THREADS / 32)), UPD_THREADS, 0,
                s, src, w);
  } else {
    static const int g_apply = persistent_grid((const void *)k_apply_append<V, Src>, UPD_THREADS, 0);
    DCSR_LAUNCH((k_apply_append<V, Src>), (int)std::min<int64_t>(g_apply, div_up(T, UPD_THREADS / 8)), UPD_THREADS, 0,
                s, src, w);
  }
  DCSR_LAUNCH((k_finish<V, Src>), grid_for(std::max<int64_t>(count, merge ? div_up(T, 64) : 1), 256), 256, 0, s, src, w, count, merge ? 1 : 0);
  return DCSR_OK;
}

template <typename V>
static int update_one(dcsr_handle h, const int32_t *rows, const int32_t *cols, const V *vals, int64_t T,
                      cudaStream_t s, Arena &ar) {
  UpdOne<V> src{h->view<V>(), rows, cols, vals};
  DCSR_TRY((update_pipeline<V, true>(src, 1, T, h->pool_cap, h->o.mode == DCSR_MERGE, bits_for(h->n_rows), bits_for(h->n_cols), h->stat,
                                     ar, s)));
  const unsigned long long cap = capture_id(s);
  h->bins.changed(cap);
  h->flat.changed(cap);
  return DCSR_OK;
}

int update_async(dcsr_handle h, const int32_t *rows, const int32_t *cols, const void *vals, int64_t nnz,
                 cudaStream_t s, Arena *ar) {
  if (nnz == 0) return DCSR_OK;
  if (nnz > 0x7ffffff0LL) return DCSR_BAD_ARG;
  Arena &a = ar ? *ar : h->scratch;
  a.status = h->stat + ST_STATUS;  // a look-back wait that gives up reports DCSR_TIMEOUT here
  if (h->dtype == DCSR_F32) return update_one<float>(h, rows, cols, (const float *)vals, nnz, s, a);
  return update_one<double>(h, rows, cols, (const double *)vals, nnz, s, a);
}

template <typename V>
static int update_many_t(const BatchItem<V> *items_dev, int count, int64_t T, int64_t pool, bool merge, int rb, int cb,
                         long long *gstat, Arena &ar, cudaStream_t s) {
  UpdMany<V> src{items_dev, count};
  return update_pipeline<V, false>(src, count, T, pool, merge, rb, cb, gstat, ar, s);
}

int update_many(const void *items_dev, int dtype, int count, int64_t T, int64_t pool, bool merge, int rb, int cb,
                long long *gstat, Arena &ar, cudaStream_t s) {
  if (T == 0 || count == 0) return DCSR_OK;
  ar.status = gstat + ST_STATUS;  // a look-back wait that gives up reports DCSR_TIMEOUT for the batch
  if (dtype == DCSR_F32)
    return update_many_t<float>((const BatchItem<float> *)items_dev, count, T, pool, merge, rb, cb, gstat, ar, s);
  return update_many_t<double>((const BatchItem<double> *)items_dev, count, T, pool, merge, rb, cb, gstat, ar, s);
}

// ------------------------------------------------------------- COO -> CSR

__global__ void k_coo_keys(const int32_t *rows, const int32_t *cols, int64_t n, int32_t n_rows, int32_t n_cols,
                           int cb, int merge, unsigned long long *keys, unsigned *perm, long long *stat) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    int32_t r = rows[i], c = cols[i];
    if (r < 0 || r >= n_rows || c < 0 || c >= n_cols) {
      atomicOr((unsigned long long *)&stat[ST_AUX], (unsigned long long)AUX_BAD_INDEX);
      r = 0;
      c = 0;
    }
    keys[i] = merge ? (((unsigned long long)r << cb) | (unsigned long long)c) : (unsigned long long)r;
    perm[i] = (unsigned)i;
  }
}

// Sorted triples -> CSR columns and values and the rows' counts, in one pass:
// a scan over group heads (MERGE: the first triple of each (row, column), the
// group's values added up in input order; else every triple), whose position
// is where the entry goes.  The pass is bound by the gather of the values
// through the permutation (a random sector each: 540 MB of L2 traffic of 16.7M
// triples), so a thread has its 8 triples' keys, then indices, then values in
// flight together, before the look-back.  With a pass for flags, their scan
// and a pass for the entries, 16 bytes of flags a triple written and read
// twice, the three took 492 us of 16.7M triples; this one 272 us (3 blocks per
// SM; 2 or 4, with more spilled registers: 20-40 us more).
template <typename V, bool MERGE>
struct CooScan {
  static constexpr int NS = 1, IT = SM_LIGHT;
  static constexpr bool LOAD_ALL = true, EMIT_ALL = MERGE;  // (no groups to add up in append mode)
  using T = int32_t;
  struct State {
    unsigned long long key;
    V val;
    int32_t col;
  };
  const unsigned long long *keys;
  const unsigned *perm;
  const int32_t *cols;
  const V *vals;
  int64_t n;
  int cb;
  int32_t n_cols;
  int32_t *ocols;
  V *ovals;
  int32_t *rowcnt;
  __device__ __forceinline__ int32_t row(unsigned long long k) const { return (int32_t)(MERGE ? k >> cb : k); }
  __device__ __forceinline__ void load_all(int64_t base, int64_t, State (&st)[IT], T (&v)[IT][1]) const {
    const int lane = lane_id();
    unsigned at[IT];
#pragma unroll
    for (int j = 0; j < IT; j++) {
      const int64_t i = base + 32 * j;
      st[j].key = i < n ? __ldcs(keys + i) : ~0ull;
      at[j] = i < n ? __ldcs(perm + i) : 0u;
    }
#pragma unroll
    for (int j = 0; j < IT; j++) {
      const int64_t i = base + 32 * j;
      st[j].val = i < n ? vals[at[j]] : V(0);
      st[j].col = 0;
      if constexpr (!MERGE) st[j].col = i < n ? cols[at[j]] : 0;
    }
    // a triple is in the group of the one before it, or starts its own
    const int64_t w0 = base - lane;  // the warp's first triple
    unsigned long long carry = ~0ull;
    if (MERGE && lane == 0 && w0 > 0 && w0 <= n) carry = keys[w0 - 1];
#pragma unroll
    for (int j = 0; j < IT; j++) {
      const int64_t i = base + 32 * j;
      unsigned long long prev = __shfl_up_sync(FULL, st[j].key, 1);
      if (lane == 0) prev = carry;
      carry = __shfl_sync(FULL, st[j].key, 31);
      v[j][0] = i < n && !(MERGE && i > 0 && prev == st[j].key) ? 1 : 0;
    }
  }
  // Groups of several triples: the head's value takes the others' in input
  // order.  The triples of a warp are added by shuffle -- a step's groups side
  // by side, a group that began in an earlier step by the whole warp -- and
  // those past the warp's last 32 at a time, so a group's sum is a chain of
  // additions, not of loads (a power-law graph's hottest edge comes up
  // hundreds of times; a thread that walked its group through keys, indices
  // and values held its warp for 0.6 us a triple).
  __device__ __forceinline__ void emit_all(int64_t base, int64_t, State (&st)[IT], const T (&v)[IT][1]) const {
    const int lane = lane_id();
    const int64_t w1 = base - lane + 32 * IT;  // past the warp's triples
    V cx = V(0);  // the sum of the last group so far, and where its head is
    int jo = -1, lo = 0;
#pragma unroll
    for (int j = 0; j < IT; j++) {
      const unsigned heads = __ballot_sync(FULL, v[j][0] != 0);
      const unsigned same = __ballot_sync(FULL, base + 32 * j < n) & ~heads;
      V x = st[j].val;
      if (same) {
        const unsigned rest = lane < 31 ? ~(same >> (lane + 1)) : FULL;
        const int run = v[j][0] && rest ? __ffs(rest) - 1 : 0;  // triples of this head's group in this step
        const int longest = (int)__reduce_max_sync(FULL, (unsigned)run);
        for (int d = 1; d <= longest; d++) {
          const V o = __shfl_down_sync(FULL, st[j].val, d);
          if (d <= run) x = x + o;
        }
        if ((same & 1u) && jo >= 0) {  // the group open from an earlier step
          const int lead = ~same ? __ffs(~same) - 1 : 32;
          for (int q = 0; q < lead; q++) cx = cx + __shfl_sync(FULL, st[j].val, q);
#pragma unroll
          for (int i = 0; i < j; i++)
            if (i == jo && lane == lo) st[i].val = cx;
        }
        st[j].val = x;
      }
      if (heads) {
        jo = j;
        lo = 31 - __clz(heads);
        cx = __shfl_sync(FULL, x, lo);
      }
    }
    if (jo < 0 || w1 >= n) return;
    const unsigned long long k = __shfl_sync(FULL, st[IT - 1].key, 31);
    bool more = keys[w1] == k;
    if (!more) return;
    for (int64_t at = w1; more; at += 32) {
      const int64_t i = at + lane;
      const unsigned in = __ballot_sync(FULL, i < n && keys[i < n ? i : w1] == k);
      const int cnt = ~in ? __ffs(~in) - 1 : 32;
      const V o = lane < cnt ? vals[perm[i]] : V(0);
      for (int q = 0; q < cnt; q++) cx = cx + __shfl_sync(FULL, o, q);
      more = cnt == 32;
    }
#pragma unroll
    for (int i = 0; i < IT; i++)
      if (i == jo && lane == lo) st[i].val = cx;
  }
  __device__ __forceinline__ void emit(int64_t i, bool ok, const State &st, const long long (&p)[1],
                                       const T (&v)[1]) const {
    const int lane = lane_id();
    if (v[0]) {
      int32_t c = MERGE ? (int32_t)(st.key & ((1ull << cb) - 1)) : st.col;
      if (c < 0 || c >= n_cols) c = 0;
      ocols[p[0]] = c;
      ovals[p[0]] = st.val;
    }
    // row counts, one atomic per row and warp step: the keys are sorted, so 32
    // triples are a few runs of one row each
    const int32_t r = ok ? row(st.key) : -1;
    const int32_t prev = __shfl_up_sync(FULL, r, 1);
    const unsigned starts = __ballot_sync(FULL, lane == 0 || prev != r);
    const unsigned heads = __ballot_sync(FULL, v[0] != 0);
    if (r >= 0 && (starts >> lane & 1u)) {
      const unsigned later = starts & ~((2u << lane) - 1u);  // lane 31: 2u << 31 is 0
      const unsigned run = (later ? (later & -later) - 1u : FULL) & ~((1u << lane) - 1u);
      const int c = __popc(heads & run);
      if (c) atomicAdd(&rowcnt[r], c);
    }
  }
  __device__ __forceinline__ void total(const long long (&)[1]) const {}
};

size_t coo_to_csr_scratch(dcsr_handle h, int64_t T) {
  return 2 * arena_bytes(T, 8) + 2 * arena_bytes(T, 4) + arena_bytes(T, 4) + arena_bytes(T, 8) +
         3 * arena_bytes(h->n_rows + 2, 4) + radix_scratch_bytes(T) +
         scan_scratch_bytes(std::max<int64_t>(T, h->n_rows + 1));
}

template <typename V>
static int coo_impl(dcsr_handle h, const int32_t *rows, const int32_t *cols, const V *vals, int64_t T, bool merge,
                    Arena &ar, int32_t **rp, int32_t **caps, int32_t **ocols, void **ovals, cudaStream_t s) {
  const int cb = bits_for(h->n_cols), rb = bits_for(h->n_rows);
  unsigned long long *k0 = ar.take<unsigned long long>(T), *k1 = ar.take<unsigned long long>(T);
  unsigned *p0 = ar.take<unsigned>(T), *p1 = ar.take<unsigned>(T);
  int32_t *oc = ar.take<int32_t>(T);
  V *ov = (V *)ar.take<double>(T);
  int32_t *cnt = ar.take<int32_t>(h->n_rows + 2);
  *rp = ar.take<int32_t>(h->n_rows + 2);
  *caps = ar.take<int32_t>(h->n_rows + 2);
  if (ar.overflow) return DCSR_OOM;  // scratch sizing bug: no kernel sees a null pointer
  DCSR_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int32_t) * (h->n_rows + 2), s));
  if (T > 0) {
    DCSR_LAUNCH(k_coo_keys, grid_for(T, 256), 256, 0, s, rows, cols, T, h->n_rows, h->n_cols, cb, merge ? 1 : 0, k0,
                p0, h->stat);
    DCSR_TRY(radix_sort_pairs(&k0, &p0, &k1, &p1, T, merge ? rb + cb : rb, ar, s));
    if (merge) DCSR_TRY(scan_map(CooScan<V, true>{k0, p0, cols, vals, T, cb, h->n_cols, oc, ov, cnt}, T, ar, s));
    else DCSR_TRY(scan_map(CooScan<V, false>{k0, p0, cols, vals, T, cb, h->n_cols, oc, ov, cnt}, T, ar, s));
  }
  DCSR_TRY(counts_scan(h, cnt, *rp, *caps, ar, s));
  *ocols = oc;
  *ovals = ov;
  return DCSR_OK;
}

int coo_to_csr(dcsr_handle h, const int32_t *rows, const int32_t *cols, const void *vals, int64_t nnz, bool merge,
               Arena &ar, int32_t **rp, int32_t **caps, int32_t **ocols, void **ovals, cudaStream_t s) {
  if (h->dtype == DCSR_F32)
    return coo_impl<float>(h, rows, cols, (const float *)vals, nnz, merge, ar, rp, caps, ocols, ovals, s);
  return coo_impl<double>(h, rows, cols, (const double *)vals, nnz, merge, ar, rp, caps, ocols, ovals, s);
}

}  // namespace dcsr
