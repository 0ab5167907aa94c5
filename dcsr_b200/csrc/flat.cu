// flat.cu -- entry-parallel copies between CSR order and a matrix's pool: the
// CSR/COO load (CSR -> pool), SpGEMM's placement (staged rows -> pool), the
// export (pool -> CSR/COO) and the compaction (pool -> fresh pool), all in
// tiles of FT_TILE entries (flat.cuh).
//
// Bound: HBM, 2*(4+sV) bytes per entry plus the offsets.  A warp or group of
// lanes per row left most lanes idle on the short rows of a power-law matrix
// and its hub rows to single warps; tiles of equal entry counts keep every
// lane at eight entries in flight and both sides coalesced row by row.
//
// Reference: CompactIndices include/sparse_update.inl:916-1007,
// DCSRtoCSROffsets :1101-1116, LoadMatrix include/load.h:207-253.
#include "flat.cuh"
#include "internal.cuh"
#include "lookback.cuh"

namespace dcsr {

namespace {

// Row lengths -> CSR row pointer and tile rows.
struct OffsetsScan {
  static constexpr int NS = 1, IT = SM_LIGHT;
  using T = int32_t;
  struct State {};
  const int32_t *sizes;
  int32_t n;
  int32_t *off, *tile_row;
  int64_t tiles;
  __device__ __forceinline__ void load(int64_t i, bool ok, State &, T (&v)[1]) const { v[0] = ok && i < n ? sizes[i] : 0; }
  __device__ __forceinline__ void emit(int64_t i, bool ok, const State &, const long long (&p)[1],
                                       const T (&v)[1]) const {
    if (ok && i < n) off[i] = (int32_t)p[0];
    flat_mark_tiles((int32_t)i, p[0], v[0], tile_row, tiles);
  }
  __device__ __forceinline__ void total(const long long (&t)[1]) const { off[n] = (int32_t)t[0]; }
  __device__ __forceinline__ void fault() const { off[n] = FLAT_BAD; }
};

// Row lengths -> CSR row pointer, tile rows and the offsets of the policy's
// capacities (compaction); the capacities' sum goes to *top.
struct CompactScan {
  static constexpr int NS = 2, IT = SM_LIGHT;
  using T = long long;
  struct State {};
  const int32_t *sizes;
  int32_t n;
  dcsr_opts o;
  int32_t *off, *tile_row, *caps;
  int64_t tiles;
  long long *top;
  __device__ __forceinline__ void load(int64_t i, bool ok, State &, T (&v)[2]) const {
    v[1] = ok && i < n ? sizes[i] : 0;
    v[0] = ok && i < n ? policy_cap(o, v[1]) : 0;
  }
  __device__ __forceinline__ void emit(int64_t i, bool ok, const State &, const long long (&p)[2],
                                       const T (&v)[2]) const {
    if (ok && i < n) {
      off[i] = (int32_t)p[1];
      caps[i] = (int32_t)p[0];
    }
    flat_mark_tiles((int32_t)i, p[1], v[1], tile_row, tiles);
  }
  __device__ __forceinline__ void total(const long long (&t)[2]) const {
    off[n] = (int32_t)t[1];
    caps[n] = (int32_t)t[0];
    *top = t[0];
  }
};

// CSR row pointer -> offsets of the policy's capacities; their sum to *top.
struct CapsScan {
  static constexpr int NS = 1, IT = SM_LIGHT;
  using T = long long;
  struct State {};
  const int32_t *rp;
  int32_t n;
  dcsr_opts o;
  int32_t *caps;
  long long *top;
  __device__ __forceinline__ void load(int64_t i, bool ok, State &, T (&v)[1]) const {
    v[0] = ok && i < n ? policy_cap(o, rp[i + 1] - rp[i]) : 0;
  }
  __device__ __forceinline__ void emit(int64_t i, bool ok, const State &, const long long (&p)[1],
                                       const T (&)[1]) const {
    if (ok && i < n) caps[i] = (int32_t)p[0];
  }
  __device__ __forceinline__ void total(const long long (&t)[1]) const {
    caps[n] = (int32_t)t[0];
    *top = t[0];
  }
};

// Row counts of a grouped COO batch -> CSR row pointer and the offsets of the
// policy's capacities; the capacities' sum to *top.
struct CountScan {
  static constexpr int NS = 2, IT = SM_LIGHT;
  using T = long long;
  struct State {};
  const int32_t *cnt;
  int32_t n;
  dcsr_opts o;
  int32_t *rp, *caps;
  long long *top;
  __device__ __forceinline__ void load(int64_t i, bool ok, State &, T (&v)[2]) const {
    v[1] = ok && i < n ? cnt[i] : 0;
    v[0] = ok && i < n ? policy_cap(o, v[1]) : 0;
  }
  __device__ __forceinline__ void emit(int64_t i, bool ok, const State &, const long long (&p)[2],
                                       const T (&)[2]) const {
    if (ok && i < n) {
      rp[i] = (int32_t)p[1];
      caps[i] = (int32_t)p[0];
    }
  }
  __device__ __forceinline__ void total(const long long (&t)[2]) const {
    rp[n] = (int32_t)t[1];
    caps[n] = (int32_t)t[0];
    *top = t[0];
  }
};

// Staged rows of given lengths -> CSR offsets, tile rows, capacity offsets and
// the new layout itself (row lengths, layer 0, other layers cleared).
struct PlaceScan {
  static constexpr int NS = 2, IT = SM_LIGHT;
  using T = long long;
  struct State {};
  const long long *lens;
  int32_t n;
  dcsr_opts o;
  int32_t *off, *tile_row, *caps, *row_sizes, *seg;
  int32_t pitch, max_segs;
  int64_t tiles;
  long long *top;
  __device__ __forceinline__ void load(int64_t i, bool ok, State &, T (&v)[2]) const {
    v[1] = ok && i < n ? lens[i] : 0;
    v[0] = ok && i < n ? policy_cap(o, v[1]) : 0;
  }
  __device__ __forceinline__ void emit(int64_t i, bool ok, const State &, const long long (&p)[2],
                                       const T (&v)[2]) const {
    if (ok && i < n) {
      off[i] = (int32_t)p[1];
      caps[i] = (int32_t)p[0];
      row_sizes[i] = (int32_t)v[1];
      *reinterpret_cast<int2 *>(seg + 2 * i) = make_int2((int32_t)p[0], (int32_t)(p[0] + v[0]));
      for (int l = 1; l < max_segs; l++)
        *reinterpret_cast<int2 *>(seg + (int64_t)l * pitch + 2 * i) = make_int2(-1, -1);
    }
    flat_mark_tiles((int32_t)i, p[1], v[1], tile_row, tiles);
  }
  __device__ __forceinline__ void total(const long long (&t)[2]) const {
    off[n] = (int32_t)t[1];
    caps[n] = row_sizes[n] = (int32_t)t[0];
    *top = t[0];
  }
  __device__ __forceinline__ void fault() const { off[n] = FLAT_BAD; }
};

// Where the entries come from / go to: CSR order, a row's start given by an
// array, or the row's segments in the pool.
enum { AT_FLAT = 0, AT_OFFS = 1, AT_POOL = 2 };

template <typename V>
struct FlatCopy {
  const int32_t *off, *tile_row;
  int32_t n;
  int64_t limit;  // entries at positions >= limit are not copied
  // source: AT_FLAT / AT_OFFS arrays (row starts in src_off), AT_POOL: seg, pitch, max_segs
  const int32_t *scols;
  const V *svals;
  const long long *src_off;
  const int32_t *seg;
  int32_t pitch, max_segs;
  // destination (AT_OFFS: row starts in dst_off), its capacity in entries
  int32_t *dcols;
  V *dvals;
  int32_t *drows;
  const int32_t *dst_off;
  int64_t dcap;
};

// A tile's first 32 rows, one per lane: offsets, destination distance,
// source start (a segment, or a staged row's).
struct FlatRows {
  int32_t r0, r1;  // rows that hold the tile's first entry and the next tile's
  int32_t o, o1, dd;
  int2 sg;
  long long so;
};

// Eight windows' loads in flight per lane; entry numbers, pool slots and
// destinations are below 2^31 (staged rows' sources are not: SD).  A tile's
// chain of loads (tile row -> row offsets and segments -> entries) is three
// round trips to HBM, so the warp works on three tiles at once: it copies
// tile t while the row data of its next tile and the tile rows of the one
// after are on their way.
template <typename V, int SRC, int DST, bool ROWS>
__global__ void __launch_bounds__(FT_THREADS) k_flat_copy(FlatCopy<V> a) {
  // distances from an entry's number to its source and to its destination
  using SD = typename std::conditional<SRC == AT_OFFS, long long, int32_t>::type;
  constexpr int NS = SRC == AT_FLAT ? 1 : FT_TILE, ND = DST == AT_FLAT ? 1 : FT_TILE, NR = ROWS ? FT_TILE : 1;
  __shared__ __align__(16) unsigned s_mask[FT_WARPS][FT_WIN];
  __shared__ SD s_sdel[FT_WARPS][NS];
  __shared__ int32_t s_ddel[FT_WARPS][ND];
  __shared__ int32_t s_row[FT_WARPS][NR];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned *mask = s_mask[w];
  SD *sdel = s_sdel[w];
  int32_t *ddel = s_ddel[w], *hrow = s_row[w];
  const int64_t nnz = a.off[a.n], total = nnz < a.limit ? nnz : a.limit;
  const int32_t nt = (int32_t)((total + FT_TILE - 1) / FT_TILE), last_row = a.n - 1;
  const int32_t nw = gridDim.x * FT_WARPS;
  const unsigned dcap = (unsigned)(a.dcap < 0xffffffffLL ? a.dcap : 0xffffffffLL);
  auto tile_rows = [&](int64_t t) -> int2 {
    if (t >= nt) return make_int2(0, -1);
    return make_int2(max(__ldg(a.tile_row + t), 0),
                     (t + 1) * FT_TILE < nnz ? min(__ldg(a.tile_row + t + 1), last_row) : last_row);
  };
  auto load_rows = [&](int2 tr) {
    FlatRows d;
    d.r0 = tr.x;
    d.r1 = tr.y;
    d.o = d.o1 = d.dd = 0;
    d.sg = make_int2(-1, -1);
    d.so = 0;
    const int32_t r = tr.x + lane;
    if (r <= tr.y) {
      d.o = __ldg(a.off + r);
      d.o1 = __ldg(a.off + r + 1);
      if constexpr (DST == AT_OFFS) d.dd = __ldg(a.dst_off + r);
      if constexpr (SRC == AT_POOL) d.sg = __ldg(reinterpret_cast<const int2 *>(a.seg + 2 * (int64_t)r));
      if constexpr (SRC == AT_OFFS) d.so = __ldg(a.src_off + r);
    }
    return d;
  };
  int64_t t = (int64_t)blockIdx.x * FT_WARPS + w;
  FlatRows cur = load_rows(tile_rows(t));
  int2 ntr = tile_rows(t + nw);
  for (; t < nt; t += nw) {
    const int32_t e0 = (int32_t)(t * FT_TILE);
    const int cnt = total - e0 < FT_TILE ? (int)(total - e0) : FT_TILE;
    const int32_t r0 = cur.r0, r1 = cur.r1;
    int32_t c[FT_WIN], row[ROWS ? FT_WIN : 1];
    V v[FT_WIN];
    unsigned dst[FT_WIN];
    if constexpr (SRC == AT_FLAT) {  // the entries do not depend on the rows
#pragma unroll
      for (int i = 0; i < FT_WIN; i++) {
        const int p = 32 * i + lane;
        if (p < cnt) {
          c[i] = __ldcs(a.scols + e0 + p);
          v[i] = __ldcs(a.svals + e0 + p);
        }
      }
    }
    const bool marked = r1 - r0 <= FT_ROWS;
    // a tile inside one row (and its first segment): one distance, no marks
    // (copies into the pool know their sources at once and gain nothing)
    bool inner = false;
    if constexpr (SRC == AT_POOL)
      inner = r0 == r1 && e0 + cnt - __shfl_sync(FULL, cur.o, 0) <=
                           __shfl_sync(FULL, cur.sg.y, 0) - __shfl_sync(FULL, cur.sg.x, 0) &&
              __shfl_sync(FULL, cur.sg.x, 0) >= 0;
    if (inner) {
      const int32_t o = __shfl_sync(FULL, cur.o, 0), dd = __shfl_sync(FULL, cur.dd, 0) - o;
      const int32_t sd = __shfl_sync(FULL, cur.sg.x, 0) - o;
#pragma unroll
      for (int i = 0; i < FT_WIN; i++) {
        const int p = 32 * i + lane;
        dst[i] = 0xffffffffu;
        if (p < cnt) {
          if constexpr (SRC == AT_POOL) {  // (only there)
            c[i] = __ldcs(a.scols + (e0 + p + sd));
            v[i] = __ldcs(a.svals + (e0 + p + sd));
          }
          dst[i] = (unsigned)(DST == AT_FLAT ? e0 + p : e0 + p + dd);
          if constexpr (ROWS) row[i] = r0;
        }
      }
    } else if (marked) {
      if (lane < FT_WIN) mask[lane] = 0;
      __syncwarp();
      auto mark_row = [&](int32_t r, const FlatRows &d) {
        const int32_t o = d.o, o1 = d.o1;
        if (o1 <= o || o - e0 >= cnt) return;
        const int32_t dd = d.dd - o;
        // marks the run of entries [pos, end) (relative to the tile; clipped to it)
        auto mark = [&](int pos, int end, SD sd) {
          if (end <= 0 || pos >= cnt || end <= pos) return;
          const int p = pos > 0 ? pos : 0;
          atomicOr(&mask[p >> 5], 1u << (p & 31));
          if constexpr (SRC != AT_FLAT) sdel[p] = sd;
          if constexpr (DST != AT_FLAT) ddel[p] = dd;
          if constexpr (ROWS) hrow[p] = r;
        };
        if constexpr (SRC == AT_POOL) {
          int32_t pos = o;
          int2 sg = d.sg;
          for (int l = 1; sg.x >= 0; l++) {
            const int32_t len = min(sg.y - sg.x, o1 - pos);
            mark(pos - e0, pos + len - e0, sg.x - pos);
            pos += len;
            if (pos >= o1 || l >= a.max_segs) break;
            sg = __ldg(reinterpret_cast<const int2 *>(a.seg + (int64_t)l * a.pitch + 2 * (int64_t)r));
          }
        } else {
          mark(o - e0, o1 - e0, (SD)(d.so - o));
        }
      };
      mark_row(r0 + lane, cur);
      for (int32_t rb = r0 + 32; rb <= r1; rb += 128) {  // past the first 32 rows: 128 at a time
        FlatRows d[4];
#pragma unroll
        for (int q = 0; q < 4; q++) d[q] = load_rows(make_int2(rb + 32 * q, r1));
#pragma unroll
        for (int q = 0; q < 4; q++) mark_row(rb + 32 * q + lane, d[q]);
      }
      __syncwarp();
      int h[FT_WIN];
      flat_heads(mask, h);
#pragma unroll
      for (int i = 0; i < FT_WIN; i++) {
        const int p = 32 * i + lane;
        dst[i] = 0xffffffffu;
        if (p < cnt) {
          const int32_t e = e0 + p;
          if constexpr (SRC != AT_FLAT) {
            const SD src = (SD)e + sdel[h[i]];
            c[i] = __ldcs(a.scols + src);
            v[i] = __ldcs(a.svals + src);
          }
          dst[i] = (unsigned)(DST == AT_FLAT ? e : e + ddel[DST == AT_FLAT ? 0 : h[i]]);
          if constexpr (ROWS) row[i] = hrow[h[i]];
        }
      }
    }
    // the next tile's rows and the tile rows of the one after
    cur = load_rows(ntr);
    ntr = tile_rows(t + 2 * (int64_t)nw);
    if (marked) {
#pragma unroll
      for (int i = 0; i < FT_WIN; i++) {
        if (dst[i] >= dcap) continue;
        a.dcols[dst[i]] = c[i];
        a.dvals[dst[i]] = v[i];
        if constexpr (ROWS) a.drows[dst[i]] = row[i];
      }
    } else {  // a long stretch of empty rows: each entry's row by a search
      int32_t rows[FT_WIN];
      flat_find_rows(a.off, e0, cnt, r0, r1, rows);
#pragma unroll
      for (int i = 0; i < FT_WIN; i++) {
        const int p = 32 * i + lane;
        if (p >= cnt) continue;
        const int32_t e = e0 + p, r = rows[i], o = a.off[r];
        int64_t src = e;
        if constexpr (SRC == AT_OFFS) src = a.src_off[r] + (e - o);
        if constexpr (SRC == AT_POOL) {
          int32_t q = e - o;
          for (int l = 0; l < a.max_segs; l++) {
            const int2 sg = __ldg(reinterpret_cast<const int2 *>(a.seg + (int64_t)l * a.pitch + 2 * (int64_t)r));
            if (sg.x < 0) break;
            src = sg.x + q;
            if (q < sg.y - sg.x) break;
            q -= sg.y - sg.x;
          }
        }
        const unsigned d = (unsigned)(DST == AT_OFFS ? a.dst_off[r] + (e - o) : e);
        if (d < dcap) {
          a.dcols[d] = a.scols[src];
          a.dvals[d] = a.svals[src];
          if constexpr (ROWS) a.drows[d] = r;
        }
      }
    }
    __syncwarp();  // the marks are cleared for the next tile
  }
}

template <typename V, int SRC, int DST, bool ROWS>
int launch_flat(const FlatCopy<V> &a, int64_t entries, cudaStream_t s) {
  static const int g = persistent_grid((const void *)k_flat_copy<V, SRC, DST, ROWS>, FT_THREADS, 0);
  const int64_t nt = flat_tiles(entries);
  if (nt < 1) return DCSR_OK;
  const int64_t nb = div_up(nt, FT_WARPS);
  DCSR_LAUNCH((k_flat_copy<V, SRC, DST, ROWS>), (unsigned)(nb < g ? nb : g), FT_THREADS, 0, s, a);
  return DCSR_OK;
}

// Layer 0 = [caps[r], caps[r+1]), other layers cleared, row lengths and the
// flat tables (offsets, tile rows) from the row pointer; pool top = caps[n].
__global__ void k_layout_rp(int32_t *seg, int32_t *row_sizes, int32_t n, int32_t pitch, int max_segs,
                            const int32_t *caps, const int32_t *rp, int32_t *off, int32_t *tile_row, int64_t tiles) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t r0 = (int64_t)blockIdx.x * blockDim.x; r0 <= n; r0 += stride) {
    const int64_t r = r0 + threadIdx.x;
    int32_t o = 0, len = 0;
    if (r < n) {
      *reinterpret_cast<int2 *>(seg + 2 * r) = make_int2(caps[r], caps[r + 1]);
      for (int l = 1; l < max_segs; l++)
        *reinterpret_cast<int2 *>(seg + (int64_t)l * pitch + 2 * r) = make_int2(-1, -1);
      o = rp[r];
      len = rp[r + 1] - o;
      row_sizes[r] = len;
      off[r] = o;
      if (r == n - 1) off[n] = o + len;
    } else if (r == n) {
      row_sizes[n] = caps[n];
      if (n == 0) off[0] = 0;
    }
    flat_mark_tiles((int32_t)r, o, len, tile_row, tiles);
  }
}

// Layer 0 = [caps[r], caps[r+1]), other layers cleared; pool top = caps[n].
__global__ void k_layout_caps(int32_t *seg, int32_t *row_sizes, int32_t n, int32_t pitch, int max_segs,
                              const int32_t *caps) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r <= n; r += stride) {
    if (r == n) {
      row_sizes[n] = caps[n];
      continue;
    }
    *reinterpret_cast<int2 *>(seg + 2 * r) = make_int2(caps[r], caps[r + 1]);
    for (int l = 1; l < max_segs; l++)
      *reinterpret_cast<int2 *>(seg + (int64_t)l * pitch + 2 * r) = make_int2(-1, -1);
  }
}

int grid_for(int64_t n, int block) {
  const int64_t g = div_up(n, block), cap = (int64_t)sm_count() * 16;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

template <typename V>
FlatCopy<V> flat_args(dcsr_handle h, const int32_t *off, const int32_t *tile_row) {
  FlatCopy<V> a;
  std::memset(&a, 0, sizeof(a));
  a.off = off;
  a.tile_row = tile_row;
  a.n = h->n_rows;
  a.limit = INT64_MAX;
  a.seg = h->seg;
  a.pitch = h->pitch;
  a.max_segs = h->o.max_segs;
  return a;
}

template <typename V>
int export_t(dcsr_handle h, const int32_t *off, const int32_t *tile_row, int32_t *cols, V *vals, int32_t *rows,
             int64_t limit, cudaStream_t s) {
  FlatCopy<V> a = flat_args<V>(h, off, tile_row);
  a.limit = limit;
  a.scols = h->cols;
  a.svals = (const V *)h->vals;
  a.dcols = cols;
  a.dvals = vals;
  a.drows = rows;
  a.dcap = INT64_MAX;
  if (rows) return launch_flat<V, AT_POOL, AT_FLAT, true>(a, h->pool_cap, s);
  return launch_flat<V, AT_POOL, AT_FLAT, false>(a, h->pool_cap, s);
}

template <typename V>
int compact_t(dcsr_handle h, const int32_t *off, const int32_t *tile_row, const int32_t *caps, int32_t *cols, V *vals,
              int64_t cap, cudaStream_t s) {
  FlatCopy<V> a = flat_args<V>(h, off, tile_row);
  a.scols = h->cols;
  a.svals = (const V *)h->vals;
  a.dcols = cols;
  a.dvals = vals;
  a.dst_off = caps;
  a.dcap = cap;
  return launch_flat<V, AT_POOL, AT_OFFS, false>(a, h->pool_cap, s);
}

template <typename V>
int load_t(dcsr_handle h, const int32_t *rp, const int32_t *tile_row, const int32_t *caps, const int32_t *cols,
           const V *vals, int64_t nnz, cudaStream_t s) {
  FlatCopy<V> a = flat_args<V>(h, rp, tile_row);
  a.scols = cols;
  a.svals = vals;
  a.dcols = h->cols;
  a.dvals = (V *)h->vals;
  a.dst_off = caps;
  a.dcap = h->buf_cap;
  return launch_flat<V, AT_FLAT, AT_OFFS, false>(a, nnz, s);
}

template <typename V>
int place_t(dcsr_handle h, const int32_t *off, const int32_t *tile_row, const int32_t *caps, const long long *src_off,
            const int32_t *scols, const V *svals, int64_t bound, cudaStream_t s) {
  FlatCopy<V> a = flat_args<V>(h, off, tile_row);
  a.scols = scols;
  a.svals = svals;
  a.src_off = src_off;
  a.dcols = h->cols;
  a.dvals = (V *)h->vals;
  a.dst_off = caps;
  a.dcap = h->buf_cap;
  return launch_flat<V, AT_OFFS, AT_OFFS, false>(a, bound, s);
}

}  // namespace

int caps_scan(dcsr_handle h, const int32_t *rp, int32_t *caps, Arena &ar, cudaStream_t s) {
  const CapsScan f{rp, h->n_rows, h->o, caps, h->stat + ST_TOTAL};
  return scan_map(f, h->n_rows > 0 ? h->n_rows : 1, ar, s);
}

int counts_scan(dcsr_handle h, const int32_t *cnt, int32_t *rp, int32_t *caps, Arena &ar, cudaStream_t s) {
  const CountScan f{cnt, h->n_rows, h->o, rp, caps, h->stat + ST_TOTAL};
  return scan_map(f, h->n_rows > 0 ? h->n_rows : 1, ar, s);
}

int place_csr(dcsr_handle h, const int32_t *rp, const int32_t *caps, const int32_t *cols, const void *vals,
              int64_t nnz, cudaStream_t s) {
  DCSR_LAUNCH(k_layout_rp, grid_for((int64_t)h->n_rows + 1, 256), 256, 0, s, h->seg, h->row_sizes, h->n_rows, h->pitch,
              h->o.max_segs, caps, rp, h->flat_off, h->flat_tile, h->flat_tiles);
  if (h->dtype == DCSR_F32) return load_t<float>(h, h->flat_off, h->flat_tile, caps, cols, (const float *)vals, nnz, s);
  return load_t<double>(h, h->flat_off, h->flat_tile, caps, cols, (const double *)vals, nnz, s);
}

int place_rows_scan(dcsr_handle h, const long long *lens, int32_t *caps, Arena &ar, cudaStream_t s) {
  const PlaceScan f{lens,   h->n_rows, h->o,          h->flat_off,   h->flat_tile,      caps, h->row_sizes,
                    h->seg, h->pitch,  h->o.max_segs, h->flat_tiles, h->stat + ST_TOTAL};
  return scan_map(f, h->n_rows > 0 ? h->n_rows : 1, ar, s);
}

int place_rows_copy(dcsr_handle h, const int32_t *caps, const long long *src_off, const int32_t *scols,
                    const void *svals, int64_t bound, cudaStream_t s) {
  if (h->dtype == DCSR_F32)
    return place_t<float>(h, h->flat_off, h->flat_tile, caps, src_off, scols, (const float *)svals, bound, s);
  return place_t<double>(h, h->flat_off, h->flat_tile, caps, src_off, scols, (const double *)svals, bound, s);
}

int compact_scan(dcsr_handle h, int32_t *off, int32_t *caps, int32_t *tile_row, Arena &ar, cudaStream_t s) {
  const CompactScan f{h->row_sizes, h->n_rows, h->o, off, tile_row, caps, flat_tiles(h->pool_cap), h->stat + ST_TOTAL};
  return scan_map(f, h->n_rows > 0 ? h->n_rows : 1, ar, s);
}

int compact_copy(dcsr_handle h, const int32_t *off, const int32_t *caps, const int32_t *tile_row, int32_t *cols,
                 void *vals, int64_t cap, cudaStream_t s) {
  const int st = h->dtype == DCSR_F32 ? compact_t<float>(h, off, tile_row, caps, cols, (float *)vals, cap, s)
                                      : compact_t<double>(h, off, tile_row, caps, cols, (double *)vals, cap, s);
  if (st != DCSR_OK) return st;
  DCSR_LAUNCH(k_layout_caps, grid_for((int64_t)h->n_rows + 1, 256), 256, 0, s, h->seg, h->row_sizes, h->n_rows, h->pitch,
              h->o.max_segs, caps);
  return DCSR_OK;
}

int flat_offsets(dcsr_handle h, int32_t *off, int32_t *tile_row, int64_t tiles, Arena &ar, cudaStream_t s) {
  const OffsetsScan f{h->row_sizes, h->n_rows, off, tile_row, tiles};
  return scan_map(f, h->n_rows > 0 ? h->n_rows : 1, ar, s);
}

int export_rows(dcsr_handle h, const int32_t *off, const int32_t *tile_row, int32_t *cols, void *vals, int32_t *rows,
                int64_t limit, cudaStream_t s) {
  if (h->dtype == DCSR_F32) return export_t<float>(h, off, tile_row, cols, (float *)vals, rows, limit, s);
  return export_t<double>(h, off, tile_row, cols, (double *)vals, rows, limit, s);
}

}  // namespace dcsr
