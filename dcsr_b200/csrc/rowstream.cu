// rowstream.cu -- passes over the rows of one DCSR matrix or a set of them:
// SpMV (1..8 RHS) and row reductions.
//
// One value per entry (SpMV with one right-hand side, row reductions): the
// flat pass, a warp per tile of 256 consecutive entries (k_flat_rows).
//
// SpMV with k >= 2: rows are split into three classes by the schedule (rebuilt
// lazily after any change of row lengths), whose units carry bounded work:
//   short  (<= short_max entries)  a warp takes 32 consecutive rows and splits
//          into groups of G lanes, G in {1..16} from the block's mean row
//          length; a group walks one row with several loads in flight per
//          lane and reduces over its lanes with log2(G) shuffles.
//   medium (<= long_min)          one warp per row, lanes strided, U loads in
//          flight per lane, one warp reduction per row.
//   long                          CHUNK-entry chunks, one CTA per chunk;
//          multi-chunk rows combine their partials in chunk order (the CTA
//          that finishes the last chunk sums them).
// A row's result depends only on the row and its matrix (its length picks its
// class, the block's lengths pick G, its position its tiles), never on which
// launch or batch it runs in.  Sums are FP64, products too (k = 1, FP32
// matrices of more than FLAT_EXACT_ROWS rows: products rounded to FP32);
// every rounding step is an explicit round-to-nearest intrinsic.
//
// Reference: spmv_dcsr_bin* include/spmv.inl:364-622 (seven bin kernels on
// seven streams, rows read with stale Prow_sizes), CompactIndices
// include/sparse_update.inl:916-1007, DCSRtoCSROffsets :1101-1116.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "flat.cuh"
#include "internal.cuh"
#include "lookback.cuh"

namespace dcsr {

constexpr int RS_THREADS_ = 256;
constexpr int RS_WARPS = RS_THREADS_ / 32;
// Long-row entries per chunk unit (a CTA's).  Small enough that a power-law
// matrix's hottest rows spread over many CTAs; multi-chunk rows combine their
// partials in chunk order.
#ifndef DCSR_CHUNK
#define DCSR_CHUNK 2048
#endif
constexpr int CHUNK = DCSR_CHUNK;
enum { P_BLOCKS = 0, P_CHUNKS = 1, P_MED = 2 };
// The flat pass's units (one value per entry): tiles; blocks of FT_THREADS
// tiles and rows for k_flat_fix.
enum { P_TILES = 0, P_TBLOCKS = 1, P_RBLOCKS = 2 };

// ------------------------------------------------------------- sources
// A row pass runs over one matrix (RowOne, descriptor passed by value) or a
// set of matrices laid end to end in one row space (RowMany, descriptors in
// device memory, per-class unit prefixes computed on the device).

// split: warps sharing one 32-row block of short rows in the k >= 2 pass
// (each takes every split-th group pass), so a small matrix's few blocks
// still fill the GPU; 1 for everything else.
template <typename V>
struct RowOne {
  RowItem<V> it;
  int split = 1;
  __device__ __forceinline__ const RowItem<V> &item(int) const { return it; }
  __device__ __forceinline__ int find_row(int64_t) const { return 0; }
  __device__ __forceinline__ int64_t units(int part) const {
    if (part == P_CHUNKS) return it.info[1];
    if (part == P_MED) return div_up(it.info[2], RS_WARPS);
    return div_up(div_up(it.m.n_rows, 32) * split, RS_WARPS);
  }
  __device__ __forceinline__ int locate(int, int64_t u, int64_t &lu) const {
    lu = u;
    return 0;
  }
};

// One matrix of a flat pass.
template <typename V>
struct FlatOne {
  RowItem<V> it;
  __device__ __forceinline__ const RowItem<V> &item(int) const { return it; }
  __device__ __forceinline__ int find_row(int64_t) const { return 0; }
  __device__ __forceinline__ int64_t units(int part) const {
    if (part == P_RBLOCKS) return div_up(it.m.n_rows, FT_THREADS);
    const int64_t tiles = div_up(it.off[it.m.n_rows], FT_TILE);
    return part == P_TILES ? tiles : div_up(tiles, FT_THREADS);
  }
  __device__ __forceinline__ int locate(int, int64_t u, int64_t &lu) const {
    lu = u;
    return 0;
  }
};

template <typename V>
struct RowMany {
  const RowItem<V> *its;
  int count;
  const long long *pref;  // [3][count+1] unit prefixes per class (short blocks counted split times)
  int split = 1;
  __device__ __forceinline__ const RowItem<V> &item(int i) const { return its[i]; }
  __device__ __forceinline__ int find_row(int64_t g) const {  // matrix holding global row g
    int lo = 0, hi = count;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (its[mid].row0 <= g) lo = mid;
      else hi = mid;
    }
    return lo;
  }
  __device__ __forceinline__ int next_row(int i, int64_t g) const {  // the same, i holding an earlier row
    while (i + 1 < count && its[i + 1].row0 <= g) i++;
    return i;
  }
  __device__ __forceinline__ int64_t units(int part) const { return pref[part * (count + 1) + count]; }
  __device__ __forceinline__ int locate(int part, int64_t u, int64_t &lu) const {
    const long long *p = pref + part * (count + 1);
    int lo = 0, hi = count;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (p[mid] <= u) lo = mid;
      else hi = mid;
    }
    lu = u - p[lo];
    return lo;
  }
};

// ---------------------------------------------------------------- schedule
// The long rows' indices and first chunks and the medium rows' slots, per
// matrix: one scan over the rows of all matrices (sums modulo 2^32: only
// differences within a matrix are used), which leaves the prefixes of the rows
// that need one, and a pass that lists them.  A batch's first row of a matrix
// may lie in any block, so the differences take the second pass.  (With flags
// and their scan in memory, four kernels: 58 us in a batch of 48 matrices of 1000 to
// 128000 rows, now 36.)

template <typename V, typename Src>
struct SchedScan {
  static constexpr int NS = 3, IT = SM_LIGHT;
  using T = int32_t;
  struct State {
    bool keep;  // long or medium, or the first or last row of its matrix
  };
  Src src;
  int64_t R;
  uint4 *tmp;  // [R + 1]: the last one nonzero when the scan gave up
  // (a search per row: with one a thread and its rows following, as below, the
  // kernel took 31 us instead of 24)
  __device__ __forceinline__ void load(int64_t g, bool ok, State &st, T (&v)[3]) const {
    v[0] = v[1] = v[2] = 0;
    st.keep = false;
    if (ok) {
      const RowItem<V> &it = src.item(src.find_row(g));
      const int64_t r = g - it.row0;
      const int32_t L = it.m.row_sizes[r];
      if (L > it.long_min) {
        v[0] = 1;
        v[1] = (int32_t)(((int64_t)L + CHUNK - 1) / CHUNK);
      } else if (L > it.short_max) {
        v[2] = 1;
      }
      st.keep = L > it.short_max || r == 0 || r == it.m.n_rows - 1;
    }
  }
  __device__ __forceinline__ void emit(int64_t g, bool, const State &st, const long long (&p)[3],
                                       const T (&)[3]) const {
    if (st.keep) tmp[g] = make_uint4((unsigned)p[0], (unsigned)p[1], (unsigned)p[2], 0);
  }
  __device__ __forceinline__ void total(const long long (&)[3]) const { tmp[R].x = 0; }
  __device__ __forceinline__ void fault() const { tmp[R].x = 1; }
};

// Lists of the long and medium rows; per matrix the class counts and the
// long-row offset sentinel (its last row's thread).  None of either when the
// scan gave up.
template <typename V, typename Src>
__global__ void k_sched_emit(Src src, int64_t R, const uint4 *tmp) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const bool bad = tmp[R].x != 0;
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < R; g += stride) {
    const RowItem<V> &it = src.item(src.find_row(g));
    const int64_t r = g - it.row0;
    const int32_t L = bad ? 0 : it.m.row_sizes[r];
    const bool last = r == it.m.n_rows - 1;
    if (L <= it.short_max && !last) continue;
    const uint4 at = bad ? make_uint4(0, 0, 0, 0) : tmp[g], a0 = bad ? at : tmp[it.row0];
    unsigned li = at.x - a0.x, c0 = at.y - a0.y, mi = at.z - a0.z;
    if (L > it.long_min) {
      const unsigned nc = (unsigned)(((int64_t)L + CHUNK - 1) / CHUNK);
      const_cast<int32_t *>(it.long_rows)[li] = (int32_t)r;
      const_cast<long long *>(it.long_off)[li] = c0;
      it.long_cnt[li] = 0;
      for (unsigned c = c0; c < c0 + nc; c++) const_cast<int2 *>(it.chunk_rl)[c] = make_int2((int32_t)r, (int32_t)li);
      li++;
      c0 += nc;
    } else if (L > it.short_max) {
      const_cast<int32_t *>(it.med_rows)[mi] = (int32_t)r;
      mi++;
    }
    if (last) {
      it.info[0] = (int32_t)li;
      it.info[1] = (int32_t)c0;
      it.info[2] = (int32_t)mi;
      const_cast<long long *>(it.long_off)[li] = c0;
    }
  }
}

static int64_t max_chunks(dcsr_handle h) { return h->pool_cap / CHUNK + h->pool_cap / h->long_min + 2; }

int ensure_part(dcsr_handle h, int K, cudaStream_t s) {
  if (max_chunks(h) > h->chunk_cap) {
    if (h->chunk_rl) DCSR_CUDA(dcsr::dev_free(h->chunk_rl, s));
    h->chunk_rl = nullptr;
    h->chunk_cap = 0;  // (should the allocation fail)
    DCSR_CUDA(dcsr::dev_alloc((void **)&h->chunk_rl, sizeof(int2) * max_chunks(h), s));
    h->chunk_cap = max_chunks(h);
    h->bins.drop();  // the chunk table is gone
  }
  const int64_t need = max_chunks(h) * K;
  if (need <= h->part_cap) return DCSR_OK;
  if (h->part) DCSR_CUDA(dcsr::dev_free(h->part, s));
  h->part = nullptr;
  h->part_cap = 0;
  DCSR_CUDA(dcsr::dev_alloc((void **)&h->part, sizeof(double) * need, s));
  h->part_cap = need;
  return DCSR_OK;
}

template <typename V>
RowItem<V> row_item(dcsr_handle h, const void *x, void *y, int64_t ldx, int64_t ldy, double alpha, double beta) {
  RowItem<V> it;
  std::memset(&it, 0, sizeof(it));  // padding too: batch descriptor images are compared bytewise
  it.m = h->view<V>();
  it.long_rows = h->long_rows;
  it.long_off = h->long_off;
  it.chunk_rl = h->chunk_rl;
  it.med_rows = h->med_rows;
  it.info = h->sched_info;
  it.long_cnt = h->long_cnt;
  it.part = h->part;
  it.x = (const V *)x;
  it.y = (V *)y;
  it.ldx = ldx;
  it.ldy = ldy;
  it.alpha = alpha;
  it.beta = beta;
  it.row0 = 0;
  it.off = h->flat_off;
  it.tile_row = h->flat_tile;
  it.fpart = h->flat_part;
  it.tiles = h->flat_tiles;
  it.short_max = h->short_max;
  it.long_min = h->long_min;
  it.skip = nullptr;
  it.k = 1;
  it.vec = 0;
  return it;
}
template RowItem<float> row_item<float>(dcsr_handle, const void *, void *, int64_t, int64_t, double, double);
template RowItem<double> row_item<double>(dcsr_handle, const void *, void *, int64_t, int64_t, double, double);

static int grid_for(int64_t n, int block) {
  int64_t g = div_up(n, block);
  int64_t cap = (int64_t)sm_count() * 16;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

size_t schedule_scratch_bytes(int64_t R) { return arena_bytes(R + 1, 16) + scan_scratch_bytes(R + 1); }

// Needs schedule_scratch_bytes(R) free in the arena (reserved by the caller).
template <typename V, typename Src>
static int schedule_src(const Src &src, int64_t R, Arena &ar, cudaStream_t s) {
  if (R <= 0) return DCSR_OK;
  uint4 *tmp = ar.take<uint4>(R + 1);
  if (ar.overflow) return DCSR_OOM;  // scratch sizing bug: no kernel sees a null pointer
  DCSR_TRY((scan_map(SchedScan<V, Src>{src, R, tmp}, R, ar, s)));
  DCSR_LAUNCH((k_sched_emit<V, Src>), grid_for(R, 256), 256, 0, s, src, R, tmp);
  return DCSR_OK;
}

int schedule_many(const void *items_dev, int dtype, int count, int64_t R, Arena &ar, cudaStream_t s) {
  if (count == 0) return DCSR_OK;
  if (dtype == DCSR_F32)
    return schedule_src<float>(RowMany<float>{(const RowItem<float> *)items_dev, count, nullptr}, R, ar, s);
  return schedule_src<double>(RowMany<double>{(const RowItem<double> *)items_dev, count, nullptr}, R, ar, s);
}

template <typename V>
static int build_schedule_t(dcsr_handle h, cudaStream_t s, Arena &ar) {
  const unsigned long long cap = capture_id(s);
  if (!cap) DCSR_TRY(ensure_flat(h, s));  // (so that a capture may build those tables too)
  DCSR_TRY(ensure_part(h, 1, s));
  DCSR_TRY(ar.reserve(schedule_scratch_bytes(h->n_rows), s));
  RowOne<V> src{row_item<V>(h, nullptr, nullptr, 0, 0, 0.0, 0.0)};
  DCSR_TRY(schedule_src<V>(src, h->n_rows, ar, s));
  h->bins.built(cap);
  return DCSR_OK;
}

int build_schedule(dcsr_handle h, cudaStream_t s, Arena *ar) {
  Arena &a = ar ? *ar : h->scratch;
  a.status = h->stat + ST_STATUS;
  if (h->dtype == DCSR_F32) return build_schedule_t<float>(h, s, a);
  return build_schedule_t<double>(h, s, a);
}

// Flat tables: offsets, tile rows and tile partials of a matrix (one scan of
// its row lengths), sized for its pool.
int ensure_flat(dcsr_handle h, cudaStream_t s, int64_t entries) {
  const int64_t need = flat_tiles(std::max(h->pool_cap, entries)) + 1;
  if (h->flat_off && need <= h->flat_tiles) return DCSR_OK;
  if (capture_id(s)) return DCSR_NOT_SUPPORTED;  // (memory allocated in a capture is the graph's)
  if (!h->flat_off) DCSR_CUDA(dcsr::dev_alloc((void **)&h->flat_off, sizeof(int32_t) * ((size_t)h->n_rows + 2), s));
  if (h->flat_tile) DCSR_CUDA(dcsr::dev_free(h->flat_tile, s));
  if (h->flat_part) DCSR_CUDA(dcsr::dev_free(h->flat_part, s));
  h->flat_tile = nullptr;
  h->flat_part = nullptr;
  h->flat_tiles = 0;
  h->flat.drop();
  const int64_t want = need + need / 4;
  DCSR_CUDA(dcsr::dev_alloc((void **)&h->flat_tile, sizeof(int32_t) * want, s));
  DCSR_CUDA(dcsr::dev_alloc((void **)&h->flat_part, sizeof(double) * 2 * want, s));
  h->flat_tiles = want;
  return DCSR_OK;
}

int build_flat(dcsr_handle h, cudaStream_t s, Arena *ar) {
  Arena &a = ar ? *ar : h->scratch;
  a.status = h->stat + ST_STATUS;
  DCSR_TRY(ensure_flat(h, s));
  DCSR_TRY(flat_offsets(h, h->flat_off, h->flat_tile, h->flat_tiles, a, s));
  h->flat.built(capture_id(s));
  return DCSR_OK;
}

size_t table_slots(dcsr_handle h) {
  if (h->n_rows <= SM_ONE) return 0;
  return (size_t)(LB_SCAN_WORDS * div_up(h->n_rows, SM_THREADS * (h->n_rows <= SM_FEW ? SM_THIN : SM_LIGHT)));
}

int ready_flat(dcsr_handle h, cudaStream_t s, Arena *ar) {
  const bool seen = h->flat.seen_capture();
  if (!h->flat.ready(seen ? capture_id(s) : 0)) return build_flat(h, s, ar);
  // A load leaves the tables built: the area that a build in a capture needs is
  // sized by the first call that finds them so.
  if (!ar && table_slots(h) > h->scratch.lb_slots && !capture_id(s)) {
    Lookback lb;
    DCSR_TRY(h->scratch.lookback(table_slots(h), s, &lb));
  }
  return DCSR_OK;
}

size_t flat_scratch_bytes(int64_t R) { return arena_bytes(R + 2, 4); }

template <typename V>
static int flat_many_t(const RowItem<V> *its, int count, int64_t R, Arena &ar, cudaStream_t s);

int flat_many(const void *items_dev, int dtype, int count, int64_t R, Arena &ar, cudaStream_t s) {
  if (count == 0 || R == 0) return DCSR_OK;
  if (dtype == DCSR_F32) return flat_many_t<float>((const RowItem<float> *)items_dev, count, R, ar, s);
  return flat_many_t<double>((const RowItem<double> *)items_dev, count, R, ar, s);
}

// Exclusive prefix over the matrices of each class's unit count (one block
// of 1024 threads, 1024 matrices per round).
template <typename V>
__device__ __forceinline__ void unit_prefix_block(const RowItem<V> *its, int count, long long *pref, int split) {
  __shared__ long long wsum[3][32];
  __shared__ long long carry[3];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x < 3) carry[threadIdx.x] = 0;
  __syncthreads();
  for (int b = 0; b < count; b += 1024) {
    const int i = b + threadIdx.x;
    long long u[3] = {0, 0, 0}, inc[3];
    if (i < count && split == 0) {  // a flat group
      const int64_t tiles = div_up(its[i].off[its[i].m.n_rows], FT_TILE);
      u[P_TILES] = tiles;
      u[P_TBLOCKS] = div_up(tiles, FT_THREADS);
      u[P_RBLOCKS] = div_up(its[i].m.n_rows, FT_THREADS);
    } else if (i < count) {
      u[P_BLOCKS] = div_up(div_up(its[i].m.n_rows, 32) * split, RS_WARPS);
      u[P_CHUNKS] = its[i].info[1];
      u[P_MED] = div_up(its[i].info[2], RS_WARPS);
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      inc[c] = warp_incl_scan(u[c]);
      if (lane == 31) wsum[c][w] = inc[c];
    }
    __syncthreads();
    if (w == 0) {
#pragma unroll
      for (int c = 0; c < 3; c++) wsum[c][lane] = warp_incl_scan(wsum[c][lane]);
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 3; c++)
      if (i < count) pref[c * (count + 1) + i] = carry[c] + (w ? wsum[c][w - 1] : 0) + inc[c] - u[c];
    __syncthreads();
    if (threadIdx.x < 3) carry[threadIdx.x] += wsum[threadIdx.x][31];
    __syncthreads();
  }
  if (threadIdx.x < 3) pref[threadIdx.x * (count + 1) + count] = carry[threadIdx.x];
}

// The SpMV groups' prefixes in one launch, one block per group.
template <typename V>
struct PrefixJobs {
  const RowItem<V> *its[MAX_PREFIX_JOBS];
  int count[MAX_PREFIX_JOBS];
  long long *pref[MAX_PREFIX_JOBS];
  int split[MAX_PREFIX_JOBS];
};

template <typename V>
__global__ void __launch_bounds__(1024) k_unit_prefix_many(PrefixJobs<V> jobs) {
  unit_prefix_block(jobs.its[blockIdx.x], jobs.count[blockIdx.x], jobs.pref[blockIdx.x], jobs.split[blockIdx.x]);
}

// ------------------------------------------------------------- helpers

struct RowBlock {
  int32_t row;  // row id within its matrix (or -1)
  int32_t len;  // logical length
  bool stream;  // streamed by the block (non-empty and short)
};

template <typename V>
__device__ __forceinline__ RowBlock load_block(const Mat<V> &m, int64_t r0, int lane, int32_t smax) {
  RowBlock b;
  const int64_t r = r0 + lane;
  b.row = r < m.n_rows ? (int32_t)r : -1;
  b.len = b.row >= 0 ? __ldg(m.row_sizes + r) : 0;
  b.stream = b.len > 0 && b.len <= smax;
  return b;
}

// Lanes per row for a block of 32 short rows: the largest power of two
// G <= mean length / 4 (1..16), so a lane has about four or more entries of
// its row in flight and a block takes G passes of 32/G rows.
__device__ __forceinline__ int group_width(int32_t total) {
  const int32_t mean = total >> 5;
  return mean < 8 ? 1 : mean < 16 ? 2 : mean < 32 ? 4 : mean < 64 ? 8 : 16;
}

enum { OP_SPMV = 0, OP_SUM = 1, OP_MAX = 2, OP_MIN = 3, OP_COUNT = 4 };

template <typename T, int OP>
__device__ __forceinline__ T op_init() {
  return OP == OP_MAX ? (T)-INFINITY : OP == OP_MIN ? (T)INFINITY : (T)0;
}
// Every rounding step is an explicit round-to-nearest intrinsic: the
// compiler may not contract a product into a later sum (it could choose
// differently in different instantiations, and the batched and per-call
// passes must agree bit for bit).
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// Maxima and minima take a where it beats b, so a NaN in b stays and one in a
// is passed over.  A row's result is NaN when its first entry is, and else the
// extreme of its entries that are numbers: a row starts from its first entry,
// later ones are a, earlier results b.
constexpr bool op_extreme(int op) { return op == OP_MAX || op == OP_MIN; }
template <typename T, int OP>
__device__ __forceinline__ T op_comb(T a, T b) {
  if (OP == OP_MAX) return a > b ? a : b;
  if (OP == OP_MIN) return a < b ? a : b;
  return add_rn(a, b);
}

// y[row*ldy + k] = alpha*v + beta*y (SpMV), or v.
template <typename V, int OP>
__device__ __forceinline__ void write_y(V *y, double v, double alpha, double beta) {
  if (OP == OP_SPMV) {
    v = mul_rn(v, alpha);
    if (beta != 0.0) v = __fma_rn(beta, (double)*y, v);
  }
  *y = (V)v;
}

// ------------------------------------------------------- k >= 2 right-hand sides
// A lane takes an entry with all of its K right-hand sides (K accumulators; a
// packed, aligned row of x in 16-byte loads): what counts is how many rows of
// x a warp has in flight.  Sharing an entry among lanes (2 of 4 values each
// for k = 8) touched half the cache lines per gather but left fewer rows in
// flight: 131 against 101 us for 8M entries with k = 8 (FP32), 59 against 36 us
// for 2M with k = 3 (FP64).  Kernels are compiled per family (k = 2, 3..4,
// 5..8; one launch serves matrices of different k) and branch to the code of a
// matrix's own K -- a runtime k in the inner loop ran the batched passes at
// half the speed.
template <typename V, int K, bool VEC>
__device__ __forceinline__ void load_x(const V *__restrict__ p, V (&v)[K]) {
  if constexpr (VEC && K * sizeof(V) % 16 == 0) {
#pragma unroll
    for (int q = 0; q < K; q += 16 / (int)sizeof(V)) {
      if constexpr (sizeof(V) == 4) {
        const float4 t = __ldg(reinterpret_cast<const float4 *>(p + q));
        v[q] = t.x; v[q + 1] = t.y; v[q + 2] = t.z; v[q + 3] = t.w;
      } else {
        const double2 t = __ldg(reinterpret_cast<const double2 *>(p + q));
        v[q] = t.x; v[q + 1] = t.y;
      }
    }
  } else if constexpr (VEC) {  // FP32, K = 2 or 6
#pragma unroll
    for (int q = 0; q < K; q += 2) {
      const float2 t = __ldg(reinterpret_cast<const float2 *>(p + q));
      v[q] = t.x; v[q + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int q = 0; q < K; q++) v[q] = __ldg(p + q);
  }
}

// acc += a*x over logical entries [c0, c1) of a row, lane j of G: entries j,
// j+G, ... of each segment, UN of them in flight.
template <typename V, int K, bool VEC, int UN = (K <= 2 ? 8 : 4)>
__device__ __forceinline__ void accum_row(const Mat<V> &m, const V *__restrict__ x, int64_t ldx, const Chain &ch,
                                          int32_t c0, int32_t c1, int j, int G, double (&acc)[K]) {
  int32_t before = 0;
#pragma unroll
  for (int l = 0; l < MAX_SEGS; l++) {
    if (l < ch.ns && before < c1) {
      const int32_t from = c0 > before ? c0 - before : 0, take = ch.cp[l] < c1 - before ? ch.cp[l] : c1 - before;
      const int64_t st = ch.st[l];
      for (int32_t p = from + j; p < take; p += UN * G) {
        V a[UN];
        int32_t col[UN];
#pragma unroll
        for (int i = 0; i < UN; i++) {
          const int32_t pp = p + i * G;
          const int64_t q = st + (pp < take ? pp : p);
          a[i] = __ldcs(m.vals + q);
          col[i] = __ldcs(m.cols + q);
        }
#pragma unroll
        for (int i = 0; i < UN; i++)
          if (p + i * G < take) {
            V xv[K];
            load_x<V, K, VEC>(x + (int64_t)col[i] * ldx, xv);
#pragma unroll
            for (int q = 0; q < K; q++) acc[q] = __fma_rn((double)a[i], (double)xv[q], acc[q]);
          }
      }
      before += ch.cp[l];
    }
  }
}

template <typename V, int K>
__device__ __forceinline__ void write_rhs(const RowItem<V> &it, int32_t row, const double (&acc)[K]) {
#pragma unroll
  for (int q = 0; q < K; q++)
    write_y<V, OP_SPMV>(it.y + (int64_t)row * it.ldy + q, acc[q], it.alpha, it.beta);
}

// One unit of a class (lu within matrix it).
template <typename V, int K, bool VEC, int PART>
__device__ __forceinline__ void rows_unit(const RowItem<V> &it, int64_t lu, int split, double (*red)[8],
                                          int *last_flag) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const Mat<V> &m = it.m;
  const V *__restrict__ x = it.x;
  double acc[K];
#pragma unroll
  for (int q = 0; q < K; q++) acc[q] = 0.0;
  auto reduce = [&](int G) {  // over the lanes of a group
    for (int o = G >> 1; o > 0; o >>= 1) {
#pragma unroll
      for (int q = 0; q < K; q++) acc[q] = add_rn(acc[q], __shfl_xor_sync(FULL, acc[q], o));
    }
  };
  if constexpr (PART == P_CHUNKS) {
    // ---- one chunk of a long row, whole CTA
    const int2 rl = it.chunk_rl[lu];
    const int32_t row = rl.x, len = m.row_sizes[row];
    const int64_t li = rl.y;
    const int32_t nch = (len + CHUNK - 1) / CHUNK, chunk = nch == 1 ? 0 : (int32_t)(lu - it.long_off[li]);
    const Chain ch = load_chain(m, row);
    const int32_t c0 = chunk * CHUNK, c1 = len - c0 > CHUNK ? c0 + CHUNK : len;
    // FP64: four entries in flight as well for K = 2 (rows of 600 entries: 74 us of
    // 6M, 90 with eight, of which a thread has two or three; of 5000: 79 and 85)
    accum_row<V, K, VEC, K <= 2 && sizeof(V) == 4 ? 8 : 4>(m, x, it.ldx, ch, c0, c1, threadIdx.x, RS_THREADS_, acc);
    reduce(32);
    if (lane == 0)
#pragma unroll
      for (int q = 0; q < K; q++) red[w][q] = acc[q];
    __syncthreads();
    if (threadIdx.x < K) {  // a thread per right-hand side: warps in order
      double t = red[0][threadIdx.x];
      for (int q = 1; q < RS_WARPS; q++) t = add_rn(t, red[q][threadIdx.x]);
      if (nch == 1) {
        write_y<V, OP_SPMV>(it.y + (int64_t)row * it.ldy + threadIdx.x, t, it.alpha, it.beta);
      } else {
        it.part[(it.long_off[li] + chunk) * K + threadIdx.x] = t;
        __threadfence();
      }
    }
    if (nch > 1) {
      __syncthreads();
      if (threadIdx.x == 0) *last_flag = atomicAdd(&it.long_cnt[li], 1) == nch - 1;
      __syncthreads();
      if (*last_flag && threadIdx.x < K) {  // every chunk's sums are there: in chunk order
        __threadfence();
        double t = 0.0;
        for (int32_t q = 0; q < nch; q++) t = add_rn(t, __ldcg(it.part + (it.long_off[li] + q) * K + threadIdx.x));
        write_y<V, OP_SPMV>(it.y + (int64_t)row * it.ldy + threadIdx.x, t, it.alpha, it.beta);
        if (threadIdx.x == 0) it.long_cnt[li] = 0;
      }
    }
    __syncthreads();
  } else if constexpr (PART == P_MED) {
    // ---- one medium row per warp
    const int64_t mi = lu * RS_WARPS + w;
    if (mi >= it.info[2]) return;
    const int32_t row = it.med_rows[mi], len = m.row_sizes[row];
    const Chain ch = load_chain_used(m, row, len);
    accum_row<V, K, VEC>(m, x, it.ldx, ch, 0, len, lane, 32, acc);
    reduce(32);
    if (lane == 0) write_rhs<V, K>(it, row, acc);
  } else {
    // ---- short rows: a warp takes 32 consecutive rows, G lanes per row
    const int64_t wu = lu * RS_WARPS + w;
    const int64_t blk = wu / split;
    const int sub = (int)(wu - blk * split);
    if (blk * 32 >= m.n_rows) return;
    const RowBlock rb = load_block(m, blk * 32, lane, it.short_max);
    const Chain own = load_chain_used(m, rb.row >= 0 ? rb.row : 0, rb.stream ? rb.len : 0);
    const int G = group_width(warp_sum(rb.stream ? rb.len : 0));
    const int per = 32 / G, j = lane & (G - 1), g = lane / G;
    for (int pass = sub; pass < G; pass += split) {
      const int owner = pass * per + g;
      const int32_t row = __shfl_sync(FULL, rb.row, owner);
      const int32_t len = __shfl_sync(FULL, rb.len, owner);
      const Chain ch = shfl_chain(own, owner);
#pragma unroll
      for (int q = 0; q < K; q++) acc[q] = 0.0;
      if (row >= 0 && len > 0 && len <= it.short_max) accum_row<V, K, VEC>(m, x, it.ldx, ch, 0, len, j, G, acc);
      reduce(G);
      if (j == 0 && row >= 0 && len <= it.short_max) write_rhs<V, K>(it, row, acc);
    }
  }
}

// Blocks per SM: three (80 registers) measured fastest for every family; the
// compiler's own choice (94-158 registers) left two or one: 121 us for 8M
// entries with k = 8 against 101, four blocks 106.
#ifndef DCSR_RHS_MINB
#define DCSR_RHS_MINB 3
#endif
template <typename V, int FAM, int PART>
__device__ __forceinline__ void rows_unit_k(const RowItem<V> &it, int64_t lu, int split, double (*red)[8],
                                            int *last_flag) {
  if (it.skip && *it.skip) return;  // a batch matrix whose update was rejected: y untouched
  if (FAM == 8 && it.vec && it.k == 6) {
    rows_unit<V, FAM == 8 ? 6 : FAM, true, PART>(it, lu, split, red, last_flag);
  } else if (it.vec) {  // k = 2, 4 or 8
    rows_unit<V, FAM, true, PART>(it, lu, split, red, last_flag);
  } else if constexpr (FAM == 2) {
    rows_unit<V, 2, false, PART>(it, lu, split, red, last_flag);
  } else if constexpr (FAM == 4) {
    if (it.k == 3) rows_unit<V, 3, false, PART>(it, lu, split, red, last_flag);
    else rows_unit<V, 4, false, PART>(it, lu, split, red, last_flag);
  } else {
    if (it.k == 5) rows_unit<V, 5, false, PART>(it, lu, split, red, last_flag);
    else if (it.k == 6) rows_unit<V, 6, false, PART>(it, lu, split, red, last_flag);
    else if (it.k == 7) rows_unit<V, 7, false, PART>(it, lu, split, red, last_flag);
    else rows_unit<V, 8, false, PART>(it, lu, split, red, last_flag);
  }
}

// All classes in one launch, the long rows' chunks first: a class of few units
// (the batched matrices have hundreds of medium rows) no longer has the GPU
// to itself for its tail.
template <typename V, int FAM, typename Src>
__global__ void __launch_bounds__(RS_THREADS_, DCSR_RHS_MINB) k_rows_rhs(Src src) {
  __shared__ double red[RS_WARPS][8];
  __shared__ int last_flag;
  const int64_t nc = src.units(P_CHUNKS), nm = src.units(P_MED), total = nc + nm + src.units(P_BLOCKS);
  for (int64_t u = blockIdx.x; u < total; u += gridDim.x) {
    int64_t lu;
    if (u < nc) {
      const RowItem<V> &it = src.item(src.locate(P_CHUNKS, u, lu));
      rows_unit_k<V, FAM, P_CHUNKS>(it, lu, src.split, red, &last_flag);
    } else if (u < nc + nm) {
      const RowItem<V> &it = src.item(src.locate(P_MED, u - nc, lu));
      rows_unit_k<V, FAM, P_MED>(it, lu, src.split, red, &last_flag);
    } else {
      const RowItem<V> &it = src.item(src.locate(P_BLOCKS, u - nc - nm, lu));
      rows_unit_k<V, FAM, P_BLOCKS>(it, lu, src.split, red, &last_flag);
    }
  }
}

// --------------------------------------------- one value per entry: flat pass
// SpMV with one right-hand side and the row reductions: a warp per tile of 256
// consecutive entries (flat.cuh), whatever the rows' lengths.  The entries are
// loaded striped (coalesced along each row), x gathered, the products put in
// tile order through shared memory so that each lane holds eight consecutive
// entries; a lane sums its pieces of rows left to right in FP64, a segmented
// scan over the lanes carries the open piece on, and every row that lies in
// the tile is written.  A row over several tiles leaves its sums in part[2t]
// (the part of a row that began in an earlier tile) and part[2t+1] (the part
// of one that goes on in the next); k_flat_fix adds them in tile order and
// writes the empty rows.  A row's result depends on the row and on its
// position among the matrix's entries, never on the launch or batch it runs in.
//
// Bound by the x gathers (random reads of x, a sector each) and the per-entry
// instructions; the row classes it replaces (32-row blocks with a segmented
// scan per window of 32 entries, streamed long and medium rows taken from a
// counter) left it to latency: the R-MAT 2^20 stream matrix (17.8M entries,
// FP32) took 118 + 63 us.

// A tile of a flat pass: its matrix, its entries, and the row data of its
// first 32 rows, one per lane (loaded ahead).
struct FlatTile {
  int32_t item, lt;  // matrix; tile within it
  int32_t r0, r1;    // rows that hold its first entry and the next tile's
  int32_t cnt;       // entries (0: past the end, or a skipped matrix)
  int32_t nnz;       // of the matrix
  int32_t o, o1;     // the lane's row: offsets
  int2 sg;           // and first segment
};

template <typename V, typename Src>
__device__ __forceinline__ void flat_tile_head(const Src &src, int64_t t, int64_t total, FlatTile &x) {
  x.item = 0;
  x.lt = 0;
  x.cnt = 0;
  x.r0 = 0;
  x.r1 = -1;
  x.nnz = 0;
  if (t >= total) return;
  int64_t lt;
  x.item = src.locate(P_TILES, t, lt);
  const RowItem<V> &it = src.item(x.item);
  if (it.skip && *it.skip) return;
  x.lt = (int32_t)lt;
  x.nnz = __ldg(it.off + it.m.n_rows);
  const int64_t e0 = lt * FT_TILE, left = x.nnz - e0;
  if (left <= 0) return;
  x.cnt = left < FT_TILE ? (int32_t)left : FT_TILE;
  x.r0 = max(__ldg(it.tile_row + lt), 0);
  x.r1 = left > FT_TILE ? min(__ldg(it.tile_row + lt + 1), it.m.n_rows - 1) : it.m.n_rows - 1;
}

template <typename V, typename Src>
__device__ __forceinline__ void flat_tile_rows(const Src &src, FlatTile &x) {
  const int32_t r = x.r0 + lane_id();
  x.o = x.o1 = 0;
  x.sg = make_int2(-1, -1);
  if (r <= x.r1) {
    const RowItem<V> &it = src.item(x.item);
    x.o = __ldg(it.off + r);
    x.o1 = __ldg(it.off + r + 1);
    x.sg = __ldg(reinterpret_cast<const int2 *>(it.m.seg + 2 * (int64_t)r));
  }
}

template <typename V, int OP>
__device__ __forceinline__ void write_row(const RowItem<V> &it, int32_t row, double v) {
  write_y<V, OP>(it.y + (int64_t)row * it.ldy, v, it.alpha, it.beta);
}

// FP32 matrices of at most this many rows multiply in FP64 (every product
// exact, and within range whatever the factors), larger ones in FP32; both sum
// in FP64.  FP64 products cost two conversions an entry: 132 against 99 us on
// the R-MAT matrix of 2^20 rows, whose error against 64 bits is 3.7e-8 with
// FP32 products (2.6e-8 with exact ones, most of it the result's own rounding).
// The line is the one the library always had between its small and its large
// matrices, so that results keep their precision and range on either side.
constexpr int32_t FLAT_EXACT_ROWS = 32768;

#ifndef DCSR_FLAT_MINB
#define DCSR_FLAT_MINB 4
#endif
// EXACT: an FP32 SpMV's products are kept in FP64 (FP64 products of a set's
// matrices of up to FLAT_EXACT_ROWS rows, FP32 ones of the larger).
template <typename V, int OP, typename Src, bool XU, bool EXACT>
__global__ void __launch_bounds__(FT_THREADS, DCSR_FLAT_MINB) k_flat_rows(Src src) {
  __shared__ __align__(16) unsigned s_run[FT_WARPS][FT_WIN], s_row[FT_WARPS][FT_WIN];
  // Products in tile order; before them, in an SpMV, the distances from an
  // entry's number to its slot, by run; and the rows by their first entries.
  // Shared memory is kept small: what it takes, the x gathers' L1 loses (33 KB
  // a block ran 118 us on the R-MAT matrix where 25 KB ran 102, 17 KB 99).
  constexpr bool OWN = OP != OP_SPMV, WIDE = EXACT && OP == OP_SPMV && sizeof(V) == 4;
  using P = typename std::conditional<WIDE, double, V>::type;
  __shared__ __align__(16) P s_prod[FT_WARPS][FT_TILE];
  __shared__ int32_t s_sdel[OWN ? FT_WARPS : 1][OWN ? FT_TILE : 1];  // (the reductions': room of their own)
  __shared__ int32_t s_hrow[FT_WARPS][FT_TILE];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned *runs = s_run[w], *starts = s_row[w];
  int32_t *hrow = s_hrow[w], *sdel = OWN ? s_sdel[OWN ? w : 0] : reinterpret_cast<int32_t *>(s_prod[w]);
  P *prod = s_prod[w];
  const int64_t total = src.units(P_TILES), nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + w;
  FlatTile cur, nx;
  flat_tile_head<V>(src, t, total, cur);
  flat_tile_rows<V>(src, cur);
  flat_tile_head<V>(src, t + nw, total, nx);
  for (; t < total; t += nw) {
    const RowItem<V> &it = src.item(cur.item);
    const int32_t e0 = cur.lt * FT_TILE, cnt = cur.cnt, r0 = cur.r0, r1 = cur.r1;
    // a tile inside one row's first segment: no marks, one sum (half of the
    // tiles of a power-law matrix)
    const int32_t o0 = __shfl_sync(FULL, cur.o, 0), o01 = __shfl_sync(FULL, cur.o1, 0);
    const int32_t sx = __shfl_sync(FULL, cur.sg.x, 0), sy = __shfl_sync(FULL, cur.sg.y, 0);
    const bool inner = cnt > 0 && r0 == r1 && sx >= 0 && e0 + cnt - o0 <= sy - sx;
    const bool cont = o0 < e0;  // its first row began in an earlier tile
    const bool exact = WIDE && it.m.n_rows <= FLAT_EXACT_ROWS;  // (a set's larger matrices: as on their own)
    auto product = [&](V a, V x) -> P {
      if constexpr (WIDE)
        if (exact) return mul_rn((double)a, (double)x);
      return (P)mul_rn(a, x);
    };
    double isum = op_init<double, OP>(), lead = 0.0;
    if (inner) {
      const int32_t base = sx + (e0 - o0) + lane;
      V a[FT_WIN];
      int32_t col[FT_WIN];
#pragma unroll
      for (int i = 0; i < FT_WIN; i++) {
        a[i] = V(0);
        col[i] = 0;
        if (32 * i + lane < cnt) {
          a[i] = __ldcs(it.m.vals + base + 32 * i);
          col[i] = OP == OP_SPMV ? __ldcs(it.m.cols + base + 32 * i) : 0;
        }
      }
      if constexpr (OP == OP_SPMV) {
        const V *__restrict__ x = it.x;
        V xv[FT_WIN];
#pragma unroll
        for (int i = 0; i < FT_WIN; i++)
          xv[i] = 32 * i + lane < cnt ? (XU ? __ldg(x + col[i]) : __ldg(x + (int64_t)col[i] * it.ldx)) : V(0);
#pragma unroll
        for (int i = 0; i < FT_WIN; i++)
          if (32 * i + lane < cnt) isum = __dadd_rn((double)product(a[i], xv[i]), isum);
      } else {
        lead = (double)a[0];
#pragma unroll
        for (int i = 0; i < FT_WIN; i++)
          if (32 * i + lane < cnt) isum = op_comb<double, OP>(OP == OP_COUNT ? 1.0 : (double)a[i], isum);
      }
    } else if (cnt > 0) {
      // ---- runs and row starts
      if (lane < FT_WIN) runs[lane] = starts[lane] = 0;
      __syncwarp();
      auto mark_row = [&](int32_t r, int32_t o, int32_t o1, int2 sg) {
        if (o1 <= o || o - e0 >= cnt) return;
        hrow[o > e0 ? o - e0 : 0] = r;
        if (o > e0) atomicOr(&starts[(o - e0) >> 5], 1u << ((o - e0) & 31));  // (position 0 needs no bit)
        int32_t pos = o;
        for (int l = 1; sg.x >= 0; l++) {
          const int32_t len = min(sg.y - sg.x, o1 - pos);
          const int a = pos - e0, b = a + len;
          if (b > 0 && a < cnt && len > 0) {
            const int p = a > 0 ? a : 0;
            atomicOr(&runs[p >> 5], 1u << (p & 31));
            sdel[p] = sg.x - pos;
          }
          pos += len;
          if (pos >= o1 || l >= it.m.max_segs) break;
          sg = __ldg(reinterpret_cast<const int2 *>(it.m.seg + (int64_t)l * it.m.pitch + 2 * (int64_t)r));
        }
      };
      if (r1 - r0 <= FT_ROWS) {
        mark_row(r0 + lane, cur.o, cur.o1, cur.sg);
        for (int32_t rb = r0 + 32; rb <= r1; rb += 128) {  // past the first 32 rows: 128 at a time
          int32_t o[4], o1[4];
          int2 sg[4];
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const int32_t r = rb + 32 * q + lane;
            o[q] = o1[q] = 0;
            sg[q] = make_int2(-1, -1);
            if (r <= r1) {
              o[q] = __ldg(it.off + r);
              o1[q] = __ldg(it.off + r + 1);
              sg[q] = __ldg(reinterpret_cast<const int2 *>(it.m.seg + 2 * (int64_t)r));
            }
          }
#pragma unroll
          for (int q = 0; q < 4; q++) mark_row(rb + 32 * q + lane, o[q], o1[q], sg[q]);
        }
      } else {  // a long stretch of empty rows: each entry's row by a search, marked by its first entry here
        int32_t rows[FT_WIN];
        flat_find_rows(it.off, e0, cnt, r0, r1, rows);
#pragma unroll
        for (int i = 0; i < FT_WIN; i++) {
          const int p = 32 * i + lane;
          if (p >= cnt) continue;
          const int32_t r = rows[i], o = it.off[r];
          if (p == 0 || e0 + p == o)
            mark_row(r, o, it.off[r + 1], *reinterpret_cast<const int2 *>(it.m.seg + 2 * (int64_t)r));
        }
      }
      __syncwarp();
      // ---- entries
      int h[FT_WIN];
      flat_heads(runs, h);
      V a[FT_WIN];
      int32_t col[FT_WIN];
#pragma unroll
      for (int i = 0; i < FT_WIN; i++) {
        const int p = 32 * i + lane;
        a[i] = V(0);
        col[i] = 0;
        if (p < cnt) {
          const int32_t q = e0 + p + sdel[h[i]];
          a[i] = __ldcs(it.m.vals + q);
          col[i] = OP == OP_SPMV ? __ldcs(it.m.cols + q) : 0;
        }
      }
      if constexpr (!OWN) __syncwarp();  // the distances are read: the products take their place
      if constexpr (OP == OP_SPMV) {
        const V *__restrict__ x = it.x;
        V xv[FT_WIN];
#pragma unroll
        for (int i = 0; i < FT_WIN; i++)
          xv[i] = 32 * i + lane < cnt ? (XU ? __ldg(x + col[i]) : __ldg(x + (int64_t)col[i] * it.ldx)) : V(0);
#pragma unroll
        for (int i = 0; i < FT_WIN; i++) prod[32 * i + lane] = 32 * i + lane < cnt ? product(a[i], xv[i]) : P(0);
      } else {
#pragma unroll
        for (int i = 0; i < FT_WIN; i++)
          prod[32 * i + lane] = 32 * i + lane >= cnt ? op_init<V, OP>() : OP == OP_COUNT ? V(1) : a[i];
      }
    }
    // the next tile's rows and the tile after it, on their way meanwhile
    FlatTile next = nx;
    flat_tile_rows<V>(src, next);
    flat_tile_head<V>(src, t + 2 * nw, total, nx);
    if (inner) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) isum = op_comb<double, OP>(isum, __shfl_xor_sync(FULL, isum, o));
      if (lane == 0) {
        double *part = it.fpart + 2 * (int64_t)cur.lt;
        if (op_extreme(OP) && !cont) isum = op_comb<double, OP>(isum, lead);  // (the row's first entry)
        if (cont) part[0] = isum;
        else if (o01 > e0 + cnt) part[1] = isum;
        else write_row<V, OP>(it, r0, isum);
      }
    } else if (cnt > 0) {
      __syncwarp();
      // ---- sums: lane l holds entries 8l .. 8l+7
      P pv[FT_WIN];
#pragma unroll
      for (int q = 0; q < FT_WIN; q += 16 / (int)sizeof(P)) {
        if constexpr (sizeof(P) == 4) {
          const float4 f = *reinterpret_cast<const float4 *>(prod + 8 * lane + q);
          pv[q] = f.x; pv[q + 1] = f.y; pv[q + 2] = f.z; pv[q + 3] = f.w;
        } else {
          const double2 f = *reinterpret_cast<const double2 *>(prod + 8 * lane + q);
          pv[q] = f.x; pv[q + 1] = f.y;
        }
      }
      const unsigned bits = (starts[lane >> 2] >> (8 * (lane & 3))) & 0xffu;
      double acc = op_init<double, OP>(), first = acc;
      if (op_extreme(OP) && lane == 0 && !cont) acc = (double)pv[0];  // (position 0 has no start bit)
      int at = -1;  // last row start in this lane
#pragma unroll
      for (int q = 0; q < 8; q++) {
        if ((bits >> q) & 1) {
          if (at < 0) first = acc;  // closes a row that began in an earlier lane (or the tile's first)
          else write_row<V, OP>(it, hrow[at], acc);
          at = 8 * lane + q;
          acc = op_extreme(OP) ? (double)pv[q] : op_init<double, OP>();
        }
        acc = op_comb<double, OP>((double)pv[q], acc);
      }
      // open pieces carried over the lanes; the last start before each lane
      double open = acc;
      bool seen = at >= 0;
      int last = at < 0 ? 0 : at;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const double ov = __shfl_up_sync(FULL, open, d);
        const int os = __shfl_up_sync(FULL, (int)seen, d), ol = __shfl_up_sync(FULL, last, d);
        if (lane >= d) {
          if (!seen) open = op_comb<double, OP>(open, ov);  // ov: the earlier lanes'
          seen = seen || os;
          last = max(last, ol);
        }
      }
      double carry = __shfl_up_sync(FULL, open, 1);
      int before = __shfl_up_sync(FULL, last, 1);
      if (lane == 0) {
        carry = op_extreme(OP) ? first : op_init<double, OP>();  // nothing came before
        before = 0;
      }
      double *part = it.fpart + 2 * (int64_t)cur.lt;
      if (at >= 0) {  // the row open before this lane ends here
        const double v = op_comb<double, OP>(first, carry);
        if (before == 0 && cont) part[0] = v;
        else write_row<V, OP>(it, hrow[before], v);
      }
      if (lane == 31) {  // the row open at the tile's end
        const int32_t r = hrow[last];
        if (last == 0 && cont) part[0] = open;
        else if (it.off[r + 1] > e0 + cnt) part[1] = open;
        else write_row<V, OP>(it, r, open);
      }
      __syncwarp();  // the tile's marks and products are free
    }
    cur = next;
  }
}

// Rows over several tiles (a thread per tile in which one begins, a warp for
// more than 16 tiles, the block for more than 512: a row of 2M entries has 7800,
// 60 us a load at a time by one warp, 7 to 10 by the block) and empty rows (a thread
// per row).  The row's length alone gives the order of the additions.
constexpr int FIX_WARP = 16, FIX_BLOCK = 512;
template <typename V, int OP, typename Src>
__global__ void __launch_bounds__(FT_THREADS) k_flat_fix(Src src) {
  __shared__ double s_sum[FT_WARPS];
  __shared__ int64_t s_tile;
  __shared__ int s_n;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t nt = src.units(P_TBLOCKS), total = nt + src.units(P_RBLOCKS);
  for (int64_t u = blockIdx.x; u < total; u += gridDim.x) {
    int64_t lu;
    const bool tiles = u < nt;
    const RowItem<V> &it = src.item(tiles ? src.locate(P_TBLOCKS, u, lu) : src.locate(P_RBLOCKS, u - nt, lu));
    if (it.skip && *it.skip) continue;
    const int64_t i = lu * FT_THREADS + threadIdx.x;
    if (!tiles) {
      if (i < it.m.n_rows && it.off[i] == it.off[i + 1]) write_row<V, OP>(it, (int32_t)i, 0.0);  // (max, min: 0 too)
      continue;
    }
    const int64_t nnz = it.off[it.m.n_rows], e1 = (i + 1) * FT_TILE;
    int32_t r = -1, nh = 0;  // the row that begins in tile i and goes on, and in how many more tiles
    if (e1 < nnz) {
      r = it.tile_row[i + 1];
      const int32_t o = it.off[r];
      if (o >= e1 - FT_TILE && o < e1) nh = (int32_t)((it.off[r + 1] - 1) / FT_TILE - i);
      else r = -1;
    }
    double v = 0.0;
    if (r >= 0) {
      v = it.fpart[2 * i + 1];
      if (nh <= FIX_WARP)
        for (int32_t q = 1; q <= nh; q++) v = op_comb<double, OP>(it.fpart[2 * (i + q)], v);
    }
    // the heads a .. b of the row that begins in tile t: lanes take every 32nd
    // in order, then a fixed tree
    auto heads = [&](int64_t t, int32_t a, int32_t b) {
      double p = op_init<double, OP>();
#pragma unroll 4
      for (int32_t q = a + lane; q <= b; q += 32) p = op_comb<double, OP>(it.fpart[2 * (t + q)], p);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) p = op_comb<double, OP>(p, __shfl_xor_sync(FULL, p, o));
      return p;
    };
    unsigned big = __ballot_sync(FULL, nh > FIX_WARP && nh <= FIX_BLOCK);
    while (big) {
      const int s = __ffs(big) - 1;
      big &= big - 1;
      const double p = heads(__shfl_sync(FULL, i, s), 1, __shfl_sync(FULL, nh, s));
      if (lane == s) v = op_comb<double, OP>(p, v);
    }
    // (of FT_THREADS tiles, one at most begins such a row)
    static_assert(FIX_BLOCK >= FT_THREADS, "one row per unit");
    if (__syncthreads_or(nh > FIX_BLOCK)) {
      if (nh > FIX_BLOCK) {
        s_tile = i;
        s_n = nh;
      }
      __syncthreads();
      const int32_t per = (s_n + FT_WARPS - 1) / FT_WARPS, to = (w + 1) * per;
      const double p = heads(s_tile, 1 + w * per, to < s_n ? to : s_n);
      if (lane == 0) s_sum[w] = p;
      __syncthreads();
      if (nh > FIX_BLOCK)
        for (int q = 0; q < FT_WARPS; q++) v = op_comb<double, OP>(s_sum[q], v);
      __syncthreads();  // (the shared words are free)
    }
    if (r >= 0) write_row<V, OP>(it, r, v);
  }
}

// Row lengths -> offsets within a set of matrices' concatenated rows (mod
// 2^32: only differences within one matrix are used).
template <typename V, typename Src>
struct FlatManyScan {
  static constexpr int NS = 1, IT = SM_LIGHT;
  using T = int32_t;
  struct State {};
  Src src;
  int64_t R;
  unsigned *tmp;
  static constexpr bool LOAD_ALL = true;
  __device__ __forceinline__ void load_all(int64_t base, int64_t n, State (&)[IT], T (&v)[IT][1]) const {
    int i = base < n ? src.find_row(base) : 0;  // one search a thread; its other rows follow
#pragma unroll
    for (int j = 0; j < IT; j++) {
      const int64_t g = base + 32 * j;
      v[j][0] = 0;
      if (g < n) {
        i = src.next_row(i, g);
        const RowItem<V> &it = src.item(i);
        v[j][0] = it.m.row_sizes[g - it.row0];
      }
    }
  }
  __device__ __forceinline__ void emit(int64_t g, bool ok, const State &, const long long (&p)[1], const T (&)[1]) const {
    if (ok) tmp[g] = (unsigned)p[0];
  }
  __device__ __forceinline__ void total(const long long (&t)[1]) const {
    tmp[R] = (unsigned)t[0];
    tmp[R + 1] = 0;
  }
  __device__ __forceinline__ void fault() const { tmp[R + 1] = 1; }
};

// (tmp[R + 1]: the scan gave up, every matrix's tables are bad)
template <typename V, typename Src>
__global__ void __launch_bounds__(256) k_flat_tables(Src src, int64_t R, const unsigned *tmp) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const bool bad = tmp[R + 1] != 0;
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x; b < R; b += stride) {
    const int64_t g = b + threadIdx.x;
    int32_t r = 0, o = 0, len = 0;
    int i = 0;
    if (g < R) {
      i = src.find_row(g);
      const RowItem<V> &it = src.item(i);
      r = (int32_t)(g - it.row0);
      if (!bad) {
        o = (int32_t)(tmp[g] - tmp[it.row0]);
        len = (int32_t)(tmp[g + 1] - tmp[g]);
      }
      const_cast<int32_t *>(it.off)[r] = o;
      if (r == it.m.n_rows - 1) const_cast<int32_t *>(it.off)[r + 1] = bad ? FLAT_BAD : o + len;
    }
    // (a warp may hold rows of several matrices: tiles are marked per row)
    const RowItem<V> &it = src.item(i);
    const unsigned t0 = ((unsigned)o + (FT_TILE - 1)) / FT_TILE;
    const unsigned t1 = len > 0 ? min(((unsigned)o + (unsigned)len - 1) / FT_TILE + 1, (unsigned)it.tiles) : 0;
    const bool many = t1 > t0 && t1 - t0 > 16;
    if (!many)
      for (unsigned t = t0; t < t1; t++) const_cast<int32_t *>(it.tile_row)[t] = r;
    unsigned big = __ballot_sync(FULL, many);
    while (big) {
      const int s = __ffs(big) - 1;
      big &= big - 1;
      const unsigned a = __shfl_sync(FULL, t0, s), z = __shfl_sync(FULL, t1, s);
      const int32_t rr = __shfl_sync(FULL, r, s);
      int32_t *tr = const_cast<int32_t *>(src.item(__shfl_sync(FULL, i, s)).tile_row);
      for (unsigned t = a + lane_id(); t < z; t += 32) tr[t] = rr;
    }
  }
}

template <typename V>
static int flat_many_t(const RowItem<V> *its, int count, int64_t R, Arena &ar, cudaStream_t s) {
  const RowMany<V> src{its, count, nullptr};
  unsigned *tmp = ar.take<unsigned>(R + 2);
  if (ar.overflow) return DCSR_OOM;  // scratch sizing bug: no kernel sees a null pointer
  DCSR_TRY((scan_map(FlatManyScan<V, RowMany<V>>{src, R, tmp}, R, ar, s)));
  DCSR_LAUNCH((k_flat_tables<V, RowMany<V>>), grid_for(R, 256), 256, 0, s, src, R, tmp);
  return DCSR_OK;
}

static int grid_of(const void *k) { return persistent_grid(k, RS_THREADS_, 0); }

template <typename V, int FAM, typename Src>
static int launch_rhs(const Src &src, cudaStream_t s) {
  static const int g = grid_of((const void *)k_rows_rhs<V, FAM, Src>);
  DCSR_LAUNCH((k_rows_rhs<V, FAM, Src>), g, RS_THREADS_, 0, s, src);
  return DCSR_OK;
}

// The flat pass over `tiles` tiles and `rows` rows at most (-1: not known on
// the host).  Few tiles: two warps per block, so that they spread over the SMs.
template <typename V, int OP, bool XU, bool EXACT, typename Src>
static int launch_flat_src(const Src &src, int64_t tiles, int64_t rows, cudaStream_t s) {
  static const int g = grid_of((const void *)k_flat_rows<V, OP, Src, XU, EXACT>);
  static const int gf = grid_of((const void *)k_flat_fix<V, OP, Src>);
  const int64_t cap = (int64_t)g * FT_WARPS;  // resident warps
  int threads = FT_THREADS;
  int64_t blocks = g, fix = gf;
  if (tiles >= 0) {
    if (tiles < cap / 4) threads = 64;
    blocks = std::max<int64_t>(1, std::min<int64_t>(div_up(tiles, threads / 32), threads == 64 ? cap / 2 : g));
    fix = std::max<int64_t>(1, std::min<int64_t>(div_up(tiles, FT_THREADS) + div_up(rows, FT_THREADS), gf));
  }
  DCSR_LAUNCH((k_flat_rows<V, OP, Src, XU, EXACT>), (unsigned)blocks, threads, 0, s, src);
  DCSR_LAUNCH((k_flat_fix<V, OP, Src>), (unsigned)fix, FT_THREADS, 0, s, src);
  return DCSR_OK;
}

template <typename V, int OP>
static int launch_flat(dcsr_handle h, const V *x, int64_t ldx, V *y, int64_t ldy, double alpha, double beta,
                       cudaStream_t s) {
  const FlatOne<V> src{row_item<V>(h, x, y, ldx, ldy, alpha, beta)};
  const int64_t tiles = flat_tiles(h->pool_cap);
  constexpr bool F32 = OP == OP_SPMV && sizeof(V) == 4;
  if (OP == OP_SPMV && ldx == 1) {
    if (F32 && h->n_rows <= FLAT_EXACT_ROWS) return launch_flat_src<V, OP, OP == OP_SPMV, F32>(src, tiles, h->n_rows, s);
    return launch_flat_src<V, OP, OP == OP_SPMV, false>(src, tiles, h->n_rows, s);
  }
  if (F32 && h->n_rows <= FLAT_EXACT_ROWS) return launch_flat_src<V, OP, false, F32>(src, tiles, h->n_rows, s);
  return launch_flat_src<V, OP, false, false>(src, tiles, h->n_rows, s);
}

// Warps per 32-row block of short rows for the k >= 2 pass: doubled (up to
// 8) while the blocks times the split stay under 12 warps per SM, so a
// matrix of a few thousand rows is not left to a few dozen warps, each
// walking 32 rows' groups one after another.
int short_split(int64_t blocks, int k) {
  if (k == 1) return 1;
  int S = 1;
  while (S < 8 && blocks * S * 2 <= (int64_t)sm_count() * 12) S *= 2;
  return S;
}

bool rhs_vec(const void *x, int32_t k, int64_t ldx, size_t vsize) {
  const size_t al = (size_t)k * vsize % 16 == 0 ? 16 : 8;  // a lane's load
  return k % 2 == 0 && ldx == k && (uintptr_t)x % al == 0;
}

template <typename V>
static int spmv_dispatch(dcsr_handle h, const V *x, int32_t k, int64_t ldx, V *y, int64_t ldy, double alpha,
                         double beta, cudaStream_t s) {
  if (k == 1) return launch_flat<V, OP_SPMV>(h, x, ldx, y, ldy, alpha, beta, s);
  RowOne<V> src{row_item<V>(h, x, y, ldx, ldy, alpha, beta)};
  src.it.k = k;
  src.it.vec = rhs_vec(x, k, ldx, sizeof(V)) ? 1 : 0;
  src.split = short_split(div_up(h->n_rows, 32), k);
  switch (rhs_family(k)) {
    case 2: return launch_rhs<V, 2>(src, s);
    case 4: return launch_rhs<V, 4>(src, s);
    case 8: return launch_rhs<V, 8>(src, s);
  }
  return DCSR_BAD_ARG;
}

template <typename V>
static int reduce_dispatch(dcsr_handle h, int32_t op, V *y, cudaStream_t s) {
  switch (op) {
    case DCSR_REDUCE_SUM: return launch_flat<V, OP_SUM>(h, nullptr, 0, y, 1, 1.0, 0.0, s);
    case DCSR_REDUCE_MAX: return launch_flat<V, OP_MAX>(h, nullptr, 0, y, 1, 1.0, 0.0, s);
    case DCSR_REDUCE_MIN: return launch_flat<V, OP_MIN>(h, nullptr, 0, y, 1, 1.0, 0.0, s);
    case DCSR_REDUCE_COUNT: return launch_flat<V, OP_COUNT>(h, nullptr, 0, y, 1, 1.0, 0.0, s);
  }
  return DCSR_BAD_ARG;
}

// Batched SpMV over a set of matrices of one k family: kf = 1 (flat pass), 2,
// 4 or 8 (each item's k <= kf, read by the kernel).
template <typename V>
static int spmv_many_t(const RowItem<V> *its, int count, int kf, const long long *pref, int split, cudaStream_t s) {
  RowMany<V> src{its, count, pref, split};
  switch (kf) {
    case 1: return launch_flat_src<V, OP_SPMV, false, sizeof(V) == 4>(src, -1, -1, s);
    case 2: return launch_rhs<V, 2>(src, s);
    case 4: return launch_rhs<V, 4>(src, s);
    case 8: return launch_rhs<V, 8>(src, s);
  }
  return DCSR_BAD_ARG;
}

int spmv_many(const void *items_dev, int dtype, int count, int k, const long long *pref, int split, cudaStream_t s) {
  if (count == 0) return DCSR_OK;
  if (dtype == DCSR_F32)
    return spmv_many_t<float>((const RowItem<float> *)items_dev, count, k, pref, split, s);
  return spmv_many_t<double>((const RowItem<double> *)items_dev, count, k, pref, split, s);
}

template <typename V>
static int unit_prefix_many_t(const void *const *items, const int *counts, long long *const *prefs,
                              const int *splits, int n, cudaStream_t s) {
  PrefixJobs<V> jobs;
  std::memset(&jobs, 0, sizeof(jobs));
  for (int i = 0; i < n; i++) {
    jobs.its[i] = (const RowItem<V> *)items[i];
    jobs.count[i] = counts[i];
    jobs.pref[i] = prefs[i];
    jobs.split[i] = splits[i];
  }
  DCSR_LAUNCH(k_unit_prefix_many<V>, n, 1024, 0, s, jobs);
  return DCSR_OK;
}

int unit_prefix_many(const void *const *items, const int *counts, long long *const *prefs, const int *splits, int n,
                     int dtype, cudaStream_t s) {
  if (n < 1) return DCSR_OK;
  if (n > MAX_PREFIX_JOBS) return DCSR_BAD_ARG;
  if (dtype == DCSR_F32) return unit_prefix_many_t<float>(items, counts, prefs, splits, n, s);
  return unit_prefix_many_t<double>(items, counts, prefs, splits, n, s);
}

}  // namespace dcsr

using namespace dcsr;

namespace dcsr {
int spmv_call(dcsr_handle h, const void *x, int32_t k, int64_t ldx, void *y, int64_t ldy, double alpha, double beta,
              cudaStream_t s, Arena *ar) {
  if (h->n_rows == 0) return DCSR_OK;
  if (k == 1) {
    DCSR_TRY(ready_flat(h, s, ar));
  } else {
    DCSR_TRY(ensure_part(h, rhs_family(k), s));
    if (!h->bins.ready(h->bins.seen_capture() ? capture_id(s) : 0)) DCSR_TRY(build_schedule(h, s, ar));
  }
  if (h->dtype == DCSR_F32)
    return spmv_dispatch<float>(h, (const float *)x, k, ldx, (float *)y, ldy, alpha, beta, s);
  return spmv_dispatch<double>(h, (const double *)x, k, ldx, (double *)y, ldy, alpha, beta, s);
}
}  // namespace dcsr

extern "C" int dcsr_spmv(dcsr_handle h, const void *x, int32_t k, int64_t ldx, void *y, int64_t ldy, double alpha,
                         double beta, void *stream) {
  if (!h || k < 1 || k > 8 || ldx < k || ldy < k || (h->n_rows > 0 && !y) || (h->n_cols > 0 && !x))
    return DCSR_BAD_ARG;
  return spmv_call(h, x, k, ldx, y, ldy, alpha, beta, (cudaStream_t)stream);
}

extern "C" int dcsr_row_reduce(dcsr_handle h, int32_t op, void *y, void *stream) {
  if (!h || (h->n_rows > 0 && !y) || op < 0 || op > 3) return DCSR_BAD_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (h->n_rows == 0) return DCSR_OK;
  DCSR_TRY(ready_flat(h, s));
  if (h->dtype == DCSR_F32) return reduce_dispatch<float>(h, op, (float *)y, s);
  return reduce_dispatch<double>(h, op, (double *)y, s);
}
