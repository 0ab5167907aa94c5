// internal.cuh -- cross-file internal API of the DCSR library.
#pragma once
#include <vector>

#include "common.cuh"

namespace dcsr {

// Entry-parallel copies between CSR order and a matrix's pool (flat.cu).
// Offsets of the layout policy's capacities of rows given by a row pointer
// (caps_scan) or by counts (counts_scan, which also makes the row pointer):
// caps[n+1]; their sum, the pool top the rows need, goes to the handle's
// ST_TOTAL word.
int caps_scan(dcsr_handle h, const int32_t *rp, int32_t *caps, Arena &ar, cudaStream_t s);
int counts_scan(dcsr_handle h, const int32_t *cnt, int32_t *rp, int32_t *caps, Arena &ar, cudaStream_t s);
// The CSR's rows become the matrix's content: layout (layer 0 from caps), flat
// tables (ensure_flat first) and entries into the handle's pool; nnz bounds
// the entries.
int place_csr(dcsr_handle h, const int32_t *rp, const int32_t *caps, const int32_t *cols, const void *vals,
              int64_t nnz, cudaStream_t s);
// Staged rows (row r: lens[r] entries from src_off[r]) likewise: the layout
// and tables with the capacities' offsets, then the entries; bound bounds
// their number.
int place_rows_scan(dcsr_handle h, const long long *lens, int32_t *caps, Arena &ar, cudaStream_t s);
int place_rows_copy(dcsr_handle h, const int32_t *caps, const long long *src_off, const int32_t *scols,
                    const void *svals, int64_t bound, cudaStream_t s);
// Compaction: the offsets of the current content and of its policy
// capacities (sum to ST_TOTAL), then the entries into the new pool (cap
// entries) and the new layout.  tile_row: flat_tiles(pool_cap) words.
int compact_scan(dcsr_handle h, int32_t *off, int32_t *caps, int32_t *tile_row, Arena &ar, cudaStream_t s);
int compact_copy(dcsr_handle h, const int32_t *off, const int32_t *caps, const int32_t *tile_row, int32_t *cols,
                 void *vals, int64_t cap, cudaStream_t s);
// Export: every row's entries in CSR order (off, tile_row: flat_offsets),
// optionally with their rows; entries at positions >= limit are not written.
int export_rows(dcsr_handle h, const int32_t *off, const int32_t *tile_row, int32_t *cols, void *vals, int32_t *rows,
                int64_t limit, cudaStream_t s);

// Rows staged elsewhere (row r: lens[r] entries at src_off[r]) become the
// matrix's content with policy capacities, in a pool allocated at cap_bound
// entries (an upper bound of the pool capacity the rows need; bound: of their
// entries); synchronises once at the end (pool top).  Uses the handle's
// scratch arena.
int load_from_rows(dcsr_handle h, const long long *src_off, const long long *lens, const int32_t *scols,
                   const void *svals, int64_t bound, int64_t cap_bound, cudaStream_t s);

// Sort + group a COO batch (any order) into CSR form in the arena:
// MERGE: sorted by (row, col), duplicates summed in input order;
// APPEND: stably sorted by row.  *rp and *caps (counts_scan) have n_rows+1
// entries.  Out-of-range input sets AUX_BAD_INDEX in the handle's ST_AUX word.
int coo_to_csr(dcsr_handle h, const int32_t *rows, const int32_t *cols, const void *vals, int64_t nnz, bool merge,
               Arena &ar, int32_t **rp, int32_t **caps, int32_t **ocols, void **ovals, cudaStream_t s);
size_t coo_to_csr_scratch(dcsr_handle h, int64_t nnz);

// Per-call operators that take a scratch arena (default: the handle's own);
// a server passes its slot's arena so resident matrices keep no scratch.
int update_async(dcsr_handle h, const int32_t *rows, const int32_t *cols, const void *vals, int64_t nnz,
                 cudaStream_t s, Arena *ar = nullptr);

// One matrix of a batched update (device-resident array element).
template <typename V>
struct BatchItem {
  Mat<V> m;
  const int32_t *rows, *cols;
  const V *vals;
  long long toff;  // first index of this matrix's triples in the batch
  long long T;     // its triple count
};
// Update `count` matrices at once (items_dev: device BatchItem<V>[count],
// toff prefix over T); pool: their pools' entries together; gstat: batch-global
// status words.
int update_many(const void *items_dev, int dtype, int count, int64_t T, int64_t pool, bool merge, int rb, int cb,
                long long *gstat, Arena &ar, cudaStream_t s);
size_t update_scratch_bytes(int64_t T, size_t vsize);
int compact(dcsr_handle h, cudaStream_t s);
int build_schedule(dcsr_handle h, cudaStream_t s, Arena *ar = nullptr);
int spmv_call(dcsr_handle h, const void *x, int32_t k, int64_t ldx, void *y, int64_t ldy, double alpha, double beta,
              cudaStream_t s, Arena *ar = nullptr);

// One matrix of a row pass (SpMV / reduction) over a set of matrices.
template <typename V>
struct RowItem {
  Mat<V> m;
  const int32_t *long_rows;
  const long long *long_off;
  const int2 *chunk_rl;   // per chunk: (row, long-row index)
  const int32_t *med_rows; // medium rows
  int32_t *info;  // [0] long rows, [1] chunks, [2] medium rows
  int32_t *long_cnt;
  double *part;
  const V *x;
  V *y;
  int64_t ldx, ldy;
  double alpha, beta;
  long long row0;             // first row of this matrix in the batch's row space
  // flat pass (k = 1, row reductions): CSR offsets, tile rows, tile partials, tiles the tables hold
  const int32_t *off, *tile_row;
  double *fpart;
  long long tiles;
  int32_t short_max, long_min; // row classes: short <= short_max < medium <= long_min < long
  const int32_t *skip;        // batch: nonzero -> this matrix's pass is skipped (may be null)
  int32_t k, vec;             // runtime-k passes: right-hand sides, x rows loadable as vectors
};
// Rebuild the schedules of `count` matrices at once (items: device
// RowItem<V>[count] in row-space order; R = total rows).  Needs
// schedule_scratch_bytes(R) free in the arena.
int schedule_many(const void *items_dev, int dtype, int count, int64_t R, Arena &ar, cudaStream_t s);
size_t schedule_scratch_bytes(int64_t R);
// y = A x for `count` matrices (items: device RowItem<V>[count]) of one k
// family: kf = 1 (flat pass), 2, 4 or 8, every item's k <= kf (each item's own
// k / vec are read by the kernel); pref: the group's unit prefixes, 3*(count+1)
// long longs on the device, computed by unit_prefix_many with the same split:
// warps per 32-row block of short rows (short_split; 0 for the flat pass).
int spmv_many(const void *items_dev, int dtype, int count, int k, const long long *pref, int split, cudaStream_t s);
// The kernel family of a k: 1 (flat pass), 2, 4 or 8; and whether x's rows can
// be read in vectors of 16 bytes (8 where a row is no multiple of 16): packed,
// aligned, k even.
inline int rhs_family(int32_t k) { return k == 1 ? 1 : k == 2 ? 2 : k <= 4 ? 4 : 8; }
bool rhs_vec(const void *x, int32_t k, int64_t ldx, size_t vsize);
// Warps per 32-row short-row block for an SpMV pass over `blocks` blocks with k RHS.
int short_split(int64_t blocks, int k);
// Flat tables of a handle (row offsets, tile rows, tile partials): sized for
// its pool (or for `entries`); built from its row lengths when they are not
// valid.
int ensure_flat(dcsr_handle h, cudaStream_t s, int64_t entries = 0);
int build_flat(dcsr_handle h, cudaStream_t s, Arena *ar = nullptr);
// Those tables ready for a call on s: built unless they are valid.
int ready_flat(dcsr_handle h, cudaStream_t s, Arena *ar = nullptr);
// Look-back words that a build of either kind of tables needs.
size_t table_slots(dcsr_handle h);
// Of `count` matrices at once (items: device RowItem<V>[count], row0 = their
// first rows in a common row space of R rows).  Needs flat_scratch_bytes(R)
// free in the arena.
int flat_many(const void *items_dev, int dtype, int count, int64_t R, Arena &ar, cudaStream_t s);
size_t flat_scratch_bytes(int64_t R);
// The offsets and tile rows of a matrix (flat.cu): off n_rows+1 words.
int flat_offsets(dcsr_handle h, int32_t *off, int32_t *tile_row, int64_t tiles, Arena &ar, cudaStream_t s);
// The unit prefixes of up to MAX_PREFIX_JOBS SpMV groups in one launch.
constexpr int MAX_PREFIX_JOBS = 8;
int unit_prefix_many(const void *const *items, const int *counts, long long *const *prefs, const int *splits, int n,
                     int dtype, cudaStream_t s);
template <typename V>
RowItem<V> row_item(dcsr_handle h, const void *x, void *y, int64_t ldx, int64_t ldy, double alpha, double beta);
// An operation of the handle reported `status`: after a timeout its tables may
// be those of the scan that gave up, and are built anew.
inline void note_status(dcsr_handle h, int status) {
  if (status != DCSR_TIMEOUT) return;
  h->flat.drop();
  h->bins.drop();
}
// Size the handle's chunk table and chunk partials (K results per chunk).
int ensure_part(dcsr_handle h, int K, cudaStream_t s);
// DCSR -> CSR writing at most `limit` entries (the row pointer is complete).
int export_csr(dcsr_handle h, int32_t *row_ptr, int32_t *cols, void *vals, int64_t limit, cudaStream_t s,
               Arena *ar = nullptr);
int reserve(dcsr_handle h, int64_t cap, cudaStream_t s);
// Pool capacity for a matrix whose pool top reached `need` and is nearly
// full: the policy's capacity for that top, and at least a quarter more than
// the current capacity (so the growth is never a no-op).
inline int64_t grow_target(dcsr_handle h, int64_t need) {
  const int64_t p = pool_capacity(h->o, need), q = h->pool_cap + h->pool_cap / 4;
  const int64_t t = p > q ? p : q;
  return t < 0x7fffffffLL ? t : 0x7fffffffLL;  // the pool's index range
}

// The device side of a batch (batch.cu): a plan over a set of
// dcsr_batch_items, their descriptor image, and the enqueue of the merged
// update + schedule rebuild + grouped SpMV.  Buffers grow, never shrink, so
// one core can serve many batches (the server re-plans one per slot).
struct BatchCore {
  struct Group {
    int k = 1;          // k family: 1, 2, 4 (k 3..4) or 8 (k 5..8)
    bool side = false;  // no update and a valid schedule: may run beside the update
    int split = 1;      // warps per 32-row short-row block (short_split of its rows)
    std::vector<int> idx;  // items of this group, in item order
    size_t off = 0;        // descriptor offset in the image
    size_t pref_off = 0;   // unit-prefix offset in pref
  };
  int count = 0, dtype = 0, mode = 0;
  int64_t R1 = 0;       // rows of the flat (k = 1) items whose tables the run rebuilds
  int split_force = 0;  // > 0: warps per short-row block of every k >= 2 group (else short_split)
  std::vector<dcsr_batch_item> items;
  int64_t T = 0, R = 0;
  int rb = 1, cb = 1;
  std::vector<Group> groups;
  std::vector<int> sched;   // items whose row classes the run rebuilds (k >= 2)
  std::vector<int> upd;     // items with update triples (the update pipeline's items)
  std::vector<int> upd_of;  // per item: its index in upd, or -1
  // image: BatchItem[upd] | RowItem[sched] (row space) | group RowItems
  size_t off_row = 0, img_bytes = 0, img_cap = 0;
  unsigned char *img_dev = nullptr;
  unsigned char *img_host = nullptr;  // pinned copy of the last upload
  cudaEvent_t up_ev = nullptr;        // recorded after the last upload from img_host
  std::vector<unsigned char> img_new;
  int cnt_cap = 0;
  int32_t *skip = nullptr;        // [upd] 1: the matrix's update was rejected this run
  long long *status_dev = nullptr;  // [2*upd] (status, pool top needed) per updated matrix
  size_t pref_cap = 0;
  long long *pref = nullptr;
  long long *gstat = nullptr;
  Arena ar;

  // Validate and plan `items` (one dtype and mode, each matrix once); grows
  // buffers with stream-ordered allocation on s.  all_schedules: every run
  // rebuilds every matrix's schedule (a captured graph must not depend on
  // host state); else only updated matrices and stale schedules.
  int plan(const dcsr_batch_item *items, int count, cudaStream_t s, bool all_schedules);
  // Size every matrix's schedule buffers for its pool (before an upload).
  int ensure_buffers(cudaStream_t s);
  // Size the image and per-item buffers for up to `items` items at once, so
  // later plans of that size allocate nothing (pinned host allocation and
  // release synchronise the device).
  int reserve_items(int items, int dtype, cudaStream_t s);
  // Rebuild the descriptor image from the handles and upload it if it changed.  sync=true waits for the
  // upload; otherwise the caller guarantees the previous upload of this core
  // has completed before the next call (the pinned image is reused).
  int upload(cudaStream_t s, bool sync, bool force = false);
  // Reserve the arena for this plan (before a capture: runs must not allocate).
  int reserve_scratch(cudaStream_t s);
  // Merged update, skip flags, schedule rebuild, grouped SpMV (capturable).
  // With a second stream s2 (and two events), the SpMVs of matrices without
  // an update and with a valid schedule run on s2 beside the update; s waits
  // for them before returning to the caller's stream order.
  int enqueue(cudaStream_t s, cudaStream_t s2 = nullptr, cudaEvent_t fork = nullptr, cudaEvent_t join = nullptr);
  // (status, needed pool top) of every updated matrix (item upd[j] -> words
  // 2j, 2j+1) into host memory (async); clears the device statuses.
  int status_async(long long *host, cudaStream_t s);
  void mark_scheduled();
  // The words status_async fetched have arrived: a timeout's tables are stale.
  void note_statuses(const long long *host);
  void release();
};

}  // namespace dcsr
