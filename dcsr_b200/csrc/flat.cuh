// flat.cuh -- passes over the stored entries in row order, in tiles of
// FT_TILE entries whatever the rows' lengths: a warp per tile, eight windows
// of 32 entries, no block-wide barrier.
//
// The entries of all rows laid end to end are numbered 0 .. nnz-1 (entry e of
// row r: off[r] <= e < off[r+1], off the CSR row pointer); tile_row[t] is the
// row that holds entry t*FT_TILE.  A tile finds the run (a row's part in one
// segment) of each of its entries without a search: the runs that start in
// it set a bit at their first entry, and an entry's run starts at the nearest
// set bit at or before it.  Empty rows and hub rows cost nothing extra; a tile
// that spans more than FT_ROWS rows (long stretches of empty ones) searches
// per entry instead, so no tile walks an unbounded number of rows.
//
// Measured on the R-MAT 2^20 graph (16.1M entries, FP32): CSR load copy 95 us,
// export copy 77-87 us (220 and 124 us with a warp or a lane group per row);
// a CTA per 2048 entries with marks in shared memory and a block-wide maximum
// scan ran 113 and 108 us (57 instructions per 32 entries, warps at barriers).
// On rows of about 145 entries (FP64) the export copy moves 5.9 TB/s.
#pragma once
#include "common.cuh"

namespace dcsr {

constexpr int FT_WIN = 8;            // windows of 32 entries per tile
constexpr int FT_TILE = 32 * FT_WIN;
constexpr int32_t FT_ROWS = 512;
constexpr int FT_THREADS = 256;
constexpr int FT_WARPS = FT_THREADS / 32;

// The entry count (off[n]) of tables whose scan gave up a look-back wait: no
// tile, so no pass reads a row's offsets or a tile's row from them.
constexpr int32_t FLAT_BAD = -1;
inline int64_t flat_tiles(int64_t entries) { return div_up(entries, FT_TILE); }

// The tiles that start within row r's entries [off, off+len) (called by whole
// warps; len 0: none).  A row over many tiles is written by its whole warp.
// Tiles past `tiles` are not written (offsets from a scan whose wait gave up
// are not to be trusted).
__device__ __forceinline__ void flat_mark_tiles(int32_t r, int64_t off, int64_t len, int32_t *tile_row, int64_t tiles) {
  // 32-bit tile numbers: offsets are below 2^31 (or not to be trusted)
  const unsigned lim = (unsigned)tiles, o = (unsigned)off, t0 = (o + (FT_TILE - 1)) / FT_TILE;
  unsigned t1 = len > 0 ? (o + (unsigned)len - 1) / FT_TILE + 1 : 0;
  t1 = t1 < lim ? t1 : lim;
  const bool many = t1 > t0 && t1 - t0 > 16;
  if (!many)
    for (unsigned t = t0; t < t1; t++) tile_row[t] = r;
  unsigned big = __ballot_sync(FULL, many);
  while (big) {
    const int src = __ffs(big) - 1;
    big &= big - 1;
    const unsigned a = __shfl_sync(FULL, t0, src), b = __shfl_sync(FULL, t1, src);
    const int32_t rr = __shfl_sync(FULL, r, src);
    for (unsigned t = a + lane_id(); t < b; t += 32) tile_row[t] = rr;
  }
}

// The first entry (0 .. FT_TILE-1) of the run that holds the lane's entry of
// each window, from the tile's start bits.
__device__ __forceinline__ void flat_heads(const unsigned *mask, int (&h)[FT_WIN]) {
  const unsigned le = (2u << lane_id()) - 1u;
  int carry = 0;
#pragma unroll
  for (int i = 0; i < FT_WIN; i++) {
    const unsigned m = mask[i], mine = m & le;
    h[i] = mine ? 32 * i + 31 - __clz(mine) : carry;
    carry = m ? 32 * i + 31 - __clz(m) : carry;
  }
}

// The rows of the lane's entries e0 + 32*i + lane (< e0 + cnt) among rows
// [lo, hi]: the last one whose offset is at most the entry's number, all
// windows' searches in step (independent loads).
__device__ __forceinline__ void flat_find_rows(const int32_t *off, int32_t e0, int cnt, int32_t lo, int32_t hi,
                                               int32_t (&row)[FT_WIN]) {
  int32_t len = hi - lo + 1;
#pragma unroll
  for (int i = 0; i < FT_WIN; i++) row[i] = lo;
  while (len > 1) {
    const int32_t half = len >> 1;
#pragma unroll
    for (int i = 0; i < FT_WIN; i++) {
      const int p = 32 * i + lane_id();
      if (p < cnt && __ldg(off + row[i] + half) <= e0 + p) row[i] += half;
    }
    len -= half;
  }
}

}  // namespace dcsr
