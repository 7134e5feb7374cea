// Stages O/E/S: per-row top-k lists -> key-block-major CSC pattern, without atomics on
// global memory and without a sort pass.
//
// The reference counts with global atomics, scans with one thread, scatters with global
// atomics (unordered) and then runs a segmented sort
// (csrc/flash_topk/src/flash_topk_kernel.h:303-312, 376-402, 407-478;
//  csrc/flash_topk/src/varlen_sort.cu:29-124).  Here:
//   1. tile_hist : a CTA takes kTileRows query rows of one (b,h) and counts its entries per column
//                  in shared memory -> hist[bh][tile][col]
//   2. tile_scan : per (b,h) and group of columns: running sum over tiles per column (hist becomes the
//                  tile's write cursor), col_nnz.  Left out for sequences of few tiles, whose scatter
//                  CTAs sum the tiles before their own themselves
//   3. scatter   : the column offsets (a scan over col_nnz, repeated by every CTA: a few hundred numbers);
//                  a bitmap (column x row) of the tile in shared memory with a running count per 32 rows, from
//                  which every entry's place in its column follows directly: columns come out ascending,
//                  bit-exact and run-to-run deterministic.  Lists of up to 16 are put in order column by column in shared
//                  memory first, so that a warp's stores fill whole sectors of a few columns instead of 4 bytes in each of 32.
//                  On request the same thread also writes the row's places in `indices`, in ascending
//                  order (row_slots): the row-major view of the pattern that the attention kernels' merge
//                  needs, so that an attention call on this pattern builds no lists of its own.
// Measured (B200, three kernels with bitmap walks before / now): 64K tokens x 32 heads, 512 columns 297 / 192 us; 32K x 16
// 71 / 45; 317K tokens, lists of 16 2.19 / 1.63 ms; 512K x 4 heads, 2,048 columns 1.49 / 0.84 ms.  The scatter with its counts per 32
// rows laid out column by column (stores of a warp eight to a bank) and 64-bit scans / row group by row group and 32-bit scans:
// 64K 143 / 129 us, 317K 1.32 / 1.23 ms, 512K 0.80 / 0.71 ms.  Entries stored by the row's thread, lists read behind the scan, a
// bitonic network per row / in column order, read ahead of it, networks of 19 exchanges, all three kernels: 64K 159 / 146 us,
// 32K x 16 39.5 / 37.3, d 64, 9K x 12 13.8 / 12.5, 8 x 8K 128 / 130, 317K 1460 / 1231, 512K 642 / 607.  (Three CTAs per SM with 40 registers: 64K 1 % more, 8 x 8K 8 % less, but 9K x 12 20 % more.  A histogram that trusts the lists to be distinct would
// save 3 %; a chunk that is named twice counts once instead.)
// What bounds it: the scatter's instructions (1,070 a warp of 32 rows, 57 % issue) and its shared-memory accesses at random columns
// (two thirds to four fifths of the wavefronts); HBM 8 - 25 %.  Algorithmic bytes: 4*nnz read + 4*nnz written + 12*B*H*ncol.
#include <mutex>
#include <type_traits>

#include "fmb_common.cuh"

namespace fmb {

constexpr int kTileRows = 512;                 // query rows per tile
constexpr int kTileWords = kTileRows / 32;     // bitmap words per column
constexpr int kBmStride = kTileWords + 1;      // padded: conflict-free column walks
constexpr int kMaxHistCols = 8192;             // columns per CTA of the histogram (32 KB of counters)
constexpr int kMaxColsPerCta = 1024;           // columns per CTA of the scatter
constexpr int kColBytes = kBmStride * 4 + kTileWords * 2 + 8;   // shared memory of the scatter per column
constexpr int kCscThreads = 512;
// Up to this many columns the row's thread stores the entries: a warp's 32 rows then put eight (lists of eight) or more into a column's
// sectors at once, and putting them in order costs more than it saves.  Measured, three kernels, by the row's thread / in order, us: 16
// columns, 128 x 2K tokens x 16 heads 224 / 242; 32 columns, 16 x 4K x 32 118 / 125, lists of 16 102 / 109, without a causal mask 46.4 / 45.4;
// 64 columns, 8 x 8K x 32 127 / 130, without a mask, 16 x 4K x 12 52 / 47, 4 x 4K 18.4 / 16.7.
constexpr int kDirectCols = 32;
// shared memory of the scatter: the columns' arrays; the tile's entries (lists of up to `kmax`) take the place of all but the cursors
constexpr size_t scatter_bytes(int ncols, int kmax) {
  return (size_t)ncols * 8 + ((size_t)ncols * (kColBytes - 8) > (size_t)kTileRows * kmax * 4 ? (size_t)ncols * (kColBytes - 8) : (size_t)kTileRows * kmax * 4);
}

struct CscParams {
  const int32_t* topk_idx; int64_t idx_rs, idx_hs;   // element strides of (row, head)
  const int32_t* cu_q;
  int64_t* col_offsets; int32_t* col_nnz; int32_t* indices;
  int32_t* hist;                                      // [B*H][ntiles][ncol]
  uint32_t* row_slots;                                // optional: [(h*total_q + token)*topk + ...], ascending, 0xffffffff = no entry
  int64_t total_q;
  int batch, heads, topk, ncol, ntiles, cols_per_cta;
  int scanned;                                        // 1: hist holds cursors (tile_scan has run), 0: counts
};

// ascending sorting networks on 8 and 16 ids: 19 compare-exchanges; two sorted eights and a bitonic merge
__device__ __forceinline__ void csc_ce(int& a, int& b) {
  const int lo = min(a, b), hi = max(a, b);
  a = lo;
  b = hi;
}
__device__ __forceinline__ void csc_sort8(int* x) {
  csc_ce(x[0], x[1]); csc_ce(x[2], x[3]); csc_ce(x[4], x[5]); csc_ce(x[6], x[7]);
  csc_ce(x[0], x[2]); csc_ce(x[1], x[3]); csc_ce(x[4], x[6]); csc_ce(x[5], x[7]);
  csc_ce(x[1], x[2]); csc_ce(x[5], x[6]); csc_ce(x[0], x[4]); csc_ce(x[3], x[7]);
  csc_ce(x[1], x[5]); csc_ce(x[2], x[6]);
  csc_ce(x[1], x[4]); csc_ce(x[3], x[6]);
  csc_ce(x[2], x[4]); csc_ce(x[3], x[5]);
  csc_ce(x[3], x[4]);
}
template <int N>
__device__ __forceinline__ void csc_sort(int* x) {
#pragma unroll
  for (int i = 0; i < N; i += 8) csc_sort8(x + i);
  if constexpr (N == 16) {
#pragma unroll
    for (int i = 0; i < 8; ++i) csc_ce(x[i], x[15 - i]);
#pragma unroll
    for (int o = 4; o; o >>= 1)
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if ((i & o) == 0) csc_ce(x[i], x[i + o]);
  }
}

constexpr int kCscNone = 0x7fffffff;
// the list of row `r` of a tile (src: the tile's first row), places without a chunk of the pattern as kCscNone
template <int KMAX>
__device__ __forceinline__ void csc_load_row(const CscParams& p, const int32_t* src, int r, int (&id)[KMAX]) {
  const int32_t* mine = src + (int64_t)r * p.idx_rs;
  if (p.topk == KMAX && (p.idx_rs & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll
    for (int j = 0; j < KMAX; j += 4) {
      const int4 q = *reinterpret_cast<const int4*>(mine + j);
      id[j] = q.x; id[j + 1] = q.y; id[j + 2] = q.z; id[j + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < KMAX; ++j) id[j] = j < p.topk ? mine[j] : kCscNone;
  }
#pragma unroll
  for (int j = 0; j < KMAX; ++j)
    if (id[j] < 0 || id[j] >= p.ncol) id[j] = kCscNone;
}

// KMAX as for the scatter kernel below.  A chunk that a row names twice counts once.
template <int KMAX>
__global__ void __launch_bounds__(kCscThreads) csc_tile_hist_kernel(CscParams p) {
  follow_on();
  extern __shared__ uint32_t sm[];
  const int bh = blockIdx.x, tile = blockIdx.y, c0 = blockIdx.z * p.cols_per_cta;
  const int b = bh / p.heads, h = bh - b * p.heads;
  const int seq0 = p.cu_q[b], len_q = p.cu_q[b + 1] - seq0;
  const int ncols = min(p.cols_per_cta, p.ncol - c0);
  int32_t* hist = p.hist + ((int64_t)bh * p.ntiles + tile) * p.ncol + c0;
  const int r0 = tile * kTileRows, rows = min(kTileRows, len_q - r0);
  if (rows <= 0) {   // tile beyond this sequence: empty counts
    for (int c = threadIdx.x; c < ncols; c += kCscThreads) hist[c] = 0;
    return;
  }
  for (int c = threadIdx.x; c < ncols; c += kCscThreads) sm[c] = 0u;
  __syncthreads();
  const int32_t* src = p.topk_idx + (int64_t)(seq0 + r0) * p.idx_rs + (int64_t)h * p.idx_hs;
  auto count = [&](int c) {
    if ((uint32_t)(c - c0) < (uint32_t)ncols) atomicAdd(&sm[c - c0], 1u);
  };
  if constexpr (KMAX > 0) {
    if ((int)threadIdx.x < rows) {
      int id[KMAX];
      csc_load_row<KMAX>(p, src, threadIdx.x, id);
      csc_sort<KMAX>(id);
#pragma unroll
      for (int j = 0; j < KMAX; ++j)
        if (j == 0 || id[j] != id[j > 0 ? j - 1 : 0]) count(id[j]);
    }
  } else {
    for (int e = threadIdx.x; e < rows * p.topk; e += kCscThreads) {
      const int r = e / p.topk, j = e - r * p.topk;
      const int32_t* list = src + (int64_t)r * p.idx_rs;
      const int c = list[j];
      bool again = false;
      for (int i = 0; i < j; ++i) again = again || list[i] == c;
      if (!again) count(c);
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < ncols; c += kCscThreads) hist[c] = (int)sm[c];
}

// grid (b*h, groups of 32 columns): 32 warps, lane = column; the tiles are cut into 32 runs, one per warp
__global__ void __launch_bounds__(1024) csc_tile_scan_kernel(CscParams p) {
  follow_on();
  __shared__ int run_sum[32][33];
  const int bh = blockIdx.x, b = bh / p.heads;
  const int ntiles_b = (p.cu_q[b + 1] - p.cu_q[b] + kTileRows - 1) / kTileRows;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.y * 32 + lane;
  const int per = (ntiles_b + 31) / 32, t0 = warp * per, t1 = min(ntiles_b, t0 + per);
  int32_t* hist = p.hist + (int64_t)bh * p.ntiles * p.ncol + c;
  int sum = 0;
  if (c < p.ncol) {
#pragma unroll 4
    for (int t = t0; t < t1; ++t) sum += hist[(int64_t)t * p.ncol];
  }
  run_sum[warp][lane] = sum;
  __syncthreads();
  int before = 0, total = 0;
  for (int w = 0; w < 32; ++w) {
    const int x = run_sum[w][lane];
    before += w < warp ? x : 0;
    total += x;
  }
  if (c >= p.ncol) return;
  for (int t = t0; t < t1; ++t) {
    const int x = hist[(int64_t)t * p.ncol];
    hist[(int64_t)t * p.ncol] = before;
    before += x;
  }
  if (warp == 0) p.col_nnz[(int64_t)bh * p.ncol + c] = total;
}

// KMAX: 8 or 16: lists of at most that many ids are sorted in registers by one thread per row; 0: any length,
// a thread per entry
// OWN: a sequence is one tile: its columns are the tile's, nobody has counted them before
template <int KMAX, bool OWN>
__global__ void __launch_bounds__(kCscThreads, 2) csc_scatter_kernel(CscParams p) {
  follow_on();
  extern __shared__ __align__(16) uint32_t sm[];
  // places inside a (b, h)'s region: fewer than 65,535 tiles of 512 rows, of lists of up to 16, fit 32 bits
  using Off = typename std::conditional<(KMAX > 0), int, int64_t>::type;
  __shared__ Off warp_sums[kCscThreads / 32];
  const int bh = blockIdx.x, tile = blockIdx.y, c0 = blockIdx.z * p.cols_per_cta;
  const int b = bh / p.heads, h = bh - b * p.heads;
  const int lead = p.cu_q[0], seq0 = p.cu_q[b], len_q = p.cu_q[b + 1] - seq0;
  const int r0 = tile * kTileRows, rows = min(kTileRows, len_q - r0);
  if (rows <= 0 && tile > 0) return;            // (the first tile of an empty sequence still writes its columns)
  const int ncols = min(p.cols_per_cta, p.ncol - c0);
  const int ntiles_b = (len_q + kTileRows - 1) / kTileRows;
  // [ncols] x: first of the column's entries among the tile's (column by column), y: from there to their places in the region
  uint2* base = reinterpret_cast<uint2*>(sm);
  uint32_t* bm = sm + ncols * 2;                                  // [ncols][kBmStride] bit (row) of every column
  uint16_t* before = reinterpret_cast<uint16_t*>(bm + ncols * kBmStride);   // [kTileWords][ncols] rows ahead of each 32
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t region = ((int64_t)seq0 * p.heads + (int64_t)len_q * h) * p.topk;   // first place of this (b, h) in `indices`
  {
    uint4* zero = reinterpret_cast<uint4*>(sm);                   // (the cursors as well: they are written further down)
    const int n = (ncols * (2 + kBmStride) + 3) / 4;              // (at most 12 bytes into `before`)
    for (int i = tid; i < n; i += kCscThreads) zero[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  // the row's list, on its way while the columns are looked up
  const int32_t* src = p.topk_idx + (int64_t)(seq0 + r0) * p.idx_rs + (int64_t)h * p.idx_hs;
  static_assert(kTileRows == kCscThreads, "a thread per row");
  int id[KMAX > 0 ? KMAX : 1];
  if constexpr (KMAX > 0) {
    if (tid < rows) csc_load_row<KMAX>(p, src, tid, id);
  }

  const int32_t* hist = p.hist + (int64_t)bh * p.ntiles * p.ncol;
  // exclusive sum over the CTA's threads; `total`: of all
  auto scan = [&](Off x, Off& total) {
    const Off own = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const Off y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    constexpr int W = kCscThreads / 32;
    Off sums = warp_sums[lane % W];
#pragma unroll
    for (int o = 1; o < W; o <<= 1) {
      const Off y = __shfl_up_sync(0xffffffffu, sums, o, W);
      if (lane % W >= o) sums += y;
    }
    total = __shfl_sync(0xffffffffu, sums, W - 1);
    const Off ahead = __shfl_sync(0xffffffffu, sums, max(warp - 1, 0));
    __syncthreads();
    return (warp > 0 ? ahead : 0) + x - own;
  };
  auto put_column = [&](int c, int64_t off, int nnz) {
    p.col_offsets[(int64_t)bh * p.ncol + c] = region + off;
    if (OWN || !p.scanned) p.col_nnz[(int64_t)bh * p.ncol + c] = nnz;
  };
  // ---- column offsets (places inside the region) and this tile's cursor in every column
  Off carry = 0, total;
  for (int g0 = 0; !OWN && g0 < p.ncol; g0 += kCscThreads) {
    const int c = g0 + tid;
    int nnz = 0, cursor = 0;
    if (c < p.ncol) {
      if (p.scanned) {
        nnz = p.col_nnz[(int64_t)bh * p.ncol + c];
        cursor = tile < ntiles_b ? hist[(int64_t)tile * p.ncol + c] : 0;
      } else {
#pragma unroll 4
        for (int t = 0; t < ntiles_b; ++t) {
          const int x = hist[(int64_t)t * p.ncol + c];
          cursor += t < tile ? x : 0;
          nnz += x;
        }
      }
    }
    const Off off = carry + scan(nnz, total);
    if (c < p.ncol) {
      if (c >= c0 && c < c0 + ncols) base[c - c0].y = (uint32_t)(off + cursor);
      if (tile == 0 && blockIdx.z == 0) put_column(c, off, nnz);
    }
    carry += total;
  }
  // the unused tail of the region stays zero, as in the reference's zero-initialised buffer
  // (csrc/flash_topk/flash_topk_api.cpp:217); its tiles share it
  auto clear_tail = [&](int64_t used) {
    if (blockIdx.z == 0 && ntiles_b > 0)
      for (int64_t i = used + (int64_t)tile * kCscThreads + tid; i < (int64_t)len_q * p.topk; i += (int64_t)ntiles_b * kCscThreads)
        p.indices[region + i] = 0;
  };
  if (!OWN) clear_tail(carry);
  // rows of no sequence (q padded to a fixed size): their lists are empty.  The merge goes over all rows of q
  if (p.row_slots != nullptr && b == p.batch - 1 && blockIdx.z == 0 && (lead > 0 || seq0 + len_q < p.total_q)) {
    uint32_t* lists = p.row_slots + (int64_t)h * p.total_q * p.topk;
    const int64_t first = (int64_t)tile * kCscThreads + tid, step = (int64_t)max(1, ntiles_b) * kCscThreads;
    for (int64_t i = first; i < (int64_t)lead * p.topk; i += step) lists[i] = 0xffffffffu;
    for (int64_t i = (int64_t)(seq0 + len_q) * p.topk + first; i < p.total_q * p.topk; i += step) lists[i] = 0xffffffffu;
  }
  if (!OWN && rows <= 0) return;

  // ---- bitmap of the tile
  if (OWN) __syncthreads();                                       // (it has been cleared: otherwise a scan has come in between)
  if constexpr (KMAX > 0) {
    if (tid < rows) {
#pragma unroll
      for (int j = 0; j < KMAX; ++j) {
        const int c = id[j] - c0;
        if ((uint32_t)c < (uint32_t)ncols) atomicOr(&bm[c * kBmStride + warp], 1u << lane);
      }
    }
  } else {
    for (int e = tid; e < rows * p.topk; e += kCscThreads) {
      const int r = e / p.topk, c = src[(int64_t)r * p.idx_rs + (e - r * p.topk)] - c0;
      if (c >= 0 && c < ncols) atomicOr(&bm[c * kBmStride + (r >> 5)], 1u << (r & 31));
    }
  }
  __syncthreads();
  int entries = 0;                                                // of the tile, in this CTA's columns
  for (int g0 = 0; g0 < ncols; g0 += kCscThreads) {
    const int c = g0 + tid;
    int run = 0;
    if (c < ncols) {
#pragma unroll
      for (int w = 0; w < kTileWords; ++w) {
        before[w * ncols + c] = (uint16_t)run;           // (neighbouring lanes, neighbouring places: no bank conflicts)
        run += __popc(bm[c * kBmStride + w]);
      }
    }
    const int first = entries + (int)scan(run, total);
    if (OWN && c < ncols) put_column(c, first, run);
    if (c < ncols) base[c] = make_uint2((uint32_t)first, OWN ? 0u : base[c].y - (uint32_t)first);
    entries += (int)total;
  }
  __syncthreads();
  if (OWN) clear_tail(entries);
  if (OWN && rows <= 0) return;

  // ---- places: first of the column's entries in this tile, plus its rows ahead of this one
  auto place = [&](int c, int r) {
    return before[(r >> 5) * ncols + c] + (uint32_t)__popc(bm[c * kBmStride + (r >> 5)] & ((1u << (r & 31)) - 1u));
  };
  if constexpr (KMAX > 0) {
    uint32_t local[KMAX];                                         // place among the tile's entries
    int32_t* into = p.indices + region;
    const bool direct = ncols <= kDirectCols;                     // (CTA-uniform)
    if (tid < rows) {
      if (p.row_slots != nullptr) csc_sort<KMAX>(id);             // ascending columns are ascending places
      uint32_t at[KMAX];
#pragma unroll
      for (int j = 0; j < KMAX; ++j) {
        const int c = id[j] - c0;
        at[j] = local[j] = 0xffffffffu;
        if ((uint32_t)c < (uint32_t)ncols) {
          const uint2 f = base[c];
          local[j] = f.x + place(c, tid);
          at[j] = (uint32_t)region + local[j] + f.y;              // (row_slots are kept for fewer than 2^32 entries only)
          if (direct) into[local[j] + f.y] = r0 + tid;
        }
      }
      if (p.row_slots != nullptr) {
        uint32_t* out = p.row_slots + ((int64_t)h * p.total_q + seq0 + r0 + tid) * p.topk;
        if (p.topk == KMAX && gridDim.z == 1 && (reinterpret_cast<uintptr_t>(p.row_slots) & 15) == 0) {
#pragma unroll
          for (int j = 0; j < KMAX; j += 4) *reinterpret_cast<uint4*>(out + j) = make_uint4(at[j], at[j + 1], at[j + 2], at[j + 3]);
        } else {                                                  // a CTA writes the entries of its own columns
#pragma unroll
          for (int j = 0; j < KMAX; ++j)
            if (j < p.topk && (at[j] != 0xffffffffu || (id[j] == kCscNone && blockIdx.z == 0))) out[j] = at[j];
        }
      }
    }
    if (direct) return;
    __syncthreads();                                              // the bitmap is done with: its place takes the entries
    uint32_t* entry = bm;                                         // column and row of every entry, column by column
    if (tid < rows) {
#pragma unroll
      for (int j = 0; j < KMAX; ++j)
        if (local[j] != 0xffffffffu) entry[local[j]] = (uint32_t)(id[j] - c0) << 16 | (uint32_t)tid;
    }
    __syncthreads();
    for (int i = tid; i < entries; i += kCscThreads) {
      const uint32_t e = entry[i];
      into[i + base[e >> 16].y] = r0 + (int)(e & 0xffffu);
    }
  } else {
    uint32_t* out = p.row_slots ? p.row_slots + ((int64_t)h * p.total_q + seq0 + r0) * p.topk : nullptr;
    for (int e = tid; e < rows * p.topk; e += kCscThreads) {
      const int r = e / p.topk, j = e - r * p.topk;
      const int32_t* list = src + (int64_t)r * p.idx_rs;
      const int cg = list[j];
      const bool used = cg >= 0 && cg < p.ncol;
      const int c = cg - c0;
      const bool here = used && c >= 0 && c < ncols;
      uint32_t x = 0;
      if (here) {
        x = base[c].x + place(c, r) + base[c].y;
        p.indices[region + x] = r0 + r;
      }
      if (out != nullptr && (here || (!used && blockIdx.z == 0))) {
        int rank = 0;                                             // places in ascending order, empty ones last
        for (int i = 0; i < p.topk; ++i) {
          const int o = list[i];
          const bool o_used = o >= 0 && o < p.ncol;
          rank += (used ? (o_used && o < cg) : (o_used || i < j)) ? 1 : 0;
        }
        out[(int64_t)r * p.topk + rank] = here ? (uint32_t)region + x : 0xffffffffu;
      }
    }
  }
}

static int csc_ntiles(int max_q) { return max(1, ceil_div(max_q, kTileRows)); }

size_t csc_workspace_bytes(int batch, int heads, int max_q, int ncol) {
  return align_up((size_t)batch * heads * csc_ntiles(max_q) * (size_t)max(ncol, 1) * sizeof(int32_t), 256);
}

int launch_build_csc(const int32_t* topk_idx, int64_t idx_rs, int64_t idx_hs, const int32_t* cu_q, int64_t* col_offsets, int32_t* col_nnz,
                     int32_t* indices, void* ws, size_t ws_bytes, int batch, int heads, int topk, int max_q,
                     int ncol, cudaStream_t s, uint32_t* row_slots, int64_t total_q) {
  if (batch == 0 || heads == 0 || ncol == 0) return FMB_OK;
  if (ws == nullptr || ws_bytes < csc_workspace_bytes(batch, heads, max_q, ncol))
    return fail(FMB_ERR_WORKSPACE, "build_csc: workspace too small (%zu < %zu)", ws_bytes,
                csc_workspace_bytes(batch, heads, max_q, ncol));
  CscParams p;
  p.topk_idx = topk_idx;
  p.idx_rs = idx_rs;
  p.idx_hs = idx_hs;
  p.cu_q = cu_q; p.col_offsets = col_offsets; p.col_nnz = col_nnz; p.indices = indices;
  p.hist = static_cast<int32_t*>(ws);
  p.row_slots = row_slots; p.total_q = total_q;
  p.batch = batch; p.heads = heads; p.topk = topk; p.ncol = ncol; p.ntiles = csc_ntiles(max_q);
  // few tiles: their scatter CTAs add up the counts of the tiles before their own (at most 16 numbers per
  // column) instead of waiting for one more launch
  p.scanned = p.ntiles > 16 ? 1 : 0;
  // A tile a sequence: the scatter's bitmap has the columns' entries anyway, nobody counts them ahead of it.  Both kernels / the scatter alone, us: four
  // sequences of 512, 16 heads 7.26 / 4.59, eight of 500, lists of 16 14.55 / 6.97, one of 200, 4 heads 5.94 / 3.69; the whole pattern of 64 of 500, 16
  // heads 95.1 / 87.3, of 200 of 120 102.9 / 84.4.  Two to four tiles, two kernels / scatter CTAs that each count all tiles of their (b, h): 1K and
  // 2K tokens, 8 heads, lists of four 7.2 / 8.3, of eight 8.1 / 11.2, of 16 12.4 / 20.0 (the whole pattern 27.2 / 44.7)
  const bool own = topk <= 16 && p.ntiles == 1 && ncol <= kMaxColsPerCta;
  prof_begin(6, s);
  if (!own) {
    p.cols_per_cta = min(kMaxHistCols, ncol);
    auto count = topk <= 8 ? csc_tile_hist_kernel<8> : topk <= 16 ? csc_tile_hist_kernel<16> : csc_tile_hist_kernel<0>;
    launch_follow_on(count, dim3(batch * heads, p.ntiles, ceil_div(ncol, p.cols_per_cta)), dim3(kCscThreads),
                     (size_t)p.cols_per_cta * sizeof(uint32_t), s, p);
    FMB_LAUNCH_CHECK("csc_tile_hist_kernel");
  }
  if (p.scanned) {
    launch_follow_on(csc_tile_scan_kernel, dim3(batch * heads, ceil_div(ncol, 32)), dim3(1024), 0, s, p);
    FMB_LAUNCH_CHECK("csc_tile_scan_kernel");
  }
  p.cols_per_cta = min(kMaxColsPerCta, ncol);
  const dim3 grid(batch * heads, p.ntiles, ceil_div(ncol, p.cols_per_cta));
  const int kmax = topk <= 8 ? 8 : topk <= 16 ? 16 : 0;
  const size_t smem = scatter_bytes(p.cols_per_cta, kmax);
  auto scatter = own ? (topk <= 8 ? csc_scatter_kernel<8, true> : csc_scatter_kernel<16, true>)
               : topk <= 8 ? csc_scatter_kernel<8, false> : topk <= 16 ? csc_scatter_kernel<16, false> : csc_scatter_kernel<0, false>;
  // the attribute belongs to the current device: set on every call (cheap, idempotent, thread-safe)
  FMB_CUDA(cudaFuncSetAttribute(scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)scatter_bytes(kMaxColsPerCta, kmax)));
  launch_follow_on(scatter, grid, dim3(kCscThreads), smem, s, p);
  prof_end(6, s);
  FMB_LAUNCH_CHECK("csc_scatter_kernel");
  return FMB_OK;
}

// ---------------------------------------------------------------------------------------
// Pattern build for callers that cannot allocate device memory.
//
// Some hosts of this library have no way to hand over a workspace: a serving runtime that
// claims all device memory at start-up and forbids cudaMalloc afterwards (the call
// synchronises the whole device and can fail once the arena owns the memory), or a thin
// FFI shim in another language that only forwards the pointers it was given.  For them the
// tile-histogram scratch of the builder lives in this file-scope device array instead.
//   * capacity: kStaticScratchBytes (8 MiB), i.e. batch*heads*ceil(max_seqlen_q/512)*ncol
//     <= 2,097,152 counters (e.g. one 64K-token sequence x 32 heads x 512 chunks); larger
//     problems are rejected with FMB_ERR_WORKSPACE and must use fmb_build_csc;
//   * every GPU that loads the library holds the array until the process exits;
//   * the array is shared by all calls and keeps the previous call's contents.  Nothing has
//     to start at zero: the histogram kernel writes every counter the later kernels read;
//   * two calls that overlap on the GPU (different streams, or different host threads)
//     race on the array: issue them on one stream, or order them with events.
// In host code the array's name is only a stand-in; the device address is obtained once per
// device with cudaGetSymbolAddress, on the first call made with that device current.  That
// first call should therefore be made outside any stream capture.
// ---------------------------------------------------------------------------------------
constexpr size_t kStaticScratchBytes = 8u << 20;
static __device__ __align__(256) int32_t g_csc_static_scratch[kStaticScratchBytes / sizeof(int32_t)];

static int csc_static_scratch_ptr(int32_t** out) {
  constexpr int kMaxDevices = 64;
  static std::mutex mu;
  static int32_t* ptrs[kMaxDevices] = {};
  int dev = 0;
  FMB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail(FMB_ERR_CUDA, "build_csc_static: device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (ptrs[dev] == nullptr) {
    int32_t* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_csc_static_scratch);
    if (e != cudaSuccess || p == nullptr)
      return fail(FMB_ERR_CUDA, "build_csc_static: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
    ptrs[dev] = p;
  }
  *out = ptrs[dev];
  return FMB_OK;
}

size_t csc_static_scratch_bytes() { return kStaticScratchBytes; }

int launch_build_csc_static(const int32_t* topk_idx, int64_t idx_rs, int64_t idx_hs, const int32_t* cu_q,
                            int64_t* col_offsets, int32_t* col_nnz, int32_t* indices, int batch, int heads,
                            int topk, int max_q, int ncol, cudaStream_t s) {
  if (batch == 0 || heads == 0 || ncol == 0) return FMB_OK;
  const size_t need = csc_workspace_bytes(batch, heads, max_q, ncol);
  if (need > kStaticScratchBytes)
    return fail(FMB_ERR_WORKSPACE,
                "build_csc_static: this problem needs %zu bytes of scratch, the built-in array holds %zu "
                "(batch*heads*ceil(max_seqlen_q/512)*ncol must be <= %zu); use fmb_build_csc with a workspace",
                need, kStaticScratchBytes, kStaticScratchBytes / sizeof(int32_t));
  int32_t* scratch = nullptr;
  const int rc = csc_static_scratch_ptr(&scratch);
  if (rc) return rc;
  return launch_build_csc(topk_idx, idx_rs, idx_hs, cu_q, col_offsets, col_nnz, indices, scratch,
                          kStaticScratchBytes, batch, heads, topk, max_q, ncol, s);
}

// ---------------------------------------------------------------------------------------
// Stand-alone segmented ascending sort (the reference's varlen_sort entry point,
// csrc/flash_topk/src/varlen_sort.cu:127-162).  The pattern builder above never needs it;
// it exists for callers that sort their own column lists.  One CTA per segment runs a
// direction-free bitonic network in place on dst: every compare-exchange puts the smaller
// key at the lower index, so virtual +inf padding above the segment end never moves.
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) varlen_sort_kernel(const int64_t* __restrict__ starts,
                                                          const int64_t* __restrict__ ends,
                                                          const int32_t* __restrict__ src,
                                                          int32_t* __restrict__ dst, int64_t nitems) {
  const int64_t s0 = starts[blockIdx.x], s1 = ends[blockIdx.x];
  if (s1 <= s0 || s0 < 0 || s1 > nitems) return;
  const int64_t n = s1 - s0;
  int32_t* a = dst + s0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) a[i] = src[s0 + i];
  __syncthreads();
  int64_t N = 1;
  while (N < n) N <<= 1;
  for (int64_t k = 2; k <= N; k <<= 1) {
    for (int64_t j = k >> 1; j >= 1; j >>= 1) {
      const bool flip = (j == (k >> 1));
      for (int64_t i = threadIdx.x; i < N; i += blockDim.x) {
        const int64_t l = flip ? (i ^ (k - 1)) : (i ^ j);
        if (l > i && l < n) {
          const int32_t x = a[i], y = a[l];
          if (x > y) { a[i] = y; a[l] = x; }
        }
      }
      __syncthreads();
    }
  }
}

int launch_varlen_sort(const int64_t* starts, const int64_t* ends, const int32_t* src, int32_t* dst,
                       int64_t nseg, int64_t nitems, cudaStream_t s) {
  FMB_CUDA(cudaMemsetAsync(dst, 0, (size_t)nitems * sizeof(int32_t), s));
  if (nseg == 0 || nitems == 0) return FMB_OK;
  FMB_CHECK_ARG(nseg <= 0x7fffffff, "varlen_sort: too many segments");
  varlen_sort_kernel<<<(unsigned)nseg, 256, 0, s>>>(starts, ends, src, dst, nitems);
  FMB_LAUNCH_CHECK("varlen_sort_kernel");
  return FMB_OK;
}

}  // namespace fmb
