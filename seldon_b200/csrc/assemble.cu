// Device assembly of CSR matrices from coordinate triplets: Seldon's
// ConvertMatrix_from_Coordinates (matrix_sparse/Matrix_Conversions.cxx:
// 1291-1334 for RowSparse, 1397-1467 for RowSymSparse) on the GPU.
//
// Seldon sorts the triplets by row, then each row by column, both times with
// its bottom-up merge sort (vector/Functions_Arrays.cxx:412-500), which keeps
// equal keys in input order.  The result is the triplets in stable
// (row, column) order, duplicates kept as separate entries.  Here:
//
//   k_coo_stats       sizes: largest row and column, bad indices, kept count,
//                     and whether the triplets come in order already
//   k_coo_sorted      triplets in order: copies, and ptr from the row changes
//   k_coo_rows        or, across long runs of empty rows, from a search a row
//   k_bkt_*           the rest, where buckets of rows fit a CTA (see there)
//   otherwise:
//   k_row_count       entries per row (warp-aggregated atomics), scanned
//                     into ptr
//   k_row_scatter     each entry's key (column << ib | input position) to a
//                     free slot of its row (atomics: any order inside a row)
//   k_row_sort_short  rows of up to 32 entries, one thread each: an entry's
//                     place is the number of smaller keys in its row; the
//                     keys are distinct (they hold the input position), so
//                     the order is (column, input position) exactly
//   k_row_sort_cta    rows of 33..4096 entries, one CTA each: bitonic sort
//                     in shared memory
//   longer rows       the stable LSD radix sort below, on the row's keys
//   (the sorted keys give ind directly and val through the position)
//
// The whole call, from Python: 14.6M shuffled triplets of the 128^3 operator
// 615 us (1030 with the last form), the same in order 206 us (483), 13.7M in
// order of power-law rows 195 us (1274).
//
// All of it is integer and byte movement bound by HBM bandwidth and L2
// atomics; the matrix comes out deterministic whatever order the atomics
// take, because every row is sorted on distinct keys afterwards.
#include <algorithm>
#include <climits>
#include <utility>

#include "sb2_internal.cuh"

namespace sb2 {
namespace {

constexpr int kAsmThreads = 256;
constexpr int kAsmWarps = kAsmThreads / 32;
constexpr int kChunks = 16;
constexpr int kTile = kAsmThreads * kChunks;  // triplets per tile
constexpr int kBins = 256;                     // 8-bit digits

struct CooStats {
  int row_max;  // largest row - index (0 when empty)
  int col_max;
  int bad;      // some index - index < 0 or too large
  int kept;     // entries with row <= col
  int unsorted; // the triplets are not in (row, column) order
  int gap;      // most rows between a triplet and the next (of the first: from -1)
};

// Also whether the triplets come in (row, column) order already: each is
// compared with the next.
__global__ void __launch_bounds__(kAsmThreads)
k_coo_stats(const int* __restrict__ row, const int* __restrict__ col, long long nnz, int index,
            CooStats* st) {
  constexpr int U = 4;
  int rmax = 0, cmax = 0, bad = 0, kept = 0, unsorted = 0, gap = 0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  for (long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < nnz;
       i0 += U * stride) {
    int rv[U], cv[U], rn[U], cn[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const long long i = i0 + u * stride + lane;
      rv[u] = i < nnz ? __ldg(row + i) : index;
      cv[u] = i < nnz ? __ldg(col + i) : index;
      // the next triplet comes from the next lane, the last lane's from memory
      const bool edge = lane == 31 && i + 1 < nnz;
      rn[u] = edge ? __ldg(row + i + 1) : INT_MAX;
      cn[u] = edge ? __ldg(col + i + 1) : INT_MAX;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const long long i = i0 + u * stride + lane;
      const long long r = (long long)rv[u] - index, c = (long long)cv[u] - index;
      const int r2 = __shfl_down_sync(0xffffffffu, rv[u], 1), c2 = __shfl_down_sync(0xffffffffu, cv[u], 1);
      if (lane < 31) {
        rn[u] = r2;
        cn[u] = c2;
      }
      if (i + 1 < nnz) {
        unsorted |= rn[u] < rv[u] || (rn[u] == rv[u] && cn[u] < cv[u]);
        if (rn[u] > rv[u]) gap = max(gap, (int)((unsigned)rn[u] - (unsigned)rv[u]));
      }
      const bool out = r < 0 || c < 0 || r >= INT_MAX || c >= INT_MAX;
      bad |= out;
      if (!out && i < nnz) {
        rmax = max(rmax, (int)r);
        cmax = max(cmax, (int)c);
        kept += (r <= c);
        if (i == 0) gap = max(gap, (int)r + 1);
      }
    }
  }
  rmax = __reduce_max_sync(0xffffffffu, rmax);
  cmax = __reduce_max_sync(0xffffffffu, cmax);
  bad = __reduce_or_sync(0xffffffffu, bad);
  kept = __reduce_add_sync(0xffffffffu, kept);
  unsorted = __reduce_or_sync(0xffffffffu, unsorted);
  gap = __reduce_max_sync(0xffffffffu, gap);
  // one set of atomics per CTA: with one per warp they took longer than the reads
  __shared__ int s_st[kAsmWarps][6];
  if (lane == 0) {
    int* w = s_st[threadIdx.x >> 5];
    w[0] = rmax; w[1] = cmax; w[2] = bad; w[3] = kept; w[4] = unsorted; w[5] = gap;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kAsmWarps; w++) {
      rmax = max(rmax, s_st[w][0]);
      cmax = max(cmax, s_st[w][1]);
      bad |= s_st[w][2];
      kept += s_st[w][3];
      unsorted |= s_st[w][4];
      gap = max(gap, s_st[w][5]);
    }
    atomicMax(&st->row_max, rmax);
    atomicMax(&st->col_max, cmax);
    if (bad) atomicOr(&st->bad, 1);
    atomicAdd(&st->kept, kept);
    if (unsorted) atomicOr(&st->unsorted, 1);
    atomicMax(&st->gap, gap);
  }
}

// Rows that one thread of k_coo_sorted fills ptr for at most.  1M triplets, gaps
// of 1024 rows: 132 us a call so, 175 with the searches; of 4096: 179 and 173; one
// gap of 16M rows: 56 ms and 0.44.
constexpr int kGapRows = 2048;

// Triplets that are in order: ind and val are copies, and ptr[r] is the place
// of the first triplet of row r or beyond: the triplet's thread fills ptr from
// the row of the one before.  Where that may be many rows (GAPS) k_coo_rows
// fills it instead.
template <bool GAPS>
__global__ void __launch_bounds__(kAsmThreads)
k_coo_sorted(const int* __restrict__ row, const int* __restrict__ col,
             const double* __restrict__ val, long long nnz, int index, int m,
             int* __restrict__ ptr, int* __restrict__ ind, double* __restrict__ vout) {
  const long long stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += stride) {
    const int r = __ldg(row + i) - index, before = i ? __ldg(row + i - 1) - index : -1;
    ind[i] = __ldcs(col + i) - index;
    vout[i] = __ldcs(val + i);
    if (!GAPS) {
      for (int q = before + 1; q <= r; q++) ptr[q] = (int)i;
      if (i == nnz - 1)
        for (int q = r + 1; q <= m; q++) ptr[q] = (int)nnz;
    }
  }
}

// ptr of triplets in order by a search for each row.
__global__ void __launch_bounds__(kAsmThreads)
k_coo_rows(const int* __restrict__ row, long long nnz, int index, int m, int* __restrict__ ptr) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r <= m; r += stride) {
    long long lo = 0, hi = nnz;  // the first triplet of row r or beyond lies in [lo, hi]
    while (lo < hi) {
      const long long mid = (lo + hi) >> 1;
      if ((long long)__ldg(row + mid) - index < r) lo = mid + 1;
      else hi = mid;
    }
    ptr[r] = (int)lo;
  }
}

// Digit counts of each tile, stored digit-major: hist[d * ntiles + tile].
template <typename K>
__global__ void __launch_bounds__(kAsmThreads)
k_radix_hist(const K* __restrict__ key, long long nnz, int ntiles, int shift,
             int* __restrict__ hist) {
  __shared__ int h[kBins];
  h[threadIdx.x] = 0;
  __syncthreads();
  const long long t0 = (long long)blockIdx.x * kTile;
  for (int c = 0; c < kChunks; ++c) {
    const long long i = t0 + c * kAsmThreads + threadIdx.x;
    if (i < nnz) atomicAdd(&h[(unsigned)(key[i] >> shift) & (kBins - 1)], 1);
  }
  __syncthreads();
  hist[(long long)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// Stable scatter of one tile: entry i goes to the tile's first position for
// its digit plus the number of earlier entries of the tile with that digit.
template <typename K>
__global__ void __launch_bounds__(kAsmThreads)
k_radix_scatter(const K* __restrict__ kin, const int* __restrict__ pin, long long nnz,
                int ntiles, int shift, const int* __restrict__ off, K* __restrict__ kout,
                int* __restrict__ pout) {
  __shared__ int s_cnt[kAsmWarps][kBins];  // digit counts of each warp's 32 entries
  __shared__ int s_off[kAsmWarps][kBins];  // first position of each warp's run
  __shared__ int s_base[kBins];            // next free position of each digit
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int w = 0; w < kAsmWarps; ++w) s_cnt[w][tid] = 0;
  s_base[tid] = off[(long long)tid * ntiles + blockIdx.x];
  __syncthreads();
  const long long t0 = (long long)blockIdx.x * kTile;
  for (int c = 0; c < kChunks; ++c) {
    const long long c0 = t0 + c * kAsmThreads;
    if (c0 >= nnz) break;  // uniform across the block
    const long long i = c0 + tid;
    const bool valid = i < nnz;
    const K k = valid ? kin[i] : K(0);
    const int p = (valid && pin) ? pin[i] : 0;
    const unsigned d = valid ? ((unsigned)(k >> shift) & (kBins - 1)) : (unsigned)kBins;
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const unsigned before = peers & ((1u << lane) - 1u);
    if (valid && before == 0) s_cnt[warp][d] = __popc(peers);
    __syncthreads();
    {
      int run = s_base[tid];
#pragma unroll
      for (int w = 0; w < kAsmWarps; ++w) {
        const int n = s_cnt[w][tid];
        s_off[w][tid] = run;
        run += n;
        s_cnt[w][tid] = 0;
      }
      s_base[tid] = run;
    }
    __syncthreads();
    if (valid) {
      const int q = s_off[warp][d] + __popc(before);
      kout[q] = k;
      if (pout) pout[q] = p;
    }
  }
}

// Exclusive scan of n ints in three launches: tile sums, a scan of the sums
// in one CTA, and the tiles rescanned from their base.
constexpr int kScanTile = kTile;

__device__ __forceinline__ int block_excl_scan(int v, int* s_warp, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  int wbase = 0, sum = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    const int s = s_warp[w];
    if (w < warp) wbase += s;
    sum += s;
  }
  __syncthreads();
  *total = sum;
  return wbase + incl - v;
}

__global__ void __launch_bounds__(kAsmThreads)
k_scan_sums(const int* __restrict__ a, long long n, int* __restrict__ sums) {
  __shared__ int s_warp[kAsmWarps];
  const long long t0 = (long long)blockIdx.x * kScanTile;
  int v = 0;
  for (int c = 0; c < kChunks; ++c) {
    const long long i = t0 + c * kAsmThreads + threadIdx.x;
    if (i < n) v += a[i];
  }
  int total;
  block_excl_scan(v, s_warp, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) k_scan_top(int* __restrict__ sums, int nb) {
  __shared__ int s_warp[32];
  const int per = (nb + 1023) / 1024;
  const int b0 = threadIdx.x * per;
  int v = 0;
  for (int j = 0; j < per; ++j)
    if (b0 + j < nb) v += sums[b0 + j];
  int total;
  int run = block_excl_scan(v, s_warp, &total);
  for (int j = 0; j < per; ++j)
    if (b0 + j < nb) {
      const int s = sums[b0 + j];
      sums[b0 + j] = run;
      run += s;
    }
}

__global__ void __launch_bounds__(kAsmThreads)
k_scan_tiles(int* __restrict__ a, long long n, const int* __restrict__ sums) {
  __shared__ int s_warp[kAsmWarps];
  const long long t0 = (long long)blockIdx.x * kScanTile;
  int base = sums[blockIdx.x];
  for (int c = 0; c < kChunks; ++c) {
    const long long c0 = t0 + c * kAsmThreads;
    if (c0 >= n) break;  // uniform
    const long long i = c0 + threadIdx.x;
    const int v = i < n ? a[i] : 0;
    int total;
    const int ex = block_excl_scan(v, s_warp, &total);
    if (i < n) a[i] = base + ex;
    base += total;
  }
}

// Entries per row.  Lanes of a warp that hit the same row add once.
__global__ void __launch_bounds__(kAsmThreads)
k_row_count(const int* __restrict__ row, const int* __restrict__ col, long long nnz, int index,
            int sym, int* __restrict__ cnt) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  for (long long i0 = (long long)blockIdx.x * blockDim.x; i0 < nnz; i0 += stride) {
    const long long i = i0 + threadIdx.x;
    int r = -1;
    if (i < nnz) {
      r = row[i] - index;
      if (sym && r > col[i] - index) r = -1;  // below the diagonal: dropped
    }
    const unsigned peers = __match_any_sync(0xffffffffu, r);
    if (r >= 0 && lane == __ffs(peers) - 1) atomicAdd(&cnt[r], __popc(peers));
  }
}

// Each kept entry's key to a free slot of its row.
__global__ void __launch_bounds__(kAsmThreads)
k_row_scatter(const int* __restrict__ row, const int* __restrict__ col, long long nnz, int index,
              int sym, int ib, int* __restrict__ fill, unsigned long long* __restrict__ key) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  for (long long i0 = (long long)blockIdx.x * blockDim.x; i0 < nnz; i0 += stride) {
    const long long i = i0 + threadIdx.x;
    int r = -1, c = 0;
    if (i < nnz) {
      r = row[i] - index;
      c = col[i] - index;
      if (sym && r > c) r = -1;
    }
    const unsigned peers = __match_any_sync(0xffffffffu, r);
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (r >= 0 && lane == leader) base = atomicAdd(&fill[r], __popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (r >= 0) {
      const int slot = base + __popc(peers & ((1u << lane) - 1u));
      key[slot] = ((unsigned long long)(unsigned)c << ib) | (unsigned long long)i;
    }
  }
}

__device__ __forceinline__ void emit(unsigned long long k, long long at, int ib,
                                     const double* __restrict__ val, int* __restrict__ ind,
                                     double* __restrict__ vout) {
  ind[at] = (int)(k >> ib);
  vout[at] = val[k & ((1ull << ib) - 1ull)];
}

constexpr int kShortRow = 32;
constexpr int kCtaRow = 4096;

// Rows of up to kShortRow entries; longer ones are listed for the CTA and
// segment sorts.
__global__ void __launch_bounds__(kAsmThreads)
k_row_sort_short(const int* __restrict__ ptr, int m, const unsigned long long* __restrict__ key,
                 int ib, const double* __restrict__ val, int* __restrict__ ind,
                 double* __restrict__ vout, int* __restrict__ long_rows, int* __restrict__ nlong) {
  const int stride = gridDim.x * blockDim.x;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < m; r += stride) {
    const int b = ptr[r], e = ptr[r + 1];
    if (e - b > kShortRow) {
      long_rows[atomicAdd(nlong, 1)] = r;
      if (e - b > kCtaRow) atomicAdd(nlong + 1, 1);
      continue;
    }
    for (int a = b; a < e; ++a) {
      const unsigned long long ka = key[a];
      int rank = 0;
      for (int c = b; c < e; ++c) rank += key[c] < ka;
      emit(ka, b + rank, ib, val, ind, vout);
    }
  }
}

// One CTA per listed row of kShortRow+1..kCtaRow entries: bitonic sort of the
// row's keys (padded with the largest key) in shared memory.
__global__ void __launch_bounds__(kAsmThreads)
k_row_sort_cta(const int* __restrict__ ptr, const int* __restrict__ rows,
               const unsigned long long* __restrict__ key, int ib,
               const double* __restrict__ val, int* __restrict__ ind,
               double* __restrict__ vout) {
  __shared__ unsigned long long s[kCtaRow];
  const int r = rows[blockIdx.x];
  const int b = ptr[r], L = ptr[r + 1] - b;
  if (L > kCtaRow) return;  // segment-sorted on its own
  int P = 1;
  while (P < L) P <<= 1;
  for (int i = threadIdx.x; i < P; i += blockDim.x) s[i] = i < L ? key[b + i] : ~0ull;
  __syncthreads();
  for (int k = 2; k <= P; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < P; i += blockDim.x) {
        const int x = i ^ j;
        if (x > i) {
          const unsigned long long u = s[i], v = s[x];
          if ((u > v) == ((i & k) == 0)) {
            s[i] = v;
            s[x] = u;
          }
        }
      }
      __syncthreads();
    }
  for (int i = threadIdx.x; i < L; i += blockDim.x) emit(s[i], b + i, ib, val, ind, vout);
}

// A sorted segment of keys written out.
__global__ void __launch_bounds__(kAsmThreads)
k_emit_segment(const unsigned long long* __restrict__ key, long long b, long long L, int ib,
               const double* __restrict__ val, int* __restrict__ ind, double* __restrict__ vout) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < L; i += stride)
    emit(key[b + i], b + i, ib, val, ind, vout);
}

// ---------------------------------------------------------------- two-pass form
//
// The triplets' keys are first dealt to buckets of consecutive rows, then
// every bucket is sorted in shared memory and written out.  A tile of keys is
// grouped by bucket in shared memory before it goes to global memory, then its
// values through the same shared memory, so that a bucket's part of a tile is
// written as one run: two entries on the mean with 4096 buckets, more with
// fewer.  (With the values gathered by the second pass, a 32-byte sector each,
// that pass alone took 458 us for 14.6M triplets of 7 a row, against 161 us.)
// The form after it scatters one key at a time to its row and gathers one value
// at a time; it stays for what does not fit here: more than kBktMax buckets,
// buckets beyond a CTA's shared memory (rows of very uneven length), keys beyond
// 64 bits, scratch beyond the memory there is.
//   k_bkt_count  entries per bucket
//   k_bkt_scan   first entry of each bucket; whether one is too large
//   k_bkt_deal   tiles of keys (row in the bucket, column, input position) and
//                values grouped by bucket
//   k_bkt_sort   one CTA per bucket: entries placed by row (shared-memory
//                counters), then an entry's place in a row of up to kBktRank
//                entries is the number of smaller keys there, and longer rows
//                take a bitonic sort; ptr, ind and val written

constexpr int kBktMax = 4096;      // buckets
constexpr int kBktThreads = 1024;
constexpr int kDealThreads = 512;
constexpr int kBktTile = 16 * kDealThreads;
constexpr int kSortThreads = 512;
constexpr int kBktCap = 5376;      // entries of a bucket at most: two CTAs an SM
constexpr int kBktRows = 4096;     // rows of a bucket at most
// Longest row that is ranked.  A row of the bitonic sort has the CTA to itself,
// 28 CTA barriers for 80 entries and half its threads idle up to 512; a rank
// reads the row once an entry, all lanes of a row the same key.  4M triplets,
// exactly 49 / 81 / 125 / 257 a row: 235 / 272 / 284 / 387 us a call, 1289 / 1071 / 793 /
// 752 with rows past 48 sorted; at 400 the two meet (502 and 610).
constexpr int kBktRank = 448;
constexpr int kBktLong = 16;       // longer rows of one bucket, at most

struct BktArgs {
  const int* row;
  const int* col;
  const double* val;
  long long nnz, nout;
  int index, sym, m;
  int lb, cb, ib;  // bits of a row in its bucket, of a column, of an input position
  int nb;          // buckets
  int* count;      // [nb + 1] entries, then first entry, of each bucket
  int* cursor;     // [nb] next free entry
  int* over;       // a bucket is too large
  unsigned long long* key;
  double* kval;
  int* ptr;
  int* ind;
  double* vout;
};

__global__ void __launch_bounds__(kBktThreads) k_bkt_count(BktArgs a) {
  __shared__ int h[kBktMax];
  for (int b = threadIdx.x; b < a.nb; b += kBktThreads) h[b] = 0;
  __syncthreads();
  const long long stride = (long long)gridDim.x * kBktThreads;
#pragma unroll 4
  for (long long i = (long long)blockIdx.x * kBktThreads + threadIdx.x; i < a.nnz; i += stride) {
    const int r = __ldg(a.row + i);
    if (!a.sym || r <= __ldg(a.col + i)) atomicAdd(&h[(r - a.index) >> a.lb], 1);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < a.nb; b += kBktThreads)
    if (h[b]) atomicAdd(&a.count[b], h[b]);
}

// Exclusive scan of v over W warps.
template <int W>
__device__ __forceinline__ int block_scan(int v, int* s_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int w = lane < W ? s_warp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += t;
    }
    if (lane < W) s_warp[lane] = w;
  }
  __syncthreads();
  const int base = warp ? s_warp[warp - 1] : 0;
  __syncthreads();
  return base + incl - v;
}

__global__ void __launch_bounds__(kBktThreads) k_bkt_scan(BktArgs a) {
  __shared__ int s_warp[32];
  constexpr int P = kBktMax / kBktThreads;
  int c[P], sum = 0, most = 0;
#pragma unroll
  for (int j = 0; j < P; j++) {
    const int b = threadIdx.x * P + j;
    c[j] = b < a.nb ? a.count[b] : 0;
    sum += c[j];
    most = max(most, c[j]);
  }
  int at = block_scan<kBktThreads / 32>(sum, s_warp);
#pragma unroll
  for (int j = 0; j < P; j++) {
    const int b = threadIdx.x * P + j;
    if (b < a.nb) {
      a.count[b] = at;
      a.cursor[b] = at;
    }
    at += c[j];
  }
  if (most > kBktCap) *a.over = 1;
  if (threadIdx.x == 0) {
    a.count[a.nb] = (int)a.nout;
    a.ptr[a.m] = (int)a.nout;
  }
}

// shared memory of k_bkt_deal: keys and buckets of a tile, and per bucket the
// tile's first place and the distance to its place in global memory
constexpr size_t kDealSmem = kBktTile * (8 + 2) + (2 * kBktMax + 4) * 4;

__global__ void __launch_bounds__(kDealThreads, 2) k_bkt_deal(BktArgs a) {
  extern __shared__ __align__(16) unsigned char s_deal[];
  __shared__ int s_warp[32];
  unsigned long long* skey = reinterpret_cast<unsigned long long*>(s_deal);
  int* loc = reinterpret_cast<int*>(skey + kBktTile);  // [kBktMax + 1]
  int* delta = loc + kBktMax + 4;
  unsigned short* sb = reinterpret_cast<unsigned short*>(delta + kBktMax);
  constexpr int E = kBktTile / kDealThreads, P = kBktMax / kDealThreads;
  const int tid = threadIdx.x;
  if (*a.over) return;
  const long long tiles = (a.nnz + kBktTile - 1) / kBktTile;
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const long long t0 = tile * kBktTile;
    for (int b = tid; b < kBktMax; b += kDealThreads) loc[b] = 0;
    __syncthreads();
    int br[E];  // bucket << 16 | place among the tile's entries of the bucket, or -1
#pragma unroll
    for (int e = 0; e < E; e++) {
      const long long i = t0 + e * kDealThreads + tid;
      br[e] = -1;
      if (i < a.nnz) {
        const int r = __ldg(a.row + i);
        if (!a.sym || r <= __ldg(a.col + i)) br[e] = (r - a.index) >> a.lb;
      }
    }
#pragma unroll
    for (int e = 0; e < E; e++)
      if (br[e] >= 0) br[e] = (br[e] << 16) | atomicAdd(&loc[br[e]], 1);
    __syncthreads();
    int c[P], sum = 0;
#pragma unroll
    for (int j = 0; j < P; j++) {
      c[j] = loc[tid * P + j];
      sum += c[j];
    }
    int at = block_scan<kDealThreads / 32>(sum, s_warp);
#pragma unroll
    for (int j = 0; j < P; j++) {
      loc[tid * P + j] = at;
      at += c[j];
    }
    if (tid == kDealThreads - 1) loc[kBktMax] = at;
    __syncthreads();
    // consecutive threads take consecutive cursors, in every CTA the same way:
    // runs of a bucket that follow one another then meet in L2 while their
    // sector is still open (from a place that differs by CTA: 338 us, not 279)
#pragma unroll
    for (int j = 0; j < P; j++) {
      const int b = j * kDealThreads + tid;
      const int l = loc[b], n = loc[b + 1] - l;
      if (n) delta[b] = atomicAdd(&a.cursor[b], n) - l;
    }
#pragma unroll
    for (int e = 0; e < E; e++)
      if (br[e] >= 0) {
        const long long i = t0 + e * kDealThreads + tid;
        const int r = __ldg(a.row + i) - a.index, cc = __ldg(a.col + i) - a.index;
        const int b = br[e] >> 16, q = loc[b] + (br[e] & 0xffff);
        skey[q] = ((unsigned long long)(r & ((1 << a.lb) - 1)) << (a.cb + a.ib)) |
                  ((unsigned long long)(unsigned)cc << a.ib) | (unsigned long long)i;
        sb[q] = (unsigned short)b;
      }
    __syncthreads();
    const int kept = loc[kBktMax];
#pragma unroll 4
    for (int q = tid; q < kept; q += kDealThreads) a.key[delta[sb[q]] + q] = skey[q];
    __syncthreads();
    double* sval = reinterpret_cast<double*>(skey);
#pragma unroll
    for (int e = 0; e < E; e++)
      if (br[e] >= 0)
        sval[loc[br[e] >> 16] + (br[e] & 0xffff)] = __ldcs(a.val + t0 + e * kDealThreads + tid);
    __syncthreads();
#pragma unroll 4
    for (int q = tid; q < kept; q += kDealThreads) a.kval[delta[sb[q]] + q] = sval[q];
    __syncthreads();
  }
}

constexpr size_t kSortSmem = (size_t)kBktCap * (8 + 8 + 2) + (kBktRows + 4) * 4 + kBktLong * 4;

// Two CTAs per SM: while one waits for its keys or values the other works.
__global__ void __launch_bounds__(kSortThreads, 2) k_bkt_sort(BktArgs a) {
  extern __shared__ __align__(16) unsigned char s_sort[];
  __shared__ int s_warp[32];
  __shared__ int s_nlong;
  unsigned long long* skey = reinterpret_cast<unsigned long long*>(s_sort);
  double* sval = reinterpret_cast<double*>(skey + kBktCap);
  int* off = reinterpret_cast<int*>(sval + kBktCap);  // [rows + 1]
  int* lrow = off + kBktRows + 4;
  unsigned short* place = reinterpret_cast<unsigned short*>(lrow + kBktLong);
  constexpr int NS = kSortThreads, P = kBktRows / NS;
  if (*a.over) return;
  const int tid = threadIdx.x, b = blockIdx.x;
  const int rb = 1 << a.lb, row0 = b << a.lb, rows = min(rb, a.m - row0);
  const int start = __ldg(a.count + b), n = __ldg(a.count + b + 1) - start;
  const int rs = a.cb + a.ib;
  for (int r = tid; r <= rows; r += NS) off[r] = 0;
  if (tid == 0) s_nlong = 0;
  __syncthreads();
#pragma unroll 4
  for (int q = tid; q < n; q += NS)
    place[q] = (unsigned short)atomicAdd(&off[(int)(__ldg(a.key + start + q) >> rs)], 1);
  __syncthreads();
  int c[P], sum = 0;
#pragma unroll
  for (int j = 0; j < P; j++) {
    const int r = tid * P + j;
    c[j] = r < rows ? off[r] : 0;
    sum += c[j];
  }
  int at = block_scan<NS / 32>(sum, s_warp);
#pragma unroll
  for (int j = 0; j < P; j++) {
    const int r = tid * P + j;
    if (r < rows) {
      off[r] = at;
      if (c[j] > kBktRank) {
        const int k = atomicAdd(&s_nlong, 1);
        if (k < kBktLong) lrow[k] = r;
      }
    }
    at += c[j];
  }
  if (tid == NS - 1) off[rows] = n;
  __syncthreads();
  for (int r = tid; r < rows; r += NS) a.ptr[row0 + r] = start + off[r];
#pragma unroll 4
  for (int q = tid; q < n; q += NS) {
    const unsigned long long k = __ldg(a.key + start + q);
    const double v = __ldcs(a.kval + start + q);
    const int p = off[(int)(k >> rs)] + place[q];
    skey[p] = k;
    sval[p] = v;
  }
  __syncthreads();
  const unsigned long long cmask = (1ull << a.cb) - 1ull;
#pragma unroll 4
  for (int q = tid; q < n; q += NS) {
    const unsigned long long k = skey[q];
    const int r = (int)(k >> rs), r0 = off[r], r1 = off[r + 1];
    if (r1 - r0 > kBktRank) continue;
    int f = r0;
    for (int x = r0; x < r1; x++) f += skey[x] < k;
    a.ind[start + f] = (int)((k >> a.ib) & cmask);
    a.vout[start + f] = sval[q];
  }
  // (a bucket holds at most kBktCap / (kBktRank + 1) longer rows)
  static_assert(kBktCap / (kBktRank + 1) < kBktLong, "the list holds every longer row");
  for (int l = 0; l < s_nlong; l++) {
    const int r0 = off[lrow[l]], L = off[lrow[l] + 1] - r0;
    int S = 1;
    while (S < L) S <<= 1;
    // the places past the row hold keys larger than any: with the first step
    // of a merge mirrored, every exchange is ascending and leaves them there
    for (int k = 2; k <= S; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        __syncthreads();
        for (int i = tid; i < S; i += NS) {
          const int y = j == (k >> 1) ? (i ^ (k - 1)) : (i ^ j);
          if (y > i && y < L) {
            const unsigned long long u = skey[r0 + i], w = skey[r0 + y];
            if (u > w) {
              skey[r0 + i] = w;
              skey[r0 + y] = u;
              const double t = sval[r0 + i];
              sval[r0 + i] = sval[r0 + y];
              sval[r0 + y] = t;
            }
          }
        }
      }
    __syncthreads();
    for (int i = tid; i < L; i += NS) {
      a.ind[start + r0 + i] = (int)((skey[r0 + i] >> a.ib) & cmask);
      a.vout[start + r0 + i] = sval[r0 + i];
    }
  }
}

int bits_for(long long v) {  // bits needed to store 0..v
  int b = 0;
  while (v > 0) {
    ++b;
    v >>= 1;
  }
  return b;
}

int excl_scan(int* a, long long n, cudaStream_t s) {
  if (n <= 0) return SB2_OK;
  const long long nb = (n + kScanTile - 1) / kScanTile;
  if (nb > INT_MAX) return SB2_ERR_INVALID_VALUE;
  int* sums = nullptr;
  SB2_CUDA_TRY(pool_malloc((void**)&sums, sizeof(int) * nb, s));
  k_scan_sums<<<(unsigned)nb, kAsmThreads, 0, s>>>(a, n, sums);
  k_scan_top<<<1, 1024, 0, s>>>(sums, (int)nb);
  k_scan_tiles<<<(unsigned)nb, kAsmThreads, 0, s>>>(a, n, sums);
  cudaFreeAsync(sums, s);
  return map_cuda_error(cudaGetLastError());
}

// Stable sort of keys (and positions, when pos is not null) in place over
// the low `bits` bits.
template <typename K>
int radix_sort(K* key, int* pos, long long nnz, int bits, cudaStream_t s) {
  if (nnz <= 1 || bits <= 0) return SB2_OK;
  const long long ntl = (nnz + kTile - 1) / kTile;
  const long long nh = ntl * kBins;
  K* k2 = nullptr;
  int *p2 = nullptr, *hist = nullptr;
  cudaError_t e = pool_malloc((void**)&k2, sizeof(K) * nnz, s);
  if (e == cudaSuccess && pos) e = pool_malloc((void**)&p2, sizeof(int) * nnz, s);
  if (e == cudaSuccess) e = pool_malloc((void**)&hist, sizeof(int) * nh, s);
  int st = map_cuda_error(e);
  K *ka = key, *kb = k2;
  int *pa = pos, *pb = p2;
  for (int shift = 0; st == SB2_OK && shift < bits; shift += 8) {
    k_radix_hist<K><<<(unsigned)ntl, kAsmThreads, 0, s>>>(ka, nnz, (int)ntl, shift, hist);
    st = excl_scan(hist, nh, s);
    if (st != SB2_OK) break;
    k_radix_scatter<K><<<(unsigned)ntl, kAsmThreads, 0, s>>>(ka, pa, nnz, (int)ntl, shift, hist,
                                                             kb, pb);
    std::swap(ka, kb);
    std::swap(pa, pb);
    st = map_cuda_error(cudaGetLastError());
  }
  if (st == SB2_OK && ka != key) {
    e = cudaMemcpyAsync(key, ka, sizeof(K) * nnz, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess && pos)
      e = cudaMemcpyAsync(pos, pa, sizeof(int) * nnz, cudaMemcpyDeviceToDevice, s);
    st = map_cuda_error(e);
  }
  if (k2) cudaFreeAsync(k2, s);
  if (p2) cudaFreeAsync(p2, s);
  if (hist) cudaFreeAsync(hist, s);
  return st;
}

// Shared memory of the two-pass kernels, taken once per device.
cudaError_t bkt_shared_memory() {
  static std::atomic<unsigned long long> taken{0};
  const int dev = current_device();
  const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
  if (bit && (taken.load() & bit)) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(k_bkt_deal, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDealSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_bkt_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSortSmem);
  if (e == cudaSuccess) taken.fetch_or(bit);
  return e;
}

// The two-pass form.  *done false: the triplets do not suit it, or its scratch
// of 16 bytes a triplet is not to be had (the form after it takes 8); the outputs
// are then unfinished.  Synchronizes the stream.
int assemble_buckets(long long nnz, const int* row, const int* col, const double* val, int index,
                     int m, int cb, int sym, long long nout, int* ptr, int* ind, double* vout,
                     cudaStream_t s, bool* done) {
  *done = false;
  if (nout == 0) return SB2_OK;
  const int sms = num_sms(current_device());
  const int ib = bits_for(nnz - 1);
  const double target = std::max(256.0, std::min(4800.0, (double)nout / (2.0 * sms)));
  int lb = 0;
  while (lb < 12 && (2.0 * nout / m) * (double)(1 << lb) <= target) lb++;
  while (lb < 12 && ((long long)m + (1 << lb) - 1) >> lb > kBktMax) lb++;
  const long long nb = ((long long)m + (1 << lb) - 1) >> lb;
  // rows that are mostly too long to be ranked and too short for the bitonic
  // sort: 8M triplets of 500 / 700 / 1000 a row 1119 / 1170 / 1130 us here, 925 / 995 /
  // 1090 row by row; 2M of 500 382 and 421, 8M of 2000 1175 and 1325
  const double mean = (double)nout / m;
  if (mean > kBktRank - 32 && mean < 1024.0 && nout >= 4000000) return SB2_OK;
  if (nb > kBktMax || (double)nout / m * (1 << lb) > 0.9 * kBktCap || lb + cb + ib > 64)
    return SB2_OK;
  BktArgs a{row, col, val, nnz, nout, index, sym, m, lb, cb, ib, (int)nb};
  a.ptr = ptr;
  a.ind = ind;
  a.vout = vout;
  char* buf = nullptr;
  const size_t ints = 2 * (size_t)kBktMax + 64;
  cudaError_t e = pool_malloc((void**)&buf, 16 * (size_t)nout + sizeof(int) * ints, s);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    return SB2_OK;
  }
  SB2_CUDA_TRY(e);
  a.key = reinterpret_cast<unsigned long long*>(buf);
  a.kval = reinterpret_cast<double*>(buf + 8 * (size_t)nout);
  a.count = reinterpret_cast<int*>(buf + 16 * (size_t)nout);
  a.cursor = a.count + kBktMax + 1;
  a.over = a.cursor + kBktMax;
  e = cudaMemsetAsync(a.count, 0, sizeof(int) * ints, s);
  if (e == cudaSuccess) e = bkt_shared_memory();
  int over = 0;
  if (e == cudaSuccess) {
    const long long tiles = (nnz + kBktTile - 1) / kBktTile;
    const int grid = (int)std::min<long long>(tiles, 2LL * sms);
    const int cgrid = (int)std::min<long long>((nnz + kBktThreads - 1) / kBktThreads, 2LL * sms);
    k_bkt_count<<<cgrid, kBktThreads, 0, s>>>(a);
    k_bkt_scan<<<1, kBktThreads, 0, s>>>(a);
    k_bkt_deal<<<grid, kDealThreads, kDealSmem, s>>>(a);
    k_bkt_sort<<<(int)nb, kSortThreads, kSortSmem, s>>>(a);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&over, a.over, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaFreeAsync(buf, s);
  SB2_CUDA_TRY(e);
  *done = over == 0;
  return SB2_OK;
}

int assemble(long long nnz, const int* row, const int* col, const double* val, int index, int m,
             int cb, int sym, long long nout, int* ptr, int* ind, double* vout, cudaStream_t s) {
  const int grid = num_sms(current_device()) * 8;
  SB2_CUDA_TRY(cudaMemsetAsync(ptr, 0, sizeof(int) * ((size_t)m + 1), s));
  if (nout == 0) return SB2_OK;
  const int ib = bits_for(nnz - 1);  // input positions 0..nnz-1
  if (ib + cb > 64) return SB2_ERR_INVALID_VALUE;
  unsigned long long* key = nullptr;
  int *fill = nullptr, *long_rows = nullptr, *nlong = nullptr;
  cudaError_t e = pool_malloc((void**)&key, sizeof(unsigned long long) * nout, s);
  if (e == cudaSuccess) e = pool_malloc((void**)&fill, sizeof(int) * ((size_t)m + 1), s);
  if (e == cudaSuccess) e = pool_malloc((void**)&long_rows, sizeof(int) * ((size_t)m + 1), s);
  if (e == cudaSuccess) e = pool_malloc((void**)&nlong, 2 * sizeof(int), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(nlong, 0, 2 * sizeof(int), s);
  int st = map_cuda_error(e);
  int h_nlong = 0, h_long[2] = {0, 0};  // rows past kShortRow, and past kCtaRow
  std::vector<int> hrows, hptr;
  if (st == SB2_OK) {
    k_row_count<<<grid, kAsmThreads, 0, s>>>(row, col, nnz, index, sym, ptr);
    st = excl_scan(ptr, (long long)m + 1, s);
  }
  if (st == SB2_OK) {
    e = cudaMemcpyAsync(fill, ptr, sizeof(int) * ((size_t)m + 1), cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) {
      k_row_scatter<<<grid, kAsmThreads, 0, s>>>(row, col, nnz, index, sym, ib, fill, key);
      k_row_sort_short<<<grid, kAsmThreads, 0, s>>>(ptr, m, key, ib, val, ind, vout, long_rows,
                                                    nlong);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h_long, nlong, sizeof(h_long), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    st = map_cuda_error(e);
    h_nlong = h_long[0];
  }
  if (st == SB2_OK && h_nlong > 0) {
    k_row_sort_cta<<<h_nlong, kAsmThreads, 0, s>>>(ptr, long_rows, key, ib, val, ind, vout);
    st = map_cuda_error(cudaGetLastError());
  }
  if (st == SB2_OK && h_long[1] > 0) {
    // rows past the CTA sort: each sorted on its own
    hrows.resize(h_nlong);
    hptr.resize((size_t)m + 1);
    e = cudaMemcpyAsync(hrows.data(), long_rows, sizeof(int) * h_nlong, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(hptr.data(), ptr, sizeof(int) * ((size_t)m + 1), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    st = map_cuda_error(e);
    for (int k = 0; st == SB2_OK && k < h_nlong; ++k) {
      const int r = hrows[k];
      const long long b = hptr[r], L = (long long)hptr[r + 1] - b;
      if (L <= kCtaRow) continue;
      st = radix_sort<unsigned long long>(key + b, nullptr, L, ib + cb, s);
      if (st == SB2_OK) {
        const int g = (int)std::min<long long>((L + kAsmThreads - 1) / kAsmThreads, grid);
        k_emit_segment<<<g, kAsmThreads, 0, s>>>(key, b, L, ib, val, ind, vout);
        st = map_cuda_error(cudaGetLastError());
      }
    }
  }
  if (st == SB2_OK) st = map_cuda_error(cudaGetLastError());
  cudaFreeAsync(key, s);
  cudaFreeAsync(fill, s);
  cudaFreeAsync(long_rows, s);
  cudaFreeAsync(nlong, s);
  return st;
}

}  // namespace
}  // namespace sb2

using namespace sb2;

extern "C" {

int sb2_coo_to_csr(int nnz, const int* row, const int* col, const double* val, int index,
                   int m_min, int n_min, int symmetric_upper, void* stream, int* m_out,
                   int* n_out, int* nnz_out, int** ptr, int** ind, double** val_out) try {
  SB2_TRACE("sb2_coo_to_csr");
  if (nnz < 0 || m_min < 0 || n_min < 0 || !m_out || !n_out || !nnz_out || !ptr || !ind ||
      !val_out)
    return SB2_ERR_INVALID_VALUE;
  if (nnz > 0 && (!row || !col || !val)) return SB2_ERR_INVALID_VALUE;
  *ptr = nullptr;
  *ind = nullptr;
  *val_out = nullptr;
  cudaStream_t s = static_cast<cudaStream_t>(stream);

  CooStats h = {};
  if (nnz > 0) {
    CooStats* d = nullptr;
    SB2_CUDA_TRY(pool_malloc((void**)&d, sizeof(CooStats), s));
    cudaError_t e = cudaMemsetAsync(d, 0, sizeof(CooStats), s);
    if (e == cudaSuccess) {
      const long long want = (nnz + kAsmThreads - 1) / kAsmThreads;
      const int grid = (int)std::min<long long>(want, num_sms(current_device()) * 8LL);
      k_coo_stats<<<grid, kAsmThreads, 0, s>>>(row, col, nnz, index, d);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d, sizeof(CooStats), cudaMemcpyDeviceToHost, s);
    cudaFreeAsync(d, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    SB2_CUDA_TRY(e);
    if (h.bad) return SB2_ERR_INVALID_VALUE;
  }

  // Sizes as ConvertMatrix_from_Coordinates sets them: RowSparse takes
  // max(largest index + 1, current size) and is at least 1 x 1 (the norm of
  // an empty index vector is 0); RowSymSparse is (largest row + 1) square,
  // and an empty input leaves the m_min x m_min matrix unchanged.
  long long m, n, nout;
  if (symmetric_upper) {
    m = nnz > 0 ? (long long)h.row_max + 1 : m_min;
    n = m;
    nout = h.kept;
  } else {
    m = std::max<long long>((long long)h.row_max + 1, m_min);
    n = std::max<long long>((long long)h.col_max + 1, n_min);
    nout = nnz;
  }
  if (m >= INT_MAX || n >= INT_MAX) return SB2_ERR_INVALID_VALUE;
  const int cb = bits_for(nnz > 0 ? h.col_max : 0);  // columns 0..max(col)

  int *dp = nullptr, *di = nullptr;
  double* dv = nullptr;
  cudaError_t e = pool_malloc_owned((void**)&dp, sizeof(int) * (m + 1), s);
  if (e == cudaSuccess && nout > 0) e = pool_malloc_owned((void**)&di, sizeof(int) * nout, s);
  if (e == cudaSuccess && nout > 0) e = pool_malloc_owned((void**)&dv, sizeof(double) * nout, s);
  int st = map_cuda_error(e);
  bool done = false;
  if (st == SB2_OK && nnz > 0 && !h.unsorted && nout == nnz) {
    const int grid = (int)std::min<long long>((nnz + kAsmThreads - 1) / kAsmThreads,
                                              num_sms(current_device()) * 8LL);
    if (std::max<long long>(h.gap, m - h.row_max) > kGapRows) {
      k_coo_sorted<true><<<grid, kAsmThreads, 0, s>>>(row, col, val, nnz, index, (int)m, dp, di, dv);
      const int rgrid =
          (int)std::min<long long>((m + kAsmThreads) / kAsmThreads, num_sms(current_device()) * 8LL);
      k_coo_rows<<<rgrid, kAsmThreads, 0, s>>>(row, nnz, index, (int)m, dp);
    } else {
      k_coo_sorted<false><<<grid, kAsmThreads, 0, s>>>(row, col, val, nnz, index, (int)m, dp, di, dv);
    }
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    st = map_cuda_error(e);
    done = true;
  }
  if (st == SB2_OK && !done)
    st = assemble_buckets(nnz, row, col, val, index, (int)m, cb, symmetric_upper, nout, dp, di, dv, s,
                          &done);
  if (st == SB2_OK && !done)
    st = assemble(nnz, row, col, val, index, (int)m, cb, symmetric_upper, nout, dp, di, dv, s);
  if (st == SB2_OK && !done) st = map_cuda_error(cudaStreamSynchronize(s));
  if (st != SB2_OK) {
    sb2_device_free(dp);
    sb2_device_free(di);
    sb2_device_free(dv);
    return st;
  }
  *m_out = (int)m;
  *n_out = (int)n;
  *nnz_out = (int)nout;
  *ptr = dp;
  *ind = di;
  *val_out = dv;
  return SB2_OK;
} SB2_CATCH

}  // extern "C"
