// Stable LSD radix sort of (64- or 32-bit key, int32 value) pairs, the COO ->
// CSR ordering and the column sums in entry order built on it.
//
// Replaces the ordering step of tbsla::cpp::MatrixCSR(const MatrixCOO&)
// (src/cpp/matrix/MatrixCSR.cpp:49-96 with compare_row,
// src/cpp/utils/csr.cpp:3-8): entries ordered by (row, column), ties kept
// in storage order.  The reference sorts a permutation with std::sort on
// the host; here the key (row << column bits | column) is sorted on the
// GPU with 8-bit digits, stable pass by pass, so equal keys keep their
// storage order and the permutation equals the host's stable sort exactly.
//
// One pass = per-tile digit histograms (tiles of 4096 keys), an exclusive
// scan of the histograms in digit-major order (global output offsets), and
// a stable scatter: each tile walks its keys in index order 256 at a time;
// lanes with the same digit find each other with __match_any_sync, and the
// per-warp counts in shared memory give every key its place after the
// earlier warps and rounds of its tile.
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "kernels.hpp"

namespace tbsla_gpu {

namespace {

constexpr int RT = 256;
constexpr int TILE = 4096;
constexpr int RADIX = 256;
constexpr int SCAN_CHUNK = 2048;  // elements per CTA in the scan (8 per thread)
constexpr unsigned FULL = 0xffffffffu;

template <class K>
__global__ void __launch_bounds__(RT) k_hist(const K* __restrict__ keys, long n, int shift, int ntiles,
                                            unsigned* __restrict__ hist) {
  __shared__ unsigned h[RADIX];
  for (int d = threadIdx.x; d < RADIX; d += RT) h[d] = 0;
  __syncthreads();
  const long base = (long)blockIdx.x * TILE;
  for (int k = threadIdx.x; k < TILE; k += RT) {
    const long i = base + k;
    if (i < n) atomicAdd(&h[(keys[i] >> shift) & (RADIX - 1)], 1u);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < RADIX; d += RT) hist[(long)d * ntiles + blockIdx.x] = h[d];
}

template <class K>
__global__ void __launch_bounds__(RT) k_scatter(const K* __restrict__ keys, const int* __restrict__ vals,
                                               K* __restrict__ okeys, int* __restrict__ ovals, long n,
                                               int shift, int ntiles, const unsigned* __restrict__ offs) {
  __shared__ unsigned base[RADIX];
  __shared__ unsigned wcnt[RT / kWarp][RADIX];
  const int lane = threadIdx.x & 31, warp = threadIdx.x / kWarp;
  for (int d = threadIdx.x; d < RADIX; d += RT) base[d] = offs[(long)d * ntiles + blockIdx.x];
  const long t0 = (long)blockIdx.x * TILE;
  const unsigned lt = (1u << lane) - 1u;
  for (int r = 0; r < TILE / RT; r++) {
    for (int d = lane; d < RADIX; d += kWarp) wcnt[warp][d] = 0;
    __syncthreads();
    const long i = t0 + (long)r * RT + threadIdx.x;
    const bool valid = i < n;
    const K key = valid ? keys[i] : 0;
    const int dg = valid ? (int)((key >> shift) & (RADIX - 1)) : RADIX;  // RADIX: no key
    const unsigned peers = __match_any_sync(FULL, dg);
    const int rank = __popc(peers & lt);
    if (valid && rank == 0) wcnt[warp][dg] = __popc(peers);
    __syncthreads();
    if (valid) {
      unsigned p = base[dg] + rank;
      for (int w = 0; w < warp; w++) p += wcnt[w][dg];
      okeys[p] = key;
      ovals[p] = vals[i];
    }
    __syncthreads();
    for (int d = threadIdx.x; d < RADIX; d += RT) {
      unsigned s = 0;
      for (int w = 0; w < RT / kWarp; w++) s += wcnt[w][d];
      base[d] += s;
    }
    __syncthreads();
  }
}

// In-place exclusive scan of each SCAN_CHUNK-element chunk; chunk totals to
// sums[blockIdx.x].
__global__ void __launch_bounds__(RT) k_scan_chunks(unsigned* __restrict__ a, long n, unsigned* __restrict__ sums) {
  __shared__ unsigned ws[RT / kWarp];
  const long c0 = (long)blockIdx.x * SCAN_CHUNK;
  constexpr int PER = SCAN_CHUNK / RT;
  unsigned v[PER];
  unsigned t = 0;
#pragma unroll
  for (int k = 0; k < PER; k++) {
    const long i = c0 + (long)threadIdx.x * PER + k;
    v[k] = i < n ? a[i] : 0u;
    t += v[k];
  }
  // exclusive scan of the per-thread totals over the CTA
  const int lane = threadIdx.x & 31, warp = threadIdx.x / kWarp;
  unsigned incl = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) ws[warp] = incl;
  __syncthreads();
  unsigned wpre = 0;
  for (int w = 0; w < warp; w++) wpre += ws[w];
  unsigned run = wpre + incl - t;
#pragma unroll
  for (int k = 0; k < PER; k++) {
    const long i = c0 + (long)threadIdx.x * PER + k;
    if (i < n) a[i] = run;
    run += v[k];
  }
  if (threadIdx.x == RT - 1) sums[blockIdx.x] = run;
}

__global__ void k_scan_add(unsigned* __restrict__ a, long n, const unsigned* __restrict__ sums) {
  const long i = (long)blockIdx.x * SCAN_CHUNK + threadIdx.x;
  const unsigned add = sums[blockIdx.x];
  for (long k = i; k < std::min(n, (long)(blockIdx.x + 1) * SCAN_CHUNK); k += RT) a[k] += add;
}

__global__ void k_keys(const int* __restrict__ row, const int* __restrict__ col, long n, int cbits,
                       uint64_t* __restrict__ keys, int* __restrict__ idx) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    keys[i] = ((uint64_t)(unsigned)row[i] << cbits) | (unsigned)col[i];
    idx[i] = (int)i;
  }
}

__global__ void k_count_rows(const int* __restrict__ row, long n, unsigned* __restrict__ cnt) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    atomicAdd(cnt + row[i], 1u);
}

int grid_for(long n) { return (int)std::max<long>(1, std::min<long>((n + RT - 1) / RT, 152L * 32)); }

}  // namespace

// Exclusive scan of a[0..n) in place; scratch: at least scan_scratch(n) words.
long scan_scratch(long n) {
  long s = 0;
  while (n > 1) {
    n = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
    s += n;
  }
  return s + 1;
}

cudaError_t exclusive_scan(unsigned* a, long n, unsigned* scratch, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const long nb = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
  k_scan_chunks<<<(unsigned)nb, RT, 0, s>>>(a, n, scratch);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || nb == 1) return e;
  e = exclusive_scan(scratch, nb, scratch + nb, s);
  if (e != cudaSuccess) return e;
  k_scan_add<<<(unsigned)nb, RT, 0, s>>>(a, n, scratch);
  return cudaGetLastError();
}

long radix_scratch(long n) {
  const long ntiles = (n + TILE - 1) / TILE;
  return (long)RADIX * ntiles + scan_scratch((long)RADIX * ntiles);
}

namespace {
template <class K>
cudaError_t sort_pairs(K* keys, K* keys_alt, int* vals, int* vals_alt, long n, int bits, unsigned* scratch,
                       int* result_in_alt, cudaStream_t s) {
  *result_in_alt = 0;
  if (n <= 1) return cudaSuccess;
  const long ntiles = (n + TILE - 1) / TILE;
  unsigned* hist = scratch;
  unsigned* sc = scratch + RADIX * ntiles;
  int flip = 0;
  for (int shift = 0; shift < bits; shift += 8) {
    const K* ki = flip ? keys_alt : keys;
    K* ko = flip ? keys : keys_alt;
    const int* vi = flip ? vals_alt : vals;
    int* vo = flip ? vals : vals_alt;
    k_hist<<<(unsigned)ntiles, RT, 0, s>>>(ki, n, shift, (int)ntiles, hist);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = exclusive_scan(hist, (long)RADIX * ntiles, sc, s);
    if (e != cudaSuccess) return e;
    k_scatter<<<(unsigned)ntiles, RT, 0, s>>>(ki, vi, ko, vo, n, shift, (int)ntiles, hist);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    flip ^= 1;
  }
  *result_in_alt = flip;
  return cudaSuccess;
}

// 32-bit keys (columns) and their entries' indices, in entry order.
__global__ void k_column_keys(const int* __restrict__ colidx, long n, int f_col, unsigned* __restrict__ keys,
                              int* __restrict__ idx) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    keys[i] = (unsigned)(colidx[i] - f_col);
    idx[i] = (int)i;
  }
}

// start[c]: the first of the sorted keys that is c or more (c <= n_col).  A
// binary search per column: a thread per key that fills the columns up to it
// leaves a run of empty columns to one thread (2^22 columns, the first 1000
// used: 24.5 -> 10.5 ms of a first solve).
__global__ void k_column_starts(const unsigned* __restrict__ keys, long n, int n_col, int* __restrict__ start) {
  for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c <= n_col; c += (long)gridDim.x * blockDim.x) {
    long lo = 0, hi = n;
    while (lo < hi) {
      const long mid = (lo + hi) >> 1;
      if ((long)keys[mid] < c) lo = mid + 1;
      else hi = mid;
    }
    start[c] = (int)lo;
  }
}

// w[c] = sum of column c's values, added one by one in entry order from 0 (the
// order of a loop over the entries, so the same bits).  A lane per column here;
// columns of more than kLaneColumn entries go to list (lens[0]: how many,
// lens[1]: the longest's entries), 0 for now.
constexpr int kLaneColumn = 64;
template <class V>
__global__ void __launch_bounds__(RT) k_column_sums_short(const V* __restrict__ vals, const int* __restrict__ perm,
                                                         const int* __restrict__ start, int n_col,
                                                         double* __restrict__ w, int* __restrict__ list,
                                                         int* __restrict__ lens) {
  const int lane = threadIdx.x & 31;
  int most = 0;
  for (long c0 = (blockIdx.x * (long)RT + threadIdx.x) / kWarp * kWarp; c0 < n_col; c0 += (long)gridDim.x * RT) {
    const long c = c0 + lane;
    const int a = c < n_col ? start[c] : 0, e = c < n_col ? start[c + 1] : 0;
    const bool is_long = e - a > kLaneColumn;
    double sum = 0.0;
    if (!is_long) {
      int t = a;
      for (; t + 4 <= e; t += 4) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = widen(vals[perm[t + u]]);
#pragma unroll
        for (int u = 0; u < 4; u++) sum = add_rn(sum, v[u]);
      }
      for (; t < e; t++) sum = add_rn(sum, widen(vals[perm[t]]));
    } else {
      list[atomicAdd(lens, 1)] = (int)c;
      most = max(most, e - a);
    }
    if (c < n_col) w[c] = sum;
  }
  most = __reduce_max_sync(FULL, most);
  if (lane == 0 && most > 0) atomicMax(lens + 1, most);
}

// The listed columns of at most `most` entries, a warp each (columns of a list,
// not of the matrix: neighbours in the numbering may all be long): 32 values
// loaded at once, added in order by shuffles.
template <class V>
__global__ void __launch_bounds__(RT) k_column_sums_long(const V* __restrict__ vals, const int* __restrict__ perm,
                                                        const int* __restrict__ start, const int* __restrict__ list,
                                                        int count, int most, double* __restrict__ w) {
  const int lane = threadIdx.x & 31;
  for (int k = (blockIdx.x * RT + threadIdx.x) / kWarp; k < count; k += gridDim.x * (RT / kWarp)) {
    const int c = list[k], la = start[c], le = start[c + 1];
    if (le - la > most) continue;
    double s = 0.0, v = la + lane < le ? widen(vals[perm[la + lane]]) : 0.0;
    for (int t = la; t < le; t += kWarp) {
      const int next = t + kWarp + lane;
      const double vn = next < le ? widen(vals[perm[next]]) : 0.0;
      const int m = min(kWarp, le - t);
      if (m == kWarp) {
#pragma unroll
        for (int u = 0; u < kWarp; u++) s = add_rn(s, __shfl_sync(FULL, v, u));
      } else {
        for (int u = 0; u < m; u++) s = add_rn(s, __shfl_sync(FULL, v, u));
      }
      v = vn;
    }
    if (lane == 0) w[c] = s;
  }
}

// The listed columns of more than `over` entries: found[0] of them, then
// (column, first sorted entry, entries) each, the first kMostHubs of them.
constexpr int kMostHubs = 256;
__global__ void k_long_columns(const int* __restrict__ start, const int* __restrict__ list, int count, int over,
                               int* __restrict__ found) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
    const int c = list[k], a = start[c], len = start[c + 1] - a;
    if (len <= over) continue;
    const int at = atomicAdd(found, 1);
    if (at >= kMostHubs) continue;
    found[1 + 3 * at] = c;
    found[2 + 3 * at] = a;
    found[3 + 3 * at] = len;
  }
}

// Columns that the caller adds up on the host, longest first.  On the device a
// column is a chain of dependent FP64 additions, 46 ns an entry, on the host 1
// to 3; the device's columns run side by side, the host's one after another.  So
// the longest ones go to the host as long as all that it takes so far costs it
// less than the shortest of them costs the device (2^20 nodes, 200,000 entries
// and one column of 10^6: first solve 47.7 -> 2.2 ms more than the next; 32
// neighbouring columns of 100,000, on one warp before the list: 152 -> 9.0).  More than kMostHubs columns within the
// ratio of the longest are work enough for the device's many warps.
constexpr int kHubMin = 4096, kHubRatio = 12;
cudaError_t choose_hubs(const int* start, const int* list, int count, int longest, int* found,
                        std::vector<ColumnRange>* hubs, cudaStream_t s) {
  hubs->clear();
  if (longest <= kHubMin) return cudaSuccess;
  std::vector<int> h(1 + 3 * kMostHubs);
  cudaError_t e = cudaMemsetAsync(found, 0, sizeof(int), s);
  if (e != cudaSuccess) return e;
  k_long_columns<<<grid_for(count), RT, 0, s>>>(start, list, count, std::max(kHubMin, longest / kHubRatio), found);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), found, h.size() * sizeof(int), cudaMemcpyDeviceToHost, s);
  const cudaError_t w = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = w;
  if (e != cudaSuccess || h[0] > kMostHubs) return e;
  for (int k = 0; k < h[0]; k++) hubs->push_back({h[1 + 3 * k], h[2 + 3 * k], h[3 + 3 * k]});
  std::sort(hubs->begin(), hubs->end(), [](const ColumnRange& a, const ColumnRange& b) {
    return a.len != b.len ? a.len > b.len : a.col < b.col;
  });
  long taken = 0;
  size_t k = 0;
  while (k < hubs->size() && taken + (*hubs)[k].len < (long)kHubRatio * (*hubs)[k].len) taken += (*hubs)[k++].len;
  while (k > 0 && k < hubs->size() && (*hubs)[k].len == (*hubs)[k - 1].len) k--;  // the device skips by length
  hubs->resize(k);
  return cudaSuccess;
}

template <class V>
cudaError_t column_sums(const V* vals, const int* perm, const int* start, int n_col, int* list, int* found, double* w,
                        std::vector<ColumnRange>* hubs, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(found, 0, 2 * sizeof(int), s);
  if (e != cudaSuccess) return e;
  k_column_sums_short<<<grid_for(n_col), RT, 0, s>>>(vals, perm, start, n_col, w, list, found);
  e = cudaGetLastError();
  int lens[2] = {0, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(lens, found, sizeof lens, cudaMemcpyDeviceToHost, s);
  const cudaError_t done = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = done;
  if (e != cudaSuccess || lens[0] == 0) return e;
  e = choose_hubs(start, list, lens[0], lens[1], found, hubs, s);
  if (e != cudaSuccess) return e;
  const int most = hubs->empty() ? lens[1] : hubs->back().len - 1;
  k_column_sums_long<<<grid_for((long)lens[0] * kWarp), RT, 0, s>>>(vals, perm, start, list, lens[0], most, w);
  return cudaGetLastError();
}
}  // namespace

cudaError_t radix_sort_pairs(uint64_t* keys, uint64_t* keys_alt, int* vals, int* vals_alt, long n, int bits,
                             unsigned* scratch, int* result_in_alt, cudaStream_t s) {
  return sort_pairs(keys, keys_alt, vals, vals_alt, n, bits, scratch, result_in_alt, s);
}

long column_sums_scratch(long n, int n_col) {
  return 4 * n + n_col + 1 + radix_scratch(n) + n / kLaneColumn + 1 + 1 + 3 * kMostHubs;
}

cudaError_t column_sums_ordered(const void* vals, int prec, const int* colidx, long n, int f_col, int n_col,
                                unsigned* scratch, double* w, const int** sorted, std::vector<ColumnRange>* hubs,
                                cudaStream_t s) {
  hubs->clear();
  if (n_col <= 0) return cudaSuccess;
  unsigned *keys = scratch, *alt = keys + n;
  int *perm = reinterpret_cast<int*>(alt + n), *perm_alt = perm + n, *start = perm_alt + n;
  unsigned* radix = reinterpret_cast<unsigned*>(start + n_col + 1);
  int* list = reinterpret_cast<int*>(radix + radix_scratch(n));
  int* found = list + n / kLaneColumn + 1;
  int bits = 0, in_alt = 0;
  while (bits < 31 && (1L << bits) < (long)n_col) bits++;
  if (n > 0) k_column_keys<<<grid_for(n), RT, 0, s>>>(colidx, n, f_col, keys, perm);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = sort_pairs(keys, alt, perm, perm_alt, n, bits, radix, &in_alt, s);
  if (e != cudaSuccess) return e;
  const int* p = in_alt ? perm_alt : perm;
  *sorted = p;
  k_column_starts<<<grid_for((long)n_col + 1), RT, 0, s>>>(in_alt ? alt : keys, n, n_col, start);
  switch (prec) {
    case kF64: return column_sums(static_cast<const double*>(vals), p, start, n_col, list, found, w, hubs, s);
    case kF32: return column_sums(static_cast<const float*>(vals), p, start, n_col, list, found, w, hubs, s);
    case kBF16: return column_sums(static_cast<const __nv_bfloat16*>(vals), p, start, n_col, list, found, w, hubs, s);
  }
  return cudaErrorInvalidValue;
}

// COO -> DENSE (MatrixDENSE.cpp:15-37): the entries in (row, column) order,
// ties in storage order, so each run of one position sums its values in the
// reference's order (starting from 0), written once; a thread per sorted
// entry, the first of a run does the run.
__global__ void k_dense_scatter(const int* __restrict__ perm, const int* __restrict__ row,
                                const int* __restrict__ col, const double* __restrict__ val, long n, long ln_col,
                                double* __restrict__ dense) {
  for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) {
    const int p = perm[k];
    const int r = row[p], c = col[p];
    if (k > 0) {
      const int q = perm[k - 1];
      if (row[q] == r && col[q] == c) continue;  // inside a run
    }
    double sum = 0.0;
    for (long t = k; t < n; t++) {
      const int u = perm[t];
      if (row[u] != r || col[u] != c) break;
      sum = __dadd_rn(sum, val[u]);
    }
    dense[(size_t)r * ln_col + c] = sum;
  }
}

cudaError_t coo_dense_scatter(const int* perm, const int* row, const int* col, const double* val, long n,
                              long ln_col, double* dense, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_dense_scatter<<<grid_for(n), RT, 0, s>>>(perm, row, col, val, n, ln_col, dense);
  return cudaGetLastError();
}

cudaError_t coo_order(const int* row, const int* col, long n, int n_row, int n_col, uint64_t* keys,
                      uint64_t* keys_alt, int* perm, int* perm_alt, unsigned* rowcount, unsigned* scratch,
                      int* perm_in_alt, cudaStream_t s) {
  int rbits = 0, cbits = 0;
  while (rbits < 31 && (1L << rbits) < (long)n_row) rbits++;
  while (cbits < 31 && (1L << cbits) < (long)n_col) cbits++;
  cudaError_t e = cudaMemsetAsync(rowcount, 0, ((size_t)n_row + 1) * sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  if (n > 0) {
    k_keys<<<grid_for(n), RT, 0, s>>>(row, col, n, cbits, keys, perm);
    k_count_rows<<<grid_for(n), RT, 0, s>>>(row, n, rowcount);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  e = exclusive_scan(rowcount, (long)n_row + 1, scratch, s);  // row starts
  if (e != cudaSuccess) return e;
  return radix_sort_pairs(keys, keys_alt, perm, perm_alt, n, rbits + cbits, scratch, perm_in_alt, s);
}

}  // namespace tbsla_gpu
