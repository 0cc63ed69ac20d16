// rowsort.cu -- triplets into row order by buckets: the order a stable sort on
// (row, column) gives, with one scatter instead of a radix sort's passes.
//
// The rows of these systems are short (a vertex has some 15 neighbours, a raw
// row some 60 triplets), so the entries are counted per row, scattered to their
// row's bucket (in whatever order the atomics give) and each bucket is sorted
// by (column, input position) in registers: the position makes every key
// unique and the result the stable order.  At 64-bit keys a radix sort of n
// pairs reads and writes them once per 8 key bits, five times for 262,144 rows.
// Merging the 110,592-row system's triplets went from 0.92 to 0.64 ms, building
// the 262,144-row matrix from 0.87 to 0.68, the 8,000-row one from 0.25 to 0.20.
// Rows longer than kRowMost, or more rows than the triplets justify, keep the
// radix sort (the callers fall back when these functions return false).
#include <algorithm>

#include <cub/device/device_scan.cuh>

#include "maspcg_internal.cuh"

namespace maspcg {
namespace {

constexpr int kTpb = 256;
constexpr int kRowMost = 1024;  // entries of a row one warp sorts in registers (32 per lane)

// flags: [0] entries out of range, [1] longest row.
template <bool kSym>
__global__ void __launch_bounds__(kTpb) k_bucket_count(const int* __restrict__ rows, const int* __restrict__ cols, int n,
                                                      int nb, const int* __restrict__ map, int* count, int* rank,
                                                      int* flags)
{
  const int i = blockIdx.x * kTpb + threadIdx.x;
  if (i >= n) return;
  int r = rows[i], c = cols[i];
  if constexpr (kSym) {
    rank[2 * (size_t)i] = rank[2 * (size_t)i + 1] = -1;
    if ((unsigned)r >= (unsigned)nb || (unsigned)c >= (unsigned)nb) {
      atomicAdd(flags, 1);
      return;
    }
    r = __ldg(map + r);
    c = __ldg(map + c);
    rank[2 * (size_t)i] = atomicAdd(count + r, 1);
    if (r != c) rank[2 * (size_t)i + 1] = atomicAdd(count + c, 1);
  } else {
    rank[i] = atomicAdd(count + r, 1);
  }
}

__global__ void __launch_bounds__(kTpb) k_bucket_most(const int* __restrict__ count, int nrows, int* flags)
{
  __shared__ unsigned most[kTpb / 32];
  unsigned m = 0;
  for (int i = blockIdx.x * kTpb + threadIdx.x; i < nrows; i += gridDim.x * kTpb) m = max(m, (unsigned)count[i]);
  m = __reduce_max_sync(kFull, m);
  if ((threadIdx.x & 31) == 0) most[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kTpb / 32; ++w) m = max(m, most[w]);
    atomicMax(flags + 1, (int)m);
  }
}

// Entry: column in the high word, input position in the low one (kSym: the
// triplet in the upper 31 bits, bit 0 its mirror A_cr = H^T).
template <bool kSym>
__global__ void __launch_bounds__(kTpb) k_bucket_scatter(const int* __restrict__ rows, const int* __restrict__ cols,
                                                        int n, const int* __restrict__ map,
                                                        const int* __restrict__ start, const int* __restrict__ rank,
                                                        unsigned long long* entries)
{
  const int i = blockIdx.x * kTpb + threadIdx.x;
  if (i >= n) return;
  int r = rows[i], c = cols[i];
  if constexpr (kSym) {
    r = __ldg(map + r);
    c = __ldg(map + c);
    const int2 k = reinterpret_cast<const int2*>(rank)[i];
    entries[start[r] + k.x] = ((unsigned long long)(unsigned)c << 32) | (2u * (unsigned)i);
    if (k.y >= 0) entries[start[c] + k.y] = ((unsigned long long)(unsigned)r << 32) | (2u * (unsigned)i + 1u);
  } else {
    entries[start[r] + rank[i]] = ((unsigned long long)(unsigned)c << 32) | (unsigned)i;
  }
}

// Bitonic sort of 32 kE keys of a warp, element 32 e + lane in k[e].
template <int kE>
__device__ __forceinline__ void warp_sort(unsigned long long k[kE], int lane)
{
#pragma unroll
  for (int size = 2; size <= 32 * kE; size *= 2)
#pragma unroll
    for (int d = size / 2; d > 0; d /= 2) {
      if (d >= 32) {
#pragma unroll
        for (int e = 0; e < kE; ++e) {
          const int f = e ^ (d / 32);
          if (f > e) {
            const bool up = ((32 * e) & size) == 0;
            const unsigned long long a = k[e], b = k[f];
            if ((a > b) == up) k[e] = b, k[f] = a;
          }
        }
      } else {
#pragma unroll
        for (int e = 0; e < kE; ++e) {
          const unsigned long long o = __shfl_xor_sync(kFull, k[e], d);
          const bool up = ((32 * e + lane) & size) == 0, low = (lane & d) == 0;
          if ((k[e] > o) == (up == low)) k[e] = o;
        }
      }
    }
}

// Sorts a bucket in place and returns its distinct columns.
template <int kE>
__device__ __forceinline__ int sort_bucket(unsigned long long* entries, int n, int lane)
{
  unsigned long long k[kE];
#pragma unroll
  for (int e = 0; e < kE; ++e) k[e] = 32 * e + lane < n ? entries[32 * e + lane] : ~0ull;
  warp_sort<kE>(k, lane);
  int distinct = 0;
  unsigned last = 0xffffffffu;  // column of the element before lane 0's (columns are below 2^31)
#pragma unroll
  for (int e = 0; e < kE; ++e) {
    const unsigned c = (unsigned)(k[e] >> 32);
    unsigned before = __shfl_up_sync(kFull, c, 1);
    if (lane == 0) before = last;
    last = __shfl_sync(kFull, c, 31);
    const bool in = 32 * e + lane < n;
    distinct += __popc(__ballot_sync(kFull, in && c != before));
    if (in) entries[32 * e + lane] = k[e];
  }
  return distinct;
}

__global__ void __launch_bounds__(kTpb) k_bucket_sort(const int* __restrict__ start, int nrows,
                                                     unsigned long long* entries, int* distinct)
{
  const int row = (blockIdx.x * kTpb + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (row > nrows) return;  // whole warp
  if (row == nrows) {       // the scan's extra entry
    if (lane == 0) distinct[row] = 0;
    return;
  }
  const int s = start[row], n = start[row + 1] - s;
  int u = 0;
  if (n > 512)
    u = sort_bucket<32>(entries + s, n, lane);
  else if (n > 256)
    u = sort_bucket<16>(entries + s, n, lane);
  else if (n > 128)
    u = sort_bucket<8>(entries + s, n, lane);
  else if (n > 64)
    u = sort_bucket<4>(entries + s, n, lane);
  else if (n > 32)
    u = sort_bucket<2>(entries + s, n, lane);
  else if (n > 0)
    u = sort_bucket<1>(entries + s, n, lane);
  if (lane == 0) distinct[row] = u;
}

// The distinct blocks of every row: column (and row), first entry; the input
// position of every entry.
__global__ void __launch_bounds__(kTpb) k_bucket_fill(const int* __restrict__ start, const int* __restrict__ uptr,
                                                     int nrows, const unsigned long long* __restrict__ entries,
                                                     int* urow, int* ucol, int* seg_start, int* position)
{
  const int row = (blockIdx.x * kTpb + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (row >= nrows) return;  // whole warp
  const int s = start[row], n = start[row + 1] - s;
  int u = uptr[row];
  unsigned last = 0xffffffffu;
  for (int j = 0; j < n; j += 32) {
    const bool in = j + lane < n;
    const unsigned long long k = in ? entries[s + j + lane] : ~0ull;
    const unsigned c = (unsigned)(k >> 32);
    unsigned before = __shfl_up_sync(kFull, c, 1);
    if (lane == 0) before = last;
    last = __shfl_sync(kFull, c, 31);
    const unsigned heads = __ballot_sync(kFull, in && c != before);
    if (in) position[s + j + lane] = (int)(unsigned)k;
    if ((heads >> lane) & 1u) {
      const int at = u + __popc(heads & ((1u << lane) - 1u));
      if (urow) urow[at] = row;
      ucol[at] = (int)c;
      seg_start[at] = s + j + lane;
    }
    u += __popc(heads);
  }
}

// Counts, longest row, scatter, sort, distinct offsets (uptr, nrows + 1).
// False: leave it to the radix sort (nothing but scratch has been written).
template <bool kSym>
bool bucket(maspcg_handle* h, const int* rows, const int* cols, int n, int nrows, int nb, const int* map,
            unsigned long long* entries, int* rank, int* start, int* uptr, int* flags, int flags_host[2])
{
  cudaStream_t st = h->stream;
  h->row_count.resize((size_t)nrows + 1);
  int* count = h->row_count.get();
  MCK(cudaMemsetAsync(count, 0, sizeof(int) * ((size_t)nrows + 1), st));
  MCK(cudaMemsetAsync(flags, 0, 2 * sizeof(int), st));
  const int grid = ceil_div(n, kTpb);
  k_bucket_count<kSym><<<grid, kTpb, 0, st>>>(rows, cols, n, nb, map, count, rank, flags); MLAUNCHED(h);
  k_bucket_most<<<std::min(ceil_div(nrows, kTpb), 4 * h->sm_count), kTpb, 0, st>>>(count, nrows, flags); MLAUNCHED(h);
  size_t need = 0;
  MCK(cub::DeviceScan::ExclusiveSum(nullptr, need, count, start, nrows + 1, st));
  h->cub_tmp.resize(std::max(need, h->cub_tmp.n));
  size_t tb = h->cub_tmp.cap;
  MCK(cub::DeviceScan::ExclusiveSum(h->cub_tmp.get(), tb, count, start, nrows + 1, st));
  MCK(cudaMemcpyAsync(flags_host, flags, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
  if (flags_host[0] != 0 || flags_host[1] > kRowMost) return false;
  k_bucket_scatter<kSym><<<grid, kTpb, 0, st>>>(rows, cols, n, map, start, rank, entries); MLAUNCHED(h);
  k_bucket_sort<<<ceil_div(32LL * (nrows + 1LL), kTpb), kTpb, 0, st>>>(start, nrows, entries, count); MLAUNCHED(h);
  tb = h->cub_tmp.cap;
  MCK(cub::DeviceScan::ExclusiveSum(h->cub_tmp.get(), tb, count, uptr, nrows + 1, st));
  MCK(cudaGetLastError());
  return true;
}

}  // namespace

bool row_sort_matrix(maspcg_handle* h, const int* rows, const int* cols, int n)
{
  cudaStream_t st = h->stream;
  h->row_start.resize((size_t)h->nb_int + 1);
  int flags[2] = {0, 0};
  const bool ok = bucket<true>(h, rows, cols, n, h->nb_int, h->nb, h->int_of_row.get(), h->keys.get(), h->kv.get(),
                               h->row_start.get(), h->rowptr.get(), h->failed.get(), flags);
  MREQ(flags[0] == 0, MASPCG_ERR_INVALID_ARGUMENT, "matrix block index out of range");
  if (!ok) return false;
  MCK(cudaMemsetAsync(h->failed.get(), 0, 2 * sizeof(int), st));
  int ends[2] = {0, 0};
  MCK(cudaMemcpyAsync(&ends[0], h->row_start.get() + h->nb_int, sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaMemcpyAsync(&ends[1], h->rowptr.get() + h->nb_int, sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
  h->m_valid = ends[0];
  h->nnzb = ends[1];
  h->colidx.resize(h->nnzb, 4);
  k_bucket_fill<<<ceil_div(32LL * h->nb_int, kTpb), kTpb, 0, st>>>(h->row_start.get(), h->rowptr.get(), h->nb_int,
                                                                  h->keys.get(), nullptr, h->colidx.get(),
                                                                  h->seg_start.get(), h->kv_sorted.get());
  MLAUNCHED(h);
  MCK(cudaGetLastError());
  return true;
}

bool row_sort_triplets(maspcg_handle* h, const int* rows, const int* cols, int n, int last_row, MergedKeys& out)
{
  // more rows than this would make the per-row passes the longer part
  if (last_row >= 2LL * n + 4096) return false;
  const int nrows = last_row + 1;
  cudaStream_t st = h->stream;
  h->row_start.resize(2 * ((size_t)nrows + 1));
  int* start = h->row_start.get();
  int* uptr = start + nrows + 1;
  int flags[2] = {0, 0};
  int* position = h->asm_idx.get();
  if (!bucket<false>(h, rows, cols, n, nrows, 0, nullptr, h->asm_keys.get(), position, start, uptr,
                     h->asm_flags.get() + 2 * (size_t)n, flags))
    return false;
  int count = 0;
  MCK(cudaMemcpyAsync(&count, uptr + nrows, sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
  h->asm_start.resize((size_t)count + 1);
  int* urow = h->asm_flags.get();
  int* ucol = urow + n;
  k_bucket_fill<<<ceil_div(32LL * nrows, kTpb), kTpb, 0, st>>>(start, uptr, nrows, h->asm_keys.get(), urow, ucol,
                                                              h->asm_start.get(), position);
  MLAUNCHED(h);
  MCK(cudaMemcpyAsync(h->asm_start.get() + count, start + nrows, sizeof(int), cudaMemcpyDeviceToDevice, st));
  MCK(cudaGetLastError());
  out.rows = urow;
  out.cols = ucol;
  out.perm = position;
  out.start = h->asm_start.get();
  out.count = count;
  return true;
}

}  // namespace maspcg
