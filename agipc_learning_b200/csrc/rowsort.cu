// rowsort.cu -- triplets into row order by buckets: the order a stable sort on
// (row, column) gives, with one scatter instead of a radix sort's passes.
//
// The rows of these systems are short (a vertex has some 15 neighbours, a raw
// row some 60 triplets), so the entries are counted per row, scattered to their
// row's bucket (in whatever order the atomics give) and each bucket is sorted
// by (column, input position) in registers: the position makes every key
// unique and the result the stable order.  At 64-bit keys a radix sort of n
// pairs reads and writes them once per 8 key bits, five times for 262,144 rows.
// Merging the 110,592-row system's triplets went from 0.92 to 0.59 ms, building
// the 262,144-row matrix from 0.87 to 0.68, the 8,000-row one from 0.25 to 0.20.
//
// Rows longer than kRowMost, or more rows than the triplets justify
// (bucket_rows), keep the radix sort: the callers fall back when these functions
// return false.  That is known after the counting pass, which also takes the
// range of the indices, so a fallback costs little more than the range pass that
// a radix sort needs anyway: 28,100 triplets with a row of 1,100 merge in 0.27 ms
// and 127,000 with a row of 100,000 in 0.29, by the radix sort alone 0.26 and
// 0.31; as matrices 0.24 and 0.27 (0.25 and 0.29).
#include <algorithm>

#include <cub/device/device_scan.cuh>

#include "maspcg_internal.cuh"

namespace maspcg {
namespace {

constexpr int kTpb = 256;
constexpr int kRowMost = 1024;  // entries of a row one warp sorts in registers (32 per lane)

// Most rows for m entries that are sorted by buckets.  A row costs a warp of the
// sort and of the fill (some 0.35 ns), an entry a little less than in a radix
// sort, and there are fewer launches: with rows of random triplets the two ways
// meet at 133,000 rows for 0.2 M entries, 250,000 for 1.5 M and 600,000 for 6 M
// (merge), at 90,000 for 0.4 M, 214,000 for 3 M and 476,000 for 6 M (matrix).
size_t bucket_rows(size_t m) { return std::min(m / 16 + 65536, (size_t)1 << 26); }

// Places for the warp's entries in their rows' buckets (-1 where take is
// false): one atomic for each of the warp's first two rows, which are mostly the
// only ones that repeat, and one for each other entry, all of them in flight
// together.
__device__ __forceinline__ int bucket_rank(int* count, int row, bool take, int lane)
{
  unsigned todo = __ballot_sync(kFull, take), group = 1u << lane;
  int from = lane;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int lead = todo ? __ffs(todo) - 1 : 0;
    const int r = __shfl_sync(kFull, row, lead);
    const unsigned same = __ballot_sync(kFull, take && row == r) & todo;
    if ((same >> lane) & 1u) from = lead, group = same;
    todo &= ~same;
  }
  int base = 0;
  if (take && from == lane) base = atomicAdd(count + row, __popc(group));
  base = __shfl_sync(kFull, base, from);
  return take ? base + __popc(group & ((1u << lane) - 1u)) : -1;
}

// Entries per row and every entry's place among its row's.  flags: [0] an index
// out of range, [1] longest row (not its full length beyond kRowMost), [2] largest
// row and [3] largest column (kSym: not set, rows and columns are below nb; else
// rows from nb on are not counted).  The atomics of a long row queue on one
// address (71 us for 100,000 entries), so the CTAs look once a round whether there
// is one and count no further.
template <bool kSym>
__global__ void __launch_bounds__(kTpb) k_bucket_count(const int* __restrict__ rows, const int* __restrict__ cols, int n,
                                                      int nb, const int* __restrict__ map, int* count, int* rank,
                                                      int* flags)
{
  __shared__ unsigned most[3][kTpb / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned top[3] = {0u, 0u, 0u};
  bool bad = false, counting = true;
  for (unsigned base = blockIdx.x * kTpb; base < (unsigned)n; base += gridDim.x * kTpb) {  // uniform
    const unsigned i = base + threadIdx.x;
    const bool in = i < (unsigned)n;
    if (base >= gridDim.x * kTpb)
      counting = !__syncthreads_or(threadIdx.x == 0 && __ldcg(flags + 1) > kRowMost) && counting;
    int r = in ? rows[i] : -1, c = in ? cols[i] : -1;
    if constexpr (kSym) {
      const bool ok = (unsigned)r < (unsigned)nb && (unsigned)c < (unsigned)nb;
      bad |= in && !ok;
      if (ok) r = __ldg(map + r), c = __ldg(map + c);
      if (!counting) continue;
      const int2 k = make_int2(bucket_rank(count, r, ok, lane), bucket_rank(count, c, ok && r != c, lane));
      if (in) reinterpret_cast<int2*>(rank)[i] = k;
      if (k.x == kRowMost || k.y == kRowMost) atomicMax(flags + 1, kRowMost + 1);
      top[0] = max(top[0], (unsigned)(max(k.x, k.y) + 1));
    } else {
      bad |= in && (r < 0 || c < 0);
      top[1] = max(top[1], (unsigned)max(r, 0));
      top[2] = max(top[2], (unsigned)max(c, 0));
      if (!counting) continue;
      const int k = bucket_rank(count, r, (unsigned)r < (unsigned)nb, lane);
      if (in) rank[i] = k;
      if (k == kRowMost) atomicMax(flags + 1, kRowMost + 1);
      top[0] = max(top[0], (unsigned)(k + 1));
    }
  }
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    top[q] = __reduce_max_sync(kFull, top[q]);
    if (lane == 0) most[q][w] = top[q];
  }
  bad = __syncthreads_or(bad);
  if (threadIdx.x < (kSym ? 1 : 3)) {
    unsigned v = 0;
    for (int q = 0; q < kTpb / 32; ++q) v = max(v, most[threadIdx.x][q]);
    atomicMax(flags + 1 + threadIdx.x, (int)v);
  }
  if (threadIdx.x == 0 && bad) atomicExch(flags, 1);
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

// The counting pass; flags on the host after it.
template <bool kSym>
void count_rows(maspcg_handle* h, const int* rows, const int* cols, int n, int nb, const int* map, int* count,
                int* rank, int* flags, int flags_host[4])
{
  cudaStream_t st = h->stream;
  k_bucket_count<kSym><<<std::min(ceil_div(n, kTpb), 8 * h->sm_count), kTpb, 0, st>>>(rows, cols, n, nb, map, count,
                                                                                    rank, flags);
  MLAUNCHED(h);
  MCK(cudaGetLastError());
  MCK(cudaMemcpyAsync(flags_host, flags, 4 * sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
}

// Scatter, sort, and the offsets of the entries (start) and distinct columns
// (uptr) of each of nrows rows, nrows + 1 of them; count[nrows] is 0.
template <bool kSym>
void sort_rows(maspcg_handle* h, const int* rows, const int* cols, int n, int nrows, const int* map,
               unsigned long long* entries, int* count, const int* rank, int* start, int* uptr)
{
  cudaStream_t st = h->stream;
  size_t need = 0;
  MCK(cub::DeviceScan::ExclusiveSum(nullptr, need, count, start, nrows + 1, st));
  h->cub_tmp.resize(std::max(need, h->cub_tmp.n));
  size_t tb = h->cub_tmp.cap;
  MCK(cub::DeviceScan::ExclusiveSum(h->cub_tmp.get(), tb, count, start, nrows + 1, st));
  k_bucket_scatter<kSym><<<ceil_div(n, kTpb), kTpb, 0, st>>>(rows, cols, n, map, start, rank, entries); MLAUNCHED(h);
  k_bucket_sort<<<ceil_div(32LL * (nrows + 1LL), kTpb), kTpb, 0, st>>>(start, nrows, entries, count); MLAUNCHED(h);
  tb = h->cub_tmp.cap;
  MCK(cub::DeviceScan::ExclusiveSum(h->cub_tmp.get(), tb, count, uptr, nrows + 1, st));
  MCK(cudaGetLastError());
}

}  // namespace

bool row_sort_matrix(maspcg_handle* h, const int* rows, const int* cols, int n)
{
  const int nrows = h->nb_int;
  if ((size_t)nrows > bucket_rows(2 * (size_t)n)) return false;
  cudaStream_t st = h->stream;
  int* count = h->row_count.get();  // 4 more at the end, for the flags
  int* flags = count + nrows + 1;
  MCK(cudaMemsetAsync(count, 0, sizeof(int) * ((size_t)nrows + 5), st));
  int f[4] = {0, 0, 0, 0};
  count_rows<true>(h, rows, cols, n, h->nb, h->int_of_row.get(), count, h->kv.get(), flags, f);
  MREQ(f[0] == 0, MASPCG_ERR_INVALID_ARGUMENT, "matrix block index out of range");
  if (f[1] > kRowMost) return false;
  h->row_start.resize((size_t)nrows + 1);
  sort_rows<true>(h, rows, cols, n, nrows, h->int_of_row.get(), h->keys.get(), count, h->kv.get(), h->row_start.get(),
                  h->rowptr.get());
  int ends[2] = {0, 0};
  MCK(cudaMemcpyAsync(&ends[0], h->row_start.get() + nrows, sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaMemcpyAsync(&ends[1], h->rowptr.get() + nrows, sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
  h->m_valid = ends[0];
  h->nnzb = ends[1];
  h->colidx.resize(h->nnzb, 4);
  k_bucket_fill<<<ceil_div(32LL * nrows, kTpb), kTpb, 0, st>>>(h->row_start.get(), h->rowptr.get(), nrows,
                                                              h->keys.get(), nullptr, h->colidx.get(),
                                                              h->seg_start.get(), h->kv_sorted.get());
  MLAUNCHED(h);
  MCK(cudaGetLastError());
  return true;
}

bool row_sort_triplets(maspcg_handle* h, const int* rows, const int* cols, int n, TripletRange& range, MergedKeys& out)
{
  cudaStream_t st = h->stream;
  const size_t limit = bucket_rows((size_t)n);
  // one block of scratch, which the radix sort takes over: entries, their
  // places, and per row flags, counts and offsets
  const size_t ints = (size_t)n + 4 + 3 * (limit + 1);
  h->asm_keys.resize(std::max(2 * (size_t)n, (size_t)n + (ints + 1) / 2));
  unsigned long long* entries = h->asm_keys.get();
  int* position = reinterpret_cast<int*>(entries + n);  // the place in the row's bucket first
  int* flags = position + n;
  int* count = flags + 4;
  int* start = count + limit + 1;
  int* uptr = start + limit + 1;
  MCK(cudaMemsetAsync(flags, 0, sizeof(int) * (4 + limit + 1), st));
  int f[4] = {0, 0, 0, 0};
  count_rows<false>(h, rows, cols, n, (int)limit, nullptr, count, position, flags, f);
  MREQ(f[0] == 0, MASPCG_ERR_INVALID_ARGUMENT, "negative row or column index");
  range.row = f[2];
  range.col = f[3];
  if (f[1] > kRowMost || (size_t)f[2] >= limit) return false;
  const int nrows = f[2] + 1;
  sort_rows<false>(h, rows, cols, n, nrows, nullptr, entries, count, position, start, uptr);
  int distinct = 0;
  MCK(cudaMemcpyAsync(&distinct, uptr + nrows, sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
  h->asm_start.resize(3 * (size_t)distinct + 1);
  int* first = h->asm_start.get();
  int* urow = first + distinct + 1;
  int* ucol = urow + distinct;
  k_bucket_fill<<<ceil_div(32LL * nrows, kTpb), kTpb, 0, st>>>(start, uptr, nrows, entries, urow, ucol, first, position);
  MLAUNCHED(h);
  MCK(cudaMemcpyAsync(first + distinct, start + nrows, sizeof(int), cudaMemcpyDeviceToDevice, st));
  MCK(cudaGetLastError());
  out.rows = urow;
  out.cols = ucol;
  out.perm = position;
  out.start = first;
  out.count = distinct;
  return true;
}

}  // namespace maspcg
