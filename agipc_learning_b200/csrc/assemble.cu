// assemble.cu -- the two triplet steps in front of the solve, on the device:
//
// * convert_bcoo: Converter::convert (StiffGIPC/linear_system/utils/
//   converter.cu:137-284).  Triplets are put in the stable order of (row, col)
//   by row buckets (rowsort.cu), or, where rows are too long or too many for
//   those, by a radix sort of the key (row << 32) + col packed into as few bits as the
//   indices need, and each run's 3x3 blocks are summed.  The reference sums a run with
//   a warp head-segmented reduction plus FP64 atomics, whose order varies;
//   here each element of a block is summed over its run in the stable sort
//   order, so the result is deterministic (and equal to a sequential sum in input order within each
//   key).
// * partition_contacts: GIPC::partitionContactHessian (StiffGIPC/GIPC.cu:
//   9952-10128 with _partition_collision_triplets and _reorder_triplets at
//   :218-283).  Contact triplets carry a type hash (0 FEM-FEM, 1 ABD-FEM,
//   2 FEM-ABD, 3 ABD-ABD); a stable radix sort on it groups them by type
//   in that order, and the per-type counts come back with the reordered
//   triplets.
//
// Both are integer, bit-exact work apart from the FP64 sums.
#include <algorithm>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "maspcg_internal.cuh"

namespace maspcg {
namespace {

constexpr int kAsmTpb = 256;

// Key (row << col_bits) + col: the order of (row << 32) + col in as few bits
// as the indices need, so the radix sort runs only the passes it must.
__global__ void k_conv_keys(const int* __restrict__ rows, const int* __restrict__ cols, int n, int col_bits,
                            unsigned long long* keys, int* idx)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  keys[i] = ((unsigned long long)(unsigned)rows[i] << col_bits) + (unsigned long long)(unsigned)cols[i];
  idx[i] = i;
}

__global__ void k_conv_heads(const unsigned long long* __restrict__ keys, int n, int* heads)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) heads[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1 : 0;
}

// start[u] = first sorted position of unique key u; start[count] = n; its row
// and column
__global__ void k_conv_starts(const int* __restrict__ heads, const int* __restrict__ pos,
                              const unsigned long long* __restrict__ keys, int n, int col_bits, int* start, int* urow,
                              int* ucol)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && heads[i]) {
    const int u = pos[i];
    start[u] = i;
    urow[u] = (int)(keys[i] >> col_bits);
    ucol[u] = (int)(keys[i] & ((1ull << col_bits) - 1ull));
  }
  if (i == n - 1) start[pos[i] + heads[i]] = n;
}

// One thread per element of a unique key's block: the sum over its run in
// sorted (stable) order, and the row and column.  Nine consecutive threads read
// a block's 72 bytes and write the sum's, so both are coalesced; the runs'
// entries are fetched four ahead of the sums.  Bound by the latency of the
// scattered blocks.  On the 110,592-row merge the whole call went from 1.21 to
// 0.94 ms with this kernel and a range pass with fewer atomics (a thread per key
// before; 0.59 with the row buckets since).
__global__ void __launch_bounds__(kAsmTpb) k_conv_sum(MergedKeys k, const double* __restrict__ vals,
                                                     int* rows_out, int* cols_out, double* vals_out)
{
  const long long e = (long long)blockIdx.x * kAsmTpb + threadIdx.x;
  const int u = (int)(e / 9), q = (int)(e % 9);
  if (u >= k.count) return;
  const int s = k.start[u], end = k.start[u + 1];
  if (q == 0) rows_out[u] = k.rows[u];
  if (q == 1) cols_out[u] = k.cols[u];
  double a = 0.0;
  for (int t = s; t < end; t += 4) {
    double v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = t + j < end ? __ldcs(vals + 9 * (size_t)k.perm[t + j] + q) : 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (t + j < end) a = a + v[j];
  }
  vals_out[e] = a;
}

__global__ void k_part_keys(const unsigned long long* __restrict__ types, int n, unsigned* keys, int* idx, int* bad,
                            int* counts)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const unsigned long long t = types[i];
  if (t > 3ull) atomicExch(bad, 1);
  const unsigned k = (unsigned)(t & 3ull);
  keys[i] = k;
  idx[i] = i;
  // one atomic per type present in the warp
  const unsigned same = __match_any_sync(__activemask(), k);
  if (__ffs(same) - 1 == (int)(threadIdx.x & 31)) atomicAdd(counts + k, __popc(same));
}

// One thread per element of a block (coalesced reads and writes).
__global__ void k_gather_triplets(const int* __restrict__ perm, int n, const int* __restrict__ rows,
                                  const int* __restrict__ cols, const double* __restrict__ vals, int* rows_out,
                                  int* cols_out, double* vals_out)
{
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int i = (int)(e / 9), q = (int)(e % 9);
  if (i >= n) return;
  const int p = perm[i];
  if (q == 0) rows_out[i] = rows[p];
  if (q == 1) cols_out[i] = cols[p];
  vals_out[e] = vals[9 * (size_t)p + q];
}

}  // namespace

MergedKeys merge_keys(maspcg_handle* h, const int* rows, const int* cols, int n)
{
  MergedKeys out{};
  if (n <= 0) return out;
  cudaStream_t st = h->stream;
  TripletRange top{};
  if (row_sort_triplets(h, rows, cols, n, top, out)) return out;
  unsigned long long* k0 = h->asm_keys.get();  // 2n at least
  unsigned long long* k1 = k0 + n;
  h->asm_idx.resize(2 * (size_t)n);
  h->asm_flags.resize(2 * (size_t)n + 4);
  int* i0 = h->asm_idx.get();
  int* i1 = i0 + n;
  int* heads = h->asm_flags.get();
  int* pos = heads + n;
  const int grid = ceil_div(n, kAsmTpb);
  auto bits = [](unsigned v) {
    int b = 1;
    while (b < 32 && (v >> b) != 0u) ++b;
    return b;
  };
  const int col_bits = bits((unsigned)top.col), key_bits = col_bits + bits((unsigned)top.row);
  k_conv_keys<<<grid, kAsmTpb, 0, st>>>(rows, cols, n, col_bits, k0, i0); MLAUNCHED(h);
  size_t need = 0;
  MCK(cub::DeviceRadixSort::SortPairs(nullptr, need, k0, k1, i0, i1, n, 0, key_bits, st));
  size_t need2 = 0;
  MCK(cub::DeviceScan::ExclusiveSum(nullptr, need2, heads, pos, n, st));
  h->cub_tmp.resize(std::max(std::max(need, need2), h->cub_tmp.n));
  size_t tb = h->cub_tmp.cap;
  MCK(cub::DeviceRadixSort::SortPairs(h->cub_tmp.get(), tb, k0, k1, i0, i1, n, 0, key_bits, st));
  k_conv_heads<<<grid, kAsmTpb, 0, st>>>(k1, n, heads); MLAUNCHED(h);
  tb = h->cub_tmp.cap;
  MCK(cub::DeviceScan::ExclusiveSum(h->cub_tmp.get(), tb, heads, pos, n, st));
  int last[2] = {0, 0};
  MCK(cudaMemcpyAsync(&last[0], pos + (n - 1), sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaMemcpyAsync(&last[1], heads + (n - 1), sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
  const int count = last[0] + last[1];
  h->asm_start.resize((size_t)count + 1);
  // (the keys' first copy is free by now: it takes the rows and columns)
  int* urow = reinterpret_cast<int*>(k0);
  int* ucol = urow + n;
  k_conv_starts<<<grid, kAsmTpb, 0, st>>>(heads, pos, k1, n, col_bits, h->asm_start.get(), urow, ucol); MLAUNCHED(h);
  MCK(cudaGetLastError());
  out.rows = urow;
  out.cols = ucol;
  out.perm = i1;
  out.start = h->asm_start.get();
  out.count = count;
  return out;
}

int convert_bcoo(maspcg_handle* h, const int* rows, const int* cols, const double* vals, int n, int* rows_out,
                 int* cols_out, double* vals_out)
{
  const MergedKeys k = merge_keys(h, rows, cols, n);
  if (k.count == 0) return 0;
  k_conv_sum<<<ceil_div(9LL * k.count, kAsmTpb), kAsmTpb, 0, h->stream>>>(k, vals, rows_out, cols_out,
                                                                          vals_out);
  MLAUNCHED(h);
  MCK(cudaGetLastError());
  return k.count;
}

void partition_contacts(maspcg_handle* h, const int* rows, const int* cols, const double* vals,
                        const unsigned long long* types, int n, int* rows_out, int* cols_out, double* vals_out,
                        int counts[4])
{
  counts[0] = counts[1] = counts[2] = counts[3] = 0;
  if (n <= 0) return;
  cudaStream_t st = h->stream;
  h->asm_keys.resize((size_t)n);  // two 32-bit key arrays
  h->asm_idx.resize(2 * (size_t)n);
  h->asm_flags.resize(8);
  unsigned* k0 = reinterpret_cast<unsigned*>(h->asm_keys.get());
  unsigned* k1 = k0 + n;
  int* i0 = h->asm_idx.get();
  int* i1 = i0 + n;
  int* bad = h->asm_flags.get();
  int* dcount = bad + 1;
  MCK(cudaMemsetAsync(bad, 0, 5 * sizeof(int), st));
  const int grid = ceil_div(n, kAsmTpb);
  k_part_keys<<<grid, kAsmTpb, 0, st>>>(types, n, k0, i0, bad, dcount); MLAUNCHED(h);
  size_t need = 0;
  MCK(cub::DeviceRadixSort::SortPairs(nullptr, need, k0, k1, i0, i1, n, 0, 2, st));
  h->cub_tmp.resize(std::max(need, h->cub_tmp.n));
  size_t tb = h->cub_tmp.cap;
  MCK(cub::DeviceRadixSort::SortPairs(h->cub_tmp.get(), tb, k0, k1, i0, i1, n, 0, 2, st));
  int flags[5] = {0, 0, 0, 0, 0};
  MCK(cudaMemcpyAsync(flags, bad, 5 * sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
  MREQ(flags[0] == 0, MASPCG_ERR_INVALID_ARGUMENT, "contact type hash outside 0..3");
  k_gather_triplets<<<ceil_div(9LL * n, kAsmTpb), kAsmTpb, 0, st>>>(i1, n, rows, cols, vals, rows_out, cols_out, vals_out); MLAUNCHED(h);
  MCK(cudaGetLastError());
  for (int t = 0; t < 4; ++t) counts[t] = flags[1 + t];
}

}  // namespace maspcg
