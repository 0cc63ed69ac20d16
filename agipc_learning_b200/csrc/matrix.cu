// matrix.cu -- assembled BCOO -> internal full BCSR, FP64 SpMV, permutations,
// block-Jacobi (3x3) and affine-body (12x12) inverses.
//
// The conversion follows Converter::convert (converter.cu:137-284): the stable
// order of the (row, col) keys, here by row buckets (rowsort.cu) or, with rows
// too long or too many for those, by a radix sort, and a segmented sum of equal
// keys, so the block structure is bit-exact and FP64 sums are taken in input
// order.  It differs in what it produces: both triangles (the symmetric SpMV of
// spmv.cu:28-53 scatters B^T with atomics; a row-owned BCSR needs none) and
// rows renumbered into the MAS partition order.
#include <algorithm>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "maspcg_internal.cuh"
#include "spmv_row.cuh"

namespace maspcg {
namespace {

constexpr int kTpb = 256;
constexpr unsigned long long kSentinel = ~0ull;

// The internal row of every block row and back: the FEM rows [fem_off, fem_off +
// nv) take their slots in [fem_off, fem_off + c0) (padding slots: -1), the rows
// after them move up by c0 - nv.
__global__ void k_row_maps(int nb, int nb_int, int fem_off, int nv, int c0, const int* __restrict__ rmp,
                           const int* __restrict__ pmr, int* int_of_row, int* row_of_int)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nb) int_of_row[i] = i < fem_off ? i : (i < fem_off + nv ? fem_off + rmp[i - fem_off] : i + c0 - nv);
  if (i < nb_int) {
    int r = i;
    if (i >= fem_off + c0)
      r = i - (c0 - nv);
    else if (i >= fem_off)
      r = pmr[i - fem_off] >= 0 ? fem_off + pmr[i - fem_off] : -1;
    row_of_int[i] = r;
  }
}

__global__ void k_make_keys(const int* __restrict__ rows, const int* __restrict__ cols, int n, int nb,
                            const int* __restrict__ int_of_row, int bits, unsigned long long* keys, int* vals,
                            int* bad)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = rows[i], c = cols[i];
  if (r < 0 || c < 0 || r >= nb || c >= nb) {
    atomicAdd(bad, 1);
    keys[2 * (size_t)i] = kSentinel;
    keys[2 * (size_t)i + 1] = kSentinel;
    return;
  }
  const unsigned long long ri = (unsigned)int_of_row[r], ci = (unsigned)int_of_row[c];
  keys[2 * (size_t)i] = (ri << bits) | ci;
  vals[2 * (size_t)i] = i << 1;  // A_rc = H
  if (r != c) {
    keys[2 * (size_t)i + 1] = (ci << bits) | ri;
    vals[2 * (size_t)i + 1] = (i << 1) | 1;  // A_cr = H^T
  } else {
    keys[2 * (size_t)i + 1] = kSentinel;
    vals[2 * (size_t)i + 1] = -1;
    atomicAdd(bad + 2, 1);
  }
}

__global__ void k_heads(const unsigned long long* __restrict__ keys, int m, int* head)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const unsigned long long k = keys[i];
  head[i] = (k != kSentinel && (i == 0 || k != keys[i - 1])) ? 1 : 0;
}

// Block count, indices out of range and sentinels of the sorted structure in one
// place: one copy to the host (each waits for the stream) where there were three.
__global__ void k_structure_ends(const int* last_head, const int* last_index, const int* flags, int* ends)
{
  ends[0] = *last_head + *last_index;
  ends[1] = flags[0];
  ends[2] = flags[2];
}

__global__ void k_fill_structure(const unsigned long long* __restrict__ keys, const int* __restrict__ head,
                                 const int* __restrict__ uidx, int m, int bits, int* colidx, int* seg_start,
                                 int* row_count)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  if (!head[i]) return;
  const unsigned long long k = keys[i];
  const int u = uidx[i];
  const int row = (int)(k >> bits);
  colidx[u] = (int)(k & ((1ull << bits) - 1));
  seg_start[u] = i;
  atomicAdd(row_count + row, 1);
}

// One CTA per tile of 32 stored blocks, a thread per element: the input blocks
// of the element summed in sorted (= input) order, fetched four ahead.  Nine
// consecutive threads read a block's 72 bytes and write its FP64 values; the
// FP32 tile (null in the reference precision, which does not read it) is
// transposed in shared memory and written in one run.
// Bound by the scattered input blocks.  With the row maps formed on the device the
// matrix of the 64^3 contact system was built in 0.87 ms (0.68 with the row buckets
// since), 1.31 with a thread per block and the maps copied from the host.
constexpr int kFillTpb = 288;
__global__ void __launch_bounds__(kFillTpb) k_fill_values(const int* __restrict__ vals_sorted,
                                                         const int* __restrict__ seg_start, int nnzb, int m_valid,
                                                         const double* __restrict__ in_vals, double* val64,
                                                         float* val32, unsigned short* val_lo)
{
  __shared__ float hi_s[kFillTpb];
  __shared__ unsigned short lo_s[kFillTpb];
  const int tid = threadIdx.x, b = tid / 9, q = tid % 9;
  const int u = blockIdx.x * 32 + b;
  const int straight = q / 3 + 3 * (q % 3);  // element (r, c) = (q / 3, q % 3) of a column-major block; transposed: q
  double a = 0.0;
  if (u < nnzb) {
    const int s = seg_start[u], e = (u + 1 < nnzb) ? seg_start[u + 1] : m_valid;
    for (int i = s; i < e; i += 4) {
      double v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        v[k] = 0.0;
        if (i + k < e) {
          const int p = vals_sorted[i + k];  // bit 0: A_cr = H^T
          v[k] = in_vals[9 * (size_t)(p >> 1) + ((p & 1) ? q : straight)];
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (i + k < e) a += v[k];
    }
    val64[9 * (size_t)u + q] = a;
  }
  if (!val32) return;  // uniform
  const float hi = (float)a;
  hi_s[32 * q + b] = hi;  // tiles of 32 blocks, element-major
  // the remainder a - hi is exact in FP64; its BF16 rounding carries A to
  // about 2^-32 relative
  if (val_lo) lo_s[32 * q + b] = __bfloat16_as_ushort(__float2bfloat16_rn((float)(a - (double)hi)));
  __syncthreads();
  val32[(size_t)blockIdx.x * 288 + tid] = hi_s[tid];
  if (val_lo) val_lo[(size_t)blockIdx.x * 288 + tid] = lo_s[tid];
}

// y = a*A*x + b*y, FP64, half-warp per block row.
__global__ void k_spmv64(const int* __restrict__ rowptr, const int* __restrict__ colidx, const double* __restrict__ val,
                         const double* __restrict__ x, double* y, double a, double b, int nrows)
{
  constexpr int LPR = 16;
  const int gl = blockIdx.x * blockDim.x + threadIdx.x;
  const int row = gl / LPR, sub = gl % LPR;
  const bool ok = row < nrows;
  const int rs = ok ? rowptr[row] : 0, re = ok ? rowptr[row + 1] : 0;
  double acc[3];
  row_product<double, double, LPR>(rs, re, colidx, val, x, sub, acc);
  if (ok && sub < 3) {
    const double prev = (b != 0.0) ? b * y[3 * (size_t)row + sub] : 0.0;
    y[3 * (size_t)row + sub] = a * acc[sub] + prev;
  }
}

__global__ void k_permute_in(const double* __restrict__ src, double* dst, const int* __restrict__ row_of_int, int nb_int)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 3 * nb_int) return;
  const int r = row_of_int[i / 3];
  dst[i] = r >= 0 ? src[3 * (size_t)r + i % 3] : 0.0;
}

__global__ void k_permute_out(const double* __restrict__ src, double* dst, const int* __restrict__ int_of_row, int nb)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 3 * nb) return;
  dst[i] = src[3 * (size_t)int_of_row[i / 3] + i % 3];
}

// DiagPreconditioner (diag_preconditioner.cu:10-39): 3x3 inverse of the
// diagonal block, identity where it is missing.
__global__ void k_diag3(const int* __restrict__ rowptr, const int* __restrict__ colidx, const double* __restrict__ val,
                        int nrows, double* inv64, float* inv32)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nrows) return;
  int lo = rowptr[i], hi = rowptr[i + 1] - 1, t = -1;
  while (lo <= hi) {
    const int mid = (lo + hi) >> 1;
    const int c = colidx[mid];
    if (c == i) {
      t = mid;
      break;
    }
    if (c < i)
      lo = mid + 1;
    else
      hi = mid - 1;
  }
  double o[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
  if (t >= 0) {
    const double* m = val + 9 * (size_t)t;  // row-major
    const double a = m[0], b = m[1], c = m[2], d = m[3], e = m[4], f = m[5], g = m[6], hh = m[7], k = m[8];
    const double A = e * k - f * hh, B = -(d * k - f * g), C = d * hh - e * g;
    const double det = a * A + b * B + c * C;
    const double id = 1.0 / det;
    o[0] = A * id;
    o[1] = -(b * k - c * hh) * id;
    o[2] = (b * f - c * e) * id;
    o[3] = B * id;
    o[4] = (a * k - c * g) * id;
    o[5] = -(a * f - c * d) * id;
    o[6] = C * id;
    o[7] = -(a * hh - b * g) * id;
    o[8] = (a * e - b * d) * id;
  }
  for (int q = 0; q < 9; ++q) {
    inv64[9 * (size_t)i + q] = o[q];
    inv32[9 * (size_t)i + q] = (float)o[q];
  }
}

// ABDPreconditioner (setup_abd_system_gradient_and_hessian.cu:407-441): gather
// the body's 12x12 diagonal block from the blocks with row/4 == col/4 and
// invert it (Gauss-Jordan, partial pivoting), row-major.  A warp per body: lane
// c < 24 holds column c of [A | 1] in registers and takes the pivot column from
// lane k, so a step is 12 multiply-adds and as many shuffles.  Bound by that
// chain; a thread per body on a matrix in local memory took 172 us for 500
// bodies.
constexpr int kAbdWarps = 4;
__global__ void __launch_bounds__(32 * kAbdWarps) k_abd_inverse(const int* __restrict__ rowptr,
                                                                const int* __restrict__ colidx,
                                                                const double* __restrict__ val, int bodies,
                                                                double* inv64, int* failed)
{
  __shared__ double block[kAbdWarps][12][12];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, bdy = blockIdx.x * kAbdWarps + w;
  if (bdy >= bodies) return;
  double(*m)[12] = block[w];
  for (int e = lane; e < 144; e += 32) m[e / 12][e % 12] = 0.0;
  __syncwarp();
  for (int q = 0; q < 4; ++q) {
    const int row = 4 * bdy + q;
    for (int t = rowptr[row] + lane; t < rowptr[row + 1]; t += 32) {
      const int c = colidx[t];
      if (c / 4 != bdy) continue;
      if (t + 1 < rowptr[row + 1] && colidx[t + 1] == c) continue;  // of equal columns the last one, as ever
      for (int e = 0; e < 9; ++e) m[3 * q + e / 3][3 * (c % 4) + e % 3] = val[9 * (size_t)t + e];
    }
  }
  __syncwarp();
  double a[12];
#pragma unroll
  for (int r = 0; r < 12; ++r) a[r] = lane < 12 ? m[r][lane] : (lane - 12 == r ? 1.0 : 0.0);
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    double col[12];  // the pivot column
#pragma unroll
    for (int r = 0; r < 12; ++r) col[r] = __shfl_sync(kFull, a[r], k);
    int piv = k;
    double top = col[k];
#pragma unroll
    for (int r = k + 1; r < 12; ++r)
      if (fabs(col[r]) > fabs(top)) piv = r, top = col[r];
    if (top == 0.0) {
      ok = false;
      break;
    }
#pragma unroll
    for (int r = k + 1; r < 12; ++r)
      if (r == piv) {
        const double t = a[k], u = col[k];
        a[k] = a[r], col[k] = col[r];
        a[r] = t, col[r] = u;
      }
    const double inv = 1.0 / top;
    a[k] *= inv;
#pragma unroll
    for (int r = 0; r < 12; ++r)
      if (r != k && col[r] != 0.0) a[r] -= col[r] * a[k];
  }
  if (!ok && lane == 0) atomicAdd(failed, 1);
  if (lane >= 12 && lane < 24)
#pragma unroll
    for (int r = 0; r < 12; ++r)
      inv64[144 * (size_t)bdy + 12 * r + lane - 12] = ok ? a[r] : (r == lane - 12 ? 1.0 : 0.0);
}

// The reference precision runs on the FP64 values alone.
bool runs_fp32(const maspcg_handle* h) { return h->cfg.precision != MASPCG_PREC_REFERENCE; }

// The merged values of the current structure from the input blocks.
void fill_values(maspcg_handle* h, const double* vals)
{
  k_fill_values<<<ceil_div(h->nnzb, 32), kFillTpb, 0, h->stream>>>(
      h->kv_sorted.get(), h->seg_start.get(), h->nnzb, h->m_valid, vals, h->val64.get(),
      runs_fp32(h) ? h->val32.get() : nullptr,
      h->cfg.matrix_form == MASPCG_MATRIX_F32_SPLIT ? h->val_lo.get() : nullptr);
  MLAUNCHED(h);
  MCK(cudaGetLastError());
}

size_t cub_bytes_sort(int m, int end_bit)
{
  size_t b = 0;
  MCK(cub::DeviceRadixSort::SortPairs(nullptr, b, (const unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                      (const int*)nullptr, (int*)nullptr, m, 0, end_bit));
  return b;
}

// The structure by a stable radix sort of (row, col) keys (rows of any length).
void radix_sort_matrix(maspcg_handle* h, const int* rows, const int* cols, int n)
{
  cudaStream_t st = h->stream;
  const int nb = h->nb, nb_int = h->nb_int, m = 2 * n;
  int bits = 1;
  while ((1ll << bits) <= nb_int) ++bits;
  MREQ(2 * bits <= 62, MASPCG_ERR_CAPACITY, "too many block rows");
  h->keys_sorted.resize(m);
  h->seg_head.resize(m);
  MCK(cudaMemsetAsync(h->failed.get(), 0, sizeof(int) * 8, st));
  k_make_keys<<<ceil_div(n, kTpb), kTpb, 0, st>>>(rows, cols, n, nb, h->int_of_row.get(), bits, h->keys.get(),
                                                 h->kv.get(), h->failed.get()); MLAUNCHED(h);
  // keys use 2*bits bits; the all-ones sentinel still sorts last on 2*bits+1
  const int end_bit = 2 * bits + 1;
  size_t need = cub_bytes_sort(m, end_bit);
  size_t scan_b = 0;
  MCK(cub::DeviceScan::ExclusiveSum(nullptr, scan_b, (const int*)nullptr, (int*)nullptr, m));
  need = std::max(need, scan_b);
  h->cub_tmp.resize(need);
  size_t tb = h->cub_tmp.cap;
  MCK(cub::DeviceRadixSort::SortPairs(h->cub_tmp.get(), tb, h->keys.get(), h->keys_sorted.get(), h->kv.get(),
                                      h->kv_sorted.get(), m, 0, end_bit, st));
  k_heads<<<ceil_div(m, kTpb), kTpb, 0, st>>>(h->keys_sorted.get(), m, h->seg_head.get()); MLAUNCHED(h);
  // unique index = exclusive scan of heads (reuse kv as output)
  tb = h->cub_tmp.cap;
  MCK(cub::DeviceScan::ExclusiveSum(h->cub_tmp.get(), tb, h->seg_head.get(), h->kv.get(), m, st));
  int* ends = h->failed.get() + 4;
  k_structure_ends<<<1, 1, 0, st>>>(h->seg_head.get() + (m - 1), h->kv.get() + (m - 1), h->failed.get(), ends);
  MLAUNCHED(h);
  int e[3] = {0, 0, 0};
  MCK(cudaMemcpyAsync(e, ends, 3 * sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
  MCK(cudaMemsetAsync(ends, 0, 3 * sizeof(int), st));
  MREQ(e[1] == 0, MASPCG_ERR_INVALID_ARGUMENT, "matrix block index out of range");
  const int nnzb = e[0];
  const int m_valid = m - e[2];  // sentinels (one per diagonal input block) sort last
  h->m_valid = m_valid;
  h->nnzb = nnzb;
  h->colidx.resize(nnzb, 4);  // 16-byte tail for TMA bulk copies
  MCK(cudaMemsetAsync(h->row_count.get(), 0, sizeof(int) * (nb_int + 1), st));
  k_fill_structure<<<ceil_div(m, kTpb), kTpb, 0, st>>>(h->keys_sorted.get(), h->seg_head.get(), h->kv.get(), m, bits,
                                                      h->colidx.get(), h->seg_start.get(), h->row_count.get()); MLAUNCHED(h);
  // rowptr = exclusive scan of the per-row counts (the extra entry gives nnzb)
  tb = h->cub_tmp.cap;
  MCK(cub::DeviceScan::ExclusiveSum(h->cub_tmp.get(), tb, h->row_count.get(), h->rowptr.get(), nb_int + 1, st));
  MCK(cudaGetLastError());
}

}  // namespace

void build_internal_matrix(maspcg_handle* h, const double* vals, const int* rows, const int* cols, int n)
{
  cudaStream_t st = h->stream;
  const int nb = h->nb;
  // ---- internal row order
  h->mas_layout = (h->cfg.preconditioner == MASPCG_PRECOND_MAS32 || h->cfg.preconditioner == MASPCG_PRECOND_MAS16) &&
                  h->has_graph && h->nv > 0;
  int nb_int = nb;
  if (h->mas_layout) {
    MREQ(h->fem_off + h->nv <= nb, MASPCG_ERR_INVALID_ARGUMENT, "FEM range exceeds the block rows");
    nb_int = nb + h->c0 - h->nv;
  }
  h->nb_int = nb_int;
  h->int_of_row.resize(nb);
  h->row_of_int.resize(nb_int);
  k_row_maps<<<ceil_div(std::max(nb, nb_int), kTpb), kTpb, 0, st>>>(
      nb, nb_int, h->mas_layout ? h->fem_off : nb, h->mas_layout ? h->nv : 0, h->mas_layout ? h->c0 : 0, h->rmp.get(),
      h->pmr.get(), h->int_of_row.get(), h->row_of_int.get()); MLAUNCHED(h);

  // ---- structure: row buckets, or a radix sort where a row is too long
  const int m = 2 * n;
  h->keys.resize(m);
  h->kv.resize(m);
  h->kv_sorted.resize(m);
  h->seg_start.resize(m + 1);
  h->failed.resize(8);
  MCK(cudaMemsetAsync(h->failed.get(), 0, sizeof(int) * 8, st));
  h->row_count.resize((size_t)nb_int + 5);
  h->rowptr.resize(nb_int + 1);
  if (!row_sort_matrix(h, rows, cols, n)) radix_sort_matrix(h, rows, cols, n);
  const int nnzb = h->nnzb;
  h->val64.resize((size_t)9 * nnzb, 2);
  const size_t tiled = (size_t)9 * (((size_t)nnzb + 31) / 32 * 32);
  if (runs_fp32(h)) h->val32.resize(tiled);
  if (h->cfg.matrix_form == MASPCG_MATRIX_F32_SPLIT) h->val_lo.resize(tiled);
  if (h->vals_pending) {  // host values copied on the side stream
    MCK(cudaStreamWaitEvent(st, h->ev_join, 0));
    h->vals_pending = false;
  }
  fill_values(h, vals);
}

void refresh_internal_values(maspcg_handle* h, const double* vals)
{
  cudaStream_t st = h->stream;
  if (h->vals_pending) {  // host values copied on the side stream
    MCK(cudaStreamWaitEvent(st, h->ev_join, 0));
    h->vals_pending = false;
  }
  fill_values(h, vals);
}

void launch_spmv64(maspcg_handle* h, const double* x, double* y, double a, double b)
{
  const long long threads = (long long)h->nb_int * 16;
  k_spmv64<<<ceil_div(threads, kTpb), kTpb, 0, h->stream>>>(h->rowptr.get(), h->colidx.get(), h->val64.get(), x, y, a,
                                                           b, h->nb_int); MLAUNCHED(h);
  MCK(cudaGetLastError());
}

void permute_in(maspcg_handle* h, const double* src, double* dst)
{
  k_permute_in<<<ceil_div(3LL * h->nb_int, kTpb), kTpb, 0, h->stream>>>(src, dst, h->row_of_int.get(), h->nb_int); MLAUNCHED(h);
  MCK(cudaGetLastError());
}

void permute_out(maspcg_handle* h, const double* src, double* dst)
{
  k_permute_out<<<ceil_div(3LL * h->nb, kTpb), kTpb, 0, h->stream>>>(src, dst, h->int_of_row.get(), h->nb); MLAUNCHED(h);
  MCK(cudaGetLastError());
}

void build_block_jacobi(maspcg_handle* h)
{
  cudaStream_t st = h->stream;
  if (h->cfg.preconditioner == MASPCG_PRECOND_BLOCK_JACOBI) {
    h->diag_inv64.resize((size_t)9 * h->nb_int);
    h->diag_inv32.resize((size_t)9 * h->nb_int);
    k_diag3<<<ceil_div(h->nb_int, kTpb), kTpb, 0, st>>>(h->rowptr.get(), h->colidx.get(), h->val64.get(), h->nb_int,
                                                       h->diag_inv64.get(), h->diag_inv32.get()); MLAUNCHED(h);
  }
  if (h->abd_bodies > 0 && h->cfg.preconditioner != MASPCG_PRECOND_NONE) {
    h->abd_inv64.resize((size_t)144 * h->abd_bodies);
    k_abd_inverse<<<ceil_div(h->abd_bodies, kAbdWarps), 32 * kAbdWarps, 0, st>>>(
        h->rowptr.get(), h->colidx.get(), h->val64.get(), h->abd_bodies, h->abd_inv64.get(), h->failed.get() + 1);
    MLAUNCHED(h);
  }
  MCK(cudaGetLastError());
}

}  // namespace maspcg
