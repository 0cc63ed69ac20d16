// galerkin.cu -- the AGIPC coarse system on the device (StiffGIPC/agipc/
// agipc_galerkin.cu): A_c = P^T A P and b_c = P^T b for the mixed
// prolongation P of the coarse mapping, and x = P x_c back.
//
// The mapping (agipc_criterion.cuh:13-25, transform_for_block at
// agipc_galerkin.cu:200-219): fine blocks [0, prefix) pass through unchanged
// (coarse block = fine block); fine FEM node k = block prefix + k belongs to
// coarse node fine_to_coarse[k], whose blocks start at prefix +
// coarse_block_bases[c] and whose basis is the subset `basis_masks[c]` of
// (1, x, y, z) at the node's rest position: a translational node keeps 1, an
// affine node all four.  A fine block (i, j) therefore expands into
// width_i x width_j coarse blocks phi_i[a] phi_j[b] A_ij (count_expanded_blocks
// and emit_expanded_blocks, :221-283): a diagonal fine block keeps a <= b; an
// off-diagonal one that lands on a coarse diagonal block adds its transpose;
// one that lands below the diagonal is transposed to (col, row).  The
// expanded triplets are then merged like any triplet list (assemble.cu).
#include <cub/device/device_scan.cuh>

#include "maspcg_internal.cuh"

namespace maspcg {

namespace {

constexpr int kGalTpb = 256;

__device__ __forceinline__ void transform_block(const GalerkinMap& m, int block, int& base, int& width, double phi[4])
{
  phi[0] = 1.0;
  phi[1] = phi[2] = phi[3] = 0.0;
  if (block < m.prefix) {
    base = block;
    width = 1;
    return;
  }
  const int k = block - m.prefix;
  const int c = m.fine_to_coarse[k];
  base = m.prefix + m.coarse_block_bases[c];
  const int mask = m.basis_masks[c];
  width = __popc((unsigned)mask & 15u);
  const double raw[4] = {1.0, m.rest[3 * (size_t)k], m.rest[3 * (size_t)k + 1], m.rest[3 * (size_t)k + 2]};
  int o = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (mask & (1 << q)) phi[o++] = raw[q];
}

__global__ void k_gal_count(GalerkinMap m, const int* __restrict__ rows, const int* __restrict__ cols, int n,
                            int* counts, int* bad)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = rows[i], c = cols[i];
  if (r < 0 || c < 0 || r >= m.fine_blocks || c >= m.fine_blocks) {
    atomicExch(bad, 1);
    counts[i] = 0;
    return;
  }
  int rb, rw, cb, cw;
  double rp[4], cp[4];
  transform_block(m, r, rb, rw, rp);
  transform_block(m, c, cb, cw, cp);
  counts[i] = r == c ? rw * (rw + 1) / 2 : rw * cw;
}

// Expanded coarse triplets without their values: row, column, the fine block
// they come from with how it enters (0 as it is, 1 transposed, 2 the sum of
// both), and the weight phi_i[a] phi_j[b].  The merge forms a value when it adds
// it (k_gal_sum), so 20 bytes per expanded triplet pass through memory, not 80:
// 0.96 to 0.84 ms for the whole coarse system of 64,000 nodes (0.78 with the merge's
// later counting pass).
__global__ void k_gal_emit(GalerkinMap m, const int* __restrict__ rows, const int* __restrict__ cols,
                           const int* __restrict__ offsets, int n, int* out_rows, int* out_cols,
                           unsigned* out_src, double* out_weight)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = rows[i], c = cols[i];
  if (r < 0 || c < 0 || r >= m.fine_blocks || c >= m.fine_blocks) return;
  int rb, rw, cb, cw;
  double rp[4], cp[4];
  transform_block(m, r, rb, rw, rp);
  transform_block(m, c, cb, cw, cp);
  int o = offsets[i];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      if (a >= rw || b >= cw || (r == c && a > b)) continue;
      const int mr = rb + a, mc = cb + b;
      const int mode = (r != c && mr == mc) ? 2 : (mr > mc ? 1 : 0);
      out_rows[o] = min(mr, mc);
      out_cols[o] = max(mr, mc);
      out_src[o] = 4u * (unsigned)i + (unsigned)mode;
      out_weight[o] = rp[a] * cp[b];
      ++o;
    }
}

// The merge's sum over expanded triplets (k_conv_sum in assemble.cu): a thread
// per element of a coarse block, values Eigen column-major (element (i, j) at
// i + 3j).  A term that is not finite sets *bad.
__global__ void __launch_bounds__(kGalTpb) k_gal_sum(MergedKeys k, const unsigned* __restrict__ src,
                                                    const double* __restrict__ weight,
                                                    const double* __restrict__ vals, int* rows_out, int* cols_out,
                                                    double* vals_out, int* bad)
{
  const long long e = (long long)blockIdx.x * kGalTpb + threadIdx.x;
  const int u = (int)(e / 9), q = (int)(e % 9), t = q / 3 + 3 * (q % 3);
  if (u >= k.count) return;
  const int s = k.start[u], end = k.start[u + 1];
  if (q == 0) rows_out[u] = k.rows[u];
  if (q == 1) cols_out[u] = k.cols[u];
  double a = 0.0;
  bool finite = true;
  for (int j = s; j < end; j += 4) {
    double v[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      v[p] = 0.0;
      if (j + p < end) {
        const int o = k.perm[j + p];
        const unsigned x = src[o], mode = x & 3u;
        const double w = weight[o];
        const double* in = vals + 9 * (size_t)(x >> 2);
        v[p] = __dmul_rn(w, in[mode == 1 ? t : q]);
        if (mode == 2) v[p] = __dadd_rn(v[p], __dmul_rn(w, in[t]));
      }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
      if (j + p < end) {
        finite &= isfinite(v[p]);
        a += v[p];
      }
  }
  vals_out[e] = a;
  if (!finite) atomicExch(bad, 1);
}

// b_c = P^T b (FP64 atomics, as reduce_mixed_rhs at agipc_galerkin.cu:285-306)
__global__ void k_gal_restrict(GalerkinMap m, const double* __restrict__ fine, double* coarse, int* bad)
{
  const int block = blockIdx.x * blockDim.x + threadIdx.x;
  if (block >= m.fine_blocks) return;
  int base, width;
  double phi[4];
  transform_block(m, block, base, width, phi);
  for (int comp = 0; comp < 3; ++comp) {
    const double v = fine[3 * (size_t)block + comp];
    if (!isfinite(v)) {
      atomicExch(bad, 2);
      continue;
    }
    for (int a = 0; a < width; ++a) atomicAdd(coarse + 3 * (size_t)(base + a) + comp, phi[a] * v);
  }
}

// x = P x_c (prolongate_mixed, agipc_galerkin.cu:355-369)
__global__ void k_gal_prolong(GalerkinMap m, const double* __restrict__ coarse, double* fine)
{
  const int block = blockIdx.x * blockDim.x + threadIdx.x;
  if (block >= m.fine_blocks) return;
  int base, width;
  double phi[4];
  transform_block(m, block, base, width, phi);
  for (int comp = 0; comp < 3; ++comp) {
    double v = 0.0;
    for (int a = 0; a < width; ++a) v += phi[a] * coarse[3 * (size_t)(base + a) + comp];
    fine[3 * (size_t)block + comp] = v;
  }
}

// Sets the bits of the rules that the mapping breaks (galerkin_check): 4 us for a
// 64,000-node mapping, whose copies to the host and checks there took some 130.
__global__ void __launch_bounds__(kGalTpb) k_gal_check(GalerkinMap m, int fem_nodes, int coarse_nodes,
                                                      int coarse_block_nodes, int* bad)
{
  const int i = blockIdx.x * kGalTpb + threadIdx.x;
  if (i < fem_nodes && (unsigned)m.fine_to_coarse[i] >= (unsigned)coarse_nodes) atomicOr(bad, 1);
  if (i < coarse_nodes) {
    const int mask = m.basis_masks[i], base = m.coarse_block_bases[i];
    if (mask < 1 || mask > 15)
      atomicOr(bad, 2);
    else if (base < 0 || (long long)base + __popc((unsigned)mask) > coarse_block_nodes)
      atomicOr(bad, 4);
  }
}

int read_int(maspcg_handle* h, const int* d)
{
  int v = 0;
  MCK(cudaMemcpyAsync(&v, d, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
  MCK(cudaStreamSynchronize(h->stream));
  return v;
}

}  // namespace

int galerkin_check(maspcg_handle* h, const GalerkinMap& m, int fem_nodes, int coarse_nodes, int coarse_block_nodes)
{
  h->gal_counts.resize(std::max<size_t>(h->gal_counts.n, 1));
  int* bad = h->gal_counts.get();
  MCK(cudaMemsetAsync(bad, 0, sizeof(int), h->stream));
  k_gal_check<<<ceil_div(std::max(fem_nodes, coarse_nodes), kGalTpb), kGalTpb, 0, h->stream>>>(
      m, fem_nodes, coarse_nodes, coarse_block_nodes, bad); MLAUNCHED(h);
  MCK(cudaGetLastError());
  const int b = read_int(h, bad);
  return (b & 1) ? 1 : (b & 2) ? 2 : (b & 4) ? 3 : 0;
}

MergedKeys galerkin_keys(maspcg_handle* h, const GalerkinMap& m, const int* rows, const int* cols, int n)
{
  cudaStream_t st = h->stream;
  h->gal_counts.resize(2 * (size_t)n + 2);
  int* counts = h->gal_counts.get();
  int* offsets = counts + n;
  int* bad = offsets + n;
  MCK(cudaMemsetAsync(bad, 0, sizeof(int), st));
  const int grid = ceil_div(n, kGalTpb);
  k_gal_count<<<grid, kGalTpb, 0, st>>>(m, rows, cols, n, counts, bad); MLAUNCHED(h);
  size_t need = 0;
  MCK(cub::DeviceScan::ExclusiveSum(nullptr, need, counts, offsets, n, st));
  h->cub_tmp.resize(std::max(need, h->cub_tmp.n));
  size_t tb = h->cub_tmp.cap;
  MCK(cub::DeviceScan::ExclusiveSum(h->cub_tmp.get(), tb, counts, offsets, n, st));
  MREQ(read_int(h, bad) == 0, MASPCG_ERR_INVALID_ARGUMENT, "fine block index outside [0, fine_blocks)");
  int last[2] = {0, 0};
  MCK(cudaMemcpyAsync(&last[0], offsets + (n - 1), sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaMemcpyAsync(&last[1], counts + (n - 1), sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
  const long long expanded = (long long)last[0] + last[1];
  MREQ(expanded <= 0x3fffffffLL, MASPCG_ERR_CAPACITY, "expanded coarse triplets exceed 2^30");
  const size_t room = (size_t)std::max(expanded, 1LL);
  h->gal_rows.resize(room);
  h->gal_cols.resize(room);
  h->gal_src.resize(room);
  h->gal_weight.resize(room);
  k_gal_emit<<<grid, kGalTpb, 0, st>>>(m, rows, cols, offsets, n, h->gal_rows.get(), h->gal_cols.get(),
                                       h->gal_src.get(), h->gal_weight.get()); MLAUNCHED(h);
  MCK(cudaGetLastError());
  return merge_keys(h, h->gal_rows.get(), h->gal_cols.get(), (int)expanded);
}

bool galerkin_values(maspcg_handle* h, const MergedKeys& k, const double* vals, int* rows_out, int* cols_out,
                     double* vals_out)
{
  if (k.count == 0) return true;
  int* bad = h->gal_counts.get();
  MCK(cudaMemsetAsync(bad, 0, sizeof(int), h->stream));
  k_gal_sum<<<ceil_div(9LL * k.count, kGalTpb), kGalTpb, 0, h->stream>>>(k, h->gal_src.get(), h->gal_weight.get(),
                                                                        vals, rows_out, cols_out, vals_out, bad);
  MLAUNCHED(h);
  MCK(cudaGetLastError());
  return read_int(h, bad) == 0;
}

void galerkin_restrict(maspcg_handle* h, const GalerkinMap& m, const double* fine, double* coarse, int coarse_blocks)
{
  cudaStream_t st = h->stream;
  h->gal_counts.resize(std::max<size_t>(h->gal_counts.n, 1));
  int* bad = h->gal_counts.get();
  MCK(cudaMemsetAsync(bad, 0, sizeof(int), st));
  MCK(cudaMemsetAsync(coarse, 0, sizeof(double) * 3 * (size_t)coarse_blocks, st));
  if (m.fine_blocks > 0) {
    k_gal_restrict<<<ceil_div(m.fine_blocks, kGalTpb), kGalTpb, 0, st>>>(m, fine, coarse, bad); MLAUNCHED(h);
  }
  MREQ(read_int(h, bad) == 0, MASPCG_ERR_INVALID_ARGUMENT, "non-finite fine right-hand side");
}

void galerkin_prolong(maspcg_handle* h, const GalerkinMap& m, const double* coarse, double* fine)
{
  if (m.fine_blocks <= 0) return;
  k_gal_prolong<<<ceil_div(m.fine_blocks, kGalTpb), kGalTpb, 0, h->stream>>>(m, coarse, fine); MLAUNCHED(h);
  MCK(cudaGetLastError());
}

}  // namespace maspcg
