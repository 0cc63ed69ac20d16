// factor.cu -- the MAS domain inverses: gather, FP64 factorisation and store of
// one domain per CTA (MAS32: 96x96; CEMAS16: 48x48).
//
// The reference inverts each domain by Gauss-Jordan elimination without
// pivoting (__inverse6_P96x96, TraditionalMAS32Preconditioner.cu:1099-1146).
// FP32 storage runs that elimination (k_domain_eliminate).  16-bit storage
// takes the same pivots through A = L L^T and keeps the scaled factor W S^-1,
// W = L^-1 (k_domain_invert).  A pivot <= 0 or not finite counts the domain as
// failed and stands as 1 in both.
#include "maspcg_internal.cuh"

namespace maspcg {
namespace {

// ---- FP32 storage ----------------------------------------------------------

constexpr int kElimSide = 6;  // a thread's square of the matrix: two by two blocks

// In-place Gauss-Jordan of the whole matrix in registers, kB/2 x kB/2 threads
// with a 6x6 square each.  A step publishes the pivot's row and column, waits
// once, and is 36 multiply-adds per thread with two CTAs per SM to hide each
// other's wait.  Every element takes the reference's operations in the
// reference's order: x - (m / pivot) p per step, so the result is that of the
// elimination on the matrix as it is -- also where CEMAS16's assembly rules
// leave a coarse diagonal block unsymmetric, which a Cholesky factor of one
// triangle does not see (6e-3 of an inverse's largest entry on such a domain).
// Bound by the chain of steps (wait, reciprocal, 36 multiply-adds, next pivot).
// Whole factor stage with coarse sums: 1.07 ms for 3,347 domains of 96 rows and
// 0.68 for 7,675 of 48, where a 3x3 block per thread (1,024 and 512 threads, one
// CTA per SM) took 1.74 and 1.14, and the tensor-tile Cholesky below with a
// closing W^T W 0.89 and 0.68.
template <int kB>
__global__ void __launch_bounds__(kB * kB / 4, kB == 32 ? 2 : 8) k_domain_eliminate(FactorArgs a, int dom_offset)
{
  constexpr int kG = kB / 2, kT = kG * kG, kN = 3 * kB, kS = kElimSide;
  constexpr int kDiag = kB / 2 + 1, kElems = kDiag * 9 * kB;
  __shared__ __align__(16) double half[kN / 2 * kN];  // half the rows at a time; the record afterwards
  __shared__ __align__(16) double row[2][kN], col[2][kN];
  __shared__ double recip[2];
  __shared__ int rp[kB + 1], fail;
  static_assert(kElems * sizeof(float) <= sizeof(half) && kElems % 4 == 0, "the record fits the half matrix");
  const int tid = threadIdx.x, ty = tid / kG, tx = tid % kG;
  const int dom = blockIdx.x + dom_offset, d0 = a.lv.dom_begin[1];
  if (tid == 0) fail = 0;

  // ---- the domain's blocks (rows 6 ty, columns 6 tx)
  double acc[kS][kS];
  if (dom < d0) {
    const int row0 = a.fem_off + kB * dom;  // first internal row
    for (int e = tid; e <= kB; e += kT) rp[e] = a.rowptr[row0 + e];
    for (int h = 0; h < 2; ++h) {
      for (int e = tid; e < kN / 2 * kN / 2; e += kT) reinterpret_cast<double2*>(half)[e] = make_double2(0.0, 0.0);
      __syncthreads();
      const int r0 = h * kG, end = rp[r0 + kG];
      for (int t = rp[r0] + tid; t < end; t += kT) {  // a thread per block (a merged block appears once)
        const int bc = a.colidx[t] - row0;
        if (bc < 0 || bc >= kB) continue;
        int lo = r0, hi = r0 + kG;  // row lo: rp[lo] <= t < rp[lo + 1]
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (rp[mid] <= t) lo = mid; else hi = mid;
        }
        if (kB == 16 && bc != lo) {
          // CEMAS16 drops a pair whose slot order runs against its vertex order
          const int* pm = a.pmr + kB * dom;
          if ((pm[lo] < pm[bc]) != (lo < bc)) continue;
        }
        double* m = half + 3 * (lo - r0) * kN + 3 * bc;
#pragma unroll
        for (int e = 0; e < 9; ++e) m[e / 3 * kN + e % 3] = __ldcs(a.val64 + 9 * (size_t)t + e);
      }
      __syncthreads();
      if (ty / (kG / 2) == h) {
#pragma unroll
        for (int i = 0; i < kS; ++i)
#pragma unroll
          for (int k = 0; k < kS; ++k) acc[i][k] = half[(kS * ty + i - h * kN / 2) * kN + kS * tx + k];
      }
      __syncthreads();
    }
  } else {
#pragma unroll
    for (int bi = 0; bi < 2; ++bi)
#pragma unroll
      for (int bk = 0; bk < 2; ++bk) {
        const double* src = a.coarse64 + (((size_t)(dom - d0) * kB + 2 * ty + bi) * kB + 2 * tx + bk) * 9;
#pragma unroll
        for (int e = 0; e < 9; ++e) acc[3 * bi + e / 3][3 * bk + e % 3] = src[e];
      }
  }
  if (ty == tx)  // padding slots: zero diagonal -> 1
#pragma unroll
    for (int i = 0; i < kS; ++i)
      if (acc[i][i] == 0.0) acc[i][i] = 1.0;

  // ---- elimination; two copies of the row and column, so one barrier a step
  for (int q = 0; q < kG; ++q) {
#pragma unroll
    for (int c = 0; c < kS; ++c) {
      const int b = c & 1;
      if (tx == q) {
#pragma unroll
        for (int i = 0; i < kS; ++i) col[b][kS * ty + i] = acc[i][c];
      }
      if (ty == q) {
#pragma unroll
        for (int k = 0; k < kS; ++k) row[b][kS * tx + k] = acc[c][k];
        if (tx == q) {
          double pivot = acc[c][c];
          if (!(pivot > 0.0) || !isfinite(pivot)) fail = 1, pivot = 1.0;
          recip[b] = 1.0 / pivot;
        }
      }
      __syncthreads();
      const double inv = recip[b];
      double f[kS];
#pragma unroll
      for (int i = 0; i < kS; ++i) f[i] = col[b][kS * ty + i] * inv;
#pragma unroll
      for (int k = 0; k < kS; ++k) {
        const double p = row[b][kS * tx + k];
#pragma unroll
        for (int i = 0; i < kS; ++i) acc[i][k] = fma(-f[i], p, acc[i][k]);
        if (ty == q) acc[c][k] = p * inv;
      }
      if (tx == q) {
#pragma unroll
        for (int i = 0; i < kS; ++i) acc[i][c] = -f[i];
        if (ty == q) acc[c][c] = inv;
      }
    }
  }
  __syncthreads();
  if (tid == 0 && fail) atomicAdd(a.failed, 1);

  // ---- wrapped diagonals: block (l, (l + d) % kB) at [d][3i + j][l], the last
  // diagonal for l < kB / 2 only
  float* out = reinterpret_cast<float*>(half);
#pragma unroll
  for (int bi = 0; bi < 2; ++bi)
#pragma unroll
    for (int bk = 0; bk < 2; ++bk) {
      const int l = 2 * ty + bi, d = (2 * tx + bk - l) & (kB - 1);
      if (d > kB / 2) continue;
      const bool zero = d == kB / 2 && l >= kB / 2;
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          // CEMAS16 stores the diagonal blocks with their lower elements
          // taken from the upper ones (MASPreconditioner.cu:705-711)
          const bool upper = kB == 16 && d == 0 && i > j;
          const double v = upper ? acc[3 * bi + j][3 * bk + i] : acc[3 * bi + i][3 * bk + j];
          out[(9 * d + 3 * i + j) * kB + l] = zero ? 0.f : (float)v;
        }
    }
  __syncthreads();
  float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.inv) + (size_t)dom * kElems);
  for (int e = tid; e < kElems / 4; e += kT) dst[e] = reinterpret_cast<const float4*>(out)[e];
}

// ---- 16-bit storage --------------------------------------------------------
//
// The lower triangle lives in shared memory as 8x8 FP64 tiles (40 KB), and
// everything but the 8x8 diagonal tiles runs on the FP64 tensor instruction
// mma.m8n8k4.  Each step k: the tiles below the diagonal times L_kk^-T, then the
// trailing tiles less L_ik L_jk^T, while the first warp updates the next
// diagonal tile first and factors it (its chain of eight pivots is the longest
// of the step).  W needs no second factorisation-like sweep: with
// H_kj = -L_kj L_jj^-1, row i of W is
//   W_ii = L_ii^-1,  W_ij = sum over k = j+1 .. i of W_ik H_kj,
// so each warp runs whole rows in registers and the rows need three barriers.
// Bound by the chain of twelve steps: 0.73 ms for 8,192 domains in BF16 storage,
// where a gather and a 3x3-block Cholesky took 2.7.
constexpr int kFactorTpb = 128;

// Element (r, c) of an 8x8 tile: row-major, the halves of rows with bit 1 set
// swapped, so that the row-wise and column-wise operand loads of mma.m8n8k4
// (four consecutive rows or columns per half-warp) fall in distinct banks.
__device__ __forceinline__ int tpos(int r, int c) { return 8 * r + (c ^ ((r & 2) << 1)); }
__device__ __forceinline__ int tile_of(int i, int j) { return (i * (i + 1) / 2 + j) * 64; }

__device__ __forceinline__ void dmma(double c[2], double a, double b)
{
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// Operand element of k step s (columns or rows 4s .. 4s+3): entry (g, 4s + q)
// of a tile read along its rows, entry (4s + q, g) read along its columns, for
// lane = 4g + q.
__device__ __forceinline__ double by_row(const double* t, int g, int q, int s) { return t[tpos(g, 4 * s + q)]; }
__device__ __forceinline__ double by_col(const double* t, int g, int q, int s) { return t[tpos(4 * s + q, g)]; }
__device__ __forceinline__ void store_tile(double* t, int g, int q, const double c[2])
{
  *reinterpret_cast<double2*>(t + tpos(g, 2 * q)) = make_double2(c[0], c[1]);
}

// One warp: L L^T of the 8x8 tile t (its lower triangle), then t = L^-1 with
// zeros above the diagonal.  Lane r (mod 8) holds row r; scratch: 64 doubles.
__device__ __forceinline__ bool factor_diag(double* t, double* scratch, int lane)
{
  const int r = lane & 7;
  double a[8], inv[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) a[c] = t[tpos(r, c)];
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    double p = __shfl_sync(kFull, a[k], k);
    if (!(p > 0.0) || !isfinite(p)) ok = false, p = 1.0;
    inv[k] = rsqrt(p);
    const double l = (r == k ? p : a[k]) * inv[k];
    a[k] = l;
#pragma unroll
    for (int c = k + 1; c < 8; ++c) a[c] = fma(-l, __shfl_sync(kFull, l, c), a[c]);
  }
  if (lane < 8) {
#pragma unroll
    for (int c = 0; c < 8; ++c) scratch[8 * r + c] = a[c];
  }
  __syncwarp();
  // column r of L^-1: forward substitution on the identity
  double x[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = i == r ? 1.0 : 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    x[k] *= inv[k];
#pragma unroll
    for (int i = k + 1; i < 8; ++i) x[i] = fma(-scratch[8 * i + k], x[k], x[i]);
  }
  if (lane < 8) {
#pragma unroll
    for (int i = 0; i < 8; ++i) t[tpos(i, r)] = x[i];
  }
  __syncwarp();
  return ok;
}

template <typename T>
__device__ __forceinline__ unsigned short to16(double v);
template <>
__device__ __forceinline__ unsigned short to16<__nv_bfloat16>(double v)
{
  return __bfloat16_as_ushort(__float2bfloat16_rn((float)v));
}
template <>
__device__ __forceinline__ unsigned short to16<__half>(double v) { return __half_as_ushort(__float2half_rn((float)v)); }

template <typename TI>
__global__ void __launch_bounds__(kFactorTpb, 5) k_domain_invert(FactorArgs a, int dom_offset)
{
  constexpr int kB = kBank, kT = kFactorTpb, kW = kT / 32;
  constexpr int kN = 3 * kB, kR = kN / 8;  // rows, tile rows
  constexpr int kTiles = kR * (kR + 1) / 2;
  __shared__ __align__(16) double T[kTiles * 64];
  __shared__ double scratch[64];
  __shared__ float colscale[kN];
  __shared__ int rp[kB + 1], fail;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int dom = blockIdx.x + dom_offset;
  const int d0 = a.lv.dom_begin[1];

  // ---- the domain's lower blocks
  for (int e = tid; e < kTiles * 32; e += kT) reinterpret_cast<double2*>(T)[e] = make_double2(0.0, 0.0);
  if (tid == 0) fail = 0;
  const int row0 = a.fem_off + kB * dom;  // level 0: first internal row
  if (dom < d0 && tid <= kB) rp[tid] = a.rowptr[row0 + tid];
  __syncthreads();
  auto put = [&](int br, int bc, const double* v) {  // 3x3 block (br, bc), br >= bc, row-major
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int r = 3 * br + i, c = 3 * bc + j;
        if (r >= c) T[tile_of(r >> 3, c >> 3) + tpos(r & 7, c & 7)] = v[3 * i + j];
      }
  };
  if (dom < d0) {
    // the rows of a level-0 domain are consecutive, and so are their blocks: a
    // thread per block, two at a time (a merged block appears once)
    const int end = rp[kB];
    for (int t0 = rp[0] + tid; t0 < end; t0 += 2 * kT) {
      int br[2], bc[2];
      double v[2][9];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = t0 + h * kT;
        br[h] = -1;
        bc[h] = t < end ? a.colidx[t] - row0 : -1;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = t0 + h * kT;
        if (bc[h] < 0 || bc[h] >= kB) continue;
        int lo = 0, hi = kB;  // row lo: rp[lo] <= t < rp[lo + 1]
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (rp[mid] <= t) lo = mid; else hi = mid;
        }
        if (bc[h] > lo) continue;
        br[h] = lo;
#pragma unroll
        for (int e = 0; e < 9; ++e) v[h][e] = __ldcs(a.val64 + 9 * (size_t)t + e);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (br[h] >= 0) put(br[h], bc[h], v[h]);
    }
  } else {
    for (int e = tid; e < kB * (kB + 1) / 2; e += kT) {
      int br = (int)((sqrtf(8.f * e + 1.f) - 1.f) * 0.5f);
      while (br * (br + 1) / 2 > e) --br;
      while ((br + 1) * (br + 2) / 2 <= e) ++br;
      const int bc = e - br * (br + 1) / 2;
      const double* src = a.coarse64 + (((size_t)(dom - d0) * kB + br) * kB + bc) * 9;
      double v[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) v[k] = src[k];
      put(br, bc, v);
    }
  }
  __syncthreads();
  for (int r = tid; r < kN; r += kT) {  // padding slots: zero diagonal -> 1
    double& d = T[tile_of(r >> 3, r >> 3) + tpos(r & 7, r & 7)];
    if (d == 0.0) d = 1.0;
  }
  __syncthreads();

  // ---- A = L L^T; the diagonal tiles end as L_kk^-1
  if (w == 0 && !factor_diag(T, scratch, lane)) fail = 1;
  __syncthreads();
  for (int k = 0; k + 1 < kR; ++k) {
    {
      const double* D = T + tile_of(k, k);
      const double b0 = by_row(D, g, q, 0), b1 = by_row(D, g, q, 1);  // L_kk^-T
      for (int i = k + 1 + w; i < kR; i += kW) {
        double* P = T + tile_of(i, k);
        const double a0 = by_row(P, g, q, 0), a1 = by_row(P, g, q, 1);
        double c[2] = {0.0, 0.0};
        dmma(c, a0, b0);
        dmma(c, a1, b1);
        __syncwarp();
        store_tile(P, g, q, c);
      }
    }
    __syncthreads();
    // trailing tiles (i, j), k < j <= i, less L_ik L_jk^T: warp 0 takes the next
    // diagonal tile and factors it, the others the rest
    auto update = [&](int i, int j) {
      const double *Li = T + tile_of(i, k), *Lj = T + tile_of(j, k);
      double* C = T + tile_of(i, j);
      const double2 c2 = *reinterpret_cast<const double2*>(C + tpos(g, 2 * q));
      double c[2] = {c2.x, c2.y};
      dmma(c, -by_row(Li, g, q, 0), by_row(Lj, g, q, 0));
      dmma(c, -by_row(Li, g, q, 1), by_row(Lj, g, q, 1));
      store_tile(C, g, q, c);
    };
    if (w == 0) {
      update(k + 1, k + 1);
      __syncwarp();
      if (!factor_diag(T + tile_of(k + 1, k + 1), scratch, lane)) fail = 1;
    } else {
      int i = k + 2, j = k + 1;  // the remaining tiles in row order, dealt to warps 1 ..
      for (int skip = w - 1; i < kR; skip = kW - 1) {
        j += skip;
        while (i < kR && j > i) j = j - i + k, ++i;
        if (i < kR) update(i, j);
      }
    }
    __syncthreads();
  }

  // ---- H_kj = -L_kj L_jj^-1 in place
  for (int t = w; t < kTiles; t += kW) {
    int i = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
    while (i * (i + 1) / 2 > t) --i;
    while ((i + 1) * (i + 2) / 2 <= t) ++i;
    const int j = t - i * (i + 1) / 2;
    if (i == j) continue;
    double* P = T + 64 * t;
    const double* D = T + tile_of(j, j);
    const double a0 = -by_row(P, g, q, 0), a1 = -by_row(P, g, q, 1);
    double c[2] = {0.0, 0.0};
    dmma(c, a0, by_col(D, g, q, 0));
    dmma(c, a1, by_col(D, g, q, 1));
    __syncwarp();
    store_tile(P, g, q, c);
  }
  __syncthreads();
  // ---- W = L^-1, kW rows at a time from the last: a row's tiles stay in
  // registers as A operands; H rows past the current ones are no longer read
  for (int top = kR; top > 0; top -= kW) {
    const int i = top - 1 - w;
    double wa[kR][2];
    if (i >= 0) {
#pragma unroll
      for (int j = kR - 1; j >= 0; --j) {
        if (j > i) continue;
        if (j == i) {
          wa[j][0] = by_row(T + tile_of(i, i), g, q, 0);
          wa[j][1] = by_row(T + tile_of(i, i), g, q, 1);
          continue;
        }
        double c[2] = {0.0, 0.0};
#pragma unroll
        for (int k = 1; k < kR; ++k) {
          if (k <= j || k > i) continue;
          const double* B = T + tile_of(k, j);
          dmma(c, wa[k][0], by_col(B, g, q, 0));
          dmma(c, wa[k][1], by_col(B, g, q, 1));
        }
        // accumulator layout (columns 2q, 2q + 1) to operand layout (columns 4s + q)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const int from = (lane & ~3) | (2 * s + (q >> 1));
          const double lo = __shfl_sync(kFull, c[0], from), hi = __shfl_sync(kFull, c[1], from);
          wa[j][s] = (q & 1) ? hi : lo;
        }
      }
    }
    __syncthreads();
    if (i >= 0) {
#pragma unroll
      for (int j = 0; j < kR; ++j)
        if (j < i) {
          double* P = T + tile_of(i, j);
          P[tpos(g, q)] = wa[j][0];
          P[tpos(g, 4 + q)] = wa[j][1];
        }
    }
  }
  __syncthreads();
  if (tid == 0 && fail) atomicAdd(a.failed, 1);

  // ---- column scales (largest entry of each column of W) and the scaled
  // 16-bit tiles, 16 bytes (8 elements of a row) per thread
  for (int c = tid; c < kN; c += kT) {
    float m = 0.f;
#pragma unroll 8
    for (int r = 0; r < kN; ++r)
      if (r >= c) m = fmaxf(m, (float)fabs(T[tile_of(r >> 3, c >> 3) + tpos(r & 7, c & 7)]));
    if (!(m > 0.f) || !isfinite(m)) m = 1.f;
    colscale[c] = m;
    a.scale[(size_t)dom * 96 + c] = m;
  }
  __syncthreads();
  uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<unsigned short*>(a.inv) + (size_t)dom * kInvElems16);
  for (int e = tid; e < kInvElems16 / 8; e += kT) {
    const int t16 = e >> 5, r = (e >> 1) & 15, half = (e ^ (r >> 2)) & 1;  // inv16_pos
    int I = 0;
    while ((I + 1) * (I + 2) / 2 <= t16) ++I;
    const int ti = 2 * I + (r >> 3), tj = 2 * (t16 - I * (I + 1) / 2) + half;
    unsigned u[4] = {0u, 0u, 0u, 0u};
    if (tj <= ti) {
      const double* src = T + tile_of(ti, tj);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const double v = src[tpos(r & 7, k)] / (double)colscale[8 * tj + k];
        u[k >> 1] |= (unsigned)to16<TI>(v) << (16 * (k & 1));
      }
    }
    dst[e] = make_uint4(u[0], u[1], u[2], u[3]);
  }
}

}  // namespace

// Inverses of the domains [g0, g0 + n).
void factor_domains(maspcg_handle* h, const FactorArgs& a, int g0, int n, int storage)
{
  if (n <= 0) return;
  if (h->bank == 16)
    k_domain_eliminate<16><<<n, 64, 0, h->stream>>>(a, g0);
  else if (storage == MASPCG_INV_FP32)
    k_domain_eliminate<32><<<n, 256, 0, h->stream>>>(a, g0);
  else if (storage == MASPCG_INV_BF16)
    k_domain_invert<__nv_bfloat16><<<n, kFactorTpb, 0, h->stream>>>(a, g0);
  else
    k_domain_invert<__half><<<n, kFactorTpb, 0, h->stream>>>(a, g0);
  MLAUNCHED(h);
}

}  // namespace maspcg
