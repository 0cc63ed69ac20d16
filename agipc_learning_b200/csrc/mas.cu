// mas.cu -- MAS domain matrices, inverses and the preconditioner apply:
// TraditionalMAS32 (32-slot banks, 96x96 domains) and, where marked, CEMAS16
// (16-slot banks, 48x48 domains, MASPreconditioner.cu).
//
// Build (once per Newton step, after the hierarchy):
//   * member lists: for every coarse level a stable radix sort of the fine
//     slots by their level node, so each coarse node owns a contiguous,
//     fixed-order list of fine rows;
//   * the Galerkin sums P^T A P of the coarse domains (k_coarse_assemble), as
//     prepare_hessian_bcoo_kernel and prepare_hessian_bcoo_sum_kernel form them
//     (TraditionalMAS32Preconditioner.cu:2234-2464); a level-0 domain is a
//     diagonal block of the matrix itself;
//   * one CTA per domain gathers, factors and stores it (factor.cu): zero
//     diagonals become 1 (expand_symmetric_mas32 :1062-1096); FP32 storage
//     keeps the inverse as 17 wrapped diagonals x 9 elements x 32 lanes, 16-bit
//     storage the scaled Cholesky factor of the inverse (BF16/FP16 tiles);
//   * CEMAS16: the same with 16-slot banks (48x48, FP32, 9 wrapped
//     diagonals), with its assembly rules.
// Apply (every PCG iteration): MAS32 runs the coarse domains as one
// kernel beside a tensor-core level-0 apply of the 16-bit records (or a warp
// per domain on FP32 records, each stored block used for both triangles
// through a shuffle); CEMAS16 runs half a warp per domain (see the CEMAS16
// apply kernels).
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "maspcg_internal.cuh"
#include "pcg_device.cuh"
#include "tma.cuh"
#include "mas_args.cuh"

namespace maspcg {
namespace {

constexpr int kTpb = 256;

// ------------------------------------------------------------------ build --

__global__ void k_member_keys(const int* __restrict__ cmap, int c0, int count, unsigned* keys, int* vals)
{
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= c0) return;
  const int c = cmap[s];
  keys[s] = c >= 0 ? (unsigned)c : (unsigned)count;
  vals[s] = s;
}

template <int kB>
__device__ __forceinline__ int pkb(int a, int b) { return kB * a - a * (a + 1) / 2 + b; }

// CEMAS16 assembly (MASPreconditioner.cu prepare_hessian_bcoo_kernel
// :1822-1914 and prepare_hessian_bcoo_sum_kernel :1916-2037) differs from
// MAS32 on the entries (rs, u) of a fine row whose column lies in the row's
// own level-0 bank (rs, u: level-0 slots):
//  * an in-bank upper block is kept only when its column's slot is not
//    below its row's: a pair whose slot order runs against its vertex order
//    is not transposed (MAS32 transposes it) but dropped, at every level;
//  * in a bank that is one component, the coarse diagonal block receives
//    the entries of rows (2k, 2k+1) through the entry (2k, 0), so a row
//    whose even partner slot is padding adds nothing to the coarse levels.
// pmr: part_map_real; prefix_orig: components per level-0 bank (null for
// the level-0 domain itself).
__device__ __forceinline__ bool cemas16_drops(int rs, int u, const int* __restrict__ pmr,
                                              const int* __restrict__ prefix_orig)
{
  if ((u >> 4) != (rs >> 4)) return false;
  if (u != rs && ((pmr[rs] < pmr[u]) != (rs < u))) return true;
  return prefix_orig && prefix_orig[rs >> 4] == 1 && pmr[rs & ~1] < 0;
}

// Accumulate the fine row `row` into the owner lanes: every block whose
// column's level node `B` lies in bank `bank` is added by lane B % kB.
// Staging: 16 blocks per chunk through the warp's shared-memory slots, so
// the 9 doubles of a block are read coalesced and summed in block order.
// kB = 16 applies the CEMAS16 rules (pmr non-null).
template <int kB>
__device__ __forceinline__ void gather_row(const int* __restrict__ rowptr, const int* __restrict__ colidx,
                                           const double* __restrict__ val64, const int* __restrict__ cmap, int row,
                                           int fem_off, int c0, int bank, int lane, double* stage, int* sdest,
                                           double acc[9], const int* __restrict__ pmr = nullptr,
                                           const int* __restrict__ prefix_orig = nullptr)
{
  const int rs = rowptr[row], re = rowptr[row + 1];
  for (int t0 = rs; t0 < re; t0 += 16) {
    const int nblk = min(16, re - t0);
    if (lane < nblk) {
      int dest = -1;
      const int u = colidx[t0 + lane] - fem_off;
      if (u >= 0 && u < c0) {
        const int B = cmap ? cmap[u] : u;
        if (B >= 0 && B / kB == bank) dest = B % kB;
        if (kB == 16 && dest >= 0 && cemas16_drops(row - fem_off, u, pmr, prefix_orig)) dest = -1;
      }
      sdest[lane] = dest;
    }
    const double* src = val64 + 9 * (size_t)t0;
    for (int q = lane; q < nblk * 9; q += 32) stage[q] = src[q];
    __syncwarp();
    for (int j = 0; j < nblk; ++j) {
      if (sdest[j] == lane) {
#pragma unroll
        for (int e = 0; e < 9; ++e) acc[e] += stage[9 * j + e];
      }
    }
    __syncwarp();
  }
}

struct CoarseArgs {
  const int* pmr;          // CEMAS16 rules (bank 16 only)
  const int* prefix_orig;
  const int* perm[kMaxLevels];
  const int* cmap[kMaxLevels];
  int slice_base[kMaxLevels + 1];  // first warp item of each level (levels >= 1)
  int dom_begin[kMaxLevels + 1];
  int levelnum;
  int slice_rows;
  int nv;
  const int* rowptr;
  const int* colidx;
  const double* val64;
  int fem_off, c0;
  double* coarse64;  // (domains - dom_begin[1]) x kB x kB blocks, row-major 3x3
};

// Coarse-level Galerkin sums: one warp per slice of a level's member list
// (fine rows grouped by node); the slice's partial block-row is reduced in
// registers and added to the FP64 coarse domain matrix once per node.
template <int kB>
__global__ void __launch_bounds__(256) k_coarse_assemble(CoarseArgs a)
{
  __shared__ double stage_s[8][16 * 9];
  __shared__ int sdest_s[8][16];
  const int item = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31, lw = threadIdx.x >> 5;
  int L = 1;
  while (L + 1 < a.levelnum && item >= a.slice_base[L + 1]) ++L;
  if (item >= a.slice_base[a.levelnum]) return;
  const int sl = item - a.slice_base[L];
  const int p0 = sl * a.slice_rows, p1 = min(p0 + a.slice_rows, a.nv);
  const int* perm = a.perm[L];
  const int* cmap = a.cmap[L];
  double acc[9];
#pragma unroll
  for (int e = 0; e < 9; ++e) acc[e] = 0.0;
  int node = -1;
  auto flush = [&](int A) {
    if (lane >= kB) return;
    const int local = a.dom_begin[L] + A / kB - a.dom_begin[1];
    double* dst = a.coarse64 + (((size_t)local * kB + A % kB) * kB + lane) * 9;
#pragma unroll
    for (int e = 0; e < 9; ++e)
      if (acc[e] != 0.0) atomicAdd(dst + e, acc[e]);
  };
  for (int pos = p0; pos < p1; ++pos) {
    const int v = perm[pos];
    const int A = cmap[v];
    if (A != node) {
      if (node >= 0) flush(node);
#pragma unroll
      for (int e = 0; e < 9; ++e) acc[e] = 0.0;
      node = A;
    }
    gather_row<kB>(a.rowptr, a.colidx, a.val64, cmap, a.fem_off + v, a.fem_off, a.c0, A / kB, lane, stage_s[lw],
                   sdest_s[lw], acc, a.pmr, a.prefix_orig);
  }
  if (node >= 0) flush(node);
}

// The packed upper FP64 blocks of a domain (the matrix its stored inverse was
// built from, before the zero-diagonal rule): one CTA per domain, one warp per
// block row (for kB = 16 lanes 16..31 only help stage the gathered rows).
template <int kB>
__global__ void __launch_bounds__(32 * kB) k_domain_gather(FactorArgs a)
{
  __shared__ double stage[kB][16 * 9];
  __shared__ int sdest[kB][16];
  const int g = blockIdx.x, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double acc[9];
#pragma unroll
  for (int e = 0; e < 9; ++e) acc[e] = 0.0;
  const int d0 = a.lv.dom_begin[1];
  if (g < d0) {
    const int slot = kB * g + w;
    if (a.pmr[slot] >= 0)
      gather_row<kB>(a.rowptr, a.colidx, a.val64, nullptr, a.fem_off + slot, a.fem_off, a.c0, g, lane, stage[w],
                     sdest[w], acc, a.pmr);
  } else if (lane < kB) {
    const double* src = a.coarse64 + (((size_t)(g - d0) * kB + w) * kB + lane) * 9;
#pragma unroll
    for (int e = 0; e < 9; ++e) acc[e] = src[e];
  }
  if (lane >= w && lane < kB) {
    double* o = a.assembled + ((size_t)g * (kB * (kB + 1) / 2) + pkb<kB>(w, lane)) * 9;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) o[i + 3 * j] = acc[3 * i + j];
  }
}

// ------------------------------------------------------------------ apply --

// z = (M x) for one domain held by one warp, FP32 storage: the symmetric
// inverse, lane l holding block (l, (l + d) % 32) of diagonal d = 0..16, each
// stored block serving both triangles through a shuffle.  x, y: the lane's
// three rows.
__device__ __forceinline__ void domain_apply(const float* __restrict__ inv, int lane, const float x[3], float y[3])
{
  const float x0 = x[0], x1 = x[1], x2 = x[2];
  float y0 = 0.f, y1 = 0.f, y2 = 0.f;
#pragma unroll
  for (int d = 0; d < kDiags; ++d) {
    const int c = (lane + d) & 31;
    const float c0 = __shfl_sync(kFull, x0, c), c1 = __shfl_sync(kFull, x1, c), c2 = __shfl_sync(kFull, x2, c);
    float B[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) B[e] = inv[(d * 9 + e) * kBank + lane];
    y0 += B[0] * c0 + B[1] * c1 + B[2] * c2;
    y1 += B[3] * c0 + B[4] * c1 + B[5] * c2;
    y2 += B[6] * c0 + B[7] * c1 + B[8] * c2;
    if (d != 0) {
      const float t0 = B[0] * x0 + B[3] * x1 + B[6] * x2;
      const float t1 = B[1] * x0 + B[4] * x1 + B[7] * x2;
      const float t2 = B[2] * x0 + B[5] * x1 + B[8] * x2;
      const int src = (lane - d) & 31;
      y0 += __shfl_sync(kFull, t0, src);
      y1 += __shfl_sync(kFull, t1, src);
      y2 += __shfl_sync(kFull, t2, src);
    }
  }
  y[0] = y0;
  y[1] = y1;
  y[2] = y2;
}

// ---- tensor-core apply of a 16-bit factored record -------------------------
//
// M = S V^T V S with V the scaled lower factor (96 x 96, 21 tiles of 16 x 16
// in shared memory, inv16_pos).  Pass 1, t = V (S x), multiplies each tile by
// the matching 16 entries of the vector with mma.m16n8k16 (the tile as A);
// pass 2, z = V^T t, does the same with the tiles loaded transposed
// (ldmatrix .trans).  The FP32 vector enters the 16-bit B operand as three
// terms, hi + mid + lo (each the rounding of what the previous ones leave),
// in columns 0, 1, 2 of B, so the products carry the vector to FP32 precision
// and the FP32 accumulators of the three columns are added afterwards.  FP16
// records scale the vector by a power of two (its largest entry to [1, 2))
// first, as FP16 has a narrow exponent range; the scaling is exact.
constexpr int kPartStride = 104;             // 16-bit split terms: 3 rows of 104 (bank spread)
constexpr int kApplyScratch = 1024;          // per warp: 96 FP32 + 3 x 104 16-bit
constexpr int kRecBytes16 = kInvElems16 * 2;  // 10,752

template <typename TI>
struct Mma16;
template <>
struct Mma16<__nv_bfloat16> {
  static constexpr bool kNormalize = false;
  static __device__ __forceinline__ void mma(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1)
  {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  static __device__ __forceinline__ unsigned short to16(float v) { return __bfloat16_as_ushort(__float2bfloat16_rn(v)); }
  static __device__ __forceinline__ float from16(unsigned short u) { return __uint_as_float((uint32_t)u << 16); }
};
template <>
struct Mma16<__half> {
  static constexpr bool kNormalize = true;
  static __device__ __forceinline__ void mma(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1)
  {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
  static __device__ __forceinline__ unsigned short to16(float v) { return __half_as_ushort(__float2half_rn(v)); }
  static __device__ __forceinline__ float from16(unsigned short u) { return __half2float(__ushort_as_half(u)); }
};

__device__ __forceinline__ void ldsm(uint32_t addr, uint32_t a[4])
{
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm_t(uint32_t addr, uint32_t a[4])
{
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
               : "r"(addr)
               : "memory");
}

// Power-of-two factor taking the warp's largest |v| to [1, 2) (1 when the
// vector is zero or not finite), and its inverse.
__device__ __forceinline__ void pow2_normalizer(const float v[3], float& f, float& fi)
{
  const float m = fmaxf(fabsf(v[0]), fmaxf(fabsf(v[1]), fabsf(v[2])));
  const unsigned mb = __reduce_max_sync(kFull, __float_as_uint(m));
  int ex = (int)(mb >> 23) - 127;
  if (mb == 0u || mb >= 0x7f800000u) ex = 0;
  ex = max(-120, min(120, ex));
  f = __uint_as_float((unsigned)(127 - ex) << 23);
  fi = __uint_as_float((unsigned)(127 + ex) << 23);
}

// Three 16-bit terms of each of the lane's three entries (rows 3 lane + i).
template <typename TI>
__device__ __forceinline__ void split_store(unsigned short* part, int lane, const float v[3])
{
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    float r = v[i];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const unsigned short u = Mma16<TI>::to16(r);
      part[k * kPartStride + 3 * lane + i] = u;
      r -= Mma16<TI>::from16(u);
    }
  }
}

// B operand of the 16 vector entries [16 K, 16 K + 16): thread (g, q) holds
// column g (split term g; zero for g >= 3), rows 2q, 2q+1 and 2q+8, 2q+9.
__device__ __forceinline__ void b_frag(const unsigned short* part, int K, int g, int q, uint32_t& b0, uint32_t& b1)
{
  b0 = b1 = 0u;
  if (g < 3) {
    const unsigned short* p = part + g * kPartStride + 16 * K + 2 * q;
    b0 = *reinterpret_cast<const uint32_t*>(p);
    b1 = *reinterpret_cast<const uint32_t*>(p + 8);
  }
}

// Sum of the three split-term columns of accumulator tiles into out (16 rows each):
// thread (g, q = 0) holds columns 0-1 of rows g and g + 8, thread (g, 1)
// column 2.
template <int kTilesUp>
__device__ __forceinline__ void reduce_columns(float acc[kTilesUp][4], float* out, int g, int q)
{
#pragma unroll
  for (int I = 0; I < kTilesUp; ++I) {
    float t0 = acc[I][0] + acc[I][1], t1 = acc[I][2] + acc[I][3];
    t0 += __shfl_down_sync(kFull, t0, 1);
    t1 += __shfl_down_sync(kFull, t1, 1);
    if (q == 0) {
      out[16 * I + g] = t0;
      out[16 * I + g + 8] = t1;
    }
  }
}

// y = (M x) for one domain held by one warp: rec is the 16-bit record in
// shared memory, scratch this warp's kApplyScratch bytes of shared memory,
// sc the lane's three column scales.
template <typename TI>
__device__ __forceinline__ void domain_apply16(const TI* rec, unsigned char* scratch, const float sc[3], int lane,
                                               const float x[3], float y[3])
{
  using M = Mma16<TI>;
  float* vf = reinterpret_cast<float*>(scratch);
  unsigned short* part = reinterpret_cast<unsigned short*>(scratch + 96 * sizeof(float));
  const int g = lane >> 2, q = lane & 3;
  const int m = lane >> 3, rr = lane & 7;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(rec);
  const uint32_t off_n = ((((m & 1) << 3) + rr) << 5) + ((((m >> 1) ^ (rr >> 2)) & 1) << 4);
  const uint32_t off_t = ((((m >> 1) << 3) + rr) << 5) + ((((m & 1) ^ (rr >> 2)) & 1) << 4);
  const float s0 = sc[0], s1 = sc[1], s2 = sc[2];
  float v[3] = {x[0] * s0, x[1] * s1, x[2] * s2};
  float f1 = 1.f, fi1 = 1.f;
  if constexpr (M::kNormalize) {
    pow2_normalizer(v, f1, fi1);
    v[0] *= f1;
    v[1] *= f1;
    v[2] *= f1;
  }
  split_store<TI>(part, lane, v);
  __syncwarp();
  // pass 1: t = V v
  {
    float acc[6][4];
#pragma unroll
    for (int I = 0; I < 6; ++I) acc[I][0] = acc[I][1] = acc[I][2] = acc[I][3] = 0.f;
#pragma unroll
    for (int K = 0; K < 6; ++K) {
      uint32_t b0, b1;
      b_frag(part, K, g, q, b0, b1);
#pragma unroll
      for (int I = K; I < 6; ++I) {
        uint32_t a[4];
        ldsm(base + (uint32_t)((I * (I + 1) / 2 + K) * 512) + off_n, a);
        M::mma(acc[I], a, b0, b1);
      }
    }
    reduce_columns<6>(acc, vf, g, q);
  }
  __syncwarp();
  v[0] = vf[3 * lane];
  v[1] = vf[3 * lane + 1];
  v[2] = vf[3 * lane + 2];
  float f2 = 1.f, fi2 = 1.f;
  if constexpr (M::kNormalize) {
    pow2_normalizer(v, f2, fi2);
    v[0] *= f2;
    v[1] *= f2;
    v[2] *= f2;
  }
  split_store<TI>(part, lane, v);
  __syncwarp();
  // pass 2: z = V^T t
  {
    float acc[6][4];
#pragma unroll
    for (int J = 0; J < 6; ++J) acc[J][0] = acc[J][1] = acc[J][2] = acc[J][3] = 0.f;
#pragma unroll
    for (int K = 0; K < 6; ++K) {
      uint32_t b0, b1;
      b_frag(part, K, g, q, b0, b1);
#pragma unroll
      for (int J = 0; J <= K; ++J) {
        uint32_t a[4];
        ldsm_t(base + (uint32_t)((K * (K + 1) / 2 + J) * 512) + off_t, a);
        M::mma(acc[J], a, b0, b1);
      }
    }
    reduce_columns<6>(acc, vf, g, q);
  }
  __syncwarp();
  const float back = fi1 * fi2;
  y[0] = vf[3 * lane] * back * s0;
  y[1] = vf[3 * lane + 1] * back * s1;
  y[2] = vf[3 * lane + 2] * back * s2;
}

// Copy a 16-bit domain record to a warp's shared-memory slot with coalesced
// 16-byte loads (streaming: a record is read once per apply).
__device__ __forceinline__ void stage_record(const uint4* __restrict__ src, unsigned char* slot, int lane)
{
  uint4* dst = reinterpret_cast<uint4*>(slot);
  __syncwarp();
#pragma unroll 7
  for (int k = lane; k < kRecBytes16 / 16; k += 32) dst[k] = __ldcs(src + k);
  __syncwarp();
}

// Domain-apply kernels: 4 warps per CTA.  16-bit records are staged in
// shared memory (a record and the apply scratch per warp: 47,104 bytes per
// CTA, four CTAs per SM).
constexpr int kApplyTpb = 128;
constexpr int kDirectSmem16 = (kApplyTpb / 32) * (kRecBytes16 + kApplyScratch);
#define MAS_APPLY_BOUNDS(TI) __launch_bounds__(kApplyTpb, 4)

// ---- coarse levels (restriction + coarse domain applies) -------------------
//
// BuildMultiLevelR and the coarse part of _schwarzLocalXSym6.  Level 1's R is
// summed from the fine residual by the kernel that forms it (the x / r update,
// or k_restrict1); every coarse domain then runs in one launch, a CTA each,
// with no CTA waiting on another: a domain of level l >= 3 sums the levels
// below its own nodes again for itself (a few thousand values) instead of
// waiting for the CTAs that own them.  32-slot banks only: with 16 the levels are
// more and wider (6,912 level-1 nodes below one CTA at 110,592 rows), and the
// kernel per level stays ahead of this form (75.5 against 82.9 us per iteration).

// The children of every level-l node: they lie in one bank of level l - 1, so a node keeps that bank and the bits of its children's lanes.
__global__ void k_children(const int* __restrict__ going_next, int begin_prev, int count_prev, int begin_next,
                           int* child_bank, unsigned* child_mask)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if ((t & ~31) >= count_prev) return;  // whole warp past the level
  const int lane = threadIdx.x & 31;
  const int key = t < count_prev ? going_next[begin_prev + t] - begin_next : -1;
  const unsigned grp = __match_any_sync(kFull, key);
  if (key < 0 || __ffs(grp) - 1 != lane) return;
  child_bank[key] = t / kBank;
  child_mask[key] = grp;
}

struct CoarseLevels {
  const int* child_bank[kMaxLevels];       // l >= 2
  const unsigned* child_mask[kMaxLevels];
  const int* going_next;
  int2* span;                   // per coarse domain, kMaxLevels entries: [first, last) node of level m below it
  const float* r1;              // R of level 1, 3 per node (padding zero)
  float* scratch;               // per level l >= 3, R of the levels 2 .. l - 1 below it where it does not fit on chip
  float* z;                     // Z of every coarse level
  const void* inv;
  const float* scale;
  LevelInfo lv;
  int c0;
};
constexpr int kCoarseOnChip = 512;   // nodes of one level whose R a CTA holds in shared memory
constexpr int kCoarseStage = 11600;  // floats of a level staged at a time: 116 banks

// Scratch floats of one level l >= 3: R of levels 2 .. l - 1 (16-byte runs).
__host__ __device__ __forceinline__ size_t coarse_scratch_level(const LevelInfo& lv, int m)
{
  return (3 * (size_t)lv.count[m] + 3) / 4 * 4;
}
__host__ __device__ __forceinline__ size_t coarse_scratch(const LevelInfo& lv, int l)
{
  size_t n = 0;
  for (int m = 2; m < l; ++m) n += coarse_scratch_level(lv, m);
  return n;
}

// Level of a coarse domain g.
__device__ __forceinline__ int domain_level(const LevelInfo& lv, int g)
{
  int l = 1;
  while (l + 1 < lv.levelnum && g >= lv.dom_begin[l + 1]) ++l;
  return l;
}

// The nodes of every level below a coarse domain of level l >= 2, down to level
// 1 (whole banks: a span may hold a few nodes of a neighbouring domain).
__global__ void k_coarse_spans(CoarseLevels a)
{
  const int g = a.lv.dom_begin[1] + blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= a.lv.domains) return;
  const int l = domain_level(a.lv, g);
  int2* span = a.span + (size_t)(g - a.lv.dom_begin[1]) * kMaxLevels;
  int lo = kBank * g - a.lv.begin[l], hi = min(lo + kBank, a.lv.count[l]);
  span[l] = make_int2(lo, hi);
  for (int m = l; m >= 2; --m) {
    lo = kBank * a.child_bank[m][lo];
    hi = min(a.lv.count[m - 1], kBank * (a.child_bank[m][hi - 1] + 1));
    span[m - 1] = make_int2(lo, hi);
  }
}

// Threads of a coarse domain's CTA: one 16-byte load per thread fetches a 16-bit
// record (21 tiles of 16x16, six warps apply them), a thread per block of the
// wrapped diagonals of an FP32 one.
template <typename TI>
constexpr int coarse_threads() { return sizeof(TI) == 2 ? 32 * kTiles16 : kDiags * kBank; }

// One coarse domain per CTA: R of its nodes, then Z = M R with the whole record
// on the chip, loaded before R is needed.  Latency is all that counts here
// (a few hundred domains of 10-20 KB): a few dependent loads and barriers,
// where the form before walked up the hierarchy through counters that the CTAs
// waited on, and one warp applied a domain: 30.7 to 28.2 us per iteration on the
// 8,000-row system and 50.8 to 44.5 at 64,000 rows with FP16 storage, where it is
// on the critical path.
// pair: the level-0 apply runs concurrently and leaves the coarse correction
// to the p update; this kernel then also sums r.z of the coarse levels, the
// sum over domains of R.Z (= r . P Z), and completes r.z with the level-0
// part (rz_part_done, mode as in rz_update).
template <typename TI>
__global__ void __launch_bounds__(coarse_threads<TI>(), 2) k_coarse_levels(CoarseLevels a, PcgScalars* s, int mode,
                                                                          int pair, double* dots)
{
  constexpr int kT = coarse_threads<TI>(), kN = 3 * kBank;
  constexpr bool kTiled = sizeof(TI) == 2;
  // dynamic: R of the levels below (two of them), then R of a level on the way
  // up (the partial products afterwards)
  extern __shared__ __align__(16) float coarse_smem[];
  float* stage = coarse_smem + 2 * 3 * kCoarseOnChip;
  __shared__ float xs[kN], vs[kN], norm[2];
  __shared__ __align__(4) unsigned short part[kTiled ? 3 * kPartStride : 1];
  float* p1 = stage;
  float* p2 = stage + kDiags * kN;
  static_assert(2 * kDiags * 3 * kBank <= kCoarseStage, "partial products share the stage");
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int g = a.lv.domains - 1 - blockIdx.x;  // the top levels, with most below them, start first
  // the record does not change during a solve: it is fetched before the wait
  uint4 rec;
  float sc = 1.f, B[9];
  const int d = tid / kBank, ln = tid % kBank;
  if constexpr (kTiled) {
    rec = __ldg(reinterpret_cast<const uint4*>(a.inv) + (size_t)g * (kRecBytes16 / 16) + tid);
    if (tid < kN) sc = __ldg(a.scale + (size_t)g * 96 + tid);
  } else if (d < kDiags) {
    const float* src = reinterpret_cast<const float*>(a.inv) + (size_t)g * (kDiags * 9 * kBank);
#pragma unroll
    for (int e = 0; e < 9; ++e) B[e] = __ldg(src + (d * 9 + e) * kBank + ln);
  }
  pdl_wait();
  if (s && s->status != MASPCG_SOLVE_RUNNING) return;  // uniform: nothing changes the status meanwhile
  // ---- R
  const int l = domain_level(a.lv, g);
  const int2* span = a.span + (size_t)(g - a.lv.dom_begin[1]) * kMaxLevels;
  if (l == 1) {
    const int2 own = span[1];
    if (tid < kN) xs[tid] = tid < 3 * (own.y - own.x) ? a.r1[3 * (size_t)own.x + tid] : 0.f;
  } else {
    // R of level m from level m - 1: a thread per component of a bank adds the
    // children of each of the bank's parents in order.  What that takes besides
    // the values (parents, child masks) does not depend on them and is loaded
    // ahead: level 2's with the staging loads, the upper levels' at the start.
    struct Parents {
      int first, end;  // a bank's parents are numbered one after another
      unsigned mask;   // children of the first (mostly the only one)
    };
    auto parents = [&](int m, int bank) {
      const int* next = a.going_next + a.lv.begin[m - 1];
      Parents t;
      t.first = __ldg(next + kBank * bank) - a.lv.begin[m];
      t.end = kBank * (bank + 1) < a.lv.count[m - 1] ? __ldg(next + kBank * (bank + 1)) - a.lv.begin[m] : a.lv.count[m];
      t.mask = __ldg(a.child_mask[m] + t.first);
      return t;
    };
    auto add_children = [&](int m, const Parents& t, const float* c, int q, float* dst, const int2& to) {
      for (int node = t.first; node < t.end; ++node) {
        unsigned mask = node == t.first ? t.mask : __ldg(a.child_mask[m] + node);
        float v = 0.f;
        if (mask == kFull) {
#pragma unroll
          for (int k = 0; k < kBank; ++k) v += c[3 * k + q];
        } else {
          for (; mask; mask &= mask - 1u) v += c[3 * (__ffs(mask) - 1) + q];
        }
        if (node >= to.x && node < to.y) dst[3 * (node - to.x) + q] = v;
      }
    };
    int2 sp[kMaxLevels];
#pragma unroll
    for (int m = 1; m < kMaxLevels; ++m) sp[m] = m <= l ? __ldg(span + m) : make_int2(0, 0);
    Parents up[kMaxLevels];
#pragma unroll
    for (int m = 3; m < kMaxLevels; ++m)
      if (m <= l && kBank * (tid / 3) < sp[m - 1].y - sp[m - 1].x) up[m] = parents(m, sp[m - 1].x / kBank + tid / 3);
    float* far = a.scratch;
    for (int m = 3; m < l; ++m) far += coarse_scratch(a.lv, m);
    auto place = [&](int m) {  // where level m's R goes
      return m == l ? xs : (sp[m].y - sp[m].x <= kCoarseOnChip ? coarse_smem + (m & 1) * 3 * kCoarseOnChip
                                                               : far + 3 * (size_t)sp[m].x);
    };
    // level 2 from level 1, staged kStageBanks banks at a time with 16-byte
    // loads (spans start at whole banks), a bank's stride padded by 16 bytes so
    // that the sums of neighbouring banks read distinct shared-memory banks
    constexpr int kStride = kN + 4;
    constexpr int kStageBanks = kCoarseStage / kStride < kT / 3 ? kCoarseStage / kStride : kT / 3;
    float* dst = place(2);
    for (int p = sp[1].x; p < sp[1].y; p += kStageBanks * kBank) {
      const int pe = min(p + kStageBanks * kBank, sp[1].y);
      const float4* from4 = reinterpret_cast<const float4*>(a.r1 + 3 * (size_t)p);
      const int n4 = (3 * (pe - p) + 3) / 4;  // the arrays are padded to whole 16-byte words
#pragma unroll 6
      for (int e = tid; e < n4; e += kT) reinterpret_cast<float4*>(stage)[e + e / (kN / 4)] = from4[e];
      const bool mine = p + kBank * (tid / 3) < pe;
      Parents t;
      if (mine) t = parents(2, p / kBank + tid / 3);
      __syncthreads();
      if (mine) add_children(2, t, stage + (tid / 3) * kStride, tid % 3, dst, sp[2]);
      __syncthreads();
    }
#pragma unroll
    for (int m = 3; m < kMaxLevels; ++m) {
      if (m > l) break;
      const float* src = dst;
      const int banks = (sp[m - 1].y - sp[m - 1].x + kBank - 1) / kBank, bank0 = sp[m - 1].x / kBank;
      far += coarse_scratch_level(a.lv, m - 1);
      dst = place(m);
      for (int e = tid; e < 3 * banks; e += kT)
        add_children(m, e == tid ? up[m] : parents(m, bank0 + e / 3), src + (size_t)(e / 3) * kN, e % 3, dst, sp[m]);
      __syncthreads();
    }
    if (tid >= 3 * min(kBank, a.lv.count[l] - (kBank * g - a.lv.begin[l])) && tid < kN) xs[tid] = 0.f;
  }
  if constexpr (kTiled) {
    if (tid < kN) vs[tid] = xs[tid] * sc;  // (by the thread that wrote xs[tid], or after its barrier)
    reinterpret_cast<uint4*>(stage)[tid] = rec;
  }
  __syncthreads();
  // ---- Z = M R
  float y = 0.f;
  if constexpr (kTiled) {
    // The products of domain_apply16 in its order, so a domain's Z is the same
    // to the bit whichever kernel forms it: warp I < 6 holds row tile I of pass
    // 1 and column tile I of pass 2, and warp 0 splits the vector for both.
    // (Plain FP32 products, a warp per tile, were 1% faster on whole solves,
    // 75.2 against 76.0 ms at 64,000 rows.  Where FP32 values barely converge,
    // as with dense contacts on small boxes, that rounding decided between
    // 4,034 iterations and the cap.)
    using M = Mma16<TI>;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(stage);
    const int g8 = lane >> 2, q4 = lane & 3, m8 = lane >> 3, rr = lane & 7;
    const uint32_t off_n = ((((m8 & 1) << 3) + rr) << 5) + ((((m8 >> 1) ^ (rr >> 2)) & 1) << 4);
    const uint32_t off_t = ((((m8 >> 1) << 3) + rr) << 5) + ((((m8 & 1) ^ (rr >> 2)) & 1) << 4);
    float back = 1.f;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
      if (w == 0) {
        float v[3] = {vs[3 * lane], vs[3 * lane + 1], vs[3 * lane + 2]};
        if constexpr (M::kNormalize) {
          float f, fi;
          pow2_normalizer(v, f, fi);
          v[0] *= f;
          v[1] *= f;
          v[2] *= f;
          if (lane == 0) norm[pass] = fi;
        }
        split_store<TI>(part, lane, v);
      }
      __syncthreads();
      if (w < kN / 16) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (int K = pass == 0 ? 0 : w; K < (pass == 0 ? w + 1 : kN / 16); ++K) {
          uint32_t b0, b1, t[4];
          b_frag(part, K, g8, q4, b0, b1);
          if (pass == 0)
            ldsm(base + (uint32_t)((w * (w + 1) / 2 + K) * 512) + off_n, t);
          else
            ldsm_t(base + (uint32_t)((K * (K + 1) / 2 + w) * 512) + off_t, t);
          M::mma(acc, t, b0, b1);
        }
        reduce_columns<1>(&acc, vs + 16 * w, g8, q4);
      }
      __syncthreads();
    }
    if constexpr (M::kNormalize) back = norm[0] * norm[1];
    if (tid < kN) y = vs[tid] * back * sc;
  } else {
    // the symmetric inverse: block (ln, ln + d) serves both triangles; the
    // products and the order of the sums are those of domain_apply
    if (d < kDiags) {
      const int c = (ln + d) & (kBank - 1);
      const float x0 = xs[3 * ln], x1 = xs[3 * ln + 1], x2 = xs[3 * ln + 2];
      const float c0 = xs[3 * c], c1 = xs[3 * c + 1], c2 = xs[3 * c + 2];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        p1[kN * d + 3 * ln + i] = B[3 * i] * c0 + B[3 * i + 1] * c1 + B[3 * i + 2] * c2;
        p2[kN * d + 3 * c + i] = B[i] * x0 + B[3 + i] * x1 + B[6 + i] * x2;
      }
    }
    __syncthreads();
    if (tid < kN) {
      y = p1[tid];
#pragma unroll
      for (int q = 1; q < kDiags; ++q) {
        y += p1[kN * q + tid];
        y += p2[kN * q + tid];
      }
    }
  }
  if (tid < kN) a.z[3 * (size_t)(kBank * g - a.c0) + tid] = y;
  if (!pair || !s) return;
  double total = 0.0;
  if (grid_finish<double, kT>(tid < kN ? (double)xs[tid] * y : 0.0, dots, blockIdx.x, gridDim.x,
                              &s->tickets[kTicketCoarse], gridDim.x, total) &&
      tid == 0)
    rz_part_done(s, 1, total, mode);
}

CoarseLevels coarse_levels_args(maspcg_handle* h)
{
  CoarseLevels c{};
  for (int l = 2; l < h->lv.levelnum; ++l) {
    c.child_bank[l] = h->child_bank[l].get();
    c.child_mask[l] = h->child_mask[l].get();
  }
  c.going_next = h->going_next.get();
  c.span = reinterpret_cast<int2*>(h->coarse_span.get());
  c.r1 = h->coarse_r.get();
  c.scratch = h->coarse_below.get();
  c.z = h->coarse_z.get();
  c.inv = h->inv.get();
  c.scale = h->cfg.inverse_storage == MASPCG_INV_FP32 ? nullptr : h->inv_scale.get();
  c.lv = h->lv;
  c.c0 = h->c0;
  return c;
}

// R of level 1 from the residual on its own (a warp per 32 slots), where no
// kernel in front summed it: the initial and standalone applies, after a
// residual replacement, and with the fused x / r update or iteration head.
template <typename Tv, bool kFused>
__global__ void __launch_bounds__(kTpb) k_restrict1(ApplyArgs a, const Tv* __restrict__ r, PcgScalars* s, FusedArgs fa)
{
  pdl_wait();
  if (s && s->status != MASPCG_SOLVE_RUNNING) return;
  const int slot = blockIdx.x * kTpb + threadIdx.x;
  if ((slot & ~31) >= a.c0) return;  // whole warp past the slots
  FusedScal fs{};
  if constexpr (kFused) fs = fused_scalars(s);
  float v[3] = {0.f, 0.f, 0.f};
  if (slot < a.c0) {
    if constexpr (kFused) {
      // r' of the iteration's update, formed as the level-0 apply forms it
      fused_input_row(fa, fs, a.fem_off + slot, false, v);
    } else {
      const Tv* rp = r + 3 * (size_t)(a.fem_off + slot);
      v[0] = (float)rp[0];
      v[1] = (float)rp[1];
      v[2] = (float)rp[2];
    }
  }
  restrict_bank(slot < a.c0 ? __ldg(a.cmap1 + slot) : -1, a.coarse_r, v);
}

// The leader of each key group gets the group's sum, its lanes in ascending order.
__device__ __forceinline__ void group_sum(int key, const float v[3], float out[3], bool& leader)
{
  const unsigned grp = __match_any_sync(kFull, key);
  float s0 = 0.f, s1 = 0.f, s2 = 0.f;
  for (int src = 0; src < 32; ++src) {
    const float a0 = __shfl_sync(kFull, v[0], src), a1 = __shfl_sync(kFull, v[1], src),
                a2 = __shfl_sync(kFull, v[2], src);
    if ((grp >> src) & 1u) {
      s0 += a0;
      s1 += a1;
      s2 += a2;
    }
  }
  out[0] = s0;
  out[1] = s1;
  out[2] = s2;
  leader = (__ffs(grp) - 1) == (int)(threadIdx.x & 31);
}

// ---- CEMAS16 apply (MASPreconditioner::preconditioning, :2250-2291) -------
//
// Over 16-slot banks:
//   * the restriction, one launch per coarse level (L-1 launches): a node of
//     level l+1 is a connected component inside one bank of level l, so its
//     children sit in one half-warp; each group is summed in lane order and
//     its lowest lane writes the parent's R once (no atomics; the reference
//     adds the same FP32 terms with atomics, __buildMultiLevelR_optimized_new
//     :729-847);
//   * the coarse domain applies (levels >= 1) and the level-0 domain apply:
//     half a warp per 48x48 domain, lane l holding block (l, (l + d) % 16) of
//     the wrapped diagonals d = 0..8, each stored block serving both
//     triangles through a shuffle of width 16 (_schwarzLocalXSym6 :957-1027);
//   * the prolongation: a vertex's z is its level-0 result plus the coarse
//     results along its coarse table, in level order (__collectFinalZ_new
//     :850-881), with r.z.  Sequentially it is fused into the level-0 apply;
//     with the coarse levels on the side stream beside the level-0 apply it
//     is a pass of its own after the join (the same FP32 sums either way).
struct Mas16Args {
  const int* pmr;
  const int* going_next;
  const int* coarse_table;  // 6 global slots per vertex (levels 1..L-1)
  LevelInfo lv;
  const float* inv;  // kMas16InvElems per domain
  float* coarse_r;   // (total_clusters - c0) x 3
  float* coarse_z;
  int fem_off, c0;
};

// R of level l+1 from level l (l = 0: from r).
template <typename Tv>
__global__ void __launch_bounds__(kTpb) k16_restrict(Mas16Args a, const Tv* __restrict__ r, int level, PcgScalars* s)
{
  pdl_wait();
  if (s && s->status != MASPCG_SOLVE_RUNNING) return;
  const int count = level == 0 ? a.c0 : a.lv.count[level];
  const int padded = (count + 15) & ~15;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if ((t & ~31) >= padded) return;  // whole warp past the level
  float v[3] = {0.f, 0.f, 0.f};
  int parent = -1;
  if (t < count) {
    if (level == 0) {
      const int vtx = a.pmr[t];
      if (vtx >= 0) {
        const size_t base = 3 * (size_t)(a.fem_off + t);
        v[0] = (float)r[base];
        v[1] = (float)r[base + 1];
        v[2] = (float)r[base + 2];
        parent = a.going_next[vtx];
      }
    } else {
      const int slot = a.lv.begin[level] + t;
      const float* x = a.coarse_r + 3 * (size_t)(slot - a.c0);
      v[0] = x[0];
      v[1] = x[1];
      v[2] = x[2];
      parent = a.going_next[slot];
    }
  }
  float o[3];
  bool leader;
  group_sum(parent >= 0 ? parent : -1 - (int)(threadIdx.x & 31), v, o, leader);
  if (parent >= 0 && leader) {
    float* d = a.coarse_r + 3 * (size_t)(parent - a.c0);
    d[0] = o[0];
    d[1] = o[1];
    d[2] = o[2];
  }
}

// y = M x for the domain of this half-warp (lane = t & 15); x of the lane's
// node; all 32 lanes of the warp take part (in = false: x = 0, no loads).
// The lane's 81 record elements are all loaded before the arithmetic, so a
// warp has its whole 10 KB in flight at once.
__device__ __forceinline__ void domain_apply16(const float* __restrict__ inv, bool in, int lane, const float x[3],
                                               float y[3])
{
  float Bm[kMas16Diags * 9];
#pragma unroll
  for (int k = 0; k < kMas16Diags * 9; ++k) Bm[k] = in ? __ldcs(inv + k * 16 + lane) : 0.f;
  float y0 = 0.f, y1 = 0.f, y2 = 0.f;
#pragma unroll
  for (int d = 0; d < kMas16Diags; ++d) {
    const int c = (lane + d) & 15;
    const float c0 = __shfl_sync(kFull, x[0], c, 16), c1 = __shfl_sync(kFull, x[1], c, 16),
                c2 = __shfl_sync(kFull, x[2], c, 16);
    const float* B = Bm + 9 * d;
    y0 += B[0] * c0 + B[1] * c1 + B[2] * c2;
    y1 += B[3] * c0 + B[4] * c1 + B[5] * c2;
    y2 += B[6] * c0 + B[7] * c1 + B[8] * c2;
    if (d != 0) {
      const float t0 = B[0] * x[0] + B[3] * x[1] + B[6] * x[2];
      const float t1 = B[1] * x[0] + B[4] * x[1] + B[7] * x[2];
      const float t2 = B[2] * x[0] + B[5] * x[1] + B[8] * x[2];
      const int src = (lane - d) & 15;
      y0 += __shfl_sync(kFull, t0, src, 16);
      y1 += __shfl_sync(kFull, t1, src, 16);
      y2 += __shfl_sync(kFull, t2, src, 16);
    }
  }
  y[0] = y0;
  y[1] = y1;
  y[2] = y2;
}

// All coarse domains (levels >= 1).  pair: the grid's R.Z (= r . P Z, the
// coarse part of r.z) completes part 1 of the pair r.z.
template <typename Tacc>
__global__ void __launch_bounds__(kTpb, 2) k16_apply_coarse(Mas16Args a, Tacc* cpart, PcgScalars* s, int mode,
                                                           int pair)
{
  pdl_wait();
  if (s && s->status != MASPCG_SOLVE_RUNNING) return;  // uniform: nothing changes the status meanwhile
  const int d1 = a.lv.dom_begin[1];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int g = d1 + (t >> 4), lane = t & 15;
  const bool in = g < a.lv.domains;
  const size_t base = 3 * (size_t)(16 * g + lane - a.c0);
  float x[3] = {0.f, 0.f, 0.f}, y[3];
  if (in) {
    x[0] = a.coarse_r[base];
    x[1] = a.coarse_r[base + 1];
    x[2] = a.coarse_r[base + 2];
  }
  domain_apply16(a.inv + (size_t)(in ? g : 0) * kMas16InvElems, in, lane, x, y);
  Tacc dot = 0;
  if (in) {
    a.coarse_z[base] = y[0];
    a.coarse_z[base + 1] = y[1];
    a.coarse_z[base + 2] = y[2];
    dot = (Tacc)x[0] * (Tacc)y[0] + (Tacc)x[1] * (Tacc)y[1] + (Tacc)x[2] * (Tacc)y[2];
  }
  if (!pair || !s) return;
  Tacc total = 0;
  if (grid_finish<Tacc>(dot, cpart, blockIdx.x, gridDim.x, &s->tickets[kTicketCoarse], gridDim.x, total) &&
      threadIdx.x == 0)
    rz_part_done(s, 1, (double)total, mode);
}

// CTAs of k16_apply_coarse.
inline int mas16_coarse_grid(const maspcg_handle* h)
{
  return std::max(1, ceil_div((long long)(h->lv.domains - h->lv.dom_begin[1]) * 16, kTpb));
}

// The coarse correction and r.z of one slot's z (y holds the level-0 result
// in FP32 precision).
template <typename Tv, typename Tacc>
__device__ __forceinline__ Tacc prolong16(const Mas16Args& a, int vtx, const Tv rv[3], float y[3], Tv* zp)
{
  if (vtx >= 0) {
    const int* ct = a.coarse_table + 6 * (size_t)vtx;
    for (int l = 1; l < a.lv.levelnum; ++l) {
      const float* zc = a.coarse_z + 3 * (size_t)(ct[l - 1] - a.c0);
      y[0] += zc[0];
      y[1] += zc[1];
      y[2] += zc[2];
    }
  } else {
    y[0] = y[1] = y[2] = 0.f;
  }
  Tacc dot = 0;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const Tv zv = (Tv)y[q];
    zp[q] = zv;
    dot += (Tacc)rv[q] * (Tacc)zv;
  }
  return dot;
}

template <typename Tacc>
__device__ __forceinline__ void rz_finish(Tacc dot, Tacc* partial, int part_base, int total_parts, int mode,
                                          PcgScalars* s)
{
  if (!partial) return;
  Tacc total = 0;
  if (grid_finish<Tacc>(dot, partial, part_base + blockIdx.x, total_parts, &s->tickets[kTicketRz], gridDim.x, total) &&
      threadIdx.x == 0 && mode > 0)
    rz_update(s, (double)total, mode);
}

// kProlong: add the coarse correction and sum r.z (the coarse levels ran
// before).  Else z = the level-0 result (the next p update adds the coarse
// correction), and r.z0 completes part 0 of the pair r.z.
template <typename Tv, typename Tacc, bool kProlong>
__global__ void __launch_bounds__(kTpb, 2) k16_apply_level0(Mas16Args a, const Tv* __restrict__ r, Tv* z, Tacc* partial,
                                                         int part_base, int total_parts, int mode, PcgScalars* s)
{
  pdl_wait();
  if (s && s->status != MASPCG_SOLVE_RUNNING) return;
  const int d0 = a.lv.dom_begin[1];
  Tacc dot = 0;
  const int stride = gridDim.x * blockDim.x;
  const int span = (d0 * 16 + 31) & ~31;  // whole warps
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < span; t += stride) {
    const int g = t >> 4, lane = t & 15;
    const bool in = g < d0;
    const int slot = 16 * g + lane;
    const int vtx = in ? a.pmr[slot] : -1;
    const size_t base = 3 * (size_t)(a.fem_off + slot);
    Tv rv[3] = {0, 0, 0};
    float x[3] = {0.f, 0.f, 0.f}, y[3];
    if (vtx >= 0) {
      rv[0] = r[base];
      rv[1] = r[base + 1];
      rv[2] = r[base + 2];
      x[0] = (float)rv[0];
      x[1] = (float)rv[1];
      x[2] = (float)rv[2];
    }
    domain_apply16(a.inv + (size_t)(in ? g : 0) * kMas16InvElems, in, lane, x, y);
    if (!in) continue;
    if (kProlong) {
      dot += prolong16<Tv, Tacc>(a, vtx, rv, y, z + base);
    } else {
      const bool real = vtx >= 0;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const Tv zv = real ? (Tv)y[q] : Tv(0);
        z[base + q] = zv;
        dot += (Tacc)rv[q] * (Tacc)zv;
      }
    }
  }
  pdl_trigger();
  if (kProlong) {
    rz_finish(dot, partial, part_base, total_parts, mode, s);
  } else if (partial) {
    Tacc total = 0;
    if (grid_finish<Tacc>(dot, partial, part_base + blockIdx.x, total_parts, &s->tickets[kTicketRz], gridDim.x,
                          total) &&
        threadIdx.x == 0)
      rz_part_done(s, 0, (double)total, mode);
  }
}

Mas16Args make_mas16_args(maspcg_handle* h)
{
  Mas16Args a{};
  a.pmr = h->pmr.get();
  a.going_next = h->going_next.get();
  a.coarse_table = h->coarse_table.get();
  a.lv = h->lv;
  a.inv = reinterpret_cast<const float*>(h->inv.get());
  a.coarse_r = h->coarse_r.get();
  a.coarse_z = h->coarse_z.get();
  a.fem_off = h->fem_off;
  a.c0 = h->c0;
  return a;
}

}  // namespace

// Level-0 apply + prolongation + r.z; with `partial` set, the last block
// completes the r.z reduction over [0, total_parts) and, for mode > 0,
// updates the PCG scalars (rz0 / beta / k).
template <typename TI, typename Tv, typename Tacc, bool kFused, bool kLevel1>
__global__ void MAS_APPLY_BOUNDS(TI) k_level0_apply(ApplyArgs a, const Tv* __restrict__ r, Tv* z, Tacc* partial,
                                                      int part_base, int total_parts, int mode, PcgScalars* s,
                                                      int coarse_add, int pair, FusedArgs fa, double* partial_rr)
{
  pdl_wait();
  if (s && s->status != MASPCG_SOLVE_RUNNING) return;
  const int lane = threadIdx.x & 31;
  const int warps_total = gridDim.x * (blockDim.x >> 5);
  Tacc dot = 0;
  double rr = 0.0;
  FusedScal fs{};
  if constexpr (kFused) fs = fused_scalars(s);
  for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < a.lv.dom_begin[kLevel1 ? 2 : 1]; g += warps_total) {
    const int slot = kBank * g + lane;
    const bool level0 = !kLevel1 || g < a.lv.dom_begin[1];
    const size_t row3 = 3 * (size_t)(level0 ? a.fem_off + slot : slot - a.c0);
    Tv r0, r1, r2;
    if (!level0) {
      r0 = a.coarse_r[row3], r1 = a.coarse_r[row3 + 1], r2 = a.coarse_r[row3 + 2];
    } else if constexpr (kFused) {
      float rn[3];
      fused_input_row(fa, fs, a.fem_off + slot, true, rn);
      r0 = rn[0], r1 = rn[1], r2 = rn[2];
      if (fa.update) rr += (double)rn[0] * rn[0] + (double)rn[1] * rn[1] + (double)rn[2] * rn[2];
    } else {
      r0 = r[row3], r1 = r[row3 + 1], r2 = r[row3 + 2];
    }
    const float x[3] = {(float)r0, (float)r1, (float)r2};
    float y[3];
    if constexpr (sizeof(TI) == 2) {
      extern __shared__ __align__(16) unsigned char direct_slots[];
      unsigned char* slot = direct_slots + (size_t)(threadIdx.x >> 5) * (kRecBytes16 + kApplyScratch);
      stage_record(reinterpret_cast<const uint4*>(a.inv) + (size_t)g * (kRecBytes16 / 16), slot, lane);
      const float* scg = a.scale + (size_t)g * 96 + 3 * lane;
      const float sc[3] = {scg[0], scg[1], scg[2]};
      domain_apply16<TI>(reinterpret_cast<const TI*>(slot), slot + kRecBytes16, sc, lane, x, y);
    } else {
      domain_apply(reinterpret_cast<const float*>(a.inv) + (size_t)g * kInvElems, lane, x, y);
    }
    if (!level0) {
      a.coarse_z[row3] = y[0], a.coarse_z[row3 + 1] = y[1], a.coarse_z[row3 + 2] = y[2];
      dot += (Tacc)r0 * (Tacc)y[0] + (Tacc)r1 * (Tacc)y[1] + (Tacc)r2 * (Tacc)y[2];
      continue;
    }
    float cc[3];
    const bool real = coarse_add ? coarse_correction(a, slot, cc) : a.pmr[slot] >= 0;
    if (!real) {
      y[0] = y[1] = y[2] = 0.f;
    } else if (coarse_add) {
      y[0] += cc[0];
      y[1] += cc[1];
      y[2] += cc[2];
    }
    z[row3] = (Tv)y[0];
    z[row3 + 1] = (Tv)y[1];
    z[row3 + 2] = (Tv)y[2];
    dot += (Tacc)r0 * (Tacc)(Tv)y[0] + (Tacc)r1 * (Tacc)(Tv)y[1] + (Tacc)r2 * (Tacc)(Tv)y[2];
  }
  pdl_trigger();
  if (kFused && fa.update) {
    double rt = 0.0;
    if (grid_finish<double, kApplyTpb>(rr, partial_rr, part_base + blockIdx.x, total_parts, &s->tickets[kTicketXr],
                                       gridDim.x, rt) &&
        threadIdx.x == 0)
      s->rr = rt;
  }
  if (partial) {
    Tacc total = 0;
    if (grid_finish<Tacc, kApplyTpb>(dot, partial, part_base + blockIdx.x, total_parts, &s->tickets[kTicketRz], gridDim.x,
                          total) &&
        threadIdx.x == 0 && mode > 0) {
      if (pair)
        rz_part_done(s, 0, (double)total, mode);
      else
        rz_update(s, (double)total, mode);
    }
  }
}

// Domain apply with the inverse staged by TMA: each warp streams its
// domains' stored records (one contiguous bulk copy per domain) into kBuf
// shared-memory slots of its own and applies them from there, so the two
// passes of the factored form read global memory once.  kBuf = 2 overlaps a
// warp's next copy with its arithmetic; kBuf = 1 halves the shared memory per
// warp and fits more warps per SM.  Level 0 reads r / writes z (plus the
// coarse correction and r.z); domains of level 1 (kLevel1, see
// takes_level1) read and write the coarse R/Z arrays.  Every wait is bounded; on expiry the warp drains its copies,
// records the error and the whole CTA leaves.
constexpr int kApplyWarps = 4;

template <typename TI, typename Tv, typename Tacc, int kBuf, bool kFused, bool kLevel1>
__global__ void __launch_bounds__(kApplyWarps * 32, kBuf == 1 ? 4 : 2)
    k_apply_tma(ApplyArgs a, const Tv* __restrict__ r, Tv* z, Tacc* partial, int part_base, int total_parts, int mode,
                PcgScalars* s, int g_end, int* err, int coarse_add, int pair, FusedArgs fa,
                double* partial_rr)
{
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t bar[kApplyWarps][kBuf];
  pdl_wait();
  if (s && s->status != MASPCG_SOLVE_RUNNING) return;
  static_assert(sizeof(TI) == 2, "the staged apply holds 16-bit records");
  constexpr unsigned kBytes = kRecBytes16;
  const int lw = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warps_total = gridDim.x * kApplyWarps;
  const int gw = blockIdx.x * kApplyWarps + lw;
  unsigned char* buf = smem + (size_t)lw * (kBuf * kBytes + kApplyScratch);
  const TI* inv = reinterpret_cast<const TI*>(a.inv);
  if (lane == 0) {
#pragma unroll
    for (int j = 0; j < kBuf; ++j) mbar_init(&bar[lw][j], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
#pragma unroll
    for (int j = 0; j < kBuf; ++j) {
      const int gj = gw + j * warps_total;
      if (gj < g_end) {
        mbar_expect_tx(&bar[lw][j], kBytes);
        tma_bulk_g2s(buf + j * kBytes, inv + (size_t)gj * inv_elems<TI>(), kBytes, &bar[lw][j]);
      }
    }
  }
  __syncwarp();
  unsigned ph[kBuf];
#pragma unroll
  for (int j = 0; j < kBuf; ++j) ph[j] = 0;
  Tacc dot = 0;
  double rr = 0.0;
  FusedScal fs{};
  if constexpr (kFused) fs = fused_scalars(s);
  int i = 0;
  bool ok = true;
  for (int g = gw; g < g_end; g += warps_total, ++i) {
    const int st = kBuf == 1 ? 0 : (i & 1);
    // loads that do not depend on the record go out before its wait
    const float* scg = a.scale + (size_t)g * 96 + 3 * lane;
    const float sc[3] = {__ldg(scg), __ldg(scg + 1), __ldg(scg + 2)};
    float x[3], y[3];
    Tv rv[3];
    size_t base;
    const bool level0 = !kLevel1 || g < a.lv.dom_begin[1];
    if (level0) {
      base = 3 * (size_t)(a.fem_off + kBank * g + lane);
      if constexpr (kFused) {
        float rn[3];
        fused_input_row(fa, fs, a.fem_off + kBank * g + lane, true, rn);
        rv[0] = rn[0];
        rv[1] = rn[1];
        rv[2] = rn[2];
        if (fa.update) rr += (double)rn[0] * rn[0] + (double)rn[1] * rn[1] + (double)rn[2] * rn[2];
      } else {
        rv[0] = r[base];
        rv[1] = r[base + 1];
        rv[2] = r[base + 2];
      }
      x[0] = (float)rv[0];
      x[1] = (float)rv[1];
      x[2] = (float)rv[2];
    } else {
      base = (size_t)(kBank * g + lane - a.c0) * 3;
      x[0] = a.coarse_r[base];
      x[1] = a.coarse_r[base + 1];
      x[2] = a.coarse_r[base + 2];
      rv[0] = x[0];
      rv[1] = x[1];
      rv[2] = x[2];
    }
    const bool padded = level0 && !coarse_add && a.pmr[kBank * g + lane] < 0;
    const bool w = mbar_wait(&bar[lw][st], ph[st]);
    if (w) ph[st] ^= 1u;
    if (!__all_sync(kFull, w)) {
      ok = false;
      break;
    }
    const TI* blk = reinterpret_cast<const TI*>(buf + st * kBytes);
    domain_apply16<TI>(blk, buf + kBuf * kBytes, sc, lane, x, y);
    __syncwarp();
    const int gn = g + kBuf * warps_total;
    if (lane == 0 && gn < g_end) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_expect_tx(&bar[lw][st], kBytes);
      tma_bulk_g2s(buf + st * kBytes, inv + (size_t)gn * inv_elems<TI>(), kBytes, &bar[lw][st]);
    }
    if (level0) {
      const int slot = kBank * g + lane;
      float cc[3];
      const bool real = coarse_add ? coarse_correction(a, slot, cc) : !padded;
      if (!real) {
        y[0] = y[1] = y[2] = 0.f;
      } else if (coarse_add) {
        y[0] += cc[0];
        y[1] += cc[1];
        y[2] += cc[2];
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const Tv zv = (Tv)y[q];
        z[base + q] = zv;
        dot += (Tacc)rv[q] * (Tacc)zv;
      }
    } else {
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        a.coarse_z[base + q] = y[q];
        dot += (Tacc)rv[q] * (Tacc)y[q];
      }
    }
  }
  pdl_trigger();
  if (!ok && lane == 0) {
    // drain this warp's copies still in flight (bounded), report
    atomicExch(err, 1);
#pragma unroll
    for (int j = 0; j < kBuf; ++j) {
      const int gj = gw + (i + j) * warps_total;
      const int sj = kBuf == 1 ? 0 : ((i + j) & 1);
      if (gj < g_end) mbar_wait(&bar[lw][sj], ph[sj]);
    }
    if (s) s->status = MASPCG_SOLVE_NONFINITE;
  }
  if (__syncthreads_or(!ok)) return;  // the whole CTA leaves together
  if (kFused && fa.update) {
    // r.r of the updated residual first: its last block stores it before its
    // arrival on the r.z ticket, so the r.z completion below sees it
    double rt = 0.0;
    if (grid_finish<double, kApplyWarps * 32>(rr, partial_rr, part_base + blockIdx.x, total_parts,
                                              &s->tickets[kTicketXr], gridDim.x, rt) &&
        threadIdx.x == 0)
      s->rr = rt;
  }
  if (partial) {
    Tacc total = 0;
    if (grid_finish<Tacc, kApplyWarps * 32>(dot, partial, part_base + blockIdx.x, total_parts, &s->tickets[kTicketRz],
                                            gridDim.x, total) &&
        threadIdx.x == 0 && mode > 0) {
      if (pair)
        rz_part_done(s, 0, (double)total, mode);
      else
        rz_update(s, (double)total, mode);
    }
  }
}

void launch_factor(maspcg_handle* h);
void build_mas_domains(maspcg_handle* h)
{
  cudaStream_t st = h->stream;
  const LevelInfo& lv = h->lv;
  const int c0 = h->c0;
  // member lists per coarse level
  h->sort_keys.resize(c0);
  h->sort_keys_out.resize(c0);
  h->sort_vals.resize(c0);
  size_t need = 0;
  MCK(cub::DeviceRadixSort::SortPairs(nullptr, need, (const unsigned*)nullptr, (unsigned*)nullptr, (const int*)nullptr,
                                      (int*)nullptr, c0, 0, 32));
  h->cub_tmp.resize(std::max(need, h->cub_tmp.n));
  for (int l = 1; l < lv.levelnum; ++l) {
    const int count = lv.count[l];
    int bits = 1;
    while ((1ll << bits) <= count) ++bits;
    k_member_keys<<<ceil_div(c0, kTpb), kTpb, 0, st>>>(h->cmap[l].get(), c0, count,
                                                      reinterpret_cast<unsigned*>(h->sort_keys.get()),
                                                      h->sort_vals.get()); MLAUNCHED(h);
    h->perm[l].resize(c0);
    size_t tb = h->cub_tmp.cap;
    MCK(cub::DeviceRadixSort::SortPairs(h->cub_tmp.get(), tb, reinterpret_cast<const unsigned*>(h->sort_keys.get()),
                                        reinterpret_cast<unsigned*>(h->sort_keys_out.get()), h->sort_vals.get(),
                                        h->perm[l].get(), c0, 0, bits, st));
  }
  // storage (16-slot banks: FP32 only)
  const int storage = h->bank == 16 ? (int)MASPCG_INV_FP32 : h->cfg.inverse_storage;
  const size_t esize = storage == MASPCG_INV_FP32 ? 4 : 2;
  h->inv.resize((size_t)lv.domains * (h->bank == 16 ? kMas16InvElems : inv_elems_for(storage)) * esize, 16);
  if (storage != MASPCG_INV_FP32) h->inv_scale.resize((size_t)lv.domains * 96);
  MCK(cudaMemsetAsync(h->failed.get() + 3, 0, sizeof(int), st));
  launch_factor(h);
  const int coarse_domains = lv.domains - lv.dom_begin[1];
  // coarse work vectors (padding entries stay zero)
  const size_t coarse = (size_t)(lv.total_clusters - c0) * 3;
  if (h->bank == 32) {
    // children of the coarse nodes and spans below the coarse domains
    // (k_coarse_levels, which keeps R above level 1 on the chip)
    size_t below = 0;
    for (int l = 2; l < lv.levelnum; ++l) {
      h->child_bank[l].resize((size_t)lv.count[l]);
      h->child_mask[l].resize((size_t)lv.count[l]);
      k_children<<<ceil_div(lv.count[l - 1], kTpb), kTpb, 0, st>>>(
          h->going_next.get(), lv.begin[l - 1], lv.count[l - 1], lv.begin[l], h->child_bank[l].get(),
          h->child_mask[l].get());
      MLAUNCHED(h);
      below += coarse_scratch(lv, l);
    }
    h->coarse_below.resize(std::max<size_t>(below, 1), 4);
    h->coarse_span.resize((size_t)std::max(coarse_domains, 1) * kMaxLevels);
    h->coarse_r.resize(std::max<size_t>(lv.levelnum > 1 ? 3 * (size_t)(lv.begin[2] - lv.begin[1]) : 0, 3));
    if (coarse_domains > 0) {
      k_coarse_spans<<<ceil_div(coarse_domains, 64), 64, 0, st>>>(coarse_levels_args(h));
      MLAUNCHED(h);
    }
  } else {
    h->coarse_r.resize(std::max<size_t>(coarse, 3));
  }
  h->coarse_z.resize(coarse > 0 ? coarse : 3);
  h->chain_dot.resize((size_t)std::max(coarse_domains, 1));  // >= CTAs of k16_apply_coarse
  MCK(cudaMemsetAsync(h->coarse_r.get(), 0, h->coarse_r.bytes(), st));
  MCK(cudaMemsetAsync(h->coarse_z.get(), 0, h->coarse_z.bytes(), st));
  int f = 0;
  MCK(cudaMemcpyAsync(&f, h->failed.get() + 3, sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
  h->failed_domains = f;
}

FactorArgs factor_args(maspcg_handle* h)
{
  FactorArgs fa{};
  fa.lv = h->lv;
  fa.pmr = h->pmr.get();
  fa.rowptr = h->rowptr.get();
  fa.colidx = h->colidx.get();
  fa.val64 = h->val64.get();
  fa.fem_off = h->fem_off;
  fa.c0 = h->c0;
  fa.inv = h->inv.get();
  fa.scale = h->inv_scale.get();
  fa.failed = h->failed.get() + 3;
  fa.coarse64 = h->coarse64.get();
  return fa;
}

// Coarse-level Galerkin sums, then the inverse of every domain (factor.cu).
template <int kB>
void launch_factor_t(maspcg_handle* h)
{
  cudaStream_t st = h->stream;
  const LevelInfo& lv = h->lv;
  const int storage = kB == 16 ? (int)MASPCG_INV_FP32 : h->cfg.inverse_storage;
  const int d0 = lv.dom_begin[1];
  const int coarse_domains = lv.domains - d0;
  h->coarse64.resize((size_t)std::max(coarse_domains, 1) * kB * kB * 9);
  CoarseArgs ca{};
  ca.pmr = h->pmr.get();
  ca.prefix_orig = h->prefix_orig.get();
  ca.levelnum = lv.levelnum;
  ca.slice_rows = 64;
  ca.nv = h->nv;
  int items = 0;
  for (int l = 1; l < lv.levelnum; ++l) {
    ca.perm[l] = h->perm[l].get();
    ca.cmap[l] = h->cmap[l].get();
    ca.slice_base[l] = items;
    items += ceil_div(h->nv, ca.slice_rows);
  }
  ca.slice_base[lv.levelnum] = items;
  for (int l = 0; l <= lv.levelnum; ++l) ca.dom_begin[l] = lv.dom_begin[l];
  ca.rowptr = h->rowptr.get();
  ca.colidx = h->colidx.get();
  ca.val64 = h->val64.get();
  ca.fem_off = h->fem_off;
  ca.c0 = h->c0;
  ca.coarse64 = h->coarse64.get();
  // The coarse sums feed only the coarse domains: with level-0 domains to
  // factor they are assembled on the side stream meanwhile, and the coarse
  // domains are factored after the join.
  const bool split = items > 0 && d0 > 0 && coarse_domains > 0;
  cudaStream_t cs = st;
  if (split) {
    MCK(cudaEventRecord(h->ev_fork, st));
    MCK(cudaStreamWaitEvent(h->side_stream, h->ev_fork, 0));
    cs = h->side_stream;
  }
  MCK(cudaMemsetAsync(h->coarse64.get(), 0, (size_t)coarse_domains * kB * kB * 9 * sizeof(double), cs));
  if (items > 0) {
    k_coarse_assemble<kB><<<ceil_div((long long)items * 32, 256), 256, 0, cs>>>(ca);
    MLAUNCHED(h);
  }
  if (split) MCK(cudaEventRecord(h->ev_join, cs));
  const FactorArgs fa = factor_args(h);
  if (split) {
    factor_domains(h, fa, 0, d0, storage);
    MCK(cudaStreamWaitEvent(st, h->ev_join, 0));
    factor_domains(h, fa, d0, coarse_domains, storage);
  } else {
    factor_domains(h, fa, 0, lv.domains, storage);
  }
  MCK(cudaGetLastError());
}

void launch_factor(maspcg_handle* h)
{
  if (h->bank == 16)
    launch_factor_t<16>(h);
  else
    launch_factor_t<32>(h);
}

void gather_mas_domains(maspcg_handle* h, double* assembled_out)
{
  FactorArgs fa = factor_args(h);
  fa.assembled = assembled_out;
  if (h->lv.domains <= 0) return;
  if (h->bank == 16)
    k_domain_gather<16><<<h->lv.domains, 512, 0, h->stream>>>(fa);
  else
    k_domain_gather<32><<<h->lv.domains, 1024, 0, h->stream>>>(fa);
  MLAUNCHED(h);
  MCK(cudaGetLastError());
}

namespace {
ApplyArgs make_apply_args(maspcg_handle* h)
{
  ApplyArgs a{};
  a.cmap1 = h->cmap[1].get();
  a.coarse_r = h->coarse_r.get();
  a.coarse_z = h->coarse_z.get();
  for (int l = 1; l < h->lv.levelnum && l < kMaxLevels; ++l) a.cmap[l] = h->cmap[l].get();
  a.pmr = h->pmr.get();
  a.inv = h->inv.get();
  a.scale = h->cfg.inverse_storage == MASPCG_INV_FP32 ? nullptr : h->inv_scale.get();
  a.fem_off = h->fem_off;
  a.c0 = h->c0;
  a.lv = h->lv;
  return a;
}

// Level-0 domain apply variants (the solve uses h->apply_variant).
enum ApplyVariant { kApplyDirect = 0, kApplyStaged2 = 1, kApplyStaged1 = 2 };

template <typename TI, typename Tv, typename Tacc, int kBuf, bool kFused, bool kLevel1>
void launch_apply_tma(maspcg_handle* h, const ApplyArgs& a, const Tv* r, Tv* z, Tacc* partial, int part_base,
                      int total_parts, int mode, PcgScalars* s, int g_end, int grid, int coarse_add, int pair,
                      const FusedArgs& fa, double* partial_rr)
{
  constexpr int bytes = kApplyWarps * (kBuf * kRecBytes16 + kApplyScratch);
  auto kern = k_apply_tma<TI, Tv, Tacc, kBuf, kFused, kLevel1>;
  allow_smem(h, kern, bytes);
  launch_pdl(h, kern, dim3(grid), dim3(kApplyWarps * 32), bytes, a, r, z, partial, part_base, total_parts, mode, s,
             g_end, h->failed.get() + 4, coarse_add, pair, fa, partial_rr);
}

// CTAs of a staged apply over `domains` domains: one wave of resident CTAs.
inline int staged_grid(const maspcg_handle* h, int domains, int kbuf)
{
  return std::max(1, std::min(ceil_div(domains, kApplyWarps), (kbuf == 1 ? 4 : 2) * h->sm_count));
}

// CTAs of the level-0 apply in a variant (level1: level 1's domains with it).
// The r.z partial sums occupy one slot per CTA, so the PCG engine sizes its
// reduction with this same count.
inline int level0_grid(const maspcg_handle* h, int variant, bool level1)
{
  const int d0 = h->lv.dom_begin[level1 ? 2 : 1];
  if (h->cfg.inverse_storage == MASPCG_INV_FP32) variant = kApplyDirect;
  switch (variant) {
    case kApplyStaged2: return staged_grid(h, d0, 2);
    case kApplyStaged1: return staged_grid(h, d0, 1);
    default:
      return std::max(1, std::min(ceil_div((long long)d0 * 32, kApplyTpb),
                                  (h->cfg.inverse_storage == MASPCG_INV_FP32 ? 16 : 4) * h->sm_count));
  }
}

// Level-0 apply (with r.z) in the given variant; coarse_add: z includes the
// coarse correction (else the p update adds it); pair: r.z is completed
// together with the concurrently running coarse levels.
template <typename TI, typename Tv, typename Tacc, bool kFused = false, bool kLevel1 = false>
void level0_apply(maspcg_handle* h, const ApplyArgs& a, int variant, const Tv* r, Tv* z, Tacc* partial, int part_base,
                  int total_parts, int mode, PcgScalars* s, int grid0, int coarse_add = 1, int pair = 0,
                  const FusedArgs& fa = FusedArgs{}, double* partial_rr = nullptr)
{
  const int g_end = h->lv.dom_begin[kLevel1 ? 2 : 1];
  if (std::is_same<TI, float>::value) variant = kApplyDirect;
  // grid0: at least level0_grid(h, variant, kLevel1), every CTA owns one r.z slot
  switch (variant) {
    case kApplyStaged2:
      if constexpr (sizeof(TI) == 2)
        launch_apply_tma<TI, Tv, Tacc, 2, kFused, kLevel1>(h, a, r, z, partial, part_base, total_parts, mode, s, g_end, grid0,
                                                  coarse_add, pair, fa, partial_rr);
      break;
    case kApplyStaged1:
      if constexpr (sizeof(TI) == 2)
        launch_apply_tma<TI, Tv, Tacc, 1, kFused, kLevel1>(h, a, r, z, partial, part_base, total_parts, mode, s, g_end, grid0,
                                                  coarse_add, pair, fa, partial_rr);
      break;

    default:
      launch_pdl(h, k_level0_apply<TI, Tv, Tacc, kFused, kLevel1>, dim3(grid0), dim3(kApplyTpb),
                 sizeof(TI) == 2 ? kDirectSmem16 : 0, a, r, z, partial, part_base, total_parts, mode, s, coarse_add,
                 pair, fa, partial_rr);
      break;
  }
}

// The coarse levels on `st`.  fa set: the residual is the fused x / r
// update's; else restricted says that the kernel in front summed level 1's R.
template <typename TI, typename Tv, bool kFused = false>
void launch_coarse(maspcg_handle* h, cudaStream_t st, const ApplyArgs& a, const Tv* r, PcgScalars* s, int mode,
                   int pair, bool restricted, const FusedArgs& fa = FusedArgs{}, int from_level = 1)
{
  if (kFused || !restricted)
    launch_pdl_on(h, st, k_restrict1<Tv, kFused>, dim3(ceil_div(h->c0, kTpb)), dim3(kTpb), 0, a, r, s, fa);
  if (from_level >= a.lv.levelnum) return;
  constexpr int bytes = (kCoarseStage + 2 * 3 * kCoarseOnChip) * sizeof(float);
  allow_smem(h, k_coarse_levels<TI>, bytes);
  launch_pdl_on(h, st, k_coarse_levels<TI>, dim3(a.lv.domains - a.lv.dom_begin[from_level]),
                dim3(coarse_threads<TI>()), bytes, coarse_levels_args(h), s, mode, pair, h->chain_dot.get());
}

// Whether the overlapped apply takes level 1's domains into the level-0 kernel:
// their R is there before it starts, they are the same work, and there are 1/32
// as many.  Beside it as CTAs of k_coarse_levels they hold the registers of most
// SMs while its own CTAs wait.  Per iteration on cubes in BF16 storage, beside it
// -> this way: 74,088 rows 45.5 -> 45.6 us, 85,184 49.5 -> 49.8, 97,336 51.5 -> 50.9,
// 140,608 60.3 -> 58.8, 262,144 84.0 -> 80.5 (91.6 -> 86.4 with 50,000 contacts).
// The line is where the level-0 domains are more than one round of resident
// warps, 75,776 rows on 148 SMs; below it no CTA waits and the two ways are equal.
// Not where r.z is summed in FP32: the coarse share of it is an FP64 sum.
template <typename Tv, typename Tacc>
bool takes_level1(const maspcg_handle* h)
{
  return sizeof(Tv) == 4 && sizeof(Tacc) == 8 && h->lv.levelnum > 1 &&
         h->lv.dom_begin[2] > 4 * kApplyWarps * h->sm_count;
}

// The MAS apply.  Sequential form: the coarse levels, then the level-0 apply
// adding the coarse correction.  Overlapped form (inside the solve): the
// coarse levels run on the side stream beside the level-0 apply, the two
// complete r.z together, and the next p update adds the coarse correction.
template <typename TI, typename Tv, typename Tacc>
void mas_apply_t(maspcg_handle* h, const Tv* r, Tv* z, Tacc* partial, int part_base, int total_parts, int mode,
                 int grid0, PcgScalars* s, bool overlap, bool restricted)
{
  ApplyArgs a = make_apply_args(h);
  const LevelInfo& lv = h->lv;
  const int variant = std::is_same<TI, float>::value ? (int)kApplyDirect : h->apply_variant;
  if (lv.levelnum <= 1) {
    level0_apply<TI, Tv, Tacc>(h, a, variant, r, z, partial, part_base, total_parts, mode, s, grid0);
    return;
  }
  if (!overlap || !s) {
    launch_coarse<TI, Tv>(h, h->stream, a, r, s, mode, 0, restricted);
    level0_apply<TI, Tv, Tacc>(h, a, variant, r, z, partial, part_base, total_parts, mode, s, grid0);
    return;
  }
  const bool level1 = takes_level1<Tv, Tacc>(h);
  const auto level0 = [&](int pair) {
    if constexpr (sizeof(Tv) == 4 && sizeof(Tacc) == 8) {
      if (level1) {
        level0_apply<TI, Tv, Tacc, false, true>(h, a, variant, r, z, partial, part_base, total_parts, mode, s, grid0, 0,
                                                pair);
        return;
      }
    }
    level0_apply<TI, Tv, Tacc>(h, a, variant, r, z, partial, part_base, total_parts, mode, s, grid0, 0, pair);
  };
  if (level1 && !restricted)
    launch_pdl(h, k_restrict1<Tv, false>, dim3(ceil_div(h->c0, kTpb)), dim3(kTpb), 0, a, r, s, FusedArgs{});
  if (level1 && lv.levelnum == 2) {
    level0(0);
    return;
  }
  MCK(cudaEventRecord(h->ev_fork, h->stream));
  MCK(cudaStreamWaitEvent(h->side_stream, h->ev_fork, 0));
  launch_coarse<TI, Tv>(h, h->side_stream, a, r, s, mode, 1, level1 || restricted, FusedArgs{}, level1 ? 2 : 1);
  MCK(cudaEventRecord(h->ev_join, h->side_stream));
  level0(1);
  MCK(cudaStreamWaitEvent(h->stream, h->ev_join, 0));
}

// The MAS apply behind the iteration's fused x / r update (fa.update; else
// fa.r[cur] is the residual): the level-0 apply updates its rows and
// preconditions r', the coarse levels restrict the same r' formed again.
// Overlapped (inside the solve, outside the reference precision): the coarse
// levels run on the side stream, r.z is completed from the two parts and the
// next p update adds the coarse correction; else they run first and the
// level-0 apply adds it.  r.r of the update comes from the level-0 apply.
template <typename TI, typename Tacc>
void mas_apply_fused_t(maspcg_handle* h, const FusedArgs& fa, float* z, Tacc* partial, double* partial_rr,
                       int part_base, int total_parts, int mode, int grid0, PcgScalars* s, bool overlap)
{
  ApplyArgs a = make_apply_args(h);
  const LevelInfo& lv = h->lv;
  const int variant = std::is_same<TI, float>::value ? (int)kApplyDirect : h->apply_variant;
  if (lv.levelnum <= 1) {
    level0_apply<TI, float, Tacc, true>(h, a, variant, nullptr, z, partial, part_base, total_parts, mode, s, grid0, 1,
                                        0, fa, partial_rr);
    return;
  }
  if (!overlap) {
    launch_coarse<TI, float, true>(h, h->stream, a, nullptr, s, mode, 0, false, fa);
    level0_apply<TI, float, Tacc, true>(h, a, variant, nullptr, z, partial, part_base, total_parts, mode, s, grid0, 1,
                                        0, fa, partial_rr);
    return;
  }
  MCK(cudaEventRecord(h->ev_fork, h->stream));
  MCK(cudaStreamWaitEvent(h->side_stream, h->ev_fork, 0));
  launch_coarse<TI, float, true>(h, h->side_stream, a, nullptr, s, mode, 1, false, fa);
  MCK(cudaEventRecord(h->ev_join, h->side_stream));
  level0_apply<TI, float, Tacc, true>(h, a, variant, nullptr, z, partial, part_base, total_parts, mode, s, grid0, 0, 1,
                                      fa, partial_rr);
  MCK(cudaStreamWaitEvent(h->stream, h->ev_join, 0));
}

}  // namespace

ApplyArgs mas_apply_args(maspcg_handle* h) { return make_apply_args(h); }



// Explicit launcher used by pcg.cu.
template <typename Tv, typename Tacc>
void mas_apply(maspcg_handle* h, const Tv* r, Tv* z, Tacc* partial, int part_base, int total_parts, int mode,
               int grid0, PcgScalars* s, bool overlap, bool restricted)
{
  switch (h->cfg.inverse_storage) {
    case MASPCG_INV_BF16:
      mas_apply_t<__nv_bfloat16, Tv, Tacc>(h, r, z, partial, part_base, total_parts, mode, grid0, s, overlap, restricted);
      break;
    case MASPCG_INV_FP16:
      mas_apply_t<__half, Tv, Tacc>(h, r, z, partial, part_base, total_parts, mode, grid0, s, overlap, restricted);
      break;
    default:
      mas_apply_t<float, Tv, Tacc>(h, r, z, partial, part_base, total_parts, mode, grid0, s, overlap, restricted);
      break;
  }
  MCK(cudaGetLastError());
}

template <typename Tacc>
void mas_apply_fused(maspcg_handle* h, const FusedArgs& fa, float* z, Tacc* partial, double* partial_rr, int part_base,
                     int total_parts, int mode, int grid0, PcgScalars* s, bool overlap)
{
  switch (h->cfg.inverse_storage) {
    case MASPCG_INV_BF16:
      mas_apply_fused_t<__nv_bfloat16, Tacc>(h, fa, z, partial, partial_rr, part_base, total_parts, mode, grid0, s,
                                             overlap);
      break;
    case MASPCG_INV_FP16:
      mas_apply_fused_t<__half, Tacc>(h, fa, z, partial, partial_rr, part_base, total_parts, mode, grid0, s, overlap);
      break;
    default:
      mas_apply_fused_t<float, Tacc>(h, fa, z, partial, partial_rr, part_base, total_parts, mode, grid0, s, overlap);
      break;
  }
  MCK(cudaGetLastError());
}
template void mas_apply_fused<float>(maspcg_handle*, const FusedArgs&, float*, float*, double*, int, int, int, int,
                                     PcgScalars*, bool);
template void mas_apply_fused<double>(maspcg_handle*, const FusedArgs&, float*, double*, double*, int, int, int, int,
                                      PcgScalars*, bool);

// Stage timing helpers: the level-0 domain apply alone, and the domain
// assembly + inversion alone (member lists from the last build).
template <typename Tv, typename Tacc>
void mas_level0_only(maspcg_handle* h, const Tv* r, Tv* z, Tacc* partial, PcgScalars* s, int variant)
{
  ApplyArgs a = make_apply_args(h);
  if (variant < 0) variant = h->apply_variant;
  const int grid = level0_grid(h, variant, false);
  switch (h->cfg.inverse_storage) {
    case MASPCG_INV_BF16:
      level0_apply<__nv_bfloat16, Tv, Tacc>(h, a, variant, r, z, partial, 0, grid, 0, s, grid);
      break;
    case MASPCG_INV_FP16: level0_apply<__half, Tv, Tacc>(h, a, variant, r, z, partial, 0, grid, 0, s, grid); break;
    default:
      MREQ(variant == kApplyDirect || variant == h->apply_variant, MASPCG_ERR_UNSUPPORTED,
           "the staged apply exists for 16-bit inverses only");
      level0_apply<float, Tv, Tacc>(h, a, kApplyDirect, r, z, partial, 0, grid, 0, s, grid);
      break;
  }
  MCK(cudaGetLastError());
}
template void mas_level0_only<float, float>(maspcg_handle*, const float*, float*, float*, PcgScalars*, int);
template void mas_level0_only<float, double>(maspcg_handle*, const float*, float*, double*, PcgScalars*, int);
template void mas_level0_only<double, double>(maspcg_handle*, const double*, double*, double*, PcgScalars*, int);

template void mas_apply<float, float>(maspcg_handle*, const float*, float*, float*, int, int, int, int, PcgScalars*,
                                      bool, bool);
template void mas_apply<float, double>(maspcg_handle*, const float*, float*, double*, int, int, int, int, PcgScalars*,
                                       bool, bool);
template void mas_apply<double, double>(maspcg_handle*, const double*, double*, double*, int, int, int, int,
                                        PcgScalars*, bool, bool);

template <typename Tv, typename Tacc>
int mas_level0_grid(maspcg_handle* h, bool overlap)
{
  return level0_grid(h, h->apply_variant, overlap && takes_level1<Tv, Tacc>(h));
}
template int mas_level0_grid<float, float>(maspcg_handle*, bool);
template int mas_level0_grid<float, double>(maspcg_handle*, bool);
template int mas_level0_grid<double, double>(maspcg_handle*, bool);

// CTAs of the level-0 apply, which completes r.z (or part 0 of it).  When
// the coarse levels run beside it (inside the solve, outside the reference
// precision) it leaves 16 SMs' worth of CTA slots free: its CTAs take every
// register of an SM, two per SM, so the chain's small launches start at once
// instead of after the apply drains.
int mas16_grid(maspcg_handle* h)
{
  const int sms = (h->overlap_coarse && h->lv.levelnum > 1) ? std::max(h->sm_count - 16, 1) : 4 * h->sm_count;
  return std::max(1, std::min(ceil_div(h->c0, kTpb), 2 * sms));
}

// CEMAS16 apply.  Sequential: the restriction level by level, the coarse
// domain applies, then the level-0 apply with the prolongation and r.z.
// overlap (with s): the restriction and the coarse applies on the side
// stream beside the level-0 apply; z leaves the coarse correction to the
// next p update (as the MAS32 apply does) and r.z is completed from a pair
// of parts, r.z0 over the fine rows and R.Z over the coarse domains.
template <typename Tv, typename Tacc>
void mas16_apply(maspcg_handle* h, const Tv* r, Tv* z, Tacc* partial, int part_base, int total_parts, int mode,
                 int grid, PcgScalars* s, bool overlap)
{
  const Mas16Args a = make_mas16_args(h);
  const LevelInfo& lv = h->lv;
  const bool pair = overlap && s && lv.levelnum > 1;
  auto coarse_levels = [&](cudaStream_t st) {
    for (int l = 0; l + 1 < lv.levelnum; ++l) {
      const int count = l == 0 ? h->c0 : lv.count[l];
      launch_pdl_on(h, st, k16_restrict<Tv>, dim3(std::max(1, ceil_div((count + 15) & ~15, kTpb))), dim3(kTpb), 0,
                    a, r, l, s);
    }
    launch_pdl_on(h, st, k16_apply_coarse<Tacc>, dim3(mas16_coarse_grid(h)), dim3(kTpb), 0, a,
                  reinterpret_cast<Tacc*>(h->chain_dot.get()), s, mode, pair ? 1 : 0);
  };
  if (pair) {
    MCK(cudaEventRecord(h->ev_fork, h->stream));
    MCK(cudaStreamWaitEvent(h->side_stream, h->ev_fork, 0));
    coarse_levels(h->side_stream);
    MCK(cudaEventRecord(h->ev_join, h->side_stream));
    launch_pdl(h, k16_apply_level0<Tv, Tacc, false>, dim3(grid), dim3(kTpb), 0, a, r, z, partial, part_base,
               total_parts, mode, s);
    MCK(cudaStreamWaitEvent(h->stream, h->ev_join, 0));
  } else {
    if (lv.levelnum > 1) coarse_levels(h->stream);
    launch_pdl(h, k16_apply_level0<Tv, Tacc, true>, dim3(grid), dim3(kTpb), 0, a, r, z, partial, part_base,
               total_parts, mode, s);
  }
  MCK(cudaGetLastError());
}
template void mas16_apply<float, float>(maspcg_handle*, const float*, float*, float*, int, int, int, int,
                                        PcgScalars*, bool);
template void mas16_apply<float, double>(maspcg_handle*, const float*, float*, double*, int, int, int, int,
                                         PcgScalars*, bool);
template void mas16_apply<double, double>(maspcg_handle*, const double*, double*, double*, int, int, int, int,
                                          PcgScalars*, bool);

// Decode the stored inverses into the reference's packed FP32 layout.
void decode_inverses(maspcg_handle* h, float* out)
{
  const int D = h->lv.domains;
  const int storage = h->bank == 16 ? (int)MASPCG_INV_FP32 : h->cfg.inverse_storage;
  const size_t esize = storage == MASPCG_INV_FP32 ? 4 : 2;
  std::vector<unsigned char> raw((size_t)D * (h->bank == 16 ? kMas16InvElems : inv_elems_for(storage)) * esize);
  std::vector<float> sc;
  MCK(cudaMemcpyAsync(raw.data(), h->inv.get(), raw.size(), cudaMemcpyDeviceToHost, h->stream));
  if (storage != MASPCG_INV_FP32) {
    sc.resize((size_t)D * 96);
    MCK(cudaMemcpyAsync(sc.data(), h->inv_scale.get(), sc.size() * 4, cudaMemcpyDeviceToHost, h->stream));
  }
  MCK(cudaStreamSynchronize(h->stream));
  auto elem = [&](size_t idx) -> float {
    if (storage == MASPCG_INV_FP32) {
      float f;
      std::memcpy(&f, raw.data() + idx * 4, 4);
      return f;
    }
    uint16_t u;
    std::memcpy(&u, raw.data() + idx * 2, 2);
    if (storage == MASPCG_INV_BF16) {
      uint32_t w = (uint32_t)u << 16;
      float f;
      std::memcpy(&f, &w, 4);
      return f;
    }
    // IEEE half -> float
    const uint32_t sign = (u >> 15) & 1, ex = (u >> 10) & 0x1f, man = u & 0x3ff;
    float f;
    if (ex == 0)
      f = std::ldexp((float)man, -24);
    else if (ex == 31)
      f = man ? NAN : INFINITY;
    else
      f = std::ldexp((float)(man | 0x400), (int)ex - 25);
    return sign ? -f : f;
  };
  if (h->bank == 16) {
    for (int g = 0; g < D; ++g)
      for (int a = 0; a < 16; ++a)
        for (int b = a; b < 16; ++b) {
          const int d = b - a;
          const bool direct = d <= 8;
          const int lane = direct ? a : b, dd = direct ? d : 16 - d;
          float* o = out + ((size_t)g * kMas16Packed + (16 * a - a * (a + 1) / 2 + b)) * 9;
          for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) {
              const int ei = direct ? 3 * i + j : 3 * j + i;
              o[i + 3 * j] = elem((size_t)g * kMas16InvElems + (size_t)(dd * 9 + ei) * 16 + lane);
            }
        }
    return;
  }
  if (storage == MASPCG_INV_FP32) {
    for (int g = 0; g < D; ++g)
      for (int a = 0; a < kBank; ++a)
        for (int b = a; b < kBank; ++b) {
          // block (a,b) lives at lane a, diagonal b-a when that is <= 16, else it
          // is the transpose of (b,a) at lane b, diagonal 32-(b-a).
          const int d = b - a;
          const bool direct = d <= 16;
          const int lane = direct ? a : b, dd = direct ? d : 32 - d;
          float* o = out + ((size_t)g * kPacked + (kBank * a - a * (a + 1) / 2 + b)) * 9;
          for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) {
              const int ei = direct ? 3 * i + j : 3 * j + i;
              o[i + 3 * j] = elem((size_t)g * kInvElems + (size_t)(dd * 9 + ei) * kBank + lane);
            }
        }
    return;
  }
  // factored storage: rebuild W (lower, column-scaled) and form W^T W
  std::vector<double> W(96 * 96), M(96 * 96);
  for (int g = 0; g < D; ++g) {
    std::fill(W.begin(), W.end(), 0.0);
    const float* scg = sc.data() + (size_t)g * 96;
    for (int i = 0; i < 96; ++i)
      for (int j = 0; j <= i; ++j)
        W[i * 96 + j] = (double)elem((size_t)g * kInvElems16 + (size_t)inv16_pos(i, j)) * scg[j];
    for (int r = 0; r < 96; ++r)
      for (int q = r; q < 96; ++q) {
        double acc = 0;
        for (int k = std::max(r, q); k < 96; ++k) acc += W[k * 96 + r] * W[k * 96 + q];
        M[r * 96 + q] = M[q * 96 + r] = acc;
      }
    for (int a = 0; a < kBank; ++a)
      for (int b = a; b < kBank; ++b) {
        float* o = out + ((size_t)g * kPacked + (kBank * a - a * (a + 1) / 2 + b)) * 9;
        for (int i = 0; i < 3; ++i)
          for (int j = 0; j < 3; ++j) o[i + 3 * j] = (float)M[(3 * a + i) * 96 + 3 * b + j];
      }
  }
}

}  // namespace maspcg
