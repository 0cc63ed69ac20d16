// fem.cu -- the producer of the FEM part of A: per-tet gradient and
// PSD-projected Hessian of the stable Neo-Hookean energy (SNK1),
// _calculate_fem_gradient_hessian (StiffGIPC/femEnergy.cu:1720-1856) with
// __computePEPF_StableNHK3D1_double (:432-455), __computePFPX3D_Eigen_double
// (:1389), BuildTwistAndFlipEigenvectors (:1593-1639) and
// __project_StabbleNHK_H_3D1_makePD (:1641-1717).
//
// Per tet: F = Ds Dm^-1, energy u/2 (I2 - 3) + r/2 (I3 - 1 - u/r)^2 with the
// Lame rates u (length) and r (volume).  The gradient dt^2 V dF/dx^T P(F) is
// accumulated into the vertex gradient with FP64 atomics (as the reference
// does).  The 9x9 Hessian in F is projected through its closed-form
// eigensystem: six twist/flip pairs from the signed SVD F = U diag(S) V^T,
// and three scaling modes from a 3x3 eigenproblem; negative eigenvalues are
// clamped to zero.  The 12x12 element Hessian dt^2 V dF/dx^T H_F dF/dx is
// written as the 10 upper 3x3 blocks of the tet, rows <= cols (a block below
// the diagonal is transposed), values Eigen column-major.
//
// One thread per tet, FP64 throughout.  920 bytes per tet leave and arrive, 0.21
// ms for 1,500,282 tets at the measured bandwidth; the FP64 arithmetic of the
// eigensystem and the stores' 72-byte runs bound it.  The Hessian is formed in
// the frame of the singular vectors (sparse there) and rotated block by block,
// the Jacobi rotations need no division, and a warp's values leave through
// shared memory as coalesced runs: 0.47 ms, 1.36 ms with a 12-vector per
// eigenpair and each thread writing its own 720 bytes.
#include "maspcg_internal.cuh"

namespace maspcg {
namespace {

constexpr int kFemTpb = 128;

// Cyclic Jacobi on a symmetric 3x3, a = {a00, a11, a22, a01, a02, a12}
// (destroyed): eigenvalues in a[0..2], eigenvectors in the columns of v
// (row-major).  A rotation's cosine and sine come from two reciprocal square
// roots (cos 2t = |d| / h with d the diagonal difference, h = hypot(d, 2 apq)),
// no division.  The caller scales the matrix to a trace of about 1; an entry
// below 1e-18 is left alone, so no square underflows.
__device__ __forceinline__ void sym3_eigen(double a[6], double v[9])
{
#pragma unroll
  for (int i = 0; i < 9; ++i) v[i] = (i % 4 == 0) ? 1.0 : 0.0;
#pragma unroll 1
  for (int sweep = 0; sweep < 32; ++sweep) {
    const double off = a[3] * a[3] + a[4] * a[4] + a[5] * a[5];
    const double dia = a[0] * a[0] + a[1] * a[1] + a[2] * a[2];
    if (!(off > 1e-34 * dia)) break;
#pragma unroll
    for (int pr = 0; pr < 3; ++pr) {
      // pairs (0,1), (0,2), (1,2); r the third index
      const int p = pr == 2 ? 1 : 0, q = pr == 0 ? 1 : 2;
      const int pq = 3 + pr;
      const int rp = pr == 0 ? 4 : 3, rq = pr == 2 ? 4 : 5;  // entries (r, p) and (r, q)
      const double apq = a[pq];
      if (!(fabs(apq) > 1e-18)) continue;
      const double dd = a[q] - a[p], bb = 2.0 * apq;
      const double rh = rsqrt(dd * dd + bb * bb);
      const double c2 = 0.5 + 0.5 * fabs(dd) * rh;
      const double rc = rsqrt(c2);
      const double c = c2 * rc, sn = copysign(0.5 * rh * rc, dd) * bb, t = sn * rc;
      a[p] -= t * apq;
      a[q] += t * apq;
      a[pq] = 0.0;
      const double arp = a[rp], arq = a[rq];
      a[rp] = c * arp - sn * arq;
      a[rq] = sn * arp + c * arq;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double vkp = v[3 * k + p], vkq = v[3 * k + q];
        v[3 * k + p] = c * vkp - sn * vkq;
        v[3 * k + q] = sn * vkp + c * vkq;
      }
    }
  }
}

// Power of two that brings m > 0 to [1, 2) (1 when m is zero or not finite).
__device__ __forceinline__ double pow2_scale(double m)
{
  const int ex = ((__double2hiint(m) >> 20) & 0x7ff) - 1023;
  if (!(m > 0.0) || ex == 1024 || ex < -1000) return 1.0;
  return __hiloint2double((1023 - max(ex, -1000)) << 20, 0);
}

__device__ __forceinline__ void cross3(const double* a, const double* b, double* o)
{
  o[0] = a[1] * b[2] - a[2] * b[1];
  o[1] = a[2] * b[0] - a[0] * b[2];
  o[2] = a[0] * b[1] - a[1] * b[0];
}

// Signed SVD of a 3x3 (row-major): F = U diag(S) V^T with U, V rotations and
// S[2] carrying the sign of det F.  V from the eigenvectors of F^T F
// (descending), U and S from a Gram-Schmidt QR of F V.
__device__ __forceinline__ void signed_svd3(const double F[9], double U[9], double S[3], double V[9])
{
  double c[6] = {F[0] * F[0] + F[3] * F[3] + F[6] * F[6], F[1] * F[1] + F[4] * F[4] + F[7] * F[7],
                 F[2] * F[2] + F[5] * F[5] + F[8] * F[8], F[0] * F[1] + F[3] * F[4] + F[6] * F[7],
                 F[0] * F[2] + F[3] * F[5] + F[6] * F[8], F[1] * F[2] + F[4] * F[5] + F[7] * F[8]};
  const double f = pow2_scale(c[0] + c[1] + c[2]);
#pragma unroll
  for (int i = 0; i < 6; ++i) c[i] *= f;
  sym3_eigen(c, V);
  // columns in descending order of their eigenvalues (selects: no indexing)
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int p = k == 1 ? 1 : 0, q = p + 1;
    const bool sw = c[p] < c[q];
    const double cp = c[p];
    c[p] = sw ? c[q] : c[p];
    c[q] = sw ? cp : c[q];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double vp = V[3 * i + p];
      V[3 * i + p] = sw ? V[3 * i + q] : vp;
      V[3 * i + q] = sw ? vp : V[3 * i + q];
    }
  }
  const double detv = V[0] * (V[4] * V[8] - V[5] * V[7]) - V[1] * (V[3] * V[8] - V[5] * V[6]) +
                      V[2] * (V[3] * V[7] - V[4] * V[6]);
  if (detv < 0.0) V[2] = -V[2], V[5] = -V[5], V[8] = -V[8];
  double b[3][3];  // columns of F V
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int i = 0; i < 3; ++i) b[k][i] = F[3 * i] * V[k] + F[3 * i + 1] * V[3 + k] + F[3 * i + 2] * V[6 + k];
  double u0[3] = {1.0, 0.0, 0.0}, u1[3], u2[3];
  const double q0 = b[0][0] * b[0][0] + b[0][1] * b[0][1] + b[0][2] * b[0][2];
  S[0] = 0.0;
  if (q0 > 0.0) {
    const double ri = rsqrt(q0);
    S[0] = q0 * ri;
    for (int i = 0; i < 3; ++i) u0[i] = b[0][i] * ri;
  }
  const double p = u0[0] * b[1][0] + u0[1] * b[1][1] + u0[2] * b[1][2];
  double r1[3] = {b[1][0] - p * u0[0], b[1][1] - p * u0[1], b[1][2] - p * u0[2]};
  double q1 = r1[0] * r1[0] + r1[1] * r1[1] + r1[2] * r1[2];
  S[1] = 0.0;
  if (q1 > 0.0) {
    const double ri = rsqrt(q1);
    S[1] = q1 * ri;
    for (int i = 0; i < 3; ++i) u1[i] = r1[i] * ri;
  } else {  // any unit vector orthogonal to u0
    const double e[3] = {fabs(u0[0]) < 0.9 ? 1.0 : 0.0, fabs(u0[0]) < 0.9 ? 0.0 : 1.0, 0.0};
    cross3(u0, e, r1);
    const double ri = rsqrt(r1[0] * r1[0] + r1[1] * r1[1] + r1[2] * r1[2]);
    for (int i = 0; i < 3; ++i) u1[i] = r1[i] * ri;
  }
  cross3(u0, u1, u2);
  S[2] = u2[0] * b[2][0] + u2[1] * b[2][1] + u2[2] * b[2][2];
  for (int i = 0; i < 3; ++i) {
    U[3 * i] = u0[i];
    U[3 * i + 1] = u1[i];
    U[3 * i + 2] = u2[i];
  }
}

// The warp's 32 x 9 values (a block of each tet, lane by lane in stage) to
// out + 90 lane for the tets of the mask: runs of 72 bytes, nine coalesced stores.
__device__ __forceinline__ void store_blocks(double* stage, const double K[9], bool swap, double* out, int lane,
                                             unsigned tets)
{
  double* mine = stage + 9 * lane;  // Eigen column-major; a swapped block is transposed
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) mine[swap ? 3 * i + j : i + 3 * j] = K[3 * i + j];
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int e = lane + 32 * k, t = e / 9;
    if ((tets >> t) & 1u) __stcs(out + 90 * (size_t)t + e % 9, stage[e]);
  }
  __syncwarp();
}

__global__ void __launch_bounds__(kFemTpb, 3) k_fem_snk1(int ntet, const unsigned* __restrict__ tets,
                                                      const double* __restrict__ x, const double* __restrict__ dm_inv,
                                                      const double* __restrict__ volume,
                                                      const double* __restrict__ len_rate,
                                                      const double* __restrict__ vol_rate, double dt2, int offset,
                                                      int nverts, double* gradient, int* rows, int* cols,
                                                      double* vals, int* bad)
{
  __shared__ double stage_s[kFemTpb / 32][9 * 32];
  const int lane = threadIdx.x & 31;
  double* stage = stage_s[threadIdx.x >> 5];
  const int first = blockIdx.x * blockDim.x + (threadIdx.x & ~31);
  if (first >= ntet) return;  // whole warp
  // lanes past the end repeat the last tet without writing
  const int t = min(first + lane, ntet - 1);
  const bool own = first + lane < ntet;
  unsigned v[4] = {tets[4 * (size_t)t], tets[4 * (size_t)t + 1], tets[4 * (size_t)t + 2], tets[4 * (size_t)t + 3]};
  const bool fits = v[0] < (unsigned)nverts && v[1] < (unsigned)nverts && v[2] < (unsigned)nverts &&
                    v[3] < (unsigned)nverts;
  if (!fits) {
    atomicExch(bad, 1);  // the tet is skipped; the call reports the error
#pragma unroll
    for (int a = 0; a < 4; ++a) v[a] = 0;
  }
  const unsigned tets_here = __ballot_sync(kFull, own && fits);
  double Di[9];  // row-major Dm^-1
#pragma unroll
  for (int e = 0; e < 9; ++e) Di[e] = dm_inv[9 * (size_t)t + e];
  double Ds[9];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) Ds[3 * r + c] = x[3 * (size_t)v[c + 1] + r] - x[3 * (size_t)v[0] + r];
  double F[9];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) F[3 * r + c] = Ds[3 * r] * Di[c] + Ds[3 * r + 1] * Di[3 + c] + Ds[3 * r + 2] * Di[6 + c];
  const double u = len_rate[t], rr = vol_rate[t], vol = volume[t];
  // dI3/dF (cofactor matrix) and I3
  double g[9];
  g[0] = F[4] * F[8] - F[5] * F[7];
  g[1] = F[5] * F[6] - F[3] * F[8];
  g[2] = F[3] * F[7] - F[4] * F[6];
  g[3] = F[7] * F[2] - F[8] * F[1];
  g[4] = F[8] * F[0] - F[6] * F[2];
  g[5] = F[6] * F[1] - F[7] * F[0];
  g[6] = F[1] * F[5] - F[4] * F[2];
  g[7] = F[2] * F[3] - F[0] * F[5];
  g[8] = F[0] * F[4] - F[1] * F[3];
  const double I3 = F[0] * g[0] + F[1] * g[1] + F[2] * g[2];
  const double scale = dt2 * vol;
  // gradient: P = u F + (r (I3 - 1) - u) dI3/dF; dF_ij / dx_{a,i} = Dm^-1_{a-1,j} for
  // a >= 1, and vertex 0 takes minus the sum of the other three
  if (own && fits) {
    const double k = scale * (rr * (I3 - 1.0) - u), su = scale * u;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      double f0 = 0.0;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        double f = 0.0;
#pragma unroll
        for (int j = 0; j < 3; ++j) f += Di[3 * a + j] * (su * F[3 * i + j] + k * g[3 * i + j]);
        atomicAdd(gradient + 3 * (size_t)v[a + 1] + i, f);
        f0 -= f;
      }
      atomicAdd(gradient + 3 * (size_t)v[0] + i, f0);
    }
  }
  // ---- triplet indices: 10 upper blocks, rows <= cols (staged as 320 ints)
  {
    int* st = reinterpret_cast<int*>(stage);
    for (int which = 0; which < 2; ++which) {
      int bi = 0;
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = a; b < 4; ++b, ++bi)
          st[10 * lane + bi] = (int)(which ? max(v[a], v[b]) : min(v[a], v[b])) + offset;
      __syncwarp();
      int* out = (which ? cols : rows) + 10 * (size_t)first;
#pragma unroll
      for (int k = 0; k < 10; ++k)
        if ((tets_here >> ((lane + 32 * k) / 10)) & 1u) out[lane + 32 * k] = st[lane + 32 * k];
      __syncwarp();
    }
  }
  // ---- the Hessian in F in the frame of the signed SVD, projected, times
  // dt^2 V: scaling modes A (3x3 over the diagonal entries of U^T dF V), and
  // for every axis pair opposite axis m the twist and flip eigenvalues, as
  // al[m] on both off-diagonal entries and be[m] between them
  double U[9], S[3], V[9];
  signed_svd3(F, U, S, V);
  const double ev1 = rr * (I3 - 1.0) - u;
  double al[3], be[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double tw = fmax(u + S[i] * ev1, 0.0), fl = fmax(u - S[i] * ev1, 0.0);
    al[i] = 0.5 * scale * (tw + fl);
    be[i] = 0.5 * scale * (fl - tw);
  }
  const double ev2 = rr * (2.0 * I3 - 1.0) - u;
  double A[6] = {u + rr * S[1] * S[1] * S[2] * S[2], u + rr * S[0] * S[0] * S[2] * S[2],
                 u + rr * S[0] * S[0] * S[1] * S[1], ev2 * S[2], ev2 * S[1], ev2 * S[0]};  // 00 11 22 01 02 12
  // leading minors positive beyond their own rounding (some 1e-15 of the trace's
  // powers): the projection changes nothing (most tets; the determinant is 1e-2 of
  // the trace cubed at a Poisson ratio of 0.45, 1e-7 at 0.4999).  Otherwise the
  // eigenvalues below zero are cut off
  const double m01 = A[0] * A[1] - A[3] * A[3];
  const double det = A[2] * m01 - A[0] * A[5] * A[5] - A[1] * A[4] * A[4] + 2.0 * A[3] * A[4] * A[5];
  const double tr = A[0] + A[1] + A[2];
  if (!(A[0] > 1e-12 * tr && m01 > 1e-12 * tr * tr && det > 1e-12 * tr * tr * tr)) {
    const double f = pow2_scale(fmax(fabs(A[0]), fmax(fabs(A[1]), fmax(fabs(A[2]), fmax(fabs(A[3]),
                                                                    fmax(fabs(A[4]), fabs(A[5])))))));
    double d[6], W[9];
#pragma unroll
    for (int i = 0; i < 6; ++i) d[i] = A[i] * f;
    sym3_eigen(d, W);
    const double fi = 1.0 / f;
#pragma unroll
    for (int i = 0; i < 3; ++i) d[i] = fmax(d[i], 0.0) * fi;
#pragma unroll
    for (int e = 0; e < 6; ++e) {
      const int i = e < 3 ? e : (e == 5 ? 1 : 0), j = e < 3 ? e : (e == 3 ? 1 : 2);
      A[e] = d[0] * W[3 * i] * W[3 * j] + d[1] * W[3 * i + 1] * W[3 * j + 1] + d[2] * W[3 * i + 2] * W[3 * j + 2];
    }
  }
#pragma unroll
  for (int e = 0; e < 6; ++e) A[e] *= scale;
  // dF/dx in that frame: U^T dF V = sum_a (U^T x_a) c_a^T with c_a = V^T (row a - 1 of Dm^-1)
  double c[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int j = 0; j < 3; ++j) c[a][j] = V[j] * Di[3 * a] + V[3 + j] * Di[3 * a + 1] + V[6 + j] * Di[3 * a + 2];
  // blocks (a, b) of vertices 1..3, K = U M U^T with
  //   M_ik = A_ik c_a[i] c_b[k] + be[j] c_a[k] c_b[i] (j the third axis), i != k
  //   M_ii = A_ii c_a[i] c_b[i] + sum over j != i of al[third of i, j] c_a[j] c_b[j]
  // and vertex 0's blocks from the rows summing to zero (a rigid translation
  // changes no energy); R holds sum over a of K_ab
  double* base = vals + 90 * (size_t)first;
  double R[3][9];
#pragma unroll
  for (int b = 0; b < 3; ++b)
#pragma unroll
    for (int e = 0; e < 9; ++e) R[b][e] = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      const double* ca = c[a];
      const double* cb = c[b];
      double M[9], K[9];
      const double p0 = ca[0] * cb[0], p1 = ca[1] * cb[1], p2 = ca[2] * cb[2];
      M[0] = A[0] * p0 + al[2] * p1 + al[1] * p2;
      M[4] = A[1] * p1 + al[2] * p0 + al[0] * p2;
      M[8] = A[2] * p2 + al[1] * p0 + al[0] * p1;
      const double q01 = ca[0] * cb[1], q10 = ca[1] * cb[0], q02 = ca[0] * cb[2], q20 = ca[2] * cb[0],
                   q12 = ca[1] * cb[2], q21 = ca[2] * cb[1];
      M[1] = A[3] * q01 + be[2] * q10;
      M[3] = A[3] * q10 + be[2] * q01;
      M[2] = A[4] * q02 + be[1] * q20;
      M[6] = A[4] * q20 + be[1] * q02;
      M[5] = A[5] * q12 + be[0] * q21;
      M[7] = A[5] * q21 + be[0] * q12;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        double w[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) w[k] = U[3 * i] * M[k] + U[3 * i + 1] * M[3 + k] + U[3 * i + 2] * M[6 + k];
#pragma unroll
        for (int k = 0; k < 3; ++k) K[3 * i + k] = w[0] * U[3 * k] + w[1] * U[3 * k + 1] + w[2] * U[3 * k + 2];
      }
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          R[b][3 * i + k] += K[3 * i + k];
          if (a != b) R[a][3 * k + i] += K[3 * i + k];
        }
      constexpr int kBlock[3][3] = {{4, 5, 6}, {0, 7, 8}, {0, 0, 9}};
      store_blocks(stage, K, v[a + 1] > v[b + 1], base + 9 * kBlock[a][b], lane, tets_here);
    }
  double K0[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int k = 0; k < 3; ++k) K0[3 * i + k] = R[0][3 * k + i] + R[1][3 * k + i] + R[2][3 * k + i];
  store_blocks(stage, K0, false, base, lane, tets_here);
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    double K[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) K[e] = -R[b][e];
    store_blocks(stage, K, v[0] > v[b + 1], base + 9 * (b + 1), lane, tets_here);
  }
}

}  // namespace

void fem_snk1(maspcg_handle* h, int ntet, int nverts, const unsigned* tets, const double* x, const double* dm_inv,
              const double* volume, const double* len_rate, const double* vol_rate, double dt, int offset,
              double* gradient, int* rows, int* cols, double* vals)
{
  if (ntet <= 0) return;
  MREQ(nverts > 0, MASPCG_ERR_INVALID_ARGUMENT, "tet vertex id out of range");
  h->asm_flags.resize(std::max<size_t>(h->asm_flags.n, 1));
  int* bad = h->asm_flags.get();
  MCK(cudaMemsetAsync(bad, 0, sizeof(int), h->stream));
  k_fem_snk1<<<ceil_div(ntet, kFemTpb), kFemTpb, 0, h->stream>>>(ntet, tets, x, dm_inv, volume, len_rate, vol_rate,
                                                                 dt * dt, offset, nverts, gradient, rows, cols, vals,
                                                                 bad);
  MLAUNCHED(h);
  MCK(cudaGetLastError());
  int flag = 0;
  MCK(cudaMemcpyAsync(&flag, bad, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
  MCK(cudaStreamSynchronize(h->stream));
  MREQ(flag == 0, MASPCG_ERR_INVALID_ARGUMENT, "tet vertex id out of range");
}

}  // namespace maspcg
