// mas_args.cuh -- what the MAS apply kernels read about the hierarchy and
// the stored inverses, and the prolongation of the coarse levels to a fine
// slot (shared by the apply kernels and the fused PCG iteration kernel).
#pragma once
#include "maspcg_internal.cuh"

namespace maspcg {

struct ApplyArgs {
  const int* cmap1;
  const int* cmap[kMaxLevels];  // fine slot -> level-l local node (-1 padding), l >= 1
  const int* pmr;               // part_map_real: -1 marks a padding slot
  float* coarse_r;
  float* coarse_z;
  const void* inv;
  const float* scale;
  int fem_off, c0;
  LevelInfo lv;
};

// Coarse correction of a level-0 slot: the sum over the coarse levels of the
// level's z at the slot's ancestor (the prolongation, CollectFinalZ).  Returns
// false for a padding slot, whose z is zero.  The ancestors are loaded
// together with the padding mark (none depends on another), so the
// correction costs two dependent loads, not three.
__device__ __forceinline__ bool coarse_correction(const ApplyArgs& a, int slot, float c[3])
{
  c[0] = c[1] = c[2] = 0.f;
  int node[kMaxLevels];
#pragma unroll
  for (int l = 1; l < kMaxLevels; ++l) node[l] = l < a.lv.levelnum ? __ldg(a.cmap[l] + slot) : -1;
  if (a.pmr[slot] < 0) return false;
#pragma unroll
  for (int l = 1; l < kMaxLevels; ++l) {
    if (l < a.lv.levelnum) {
      const float* q = a.coarse_z + 3 * (size_t)(a.lv.begin[l] - a.c0 + node[l]);
      c[0] += q[0];
      c[1] += q[1];
      c[2] += q[2];
    }
  }
  return true;
}

// R of level 1 from one warp's 32 slots (key: the lane's level-1 node, -1 past
// the slots and for padding, which takes no part; v: its residual row).  A
// level-1 node's children all lie in one bank, so its sum is written, not
// accumulated: a butterfly when every bank of the warp is one component (the
// common case), else the component's lanes in ascending order.  Both orders are
// fixed.
__device__ __forceinline__ void restrict_bank(int key, float* coarse_r, const float v[3])
{
  const int lane = threadIdx.x & 31;
  const unsigned grp = __match_any_sync(kFull, key >= 0 ? key : -1 - lane);
  float s0 = 0.f, s1 = 0.f, s2 = 0.f;
  if (grp == kFull) {
    s0 = v[0], s1 = v[1], s2 = v[2];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s0 += __shfl_xor_sync(kFull, s0, o);
      s1 += __shfl_xor_sync(kFull, s1, o);
      s2 += __shfl_xor_sync(kFull, s2, o);
    }
  } else {
    for (unsigned m = grp; __any_sync(kFull, m != 0u); m &= m - 1u) {
      const int src = m ? __ffs(m) - 1 : lane;
      const float a0 = __shfl_sync(kFull, v[0], src), a1 = __shfl_sync(kFull, v[1], src),
                  a2 = __shfl_sync(kFull, v[2], src);
      if (m) s0 += a0, s1 += a1, s2 += a2;
    }
  }
  if (key >= 0 && __ffs(grp) - 1 == lane) {
    float* d = coarse_r + 3 * (size_t)key;
    d[0] = s0;
    d[1] = s1;
    d[2] = s2;
  }
}

ApplyArgs mas_apply_args(maspcg_handle* h);

}  // namespace maspcg
