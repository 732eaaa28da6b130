// cgfd_source.cuh -- source injection (sv_curv_col_el_gpu.cu:227-301) of one smoothing point and
// component, shared by the source kernel and the bulk stage's tiles.
#pragma once

#include "cgfd_dev.cuh"
#include "cgfd_launch.h"

namespace cgfd {

// Right-hand side contribution of component c at smoothing point e of source `is`, with the RK weights
// of the stage, added to the stage output and w_end. it: the step. The reductions return no value
// except where the FP16 scale collector needs it.
template <typename R>
__device__ __forceinline__ void source_add(const SrcPT<R> &s, int is, int e, int c, int it, int shot) {
  if (c < 3 ? !s.force : !s.moment) return;
  const long long q = (long long)is * s.max_ext + e;
  const long long id = s.ext_idx[q] + ((long long)shot * 9 + c) * s.sf;
  const R w = (c < 3 ? s.ext_wv : s.ext_wt)[q];
  const R v = s.stf[(((long long)is * s.max_nt + (it - s.it_begin[is])) * 4 + s.stage) * 9 + c];
  const R h = c < 3 ? v * w : -v * w;
  if (s.stage < 3) {
    if constexpr (std::is_same<R, float>::value) {
      if (s.wave16)
        atomicAdd(reinterpret_cast<__half *>(s.tmp_out) + id, __float2half_rn(s.ca * h * s.wsc[18 * shot + 9 + c]));
      else atomicAdd(s.tmp_out + id, s.ca * h);
    } else {
      atomicAdd(s.tmp_out + id, s.ca * h);
    }
  }
  if constexpr (std::is_same<R, float>::value) {
    if (s.wave16 && s.stage == 3) {
      const R old = atomicAdd(s.end + id, s.cb * h);
      atomic_max_abs(&s.amax[2 * shot + wgroup(c)], old + s.cb * h);
      return;
    }
  }
  atomicAdd(s.end + id, s.cb * h);
}

// whether source `is` acts at step it
template <typename R>
__device__ __forceinline__ bool source_active(const SrcPT<R> &s, int is, int it) {
  const int ib = s.it_begin[is];
  return it >= ib && it <= ib + s.max_nt - 1;
}

// The shot's sources at the smoothing points inside one tile [i0, i1) x [j0, j1) x [k0, k1), by the block
// that has stored the tile.
template <typename R>
__device__ __noinline__ void tile_sources(const StagePT<R> &p, const SrcPT<R> &s, int shot, int i0, int i1, int j0, int j1,
                                          int k0, int k1, int tid, int threads) {
  const int it = *s.d_it;
  for (int is = 0; is < s.nsrc; is++) {
    if (s.src_shot[is] != shot || !source_active(s, is, it)) continue;
    for (int e = tid; e < s.ext_num[is]; e += threads) {
      long long r = s.ext_idx[(long long)is * s.max_ext + e] - p.off0;
      const int k = (int)(r / p.sz);
      r -= k * p.sz;
      const int j = (int)(r / p.sx), i = (int)(r - j * p.sx);
      if (i < i0 || i >= i1 || j < j0 || j >= j1 || k < k0 || k >= k1) continue;
      for (int c = 0; c < 9; c++) source_add(s, is, e, c, it, shot);
    }
  }
}

}  // namespace cgfd
