// cgfd_visco.cuh -- the attenuation of one point of a visco-elastic medium (generalized Maxwell
// body), shared by the bulk stage kernel's visco-elastic form and the surface slab's pass.
// Reference: sv_curv_col_vis_iso_gpu.cu:285-433 (sv_curv_col_vis_iso_atten_gpu).
#pragma once

#include "cgfd_dev.cuh"
#include "cgfd_launch.h"

namespace cgfd {

// At the point of device index id: the strain rate recovered from the stress right-hand side
// h[3..8] (xx yy zz yz xz xy), each mechanism's right-hand side wl (strain rate - J) and RK combine,
// and the anelastic stress sum (lambda Ylam tr J + 2 mu Ymu J) taken off h. NM mechanisms, unrolled.
// The values of a mechanism are loaded ahead of the stores of the one before it, so that its memory
// round trip runs beside that one's arithmetic.
template <int NM>
__device__ __forceinline__ void vis_atten(const VisP &q, int stage, long long id, float lam, float mu, float h[9]) {
  const long long sf = q.sf;
  // isotropic compliance, in double as the reference's double literals make it; one division for the
  // six quotients by 2 mu (each within 2^-52 before it is rounded to float)
  const float tr = (h[3] + h[4] + h[5]) / (3.f * lam + 2.f * mu);
  const double inv2mu = 1.0 / (double)(2.f * mu);
  constexpr double third = 1.0 / 3.0;
  float ev[6];
  ev[0] = (float)(((2.0 * h[3] - h[4] - h[5]) * inv2mu + tr) * third);
  ev[1] = (float)(((2.0 * h[4] - h[3] - h[5]) * inv2mu + tr) * third);
  ev[2] = (float)(((2.0 * h[5] - h[3] - h[4]) * inv2mu + tr) * third);
  ev[3] = (float)((double)h[6] * inv2mu);
  ev[4] = (float)((double)h[7] * inv2mu);
  ev[5] = (float)((double)h[8] * inv2mu);
  float sl = 0.f, sm[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const bool need_pre = stage == 1 || stage == 2, need_end = stage >= 1;
  struct Mech { float ylam, ymu, j[6], pre[6], end[6]; };
  auto load = [&](int m, Mech &v) {
    v.ylam = __ldg(q.y + (long long)m * sf + id);
    v.ymu = __ldg(q.y + (long long)(NM + m) * sf + id);
#pragma unroll
    for (int c = 0; c < 6; c++) v.j[c] = __ldg(q.jcur + (long long)(6 * m + c) * sf + id);
#pragma unroll
    for (int c = 0; c < 6; c++) v.end[c] = need_end ? q.jend[(long long)(6 * m + c) * sf + id] : 0.f;
#pragma unroll
    for (int c = 0; c < 6; c++) v.pre[c] = need_pre ? __ldg(q.jpre + (long long)(6 * m + c) * sf + id) : 0.f;
  };
  Mech a;
  load(0, a);
#pragma unroll
  for (int m = 0; m < NM; m++) {
    Mech b;
    if (m + 1 < NM) load(m + 1, b);
    float hj[6];
#pragma unroll
    for (int c = 0; c < 6; c++) hj[c] = q.wl[m] * (ev[c] - a.j[c]);
    sl += a.ylam * (a.j[0] + a.j[1] + a.j[2]);
#pragma unroll
    for (int c = 0; c < 6; c++) sm[c] += a.ymu * a.j[c];
    // RK combine of the memory variables
#pragma unroll
    for (int c = 0; c < 6; c++) {
      const long long o = (long long)(6 * m + c) * sf + id;
      if (stage == 0) {
        q.jtmp[o] = a.j[c] + q.ca * hj[c];
        q.jend[o] = a.j[c] + q.cb * hj[c];
      } else {
        if (need_pre) q.jtmp[o] = a.pre[c] + q.ca * hj[c];
        q.jend[o] = a.end[c] + q.cb * hj[c];
      }
    }
    if (m + 1 < NM) a = b;
  }
  const float ls = lam * sl;
  const double mu2 = 2.0 * (double)mu;
#pragma unroll
  for (int c = 0; c < 3; c++) h[3 + c] -= (float)((double)ls + mu2 * (double)sm[c]);
#pragma unroll
  for (int c = 3; c < 6; c++) h[3 + c] -= (float)(mu2 * (double)sm[c]);
}

}  // namespace cgfd
