// y = R(x) for the self pathway's Q and K, written as bf16.  A thread rotates 8 dims of the lower half together with their partners in
// the upper half (16-byte loads and stores, rows contiguous in memory): part `idx` of rows * D / 16.
#pragma once

#include "common.cuh"

namespace mintb {

__device__ __forceinline__ void rope_rotate_part(size_t idx, const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                                                 __nv_bfloat16* __restrict__ qr, __nv_bfloat16* __restrict__ kr, const float* __restrict__ cos_tab,
                                                 const float* __restrict__ sin_tab, size_t rows, int T, int D) {
  const int h = D / 2, cpr = h / 8;  // chunks per row
  if (idx >= rows * cpr) return;
  const int c = int(idx % cpr);
  const size_t row = idx / cpr;
  const int t = int(row % T);
  const float4* ct = reinterpret_cast<const float4*>(cos_tab + size_t(t) * h + c * 8);
  const float4* st = reinterpret_cast<const float4*>(sin_tab + size_t(t) * h + c * 8);
  const float4 c0 = ct[0], c1 = ct[1], s0 = st[0], s1 = st[1];
  const float cs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
  const float sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    const __nv_bfloat16* src = (which == 0 ? q : k) + row * D + c * 8;
    __nv_bfloat16* dst = (which == 0 ? qr : kr) + row * D + c * 8;
    uint4 lo = *reinterpret_cast<const uint4*>(src), hi = *reinterpret_cast<const uint4*>(src + h);
    const __nv_bfloat16* lp = reinterpret_cast<const __nv_bfloat16*>(&lo);
    const __nv_bfloat16* hp = reinterpret_cast<const __nv_bfloat16*>(&hi);
    uint4 olo, ohi;
    __nv_bfloat16* olp = reinterpret_cast<__nv_bfloat16*>(&olo);
    __nv_bfloat16* ohp = reinterpret_cast<__nv_bfloat16*>(&ohi);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float a = __bfloat162float(lp[e]), b = __bfloat162float(hp[e]);
      olp[e] = __float2bfloat16_rn(a * cs[e] - b * sn[e]);
      ohp[e] = __float2bfloat16_rn(b * cs[e] + a * sn[e]);
    }
    *reinterpret_cast<uint4*>(dst) = olo;
    *reinterpret_cast<uint4*>(dst + h) = ohi;
  }
}

}  // namespace mintb
