// 1 x 128 block-scaled e4m3 quantisation of bf16 rows (scale = amax / 448 per 128 values, 1 for
// an all-zero block; saturating round-to-nearest-even convert), shared by the all-to-all dispatch
// and the dense dispatch.
#pragma once
#include <cuda_fp8.h>

#include "mcb_ptx.cuh"

namespace mcb {

// The quotients below are v / scale and amax / 448 rounded to fp32, as an fp32 reference has them.  For ordinary scales
// they are a product with the reciprocal and one correction by its residual (Markstein, IBM J. Res. Dev. 34(1), 1990):
// three instructions where a division takes about twelve and a branch, and the quantisation is most of what a dispatching
// warp issues.  That the results are the same follows by exhaustion, with the reciprocal up to three units in the last
// place off (the hardware's approximation is within one): a scale is (bf16 value) / 448, so there are 128 x 128 pairs of
// significands and some twenty exponents apart before everything rounds to zero.  The range of scales keeps the residuals
// out of underflow, the order of the signs keeps negative zeros.
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float div_corrected(float v, float d, float rcp) {
  const float q = __fmul_rn(v, rcp);
  return __fmaf_rn(__fmaf_rn(q, d, -v), -rcp, q);
}
__device__ __forceinline__ bool e4m3_ordinary(float scale) { return scale > 0x1p-80f && scale < 0x1p80f; }

// Quantise 8 bf16 values (one 16-byte pack) to 8 e4m3 bytes: saturating RNE of v / scale.
__device__ __forceinline__ uint2 quant_pack_e4m3(uint4 v, float scale) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t q[4];
  if (e4m3_ordinary(scale)) {
    const float r = rcp_approx(scale);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      q[i] = __nv_cvt_float2_to_fp8x2(make_float2(div_corrected(bf16_lo(w[i]), scale, r), div_corrected(bf16_hi(w[i]), scale, r)),
                                      __NV_SATFINITE, __NV_E4M3);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      q[i] = __nv_cvt_float2_to_fp8x2(make_float2(__fdiv_rn(bf16_lo(w[i]), scale), __fdiv_rn(bf16_hi(w[i]), scale)), __NV_SATFINITE,
                                      __NV_E4M3);
  }
  // By a move of halves, which the conversion can do itself; as byte permutations the steps with e4m3 rows were 1 to 4 % slower.
  auto join = [](uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mov.b32 %0, {%1, %2};" : "=r"(r) : "h"((uint16_t)a), "h"((uint16_t)b));
    return r;
  };
  return make_uint2(join(q[0], q[1]), join(q[2], q[3]));
}

// Largest magnitudes of the even and of the odd values of a pack, as bf16x2 (NaNs are passed over).
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t pack_absmax2(uint4 v) {
  // Of magnitudes, with a sign that is cleared once (cleared on the way in, 1 to 2 % of the steps with e4m3 rows, which are bound by the ALU pipe).
  auto absmax = [](uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
  };
  return absmax(absmax(v.x, v.y), absmax(v.z, v.w)) & 0x7fff7fffu;
}
__device__ __forceinline__ float pack_absmax(uint4 v) {
  const uint32_t m = pack_absmax2(v);
  return fmaxf(0.f, fmaxf(bf16_lo(m), bf16_hi(m)));
}
// Largest magnitudes of the 128-value blocks of two packs per lane, 16 neighbouring lanes holding a block; all 32 lanes.
__device__ __forceinline__ void block_absmax_pair(uint4 v0, uint4 v1, float& m0, float& m1) {
  const uint32_t a = pack_absmax2(v0), b = pack_absmax2(v1);
  uint32_t m = max_bf16x2(__byte_perm(a, b, 0x5410), __byte_perm(a, b, 0x7632));     // pack 0 in the low half, pack 1 in the high
#pragma unroll
  for (int sh = 8; sh >= 1; sh >>= 1) m = max_bf16x2(m, __shfl_xor_sync(0xffffffffu, m, sh));
  m0 = bf16_lo(m);
  m1 = bf16_hi(m);
}

// The same where a lane holds two neighbouring packs and eight lanes a block: of the lane's packs p0 and of its packs p1.
__device__ __forceinline__ void block_absmax_wide(const uint4* p0, const uint4* p1, float& m0, float& m1) {
  const uint32_t a = max_bf16x2(pack_absmax2(p0[0]), pack_absmax2(p0[1])), b = max_bf16x2(pack_absmax2(p1[0]), pack_absmax2(p1[1]));
  uint32_t m = max_bf16x2(__byte_perm(a, b, 0x5410), __byte_perm(a, b, 0x7632));
#pragma unroll
  for (int sh = 4; sh >= 1; sh >>= 1) m = max_bf16x2(m, __shfl_xor_sync(0xffffffffu, m, sh));
  m0 = bf16_lo(m);
  m1 = bf16_hi(m);
}

// Scale of a 128-value block from its largest magnitude (1 if that is zero or the block has only NaNs).
__device__ __forceinline__ float e4m3_scale(float amax) {
  if (e4m3_ordinary(amax)) return div_corrected(amax, 448.0f, 1.0f / 448.0f);
  return amax > 0.f ? __fdiv_rn(amax, 448.0f) : 1.0f;
}

// Two times two neighbouring packs per lane, eight lanes a block: where want(k), put(k, the sixteen values of packs k in e4m3, their block's
// scale).  All 32 lanes.  (Values of packs that nobody wants are not worked out: one in two of a run of one layer, 13 % of the smallest steps.)
template <class Want, class Put>
__device__ __forceinline__ void quant_wide_pair(const uint4* p0, const uint4* p1, Want want, Put put) {
  float m[2];
  block_absmax_wide(p0, p1, m[0], m[1]);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (!want(k)) continue;
    const uint4* p = k ? p1 : p0;
    const float scale = e4m3_scale(m[k]);
    const uint2 q0 = quant_pack_e4m3(p[0], scale), q1 = quant_pack_e4m3(p[1], scale);
    put(k, make_uint4(q0.x, q0.y, q1.x, q1.y), scale);
  }
}

// Largest magnitude of the 128-value block that starts at `block` (16 packs of 16 bytes), read by
// ONE thread (for the packet mode, where the threads that share a block are not neighbours).
__device__ __forceinline__ float block_absmax_serial(const uint8_t* block) {
  float m = 0.f;
#pragma unroll 4
  for (int p = 0; p < 16; ++p) m = fmaxf(m, pack_absmax(ld_v4(block + p * 16)));
  return m;
}

}  // namespace mcb
