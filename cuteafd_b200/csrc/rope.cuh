// Head norm and rotation of one 128-wide head by one warp: lane holds elements {2l, 2l+1} (a) and {64+2l, 64+2l+1} (b) as bf16 pairs.
// Rounding points follow the oracle: norm -> bf16 -> rope (fp32) -> bf16.
#pragma once

#include "common.cuh"

namespace cafd {

struct HeadAngles {
  float s0, c0, s1, c1;
};

// Angles of a token, the same for all its heads.  Pairs: whole head interleaved (2i, 2i+1), lane l holds pairs l and 32+l; whole head in halves
// (i, i+64), i = 2l and 2l+1; half a head (rot 64) interleaved, pair l; half a head in halves (i, i+32), lanes 0..15 hold i = 2l, 2l+1, lanes
// 16..31 their partners.
__device__ __forceinline__ HeadAngles head_angles(float pos, const float* __restrict__ inv_freq, int lane, int interleaved, int rot) {
  HeadAngles r{0.f, 1.f, 0.f, 1.f};
  const int f0 = interleaved ? lane : rot == 64 ? (2 * lane) & 31 : 2 * lane;
  const int f1 = interleaved ? 32 + lane : f0 + 1;
  sincosf(pos * inv_freq[f0], &r.s0, &r.c0);
  if (!(interleaved && rot == 64)) sincosf(pos * inv_freq[f1], &r.s1, &r.c1);
  return r;
}

// bias [128] of the head: added to the projection's bf16 output and rounded again.
__device__ __forceinline__ void head_bias(uint32_t& a, uint32_t& b, const __nv_bfloat16* __restrict__ bias, int lane) {
  const uint32_t ba = *reinterpret_cast<const uint32_t*>(bias + 2 * lane);
  const uint32_t bb = *reinterpret_cast<const uint32_t*>(bias + 64 + 2 * lane);
  a = pack_bf16(bf16_lo(a) + bf16_lo(ba), bf16_hi(a) + bf16_hi(ba));
  b = pack_bf16(bf16_lo(b) + bf16_lo(bb), bf16_hi(b) + bf16_hi(bb));
}

// In place; nw: norm weights or null.
__device__ __forceinline__ void head_norm_rope(uint32_t& a, uint32_t& b, const __nv_bfloat16* __restrict__ nw, float eps, const HeadAngles& r,
                                               int lane, int interleaved, int rot) {
  float x0 = bf16_lo(a), x1 = bf16_hi(a), x2 = bf16_lo(b), x3 = bf16_hi(b);
  if (nw) {
    const float ss = warp_sum(x0 * x0 + x1 * x1 + x2 * x2 + x3 * x3);
    const float inv = rsqrtf(ss / 128.0f + eps);
    const uint32_t wa = *reinterpret_cast<const uint32_t*>(nw + 2 * lane);
    const uint32_t wb = *reinterpret_cast<const uint32_t*>(nw + 64 + 2 * lane);
    const uint32_t ra = pack_bf16(x0 * inv * bf16_lo(wa), x1 * inv * bf16_hi(wa));
    const uint32_t rb = pack_bf16(x2 * inv * bf16_lo(wb), x3 * inv * bf16_hi(wb));
    x0 = bf16_lo(ra); x1 = bf16_hi(ra); x2 = bf16_lo(rb); x3 = bf16_hi(rb);
  }
  float y0, y1, y2, y3;
  if (rot == 64) {
    y2 = x2; y3 = x3;
    if (interleaved) {
      y0 = x0 * r.c0 - x1 * r.s0; y1 = x0 * r.s0 + x1 * r.c0;
    } else {
      const float p0 = __shfl_xor_sync(0xffffffffu, x0, 16), p1 = __shfl_xor_sync(0xffffffffu, x1, 16);
      if (lane < 16) { y0 = x0 * r.c0 - p0 * r.s0; y1 = x1 * r.c1 - p1 * r.s1; }
      else           { y0 = p0 * r.s0 + x0 * r.c0; y1 = p1 * r.s1 + x1 * r.c1; }
    }
  } else if (interleaved) {
    y0 = x0 * r.c0 - x1 * r.s0; y1 = x0 * r.s0 + x1 * r.c0;
    y2 = x2 * r.c1 - x3 * r.s1; y3 = x2 * r.s1 + x3 * r.c1;
  } else {
    y0 = x0 * r.c0 - x2 * r.s0; y2 = x0 * r.s0 + x2 * r.c0;
    y1 = x1 * r.c1 - x3 * r.s1; y3 = x1 * r.s1 + x3 * r.c1;
  }
  a = pack_bf16(y0, y1);
  b = pack_bf16(y2, y3);
}

}  // namespace cafd
