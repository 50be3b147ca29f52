// Stick-breaking weights of eight neighbouring keys of one row, shared by the forward and the backward
// of sb_attention.cu: the backward's running sum of weight gradients has to meet the total the forward's weights imply, so both
// form the same fp32 weights in the same order.
//
//   sigma = t / (1 + t), t = 2^x (x: logit in log2 units),   att_i = sigma_i * prod_{m > i} (1 - sigma_m),   1 - sigma = 1 / (1 + t)
//
// Keys are consumed from the right.  The products inside the group do not depend on the product E carried from the right,
// so the eight exponentials, reciprocals and local products of a group overlap with its neighbours'; only E is a chain, one
// multiplication per group (one per key, behind a correctly rounded reciprocal subroutine, held the softmax warps up before).
// Two keys share one hardware reciprocal, of the product of their denominators (three special functions for two keys instead of
// four: forward 854 -> 819 us, backward 1,934 -> 1,872 at eight rows of 4,096 tokens, 16 heads), and each gets a Newton step, which
// takes out the roundings of the products as well (the remainder against fp64: mean error 3.18e-7, as with one each).  A logit
// counts as at most 2^100 : 1.  The product of two denominators has to stay below 2^126, so that its reciprocal is a normal number:
// the left one of two keys that together exceed 2^124 : 1 counts as what is left of that.  Its weight's sigma is 1 in fp32 all
// the same (the rest is 2^24 : 1 or more), and what both leave of the row, less than 2^-124, is at the end of the range of fp32.
// (One clamp at 2^60 : 1 was 22 us less forward and 12 less backward, 31 more with the remainder's gradient; one denominator
// times 2^-76 instead is 5 us more forward and holds short rows up, 4,096 tokens 3 %.)
//
// Two keys share an instruction wherever there is a packed one.  It has no negation, so the reciprocal is formed with its sign
// turned, m = -1 / (1 + t): then 1 + y m is the Newton residual, t m = -sigma, and the sign of the product over k keys, (-1)^k,
// is put right by the pair (E, -E).
#pragma once
#include <stdint.h>
#include "tc05.cuh"

typedef unsigned long long sb2;  // two fp32 values, the lower key in the lower half
__device__ __forceinline__ sb2 sb_pk(float a, float b) {
  sb2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void sb_up(sb2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ sb2 sb_mul2(sb2 a, sb2 b) {
  sb2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ sb2 sb_add2(sb2 a, sb2 b) {
  sb2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ sb2 sb_fma2(sb2 a, sb2 b, sb2 c) {
  sb2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint32_t sb_pack(sb2 v) {  // bf16
  float a, b;
  sb_up(v, a, b);
  return tc05::pack_bf16(a, b);
}

// What does not depend on the keys to the right.  nsig: -sigma, ninv: sigma - 1; nsig[i] holds keys 2 i and 2 i + 1
template <bool MASK>
__device__ __forceinline__ void sb_sigma(const uint32_t* x8, float scale_log2, uint32_t dead, sb2 (&nsig)[4], float (&ninv)[8]) {
  const sb2 one = sb_pk(1.f, 1.f), scale = sb_pk(scale_log2, scale_log2);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float x0, x1, t0, t1, y0, y1;
    sb_up(sb_mul2(sb_pk(__uint_as_float(x8[2 * i]), __uint_as_float(x8[2 * i + 1])), scale), x0, x1);
    if (MASK && ((dead >> (2 * i + 1)) & 1u)) x1 = -100.f;  // a key that does not count takes nothing from its neighbour
    x1 = fminf(fmaxf(x1, -100.f), 100.f);
    x0 = fminf(fminf(fmaxf(x0, -100.f), 100.f), 124.f - x1);
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(t0) : "f"(x0));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(t1) : "f"(x1));
    const sb2 t = sb_pk(t0, t1), y = sb_add2(t, one);
    sb_up(y, y0, y1);
    float both;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(both) : "f"(-y0 * y1));
    sb2 m = sb_pk(both * y1, both * y0);
    m = sb_fma2(m, sb_fma2(y, m, one), m);
    nsig[i] = sb_mul2(t, m);
    sb_up(m, ninv[2 * i], ninv[2 * i + 1]);
    if (MASK) {
      float s0, s1;
      sb_up(nsig[i], s0, s1);
      const bool gone0 = (dead >> (2 * i)) & 1u, gone1 = (dead >> (2 * i + 1)) & 1u;
      nsig[i] = sb_pk(gone0 ? 0.f : s0, gone1 ? 0.f : s1);
      ninv[2 * i] = gone0 ? -1.f : ninv[2 * i];
      ninv[2 * i + 1] = gone1 ? -1.f : ninv[2 * i + 1];
    }
  }
}

// att: the weights, and E past these keys
__device__ __forceinline__ void sb_weights(float& E, const sb2 (&nsig)[4], const float (&ninv)[8], sb2 (&att)[4]) {
  const sb2 e2 = sb_pk(E, -E);
  float p = 1.f;
#pragma unroll
  for (int i = 3; i >= 0; --i) {
    const float p1 = p;
    p *= ninv[2 * i + 1];
    att[i] = sb_mul2(sb_mul2(nsig[i], sb_pk(p, p1)), e2);
    p *= ninv[2 * i];
  }
  E *= p;
}

// bit i set: key kv + i of this group is not before the row (kv >= q), or the row does not exist
__device__ __forceinline__ uint32_t sb_dead_bits(bool row_dead, bool diag, int kv, int q_idx) {
  if (row_dead) return 0xffu;
  if (!diag) return 0u;
  const int live = q_idx - kv;  // keys kv .. q_idx - 1
  return live >= 8 ? 0u : (live <= 0 ? 0xffu : (0xffu << live) & 0xffu);
}
