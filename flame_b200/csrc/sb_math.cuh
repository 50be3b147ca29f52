// Stick-breaking weights of eight neighbouring keys of one row, shared by the forward (attention.cu) and the backward
// (sb_attention.cu): the backward's running sum of weight gradients has to meet the total the forward's weights imply, so both
// form the same fp32 weights in the same order.
//
//   sigma = t / (1 + t), t = 2^x (x: logit in log2 units),   att_i = sigma_i * prod_{m > i} (1 - sigma_m),   1 - sigma = 1 / (1 + t)
//
// Keys are consumed from the right.  The products inside the group do not depend on the product E carried from the right,
// so the eight exponentials, reciprocals and local products of a group overlap with its neighbours'; only E is a chain, one
// multiplication per group (one per key, behind a correctly rounded reciprocal subroutine, held the softmax warps up before).
// The reciprocal is the hardware approximation and one Newton step: against fp64 the remainder's mean error is that of the
// correctly rounded one (4.87e-7 both at 512 keys, 4.84e-7 and 4.81e-7 at 4,096).
#pragma once
#include <stdint.h>

template <bool MASK>
__device__ __forceinline__ void sb_group(const uint32_t* x8, float scale_log2, uint32_t dead, float& E, float (&sig)[8], float (&att)[8]) {
  float inv[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float x = fminf(fmaxf(__uint_as_float(x8[i]) * scale_log2, -100.f), 100.f);
    float t, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(x));
    const float y = 1.f + t;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
    r = fmaf(r, fmaf(-y, r, 1.f), r);
    const bool gone = MASK && ((dead >> i) & 1u);
    inv[i] = gone ? 1.f : r;
    sig[i] = gone ? 0.f : t * r;
  }
  float p = 1.f;
#pragma unroll
  for (int i = 7; i >= 0; --i) {
    att[i] = (sig[i] * p) * E;
    p *= inv[i];
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
