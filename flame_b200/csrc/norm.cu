// Fused RMSNorm (+ residual add) forward and backward, and the gated variant used by the linear-attention
// layers.  Bandwidth-bound: 16-byte loads, fp32 math, a single pass over HBM.
//
//   forward :  r = x (+ residual_in);  y = r * rsqrt(mean(r^2) + eps) * w;   optionally writes r and rstd
//   backward:  dx = rstd * (dy*w - xhat * mean(dy*w*xhat)) (+ d_residual);   dw = sum_rows dy * xhat
//
// Semantics follow fla/modules/layernorm.py:1084-1134 (RMSNorm with prenorm residual) and
// fla/modules/fused_norm_gate.py:992 (norm(x) * w * g * sigmoid(g)); the row-parallel design, the fixed-order
// two-stage dw reduction and the fused residual-gradient add are this library's own.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include "host_utils.cuh"
#include "flame_b200_noalloc.h"

namespace {

constexpr int WARPS = 8;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void unpack8(const uint4& q, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 q;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return q;
}
__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + __expf(-x)); }

// Where rows lie.  A row is one head of a token.  `map`: the normalised tensor is in the chunk layout of the linear-attention kernels
// (padded rows), everything else in packed rows: forward map[token] = padded row, backward map[padded row] = token or -1.  The
// gate may be a column block of a wider matrix: `ldg` elements from token to token (`lddg`: its gradient's).
struct Rows {
  const int* map;
  unsigned heads;
  long long ldg, lddg;
};
__device__ __forceinline__ long long mapped_row(const Rows& rs, long long row) {  // -1: padding
  if (rs.map == nullptr) return row;
  const unsigned t = (unsigned)row / rs.heads;
  const int to = rs.map[t];
  return to < 0 ? -1 : (long long)to * rs.heads + ((unsigned)row - t * rs.heads);
}
__device__ __forceinline__ long long gate_at(unsigned heads, long long ld, long long row, int D) {
  if (ld == (long long)heads * D) return row * D;
  const unsigned t = (unsigned)row / heads;
  return t * ld + (long long)((unsigned)row - t * heads) * D;
}

// gate_mode: 0 none, 1 swish (g * sigmoid(g)), 2 sigmoid
template <bool HAS_RES, bool WRITE_RES, int GATE>
__global__ void __launch_bounds__(WARPS * 32)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res_in,
                   const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ gate,
                   __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ res_out, float* __restrict__ rstd,
                   long long rows, int D, float eps, const Rows at) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * WARPS + warp;
  if (row >= rows) return;
  const int nvec = D >> 3;
  const uint4* xr = reinterpret_cast<const uint4*>(x + mapped_row(at, row) * D);
  const uint4* rr = HAS_RES ? reinterpret_cast<const uint4*>(res_in + row * D) : nullptr;
  uint4* ro = WRITE_RES ? reinterpret_cast<uint4*>(res_out + row * D) : nullptr;
  float ss = 0.f;
  for (int i = lane; i < nvec; i += 32) {
    float a[8];
    unpack8(xr[i], a);
    if (HAS_RES) {
      float b[8];
      unpack8(rr[i], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += b[j];
    }
    if (WRITE_RES) {
      uint4 q = pack8(a);
      ro[i] = q;
      unpack8(q, a);  // normalise what was stored, so backward sees identical values
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += a[j] * a[j];
  }
  ss = warp_sum(ss);
  const float rs = rsqrtf(ss / (float)D + eps);
  if (lane == 0 && rstd != nullptr) rstd[row] = rs;
  const uint4* src = WRITE_RES ? reinterpret_cast<const uint4*>(res_out + row * D) : xr;
  const uint4* wv = reinterpret_cast<const uint4*>(w);
  const uint4* gv = GATE ? reinterpret_cast<const uint4*>(gate + gate_at(at.heads, at.ldg, row, D)) : nullptr;
  uint4* yo = reinterpret_cast<uint4*>(y + row * D);
  for (int i = lane; i < nvec; i += 32) {
    float a[8], ww[8];
    unpack8(src[i], a);
    if (HAS_RES && !WRITE_RES) {
      float b[8];
      unpack8(rr[i], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += b[j];
    }
    if (w != nullptr) unpack8(wv[i], ww);
    float o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = a[j] * rs * (w != nullptr ? ww[j] : 1.f);
    if (GATE) {
      float g[8];
      unpack8(gv[i], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] *= (GATE == 1) ? g[j] * sigmoidf_(g[j]) : sigmoidf_(g[j]);
    }
    yo[i] = pack8(o);
  }
}

// The same for rows that a warp's registers hold (D <= 2048): NV vectors per lane of every operand, loaded at once and kept packed,
// so nothing is read twice and the second sweep waits for nothing: 32,768 rows of 2,048 65 -> 49 us, 65,536 of 1,024 64 -> 47 (with a
// residual 94 -> 86), 98,304 of 512 55 -> 37, with a gate 65 -> 59.  Vectors that a row does not fill cost warps: with a gate, three per lane
// for rows of up to 768 (131,072 of 520: 102 us with four, 84 with three, 92 by the form above), with a residual five for up to 1,280 (65,536
// of 1,152: 113 with eight, 91, 104).  A gate of 2,048 leaves too few warps (84 -> 88): that and wider rows take the form above.
template <bool HAS_RES, bool WRITE_RES, int GATE, int NV>
__global__ void __launch_bounds__(WARPS * 32)
rmsnorm_fwd_row_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res_in, const __nv_bfloat16* __restrict__ w,
                       const __nv_bfloat16* __restrict__ gate, __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ res_out,
                       float* __restrict__ rstd, long long rows, int D, float eps, const Rows at) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * WARPS + warp;
  if (row >= rows) return;
  const int count = ((D >> 3) - lane + 31) >> 5;  // vectors of this lane (none: 0)
  const uint4* xr = reinterpret_cast<const uint4*>(x + mapped_row(at, row) * D) + lane;
  const uint4* rr = HAS_RES ? reinterpret_cast<const uint4*>(res_in + row * D) + lane : nullptr;
  const uint4* gv = GATE ? reinterpret_cast<const uint4*>(gate + gate_at(at.heads, at.ldg, row, D)) + lane : nullptr;
  const uint4 none = make_uint4(0, 0, 0, 0);
  uint4 xa[NV], ra[HAS_RES ? NV : 1], ta[GATE ? NV : 1];
#pragma unroll
  for (int k = 0; k < NV; ++k) xa[k] = k < count ? xr[k * 32] : none;
  if (HAS_RES) {
#pragma unroll
    for (int k = 0; k < NV; ++k) ra[k] = k < count ? rr[k * 32] : none;
  }
  if (GATE) {
#pragma unroll
    for (int k = 0; k < NV; ++k) ta[k] = k < count ? gv[k * 32] : none;
  }
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    float a[8];
    unpack8(xa[k], a);
    if (HAS_RES) {
      float b[8];
      unpack8(ra[k], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += b[j];
    }
    if (WRITE_RES) {
      xa[k] = pack8(a);
      if (k < count) reinterpret_cast<uint4*>(res_out + row * D)[lane + k * 32] = xa[k];
      unpack8(xa[k], a);  // normalise what was stored, so backward sees identical values
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += a[j] * a[j];
  }
  ss = warp_sum(ss);
  const float rs = rsqrtf(ss / (float)D + eps);
  if (lane == 0 && rstd != nullptr) rstd[row] = rs;
  const uint4* wv = reinterpret_cast<const uint4*>(w) + lane;
  uint4* yo = reinterpret_cast<uint4*>(y + row * D) + lane;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    if (k >= count) break;
    float a[8], ww[8];
    unpack8(xa[k], a);
    if (HAS_RES && !WRITE_RES) {
      float b[8];
      unpack8(ra[k], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += b[j];
    }
    if (w != nullptr) unpack8(__ldg(wv + k * 32), ww);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = a[j] * rs * (w != nullptr ? ww[j] : 1.f);
    if (GATE) {
      float g[8];
      unpack8(ta[k], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] *= (GATE == 1) ? g[j] * sigmoidf_(g[j]) : sigmoidf_(g[j]);
    }
    yo[k * 32] = pack8(a);
  }
}

// Forward for short rows (D <= 256): LPR = D / 8 lanes (rounded up to a power of two) share a row, so that a warp of the
// per-head norms is full, and a thread takes FR rows at once to keep FR (gated: 2 FR) 16-byte loads in flight.  D = 128,
// 524,288 rows: the one-warp-per-row form above took 0.107 ms (2.5 TB/s), half of its lanes without work.
constexpr int FR = 4;
template <bool HAS_RES, bool WRITE_RES, int GATE, int LPR>
__global__ void __launch_bounds__(WARPS * 32)
rmsnorm_fwd_short_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res_in, const __nv_bfloat16* __restrict__ w,
                         const __nv_bfloat16* __restrict__ gate, __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ res_out,
                         float* __restrict__ rstd, long long rows, int D, float eps, const Rows at) {
  constexpr int SLOTS = WARPS * 32 / LPR;
  const int l = threadIdx.x % LPR, col = l * 8;
  const bool live = col < D;
  const long long r0 = (long long)blockIdx.x * (SLOTS * FR) + threadIdx.x / LPR;
  float ww[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) ww[j] = 1.f;
  if (w != nullptr && live) unpack8(*reinterpret_cast<const uint4*>(w + col), ww);
  uint4 xa[FR], ra[HAS_RES ? FR : 1], ta[GATE ? FR : 1];
#pragma unroll
  for (int k = 0; k < FR; ++k) {
    const long long row = r0 + k * SLOTS;
    const bool ok = live && row < rows;
    xa[k] = ok ? *reinterpret_cast<const uint4*>(x + mapped_row(at, row) * D + col) : make_uint4(0, 0, 0, 0);
    if (HAS_RES) ra[k] = ok ? *reinterpret_cast<const uint4*>(res_in + row * D + col) : make_uint4(0, 0, 0, 0);
    if (GATE) ta[k] = ok ? *reinterpret_cast<const uint4*>(gate + gate_at(at.heads, at.ldg, row, D) + col) : make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int k = 0; k < FR; ++k) {
    const long long row = r0 + k * SLOTS;
    const bool ok = live && row < rows;
    float a[8];
    unpack8(xa[k], a);
    if (HAS_RES) {
      float b[8];
      unpack8(ra[k], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += b[j];
    }
    if (WRITE_RES) {
      const uint4 q = pack8(a);
      if (ok) *reinterpret_cast<uint4*>(res_out + row * D + col) = q;
      unpack8(q, a);  // normalise what was stored, so backward sees identical values
    }
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += a[j] * a[j];
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float rs = rsqrtf(ss / (float)D + eps);
    if (l == 0 && row < rows && rstd != nullptr) rstd[row] = rs;
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = a[j] * rs * ww[j];
    if (GATE) {
      float g[8];
      unpack8(ta[k], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] *= (GATE == 1) ? g[j] * sigmoidf_(g[j]) : sigmoidf_(g[j]);
    }
    if (ok) *reinterpret_cast<uint4*>(y + row * D + col) = pack8(a);
  }
}

// Backward.  `xin` is the tensor that was normalised (the stored residual sum when a residual was fused).  A thread owns
// eight columns and keeps their dw in registers over all rows of its CTA; a row belongs to LPR lanes (D <= 512, LPR = D / 8
// rounded up to a power of two, several rows side by side; 64 lanes are two warps, whose sums meet in shared memory) or to the
// whole CTA (LPR = 0, D / 8 threads rounded up to warps, sums through shared memory).  Rows of 257 to 512 as CTAs of 64 threads
// left an SM with eight warps: 98,304 rows of 512 with a gate 157 us, 65,536 of 320 107; four rows side by side take 118 and 77.
// For 1,024 two rows side by side and one CTA each are equal (105 : 111 us with a residual, 91 : 87 without): one CTA each stays.
// BR rows per trip: their 2 BR to 3 BR 16-byte loads are issued together and stay packed in registers, so every operand is read
// once.  The next trip's go out before this trip's sums (AHEAD), so memory is busy while the CTA computes; what 128 registers hold
// of two trips sets BR, and 80 where a gate leaves more to compute and three CTAs pay: 98,304 rows of 512 with a gate 118 -> 101 us,
// 262,144 of 256 142 -> 130 (of the chunk layout 156 -> 148), 65,536 of 320 77 -> 66, of 1,024 with a residual 111 -> 101, 32,768 of 2,048
// 95 -> 89.  Gated rows of a whole CTA are slower with it (150 -> 158) and keep two rows and no lead.
// Rows of up to 256 without gate and residual: two per trip while the operands stay in L2 (below 2^24 elements), 65,536 of 64 12.9 us and
// 8,192 9.7 where four per trip take 13.3 and 11.4; four beyond, 1,048,576 of 64 73 us where two take 83.  A lead and four rows of 129 to 256
// are more than the registers hold (spilled): 262,144 of 256 75 us without the lead, 90 with it.
// dw partials: one row per CTA, which a second kernel sums in order.
template <bool HAS_DRES, int GATE, int LPR, int BR, int TPB, bool MAP>
__global__ void __launch_bounds__(TPB, TPB != 256 ? 1 : GATE && LPR ? 3 : 2)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ xin, const __nv_bfloat16* __restrict__ w,
                   const float* __restrict__ rstd, const __nv_bfloat16* __restrict__ gate, const __nv_bfloat16* __restrict__ dres,
                   __nv_bfloat16* __restrict__ dx, __nv_bfloat16* __restrict__ dgate, float* __restrict__ dw_part, long long rows, int D,
                   int rows_per_cta, const Rows at) {
  constexpr int SLOTS = LPR ? WARPS * 32 / (LPR ? LPR : 1) : 1;
  // the next trip's loads go out before this trip's sums
  constexpr bool AHEAD = TPB == 256 && !(GATE && LPR == 0) && !(BR == 4 && LPR == 32);
  constexpr bool WIDE = LPR == 0 || LPR > 32;  // a row belongs to several warps
  __shared__ float s_c[WIDE ? 2 : 1][WIDE ? BR : 1][WIDE ? 32 : 1];
  __shared__ float s_dw[LPR ? SLOTS : 1][LPR ? LPR * 8 + 1 : 1];
  const int l = LPR ? threadIdx.x % (LPR ? LPR : 1) : threadIdx.x, slot = LPR ? threadIdx.x / (LPR ? LPR : 1) : 0;
  const int col = l * 8;
  const bool live = col < D;
  const long long row0 = (long long)blockIdx.x * rows_per_cta, row1 = min(rows, row0 + rows_per_cta);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = (LPR ? LPR : blockDim.x) >> 5;
  float ww[8], dw[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) ww[j] = 1.f, dw[j] = 0.f;
  if (w != nullptr && live) unpack8(*reinterpret_cast<const uint4*>(w + col), ww);
  const float inv_d = 1.f / (float)D;
  int flip = 0;
  int ahead[MAP ? BR : 1];  // the next trip's `from`, on its way while this trip works: without it every trip waits twice
  auto look = [&](long long rb) {
#pragma unroll
    for (int k = 0; k < BR; ++k) {
      const long long row = rb + slot + k * SLOTS;
      if (MAP) ahead[k] = row < row1 ? (int)mapped_row(at, row) : -1;
    }
  };
  if (MAP) look(row0);
  uint4 xa[BR], ga[BR], ra[HAS_DRES ? BR : 1], ta[GATE ? BR : 1];
  float rs[BR], c[BR];
  int from[MAP ? BR : 1];  // the packed row, -1 where there is none: its gradient is zero
  auto load = [&](long long rb, uint4 (&xa)[BR], uint4 (&ga)[BR], uint4 (&ra)[HAS_DRES ? BR : 1], uint4 (&ta)[GATE ? BR : 1], float (&rs)[BR],
                  int (&from)[MAP ? BR : 1]) {
#pragma unroll
    for (int k = 0; k < (MAP ? BR : 1); ++k)
      if (MAP) from[k] = ahead[k];
#pragma unroll
    for (int k = 0; k < BR; ++k) {
      const long long row = rb + slot + k * SLOTS, pr = MAP ? from[k] : row;
      const bool there = MAP ? pr >= 0 : row < row1, ok = live && there;
      // streaming loads: every operand row is read exactly once
      const uint4 none = make_uint4(0, 0, 0, 0);
      xa[k] = ok ? __ldcs(reinterpret_cast<const uint4*>(xin + row * D + col)) : none;
      ga[k] = ok ? __ldcs(reinterpret_cast<const uint4*>(dy + pr * D + col)) : none;
      if (HAS_DRES) ra[k] = ok ? __ldcs(reinterpret_cast<const uint4*>(dres + pr * D + col)) : none;
      if (GATE) ta[k] = ok ? __ldcs(reinterpret_cast<const uint4*>(gate + gate_at(at.heads, at.ldg, pr, D) + col)) : none;
      rs[k] = there ? rstd[pr] : 0.f;
    }
    if (MAP) look(rb + SLOTS * BR);
  };
  uint4 xn[BR], gn[BR], rn[HAS_DRES ? BR : 1], tn[GATE ? BR : 1];  // AHEAD: the next trip's
  float sn[BR];
  int fn[MAP ? BR : 1];
  if constexpr (AHEAD) load(row0, xn, gn, rn, tn, sn, fn);
  for (long long rb = row0; rb < row1; rb += SLOTS * BR, flip ^= 1) {
    if constexpr (AHEAD) {
#pragma unroll
      for (int k = 0; k < BR; ++k) {
        xa[k] = xn[k], ga[k] = gn[k], rs[k] = sn[k];
        if (HAS_DRES) ra[k] = rn[k];
        if (GATE) ta[k] = tn[k];
        if (MAP) from[k] = fn[k];
      }
      load(rb + SLOTS * BR, xn, gn, rn, tn, sn, fn);
    } else {
      load(rb, xa, ga, ra, ta, rs, from);
    }
#pragma unroll
    for (int k = 0; k < BR; ++k) {
      float a[8], g[8];
      unpack8(xa[k], a);
      unpack8(ga[k], g);
      if (GATE) {
        float gt[8];
        unpack8(ta[k], gt);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float sg = sigmoidf_(gt[j]);
          g[j] *= (GATE == 1) ? gt[j] * sg : sg;
        }
      }
      float s = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) s += g[j] * ww[j] * a[j] * rs[k];
#pragma unroll
      for (int o = (WIDE ? 32 : LPR) / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      c[k] = s * inv_d;
    }
    if constexpr (WIDE) {
      if (lane == 0) {
#pragma unroll
        for (int k = 0; k < BR; ++k) s_c[flip][k][warp] = c[k];
      }
      __syncthreads();  // the two buffers alternate: one barrier per trip separates the writes of a buffer from its last reads
#pragma unroll
      for (int k = 0; k < BR; ++k) {
        float s = 0.f;
        for (int i = 0; i < nwarps; ++i) s += s_c[flip][k][slot * nwarps + i];
        c[k] = s;
      }
    }
    // keep the compiler from carrying the unpacked fp32 values of the first pass (twice the registers) into the second
#pragma unroll
    for (int k = 0; k < BR; ++k) {
      asm volatile("" : "+r"(xa[k].x), "+r"(xa[k].y), "+r"(xa[k].z), "+r"(xa[k].w));
      asm volatile("" : "+r"(ga[k].x), "+r"(ga[k].y), "+r"(ga[k].z), "+r"(ga[k].w));
      if (GATE) asm volatile("" : "+r"(ta[k].x), "+r"(ta[k].y), "+r"(ta[k].z), "+r"(ta[k].w));
    }
#pragma unroll
    for (int k = 0; k < BR; ++k) {
      const long long row = rb + slot + k * SLOTS;
      float a[8], g[8], o[8], gt[8], dgo[8];
      unpack8(xa[k], a);
      unpack8(ga[k], g);
      if (GATE) unpack8(ta[k], gt);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xhat = a[j] * rs[k];
        float gy = g[j];
        if (GATE) {
          const float sg = sigmoidf_(gt[j]);
          const float act = (GATE == 1) ? gt[j] * sg : sg;
          const float dact = (GATE == 1) ? sg * (1.f + gt[j] * (1.f - sg)) : sg * (1.f - sg);
          dgo[j] = g[j] * xhat * ww[j] * dact;
          gy = g[j] * act;
        }
        o[j] = rs[k] * (gy * ww[j] - xhat * c[k]);
        dw[j] += gy * xhat;
      }
      if (HAS_DRES) {
        float b[8];
        unpack8(ra[k], b);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] += b[j];
      }
      if (live && row < row1) {
        __stcs(reinterpret_cast<uint4*>(dx + row * D + col), pack8(o));
        if (GATE && (!MAP || from[k] >= 0))
          __stcs(reinterpret_cast<uint4*>(dgate + gate_at(at.heads, at.lddg, MAP ? from[k] : row, D) + col), pack8(dgo));
      }
    }
  }
  if (w == nullptr) return;
  if constexpr (LPR == 0) {
    if (live) {
#pragma unroll
      for (int j = 0; j < 8; ++j) dw_part[(long long)blockIdx.x * D + col + j] = dw[j];
    }
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) s_dw[slot][col + j] = dw[j];
    __syncthreads();
    for (int i = threadIdx.x; i < D; i += blockDim.x) {
      float t = 0.f;
#pragma unroll 8
      for (int k = 0; k < SLOTS; ++k) t += s_dw[k][i];
      dw_part[(long long)blockIdx.x * D + i] = t;
    }
  }
}

// Column sums of the CTAs' partial rows in a fixed order: 32 columns x 16 groups of rows per block.
constexpr int CS_GROUPS = 16;
__global__ void __launch_bounds__(32 * CS_GROUPS) colsum_partials_kernel(const float* __restrict__ part, int nparts, int D,
                                                                         float* __restrict__ out, int accumulate) {
  __shared__ float red[CS_GROUPS][33];
  const int i = blockIdx.x * 32 + threadIdx.x;
  float s = 0.f;
  if (i < D) {
#pragma unroll 8
    for (int p = threadIdx.y; p < nparts; p += CS_GROUPS) s += part[(long long)p * D + i];
  }
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y != 0 || i >= D) return;
#pragma unroll
  for (int k = 1; k < CS_GROUPS; ++k) s += red[k][threadIdx.x];
  out[i] = accumulate ? out[i] + s : s;
}

// Column sums of a bf16 matrix (a bias' gradient): 256 columns x 8 groups of rows per block, four rows' loads in flight per thread.
// 65,536 x 512: torch's reduction took 0.057 ms, the bytes take 0.010.
constexpr int CB_ROWS = 8;
__global__ void __launch_bounds__(32 * CB_ROWS) colsum_bf16_kernel(const __nv_bfloat16* __restrict__ x, long long ld, long long rows, int cols,
                                                                   float* __restrict__ part) {
  __shared__ float red[CB_ROWS][257];
  const int col = (blockIdx.x * 32 + threadIdx.x) * 8;
  float s[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) s[j] = 0.f;
  if (col < cols) {
    const long long step = (long long)gridDim.y * CB_ROWS;
    for (long long r = (long long)blockIdx.y * CB_ROWS + threadIdx.y; r < rows; r += 4 * step) {
      uint4 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = r + k * step < rows ? *reinterpret_cast<const uint4*>(x + (r + k * step) * ld + col) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float f[8];
        unpack8(v[k], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] += f[j];
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) red[threadIdx.y][threadIdx.x * 8 + j] = s[j];
  __syncthreads();
  const int t = threadIdx.y * 32 + threadIdx.x, c = blockIdx.x * 256 + t;
  if (c >= cols) return;
  float v = 0.f;
#pragma unroll
  for (int k = 0; k < CB_ROWS; ++k) v += red[k][t];
  part[(long long)blockIdx.y * cols + c] = v;
}

}  // namespace

extern "C" {

int fb_colsum_bf16_parts(long long rows, int cols) {
  const long long want = (rows + 4 * CB_ROWS - 1) / (4 * CB_ROWS), most = 592 / ((cols + 255) / 256);
  return (int)(want < 1 ? 1 : want < most ? want : most < 1 ? 1 : most);
}
// out[cols] (fp32) = column sums of x [rows, cols] bf16, rows ld elements apart; part: fp32 [fb_colsum_bf16_parts, cols] scratch
int fb_colsum_bf16(const void* x, long long ld, long long rows, int cols, float* part, float* out, cudaStream_t stream) {
  if (cols == 0) return 0;
  if ((cols & 7) || (ld & 7) || !fb::aligned(16, x)) return -2;
  const int parts = fb_colsum_bf16_parts(rows, cols);
  colsum_bf16_kernel<<<dim3((cols + 255) / 256, parts), dim3(32, CB_ROWS), 0, stream>>>((const __nv_bfloat16*)x, ld, rows, cols, part);
  int rc = fb::launch_ok("colsum_bf16_kernel");
  if (rc) return rc;
  colsum_partials_kernel<<<(cols + 31) / 32, dim3(32, CS_GROUPS), 0, stream>>>(part, parts, cols, out, 0);
  return fb::launch_ok("colsum_partials_kernel");
}

// out[cols] = column sums of the fp32 partials [parts, cols], in a fixed order (the scan's gradients of A and D, [518, 16, 2048] and
// [518, 2048]: 28 + 22 us by the general reduction, which takes few blocks along the columns; 22 us here, the bytes take 11)
int fb_colsum_parts(const float* part, int parts, int cols, float* out, cudaStream_t stream) {
  if (cols <= 0) return 0;
  colsum_partials_kernel<<<(cols + 31) / 32, dim3(32, CS_GROUPS), 0, stream>>>(part, parts, cols, out, 0);
  return fb::launch_ok("colsum_partials_kernel");
}

// Number of CTAs (= rows of the dw partial buffer) the backward launches for `rows` rows.
int fb_rmsnorm_bwd_parts(long long rows) {
  long long want = (rows + WARPS - 1) / WARPS;
  return (int)(want < 592 ? (want < 1 ? 1 : want) : 592);  // two resident CTAs on each of 148 SMs: two full waves
}

// map, heads, ldg (0: the gate's rows are side by side): see Rows
int fb_rmsnorm_fwd(const void* x, const void* res_in, const void* w, const void* gate, void* y, void* res_out,
                   float* rstd, long long rows, int D, float eps, int gate_mode, const int* map, int heads, long long ldg, cudaStream_t stream) {
  if (rows == 0) return 0;
  if (D % 8 || heads < 1 || rows % heads || ldg % 8 || (rows >= (1ll << 31) && (map || ldg)) || !fb::aligned(16, x, res_in, w, gate, y, res_out))
    return -2;
  const Rows at{map, (unsigned)heads, ldg ? ldg : (long long)heads * D, 0};
  const int lpr = D <= 64 ? 8 : D <= 128 ? 16 : 32;  // lanes of a row, D <= 256
  const int per_block = D <= 256 ? WARPS * 32 / lpr * FR : WARPS;
  const unsigned grid = (unsigned)((rows + per_block - 1) / per_block);
  const auto X = (const __nv_bfloat16*)x;
  const auto R = (const __nv_bfloat16*)res_in;
  const auto W = (const __nv_bfloat16*)w;
  const auto G = (const __nv_bfloat16*)gate;
  auto Y = (__nv_bfloat16*)y;
  auto RO = (__nv_bfloat16*)res_out;
#define FWD_S(HR, WR, GM, LP) \
  rmsnorm_fwd_short_kernel<HR, WR, GM, LP><<<grid, WARPS * 32, 0, stream>>>(X, R, W, G, Y, RO, rstd, rows, D, eps, at)
#define FWD_R(HR, WR, GM, NV) \
  rmsnorm_fwd_row_kernel<HR, WR, GM, NV><<<grid, WARPS * 32, 0, stream>>>(X, R, W, G, Y, RO, rstd, rows, D, eps, at)
#define FWD(HR, WR, GM)                                                                                            \
  do {                                                                                                             \
    if (D <= 64) FWD_S(HR, WR, GM, 8);                                                                             \
    else if (D <= 128) FWD_S(HR, WR, GM, 16);                                                                      \
    else if (D <= 256) FWD_S(HR, WR, GM, 32);                                                                      \
    else if (D <= 512) FWD_R(HR, WR, GM, 2);                                                                       \
    else if (D <= 768) FWD_R(HR, WR, GM, (GM ? 3 : 4));                                                            \
    else if (D <= 1024) FWD_R(HR, WR, GM, 4);                                                                      \
    else if (D <= 1280 && !GM) FWD_R(HR, WR, GM, (GM ? 4 : HR ? 5 : 8));                                           \
    else if (D <= 2048 && !GM) FWD_R(HR, WR, GM, (GM ? 4 : 8));                                                    \
    else rmsnorm_fwd_kernel<HR, WR, GM><<<grid, WARPS * 32, 0, stream>>>(X, R, W, G, Y, RO, rstd, rows, D, eps, at);   \
  } while (0)
  if (gate_mode == 0) {
    if (res_in && res_out) FWD(true, true, 0);
    else if (res_in) FWD(true, false, 0);
    else FWD(false, false, 0);
  } else if (gate_mode == 1) {
    FWD(false, false, 1);
  } else {
    FWD(false, false, 2);
  }
#undef FWD
#undef FWD_S
#undef FWD_R
  return fb::launch_ok("rmsnorm_fwd_kernel");
}

// rows: of xin and dx.  dw_part: fp32 [fb_rmsnorm_bwd_parts(rows), D] scratch; dw: fp32 [D] (accumulated when accumulate_dw != 0).
int fb_rmsnorm_bwd_rows(const void* dy, const void* xin, const void* w, const float* rstd, const void* gate,
                        const void* dres, void* dx, void* dgate, float* dw_part, float* dw, long long rows, int D,
                        int gate_mode, int accumulate_dw, const int* map, int heads, long long ldg, long long lddg, cudaStream_t stream) {
  if (rows == 0) return 0;
  if (D % 8 || heads < 1 || rows % heads || ldg % 8 || lddg % 8 || (rows >= (1ll << 31) && (map || ldg || lddg)) ||
      !fb::aligned(16, dy, xin, w, gate, dres, dx, dgate))
    return -2;
  const Rows at{map, (unsigned)heads, ldg ? ldg : (long long)heads * D, lddg ? lddg : (long long)heads * D};
  // resident CTAs: two on each of 148 SMs, two waves of them; three with a gate and rows side by side, one wave
  const int most = fb_rmsnorm_bwd_parts(rows), parts = gate_mode && D <= 512 && most > 444 ? 444 : most;
  const int rows_per_cta = (int)((rows + parts - 1) / parts);
  if (D > 7040) return -3;
  const int threads = D <= 512 ? WARPS * 32 : (D / 8 + 31) / 32 * 32;
#define BWD_N(HD, GM, LP, NR, TPB)                                                                                  \
  (map ? rmsnorm_bwd_kernel<HD, GM, LP, NR, TPB, true> : rmsnorm_bwd_kernel<HD, GM, LP, NR, TPB, false>)<<<parts, threads, 0, stream>>>( \
      (const __nv_bfloat16*)dy, (const __nv_bfloat16*)xin, (const __nv_bfloat16*)w, rstd, (const __nv_bfloat16*)gate, \
      (const __nv_bfloat16*)dres, (__nv_bfloat16*)dx, (__nv_bfloat16*)dgate, dw_part, rows, D, rows_per_cta, at)
  const bool four = rows * D >= (1ll << 24);
#define BWD_S(HD, GM, LP)                                                                                         \
  do {                                                                                                            \
    if (!GM && !HD && four) BWD_N(HD, GM, LP, (GM || HD ? 2 : 4), 256);                                           \
    else BWD_N(HD, GM, LP, (GM ? 1 : 2), 256);                                                                    \
  } while (0)
  // rows per trip by what the registers hold packed; one row and no lead where a CTA has more than eight warps to overlap (64 registers)
#define BWD(HD, GM)                                                                                               \
  do {                                                                                                            \
    if (D <= 64) BWD_S(HD, GM, 8);                                                                                \
    else if (D <= 128) BWD_S(HD, GM, 16);                                                                         \
    else if (D <= 256) BWD_S(HD, GM, 32);                                                                         \
    else if (D <= 512) BWD_N(HD, GM, 64, (GM ? 1 : 2), 256);                                                      \
    else if (D <= 2048) BWD_N(HD, GM, 0, 2, 256);                                                                 \
    else BWD_N(HD, GM, 0, 1, 1024);                                                                               \
  } while (0)
  if (gate_mode == 0) {
    if (dres) { BWD(true, 0); } else { BWD(false, 0); }
  } else if (gate_mode == 1) {
    BWD(false, 1);
  } else {
    BWD(false, 2);
  }
#undef BWD
#undef BWD_S
#undef BWD_N
  int rc = fb::launch_ok("rmsnorm_bwd_kernel");
  if (rc) return rc;
  if (w != nullptr) {
    colsum_partials_kernel<<<(D + 31) / 32, dim3(32, CS_GROUPS), 0, stream>>>(dw_part, parts, D, dw, accumulate_dw);
    rc = fb::launch_ok("colsum_partials_kernel");
  }
  return rc;
}

// The same with every row in its place.
int fb_rmsnorm_bwd(const void* dy, const void* xin, const void* w, const float* rstd, const void* gate,
                   const void* dres, void* dx, void* dgate, float* dw_part, float* dw, long long rows, int D,
                   int gate_mode, int accumulate_dw, cudaStream_t stream) {
  return fb_rmsnorm_bwd_rows(dy, xin, w, rstd, gate, dres, dx, dgate, dw_part, dw, rows, D, gate_mode, accumulate_dw, nullptr, 1, 0, 0, stream);
}

}  // extern "C"

// ------------------------------------------------------------------------------------------------
// Allocation-free variant (declared in flame_b200_noalloc.h)
// ------------------------------------------------------------------------------------------------
namespace {
constexpr int kNoAllocParts = 592;   // upper bound of fb_rmsnorm_bwd_parts()
constexpr int kNoAllocMaxDevices = 64;
// Scratch for the per-CTA dw partial sums.  In host code this name is only a stand-in for the symbol; the
// address a kernel can use is obtained once per device with cudaGetSymbolAddress below.
static __device__ __align__(256) float g_noalloc_dw_part[(size_t)kNoAllocParts * FB_NOALLOC_MAX_D];
static float* g_noalloc_dw_part_addr[kNoAllocMaxDevices] = {nullptr};
}  // namespace

extern "C" int fb_rmsnorm_bwd_noalloc(const void* dy, const void* xin, const void* w, const float* rstd, void* dx,
                                      float* dw, long long rows, int D, int accumulate_dw, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (D <= 0 || (D % 8) != 0) {
    fprintf(stderr, "[flame_b200] fb_rmsnorm_bwd_noalloc: D=%d must be a positive multiple of 8\n", D);
    return -2;
  }
  if (D > FB_NOALLOC_MAX_D) {
    fprintf(stderr,
            "[flame_b200] fb_rmsnorm_bwd_noalloc: D=%d exceeds the built-in scratch (max D = %d); use fb_rmsnorm_bwd "
            "with caller-provided scratch instead\n", D, FB_NOALLOC_MAX_D);
    return -3;
  }
  if (w == nullptr || dw == nullptr) {
    fprintf(stderr, "[flame_b200] fb_rmsnorm_bwd_noalloc: w and dw are required\n");
    return -4;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices) {
    fprintf(stderr, "[flame_b200] fb_rmsnorm_bwd_noalloc: cannot identify the current device\n");
    return -5;
  }
  if (g_noalloc_dw_part_addr[dev] == nullptr) {
    // one-time set-up for this device, with this device current
    float* p = nullptr;
    e = cudaGetSymbolAddress((void**)&p, g_noalloc_dw_part);
    if (e != cudaSuccess || p == nullptr) {
      fprintf(stderr, "[flame_b200] fb_rmsnorm_bwd_noalloc: cudaGetSymbolAddress failed: %s\n", cudaGetErrorString(e));
      return (int)(e != cudaSuccess ? e : cudaErrorInvalidSymbol);
    }
    g_noalloc_dw_part_addr[dev] = p;
  }
  // same kernels and launch shape as fb_rmsnorm_bwd; only the origin of the scratch differs
  return fb_rmsnorm_bwd(dy, xin, w, rstd, nullptr, nullptr, dx, nullptr, g_noalloc_dw_part_addr[dev], dw, rows, D, 0,
                        accumulate_dw, stream);
}

