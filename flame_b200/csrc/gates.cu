// Fused gate arithmetic of the linear-attention layers: what the reference leaves to a chain of elementwise framework
// kernels (ten passes forward, fifteen backward over [tokens, hidden] fp32 tensors for HGRN2), one pass each way.
//
// HGRN2 (fla/layers/hgrn2.py:160-190):
//   q = silu(q_raw)
//   g = logsigmoid(f_raw)                                        (no lower bound)
//   g = log(lb + (1 - lb) sigmoid(f_raw))                        (with a per-channel lower bound lb in (0, 1))
//   k = 1 - exp(g)
// Outputs: q, k in bf16, g in fp32 (the log decay the chunk kernels consume).  The backward takes dq, dk (bf16) and dg
// (fp32), recomputes the gate from f_raw and returns dq_raw, df_raw and the per-channel sum of dlb.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "fine_math.cuh"
#include "host_utils.cuh"

namespace {

__device__ __forceinline__ void unpack8(const uint4& q, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = __bfloat1622float2(h[i]);
    f[2 * i] = v.x;
    f[2 * i + 1] = v.y;
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
// log(sigmoid(x)) without cancellation or underflow
__device__ __forceinline__ float logsigmoidf_(float x) { return fminf(x, 0.f) - log1pf(__expf(-fabsf(x))); }

// g = logsigmoid(x) / n in fp32 from bf16 x, and with SLOTS s = 1 - exp(g) too (GLA's and GSA's forget gates,
// fla/layers/gla.py:205-212, fla/layers/gsa.py:173-176).  Bound by memory: torch's chain (widen, logsigmoid, divide, and the same
// back) moved 24 bytes per element forward and 30 backward where 6 and 8 are needed.  x may be a column block (ldx); with a map g and s are
// in the padded rows of the chunk layout: forward map[padded row] = row of x or -1 (zeros), backward map[row of x] = padded row.
template <bool SLOTS>
__global__ void logsigmoid_gate_fwd_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const int* __restrict__ map, float* __restrict__ g,
                                           float* __restrict__ s, float n, long long total, long long vecs) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const long long row = i / vecs, from = map == nullptr ? row : map[row];
  float f[8], sv[8];
  unpack8(from >= 0 ? *reinterpret_cast<const uint4*>(x + from * ldx + (i - row * vecs) * 8) : make_uint4(0, 0, 0, 0), f);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    f[c] = from >= 0 ? __fdiv_rn(logsigmoidf_(f[c]), n) : 0.f;
    if (SLOTS) sv[c] = -expm1f(f[c]);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    reinterpret_cast<float4*>(g)[2 * i + h] = make_float4(f[4 * h], f[4 * h + 1], f[4 * h + 2], f[4 * h + 3]);
    if (SLOTS) reinterpret_cast<float4*>(s)[2 * i + h] = make_float4(sv[4 * h], sv[4 * h + 1], sv[4 * h + 2], sv[4 * h + 3]);
  }
}

// dx = (dg - exp(g) ds) sigmoid(-x) / n
template <bool SLOTS>
__global__ void logsigmoid_gate_bwd_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const int* __restrict__ map, const float* __restrict__ dg,
                                           const float* __restrict__ ds, __nv_bfloat16* __restrict__ dx, long long lddx, float n, long long total,
                                           long long vecs) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const long long row = i / vecs, col = i - row * vecs, at = (map == nullptr ? row : map[row]) * vecs + col;
  float f[8], o[8];
  unpack8(*reinterpret_cast<const uint4*>(x + row * ldx + col * 8), f);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float4 a = reinterpret_cast<const float4*>(dg)[2 * at + h];
    o[4 * h] = a.x, o[4 * h + 1] = a.y, o[4 * h + 2] = a.z, o[4 * h + 3] = a.w;
    if (SLOTS) {
      const float4 b = reinterpret_cast<const float4*>(ds)[2 * at + h];
      const float bs[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int c = 0; c < 4; ++c) o[4 * h + c] -= __expf(__fdiv_rn(logsigmoidf_(f[4 * h + c]), n)) * bs[c];
    }
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) o[c] = __fdiv_rn(o[c] * sigmoidf_(-f[c]), n);
  *reinterpret_cast<uint4*>(dx + row * lddx + col * 8) = pack8(o);
}

// one thread per (row, 8 channels)
template <bool HAS_LB>
__global__ void hgrn2_gate_fwd_kernel(const __nv_bfloat16* __restrict__ qr, const __nv_bfloat16* __restrict__ fr,
                                      const float* __restrict__ lb, __nv_bfloat16* __restrict__ q,
                                      __nv_bfloat16* __restrict__ k, float* __restrict__ g, long long rows, int D) {
  const int vecs = D >> 3;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long row = gid / vecs;
  if (row >= rows) return;
  const int d0 = (int)(gid - row * vecs) * 8;
  const long long off = row * D + d0;
  float a[8], f[8], qo[8], ko[8], go[8];
  unpack8(*reinterpret_cast<const uint4*>(qr + off), a);
  unpack8(*reinterpret_cast<const uint4*>(fr + off), f);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    qo[c] = a[c] * sigmoidf_(a[c]);
    float gs = logsigmoidf_(f[c]);
    if (HAS_LB) {
      const float l = lb[d0 + c];
      gs = __logf(l + (1.f - l) * __expf(gs));
    }
    go[c] = gs;
    ko[c] = 1.f - __expf(gs);
  }
  *reinterpret_cast<uint4*>(q + off) = pack8(qo);
  *reinterpret_cast<uint4*>(k + off) = pack8(ko);
  *reinterpret_cast<float4*>(g + off) = make_float4(go[0], go[1], go[2], go[3]);
  *reinterpret_cast<float4*>(g + off + 4) = make_float4(go[4], go[5], go[6], go[7]);
}

constexpr int GATE_TILE_ROWS = 64;  // rows per block of the backward; a block covers 256 channels

// block = 32 channel vectors x 8 row lanes; a block walks 64 rows and leaves one partial row of dlb sums
template <bool HAS_LB>
__global__ void __launch_bounds__(256)
hgrn2_gate_bwd_kernel(const __nv_bfloat16* __restrict__ qr, const __nv_bfloat16* __restrict__ fr, const float* __restrict__ lb,
                      const __nv_bfloat16* __restrict__ dq, const __nv_bfloat16* __restrict__ dk, const float* __restrict__ dg,
                      __nv_bfloat16* __restrict__ dqr, __nv_bfloat16* __restrict__ dfr, float* __restrict__ dlb_part,
                      long long rows, int D) {
  __shared__ float red[8][256];
  const int vx = threadIdx.x & 31, ry = threadIdx.x >> 5;
  const int d0 = (blockIdx.x * 32 + vx) * 8;
  const bool col_ok = d0 < D;
  const long long r0 = (long long)blockIdx.y * GATE_TILE_ROWS;
  float lbv[8], acc[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    lbv[c] = (HAS_LB && col_ok) ? lb[d0 + c] : 0.f;
    acc[c] = 0.f;
  }
  if (col_ok) {
#pragma unroll 2
    for (int i = ry; i < GATE_TILE_ROWS; i += 8) {
      const long long row = r0 + i;
      if (row >= rows) break;
      const long long off = row * D + d0;
      float a[8], f[8], gq[8], gk[8], gg[8], oq[8], of[8];
      unpack8(*reinterpret_cast<const uint4*>(qr + off), a);
      unpack8(*reinterpret_cast<const uint4*>(fr + off), f);
      unpack8(*reinterpret_cast<const uint4*>(dq + off), gq);
      unpack8(*reinterpret_cast<const uint4*>(dk + off), gk);
      const float4 g0 = *reinterpret_cast<const float4*>(dg + off), g1 = *reinterpret_cast<const float4*>(dg + off + 4);
      gg[0] = g0.x; gg[1] = g0.y; gg[2] = g0.z; gg[3] = g0.w;
      gg[4] = g1.x; gg[5] = g1.y; gg[6] = g1.z; gg[7] = g1.w;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float sq = sigmoidf_(a[c]);
        oq[c] = gq[c] * sq * (1.f + a[c] * (1.f - sq));
        const float s = sigmoidf_(f[c]);
        if (HAS_LB) {
          const float l = lbv[c];
          const float e = l + (1.f - l) * s;           // exp(g), at least l > 0
          const float de = gg[c] / e - gk[c];          // g = log e, k = 1 - e
          of[c] = de * (1.f - l) * s * (1.f - s);
          acc[c] += de * (1.f - s);
        } else {
          // e = s: dg / s * s (1 - s) = dg (1 - s), which stays finite where s underflows
          of[c] = (gg[c] - gk[c] * s) * (1.f - s);
        }
      }
      *reinterpret_cast<uint4*>(dqr + off) = pack8(oq);
      *reinterpret_cast<uint4*>(dfr + off) = pack8(of);
    }
  }
  if (!HAS_LB) return;
#pragma unroll
  for (int c = 0; c < 8; ++c) red[ry][vx * 8 + c] = acc[c];
  __syncthreads();
  const int ch = threadIdx.x;  // one of the block's 256 channels
  const int d = blockIdx.x * 256 + ch;
  if (d < D) {
    float s = 0.f;
#pragma unroll
    for (int y = 0; y < 8; ++y) s += red[y][ch];
    dlb_part[(long long)blockIdx.y * D + d] = s;
  }
}

// out[d] = sum over `parts` partial rows, in a fixed order; block = 32 channels x 8 part lanes
__global__ void colsum_rows_kernel(const float* __restrict__ part, int parts, int D, float* __restrict__ out) {
  __shared__ float red[8][32];
  const int ix = threadIdx.x & 31, ky = threadIdx.x >> 5;
  const int d = blockIdx.x * 32 + ix;
  float s = 0.f;
  if (d < D)
    for (int k = ky; k < parts; k += 8) s += part[(long long)k * D + d];
  red[ky][ix] = s;
  __syncthreads();
  if (ky != 0 || d >= D) return;
#pragma unroll
  for (int k = 1; k < 8; ++k) s += red[k][ix];
  out[d] = s;
}

// ---------------------------------------------------------------------------------------------------------------
// The delta rule's gates (fla/layers/delta_net.py:246-252, fla/ops/gated_delta_rule/gate.py:20-44), per token and head:
//   beta = mul sigmoid(b),   g = -exp(A_log) softplus(a + dt_bias)
// read from column blocks of the projection and written as fp32 in the padded rows of the chunk layout (zeros in the
// padding).  A few scalars per token: what they cost is launches, not arithmetic, which is that of torch's fp32 functions or closer
// to the exact result (fine_math.cuh); one kernel stands for ten of torch's forward and one
// (and the sum of its partials) for fifteen backward.  src: packed token of a padded row (-1: padding), or null: the same.
template <bool BF16>
__device__ __forceinline__ float param(const void* p, int h) {
  return BF16 ? __bfloat162float(((const __nv_bfloat16*)p)[h]) : ((const float*)p)[h];
}
// softplus(x), with sigmoid(x) from the same exponential, which never overflows and whose logarithm does not round 1 + exp first
__device__ __forceinline__ float softplus_fine(float x, float& sigmoid) {
  const float e = exp_rn(-fabsf(x));
  sigmoid = __fdiv_rn(x >= 0.f ? 1.f : e, 1.f + e);
  return fmaxf(x, 0.f) + log1pf(e);
}

template <bool BF16>
__global__ void delta_gates_fwd_kernel(const __nv_bfloat16* __restrict__ b, long long ldb, const __nv_bfloat16* __restrict__ a, long long lda,
                                       const void* __restrict__ A_log, const void* __restrict__ dt_bias, const int* __restrict__ src,
                                       long long rows, int H, float mul, float* __restrict__ beta, float* __restrict__ g) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * H) return;
  const long long r = i / H;
  const int h = (int)(i - r * H);
  const long long t = src == nullptr ? r : src[r];
  float be = 0.f, ge = 0.f;
  if (t >= 0) {
    float s;
    be = mul * sigmoid_fine(__bfloat162float(b[t * ldb + h]));
    if (a != nullptr) ge = -exp_rn(param<BF16>(A_log, h)) * softplus_fine(__bfloat162float(a[t * lda + h]) + param<BF16>(dt_bias, h), s);
  }
  beta[i] = be;
  if (a != nullptr) g[i] = ge;
}

// db, da at their packed rows; part [blocks][2][H]: sums of dg g (for A_log) and of da (for dt_bias)
constexpr int DG_THREADS = 256, DG_MAXH = 128;
template <bool BF16>
__global__ void __launch_bounds__(DG_THREADS) delta_gates_bwd_kernel(
    const __nv_bfloat16* __restrict__ b, long long ldb, const __nv_bfloat16* __restrict__ a, long long lda, const void* __restrict__ A_log,
    const void* __restrict__ dt_bias, const int* __restrict__ src, long long rows, int H, float mul, const float* __restrict__ dbeta,
    const float* __restrict__ dg, __nv_bfloat16* __restrict__ db, long long lddb, __nv_bfloat16* __restrict__ da, long long ldda,
    float* __restrict__ part) {
  __shared__ float red[2][DG_THREADS];
  const int per = DG_THREADS / H;  // rows of the block at a time
  const int h = threadIdx.x % H, slot = threadIdx.x / H;
  float sA = 0.f, sdt = 0.f;
  if (slot < per) {
    const float nA = a == nullptr ? 0.f : -exp_rn(param<BF16>(A_log, h)), dt = a == nullptr ? 0.f : param<BF16>(dt_bias, h);
    for (long long r = (long long)blockIdx.x * per + slot; r < rows; r += (long long)gridDim.x * per) {
      const long long t = src == nullptr ? r : src[r];
      if (t < 0) continue;
      const float s = sigmoid_fine(__bfloat162float(b[t * ldb + h]));
      db[t * lddb + h] = __float2bfloat16(dbeta[r * H + h] * mul * s * (1.f - s));
      if (a != nullptr) {
        const float x = __bfloat162float(a[t * lda + h]) + dt, d = dg[r * H + h];
        float sx;
        const float plus = softplus_fine(x, sx), v = d * nA * sx;
        da[t * ldda + h] = __float2bfloat16(v);
        sA = fmaf(d, nA * plus, sA);
        sdt += v;
      }
    }
  }
  if (a == nullptr) return;
  red[0][threadIdx.x] = sA;
  red[1][threadIdx.x] = sdt;
  __syncthreads();
  if (threadIdx.x < 2 * H) {
    const int which = threadIdx.x / H, hh = threadIdx.x % H;
    float v = 0.f;
    for (int k = 0; k < per; ++k) v += red[which][k * H + hh];
    part[(long long)blockIdx.x * 2 * H + threadIdx.x] = v;
  }
}
__global__ void delta_gates_sum_kernel(const float* __restrict__ part, int blocks, int H, float* __restrict__ dA, float* __restrict__ ddt, int accumulate) {
  const int i = blockIdx.x, lane = threadIdx.x;  // one warp per value
  float* to = i < H ? dA : ddt;
  if (to == nullptr) return;  // frozen
  float v = 0.f;
  for (int k = lane; k < blocks; k += 32) v += part[(long long)k * 2 * H + i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane != 0) return;
  to += i < H ? i : i - H;
  *to = accumulate ? *to + v : v;
}

// ---------------------------------------------------------------------------------------------------------------
// Mamba2 (fla/layers/mamba2.py:241-331): the elementwise work around the SSD core, H heads of P channels.
//   pre :  dt = softplus(dt_raw + dt_bias),  g = -exp(A_log) dt,  xv = x dt                 (x, dt_raw: strided views)
//   post:  out = (y + D x) silu(z)                                                           (z: strided view)
// A thread owns 8 channels of one token; the P / 8 threads of a head reduce over the head with shuffles.  x, y, xv, dt, g and their
// gradients may be in the padded rows of the chunk layout: src[row] is the token of a padded row (-1: padding), null the row itself;
// dt_raw, z, out and theirs are always per token.  The padding's dt, g, dy and dx are zero.  All four are bound by
// memory; what the mapping saves is the passes that moved x, B, C and y between the two orders around them (layer at 32,761 tokens,
// 32 heads of 64, forward and backward: 3.90 -> 3.76 ms).
__device__ __forceinline__ float softplusf_(float x) { return x > 20.f ? x : log1pf(__expf(x)); }

template <int LANES>  // LANES = P / 8 threads per head: 8, 16 or 32
__global__ void mamba2_pre_fwd_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const __nv_bfloat16* __restrict__ dt_raw,
                                      long long ld_dt, const float* __restrict__ dt_bias, const float* __restrict__ A_log,
                                      __nv_bfloat16* __restrict__ xv, float* __restrict__ dt_out, float* __restrict__ g_out,
                                      const int* __restrict__ src, long long T, int H) {
  const int vecs = H * LANES;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long t = gid / vecs;
  if (t >= T) return;
  const int v = (int)(gid - t * vecs);
  const int h = v / LANES;
  const long long tok = src == nullptr ? t : src[t];
  const float dt = tok < 0 ? 0.f : softplusf_(__bfloat162float(dt_raw[tok * ld_dt + h]) + dt_bias[h]);
  float a[8];
  unpack8(*reinterpret_cast<const uint4*>(x + t * ldx + v * 8), a);
#pragma unroll
  for (int c = 0; c < 8; ++c) a[c] *= dt;
  *reinterpret_cast<uint4*>(xv + (t * vecs + v) * 8) = pack8(a);
  if (v % LANES == 0) {
    dt_out[t * H + h] = dt;
    g_out[t * H + h] = -__expf(A_log[h]) * dt;
  }
}

// dx = dxv dt + add;  d_raw = (sum_p dxv x + dg A + ddt) sigmoid(dt_raw + bias)   (ddt: gradient reaching dt directly, add: what x's
// other reader, the D skip, sends back in rows of H * P; both may be null).  dx may be a block of a wider matrix.  At 32,761 tokens and
// 32 heads of 64 the addition takes the kernel from 93 to 119 us; torch's sum (59 us) and the pass that put the gradients of x, B and C
// side by side (47 us) go: layer forward and backward 3.86 -> 3.78 ms.
template <int LANES>
__global__ void mamba2_pre_bwd_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const __nv_bfloat16* __restrict__ dt_raw,
                                      long long ld_dt, const float* __restrict__ dt_bias, const float* __restrict__ A_log,
                                      const __nv_bfloat16* __restrict__ dxv, const float* __restrict__ dg,
                                      const float* __restrict__ ddt, const __nv_bfloat16* __restrict__ add,
                                      __nv_bfloat16* __restrict__ dx, long long lddx, float* __restrict__ d_raw,
                                      const int* __restrict__ src, long long T, int H) {
  const int vecs = H * LANES;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long t = gid / vecs;
  const long long tok = t >= T ? -1 : src == nullptr ? t : src[t];
  const bool live = tok >= 0;
  const int v = t < T ? (int)(gid - t * vecs) : 0;
  const int h = v / LANES;
  float part = 0.f, pre = 0.f;
  if (t < T && !live) {
    *reinterpret_cast<uint4*>(dx + t * lddx + v * 8) = make_uint4(0, 0, 0, 0);
  } else if (live) {
    pre = __bfloat162float(dt_raw[tok * ld_dt + h]) + dt_bias[h];
    const float dt = softplusf_(pre);
    float a[8], g[8], o[8];
    const uint4 more = add == nullptr ? make_uint4(0, 0, 0, 0) : *reinterpret_cast<const uint4*>(add + (t * vecs + v) * 8);
    unpack8(*reinterpret_cast<const uint4*>(x + t * ldx + v * 8), a);
    unpack8(*reinterpret_cast<const uint4*>(dxv + (t * vecs + v) * 8), g);
    unpack8(more, o);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      part = fmaf(g[c], a[c], part);
      o[c] = fmaf(g[c], dt, o[c]);
    }
    *reinterpret_cast<uint4*>(dx + t * lddx + v * 8) = pack8(o);
  }
  // blockDim is a multiple of 32 and LANES divides 32, so a head's threads sit in one warp; dead threads add zero
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (live && v % LANES == 0) {
    float total = part + dg[t * H + h] * (-__expf(A_log[h]));
    if (ddt != nullptr) total += ddt[t * H + h];
    d_raw[tok * H + h] = total * sigmoidf_(pre);
  }
}

template <int LANES>
__global__ void mamba2_post_fwd_kernel(const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ x, long long ldx,
                                       const __nv_bfloat16* __restrict__ z, long long ldz, const float* __restrict__ D,
                                       __nv_bfloat16* __restrict__ out, const int* __restrict__ src, long long T, int H) {
  const int vecs = H * LANES;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long t = gid / vecs;
  const long long tok = t >= T ? -1 : src == nullptr ? t : src[t];
  if (tok < 0) return;
  const int v = (int)(gid - t * vecs);
  const float d = D[v / LANES];
  float a[8], b[8], g[8], o[8];
  unpack8(*reinterpret_cast<const uint4*>(y + (t * vecs + v) * 8), a);
  unpack8(*reinterpret_cast<const uint4*>(x + t * ldx + v * 8), b);
  unpack8(*reinterpret_cast<const uint4*>(z + tok * ldz + v * 8), g);
#pragma unroll
  for (int c = 0; c < 8; ++c) o[c] = fmaf(d, b[c], a[c]) * g[c] * sigmoidf_(g[c]);
  *reinterpret_cast<uint4*>(out + (tok * vecs + v) * 8) = pack8(o);
}

// du = dout silu(z): dy = du, dx = du D, dz = dout (y + D x) silu'(z), dD_part[t, h] = sum_p du x
template <int LANES>
__global__ void mamba2_post_bwd_kernel(const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ x, long long ldx,
                                       const __nv_bfloat16* __restrict__ z, long long ldz, const float* __restrict__ D,
                                       const __nv_bfloat16* __restrict__ dout, __nv_bfloat16* __restrict__ dy,
                                       __nv_bfloat16* __restrict__ dx, __nv_bfloat16* __restrict__ dz, long long lddz,
                                       float* __restrict__ dD_part, const int* __restrict__ src, long long T, int H) {
  const int vecs = H * LANES;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long t = gid / vecs;
  const bool live = t < T;
  const long long tok = !live ? -1 : src == nullptr ? t : src[t];
  const int v = live ? (int)(gid - t * vecs) : 0;
  const int h = v / LANES;
  float part = 0.f;
  if (live && tok < 0) {
    *reinterpret_cast<uint4*>(dy + (t * vecs + v) * 8) = make_uint4(0, 0, 0, 0);
    *reinterpret_cast<uint4*>(dx + (t * vecs + v) * 8) = make_uint4(0, 0, 0, 0);
  } else if (live) {
    const float d = D[h];
    float a[8], b[8], g[8], go[8], oy[8], ox[8], oz[8];
    const long long off = (t * vecs + v) * 8;
    unpack8(*reinterpret_cast<const uint4*>(y + off), a);
    unpack8(*reinterpret_cast<const uint4*>(x + t * ldx + v * 8), b);
    unpack8(*reinterpret_cast<const uint4*>(z + tok * ldz + v * 8), g);
    unpack8(*reinterpret_cast<const uint4*>(dout + (tok * vecs + v) * 8), go);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float sg = sigmoidf_(g[c]);
      const float du = go[c] * g[c] * sg;
      oy[c] = du;
      ox[c] = du * d;
      oz[c] = go[c] * fmaf(d, b[c], a[c]) * sg * (1.f + g[c] * (1.f - sg));
      part = fmaf(du, b[c], part);
    }
    *reinterpret_cast<uint4*>(dy + off) = pack8(oy);
    *reinterpret_cast<uint4*>(dx + off) = pack8(ox);
    *reinterpret_cast<uint4*>(dz + tok * lddz + v * 8) = pack8(oz);
  }
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if (live && v % LANES == 0) dD_part[t * H + h] = part;
}

}  // namespace

extern "C" {

int fb_delta_gates_blocks(long long rows, int H) {
  const long long per = DG_THREADS / H, n = (rows + per * 8 - 1) / (per * 8);
  return (int)(n < 1 ? 1 : n > 592 ? 592 : n);
}
// a, g null: beta alone.  bf16: A_log and dt_bias are bf16, else fp32.  H up to DG_MAXH.
int fb_delta_gates_fwd(const void* b, long long ldb, const void* a, long long lda, const void* A_log, const void* dt_bias, int bf16, const int* src,
                       long long rows, int H, float mul, float* beta, float* g, cudaStream_t stream) {
  if (rows == 0) return 0;
  if (H < 1 || H > DG_MAXH) return -2;
  const unsigned grid = (unsigned)((rows * H + 255) / 256);
  const auto kernel = bf16 ? delta_gates_fwd_kernel<true> : delta_gates_fwd_kernel<false>;
  kernel<<<grid, 256, 0, stream>>>((const __nv_bfloat16*)b, ldb, (const __nv_bfloat16*)a, lda, A_log, dt_bias, src, rows, H, mul, beta, g);
  return fb::launch_ok("delta_gates_fwd_kernel");
}
// part: fp32 [fb_delta_gates_blocks(rows, H), 2, H] scratch; dA, ddt: fp32 [H] (either may be null), added to with `accumulate`
int fb_delta_gates_bwd(const void* b, long long ldb, const void* a, long long lda, const void* A_log, const void* dt_bias, int bf16, const int* src,
                       long long rows, int H, float mul, const float* dbeta, const float* dg, void* db, long long lddb, void* da, long long ldda,
                       float* part, float* dA, float* ddt, int accumulate, cudaStream_t stream) {
  if (rows == 0) return 0;
  if (H < 1 || H > DG_MAXH) return -2;
  const int blocks = fb_delta_gates_blocks(rows, H);
  const auto kernel = bf16 ? delta_gates_bwd_kernel<true> : delta_gates_bwd_kernel<false>;
  kernel<<<blocks, DG_THREADS, 0, stream>>>((const __nv_bfloat16*)b, ldb, (const __nv_bfloat16*)a, lda, A_log, dt_bias, src, rows, H, mul, dbeta, dg,
                                            (__nv_bfloat16*)db, lddb, (__nv_bfloat16*)da, ldda, part);
  int rc = fb::launch_ok("delta_gates_bwd_kernel");
  if (rc || a == nullptr) return rc;
  delta_gates_sum_kernel<<<2 * H, 32, 0, stream>>>(part, blocks, H, dA, ddt, accumulate);
  return fb::launch_ok("delta_gates_sum_kernel");
}


// x: bf16 [T, H * P] view with row stride ldx (elements); dt_raw: bf16 [T, H] view with row stride ld_dt; dt_bias, A_log: fp32 [H]
// xv: bf16 [T, H, P]; dt, g: fp32 [T, H].  P in {64, 128, 256}; ldx a multiple of 8, x 16-byte aligned.
int fb_mamba2_pre_fwd(const void* x, long long ldx, const void* dt_raw, long long ld_dt, const float* dt_bias, const float* A_log,
                      void* xv, float* dt, float* g, const int* src, long long T, int H, int P, cudaStream_t stream) {
  if (T <= 0) return 0;
  if ((P != 64 && P != 128 && P != 256) || (ldx % 8) || ((uintptr_t)x & 15)) return -2;
  const long long threads = T * H * (P / 8);
  const unsigned blocks = (unsigned)((threads + 255) / 256);
#define FB_PRE_FWD(L) mamba2_pre_fwd_kernel<L><<<blocks, 256, 0, stream>>>((const __nv_bfloat16*)x, ldx, (const __nv_bfloat16*)dt_raw, \
      ld_dt, dt_bias, A_log, (__nv_bfloat16*)xv, dt, g, src, T, H)
  if (P == 64) FB_PRE_FWD(8); else if (P == 128) FB_PRE_FWD(16); else FB_PRE_FWD(32);
#undef FB_PRE_FWD
  return fb::launch_ok("mamba2_pre_fwd_kernel");
}

// dxv: bf16 [T, H, P]; dg: fp32 [T, H]; ddt: fp32 [T, H] or null; add: bf16 [T, H * P] or null; dx: bf16 [T, H * P] with row stride lddx;
// d_raw: fp32 [T, H]
int fb_mamba2_pre_bwd(const void* x, long long ldx, const void* dt_raw, long long ld_dt, const float* dt_bias, const float* A_log,
                      const void* dxv, const float* dg, const float* ddt, const void* add, void* dx, long long lddx, float* d_raw,
                      const int* src, long long T, int H, int P, cudaStream_t stream) {
  if (T <= 0) return 0;
  if ((P != 64 && P != 128 && P != 256) || (ldx % 8) || (lddx % 8) || ((uintptr_t)x & 15) || ((uintptr_t)dx & 15) || ((uintptr_t)add & 15)) return -2;
  const long long threads = T * H * (P / 8);
  const unsigned blocks = (unsigned)((threads + 255) / 256);
#define FB_PRE_BWD(L) mamba2_pre_bwd_kernel<L><<<blocks, 256, 0, stream>>>((const __nv_bfloat16*)x, ldx, (const __nv_bfloat16*)dt_raw, \
      ld_dt, dt_bias, A_log, (const __nv_bfloat16*)dxv, dg, ddt, (const __nv_bfloat16*)add, (__nv_bfloat16*)dx, lddx, d_raw, src, T, H)
  if (P == 64) FB_PRE_BWD(8); else if (P == 128) FB_PRE_BWD(16); else FB_PRE_BWD(32);
#undef FB_PRE_BWD
  return fb::launch_ok("mamba2_pre_bwd_kernel");
}

// y: bf16 [T, H, P]; x, z: bf16 views with row strides ldx / ldz; D: fp32 [H]; out: bf16 [T, H * P]
int fb_mamba2_post_fwd(const void* y, const void* x, long long ldx, const void* z, long long ldz, const float* D, void* out,
                       const int* src, long long T, int H, int P, cudaStream_t stream) {
  if (T <= 0) return 0;
  if ((P != 64 && P != 128 && P != 256) || (ldx % 8) || (ldz % 8) || ((uintptr_t)x & 15) || ((uintptr_t)z & 15)) return -2;
  const long long threads = T * H * (P / 8);
  const unsigned blocks = (unsigned)((threads + 255) / 256);
#define FB_POST_FWD(L) mamba2_post_fwd_kernel<L><<<blocks, 256, 0, stream>>>((const __nv_bfloat16*)y, (const __nv_bfloat16*)x, ldx, \
      (const __nv_bfloat16*)z, ldz, D, (__nv_bfloat16*)out, src, T, H)
  if (P == 64) FB_POST_FWD(8); else if (P == 128) FB_POST_FWD(16); else FB_POST_FWD(32);
#undef FB_POST_FWD
  return fb::launch_ok("mamba2_post_fwd_kernel");
}

// dout: bf16 [T, H * P]; dy, dx: bf16 [T, H * P]; dz the same with row stride lddz; dD_part: fp32 [T, H] (summed over T by the caller)
int fb_mamba2_post_bwd(const void* y, const void* x, long long ldx, const void* z, long long ldz, const float* D, const void* dout,
                       void* dy, void* dx, void* dz, long long lddz, float* dD_part, const int* src, long long T, int H, int P, cudaStream_t stream) {
  if (T <= 0) return 0;
  if ((P != 64 && P != 128 && P != 256) || (ldx % 8) || (ldz % 8) || (lddz % 8) || ((uintptr_t)dz & 15) || ((uintptr_t)x & 15) || ((uintptr_t)z & 15)) return -2;
  const long long threads = T * H * (P / 8);
  const unsigned blocks = (unsigned)((threads + 255) / 256);
#define FB_POST_BWD(L) mamba2_post_bwd_kernel<L><<<blocks, 256, 0, stream>>>((const __nv_bfloat16*)y, (const __nv_bfloat16*)x, ldx, \
      (const __nv_bfloat16*)z, ldz, D, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dy, (__nv_bfloat16*)dx, (__nv_bfloat16*)dz, \
      lddz, dD_part, src, T, H)
  if (P == 64) FB_POST_BWD(8); else if (P == 128) FB_POST_BWD(16); else FB_POST_BWD(32);
#undef FB_POST_BWD
  return fb::launch_ok("mamba2_post_bwd_kernel");
}

// x, dx: bf16, rows ldx / lddx elements apart; g, s (optional), dg, ds (with s): fp32, rows side by side; rows: of g (forward) or of x
// (backward), cols of each; map: see the kernels.  cols, ldx and lddx multiples of 8, all 16-byte aligned.
int fb_logsigmoid_gate_fwd(const void* x, long long ldx, const int* map, float* g, float* s, float normalizer, long long rows, long long cols,
                           cudaStream_t stream) {
  if (rows == 0 || cols == 0) return 0;
  if ((cols & 7) || (ldx & 7) || !fb::aligned(16, x, g, s)) return -2;
  const long long vecs = cols / 8, total = rows * vecs;
  const auto kernel = s != nullptr ? logsigmoid_gate_fwd_kernel<true> : logsigmoid_gate_fwd_kernel<false>;
  kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>((const __nv_bfloat16*)x, ldx, map, g, s, normalizer, total, vecs);
  return fb::launch_ok("logsigmoid_gate_fwd_kernel");
}

int fb_logsigmoid_gate_bwd(const void* x, long long ldx, const int* map, const float* dg, const float* ds, void* dx, long long lddx, float normalizer,
                           long long rows, long long cols, cudaStream_t stream) {
  if (rows == 0 || cols == 0) return 0;
  if ((cols & 7) || (ldx & 7) || (lddx & 7) || !fb::aligned(16, x, dg, ds, dx)) return -2;
  const long long vecs = cols / 8, total = rows * vecs;
  const auto kernel = ds != nullptr ? logsigmoid_gate_bwd_kernel<true> : logsigmoid_gate_bwd_kernel<false>;
  kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>((const __nv_bfloat16*)x, ldx, map, dg, ds, (__nv_bfloat16*)dx, lddx, normalizer, total, vecs);
  return fb::launch_ok("logsigmoid_gate_bwd_kernel");
}

int fb_hgrn2_gate_tiles(long long rows) { return (int)((rows + GATE_TILE_ROWS - 1) / GATE_TILE_ROWS); }

// q_raw, f_raw, q, k: bf16 [rows, D]; g: fp32 [rows, D]; lb: fp32 [D] or null.  D a multiple of 8.
int fb_hgrn2_gate_fwd(const void* q_raw, const void* f_raw, const float* lb, void* q, void* k, float* g, long long rows, int D,
                      cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (D % 8) return -2;
  const long long threads = rows * (D / 8);
  const unsigned blocks = (unsigned)((threads + 255) / 256);
  if (lb)
    hgrn2_gate_fwd_kernel<true><<<blocks, 256, 0, stream>>>((const __nv_bfloat16*)q_raw, (const __nv_bfloat16*)f_raw, lb,
                                                            (__nv_bfloat16*)q, (__nv_bfloat16*)k, g, rows, D);
  else
    hgrn2_gate_fwd_kernel<false><<<blocks, 256, 0, stream>>>((const __nv_bfloat16*)q_raw, (const __nv_bfloat16*)f_raw, lb,
                                                             (__nv_bfloat16*)q, (__nv_bfloat16*)k, g, rows, D);
  return fb::launch_ok("hgrn2_gate_fwd_kernel");
}

// dlb_part: fp32 [fb_hgrn2_gate_tiles(rows), D] scratch and dlb: fp32 [D], both only read / written when lb is given
int fb_hgrn2_gate_bwd(const void* q_raw, const void* f_raw, const float* lb, const void* dq, const void* dk, const float* dg,
                      void* dq_raw, void* df_raw, float* dlb_part, float* dlb, long long rows, int D, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (D % 8) return -2;
  const int tiles = fb_hgrn2_gate_tiles(rows);
  dim3 grid((D + 255) / 256, tiles);
  if (lb) {
    hgrn2_gate_bwd_kernel<true><<<grid, 256, 0, stream>>>(
        (const __nv_bfloat16*)q_raw, (const __nv_bfloat16*)f_raw, lb, (const __nv_bfloat16*)dq, (const __nv_bfloat16*)dk, dg,
        (__nv_bfloat16*)dq_raw, (__nv_bfloat16*)df_raw, dlb_part, rows, D);
    int rc = fb::launch_ok("hgrn2_gate_bwd_kernel");
    if (rc) return rc;
    colsum_rows_kernel<<<(D + 31) / 32, 256, 0, stream>>>(dlb_part, tiles, D, dlb);
    return fb::launch_ok("colsum_rows_kernel");
  }
  hgrn2_gate_bwd_kernel<false><<<grid, 256, 0, stream>>>(
      (const __nv_bfloat16*)q_raw, (const __nv_bfloat16*)f_raw, lb, (const __nv_bfloat16*)dq, (const __nv_bfloat16*)dk, dg,
      (__nv_bfloat16*)dq_raw, (__nv_bfloat16*)df_raw, dlb_part, rows, D);
  return fb::launch_ok("hgrn2_gate_bwd_kernel");
}

}  // extern "C"
