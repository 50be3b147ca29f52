// Small CUDA-core kernels of the chunk-parallel token mixers (everything GEMM-shaped runs on bgemm.cu).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

#include "fine_math.cuh"
#include "host_utils.cuh"

namespace {

__device__ __forceinline__ void unpack8f(const uint4& q, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x, f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8f(const float (&f)[8]) {
  uint4 q;
#pragma unroll
  for (int i = 0; i < 4; ++i) reinterpret_cast<__nv_bfloat162*>(&q)[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return q;
}

// T = (I + diag(beta) P)^-1 of the strictly lower-triangular score blocks P (the WY "solve" of the delta rule; the reference
// does it by blockwise forward substitution in fla/ops/utils/solve_tril.py).  One 64-thread block per 64 x 64 diagonal block:
// thread c solves (I + A) x = e_c by forward substitution, 16 rows at a time: what the rows before contribute is sixteen sums
// side by side, A in 16-byte broadcasts from shared memory, then the 16 x 16 corner in registers.  Warp 1 skips the zeros that
// its columns have above row 32, and T is written in 16-byte vectors over the rows of A that are done with (more shared memory
// than the 16 KB of A costs resident blocks: with T beside it the gated form took 72 us instead of 32).  Written out over all 64
// rows it was one chain of 2,016 multiply-adds and as many reads: 150 us at 65,536 tokens, 8 heads of 128, where the bytes take
// 41; this takes 89, in the same order of operations.
// P: [n, C, C] fp32, C = 64 or 128; T: [n, C, C] bf16.
//   C = 64:  also Tu = T diag(beta) and (b given) Tw = T diag(beta e^b), the matrices the values and keys are multiplied with,
//            which used to be passes of their own over T
//   C = 128: the two diagonal blocks of T, zeros above them, and A21 = the scaled lower-left block in bf16, from which two
//            products make T's lower-left block
// beta, b: element (chunk, head, i) at ((chunk * C + i) * H + head).
__global__ void __launch_bounds__(64) delta_inverse_kernel(const float* __restrict__ P, const float* __restrict__ beta, const float* __restrict__ b,
                                                           int C, int H, __nv_bfloat16* __restrict__ T, __nv_bfloat16* __restrict__ Tu,
                                                           __nv_bfloat16* __restrict__ Tw, __nv_bfloat16* __restrict__ A21) {
  __shared__ alignas(16) float sA[64 * 64];  // from the top down, the rows of A that are done with make room for those of T
  __shared__ float sbeta[64], sw[64];
  const int halves = C >> 6;
  const long long m = blockIdx.x / halves;
  const int half = (int)(blockIdx.x - m * halves), ch = (int)(m / H), h = (int)(m - (long long)ch * H);
  const float* a = P + m * C * C + (long long)half * 64 * (C + 1);
  const int c = threadIdx.x;
  const long long at = ((long long)ch * C + half * 64 + c) * H + h;
  sbeta[c] = beta[at];
  if (Tw != nullptr) sw[c] = sbeta[c] * __expf(b[at]);
  __syncthreads();
#pragma unroll 4
  for (int i = c; i < 4096 / 4; i += 64) {
    const int r = i >> 4;
    float4 v = __ldcs(reinterpret_cast<const float4*>(a + (long long)r * C + (i & 15) * 4));
    const float f = sbeta[r];
    v.x *= f, v.y *= f, v.z *= f, v.w *= f;
    reinterpret_cast<float4*>(sA)[i] = v;
  }
  __syncthreads();
  const int first = c & 32;  // T is lower triangular: the second warp's columns are zero above row 32
#pragma unroll 1
  for (int I = 0; I < 64; I += 16) {
    float s[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) s[i] = I + i == c ? 1.f : 0.f;
    const float4* row = reinterpret_cast<const float4*>(sA + I * 64);
    if (I >= first) {
#pragma unroll 1
      for (int j = first; j < I; j += 4) {
        float x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = sA[(j + k) * 64 + c];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float4 v = row[i * 16 + j / 4];
          s[i] = fmaf(-v.x, x[0], s[i]);
          s[i] = fmaf(-v.y, x[1], s[i]);
          s[i] = fmaf(-v.z, x[2], s[i]);
          s[i] = fmaf(-v.w, x[3], s[i]);
        }
      }
#pragma unroll
      for (int i = 1; i < 16; ++i)
#pragma unroll
        for (int j = 0; j < i; j += 4) {
          const float4 v = row[i * 16 + (I + j) / 4];
          s[i] = fmaf(-v.x, s[j], s[i]);
          if (j + 1 < i) s[i] = fmaf(-v.y, s[j + 1], s[i]);
          if (j + 2 < i) s[i] = fmaf(-v.z, s[j + 2], s[i]);
          if (j + 3 < i) s[i] = fmaf(-v.w, s[j + 3], s[i]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 16; ++i) sA[(I + i) * 64 + c] = s[i];
  }
  __syncthreads();
  // out in vectors of eight columns
  __nv_bfloat16* o = T + m * C * C + (long long)half * 64 * (C + 1);
  const int v8 = (c & 7) * 8;
#pragma unroll 2
  for (int r = c >> 3; r < 64; r += 8) {
    float x[8], y[8];
#pragma unroll
    for (int k = 0; k < 8; k += 4) *reinterpret_cast<float4*>(x + k) = *reinterpret_cast<const float4*>(sA + r * 64 + v8 + k);
    *reinterpret_cast<uint4*>(o + (long long)r * C + v8) = pack8f(x);
    if (Tu != nullptr) {
#pragma unroll
      for (int k = 0; k < 8; ++k) y[k] = x[k] * sbeta[v8 + k];
      *reinterpret_cast<uint4*>(Tu + m * 4096 + r * 64 + v8) = pack8f(y);
      if (Tw != nullptr) {
#pragma unroll
        for (int k = 0; k < 8; ++k) y[k] = x[k] * sw[v8 + k];
        *reinterpret_cast<uint4*>(Tw + m * 4096 + r * 64 + v8) = pack8f(y);
      }
    }
  }
  if (C == 128) {
    if (half == 0) {
      __nv_bfloat16* z = T + m * C * C + 64 + v8;
#pragma unroll
      for (int r = c >> 3; r < 64; r += 8) *reinterpret_cast<uint4*>(z + (long long)r * C) = make_uint4(0, 0, 0, 0);
    } else {
      const float* a21 = P + m * C * C + 64ll * C + v8;
#pragma unroll 4
      for (int r = c >> 3; r < 64; r += 8) {
        float x[8];
#pragma unroll
        for (int k = 0; k < 8; k += 4) *reinterpret_cast<float4*>(x + k) = __ldcs(reinterpret_cast<const float4*>(a21 + (long long)r * C + k));
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] *= sbeta[r];
        *reinterpret_cast<uint4*>(A21 + m * 4096 + r * 64 + v8) = pack8f(x);
      }
    }
  }
}

// Tu = T diag(beta), Tw = T diag(beta e^b) (C = 128, where T's corner comes from a product).  One block per matrix.
__global__ void __launch_bounds__(256) delta_scale_kernel(const __nv_bfloat16* __restrict__ T, const float* __restrict__ beta, const float* __restrict__ b,
                                                          int C, int H, __nv_bfloat16* __restrict__ Tu, __nv_bfloat16* __restrict__ Tw) {
  __shared__ float fu[128], fw[128];
  const long long m = blockIdx.x;
  const int ch = (int)(m / H), h = (int)(m - (long long)ch * H);
  for (int i = threadIdx.x; i < C; i += 256) {
    const long long o = ((long long)ch * C + i) * H + h;
    fu[i] = beta[o];
    fw[i] = b != nullptr ? beta[o] * __expf(b[o]) : 0.f;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < C * C / 8; i += 256) {
    const int j0 = (i * 8) & (C - 1);
    const uint4 q = reinterpret_cast<const uint4*>(T + m * C * C)[i];
    const __nv_bfloat162* t2 = reinterpret_cast<const __nv_bfloat162*>(&q);
    uint4 qu, qw;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 t = __bfloat1622float2(t2[e]);
      reinterpret_cast<__nv_bfloat162*>(&qu)[e] = __floats2bfloat162_rn(t.x * fu[j0 + 2 * e], t.y * fu[j0 + 2 * e + 1]);
      reinterpret_cast<__nv_bfloat162*>(&qw)[e] = __floats2bfloat162_rn(t.x * fw[j0 + 2 * e], t.y * fw[j0 + 2 * e + 1]);
    }
    reinterpret_cast<uint4*>(Tu + m * C * C)[i] = qu;
    if (Tw != nullptr) reinterpret_cast<uint4*>(Tw + m * C * C)[i] = qw;
  }
}

// Backward of Tu and Tw: dT = dTu diag(beta) + dTw diag(beta e^b) (bf16), and over the rows
//   dbeta_j = scale sum_i T_ij (dTu_ij + e^{b_j} dTw_ij),   db_j = scale sum_i beta_j e^{b_j} T_ij dTw_ij      (written, not added).
// dTw and b null: one matrix served both products.  One block of 256 threads per (chunk, head); a thread keeps eight
// columns' sums over its rows in registers, so a row costs no atomics.  A thread has two (C = 64) or eight rows: their loads go
// out two rows at a time, the first before the factors are fetched, and T above its diagonal is not read.  One row after the
// other it waited for memory four times per block: 70 us at 65,536 tokens, 8 heads of 128 (the bytes take 26); this takes 40.
template <int C, bool W>
__global__ void __launch_bounds__(256) delta_bwd_t_kernel(const __nv_bfloat16* __restrict__ T, const __nv_bfloat16* __restrict__ dTu,
                                                          const __nv_bfloat16* __restrict__ dTw, const float* __restrict__ beta,
                                                          const float* __restrict__ b, int H, float scale, __nv_bfloat16* __restrict__ dT,
                                                          float* __restrict__ dbeta, float* __restrict__ db) {
  constexpr int nv = C / 8, groups = 256 / nv;  // 32 or 16 groups of rows
  __shared__ float su[8][C + 4], sw[8][C + 4];
  const long long m = blockIdx.x;
  const int ch = (int)(m / H), h = (int)(m - (long long)ch * H);
  const int v = threadIdx.x % nv, r0 = threadIdx.x / nv;
  uint4 rt[2], ru[2], rw[2];
  auto load = [&](int i0) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = i0 + u * groups;
      const long long o = (m * C * C + (long long)i * C) / 8 + v;
      rt[u] = v * 8 <= i ? __ldcs(reinterpret_cast<const uint4*>(T) + o) : make_uint4(0, 0, 0, 0);  // T is lower triangular
      ru[u] = __ldcs(reinterpret_cast<const uint4*>(dTu) + o);
      if constexpr (W) rw[u] = __ldcs(reinterpret_cast<const uint4*>(dTw) + o);
    }
  };
  load(r0);
  float fu[8], fe[8], au[8], aw[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const long long o = ((long long)ch * C + v * 8 + e) * H + h;
    fu[e] = beta[o];
    if constexpr (W) fe[e] = __expf(b[o]);
    au[e] = aw[e] = 0.f;
  }
#pragma unroll 1
  for (int i0 = r0; i0 < C; i0 += 2 * groups) {
    if (i0 != r0) load(i0);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float t[8], gu[8], gw[8];
      unpack8f(rt[u], t);
      unpack8f(ru[u], gu);
      if constexpr (W) unpack8f(rw[u], gw);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float w = W ? gw[e] * fe[e] : 0.f;
        au[e] = fmaf(t[e], gu[e] + w, au[e]);
        if constexpr (W) aw[e] = fmaf(t[e], w, aw[e]);
        gu[e] = fu[e] * (gu[e] + w);
      }
      reinterpret_cast<uint4*>(dT)[(m * C * C + (long long)(i0 + u * groups) * C) / 8 + v] = pack8f(gu);
    }
  }
  // lanes of a warp hold the same columns for 32 / nv groups: add those by shuffle, the warps through shared memory
#pragma unroll
  for (int e = 0; e < 8; ++e)
    for (int o = nv; o < 32; o <<= 1) {
      au[e] += __shfl_xor_sync(0xffffffffu, au[e], o);
      if constexpr (W) aw[e] += __shfl_xor_sync(0xffffffffu, aw[e], o);
    }
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) < nv) {
#pragma unroll
    for (int e = 0; e < 8; ++e) su[warp][v * 8 + e] = au[e], sw[warp][v * 8 + e] = aw[e];
  }
  __syncthreads();
  for (int j = threadIdx.x; j < C; j += 256) {
    float x = 0.f, y = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) x += su[w][j], y += sw[w][j];
    const long long o = ((long long)ch * C + j) * H + h;
    dbeta[o] = scale * x;
    if (db != nullptr) db[o] = scale * beta[o] * y;
  }
}

// Backward of the score blocks A = diag(beta) P (strict, P = k k^T decayed) and Q = tril(q k^T decayed):
//   g_ij  = beta_i dA_ij e^{b_i - b_j} [j < i],   gq_ij = q_scale dQ_ij e^{b_i - b_j} [j <= i]   (bf16 operands of the dq, dk products)
//   dbeta_i += scale sum_j dA_ij P_ij,   db_i += scale (row sum_i - column sum_i) of beta dA P + dQ Q
// dA, P fp32 (null: only the second block, for the scalar-gated attention without a delta rule); dQ, Q bf16 and b only with a
// decay (without one the products' epilogues already give gq).  A, B: which of the two there are; one kernel for all three cases
// held the registers of both (80 instead of 48), and with that two thirds of the warps.  Loads as in delta_bwd_t_kernel, and
// nothing above the diagonal is read.  Before and after: 185 and 76 us (Q alone, 512 chunks of 64, 32 heads; the bytes take 45),
// 85 and 54 us (A alone, 1,024 chunks of 64, 8 heads; 33), 69 and 46 us (both, 128 chunks of 128, 6 heads).
template <int C, bool A, bool B>
__global__ void __launch_bounds__(256) delta_bwd_scores_kernel(const float* __restrict__ dA, const float* __restrict__ P,
                                                               const __nv_bfloat16* __restrict__ dQ, const __nv_bfloat16* __restrict__ Q,
                                                               const float* __restrict__ beta, const float* __restrict__ b, int H, float scale,
                                                               float q_scale, __nv_bfloat16* __restrict__ g, __nv_bfloat16* __restrict__ gq,
                                                               float* __restrict__ dbeta, float* __restrict__ db) {
  constexpr int nv = C / 8, groups = 256 / nv;
  __shared__ float sb[C], sbeta[C], srow[C], scol[8][C + 4];
  const long long m = blockIdx.x;
  const int ch = (int)(m / H), h = (int)(m - (long long)ch * H);
  const int v = threadIdx.x % nv, r0 = threadIdx.x / nv;
  float4 da[2][2], pp[2][2];
  uint4 dq[2], qq[2];
  auto load = [&](int i0) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = i0 + u * groups;
      const long long row = m * C * C + (long long)i * C + v * 8;
      if (v * 8 > i) continue;
      if constexpr (A) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          da[u][k] = __ldcs(reinterpret_cast<const float4*>(dA + row + 4 * k));
          pp[u][k] = __ldcs(reinterpret_cast<const float4*>(P + row + 4 * k));
        }
      }
      if constexpr (B) {
        dq[u] = __ldcs(reinterpret_cast<const uint4*>(dQ + row));
        qq[u] = __ldcs(reinterpret_cast<const uint4*>(Q + row));
      }
    }
  };
  load(r0);
  float db_old = 0.f;  // read ahead: each is this block's own to add to
  if (threadIdx.x < C) {
    const long long at = ((long long)ch * C + threadIdx.x) * H + h;
    sb[threadIdx.x] = b != nullptr ? b[at] : 0.f;
    if constexpr (A) sbeta[threadIdx.x] = beta != nullptr ? beta[at] : 0.f;
    if (db != nullptr) db_old = db[at];
  }
  __syncthreads();
  float col[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) col[e] = 0.f;
#pragma unroll 1
  for (int i0 = r0; i0 < C; i0 += 2 * groups) {
    if (i0 != r0) load(i0);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = i0 + u * groups;
      const long long row = m * C * C + (long long)i * C + v * 8;
      float rs = 0.f, rd = 0.f;
      if (v * 8 > i) {  // nothing above the diagonal
        if constexpr (A) *reinterpret_cast<uint4*>(g + row) = make_uint4(0, 0, 0, 0);
        if constexpr (B) *reinterpret_cast<uint4*>(gq + row) = make_uint4(0, 0, 0, 0);
      } else {
        const float bi = sb[i], be = A ? sbeta[i] : 0.f;
        float gg[8];
        if constexpr (A) {
          const float *a = reinterpret_cast<const float*>(da[u]), *p = reinterpret_cast<const float*>(pp[u]);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int j = v * 8 + e;
            const float x = j < i ? a[e] : 0.f, y = j < i ? x * p[e] : 0.f;
            gg[e] = j < i ? x * be * (b != nullptr ? __expf(bi - sb[j]) : 1.f) : 0.f;
            rs += y;
            rd += be * y;
            col[e] += be * y;
          }
          *reinterpret_cast<uint4*>(g + row) = pack8f(gg);
        }
        if constexpr (B) {
          float x[8], q[8];
          unpack8f(dq[u], x);
          unpack8f(qq[u], q);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int j = v * 8 + e;
            const float y = j <= i ? x[e] * q[e] : 0.f;
            gg[e] = j <= i ? x[e] * __expf(bi - sb[j]) * q_scale : 0.f;
            rd += y;
            col[e] += y;
          }
          *reinterpret_cast<uint4*>(gq + row) = pack8f(gg);
        }
      }
#pragma unroll
      for (int o = nv >> 1; o > 0; o >>= 1) {
        if constexpr (A) rs += __shfl_xor_sync(0xffffffffu, rs, o);
        rd += __shfl_xor_sync(0xffffffffu, rd, o);
      }
      if (v == 0) {
        if (A && dbeta != nullptr) dbeta[((long long)ch * C + i) * H + h] += scale * rs;
        srow[i] = rd;
      }
    }
  }
  if (db == nullptr) return;
#pragma unroll
  for (int e = 0; e < 8; ++e)
    for (int o = nv; o < 32; o <<= 1) col[e] += __shfl_xor_sync(0xffffffffu, col[e], o);
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) < nv) {
#pragma unroll
    for (int e = 0; e < 8; ++e) scol[warp][v * 8 + e] = col[e];
  }
  __syncthreads();
  if (threadIdx.x < C) {
    const int j = threadIdx.x;
    float x = srow[j];
#pragma unroll
    for (int w = 0; w < 8; ++w) x -= scol[w][j];
    db[((long long)ch * C + j) * H + h] = db_old + scale * x;
  }
}

}  // namespace

extern "C" {

int fb_delta_inverse(const float* P, const float* beta, const float* b, int NC, int H, int C, void* T, void* Tu, void* Tw, void* A21,
                     cudaStream_t stream) {
  if (NC <= 0) return 0;
  if ((C != 64 && C != 128) || !fb::aligned(16, P, T, Tu, Tw, A21)) return -2;
  delta_inverse_kernel<<<(unsigned)(NC * H * (C / 64)), 64, 0, stream>>>(P, beta, b, C, H, (__nv_bfloat16*)T, (__nv_bfloat16*)(C == 64 ? Tu : nullptr),
                                                                         (__nv_bfloat16*)Tw, (__nv_bfloat16*)A21);
  return fb::launch_ok("delta_inverse_kernel");
}

int fb_delta_scale(const void* T, const float* beta, const float* b, int NC, int H, int C, void* Tu, void* Tw, cudaStream_t stream) {
  if (NC <= 0) return 0;
  if ((C != 64 && C != 128) || !fb::aligned(16, T, Tu, Tw)) return -2;
  delta_scale_kernel<<<(unsigned)(NC * H), 256, 0, stream>>>((const __nv_bfloat16*)T, beta, b, C, H, (__nv_bfloat16*)Tu, (__nv_bfloat16*)Tw);
  return fb::launch_ok("delta_scale_kernel");
}

int fb_delta_bwd_t(const void* T, const void* dTu, const void* dTw, const float* beta, const float* b, int NC, int H, int C, float scale, void* dT,
                   float* dbeta, float* db, cudaStream_t stream) {
  if (NC <= 0) return 0;
  if ((C != 64 && C != 128) || !fb::aligned(16, T, dTu, dTw, dT)) return -2;
  if ((dTw == nullptr) != (b == nullptr)) return -2;
  const auto kernel = C == 64 ? (b != nullptr ? delta_bwd_t_kernel<64, true> : delta_bwd_t_kernel<64, false>)
                              : (b != nullptr ? delta_bwd_t_kernel<128, true> : delta_bwd_t_kernel<128, false>);
  kernel<<<(unsigned)(NC * H), 256, 0, stream>>>((const __nv_bfloat16*)T, (const __nv_bfloat16*)dTu, (const __nv_bfloat16*)dTw, beta, b, H, scale,
                                                 (__nv_bfloat16*)dT, dbeta, db);
  return fb::launch_ok("delta_bwd_t_kernel");
}

int fb_delta_bwd_scores(const float* dA, const float* P, const void* dQ, const void* Q, const float* beta, const float* b, int NC, int H, int C,
                        float scale, float q_scale, void* g, void* gq, float* dbeta, float* db, cudaStream_t stream) {
  if (NC <= 0) return 0;
  if ((C != 64 && C != 128) || !fb::aligned(16, dA, P, dQ, Q, g, gq)) return -2;
  auto go = [&](auto kernel) {
    kernel<<<(unsigned)(NC * H), 256, 0, stream>>>(dA, P, (const __nv_bfloat16*)dQ, (const __nv_bfloat16*)Q, beta, b, H, scale, q_scale,
                                                   (__nv_bfloat16*)g, (__nv_bfloat16*)gq, dbeta, db);
  };
  if (dA == nullptr)
    go(C == 64 ? delta_bwd_scores_kernel<64, false, true> : delta_bwd_scores_kernel<128, false, true>);
  else if (dQ == nullptr)
    go(C == 64 ? delta_bwd_scores_kernel<64, true, false> : delta_bwd_scores_kernel<128, true, false>);
  else
    go(C == 64 ? delta_bwd_scores_kernel<64, true, true> : delta_bwd_scores_kernel<128, true, true>);
  return fb::launch_ok("delta_bwd_scores_kernel");
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------------------------
// Scalar-gated attention with queries and keys shared by groups of heads (Mamba2's SSD): what is elementwise around its
// products, on the value side.  v, do, ..: [NC, C, H, dv] bf16; g, b: [NC, C, H] fp32; one block per (chunk, head), a row of
// dv in dv / 8 lanes (a power of two up to 32), so that the row sums are shuffles.
namespace {

__device__ __forceinline__ void group_rows(int C, int H, int dv, int& ch, int& h, int& v, int& r0, int& groups) {
  ch = blockIdx.x / H, h = blockIdx.x - ch * H;
  const int nv = dv >> 3;
  v = threadIdx.x % nv, r0 = threadIdx.x / nv, groups = blockDim.x / nv;
}

// b = cumsum(g), eb = scale e^b (fp32, the factor of an output row), alpha = e^{b_last}, vhat = v e^{b_last - b}.  The rows of v
// are fetched before the sum of the gates, which is a chain: 67 -> 58 us at 32,768 tokens, 32 heads of 64 (the bytes take 41).
// (Two rows at a time made group_bwd2_kernel slower, 101 -> 117 us: three operands of two rows cost it warps.)
__global__ void __launch_bounds__(256) group_prep_fwd_kernel(const __nv_bfloat16* __restrict__ v, const float* __restrict__ g, int C, int H, int dv,
                                                             float scale, float* __restrict__ b, float* __restrict__ eb, float* __restrict__ alpha,
                                                             __nv_bfloat16* __restrict__ vhat) {
  __shared__ float sb[128];
  int ch, h, vv, r0, groups;
  group_rows(C, H, dv, ch, h, vv, r0, groups);
  uint4 raw[2];
  auto load = [&](int i0) {
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (i0 + u * groups < C) raw[u] = __ldcs(reinterpret_cast<const uint4*>(v + (((long long)ch * C + i0 + u * groups) * H + h) * dv + vv * 8));
  };
  load(r0);  // on their way while the gates are summed up
  if (threadIdx.x < 32) {  // warp 0: inclusive sum of up to 128 steps, four per lane
    const int lane = threadIdx.x, per = C >> 5;
    float loc[4], s = 0.f;
    for (int k = 0; k < per; ++k) {
      s += g[((long long)ch * C + lane * per + k) * H + h];
      loc[k] = s;
    }
    float pre = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float t = __shfl_up_sync(0xffffffffu, pre, o);
      if (lane >= o) pre += t;
    }
    pre -= s;
    for (int k = 0; k < per; ++k) sb[lane * per + k] = pre + loc[k];
  }
  __syncthreads();
  const float last = sb[C - 1];
  for (int i = threadIdx.x; i < C; i += blockDim.x) {
    const long long o = ((long long)ch * C + i) * H + h;
    b[o] = sb[i];
    eb[o] = scale * __expf(sb[i]);
  }
  if (threadIdx.x == 0) alpha[(long long)ch * H + h] = __expf(last);
  for (int i0 = r0; i0 < C; i0 += 2 * groups) {
    if (i0 != r0) load(i0);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = i0 + u * groups;
      if (i >= C) break;
      float x[8];
      unpack8f(raw[u], x);
      const float f = __expf(last - sb[i]);
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] *= f;
      *reinterpret_cast<uint4*>(vhat + (((long long)ch * C + i) * H + h) * dv + vv * 8) = pack8f(x);
    }
  }
}

// dos = do eb (the gradient of q S), db_i = sum do_i o1_i with o1 = eb (q S) (written, not added)
__global__ void __launch_bounds__(256) group_bwd1_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ o1,
                                                         const float* __restrict__ eb, int C, int H, int dv, __nv_bfloat16* __restrict__ dos,
                                                         float* __restrict__ db) {
  int ch, h, vv, r0, groups;
  group_rows(C, H, dv, ch, h, vv, r0, groups);
  const int nv = dv >> 3;
  for (int i = r0; i < C; i += groups) {
    const long long ob = ((long long)ch * C + i) * H + h, o = ob * dv + vv * 8;
    float x[8], y[8], s = 0.f;
    unpack8f(*reinterpret_cast<const uint4*>(dout + o), x);
    unpack8f(*reinterpret_cast<const uint4*>(o1 + o), y);
    const float f = eb[ob];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      s = fmaf(x[e], y[e], s);
      x[e] *= f;
    }
    *reinterpret_cast<uint4*>(dos + o) = pack8f(x);
    for (int k = nv >> 1; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
    if (vv == 0) db[ob] = s;
  }
}

// dv = dv1 + dvhat e^{b_last - b}; db_i -= sum dvhat vhat, the chunk's last step gets that sum over all steps and
// alpha dalpha; dg = reverse cumulative sum of db.  dv1 and dvo null: dv is not wanted; dalpha and dg null: dg is not.
template <bool DV>
__global__ void __launch_bounds__(256) group_bwd2_kernel(const __nv_bfloat16* __restrict__ dvhat, const __nv_bfloat16* __restrict__ vhat,
                                                         const __nv_bfloat16* __restrict__ dv1, const float* __restrict__ b,
                                                         const float* __restrict__ db, const float* __restrict__ alpha, const float* __restrict__ dalpha,
                                                         int C, int H, int dv, __nv_bfloat16* __restrict__ dvo, float* __restrict__ dg) {
  __shared__ float sdb[128], sv[128];
  int ch, h, vv, r0, groups;
  group_rows(C, H, dv, ch, h, vv, r0, groups);
  const int nv = dv >> 3;
  const float last = b[((long long)ch * C + C - 1) * H + h];
  for (int i = r0; i < C; i += groups) {
    const long long ob = ((long long)ch * C + i) * H + h, o = ob * dv + vv * 8;
    float x[8], y[8], z[8], s = 0.f;
    unpack8f(*reinterpret_cast<const uint4*>(dvhat + o), x);
    unpack8f(*reinterpret_cast<const uint4*>(vhat + o), y);
    unpack8f(*reinterpret_cast<const uint4*>((DV ? dv1 : vhat) + o), z);
    const float f = __expf(last - b[ob]);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      s = fmaf(x[e], y[e], s);
      z[e] = fmaf(x[e], f, z[e]);
    }
    if (DV) *reinterpret_cast<uint4*>(dvo + o) = pack8f(z);
    for (int k = nv >> 1; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
    if (vv == 0) {
      sdb[i] = db[ob] - s;
      sv[i] = s;
    }
  }
  if (dg == nullptr) return;
  __syncthreads();
  if (threadIdx.x < 32) {  // warp 0: suffix sums, up to four steps per lane
    const int lane = threadIdx.x, per = C >> 5;
    float tot = 0.f, mine = 0.f, loc[4];
    for (int k = 0; k < per; ++k) tot += sv[lane * per + k];
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    tot += alpha[(long long)ch * H + h] * dalpha[(long long)ch * H + h];  // everything that enters through the last step
    for (int k = per - 1; k >= 0; --k) {
      mine += sdb[lane * per + k];
      loc[k] = mine;
    }
    float suf = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float t = __shfl_down_sync(0xffffffffu, suf, o);
      if (lane + o < 32) suf += t;
    }
    suf -= mine;
    for (int k = 0; k < per; ++k) dg[((long long)ch * C + lane * per + k) * H + h] = loc[k] + suf + tot;
  }
}

inline bool group_shape_ok(int C, int dv) {
  const int nv = dv >> 3;
  return (C == 64 || C == 128) && (dv & 7) == 0 && nv >= 1 && nv <= 32 && (nv & (nv - 1)) == 0;
}

}  // namespace

extern "C" {

int fb_group_prep_fwd(const void* v, const float* g, int NC, int C, int H, int dv, float scale, float* b, float* eb, float* alpha, void* vhat,
                      cudaStream_t stream) {
  if (NC <= 0) return 0;
  if (!group_shape_ok(C, dv) || !fb::aligned(16, v, vhat)) return -2;
  group_prep_fwd_kernel<<<(unsigned)(NC * H), 256, 0, stream>>>((const __nv_bfloat16*)v, g, C, H, dv, scale, b, eb, alpha, (__nv_bfloat16*)vhat);
  return fb::launch_ok("group_prep_fwd_kernel");
}

int fb_group_bwd1(const void* dout, const void* o1, const float* eb, int NC, int C, int H, int dv, void* dos, float* db, cudaStream_t stream) {
  if (NC <= 0) return 0;
  if (!group_shape_ok(C, dv) || !fb::aligned(16, dout, o1, dos)) return -2;
  group_bwd1_kernel<<<(unsigned)(NC * H), 256, 0, stream>>>((const __nv_bfloat16*)dout, (const __nv_bfloat16*)o1, eb, C, H, dv, (__nv_bfloat16*)dos, db);
  return fb::launch_ok("group_bwd1_kernel");
}

int fb_group_bwd2(const void* dvhat, const void* vhat, const void* dv1, const float* b, const float* db, const float* alpha, const float* dalpha, int NC,
                  int C, int H, int dv, void* dvo, float* dg, cudaStream_t stream) {
  if (NC <= 0) return 0;
  if (!group_shape_ok(C, dv) || !fb::aligned(16, dvhat, vhat, dv1, dvo)) return -2;
  const auto kernel = dvo != nullptr ? group_bwd2_kernel<true> : group_bwd2_kernel<false>;
  kernel<<<(unsigned)(NC * H), 256, 0, stream>>>((const __nv_bfloat16*)dvhat, (const __nv_bfloat16*)vhat, (const __nv_bfloat16*)dv1, b, db, alpha, dalpha,
                                                 C, H, dv, (__nv_bfloat16*)dvo, dg);
  return fb::launch_ok("group_bwd2_kernel");
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------------------------
// GLA intra-chunk scores  A_ij = scale * sum_d q_id k_jd exp(b_id - b_jd),  j <= i, of 64-token chunks.  The diagonal 16 x 16
// sub-blocks are evaluated pairwise so that no exponent is positive whatever the gates are (the "secondary chunking" of
// fla/ops/gla/chunk.py:88-170); the sub-blocks left of them come in from a batched GEMM on re-based operands.
// q, k: [NC, 64, H, dk] bf16; b: [NC, 64, H, dk] fp32 (within-chunk cumulative log decay); blk: [3 NC, H, 16, 48] bf16, entry
// (3 c + I - 1) holding the 16 rows of sub-block I; A: [NC, H, 64, 64] bf16, written in full.
// One block per (chunk, head).  Four lanes share a tile of 2 x 2 pairs, a quarter of the channels each: 4 x 36 tiles (of those on
// the diagonal three pairs count) = 576 threads.  Operands of 64 channels at a time in shared memory, rows 4 words apart modulo
// the banks; eight 16-byte reads and sixteen exponentials per tile and four
// channels.  With a thread per pair (four reads for four exponentials, operands brought in two bytes at a time) shared memory
// bound it: 0.271 ms at 65,536 tokens, 4 heads of 128; this takes 0.193.
namespace {

// Where the rows of a chunk's q, k and gate lie: packed tokens (src [64 NC]: the token of every chunk row, -1: padding, a chunk's
// tokens follow one another), ld* elements from row to row, or, src null, in the padded rows themselves.
struct GlaRows {
  const int* src;
  long long ldq, ldk, ldg;  // (the scores read no gate)
};
// log(sigmoid(x)) / norm without cancellation or underflow (inv: 1 / norm): log(1 + e), e = exp(-|x|) <= 1, is 2 artanh(s), s = e / (2 + e), by the
// artanh series up to s^13 for s <= 1/3 (off by 1.5e-8 relative at most).  Both quotients are corrected by their remainders, so that the
// exponential (2^-22) is what is left: closer than the chain of kernels before it, whose exponent was rounded to one float.
__device__ __forceinline__ float log_sigmoid(float x, float norm, float inv) {
  const float e = exp_neg_fine(-fabsf(x)), y = 2.f + e, r = __fdividef(1.f, y), s0 = e * r, s = fmaf(fmaf(-y, s0, e), r, s0), w = s * s;
  float p = fmaf(w, 1.f / 13.f, 1.f / 11.f);
  p = fmaf(p, w, 1.f / 9.f);
  p = fmaf(p, w, 1.f / 7.f);
  p = fmaf(p, w, 1.f / 5.f);
  p = fmaf(p, w, 1.f / 3.f);
  p = fmaf(p, w, 1.f);
  const float l = fminf(x, 0.f) - 2.f * s * p, q = l * inv;
  return l > -3e38f ? fmaf(fmaf(-norm, q, l), inv, q) : q;  // (-inf leaves no remainder)
}
__device__ __forceinline__ void unpack8_bf16(const uint4& v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) f[2 * i] = __uint_as_float(w[i] << 16), f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
}
// first row of chunk c and how many rows it has
__device__ __forceinline__ void gla_rows(const int* __restrict__ src, int c, long long& row0, int& n) {
  row0 = 64ll * c, n = 64;
  if (src == nullptr) return;
  const int lane = threadIdx.x & 31;
  const int* s = src + 64ll * c;
  n = __popc(__ballot_sync(0xffffffffu, s[lane] >= 0)) + __popc(__ballot_sync(0xffffffffu, s[lane + 32] >= 0));
  row0 = s[0];
}

constexpr int GD_T = 64;        // channels per trip
constexpr int GD_LD = GD_T + 4;
constexpr int GD_THREADS = 576;

template <typename TQ>
__global__ void __launch_bounds__(GD_THREADS, 2) gla_scores_kernel(const TQ* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                                                                const float* __restrict__ b, const __nv_bfloat16* __restrict__ blk,
                                                                __nv_bfloat16* __restrict__ A, const GlaRows at, int H, int dk, float scale, int vec) {
  extern __shared__ __align__(16) float sm[];
  float *sq = sm, *sk = sq + 64 * GD_LD, *sb = sk + 64 * GD_LD;
  const int ch = blockIdx.x, c = ch / H, h = ch - c * H, tid = threadIdx.x;
  long long row0;
  int n;
  gla_rows(at.src, c, row0, n);
  const int tile = tid >> 2, part = tid & 3, sub = tile / 36, tt = tile - sub * 36;
  int ti = (int)((sqrtf(8.f * tt + 1.f) - 1.f) * 0.5f);
  while ((ti + 1) * (ti + 2) / 2 <= tt) ++ti;
  while (ti * (ti + 1) / 2 > tt) --ti;
  const int tj = tt - ti * (ti + 1) / 2;
  const int ri = (sub * 16 + 2 * ti) * GD_LD + part * 4, rj = (sub * 16 + 2 * tj) * GD_LD + part * 4;
  constexpr float LOG2E = 1.4426950408889634f;
  const TQ* qp = q + row0 * at.ldq + (long long)h * dk;
  const __nv_bfloat16* kp = k + row0 * at.ldk + (long long)h * dk;
  const float* bp = b + ((long long)c * 64 * H + h) * dk;
  const long long ldb = (long long)H * dk;
  // a thread brings eight channels of a row
  const int lr = tid >> 3, lc = (tid & 7) * 8;
  uint4 nq[sizeof(TQ) / 2], nk;
  float4 nb[2];  // a trip's operands between global and shared memory
  auto fetch = [&](int d0) {
    const bool in = tid < 512 && d0 + lc < dk, there = in && lr < n;  // dk is a multiple of 8 here
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int t = 0; t < (int)sizeof(TQ) / 2; ++t) nq[t] = there ? reinterpret_cast<const uint4*>(qp + lr * at.ldq + d0 + lc)[t] : none;
    nk = there ? *reinterpret_cast<const uint4*>(kp + lr * at.ldk + d0 + lc) : none;
#pragma unroll
    for (int t = 0; t < 2; ++t) nb[t] = in ? reinterpret_cast<const float4*>(bp + lr * ldb + d0 + lc)[t] : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  auto put = [&]() {
    if (tid >= 512) return;
    float f[8];
    float4 *oq = reinterpret_cast<float4*>(sq + lr * GD_LD + lc), *ok = reinterpret_cast<float4*>(sk + lr * GD_LD + lc),
           *ob = reinterpret_cast<float4*>(sb + lr * GD_LD + lc);
    if constexpr (sizeof(TQ) == 4) {
      oq[0] = *reinterpret_cast<const float4*>(&nq[0]);
      oq[1] = *reinterpret_cast<const float4*>(&nq[1]);
    } else {
      unpack8_bf16(nq[0], f);
      oq[0] = make_float4(f[0], f[1], f[2], f[3]), oq[1] = make_float4(f[4], f[5], f[6], f[7]);
    }
    unpack8_bf16(nk, f);
    ok[0] = make_float4(f[0], f[1], f[2], f[3]), ok[1] = make_float4(f[4], f[5], f[6], f[7]);
#pragma unroll
    for (int t = 0; t < 2; ++t) ob[t] = make_float4(nb[t].x * LOG2E, nb[t].y * LOG2E, nb[t].z * LOG2E, nb[t].w * LOG2E);
  };
  float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
  for (int d0 = 0; d0 < dk; d0 += GD_T) {
    if (vec) fetch(d0);
    __syncthreads();
    if (vec) {
      put();
    } else {  // rows that are not whole vectors
      for (int idx = tid; idx < 64 * GD_T; idx += GD_THREADS) {
        const int r = idx / GD_T, d = idx % GD_T;
        const bool in = d0 + d < dk, there = in && r < n;
        sq[r * GD_LD + d] = there ? (float)qp[r * at.ldq + d0 + d] : 0.f;
        sk[r * GD_LD + d] = there ? __bfloat162float(kp[r * at.ldk + d0 + d]) : 0.f;
        sb[r * GD_LD + d] = in ? bp[r * ldb + d0 + d] * LOG2E : 0.f;
      }
    }
    __syncthreads();
#pragma unroll 2
    for (int d = 0; d < GD_T; d += 16) {
      float4 qi[2], bi[2], kj[2], bj[2];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        qi[t] = *reinterpret_cast<const float4*>(sq + ri + t * GD_LD + d);
        bi[t] = *reinterpret_cast<const float4*>(sb + ri + t * GD_LD + d);
        kj[t] = *reinterpret_cast<const float4*>(sk + rj + t * GD_LD + d);
        bj[t] = *reinterpret_cast<const float4*>(sb + rj + t * GD_LD + d);
      }
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          acc[x][y] = fmaf(qi[x].x * kj[y].x, exp2f(bi[x].x - bj[y].x), acc[x][y]);
          acc[x][y] = fmaf(qi[x].y * kj[y].y, exp2f(bi[x].y - bj[y].y), acc[x][y]);
          acc[x][y] = fmaf(qi[x].z * kj[y].z, exp2f(bi[x].z - bj[y].z), acc[x][y]);
          acc[x][y] = fmaf(qi[x].w * kj[y].w, exp2f(bi[x].w - bj[y].w), acc[x][y]);
        }
    }
  }
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      acc[x][y] += __shfl_xor_sync(0xffffffffu, acc[x][y], 1);
      acc[x][y] += __shfl_xor_sync(0xffffffffu, acc[x][y], 2);
    }
  __nv_bfloat16* o = A + (long long)ch * 4096;
  {
    const int x = part >> 1, y = part & 1, i = 2 * ti + x, j = 2 * tj + y;  // the pair of the tile that this lane writes
    const float v = x ? (y ? acc[1][1] : acc[1][0]) : (y ? acc[0][1] : acc[0][0]);
    // above the diagonal the exponent is positive and the sum means nothing
    o[(sub * 16 + i) * 64 + sub * 16 + j] = __float2bfloat16(j <= i ? v * scale : 0.f);
  }
  // the rest of the matrix: sub-blocks to the left from the GEMM, zeros to the right (16-byte pieces), zeros above the diagonal
  for (int idx = tid; idx < 64 * 8; idx += GD_THREADS) {
    const int r = idx >> 3, c8 = (idx & 7) * 8, I = r >> 4;
    if ((c8 >> 4) == I) continue;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (c8 < 16 * I) v = *reinterpret_cast<const uint4*>(blk + ((((long long)c * 3 + I - 1) * H + h) * 16 + (r & 15)) * 48 + c8);
    *reinterpret_cast<uint4*>(o + r * 64 + c8) = v;
  }
  for (int idx = tid; idx < 4 * 256; idx += GD_THREADS) {
    const int I = idx >> 8, r = (idx >> 4) & 15, cc = idx & 15;
    if ((cc >> 1) > (r >> 1)) o[(I * 16 + r) * 64 + I * 16 + cc] = __float2bfloat16(0.f);
  }
}

// The whole channel-wise backward of a chunk: diagonal sub-blocks and preparation.  A thread owns one channel of one (chunk,
// head); per sub-block its 16 rows of q, k and b sit in registers and each of the 136 pairs costs one exponential that serves
// dq and dk (the pairwise kernel took one for each, read its operands from shared memory, and added into fp32 arrays that
// others had to clear, convert and add up: 0.66 ms + 0.44 ms + about 0.6 ms of passes at 65,536 tokens, 4 heads of 128).
//   dq_id = scale sum_{j<=i} dA_ij k_jd e^{b_id-b_jd} + dqbar_id scale e^{b_id} + dqt_id e^{b_id-r_I}
//   dk_jd = scale sum_{i>=j} dA_ij q_id e^{b_id-b_jd} + dkhat_jd e^{b_last-b_jd} + sum_I dk3[I]_jd e^{r_I-b_jd}
//   db    = q dq - k dk (+ what enters through b_last: khat and alpha), dg = reverse cumulative sum of db
// dA: bf16 [NC, H, 64, 64] (only the diagonal sub-blocks are read).  q, k, dq, dk and the gate's gradient lie as GlaRows says (`to`: the
// gradients).  With `raw` the gate is g = logsigmoid(raw) norm, and its gradient is that of raw in bf16.
// FULL: the chunk has all of its 64 rows; a test per row keeps the loads of the next rows behind it, so only the chunks at the
// documents' ends make it.  What the second half of a sub-block needs is loaded in front of the pairs, whose 136 exponentials it takes
// to come: loaded after them, and each under a test of its own, they doubled the waits (0.70 ms at 65,536 tokens, 4 heads of 128; this takes
// 0.418 with the gate's argument, 0.105 instead of 0.166 for 64 channels, 32,767 tokens).  Two blocks of 128 threads per SM (three: 0.451).
__device__ __forceinline__ unsigned short ld_now(const __nv_bfloat16* p, bool yes) {  // a read-only load that stays where it is written
  unsigned short v;
  asm volatile("{.reg .pred p; setp.ne.s32 p, %2, 0; mov.b16 %0, 0; @p ld.global.nc.u16 %0, [%1];}" : "=h"(v) : "l"(p), "r"((int)yes));
  return v;
}
__device__ __forceinline__ float ld_now(const float* p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float bf16_of(unsigned short v) { return __uint_as_float((uint32_t)v << 16); }
template <bool FULL, int TPB>
__device__ __forceinline__ void gla_bwd_rows(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, const float* __restrict__ b,
                                             const __nv_bfloat16* __restrict__ dkhat, const __nv_bfloat16* __restrict__ dqbar,
                                             const __nv_bfloat16* __restrict__ dqt, const __nv_bfloat16* __restrict__ dk3,
                                             __nv_bfloat16* __restrict__ dq, __nv_bfloat16* __restrict__ dk_, void* __restrict__ dg,
                                             const __nv_bfloat16* __restrict__ raw, float norm, const float (&sA)[4][16][16], float (&sgb)[64][TPB],
                                             int rs, int ldq, int ldk, int ldg, int lddq, int lddk, int lddg, int n, float dalpha, float scale) {
  constexpr float LOG2E = 1.4426950408889634f;
  float r[4];
#pragma unroll
  for (int I = 0; I < 4; ++I) r[I] = __ldg(b + 16 * I * rs) * LOG2E;
  const float b_last = __ldg(b + 63 * rs) * LOG2E;
  float acc_last = 0.f;
#pragma unroll 1
  for (int I = 0; I < 4; ++I) {
    float qv[16], kv[16], bv[16], gq[16], gk[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int row = I * 16 + i;
      qv[i] = FULL || row < n ? __bfloat162float(__ldg(q + row * ldq)) : 0.f;
      kv[i] = FULL || row < n ? __bfloat162float(__ldg(k + row * ldk)) : 0.f;
      bv[i] = __ldg(b + row * rs) * LOG2E;
      gq[i] = gk[i] = 0.f;
    }
    unsigned short a_khat[16], a_qbar[16], a_qt[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int off = (I * 16 + i) * rs;
      a_khat[i] = ld_now(dkhat + off, true);
      a_qbar[i] = ld_now(dqbar + off, true);
      a_qt[i] = ld_now(dqt + off, I > 0);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) {
        const float t = i == j ? sA[I][i][j] : sA[I][i][j] * exp2f(bv[i] - bv[j]);
        gq[i] = fmaf(t, kv[j], gq[i]);
        gk[j] = fmaf(t, qv[i], gk[j]);
      }
    const float rI = r[0] * (I == 0) + r[1] * (I == 1) + r[2] * (I == 2) + r[3] * (I == 3);
#pragma unroll
    for (int half = 0; half < 16; half += 8) {
      unsigned short a_k3[3][8];  // all that eight rows need, together: each load under its own test waited for the one before
#pragma unroll
      for (int J = 0; J < 3; ++J)
#pragma unroll
        for (int i = 0; i < 8; ++i) a_k3[J][i] = ld_now(dk3 + (J * 48 + min(I, 2) * 16 + half + i) * rs, J >= I);
#pragma unroll
      for (int ii = 0; ii < 8; ++ii) {
        const int i = half + ii, row = I * 16 + i;
        const float g_khat = bf16_of(a_khat[i]) * exp2f(b_last - bv[i]);
        gq[i] = fmaf(bf16_of(a_qbar[i]), exp2f(bv[i]) * scale, gq[i]);
        if (I > 0) gq[i] = fmaf(bf16_of(a_qt[i]), exp2f(bv[i] - rI), gq[i]);
        gk[i] += g_khat;
        acc_last = fmaf(g_khat, kv[i], acc_last);
#pragma unroll
        for (int J = 0; J < 3; ++J)
          if (J >= I) gk[i] = fmaf(bf16_of(a_k3[J][ii]), exp2f(r[J + 1] - bv[i]), gk[i]);
        if (FULL || row < n) {
          dq[row * lddq] = __float2bfloat16(gq[i]);
          dk_[row * lddk] = __float2bfloat16(gk[i]);
        }
        sgb[row][threadIdx.x] = qv[i] * gq[i] - kv[i] * gk[i];
      }
    }
  }
  float tail = acc_last + dalpha * exp2f(b_last);  // gradient of b_last
  if (raw == nullptr) {
#pragma unroll 8
    for (int i = 63; i >= 0; --i) {
      tail += sgb[i][threadIdx.x];
      if (FULL || i < n) ((float*)dg)[i * lddg] = tail;
    }
  } else {
#pragma unroll 8
    for (int i = 63; i >= 0; --i) {
      tail += sgb[i][threadIdx.x];
      if (FULL || i < n) ((__nv_bfloat16*)dg)[i * lddg] = __float2bfloat16(tail * norm / (1.f + __expf(__bfloat162float(__ldg(raw + i * ldg)))));
    }
  }
}

// TPB: 64 where a head has no more channels, else 128
template <int TPB>
__global__ void __launch_bounds__(TPB, 256 / TPB) gla_bwd_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                                                      const float* __restrict__ b, const __nv_bfloat16* __restrict__ dA,
                                                      const __nv_bfloat16* __restrict__ dkhat, const __nv_bfloat16* __restrict__ dqbar,
                                                      const __nv_bfloat16* __restrict__ dqt, const __nv_bfloat16* __restrict__ dk3,
                                                      const float* __restrict__ dalpha, __nv_bfloat16* __restrict__ dq,
                                                      __nv_bfloat16* __restrict__ dk_, void* __restrict__ dg, const __nv_bfloat16* __restrict__ raw,
                                                      float norm, const GlaRows at, const GlaRows to, int H, int dk, float scale) {
  __shared__ float sA[4][16][16];
  __shared__ float sgb[64][TPB];
  const int d = blockIdx.y * TPB + threadIdx.x;
  const int ch = blockIdx.x, c = ch / H, h = ch - c * H;
  long long row0;
  int n;
  gla_rows(at.src, c, row0, n);
  for (int idx = threadIdx.x; idx < 1024; idx += TPB) {
    const int I = idx >> 8, r = (idx >> 4) & 15, cc = idx & 15;
    sA[I][r][cc] = cc <= r ? __bfloat162float(dA[((long long)ch * 64 + I * 16 + r) * 64 + I * 16 + cc]) * scale : 0.f;
  }
  __syncthreads();
  if (d >= dk) return;
  // every row of the chunk lies within 32 bits of its first
  const int rs = H * dk;
  const long long base = ((long long)c * 64 * H + h) * dk + d, col = (long long)h * dk + d;
  const long long g0 = row0 * to.ldg + col;
  void* dgp = raw == nullptr ? (void*)((float*)dg + g0) : (void*)((__nv_bfloat16*)dg + g0);
  auto rows = [&](auto full) {
    gla_bwd_rows<decltype(full)::value, TPB>(q + row0 * at.ldq + col, k + row0 * at.ldk + col, b + base, dkhat + base, dqbar + base,
                                        dqt + ((long long)c * 48 - 16) * rs + col,  // rows of sub-blocks 1..3 only, read at the others' offsets
                                        dk3 + (long long)c * 144 * rs + col, dq + row0 * to.ldq + col, dk_ + row0 * to.ldk + col, dgp,
                                        raw == nullptr ? nullptr : raw + row0 * at.ldg + col, norm, sA, sgb, rs, (int)at.ldq, (int)at.ldk, (int)at.ldg,
                                        (int)to.ldq, (int)to.ldk, (int)to.ldg, n, dalpha[(long long)ch * dk + d], scale);
  };
  if (n == 64) rows(std::true_type{});
  else rows(std::false_type{});
}

}  // namespace

extern "C" {

// rows: src, ldq, ldk, ldg of GlaRows
int fb_gla_scores(const void* q, int q32, const void* k, const float* b, const void* blk, void* A, const int* src, long long ldq, long long ldk, int NC,
                  int H, int dk, float scale, cudaStream_t stream) {
  if (NC <= 0) return 0;
  if (!fb::aligned(16, blk, A)) return -2;
  constexpr int smem = 3 * 64 * GD_LD * 4;
  const GlaRows at{src, ldq, ldk, 0};
  const int vec = dk % 8 == 0 && ldq % 8 == 0 && ldk % 8 == 0 && fb::aligned(16, q, k, b);
  auto launch = [&](auto kernel, auto* qq) -> int {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    kernel<<<NC * H, GD_THREADS, smem, stream>>>(qq, (const __nv_bfloat16*)k, b, (const __nv_bfloat16*)blk, (__nv_bfloat16*)A, at, H, dk, scale, vec);
    return fb::launch_ok("gla_scores_kernel");
  };
  return q32 ? launch(gla_scores_kernel<float>, (const float*)q) : launch(gla_scores_kernel<__nv_bfloat16>, (const __nv_bfloat16*)q);
}

int fb_gla_bwd(const void* q, const void* k, const float* b, const void* dA, const void* dkhat, const void* dqbar, const void* dqt,
               const void* dk3, const float* dalpha, void* dq, void* dk_, void* dg, const void* raw, float norm, const int* src, long long ldq,
               long long ldk, long long ldg, long long lddq, long long lddk, long long lddg, int NC, int H, int dk, float scale, cudaStream_t stream) {
  if (NC <= 0) return 0;
  const int tpb = dk <= 64 ? 64 : 128;
  const auto kernel = dk <= 64 ? gla_bwd_kernel<64> : gla_bwd_kernel<128>;
  kernel<<<dim3(NC * H, (dk + tpb - 1) / tpb), tpb, 0, stream>>>(
      (const __nv_bfloat16*)q, (const __nv_bfloat16*)k, b, (const __nv_bfloat16*)dA, (const __nv_bfloat16*)dkhat, (const __nv_bfloat16*)dqbar,
      (const __nv_bfloat16*)dqt, (const __nv_bfloat16*)dk3, dalpha, (__nv_bfloat16*)dq, (__nv_bfloat16*)dk_, dg, (const __nv_bfloat16*)raw, norm,
      GlaRows{src, ldq, ldk, ldg}, GlaRows{src, lddq, lddk, lddg}, H, dk, scale);
  return fb::launch_ok("gla_bwd_kernel");
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------------------------
// L2 normalisation of q / k heads (fla/modules/l2norm.py): y = x * rsqrt(sum x^2 + eps); one warp per row of D <= 1024.
namespace {

__global__ void l2norm_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, float* __restrict__ rstd,
                                  long long rows, int D, float eps) {
  const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const __nv_bfloat16* xr = x + row * D;
  float v[32];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int d = lane + i * 32;
    v[i] = d < D ? __bfloat162float(xr[d]) : 0.f;
    ss = fmaf(v[i], v[i], ss);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float r = rsqrtf(ss + eps);
  if (lane == 0) rstd[row] = r;
  __nv_bfloat16* yr = y + row * D;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int d = lane + i * 32;
    if (d < D) yr[d] = __float2bfloat16(v[i] * r);
  }
}

__global__ void l2norm_bwd_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ rstd,
                                  const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dx, long long rows, int D) {
  const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const __nv_bfloat16* xr = x + row * D;
  const __nv_bfloat16* gr = dy + row * D;
  const float r = rstd[row];
  float y[32], g[32];
  float dot = 0.f;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int d = lane + i * 32;
    y[i] = d < D ? __bfloat162float(xr[d]) * r : 0.f;
    g[i] = d < D ? __bfloat162float(gr[d]) : 0.f;
    dot = fmaf(y[i], g[i], dot);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
  __nv_bfloat16* dr = dx + row * D;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int d = lane + i * 32;
    if (d < D) dr[d] = __float2bfloat16(r * (g[i] - y[i] * dot));
  }
}

// The same two kernels for head dims that are a multiple of 64: LANES threads share a row and move 8 bf16 per access,
// so a warp covers 32 / LANES rows with 16-byte loads (the one-warp-per-row kernels above spend most of their 32
// predicated 2-byte accesses idle at the usual head dims of 64..256).
template <int LANES, int ITERS>
__global__ void l2norm_fwd_vec_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y,
                                      float* __restrict__ rstd, long long rows, float eps) {
  constexpr int D = LANES * ITERS * 8;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long row = gid / LANES;
  const int sub = (int)(gid % LANES);
  const bool live = row < rows;
  uint4 v[ITERS];
  float ss = 0.f;
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    v[it] = live ? *reinterpret_cast<const uint4*>(x + row * D + (it * LANES + sub) * 8) : make_uint4(0, 0, 0, 0);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[it]);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = __bfloat1622float2(h[e]);
      ss = fmaf(f.x, f.x, fmaf(f.y, f.y, ss));
    }
  }
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float r = rsqrtf(ss + eps);
  if (!live) return;
  if (sub == 0) rstd[row] = r;
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[it]);
    uint4 o;
    __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = __bfloat1622float2(h[e]);
      oh[e] = __floats2bfloat162_rn(f.x * r, f.y * r);
    }
    *reinterpret_cast<uint4*>(y + row * D + (it * LANES + sub) * 8) = o;
  }
}

template <int LANES, int ITERS>
__global__ void l2norm_bwd_vec_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ rstd,
                                      const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dx, long long rows) {
  constexpr int D = LANES * ITERS * 8;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long row = gid / LANES;
  const int sub = (int)(gid % LANES);
  const bool live = row < rows;
  const float r = live ? rstd[row] : 0.f;
  uint4 xv[ITERS], gv[ITERS];
  float dot = 0.f;
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const long long off = row * D + (it * LANES + sub) * 8;
    xv[it] = live ? *reinterpret_cast<const uint4*>(x + off) : make_uint4(0, 0, 0, 0);
    gv[it] = live ? *reinterpret_cast<const uint4*>(dy + off) : make_uint4(0, 0, 0, 0);
    const __nv_bfloat162* xh = reinterpret_cast<const __nv_bfloat162*>(&xv[it]);
    const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gv[it]);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 a = __bfloat1622float2(xh[e]), g = __bfloat1622float2(gh[e]);
      dot = fmaf(a.x * r, g.x, fmaf(a.y * r, g.y, dot));
    }
  }
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
  if (!live) return;
#pragma unroll
  for (int it = 0; it < ITERS; ++it) {
    const __nv_bfloat162* xh = reinterpret_cast<const __nv_bfloat162*>(&xv[it]);
    const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gv[it]);
    uint4 o;
    __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 a = __bfloat1622float2(xh[e]), g = __bfloat1622float2(gh[e]);
      oh[e] = __floats2bfloat162_rn(r * (g.x - a.x * r * dot), r * (g.y - a.y * r * dot));
    }
    *reinterpret_cast<uint4*>(dx + row * D + (it * LANES + sub) * 8) = o;
  }
}

template <int LANES, int ITERS>
void l2norm_fwd_vec(const void* x, void* y, float* rstd, long long rows, float eps, cudaStream_t stream) {
  const long long threads = rows * LANES;
  l2norm_fwd_vec_kernel<LANES, ITERS><<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>(
      (const __nv_bfloat16*)x, (__nv_bfloat16*)y, rstd, rows, eps);
}
template <int LANES, int ITERS>
void l2norm_bwd_vec(const void* x, const float* rstd, const void* dy, void* dx, long long rows, cudaStream_t stream) {
  const long long threads = rows * LANES;
  l2norm_bwd_vec_kernel<LANES, ITERS><<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>(
      (const __nv_bfloat16*)x, rstd, (const __nv_bfloat16*)dy, (__nv_bfloat16*)dx, rows);
}
bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

}  // namespace

extern "C" {

int fb_l2norm_fwd(const void* x, void* y, float* rstd, long long rows, int D, float eps, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (D > 1024) return -2;
  if (aligned16(x) && aligned16(y)) {
    switch (D) {
      case 64: l2norm_fwd_vec<8, 1>(x, y, rstd, rows, eps, stream); return fb::launch_ok("l2norm_fwd_vec_kernel");
      case 128: l2norm_fwd_vec<16, 1>(x, y, rstd, rows, eps, stream); return fb::launch_ok("l2norm_fwd_vec_kernel");
      case 256: l2norm_fwd_vec<32, 1>(x, y, rstd, rows, eps, stream); return fb::launch_ok("l2norm_fwd_vec_kernel");
      case 512: l2norm_fwd_vec<32, 2>(x, y, rstd, rows, eps, stream); return fb::launch_ok("l2norm_fwd_vec_kernel");
      case 1024: l2norm_fwd_vec<32, 4>(x, y, rstd, rows, eps, stream); return fb::launch_ok("l2norm_fwd_vec_kernel");
      default: break;
    }
  }
  l2norm_fwd_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, stream>>>((const __nv_bfloat16*)x, (__nv_bfloat16*)y, rstd, rows, D, eps);
  return fb::launch_ok("l2norm_fwd_kernel");
}

int fb_l2norm_bwd(const void* x, const float* rstd, const void* dy, void* dx, long long rows, int D, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (D > 1024) return -2;
  if (aligned16(x) && aligned16(dy) && aligned16(dx)) {
    switch (D) {
      case 64: l2norm_bwd_vec<8, 1>(x, rstd, dy, dx, rows, stream); return fb::launch_ok("l2norm_bwd_vec_kernel");
      case 128: l2norm_bwd_vec<16, 1>(x, rstd, dy, dx, rows, stream); return fb::launch_ok("l2norm_bwd_vec_kernel");
      case 256: l2norm_bwd_vec<32, 1>(x, rstd, dy, dx, rows, stream); return fb::launch_ok("l2norm_bwd_vec_kernel");
      case 512: l2norm_bwd_vec<32, 2>(x, rstd, dy, dx, rows, stream); return fb::launch_ok("l2norm_bwd_vec_kernel");
      case 1024: l2norm_bwd_vec<32, 4>(x, rstd, dy, dx, rows, stream); return fb::launch_ok("l2norm_bwd_vec_kernel");
      default: break;
    }
  }
  l2norm_bwd_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, stream>>>((const __nv_bfloat16*)x, rstd, (const __nv_bfloat16*)dy,
                                                                   (__nv_bfloat16*)dx, rows, D);
  return fb::launch_ok("l2norm_bwd_kernel");
}

}  // extern "C"

// out[b (, r)] = sum x[b, ...] * y[b, ...] in fp32 for bf16 x, y of shape [B, R, C]: per_row = 0 sums over R x C (one
// value per batch), per_row = 1 sums over C (one value per row).  One block per batch.
namespace {
__global__ void __launch_bounds__(256) pair_dot_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ y,
                                                       float* __restrict__ out, int R, int C, int per_row) {
  const long long b = blockIdx.x;
  const __nv_bfloat16* xb = x + b * (long long)R * C;
  const __nv_bfloat16* yb = y + b * (long long)R * C;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto dot8 = [](const uint4& a, const uint4& d, float s) {
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, dw[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      s = fmaf(__uint_as_float(aw[t] << 16), __uint_as_float(dw[t] << 16), s);
      s = fmaf(__uint_as_float(aw[t] & 0xffff0000u), __uint_as_float(dw[t] & 0xffff0000u), s);
    }
    return s;
  };
  if (per_row) {
    for (int r = warp; r < R; r += 8) {
      float s = 0.f;
      for (int c = lane * 8; c < C; c += 256)
        s = dot8(*reinterpret_cast<const uint4*>(xb + (long long)r * C + c), *reinterpret_cast<const uint4*>(yb + (long long)r * C + c), s);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) out[b * R + r] = s;
    }
    return;
  }
  // one sum: the block takes the matrix as one run of 16-byte vectors, four in flight per thread (row by row, rows of 64 left
  // 24 of 32 lanes idle: 0.217 ms for 16,576 pairs of 128 x 64, now 0.084)
  __shared__ float red[8];
  const uint4 *xv = reinterpret_cast<const uint4*>(xb), *yv = reinterpret_cast<const uint4*>(yb);
  const int n = R * C / 8;
  float s = 0.f;
  for (int v = threadIdx.x; v < n; v += 4 * 256) {
    uint4 a[4], d[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const bool in = v + t * 256 < n;
      a[t] = in ? xv[v + t * 256] : make_uint4(0u, 0u, 0u, 0u);
      d[t] = in ? yv[v + t * 256] : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) s = dot8(a[t], d[t], s);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) red[warp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int i = 0; i < 8; ++i) t += red[i];
    out[b] = t;
  }
}
}  // namespace

extern "C" int fb_pair_dot(const void* x, const void* y, float* out, long long B, int R, int C, int per_row, cudaStream_t stream) {
  if (B <= 0) return 0;
  if ((C & 7) || !fb::aligned(16, x, y)) return -2;
  pair_dot_kernel<<<(unsigned)B, 256, 0, stream>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)y, out, R, C, per_row);
  return fb::launch_ok("pair_dot_kernel");
}

// ---------------------------------------------------------------------------------------------------------------
// Chunk-state recurrence without a transition matrix (GLA, GSA, SSD), all chunks of every document in one launch:
//   forward   out[c] = state entering chunk c:            s = 0;  out[c] = s;  s = alpha[c] s + x[c],   c ascending
//   reverse   out[c] = adjoint of the state leaving c:    s = 0;  out[c] = s;  s = alpha[c] s + x[c],   c descending
// x: increments (fp32) or gradients of the states (bf16) [NC, H, rows, cols]; out bf16; alpha: [NC, H] (per_row = 0) or
// [NC, H, rows] (per_row = 1).  Each thread owns V state elements (16 bytes of x) of one document and carries them in
// registers, with four chunks' loads in flight.  Nothing but the bf16 states is written: writing the running fp32 state beside
// them, which nobody reads, and copying bf16 gradients to fp32 first took twice the traffic.  Bound by memory: with fp32 x
// 0.13 ms for 136 M elements (6.3 TB/s); with bf16 x 8 bytes per
// thread and chunk took 0.142 ms, 16 bytes take 0.090 (6.0 TB/s).
// Grid: (ceil(H*rows*cols/V / 256), documents).
namespace {
template <typename TIn, int V>
__global__ void __launch_bounds__(256) state_scan_kernel(const long long* __restrict__ first, const long long* __restrict__ last,
                                                         const float* __restrict__ alpha, int per_row, const TIn* __restrict__ X,
                                                         __nv_bfloat16* __restrict__ out, int H, int rows, int cols, int reverse) {
  using InVec = typename std::conditional<sizeof(TIn) * V == 16, uint4, uint2>::type;
  using OutVec = typename std::conditional<V == 8, uint4, uint2>::type;
  const long long per_chunk = (long long)H * rows * cols;
  const long long e = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * V;
  if (e >= per_chunk) return;
  const int doc = blockIdx.y;
  const long long c0 = first[doc];
  const int cnt = (int)(last[doc] - c0) + 1;
  const int h = (int)(e / ((long long)rows * cols));
  const int row = (int)((e / cols) % rows);
  float s[V];
#pragma unroll
  for (int j = 0; j < V; ++j) s[j] = 0.f;
  for (int i0 = 0; i0 < cnt; i0 += 4) {
    InVec x[4];
    float al[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i0 + k >= cnt) break;
      const long long c = c0 + (reverse ? cnt - 1 - i0 - k : i0 + k);
      al[k] = per_row ? alpha[(c * H + h) * rows + row] : alpha[c * H + h];
      x[k] = *reinterpret_cast<const InVec*>(X + c * per_chunk + e);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i0 + k >= cnt) break;
      const long long c = c0 + (reverse ? cnt - 1 - i0 - k : i0 + k);
      OutVec q;
      __nv_bfloat162* q2 = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
      for (int j = 0; j < V / 2; ++j) q2[j] = __floats2bfloat162_rn(s[2 * j], s[2 * j + 1]);
      *reinterpret_cast<OutVec*>(out + c * per_chunk + e) = q;
      const uint32_t* w = reinterpret_cast<const uint32_t*>(&x[k]);
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const float xj = sizeof(TIn) == 4 ? __uint_as_float(w[j]) : __uint_as_float((j & 1) ? w[j >> 1] & 0xffff0000u : w[j >> 1] << 16);
        s[j] = fmaf(al[k], s[j], xj);
      }
    }
  }
}
}  // namespace

extern "C" int fb_state_scan(const long long* first, const long long* last, int n_docs, const float* alpha, int per_row, const void* X,
                             int x16, void* out, int H, int rows, int cols, int reverse, cudaStream_t stream) {
  if (n_docs <= 0) return 0;
  if ((cols & 3) || !fb::aligned(x16 ? 8 : 16, X) || !fb::aligned(8, out)) return -2;
  const long long per_chunk = (long long)H * rows * cols;
  const bool wide = x16 && (cols & 7) == 0 && !(((uintptr_t)X | (uintptr_t)out) & 15);  // eight bf16 are 16 bytes
  const int v = wide ? 8 : 4;
  const dim3 grid((unsigned)((per_chunk / v + 255) / 256), (unsigned)n_docs);
  __nv_bfloat16* o = (__nv_bfloat16*)out;
  if (wide) state_scan_kernel<__nv_bfloat16, 8><<<grid, 256, 0, stream>>>(first, last, alpha, per_row, (const __nv_bfloat16*)X, o, H, rows, cols, reverse);
  else if (x16) state_scan_kernel<__nv_bfloat16, 4><<<grid, 256, 0, stream>>>(first, last, alpha, per_row, (const __nv_bfloat16*)X, o, H, rows, cols, reverse);
  else state_scan_kernel<float, 4><<<grid, 256, 0, stream>>>(first, last, alpha, per_row, (const float*)X, o, H, rows, cols, reverse);
  return fb::launch_ok("state_scan_kernel");
}

// ---------------------------------------------------------------------------------------------------------------
// GLA chunk preparation (one pass over q, k, g of a chunk; stands in for fla/ops/utils/cumsum.py and the scaling
// prologues of fla/ops/gla/chunk.py).  Chunk layout [NC, 64, H, dk]; a thread owns one channel of one (chunk, head).
//   b     = within-chunk cumulative sum of the log decay g                      (fp32)
//   khat  = k * exp(b_last - b)        key decayed to the end of its chunk      (state update operand)
//   qbar  = q * exp(b) * scale         query against the state entering the chunk
//   qt    = q * exp(b - r_I)           query re-based on the first row of its 16-row sub-block I = 1..3 (48 rows: there is
//                                      nothing before sub-block 0)
//   k3[I-1, j] = k_j * exp(r_I - b_j)  for j < 16 I, zero otherwise (I = 1..3; 48 rows): keys re-based for sub-block I
//   alpha = exp(b_last)                per-channel decay of the state across the chunk
// Every exponent is <= 0.
namespace {

// Bound by memory: 20 bytes per channel and row with the gate's bf16 argument (6 in, 14 out: b 4, khat and qbar 2 each, qt 1.5, k3 4.5), 22
// with the gate in fp32; 0.104 ms at 65,536 tokens, 4 heads of 128.  A thread owns two channels of one
// 16-row sub-block and loads all it needs of q, k and g before it uses any; the sub-blocks' sums meet in shared memory.  A
// thread that walked the 64 rows of a chunk waited for memory sub-block after sub-block and read b back: 0.205 ms.  This takes 0.155, with the
// gate's own arithmetic (0.05 by a kernel before; 0.146 with an exponent rounded to one float).
template <bool RAW>
__global__ void __launch_bounds__(256, 2) gla_prep_fwd_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                                                          const void* __restrict__ g, float norm, const GlaRows at, float* __restrict__ b,
                                                          __nv_bfloat16* __restrict__ khat, __nv_bfloat16* __restrict__ qbar,
                                                          __nv_bfloat16* __restrict__ qt, __nv_bfloat16* __restrict__ k3,
                                                          float* __restrict__ alpha, int H, int dk, float scale) {
  __shared__ float2 total[4][64], first[4][64], last[64];
  const int x = threadIdx.x & 63, Iq = threadIdx.x >> 6;
  const int d = blockIdx.y * 128 + 2 * x;
  const bool live = d < dk;
  const int ch = blockIdx.x, c = ch / H, h = ch - c * H;
  long long row0;
  int n;
  gla_rows(at.src, c, row0, n);
  const long long col = (long long)h * dk + d;
  const __nv_bfloat16 *qp = q + (row0 + Iq * 16) * at.ldq + col, *kp = k + (row0 + Iq * 16) * at.ldk + col;
  const int there = live ? n - Iq * 16 : 0;  // rows of this sub-block
  uint32_t qv[16], kv[16];
  float2 bv[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const long long o = (row0 + Iq * 16 + i) * at.ldg + col;
    if constexpr (RAW) {
      const uint32_t v = i < there ? *reinterpret_cast<const uint32_t*>((const __nv_bfloat16*)g + o) : 0u;
      bv[i] = make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
    } else {
      bv[i] = i < there ? *reinterpret_cast<const float2*>((const float*)g + o) : make_float2(0.f, 0.f);
    }
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    qv[i] = i < there ? *reinterpret_cast<const uint32_t*>(qp + i * at.ldq) : 0u;
    kv[i] = i < there ? *reinterpret_cast<const uint32_t*>(kp + i * at.ldk) : 0u;
  }
  float2 run = make_float2(0.f, 0.f);
  const float inv = RAW ? __frcp_rn(norm) : 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    if (RAW) bv[i] = i < there ? make_float2(log_sigmoid(bv[i].x, norm, inv), log_sigmoid(bv[i].y, norm, inv)) : make_float2(0.f, 0.f);
    run.x += bv[i].x;
    run.y += bv[i].y;
    bv[i] = run;
  }
  total[Iq][x] = run;
  __syncthreads();
  float2 pre = make_float2(0.f, 0.f);
  for (int I = 0; I < Iq; ++I) pre.x += total[I][x].x, pre.y += total[I][x].y;
#pragma unroll
  for (int i = 0; i < 16; ++i) bv[i].x += pre.x, bv[i].y += pre.y;
  first[Iq][x] = bv[0];
  if (Iq == 3) last[x] = bv[15];
  __syncthreads();
  if (!live) return;
  const long long rs = (long long)H * dk;                                            // distance of padded rows
  const long long base = ((long long)c * 64 + Iq * 16) * rs + col;                   // row 0 of the sub-block
  const long long qtbase = ((long long)c * 48 + Iq * 16 - 16) * rs + col;
  const long long k3base = ((long long)c * 3 * 48 + Iq * 16) * rs + col;             // (I - 1 = 0, row 0 of the sub-block)
  const float2 b_last = last[x], rq = bv[0], r1 = first[1][x], r2 = first[2][x], r3 = first[3][x];
  if (Iq == 0) *reinterpret_cast<float2*>(alpha + (long long)ch * dk + d) = make_float2(__expf(b_last.x), __expf(b_last.y));
  auto put = [](__nv_bfloat16* p, long long off, float a, float e) {
    *reinterpret_cast<__nv_bfloat162*>(p + off) = __floats2bfloat162_rn(a, e);
  };
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float2 bi = bv[i];
    const float2 qi = make_float2(__uint_as_float(qv[i] << 16), __uint_as_float(qv[i] & 0xffff0000u));
    const float2 ki = make_float2(__uint_as_float(kv[i] << 16), __uint_as_float(kv[i] & 0xffff0000u));
    const long long off = base + i * rs;
    *reinterpret_cast<float2*>(b + off) = bi;
    put(khat, off, ki.x * __expf(b_last.x - bi.x), ki.y * __expf(b_last.y - bi.y));
    put(qbar, off, qi.x * __expf(bi.x) * scale, qi.y * __expf(bi.y) * scale);
    if (Iq > 0) put(qt, qtbase + i * rs, qi.x * __expf(bi.x - rq.x), qi.y * __expf(bi.y - rq.y));
    if (Iq < 3) {
#pragma unroll
      for (int I = 1; I <= 3; ++I) {
        const float2 r = I == 1 ? r1 : I == 2 ? r2 : r3;
        const bool before = Iq < I;
        put(k3, k3base + ((long long)(I - 1) * 48 + i) * rs, before ? ki.x * __expf(r.x - bi.x) : 0.f, before ? ki.y * __expf(r.y - bi.y) : 0.f);
      }
    }
  }
}

}  // namespace

extern "C" {

// g: fp32 (raw 0), or bf16 whose logsigmoid over norm is the gate; src, ld*: see GlaRows
int fb_gla_prep_fwd(const void* q, const void* k, const void* g, int raw, float norm, const int* src, long long ldq, long long ldk, long long ldg,
                    float* b, void* khat, void* qbar, void* qt, void* k3, float* alpha, int NC, int H, int dk, float scale, cudaStream_t stream) {
  if (NC <= 0) return 0;
  if ((dk & 1) || (ldq & 1) || (ldk & 1) || (ldg & 1) || !fb::aligned(4, q, k, khat, qbar, qt, k3) || !fb::aligned(8, b, alpha) ||
      !fb::aligned(raw ? 4 : 8, g))
    return -2;
  const dim3 grid(NC * H, (dk + 127) / 128);
  const auto kernel = raw ? gla_prep_fwd_kernel<true> : gla_prep_fwd_kernel<false>;
  kernel<<<grid, 256, 0, stream>>>((const __nv_bfloat16*)q, (const __nv_bfloat16*)k, g, norm, GlaRows{src, ldq, ldk, ldg}, b, (__nv_bfloat16*)khat,
                                   (__nv_bfloat16*)qbar, (__nv_bfloat16*)qt, (__nv_bfloat16*)k3, alpha, H, dk, scale);
  return fb::launch_ok("gla_prep_fwd_kernel");
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------------------------
// Preparation of the scalar-gated chunk algorithms (gated delta rule, SSD): one log decay per token and head.
//   b = within-chunk cumulative sum of g,  khat = k * exp(b_last - b),  qbar = q * exp(b) * scale,  alpha = exp(b_last)
// q, k: [NC, C, H, dk] bf16 (C = 64 or 128); g, b: [NC, C, H] fp32; alpha: [NC, H].  One block per (chunk, head).
namespace {

__global__ void __launch_bounds__(256) scalar_prep_fwd_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                                                              const float* __restrict__ g, float* __restrict__ b,
                                                              __nv_bfloat16* __restrict__ khat, __nv_bfloat16* __restrict__ qbar,
                                                              float* __restrict__ alpha, int C, int H, int dk, float scale) {
  __shared__ float sb[128];
  const int ch = blockIdx.x, c = ch / H, h = ch - c * H;
  for (int i = threadIdx.x; i < C; i += blockDim.x) sb[i] = g[((long long)c * C + i) * H + h];
  __syncthreads();
  if (threadIdx.x == 0) {
    float run = 0.f;
    for (int i = 0; i < C; ++i) {
      run += sb[i];
      sb[i] = run;
    }
    alpha[ch] = __expf(run);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < C; i += blockDim.x) b[((long long)c * C + i) * H + h] = sb[i];
  const float b_last = sb[C - 1];
  const int nv = dk >> 3;  // 8 channels per thread and row
  for (int idx = threadIdx.x; idx < C * nv; idx += blockDim.x) {
    const int i = idx / nv, v = idx - i * nv;
    const long long off = (((long long)c * C + i) * H + h) * dk + v * 8;
    const float ek = __expf(b_last - sb[i]), eq = __expf(sb[i]) * scale;
    const uint4 qa = *reinterpret_cast<const uint4*>(q + off), ka = *reinterpret_cast<const uint4*>(k + off);
    const __nv_bfloat162* q2 = reinterpret_cast<const __nv_bfloat162*>(&qa);
    const __nv_bfloat162* k2 = reinterpret_cast<const __nv_bfloat162*>(&ka);
    uint4 qo, ko;
    __nv_bfloat162* qo2 = reinterpret_cast<__nv_bfloat162*>(&qo);
    __nv_bfloat162* ko2 = reinterpret_cast<__nv_bfloat162*>(&ko);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 qf = __bfloat1622float2(q2[j]), kf = __bfloat1622float2(k2[j]);
      qo2[j] = __floats2bfloat162_rn(qf.x * eq, qf.y * eq);
      ko2[j] = __floats2bfloat162_rn(kf.x * ek, kf.y * ek);
    }
    *reinterpret_cast<uint4*>(qbar + off) = qo;
    *reinterpret_cast<uint4*>(khat + off) = ko;
  }
}

// Backward: dq = dqbar e^{b} scale, dk = dkhat e^{b_last - b}; db_i = sum_d (q dq - k dk) + db_in_i, the b_last uses
// (sum_i sum_d k dk, and alpha) go to the last row, and dg is the reverse cumulative sum of db.
__global__ void __launch_bounds__(256) scalar_prep_bwd_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                                                              const float* __restrict__ b, const __nv_bfloat16* __restrict__ dkhat,
                                                              const __nv_bfloat16* __restrict__ dqbar, const float* __restrict__ dalpha,
                                                              const float* __restrict__ db_in, __nv_bfloat16* __restrict__ dq,
                                                              __nv_bfloat16* __restrict__ dk_, float* __restrict__ dg, int C, int H,
                                                              int dk, float scale) {
  __shared__ float sb[128], sdb[128];
  __shared__ float slast;
  const int ch = blockIdx.x, c = ch / H, h = ch - c * H;
  for (int i = threadIdx.x; i < C; i += blockDim.x) {
    sb[i] = b[((long long)c * C + i) * H + h];
    sdb[i] = db_in != nullptr ? db_in[((long long)c * C + i) * H + h] : 0.f;
  }
  if (threadIdx.x == 0) slast = 0.f;
  __syncthreads();
  const float b_last = sb[C - 1];
  const int nv = dk >> 3;
  // dk / 8 is a power of two for every supported head size, so a row's vectors sit in aligned lane groups
  for (int idx = threadIdx.x; idx < C * nv; idx += blockDim.x) {
    const int i = idx / nv, v = idx - i * nv;
    const long long off = (((long long)c * C + i) * H + h) * dk + v * 8;
    const float ek = __expf(b_last - sb[i]), eq = __expf(sb[i]) * scale;
    const uint4 qa = *reinterpret_cast<const uint4*>(q + off), ka = *reinterpret_cast<const uint4*>(k + off);
    uint4 gqa = make_uint4(0, 0, 0, 0), gka = make_uint4(0, 0, 0, 0);
    if (dqbar != nullptr) gqa = *reinterpret_cast<const uint4*>(dqbar + off);
    if (dkhat != nullptr) gka = *reinterpret_cast<const uint4*>(dkhat + off);
    const __nv_bfloat162* q2 = reinterpret_cast<const __nv_bfloat162*>(&qa);
    const __nv_bfloat162* k2 = reinterpret_cast<const __nv_bfloat162*>(&ka);
    const __nv_bfloat162* gq2 = reinterpret_cast<const __nv_bfloat162*>(&gqa);
    const __nv_bfloat162* gk2 = reinterpret_cast<const __nv_bfloat162*>(&gka);
    uint4 qo, ko;
    __nv_bfloat162* qo2 = reinterpret_cast<__nv_bfloat162*>(&qo);
    __nv_bfloat162* ko2 = reinterpret_cast<__nv_bfloat162*>(&ko);
    float tq = 0.f, tk = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 qf = __bfloat1622float2(q2[j]), kf = __bfloat1622float2(k2[j]);
      const float2 gq = __bfloat1622float2(gq2[j]), gk = __bfloat1622float2(gk2[j]);
      const float dqx = gq.x * eq, dqy = gq.y * eq, dkx = gk.x * ek, dky = gk.y * ek;
      qo2[j] = __floats2bfloat162_rn(dqx, dqy);
      ko2[j] = __floats2bfloat162_rn(dkx, dky);
      tq += qf.x * dqx + qf.y * dqy;
      tk += kf.x * dkx + kf.y * dky;
    }
    *reinterpret_cast<uint4*>(dq + off) = qo;
    *reinterpret_cast<uint4*>(dk_ + off) = ko;
    // reduce over the lanes that share the row (a row's vectors are consecutive lanes), then one atomic per group
    const int grp = nv < 32 ? nv : 32;
    float s1 = tq - tk, s2 = tk;
    for (int o = grp >> 1; o > 0; o >>= 1) s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    if ((threadIdx.x & (grp - 1)) == 0) atomicAdd(&sdb[i], s1);
    if ((threadIdx.x & 31) == 0) atomicAdd(&slast, s2);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float tail = slast + (dalpha != nullptr ? dalpha[ch] * __expf(b_last) : 0.f);
    for (int i = C - 1; i >= 0; --i) {
      tail += sdb[i];
      sdb[i] = tail;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < C; i += blockDim.x) dg[((long long)c * C + i) * H + h] = sdb[i];
}

}  // namespace

extern "C" {

int fb_scalar_prep_fwd(const void* q, const void* k, const float* g, float* b, void* khat, void* qbar, float* alpha, int NC,
                       int C, int H, int dk, float scale, cudaStream_t stream) {
  if (NC <= 0) return 0;
  if (C > 128 || (dk & 7) || !fb::aligned(16, q, k, khat, qbar)) return -2;
  scalar_prep_fwd_kernel<<<NC * H, 256, 0, stream>>>((const __nv_bfloat16*)q, (const __nv_bfloat16*)k, g, b, (__nv_bfloat16*)khat,
                                                     (__nv_bfloat16*)qbar, alpha, C, H, dk, scale);
  return fb::launch_ok("scalar_prep_fwd_kernel");
}

int fb_scalar_prep_bwd(const void* q, const void* k, const float* b, const void* dkhat, const void* dqbar, const float* dalpha,
                       const float* db_in, void* dq, void* dk_, float* dg, int NC, int C, int H, int dk, float scale,
                       cudaStream_t stream) {
  if (NC <= 0) return 0;
  if (C > 128 || (dk & 7) || ((dk >> 3) & ((dk >> 3) - 1))) return -2;  // dk / 8 must be a power of two
  if (!fb::aligned(16, q, k, dkhat, dqbar, dq, dk_)) return -2;
  scalar_prep_bwd_kernel<<<NC * H, 256, 0, stream>>>((const __nv_bfloat16*)q, (const __nv_bfloat16*)k, b, (const __nv_bfloat16*)dkhat,
                                                     (const __nv_bfloat16*)dqbar, dalpha, db_in, (__nv_bfloat16*)dq,
                                                     (__nv_bfloat16*)dk_, dg, C, H, dk, scale);
  return fb::launch_ok("scalar_prep_bwd_kernel");
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------------------------
// First pass of gated slot attention: o_ic = scale sum_{j<=i} (q_i . k_j) v_jc exp(b_ic - b_jc), a decay along the VALUE
// dimension c (the slots, M of them), then a softmax over the slots (fla/ops/gsa/chunk.py:826-871).  64-token chunks, layouts
// as for GLA: v [NC, 64, H, M] bf16; g, b, o: [NC, 64, H, M] fp32; P = tril(q k^T) [NC, H, 64, 64].  A thread owns a channel of
// a (chunk, head) and keeps 16 rows in registers; the products of rows across sub-blocks and chunks come from batched
// GEMMs.  These kernels are everything between the GEMMs: as a chain of elementwise passes over fp32 [.., H, M] arrays and
// pairwise kernels over padded matrices this pass took 236 launches with the rest of the layer and 2.5 ms at 32,767 tokens.
namespace {

constexpr float VD_LOG2E = 1.4426950408889634f;

// b = cumsum(g); vhat = v e^{b_last - b}; v3[I-1]_j = v_j e^{r_I - b_j} for j < 16 I (zero beyond); alpha = e^{b_last}
__global__ void __launch_bounds__(128) vdecay_prep_kernel(const __nv_bfloat16* __restrict__ v, const float* __restrict__ g, float* __restrict__ b,
                                                          __nv_bfloat16* __restrict__ vhat, __nv_bfloat16* __restrict__ v3, float* __restrict__ alpha,
                                                          int H, int M, int n) {
  const int e = blockIdx.x * 128 + threadIdx.x;  // (chunk, head, channel)
  if (e >= n) return;
  const int c = e / (H * M), hm = e - c * H * M;
  const long long rs = (long long)H * M, base = (long long)c * 64 * rs + hm, base3 = (long long)c * 144 * rs + hm;
  float run = 0.f, r[4];
#pragma unroll 8
  for (int i = 0; i < 64; ++i) {
    run += g[base + i * rs];
    b[base + i * rs] = run;
    if ((i & 15) == 0) r[i >> 4] = run;
  }
  alpha[e] = __expf(run);
#pragma unroll 4
  for (int i = 0; i < 64; ++i) {
    const float bi = b[base + i * rs], x = __bfloat162float(v[base + i * rs]);
    vhat[base + i * rs] = __float2bfloat16(x * __expf(run - bi));
    if (i < 48) {
#pragma unroll
      for (int I = 1; I <= 3; ++I) v3[base3 + ((I - 1) * 48 + i) * rs] = __float2bfloat16(i < 16 * I ? x * __expf(r[I] - bi) : 0.f);
    }
  }
}

// o = scale (o1 e^b + acc e^{b - r_I} + diagonal sub-blocks), qv = softmax over the slots (null: not wanted).  One block per (chunk, head), 4 threads
// per slot: thread (I, c) forms the 16 rows of sub-block I.  o1 [NC, 64, H, M] fp32, acc [NC, 48, H, M] fp32 (rows 16..63).
__global__ void vdecay_out_kernel(const float* __restrict__ o1, const float* __restrict__ acc, const float* __restrict__ P,
                                  const __nv_bfloat16* __restrict__ v, const float* __restrict__ b, int H, int M, float scale,
                                  float* __restrict__ o, __nv_bfloat16* __restrict__ qv) {
  extern __shared__ float sm[];
  float* sP = sm;          // [4][16][16]
  float* so = sm + 1024;   // [64][M + 1]
  const int ch = blockIdx.x, c = ch / H, h = ch - c * H;
  for (int idx = threadIdx.x; idx < 1024; idx += blockDim.x) {
    const int I = idx >> 8, r = (idx >> 4) & 15, cc = idx & 15;
    sP[idx] = P[((long long)ch * 64 + I * 16 + r) * 64 + I * 16 + cc];
  }
  __syncthreads();
  const long long rs = (long long)H * M;
  for (int t = threadIdx.x; t < 4 * M; t += blockDim.x) {
    const int I = t / M, m = t - I * M;
    const long long base = ((long long)c * 64 + I * 16) * rs + (long long)h * M + m;
    const long long basea = ((long long)c * 48 + (I - 1) * 16) * rs + (long long)h * M + m;
    float vv[16], bv[16], out[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      vv[i] = __bfloat162float(v[base + i * rs]);
      bv[i] = b[base + i * rs] * VD_LOG2E;
      out[i] = o1[base + i * rs] * exp2f(bv[i]);
    }
    if (I > 0) {
#pragma unroll
      for (int i = 0; i < 16; ++i) out[i] = fmaf(acc[basea + i * rs], exp2f(bv[i] - bv[0]), out[i]);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) out[i] = fmaf(sP[I * 256 + i * 16 + j] * vv[j], i == j ? 1.f : exp2f(bv[i] - bv[j]), out[i]);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (qv != nullptr) so[(I * 16 + i) * (M + 1) + m] = out[i] * scale;
      else o[base + i * rs] = out[i] * scale;
    }
  }
  if (qv == nullptr) return;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int i = warp; i < 64; i += warps) {
    const float* row = so + i * (M + 1);
    float mx = -INFINITY, s = 0.f;
    for (int m = lane; m < M; m += 32) mx = fmaxf(mx, row[m]);
    for (int k = 16; k > 0; k >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, k));
    for (int m = lane; m < M; m += 32) s += __expf(row[m] - mx);
    for (int k = 16; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
    const float inv = 1.f / s;
    const long long g = ((long long)c * 64 + i) * rs + (long long)h * M;
    for (int m = lane; m < M; m += 32) {
      o[g + m] = row[m];
      qv[g + m] = __float2bfloat16(__expf(row[m] - mx) * inv);
    }
  }
}

// Softmax backward and the two scaled operands: d = p (dqv - sum p dqv) (the gradient of o; or given as d32), do = scale d (fp32),
// do1 = do e^b, dacc = do e^{b - r_I} (rows 16..63), both bf16.  One warp per (token, head).
__global__ void __launch_bounds__(256) vdecay_bwd1_kernel(const float* __restrict__ o, const __nv_bfloat16* __restrict__ dqv,
                                                          const float* __restrict__ d32, const float* __restrict__ b,
                                                          int H, int M, float scale, long long rows, float* __restrict__ dout,
                                                          __nv_bfloat16* __restrict__ do1, __nv_bfloat16* __restrict__ dacc) {
  const long long row = ((long long)blockIdx.x * 256 + threadIdx.x) >> 5;  // (chunk, i, head)
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const int h = (int)(row % H);
  const long long tok = row / H;
  const int i = (int)(tok & 63);
  const long long c = tok >> 6, g = row * M;
  const float* r0 = b + ((c * 64 + (i & 48)) * H + h) * M;  // first row of the sub-block
  float mx = -INFINITY, s = 0.f, dot = 0.f;
  if (d32 == nullptr)
    for (int m = lane; m < M; m += 32) mx = fmaxf(mx, o[g + m]);
  for (int k = 16; k > 0; k >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, k));
  for (int m = lane; d32 == nullptr && m < M; m += 32) {
    const float e = __expf(o[g + m] - mx);
    s += e;
    dot = fmaf(e, __bfloat162float(dqv[g + m]), dot);
  }
  for (int k = 16; k > 0; k >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, k);
    dot += __shfl_xor_sync(0xffffffffu, dot, k);
  }
  const float inv = 1.f / s;
  dot *= inv;
  for (int m = lane; m < M; m += 32) {
    const float bi = b[g + m];
    const float d = scale * (d32 != nullptr ? d32[g + m] : __expf(o[g + m] - mx) * inv * (__bfloat162float(dqv[g + m]) - dot));
    dout[g + m] = d;
    do1[g + m] = __float2bfloat16(d * __expf(bi));
    if (i >= 16) dacc[((c * 48 + i - 16) * H + h) * M + m] = __float2bfloat16(d * __expf(bi - r0[m]));
  }
}

// dv = dvhat e^{b_last - b} + sum_I dv3[I] e^{r_I - b} + diagonal sub-blocks;  db = do o / scale - v dv (+ what enters through
// b_last: vhat and alpha), dg = reverse cumulative sum.  `o` carries the factor scale and so does `do`, hence the division.
// TPB: 64 where a head has no more slots, else 128; loads as in gla_bwd_rows (half of the threads idle and each load of dv3 behind the
// one before: 0.250 ms at 32,767 tokens, 4 heads of 64 slots; this takes 0.105)
template <int TPB>
__global__ void __launch_bounds__(TPB, 256 / TPB) vdecay_bwd2_kernel(const float* __restrict__ P, const __nv_bfloat16* __restrict__ v, const float* __restrict__ b,
                                                          const float* __restrict__ dout, const float* __restrict__ o,
                                                          const __nv_bfloat16* __restrict__ dvhat, const __nv_bfloat16* __restrict__ dv3,
                                                          const float* __restrict__ dalpha, int H, int M, float inv_scale, __nv_bfloat16* __restrict__ dv,
                                                          float* __restrict__ dg) {
  __shared__ float sP[4][16][16];
  __shared__ float sgb[64][TPB];
  const int ch = blockIdx.x, c = ch / H, h = ch - c * H;
  for (int idx = threadIdx.x; idx < 1024; idx += TPB) {
    const int I = idx >> 8, r = (idx >> 4) & 15, cc = idx & 15;
    sP[I][r][cc] = P[((long long)ch * 64 + I * 16 + r) * 64 + I * 16 + cc];
  }
  __syncthreads();
  const int m = blockIdx.y * TPB + threadIdx.x;
  if (m >= M) return;
  const long long rs = (long long)H * M, base = (long long)c * 64 * rs + (long long)h * M + m, base3 = (long long)c * 144 * rs + (long long)h * M + m;
  float r[4];
#pragma unroll
  for (int I = 0; I < 4; ++I) r[I] = b[base + 16 * I * rs] * VD_LOG2E;
  const float b_last = b[base + 63 * rs] * VD_LOG2E;
  float acc_last = 0.f;
#pragma unroll 1
  for (int I = 0; I < 4; ++I) {
    float bv[16], dd[16], gv[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const long long off = base + (I * 16 + i) * rs;
      bv[i] = b[off] * VD_LOG2E;
      dd[i] = dout[off];
      gv[i] = 0.f;
    }
    unsigned short a_v[16], a_vhat[16];
    float a_o[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const long long off = base + (I * 16 + i) * rs;
      a_v[i] = ld_now(v + off, true);
      a_vhat[i] = ld_now(dvhat + off, true);
      a_o[i] = ld_now(o + off);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) gv[j] = fmaf(sP[I][i][j] * dd[i], i == j ? 1.f : exp2f(bv[i] - bv[j]), gv[j]);
#pragma unroll
    for (int half = 0; half < 16; half += 8) {
      unsigned short a_v3[3][8];
#pragma unroll
      for (int J = 0; J < 3; ++J)
#pragma unroll
        for (int i = 0; i < 8; ++i) a_v3[J][i] = ld_now(dv3 + base3 + (J * 48 + min(I, 2) * 16 + half + i) * rs, J >= I);
#pragma unroll
      for (int ii = 0; ii < 8; ++ii) {
        const int i = half + ii;
        const float x = bf16_of(a_v[i]);
        const float gl = bf16_of(a_vhat[i]) * exp2f(b_last - bv[i]);
        gv[i] += gl;
        acc_last = fmaf(gl, x, acc_last);
#pragma unroll
        for (int J = 0; J < 3; ++J)
          if (J >= I) gv[i] = fmaf(bf16_of(a_v3[J][ii]), exp2f(r[J + 1] - bv[i]), gv[i]);
        dv[base + (I * 16 + i) * rs] = __float2bfloat16(gv[i]);
        sgb[I * 16 + i][threadIdx.x] = dd[i] * a_o[i] * inv_scale - x * gv[i];
      }
    }
  }
  float tail = acc_last + dalpha[(long long)ch * M + m] * exp2f(b_last);
#pragma unroll 8
  for (int i = 63; i >= 0; --i) {
    tail += sgb[i][threadIdx.x];
    dg[base + i * rs] = tail;
  }
}

}  // namespace

extern "C" {

int fb_vdecay_prep(const void* v, const float* g, float* b, void* vhat, void* v3, float* alpha, int NC, int H, int M, cudaStream_t stream) {
  if (NC <= 0) return 0;
  const int n = NC * H * M;
  vdecay_prep_kernel<<<(n + 127) / 128, 128, 0, stream>>>((const __nv_bfloat16*)v, g, b, (__nv_bfloat16*)vhat, (__nv_bfloat16*)v3, alpha, H, M, n);
  return fb::launch_ok("vdecay_prep_kernel");
}

int fb_vdecay_out(const float* o1, const float* acc, const float* P, const void* v, const float* b, int NC, int H, int M, float scale, float* o,
                  void* qv, cudaStream_t stream) {
  if (NC <= 0) return 0;
  if (qv != nullptr && M > 512) return -2;
  const int smem = (1024 + (qv != nullptr ? 64 * (M + 1) : 0)) * 4;
  if (cudaFuncSetAttribute(vdecay_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -3;
  vdecay_out_kernel<<<NC * H, 256, smem, stream>>>(o1, acc, P, (const __nv_bfloat16*)v, b, H, M, scale, o, (__nv_bfloat16*)qv);
  return fb::launch_ok("vdecay_out_kernel");
}

int fb_vdecay_bwd1(const float* o, const void* dqv, const float* d32, const float* b, int NC, int H, int M, float scale, float* dout, void* do1, void* dacc,
                   cudaStream_t stream) {
  if (NC <= 0) return 0;
  const long long rows = (long long)NC * 64 * H;
  vdecay_bwd1_kernel<<<(unsigned)((rows * 32 + 255) / 256), 256, 0, stream>>>(o, (const __nv_bfloat16*)dqv, d32, b, H, M, scale, rows, dout,
                                                                              (__nv_bfloat16*)do1, (__nv_bfloat16*)dacc);
  return fb::launch_ok("vdecay_bwd1_kernel");
}

int fb_vdecay_bwd2(const float* P, const void* v, const float* b, const float* dout, const float* o, const void* dvhat, const void* dv3,
                   const float* dalpha, int NC, int H, int M, float inv_scale, void* dv, float* dg, cudaStream_t stream) {
  if (NC <= 0) return 0;
  const int tpb = M <= 64 ? 64 : 128;
  const auto kernel = M <= 64 ? vdecay_bwd2_kernel<64> : vdecay_bwd2_kernel<128>;
  kernel<<<dim3(NC * H, (M + tpb - 1) / tpb), tpb, 0, stream>>>(P, (const __nv_bfloat16*)v, b, dout, o, (const __nv_bfloat16*)dvhat,
                                                                (const __nv_bfloat16*)dv3, dalpha, H, M, inv_scale, (__nv_bfloat16*)dv, dg);
  return fb::launch_ok("vdecay_bwd2_kernel");
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------------------------
// Backward helper of the decayed / masked score blocks C_ij = alpha (a_i . b_j) exp(d_i - d_j):
//   g_ij  = dC_ij * keep_ij * exp(d_i - d_j)      (bf16, the operand of the two gradient GEMMs)
//   dd_i  = sum_j dC_ij C_ij - sum_j dC_ji C_ji    (gradient of the cumulative log decay)
// dC and C may each be fp32 or bf16 (exactly one pointer of each pair is non-null).  One block per (chunk, head).
namespace {

__global__ void __launch_bounds__(256) scores_bwd_prep_kernel(const float* __restrict__ dc32, const __nv_bfloat16* __restrict__ dc16,
                                                              const float* __restrict__ c32, const __nv_bfloat16* __restrict__ c16,
                                                              const float* __restrict__ d, long long d_hi, long long d_lo,
                                                              long long d_r, int H, int C, int mask_mode,
                                                              __nv_bfloat16* __restrict__ g, float* __restrict__ dd) {
  __shared__ float sd[128], srow[128], scol[128];
  const int ch = blockIdx.x, c = ch / H, h = ch - c * H;
  const float* dv = d + (long long)c * d_hi + (long long)h * d_lo;
  for (int i = threadIdx.x; i < C; i += 256) {
    sd[i] = dv[(long long)i * d_r];
    srow[i] = 0.f;
    scol[i] = 0.f;
  }
  __syncthreads();
  const long long base = (long long)ch * C * C;
  for (int idx = threadIdx.x; idx < C * C; idx += 256) {
    const int i = idx / C, j = idx - i * C;  // a warp covers 32 consecutive j of one row (C is a multiple of 32)
    const bool keep = mask_mode == 0 || (mask_mode == 1 ? j <= i : j < i);
    const float dcv = dc32 != nullptr ? dc32[base + idx] : __bfloat162float(dc16[base + idx]);
    const float cv = c32 != nullptr ? c32[base + idx] : __bfloat162float(c16[base + idx]);
    g[base + idx] = __float2bfloat16(keep ? dcv * __expf(sd[i] - sd[j]) : 0.f);
    const float e = dcv * cv;  // C is zero where masked
    float r = e;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(&srow[i], r);
    atomicAdd(&scol[j], e);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < C; i += 256) dd[(long long)ch * C + i] = srow[i] - scol[i];
}

}  // namespace

extern "C" int fb_scores_bwd_prep(const float* dc32, const void* dc16, const float* c32, const void* c16, const float* d,
                                  long long d_hi, long long d_lo, long long d_r, int NC, int H, int C, int mask_mode, void* g,
                                  float* dd, cudaStream_t stream) {
  if (NC <= 0) return 0;
  if (C > 128 || (C & 31)) return -2;
  scores_bwd_prep_kernel<<<NC * H, 256, 0, stream>>>(dc32, (const __nv_bfloat16*)dc16, c32, (const __nv_bfloat16*)c16, d, d_hi, d_lo,
                                                     d_r, H, C, mask_mode, (__nv_bfloat16*)g, dd);
  return fb::launch_ok("scores_bwd_prep_kernel");
}
