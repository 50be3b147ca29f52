// Depthwise causal short convolution (kernel width <= 8) over packed sequences, with optional bias and SiLU.
//   pre[t, d] = b[d] + sum_{j < W, j <= pos[t]} w[d, W-1-j] * x[t-j, d];   y = act(pre)
// `pos[t]` is the token's offset inside its document, so taps never reach into the previous document.
// Backward: dpre = dy * act'(pre) with pre recomputed, dx[t] = sum_j w[., W-1-j] dpre[t+j] (same document only) and partial
// sums of dw / db per strip of rows, then a fixed-order reduction of the partials.  Width 4 (every configuration's) does
// the first three in one kernel and never stores dpre; the other widths take a dpre pass and a strip pass.
// Semantics of fla/modules/conv/triton/kernels.py:37-345; the row-strip partial reduction replaces its atomics.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stddef.h>
#include <stdint.h>
#include <type_traits>
#include "host_utils.cuh"

namespace {

constexpr int MAXW = 8;

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

// weights are read as bf16 [D, W]; one thread = one token x 8 channels
template <bool SILU, bool WRITE_DPRE>
__global__ void conv_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                const __nv_bfloat16* __restrict__ b, const int* __restrict__ pos,
                                const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ out, long long T,
                                int D, int W, long long ldx, long long ldo) {
  const int vec = D >> 3;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= T * vec) return;
  const long long t = idx / vec;
  const int d0 = (int)(idx - t * vec) * 8;
  const int p = pos[t];
  float acc[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) acc[c] = b ? __bfloat162float(b[d0 + c]) : 0.f;
  for (int j = 0; j < W && j <= p; ++j) {
    float xv[8];
    unpack8(*reinterpret_cast<const uint4*>(x + (t - j) * ldx + d0), xv);
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c] += __bfloat162float(w[(d0 + c) * W + (W - 1 - j)]) * xv[c];
  }
  float o[8];
  if (WRITE_DPRE) {
    float g[8];
    unpack8(*reinterpret_cast<const uint4*>(dy + t * ldo + d0), g);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (SILU) {
        const float s = sigmoidf_(acc[c]);
        o[c] = g[c] * s * (1.f + acc[c] * (1.f - s));
      } else {
        o[c] = g[c];
      }
    }
  } else {
#pragma unroll
    for (int c = 0; c < 8; ++c) o[c] = SILU ? acc[c] * sigmoidf_(acc[c]) : acc[c];
  }
  *reinterpret_cast<uint4*>(out + t * ldo + d0) = pack8(o);
}

// Width-specialised forward (and dpre) kernel: a thread owns 8 channels and walks a strip of consecutive tokens with the
// last W-1 inputs in registers, so every input row is read once and the taps are read once per strip.
// grid = (channel vectors / 64, strips of `rows` tokens).
template <bool SILU, bool WRITE_DPRE, int W>
__global__ void __launch_bounds__(64) conv_strip_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                        const __nv_bfloat16* __restrict__ b, const int* __restrict__ pos,
                                                        const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ out,
                                                        long long T, int D, long long ldx, long long ldo, int rows) {
  const int v = blockIdx.x * 64 + threadIdx.x;
  if (v >= (D >> 3)) return;
  const int d0 = v * 8;
  const long long r0 = (long long)blockIdx.y * rows;
  const long long r1 = min(T, r0 + rows);
  float wv[W][8], bias[8], win[W > 1 ? W - 1 : 1][8];
#pragma unroll
  for (int j = 0; j < W; ++j)
#pragma unroll
    for (int c = 0; c < 8; ++c) wv[j][c] = __bfloat162float(w[(d0 + c) * W + (W - 1 - j)]);  // tap at distance j
#pragma unroll
  for (int c = 0; c < 8; ++c) bias[c] = b ? __bfloat162float(b[d0 + c]) : 0.f;
#pragma unroll
  for (int j = 1; j < W; ++j) {
    if (r0 - j >= 0) {
      unpack8(*reinterpret_cast<const uint4*>(x + (r0 - j) * ldx + d0), win[j - 1]);
    } else {
#pragma unroll
      for (int c = 0; c < 8; ++c) win[j - 1][c] = 0.f;
    }
  }
#pragma unroll 4
  for (long long t = r0; t < r1; ++t) {
    float xc[8], acc[8];
    unpack8(*reinterpret_cast<const uint4*>(x + t * ldx + d0), xc);
    const int p = pos[t];
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c] = fmaf(wv[0][c], xc[c], bias[c]);
#pragma unroll
    for (int j = 1; j < W; ++j) {
      if (j <= p) {
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[c] = fmaf(wv[j][c], win[j - 1][c], acc[c]);
      }
    }
#pragma unroll
    for (int j = W - 2; j >= 1; --j)
#pragma unroll
      for (int c = 0; c < 8; ++c) win[j][c] = win[j - 1][c];
    if (W > 1) {
#pragma unroll
      for (int c = 0; c < 8; ++c) win[0][c] = xc[c];
    }
    float o[8];
    if (WRITE_DPRE) {
      float g[8];
      unpack8(*reinterpret_cast<const uint4*>(dy + t * ldo + d0), g);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (SILU) {
          const float sg = sigmoidf_(acc[c]);
          o[c] = g[c] * sg * (1.f + acc[c] * (1.f - sg));
        } else {
          o[c] = g[c];
        }
      }
    } else {
#pragma unroll
      for (int c = 0; c < 8; ++c) o[c] = SILU ? acc[c] * sigmoidf_(acc[c]) : acc[c];
    }
    *reinterpret_cast<uint4*>(out + t * ldo + d0) = pack8(o);
  }
}

template <bool SILU, bool WRITE_DPRE>
int launch_conv_point(const void* x, const void* w, const void* b, const int* pos, const void* dy, void* out, long long T, int D,
                      int W, long long ldx, long long ldo, cudaStream_t stream) {
  const __nv_bfloat16 *xx = (const __nv_bfloat16*)x, *ww = (const __nv_bfloat16*)w, *bb = (const __nv_bfloat16*)b,
                      *gg = (const __nv_bfloat16*)dy;
  __nv_bfloat16* oo = (__nv_bfloat16*)out;
  if (W == 2 || W == 3) {
    const int rows = 32;
    dim3 grid((D / 8 + 63) / 64, (unsigned)((T + rows - 1) / rows));
    if (W == 3) conv_strip_kernel<SILU, WRITE_DPRE, 3><<<grid, 64, 0, stream>>>(xx, ww, bb, pos, gg, oo, T, D, ldx, ldo, rows);
    else conv_strip_kernel<SILU, WRITE_DPRE, 2><<<grid, 64, 0, stream>>>(xx, ww, bb, pos, gg, oo, T, D, ldx, ldo, rows);
    return fb::launch_ok("conv_strip_kernel");
  }
  const unsigned blocks = (unsigned)((T * (D / 8) + 255) / 256);
  conv_fwd_kernel<SILU, WRITE_DPRE><<<blocks, 256, 0, stream>>>(xx, ww, bb, pos, gg, oo, T, D, W, ldx, ldo);
  return fb::launch_ok("conv_fwd_kernel");
}

// dx and per-strip partial sums of dw (and db).  grid = (channel vectors / 32, strips); a warp's lanes cover 32
// consecutive channel vectors, each thread walks its strip of rows.
__global__ void conv_bwd_kernel(const __nv_bfloat16* __restrict__ dpre, const __nv_bfloat16* __restrict__ x,
                                const __nv_bfloat16* __restrict__ w, const int* __restrict__ pos,
                                __nv_bfloat16* __restrict__ dx, float* __restrict__ part, long long T, int D, int W,
                                long long ldx, long long ldd, int rows_per_strip) {
  const int vec = D >> 3;
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= vec) return;
  const int d0 = v * 8;
  const long long r0 = (long long)blockIdx.y * rows_per_strip;
  const long long r1 = min(T, r0 + rows_per_strip);
  float wv[MAXW][8];
  for (int j = 0; j < W; ++j)
#pragma unroll
    for (int c = 0; c < 8; ++c) wv[j][c] = __bfloat162float(w[(d0 + c) * W + (W - 1 - j)]);  // tap at distance j
  float dw[MAXW][8], db[8];
  for (int j = 0; j < MAXW; ++j)
#pragma unroll
    for (int c = 0; c < 8; ++c) dw[j][c] = 0.f;
#pragma unroll
  for (int c = 0; c < 8; ++c) db[c] = 0.f;
  for (long long t = r0; t < r1; ++t) {
    float g[8];
    unpack8(*reinterpret_cast<const uint4*>(dpre + t * ldd + d0), g);
    const int p = pos[t];
    // weight / bias gradients: dw[tap j] += dpre[t] * x[t - j]
#pragma unroll
    for (int c = 0; c < 8; ++c) db[c] += g[c];
    for (int j = 0; j < W && j <= p; ++j) {
      float xv[8];
      unpack8(*reinterpret_cast<const uint4*>(x + (t - j) * ldx + d0), xv);
#pragma unroll
      for (int c = 0; c < 8; ++c) dw[j][c] += g[c] * xv[c];
    }
    // input gradient: dx[t] = sum_j w[tap j] * dpre[t + j] while t + j is in the same document
    float acc[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c] = wv[0][c] * g[c];
    for (int j = 1; j < W; ++j) {
      const long long tj = t + j;
      if (tj >= T || pos[tj] < j) break;  // crossed into the next document (positions restart at 0)
      float gj[8];
      unpack8(*reinterpret_cast<const uint4*>(dpre + tj * ldd + d0), gj);
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[c] += wv[j][c] * gj[c];
    }
    *reinterpret_cast<uint4*>(dx + t * ldx + d0) = pack8(acc);
  }
  // partial layout: [strip][D][W + 1]
  float* dst = part + ((long long)blockIdx.y * D + d0) * (W + 1);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    for (int j = 0; j < W; ++j) dst[c * (W + 1) + (W - 1 - j)] = dw[j][c];
    dst[c * (W + 1) + W] = db[c];
  }
}

// Width 4.  Both directions move each row once and compute little, so what bounds them is bytes in flight: a thread owns
// four channels (8-byte accesses, a warp covers 128 channels of a row) and a few consecutive rows, and issues all of its
// loads before it uses any of them; the rows around its own come from L1, where the neighbouring warps of the block bring
// them.  At 65,536 x 1,024 the walking form of one thread per eight channels took 0.086 ms forward (3.1 TB/s) and
// 0.33 ms backward in three kernels; this forward takes 0.078 ms.
constexpr int CW = 4;          // taps
constexpr int CLANES = 32;     // threads along the channels
constexpr int CGROUPS = 8;     // row groups of a block
constexpr int FROWS = 8;       // rows of a thread, forward
constexpr int BROWS = 8;       // rows of a thread, backward
constexpr int BTILE = BROWS * CGROUPS;

__device__ __forceinline__ void unpack4(const uint2& q, float (&f)[4]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
  const float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
  f[0] = a.x, f[1] = a.y, f[2] = b.x, f[3] = b.y;
}
__device__ __forceinline__ uint2 pack4(const float (&f)[4]) {
  uint2 q;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
  h[0] = __floats2bfloat162_rn(f[0], f[1]);
  h[1] = __floats2bfloat162_rn(f[2], f[3]);
  return q;
}
__device__ __forceinline__ void load_taps(const __nv_bfloat16* w, const __nv_bfloat16* b, int d0, float (&wv)[CW][4], float (&bias)[4]) {
  // four channels' taps are 32 contiguous bytes; as sixteen 2-byte loads they cost the L1 more than the rows themselves
  const uint4* w4 = reinterpret_cast<const uint4*>(w + (long long)d0 * CW);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float f[8];
    unpack8(w4[h], f);
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int j = 0; j < CW; ++j) wv[j][2 * h + c] = f[c * CW + (CW - 1 - j)];  // tap at distance j
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) bias[c] = 0.f;
  if (b != nullptr) unpack4(*reinterpret_cast<const uint2*>(b + d0), bias);
}

template <bool SILU>
__global__ void __launch_bounds__(CLANES * CGROUPS) conv4_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                                     const __nv_bfloat16* __restrict__ b, const int* __restrict__ pos,
                                                                     __nv_bfloat16* __restrict__ y, long long T, int D, long long ldx,
                                                                     long long ldy) {
  const int d0 = (blockIdx.x * CLANES + threadIdx.x) * 4;
  const long long r0 = ((long long)blockIdx.y * CGROUPS + threadIdx.y) * FROWS;
  if (d0 >= D || r0 >= T) return;
  uint2 xq[FROWS + CW - 1];
  int p[FROWS];
#pragma unroll
  for (int i = 0; i < FROWS + CW - 1; ++i) {
    const long long r = r0 + i - (CW - 1);
    xq[i] = r >= 0 && r < T ? *reinterpret_cast<const uint2*>(x + r * ldx + d0) : make_uint2(0u, 0u);
  }
#pragma unroll
  for (int i = 0; i < FROWS; ++i) p[i] = r0 + i < T ? pos[r0 + i] : 0;
  float wv[CW][4], bias[4];
  load_taps(w, b, d0, wv, bias);
  bool whole = r0 + FROWS <= T;  // every tap of every row lies in the row's document (the same for the whole warp)
#pragma unroll
  for (int i = 0; i < FROWS; ++i) whole = whole && p[i] >= CW - 1;
  auto rows = [&](auto all) {
#pragma unroll
  for (int i = 0; i < FROWS; ++i) {
    if (!decltype(all)::value && r0 + i >= T) break;
    float acc[4] = {bias[0], bias[1], bias[2], bias[3]};
#pragma unroll
    for (int j = 0; j < CW; ++j) {
      if (decltype(all)::value || j <= p[i]) {
        float xv[4];
        unpack4(xq[i + CW - 1 - j], xv);
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] = fmaf(wv[j][c], xv[c], acc[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (SILU) acc[c] *= sigmoidf_(acc[c]);
    *reinterpret_cast<uint2*>(y + (r0 + i) * ldy + d0) = pack4(acc);
  }
  };
  if (whole) rows(std::true_type{});
  else rows(std::false_type{});
}

// Two fp32 lanes per instruction (sm_100): the backward forms about 60 products per channel and row.
using f2 = unsigned long long;
__device__ __forceinline__ f2 f2_make(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 f2_get(f2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_unpack2(uint32_t q) { return f2_make(__uint_as_float(q << 16), __uint_as_float(q & 0xffff0000u)); }
// 8 bytes into shared memory, zeros where `in` is false (nothing is read then)
__device__ __forceinline__ void cp_async8(void* dst, const void* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 8 : 0) : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr int BCH = 2 * CLANES;  // channels of a block, backward: a thread owns two
struct alignas(16) ConvTile {  // the stages follow one another: each has to start where 8-byte copies may
  uint32_t x[BTILE + 2 * (CW - 1)][CLANES];  // rows r0 - 3 .. r0 + 66, two channels a word
  uint32_t g[BTILE + CW - 1][CLANES];        // rows r0 .. r0 + 66
  int pos[BTILE + CW + 1];
};
constexpr int CSTAGES = 2;
static_assert(sizeof(ConvTile) % 16 == 0 && offsetof(ConvTile, g) % 8 == 0, "alignment of the copies");

// A block walks the tiles of 64 rows of its strip, the next tile on its way into shared memory (cp.async) while it works on
// this one; there are as many strips as fill the GPU once (four blocks per SM), so that the partial sums of the taps'
// gradients are few.  dpre of the three rows behind a thread's own is recomputed (11 rows for 8).  At 65,536 x 1,024 0.155 ms
// and 0.003 ms to sum the strips' partials; the form that loaded one tile per block into registers before it used any of it took
// 0.194 ms and 0.035 ms (1,024 strips), four channels per thread with 127 registers 0.16 ms.
template <bool SILU>
__global__ void __launch_bounds__(CLANES * CGROUPS, 4) conv4_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                                                        const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b,
                                                                        const int* __restrict__ pos, __nv_bfloat16* __restrict__ dx,
                                                                        float* __restrict__ part, long long T, int D, long long ldx, long long ldy,
                                                                        long long ldd, int tiles_per_strip) {
  extern __shared__ __align__(16) uint8_t conv_smem[];
  ConvTile* stage = reinterpret_cast<ConvTile*>(conv_smem);
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * CLANES + tx;
  const int c_block = blockIdx.x * BCH, d0 = c_block + 2 * tx;
  const bool live = d0 < D;
  constexpr int H = CW - 1;
  const long long tile0 = (long long)blockIdx.y * tiles_per_strip;
  auto fetch = [&](int tile) {
    const long long r0 = (tile0 + tile) * BTILE;
    if (tile < tiles_per_strip && r0 < T) {
      ConvTile& s = stage[tile % CSTAGES];
      constexpr int PER_ROW = BCH / 4;  // 8-byte pieces
      const int piece = tid % PER_ROW, c = c_block + piece * 4;
      if (c < D) {
        for (int i = tid / PER_ROW; i < BTILE + 2 * H; i += CLANES * CGROUPS / PER_ROW) {
          const long long r = r0 + i - H;
          const bool in = r >= 0 && r < T;
          cp_async8(&s.x[i][piece * 2], in ? x + r * ldx + c : x, in);
        }
        for (int i = tid / PER_ROW; i < BTILE + H; i += CLANES * CGROUPS / PER_ROW) {
          const bool in = r0 + i < T;
          cp_async8(&s.g[i][piece * 2], in ? dy + (r0 + i) * ldy + c : dy, in);
        }
      }
      if (tid < BTILE + H) s.pos[tid] = r0 + tid < T ? pos[r0 + tid] : -1;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  f2 wv[CW], bias = 0ull, dw[CW], db = 0ull;
  if (live) {
    float f[8];
    unpack8(*reinterpret_cast<const uint4*>(w + (long long)d0 * CW), f);
#pragma unroll
    for (int j = 0; j < CW; ++j) wv[j] = f2_make(f[CW - 1 - j], f[CW + CW - 1 - j]);  // tap at distance j
    if (b != nullptr) bias = f2_unpack2(*reinterpret_cast<const uint32_t*>(b + d0));
  }
#pragma unroll
  for (int j = 0; j < CW; ++j) dw[j] = 0ull;
  fetch(0);
  for (int tile = 0; tile < tiles_per_strip && (tile0 + tile) * BTILE < T; ++tile) {
    fetch(tile + 1);
    cp_async_wait<1>();
    __syncthreads();
    const ConvTile& s = stage[tile % CSTAGES];
    const int first = ty * BROWS;
    const long long r0 = (tile0 + tile) * BTILE + first;
    if (live && r0 < T) {
      bool whole = true;  // every tap of every row lies in the row's document (the same for the whole warp)
#pragma unroll
      for (int i = 0; i < BROWS + H; ++i) whole = whole && s.pos[first + i] >= H;
      __nv_bfloat16* out = dx + r0 * ldd + d0;
      // straight-line code for whole rows: with a branch per tap the warp waits out each row's sigmoid by itself
      auto rows = [&](auto all) {
        f2 g[CW], xv[CW];  // dpre and x of the last four rows, [0] the newest
        int p[CW];         // their positions
#pragma unroll
        for (int j = 1; j < CW; ++j) xv[j - 1] = f2_unpack2(s.x[first + H - j][tx]);
#pragma unroll
        for (int i = 0; i < BROWS + H; ++i) {
#pragma unroll
          for (int j = CW - 1; j >= 1; --j) g[j] = g[j - 1], xv[j] = xv[j - 1], p[j] = p[j - 1];
          p[0] = decltype(all)::value ? H : s.pos[first + i];
          g[0] = f2_unpack2(s.g[first + i][tx]);
          xv[0] = f2_unpack2(s.x[first + i + H][tx]);
          if (SILU) {
            f2 pre = bias;
#pragma unroll
            for (int j = 0; j < CW; ++j)
              if (decltype(all)::value || j <= p[0]) pre = f2_fma(wv[j], xv[j], pre);
            const float2 z = f2_get(pre);
            const float s0 = sigmoidf_(z.x), s1 = sigmoidf_(z.y);
            g[0] = f2_mul(g[0], f2_make(s0 * (1.f + z.x * (1.f - s0)), s1 * (1.f + z.y * (1.f - s1))));
          }
          if (i < BROWS) {  // the rows behind belong to other threads' sums
            db = f2_add(db, g[0]);
#pragma unroll
            for (int j = 0; j < CW; ++j)
              if (decltype(all)::value || j <= p[0]) dw[j] = f2_fma(g[0], xv[j], dw[j]);
          }
          if (i >= H && (decltype(all)::value || r0 + i - H < T)) {
            // dx[s] = sum_j w[tap j] dpre[s + j] while row s + j is at least j tokens into its document
            f2 acc = f2_mul(wv[0], g[H]);
            bool alive = true;
#pragma unroll
            for (int j = 1; j < CW; ++j) {
              alive = decltype(all)::value || (alive && p[H - j] >= j);
              if (alive) acc = f2_fma(wv[j], g[H - j], acc);
            }
            const float2 a = f2_get(acc);
            *reinterpret_cast<__nv_bfloat162*>(out + (i - H) * ldd) = __floats2bfloat162_rn(a.x, a.y);
          }
        }
      };
      if (whole) rows(std::true_type{});
      else rows(std::false_type{});
    }
    __syncthreads();  // the stage is free for the tile after next
  }
  cp_async_wait<0>();
  float* red = reinterpret_cast<float*>(conv_smem);  // [CGROUPS][BCH * (CW + 1)]: the stages are done with
  constexpr int NRED = BCH * (CW + 1);
  float* mine = red + ty * NRED + tx * 2 * (CW + 1);
#pragma unroll
  for (int j = 0; j < CW; ++j) {
    const float2 v = f2_get(dw[j]);
    mine[CW - 1 - j] = v.x;
    mine[CW + 1 + CW - 1 - j] = v.y;
  }
  const float2 vb = f2_get(db);
  mine[CW] = vb.x;
  mine[CW + 1 + CW] = vb.y;
  __syncthreads();
  const int n = min(BCH, D - c_block) * (CW + 1);
  float* dst = part + ((long long)blockIdx.y * D + c_block) * (CW + 1);
  for (int i = tid; i < n; i += CLANES * CGROUPS) {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < CGROUPS; ++k) v += red[k * NRED + i];
    dst[i] = v;
  }
}

template <bool SILU>
int launch_conv4_bwd(const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* w, const __nv_bfloat16* b, const int* pos,
                     __nv_bfloat16* dx, float* part, long long T, int D, long long ldx, long long ldy, long long ldd, int per, dim3 grid,
                     cudaStream_t stream) {
  constexpr int bytes = CSTAGES * (int)sizeof(ConvTile);
  static_assert(bytes >= CGROUPS * BCH * (CW + 1) * 4, "the partial sums of a block reuse the stages");
  static const cudaError_t rc = cudaFuncSetAttribute(conv4_bwd_kernel<SILU>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (rc != cudaSuccess) return (int)rc;
  conv4_bwd_kernel<SILU><<<grid, dim3(CLANES, CGROUPS), bytes, stream>>>(dy, x, w, b, pos, dx, part, T, D, ldx, ldy, ldd, per);
  return fb::launch_ok("conv4_bwd_kernel");
}

// Sums the per-strip partials in a fixed order: a block of 32 outputs x 8 strip groups reads coalesced rows of partials.
__global__ void conv_reduce_kernel(const float* __restrict__ part, int strips, int D, int W, float* __restrict__ dw,
                                   float* __restrict__ db, int accumulate) {
  __shared__ float red[8][32];
  const int n = D * (W + 1);
  const int ix = threadIdx.x & 31, ky = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + ix;
  float s = 0.f;
  if (i < n)
    for (int k = ky; k < strips; k += 8) s += part[(long long)k * n + i];
  red[ky][ix] = s;
  __syncthreads();
  if (ky != 0 || i >= n) return;
#pragma unroll
  for (int k = 1; k < 8; ++k) s += red[k][ix];
  const int d = i / (W + 1), j = i % (W + 1);
  if (j < W) {
    float* o = dw + d * W + j;
    *o = accumulate ? *o + s : s;
  } else if (db != nullptr) {
    float* o = db + d;
    *o = accumulate ? *o + s : s;
  }
}

}  // namespace

extern "C" {

// Strips of rows whose weight-gradient partials the reduction adds up: of at least 64 rows, at most 2,048 of them, and for width 4
// no more than fill the GPU once (four blocks on each of 148 SMs): 37 for 65,536 tokens and 1,024 channels.
int fb_short_conv_strips(long long T, int D, int W) {
  const long long tiles = (T + BTILE - 1) / BTILE;
  long long s = tiles < 1 ? 1 : (tiles > 2048 ? 2048 : tiles);
  if (W == CW) {
    const int blocks_x = (D + BCH - 1) / BCH;
    s = min(s, (long long)max(1, 4 * 148 / max(blocks_x, 1)));
    const long long per = max(1ll, (tiles + s - 1) / s);
    s = max(1ll, (tiles + per - 1) / per);
  }
  return (int)s;
}

int fb_short_conv_fwd(const void* x, const void* w, const void* b, const int* pos, void* y, long long T, int D, int W,
                      long long ldx, long long ldy, int silu, cudaStream_t stream) {
  if (T == 0) return 0;
  if ((D % 8) || W > MAXW || (ldx % 8) || (ldy % 8)) return -2;
  if (W == CW) {
    if (((uintptr_t)w & 15) || ((uintptr_t)b & 7) || ((uintptr_t)x & 7)) return -2;
    const dim3 grid((D / 4 + CLANES - 1) / CLANES, (unsigned)((T + FROWS * CGROUPS - 1) / (FROWS * CGROUPS))), block(CLANES, CGROUPS);
    const __nv_bfloat16 *xx = (const __nv_bfloat16*)x, *ww = (const __nv_bfloat16*)w, *bb = (const __nv_bfloat16*)b;
    if (grid.y > 65535) return -2;
    if (silu) conv4_fwd_kernel<true><<<grid, block, 0, stream>>>(xx, ww, bb, pos, (__nv_bfloat16*)y, T, D, ldx, ldy);
    else conv4_fwd_kernel<false><<<grid, block, 0, stream>>>(xx, ww, bb, pos, (__nv_bfloat16*)y, T, D, ldx, ldy);
    return fb::launch_ok("conv4_fwd_kernel");
  }
  return silu ? launch_conv_point<true, false>(x, w, b, pos, nullptr, y, T, D, W, ldx, ldy, stream)
              : launch_conv_point<false, false>(x, w, b, pos, nullptr, y, T, D, W, ldx, ldy, stream);
}

// dx: bf16 [T, D], row stride ldd (= ldx unless W is 4); dpre: bf16 [T, D] scratch with dy's row stride, not used when W is 4;
// part: fp32 [fb_short_conv_strips(T, D, W), D, W + 1] scratch; dw: fp32 [D, W]; db: fp32 [D] or null
int fb_short_conv_bwd(const void* dy, const void* x, const void* w, const void* b, const int* pos, void* dx, void* dpre,
                      float* part, float* dw, float* db, long long T, int D, int W, long long ldx, long long ldy, long long ldd, int silu,
                      int accumulate, cudaStream_t stream) {
  if (T == 0) return 0;
  if ((D % 8) || W > MAXW || (ldx % 8) || (ldy % 8) || (ldd % 8)) return -2;
  const int strips = fb_short_conv_strips(T, D, W);
  int rc;
  const __nv_bfloat16 *gg = (const __nv_bfloat16*)dy, *xx = (const __nv_bfloat16*)x, *ww = (const __nv_bfloat16*)w, *bb = (const __nv_bfloat16*)b;
  if (W == CW) {
    if (((uintptr_t)w & 15) || ((uintptr_t)b & 7) || ((uintptr_t)x & 7) || ((uintptr_t)dy & 7)) return -2;
    const long long tiles = (T + BTILE - 1) / BTILE;
    const int per = (int)((tiles + strips - 1) / strips);  // the number of strips is such that none is empty
    const dim3 grid((D + BCH - 1) / BCH, strips);
    rc = silu ? launch_conv4_bwd<true>(gg, xx, ww, bb, pos, (__nv_bfloat16*)dx, part, T, D, ldx, ldy, ldd, per, grid, stream)
              : launch_conv4_bwd<false>(gg, xx, ww, bb, pos, (__nv_bfloat16*)dx, part, T, D, ldx, ldy, ldd, per, grid, stream);
  } else {
    if (ldd != ldx) return -2;
    rc = silu ? launch_conv_point<true, true>(x, w, b, pos, dy, dpre, T, D, W, ldx, ldy, stream)
              : launch_conv_point<false, true>(x, w, b, pos, dy, dpre, T, D, W, ldx, ldy, stream);
    if (rc) return rc;
    const int rows_per_strip = (int)((T + strips - 1) / strips);
    conv_bwd_kernel<<<dim3((D / 8 + 63) / 64, strips), 64, 0, stream>>>((const __nv_bfloat16*)dpre, xx, ww, pos, (__nv_bfloat16*)dx, part, T, D,
                                                                        W, ldx, ldy, rows_per_strip);
    rc = fb::launch_ok("conv_bwd_kernel");
  }
  if (rc) return rc;
  conv_reduce_kernel<<<(D * (W + 1) + 31) / 32, 256, 0, stream>>>(part, strips, D, W, dw, db, accumulate);
  return fb::launch_ok("conv_reduce_kernel");
}

}  // extern "C"
