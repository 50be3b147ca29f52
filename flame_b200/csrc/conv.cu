// Depthwise causal short convolution (kernel width <= 8) over packed sequences, with optional bias and SiLU.
//   pre[t, d] = b[d] + sum_{j < W, j <= pos[t]} w[d, W-1-j] * x[t-j, d];   y = act(pre)
// `pos[t]` is the token's offset inside its document, so taps never reach into the previous document.
// Backward: dpre = dy * act'(pre) with pre recomputed, dx[t] = sum_j w[., W-1-j] dpre[t+j] (same document only) and partial
// sums of dw / db per strip of rows, then a fixed-order reduction of the partials.  Width 4 (every configuration's) does
// the first three in one kernel and never stores dpre; the other widths take a dpre pass and a strip pass.
// Semantics of fla/modules/conv/triton/kernels.py:37-345; the row-strip partial reduction replaces its atomics.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include "host_utils.cuh"
#include "tc05.cuh"

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

// Width 4.  Both directions move each row once, so what should bound them is memory; what did was instructions (21 and 55 per
// element, 0.078 and 0.158 ms at 65,536 x 1,024, 38 % and 29 % of the memory's rate).  So: a warp owns 64 channels of a strip
// of rows, two channels per lane as packed fp32 pairs, and walks it with the last three rows in registers.  dpre, which the gradient of
// a row needs from the three rows behind it, is formed once too: dx lags three rows.  Only the three rows in front of a strip are
// read twice, and in the backward those behind it, with their dpre.  The rows come
// by TMA (no address arithmetic), each warp through a ring of its own: there is no barrier in the walk.
//
// Rows may be taken in a padded order (`src`): the chunk layout of the linear-attention kernels, where every document starts on
// a chunk boundary.  Tiles of 16 rows divide a chunk, so a tile's rows follow one another in both orders; the forward then
// writes its result there (zeros where a document is padded), the backward reads its gradient from there, and no pass
// gathers rows in between.
constexpr int CW = 4;          // taps
constexpr int H3 = CW - 1;
constexpr int BCH = 64;        // channels of a warp
constexpr int WARPS = 4;       // of a block: consecutive strips of the same channels
constexpr int MAXPART = 3;     // convolutions of one launch
constexpr int NO_ROW = -(1 << 20);  // position of a row that is padding (a halo row in front of a document has a small negative one)
// Rows of a tile, stages of the ring, blocks per SM.  At 65,536 x 1,024 on the device, forward 0.072 -> 0.055 ms and backward 0.158 ->
// 0.091 ms (the copy of 268 MB takes 0.049); tiles of 8 rows took 0.061 and 0.120, of 32 rows 0.063 (host included).  The warps
// still wait for the special function unit (two results per element, 63 % busy in the forward) and for one another's issue.
constexpr int FROWS = 16, FSTAGES = 3, FOCC = 6;
constexpr int BROWS = 16, BSTAGES = 2, BOCC = 4;

struct ConvPart {
  const __nv_bfloat16 *x, *g, *w, *b;  // g: dy (backward)
  __nv_bfloat16* out;                  // y or dx
  long long ldx, ldg, ldo;
  int D, block0;                       // channels, first block along x
};
struct ConvArgs {
  ConvPart part[MAXPART];
  int parts, rows, per, D;  // rows to walk (padded ones included), tiles of a strip, all channels
  const int* src;           // [rows] packed row of a padded row (-1: padding); null: the rows themselves
  const int* pos;           // [T] offset of a packed row in its document
  float* partial;           // [blocks along y][D][W + 1]
  long long T;              // rows of x
  int* status;
};
struct ConvMaps {
  CUtensorMap x[MAXPART], g[MAXPART];
};

// Two fp32 values per instruction (sm_100).
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
__device__ __forceinline__ f2 f2_all(float a) { return f2_make(a, a); }
__device__ __forceinline__ f2 f2_sigmoid(f2 z) {
  const float2 e = f2_get(f2_mul(z, f2_all(-1.4426950408889634f)));
  const float2 d = f2_get(f2_add(f2_make(exp2f(e.x), exp2f(e.y)), f2_all(1.f)));
  return f2_make(1.f / d.x, 1.f / d.y);
}
__device__ __forceinline__ uint32_t f2_pack(f2 v) {
  const float2 a = f2_get(v);
  return tc05::pack_bf16(a.x, a.y);
}

// The ring of one warp: BUFS tiles of ROWS rows x 64 channels per stage.
template <int ROWS, int STAGES, int BUFS>
struct ConvRing {
  uint32_t data[STAGES][BUFS][ROWS][BCH / 2];
};
template <int ROWS, int STAGES, int BUFS>
struct ConvSmem {
  ConvRing<ROWS, STAGES, BUFS> ring[WARPS];
  uint64_t full[WARPS][STAGES];
  int abort_flag;
};

// What both directions share: which strip, the ring, and the packed row of every tile, read 32 tiles at a time.
template <int ROWS, int STAGES, int BUFS>
struct ConvWalk {
  const ConvArgs& a;
  const CUtensorMap *mx, *mg;
  ConvRing<ROWS, STAGES, BUFS>& ring;
  uint64_t* full;
  volatile int* abort_flag;
  int lane, c0, tiles, k0, k1, batch0, batch;  // tiles [k0, k1) are this warp's; `batch`: this lane's of batch0 ...

  __device__ __forceinline__ void load_batch(int k) {
    batch0 = k;
    const int t = k + lane;
    batch = t >= tiles ? -1 : a.src == nullptr ? t * ROWS : a.src[t * ROWS];
  }
  // packed row of a tile's first row, -1 where the whole tile is padding (or there is none): k does not decrease
  __device__ __forceinline__ int row_of(int k) {
    if (k - batch0 >= 32) load_batch(k);
    return __shfl_sync(0xffffffffu, batch, k - batch0);
  }
  // lane i: position of the i-th packed row from s on.  A padded tile whose first row is s holds those that follow it in its document, which
  // `in_tile` tells by the positions alone (and only when they are needed: it waits for them).
  __device__ __forceinline__ int pos_of(int s) const {
    const long long r = (long long)s + lane;
    return s >= 0 && lane < ROWS && r < a.T ? a.pos[r] : NO_ROW;
  }
  __device__ __forceinline__ int in_tile(int p) const {
    return a.src == nullptr || p == __shfl_sync(0xffffffffu, p, 0) + lane ? p : NO_ROW;
  }
  __device__ __forceinline__ void fetch(int k, int s) {  // row s of x (and the tile of g) into the ring
    if (k < k1 && s >= 0 && lane == 0) {
      const int st = (k - k0) % STAGES;
      tc05::mbar_expect_tx(&full[st], BUFS * ROWS * BCH * 2);
      tc05::tma_load_2d(&ring.data[st][0][0][0], mx, &full[st], c0, s);
      if (BUFS == 2) tc05::tma_load_2d(&ring.data[st][BUFS - 1][0][0], mg, &full[st], c0, k * ROWS);
    }
  }
};

__device__ __forceinline__ void load_taps2(const ConvPart& p, int d0, bool live, f2 (&wv)[CW], f2& bias) {
  bias = 0ull;
#pragma unroll
  for (int j = 0; j < CW; ++j) wv[j] = 0ull;
  if (!live) return;
  float f[8];
  unpack8(*reinterpret_cast<const uint4*>(p.w + (long long)d0 * CW), f);
#pragma unroll
  for (int j = 0; j < CW; ++j) wv[j] = f2_make(f[CW - 1 - j], f[CW + CW - 1 - j]);  // tap at distance j
  if (p.b != nullptr) bias = f2_unpack2(*reinterpret_cast<const uint32_t*>(p.b + d0));
}

template <bool SILU>
__global__ void __launch_bounds__(32 * WARPS, FOCC) conv4_fwd_kernel(const __grid_constant__ ConvMaps maps, const __grid_constant__ ConvArgs a) {
  using Sm = ConvSmem<FROWS, FSTAGES, 1>;
  extern __shared__ __align__(128) uint8_t conv_smem[];
  Sm& sm = *reinterpret_cast<Sm*>(conv_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int pi = 0;
  while (pi + 1 < a.parts && (int)blockIdx.x >= a.part[pi + 1].block0) ++pi;
  const ConvPart& p = a.part[pi];
  const int c0 = ((int)blockIdx.x - p.block0) * BCH, d0 = c0 + 2 * lane;
  const bool live = d0 < p.D;
  if (lane == 0)
    for (int s = 0; s < FSTAGES; ++s) tc05::mbar_init(&sm.full[warp][s], 1);
  if (threadIdx.x == 0) sm.abort_flag = 0;
  tc05::mbar_fence_init();
  __syncthreads();

  ConvWalk<FROWS, FSTAGES, 1> w{a, &maps.x[pi], nullptr, sm.ring[warp], sm.full[warp], &sm.abort_flag, lane, c0, (a.rows + FROWS - 1) / FROWS};
  w.k0 = min(w.tiles, ((int)blockIdx.y * WARPS + warp) * a.per);
  w.k1 = min(w.tiles, w.k0 + a.per);
  if (w.k0 == w.k1) return;
  w.load_batch(w.k0);
  int row[FSTAGES];  // packed rows of the tiles on their way
#pragma unroll
  for (int s = 0; s < FSTAGES; ++s) {
    row[s] = w.row_of(w.k0 + s);
    w.fetch(w.k0 + s, row[s]);
  }
  f2 wv[CW], bias, xv[CW];  // x of the last rows, [0] the newest
  load_taps2(p, d0, live, wv, bias);
  int pos_l = w.in_tile(w.pos_of(row[0]));
#pragma unroll
  for (int j = 0; j < H3; ++j) {
    const bool in = live && row[0] - 1 - j >= 0;
    xv[j] = in ? f2_unpack2(*reinterpret_cast<const uint32_t*>(p.x + (long long)(row[0] - 1 - j) * p.ldx + d0)) : 0ull;
  }
  xv[H3] = 0ull;
  int stage = 0, phase = 0;
  for (int k = w.k0; k < w.k1; ++k) {
    const int pos_next = w.pos_of(row[1]);
    const uint32_t* xs = &w.ring.data[stage][0][0][lane];
    __nv_bfloat16* out = p.out + (long long)k * FROWS * p.ldo + d0;
    const int src = row[0];
    if (src >= 0 && !tc05::mbar_wait_warp(&w.full[stage], (phase >> stage) & 1, a.status, w.abort_flag, tc05::ERR_WAIT_FULL)) break;
    if (src >= 0) phase ^= 1 << stage;
    // straight-line code where every tap of every row lies in the row's document (the same for the whole warp)
    if (__all_sync(0xffffffffu, lane >= FROWS || pos_l >= H3)) {
#pragma unroll
      for (int i = 0; i < FROWS; ++i) {
#pragma unroll
        for (int j = CW - 1; j >= 1; --j) xv[j] = xv[j - 1];
        xv[0] = f2_unpack2(xs[i * (BCH / 2)]);
        f2 acc = f2_fma(wv[0], xv[0], bias);
#pragma unroll
        for (int j = 1; j < CW; ++j) acc = f2_fma(wv[j], xv[j], acc);
        if (SILU) acc = f2_mul(acc, f2_sigmoid(acc));
        if (live) *reinterpret_cast<uint32_t*>(out) = f2_pack(acc);
        out += p.ldo;
      }
    } else {
#pragma unroll 4
      for (int i = 0; i < FROWS; ++i) {
        const int q = __shfl_sync(0xffffffffu, pos_l, i);
#pragma unroll
        for (int j = CW - 1; j >= 1; --j) xv[j] = xv[j - 1];
        uint32_t y = 0;
        if (q != NO_ROW) {
          xv[0] = f2_unpack2(xs[i * (BCH / 2)]);
          f2 acc = bias;
#pragma unroll
          for (int j = 0; j < CW; ++j)
            if (j <= q) acc = f2_fma(wv[j], xv[j], acc);
          if (SILU) acc = f2_mul(acc, f2_sigmoid(acc));
          y = f2_pack(acc);
        }
        if (live && (long long)k * FROWS + i < a.rows) *reinterpret_cast<uint32_t*>(out) = y;
        out += p.ldo;
      }
    }
    __syncwarp();  // the stage is free
#pragma unroll
    for (int s = 0; s + 1 < FSTAGES; ++s) row[s] = row[s + 1];
    row[FSTAGES - 1] = w.row_of(k + FSTAGES);
    w.fetch(k + FSTAGES, row[FSTAGES - 1]);
    pos_l = w.in_tile(pos_next);
    stage = stage + 1 == FSTAGES ? 0 : stage + 1;
  }
}

template <bool SILU>
__global__ void __launch_bounds__(32 * WARPS, BOCC) conv4_bwd_kernel(const __grid_constant__ ConvMaps maps, const __grid_constant__ ConvArgs a) {
  using Sm = ConvSmem<BROWS, BSTAGES, 2>;
  extern __shared__ __align__(128) uint8_t conv_smem[];
  Sm& sm = *reinterpret_cast<Sm*>(conv_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int pi = 0, ch = 0;  // ch: channels of the convolutions before this one
  while (pi + 1 < a.parts && (int)blockIdx.x >= a.part[pi + 1].block0) ch += a.part[pi++].D;
  const ConvPart& p = a.part[pi];
  const int c0 = ((int)blockIdx.x - p.block0) * BCH, d0 = c0 + 2 * lane;
  const bool live = d0 < p.D;
  if (lane == 0)
    for (int s = 0; s < BSTAGES; ++s) tc05::mbar_init(&sm.full[warp][s], 1);
  if (threadIdx.x == 0) sm.abort_flag = 0;
  tc05::mbar_fence_init();
  __syncthreads();

  ConvWalk<BROWS, BSTAGES, 2> w{a, &maps.x[pi], &maps.g[pi], sm.ring[warp], sm.full[warp], &sm.abort_flag, lane, c0, (a.rows + BROWS - 1) / BROWS};
  w.k0 = min(w.tiles, ((int)blockIdx.y * WARPS + warp) * a.per);
  w.k1 = min(w.tiles, w.k0 + a.per);
  f2 dw[CW], db = 0ull;
#pragma unroll
  for (int j = 0; j < CW; ++j) dw[j] = 0ull;
  if (w.k0 < w.k1) {
    w.load_batch(w.k0);
    int row[BSTAGES];  // packed rows of the tiles on their way
#pragma unroll
    for (int s = 0; s < BSTAGES; ++s) {
      row[s] = w.row_of(w.k0 + s);
      w.fetch(w.k0 + s, row[s]);
    }
    f2 wv[CW], bias, xv[CW], g[CW];  // x and dpre of the last four rows, [0] the newest
    int q[CW];                       // their positions
    load_taps2(p, d0, live, wv, bias);
#pragma unroll
    for (int j = 0; j < CW; ++j) g[j] = 0ull, q[j] = NO_ROW;
    int pos_l = w.in_tile(w.pos_of(row[0]));
#pragma unroll
    for (int j = 0; j < H3; ++j) {
      const bool in = live && row[0] - 1 - j >= 0;
      xv[j] = in ? f2_unpack2(*reinterpret_cast<const uint32_t*>(p.x + (long long)(row[0] - 1 - j) * p.ldx + d0)) : 0ull;
    }
    xv[H3] = 0ull;
    int stage = 0, phase = 0, before = -1;  // before: the packed row of the tile before
    auto dpre = [&](f2 dy, f2 pre) {
      if (!SILU) return dy;
      const f2 s = f2_sigmoid(pre);
      const f2 t = f2_fma(pre, f2_fma(s, f2_all(-1.f), f2_all(1.f)), f2_all(1.f));
      return f2_mul(f2_mul(dy, s), t);
    };
    // one row whose document may begin or end nearby; `own`: its products belong to this strip's sums
    auto edge_row = [&](uint32_t xr, uint32_t gr, int pos, bool own, __nv_bfloat16* out) {
#pragma unroll
      for (int j = CW - 1; j >= 1; --j) g[j] = g[j - 1], xv[j] = xv[j - 1], q[j] = q[j - 1];
      q[0] = pos;
      g[0] = 0ull;
      if (pos != NO_ROW) {
        xv[0] = f2_unpack2(xr);
        f2 pre = bias;
#pragma unroll
        for (int j = 0; j < CW; ++j)
          if (j <= pos) pre = f2_fma(wv[j], xv[j], pre);
        g[0] = dpre(f2_unpack2(gr), pre);
        if (own) {
          db = f2_add(db, g[0]);
#pragma unroll
          for (int j = 0; j < CW; ++j)
            if (j <= pos) dw[j] = f2_fma(g[0], xv[j], dw[j]);
        }
      }
      if (q[H3] != NO_ROW) {
        // dx[s] = sum_j w[tap j] dpre[s + j] while row s + j is at least j tokens into its document
        f2 acc = f2_mul(wv[0], g[H3]);
        bool alive = true;
#pragma unroll
        for (int j = 1; j < CW; ++j) {
          alive = alive && q[H3 - j] >= j;
          if (alive) acc = f2_fma(wv[j], g[H3 - j], acc);
        }
        if (live) *reinterpret_cast<uint32_t*>(out) = f2_pack(acc);
      }
    };
    int k = w.k0;
    for (; k < w.k1; ++k) {
      const int pos_next = w.pos_of(row[1]);
      const uint32_t *xs = &w.ring.data[stage][0][0][lane], *gs = &w.ring.data[stage][1][0][lane];
      const int src = row[0];
      if (src >= 0 && !tc05::mbar_wait_warp(&w.full[stage], (phase >> stage) & 1, a.status, w.abort_flag, tc05::ERR_WAIT_FULL)) break;
      if (src >= 0) phase ^= 1 << stage;
      // straight-line code where every tap of every row lies in the row's document (the same for the whole warp)
      if (__all_sync(0xffffffffu, lane >= BROWS || pos_l >= H3)) {
        __nv_bfloat16* out = p.out + (long long)(src - H3) * p.ldo + d0;
        const bool first = k == w.k0;  // the three rows before belong to another strip
#pragma unroll
        for (int i = 0; i < BROWS; ++i) {
#pragma unroll
          for (int j = CW - 1; j >= 1; --j) g[j] = g[j - 1], xv[j] = xv[j - 1];
          xv[0] = f2_unpack2(xs[i * (BCH / 2)]);
          g[0] = f2_unpack2(gs[i * (BCH / 2)]);
          if (SILU) {
            f2 pre = f2_fma(wv[0], xv[0], bias);
#pragma unroll
            for (int j = 1; j < CW; ++j) pre = f2_fma(wv[j], xv[j], pre);
            g[0] = dpre(g[0], pre);
          }
          db = f2_add(db, g[0]);
#pragma unroll
          for (int j = 0; j < CW; ++j) dw[j] = f2_fma(g[0], xv[j], dw[j]);
          f2 acc = f2_mul(wv[0], g[H3]);
#pragma unroll
          for (int j = 1; j < CW; ++j) acc = f2_fma(wv[j], g[H3 - j], acc);
          if (live && (i >= H3 || !first)) *reinterpret_cast<uint32_t*>(out) = f2_pack(acc);
          out += p.ldo;
        }
#pragma unroll
        for (int j = 0; j < CW; ++j) q[j] = H3;  // any position of at least three
      } else {
#pragma unroll 4
        for (int i = 0; i < BROWS; ++i) {
          const int row_out = i >= H3 ? src + i - H3 : before + BROWS + i - H3;
          edge_row(xs[i * (BCH / 2)], gs[i * (BCH / 2)], __shfl_sync(0xffffffffu, pos_l, i), true, p.out + (long long)row_out * p.ldo + d0);
        }
      }
      __syncwarp();  // the stage is free
      before = src;
#pragma unroll
      for (int s = 0; s + 1 < BSTAGES; ++s) row[s] = row[s + 1];
      row[BSTAGES - 1] = w.row_of(k + BSTAGES);
      w.fetch(k + BSTAGES, row[BSTAGES - 1]);
      pos_l = w.in_tile(pos_next);
      stage = stage + 1 == BSTAGES ? 0 : stage + 1;
    }
    if (k == w.k1) {  // the three rows behind the strip, for the gradients of its last three
      const int src = row[0];
#pragma unroll
      for (int i = 0; i < H3; ++i) {
        const int pos = __shfl_sync(0xffffffffu, pos_l, i);
        uint32_t xr = 0, gr = 0;
        if (live && pos != NO_ROW) {
          xr = *reinterpret_cast<const uint32_t*>(p.x + (long long)(src + i) * p.ldx + d0);
          gr = *reinterpret_cast<const uint32_t*>(p.g + ((long long)k * BROWS + i) * p.ldg + d0);
        }
        edge_row(xr, gr, pos, false, p.out + (long long)(before + BROWS + i - H3) * p.ldo + d0);
      }
    }
  }
  __syncthreads();  // the rings are done with
  float* red = reinterpret_cast<float*>(conv_smem);  // [WARPS][BCH * (CW + 1)]
  constexpr int NRED = BCH * (CW + 1);
  float* mine = red + warp * NRED + lane * 2 * (CW + 1);
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
  const int n = min(BCH, p.D - c0) * (CW + 1);
  float* dst = a.partial + ((long long)blockIdx.y * a.D + ch + c0) * (CW + 1);
  for (int i = threadIdx.x; i < n; i += 32 * WARPS) {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < WARPS; ++k) v += red[k * NRED + i];
    dst[i] = v;
  }
}

struct ConvSums {
  float *dw[MAXPART], *db[MAXPART];
  int D[MAXPART];
};
// Sums the per-strip partials in a fixed order: a block of 32 outputs x 8 strip groups reads coalesced rows of partials.
__global__ void conv_reduce_kernel(const float* __restrict__ part, int strips, int D, int W, const ConvSums to, int accumulate) {
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
  int d = i / (W + 1), pi = 0;
  const int j = i % (W + 1);
  while (d >= to.D[pi]) d -= to.D[pi++];
  float* o = j < W ? to.dw[pi] + d * W + j : to.db[pi];
  if (o == nullptr) return;
  if (j == W) o += d;
  *o = accumulate ? *o + s : s;
}


// Strips of the width-4 kernels along the rows (blocks of WARPS each): no more than fill the GPU once.
int strip_blocks(int rows, int tile, int blocks_x, int per_sm, int* per) {
  const int tiles = (rows + tile - 1) / tile;
  const int most = max(1, per_sm * 148 / max(blocks_x, 1));
  const int blocks = max(1, min((tiles + WARPS - 1) / WARPS, most));
  *per = (tiles + blocks * WARPS - 1) / (blocks * WARPS);
  return (tiles + *per * WARPS - 1) / (*per * WARPS);
}
int blocks_x(int parts, const long long* table, int stride, int at) {
  int n = 0;
  for (int i = 0; i < parts; ++i) n += ((int)table[i * stride + at] + BCH - 1) / BCH;
  return n;
}

constexpr int FWD_ENTRIES = 7, BWD_ENTRIES = 11;

template <class Kernel, class Sm>
int launch_walk(Kernel kernel, dim3 grid, const ConvMaps& maps, const ConvArgs& a, cudaStream_t stream, const char* name) {
  // per call and thread-safe: the attribute belongs to the device, of which a process may use several
  const cudaError_t rc = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Sm));
  if (rc != cudaSuccess) return (int)rc;
  kernel<<<grid, 32 * WARPS, sizeof(Sm), stream>>>(maps, a);
  return fb::launch_ok(name);
}

}  // namespace

extern "C" {

// Strips of rows whose weight-gradient partials the reduction adds up: of at least 64 rows, at most 2,048 of them.
int fb_short_conv_strips(long long T, int D, int W) {
  const long long tiles = (T + 63) / 64;
  return (int)(tiles < 1 ? 1 : (tiles > 2048 ? 2048 : tiles));
}
int fb_short_conv4_strips(int parts, const long long* table, int rows) {
  int per;
  return strip_blocks(rows, BROWS, blocks_x(parts, table, BWD_ENTRIES, 7), BOCC, &per);
}

// Width 4: up to three convolutions of the same rows.  table: per convolution x, w, b (or 0), y, D, ldx, ldy.  rows: of y; src, pos:
// see ConvArgs; T: rows of x.
int fb_short_conv4_fwd(int parts, const long long* table, int rows, const int* src, const int* pos, long long T, int silu, cudaStream_t stream) {
  if (rows == 0) return 0;
  if (parts < 1 || parts > MAXPART) return -2;
  ConvMaps maps;
  ConvArgs a{};
  a.parts = parts, a.rows = rows, a.src = src, a.pos = pos, a.T = T, a.status = fb::status_ptr();
  int block0 = 0;
  for (int i = 0; i < parts; ++i) {
    const long long* t = table + i * FWD_ENTRIES;
    ConvPart& p = a.part[i];
    p.x = (const __nv_bfloat16*)t[0], p.w = (const __nv_bfloat16*)t[1], p.b = (const __nv_bfloat16*)t[2], p.out = (__nv_bfloat16*)t[3];
    p.D = (int)t[4], p.ldx = t[5], p.ldo = t[6], p.block0 = block0;
    if ((p.D % 8) || (p.ldx % 8) || (p.ldo % 2) || !fb::aligned(16, p.x, p.w) || !fb::aligned(4, p.b, p.out)) return -2;
    if (int rc = fb::make_tmap_2d(&maps.x[i], p.x, 2, (uint64_t)T, p.D, p.ldx, FROWS, BCH, false)) return rc;
    block0 += (p.D + BCH - 1) / BCH;
  }
  const dim3 grid(block0, strip_blocks(rows, FROWS, block0, FOCC, &a.per));
  using Sm = ConvSmem<FROWS, FSTAGES, 1>;
  return silu ? launch_walk<decltype(&conv4_fwd_kernel<true>), Sm>(conv4_fwd_kernel<true>, grid, maps, a, stream, "conv4_fwd_kernel")
              : launch_walk<decltype(&conv4_fwd_kernel<false>), Sm>(conv4_fwd_kernel<false>, grid, maps, a, stream, "conv4_fwd_kernel");
}

// table: per convolution x, dy, w, b (or 0), dx, dw, db (or 0), D, ldx, ldy, lddx; dy has `rows` rows, dx T.  partial: fp32
// [fb_short_conv4_strips, channels of all, W + 1] scratch; dw: fp32 [D, W]; db: fp32 [D] or null
int fb_short_conv4_bwd(int parts, const long long* table, int rows, const int* src, const int* pos, float* partial, long long T, int silu,
                       int accumulate, cudaStream_t stream) {
  if (rows == 0) return 0;
  if (parts < 1 || parts > MAXPART) return -2;
  ConvMaps maps;
  ConvArgs a{};
  ConvSums to{};
  a.parts = parts, a.rows = rows, a.src = src, a.pos = pos, a.T = T, a.partial = partial, a.status = fb::status_ptr();
  int block0 = 0;
  for (int i = 0; i < parts; ++i) {
    const long long* t = table + i * BWD_ENTRIES;
    ConvPart& p = a.part[i];
    p.x = (const __nv_bfloat16*)t[0], p.g = (const __nv_bfloat16*)t[1], p.w = (const __nv_bfloat16*)t[2], p.b = (const __nv_bfloat16*)t[3];
    p.out = (__nv_bfloat16*)t[4], to.dw[i] = (float*)t[5], to.db[i] = (float*)t[6];
    p.D = to.D[i] = (int)t[7], p.ldx = t[8], p.ldg = t[9], p.ldo = t[10], p.block0 = block0;
    if ((p.D % 8) || (p.ldx % 8) || (p.ldg % 8) || (p.ldo % 2) || !fb::aligned(16, p.x, p.g, p.w) || !fb::aligned(4, p.b, p.out)) return -2;
    if (int rc = fb::make_tmap_2d(&maps.x[i], p.x, 2, (uint64_t)T, p.D, p.ldx, BROWS, BCH, false)) return rc;
    if (int rc = fb::make_tmap_2d(&maps.g[i], p.g, 2, (uint64_t)rows, p.D, p.ldg, BROWS, BCH, false)) return rc;
    block0 += (p.D + BCH - 1) / BCH;
    a.D += p.D;
  }
  const int strips = strip_blocks(rows, BROWS, block0, BOCC, &a.per);
  const dim3 grid(block0, strips);
  using Sm = ConvSmem<BROWS, BSTAGES, 2>;
  static_assert(sizeof(Sm) >= WARPS * BCH * (CW + 1) * 4, "the partial sums of a block reuse the rings");
  const int rc = silu ? launch_walk<decltype(&conv4_bwd_kernel<true>), Sm>(conv4_bwd_kernel<true>, grid, maps, a, stream, "conv4_bwd_kernel")
                      : launch_walk<decltype(&conv4_bwd_kernel<false>), Sm>(conv4_bwd_kernel<false>, grid, maps, a, stream, "conv4_bwd_kernel");
  if (rc) return rc;
  conv_reduce_kernel<<<(a.D * (CW + 1) + 31) / 32, 256, 0, stream>>>(partial, strips, a.D, CW, to, accumulate);
  return fb::launch_ok("conv_reduce_kernel");
}

int fb_short_conv_fwd(const void* x, const void* w, const void* b, const int* pos, void* y, long long T, int D, int W,
                      long long ldx, long long ldy, int silu, cudaStream_t stream) {
  if (T == 0) return 0;
  if ((D % 8) || W > MAXW || W == CW || (ldx % 8) || (ldy % 8)) return -2;
  return silu ? launch_conv_point<true, false>(x, w, b, pos, nullptr, y, T, D, W, ldx, ldy, stream)
              : launch_conv_point<false, false>(x, w, b, pos, nullptr, y, T, D, W, ldx, ldy, stream);
}

// dx: bf16 [T, D], row stride ldx; dpre: bf16 [T, D] scratch with dy's row stride; part: fp32 [fb_short_conv_strips(T, D, W), D,
// W + 1] scratch; dw: fp32 [D, W]; db: fp32 [D] or null
int fb_short_conv_bwd(const void* dy, const void* x, const void* w, const void* b, const int* pos, void* dx, void* dpre,
                      float* part, float* dw, float* db, long long T, int D, int W, long long ldx, long long ldy, int silu,
                      int accumulate, cudaStream_t stream) {
  if (T == 0) return 0;
  if ((D % 8) || W > MAXW || W == CW || (ldx % 8) || (ldy % 8)) return -2;
  const int strips = fb_short_conv_strips(T, D, W);
  const __nv_bfloat16 *xx = (const __nv_bfloat16*)x, *ww = (const __nv_bfloat16*)w;
  int rc = silu ? launch_conv_point<true, true>(x, w, b, pos, dy, dpre, T, D, W, ldx, ldy, stream)
                : launch_conv_point<false, true>(x, w, b, pos, dy, dpre, T, D, W, ldx, ldy, stream);
  if (rc) return rc;
  const int rows_per_strip = (int)((T + strips - 1) / strips);
  conv_bwd_kernel<<<dim3((D / 8 + 63) / 64, strips), 64, 0, stream>>>((const __nv_bfloat16*)dpre, xx, ww, pos, (__nv_bfloat16*)dx, part, T, D,
                                                                      W, ldx, ldy, rows_per_strip);
  rc = fb::launch_ok("conv_bwd_kernel");
  if (rc) return rc;
  ConvSums to{};
  to.dw[0] = dw, to.db[0] = db, to.D[0] = D;
  conv_reduce_kernel<<<(D * (W + 1) + 31) / 32, 256, 0, stream>>>(part, strips, D, W, to, accumulate);
  return fb::launch_ok("conv_reduce_kernel");
}

}  // extern "C"
