// Mamba-1 selective scan, forward and backward, chunk-parallel (state size N = 16), on packed tokens.
//
//   h_t[d, n] = exp(delta_t[d] A[d, n]) h_{t-1}[d, n] + delta_t[d] B_t[n] u_t[d],     y_t[d] = sum_n h_t[d, n] C_t[n] + D[d] u_t[d]
//
// Optionally delta = softplus(raw) with raw in bf16, and the output is y * silu(z): what stands around the scan in the layer.
// A chunk is up to 64 consecutive tokens of one document: chunk c starts at token inv[64 c] and holds as many tokens as
// inv[64 c ..] has entries >= 0, so operands are read where the projections left them.  Steps past the end run with
// delta = u = dy = 0, which leaves state and adjoint untouched.
//   forward:  (1) chunk-local end state from a zero start and the chunk's sum of delta (its decay is exp(A sum))
//             (2) carry across the chunks of each document: h_in[c+1] = P[c] h_in[c] + h_loc[c]
//             (3) outputs from the true chunk-start state; the states at steps 0, 16, 32, 48 are kept for the backward
//   backward: (4) chunk-local adjoint of the chunk-start state, (5) reverse carry, (6) all gradients, 16 steps at a time.
// Replaces the sequential loop of fla/layers/mamba.py:361-397 (the reference's fast path, mamba_ssm's CUDA scan, is not
// installed in the reference environment).
//
// What bounds it: one exponential per state element and sweep, 16 MUFU results per clock and SM: 0.24 ms per sweep at 32,768
// tokens x 2,048 channels; the forward needs two sweeps, the backward three.  Everything else has to stay below that in
// issue slots: sweeps (1), (3), (4) give a thread a whole channel (16 states, B / C read as float4 broadcasts, no
// shuffles), sweep (6) gives it 2 channels x 4 states, so that the sums over states and over channels are mostly
// additions in registers, finished through shared memory; pairs of states use the packed fp32x2 instructions.  Every
// sweep fetches its operands a group of four steps ahead: waiting for memory at each group, not the MUFU, set the pace before.
// At that size with gate and softplus, before and after: (1) 0.44 -> 0.31 ms, (3) 0.84 -> 0.47, (4) 0.59 -> 0.36,
// (6) 2.17 -> 1.63.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "host_utils.cuh"

namespace {

constexpr int N = 16;        // state size
constexpr int L = 64;        // chunk length
constexpr int SEG = 16;      // steps between kept states
constexpr int NSEG = L / SEG;
constexpr int CT = 128;      // sweeps (1), (3), (4): threads = channels per block
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;

struct ScanArgs {
  const __nv_bfloat16* u;  // [T, Di], row stride us
  const void* dl;          // delta fp32 or raw bf16 [T, Di], row stride ds
  const __nv_bfloat16* z;  // gate [T, Di], row stride zs, or null
  const void* B;           // [T, N], row stride bs, bf16 or fp32
  const void* C;           // [T, N], row stride cs
  const float* A;          // [Di, N]
  const float* Dv;         // [Di]
  const int* inv;          // [64 NC]: token of every chunk step, -1 = past the end
  int us, ds, zs, bs, cs;
  int Di, DiP, bc16;       // DiP: Di rounded up to 128, the row length of the state arrays
  int kept;                // states kept per chunk: NSEG, or 1 where no backward follows
};

// two fp32 lanes per instruction
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void up(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 ex2v(f2 v) {
  float a, b;
  up(v, a, b);
  return pk(exp2f(a), exp2f(b));
}
__device__ __forceinline__ float sum2(f2 v) {
  float a, b;
  up(v, a, b);
  return a + b;
}
struct alignas(16) F4 { f2 a, b; };

__device__ __forceinline__ float sigm(float x) { return 1.f / (1.f + __expf(-x)); }
// max(x, 0) + log(1 + e), e = exp(-|x|) <= 1, by log(1 + e) = 2 artanh(e / (2 + e)) with the artanh series up to s^13, s <= 1/3:
// relative error below 1e-7 plus rounding also where e is tiny (log(1 + e) itself would round 1 + e first)
__device__ __forceinline__ float softplus(float x) {
  const float e = __expf(-fabsf(x));
  const float s = __fdividef(e, 2.f + e), w = s * s;
  float p = fmaf(w, 1.f / 13.f, 1.f / 11.f);
  p = fmaf(p, w, 1.f / 9.f);
  p = fmaf(p, w, 1.f / 7.f);
  p = fmaf(p, w, 1.f / 5.f);
  p = fmaf(p, w, 1.f / 3.f);
  p = fmaf(p, w, 1.f);
  return fmaf(2.f * s, p, fmaxf(x, 0.f));
}

__device__ __forceinline__ float load_bc(const ScanArgs& a, const void* p, int stride, long long row, int n) {
  return a.bc16 ? __bfloat162float(((const __nv_bfloat16*)p)[row * stride + n]) : ((const float*)p)[row * stride + n];
}

// token of the chunk's first step and its number of steps (1..64)
__device__ __forceinline__ void chunk_rows(const ScanArgs& a, int c, long long& row0, int& len) {
  const int* iv = a.inv + (long long)c * L;
  row0 = iv[0];
  const int lane = threadIdx.x & 31;
  len = __popc(__ballot_sync(0xffffffffu, iv[lane] >= 0)) + __popc(__ballot_sync(0xffffffffu, iv[32 + lane] >= 0));
}

__device__ __forceinline__ void stage_bc(const ScanArgs& a, const void* p, int stride, long long row0, int len, float* s) {
  for (int i = threadIdx.x; i < L * N; i += CT) s[i] = (i / N) < len ? load_bc(a, p, stride, row0 + i / N, i % N) : 0.f;
}

__device__ __forceinline__ void load_A(const ScanArgs& a, int d, bool live, f2* A2) {
#pragma unroll
  for (int p = 0; p < N / 4; ++p) {
    const float4 v = live ? reinterpret_cast<const float4*>(a.A + (long long)d * N)[p] : make_float4(0.f, 0.f, 0.f, 0.f);
    A2[2 * p] = pk(v.x * LOG2E, v.y * LOG2E);
    A2[2 * p + 1] = pk(v.z * LOG2E, v.w * LOG2E);
  }
}

// A channel's column of a row-major operand, starting at the chunk's first token; rows by 32-bit offsets.  Loads and
// conversions are apart: the loads go out together, a group of steps ahead of their use (ncu on the form that loaded a group
// right before its use: 10 of 16 stall cycles per issue on these loads, the exponential pipe at 0.33 to 0.60 of its peak), and
// as read-only loads they may pass the kernels' stores.
typedef unsigned short u16;
__device__ __forceinline__ float bf(u16 v) { return __uint_as_float((uint32_t)v << 16); }
struct Col16 {
  const u16* p;
  int stride;
  __device__ __forceinline__ Col16(const __nv_bfloat16* base, long long row0, int stride_, int d)
      : p(reinterpret_cast<const u16*>(base) + row0 * stride_ + d), stride(stride_) {}
  __device__ __forceinline__ u16 operator()(int t, bool ok) const { return ok ? __ldg(p + t * stride) : (u16)0; }
};
template <bool RAW>
struct DeltaCol;
template <>
struct DeltaCol<true> {
  typedef u16 T;
  Col16 c;
  __device__ __forceinline__ DeltaCol(const ScanArgs& a, long long row0, int d) : c((const __nv_bfloat16*)a.dl, row0, a.ds, d) {}
  __device__ __forceinline__ T operator()(int t, bool ok) const { return c(t, ok); }
  static __device__ __forceinline__ float value(T v, bool ok) { return ok ? softplus(bf(v)) : 0.f; }
};
template <>
struct DeltaCol<false> {
  typedef float T;
  const float* p;
  int stride;
  __device__ __forceinline__ DeltaCol(const ScanArgs& a, long long row0, int d) : p((const float*)a.dl + row0 * a.ds + d), stride(a.ds) {}
  __device__ __forceinline__ T operator()(int t, bool ok) const { return ok ? __ldg(p + t * stride) : 0.f; }
  static __device__ __forceinline__ float value(T v, bool) { return v; }
};

constexpr int PF = 4;  // steps whose operands are fetched together, one group ahead

// (1)
template <bool RAW>
__global__ void __launch_bounds__(CT) sscan_local_kernel(ScanArgs a, float* __restrict__ st, float* __restrict__ sdl) {
  __shared__ alignas(16) float sB[L * N];
  const int c = blockIdx.x, d = blockIdx.y * CT + threadIdx.x;
  const bool live = d < a.Di;
  long long row0;
  int len;
  chunk_rows(a, c, row0, len);
  stage_bc(a, a.B, a.bs, row0, len, sB);
  f2 A2[N / 2], h[N / 2];
  load_A(a, d, live, A2);
#pragma unroll
  for (int p = 0; p < N / 2; ++p) h[p] = 0ull;
  float s = 0.f;
  const DeltaCol<RAW> delta(a, row0, d);
  const Col16 ucol(a.u, row0, a.us, d);
  typename DeltaCol<RAW>::T nd[PF];
  u16 nu[PF];
  auto fetch = [&](int t0) {
#pragma unroll
    for (int i = 0; i < PF; ++i) {
      const bool ok = live && t0 + i < len;
      nd[i] = delta(t0 + i, ok);
      nu[i] = ucol(t0 + i, ok);
    }
  };
  fetch(0);
  __syncthreads();
  for (int t0 = 0; t0 < len; t0 += PF) {
    float dl[PF], u[PF];
#pragma unroll
    for (int i = 0; i < PF; ++i) {
      dl[i] = DeltaCol<RAW>::value(nd[i], live && t0 + i < len);
      u[i] = bf(nu[i]);
    }
    if (t0 + PF < len) fetch(t0 + PF);
#pragma unroll
    for (int i = 0; i < PF; ++i) {
      const F4* b4 = reinterpret_cast<const F4*>(sB + (t0 + i) * N);
      const f2 d2 = pk(dl[i], dl[i]), x2 = pk(dl[i] * u[i], dl[i] * u[i]);
      s += dl[i];
#pragma unroll
      for (int p = 0; p < N / 4; ++p) {
        const F4 b = b4[p];
        h[2 * p] = fma2(ex2v(mul2(d2, A2[2 * p])), h[2 * p], mul2(x2, b.a));
        h[2 * p + 1] = fma2(ex2v(mul2(d2, A2[2 * p + 1])), h[2 * p + 1], mul2(x2, b.b));
      }
    }
  }
  float* o = st + (long long)c * a.kept * N * a.DiP + d;
#pragma unroll
  for (int p = 0; p < N / 2; ++p) {
    float x, y;
    up(h[p], x, y);
    o[(2 * p) * a.DiP] = x;
    o[(2 * p + 1) * a.DiP] = y;
  }
  sdl[(long long)c * a.DiP + d] = s;
}

// (2) and (5): carry over the chunks of each document, in place.  forward: st[c] = state entering chunk c; reverse: st[c] =
// adjoint of the state leaving chunk c.  `step`: distance of consecutive chunks' entries.  Eight loads in flight per thread.
__global__ void sscan_carry_kernel(const long long* __restrict__ first, const long long* __restrict__ last, const float* __restrict__ A,
                                   const float* __restrict__ sdl, float* __restrict__ st, long long step, int Di, int DiP, int reverse) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = e / DiP, d = e - n * DiP;
  const int doc = blockIdx.y;
  const int c0 = (int)first[doc], cnt = (int)last[doc] - c0 + 1;
  const float A2 = d < Di ? A[(long long)d * N + n] * LOG2E : 0.f;
  float s = 0.f;
  for (int i0 = 0; i0 < cnt; i0 += 8) {
    float v[8], q[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (i0 + k >= cnt) break;
      const int c = c0 + (reverse ? cnt - 1 - i0 - k : i0 + k);
      v[k] = st[(long long)c * step + e];
      q[k] = sdl[(long long)c * DiP + d];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (i0 + k >= cnt) break;
      const int c = c0 + (reverse ? cnt - 1 - i0 - k : i0 + k);
      st[(long long)c * step + e] = s;
      s = fmaf(exp2f(A2 * q[k]), s, v[k]);
    }
  }
}

// (3)
template <bool RAW, bool GATE>
__global__ void __launch_bounds__(CT, 4) sscan_out_kernel(ScanArgs a, float* __restrict__ st, __nv_bfloat16* __restrict__ y,
                                                       __nv_bfloat16* __restrict__ out) {
  __shared__ alignas(16) float sB[L * N];
  __shared__ alignas(16) float sC[L * N];
  const int c = blockIdx.x, d = blockIdx.y * CT + threadIdx.x;
  const bool live = d < a.Di;
  long long row0;
  int len;
  chunk_rows(a, c, row0, len);
  stage_bc(a, a.B, a.bs, row0, len, sB);
  stage_bc(a, a.C, a.cs, row0, len, sC);
  f2 A2[N / 2], h[N / 2];
  load_A(a, d, live, A2);
  const bool keep = a.kept == NSEG;
  float* s0 = st + (long long)c * a.kept * N * a.DiP + d;
#pragma unroll
  for (int p = 0; p < N / 2; ++p) h[p] = pk(s0[(2 * p) * a.DiP], s0[(2 * p + 1) * a.DiP]);
  const float Dd = live ? a.Dv[d] : 0.f;
  const DeltaCol<RAW> delta(a, row0, d);
  const Col16 ucol(a.u, row0, a.us, d), zcol(GATE ? a.z : a.u, row0, GATE ? a.zs : a.us, d);
  typename DeltaCol<RAW>::T nd[PF];
  u16 nu[PF], nz[PF];
  auto fetch = [&](int t0) {
#pragma unroll
    for (int i = 0; i < PF; ++i) {
      const bool ok = live && t0 + i < len;
      nd[i] = delta(t0 + i, ok);
      nu[i] = ucol(t0 + i, ok);
      if (GATE) nz[i] = zcol(t0 + i, ok);
    }
  };
  fetch(0);
  y += row0 * a.Di + d;
  out += row0 * a.Di + d;
  __syncthreads();
  for (int t0 = 0; t0 < len; t0 += PF) {
    if (keep && t0 > 0 && (t0 % SEG) == 0) {
      float* o = s0 + (long long)(t0 / SEG) * N * a.DiP;
#pragma unroll
      for (int p = 0; p < N / 2; ++p) {
        float x, w;
        up(h[p], x, w);
        o[(2 * p) * a.DiP] = x;
        o[(2 * p + 1) * a.DiP] = w;
      }
    }
    float dl[PF], u[PF], zz[PF];
#pragma unroll
    for (int i = 0; i < PF; ++i) {
      dl[i] = DeltaCol<RAW>::value(nd[i], live && t0 + i < len);
      u[i] = bf(nu[i]);
      if (GATE) zz[i] = bf(nz[i]);
    }
    if (t0 + PF < len) fetch(t0 + PF);
#pragma unroll
    for (int i = 0; i < PF; ++i) {
      const F4* b4 = reinterpret_cast<const F4*>(sB + (t0 + i) * N);
      const F4* c4 = reinterpret_cast<const F4*>(sC + (t0 + i) * N);
      const f2 d2 = pk(dl[i], dl[i]), x2 = pk(dl[i] * u[i], dl[i] * u[i]);
      f2 acc = 0ull, acc1 = 0ull;
#pragma unroll
      for (int p = 0; p < N / 4; ++p) {
        const F4 b = b4[p], cc = c4[p];
        h[2 * p] = fma2(ex2v(mul2(d2, A2[2 * p])), h[2 * p], mul2(x2, b.a));
        h[2 * p + 1] = fma2(ex2v(mul2(d2, A2[2 * p + 1])), h[2 * p + 1], mul2(x2, b.b));
        acc = fma2(h[2 * p], cc.a, acc);
        acc1 = fma2(h[2 * p + 1], cc.b, acc1);
      }
      if (live && t0 + i < len) {
        const float v = fmaf(Dd, u[i], sum2(add2(acc, acc1)));
        const int o = (t0 + i) * a.Di;
        if (!GATE || keep) y[o] = __float2bfloat16(v);
        if (GATE) out[o] = __float2bfloat16(v * zz[i] * sigm(zz[i]));
      }
    }
  }
}

// (4): adjoint of the state entering the chunk, from a zero adjoint at its end: c <- a_t (c + C_t dy_t), t descending
template <bool RAW, bool GATE>
__global__ void __launch_bounds__(CT) sscan_local_bwd_kernel(ScanArgs a, const __nv_bfloat16* __restrict__ dout, float* __restrict__ adj) {
  __shared__ alignas(16) float sC[L * N];
  const int c = blockIdx.x, d = blockIdx.y * CT + threadIdx.x;
  const bool live = d < a.Di;
  long long row0;
  int len;
  chunk_rows(a, c, row0, len);
  stage_bc(a, a.C, a.cs, row0, len, sC);
  f2 A2[N / 2], g[N / 2];
  load_A(a, d, live, A2);
#pragma unroll
  for (int p = 0; p < N / 2; ++p) g[p] = 0ull;
  const DeltaCol<RAW> delta(a, row0, d);
  const Col16 ocol(dout, row0, a.Di, d), zcol(GATE ? a.z : dout, row0, GATE ? a.zs : a.Di, d);
  typename DeltaCol<RAW>::T nd[PF];
  u16 no[PF], nz[PF];
  auto fetch = [&](int t0) {
#pragma unroll
    for (int i = 0; i < PF; ++i) {
      const bool ok = live && t0 + i < len;
      nd[i] = delta(t0 + i, ok);
      no[i] = ocol(t0 + i, ok);
      if (GATE) nz[i] = zcol(t0 + i, ok);
    }
  };
  const int t_first = (len - 1) / PF * PF;
  fetch(t_first);
  __syncthreads();
  for (int t0 = t_first; t0 >= 0; t0 -= PF) {
    float dl[PF], dy[PF];
#pragma unroll
    for (int i = 0; i < PF; ++i) {
      dl[i] = DeltaCol<RAW>::value(nd[i], live && t0 + i < len);
      dy[i] = bf(no[i]);
      if (GATE) {
        const float z = bf(nz[i]);
        dy[i] *= z * sigm(z);
      }
    }
    if (t0 > 0) fetch(t0 - PF);
#pragma unroll
    for (int i = PF - 1; i >= 0; --i) {
      const F4* c4 = reinterpret_cast<const F4*>(sC + (t0 + i) * N);
      const f2 d2 = pk(dl[i], dl[i]), y2 = pk(dy[i], dy[i]);
#pragma unroll
      for (int p = 0; p < N / 4; ++p) {
        const F4 cc = c4[p];
        g[2 * p] = mul2(ex2v(mul2(d2, A2[2 * p])), fma2(cc.a, y2, g[2 * p]));
        g[2 * p + 1] = mul2(ex2v(mul2(d2, A2[2 * p + 1])), fma2(cc.b, y2, g[2 * p + 1]));
      }
    }
  }
  float* o = adj + (long long)c * N * a.DiP + d;
#pragma unroll
  for (int p = 0; p < N / 2; ++p) {
    float x, w;
    up(g[p], x, w);
    o[(2 * p) * a.DiP] = x;
    o[(2 * p + 1) * a.DiP] = w;
  }
}

// (6): all gradients of one chunk and 64 channels, 16 steps at a time from the back.  Lane = (channel pair cg, state quad q).
// Per 16 steps: recompute the states from the kept one, leaving one every four steps in shared memory; then per four steps
// recompute decay and decayed state into registers and walk back.  Four steps' partial sums go to shared memory, from
// where the warp adds them: over the four quads (ddelta, du) and over the eight channel pairs (dB, dC).
constexpr int BT = 128;                    // threads
constexpr int BC = 64;                     // channels per block
constexpr int RROW = 36;                   // float4 per row of the reduction buffer (32 lanes + 4: rows start on other banks)
struct BwdSmem {
  float4 dl[SEG][BC / 2];                  // (delta, delta) of two channels
  float4 x[SEG][BC / 2];                   // (delta u, delta u)
  float4 dy[SEG][BC / 2];
  float B[SEG][N];
  float C[SEG][N];
  float4 ck[3][2][BT];                     // states entering steps 0, 4, 8 of the segment
  float4 red[BT / 32][4 * 3 * RROW];
  float bc[BT / 32][SEG][2 * N];           // per-warp dB | dC
};

template <bool RAW, bool GATE>
__global__ void __launch_bounds__(BT, 3) sscan_bwd_kernel(ScanArgs a, const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ y,
                                                          const float* __restrict__ st, const float* __restrict__ adj,
                                                          __nv_bfloat16* __restrict__ du, void* __restrict__ ddl,
                                                          __nv_bfloat16* __restrict__ dz, int dzs, float* __restrict__ dA,
                                                          float* __restrict__ part, float* __restrict__ dD, long long T) {
  extern __shared__ __align__(16) unsigned char raw_smem[];
  BwdSmem& s = *reinterpret_cast<BwdSmem*>(raw_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q = lane & 3, cg = lane >> 2;
  const int c = blockIdx.x, d0 = blockIdx.y * BC;
  long long row0;
  int len;
  chunk_rows(a, c, row0, len);
  const int cp = warp * 8 + cg;            // channel pair of this lane within the block
  const int dc = d0 + 2 * cp;
  f2 A2[2][2], carry[2][2], dAa[2][2], h[2][2];
  const float* ad = adj + (long long)c * N * a.DiP + dc;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float4 v = dc + k < a.Di ? *reinterpret_cast<const float4*>(a.A + (long long)(dc + k) * N + q * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    A2[k][0] = pk(v.x * LOG2E, v.y * LOG2E);
    A2[k][1] = pk(v.z * LOG2E, v.w * LOG2E);
    dAa[k][0] = dAa[k][1] = 0ull;
  }
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const int n = q * 4 + 2 * p;
    const float2 lo = *reinterpret_cast<const float2*>(ad + n * a.DiP), hi = *reinterpret_cast<const float2*>(ad + (n + 1) * a.DiP);
    carry[0][p] = pk(lo.x, hi.x);
    carry[1][p] = pk(lo.y, hi.y);
  }
  // the lane that finishes sums over states handles step t = lane / 8 (of four) and channel pair lane % 8 of its warp
  const int fcp = warp * 8 + (lane & 7), fd = d0 + 2 * fcp;
  const float D0 = fd < a.Di ? a.Dv[fd] : 0.f, D1 = fd + 1 < a.Di ? a.Dv[fd + 1] : 0.f;
  float dD0 = 0.f, dD1 = 0.f;
  const int st_ch = tid % BC, st_t = tid / BC, st_d = d0 + st_ch;
  const bool st_live = st_d < a.Di;
  const DeltaCol<RAW> delta(a, row0, st_d), fdelta(a, row0, fd);
  const Col16 ucol(a.u, row0, a.us, st_d), ocol(dout, row0, a.Di, st_d), zcol(GATE ? a.z : dout, row0, GATE ? a.zs : a.Di, st_d),
      ycol(GATE ? y : dout, row0, a.Di, st_d), fu(a.u, row0, a.us, fd);
  __nv_bfloat16* pdz = GATE ? dz + row0 * dzs + st_d : nullptr;

  for (int seg = (len - 1) / SEG; seg >= 0; --seg) {
    const int tb = seg * SEG;
    __syncthreads();
    // a thread stages one channel of eight steps; all of its loads go out first, the kept states' with them
    const float* hs = st + ((long long)c * NSEG + seg) * N * a.DiP + dc;
    float2 hv[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) hv[p] = __ldg(reinterpret_cast<const float2*>(hs + (q * 4 + p) * a.DiP));
    {
      constexpr int NT = SEG * BC / BT;
      typename DeltaCol<RAW>::T rd[NT];
      u16 ru[NT], ro[NT], rz[NT], ry[NT];
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        const int r = tb + i * (BT / BC) + st_t;
        const bool ok = r < len && st_live;
        rd[i] = delta(r, ok);
        ru[i] = ucol(r, ok);
        ro[i] = ocol(r, ok);
        if (GATE) {
          rz[i] = zcol(r, ok);
          ry[i] = ycol(r, ok);
        }
      }
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        const int t = i * (BT / BC) + st_t, r = tb + t;
        const bool ok = r < len && st_live;
        const float dlv = DeltaCol<RAW>::value(rd[i], ok), uv = bf(ru[i]);
        float dyv = bf(ro[i]);
        if (GATE) {
          const float z = bf(rz[i]), sg = sigm(z), sl = z * sg;
          if (ok) pdz[r * dzs] = __float2bfloat16(dyv * bf(ry[i]) * (sg + sl * (1.f - sg)));
          dyv *= sl;
        }
        reinterpret_cast<float2*>(&s.dl[t][0])[st_ch] = make_float2(dlv, dlv);
        reinterpret_cast<float2*>(&s.x[t][0])[st_ch] = make_float2(dlv * uv, dlv * uv);
        reinterpret_cast<float2*>(&s.dy[t][0])[st_ch] = make_float2(dyv, dyv);
      }
    }
    for (int i = tid; i < SEG * N; i += BT) {
      const int t = i / N, n = i % N;
      const bool ok = tb + t < len;
      s.B[t][n] = ok ? load_bc(a, a.B, a.bs, row0 + tb + t, n) : 0.f;
      s.C[t][n] = ok ? load_bc(a, a.C, a.cs, row0 + tb + t, n) : 0.f;
    }
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      h[0][p] = pk(hv[2 * p].x, hv[2 * p + 1].x);
      h[1][p] = pk(hv[2 * p].y, hv[2 * p + 1].y);
    }
    __syncthreads();
    // states entering steps 4, 8, 12
#pragma unroll
    for (int sb = 0; sb < 3; ++sb) {
      *reinterpret_cast<F4*>(&s.ck[sb][0][tid]) = F4{h[0][0], h[0][1]};
      *reinterpret_cast<F4*>(&s.ck[sb][1][tid]) = F4{h[1][0], h[1][1]};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = sb * 4 + i;
        const F4 b = *reinterpret_cast<const F4*>(&s.B[t][q * 4]);
        const F4 dl = *reinterpret_cast<const F4*>(&s.dl[t][cp]), x = *reinterpret_cast<const F4*>(&s.x[t][cp]);
        h[0][0] = fma2(ex2v(mul2(dl.a, A2[0][0])), h[0][0], mul2(x.a, b.a));
        h[0][1] = fma2(ex2v(mul2(dl.a, A2[0][1])), h[0][1], mul2(x.a, b.b));
        h[1][0] = fma2(ex2v(mul2(dl.b, A2[1][0])), h[1][0], mul2(x.b, b.a));
        h[1][1] = fma2(ex2v(mul2(dl.b, A2[1][1])), h[1][1], mul2(x.b, b.b));
      }
    }
#pragma unroll 1
    for (int sb = 3; sb >= 0; --sb) {
      if (sb < 3) {
        const F4 k0 = *reinterpret_cast<const F4*>(&s.ck[sb][0][tid]), k1 = *reinterpret_cast<const F4*>(&s.ck[sb][1][tid]);
        h[0][0] = k0.a, h[0][1] = k0.b, h[1][0] = k1.a, h[1][1] = k1.b;
      }
      // what the finishing lanes need of u and raw, on its way while the states are recomputed
      const int ft = tb + sb * 4 + (lane >> 3);
      const bool f0 = ft < len && fd < a.Di, f1 = ft < len && fd + 1 < a.Di;
      const u16 fu0 = fu(ft, f0), fu1 = f1 ? __ldg(fu.p + ft * fu.stride + 1) : (u16)0;
      u16 fr0 = 0, fr1 = 0;
      if constexpr (RAW) {
        fr0 = fdelta(ft, f0);
        fr1 = f1 ? __ldg(fdelta.c.p + ft * fdelta.c.stride + 1) : (u16)0;
      }
      f2 dec[4][2][2], w[4][2][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = sb * 4 + i;
        const F4 b = *reinterpret_cast<const F4*>(&s.B[t][q * 4]);
        const F4 dl = *reinterpret_cast<const F4*>(&s.dl[t][cp]), x = *reinterpret_cast<const F4*>(&s.x[t][cp]);
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int p = 0; p < 2; ++p) {
            dec[i][k][p] = ex2v(mul2(k ? dl.b : dl.a, A2[k][p]));
            w[i][k][p] = mul2(dec[i][k][p], h[k][p]);
            h[k][p] = fma2(k ? x.b : x.a, p ? b.b : b.a, w[i][k][p]);
          }
      }
      __syncwarp();  // the previous four steps' sums have been read
#pragma unroll
      for (int i = 3; i >= 0; --i) {
        const int t = sb * 4 + i;
        const F4 b = *reinterpret_cast<const F4*>(&s.B[t][q * 4]), cc = *reinterpret_cast<const F4*>(&s.C[t][q * 4]);
        const F4 dl = *reinterpret_cast<const F4*>(&s.dl[t][cp]), x = *reinterpret_cast<const F4*>(&s.x[t][cp]);
        const F4 dy = *reinterpret_cast<const F4*>(&s.dy[t][cp]);
        f2 s1[2], s2[2], vb[2], vc[2];
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int p = 0; p < 2; ++p) {
            const f2 bb = p ? b.b : b.a, xx = k ? x.b : x.a, dd = k ? dl.b : dl.a, yy = k ? dy.b : dy.a;
            const f2 g = fma2(p ? cc.b : cc.a, yy, carry[k][p]);
            const f2 ht = fma2(xx, bb, w[i][k][p]);
            const f2 gw = mul2(g, w[i][k][p]);
            vb[p] = k ? fma2(g, xx, vb[p]) : mul2(g, xx);
            vc[p] = k ? fma2(ht, yy, vc[p]) : mul2(ht, yy);
            s1[k] = p ? fma2(gw, A2[k][p], s1[k]) : mul2(gw, A2[k][p]);
            s2[k] = p ? fma2(g, bb, s2[k]) : mul2(g, bb);
            dAa[k][p] = fma2(gw, dd, dAa[k][p]);
            carry[k][p] = mul2(dec[i][k][p], g);
          }
        float4* r = s.red[warp] + i * 3 * RROW + lane;
        r[0] = make_float4(sum2(s1[0]), sum2(s2[0]), sum2(s1[1]), sum2(s2[1]));
        *reinterpret_cast<F4*>(r + RROW) = F4{vb[0], vb[1]};
        *reinterpret_cast<F4*>(r + 2 * RROW) = F4{vc[0], vc[1]};
      }
      __syncwarp();
      {
        // over the four state quads; the order of the quads is rotated per lane so that eight lanes read eight banks groups
        const int i = lane >> 3, g8 = lane & 7, t = sb * 4 + i;
        const F4* r = reinterpret_cast<const F4*>(s.red[warp] + i * 3 * RROW + g8 * 4);
        F4 v = r[(g8 >> 1) & 3];
#pragma unroll
        for (int k = 1; k < 4; ++k) {
          const F4 o = r[(k + (g8 >> 1)) & 3];
          v.a = add2(v.a, o.a);
          v.b = add2(v.b, o.b);
        }
        if (tb + t < len) {
          const long long row = row0 + tb + t;
          const F4 dl = *reinterpret_cast<const F4*>(&s.dl[t][fcp]), dy = *reinterpret_cast<const F4*>(&s.dy[t][fcp]);
          float dlv[2], dyv[2], tmp, m1[2], m2[2];
          up(dl.a, dlv[0], tmp), up(dl.b, dlv[1], tmp);
          up(dy.a, dyv[0], tmp), up(dy.b, dyv[1], tmp);
          up(v.a, m1[0], m2[0]), up(v.b, m1[1], m2[1]);
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int d = fd + k;
            if (d < a.Di) {
              const float uv = bf(k ? fu1 : fu0);
              float dd = fmaf(uv, m2[k], m1[k] * LN2);
              du[row * a.Di + d] = __float2bfloat16(fmaf(k ? D1 : D0, dyv[k], dlv[k] * m2[k]));
              if (RAW) {
                dd *= sigm(bf(k ? fr1 : fr0));
                ((__nv_bfloat16*)ddl)[row * a.Di + d] = __float2bfloat16(dd);
              } else {
                ((float*)ddl)[row * a.Di + d] = dd;
              }
              if (k) dD1 = fmaf(dyv[k], uv, dD1);
              else dD0 = fmaf(dyv[k], uv, dD0);
            }
          }
        }
      }
      {
        // over the eight channel pairs
        const int i = lane >> 3, k = (lane >> 2) & 1, q8 = lane & 3;
        const F4* r = reinterpret_cast<const F4*>(s.red[warp] + (i * 3 + 1 + k) * RROW + q8);
        F4 v = r[0];
#pragma unroll
        for (int g = 1; g < 8; ++g) {
          v.a = add2(v.a, r[g * 4].a);
          v.b = add2(v.b, r[g * 4].b);
        }
        *reinterpret_cast<F4*>(&s.bc[warp][sb * 4 + i][k * N + q8 * 4]) = v;
      }
    }
    __syncthreads();
    for (int i = tid; i < SEG * 2 * N; i += BT) {
      const int t = i / (2 * N);
      if (tb + t < len) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < BT / 32; ++w) v += s.bc[w][t][i % (2 * N)];
        part[((long long)blockIdx.y * T + row0 + tb + t) * (2 * N) + i % (2 * N)] = v;
      }
    }
  }
  // dA per chunk, dD per chunk: the caller adds the chunks up
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    float lo0, hi0, lo1, hi1;
    up(dAa[0][p], lo0, hi0);
    up(dAa[1][p], lo1, hi1);
    float* o = dA + ((long long)c * N + q * 4 + 2 * p) * a.DiP + dc;
    *reinterpret_cast<float2*>(o) = make_float2(lo0, lo1);
    *reinterpret_cast<float2*>(o + a.DiP) = make_float2(hi0, hi1);
  }
#pragma unroll
  for (int o = 8; o < 32; o <<= 1) {
    dD0 += __shfl_xor_sync(0xffffffffu, dD0, o);
    dD1 += __shfl_xor_sync(0xffffffffu, dD1, o);
  }
  if (lane < 8) *reinterpret_cast<float2*>(dD + (long long)c * a.DiP + fd) = make_float2(dD0, dD1);
}

// dB, dC: sum of the channel blocks' partials, written in the operands' type
__global__ void sscan_bc_reduce_kernel(const float* __restrict__ part, int nblk, long long T, void* __restrict__ dB, void* __restrict__ dC, int out16) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // one float4 of the 32 columns of a row
  if (i >= T * (2 * N / 4)) return;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int b = 0; b < nblk; ++b) {
    const float4 p = reinterpret_cast<const float4*>(part)[(long long)b * T * (2 * N / 4) + i];
    v.x += p.x, v.y += p.y, v.z += p.z, v.w += p.w;
  }
  const long long row = i / (2 * N / 4);
  const int col = (int)(i % (2 * N / 4)) * 4;
  const long long o = row * N + (col & (N - 1));
  void* dst = col < N ? dB : dC;
  if (out16) {
    __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>((__nv_bfloat16*)dst + o);
    p[0] = __floats2bfloat162_rn(v.x, v.y);
    p[1] = __floats2bfloat162_rn(v.z, v.w);
  } else {
    *reinterpret_cast<float4*>((float*)dst + o) = v;
  }
}

ScanArgs make_args(const void* u, long long us, const void* dl, long long ds, const void* z, long long zs, const void* B, long long bs,
                   const void* C, long long cs, int bc16, const float* A, const float* Dv, const int* inv, int Di, int keep) {
  ScanArgs a;
  a.kept = keep ? NSEG : 1;
  a.u = (const __nv_bfloat16*)u, a.dl = dl, a.z = (const __nv_bfloat16*)z, a.B = B, a.C = C, a.A = A, a.Dv = Dv, a.inv = inv;
  a.us = (int)us, a.ds = (int)ds, a.zs = (int)zs, a.bs = (int)bs, a.cs = (int)cs;  // 64 rows of any of them fit 32 bits
  a.Di = Di, a.DiP = (Di + CT - 1) / CT * CT, a.bc16 = bc16;
  return a;
}

}  // namespace

extern "C" {

// Row length of the state arrays: Di rounded up to whole blocks.
int fb_sscan_padded(int Di) { return (Di + CT - 1) / CT * CT; }
int fb_sscan_channel_blocks(int Di) { return (Di + BC - 1) / BC; }

// Forward.  raw: dl is bf16 and goes through softplus.  z: null, or the gate; then y is the ungated output (null: not wanted)
// and out = y silu(z).  st: fp32 [NC, 4, 16, DiP], states entering steps 0, 16, 32, 48; without keep (no backward) [NC, 1, 16, DiP];
// sdl: fp32 [NC, DiP]; y, out: bf16 [T, Di].
int fb_sscan_fwd(const void* u, long long us, const void* dl, long long ds, int raw, const void* z, long long zs, const void* B, long long bs,
                 const void* C, long long cs, int bc16, const float* A, const float* Dv, const int* inv, const long long* first,
                 const long long* last, int n_docs, float* st, float* sdl, void* y, void* out, int keep, int NC, int Di, int n_state,
                 cudaStream_t stream) {
  if (NC <= 0) return 0;
  if (n_state != N) return -2;
  const ScanArgs a = make_args(u, us, dl, ds, z, zs, B, bs, C, cs, bc16, A, Dv, inv, Di, keep);
  const dim3 grid(NC, a.DiP / CT);
  if (raw) sscan_local_kernel<true><<<grid, CT, 0, stream>>>(a, st, sdl);
  else sscan_local_kernel<false><<<grid, CT, 0, stream>>>(a, st, sdl);
  int rc = fb::launch_ok("sscan_local_kernel");
  if (rc) return rc;
  sscan_carry_kernel<<<dim3(a.DiP * N / 256, n_docs), 256, 0, stream>>>(first, last, A, sdl, st, (long long)a.kept * N * a.DiP, Di, a.DiP, 0);
  rc = fb::launch_ok("sscan_carry_kernel");
  if (rc) return rc;
  __nv_bfloat16 *yy = (__nv_bfloat16*)y, *oo = (__nv_bfloat16*)out;
  if (z) {
    if (raw) sscan_out_kernel<true, true><<<grid, CT, 0, stream>>>(a, st, yy, oo);
    else sscan_out_kernel<false, true><<<grid, CT, 0, stream>>>(a, st, yy, oo);
  } else {
    if (raw) sscan_out_kernel<true, false><<<grid, CT, 0, stream>>>(a, st, yy, oo);
    else sscan_out_kernel<false, false><<<grid, CT, 0, stream>>>(a, st, yy, oo);
  }
  return fb::launch_ok("sscan_out_kernel");
}

// Backward.  dout: gradient of the (gated) output, bf16 [T, Di]; y: ungated output (with z).  adj: fp32 [NC, 16, DiP] scratch;
// du: bf16 [T, Di]; ddl: bf16 (raw) or fp32 [T, Di]; dz: bf16 [T, Di], row stride dzs (with z); dB, dC: [T, 16] in B's type.  Partial results
// for the caller to add over the chunks: dA [NC, 16, DiP], dD [NC, DiP].  part: fp32 [channel blocks, T, 32] scratch.
int fb_sscan_bwd(const void* u, long long us, const void* dl, long long ds, int raw, const void* z, long long zs, const void* B, long long bs,
                 const void* C, long long cs, int bc16, const float* A, const float* Dv, const int* inv, const long long* first,
                 const long long* last, int n_docs, const float* st, const float* sdl, const void* y, const void* dout, float* adj, void* du,
                 void* ddl, void* dz, long long dzs, float* dA, float* part, float* dD, void* dB, void* dC, long long T, int NC, int Di, int n_state,
                 cudaStream_t stream) {
  if (NC <= 0) return 0;
  if (n_state != N) return -2;
  const ScanArgs a = make_args(u, us, dl, ds, z, zs, B, bs, C, cs, bc16, A, Dv, inv, Di, 1);
  const dim3 grid(NC, a.DiP / CT);
  const __nv_bfloat16* go = (const __nv_bfloat16*)dout;
  if (z) {
    if (raw) sscan_local_bwd_kernel<true, true><<<grid, CT, 0, stream>>>(a, go, adj);
    else sscan_local_bwd_kernel<false, true><<<grid, CT, 0, stream>>>(a, go, adj);
  } else {
    if (raw) sscan_local_bwd_kernel<true, false><<<grid, CT, 0, stream>>>(a, go, adj);
    else sscan_local_bwd_kernel<false, false><<<grid, CT, 0, stream>>>(a, go, adj);
  }
  int rc = fb::launch_ok("sscan_local_bwd_kernel");
  if (rc) return rc;
  sscan_carry_kernel<<<dim3(a.DiP * N / 256, n_docs), 256, 0, stream>>>(first, last, A, sdl, adj, (long long)N * a.DiP, Di, a.DiP, 1);
  rc = fb::launch_ok("sscan_carry_kernel(reverse)");
  if (rc) return rc;
  const int nblk = fb_sscan_channel_blocks(Di);
  auto go_bwd = [&](auto kernel) -> int {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BwdSmem));
    if (e != cudaSuccess) return -3;
    kernel<<<dim3(NC, nblk), BT, sizeof(BwdSmem), stream>>>(a, go, (const __nv_bfloat16*)y, st, adj, (__nv_bfloat16*)du, ddl,
                                                                 (__nv_bfloat16*)dz, (int)dzs, dA, part, dD, T);
    return fb::launch_ok("sscan_bwd_kernel");
  };
  if (z) rc = raw ? go_bwd(sscan_bwd_kernel<true, true>) : go_bwd(sscan_bwd_kernel<false, true>);
  else rc = raw ? go_bwd(sscan_bwd_kernel<true, false>) : go_bwd(sscan_bwd_kernel<false, false>);
  if (rc) return rc;
  const long long n4 = T * (2 * N / 4);
  sscan_bc_reduce_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, stream>>>(part, nblk, T, dB, dC, bc16);
  return fb::launch_ok("sscan_bc_reduce_kernel");
}

}  // extern "C"
