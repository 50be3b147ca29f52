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
// shuffles), sweep (6) gives it 4 channels x 4 states (see there); pairs of states, or of channels, use the packed fp32x2
// instructions.  Every sweep fetches its operands ahead: waiting for memory at each group of steps, not the MUFU, set the pace
// before.  At that size with gate and softplus, before and after: (1) 0.44 -> 0.31 ms, (3) 0.84 -> 0.47, (4) 0.59 -> 0.36,
// (6) 2.17 -> 1.63 -> 1.26.  (1) and (4) keep the MUFU 80 and 78 % busy.  (3) keeps it and the issue slots at 59 % (126 registers leave 15
// warps an SM, whose stalls are fixed latencies); an eighth of its decays as polynomials on the multiply-add pipe made it 40 us slower.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

#include "host_utils.cuh"
#include "tc05.cuh"

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

// two channels at a time
__device__ __forceinline__ f2 dup(float v) { return pk(v, v); }
__device__ __forceinline__ f2 rcp2(f2 v) {
  float a, b;
  up(v, a, b);
  return pk(__fdividef(1.f, a), __fdividef(1.f, b));
}
__device__ __forceinline__ f2 sigm2(f2 x) { return rcp2(add2(ex2v(mul2(x, dup(-LOG2E))), dup(1.f))); }
// softplus and its derivative from one exponential
__device__ __forceinline__ void softplus2(f2 x, f2& sp, f2& sg) {
  float x0, x1;
  up(x, x0, x1);
  const f2 e = ex2v(mul2(pk(-fabsf(x0), -fabsf(x1)), dup(LOG2E))), s = mul2(e, rcp2(add2(e, dup(2.f)))), w = mul2(s, s);
  f2 p = fma2(w, dup(1.f / 13.f), dup(1.f / 11.f));
  p = fma2(p, w, dup(1.f / 9.f));
  p = fma2(p, w, dup(1.f / 7.f));
  p = fma2(p, w, dup(1.f / 5.f));
  p = fma2(p, w, dup(1.f / 3.f));
  p = fma2(p, w, dup(1.f));
  sp = fma2(add2(s, s), p, pk(fmaxf(x0, 0.f), fmaxf(x1, 0.f)));
  float r0, r1, e0, e1;
  up(rcp2(add2(e, dup(1.f))), r0, r1);
  up(e, e0, e1);
  sg = pk(x0 >= 0.f ? r0 : e0 * r0, x1 >= 0.f ? r1 : e1 * r1);
}
__device__ __forceinline__ f2 bf2(uint32_t v) { return pk(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); }

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

// (6): all gradients of one chunk and 128 channels, 16 steps at a time from the back.  A warp has 32 channels: lane = (channel
// quad cg, state quad q), a thread 4 channels x 4 states in eight channel pairs.  Per 16 steps: recompute the states from the
// kept one, leaving one every four steps in shared memory; then per four steps recompute decays and states, leaving them in
// tensor memory (32 columns a step, the thread's own lane: the 128 registers they would take cost a third of the warps), and
// walk back.  What bounds it: issue slots (355 instructions per warp and step, two per clock with 12 warps an SM), of which eight
// packed multiply-adds per pair on the way back and three forward are the work.  The sums over states (ddelta, du) and over
// channels (dB, dC) are halved from lane to lane by shuffles: a thread's registers are numbered so that what a lane keeps lies
// in the same registers on every lane (register k holds state k ^ (cg & 3) of the quad, register j channel pair j ^ (q >> 1)),
// which leaves six selects per step instead of 26.  Measured at 32,768 tokens x 2,048 channels: 2 channels x 4 states and sums
// through shared memory (73 % of its bandwidth) 1.62 ms; this split with all four steps in registers (8 warps) 1.85, in tensor
// memory 1.48, a step's sums under the next one's loads and results through shared memory 1.39, two channels staged at a
// time 1.26.
constexpr int BT = 128;                    // threads
constexpr int BC = 128;                    // channels per block
constexpr int G = 4;                       // steps recomputed into registers together
struct BwdSmem {
  float dl[SEG][BC];
  float sg[SEG][BC];                       // derivative of delta by its argument
  float u[SEG][BC];
  float dy[SEG][BC];
  float2 B[SEG][N];                        // (value, value)
  float2 C[SEG][N];
  f2 ck[SEG / G - 1][8][BT];               // states entering steps 0, 4, 8 of the segment
  float bc[BT / 32][SEG][2 * N];           // per-warp dB | dC
  uint32_t tmem;
};

__device__ __forceinline__ f2 lds2(const void* p) { return *reinterpret_cast<const f2*>(p); }
__device__ __forceinline__ float shx(float v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }

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
  if (warp == 0) {
    tc05::tmem_alloc(&s.tmem, 32 * G);
    tc05::tmem_relinquish();
  }
  tc05::tc_fence_before();
  __syncthreads();
  tc05::tc_fence_after();
  const uint32_t taddr = s.tmem + ((uint32_t)(warp * 32) << 16);
  int ch[2], nn[4];                        // channel pairs within the block and states of this thread's registers
#pragma unroll
  for (int j = 0; j < 2; ++j) ch[j] = warp * 32 + cg * 4 + 2 * (j ^ (q >> 1));
#pragma unroll
  for (int k = 0; k < 4; ++k) nn[k] = q * 4 + (k ^ (cg & 3));
  f2 A2[2][4], carry[2][4], dAa[2][4], h[2][4];
  const float* ad = adj + (long long)c * N * a.DiP + d0;
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int d = d0 + ch[j];
      const float lo = d < a.Di ? a.A[(long long)d * N + nn[k]] : 0.f, hi = d + 1 < a.Di ? a.A[(long long)(d + 1) * N + nn[k]] : 0.f;
      A2[j][k] = pk(lo * LOG2E, hi * LOG2E);
      carry[j][k] = lds2(ad + nn[k] * a.DiP + ch[j]);
      dAa[j][k] = 0ull;
    }
  // after the sums over states a lane holds one channel pair: ddelta where q is even, du where it is odd
  const bool is_du = q & 1;
  const int fch = ch[0], fd = d0 + fch;
  const f2 Df = is_du ? pk(fd < a.Di ? a.Dv[fd] : 0.f, fd + 1 < a.Di ? a.Dv[fd + 1] : 0.f) : 0ull;
  const float* ffac = is_du ? &s.dl[0][fch] : &s.sg[0][fch];
  const bool hi = cg & 4;
  const bool even = (a.Di & 1) == 0;
  const f2 ln2 = pk(LN2, LN2);

  // a thread stages two neighbouring channels of eight steps
  const int sc = 2 * (tid & 63), st0 = (tid >> 6) * 8, sd = d0 + sc;
  const bool live0 = sd < a.Di, live1 = sd + 1 < a.Di;
  const uintptr_t bases = (uintptr_t)a.u | (RAW ? (uintptr_t)a.dl : (uintptr_t)a.dl >> 1) | (uintptr_t)dout | (GATE ? (uintptr_t)a.z | (uintptr_t)y | (uintptr_t)dz : 0);
  const bool vec = live1 && even && (bases & 3) == 0 && ((a.us | a.ds | (GATE ? a.zs | dzs : 0)) & 1) == 0;
  f2 dDa = 0ull;
  const u16* pu = reinterpret_cast<const u16*>(a.u) + row0 * a.us + sd;
  const u16* po = reinterpret_cast<const u16*>(dout) + row0 * a.Di + sd;
  const u16* pz = GATE ? reinterpret_cast<const u16*>(a.z) + row0 * a.zs + sd : nullptr;
  const u16* py = GATE ? reinterpret_cast<const u16*>(y) + row0 * a.Di + sd : nullptr;
  const u16* pr = RAW ? reinterpret_cast<const u16*>(a.dl) + row0 * a.ds + sd : nullptr;
  const float* pf = RAW ? nullptr : reinterpret_cast<const float*>(a.dl) + row0 * a.ds + sd;
  u16* pdz = GATE ? reinterpret_cast<u16*>(dz) + row0 * dzs + sd : nullptr;
  u16* pdu = reinterpret_cast<u16*>(du) + row0 * a.Di + sd;
  u16* pdd = reinterpret_cast<u16*>(ddl) + row0 * a.Di + sd;
  // a row's two values; FULL: both channels and all rows exist and lie on four bytes
  auto two = [&](auto full, const u16* p, bool row) -> uint32_t {
    if constexpr (decltype(full)::value) return __ldg(reinterpret_cast<const uint32_t*>(p));
    const uint32_t lo = row && live0 ? __ldg(p) : (u16)0, hi = row && live1 ? __ldg(p + 1) : (u16)0;
    return lo | hi << 16;
  };
  auto stage = [&](auto full, int tb) {
    constexpr bool FULL = decltype(full)::value;
    uint32_t rd[8], ru[8], ro[8], rz[8], ry[8];
    f2 rf[8];
    const int r0 = tb + st0;
    const u16 *qu = pu + r0 * a.us, *qo = po + r0 * a.Di, *qz = GATE ? pz + r0 * a.zs : nullptr, *qy = GATE ? py + r0 * a.Di : nullptr,
              *qr = RAW ? pr + r0 * a.ds : nullptr;
    u16* qdz = GATE ? pdz + r0 * dzs : nullptr;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const bool row = FULL || r0 + i < len;
      ru[i] = two(full, qu + i * a.us, row);
      ro[i] = two(full, qo + i * a.Di, row);
      if (RAW) {
        rd[i] = two(full, qr + i * a.ds, row);
      } else {
        const float* q = pf + (r0 + i) * a.ds;
        rf[i] = pk(row && live0 ? __ldg(q) : 0.f, row && live1 ? __ldg(q + 1) : 0.f);
      }
      if (GATE) {
        rz[i] = two(full, qz + i * a.zs, row);
        ry[i] = two(full, qy + i * a.Di, row);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = st0 + i;
      const bool row = FULL || r0 + i < len;
      const f2 uv = bf2(ru[i]);
      f2 dyv = bf2(ro[i]);
      if (GATE) {
        const f2 z = bf2(rz[i]), g = sigm2(z), l = mul2(z, g), om = fma2(g, dup(-1.f), dup(1.f));
        float q0, q1;
        up(mul2(mul2(dyv, bf2(ry[i])), fma2(l, om, g)), q0, q1);
        const uint32_t q = tc05::pack_bf16(q0, q1);
        if (FULL) {
          *reinterpret_cast<uint32_t*>(qdz + i * dzs) = q;
        } else {
          if (row && live0) qdz[i * dzs] = (u16)q;
          if (row && live1) qdz[i * dzs + 1] = (u16)(q >> 16);
        }
        dyv = mul2(dyv, l);
      }
      f2 dl, sg = dup(1.f);
      if (RAW) {
        softplus2(bf2(rd[i]), dl, sg);
        if (!FULL) {
          float d0_, d1_;
          up(dl, d0_, d1_);
          dl = pk(row && live0 ? d0_ : 0.f, row && live1 ? d1_ : 0.f);
        }
      } else {
        dl = rf[i];
      }
      *reinterpret_cast<f2*>(&s.dl[t][sc]) = dl;
      *reinterpret_cast<f2*>(&s.sg[t][sc]) = sg;
      *reinterpret_cast<f2*>(&s.u[t][sc]) = uv;
      *reinterpret_cast<f2*>(&s.dy[t][sc]) = dyv;
      dDa = fma2(dyv, uv, dDa);
    }
  };

#pragma unroll 1
  for (int seg = (len - 1) / SEG; seg >= 0; --seg) {
    const int tb = seg * SEG;
    __syncthreads();
    const float* hs = st + ((long long)c * NSEG + seg) * N * a.DiP + d0;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) h[j][k] = __ldg(reinterpret_cast<const f2*>(hs + nn[k] * a.DiP + ch[j]));
    if (vec && tb + SEG <= len) stage(std::true_type(), tb);
    else stage(std::false_type(), tb);
    for (int i = tid; i < SEG * N; i += BT) {
      const int t = i / N, n = i % N;
      const bool ok = tb + t < len;
      const float b = ok ? load_bc(a, a.B, a.bs, row0 + tb + t, n) : 0.f, cc = ok ? load_bc(a, a.C, a.cs, row0 + tb + t, n) : 0.f;
      s.B[t][n] = make_float2(b, b);
      s.C[t][n] = make_float2(cc, cc);
    }
    __syncthreads();
    // states entering steps 4, 8, 12
#pragma unroll 1
    for (int sb = 0; sb < SEG / G - 1; ++sb) {
#pragma unroll
      for (int e = 0; e < 8; ++e) s.ck[sb][e][tid] = h[e >> 2][e & 3];
#pragma unroll
      for (int i = 0; i < G; ++i) {
        const int t = sb * G + i;
        f2 bb[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) bb[k] = lds2(&s.B[t][nn[k]]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const f2 dl = lds2(&s.dl[t][ch[j]]), x = mul2(dl, lds2(&s.u[t][ch[j]]));
#pragma unroll
          for (int k = 0; k < 4; ++k) h[j][k] = fma2(ex2v(mul2(dl, A2[j][k])), h[j][k], mul2(x, bb[k]));
        }
      }
    }
#pragma unroll 1
    for (int sb = SEG / G - 1; sb >= 0; --sb) {
      if (sb < SEG / G - 1) {
#pragma unroll
        for (int e = 0; e < 8; ++e) h[e >> 2][e & 3] = s.ck[sb][e][tid];
      }
      // decay of a step and the state before it: 32 columns of tensor memory a step, a lane a thread
#pragma unroll
      for (int i = 0; i < G; ++i) {
        const int t = sb * G + i;
        union { f2 p[2][2][4]; uint32_t r[32]; } hist;
        f2 bb[4], xb[2][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) bb[k] = lds2(&s.B[t][nn[k]]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const f2 dl = lds2(&s.dl[t][ch[j]]), x = mul2(dl, lds2(&s.u[t][ch[j]]));
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            hist.p[1][j][k] = h[j][k];
            hist.p[0][j][k] = ex2v(mul2(dl, A2[j][k]));
            xb[j][k] = mul2(x, bb[k]);
          }
        }
        tc05::tmem_st_32x32(taddr + i * 32, hist.r);
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int k = 0; k < 4; ++k) h[j][k] = fma2(hist.p[0][j][k], h[j][k], xb[j][k]);
      }
      tc05::tmem_st_wait();
      // back through the four steps.  A step's sums over lanes are formed while the next step's operands are on their way; dC of a
      // step is formed a step late, when the state after it (the next one's state before) has been fetched.
      union { f2 p[2][2][4]; uint32_t r[32]; } hist;
      f2 bb[4], cc[4], dl[2], uu[2], dy[2];
      float vc3[4];                          // the group's last step's
      f2 val[G];
      auto fetch = [&](int i) {
        const int t = sb * G + i;
        tc05::tmem_ld_32x32(taddr + i * 32, hist.r);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          bb[k] = lds2(&s.B[t][nn[k]]);
          cc[k] = lds2(&s.C[t][nn[k]]);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          dl[j] = lds2(&s.dl[t][ch[j]]);
          uu[j] = lds2(&s.u[t][ch[j]]);
        }
      };
#pragma unroll
      for (int j = 0; j < 2; ++j) dy[j] = lds2(&s.dy[sb * G + G - 1][ch[j]]);
      fetch(G - 1);
#pragma unroll
      for (int k = 0; k < 4; ++k) vc3[k] = sum2(fma2(h[1][k], dy[1], mul2(h[0][k], dy[0])));
#pragma unroll
      for (int i = G - 1; i >= 0; --i) {
        const int t = sb * G + i;
        f2 vb[4], s1[2], s2[2], dyb[2];
        float vc[4];
        if (i > 0) {
#pragma unroll
          for (int j = 0; j < 2; ++j) dyb[j] = lds2(&s.dy[t - 1][ch[j]]);
        }
        const f2 fac = lds2(ffac + t * BC), dyf = lds2(&s.dy[t][fch]);
        tc05::tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const f2 x = mul2(dl[j], uu[j]);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const f2 g = fma2(cc[k], dy[j], carry[j][k]);
            vb[k] = j ? fma2(g, x, vb[k]) : mul2(g, x);
            s2[j] = k ? fma2(g, bb[k], s2[j]) : mul2(g, bb[k]);
            carry[j][k] = mul2(hist.p[0][j][k], g);
            const f2 gw = mul2(carry[j][k], hist.p[1][j][k]);
            s1[j] = k ? fma2(gw, A2[j][k], s1[j]) : mul2(gw, A2[j][k]);
            dAa[j][k] = fma2(gw, dl[j], dAa[j][k]);
          }
          s1[j] = fma2(uu[j], s2[j], mul2(s1[j], ln2));
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) vc[k] = i > 0 ? sum2(fma2(hist.p[1][1][k], dyb[1], mul2(hist.p[1][0][k], dyb[0]))) : vc3[k];
        if (i > 0) {
          dy[0] = dyb[0], dy[1] = dyb[1];
          fetch(i - 1);
        }
        // over the channels: states by bits 1 and 0 of cg, dB or dC by bit 2
        float b0 = sum2(vb[0]) + shx(sum2(vb[2]), 8), b1 = sum2(vb[1]) + shx(sum2(vb[3]), 8);
        float c0 = vc[0] + shx(vc[2], 8), c1 = vc[1] + shx(vc[3], 8);
        b0 += shx(b1, 4);
        c0 += shx(c1, 4);
        // over the states: channel pair by bit 1 of q, ddelta or du by bit 0
        float e0, e1, f0, f1, x0, x1;
        up(s1[1], x0, x1);
        up(add2(s1[0], pk(shx(x0, 2), shx(x1, 2))), e0, e1);
        up(s2[1], x0, x1);
        up(add2(s2[0], pk(shx(x0, 2), shx(x1, 2))), f0, f1);
        s.bc[warp][hi ? (i > 0 ? t - 1 : sb * G + G - 1) : t][(hi ? N : 0) + nn[0]] = (hi ? c0 : b0) + shx(hi ? b0 : c0, 16);
        const f2 got = pk(shx(is_du ? e0 : f0, 1), shx(is_du ? e1 : f1, 1));
        val[i] = fma2(add2(pk(is_du ? f0 : e0, is_du ? f1 : e1), got), fac, mul2(Df, dyf));
      }
      if (RAW) {  // the place of the pair's factor, which this group has read, takes both results
        __syncwarp();
#pragma unroll
        for (int i = 0; i < G; ++i) {
          float v0, v1;
          up(val[i], v0, v1);
          reinterpret_cast<uint32_t*>(&s.sg[sb * G + i][fch])[is_du] = tc05::pack_bf16(v0, v1);
        }
      } else {
#pragma unroll
        for (int i = 0; i < G; ++i) {
          const int t = sb * G + i;
          const long long o = (row0 + tb + t) * a.Di + fd;
          float v0, v1;
          up(val[i], v0, v1);
          if (tb + t < len) {
            if (is_du) {
              if (fd < a.Di) du[o] = __float2bfloat16(v0);
              if (fd + 1 < a.Di) du[o + 1] = __float2bfloat16(v1);
            } else {
              if (fd < a.Di) ((float*)ddl)[o] = v0;
              if (fd + 1 < a.Di) ((float*)ddl)[o + 1] = v1;
            }
          }
        }
      }
    }
    __syncthreads();
    if (RAW) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int t = st0 + i, r = tb + t;
        const uint2 v = *reinterpret_cast<const uint2*>(&s.sg[t][sc]);  // ddelta, du
        u16 *p0 = pdd + r * a.Di, *p1 = pdu + r * a.Di;
        if (r < len && live0) {
          if (even) {
            *reinterpret_cast<uint32_t*>(p0) = v.x;
            *reinterpret_cast<uint32_t*>(p1) = v.y;
          } else {
            p0[0] = (u16)v.x, p1[0] = (u16)v.y;
            if (live1) p0[1] = (u16)(v.x >> 16), p1[1] = (u16)(v.y >> 16);
          }
        }
      }
    }
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
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int k = 0; k < 4; ++k) *reinterpret_cast<f2*>(dA + ((long long)c * N + nn[k]) * a.DiP + d0 + ch[j]) = dAa[j][k];
  __syncthreads();
  if (st0) *reinterpret_cast<f2*>(&s.dl[0][sc]) = dDa;
  tc05::tc_fence_before();
  __syncthreads();
  if (!st0) {
    *reinterpret_cast<f2*>(dD + (long long)c * a.DiP + sd) = add2(dDa, lds2(&s.dl[0][sc]));
  }
  if (warp == 0) {
    tc05::tc_fence_after();
    tc05::tmem_dealloc(s.tmem, 32 * G);
  }
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
