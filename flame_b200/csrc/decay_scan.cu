// Chunk states of a decaying outer-product recurrence (GLA, GSA, SSD), increments and recurrence in one launch per direction:
//   forward   out[c] = state entering chunk c:            s = 0;  out[c] = s;  s = alpha[c] s + A_c^T B_c,   c ascending
//   reverse   out[c] = adjoint of the state leaving c:    s = 0;  out[c] = s;  s = alpha[c] s + A_c^T B_c,   c descending
// A_c [64, rows] and B_c [64, cols] are a chunk's tokens of one head (keys and values, or queries and output gradients), bf16; the state
// is fp32, what leaves is bf16; alpha is one decay per state row, or one per head.
//
// A CTA walks one document's chunks for one head and 64 columns.  The increments do not depend on the state, so their products run
// ahead through a ring of TMA stages and two accumulators; a thread owns a state row, 64 fp32 registers, adds the
// accumulator's row to it and sends the bf16 copy out by TMA.  What bounds it is memory: operands once, states once.  As a
// product that wrote the increments (fp32 forward, bf16 backward) and a scan that read them, at 65,536 tokens, 4 heads of
// 128 x 256: 0.25 ms forward, 0.17 backward and 0.10 for the decay's gradient (the sums of state times adjoint, for which both were
// read again); this: 0.10 and 0.15 with the gradient.
// Stands in for fla/ops/common/chunk_h.py.
#include "tc05.cuh"
#include "host_utils.cuh"

using namespace tc05;

namespace {

constexpr int C = 64;        // tokens per chunk
constexpr int W = 64;        // columns per CTA
constexpr int THREADS = 192; // warp 0 TMA, warp 1 MMA, warps 2..5 the state: warp w has rows 32 (w & 3) .. (two warps for 32 rows, half of
                             // the columns each, took the same time)

struct DecayScanParams {
  const int* first;          // [n_docs] first chunk of every document
  const int* last;           // [n_docs] last chunk
  int H, a_div, b_div;       // heads; consecutive heads that share a head of A, of B
  int reverse, per_row;
  const float* alpha;        // [NC, H] or [NC, H, rows]
  float* part;               // DOT: [slices, NC, H, rows] (per_row) or [slices * rows / 32, NC, H]
  long long part_step;       // NC H rows, or NC H
  int* status;
};

// DOT (reverse): the states that the forward left come back in, and their products with the adjoints are summed
template <int R, bool DOT>
struct Smem {
  static constexpr int STAGES = R == 64 ? 4 : DOT ? 2 : 3;
  static constexpr int A_BYTES = C * R * 2;              // groups of [64 tokens][64 rows of the state]
  static constexpr int STAGE_BYTES = A_BYTES + C * W * 2;
  static constexpr int BOX_BYTES = 32 * W * 2;           // 32 rows x 64 columns bf16, OUT per warp, and two to come in
  static constexpr int OUT = DOT && R == 128 ? 1 : 2;    // two do not fit beside another CTA
  static constexpr int BOXES = OUT + (DOT ? 2 : 0);
  static constexpr int BOX_OFF = STAGES * STAGE_BYTES;
  static constexpr int BAR_OFF = BOX_OFF + (R / 32) * BOXES * BOX_BYTES;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

template <int R, bool DOT>
__global__ void __launch_bounds__(THREADS, 2)
decay_scan_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmOut,
                  const __grid_constant__ CUtensorMap tmS, const DecayScanParams p) {
  using L = Smem<R, DOT>;
  constexpr int STAGES = L::STAGES;
  const int vt = blockIdx.x, head = blockIdx.y, doc = blockIdx.z;
  const int c_first = p.first[doc], c_last = p.last[doc], cnt = c_last - c_first + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto chunk = [&](int i) { return p.reverse ? c_last - i : c_first + i; };

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full_bar = (uint64_t*)(smem + L::BAR_OFF);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint64_t* in_bar = tempty_bar + 2;  // DOT: two per warp of the state
  uint32_t* tmem_slot = (uint32_t*)(in_bar + 8);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], R / 32);
    }
    for (int b = 0; b < 8; ++b) mbar_init(&in_bar[b], 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmOut);
    if (DOT) tma_prefetch_desc(&tmS);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * W);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      const int ha = head / p.a_div, hb = head / p.b_div;
      for (int i = 0; i < cnt - 1; ++i) {  // the last chunk's increment goes nowhere
        const int stage = i % STAGES;
        if (!mbar_wait(&empty_bar[stage], ((i / STAGES) & 1) ^ 1, p.status, abort_flag, ERR_WAIT_EMPTY)) break;
        uint8_t* dst = smem + stage * L::STAGE_BYTES;
        mbar_expect_tx(&full_bar[stage], L::STAGE_BYTES);
#pragma unroll
        for (int g = 0; g < R / 64; ++g) tma_load_4d(dst + g * (C * 128), &tmA, &full_bar[stage], g * 64, 0, ha, chunk(i));
        tma_load_4d(dst + L::A_BYTES, &tmB, &full_bar[stage], vt * W, 0, hb, chunk(i));
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // both operands have tokens as K and lie MN-major.  With 64 rows the product's upper 64 rows read what follows A (B's tile,
      // inside the stage); nobody reads them
      constexpr uint32_t idesc = make_idesc_bf16(128, W, 1, 1);
      for (int i = 0; i < cnt - 1; ++i) {
        const int stage = i % STAGES, acc = i & 1;
        if (!mbar_wait(&tempty_bar[acc], ((i >> 1) & 1) ^ 1, p.status, abort_flag, ERR_WAIT_TMEM_EMPTY)) break;
        if (!mbar_wait(&full_bar[stage], (i / STAGES) & 1, p.status, abort_flag, ERR_WAIT_FULL)) break;
        tc_fence_after();
        const uint32_t sA = smem_u32(smem + stage * L::STAGE_BYTES);
        const uint64_t ad = make_smem_desc(sA, C * 128, 1024), bd = make_smem_desc(sA + L::A_BYTES, C * 128, 1024);
#pragma unroll
        for (int k = 0; k < C / 16; ++k)
          mma_ss(tmem_base + acc * W, desc_advance(ad, k * 2048), desc_advance(bd, k * 2048), idesc, k ? 1u : 0u);
        mma_commit(&empty_bar[stage]);
        mma_commit(&tfull_bar[acc]);
      }
    }
  } else if ((warp & 3) * 32 < R) {
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const bool lead = lane == 0;
    const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
    uint8_t* boxes = smem + L::BOX_OFF + quarter * L::BOXES * L::BOX_BYTES;
    auto state_row = [&](int i) { return (chunk(i) * p.H + head) * R + quarter * 32; };
    int fetched = 0;
    auto fetch = [&](int i) {  // the forward's state of chunk(i)
      if (i >= cnt) return;
      ++fetched;
      uint64_t* bar = &in_bar[quarter * 2 + (i & 1)];
      mbar_expect_tx(bar, L::BOX_BYTES);
      tma_load_2d(boxes + (L::OUT + (i & 1)) * L::BOX_BYTES, &tmS, bar, vt * W, state_row(i));
    };
    if (DOT && lead) fetch(0), fetch(1);
    auto decay = [&](int i) {
      const long long at = (long long)chunk(min(i, cnt - 1)) * p.H + head;
      return __ldg(p.alpha + (p.per_row ? at * R + row : at));
    };
    float s[W];
#pragma unroll
    for (int j = 0; j < W; ++j) s[j] = 0.f;
    float a0 = decay(0), a1 = decay(1);
    bool ok = true;
    for (int i = 0; i < cnt; ++i) {
      const float a2 = decay(i + 2);
      uint8_t* box = boxes + (i & (L::OUT - 1)) * L::BOX_BYTES;
      if (lead) tma_store_wait_read<L::OUT - 1>();  // the last state in this box has left it
      __syncwarp();
      uint32_t s16[W / 2];
#pragma unroll
      for (int j = 0; j < W / 2; ++j) s16[j] = pack_bf16(s[2 * j], s[2 * j + 1]);
#pragma unroll
      for (int j = 0; j < W / 8; ++j)
        *reinterpret_cast<uint4*>(box + lane * 128 + ((j ^ (lane & 7)) << 4)) =
            make_uint4(s16[4 * j], s16[4 * j + 1], s16[4 * j + 2], s16[4 * j + 3]);
      fence_async_smem();
      __syncwarp();
      if (lead) {
        tma_store_2d(&tmOut, box, vt * W, state_row(i));
        tma_store_commit();
      }
      if (DOT) {
        ok = mbar_wait_warp(&in_bar[quarter * 2 + (i & 1)], (i >> 1) & 1, p.status, abort_flag, ERR_WAIT_MISC);
        if (!ok) break;
        const uint8_t* in = boxes + (L::OUT + (i & 1)) * L::BOX_BYTES;
        // of the rounded adjoint, the one that the other gradients see: parts of the gate's gradient cancel
        float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < W / 8; ++j) {
          const uint4 v = *reinterpret_cast<const uint4*>(in + lane * 128 + ((j ^ (lane & 7)) << 4));
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const uint32_t v16 = s16[4 * j + e];
            d[e] = fmaf(__uint_as_float(v16 << 16), __uint_as_float(w[e] << 16), d[e]);
            d[e] = fmaf(__uint_as_float(v16 & 0xffff0000u), __uint_as_float(w[e] & 0xffff0000u), d[e]);
          }
        }
        float d0 = (d[0] + d[1]) + (d[2] + d[3]);
        const long long at = (long long)chunk(i) * p.H + head;
        if (p.per_row) {
          p.part[vt * p.part_step + at * R + row] = d0;
        } else {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) d0 += __shfl_xor_sync(0xffffffffu, d0, o);
          if (lane == 0) p.part[(vt * (R / 32) + quarter) * p.part_step + at] = d0;
        }
        __syncwarp();
        if (lead) fetch(i + 2);                 // its box has been read
      }
      if (i + 1 == cnt) break;
      const int acc = i & 1;
      ok = mbar_wait_warp(&tfull_bar[acc], (i >> 1) & 1, p.status, abort_flag, ERR_WAIT_TMEM_FULL);
      if (!ok) break;
      tc_fence_after();
      uint32_t x[W];
      tmem_ld_32x32(t_row + acc * W, *reinterpret_cast<uint32_t(*)[32]>(&x[0]));
      tmem_ld_32x32(t_row + acc * W + 32, *reinterpret_cast<uint32_t(*)[32]>(&x[32]));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty_bar[acc]);
#pragma unroll
      for (int j = 0; j < W; ++j) s[j] = fmaf(a0, s[j], __uint_as_float(x[j]));
      a0 = a1, a1 = a2;
    }
    if (lead) {
      tma_store_wait_all<0>();
      // every copy has landed (a wait that has passed returns at once): nothing may land in this shared memory once it belongs to
      // another block
      if (DOT && !ok)
        for (int k = max(fetched - 2, 0); k < fetched; ++k)
          for (int tries = 0; tries < 50000 && !mbar_try_wait(&in_bar[quarter * 2 + (k & 1)], (k >> 1) & 1); ++tries) {}
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * W);
  }
}

template <int R, bool DOT>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& to, const CUtensorMap& ts, const DecayScanParams& p, int cols,
           int n_docs, cudaStream_t stream) {
  auto kern = decay_scan_kernel<R, DOT>;
  constexpr int TOTAL = Smem<R, DOT>::TOTAL;
  static bool configured = false;
  if (!configured) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TOTAL);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  kern<<<dim3(cols / W, p.H, n_docs), THREADS, TOTAL, stream>>>(ta, tb, to, ts, p);
  return fb::launch_ok("decay_scan_kernel");
}

}  // namespace

extern "C" {

// A [NC, Ha, 64, rows] and B [NC, Hb, 64, cols] bf16, inner contiguous, any other strides of whole 16-byte vectors (elements), Ha and
// Hb dividing H; out [NC, H, rows, cols] bf16 contiguous; alpha fp32 [NC, H], or with per_row [NC, H, rows]; first / last [n_docs]
// chunk indices.  S (or null) as out, with part: the sums of S out over the columns, [cols / 64, NC, H, rows] if per_row, else over the rows
// too, [cols / 64 * rows / 32, NC, H]; the caller adds up the first dimension.  rows 64 or 128, cols a multiple of 64; at most 65,535 documents and heads (-2 otherwise, and for misaligned operands).
int fb_decay_scan(const void* A, long long a_ld, long long a_lo, long long a_hi, int Ha, const void* B, long long b_ld, long long b_lo,
                  long long b_hi, int Hb, const float* alpha, int per_row, void* out, const void* S, float* part, const int* first, const int* last, int n_docs, int H,
                  int NC, int rows, int cols, int reverse, cudaStream_t stream) {
  if (n_docs <= 0 || NC <= 0 || H <= 0 || cols <= 0) return 0;
  if ((rows != 64 && rows != 128) || cols % W || Ha <= 0 || Hb <= 0 || H % Ha || H % Hb || n_docs > 65535 || H > 65535) return -2;
  if (((a_ld | a_lo | a_hi | b_ld | b_lo | b_hi) & 7) || !fb::aligned(16, A, B, out, S)) return -2;
  if ((long long)NC * H * rows > 0x7fffffffll) return -2;  // rows of the states' tensor map
  CUtensorMap ta, tb, to, ts;
  int rc = fb::make_tmap_4d(&ta, A, 2, NC, Ha, C, rows, a_hi, a_lo, a_ld, C, 64, true);
  if (rc) return rc;
  rc = fb::make_tmap_4d(&tb, B, 2, NC, Hb, C, cols, b_hi, b_lo, b_ld, C, 64, true);
  if (rc) return rc;
  rc = fb::make_tmap_2d(&to, out, 2, (uint64_t)NC * H * rows, cols, cols, 32, W, true);
  if (rc) return rc;
  ts = to;
  if (S) {
    rc = fb::make_tmap_2d(&ts, S, 2, (uint64_t)NC * H * rows, cols, cols, 32, W, true);
    if (rc) return rc;
  }
  DecayScanParams p;
  p.part = part; p.part_step = (long long)NC * H * (per_row ? rows : 1);
  p.first = first; p.last = last; p.H = H; p.a_div = H / Ha; p.b_div = H / Hb;
  p.reverse = reverse; p.per_row = per_row; p.alpha = alpha; p.status = fb::status_ptr();
  if (S)
    return rows == 64 ? launch<64, true>(ta, tb, to, ts, p, cols, n_docs, stream) : launch<128, true>(ta, tb, to, ts, p, cols, n_docs, stream);
  return rows == 64 ? launch<64, false>(ta, tb, to, ts, p, cols, n_docs, stream) : launch<128, false>(ta, tb, to, ts, p, cols, n_docs, stream);
}

}  // extern "C"
