// Batched bf16 GEMM for the chunk-parallel token mixers (linear attention, delta rule, SSD):
//
//   C[b] = epilogue( alpha * sum_i (+-) A_i[b] * B_i[b]^T )      b = (hi, lo) = (chunk, head), up to six products i
//
// Thousands of small problems (64 x 64 x dk score blocks, dk x dv chunk states, 64 x dv outputs) run as ONE persistent
// launch: every operand is a 4-D tensor map (inner, row, lo, hi), so a tile of any batch is a TMA box and the batch
// coordinates come from the work-unit index (optionally through an index table, which is how the chunk-by-chunk state
// recurrence of documents with different lengths addresses "chunk s of every document that has one").  The main loop is
// the single-CTA tcgen05 pipeline of gemm.cu (TMA warp, MMA warp, epilogue warps, two or four TMEM accumulators); the
// several products of one result (the state's and the scores' share of an output, the terms of a gradient) accumulate in
// tensor memory one after the other, so that no partial result is written and read back.  The
// epilogue adds what the chunk algorithms need so no elementwise pass follows the GEMM:
//   * causal masks (keep col <= row, or col < row),
//   * a decay factor exp(d[row] - d[col]) from a per-batch fp32 vector (scalar-gated attention scores), a factor per row,
//   * the state step   C = alpha * acc + gamma[b] * Cin[b'] + add16[b''] (+ C)   with a bf16 copy of the result written
//     to a batch of its own (C may be its own Cin: an fp32 state updated in place, small enough to stay in L2).
//
// Stands in for the tl.dot bodies of the reference's Triton chunk kernels (fla/ops/common/chunk_h.py,
// fla/ops/common/chunk_o.py, fla/ops/gated_delta_rule/wy_fast.py, fla/ops/common/chunk_scaled_dot_kkt.py).
#include "tc05.cuh"
#include "host_utils.cuh"

using namespace tc05;

namespace {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int MAX_STAGES = 8;
// warp 0 TMA, warp 1 MMA, warps 2..9 epilogue: two warps per TMEM lane quarter, each taking half of the tile's columns.
// The chunk algorithms' problems mostly have 64 rows, which live in two lane quarters only; with one warp per quarter
// two warps would drain every accumulator and the epilogue, not memory, would set the pace.
constexpr int BGEMM_THREADS = 320;
// A work unit of the chunk algorithms is one to four K blocks, so a CTA spends its time in hand-offs between its warps: tiles of
// at most 128 columns leave room for two CTAs per SM (half of tensor memory and of shared memory each), whose chains overlap.
constexpr int MAX_BN = 128;
constexpr int TMEM_COLS = 256;
// Shared memory of a CTA: the ring, and where results leave by TMA 4 KB for every epilogue warp that has rows.
constexpr int MAIN_BYTES = 104 * 1024;
constexpr int STG_BYTES = 4096;

struct BOperandIdx {
  const int* hi_index;  // optional: hi coordinate = hi_index[hi_raw]
  int hi_offset;        // added to the hi coordinate
  int lo_div;           // lo coordinate = lo / lo_div (grouped value heads)
};

constexpr int MAX_PAIRS = 6;

struct BPair {
  BOperandIdx a, b;
  int num_kb, a_mn, b_mn, neg;
};

struct BMaps {
  CUtensorMap a[MAX_PAIRS], b[MAX_PAIRS];
  CUtensorMap c, add;  // TMA_OUT: boxes of 32 rows x 128 bytes of the result and of the bf16 addend
};

struct BGemmParams {
  int M, N;
  int tiles_m, tiles_n, n_pairs, bn;
  int sum_lo;          // every product is summed over this many lo coordinates (the heads of a group): lo * sum_lo + 0, 1, ..
  BPair pair[MAX_PAIRS];
  int a_rows, stages;  // rows of the A box (64 when M <= 64: the tile's other rows are never looked at), depth of the ring
  int n_lo, n_batch;
  BOperandIdx c, cin, c16i, add16i;
  void* C;
  long long ldc, c_stride_lo, c_stride_hi;
  const float* Cin;    // optional fp32 addend, same layout as C (may BE C: in-place state), scaled by gamma[hi(A) * n_lo + lo]
  const float* gamma;
  // bf16 side tensors of the fp32 modes, sharing one layout (ld16, stride_lo16, stride_hi16) but with hi coordinates of
  // their own: C16 receives a bf16 copy of the result, add16 is added to it
  __nv_bfloat16* C16;
  const __nv_bfloat16* add16;
  long long ld16, stride_lo16, stride_hi16;
  const float* decay;  // optional: value *= exp(decay[row] - decay[col]); element (hi, lo, r) at hi*d_hi + lo*d_lo + r*d_r
  long long d_hi, d_lo, d_r;
  const float* rowscale;  // optional: value *= rowscale[row], element (hi, lo, r) at hi*r_hi + lo*r_lo + r*r_r
  long long r_hi, r_lo, r_r;
  float alpha;
  int out_mode;        // 0 bf16 store, 1 fp32 store, 2 fp32 accumulate
  int mask_mode;       // 0 none, 1 keep col <= row, 2 keep col < row
  int stg_offset;      // TMA_OUT: the epilogue warps' boxes begin here
  int arrivals;        // epilogue warps that drain an accumulator
  int* status;
};

struct Smem {
  static constexpr int BAR_OFFSET = MAIN_BYTES;
  static constexpr int TOTAL = BAR_OFFSET + 512 + 1024;
};

struct Unit {
  int hi_raw, lo, tm, tn;
};

__device__ __forceinline__ Unit decode(const BGemmParams& p, int unit) {
  Unit u;
  const int per_batch = p.tiles_m * p.tiles_n;
  const int batch = unit / per_batch;
  const int r = unit - batch * per_batch;
  u.tn = r / p.tiles_m;
  u.tm = r - u.tn * p.tiles_m;
  u.hi_raw = batch / p.n_lo;
  u.lo = batch - u.hi_raw * p.n_lo;
  return u;
}
// The unit `step` (a decoded distance) further on, without divisions.
__device__ __forceinline__ void advance(const BGemmParams& p, Unit& u, const Unit& step) {
  u.tm += step.tm;
  u.tn += step.tn;
  u.lo += step.lo;
  u.hi_raw += step.hi_raw;
  if (u.tm >= p.tiles_m) u.tm -= p.tiles_m, ++u.tn;
  if (u.tn >= p.tiles_n) u.tn -= p.tiles_n, ++u.lo;
  if (u.lo >= p.n_lo) u.lo -= p.n_lo, ++u.hi_raw;
}
__device__ __forceinline__ int lo_of(const BOperandIdx& o, int lo) { return o.lo_div == 1 ? lo : lo / o.lo_div; }
__device__ __forceinline__ int hi_of(const BOperandIdx& o, int hi_raw) {
  return (o.hi_index != nullptr ? o.hi_index[hi_raw] : hi_raw) + o.hi_offset;
}

// TMA_OUT: each epilogue warp puts 32 rows x 128 bytes of the result into shared memory and one thread hands them to the TMA
// unit (the accumulating mode adds in L2, a bf16 addend comes in the same way while the products are formed).  Results with a
// state step, a hi index or a layout that has no tensor map are stored row by row: a warp's 16-byte stores to 32 different
// rows then take the load/store unit 64 cycles each, and that unit, not memory, set the pace (a unit of 128 x 128 took 13,000
// clocks in two CTAs, 8,200 of them in these stores).  The ten to twenty-five launches of a layer's forward and backward,
// row by row and by TMA: DeltaNet 3.77 -> 1.90 ms (65,536 tokens, 8 heads of 128), GLA 1.79 -> 0.84, GSA 1.49 -> 0.66, Mamba2
// 2.38 -> 1.06, Gated DeltaNet 2.14 -> 1.28.
template <bool TMA_OUT>
__global__ void __launch_bounds__(BGEMM_THREADS, 2)
bgemm_bf16_kernel(const __grid_constant__ BMaps maps, const __grid_constant__ BGemmParams p) {
  using L = Smem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full_bar = (uint64_t*)(smem + L::BAR_OFFSET);
  uint64_t* empty_bar = full_bar + MAX_STAGES;
  uint64_t* tfull_bar = empty_bar + MAX_STAGES;
  uint64_t* tempty_bar = tfull_bar + 4;
  uint64_t* stg_bar = tempty_bar + 4;
  uint32_t* tmem_slot = (uint32_t*)(stg_bar + 8);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int total_units = p.n_batch * p.tiles_m * p.tiles_n;
  const int BN = p.bn, STAGES = p.stages;
  const int a_bytes = p.a_rows * BK * 2;
  const int stage_bytes = a_bytes + BN * BK * 2;
  const int n_acc = TMEM_COLS / BN;  // accumulators in flight: 2 (BN = 128) or 4

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < n_acc; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], p.arrivals);
    }
    for (int w = 0; w < 8; ++w) mbar_init(&stg_bar[w], 1);
    *abort_flag = 0;
    mbar_fence_init();
    for (int i = 0; i < p.n_pairs; ++i) {
      tma_prefetch_desc(&maps.a[i]);
      tma_prefetch_desc(&maps.b[i]);
    }
    if (TMA_OUT) tma_prefetch_desc(&maps.c);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      Unit u = decode(p, blockIdx.x);
      const Unit step = decode(p, gridDim.x);
      for (int unit = blockIdx.x; unit < total_units && ok; unit += gridDim.x, advance(p, u, step)) {
        for (int i = 0; i < p.n_pairs && ok; ++i) {
          const BPair& pr = p.pair[i];
          const int a_hi = hi_of(pr.a, u.hi_raw), b_hi = hi_of(pr.b, u.hi_raw);
          for (int sk = 0, kb = 0, lo = u.lo * p.sum_lo; sk < p.sum_lo * pr.num_kb; ++sk) {
            const int a_lo = lo_of(pr.a, lo), b_lo = lo_of(pr.b, lo);
            if (!mbar_wait(&empty_bar[stage], phase ^ 1, p.status, abort_flag, ERR_WAIT_EMPTY)) { ok = false; break; }
            uint8_t* sA = smem + stage * stage_bytes;
            uint8_t* sB = sA + a_bytes;
            mbar_expect_tx(&full_bar[stage], (uint32_t)stage_bytes);
            if (!pr.a_mn) {
              tma_load_4d(sA, &maps.a[i], &full_bar[stage], kb * BK, u.tm * BM, a_lo, a_hi);
            } else {
              for (int g = 0; g < p.a_rows / 64; ++g)
                tma_load_4d(sA + g * (64 * BK * 2), &maps.a[i], &full_bar[stage], u.tm * BM + g * 64, kb * BK, a_lo, a_hi);
            }
            if (!pr.b_mn) {
              tma_load_4d(sB, &maps.b[i], &full_bar[stage], kb * BK, u.tn * BN, b_lo, b_hi);
            } else {
              for (int g = 0; g < BN / 64; ++g)
                tma_load_4d(sB + g * (64 * BK * 2), &maps.b[i], &full_bar[stage], u.tn * BN + g * 64, kb * BK, b_lo, b_hi);
            }
            if (++kb == pr.num_kb) { kb = 0; ++lo; }
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int unit = blockIdx.x; unit < total_units && ok; unit += gridDim.x) {
        if (!mbar_wait(&tempty_bar[acc], acc_phase ^ 1, p.status, abort_flag, ERR_WAIT_TMEM_EMPTY)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        bool first = true;
        for (int i = 0; i < p.n_pairs && ok; ++i) {
          const BPair& pr = p.pair[i];
          const uint32_t idesc = make_idesc_bf16(BM, BN, pr.a_mn, pr.b_mn) | (pr.neg ? 1u << 13 : 0u);  // bit 13: negate A
          const uint32_t a_lbo = pr.a_mn ? 64 * BK * 2 : 16, b_lbo = pr.b_mn ? 64 * BK * 2 : 16;
          const uint32_t a_kstep = pr.a_mn ? 16 * 128 : 32, b_kstep = pr.b_mn ? 16 * 128 : 32;
          for (int kb = 0; kb < p.sum_lo * pr.num_kb; ++kb) {
            if (!mbar_wait(&full_bar[stage], phase, p.status, abort_flag, ERR_WAIT_FULL)) { ok = false; break; }
            tc_fence_after();
            const uint32_t sA = smem_u32(smem + stage * stage_bytes);
            const uint32_t sB = sA + a_bytes;
            const uint64_t adesc = make_smem_desc(sA, a_lbo, 1024);
            const uint64_t bdesc = make_smem_desc(sB, b_lbo, 1024);
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              mma_ss(d_tmem, desc_advance(adesc, k * a_kstep), desc_advance(bdesc, k * b_kstep), idesc, (!first || k > 0) ? 1u : 0u);
            first = false;
            mma_commit(&empty_bar[stage]);
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
          }
        }
        if (ok) mma_commit(&tfull_bar[acc]);
        if (++acc == n_acc) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else if constexpr (TMA_OUT) {
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    // Tiles of 128 columns: the two warps of a lane quarter take half of the columns each.  Tiles of 64: every second unit, so
    // that a box of the result is 128 bytes wide there too.  Either way a warp drains two groups of 32 columns.
    const bool alt = BN == 64;
    const int c_begin = alt ? 0 : half * 64;
    const bool b16 = p.out_mode == 0, add = p.add16 != nullptr;
    int acc = 0, n = 0;
    uint32_t acc_phase = 0, stg_phase = 0;
    bool ok = quarter * 32 < p.a_rows;  // warps of rows that the tile does not have
    const int slot = half * (p.a_rows >> 5) + quarter;
    uint8_t* stg = smem + p.stg_offset + (ok ? slot : 0) * STG_BYTES;
    uint64_t* my_bar = &stg_bar[warp - 2];
    auto at = [&](int chunk) { return stg + lane * 128 + ((chunk ^ (lane & 7)) << 4); };  // the 128-byte swizzle of the maps
    Unit u = decode(p, blockIdx.x);
    const Unit step = decode(p, gridDim.x);
    for (int unit = blockIdx.x; unit < total_units && ok; unit += gridDim.x, advance(p, u, step), ++n) {
      if (!alt || (n & 1) == half) {
        const int row0 = u.tm * BM + quarter * 32, row = row0 + lane, colw = u.tn * BN + c_begin;
        const bool any = row0 < p.M && colw < p.N;
        if (add && any && lane == 0) {
          tma_store_wait_read<0>();
          mbar_expect_tx(my_bar, STG_BYTES);
          tma_load_4d(stg, &maps.add, my_bar, colw, row0, u.lo, u.hi_raw + p.add16i.hi_offset);
        }
        float scale = p.alpha, dec_row = 0.f;
        const float* dec = nullptr;
        if (p.rowscale != nullptr && row < p.M)
          scale *= p.rowscale[(long long)u.hi_raw * p.r_hi + (long long)u.lo * p.r_lo + (long long)row * p.r_r];
        if (p.decay != nullptr) {
          dec = p.decay + (long long)u.hi_raw * p.d_hi + (long long)u.lo * p.d_lo;
          if (row < p.M) dec_row = dec[(long long)row * p.d_r];
        }
        if (!mbar_wait_warp(&tfull_bar[acc], acc_phase, p.status, abort_flag, ERR_WAIT_TMEM_FULL)) { ok = false; break; }
        tc_fence_after();
        const uint32_t t_row = tmem_base + acc * BN + ((uint32_t)(quarter * 32) << 16) + c_begin;
#pragma unroll 1
        for (int k = 0; k < 2; ++k) {
          const int col = colw + 32 * k;
          const bool live = any && col < p.N;  // warp-uniform
          uint32_t r[32];
          float dec_col = 0.f;
          if (live) {
            tmem_ld_32x32(t_row + 32 * k, r);
            if (dec != nullptr && col + lane < p.N) dec_col = dec[(long long)(col + lane) * p.d_r];
            if (!b16 || k == 0) {  // the box is free: its last store has been read, or the addend has come
              if (add) {
                if (!mbar_wait_warp(my_bar, stg_phase, p.status, abort_flag, ERR_WAIT_TMEM_FULL)) ok = false;
                stg_phase ^= 1;
              } else {
                if (lane == 0) tma_store_wait_read<0>();
                __syncwarp();
              }
            }
            tmem_ld_wait();
          }
          if (k == 1) {  // everything is in registers
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty_bar[acc]);
          }
          if (!live) continue;
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * scale);
          if (dec != nullptr) {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float dj = __shfl_sync(0xffffffffu, dec_col, j);
              // masked entries may have a positive exponent: they are dropped, never multiplied
              const bool keep = p.mask_mode == 0 || (p.mask_mode == 1 ? col + j <= row : col + j < row);
              r[j] = keep ? __float_as_uint(__uint_as_float(r[j]) * __expf(dec_row - dj)) : 0u;
            }
          } else if (p.mask_mode != 0) {
            const int first_out = row - col + (p.mask_mode == 1 ? 1 : 0);  // the first column that is dropped
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j >= first_out) r[j] = 0u;
          }
          if (b16) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4* dst = reinterpret_cast<uint4*>(at(4 * k + j));
              if (add) {  // v_new = u - w S, o = q S + A v
                const uint4 a4 = *dst;
                const uint32_t w4[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                  r[8 * j + 2 * t] = __float_as_uint(__uint_as_float(r[8 * j + 2 * t]) + __uint_as_float(w4[t] << 16));
                  r[8 * j + 2 * t + 1] = __float_as_uint(__uint_as_float(r[8 * j + 2 * t + 1]) + __uint_as_float(w4[t] & 0xffff0000u));
                }
              }
              uint4 q;
              q.x = pack_bf16(__uint_as_float(r[8 * j]), __uint_as_float(r[8 * j + 1]));
              q.y = pack_bf16(__uint_as_float(r[8 * j + 2]), __uint_as_float(r[8 * j + 3]));
              q.z = pack_bf16(__uint_as_float(r[8 * j + 4]), __uint_as_float(r[8 * j + 5]));
              q.w = pack_bf16(__uint_as_float(r[8 * j + 6]), __uint_as_float(r[8 * j + 7]));
              *dst = q;
            }
            if (k == 0 && col + 32 < p.N) continue;  // the box's other half follows
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<uint4*>(at(j)) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) {
            const int x = b16 ? colw : col, hi = u.hi_raw + p.c.hi_offset;
            if (p.out_mode == 2) tma_reduce_add_4d(&maps.c, stg, x, row0, u.lo, hi);
            else tma_store_4d(&maps.c, stg, x, row0, u.lo, hi);
            tma_store_commit();
          }
        }
      }
      if (++acc == n_acc) { acc = 0; acc_phase ^= 1; }
    }
    if (lane == 0) tma_store_wait_all<0>();
  } else {
    const int quarter = warp & 3;
    // two warps per lane quarter, each takes half of the tile's columns (tiles are 64 or 128 wide)
    const int half = (warp - 2) >> 2;
    const int c_begin = half * (BN / 2), c_end = c_begin + BN / 2;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int unit = blockIdx.x; unit < total_units && ok; unit += gridDim.x) {
      const Unit u = decode(p, unit);
      if (!mbar_wait_warp(&tfull_bar[acc], acc_phase, p.status, abort_flag, ERR_WAIT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      const int row = u.tm * BM + quarter * 32 + lane;
      const bool row_ok = row < p.M;
      const uint32_t t_row = tmem_base + acc * BN + ((uint32_t)(quarter * 32) << 16);
      const long long c_base = (long long)hi_of(p.c, u.hi_raw) * p.c_stride_hi + (long long)(u.lo / p.c.lo_div) * p.c_stride_lo +
                               (long long)row * p.ldc;
      const float* cin_row = nullptr;
      float gamma = 0.f;
      if (p.Cin != nullptr) {
        cin_row = p.Cin + (long long)hi_of(p.cin, u.hi_raw) * p.c_stride_hi + (long long)(u.lo / p.cin.lo_div) * p.c_stride_lo +
                  (long long)row * p.ldc;
        gamma = p.gamma != nullptr ? p.gamma[(long long)hi_of(p.pair[0].a, u.hi_raw) * p.n_lo + u.lo] : 1.f;
      }
      const long long lo16 = (long long)(u.lo / p.c.lo_div) * p.stride_lo16 + (long long)row * p.ld16;
      __nv_bfloat16* c16_row = p.C16 != nullptr ? p.C16 + (long long)hi_of(p.c16i, u.hi_raw) * p.stride_hi16 + lo16 : nullptr;
      const __nv_bfloat16* add_row = p.add16 != nullptr ? p.add16 + (long long)hi_of(p.add16i, u.hi_raw) * p.stride_hi16 + lo16 : nullptr;
      const float* dec = nullptr;
      float dec_row = 0.f;
      if (p.decay != nullptr) {
        dec = p.decay + (long long)u.hi_raw * p.d_hi + (long long)u.lo * p.d_lo;
        if (row_ok) dec_row = dec[(long long)row * p.d_r];
      }
      float scale = p.alpha;
      if (p.rowscale != nullptr && row_ok)
        scale *= p.rowscale[(long long)u.hi_raw * p.r_hi + (long long)u.lo * p.r_lo + (long long)row * p.r_r];
#pragma unroll 1
      for (int c = c_begin; c < c_end; c += 32) {
        const int col0 = u.tn * BN + c;
        if (col0 >= p.N) break;  // warp-uniform
        uint32_t r[32];
        tmem_ld_32x32(t_row + c, r);
        const bool full = (col0 + 32 <= p.N);
        const bool vec = full && row_ok;
        // the addend (or, in the accumulating mode, the old result: never both in registers) is fetched while the
        // accumulator comes in
        uint4 side[8];
        float dec_col = 0.f;
        if (vec && p.out_mode == 2) {
#pragma unroll
          for (int j = 0; j < 8; ++j) side[j] = *reinterpret_cast<const uint4*>((const float*)p.C + c_base + col0 + 4 * j);
        } else if (vec && add_row != nullptr) {
#pragma unroll
          for (int j = 0; j < 4; ++j) side[j] = *reinterpret_cast<const uint4*>(add_row + col0 + 8 * j);
        }
        if (dec != nullptr && col0 + lane < p.N) dec_col = dec[(long long)(col0 + lane) * p.d_r];
        tmem_ld_wait();
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]) * scale;
        if (dec != nullptr) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int col = col0 + j;
            const float dj = __shfl_sync(0xffffffffu, dec_col, j);  // before any lane leaves
            // masked entries may have a positive exponent: they are dropped, never multiplied
            const bool keep = col < p.N && (p.mask_mode == 0 || (p.mask_mode == 1 ? col <= row : col < row));
            v[j] = keep ? v[j] * __expf(dec_row - dj) : 0.f;
          }
        } else if (p.mask_mode != 0) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int col = col0 + j;
            if (!(p.mask_mode == 1 ? col <= row : col < row)) v[j] = 0.f;
          }
        }
        if (!row_ok) continue;
        if (p.out_mode == 0) {
          __nv_bfloat16* dst = (__nv_bfloat16*)p.C + c_base + col0;
          if (add_row != nullptr) {  // bf16 result with a bf16 addend (v_new = u - w S, o = q S + A v)
            if (full) {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const uint32_t w4[4] = {side[j].x, side[j].y, side[j].z, side[j].w};
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                  v[8 * j + 2 * t] += __uint_as_float(w4[t] << 16);
                  v[8 * j + 2 * t + 1] += __uint_as_float(w4[t] & 0xffff0000u);
                }
              }
            } else {
              for (int j = 0; j < 32; ++j)
                if (col0 + j < p.N) v[j] += __bfloat162float(add_row[col0 + j]);
            }
          }
          if (full) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              uint4 q;
              q.x = pack_bf16(v[j], v[j + 1]);
              q.y = pack_bf16(v[j + 2], v[j + 3]);
              q.z = pack_bf16(v[j + 4], v[j + 5]);
              q.w = pack_bf16(v[j + 6], v[j + 7]);
              *reinterpret_cast<uint4*>(dst + j) = q;
            }
          } else {
            for (int j = 0; j < 32; ++j)
              if (col0 + j < p.N) dst[j] = __float2bfloat16(v[j]);
          }
        } else if (vec) {
          float* dst = (float*)p.C + c_base + col0;
          if (p.out_mode == 2) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              v[4 * j] += __uint_as_float(side[j].x); v[4 * j + 1] += __uint_as_float(side[j].y);
              v[4 * j + 2] += __uint_as_float(side[j].z); v[4 * j + 3] += __uint_as_float(side[j].w);
            }
          }
          if (cin_row != nullptr) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float4 o = *reinterpret_cast<const float4*>(cin_row + col0 + 4 * j);
              v[4 * j] = fmaf(gamma, o.x, v[4 * j]); v[4 * j + 1] = fmaf(gamma, o.y, v[4 * j + 1]);
              v[4 * j + 2] = fmaf(gamma, o.z, v[4 * j + 2]); v[4 * j + 3] = fmaf(gamma, o.w, v[4 * j + 3]);
            }
          }
          if (add_row != nullptr) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 a4 = p.out_mode == 2 ? *reinterpret_cast<const uint4*>(add_row + col0 + 8 * j) : side[j];
              const uint32_t w4[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                v[8 * j + 2 * t] += __uint_as_float(w4[t] << 16);
                v[8 * j + 2 * t + 1] += __uint_as_float(w4[t] & 0xffff0000u);
              }
            }
          }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<float4*>(dst + 4 * j) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          if (c16_row != nullptr) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              uint4 q;
              q.x = pack_bf16(v[j], v[j + 1]);
              q.y = pack_bf16(v[j + 2], v[j + 3]);
              q.z = pack_bf16(v[j + 4], v[j + 5]);
              q.w = pack_bf16(v[j + 6], v[j + 7]);
              *reinterpret_cast<uint4*>(c16_row + col0 + j) = q;
            }
          }
        } else {
          float* dst = (float*)p.C + c_base + col0;
          for (int j = 0; j < 32; ++j) {
            if (col0 + j >= p.N) continue;
            float x = v[j];
            if (p.out_mode == 2) x += dst[j];
            if (cin_row != nullptr) x += gamma * cin_row[col0 + j];
            if (add_row != nullptr) x += __bfloat162float(add_row[col0 + j]);
            dst[j] = x;
            if (c16_row != nullptr) c16_row[col0 + j] = __float2bfloat16(x);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty_bar[acc]);
      if (++acc == n_acc) { acc = 0; acc_phase ^= 1; }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <bool TMA_OUT>
int launch_b(const BMaps& maps, const BGemmParams& p, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(bgemm_bf16_kernel<TMA_OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem::TOTAL);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  const long long units = (long long)p.n_batch * p.tiles_m * p.tiles_n;
  const int grid = (int)(units < 2 * sms ? units : 2 * sms);
  bgemm_bf16_kernel<TMA_OUT><<<grid, BGEMM_THREADS, Smem::TOTAL, stream>>>(maps, p);
  return fb::launch_ok("bgemm_bf16_kernel");
}

// A [hi, lo, rows, cols] layout that a tensor map can describe (a stride counts only where there is something to step to).
bool mappable(const void* ptr, long long ld, long long lo, long long hi, int n_lo, int n_hi, int rows) {
  return !((uintptr_t)ptr & 15) && (ld > 0 || rows == 1) && (lo > 0 || n_lo == 1) && (hi > 0 || n_hi == 1);
}

}  // namespace

extern "C" {

// Operand of a batched GEMM: a [rows, inner] bf16 matrix per batch (hi, lo) at ptr + hi*stride_hi + lo*stride_lo, `ld`
// elements between rows, inner contiguous.  `mn` = 0: rows are the M (or N) dimension and inner is K; `mn` = 1: rows are K
// and inner is the M (or N) dimension.  n_hi / n_lo are the EXTENTS of the storage (coordinates may come from an index).
struct FbBOperand {
  const void* ptr;
  long long ld, stride_lo, stride_hi;
  int n_lo, n_hi;
  int mn;
  int lo_div;
  int hi_offset;
  const int* hi_index;
  int k;               // K of the product this operand belongs to
  int neg;             // A operands: subtract this product
};

struct FbBEpilogue {
  void* C;             // [.., M, N] bf16 (out_mode 0) or fp32 (1 store, 2 accumulate)
  long long ldc, stride_lo, stride_hi;
  int c_lo_div, c_hi_offset;
  const int* c_hi_index;
  const float* Cin;    // optional fp32 addend (layout of C; may be C itself), scaled by gamma[hi coordinate of A * n_lo_batch + lo] (null = 1)
  int cin_hi_offset;
  const int* cin_hi_index;
  const float* gamma;
  void* C16;           // optional bf16 copy of the result (fp32 modes), own hi coordinate
  int c16_hi_offset;
  const int* c16_hi_index;
  const void* add16;   // optional bf16 addend (fp32 modes), own hi coordinate; shares the layout below with C16
  int add16_hi_offset;
  const int* add16_hi_index;
  long long ld16, stride_lo16, stride_hi16;
  const float* decay;  // optional fp32 vector per batch, see bgemm.cu header
  long long d_hi, d_lo, d_r;
  const float* rowscale;  // optional fp32 factor per row
  long long r_hi, r_lo, r_r;
  float alpha;
  int out_mode, mask_mode;
};

// n_hi_batch x n_lo_batch problems of size M x N; ops: n_pairs times (A, B), each product summed over sum_lo consecutive lo
// coordinates.  Returns 0 on success.
int fb_bgemm_bf16(const FbBOperand* ops, int n_pairs, const FbBEpilogue* e, int n_hi_batch, int n_lo_batch, int sum_lo, int M, int N,
                  cudaStream_t stream) {
  if (n_hi_batch <= 0 || n_lo_batch <= 0 || M <= 0 || N <= 0) return 0;
  if (n_pairs < 1 || n_pairs > MAX_PAIRS || sum_lo < 1) return -2;
  for (int i = 0; i < 2 * n_pairs; ++i) {
    const FbBOperand& o = ops[i];
    if ((o.ld & 7) || (o.stride_lo & 7) || (o.stride_hi & 7) || ((uintptr_t)o.ptr & 15) || o.k <= 0) {
      fprintf(stderr, "[flame_b200] bgemm: operand bases and strides must be multiples of 16 bytes\n");
      return -2;
    }
  }
  if ((e->ldc & 7) || (e->stride_lo & 7) || (e->stride_hi & 7) || ((uintptr_t)e->C & 15)) {
    fprintf(stderr, "[flame_b200] bgemm: output base and strides must be multiples of 8 elements\n");
    return -2;
  }
  BGemmParams p;
  p.M = M; p.N = N; p.n_pairs = n_pairs; p.sum_lo = sum_lo;
  p.bn = N <= 64 ? 64 : MAX_BN;
  p.a_rows = M <= 64 ? 64 : BM;
  p.tiles_m = (M + BM - 1) / BM;
  p.tiles_n = (N + p.bn - 1) / p.bn;
  p.n_lo = n_lo_batch;
  p.n_batch = n_hi_batch * n_lo_batch;
  p.c = {e->c_hi_index, e->c_hi_offset, e->c_lo_div > 0 ? e->c_lo_div : 1};
  p.cin = {e->cin_hi_index, e->cin_hi_offset, p.c.lo_div};
  p.C = e->C; p.ldc = e->ldc; p.c_stride_lo = e->stride_lo; p.c_stride_hi = e->stride_hi;
  p.c16i = {e->c16_hi_index, e->c16_hi_offset, p.c.lo_div};
  p.add16i = {e->add16_hi_index, e->add16_hi_offset, p.c.lo_div};
  p.C16 = (__nv_bfloat16*)e->C16;
  p.add16 = (const __nv_bfloat16*)e->add16;
  p.ld16 = e->ld16; p.stride_lo16 = e->stride_lo16; p.stride_hi16 = e->stride_hi16;
  p.Cin = e->Cin; p.gamma = e->gamma;
  p.decay = e->decay; p.d_hi = e->d_hi; p.d_lo = e->d_lo; p.d_r = e->d_r;
  p.rowscale = e->rowscale; p.r_hi = e->r_hi; p.r_lo = e->r_lo; p.r_r = e->r_r;
  p.alpha = e->alpha; p.out_mode = e->out_mode; p.mask_mode = e->mask_mode;
  p.status = fb::status_ptr();
  if ((p.C16 != nullptr || p.Cin != nullptr) && p.out_mode == 0) return -3;
  if ((p.C16 != nullptr || p.add16 != nullptr) && ((p.ld16 & 7) || (p.stride_lo16 & 7) || (p.stride_hi16 & 7))) return -2;
  if (!fb::aligned(16, e->C16, e->add16, e->Cin)) return -2;
  // results leave by TMA unless there is a state step or an index in the way (see the kernel)
  const bool out16 = p.out_mode == 0;
  const int hi_c = p.c.hi_offset + n_hi_batch, hi_add = p.add16i.hi_offset + n_hi_batch;
  const bool tma_out = p.Cin == nullptr && p.C16 == nullptr && p.c.hi_index == nullptr && p.c.lo_div == 1 && p.c.hi_offset >= 0 &&
                       mappable(p.C, p.ldc, p.c_stride_lo, p.c_stride_hi, n_lo_batch, hi_c, M) &&
                       (p.add16 == nullptr ||
                        (out16 && p.add16i.hi_index == nullptr && p.add16i.hi_offset >= 0 &&
                         mappable(p.add16, p.ld16, p.stride_lo16, p.stride_hi16, n_lo_batch, hi_add, M)));
  const int stage_bytes = (p.a_rows + p.bn) * BK * 2;
  const int stg_warps = !tma_out ? 0 : 2 * (p.a_rows / 32);
  p.stages = (MAIN_BYTES - stg_warps * STG_BYTES) / stage_bytes;
  if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
  p.stg_offset = p.stages * stage_bytes;
  p.arrivals = !tma_out ? 8 : (p.a_rows / 32) * (p.bn == 64 ? 1 : 2);
  BMaps maps;
  if (tma_out) {
    const long long some = 8;  // a stride that is never used
    int rc = fb::make_tmap_4d(&maps.c, p.C, out16 ? 2 : 4, hi_c, n_lo_batch, M, N, hi_c > 1 ? p.c_stride_hi : some,
                              n_lo_batch > 1 ? p.c_stride_lo : some, M > 1 ? p.ldc : some, 32, out16 ? 64 : 32, true);
    if (rc) return rc;
    if (p.add16 != nullptr) {
      rc = fb::make_tmap_4d(&maps.add, p.add16, 2, hi_add, n_lo_batch, M, N, hi_add > 1 ? p.stride_hi16 : some,
                            n_lo_batch > 1 ? p.stride_lo16 : some, M > 1 ? p.ld16 : some, 32, 64, true);
      if (rc) return rc;
    }
  }
  for (int i = 0; i < n_pairs; ++i) {
    const FbBOperand &a = ops[2 * i], &b = ops[2 * i + 1];
    BPair& pr = p.pair[i];
    pr.a = {a.hi_index, a.hi_offset, a.lo_div > 0 ? a.lo_div : 1};
    pr.b = {b.hi_index, b.hi_offset, b.lo_div > 0 ? b.lo_div : 1};
    pr.num_kb = (a.k + BK - 1) / BK;
    pr.a_mn = a.mn; pr.b_mn = b.mn; pr.neg = a.neg;
    // dims: (inner, rows, lo, hi)
    int rc = a.mn ? fb::make_tmap_4d(&maps.a[i], a.ptr, 2, a.n_hi, a.n_lo, a.k, M, a.stride_hi, a.stride_lo, a.ld, BK, 64, true)
                  : fb::make_tmap_4d(&maps.a[i], a.ptr, 2, a.n_hi, a.n_lo, M, a.k, a.stride_hi, a.stride_lo, a.ld, p.a_rows, BK, true);
    if (rc) return rc;
    rc = b.mn ? fb::make_tmap_4d(&maps.b[i], b.ptr, 2, b.n_hi, b.n_lo, b.k, N, b.stride_hi, b.stride_lo, b.ld, BK, 64, true)
              : fb::make_tmap_4d(&maps.b[i], b.ptr, 2, b.n_hi, b.n_lo, N, b.k, b.stride_hi, b.stride_lo, b.ld, p.bn, BK, true);
    if (rc) return rc;
  }
  return tma_out ? launch_b<true>(maps, p, stream) : launch_b<false>(maps, p, stream);
}

}  // extern "C"
