// Stick-breaking attention for sm_100a (head dim 64), packed variable-length documents: backward, then forward.
//
//   att_ij = sigma_ij * prod_{j<m<i} (1 - sigma_im)   (j < i),   o_i = sum_j att_ij v_j,   rem_i = 1 - sum_j att_ij
//   g_ij   = do_i . v_j - drem_i,   dA = att * g,   dl_ij = dA_ij - sigma_ij * sum_{k<=j} dA_ik
//   dq_i = scale sum_j dl_ij k_j,   dk_j = scale sum_i dl_ij q_i,   dv_j = sum_i att_ij do_i
//
// One CTA owns a 128-query tile of one (document, head) and walks the keys, 64 at a time, from the diagonal backwards - the
// direction in which both running quantities of a row are available: E = prod (1 - sigma) over the keys already
// seen (so att = sigma * E) and R = sum of dA over the keys already seen; the prefix sum the gradient needs is
// Tot_i - R with Tot_i = do_i . o_i - drem_i (1 - rem_i), known up front.  Per key tile the tensor core forms S and dP,
// one thread per query row turns them into P = att and dS = dl (bf16, swizzled smem), and three more products make the
// tile's dV and dK (fresh each tile, added to fp32 accumulators in global memory) and dQ (accumulated in
// TMEM across the whole walk, no atomics).  Warps: TMA, MMA, four that form P and dS, four that move dV and dK out.
//
// What bounds it is the chain of a tile: clock stamps give 7,500 cycles per 64 keys, of them 4,100 in the weight warps, which issue
// a quarter of the time, the rest waits for products and hand-overs.  So two CTAs share an SM: 256
// tensor-memory columns and 112 KB each.  That is why dV and dK are formed transposed, in ONE accumulator of 128 rows (64
// of dV, 64 of dK) and 64 columns (keys): [dO | 0]^T P + [0 | Q]^T dS, the zeros a tile in shared memory between the two.  (A
// dS that is not finite would reach dV as 0 x dS; it is taken out of its tile, and dQ of its query and dK of its key become NaN.)  A
// row of the accumulator is one channel of 64 keys, so 32 lanes hold 32 neighbouring floats of a key's gradient and add them
// to global memory as they are (red.add, 128 bytes per instruction), without a staging tile.  S and dP of the next tile are
// issued ahead of this tile's other products, and the weights of eight keys finished while the next eight's exponentials and
// reciprocals run (one loop for masked tiles and one for the others: with both in one the compiler kept the parts apart, 2.18 ms).
// Eight rows of 4,096 tokens, 16 heads: 2.46 ms with one CTA of 128 x 128 tiles per SM, 2.03 with two, 1.94 with the eights
// interleaved, 1.87 with one reciprocal for two keys.  The reference reaches the same sums with spin-locked adds
// (custom_models/sba/stickbreaking_attention/sb_varlen/sb_varlen_bwd.py:13-52); here nothing spins unbounded.
#include "attn_tiles.cuh"
#include "sb_math.cuh"
#include "tc05.cuh"
#include "host_utils.cuh"
#include <math.h>
#include <type_traits>

using namespace tc05;

namespace {

constexpr int BQ = 128, BKV = 64, DH = 64;
constexpr float kLog2e = 1.4426950408889634f;

struct SbBwdParams {
  const int* cu_seqlens;
  const int* tile_list;
  int nseq, H, total_tokens;
  float scale, scale_log2;
  const float* tot;    // [H, T]  do.o - drem (1 - rem)
  const float* drem;   // [H, T] or null
  float *dK, *dV;      // [T, H, DH] fp32, added to
  __nv_bfloat16* dQ;   // [T, H, DH] with token stride dq_stride_t
  long long dq_stride_t;
  int* status;
};

__device__ __forceinline__ uint32_t sw128_offset(int row, int col) {
  const int chunk = (col >> 3) ^ (row & 7);
  return (uint32_t)(row * 128 + chunk * 16 + (col & 7) * 2);
}

struct Smem {
  static constexpr int TILE = BQ * DH * 2;           // 16 KB
  static constexpr int DO_OFF = 0, ZERO_OFF = TILE, Q_OFF = 2 * TILE;  // in this order: the transposed products' A operands
  static constexpr int NSTAGE = 2;
  static constexpr int KV = BKV * DH * 2;            // 8 KB
  static constexpr int RING_OFF = 3 * TILE;          // stage = K tile + V tile
  static constexpr int STAGE = 2 * KV;
  static constexpr int P_OFF = RING_OFF + NSTAGE * STAGE;
  static constexpr int DS_OFF = P_OFF + BQ * BKV * 2;
  static constexpr int BAR_OFF = DS_OFF + BQ * BKV * 2;
  static constexpr int TOTAL = BAR_OFF + 256;        // 112 KB and the barriers: two CTAs per SM, without room to align the base
};

constexpr int SB_THREADS = 320;

// Takes the values that are not finite out of row r of a tile of dS: the accumulator shared by dV and dK forms 0 x dS in dV's rows, which
// P and dO alone decide.  Their keys' dK (n of them belong to the document; `dst`: the first one's) becomes NaN here instead.  Whether
// there was any.
__device__ __noinline__ bool take_out_not_finite(uint8_t* sDS, int r, int n, float* dst, long long row) {
  bool any = false;
  for (int c = 0; c < BKV; ++c) {
    uint16_t* v = reinterpret_cast<uint16_t*>(sDS + sw128_offset(r, c));
    if ((*v & 0x7f80) != 0x7f80) continue;
    *v = 0;
    any = true;
    float* k = dst + c * row;
    if (c >= n || isnan(*reinterpret_cast<volatile float*>(k))) continue;  // (NaN stays NaN whatever is added)
    for (int i = 0; i < DH; ++i) k[i] = __uint_as_float(0x7fc00000u);
  }
  return any;
}

template <bool DREM>
__global__ void __launch_bounds__(SB_THREADS, 2)
sb_attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO, SbBwdParams p) {
  using L = Smem;
  int head, doc, ti;
  if (!attn_tile(p.tile_list, p.nseq, p.H, true, head, doc, ti)) return;
  const int doc_start = p.cu_seqlens[doc];
  const int doc_len = p.cu_seqlens[doc + 1] - doc_start;
  const int q0 = ti * BQ;
  const int n_iter = min((q0 + BQ) / BKV, (doc_len + BKV - 1) / BKV);  // key tiles n_iter - 1, ..., 0

  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023) {  // the swizzled tiles need it
    if (threadIdx.x == 0) report(p.status, ERR_BAD_ARG);
    return;
  }
  uint64_t* full_bar = (uint64_t*)(smem + L::BAR_OFF);
  uint64_t* empty_bar = full_bar + L::NSTAGE;
  uint64_t* q_full = empty_bar + L::NSTAGE;
  uint64_t* sdp_full = q_full + 1;
  uint64_t* pds_ready = sdp_full + 1;
  uint64_t* dkv_full = pds_ready + 1;  // also: P and dS may be overwritten
  uint64_t* dkv_free = dkv_full + 1;
  uint64_t* dq_full = dkv_free + 1;
  uint32_t* tmem_slot = (uint32_t*)(dq_full + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < L::NSTAGE; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(q_full, 1);
    mbar_init(sdp_full, 1);
    mbar_init(pds_ready, 128);
    mbar_init(dkv_full, 1);
    mbar_init(dkv_free, 128);
    mbar_init(dq_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmdO);
  }
  for (int i = threadIdx.x; i < L::TILE / 16; i += SB_THREADS) reinterpret_cast<uint4*>(smem + L::ZERO_OFF)[i] = make_uint4(0u, 0u, 0u, 0u);
  fence_async_smem();
  if (warp == 1) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_S = tmem_base, tmem_dP = tmem_base + 64, tmem_dKV = tmem_base + 128, tmem_dQ = tmem_base + 192;

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(q_full, 2 * L::TILE);
      tma_load_3d(smem + L::Q_OFF, &tmQ, q_full, 0, head, doc_start + q0);
      tma_load_3d(smem + L::DO_OFF, &tmdO, q_full, 0, head, doc_start + q0);
      for (int it = 0; it < n_iter; ++it) {
        const int stage = it % L::NSTAGE;
        if (!mbar_wait(&empty_bar[stage], ((it / L::NSTAGE) & 1) ^ 1, p.status, abort_flag, ERR_WAIT_EMPTY)) break;
        const int row = doc_start + (n_iter - 1 - it) * BKV;
        uint8_t* dst = smem + L::RING_OFF + stage * L::STAGE;
        mbar_expect_tx(&full_bar[stage], L::STAGE);
        tma_load_3d(dst, &tmK, &full_bar[stage], 0, head, row);
        tma_load_3d(dst + L::KV, &tmV, &full_bar[stage], 0, head, row);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16(BQ, BKV, 0, 0);
      constexpr uint32_t idesc_kv = make_idesc_bf16(2 * DH, BKV, 1, 1);
      constexpr uint32_t idesc_dq = make_idesc_bf16(BQ, DH, 0, 1);
      const uint32_t sQ = smem_u32(smem + L::Q_OFF), sdO = smem_u32(smem + L::DO_OFF);
      const uint32_t sP = smem_u32(smem + L::P_OFF), sDS = smem_u32(smem + L::DS_OFF);
      auto issue_sdp = [&](int it) -> bool {
        const int stage = it % L::NSTAGE;
        if (!mbar_wait(&full_bar[stage], (it / L::NSTAGE) & 1, p.status, abort_flag, ERR_WAIT_FULL)) return false;
        tc_fence_after();
        const uint32_t sK = smem_u32(smem + L::RING_OFF + stage * L::STAGE), sV = sK + L::KV;
        const uint64_t aq = make_smem_desc(sQ, 16, 1024), bk = make_smem_desc(sK, 16, 1024);
        const uint64_t ad = make_smem_desc(sdO, 16, 1024), bv = make_smem_desc(sV, 16, 1024);
#pragma unroll
        for (int k = 0; k < DH / 16; ++k) mma_ss(tmem_S, desc_advance(aq, k * 32), desc_advance(bk, k * 32), idesc_s, k ? 1u : 0u);
#pragma unroll
        for (int k = 0; k < DH / 16; ++k) mma_ss(tmem_dP, desc_advance(ad, k * 32), desc_advance(bv, k * 32), idesc_s, k ? 1u : 0u);
        mma_commit(sdp_full);
        return true;
      };
      bool ok = mbar_wait(q_full, 0, p.status, abort_flag, ERR_WAIT_FULL);
      if (ok) ok = issue_sdp(0);
      for (int it = 0; it < n_iter && ok; ++it) {
        const int stage = it % L::NSTAGE;
        const uint32_t sK = smem_u32(smem + L::RING_OFF + stage * L::STAGE);
        if (!mbar_wait(pds_ready, it & 1, p.status, abort_flag, ERR_WAIT_MISC)) break;
        tc_fence_after();
        if (it + 1 < n_iter && !issue_sdp(it + 1)) break;
        // dO | zeros and zeros | Q: 64-wide groups of the M dimension one tile apart
        const uint64_t a_do = make_smem_desc(sdO, L::TILE, 1024), a_q = make_smem_desc(smem_u32(smem + L::ZERO_OFF), L::TILE, 1024);
        const uint64_t bp = make_smem_desc(sP, 16, 1024), bds = make_smem_desc(sDS, 16, 1024);
        const uint64_t ads = make_smem_desc(sDS, 16, 1024), bk = make_smem_desc(sK, 16, 1024);
#pragma unroll
        for (int k = 0; k < BKV / 16; ++k) mma_ss(tmem_dQ, desc_advance(ads, k * 32), desc_advance(bk, k * 2048), idesc_dq, (it > 0 || k > 0) ? 1u : 0u);
        if (it > 0) {  // the previous tile's dK / dV must have left TMEM
          if (!mbar_wait(dkv_free, (it - 1) & 1, p.status, abort_flag, ERR_WAIT_TMEM_EMPTY)) break;
          tc_fence_after();
        }
#pragma unroll
        for (int k = 0; k < BQ / 16; ++k) mma_ss(tmem_dKV, desc_advance(a_do, k * 2048), desc_advance(bp, k * 2048), idesc_kv, k ? 1u : 0u);
#pragma unroll
        for (int k = 0; k < BQ / 16; ++k) mma_ss(tmem_dKV, desc_advance(a_q, k * 2048), desc_advance(bds, k * 2048), idesc_kv, 1u);
        mma_commit(&empty_bar[stage]);
        mma_commit(dkv_full);
        if (it + 1 == n_iter) mma_commit(dq_full);
      }
    }
  } else if (warp < 6) {
    // ------------------------------------------------------------------ weights: one thread per query row
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const uint32_t lane_sel = (uint32_t)(quarter * 32) << 16;
    uint8_t* sP = smem + L::P_OFF;
    uint8_t* sDS = smem + L::DS_OFF;
    const int q_idx = q0 + r;
    const bool valid = q_idx < doc_len;
    const bool ragged = q0 + BQ > doc_len;
    const long long tok = (long long)doc_start + q_idx;
    const float tot = valid ? p.tot[(long long)head * p.total_tokens + tok] : 0.f;
    const float drem = (DREM && valid) ? p.drem[(long long)head * p.total_tokens + tok] : 0.f;
    const sb2 ndrem = sb_pk(-drem, -drem);
    float E = 1.f;  // product of (1 - sigma) over the keys already seen
    float R = 0.f;  // sum of dA over the keys already seen
    // dS is made of tot, R and their differences, and a dA that is not finite stays in R: as long as this sum over every eighth R is far
    // from overflow all of dS is finite (backward with its sums 2.20 -> 2.24 ms, 8 x 4,096 tokens, 16 heads; value by value twice that)
    float size = fabsf(tot);
    bool ok = true, lost = false;  // lost: some dS of this row was not finite
    for (int it = 0; it < n_iter && ok; ++it) {
      const int kv0 = (n_iter - 1 - it) * BKV;
      const bool diag = kv0 + BKV > q0;
      if (!mbar_wait_warp(sdp_full, it & 1, p.status, abort_flag, ERR_WAIT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      auto walk = [&](auto mask) -> bool {
      constexpr bool MASK = decltype(mask)::value;
      uint32_t xr[2][8], dr[2][8];  // a group's logits and dP, the next group's on their way
      sb2 nsig_n[4];
      float ninv_n[8];
      auto sigma = [&](int g, const uint32_t* x) {
        const int c = BKV - 8 - g * 8;
        sb_sigma<MASK>(x, p.scale_log2, MASK ? sb_dead_bits(!valid, diag, kv0 + c, q_idx) : 0u, nsig_n, ninv_n);
      };
      tmem_ld_32x8(tmem_S + lane_sel + BKV - 8, xr[0]);
      tmem_ld_wait();
      tmem_ld_32x8(tmem_S + lane_sel + BKV - 16, xr[1]);
      tmem_ld_32x8(tmem_dP + lane_sel + BKV - 8, dr[0]);
      sigma(0, xr[0]);
      // the previous tile's products have read P and dS
      if (it > 0 && !mbar_wait_warp(dkv_full, (it - 1) & 1, p.status, abort_flag, ERR_WAIT_MISC)) return false;
#pragma unroll 2
      for (int g = 0; g < BKV / 8; ++g) {
        const int c = BKV - 8 - g * 8;
        tmem_ld_wait();
        uint32_t(&dp)[8] = dr[g & 1];
        sb2 nsig[4], a[4], d[4];
        float ninv[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) nsig[i] = nsig_n[i];
#pragma unroll
        for (int i = 0; i < 8; ++i) ninv[i] = ninv_n[i];
        if (c > 8) tmem_ld_32x8(tmem_S + lane_sel + c - 16, xr[g & 1]);
        if (c > 0) {
          tmem_ld_32x8(tmem_dP + lane_sel + c - 8, dr[(g & 1) ^ 1]);
          sigma(g + 1, xr[(g & 1) ^ 1]);
        }
        sb_weights(E, nsig, ninv, a);
        if (MASK) {
          const uint32_t dead = sb_dead_bits(!valid, diag, kv0 + c, q_idx);
#pragma unroll
          for (int i = 0; i < 8; ++i)  // what stands in another document's rows does not count, whatever it is
            if ((dead >> i) & 1u) dp[i] = 0u;
        }
        const uint4 q = make_uint4(sb_pack(a[0]), sb_pack(a[1]), sb_pack(a[2]), sb_pack(a[3]));
        // The forward formed o from the bf16 rounding of att, and tot = do . o is the total the running sum of dA has to
        // meet exactly at the end of the walk: the same rounded weight enters dA here (the remainder term keeps the
        // fp32 weight, as rem was formed from it).  With fp32 att in this place the mismatch of the two roundings,
        // multiplied by sigma for every key of the row, was a 20 % error in dq at 4096-token rows.
        const uint32_t qw[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 3; i >= 0; --i) {  // dA is zero for keys that do not count
          const sb2 att16 = sb_pk(__uint_as_float(qw[i] << 16), __uint_as_float(qw[i] & 0xffff0000u));
          sb2 dA = sb_mul2(att16, sb_pk(__uint_as_float(dp[2 * i]), __uint_as_float(dp[2 * i + 1])));
          if (DREM) dA = sb_fma2(a[i], ndrem, dA);
          float dA0, dA1;
          sb_up(dA, dA0, dA1);
          const float R1 = R;
          R += dA1;
          d[i] = sb_fma2(nsig[i], sb_pk(tot - R, tot - R1), dA);
          R += dA0;
        }
        const uint32_t off = sw128_offset(r, c);
        *reinterpret_cast<uint4*>(sP + off) = q;
        *reinterpret_cast<uint4*>(sDS + off) = make_uint4(sb_pack(d[0]), sb_pack(d[1]), sb_pack(d[2]), sb_pack(d[3]));
        size += fabsf(R);
      }
      return true;
      };
      ok = diag || ragged ? walk(std::true_type()) : walk(std::false_type());
      if (!ok) break;
      if (!(size < 1e38f))
        lost |= take_out_not_finite(sDS, r, doc_len - kv0, p.dK + (long long)(doc_start + kv0) * p.H * DH + head * DH, (long long)p.H * DH);
      tc_fence_before();
      fence_async_smem();
      mbar_arrive(pds_ready);
    }
    if (ok) ok = mbar_wait_warp(dq_full, 0, p.status, abort_flag, ERR_WAIT_TMEM_FULL);
    if (ok) {
      // dQ of this query tile
      tc_fence_after();
      __nv_bfloat16* dqrow = p.dQ + tok * p.dq_stride_t + (long long)head * DH;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t v[32];
        tmem_ld_32x32(tmem_dQ + lane_sel + half * 32, v);
        tmem_ld_wait();
        if (lost) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0x7fc00000u;
        }
        if (valid) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint4 q;
            q.x = pack_bf16(__uint_as_float(v[g * 8 + 0]) * p.scale, __uint_as_float(v[g * 8 + 1]) * p.scale);
            q.y = pack_bf16(__uint_as_float(v[g * 8 + 2]) * p.scale, __uint_as_float(v[g * 8 + 3]) * p.scale);
            q.z = pack_bf16(__uint_as_float(v[g * 8 + 4]) * p.scale, __uint_as_float(v[g * 8 + 5]) * p.scale);
            q.w = pack_bf16(__uint_as_float(v[g * 8 + 6]) * p.scale, __uint_as_float(v[g * 8 + 7]) * p.scale);
            *reinterpret_cast<uint4*>(dqrow + half * 32 + g * 8) = q;
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ dV and dK of every tile: a lane is one channel
    const int quarter = warp & 3;
    const uint32_t lane_sel = (uint32_t)(quarter * 32) << 16;
    const long long row = (long long)p.H * DH;
    float* out = (quarter < 2 ? p.dV : p.dK) + (long long)doc_start * row + head * DH + (quarter & 1) * 32 + lane;
    const float mul = quarter < 2 ? 1.f : p.scale;
    for (int it = 0; it < n_iter; ++it) {
      const int kv0 = (n_iter - 1 - it) * BKV;
      if (!mbar_wait_warp(dkv_full, it & 1, p.status, abort_flag, ERR_WAIT_TMEM_FULL)) break;
      tc_fence_after();
      uint32_t v[2][32];
      tmem_ld_32x32(tmem_dKV + lane_sel, v[0]);
      tmem_ld_32x32(tmem_dKV + lane_sel + 32, v[1]);
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive(dkv_free);
      float* dst = out + kv0 * row;
      const int n = min(BKV, doc_len - kv0);  // keys of the document
      if (n == BKV) {
#pragma unroll
        for (int c = 0; c < BKV; ++c) atomicAdd(dst + c * row, __uint_as_float(v[c / 32][c % 32]) * mul);
      } else {
#pragma unroll
        for (int c = 0; c < BKV; ++c)
          if (c < n) atomicAdd(dst + c * row, __uint_as_float(v[c / 32][c % 32]) * mul);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

// tot[h, t] = do.o - drem * (1 - rem).  The prefix sums the gradient needs are formed as tot - (running sum of dA), a
// difference of nearly equal numbers for the far keys, and every key's dl carries sigma times its error: with o rounded
// to bf16 the error of dq / dk grows with the row length (7 % at 1000 tokens, 22 % at 4096).  So o enters as the
// two-term split o + o_lo that the forward kernel writes (16 mantissa bits), which makes tot agree with the running sum
// to fp32 accuracy.
__global__ void sb_tot_kernel(const __nv_bfloat16* __restrict__ O, const __nv_bfloat16* __restrict__ O_lo,
                              const __nv_bfloat16* __restrict__ dO,
                              const float* __restrict__ rem, const float* __restrict__ drem, float* __restrict__ tot,
                              long long T, int H, long long o_stride_t, long long do_stride_t) {
  constexpr int LANES = DH / 8;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long row = gid / LANES;
  const int sub = (int)(gid % LANES);
  float acc = 0.f;
  long long t = 0;
  int h = 0;
  const bool live = row < T * H;
  if (live) {
    t = row / H;
    h = (int)(row - t * H);
    const uint4 a = *reinterpret_cast<const uint4*>(O + t * o_stride_t + (long long)h * DH + sub * 8);
    const uint4 b = *reinterpret_cast<const uint4*>(dO + t * do_stride_t + (long long)h * DH + sub * 8);
    uint4 l = make_uint4(0u, 0u, 0u, 0u);
    if (O_lo != nullptr) l = *reinterpret_cast<const uint4*>(O_lo + (t * H + h) * DH + sub * 8);
    const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&a);
    const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&b);
    const __nv_bfloat162* pl = reinterpret_cast<const __nv_bfloat162*>(&l);
    float lo_acc = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 x = __bfloat1622float2(pa[i]), y = __bfloat1622float2(pb[i]), z = __bfloat1622float2(pl[i]);
      acc += x.x * y.x + x.y * y.y;
      lo_acc += z.x * y.x + z.y * y.y;
    }
    acc += lo_acc;
  }
#pragma unroll
  for (int s = LANES / 2; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if (live && sub == 0) {
    const long long i = (long long)h * T + t;
    tot[i] = acc - (drem ? drem[i] * (1.f - rem[i]) : 0.f);
  }
}

// ------------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------------
//   o_i = sum_j att_ij v_j (att of the head of this file),   rem_i = 1 - sum_j att_ij = prod_j (1 - sigma_ij)
//
// One CTA per 128-query tile, two per SM, the keys from the diagonal backwards, 64 at a time, a thread per query row.  Weights
// never exceed one, so there is no running maximum and the output is never rescaled.  What bounds it is the weight warps' chain
// (special functions 61 % of their peak): the scores of the next tile and a second tile of weights are there, so that they
// wait for no product, and the weights of eight keys are finished while the next eight's exponentials and reciprocals run.
// Eight rows of 4,096 tokens, 16 heads: 128 keys at a time with one tile of scores and weights 1.00 ms, eights finished under the
// next 0.94, two tiles of 64 keys 0.85 (and one reciprocal for two keys 0.82).
struct FwdParams {
  const int* cu_seqlens;
  const int* tile_list;
  int nseq, H, total_tokens;
  float scale_log2;
  __nv_bfloat16* O;
  long long o_stride_t;
  // Optional second output [T, H, DH] (contiguous): the bf16 rounding of (O_fp32 - O), i.e. the low half of a two-term
  // bf16 split of the fp32 result.  The backward needs do . o to fp32 accuracy.
  __nv_bfloat16* O_lo;
  float* rem;  // [H, T]
  int* status;
};

struct FwdSmem {
  static constexpr int TILE = BQ * DH * 2;   // 16 KB
  static constexpr int KV = BKV * DH * 2;    // 8 KB
  static constexpr int NSLOT = 6;            // K and V tiles in turn
  static constexpr int Q_OFF = 0, RING_OFF = TILE, P_OFF = RING_OFF + NSLOT * KV;
  static constexpr int BAR_OFF = P_OFF + 2 * BQ * BKV * 2;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

__global__ void __launch_bounds__(192, 2)
sb_attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                   FwdParams p) {
  using L = FwdSmem;
  int head, doc, ti;
  if (!attn_tile(p.tile_list, p.nseq, p.H, true, head, doc, ti)) return;
  const int doc_start = p.cu_seqlens[doc];
  const int doc_len = p.cu_seqlens[doc + 1] - doc_start;
  const int q0 = ti * BQ;
  const int n_iter = min((q0 + BQ) / BKV, (doc_len + BKV - 1) / BKV);  // key tiles n_iter - 1, ..., 0

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full_bar = (uint64_t*)(smem + L::BAR_OFF);
  uint64_t* empty_bar = full_bar + L::NSLOT;
  uint64_t* q_full = empty_bar + L::NSLOT;
  uint64_t* s_full = q_full + 1;    // [2] scores of a tile
  uint64_t* p_ready = s_full + 2;   // [2] its weights, and its scores have been read
  uint64_t* pv_done = p_ready + 2;  // [2] its product, which has read the weights
  uint32_t* tmem_slot = (uint32_t*)(pv_done + 2);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < L::NSLOT; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(q_full, 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&s_full[b], 1);
      mbar_init(&p_ready[b], 128);
      mbar_init(&pv_done[b], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_S = tmem_base, tmem_O = tmem_base + 2 * BKV;  // two tiles of scores

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(q_full, L::TILE);
      tma_load_3d(smem + L::Q_OFF, &tmQ, q_full, 0, head, doc_start + q0);
      // in the order in which the products take them: K 0, K 1, V 0, K 2, V 1, ..., the last V
      for (int n = 0, k = 0, v = 0; n < 2 * n_iter; ++n) {
        const bool is_k = k < n_iter && k <= v + 1;
        const int row = doc_start + (n_iter - 1 - (is_k ? k++ : v++)) * BKV, slot = n % L::NSLOT;
        if (!mbar_wait(&empty_bar[slot], ((n / L::NSLOT) & 1) ^ 1, p.status, abort_flag, ERR_WAIT_EMPTY)) break;
        mbar_expect_tx(&full_bar[slot], L::KV);
        tma_load_3d(smem + L::RING_OFF + slot * L::KV, is_k ? &tmK : &tmV, &full_bar[slot], 0, head, row);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16(BQ, BKV, 0, 0);
      constexpr uint32_t idesc_o = make_idesc_bf16(BQ, DH, 0, 1);
      const uint32_t sQ = smem_u32(smem + L::Q_OFF);
      int n = 0;  // tiles taken from the ring
      auto tile = [&](uint32_t& addr) -> uint64_t* {
        const int slot = n % L::NSLOT;
        if (!mbar_wait(&full_bar[slot], (n / L::NSLOT) & 1, p.status, abort_flag, ERR_WAIT_FULL)) return nullptr;
        tc_fence_after();
        ++n;
        addr = smem_u32(smem + L::RING_OFF + slot * L::KV);
        return &empty_bar[slot];
      };
      auto scores = [&](int it) -> bool {
        uint32_t sK;
        uint64_t* done = tile(sK);
        if (!done) return false;
        const uint64_t a = make_smem_desc(sQ, 16, 1024), b = make_smem_desc(sK, 16, 1024);
#pragma unroll
        for (int k = 0; k < DH / 16; ++k)
          mma_ss(tmem_S + (it & 1) * BKV, desc_advance(a, k * 32), desc_advance(b, k * 32), idesc_s, k ? 1u : 0u);
        mma_commit(done);
        mma_commit(&s_full[it & 1]);
        return true;
      };
      bool ok = mbar_wait(q_full, 0, p.status, abort_flag, ERR_WAIT_FULL) && scores(0);
      if (ok && n_iter > 1) ok = scores(1);
      for (int it = 0; it < n_iter && ok; ++it) {
        if (!mbar_wait(&p_ready[it & 1], (it >> 1) & 1, p.status, abort_flag, ERR_WAIT_MISC)) break;
        tc_fence_after();
        uint32_t sV;
        uint64_t* done = tile(sV);
        if (!done) break;
        const uint64_t a = make_smem_desc(smem_u32(smem + L::P_OFF) + (it & 1) * (BQ * BKV * 2), 16, 1024), b = make_smem_desc(sV, 16, 1024);
#pragma unroll
        for (int k = 0; k < BKV / 16; ++k)
          mma_ss(tmem_O, desc_advance(a, k * 32), desc_advance(b, k * 2048), idesc_o, (it > 0 || k > 0) ? 1u : 0u);
        mma_commit(done);
        mma_commit(&pv_done[it & 1]);
        if (it + 2 < n_iter) ok = scores(it + 2);
      }
    }
  } else {
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int q_idx = q0 + r;
    const uint32_t lane_sel = (uint32_t)(quarter * 32) << 16;
    float E = 1.f;  // product of (1 - sigma) over the keys already seen
    bool ok = true;
    for (int it = 0; it < n_iter && ok; ++it) {
      const int kv0 = (n_iter - 1 - it) * BKV;
      const uint32_t t_s = tmem_S + (it & 1) * BKV + lane_sel;
      uint8_t* sP = smem + L::P_OFF + (it & 1) * (BQ * BKV * 2);
      if (!mbar_wait_warp(&s_full[it & 1], (it >> 1) & 1, p.status, abort_flag, ERR_WAIT_TMEM_FULL)) { ok = false; break; }
      if (it > 1 && !mbar_wait_warp(&pv_done[it & 1], ((it >> 1) - 1) & 1, p.status, abort_flag, ERR_WAIT_MISC)) { ok = false; break; }
      tc_fence_after();
      auto walk = [&](auto mask) {
        constexpr bool MASK = decltype(mask)::value;
        uint32_t x[BKV];  // the row's scores, sixteen at a time from the right
        sb2 nsig[4], att[4];
        float ninv[8];
        auto sigma = [&](int c) {
          sb_sigma<MASK>(x + c, p.scale_log2, MASK ? sb_dead_bits(false, true, kv0 + c, q_idx) : 0u, nsig, ninv);
        };
        auto load = [&](int c) { tmem_ld_32x16(t_s + c, *reinterpret_cast<uint32_t(*)[16]>(&x[c])); };
        load(BKV - 16);
        tmem_ld_wait();
        load(BKV - 32);
        sigma(BKV - 8);
#pragma unroll
        for (int c = BKV - 8; c >= 0; c -= 8) {  // the weights of the eight keys at c
          sb2 ns[4];
          float ni[8];
#pragma unroll
          for (int i = 0; i < 4; ++i) ns[i] = nsig[i];
#pragma unroll
          for (int i = 0; i < 8; ++i) ni[i] = ninv[i];
          if (c > 0) {
            if (c % 16 == 0) {
              tmem_ld_wait();
              if (c > 16) load(c - 32);
            }
            sigma(c - 8);
          }
          sb_weights(E, ns, ni, att);
          *reinterpret_cast<uint4*>(sP + sw128_offset(r, c)) = make_uint4(sb_pack(att[0]), sb_pack(att[1]), sb_pack(att[2]), sb_pack(att[3]));
        }
      };
      if (kv0 + BKV > q0) walk(std::true_type());
      else walk(std::false_type());
      tc_fence_before();
      fence_async_smem();
      mbar_arrive(&p_ready[it & 1]);
    }
    if (ok) ok = mbar_wait_warp(&pv_done[(n_iter - 1) & 1], ((n_iter - 1) >> 1) & 1, p.status, abort_flag, ERR_WAIT_MISC);
    if (ok) {
      tc_fence_after();
      const bool valid = q_idx < doc_len;
      const long long tok = (long long)doc_start + q_idx;
      __nv_bfloat16* orow = p.O + tok * p.o_stride_t + (long long)head * DH;
#pragma unroll 1
      for (int c = 0; c < DH; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32(tmem_O + lane_sel + c, v);
        tmem_ld_wait();
        if (!valid) continue;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint4 q, lo;
          uint32_t *qw = reinterpret_cast<uint32_t*>(&q), *lw = reinterpret_cast<uint32_t*>(&lo);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float v0 = __uint_as_float(v[g * 8 + 2 * e]), v1 = __uint_as_float(v[g * 8 + 2 * e + 1]);
            qw[e] = pack_bf16(v0, v1);
            lw[e] = pack_bf16(v0 - __uint_as_float(qw[e] << 16), v1 - __uint_as_float(qw[e] & 0xffff0000u));
          }
          *reinterpret_cast<uint4*>(orow + c + g * 8) = q;
          if (p.O_lo != nullptr) *reinterpret_cast<uint4*>(p.O_lo + (tok * p.H + head) * DH + c + g * 8) = lo;
        }
      }
      if (valid) p.rem[(long long)head * p.total_tokens + tok] = E;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

// dims (inner to outer): [DH, H, T]; box [64, 1, rows]
int make_map(CUtensorMap* m, const void* base, long long T, int H, long long stride, uint32_t rows) {
  return fb::make_tmap_3d(m, base, 2, (uint64_t)T, (uint64_t)H, (uint64_t)DH, (uint64_t)stride, (uint64_t)DH, rows, 1, 64, true);
}

}  // namespace

extern "C" {

// o = sum_j att_ij v_j without normalisation (head dim 64), rem[h, t] = 1 - sum_j att_ij.
// o_lo: optional bf16 [T, H, 64] that receives the part of the fp32 result the bf16 output lost (null: not written).
int fb_sb_attn_fwd(const void* q, const void* k, const void* v, void* o, void* o_lo, float* rem, const int* cu_seqlens,
                   const int* tile_list, int nseq, int max_tiles, long long T, int H, int dh, long long q_stride_t,
                   long long k_stride_t, long long v_stride_t, long long o_stride_t, float scale, cudaStream_t stream) {
  if (T == 0) return 0;
  if (dh != DH) return -2;
  if ((q_stride_t % 8) || (k_stride_t % 8) || (v_stride_t % 8) || (o_stride_t % 8)) return -3;
  CUtensorMap tmQ, tmK, tmV;
  int rc = make_map(&tmQ, q, T, H, q_stride_t, BQ);
  if (!rc) rc = make_map(&tmK, k, T, H, k_stride_t, BKV);
  if (!rc) rc = make_map(&tmV, v, T, H, v_stride_t, BKV);
  if (rc) return rc;
  FwdParams p;
  p.cu_seqlens = cu_seqlens;
  p.tile_list = tile_list;
  p.nseq = nseq;
  p.H = H;
  p.total_tokens = (int)T;
  p.scale_log2 = scale * kLog2e;
  p.O = (__nv_bfloat16*)o;
  p.o_stride_t = o_stride_t;
  p.O_lo = (__nv_bfloat16*)o_lo;
  p.rem = rem;
  p.status = fb::status_ptr();
  const cudaError_t e = cudaFuncSetAttribute(sb_attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FwdSmem::TOTAL);
  if (e != cudaSuccess) return (int)e;
  sb_attn_fwd_kernel<<<(unsigned)max_tiles * H, 192, FwdSmem::TOTAL, stream>>>(tmQ, tmK, tmV, p);
  return fb::launch_ok("sb_attn_fwd_kernel");
}

// dk_acc, dv_acc: fp32 [T, H, 64], zero on entry (added to); dq: bf16 [T, H, 64] (token stride given).
// tot: fp32 [H, T] scratch.  rem: fp32 [H, T] from the forward; drem may be null.  o_lo: the forward's second output
// (bf16 [T, H, 64], contiguous) or null.
int fb_sb_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* o_lo, const void* dout, const float* rem,
                   const float* drem, float* tot, void* dq, float* dk_acc, float* dv_acc, const int* cu_seqlens,
                   const int* tile_list, int nseq, int max_tiles, long long T, int H, long long q_stride_t,
                   long long k_stride_t, long long v_stride_t, long long o_stride_t, long long do_stride_t,
                   long long dq_stride_t, float scale, cudaStream_t stream) {
  if (T == 0) return 0;
  if ((q_stride_t % 8) || (k_stride_t % 8) || (v_stride_t % 8) || (o_stride_t % 8) || (do_stride_t % 8) || (dq_stride_t % 8))
    return -3;
  if (!fb::aligned(16, o, o_lo, dout, dq)) return -2;
  {
    const long long threads = T * H * (DH / 8);
    sb_tot_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>((const __nv_bfloat16*)o, (const __nv_bfloat16*)o_lo,
                                                                       (const __nv_bfloat16*)dout, rem, drem, tot, T, H,
                                                                       o_stride_t, do_stride_t);
    int rc = fb::launch_ok("sb_tot_kernel");
    if (rc) return rc;
  }
  CUtensorMap tmQ, tmK, tmV, tmdO;
  int rc = make_map(&tmQ, q, T, H, q_stride_t, BQ);
  if (!rc) rc = make_map(&tmK, k, T, H, k_stride_t, BKV);
  if (!rc) rc = make_map(&tmV, v, T, H, v_stride_t, BKV);
  if (!rc) rc = make_map(&tmdO, dout, T, H, do_stride_t, BQ);
  if (rc) return rc;
  SbBwdParams p;
  p.cu_seqlens = cu_seqlens;
  p.tile_list = tile_list;
  p.nseq = nseq;
  p.H = H;
  p.total_tokens = (int)T;
  p.scale = scale;
  p.scale_log2 = scale * kLog2e;
  p.tot = tot;
  p.drem = drem;
  p.dK = dk_acc, p.dV = dv_acc;
  p.dQ = (__nv_bfloat16*)dq;
  p.dq_stride_t = dq_stride_t;
  p.status = fb::status_ptr();
  auto launch = [&](auto kernel) -> int {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem::TOTAL);
    if (e != cudaSuccess) return (int)e;
    kernel<<<(unsigned)max_tiles * H, SB_THREADS, Smem::TOTAL, stream>>>(tmQ, tmK, tmV, tmdO, p);
    return 0;
  };
  rc = drem != nullptr ? launch(sb_attn_bwd_kernel<true>) : launch(sb_attn_bwd_kernel<false>);
  if (rc) return rc;
  return fb::launch_ok("sb_attn_bwd_kernel");
}

}  // extern "C"
