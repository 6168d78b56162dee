// Flash attention backward for sm_100a with one writer for every row, for gradients whose bits repeat, for softmax scales that are next
// to nothing and for calls whose sums of dq would outgrow the scratch; attention_bwd_fused.cuh is the faster form, whose sums have no
// fixed order.
// Two tcgen05 kernels that recompute the probabilities from
// the saved log-sum-exp (natural log of the scaled scores) and delta = rowsum(dO * O):
//
//   attn_bwd_dq_kernel   one CTA per (128-query block, query head, sequence), loops over key blocks:
//        S = Q K^T, dP = dO V^T            (SS MMAs into TMEM)
//        dS = P * (dP - delta)              (lanes = queries; bf16 dS over S in TMEM)
//        dQ += dS K                         (TS MMA; K tile read MN-major from the same shared tile)
//   attn_bwd_dkv_kernel  one CTA per (128-key block, KV head, sequence), loops over the G query heads
//        of the group and the query blocks that see this key block:
//        S^T = K Q^T, dP^T = V dO^T         (lanes = keys, columns = queries)
//        P^T, dS^T -> bf16 in TMEM
//        dV += P^T dO,  dK += dS^T Q        (TS MMAs; dO and Q tiles read MN-major)
//   Both scale by the softmax scale in the epilogue.  No atomics: every output row has one writer.
//
// What bounds them: a 128 x 128 block takes 16 D cycles of the tensor core in the dK/dV kernel and 12 D in the dQ kernel, and
// 16384 exponentials in either.  The conversions of a block are two phases, P from the scores and dS from dP, each behind a
// barrier of its own, so that the tensor core computes the other product of this block or the next block's scores
// meanwhile; all products are 128 wide (64-wide ones wait for shared memory: 6 KB per 32 cycles).
// Measured, before (64-wide halves, eight softmax warps, 2^x on bf16 pairs) and now: 1 x 16384, 32 / 8 heads of 128, causal
// 9047 -> 6461 us (608 -> 851 TFLOP/s of the five products that a backward pass cannot do without); 2 x 4096 1473 -> 1083 us;
// 4 x 5329, 16 heads of 64, not causal 4046 -> 2392 us (287 -> 486).  Eight warps with 64 columns each: 7108, 1183, 2694 us.
#pragma once
#include "attention_math.cuh"

namespace yv {

struct AttnBwdParams {
  CUtensorMap tma_q, tma_k, tma_v, tma_do;   // 3-D (d, head, token), box (64, 1, 128)
  __nv_bfloat16* dq;
  __nv_bfloat16* dk;
  __nv_bfloat16* dv;
  const float* lse;      // [hq, total_q] natural log
  const float* delta;    // [hq, total_q]
  const int* cu_q;
  const int* cu_k;
  int hq, hk;
  int64_t dq_stride, dk_stride, dv_stride;
  int64_t total_q;
  int causal;
  float scale;           // softmax scale
  float scale_log2;      // scale * log2(e)
  uint32_t* status;
};

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kAttnBwdPoly = 4;     // pairs of 16 whose 2^x is a polynomial
// Backward CTAs: TMA warp, MMA warp and sixteen softmax warps (four per TMEM lane quarter, each converting a quarter of a
// block's columns): four warps per scheduler hide one another's latencies.
constexpr int kAttnBwdSoftmaxWarps = 16;
constexpr int kAttnBwdSoftmaxThreads = 32 * kAttnBwdSoftmaxWarps;
constexpr int kAttnBwdThreads = 64 + kAttnBwdSoftmaxThreads;

template <int D>
struct AttnBwdSmem {
  static constexpr int kTile = 128 * D * 2;
  static constexpr int kStages = 2;
  static constexpr int kTotal = kTile * (2 + 2 * kStages) + 2 * 2 * 128 * 4 + 256 + 1024;
  // dQ kernel: a third K stage, because a block's K is read until its dQ product, after which the scores of the block two
  // further on are issued
  static constexpr int kStagesK = 3;
  static constexpr int kTotalDQ = kTile * (2 + kStages + kStagesK) + 256 + 1024;
};

// --------------------------------------------------------------------------------------------------
// dQ kernel
// --------------------------------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(kAttnBwdThreads, 1) attn_bwd_dq_kernel(const __grid_constant__ AttnBwdParams p) {
  using S = AttnBwdSmem<D>;
  constexpr int kStages = S::kStages, kStagesK = S::kStagesK;
  constexpr int kDBoxes = D / 64;
  constexpr uint32_t kBoxBytes = 128 * 128;
  // TMEM: S of key block j at [128 (j % 2), + 128), dS over it (bf16: the 32 keys of a warp's columns in the first 16 of
  // them); dP at [256, 384); dQ at [384, 384 + D).  The scores of block j + 1 are ready before dS of block j is.
  constexpr uint32_t kIdescNT = make_idesc_bf16(128, 128, false, false);   // S, dP: 128 queries x 128 keys
  constexpr uint32_t kIdescDQ = make_idesc_bf16(128, D, false, true);      // dS (TMEM) x K (MN-major)
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kColDP = 256, kColDQ = 384;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sDO = sQ + S::kTile;
  uint8_t* sK = sDO + S::kTile;
  uint8_t* sV = sK + kStagesK * S::kTile;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + kStages * S::kTile);
  uint64_t* qdo_full = bars;            // [1]
  uint64_t* v_full = bars + 1;          // [2]
  uint64_t* v_empty = bars + 3;         // [2]  released after dP MMA
  uint64_t* s_full = bars + 5;          // [2]  scores of a TMEM stage ready
  uint64_t* dp_full = bars + 7;         // [1]
  uint64_t* ds_full = bars + 8;         // [1]  one arrival per softmax warp: dS written, dP read
  uint64_t* dq_done = bars + 9;         // [1]
  uint64_t* k_full = bars + 10;         // [3]
  uint64_t* k_empty = bars + 13;        // [3]  released after dQ MMA (last reader of K_j)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.z, h = blockIdx.y;
  const int hkv = h / (p.hq / p.hk);
  const int q_begin = p.cu_q[b], q_len = p.cu_q[b + 1] - q_begin;
  const int k_begin = p.cu_k[b], k_len = p.cu_k[b + 1] - k_begin;
  const int n_qblk = (q_len + 127) / 128;
  const int q_blk = n_qblk - 1 - static_cast<int>(blockIdx.x);
  if (q_blk < 0) return;
  const int q0 = q_blk * 128;
  const int causal_shift = k_len - q_len;
  int n_kv = (k_len + 127) / 128;
  if (p.causal) {
    const int last_key = q0 + 127 + causal_shift;
    const int lim = last_key / 128 + 1;
    n_kv = last_key < 0 ? 0 : (lim < n_kv ? lim : n_kv);
  }

  if (threadIdx.x == 0) {
    mbar_init(qdo_full, 1);
    for (int s = 0; s < kStagesK; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); mbar_init(&s_full[s], 1); }
    mbar_init(dp_full, 1);
    mbar_init(ds_full, kAttnBwdSoftmaxWarps);
    mbar_init(dq_done, 1);
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, kTmemCols); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one() && n_kv > 0) {
      mbar_expect_tx(qdo_full, 2 * S::kTile);
#pragma unroll
      for (int c = 0; c < kDBoxes; ++c) {
        tma_load_3d(sQ + c * kBoxBytes, &p.tma_q, qdo_full, c * 64, h, q_begin + q0);
        tma_load_3d(sDO + c * kBoxBytes, &p.tma_do, qdo_full, c * 64, h, q_begin + q0);
      }
      bool ok = true;
      for (int j = 0; j < n_kv && ok; ++j) {
        const int s = j % kStages, sk = j % kStagesK;
        const uint32_t ph = (j / kStages) & 1u;
        ok = mbar_wait(&k_empty[sk], ((j / kStagesK) & 1u) ^ 1u, p.status);
        if (!ok) break;
        mbar_expect_tx(&k_full[sk], S::kTile);
#pragma unroll
        for (int c = 0; c < kDBoxes; ++c)
          tma_load_3d(sK + sk * S::kTile + c * kBoxBytes, &p.tma_k, &k_full[sk], c * 64, hkv, k_begin + j * 128);
        ok = mbar_wait(&v_empty[s], ph ^ 1u, p.status);
        if (!ok) break;
        mbar_expect_tx(&v_full[s], S::kTile);
#pragma unroll
        for (int c = 0; c < kDBoxes; ++c)
          tma_load_3d(sV + s * S::kTile + c * kBoxBytes, &p.tma_v, &v_full[s], c * 64, hkv, k_begin + j * 128);
      }
    }
  } else if (warp == 1) {
    if (elect_one() && n_kv > 0) {
      bool ok = mbar_wait(qdo_full, 0, p.status);
      const uint32_t aQ = smem_u32(sQ), aDO = smem_u32(sDO);
      auto issue_s = [&](int j) -> bool {
        const int s = j % kStagesK;
        if (!mbar_wait(&k_full[s], (j / kStagesK) & 1u, p.status)) return false;
        tc_fence_after_sync();
        const uint32_t aK = smem_u32(sK + s * S::kTile);
        const uint32_t tS = tmem_base + static_cast<uint32_t>((j & 1) * 128);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk / 4) * kBoxBytes + (kk % 4) * 32;
          tc_mma_f16_ss(tS, make_smem_desc(aQ + off, 16, 1024), make_smem_desc(aK + off, 16, 1024), kIdescNT,
                        kk != 0 ? 1u : 0u);
        }
        tc_commit(&s_full[j & 1]);
        return true;
      };
      auto issue_dp = [&](int j) -> bool {
        const int s = j % kStages;
        if (!mbar_wait(&v_full[s], (j / kStages) & 1u, p.status)) return false;
        tc_fence_after_sync();
        const uint32_t aV = smem_u32(sV + s * S::kTile);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk / 4) * kBoxBytes + (kk % 4) * 32;
          tc_mma_f16_ss(tmem_base + kColDP, make_smem_desc(aDO + off, 16, 1024), make_smem_desc(aV + off, 16, 1024),
                        kIdescNT, kk != 0 ? 1u : 0u);
        }
        tc_commit(&v_empty[s]);                          // V_j is read by the dP product only
        tc_commit(dp_full);
        return true;
      };
      if (ok) ok = issue_s(0);
      if (ok) ok = issue_dp(0);
      if (ok && n_kv > 1) ok = issue_s(1);
      for (int j = 0; j < n_kv && ok; ++j) {
        ok = mbar_wait(ds_full, j & 1u, p.status);
        if (!ok) break;
        tc_fence_after_sync();
        if (j + 1 < n_kv) {                              // dP first: the softmax threads wait for it next
          ok = issue_dp(j + 1);
          if (!ok) break;
        }
        const int s = j % kStagesK;
        const uint32_t aK = smem_u32(sK + s * S::kTile);
        const uint32_t tS = tmem_base + static_cast<uint32_t>((j & 1) * 128);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {                 // 128 keys = 8 K-steps of 16
          tc_mma_f16_ts(tmem_base + kColDQ, tS + (kk >> 1) * 32 + (kk & 1) * 8,
                        make_smem_desc(aK + kk * 2048, kBoxBytes, 1024), kIdescDQ, (j | kk) != 0 ? 1u : 0u);
        }
        tc_commit(&k_empty[s]);
        if (j == n_kv - 1) tc_commit(dq_done);           // one completion, after the last product
        if (j + 2 < n_kv) ok = issue_s(j + 2);
      }
    }
  } else {
    const int quarter = warp & 3;
    const int part = (warp - 2) >> 2;                    // four warps per TMEM lane quarter split the columns
    const int row = quarter * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    const int q_pos = q0 + row;
    const bool q_valid = q_pos < q_len;
    const int key_limit = p.causal ? (q_pos + causal_shift) : (k_len - 1);
    const int64_t stat_idx = static_cast<int64_t>(h) * p.total_q + q_begin + q_pos;
    const float lse2 = q_valid ? p.lse[stat_idx] * kLog2e : 0.f;
    const float delta = q_valid ? p.delta[stat_idx] : 0.f;
    bool ok = true;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    const float2 nl2 = make_float2(-lse2, -lse2), nd2 = make_float2(-delta, -delta);
    for (int j = 0; j < n_kv && ok; ++j) {
      ok = mbar_wait(&s_full[j & 1], (j >> 1) & 1u, p.status);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t tS = tmem_base + lane_off + static_cast<uint32_t>((j & 1) * 128);
      const int c0 = part * 32;
      // last visible column of this thread's 32; the select per element is only needed on blocks that touch the causal
      // diagonal, the end of the keys or a query row past the end
      const int last = q_valid ? min(key_limit, k_len - 1) - j * 128 - c0 : -1;
      uint32_t sv[32];
      tmem_ld32(tS + c0, sv);
      tc_wait_ld();
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float2 x = __ffma2_rn(make_float2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), sc2, nl2);
        if (last < 31) {
          if (2 * i > last) x.x = -INFINITY;
          if (2 * i + 1 > last) x.y = -INFINITY;
        }
        const float2 e = ex2_pair<kAttnBwdPoly, true>(i, x);
        sv[2 * i] = __float_as_uint(e.x);
        sv[2 * i + 1] = __float_as_uint(e.y);
      }
      ok = mbar_wait(dp_full, j & 1u, p.status);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t dv[32], pk[16];
      tmem_ld32(tmem_base + lane_off + kColDP + c0, dv);
      tc_wait_ld();
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 dd = __fadd2_rn(make_float2(__uint_as_float(dv[2 * i]), __uint_as_float(dv[2 * i + 1])), nd2);
        const float2 r = __fmul2_rn(make_float2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), dd);
        pk[i] = pack_bf16(r.x, r.y);
      }
      tmem_st16(tS + c0, pk);                            // over this warp's own columns of the scores
      tc_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
    }
    if (ok && n_kv > 0) {
      ok = mbar_wait(dq_done, 0u, p.status);
      ok = __all_sync(0xFFFFFFFFu, ok);
    }
    if (ok) {
      tc_fence_after_sync();
      __nv_bfloat16* orow = p.dq + static_cast<int64_t>(q_begin + q_pos) * p.dq_stride + static_cast<int64_t>(h) * D;
#pragma unroll
      for (int c = part; c < D / 32; c += 4) {             // the warps of a quarter share the columns
        uint32_t ov[32];
        if (n_kv > 0) {
          tmem_ld32(tmem_base + lane_off + kColDQ + c * 32, ov);
          tc_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) ov[i] = 0u;
        }
        if (q_valid) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 v;
            v.x = pack_bf16(__uint_as_float(ov[8 * i + 0]) * p.scale, __uint_as_float(ov[8 * i + 1]) * p.scale);
            v.y = pack_bf16(__uint_as_float(ov[8 * i + 2]) * p.scale, __uint_as_float(ov[8 * i + 3]) * p.scale);
            v.z = pack_bf16(__uint_as_float(ov[8 * i + 4]) * p.scale, __uint_as_float(ov[8 * i + 5]) * p.scale);
            v.w = pack_bf16(__uint_as_float(ov[8 * i + 6]) * p.scale, __uint_as_float(ov[8 * i + 7]) * p.scale);
            *reinterpret_cast<uint4*>(orow + c * 32 + i * 8) = v;
          }
        }
      }
    }
  }

  tc_fence_before_sync();
  block_settle(p.status);
  if (warp == 1) { tc_fence_after_sync(); tmem_dealloc(tmem_base, kTmemCols); }
}

}  // namespace yv

#include "attention_bwd_dkv.cuh"
