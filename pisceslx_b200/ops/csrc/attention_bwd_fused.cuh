// Flash attention backward in one pass over the score blocks (see attention_bwd.cuh for the two-kernel form).
//
//   attn_stats_kernel       per (head, token): delta = <dO, O>; -lse / scale and -delta as three bf16 terms each, 16 bytes
//   attn_bwd_fused_kernel   one CTA per (128-key block, KV head, sequence), loops over the G query heads of the group and the
//                           query blocks that see this key block:
//        S^T = K Q^T - lse / scale, dP^T = V dO^T - delta      (SS MMAs; lanes = keys, columns = queries)
//        P^T, dS^T -> bf16 in TMEM, dS^T also into shared memory
//        dV += P^T dO,  dK += dS^T Q                           (TS MMAs)
//        dQ  = dS K                                            (SS MMA, dS read MN-major from the tile of dS^T)
//        dQ is added to an fp32 sum in memory by bulk reductions, 16 columns of 128 queries at a time
//   attn_dq_finish_kernel   scaled sums -> bf16 rows
//
// Five products a block where the two kernels computed seven, and one set of exponentials and dS instead of two.  The order in
// which blocks are added to a query's sum is not fixed; where the caller asks for reproducible bits, the two kernels run.
//
// The statistics of the queries, which are columns here, enter through the tensor core: one more step of 16 along the summed
// dimension, ones times the three terms of each, whose sum has the 24 bits of the fp32 value.  Read from shared memory by the
// threads they cost 16 LDS.128 a warp and block, 128 KB that come back at 128 bytes a cycle.
//
// What bounds it (cycles a block of 128 x 128 and SM, of which the tensor core needs 2690 at 128 and 1540 at 64): at 128 4510, the
// chain dQ product - dQ out of TMEM - dP^T over its columns - dS^T, and the 64 KB of adds, of which L2 takes 6.2 TB/s in all
// (3000 cycles); without the adds it is 4130.  At 64 3030, the softmax warps' chain of loads, exponentials and stores, whose special
// functions alone are 768.  Issuing from a whole warp, so that descriptors live in uniform registers, took 8 %, the statistics
// through the tensor core 15 % at 64, dQ in two steps instead of four waits for the adds 20 % at 128.
// Measured, delta to the last row of dq, two kernels and one: 1 x 16384, 32 / 8 heads of 128, causal 6640 -> 5170 us (830 -> 1060
// TFLOP/s of the five products); 2 x 4096 1083 -> 760; 4 x 5329, 16 heads of 64, not causal 2390 -> 1440 us.
#pragma once

namespace yv {

struct AttnBwdFusedParams {
  AttnBwdParams b;
  float* dq_acc;         // [heads of this launch][D / 16][total_q][16], see dq_piece
  const uint4* stats;    // [hq][total_q] terms of -lse / scale and -delta
  int hk0, heads;        // KV heads of this launch
  int batch, blocks;     // sequences; key blocks of the longest
};

constexpr int kFusedSoftmaxWarps = 16, kFusedDqWarps = 4;
// Warpgroups: 0 TMA (warp 0) and MMA (warp 1), 1 to 4 softmax, 5 dQ.  Registers a thread: 80 at launch, 6 x 80 = 48 + 4 x 88 + 80.
constexpr int kFusedThreads = 128 + 32 * (kFusedSoftmaxWarps + kFusedDqWarps);
constexpr int kFusedRegsIssue = 48, kFusedRegsSoftmax = 88;

template <int D>
struct AttnBwdFusedSmem {
  static constexpr int kTile = 128 * D * 2;
  static constexpr int kStagesQ = 2;
  static constexpr int kStagesDO = D == 128 ? 1 : 2;    // at 128 a second one does not fit beside dS
  static constexpr int kDS = 128 * 128 * 2;
  static constexpr int kStagesDS = D == 128 ? 1 : 2;
  // statistics: ones for the scores and for dP^T (a group of 8 rows each, which all rows share), two stages of 128 rows of 16
  // bytes, and 128 rows of zeros, the second half of the summed 16
  static constexpr int kStats = 2 * 128 + 3 * 2048;
  static constexpr int kChunk = 128 * 16 * 4;           // 16 columns of dQ
  static constexpr int kChunks = D == 128 ? 3 : 4;
  static constexpr int kTotal = kTile * (2 + kStagesQ + kStagesDO) + kStagesDS * kDS + kChunks * kChunk + kStats + 256 + 1024;
  static_assert(kTotal <= 227 * 1024, "shared memory of an SM");
};

// Place of the 16-byte piece j of a token's 16 columns in the sums of dq: pieces are turned with the token, so that the threads of
// a warp, a token each, meet no bank of shared memory twice.
__device__ __forceinline__ int dq_piece(int64_t token, int j) { return j ^ (static_cast<int>(token >> 1) & 3); }

// Unswizzled K-major operand of 16 along the summed dimension: rows of 16 bytes, the groups of 8 rows `sbo` bytes apart, the second
// 8 of the 16 `lbo` bytes behind the first.
__device__ __forceinline__ uint64_t make_smem_desc_plain(const uint8_t* tile, uint32_t lbo, uint32_t sbo) {
  return static_cast<uint64_t>((smem_u32(tile) & 0x3FFFFu) >> 4) | static_cast<uint64_t>(lbo >> 4) << 16 |
         static_cast<uint64_t>(sbo >> 4) << 32 | static_cast<uint64_t>(1) << 46;
}

__device__ __forceinline__ void bulk_reduce_add_f32(float* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)),
               "r"(bytes)
               : "memory");
}

// Three bf16 terms whose sum is v (to its 24 bits).  An infinite v is held at the largest bf16 value: it stands for a query that
// sees no key, whose scores are masked, and has to stay finite beside the zeros that it is multiplied with.
__device__ __forceinline__ void bf16_terms(float v, uint32_t (&t)[3]) {
  const float top = __uint_as_float(0x7F7F0000u);
  if (fabsf(v) > top) v = copysignf(top, v);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat16 b = __float2bfloat16_rn(v);
    t[i] = __bfloat16_as_ushort(b);
    v -= __bfloat162float(b);
  }
}

// D / 8 lanes per (token, head), as attn_delta_kernel.
template <int D, bool VEC>
__global__ void __launch_bounds__(256) attn_stats_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                                                         const float* __restrict__ lse, uint4* __restrict__ stats,
                                                         int64_t total_q, int hq, int64_t o_stride, int64_t do_stride,
                                                         float inv_scale) {
  constexpr int kLanes = D / 8;
  const int64_t w = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) / kLanes;
  const int c = threadIdx.x & (kLanes - 1);
  const int64_t t = w / hq;
  const int h = static_cast<int>(w - t * hq);
  const int64_t at = static_cast<int64_t>(h) * total_q + t;
  const float l = c == 0 && t < total_q ? lse[at] : 0.f;
  const float s = attn_delta_row<D, VEC>(o, dout, t, h, c, t < total_q, o_stride, do_stride);
  if (c == 0 && t < total_q) {
    uint32_t lt[3], dt[3];
    bf16_terms(-l * inv_scale, lt);
    bf16_terms(-s, dt);
    stats[at] = make_uint4(lt[0] | lt[1] << 16, lt[2] | dt[0] << 16, dt[1] | dt[2] << 16, 0u);
  }
}

template <int D>
__global__ void __launch_bounds__(kFusedThreads, 1) attn_bwd_fused_kernel(const __grid_constant__ AttnBwdFusedParams fp) {
  using S = AttnBwdFusedSmem<D>;
  const AttnBwdParams& p = fp.b;
  constexpr int kStagesQ = S::kStagesQ, kStagesDO = S::kStagesDO;
  constexpr int kDBoxes = D / 64;
  constexpr uint32_t kBoxBytes = 128 * 128;
  constexpr uint32_t kIdescNT = make_idesc_bf16(128, 128, false, false);    // 128 keys x 128 queries
  constexpr uint32_t kIdescAcc = make_idesc_bf16(128, D, false, true);      // dV, dK: 128 keys x D
  constexpr uint32_t kIdescDQ = make_idesc_bf16(128, D, true, true);        // 128 queries x D over keys
  // TMEM columns: [0,128) S^T; [128,256) dP^T, then dS^T over it (bf16: the 32 queries of a warp's columns in the first 16 of
  // them).  At 64: dQ [256,320), dV [320,384), dK [384,448), P^T [448,512), so that the next scores are computed as soon as
  // these have been read.  At 128: dV, dK behind dP^T, P^T over S^T like dS^T, and dQ over dS^T once dK has read it.
  constexpr bool kRoom = D == 64;
  constexpr uint32_t kTmemCols = 512, kColDP = 128;
  constexpr uint32_t kColDQ = kRoom ? 256 : 128, kColDV = kRoom ? 320 : 256, kColDK = 384;
  constexpr uint32_t kColP = kRoom ? 448 : 0, kPPitch = kRoom ? 16 : 32;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + S::kTile;
  uint8_t* sQ = sV + S::kTile;
  uint8_t* sDO = sQ + kStagesQ * S::kTile;
  uint8_t* sDS = sDO + kStagesDO * S::kTile;            // dS^T: 128 key rows of 64 queries, two boxes, 128-byte swizzle
  uint8_t* sDQ = sDS + S::kStagesDS * S::kDS;                          // chunks of dQ on their way to memory: [128 queries][16] fp32
  uint8_t* sOnes = sDQ + S::kChunks * S::kChunk;        // ones that pick the terms of -lse / scale, then those of -delta
  uint8_t* sStat = sOnes + 2 * 128;
  uint8_t* sZero = sStat + 2 * 2048;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sZero + 2048);
  uint64_t* kv_full = bars;             // [1]
  uint64_t* q_full = bars + 1;          // [2]
  uint64_t* q_empty = bars + 3;         // [2]
  uint64_t* do_full = bars + 5;         // [2]
  uint64_t* do_empty = bars + 7;        // [2]
  uint64_t* s_full = bars + 9;          // [1]
  uint64_t* dp_full = bars + 10;        // [1]
  uint64_t* p_full = bars + 11;         // [1] one arrival per softmax warp: P^T written
  uint64_t* ds_full = bars + 12;        // [1] likewise: dS^T written, dP^T read
  uint64_t* dq_full = bars + 13;        // [1] dQ of the block ready, the tile of dS^T read
  uint64_t* dq_read = bars + 14;        // [1] one arrival per dQ warp
  uint64_t* acc_done = bars + 15;       // [1]
  uint64_t* s_read = bars + 16;         // [1] one arrival per softmax warp: S^T read
  uint64_t* ds_free = bars + 17;        // [1] the tile of dS^T, which dQ has passed through on its way, may be written
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);

  const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  // With the causal mask the first key blocks of all heads and sequences come first, since they see the most queries: the short
  // ones fill the end.  Without it the blocks of a head are neighbours.
  const int units = fp.heads * fp.batch;
  const int unit = p.causal ? blockIdx.x % units : blockIdx.x / fp.blocks;
  const int k_blk = p.causal ? blockIdx.x / units : blockIdx.x % fp.blocks;
  const int b = unit / fp.heads, head0 = unit % fp.heads, hkv = fp.hk0 + head0;
  const int G = p.hq / p.hk;
  const int q_begin = p.cu_q[b], q_len = p.cu_q[b + 1] - q_begin;
  const int k_begin = p.cu_k[b], k_len = p.cu_k[b + 1] - k_begin;
  const int n_kblk = (k_len + 127) / 128;
  if (k_blk >= n_kblk) return;
  const int k0 = k_blk * 128;
  const int causal_shift = k_len - q_len;
  const int n_qblk = (q_len + 127) / 128;
  int i_start = 0;
  if (p.causal) {
    const int first_q = k0 - causal_shift;          // first query position that sees key k0
    i_start = first_q > 0 ? first_q / 128 : 0;
  }
  const int n_i = n_qblk > i_start ? n_qblk - i_start : 0;
  const int n_it = n_i * G;
  // Steps of the loop: query blocks of a head, then the next head.  CTAs of one head start at blocks of their own, so that
  // they do not add to the same sums at once (with the causal mask they do by themselves).
  struct Step {
    int i, g, left;
  };
  const int turn = n_i > 0 && !p.causal ? k_blk % n_i : 0;
  auto first_step = [&]() -> Step { return Step{i_start + turn, 0, n_i}; };
  auto advance = [&](Step& s) {
    if (++s.i == n_qblk) s.i = i_start;
    if (--s.left == 0) { s.left = n_i; ++s.g; s.i = i_start + turn; }
  };

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 1); mbar_init(&do_full[s], 1);
      mbar_init(&q_empty[s], 1); mbar_init(&do_empty[s], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_full, kFusedSoftmaxWarps);
    mbar_init(ds_full, kFusedSoftmaxWarps);
    mbar_init(dq_full, 1);
    mbar_init(dq_read, kFusedDqWarps);
    mbar_init(acc_done, 1);
    mbar_init(s_read, kFusedSoftmaxWarps);
    mbar_init(ds_free, 1);
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, kTmemCols); tmem_relinquish(); }
  for (int i = threadIdx.x; i < S::kStats / 16; i += kFusedThreads)
    reinterpret_cast<uint4*>(sOnes)[i] = i < 8 ? make_uint4(0x3F803F80u, 0x00003F80u, 0u, 0u)
                                         : i < 16 ? make_uint4(0u, 0x3F800000u, 0x3F803F80u, 0u) : make_uint4(0u, 0u, 0u, 0u);
  fence_proxy_async_smem();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < 4) {
    regs_give<kFusedRegsIssue>();
    if (warp == 0 && elect_one() && n_it > 0) {
      mbar_expect_tx(kv_full, 2 * S::kTile);
#pragma unroll
      for (int c = 0; c < kDBoxes; ++c) {
        tma_load_3d(sK + c * kBoxBytes, &p.tma_k, kv_full, c * 64, hkv, k_begin + k0);
        tma_load_3d(sV + c * kBoxBytes, &p.tma_v, kv_full, c * 64, hkv, k_begin + k0);
      }
      bool ok = true;
      Step at = first_step();
      for (int it = 0; it < n_it && ok; ++it, advance(at)) {
        const int h = hkv * G + at.g, row = q_begin + at.i * 128;
        const int s = it % kStagesQ, sd = it % kStagesDO;
        ok = mbar_wait(&q_empty[s], ((it / kStagesQ) & 1u) ^ 1u, p.status);
        if (!ok) break;
        const uint32_t stat_bytes = 16u * static_cast<uint32_t>(min(static_cast<int64_t>(128), p.total_q - row));
        mbar_expect_tx(&q_full[s], S::kTile + stat_bytes);
        bulk_load_1d(sStat + s * 2048, fp.stats + static_cast<int64_t>(h) * p.total_q + row, stat_bytes, &q_full[s]);
#pragma unroll
        for (int c = 0; c < kDBoxes; ++c)
          tma_load_3d(sQ + s * S::kTile + c * kBoxBytes, &p.tma_q, &q_full[s], c * 64, h, row);
        ok = mbar_wait(&do_empty[sd], ((it / kStagesDO) & 1u) ^ 1u, p.status);
        if (!ok) break;
        mbar_expect_tx(&do_full[sd], S::kTile);
#pragma unroll
        for (int c = 0; c < kDBoxes; ++c)
          tma_load_3d(sDO + sd * S::kTile + c * kBoxBytes, &p.tma_do, &do_full[sd], c * 64, h, row);
      }
    }
    if (warp == 1 && n_it > 0) {
      // The whole warp runs this and one thread issues: descriptors stay in uniform registers.
      const uint32_t lead = elect_one() ? 1u : 0u;
      bool ok = mbar_wait_warp(kv_full, 0, p.status);
      // Descriptors of the tiles, made anew from these at each product (kept for every step of every product they would not fit
      // into the registers).  K-major: a step of 16 along d; MN-major: of 16 rows.
      auto k_major = [](const uint8_t* tile) { return (make_smem_desc(smem_u32(tile), 16, 1024)); };
      auto mn_major = [](const uint8_t* tile) { return (make_smem_desc(smem_u32(tile), kBoxBytes, 1024)); };
      auto along_d = [](int kk) -> uint64_t { return ((kk / 4) * kBoxBytes + (kk % 4) * 32) >> 4; };
      auto along_rows = [](int kk) -> uint64_t { return kk * 2048 >> 4; };
      auto ones = [&](int which) { return make_smem_desc_plain(sOnes + which * 128, smem_u32(sZero) - smem_u32(sOnes + which * 128), 0); };
      auto stat_rows = [&](int it) {
        const uint8_t* tile = sStat + (it % kStagesQ) * 2048;
        return make_smem_desc_plain(tile, smem_u32(sZero) - smem_u32(tile), 128);
      };
      auto issue_s = [&](int it) -> bool {
        const int s = it % kStagesQ;
        if (!mbar_wait_warp(&q_full[s], (it / kStagesQ) & 1u, p.status)) return false;
        tc_fence_after_sync();
        const uint64_t dk = k_major(sK), dq = k_major(sQ + s * S::kTile);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          tc_mma_f16_ss_if(lead, tmem_base, dk + along_d(kk), dq + along_d(kk), kIdescNT, kk != 0 ? 1u : 0u);
        tc_mma_f16_ss_if(lead, tmem_base, ones(0), stat_rows(it), kIdescNT, 1u);
        tc_commit_if(lead, s_full);
        return true;
      };
      auto issue_dp = [&](int it) -> bool {
        const int s = it % kStagesDO;
        if (!mbar_wait_warp(&do_full[s], (it / kStagesDO) & 1u, p.status)) return false;
        tc_fence_after_sync();
        const uint64_t dv = k_major(sV), ddo = k_major(sDO + s * S::kTile);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          tc_mma_f16_ss_if(lead, tmem_base + kColDP, dv + along_d(kk), ddo + along_d(kk), kIdescNT, kk != 0 ? 1u : 0u);
        tc_mma_f16_ss_if(lead, tmem_base + kColDP, ones(1), stat_rows(it), kIdescNT, 1u);   // with the scores' terms: Q has arrived
        tc_commit_if(lead, dp_full);
        return true;
      };
      // dV of block `it`; the block's dO has arrived or is waited for
      auto issue_dv = [&](int it) -> bool {
        const int s = it % kStagesDO;
        if (!kRoom && !mbar_wait_warp(p_full, it & 1u, p.status)) return false;
        if (!mbar_wait_warp(&do_full[s], (it / kStagesDO) & 1u, p.status)) return false;
        tc_fence_after_sync();
        const uint64_t ddo = mn_major(sDO + s * S::kTile);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)                   // 128 queries = 8 K-steps of 16
          tc_mma_f16_ts_if(lead, tmem_base + kColDV, tmem_base + kColP + (kk >> 1) * kPPitch + (kk & 1) * 8, ddo + along_rows(kk), kIdescAcc,
                        (it | kk) != 0 ? 1u : 0u);
        return true;
      };
      if (ok) ok = issue_s(0);
      if (ok) ok = issue_dp(0);
      if (!kRoom) {
        if (ok) ok = issue_dv(0);
        if (ok) {
          tc_commit_if(lead, &do_empty[0]);
          if (n_it > 1) ok = issue_s(1);                 // over P^T, which dV has read
        }
      }
      for (int it = 0; it < n_it && ok; ++it) {
        const bool more = it + 1 < n_it;
        if (kRoom && more) {
          ok = mbar_wait_warp(s_read, it & 1u, p.status) && issue_s(it + 1);
          if (!ok) break;
        }
        ok = mbar_wait_warp(ds_full, it & 1u, p.status);
        if (!ok) break;
        tc_fence_after_sync();
        if (kRoom) {                                     // P^T and dS^T arrive together
          ok = issue_dv(it);
          if (!ok) break;
          tc_commit_if(lead, &do_empty[it % kStagesDO]);
        }
        const uint64_t dq = mn_major(sQ + (it % kStagesQ) * S::kTile);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          tc_mma_f16_ts_if(lead, tmem_base + kColDK, tmem_base + kColDP + (kk >> 1) * 32 + (kk & 1) * 8, dq + along_rows(kk),
                        kIdescAcc, (it | kk) != 0 ? 1u : 0u);
        tc_commit_if(lead, &q_empty[it % kStagesQ]);
        if (!more) tc_commit_if(lead, acc_done);
        if (kRoom) {
          if (more) ok = issue_dp(it + 1);               // over dS^T, which dK has read
          if (ok && it > 0) ok = mbar_wait_warp(dq_read, (it - 1) & 1u, p.status);
          if (!ok) break;
          tc_fence_after_sync();
        }
        const uint64_t dds = mn_major(sDS + (it % S::kStagesDS) * S::kDS), dk = mn_major(sK);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)                   // 128 keys = 8 K-steps of 16
          tc_mma_f16_ss_if(lead, tmem_base + kColDQ, dds + along_rows(kk), dk + along_rows(kk), kIdescDQ, kk != 0 ? 1u : 0u);
        tc_commit_if(lead, dq_full);
        if (!more) break;
        if (!kRoom) {
          ok = mbar_wait_warp(dq_read, it & 1u, p.status);    // dQ leaves the columns of dP^T
          if (ok) ok = issue_dp(it + 1);
          if (ok) ok = issue_dv(it + 1);
          if (!ok) break;
          tc_commit_if(lead, &do_empty[(it + 1) % kStagesDO]);
          if (it + 2 < n_it) ok = issue_s(it + 2);
        }
      }
    }
  } else if (warp < 4 + kFusedSoftmaxWarps) {
    regs_take<kFusedRegsSoftmax>();
    // Sixteen softmax warps: four warps share each TMEM lane quarter (a warp may only touch lanes 32 (warp % 4) ..) and
    // split the 128 query columns of a block between them, 32 each.
    const int quarter = warp & 3;
    const int part = (warp - 4) >> 2;                    // which 32 of the 128 columns this warp converts
    const int row = quarter * 32 + lane;                 // key row of the tile
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    const int key = k0 + row;
    const bool key_valid = key < k_len;
    const uint32_t tST = tmem_base + lane_off + part * 32, tDPT = tST + kColDP;
    const uint32_t tP = tmem_base + lane_off + kColP + part * kPPitch;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    uint8_t* ds_row = sDS + (part >> 1) * kBoxBytes + row * 128;
    bool ok = true;
    Step at = first_step();
    for (int it = 0; it < n_it && ok; ++it, advance(at)) {
      const int qb = at.i * 128;
      ok = mbar_wait(s_full, it & 1u, p.status);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (!ok) break;
      tc_fence_after_sync();
      // query column c of this warp's 32 is visible to this key iff key <= (qb + c) + shift, and is one iff it lies before the end
      const int first_vis = !key_valid ? 32 : p.causal ? (key - causal_shift - qb - part * 32) : 0;
      const int end_vis = q_len - qb - part * 32;
      // every (key, query) pair of this block is visible: no per-element selects (uniform over the CTA)
      const bool full_vis = (!p.causal || qb >= k0 + 127 - causal_shift) && k0 + 128 <= k_len && qb + 128 <= q_len;
      uint32_t sv[32], pp[16];
      tmem_ld32(tST, sv);
      tc_wait_ld();
      if (kRoom) {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_read);
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float2 x = __fmul2_rn(make_float2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), sc2);
        if (!full_vis) {
          if (2 * i < first_vis || 2 * i >= end_vis) x.x = -INFINITY;
          if (2 * i + 1 < first_vis || 2 * i + 1 >= end_vis) x.y = -INFINITY;
        }
        const float2 e = ex2_pair<kAttnBwdPoly, true>(i, x);
        sv[2 * i] = __float_as_uint(e.x);
        sv[2 * i + 1] = __float_as_uint(e.y);
        pp[i] = pack_bf16(e.x, e.y);
      }
      if (!kRoom) {
        tmem_st16(tP, pp);
        tc_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
      }
      ok = mbar_wait(dp_full, it & 1u, p.status);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t dv[32], ds[16];
      tmem_ld32(tDPT, dv);
      if (kRoom) tmem_st16(tP, pp);                      // dV of the block before, which read P^T, is done: dP^T came behind it
      tc_wait_ld();
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 r = __fmul2_rn(make_float2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])),
                                    make_float2(__uint_as_float(dv[2 * i]), __uint_as_float(dv[2 * i + 1])));
        ds[i] = pack_bf16(r.x, r.y);
      }
      tmem_st16(tDPT, ds);
      // The tile of dS^T: at 64 there are two, and the dQ product of two blocks ago is done, because dP^T came behind it; at 128
      // the dQ of the block before has been computed from it and has left through it.
      if (!kRoom && it > 0) {
        ok = mbar_wait(ds_free, (it - 1) & 1u, p.status);
        ok = __all_sync(0xFFFFFFFFu, ok);
        if (!ok) break;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<uint4*>(ds_row + (it % S::kStagesDS) * S::kDS + ((((part & 1) * 4 + i) ^ (row & 7)) * 16)) =
            make_uint4(ds[4 * i], ds[4 * i + 1], ds[4 * i + 2], ds[4 * i + 3]);
      tc_wait_st();
      tc_fence_before_sync();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
    }
    if (ok && n_it > 0) {
      ok = mbar_wait(acc_done, 0u, p.status);
      ok = __all_sync(0xFFFFFFFFu, ok);
    }
    if (ok) {
      tc_fence_after_sync();
      const int64_t tok = k_begin + key;
      const int which = part >> 1;                         // two warps of the quarter write dV, two dK
      const uint32_t col = which == 0 ? kColDV : kColDK;
      const float sc = which == 0 ? 1.f : p.scale;
      __nv_bfloat16* orow = which == 0 ? p.dv + tok * p.dv_stride + static_cast<int64_t>(hkv) * D
                                       : p.dk + tok * p.dk_stride + static_cast<int64_t>(hkv) * D;
#pragma unroll
      for (int c = 0; c < D / 64; ++c) {
        const int c32 = (part & 1) * (D / 64) + c;
        uint32_t ov[32];
        if (n_it > 0) {
          tmem_ld32(tmem_base + lane_off + col + c32 * 32, ov);
          tc_wait_ld();
        } else {
#pragma unroll
          for (int i2 = 0; i2 < 32; ++i2) ov[i2] = 0u;
        }
        if (key_valid) {
#pragma unroll
          for (int i2 = 0; i2 < 4; ++i2) {
            uint4 v;
            v.x = pack_bf16(__uint_as_float(ov[8 * i2 + 0]) * sc, __uint_as_float(ov[8 * i2 + 1]) * sc);
            v.y = pack_bf16(__uint_as_float(ov[8 * i2 + 2]) * sc, __uint_as_float(ov[8 * i2 + 3]) * sc);
            v.z = pack_bf16(__uint_as_float(ov[8 * i2 + 4]) * sc, __uint_as_float(ov[8 * i2 + 5]) * sc);
            v.w = pack_bf16(__uint_as_float(ov[8 * i2 + 6]) * sc, __uint_as_float(ov[8 * i2 + 7]) * sc);
            *reinterpret_cast<uint4*>(orow + c32 * 32 + i2 * 8) = v;
          }
        }
      }
    }
  } else {
    // Four dQ warps, one per TMEM lane quarter, a query per thread: 16 columns at a time into shared memory, from where a bulk
    // reduction adds them to the sums.  Of 128 columns 64 wait in registers, so that TMEM is free before they have left.
    const int quarter = warp & 3;
    const uint32_t tDQ = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + kColDQ;
    const int row = quarter * 32 + lane;
    const bool leader = threadIdx.x == kFusedThreads - 128;
    constexpr int kHeld = 4;                             // chunks in registers
    Step at = first_step();
    for (int it = 0; it < n_it; ++it, advance(at)) {
      const int64_t token = q_begin + at.i * 128;
      const uint32_t bytes = 64u * static_cast<uint32_t>(min(128, q_len - at.i * 128));
      float* acc = fp.dq_acc + ((static_cast<int64_t>(head0) * G + at.g) * (D / 16) * p.total_q + token) * 16;
      const bool mine = mbar_wait(dq_full, it & 1u, p.status);
      if (leader) tma_store_wait_read<0>();              // the block before has left its chunks
      uint32_t all_ok;                                   // the four warps go on together or not at all
      asm volatile(
          "{\n"
          ".reg .pred pin, pout;\n"
          "setp.ne.u32 pin, %1, 0;\n"
          "bar.red.and.pred pout, 1, 128, pin;\n"
          "selp.u32 %0, 1, 0, pout;\n"
          "}\n"
          : "=r"(all_ok)
          : "r"(static_cast<uint32_t>(mine))
          : "memory");
      if (all_ok == 0u) break;
      tc_fence_after_sync();
      uint32_t r[kHeld][16];
      auto load = [&](int c) { tmem_ld16(tDQ + c * 16, r[c % kHeld]); };
      auto release = [&]() {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(dq_read);
      };
      auto store = [&](int c, uint8_t* chunk) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          *reinterpret_cast<uint4*>(chunk + row * 64 + dq_piece(token + row, j) * 16) =
              make_uint4(r[c % kHeld][4 * j], r[c % kHeld][4 * j + 1], r[c % kHeld][4 * j + 2], r[c % kHeld][4 * j + 3]);
      };
      auto stored = []() {
        fence_proxy_async_smem();
        asm volatile("bar.sync 1, 128;" ::: "memory");
      };
      auto send = [&](int c, const uint8_t* chunk) { bulk_reduce_add_f32(acc + static_cast<int64_t>(c) * p.total_q * 16, chunk, bytes); };
#pragma unroll
      for (int c = 0; c < kHeld; ++c) load(c);
      tc_wait_ld();
      if (D == 64) {
        release();
#pragma unroll
        for (int c = 0; c < 4; ++c) store(c, sDQ + c * S::kChunk);
        stored();
        if (leader) {
#pragma unroll
          for (int c = 0; c < 4; ++c) send(c, sDQ + c * S::kChunk);
          tma_store_commit();
        }
      } else {
        // Two chunks through the tile of dS^T, which the product was the last to read, three through places of their own; the
        // other three wait in registers for those.
        store(0, sDS);
        store(1, sDS + S::kChunk);
        store(2, sDQ);
        store(3, sDQ + S::kChunk);
#pragma unroll
        for (int c = 4; c < 8; ++c) load(c);
        tc_wait_ld();
        release();
        store(4, sDQ + 2 * S::kChunk);
        stored();
        if (leader) {
          send(0, sDS);
          send(1, sDS + S::kChunk);
          tma_store_commit();
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            send(2 + i, sDQ + i * S::kChunk);
            tma_store_commit();
          }
          tma_store_wait_read<3>();
          mbar_arrive(ds_free);
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          if (leader) tma_store_wait_read<2>();
          asm volatile("bar.sync 1, 128;" ::: "memory"); // the chunk that was here has left
          store(5 + i, sDQ + i * S::kChunk);
          stored();
          if (leader) {
            send(5 + i, sDQ + i * S::kChunk);
            tma_store_commit();
          }
        }
      }
    }
    if (leader) tma_store_wait_all<0>();
  }

  tc_fence_before_sync();
  block_settle(p.status);
  if (warp == 1) { tc_fence_after_sync(); tmem_dealloc(tmem_base, kTmemCols); }
}

// dq[t][h * D ..] = scale * sums: a thread turns 8 columns of a token, its two pieces of the sums, into 16 bytes of a row; the threads
// of a warp cover 64 contiguous bytes of sums a token and 16 tokens, or 32 bytes of a row.
template <int D>
__global__ void __launch_bounds__(256) attn_dq_finish_kernel(const float4* __restrict__ acc, __nv_bfloat16* __restrict__ dq,
                                                             int64_t total_q, int64_t dq_stride, int h0, float scale) {
  __shared__ uint4 tile[32 * (D / 8)];
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * 32;
  const int h = blockIdx.y;
  constexpr int kItems = 32 * (D / 8);                   // (16 columns, token, half)
#pragma unroll
  for (int i = threadIdx.x; i < kItems; i += 256) {
    const int c = i / 64, t = (i >> 1) & 31, half = i & 1;
    if (t0 + t < total_q) {
      const float4* src = acc + ((static_cast<int64_t>(h) * (D / 16) + c) * total_q + t0 + t) * 4;
      const float4 a = src[dq_piece(t0 + t, 2 * half)], b = src[dq_piece(t0 + t, 2 * half + 1)];
      const int k = c * 2 + half;
      tile[t * (D / 8) + (k ^ (t & 7))] = make_uint4(pack_bf16(a.x * scale, a.y * scale), pack_bf16(a.z * scale, a.w * scale),
                                                      pack_bf16(b.x * scale, b.y * scale), pack_bf16(b.z * scale, b.w * scale));
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = threadIdx.x; i < kItems; i += 256) {
    const int t = i / (D / 8), k = i % (D / 8);
    if (t0 + t < total_q)
      *reinterpret_cast<uint4*>(dq + (t0 + t) * dq_stride + static_cast<int64_t>(h0 + h) * D + k * 8) = tile[t * (D / 8) + (k ^ (t & 7))];
  }
}

}  // namespace yv
