// Flash attention forward for sm_100a: GQA, causal or full, packed variable-length sequences.
//
// One persistent CTA per SM walks (query block, query head, sequence) items, heavy blocks first.  A block has two tiles of 128
// queries or one; the key tiles of a lone query tile are dealt out to both halves of the CTA in turn, whose sums are added at
// the end (the tile is "split").  384 threads:
//   warps 0..3  softmax of tile 0, warps 4..7 of tile 1 (split: of every other key tile): a thread owns one query row (= TMEM
//               lane): tcgen05.ld the 128 scores, online softmax with lazy rescaling of the O accumulator, pack P to bf16, tcgen05.st
//   warp 8      TMA producer: the item's two 128-row Q tiles, then K_j / V_j tiles through rings
//   warp 9      MMA issuer: per tile S = Q K_j^T (SS), O += P_j V_j (TS: P is read from TMEM where the softmax warps wrote it
//               over S); the two tiles take turns, so the tensor core works on one while the other is in softmax
//   warps 10,11 only give their registers to the softmax warps, which keep a row's 128 scores in registers
// TMEM columns: [0,128) S0/P0, [128,256) S1/P1, [256,256+D) O0, [384,384+D) O1.
//
// What bounds it: per 128 x 128 tile the tensor core needs 4 D cycles per product pair, one softmax group some 1000 cycles of
// issue and special-function work.  With one tile per CTA the two took turns; two tiles overlap them.  An item's
// Q loads, first scores and epilogue overlap the neighbouring items' work: nothing is allocated or set up per item.
// Measured, before (one tile per CTA, 2^x on bf16 pairs) and now: 1 x 16384, 32 / 8 heads of 128, causal 2368 -> 1810 us (929 ->
// 1215 TFLOP/s); 2 x 4096 390 -> 283 us; 4 x 5329, 16 heads of 64, not causal 1036 -> 775 us (449 -> 601 TFLOP/s).
// A lone tile, one half of the CTA idle and now split (and one tile per CTA): 64 queries of 8192 keys, 32 / 8 heads of 128 110 ->
// 67 us (86), 16 / 4 of 64 88 -> 56 (84); one after the other, S, softmax and P V of a tile leave nothing to overlap.
#pragma once
#include "attention_math.cuh"

namespace yv {

struct AttnFwdParams {
  CUtensorMap tma_q;   // 3-D (d, head, token), box (64, 1, 128)
  CUtensorMap tma_k;
  CUtensorMap tma_v;
  __nv_bfloat16* o;
  float* lse;          // [hq, total_q]
  const int* cu_q;     // [B+1]
  const int* cu_k;     // [B+1]
  int hq, hk, batch;
  int two;             // 1: items of two query tiles, 0: of one
  int64_t items;       // query blocks of the longest sequence times hq * batch, in descending order of work
  int64_t o_stride;    // elements between consecutive tokens of o
  int64_t total_q;
  int causal;
  float scale_log2;    // softmax scale * log2(e)
  uint32_t* status;
};

constexpr int kAttnThreads = 384;
constexpr int kAttnSoftmaxRegs = 208, kAttnOtherRegs = 88;   // 2 x 128 x 208 + 128 x 88 = 384 x 168, the launch's registers
constexpr int kAttnBlock = 128;     // query rows and key rows per tile
constexpr int kAttnFwdPoly = 4;     // pairs of 16 whose 2^x is a polynomial
constexpr float kMaskValue = -1.0e30f;
constexpr float kRescaleThreshold = 8.0f;   // log2 units: O is rescaled only when the row max grew by more

template <int D>
struct AttnFwdSmem {
  static constexpr int kTile = kAttnBlock * D * 2;       // bytes of one Q/K/V tile
  static constexpr int kStages = D == 64 ? 3 : 2;
  static constexpr int kTotal = kTile * (2 + 2 * kStages) + kAttnBlock * 8 + 256 + 1024;
};

// Item of round r of a CTA.  Every other round runs backwards, so that no CTA gets the heaviest item of each (16 rounds of a
// causal 8192-token prompt: the last CTA would otherwise work 28 % longer than the mean).
__device__ __forceinline__ int64_t attn_item_of(int64_t r) {
  return r * gridDim.x + ((r & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
}

// One item: a block of queries of one head of one sequence, and how many key tiles each half of the CTA works on.
struct AttnItem {
  int h, q0, q_begin, q_len, k_begin, k_len, shift;
  bool second;         // there is a second query tile
  bool split;          // both halves have the first query tile, and every other key tile of it
  int n[2];            // key tiles; a query tile that sees none is written as zeros
  __device__ __forceinline__ bool load(const AttnFwdParams& p, int64_t r) {
    const int64_t w = attn_item_of(r);
    if (w >= p.items) return false;
    const int per = p.hq * p.batch;
    const int rank = static_cast<int>(w / per), rest = static_cast<int>(w - static_cast<int64_t>(rank) * per);
    const int b = rest / p.hq;
    h = rest - b * p.hq;
    q_begin = p.cu_q[b];
    q_len = p.cu_q[b + 1] - q_begin;
    k_begin = p.cu_k[b];
    k_len = p.cu_k[b + 1] - k_begin;
    const int log_rows = 7 + p.two;
    const int blk = ((q_len + (1 << log_rows) - 1) >> log_rows) - 1 - rank;       // heavy (late) blocks first
    if (blk < 0) return false;
    q0 = blk << log_rows;
    second = p.two != 0 && q0 + kAttnBlock < q_len;
    // causal: query i (bottom-right aligned when k_len != q_len) sees keys <= i + (k_len - q_len)
    shift = k_len - q_len;
    const int all = (k_len + kAttnBlock - 1) / kAttnBlock;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      int v = all;
      if (p.causal) {
        const int last_key = q0 + (t + 1) * kAttnBlock - 1 + shift;
        const int lim = last_key / kAttnBlock + 1;
        v = last_key < 0 ? 0 : (lim < all ? lim : all);
      }
      n[t] = t == 0 || second ? v : 0;
    }
    split = !second && n[0] > 1;
    if (split) {
      n[1] = n[0] / 2;
      n[0] -= n[1];
    }
    return true;
  }
  __device__ __forceinline__ int count(int t) const { return t == 0 ? n[0] : n[1]; }
  __device__ __forceinline__ int tiles() const { return split ? n[0] + n[1] : n[0] > n[1] ? n[0] : n[1]; }
  __device__ __forceinline__ int steps() const { return n[0] > n[1] ? n[0] : n[1]; }
  // key tile of step j of a half, and first query of its tile
  __device__ __forceinline__ int key_tile(int t, int j) const { return split ? 2 * j + t : j; }
  __device__ __forceinline__ int first_query(int t) const { return q0 + (split ? 0 : t * kAttnBlock); }
  // whether a half's products of step j are the last that read its key tile
  __device__ __forceinline__ bool last_reader(int t, int j) const { return split || t == 1 || j >= n[1]; }
};

template <int D>
__global__ void __launch_bounds__(kAttnThreads, 1) attn_fwd_kernel(const __grid_constant__ AttnFwdParams p) {
  using S = AttnFwdSmem<D>;
  constexpr int kStages = S::kStages;
  constexpr int kDBoxes = D / 64;
  constexpr uint32_t kBoxBytes = kAttnBlock * 128;     // one (128 rows x 64 cols) box
  constexpr uint32_t kIdescQK = make_idesc_bf16(128, 128, false, false);
  constexpr uint32_t kIdescPV = make_idesc_bf16(128, D, false, true);
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kOCol = 256;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                                  // [2]
  uint8_t* sK = sQ + 2 * S::kTile;
  uint8_t* sV = sK + kStages * S::kTile;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + kStages * S::kTile);
  uint64_t* q_full = bars;                 // [2]
  uint64_t* q_empty = bars + 2;            // [2]
  uint64_t* s_full = bars + 4;             // [2]
  uint64_t* p_full = bars + 6;             // [2]
  uint64_t* o_full = bars + 8;             // [2] the item's last product of the tile has landed
  uint64_t* k_full = bars + 10;            // [kStages]
  uint64_t* k_empty = k_full + kStages;
  uint64_t* v_full = k_empty + kStages;
  uint64_t* v_empty = v_full + kStages;
  uint64_t* ml_full = v_empty + kStages;   // split: the second half's maxima and sums are in ml
  uint64_t* ml_empty = ml_full + 1;        //        they and its O have been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ml_empty + 1);
  float2* ml = reinterpret_cast<float2*>(reinterpret_cast<uint8_t*>(bars) + 256);     // [128] per query row

  // At 128 the products are issued by a whole warp (1 x 16384, 32 / 8 heads, causal 1797 -> 1753 us; 2 x 4096 254 -> 247); at 64,
  // where the softmax warps have no issue slots to spare, by one thread (4 x 5329, 16 heads: 675 us, by the warp 704).
  constexpr bool kWarpIssues = D == 128;
  const int warp = kWarpIssues ? __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0) : threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&p.tma_q);
    tma_prefetch_desc(&p.tma_k);
    tma_prefetch_desc(&p.tma_v);
    for (int t = 0; t < 2; ++t) {
      mbar_init(&q_full[t], 1);
      mbar_init(&q_empty[t], 1);
      mbar_init(&s_full[t], 1);
      mbar_init(&p_full[t], 4);
      mbar_init(&o_full[t], 1);
    }
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    mbar_init(ml_full, 4);
    mbar_init(ml_empty, 4);
    fence_barrier_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp >= 8) regs_give<kAttnOtherRegs>();
  if (warp == 8) {
    // ------------------------------------ producer ------------------------------------------
    if (elect_one()) {
      bool ok = true;
      uint32_t kv = 0, nq[2] = {0u, 0u};          // key tiles and Q tiles so far
      for (int64_t r = 0; r * gridDim.x < p.items && ok; ++r) {
        AttnItem it;
        if (!it.load(p, r)) continue;
        const int hkv = it.h / (p.hq / p.hk);
        const int n = it.tiles();
        for (int t = 0; t < 2 && ok; ++t) {
          if (it.count(t) == 0) continue;
          ok = mbar_wait(&q_empty[t], (nq[t] & 1u) ^ 1u, p.status);
          if (!ok) break;
          ++nq[t];
          mbar_expect_tx(&q_full[t], S::kTile);
#pragma unroll
          for (int c = 0; c < kDBoxes; ++c)
            tma_load_3d(sQ + t * S::kTile + c * kBoxBytes, &p.tma_q, &q_full[t], c * 64, it.h,
                        it.q_begin + it.first_query(t));
        }
        for (int j = 0; j < n && ok; ++j, ++kv) {
          const uint32_t s = kv % kStages, ph = (kv / kStages) & 1u;
          ok = mbar_wait(&k_empty[s], ph ^ 1u, p.status);
          if (!ok) break;
          mbar_expect_tx(&k_full[s], S::kTile);
#pragma unroll
          for (int c = 0; c < kDBoxes; ++c)
            tma_load_3d(sK + s * S::kTile + c * kBoxBytes, &p.tma_k, &k_full[s], c * 64, hkv,
                        it.k_begin + j * kAttnBlock);
          ok = mbar_wait(&v_empty[s], ph ^ 1u, p.status);
          if (!ok) break;
          mbar_expect_tx(&v_full[s], S::kTile);
#pragma unroll
          for (int c = 0; c < kDBoxes; ++c)
            tma_load_3d(sV + s * S::kTile + c * kBoxBytes, &p.tma_v, &v_full[s], c * 64, hkv,
                        it.k_begin + j * kAttnBlock);
        }
      }
    }
  } else if (warp == 9) {
    // ------------------------------------ MMA issuer ----------------------------------------
    const uint32_t lead = elect_one() ? 1u : 0u;
    auto commit = [&](uint64_t* bar) {
      if (kWarpIssues) tc_commit_if(lead, bar); else tc_commit(bar);
    };
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      return kWarpIssues ? mbar_wait_warp(bar, parity, p.status) : mbar_wait(bar, parity, p.status);
    };
    if (kWarpIssues || lead != 0u) {
      bool ok = true;
      uint32_t kv = 0, nq[2] = {0u, 0u}, np[2] = {0u, 0u};   // key tiles, Q tiles and P tiles so far
      for (int64_t r = 0; r * gridDim.x < p.items && ok; ++r) {
        AttnItem it;
        if (!it.load(p, r)) continue;
        // S_t of step j; the products of one thread execute in order, so it follows the P V that read the same columns
        auto issue_qk = [&](int t, int j) -> bool {
          const uint32_t at = kv + it.key_tile(t, j), s = at % kStages;
          if (!wait(&k_full[s], (at / kStages) & 1u)) return false;
          tc_fence_after_sync();
          const uint32_t aQ = smem_u32(sQ + t * S::kTile), aK = smem_u32(sK + s * S::kTile);
          const uint32_t tS = tmem_base + static_cast<uint32_t>(t * 128);
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t off = (kk / 4) * kBoxBytes + (kk % 4) * 32;
            const uint64_t dq = make_smem_desc(aQ + off, 16, 1024), dk = make_smem_desc(aK + off, 16, 1024);
            if (kWarpIssues) tc_mma_f16_ss_if(lead, tS, dq, dk, kIdescQK, kk != 0 ? 1u : 0u);
            else tc_mma_f16_ss(tS, dq, dk, kIdescQK, kk != 0 ? 1u : 0u);
          }
          commit(&s_full[t]);
          if (j + 1 == it.count(t)) commit(&q_empty[t]);
          // the tile is free once the last query tile that sees it has been multiplied
          if (it.last_reader(t, j)) commit(&k_empty[s]);
          return true;
        };
        for (int t = 0; t < 2 && ok; ++t) {
          if (it.count(t) == 0) continue;
          ok = wait(&q_full[t], nq[t] & 1u);
          if (!ok) break;
          ++nq[t];
          ok = issue_qk(t, 0);
        }
        for (int j = 0; j < it.steps() && ok; ++j) {
          for (int t = 0; t < 2 && ok; ++t) {
            if (j >= it.count(t)) continue;
            const uint32_t at = kv + it.key_tile(t, j), s = at % kStages;
            ok = wait(&p_full[t], np[t] & 1u);
            if (!ok) break;
            ++np[t];
            ok = wait(&v_full[s], (at / kStages) & 1u);
            if (!ok) break;
            tc_fence_after_sync();
            const uint32_t aV = smem_u32(sV + s * S::kTile);
            const uint32_t tP = tmem_base + static_cast<uint32_t>(t * 128);
            const uint32_t tO = tmem_base + kOCol + static_cast<uint32_t>(t * 128);
#pragma unroll
            for (int kk = 0; kk < kAttnBlock / 16; ++kk) {
              // 16 keys per step: 8 packed bf16x2 columns of P; 16 key rows (2048 B) of the V tile
              const uint64_t dv = make_smem_desc(aV + kk * 2048, kBoxBytes, 1024);
              if (kWarpIssues) tc_mma_f16_ts_if(lead, tO, tP + kk * 8, dv, kIdescPV, (j | kk) != 0 ? 1u : 0u);
              else tc_mma_f16_ts(tO, tP + kk * 8, dv, kIdescPV, (j | kk) != 0 ? 1u : 0u);
            }
            if (j + 1 == it.count(t)) commit(&o_full[t]);
            if (it.last_reader(t, j)) commit(&v_empty[s]);
            if (j + 1 < it.count(t)) ok = issue_qk(t, j + 1);
          }
        }
        kv += it.tiles();
      }
    }
  } else if (warp < 8) {
    // ------------------------------------ softmax / epilogue --------------------------------
    regs_take<kAttnSoftmaxRegs>();
    const int t = warp >> 2;                          // query tile of this warp
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;              // query row inside the tile
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t tS = tmem_base + lane_off + static_cast<uint32_t>(t * 128);
    const uint32_t tO = tmem_base + lane_off + kOCol + static_cast<uint32_t>(t * 128);
    bool ok = true;
    uint32_t ns = 0, no0 = 0, no1 = 0, nx = 0;        // score tiles, finished items of either half and split items so far
    for (int64_t r = 0; r * gridDim.x < p.items && ok; ++r) {
      AttnItem it;
      if (!it.load(p, r)) continue;
      const int n_kv = it.count(t);
      const int q_pos = it.first_query(t) + row;      // position inside the sequence
      const int key_limit = p.causal ? min(q_pos + it.shift, it.k_len - 1) : (it.k_len - 1);   // last visible key
      float m_used = -1.0e29f;                        // running max (log2 domain); above kMaskValue so masked scores give 0
      float l_sum = 0.f;
      for (int j = 0; j < n_kv && ok; ++j, ++ns) {
        ok = mbar_wait(&s_full[t], ns & 1u, p.status);
        ok = __all_sync(0xFFFFFFFFu, ok);
        if (!ok) break;
        tc_fence_after_sync();
        uint32_t sreg[128];
        {
          uint32_t(&c0)[32] = *reinterpret_cast<uint32_t(*)[32]>(&sreg[0]);
          uint32_t(&c1)[32] = *reinterpret_cast<uint32_t(*)[32]>(&sreg[32]);
          uint32_t(&c2)[32] = *reinterpret_cast<uint32_t(*)[32]>(&sreg[64]);
          uint32_t(&c3)[32] = *reinterpret_cast<uint32_t(*)[32]>(&sreg[96]);
          tmem_ld32(tS, c0);
          tmem_ld32(tS + 32, c1);
          tmem_ld32(tS + 64, c2);
          tmem_ld32(tS + 96, c3);
          tc_wait_ld();
        }
        // The row maximum is taken over the raw scores (the scale is positive); scaling and the subtraction of the
        // reference maximum are one fused multiply-add per pair of scores further down.
        const int last = key_limit - it.key_tile(t, j) * kAttnBlock;  // last visible column of this tile
        if (last < kAttnBlock - 1) {
#pragma unroll
          for (int i = 0; i < 128; ++i)
            if (i > last) sreg[i] = 0xFF800000u;      // -inf: 2^(-inf) = 0
        }
        float m4[4] = {kMaskValue, kMaskValue, kMaskValue, kMaskValue};
#pragma unroll
        for (int i = 0; i < 128; i += 8) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            m4[c] = max_nan(m4[c], max_nan(__uint_as_float(sreg[i + 2 * c]), __uint_as_float(sreg[i + 2 * c + 1])));
        }
        float mx = max_nan(max_nan(m4[0], m4[1]), max_nan(m4[2], m4[3]));
        mx = (mx <= 0.5f * kMaskValue) ? kMaskValue : mx * p.scale_log2;
        mx += mx - mx;                                // a NaN or an infinite score makes the whole row NaN
        // lazy rescale: keep the old reference max unless the new one is much larger
        float alpha = 1.f;
        bool rescale = false;
        if (!(mx <= m_used + kRescaleThreshold)) {
          alpha = exp2f(m_used - mx);
          m_used = mx;
          rescale = (j > 0);
        }
        if (__any_sync(0xFFFFFFFFu, rescale)) {
          // O holds sums relative to the old max; the products that wrote it precede the scores just read
#pragma unroll 1
          for (int c = 0; c < D / 32; ++c) {
            uint32_t ov[32];
            tmem_ld32(tO + c * 32, ov);
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
            tmem_st32(tO + c * 32, ov);
          }
        }
        // p = 2^(s * scale - m): one packed fp32 FMA per pair of scores, 2^x, and one conversion of the pair to the packed
        // bf16 operand.  (2^x on a bf16 pair is no faster than on two floats, and rounds its argument.)
        float2 rs2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
        const float2 nm2 = make_float2(-m_used, -m_used);
#pragma unroll
        for (int hlf = 0; hlf < 2; ++hlf) {
          uint32_t pk[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int at = hlf * 64 + 2 * i;
            const float2 x = __ffma2_rn(make_float2(__uint_as_float(sreg[at]), __uint_as_float(sreg[at + 1])), sc2, nm2);
            const float2 e = ex2_pair<kAttnFwdPoly, false>(at / 2, x);
            rs2[i & 1] = __fadd2_rn(rs2[i & 1], e);
            pk[i] = pack_bf16(e.x, e.y);
          }
          tmem_st32(tS + hlf * 32, pk);
        }
        tc_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[t]);       // one arrival per warp: 32 on one word would be served one by one
        const float2 rs = __fadd2_rn(rs2[0], rs2[1]);
        l_sum = l_sum * alpha + (rs.x + rs.y);
      }
      // ---- epilogue: O / l, LSE ----
      const uint32_t done0 = no0 & 1u, done1 = no1 & 1u, turn = nx & 1u;
      no0 += it.n[0] > 0 ? 1u : 0u;
      no1 += it.n[1] > 0 ? 1u : 0u;
      if (it.split) {
        ++nx;
        if (t == 1) {
          // hand this half's maxima and sums over; its O stays where it is until it has been read
          if (ok) {
            ml[row] = make_float2(m_used, l_sum);
            __syncwarp();
            if (lane == 0) mbar_arrive(ml_full);
            ok = mbar_wait(ml_empty, turn, p.status);
            ok = __all_sync(0xFFFFFFFFu, ok);
            tc_fence_after_sync();
          }
          continue;
        }
        if (ok) {
          // in this order: once the second half has handed over, its earlier items' products are known to have landed, so that
          // the phase that is waited for next is this item's
          ok = mbar_wait(ml_full, turn, p.status) && mbar_wait(&o_full[1], done1, p.status);
          ok = __all_sync(0xFFFFFFFFu, ok);
        }
      }
      if (ok && n_kv > 0) {
        ok = mbar_wait(&o_full[t], t == 0 ? done0 : done1, p.status);
        ok = __all_sync(0xFFFFFFFFu, ok);
      }
      if (ok) {
        tc_fence_after_sync();
        float f0 = 1.f, f1 = 0.f;                     // factors of the halves' sums
        if (it.split) {
          const float2 other = ml[row];
          const float m = max_nan(m_used, other.x);
          f0 = exp2f(m_used - m);
          f1 = exp2f(other.x - m);
          m_used = m;
          l_sum = l_sum * f0 + other.y * f1;
        }
        const bool valid = q_pos < it.q_len && (t == 0 || it.second);
        const float inv_l = (l_sum > 0.f) ? 1.f / l_sum : 0.f;
        f0 *= inv_l;
        f1 *= inv_l;
        __nv_bfloat16* orow = p.o + (static_cast<int64_t>(it.q_begin + q_pos) * p.o_stride) + static_cast<int64_t>(it.h) * D;
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {             // a loop, since short items run it once each: the code has to stay small
          uint32_t ov[32];
          if (n_kv > 0) {
            tmem_ld32(tO + c * 32, ov);
            tc_wait_ld();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) ov[i] = 0u;
          }
          if (it.split) {
            uint32_t o1[32];
            tmem_ld32(tO + 128 + c * 32, o1);
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i)
              ov[i] = __float_as_uint(__uint_as_float(ov[i]) * f0 + __uint_as_float(o1[i]) * f1);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * f0);
          }
          if (valid) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint4 v;
              v.x = pack_bf16(__uint_as_float(ov[8 * i + 0]), __uint_as_float(ov[8 * i + 1]));
              v.y = pack_bf16(__uint_as_float(ov[8 * i + 2]), __uint_as_float(ov[8 * i + 3]));
              v.z = pack_bf16(__uint_as_float(ov[8 * i + 4]), __uint_as_float(ov[8 * i + 5]));
              v.w = pack_bf16(__uint_as_float(ov[8 * i + 6]), __uint_as_float(ov[8 * i + 7]));
              *reinterpret_cast<uint4*>(orow + c * 32 + i * 8) = v;
            }
          }
        }
        tc_fence_before_sync();                       // O is read before the next item's first P is announced
        if (it.split) {
          __syncwarp();
          if (lane == 0) mbar_arrive(ml_empty);
        }
        if (valid && p.lse != nullptr) {
          // natural-log LSE of the scaled scores
          p.lse[static_cast<int64_t>(it.h) * p.total_q + it.q_begin + q_pos] =
              (l_sum > 0.f) ? (m_used + log2f(l_sum)) * 0.6931471805599453f : -INFINITY;
        }
      }
    }
  }

  tc_fence_before_sync();
  block_settle(p.status);
  if (warp == 9) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace yv
