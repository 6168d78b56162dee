// dK / dV kernel of the flash attention backward (see attention_bwd.cuh for the scheme).
// TMEM columns: [0,128) S^T, then P^T over it (bf16: the 32 queries of a warp's columns in the first 16 of them); [128,256)
// dP^T, then dS^T over it likewise; [256,256+D) dV, [384,384+D) dK.  While the softmax threads turn S^T into P^T the tensor
// core computes dK of the block before and dP^T; while they turn dP^T into dS^T it computes dV and the next block's S^T.
#pragma once

namespace yv {

template <int D>
__global__ void __launch_bounds__(kAttnBwdThreads, 1) attn_bwd_dkv_kernel(const __grid_constant__ AttnBwdParams p) {
  using S = AttnBwdSmem<D>;
  constexpr int kStages = S::kStages;
  constexpr int kDBoxes = D / 64;
  constexpr uint32_t kBoxBytes = 128 * 128;
  constexpr uint32_t kIdescNT = make_idesc_bf16(128, 128, false, false);    // 128 keys x 128 queries
  constexpr uint32_t kIdescAcc = make_idesc_bf16(128, D, false, true);
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kColDP = 128, kColDV = 256, kColDK = 384;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + S::kTile;
  uint8_t* sQ = sV + S::kTile;
  uint8_t* sDO = sQ + kStages * S::kTile;
  float* s_lse = reinterpret_cast<float*>(sDO + kStages * S::kTile);   // [2][128]
  float* s_delta = s_lse + 2 * 128;                                     // [2][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_delta + 2 * 128);
  uint64_t* kv_full = bars;             // [1]
  uint64_t* q_full = bars + 1;          // [2]
  uint64_t* do_full = bars + 3;         // [2]
  uint64_t* q_empty = bars + 5;         // [2]
  uint64_t* do_empty = bars + 7;        // [2]
  uint64_t* s_full = bars + 9;          // [1]
  uint64_t* dp_full = bars + 10;        // [1]
  uint64_t* p_full = bars + 11;         // [1] one arrival per softmax warp: P^T written
  uint64_t* ds_full = bars + 12;        // [1] likewise: dS^T written
  uint64_t* acc_done = bars + 13;       // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.z, hkv = blockIdx.y;
  const int G = p.hq / p.hk;
  const int q_begin = p.cu_q[b], q_len = p.cu_q[b + 1] - q_begin;
  const int k_begin = p.cu_k[b], k_len = p.cu_k[b + 1] - k_begin;
  const int n_kblk = (k_len + 127) / 128;
  const int k_blk = static_cast<int>(blockIdx.x);
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

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 1); mbar_init(&do_full[s], 1);
      mbar_init(&q_empty[s], 1); mbar_init(&do_empty[s], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_full, kAttnBwdSoftmaxWarps);
    mbar_init(ds_full, kAttnBwdSoftmaxWarps);
    mbar_init(acc_done, 1);
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, kTmemCols); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one() && n_it > 0) {
      mbar_expect_tx(kv_full, 2 * S::kTile);
#pragma unroll
      for (int c = 0; c < kDBoxes; ++c) {
        tma_load_3d(sK + c * kBoxBytes, &p.tma_k, kv_full, c * 64, hkv, k_begin + k0);
        tma_load_3d(sV + c * kBoxBytes, &p.tma_v, kv_full, c * 64, hkv, k_begin + k0);
      }
      bool ok = true;
      for (int it = 0; it < n_it && ok; ++it) {
        const int g = it / n_i, i = i_start + it % n_i;
        const int h = hkv * G + g;
        const int s = it % kStages;
        const uint32_t ph = (it / kStages) & 1u;
        ok = mbar_wait(&q_empty[s], ph ^ 1u, p.status);
        if (!ok) break;
        mbar_expect_tx(&q_full[s], S::kTile);
#pragma unroll
        for (int c = 0; c < kDBoxes; ++c)
          tma_load_3d(sQ + s * S::kTile + c * kBoxBytes, &p.tma_q, &q_full[s], c * 64, h, q_begin + i * 128);
        ok = mbar_wait(&do_empty[s], ph ^ 1u, p.status);
        if (!ok) break;
        mbar_expect_tx(&do_full[s], S::kTile);
#pragma unroll
        for (int c = 0; c < kDBoxes; ++c)
          tma_load_3d(sDO + s * S::kTile + c * kBoxBytes, &p.tma_do, &do_full[s], c * 64, h, q_begin + i * 128);
      }
    }
  } else if (warp == 1) {
    if (elect_one() && n_it > 0) {
      bool ok = mbar_wait(kv_full, 0, p.status);
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV);
      auto issue_s = [&](int it) -> bool {
        const int s = it % kStages;
        if (!mbar_wait(&q_full[s], (it / kStages) & 1u, p.status)) return false;
        tc_fence_after_sync();
        const uint32_t aQ = smem_u32(sQ + s * S::kTile);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk / 4) * kBoxBytes + (kk % 4) * 32;
          tc_mma_f16_ss(tmem_base, make_smem_desc(aK + off, 16, 1024), make_smem_desc(aQ + off, 16, 1024), kIdescNT,
                        kk != 0 ? 1u : 0u);
        }
        tc_commit(s_full);
        return true;
      };
      auto issue_dp = [&](int it) -> bool {
        const int s = it % kStages;
        if (!mbar_wait(&do_full[s], (it / kStages) & 1u, p.status)) return false;
        tc_fence_after_sync();
        const uint32_t aDO = smem_u32(sDO + s * S::kTile);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk / 4) * kBoxBytes + (kk % 4) * 32;
          tc_mma_f16_ss(tmem_base + kColDP, make_smem_desc(aV + off, 16, 1024), make_smem_desc(aDO + off, 16, 1024),
                        kIdescNT, kk != 0 ? 1u : 0u);
        }
        tc_commit(dp_full);
        return true;
      };
      if (ok) ok = issue_s(0);
      if (ok) ok = issue_dp(0);
      for (int it = 0; it < n_it && ok; ++it) {
        const int s = it % kStages;
        const uint32_t aQ = smem_u32(sQ + s * S::kTile), aDO = smem_u32(sDO + s * S::kTile);
        ok = mbar_wait(p_full, it & 1u, p.status);
        if (!ok) break;
        tc_fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {                 // 128 queries = 8 K-steps of 16
          tc_mma_f16_ts(tmem_base + kColDV, tmem_base + (kk >> 1) * 32 + (kk & 1) * 8,
                        make_smem_desc(aDO + kk * 2048, kBoxBytes, 1024), kIdescAcc, (it | kk) != 0 ? 1u : 0u);
        }
        tc_commit(&do_empty[s]);                         // dP^T of this block precedes it
        if (it + 1 < n_it) {
          ok = issue_s(it + 1);                          // over P^T, which dV has read
          if (!ok) break;
        }
        ok = mbar_wait(ds_full, it & 1u, p.status);
        if (!ok) break;
        tc_fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          tc_mma_f16_ts(tmem_base + kColDK, tmem_base + kColDP + (kk >> 1) * 32 + (kk & 1) * 8,
                        make_smem_desc(aQ + kk * 2048, kBoxBytes, 1024), kIdescAcc, (it | kk) != 0 ? 1u : 0u);
        }
        tc_commit(&q_empty[s]);
        if (it + 1 < n_it) ok = issue_dp(it + 1);
        else tc_commit(acc_done);
      }
    }
  } else {
    // Sixteen softmax warps: four warps share each TMEM lane quarter (a warp may only touch lanes 32 (warp % 4) ..) and
    // split the 128 query columns of a block between them, 32 each.
    const int quarter = warp & 3;
    const int part = (warp - 2) >> 2;                    // which 32 of the 128 columns this warp converts
    const int row = quarter * 32 + lane;                 // key row of the tile
    const int tix = threadIdx.x - 64;                    // 0..511 among the softmax threads
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    const int key = k0 + row;
    const bool key_valid = key < k_len;
    const uint32_t tST = tmem_base + lane_off, tDPT = tST + kColDP;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    // Statistics of a block's queries, one value per thread: 0..127 the log-sum-exp, 128..255 delta; stored negated, so that
    // they fold into packed FMAs and adds (-inf makes the probability of rows past the end 0).
    auto stat = [&](int it) -> float {
      const int g = it / n_i, i = i_start + it % n_i;
      const int qpos = i * 128 + (tix & 127);
      const bool v = it < n_it && qpos < q_len;
      const int64_t idx = static_cast<int64_t>(hkv * G + g) * p.total_q + q_begin + qpos;
      return tix < 128 ? (v ? -p.lse[idx] * kLog2e : -INFINITY) : (v ? -p.delta[idx] : 0.f);
    };
    bool ok = true;
    if (n_it > 0) {
      if (tix < 256) (tix < 128 ? s_lse : s_delta)[tix & 127] = stat(0);
      asm volatile("bar.sync 1, 512;" ::: "memory");
    }
    for (int it = 0; it < n_it && ok; ++it) {
      const int qb = (i_start + it % n_i) * 128;
      const float* lse_b = s_lse + (it & 1) * 128 + part * 32;
      const float* del_b = s_delta + (it & 1) * 128 + part * 32;
      const float next = tix < 256 ? stat(it + 1) : 0.f; // in flight during the block
      ok = mbar_wait(s_full, it & 1u, p.status);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (ok) {
        tc_fence_after_sync();
        // a query column c is visible to this key iff key <= (qb + c) + shift
        const int first_vis = !key_valid ? 128 : p.causal ? (key - causal_shift - qb - part * 32) : 0;
        // every (key, query) pair of this block is visible: no per-element selects (uniform over the CTA)
        const bool full_vis = (!p.causal || qb >= k0 + 127 - causal_shift) && (k0 + 127 < k_len);
        uint32_t sv[32], pp[16];
        tmem_ld32(tST + part * 32, sv);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float4 nl4 = *reinterpret_cast<const float4*>(lse_b + (i & ~1) * 2);
          const float2 nl = (i & 1) ? make_float2(nl4.z, nl4.w) : make_float2(nl4.x, nl4.y);
          float2 x = __ffma2_rn(make_float2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), sc2, nl);
          if (!full_vis) {
            if (2 * i < first_vis) x.x = -INFINITY;
            if (2 * i + 1 < first_vis) x.y = -INFINITY;
          }
          const float2 e = ex2_pair<kAttnBwdPoly, true>(i, x);
          sv[2 * i] = __float_as_uint(e.x);
          sv[2 * i + 1] = __float_as_uint(e.y);
          pp[i] = pack_bf16(e.x, e.y);
        }
        tmem_st16(tST + part * 32, pp);
        tc_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
        ok = mbar_wait(dp_full, it & 1u, p.status);
        ok = __all_sync(0xFFFFFFFFu, ok);
        if (ok) {
          tc_fence_after_sync();
          uint32_t dv[32], ds[16];
          tmem_ld32(tDPT + part * 32, dv);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float4 nd4 = *reinterpret_cast<const float4*>(del_b + (i & ~1) * 2);
            const float2 nd = (i & 1) ? make_float2(nd4.z, nd4.w) : make_float2(nd4.x, nd4.y);
            const float2 dd = __fadd2_rn(make_float2(__uint_as_float(dv[2 * i]), __uint_as_float(dv[2 * i + 1])), nd);
            const float2 r = __fmul2_rn(make_float2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), dd);
            ds[i] = pack_bf16(r.x, r.y);
          }
          tmem_st16(tDPT + part * 32, ds);
          tc_wait_st();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(ds_full);
        }
      }
      // the other buffer was last read in the block before
      if (tix < 256) (tix < 128 ? s_lse : s_delta)[((it + 1) & 1) * 128 + (tix & 127)] = next;
      uint32_t all_ok;
      asm volatile(
          "{\n"
          ".reg .pred pin, pout;\n"
          "setp.ne.u32 pin, %1, 0;\n"
          "bar.red.and.pred pout, 1, 512, pin;\n"
          "selp.u32 %0, 1, 0, pout;\n"
          "}\n"
          : "=r"(all_ok)
          : "r"(static_cast<uint32_t>(ok))
          : "memory");
      ok = all_ok != 0u;
    }
    if (ok && n_it > 0) {
      ok = mbar_wait(acc_done, 0u, p.status);
      ok = __all_sync(0xFFFFFFFFu, ok);
    }
    if (ok) {
      tc_fence_after_sync();
      const int64_t tok = k_begin + key;
      __nv_bfloat16* dkrow = p.dk + tok * p.dk_stride + static_cast<int64_t>(hkv) * D;
      __nv_bfloat16* dvrow = p.dv + tok * p.dv_stride + static_cast<int64_t>(hkv) * D;
      {
        const int which = part >> 1;                       // two warps of the quarter write dV, two dK
        const uint32_t col = which == 0 ? kColDV : kColDK;
        const float sc = which == 0 ? 1.f : p.scale;
        __nv_bfloat16* orow = which == 0 ? dvrow : dkrow;
#pragma unroll
        for (int c = (part & 1) * (D / 64); c < ((part & 1) + 1) * (D / 64); ++c) {
          uint32_t ov[32];
          if (n_it > 0) {
            tmem_ld32(tmem_base + lane_off + col + c * 32, ov);
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
              *reinterpret_cast<uint4*>(orow + c * 32 + i2 * 8) = v;
            }
          }
        }
      }
    }
  }

  tc_fence_before_sync();
  block_settle(p.status);
  if (warp == 1) { tc_fence_after_sync(); tmem_dealloc(tmem_base, kTmemCols); }
}

// delta[h, t] = sum_d dO[t,h,d] * O[t,h,d]: D / 8 lanes per (token, head), 16 bytes of either operand each, so that a warp
// reads 512 contiguous bytes twice.  Bound by memory:
// 16384 tokens of 32 heads of 128 in 48 us (5.5 TB/s) instead of 107 with one warp and 4-byte loads per head.  O that is not aligned to 16 bytes is read in pairs.
template <int D, bool VEC>
__device__ __forceinline__ float attn_delta_row(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                                                int64_t t, int h, int c, bool valid, int64_t o_stride, int64_t do_stride) {
  constexpr int kLanes = D / 8;
  float s = 0.f;
  if (valid) {
    const __nv_bfloat16* orow = o + t * o_stride + static_cast<int64_t>(h) * D + c * 8;
    uint4 a;
    if (VEC) {
      a = *reinterpret_cast<const uint4*>(orow);
    } else {
      const uint32_t* pairs = reinterpret_cast<const uint32_t*>(orow);
      a = make_uint4(pairs[0], pairs[1], pairs[2], pairs[3]);
    }
    const uint4 b = *reinterpret_cast<const uint4*>(dout + t * do_stride + static_cast<int64_t>(h) * D + c * 8);
    const uint32_t av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s += __uint_as_float(av[i] << 16) * __uint_as_float(bv[i] << 16);
      s += __uint_as_float(av[i] & 0xFFFF0000u) * __uint_as_float(bv[i] & 0xFFFF0000u);
    }
  }
#pragma unroll
  for (int off = kLanes / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, off);
  return s;
}

template <int D, bool VEC>
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ o,
                                                         const __nv_bfloat16* __restrict__ dout, float* __restrict__ delta,
                                                         int64_t total_q, int hq, int64_t o_stride, int64_t do_stride) {
  constexpr int kLanes = D / 8;
  const int64_t w = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) / kLanes;
  const int c = threadIdx.x & (kLanes - 1);
  const int64_t t = w / hq;
  const int h = static_cast<int>(w - t * hq);
  const float s = attn_delta_row<D, VEC>(o, dout, t, h, c, t < total_q, o_stride, do_stride);
  if (c == 0 && t < total_q) delta[static_cast<int64_t>(h) * total_q + t] = s;
}

}  // namespace yv
