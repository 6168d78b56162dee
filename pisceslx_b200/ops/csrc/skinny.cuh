// Products of a few token rows with large weights (decoding, short prompts): out[t, n] = sum_k x[t, k] * w[n, k].
//
// Every weight is used by at most 128 tokens, so the time is that of streaming the weights from HBM.  The operands are
// swapped against the general kernel: 128 weight rows fill the M side of tcgen05.mma and the tokens, padded to 16, the N
// side, so that shared memory and the L2 carry weights and not the rows of an empty 128-row token tile, and nothing but
// live outputs is written.  Two CTAs per SM, about 100 KB of loads in flight each.
//
//   dense    One CTA per (128 weight rows, slice of K); the slices of a tile form a cluster and add their fp32 sums, in
//            the order of the slices, through distributed shared memory: no workspace, no second kernel.  The number of
//            slices depends on N and K alone, so a row's result does not depend on the rows it is batched with.
//            With SWIGLU as below; a factor per segment of the outputs (a shared expert's weight) may go with it.
//   grouped  Persistent CTAs over (tile of <= 128 tokens of one expert, 128 weight rows).  With SWIGLU the 128 rows are 64
//            gate rows and their 64 up rows, and silu(gate) * up leaves the kernel; the products stay in fp32 until then.
//
// Bound by HBM and, for the smaller matrices, by some 4 us of start and end.  Measured in a graph, weights not in L2, one token
// (before: the split of K by the general kernel and a second kernel that added the parts): 11264 x 4096 16.8 us, 32000 x 4096
// 44.4 (5.9 TB/s; before 57), 6144 x 4096 12.4, 4096 x 4096 9.2, 4096 x 5632 11.1, 64 x 4096 4.7 (before 8); 128 tokens
// 23.2 (28), 49.7 (50), 18.4 (18), 14.7 (16), 16.6 (17), 7.0 (8); 64 experts of 4096 x 1408 with 64 tokens, top-6, both
// products and the activation 350 us (6.3 TB/s; before 435).
#pragma once
#include "chain.cuh"
#include "sm100.cuh"

namespace yv {

struct SkinnyParams {
  CUtensorMap tma_w;            // [weight rows, K], box 64 x 128 (SWIGLU: 64 x 64)
  CUtensorMap tma_x;            // [token rows, K], box 64 x 16
  int M, N, K;                  // dense: tokens; outputs per token (SWIGLU: F); depth
  int out_fp32;                 // dense only
  int tiles_w;                  // tiles of weight rows (of one expert)
  int w_rows;                   // grouped: weight rows per expert
  int seg;                      // dense SWIGLU: outputs per segment (its gate rows are followed by its up rows)
  const void* scale;            // dense SWIGLU, optional: one factor per segment (bf16, or fp32 with scale_fp32)
  int scale_fp32;
  int scale_softmax;            // the factors are the softmax of `scale` over the segments
  void* out;
  long long ldo;                // elements between output rows
  const __nv_bfloat16* bias;    // dense, optional
  const int* tile_expert;       // grouped: the dispatch plan
  const int* num_m_tiles;
  const int* seg_offsets;
  const int* counts;
  uint32_t* status;
};

constexpr int kSkThreads = 192;              // TMA producer, MMA issuer, four epilogue warps
constexpr int kSkRows = 128;                 // weight rows per tile
constexpr int kSkWBytes = kSkRows * 128;     // one stage of weights: 128 rows x 64 bf16
constexpr int kSkXBox = 16 * 128;            // 16 tokens x 64 bf16
constexpr int kSkAhead = 16;                  // 64-wide steps of K that a dense CTA fetches ahead of the kernel before it
constexpr int kSkEpiBytes = 16 * kSkRows * 4;

// NT: token slots (16, 32, 64 or 128).  A tile with more live tokens than slots is worked off in passes.
template <int NT>
struct SkinnySmem {
  static constexpr int kStageBytes = kSkWBytes + (NT / 16) * kSkXBox;
  static constexpr int kStages = NT == 128 ? 3 : (NT == 64 ? 4 : 5);
  static constexpr int kRing = kStages * kStageBytes;
  static constexpr int kTotal = kRing + kSkEpiBytes + 256;       // two CTAs per SM: at most 113 KB each
  static_assert(kTotal <= 115712 && NT * kSkRows * 4 <= kRing, "two CTAs per SM; the dense sums reuse the ring");
};

struct SkinnyTile {
  int w_row, w_row2;            // first weight row (SWIGLU: of the gate rows and of the up rows)
  int x_row;                    // first token row
  int cnt;                      // live tokens
  int col;                      // first output column
};

// MODE: 0 dense, 1 grouped, 2 grouped with SWIGLU, 3 dense with SWIGLU
__host__ __device__ constexpr bool skinny_dense(int mode) { return mode == 0 || mode == 3; }
__host__ __device__ constexpr bool skinny_swiglu(int mode) { return mode >= 2; }

// Factor of a segment of the outputs.  The softmax of the few values is taken here, from the parameter itself, so that nothing
// derived from it has to be kept between launches.
__device__ __forceinline__ float skinny_factor(const SkinnyParams& p, int segment) {
  if (p.scale == nullptr) return 1.f;
  auto at = [&](int i) {
    return p.scale_fp32 ? static_cast<const float*>(p.scale)[i]
                        : __bfloat162float(static_cast<const __nv_bfloat16*>(p.scale)[i]);
  };
  const float mine = at(segment);
  if (!p.scale_softmax) return mine;
  const int n = p.N / p.seg;
  float top = mine, sum = 0.f;
  for (int i = 0; i < n; ++i) top = fmaxf(top, at(i));
  for (int i = 0; i < n; ++i) sum += expf(at(i) - top);
  return expf(mine - top) / sum;
}

__device__ __forceinline__ float swiglu1(float gate, float up) { return gate / (1.f + __expf(-gate)) * up; }

template <int MODE>
__device__ __forceinline__ bool skinny_tile(const SkinnyParams& p, int unit, int units, SkinnyTile& t) {
  if (unit >= units) return false;
  if (skinny_dense(MODE)) {
    t.col = unit * (MODE == 3 ? 64 : kSkRows);
    t.w_row = MODE == 3 ? t.col + t.col / p.seg * p.seg : t.col;
    t.w_row2 = t.w_row + p.seg;
    t.x_row = 0;
    t.cnt = p.M;
    return true;
  }
  const int j = unit / p.tiles_w, i = unit - j * p.tiles_w;
  const int e = p.tile_expert[j];
  t.x_row = j * 128;
  t.cnt = max(1, min(128, p.seg_offsets[e] + p.counts[e] - t.x_row));
  if (MODE == 2) {
    t.col = i * 64;
    t.w_row = e * p.w_rows + t.col;
    t.w_row2 = t.w_row + p.N;
  } else {
    t.col = i * kSkRows;
    t.w_row = e * p.w_rows + t.col;
    t.w_row2 = 0;
  }
  return true;
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr, uint32_t rank) {
  float4 v;
  asm volatile(
      "{\n"
      ".reg .b32 ra;\n"
      "mapa.shared::cluster.u32 ra, %4, %5;\n"
      "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [ra];\n"
      "}\n"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "r"(addr), "r"(rank)
      : "memory");
  return v;
}

__device__ __forceinline__ uint32_t ld_cluster_u32(uint32_t addr, uint32_t rank) {
  uint32_t v;
  asm volatile(
      "{\n"
      ".reg .b32 ra;\n"
      "mapa.shared::cluster.u32 ra, %1, %2;\n"
      "ld.shared::cluster.u32 %0, [ra];\n"
      "}\n"
      : "=r"(v)
      : "r"(addr), "r"(rank)
      : "memory");
  return v;
}

// Four consecutive outputs of one token, as one vector if `whole`; columns at or past `n` are dropped.
__device__ __forceinline__ void skinny_store4(void* out, int fp32, long long at, int col, int n, bool whole, float4 v) {
  float f[4] = {v.x, v.y, v.z, v.w};
  if (fp32) {
    float* o = static_cast<float*>(out) + at;
    if (whole) {
      *reinterpret_cast<float4*>(o) = v;
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (col + i < n) o[i] = f[i];
    }
  } else {
    __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out) + at;
    if (whole) {
      *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]));
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (col + i < n) o[i] = __float2bfloat16(f[i]);
    }
  }
}

// Outputs of a dense tile: the sums of the SLICES CTAs of the cluster in their order.  A thread owns four neighbouring columns
// and takes every kRows-th token, eight loads ahead of their use: the few warps have nothing else to hide a load or an address
// behind (one token at a time with its own addresses, 128 tokens of one slice took 6500 cycles).
// A slice whose sums did not arrive gives zeros, so that no stale memory is read further on; what other kernels reported is no
// reason to leave the product out.
template <int MODE, int SLICES>
__device__ __forceinline__ void skinny_sum(const SkinnyParams& p, uint8_t* smem, int slice, int col0, float f, uint32_t failed) {
  constexpr int kQuads = MODE == 3 ? 16 : 32;              // groups of four outputs per token
  constexpr int kLoads = SLICES * (MODE == 3 ? 2 : 1);
  constexpr int kAtOnce = kLoads >= 8 ? 1 : 8 / kLoads;
  constexpr int kRows = SLICES * kSkThreads / kQuads;      // tokens that the cluster's threads cover at a time
  const int c = (static_cast<int>(threadIdx.x) % kQuads) * 4, col = col0 + c;
  if (col >= p.N) return;
  const bool whole = col + 4 <= p.N && (p.ldo & 3) == 0;
  uint32_t bad = 0u;
#pragma unroll
  for (int s = 0; s < SLICES; ++s) bad |= ld_cluster_u32(failed, static_cast<uint32_t>(s));
  float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
  if (p.bias != nullptr) {
    bias.x = __bfloat162float(p.bias[col]);
    if (col + 1 < p.N) bias.y = __bfloat162float(p.bias[col + 1]);
    if (col + 2 < p.N) bias.z = __bfloat162float(p.bias[col + 2]);
    if (col + 3 < p.N) bias.w = __bfloat162float(p.bias[col + 3]);
  }
  const int tok0 = slice * (kSkThreads / kQuads) + static_cast<int>(threadIdx.x) / kQuads;
  const float* mine = reinterpret_cast<const float*>(smem) + tok0 * kSkRows + c;
  const uint32_t mine_addr = smem_u32(smem) + static_cast<uint32_t>(tok0 * kSkRows + c) * 4u;
  auto load = [&](int row, int s) -> float4 {              // `row`: tokens past tok0, or half a row for the up part
    if (SLICES == 1) return *reinterpret_cast<const float4*>(mine + row);
    return ld_cluster_f4(mine_addr + static_cast<uint32_t>(row) * 4u, static_cast<uint32_t>(s));
  };
  const long long step = static_cast<long long>(kRows) * p.ldo;
  long long at = static_cast<long long>(tok0) * p.ldo + col;
  int row = 0;
  for (int tok = tok0; tok < p.M; tok += kAtOnce * kRows) {
    float4 v[kAtOnce][SLICES], up[kAtOnce][MODE == 3 ? SLICES : 1];
#pragma unroll
    for (int j = 0; j < kAtOnce; ++j) {
      if (tok + j * kRows < p.M) {
#pragma unroll
        for (int s = 0; s < SLICES; ++s) {
          v[j][s] = load(row + j * kRows * kSkRows, s);
          if (MODE == 3) up[j][s] = load(row + j * kRows * kSkRows + 64, s);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < kAtOnce; ++j) {
      if (tok + j * kRows < p.M) {
        float4 o = v[j][0];
#pragma unroll
        for (int s = 1; s < SLICES; ++s) { o.x += v[j][s].x; o.y += v[j][s].y; o.z += v[j][s].z; o.w += v[j][s].w; }
        if (MODE == 3) {
          float4 u = up[j][0];
#pragma unroll
          for (int s = 1; s < SLICES; ++s) { u.x += up[j][s].x; u.y += up[j][s].y; u.z += up[j][s].z; u.w += up[j][s].w; }
          o = make_float4(f * swiglu1(o.x, u.x), f * swiglu1(o.y, u.y), f * swiglu1(o.z, u.z), f * swiglu1(o.w, u.w));
        } else {
          o.x += bias.x; o.y += bias.y; o.z += bias.z; o.w += bias.w;
        }
        if (bad != 0u) o = make_float4(0.f, 0.f, 0.f, 0.f);
        skinny_store4(p.out, p.out_fp32, at, col, p.N, whole, o);
        at += step;
      }
    }
    row += kAtOnce * kRows * kSkRows;
  }
}

template <int NT, int MODE>
__global__ void __launch_bounds__(kSkThreads, 2) skinny_kernel(const __grid_constant__ SkinnyParams p) {
  using S = SkinnySmem<NT>;
  constexpr int kStages = S::kStages;
  constexpr int kAccBufs = skinny_dense(MODE) ? 1 : 2;
  constexpr uint32_t kTmemCols = kAccBufs * NT < 32 ? 32 : kAccBufs * NT;

  extern __shared__ __align__(1024) uint8_t skinny_smem[];
  uint8_t* smem = skinny_smem;
  float* epi = reinterpret_cast<float*>(smem + S::kRing);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S::kRing + kSkEpiBytes);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* acc_full = empty_bar + kStages;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  uint32_t* failed = tmem_slot + 1;                // dense: a wait of this CTA ran out

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the swizzled tiles need shared memory that starts on 1024 bytes
  if ((smem_u32(smem) & 1023u) != 0u) {
    chain_wait();
    if (threadIdx.x == 0 && p.status != nullptr) atomicOr(p.status, kStatusBadArgument);
    return;
  }
  const int kc = (p.K + 63) / 64;
  int slices = 1, slice = 0, units = 0, first, step;
  if (skinny_dense(MODE)) {
    uint32_t n;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
    slices = static_cast<int>(n);
    slice = static_cast<int>(cluster_rank());
    first = static_cast<int>(blockIdx.x) / slices;
    units = p.tiles_w;
    step = units;                                  // one tile per cluster
  } else {
    first = blockIdx.x;
    step = gridDim.x;
  }
  const int k0 = kc * slice / slices, k1 = kc * (slice + 1) / slices;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&p.tma_w);
    tma_prefetch_desc(&p.tma_x);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], 1);
    }
    *failed = 0u;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  chain_next();
  if (skinny_dense(MODE) && warp == 0 && elect_one()) {
    // the weights do not depend on the kernel before this one: start them on their way to the L2 (not into shared memory, where
    // weights that the kernel before wrote would be stale)
    SkinnyTile t;
    if (skinny_tile<MODE>(p, first, units, t))
      for (int k = k0; k < k1 && k < k0 + kSkAhead; ++k) {
        tma_prefetch_l2_2d(&p.tma_w, k * 64, t.w_row);
        if (skinny_swiglu(MODE)) tma_prefetch_l2_2d(&p.tma_w, k * 64, t.w_row2);
      }
  }
  chain_wait();
  if (!skinny_dense(MODE)) units = *p.num_m_tiles * p.tiles_w;

  __syncwarp();
  if (warp == 0) {
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      SkinnyTile t;
      for (int u = first; ok && skinny_tile<MODE>(p, u, units, t); u += step) {
        for (int at = 0; ok && at < t.cnt; at += NT) {
          const int boxes = (min(NT, t.cnt - at) + 15) / 16;
          const uint32_t bytes = kSkWBytes + static_cast<uint32_t>(boxes) * kSkXBox;
          for (int k = k0; k < k1; ++k, ++it) {
            const int s = it % kStages;
            ok = mbar_wait(&empty_bar[s], ((it / kStages) & 1u) ^ 1u, p.status);
            if (!ok) break;
            uint8_t* sw = smem + s * S::kStageBytes;
            uint8_t* sx = sw + kSkWBytes;
            mbar_expect_tx(&full_bar[s], bytes);
            tma_load_2d(sw, &p.tma_w, &full_bar[s], k * 64, t.w_row);
            if (skinny_swiglu(MODE)) tma_load_2d(sw + kSkWBytes / 2, &p.tma_w, &full_bar[s], k * 64, t.w_row2);
            for (int b = 0; b < boxes; ++b)
              tma_load_2d(sx + b * kSkXBox, &p.tma_x, &full_bar[s], k * 64, t.x_row + at + 16 * b);
          }
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      uint32_t it = 0, tile_it = 0;
      bool ok = true;
      SkinnyTile t;
      for (int u = first; ok && skinny_tile<MODE>(p, u, units, t); u += step) {
        for (int at = 0; ok && at < t.cnt; at += NT, ++tile_it) {
          const int acc = tile_it % kAccBufs;
          ok = mbar_wait(&acc_empty[acc], ((tile_it / kAccBufs) & 1u) ^ 1u, p.status);
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(acc * NT);
          const uint32_t idesc = make_idesc_bf16(kSkRows, ((min(NT, t.cnt - at) + 15) / 16) * 16, false, false);
          for (int k = k0; k < k1; ++k, ++it) {
            const int s = it % kStages;
            ok = mbar_wait(&full_bar[s], (it / kStages) & 1u, p.status);
            if (!ok) break;
            tc_fence_after_sync();
            const uint32_t sw = smem_u32(smem + s * S::kStageBytes), sx = sw + kSkWBytes;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              tc_mma_f16_ss(tmem_d, make_smem_desc(sw + kk * 32, 16, 1024), make_smem_desc(sx + kk * 32, 16, 1024), idesc,
                            (k > k0 || kk > 0) ? 1u : 0u);
            tc_commit(&empty_bar[s]);
          }
          if (ok) tc_commit(&acc_full[acc]);
        }
      }
    }
  } else {
    const int quarter = warp & 3;                  // TMEM lane quarter of this warp
    const int row = quarter * 32 + lane;           // weight row of the tile
    const int tid = static_cast<int>(threadIdx.x) - 64;
    uint32_t tile_it = 0;
    SkinnyTile t;
    bool live = true;
    for (int u = first; live && skinny_tile<MODE>(p, u, units, t); u += step) {
      for (int at = 0; at < t.cnt; at += NT, ++tile_it) {
        const int acc = tile_it % kAccBufs, cnt = min(NT, t.cnt - at);
        uint32_t ok = mbar_wait(&acc_full[acc], (tile_it / kAccBufs) & 1u, p.status) ? 1u : 0u;
        asm volatile(
            "{\n"
            ".reg .pred pin, pout;\n"
            "setp.ne.u32 pin, %0, 0;\n"
            "bar.red.and.pred pout, 1, 128, pin;\n"
            "selp.u32 %0, 1, 0, pout;\n"
            "}\n"
            : "+r"(ok)::"memory");
        live = ok != 0u;
        if (!live) {
          if (tid == 0) *failed = 1u;
          break;
        }
        tc_fence_after_sync();
        const uint32_t taddr = tmem_base + static_cast<uint32_t>(acc * NT) + (static_cast<uint32_t>(quarter * 32) << 16);
        const int boxes = (cnt + 15) / 16;
        if (skinny_dense(MODE)) {
          // [token][weight row], where all slices' threads find it
          float* st = reinterpret_cast<float*>(smem) + row;
          for (int b = 0; b < boxes; b += 2) {
            uint32_t v[2][16];
            tmem_ld16(taddr + 16 * b, v[0]);
            if (b + 1 < boxes) tmem_ld16(taddr + 16 * b + 16, v[1]);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 2; ++j)
              if (b + j < boxes) {
#pragma unroll
                for (int i = 0; i < 16; ++i) st[(16 * (b + j) + i) * kSkRows] = __uint_as_float(v[j][i]);
              }
          }
        }
        for (int b = 0; !skinny_dense(MODE) && b < boxes; ++b) {
          uint32_t v[16];
          tmem_ld16(taddr + 16 * b, v);
          tc_wait_ld();
          // staged as [token][weight row], so that consecutive threads write consecutive outputs of one token
          float* st = epi;
          if (b > 0) asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
          for (int i = 0; i < 16; ++i) st[i * kSkRows + row] = __uint_as_float(v[i]);
          asm volatile("bar.sync 1, 128;" ::: "memory");
          constexpr int kQuads = MODE == 2 ? 16 : 32;          // groups of four outputs per token
#pragma unroll
          for (int i = 0; i < 16 * kQuads / 128; ++i) {
            const int w = i * 128 + tid, tok = w / kQuads, c = (w % kQuads) * 4;
            float4 o = *reinterpret_cast<const float4*>(st + tok * kSkRows + c);
            if (MODE == 2) {
              const float4 up = *reinterpret_cast<const float4*>(st + tok * kSkRows + 64 + c);
              o = make_float4(swiglu1(o.x, up.x), swiglu1(o.y, up.y), swiglu1(o.z, up.z), swiglu1(o.w, up.w));
            }
            if (16 * b + tok < cnt)
              skinny_store4(p.out, 0, (t.x_row + at + 16 * b + tok) * p.ldo + t.col + c, t.col + c, p.N,
                            t.col + c + 4 <= p.N && (p.ldo & 3) == 0, o);
          }
        }
        tc_fence_before_sync();
        asm volatile("bar.sync 1, 128;" ::: "memory");         // all of the accumulator and the staging have been read
        if (tid == 0) mbar_arrive(&acc_empty[acc]);
      }
    }
  }

  __syncwarp();                                    // the aligned barriers below need whole warps
  tc_fence_before_sync();
  if (skinny_dense(MODE)) {
    if (slices > 1) cluster_sync_all(); else __syncthreads();      // every slice's sums are in its shared memory
    const int col0 = first * (MODE == 3 ? 64 : kSkRows);
    const float f = MODE == 3 ? skinny_factor(p, col0 / p.seg) : 1.f;      // a tile lies in one segment
    switch (slices) {
      case 1: skinny_sum<MODE, 1>(p, smem, slice, col0, f, smem_u32(failed)); break;
      case 2: skinny_sum<MODE, 2>(p, smem, slice, col0, f, smem_u32(failed)); break;
      case 3: skinny_sum<MODE, 3>(p, smem, slice, col0, f, smem_u32(failed)); break;
      case 4: skinny_sum<MODE, 4>(p, smem, slice, col0, f, smem_u32(failed)); break;
      case 6: skinny_sum<MODE, 6>(p, smem, slice, col0, f, smem_u32(failed)); break;
      default: skinny_sum<MODE, 8>(p, smem, slice, col0, f, smem_u32(failed));
    }
    if (slices > 1) cluster_sync_all();            // nobody reads this CTA's shared memory any more
  }
  block_settle(p.status);
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace yv
