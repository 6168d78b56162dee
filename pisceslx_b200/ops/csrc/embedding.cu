// Gradient of the token embedding: dW[v] = the sum of the gradient rows of all tokens v, in fp32 and in token order, so that its bits
// repeat; rows of words that do not occur are zero.
//
// Bound by the bytes of dW, which is written once as zeros, and of the gradient.  The tokens are put in order of their words by
// counting: a token's place is the number of smaller words plus that of equal ones before it, T^2 comparisons without a
// launch-by-launch sort.  Runs of equal words are then summed 32 places to a block; runs that cross blocks go through fp32 carries.
// 8192 tokens of 4096, 32000 words: 766 us by sort, segments and their sums in a kernel each; 90 here, of which 45 are the zeros.
// 2331 of 1024, 154856 words 204 -> 70 us; 32768 of 4096 2064 -> 268 (884 where all are the same word: one run through 1024 carries).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "yv_ops.h"

namespace yv {
namespace {

constexpr int kRankChunk = 2048;
constexpr int kPlaces = 32;          // places of the order per block of the sums

// 32 tokens per block, 8 lanes each, every lane an eighth of the comparisons.
__global__ void __launch_bounds__(256) embed_rank_kernel(const int64_t* __restrict__ ids, int T, int* __restrict__ order,
                                                         int* __restrict__ sorted) {
  __shared__ int4 chunk[kRankChunk / 4];
  int* flat = reinterpret_cast<int*>(chunk);
  const int t = blockIdx.x * 32 + (threadIdx.x >> 3), lane = threadIdx.x & 7;
  const int id = t < T ? static_cast<int>(ids[t]) : 0;
  int place = 0;
  for (int c0 = 0; c0 < T; c0 += kRankChunk) {
    __syncthreads();
    for (int i = threadIdx.x; i < kRankChunk; i += 256) flat[i] = c0 + i < T ? static_cast<int>(ids[c0 + i]) : 0x7FFFFFFF;
    __syncthreads();
    if (t < c0 || t >= c0 + kRankChunk) {
      const int below = id + (t >= c0 ? 1 : 0);        // equal words count where they come before
#pragma unroll 8
      for (int i = lane; i < kRankChunk / 4; i += 8) {
        const int4 v = chunk[i];
        place += (v.x < below) + (v.y < below) + (v.z < below) + (v.w < below);
      }
    } else {
      for (int i = lane; i < kRankChunk; i += 8) place += flat[i] < id + (c0 + i < t ? 1 : 0);
    }
  }
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) place += __shfl_xor_sync(0xFFFFFFFFu, place, off);
  if (lane == 0 && t < T) {
    order[place] = t;
    sorted[place] = id;
  }
}

__device__ __forceinline__ void store_row(__nv_bfloat16* dst, const float (&a)[8]) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(a[2 * i], a[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&p);
  }
  *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
}

// carry [2][blocks][H]: of each block the part of its first run, if that began before it, and of its last, if that began here and
// goes on.
__global__ void __launch_bounds__(256) embed_sum_kernel(const __nv_bfloat16* __restrict__ dy, const int* __restrict__ order,
                                                        const int* __restrict__ sorted, __nv_bfloat16* __restrict__ dw,
                                                        float* __restrict__ carry, int T, int H) {
  __shared__ int s_order[kPlaces], s_id[kPlaces + 2];
  const int b = blockIdx.x, first = b * kPlaces, n = min(kPlaces, T - first);
  if (threadIdx.x < n) s_order[threadIdx.x] = order[first + threadIdx.x];
  if (threadIdx.x < n + 2) {
    const int at = first + static_cast<int>(threadIdx.x) - 1;
    s_id[threadIdx.x] = at >= 0 && at < T ? sorted[at] : -1;
  }
  __syncthreads();
  const int col = (blockIdx.y * 256 + threadIdx.x) * 8;
  if (col >= H) return;
  float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  bool opened_before = s_id[0] == s_id[1];
  for (int i0 = 0; i0 < n; i0 += 8) {
    uint4 row[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (i0 + j < n) row[j] = *reinterpret_cast<const uint4*>(dy + static_cast<int64_t>(s_order[i0 + j]) * H + col);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int i = i0 + j;
      if (i >= n) break;
      const uint32_t w[4] = {row[j].x, row[j].y, row[j].z, row[j].w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        a[2 * q] += __uint_as_float(w[q] << 16);
        a[2 * q + 1] += __uint_as_float(w[q] & 0xFFFF0000u);
      }
      const bool goes_on = s_id[i + 2] == s_id[i + 1];
      if (goes_on && i + 1 < n) continue;
      if (opened_before || goes_on) {
        float* c = carry + (static_cast<int64_t>(opened_before ? 0 : gridDim.x) + b) * H + col;
        *reinterpret_cast<float4*>(c) = make_float4(a[0], a[1], a[2], a[3]);
        *reinterpret_cast<float4*>(c + 4) = make_float4(a[4], a[5], a[6], a[7]);
      } else {
        store_row(dw + static_cast<int64_t>(s_id[i + 1]) * H + col, a);
      }
      opened_before = false;
#pragma unroll
      for (int q = 0; q < 8; ++q) a[q] = 0.f;
    }
  }
}

// Runs that cross blocks: by the block in which they begin.
__global__ void __launch_bounds__(256) embed_join_kernel(const int* __restrict__ sorted, const float* __restrict__ carry,
                                                         __nv_bfloat16* __restrict__ dw, int T, int H) {
  const int b = blockIdx.x, last = b * kPlaces + kPlaces - 1;
  if (last + 1 >= T) return;
  const int id = sorted[last];
  if (sorted[last + 1] != id || (b > 0 && sorted[b * kPlaces - 1] == id)) return;
  const int col = (blockIdx.y * 256 + threadIdx.x) * 8;
  if (col >= H) return;
  float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const float* c = carry + (static_cast<int64_t>(gridDim.x) + b) * H + col;
  for (int j = b;;) {
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] += c[q];
    ++j;
    if (j * kPlaces >= T || sorted[j * kPlaces] != id) break;
    c = carry + static_cast<int64_t>(j) * H + col;
  }
  store_row(dw + static_cast<int64_t>(id) * H + col, a);
}

}  // namespace

int launch_embedding_grad(const void* dy, const int64_t* ids, void* dw, int* order, float* carry, int64_t T, int64_t V, int H,
                          cudaStream_t stream) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dw) | reinterpret_cast<uintptr_t>(carry);
  if ((H & 7) != 0 || (at & 15u) != 0 || T > kEmbeddingGradTokens || V <= 0 || V >= 0x7FFFFFFF) return -1;
  const int r = static_cast<int>(cudaMemsetAsync(dw, 0, static_cast<size_t>(V) * H * 2, stream));
  if (r != 0 || T <= 0) return r;
  const int n = static_cast<int>(T), blocks = (n + kPlaces - 1) / kPlaces, across = (H / 8 + 255) / 256;
  int* sorted = order + n;
  auto* g = reinterpret_cast<const __nv_bfloat16*>(dy);
  auto* w = reinterpret_cast<__nv_bfloat16*>(dw);
  embed_rank_kernel<<<(n + 31) / 32, 256, 0, stream>>>(ids, n, order, sorted);
  embed_sum_kernel<<<dim3(blocks, across), 256, 0, stream>>>(g, order, sorted, w, carry, n, H);
  if (blocks > 1) embed_join_kernel<<<dim3(blocks, across), 256, 0, stream>>>(sorted, carry, w, n, H);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace yv
