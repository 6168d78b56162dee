// Host side of the few-token products: tensor maps, number of K slices, choice of the token slots.
#include "per_device.h"
#include "skinny.cuh"
#include "tensormap.h"
#include "yv_ops.h"

namespace yv {

namespace {

int sm_count() {
  static PerDeviceInt n;
  int& v = n.cur();
  if (v == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    if (v <= 0) v = 148;
  }
  return v;
}

template <int NT, int MODE>
int launch(const SkinnyParams& p, int grid, int cluster, cudaStream_t stream) {
  auto kern = skinny_kernel<NT, MODE>;
  static PerDeviceInt configured;
  if (!configured.cur()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SkinnySmem<NT>::kTotal);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured.cur() = 1;
  }
  return launch_chained(kern, dim3(static_cast<unsigned>(grid)), dim3(kSkThreads), SkinnySmem<NT>::kTotal, stream, cluster, p);
}

// Clusters of `slices` CTAs that the device holds at two CTAs per SM: fewer than the CTAs would allow, since a cluster stays
// within one group of SMs (148 of two, 93 of three, 71 of four, 45 of six, 33 of eight).  An empty kernel of the same shape
// is asked about, since the answer for a kernel that allocates tensor memory counts one CTA per SM.
__global__ void __launch_bounds__(kSkThreads, 2) skinny_shape_kernel() {}

int clusters_at_once(int slices) {
  static PerDeviceInt known[9];
  int& n = known[slices].cur();
  if (n != 0) return n;
  auto kern = skinny_shape_kernel;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(slices));
  cfg.blockDim = dim3(kSkThreads);
  cfg.dynamicSmemBytes = SkinnySmem<128>::kTotal;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(slices);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int found = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SkinnySmem<128>::kTotal) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&found, kern, &cfg) != cudaSuccess || found <= 0)
    found = 1;
  return n = found;
}

template <int MODE>
int dispatch(int tokens, const SkinnyParams& p, int grid, int cluster, cudaStream_t stream) {
  if (tokens <= 16) return launch<16, MODE>(p, grid, cluster, stream);
  if (tokens <= 32) return launch<32, MODE>(p, grid, cluster, stream);
  if (tokens <= 64) return launch<64, MODE>(p, grid, cluster, stream);
  return launch<128, MODE>(p, grid, cluster, stream);
}

}  // namespace

int launch_skinny(const SkinnyArgs& a, cudaStream_t stream) {
  if (a.N <= 0 || a.K <= 0) return -1;
  SkinnyParams p = {};
  p.N = a.N; p.K = a.K;
  p.out = a.out; p.out_fp32 = a.out_fp32; p.ldo = a.ldo;
  p.bias = static_cast<const __nv_bfloat16*>(a.bias);
  p.status = a.status;
  const bool grouped = a.experts > 0;
  const int rows = a.swiglu ? 64 : kSkRows;
  p.tiles_w = (a.N + rows - 1) / rows;
  p.w_rows = a.swiglu ? 2 * a.N : a.N;
  const uint64_t w_rows = static_cast<uint64_t>(p.w_rows) * static_cast<uint64_t>(grouped ? a.experts : 1);
  int r = make_tmap_2d(&p.tma_w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.w, a.K, w_rows, a.ldw, 64, rows);
  if (r != 0) return -20 + r;
  r = make_tmap_2d(&p.tma_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a.x, a.K, a.x_rows, a.ldx, 64, 16);
  if (r != 0) return -30 + r;
  if (!grouped) {
    if (a.M < 1 || a.M > 128) return -2;
    if (a.swiglu && (a.seg <= 0 || a.seg % 64 != 0 || a.N % a.seg != 0 || a.bias != nullptr)) return -4;
    p.M = a.M;
    p.seg = a.seg;
    p.scale = a.scale;
    p.scale_fp32 = a.scale_fp32;
    p.scale_softmax = a.scale_softmax;
    // as many slices of K as keep all clusters resident and leave four 64-wide steps to each; one cluster more than fits costs
    // a second round (6144 x 4096, one token: 48 clusters of six 15.8 us, of four 12.4; 128 tokens 24.5 and 18.4)
    const int kc = (a.K + 63) / 64;
    int slices = 1;
    for (int s : {2, 3, 4, 6, 8})
      if (s * 4 <= kc && p.tiles_w <= clusters_at_once(s)) slices = s;
    const int grid = p.tiles_w * slices;
    return a.swiglu ? dispatch<3>(a.M, p, grid, slices, stream) : dispatch<0>(a.M, p, grid, slices, stream);
  }
  // a tile that reached into the next expert's rows would compute with them; its outputs past N are dropped, the gate and up
  // halves of a fused tile must be whole
  if (a.out_fp32 || a.bias != nullptr || (a.swiglu && a.N % 64 != 0)) return -3;
  p.tile_expert = a.tile_expert; p.num_m_tiles = a.num_m_tiles;
  p.seg_offsets = a.seg_offsets; p.counts = a.counts;
  const int64_t units = static_cast<int64_t>(a.max_tiles) * p.tiles_w, room = 2 * sm_count();
  const int grid = static_cast<int>(units < room ? units : room);
  if (grid <= 0) return 0;
  return a.swiglu ? dispatch<2>(a.slots, p, grid, 1, stream) : dispatch<1>(a.slots, p, grid, 1, stream);
}

}  // namespace yv
