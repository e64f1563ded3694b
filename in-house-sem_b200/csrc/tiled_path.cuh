// Host side of the tiled fused step: tiling, device numbering and launches.
#pragma once

#include <algorithm>
#include <cstdint>
#include <map>
#include <vector>

#include "device_data.cuh"
#include "tiled.cuh"

namespace insem_b200 {

// Per-point special terms of one domain, in the reference's point numbering.
struct SpecialTerms {
  std::map<int32_t, std::vector<std::pair<int32_t, std::vector<float>>>> sources;  // point -> (source, coef[ncomp])
  std::map<int32_t, std::vector<int32_t>> coupling;                               // point -> coupling entries
  std::map<int32_t, int32_t> absorbing;                                           // point -> Stacey index
  std::map<int32_t, uint8_t> zero;                                                // point -> zeroed components
  std::vector<int32_t> receivers;                                                 // points read by receivers
  std::vector<int32_t> coupled;  // coupled points in chunk order: numbered last, in this order
};

// First device points of every tile: inner points in `ni` x `ni` rows of 32,
// one per lane, whatever the tile holds (so that rows lie at fixed distances),
// then its edge points, each range starting on a multiple of 32 points; then
// the halo points.  The gaps are unused padding points.
struct TileNumbers {
  std::vector<int32_t> cbeg, ebeg;  // [tiles + 1] inner points, [tiles] edge points
  int32_t n_complete = 0;
  int32_t stride = 0;               // points of a component: all of them, rounded up to 4 (16 bytes), at least 4
};
// edge_points[t]: edge complete points of tile t.  Device points are 32-bit:
// the padding of many part-filled tiles may need more, which is refused here
// before anything is sized by it.
inline TileNumbers number_tiles(const std::vector<int32_t>& edge_points, int ni, int32_t n_halo) {
  TileNumbers t;
  t.cbeg.reserve(edge_points.size() + 1);
  t.ebeg.reserve(edge_points.size());
  int64_t at = 0;
  auto point = [&](int64_t p) {
    INSEM_REQUIRE(p <= INT32_MAX, INSEM_CUDA_ERR_UNSUPPORTED,
                  "the domain's tiles need more than 2^31 - 1 points with their padding (options.path = 1 takes none)");
    return static_cast<int32_t>(p);
  };
  for (int32_t edge : edge_points) {
    t.cbeg.push_back(point(at));
    t.ebeg.push_back(point(at + kTileLanes * ni * ni));
    at = (at + kTileLanes * ni * ni + edge + kTileLanes - 1) / kTileLanes * kTileLanes;
  }
  t.cbeg.push_back(point(at));
  t.n_complete = point(at);
  t.stride = point(std::max<int64_t>((at + n_halo + 3) / 4 * 4, 4));
  return t;
}

// One domain of the tiled path.
class TiledDomain {
 public:
  // Builds tiles of at most `te` elements per block and the device numbering.
  void build(const insem_cuda_domain& d, int ngll, int te, const SpecialTerms& sp, const std::vector<float>& abs_coef);

  // ng: component stride of the device arrays (points padded so that every
  // tile's complete range starts on a 16-byte boundary); ng_ref: the
  // reference's point count.  Halo points are [n_complete, n_complete + n_halo).
  int medium = 0, ncomp = 1, m = 0, ng = 0, ng_ref = 0, npe = 0, n_elements = 0;
  int n_complete = 0, n_halo = 0, n_tiles = 0, tp_cap = 0, nc_cap = 0, n_hbuf = 0;
  int rank_cap = 1;  // the most contributions one complete point of a tile has
  int te = 0;  // elements per tile
  bool weighted = false;
  std::vector<int32_t> perm;  // reference point -> device point
  DeviceBuffer<int32_t> device_perm;  // the same on the device, from the first state() on
  struct BlockTiles {
    int kind = 0, m = 0, tile0 = 0, ntiles = 0, n = 0;  // kind of the tile kernels
    bool any_axial = false;
    DeviceBuffer<float> data, coef0, coef1;  // [tile][tile_data_floats], [tile][32]
    DeviceBuffer<uint8_t> axial;
    BlockDev view() const;
  };
  std::vector<BlockTiles> blocks;
  // device data
  DeviceBuffer<uint16_t> sdesc, plist;
  DeviceBuffer<TileHdr> tiles;
  std::vector<TileHdr> host_tiles;  // the same headers on the host (the batched tile items copy them)
  DeviceBuffer<int32_t> halo_tp, hs_slot, hs_dst, mdst_off, mdst, cs_slot;
  DeviceBuffer<int2> cs_row;
  DeviceBuffer<float> hbuf, mass, inv_mass;
  DeviceBuffer<float> u0, u1, v, a, vn;
  DeviceBuffer<int32_t> h_off, h_spec, src_which;
  DeviceBuffer<HaloRec> h_rec;
  DeviceBuffer<CouplingEntry> h_cpl;
  DeviceBuffer<float> h_w, src_coef, abs_coef_d;
  std::vector<int32_t> cpl_entry;  // coupling entry of each h_cpl element (its partner is filled in by set_partners)
  void set_partners(const std::vector<int32_t>& partner, const std::vector<float>& cx, const std::vector<float>& cz);
  DeviceBuffer<int32_t> rows_off, rows_dofs;  // constraint rows in device numbering
  DeviceBuffer<float> rows_w;
  RowsDev rows() const { return {rows_off.get(), rows_dofs.get(), rows_w.get()}; }
  std::vector<float> host_mass;

  TiledDev view(int parity) const;  // parity 0: u0 current, u1 next
  HaloDev halo_view() const;
  float* u_cur(int parity) { return parity ? u1.get() : u0.get(); }
};

// Opts a kernel in to all the shared memory a CTA may have beside its static
// part: the same value for every solve, so that none lowers another's.
template <class Kernel>
void allow_shared_memory(Kernel kernel) {
  cudaFuncAttributes fa;
  CUDA_CHECK(cudaFuncGetAttributes(&fa, kernel));
  CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  227 * 1024 - static_cast<int>(fa.sharedSizeBytes)));
}

// Launchers, instantiated per ngll in tiled_ng.cu.
struct TileLaunch {
  const TiledDomain* dom = nullptr;
  int block = 0;
  int parity = 0;
  StepScalars sc{};
  StepState* st = nullptr;
  double* epartial = nullptr;
  bool elastic = false;
  StepIdx ix{};
  bool overlap = false;  // may start before the kernel ahead of it on the stream has ended (see DepMode)
  cudaStream_t stream = nullptr;
};
void launch_tiles_ng2(const TileLaunch&);
void launch_tiles_ng3(const TileLaunch&);
void launch_tiles_ng4(const TileLaunch&);
void launch_tiles_ng5(const TileLaunch&);
void launch_tiles_ng6(const TileLaunch&);
void launch_tiles_ng7(const TileLaunch&);
void launch_tiles_ng8(const TileLaunch&);
void launch_tiles_ng9(const TileLaunch&);
void launch_tiles(int ngll, const TileLaunch& a);
// Elements per tile of a domain: `requested` if > 0, else a registered entry
// (set_tile_elements, e.g. from the autotuner), at most the kernel's 32; by
// default 32, which leaves no lane idle and the fewest points shared between
// tiles.
int choose_tile_elements(int ngll, int kind, bool elastic, int m, int requested);
void set_tile_elements(int ngll, int kind, bool elastic, int m, int te);  // te <= 0 clears the entry
// Uploads the GLL / GLJ basis of one ngll to constant memory (must agree with earlier uploads).
void set_constant_basis(int ngll, const std::vector<float>& D, const std::vector<float>& Dj,
                        const std::vector<float>& w2);

// Batched tile launches: one launch per tile class (ngll, kind, medium,
// order) over the work items of many solves, one CTA per item.
struct TileBatchLaunch {
  int kind = 0, m = 0;
  bool elastic = false;
  const TileSeg* segs = nullptr;
  const TileItem* items = nullptr;
  TileLayout L{};  // the class layout
  uint32_t smem = 0;
  int grid = 0;
  StepIdx ix{};
  bool overlap = false;
  cudaStream_t stream = nullptr;
};
// launch == false: opts the class kernel in to its dynamic shared memory
// (outside stream capture); true: launches.
void tile_batch_ng2(const TileBatchLaunch&, bool launch);
void tile_batch_ng3(const TileBatchLaunch&, bool launch);
void tile_batch_ng4(const TileBatchLaunch&, bool launch);
void tile_batch_ng5(const TileBatchLaunch&, bool launch);
void tile_batch_ng6(const TileBatchLaunch&, bool launch);
void tile_batch_ng7(const TileBatchLaunch&, bool launch);
void tile_batch_ng8(const TileBatchLaunch&, bool launch);
void tile_batch_ng9(const TileBatchLaunch&, bool launch);
void tile_batch(int ngll, const TileBatchLaunch& a, bool launch);

template <int NG>
void tile_batch_cfg(const TileBatchLaunch& a, bool launch) {
  INSEM_REQUIRE(a.smem <= 226u * 1024u, INSEM_CUDA_ERR_UNSUPPORTED, "tile needs too much shared memory");
  auto go = [&](auto kernel) {
    if (!launch) {
      allow_shared_memory(kernel);
      return;
    }
    cudaError_t err = launch_chained(kernel, a.grid, TileCfg<NG>::THREADS, a.smem, a.stream, a.overlap, a.segs,
                                     a.items, a.ix, a.L);
    if (err == cudaSuccess) err = cudaGetLastError();
    if (err != cudaSuccess)
      throw Error(INSEM_CUDA_ERR_CUDA, "batched tile kernel launch (ngll " + std::to_string(NG) + ", kind " +
                                           std::to_string(a.kind) + ", grid " + std::to_string(a.grid) + ", smem " +
                                           std::to_string(a.smem) + "): " + cudaGetErrorString(err));
  };
  if (a.kind == kAxisymOffAxis)
    return a.m == 1 ? go(tile_batch_kernel<NG, kAxisymOffAxis, true, 1>) : go(tile_batch_kernel<NG, kAxisymOffAxis, true, 0>);
  if (a.kind == kAxisymSeparable) {
    if (a.m == 1)
      return a.elastic ? go(tile_batch_kernel<NG, kAxisymSeparable, true, 1>) : go(tile_batch_kernel<NG, kAxisymSeparable, false, 1>);
    return a.elastic ? go(tile_batch_kernel<NG, kAxisymSeparable, true, 0>) : go(tile_batch_kernel<NG, kAxisymSeparable, false, 0>);
  }
  if (a.kind == INSEM_AXISYM) {
    if (a.m == 1) return a.elastic ? go(tile_batch_kernel<NG, INSEM_AXISYM, true, 1>)
                                   : go(tile_batch_kernel<NG, INSEM_AXISYM, false, 1>);
    return a.elastic ? go(tile_batch_kernel<NG, INSEM_AXISYM, true, 0>) : go(tile_batch_kernel<NG, INSEM_AXISYM, false, 0>);
  }
  switch (a.kind) {
    case INSEM_RECT:
      return a.elastic ? go(tile_batch_kernel<NG, INSEM_RECT, true, 0>) : go(tile_batch_kernel<NG, INSEM_RECT, false, 0>);
    case INSEM_AFFINE:
      return a.elastic ? go(tile_batch_kernel<NG, INSEM_AFFINE, true, 0>)
                       : go(tile_batch_kernel<NG, INSEM_AFFINE, false, 0>);
    default:
      return a.elastic ? go(tile_batch_kernel<NG, INSEM_CURVED, true, 0>)
                       : go(tile_batch_kernel<NG, INSEM_CURVED, false, 0>);
  }
}

template <int NG>
void launch_tiles_cfg(const TileLaunch& a) {
  const TiledDomain& d = *a.dom;
  const auto& b = d.blocks[a.block];
  if (b.ntiles == 0) return;
  auto go = [&](auto one_wave, auto many_waves, int nc) {
    const TileLayout L = TileLayout::make(NG, nc, b.kind, a.elastic, d.te, d.tp_cap, d.nc_cap, d.rank_cap);
    const size_t smem = b.any_axial || !is_axisym(b.kind) ? L.total : L.ax;
    INSEM_REQUIRE(smem <= 226 * 1024, INSEM_CUDA_ERR_UNSUPPORTED, "tile needs too much shared memory");
    // The kernel with the compiler's own registers where it holds all tiles at
    // once; and the opt-in to this launch's dynamic shared memory (outside
    // stream capture; the first launch of every tile kernel happens in the
    // uncaptured initial step).
    auto kernel = many_waves;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CUDA_CHECK(cudaStreamIsCapturing(a.stream, &cap));
    if (cap == cudaStreamCaptureStatusNone)
      for (auto k : {one_wave, many_waves})
        allow_shared_memory(k);
    int per_sm = 0, device = 0, sms = 0;
    CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, one_wave, TileCfg<NG>::THREADS, smem));
    CUDA_CHECK(cudaGetDevice(&device));
    CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    if (b.ntiles <= per_sm * sms) kernel = one_wave;
    TiledDev td = d.view(a.parity);
    cudaError_t err = launch_chained(kernel, b.ntiles, TileCfg<NG>::THREADS, smem, a.stream, a.overlap, b.view(), td,
                                     a.sc, a.st, a.epartial, static_cast<int32_t>(b.tile0), a.ix, L);
    if (err == cudaSuccess) err = cudaGetLastError();
    if (err != cudaSuccess)
      throw Error(INSEM_CUDA_ERR_CUDA, "tile kernel launch (ngll " + std::to_string(NG) + ", kind " +
                                           std::to_string(b.kind) + ", tiles " + std::to_string(b.ntiles) +
                                           ", threads " + std::to_string(TileCfg<NG>::THREADS) + ", smem " +
                                           std::to_string(smem) + "): " + cudaGetErrorString(err));
  };
  if (b.kind == kAxisymOffAxis) {
    constexpr int K = kAxisymOffAxis;
    if (b.m == 1) go(tile_step_kernel<NG, K, true, 1, true>, tile_step_kernel<NG, K, true, 1, false>, 3);
    else go(tile_step_kernel<NG, K, true, 0, true>, tile_step_kernel<NG, K, true, 0, false>, 2);
    return;
  }
  if (b.kind == kAxisymSeparable) {
    constexpr int K = kAxisymSeparable;
    if (b.m == 1) {
      if (a.elastic) go(tile_step_kernel<NG, K, true, 1, true>, tile_step_kernel<NG, K, true, 1, false>, 3);
      else go(tile_step_kernel<NG, K, false, 1, true>, tile_step_kernel<NG, K, false, 1, false>, 1);
    } else {
      if (a.elastic) go(tile_step_kernel<NG, K, true, 0, true>, tile_step_kernel<NG, K, true, 0, false>, 2);
      else go(tile_step_kernel<NG, K, false, 0, true>, tile_step_kernel<NG, K, false, 0, false>, 1);
    }
    return;
  }
  if (b.kind == INSEM_AXISYM) {
    if (b.m == 1) {
      if (a.elastic) go(tile_step_kernel<NG, INSEM_AXISYM, true, 1, true>, tile_step_kernel<NG, INSEM_AXISYM, true, 1, false>, 3);
      else go(tile_step_kernel<NG, INSEM_AXISYM, false, 1, true>, tile_step_kernel<NG, INSEM_AXISYM, false, 1, false>, 1);
    } else {
      if (a.elastic) go(tile_step_kernel<NG, INSEM_AXISYM, true, 0, true>, tile_step_kernel<NG, INSEM_AXISYM, true, 0, false>, 2);
      else go(tile_step_kernel<NG, INSEM_AXISYM, false, 0, true>, tile_step_kernel<NG, INSEM_AXISYM, false, 0, false>, 1);
    }
    return;
  }
  switch (b.kind) {
    case INSEM_RECT:
      if (a.elastic) go(tile_step_kernel<NG, INSEM_RECT, true, 0, true>, tile_step_kernel<NG, INSEM_RECT, true, 0, false>, 2);
      else go(tile_step_kernel<NG, INSEM_RECT, false, 0, true>, tile_step_kernel<NG, INSEM_RECT, false, 0, false>, 1);
      break;
    case INSEM_AFFINE:
      if (a.elastic) go(tile_step_kernel<NG, INSEM_AFFINE, true, 0, true>, tile_step_kernel<NG, INSEM_AFFINE, true, 0, false>, 2);
      else go(tile_step_kernel<NG, INSEM_AFFINE, false, 0, true>, tile_step_kernel<NG, INSEM_AFFINE, false, 0, false>, 1);
      break;
    default:
      if (a.elastic) go(tile_step_kernel<NG, INSEM_CURVED, true, 0, true>, tile_step_kernel<NG, INSEM_CURVED, true, 0, false>, 2);
      else go(tile_step_kernel<NG, INSEM_CURVED, false, 0, true>, tile_step_kernel<NG, INSEM_CURVED, false, 0, false>, 1);
      break;
  }
}

}  // namespace insem_b200
