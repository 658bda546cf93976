// Entry points of the PCG path: SpMV, SYMGS, the V-cycle, CG and the vector
// routines, with the host-side drivers that sequence the kernels.
#include <atomic>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <cmath>
#include <new>
#include <thread>
#include <vector>

#include <algorithm>

#include "kernels.cuh"
#include "wave.cuh"

namespace hb {

namespace {

constexpr int kPerSm = 8;  // resident 256-thread blocks per SM targeted by grid-stride kernels

// The column array a kernel of value type T reads: the FP32 V-cycle has its own,
// in its blocked layout.
template <typename T>
const int* cols_of(const Level& L) {
  return sizeof(T) == 4 ? L.col32 : L.col;
}

inline int red_blocks(const Context* c, int64_t n) {
  int b = grid_for(c, n, kThreads, kPerSm);
  return b > kRedBlocksMax / 2 ? kRedBlocksMax / 2 : b;
}

// The tiled phase (configuration 9): one block per SM-resident slot, walking
// tiles of rows; its dynamic shared memory is enabled on first launch.
template <typename T, typename TR, bool FIRST, int CFG, int64_t CMASK, bool DOT>
void gs_tile_launch(Context* c, const Level& L, const T* val, const TR* rhs, T* x, int r0, int r1, uint32_t mask,
                    double* dot) {
  auto k = k_gs_tile<T, TR, FIRST, CFG, CMASK, DOT>;
  constexpr int smem = gs_tile_smem<T>(CFG);
  constexpr int rows = gs_tile_rows<T>(CFG);
  static int per_sm = 0;  // resident blocks per SM with that shared memory (one device's figure)
  if (per_sm == 0) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, rows, smem) != cudaSuccess || per_sm < 1) {
      cudaGetLastError();
      per_sm = 1;
    }
  }
  const int a0 = r0 & ~3;
  const int64_t tiles = ((int64_t)r1 - a0 + rows - 1) / rows;
  int g = (int)std::min<int64_t>(tiles, (int64_t)c->sms * per_sm);
  if (DOT && g > kDotStride) g = kDotStride;
  k<<<g, rows, smem, c->stream>>>(val, cols_of<T>(L), L.pitch, rhs, x, r0, r1, mask, dot);
}

// The sweep position whose rows start at r0.
inline int sweep_at(const Level& L, int r0) {
  int s = 0;
  while (s + 1 < kColours && (L.g.start[s] != r0 || L.g.start[s + 1] == r0)) ++s;
  return s;
}

// The bulk-copy pipeline (configuration 10): one block per SM (its shared
// memory allows no second), at most one per tile; PW: the level's column form
// (L.pack). false: not launched (FP64 tensor maps unavailable, or refused).
template <typename T, typename TR, bool FIRST, int64_t CMASK, bool DOT, int PW>
bool gs_bulk_launch_p(Context* c, const Level& L, const T* val, const TR* rhs, T* x, int r0, int r1,
                      uint32_t mask, double* dot) {
  auto k = k_gs_bulk<T, TR, FIRST, CMASK, DOT, PW>;
  using Shape = GsShape<T, PW>;
  constexpr int smem = Shape::smem;
  static CUtensorMap none;  // the FP32 kernels take no maps
  const CUtensorMap* tv = &none;
  const CUtensorMap* tc = &none;
  if constexpr (bulk_tensor_tile<T>()) {
    const BulkMaps* m = bulk_maps(L);
    if (!m) return false;
    tv = &m->val;
    tc = &m->col;
  }
  static std::atomic<uint64_t> attr_set{0};  // devices on which the shared-memory size is enabled
  bulk_attr(k, smem, c->device, &attr_set);
  const int a0 = r0 & ~(Shape::tile_rows - 1);
  const int64_t tiles = ((int64_t)r1 - a0 + Shape::tile_rows - 1) / Shape::tile_rows;
  int g = (int)std::min<int64_t>(tiles, (int64_t)c->sms);
  if (DOT && g > kDotStride) g = kDotStride;
  // programmatic dependent launch: the phase's producer streams its first
  // matrix tiles while the previous kernel finishes (HPCG_B200_PDL=0: off)
  const bool pdl = pdl_enabled();
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(g);
  cfg.blockDim = dim3(Shape::threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  GeoPhase geo{};
  if constexpr (PW == kPackGeo) geo = L.geo_cols->block[sweep_at(L, r0)];
  cudaError_t e = cudaLaunchKernelEx(&cfg, k, val, cols_of<T>(L), L.pitch, rhs, x, r0, r1, mask, dot, c->fault,
                                     *tv, *tc, (const unsigned char*)L.colp, sink_of(L), geo);
  if (e != cudaSuccess && pdl) {
    // refused with the early-launch attribute: record it and launch plainly
    set_error("k_gs_bulk (programmatic dependent launch)", e);
    cudaGetLastError();
    cfg.numAttrs = 0;
    e = cudaLaunchKernelEx(&cfg, k, val, cols_of<T>(L), L.pitch, rhs, x, r0, r1, mask, dot, c->fault, *tv, *tc,
                           (const unsigned char*)L.colp, sink_of(L), geo);
  }
  if (e != cudaSuccess) {
    // refused outright (nothing was queued): the caller runs the register kernel instead
    set_error("k_gs_bulk", e);
    cudaGetLastError();
    return false;
  }
  return true;
}

template <typename T, typename TR, bool FIRST, int64_t CMASK, bool DOT>
bool gs_bulk_launch(Context* c, const Level& L, const T* val, const TR* rhs, T* x, int r0, int r1, uint32_t mask,
                    double* dot) {
  if (L.geo_cols) return gs_bulk_launch_p<T, TR, FIRST, CMASK, DOT, kPackGeo>(c, L, val, rhs, x, r0, r1, mask, dot);
  if (L.pack == kPackDiag)
    return gs_bulk_launch_p<T, TR, FIRST, CMASK, DOT, kPackDiag>(c, L, val, rhs, x, r0, r1, mask, dot);
  if (L.pack == 1) return gs_bulk_launch_p<T, TR, FIRST, CMASK, DOT, 1>(c, L, val, rhs, x, r0, r1, mask, dot);
  if (L.pack == 2) return gs_bulk_launch_p<T, TR, FIRST, CMASK, DOT, 2>(c, L, val, rhs, x, r0, r1, mask, dot);
  return gs_bulk_launch_p<T, TR, FIRST, CMASK, DOT, 0>(c, L, val, rhs, x, r0, r1, mask, dot);
}

// dot != nullptr: the phase also writes its r'z block partials there (FP64
// full-slot phases only; the grid is capped at kDotStride blocks).
template <typename T, typename TR, bool FIRST, int CFG, int64_t CMASK = -1>
void gs_launch(Context* c, const Level& L, const T* val, const TR* rhs, T* x, int r0, int r1, uint32_t mask,
               double* dot = nullptr) {
  if constexpr (CFG == kBulkCfg) {
    if (r1 <= r0) return;
    bool done = false;
    if constexpr (!FIRST && CMASK < 0) {
      // the full-slot phases with the mask compiled in: the 27 gathers of a row
      // are issued back to back instead of behind one test each
      if (mask == kAllSlots) {
        if constexpr (sizeof(T) == 8) {
          if (dot) done = gs_bulk_launch<T, TR, false, kAllSlots, true>(c, L, val, rhs, x, r0, r1, mask, dot);
        }
        if (!dot) done = gs_bulk_launch<T, TR, false, kAllSlots, false>(c, L, val, rhs, x, r0, r1, mask, nullptr);
      } else {
        done = gs_bulk_launch<T, TR, FIRST, CMASK, false>(c, L, val, rhs, x, r0, r1, mask, nullptr);
      }
    } else {
      done = gs_bulk_launch<T, TR, FIRST, CMASK, false>(c, L, val, rhs, x, r0, r1, mask, nullptr);
    }
    if (!done) gs_launch<T, TR, FIRST, 1, CMASK>(c, L, val, rhs, x, r0, r1, mask, dot);  // no tensor maps here
    return;
  } else if constexpr (cfg_tiled(CFG)) {
    if (r1 <= r0) return;
    if constexpr (!FIRST && CMASK < 0 && sizeof(T) == 8) {
      if (dot) {
        gs_tile_launch<T, TR, FIRST, CFG, CMASK, true>(c, L, val, rhs, x, r0, r1, mask, dot);
        return;
      }
    }
    gs_tile_launch<T, TR, FIRST, CFG, CMASK, false>(c, L, val, rhs, x, r0, r1, mask, nullptr);
    return;
  }
  const int64_t units = ((int64_t)(r1 - r0) + cfg_rows(CFG) - 1) / cfg_rows(CFG);
  if constexpr (!FIRST && CMASK < 0 && sizeof(T) == 8) {
    if (dot) {
      auto k = k_gs_phase<T, TR, FIRST, CFG, CMASK, cfg_sched(CFG), cfg_rows(CFG), true>;
      int g = grid_of(c, k, units);
      if (g > kDotStride) g = kDotStride;
      k<<<g, kThreads, 0, c->stream>>>(val, cols_of<T>(L), L.pitch, rhs, x, r0, r1, mask, dot);
      return;
    }
  }
  auto k = k_gs_phase<T, TR, FIRST, CFG, CMASK>;
  k<<<grid_of(c, k, units), kThreads, 0, c->stream>>>(val, cols_of<T>(L), L.pitch, rhs, x, r0, r1, mask, nullptr);
}

// A configuration with R contiguous rows per thread needs the row range to start
// on a multiple of R (vector loads); otherwise the scalar configuration 1 runs.
// Interleaved rows need no alignment.
inline int usable_cfg(int cfg, int r0) {
  if (cfg >= kGeoCfg) return kBulkCfg;  // (no columns from the grid: see gs_dispatch, gs_first_dispatch)
  return cfg_tiled(cfg) || cfg_interleaved(cfg) || r0 % cfg_rows(cfg) == 0 ? cfg : 1;
}

// k_gs_geo over rows [r0, r1) of one colour block.
template <typename T, typename TR>
void gs_geo_launch(Context* c, const Level& L, const T* val, const TR* rhs, T* x, int r0, int r1, double* dot) {
  const GeoPhase& geo = L.geo_cols->block[sweep_at(L, r0)];
  if constexpr (sizeof(T) == 8) {
    if (dot) {
      auto k = k_gs_geo<T, TR, true>;
      const int g = std::min(grid_of(c, k, r1 - r0), kDotStride);
      launch_early(c->stream, k, g, kThreads, 0, val, L.pitch, rhs, x, r0, r1, sink_of(L), dot, geo);
      return;
    }
  }
  auto k = k_gs_geo<T, TR, false>;
  launch_early(c->stream, k, grid_of(c, k, r1 - r0), kThreads, 0, val, L.pitch, rhs, x, r0, r1, sink_of(L), nullptr,
               geo);
}

template <typename T, typename TR, bool FIRST>
void gs_dispatch(Context* c, const Level& L, int cfg, const T* val, const TR* rhs, T* x, int r0, int r1,
                 uint32_t mask, double* dot = nullptr) {
  if constexpr (!FIRST) {
    if (cfg == kGeoCfg && mask == kAllSlots && L.geo_cols) {
      if (r1 > r0) gs_geo_launch<T, TR>(c, L, val, rhs, x, r0, r1, dot);
      return;
    }
  }
  switch (usable_cfg(cfg, r0)) {
    case 0: gs_launch<T, TR, FIRST, 0>(c, L, val, rhs, x, r0, r1, mask, dot); break;
    case 1: gs_launch<T, TR, FIRST, 1>(c, L, val, rhs, x, r0, r1, mask, dot); break;
    case 2: gs_launch<T, TR, FIRST, 2>(c, L, val, rhs, x, r0, r1, mask, dot); break;
    case 3: gs_launch<T, TR, FIRST, 3>(c, L, val, rhs, x, r0, r1, mask, dot); break;
    case 4: gs_launch<T, TR, FIRST, 4>(c, L, val, rhs, x, r0, r1, mask, dot); break;
    case 5: gs_launch<T, TR, FIRST, 5>(c, L, val, rhs, x, r0, r1, mask, dot); break;
    case 6: gs_launch<T, TR, FIRST, 6>(c, L, val, rhs, x, r0, r1, mask, dot); break;
    case 7: gs_launch<T, TR, FIRST, 7>(c, L, val, rhs, x, r0, r1, mask, dot); break;
    case 8: gs_launch<T, TR, FIRST, 8>(c, L, val, rhs, x, r0, r1, mask, dot); break;
    case 9: gs_launch<T, TR, FIRST, 9>(c, L, val, rhs, x, r0, r1, mask, dot); break;
    default: gs_launch<T, TR, FIRST, 10>(c, L, val, rhs, x, r0, r1, mask, dot); break;
  }
}

// A first-sweep phase at sweep position s with its mask compiled in (plain
// configurations; the staged ones take the mask at run time).
template <typename T, typename TR, int CFG>
void gs_first_const(Context* c, const Level& L, const T* val, const TR* rhs, T* x, int r0, int r1, int s) {
  switch (s) {
    case 0: gs_launch<T, TR, true, CFG, first_mask_default(0)>(c, L, val, rhs, x, r0, r1, 0); break;
    case 1: gs_launch<T, TR, true, CFG, first_mask_default(1)>(c, L, val, rhs, x, r0, r1, 0); break;
    case 2: gs_launch<T, TR, true, CFG, first_mask_default(2)>(c, L, val, rhs, x, r0, r1, 0); break;
    case 3: gs_launch<T, TR, true, CFG, first_mask_default(3)>(c, L, val, rhs, x, r0, r1, 0); break;
    case 4: gs_launch<T, TR, true, CFG, first_mask_default(4)>(c, L, val, rhs, x, r0, r1, 0); break;
    case 5: gs_launch<T, TR, true, CFG, first_mask_default(5)>(c, L, val, rhs, x, r0, r1, 0); break;
    case 6: gs_launch<T, TR, true, CFG, first_mask_default(6)>(c, L, val, rhs, x, r0, r1, 0); break;
    default: gs_launch<T, TR, true, CFG, first_mask_default(7)>(c, L, val, rhs, x, r0, r1, 0); break;
  }
}

// The same on k_gs_first_geo with R rows a thread.
template <typename T, typename TR, int R, int S>
void gs_first_geo_at(Context* c, const Level& L, const T* val, const TR* rhs, T* x, int r0, int r1) {
  if (r1 <= r0) return;
  auto k = k_gs_first_geo<T, TR, first_mask_default(S), R>;
  const int64_t units = ((int64_t)r1 - r0 + R - 1) / R;
  launch_early(c->stream, k, grid_of(c, k, units), kThreads, 0, val, L.pitch, rhs, x, r0, r1, sink_of(L),
               L.geo_cols->block[S]);
}
template <typename T, typename TR, int R>
void gs_first_geo(Context* c, const Level& L, const T* val, const TR* rhs, T* x, int r0, int r1, int s) {
  switch (s) {
    case 0: gs_first_geo_at<T, TR, R, 0>(c, L, val, rhs, x, r0, r1); break;
    case 1: gs_first_geo_at<T, TR, R, 1>(c, L, val, rhs, x, r0, r1); break;
    case 2: gs_first_geo_at<T, TR, R, 2>(c, L, val, rhs, x, r0, r1); break;
    case 3: gs_first_geo_at<T, TR, R, 3>(c, L, val, rhs, x, r0, r1); break;
    case 4: gs_first_geo_at<T, TR, R, 4>(c, L, val, rhs, x, r0, r1); break;
    case 5: gs_first_geo_at<T, TR, R, 5>(c, L, val, rhs, x, r0, r1); break;
    case 6: gs_first_geo_at<T, TR, R, 6>(c, L, val, rhs, x, r0, r1); break;
    default: gs_first_geo_at<T, TR, R, 7>(c, L, val, rhs, x, r0, r1); break;
  }
}

// The first sweep of the default sweep order with compile-time masks; other
// configurations take the mask at run time.
template <typename T, typename TR>
void gs_first_dispatch(Context* c, const Level& L, int cfg, const T* val, const TR* rhs, T* x, int r0, int r1,
                       int s, uint32_t mask) {
  bool default_order = true;
  for (int i = 0; i < kColours; ++i) default_order = default_order && L.g.sweep[i] == kSweepDefault[i];
  if (cfg >= kGeoCfg && default_order && L.geo_cols) {
    if (cfg == kGeoCfg)
      gs_first_geo<T, TR, 1>(c, L, val, rhs, x, r0, r1, s);
    else
      gs_first_geo<T, TR, 2>(c, L, val, rhs, x, r0, r1, s);
    return;
  }
  const int u = usable_cfg(cfg, r0);
  if (default_order && (u == 0 || u == 1 || u == 4 || u == 5 || u == 7 || u == 8 || cfg_tiled(u))) {
    switch (u) {
      case 0: gs_first_const<T, TR, 0>(c, L, val, rhs, x, r0, r1, s); return;
      case 1: gs_first_const<T, TR, 1>(c, L, val, rhs, x, r0, r1, s); return;
      case 4: gs_first_const<T, TR, 4>(c, L, val, rhs, x, r0, r1, s); return;
      case 5: gs_first_const<T, TR, 5>(c, L, val, rhs, x, r0, r1, s); return;
      case 7: gs_first_const<T, TR, 7>(c, L, val, rhs, x, r0, r1, s); return;
      case 8: gs_first_const<T, TR, 8>(c, L, val, rhs, x, r0, r1, s); return;
      case 9: gs_first_const<T, TR, 9>(c, L, val, rhs, x, r0, r1, s); return;
      default: gs_first_const<T, TR, 10>(c, L, val, rhs, x, r0, r1, s); return;
    }
  }
  gs_dispatch<T, TR, true>(c, L, cfg, val, rhs, x, r0, r1, mask);
}

// Slab order (ORDER 2) needs even grid dimensions and slab runs that split into R-row groups.
inline bool slab_ok(const Level& L, int R) {
  const int per = (L.g.nx >> 1) * (L.g.ny >> 1);
  return L.g.nx % 2 == 0 && L.g.ny % 2 == 0 && L.g.nz % 2 == 0 && per % R == 0;
}

template <typename T, bool DOT, int CFG, int ORDER>
int spmv_launch_o(Context* c, const Level& L, const T* val, const T* x, T* y, double* partials) {
  auto k = k_spmv<T, DOT, CFG, ORDER>;
  const int r = ORDER == 1 ? 1 : cfg_rows(CFG);
  const int g = grid_of(c, k, ((int64_t)L.n + r - 1) / r);
  k<<<g, kThreads, 0, c->stream>>>(L.g, val, cols_of<T>(L), L.pitch, x, y, L.n, partials);
  return g;
}

template <typename T, bool DOT, int CFG>
int spmv_launch(Context* c, const Level& L, const T* val, const T* x, T* y, double* partials) {
  if (L.mv_order == 1) return spmv_launch_o<T, DOT, CFG, 1>(c, L, val, x, y, partials);
  if (L.mv_order == 2 && slab_ok(L, cfg_rows(CFG))) return spmv_launch_o<T, DOT, CFG, 2>(c, L, val, x, y, partials);
  return spmv_launch_o<T, DOT, CFG, 0>(c, L, val, x, y, partials);
}

// Slab-order tiles of the bulk SpMV: slab runs of whole tiles, colour blocks on
// even rows (the tensor copy's row coordinate times 8 bytes on 16).
inline bool bulk_slab_ok(const Level& L) {
  if (!slab_ok(L, kBulkRows)) return false;
  for (int s = 0; s < kColours; ++s)
    if (L.g.start[s] % 2) return false;
  return true;
}

template <typename T, bool DOT, int ORDER, int PW>
int spmv_bulk_launch(Context* c, const Level& L, const T* val, const T* x, T* y, double* partials,
                     const BulkMaps* m) {
  auto k = k_spmv_bulk<T, DOT, ORDER, PW>;
  using Shape = SpmvShape<T, PW>;
  constexpr int smem = Shape::smem;
  static std::atomic<uint64_t> attr_set{0};  // devices on which the shared-memory size is enabled
  bulk_attr(k, smem, c->device, &attr_set);
  const int64_t tiles = ((int64_t)L.n + kBulkRows - 1) / kBulkRows;
  const int g = (int)std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)c->sms));
  static const GeoGrid none{};
  const GeoGrid& geo = PW == kPackGeo ? *L.geo_cols : none;
  launch_early(c->stream, k, g, Shape::threads, smem, L.g, val, cols_of<T>(L), L.pitch, x, y, L.n, partials, c->fault,
               m->val, m->col, (const unsigned char*)L.colp, sink_of(L), geo);
  return g;
}

// Packed columns in slab order: every slab run starts a packed tile (colour
// blocks on multiples of kBulkRows).
inline bool packed_slab_ok(const Level& L) {
  if (!L.colp) return false;
  for (int s = 0; s < kColours; ++s)
    if (L.g.start[s] % kBulkRows) return false;
  return true;
}

// SpMV configuration 7 (FP64): slab order where the tiles fit it, storage order
// otherwise (the natural order has no tile form). Returns the grid, or 0 if it
// cannot run (no tensor maps): the caller falls back.
template <typename T, bool DOT>
int spmv_bulk(Context* c, const Level& L, const T* val, const T* x, T* y, double* partials) {
  if constexpr (sizeof(T) != 8) {
    return 0;
  } else {
    const BulkMaps* m = bulk_maps(L);
    if (!m) return 0;
    if (L.mv_order == 2 && bulk_slab_ok(L)) {
      if (L.geo_cols) return spmv_bulk_launch<T, DOT, 2, kPackGeo>(c, L, val, x, y, partials, m);
      if (packed_slab_ok(L)) {
        if (L.pack == kPackDiag) return spmv_bulk_launch<T, DOT, 2, kPackDiag>(c, L, val, x, y, partials, m);
        if (L.pack == 1) return spmv_bulk_launch<T, DOT, 2, 1>(c, L, val, x, y, partials, m);
        return spmv_bulk_launch<T, DOT, 2, 2>(c, L, val, x, y, partials, m);
      }
      return spmv_bulk_launch<T, DOT, 2, 0>(c, L, val, x, y, partials, m);
    }
    if (L.geo_cols) return spmv_bulk_launch<T, DOT, 0, kPackGeo>(c, L, val, x, y, partials, m);
    if (L.pack == kPackDiag) return spmv_bulk_launch<T, DOT, 0, kPackDiag>(c, L, val, x, y, partials, m);
    if (L.pack == 1) return spmv_bulk_launch<T, DOT, 0, 1>(c, L, val, x, y, partials, m);
    if (L.pack == 2) return spmv_bulk_launch<T, DOT, 0, 2>(c, L, val, x, y, partials, m);
    return spmv_bulk_launch<T, DOT, 0, 0>(c, L, val, x, y, partials, m);
  }
}

// Launches y = A x on level L; returns the grid (the number of partials written when DOT).
template <typename T, bool DOT>
int spmv_dispatch(Context* c, const Level& L, const T* val, const T* x, T* y, double* partials) {
  switch (L.mv_sched) {
    case kBulkMvCfg: {
      const int g = spmv_bulk<T, DOT>(c, L, val, x, y, partials);
      return g > 0 ? g : spmv_launch<T, DOT, 1>(c, L, val, x, y, partials);
    }
    case 0: return spmv_launch<T, DOT, 0>(c, L, val, x, y, partials);
    case 1: return spmv_launch<T, DOT, 1>(c, L, val, x, y, partials);
    case 2: return spmv_launch<T, DOT, 2>(c, L, val, x, y, partials);
    case 3: return spmv_launch<T, DOT, 3>(c, L, val, x, y, partials);
    case 4: return spmv_launch<T, DOT, 4>(c, L, val, x, y, partials);
    case 5: return spmv_launch<T, DOT, 5>(c, L, val, x, y, partials);
    default: return spmv_launch<T, DOT, 6>(c, L, val, x, y, partials);
  }
}

template <typename T, int CFG>
void restrict_launch(Context* c, const Level& L, const T* val, const T* rf, const T* xf, T* rc, int nc) {
  auto k = k_restrict<T, CFG>;
  k<<<grid_of(c, k, nc), kThreads, 0, c->stream>>>(val, cols_of<T>(L), L.pitch, rf, xf, L.tf, L.tq, rc, nc);
}

// The restriction on the bulk-copy pipeline (SpMV configuration 7, injected rows
// in one run); false if it cannot run here.
template <typename T, int PW>
bool restrict_bulk_p(Context* c, const Level& L, const T* val, const T* rf, const T* xf, T* rc, int nc) {
  static CUtensorMap none;  // the FP32 copy takes no maps
  const CUtensorMap* tv = &none;
  const CUtensorMap* tc = &none;
  if constexpr (bulk_tensor_tile<T>()) {
    const BulkMaps* m = bulk_maps(L);
    if (!m) return false;
    tv = &m->val;
    tc = &m->col;
  }
  auto k = k_restrict_bulk<T, PW>;
  using Shape = RestrictShape<T, PW>;
  constexpr int smem = Shape::smem;
  static std::atomic<uint64_t> attr_set{0};  // devices on which the shared-memory size is enabled
  bulk_attr(k, smem, c->device, &attr_set);
  const int64_t tiles = ((int64_t)L.tf_run + nc - (L.tf_run & ~(kBulkRows - 1)) + kBulkRows - 1) / kBulkRows;
  const int g = (int)std::min<int64_t>(tiles, (int64_t)c->sms);
  GeoPhase geo{};
  if constexpr (PW == kPackGeo) geo = L.geo_cols->block[sweep_at(L, L.tf_run)];
  launch_early(c->stream, k, g, Shape::threads, smem, val, cols_of<T>(L), L.pitch, rf, xf, L.tq, rc, L.tf_run, nc,
               c->fault, *tv, *tc, (const unsigned char*)L.colp, sink_of(L), geo);
  return true;
}

template <typename T>
bool restrict_bulk(Context* c, const Level& L, const T* val, const T* rf, const T* xf, T* rc, int nc) {
  if (L.tf_run < 0 || nc <= 0) return false;
  if (L.geo_cols && L.geo_f2c) return restrict_bulk_p<T, kPackGeo>(c, L, val, rf, xf, rc, nc);
  if (L.pack == kPackDiag) return restrict_bulk_p<T, kPackDiag>(c, L, val, rf, xf, rc, nc);
  if (L.pack == 1) return restrict_bulk_p<T, 1>(c, L, val, rf, xf, rc, nc);
  if (L.pack == 2) return restrict_bulk_p<T, 2>(c, L, val, rf, xf, rc, nc);
  return restrict_bulk_p<T, 0>(c, L, val, rf, xf, rc, nc);
}

template <typename T>
void restrict_dispatch(Context* c, const Level& L, const T* val, const T* rf, const T* xf, T* rc, int nc) {
  if (L.mv_sched == kBulkMvCfg && restrict_bulk<T>(c, L, val, rf, xf, rc, nc)) return;
  switch (L.mv_sched) {  // scalar configurations only: the transfer pairs need not be contiguous
    case 0: case 4: restrict_launch<T, 0>(c, L, val, rf, xf, rc, nc); break;
    case 2: restrict_launch<T, 2>(c, L, val, rf, xf, rc, nc); break;
    case 3: restrict_launch<T, 3>(c, L, val, rf, xf, rc, nc); break;
    default: restrict_launch<T, 1>(c, L, val, rf, xf, rc, nc); break;
  }
}

template <typename T, typename TR>
int launch_phase(Context* c, const Level& L, const T* val, const TR* rhs, T* x, int s, bool first, bool top,
                 double* dot = nullptr) {
  const int r0 = L.g.start[s], r1 = L.g.start[s + 1];
  if (r1 <= r0) return HPCG_B200_OK;
  const int kind = !top ? -1
                   : sizeof(T) == 4 ? (first ? kProfGs32First : kProfGs32Full)
                                    : (first ? kProfGsFirst : kProfGsFull);
  cudaEvent_t ev0 = nullptr;
  HB_TRY(prof_begin(c, kind, &ev0));
  const int at = first ? (sizeof(T) == 4 ? L.gs_first32_at[s] : L.gs_first_at[s]) : -1;
  const int cfg = at >= 0 ? at
                  : sizeof(T) == 4 ? (first ? L.gs_first32 : L.gs_sched32) : first ? L.gs_first : L.gs_sched;
  if (first)
    gs_first_dispatch<T, TR>(c, L, cfg, val, rhs, x, r0, r1, s, first_mask(L.g, s));
  else
    gs_dispatch<T, TR, false>(c, L, cfg, val, rhs, x, r0, r1, kAllSlots, dot);
  HB_CK(cudaGetLastError());
  return prof_end(c, kind, ev0, r1 - r0);
}

// The wavefront sweeps of level L (wave.cuh): their geometry and the per-unit
// counters, set up once. A level whose colour blocks do not cut into whole
// 128-row tiles per z pair (odd sides, or (nx/2)(ny/2) not a multiple of 128)
// gets none (wf_tpu stays 0). Phase j of a sweep runs `lag` z pairs behind
// phase j - 1 (2, or HPCG_B200_WAVE_LAG).
int ensure_wavefront(Level& L) {
  if (L.wf_tpu != 0) return HPCG_B200_OK;
  const ColourGrid& g = L.g;
  const int64_t per = (int64_t)(g.nx / 2) * (g.ny / 2);
  if (g.nx % 2 || g.ny % 2 || g.nz % 2 || per % kBulkRows || per == 0 || (int64_t)L.n != per * 4 * g.nz) {
    L.wf_tpu = -1;  // not eligible; not asked again
    return HPCG_B200_OK;
  }
  static const int lag = [] {
    const char* e = std::getenv("HPCG_B200_WAVE_LAG");
    const int v = e && *e ? std::atoi(e) : 2;
    return v < 1 ? 1 : v > 16 ? 16 : v;
  }();
  for (int dir = 0; dir < 2; ++dir) {
    WaveGeom& w = L.wf_geom[dir];
    w.H = g.nz / 2;
    w.P = dir == 0 ? kColours : kColours - 1;  // the backward sweep skips the turn colour
    w.lag = lag;
    w.tpu = (int)(per / kBulkRows);
    w.per = (int)per;
    // the phases that write each colour's final value add r'x: the forward
    // sweep's last, every phase of the backward sweep
    w.dot_from = dir == 0 ? w.P - 1 : 0;
    w.self_dep = -1;
    for (int j = 0; j < kColours; ++j) w.start[j] = j < w.P ? g.start[dir == 0 ? j : kColours - 2 - j] : 0;
  }
  HB_CK(cudaMalloc(&L.wf_done, sizeof(unsigned) * wave_units(L.wf_geom[0])));
  L.wf_tpu = (int)(per / kBulkRows);
  return HPCG_B200_OK;
}

// One sweep of level L as one cooperative launch of k_gs_wave over geometry w
// (x entering nonzero). dot: as gs_colour's, the block partials of the sweep's
// final-value rows (the caller's zeroed slots). false: not launched (no
// tensor maps, or the launch was refused): the caller runs the phases one by
// one.
template <int PW>
bool wave_launch_p(Context* c, const Level& L, const double* rhs, double* x, const WaveGeom& w, double* dot,
                   unsigned long long limit_ns = kBulkWaitNs) {
  const BulkMaps* m = bulk_maps(L);
  if (!m) return false;
  auto k = k_gs_wave<double, PW>;
  using Shape = WaveShape<double, PW>;
  constexpr int smem = Shape::smem;
  constexpr int threads = wave_threads<double, PW>();
  static std::atomic<uint64_t> attr_set{0};  // devices on which the shared-memory size is enabled
  bulk_attr(k, smem, c->device, &attr_set);
  const int nunits = wave_units(w);
  const int64_t ntiles = (int64_t)w.H * w.P * w.tpu;  // the non-empty units' tiles
  int g = (int)std::min<int64_t>(ntiles, (int64_t)c->sms);
  if (dot && g > kDotStride) g = kDotStride;
  if (cudaMemsetAsync(L.wf_done, 0, sizeof(unsigned) * nunits, c->stream) != cudaSuccess) {
    set_error("wavefront counters", cudaGetLastError());
    return false;
  }
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(g);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;  // every block resident: the sweep's waits always end
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k, (const double*)L.val, cols_of<double>(L), L.pitch, rhs, x, w,
                                           L.wf_done, dot, c->fault, m->val, m->col, (const unsigned char*)L.colp,
                                           sink_of(L), limit_ns);
  if (e != cudaSuccess) {
    set_error("k_gs_wave", e);
    cudaGetLastError();
    return false;
  }
  return true;
}

bool wave_launch(Context* c, const Level& L, const double* rhs, double* x, const WaveGeom& w, double* dot,
                 unsigned long long limit_ns = kBulkWaitNs) {
  if (L.wf_tpu <= 0) return false;
  if (L.pack == kPackDiag) return wave_launch_p<kPackDiag>(c, L, rhs, x, w, dot, limit_ns);
  if (L.pack == 1) return wave_launch_p<1>(c, L, rhs, x, w, dot, limit_ns);
  if (L.pack == 2) return wave_launch_p<2>(c, L, rhs, x, w, dot, limit_ns);
  return wave_launch_p<0>(c, L, rhs, x, w, dot, limit_ns);
}

// One launch of k_stream_probe over every tile of L (hpcg_b200_stream_probe).
template <int PW>
int stream_probe_p(Context* c, const Level& L, float* ms, double* bytes) {
  const BulkMaps* m = bulk_maps(L);
  if (!m) return HPCG_B200_ERR_UNSUPPORTED;
  auto k = k_stream_probe<PW>;
  using Shape = GsShape<double, PW>;
  static std::atomic<uint64_t> attr_set{0};
  bulk_attr(k, Shape::smem, c->device, &attr_set);
  const int ntiles = (int)(((int64_t)L.n + kBulkRows - 1) / kBulkRows);
  const int g = std::min(ntiles, c->sms);
  cudaEvent_t ev[2] = {nullptr, nullptr};
  cudaError_t e = cudaEventCreate(&ev[0]);
  if (e == cudaSuccess) e = cudaEventCreate(&ev[1]);
  if (e == cudaSuccess) e = cudaEventRecord(ev[0], c->stream);
  if (e == cudaSuccess) {
    k<<<g, Shape::threads, Shape::smem, c->stream>>>(L.val, L.col, L.pitch, ntiles, c->fault, m->val, m->col,
                                                       (const unsigned char*)L.colp);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaEventRecord(ev[1], c->stream);
  int st = e == cudaSuccess ? stream_sync(c) : status_of(e);
  if (e != cudaSuccess) set_error("k_stream_probe", e);
  if (st == HPCG_B200_OK && cudaEventElapsedTime(ms, ev[0], ev[1]) != cudaSuccess) st = HPCG_B200_ERR_CUDA;
  for (cudaEvent_t x : ev)
    if (x) cudaEventDestroy(x);
  *bytes = (double)ntiles * (Shape::value_bytes + Shape::col_bytes);
  return st;
}

// A whole sweep as one wavefront launch, timed as kProfGsSweep on level 0.
// false: not launched (see wave_launch).
template <typename T, typename TR>
bool wave_sweep(Context* c, const Level& L, const T* val, const TR* rhs, T* x, int dir, bool top, double* dot,
                int* status) {
  *status = HPCG_B200_OK;
  if constexpr (sizeof(T) != 8 || sizeof(TR) != 8) {
    return false;
  } else {
    if (!L.wf || L.wf_tpu <= 0 || val != L.val) return false;
    const int kind = top ? kProfGsSweep : -1;
    cudaEvent_t ev0 = nullptr;
    if ((*status = prof_begin(c, kind, &ev0)) != HPCG_B200_OK) return true;
    const WaveGeom& w = L.wf_geom[dir];
    if (!wave_launch(c, L, rhs, x, w, dot)) {
      if (ev0) c->ev_pool.push_back(ev0);  // recorded around no launch: back to the pool, not timed
      return false;
    }
    const int64_t rows = (int64_t)w.H * w.P * w.per;
    *status = prof_end(c, kind, ev0, rows);
    return true;
  }
}

// One symmetric Gauss-Seidel step in colour order: forward over the sweep
// positions, then backward. The last non-empty colour of the forward sweep is
// not repeated at the start of the backward sweep: its rows read only other
// colours, none of which changed in between, so a repeat would rewrite the
// same bits. first: x enters as zero (ComputeMG_ref.cpp:42).
// dot (x entering nonzero only): the phase that writes each colour's final
// value (the last colour's forward phase, every other colour's backward phase)
// also writes r'x block partials at dot + kDotStride * (sweep position); the
// caller zeroes the kColours * kDotStride slots first.
// With L.wf (FP64, whole-tile z pairs) each sweep that does not start from
// x = 0 is one wavefront launch instead (wave.cuh: the same bits); its r'x
// partials go to the slot of the forward sweep's last position, or of
// position 0 for the backward sweep.
template <typename T, typename TR>
int gs_colour(Context* c, const Level& L, const T* val, const TR* rhs, T* x, bool first, bool top,
              double* dot = nullptr) {
  int last = -1;
  for (int s = 0; s < kColours; ++s)
    if (L.g.start[s + 1] > L.g.start[s]) last = s;
  int st = HPCG_B200_OK;
  if (first || !wave_sweep<T, TR>(c, L, val, rhs, x, 0, top, dot ? dot + (int64_t)kDotStride * last : nullptr, &st)) {
    HB_TRY(st);
    for (int s = 0; s < kColours; ++s)
      HB_TRY((launch_phase<T, TR>(c, L, val, rhs, x, s, first, top,
                                  dot && !first && s == last ? dot + (int64_t)kDotStride * s : nullptr)));
  }
  HB_TRY(st);
  if (!wave_sweep<T, TR>(c, L, val, rhs, x, 1, top, dot, &st)) {
    HB_TRY(st);
    for (int s = last - 1; s >= 0; --s)
      HB_TRY((launch_phase<T, TR>(c, L, val, rhs, x, s, false, top, dot ? dot + (int64_t)kDotStride * s : nullptr)));
  }
  return st;
}

// Wavefronts ix + 2 iy + 4 iz: every lower neighbour (in the reference's natural
// order) of a row lies on an earlier wavefront, every upper one on a later one.
int ensure_waves(Level& L) {
  if (L.wave_rows) return HPCG_B200_OK;
  const ColourGrid& g = L.g;
  const int nw = (g.nx - 1) + 2 * (g.ny - 1) + 4 * (g.nz - 1) + 1;
  std::vector<int> count(nw + 1, 0), rows(L.n);
  std::vector<int> wave(L.n);
  for (int q = 0; q < L.n; ++q) {
    int ix, iy, iz;
    g.coords(q, ix, iy, iz);
    wave[q] = ix + 2 * iy + 4 * iz;
    ++count[wave[q] + 1];
  }
  for (int w = 0; w < nw; ++w) count[w + 1] += count[w];
  std::vector<int> fill(count.begin(), count.end() - 1);
  for (int q = 0; q < L.n; ++q) rows[fill[wave[q]]++] = q;
  int* d = nullptr;
  HB_CK(cudaMalloc(&d, sizeof(int) * L.n));
  cudaError_t e = cudaMemcpy(d, rows.data(), sizeof(int) * L.n, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(d);
    set_error("wave upload", e);
    return status_of(e);
  }
  L.wave_rows = d;
  L.nwaves = nw;
  L.wave_start = new int[nw + 1];
  for (int w = 0; w <= nw; ++w) L.wave_start[w] = count[w];
  return HPCG_B200_OK;
}

int gs_natural(Context* c, Level& L, const double* rhs, double* x) {
  HB_TRY(ensure_waves(L));
  for (int dir = 0; dir < 2; ++dir) {
    for (int t = 0; t < L.nwaves; ++t) {
      const int w = dir == 0 ? t : L.nwaves - 1 - t;
      const int b = L.wave_start[w], cnt = L.wave_start[w + 1] - b;
      if (cnt == 0) continue;
      k_gs_rows<double><<<grid_for(c, cnt, kThreads, kPerSm), kThreads, 0, c->stream>>>(
          L.val, L.col, L.pitch, rhs, x, L.wave_rows + b, cnt);
    }
  }
  HB_CK(cudaGetLastError());
  return HPCG_B200_OK;
}

// dot: see gs_colour (colour mode only).
int symgs_level(hpcg_b200_problem* p, int l, const double* rhs, double* x, bool x_is_zero, double* dot = nullptr) {
  Level& L = p->lev[l];
  Context* c = p->ctx;
  if (p->symgs_mode == HPCG_B200_SYMGS_NATURAL) {
    if (x_is_zero) HB_CK(cudaMemsetAsync(x, 0, sizeof(double) * L.n, c->stream));
    return gs_natural(c, L, rhs, x);
  }
  if (!x_is_zero && !dot && !(c->prof && l == 0) && tail_step_ok(p, l) && tail_step(p, l, rhs, x))
    return HPCG_B200_OK;
  return gs_colour<double, double>(c, L, L.val, rhs, x, x_is_zero, l == 0, dot);
}

int coarse_vcycle(hpcg_b200_problem* p, bool f32);

// ComputeMG_ref.cpp:39-63 on colour-order device vectors of level l. rtz (level
// 0, colour mode): the post-smoother also leaves the block partials of r'x in
// rtz[0 .. kColours * kDotStride), zeroed here first.
int mg_level(hpcg_b200_problem* p, int l, const double* r, double* x, double* rtz = nullptr) {
  Level& L = p->lev[l];
  Context* c = p->ctx;
  if (p->symgs_mode == HPCG_B200_SYMGS_COLOUR && !rtz && !(c->prof && l == 0) && l >= tail_first(p, false) &&
      tail_vcycle(p, l, r, x))
    return HPCG_B200_OK;
  HB_TRY(symgs_level(p, l, r, x, true));
  if (l + 1 < p->nlev) {
    Level& C = p->lev[l + 1];
    cudaEvent_t ev0 = nullptr;
    HB_TRY(prof_begin(c, l == 0 ? kProfRestrict : -1, &ev0));
    restrict_dispatch<double>(c, L, L.val, r, x, C.r, C.n);
    HB_CK(cudaGetLastError());
    HB_TRY(prof_end(c, l == 0 ? kProfRestrict : -1, ev0, C.n));
    HB_TRY(l == 0 ? coarse_vcycle(p, false) : mg_level(p, l + 1, C.r, C.x));
    HB_CK(launch_early(c->stream, k_prolong<double>, grid_for(c, C.n, kThreads, kPerSm), kThreads, 0, L.tf, L.tq, C.x,
                       x, C.n));
    if (rtz) HB_CK(cudaMemsetAsync(rtz, 0, sizeof(double) * kColours * kDotStride, c->stream));
    HB_TRY(symgs_level(p, l, r, x, false, rtz));
  }
  return HPCG_B200_OK;
}

// The CG's r'z comes out of the post-smoother (colour mode, more than one level).
// r'z from the post-smoother's partials (CG.cpp:110/113 fused into the phase
// that writes each colour's final value), except when level 0 runs the
// bulk-copy phases on 8- or 16-bit offset records: there the phases that also
// write partials measured about 12% slower than the plain ones at the same
// bytes (two consumer groups, 16-bit offsets: 0.8 ms per 512^3 iteration),
// more than a separate r'z pass over r and z (2.1 GB), so the CG runs that
// pass instead. With the diagonal form (three groups) the fused partials are
// the faster way: 32.16 against 32.79 ms per 512^3 iteration, same box.
// Read after tuning. Measurement knob HPCG_B200_RTZ: "fused" or "pass" forces
// one way (colour mode with more than one level only).
// Where the whole V-cycle is one launch (tail.cuh) the CG runs a separate pass.
bool rtz_fused(const hpcg_b200_problem* P) {
  const Level& L = P->lev[0];
  if (P->symgs_mode != HPCG_B200_SYMGS_COLOUR || P->nlev < 2) return false;
  static const int force = [] {
    const char* e = std::getenv("HPCG_B200_RTZ");
    return !e ? 0 : std::strcmp(e, "fused") == 0 ? 1 : std::strcmp(e, "pass") == 0 ? 2 : 0;
  }();
  if (force) return force == 1;
  if (!P->ctx->prof && tail_first(const_cast<hpcg_b200_problem*>(P), false) == 0) return false;
  return !(L.gs_sched == kBulkCfg && L.colp && L.pack != kPackDiag && !L.geo_cols);
}

// Autotuner, for levels that read stored columns (and, with HPCG_B200_TUNE=1,
// for those whose configurations follow from rule_config): times each kernel
// configuration (load schedule x
// registers per thread) of the Gauss-Seidel phase and of the SpMV on scratch
// vectors (Ap as x, zprev as right-hand side on level 0; the coarse r/x pair
// otherwise) and keeps the fastest. Every configuration computes the same bits,
// so the choice only affects speed. HPCG_B200_CONFIG=n forces configuration n
// (clamped to each kernel's range).
// Measurement knob HPCG_B200_LEVEL_CONFIG: the configurations of every level
// given instead of tuned, "gs,gs_first,spmv,spmv_order,gs32,gs32_first" per
// level, levels separated by ';' (a profiler run then uses the plain run's
// choices: under a profiler the tuner's timings are not the real ones). The
// two first-sweep fields may list one configuration per sweep position,
// separated by '/' (8 of them), as hpcg_b200_level_first_config reports them.
// An optional seventh field, 0 or 1, is the level's wavefront-sweep choice
// (hpcg_b200_level_wavefront). Fills v[6], *wf (-1 if absent) and the
// per-position lists at64/at32 (-1: v[1] / v[5] at every position) for level
// l; false if the variable is unset, malformed or has no such level.
bool level_config_override(int l, int v[6], int* wf, int (&at64)[kColours], int (&at32)[kColours]) {
  *wf = -1;
  const char* s = std::getenv("HPCG_B200_LEVEL_CONFIG");
  if (!s || !*s) return false;
  for (int i = 0; i < l; ++i) {
    s = std::strchr(s, ';');
    if (!s) return false;
    ++s;
  }
  for (int p = 0; p < kColours; ++p) at64[p] = at32[p] = -1;
  for (int i = 0; i < 6; ++i) {
    char* end = nullptr;
    const long x = std::strtol(s, &end, 10);
    if (end == s) return false;
    v[i] = (int)x;
    s = end;
    if ((i == 1 || i == 5) && *s == '/') {  // one configuration per sweep position
      int* at = i == 1 ? at64 : at32;
      at[0] = v[i];
      for (int p = 1; p < kColours; ++p) {
        if (*s != '/') return false;
        ++s;
        const long y = std::strtol(s, &end, 10);
        if (end == s || y < 0 || y >= kGsConfigs) return false;
        at[p] = (int)y;
        s = end;
      }
    }
    if (i < 5) {
      if (*s != ',') return false;
      ++s;
    }
  }
  const int lim[6] = {kGsFull, kGsConfigs, kConfigs, 3, kGsFull, kGsConfigs};
  for (int i = 0; i < 6; ++i)
    if (v[i] < 0 || v[i] >= lim[i]) return false;
  if (*s == ',') {
    char* end = nullptr;
    const long y = std::strtol(s + 1, &end, 10);
    if (end == s + 1 || (y != 0 && y != 1)) return false;
    *wf = (int)y;
  }
  return true;
}

// HPCG_B200_WAVE: unset or "0": no sweep runs as one wavefront launch; "1":
// every sweep does where the level allows it; "tune": the autotuner times
// both. Off unless asked for: at 512^3 the wavefront lost on every level in
// whole CG sets (levels 0 and 1 by timing; on levels 2 and 3 the tuner, which
// times launch by launch, chose it in some runs, and those CG sets ran at
// 1622 against 1647-1649 GFLOP/s with the phases, configurations otherwise
// pinned equal).
int wave_force() {
  static const int f = [] {
    const char* e = std::getenv("HPCG_B200_WAVE");
    if (!e || !*e || e[0] == '0') return 0;
    return std::strcmp(e, "tune") == 0 ? -1 : 1;
  }();
  return f;
}

// The first-sweep choice from per-position timings t[s][cfg]: the fastest
// configuration at each sweep position into at[s] (-1 for an empty colour),
// and into *one the configuration with the least time summed over the sweep
// (reported by hpcg_b200_level_config, and used where a position has none).
void pick_first(const float (&t)[kColours][kGsConfigs], int (&at)[kColours], int* one) {
  double sum[kGsConfigs] = {};
  for (int s = 0; s < kColours; ++s) {
    at[s] = -1;
    float best = 1e30f;
    for (int cfg = 0; cfg < kGsConfigs; ++cfg) {
      if (t[s][cfg] >= 1e30f) continue;
      sum[cfg] += t[s][cfg];
      if (t[s][cfg] < best) {
        best = t[s][cfg];
        at[s] = cfg;
      }
    }
  }
  int b = *one;
  for (int cfg = 0; cfg < kGsConfigs; ++cfg)
    if (sum[cfg] > 0.0 && (sum[b] <= 0.0 || sum[cfg] < sum[b])) b = cfg;
  *one = b;
}

// The configurations of a level whose columns come from the grid: on one rank
// every kernel has a form that reads the values alone, and which of them is
// fastest follows from what bounds it, so nothing is timed (timing a new
// problem's levels took 11-216 ms, and single launches of a few microseconds
// are not told apart reliably: a step of 96^3 ran in 110 or 181 us from one
// problem to the next). HPCG_B200_TUNE=1: time them all the same.
//  - phases of all slots: up to two rounds of blocks on the SMs k_gs_geo, whose
//    threads request their rows' values before the phase before has ended (a
//    symmetric step of 64^3: 55 against 62 us, 80^3: 66 against 84, 104^3: 120
//    against 130); above that the bulk-copy pipeline (128^3: 193 against 213; level
//    0 of 384^3 the more so);
//  - first-sweep phases: k_gs_first_geo, one row a thread in FP64 (384^3: 1.36 ms a
//    sweep, two rows 1.47, bulk copies 2.15, the tuner's register mix 1.53), two in
//    FP32 once the phases leave the L2 (384^3: 0.81 against 0.84 ms; 128^3: 85
//    against 83 us); the last position reads 26 of 27 slots, so there the bulk
//    copies win once the matrix comes from memory;
//  - SpMV: bulk copies, slab order once x no longer fits the L2 beside the matrix
//    stream (384^3: 1.04 ms; 128^3: 43 us, in storage order 41).
constexpr int kBeyondL2 = 4 << 20;  // rows: 32 MB a vector, 900 MB of values

// rows of a phase: two rounds of two blocks of k_gs_geo on each SM (148: 151552)
int geo_rows(const Context* c) { return 2 * 2 * c->sms * kThreads; }

bool by_rule(const Level& L) {
  const char* e = std::getenv("HPCG_B200_TUNE");
  return L.geo_cols && !(e && *e && e[0] != '0');
}

void rule_config(const Context* c, Level& L) {
  const bool large = L.n >= kBeyondL2;
  L.gs_sched = L.n / kColours <= geo_rows(c) ? kGeoCfg : kBulkCfg;
  L.gs_first = kGeoCfg;
  for (int s = 0; s < kColours; ++s) L.gs_first_at[s] = large && s == kColours - 1 ? kBulkCfg : kGeoCfg;
  L.mv_sched = kBulkMvCfg;
  L.mv_order = large ? 2 : 0;
}

void rule_config32(const Context* c, Level& L) {
  const bool large = L.n >= kBeyondL2;
  L.gs_sched32 = L.n / kColours <= geo_rows(c) ? kGeoCfg : kBulkCfg;
  L.gs_first32 = large ? kGeoCfg + 1 : kGeoCfg;
  for (int s = 0; s < kColours; ++s)
    L.gs_first32_at[s] = large && s == kColours - 1 ? kBulkCfg : L.gs_first32;
}

// small: also decide which small levels run in one launch (not for an SpMV alone).
int autotune(hpcg_b200_problem* P, bool small = true) {
  Context* c = P->ctx;
  if (small) tail_first(P, false);  // may allocate: before any capture
  const char* force = std::getenv("HPCG_B200_CONFIG");
  for (int l = 0; l < P->nlev; ++l) {
    Level& L = P->lev[l];
    if (L.tuned) continue;
    L.tuned = true;
    int ov[6], at64[kColours], at32[kColours], wf = -1;
    if (level_config_override(l, ov, &wf, at64, at32)) {
      L.gs_sched = ov[0];
      L.gs_first = ov[1];
      L.mv_sched = ov[2];
      L.mv_order = ov[3];
      for (int s = 0; s < kColours; ++s) L.gs_first_at[s] = at64[s];
      if (wf < 0) wf = wave_force() > 0 ? 1 : 0;
      if (wf) HB_TRY(ensure_wavefront(L));
      L.wf = wf && L.wf_tpu > 0 ? 1 : 0;
      continue;
    }
    if (force && *force) {
      const int f = std::atoi(force);
      L.gs_first = f < 0 ? 0 : f >= kGsConfigs ? kGsConfigs - 1 : f;
      L.gs_sched = std::min(L.gs_first, kGsFull - 1);
      L.mv_sched = f < 0 ? 0 : f >= kConfigs ? kConfigs - 1 : f;
      continue;
    }
    if (by_rule(L)) {
      rule_config(c, L);
      const char* fo = std::getenv("HPCG_B200_SPMV_ORDER");
      if (fo && *fo) L.mv_order = std::atoi(fo);
      if (wave_force() > 0) {
        HB_TRY(ensure_wavefront(L));
        L.wf = L.wf_tpu > 0 ? 1 : 0;
      }
      if (wave_force() >= 0) {
        L.mv_rule = !(fo && *fo);
        continue;
      }
    }
    double* xs = l == 0 ? P->Ap : L.x;
    double* rs = l == 0 ? P->zprev : L.r;
    double* ys = l == 0 ? P->z : L.r;  // SpMV output (coarse levels: r, rewritten before use)
    const int r0 = L.g.start[1], r1 = L.g.start[2];
    if (r1 <= r0) continue;
    cudaEvent_t e0, e1;
    HB_CK(cudaEventCreate(&e0));
    HB_CK(cudaEventCreate(&e1));
    // Repetitions run round-robin over the configurations, so that a drift of
    // the clocks during tuning (the power cap settling) biases none of them.
    const int kOrders = 3;  // SpMV row orders: storage, natural, slab
    float t_gs[kGsConfigs], t_first[kColours][kGsConfigs], t_mv[kConfigs][kOrders];
    for (int k = 0; k < kGsConfigs; ++k) {
      t_gs[k] = 1e30f;
      for (int s = 0; s < kColours; ++s) t_first[s][k] = 1e30f;
      if (k < kConfigs)
        for (int v = 0; v < kOrders; ++v) t_mv[k][v] = 1e30f;
    }
    auto time_it = [&](float& best, auto&& launch) -> int {
      HB_CK(cudaEventRecord(e0, c->stream));
      launch();
      HB_CK(cudaEventRecord(e1, c->stream));
      HB_CK(cudaEventSynchronize(e1));
      float ms = 0.f;
      HB_CK(cudaEventElapsedTime(&ms, e0, e1));
      if (ms < best) best = ms;
      return HPCG_B200_OK;
    };
    const int keep_sched = L.mv_sched, keep_order = L.mv_order;
    for (int rep = 0; rep < 4; ++rep) {
      for (int sched = 0; sched < kGsConfigs; ++sched) {
        if (sched < kGsFull) HB_TRY(time_it(t_gs[sched], [&] {
          gs_dispatch<double, double, false>(c, L, sched, L.val, rs, xs, r0, r1, kAllSlots);
        }));
        // the first-sweep phase of every sweep position (0 to 26 slots)
        for (int s = 0; s < kColours; ++s) {
          if (L.g.start[s + 1] <= L.g.start[s]) continue;
          HB_TRY(time_it(t_first[s][sched], [&] {
            gs_first_dispatch<double, double>(c, L, sched, L.val, rs, xs, L.g.start[s], L.g.start[s + 1], s,
                                              first_mask(L.g, s));
          }));
        }
        for (int v = 0; v < kOrders && sched < kConfigs; ++v) {
          if (sched == kBulkMvCfg && v == 1) continue;  // the bulk SpMV has no natural order
          L.mv_sched = sched;
          L.mv_order = v;
          // the variant CG runs: fused with the p'Ap partials
          HB_TRY(time_it(t_mv[sched][v], [&] { spmv_dispatch<double, true>(c, L, L.val, xs, ys, c->partials); }));
        }
      }
    }
    L.mv_sched = keep_sched;
    L.mv_order = keep_order;
    float best_gs = 1e30f, best_mv = 1e30f;
    for (int sched = 0; sched < kGsConfigs; ++sched) {
      if (t_gs[sched] < best_gs) { best_gs = t_gs[sched]; L.gs_sched = sched; }
      for (int v = 0; v < kOrders && sched < kConfigs; ++v)
        if (t_mv[sched][v] < best_mv) { best_mv = t_mv[sched][v]; L.mv_sched = sched; L.mv_order = v; }
    }
    pick_first(t_first, L.gs_first_at, &L.gs_first);
    const char* fo = std::getenv("HPCG_B200_SPMV_ORDER");  // measurement: force the SpMV row order
    if (fo && *fo) L.mv_order = std::atoi(fo);
    // the sweeps as wavefront launches (wave.cuh) or phase by phase: a whole
    // symmetric step from nonzero x each way, round-robin
    L.wf = 0;
    if (wave_force() != 0) HB_TRY(ensure_wavefront(L));
    if (L.wf_tpu > 0 && wave_force() > 0) {
      L.wf = 1;
    } else if (L.wf_tpu > 0 && wave_force() < 0) {
      float t_wf[2] = {1e30f, 1e30f};
      for (int rep = 0; rep < 3; ++rep)
        for (int w = 0; w < 2; ++w) {
          L.wf = w;
          HB_TRY(time_it(t_wf[w], [&] { gs_colour<double, double>(c, L, L.val, rs, xs, false, false); }));
        }
      L.wf = t_wf[1] < t_wf[0] ? 1 : 0;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    HB_CK(cudaGetLastError());
  }
  return HPCG_B200_OK;
}

int finalize(Context* c, int nparts, int op, double* out = nullptr) {
  if (nparts == kWideParts && op != kFinMax && op != kFinFlex)
    HB_CK(launch_early(c->stream, k_finalize_wide, 1, kWideThreads, 0, c->partials, op, c->scal, out));
  else
    HB_CK(launch_early(c->stream, k_finalize, 1, kThreads, 0, c->partials, nparts, op, c->scal, out));
  return HPCG_B200_OK;
}

int read_scalars(Context* c) {
  HB_CK(cudaMemcpyAsync(c->scal_host, c->scal, sizeof(Scalars), cudaMemcpyDeviceToHost, c->stream));
  HB_TRY(stream_sync(c));
  return HPCG_B200_OK;
}

struct Setter {  // selects the problem's device for the duration of a call
  int prev = -1;
  explicit Setter(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    if (prev != dev) cudaSetDevice(dev);
  }
  ~Setter() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

double now_s() {
  return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

// ---- the CG loop as one CUDA graph ------------------------------------------

bool graph_enabled() {
  const char* e = std::getenv("HPCG_B200_GRAPH");
  return !(e && e[0] == '0');
}

int mg32_level(hpcg_b200_problem* p, int l, const float* r, float* x);

// Runs `direct` (launches on c's stream, the same ones every time) as one graph
// launch once it has been captured into ex; inside a capture, with graphs off
// or refused, in the natural-order mode and under the launch profiler directly.
// The capture is on a stream of its own, through a copy of the context that only
// this problem sees: the context's stream is every problem's on the GPU, and a call
// of another thread would be recorded into the graph, or end the capture by waiting.
template <typename F>
int run_captured(hpcg_b200_problem* p, cudaGraphExec_t& ex, F&& direct) {
  Context* c = p->ctx;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  HB_CK(cudaStreamIsCapturing(c->stream, &cs));
  if (cs != cudaStreamCaptureStatusNone || p->coarse_graph_failed || !graph_enabled() || c->prof ||
      p->symgs_mode != HPCG_B200_SYMGS_COLOUR)
    return direct();
  if (!ex) {
    Context rec;
    rec.device = c->device;
    rec.sms = c->sms;
    rec.partials = c->partials;
    rec.scal = c->scal;
    rec.scal_host = c->scal_host;
    rec.fault = c->fault;
    if (take_recorder(c, &rec.stream) != HPCG_B200_OK) {
      cudaGetLastError();
      return direct();
    }
    cudaGraph_t g = nullptr;
    int st = HPCG_B200_OK;
    cudaError_t e = cudaStreamBeginCapture(rec.stream, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      p->ctx = &rec;
      st = direct();
      p->ctx = c;
      e = cudaStreamEndCapture(rec.stream, &g);
    }
    if (st == HPCG_B200_OK && e == cudaSuccess) e = cudaGraphInstantiate(&ex, g, 0);
    if (g) cudaGraphDestroy(g);
    give_recorder(c, rec.stream);
    if (st != HPCG_B200_OK || e != cudaSuccess) {  // refused: stream launches from now on
      cudaGetLastError();
      ex = nullptr;
      p->coarse_graph_failed = true;
      return direct();
    }
  }
  HB_CK(cudaGraphLaunch(ex, c->stream));
  return HPCG_B200_OK;
}

// The V-cycle below level 0 (levels 1 .. nlev-1 between the level-0 restriction
// and prolongation, on the fixed coarse vectors r, x of level 1) for the loops
// that launch kernel by kernel: one graph launch instead of one launch for each
// of its small kernels (a single launch already where tail.cuh runs them all).
// The same kernels either way, so the same bits.
int coarse_vcycle(hpcg_b200_problem* p, bool f32) {
  auto direct = [&]() -> int {
    return f32 ? mg32_level(p, 1, p->lev[1].r32, p->lev[1].x32) : mg_level(p, 1, p->lev[1].r, p->lev[1].x);
  };
  if (tail_first(p, f32) <= 1) return direct();
  return run_captured(p, p->coarse_graph[f32 ? 1 : 0], direct);
}

// A V-cycle or step on the problem's own level-0 vectors, as one graph launch
// from its second use on (a launch costs the host 2-3 us, as long as a small
// phase runs; a capture costs about what one pass does, so a single use is
// not captured).
template <typename F>
int run_cycle(hpcg_b200_problem* p, CycleKind kind, F&& direct) {
  if (tail_first(p, kind == kCycleMg32) == 0 && kind != kCycleStep) return direct();  // one launch
  if (p->cycle_uses[kind] < 1) {
    ++p->cycle_uses[kind];
    return direct();
  }
  return run_captured(p, p->cycle_graph[kind], direct);
}

int mg_cycle(hpcg_b200_problem* p) {
  return run_cycle(p, kCycleMg, [&] { return mg_level(p, 0, p->r, p->z); });
}
int mg32_cycle(hpcg_b200_problem* p) {
  return run_cycle(p, kCycleMg32, [&] { return mg32_level(p, 0, p->lev[0].r32, p->lev[0].x32); });
}

// One CG iteration (CG.cpp:101-125) with the iteration-aware kernels: the body
// of the graph's while node.
int cg_iteration_body(hpcg_b200_problem* P, bool prec) {
  const Level& L = P->lev[0];
  Context* c = P->ctx;
  const int n = L.n;
  const int nb = red_blocks(c, n);
  const int gv = grid_for(c, n, kThreads, kPerSm);
  if (prec && rtz_fused(P)) {
    HB_TRY(mg_level(P, 0, P->r, P->z, c->partials));
    HB_TRY(finalize(c, kColours * kDotStride, kFinRtzIter));
  } else {
    if (prec) {
      HB_TRY(mg_level(P, 0, P->r, P->z));
    } else {
      HB_CK(cudaMemcpyAsync(P->z, P->r, sizeof(double) * n, cudaMemcpyDeviceToDevice, c->stream));
    }
    HB_CK(launch_early(c->stream, k_dot<false>, nb, kThreads, 0, n, P->r, P->z, nullptr, c->partials));
    HB_TRY(finalize(c, nb, kFinRtzIter));
  }
  // with x of the last iteration
  HB_CK(launch_early(c->stream, k_update_px_iter, gv, kThreads, 0, n, P->z, P->p, P->x, c->scal));
  const int gs = spmv_dispatch<double, true>(c, L, L.val, P->p, P->Ap, c->partials);
  HB_CK(cudaGetLastError());
  HB_TRY(finalize(c, gs, kFinPap));
  HB_CK(launch_early(c->stream, k_update_r, nb, kThreads, 0, n, P->r, P->Ap, c->scal, c->partials, nullptr));
  return finalize(c, nb, kFinNormr);
}

// Ends a capture begun on `st` (whether or not the captured work succeeded).
int end_capture(cudaStream_t st, int status) {
  cudaGraph_t g = nullptr;
  const cudaError_t e = cudaStreamEndCapture(st, &g);
  if (status == HPCG_B200_OK && e != cudaSuccess) {
    set_error("cudaStreamEndCapture", e);
    return status_of(e);
  }
  return status;
}

// Graph: [condition before the loop] -> while (condition) { iteration; condition }.
int build_cg_graph(hpcg_b200_problem* P, bool prec, cudaGraphExec_t* out) {
  Context* c = P->ctx;
  cudaGraph_t g = nullptr;
  HB_CK(cudaGraphCreate(&g, 0));
  int st = HPCG_B200_OK;
  cudaGraphConditionalHandle h;
  cudaError_t e = cudaGraphConditionalHandleCreate(&h, g, 0, cudaGraphCondAssignDefault);
  if (e != cudaSuccess) {
    cudaGraphDestroy(g);
    set_error("cudaGraphConditionalHandleCreate", e);
    return status_of(e);
  }
  e = cudaStreamBeginCaptureToGraph(c->stream, g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    k_cg_condition<<<1, 32, 0, c->stream>>>(c->scal, h, 0);
    e = cudaGetLastError();
    st = end_capture(c->stream, e == cudaSuccess ? HPCG_B200_OK : status_of(e));
  }
  if (e != cudaSuccess || st != HPCG_B200_OK) {
    cudaGraphDestroy(g);
    set_error("graph capture (loop condition)", e);
    return st != HPCG_B200_OK ? st : status_of(e);
  }
  size_t num = 0;
  cudaGraphNode_t init = nullptr;
  e = cudaGraphGetNodes(g, nullptr, &num);
  if (e == cudaSuccess && num == 1) e = cudaGraphGetNodes(g, &init, &num);
  // zero-filled node parameters (the struct's union has no default constructor)
  alignas(cudaGraphNodeParams) unsigned char cp_buf[sizeof(cudaGraphNodeParams)];
  std::memset(cp_buf, 0, sizeof(cp_buf));
  cudaGraphNodeParams& cp = *reinterpret_cast<cudaGraphNodeParams*>(cp_buf);
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = h;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  cudaGraphNode_t loop = nullptr;
  if (e == cudaSuccess) e = cudaGraphAddNode(&loop, g, &init, 1, &cp);
  if (e == cudaSuccess)
    e = cudaStreamBeginCaptureToGraph(c->stream, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                      cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) {
    cudaGraphDestroy(g);
    set_error("graph while node", e);
    return status_of(e);
  }
  st = cg_iteration_body(P, prec);
  if (st == HPCG_B200_OK) {
    k_cg_condition<<<1, 32, 0, c->stream>>>(c->scal, h, 1);
    if (cudaGetLastError() != cudaSuccess) st = HPCG_B200_ERR_CUDA;
  }
  st = end_capture(c->stream, st);
  if (st == HPCG_B200_OK) {
    e = cudaGraphInstantiate(out, g, 0);
    if (e != cudaSuccess) {
      set_error("cudaGraphInstantiate", e);
      st = status_of(e);
    }
  }
  cudaGraphDestroy(g);
  return st;
}

// The whole loop of CG.cpp:100-126 as one graph launch after the preamble on
// the stream; no host round trip until the loop has ended.
int run_cg_graph(hpcg_b200_problem* P, int max_iter, double tol, bool prec, int* niters, double* normr_out,
                 double* normr0_out) {
  const Level& L = P->lev[0];
  Context* c = P->ctx;
  const int n = L.n;
  const int nb = red_blocks(c, n);
  spmv_dispatch<double, false>(c, L, L.val, P->x, P->Ap, nullptr);
  k_waxpby<true><<<nb, kThreads, 0, c->stream>>>(n, 1.0, P->b, -1.0, P->Ap, P->r, c->partials);
  HB_CK(cudaGetLastError());
  HB_TRY(finalize(c, nb, kFinNormr0));
  k_cg_setup<<<1, 32, 0, c->stream>>>(c->scal, max_iter, tol);
  HB_CK(cudaGetLastError());
  cudaGraphExec_t& ex = P->cg_graph[prec ? 1 : 0];
  if (!ex) HB_TRY(build_cg_graph(P, prec, &ex));
  HB_CK(cudaGraphLaunch(ex, c->stream));
  // the last iteration's x update (CG.cpp:121), if the loop ran one
  k_update_x<<<grid_for(c, n, kThreads, kPerSm), kThreads, 0, c->stream>>>(n, P->x, P->p, c->scal, 1);
  HB_CK(cudaGetLastError());
  HB_TRY(read_scalars(c));
  *niters = c->scal_host->iter;
  *normr_out = std::sqrt(c->scal_host->normr2);
  *normr0_out = c->scal_host->normr0;
  return HPCG_B200_OK;
}

// CG.cpp:59-143 on the resident vectors p->b, p->x (colour order).
int run_cg(hpcg_b200_problem* P, int max_iter, double tol, bool prec, int* niters, double* normr_out,
           double* normr0_out, double* times) {
  // the graph holds the colour-order kernels; the natural-order parity mode
  // (thousands of wavefront launches) runs on the stream
  if (!times && !P->ctx->prof && !P->cg_graph_failed && P->symgs_mode == HPCG_B200_SYMGS_COLOUR &&
      graph_enabled()) {
    HB_TRY(autotune(P));
    const int st = run_cg_graph(P, max_iter, tol, prec, niters, normr_out, normr0_out);
    if (st == HPCG_B200_OK) return st;
    // a refused capture leaves the vectors as the preamble left them: rerun on the stream
    P->cg_graph_failed = true;
    cudaGetLastError();
  }
  const Level& L = P->lev[0];
  Context* c = P->ctx;
  const int n = L.n;
  const int nb = red_blocks(c, n);
  const int gv = grid_for(c, n, kThreads, kPerSm);
  const double t_begin = now_s();
  std::vector<cudaEvent_t> ev;
  auto mark = [&](void) -> int {
    if (!times) return HPCG_B200_OK;
    cudaEvent_t e;
    HB_CK(cudaEventCreate(&e));
    ev.push_back(e);
    HB_CK(cudaEventRecord(e, c->stream));
    return HPCG_B200_OK;
  };
  HB_TRY(autotune(P));
  // p = x; Ap = A p; r = b - Ap; normr = sqrt(r'r)   (CG.cpp:86-90)
  spmv_dispatch<double, false>(c, L, L.val, P->x, P->Ap, nullptr);
  k_waxpby<true><<<nb, kThreads, 0, c->stream>>>(n, 1.0, P->b, -1.0, P->Ap, P->r, c->partials);
  HB_CK(cudaGetLastError());
  HB_TRY(finalize(c, nb, kFinNormr));
  HB_TRY(read_scalars(c));
  double normr = std::sqrt(c->scal_host->normr2);
  const double normr0 = normr;
  *niters = 0;
  for (int k = 1; k <= max_iter && normr / normr0 > tol; ++k) {
    HB_TRY(mark());
    const bool fused = prec && rtz_fused(P);
    if (prec) {
      HB_TRY(mg_level(P, 0, P->r, P->z, fused ? c->partials : nullptr));  // CG.cpp:103 (and r'z, :110 / :113)
    } else {
      HB_CK(cudaMemcpyAsync(P->z, P->r, sizeof(double) * n, cudaMemcpyDeviceToDevice, c->stream));  // :105
    }
    HB_TRY(mark());
    const int rz_parts = fused ? kColours * kDotStride : nb;
    if (!fused) {
      k_dot<false><<<nb, kThreads, 0, c->stream>>>(n, P->r, P->z, nullptr, c->partials);  // :110 / :113
      HB_CK(cudaGetLastError());
    }
    if (k == 1) {
      HB_TRY(finalize(c, rz_parts, kFinRtzFirst));
      HB_CK(cudaMemcpyAsync(P->p, P->z, sizeof(double) * n, cudaMemcpyDeviceToDevice, c->stream));  // :109
    } else {
      HB_TRY(finalize(c, rz_parts, kFinRtz));
      k_update_px<<<gv, kThreads, 0, c->stream>>>(n, P->z, P->p, P->x, c->scal);  // :115, and :121 of k - 1
      HB_CK(cudaGetLastError());
    }
    HB_TRY(mark());
    cudaEvent_t ev0 = nullptr;
    HB_TRY(prof_begin(c, kProfSpmv, &ev0));
    const int gs = spmv_dispatch<double, true>(c, L, L.val, P->p, P->Ap, c->partials);
    HB_CK(cudaGetLastError());
    HB_TRY(prof_end(c, kProfSpmv, ev0, n));
    HB_TRY(finalize(c, gs, kFinPap));                                       // :118-120
    HB_TRY(mark());
    k_update_r<<<nb, kThreads, 0, c->stream>>>(n, P->r, P->Ap, c->scal, c->partials);  // :122-123 (x: next :115)
    HB_CK(cudaGetLastError());
    HB_TRY(finalize(c, nb, kFinNormr));
    HB_TRY(mark());
    HB_TRY(read_scalars(c));
    normr = std::sqrt(c->scal_host->normr2);
    *niters = k;
  }
  if (*niters > 0) {  // the last iteration's x update (CG.cpp:121)
    k_update_x<<<gv, kThreads, 0, c->stream>>>(n, P->x, P->p, c->scal, 0);
    HB_CK(cudaGetLastError());
  }
  *normr_out = normr;
  *normr0_out = normr0;
  if (c->prof) HB_TRY(prof_flush(c));
  if (times) {
    HB_TRY(stream_sync(c));
    double t_mg = 0, t_dw = 0, t_spmv = 0, t_up = 0;
    for (size_t i = 0; i + 4 < ev.size(); i += 5) {
      float a, b2, d, e;
      cudaEventElapsedTime(&a, ev[i], ev[i + 1]);
      cudaEventElapsedTime(&b2, ev[i + 1], ev[i + 2]);
      cudaEventElapsedTime(&d, ev[i + 2], ev[i + 3]);
      cudaEventElapsedTime(&e, ev[i + 3], ev[i + 4]);
      t_mg += a * 1e-3; t_dw += b2 * 1e-3; t_spmv += d * 1e-3; t_up += e * 1e-3;
    }
    for (cudaEvent_t e : ev) cudaEventDestroy(e);
    times[1] += 0.5 * (t_dw + t_up);  // dot products (fused with the vector updates)
    times[2] += 0.5 * (t_dw + t_up);  // WAXPBY
    times[3] += t_spmv;
    times[5] += t_mg;
    times[0] += now_s() - t_begin;
  }
  return HPCG_B200_OK;
}


// ---- FP32 V-cycle ----------------------------------------------------------

// FP32 copies of the values and FP32 work vectors of every level (first use).
int ensure_f32(hpcg_b200_problem* P) {
  Context* c = P->ctx;
  for (int l = 0; l < P->nlev; ++l) {
    Level& L = P->lev[l];
    if (!L.val32 || !L.col32) {
      const int64_t cnt = blocked_entries(L.pitch, kRowBlock32);
      if (!L.val32) HB_TRY(dev_alloc((void**)&L.val32, sizeof(float) * cnt, &P->bytes));
      L.old32 = true;
      HB_TRY(dev_alloc((void**)&L.col32, sizeof(int) * cnt, &P->bytes));
      HB_CK(cudaMemsetAsync(L.val32, 0, sizeof(float) * cnt, c->stream));
      HB_CK(cudaMemsetAsync(L.col32, 0, sizeof(int) * cnt, c->stream));
    }
    if (L.old32) {
      k_block32<<<grid_for(c, (int64_t)kSlots * L.pitch, kThreads, kPerSm), kThreads, 0, c->stream>>>(
          L.val, L.col, L.pitch, L.val32, L.col32);
      HB_CK(cudaGetLastError());
      // a Gauss-Seidel phase launched next may read the copy before this
      // kernel is done (its producer does not wait): finish it here
      HB_TRY(stream_sync(c));
      L.old32 = false;
    }
    if (!L.r32) {
      HB_TRY(dev_alloc((void**)&L.r32, sizeof(float) * L.pitch, &P->bytes));
      HB_TRY(dev_alloc((void**)&L.x32, sizeof(float) * L.pitch, &P->bytes));
      HB_CK(cudaMemsetAsync(L.r32, 0, sizeof(float) * L.pitch, c->stream));
      HB_CK(cudaMemsetAsync(L.x32, 0, sizeof(float) * L.pitch, c->stream));
      // FP32 phases load half the bytes per instruction: tune them on their own
      // (on the level's FP32 work vectors, which every V-cycle rewrites)
      int ov[6], at64[kColours], at32[kColours], wf = -1;
      if (level_config_override(l, ov, &wf, at64, at32)) {
        L.gs_sched32 = ov[4];
        L.gs_first32 = ov[5];
        for (int s = 0; s < kColours; ++s) L.gs_first32_at[s] = at32[s];
        continue;
      }
      const char* force = std::getenv("HPCG_B200_CONFIG");
      if (force && *force) {
        const int f = std::atoi(force);
        L.gs_first32 = f < 0 ? 0 : f >= kGsConfigs ? kGsConfigs - 1 : f;
        L.gs_sched32 = std::min(L.gs_first32, kGsFull - 1);
        continue;
      }
      if (by_rule(L)) {
        rule_config32(c, L);
        continue;
      }
      const int r0 = L.g.start[1], r1 = L.g.start[2];
      if (r1 <= r0) continue;
      cudaEvent_t e0, e1;
      HB_CK(cudaEventCreate(&e0));
      HB_CK(cudaEventCreate(&e1));
      float t[kGsConfigs], tf[kColours][kGsConfigs];
      for (int cfg = 0; cfg < kGsConfigs; ++cfg) {
        t[cfg] = 1e30f;
        for (int s = 0; s < kColours; ++s) tf[s][cfg] = 1e30f;
      }
      auto time_it = [&](float& best_ms, auto&& launch) -> int {
        HB_CK(cudaEventRecord(e0, c->stream));
        launch();
        HB_CK(cudaEventRecord(e1, c->stream));
        HB_CK(cudaEventSynchronize(e1));
        float ms = 0.f;
        HB_CK(cudaEventElapsedTime(&ms, e0, e1));
        if (ms < best_ms) best_ms = ms;
        return HPCG_B200_OK;
      };
      for (int rep = 0; rep < 4; ++rep) {  // round-robin over the configurations, as in autotune
        for (int cfg = 0; cfg < kGsConfigs; ++cfg) {
          if (cfg < kGsFull) HB_TRY(time_it(t[cfg], [&] {
            gs_dispatch<float, float, false>(c, L, cfg, L.val32, L.r32, L.x32, r0, r1, kAllSlots);
          }));
          // the first-sweep phase of every sweep position, as in autotune
          for (int s = 0; s < kColours; ++s) {
            if (L.g.start[s + 1] <= L.g.start[s]) continue;
            HB_TRY(time_it(tf[s][cfg], [&] {
              gs_first_dispatch<float, float>(c, L, cfg, L.val32, L.r32, L.x32, L.g.start[s], L.g.start[s + 1], s,
                                              first_mask(L.g, s));
            }));
          }
        }
      }
      float best = 1e30f;
      for (int cfg = 0; cfg < kGsConfigs; ++cfg) {
        if (t[cfg] < best) {
          best = t[cfg];
          L.gs_sched32 = cfg;
        }
      }
      pick_first(tf, L.gs_first32_at, &L.gs_first32);
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      HB_CK(cudaGetLastError());
    }
  }
  return HPCG_B200_OK;
}

// ComputeMG_ref.cpp:39-63 with FP32 values, vectors and arithmetic.
int mg32_level(hpcg_b200_problem* p, int l, const float* r, float* x) {
  Level& L = p->lev[l];
  Context* c = p->ctx;
  if (!(c->prof && l == 0) && l >= tail_first(p, true) && tail_vcycle(p, l, r, x)) return HPCG_B200_OK;
  HB_TRY((gs_colour<float, float>(c, L, L.val32, r, x, true, l == 0)));
  if (l + 1 < p->nlev) {
    Level& C = p->lev[l + 1];
    restrict_dispatch<float>(c, L, L.val32, r, x, C.r32, C.n);
    HB_CK(cudaGetLastError());
    HB_TRY(l == 0 ? coarse_vcycle(p, true) : mg32_level(p, l + 1, C.r32, C.x32));
    HB_CK(launch_early(c->stream, k_prolong<float>, grid_for(c, C.n, kThreads, kPerSm), kThreads, 0, L.tf, L.tq, C.x32,
                       x, C.n));
    HB_TRY((gs_colour<float, float>(c, L, L.val32, r, x, false, l == 0)));
  }
  return HPCG_B200_OK;
}

// Flexible PCG in FP64 around the FP32 V-cycle: z = widen(MG32(narrow(r))),
// beta = r'(z - z_prev) / r_prev'z_prev (Polak-Ribiere), everything else as CG.cpp.
int run_cg_mixed(hpcg_b200_problem* P, int max_iter, double tol, int* niters, double* normr_out,
                 double* normr0_out) {
  HB_TRY(ensure_f32(P));
  Level& L = P->lev[0];
  Context* c = P->ctx;
  const int n = L.n;
  const int nb = red_blocks(c, n);
  const int gv = grid_for(c, n, kThreads, kPerSm);
  HB_TRY(autotune(P));
  spmv_dispatch<double, false>(c, L, L.val, P->x, P->Ap, nullptr);
  k_waxpby<true><<<nb, kThreads, 0, c->stream>>>(n, 1.0, P->b, -1.0, P->Ap, P->r, c->partials);
  HB_CK(cudaGetLastError());
  HB_TRY(finalize(c, nb, kFinNormr));
  HB_TRY(read_scalars(c));
  double normr = std::sqrt(c->scal_host->normr2);
  const double normr0 = normr;
  *niters = 0;
  // z and zprev alternate between two buffers; r32 is refreshed by the x/r update
  double* zc = P->z;
  double* zp = P->zprev;
  if (max_iter >= 1 && normr / normr0 > tol) {
    k_convert<float, double><<<gv, kThreads, 0, c->stream>>>(L.r32, P->r, n);
    HB_CK(cudaGetLastError());
  }
  for (int k = 1; k <= max_iter && normr / normr0 > tol; ++k) {
    HB_TRY(mg32_cycle(P));
    if (k == 1) {
      k_widen_dot<false><<<nb, kThreads, 0, c->stream>>>(n, L.x32, P->r, zc, nullptr, c->partials);
      HB_CK(cudaGetLastError());
      HB_TRY(finalize(c, nb, kFinRtzFirst));
      HB_CK(cudaMemcpyAsync(P->p, zc, sizeof(double) * n, cudaMemcpyDeviceToDevice, c->stream));
    } else {
      HB_CK(launch_early(c->stream, k_widen_dot<true>, nb, kThreads, 0, n, L.x32, P->r, zc, zp, c->partials));
      HB_TRY(finalize(c, nb, kFinFlex));
      // with x of iteration k - 1
      HB_CK(launch_early(c->stream, k_update_px, gv, kThreads, 0, n, zc, P->p, P->x, c->scal));
    }
    std::swap(zc, zp);
    const int gs = spmv_dispatch<double, true>(c, L, L.val, P->p, P->Ap, c->partials);
    HB_CK(cudaGetLastError());
    HB_TRY(finalize(c, gs, kFinPap));
    HB_CK(launch_early(c->stream, k_update_r, nb, kThreads, 0, n, P->r, P->Ap, c->scal, c->partials, L.r32));
    HB_TRY(finalize(c, nb, kFinNormr));
    HB_TRY(read_scalars(c));
    normr = std::sqrt(c->scal_host->normr2);
    *niters = k;
  }
  if (*niters > 0) {  // the last iteration's x update
    k_update_x<<<gv, kThreads, 0, c->stream>>>(n, P->x, P->p, c->scal, 0);
    HB_CK(cudaGetLastError());
  }
  *normr_out = normr;
  *normr0_out = normr0;
  return HPCG_B200_OK;
}

}  // namespace

int prepare_f32(hpcg_b200_problem* p) { return ensure_f32(p); }

// ---- pieces of the single-rank path the sharded drivers reuse (shard.cuh) ----

int autotune_problem(hpcg_b200_problem* p) { return autotune(p); }

// a launch error as the negative status (the success value of the reducing
// launchers is their partial count)
int neg_status(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) return 0;
  set_error(what, e);
  return -status_of(e);
}

int spmv_level(hpcg_b200_problem* p, int l, const double* x, double* y, bool dot) {
  Context* c = p->ctx;
  const Level& L = p->lev[l];
  const int parts = dot ? spmv_dispatch<double, true>(c, L, L.val, x, y, c->partials)
                        : spmv_dispatch<double, false>(c, L, L.val, x, y, nullptr);
  const int e = neg_status("spmv");
  if (e) return dot ? e : -e;
  return dot ? parts : HPCG_B200_OK;
}

int restrict_level(hpcg_b200_problem* p, int l, const double* rf, const double* xf, double* rc) {
  const Level& L = p->lev[l];
  restrict_dispatch<double>(p->ctx, L, L.val, rf, xf, rc, p->lev[l + 1].n);
  HB_CK(cudaGetLastError());
  return HPCG_B200_OK;
}

int prolong_level(hpcg_b200_problem* p, int l, const double* xc, double* xf) {
  const Level& L = p->lev[l];
  const int nc = p->lev[l + 1].n;
  Context* c = p->ctx;
  k_prolong<double><<<grid_for(c, nc, kThreads, kPerSm), kThreads, 0, c->stream>>>(L.tf, L.tq, xc, xf, nc);
  HB_CK(cudaGetLastError());
  return HPCG_B200_OK;
}

int symgs_step(hpcg_b200_problem* p, int l, const double* rhs, double* x, bool x_is_zero, double* dot) {
  return symgs_level(p, l, rhs, x, x_is_zero, dot);
}

bool rtz_from_smoother(const hpcg_b200_problem* p) { return rtz_fused(p); }

int reduction_blocks(const Context* c, int64_t n) { return red_blocks(c, n); }

int launch_residual(Context* c, int n, const double* b, const double* Ap, double* r) {
  const int nb = red_blocks(c, n);
  k_waxpby<true><<<nb, kThreads, 0, c->stream>>>(n, 1.0, b, -1.0, Ap, r, c->partials);
  const int e = neg_status("launch_residual");
  return e ? e : nb;
}

int launch_dot(Context* c, int n, const double* x, const double* y) {
  const int nb = red_blocks(c, n);
  k_dot<false><<<nb, kThreads, 0, c->stream>>>(n, x, y, nullptr, c->partials);
  const int e = neg_status("launch_dot");
  return e ? e : nb;
}

int launch_update_px(Context* c, int n, const double* z, double* p, double* x) {
  k_update_px<<<grid_for(c, n, kThreads, kPerSm), kThreads, 0, c->stream>>>(n, z, p, x, c->scal);
  HB_CK(cudaGetLastError());
  return HPCG_B200_OK;
}

int launch_update_r(Context* c, int n, double* r, const double* Ap) {
  const int nb = red_blocks(c, n);
  k_update_r<<<nb, kThreads, 0, c->stream>>>(n, r, Ap, c->scal, c->partials);
  const int e = neg_status("launch_update_r");
  return e ? e : nb;
}

int launch_update_x(Context* c, int n, double* x, const double* p) {
  k_update_x<<<grid_for(c, n, kThreads, kPerSm), kThreads, 0, c->stream>>>(n, x, p, c->scal, 0);
  HB_CK(cudaGetLastError());
  return HPCG_B200_OK;
}

int launch_finalize(Context* c, int nparts, int op, double* out) { return finalize(c, nparts, op, out); }

int launch_finalize_ranks(Context* c, const double* vals, int nvals, int op, double* out) {
  k_finalize_ranks<<<1, 32, 0, c->stream>>>(vals, nvals, op, c->scal, out);
  HB_CK(cudaGetLastError());
  return HPCG_B200_OK;
}

static NatGrid nat_of(const Level& L) { return nat_grid(L.g, L.n); }

// natural-order src (host or device) -> colour-order device dst
int load_vector(hpcg_b200_problem* p, int level, const double* src, double* dst) {
  const Level& L = p->lev[level];
  Context* c = p->ctx;
  if (dst == p->b) p->b_kept = false;  // b no longer holds hpcg_b200_cg's kept right-hand side
  const double* s = src;
  bool dev = false;
  HB_TRY(locate_ptr(src, p->device, &dev, "input vector"));
  if (!dev) {
    HB_TRY(ensure_stage(c, L.n));
    HB_TRY(host_to_device(c, c->stage[0], src, L.n));
    s = c->stage[0];
  }
  // (the rows of a level are those of its grid whatever its columns)
  k_permute<true><<<grid_for(c, (L.n + 3) / 4, kThreads, kPerSm), kThreads, 0, c->stream>>>(dst, s, nat_of(L));
  HB_CK(cudaGetLastError());
  return HPCG_B200_OK;
}

// colour-order device src -> natural-order dst (host or device); synchronises
int store_vector(hpcg_b200_problem* p, int level, const double* src, double* dst) {
  const Level& L = p->lev[level];
  Context* c = p->ctx;
  bool dev = false;
  HB_TRY(locate_ptr(dst, p->device, &dev, "output vector"));
  double* d = dst;
  if (!dev) {
    HB_TRY(ensure_stage(c, L.n));
    d = c->stage[1];
  }
  k_permute<false><<<grid_for(c, (L.n + 3) / 4, kThreads, kPerSm), kThreads, 0, c->stream>>>(d, src, nat_of(L));
  HB_CK(cudaGetLastError());
  if (!dev) HB_TRY(device_to_host(c, dst, d, L.n));
  HB_TRY(stream_sync(c));
  return HPCG_B200_OK;
}

// ---- hpcg_b200_cg's host inputs ------------------------------------------------
// The reference's timed loop zeroes x on the host and calls CG with the same b
// for every set (src/main.cpp:334-340). For host vectors hpcg_b200_cg therefore
// sends b only when it differs from the b it sent last (an exact comparison,
// bit for bit, against a host copy kept with the problem), and zeroes x on the
// device when the host x is all zero bits, instead of sending it. Both checks
// read host memory on several threads, which outruns a copy from pageable
// memory. hpcg_b200_set_host_reuse (or HPCG_B200_HOST_REUSE=0 at creation)
// sends both every call.

bool host_same_bits(const double* a, const double* b, int64_t n) {
  std::atomic<bool> same{true};
  host_parallel(n, [&](int64_t lo, int64_t hi) {
    constexpr int64_t kStep = 1 << 16;  // entries compared between looks at the others' verdict
    for (int64_t i = lo; i < hi && same.load(std::memory_order_relaxed); i += kStep) {
      const int64_t m = std::min(kStep, hi - i);
      if (std::memcmp(a + i, b + i, sizeof(double) * (size_t)m) != 0) same.store(false, std::memory_order_relaxed);
    }
  });
  return same.load();
}

bool host_all_zero_bits(const double* a, int64_t n) {
  std::atomic<bool> zero{true};
  host_parallel(n, [&](int64_t lo, int64_t hi) {
    const uint64_t* w = reinterpret_cast<const uint64_t*>(a);
    constexpr int64_t kStep = 1 << 16;
    for (int64_t i = lo; i < hi && zero.load(std::memory_order_relaxed); i += kStep) {
      const int64_t e = std::min(hi, i + kStep);
      uint64_t acc = 0;
      for (int64_t j = i; j < e; ++j) acc |= w[j];
      if (acc) zero.store(false, std::memory_order_relaxed);
    }
  });
  return zero.load();
}

int load_cg_rhs(hpcg_b200_problem* p, const double* b) {
  bool dev = false;
  HB_TRY(locate_ptr(b, p->device, &dev, "b"));
  const int n = p->lev[0].n;
  if (dev || !p->host_reuse) return load_vector(p, 0, b, p->b);
  if (p->b_kept && host_same_bits(p->b_kept_host, b, n)) return HPCG_B200_OK;
  if (!p->b_kept_host) p->b_kept_host = new (std::nothrow) double[n];  // no host memory: send every call
  if (p->b_kept_host)
    host_parallel(n, [&](int64_t lo, int64_t hi) {
      std::memcpy(p->b_kept_host + lo, b + lo, sizeof(double) * (size_t)(hi - lo));
    });
  HB_TRY(load_vector(p, 0, b, p->b));  // a copy from pageable memory has read b when it returns
  p->b_kept = p->b_kept_host != nullptr;
  return HPCG_B200_OK;
}

int load_cg_guess(hpcg_b200_problem* p, const double* x) {
  bool dev = false;
  HB_TRY(locate_ptr(x, p->device, &dev, "x"));
  const Level& L = p->lev[0];
  if (!dev && p->host_reuse && host_all_zero_bits(x, L.n)) {
    HB_CK(cudaMemsetAsync(p->x, 0, sizeof(double) * L.pitch, p->ctx->stream));
    return HPCG_B200_OK;
  }
  return load_vector(p, 0, x, p->x);
}

}  // namespace hb

using namespace hb;

namespace {

// A vector argument of the standalone routines as a device pointer: device
// memory is used in place, host memory is staged into stage[slot].
int device_view(Context* c, const double* v, int n, int slot, const double** out) {
  bool dev = false;
  HB_TRY(locate_ptr(v, c->device, &dev, "input vector"));
  if (dev) {
    *out = v;
    return HPCG_B200_OK;
  }
  HB_TRY(ensure_stage(c, (size_t)n));
  HB_TRY(host_to_device(c, c->stage[slot], v, (size_t)n));
  *out = c->stage[slot];
  return HPCG_B200_OK;
}

// Largest level whose SpMV call reads and writes the caller's device vectors in
// place (k_spmv_nat) instead of permuting them around the bulk-copy SpMV: 96^3 47
// against 57 us, 128^3 89 against 104, 192^3 312 against 323. Beyond, x no longer
// stays in the L2 from one colour block to the next, which the slab order of the
// bulk-copy SpMV provides for. Where the environment names the level's configurations
// or asks for timed ones, the call runs what it named (Level::mv_rule).
constexpr int kNatSpmv = 1 << 23;

// whether runs of na doubles at a and nb at b share memory
bool overlap(const double* a, int64_t na, const double* b, int64_t nb) {
  const uintptr_t u = (uintptr_t)a, v = (uintptr_t)b;
  return u < v + sizeof(double) * (uintptr_t)nb && v < u + sizeof(double) * (uintptr_t)na;
}

// The result of lone reduction `call` once the GPU has stored it: the host looks
// for it for as long as such a call usually takes, then waits for the stream
// (which also reports what went wrong).
int lone_result(Context* c, const volatile LoneResult* r, unsigned long long call, double* out) {
  const double until = now_s() + 200e-6;
  while (r->call != call)
    if (now_s() > until) {
      HB_TRY(stream_sync(c));
      break;
    }
  std::atomic_thread_fence(std::memory_order_acquire);
  *out = r->value;
  return HPCG_B200_OK;
}

template <bool MAX>
int lone_reduction(Context* c, int n, const double* x, const double* y, double* out) {
  static_assert(sizeof(LoneResult) * kLoneSlots == kLoneBytes, "the results' memory");
  const unsigned long long call = c->lone_call.fetch_add(1) + 1;
  volatile LoneResult* r = static_cast<volatile LoneResult*>(c->lone) + call % kLoneSlots;
  k_lone<MAX><<<red_blocks(c, n), kThreads, 0, c->stream>>>(n, x, y, c->partials, c->lone_count, r, call);
  HB_CK(cudaGetLastError());
  return lone_result(c, r, call, out);
}

}  // namespace

extern "C" {

int hpcg_b200_spmv(hpcg_b200_problem* p, const double* x, double* y) {
  if (!valid(p)) return HPCG_B200_ERR_HANDLE;
  if (is_rank(p)) return HPCG_B200_ERR_UNSUPPORTED;  // a rank: use the hpcg_b200_shard_* routines
  if (!x || !y) return HPCG_B200_ERR_ARG;
  Setter dev(p->device);
  const Level& L = p->lev[0];
  Context* c = p->ctx;
  HB_TRY(autotune(p, false));
  bool xdev = false, ydev = false;
  if (L.geo_cols && L.mv_rule && L.n <= kNatSpmv) {
    HB_TRY(locate_ptr(x, p->device, &xdev, "input vector"));
    HB_TRY(locate_ptr(y, p->device, &ydev, "output vector"));
    if (xdev && ydev && !overlap(x, L.n, y, L.n)) {
      FastDiv dx, dy;
      dx.init((unsigned)L.g.nx);
      dy.init((unsigned)L.g.ny);
      k_spmv_nat<<<(L.n + kThreads - 1) / kThreads, kThreads, 0, c->stream>>>(L.val, L.pitch, L.new2old, x, y, L.g.nx,
                                                                              L.g.ny, L.g.nz, dx, dy, L.n);
      HB_CK(cudaGetLastError());
      return stream_sync(c);
    }
  }
  HB_TRY(load_vector(p, 0, x, p->p));
  spmv_dispatch<double, false>(c, L, L.val, p->p, p->Ap, nullptr);
  HB_CK(cudaGetLastError());
  return store_vector(p, 0, p->Ap, y);
}

int hpcg_b200_symgs(hpcg_b200_problem* p, const double* r, double* x) {
  if (!valid(p)) return HPCG_B200_ERR_HANDLE;
  if (is_rank(p)) return HPCG_B200_ERR_UNSUPPORTED;  // a rank: use the hpcg_b200_shard_* routines
  if (!r || !x) return HPCG_B200_ERR_ARG;
  Setter dev(p->device);
  HB_TRY(load_vector(p, 0, r, p->r));
  HB_TRY(load_vector(p, 0, x, p->x));
  HB_TRY(autotune(p));
  HB_TRY(run_cycle(p, kCycleStep, [&] { return symgs_level(p, 0, p->r, p->x, false); }));
  return store_vector(p, 0, p->x, x);
}

int hpcg_b200_mg(hpcg_b200_problem* p, const double* r, double* x) {
  if (!valid(p)) return HPCG_B200_ERR_HANDLE;
  if (is_rank(p)) return HPCG_B200_ERR_UNSUPPORTED;  // a rank: use the hpcg_b200_shard_* routines
  if (!r || !x) return HPCG_B200_ERR_ARG;
  Setter dev(p->device);
  HB_TRY(load_vector(p, 0, r, p->r));
  HB_TRY(autotune(p));
  HB_TRY(mg_cycle(p));
  return store_vector(p, 0, p->z, x);
}

int hpcg_b200_cg(hpcg_b200_problem* p, const double* b, double* x, int max_iter, double tolerance,
                 int do_preconditioning, int* niters, double* normr, double* normr0, double* times) {
  if (!valid(p)) return HPCG_B200_ERR_HANDLE;
  if (is_rank(p)) return HPCG_B200_ERR_UNSUPPORTED;  // a rank: use the hpcg_b200_shard_* routines
  if (!b || !x || !niters || !normr || !normr0 || max_iter < 0) return HPCG_B200_ERR_ARG;
  Setter dev(p->device);
  HB_TRY(load_cg_rhs(p, b));
  HB_TRY(load_cg_guess(p, x));
  HB_TRY(run_cg(p, max_iter, tolerance, do_preconditioning != 0, niters, normr, normr0, times));
  return store_vector(p, 0, p->x, x);
}

int hpcg_b200_cg_mixed(hpcg_b200_problem* p, const double* b, double* x, int max_iter, double tolerance,
                       int* niters, double* normr, double* normr0) {
  if (!valid(p)) return HPCG_B200_ERR_HANDLE;
  if (is_rank(p)) return HPCG_B200_ERR_UNSUPPORTED;  // a rank: use the hpcg_b200_shard_* routines
  if (!b || !x || !niters || !normr || !normr0 || max_iter < 0) return HPCG_B200_ERR_ARG;
  Setter dev(p->device);
  HB_TRY(load_vector(p, 0, b, p->b));
  HB_TRY(load_vector(p, 0, x, p->x));
  HB_TRY(run_cg_mixed(p, max_iter, tolerance, niters, normr, normr0));
  return store_vector(p, 0, p->x, x);
}

int hpcg_b200_mg_f32(hpcg_b200_problem* p, const double* r, double* x) {
  if (!valid(p)) return HPCG_B200_ERR_HANDLE;
  if (is_rank(p)) return HPCG_B200_ERR_UNSUPPORTED;  // a rank: use the hpcg_b200_shard_* routines
  if (!r || !x) return HPCG_B200_ERR_ARG;
  Setter dev(p->device);
  HB_TRY(ensure_f32(p));
  Level& L = p->lev[0];
  Context* c = p->ctx;
  const int gv = grid_for(c, L.n, kThreads, kPerSm);
  HB_TRY(load_vector(p, 0, r, p->r));
  k_convert<float, double><<<gv, kThreads, 0, c->stream>>>(L.r32, p->r, L.n);
  HB_CK(cudaGetLastError());
  HB_TRY(mg32_cycle(p));
  k_convert<double, float><<<gv, kThreads, 0, c->stream>>>(p->z, L.x32, L.n);
  HB_CK(cudaGetLastError());
  return store_vector(p, 0, p->z, x);
}

int hpcg_b200_adjoint(hpcg_b200_problem* p, const double* x, const double* g, int max_iter, double tolerance,
                      double* grad_b, double* grad_values27, int* niters) {
  if (!valid(p)) return HPCG_B200_ERR_HANDLE;
  if (is_rank(p)) return HPCG_B200_ERR_UNSUPPORTED;  // a rank: use the hpcg_b200_shard_* routines
  if (!x || !g || !grad_b || !grad_values27 || !niters || max_iter < 0) return HPCG_B200_ERR_ARG;
  Setter dev(p->device);
  const Level& L = p->lev[0];
  Context* c = p->ctx;
  // lambda: A lambda = g with the same preconditioned CG, from lambda = 0
  HB_TRY(load_vector(p, 0, g, p->b));
  HB_CK(cudaMemsetAsync(p->x, 0, sizeof(double) * L.pitch, c->stream));
  double nr = 0, nr0 = 0;
  HB_TRY(run_cg(p, max_iter, tolerance, true, niters, &nr, &nr0, nullptr));
  HB_TRY(store_vector(p, 0, p->x, grad_b));  // dL/db = lambda
  // on grid columns the gradients are formed from the natural-order vectors:
  // lambda as just stored, x as given, or their device copies; from the problem's
  // own colour-order vectors where the gradients go over one of those
  bool xdev = false, bdev = false, dev_out = false;
  HB_TRY(locate_ptr(x, p->device, &xdev, "x"));
  HB_TRY(locate_ptr(grad_b, p->device, &bdev, "grad_b"));
  HB_TRY(locate_ptr(grad_values27, p->device, &dev_out, "grad_values27"));
  const double* xn = x;
  const double* ln = bdev ? grad_b : c->stage[1];
  const int64_t entries = (int64_t)kSlots * L.n;
  const bool natural = L.geo_cols && !(dev_out && ((xdev && overlap(grad_values27, entries, x, L.n)) ||
                                                   (bdev && overlap(grad_values27, entries, grad_b, L.n))));
  if (!natural) {
    HB_TRY(load_vector(p, 0, x, p->Ap));  // the forward solution, colour order
  } else if (!xdev) {
    if (bdev) HB_TRY(ensure_stage(c, L.n));  // (else stage[1] holds lambda and they are large enough)
    HB_TRY(host_to_device(c, c->stage[0], x, L.n));
    xn = c->stage[0];
  }
  double* out = grad_values27;
  const size_t bytes = sizeof(double) * (size_t)entries;
  if (!dev_out) HB_CK(cudaMalloc(&out, bytes));
  if (natural) {
    FastDiv dx, dy;
    dx.init((unsigned)L.g.nx);
    dy.init((unsigned)L.g.ny);
    k_adjoint_values_geo<<<(L.n + 1023) / 1024, kThreads, 0, c->stream>>>(L.g.nx, L.g.ny, L.g.nz, dx, dy, ln, xn, out);
  } else {
    k_adjoint_values<<<grid_for(c, L.n, kThreads, kPerSm), kThreads, 0, c->stream>>>(L.g, L.col, L.pitch, L.n, p->x,
                                                                                      p->Ap, out);
  }
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && !dev_out) e = cudaMemcpyAsync(grad_values27, out, bytes, cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (!dev_out) cudaFree(out);
  if (e != cudaSuccess) {
    set_error("hpcg_b200_adjoint", e);
    return status_of(e);
  }
  return HPCG_B200_OK;
}

int hpcg_b200_wait_selftest(int device, double seconds) {
  if (!(seconds > 0.0 && seconds <= 2.0)) return HPCG_B200_ERR_ARG;
  Context* c = context_for(device);
  if (!c) return HPCG_B200_ERR_CUDA;
  Setter dev(device);
  k_wait_selftest<<<1, 32, 0, c->stream>>>((unsigned long long)(seconds * 1e9), c->fault);
  HB_CK(cudaGetLastError());
  return stream_sync(c);
}

int hpcg_b200_level_config(const hpcg_b200_problem* p, int level, int* config) {
  if (!valid(p)) return HPCG_B200_ERR_HANDLE;
  if (!config || level < 0 || level >= p->nlev) return HPCG_B200_ERR_ARG;
  const Level& L = p->lev[level];
  config[0] = L.gs_sched;
  config[1] = L.gs_first;
  config[2] = L.gs_sched32;
  config[3] = L.mv_sched;
  config[4] = L.mv_order;
  config[5] = L.tuned ? 1 : 0;
  config[6] = L.gs_first32;
  return HPCG_B200_OK;
}

int hpcg_b200_wave_wait_selftest(hpcg_b200_problem* p, double limit_seconds) {
  if (!valid(p)) return HPCG_B200_ERR_HANDLE;
  if (!(limit_seconds > 0.0) || limit_seconds > 10.0) return HPCG_B200_ERR_ARG;
  HB_CK(cudaSetDevice(p->device));
  Context* c = p->ctx;
  Level& L = p->lev[0];
  HB_TRY(ensure_wavefront(L));
  if (L.wf_tpu <= 0) return HPCG_B200_ERR_UNSUPPORTED;
  // one unit (one phase, one z pair) that waits for itself: its counter cannot
  // fill before its own tiles are released, so every block's wait runs out
  WaveGeom w = L.wf_geom[0];
  w.H = 1;
  w.P = 1;
  w.dot_from = 1;
  w.self_dep = 0;
  // x: scratch (Ap), which the tiles released after the wait gave up rewrite
  const unsigned long long lim = (unsigned long long)(limit_seconds * 1e9);
  if (!wave_launch(c, L, p->zprev, p->Ap, w, nullptr, lim)) return HPCG_B200_ERR_UNSUPPORTED;
  return stream_sync(c);
}

int hpcg_b200_stream_probe(hpcg_b200_problem* p, int level, float* ms, double* bytes) {
  if (!valid(p)) return HPCG_B200_ERR_HANDLE;
  if (!ms || !bytes || level < 0 || level >= p->nlev) return HPCG_B200_ERR_ARG;
  Setter dev(p->device);
  Context* c = p->ctx;
  const Level& L = p->lev[level];
  if (L.pack == kPackDiag) return stream_probe_p<kPackDiag>(c, L, ms, bytes);
  if (L.pack == 1) return stream_probe_p<1>(c, L, ms, bytes);
  if (L.pack == 2) return stream_probe_p<2>(c, L, ms, bytes);
  return stream_probe_p<0>(c, L, ms, bytes);
}

int hpcg_b200_level_wavefront(const hpcg_b200_problem* p, int level, int* on) {
  if (!valid(p)) return HPCG_B200_ERR_HANDLE;
  if (!on || level < 0 || level >= p->nlev) return HPCG_B200_ERR_ARG;
  *on = p->lev[level].wf;
  return HPCG_B200_OK;
}

int hpcg_b200_level_first_config(const hpcg_b200_problem* p, int level, int* fp64, int* fp32) {
  if (!valid(p)) return HPCG_B200_ERR_HANDLE;
  if (level < 0 || level >= p->nlev) return HPCG_B200_ERR_ARG;
  const Level& L = p->lev[level];
  for (int s = 0; s < kColours; ++s) {
    if (fp64) fp64[s] = L.gs_first_at[s] >= 0 ? L.gs_first_at[s] : L.gs_first;
    if (fp32) fp32[s] = L.gs_first32_at[s] >= 0 ? L.gs_first32_at[s] : L.gs_first32;
  }
  return HPCG_B200_OK;
}

int hpcg_b200_dot(int n, const double* x, const double* y, double* result) {
  if (!x || !y || !result || n < 0) return HPCG_B200_ERR_ARG;
  Context* c = current_context();
  if (!c) return HPCG_B200_ERR_CUDA;
  if (n == 0) {
    *result = 0.0;
    return HPCG_B200_OK;
  }
  const double *dx, *dy;
  HB_TRY(device_view(c, x, n, 0, &dx));
  if (y == x) dy = dx;
  else HB_TRY(device_view(c, y, n, 1, &dy));
  return lone_reduction<false>(c, n, dx, dy, result);
}

int hpcg_b200_waxpby(int n, double alpha, const double* x, double beta, const double* y, double* w) {
  if (!x || !y || !w || n < 0) return HPCG_B200_ERR_ARG;
  Context* c = current_context();
  if (!c) return HPCG_B200_ERR_CUDA;
  if (n == 0) return HPCG_B200_OK;
  const double *dx, *dy;
  HB_TRY(device_view(c, x, n, 0, &dx));
  if (y == x) dy = dx;
  else HB_TRY(device_view(c, y, n, 1, &dy));
  bool wdev = false;
  HB_TRY(locate_ptr(w, c->device, &wdev, "output vector"));
  if (!wdev) HB_TRY(ensure_stage(c, (size_t)n));
  double* dw = wdev ? w : c->stage[2];
  k_waxpby<false><<<grid_for(c, n, kThreads, kPerSm), kThreads, 0, c->stream>>>(n, alpha, dx, beta, dy, dw, nullptr);
  HB_CK(cudaGetLastError());
  if (!wdev) HB_TRY(device_to_host(c, w, dw, (size_t)n));
  HB_TRY(stream_sync(c));
  return HPCG_B200_OK;
}

int hpcg_b200_residual(int n, const double* v1, const double* v2, double* residual) {
  if (!v1 || !v2 || !residual || n < 0) return HPCG_B200_ERR_ARG;
  Context* c = current_context();
  if (!c) return HPCG_B200_ERR_CUDA;
  if (n == 0) {
    *residual = 0.0;
    return HPCG_B200_OK;
  }
  const double *a, *b;
  HB_TRY(device_view(c, v1, n, 0, &a));
  HB_TRY(device_view(c, v2, n, 1, &b));
  return lone_reduction<true>(c, n, a, b, residual);
}

}  // extern "C"
