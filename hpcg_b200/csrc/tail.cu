// Host side of the one-launch small end of the V-cycle (tail.cuh): which levels
// it runs, its shape, and its launch.
#include <cstdlib>

#include "tail.cuh"

namespace hb {

namespace {

// Largest number of rows a block may have in one colour phase: one chunk of a
// block's threads. Each further chunk adds its own chain, while a phase spread
// over every SM costs its launch whatever its size. CG per iteration with the level
// in and out of this launch, FP64: 256 rows (32^3) 136 against 139 us, 288 rows
// (36x32x32 below 72x64x64) 218 against 194, 384 rows 218 against 194; FP32, whose
// launched phases read half the bytes: 256 rows 137 against 133, 288 rows 202 against
// 188. A lone step also brings x in: 64 rows (16^3) 43 against 47 us, 144 rows
// (24^3) 49 against 47, 256 rows 51 against 47.
// Measurement knob: HPCG_B200_TAIL_ROWS.
int max_rows(bool f32) {
  static const int forced = [] {
    const char* e = std::getenv("HPCG_B200_TAIL_ROWS");
    return e && *e ? std::atoi(e) : 0;
  }();
  return forced > 0 ? forced : f32 ? 240 : 256;
}
constexpr int kStepRows = 96;
constexpr int kMaxSmem = 200 * 1024;
// A level with at most this many rows to a colour stays on one block: its
// phases then end at the block's own barrier instead of the cluster's.
constexpr int kOneBlockRows = 128;

int blocks_of(const Level& L) {
  const int pairs = (L.g.nz + 1) / 2;
  const int rows = pairs * ((L.g.ny + 1) / 2) * ((L.g.nx + 1) / 2);
  return rows <= kOneBlockRows ? 1 : std::min(pairs, kTailMaxCluster);
}

// most z pairs of one block
int most_pairs(const Level& L, int act) { return ((L.g.nz + 1) / 2 + act - 1) / act; }

// most rows of one block in a phase
int64_t most_rows(const Level& L, int act) {
  return (int64_t)most_pairs(L, act) * ((L.g.ny + 1) / 2) * ((L.g.nx + 1) / 2);
}

int64_t elems_of(const Level& L, int act) {
  return (int64_t)(2 * most_pairs(L, act) + 2) * TailShape(L.g.nx, L.g.ny).sz;
}
// entries of a block's row table: its points
int64_t rows_of(const Level& L, int act) { return 2ll * most_pairs(L, act) * L.g.ny * L.g.nx; }
// shared memory of a level
int64_t bytes_of(const Level& L, int act, bool f32) {
  return elems_of(L, act) * (f32 ? 4 : 8) + rows_of(L, act) * (int64_t)sizeof(TailRow);
}

// the first level from which all levels fit a block's share of max_rows rows a
// phase and max_bytes of shared memory
int first_within(const hpcg_b200_problem* p, bool f32, int64_t rows, int64_t max_bytes) {
  int64_t bytes = 256;  // rounding of the table's place
  int f = p->nlev;
  for (int l = p->nlev - 1; l >= 0; --l) {
    const Level& L = p->lev[l];
    if (!L.geo || L.next || L.n <= 0 || (l + 1 < p->nlev && !L.geo_f2c)) break;
    const int act = blocks_of(L);
    bytes += bytes_of(L, act, f32);
    if (most_rows(L, act) > rows || bytes > max_bytes) break;
    f = l;
  }
  return f;
}

// On unless the environment pins kernel configurations or asks for wavefront
// sweeps (those are to run), HPCG_B200_TAIL=0 / 1: off / on either way.
bool wanted() {
  const char* e = std::getenv("HPCG_B200_TAIL");
  if (e && *e) return e[0] != '0';
  const char* a = std::getenv("HPCG_B200_CONFIG");
  const char* b = std::getenv("HPCG_B200_LEVEL_CONFIG");
  const char* w = std::getenv("HPCG_B200_WAVE");
  return !(a && *a) && !(b && *b) && !(w && *w && w[0] != '0');
}

__global__ void k_tail_values(const double* __restrict__ val, int64_t pitch, double* __restrict__ valt) {
  const int64_t total = (int64_t)kSlots * pitch;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int k = (int)(i / pitch);
    valt[mat_index<double, kTailBlock>(k, i - (int64_t)k * pitch, pitch)] = val[i];
  }
}

template <typename T>
int describe(hpcg_b200_problem* p, int l, int nlev, TailDesc<T>* desc, size_t* smem) {
  TailDesc<T>& D = *desc;
  std::memset(&D, 0, sizeof(D));
  D.nlev = nlev;
  int cluster = 1;
  int64_t elems = 0, rows = 0;
  for (int i = 0; i < nlev; ++i) {
    const Level& L = p->lev[l + i];
    TailLevel<T>& t = D.lev[i];
    if constexpr (sizeof(T) == 4) {
      t.val = L.val32;
      t.r = L.r32;
      t.x = L.x32;
    } else {
      t.val = L.valt;
      t.r = L.r;
      t.x = L.x;
    }
    t.nx = L.g.nx;
    t.ny = L.g.ny;
    t.nz = L.g.nz;
    for (int s = 0; s < kColours; ++s) t.start[s] = L.g.start[s];
    t.act = blocks_of(L);
    t.xoff = (int)elems;
    elems += elems_of(L, t.act);
    t.toff = (int)rows;
    rows += rows_of(L, t.act);
    cluster = std::max(cluster, t.act);
  }
  const ColourGrid& g = p->lev[l].g;
  for (int s = 0; s < kColours; ++s) {
    D.sweep[s] = g.sweep[s];
    D.pos[s] = g.pos[s];
    D.mask[s] = first_mask(g, s);
  }
  D.elems = (int)((elems + 1) & ~1ll);  // the row table behind it: 8-byte aligned
  D.rows = (int)rows;
  *smem = sizeof(T) * (size_t)D.elems + sizeof(TailRow) * (size_t)D.rows;
  int size = 1;
  while (size < cluster) size *= 2;
  return size;
}

template <typename T>
bool fits(hpcg_b200_problem* p, int l) {
  TailDesc<T> D;
  size_t smem = 0;
  const int size = describe(p, l, p->nlev - l, &D, &smem);
  return tail_fits((const void*)k_tail<T>, size, smem);
}

template <typename T>
bool launch(hpcg_b200_problem* p, int l, int nlev, const T* rhs, T* x, bool step) {
  Context* c = p->ctx;
  TailDesc<T> D;
  size_t smem = 0;
  const int size = describe(p, l, nlev, &D, &smem);
  auto k = k_tail<T>;
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(size);
  cfg.blockDim = dim3(kTailThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[2];
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = size;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k, D, rhs, x, step ? 1 : 0, c->fault);
  if (e != cudaSuccess) {
    set_error("k_tail", e);
    cudaGetLastError();
    p->tail_first[0] = p->tail_first[1] = p->nlev;
    return false;
  }
  return true;
}

}  // namespace

int tail_first(hpcg_b200_problem* p, bool f32) {
  int& first = p->tail_first[f32 ? 1 : 0];
  if (first >= 0) return first;
  first = p->nlev;
  if (!wanted()) return first;
  int f = first_within(p, f32, max_rows(f32), kMaxSmem);
  while (f < p->nlev && !(f32 ? fits<float>(p, f) : fits<double>(p, f))) ++f;
  if (!f32)
    for (int l = f; l < p->nlev; ++l)
      if (!p->lev[l].valt && tail_values(p, l) != HPCG_B200_OK) return first;  // no memory: the phases run
  first = f;
  return first;
}

int tail_first_within(const hpcg_b200_problem* p, bool f32, int64_t rows, int64_t bytes) {
  return wanted() ? first_within(p, f32, rows, std::min<int64_t>(bytes, kMaxSmem)) : p->nlev;
}

// The FP64 values of a small level in the layout tail.cuh reads, built (or,
// after the values changed, rewritten in place) from the level's own.
int tail_values(hpcg_b200_problem* p, int l) {
  Level& L = p->lev[l];
  Context* c = p->ctx;
  const int64_t cnt = blocked_entries(L.pitch, kTailBlock);
  if (!L.valt) {
    HB_TRY(dev_alloc((void**)&L.valt, sizeof(double) * cnt, &p->bytes));
    HB_CK(cudaMemsetAsync(L.valt, 0, sizeof(double) * cnt, c->stream));
  }
  k_tail_values<<<grid_for(c, (int64_t)kSlots * L.pitch, 256, 8), 256, 0, c->stream>>>(L.val, L.pitch, L.valt);
  HB_CK(cudaGetLastError());
  return HPCG_B200_OK;
}

int tail_desc(hpcg_b200_problem* p, int l, int nlev, TailDesc<double>* D, size_t* smem) {
  return describe(p, l, nlev, D, smem);
}
int tail_desc(hpcg_b200_problem* p, int l, int nlev, TailDesc<float>* D, size_t* smem) {
  return describe(p, l, nlev, D, smem);
}
bool tail_fits(const void* kernel, int size, size_t smem) {
  const char* e = std::getenv("HPCG_B200_TAIL_CLUSTER");
  if (e && *e && size > std::atoi(e)) return false;
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(size);
  cfg.blockDim = dim3(kTailThreads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = size;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem) == cudaSuccess &&
      cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
      cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess)
    return clusters > 0;
  cudaGetLastError();
  return false;
}

bool tail_step_ok(hpcg_b200_problem* p, int l) {
  return tail_first(p, false) <= l && most_rows(p->lev[l], blocks_of(p->lev[l])) <= kStepRows;
}

bool tail_vcycle(hpcg_b200_problem* p, int l, const double* r, double* x) {
  return launch<double>(p, l, p->nlev - l, r, x, false);
}
bool tail_vcycle(hpcg_b200_problem* p, int l, const float* r, float* x) {
  return launch<float>(p, l, p->nlev - l, r, x, false);
}
bool tail_step(hpcg_b200_problem* p, int l, const double* r, double* x) { return launch<double>(p, l, 1, r, x, true); }

}  // namespace hb
