// Batched solves: many independent HPCG problems of different sizes advanced
// together by flexible CG in FP64 around the FP32 V-cycle (the mixed form of
// hpcg_b200_cg_mixed, per problem).
//
// Every step of an iteration is ONE kernel launch for the whole batch: the
// launch walks a work list of row tiles that spans all problems (a colour phase
// of every problem's level, a restriction, a vector update...), so a batch of
// small problems costs the launches of one (and, in the form chosen by default,
// the small levels of all problems are one launch). The iteration loop itself is one
// CUDA graph launch: a conditional while node repeats the iteration while any
// problem is still above its tolerance and the iteration limit is not reached;
// problems that have converged skip their tiles. No kernel waits on another (an
// early launch waits on the device for the kernel before it).
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "bulk.cuh"
#include "geo.cuh"
#include "reduce.cuh"
#include "rows.cuh"
#include "tail.cuh"

namespace hb {

int prepare_f32(hpcg_b200_problem* p);
int free_problem(hpcg_b200_problem* p);
void release_accounted(size_t bytes);

namespace {

constexpr int kTile = kThreads;  // rows per tile: one thread per row
constexpr int kBlocksPerSm = 8;
constexpr uint64_t kBatchMagic = 0x48504347b2000b01ull;

// one problem's share of a Gauss-Seidel colour phase (FP32 V-cycle)
struct BGs {
  const float* val;
  const int* col;
  int64_t pitch;
  const float* rhs;
  float* x;
  int r0, r1;
  uint32_t mask;
  int first;
  int prob;
};
// residual + restriction, and prolongation, of one problem's level
struct BRes {
  const float* val;
  const int* col;
  int64_t pitch;
  const float* rf;
  const float* xf;
  const int* tf;
  const int* tq;
  float* rc;
  int nc;
  int prob;
};
// the level-0 (outer, FP64) vectors of one problem
struct BVec {
  const double* val;
  const int* col;
  int64_t pitch;
  int n;
  double *b, *x, *r, *z, *zprev, *p, *Ap;
  float *r32, *x32;
};
struct BTile {
  int item;   // index into the step's item array (or the problem for vector tiles)
  int start;  // first row of the tile
};
// per-problem CG scalars
struct BScal {
  double rtz, oldrtz, alpha, beta, pAp, normr2, normr0, rzprev;
  int active, niters;
};
struct BCtl {
  int iter;  // iterations completed
  int max_iter;
  double tol;
};

// ---- kernels -----------------------------------------------------------------

__device__ __forceinline__ void b_gs(const BGs* __restrict__ items, const BTile* __restrict__ tiles,
                                                   int ntiles, const BScal* __restrict__ sc) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BTile tl = tiles[t];
    const BGs it = items[tl.item];
    if (!sc[it.prob].active) continue;
    const int q = tl.start + threadIdx.x;
    if (q >= it.r1) continue;
    if (it.first)
      gs_row<float, float, true, kPlain, 0>(it.val, it.col, it.pitch, it.rhs, it.x, q, it.mask);
    else
      gs_row<float, float, false, kPlain, 0>(it.val, it.col, it.pitch, it.rhs, it.x, q, it.mask);
  }
}
__global__ void __launch_bounds__(kThreads) k_b_gs(const BGs* __restrict__ items, const BTile* __restrict__ tiles,
                                                   int ntiles, const BScal* __restrict__ sc) { b_gs(items, tiles, ntiles, sc); }

// ---- form 1: bulk-copy phases, columns from the grid ---------------------------
// Every batch member is generated on one rank, so its columns follow from its
// grids (geo.cuh): a phase's tile is its blocked FP32 values alone (val32 of the
// single-problem path), and the small levels of all problems are one launch
// (tail.cuh, a cluster for each problem). The same sums as k_b_gs and its kin.

// one problem's share of a step on one level: a colour phase (rhs -> x), or the
// residual at the injected rows (rhs, x -> rc through tq)
struct BGeo {
  const float* val;
  const float* rhs;
  float* x;
  float* rc;
  const int* tq;
  int r0, r1, sink, prob;
  GeoPhase geo;
};
// a tile of rows: everything a producer needs of it in one 32-byte load
struct alignas(32) BGeoTile {
  const float* vals;
  int item, start, prob, pad;
};

using BatchShape = GsShape<float, kPackGeo>;

// Descriptions kept on chip by the kernels below; those of further problems are
// read from memory. (Read from memory by every thread a full-slot phase of 0.5 M rows
// took 22 us, with the list walked by the producer alone and this 20.)
constexpr int kGeoCache = 24;

// A full-slot phase: the single-problem FP32 phase's pipeline and shape. Items
// item0 .. item0 + nitems - 1. fence: whether 32 bytes of a vector of one of them
// may hold rows of two colours (griddep_wait): sides are multiples of 16, so that is
// so on level 3, where they are multiples of 2.
__global__ void __launch_bounds__(BatchShape::threads, 1)
    k_b_gs_geo(const BGeo* __restrict__ items, int item0, int nitems, const BGeoTile* __restrict__ tiles, int ntiles,
               const BScal* __restrict__ sc, unsigned* fault, int fence) {
  __shared__ BGeo cache[kGeoCache];
  const int words = min(nitems, kGeoCache) * (int)(sizeof(BGeo) / sizeof(int));
  for (int i = threadIdx.x; i < words; i += blockDim.x)
    reinterpret_cast<int*>(cache)[i] = reinterpret_cast<const int*>(items + item0)[i];
  bulk_tiles_driven<float, BatchShape>(
      ntiles,
      [&](int t) {
        const BGeoTile tl = tiles[t];
        TileSrc<float> ts{};
        ts.q0 = (int64_t)(tl.item - item0) << 32 | (unsigned)tl.start;
        ts.vals = tl.vals;
        return ts;
      },
      [&](int t) { return !sc[tiles[t].prob].active; },
      [&](int64_t tag, const float* sv, int row, auto&& release) {
        const int at = (int)(tag >> 32), q = (int)(unsigned)tag + row;
        float a[kSlots];
#pragma unroll
        for (int k = 0; k < kSlots; ++k) a[k] = sv[k * kBulkRows];
        release();
        auto work = [&](const BGeo& it) {
          if (q < it.r0 || q >= it.r1) return;
          const GeoRow g(it.geo, q);
          const float* x = it.x;
          const int sink = it.sink;
          float sum = it.rhs[q], xd = 0.0f;
#pragma unroll
          for (int k = 0; k < kSlots; ++k) {
            const float xv = __ldg(x + g.col(it.geo, k, sink));
            sum -= a[k] * xv;
            if (k == kDiagSlot) xd = xv;
          }
          sum += xd * a[kDiagSlot];
          it.x[q] = sum / a[kDiagSlot];
        };
        if (at < kGeoCache)
          work(cache[at]);
        else
          work(items[item0 + at]);
      },
      fault, fence != 0);
}

// A first-sweep phase (k_gs_first_geo's arithmetic), 256 rows a tile.
template <uint32_t MASK>
__global__ void __launch_bounds__(kThreads, __builtin_popcount(MASK) > 16 ? 3 : 4)
    k_b_first_geo(const BGeo* __restrict__ items, const BGeoTile* __restrict__ tiles, int ntiles,
                  const BScal* __restrict__ sc) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BGeoTile tl = tiles[t];
    if (!sc[tl.prob].active) continue;
    const BGeo& it = items[tl.item];
    const int q = tl.start + threadIdx.x;
    if (q >= it.r1) continue;
    float a[kSlots];
#pragma unroll
    for (int k = 0; k < kSlots; ++k)
      if (MASK >> k & 1u) a[k] = __ldcs(it.val + mat_index<float>(k, q, 0));
    const float d = __ldcs(it.val + mat_index<float>(kDiagSlot, q, 0));
    float sum = it.rhs[q];
    if (MASK) {
      const GeoRow g(it.geo, q);
      float xv[kSlots];
#pragma unroll
      for (int k = 0; k < kSlots; ++k)
        if (MASK >> k & 1u) xv[k] = __ldg(it.x + g.col(it.geo, k, it.sink));
#pragma unroll
      for (int k = 0; k < kSlots; ++k)
        if (MASK >> k & 1u) sum -= a[k] * xv[k];
    }
    it.x[q] = sum / d;
  }
}

// Residual at the injected rows (k_b_restrict's arithmetic): rows r0 .. r1 are
// the all-even points, tq their coarse rows.
__global__ void __launch_bounds__(kThreads, 3)
    k_b_restrict_geo(const BGeo* __restrict__ items, const BGeoTile* __restrict__ tiles, int ntiles,
                     const BScal* __restrict__ sc) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BGeoTile tl = tiles[t];
    if (!sc[tl.prob].active) continue;
    const BGeo& it = items[tl.item];
    const int q = tl.start + threadIdx.x;
    if (q >= it.r1) continue;
    float a[kSlots];
#pragma unroll
    for (int k = 0; k < kSlots; ++k) a[k] = __ldcs(it.val + mat_index<float>(k, q, 0));
    const GeoRow g(it.geo, q);
    float sum = 0.0f;
#pragma unroll
    for (int k = 0; k < kSlots; ++k) sum += a[k] * __ldg(it.x + g.col(it.geo, k, it.sink));
    it.rc[it.tq[q - it.r0]] = it.rhs[q] - sum;
  }
}

// The small levels of every active problem: cluster p of the grid runs problem
// p's (tail.cuh).
__global__ void __launch_bounds__(kTailThreads, 2)
    k_b_tail(const TailDesc<float>* __restrict__ descs, const BScal* __restrict__ sc, unsigned* fault) {
  __shared__ TailDesc<float> D;
  const int p = (int)(blockIdx.x / cluster_blocks());
  if (!sc[p].active || descs[p].nlev == 0) return;  // the whole cluster
  const int* src = reinterpret_cast<const int*>(&descs[p]);
  for (int i = threadIdx.x; i < (int)(sizeof(D) / sizeof(int)); i += kTailThreads) reinterpret_cast<int*>(&D)[i] = src[i];
  __syncthreads();
  tail_run<float>(D, D.lev[0].r, D.lev[0].x, false, fault);
}

// Ap = A p (b_spmv's arithmetic) on the single-problem SpMV's pipeline, columns
// from the grid; one partial of p'Ap per warp: problem i's from 4 * tile0[i] on,
// four to each of its 128-row tiles. (Sides are multiples of 16, so every
// 256-row tile of the other kernels is two whole ones of these, and
// k_b_finalize_warps sums the partials in those kernels' order: the FP32
// V-cycle's input turns a last-bit difference of a dot into 1e-7 of a residual.)
using BatchSpmv = SpmvShape<double, kPackGeo>;
constexpr int kGridCache = 16;
struct alignas(64) BMap {
  CUtensorMap map;
};
__global__ void __launch_bounds__(BatchSpmv::threads, 1)
    k_b_spmv_geo(const BVec* __restrict__ v, const GeoGrid* __restrict__ grids, int m, const BMap* __restrict__ maps,
                 const BTile* __restrict__ tiles, int ntiles, const int* __restrict__ tile0,
                 const BScal* __restrict__ sc, double* __restrict__ partials, unsigned* fault) {
  __shared__ GeoGrid cache[kGridCache];
  const int words = min(m, kGridCache) * (int)(sizeof(GeoGrid) / sizeof(int));
  for (int i = threadIdx.x; i < words; i += blockDim.x)
    reinterpret_cast<int*>(cache)[i] = reinterpret_cast<const int*>(grids)[i];
  bulk_tiles_driven<double, BatchSpmv>(
      ntiles,
      [&](int t) {
        const BTile tl = tiles[t];
        TileSrc<double> ts{};
        ts.q0 = (int64_t)tl.item << 32 | (unsigned)tl.start;
        ts.map = &maps[tl.item].map;
        return ts;
      },
      [&](int t) { return !sc[tiles[t].item].active; },
      [&](int64_t tag, const double* sv, int row, auto&& release) {
        const int p = (int)(tag >> 32), q0 = (int)(unsigned)tag, q = q0 + row;
        double a[kSlots];
#pragma unroll
        for (int k = 0; k < kSlots; ++k) a[k] = sv[k * kBulkRows];
        release();
        const int n = v[p].n;
        const double* x = v[p].p;
        double acc = 0.0;
        auto work = [&](const GeoGrid& G) {
          int at = 0;
#pragma unroll
          for (int s = 1; s < kColours; ++s) at += q >= G.block[s].start ? 1 : 0;
          const GeoPhase& b = G.block[at];
          const GeoRow g(b, q);
          double sum = 0.0, xq = 0.0;
#pragma unroll
          for (int k = 0; k < kSlots; ++k) {
            const double xv = __ldg(x + g.col(b, k, n));
            sum += a[k] * xv;
            if (k == kDiagSlot) xq = xv;
          }
          v[p].Ap[q] = sum;
          acc = xq * sum;
        };
        if (q < n) {
          if (p < kGridCache)
            work(cache[p]);
          else
            work(grids[p]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if ((threadIdx.x & 31) == 0) partials[4 * (tile0[p] + q0 / kBulkRows) + row / 32] = acc;
      },
      fault, true);
}

// rc = (rf - A xf) at the injected rows (ComputeMG_ref.cpp:49-51, sorted pairs)
__device__ __forceinline__ void b_restrict(const BRes* __restrict__ items,
                                                         const BTile* __restrict__ tiles, int ntiles,
                                                         const BScal* __restrict__ sc) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BTile tl = tiles[t];
    const BRes it = items[tl.item];
    if (!sc[it.prob].active) continue;
    const int u = tl.start + threadIdx.x;
    if (u >= it.nc) continue;
    const int f = it.tf[u];
    float sum = 0.0f;
#pragma unroll
    for (int k = 0; k < kSlots; ++k)
      sum += it.val[mat_index<float, 0>(k, f, it.pitch)] * __ldg(it.xf + it.col[mat_index<float, 0>(k, f, it.pitch)]);
    it.rc[it.tq[u]] = it.rf[f] - sum;
  }
}
__global__ void __launch_bounds__(kThreads) k_b_restrict(const BRes* __restrict__ items,
                                                         const BTile* __restrict__ tiles, int ntiles,
                                                         const BScal* __restrict__ sc) { b_restrict(items, tiles, ntiles, sc); }

// xf[f] += xc[q] (ComputeProlongation_ref.cpp:49); prolongation items carry xc in
// rf and the fine solution in rc
__device__ __forceinline__ void b_prolong(const BRes* __restrict__ items,
                                                        const BTile* __restrict__ tiles, int ntiles,
                                                        const BScal* __restrict__ sc) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BTile tl = tiles[t];
    const BRes it = items[tl.item];
    if (!sc[it.prob].active) continue;
    const int u = tl.start + threadIdx.x;
    if (u >= it.nc) continue;
    it.rc[it.tf[u]] += it.rf[it.tq[u]];
  }
}
__global__ void __launch_bounds__(kThreads) k_b_prolong(const BRes* __restrict__ items,
                                                        const BTile* __restrict__ tiles, int ntiles,
                                                        const BScal* __restrict__ sc) { b_prolong(items, tiles, ntiles, sc); }

// y = A x (FP64 outer SpMV, CG.cpp:118); DOT: partial of x'y per tile
template <bool DOT>
__device__ __forceinline__ void b_spmv(const BVec* __restrict__ v, const BTile* __restrict__ tiles,
                                                     int ntiles, int use_p, const BScal* __restrict__ sc,
                                                     double* __restrict__ partials) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BTile tl = tiles[t];
    const BVec it = v[tl.item];
    double acc = 0.0;
    const bool act = sc == nullptr || sc[tl.item].active;
    const int q = tl.start + threadIdx.x;
    if (act && q < it.n) {
      const double* x = use_p ? it.p : it.x;
      double sum = 0.0, xq = 0.0;
#pragma unroll
      for (int k = 0; k < kSlots; ++k) {
        const double xv = __ldg(x + it.col[k * it.pitch + q]);
        sum += it.val[k * it.pitch + q] * xv;
        if (k == kDiagSlot) xq = xv;
      }
      it.Ap[q] = sum;
      if (DOT) acc = xq * sum;
    }
    if (DOT) {
      const double s = block_sum(acc);
      if (threadIdx.x == 0) partials[t] = s;
    }
  }
}
template <bool DOT>
__global__ void __launch_bounds__(kThreads) k_b_spmv(const BVec* __restrict__ v, const BTile* __restrict__ tiles,
                                                     int ntiles, int use_p, const BScal* __restrict__ sc,
                                                     double* __restrict__ partials) { b_spmv<DOT>(v, tiles, ntiles, use_p, sc, partials); }

// r = 1.0 b + (-1.0) Ap (CG.cpp:88) and partial of r'r
__device__ __forceinline__ void b_resid(const BVec* __restrict__ v, const BTile* __restrict__ tiles,
                                                      int ntiles, double* __restrict__ partials) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BTile tl = tiles[t];
    const BVec it = v[tl.item];
    const int q = tl.start + threadIdx.x;
    double acc = 0.0;
    if (q < it.n) {
      const double r = 1.0 * it.b[q] + -1.0 * it.Ap[q];
      it.r[q] = r;
      acc = r * r;
    }
    const double s = block_sum(acc);
    if (threadIdx.x == 0) partials[t] = s;
  }
}
__global__ void __launch_bounds__(kThreads) k_b_resid(const BVec* __restrict__ v, const BTile* __restrict__ tiles,
                                                      int ntiles, double* __restrict__ partials) { b_resid(v, tiles, ntiles, partials); }

// r32 = (float) r: the FP32 V-cycle's right-hand side
__device__ __forceinline__ void b_to32(const BVec* __restrict__ v, const BTile* __restrict__ tiles,
                                                     int ntiles, const BScal* __restrict__ sc) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BTile tl = tiles[t];
    if (!sc[tl.item].active) continue;
    const BVec it = v[tl.item];
    const int q = tl.start + threadIdx.x;
    if (q < it.n) it.r32[q] = (float)it.r[q];
  }
}
__global__ void __launch_bounds__(kThreads) k_b_to32(const BVec* __restrict__ v, const BTile* __restrict__ tiles,
                                                     int ntiles, const BScal* __restrict__ sc) { b_to32(v, tiles, ntiles, sc); }

// z = (double) x32; partials of r'z and r'zprev (flexible beta)
__device__ __forceinline__ void b_to64_dots(const BVec* __restrict__ v, const BTile* __restrict__ tiles,
                                                          int ntiles, const BScal* __restrict__ sc,
                                                          double* __restrict__ partials) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BTile tl = tiles[t];
    const BVec it = v[tl.item];
    const int q = tl.start + threadIdx.x;
    double a1 = 0.0, a2 = 0.0;
    if (sc[tl.item].active && q < it.n) {
      const double z = (double)it.x32[q];
      it.z[q] = z;
      const double r = it.r[q];
      a1 = r * z;
      a2 = r * it.zprev[q];
    }
    const double s1 = block_sum(a1);
    const double s2 = block_sum(a2);
    if (threadIdx.x == 0) {
      partials[t] = s1;
      partials[ntiles + t] = s2;
    }
  }
}
__global__ void __launch_bounds__(kThreads) k_b_to64_dots(const BVec* __restrict__ v, const BTile* __restrict__ tiles,
                                                          int ntiles, const BScal* __restrict__ sc,
                                                          double* __restrict__ partials) { b_to64_dots(v, tiles, ntiles, sc, partials); }

// iteration 1: p = z; later: p = z + beta p; then zprev = z
__device__ __forceinline__ void b_update_p(const BVec* __restrict__ v, const BTile* __restrict__ tiles,
                                                         int ntiles, const BScal* __restrict__ sc,
                                                         const BCtl* __restrict__ ctl) {
  const bool first = ctl->iter == 0;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BTile tl = tiles[t];
    if (!sc[tl.item].active) continue;
    const BVec it = v[tl.item];
    const double beta = sc[tl.item].beta;
    const int q = tl.start + threadIdx.x;
    if (q < it.n) {
      const double z = it.z[q];
      it.p[q] = first ? z : z + beta * it.p[q];
      it.zprev[q] = z;
    }
  }
}
__global__ void __launch_bounds__(kThreads) k_b_update_p(const BVec* __restrict__ v, const BTile* __restrict__ tiles,
                                                         int ntiles, const BScal* __restrict__ sc,
                                                         const BCtl* __restrict__ ctl) { b_update_p(v, tiles, ntiles, sc, ctl); }

// x += alpha p, r += (-alpha) Ap (CG.cpp:121-122); partial of r'r
__device__ __forceinline__ void b_update_xr(const BVec* __restrict__ v, const BTile* __restrict__ tiles,
                                                          int ntiles, const BScal* __restrict__ sc,
                                                          double* __restrict__ partials) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BTile tl = tiles[t];
    const BVec it = v[tl.item];
    const int q = tl.start + threadIdx.x;
    double acc = 0.0;
    if (q < it.n) {
      double r = it.r[q];
      if (sc[tl.item].active) {
        const double alpha = sc[tl.item].alpha;
        it.x[q] = it.x[q] + alpha * it.p[q];
        r = r + -alpha * it.Ap[q];
        it.r[q] = r;
      }
      acc = r * r;
    }
    const double s = block_sum(acc);
    if (threadIdx.x == 0) partials[t] = s;
  }
}
__global__ void __launch_bounds__(kThreads) k_b_update_xr(const BVec* __restrict__ v, const BTile* __restrict__ tiles,
                                                          int ntiles, const BScal* __restrict__ sc,
                                                          double* __restrict__ partials) { b_update_xr(v, tiles, ntiles, sc, partials); }

// ---- form 1's vector steps: the arithmetic of b_to64_dots and b_update_xr, with
// the partials left per warp (summed by k_b_finalize_warps in the same order)
// instead of two block barriers a tile, and r narrowed for the next V-cycle where
// it is made.
__global__ void __launch_bounds__(kThreads) k_b_to64_dots_w(const BVec* __restrict__ v,
                                                            const BTile* __restrict__ tiles, int ntiles,
                                                            const BScal* __restrict__ sc,
                                                            double* __restrict__ partials) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BTile tl = tiles[t];
    if (!sc[tl.item].active) continue;  // its sums are not read
    const BVec& it = v[tl.item];
    const int q = tl.start + threadIdx.x;
    double a1 = 0.0, a2 = 0.0;
    if (q < it.n) {
      const double z = (double)it.x32[q];
      it.z[q] = z;
      const double r = it.r[q];
      a1 = r * z;
      a2 = r * it.zprev[q];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a1 += __shfl_down_sync(0xffffffffu, a1, o);
      a2 += __shfl_down_sync(0xffffffffu, a2, o);
    }
    if ((threadIdx.x & 31) == 0) {
      const int64_t w = 8 * (int64_t)t + (threadIdx.x >> 5);
      partials[w] = a1;
      partials[8 * (int64_t)ntiles + w] = a2;
    }
  }
}

__global__ void __launch_bounds__(kThreads) k_b_update_xr_w(const BVec* __restrict__ v,
                                                            const BTile* __restrict__ tiles, int ntiles,
                                                            const BScal* __restrict__ sc,
                                                            double* __restrict__ partials) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BTile tl = tiles[t];
    if (!sc[tl.item].active) continue;  // its norm stays
    const BVec& it = v[tl.item];
    const int q = tl.start + threadIdx.x;
    double acc = 0.0;
    if (q < it.n) {
      const double alpha = sc[tl.item].alpha;
      it.x[q] = it.x[q] + alpha * it.p[q];
      const double r = it.r[q] + -alpha * it.Ap[q];
      it.r[q] = r;
      it.r32[q] = (float)r;
      acc = r * r;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) partials[8 * (int64_t)t + (threadIdx.x >> 5)] = acc;
  }
}

enum BFin : int { kBNorm0 = 0, kBRtz = 1, kBPap = 2, kBNormr = 3 };

// The sum of a 256-row tile from its eight warps' sums, in block_sum's order.
__device__ __forceinline__ double tile_of_warps(const double* __restrict__ w) {
  return ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
}

// Problem p's fixed-order sum over its tiles, then its scalar step; block b
// takes problems b, b + gridDim.x, ... WARPS: the partials are the tiles' warps'.
template <bool WARPS = false>
__device__ __forceinline__ void b_finalize(BScal* sc, const double* __restrict__ partials, int ntiles,
                                           const int* __restrict__ range, int op, const BCtl* __restrict__ ctl,
                                           int m) {
  for (int p = blockIdx.x; p < m; p += gridDim.x) {
    const int t0 = range[p], t1 = range[p + 1];
    if (WARPS && !sc[p].active) continue;  // no sums were left for it, and its scalars stay
    double a1 = 0.0, a2 = 0.0;
    if (WARPS) {
#pragma unroll 4
      for (int t = t0 + threadIdx.x; t < t1; t += blockDim.x) a1 += tile_of_warps(partials + 8 * (int64_t)t);
      if (op == kBRtz) {
#pragma unroll 4
        for (int t = t0 + threadIdx.x; t < t1; t += blockDim.x)
          a2 += tile_of_warps(partials + 8 * ((int64_t)ntiles + t));
      }
    } else {
      for (int t = t0 + threadIdx.x; t < t1; t += blockDim.x) {
        a1 += partials[t];
        if (op == kBRtz) a2 += partials[ntiles + t];
      }
    }
    const double s1 = block_sum(a1);
    const double s2 = op == kBRtz ? block_sum(a2) : 0.0;
    if (threadIdx.x != 0) continue;
    BScal& s = sc[p];
    switch (op) {
      case kBNorm0:
        s.normr2 = s1;
        s.normr0 = sqrt(s1);
        s.active = s.normr0 / s.normr0 > ctl->tol ? 1 : 0;
        s.niters = 0;
        break;
      case kBRtz:
        if (!s.active) break;
        if (ctl->iter == 0) {
          s.rtz = s1;
        } else {
          s.oldrtz = s.rtz;
          s.rtz = s1;
          s.rzprev = s2;
          s.beta = (s1 - s2) / s.oldrtz;  // Polak-Ribiere
        }
        break;
      case kBPap:
        if (!s.active) break;
        s.pAp = s1;
        s.alpha = s.rtz / s1;
        break;
      case kBNormr:
        s.normr2 = s1;
        if (s.active) {
          s.niters = ctl->iter + 1;
          s.active = sqrt(s1) / s.normr0 > ctl->tol ? 1 : 0;
        }
        break;
      default: break;
    }
  }
}

// One block per problem.
__global__ void __launch_bounds__(kThreads) k_b_finalize_warps(BScal* sc, const double* __restrict__ partials,
                                                               int ntiles, const int* __restrict__ range, int op,
                                                               const BCtl* __restrict__ ctl, int m) {
  b_finalize<true>(sc, partials, ntiles, range, op, ctl, m);
}
__global__ void __launch_bounds__(kThreads) k_b_finalize(BScal* sc, const double* __restrict__ partials,
                                                         int ntiles, const int* __restrict__ range, int op,
                                                         const BCtl* __restrict__ ctl, int m) {
  b_finalize(sc, partials, ntiles, range, op, ctl, m);
}

// ---- the whole iteration in one launch ------------------------------------------
// A cooperative launch (every block resident at once) walks the iteration's
// steps, the same work lists as the launches above, in the same order, with a
// grid barrier wherever a step reads what the step before wrote. So each
// problem computes the same bits as with one launch per step on the register
// kernels.
//
// The barrier: every block's thread 0 reads the generation word, arrives on
// the counter, and the last to arrive zeroes the counter and advances the
// generation; the others wait for the generation to move. The two words sit on
// separate 128-byte lines, so the waiting blocks' polls do not queue behind the
// arrivals. Each wait gives up after kBatchWaitNs of global time: it records
// fault code 5 in the context's fault word and the block leaves the kernel. A block that left stops arriving,
// so every other block's next wait runs out too and the launch ends; the
// loop's condition kernel reads the fault word and ends the loop, and the
// host's stream synchronisation returns HPCG_B200_ERR_TIMEOUT.
constexpr unsigned long long kBatchWaitNs = 1000000000ull;  // 1 s per wait

// The barrier's state (device memory): arrivals, and the generation on a line
// of its own.
struct BBar {
  unsigned count;
  unsigned pad0[31];
  unsigned gen;
  unsigned pad1[31];
};

// A load of the generation word from L2 without acquire semantics: an acquire
// at GPU scope also discards the SM's L1 contents, and a block polling on an
// SM where other blocks still work would take their cached lines away with
// every poll. The waiter orders itself once, with the fence after the loop.
__device__ __forceinline__ unsigned ld_relaxed_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// true once every one of the `expected` blocks has arrived; false if the wait
// gave up (the caller leaves the kernel)
__device__ __forceinline__ bool grid_barrier(BBar* bar, unsigned expected, unsigned* fault,
                                             unsigned long long limit_ns = kBatchWaitNs) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    ok = 1;
    const unsigned g = ld_relaxed_u32(&bar->gen);  // cannot move before this block arrives
    __threadfence();  // this block's writes are visible before its arrival
    if (atomicAdd(&bar->count, 1u) + 1u == expected) {
      bar->count = 0;  // nobody touches the counter until the generation moves
      __threadfence();
      asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&bar->gen), "r"(g + 1u) : "memory");
    } else {
      const unsigned long long t0 = global_ns();
      unsigned pause = 32;  // polls back off to one per ~0.5 us: fewer loads on the line while steps run
      while (ld_relaxed_u32(&bar->gen) == g) {
        if (global_ns() - t0 > limit_ns) {
          record_fault(fault, 5);
          ok = 0;
          break;
        }
        __nanosleep(pause);
        pause = pause < 512 ? pause * 2 : 512;
      }
    }
    __threadfence();  // with the load that saw the new generation: the other blocks' writes are visible
  }
  __syncthreads();
  return ok != 0;
}

// A step of the V-cycle on the device: 0 colour phase, 1 restriction, 2 prolongation.
struct DStep {
  int kind, tile_off, ntiles;
};

struct BIter {
  const DStep* steps;
  int nsteps;
  const BGs* gs_items;
  const BRes* res_items;
  const BTile* tiles;
  const BVec* vec;
  const BTile* vtiles;
  int nvt;
  const int* vrange;
  double* partials;
  BScal* sc;
  const BCtl* ctl;
  int m;
  BBar* bar;
  unsigned* fault;
  int vcycle_only;  // 1: the V-cycle's steps alone (timing at creation)
};

// One flexible-CG iteration of every active problem (the launches of
// iteration() below, in one launch).
__global__ void __launch_bounds__(kThreads) k_b_iteration(BIter a) {
  const unsigned nb = gridDim.x;
  if (*(volatile unsigned*)a.fault) return;  // an earlier launch gave up: do nothing
  if (!a.vcycle_only) {
    b_to32(a.vec, a.vtiles, a.nvt, a.sc);
    if (!grid_barrier(a.bar, nb, a.fault)) return;
  }
  for (int i = 0; i < a.nsteps; ++i) {
    const DStep st = a.steps[i];
    if (st.kind == 0)
      b_gs(a.gs_items, a.tiles + st.tile_off, st.ntiles, a.sc);
    else if (st.kind == 1)
      b_restrict(a.res_items, a.tiles + st.tile_off, st.ntiles, a.sc);
    else
      b_prolong(a.res_items, a.tiles + st.tile_off, st.ntiles, a.sc);
    if (!grid_barrier(a.bar, nb, a.fault)) return;
  }
  if (a.vcycle_only) return;
  b_to64_dots(a.vec, a.vtiles, a.nvt, a.sc, a.partials);
  if (!grid_barrier(a.bar, nb, a.fault)) return;
  b_finalize(a.sc, a.partials, a.nvt, a.vrange, kBRtz, a.ctl, a.m);
  if (!grid_barrier(a.bar, nb, a.fault)) return;
  b_update_p(a.vec, a.vtiles, a.nvt, a.sc, a.ctl);
  if (!grid_barrier(a.bar, nb, a.fault)) return;
  b_spmv<true>(a.vec, a.vtiles, a.nvt, 1, a.sc, a.partials);
  if (!grid_barrier(a.bar, nb, a.fault)) return;
  b_finalize(a.sc, a.partials, a.nvt, a.vrange, kBPap, a.ctl, a.m);
  if (!grid_barrier(a.bar, nb, a.fault)) return;
  b_update_xr(a.vec, a.vtiles, a.nvt, a.sc, a.partials);
  if (!grid_barrier(a.bar, nb, a.fault)) return;
  b_finalize(a.sc, a.partials, a.nvt, a.vrange, kBNormr, a.ctl, a.m);
}

// Check of the barrier's bounded wait: every block waits for one more arrival
// than the grid holds, so every wait runs out; records fault code 5 and returns.
__global__ void __launch_bounds__(kThreads) k_b_barrier_selftest(BBar* bar, unsigned long long limit_ns,
                                                                 unsigned* fault) {
  grid_barrier(bar, gridDim.x + 1, fault, limit_ns);
}

__global__ void k_b_setup(BCtl* ctl, int max_iter, double tol) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl->iter = 0;
    ctl->max_iter = max_iter;
    ctl->tol = tol;
  }
}

// while (iter < max_iter && any problem active), and no bounded wait gave up;
// also zeroes the one-launch iteration's barrier counter
__global__ void k_b_condition(BCtl* ctl, const BScal* __restrict__ sc, int m, cudaGraphConditionalHandle h,
                              int advance, BBar* bar, const unsigned* fault) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  if (advance) ctl->iter += 1;
  bool any = false;
  for (int p = 0; p < m; ++p) any = any || sc[p].active;
  bar->count = 0;
  const bool gave_up = *(volatile const unsigned*)fault != 0;
  cudaGraphSetConditional(h, any && !gave_up && ctl->iter < ctl->max_iter ? 1u : 0u);
}

// ---- host ---------------------------------------------------------------------

struct Step {
  int kind;      // 0 = GS phase, 1 = restriction, 2 = prolongation
  int item_off;  // first item of the step (tiles index the whole item array)
  int tile_off;  // first tile of the step
  int ntiles;
};

// A step of form 1's V-cycle.
struct GeoStep {
  enum Kind { kFull, kFirst, kRestrict, kProlong, kTail } kind;
  int s;         // kFirst: sweep position
  int tile_off;  // first tile
  int ntiles;
  int item_off;  // kFull: first item, items
  int nitems;
  int shared;    // kFull: whether an item's colours may meet in 32 bytes (GeoPhase::shared)
};

}  // namespace
}  // namespace hb

struct hpcg_b200_batch {
  uint64_t magic;
  int device;
  hb::Context* ctx;
  int m;
  std::vector<hpcg_b200_problem*> probs;
  // work lists (device) and the V-cycle's step sequence
  hb::BGs* gs_items;
  hb::BRes* res_items;
  hb::BTile* tiles;
  bool bulk;           // form 1
  bool persist;        // form 2: the whole iteration as one cooperative launch (k_b_iteration)
  // form 1's work lists (device) and steps
  hb::BGeo* geo_items;
  hb::BGeoTile* geo_tiles;
  hb::BRes* prolong_items;
  hb::BTile* prolong_tiles;
  hb::GeoGrid* grids;            // [m] level 0, and its tensor map
  hb::BMap* maps;
  hb::BTile* mv_tiles;           // 128-row tiles of every problem's level 0
  int mv_ntiles;
  int* mv_tile0;                 // [m + 1] first of each problem
  double* mv_partials;
  std::vector<int> tail_at;      // first level in the one-launch part
  hb::TailDesc<float>* descs;    // [m] the small levels (nlev 0: none)
  std::vector<hb::GeoStep> geo_steps;
  int tail_cluster;              // blocks of a cluster
  size_t tail_smem;
  int persist_grid;    // its blocks: as many as the SMs hold at once
  hb::DStep* dsteps;   // the V-cycle's steps for k_b_iteration
  hb::BBar* bar;       // its grid barrier
  std::vector<hb::Step> steps;
  hb::BVec* vec;
  hb::BTile* vtiles;  // row tiles of every problem's level 0
  int nvt;
  int* vrange;        // [m+1] tile range of each problem
  double* partials;   // [2 * nvt]
  hb::BScal* sc;
  hb::BScal* sc_host;
  hb::BCtl* ctl;
  // slot-major FP32 values of every problem's levels, [problem * kMaxLevels + level]:
  // the batched kernels walk tiles of 256 rows, for which the single-problem
  // path's blocked FP32 layout was measured slower
  std::vector<float*> val32;
  size_t bytes;
  cudaGraphExec_t graph;
};

namespace hb {
namespace {

bool valid_batch(const hpcg_b200_batch* b) { return b && b->magic == kBatchMagic; }

int alloc_copy(hpcg_b200_batch* B, void** dst, const void* src, size_t bytes) {
  HB_TRY(dev_alloc(dst, bytes, &B->bytes));
  HB_CK(cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice));
  return HPCG_B200_OK;
}

// FP32 copy of FP64 values, element for element (round to nearest).
__global__ void k_narrow(float* __restrict__ dst, const double* __restrict__ src, int64_t n) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) dst[i] = (float)src[i];
}

void tiles_of(std::vector<BTile>& tiles, int item, int r0, int r1) {
  for (int s = r0; s < r1; s += kTile) tiles.push_back({item, s});
}

// The V-cycle of every problem as one step sequence (ComputeMG_ref.cpp:39-63
// with the colour sweeps of the single-problem path): level l pre-smooth
// (forward from x = 0, backward without the last colour), restriction,
// recursion, prolongation, post-smooth; the coarsest level one symmetric sweep.
void build_vcycle(hpcg_b200_batch* B, int l, std::vector<BGs>& gs, std::vector<BRes>& res,
                  std::vector<BTile>& tiles) {
  auto phase = [&](int s, bool first) {
    Step st{0, (int)gs.size(), (int)tiles.size(), 0};
    for (int p = 0; p < B->m; ++p) {
      const Level& L = B->probs[p]->lev[l];
      const int item = (int)gs.size();
      BGs it;
      it.val = B->val32[p * kMaxLevels + l];
      it.col = L.col;
      it.pitch = L.pitch;
      it.rhs = L.r32;
      it.x = L.x32;
      it.r0 = L.g.start[s];
      it.r1 = L.g.start[s + 1];
      it.mask = first ? first_mask(L.g, s) : kAllSlots;
      it.first = first ? 1 : 0;
      it.prob = p;
      gs.push_back(it);
      tiles_of(tiles, item, it.r0, it.r1);
    }
    st.ntiles = (int)tiles.size() - st.tile_off;
    B->steps.push_back(st);
  };
  auto sweep = [&](bool first) {
    for (int s = 0; s < kColours; ++s) phase(s, first);
    for (int s = kColours - 2; s >= 0; --s) phase(s, false);
  };
  auto transfer = [&](int kind) {
    Step st{kind, (int)res.size(), (int)tiles.size(), 0};
    for (int p = 0; p < B->m; ++p) {
      const Level& L = B->probs[p]->lev[l];
      const Level& C = B->probs[p]->lev[l + 1];
      const int item = (int)res.size();
      BRes it;
      it.val = B->val32[p * kMaxLevels + l];
      it.col = L.col;
      it.pitch = L.pitch;
      it.tf = L.tf;
      it.tq = L.tq;
      it.nc = C.n;
      it.prob = p;
      if (kind == 1) {  // rc = rf - A xf
        it.rf = L.r32;
        it.xf = L.x32;
        it.rc = C.r32;
      } else {  // xf += xc: xc travels in rf, the fine solution in rc
        it.rf = C.x32;
        it.xf = nullptr;
        it.rc = L.x32;
      }
      res.push_back(it);
      tiles_of(tiles, item, 0, it.nc);
    }
    st.ntiles = (int)tiles.size() - st.tile_off;
    B->steps.push_back(st);
  };
  sweep(true);
  if (l + 1 < 4) {
    transfer(1);
    build_vcycle(B, l + 1, gs, res, tiles);
    transfer(2);
    sweep(false);
  }
}

// Form 1's V-cycle: as build_vcycle, problem p taking part in the steps of the
// levels above tail_first; the rest is one launch.
struct GeoLists {
  std::vector<BGeo> items;
  std::vector<BGeoTile> tiles;
  std::vector<BRes> res;
  std::vector<BTile> rtiles;
};
void build_geo(hpcg_b200_batch* B, int l, GeoLists& W) {
  const int m = B->m;
  std::vector<int> in;
  for (int p = 0; p < m; ++p)
    if (l < kMaxLevels && B->tail_at[p] > l) in.push_back(p);
  if (in.empty() || l >= kMaxLevels) {  // the others' levels are done above: now the small ones of all
    bool any = false;
    for (int p = 0; p < m; ++p) any = any || B->tail_at[p] < B->probs[p]->nlev;
    if (any) B->geo_steps.push_back(GeoStep{GeoStep::kTail, 0, 0, 0, 0, 0, 0});
    return;
  }
  auto step = [&](GeoStep::Kind kind, int s, int rows) {
    GeoStep st{kind, s, (int)W.tiles.size(), 0, (int)W.items.size(), (int)in.size(), 0};
    for (int p : in) {
      const Level& L = B->probs[p]->lev[l];
      const int item = (int)W.items.size();
      BGeo it;
      it.val = L.val32;
      it.rhs = L.r32;
      it.x = L.x32;
      it.rc = kind == GeoStep::kRestrict ? B->probs[p]->lev[l + 1].r32 : nullptr;
      it.tq = L.tq;
      it.r0 = L.g.start[s];
      it.r1 = L.g.start[s + 1];
      it.sink = sink_of(L);
      it.prob = p;
      it.geo = L.geo_cols->block[s];
      st.shared |= it.geo.shared;
      W.items.push_back(it);
      // whole-block tiles for the copies, from the first row for the others
      const int first = kind == GeoStep::kFull ? it.r0 / rows * rows : it.r0;
      for (int q = first; q < it.r1; q += rows)
        W.tiles.push_back(BGeoTile{L.val32 + mat_index<float>(0, q, 0), item, q, p, 0});
    }
    st.ntiles = (int)W.tiles.size() - st.tile_off;
    B->geo_steps.push_back(st);
  };
  auto sweep = [&](bool first) {
    for (int s = 0; s < kColours; ++s)
      step(first ? GeoStep::kFirst : GeoStep::kFull, s, first ? kTile : BatchShape::tile_rows);
    for (int s = kColours - 2; s >= 0; --s) step(GeoStep::kFull, s, BatchShape::tile_rows);
  };
  sweep(true);
  if (l + 1 < kMaxLevels) {
    step(GeoStep::kRestrict, kColours - 1, kTile);
    build_geo(B, l + 1, W);
    GeoStep st{GeoStep::kProlong, 0, (int)W.rtiles.size(), 0, 0, 0, 0};
    for (int p : in) {
      const Level& L = B->probs[p]->lev[l];
      const Level& C = B->probs[p]->lev[l + 1];
      const int item = (int)W.res.size();
      BRes it{};
      it.tf = L.tf;
      it.tq = L.tq;
      it.nc = C.n;
      it.prob = p;
      it.rf = C.x32;
      it.rc = L.x32;
      W.res.push_back(it);
      tiles_of(W.rtiles, item, 0, it.nc);
    }
    st.ntiles = (int)W.rtiles.size() - st.tile_off;
    B->geo_steps.push_back(st);
    sweep(false);
  } else {
    build_geo(B, l + 1, W);
  }
}

int grid_tiles(Context* c, int ntiles) {
  int g = c->sms * kBlocksPerSm;
  return ntiles < g ? (ntiles < 1 ? 1 : ntiles) : g;
}

int launch_step(hpcg_b200_batch* B, const Step& s) {
  Context* c = B->ctx;
  const int g = grid_tiles(c, s.ntiles);
  // tiles hold indices into the whole item array, so the items go in unshifted
  if (s.kind == 0)
    k_b_gs<<<g, kThreads, 0, c->stream>>>(B->gs_items, B->tiles + s.tile_off, s.ntiles, B->sc);
  else if (s.kind == 1)
    k_b_restrict<<<g, kThreads, 0, c->stream>>>(B->res_items, B->tiles + s.tile_off, s.ntiles, B->sc);
  else
    k_b_prolong<<<g, kThreads, 0, c->stream>>>(B->res_items, B->tiles + s.tile_off, s.ntiles, B->sc);
  HB_CK(cudaGetLastError());
  return HPCG_B200_OK;
}

template <int S>
void launch_first_geo(hpcg_b200_batch* B, const GeoStep& st) {
  Context* c = B->ctx;
  k_b_first_geo<first_mask_default(S)><<<grid_tiles(c, st.ntiles), kThreads, 0, c->stream>>>(
      B->geo_items, B->geo_tiles + st.tile_off, st.ntiles, B->sc);
}

int launch_geo_step(hpcg_b200_batch* B, const GeoStep& st) {
  Context* c = B->ctx;
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const BGeoTile* tiles = B->geo_tiles + st.tile_off;
  switch (st.kind) {
    case GeoStep::kFull: {
      static std::atomic<uint64_t> attr_set{0};  // devices on which the shared-memory size is enabled
      bulk_attr(k_b_gs_geo, BatchShape::smem, c->device, &attr_set);
      // early launch: the producer reads values and, for the tiles to skip, the
      // convergence flags, which are written before a plainly launched kernel
      // (a first-sweep phase, a prolongation) of every V-cycle
      HB_CK(launch_early(c->stream, k_b_gs_geo, std::max(1, std::min(st.ntiles, c->sms)), BatchShape::threads,
                         BatchShape::smem, B->geo_items, st.item_off, st.nitems, tiles, st.ntiles, B->sc, c->fault,
                         st.shared));
      return HPCG_B200_OK;
    }
    case GeoStep::kFirst:
      switch (st.s) {
        case 0: launch_first_geo<0>(B, st); break;
        case 1: launch_first_geo<1>(B, st); break;
        case 2: launch_first_geo<2>(B, st); break;
        case 3: launch_first_geo<3>(B, st); break;
        case 4: launch_first_geo<4>(B, st); break;
        case 5: launch_first_geo<5>(B, st); break;
        case 6: launch_first_geo<6>(B, st); break;
        default: launch_first_geo<7>(B, st); break;
      }
      break;
    case GeoStep::kRestrict:
      k_b_restrict_geo<<<grid_tiles(c, st.ntiles), kThreads, 0, c->stream>>>(B->geo_items, tiles, st.ntiles, B->sc);
      break;
    case GeoStep::kProlong:
      k_b_prolong<<<grid_tiles(c, st.ntiles), kThreads, 0, c->stream>>>(
          B->prolong_items, B->prolong_tiles + st.tile_off, st.ntiles, B->sc);
      break;
    case GeoStep::kTail:
      cfg.gridDim = dim3(B->m * B->tail_cluster);
      cfg.blockDim = dim3(kTailThreads);
      cfg.dynamicSmemBytes = B->tail_smem;
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = B->tail_cluster;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      HB_CK(cudaLaunchKernelEx(&cfg, k_b_tail, (const TailDesc<float>*)B->descs, (const BScal*)B->sc, c->fault));
      return HPCG_B200_OK;
  }
  HB_CK(cudaGetLastError());
  return HPCG_B200_OK;
}

int finalize_b(hpcg_b200_batch* B, int op) {
  k_b_finalize<<<B->m, kThreads, 0, B->ctx->stream>>>(B->sc, B->partials, B->nvt, B->vrange, op, B->ctl, B->m);
  HB_CK(cudaGetLastError());
  return HPCG_B200_OK;
}

int finalize_w(hpcg_b200_batch* B, int op) {
  k_b_finalize_warps<<<B->m, kThreads, 0, B->ctx->stream>>>(B->sc, B->mv_partials, B->nvt, B->vrange, op, B->ctl,
                                                            B->m);
  HB_CK(cudaGetLastError());
  return HPCG_B200_OK;
}

// one flexible-CG iteration of every active problem, form 1 (r32 holds r)
int iteration_geo(hpcg_b200_batch* B) {
  Context* c = B->ctx;
  const int gv = grid_tiles(c, B->nvt);
  for (const GeoStep& s : B->geo_steps) HB_TRY(launch_geo_step(B, s));
  k_b_to64_dots_w<<<gv, kThreads, 0, c->stream>>>(B->vec, B->vtiles, B->nvt, B->sc, B->mv_partials);
  HB_CK(cudaGetLastError());
  HB_TRY(finalize_w(B, kBRtz));
  k_b_update_p<<<gv, kThreads, 0, c->stream>>>(B->vec, B->vtiles, B->nvt, B->sc, B->ctl);
  static std::atomic<uint64_t> attr_set{0};  // devices on which the shared-memory size is enabled
  bulk_attr(k_b_spmv_geo, BatchSpmv::smem, c->device, &attr_set);
  k_b_spmv_geo<<<std::min(B->mv_ntiles, c->sms), BatchSpmv::threads, BatchSpmv::smem, c->stream>>>(
      B->vec, B->grids, B->m, B->maps, B->mv_tiles, B->mv_ntiles, B->mv_tile0, B->sc, B->mv_partials, c->fault);
  HB_CK(cudaGetLastError());
  HB_TRY(finalize_w(B, kBPap));
  k_b_update_xr_w<<<gv, kThreads, 0, c->stream>>>(B->vec, B->vtiles, B->nvt, B->sc, B->mv_partials);
  HB_CK(cudaGetLastError());
  return finalize_w(B, kBNormr);
}

// ... and form 0
int iteration(hpcg_b200_batch* B) {
  Context* c = B->ctx;
  const int gv = grid_tiles(c, B->nvt);
  k_b_to32<<<gv, kThreads, 0, c->stream>>>(B->vec, B->vtiles, B->nvt, B->sc);
  HB_CK(cudaGetLastError());
  for (const Step& s : B->steps) HB_TRY(launch_step(B, s));
  k_b_to64_dots<<<gv, kThreads, 0, c->stream>>>(B->vec, B->vtiles, B->nvt, B->sc, B->partials);
  HB_CK(cudaGetLastError());
  HB_TRY(finalize_b(B, kBRtz));
  k_b_update_p<<<gv, kThreads, 0, c->stream>>>(B->vec, B->vtiles, B->nvt, B->sc, B->ctl);
  k_b_spmv<true><<<gv, kThreads, 0, c->stream>>>(B->vec, B->vtiles, B->nvt, 1, B->sc, B->partials);
  HB_CK(cudaGetLastError());
  HB_TRY(finalize_b(B, kBPap));
  k_b_update_xr<<<gv, kThreads, 0, c->stream>>>(B->vec, B->vtiles, B->nvt, B->sc, B->partials);
  HB_CK(cudaGetLastError());
  return finalize_b(B, kBNormr);
}

// k_b_iteration as a cooperative launch (vcycle_only: the V-cycle's steps alone)
int launch_iteration(hpcg_b200_batch* B, bool vcycle_only) {
  Context* c = B->ctx;
  if (B->persist_grid < 1) return HPCG_B200_ERR_UNSUPPORTED;
  BIter a;
  a.steps = B->dsteps;
  a.nsteps = (int)B->steps.size();
  a.gs_items = B->gs_items;
  a.res_items = B->res_items;
  a.tiles = B->tiles;
  a.vec = B->vec;
  a.vtiles = B->vtiles;
  a.nvt = B->nvt;
  a.vrange = B->vrange;
  a.partials = B->partials;
  a.sc = B->sc;
  a.ctl = B->ctl;
  a.m = B->m;
  a.bar = B->bar;
  a.fault = c->fault;
  a.vcycle_only = vcycle_only ? 1 : 0;
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(B->persist_grid);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  HB_CK(cudaMemsetAsync(B->bar, 0, sizeof(BBar), c->stream));  // the barrier counts from zero each launch
  HB_CK(cudaLaunchKernelEx(&cfg, k_b_iteration, a));
  return HPCG_B200_OK;
}

int end_capture_b(cudaStream_t st, int status) {
  cudaGraph_t g = nullptr;
  const cudaError_t e = cudaStreamEndCapture(st, &g);
  if (status == HPCG_B200_OK && e != cudaSuccess) {
    set_error("cudaStreamEndCapture", e);
    return status_of(e);
  }
  return status;
}

int build_graph(hpcg_b200_batch* B) {
  Context* c = B->ctx;
  cudaGraph_t g = nullptr;
  HB_CK(cudaGraphCreate(&g, 0));
  cudaGraphConditionalHandle h;
  cudaError_t e = cudaGraphConditionalHandleCreate(&h, g, 0, cudaGraphCondAssignDefault);
  int st = HPCG_B200_OK;
  if (e == cudaSuccess) e = cudaStreamBeginCaptureToGraph(c->stream, g, nullptr, nullptr, 0,
                                                            cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    k_b_condition<<<1, 32, 0, c->stream>>>(B->ctl, B->sc, B->m, h, 0, B->bar, c->fault);
    e = cudaGetLastError();
    st = end_capture_b(c->stream, e == cudaSuccess ? HPCG_B200_OK : status_of(e));
  }
  size_t num = 0;
  cudaGraphNode_t init = nullptr;
  if (e == cudaSuccess && st == HPCG_B200_OK) e = cudaGraphGetNodes(g, nullptr, &num);
  if (e == cudaSuccess && st == HPCG_B200_OK && num == 1) e = cudaGraphGetNodes(g, &init, &num);
  alignas(cudaGraphNodeParams) unsigned char buf[sizeof(cudaGraphNodeParams)];
  std::memset(buf, 0, sizeof(buf));
  cudaGraphNodeParams& cp = *reinterpret_cast<cudaGraphNodeParams*>(buf);
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = h;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  cudaGraphNode_t loop = nullptr;
  if (e == cudaSuccess && st == HPCG_B200_OK) e = cudaGraphAddNode(&loop, g, &init, 1, &cp);
  if (e == cudaSuccess && st == HPCG_B200_OK)
    e = cudaStreamBeginCaptureToGraph(c->stream, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                      cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess || st != HPCG_B200_OK) {
    cudaGraphDestroy(g);
    if (e != cudaSuccess) set_error("batch graph", e);
    return st != HPCG_B200_OK ? st : status_of(e);
  }
  st = B->persist ? launch_iteration(B, false) : B->bulk ? iteration_geo(B) : iteration(B);
  if (st == HPCG_B200_OK) {
    k_b_condition<<<1, 32, 0, c->stream>>>(B->ctl, B->sc, B->m, h, 1, B->bar, c->fault);
    if (cudaGetLastError() != cudaSuccess) st = HPCG_B200_ERR_CUDA;
  }
  st = end_capture_b(c->stream, st);
  if (st == HPCG_B200_OK) {
    e = cudaGraphInstantiate(&B->graph, g, 0);
    if (e != cudaSuccess) {
      set_error("cudaGraphInstantiate (batch)", e);
      st = status_of(e);
    }
  }
  cudaGraphDestroy(g);
  return st;
}

// The form of an iteration (hpcg_b200_batch_form): 1, the bulk-copy phases with
// columns from the grid and the small levels in one launch, where every level's
// columns follow from its grid (every batch unless HPCG_B200_PACKED asks for
// stored ones), else 0, one launch per step on the register kernels.
// HPCG_B200_BATCH_PERSIST=1: 2, the whole iteration as one cooperative launch;
// HPCG_B200_BATCH_BULK=0 (or PERSIST=0 without BULK=1): 0. Sixteen problems of
// sides 32 to 128: form 1 takes 54 ms to 1e-9, form 0 105.
int choose_form(hpcg_b200_batch* B) {
  const char* fp = std::getenv("HPCG_B200_BATCH_PERSIST");
  const char* fb = std::getenv("HPCG_B200_BATCH_BULK");
  bool geo = true;
  for (hpcg_b200_problem* p : B->probs)
    for (int l = 0; l < p->nlev; ++l) geo = geo && p->lev[l].geo_cols && (l + 1 == p->nlev || p->lev[l].tf_run >= 0);
  for (hpcg_b200_problem* p : B->probs) geo = geo && bulk_maps(p->lev[0]) != nullptr;
  const bool want = fb && *fb ? std::atoi(fb) != 0 : !(fp && *fp);
  B->persist = fp && *fp && std::atoi(fp) != 0 && B->persist_grid > 0;
  B->bulk = !B->persist && geo && want;
  return HPCG_B200_OK;
}

constexpr int kBatchTailRows = 1280;

// Form 1's work lists.
int build_form1(hpcg_b200_batch* B) {
  // One cut for all problems, the first level at which every problem fits: a
  // level that some problem needs launches for costs the others' rows little
  // there, and the one-launch part as long as its longest cluster. There the
  // problems run side by side, so up to five chunks of rows a phase (2.2 us)
  // still beat a launch for every phase. With more clusters than the GPU holds
  // at one block to an SM, two blocks share one.
  int cut = 0;
  for (hpcg_b200_problem* p : B->probs)
    cut = std::max(cut, tail_first_within(p, true, kBatchTailRows, B->m > 8 ? 110 * 1024 : 200 * 1024));
  std::vector<TailDesc<float>> descs(B->m);
  for (;; ++cut) {
    B->tail_cluster = 1;
    B->tail_smem = 0;
    bool any = false;
    for (int p = 0; p < B->m; ++p) {
      hpcg_b200_problem* P = B->probs[p];
      std::memset(&descs[p], 0, sizeof(descs[p]));
      if (cut >= P->nlev) continue;
      any = true;
      size_t smem = 0;
      B->tail_cluster = std::max(B->tail_cluster, tail_desc(P, cut, P->nlev - cut, &descs[p], &smem));
      B->tail_smem = std::max(B->tail_smem, smem);
    }
    if (!any || tail_fits((const void*)k_b_tail, B->tail_cluster, B->tail_smem)) break;
  }
  B->tail_at.assign(B->m, cut);
  GeoLists W;
  build_geo(B, 0, W);
  std::vector<GeoGrid> grids;
  for (hpcg_b200_problem* P : B->probs) grids.push_back(*P->lev[0].geo_cols);
  HB_TRY(alloc_copy(B, (void**)&B->geo_items, W.items.data(), sizeof(BGeo) * W.items.size()));
  HB_TRY(alloc_copy(B, (void**)&B->geo_tiles, W.tiles.data(), sizeof(BGeoTile) * W.tiles.size()));
  HB_TRY(alloc_copy(B, (void**)&B->prolong_items, W.res.data(), sizeof(BRes) * W.res.size()));
  HB_TRY(alloc_copy(B, (void**)&B->prolong_tiles, W.rtiles.data(), sizeof(BTile) * W.rtiles.size()));
  HB_TRY(alloc_copy(B, (void**)&B->grids, grids.data(), sizeof(GeoGrid) * grids.size()));
  std::vector<BMap> maps(B->m);
  std::vector<BTile> mv;
  std::vector<int> tile0(B->m + 1, 0);
  for (int p = 0; p < B->m; ++p) {
    const Level& L = B->probs[p]->lev[0];
    std::memcpy(&maps[p].map, &bulk_maps(L)->val, sizeof(CUtensorMap));
    for (int q = 0; q < L.n; q += kBulkRows) mv.push_back(BTile{p, q});
    tile0[p + 1] = (int)mv.size();
  }
  B->mv_ntiles = (int)mv.size();
  HB_TRY(alloc_copy(B, (void**)&B->maps, maps.data(), sizeof(BMap) * maps.size()));
  HB_TRY(alloc_copy(B, (void**)&B->mv_tiles, mv.data(), sizeof(BTile) * mv.size()));
  HB_TRY(alloc_copy(B, (void**)&B->mv_tile0, tile0.data(), sizeof(int) * tile0.size()));
  HB_TRY(dev_alloc((void**)&B->mv_partials, sizeof(double) * 16 * B->nvt, &B->bytes));  // two sums, 8 warps a tile
  return alloc_copy(B, (void**)&B->descs, descs.data(), sizeof(TailDesc<float>) * descs.size());
}

// Forms 0 and 2: slot-major FP32 values and the work lists of the register kernels.
int build_register_forms(hpcg_b200_batch* B) {
  Context* c = B->ctx;
  for (hpcg_b200_problem* p : B->probs)
    for (int l = 0; l < kMaxLevels; ++l) {
      float* v = nullptr;
      if (l < p->nlev) {
        const int64_t cnt = (int64_t)kSlots * p->lev[l].pitch;
        HB_TRY(dev_alloc((void**)&v, sizeof(float) * cnt, &B->bytes));
        B->val32.push_back(v);
        k_narrow<<<grid_for(c, cnt, kThreads, 8), kThreads, 0, c->stream>>>(v, p->lev[l].val, cnt);
        HB_CK(cudaGetLastError());
      } else {
        B->val32.push_back(v);
      }
    }
  std::vector<BGs> gs;
  std::vector<BRes> res;
  std::vector<BTile> tiles;
  build_vcycle(B, 0, gs, res, tiles);
  HB_TRY(alloc_copy(B, (void**)&B->gs_items, gs.data(), sizeof(BGs) * gs.size()));
  if (!res.empty()) HB_TRY(alloc_copy(B, (void**)&B->res_items, res.data(), sizeof(BRes) * res.size()));
  HB_TRY(alloc_copy(B, (void**)&B->tiles, tiles.data(), sizeof(BTile) * tiles.size()));
  std::vector<DStep> ds;
  for (const Step& x : B->steps) ds.push_back(DStep{x.kind, x.tile_off, x.ntiles});
  return alloc_copy(B, (void**)&B->dsteps, ds.data(), sizeof(DStep) * ds.size());
}

void destroy(hpcg_b200_batch* B) {
  if (!B) return;
  cudaSetDevice(B->device);
  if (B->ctx) cudaStreamSynchronize(B->ctx->stream);
  if (B->graph) cudaGraphExecDestroy(B->graph);
  void* v[] = {B->gs_items, B->res_items, B->tiles, B->geo_items, B->geo_tiles, B->prolong_items, B->prolong_tiles,
               B->grids, B->maps, B->mv_tiles, B->mv_tile0, B->mv_partials, B->descs, B->vec, B->vtiles, B->vrange, B->partials, B->sc, B->ctl, B->dsteps, B->bar};
  for (void* q : v) cudaFree(q);
  for (float* q : B->val32) cudaFree(q);
  if (B->sc_host) cudaFreeHost(B->sc_host);
  release_accounted(B->bytes);
  for (hpcg_b200_problem* p : B->probs) free_problem(p);
  B->magic = 0;
  delete B;
}

}  // namespace
}  // namespace hb

using namespace hb;

extern "C" {

int hpcg_b200_batch_create(int count, const int* nx, const int* ny, const int* nz, int device,
                           hpcg_b200_batch** out) {
  if (!out || count < 1 || !nx || !ny || !nz) return HPCG_B200_ERR_ARG;
  *out = nullptr;
  for (int i = 0; i < count; ++i)  // every level even: all 8 colours present on every level
    if (nx[i] % 16 || ny[i] % 16 || nz[i] % 16 || nx[i] < 16 || ny[i] < 16 || nz[i] < 16)
      return HPCG_B200_ERR_UNSUPPORTED;
  Context* c = context_for(device);
  if (!c) return HPCG_B200_ERR_CUDA;
  HB_CK(cudaSetDevice(device));
  hpcg_b200_batch* B = new hpcg_b200_batch;
  B->magic = kBatchMagic;
  B->device = device;
  B->ctx = c;
  B->m = count;
  B->gs_items = nullptr; B->res_items = nullptr; B->tiles = nullptr; B->vec = nullptr; B->vtiles = nullptr;
  B->geo_items = nullptr; B->geo_tiles = nullptr; B->prolong_items = nullptr; B->prolong_tiles = nullptr;
  B->maps = nullptr; B->mv_tiles = nullptr; B->mv_tile0 = nullptr; B->mv_partials = nullptr;
  B->mv_ntiles = 0;
  B->grids = nullptr; B->descs = nullptr; B->bulk = false; B->tail_cluster = 1; B->tail_smem = 0;
  B->persist = false; B->persist_grid = 0; B->dsteps = nullptr; B->bar = nullptr;
  B->vrange = nullptr; B->partials = nullptr; B->sc = nullptr; B->sc_host = nullptr; B->ctl = nullptr;
  B->bytes = 0;
  B->graph = nullptr;
  B->nvt = 0;
  int st = HPCG_B200_OK;
  for (int i = 0; i < count && st == HPCG_B200_OK; ++i) {
    hpcg_b200_problem* p = nullptr;
    st = hpcg_b200_generate(nx[i], ny[i], nz[i], 4, device, &p);
    if (st == HPCG_B200_OK) {
      B->probs.push_back(p);
      st = prepare_f32(p);
    }
  }
  if (st == HPCG_B200_OK) {
    std::vector<BVec> vec(count);
    std::vector<BTile> vt;
    std::vector<int> range(count + 1, 0);
    for (int p = 0; p < count; ++p) {
      hpcg_b200_problem* P = B->probs[p];
      const Level& L = P->lev[0];
      vec[p] = BVec{L.val, L.col, L.pitch, L.n, P->b, P->x, P->r, P->z, P->zprev, P->p, P->Ap, L.r32, L.x32};
      range[p] = (int)vt.size();
      tiles_of(vt, p, 0, L.n);
    }
    range[count] = (int)vt.size();
    B->nvt = (int)vt.size();
    st = alloc_copy(B, (void**)&B->vec, vec.data(), sizeof(BVec) * vec.size());
    if (!st) st = alloc_copy(B, (void**)&B->vtiles, vt.data(), sizeof(BTile) * vt.size());
    if (!st) st = alloc_copy(B, (void**)&B->vrange, range.data(), sizeof(int) * range.size());
    if (!st) st = dev_alloc((void**)&B->partials, sizeof(double) * 2 * B->nvt, &B->bytes);
    if (!st) st = dev_alloc((void**)&B->sc, sizeof(BScal) * count, &B->bytes);
    if (!st) st = dev_alloc((void**)&B->ctl, sizeof(BCtl), &B->bytes);
    if (!st) st = dev_alloc((void**)&B->bar, sizeof(BBar), &B->bytes);
    if (!st && cudaMemset(B->bar, 0, sizeof(BBar)) != cudaSuccess) st = HPCG_B200_ERR_CUDA;
    if (!st) {
      int per_sm = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_b_iteration, kThreads, 0) != cudaSuccess) {
        cudaGetLastError();
        per_sm = 0;
      }
      // measurement knob HPCG_B200_BATCH_PERSIST_BLOCKS: resident blocks per SM
      const char* pb = std::getenv("HPCG_B200_BATCH_PERSIST_BLOCKS");
      const int want = pb && *pb ? std::atoi(pb) : kBlocksPerSm;
      B->persist_grid = c->sms * std::max(0, std::min({per_sm, kBlocksPerSm, want}));
    }
    if (!st && cudaMallocHost(&B->sc_host, sizeof(BScal) * count) != cudaSuccess) st = HPCG_B200_ERR_NOMEM;
    if (!st && cudaMemset(B->sc, 0, sizeof(BScal) * count) != cudaSuccess) st = HPCG_B200_ERR_CUDA;
    if (!st) st = choose_form(B);
    if (!st) st = B->bulk ? build_form1(B) : build_register_forms(B);
    if (!st) st = stream_sync(c);
  }
  if (st != HPCG_B200_OK) {
    destroy(B);
    return st;
  }
  *out = B;
  return HPCG_B200_OK;
}

int hpcg_b200_batch_problem(hpcg_b200_batch* B, int i, hpcg_b200_problem** out) {
  if (!valid_batch(B)) return HPCG_B200_ERR_HANDLE;
  if (!out || i < 0 || i >= B->m) return HPCG_B200_ERR_ARG;
  *out = B->probs[i];
  return HPCG_B200_OK;
}

int hpcg_b200_batch_cg_mixed(hpcg_b200_batch* B, const double* const* b, double* const* x, int max_iter,
                             double tolerance, int* niters, double* normr, double* normr0) {
  if (!valid_batch(B)) return HPCG_B200_ERR_HANDLE;
  if (!b || !x || !niters || !normr || !normr0 || max_iter < 0) return HPCG_B200_ERR_ARG;
  for (int p = 0; p < B->m; ++p)
    if (!b[p] || !x[p]) return HPCG_B200_ERR_ARG;
  HB_CK(cudaSetDevice(B->device));
  Context* c = B->ctx;
  for (int p = 0; p < B->m; ++p) {
    if (B->bulk) HB_TRY(prepare_f32(B->probs[p]));  // (a member's values may have been set since)
    HB_TRY(load_vector(B->probs[p], 0, b[p], B->probs[p]->b));
    HB_TRY(load_vector(B->probs[p], 0, x[p], B->probs[p]->x));
  }
  // preamble: Ap = A x; r = b - Ap; normr0 (CG.cpp:86-96), every problem
  const int gv = grid_tiles(c, B->nvt);
  k_b_setup<<<1, 32, 0, c->stream>>>(B->ctl, max_iter, tolerance);
  k_b_spmv<false><<<gv, kThreads, 0, c->stream>>>(B->vec, B->vtiles, B->nvt, 0, nullptr, nullptr);
  k_b_resid<<<gv, kThreads, 0, c->stream>>>(B->vec, B->vtiles, B->nvt, B->partials);
  HB_CK(cudaGetLastError());
  HB_TRY(finalize_b(B, kBNorm0));
  if (B->bulk) {
    k_b_to32<<<gv, kThreads, 0, c->stream>>>(B->vec, B->vtiles, B->nvt, B->sc);
    HB_CK(cudaGetLastError());
  }
  if (!B->graph) {
    int gs = build_graph(B);
    if (gs != HPCG_B200_OK && B->persist) {  // a cooperative launch refused inside a capture
      cudaGetLastError();
      B->persist = false;
      gs = build_graph(B);
    }
    HB_TRY(gs);
  }
  HB_CK(cudaGraphLaunch(B->graph, c->stream));
  HB_CK(cudaMemcpyAsync(B->sc_host, B->sc, sizeof(BScal) * B->m, cudaMemcpyDeviceToHost, c->stream));
  HB_TRY(stream_sync(c));
  for (int p = 0; p < B->m; ++p) {
    niters[p] = B->sc_host[p].niters;
    normr[p] = std::sqrt(B->sc_host[p].normr2);
    normr0[p] = B->sc_host[p].normr0;
    HB_TRY(store_vector(B->probs[p], 0, B->probs[p]->x, x[p]));
  }
  return HPCG_B200_OK;
}

int hpcg_b200_batch_form(const hpcg_b200_batch* B, int* form) {
  if (!valid_batch(B)) return HPCG_B200_ERR_HANDLE;
  if (!form) return HPCG_B200_ERR_ARG;
  *form = B->persist ? 2 : B->bulk ? 1 : 0;
  return HPCG_B200_OK;
}

int hpcg_b200_grid_wait_selftest(int device, double seconds) {
  if (!(seconds > 0.0 && seconds <= 2.0)) return HPCG_B200_ERR_ARG;
  Context* c = context_for(device);
  if (!c) return HPCG_B200_ERR_CUDA;
  HB_CK(cudaSetDevice(device));
  BBar* bar = nullptr;
  HB_CK(cudaMalloc(&bar, sizeof(BBar)));
  cudaError_t e = cudaMemsetAsync(bar, 0, sizeof(BBar), c->stream);
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(c->sms);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = c->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, k_b_barrier_selftest, bar, (unsigned long long)(seconds * 1e9), c->fault);
  }
  if (e != cudaSuccess) {
    set_error("grid wait self-test", e);
    cudaStreamSynchronize(c->stream);
    cudaFree(bar);
    return status_of(e);
  }
  const int st = stream_sync(c);
  cudaFree(bar);
  return st;
}

int hpcg_b200_batch_free(hpcg_b200_batch* B) {
  if (!valid_batch(B)) return HPCG_B200_ERR_HANDLE;
  destroy(B);
  return HPCG_B200_OK;
}

}  // extern "C"
