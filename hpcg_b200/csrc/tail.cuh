// The small end of the V-cycle in one launch: one thread-block cluster runs
// every level from a given one down (pre-smooth, residual + restriction, the
// levels below, prolongation, post-smooth), with x of each level in the
// blocks' shared memory. Launched phase by phase such a level costs 32
// launches of 2-5 us each although a phase's rows need well under 1 us, so the
// launches, not the bytes, set its time.
//
// Split. Block i of a level's `act` blocks owns a run of z pairs (planes 2h,
// 2h+1); the rows of one colour in that run are one run of storage, so a
// phase's matrix rows stream coalesced. A block keeps x of its planes and of
// one plane on either side; a thread that updates a point of its first or last
// plane also stores it into the neighbour's copy through distributed shared
// memory, so every gather of a phase is a local shared load. Between two
// phases a block waits for its own threads and its two neighbours (TailWait).
// Right-hand sides and solutions of the levels below
// the first move between owners through global memory (L2).
// x is stored with a border of zeros, [plane][y][x parity][x / 2], so a colour's
// lanes read consecutive words and a neighbour is a fixed offset: no column is
// read. The host takes this path only for levels whose columns are exactly the
// stencil's (Level::geo); the zero sink of a direction that leaves the grid is
// the border.
// The arithmetic is gs_row's and k_restrict's, in slot order: the same bits.
#pragma once

#include <type_traits>

#include "bulk.cuh"
#include "common.cuh"

namespace hb {

constexpr int kTailThreads = 256;
constexpr int kTailMaxCluster = 16;
// Rows per block of the values a small level reads: a row's 27 loads are then
// one address and 27 constant offsets (with the pitch between slots each load
// needed 64-bit arithmetic of its own, 1.2 us a phase at any size). The FP32
// copy has this layout; FP64 levels keep such a copy of their values (valt).
constexpr int kTailBlock = kRowBlock32;

template <typename T>
struct TailLevel {
  const T* val;  // values in blocks of kTailBlock rows (mat_index<T, kTailBlock>)
  T* r;          // right-hand side and solution, colour order
  T* x;
  int nx, ny, nz;
  int start[kColours];  // first row of each sweep position
  int act;              // blocks that own a slab
  int xoff;             // the level's first element in a block's shared array
  int toff;             // the level's first entry in a block's row table
};

template <typename T>
struct TailDesc {
  TailLevel<T> lev[kMaxLevels];
  int nlev;
  int elems;  // shared elements of a block
  int rows;   // entries of its row table
  int sweep[kColours];
  int pos[kColours];
  uint32_t mask[kColours];  // first_mask of each sweep position
};

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_blocks() {
  unsigned n;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
  return n;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// Without ordering: the end of a block's life only (a neighbour whose wait gave
// up may still store into it).
__device__ __forceinline__ void cluster_sync_relaxed() {
  asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
  asm volatile("barrier.cluster.wait;" ::: "memory");
}
// The same shared-memory place in another block of the cluster.
__device__ __forceinline__ unsigned cluster_addr(const void* local, unsigned rank) {
  unsigned ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_addr(local)), "r"(rank));
  return ra;
}
// Stores v into another block's shared memory; its bytes count on that block's `bar`.
__device__ __forceinline__ void st_async(unsigned addr, double v, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(addr), "d"(v),
               "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async(unsigned addr, float v, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(addr), "f"(v),
               "r"(bar)
               : "memory");
}

// What a block waits on between two phases of a level that several blocks
// hold: the bytes its neighbours send it in the phase (their new boundary
// values) and one word from each that says the phase is done there, counted on
// an mbarrier. No memory fence lies on this path: the cluster barrier's
// release waits for every load and store in flight, 930-1680 cycles measured
// with global stores outstanding against about 350 here, and it would end the
// overlap of the next row's loads with the wait. Two mbarriers alternate: a
// neighbour may be one phase ahead, never two (it waits for this block's word).
struct TailSync {
  uint64_t bar[2];
  unsigned word[2];  // where the neighbours' words land
};
struct TailWait {
  TailSync* sy;
  unsigned* fault;
  int m;            // index of the next phase's wait in this sweep
  unsigned parity;  // bit b: parity of mbarrier b's next completion
  bool dead;        // a wait gave up: no more waiting
  // ends a phase in which this block is sent `bytes` by its neighbours
  __device__ __forceinline__ void end(int rank, int act, unsigned bytes) {
    __syncthreads();
    if (act == 1) return;
    uint64_t* b = &sy->bar[m & 1];
    if (threadIdx.x == 0) {
      if (rank > 0) st_async(cluster_addr(&sy->word[0], rank - 1), 0.0f, cluster_addr(b, rank - 1));
      if (rank + 1 < act) st_async(cluster_addr(&sy->word[1], rank + 1), 0.0f, cluster_addr(b, rank + 1));
      mbar_expect_tx(b, bytes + 4u * ((rank > 0) + (rank + 1 < act)));
    }
    if (!dead && !mbar_wait(b, (parity >> (m & 1)) & 1u)) {
      record_fault(fault, 7);
      dead = true;
    }
    parity ^= 1u << (m & 1);
    ++m;
  }
};

// Strides of a level's x in shared memory.
struct TailShape {
  int hx, sy, sz;
  __host__ __device__ TailShape(int nx, int ny) : hx((nx + 1) / 2 + 2), sy(2 * hx), sz((ny + 2) * sy) {}
};
// z pairs [h0, h1) of block i of `act`
__host__ __device__ __forceinline__ int tail_cut(int pairs, int act, int i) { return (int)((int64_t)pairs * i / act); }

// A block's rows of one colour of a level, by sweep position (a table in shared
// memory: a phase starts from two 16-byte loads).
struct alignas(16) TailPhase {
  int q0, cnt;    // first row, rows
  int t0;         // first entry in the row table
  int colour;
  int per, hx;    // rows of a plane, of a line
  unsigned sent;  // bytes the neighbours send this block in the phase
  uint32_t mask;  // first_mask
};
// A row's place: its element, marked if it lies in the first / last plane of
// the slab with a block beyond.
using TailRow = unsigned;
constexpr unsigned kTailLow = 1u << 30, kTailHigh = 1u << 31;

// A block's share of one level.
template <typename T>
struct TailSlab {
  const TailLevel<T>& L;
  TailShape sh;
  T* xs;
  int rank, h0, h1, planes, lo_planes;
  __device__ TailSlab(const TailLevel<T>& l, T* base, int rank_)
      : L(l), sh(l.nx, l.ny), xs(base + l.xoff), rank(rank_) {
    const int pairs = (l.nz + 1) / 2;
    h0 = tail_cut(pairs, l.act, rank);
    h1 = tail_cut(pairs, l.act, rank + 1);
    planes = min(2 * h1, l.nz) - 2 * h0;
    lo_planes = rank > 0 ? 2 * (h0 - tail_cut(pairs, l.act, rank - 1)) : 0;
  }
  __device__ TailPhase phase(const TailDesc<T>& D, int s) const {
    TailPhase P;
    const int c = D.sweep[s], px = c & 1, py = (c >> 1) & 1, pz = (c >> 2) & 1;
    P.hx = ColourGrid::half(L.nx, px);
    P.per = ColourGrid::half(L.ny, py) * P.hx;
    P.q0 = L.start[s] + h0 * P.per;
    P.cnt = max(0, (min(h1, ColourGrid::half(L.nz, pz)) - h0) * P.per);
    P.t0 = L.toff;
    for (int u = 0; u < s; ++u) {
      const int d = D.sweep[u];
      P.t0 += max(0, (min(h1, ColourGrid::half(L.nz, (d >> 2) & 1)) - h0) * ColourGrid::half(L.ny, (d >> 1) & 1) *
                         ColourGrid::half(L.nx, d & 1));
    }
    P.colour = c;
    // the block below ends with an odd plane, the one above starts with an even one
    P.sent = (pz ? rank > 0 : rank + 1 < L.act) ? (unsigned)(P.per * sizeof(T)) : 0u;
    P.mask = D.mask[s];
    return P;
  }
  // the table entry of the i-th row of a phase
  __device__ TailRow row(const TailPhase& P, int i) const {
    const int zz = i / P.per, rem = i - zz * P.per, yy = rem / P.hx, xx = rem - yy * P.hx;
    const int px = P.colour & 1, py = (P.colour >> 1) & 1, lz = 2 * zz + ((P.colour >> 2) & 1) + 1;
    return (unsigned)(lz * sh.sz + (2 * yy + py + 1) * sh.sy + px * sh.hx + xx + 1) |
           (lz == 1 && rank > 0 ? kTailLow : 0u) | (lz == planes && rank + 1 < L.act ? kTailHigh : 0u);
  }
  // the row of the next level injected from the i-th row of the all-even points
  __device__ int coarse(const TailDesc<T>& D, const TailLevel<T>& C, const TailPhase& P, int i) const {
    const int zz = i / P.per, rem = i - zz * P.per, yy = rem / P.hx, xx = rem - yy * P.hx, zc = h0 + zz;
    const int c = (xx & 1) | ((yy & 1) << 1) | ((zc & 1) << 2);
    const int cx = ColourGrid::half(C.nx, c & 1), cy = ColourGrid::half(C.ny, (c >> 1) & 1);
    return C.start[D.pos[c]] + ((zc >> 1) * cy + (yy >> 1)) * cx + (xx >> 1);
  }
};

// One symmetric sweep of a level (the last colour of the forward sweep is not
// repeated, as in gs_colour), and with RESTRICT the residual at the injected
// rows into the next level's r. ZERO: x enters as zero. prolong: the next
// level's x is added at the injected points first. keep: each row's final x
// is also stored in xg.
// A phase is one dependent chain: 27 subtractions (14.5 cycles each in FP64 on
// B200), the division (some 300), the store, the wait for the neighbours (350),
// and its warps issue one instruction in some seven cycles (ncu: fixed-latency
// waits), so the instructions of a row set a phase's time. The code of a row is
// one straight line: the next row's 27 values are loaded into the other of two
// register sets first (they have the whole phase to arrive), then the 27
// gathers, then the chain. Measured at 8^3: 2.4 us a phase with a test per slot
// or with values loaded into the registers of the slot just used (each gather's
// latency or an L2 latency then enters the chain), 1.1 us this way; three lanes
// to a row, the sum passed between them, 1.2 us.
// A forward phase of a sweep from zero loads only its masked slots' values and
// takes zero for the others: their products are +0, which change no sum.
// ST: entries from one row's right-hand side or solution to the next's (the
// systems of a multi-system solve interleave), off: the system.
template <typename T, bool ZERO, int ST>
__device__ __forceinline__ void tail_sweep(const TailDesc<T>& D, int l, T* smem, const TailPhase* __restrict__ phases,
                                           const TailRow* __restrict__ table, int rank, const T* __restrict__ rhs,
                                           T* xg, bool keep, bool restrict_, bool prolong, TailWait& wait,
                                           int off) {
  const TailLevel<T>& L = D.lev[l];
  if (rank >= L.act) {
    cluster_sync_all();
    return;
  }
  const int nph = 15 + (restrict_ ? 1 : 0);
  wait.m = 0;
  const TailSlab<T> S(L, smem, rank);
  const TailPhase* tab = phases + l * kColours;
  const int tid = threadIdx.x, lane = tid & 31;
  // the neighbours' copies of this block's boundary planes, and their mbarriers
  const bool low = rank > 0, high = rank + 1 < L.act;
  const unsigned xlow = low ? cluster_addr(S.xs + S.lo_planes * S.sh.sz, rank - 1) : 0u;
  const unsigned xhigh =  // (the difference after the mapping: before it the address would leave the block's memory)
      high ? cluster_addr(S.xs, rank + 1) - (unsigned)(S.planes * S.sh.sz * (int)sizeof(T)) : 0u;
  const unsigned blow = low ? cluster_addr(wait.sy->bar, rank - 1) : 0u;
  const unsigned bhigh = high ? cluster_addr(wait.sy->bar, rank + 1) : 0u;
  // x of the row at t becomes v, here and in the neighbours' copies (their
  // bytes counted on the phase's mbarrier there)
  auto put = [&](unsigned t, T v) {
    const unsigned e = t & ~(kTailLow | kTailHigh);
    S.xs[e] = v;
    if (t & kTailLow) st_async(xlow + e * (unsigned)sizeof(T), v, blow + 8u * (wait.m & 1));
    if (t & kTailHigh) st_async(xhigh + e * (unsigned)sizeof(T), v, bhigh + 8u * (wait.m & 1));
  };
  // sweep position of phase j: 0 .. 7, 6 .. 0, and the injected rows (position 7)
  auto pos_of = [](int j) { return j < 8 ? j : j < 15 ? 14 - j : 7; };
  // a row's 27 values
  auto fetch = [&](T(&v)[kSlots + 1], int q, const TailPhase& P, int j) {
    const T* p = L.val + ((unsigned)q / kTailBlock * (kSlots * kTailBlock) + (unsigned)q % kTailBlock);
    if (ZERO && j < 8) {
      const uint32_t m = P.mask | 1u << kDiagSlot;
#pragma unroll
      for (int k = 0; k < kSlots; ++k) v[k] = m >> k & 1u ? __ldg(p + k * kTailBlock) : (T)0;
    } else {
#pragma unroll
      for (int k = 0; k < kSlots; ++k) v[k] = __ldg(p + k * kTailBlock);
    }
  };
  T va[kSlots + 1], vb[kSlots + 1];  // values, and the right-hand side behind them
  int j = 0, i = tid;                // phase, this thread's row in it
  TailPhase P = tab[0];
  TailRow R = table[P.t0 + (i < P.cnt ? i : 0)];
  fetch(va, P.q0 + (i < P.cnt ? i : 0), P, 0);
  cluster_sync_all();  // what the sweep reads (rhs, the next level's x) is written
  if (prolong) {
    const TailLevel<T>& C = D.lev[l + 1];
    const TailPhase PI = tab[7];
    for (int u = tid; u < PI.cnt; u += kTailThreads) {
      const unsigned t = table[PI.t0 + u];
      put(t, S.xs[t & ~(kTailLow | kTailHigh)] + __ldcg(C.x + (int64_t)S.coarse(D, C, PI, u) * ST + off));
    }
    wait.end(rank, L.act, PI.sent);
  }
  va[kSlots] = __ldcg(rhs + (int64_t)(P.q0 + (i < P.cnt ? i : 0)) * ST);
  // one row of this thread, its values in a; false after the last
  auto step = [&](const T(&a)[kSlots + 1], T(&next)[kSlots + 1]) -> bool {
    // the next row: the phase's next chunk, or the next phase's first (a thread
    // without a row takes the phase's first and drops it; a warp without any
    // passes)
    const bool same = i - tid + kTailThreads < P.cnt;
    const int nj = same ? j : j + 1;
    const bool more = nj < nph;
    const TailPhase NP = tab[pos_of(nj)];
    const int ni = same ? i + kTailThreads : tid;
    TailRow NR = R;
    if (more && ni - lane < NP.cnt) {
      const int nc = ni < NP.cnt ? ni : 0;
      NR = table[NP.t0 + nc];
      fetch(next, NP.q0 + nc, NP, nj);
      next[kSlots] = __ldcg(rhs + (int64_t)(NP.q0 + nc) * ST);
    }
    const bool res = j == 15;  // the residual at the injected rows
    if (i < P.cnt) {
      // the gathers' two bases: the row's own x parity, and the other one (the
      // neighbour at x - 1; the one at x + 1 is the next element)
      const T* xp = S.xs + (R & ~(kTailLow | kTailHigh));
      const T* xo = xp + (P.colour & 1 ? -S.sh.hx : S.sh.hx - 1);
      T xv[kSlots];
#pragma unroll
      for (int k = 0; k < kSlots; ++k) {
        const int sx = k % 3 - 1, sy = (k / 3) % 3 - 1, sz = k / 9 - 1;
        const int line = sz * S.sh.sz + sy * S.sh.sy;
        xv[k] = sx == 0 ? xp[line] : xo[line + (sx > 0 ? 1 : 0)];
      }
      const T rv = a[kSlots];
      T sum = res ? (T)0 : rv;
#pragma unroll
      for (int k = 0; k < kSlots; ++k) sum -= a[k] * xv[k];
      if (res) {
        const TailLevel<T>& C = D.lev[l + 1];
        C.r[(int64_t)S.coarse(D, C, P, i) * ST + off] = rv + sum;  // sum: minus the row's product
      } else {
        const T d = a[kDiagSlot];
        if (!(ZERO && j < 8)) sum += xv[kDiagSlot] * d;
        const T out = sum / d;
        put(R, out);
        if (keep && j >= 7) xg[(int64_t)(P.q0 + i) * ST] = out;
      }
    }
    if (!same && !res) wait.end(rank, L.act, P.sent);
    i = ni;
    j = nj;
    P = NP;
    R = NR;
    return more;
  };
  while (step(va, vb) && step(vb, va)) {
  }
}

// The V-cycle of a problem's levels from D.lev[0] down (rhs, x: level D.lev[0]'s
// vectors, at the system's first entry), or with `step` one symmetric step on x
// with right-hand side rhs.
template <typename T, int ST = 1>
__device__ __forceinline__ void tail_run(const TailDesc<T>& D, const T* __restrict__ rhs, T* x, bool step,
                                         unsigned* fault, int off = 0) {
  extern __shared__ __align__(16) unsigned char tail_smem[];
  __shared__ TailSync sync;
  __shared__ TailPhase phases[kMaxLevels * kColours];
  T* smem = reinterpret_cast<T*>(tail_smem);
  TailRow* table = reinterpret_cast<TailRow*>(smem + D.elems);
  const int rank = (int)cluster_rank();
  TailWait wait{&sync, fault, 0, 0u, false};
  if (threadIdx.x == 0) {
    mbar_init(&sync.bar[0], 1);
    mbar_init(&sync.bar[1], 1);
    mbar_init_fence();
  }
  if (threadIdx.x < (unsigned)(D.nlev * kColours)) {
    const TailLevel<T>& L = D.lev[threadIdx.x / kColours];
    if (rank < L.act) phases[threadIdx.x] = TailSlab<T>(L, smem, rank).phase(D, threadIdx.x % kColours);
  }
  for (int i = threadIdx.x; i < D.elems; i += kTailThreads) smem[i] = (T)0;
  __syncthreads();
  for (int u = 0; u < D.nlev * kColours; ++u) {
    const TailLevel<T>& L = D.lev[u / kColours];
    if (rank >= L.act) break;
    const TailSlab<T> S(L, smem, rank);
    const TailPhase P = phases[u];
    for (int i = threadIdx.x; i < P.cnt; i += kTailThreads) table[P.t0 + i] = S.row(P, i);
  }
  griddep_wait();  // (above: this block's own memory and the launch's description only)
  if (step) {
    const TailLevel<T>& L = D.lev[0];
    if (rank < L.act) {
      const TailSlab<T> S(L, smem, rank);
      const int lz0 = S.h0 > 0 ? 0 : 1, lz1 = min(S.planes + 1, L.nz - 2 * S.h0);  // planes that exist
      const int per = L.nx * L.ny;
      for (int i = threadIdx.x; i < (lz1 - lz0 + 1) * per; i += kTailThreads) {
        const int lz = lz0 + i / per, rem = i % per, iy = rem / L.nx, ix = rem - iy * L.nx;
        const int iz = 2 * S.h0 + lz - 1;
        const int c = (ix & 1) | ((iy & 1) << 1) | ((iz & 1) << 2);
        const int cx = ColourGrid::half(L.nx, c & 1), cy = ColourGrid::half(L.ny, (c >> 1) & 1);
        S.xs[lz * S.sh.sz + (iy + 1) * S.sh.sy + (ix & 1) * S.sh.hx + (ix >> 1) + 1] =
            __ldcg(x + (int64_t)(L.start[D.pos[c]] + ((iz >> 1) * cy + (iy >> 1)) * cx + (ix >> 1)) * ST);
      }
    }
    tail_sweep<T, false, ST>(D, 0, smem, phases, table, rank, rhs, x, true, false, false, wait, off);
    cluster_sync_relaxed();
    return;
  }
  for (int l = 0; l < D.nlev; ++l)
    tail_sweep<T, true, ST>(D, l, smem, phases, table, rank, l == 0 ? rhs : D.lev[l].r + off,
                            l == 0 ? x : D.lev[l].x + off, l + 1 == D.nlev, l + 1 < D.nlev, false, wait, off);
  for (int l = D.nlev - 2; l >= 0; --l)
    tail_sweep<T, false, ST>(D, l, smem, phases, table, rank, l == 0 ? rhs : D.lev[l].r + off,
                             l == 0 ? x : D.lev[l].x + off, true, false, true, wait, off);
  cluster_sync_relaxed();
}

template <typename T>
__global__ void __launch_bounds__(kTailThreads, 1)
    k_tail(const __grid_constant__ TailDesc<T> D, const T* __restrict__ rhs, T* x, int step, unsigned* fault) {
  tail_run<T>(D, rhs, x, step != 0, fault);
}

// Host side (tail.cu). tail_desc: the description of problem p's levels l ..
// l + nlev - 1, the shared memory of a block; returns the blocks of a cluster (a
// power of two). tail_fits: whether the GPU can hold one such cluster of a kernel
// built on tail_run, asked before a launch of it is planned: a refusal would come in
// the middle of a capture. It lets the kernel use as much shared memory as any
// description asks for: the limit is the kernel's, not a launch's, so one set for one
// problem's need would refuse a larger problem that is still alive.
// HPCG_B200_TAIL_CLUSTER=n: as on a GPU that holds clusters of at most n blocks.
int tail_desc(hpcg_b200_problem* p, int l, int nlev, TailDesc<double>* D, size_t* smem);
int tail_desc(hpcg_b200_problem* p, int l, int nlev, TailDesc<float>* D, size_t* smem);
bool tail_fits(const void* kernel, int size, size_t smem);
// tail_first for other bounds than the single problem's: rows of a block in one
// phase, bytes of its shared memory
int tail_first_within(const hpcg_b200_problem* p, bool f32, int64_t rows, int64_t bytes);

}  // namespace hb
