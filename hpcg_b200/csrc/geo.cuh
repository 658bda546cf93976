// Columns of a level from the grid instead of from memory. In the colour order
// the neighbour of row m of a colour (m counted inside its block, point
// (xx, yy, zz) of the colour's half-grid) in direction (sx, sy, sz) is row
// (zz + az) hy' hx' + (yy + ay) hx' + (xx + ax) of the neighbour colour's block,
// with ax, ay, az in {-1, 0, 1} fixed by the two colours' parities and hx', hy'
// the half-sides of the neighbour colour. So a slot's column is one of four
// numbers of the row (m itself where the sides are even) plus a constant of
// (colour, slot), and a direction that leaves the grid is a bit of a 27-bit word
// of the row. Used for levels whose stored columns were checked to be exactly
// these at creation (Level::geo): the same columns, no bytes read for them, on
// any sides and for any tile of rows (a packed record needs its 128 rows in one
// colour block). A packed record costs a row 4.25 bytes, two shared loads and
// four integer instructions a slot; this costs about 40 integer instructions a
// row and three a slot.
#pragma once

#include "common.cuh"

namespace hb {

// Quotients by a fixed divisor for 0 <= n < 2^31: (n * mul) >> shift.
struct FastDiv {
  unsigned mul, shift;
  __host__ void init(unsigned d) {
    unsigned p = 31;  // smallest with 2^(p - 31) >= d
    while (((uint64_t)1 << (p - 31)) < d) ++p;
    mul = (unsigned)((((uint64_t)1 << p) + d - 1) / d);
    shift = p;
  }
  __host__ __device__ __forceinline__ unsigned div(unsigned n) const {
    return (unsigned)(((uint64_t)n * mul) >> shift);
  }
};

// One colour block of a level.
struct GeoPhase {
  int d[kSlots];    // slot k's column less the row's number of its kind
  int start;        // first row of the block
  int hx, hy, hz;   // half-sides
  int ex, ey;       // what the half-sides of the other x / y parity have more
  FastDiv dx, dy;   // by hx, hy
  int shared;       // whether 32 bytes of a vector may hold rows of two colours, or rows
                    // and the zero sink behind the last one (which border rows of every colour read)
  uint32_t low[3], high[3];  // slots that leave the grid at the first / last xx, yy, zz
};

struct GeoGrid {
  GeoPhase block[kColours];  // by sweep position
};

// A row's place: the numbers of its neighbours by flipped parities of x (bit 0)
// and y (bit 1), and the slots that leave the grid.
struct GeoRow {
  int lin[4];
  uint32_t out;
  __host__ __device__ __forceinline__ GeoRow(const GeoPhase& g, int q) {
    const unsigned m = (unsigned)(q - g.start);
    const unsigned t = g.dx.div(m);
    const int xx = (int)(m - t * g.hx);
    const int zz = (int)g.dy.div(t);
    const int yy = (int)t - zz * g.hy;
    lin[0] = (int)m;
    lin[1] = (int)m + (int)t * g.ex;
    lin[2] = (int)m + zz * g.ey * g.hx;
    lin[3] = lin[2] + (zz * (g.hy + g.ey) + yy) * g.ex;
    out = (xx == 0 ? g.low[0] : 0u) | (xx == g.hx - 1 ? g.high[0] : 0u) | (yy == 0 ? g.low[1] : 0u) |
          (yy == g.hy - 1 ? g.high[1] : 0u) | (zz == 0 ? g.low[2] : 0u) | (zz == g.hz - 1 ? g.high[2] : 0u);
  }
  // column of slot k (a compile-time constant after unrolling)
  __host__ __device__ __forceinline__ int col(const GeoPhase& g, int k, int sink) const {
    const int f = slot_flip(k);
    return out >> k & 1u ? sink : lin[f & 3] + g.d[k];
  }
};

// The colour block at sweep position s of a grid.
inline GeoPhase geo_phase(const ColourGrid& g, int s) {
  GeoPhase p;
  const int c = g.sweep[s], par[3] = {c & 1, (c >> 1) & 1, (c >> 2) & 1}, n[3] = {g.nx, g.ny, g.nz};
  int h[3], other[3];
  for (int i = 0; i < 3; ++i) {
    h[i] = ColourGrid::half(n[i], par[i]);
    other[i] = ColourGrid::half(n[i], 1 - par[i]);
    p.low[i] = p.high[i] = 0;
  }
  p.start = g.start[s];
  p.shared = 0;
  for (int u = 0; u <= kColours; ++u) p.shared |= g.start[u] % 8 != 0;  // (start[kColours]: the sink)
  p.hx = h[0];
  p.hy = h[1];
  p.hz = h[2];
  p.ex = other[0] - h[0];
  p.ey = other[1] - h[1];
  p.dx.init((unsigned)std::max(1, p.hx));
  p.dy.init((unsigned)std::max(1, p.hy));
  for (int k = 0; k < kSlots; ++k) {
    const int sg[3] = {k % 3 - 1, (k / 3) % 3 - 1, k / 9 - 1};
    int a[3];  // step in the neighbour's half-grid
    for (int i = 0; i < 3; ++i) {
      a[i] = par[i] ? (sg[i] > 0 ? 1 : 0) : (sg[i] < 0 ? -1 : 0);
      if (par[i] == 0 && sg[i] < 0) p.low[i] |= 1u << k;                       // before point 0
      if (2 * (h[i] - 1) + par[i] == n[i] - 1 && sg[i] > 0) p.high[i] |= 1u << k;  // behind the last
    }
    const int nhx = sg[0] ? other[0] : h[0], nhy = sg[1] ? other[1] : h[1];
    p.d[k] = g.start[g.pos[c ^ slot_flip(k)]] + (a[2] * nhy + a[1]) * nhx + a[0];
  }
  return p;
}

inline GeoGrid geo_grid(const ColourGrid& g) {
  GeoGrid r;
  for (int s = 0; s < kColours; ++s) r.block[s] = geo_phase(g, s);
  return r;
}

}  // namespace hb
