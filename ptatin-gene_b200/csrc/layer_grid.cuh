// Index arithmetic of the layer tiles (kernels_layer.cuh), host and device so
// that the CPU self-check (tests/core_host_check.cpp) walks the same code.
//
// A layer tile is E consecutive elements (element number ex + mx*(ej + my*ek),
// one thread each), so every thread has an element whatever the row length
// and a warp's K is whole blocks.  The tile's pieces of element rows
// ("segments", at most END of them) each keep their own 3 x 3 node rows and
// share nothing with each other.  One component's node row of a tile is
// [even | odd | end]: thread tid has its node 2t at tid, its node 2t+1 at
// ODD + tid, and its node 2t+2 at tid + 1, the next element's 2t -- except the
// last thread of a segment, whose 2t+2 is the segment's end entry.  A warp
// reads consecutive words.  Short rows make many segments, so a box of them
// takes fewer elements per tile and the room of their odd entries for ends.
#pragma once

#include <cstdint>

#ifndef PT_HD
#ifdef __CUDACC__
#define PT_HD __host__ __device__ __forceinline__
#else
#define PT_HD inline
#endif
#endif

namespace ptk {

// Division of values below 2^31 by a fixed divisor: one high multiply (the
// round-up method: ceil(2^(32+s) / d) with 2^s >= d has 33 bits; m holds the
// low 32, and the top one is the n added back after the multiply).
struct FastDiv {
  uint32_t d, m, s;
  PT_HD uint32_t div(uint32_t n) const
  {
#ifdef __CUDA_ARCH__
    const uint32_t h = __umulhi(n, m);
#else
    const uint32_t h = (uint32_t)(((uint64_t)n * m) >> 32);
#endif
    return (h + n) >> s;  // h < n < 2^31: no overflow
  }
};

inline FastDiv fast_div(uint32_t d)
{
  FastDiv f;
  f.d = d;
  f.s = 0;
  while (((uint64_t)1 << f.s) < d) f.s++;
  f.m = (uint32_t)((((uint64_t)1 << 32) * (((uint64_t)1 << f.s) - d)) / d + 1);
  return f;
}

template <int NT>
struct LayerLayout {
  static constexpr int ROW = 2 * NT + 8;     // one component's node row
  static constexpr int PLANE = 3 * ROW;      // three node rows
  // 11 values of padding: the plane fetch walks the (node, component) order;
  // with 3 modulo 16 between components its stores fall in different banks
  static constexpr int COMP = 3 * PLANE + 11;
  static constexpr int TILE = (3 * COMP + 3) / 4 * 4;  // a multiple of 16 bytes in both precisions
  static constexpr int NW = NT / 32;
  static constexpr int SIDE = NW * 27;       // 2t+2 column of each warp's last lane
};

struct LayerGrid {
  int mx, my, mz;
  int64_t X, XY, off;  // node strides and first node of the element box
  int nel, E, tiles;   // elements, elements per tile, tiles
  int odd;             // first odd entry of a node row; the end entries start at 2 odd
  FastDiv dNX, dNY, dmx, dmy, dE;  // by 2mx+1, 2my+1, mx, my, E
  PT_HD uint32_t nodes() const { return dNX.d * dNY.d * (uint32_t)(2 * mz + 1); }
};

// Most segments that E consecutive elements in rows of mx can touch, tiles
// starting at multiples of E.
inline int layer_segments(int E, int mx)
{
  if (E % mx == 0) return E / mx;
  if (mx % E == 0) return 1;
  return (E - 2) / mx + 2;
}

// Elements per tile: NT where their segments fit the 8 end entries beside NT
// even and odd ones (rows of 21 elements and more, and of 16), else 7/8 of NT
// (40 end entries with NT = 128), fewer only for rows of one or two elements.
// The shape depends on the box alone, so its sums are the same in any batch.
template <int NT>
inline LayerGrid layer_grid(int mx, int my, int mz, int64_t X, int64_t XY, int64_t off)
{
  LayerGrid g;
  g.mx = mx; g.my = my; g.mz = mz;
  g.X = X; g.XY = XY; g.off = off;
  g.nel = mx * my * mz;
  g.odd = layer_segments(NT, mx) <= LayerLayout<NT>::ROW - 2 * NT ? NT : NT * 7 / 8;
  const int ends = LayerLayout<NT>::ROW - 2 * g.odd;
  g.E = g.odd;
  while (layer_segments(g.E, mx) > ends) g.E--;
  g.tiles = (g.nel + g.E - 1) / g.E;
  g.dNX = fast_div(2 * mx + 1);
  g.dNY = fast_div(2 * my + 1);
  g.dmx = fast_div(mx);
  g.dmy = fast_div(my);
  g.dE = fast_div(g.E);
  return g;
}

// Segment sg of a tile that starts at element e0 (in row row0 = e0 / mx): its
// first thread and its length within [e0, e0 + n).
PT_HD void layer_segment(const LayerGrid &g, int e0, int row0, int n, int sg, int &t0, int &len)
{
  const int a = (row0 + sg) * g.mx - e0;  // thread of the row's first element
  t0 = a > 0 ? a : 0;
  const int b = a + g.mx < n ? a + g.mx : n;
  len = b - t0;
}

// One axis of a node: its elements and local node indices, lower element first.
struct AxisNode {
  int e[2], l[2], n;
};
PT_HD AxisNode axis_node(int i, int m)
{
  AxisNode a;
  const int h = i >> 1;
  if (i & 1) { a.e[0] = a.e[1] = h; a.l[0] = a.l[1] = 1; a.n = 1; }
  else if (h == 0) { a.e[0] = a.e[1] = 0; a.l[0] = a.l[1] = 0; a.n = 1; }
  else {
    a.e[0] = h - 1; a.l[0] = 2;
    a.e[1] = h; a.l[1] = 0;
    a.n = h < m ? 2 : 1;
  }
  return a;
}

// Scratch offsets (component 0, node plane 0, row 0) of the entries that hold
// node i's sum from element row `row`: at[0] the end entry of element
// (i/2 - 1)'s segment where that is not an even entry of element i/2, at[1]
// element i/2's even or odd entry; -1 where there is none.
template <int NT>
PT_HD void layer_slots(const LayerGrid &g, int i, int row, int64_t at[2])
{
  using L = LayerLayout<NT>;
  const int h = i >> 1;
  const int e = row * g.mx + h;  // element i/2 of the row (one past the row for the last node)
  const int tile = (int)g.dE.div((uint32_t)e), tid = e - tile * g.E;
  at[0] = at[1] = -1;
  if (h < g.mx) at[1] = (int64_t)tile * L::TILE + ((i & 1) ? g.odd + tid : tid);
  if (!(i & 1) && h > 0 && (h == g.mx || tid == 0)) {
    const int tl = tid == 0 ? tile - 1 : tile;  // tile of element i/2 - 1
    const int row0 = (int)g.dmx.div((uint32_t)(tl * g.E));
    at[0] = (int64_t)tl * L::TILE + 2 * g.odd + (row - row0);
  }
}

}  // namespace ptk
