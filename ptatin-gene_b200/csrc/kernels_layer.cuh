// Layer tiles ("b200_layer"): the streaming A11 kernel's arithmetic on
// single-layer tiles, for boxes too small to hide a z-march.
//
// What bounds a small box is latency, not bandwidth: one element takes a
// thread about 20 us (4,700 dependent FP64 operations at two warps per
// scheduler), and the coloured z-march puts a chunk's layers and four colour
// launches one behind the other (41x37x29: 115 us for 1,375 warps of work, on
// a chip that holds 1,184).  Here every element runs at once: each tile
// writes its node sums to scratch, and one gather adds the (at most 4 per
// row, 8 at an x-tile edge) sums of a node in a fixed order, with the
// Dirichlet rows in the same pass.  Two launches, deterministic, no colours.
// The price is the scratch, about 450 B written and read per element next to
// 1.9 KB of K, which is why long boxes with full rows keep the z-march (the rule
// and its figures: auto_kernel in pt_b200.cu).
//
// A tile is E consecutive elements whatever the row length (layer_grid.cuh),
// so rows that do not divide it leave no thread idle.
#pragma once

#include <cstdint>

#include "kernels_diag.cuh"
#include "layer_grid.cuh"

namespace ptk {

constexpr int LAYER_NT = 128;

template <typename T, int NT>
constexpr size_t layer_smem_bytes()
{
  return sizeof(T) * (2 * (size_t)LayerLayout<NT>::TILE + LayerLayout<NT>::SIDE);
}

template <typename T, int NT>
constexpr size_t layer_diag_smem_bytes()
{
  return sizeof(T) * ((size_t)LayerLayout<NT>::TILE + LayerLayout<NT>::SIDE);
}

// The thread's element and its entries of a tile's node row.
struct LayerThread {
  int e;         // element
  bool active;
  int od, en;    // 2t+1, and 2t+2: tid + 1 or the segment's end entry
  bool to_side;  // 2t+2 is the next warp's first column: kept in the side buffer
};

template <int NT>
__device__ __forceinline__ LayerThread layer_thread(const LayerGrid &g, int tile)
{
  LayerThread a;
  const int tid = threadIdx.x, e0 = tile * g.E;
  a.e = e0 + tid;
  a.active = tid < g.E && a.e < g.nel;
  const int row = (int)g.dmx.div((uint32_t)a.e), row0 = (int)g.dmx.div((uint32_t)e0);
  const bool last = a.e + 1 == (row + 1) * g.mx || tid + 1 == g.E;  // of its segment
  a.od = g.odd + tid;
  a.en = last ? 2 * g.odd + (row - row0) : tid + 1;
  a.to_side = (tid & 31) == 31 && !last;
  return a;
}

// A segment's first dof (node row 0 of node plane 0), first thread and length.
struct LayerSeg {
  int64_t k0;
  int t0, len;
};

// Segment table and lines of a tile (a line is one of a segment's 9 node rows).
struct LayerLines {
  const LayerSeg *seg;
  int lines;
  int words;  // mask words that cover a line, wherever it starts
};

// Line `line`: its first dof, its first entry in the tile, its nodes' elements
// and its end entry from the first one.
template <int NT>
__device__ __forceinline__ int64_t layer_line(const LayerGrid &g, const LayerLines &ll, int line, int &first, int &len,
                                              int &end)
{
  using L = LayerLayout<NT>;
  const int sg = line / 9, kj = line - 9 * sg, k = kj / 3, j = kj - 3 * k;
  const LayerSeg s = ll.seg[sg];
  first = k * L::PLANE + j * L::ROW + s.t0;
  len = s.len;
  end = 2 * g.odd + sg - s.t0;
  return s.k0 + 3 * (j * g.X + k * g.XY);
}

// Entry of value d (node d/3, component d%3) of a line, from the line's first.
template <int NT>
__device__ __forceinline__ int layer_entry(const LayerGrid &g, int d, int len, int end)
{
  const int m = (d * 43691) >> 17, c = d - 3 * m;  // d / 3 for d < 2^16
  const int h = m >> 1;
  return c * LayerLayout<NT>::COMP + ((m & 1) ? g.odd + h : (h == len ? end : h));
}

// Fetches the tile's node values of u with asynchronous copies, every copy of
// the tile in flight at once, a warp to a line: a lane works out one of its
// warp's lines and the warp then takes them from lane to lane (worked out by
// the whole warp one after the other, the lines of a tile of short rows took
// 8 us of a 27 us apply).  `stage`: shared memory for the segment table.  Ends
// with the copies committed.
template <typename T, int NT>
__device__ __forceinline__ LayerLines layer_fetch(T *ut, void *stage, const LayerGrid &g, int tile,
                                                  const T *__restrict__ u)
{
  using L = LayerLayout<NT>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e0 = tile * g.E, n = min(g.E, g.nel - e0);
  const int row0 = (int)g.dmx.div((uint32_t)e0);
  const int segs = (int)g.dmx.div((uint32_t)(e0 + n - 1)) - row0 + 1;
  LayerSeg *seg = reinterpret_cast<LayerSeg *>(stage);
  LayerLines ll;
  ll.seg = seg;
  ll.lines = 9 * segs;
  ll.words = (3 * (2 * min(g.mx, n) + 1) + 31) / 32 + 1;
  if ((int)threadIdx.x < segs) {
    LayerSeg s;
    const int row = row0 + threadIdx.x;
    const int ek = (int)g.dmy.div((uint32_t)row), ej = row - ek * g.my;
    layer_segment(g, e0, row0, n, threadIdx.x, s.t0, s.len);
    s.k0 = 3 * (g.off + 2 * (int64_t)(e0 + s.t0 - row * g.mx) + 2 * (int64_t)ej * g.X + 2 * (int64_t)ek * g.XY);
    seg[threadIdx.x] = s;
  }
  __syncthreads();
  const int nl = (ll.lines - warp + L::NW - 1) / L::NW;  // lines of this warp
  for (int b = 0; b < nl; b += 32) {
    int64_t k0 = 0;
    uint32_t pack = 0;  // first (12 bits), len (8), end (10)
    if (b + lane < nl) {
      int first, len, end;
      k0 = layer_line<NT>(g, ll, warp + L::NW * (b + lane), first, len, end);
      pack = (uint32_t)first | (uint32_t)len << 12 | (uint32_t)end << 20;
    }
    const int cnt = min(32, nl - b);
    for (int i = 0; i < cnt; i++) {
      const uint32_t pk = __shfl_sync(0xffffffffu, pack, i);
      const T *src = u + __shfl_sync(0xffffffffu, k0, i);
      const int len = (pk >> 12) & 255, end = pk >> 20, nd = 3 * (2 * len + 1);
      T *row = ut + (pk & 4095);
#pragma unroll 4
      for (int d = lane; d < nd; d += 32) {
        const uint32_t sd = (uint32_t)__cvta_generic_to_shared(row + layer_entry<NT>(g, d, len, end));
        if (sizeof(T) == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sd), "l"(src + d) : "memory");
        else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sd), "l"(src + d) : "memory");
      }
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  return ll;
}

// Waits for the tile's copies and zeroes its Dirichlet entries (mbits not
// null): a thread per mask word of a line, read while the copies fly.  The
// tile is complete for every thread on return, the stage free.
template <typename T, int NT>
__device__ __forceinline__ void layer_land(T *ut, const LayerGrid &g, const LayerLines &ll,
                                           const uint32_t *__restrict__ mbits)
{
  constexpr int AHEAD = 4;  // words per thread in flight (a tile of 128 elements has about 250 to 400)
  if (!mbits) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    return;
  }
  const int total = ll.lines * ll.words;
  for (int i0 = threadIdx.x; i0 - (int)threadIdx.x < total; i0 += AHEAD * NT) {
    uint32_t w[AHEAD];
    int d0[AHEAD], line[AHEAD];  // value of the word's first bit
#pragma unroll
    for (int a = 0; a < AHEAD; a++) {
      const int i = i0 + a * NT;
      w[a] = 0;
      if (i < total) {
        line[a] = i / ll.words;
        int first, len, end;
        const int64_t k0 = layer_line<NT>(g, ll, line[a], first, len, end);
        const int64_t wi = (k0 >> 5) + (i - line[a] * ll.words);
        const int nd = 3 * (2 * len + 1);
        d0[a] = (int)(32 * wi - k0);
        if (d0[a] < nd) {
          w[a] = mbits[wi];
          if (d0[a] < 0) w[a] &= ~0u << -d0[a];           // the line starts within the word
          if (nd - d0[a] < 32) w[a] &= (1u << (nd - d0[a])) - 1;  // or ends in it
        }
      }
    }
    if (i0 == (int)threadIdx.x) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < AHEAD; a++)
      if (w[a]) {
        int first, len, end;
        (void)layer_line<NT>(g, ll, line[a], first, len, end);
        while (w[a]) {
          const int d = d0[a] + __ffs(w[a]) - 1;
          w[a] &= w[a] - 1;
          ut[first + layer_entry<NT>(g, d, len, end)] = T(0);
        }
      }
  }
  __syncthreads();
}

template <typename T, int NT>
__device__ __forceinline__ void layer_zero(T *yt)
{
  using L = LayerLayout<NT>;
  // the tile and the side buffer behind it
  constexpr int N16 = (int)(sizeof(T) * (L::TILE + L::SIDE) / 16);
  static_assert(sizeof(T) * (L::TILE + L::SIDE) % 16 == 0, "16-byte stores");
  for (int i = threadIdx.x; i < N16; i += NT) reinterpret_cast<uint4 *>(yt)[i] = make_uint4(0, 0, 0, 0);
}

// Adds V (27 node values [k*9 + j*3 + i]) to component l of the thread's
// nodes, columns 2t and 2t+1 first, then (after the warp's other lanes) 2t+2:
// the order in which a column shared by two elements is summed is fixed.  A
// group's entries are all read before any is written (tile_add_nodes).
template <typename T, int NT>
__device__ __forceinline__ void layer_add(T *yt, T *side, const LayerThread &a, unsigned amask, int l, const T V[27])
{
  using L = LayerLayout<NT>;
  {
    T *b0 = yt + l * L::COMP + threadIdx.x, *b1 = yt + l * L::COMP + a.od;
    T c[18];
#pragma unroll
    for (int kj = 0; kj < 9; kj++) {
      c[2 * kj] = b0[kj * L::ROW];
      c[2 * kj + 1] = b1[kj * L::ROW];
    }
#pragma unroll
    for (int kj = 0; kj < 9; kj++) {
      b0[kj * L::ROW] = c[2 * kj] + V[3 * kj];
      b1[kj * L::ROW] = c[2 * kj + 1] + V[3 * kj + 1];
    }
  }
  __syncwarp(amask);
  {
    T *b2 = a.to_side ? side + (threadIdx.x >> 5) * 27 + l : yt + l * L::COMP + a.en;
    const int s = a.to_side ? 3 : L::ROW;
    T c[9];
#pragma unroll
    for (int kj = 0; kj < 9; kj++) c[kj] = b2[kj * s];
#pragma unroll
    for (int kj = 0; kj < 9; kj++) b2[kj * s] = c[kj] + V[3 * kj + 2];
  }
  __syncwarp(amask);
}

// The tile's sums to scratch: the side buffer's columns added to their tile
// entries, then one bulk copy of the tile.
template <typename T, int NT>
__device__ __forceinline__ void layer_dump(T *yt, T *side, const LayerThread &a, T *__restrict__ out)
{
  using L = LayerLayout<NT>;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned last = __ballot_sync(0xffffffffu, a.active && a.to_side);
  if (last && lane < 27) {
    const int kj = lane / 3, l = lane - 3 * kj;
    yt[l * L::COMP + kj * L::ROW + 32 * (warp + 1)] += side[warp * 27 + lane];
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(yt);
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(out), "r"(s),
                 "r"((uint32_t)(sizeof(T) * L::TILE))
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // before the tile's memory is given back
  }
}

// One element (thread a), Gauss plane A: element_plane of the streaming
// kernel on the layer tile's entries.
template <typename T, int NT>
__device__ __forceinline__ void layer_plane(int A, const T *ut, T *yt, T *side, const LayerThread &a, unsigned amask,
                                            const T *__restrict__ Ke)
{
  using L = LayerLayout<NT>;
  T G[3][3][9];  // [d][l][b*3+c]
#pragma unroll
  for (int l = 0; l < 3; l++) {
    T Q[9], R[9];
    const T *ul = ut + l * L::COMP;
#pragma unroll
    for (int j = 0; j < 3; j++)
#pragma unroll
      for (int i = 0; i < 3; i++) {
        const T *p = ul + (i == 0 ? (int)threadIdx.x : (i == 1 ? a.od : a.en)) + j * L::ROW;
        zeta_fwd_rt<T>(A, p[0], p[L::PLANE], p[2 * L::PLANE], Q[3 * j + i], R[3 * j + i]);
      }
    q2::plane_fwd(Q, R, G[0][l], G[1][l], G[2][l]);
  }
  // K of the next two points in flight while one computes, as in the streaming kernel
  const T *kp = Ke + koff(9 * A, 0);
  T Kn[9], Kn2[9];
#pragma unroll
  for (int r = 0; r < 9; r++) Kn[r] = ldk(kp + koff(0, r));
#pragma unroll
  for (int r = 0; r < 9; r++) Kn2[r] = ldk(kp + koff(1, r));
#pragma unroll
  for (int p = 0; p < 9; p++) {
    T Kq[9];
#pragma unroll
    for (int r = 0; r < 9; r++) Kq[r] = Kn[r];
#pragma unroll
    for (int r = 0; r < 9; r++) Kn[r] = Kn2[r];
    if (p < 7) {
#pragma unroll
      for (int r = 0; r < 9; r++) Kn2[r] = ldk(kp + koff(p + 2, r));
    }
    q2::qp_action_K(Kq, G, p);
  }
#pragma unroll
  for (int l = 0; l < 3; l++) {
    T Qt[9], Rt[9];
    q2::plane_bwd(G[0][l], G[1][l], G[2][l], Qt, Rt);
    T C[27];
#pragma unroll
    for (int ji = 0; ji < 9; ji++) zeta_bwd_rt<T>(A, Qt[ji], Rt[ji], C[ji], C[9 + ji], C[18 + ji]);
    layer_add<T, NT>(yt, side, a, amask, l, C);
  }
}

// One tile; the whole CTA.  mbits: packed Dirichlet mask or null.
template <typename T, int NT>
__device__ __forceinline__ void layer_tile(const LayerGrid &g, int tile, const T *__restrict__ K,
                                           const T *__restrict__ u, const uint32_t *__restrict__ mbits,
                                           T *__restrict__ out)
{
  using L = LayerLayout<NT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *ut = reinterpret_cast<T *>(smem_raw);
  T *yt = ut + L::TILE;
  T *side = yt + L::TILE;
  // the gather may be scheduled as soon as every tile has started; it waits
  // for this grid's stores before it reads
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const LayerThread a = layer_thread<NT>(g, tile);
  const int64_t e0 = (int64_t)tile * g.E, e1 = min(e0 + g.E, (int64_t)g.nel);
  prefetch_k(K, 0, e0, e1);
  const LayerLines ll = layer_fetch<T, NT>(ut, yt, g, tile, u);
  layer_land<T, NT>(ut, g, ll, mbits);
  layer_zero<T, NT>(yt);  // the stage was there
  __syncthreads();
  const unsigned amask = __ballot_sync(0xffffffffu, a.active);
  const T *Ke = K + kelem(a.e);
#pragma unroll 1
  for (int A = 0; A < 3; A++) {
    if (A < 2) prefetch_k(K, A + 1, e0, e1);
    if (a.active) layer_plane<T, NT>(A, ut, yt, side, a, amask, Ke);
  }
  layer_dump<T, NT>(yt, side, a, out + (int64_t)tile * L::TILE);
}

// FP64 256 threads per SM (252 registers, the streaming kernel's budget), FP32 512.
template <typename T, int NT>
constexpr int layer_min_blocks()
{
  return (sizeof(T) == 4 ? 512 : 256) / NT;
}

template <typename T, int NT>
__global__ void __launch_bounds__(NT, layer_min_blocks<T, NT>()) a11_layer_kernel(LayerGrid g, int tile0,
                                                                                  const T *__restrict__ K,
                                                                                  const T *__restrict__ u,
                                                                                  const uint32_t *__restrict__ mbits,
                                                                                  T *__restrict__ out)
{
  layer_tile<T, NT>(g, tile0 + (int)blockIdx.x, K, u, mbits, out);
}

// P: four factors per point beyond K, in blocks like K (geom_layer_kernel).
constexpr int PN = 4;
constexpr int PBLOCK = 27 * PN * KB;
__host__ __device__ __forceinline__ int64_t pelem(int64_t e) { return e / KB * PBLOCK + e % KB; }
__host__ __device__ constexpr int poff(int q, int r) { return (PN * q + r) * KB; }
__host__ __device__ __forceinline__ int64_t psize(int64_t nel) { return (nel + KB - 1) / KB * PBLOCK; }

// Gradient of component l of a tile's field at Gauss plane A (h^-1 d/dxi).
template <int NT>
__device__ __forceinline__ void layer_gradient(int A, const double *t, const LayerThread &a, int l, double G0[9],
                                               double G1[9], double G2[9])
{
  using L = LayerLayout<NT>;
  double Q[9], R[9];
  const double *tl = t + l * L::COMP;
#pragma unroll
  for (int j = 0; j < 3; j++)
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double *p = tl + (i == 0 ? (int)threadIdx.x : (i == 1 ? a.od : a.en)) + j * L::ROW;
      zeta_fwd_rt<double>(A, p[0], p[L::PLANE], p[2 * L::PLANE], Q[3 * j + i], R[3 * j + i]);
    }
  q2::plane_fwd(Q, R, G0, G1, G2);
}

// G[d][l][p] = h^-1 d x_l / d xi_d at the 9 points of Gauss plane A.
template <int NT>
__device__ __forceinline__ void layer_jacobian(int A, const double *xt, const LayerThread &a, double G[3][3][9])
{
#pragma unroll
  for (int l = 0; l < 3; l++) layer_gradient<NT>(A, xt, a, l, G[0][l], G[1][l], G[2][l]);
}

// Element e's four pressure sums.
__device__ __forceinline__ void store_p(double *yp, int e, const double Y[4])
{
  double *y = yp + 4 * (int64_t)e;
  if ((reinterpret_cast<uintptr_t>(yp) & 15) == 0) {
    reinterpret_cast<double2 *>(y)[0] = make_double2(Y[0], Y[1]);
    reinterpret_cast<double2 *>(y)[1] = make_double2(Y[2], Y[3]);
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++) y[i] = Y[i];
  }
}

// The whole Stokes operator on the A11 tiles: with P (four more factors per
// point, see the set-up) the pressure is one number added to the symmetric
// stress before it meets K again, and the divergence is the trace that the
// viscous action has formed, so A12 and A21 cost neither a forward nor a
// transposed contraction nor a scatter of their own.  DIV: yp = B u.
template <int NT, bool DIV>
__device__ __forceinline__ void stokes_plane(int A, const double *ut, double *yt, double *side, const LayerThread &a,
                                             unsigned amask, const double *__restrict__ Ke,
                                             const double *__restrict__ Pe, const double pe[4], double Y[4])
{
  double G[3][3][9];
  layer_jacobian<NT>(A, ut, a, G);
  // the next point's factors are in flight while one computes
  const double *kp = Ke + koff(9 * A, 0), *pp = Pe + poff(9 * A, 0);
  double Kn[9], Pn[4];
#pragma unroll
  for (int r = 0; r < 9; r++) Kn[r] = ldk(kp + koff(0, r));
#pragma unroll
  for (int r = 0; r < 4; r++) Pn[r] = ldk(pp + poff(0, r));
#pragma unroll
  for (int p = 0; p < 9; p++) {
    double Kq[9], Pq[4];
#pragma unroll
    for (int r = 0; r < 9; r++) Kq[r] = Kn[r];
#pragma unroll
    for (int r = 0; r < 4; r++) Pq[r] = Pn[r];
    if (p < 8) {
#pragma unroll
      for (int r = 0; r < 9; r++) Kn[r] = ldk(kp + koff(p + 1, r));
#pragma unroll
      for (int r = 0; r < 4; r++) Pn[r] = ldk(pp + poff(p + 1, r));
    }
    const double pq = pe[0] + (pe[1] * Pq[1] + (pe[2] * Pq[2] + pe[3] * Pq[3]));
    const double f = Pq[0] * q2::qp_action_Ks<double, true>(Kq, G, p, Pq[0] * pq);
    if (DIV) {
      Y[0] += f;
#pragma unroll
      for (int d = 0; d < 3; d++) Y[1 + d] = fma(f, Pq[1 + d], Y[1 + d]);
    }
  }
#pragma unroll
  for (int l = 0; l < 3; l++) {
    double Qt[9], Rt[9], C[27];
    q2::plane_bwd(G[0][l], G[1][l], G[2][l], Qt, Rt);
#pragma unroll
    for (int ji = 0; ji < 9; ji++) zeta_bwd_rt<double>(A, Qt[ji], Rt[ji], C[ji], C[9 + ji], C[18 + ji]);
    layer_add<double, NT>(yt, side, a, amask, l, C);
  }
}

// pr and yp may be one vector: an element's thread reads its four entries before it
// writes them.
template <int NT, bool DIV>
__global__ void __launch_bounds__(NT, 256 / NT) stokes_layer_kernel(LayerGrid g, const double *__restrict__ K,
                                                                    const double *__restrict__ P,
                                                                    const double *__restrict__ u,
                                                                    const double *pr,
                                                                    const uint32_t *__restrict__ mbits,
                                                                    double *__restrict__ out, double *yp)
{
  using L = LayerLayout<NT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *ut = reinterpret_cast<double *>(smem_raw);
  double *yt = ut + L::TILE;
  double *side = yt + L::TILE;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int tile = blockIdx.x;
  const LayerThread a = layer_thread<NT>(g, tile);
  const int64_t e0 = (int64_t)tile * g.E, e1 = min(e0 + g.E, (int64_t)g.nel);
  prefetch_k(K, 0, e0, e1);
  prefetch_k<double, PN>(P, 0, e0, e1);
  const LayerLines ll = layer_fetch<double, NT>(ut, yt, g, tile, u);
  double pe[4], Y[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int i = 0; i < 4; i++) pe[i] = a.active ? pr[4 * (int64_t)a.e + i] : 0.0;
  layer_land<double, NT>(ut, g, ll, mbits);
  layer_zero<double, NT>(yt);  // the stage was there
  __syncthreads();
  const unsigned amask = __ballot_sync(0xffffffffu, a.active);
  const double *Ke = K + kelem(a.e), *Pe = P + pelem(a.e);
#pragma unroll 1
  for (int A = 0; A < 3; A++) {
    if (A < 2) {
      prefetch_k(K, A + 1, e0, e1);
      prefetch_k<double, PN>(P, A + 1, e0, e1);
    }
    if (a.active) stokes_plane<NT, DIV>(A, ut, yt, side, a, amask, Ke, Pe, pe, Y);
  }
  if (DIV && a.active) store_p(yp, a.e, Y);
  layer_dump<double, NT>(yt, side, a, out + (int64_t)tile * L::TILE);
}

// diag(A11): the same tiles without an input, q2::diag_form_plane per plane
// and component as in the streaming diagonal (kernels_diag.cuh).
template <int NT>
__global__ void __launch_bounds__(NT, 256 / NT) diag_layer_kernel(LayerGrid g, const double *__restrict__ K,
                                                                  double *__restrict__ out)
{
  using L = LayerLayout<NT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *yt = reinterpret_cast<double *>(smem_raw);
  double *side = yt + L::TILE;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int tile = blockIdx.x;
  const LayerThread a = layer_thread<NT>(g, tile);
  const int64_t e0 = (int64_t)tile * g.E, e1 = min(e0 + g.E, (int64_t)g.nel);
  prefetch_k(K, 0, e0, e1);
  layer_zero<double, NT>(yt);
  __syncthreads();
  const unsigned amask = __ballot_sync(0xffffffffu, a.active);
  const double *Ke = K + kelem(a.e);
#pragma unroll 1
  for (int A = 0; A < 3; A++) {
    if (A < 2) prefetch_k(K, A + 1, e0, e1);
    if (!a.active) continue;
    double z[3][3];
#pragma unroll
    for (int s = 0; s < 3; s++)
#pragma unroll
      for (int k = 0; k < 3; k++) z[s][k] = c_zdiag[A][s][k];
    const double *kp = Ke + koff(9 * A, 0);
    double S[27];
#pragma unroll 1
    for (int m = 0; m < 3; m++) {
      const double *km = kp + koff(0, 3 * m);
      double Q[27];
      q2::diag_form_plane<double>([&](int p, int d) { return ldk(km + koff(p, d)); }, z, Q);
#pragma unroll
      for (int n = 0; n < 27; n++) S[n] = m == 0 ? Q[n] : S[n] + Q[n];
      layer_add<double, NT>(yt, side, a, amask, m, Q);
    }
#pragma unroll 1
    for (int l = 0; l < 3; l++) layer_add<double, NT>(yt, side, a, amask, l, S);
  }
  layer_dump<double, NT>(yt, side, a, out + (int64_t)tile * L::TILE);
}

// ---------------------------------------------------------------------------
// Set-up on the same tiles: the coordinates take the place of u
// ---------------------------------------------------------------------------
// J at point p of a plane's scaled gradient
__device__ __forceinline__ void layer_point(const double G[3][3][9], int p, double J[3][3])
{
#pragma unroll
  for (int k = 0; k < 3; k++)
#pragma unroll
    for (int l = 0; l < 3; l++) J[k][l] = q2::DH * G[k][l][p];
}

// The tile's coordinates in shared memory, for every thread.
template <int NT>
__device__ __forceinline__ void layer_fetch_coords(double *xt, void *stage, const LayerGrid &g, int tile,
                                                   const double *__restrict__ coords)
{
  const LayerLines ll = layer_fetch<double, NT>(xt, stage, g, tile, coords);
  layer_land<double, NT>(xt, g, ll, nullptr);
}

constexpr int LAYER_STAGE_BYTES = 1024;  // segment table of a fetch that has no second tile (at most 40 entries)

template <int NT>
constexpr size_t layer_geom_smem_bytes()
{
  return sizeof(double) * (size_t)LayerLayout<NT>::TILE + LAYER_STAGE_BYTES;
}

// Node n of component l of the thread's element in a tile.
template <int NT>
__device__ __forceinline__ double layer_node(const double *t, const LayerThread &a, int l, int n)
{
  using L = LayerLayout<NT>;
  return t[l * L::COMP + n / 9 * L::PLANE + n / 3 % 3 * L::ROW +
           (n % 3 == 0 ? (int)threadIdx.x : (n % 3 == 1 ? a.od : a.en))];
}

// I[l][q] = coordinate l at the element's 27 Gauss points.
template <int NT>
__device__ __forceinline__ void layer_points(const double *xt, const LayerThread &a, double I[3][27])
{
#pragma unroll
  for (int l = 0; l < 3; l++) {
    double f[27];
#pragma unroll
    for (int n = 0; n < 27; n++) f[n] = layer_node<NT>(xt, a, l, n);
    q2::interp(f, I[l]);
  }
}

// The P1GRel frame: mean of the element's nodes and inverse extents.
template <int NT>
__device__ __forceinline__ void layer_frame(const double *xt, const LayerThread &a, double mean[3], double invL[3])
{
#pragma unroll
  for (int l = 0; l < 3; l++) {
    double s = 0.0;
#pragma unroll
    for (int n = 0; n < 27; n++) s += layer_node<NT>(xt, a, l, n);
    mean[l] = (1.0 / 27.0) * s;
  }
  invL[0] = 1.0 / (layer_node<NT>(xt, a, 0, 14) - layer_node<NT>(xt, a, 0, 12));
  invL[1] = 1.0 / (layer_node<NT>(xt, a, 1, 16) - layer_node<NT>(xt, a, 1, 10));
  invL[2] = 1.0 / (layer_node<NT>(xt, a, 2, 22) - layer_node<NT>(xt, a, 2, 4));
}

// J at point q from the coordinates at the points
__device__ __forceinline__ void layer_point_jacobian(const double I[3][27], int q, double J[3][3])
{
  const int qa = q / 9, qb = q / 3 % 3, qc = q % 3;
#pragma unroll
  for (int l = 0; l < 3; l++) {
    const double *x = I[l];
    J[0][l] = q2::lineD_at(x[9 * qa + 3 * qb], x[9 * qa + 3 * qb + 1], x[9 * qa + 3 * qb + 2], qc);
    J[1][l] = q2::lineD_at(x[9 * qa + qc], x[9 * qa + 3 + qc], x[9 * qa + 6 + qc], qb);
    J[2][l] = q2::lineD_at(x[3 * qb + qc], x[9 + 3 * qb + qc], x[18 + 3 * qb + qc], qa);
  }
}

// K at every Gauss point, in FP64 and (K32 not null) FP32 in one pass over the
// coordinates; *bad counts the points with c = w eta / det <= 0 or not finite.
// The live state is the coordinates at the element's 27 points, 81 values in
// registers (arrays in local memory and a pass per precision took 4.1 ms at
// 128^3), and the stores are whole lines of the K blocks.  J is formed by the
// operations of element_jacobian in their order -- its entries are differences
// of nearby coordinates, so another order moves K by 1e-14 -- which is why
// this does not go plane by plane like the apply.
//
// PRESSURE: also P, the factors of the whole Stokes operator beyond K, four per
// point and blocked like K: S = -w / sqrt(c), and the P1GRel basis functions
// x^_d of P3D_ConstructNi_P1GRel_3D (src/element_utils_q2.c:183-224).
template <int NT, bool PRESSURE>
__global__ void __launch_bounds__(NT, 256 / NT) geom_layer_kernel(LayerGrid g, const double *__restrict__ coords,
                                                                  const double *__restrict__ eta,
                                                                  double *__restrict__ K, float *__restrict__ K32,
                                                                  double *__restrict__ P,
                                                                  unsigned int *__restrict__ bad)
{
  using L = LayerLayout<NT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *xt = reinterpret_cast<double *>(smem_raw);
  const int tile = blockIdx.x;
  const LayerThread a = layer_thread<NT>(g, tile);
  layer_fetch_coords<NT>(xt, xt + L::TILE, g, tile, coords);
  if (!a.active) return;
  double mean[3], invL[3];
  if (PRESSURE) layer_frame<NT>(xt, a, mean, invL);
  double I[3][27];
  layer_points<NT>(xt, a, I);
  const double *ee = eta + 27 * (int64_t)a.e;
  const int64_t k0 = kelem(a.e);
  unsigned nbad = 0;
#pragma unroll
  for (int q = 0; q < 27; q++) {
    double J[3][3], Kq[9], e;
    // one point at a time: square roots and divisions of several in flight spill
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(e) : "l"(ee + q) : "memory");
    layer_point_jacobian(I, q, J);
    double root;
    if (!q2::geom_K(J, q2::weight(q) * e, Kq, &root)) nbad++;
#pragma unroll
    for (int r = 0; r < 9; r++) {
      K[k0 + koff(q, r)] = Kq[r];
      if (K32) K32[k0 + koff(q, r)] = (float)Kq[r];
    }
    if (PRESSURE) {
      double *Pe = P + pelem(a.e) + poff(q, 0);
      Pe[0] = -q2::weight(q) / root;
#pragma unroll
      for (int d = 0; d < 3; d++) Pe[(1 + d) * KB] = (I[d][q] - mean[d]) * invL[d];
    }
  }
  if (nbad) atomicAdd(bad, nbad);
}

// Body-force load of the momentum residual (src/stokes_form_function.c:201-213):
// F[n,l] = sum_q w_q det(J_q) N_n(q) Fu_l(q), fu = [27 nel][3], to scratch.
template <int NT>
__global__ void __launch_bounds__(NT, 256 / NT) body_force_layer_kernel(LayerGrid g, const double *__restrict__ coords,
                                                                        const double *__restrict__ fu,
                                                                        double *__restrict__ out)
{
  using L = LayerLayout<NT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *xt = reinterpret_cast<double *>(smem_raw);
  double *yt = xt + L::TILE;
  double *side = yt + L::TILE;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int tile = blockIdx.x;
  const LayerThread a = layer_thread<NT>(g, tile);
  layer_fetch_coords<NT>(xt, yt, g, tile, coords);
  layer_zero<double, NT>(yt);
  __syncthreads();
  const unsigned amask = __ballot_sync(0xffffffffu, a.active);
#pragma unroll 1
  for (int A = 0; A < 3; A++) {
    if (!a.active) continue;
    double G[3][3][9], wd[9];
    layer_jacobian<NT>(A, xt, a, G);
#pragma unroll
    for (int p = 0; p < 9; p++) {
      double J[3][3], adj[3][3];
      layer_point(G, p, J);
      wd[p] = q2::weight(p) * (A == 1 ? q2::W1 / q2::W0 : 1.0) * q2::adjugate(J, adj);
    }
    const double *f = fu + 3 * (27 * (int64_t)a.e + 9 * A);
#pragma unroll 1
    for (int l = 0; l < 3; l++) {
      double r[9], Sx[9], Qt[9], V[27];
#pragma unroll
      for (int p = 0; p < 9; p++) r[p] = wd[p] * f[3 * p + l];
#pragma unroll
      for (int c = 0; c < 3; c++) q2::lineBt(r[c], r[3 + c], r[6 + c], Sx[c], Sx[3 + c], Sx[6 + c]);
#pragma unroll
      for (int j = 0; j < 3; j++)
        q2::lineBt(Sx[3 * j], Sx[3 * j + 1], Sx[3 * j + 2], Qt[3 * j], Qt[3 * j + 1], Qt[3 * j + 2]);
#pragma unroll
      for (int ji = 0; ji < 9; ji++) zeta_bwd_rt<double>(A, Qt[ji], 0.0, V[ji], V[9 + ji], V[18 + ji]);
      layer_add<double, NT>(yt, side, a, amask, l, V);
    }
  }
  layer_dump<double, NT>(yt, side, a, out + (int64_t)tile * L::TILE);
}

// ---------------------------------------------------------------------------
// Divergence and gradient
// ---------------------------------------------------------------------------
// D: the factors of B and B^T, 12 per Gauss point, blocked like K: entries
// 3k + d (k, d = 0..2) are -h w adj(J)[k][d] and 9 + d the P1GRel basis
// function x^_d of P3D_ConstructNi_P1GRel_3D (src/element_utils_q2.c:183-224).
// With G' = h^-1 grad_xi u, w det div u = -sum_kd D[3k+d] G'[d][k], so
//   (B u)_i = sum_q Np_i sum_kd D[3k+d] G'[d][k],    Np = {1, x^_0, x^_1, x^_2}
//   dv'[d][l] = (sum_i p_i Np_i) D[3l+d]              (the transpose's input)
// (MatMultMF_Stokes_MixedFEM3d_A21 / _A12, src/stokes_q2p1_mf_operators_def.c:
// 423-538).  324 values per element like the 4 x 81 blocks of B itself (which
// small one-rank boxes form from D, kernels_bmat.cuh), but formed in one pass
// over the coordinates (64x48x40 70 us; the blocks straight from the coordinates
// 1,031 us) and read in whole lines by one thread per element.  Coordinates only:
// a viscosity update keeps them.
constexpr int DN = 12;
constexpr int DBLOCK = 27 * DN * KB;
__host__ __device__ __forceinline__ int64_t delem(int64_t e) { return e / KB * DBLOCK + e % KB; }
__host__ __device__ constexpr int doff(int q, int r) { return (DN * q + r) * KB; }
__host__ __device__ __forceinline__ int64_t dsize(int64_t nel) { return (nel + KB - 1) / KB * DBLOCK; }

template <int NT>
__global__ void __launch_bounds__(NT, 256 / NT) div_layer_kernel(LayerGrid g, const double *__restrict__ coords,
                                                                 double *__restrict__ D)
{
  using L = LayerLayout<NT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *xt = reinterpret_cast<double *>(smem_raw);
  const int tile = blockIdx.x;
  const LayerThread a = layer_thread<NT>(g, tile);
  layer_fetch_coords<NT>(xt, xt + L::TILE, g, tile, coords);
  if (!a.active) return;
  double mean[3], invL[3];
  layer_frame<NT>(xt, a, mean, invL);
  double I[3][27];
  layer_points<NT>(xt, a, I);
  double *De = D + delem(a.e);
#pragma unroll
  for (int q = 0; q < 27; q++) {
    double J[3][3], adj[3][3];
    layer_point_jacobian(I, q, J);
    (void)q2::adjugate(J, adj);
    const double s = -q2::DH * q2::weight(q);
#pragma unroll
    for (int r = 0; r < 9; r++) De[doff(q, r)] = s * adj[r / 3][r % 3];
#pragma unroll
    for (int d = 0; d < 3; d++) De[doff(q, 9 + d)] = (I[d][q] - mean[d]) * invL[d];
    asm volatile("" ::: "memory");  // one point at a time
  }
}

// B and B^T go component by component, so their live state is one component's
// gradient (27 values) and three tiles fit an SM instead of the apply's two.
constexpr int DIV_TILES_PER_SM = 3;

// yp = B u (Dirichlet entries of u as zeros where mbits is given): gradient and
// divergence per point, four sums per element, nothing to scatter.
template <int NT>
__global__ void __launch_bounds__(NT, DIV_TILES_PER_SM) a21_layer_kernel(LayerGrid g, const double *__restrict__ D,
                                                                         const double *__restrict__ u,
                                                                         const uint32_t *__restrict__ mbits,
                                                                         double *__restrict__ yp)
{
  using L = LayerLayout<NT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *ut = reinterpret_cast<double *>(smem_raw);
  const int tile = blockIdx.x;
  const LayerThread a = layer_thread<NT>(g, tile);
  const int64_t e0 = (int64_t)tile * g.E, e1 = min(e0 + g.E, (int64_t)g.nel);
  prefetch_k<double, DN>(D, 0, e0, e1);
  const LayerLines ll = layer_fetch<double, NT>(ut, ut + L::TILE, g, tile, u);
  layer_land<double, NT>(ut, g, ll, mbits);
  const double *De = D + delem(a.e);
  double Y[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
  for (int A = 0; A < 3; A++) {
    if (A < 2) prefetch_k<double, DN>(D, A + 1, e0, e1);
    if (!a.active) continue;
    const double *dp = De + doff(9 * A, 0);
    double f[9];
#pragma unroll
    for (int p = 0; p < 9; p++) f[p] = 0.0;
#pragma unroll 1
    for (int k = 0; k < 3; k++) {
      double m[27], G[3][9];
#pragma unroll
      for (int p = 0; p < 9; p++)
#pragma unroll
        for (int d = 0; d < 3; d++) m[3 * p + d] = ldk(dp + doff(p, 0) + (3 * k + d) * KB);
      layer_gradient<NT>(A, ut, a, k, G[0], G[1], G[2]);
#pragma unroll
      for (int p = 0; p < 9; p++)
#pragma unroll
        for (int d = 0; d < 3; d++) f[p] = fma(m[3 * p + d], G[d][p], f[p]);
    }
#pragma unroll
    for (int p = 0; p < 9; p++) {
      Y[0] += f[p];
#pragma unroll
      for (int d = 0; d < 3; d++) Y[1 + d] = fma(f[p], ldk(dp + doff(p, 9 + d)), Y[1 + d]);
    }
  }
  if (a.active) store_p(yp, a.e, Y);
}

// B^T p to scratch.
template <int NT>
__global__ void __launch_bounds__(NT, DIV_TILES_PER_SM) a12_layer_kernel(LayerGrid g, const double *__restrict__ D,
                                                                         const double *__restrict__ p,
                                                                         double *__restrict__ out)
{
  using L = LayerLayout<NT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *yt = reinterpret_cast<double *>(smem_raw);
  double *side = yt + L::TILE;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int tile = blockIdx.x;
  const LayerThread a = layer_thread<NT>(g, tile);
  const int64_t e0 = (int64_t)tile * g.E, e1 = min(e0 + g.E, (int64_t)g.nel);
  prefetch_k<double, DN>(D, 0, e0, e1);
  layer_zero<double, NT>(yt);
  double pe[4];
#pragma unroll
  for (int i = 0; i < 4; i++) pe[i] = a.active ? p[4 * (int64_t)a.e + i] : 0.0;
  __syncthreads();
  const unsigned amask = __ballot_sync(0xffffffffu, a.active);
  const double *De = D + delem(a.e);
#pragma unroll 1
  for (int A = 0; A < 3; A++) {
    if (A < 2) prefetch_k<double, DN>(D, A + 1, e0, e1);
    if (!a.active) continue;
    const double *dp = De + doff(9 * A, 0);
    double pq[9];
#pragma unroll
    for (int q = 0; q < 9; q++)
      pq[q] = pe[0] + (pe[1] * ldk(dp + doff(q, 9)) + (pe[2] * ldk(dp + doff(q, 10)) + pe[3] * ldk(dp + doff(q, 11))));
#pragma unroll 1
    for (int l = 0; l < 3; l++) {
      double G[3][9], Qt[9], Rt[9], V[27];
#pragma unroll
      for (int q = 0; q < 9; q++)
#pragma unroll
        for (int d = 0; d < 3; d++) G[d][q] = pq[q] * ldk(dp + doff(q, 0) + (3 * l + d) * KB);
      q2::plane_bwd(G[0], G[1], G[2], Qt, Rt);
#pragma unroll
      for (int ji = 0; ji < 9; ji++) zeta_bwd_rt<double>(A, Qt[ji], Rt[ji], V[ji], V[9 + ji], V[18 + ji]);
      layer_add<double, NT>(yt, side, a, amask, l, V);
    }
  }
  layer_dump<double, NT>(yt, side, a, out + (int64_t)tile * L::TILE);
}

// ---------------------------------------------------------------------------
// The gather
// ---------------------------------------------------------------------------
enum { LAYER_PLAIN = 0, LAYER_BC_COPY = 1, LAYER_BC_ONE = 2, LAYER_BC_ZERO = 3, LAYER_ADD = 4, LAYER_SUB = 5 };

// Node t of the element box (i + NX (j + NY k)): the sum of its tile entries,
// along x innermost, then rows, then layers, lower first.  BC_COPY: y_k = x_k
// on Dirichlet dofs, BC_ONE / BC_ZERO: 1 / 0 there, ADD: added to y,
// SUB: x subtracted.
struct LayerNode {
  int64_t at[2][2][2];  // scratch offsets of the node's sums, -1 where there is none
  int64_t k0;           // its first dof
};
template <int NT>
__device__ __forceinline__ LayerNode layer_node_slots(const LayerGrid &g, uint32_t t)
{
  using L = LayerLayout<NT>;
  LayerNode n;
  const uint32_t jk = g.dNX.div(t);
  const int i = (int)(t - jk * g.dNX.d);
  const int k = (int)g.dNY.div(jk);
  const int j = (int)(jk - (uint32_t)k * g.dNY.d);
  const AxisNode ay = axis_node(j, g.my), az = axis_node(k, g.mz);
#pragma unroll
  for (int q = 0; q < 2; q++)
#pragma unroll
    for (int p = 0; p < 2; p++) {
      n.at[q][p][0] = n.at[q][p][1] = -1;
      if (q < az.n && p < ay.n) {
        layer_slots<NT>(g, i, ay.e[p] + g.my * az.e[q], n.at[q][p]);
        const int o = az.l[q] * L::PLANE + ay.l[p] * L::ROW;
#pragma unroll
        for (int b = 0; b < 2; b++)
          if (n.at[q][p][b] >= 0) n.at[q][p][b] += o;
      }
    }
  n.k0 = 3 * (g.off + i + j * g.X + k * g.XY);
  return n;
}

template <typename T, int NT, int MODE>
__device__ __forceinline__ void layer_gather_node(const LayerNode &n, const T *s, const T *__restrict__ x,
                                                  const uint32_t *__restrict__ mbits, T *__restrict__ y)
{
  using L = LayerLayout<NT>;
  T acc[3] = {T(0), T(0), T(0)};
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int64_t at = n.at[i >> 2][i >> 1 & 1][i & 1];
    if (at >= 0) {
#pragma unroll
      for (int l = 0; l < 3; l++) acc[l] += __ldcg(s + at + l * L::COMP);  // not before the wait
    }
  }
#pragma unroll
  for (int l = 0; l < 3; l++) {
    const int64_t k = n.k0 + l;
    T v = acc[l];
    if (MODE == LAYER_ADD) v += y[k];
    else if (MODE == LAYER_SUB) v -= x[k];
    else if (MODE != LAYER_PLAIN && mbits && ((mbits[k >> 5] >> (k & 31)) & 1u))
      v = MODE == LAYER_BC_COPY ? x[k] : T(MODE == LAYER_BC_ONE ? 1 : 0);
    y[k] = v;
  }
}

// Nodes [t0, t1) of the element box.  The offsets are worked out while the
// tiles' kernel runs.
template <typename T, int NT, int MODE>
__global__ void __launch_bounds__(256) layer_gather_kernel(LayerGrid g, uint32_t t0, uint32_t t1,
                                                           const T *s, const T *__restrict__ x,
                                                           const uint32_t *__restrict__ mbits, T *__restrict__ y)
{
  const uint32_t t = t0 + blockIdx.x * 256u + threadIdx.x;
  if (t >= t1) return;
  const LayerNode n = layer_node_slots<NT>(g, t);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  layer_gather_node<T, NT, MODE>(n, s, x, mbits, y);
}

// Batched forms: one work item per tile (problem, tile) and one per
// LAYER_GATHER_NODES nodes (problem, first node); a problem's sums lie at its
// own offset of the batch's scratch.
constexpr int LAYER_GATHER_NODES = 512;

template <typename T, int NT, bool MASKED>
__global__ void __launch_bounds__(NT, layer_min_blocks<T, NT>()) a11_layer_batch_kernel(const BatchProb *__restrict__ probs,
                                                                                        const int2 *__restrict__ items,
                                                                                        const T *const *__restrict__ uptr,
                                                                                        T *__restrict__ scratch)
{
  const int2 it = items[blockIdx.x];
  const BatchProb &p = probs[it.x];
  layer_tile<T, NT>(p.lg, it.y, reinterpret_cast<const T *>(p.K), uptr[it.x], MASKED ? p.mbits : nullptr,
                    scratch + p.lay_off);
}

template <typename T, int NT, bool MASKED>
__global__ void __launch_bounds__(256) layer_gather_batch_kernel(const BatchProb *__restrict__ probs,
                                                                 const int2 *__restrict__ items,
                                                                 const T *const *__restrict__ uptr, const T *scratch,
                                                                 T *const *__restrict__ yptr)
{
  const int2 it = items[blockIdx.x];
  const BatchProb &p = probs[it.x];
  const LayerGrid g = p.lg;
  const uint32_t nodes = g.nodes();
  const T *s = scratch + p.lay_off, *u = uptr[it.x];
  const uint32_t *mb = MASKED ? p.mbits : nullptr;
  T *y = yptr[it.x];
  uint32_t t = (uint32_t)it.y + threadIdx.x;
  if (t >= nodes) return;
  const uint32_t t1 = min(nodes, (uint32_t)it.y + LAYER_GATHER_NODES);
  LayerNode n = layer_node_slots<NT>(g, t);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (;;) {
    layer_gather_node<T, NT, MASKED ? LAYER_BC_COPY : LAYER_PLAIN>(n, s, u, mb, y);
    t += 256;
    if (t >= t1) break;
    n = layer_node_slots<NT>(g, t);
  }
}

}  // namespace ptk
