// Gauss-point viscosity and density from material points: the reference's
// default coefficient projection (coefficient_projection_type 1, "Q1") on one
// rank, src/material_point_utils.c:1090-1190 and 957-1088.
//
//   node sums over the markers of each element:  A1 += N_i eta_p,
//   A2 += N_i rho_p, B += N_i, with N_i the Q1 basis at the marker's local
//   coordinates on the element's 8 vertices (Q2 nodes 0,2,6,8,18,20,24,26)
//   and 1 on its other 19 nodes;  A1 /= B, A2 /= B;  at each Gauss point the
//   Q1 interpolant of the vertex values, clamped to the range of the
//   element's 27 node values.
//
// Deterministic without atomics: markers are sorted by element (stable radix
// sort, so each element keeps its markers in input order), eight lanes sum an
// element's markers (lane = vertex), and a per-node gather adds the (<= 8)
// element sums in a fixed order.  Node arrays are indexed compactly over the
// element box's own nodes.
#pragma once

#include <cstdint>

namespace ptk {

// Q1 basis of pTatinConstructNI_Q1_3D (src/material_point_utils.c:503-520),
// vertex v = k*4 + j*2 + i.
__device__ __forceinline__ double mk_q1(int v, double x, double y, double z)
{
  const double a = (v & 1) ? 1.0 + x : 1.0 - x;
  const double b = (v & 2) ? 1.0 + y : 1.0 - y;
  const double c = (v & 4) ? 1.0 + z : 1.0 - z;
  return 0.125 * a * b * c;
}

// Sort keys and payload: key = element index, with every index outside
// [0, nel) mapped to nel so that a radix sort over the bits of nel suffices;
// payload = marker index.
__global__ void mk_keys_kernel(const int32_t *__restrict__ wil, int64_t n, int32_t nel, int32_t *__restrict__ key,
                               int32_t *__restrict__ idx)
{
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t w = wil[i];
    key[i] = (w >= 0 && w < nel) ? w : nel;
    idx[i] = (int32_t)i;
  }
}

// start[e] = first sorted position with key >= e, e = 0..nel
__global__ void mk_starts_kernel(const int32_t *__restrict__ keys, int64_t n, int64_t nel, int64_t *__restrict__ start)
{
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e <= nel; e += (int64_t)gridDim.x * blockDim.x) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (keys[mid] < e) lo = mid + 1;
      else hi = mid;
    }
    start[e] = lo;
  }
}

// Sums over an element's markers, 27 values: (N eta, N rho, N) for its 8
// vertices and, once for the other 19 nodes whose weight is 1, (eta, rho, 1).
// Eight lanes per element, lane v = vertex v, four elements per warp; every
// lane walks the element's markers in order (the eight read the same address),
// MK_AHEAD of them loaded before they are used.  A warp per element with one
// lane per node kept 81 sums per element, 19 times the same ones, and moved
// every marker through ten shuffles: 64^3 with 2.1 M markers 186 us.
//
// A crowded element, which the others do not hide, pays two dependent round trips
// per MK_AHEAD markers (160 ns a marker).  There lane v takes marker v of every
// eight, an index ahead of its data and the data ahead of their sums, and the eight
// are passed from lane to lane in order (same sums, 124 ns; 8^3 with 4096 per
// element 1,215 -> 717 us, 100,000 in one element 16.0 -> 12.4 ms).  Where there
// are elements enough to hide the trips the shuffles cost more than they save
// (32^3 with 256 per element 444 vs 578 us), so a box that fills the chip (about
// MK_FEW elements) goes that way for its outliers only.
constexpr int MK_SUMS = 27;
constexpr int MK_AHEAD = 4;
constexpr int64_t MK_FEW = 16384;                      // elements
constexpr int64_t MK_CROWDED_FEW = 256, MK_CROWDED = 1024;  // markers in an element

__device__ __forceinline__ void mk_store(double *o, int v, double s1, double s2, double sb, double c1, double c2,
                                         int64_t n)
{
  o[3 * v] = s1;
  o[3 * v + 1] = s2;
  o[3 * v + 2] = sb;
  if (v == 0) {
    o[24] = c1;
    o[25] = c2;
    o[26] = (double)n;
  }
}

// A crowded element, lane v; out of line so that the common loop keeps its registers.
__device__ __noinline__ void mk_crowded(int v, int64_t m0, int64_t m1, const int32_t *__restrict__ order,
                                        const double *__restrict__ xi, const double *__restrict__ eta,
                                        const double *__restrict__ rho, double *__restrict__ o)
{
  const unsigned group = 0xffu << (threadIdx.x & 24);
  double s1 = 0.0, s2 = 0.0, sb = 0.0, c1 = 0.0, c2 = 0.0;
  double a[5] = {};  // lane v: marker v of the eight under way
  const auto index = [&](int64_t c) { return c + v < m1 ? order[c + v] : -1; };
  const auto load = [&](int64_t p) {
    if (p < 0) return;
    a[0] = xi[3 * p];
    a[1] = xi[3 * p + 1];
    a[2] = xi[3 * p + 2];
    a[3] = eta[p];
    a[4] = rho[p];
  };
  load(index(m0));
  int64_t next = index(m0 + 8);
  for (int64_t c0 = m0; c0 < m1; c0 += 8) {
    double m[5];
#pragma unroll
    for (int i = 0; i < 5; i++) m[i] = a[i];
    load(next);  // in flight while this eight is summed
    next = index(c0 + 16);
    const int n = (int)min((int64_t)8, m1 - c0);
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (k < n) {
        double w[5];
#pragma unroll
        for (int i = 0; i < 5; i++) w[i] = __shfl_sync(group, m[i], k, 8);
        const double N = mk_q1(v, w[0], w[1], w[2]);
        s1 += N * w[3];
        s2 += N * w[4];
        sb += N;
        c1 += w[3];
        c2 += w[4];
      }
  }
  mk_store(o, v, s1, s2, sb, c1, c2, m1 - m0);
}

__global__ void __launch_bounds__(128) mk_element_kernel(int64_t nel, const int64_t *__restrict__ start,
                                                         const int32_t *__restrict__ order,
                                                         const double *__restrict__ xi, const double *__restrict__ eta,
                                                         const double *__restrict__ rho, double *__restrict__ part)
{
  const int64_t e = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const int v = threadIdx.x & 7;
  if (e >= nel) return;
  double s1 = 0.0, s2 = 0.0, sb = 0.0, c1 = 0.0, c2 = 0.0;
  const int64_t m0 = start[e], m1 = start[e + 1];
  if (m1 - m0 > (nel <= MK_FEW ? MK_CROWDED_FEW : MK_CROWDED)) {
    mk_crowded(v, m0, m1, order, xi, eta, rho, part + e * MK_SUMS);
    return;
  }
  for (int64_t c0 = m0; c0 < m1; c0 += MK_AHEAD) {
    double x[MK_AHEAD], y[MK_AHEAD], z[MK_AHEAD], ee[MK_AHEAD], rr[MK_AHEAD];
#pragma unroll
    for (int k = 0; k < MK_AHEAD; k++)
      if (c0 + k < m1) {
        const int64_t p = order[c0 + k];
        x[k] = xi[3 * p];
        y[k] = xi[3 * p + 1];
        z[k] = xi[3 * p + 2];
        ee[k] = eta[p];
        rr[k] = rho[p];
      }
#pragma unroll
    for (int k = 0; k < MK_AHEAD; k++)
      if (c0 + k < m1) {
        const double N = mk_q1(v, x[k], y[k], z[k]);
        s1 += N * ee[k];
        s2 += N * rr[k];
        sb += N;
        c1 += ee[k];
        c2 += rr[k];
      }
  }
  mk_store(part + e * MK_SUMS, v, s1, s2, sb, c1, c2, m1 - m0);
}

// Per node of the element box (compact index i + j X + k X Y, X = 2mx+1):
// the element sums in a fixed order, divided; (viscosity, density) side by side.
__global__ void mk_node_kernel(int mx, int my, int mz, const double *__restrict__ part, double2 *__restrict__ v12)
{
  // node count < 2^31 (checked by the caller): 32-bit index arithmetic
  const unsigned X = 2 * mx + 1, Y = 2 * my + 1;
  const unsigned nn = X * Y * (2 * mz + 1);
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < nn; t += gridDim.x * blockDim.x) {
    const unsigned txy = t / X;
    const int i = (int)(t - txy * X), j = (int)(txy % Y), k = (int)(txy / Y);
    const bool vertex = !((i | j | k) & 1);
    double a1 = 0.0, a2 = 0.0, b = 0.0;
#pragma unroll
    for (int cz = 0; cz < 2; cz++)
#pragma unroll
      for (int cy = 0; cy < 2; cy++)
#pragma unroll
        for (int cx = 0; cx < 2; cx++) {
          // elements i/2 - 1 and i/2 of an even node, i/2 of an odd one
          const int ex = (i >> 1) - 1 + cx, ey = (j >> 1) - 1 + cy, ez = (k >> 1) - 1 + cz;
          if ((cx == 0 && (i & 1)) || (cy == 0 && (j & 1)) || (cz == 0 && (k & 1))) continue;
          if (ex < 0 || ey < 0 || ez < 0 || ex >= mx || ey >= my || ez >= mz) continue;
          const int64_t e = ex + (int64_t)mx * (ey + (int64_t)my * ez);
          // this node within the element: its high vertex where the element is the lower one
          const int w = vertex ? (1 - cx) + 2 * (1 - cy) + 4 * (1 - cz) : 8;
          const double *o = part + e * MK_SUMS + 3 * w;
          a1 += o[0];
          a2 += o[1];
          b += o[2];
        }
    v12[t] = make_double2(a1 / b, a2 / b);
  }
}

// Gauss point q of element e: Q1 interpolant of the vertex values, clamped to
// the element's 27 node values, abscissae of QuadratureCreateGauss_3pnt_3D
// (src/quadrature.c:136-167).  One thread per element: the interpolant is
// formed axis by axis (a warp per element paid 72 shuffles for the range and
// the vertices: 64^3 122 us), and a block's points, which lie side by side in
// the result, leave through shared memory in whole lines.  eta2: a second copy
// of the viscosity, or null.
constexpr int MK_QP_THREADS = 128;

__global__ void __launch_bounds__(MK_QP_THREADS) mk_qp_kernel(int mx, int my, int mz, const double2 *__restrict__ v12,
                                                              double *__restrict__ eta_qp, double *__restrict__ eta2,
                                                              double *__restrict__ rho_qp)
{
  __shared__ double sh[27 * MK_QP_THREADS];
  // element count < 2^31 (checked by the caller): 32-bit index arithmetic
  const unsigned nel = (unsigned)mx * my * mz;
  const unsigned e0 = blockIdx.x * MK_QP_THREADS, e = e0 + threadIdx.x;
  const unsigned n = min((unsigned)MK_QP_THREADS, nel - e0);
  double lo[2], hi[2], vx[2][8];
  if (e < nel) {
    const int X = 2 * mx + 1, Y = 2 * my + 1;
    const unsigned exy = e / mx;
    const int ei = (int)(e - exy * mx), ej = (int)(exy % my), ek = (int)(exy / my);
    const double2 *base = v12 + 2 * (int64_t)ei + 2 * (int64_t)ej * X + 2 * (int64_t)ek * X * Y;
#pragma unroll
    for (int m = 0; m < 27; m++) {
      const double2 a = base[(m % 3) + ((m / 3) % 3) * (int64_t)X + (m / 9) * (int64_t)X * Y];
      lo[0] = m == 0 ? a.x : fmin(lo[0], a.x);
      hi[0] = m == 0 ? a.x : fmax(hi[0], a.x);
      lo[1] = m == 0 ? a.y : fmin(lo[1], a.y);
      hi[1] = m == 0 ? a.y : fmax(hi[1], a.y);
      if (m % 3 != 1 && m / 3 % 3 != 1 && m / 9 != 1) {
        const int v = (m % 3) / 2 + (m / 3 % 3) + 2 * (m / 9);
        vx[0][v] = a.x;
        vx[1][v] = a.y;
      }
    }
  }
  const double g = 0.774596669241483;
  const double w0[3] = {0.5 * (1.0 + g), 0.5, 0.5 * (1.0 - g)};  // weight of the lower node; the upper one's mirrored
#pragma unroll
  for (int f = 0; f < 2; f++) {
    double *const out = f == 0 ? eta_qp : rho_qp;
    if (f == 1 && !out) break;
    if (e < nel) {
      double a[3][4];  // along x
#pragma unroll
      for (int c = 0; c < 3; c++)
#pragma unroll
        for (int yz = 0; yz < 4; yz++) a[c][yz] = w0[c] * vx[f][2 * yz] + w0[2 - c] * vx[f][2 * yz + 1];
#pragma unroll
      for (int b = 0; b < 3; b++)
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const double b0 = w0[b] * a[c][0] + w0[2 - b] * a[c][1], b1 = w0[b] * a[c][2] + w0[2 - b] * a[c][3];
#pragma unroll
          for (int d = 0; d < 3; d++) {
            double s = w0[d] * b0 + w0[2 - d] * b1;
            if (s < lo[f]) s = lo[f];
            if (s > hi[f]) s = hi[f];
            sh[27 * threadIdx.x + 9 * d + 3 * b + c] = s;
          }
        }
    }
    __syncthreads();
    for (unsigned i = threadIdx.x; i < 27 * n; i += MK_QP_THREADS) {
      if (out) out[27 * (int64_t)e0 + i] = sh[i];
      if (f == 0 && eta2) eta2[27 * (int64_t)e0 + i] = sh[i];
    }
    __syncthreads();
  }
}

}  // namespace ptk
