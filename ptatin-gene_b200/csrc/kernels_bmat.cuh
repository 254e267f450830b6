// Stored divergence blocks for B u (A21) and B^T p (A12) on small one-rank boxes.
//
// Per element, B_e is the 4 x 81 block of the discrete divergence,
//     B_e[i][3n+l] = -sum_q w_q Np_i(q) (adj(J_q) grad_xi N_n)_l,
// with the P1GRel pressure basis Np of P3D_ConstructNi_P1GRel_3D
// (src/element_utils_q2.c:183-224): the element operator of
// MatMultMF_Stokes_MixedFEM3d_A21 / _A12 (src/stokes_q2p1_mf_operators_def.c:
// 423-538), stored column-major [e][3n+l][i] (a column's four entries are one
// 32-byte sector).  It depends on the coordinates only.
//
// B u is a 4 x 81 GEMV per element (one warp, a fixed-order reduction) and
// B^T p a node-centred sum over the (<= 8) elements of each node, both one
// launch with every element or dof at work at once.  On layer tiles a small box
// waits for the one thread that an element has (8^3 B u 5.6 vs 14.5 us, B^T p 7 vs
// 14.5 us), and B^T p writes and reads the tiles' sums besides (64x48x40 92 vs 103
// us); where the line lies: DIV_BLOCKS_MAX_ELEMENTS.
#pragma once

#include <cstdint>

#include "kernels_layer.cuh"

namespace ptk {

constexpr int BMAT_LD = 324;  // 4 x 81 per element
constexpr int BMAT_EL = 4;    // elements per CTA of the set-up: a 32-byte sector of D

// A Q2 node's 1-D basis function and derivative (scaled by 1/h: D carries the h)
// at the three Gauss points.
__device__ __forceinline__ void bmat_line(int node, double b[3], double d[3])
{
  const double x[3] = {-q2::GS, 0.0, q2::GS};
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const double t = x[q];
    b[q] = node == 0 ? 0.5 * t * (t - 1.0) : (node == 1 ? (1.0 + t) * (1.0 - t) : 0.5 * (1.0 + t) * t);
    d[q] = (node == 0 ? t - 0.5 : (node == 1 ? -2.0 * t : t + 0.5)) * (1.0 / q2::DH);
  }
}

// The blocks from the factors D: a warp per element, lane n = node n with its 12
// entries, so that the lanes read the same factors (broadcasts from shared memory,
// filled in whole sectors of D) and a point's 12 values feed 21 multiply-adds: 3.3
// ns per element (a thread per column 7.4), 7.3 with D from the coordinates.
__global__ void __launch_bounds__(32 * BMAT_EL) bmat_kernel(int64_t nel, const double *__restrict__ D,
                                                           double *__restrict__ Be)
{
  __shared__ __align__(16) double sh[BMAT_EL][27 * DN];
  const int64_t e0 = (int64_t)blockIdx.x * BMAT_EL;
  const double *src = D + delem(e0);
  for (int i = threadIdx.x; i < 27 * DN * BMAT_EL; i += 32 * BMAT_EL) {
    const int r = i / BMAT_EL, k = i % BMAT_EL;
    if (e0 + k < nel) sh[k][r] = src[(int64_t)r * KB + k];
  }
  __syncthreads();
  const int k = threadIdx.x / 32, n = threadIdx.x % 32;
  if (n >= 27 || e0 + k >= nel) return;
  double bx[3], dx[3], by[3], dy[3], bz[3], dz[3], f[3][4];
  bmat_line(n % 3, bx, dx);
  bmat_line(n / 3 % 3, by, dy);
  bmat_line(n / 9, bz, dz);
#pragma unroll
  for (int i = 0; i < 12; i++) f[i / 4][i % 4] = 0.0;
#pragma unroll
  for (int ab = 0; ab < 9; ab++) {
    const int a = ab / 3, b = ab % 3;
    const double bb = by[b] * bz[a], db = dy[b] * bz[a], bd = by[b] * dz[a];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const double *d = &sh[k][DN * (3 * ab + c)];
      const double c0 = dx[c] * bb, c1 = bx[c] * db, c2 = bx[c] * bd;
#pragma unroll
      for (int l = 0; l < 3; l++) {
        const double g = fma(c0, d[3 * l], fma(c1, d[3 * l + 1], c2 * d[3 * l + 2]));
        f[l][0] += g;
#pragma unroll
        for (int i = 0; i < 3; i++) f[l][1 + i] = fma(g, d[9 + i], f[l][1 + i]);
      }
    }
  }
  double2 *out = reinterpret_cast<double2 *>(Be + (e0 + k) * BMAT_LD + 12 * n);
#pragma unroll
  for (int l = 0; l < 3; l++) {
    out[2 * l] = make_double2(f[l][0], f[l][1]);
    out[2 * l + 1] = make_double2(f[l][2], f[l][3]);
  }
}

// yp[4e+i] = sum_j B_e[i][j] u_j (mask: Dirichlet entries of u as 0, or null).
// One warp per element.  The block is read as 162 16-byte pairs (rows 0 and 1,
// or 2 and 3, of a column), 32 consecutive pairs per warp load: even lanes sum
// rows 0 and 1, odd lanes rows 2 and 3, then a fixed xor-tree over the lanes of
// each parity.
__global__ void __launch_bounds__(128) bmat_a21_kernel(Box bx, const double *__restrict__ Be,
                                                       const double *__restrict__ u,
                                                       const uint8_t *__restrict__ mask, double *__restrict__ yp)
{
  const int64_t e = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (e >= (int64_t)bx.mx * bx.my * bx.mz) return;  // whole warp
  const int ei = (int)(e % bx.mx), ej = (int)((e / bx.mx) % bx.my), ek = (int)(e / ((int64_t)bx.mx * bx.my));
  const int64_t node0 = bx.off + 2 * (int64_t)ei + 2 * (int64_t)ej * bx.X + 2 * (int64_t)ek * bx.XY;
  const double2 *b2 = reinterpret_cast<const double2 *>(Be + e * BMAT_LD);
  double s0 = 0.0, s1 = 0.0;
#pragma unroll
  for (int it = 0; it < 6; it++) {
    const int idx = lane + 32 * it;
    if (idx < 162) {
      const int j = idx >> 1, n = j / 3, l = j - 3 * n;
      const int64_t k = 3 * (node0 + (n % 3) + ((n / 3) % 3) * bx.X + (n / 9) * bx.XY) + l;
      double v = u[k];
      if (mask && mask[k]) v = 0.0;
      const double2 c = b2[idx];
      s0 = fma(c.x, v, s0);
      s1 = fma(c.y, v, s1);
    }
  }
#pragma unroll
  for (int o = 16; o > 1; o >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
  }
  if (lane < 2) {
    double *y = yp + 4 * e + 2 * lane;
    y[0] = s0;
    y[1] = s1;
  }
}

// B^T p node by node, the elements in the order of ebe_gather_kernel; MODE as in
// the layer gather (PLAIN, ADD, BC_ZERO).
template <int MODE>
__global__ void bmat_a12_kernel(Box b, const double *__restrict__ Be, const double *__restrict__ p,
                                const uint8_t *__restrict__ mask, double *__restrict__ y)
{
  const int64_t n = 3 * b.XY * (2 * (int64_t)b.mz + 1);
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    const int l = (int)(t % 3);
    const int64_t node = t / 3;
    const int i = (int)(node % b.X), j = (int)((node / b.X) % (2 * b.my + 1)), k = (int)(node / b.XY);
    const AxisNode ax = axis_node(i, b.mx), ay = axis_node(j, b.my), az = axis_node(k, b.mz);
    double acc = 0.0;
    for (int c = 0; c < az.n; c++)
      for (int d = 0; d < ay.n; d++)
        for (int a = 0; a < ax.n; a++) {
          const int64_t e = ax.e[a] + (int64_t)b.mx * (ay.e[d] + (int64_t)b.my * az.e[c]);
          const double *be = Be + e * BMAT_LD + 4 * (3 * (ax.l[a] + 3 * ay.l[d] + 9 * az.l[c]) + l);
          const double2 c01 = *reinterpret_cast<const double2 *>(be);
          const double2 c23 = *reinterpret_cast<const double2 *>(be + 2);
          const double *pe = p + 4 * e;
          acc += fma(c23.y, pe[3], fma(c23.x, pe[2], fma(c01.y, pe[1], c01.x * pe[0])));
        }
    if (MODE == LAYER_ADD) acc += y[t];
    y[t] = MODE == LAYER_BC_ZERO && mask[t] ? 0.0 : acc;
  }
}

}  // namespace ptk
