// Dense inverse of a small multigrid level's operator on the device.
//
// The masked operator (Dirichlet rows and columns replaced by the identity) is
// assembled row by row from the packed element matrices and inverted in place
// by blocked Gauss-Jordan elimination without pivoting (the matrix is symmetric
// positive definite, so every pivot block is).  Per block of DN_B rows three
// launches: the pivot block's inverse, the row and column panels, the rank-DN_B
// update of the rest; 1,029 dofs (a 3^3 level) are 2.2 GFLOP in 33 steps.  By
// Cholesky on one host core the 525 dofs of a 16x24x16 box's coarsest level
// were 35 of the 41 ms of its hierarchy's set-up (now 6 ms).
#pragma once

#include <cstdint>

#include "kernels_ebe.cuh"

namespace ptk {

constexpr int DN_B = 32;

// Row blockIdx.x of A (np x np, row stride np; rows and columns n..np-1 are the
// identity's).  The row's elements one after the other, lower first.
__global__ void __launch_bounds__(96) dense_assemble_kernel(Box b, const double *__restrict__ Ae,
                                                            const uint8_t *__restrict__ mask, int n, int np,
                                                            double *__restrict__ A)
{
  const int i = blockIdx.x;
  double *row = A + (int64_t)i * np;
  for (int j = threadIdx.x; j < np; j += blockDim.x) row[j] = 0.0;
  __syncthreads();
  if (i >= n || mask[i]) {
    if (threadIdx.x == 0) row[i] = 1.0;
    return;
  }
  const int l = i % 3;
  const int64_t node = i / 3;
  const int X = (int)b.X, Y = 2 * b.my + 1;
  const int x = (int)(node % X), y = (int)(node / X % Y), z = (int)(node / b.XY);
  for (int c = 0; c < 8; c++) {
    // element h-1 (local node 2) and h (0) of an even node, h (1) of an odd one
    const int cx = c & 1, cy = c >> 1 & 1, cz = c >> 2;
    if ((!cx && (x & 1)) || (!cy && (y & 1)) || (!cz && (z & 1))) continue;
    const int ex = (x >> 1) - 1 + cx, ey = (y >> 1) - 1 + cy, ez = (z >> 1) - 1 + cz;
    if (ex < 0 || ey < 0 || ez < 0 || ex >= b.mx || ey >= b.my || ez >= b.mz) continue;
    const int nl = (x - 2 * ex) + 3 * (y - 2 * ey) + 9 * (z - 2 * ez), ii = 3 * nl + l;
    const double *m = Ae + (ex + (int64_t)b.mx * (ey + (int64_t)b.my * ez)) * EBE_LD;
    const int jj = threadIdx.x;
    if (jj < 81) {
      const int q = jj / 3;
      const int64_t g = 3 * ((2 * ex + q % 3) + (2 * ey + q / 3 % 3) * b.X + (2 * ez + q / 9) * b.XY) + jj % 3;
      if (!mask[g]) row[g] += m[ebe_sym(ii, jj)];
    }
    __syncthreads();
  }
}

// D = inverse of the pivot block k; *bad = 1 if a pivot is not positive.
__global__ void __launch_bounds__(DN_B *DN_B) dense_pivot_kernel(const double *__restrict__ A, int np, int k,
                                                                double *__restrict__ D, int *__restrict__ bad)
{
  __shared__ double s[DN_B][DN_B + 1];
  const int j = threadIdx.x % DN_B, i = threadIdx.x / DN_B;
  s[i][j] = A[(int64_t)(k * DN_B + i) * np + k * DN_B + j];
  __syncthreads();
  for (int p = 0; p < DN_B; p++) {
    const double d = s[p][p], r = 1.0 / d, a = s[i][j], ip = s[i][p], pj = s[p][j];
    if (threadIdx.x == 0 && !(d > 0.0)) *bad = 1;
    __syncthreads();
    s[i][j] = i == p ? (j == p ? r : pj * r) : (j == p ? -ip * r : a - ip * (pj * r));
    __syncthreads();
  }
  D[threadIdx.x] = s[i][j];
}

// Block t != k: row panel A[k][t] <- D A[k][t] (kept in R, DN_B x np) and column
// panel A[t][k] -> C (np x DN_B), A[t][k] <- -A[t][k] D.  Block k: A[k][k] <- D.
__global__ void __launch_bounds__(256) dense_panel_kernel(double *__restrict__ A, int np, int k,
                                                          const double *__restrict__ D, double *__restrict__ R,
                                                          double *__restrict__ C)
{
  __shared__ double sd[DN_B][DN_B + 1], sr[DN_B][DN_B + 1], sc[DN_B][DN_B + 1];
  const int t = blockIdx.x, j = threadIdx.x % DN_B, i0 = threadIdx.x / DN_B;
  for (int i = i0; i < DN_B; i += 8) {
    sd[i][j] = D[i * DN_B + j];
    sr[i][j] = A[(int64_t)(k * DN_B + i) * np + t * DN_B + j];
    sc[i][j] = A[(int64_t)(t * DN_B + i) * np + k * DN_B + j];
  }
  __syncthreads();
  for (int i = i0; i < DN_B; i += 8) {
    if (t == k) {
      A[(int64_t)(k * DN_B + i) * np + k * DN_B + j] = sd[i][j];
      continue;
    }
    double r = 0.0, c = 0.0;
#pragma unroll 8
    for (int m = 0; m < DN_B; m++) {
      r = fma(sd[i][m], sr[m][j], r);
      c = fma(sc[i][m], sd[m][j], c);
    }
    A[(int64_t)(k * DN_B + i) * np + t * DN_B + j] = r;
    R[(int64_t)i * np + t * DN_B + j] = r;
    A[(int64_t)(t * DN_B + i) * np + k * DN_B + j] = -c;
    C[(int64_t)(t * DN_B + i) * DN_B + j] = sc[i][j];
  }
}

// A[i][j] -= C[i] R[j] for blocks i, j != k.
__global__ void __launch_bounds__(256) dense_update_kernel(double *__restrict__ A, int np, int k,
                                                           const double *__restrict__ R, const double *__restrict__ C)
{
  __shared__ double sr[DN_B][DN_B + 1], sc[DN_B][DN_B + 1];
  const int bi = blockIdx.y, bj = blockIdx.x, j = threadIdx.x % DN_B, i0 = threadIdx.x / DN_B;
  if (bi == k || bj == k) return;
  for (int i = i0; i < DN_B; i += 8) {
    sr[i][j] = R[(int64_t)i * np + bj * DN_B + j];
    sc[i][j] = C[(int64_t)(bi * DN_B + i) * DN_B + j];
  }
  __syncthreads();
  double *a = A + (int64_t)(bi * DN_B) * np + bj * DN_B + j;
  double v[DN_B / 8];
#pragma unroll
  for (int q = 0; q < DN_B / 8; q++) v[q] = a[(int64_t)(i0 + 8 * q) * np];
#pragma unroll 8
  for (int m = 0; m < DN_B; m++)
#pragma unroll
    for (int q = 0; q < DN_B / 8; q++) v[q] = fma(-sc[i0 + 8 * q][m], sr[m][j], v[q]);
#pragma unroll
  for (int q = 0; q < DN_B / 8; q++) a[(int64_t)(i0 + 8 * q) * np] = v[q];
}

// The leading n x n part as T.
template <typename T>
__global__ void dense_copy_kernel(const double *__restrict__ A, int np, int n, T *__restrict__ out)
{
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < (int64_t)n * n; t += (int64_t)gridDim.x * blockDim.x)
    out[t] = (T)A[t / n * np + t % n];
}

}  // namespace ptk
