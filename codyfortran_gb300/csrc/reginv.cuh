// reginv.cuh -- in-block inverse of a small complex matrix, for the regularised
// inverse of the one-body density matrix: with s = sqrt(eps),
// n / (n^2 + eps) = Re 1 / (n + i s), so U f(n) U^H is the Hermitian part of
// (rho + i s)^-1.
#pragma once
#include "common.cuh"

constexpr int RI_MAX = 32;
struct RegInvScratch {
  z_t A[RI_MAX][RI_MAX + 1];
  z_t row[RI_MAX], col[RI_MAX];
  int perm[RI_MAX], at[RI_MAX];
  // entry (i, j) of the inverse after reg_invert
  __device__ z_t inv(int i, int j) const { return A[i][at[j]]; }
};

// Gauss-Jordan with partial pivoting by the whole block (n <= 32, at least one
// warp): s.A holds the matrix, then the inverse as s.inv(i, j).  Per column, warp 0
// finds the pivot, swaps the rows and scales the pivot row, then the block updates.
// Callers synchronise the block after filling s.A.
__device__ inline void reg_invert(RegInvScratch& s, int n) {
  const int tid = threadIdx.x;
  if (tid < n) s.perm[tid] = tid;
  __syncthreads();
  for (int k = 0; k < n; k++) {
    if (tid < 32) {
      const int l = tid;
      const z_t ck = l < n ? s.A[l][k] : zmk(0.0, 0.0);
      // pivot: the largest |re| + |im| at or below the diagonal, by its FP32 size (any near-largest entry serves)
      float mag = l >= k && l < n ? fabsf((float)ck.x) + fabsf((float)ck.y) : -1.0f;
      int p = l;
      for (int o = 16; o > 0; o >>= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, mag, o);
        const int p2 = __shfl_xor_sync(0xffffffffu, p, o);
        if (m2 > mag || (m2 == mag && p2 < p)) {
          mag = m2;
          p = p2;
        }
      }
      if (!(mag >= 0.0f) || p < k || p >= n) p = k;  // NaN entries: any pivot, the result is NaN
      const z_t a = s.A[p][k], akk = s.A[k][k];
      const double d = 1.0 / fma(a.x, a.x, a.y * a.y);
      const z_t inv = zmk(a.x * d, -a.y * d);
      const z_t t = l < n ? s.A[p][l] : zmk(0.0, 0.0), u = l < n ? s.A[k][l] : zmk(0.0, 0.0);
      __syncwarp();  // every lane has read rows k and p and column k
      if (l < n) {
        s.row[l] = l == k ? inv : zmul(t, inv);
        if (p != k) s.A[p][l] = u;
        s.col[l] = l == p && p != k ? akk : ck;  // column k after the swap
      }
      if (l == 0 && p != k) {
        const int q = s.perm[k];
        s.perm[k] = s.perm[p];
        s.perm[p] = q;
      }
    }
    __syncthreads();
    for (int e = tid; e < n * n; e += blockDim.x) {
      const int i = e / n, j = e - i * n;
      if (i == k) {
        s.A[k][j] = s.row[j];
      } else {
        z_t v = j == k ? zmk(0.0, 0.0) : s.A[i][j];
        const z_t c = s.col[i], r = s.row[j];
        v.x = fma(-c.x, r.x, fma(c.y, r.y, v.x));
        v.y = fma(-c.x, r.y, fma(-c.y, r.x, v.y));
        s.A[i][j] = v;
      }
    }
    __syncthreads();
  }
  // A holds (P B)^-1: column r of it is column perm[r] of B^-1
  if (tid < n) s.at[s.perm[tid]] = tid;
  __syncthreads();
}
