// k_adjoint_mc.cu -- gradient of a final-time MCTDHF objective with respect to
// every sample of the laser field, by the exact discrete adjoint of the Strang
// step (no counterpart in the reference; the forward map is the reference's
// step: src/Propagator/SplitStep/Order2/S_Propagator_SplitStep_Order2.f90:52-77
// with fixed-order SIL on OrbsLin, src/IntegratorList/Sil/S_IntegratorList_Sil.f90:207-310,
// and RK4 on CoeffsPlusOrbsNonLin, src/Method/Mb/OrbBased/Mctdhx/S_Method_Mb_OrbBased_Mctdhx.f90:180-226).
//
// Systems: restricted MCTDHF with two body types (spins) of one particle each,
// M <= 16 spatial orbitals: the two-electron problem of the 1D helium model.
// There the configuration space is the M x M matrix C (C[a, b]: orbital a of
// body type 1, b of body type 2; state index a + M b) and the reference's
// generic CI traversals reduce to dense algebra, checked against the
// configuration-table path to rounding:
//   H1 C = h1^T C + C h1,  H2 C = sum_ab g(a, b; c, d) C[a, b],
//   g(a, b; c, d) = <phi_a| W_bd |phi_c>_w,  W_bd(x) = sum_y V(x, y) conj(phi_b(y)) phi_d(y) w(y),
//   rho1 = conj(C) C^T + C^H C (spin-summed),
//   rho2[a, b, c, d] = C[c, d] conj(C[a, b]) + C[d, c] conj(C[b, a]),
//   Mreg = U n/(n^2 + eps) U^H (rho1 = U n U^H),
//   dphi_j(x) += sum_{a, k, l, q} W_lk(x) phi_a(x) rho2[a, k, q, l] Mreg[q, j],
// then the (1 - P) projector on the orbitals, P_C on the coefficients and -i.
//
// rho2 has rank two, so neither it nor g is formed.  With
//   u_k = sum_a conj(C_ak) phi_a,  u'_k = sum_a conj(C_ka) phi_a,
//   z_l = sum_k W_lk u_k,          z'_l = sum_k W_lk u'_k,
//   X_jl = sum_q C_ql Mreg_qj,     Y_jl = sum_q C_lq Mreg_qj
// (W_bd = conj(W_db), V real)
//   H2 C [c, d] = sum_x w phi_c conj(z_d),  dphi_j += sum_l X_jl z_l + Y_jl z'_l,
// M^2 products a point instead of M^4 (and M^5 for rho2 Mreg), and the potentials of
// the M (M + 1) / 2 pairs l <= k only.  Every step of it is differentiated
// below in the reverse order; Mreg as the Hermitian part of K = (rho1 + i
// sqrt(eps))^-1 (reginv.cuh): with B the co-state of rho1 plus its adjoint,
// B = -(P + P^H), P = K herm(Mbar) K.
//
// Field: piecewise constant, E(t) = field[floor(t / dt)] (zero outside), the
// convention of the sampled laser; the one-body operator is
// h = T + V0(x) + E(t) x.  Stage times are the reference's, so step n reads
// field[n] (both SIL halves, RK4 stages 1-3) and field[n + 1] (RK4 stage 4).
//
// Objective: J = 1 - |<Psi_ref | Psi_N>|^2 with the MCTDHF overlap
// <Psi_ref|Psi> = sum conj(C_ref[a, b]) (S C S^T)[a, b], S = phi_ref^H W phi.
//
// Adjoint: co-states in the convention dL = Re sum conj(xbar) dx.  The Lanczos
// step and its reverse are one launch each (k_sil.cu).  The forward sweep keeps the
// state every `checkpoint` steps and those of the last segment; the backward sweep
// recomputes the other segments one at a time, and each step's intermediates
// (Krylov bases, the four RK4 stages) once before it is differentiated.
//
// A step is 22 launches forward and 40 more backward, most of them 3 to 10 us of
// latencies: the sums over the grid, M x M algebra by one block (beside another
// kernel's blocks where it can be), FP64 chains.  The FP64 pipe bounds the pair
// potentials (k_mc_potentials).  501 points x 8 orbitals, K = 12, per field sample:
// 27.5 ms with g, rho2 and their co-states formed, a launch per vector operation and
// the stages recomputed for every use; 1.9 ms now.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "reginv.cuh"

namespace {

constexpr int MC_T = 256;
constexpr int MC_MAXM = 16;
constexpr int MC_MAXK = 32;
constexpr int MC_RED = 512;  // threads of the one-block reductions
constexpr int MC_TX = 4;     // grid points of a block of the pointwise kernels
constexpr int MC_TT = 128;   // their threads

unsigned nblk(size_t n) { return (unsigned)std::min<size_t>((n + MC_T - 1) / MC_T, 4096); }

#define MC_LOOP(e, n) for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < (size_t)(n); e += (size_t)gridDim.x * blockDim.x)

// pair (l, k), l <= k
__host__ __device__ __forceinline__ int mc_pair(int l, int k) { return k * (k + 1) / 2 + l; }

// What one RK4 stage leaves for its reverse
struct McStage {
  z_t *Aphi, *W, *z, *zp, *dphi0;             // h phi, pair potentials, z, z', unprojected orbital derivative
  z_t *h1, *G, *Gp, *X1;                      // M x M: phi^H w h phi, phi^H w z, phi^H w dphi0, phi^H w x phi
  z_t *X, *Y, *Kinv, *Mreg, *dC0, *sc;
};

// ---- sums over the grid: out[i + M j] = sum_x conj(a_i) wgt b_j, a warp each, fixed order
struct McSum {
  const z_t *a, *b;
  const double* wgt;  // may be null
  z_t* out;
};
struct McSums {
  McSum s[4];
  int n;
};

__device__ void mc_sums(const McSums& S, int blk, int nG, int M) {
  const int lane = threadIdx.x & 31, Q = M * M;
  const int t = blk * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= S.n * Q) return;
  const int set = t / Q, o = t - set * Q;
  const McSum& D = S.s[set];
  const z_t *a = D.a + (size_t)nG * (o % M), *b = D.b + (size_t)nG * (o / M);
  z_t s = zmk(0.0, 0.0);
#pragma unroll 4
  for (int x = lane; x < nG; x += 32) {
    z_t v = b[x];
    if (D.wgt) v = zscale(v, D.wgt[x]);
    zcfma(s, a[x], v);
  }
  for (int k = 16; k > 0; k >>= 1) {
    s.x += __shfl_xor_sync(0xffffffffu, s.x, k);
    s.y += __shfl_xor_sync(0xffffffffu, s.y, k);
  }
  if (lane == 0) D.out[o] = s;
}
int mc_sum_blocks(int n, int M, int threads) { return (n * M * M + threads / 32 - 1) / (threads / 32); }

// 64 threads, so that the warps' FP64 chains lie on many SMs: 17.4 us for 4 x 64 sums
// over 501 points with 256 threads, 14.0 with 64.
constexpr int MC_ST = 64;
__global__ void __launch_bounds__(MC_ST) k_mc_sums(const McSums S, int nG, int M) { mc_sums(S, blockIdx.x, nG, M); }

// ---- M x M algebra by one block, matrices in shared memory
typedef z_t McMat[MC_MAXM * MC_MAXM];

// f(i, j) for every entry of an M x M matrix
template <class F>
__device__ __forceinline__ void mc_each(int M, F f) {
  for (int e = threadIdx.x; e < M * M; e += blockDim.x) f(e % M, e / M, e);
  __syncthreads();
}
__device__ __forceinline__ void mc_load(z_t* dst, const z_t* src, int M) {
  for (int e = threadIdx.x; e < M * M; e += blockDim.x) dst[e] = src[e];
}

// rho1 of C, K = (rho1 + i sqrt(eps))^-1, Mreg, X and Y
__device__ void mc_density(const McStage& S, const z_t* C, int M, double eps) {
  __shared__ RegInvScratch R;
  __shared__ McMat c, m;
  mc_load(c, C, M);
  __syncthreads();
  const double s0 = sqrt(eps);
  mc_each(M, [&](int i, int k, int) {
    z_t s = zmk(0.0, 0.0);
    for (int j = 0; j < M; j++) {
      zfma(s, zconj(c[i + M * j]), c[k + M * j]);
      zcfma(s, c[j + M * i], c[j + M * k]);
    }
    R.A[i][k] = i == k ? zmk(s.x, s0) : s;
  });
  reg_invert(R, M);
  mc_each(M, [&](int i, int j, int e) {
    const z_t v = R.inv(i, j), w = R.inv(j, i);
    S.Kinv[e] = v;
    m[e] = zmk(0.5 * (v.x + w.x), 0.5 * (v.y - w.y));
    S.Mreg[e] = m[e];
  });
  mc_each(M, [&](int j, int l, int e) {
    z_t x = zmk(0.0, 0.0), y = zmk(0.0, 0.0);
    for (int q = 0; q < M; q++) {
      zfma(x, c[q + M * l], m[q + M * j]);
      zfma(y, c[l + M * q], m[q + M * j]);
    }
    S.X[e] = x;
    S.Y[e] = y;
  });
}

// Pair sources conj(phi_l) phi_k w, l <= k, and h phi
__global__ void k_mc_sources(z_t* __restrict__ Sp, z_t* __restrict__ Aphi, const z_t* __restrict__ phi,
                             const double* __restrict__ w, const double* __restrict__ T,
                             const double* __restrict__ V0, const double* __restrict__ x, double E, int nG, int band,
                             int M) {
  const size_t nP = (size_t)nG * (M * (M + 1) / 2);
  const int nd = 2 * band + 1;
  MC_LOOP(e, nP + (size_t)nG * M) {
    if (e < nP) {
      const int g = (int)(e % nG), p = (int)(e / nG);
      int k = 0;
      while (mc_pair(0, k + 1) <= p) k++;
      const int l = p - mc_pair(0, k);
      Sp[e] = zscale(zcmul(phi[g + (size_t)nG * l], phi[g + (size_t)nG * k]), w[g]);
    } else {
      const size_t f = e - nP;
      const int g = (int)(f % nG);
      const z_t* col = phi + (f - g);
      z_t acc = zscale(col[g], fma(E, x[g], V0[g]));
      for (int d = max(0, band - g); d < min(nd, nG - g + band); d++) {
        const double c = T[(size_t)d * nG + g];
        const z_t v = col[g - band + d];
        acc.x = fma(c, v.x, acc.x);
        acc.y = fma(c, v.y, acc.y);
      }
      Aphi[f] = acc;
    }
  }
}

// out = V in over N columns (V the nG x nG interaction matrix), and beside it,
// in the first nExtra blocks, the density's algebra (density) or sums over the grid.
// 2 nG^2 N FP64 FMA at two a cycle and SM bound it: 30 us at 501 points x 36 columns.
// A block takes 16 rows x 4 columns, so that those 288 blocks load the SMs evenly
// (a 32 x 8 tile leaves a third of them idle), and splits the row over four
// threads.  A warp per output without tiles: 101 us for all 64 columns, 42 now.
constexpr int PT_R = 16, PT_C = 4, PT_K = 64;
__global__ void __launch_bounds__(MC_T) k_mc_potentials(z_t* __restrict__ out, const z_t* __restrict__ in,
                                                        const double* __restrict__ V, int nG, int N, int nExtra,
                                                        int density, const McStage S, const z_t* __restrict__ C,
                                                        double eps, const McSums sums, int M) {
  if ((int)blockIdx.x < nExtra) {
    if (density) mc_density(S, C, M, eps);
    else mc_sums(sums, blockIdx.x, nG, M);
    return;
  }
  __shared__ double sV[PT_R][PT_K + 1];
  __shared__ z_t sS[PT_C][PT_K], red[3][PT_R * PT_C];
  const int tid = threadIdx.x, nR = (nG + PT_R - 1) / PT_R;
  const int b = blockIdx.x - nExtra, r0 = b % nR * PT_R, c0 = b / nR * PT_C;
  const int x = tid % PT_R, col = tid / PT_R % PT_C, ks = tid / (PT_R * PT_C);
  double fv[PT_R * PT_K / MC_T];
  z_t fs;
  auto fetch = [&](int y0) {
    for (int i = 0; i < PT_R * PT_K / MC_T; i++) {
      const int e = tid + i * MC_T, r = r0 + e / PT_K, y = y0 + e % PT_K;
      fv[i] = r < nG && y < nG ? V[(size_t)r * nG + y] : 0.0;
    }
    const int c = c0 + tid / PT_K, y = y0 + tid % PT_K;
    fs = c < N && y < nG ? in[(size_t)c * nG + y] : zmk(0.0, 0.0);
  };
  z_t s = zmk(0.0, 0.0);
  fetch(0);
  for (int y0 = 0; y0 < nG; y0 += PT_K) {
    __syncthreads();
    for (int i = 0; i < PT_R * PT_K / MC_T; i++) sV[(tid + i * MC_T) / PT_K][(tid + i * MC_T) % PT_K] = fv[i];
    sS[tid / PT_K][tid % PT_K] = fs;
    __syncthreads();
    if (y0 + PT_K < nG) fetch(y0 + PT_K);
#pragma unroll 4
    for (int y = ks; y < PT_K; y += 4) {
      const double v = sV[x][y];
      const z_t q = sS[col][y];
      s.x = fma(v, q.x, s.x);
      s.y = fma(v, q.y, s.y);
    }
  }
  if (ks > 0) red[ks - 1][tid % (PT_R * PT_C)] = s;
  __syncthreads();
  if (ks == 0 && r0 + x < nG && c0 + col < N) {
    for (int i = 0; i < 3; i++) s = zadd(s, red[i][tid]);
    out[(size_t)(c0 + col) * nG + r0 + x] = s;
  }
}

// W_lk(x) from the potentials of the pairs l <= k
__device__ __forceinline__ z_t mc_w(const z_t* W, int nG, int x, int l, int k) {
  return l <= k ? W[(size_t)nG * mc_pair(l, k) + x] : zconj(W[(size_t)nG * mc_pair(k, l) + x]);
}

// f(point in the tile, orbital, x) for the points of a tile, MC_TX at a time
template <class F>
__device__ __forceinline__ void mc_tile(int nG, int M, F f) {
  for (int e = threadIdx.x; e < MC_TX * M; e += blockDim.x) {
    const int t = e % MC_TX, x = blockIdx.x * MC_TX + t;
    if (x < nG) f(t, e / MC_TX, x);
  }
  __syncthreads();
}

// u and u' of a tile
__device__ __forceinline__ void mc_u(z_t (*u)[MC_TX], z_t (*up)[MC_TX], const z_t (*ph)[MC_TX], const z_t* c, int nG,
                                     int M) {
  mc_tile(nG, M, [&](int t, int k, int) {
    z_t a = zmk(0.0, 0.0), b = zmk(0.0, 0.0);
    for (int i = 0; i < M; i++) {
      zcfma(a, c[i + M * k], ph[i][t]);
      zcfma(b, c[k + M * i], ph[i][t]);
    }
    u[k][t] = a;
    up[k][t] = b;
  });
}

// z, z' and dphi0
__global__ void __launch_bounds__(MC_TT) k_mc_meanfield(const McStage S, const z_t* __restrict__ s, int nG, int M) {
  __shared__ McMat c, X, Y;
  __shared__ z_t ph[MC_MAXM][MC_TX], u[MC_MAXM][MC_TX], up[MC_MAXM][MC_TX], z[MC_MAXM][MC_TX], zp[MC_MAXM][MC_TX];
  const z_t* phi = s + M * M;
  mc_load(c, s, M);
  mc_load(X, S.X, M);
  mc_load(Y, S.Y, M);
  mc_tile(nG, M, [&](int t, int i, int x) { ph[i][t] = phi[x + (size_t)nG * i]; });
  mc_u(u, up, ph, c, nG, M);
  mc_tile(nG, M, [&](int t, int l, int x) {
    z_t a = zmk(0.0, 0.0), b = zmk(0.0, 0.0);
    for (int k = 0; k < M; k++) {
      const z_t W = mc_w(S.W, nG, x, l, k);
      zfma(a, W, u[k][t]);
      zfma(b, W, up[k][t]);
    }
    z[l][t] = a;
    zp[l][t] = b;
    S.z[x + (size_t)nG * l] = a;
    S.zp[x + (size_t)nG * l] = b;
  });
  mc_tile(nG, M, [&](int t, int j, int x) {
    z_t a = zmk(0.0, 0.0);
    for (int l = 0; l < M; l++) {
      zfma(a, X[j + M * l], z[l][t]);
      zfma(a, Y[j + M * l], zp[l][t]);
    }
    S.dphi0[x + (size_t)nG * j] = a;
  });
}

// The derivative k = -i [dC0 - sc C ; dphi0 - phi Gp] of a stage and what follows it in
// RK4: next = s + cs k, or after the last stage the step's result
// s + (dt/6 k1 + dt/3 k2 + dt/3 k3 + dt/6 k4) (the reference's order).  Block 0 takes the
// coefficients.
struct McOut {
  const z_t *base, *k1, *k2, *k3;  // k1..k3: last stage only
  z_t *k, *next;
  double cs, dt;
};
__global__ void __launch_bounds__(MC_T) k_mc_out(const McOut O, const McStage S, const z_t* __restrict__ s, int nG,
                                                 int M) {
  const int Q = M * M;
  auto emit = [&](size_t e, z_t v) {
    const z_t k = zmi(v);
    O.k[e] = k;
    if (!O.next) return;
    if (!O.k1) {
      O.next[e] = zadd(zscale(k, O.cs), O.base[e]);
    } else {
      z_t t = zadd(zscale(O.k2[e], O.dt / 3.0), zscale(O.k1[e], O.dt / 6.0));
      t = zadd(zscale(O.k3[e], O.dt / 3.0), t);
      t = zadd(zscale(k, O.dt / 6.0), t);
      O.next[e] = zadd(t, O.base[e]);
    }
  };
  if (blockIdx.x == 0) {
    __shared__ McMat c, h, d;
    __shared__ z_t part[MC_T / 32];
    mc_load(c, s, M);
    mc_load(h, S.h1, M);
    __syncthreads();
    z_t p = zmk(0.0, 0.0);
    mc_each(M, [&](int i, int j, int e) {
      z_t v = zconj(S.G[e]);
      for (int a = 0; a < M; a++) {
        zfma(v, h[a + M * i], c[a + M * j]);
        zfma(v, c[i + M * a], h[a + M * j]);
      }
      d[e] = v;
      S.dC0[e] = v;
      zcfma(p, c[e], v);
    });
    for (int k = 16; k > 0; k >>= 1) {
      p.x += __shfl_xor_sync(0xffffffffu, p.x, k);
      p.y += __shfl_xor_sync(0xffffffffu, p.y, k);
    }
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = p;
    __syncthreads();
    z_t sc = part[0];
    for (int i = 1; i < MC_T / 32; i++) sc = zadd(sc, part[i]);
    if (threadIdx.x == 0) *S.sc = sc;
    mc_each(M, [&](int, int, int e) { emit(e, zsub(d[e], zmul(sc, c[e]))); });
    return;
  }
  const z_t* phi = s + Q;
  for (size_t e = (blockIdx.x - 1) * (size_t)MC_T + threadIdx.x; e < (size_t)nG * M;
       e += (size_t)(gridDim.x - 1) * MC_T) {
    const int x = (int)(e % nG), j = (int)(e / nG);
    z_t v = zmk(0.0, 0.0);
    for (int i = 0; i < M; i++) zfma(v, phi[x + (size_t)nG * i], S.Gp[i + M * j]);
    emit(Q + e, zsub(S.dphi0[e], v));
  }
}

// ---- reverse of a stage: obar (co-state of k) -> co-state of the stage's state
struct McBack {
  z_t *B, *Hs, *Cb;                           // M x M: co-state of dC0, h1bar + h1bar^H, co-state of C so far
  z_t *G1;                                    // phi^H obar (without the factor i of u = i obar)
  z_t *D, *ub, *ubp, *phibar, *Wh;            // co-states of dphi0, u, u', phi so far, the Hermitian pair co-states
  z_t *Xs, *Ys, *C1, *C2;                     // conjugates of the co-states of X, Y and of C through u and u'
};

// Sums phi^H obar; in block 0 the reverse of the coefficients' projector and of
// dC0 = h1^T C + C h1 + .., and the field's part Re sum conj(h1bar) X1
__global__ void __launch_bounds__(MC_T) k_mc_back_coeffs(const McBack K, const McStage S, const z_t* __restrict__ s,
                                                         const z_t* __restrict__ obar, double* __restrict__ grad,
                                                         const McSums sums, int nG, int M) {
  if (blockIdx.x > 0) {
    mc_sums(sums, blockIdx.x - 1, nG, M);
    return;
  }
  __shared__ McMat c, h, B, hb;
  __shared__ z_t part[MC_T / 32];
  const int tid = threadIdx.x;
  auto total = [&](z_t p) {
    for (int k = 16; k > 0; k >>= 1) {
      p.x += __shfl_xor_sync(0xffffffffu, p.x, k);
      p.y += __shfl_xor_sync(0xffffffffu, p.y, k);
    }
    __syncthreads();
    if ((tid & 31) == 0) part[tid >> 5] = p;
    __syncthreads();
    z_t t = part[0];
    for (int i = 1; i < MC_T / 32; i++) t = zadd(t, part[i]);
    return t;
  };
  mc_load(c, s, M);
  mc_load(h, S.h1, M);
  z_t p = zmk(0.0, 0.0);
  mc_each(M, [&](int, int, int e) { zcfma(p, s[e], zpi(obar[e])); });
  const z_t t = total(p), sc = *S.sc;
  mc_each(M, [&](int, int, int e) {
    B[e] = zsub(zpi(obar[e]), zmul(c[e], t));
    K.B[e] = B[e];
  });
  p = zmk(0.0, 0.0);
  mc_each(M, [&](int i, int j, int e) {
    z_t v = zsub(zmul(zscale(zconj(sc), -1.0), zpi(obar[e])), zmul(zconj(t), S.dC0[e]));
    z_t g = zmk(0.0, 0.0);
    for (int a = 0; a < M; a++) {
      zcfma(v, h[i + M * a], B[a + M * j]);           // conj(h1) B
      zcfma(v, h[j + M * a], B[i + M * a]);           // B h1^H
      zcfma(g, c[i + M * a], B[j + M * a]);           // conj(C) B^T
      zcfma(g, c[a + M * i], B[a + M * j]);           // C^H B
    }
    K.Cb[e] = v;
    hb[e] = g;
    zcfma(p, g, S.X1[e]);
  });
  mc_each(M, [&](int i, int j, int e) { K.Hs[e] = zadd(hb[e], zconj(hb[j + M * i])); });
  const z_t g = total(p);
  if (tid == 0 && grad) *grad += g.x;
}

// The pointwise part: D, the co-states of z, z', u and u', phi's so far and the
// Hermitian part of the pair potentials' (both halves of a pair act through it)
__global__ void __launch_bounds__(MC_TT) k_mc_back_points(const McBack K, const McStage S, const z_t* __restrict__ s,
                                                          const z_t* __restrict__ obar, const double* __restrict__ w,
                                                          int nG, int M) {
  __shared__ McMat c, g1, mA, mB;
  __shared__ z_t ph[MC_MAXM][MC_TX], u[MC_MAXM][MC_TX], up[MC_MAXM][MC_TX], D[MC_MAXM][MC_TX], pb[MC_MAXM][MC_TX],
      zb[MC_MAXM][MC_TX], zbp[MC_MAXM][MC_TX], U[MC_MAXM][MC_TX];
  const z_t *phi = s + M * M, *ob = obar + M * M;
  for (int e = threadIdx.x; e < M * M; e += blockDim.x) {
    c[e] = s[e];
    g1[e] = zpi(K.G1[e]);
    mA[e] = S.Gp[e];
    mB[e] = K.Hs[e];
  }
  mc_tile(nG, M, [&](int t, int i, int x) {
    ph[i][t] = phi[x + (size_t)nG * i];
    U[i][t] = zpi(ob[x + (size_t)nG * i]);
  });
  mc_u(u, up, ph, c, nG, M);
  mc_tile(nG, M, [&](int t, int a, int x) {
    z_t d = zmk(0.0, 0.0), p = zmk(0.0, 0.0), q = zmk(0.0, 0.0);
    for (int i = 0; i < M; i++) {
      zfma(d, ph[i][t], g1[i + M * a]);
      zfma(p, zconj(mA[a + M * i]), U[i][t]);
      zfma(q, zconj(zscale(g1[a + M * i], -1.0)), S.dphi0[x + (size_t)nG * i]);
      zfma(q, mB[i + M * a], S.Aphi[x + (size_t)nG * i]);
    }
    D[a][t] = zsub(U[a][t], zscale(d, w[x]));
    K.D[x + (size_t)nG * a] = D[a][t];
    pb[a][t] = zsub(zscale(q, w[x]), p);
  });
  mc_load(g1, K.B, M);
  mc_load(mA, S.X, M);
  mc_load(mB, S.Y, M);
  __syncthreads();
  mc_tile(nG, M, [&](int t, int l, int x) {
    z_t a = zmk(0.0, 0.0), b = zmk(0.0, 0.0), g = zmk(0.0, 0.0), q = zmk(0.0, 0.0);
    for (int j = 0; j < M; j++) {
      zcfma(a, mA[j + M * l], D[j][t]);
      zcfma(b, mB[j + M * l], D[j][t]);
      zcfma(g, g1[j + M * l], ph[j][t]);
      zfma(q, g1[l + M * j], S.z[x + (size_t)nG * j]);
    }
    zb[l][t] = zadd(a, zscale(g, w[x]));
    zbp[l][t] = b;
    pb[l][t] = zadd(pb[l][t], zscale(q, w[x]));
  });
  mc_tile(nG, M, [&](int t, int k, int x) {
    z_t a = zmk(0.0, 0.0), b = zmk(0.0, 0.0);
    for (int l = 0; l < M; l++) {
      const z_t W = zconj(mc_w(S.W, nG, x, l, k));
      zfma(a, W, zb[l][t]);
      zfma(b, W, zbp[l][t]);
    }
    D[k][t] = a;  // ubar, u'bar in place of D and U
    U[k][t] = b;
    K.ub[x + (size_t)nG * k] = a;
    K.ubp[x + (size_t)nG * k] = b;
    for (int l = 0; l <= k; l++) {
      z_t v = zcmul(u[k][t], zb[l][t]);
      zcfma(v, up[k][t], zbp[l][t]);
      zcfma(v, zb[k][t], u[l][t]);
      zcfma(v, zbp[k][t], up[l][t]);
      K.Wh[x + (size_t)nG * mc_pair(l, k)] = v;
    }
  });
  mc_tile(nG, M, [&](int t, int a, int x) {
    z_t v = pb[a][t];
    for (int k = 0; k < M; k++) {
      zfma(v, c[a + M * k], D[k][t]);
      zfma(v, c[k + M * a], U[k][t]);
    }
    K.phibar[x + (size_t)nG * a] = v;
  });
}

// The pair sources' reverse (Hb = V Wh) and the density's, and what follows in RK4's
// reverse: sbar = sIn + co-state of this stage's state, next = wgt obar0 + cs times it
// (the co-state of the stage before; may be null).  Block 0 takes the coefficients.
struct McBackOut {
  const z_t *sIn, *obar0;
  z_t *sbar, *next;
  double cs, wgt;
};
__global__ void __launch_bounds__(MC_T) k_mc_back_out(const McBackOut O, const McBack K, const McStage S,
                                                      const z_t* __restrict__ s, const z_t* __restrict__ Hb,
                                                      const double* __restrict__ w, int nG, int M) {
  const int Q = M * M;
  auto emit = [&](size_t e, z_t v) {
    const z_t o = O.obar0[e];  // sbar may be obar0's buffer: read first
    O.sbar[e] = zadd(O.sIn[e], v);
    if (O.next) O.next[e] = zadd(zscale(v, O.cs), zscale(o, O.wgt));
  };
  if (blockIdx.x == 0) {
    __shared__ McMat c, m, xb, yb, k, t, cb;
    mc_load(c, s, M);
    mc_load(m, S.Mreg, M);
    mc_load(k, S.Kinv, M);
    mc_each(M, [&](int i, int j, int e) {
      xb[e] = zconj(K.Xs[e]);
      yb[e] = zconj(K.Ys[e]);
      cb[e] = zadd(K.Cb[e], zadd(zconj(K.C1[e]), zconj(K.C2[j + M * i])));
    });
    mc_each(M, [&](int q, int l, int e) {
      z_t v = cb[e], n = zmk(0.0, 0.0);
      for (int j = 0; j < M; j++) {
        zcfma(v, m[q + M * j], xb[j + M * l]);
        zcfma(v, m[l + M * j], yb[j + M * q]);
        zcfma(n, c[q + M * j], xb[l + M * j]);   // Mbar[q, l] = sum_j Xbar[l, j] conj(C[q, j]) + Ybar[l, j] conj(C[j, q])
        zcfma(n, c[j + M * q], yb[l + M * j]);
      }
      cb[e] = v;
      t[e] = n;
    });
    mc_each(M, [&](int i, int j, int e) {
      const z_t a = t[i + M * j], b = t[j + M * i];
      xb[e] = zmk(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
    });
    mc_each(M, [&](int i, int j, int e) {  // K herm(Mbar)
      z_t v = zmk(0.0, 0.0);
      for (int a = 0; a < M; a++) zfma(v, k[i + M * a], xb[a + M * j]);
      yb[e] = v;
    });
    mc_each(M, [&](int i, int j, int e) {
      z_t v = zmk(0.0, 0.0);
      for (int a = 0; a < M; a++) zfma(v, yb[i + M * a], k[a + M * j]);
      t[e] = v;
    });
    mc_each(M, [&](int i, int j, int e) { xb[e] = zscale(zadd(t[e], zconj(t[j + M * i])), -1.0); });
    mc_each(M, [&](int i, int j, int e) {
      z_t v = cb[e];
      for (int a = 0; a < M; a++) {
        zfma(v, xb[a + M * i], c[a + M * j]);
        zfma(v, c[i + M * a], xb[a + M * j]);
      }
      emit(e, v);
    });
    return;
  }
  const z_t* phi = s + Q;
  for (size_t e = (blockIdx.x - 1) * (size_t)MC_T + threadIdx.x; e < (size_t)nG * M;
       e += (size_t)(gridDim.x - 1) * MC_T) {
    const int x = (int)(e % nG), m = (int)(e / nG);
    z_t v = zmk(0.0, 0.0);
    for (int l = 0; l < M; l++) zfma(v, mc_w(Hb, nG, x, l, m), phi[x + (size_t)nG * l]);
    emit(Q + e, zadd(K.phibar[e], zscale(v, w[x])));
  }
}

// y = a x
__global__ void k_mc_scale(z_t* __restrict__ y, const z_t* __restrict__ x, double a, int n) {
  MC_LOOP(e, n) y[e] = zscale(x[e], a);
}

// wx = w x on the grid
__global__ void k_mc_weights(double* __restrict__ wx, const double* __restrict__ w, const double* __restrict__ x,
                             int nG) {
  MC_LOOP(e, nG) wx[e] = w[e] * x[e];
}

// The objective's co-state: [Cbar ; w (ref Sbar)]
__global__ void k_mc_final_costate(z_t* __restrict__ dst, const z_t* __restrict__ Cbar, const z_t* __restrict__ Sbar,
                                   const z_t* __restrict__ ref, const double* __restrict__ w, int nG, int M) {
  const int Q = M * M;
  MC_LOOP(e, (size_t)Q + (size_t)nG * M) {
    if ((int)e < Q) {
      dst[e] = Cbar[e];
      continue;
    }
    const int x = (int)((e - Q) % nG), j = (int)((e - Q) / nG);
    z_t s = zmk(0.0, 0.0);
    for (int k = 0; k < M; k++) zfma(s, ref[Q + x + (size_t)nG * k], Sbar[k + M * j]);
    dst[e] = zscale(s, w[x]);
  }
}

// ---- objective: O = sum conj(Cr) (S C S^T), S = phi_ref^H W phi
__global__ void k_mc_overlap(z_t* __restrict__ O, const z_t* __restrict__ Cr, const z_t* __restrict__ S,
                             const z_t* __restrict__ C, int M) {
  __shared__ double sx[MC_RED], sy[MC_RED];
  z_t s = zmk(0.0, 0.0);
  for (int e = threadIdx.x; e < M * M; e += MC_RED) {
    const int a = e % M, b = e / M;
    z_t t = zmk(0.0, 0.0);
    for (int d = 0; d < M; d++)
      for (int c = 0; c < M; c++) zfma(t, zmul(S[a + M * c], C[c + M * d]), S[b + M * d]);
    s = zadd(s, zcmul(Cr[e], t));
  }
  sx[threadIdx.x] = s.x;
  sy[threadIdx.x] = s.y;
  __syncthreads();
  for (int o = MC_RED / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      sx[threadIdx.x] += sx[threadIdx.x + o];
      sy[threadIdx.x] += sy[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *O = zmk(sx[0], sy[0]);
}
// Cbar = Ob S^H Cr conj(S);  Sbar = Ob conj(P S C^T + P^T S C), P = conj(Cr), Ob = -2 O
__global__ void k_mc_overlap_vjp(z_t* __restrict__ Cbar, z_t* __restrict__ Sbar, const z_t* __restrict__ Cr,
                                 const z_t* __restrict__ S, const z_t* __restrict__ C, const z_t* __restrict__ O, int M) {
  const z_t Ob = zscale(*O, -2.0);
  for (int e = threadIdx.x; e < M * M; e += blockDim.x) {
    const int p = e % M, q = e / M;
    z_t cb = zmk(0.0, 0.0), g = zmk(0.0, 0.0);
    for (int b = 0; b < M; b++)
      for (int a = 0; a < M; a++) {
        // (S^H Cr conj(S))[p, q] = sum_ab conj(S[a, p]) Cr[a, b] conj(S[b, q])
        zfma(cb, zconj(S[a + M * p]), zmul(Cr[a + M * b], zconj(S[b + M * q])));
        // (P S C^T)[p, q] = sum_ab conj(Cr[p, a]) S[a, b] C[q, b];  (P^T S C)[p, q] = sum_ab conj(Cr[a, p]) S[a, b] C[b, q]
        zfma(g, zconj(Cr[p + M * a]), zmul(S[a + M * b], C[q + M * b]));
        zfma(g, zconj(Cr[a + M * p]), zmul(S[a + M * b], C[b + M * q]));
      }
    Cbar[e] = zmul(Ob, cb);
    Sbar[e] = zmul(Ob, zconj(g));
  }
}
__global__ void k_mc_objective(double* __restrict__ J, const z_t* __restrict__ O) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *J = 1.0 - (O->x * O->x + O->y * O->y);
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct McAdjoint {
  int nG = 0, M = 0, Q = 0, nS = 0, nP = 0, band = 0, K = 0, nT = 0, chk = 0;
  int segAt = -1;  // the segment whose states seg holds
  double dt = 0.0, eps = 1e-10;
  std::vector<double> field;
  double *wx = nullptr, *grad = nullptr, *J = nullptr;
  // state vectors
  z_t *ref = nullptr, *cur = nullptr, *chkStates = nullptr, *seg = nullptr, *co = nullptr;
  z_t *sA = nullptr, *sB = nullptr, *tmpS = nullptr, *lam = nullptr, *lamB = nullptr;
  z_t *stage[4] = {}, *kv[4] = {};  // stage[0] is the step's own vector
  SilKeep lzA{}, lzC{};             // the two half steps
  McStage st[4] = {};
  z_t* Sp = nullptr;  // pair sources; in the reverse the pair co-states' potentials
  McBack bk{};
  z_t *Sov = nullptr, *Sbar = nullptr, *Ov = nullptr;
  std::vector<void*> allocs;
  bool ready = false;

  template <class T>
  T* alloc(size_t n) {
    void* p = nullptr;
    CODY_CUDA(cudaMalloc(&p, sizeof(T) * std::max<size_t>(n, 1)));
    CODY_CUDA(cudaMemset(p, 0, sizeof(T) * std::max<size_t>(n, 1)));
    allocs.push_back(p);
    return (T*)p;
  }
  ~McAdjoint() {
    for (void* p : allocs) cudaFree(p);
  }
};

namespace {

double field_at(const McAdjoint& A, double t, int* idx) {
  const int n = (int)std::floor(t / A.dt + 1e-9);
  *idx = n;
  return (n >= 0 && n < A.nT) ? A.field[n] : 0.0;
}
double* grad_at(const McAdjoint& A, int n) { return n >= 0 && n < A.nT ? A.grad + n : nullptr; }

int tiles(const McAdjoint& A) { return (A.nG + MC_TX - 1) / MC_TX; }

// out = V in over the pairs, with the density's algebra of state s beside it (S) or sums
void potentials(cgpu_ctx* c, McAdjoint& A, z_t* out, const z_t* in, const McStage* S, const z_t* s,
                const McSums* sums) {
  const int nExtra = S ? 1 : mc_sum_blocks(sums->n, A.M, MC_T);
  const int nB = (A.nG + PT_R - 1) / PT_R * ((A.nP + PT_C - 1) / PT_C);
  k_mc_potentials<<<nExtra + nB, MC_T, 0, c->stream>>>(out, in, c->Vint_d, A.nG, A.nP, nExtra, S != nullptr,
                                                       S ? *S : McStage{}, s, A.eps, sums ? *sums : McSums{}, A.M);
  CODY_LAUNCHED(c);
}

// NonLin derivative of state s with field E, stage i of RK4 (see k_mc_out)
void nonlin_forward(cgpu_ctx* c, McAdjoint& A, const z_t* s, double E, int i, const McOut& O) {
  const int nG = A.nG, M = A.M;
  const McStage& S = A.st[i];
  const z_t* phi = s + A.Q;
  k_mc_sources<<<nblk((size_t)nG * (A.nP + M)), MC_T, 0, c->stream>>>(A.Sp, S.Aphi, phi, c->w_d, c->T_d, c->V0_d,
                                                                      c->x_d, E, nG, A.band, M);
  CODY_LAUNCHED(c);
  potentials(c, A, S.W, A.Sp, &S, s, nullptr);
  k_mc_meanfield<<<tiles(A), MC_TT, 0, c->stream>>>(S, s, nG, M);
  CODY_LAUNCHED(c);
  const McSums sums = {{{phi, S.Aphi, c->w_d, S.h1},
                        {phi, S.z, c->w_d, S.G},
                        {phi, S.dphi0, c->w_d, S.Gp},
                        {phi, phi, A.wx, S.X1}},
                       4};
  k_mc_sums<<<mc_sum_blocks(4, M, MC_ST), MC_ST, 0, c->stream>>>(sums, nG, M);
  CODY_LAUNCHED(c);
  k_mc_out<<<1 + nblk((size_t)nG * M), MC_T, 0, c->stream>>>(O, S, s, nG, M);
  CODY_LAUNCHED(c);
}

// The reverse of stage i at its state s, from the co-state obar of its derivative
void nonlin_vjp(cgpu_ctx* c, McAdjoint& A, const z_t* s, const z_t* obar, int i, int nIdx, const McBackOut& O) {
  const int nG = A.nG, M = A.M;
  const McStage& S = A.st[i];
  const McBack& K = A.bk;
  const z_t* phi = s + A.Q;
  const McSums g1 = {{{phi, obar + A.Q, nullptr, K.G1}}, 1};
  k_mc_back_coeffs<<<1 + mc_sum_blocks(1, M, MC_T), MC_T, 0, c->stream>>>(K, S, s, obar, grad_at(A, nIdx), g1, nG, M);
  CODY_LAUNCHED(c);
  k_mc_back_points<<<tiles(A), MC_TT, 0, c->stream>>>(K, S, s, obar, c->w_d, nG, M);
  CODY_LAUNCHED(c);
  const McSums sums = {{{K.D, S.z, nullptr, K.Xs},
                        {K.D, S.zp, nullptr, K.Ys},
                        {phi, K.ub, nullptr, K.C1},
                        {phi, K.ubp, nullptr, K.C2}},
                       4};
  potentials(c, A, A.Sp, K.Wh, nullptr, s, &sums);
  k_mc_back_out<<<1 + nblk((size_t)nG * M), MC_T, 0, c->stream>>>(O, K, S, s, A.Sp, c->w_d, nG, M);
  CODY_LAUNCHED(c);
}

// RK4 of the NonLin derivative from s (t0, dt) into out; the stages are kept
void rk4_forward(cgpu_ctx* c, McAdjoint& A, z_t* s, z_t* out, double t0) {
  const double dt = A.dt;
  const double ts[4] = {t0, t0 + 0.5 * dt, t0 + 0.5 * dt, t0 + dt}, cs[4] = {0.5 * dt, 0.5 * dt, dt, 0.0};
  A.stage[0] = s;
  for (int i = 0; i < 4; i++) {
    int n;
    McOut O = {s, nullptr, nullptr, nullptr, A.kv[i], i < 3 ? A.stage[i + 1] : out, cs[i], dt};
    if (i == 3) {
      O.k1 = A.kv[0];
      O.k2 = A.kv[1];
      O.k3 = A.kv[2];
    }
    nonlin_forward(c, A, A.stage[i], field_at(A, ts[i], &n), i, O);
  }
}

// sbar = (d RK4 / d s)^H obar at the stages of the last rk4_forward; grad += field parts
void rk4_vjp(cgpu_ctx* c, McAdjoint& A, const z_t* obar, z_t* sbar, double t0) {
  const double dt = A.dt;
  const double ts[4] = {t0, t0 + 0.5 * dt, t0 + 0.5 * dt, t0 + dt};
  const double wgt[4] = {dt / 6.0, dt / 3.0, dt / 3.0, dt / 6.0}, cs[4] = {0.5 * dt, 0.5 * dt, dt, 0.0};
  k_mc_scale<<<nblk(A.nS), MC_T, 0, c->stream>>>(A.kv[3], obar, wgt[3], A.nS);
  CODY_LAUNCHED(c);
  for (int i = 3; i >= 0; i--) {
    int n;
    field_at(A, ts[i], &n);
    McBackOut O = {i == 3 ? obar : sbar, obar, sbar, nullptr, 0.0, 0.0};
    if (i > 0) {
      O.next = A.kv[i - 1];
      O.cs = cs[i - 1];
      O.wgt = wgt[i - 1];
    }
    nonlin_vjp(c, A, A.stage[i], A.kv[i], i, n, O);
  }
}

// One Strang step n: s -> out; the Krylov bases and RK4 stages are kept
void step_forward(cgpu_ctx* c, McAdjoint& A, const z_t* s, z_t* out, int n) {
  const double dt = A.dt, t0 = n * dt;
  int na, nc;
  launch_sil_keep(c, s, A.sA, field_at(A, t0 + 0.25 * dt, &na), 0.5 * dt, A.lzA);
  rk4_forward(c, A, A.sA, A.sB, t0);
  launch_sil_keep(c, A.sB, out, field_at(A, t0 + 0.75 * dt, &nc), 0.5 * dt, A.lzC);
}

// lam (co-state of the step's output) -> lam (co-state of its input s)
void step_vjp(cgpu_ctx* c, McAdjoint& A, const z_t* s, z_t* lam, int n) {
  const double dt = A.dt, t0 = n * dt;
  int na, nc;
  const double Ea = field_at(A, t0 + 0.25 * dt, &na), Ec = field_at(A, t0 + 0.75 * dt, &nc);
  step_forward(c, A, s, A.tmpS, n);  // the step's intermediates
  launch_sil_vjp(c, lam, A.lamB, Ec, 0.5 * dt, A.lzC, grad_at(A, nc));
  rk4_vjp(c, A, A.lamB, A.lam, t0);
  launch_sil_vjp(c, A.lam, lam, Ea, 0.5 * dt, A.lzA, grad_at(A, na));
}

}  // namespace

// ---------------------------------------------------------------------------
// Entry points (called from ctx.cu's C ABI)
// ---------------------------------------------------------------------------
void mc_adjoint_free(cgpu_ctx* c) {
  delete c->mcAdj;
  c->mcAdj = nullptr;
}

void mc_adjoint_forward(cgpu_ctx* c, const z_t* state0_h, const z_t* ref_h, const double* field_h, int nT, double dt,
                        int K, int checkpoint, double* J, double* overlap, z_t* final_h) {
  if (c->nb != 1) throw std::string("mc_adjoint: a single-system context");
  if (c->method != CGPU_METHOD_MCTDHX) throw std::string("mc_adjoint: an MCTDHX context");
  if (c->precision != CGPU_PREC_FP64) throw std::string("mc_adjoint: the FP64 form");
  const SysHost& s = c->sys[0];
  if (!c->restricted || c->nBt != 2 || s.nBodies[0] != 1 || s.nBodies[1] != 1)
    throw std::string("mc_adjoint: restricted systems of two body types with one particle each");
  if (s.nOS > MC_MAXM) throw std::string("mc_adjoint: at most 16 spatial orbitals");
  if (K < 1 || K > MC_MAXK) throw std::string("mc_adjoint: Krylov order in 1..32");
  if (nT < 1 || !(dt > 0.0)) throw std::string("mc_adjoint: need n_steps >= 1 and dt > 0");
  if (!c->hasInteraction) throw std::string("mc_adjoint: needs the interaction");
  if (checkpoint <= 0) checkpoint = 64;
  const int M = s.nOS, nG = s.nG, Q = M * M, nS = Q + nG * M;
  if (s.nC != Q) throw std::string("mc_adjoint: configuration count");
  McAdjoint* A = c->mcAdj;
  const int nChk = (nT + checkpoint - 1) / checkpoint;
  if (!A || A->K != K || A->nT != nT || A->chk != checkpoint) {
    delete A;
    A = new McAdjoint();
    c->mcAdj = A;
    A->nG = nG;
    A->M = M;
    A->Q = Q;
    A->nS = nS;
    A->band = s.band;
    A->K = K;
    A->nT = nT;
    A->chk = checkpoint;
    A->eps = s.regEps;
    A->nP = M * (M + 1) / 2;
    A->wx = A->alloc<double>(nG);
    A->grad = A->alloc<double>(nT);
    A->J = A->alloc<double>(4);
    auto state = [&]() { return A->alloc<z_t>(nS); };
    A->ref = state();
    A->cur = state();
    A->co = state();
    A->chkStates = A->alloc<z_t>((size_t)nS * nChk);
    A->seg = A->alloc<z_t>((size_t)nS * (checkpoint + 1));
    A->sA = state();
    A->sB = state();
    A->tmpS = state();
    A->lam = state();
    A->lamB = state();
    z_t* spill = sil_spill(c) ? A->alloc<z_t>(sil_spill(c)) : nullptr;
    for (SilKeep* k : {&A->lzA, &A->lzC}) {
      k->K = K;
      k->V = A->alloc<z_t>((size_t)nS * K);
      k->last = state();
      k->phi = A->alloc<z_t>(MC_MAXK);
      k->parts = A->alloc<z_t>((size_t)MC_MAXK * SIL_KEEP_PARTS);
      k->spill = spill;
      k->alpha = A->alloc<double>(MC_MAXK);
      k->beta = A->alloc<double>(MC_MAXK);
      k->norm = A->alloc<double>(1);
    }
    const size_t GM = (size_t)nG * M, GP = (size_t)nG * A->nP;
    for (int i = 0; i < 4; i++) {
      if (i > 0) A->stage[i] = state();
      A->kv[i] = state();
      McStage& S = A->st[i];
      for (z_t** p : {&S.Aphi, &S.z, &S.zp, &S.dphi0}) *p = A->alloc<z_t>(GM);
      S.W = A->alloc<z_t>(GP);
      for (z_t** p : {&S.h1, &S.G, &S.Gp, &S.X1, &S.X, &S.Y, &S.Kinv, &S.Mreg, &S.dC0}) *p = A->alloc<z_t>(Q);
      S.sc = A->alloc<z_t>(1);
    }
    A->Sp = A->alloc<z_t>(GP);
    McBack& B = A->bk;
    for (z_t** p : {&B.B, &B.Hs, &B.Cb, &B.G1, &B.Xs, &B.Ys, &B.C1, &B.C2}) *p = A->alloc<z_t>(Q);
    for (z_t** p : {&B.D, &B.ub, &B.ubp, &B.phibar}) *p = A->alloc<z_t>(GM);
    B.Wh = A->alloc<z_t>(GP);
    A->Sov = A->alloc<z_t>(Q);
    A->Sbar = A->alloc<z_t>(Q);
    A->Ov = A->alloc<z_t>(2);
    k_mc_weights<<<nblk(nG), MC_T, 0, c->stream>>>(A->wx, c->w_d, c->x_d, nG);
    CODY_LAUNCHED(c);
  }
  A->dt = dt;
  A->field.assign(field_h, field_h + nT);
  CODY_CUDA(cudaMemcpyAsync(A->cur, state0_h, sizeof(z_t) * nS, cudaMemcpyHostToDevice, c->stream));
  CODY_CUDA(cudaMemcpyAsync(A->ref, ref_h ? ref_h : state0_h, sizeof(z_t) * nS, cudaMemcpyHostToDevice, c->stream));
  A->ready = false;
  for (int n = 0; n < nT; n++) {
    z_t* s = A->seg + (size_t)nS * (n % checkpoint);
    if (n % checkpoint == 0) {
      const z_t* from = n == 0 ? A->cur : A->seg + (size_t)nS * checkpoint;
      for (z_t* to : {s, A->chkStates + (size_t)nS * (n / checkpoint)})
        CODY_CUDA(cudaMemcpyAsync(to, from, sizeof(z_t) * nS, cudaMemcpyDeviceToDevice, c->stream));
    }
    step_forward(c, *A, s, n + 1 < nT ? s + nS : A->cur, n);
  }
  A->segAt = nChk - 1;
  // objective
  const McSums sov = {{{A->ref + Q, A->cur + Q, c->w_d, A->Sov}}, 1};
  k_mc_sums<<<mc_sum_blocks(1, M, MC_ST), MC_ST, 0, c->stream>>>(sov, nG, M);
  CODY_LAUNCHED(c);
  k_mc_overlap<<<1, MC_RED, 0, c->stream>>>(A->Ov, A->ref, A->Sov, A->cur, M);
  CODY_LAUNCHED(c);
  k_mc_objective<<<1, 32, 0, c->stream>>>(A->J, A->Ov);
  CODY_LAUNCHED(c);
  double jo[1];
  z_t ov;
  CODY_CUDA(cudaMemcpyAsync(jo, A->J, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  CODY_CUDA(cudaMemcpyAsync(&ov, A->Ov, sizeof(z_t), cudaMemcpyDeviceToHost, c->stream));
  if (final_h) CODY_CUDA(cudaMemcpyAsync(final_h, A->cur, sizeof(z_t) * nS, cudaMemcpyDeviceToHost, c->stream));
  ctx_sync(c);
  if (J) *J = jo[0];
  if (overlap) {
    overlap[0] = ov.x;
    overlap[1] = ov.y;
  }
  A->ready = true;
}

void mc_adjoint_backward(cgpu_ctx* c, double* grad_h) {
  McAdjoint* A = c->mcAdj;
  if (!A || !A->ready) throw std::string("mc_adjoint_backward: call cgpu_mc_adjoint_forward first");
  const int nS = A->nS, M = A->M, nG = A->nG, nT = A->nT, chk = A->chk;
  CODY_CUDA(cudaMemsetAsync(A->grad, 0, sizeof(double) * nT, c->stream));
  // co-state of the final state: d J / d Psi_N
  k_mc_overlap_vjp<<<1, 256, 0, c->stream>>>(A->bk.Cb, A->Sbar, A->ref, A->Sov, A->cur, A->Ov, M);
  CODY_LAUNCHED(c);
  k_mc_final_costate<<<nblk(nS), MC_T, 0, c->stream>>>(A->co, A->bk.Cb, A->Sbar, A->ref, c->w_d, nG, M);
  CODY_LAUNCHED(c);
  const int nChk = (nT + chk - 1) / chk;
  for (int sgm = nChk - 1; sgm >= 0; sgm--) {
    const int n0 = sgm * chk, n1 = std::min(nT, n0 + chk);
    if (A->segAt != sgm) {
      CODY_CUDA(cudaMemcpyAsync(A->seg, A->chkStates + (size_t)nS * sgm, sizeof(z_t) * nS, cudaMemcpyDeviceToDevice,
                                c->stream));
      for (int n = n0; n < n1 - 1; n++)
        step_forward(c, *A, A->seg + (size_t)nS * (n - n0), A->seg + (size_t)nS * (n - n0 + 1), n);
      A->segAt = sgm;
    }
    for (int n = n1 - 1; n >= n0; n--) step_vjp(c, *A, A->seg + (size_t)nS * (n - n0), A->co, n);
  }
  CODY_CUDA(cudaMemcpyAsync(grad_h, A->grad, sizeof(double) * nT, cudaMemcpyDeviceToHost, c->stream));
  ctx_sync(c);
}
