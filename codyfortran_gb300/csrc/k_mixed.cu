// k_mixed.cu -- mixed-precision form of ApplyCorrelationOp
// (src/Method/Mb/OrbBased/S_Method_Mb_OrbBased.f90:647-872).
//
// The three contractions run on the tcgen05 GEMM (k_tc.cu) with split-bf16
// operands and FP32 accumulation; split-K partials, the correlation
// epilogue, the RDMs, rho^-1 and everything else stay FP64.
//
//   GEMM1  W[g][2p+s]   = sum_g' V[g][g'] S_s(p, g')            (M=nG, N=2P, K=nG)
//   GEMM2  Z[g][2q+s]   = sum_k  W[g][k] R''[2q+s][k]           (M=nG, N=2Q, K=2P)
//   GEMM3  G[2p+s][2p'+t] = sum_g S_s(p,g) W_t(p',g)            (M=N=2P, K=nG)
// with p, p' unordered orbital pairs (l <= k), s,t in {re, im}, q = (k1, j)
// an ordered pair.  The conjugate symmetry W_(k,l) = conj(W_(l,k)) folds the
// ordered-pair sums into real GEMMs over unordered pairs:
//   sum_(l2,k2) W_(l2k2) R'[(l2,k2), q] = sum_p a_p X_p[q] + b_p Y_p[q],
//   W_p = a_p + i b_p,  X_p = R1 + R2,  Y_p = i (R1 - R2),
//   R1 = R'[(l,k), q], R2 = R'[(k,l), q] (0 when l = k).
//
// The fixed-point forms (FP64, mixed_fx, mixed_fx6) carry every operand row as L
// base-256 digit slices under one power of two per row (k_fx.cu) and return
// FP64 results whose only error is the operand truncation (fx_slices: at least 63
// / 31 / 39 bits of each row's maximum): S and V rows for GEMM1, W rows and R''
// rows for GEMM2, W columns for GEMM3.  FillH2 (energies) runs GEMM1 and GEMM3 with the
// eight or nine slices of the FP64 form in all three, or on the FP64 pipe where that
// form runs there (cgpu_ctx::fx64).  The row exponents of W come from
// the GEMM1 epilogue, or from the reduction of its K splits.  The bf16x3 /
// bf16x6 forms keep their own operands (k_tc.cu) and the FP64 pipe's FillH2.
#include <cuda_bf16.h>

#include <array>
#include <type_traits>

#include <algorithm>

#include "common.cuh"
#include "tc.cuh"


// One fixed-point GEMM: N-tile width, two-CTAs-per-SM configuration, K splits, its tile list.
struct FxGemm {
  int bn = 64, s = 1, nTiles = 0;
  bool compact = false;
  void* tiles = nullptr;
};

struct MixedBufs {
  int terms = 3;            // 3: bf16x3, 6: bf16x6
  int KgMax = 0, KpMax = 0; // segment pitches: the largest padded K of the grid / pair contractions
  int bn1 = 64, bn2 = 64, bn3 = 64;  // bf16x3 / bf16x6
  int s1 = 1, s2 = 1, s3 = 1;        // K splits of the three GEMMs (bf16x3 / bf16x6)
  __nv_bfloat16 *VxB = nullptr, *SxA = nullptr, *WxA = nullptr, *WTxB = nullptr, *RxB = nullptr;
  float *P1 = nullptr, *P2 = nullptr, *P3 = nullptr;
  int* err = nullptr;       // GEMM error flag: page-locked host memory, and its device address
  volatile int* err_h = nullptr;
  double* Zd = nullptr;     // (nG, Q) complex
  CUtensorMap mV, mS, mSasB, mW, mWT, mR;  // TMA maps (A operands box 128 rows, B operands box BN rows)
  // fixed-point forms (L > 0): digit slices of GEMM1 / GEMM3 and of GEMM2 (L2); V
  // carries LV slices of which a GEMM reads the first L
  int L = 0, L2 = 0;
  int L64 = 0, LV = 0;              // slices of the FP64 form (cgpu_ctx::fx64; 0: FP64 pipe), of V and S: the most of both
  FxGemm gW, gZ, gH, gWx, gHx;      // the form's three GEMMs; W and h2 at L64 slices for FillH2
  int sCapW = 1, sCapZ = 1, sCapH = 1;  // K splits the FP64 partial buffers hold (the tuner stays within them)
  FxMaps bS, bWT, bR, bSx, bWTx;    // B operands (x: at L64 slices)
  CUtensorMap mSxasB;               // S rows as the A operand at L64 slices
  // one interaction matrix per root grid (cgpu_ctx::fxShared): slices [root][c->nG][LV KgBig]
  // and row exponents [root][c->nG], outside the per-trajectory arena
  int KgBig = 0;
  __nv_bfloat16* Vsh = nullptr;
  int* eVsh = nullptr;
  CUtensorMap mVsh;
  int *eV = nullptr, *eS = nullptr, *sS = nullptr, *eWr = nullptr, *eWc = nullptr, *eR = nullptr;  // row exponents (sS: see fx_scale_key)
  unsigned *mWr = nullptr, *mWc = nullptr;  // largest biased exponent of |W| per row g / column n
  double *Wd = nullptr, *Zp = nullptr, *Gd = nullptr;  // FP64 results [split][M][N]
};

namespace {

// Segment patterns: A operands [hi,hi,lo] / [hi,hi,mid,hi,mid,lo],
// B operands [hi,lo,hi] / [hi,mid,hi,lo,mid,hi]; part index 0=hi, 1=mid, 2=lo.
__device__ __forceinline__ int seg_part(int terms, int isB, int seg) {
  if (terms == 3) {
    const int a[3] = {0, 0, 2}, b[3] = {0, 2, 0};
    return isB ? b[seg] : a[seg];
  }
  const int a[6] = {0, 0, 1, 0, 1, 2}, b[6] = {0, 1, 0, 2, 1, 0};
  return isB ? b[seg] : a[seg];
}

// x = hi + mid + lo in bf16 (for terms == 3 the low part is bf16(x - hi)).
__device__ __forceinline__ __nv_bfloat16 split_part(double x, int terms, int part) {
  __nv_bfloat16 hi = __double2bfloat16(x);
  if (part == 0) return hi;
  double r1 = x - (double)__bfloat162float(hi);
  __nv_bfloat16 mid = __double2bfloat16(r1);
  if (terms == 3) return mid;  // the "lo" part of the two-term split
  if (part == 1) return mid;
  return __double2bfloat16(r1 - (double)__bfloat162float(mid));
}

// out[row][seg*pitch + k] = part(value(row,k)), zero for k >= K.
__device__ __forceinline__ void write_split(__nv_bfloat16* out, int row, int k, int K, int pitch, int terms, int isB,
                                            double v) {
  size_t base = (size_t)row * terms * pitch;
  for (int seg = 0; seg < terms; seg++) {
    __nv_bfloat16 h = (k < K) ? split_part(v, terms, seg_part(terms, isB, seg)) : __double2bfloat16(0.0);
    out[base + (size_t)seg * pitch + k] = h;
  }
}

// FP64 -> FP32 by truncating the significand (integer operations only: the FP64
// pipes are the scarce resource).  |x| below the FP32 normal range flushes to
// zero; relative error < 2^-23, below the bf16x3 form's ~2^-16.
__device__ __forceinline__ float f64_to_f32(double x) {
  unsigned long long u = (unsigned long long)__double_as_longlong(x);
  unsigned hi = (unsigned)(u >> 32);
  unsigned sign = hi & 0x80000000u;
  int e = (int)((hi >> 20) & 0x7FFu) - 1023 + 127;
  if (e <= 0) return __int_as_float((int)sign);
  if (e >= 255) return __int_as_float((int)(sign | 0x7F800000u));
  unsigned mant = ((hi & 0xFFFFFu) << 3) | (unsigned)((u >> 29) & 7u);
  return __int_as_float((int)(sign | ((unsigned)e << 23) | mant));
}

// bf16x3 split in FP32: hi = bf16(v), lo = bf16(v - hi); A rows [hi,hi,lo], B rows [hi,lo,hi].
__device__ __forceinline__ void write_split3(__nv_bfloat16* out, int row, int k, int K, int pitch, int isB, float v) {
  size_t base = (size_t)row * 3 * pitch + k;
  __nv_bfloat16 hi = __float2bfloat16_rn(0.0f), lo = hi;
  if (k < K) {
    hi = __float2bfloat16_rn(v);
    lo = __float2bfloat16_rn(v - __bfloat162float(hi));
  }
  out[base] = hi;
  out[base + pitch] = isB ? lo : hi;
  out[base + 2 * (size_t)pitch] = isB ? hi : lo;
}

__global__ void k_split_V(__nv_bfloat16* __restrict__ out, const double* __restrict__ V, int pitch, int terms,
                          TRAJ_ARGS) {
  const TrajShape& T = shp[blockIdx.z];
  const int nG = T.nG, Kpad = T.Kg;
  out = bat(out, bs);
  V = bat(V, bs);
  GRID_STRIDE(e, (size_t)nG * Kpad) {
    int row = (int)(e / Kpad), k = (int)(e % Kpad);
    double v = (k < nG) ? V[(size_t)row * nG + k] : 0.0;
    write_split(out, row, k, nG, pitch, terms, 1, v);
  }
}

// S_s(p, g) = (re, im)[conj(phi_l) phi_k w] for pair p = (l, k), A pattern.
__global__ void k_split_S(__nv_bfloat16* __restrict__ outA, const z_t* __restrict__ orbs, const double* __restrict__ w,
                          const int* __restrict__ pl, const int* __restrict__ pk, int pitch, int terms, TRAJ_ARGS) {
  const TrajShape& T = shp[blockIdx.z];
  const int nG = T.nG, nP = T.nPairs, Kpad = T.Kg;
  outA = bat(outA, bs);
  orbs = bat(orbs, bs);
  w = bat(w, bs);
  pl = bat(pl, bs);
  pk = bat(pk, bs);
  GRID_STRIDE(e, (size_t)2 * nP * Kpad) {
    int row = (int)(e / Kpad), g = (int)(e % Kpad);
    int p = row >> 1, s = row & 1;
    if (terms == 3) {
      float v = 0.0f;
      if (g < nG) {
        z_t a = orbs[(size_t)nG * pl[p] + g], b = orbs[(size_t)nG * pk[p] + g];
        float ar = f64_to_f32(a.x), ai = f64_to_f32(a.y), br = f64_to_f32(b.x), bi = f64_to_f32(b.y);
        float wg = f64_to_f32(w[g]);
        v = s ? (ar * bi - ai * br) * wg : (ar * br + ai * bi) * wg;
      }
      write_split3(outA, row, g, nG, pitch, 0, v);
    } else {
      double v = 0.0;
      if (g < nG) {
        z_t a = orbs[(size_t)nG * pl[p] + g], b = orbs[(size_t)nG * pk[p] + g];
        z_t sv = zscale(zcmul(a, b), w[g]);
        v = s ? sv.y : sv.x;
      }
      write_split(outA, row, g, nG, pitch, terms, 0, v);
    }
  }
}

// W[g][n] = sum_z P1[z][g][n] (FP64), split to WxA (g-major, K = 2P, zero for
// n >= 2P) and WTxB (pair-major, K = nG, zero for g >= nG).  A 32 x 32 tile of
// (g, n) per block: read along n, transposed through shared memory, written
// along n (WxA) and along g (WTxB).
constexpr int SW_T = 32;

__global__ void __launch_bounds__(256) k_split_W(__nv_bfloat16* __restrict__ WxA, __nv_bfloat16* __restrict__ WTxB,
                                                 const float* __restrict__ P1, int nSplit, int pitchP, int pitchG,
                                                 int terms, TRAJ_ARGS) {
  __shared__ double tile[SW_T][SW_T + 1];
  const TrajShape& T = shp[blockIdx.z];
  const int nG = T.nG, N2P = 2 * T.nPairs, KpP = T.Kp, KpG = T.Kg;
  const int g0 = blockIdx.x * SW_T, n0 = blockIdx.y * SW_T;
  if (g0 >= KpG || n0 >= KpP) return;
  WxA = bat(WxA, bs);
  WTxB = bat(WTxB, bs);
  P1 = bat(P1, bs);
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  for (int r = ty; r < SW_T; r += 8) {
    int g = g0 + r, n = n0 + tx;
    double v = 0.0;
    if (g < nG && n < N2P)
      for (int z = 0; z < nSplit; z++) v += (double)P1[((size_t)z * nG + g) * N2P + n];
    tile[r][tx] = v;
    if (g < nG && n < KpP) {
      if (terms == 3) write_split3(WxA, g, n, N2P, pitchP, 0, (float)v);
      else write_split(WxA, g, n, N2P, pitchP, terms, 0, v);
    }
  }
  __syncthreads();
  for (int r = ty; r < SW_T; r += 8) {
    int n = n0 + r, g = g0 + tx;
    if (n < N2P && g < KpG) {
      if (terms == 3) write_split3(WTxB, n, g, nG, pitchG, 1, (float)tile[tx][r]);
      else write_split(WTxB, n, g, nG, pitchG, terms, 1, tile[tx][r]);
    }
  }
}

// R'' rows n = 2q + s (s: re/im of the output), K = 2p + t (t: a or b of W_p).
__global__ void k_split_R(__nv_bfloat16* __restrict__ RxB, const z_t* __restrict__ Rp, const int* __restrict__ pl,
                          const int* __restrict__ pk, int pitchP, int terms, TRAJ_ARGS) {
  const TrajShape& T = shp[blockIdx.z];
  const int n = T.nOS, nP = T.nPairs, KpP = T.Kp;
  int Q = n * n;
  RxB = bat(RxB, bs);
  Rp = bat(Rp, bs);
  pl = bat(pl, bs);
  pk = bat(pk, bs);
  GRID_STRIDE(e, (size_t)2 * Q * KpP) {
    int row = (int)(e / KpP), k = (int)(e % KpP);
    int q = row >> 1, s = row & 1;
    double v = 0.0;
    if (k < 2 * nP) {
      int p = k >> 1, t = k & 1;
      int l = pl[p], kk = pk[p];
      z_t R1 = Rp[(size_t)(l * n + kk) * Q + q];
      z_t R2 = (l < kk) ? Rp[(size_t)(kk * n + l) * Q + q] : zmk(0.0, 0.0);
      // X = R1 + R2, Y = i (R1 - R2): re/im parts of the selected one
      double r1 = s ? (t ? R1.x : R1.y) : (t ? -R1.y : R1.x);
      double r2 = s ? (t ? R2.x : R2.y) : (t ? -R2.y : R2.x);
      v = t ? r1 - r2 : r1 + r2;
    }
    if (terms == 3) write_split3(RxB, row, k, 2 * nP, pitchP, 1, f64_to_f32(v));
    else write_split(RxB, row, k, 2 * nP, pitchP, terms, 1, v);
  }
}

// Z[g][q] (complex) = sum_z P2[z][g][2q+s]
template <class PT>
__global__ void k_reduce_Z(z_t* __restrict__ Z, const PT* __restrict__ P2, int nSplit, TRAJ_ARGS) {
  const TrajShape& T = shp[blockIdx.z];
  const int nG = T.nG, Q = T.nOS * T.nOS;
  Z = bat(Z, bs);
  P2 = bat(P2, bs);
  GRID_STRIDE(e, (size_t)nG * Q) {
  int g = (int)(e / Q), q = (int)(e % Q);
  double re = 0.0, im = 0.0;
  for (int z = 0; z < nSplit; z++) {
    const PT* r = P2 + ((size_t)z * nG + g) * 2 * Q + 2 * q;
    re += (double)r[0];
    im += (double)r[1];
  }
  Z[e] = zmk(re, im);
  }
}

// H2s[(i1*n+j1)][(l2*n+k2)] = 1/2 sum_g S_(i1j1) W_(l2k2) from the unordered-pair products.
template <class PT>
__global__ void k_reduce_H2(z_t* __restrict__ H2s, const PT* __restrict__ P3, int nSplit,
                            const int* __restrict__ pidx, TRAJ_ARGS) {
  const TrajShape& T = shp[blockIdx.z];
  const int n = T.nOS, nP = T.nPairs;
  int Q = n * n;
  H2s = bat(H2s, bs);
  P3 = bat(P3, bs);
  pidx = bat(pidx, bs);
  GRID_STRIDE(e, (size_t)Q * Q) {
  int row = (int)(e / Q), col = (int)(e % Q);
  int i1 = row / n, j1 = row % n, l2 = col / n, k2 = col % n;
  bool c1 = i1 > j1, c2 = l2 > k2;
  int p = c1 ? pidx[j1 * n + i1] : pidx[i1 * n + j1];
  int pp = c2 ? pidx[k2 * n + l2] : pidx[l2 * n + k2];
  z_t v = zmk(0.0, 0.0);
  if (p >= 0 && pp >= 0) {
    int N2 = 2 * nP;
    double rr = 0, ii = 0, ri = 0, ir = 0;
    for (int z = 0; z < nSplit; z++) {
      const PT* G = P3 + (size_t)z * N2 * N2;
      rr += G[(size_t)(2 * p) * N2 + 2 * pp];
      ii += G[(size_t)(2 * p + 1) * N2 + 2 * pp + 1];
      ri += G[(size_t)(2 * p) * N2 + 2 * pp + 1];
      ir += G[(size_t)(2 * p + 1) * N2 + 2 * pp];
    }
    z_t G1 = zmk(rr - ii, ri + ir);   // sum S_p W_p'
    z_t G2 = zmk(rr + ii, ir - ri);   // sum S_p conj(W_p')
    if (!c1 && !c2) v = G1;
    else if (!c1 && c2) v = G2;
    else if (c1 && !c2) v = zconj(G2);
    else v = zconj(G1);
    v = zscale(v, 0.5);
  }
  H2s[e] = v;
  }
}


// ---- fixed-point digit slices -------------------------------------------------

// Slices of the contractions over the grid (L) and over the pairs (L2).  The
// mixed forms' targets are 30 and 36 bits of the row maxima; at a contraction
// length of at most 1024 they held 35 and 42 with the 7-bit digits they used to
// have there (up to 256: 32 and 40), which five or six 8-bit slices keep.
void fx_slices(int precision, int fx64, int kTiles, int pTiles, int* L, int* L2) {
  if (precision == CGPU_PREC_FP64) {
    *L = *L2 = fx64;
  } else {
    const int x6 = precision == CGPU_PREC_MIXED_FX6 ? 1 : 0;
    *L = x6 && kTiles <= 16 ? 6 : 5;
    *L2 = (pTiles <= 4 ? 4 : 5) + x6;
  }
}

// Signed base-256 digits of x relative to 2^e (|x| < 2^(e-1), or < 2^e for L <= 6): X = round(x 2^(8L-e))
// = sum_i d_i 2^(8(L-1-i)), d_i in [-128, 128) for i > 0, |d_0| <= 128.
// Integer operations only.  With H = 128 sum_{k<L-1} 256^k, the digits of Y = X + H
// below the top one are the plain base-256 digits d_i + 128, so every digit is an
// independent byte of Y: d_i = byte_i(Y) - 128, d_0 = Y >> 8(L-1) (arithmetic shift).
// FP64 subnormals (below 2^-1022 of anything) count as zero.
template <int L>
__device__ __forceinline__ void fx_digits(double x, int e, int (&d)[L]) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)((u >> 52) & 0x7FF);
  using Int = std::conditional_t<(L > 7), __int128, long long>;  // |Y| <= 2^(8L - 1) + H
  Int X = 0;
  if (ex != 0) {
    const unsigned long long mant = (u & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    const int sh = 1075 - ex - 8 * L + e;  // >= 54 - 8L because |x| < 2^(e-1) (53 - 8L: < 2^e)
    if (8 * L > 53 && sh <= 0) X = (Int)mant << -sh;
    else if (sh < 63) X = (Int)((mant + (1ull << (sh - 1))) >> sh);
    if (u >> 63) X = -X;
  }
  constexpr Int H = [] {
    Int h = 0;
    for (int i = 1; i < L; i++) h = (h << 8) | 128;
    return h;
  }();
  const Int Y = X + H;
#pragma unroll
  for (int i = 1; i < L; i++) d[i] = (int)(Y >> (8 * (L - 1 - i)) & 255) - 128;
  d[0] = (int)(Y >> (8 * (L - 1)));
}

// Two integers |d| <= 128 as a bf16 pair without conversion instructions: the
// FP32 magic-number sum 1.5 2^23 + d is exact, subtracting 1.5 2^23 leaves d as an
// FP32 with at most 8 significant bits, whose upper half is its bf16.
__device__ __forceinline__ unsigned fx_bf16x2(int d0, int d1) {
  const float f0 = __int_as_float(0x4B400000 + d0) - 12582912.0f, f1 = __int_as_float(0x4B400000 + d1) - 12582912.0f;
  return __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
}

__device__ __forceinline__ unsigned fx_biased_exp(double v) { return (unsigned)(__double2hiint(v) >> 20) & 0x7FFu; }
// smallest e with |x| < 2^(e-1) (wide: < 2^e) for the largest biased exponent m
// of a row (0: all zero; 2047: infinity or NaN).  wide is for the pair
// contractions of the mixed forms (K <= 256: |d_0| <= 256 stays exact).
__device__ __forceinline__ int fx_exp(unsigned m, bool wide = false) {
  return m == 0 ? 0 : m == 2047u ? FX_EXP_NAN : (int)m - (wide ? 1022 : 1021);
}

// Columns k, k + 1 (k even) of a row's L digit planes, relative to 2^e0 and 2^e1.
template <int L>
__device__ __forceinline__ void fx_store2(__nv_bfloat16* rowBase, size_t pitch, int k, double v0, double v1, int e0,
                                          int e1) {
  int d0[L], d1[L];
  fx_digits<L>(v0, e0, d0);
  fx_digits<L>(v1, e1, d1);
#pragma unroll
  for (int l = 0; l < L; l++) *reinterpret_cast<unsigned*>(rowBase + (size_t)l * pitch + k) = fx_bf16x2(d0[l], d1[l]);
}

// Sums of two values over the block, to its first warp.
__device__ z_t fx_block_sum(double a, double b) {
  __shared__ double red[2][32];
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (lane == 0) {
    red[0][threadIdx.x >> 5] = a;
    red[1][threadIdx.x >> 5] = b;
  }
  __syncthreads();
  a = b = 0.0;
  for (int w = 0; w < nw; w++) {
    a += red[0][w];
    b += red[1][w];
  }
  return zmk(a, b);
}

__device__ unsigned fx_block_max(unsigned m) {
  __shared__ unsigned red[32];
  m = __reduce_max_sync(0xffffffffu, m);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[wid] = m;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  unsigned r = 0;
  for (int i = 0; i < nw; i++) r = max(r, red[i]);
  return r;
}

// Scales of the pair contraction Z = W R'' in the FP64 form.  Its K index runs over the
// pairs, and a pair of orbitals that hardly overlap has a potential many orders below the
// others' with perhaps a large coefficient: rounded to their row's maximum, W's entry and R''s
// would lose what an FP64 sum keeps.  So W's column of pair p is taken times 2^-s_p and R''s
// row times 2^s_p, with sum_y |S_p| < 2^s_p: then the entries of a row of W lie within V's range
// of one another or below their own rounding error.  The scales enter as exponents
// alone (fx_scale_key).

// One block per row of K values: the exponent of its maximum, then the L digit
// planes, zero in [K, Kpad).  The values are staged in dynamic shared memory
// when `staged`, else formed twice (rows longer than shared memory).  scale (null: none):
// value k counts as value times 2^scale[k].
template <int L, class F>
__device__ void fx_row(__nv_bfloat16* rowBase, int* expOut, int K, int Kpad, int pitch, int staged, bool wide,
                       const int* scale, F value) {
  extern __shared__ double fxbuf[];
  unsigned m = 0;
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const double v = value(k);
    if (staged) fxbuf[k] = v;
    m = max(m, scale ? fx_scale_key(fx_biased_exp(v), scale[k]) : fx_biased_exp(v));
  }
  const unsigned M = fx_block_max(m);
  const int e = scale ? fx_key_exp(M) : fx_exp(M, wide);
  if (threadIdx.x == 0) *expOut = e;
  auto at = [&](int k) { return k < K ? (staged ? fxbuf[k] : value(k)) : 0.0; };
  auto ex = [&](int k) { return scale && k < K ? e - scale[k] : e; };
  for (int k = 2 * threadIdx.x; k < Kpad; k += 2 * blockDim.x)
    fx_store2<L>(rowBase, pitch, k, at(k), at(k + 1), ex(k), ex(k + 1));
}

constexpr size_t FX_STAGE_MAX = 200 * 1024;  // shared memory for staged rows; longer rows are formed twice

template <int L>
__global__ void __launch_bounds__(256) k_fx_split_V(__nv_bfloat16* __restrict__ out, int* __restrict__ eV,
                                                     const double* __restrict__ V, int pitch, TRAJ_ARGS) {
  const TrajShape& T = shp[blockIdx.z];
  const int g = blockIdx.x, nG = T.nG;
  if (g >= nG) return;
  out = bat(out, bs);
  eV = bat(eV, bs);
  V = bat(V, bs);
  const double* row = V + (size_t)g * nG;
  fx_row<L>(out + (size_t)g * L * pitch, eV + g, nG, (nG + 63) / 64 * 64, pitch, 0, false,
            nullptr, [&](int k) { return row[k]; });
}

// Rows 2p (real part) and 2p + 1 (imaginary part) of S = conj(phi_l) phi_k w
// over the grid (p = (l, k)), one block per pair, both rows staged in shared
// memory, each with the exponent of its own maximum.  In the mixed forms the
// complex product and the weight are double-float (FP32 pipe; ~2^-44 relative,
// below the digits' 2^-31 / 2^-39 of the row maximum); in the FP64 form they
// are FP64, rounded as FillInteractionSrc rounds them.  Block 0 of a trajectory
// also clears the W exponent maxima for GEMM1.
template <int L>
__global__ void __launch_bounds__(256) k_fx_split_S(__nv_bfloat16* __restrict__ out, int* __restrict__ eS,
                                                     unsigned* __restrict__ mWr, unsigned* __restrict__ mWc,
                                                     const z_t* __restrict__ orbs, const double* __restrict__ w,
                                                     const int* __restrict__ pl, const int* __restrict__ pk, int pitch,
                                                     int* __restrict__ sS, int staged, TRAJ_ARGS) {
  const TrajShape& T = shp[blockIdx.z];
  const int p = blockIdx.x, nG = T.nG, nP = T.nPairs;
  if (p >= nP) return;
  sS = bat(sS, bs);
  out = bat(out, bs);
  eS = bat(eS, bs);
  orbs = bat(orbs, bs);
  w = bat(w, bs);
  pl = bat(pl, bs);
  pk = bat(pk, bs);
  if (p == 0) {
    mWr = bat(mWr, bs);
    mWc = bat(mWc, bs);
    for (int i = threadIdx.x; i < nG; i += blockDim.x) mWr[i] = 0u;
    for (int i = threadIdx.x; i < 2 * nP; i += blockDim.x) mWc[i] = 0u;
  }
  extern __shared__ double fxbuf[];  // [2][pitch]: the real and the imaginary row
  const z_t* a = orbs + (size_t)nG * pl[p];
  const z_t* bo = orbs + (size_t)nG * pk[p];
  auto value = [&](int g) -> z_t {
    const z_t av = a[g], bv = bo[g];
    if (L > 6) return zscale(zcmul(av, bv), w[g]);
    const float2 ar = df_split(av.x), ai = df_split(av.y), br = df_split(bv.x), bi = df_split(bv.y);
    const float2 wg = df_split(w[g]);
    // conj(a) b = (ar br + ai bi) + i (ar bi - ai br)
    const float2 re = df_dot2(ar, br, ai, bi);
    const float2 im = df_dot2(ar, bi, make_float2(-ai.x, -ai.y), br);
    float s0 = 0.0f, c0 = 0.0f, s1 = 0.0f, c1 = 0.0f;
    df_mul_acc(s0, c0, re.x, re.y, wg.x, wg.y);
    df_mul_acc(s1, c1, im.x, im.y, wg.x, wg.y);
    return zmk(df_to_d(make_float2(s0, c0)), df_to_d(make_float2(s1, c1)));
  };
  unsigned mr = 0, mi = 0;
  double sr = 0.0, si = 0.0;  // sums of the sizes (FP64 form)
  for (int g = threadIdx.x; g < nG; g += blockDim.x) {
    const z_t v = value(g);
    if (staged) {
      fxbuf[g] = v.x;
      fxbuf[pitch + g] = v.y;
    }
    mr = max(mr, fx_biased_exp(v.x));
    mi = max(mi, fx_biased_exp(v.y));
    if (L > 6) {
      sr += fabs(v.x);
      si += fabs(v.y);
    }
  }
  if (L > 6) {
    const z_t sum = fx_block_sum(sr, si);
    if (threadIdx.x < 2) {
      const unsigned ex = fx_biased_exp(threadIdx.x ? sum.y : sum.x);
      sS[2 * p + threadIdx.x] = ex ? (int)ex - 1022 : FX_NO_SOURCE;
    }
  }
  const int er = fx_exp(fx_block_max(mr));
  const int ei = fx_exp(fx_block_max(mi));
  if (threadIdx.x == 0) {
    eS[2 * p] = er;
    eS[2 * p + 1] = ei;
  }
  __nv_bfloat16* rowR = out + (size_t)(2 * p) * L * pitch;
  __nv_bfloat16* rowI = out + (size_t)(2 * p + 1) * L * pitch;
  const int Kpad = T.Kg, shift = T.gShift;
  auto at = [&](int g) -> z_t {
    if (g < 0 || g >= nG) return zmk(0.0, 0.0);
    return staged ? zmk(fxbuf[g], fxbuf[pitch + g]) : value(g);
  };
  for (int k = 2 * threadIdx.x; k < Kpad; k += 2 * blockDim.x) {
    const z_t v0 = at(k - shift), v1 = at(k + 1 - shift);
    fx_store2<L>(rowR, pitch, k, v0.x, v1.x, er, er);
    fx_store2<L>(rowI, pitch, k, v0.y, v1.y, ei, ei);
  }
}

// Row n = 2q + s of R'' (K = 2p + t), as k_split_R.
template <int L>
__global__ void k_fx_split_R(__nv_bfloat16* __restrict__ out, int* __restrict__ eR, const z_t* __restrict__ Rp,
                             const int* __restrict__ pl, const int* __restrict__ pk, int pitch,
                             const int* __restrict__ sS, TRAJ_ARGS) {
  const TrajShape& T = shp[blockIdx.z];
  const int n = T.nOS, nP = T.nPairs, Q = n * n;
  const int row = blockIdx.x;
  if (row >= 2 * Q) return;
  out = bat(out, bs);
  eR = bat(eR, bs);
  sS = bat(sS, bs);
  Rp = bat(Rp, bs);
  pl = bat(pl, bs);
  pk = bat(pk, bs);
  const int q = row >> 1, s = row & 1;
  fx_row<L>(out + (size_t)row * L * pitch, eR + row, 2 * nP, T.Kp, pitch, 1, L <= 6, L > 6 ? sS : nullptr, [&](int k) {
    const int p = k >> 1, t = k & 1;
    const int l = pl[p], kk = pk[p];
    const z_t R1 = Rp[(size_t)(l * n + kk) * Q + q];
    const z_t R2 = (l < kk) ? Rp[(size_t)(kk * n + l) * Q + q] : zmk(0.0, 0.0);
    const double r1 = s ? (t ? R1.x : R1.y) : (t ? -R1.y : R1.x);
    const double r2 = s ? (t ? R2.x : R2.y) : (t ? -R2.y : R2.x);
    return t ? r1 - r2 : r1 + r2;
  });
}

// W = sum of the K-split partials (into slot 0) and the exponent maxima of its
// rows and columns (used when GEMM1 ran with split K).  A maximum is read before
// it is raised: almost every entry is below it, and an atomic each would queue
// the whole matrix on 2P + nG words.
__global__ void k_fx_reduce_W(double* __restrict__ Wd, unsigned* __restrict__ mWr, unsigned* __restrict__ mWc,
                              const int* __restrict__ sS, int nSplit, TRAJ_ARGS) {
  const TrajShape& T = shp[blockIdx.z];
  const int nG = T.nG, N = 2 * T.nPairs;
  Wd = bat(Wd, bs);
  mWr = bat(mWr, bs);
  mWc = bat(mWc, bs);
  sS = bat(sS, bs);  // null: no scales
  const size_t tot = (size_t)nG * N;
  GRID_STRIDE(e, tot) {
    double v = 0.0;
    for (int z = 0; z < nSplit; z++) v += Wd[(size_t)z * tot + e];
    Wd[e] = v;
    const unsigned ex = fx_biased_exp(v);
    unsigned *r = mWr + e / N, *q = mWc + e % N;
    const unsigned key = sS ? fx_scale_key(ex, -sS[e % N]) : ex;
    if (key > *(volatile unsigned*)r) atomicMax(r, key);
    if (ex > *(volatile unsigned*)q) atomicMax(q, ex);
  }
}

// W (FP64 [nG][2P]) to WxA (rows g, K = 2P, L2 digits; null: not wanted) and WTxB
// (rows n, K = nG at columns gShift + g, L digits) planes, with the row
// exponents eWr[g] / eWc[n].  One block per 64 x 64 tile (columns of WTxB by
// columns of W), transposed through shared memory; a lane forms two adjacent
// columns of a plane, so that the digits leave as 128-byte rows.
constexpr int FW_T = 64;
template <int L, int L2, int THREADS>
__global__ void __launch_bounds__(THREADS) k_fx_split_W(__nv_bfloat16* __restrict__ WxA, __nv_bfloat16* __restrict__ WTxB,
                                                     int* __restrict__ eWr, int* __restrict__ eWc,
                                                     const double* __restrict__ Wd, const unsigned* __restrict__ mWr,
                                                     const unsigned* __restrict__ mWc, const int* __restrict__ sS,
                                                     int pitchP, int pitchG, TRAJ_ARGS) {
  __shared__ double tile[FW_T][FW_T + 1];
  const TrajShape& T = shp[blockIdx.z];
  const int nG = T.nG, N2P = 2 * T.nPairs, KpP = T.Kp, KpG = T.Kg, sh = T.gShift;
  const int c0 = blockIdx.x * FW_T, n0 = blockIdx.y * FW_T;
  if (c0 >= KpG || n0 >= KpP) return;
  WxA = bat(WxA, bs);
  WTxB = bat(WTxB, bs);
  eWr = bat(eWr, bs);
  eWc = bat(eWc, bs);
  Wd = bat(Wd, bs);
  mWr = bat(mWr, bs);
  mWc = bat(mWc, bs);
  sS = bat(sS, bs);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < FW_T * FW_T; i += THREADS) {
    const int r = i / FW_T, c = i % FW_T, g = c0 + r - sh, n = n0 + c;
    tile[r][c] = (g >= 0 && g < nG && n < N2P) ? Wd[(size_t)g * N2P + n] : 0.0;
  }
  __syncthreads();
  if (WxA) {
    const int n = n0 + 2 * lane;
    const bool scaled = L2 > 6 && n < N2P;
    const int s0 = scaled ? sS[n] : 0, s1 = scaled ? sS[n + 1] : 0;
    for (int r = warp; r < FW_T; r += THREADS / 32) {
      const int g = c0 + r - sh;
      if (g < 0 || g >= nG) continue;
      const int e = L2 > 6 ? fx_key_exp(mWr[g]) : fx_exp(mWr[g], true);
      if (n0 == 0 && lane == 0) eWr[g] = e;
      fx_store2<L2>(WxA + (size_t)g * L2 * pitchP, pitchP, n, tile[r][2 * lane], tile[r][2 * lane + 1], e + s0, e + s1);
    }
  }
  for (int r = warp; r < FW_T; r += THREADS / 32) {
    const int n = n0 + r;
    if (n >= N2P) break;
    const int e = fx_exp(mWc[n]);
    if (c0 == 0 && lane == 0) eWc[n] = e;
    fx_store2<L>(WTxB + (size_t)n * L * pitchG, pitchG, c0 + 2 * lane, tile[2 * lane][r], tile[2 * lane + 1][r], e,
                 e);
  }
}

size_t take(size_t& off, size_t bytes) {
  size_t o = (off + 255) & ~(size_t)255;
  off = o + std::max<size_t>(bytes, 1);
  return o;
}

}  // namespace

// Sizes (base == nullptr) or places (base = the arena) the mixed-form buffers of
// one trajectory block starting at byte offset `off`; returns the end offset.
size_t mixed_layout(cgpu_ctx* c, char* base, size_t off) {
  if ((c->precision == CGPU_PREC_FP64 && !c->fxOn) || !c->hasInteraction) return off;
  if (!c->mixed) c->mixed = new MixedBufs();
  MixedBufs* m = c->mixed;
  m->terms = c->precision == CGPU_PREC_MIXED_X6 ? 6 : 3;
  int nG = c->nG, nP = c->nPairs, Q = c->nOS * c->nOS, T = m->terms;
  m->KgMax = (nG + 63) / 64 * 64;
  m->KpMax = (2 * nP + 63) / 64 * 64;
  typedef __nv_bfloat16 bf;
  if (c->fxOn) {
    m->KgMax = c->fxKgMax;  // includes the K-tile offsets of a shared interaction matrix
    const int kg = m->KgMax / 64, kp = m->KpMax / 64;
    fx_slices(c->precision, c->fx64, kg, kp, &m->L, &m->L2);
    m->L64 = c->fx64;
    m->LV = std::max(m->L, m->L64);
    const int L = m->L, L2 = m->L2, L64 = m->L64, LV = m->LV;
    auto plan = [&](FxGemm& g, int Lg, int M, int N, int kTiles, bool compact, bool extra) {
      g.compact = compact;
      g.bn = fx_tile_n(N, Lg, compact);
      g.s = fx_split_count(M, N, g.bn, Lg, kTiles, c->nb, extra);
    };
    plan(m->gW, L, nG, 2 * nP, kg, false, true);
    plan(m->gZ, L2, nG, 2 * Q, kp, c->nb > 1 && fx_compact_ok(L2), true);
    plan(m->gH, L, 2 * nP, 2 * nP, kg, false, false);
    if (L64) {
      plan(m->gWx, L64, nG, 2 * nP, kg, false, true);
      plan(m->gHx, L64, 2 * nP, 2 * nP, kg, false, false);
    }
    // partial buffers: a single system of a tunable form holds twice the
    // heuristic's K splits (room for the tile tuner), else exactly the heuristic's
    const int grow = c->nb == 1 && L != L64 ? 2 : 1;
    m->sCapW = std::max(std::min(m->gW.s * grow, kg), m->gWx.s);
    m->sCapZ = std::min(m->gZ.s * grow, kp);
    m->sCapH = std::max(std::min(m->gH.s * grow, kg), m->gHx.s);
    const size_t perTrajV = c->fxShared ? 0 : 1;
    size_t oV = take(off, perTrajV * sizeof(bf) * (size_t)nG * LV * m->KgMax);
    size_t oS = take(off, sizeof(bf) * (size_t)2 * nP * LV * m->KgMax);
    size_t oW = take(off, sizeof(bf) * (size_t)nG * L2 * m->KpMax);
    size_t oWT = take(off, sizeof(bf) * (size_t)2 * nP * LV * m->KgMax);
    size_t oR = take(off, sizeof(bf) * (size_t)2 * Q * L2 * m->KpMax);
    size_t oWd = take(off, sizeof(double) * (size_t)m->sCapW * nG * 2 * nP);
    size_t oZp = take(off, m->sCapZ > 1 ? sizeof(double) * (size_t)m->sCapZ * nG * 2 * Q : 0);
    size_t oGd = take(off, sizeof(double) * (size_t)m->sCapH * 2 * nP * 2 * nP);
    size_t oZ = take(off, sizeof(double) * (size_t)2 * nG * Q);
    size_t oeV = take(off, perTrajV * sizeof(int) * (size_t)nG);
    size_t oeS = take(off, sizeof(int) * (size_t)2 * nP);
    size_t osS = take(off, sizeof(int) * (size_t)2 * nP);
    size_t oeWr = take(off, sizeof(int) * (size_t)nG);
    size_t oeWc = take(off, sizeof(int) * (size_t)2 * nP);
    size_t oeR = take(off, sizeof(int) * (size_t)2 * Q);
    size_t omWr = take(off, sizeof(unsigned) * (size_t)nG);
    size_t omWc = take(off, sizeof(unsigned) * (size_t)2 * nP);
    if (base) {
      m->VxB = perTrajV ? (bf*)(base + oV) : nullptr;
      m->SxA = (bf*)(base + oS);
      m->WxA = (bf*)(base + oW);
      m->WTxB = (bf*)(base + oWT);
      m->RxB = (bf*)(base + oR);
      m->Wd = (double*)(base + oWd);
      m->Zp = m->sCapZ > 1 ? (double*)(base + oZp) : nullptr;
      m->Gd = (double*)(base + oGd);
      m->Zd = (double*)(base + oZ);
      m->eV = perTrajV ? (int*)(base + oeV) : nullptr;
      m->eS = (int*)(base + oeS);
      m->sS = (int*)(base + osS);
      m->eWr = (int*)(base + oeWr);
      m->eWc = (int*)(base + oeWc);
      m->eR = (int*)(base + oeR);
      m->mWr = (unsigned*)(base + omWr);
      m->mWc = (unsigned*)(base + omWc);
    }
    return off;
  }
  // W = V S: in a batch one N tile of 256 covers all pairs (2P <= 156 for 12
  // orbitals), so the large V operand streams once per trajectory
  m->bn1 = (c->nb > 1 && 2 * nP <= 256) ? 256 : tc_tile_n(2 * nP);
  m->bn2 = tc_tile_n(2 * Q);
  m->bn3 = tc_tile_n(2 * nP);
  m->s1 = tc_split_count(nG, 2 * nP, m->bn1, T * m->KgMax / 64, c->nb);
  m->s2 = tc_split_count(nG, 2 * Q, m->bn2, T * m->KpMax / 64, c->nb);
  m->s3 = tc_split_count(2 * nP, 2 * nP, m->bn3, T * m->KgMax / 64, c->nb);
  size_t oV = take(off, sizeof(bf) * (size_t)nG * T * m->KgMax);
  size_t oS = take(off, sizeof(bf) * (size_t)2 * nP * T * m->KgMax);
  size_t oW = take(off, sizeof(bf) * (size_t)nG * T * m->KpMax);
  size_t oWT = take(off, sizeof(bf) * (size_t)2 * nP * T * m->KgMax);
  size_t oR = take(off, sizeof(bf) * (size_t)2 * Q * T * m->KpMax);
  size_t o1 = take(off, sizeof(float) * (size_t)m->s1 * nG * 2 * nP);
  size_t o2 = take(off, sizeof(float) * (size_t)m->s2 * nG * 2 * Q);
  size_t o3 = take(off, sizeof(float) * (size_t)m->s3 * 2 * nP * 2 * nP);
  size_t oZ = take(off, sizeof(double) * (size_t)2 * nG * Q);
  if (base) {
    m->VxB = (bf*)(base + oV);
    m->SxA = (bf*)(base + oS);
    m->WxA = (bf*)(base + oW);
    m->WTxB = (bf*)(base + oWT);
    m->RxB = (bf*)(base + oR);
    m->P1 = (float*)(base + o1);
    m->P2 = (float*)(base + o2);
    m->P3 = (float*)(base + o3);
    m->Zd = (double*)(base + oZ);
  }
  return off;
}

size_t mixed_outside_bytes(const cgpu_ctx* c) {
  if (!c->fxOn || !c->fxShared || !c->mixed) return 0;
  const size_t kgBig = (c->nG + 63) / 64 * 64;
  return c->fxRoots.size() * (size_t)c->nG * (c->mixed->LV * kgBig * sizeof(__nv_bfloat16) + sizeof(int));
}

bool mixed_alloc_outside(cgpu_ctx* c) {
  MixedBufs* m = c->mixed;
  if (!m || mixed_outside_bytes(c) == 0) return true;
  const size_t rows = (size_t)c->nG * c->fxRoots.size();
  m->KgBig = (c->nG + 63) / 64 * 64;
  return cudaMalloc(&m->Vsh, sizeof(__nv_bfloat16) * rows * m->LV * m->KgBig) == cudaSuccess &&
         cudaMalloc(&m->eVsh, sizeof(int) * rows) == cudaSuccess;
}

void mixed_free(cgpu_ctx* c) {
  if (c->mixed) {
    MixedBufs* m = c->mixed;
    if (m->Vsh) cudaFree(m->Vsh);
    if (m->eVsh) cudaFree(m->eVsh);
    for (FxGemm* g : {&m->gW, &m->gZ, &m->gH, &m->gWx, &m->gHx})
      if (g->tiles) cudaFree(g->tiles);
    if (m->err_h) cudaFreeHost((void*)m->err_h);
  }
  delete c->mixed;  // the other buffers belong to the arena
  c->mixed = nullptr;
}

// After the arena holds V: bf16 splits of V (static) and the TMA maps.
void mixed_init(cgpu_ctx* c) {
  MixedBufs* m = c->mixed;
  if (!m) return;
  {
    void* h = nullptr;
    CODY_CUDA(cudaHostAlloc(&h, sizeof(int), cudaHostAllocMapped));
    *(int*)h = 0;
    m->err_h = (volatile int*)h;
    CODY_CUDA(cudaHostGetDevicePointer((void**)&m->err, h, 0));
  }
  const int P2 = 2 * c->nPairs, Q2 = 2 * c->nOS * c->nOS;
  if (m->L) {
    const int L = m->L, L64 = m->L64, LV = m->LV, pV = LV * m->KgMax, pG = L * m->KgMax, pP = m->L2 * m->KpMax;
    auto splitV = LV == 9 ? k_fx_split_V<9> : LV == 8 ? k_fx_split_V<8> : LV == 6 ? k_fx_split_V<6> : k_fx_split_V<5>;
    if (c->fxShared) {
      // each root trajectory's interaction matrix, sliced once for the batch
      const int nR = (int)c->fxRoots.size();
      const size_t plane = (size_t)c->nG * LV * m->KgBig;  // elements per root
      CODY_CUDA(cudaMemsetAsync(m->Vsh, 0, sizeof(__nv_bfloat16) * plane * nR, c->stream));
      for (int r = 0; r < nR; r++) {
        const int root = c->fxRoots[r], nGb = c->sys[root].nG;
        const double* Vb = (const double*)((const char*)c->Vint_d + (size_t)root * c->bs);
        splitV<<<dim3(nGb, 1, 1), 256, 0, c->stream>>>(m->Vsh + plane * r, m->eVsh + (size_t)c->nG * r, Vb,
                                                             m->KgBig, c->shape_d + root, 0);
        CODY_LAUNCHED(c);
      }
      m->mVsh = tc_make_map_planes(m->Vsh, c->nG, LV * m->KgBig, 128, nR, sizeof(__nv_bfloat16) * plane);
    } else {
      splitV<<<dim3(c->nG, 1, c->nb), 256, 0, c->stream>>>(m->VxB, m->eV, c->Vint_d, m->KgMax, TRAJ_PASS(c));
      CODY_LAUNCHED(c);
      m->mV = tc_make_map(c, m->VxB, c->nG, pV, 128);
    }
    m->mSasB = tc_make_map(c, m->SxA, P2, pG, 128);
    m->mW = tc_make_map(c, m->WxA, c->nG, pP, 128);
    m->bS = fx_make_maps(c, m->SxA, P2, m->KgMax, L);
    m->bWT = fx_make_maps(c, m->WTxB, P2, m->KgMax, L);
    m->bR = fx_make_maps(c, m->RxB, Q2, m->KpMax, m->L2);
    auto tiles = [&](FxGemm& g, int id) { g.tiles = fx_build_tiles(c, id, g.bn, g.s, &g.nTiles); };
    tiles(m->gW, TC_GEMM_W);
    tiles(m->gZ, TC_GEMM_Z);
    tiles(m->gH, TC_GEMM_H2);
    if (L64) {
      m->mSxasB = tc_make_map(c, m->SxA, P2, L64 * m->KgMax, 128);
      m->bSx = fx_make_maps(c, m->SxA, P2, m->KgMax, L64);
      m->bWTx = fx_make_maps(c, m->WTxB, P2, m->KgMax, L64);
    }
    if (L64 && L != L64) {  // the FP64 form's FillH2 uses its own gW, gH
      tiles(m->gWx, TC_GEMM_W);
      tiles(m->gHx, TC_GEMM_H2);
    }
  } else {
    const int T = m->terms, pG = T * m->KgMax, pP = T * m->KpMax;
    k_split_V<<<bgrid(c, ew_blocks(c, (size_t)c->nG * m->KgMax)), 256, 0, c->stream>>>(m->VxB, c->Vint_d, m->KgMax, T,
                                                                                    TRAJ_PASS(c));
    CODY_LAUNCHED(c);
    m->mV = tc_make_map(c, m->VxB, c->nG, pG, 128);
    m->mS = tc_make_map(c, m->SxA, P2, pG, m->bn1);
    m->mW = tc_make_map(c, m->WxA, c->nG, pP, 128);
    m->mR = tc_make_map(c, m->RxB, Q2, pP, m->bn2);
    m->mSasB = tc_make_map(c, m->SxA, P2, pG, 128);
    m->mWT = tc_make_map(c, m->WTxB, P2, pG, m->bn3);
  }
  CODY_CUDA(cudaStreamSynchronize(c->stream));
}

// The kernels set the flag in host memory, so reading it after a
// synchronisation costs nothing.
int mixed_error(cgpu_ctx* c) { return c->mixed && c->mixed->err_h ? *c->mixed->err_h : 0; }

// The three fixed-point contractions with their K-split reductions, on the
// operands the digit splits left in the arena (one call = one launch of the
// GEMM, plus the reduction when K is split).  exact: L64 slices (FillH2).
// W = V S (pair potentials; row / column exponent maxima for the W split).
static void fx_run_W(cgpu_ctx* c, bool exact) {
  MixedBufs* m = c->mixed;
  const int nG = c->nG, nP = c->nPairs;
  const FxGemm& g = exact && m->L != m->L64 ? m->gWx : m->gW;
  const bool one = g.s == 1;
  const int* scale = exact || m->L == m->L64 ? m->sS : nullptr;  // the FP64 form's slices
  fx_gemm(c, exact ? m->L64 : m->L, g.compact, TC_GEMM_W, c->fxShared ? m->mVsh : m->mV, exact ? m->bSx : m->bS, g.bn,
          m->Wd, c->fxShared ? m->eVsh : m->eV, m->eS, one ? m->mWr : nullptr, one ? m->mWc : nullptr,
          c->fxShared ? m->KgBig : m->KgMax, m->KgMax, c->fxShared, g.s, g.tiles, g.nTiles, m->err, scale);
  if (!one) {
    k_fx_reduce_W<<<bgrid(c, ew_blocks(c, (size_t)nG * 2 * nP)), 256, 0, c->stream>>>(m->Wd, m->mWr, m->mWc, scale, g.s,
                                                                                   TRAJ_PASS(c));
    CODY_LAUNCHED(c);
  }
}

// Z = W R'' (the correlation contraction) into Zd.
static void fx_run_Z(cgpu_ctx* c) {
  MixedBufs* m = c->mixed;
  const int nG = c->nG, Q = c->nOS * c->nOS;
  const FxGemm& g = m->gZ;
  fx_gemm(c, m->L2, g.compact, TC_GEMM_Z, m->mW, m->bR, g.bn, g.s > 1 ? m->Zp : m->Zd, m->eWr, m->eR, nullptr, nullptr,
          m->KpMax, m->KpMax, 0, g.s, g.tiles, g.nTiles, m->err);
  if (g.s > 1) {
    k_reduce_Z<<<bgrid(c, ew_blocks(c, (size_t)nG * Q)), 256, 0, c->stream>>>((z_t*)m->Zd, m->Zp, g.s, TRAJ_PASS(c));
    CODY_LAUNCHED(c);
  }
}

// G = S^T W (h2) and its reduction into the spatial h2 block.
static void fx_run_H2(cgpu_ctx* c, bool exact) {
  MixedBufs* m = c->mixed;
  const int Q = c->nOS * c->nOS;
  const FxGemm& g = exact && m->L != m->L64 ? m->gHx : m->gH;
  fx_gemm(c, exact ? m->L64 : m->L, g.compact, TC_GEMM_H2, exact ? m->mSxasB : m->mSasB, exact ? m->bWTx : m->bWT, g.bn,
          m->Gd, m->eS, m->eWc, nullptr, nullptr, m->KgMax, m->KgMax, 0, g.s, g.tiles, g.nTiles, m->err);
  k_reduce_H2<<<bgrid(c, ew_blocks(c, (size_t)Q * Q)), 256, 0, c->stream>>>(c->h2s_d, m->Gd, g.s, c->pidx_d,
                                                                      TRAJ_PASS(c));
  CODY_LAUNCHED(c);
}

// ---- tile tuner hooks ---------------------------------------------------------
// The FP64 form has one tile width and is not tuned.
static bool fx_tunable(const cgpu_ctx* c) { return c->mixed && c->mixed->L && c->precision != CGPU_PREC_FP64; }

void fx_slice_plan(const cgpu_ctx* c, int* L, int* L2) {
  *L = c->mixed ? c->mixed->L : 0;
  *L2 = c->mixed ? c->mixed->L2 : 0;
}

bool fx_tiles_get(const cgpu_ctx* c, int* t) {
  if (!fx_tunable(c)) return false;
  const MixedBufs* m = c->mixed;
  int i = 0;
  for (const FxGemm* g : {&m->gW, &m->gZ, &m->gH}) {
    t[i++] = g->bn;
    t[i++] = g->compact;
    t[i++] = g->s;
  }
  return true;
}

// K blocks, split capacity and output columns of GEMM g.
static void fx_gemm_plan(const cgpu_ctx* c, int g, int& kTiles, int& cap, int& N) {
  const MixedBufs* m = c->mixed;
  if (g == TC_GEMM_W) { kTiles = m->KgMax / 64; cap = m->sCapW; N = 2 * c->nPairs; }
  else if (g == TC_GEMM_Z) { kTiles = m->KpMax / 64; cap = m->sCapZ; N = 2 * c->nOS * c->nOS; }
  else { kTiles = m->KgMax / 64; cap = m->sCapH; N = 2 * c->nPairs; }
}

const char* fx_tiles_refused(const cgpu_ctx* c, const int* t) {
  const MixedBufs* m = c->mixed;
  if (!fx_tunable(c)) return "tiles: not a fixed-point context";
  for (int g = 0; g < 3; g++) {
    int kTiles, cap, N;
    fx_gemm_plan(c, g, kTiles, cap, N);
    if (!fx_tile_supported(t[3 * g], g == TC_GEMM_Z ? m->L2 : m->L, t[3 * g + 1] != 0))
      return "tiles: no fixed-point GEMM configuration for that tile";
    if (t[3 * g + 2] < 1 || t[3 * g + 2] > kTiles) return "tiles: K split count outside 1..K blocks";
    const int s = fx_normalize_splits(kTiles, t[3 * g + 2]);
    // every split keeps at least two K blocks, as the set-up heuristic does
    if (s < fx_min_splits(kTiles, g == TC_GEMM_Z ? m->L2 : m->L) || s > cap || (s > 1 && s > kTiles / 2))
      return "tiles: K split outside the range of the level sums or the partial buffers";
  }
  return nullptr;
}

void fx_tiles_set(cgpu_ctx* c, const int* t) {
  if (const char* why = fx_tiles_refused(c, t)) throw std::string(why);
  MixedBufs* m = c->mixed;
  ctx_sync(c);
  FxGemm* gm[3] = {&m->gW, &m->gZ, &m->gH};
  for (int g = 0; g < 3; g++) {
    FxGemm& G = *gm[g];
    if (G.tiles) CODY_CUDA(cudaFree(G.tiles));
    G.tiles = nullptr;
    int kTiles, cap, N;
    fx_gemm_plan(c, g, kTiles, cap, N);
    const int s = fx_normalize_splits(kTiles, t[3 * g + 2]);
    G.tiles = fx_build_tiles(c, g, t[3 * g], s, &G.nTiles);
    G.bn = t[3 * g];
    G.compact = t[3 * g + 1] != 0;
    G.s = s;
  }
}

void fx_tile_candidates(const cgpu_ctx* c, int g, std::vector<std::array<int, 3>>& out) {
  out.clear();
  if (!fx_tunable(c)) return;
  int kTiles, cap, N;
  fx_gemm_plan(c, g, kTiles, cap, N);
  std::vector<std::pair<int, bool>> cfgs;
  fx_tile_configs(g == TC_GEMM_Z ? c->mixed->L2 : c->mixed->L, cfgs);
  std::vector<int> splits;
  for (int s : {1, 2, 3, 4, cap}) {
    int v = fx_normalize_splits(kTiles, s);
    if (v >= fx_min_splits(kTiles, g == TC_GEMM_Z ? c->mixed->L2 : c->mixed->L) && v <= cap && (v == 1 || v <= kTiles / 2) &&
        std::find(splits.begin(), splits.end(), v) == splits.end())
      splits.push_back(v);
  }
  for (const auto& cf : cfgs) {
    if (cf.first >= 2 * ((N + 15) / 16 * 16)) continue;  // wider than twice the output: idle MMA columns only
    for (int v : splits) out.push_back({cf.first, cf.second ? 1 : 0, v});
  }
}

double fx_time_contraction(cgpu_ctx* c, int g, int reps) {
  auto run = [&]() {
    if (g == TC_GEMM_W) fx_run_W(c, false);
    else if (g == TC_GEMM_Z) fx_run_Z(c);
    else fx_run_H2(c, false);
  };
  run();
  cudaEvent_t e0, e1;
  CODY_CUDA(cudaEventCreate(&e0));
  CODY_CUDA(cudaEventCreate(&e1));
  CODY_CUDA(cudaEventRecord(e0, c->stream));
  for (int r = 0; r < reps; r++) run();
  CODY_CUDA(cudaEventRecord(e1, c->stream));
  CODY_CUDA(cudaEventSynchronize(e1));
  float ms = 0.f;
  CODY_CUDA(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (mixed_error(c)) throw std::string("tiles: a fixed-point GEMM reported a wait timeout while timing");
  return ms / reps;
}

// S rows as L digit slices, W = V S, W columns as L and (wantW) rows as L2 digit slices.
template <int L, int L2>
static void fx_potentials(cgpu_ctx* c, const z_t* orbs, bool exact, bool wantW) {
  MixedBufs* m = c->mixed;
  ProfScope prof(c, CGPU_KERNEL_PAIR_POTENTIALS);
  const size_t need = 2 * sizeof(double) * m->KgMax;
  const int staged = need <= FX_STAGE_MAX;
  if (staged && need > 48 * 1024)
    CODY_CUDA(cudaFuncSetAttribute(k_fx_split_S<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FX_STAGE_MAX));
  k_fx_split_S<L><<<dim3(c->nPairs, 1, c->nb), 256, staged ? need : 0, c->stream>>>(
      m->SxA, m->eS, m->mWr, m->mWc, orbs, c->w_d, c->pairL_d, c->pairK_d, m->KgMax, m->sS, staged, TRAJ_PASS(c));
  CODY_LAUNCHED(c);
  branch_record(c, BR_SOURCES);
  fx_run_W(c, exact);
  dim3 gw(m->KgMax / FW_T, m->KpMax / FW_T, c->nb);
  // fewer than two tiles an SM: four times the warps a tile, whose rows are then two in turn instead
  // of eight (8 tiles, 501 points x 10 pairs: 16.2 -> 8.0 us; 220 tiles, 2801 x 136: 19.2 -> 12.5)
  const bool few = gw.x * gw.y * gw.z < 2 * (unsigned)c->numSms;
  auto split = few ? k_fx_split_W<L, L2, 1024> : k_fx_split_W<L, L2, 256>;
  split<<<gw, few ? 1024 : 256, 0, c->stream>>>(wantW ? m->WxA : nullptr, m->WTxB, m->eWr, m->eWc, m->Wd, m->mWr,
                                                 m->mWc, m->sS, m->KpMax, m->KgMax, TRAJ_PASS(c));
  CODY_LAUNCHED(c);
}

// Calls f<L, L2>() of the context's slice plan.
template <class F>
static void fx_plan(const cgpu_ctx* c, F f) {
  const int L = c->mixed->L, L2 = c->mixed->L2;
  if (L == 8) return f(std::integral_constant<int, 8>(), std::integral_constant<int, 8>());
  if (L == 9) return f(std::integral_constant<int, 9>(), std::integral_constant<int, 9>());
  if (L == 5 && L2 == 4) return f(std::integral_constant<int, 5>(), std::integral_constant<int, 4>());
  if (L == 5 && L2 == 5) return f(std::integral_constant<int, 5>(), std::integral_constant<int, 5>());
  if (L == 5 && L2 == 6) return f(std::integral_constant<int, 5>(), std::integral_constant<int, 6>());
  if (L == 6 && L2 == 5) return f(std::integral_constant<int, 6>(), std::integral_constant<int, 5>());
  if (L == 6 && L2 == 6) return f(std::integral_constant<int, 6>(), std::integral_constant<int, 6>());
  throw std::string("internal: no kernels for this slice plan");
}

// The pieces of the correlation in the fixed-point forms, for callers that place
// them on several streams: the pair potentials; the digits of rho^-1 rho2 (after
// launch_rdm_inverse and, in the FP64 form, the pair sources' scales: BR_SOURCES); Z from
// both, dOrbs += its contraction with the orbitals; h2 from the potentials.
bool fx_ready(const cgpu_ctx* c) { return c->fxOn && c->mixed && c->mixed->L > 0 && c->hasInteraction; }

void launch_fx_potentials(cgpu_ctx* c, const z_t* orbs) {
  fx_plan(c, [&](auto L, auto L2) { fx_potentials<L(), L2()>(c, orbs, false, true); });
}

void launch_fx_split_R(cgpu_ctx* c) {
  ProfScope prof(c, CGPU_KERNEL_CORRELATION);
  MixedBufs* m = c->mixed;
  fx_plan(c, [&](auto, auto L2) {
    k_fx_split_R<L2()><<<dim3(2 * c->nOS * c->nOS, 1, c->nb), 64, sizeof(double) * m->KpMax, c->stream>>>(
        m->RxB, m->eR, c->Rp_d, c->pairL_d, c->pairK_d, m->KpMax, m->sS, TRAJ_PASS(c));
  });
  CODY_LAUNCHED(c);
}

void launch_fx_Z(cgpu_ctx* c) {
  ProfScope prof(c, CGPU_KERNEL_CORRELATION);
  fx_run_Z(c);
}

void launch_fx_epilogue(cgpu_ctx* c, z_t* dOrbs, const z_t* orbs) {
  ProfScope prof(c, CGPU_KERNEL_CORRELATION);
  launch_corr_epilogue(c, dOrbs, orbs, (z_t*)c->mixed->Zd);
}

void launch_fx_h2(cgpu_ctx* c) {
  ProfScope prof(c, CGPU_KERNEL_H2);
  fx_run_H2(c, false);
  launch_h2_layout(c);
}

// In one row, or (no kernel family being profiled) the density's inverse beside the
// potentials and h2 beside Z, as in the equation of motion: a mean field of 10
// orbitals over 806 points 323 -> 263 us with its copies.
static void correlation_fx(cgpu_ctx* c, z_t* dOrbs, const z_t* orbs, int wantH2) {
  if (!c->profTarget) {
    branch_record(c, BR_START);
    launch_fx_potentials(c, orbs);
    branch_record(c, BR_POTENTIALS);
    {
      BranchStream on(c, c->side[0]);
      branch_wait(c, BR_START);
      launch_rdm_inverse(c);
      branch_wait(c, BR_SOURCES);
      launch_fx_split_R(c);
      branch_record(c, BR_DENSITY);
    }
    if (wantH2) {
      BranchStream on(c, c->side[1]);
      branch_wait(c, BR_POTENTIALS);
      launch_fx_h2(c);
      branch_record(c, BR_COEFFS);
    }
    branch_wait(c, BR_DENSITY);
    launch_fx_Z(c);
    launch_fx_epilogue(c, dOrbs, orbs);
    if (wantH2) branch_wait(c, BR_COEFFS);
    return;
  }
  launch_rdm_inverse(c);
  launch_fx_potentials(c, orbs);
  launch_fx_split_R(c);
  launch_fx_Z(c);
  launch_fx_epilogue(c, dOrbs, orbs);
  if (wantH2) launch_fx_h2(c);
}

void launch_fill_h2_fx(cgpu_ctx* c, const z_t* orbs) {
  if (c->fx64 == 9) fx_potentials<9, 9>(c, orbs, true, false);
  else fx_potentials<8, 8>(c, orbs, true, false);
  ProfScope prof(c, CGPU_KERNEL_H2);
  fx_run_H2(c, true);
  launch_h2_layout(c);
}

// ApplyCorrelationOp in the mixed form: dOrbs += rho^-1 rho2 W phi; h2 (FP64 nO^4) when wantH2.
void launch_correlation_mixed(cgpu_ctx* c, z_t* dOrbs, const z_t* orbs, int wantH2) {
  if (fx_ready(c)) return correlation_fx(c, dOrbs, orbs, wantH2);
  launch_rdm_inverse(c);
  if (!c->hasInteraction) {
    if (wantH2) {
      batch_zero(c, c->h2_d, sizeof(z_t) * (size_t)c->nO * c->nO * c->nO * c->nO);
      batch_zero(c, c->h2s_d, sizeof(z_t) * (size_t)c->nOS * c->nOS * c->nOS * c->nOS);
    }
    return;
  }
  MixedBufs* m = c->mixed;
  int nG = c->nG, nP = c->nPairs, n = c->nOS, Q = n * n, T = m->terms;
  {
    ProfScope prof(c, CGPU_KERNEL_PAIR_POTENTIALS);
    k_split_S<<<bgrid(c, ew_blocks(c, (size_t)2 * nP * m->KgMax)), 256, 0, c->stream>>>(
        m->SxA, orbs, c->w_d, c->pairL_d, c->pairK_d, m->KgMax, T, TRAJ_PASS(c));
    CODY_LAUNCHED(c);
    // V carries the B split pattern, S the A pattern: hi*hi + lo*hi + hi*lo (x3)
    tc_gemm(c, TC_GEMM_W, m->mV, m->mS, m->bn1, m->P1, T, m->KgMax, m->s1, nG, 2 * nP, m->err);
    dim3 gw(ceil_div(m->KgMax, SW_T), ceil_div(m->KpMax, SW_T), c->nb);
    k_split_W<<<gw, 256, 0, c->stream>>>(m->WxA, m->WTxB, m->P1, m->s1, m->KpMax, m->KgMax, T, TRAJ_PASS(c));
    CODY_LAUNCHED(c);
  }
  {
    ProfScope prof(c, CGPU_KERNEL_CORRELATION);
    k_split_R<<<bgrid(c, ew_blocks(c, (size_t)2 * Q * m->KpMax)), 256, 0, c->stream>>>(m->RxB, c->Rp_d, c->pairL_d,
                                                                                   c->pairK_d, m->KpMax, T,
                                                                                   TRAJ_PASS(c));
    CODY_LAUNCHED(c);
    tc_gemm(c, TC_GEMM_Z, m->mW, m->mR, m->bn2, m->P2, T, m->KpMax, m->s2, nG, 2 * Q, m->err);
    z_t* Z = (z_t*)m->Zd;
    k_reduce_Z<<<bgrid(c, ew_blocks(c, (size_t)nG * Q)), 256, 0, c->stream>>>(Z, m->P2, m->s2, TRAJ_PASS(c));
    CODY_LAUNCHED(c);
    launch_corr_epilogue(c, dOrbs, orbs, Z);
  }
  if (wantH2) {
    ProfScope prof(c, CGPU_KERNEL_H2);
    tc_gemm(c, TC_GEMM_H2, m->mSasB, m->mWT, m->bn3, m->P3, T, m->KgMax, m->s3, 2 * nP, 2 * nP, m->err);
    k_reduce_H2<<<bgrid(c, ew_blocks(c, (size_t)Q * Q)), 256, 0, c->stream>>>(c->h2s_d, m->P3, m->s3, c->pidx_d,
                                                                        TRAJ_PASS(c));
    CODY_LAUNCHED(c);
    launch_h2_layout(c);
  }
}
