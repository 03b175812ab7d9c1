// k_sil.cu -- a whole short-iterative-Lanczos integration of the one-body part
// in one launch (Integrate / PerformLanczosStep / EvaluateExpInSubspace,
// src/IntegratorList/Sil/S_IntegratorList_Sil.f90:114-310, on
// TimeDerivativeOrbsLin, S_Method_Mb_OrbBased_Mctdhx.f90:152-177).
//
// The launch-per-pass form (k_lanczos.cu) spends seven launches and five passes
// over the vectors on every Krylov iteration.  Here each trajectory has a group
// of blocks, every block owns a contiguous piece of its state vector, and an
// iteration has one barrier of the group.  With w_j = beta_{j-1} v_j not yet normalised,
//   before it  g = H w_j on the piece, published for the neighbours' halo of `band`
//              points; partials of <v_k, g>, <w_j, g>, ||g||^2 and ||w_j||^2;
//   after it   beta_{j-1} = ||w_j||, v_j = w_j / beta_{j-1}, h = g / beta_{j-1},
//              w_{j+1} = h - sum_k c_k v_k on the piece and on its halo, whose basis
//              vectors every block keeps.
// The second Gram-Schmidt pass (its own barrier) is decided by ||h||^2 - sum |c_k|^2;
// the norms in T are always sums over the vectors.  The piece, its metric and (where they
// fit) its basis vectors stay in shared memory.  Every block sums the same partials in
// the same order and evaluates exp(-i dt T) e1 itself, so all of them take the same
// decisions: second pass, breakdown, convergence, halving of the step.  An adaptive
// integration runs without the host for SIL_PASSES Krylov passes; what is left then (a
// tolerance that is never met, a long interval) is handed back, and the host launches the
// next part, so that no launch holds the GPU for longer than a fraction of a second.
//
// FP64 throughout, also for the mixed forms: up to one group block per SM the
// FP64 pipe is not the bound of this kernel (44 to 100 FMA an entry and
// iteration): the barriers, the reductions and the chains of dependent FP64
// instructions are.  One half step of 2801 points x 16 orbitals, K = 16: 1330 us as
// launches, 460 with two barriers an order, 370 here; 501 x 4, K = 12: 830, 170 and 133.
//
// The groups' blocks wait on one another, so the launch is cooperative (at most
// one block per SM) and every wait is bounded.
#include <algorithm>
#include <cstring>

#include "common.cuh"

namespace {

constexpr int SIL_K = 32;
constexpr int SIL_PART = SIL_K + 8;            // partial sums of a block (two sets)
constexpr int SIL_MIN = 32;                    // smallest piece worth a block of its own
constexpr size_t SIL_SMEM = 200 * 1024;
constexpr long long SIL_WAIT = 4000000000LL;   // cycles after which a barrier gives up
constexpr int SIL_PASSES = 64;                 // Krylov passes of one launch (about 1 ms each at most)
constexpr double SIL_ZERO = 1.0e-14, SIL_ETA2 = 1.0e-2;  // as k_lanczos.cu

// One block's place: its trajectory, its rank in the trajectory's group, the group's size.
struct SilBlock {
  int traj, rank, n;
};

// Barrier of one group: monotonic count, reset by the last block that leaves the kernel.
__device__ bool group_barrier(unsigned* ctr, unsigned target, int n, int* err) {
  __shared__ int ok;
  __syncthreads();
  if (n > 1 && threadIdx.x == 0) {
    ok = 1;
    __threadfence();
    atomicAdd(ctr, 1u);
    const long long t0 = clock64();
    unsigned v;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
      if (v >= target) break;
      if (clock64() - t0 > SIL_WAIT) {
        ok = 0;
        atomicExch(err, 21);
        break;
      }
    }
  } else if (threadIdx.x == 0) {
    ok = 1;
  }
  __syncthreads();
  return ok != 0;
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Warp sums of two / four values at once: a lane hands on the values it does not
// keep, so that the reduction costs 5 / 6 FP64 adds (each holds the pipe for 64
// cycles) instead of 10 / 20.  Value i ends in lane 16 i / 8 i (and its neighbours).
__device__ __forceinline__ double warp_sum2(double v0, double v1) {
  const bool u = threadIdx.x & 16;
  double x = u ? v1 : v0;
  x += __shfl_xor_sync(0xffffffffu, u ? v0 : v1, 16);
  for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
__device__ __forceinline__ double warp_sum4(double v0, double v1, double v2, double v3) {
  const bool u = threadIdx.x & 16, t = threadIdx.x & 8;
  double a = u ? v2 : v0, b = u ? v3 : v1;
  a += __shfl_xor_sync(0xffffffffu, u ? v0 : v2, 16);
  b += __shfl_xor_sync(0xffffffffu, u ? v1 : v3, 16);
  double x = t ? b : a;
  x += __shfl_xor_sync(0xffffffffu, t ? a : b, 8);
  for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

}  // namespace

// phi = exp(-i dt T) e1 of the m x m tridiagonal (alpha, beta), by one warp
// (lane i = row i, m <= 32).  The reference diagonalises T (DSYEV); the same vector
// comes from the Chebyshev (Jacobi-Anger) expansion of the exponential (Tal-Ezer &
// Kosloff, J. Chem. Phys. 81, 3967 (1984)):
//   T' = (T - c)/R with spectrum in [-1, 1] (Gershgorin bounds),
//   exp(-i z x) = J_0(z) + 2 sum_k (-i)^k J_k(z) T_k(x),  z = dt R,
//   phi = exp(-i dt c) sum_k a_k q_k,  q_0 = e1, q_1 = T' e1, q_{k+1} = 2 T' q_k - q_{k-1}.
// The Bessel values come from Miller's backward recurrence J_{k-1} = (2k/z) J_k -
// J_{k+1}, normalised by J_0 + 2 sum J_2k = 1, and the series runs to machine
// precision.  A warp's FP64 instruction holds its sub-partition's pipe for 64
// cycles, so the chains are kept short: the factors 2k/z are formed 32 at a time by
// the lanes, the normalisation is a warp sum, a Chebyshev term costs four FMA, and
// both recurrences start where (z/2)^n / n!, a bound on |J_n|, falls below 1e-19
// (52 -> 10 us at K = 16).  jb: 1216 doubles of shared memory.
//
// lz_series_warp: centre c, radius R, last term K and the coefficients jb[0] = J_0,
// jb[k] = 2 J_k of the series of exp(-i dt/n T); PARTS (the pulse gradient): n > 1
// where |dt| R is above LZ_PART, so that jb holds every term.
constexpr double LZ_PART = 700.0;
// Below it J_0 is 1 and the other terms are nothing.  The recurrence's 2k/z would overflow: one
// Krylov vector (m = 1: R is the 1e-300 added to a spectrum of no width) with |dt| >= 1.
constexpr double LZ_TINY = 1e-30;
template <bool PARTS>
__device__ void lz_series_warp(const double* alpha, const double* beta, int m, double dt, double* jb, double& c,
                               double& R, int& K, int& n) {
  constexpr int KMAX = 1180;
  const int lane = threadIdx.x & 31;
  const double a = lane < m ? alpha[lane] : 0.0;
  const double bl = lane >= 1 && lane < m ? beta[lane - 1] : 0.0;  // couples i-1, i
  const double br = lane + 1 < m ? beta[lane] : 0.0;               // couples i, i+1
  double lo = lane < m ? a - fabs(bl) - fabs(br) : 1e300, hi = lane < m ? a + fabs(bl) + fabs(br) : -1e300;
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  c = 0.5 * (hi + lo);
  R = 0.5 * (hi - lo) * (1.0 + 1e-12) + 1e-300;
  n = 1;
  if (PARTS) n = (int)fmin(fmax(ceil(fabs(dt) * R / LZ_PART), 1.0), (double)SIL_KEEP_PARTS);
  const double z = PARTS ? fabs(dt) * R / n : fabs(dt) * R;
  K = 1;
  if (z >= LZ_TINY) {
    // log2 of (z/2)^n / n! below -64
    const float l2 = log2f((float)fmin(z, 1e30) * 0.5f);
    float lg = 0.0f;
    for (K = 1; K < KMAX; K++) {
      lg += l2 - log2f((float)K);
      if (lg < -64.0f && (float)K > (float)z) break;
    }
  }
  __syncwarp();
  if (z < LZ_TINY) {
    if (lane == 0) {
      jb[0] = 1.0;
      jb[1] = 0.0;
    }
  } else {
    const double tz = 2.0 / z;
    double jp = 0.0, jc = 1e-280;
    for (int k0 = K + 12; k0 >= 1; k0 -= 32) {
      const double f = (double)(k0 - lane) * tz;  // 2k/z for k = k0 - lane
      const int n = min(32, k0);
      for (int i = 0; i < n; i++) {
        const double jm = fma(__shfl_sync(0xffffffffu, f, i), jc, -jp);
        jp = jc;
        jc = jm;
        const int k = k0 - i - 1;
        if (lane == 0 && k <= K) jb[k] = jc;
        if (((__double2hiint(jc) >> 20) & 0x7FF) > 1023 + 830) {  // rescale to keep the recurrence finite
          jc *= 1e-250;
          jp *= 1e-250;
          __syncwarp();
          for (int q = k + lane; q <= K; q += 32) jb[q] *= 1e-250;
          __syncwarp();
        }
      }
    }
    __syncwarp();
    double s = 0.0;
    for (int k = 2 * lane; k <= K; k += 64) s += k == 0 ? jb[0] : 2.0 * jb[k];
    const double inv = 1.0 / warp_sum(s);
    for (int k = lane; k <= K; k += 32) jb[k] *= k == 0 ? inv : 2.0 * inv;
  }
  __syncwarp();
}

// The tridiagonal 2 T' of a series, a lane a row.
struct LzRow {
  double ta, tl, tr;
  __device__ LzRow(const double* alpha, const double* beta, int m, double c, double iR) {
    const int lane = threadIdx.x & 31;
    ta = lane < m ? (alpha[lane] - c) * iR : 0.0;
    tl = lane >= 1 && lane < m ? beta[lane - 1] * iR : 0.0;
    tr = lane + 1 < m ? beta[lane] * iR : 0.0;
  }
  __device__ double mul(double v, double minus) const {  // 2 T' v - minus
    const double l = __shfl_up_sync(0xffffffffu, v, 1), r = __shfl_down_sync(0xffffffffu, v, 1);
    return fma(ta, v, fma(tl, l, fma(tr, r, -minus)));
  }
};

// The parts after one another, on a complex vector; parts: the vector at the start of
// each, 32 entries a part (may be null).
__device__ __noinline__ z_t lz_expsub_parts(LzRow T, const double* jb, int K, int n, double dt, double c,
                                            z_t* parts) {
  const int lane = threadIdx.x & 31;
  double vr = lane == 0 ? 1.0 : 0.0, vi = 0.0, sn, cs;
  sincos(dt / n * c, &sn, &cs);
  for (int s = 0; s < n; s++) {
    if (parts) parts[32 * s + lane] = zmk(vr, vi);
    double mr = vr, mi = vi, qr = 0.5 * T.mul(vr, 0.0), qi = 0.5 * T.mul(vi, 0.0);
    double er = jb[0] * vr, ei = jb[0] * vi, orr = jb[1] * qr, oi = jb[1] * qi;  // even terms; odd terms without -i
    for (int k = 2; k <= K; k++) {
      const double nr = T.mul(qr, mr), ni = T.mul(qi, mi);
      mr = qr;
      mi = qi;
      qr = nr;
      qi = ni;
      const double co = (k & 2) == 0 ? jb[k] : -jb[k];
      if (k & 1) {
        orr = fma(co, qr, orr);
        oi = fma(co, qi, oi);
      } else {
        er = fma(co, qr, er);
        ei = fma(co, qi, ei);
      }
    }
    if (dt < 0.0) {
      orr = -orr;
      oi = -oi;
    }
    const double pr = er + oi, pi = ei - orr;
    vr = cs * pr + sn * pi;
    vi = cs * pi - sn * pr;
  }
  return zmk(vr, vi);
}

template <bool PARTS>
__device__ void lz_expsub_warp(const double* alpha, const double* beta, int m, double dt, double* jb, double& fr,
                               double& fi, z_t* parts = nullptr) {
  const int lane = threadIdx.x & 31;
  double c, R;
  int K, n;
  lz_series_warp<PARTS>(alpha, beta, m, dt, jb, c, R, K, n);
  const LzRow T(alpha, beta, m, c, 2.0 / R);
  if (PARTS && n > 1) {
    const z_t v = lz_expsub_parts(T, jb, K, n, dt, c, parts);
    fr = v.x;
    fi = v.y;
    return;
  }
  // a_k = 2 (-i)^k J_k: 1, -i, -1, i in turn
  double qm = lane == 0 ? 1.0 : 0.0, q = 0.5 * T.mul(qm, 0.0);
  double pr = jb[0] * qm, pi = -jb[1] * q;
  for (int k = 2; k <= K; k++) {
    const double qn = T.mul(q, qm);
    qm = q;
    q = qn;
    const double co = (k & 2) == 0 ? jb[k] : -jb[k];  // k mod 4 = 0: 1, 1: -i, 2: -1, 3: i
    if (k & 1) pi = fma(-co, q, pi);
    else pr = fma(co, q, pr);
  }
  if (dt < 0.0) pi = -pi;  // the complex conjugate series
  double sn, cs;
  sincos(dt * c, &sn, &cs);
  fr = cs * pr + sn * pi;
  fi = cs * pi - sn * pr;
}

// Co-states of alpha and beta (lane i: alpha_i, beta_i) from that of phi (lane i:
// yb, in the convention dL = Re sum conj(yb) dphi): the reverse of the Chebyshev
// recurrence, part by part from the last.  With the series' coefficients a_k (and
// the phase) and the co-states conj(a_k) yb of the terms q_k,
//   l_k = conj(a_k) yb + 2 T' l_{k+1} - l_{k+2},
//   T'bar = l_1 q_0^T + sum_{k>1} 2 l_k q_{k-1}^T,  q_0bar = conj(a_0) yb + T' l_1 - l_2,
// the q_k run back by q_{k-1} = 2 T' q_k - q_{k+1}.  c and R are constants of the
// expansion: phi does not depend on them.
__device__ void lz_expsub_vjp_warp(const double* alpha, const double* beta, int m, double dt, double* jb, z_t yb,
                                   const z_t* parts, double& abar, double& bbar) {
  const int lane = threadIdx.x & 31;
  double c, R;
  int K, n;
  lz_series_warp<true>(alpha, beta, m, dt, jb, c, R, K, n);
  const double iR = 2.0 / R;
  const LzRow T(alpha, beta, m, c, iR);
  double sn, cs;
  sincos(dt / n * c, &sn, &cs);
  double sa = 0.0, sb = 0.0;
  for (int s = n - 1; s >= 0; s--) {
    const z_t v = s == 0 ? zmk(lane == 0 ? 1.0 : 0.0, 0.0) : parts[32 * s + lane];
    double mr = v.x, mi = v.y, qr = 0.5 * T.mul(mr, 0.0), qi = 0.5 * T.mul(mi, 0.0);  // q_0, q_1
    for (int k = 2; k <= K; k++) {
      const double nr = T.mul(qr, mr), ni = T.mul(qi, mi);
      mr = qr;
      mi = qi;
      qr = nr;
      qi = ni;
    }
    // f = conj(phase) yb; conj((-i)^k) f: f, i f, -f, -i f in turn (conjugate series: the odd ones negated)
    const double f0 = fma(yb.x, cs, -yb.y * sn), f1 = fma(yb.x, sn, yb.y * cs), od = dt < 0.0 ? -1.0 : 1.0;
    double l1r = 0.0, l1i = 0.0, l2r = 0.0, l2i = 0.0;  // l_{k+1}, l_{k+2}
    for (int k = K; k >= 1; k--) {                      // q = q_k, qm = q_{k-1}
      const double co = ((k & 2) ? -jb[k] : jb[k]) * ((k & 1) ? od : 1.0);
      const double gr = (k & 1) ? -f1 : f0, gi = (k & 1) ? f0 : f1;
      const double lr = fma(co, gr, T.mul(l1r, l2r)), li = fma(co, gi, T.mul(l1i, l2i));
      l2r = l1r;
      l2i = l1i;
      l1r = lr;
      l1i = li;
      const double h = k == 1 ? 0.5 : 1.0;
      const double nlr = __shfl_down_sync(0xffffffffu, lr, 1), nli = __shfl_down_sync(0xffffffffu, li, 1);
      const double nqr = __shfl_down_sync(0xffffffffu, mr, 1), nqi = __shfl_down_sync(0xffffffffu, mi, 1);
      sa = fma(h, fma(lr, mr, li * mi), sa);
      sb = fma(h, fma(lr, nqr, fma(li, nqi, fma(nlr, mr, nli * mi))), sb);
      if (k > 1) {
        const double pr = T.mul(mr, qr), pi = T.mul(mi, qi);  // q_{k-2}
        qr = mr;
        qi = mi;
        mr = pr;
        mi = pi;
      }
    }
    yb = zmk(fma(jb[0], f0, 0.5 * T.mul(l1r, 2.0 * l2r)), fma(jb[0], f1, 0.5 * T.mul(l1i, 2.0 * l2i)));
  }
  abar = lane < m ? sa * iR : 0.0;
  bbar = lane + 1 < m ? sb * iR : 0.0;
}

namespace {

// Vectors of a block: w_j with its halo, g, m g, the basis on the halo and (smemV) on the piece.
__host__ __device__ __forceinline__ size_t sil_entries(int cap, int band, int K, bool smemV) {
  return (size_t)cap * (3 + (smemV ? K : 0)) + 2 * (size_t)band * (1 + K);
}

struct SilArgs {
  const z_t* start;  // the vector to propagate, and its result (may be the same)
  z_t *state, *w0, *w1, *basis;
  size_t ldv;
  const double *m, *T, *V0, *x;
  const int* btOf;
  const SilBlock* blk;
  z_t* part;       // per block: SIL_K + 1 dot / norm partials, then one norm partial
  unsigned* bar;   // per trajectory: barrier count, blocks that have left
  const double* tBase;
  double tOff, dt;
  int K, window;
  double tol;
  double dtSub;    // the step to try first, and the halvings that led to it
  int restarts, maxRestarts;
  SilFlags* flags;  // host memory: the error word, and what an adaptive integration (trajectory 0) leaves
  int place;
  int cap, smemV;  // entries of the largest piece; basis vectors in shared memory
  int pt;          // threads per entry (4 where the pieces leave most of the block idle, else 1)
  // for the pulse gradient: a given field value, and what its reverse pass reads
  double E;
  SilKeep keep;
};

// MODE: a propagation, the pass kept for its reverse, the same with the vectors in
// global memory.
constexpr int SIL_STEP = 0, SIL_KEPT = 1, SIL_SPILLED = 2;

// SIL_T threads a block: 256 for the small pieces (four threads an entry), whose
// iteration is a chain of latencies; 512 where the basis fits shared memory; 1024
// where it is read from L2 (with two barriers an order, before the other steps of the
// propagation were shortened: 10 helium steps 10.1 / 10.6 / 11.9 ms with 256 / 512 /
// 1024, 2801 x 16 points 462 / 414 / 488 us, a scan of 24 8.78 / 8.37 / 8.13 ms).
template <int SIL_T, int MODE = SIL_STEP>
__global__ void __launch_bounds__(SIL_T, 1) k_sil(const SilArgs A, TRAJ_ARGS) {
  constexpr int SIL_W = SIL_T / 32;
  constexpr bool KEEP = MODE != SIL_STEP;
  const double tol = KEEP ? 0.0 : A.tol;  // the kept pass is of fixed order
  const SilBlock B = A.blk[blockIdx.x];
  const TrajShape& S = shp[B.traj];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nG = S.nG, band = S.band, nd = 2 * band + 1, nC = S.nC, cap = A.cap;
  z_t* state = batn(A.state, bs, B.traj);
  const z_t* start = batn(A.start, bs, B.traj);
  z_t* wb[2] = {batn(A.w0, bs, B.traj), batn(A.w1, bs, B.traj)};
  z_t* basis = batn(A.basis, bs, B.traj);
  const double* m = batn(A.m, bs, B.traj);
  const double* T = batn(A.T, bs, B.traj);
  const double* V0 = batn(A.V0, bs, B.traj);
  const double* x = batn(A.x, bs, B.traj);
  const int* btOf = batn(A.btOf, bs, B.traj);
  constexpr int PS = 2 * SIL_PART;
  z_t* part0 = A.part + (size_t)(blockIdx.x - B.rank) * PS;  // the group's partials, two sets in turn:
  int set = 0;                                               // a slow block may still read the last one
  unsigned* bar = A.bar + 2 * B.traj;
  unsigned target = 0;

  extern __shared__ z_t smDyn[];
  z_t* sm = MODE == SIL_SPILLED ? A.keep.spill + blockIdx.x * sil_entries(cap, band, SIL_K, false) : smDyn;
  z_t* vt = sm;                          // w_j with its halo: entries l0 - band .. l1 + band
  z_t* g = vt + cap + 2 * band;          // H w_j
  z_t* mw = g + cap;                     // m g
  z_t* Vh = mw + cap;                    // [K][2 band]: the basis on the halo
  z_t* V = Vh + 2 * band * A.K;          // [K][cap] when smemV
  __shared__ z_t coef[SIL_K + 2];
  __shared__ double alpha[SIL_K], beta[SIL_K], red[2 * SIL_W], jb[1216], errEst, shE, shBe, shInv, shN0, shN1;
  __shared__ z_t phi[SIL_K];

  const int per = (S.nS + B.n - 1) / B.n, l0 = min(S.nS, B.rank * per), cnt = min(S.nS, l0 + per) - l0;
  auto vec = [&](int k, int e) -> z_t& { return A.smemV ? V[(size_t)k * cap + e] : basis[A.ldv * k + vidx(S, l0 + e)]; };
  auto barrier = [&]() {
    target += B.n;
    return group_barrier(bar, target, B.n, &A.flags->err);
  };
  auto mine = [&]() { return part0 + (size_t)B.rank * PS + set * SIL_PART; };
  // after a barrier: sums over the group of the partial slots [0, n), one or two slots a
  // warp, into coef[0..n); the next partials go to the other set
  double* cf = reinterpret_cast<double*>(coef);
  auto gather = [&](int n) {
    const z_t* part = part0 + set * SIL_PART;
    if (n <= SIL_W) {
      if (wid < n) {
        double x0 = 0.0, y0 = 0.0;
        for (int b = lane; b < B.n; b += 32) {
          const z_t p = __ldcg(part + (size_t)b * PS + wid);
          x0 += p.x;
          y0 += p.y;
        }
        const double x = warp_sum2(x0, y0);
        if ((lane & 15) == 0) cf[2 * wid + (lane >> 4)] = x;
      }
    } else {
      for (int k = 2 * wid; k < n; k += 2 * SIL_W) {
        double x0 = 0.0, y0 = 0.0, x1 = 0.0, y1 = 0.0;
        for (int b = lane; b < B.n; b += 32) {
          const z_t* r = part + (size_t)b * PS + k;
          const z_t p = __ldcg(r), q = __ldcg(r + 1);  // slot k + 1 exists (SIL_PART slots a set)
          x0 += p.x;
          y0 += p.y;
          x1 += q.x;
          y1 += q.y;
        }
        const double x = warp_sum4(x0, y0, x1, y1);
        if ((lane & 7) == 0 && k + (lane >> 4) < n) cf[2 * k + (lane >> 3)] = x;
      }
    }
    set ^= 1;
    __syncthreads();
  };
  // entry e of vector k of a dots call: basis vector b0 + k, or w_j itself after the n0 of them
  auto dot_vec = [&](int b0, int n0, int k, int e) { return k < n0 ? vec(b0 + k, e) : vt[band + e]; };
  // partials of <v_k, .> with mw for k in [b0, b0 + n0) and, with self, w_j into slots 0..
  auto dots = [&](int b0, int n0, int self) {
    double* out = reinterpret_cast<double*>(mine());
    const int n = n0 + self;
    if (n <= SIL_W) {
      if (wid < n) {
        double ax = 0.0, ay = 0.0;
        for (int e = lane; e < cnt; e += 32) {
          const z_t v = dot_vec(b0, n0, wid, e), u = mw[e];
          ax = fma(v.x, u.x, fma(v.y, u.y, ax));
          ay = fma(v.x, u.y, fma(-v.y, u.x, ay));
        }
        const double x = warp_sum2(ax, ay);
        if ((lane & 15) == 0) out[2 * wid + (lane >> 4)] = x;
      }
    } else {
      for (int k = 2 * wid; k < n; k += 2 * SIL_W) {
        double ax = 0.0, ay = 0.0, bx = 0.0, by = 0.0;
        const int k1 = min(k + 1, n - 1);
        for (int e = lane; e < cnt; e += 32) {
          const z_t v = dot_vec(b0, n0, k, e), t = dot_vec(b0, n0, k1, e), u = mw[e];
          ax = fma(v.x, u.x, fma(v.y, u.y, ax));
          ay = fma(v.x, u.y, fma(-v.y, u.x, ay));
          bx = fma(t.x, u.x, fma(t.y, u.y, bx));
          by = fma(t.x, u.y, fma(-t.y, u.x, by));
        }
        const double x = warp_sum4(ax, ay, bx, by);
        if ((lane & 7) == 0 && k + (lane >> 4) < n) out[2 * k + (lane >> 3)] = x;
      }
    }
  };
  // block sums of p and q into the real and imaginary part of a slot (also orders mw)
  auto publish = [&](double p, double q, int slot) {
    const double x = warp_sum2(p, q);
    if ((lane & 15) == 0) red[2 * wid + (lane >> 4)] = x;
    __syncthreads();
    if (wid == 0) {
      const double y = warp_sum2(lane < SIL_W ? red[2 * lane] : 0.0, lane < SIL_W ? red[2 * lane + 1] : 0.0);
      if ((lane & 15) == 0) reinterpret_cast<double*>(mine() + slot)[lane >> 4] = y;
    }
  };
  const int pt = A.pt, eq = tid % pt, e0 = tid / pt, eStep = SIL_T / pt;
  // sum over the pt threads of an entry, to each of them
  auto entry_sum = [&](z_t r) {
    for (int o = 1; o < pt; o <<= 1) {
      r.x += __shfl_xor_sync(0xffffffffu, r.x, o);
      r.y += __shfl_xor_sync(0xffffffffu, r.y, o);
    }
    return r;
  };
  // vt = from - sum_k coef_k v_{b0 + k} on the piece and its halo (first: from = gIn inv, and
  // coef_{n0} v with v = vt inv, which becomes basis vector b0 + n0; else from = vt)
  auto subtract = [&](int b0, int n0, bool first, double inv, const z_t* gIn) {
    for (int qb = 0; qb < cnt + 2 * band; qb += eStep) {  // the piece (its accesses aligned), then the halo
      const int e = qb + e0, hh = e - cnt;
      const bool own = e < cnt;
      const int t = own ? band + e : hh < band ? hh : cnt + hh, l = l0 - band + t;
      const bool in = e < cnt + 2 * band && l >= 0 && l < S.nS;
      z_t r = zmk(0.0, 0.0);
      if (in) {
        if (eq == 0) r = first ? zscale(own ? g[e] : __ldcg(gIn + vidx(S, l)), inv) : vt[t];
        for (int k = eq; k < n0; k += pt) {
          const z_t v = own ? vec(b0 + k, e) : Vh[2 * band * (b0 + k) + hh], c = coef[k];
          r.x = fma(-c.x, v.x, fma(c.y, v.y, r.x));
          r.y = fma(-c.x, v.y, fma(-c.y, v.x, r.y));
        }
        if (first && eq == n0 % pt) {
          const z_t v = zscale(vt[t], inv), c = coef[n0];
          if (own) {
            vec(b0 + n0, e) = v;
            if (KEEP && A.smemV) A.keep.V[A.ldv * (b0 + n0) + vidx(S, l)] = v;
          } else {
            Vh[2 * band * (b0 + n0) + hh] = v;
          }
          r.x = fma(-c.x, v.x, fma(c.y, v.y, r.x));
          r.y = fma(-c.x, v.y, fma(-c.y, v.x, r.y));
        }
      }
      r = entry_sum(r);
      if (in && eq == 0) vt[t] = r;
    }
  };

  double tCur = A.tOff, rem = A.dt, dtS = A.dtSub;
  int warnings = 0, it = 0, restarts = A.restarts, pass = 0, notFinite = 0;
  bool ok = true;
  while (ok && fabs(rem) > SIL_ZERO && pass < SIL_PASSES) {
    double nrm = 0.0;
    bool conv = false, done = false, bad = false;
    while (pass < SIL_PASSES) {
      pass++;
      __syncthreads();
      // w_1 and its halo; the field takes a few microseconds of FP64 on one lane beside it
      if (tid == SIL_T - 1)
        shE = KEEP ? A.E : S.hasPot ? field_amplitude_dev(S.laser, *batn(A.tBase, bs, B.traj) + tCur + 0.5 * dtS) : 0.0;
      for (int t = tid; t < cnt + 2 * band; t += SIL_T) {
        const int l = l0 - band + t;
        vt[t] = l >= 0 && l < S.nS ? __ldcg(start + vidx(S, l)) : zmk(0.0, 0.0);
      }
      __syncthreads();
      const double E = shE;
      int mDim = A.K;
      for (int j = 1; j <= A.K; j++, it++) {
        z_t* gOut = wb[it & 1];
        if (j > 1) __syncthreads();
        double h2 = 0.0, n2 = 0.0;
        for (int eb = 0; eb < cnt; eb += eStep) {
          const int e = eb + e0, l = l0 + e;
          z_t h = zmk(0.0, 0.0);
          if (e < cnt && l >= nC) {  // the coefficients do not move
            const int r = l - nC, i = r / nG, x0 = r - i * nG;
            const double* Tb = T + (size_t)(S.restricted ? 0 : btOf[i]) * nd * nG + x0;
            const z_t* vv = vt + e;
            const int d0 = max(0, band - x0), d1 = min(nd, nG - x0 + band);  // inside the orbital
            for (int d = eq; d < d1; d += pt) {
              if (d < d0) continue;
              const double c = __ldg(Tb + (size_t)d * nG);
              h.x = fma(c, vv[d].x, h.x);
              h.y = fma(c, vv[d].y, h.y);
            }
            if ((S.hasPot || KEEP) && eq == pt - 1) {
              const double p = fma(E, x[x0], V0[x0]);
              h.x = fma(p, vv[band].x, h.x);
              h.y = fma(p, vv[band].y, h.y);
            }
          }
          h = entry_sum(h);
          if (e < cnt && eq == 0) {
            const size_t i = vidx(S, l);
            const double mi = m[i];
            const z_t u = zscale(h, mi), v = vt[band + e];
            g[e] = h;
            mw[e] = u;
            gOut[i] = h;
            h2 = fma(u.x, h.x, fma(u.y, h.y, h2));
            n2 = fma(mi, fma(v.x, v.x, v.y * v.y), n2);
          }
        }
        // the window's vectors; the three-term recurrence takes v_{j-1} too, for ||h||^2 and its beta
        const int b0 = A.window > 0 ? max(0, j - (A.window == 1 ? 2 : A.window)) : 0, n0 = j - 1 - b0;
        publish(h2, n2, n0 + 1);  // also orders mw before the dots
        dots(b0, n0, 1);
        if (!(ok = barrier())) break;
        gather(n0 + 2);
        if (wid == 0) {  // beta_{j-1} and the coefficients against normalised vectors
          const double be = sqrt(coef[n0 + 1].y), inv = 1.0 / be;
          z_t c = lane <= n0 ? zscale(coef[lane], lane < n0 ? inv : inv * inv) : zmk(0.0, 0.0);
          double q0 = coef[n0 + 1].x * (inv * inv);
          __syncwarp();
          if (A.window == 1) {
            c.y = 0.0;
            if (n0 == 1) {  // h = H v_j - beta_{j-1} v_{j-1}
              const double cp = __shfl_sync(0xffffffffu, c.x, 0);
              q0 += be * (be - 2.0 * cp);
              if (lane == 0) c.x = be;
            }
          }
          const double sq = A.window == 1 && lane < n0 ? 0.0 : fma(c.x, c.x, c.y * c.y);
          const double q1 = q0 - warp_sum(sq);
          if (lane <= n0) coef[lane] = c;
          if (lane == n0) alpha[j - 1] = c.x;
          if (lane == 0) {
            if (j > 1) beta[j - 2] = be;
            shBe = be;
            shInv = inv;
            shN0 = q0;
            shN1 = q1;
          }
        }
        __syncthreads();
        if (j == 1) {
          nrm = shBe;
          if (nrm <= SIL_ZERO && !KEEP) {  // nothing to propagate: the state stays
            conv = true;
            mDim = 0;
            it++;
            break;
          }
        }
        double n1 = shN1;
        subtract(b0, n0, true, shInv, gOut);
        if (n1 <= SIL_ETA2 * shN0) {  // most of h cancelled: project once more
          __syncthreads();
          double q = 0.0;
          for (int e = tid; e < cnt; e += SIL_T) {
            const z_t v = vt[band + e], u = zscale(v, m[vidx(S, l0 + e)]);
            mw[e] = u;
            q = fma(u.x, v.x, fma(u.y, v.y, q));
          }
          const int p0 = A.window > 0 ? max(0, j - A.window) : 0, np = j - p0;
          publish(q, 0.0, np);
          dots(p0, np, 0);
          if (!(ok = barrier())) break;
          gather(np + 1);
          if (wid == 0) {
            const z_t c = lane < np ? coef[lane] : zmk(0.0, 0.0);
            const double q1 = coef[np].x - warp_sum(fma(c.x, c.x, c.y * c.y));
            if (lane == 0) shN1 = q1;
          }
          subtract(p0, np, false, 0.0, nullptr);
          __syncthreads();
          n1 = shN1;
        }
        // a rounding below zero is zero; NaN (an infinity or a NaN in the state) stays NaN: no breakdown
        const double be = n1 < 0.0 ? 0.0 : sqrt(n1);
        const bool broke = be <= SIL_ZERO && !KEEP;  // the kept pass runs over all orders
        const bool last = broke || j == A.K;
        if (tol > 0.0 || last) {
          __syncthreads();
          if (wid == 0) {
            if (lane == 0) beta[j - 1] = be;
            double fr, fi;
            lz_expsub_warp<KEEP>(alpha, beta, j, dtS, jb, fr, fi, KEEP && B.rank == 0 ? A.keep.parts : nullptr);
            if (lane < j) phi[lane] = zmk(fr, fi);
            if (lane == j - 1) errEst = broke ? 0.0 : be * sqrt(fr * fr + fi * fi);
          }
          __syncthreads();
          conv = errEst <= tol;
          // not finite: no step converges from here, however short (the fixed orders run on)
          bad = tol > 0.0 && !(fabs(nrm) + fabs(alpha[j - 1]) + be < INFINITY);
          if (bad || (tol > 0.0 && conv) || last) {
            mDim = j;
            it++;
            break;
          }
        }
      }
      done = mDim == 0;
      if (!ok || done) break;
      if (conv || bad || !(tol > 0.0) || fabs(dtS) <= SIL_ZERO || restarts >= A.maxRestarts) {
        for (int e = tid; e < cnt; e += SIL_T) {
          z_t acc = zmk(0.0, 0.0);
          for (int k = 0; k < mDim; k++) zfma(acc, vec(k, e), phi[k]);
          state[vidx(S, l0 + e)] = zscale(acc, nrm);
        }
        if (KEEP) {
          for (int e = tid; e < cnt; e += SIL_T) A.keep.last[l0 + e] = vt[band + e];
          if (B.rank == 0 && tid < A.K) {
            A.keep.alpha[tid] = alpha[tid];
            A.keep.beta[tid] = beta[tid];
            A.keep.phi[tid] = phi[tid];
            if (tid == 0) *A.keep.norm = nrm;
          }
        }
        done = true;
        break;
      }
      dtS = 0.5 * dtS;
      restarts++;
    }
    if (!ok || !done) break;
    if (!conv && !bad) warnings++;
    if (bad) {
      notFinite = 1;
      break;
    }
    if (!(tol > 0.0)) break;  // fixed order: one pass over the whole step
    tCur += dtS;
    rem -= dtS;
    dtS = rem;
    restarts = 0;
    if (fabs(rem) > SIL_ZERO) ok = barrier();  // the neighbours' pieces of the new start
  }
  if (tid == 0) {
    if (B.traj == 0 && B.rank == 0 && tol > 0.0) {
      SilLeft& left = A.flags->left[A.place];
      left.warnings = warnings;
      left.t = tCur;
      left.rem = rem;
      left.dtSub = dtS;
      left.restarts = restarts;
      left.notFinite = notFinite;
    }
    if (B.n > 1 && atomicAdd(bar + 1, 1u) == (unsigned)B.n - 1) {
      bar[0] = 0u;
      bar[1] = 0u;
      __threadfence();
    }
  }
}

size_t sil_smem(int cap, int band, int K, bool smemV) { return sizeof(z_t) * sil_entries(cap, band, K, smemV); }

}  // namespace

namespace {

struct SilVjpArgs {
  SilKeep k;
  const z_t* obar;
  const double *m, *T, *V0, *x;
  z_t *sbar, *vb0, *vb1;
  double *grad, E, dt;
  z_t* part;
  unsigned* bar;
  int cap, nBlk;
  SilFlags* flags;
};

// The reverse of one kept pass: sbar = (d out / d start)^H obar, grad += the field
// part, differentiating the three-term recurrence (its re-orthogonalisation is the
// identity in exact arithmetic).  With r_j = H v_j - beta_{j-1} v_{j-1} - alpha_j v_j =
// beta_j v_{j+1} the reverse step of order j is local in the vectors once two sums
// over the previous one are known:
//   bb = bbar_j - <vbar_{j+1}, v_{j+1}> / beta_j,   rbar = vbar_{j+1} / beta_j + bb m v_{j+1},
//   ab = abar_j - <vbar_{j+1}, v_j> / beta_j,       wbar_j = rbar + ab m v_j,
//   vbar_j = ||s|| conj(phi_j) obar - beta_j wbar_{j+1} - alpha_j rbar + ab m (r_j + alpha_j v_j) + H^T wbar_j,
// with bbar_j reduced by <wbar_{j+1}, v_j>, so there is one barrier per order.  A
// block forms wbar on its halo itself.  12 orders, 501 x 8 points: 1200 us as
// launches per operation, 148 here.
template <bool SPILL>
__global__ void __launch_bounds__(256, 1) k_sil_vjp(const SilVjpArgs A, TRAJ_ARGS) {
  constexpr int T = 256, W = T / 32;
  const TrajShape& S = shp[0];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, rank = blockIdx.x;
  const int nG = S.nG, band = S.band, nd = 2 * band + 1, nC = S.nC, nS = S.nS, K = A.k.K;
  constexpr int PS = SIL_PART;
  z_t* mine = A.part + (size_t)rank * PS;
  unsigned target = 0;
  extern __shared__ z_t smDyn[];
  z_t* sm = SPILL ? A.k.spill + rank * (size_t)(3 * A.cap + 2 * band) : smDyn;
  z_t* wh = sm;                       // wbar_j with its halo
  z_t* vbj = wh + A.cap + 2 * band;   // vbar of the last order
  z_t* wPrev = vbj + A.cap;           // wbar of the last order
  __shared__ z_t coef[SIL_K + 1], phi[SIL_K];
  __shared__ double alpha[SIL_K], beta[SIL_K], abar[SIL_K], bbar[SIL_K], red[4][W], jb[1216];
  const int per = (nS + A.nBlk - 1) / A.nBlk, l0 = min(nS, rank * per), cnt = min(nS, l0 + per) - l0;
  auto barrier = [&]() {
    target += A.nBlk;
    return group_barrier(A.bar, target, A.nBlk, &A.flags->err);
  };
  auto gather = [&](int s0, int n) {
    for (int k = wid; k < n; k += W) {
      double x0 = 0.0, y0 = 0.0;
      for (int b = lane; b < A.nBlk; b += 32) {
        const z_t p = __ldcg(A.part + (size_t)b * PS + s0 + k);
        x0 += p.x;
        y0 += p.y;
      }
      const double x = warp_sum2(x0, y0);
      if ((lane & 15) == 0) reinterpret_cast<double*>(coef)[2 * k + (lane >> 4)] = x;
    }
    __syncthreads();
  };
  if (tid < K) {
    alpha[tid] = A.k.alpha[tid];
    beta[tid] = A.k.beta[tid];
    phi[tid] = A.k.phi[tid];
  }
  const double nrm = *A.k.norm;
  bool ok = true;
  // phibar_j = ||s|| <v_j, obar> (no metric)
  for (int k = wid; k < K; k += W) {
    const z_t* v = A.k.V + (size_t)nS * k + l0;
    double ax = 0.0, ay = 0.0;
    for (int e = lane; e < cnt; e += 32) {
      const z_t a = v[e], b = A.obar[l0 + e];
      ax = fma(a.x, b.x, fma(a.y, b.y, ax));
      ay = fma(a.x, b.y, fma(-a.y, b.x, ay));
    }
    const double x = warp_sum2(ax, ay);
    if ((lane & 15) == 0) reinterpret_cast<double*>(mine)[2 * k + (lane >> 4)] = x;
  }
  ok = barrier();
  double nbar = 0.0, gx = 0.0;
  if (ok) {
    gather(0, K);
    for (int j = 0; j < K; j++) nbar += coef[j].x * phi[j].x + coef[j].y * phi[j].y;
    if (wid == 0) {
      const z_t yb = lane < K ? zscale(coef[lane], nrm) : zmk(0.0, 0.0);
      double a, b;
      lz_expsub_vjp_warp(alpha, beta, K, A.dt, jb, yb, A.k.parts, a, b);
      if (lane < K) {
        abar[lane] = a;
        bbar[lane] = b;
      }
    }
    __syncthreads();
  }
  double d1 = 0.0, e1 = 0.0, f1 = 0.0;  // <vbar_{j+1}, v_{j+1}>, <vbar_{j+1}, v_j>, <wbar_{j+1}, v_j>
  for (int j = K - 1; ok && j >= 0; j--) {
    const bool last = j == K - 1;
    const double be = beta[j], al = alpha[j];
    const double bb = last ? 0.0 : bbar[j] - f1 - d1 / be, ab = last ? abar[j] : abar[j] - e1 / be, ib = 1.0 / be;
    const z_t* vj = A.k.V + (size_t)nS * j;
    const z_t* vn = last ? A.k.last : vj + nS;
    const z_t* vbn = (j & 1) ? A.vb0 : A.vb1;  // vbar_{j+1}, published by the previous order
    z_t* vbo = (j & 1) ? A.vb1 : A.vb0;
    for (int t = tid; t < cnt + 2 * band; t += T) {
      const int l = l0 - band + t;
      z_t wv = zmk(0.0, 0.0);
      if (l >= 0 && l < nS) {
        const double mi = A.m[l];
        wv = zscale(vj[l], ab * mi);
        if (!last) {
          const z_t r = zadd(zscale(__ldcg(vbn + l), ib), zscale(vn[l], bb * mi));
          wv = zadd(wv, r);
        }
      }
      wh[t] = wv;
    }
    __syncthreads();
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int e = tid; e < cnt; e += T) {
      const int l = l0 + e;
      const z_t v = vj[l], n = vn[l], wv = wh[band + e], ob = A.obar[l];
      const double mi = A.m[l];
      z_t o = zscale(zcmul(phi[j], ob), nrm);
      // ab m (r + alpha v): r = beta_j v_{j+1}, or the kept residual of the last order
      const double rs = last ? 1.0 : be;
      o.x = fma(ab * mi, fma(rs, n.x, al * v.x), o.x);
      o.y = fma(ab * mi, fma(rs, n.y, al * v.y), o.y);
      if (!last) {
        const z_t vb = vbj[e], wp = wPrev[e];
        o.x = fma(-be, wp.x, fma(-al, fma(ib, vb.x, bb * mi * n.x), o.x));
        o.y = fma(-be, wp.y, fma(-al, fma(ib, vb.y, bb * mi * n.y), o.y));
      }
      if (l >= nC) {
        const int r = l - nC, g = r % nG;
        const double p = fma(A.E, A.x[g], A.V0[g]);
        o.x = fma(p, wv.x, o.x);
        o.y = fma(p, wv.y, o.y);
        // row gg of T at column g is T[2 band - d][gg]
        for (int d = max(0, band - g); d < min(nd, nG - g + band); d++) {
          const double cf = __ldg(A.T + (size_t)(nd - 1 - d) * nG + (g - band + d));
          const z_t q = wh[e + d];
          o.x = fma(cf, q.x, o.x);
          o.y = fma(cf, q.y, o.y);
        }
        gx = fma(A.x[g], fma(wv.x, v.x, wv.y * v.y), gx);
      }
      vbj[e] = o;
      wPrev[e] = wv;
      vbo[l] = o;
      s0 = fma(o.x, v.x, fma(o.y, v.y, s0));
      if (j > 0) {
        const z_t p = vj[l - nS];
        s1 = fma(o.x, p.x, fma(o.y, p.y, s1));
        s2 = fma(wv.x, p.x, fma(wv.y, p.y, s2));
      }
    }
    // block sums of s0, s1, s2 and, at the end, gx
    const double x = warp_sum4(s0, s1, s2, j == 0 ? gx : 0.0);
    if ((lane & 7) == 0) red[lane >> 3][wid] = x;
    __syncthreads();
    if (tid < 4) {
      double t = 0.0;
      for (int i = 0; i < W; i++) t += red[tid][i];
      mine[SIL_K + 4 * (j & 1) + tid] = zmk(t, 0.0);  // a slow block may still read the last order's
    }
    if (!(ok = barrier())) break;
    gather(SIL_K + 4 * (j & 1), 4);
    d1 = coef[0].x;
    e1 = coef[1].x;
    f1 = coef[2].x;
    __syncthreads();
  }
  if (ok) {
    const double nb = nbar - d1 / nrm;
    for (int e = tid; e < cnt; e += T) {
      const int l = l0 + e;
      const z_t v = A.k.V[l];
      A.sbar[l] = zadd(zscale(vbj[e], 1.0 / nrm), zscale(v, nb * A.m[l]));
    }
    if (rank == 0 && tid == 0 && A.grad) *A.grad += coef[3].x;
  }
  if (tid == 0 && A.nBlk > 1 && atomicAdd(A.bar + 1, 1u) == (unsigned)A.nBlk - 1) {
    A.bar[0] = 0u;
    A.bar[1] = 0u;
    __threadfence();
  }
}

}  // namespace

static const void* const sil_kernels[2][3] = {
    {(const void*)k_sil<256>, (const void*)k_sil<512>, (const void*)k_sil<1024>},
    {(const void*)k_sil<256, SIL_KEPT>, (const void*)k_sil<512, SIL_KEPT>, (const void*)k_sil<1024, SIL_KEPT>}};

// Shares the SMs out to the trajectories in proportion to their state sizes (at
// least one block each, none with less than SIL_MIN entries).  Left off where
// the trajectories outnumber the SMs, and not used for the propagation where a piece
// does not fit a block's shared memory: there the launch-per-pass form fills the chip.
void sil_init(cgpu_ctx* c) {
  c->silGroup = 0;
  if (c->method == CGPU_METHOD_TDCI || c->nb > c->numSms) return;
  std::vector<SilBlock> v;
  double total = 0.0;
  for (const SysHost& s : c->sys) total += s.nS;
  int left = c->numSms - c->nb;  // beyond the first block of each
  int cap = 0;
  for (int b = 0; b < c->nb; b++) {
    const int nS = c->sys[b].nS;
    const int want = (int)(nS / total * c->numSms);
    const int n = std::max(1, std::min({want, (nS + SIL_MIN - 1) / SIL_MIN, left + 1}));
    left -= n - 1;
    for (int r = 0; r < n; r++) v.push_back(SilBlock{b, r, n});
    cap = std::max(cap, (nS + n - 1) / n);
  }
  CODY_CUDA(cudaMalloc(&c->silBlk_d, sizeof(SilBlock) * v.size()));
  CODY_CUDA(cudaMemcpy(c->silBlk_d, v.data(), sizeof(SilBlock) * v.size(), cudaMemcpyHostToDevice));
  CODY_CUDA(cudaMalloc(&c->silPart_d, sizeof(z_t) * v.size() * 2 * SIL_PART));
  CODY_CUDA(cudaMalloc(&c->silBar_d, sizeof(unsigned) * 2 * c->nb));
  CODY_CUDA(cudaMemset(c->silBar_d, 0, sizeof(unsigned) * 2 * c->nb));
  for (const void* k : {sil_kernels[0][0], sil_kernels[0][1], sil_kernels[0][2], sil_kernels[1][0], sil_kernels[1][1],
                        sil_kernels[1][2], (const void*)k_sil_vjp<false>})
    CODY_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SIL_SMEM));
  c->silGroup = (int)v.size();
  c->silCap = cap;
  c->silFits = sil_smem(cap, c->band, SIL_K, false) <= SIL_SMEM;
}

void sil_check(cgpu_ctx* c) {
  if (c->flags_h && c->flags_h->err) throw std::string("SIL: a bounded wait between blocks expired");
}

void sil_free(cgpu_ctx* c) {
  for (void* p : {c->silBlk_d, (void*)c->silPart_d, (void*)c->silBar_d})
    if (p) cudaFree(p);
}

static SilArgs sil_args(cgpu_ctx* c, const z_t* start, z_t* state, double dt, int K) {
  SilArgs a;
  std::memset(&a, 0, sizeof(a));
  a.start = start;
  a.state = state;
  a.w0 = c->lw_d;
  a.w1 = c->work_d;
  a.basis = c->basis_d;
  a.ldv = c->nS;
  a.m = c->metric_d;
  a.T = c->T_d;
  a.V0 = c->V0_d;
  a.x = c->x_d;
  a.btOf = c->btOfOrb_d;
  a.blk = (const SilBlock*)c->silBlk_d;
  a.part = c->silPart_d;
  a.bar = c->silBar_d;
  a.tBase = c->zero_d;
  a.dt = a.dtSub = dt;
  a.K = K;
  a.window = c->krylovWindow;
  a.flags = c->flags_d;
  a.cap = c->silCap;
  a.smemV = sil_smem(c->silCap, c->band, K, true) <= SIL_SMEM;
  return a;
}

static void sil_launch(cgpu_ctx* c, SilArgs& a, int mode) {
  const int T = mode == SIL_SPILLED ? 1024 : 4 * c->silCap <= 256 ? 256 : a.smemV ? 512 : 1024;
  a.pt = T == 256 ? 4 : 1;
  void* args[] = {&a, (void*)&c->shape_d, (void*)&c->bs};
  const int i = T == 256 ? 0 : T == 512 ? 1 : 2;
  const void* kern = mode == SIL_SPILLED ? (const void*)k_sil<1024, SIL_SPILLED> : sil_kernels[mode][i];
  CODY_CUDA(cudaLaunchCooperativeKernel(kern, dim3(c->silGroup), dim3(T), args,
                                        mode == SIL_SPILLED ? 0 : sil_smem(c->silCap, c->band, a.K, a.smemV),
                                        c->stream));
  CODY_LAUNCHED(c);
}

// SIL on OrbsLin from t over dt on a state (all trajectories), in place.  With a tolerance
// it may leave some of dt: flags_h->left[place] holds, after a synchronisation, the time reached,
// what is left of dt, and the step and the halvings to go on with (dtSub, restarts).
void launch_sil(cgpu_ctx* c, z_t* state, double t, double dt, int K, double tol, int maxRestarts, double dtSub,
                int restarts, int place) {
  ProfScope prof(c, CGPU_KERNEL_LANCZOS);
  SilArgs a = sil_args(c, state, state, dt, K);
  a.m = c->metric_d;
  a.tBase = (c->inCapture || c->useStepTime) ? c->stepT_d : c->zero_d;
  a.tOff = c->inCapture ? t - c->captureT0 : t;
  a.tol = tol;
  a.dtSub = dtSub;
  a.restarts = restarts;
  a.place = place;
  a.maxRestarts = maxRestarts;
  sil_launch(c, a, SIL_STEP);
}

size_t sil_spill(const cgpu_ctx* c) {
  return c->silFits ? 0 : (size_t)c->silGroup * sil_entries(c->silCap, c->band, SIL_K, false);
}

// One fixed-order pass exp(-i dt h(E)) from start into out in the grid metric (a
// single system), keeping what its reverse needs.
void launch_sil_keep(cgpu_ctx* c, const z_t* start, z_t* out, double E, double dt, const SilKeep& k) {
  SilArgs a = sil_args(c, start, out, dt, k.K);
  a.m = c->metricW_d;
  a.window = 0;
  a.E = E;
  a.keep = k;
  if (!a.smemV) a.basis = k.V;
  sil_launch(c, a, k.spill ? SIL_SPILLED : SIL_KEPT);
}

// sbar may be obar; grad may be null.
void launch_sil_vjp(cgpu_ctx* c, const z_t* obar, z_t* sbar, double E, double dt, const SilKeep& k, double* grad) {
  SilVjpArgs a;
  a.k = k;
  a.obar = obar;
  a.m = c->metricW_d;
  a.T = c->T_d;
  a.V0 = c->V0_d;
  a.x = c->x_d;
  a.sbar = sbar;
  a.vb0 = c->lw_d;
  a.vb1 = c->work_d;
  a.grad = grad;
  a.E = E;
  a.dt = dt;
  a.part = c->silPart_d;
  a.bar = c->silBar_d;
  a.cap = c->silCap;
  a.nBlk = c->silGroup;
  a.flags = c->flags_d;
  void* args[] = {&a, (void*)&c->shape_d, (void*)&c->bs};
  const void* kern = k.spill ? (const void*)k_sil_vjp<true> : (const void*)k_sil_vjp<false>;
  CODY_CUDA(cudaLaunchCooperativeKernel(kern, dim3(c->silGroup), dim3(256), args,
                                        k.spill ? 0 : sil_smem(c->silCap, c->band, 0, false), c->stream));
  CODY_LAUNCHED(c);
}

__global__ void k_lz_expsub(double* __restrict__ lz, int mFixed, double dt, size_t bs) {
  __shared__ double jb[1216];
  lz = bat(lz, bs);
  int m = mFixed > 0 ? mFixed : (int)lz[CODY_LZ_MDIM];
  if (m > 32) m = 32;
  if (m < 1) return;
  double fr, fi;
  lz_expsub_warp<false>(lz, lz + CODY_LZ_BETA, m, dt, jb, fr, fi);
  const int lane = threadIdx.x;
  if (lane < m) {
    lz[CODY_LZ_PHI + 2 * lane] = fr;
    lz[CODY_LZ_PHI + 2 * lane + 1] = fi;
  }
  if (lane == m - 1)
    lz[CODY_LZ_ERR] = lz[CODY_LZ_BREAKJ] == (double)m ? 0.0 : lz[CODY_LZ_BETA + m - 1] * sqrt(fr * fr + fi * fi);
}

// EvaluateExpInSubspace on the scalar block of the launch-per-pass form.
void launch_lz_expsub(cgpu_ctx* c, int j, double dt) {
  k_lz_expsub<<<bgrid(c, 1), 32, 0, c->stream>>>(c->lz_d, j, dt, c->bs);
  CODY_LAUNCHED(c);
}
