// k_sil.cu -- a whole short-iterative-Lanczos integration of the one-body part
// in one launch (Integrate / PerformLanczosStep / EvaluateExpInSubspace,
// src/IntegratorList/Sil/S_IntegratorList_Sil.f90:114-310, on
// TimeDerivativeOrbsLin, S_Method_Mb_OrbBased_Mctdhx.f90:152-177).
//
// The launch-per-pass form (k_lanczos.cu) spends seven launches and five passes
// over the vectors on every Krylov iteration.  Here each trajectory has a group
// of blocks, every block owns a contiguous piece of its state vector, and an
// iteration is two phases between barriers of the group:
//   A  h = H v_j on the piece (halo of `band` points from the neighbours),
//      partials of the dots with the basis vectors and of ||h||^2;
//   B  h -= sum_k c_k v_k from the summed partials, ||.||^2 partials, h published
//      for the neighbours' next halo.
// v_{j+1} = h / beta_j is formed where it is read.  The piece, its metric and
// (where they fit) its basis vectors stay in shared memory.  Every block sums
// the same partials in the same order and evaluates exp(-i dt T) e1 itself, so
// all of them take the same decisions: second Gram-Schmidt pass, breakdown,
// convergence, halving of the step.  An adaptive integration therefore runs to
// its end without the host.
//
// FP64 throughout, also for the mixed forms: up to one group block per SM the
// FP64 pipe is not the bound of this kernel (44 to 100 FMA an entry and
// iteration): the barriers, the reductions and the chains of dependent FP64
// instructions are.  One half step of 2801 points x 16 orbitals, K = 16: 1330 us as
// launches, 460 here; 501 x 4, K = 12: 830 and 170.
//
// The groups' blocks wait on one another, so the launch is cooperative (at most
// one block per SM) and every wait is bounded.
#include <algorithm>

#include "common.cuh"

namespace {

constexpr int SIL_K = 32;
constexpr int SIL_MIN = 32;                    // smallest piece worth a block of its own
constexpr size_t SIL_SMEM = 200 * 1024;
constexpr long long SIL_WAIT = 4000000000LL;   // cycles after which a barrier gives up
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
__device__ void lz_expsub_warp(const double* alpha, const double* beta, int m, double dt, double* jb, double& fr,
                               double& fi) {
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
  const double c = 0.5 * (hi + lo), R = 0.5 * (hi - lo) * (1.0 + 1e-12) + 1e-300, z = fabs(dt) * R;
  int K = 1;  // last term of the series
  if (z >= 1e-300) {
    // log2 of (z/2)^n / n! below -64
    const float l2 = log2f((float)fmin(z, 1e30) * 0.5f);
    float lg = 0.0f;
    for (K = 1; K < KMAX; K++) {
      lg += l2 - log2f((float)K);
      if (lg < -64.0f && (float)K > (float)z) break;
    }
  }
  __syncwarp();
  if (z < 1e-300) {
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
  // 2 T' and the recurrence; a_k = 2 (-i)^k J_k: 1, -i, -1, i in turn
  const double iR = 2.0 / R, ta = (a - c) * iR, tl = bl * iR, tr = br * iR;
  double qm = lane == 0 ? 1.0 : 0.0, q;
  {
    const double ql = __shfl_up_sync(0xffffffffu, qm, 1), qr = __shfl_down_sync(0xffffffffu, qm, 1);
    q = 0.5 * fma(ta, qm, fma(tl, ql, tr * qr));
  }
  double pr = jb[0] * qm, pi = -jb[1] * q;
  for (int k = 2; k <= K; k++) {
    const double ql = __shfl_up_sync(0xffffffffu, q, 1), qr = __shfl_down_sync(0xffffffffu, q, 1);
    const double qn = fma(ta, q, fma(tl, ql, fma(tr, qr, -qm)));
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

namespace {

struct SilArgs {
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
  int maxRestarts;
  int* flags;      // host memory: [0] error, [1] warnings of trajectory 0
  int cap, smemV;  // entries of the largest piece; basis vectors in shared memory
  int pt;          // threads per entry (4 where the pieces leave most of the block idle, else 1)
};

// SIL_T threads a block: 256 for the small pieces (four threads an entry), whose
// iteration is a chain of latencies; 512 where the basis fits shared memory; 1024
// where it is read from L2 (10 helium steps 10.1 / 10.6 / 11.9 ms with 256 / 512 /
// 1024, 2801 x 16 points 462 / 414 / 488 us, a scan of 24 8.78 / 8.37 / 8.13 ms).
template <int SIL_T>
__global__ void __launch_bounds__(SIL_T, 1) k_sil(const SilArgs A, TRAJ_ARGS) {
  constexpr int SIL_W = SIL_T / 32;
  const SilBlock B = A.blk[blockIdx.x];
  const TrajShape& S = shp[B.traj];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nG = S.nG, band = S.band, nd = 2 * band + 1, nC = S.nC, cap = A.cap;
  z_t* state = batn(A.state, bs, B.traj);
  z_t* wb[2] = {batn(A.w0, bs, B.traj), batn(A.w1, bs, B.traj)};
  z_t* basis = batn(A.basis, bs, B.traj);
  const double* m = batn(A.m, bs, B.traj);
  const double* T = batn(A.T, bs, B.traj);
  const double* V0 = batn(A.V0, bs, B.traj);
  const double* x = batn(A.x, bs, B.traj);
  const int* btOf = batn(A.btOf, bs, B.traj);
  constexpr int PS = SIL_K + 2;
  z_t* part = A.part + (size_t)(blockIdx.x - B.rank) * PS;  // the group's partials
  z_t* mine = part + (size_t)B.rank * PS;
  unsigned* bar = A.bar + 2 * B.traj;
  unsigned target = 0;

  extern __shared__ z_t sm[];
  z_t* vt = sm;                          // v_j with its halo: entries l0 - band .. l1 + band
  z_t* w = vt + cap + 2 * band;
  z_t* mw = w + cap;                     // m w
  z_t* V = mw + cap;                     // [K][cap] when smemV
  __shared__ z_t coef[SIL_K + 1];
  __shared__ double alpha[SIL_K], beta[SIL_K], red[SIL_W], jb[1216], errEst, shE;
  __shared__ z_t phi[SIL_K];

  const int per = (S.nS + B.n - 1) / B.n, l0 = min(S.nS, B.rank * per), cnt = min(S.nS, l0 + per) - l0;
  auto vec = [&](int k, int e) -> z_t& { return A.smemV ? V[(size_t)k * cap + e] : basis[A.ldv * k + vidx(S, l0 + e)]; };
  auto barrier = [&]() {
    target += B.n;
    return group_barrier(bar, target, B.n, A.flags);
  };
  // sums over the group of partial slots [s0, s0 + n), one or two slots a warp, into coef[0..n)
  double* cf = reinterpret_cast<double*>(coef);
  auto gather = [&](int s0, int n) {
    if (n <= SIL_W) {
      if (wid < n) {
        double x0 = 0.0, y0 = 0.0;
        for (int b = lane; b < B.n; b += 32) {
          const z_t p = __ldcg(part + (size_t)b * PS + s0 + wid);
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
          const z_t* r = part + (size_t)b * PS + s0 + k;
          const z_t p = __ldcg(r), q = __ldcg(r + 1);  // slot k + 1 exists (PS slots a block)
          x0 += p.x;
          y0 += p.y;
          x1 += q.x;
          y1 += q.y;
        }
        const double x = warp_sum4(x0, y0, x1, y1);
        if ((lane & 7) == 0 && k + (lane >> 4) < n) cf[2 * k + (lane >> 3)] = x;
      }
    }
    __syncthreads();
  };
  // partials of <v_k, w>_m for k in [b0, b1) into slots 0..
  auto dots = [&](int b0, int b1) {
    double* out = reinterpret_cast<double*>(mine);
    if (b1 - b0 <= SIL_W) {
      const int k = b0 + wid;
      if (k < b1) {
        double ax = 0.0, ay = 0.0;
        for (int e = lane; e < cnt; e += 32) {
          const z_t v = vec(k, e), u = mw[e];
          ax = fma(v.x, u.x, fma(v.y, u.y, ax));
          ay = fma(v.x, u.y, fma(-v.y, u.x, ay));
        }
        const double x = warp_sum2(ax, ay);
        if ((lane & 15) == 0) out[2 * wid + (lane >> 4)] = x;
      }
    } else {
      for (int k = b0 + 2 * wid; k < b1; k += 2 * SIL_W) {
        double ax = 0.0, ay = 0.0, bx = 0.0, by = 0.0;
        const int k1 = min(k + 1, b1 - 1);
        for (int e = lane; e < cnt; e += 32) {
          const z_t v = vec(k, e), t = vec(k1, e), u = mw[e];
          ax = fma(v.x, u.x, fma(v.y, u.y, ax));
          ay = fma(v.x, u.y, fma(-v.y, u.x, ay));
          bx = fma(t.x, u.x, fma(t.y, u.y, bx));
          by = fma(t.x, u.y, fma(-t.y, u.x, by));
        }
        const double x = warp_sum4(ax, ay, bx, by);
        if ((lane & 7) == 0 && k + (lane >> 4) < b1) out[2 * (k - b0) + (lane >> 3)] = x;
      }
    }
  };
  // block sum of q into the real part of slot `slot` (warps to shared memory, then warp 0)
  auto publish = [&](double q, int slot) {
    q = warp_sum(q);
    if (lane == 0) red[wid] = q;
    __syncthreads();
    if (wid == 0) {
      double x = lane < SIL_W ? red[lane] : 0.0;
      for (int o = SIL_W / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if (lane == 0) mine[slot] = zmk(x, 0.0);
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
  // w -= sum coef_k v_{b0+k}; w published in out; its norm partial in the last slot
  auto subtract = [&](int b0, int n, z_t* out) {
    double q = 0.0;
    for (int eb = 0; eb < cnt; eb += eStep) {
      const int e = eb + e0;
      z_t r = zmk(0.0, 0.0);
      if (e < cnt) {
        if (eq == 0) r = w[e];
        for (int k = eq; k < n; k += pt) {
          const z_t v = vec(b0 + k, e), c = coef[k];
          r.x = fma(-c.x, v.x, fma(c.y, v.y, r.x));
          r.y = fma(-c.x, v.y, fma(-c.y, v.x, r.y));
        }
      }
      r = entry_sum(r);
      if (e < cnt && eq == 0) {
        const size_t i = vidx(S, l0 + e);
        const z_t u = zscale(r, m[i]);
        w[e] = r;
        mw[e] = u;
        out[i] = r;
        q = fma(u.x, r.x, fma(u.y, r.y, q));
      }
    }
    publish(q, SIL_K + 1);
  };

  double tCur = A.tOff, rem = A.dt;
  int warnings = 0;
  bool ok = true;
  while (ok && fabs(rem) > SIL_ZERO) {
    double dtS = rem;
    int restarts = 0;
    bool conv = false;
    // ||state||
    double q = 0.0;
    for (int e = tid; e < cnt; e += SIL_T) {
      const size_t i = vidx(S, l0 + e);
      const z_t v = state[i];
      q = fma(m[i], fma(v.x, v.x, v.y * v.y), q);
    }
    // the field takes a few microseconds of FP64 on one lane: beside the norm
    auto field = [&]() {
      if (tid == SIL_T - 1)
        shE = S.hasPot ? field_amplitude_dev(S.laser, *batn(A.tBase, bs, B.traj) + tCur + 0.5 * dtS) : 0.0;
    };
    field();
    publish(q, SIL_K + 1);
    if (!(ok = barrier())) break;
    gather(SIL_K + 1, 1);
    const double nrm = sqrt(coef[0].x);
    if (nrm <= SIL_ZERO) {  // nothing to propagate: the state stays
      conv = true;
    } else {
      for (;;) {
        if (restarts > 0) {
          __syncthreads();
          field();
          __syncthreads();
        }
        const double E = shE;
        double inv = 1.0 / nrm, bPrev = 0.0;
        const z_t* src = state;
        int mDim = A.K;
        for (int j = 1; j <= A.K; j++) {
          // v_j and its halo
          __syncthreads();
          for (int t = tid; t < cnt + 2 * band; t += SIL_T) {
            const int l = l0 - band + t;
            z_t v = zmk(0.0, 0.0);
            if (l >= 0 && l < S.nS) v = zscale(__ldcg(src + vidx(S, l)), inv);
            vt[t] = v;
            if (t >= band && t < band + cnt) vec(j - 1, t - band) = v;
          }
          __syncthreads();
          double h2 = 0.0;
          for (int eb = 0; eb < cnt; eb += eStep) {
            const int e = eb + e0, l = l0 + e;
            z_t h = zmk(0.0, 0.0);
            if (e < cnt && l >= nC) {  // the coefficients do not move
              const int r = l - nC, i = r / nG, g = r - i * nG;
              const double* Tb = T + (size_t)(S.restricted ? 0 : btOf[i]) * nd * nG + g;
              const z_t* vv = vt + e;
              const int d0 = max(0, band - g), d1 = min(nd, nG - g + band);  // inside the orbital
              for (int d = eq; d < d1; d += pt) {
                if (d < d0) continue;
                const double cf = __ldg(Tb + (size_t)d * nG);
                h.x = fma(cf, vv[d].x, h.x);
                h.y = fma(cf, vv[d].y, h.y);
              }
              if (S.hasPot && eq == pt - 1) {
                const double p = fma(E, x[g], V0[g]);
                h.x = fma(p, vv[band].x, h.x);
                h.y = fma(p, vv[band].y, h.y);
              }
            }
            if (e < cnt && eq == 0 && A.window == 1 && j > 1) {  // three-term recurrence
              const z_t v = vec(j - 2, e);
              h.x = fma(-bPrev, v.x, h.x);
              h.y = fma(-bPrev, v.y, h.y);
            }
            h = entry_sum(h);
            if (e < cnt && eq == 0) {
              const z_t u = zscale(h, m[vidx(S, l)]);
              w[e] = h;
              mw[e] = u;
              h2 = fma(u.x, h.x, fma(u.y, h.y, h2));
            }
          }
          const int b0 = A.window > 0 ? max(0, j - A.window) : 0, nv = j - b0;
          publish(h2, nv);  // also orders mw before the dots
          dots(b0, j);
          if (!(ok = barrier())) break;
          gather(0, nv + 1);
          const double a = coef[nv - 1].x, n0 = coef[nv].x;
          if (A.window == 1) {
            __syncthreads();
            if (tid == 0) coef[0].y = 0.0;
            __syncthreads();
          }
          subtract(b0, nv, wb[j & 1]);
          if (!(ok = barrier())) break;
          gather(SIL_K + 1, 1);
          double n1 = coef[0].x;
          if (n1 <= SIL_ETA2 * n0) {  // most of h cancelled: project once more
            __syncthreads();
            dots(b0, j);
            if (!(ok = barrier())) break;
            gather(0, nv);
            subtract(b0, nv, wb[j & 1]);
            if (!(ok = barrier())) break;
            gather(SIL_K + 1, 1);
            n1 = coef[0].x;
          }
          const double be = sqrt(n1);
          if (tid == 0) {
            alpha[j - 1] = a;
            beta[j - 1] = be;
          }
          const bool broke = be <= SIL_ZERO;
          const bool last = broke || j == A.K;
          if (A.tol > 0.0 || last) {
            __syncthreads();
            if (wid == 0) {
              double fr, fi;
              lz_expsub_warp(alpha, beta, j, dtS, jb, fr, fi);
              if (lane < j) phi[lane] = zmk(fr, fi);
              if (lane == j - 1) errEst = broke ? 0.0 : be * sqrt(fr * fr + fi * fi);
            }
            __syncthreads();
            conv = errEst <= A.tol;
            if ((A.tol > 0.0 && conv) || last) {
              mDim = j;
              break;
            }
          }
          src = wb[j & 1];
          inv = 1.0 / be;
          bPrev = be;
        }
        if (!ok) break;
        if (conv || !(A.tol > 0.0) || fabs(dtS) <= SIL_ZERO || restarts >= A.maxRestarts) {
          for (int e = tid; e < cnt; e += SIL_T) {
            z_t acc = zmk(0.0, 0.0);
            for (int k = 0; k < mDim; k++) zfma(acc, vec(k, e), phi[k]);
            state[vidx(S, l0 + e)] = zscale(acc, nrm);
          }
          break;
        }
        dtS = 0.5 * dtS;
        restarts++;
      }
    }
    if (!ok) break;
    if (!conv) warnings++;
    if (!(A.tol > 0.0)) break;  // fixed order: one pass over the whole step
    tCur += dtS;
    rem -= dtS;
  }
  if (tid == 0) {
    if (B.traj == 0 && B.rank == 0) A.flags[1] = A.tol > 0.0 ? warnings : 1;
    if (B.n > 1 && atomicAdd(bar + 1, 1u) == (unsigned)B.n - 1) {
      bar[0] = 0u;
      bar[1] = 0u;
      __threadfence();
    }
  }
}

size_t sil_smem(int cap, int band, int K, bool smemV) {
  return sizeof(z_t) * ((size_t)cap * (3 + (smemV ? K : 0)) + 2 * band);
}

}  // namespace

// Shares the SMs out to the trajectories in proportion to their state sizes (at
// least one block each, none with less than SIL_MIN entries).  Left off where
// the trajectories outnumber the SMs or a piece would not fit a block's shared
// memory: there the launch-per-pass form fills the chip.
void sil_init(cgpu_ctx* c) {
  c->silBlocks = 0;
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
  if (sil_smem(cap, c->band, 0, false) > SIL_SMEM) return;
  CODY_CUDA(cudaMalloc(&c->silBlk_d, sizeof(SilBlock) * v.size()));
  CODY_CUDA(cudaMemcpy(c->silBlk_d, v.data(), sizeof(SilBlock) * v.size(), cudaMemcpyHostToDevice));
  CODY_CUDA(cudaMalloc(&c->silPart_d, sizeof(z_t) * v.size() * (SIL_K + 2)));
  CODY_CUDA(cudaMalloc(&c->silBar_d, sizeof(unsigned) * 2 * c->nb));
  CODY_CUDA(cudaMemset(c->silBar_d, 0, sizeof(unsigned) * 2 * c->nb));
  for (const void* k : {(const void*)k_sil<256>, (const void*)k_sil<512>, (const void*)k_sil<1024>})
    CODY_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SIL_SMEM));
  c->silBlocks = (int)v.size();
  c->silCap = cap;
}

void sil_free(cgpu_ctx* c) {
  for (void* p : {c->silBlk_d, (void*)c->silPart_d, (void*)c->silBar_d})
    if (p) cudaFree(p);
}

// SIL on OrbsLin from t over dt on a state (all trajectories), in place.
void launch_sil(cgpu_ctx* c, z_t* state, double t, double dt, int K, double tol, int maxRestarts) {
  ProfScope prof(c, CGPU_KERNEL_LANCZOS);
  SilArgs a;
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
  a.tBase = (c->inCapture || c->useStepTime) ? c->stepT_d : c->zero_d;
  a.tOff = c->inCapture ? t - c->captureT0 : t;
  a.dt = dt;
  a.K = K;
  a.window = c->krylovWindow;
  a.tol = tol;
  a.maxRestarts = maxRestarts;
  a.flags = c->flags_d;
  a.cap = c->silCap;
  a.smemV = sil_smem(c->silCap, c->band, K, true) <= SIL_SMEM;
  const int T = 4 * c->silCap <= 256 ? 256 : a.smemV ? 512 : 1024;
  a.pt = T == 256 ? 4 : 1;
  void* args[] = {&a, (void*)&c->shape_d, (void*)&c->bs};
  const void* kern = T == 256 ? (const void*)k_sil<256> : T == 512 ? (const void*)k_sil<512> : (const void*)k_sil<1024>;
  CODY_CUDA(cudaLaunchCooperativeKernel(kern, dim3(c->silBlocks), dim3(T), args,
                                        sil_smem(c->silCap, c->band, K, a.smemV), c->stream));
  CODY_LAUNCHED(c);
}

__global__ void k_lz_expsub(double* __restrict__ lz, int mFixed, double dt, size_t bs) {
  __shared__ double jb[1216];
  lz = bat(lz, bs);
  int m = mFixed > 0 ? mFixed : (int)lz[CODY_LZ_MDIM];
  if (m > 32) m = 32;
  if (m < 1) return;
  double fr, fi;
  lz_expsub_warp(lz, lz + CODY_LZ_BETA, m, dt, jb, fr, fi);
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
