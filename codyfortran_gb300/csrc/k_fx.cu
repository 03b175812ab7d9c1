// k_fx.cu -- fixed-point split GEMM on tcgen05 tensor cores (the FP64 and the
// mixed_fx forms of the contractions of ApplyCorrelationOp and FillH2,
// src/Method/Mb/OrbBased/S_Method_Mb_OrbBased.f90:227-329, 647-872).
//
// An FP64 operand row x[0..K) is carried as L slices of base-256 digits under
// one power of two per row:
//     x[k] ~= 2^e sum_{i<L} d_i[k] 2^(-8(i+1)),   max_k |x[k]| < 2^(e-1),
//     |d_i| <= 128 (bf16 holds them exactly),
// i.e. x rounded to 8L - 1 fractional bits of its row maximum.  The product of
// an A row and a B row splits into levels l = i + j:
//     C = 2^(ea + eb) sum_l 2^(-8(l+2)) D_l,   D_l = sum_{i+j=l} sum_k a_i[k] b_j[k].
// Each level has its own FP32 accumulator in tensor memory (L accumulators of
// nT columns), fed by the slice products of that level.  A slice product is an
// integer of magnitude <= 2^14, so over a chunk of K a level sum of l + 1 products
// stays below (l + 1) K 2^14: exact in FP32 up to 2^24.  K = 256 in the mixed forms:
// the four leading levels whatever the operands, the others unless the digits of both
// rows are near their extremes with one sign (a few units of level 4, 2^-43 of the rows'
// maxima, then).  K = 128 in the FP64 form: eight levels whatever the operands, and the
// ninth lies below what is kept.  After every chunk the epilogue adds the level sums to
// 64-bit integers, so C is the product of the truncated operands whatever the summation
// order.  Levels l >= L are not formed; with the operand truncation (2^-8L of each row
// maximum) they bound the error at about 2^-8L max|a| max|b| sqrt(K).
//
// L = 4 to 6 serve the mixed_fx / mixed_fx6 forms (their Z operands with
// max_k |x[k]| < 2^e, |d_0| <= 256: one bit more, K <= 256).  L = 8 and 9 are the FP64
// form (fx_slices_fp64 in ctx.cu: how many, and why that is no less than FP64 sums keep):
// the FP64 pipe of this GPU does two FMA a cycle and SM (1.2 TFLOP/s), 36 slice products
// on the tensor cores about 45 TFLOP/s of the same contraction, and the sum of a row
// rounds once instead of K times.
//
// Pipeline: one TMA producer thread, one MMA issuer thread, eight epilogue
// warps (two per tensor-memory lane quarter).  Per 64-wide K block the producer
// loads the L slices of the B tile (only the rows of the tile's own nT columns,
// slice after slice) into one ring stage and the L slices of the A tile into L
// stages of a second ring.  A TMA instruction costs its thread about 100 cycles
// (measured: 16 KB per stage in one box 5.8 TB/s over all SMs, in eight boxes
// 3.1), so the B group is one instruction: a 4D box of 64 columns, nT rows, L
// slices, from the map made for that nT (in 16-row boxes, W = V S of the
// 512-trajectory batch in the 39-bit form 2.48 ms, this way 2.25).
//
// The B slices of a stage are consecutive rows of one operand (slice j at row
// j nT), and level l's accumulator sits at tensor-memory column l nT, so the
// products of A slice i with the B slices 0..L-1-i are ONE product with an N of
// (L - i) nT columns landing on the columns from i nT on.  The issuer runs it
// as one or two MMAs of up to 256 columns.  An MMA of N columns takes
// max(N / 2, 32 + N / 4) cycles (it reads 4 KB of A and 32 N bytes of B from
// shared memory at 128 bytes a cycle; tests/mma_rate.cu), so per-slice MMAs of
// N = 80 run at 77% of the pipe's rate and those of 128 and more at all of it;
// there are also 2.3 times fewer of them to issue (six 6-bit slices, N = 80,
// W = V S of the 512-trajectory batch: 4.13 ms with one MMA per slice pair,
// 2.52 this way).
//
// The epilogue adds the accumulators of a chunk to integers in registers and
// hands the tensor memory back; scaling and stores follow the tile's last
// chunk.  Tiles with L nT <= half the tensor-memory columns alternate between
// the two halves, so that the next chunk's MMAs run during the drain; wider
// ones wait for it (about 1.5 k of 13 k cycles, of 9 k in the FP64 form).  The wide configuration (two B
// stages, deep A ring) holds one CTA per SM; the compact one (one B stage, L A
// stages, <= 256 TMEM columns) two.  Every wait is bounded: on expiry the
// kernel sets an error flag, drains its copies, frees its tensor memory and
// returns.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "tc.cuh"

// B operand [nb][rowsMax][L][pitch] as 4D maps (column, row, slice, trajectory)
// with boxes of 64 columns, 16 (i + 1) rows and all L slices.
FxMaps fx_make_maps(const cgpu_ctx* c, const __nv_bfloat16* base, int rowsMax, int pitch, int L) {
  FxMaps f;
  for (int i = 0; i < FX_MAPS; i++) {
    const unsigned long long dims[4] = {(unsigned long long)pitch, (unsigned long long)rowsMax, (unsigned long long)L,
                                        (unsigned long long)c->nb};
    const unsigned long long strides[3] = {(unsigned long long)pitch * L * 2, (unsigned long long)pitch * 2,
                                           c->nb > 1 ? c->bs : (unsigned long long)pitch * L * 2 * rowsMax};
    const unsigned box[4] = {tcdev::TC_BK, 16u * (i + 1), (unsigned)L, 1};
    f.m[i] = tc_encode_map(base, 4, dims, strides, box);
  }
  return f;
}

namespace {

using namespace tcdev;

constexpr int FX_SMEM_MAX = 232448;

// 64-wide K blocks per accumulation in tensor memory: K = 256, in the FP64 form 128
__host__ __device__ constexpr int fx_chunk(int L) { return L > 6 ? 2 : 4; }

template <int BN, int L, int NA_, int NB_>
struct FxCfg {
  static constexpr int A_BYTES = TC_BM * TC_BK * 2;
  static constexpr int B_BYTES = BN * TC_BK * 2;
  static constexpr int BG_BYTES = L * B_BYTES;
  static constexpr int NB = NB_;
  // NA_ == 0: as many A stages as fit (at most 8)
  static constexpr int NA = NA_ > 0 ? NA_ : std::min(8, (FX_SMEM_MAX - 2048 - NB * BG_BYTES) / A_BYTES);
  static constexpr int RING = NA * A_BYTES + NB * BG_BYTES;
  static constexpr int SMEM = RING + 1024;
  static constexpr uint32_t TMEM_COLS = (L * BN) <= 32 ? 32 : (L * BN) <= 64 ? 64 : (L * BN) <= 128 ? 128
                                        : (L * BN) <= 256 ? 256 : 512;
  static_assert(L * BN <= 512, "tensor memory holds 512 columns");
  static_assert(BN % 16 == 0 && BN >= 16 && BN <= 16 * FX_MAPS, "N tile: multiple of 16 with a B map");
  static_assert(NA >= 2, "A ring");
  static_assert(SMEM + 2048 <= FX_SMEM_MAX, "shared memory");
};

// The level sums of one output over its chunks as integers: T = sum_l D_l
// 256^(L-1-l).  L <= 5 fits 64 bits (|D_0| <= 2^22 a chunk: below 2^63 for 512
// chunks, which fx_min_splits keeps); longer ones are held as hi 256^(L - LH) + lo
// (L = 9: lo of five levels of at most 9 2^21 a chunk is below 2^56 a chunk, 2^63 for 128).
template <int L>
struct FxAcc {
  static constexpr int LH = L <= 5 ? L : L == 6 ? 3 : 4;  // levels in hi
  long long hi, lo;
  __device__ __forceinline__ void clear() { hi = lo = 0; }
  // levels [l0, l0 + n) of column j
  template <int N, int CB>
  __device__ __forceinline__ void add(const uint32_t (&d)[N][CB], int j, int l0, int n) {
#pragma unroll
    for (int i = 0; i < N; i++) {
      if (i >= n) break;
      const int l = l0 + i, v = __float2int_rn(__uint_as_float(d[i][j]));
      const int sh = 8 * (l < LH ? LH - 1 - l : L - 1 - l);
      const long long t = sh > 24 ? (long long)((unsigned long long)(long long)v << sh)
                                  : (long long)v * (1 << (sh > 24 ? 0 : sh));
      if (l < LH) hi += t;
      else lo += t;
    }
  }
  __device__ __forceinline__ double value(int e) const;  // T 2^e
};

// ldexp out of line: results outside the normal range (the epilogue is unrolled
// over a warp's columns, and its instructions have to stay in the cache).
__device__ __noinline__ double ll_scaled_far(long long T, int e) { return ldexp((double)T, e); }

__device__ __noinline__ double ldexp_far(double v, int e) { return ldexp(v, e); }

// v 2^e, exponent arithmetic on the bits where the result is normal.
__device__ __forceinline__ double d_scaled(double v, int e) {
  if (v == 0.0) return 0.0;
  const int be = ((__double2hiint(v) >> 20) & 0x7FF) + e;
  if (be <= 0 || be >= 2047) return ldexp_far(v, e);
  return __hiloint2double(__double2hiint(v) + (e << 20), __double2loint(v));
}

// T 2^e as a double by integer operations (the FP64 pipes are the scarce
// resource): round-to-nearest-even when |T| needs more than 53 bits.
__device__ __forceinline__ double ll_scaled(long long T, int e) {
  const unsigned long long sign = (unsigned long long)T & 0x8000000000000000ull;
  unsigned long long a = T < 0 ? (unsigned long long)(-T) : (unsigned long long)T;
  if (a == 0) return 0.0;
  const int lz = __clzll((long long)a);
  a <<= lz;
  const unsigned rem = (unsigned)a & 0x7FFu;
  a >>= 11;  // 53 bits; a rounding carry runs on into the exponent
  a += (rem > 0x400u || (rem == 0x400u && (a & 1ull))) ? 1ull : 0ull;
  const int be = e - lz + 1086;  // biased exponent of a 2^(e - lz + 11)
  if (be <= 0 || be >= 2046) return ll_scaled_far(T, e);
  return __longlong_as_double((long long)(sign | (((unsigned long long)(be - 1) << 52) + a)));
}

template <int L>
__device__ __forceinline__ double FxAcc<L>::value(int e) const {
  // hi is exact as a double (below 2^46 a chunk), lo too unless its top levels add up to a
  // million times the last one, so the fma is the one rounding that counts
  if constexpr (L > 5) return d_scaled(fma((double)hi, (double)(1ll << (8 * (L - LH))), (double)lo), e);
  else return ll_scaled(hi, e);
}

// One work item of a persistent CTA: trajectory, first output row, first
// output column and column count (a multiple of 16), K split.
struct FxTile {
  int traj, m0, n0, nT, split;
};

// out[traj][split][M][N] = C (FP64) over the tile list; a persistent CTA takes
// tiles blockIdx.x, blockIdx.x + gridDim.x, ...  Warps 0..EW-1: epilogue (TMEM
// lanes 32(w%4)..32(w%4)+31, column batches of CB); warp EW: TMA producer;
// warp EW+1: MMA issuer.  The rings and their phases run on across tiles, so
// the producer loads the next tile while the epilogue drains the current one.
// One accumulator phase per chunk, numbered over the CTA's life: phase p signals
// accFull[p % 2] (MMA -> epilogue) and accEmpty[p % 2] (epilogue -> MMA) and uses
// the tensor-memory half p % 2 if its tile fits one.  Its MMAs wait for the
// drain of phase p - 2 (same half), and of p - 1 too where either tile needs
// both halves.  K splits: a trajectory of segTiles K blocks takes
// ceil(segTiles / kPer) balanced splits; the tiles of the list beyond them
// write zero partials.  maxRow/maxCol (unsplit K only): the largest biased
// exponent of |C| per output row / column.  A row or column whose exponent is
// FX_EXP_NAN (an operand with an infinity or a NaN) gives NaN.
// aShared: A is shared by the trajectories (3D map with one plane per root
// grid); the trajectory's rows start at vRow of plane vRoot, its K range at
// vRow - gShift, its row exponents at expA[vExp].
template <int BN, int L, int NA_, int NB_, int EW>
__global__ void __launch_bounds__(32 * (EW + 2), NA_ > 0 ? 2 : 1)
    k_fx_gemm(const __grid_constant__ CUtensorMap tA, const __grid_constant__ FxMaps tB, double* __restrict__ out,
              const int* __restrict__ expA, const int* __restrict__ expB, unsigned* __restrict__ maxRow,
              unsigned* __restrict__ maxCol, TRAJ_ARGS, int gemmId, int segPitchA, int aShared, int kPer,
              const FxTile* __restrict__ tiles, int nTiles, int* __restrict__ err, const int* __restrict__ colScale) {
  using C = FxCfg<BN, L, NA_, NB_>;
  constexpr int NA = C::NA, NB = C::NB, CB = 8, CH = fx_chunk(L);
  static_assert(EW % 4 == 0 && BN % CB == 0, "epilogue warps / column batch");
  constexpr int NBAT = (BN / CB + EW / 4 - 1) / (EW / 4);  // column batches of one epilogue warp
  constexpr uint32_t HALF = C::TMEM_COLS / 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* ringA = smem;
  uint8_t* ringB = smem + NA * C::A_BYTES;
  __shared__ __align__(8) uint64_t aFull[NA], aEmpty[NA], bFull[NB], bEmpty[NB], accFull[2], accEmpty[2], finalBar;
  __shared__ uint32_t tmemSlot;
  __shared__ volatile int abortFlag;
  __shared__ int consumedA, consumedB, issuedA, issuedB;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    abortFlag = 0;
    consumedA = consumedB = issuedA = issuedB = 0;
    for (int s = 0; s < NA; s++) {
      mbar_init(&aFull[s], 1);
      mbar_init(&aEmpty[s], 1);
    }
    for (int s = 0; s < NB; s++) {
      mbar_init(&bFull[s], 1);
      mbar_init(&bEmpty[s], 1);
    }
    for (int s = 0; s < 2; s++) {
      mbar_init(&accFull[s], 1);
      mbar_init(&accEmpty[s], EW);
    }
    mbar_init(&finalBar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmemSlot)),
                 "r"(C::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmemSlot;

  // per-tile geometry (every role derives the same values)
  auto geometry = [&](const FxTile& tl, int& M, int& N, int& kt0, int& nk) {
    int segTiles;
    tc_dims(shp[tl.traj], gemmId, M, N, segTiles);
    const int sT = max(1, (segTiles + kPer - 1) / kPer);  // this trajectory's splits
    const int per = (segTiles + sT - 1) / sT;              // <= kPer
    kt0 = tl.split * per;
    nk = tl.split < sT ? max(0, min(segTiles, kt0 + per) - kt0) : 0;
  };

  if (warp == EW) {
    if (lane == 0) {
      // TMA producer: per K block the L B slices of the tile's rows, then the L A slices
      int ta = 0, tb = 0;
      for (int t = blockIdx.x; t < nTiles && !abortFlag; t += gridDim.x) {
        const FxTile tl = tiles[t];
        int M, N, kt0, nk;
        geometry(tl, M, N, kt0, nk);
        const TrajShape& T = shp[tl.traj];
        const int aRow0 = aShared ? T.vRow : 0, aCol0 = aShared ? T.vRow - T.gShift : 0;
        const int aZ = aShared ? T.vRoot : tl.traj;
        for (int kb = 0; kb < nk && !abortFlag; kb++) {
          const int sb = tb % NB, rb = tb / NB;
          if (!mbar_wait(&bEmpty[sb], (rb & 1) ^ 1, &abortFlag)) {
            abortFlag = 1;
            atomicExch(err, 11);
            break;
          }
          const int x0 = (kt0 + kb) * TC_BK;
          mbar_expect_tx(&bFull[sb], (uint32_t)(L * tl.nT * TC_BK * 2));
          tma_load_4d(ringB + sb * C::BG_BYTES, &tB.m[tl.nT / 16 - 1], &bFull[sb], x0, tl.n0, 0, tl.traj);
          tb++;
          issuedB = tb;
          for (int i = 0; i < L; i++) {
            const int sa = ta % NA, ra = ta / NA;
            if (!mbar_wait(&aEmpty[sa], (ra & 1) ^ 1, &abortFlag)) {
              abortFlag = 1;
              atomicExch(err, 12);
              break;
            }
            mbar_expect_tx(&aFull[sa], C::A_BYTES);
            tma_load_3d(ringA + sa * C::A_BYTES, &tA, &aFull[sa], i * segPitchA + aCol0 + x0, aRow0 + tl.m0, aZ);
            ta++;
            issuedA = ta;
          }
        }
      }
    }
  } else if (warp == EW + 1) {
    if (lane == 0) {
      // MMA issuer: kind::f16, D=F32, A=B=BF16, K-major, M=128; descriptors
      // advance by address / 16: +2 per 16-wide K step, +8 per B row
      const uint64_t bdesc0 = sw128_desc(smem_u32(ringB));
      const uint64_t adesc0 = sw128_desc(smem_u32(ringA));
      int ca = 0, cb = 0, ph = 0;  // ph: accumulator phases (chunks)
      bool prevNarrow = true, ok = true;
      for (int t = blockIdx.x; t < nTiles && !abortFlag && ok; t += gridDim.x) {
        const FxTile tl = tiles[t];
        int M, N, kt0, nk;
        geometry(tl, M, N, kt0, nk);
        if (nk == 0) continue;  // the epilogue writes the empty split's zeros
        const bool narrow = (uint32_t)(L * tl.nT) <= HALF;
        // A slice i covers (L - i) nT columns: one MMA up to 256 of them, else two halves
        uint32_t id0[L], id1[L], half[L];
#pragma unroll
        for (int i = 0; i < L; i++) {
          const int cols = (L - i) * tl.nT;
          const int n0 = cols <= 256 ? cols : (cols / 2 + 15) / 16 * 16;
          const uint32_t base = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TC_BM >> 4) << 24);
          half[i] = (uint32_t)n0;
          id0[i] = base | ((uint32_t)(n0 >> 3) << 17);
          id1[i] = cols > n0 ? base | ((uint32_t)((cols - n0) >> 3) << 17) : 0u;
        }
        for (int kb = 0; kb < nk && ok; kb++) {
          const bool first = kb % CH == 0;
          if (first) {  // a new phase: its half (or both) drained by the epilogue
            if ((ph > 1 && !mbar_wait(&accEmpty[ph & 1], ((ph >> 1) - 1) & 1, &abortFlag)) ||
                (ph > 0 && !(narrow && prevNarrow) &&
                 !mbar_wait(&accEmpty[(ph - 1) & 1], ((ph - 1) >> 1) & 1, &abortFlag))) {
              abortFlag = 1;
              atomicExch(err, 16);
              ok = false;
              break;
            }
            prevNarrow = narrow;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          }
          const int sb = cb % NB, rb = cb / NB;
          if (!mbar_wait(&bFull[sb], rb & 1, &abortFlag)) {
            abortFlag = 1;
            atomicExch(err, 13);
            ok = false;
            break;
          }
          cb++;
          consumedB = cb;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t bd = bdesc0 + (uint64_t)((sb * C::BG_BYTES) >> 4);
          const uint32_t tcol = tmem + (narrow && (ph & 1) ? HALF : 0u);
#pragma unroll
          for (int i = 0; i < L; i++) {
            const int sa = ca % NA, ra = ca / NA;
            if (!mbar_wait(&aFull[sa], ra & 1, &abortFlag)) {
              abortFlag = 1;
              atomicExch(err, 14);
              ok = false;
              break;
            }
            ca++;
            consumedA = ca;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t ad = adesc0 + (uint64_t)((sa * C::A_BYTES) >> 4);
            const uint32_t d0 = tcol + (uint32_t)(i * tl.nT), d1 = d0 + half[i];
            const uint64_t bd1 = bd + 8 * half[i];
            if (id1[i]) {
              // both halves of a K step read the same 4 KB of A: the second from the collector
#pragma unroll
              for (int k = 0; k < TC_BK / 16; k++) {
                const uint32_t acc = (!first || i > 0 || k > 0) ? 1u : 0u;
                umma_bf16_coll(1, d0, ad + 2 * k, bd + 2 * k, id0[i], acc);
                umma_bf16_coll(3, d1, ad + 2 * k, bd1 + 2 * k, id1[i], acc);
              }
            } else {
#pragma unroll
              for (int k = 0; k < TC_BK / 16; k++)
                umma_bf16(d0, ad + 2 * k, bd + 2 * k, id0[i], (!first || i > 0 || k > 0) ? 1u : 0u);
            }
            umma_commit(&aEmpty[sa]);
          }
          if (!ok) break;
          umma_commit(&bEmpty[sb]);
          if (kb % CH == CH - 1 || kb == nk - 1) {
            umma_commit(&accFull[ph & 1]);
            ph++;
          }
        }
      }
      umma_commit(&finalBar);  // arrives when every issued MMA has completed
    }
  } else {
    // epilogue: warp w owns TMEM lanes [32q, 32q+32) = tile rows, q = w % 4
    // (the lane quarter a warp may access), and every (EW/4)-th batch of CB
    // columns starting at batch w / 4
    const int q = warp & 3, cg = warp >> 2;
    int ph = 0;
    for (int t = blockIdx.x; t < nTiles; t += gridDim.x) {
      const FxTile tl = tiles[t];
      int M, N, kt0, nk;
      geometry(tl, M, N, kt0, nk);
      double* Oz = batn(out, bs, tl.traj) + (size_t)tl.split * (size_t)M * N;
      const int r = q * 32 + lane, row = tl.m0 + r;
      const bool rowOk = row < M;
      if (nk == 0) {  // empty split: its partial is zero
        if (rowOk && cg == 0)
          for (int col = tl.n0; col < min(N, tl.n0 + tl.nT); col++) Oz[(size_t)row * N + col] = 0.0;
        continue;
      }
      const bool narrow = (uint32_t)(L * tl.nT) <= HALF;
      FxAcc<L> T[NBAT][CB];  // the level sums of this warp's columns
#pragma unroll
      for (int bt = 0; bt < NBAT; bt++)
#pragma unroll
        for (int j = 0; j < CB; j++) T[bt][j].clear();
      bool waited = true;
      for (int k0 = 0; k0 < nk; k0 += CH) {
        waited = mbar_wait(&accFull[ph & 1], (ph >> 1) & 1, &abortFlag);
        if (__any_sync(0xffffffffu, !waited)) {
          waited = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tcol = tmem + ((uint32_t)(q * 32) << 16) + (narrow && (ph & 1) ? HALF : 0u);
#pragma unroll
        for (int bt = 0; bt < NBAT; bt++) {
          const int c = (cg + bt * (EW / 4)) * CB;
          if (c < tl.nT) {
            // registers for one group of levels at a time
            constexpr int G = L <= 5 ? L : L == 6 ? 3 : 4;
#pragma unroll
            for (int l0 = 0; l0 < L; l0 += G) {
              uint32_t d[G][CB];
#pragma unroll
              for (int l = 0; l < G; l++)
                if (l0 + l < L) TMEM_LD_X8(tcol + (uint32_t)((l0 + l) * tl.nT + c), d[l]);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int j = 0; j < CB; j++) T[bt][j].add(d, j, l0, L - l0);
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&accEmpty[ph & 1]);
        ph++;
      }
      if (!waited) {
        if (lane == 0) atomicExch(err, 15);
        break;
      }
      const TrajShape& S = shp[tl.traj];
      const int* eA = aShared ? expA + S.vExp : batn(expA, bs, tl.traj);
      const int* eB = batn(expB, bs, tl.traj);
      const int ea = rowOk ? eA[row] - 8 * (L + 1) : 0;
      unsigned rowMaxEx = 0;
#pragma unroll
      for (int bt = 0; bt < NBAT; bt++) {
        const int c = (cg + bt * (EW / 4)) * CB;
        if (c < tl.nT) {
          double v[CB];
#pragma unroll
          for (int j = 0; j < CB; j++) {
            const int col = tl.n0 + c + j;
            unsigned ex = 0;
            v[j] = 0.0;
            if (rowOk && col < N) {
              const int e = ea + eB[col];
              v[j] = T[bt][j].value(e);
              if (e > FX_EXP_NAN / 2) v[j] = __longlong_as_double(0x7FF8000000000000LL);
              ex = (unsigned)(__double2hiint(v[j]) >> 20) & 0x7FFu;
              // the FP64 form: the row's maximum over the scaled columns (fx_scale_key)
              if (L > 6 && colScale) rowMaxEx = max(rowMaxEx, fx_scale_key(ex, -batn(colScale, bs, tl.traj)[col]));
              else rowMaxEx = max(rowMaxEx, ex);
            }
            if (maxCol) {
              unsigned m = __reduce_max_sync(0xffffffffu, ex);
              if (lane == 0 && m) atomicMax(batn(maxCol, bs, tl.traj) + col, m);
            }
          }
          if (rowOk) {
            double* dst = Oz + (size_t)row * N + tl.n0 + c;
#pragma unroll
            for (int j = 0; j < CB; j += 2)
              if (tl.n0 + c + j < N) *reinterpret_cast<double2*>(dst + j) = make_double2(v[j], v[j + 1]);
          }
        }
      }
      if (maxRow && rowOk && rowMaxEx) atomicMax(batn(maxRow, bs, tl.traj) + row, rowMaxEx);
    }
  }
  __syncthreads();
  // every issued MMA has completed before the tensor memory is freed; after an
  // abort also the TMA copies that were issued but never consumed (bounded waits)
  if (warp == EW && lane == 0) {
    volatile int dummy = 0;
    mbar_wait(&finalBar, 0, &dummy);
    if (abortFlag) {
      for (int t = consumedA; t < issuedA; t++) mbar_wait(&aFull[t % NA], (t / NA) & 1, &dummy);
      for (int t = consumedB; t < issuedB; t++) mbar_wait(&bFull[t % NB], (t / NB) & 1, &dummy);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::TMEM_COLS) : "memory");
}

template <int BN, int L, int NA_, int NB_>
void launch_fx_t(cgpu_ctx* c, const CUtensorMap& ta, const FxMaps& tb, double* out, const int* expA,
                 const int* expB, unsigned* maxRow, unsigned* maxCol, int gemmId, int segPitchA, int aShared, int kPer,
                 const FxTile* tiles, int nTiles, int ctasPerSm, int* err, const int* colScale) {
  using C = FxCfg<BN, L, NA_, NB_>;
  // eight epilogue warps (two per tensor-memory lane quarter); sixteen for L >
  // 5, whose two 64-bit sums per output would not fit the registers of eight
  constexpr int EW = L > 5 ? 16 : 8;
  auto kern = k_fx_gemm<BN, L, NA_, NB_, EW>;
  static bool attr = false;
  if (!attr) {
    CODY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
    attr = true;
  }
  if (nTiles <= 0) return;
  const int grid = std::min(nTiles, c->numSms * ctasPerSm);
  kern<<<grid, 32 * (EW + 2), C::SMEM, c->stream>>>(ta, tb, out, expA, expB, maxRow, maxCol, TRAJ_PASS(c), gemmId,
                                                    segPitchA, aShared, kPer, tiles, nTiles, err, colScale);
  CODY_LAUNCHED(c);
}

}  // namespace

// The instantiated N tiles (fx_gemm's cases): L accumulators of BN columns in
// 512 (wide) or 256 (compact, two CTAs per SM) tensor-memory columns.
struct FxTileCfg {
  int bn, L;
  bool compact;
};
static const FxTileCfg kFxTiles[] = {{32, 4, false}, {64, 4, false}, {96, 4, false},
                                     {32, 5, false}, {64, 5, false}, {80, 5, false}, {96, 5, false},
                                     {32, 6, false}, {64, 6, false}, {64, 8, false}, {48, 9, false}, {32, 4, true}, {64, 4, true},
                                     {32, 5, true},  {48, 5, true}};

static int fx_max_bn(int L, bool compact) {
  int m = 0;
  for (const FxTileCfg& t : kFxTiles)
    if (t.L == L && t.compact == compact) m = std::max(m, t.bn);
  return m;
}

bool fx_compact_ok(int L) { return fx_max_bn(L, true) > 0; }

void fx_tile_configs(int L, std::vector<std::pair<int, bool>>& out) {
  out.clear();
  for (const FxTileCfg& t : kFxTiles)
    if (t.L == L) out.push_back({t.bn, t.compact});
}

bool fx_tile_supported(int bn, int L, bool compact) {
  for (const FxTileCfg& t : kFxTiles)
    if (t.bn == bn && t.L == L && t.compact == compact) return true;
  return false;
}

// 512 chunks (K = 131072), in the FP64 form 128 (K = 16384), keep the integer level sums
// inside 64 bits.
int fx_min_splits(int kTiles, int L) {
  const int most = (L > 6 ? 128 : 512) * fx_chunk(L);
  return std::max(1, (kTiles + most - 1) / most);
}

int fx_normalize_splits(int kTiles, int s) {
  s = std::max(1, std::min(s, kTiles));
  const int per = (kTiles + s - 1) / s;
  return (kTiles + per - 1) / per;
}

int fx_tile_n(int N, int L, bool compact) {
  const int maxBn = fx_max_bn(L, compact);
  if (maxBn == 0) throw std::string("fx_tile_n: no configuration for this slice count");
  const int tiles = (N + maxBn - 1) / maxBn;
  const int want = ((N + tiles - 1) / tiles + 15) / 16 * 16;  // balanced tiles
  int best = maxBn;
  for (const FxTileCfg& t : kFxTiles)
    if (t.L == L && t.compact == compact && t.bn >= want && t.bn < best) best = t.bn;
  return best;
}

// K splits of one GEMM over the context's trajectories.  A batch of more tiles
// than SMs takes none.  Otherwise the cheapest by this estimate in SM cycles:
// waves of tiles, each its K blocks at the MMA rate (4 K steps of L (L + 1) / 2
// slice products of N / 2 cycles) plus about 8000 to fill the pipeline, drain
// and store; a split adds its FP64 partials, written and read at about 3 KB a
// cycle, and (reduceExtra) a reduction kernel of about 6000.
int fx_split_count(int M, int N, int BN, int L, int kTiles, int nb, bool reduceExtra) {
  const int nt = (N + BN - 1) / BN, nT = ((N + nt - 1) / nt + 15) / 16 * 16;
  const long tiles = (long)((M + TC_BM - 1) / TC_BM) * nt * nb;
  const int lo = fx_min_splits(kTiles, L);
  if (tiles >= 152) return fx_normalize_splits(kTiles, lo);
  int best = lo;
  double bestCost = 1e300;
  for (int s = lo; s <= std::max(lo, kTiles / 2); s++) {
    const int per = (kTiles + s - 1) / s;
    if ((kTiles + per - 1) / per != s) continue;
    const double wave = (double)((tiles * s + 151) / 152);
    double cost = wave * (per * 2.0 * L * (L + 1) / 2 * nT * 1.2 + 8000.0);
    if (s > 1) cost += (reduceExtra ? 6000.0 : 0.0) + 16.0 * s * M * N * nb / 3000.0;
    if (cost < bestCost) {
      bestCost = cost;
      best = s;
    }
  }
  return fx_normalize_splits(kTiles, best);
}

// The columns of a trajectory go to ceil(N / bn) tiles of equal width (to 16
// columns): a full tile and a narrow remainder would take the same MMA columns
// but issue the remainder's in short MMAs.  The tiles are sorted by their work
// (K blocks times columns), largest first, so that the CTAs, which take every
// gridDim-th tile, end together; tiles of one trajectory stay neighbours.
void* fx_build_tiles(cgpu_ctx* c, int gemmId, int bn, int nSplit, int* nTiles) {
  std::vector<FxTile> v;
  std::vector<std::pair<long, int>> order;  // (work of the widest tile, trajectory)
  for (int b = 0; b < c->nb; b++) {
    const TrajShape& S = c->shape_h[b];
    const int kTiles = gemmId == TC_GEMM_Z ? S.Kp / TC_BK : S.Kg / TC_BK;
    const int units = ceil_div(gemmId == TC_GEMM_Z ? 2 * S.nOS * S.nOS : 2 * S.nPairs, 16);
    const int nt = ceil_div(units, bn / 16);
    order.push_back({-(long)kTiles * ceil_div(units, nt), b});
  }
  std::stable_sort(order.begin(), order.end());
  for (const auto& o : order) {
    const int b = o.second;
    const TrajShape& S = c->shape_h[b];
    int P2 = 2 * S.nPairs, Q2 = 2 * S.nOS * S.nOS, M, N;
    if (gemmId == TC_GEMM_W) { M = S.nG; N = P2; }
    else if (gemmId == TC_GEMM_Z) { M = S.nG; N = Q2; }
    else { M = P2; N = P2; }
    const int units = ceil_div(N, 16), nt = ceil_div(units, bn / 16);
    for (int m0 = 0; m0 < M; m0 += TC_BM)
      for (int z = 0; z < nSplit; z++)
        for (int k = 0, u = 0; k < nt; k++) {
          const int w = units / nt + (k < units % nt ? 1 : 0);
          v.push_back(FxTile{b, m0, 16 * u, 16 * w, z});
          u += w;
        }
  }
  *nTiles = (int)v.size();
  void* d = nullptr;
  CODY_CUDA(cudaMalloc(&d, sizeof(FxTile) * std::max<size_t>(v.size(), 1)));
  if (!v.empty()) CODY_CUDA(cudaMemcpy(d, v.data(), sizeof(FxTile) * v.size(), cudaMemcpyHostToDevice));
  return d;
}

void fx_gemm(cgpu_ctx* c, int L, bool compact, int gemmId, const CUtensorMap& ta, const FxMaps& tb, int bn,
             double* out, const int* expA, const int* expB, unsigned* maxRow, unsigned* maxCol, int segPitchA,
             int segPitch, int aShared, int nSplit, const void* tiles, int nTiles, int* err, const int* colScale) {
  if (segPitch % TC_BK != 0 || segPitchA % TC_BK != 0)
    throw std::string("fx_gemm: segment pitch must be a multiple of 64");
  if (nSplit > 1 && (maxRow || maxCol)) throw std::string("fx_gemm: output maxima need an unsplit K");
  const int kTiles = segPitch / TC_BK, kPer = (kTiles + nSplit - 1) / nSplit;  // K blocks per split
  if (nSplit < fx_min_splits(kTiles, L)) throw std::string("fx_gemm: K split beyond the range of the level sums");
  const FxTile* tl = (const FxTile*)tiles;
#define FX_CASE(BN_, L_, NA_, NB_, CMP_)                                                                        \
  if (bn == BN_ && L == L_ && compact == CMP_) {                                                                \
    launch_fx_t<BN_, L_, NA_, NB_>(c, ta, tb, out, expA, expB, maxRow, maxCol, gemmId, segPitchA, aShared,     \
                                   kPer, tl, nTiles, CMP_ ? 2 : 1, err, colScale);                    \
    return;                                                                                                     \
  }
  FX_CASE(32, 4, 0, 2, false) FX_CASE(64, 4, 0, 2, false) FX_CASE(96, 4, 0, 2, false)
  FX_CASE(32, 5, 0, 2, false) FX_CASE(64, 5, 0, 2, false) FX_CASE(80, 5, 0, 2, false) FX_CASE(96, 5, 0, 2, false)
  FX_CASE(32, 6, 0, 2, false) FX_CASE(64, 6, 0, 2, false) FX_CASE(64, 8, 0, 2, false)
  FX_CASE(48, 9, 0, 2, false)
  FX_CASE(32, 4, 4, 1, true) FX_CASE(64, 4, 4, 1, true)
  FX_CASE(32, 5, 5, 1, true) FX_CASE(48, 5, 5, 1, true)
#undef FX_CASE
  throw std::string("fx_gemm: unsupported tile");
}
