// core_f64_ns.cu -- FP64 plain form of letkf_core without an eigendecomposition, for k <= 64.
//
// One CTA of 128 threads per grid point.  The quantities are those of
// common/common_letkf.f90:50-243: with
// A = hdxb^T R^-1 hdxb + (k-1)/rho I, T = sqrt((k-1) A^-1) (the symmetric
// square root), Pa = A^-1 and wbar = Pa hdxb^T R^-1 dep.  They are reached as
//   1. the Gram matrix in FP64, lower 8 x 8 blocks only, rows staged by
//      cp.async two chunks deep;
//   2. Z ~ (A/s)^(-1/2) in FP32 by the spectrum-scaled coupled Newton-Schulz
//      iteration (mixed_core.cuh describes it), a starting value only;
//   3. Newton's method for Z (A/s) Z = I: the residual R = I - Z (A/s) Z is
//      formed to more than FP32 (pairs of floats the first time, FP64
//      afterwards), and the correction D of the linearised equation
//      M D + D M = R, M = (A/s)^(1/2) ~ (A/s) Z, is solved in FP32 by the sign
//      iteration of [[M, R], [0, -M]] (its (1,2) block tends to 2 D; the part
//      of an error that does not commute with A, which a plain Newton-Schulz
//      step leaves standing or enlarges, is solved for as well).  A correction
//      takes the residual r to about max(1e-5 r, r^2): 1e-5 -> 1e-10 -> FP64
//      rounding, two residuals for lambda_max / c up to about 100, three above.
// The last residual is always FP64 against the FP64 A: FP32 decides how fast
// the result is reached.  The correction of at most 5e-10 that follows it is not
// checked by another; measured against quadruple precision the result is no
// further off than the eigensolver's at any conditioning (k = 40, geometric means
// over 32 points, eigensolver / here: T 2.7e-16 / 2.8e-17 at lambda_max / c = 2,
// 2.2e-15 / 6.9e-16 at 345, 9.8e-14 / 2.5e-14 at 8,400; wbar 7.1e-16 / 2.4e-16,
// 8.7e-15 / 5.0e-15, 1.3e-13 / 1.3e-13).
//
// Bound: the FP64 pipe, 1.2 TFLOP/s on this chip against 75 in FP32, with a
// 64-cycle latency.  The EISPACK form (core_f64.cu) walks its rotations on one
// thread's scalar chain (a division takes 440 cycles, a square root 690); here
// the FP64 work is L k^2 / 2 + 1.5 k^3 multiply-adds, all independent.  A warp
// instruction holds a sub-partition's FP64 unit for 64 cycles, so operands
// come straight from shared memory and one warp per sub-partition keeps it
// busy; the FP32 phases of one CTA overlap the FP64 phases of the others on
// the SM.  Measured: 8,640 regional points of k = 64 (mean list about 300)
// 183 -> 26 ms (FP64 pipe 69 % busy); 32,256 SPEEDY-grid points of k = 40 (mean
// list 86) 233 -> 21 ms (23 with FP32 products over the 48 columns of the tiles,
// not the 40 members; FP64 pipe 59 %, FP32 28 %); with every residual in
// FP64 a tenth more; a 40-point ring of k = 20, one point per SM, 1.43 -> 0.1.
//
// A point is left to core_f64.cu (status LETKF_PENDING until its launch) where
// mtx_eigen's truncation or the conditioning could matter (c <= 0, or
// s / c >= 1e5 where s >= lambda_max), or where the iteration does not reach
// its residual.
#include <math.h>

#include <type_traits>

#include "letkf_common.cuh"

namespace letkf {

constexpr int FN_NT = 128;

template <int NP>
struct FnCfg {
  // FP32 product tile of a thread: TR consecutive rows, TC columns; the lanes' fast index runs along the
  // columns, so a warp reads and writes consecutive words of a row
  static constexpr int TR = NP / 8, TC = NP / 16;
  static constexpr int CH = NP >= 32 ? 16 : 8;            // observations per staged chunk
  static constexpr int NB = NP / 8;                       // 8 x 8 blocks a side
  static constexpr int MAXL = (NB * (NB + 1) / 2 + 3) / 4;  // lower blocks of a warp
  static constexpr int MAXF = (NB * NB + 3) / 4;            // blocks of a warp, full matrix
  // and the fewest for the ensembles this width serves (NB - 1 blocks a side; a warp may have none at 16)
  static constexpr int MINL = NP == 16 ? 1 : NB * (NB - 1) / 2 / 4, MINF = NP == 16 ? 1 : (NB - 1) * (NB - 1) / 4;
  // CTAs an SM holds: three FP64 matrices each (96, 54, 24, 6 KB)
  static constexpr int MINB = NP == 64 ? 2 : NP == 48 ? 4 : NP == 32 ? 6 : 8;
  // doubles after the matrices: b, wbar, scratch, four partial b, two chunks' weights / departures / rloc, reductions
  static constexpr int TAIL = 7 * NP + 6 * CH + 64;
  static constexpr size_t BYTES = sizeof(double) * (3 * (size_t)NP * NP + TAIL);
};

template <int N>
__device__ __forceinline__ void fn_ld(const float* p, float (&v)[N]) {
  if constexpr (N % 4 == 0) {
#pragma unroll
    for (int q = 0; q < N; q += 4) {
      const float4 t = *reinterpret_cast<const float4*>(p + q);
      v[q] = t.x;
      v[q + 1] = t.y;
      v[q + 2] = t.z;
      v[q + 3] = t.w;
    }
  } else if constexpr (N % 2 == 0) {
#pragma unroll
    for (int q = 0; q < N; q += 2) {
      const float2 t = *reinterpret_cast<const float2*>(p + q);
      v[q] = t.x;
      v[q + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int q = 0; q < N; q++) v[q] = p[q];
  }
}

// column of element b of a thread's tile, tx = threadIdx.x % 16
template <int NP>
__device__ __forceinline__ int fn_col(int tx, int b) {
  constexpr int TC = FnCfg<NP>::TC;
  return TC == 3 ? 16 * b + tx : TC * tx + b;
}

template <int NP>
__device__ __forceinline__ void fn_ldc(const float* p, int tx, float (&v)[FnCfg<NP>::TC]) {
  if constexpr (FnCfg<NP>::TC == 3) {
#pragma unroll
    for (int b = 0; b < 3; b++) v[b] = p[16 * b + tx];
  } else {
    fn_ld<FnCfg<NP>::TC>(p + FnCfg<NP>::TC * tx, v);
  }
}

// acc = X^T Yb for this thread's tile (X symmetric, or its transpose is meant),
// over k < n8: the padding's rows and columns of both are zero off its diagonal,
// so that it leaves the ensemble's part alone, and its own values are not used
template <int NP>
__device__ __forceinline__ void fn_gemm(const float* X, const float* Yb, int n8, int i0, int tx,
                                        float (&acc)[FnCfg<NP>::TR][FnCfg<NP>::TC]) {
  using C = FnCfg<NP>;
#pragma unroll
  for (int a = 0; a < C::TR; a++)
#pragma unroll
    for (int b = 0; b < C::TC; b++) acc[a][b] = 0.f;
#pragma unroll 4
  for (int k = 0; k < n8; k++) {
    float av[C::TR], bv[C::TC];
    fn_ld<C::TR>(X + k * NP + i0, av);
    fn_ldc<NP>(Yb + k * NP, tx, bv);
#pragma unroll
    for (int a = 0; a < C::TR; a++)
#pragma unroll
      for (int b = 0; b < C::TC; b++) acc[a][b] = fmaf(av[a], bv[b], acc[a][b]);
  }
}

// Row and column block of block `id` of the lower triangle (row by row)
__device__ __forceinline__ int2 fn_lower(int id) {
  int bi = 0;
  while (id > bi) {
    id -= bi + 1;
    bi++;
  }
  return make_int2(bi, id);
}

// acc[b] += X^T Yb over k < n8 on M 8 x 8 blocks (a lane has row lane / 4 and
// the two columns 2 (lane % 4) of each)
template <int NP, int M, int N>
__device__ __forceinline__ void fn_product(const double* X, const double* Yb, int n8, const int (&xo)[N],
                                           const int (&yo)[N], double (&acc)[N][2]) {
#pragma unroll(M <= 8 ? 2 : 1)
  for (int k = 0; k < n8; k++) {
    const double* xk = X + k * NP;
    const double* yk = Yb + k * NP;
#pragma unroll
    for (int b = 0; b < M; b++) {
      const double a = xk[xo[b]];
      const double2 y = *reinterpret_cast<const double2*>(yk + yo[b]);
      acc[b][0] = fma(a, y.x, acc[b][0]);
      acc[b][1] = fma(a, y.y, acc[b][1]);
    }
  }
}

// f(std::integral_constant<int, m>) for this warp's block count, LO .. N: one
// loop per count, because a multiply-add that is only predicated off still
// takes its FP64 slot (k = 40 in the 48-wide kernel: 4 of 6 blocks are real)
template <int N, int LO, typename F>
__device__ __forceinline__ void fn_counted(int m, F&& f) {
  if constexpr (N >= LO) {
    if (m == N)
      f(std::integral_constant<int, N>());
    else
      fn_counted<N - 1, LO>(m, f);
  }
}

// Coupled Newton-Schulz in FP32 from Y = A/s, Z = I (spectrum of ZY in
// [lo, 1]); false when it does not converge.  T = Z Y, Y <- Y (3I - aT), Z <-
// (3I - aT) Z: with the other order in the Z update (T^T) rounding errors that
// do not commute with A grow (measured: residual 1e-2 instead of 1e-6 at
// lambda_max / c = 100), so T is also kept transposed, in TT.
template <int NP>
__device__ bool fn_newton_schulz(float* Y, float* Z, float* T, float* TT, float* redf, int n8, float lo) {
  using C = FnCfg<NP>;
  const int tid = threadIdx.x, i0 = (tid >> 4) * C::TR, tx = tid & 15;
  float acc[C::TR][C::TC], yn[C::TR][C::TC];
  float prev = INFINITY;
  for (int it = 0; it < 24; it++) {
    fn_gemm<NP>(Z, Y, n8, i0, tx, acc);
    float e2 = 0.f;
#pragma unroll
    for (int a = 0; a < C::TR; a++)
#pragma unroll
      for (int b = 0; b < C::TC; b++) {
        T[(i0 + a) * NP + fn_col<NP>(tx, b)] = acc[a][b];
        TT[fn_col<NP>(tx, b) * NP + i0 + a] = acc[a][b];
        const float d = acc[a][b] - (i0 + a == fn_col<NP>(tx, b) ? 1.f : 0.f);
        if (i0 + a < n8 && fn_col<NP>(tx, b) < n8) e2 = fmaf(d, d, e2);
      }
    e2 = block_sum<float, FN_NT>(e2, redf);  // publishes T
    if (!isfinite(e2)) return false;
    const float al = ns_scale(lo), sa = sqrtf(al);
    const float ka = 1.5f * sa, kb = 0.5f * al * sa;
    lo = f_ns(al * lo);
    fn_gemm<NP>(Y, T, n8, i0, tx, acc);
#pragma unroll
    for (int a = 0; a < C::TR; a++)
#pragma unroll
      for (int b = 0; b < C::TC; b++) yn[a][b] = ka * Y[(i0 + a) * NP + fn_col<NP>(tx, b)] - kb * acc[a][b];
    fn_gemm<NP>(TT, Z, n8, i0, tx, acc);
#pragma unroll
    for (int a = 0; a < C::TR; a++)
#pragma unroll
      for (int b = 0; b < C::TC; b++) acc[a][b] = ka * Z[(i0 + a) * NP + fn_col<NP>(tx, b)] - kb * acc[a][b];
    __syncthreads();
#pragma unroll
    for (int a = 0; a < C::TR; a++)
#pragma unroll
      for (int b = 0; b < C::TC; b++) {
        Y[(i0 + a) * NP + fn_col<NP>(tx, b)] = yn[a][b];
        Z[(i0 + a) * NP + fn_col<NP>(tx, b)] = acc[a][b];
      }
    __syncthreads();
    // converged, or at the FP32 floor of this spectrum (Newton's method takes it from there)
    if (e2 < 1.0e-8f || (e2 < 1.0e-3f && e2 > 0.25f * prev)) return true;
    prev = e2;
  }
  return false;
}

// Sign iteration of [[Y, R], [0, -Y]] in FP32, spectrum of Y^2 in [lo, 1]:
// Y tends to I and R to 2 D with Y0 D + D Y0 = R0.  Scaled steps as in the
// Newton-Schulz iteration (the eigenvalue map of Y^2 is the same).
template <int NP>
__device__ void fn_sign(float* Y, float* Y2, float* R, float* U, int n8, float lo) {
  using C = FnCfg<NP>;
  const int tid = threadIdx.x, i0 = (tid >> 4) * C::TR, tx = tid & 15;
  float acc[C::TR][C::TC], yn[C::TR][C::TC], rn[C::TR][C::TC];
  for (int it = 0; it < 20; it++) {
    const bool last = lo > 0.999f;
    fn_gemm<NP>(Y, Y, n8, i0, tx, acc);
#pragma unroll
    for (int a = 0; a < C::TR; a++)
#pragma unroll
      for (int b = 0; b < C::TC; b++) Y2[(i0 + a) * NP + fn_col<NP>(tx, b)] = acc[a][b];
    fn_gemm<NP>(R, Y, n8, i0, tx, acc);
#pragma unroll
    for (int a = 0; a < C::TR; a++)
#pragma unroll
      for (int b = 0; b < C::TC; b++) U[(i0 + a) * NP + fn_col<NP>(tx, b)] = acc[a][b];
    __syncthreads();
    const float al = ns_scale(lo), sa = sqrtf(al);
    const float ka = 1.5f * sa, kb = 0.5f * al * sa;
    lo = f_ns(al * lo);
    if (!last) {
      fn_gemm<NP>(Y, Y2, n8, i0, tx, acc);
#pragma unroll
      for (int a = 0; a < C::TR; a++)
#pragma unroll
        for (int b = 0; b < C::TC; b++) yn[a][b] = ka * Y[(i0 + a) * NP + fn_col<NP>(tx, b)] - kb * acc[a][b];
    }
    fn_gemm<NP>(Y, U, n8, i0, tx, acc);  // Y R Y
#pragma unroll
    for (int a = 0; a < C::TR; a++)
#pragma unroll
      for (int b = 0; b < C::TC; b++) rn[a][b] = ka * R[(i0 + a) * NP + fn_col<NP>(tx, b)] + kb * acc[a][b];
    fn_gemm<NP>(Y2, R, n8, i0, tx, acc);  // Y^2 R; R Y^2 is its transpose
    __syncthreads();
#pragma unroll
    for (int a = 0; a < C::TR; a++)
#pragma unroll
      for (int b = 0; b < C::TC; b++) {
        U[(i0 + a) * NP + fn_col<NP>(tx, b)] = acc[a][b];
        if (!last) Y[(i0 + a) * NP + fn_col<NP>(tx, b)] = yn[a][b];
      }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < C::TC; b++) {
      float m[C::TR];
      fn_ld<C::TR>(U + fn_col<NP>(tx, b) * NP + i0, m);
#pragma unroll
      for (int a = 0; a < C::TR; a++) R[(i0 + a) * NP + fn_col<NP>(tx, b)] = rn[a][b] - kb * (acc[a][b] + m[a]);
    }
    __syncthreads();
    if (last) return;
  }
}

// (hi, lo) += a z in pairs of floats, a = (x, y) with |y| < ulp(x) / 2.  hi
// carries an offset that keeps its exponent fixed, so the part of the product
// it cannot hold is r exactly (three operations where a general two-sum takes
// six); lo collects those parts and the product's own rounding error.
__device__ __forceinline__ void fn_df_mac(float& hi, float& lo, float2 a, float z) {
  const float p = __fmul_rn(a.x, z);
  const float e = fmaf(a.y, z, fmaf(a.x, z, -p));
  const float t = __fadd_rn(hi, p);
  const float r = __fsub_rn(p, __fsub_rn(t, hi));
  hi = t;
  lo = __fadd_rn(lo, __fadd_rn(r, e));
}

// the pair's value, offset removed, as a normalised pair
__device__ __forceinline__ float2 fn_df_value(float hi, float lo, float offset) {
  const float h = __fsub_rn(hi, offset);
  const float v = __fadd_rn(h, lo);
  return make_float2(v, __fsub_rn(lo, __fsub_rn(v, h)));
}

__device__ __forceinline__ void fn_cp8(double* dst, const double* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}

template <int NP>
__global__ void __launch_bounds__(FN_NT, FnCfg<NP>::MINB) core_f64_ns_kernel(
    int n, int npts, const int64_t* __restrict__ offs, const double* __restrict__ rows,
    const double* __restrict__ rdiag, const double* __restrict__ rloc, const double* __restrict__ dep,
    double* parm_infl, double* trans, double* transm, double* pao, int rdiag_wloc, double minfl, int* status) {
  using C = FnCfg<NP>;
  constexpr int Q = NP * NP, CH = C::CH, MAXL = C::MAXL, MAXF = C::MAXF, MINL = C::MINL, MINF = C::MINF;
  extern __shared__ __align__(16) double sm[];
  double* A = sm;           // A; in the sign iteration Y, Y^2 (FP32)
  double* Z = sm + Q;       // FP32 Z, T, then FP64 Z; with P: the staged rows
  double* P = sm + 2 * Q;   // FP32 Y; (A/s) Z; in the sign iteration R, R Y (FP32)
  double* bv = sm + 3 * Q;  // NP
  double* e = bv + NP;      // NP wbar
  double* g = e + NP;       // NP
  double* bw = g + NP;      // 4 NP partial b of the warps
  double* wts = bw + 4 * NP;  // CH weight, CH departure, CH rloc (two chunks)
  double* red = wts + 6 * CH;
  float* redf = reinterpret_cast<float*>(red + 32);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int li = lane >> 2, lj = 2 * (lane & 3);
  const int nb = (n + 7) / 8, n8 = 8 * nb;
  // this warp's lower blocks: offsets of its row and column lanes
  const int nlow = nb * (nb + 1) / 2, mine = nlow > wid ? (nlow - wid + 3) / 4 : 0;
  int xo[MAXL], yo[MAXL];
#pragma unroll
  for (int b = 0; b < MAXL; b++) {
    const int2 q = b < mine ? fn_lower(wid + 4 * b) : make_int2(0, 0);
    xo[b] = 8 * q.x + li;
    yo[b] = 8 * q.y + lj;
  }
  const int nful = nb * nb, minef = nful > wid ? (nful - wid + 3) / 4 : 0;

  // one point per CTA (the launch's grid), handed out by the hardware
  for (int p = blockIdx.x; p < npts; p += gridDim.x) {
    const int64_t r0 = offs[p];
    const int L = (int)(offs[p + 1] - r0);
    double infl = parm_infl[p];
    double* T = trans + (size_t)p * n * n;
    if (L == 0) {  // common_letkf.f90:82-96
      const double sq = sqrt(infl);
      for (int idx = tid; idx < n * n; idx += FN_NT) {
        const int j = idx / n, i = idx - j * n;
        T[idx] = (i == j) ? sq : 0.0;
        if (pao) pao[(size_t)p * n * n + idx] = (i == j) ? infl / (double)(n - 1) : 0.0;
      }
      if (transm)
        for (int i = tid; i < n; i += FN_NT) transm[(size_t)p * n + i] = 0.0;
      if (tid == 0) status[p] = LETKF_OK;
      __syncthreads();
      continue;
    }
    if (minfl > 0.0 && infl < minfl) infl = minfl;
    const double c = (double)(n - 1) * (1.0 / infl);
    bool ok = c > 0.0;

    // ---- 1. Gram (lower blocks), b = hdxb_rinv^T dep, inflation sums ----
    double* Yw = Z;                   // CH x NP weighted rows
    double* Yc = Z + CH * NP;         // two chunks of CH x NP rows
    for (int i = tid; i < Q; i += FN_NT) A[i] = 0.0;
    for (int i = tid; i < 3 * CH * NP; i += FN_NT) Z[i] = 0.0;  // columns n .. NP-1 stay zero
    __syncthreads();
    double acc[MAXL][2];
#pragma unroll
    for (int b = 0; b < MAXL; b++) acc[b][0] = acc[b][1] = 0.0;
    constexpr int BPL = (NP + 31) / 32;
    double bacc[BPL];
#pragma unroll
    for (int q = 0; q < BPL; q++) bacc[q] = 0.0;
    double p1 = 0.0, p3 = 0.0;
    auto stage = [&](int c0, int buf) {
      const int nr = min(CH, L - c0);
      const double* src = rows + (size_t)(r0 + c0) * n;
      double* dst = Yc + buf * CH * NP;
      for (int t = tid; t < nr * n; t += FN_NT) {
        const int r = t / n;
        fn_cp8(dst + r * NP + (t - r * n), src + t);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (tid < nr) {
        const double rd = rdiag[r0 + c0 + tid], rl = rloc[r0 + c0 + tid];
        double* w = wts + buf * 3 * CH;
        w[tid] = rdiag_wloc ? 1.0 / rd : rl / rd;
        w[CH + tid] = dep[r0 + c0 + tid];
        w[2 * CH + tid] = rl;
      }
    };
    stage(0, 0);
    for (int c0 = 0, buf = 0; c0 < L; c0 += CH, buf ^= 1) {
      const int nr = min(CH, L - c0);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      if (c0 + CH < L) stage(c0 + CH, buf ^ 1);
      const double* y = Yc + buf * CH * NP;
      const double* w = wts + buf * 3 * CH;
      for (int t = tid; t < nr * NP; t += FN_NT) Yw[t] = y[t] * w[t / NP];
      if (tid < nr) {
        const double d = w[CH + tid];
        p1 = p1 + d * d * w[tid];
        p3 = p3 + w[2 * CH + tid];
      }
      __syncthreads();
      fn_counted<MAXL, MINL>(mine, [&](auto m) { fn_product<NP, decltype(m)::value>(Yw, y, nr, xo, yo, acc); });
      for (int r = wid; r < nr; r += 4) {
        const double d = w[CH + r];
#pragma unroll
        for (int q = 0; q < BPL; q++) bacc[q] = fma(Yw[r * NP + (lane + 32 * q) % NP], d, bacc[q]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < MAXL; b++)
      if (b < mine) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
          A[xo[b] * NP + yo[b] + q] = acc[b][q];
          A[(yo[b] + q) * NP + xo[b]] = acc[b][q];
        }
      }
#pragma unroll
    for (int q = 0; q < BPL; q++)
      if (lane + 32 * q < NP) bw[wid * NP + lane + 32 * q] = bacc[q];
    __syncthreads();
    double tr = 0.0;
    for (int i = tid; i < n; i += FN_NT) tr += A[i * NP + i];
    double sums[3] = {tr, p1, p3};
    block_sum_k<double, FN_NT, 3>(sums, red);
    tr = sums[0];
    for (int i = tid; i < NP; i += FN_NT) {
      A[i * NP + i] += c;
      bv[i] = (bw[i] + bw[NP + i]) + (bw[2 * NP + i] + bw[3 * NP + i]);
    }
    __syncthreads();

    // ---- 2. FP32 start: s = min(Gershgorin, Frobenius) >= lambda_max ----
    // A is kept in the point's output matrix while the sign iteration uses its place
    float* Y32 = reinterpret_cast<float*>(P);
    float* Z32 = reinterpret_cast<float*>(Z);
    float* T32 = Z32 + Q;
    const double trA = tr + (double)NP * c;  // of the padded matrix
    const float itr = (float)(1.0 / trA);
    for (int idx = tid; idx < Q; idx += FN_NT) {
      const int i = idx / NP, j = idx - i * NP;
      const double a = A[idx];
      if (i < n && j < n) T[i * n + j] = a;
      Y32[idx] = (float)a * itr;  // conversions share the FP64 pipe: one per element
      Z32[idx] = i == j ? 1.f : 0.f;
    }
    __syncthreads();
    float sfac;
    {
      float gs = 0.f, f2 = 0.f;
      if (tid < NP)
        for (int j = 0; j < NP; j++) {
          const float x = Y32[j * NP + tid];
          gs += fabsf(x);
          f2 = fmaf(x, x, f2);
        }
      gs = warp_max(gs);
      f2 = warp_sum(f2);
      if (lane == 0) {
        redf[wid] = gs;
        redf[4 + wid] = f2;
      }
      __syncthreads();
      const float gm = fmaxf(fmaxf(redf[0], redf[1]), fmaxf(redf[2], redf[3]));
      sfac = fminf(gm, sqrtf((redf[4] + redf[5]) + (redf[6] + redf[7]))) * 1.00001f;
    }
    const double s = trA * (double)sfac, inv_s = 1.0 / s;
    const float is32 = (float)inv_s;
    const float lo = 0.9f * (float)(c * inv_s);
    ok = ok && s < 1.0e5 * c;
    if (ok) {
      const float isf = 1.f / sfac;
      for (int idx = tid; idx < Q; idx += FN_NT) Y32[idx] *= isf;
      __syncthreads();
      ok = fn_newton_schulz<NP>(Y32, Z32, T32, Y32 + Q, redf, n8, lo);
    }
    if (ok) {
      // Z exactly symmetric; A/s as pairs of floats in A's place (A is in T)
      const int i0 = (tid >> 4) * C::TR, tx = tid & 15;
      float z[C::TR][C::TC];
#pragma unroll
      for (int b = 0; b < C::TC; b++) {
        float m[C::TR];
        fn_ld<C::TR>(Z32 + fn_col<NP>(tx, b) * NP + i0, m);
#pragma unroll
        for (int a = 0; a < C::TR; a++) z[a][b] = 0.5f * (Z32[(i0 + a) * NP + fn_col<NP>(tx, b)] + m[a]);
      }
      float2* A2 = reinterpret_cast<float2*>(A);
      for (int idx = tid; idx < Q; idx += FN_NT) {
        const double a = A[idx] * inv_s;
        const float h = (float)a;
        A2[idx] = make_float2(h, (float)(a - (double)h));
      }
      __syncthreads();
#pragma unroll
      for (int a = 0; a < C::TR; a++)
#pragma unroll
        for (int b = 0; b < C::TC; b++) Z32[(i0 + a) * NP + fn_col<NP>(tx, b)] = z[a][b];
      __syncthreads();

      // ---- 3. Newton's method anchored to A ----
      // a correction takes the residual r to about max(1e-5 r, r^2), so below
      // rtol the next one reaches FP64 rounding
      const float rtol = 5.0e-10f;
      ok = false;
      for (int it = 0; it < 5; it++) {
        int fx[MAXF], fy[MAXF];
#pragma unroll
        for (int b = 0; b < MAXF; b++) {
          const int id = wid + 4 * b, bi = id / nb;
          fx[b] = 8 * bi + li;
          fy[b] = 8 * (id - bi * nb) + lj;
        }
        float e2 = 0.f;
        float rv[MAXL][2];
        if (it == 0) {
          // The first residual, about 1e-6, is wanted to 1e-11 only: pairs of
          // floats, 8 FP32 operations where an FP64 one takes 62 of their slots.
          // Partial sums of P = (A/s) Z and of Z P stay below sqrt(s/c).
          const float off = scalbnf(1.5f, ilogbf(rsqrtf(lo)) + 2);
          float ph[MAXF][2], pl[MAXF][2];
#pragma unroll
          for (int b = 0; b < MAXF; b++) {
            ph[b][0] = ph[b][1] = off;
            pl[b][0] = pl[b][1] = 0.f;
          }
          fn_counted<MAXF, MINF>(minef, [&](auto m) {
            for (int k = 0; k < n8; k++) {
              const float2* ak = A2 + k * NP;
              const float* zk = Z32 + k * NP;
#pragma unroll
              for (int b = 0; b < decltype(m)::value; b++) {
                const float2 a = ak[fx[b]];
                const float2 y = *reinterpret_cast<const float2*>(zk + fy[b]);
                fn_df_mac(ph[b][0], pl[b][0], a, y.x);
                fn_df_mac(ph[b][1], pl[b][1], a, y.y);
              }
            }
          });
          float2* P2 = reinterpret_cast<float2*>(P);
#pragma unroll
          for (int b = 0; b < MAXF; b++)
            if (b < minef) {
              P2[fx[b] * NP + fy[b]] = fn_df_value(ph[b][0], pl[b][0], off);
              P2[fx[b] * NP + fy[b] + 1] = fn_df_value(ph[b][1], pl[b][1], off);
            }
          __syncthreads();
          float qh[MAXL][2], ql[MAXL][2];
#pragma unroll
          for (int b = 0; b < MAXL; b++) {
            qh[b][0] = qh[b][1] = off;
            ql[b][0] = ql[b][1] = 0.f;
          }
          fn_counted<MAXL, MINL>(mine, [&](auto m) {
            for (int k = 0; k < n8; k++) {
              const float* zk = Z32 + k * NP;
              const float2* pk = P2 + k * NP;
#pragma unroll
              for (int b = 0; b < decltype(m)::value; b++) {
                const float z = zk[xo[b]];
                const float4 y = *reinterpret_cast<const float4*>(pk + yo[b]);
                fn_df_mac(qh[b][0], ql[b][0], make_float2(y.x, y.y), z);
                fn_df_mac(qh[b][1], ql[b][1], make_float2(y.z, y.w), z);
              }
            }
          });
#pragma unroll
          for (int b = 0; b < MAXL; b++)
#pragma unroll
            for (int q = 0; q < 2; q++) {
              const float2 v = fn_df_value(qh[b][q], ql[b][q], off);
              rv[b][q] = ((xo[b] == yo[b] + q ? 1.f : 0.f) - v.x) - v.y;
            }
        } else {
          double pf[MAXF][2];
#pragma unroll
          for (int b = 0; b < MAXF; b++) pf[b][0] = pf[b][1] = 0.0;
          fn_counted<MAXF, MINF>(minef, [&](auto m) { fn_product<NP, decltype(m)::value>(A, Z, n8, fx, fy, pf); });
#pragma unroll
          for (int b = 0; b < MAXF; b++)
            if (b < minef) *reinterpret_cast<double2*>(P + fx[b] * NP + fy[b]) = make_double2(pf[b][0], pf[b][1]);
          __syncthreads();
#pragma unroll
          for (int b = 0; b < MAXL; b++) acc[b][0] = acc[b][1] = 0.0;
          fn_counted<MAXL, MINL>(mine, [&](auto m) { fn_product<NP, decltype(m)::value>(Z, P, n8, xo, yo, acc); });
#pragma unroll
          for (int b = 0; b < MAXL; b++)
#pragma unroll
            for (int q = 0; q < 2; q++)
              rv[b][q] = (float)((xo[b] == yo[b] + q ? 1.0 : 0.0) - acc[b][q] * inv_s);
        }
        // R = I - Z (A/s) Z; M = (A/s) Z takes A's place
#pragma unroll
        for (int b = 0; b < MAXL; b++)
#pragma unroll
          for (int q = 0; q < 2; q++)
            if (b < mine) {
              const float x2 = rv[b][q] * rv[b][q];
              e2 += (xo[b] >> 3) == (yo[b] >> 3) ? x2 : 2.f * x2;
            }
        e2 = block_sum<float, FN_NT>(e2, redf);
        if (!(e2 < 0.09f)) break;
        float* M32 = reinterpret_cast<float*>(A);
        for (int idx = tid; idx < Q; idx += FN_NT) {
          const int i = idx / NP, j = idx - i * NP;
          M32[idx] = (i < n8 && j < n8) ? (it == 0 ? reinterpret_cast<const float2*>(P)[idx].x : (float)P[idx] * is32)
                                        : (i == j ? 1.f : 0.f);
        }
        __syncthreads();
        float* R32 = reinterpret_cast<float*>(P);
        for (int idx = tid; idx < Q; idx += FN_NT) {
          const int i = idx / NP, j = idx - i * NP;
          if (i >= n8 || j >= n8) R32[idx] = 0.f;
        }
#pragma unroll
        for (int b = 0; b < MAXL; b++)
          if (b < mine) {
#pragma unroll
            for (int q = 0; q < 2; q++) {
              // a diagonal block's elements are set from its lower half, so R is exactly symmetric
              if (xo[b] >= yo[b] + q) {
                R32[xo[b] * NP + yo[b] + q] = rv[b][q];
                R32[(yo[b] + q) * NP + xo[b]] = rv[b][q];
              }
            }
          }
        __syncthreads();
        fn_sign<NP>(M32, M32 + Q, R32, R32 + Q, n8, lo);
        // Z <- Z + D, D symmetrised; after the first correction Z is FP64
        if (it == 0) {
#pragma unroll
          for (int a = 0; a < C::TR; a++)
#pragma unroll
            for (int b = 0; b < C::TC; b++) z[a][b] = Z32[(i0 + a) * NP + fn_col<NP>(tx, b)];
          __syncthreads();
        }
#pragma unroll
        for (int b = 0; b < C::TC; b++) {
          float m[C::TR];
          fn_ld<C::TR>(R32 + fn_col<NP>(tx, b) * NP + i0, m);
#pragma unroll
          for (int a = 0; a < C::TR; a++) {
            double* zz = Z + (i0 + a) * NP + fn_col<NP>(tx, b);
            *zz = (it == 0 ? (double)z[a][b] : *zz) + (double)(0.25f * (R32[(i0 + a) * NP + fn_col<NP>(tx, b)] + m[a]));
          }
        }
        __syncthreads();
        if (it > 0 && sqrtf(e2) <= rtol) {
          ok = true;
          break;
        }
        for (int idx = tid; idx < Q; idx += FN_NT) {
          const int i = idx / NP, j = idx - i * NP;
          A[idx] = (i < n && j < n) ? T[i * n + j] : (i == j ? c : 0.0);
        }
        __syncthreads();
      }
    }
    if (!ok) {  // uniform: left to the eigensolver
      if (tid == 0) status[p] = LETKF_PENDING;
      __syncthreads();
      continue;
    }
    // ---- wbar = Z (Z b) / s, T, Pa, inflation ----
    if (tid < NP) {
      double a = 0.0;
      for (int j = 0; j < n; j++) a = fma(Z[j * NP + tid], bv[j], a);
      g[tid] = a;
    }
    if (tid == FN_NT - 1) {  // adaptive inflation (:218-239); p2 = trace(Gram)/(ne-1)
      const double q1 = sums[1], q2 = tr / (double)(n - 1), q3 = sums[2];
      const double q4 = (q1 - q3) / q2 - infl;
      const double t = (infl * q2 + q3) / q2;
      const double sigma_o = 2.0 / q3 * (t * t);
      const double gain = (kSigmaB * kSigmaB) / (sigma_o + kSigmaB * kSigmaB);
      parm_infl[p] = infl + gain * q4;
      status[p] = LETKF_OK;
    }
    __syncthreads();
    if (tid < n) {
      double a = 0.0;
      for (int j = 0; j < n; j++) a = fma(Z[j * NP + tid], g[j], a);
      a = a * inv_s;
      e[tid] = a;
      if (transm) transm[(size_t)p * n + tid] = a;
    }
    __syncthreads();
    const double coef = sqrt((double)(n - 1) * inv_s);
    for (int idx = tid; idx < n * n; idx += FN_NT) {
      const int j = idx / n, i = idx - j * n;
      const double w = coef * Z[j * NP + i];
      T[idx] = transm ? w : w + e[i];
    }
    if (pao) {
      double* Pa = pao + (size_t)p * n * n;
#pragma unroll
      for (int b = 0; b < MAXL; b++) acc[b][0] = acc[b][1] = 0.0;
      fn_counted<MAXL, MINL>(mine, [&](auto m) { fn_product<NP, decltype(m)::value>(Z, Z, n8, xo, yo, acc); });
#pragma unroll
      for (int b = 0; b < MAXL; b++)
        if (b < mine) {
#pragma unroll
          for (int q = 0; q < 2; q++) {
            const int i = xo[b], j = yo[b] + q;
            if (i < n && j < n) {
              Pa[i * n + j] = acc[b][q] * inv_s;
              Pa[j * n + i] = acc[b][q] * inv_s;
            }
          }
        }
    }
    __syncthreads();
  }
}

template <int NP>
static int launch_ns(int ne, int npts, const int64_t* offs, const double* rows, const double* rdiag,
                     const double* rloc, const double* dep, double* parm_infl, double* trans, double* transm,
                     double* pao, int rdiag_wloc, double minfl, int* status, cudaStream_t stream) {
  static std::atomic<uint32_t> done{0};
  auto kern = core_f64_ns_kernel<NP>;
  const cudaError_t err = set_smem_once(kern, FnCfg<NP>::BYTES, done);
  if (err != cudaSuccess) return cuda_status(err);
  // A CTA per point: their local counts differ by orders of magnitude and
  // neighbours are alike, so a fixed stride over a resident grid leaves some SMs
  // with 1.6 times the work of others.  A counter in device memory does as well
  // on large batches but costs an allocation a call: 1,000 points of k = 20 with
  // 25 observations 447 us with it, 289 so; 30,000 of k = 40 17.2 ms and 16.8.
  kern<<<npts, FN_NT, FnCfg<NP>::BYTES, stream>>>(ne, npts, offs, rows, rdiag, rloc, dep, parm_infl, trans, transm,
                                                  pao, rdiag_wloc, minfl, status);
  note_launch();
  return cuda_status(cudaGetLastError());
}

// Points it leaves to the eigensolver get the status LETKF_PENDING.
int launch_core_f64_ns(int ne, int npts, const int64_t* offs, const double* rows, const double* rdiag,
                       const double* rloc, const double* dep, double* parm_infl, double* trans, double* transm,
                       double* pao, int rdiag_wloc, double minfl, int* status, cudaStream_t stream) {
#define FN_LAUNCH(NP)                                                                                              \
  return launch_ns<NP>(ne, npts, offs, rows, rdiag, rloc, dep, parm_infl, trans, transm, pao, rdiag_wloc, minfl, \
                       status, stream)
  if (ne <= 16) FN_LAUNCH(16);
  if (ne <= 32) FN_LAUNCH(32);
  if (ne <= 48) FN_LAUNCH(48);
  FN_LAUNCH(64);
#undef FN_LAUNCH
}

}  // namespace letkf
