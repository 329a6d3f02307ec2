// core_mixed.cu -- batched mixed-precision letkf_core on packed local rows.
//
// FP32 Gram and transform, FP64 for the inflation sums.  Two launches:
//   core_mixed_ns_kernel   every point with c > 0 and tr(G) < 1e6 c (where
//       mtx_eigen's truncation cannot act): W = sqrt((k-1)/s) (A/s)^(-1/2) by
//       the spectrum-scaled Newton-Schulz iteration, wbar = Z (Z b) / s.
//   core_mixed_kernel      the points the first launch leaves (status
//       LETKF_PENDING, or MN_PENDING_GRAM with their sums in trans): the
//       parallel Jacobi eigensolver with the reference's truncation.
// Outputs FP32 trans / transm with the semantics of
// common/common_letkf.f90:50-243 (transm present: trans = T, transm = wbar;
// absent: trans = T + wbar 1^T).
#include "mixed_core.cuh"

namespace letkf {

// ---- Newton-Schulz form ----------------------------------------------------
// Bound: FP32 multiply-adds, 3 k^3 per step in k x k products whose operands
// come from shared memory.  The products waited for shared memory and barriers
// (FMA pipe 27 % busy): a warp's lanes ran down the rows of a tile, so storing
// a tile or reading one back met 8-fold bank conflicts that cost as much as
// the product.  Here the lanes run along the columns; a thread's tile is 8 x 8
// where it can be (16 bytes a lane return at a quarter of the rate, so a wide
// tile is what balances loads and multiply-adds); operands are loaded one step
// ahead; up to k = 32 one warp takes a point by itself and never meets a
// barrier; padding is to 16, 32, 48, 64, 96 or 128; the first step has Z = I
// (one product instead of three) and the last needs no new Y; a CTA's points
// are handed out by the hardware.  100,000 points of k = 32 with 21 local observations: 5.49
// -> 2.19 ms (FMA pipe 54 % busy); 4,001 points of k = 50 with 133 on average:
// 1.77 -> 0.86 ms (48 %).  Every sum keeps the order that the eigensolver form
// (and this one before) adds in, so transforms and inflation are unchanged to
// the bit.
// TX threads along the columns (the lanes' fast index), TY along the rows
template <int NP>
struct MnCfg;
template <>
struct MnCfg<16> {
  static constexpr int TX = 8, TY = 4, CH = 16, MINB = 16;
};
template <>
struct MnCfg<32> {
  static constexpr int TX = 8, TY = 4, CH = 32, MINB = 8;
};
template <>
struct MnCfg<48> {
  static constexpr int TX = 8, TY = 8, CH = 32, MINB = 7;
};
template <>
struct MnCfg<64> {
  static constexpr int TX = 8, TY = 8, CH = 32, MINB = 4;
};
template <>
struct MnCfg<96> {
  static constexpr int TX = 16, TY = 12, CH = 16, MINB = 2;
};
template <>
struct MnCfg<128> {
  static constexpr int TX = 16, TY = 16, CH = 16, MINB = 1;
};

template <int NP>
struct Mn {
  using C = MnCfg<NP>;
  static constexpr int TP = C::TX * C::TY;               // threads of a point
  // points of a CTA: lists differ from point to point, and the CTA's shared memory is held until its last one is
  // done; with one point 15 warps fit an SM where two leave 16 (100,000 points of k = 20, lists 0..150: four 2.36 ms,
  // two 2.26, one 2.30).  Points taken from a counter in device memory take 2.22 there, but an allocation a call: 20,000
  // points of k = 16 300 us against 165, 4,000 of k = 50 797 against 680 (calls in a row, that wait for nothing: 979, 993)
  static constexpr int PPC = TP == 32 ? 2 : 1;
  // product tile of a thread: TR consecutive rows, TC columns in groups of G (4 where TC allows it) that lie
  // G TX apart, so that the lanes of a quarter warp read and write 128 consecutive bytes
  static constexpr int TR = NP / C::TY, TC = NP / C::TX, G = TC % 4 == 0 ? 4 : 2;
  // floats of a point: Y, Z, T (the staged rows alias Z and T), b, wbar, scratch, two chunks' weights,
  // departures and rloc, reductions
  static constexpr int TAIL = 3 * NP + 6 * C::CH + 32;
  static constexpr int POINT = 3 * NP * NP + TAIL;
  static constexpr size_t BYTES = sizeof(float) * (size_t)POINT * PPC;
};

template <int NP>
__device__ __forceinline__ void mn_sync() {
  if constexpr (Mn<NP>::TP == 32)
    __syncwarp();
  else
    __syncthreads();
}

// sum (or maximum) over a point's threads; every thread gets it, and what was
// written to shared memory before is visible after
template <int NP, typename T, bool MAX = false>
__device__ __forceinline__ T mn_reduce(T v, float* scratch) {
  v = MAX ? warp_max(v) : warp_sum(v);
  if constexpr (Mn<NP>::TP == 32) {
    __syncwarp();
    return v;
  } else {
    T* red = reinterpret_cast<T*>(scratch);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    T s = red[0];
#pragma unroll
    for (int w = 1; w < Mn<NP>::TP / 32; w++) s = MAX ? (red[w] > s ? red[w] : s) : s + red[w];
    return s;
  }
}

// v[0] + .. + v[NV-1], v[i] = pad from NP on: by 32s as warps of one thread per
// element add them, then the partial sums as a warp does
template <int NP, int NV>
__device__ __forceinline__ float mn_sum32(const float* v, float pad) {
  float w[NV / 32];
#pragma unroll
  for (int q = 0; q < NV / 32; q++) {
    const int i = 32 * q + (threadIdx.x & 31);
    w[q] = warp_sum(i < NP ? v[i] : pad);
  }
  if constexpr (NV == 32)
    return w[0];
  else if constexpr (NV == 64)
    return w[0] + w[1];
  else
    return (w[0] + w[2]) + (w[1] + w[3]);
}

template <int N>
__device__ __forceinline__ void mn_ld(const float* p, float (&v)[N]) {
  if constexpr (N % 4 == 0) {
#pragma unroll
    for (int q = 0; q < N; q += 4) {
      const float4 t = *reinterpret_cast<const float4*>(p + q);
      v[q] = t.x;
      v[q + 1] = t.y;
      v[q + 2] = t.z;
      v[q + 3] = t.w;
    }
  } else {
    static_assert(N % 2 == 0, "tile");
#pragma unroll
    for (int q = 0; q < N; q += 2) {
      const float2 t = *reinterpret_cast<const float2*>(p + q);
      v[q] = t.x;
      v[q + 1] = t.y;
    }
  }
}

template <int N>
__device__ __forceinline__ void mn_st(float* p, const float (&v)[N]) {
  if constexpr (N % 4 == 0) {
#pragma unroll
    for (int q = 0; q < N; q += 4) *reinterpret_cast<float4*>(p + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
  } else {
#pragma unroll
    for (int q = 0; q < N; q += 2) *reinterpret_cast<float2*>(p + q) = make_float2(v[q], v[q + 1]);
  }
}

// column of element b of a thread's tile
template <int NP>
__device__ __forceinline__ int mn_col(int tx, int b) {
  constexpr int G = Mn<NP>::G;
  return (b / G) * (G * MnCfg<NP>::TX) + G * tx + b % G;
}

// a thread's columns of the row at p
template <int NP>
__device__ __forceinline__ void mn_ldc(const float* p, int tx, float (&v)[Mn<NP>::TC]) {
  constexpr int G = Mn<NP>::G;
#pragma unroll
  for (int q = 0; q < Mn<NP>::TC; q += G) {
    float t[G];
    mn_ld<G>(p + mn_col<NP>(tx, q), t);
#pragma unroll
    for (int e = 0; e < G; e++) v[q + e] = t[e];
  }
}

template <int NP>
__device__ __forceinline__ void mn_stc(float* p, int tx, const float (&v)[Mn<NP>::TC]) {
  constexpr int G = Mn<NP>::G;
#pragma unroll
  for (int q = 0; q < Mn<NP>::TC; q += G) {
    float t[G];
#pragma unroll
    for (int e = 0; e < G; e++) t[e] = v[q + e];
    mn_st<G>(p + mn_col<NP>(tx, q), t);
  }
}

// acc = X^T Yb for this thread's tile
template <int NP>
__device__ __forceinline__ void mn_gemm(const float* X, const float* Yb, int i0, int tx,
                                        float (&acc)[Mn<NP>::TR][Mn<NP>::TC]) {
  constexpr int TR = Mn<NP>::TR, TC = Mn<NP>::TC;
#pragma unroll
  for (int a = 0; a < TR; a++)
#pragma unroll
    for (int b = 0; b < TC; b++) acc[a][b] = 0.f;
  // operands of k + 1 are loaded before the products of k
  float av[2][TR], bv[2][TC];
  mn_ld<TR>(X + i0, av[0]);
  mn_ldc<NP>(Yb, tx, bv[0]);
#pragma unroll 2
  for (int k = 0; k < NP; k += 2) {
    mn_ld<TR>(X + (k + 1) * NP + i0, av[1]);
    mn_ldc<NP>(Yb + (k + 1) * NP, tx, bv[1]);
#pragma unroll
    for (int a = 0; a < TR; a++)
#pragma unroll
      for (int b = 0; b < TC; b++) acc[a][b] = fmaf(av[0][a], bv[0][b], acc[a][b]);
    if (k + 2 < NP) {
      mn_ld<TR>(X + (k + 2) * NP + i0, av[0]);
      mn_ldc<NP>(Yb + (k + 2) * NP, tx, bv[0]);
    }
#pragma unroll
    for (int a = 0; a < TR; a++)
#pragma unroll
      for (int b = 0; b < TC; b++) acc[a][b] = fmaf(av[1][a], bv[1][b], acc[a][b]);
  }
}

__device__ __forceinline__ void mn_cp4(float* dst, const float* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

// a x - b y, one rounding for the product by b
__device__ __forceinline__ float mn_axmb(float a, float x, float b, float y) {
  return fmaf(a, x, -__fmul_rn(b, y));
}

// Z = (A/s)^(-1/2) from Y = A/s (spectrum in [lo, 1]): T = Z Y, Y <- Y (3I -
// aT) / 2, Z <- (3I - aT) Z / 2 with steps scaled to the spectrum, until
// ||T - I||_F < 1e-4 and one step more (the FP32 floor).  Leaves Z in Z and its
// transpose in T; false when it does not converge.  `pads` scalars stand for
// the coordinates by which the eigensolver's padding is wider.
template <int NP>
__device__ bool mn_newton_schulz(float* Y, float* Z, float* T, float* red, int tp, float lo, float ypad, int pads) {
  using M = Mn<NP>;
  constexpr int TR = M::TR, TC = M::TC;
  const int i0 = (tp / MnCfg<NP>::TX) * TR, tx = tp % MnCfg<NP>::TX;
  float acc[TR][TC], yn[TR][TC];
  float zpad = 1.f;
  for (int it = 0; it < 24; it++) {
    if (it) {
      mn_gemm<NP>(Z, Y, i0, tx, acc);
#pragma unroll
      for (int a = 0; a < TR; a++) mn_stc<NP>(T + (i0 + a) * NP, tx, acc[a]);
    } else {  // Z = I: T = Y
#pragma unroll
      for (int a = 0; a < TR; a++) mn_ldc<NP>(Y + (i0 + a) * NP, tx, acc[a]);
    }
    float e2 = 0.f;
#pragma unroll
    for (int a = 0; a < TR; a++)
#pragma unroll
      for (int b = 0; b < TC; b++) {
        const float d = acc[a][b] - (i0 + a == mn_col<NP>(tx, b) ? 1.f : 0.f);
        e2 = fmaf(d, d, e2);
      }
    const float tpad = zpad * ypad;
    e2 = mn_reduce<NP, float>(e2, red) + (float)pads * ((tpad - 1.f) * (tpad - 1.f));  // publishes T
    if (!isfinite(e2)) return false;
    const bool last = e2 < 1.0e-8f;
    const float al = ns_scale(lo), sa = sqrtf(al);
    const float ka = 1.5f * sa, kb = 0.5f * al * sa;
    lo = f_ns(al * lo);
    ypad = ka * ypad - kb * (ypad * tpad);
    zpad = ka * zpad - kb * (tpad * zpad);
    if (!last) {
      mn_gemm<NP>(Y, it ? T : Y, i0, tx, yn);
#pragma unroll
      for (int a = 0; a < TR; a++) {
        float y[TC];
        mn_ldc<NP>(Y + (i0 + a) * NP, tx, y);
#pragma unroll
        for (int b = 0; b < TC; b++) yn[a][b] = mn_axmb(ka, y[b], kb, yn[a][b]);
      }
    }
    if (it) {
      mn_gemm<NP>(T, Z, i0, tx, acc);
#pragma unroll
      for (int a = 0; a < TR; a++) {
        float z[TC];
        mn_ldc<NP>(Z + (i0 + a) * NP, tx, z);
#pragma unroll
        for (int b = 0; b < TC; b++) acc[a][b] = mn_axmb(ka, z[b], kb, acc[a][b]);
      }
    } else {  // T^T I, T symmetric
#pragma unroll
      for (int a = 0; a < TR; a++)
#pragma unroll
        for (int b = 0; b < TC; b++) acc[a][b] = mn_axmb(ka, i0 + a == mn_col<NP>(tx, b) ? 1.f : 0.f, kb, acc[a][b]);
    }
    mn_sync<NP>();
#pragma unroll
    for (int a = 0; a < TR; a++) {
      if (!last) mn_stc<NP>(Y + (i0 + a) * NP, tx, yn[a]);
      mn_stc<NP>(Z + (i0 + a) * NP, tx, acc[a]);
    }
    if (last) {
#pragma unroll
      for (int b = 0; b < TC; b++) {
        float col[TR];
#pragma unroll
        for (int a = 0; a < TR; a++) col[a] = acc[a][b];
        mn_st<TR>(T + mn_col<NP>(tx, b) * NP + i0, col);
      }
    }
    mn_sync<NP>();
    if (last) return true;
  }
  return false;
}

// A point that the iteration is not tried for leaves its Gram matrix (lower
// triangle), b, p1 and p3 (above the diagonal) in its place in trans: the
// eigensolver forming them again took up to 18 % of small batches with long
// lists (1,000 points of k = 20 with 300 to 500 observations, three in ten left
// to it: 521 us with one kernel for both, 613 with the Gram twice, 538 so).
constexpr int MN_PENDING_GRAM = -LETKF_PENDING;  // of status, until the eigensolver's launch
constexpr int MN_GRAM_MIN = 5;  // fewest members whose rows 0 and 1 hold the n + 2 values above the diagonal

// place of value e < n + 2 above the diagonal: row 0 from column 1, row 1 from column 2
__device__ __forceinline__ int mn_spare(int n, int e) { return e < n - 1 ? 1 + e : e + 3; }

template <int NP>
__global__ void __launch_bounds__(Mn<NP>::TP* Mn<NP>::PPC, MnCfg<NP>::MINB) core_mixed_ns_kernel(
    int n, int npts, const int64_t* __restrict__ offs, const float* __restrict__ rows,
    const float* __restrict__ rdiag, const float* __restrict__ rloc, const float* __restrict__ dep,
    double* parm_infl, float* trans, float* transm, int rdiag_wloc, double minfl, int* status) {
  using M = Mn<NP>;
  using C = MnCfg<NP>;
  constexpr int TR = M::TR, TC = M::TC, TP = M::TP, CH = C::CH, Q = NP * NP;
  extern __shared__ __align__(16) float smf[];
  const int tp = threadIdx.x % TP, slot = threadIdx.x / TP;
  float* Y = smf + (size_t)slot * M::POINT;
  float* Z = Y + Q;
  float* T = Z + Q;
  float* bv = T + Q;
  float* wb = bv + NP;
  float* g = wb + NP;
  float* wts = g + NP;        // weight, departure, rloc of a chunk, twice
  float* red = wts + 6 * CH;  // 32
  const int i0 = (tp / C::TX) * TR, tx = tp % C::TX;
  for (int p = blockIdx.x * M::PPC + slot; p < npts; p += gridDim.x * M::PPC) {
    const int64_t r0 = offs[p];
    const int L = (int)(offs[p + 1] - r0);
    double infl = parm_infl[p];
    float* Tp = trans + (size_t)p * n * n;
    if (L == 0) {
      const float sq = (float)sqrt(infl);
      for (int idx = tp; idx < n * n; idx += TP) Tp[idx] = (idx / n == idx % n) ? sq : 0.f;
      if (transm)
        for (int i = tp; i < n; i += TP) transm[(size_t)p * n + i] = 0.f;
      if (tp == 0) status[p] = LETKF_OK;
      mn_sync<NP>();
      continue;
    }
    // ---- Gram: rows staged two chunks deep, columns n .. NP-1 zero ----
    static_assert(CH <= NP, "a chunk of rows fits a matrix");
    auto stage = [&](int c0, int buf) {
      const int nr = min(CH, L - c0);
      const float* src = rows + (size_t)(r0 + c0) * n;
      float* dst = buf ? T : Z;
      if (n == NP) {
        for (int t = tp; t < nr * NP; t += TP) mn_cp4(dst + t, src + t);
      } else {
        for (int t = tp; t < nr * n; t += TP) {
          const int r = t / n;
          mn_cp4(dst + r * NP + (t - r * n), src + t);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      float* w = wts + buf * 3 * CH;
      for (int r = tp; r < nr; r += TP) {
        const float rd = rdiag[r0 + c0 + r], rl = rloc[r0 + c0 + r];
        w[r] = rdiag_wloc ? 1.f / rd : rl / rd;
        w[CH + r] = dep[r0 + c0 + r];
        w[2 * CH + r] = rl;
      }
    };
    if (n < NP)
      for (int t = tp; t < CH * NP; t += TP) Z[t] = T[t] = 0.f;
    mn_sync<NP>();
    float acc[TR][TC], bacc[TR];
    float p1 = 0.f, p3 = 0.f;
#pragma unroll
    for (int a = 0; a < TR; a++) {
      bacc[a] = 0.f;
#pragma unroll
      for (int b = 0; b < TC; b++) acc[a][b] = 0.f;
    }
    stage(0, 0);
    for (int c0 = 0, buf = 0; c0 < L; c0 += CH, buf ^= 1) {
      const int nr = min(CH, L - c0);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      mn_sync<NP>();
      if (c0 + CH < L) stage(c0 + CH, buf ^ 1);
      const float* y = buf ? T : Z;
      const float* w = wts + buf * 3 * CH;
#pragma unroll 4
      for (int r = 0; r < nr; r++) {
        float av[TR], yv[TC];
        mn_ld<TR>(y + r * NP + i0, av);
        mn_ldc<NP>(y + r * NP, tx, yv);
        const float wr = w[r], d = w[CH + r];
#pragma unroll
        for (int a = 0; a < TR; a++) {
          av[a] *= wr;
          bacc[a] = fmaf(av[a], d, bacc[a]);
#pragma unroll
          for (int b = 0; b < TC; b++) acc[a][b] = fmaf(av[a], yv[b], acc[a][b]);
        }
      }
      // row r of 32 to lane r, for every chunk size up to k = 64
      const int r = tp - (NP == 16 ? (c0 & 16) : 0);
      if (r >= 0 && r < nr) {
        const float d = w[CH + r];
        p1 = fmaf(d * d, w[r], p1);
        p3 += w[2 * CH + r];
      }
    }
    // lower triangle mirrored, c on the diagonal; the staged rows are done with
    // once every thread is past the sums' barrier
    p1 = mn_reduce<NP, float>(p1, red);
    p3 = mn_reduce<NP, float>(p3, red);
    if (minfl > 0.0 && infl < minfl) infl = minfl;
    const float c = (float)((double)(n - 1) / infl);
#pragma unroll
    for (int a = 0; a < TR; a++)
#pragma unroll
      for (int b = 0; b < TC; b++) {
        const int i = i0 + a, j = mn_col<NP>(tx, b);
        if (i == j) g[i] = acc[a][b];
        if (i > j) Y[i * NP + j] = Y[j * NP + i] = acc[a][b];
        if (i == j) Y[i * NP + j] = acc[a][b] + c;
      }
    if (tx == 0) {
#pragma unroll
      for (int a = 0; a < TR; a++) bv[i0 + a] = bacc[a];
    }
    mn_sync<NP>();
    const double trace = (double)mn_sum32<NP, (NP <= 32 ? 32 : NP <= 64 ? 64 : 128)>(g, 0.f);
    mn_sync<NP>();
    bool ok = c > 0.f && trace < 1.0e6 * (double)c;
    const bool tried = ok;
    float s = 1.f;
    if (ok) {
      // s = min(Gershgorin, Frobenius) >= lambda_max of the matrix padded to NV
      constexpr int NV = NP <= 32 ? 32 : NP <= 64 ? 64 : 128;
      float gs = c;
      for (int i = tp; i < NP; i += TP) {
        float gi = 0.f, f2 = 0.f;
#pragma unroll 4
        for (int j = 0; j < NP; j++) {
          const float x = Y[j * NP + i];
          gi += fabsf(x);
          f2 = fmaf(x, x, f2);
        }
        gs = fmaxf(gs, gi);
        g[i] = f2;
      }
      gs = mn_reduce<NP, float, true>(gs, red);
      s = fminf(gs, sqrtf(mn_sum32<NP, NV>(g, c * c)));
      const float inv_s = 1.f / s;
      for (int t = tp; t < Q; t += TP) Y[t] *= inv_s;
      mn_sync<NP>();
      ok = mn_newton_schulz<NP>(Y, Z, T, red, tp, 0.9f * c * inv_s, c * inv_s, NV - NP);
    }
    if (!ok) {  // uniform over the point's threads: left to the eigensolver
      // with its sums, where the iteration has not overwritten them
      const bool gram = n >= MN_GRAM_MIN && !tried;
      if (gram) {
        for (int idx = tp; idx < n * n; idx += TP) {
          const int i = idx / n, j = idx - i * n;
          if (j <= i) Tp[idx] = i == j ? g[i] : Y[i * NP + j];
        }
        for (int e = tp; e < n + 2; e += TP) Tp[mn_spare(n, e)] = e < n ? bv[e] : e == n ? p1 : p3;
      }
      if (tp == 0) status[p] = gram ? MN_PENDING_GRAM : LETKF_PENDING;
      mn_sync<NP>();
      continue;
    }
    // ---- wbar = Z (Z b) / s, W, inflation ----
    for (int i = tp; i < NP; i += TP) {
      float a = 0.f;
#pragma unroll 4
      for (int j = 0; j < NP; j++) a = fmaf(Z[j * NP + i], bv[j], a);
      g[i] = a;
    }
    if (tp == TP - 1) {
      parm_infl[p] = infl_update(n, infl, p1, trace, p3);
      status[p] = LETKF_OK;
    }
    mn_sync<NP>();
    for (int i = tp; i < NP; i += TP) {
      float a = 0.f;
#pragma unroll 4
      for (int j = 0; j < NP; j++) a = fmaf(Z[j * NP + i], g[j], a);
      wb[i] = a / s;
      if (transm && i < n) transm[(size_t)p * n + i] = a / s;
    }
    mn_sync<NP>();
    const float coef = sqrtf((float)(n - 1) / s);
    const bool sep = transm != nullptr;
    // trans(i, j): background member i, analysis member j; T holds the transpose of Z
    for (int idx = tp; idx < n * n; idx += TP) {
      const int j = n == NP ? idx / NP : idx / n, i = idx - j * n;
      const float w = coef * T[j * NP + i];
      Tp[idx] = sep ? w : w + wb[i];
    }
    mn_sync<NP>();
  }
}

// ---- eigensolver form, for the points left ----------------------------------
template <int NP>
__global__ void __launch_bounds__(MixedCfg<NP>::NT) core_mixed_kernel(
    int n, int npts, const int64_t* __restrict__ offs, const float* __restrict__ rows,
    const float* __restrict__ rdiag, const float* __restrict__ rloc, const float* __restrict__ dep,
    double* parm_infl, float* trans, float* transm, int rdiag_wloc, double minfl, int* status, int max_sweeps) {
  using C = MixedCfg<NP>;
  using S = MixedSmem<NP>;
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x;
  for (int p = blockIdx.x; p < npts; p += gridDim.x) {
    const int pending = status[p];
    if (pending != LETKF_PENDING && pending != MN_PENDING_GRAM) continue;
    __syncthreads();  // every thread has read the status before it is set
    const int64_t r0 = offs[p];
    const int L = (int)(offs[p + 1] - r0);
    double infl = parm_infl[p];
    float* T = trans + (size_t)p * n * n;
    GramAcc<NP> acc;
    double trace;
    if (pending == MN_PENDING_GRAM) {
      for (int idx = tid; idx < NP * NP; idx += C::NT) {
        const int i = idx / NP, j = idx - i * NP;
        sm[S::A + idx] = i < n && j < n ? T[i < j ? j * n + i : i * n + j] : 0.f;
      }
      for (int i = tid; i < NP; i += C::NT) sm[S::B + i] = i < n ? T[mn_spare(n, i)] : 0.f;
      acc.p1 = T[mn_spare(n, n)];
      acc.p3 = T[mn_spare(n, n + 1)];
      __syncthreads();
      trace = gram_trace<NP>(sm);
    } else {
      acc.zero();
      for (int c0 = 0; c0 < L; c0 += S::CH) {
        const int nr = min(S::CH, L - c0);
        __syncthreads();
        for (int t = tid; t < S::CH * NP; t += C::NT) {
          const int r = t / NP, m = t - r * NP;
          sm[S::Y + t] = (r < nr && m < n) ? rows[(size_t)(r0 + c0 + r) * n + m] : 0.f;
        }
        if (tid < nr) {
          const float rd = rdiag[r0 + c0 + tid], rl = rloc[r0 + c0 + tid];
          sm[S::WR + tid] = rdiag_wloc ? 1.f / rd : rl / rd;
          sm[S::DR + tid] = dep[r0 + c0 + tid];
          sm[S::RL + tid] = rl;
        }
        __syncthreads();
        for (int t = tid; t < nr * NP; t += C::NT) sm[S::YW + t] = sm[S::Y + t] * sm[S::WR + t / NP];
        __syncthreads();
        gram_chunk<NP>(sm, nr, acc);
      }
      trace = gram_finish<NP>(sm, acc);
    }
    if (minfl > 0.0 && infl < minfl) infl = minfl;
    const float c = (float)((double)(n - 1) / infl);
    for (int i = tid; i < NP; i += C::NT) sm[S::A + i * NP + i] += c;
    __syncthreads();
    jacobi_eig<NP>(sm, max_sweeps);
    const int st = eig_postprocess<NP>(sm, n);
    if (st != LETKF_OK) {
      for (int idx = tid; idx < n * n; idx += C::NT) T[idx] = NAN;
      if (tid == 0) status[p] = st;
      __syncthreads();
      continue;
    }
    const float* wb = sm + S::WB;
    const bool sep = transm != nullptr;
    form_w<NP>(sm, [&](int i, int j, float w) {
      if (i < n && j < n) T[(size_t)j * n + i] = sep ? w : w + wb[i];
    });
    if (sep)
      for (int i = tid; i < n; i += C::NT) transm[(size_t)p * n + i] = wb[i];
    if (tid == 0) {
      parm_infl[p] = infl_update(n, infl, acc.p1, trace, acc.p3);
      status[p] = LETKF_OK;
    }
    __syncthreads();
  }
}

template <int NP>
static int launch_ns(int ne, int npts, const int64_t* offs, const float* rows, const float* rdiag, const float* rloc,
                     const float* dep, double* parm_infl, float* trans, float* transm, int rdiag_wloc, double minfl,
                     int* status, cudaStream_t stream) {
  using M = Mn<NP>;
  static std::atomic<uint32_t> done{0};
  auto kern = core_mixed_ns_kernel<NP>;
  const cudaError_t err = set_smem_once(kern, M::BYTES, done);
  if (err != cudaSuccess) return cuda_status(err);
  const int grid = (npts + M::PPC - 1) / M::PPC;
  kern<<<grid, M::TP * M::PPC, M::BYTES, stream>>>(ne, npts, offs, rows, rdiag, rloc, dep, parm_infl, trans, transm,
                                                   rdiag_wloc, minfl, status);
  note_launch();
  return cuda_status(cudaGetLastError());
}

template <int NP>
static int launch_mixed_np(int ne, int npts, const int64_t* offs, const float* rows, const float* rdiag,
                           const float* rloc, const float* dep, double* parm_infl, float* trans, float* transm,
                           int rdiag_wloc, double minfl, int* status, cudaStream_t stream) {
  const size_t bytes = sizeof(float) * (size_t)MixedSmem<NP>::TOTAL;
  static std::atomic<uint32_t> done{0};
  auto kern = core_mixed_kernel<NP>;
  const cudaError_t err = set_smem_once(kern, bytes, done);
  if (err != cudaSuccess) return cuda_status(err);
  int dev = 0, nsm = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, MixedCfg<NP>::NT, bytes);
  if (per_sm < 1) per_sm = 1;
  // Four times what is resident: a CTA without a point to solve leaves at once,
  // and those with one seldom have a second behind it (1,000 points of k = 50, a
  // twentieth of them beyond the iteration: a resident grid 4.1 ms, 2.9 so).  A
  // grid of what shared memory alone allows left its last CTAs to a wave of their
  // own (5,000 points of k = 16, all of them beyond it: 2.7 ms, 2.1 so).
  const int most = 4 * nsm * per_sm, grid = npts < most ? npts : most;
  kern<<<grid, MixedCfg<NP>::NT, bytes, stream>>>(ne, npts, offs, rows, rdiag, rloc, dep, parm_infl, trans, transm,
                                                   rdiag_wloc, minfl, status, 12);
  note_launch();
  return cuda_status(cudaGetLastError());
}

int launch_core_mixed(int ne, int npts, const int64_t* offs, const float* rows, const float* rdiag,
                      const float* rloc, const float* dep, double* parm_infl, float* trans, float* transm,
                      int rdiag_wloc, double minfl, int* status, cudaStream_t stream) {
  if (ne < 2 || npts < 0) return LETKF_ERR_ARG;
  if (ne > LETKF_MAX_NE) return LETKF_ERR_CAPACITY;
  if (npts == 0) return LETKF_OK;
#define MN_ARGS ne, npts, offs, rows, rdiag, rloc, dep, parm_infl, trans, transm, rdiag_wloc, minfl, status, stream
  int st;
  if (ne <= 16)
    st = launch_ns<16>(MN_ARGS);
  else if (ne <= 32)
    st = launch_ns<32>(MN_ARGS);
  else if (ne <= 48)
    st = launch_ns<48>(MN_ARGS);
  else if (ne <= 64)
    st = launch_ns<64>(MN_ARGS);
  else if (ne <= 96)
    st = launch_ns<96>(MN_ARGS);
  else
    st = launch_ns<128>(MN_ARGS);
  if (st != LETKF_OK) return st;
  if (ne <= 32) return launch_mixed_np<32>(MN_ARGS);
  if (ne <= 64) return launch_mixed_np<64>(MN_ARGS);
  return launch_mixed_np<128>(MN_ARGS);
#undef MN_ARGS
}

}  // namespace letkf
