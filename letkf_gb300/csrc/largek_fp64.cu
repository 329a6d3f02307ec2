// largek_fp64.cu -- FP64 pass of the large-ensemble core for points the
// mixed-precision transform cannot certify.
//
// The large-k core (largek.cu) forms the Gram and the Newton-Schulz products
// from TF32 splits with FP32 accumulation, about 1e-6 relative.  Where
// lambda_max / c of A = Gram + (k-1)/rho I reaches about 1e3..1e4 (long local
// lists, small observation errors), the smallest eigen-directions of W are
// then not resolved and the core reports LETKF_ERR_EIG.  This pass redoes those
// points in FP64, the reference's precision (common/common_letkf.f90:101-239),
// its products on the tensor cores by exact digit splitting (ozaki_gemm.cuh):
//   1. the point's rows scaled, B = sqrt(w) Y with w = rloc / rdiag (1 / rdiag
//      with rdiag_wloc), split into digits member by member in chunks of the
//      lists, G = B^T B (lower triangle) over all points of a group at once;
//      b = B^T (sqrt(w) dep) in FP64;
//   2. A = G + cI, s = Gershgorin bound, Y = A / s, Z = I;
//   3. coupled Newton-Schulz, T = Z Y, Y <- Y M, Z <- M Z with M = sqrt(a)
//      (3I - aT) / 2, spectrum-scaled steps from the lower bound 0.9 c / s, up to
//      the step after ||ZY - I||_F^2 < 1e-14 (its quadratic convergence reaches
//      FP64 rounding); Y M = Y Z Y and M Z are symmetric, so their lower
//      triangles are formed and mirrored;
//   4. certificate ||Z (A/s) Z - I||_F^2 < 1e-16, then W = sqrt((k-1)/s) Z,
//      wbar = Z (Z b) / s and the adaptive inflation (:218-239).
// The core reports LETKF_ERR_CAPACITY where tr(G) >= 1e6 c, a cheap sufficient
// test that mtx_eigen's truncation (common/common_mtx.f90:66-72: eigenvalues
// below lambda_max sqrt(eps) are dropped) cannot act.  Every eigenvalue of A is
// at least c, so truncation needs lambda_max > c / sqrt(eps) = 6.7e7 c: this
// pass takes those points too and keeps the flag only where the sharper upper
// bound min(Gershgorin, ||A||_F) of lambda_max reaches 3e7 c, or where c <= 0.
//
// Matrices are padded to np, a multiple of 64 (A's padding is c I and decouples).
// With DGEMM on the FP64 pipe (0.92 TFLOP/s of its 1.2) four points of k = 512
// with 24,000 local observations took 41 ms in the Gram and 42 in the
// iteration; the digit products take 2.8 and 2.7, and the whole pass 6.4 ms.
#include <cuda_bf16.h>

#include <vector>

#include "mixed_core.cuh"
#include "ozaki_gemm.cuh"

namespace letkf {

constexpr int L64_NT = 256;
constexpr int L64_NS_MAX = 60;
constexpr double L64_NS_LAST = 1.0e-14;  // the step after this residual is the last
constexpr double L64_CERT_TOL = 1.0e-16;
// lambda_max bound / c from which mtx_eigen's truncation could act (half of 1 / sqrt(eps))
constexpr double L64_TRUNC_RATIO = 3.0e7;
constexpr int L64_SPLIT = 64;  // pieces of a list in the FP64 sums
constexpr int L64_PART = 32;   // pieces of a matrix in the residuals
constexpr size_t L64_DIGITS = (size_t)512 << 20;  // bytes of list digits held at a time

struct L64Point {
  double s, c, p1, p3, trace, infl, lo, ka, kb;
  int done, skip;
};

// the local lists of a group of points
struct L64Lists {
  const int64_t* r0;  // first entry of each point's list
  const int* L;
  const int64_t* o;   // first entry of the point in the group's arrays
  const float* rows;
  const __nv_bfloat16* rows16;
  const int* ridx;
  const float *rdiag, *rloc, *dep;
  int ne, wloc;
  double *sw, *ed;    // sqrt(w) and sqrt(w) dep of each entry of the group
};

__device__ __forceinline__ double l64_row(const L64Lists& q, int64_t e, int m) {
  const size_t ri = q.ridx ? (size_t)q.ridx[e] : (size_t)e;
  return q.rows16 ? (double)__bfloat162float(q.rows16[ri * q.ne + m]) : (double)q.rows[ri * q.ne + m];
}

__global__ void l64_weight_kernel(L64Lists q) {
  const int b = blockIdx.y, l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= q.L[b]) return;
  const int64_t e = q.r0[b] + l;
  const double sw = sqrt(q.wloc ? 1.0 / (double)q.rdiag[e] : (double)q.rloc[e] / (double)q.rdiag[e]);
  q.sw[q.o[b] + l] = sw;
  q.ed[q.o[b] + l] = sw * (double)q.dep[q.ridx ? (size_t)q.ridx[e] : (size_t)e];
}

// one piece of a list, L64_NT members a CTA: b = B^T (sqrt(w) dep) and the
// largest |B| of each member; p1 = sum w dep^2 and p3 = sum rloc
__global__ void __launch_bounds__(L64_NT) l64_stats_kernel(L64Lists q, int np, double* pb, unsigned long long* pm,
                                                           double* pp) {
  __shared__ double red[L64_NT / 32];
  const int b = blockIdx.y, s = blockIdx.x, tid = threadIdx.x;
  const int L = q.L[b], per = (L + L64_SPLIT - 1) / L64_SPLIT, l0 = s * per, l1 = min(L, l0 + per);
  const int64_t r0 = q.r0[b], o = q.o[b];
  const size_t at = ((size_t)b * L64_SPLIT + s) * np;
  const int m = blockIdx.z * L64_NT + tid;
  if (m < np) {
    double acc = 0.0;
    unsigned long long mx = 0;
    if (m < q.ne) {
#pragma unroll 8
      for (int l = l0; l < l1; l++) {
        const double v = q.sw[o + l] * l64_row(q, r0 + l, m);
        acc = fma(v, q.ed[o + l], acc);
        const unsigned long long bits = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
        mx = bits > mx ? bits : mx;
      }
    }
    pb[at + m] = acc;
    pm[at + m] = mx;
  }
  if (blockIdx.z > 0) return;
  double p1 = 0.0, p3 = 0.0;
  for (int l = l0 + tid; l < l1; l += L64_NT) {
    p1 += q.ed[o + l] * q.ed[o + l];
    p3 += (double)q.rloc[r0 + l];
  }
  p1 = block_sum<double, L64_NT>(p1, red);
  p3 = block_sum<double, L64_NT>(p3, red);
  if (tid == 0) {
    pp[2 * (b * L64_SPLIT + s)] = p1;
    pp[2 * (b * L64_SPLIT + s) + 1] = p3;
  }
}

__global__ void __launch_bounds__(L64_NT) l64_stats_sum_kernel(int np, const double* pb, const unsigned long long* pm,
                                                               const double* pp, double* bvec, double* scale,
                                                               L64Point* pt) {
  const int b = blockIdx.y, m = blockIdx.x * L64_NT + threadIdx.x;
  if (m < np) {
    double acc = 0.0;
    unsigned long long mx = 0;
    for (int s = 0; s < L64_SPLIT; s++) {
      const size_t at = ((size_t)b * L64_SPLIT + s) * np + m;
      acc += pb[at];
      mx = pm[at] > mx ? pm[at] : mx;
    }
    bvec[(size_t)b * np + m] = acc;
    scale[(size_t)b * np + m] = oz_scale(mx);
  }
  if (m == 0) {
    double p1 = 0.0, p3 = 0.0;
    for (int s = 0; s < L64_SPLIT; s++) {
      p1 += pp[2 * (b * L64_SPLIT + s)];
      p3 += pp[2 * (b * L64_SPLIT + s) + 1];
    }
    pt[b].p1 = p1;
    pt[b].p3 = p3;
  }
}

// digits of B^T for list entries k0 .. k0 + kc - 1: [point][digit][member][kc],
// 64 entries x 64 members a CTA, turned in shared memory
constexpr int L64_TLD = 66;  // entries of a member's row in the tile: an odd number of words
__global__ void __launch_bounds__(L64_NT) l64_list_digits_kernel(L64Lists q, int np, int k0, int kc,
                                                                 const double* __restrict__ scale, uint16_t* dig) {
  extern __shared__ __align__(16) uint16_t tile[];  // [OZ_D][64][L64_TLD]
  const int b = blockIdx.z, lt = blockIdx.x * 64, m0 = blockIdx.y * 64, tid = threadIdx.x;
  const int L = q.L[b];
  if (k0 + lt >= L) return;
  const int m = tid & 63;
  const double inv55 = m0 + m < q.ne ? 36028797018963968.0 / scale[(size_t)b * np + m0 + m] : 0.0;  // 2^55
  const int64_t r0 = q.r0[b], o = q.o[b];
#pragma unroll 4
  for (int i = 0; i < 16; i++) {
    const int l = (tid >> 6) + 4 * i, e = k0 + lt + l;
    double v = 0.0;
    if (e < L && m0 + m < q.ne) v = q.sw[o + e] * l64_row(q, r0 + e, m0 + m);
    uint16_t d[OZ_D];
    oz_digits(v, inv55, d);
#pragma unroll
    for (int j = 0; j < OZ_D; j++) tile[(j * 64 + m) * L64_TLD + l] = d[j];
  }
  __syncthreads();
  const uint32_t* t32 = reinterpret_cast<const uint32_t*>(tile);
  uint32_t* out = reinterpret_cast<uint32_t*>(dig);
  for (int t = tid; t < OZ_D * 64 * 32; t += L64_NT) {
    const int w = t & 31, r = (t >> 5) & 63, j = t >> 11;
    out[((((size_t)b * OZ_D + j) * np + m0 + r) * kc + lt) / 2 + w] = t32[((j * 64 + r) * L64_TLD) / 2 + w];
  }
}

// G from the lower triangles of its splits, mirrored; c on the diagonal
__global__ void __launch_bounds__(L64_NT) l64_assemble_kernel(int ne, int np, int nsplit, const double* __restrict__ Gp,
                                                              const double* __restrict__ infl_in, double minfl,
                                                              double* A, double* diag) {
  const int b = blockIdx.y, i = blockIdx.x;
  double infl = infl_in[b];
  if (minfl > 0.0 && infl < minfl) infl = minfl;
  const double c = (double)(ne - 1) / infl;
  const size_t mat = (size_t)np * np;
  for (int j = threadIdx.x; j <= i; j += L64_NT) {
    double g = 0.0;
    for (int s = 0; s < nsplit; s++) g += Gp[((size_t)b * nsplit + s) * mat + (size_t)i * np + j];
    if (i == j) {
      diag[(size_t)b * np + i] = g;
      g += c;
    }
    A[b * mat + (size_t)i * np + j] = g;
    A[b * mat + (size_t)j * np + i] = g;
  }
}

// absolute sum and sum of squares of each row of A
__global__ void __launch_bounds__(L64_NT) l64_rows_kernel(int np, const double* __restrict__ A, double* rsum,
                                                          double* rsq) {
  const int b = blockIdx.y, i = blockIdx.x * (L64_NT / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const double* a = A + (size_t)b * np * np + (size_t)i * np;
  double g = 0.0, f = 0.0;
  for (int j = lane; j < np; j += 32) {
    g += fabs(a[j]);
    f = fma(a[j], a[j], f);
  }
  g = warp_sum(g);
  f = warp_sum(f);
  if (lane == 0) {
    rsum[(size_t)b * np + i] = g;
    rsq[(size_t)b * np + i] = f;
  }
}

__global__ void __launch_bounds__(L64_NT) l64_prep_kernel(int ne, int np, const double* __restrict__ rsum,
                                                          const double* __restrict__ rsq,
                                                          const double* __restrict__ diag,
                                                          const double* __restrict__ infl_in, double minfl,
                                                          L64Point* pt, int* skip) {
  __shared__ double red[L64_NT / 32];
  __shared__ double gmx[L64_NT / 32];
  const int b = blockIdx.x, tid = threadIdx.x;
  double infl = infl_in[b];
  if (minfl > 0.0 && infl < minfl) infl = minfl;
  const double c = (double)(ne - 1) / infl;
  double g = 0.0, f2 = 0.0, tr = 0.0;
  bool bad = false;
  for (int i = tid; i < ne; i += L64_NT) {
    g = fmax(g, rsum[(size_t)b * np + i]);
    bad |= !isfinite(rsum[(size_t)b * np + i]);
    f2 += rsq[(size_t)b * np + i];
    tr += diag[(size_t)b * np + i];
  }
  g = warp_max(g);
  if ((tid & 31) == 0) gmx[tid >> 5] = g;
  f2 = block_sum<double, L64_NT>(f2, red);  // (its barriers publish gmx)
  tr = block_sum<double, L64_NT>(tr, red);
  double s = 0.0;
  for (int w = 0; w < L64_NT / 32; w++) s = fmax(s, gmx[w]);
  // c <= 0, or truncation in mtx_eigen possible, or a value that is not finite: the point keeps the core's flag
  const bool sk = __syncthreads_or(bad) || !(c > 0.0) || !(fmin(s, sqrt(f2)) < L64_TRUNC_RATIO * c);
  if (sk) s = 1.0;
  if (tid == 0) {
    L64Point q = pt[b];
    q.s = s;
    q.c = c;
    q.trace = tr;
    q.infl = infl;
    q.lo = 0.9 * c / s;
    q.ka = 1.0;
    q.kb = 0.0;
    q.done = sk;
    q.skip = sk;
    pt[b] = q;
    skip[b] = sk;
  }
}

// Y = A / s, Z = I
__global__ void __launch_bounds__(L64_NT) l64_init_kernel(int np, const double* __restrict__ A, double* Y, double* Z,
                                                          const L64Point* __restrict__ pt) {
  const int b = blockIdx.y;
  const double inv_s = 1.0 / pt[b].s;
  const size_t mat = (size_t)np * np;
  for (size_t t = blockIdx.x * L64_NT + threadIdx.x; t < mat; t += (size_t)gridDim.x * L64_NT) {
    Y[b * mat + t] = A[b * mat + t] * inv_s;
    Z[b * mat + t] = t / np == t % np ? 1.0 : 0.0;
  }
}

// digits of the rows of X, or of ka I - kb X (the step matrix); a warp per row
template <bool STEP>
__global__ void __launch_bounds__(L64_NT) l64_digits_kernel(int np, const double* __restrict__ X,
                                                            const L64Point* __restrict__ pt,
                                                            const int* __restrict__ skip, uint16_t* dig,
                                                            double* scale) {
  const int b = blockIdx.y, i = blockIdx.x * (L64_NT / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (skip[b]) return;
  const double* x = X + (size_t)b * np * np + (size_t)i * np;
  const double ka = STEP ? pt[b].ka : 0.0, kb = STEP ? pt[b].kb : 0.0;
  auto value = [&](double v, int j) { return STEP ? (i == j ? ka : 0.0) - kb * v : v; };
  unsigned long long mx = 0;
  for (int j = 2 * lane; j < np; j += 64) {
    const double2 v = *reinterpret_cast<const double2*>(x + j);
    const unsigned long long b0 =
        (unsigned long long)__double_as_longlong(value(v.x, j)) & 0x7fffffffffffffffull;
    const unsigned long long b1 =
        (unsigned long long)__double_as_longlong(value(v.y, j + 1)) & 0x7fffffffffffffffull;
    mx = b0 > mx ? b0 : mx;
    mx = b1 > mx ? b1 : mx;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = w > mx ? w : mx;
  }
  const double sc = oz_scale(mx), inv55 = 36028797018963968.0 / sc;  // 2^55
  if (lane == 0) scale[(size_t)b * np + i] = sc;
  uint32_t* out = reinterpret_cast<uint32_t*>(dig);
  for (int j = 2 * lane; j < np; j += 64) {
    const double2 v = *reinterpret_cast<const double2*>(x + j);
    uint16_t d0[OZ_D], d1[OZ_D];
    oz_digits(value(v.x, j), inv55, d0);
    oz_digits(value(v.y, j + 1), inv55, d1);
#pragma unroll
    for (int k = 0; k < OZ_D; k++)
      out[((((size_t)b * OZ_D + k) * np + i) * np + j) / 2] = (uint32_t)d0[k] | (uint32_t)d1[k] << 16;
  }
}

// pieces of ||X f - I||_F^2, f = 1 or 1 / s
__global__ void __launch_bounds__(L64_NT) l64_residual_kernel(int np, const double* __restrict__ X,
                                                              const L64Point* __restrict__ pt, int scaled,
                                                              double* part) {
  __shared__ double red[L64_NT / 32];
  const int b = blockIdx.y;
  const size_t mat = (size_t)np * np;
  const double f = scaled ? 1.0 / pt[b].s : 1.0;
  double e2 = 0.0;
  for (size_t t = blockIdx.x * L64_NT + threadIdx.x; t < mat; t += (size_t)L64_PART * L64_NT) {
    const double d = X[b * mat + t] * f - (t / np == t % np ? 1.0 : 0.0);
    e2 = fma(d, d, e2);
  }
  e2 = block_sum<double, L64_NT>(e2, red);
  if (threadIdx.x == 0) part[b * L64_PART + blockIdx.x] = e2;
}

// the step of each point: its coefficients, or skip; counts: points that take
// this step, points that go on after it
__global__ void l64_step_kernel(int nb, const double* __restrict__ part, L64Point* pt, int* skip, int* counts) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nb) return;
  L64Point q = pt[b];
  if (!q.done) {
    double e2 = 0.0;
    for (int i = 0; i < L64_PART; i++) e2 += part[b * L64_PART + i];
    if (!isfinite(e2)) {  // not certified
      q.done = 1;
      skip[b] = 1;
    } else {
      // balanced scale of the step from the lower bound lo of the spectrum of ZY
      // (as ns_scale in FP32): f(a lo) = f(a (1 + d)), d = 0.02
      const double d1 = 1.02;
      const double l = fmin(fmax(q.lo / d1, 0.0), 0.999);
      const double r = sqrt(l);
      const double al = fmax(3.0 * (1.0 - r) / ((1.0 - l * r) * d1), 1.0);
      const double sa = sqrt(al);
      q.ka = 1.5 * sa;
      q.kb = 0.5 * al * sa;
      const double x = al * q.lo, t3 = 3.0 - x;
      q.lo = 0.25 * x * t3 * t3;
      atomicAdd(&counts[0], 1);
      if (e2 < L64_NS_LAST)
        q.done = 1;  // after this step; skip follows at the next one
      else
        atomicAdd(&counts[1], 1);
    }
    pt[b] = q;
  } else {
    skip[b] = 1;
  }
}

// g = Z b, a warp per row
__global__ void __launch_bounds__(L64_NT) l64_matvec_kernel(int np, const double* __restrict__ Z,
                                                            const double* __restrict__ x, double* y) {
  const int b = blockIdx.y, i = blockIdx.x * (L64_NT / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const double* z = Z + (size_t)b * np * np + (size_t)i * np;
  double acc = 0.0;
  for (int j = lane; j < np; j += 32) acc = fma(z[j], x[(size_t)b * np + j], acc);
  acc = warp_sum(acc);
  if (lane == 0) y[(size_t)b * np + i] = acc;
}

// points whose certificate holds: W, wbar = Z g / s, inflation; a warp per row
__global__ void __launch_bounds__(L64_NT) l64_finalize_kernel(int ne, int np, const double* __restrict__ part,
                                                              const double* __restrict__ Z,
                                                              const double* __restrict__ gvec,
                                                              const L64Point* __restrict__ pt,
                                                              const int* __restrict__ which, double* infl,
                                                              float* trans, float* transm, int* status) {
  const int b = blockIdx.y, i = blockIdx.x * (L64_NT / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const L64Point q = pt[b];
  if (q.skip) return;
  double e2 = 0.0;
  for (int k = 0; k < L64_PART; k++) e2 += part[b * L64_PART + k];
  if (!(e2 < L64_CERT_TOL)) return;  // keeps the core's status and identity
  const int p = which[b];
  const double inv_s = 1.0 / q.s;
  if (i < ne) {
    const double* z = Z + (size_t)b * np * np + (size_t)i * np;
    const double coef = sqrt((double)(ne - 1) * inv_s);
    // trans(k, m) = W[k][m] at column-major index m * ne + k (W symmetric)
    float* tr = trans + (size_t)p * ne * ne + (size_t)i * ne;
    double acc = 0.0;
    for (int j = lane; j < ne; j += 32) {
      acc = fma(z[j], gvec[(size_t)b * np + j], acc);
      tr[j] = (float)(coef * z[j]);
    }
    acc = warp_sum(acc);
    if (transm && lane == 0) transm[(size_t)p * ne + i] = (float)(acc * inv_s);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    infl[p] = infl_update(ne, q.infl, q.p1, q.trace, q.p3);
    status[p] = LETKF_OK;
  }
}

// The FP64 pass over the points whose status is LETKF_ERR_EIG or
// LETKF_ERR_CAPACITY after the mixed-precision core; their parm_infl is still
// the input value.
int largek_fp64_pass(int ne, int npts, const int64_t* offs, const float* rows, const __nv_bfloat16* rows16,
                     const int* ridx, const float* rdiag, const float* rloc, const float* dep, double* parm_infl,
                     float* trans, float* transm, int rdiag_wloc, double minfl, int* status, cudaStream_t s) {
  std::vector<int> st(npts);
  std::vector<int64_t> ho(npts + 1);
  cudaMemcpyAsync(st.data(), status, sizeof(int) * npts, cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(ho.data(), offs, sizeof(int64_t) * (npts + 1), cudaMemcpyDeviceToHost, s);
  int rc = cuda_status(cudaStreamSynchronize(s));
  if (rc != LETKF_OK) return rc;
  std::vector<int> todo;
  for (int p = 0; p < npts; p++)
    if ((st[p] == LETKF_ERR_EIG || st[p] == LETKF_ERR_CAPACITY) && ho[p + 1] > ho[p]) todo.push_back(p);
  if (todo.empty()) return LETKF_OK;
  const int np = (ne + OZ_TILE - 1) / OZ_TILE * OZ_TILE, nt = np / OZ_TILE;
  const size_t mat = (size_t)np * np;
  const int R = (int)std::min<size_t>(todo.size(), 32);  // points per group
  // list entries of a group, at most, and of its longest list
  int64_t emax = 0;
  int lmax = 0;
  for (size_t g0 = 0; g0 < todo.size(); g0 += R) {
    int64_t e = 0;
    for (size_t j = g0; j < std::min(todo.size(), g0 + R); j++) {
      const int64_t L = ho[todo[j] + 1] - ho[todo[j]];
      e += L;
      lmax = std::max(lmax, (int)L);
    }
    emax = std::max(emax, e);
  }
  // chunk of the lists whose digits are held at a time; CTAs enough for two
  // waves by splitting K where the points of a group alone are too few
  int kc = (int)std::min<size_t>(L64_DIGITS / (2 * OZ_D * (size_t)np * R) / OZ_KEXACT * OZ_KEXACT, 1 << 20);
  kc = std::max(std::min(kc, (lmax + OZ_KEXACT - 1) / OZ_KEXACT * OZ_KEXACT), OZ_KEXACT);
  int nsm = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int nsplit = std::max(1, std::min(8, 2 * nsm / (R * nt * (nt + 1) / 2)));
  double *Gp = nullptr, *A = nullptr, *Y = nullptr, *Z = nullptr, *T = nullptr, *TT = nullptr;
  uint16_t *dl = nullptr, *dz = nullptr, *dy = nullptr, *dm = nullptr, *dt = nullptr;
  double *sw = nullptr, *ed = nullptr, *pb = nullptr, *pp = nullptr, *vec = nullptr, *part = nullptr, *pinf = nullptr;
  unsigned long long* pm = nullptr;
  int64_t* r0 = nullptr;
  int *Ls = nullptr, *counts = nullptr, *which = nullptr, *skip = nullptr;
  L64Point* pt = nullptr;
  std::vector<void*> held;
  bool okm = true;
  auto alloc = [&](auto** p, size_t bytes) {
    okm = okm && cudaMallocAsync((void**)p, bytes, s) == cudaSuccess;
    if (okm) held.push_back(*p);
  };
  alloc(&Gp, sizeof(double) * mat * R * nsplit);
  for (double** p : {&A, &Y, &Z, &T, &TT}) alloc(p, sizeof(double) * mat * R);
  alloc(&dl, sizeof(uint16_t) * OZ_D * (size_t)np * kc * R);
  for (uint16_t** p : {&dz, &dy, &dm, &dt}) alloc(p, sizeof(uint16_t) * OZ_D * mat * R);
  alloc(&sw, sizeof(double) * (size_t)emax);
  alloc(&ed, sizeof(double) * (size_t)emax);
  alloc(&pb, sizeof(double) * (size_t)np * R * L64_SPLIT);
  alloc(&pm, sizeof(double) * (size_t)np * R * L64_SPLIT);
  alloc(&pp, sizeof(double) * 2 * R * L64_SPLIT);
  alloc(&vec, sizeof(double) * (size_t)np * R * 9);
  alloc(&part, sizeof(double) * R * L64_PART);
  alloc(&pinf, sizeof(double) * R);
  alloc(&r0, sizeof(int64_t) * 2 * R);
  alloc(&Ls, sizeof(int) * R);
  alloc(&counts, sizeof(int) * 2);
  alloc(&which, sizeof(int) * R);
  alloc(&skip, sizeof(int) * R);
  alloc(&pt, sizeof(L64Point) * R);
  rc = okm ? LETKF_OK : LETKF_ERR_CUDA;
  const size_t vs = (size_t)np * R;
  double *bvec = vec, *gvec = vec + vs, *diag = vec + 2 * vs, *rsum = vec + 3 * vs, *rsq = vec + 4 * vs;
  double *sl = vec + 5 * vs, *sz = vec + 6 * vs, *sy = vec + 7 * vs, *sm = vec + 8 * vs;
  double* sT = rsum;  // row sums are done with by then
  static std::atomic<uint32_t> attr{0};
  const size_t tile_bytes = sizeof(uint16_t) * OZ_D * 64 * L64_TLD;
  if (rc == LETKF_OK) rc = cuda_status(set_smem_once(l64_list_digits_kernel, tile_bytes, attr));

  L64Lists q;
  memset(&q, 0, sizeof(q));
  q.r0 = r0;
  q.L = Ls;
  q.o = r0 + R;
  q.rows = rows;
  q.rows16 = rows16;
  q.ridx = ridx;
  q.rdiag = rdiag;
  q.rloc = rloc;
  q.dep = dep;
  q.ne = ne;
  q.wloc = rdiag_wloc;
  q.sw = sw;
  q.ed = ed;
  OzGemm g;
  memset(&g, 0, sizeof(g));
  g.n = np;
  g.obatch = (int64_t)mat;
  g.nsplit = 1;
  // out = X Y from digit sets of X's rows and of Y's columns
  auto product = [&](const uint16_t* da, const double* sa, const uint16_t* db, const double* sb, double* out,
                     double* outT, bool sym, int nb) {
    OzGemm h = g;
    h.K = np;
    h.A = da;
    h.sa = sa;
    h.B = db;
    h.sb = sb;
    h.out = out;
    h.outT = outT;
    h.lower = h.mirror = sym;
    h.skip = skip;
    return oz_gemm(h, nb, s);
  };
  // sources of the group's copies: written again only after the group's last synchronisation
  std::vector<int64_t> hr(2 * R, 0);
  std::vector<int> hL(R, 0);
  for (size_t g0 = 0; g0 < todo.size() && rc == LETKF_OK; g0 += R) {
    const int nb = (int)std::min<size_t>(R, todo.size() - g0);
    const dim3 rg(np / (L64_NT / 32), nb);
    int64_t o = 0;
    int gl = 0;
    for (int j = 0; j < nb; j++) {
      const int p = todo[g0 + j];
      hr[j] = ho[p];
      hr[R + j] = o;
      hL[j] = (int)(ho[p + 1] - ho[p]);
      o += hL[j];
      gl = std::max(gl, hL[j]);
      cudaMemcpyAsync(pinf + j, parm_infl + p, sizeof(double), cudaMemcpyDeviceToDevice, s);
    }
    cudaMemcpyAsync(which, todo.data() + g0, sizeof(int) * nb, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(r0, hr.data(), sizeof(int64_t) * 2 * R, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(Ls, hL.data(), sizeof(int) * nb, cudaMemcpyHostToDevice, s);
    // 1. Gram and the sums of the lists
    l64_weight_kernel<<<dim3((gl + 255) / 256, nb), 256, 0, s>>>(q);
    l64_stats_kernel<<<dim3(L64_SPLIT, nb, (np + L64_NT - 1) / L64_NT), L64_NT, 0, s>>>(q, np, pb, pm, pp);
    l64_stats_sum_kernel<<<dim3((np + L64_NT - 1) / L64_NT, nb), L64_NT, 0, s>>>(np, pb, pm, pp, bvec, sl, pt);
    note_launch();
    note_launch();
    note_launch();
    cudaMemsetAsync(Gp, 0, sizeof(double) * mat * nb * nsplit, s);
    for (int k0 = 0; k0 < gl && rc == LETKF_OK; k0 += kc) {
      l64_list_digits_kernel<<<dim3((std::min(kc, gl - k0) + 63) / 64, nt, nb), L64_NT, tile_bytes, s>>>(q, np, k0, kc,
                                                                                                       sl, dl);
      note_launch();
      OzGemm h = g;
      h.K = kc;
      h.A = h.B = dl;
      h.sa = h.sb = sl;
      h.out = Gp;
      h.obatch = (int64_t)mat * nsplit;
      h.osplit = (int64_t)mat;
      h.nsplit = nsplit;
      h.lower = 1;
      h.accumulate = 1;
      h.len = Ls;
      h.k0 = k0;
      rc = oz_gemm(h, nb, s);
    }
    if (rc != LETKF_OK) break;
    // 2. A, s, Y, Z
    l64_assemble_kernel<<<dim3(np, nb), L64_NT, 0, s>>>(ne, np, nsplit, Gp, pinf, minfl, A, diag);
    l64_rows_kernel<<<rg, L64_NT, 0, s>>>(np, A, rsum, rsq);
    l64_prep_kernel<<<nb, L64_NT, 0, s>>>(ne, np, rsum, rsq, diag, pinf, minfl, pt, skip);
    l64_init_kernel<<<dim3(64, nb), L64_NT, 0, s>>>(np, A, Y, Z, pt);
    for (int i = 0; i < 4; i++) note_launch();
    // 3. coupled Newton-Schulz; the first T = Z Y is Y
    for (int it = 0; it < L64_NS_MAX && rc == LETKF_OK; it++) {
      const double *t = T, *tt = TT;
      if (it) {
        l64_digits_kernel<false><<<rg, L64_NT, 0, s>>>(np, Z, pt, skip, dz, sz);
        l64_digits_kernel<false><<<rg, L64_NT, 0, s>>>(np, Y, pt, skip, dy, sy);
        note_launch();
        note_launch();
        rc = product(dz, sz, dy, sy, T, TT, false, nb);
        if (rc != LETKF_OK) break;
      } else {
        t = tt = Y;
      }
      l64_residual_kernel<<<dim3(L64_PART, nb), L64_NT, 0, s>>>(np, t, pt, 0, part);
      cudaMemsetAsync(counts, 0, sizeof(int) * 2, s);
      l64_step_kernel<<<(nb + 31) / 32, 32, 0, s>>>(nb, part, pt, skip, counts);
      note_launch();
      note_launch();
      int hc[2] = {0, 0};
      cudaMemcpyAsync(hc, counts, sizeof(hc), cudaMemcpyDeviceToHost, s);
      rc = cuda_status(cudaStreamSynchronize(s));
      if (rc != LETKF_OK || hc[0] == 0) break;
      if (it == 0) {
        l64_digits_kernel<false><<<rg, L64_NT, 0, s>>>(np, Z, pt, skip, dz, sz);
        l64_digits_kernel<false><<<rg, L64_NT, 0, s>>>(np, Y, pt, skip, dy, sy);
        note_launch();
        note_launch();
      }
      l64_digits_kernel<true><<<rg, L64_NT, 0, s>>>(np, t, pt, skip, dm, sm);
      note_launch();
      if (hc[1] > 0) {  // Y <- Y M, from the rows of Y and the columns of M
        l64_digits_kernel<true><<<rg, L64_NT, 0, s>>>(np, tt, pt, skip, dt, sT);
        note_launch();
        rc = product(dy, sy, dt, sT, Y, nullptr, true, nb);
      }
      if (rc == LETKF_OK) rc = product(dm, sm, dz, sz, Z, nullptr, true, nb);  // Z <- M Z
      if (hc[1] == 0) break;
    }
    if (rc != LETKF_OK) break;
    // 4. certificate against A: Q = Z (A Z), then W, wbar, inflation
    cudaMemsetAsync(skip, 0, sizeof(int) * nb, s);
    l64_digits_kernel<false><<<rg, L64_NT, 0, s>>>(np, A, pt, skip, dm, sm);
    l64_digits_kernel<false><<<rg, L64_NT, 0, s>>>(np, Z, pt, skip, dz, sz);
    rc = product(dm, sm, dz, sz, T, TT, false, nb);
    if (rc != LETKF_OK) break;
    l64_digits_kernel<false><<<rg, L64_NT, 0, s>>>(np, TT, pt, skip, dt, sT);
    rc = product(dz, sz, dt, sT, Y, nullptr, true, nb);
    if (rc != LETKF_OK) break;
    l64_residual_kernel<<<dim3(L64_PART, nb), L64_NT, 0, s>>>(np, Y, pt, 1, part);
    l64_matvec_kernel<<<rg, L64_NT, 0, s>>>(np, Z, bvec, gvec);
    l64_finalize_kernel<<<rg, L64_NT, 0, s>>>(ne, np, part, Z, gvec, pt, which, parm_infl, trans, transm, status);
    for (int i = 0; i < 6; i++) note_launch();
    rc = cuda_status(cudaStreamSynchronize(s));
  }
  for (void* p : held) cudaFreeAsync(p, s);
  const int rc2 = cuda_status(cudaStreamSynchronize(s));
  return rc != LETKF_OK ? rc : rc2;
}

}  // namespace letkf
