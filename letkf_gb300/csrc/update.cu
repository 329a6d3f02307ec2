// update.cu -- ensemble update with the analysis weights (FP64 plain form) and
// the relaxed update of the SCALE driver.
//
//   mean(p,v) = (x(p,1,v) + ... + x(p,ne,v)) / ne      speedy/common/common_speedy.f90:335-370
//   xa(p,m,v) = mean + sum_k (x(p,k,v) - mean) * (trans(k,m) + transm(k))
//                                                     speedy/letkf/letkf_tools.f90:164-170,
//                                                     scale/letkf/letkf_tools.f90:237-251 (beta = 1)
// and with relaxation (scale/letkf/letkf_tools.f90:215-268), per point and
// variable, W_rlx = RTPP (1-a) W + a I (:1224-1237) or RTPS infl W with infl =
// a sqrt(var_g / (var_a (k-1))) - a + 1 (:1240-1268), T = (W_rlx + transm 1^T)
// beta + (1 - beta) I, xa = mean + xb' T; beta == 0 leaves mean + xb'; optional
// clipping of the relative spread of one variable (Q_SPRD_MAX).
//
// update_f64_kernel has one CTA per point and serves both entry points (mode 0
// where beta is 1, no array or an element of it, is the plain update bit for
// bit); forms for few members, few variables or few points follow it, with the
// same operations in the same order.  The factors that do not depend on k stay out
// of the sum: t(m) = sum_k x(k) W(k,m) and sum_k x(k) transm(k) once, then xa =
// mean + beta (fac t + tx) + (1 - beta) x(m): one multiply-add per element of W and
// variable where forming each weight first took five FP64 operations, and
// increments added up before they meet the mean, in every form: with the mean
// first each of k additions rounds at its size (error of the plain update against exact arithmetic, merged weights, of the rms
// value: k = 8 1.5e-16 so and 8.1e-17 here, k = 40 2.9e-16 and 9.4e-17, k = 100 4.3e-16
// and 1.3e-16).
//
// Bound: the FP64 pipe (1.2 TFLOP/s; a warp instruction takes 16 cycles of an
// SM), so lanes are kept full: outputs (variable, member) are flattened over
// the lanes, W is kept k-major with an odd row length (consecutive lanes read
// consecutive members and the transposing stores spread over the banks), and
// the quadratic form of RTPS goes over unordered pairs: x' Pa x = sum_d sum_i
// x(i) D(d,i) x(i+d mod k), D(d,i) = Pa(i,i+d) + Pa(i+d,i), d = 0..k/2, formed
// once per point for all variables, half the products of the full form and
// every lane busy.  RTPS, 20,000 points, k = 50, 11 variables: 7.77 -> 2.53 ms.
#include <algorithm>

#include "letkf_common.cuh"

namespace letkf {

constexpr int UPD_NT = 128;
constexpr int UPD_VC = 16;  // variables handled at a time, at most

struct RelaxArgs {
  int mode;           // 0 none, 1 RTPP, 2 RTPS
  double alpha;
  const double* beta; // [nv][npts] or NULL (1)
  int q_var;          // variable index of the spread clip, -1 none
  double q_sprd_max;  // <= 0: off
  double* rtps_infl;  // [nv][npts] or NULL
};

// doubles of shared memory: W, D (RTPS), transm, x and the products of a chunk
// of variables, mean / factor / beta / x . transm, the clipped variable
static size_t upd_smem_doubles(int n, int vc, int mode) {
  const size_t d = mode == 2 ? (size_t)(n / 2 + 1) * n + (size_t)vc * n : 0;
  return (size_t)n * (n | 1) + d + n + (size_t)vc * n + 4 * (size_t)vc + n;
}

// a[u] += sum_k x(v_u, k) W(k, m_u) for the first N of a thread's outputs (mm: offset of member m_u)
template <int N, int U>
__device__ __forceinline__ void upd_sums(int n, int sk, const double* xp, const double* W, const int (&vv)[U],
                                         const int (&mm)[U], double (&a)[U]) {
#pragma unroll(N == 1 ? 8 : 4)
  for (int k = 0; k < n; k++)
#pragma unroll
    for (int u = 0; u < N; u++) a[u] = fma(xp[vv[u] * n + k], W[k * sk + mm[u]], a[u]);
}

// Points p0 .. p0+cnt-1 of arrays holding npts points; trans / transm / pao
// are indexed from p0; CAP variables at a time.  MODE and BETA (r.beta given)
// are compiled in: an operation that is only predicated off still takes its FP64
// slot; CAP is because a loop of unknown step costs up to 7 % (k = 50, one
// variable, beta given, 6,000 points: 88 us with it compiled in, 95 without).
template <int MODE, bool BETA, int CAP>
__global__ void __launch_bounds__(UPD_NT) update_f64_kernel(int n, int npts, int p0, int cnt, int nv,
                                                             const double* __restrict__ xb,
                                                             const double* __restrict__ trans,
                                                             const double* __restrict__ transm,
                                                             const double* __restrict__ pao, RelaxArgs r, double* xa) {
  extern __shared__ __align__(16) double su[];
  const int ld = n | 1, nh = n / 2, vcm = nv < CAP ? nv : CAP;
  // W(k, m) at k sk + m sm: as in memory, or transposed where the row length
  // would put the lanes' members on few banks
  const bool tr = n % 16 == 0;
  const int sk = tr ? ld : 1, sm = tr ? 1 : n;
  double* W = su;
  double* D = W + (size_t)n * ld;          // [nh + 1][n] (RTPS)
  double* prod = D + (MODE == 2 ? (size_t)(nh + 1) * n : 0);  // [vcm][n] (RTPS)
  double* tm = prod + (MODE == 2 ? (size_t)vcm * n : 0);      // [n]
  double* xp = tm + n;                     // [vcm][n]
  double* mean = xp + (size_t)vcm * n;     // [vcm] each
  double* fac = mean + vcm;
  double* bet = fac + vcm;
  double* tx = bet + vcm;
  double* qv = tx + vcm;                   // [n]
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int pl = blockIdx.x; pl < cnt; pl += gridDim.x) {
    const int p = p0 + pl;
    __syncthreads();
    const double* Tp = trans + (size_t)pl * n * n;
    if (tr) {
#pragma unroll 4
      for (int idx = tid; idx < n * n; idx += UPD_NT) {
        const int m = idx / n, k = idx - m * n;
        W[k * ld + m] = Tp[idx];
      }
    } else {
#pragma unroll 4
      for (int idx = tid; idx < n * n; idx += UPD_NT) W[idx] = Tp[idx];
    }
    if (transm)
      for (int k = tid; k < n; k += UPD_NT) tm[k] = transm[(size_t)pl * n + k];
    if (MODE == 2) {
      // first the element of each pair that starts it, then the other one onto it
      const double* Pp = pao + (size_t)pl * n * n;
#pragma unroll 4
      for (int idx = tid; idx < n * n; idx += UPD_NT) {
        const int i = idx / n, j = idx - i * n;
        const int d = j >= i ? j - i : j - i + n;
        if (2 * d < n || (2 * d == n && i < j)) D[d * n + i] = Pp[idx];
        if (2 * d == n && i > j) D[d * n + i] = 0.0;
      }
      __syncthreads();
#pragma unroll 4
      for (int idx = tid; idx < n * n; idx += UPD_NT) {
        const int i = idx / n, j = idx - i * n;
        const int d = i >= j ? i - j : i - j + n;
        if (d != 0 && (2 * d < n || (2 * d == n && j < i))) D[d * n + j] += Pp[idx];
      }
    }
    for (int v0 = 0; v0 < nv; v0 += CAP) {
      const int vc = min(CAP, nv - v0), total = vc * n;
      if (v0) __syncthreads();
      for (int t = tid; t < total; t += UPD_NT) {
        const int v = t / n;
        xp[t] = xb[((size_t)(v0 + v) * npts + p) * n + (t - v * n)];
      }
      __syncthreads();
      for (int v = tid; v < vc; v += UPD_NT) {
        double s = xp[v * n];
        for (int m = 1; m < n; m++) s = s + xp[v * n + m];
        mean[v] = s / (double)n;
        if (BETA) bet[v] = r.beta[(size_t)(v0 + v) * npts + p];
        fac[v] = 1.0;
      }
      __syncthreads();
      for (int t = tid; t < total; t += UPD_NT) xp[t] = xp[t] - mean[t / n];
      __syncthreads();
      const int nch = (total + 31) / 32;  // 32 outputs (variable, member) a chunk, chunks over the warps
      if (MODE == 2) {
        for (int c = wid; c < nch; c += UPD_NT / 32) {
          const int t = min(32 * c + lane, total - 1);
          const int v = t / n, i = t - v * n;
          const double* x = xp + v * n;
          double a = 0.0;
          int j = i;
#pragma unroll 4
          for (int d = 0; d <= nh; d++) {
            a = fma(D[d * n + i], x[j], a);
            j = j + 1 == n ? 0 : j + 1;
          }
          if (32 * c + lane < total) prod[t] = a * x[i];
        }
        __syncthreads();
      }
      // sums over the members by eight lanes per variable (a full warp would
      // spend more FP64 slots on the reduction than on the sum)
      if (transm || MODE == 2) {
        for (int vb = 4 * wid; vb < vc; vb += UPD_NT / 8) {
          const int v = min(vb + (lane >> 3), vc - 1);
          const double* x = xp + v * n;
          double sx = 0.0, va = 0.0, vg = 0.0;
          if (transm)
            for (int k = lane & 7; k < n; k += 8) sx = fma(x[k], tm[k], sx);
          if (MODE == 2)
            for (int k = lane & 7; k < n; k += 8) {
              va = va + prod[v * n + k];
              vg = fma(x[k], x[k], vg);
            }
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) {
            if (transm) sx += __shfl_xor_sync(0xffffffffu, sx, o);
            if (MODE == 2) {
              va += __shfl_xor_sync(0xffffffffu, va, o);
              vg += __shfl_xor_sync(0xffffffffu, vg, o);
            }
          }
          if ((lane & 7) == 0 && vb + (lane >> 3) < vc) {
            tx[v] = sx;
            if (MODE == 2) {  // beta == 0 skips weight_RTPS (factor 1)
              double f = 1.0;
              if ((!BETA || bet[v] != 0.0) && vg > 0.0 && va > 0.0)
                f = r.alpha * sqrt(vg / (va * (double)(n - 1))) - r.alpha + 1.0;
              fac[v] = f;
              if (r.rtps_infl) r.rtps_infl[(size_t)(v0 + v) * npts + p] = f;
            }
          }
        }
      }
      if (transm || MODE == 2) __syncthreads();
      const bool clip = r.q_sprd_max > 0.0 && r.q_var >= v0 && r.q_var < v0 + vc;
      constexpr int U = 4;
      for (int c0 = wid; c0 < nch; c0 += U * (UPD_NT / 32)) {
        const int nu = min(U, (nch - c0 + UPD_NT / 32 - 1) / (UPD_NT / 32));
        double a[U];
        int vv[U], mm[U], off[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int t = min(32 * (c0 + u * (UPD_NT / 32)) + lane, total - 1);
          vv[u] = t / n;
          mm[u] = t - vv[u] * n;
          a[u] = 0.0;
          off[u] = mm[u] * sm;
        }
        // one loop per count: a multiply-add that is only predicated off takes its FP64 slot
        if (nu == 4)
          upd_sums<4>(n, sk, xp, W, vv, off, a);
        else if (nu == 3)
          upd_sums<3>(n, sk, xp, W, vv, off, a);
        else if (nu == 2)
          upd_sums<2>(n, sk, xp, W, vv, off, a);
        else
          upd_sums<1>(n, sk, xp, W, vv, off, a);
#pragma unroll
        for (int u = 0; u < U; u++) {
          if (u >= nu || 32 * (c0 + u * (UPD_NT / 32)) + lane >= total) continue;
          const int v = vv[u], m = mm[u];
          const double x = xp[v * n + m];
          double inc = a[u];
          if (MODE == 1) inc = (1.0 - r.alpha) * inc + r.alpha * x;
          if (MODE == 2) inc = fac[v] * inc;
          if (transm) inc = inc + tx[v];
          if (BETA) {
            const double b = bet[v];
            inc = b == 0.0 ? x : b == 1.0 ? inc : b * inc + (1.0 - b) * x;
          }
          const double y = mean[v] + inc;
          if (clip && v0 + v == r.q_var)
            qv[m] = y;
          else
            xa[((size_t)(v0 + v) * npts + p) * n + m] = y;
        }
      }
      if (clip) {
        __syncthreads();
        if (wid == 0) {
          double s = 0.0;
          for (int m = lane; m < n; m += 32) s = s + qv[m];
          const double qm = warp_sum(s) / (double)n;
          double sp = 0.0;
          for (int m = lane; m < n; m += 32) sp = fma(qv[m] - qm, qv[m] - qm, sp);
          sp = sqrt(warp_sum(sp) / (double)(n - 1)) / qm;
          const double f = r.q_sprd_max / sp;
          for (int m = lane; m < n; m += 32) {
            double y = qv[m];
            if (sp > r.q_sprd_max) y = qm + (y - qm) * f;
            xa[((size_t)r.q_var * npts + p) * n + m] = y;
          }
        }
      }
    }
  }
}

// The plain update of more variables than the rows kernel below takes: a CTA per
// point, a thread per output.  TM: transm given, its product with x formed as in
// the general kernel; the results of both are the same bits.  The general
// kernel's extra passes and barriers cost more than what it leaves out of the
// sums saves (320 MB of weights, at most 20,000 points, merged: k = 20, 7
// variables 172 us here and 190 there, k = 33, 4 variables 257 and 270, k = 46, 8
// variables 648 and 682; with transm k = 2..8, 5 variables 0.84 to 0.95 of the time
// of a thread per output with W + transm formed in its sum, and 1.08 to 1.40
// there).  Bound: the FP64 pipe.  W lies as in memory, or transposed where the
// row length would put the lanes' members on two banks or one (k = 40, 4
// variables: 360 -> 305 us; from k = 100, two CTAs an SM, the transposing stores
// are no longer hidden and only the latter is worth them).  The points are handed
// out by the hardware: a grid of 8 CTAs an SM in fixed strides ends with its last
// CTAs alone where 8 are not resident (k = 60, 4 variables: 450 us so, 360 here).
template <bool TM>
__global__ void __launch_bounds__(UPD_NT) update_point_kernel(int n, int npts, int p0, int cnt, int nv, int vcm,
                                                              const double* __restrict__ xb,
                                                              const double* __restrict__ trans,
                                                              const double* __restrict__ transm, double* xa) {
  extern __shared__ __align__(16) double su[];
  const int ld = n | 1;
  const bool tr = n % 16 == 0 || (n % 8 == 0 && n < 100);
  const int sk = tr ? ld : 1, sm = tr ? 1 : n;  // W(k, m) at k sk + m sm
  double* W = su;
  double* xp = W + (size_t)n * ld;      // [vcm][n]
  double* mean = xp + (size_t)vcm * n;  // [vcm] each
  double* tx = mean + vcm;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int pl = blockIdx.x; pl < cnt; pl += gridDim.x) {
    const int p = p0 + pl;
    __syncthreads();
    const double* Tp = trans + (size_t)pl * n * n;
    if (tr) {
      for (int idx = tid; idx < n * n; idx += UPD_NT) {
        const int m = idx / n, k = idx - m * n;
        W[k * ld + m] = Tp[idx];
      }
    } else {
      for (int idx = tid; idx < n * n; idx += UPD_NT) W[idx] = Tp[idx];
    }
    for (int v0 = 0; v0 < nv; v0 += vcm) {
      const int vc = min(vcm, nv - v0), total = vc * n;
      if (v0) __syncthreads();
      for (int t = tid; t < total; t += UPD_NT) {
        const int v = t / n;
        xp[t] = xb[((size_t)(v0 + v) * npts + p) * n + (t - v * n)];
      }
      __syncthreads();
      for (int v = tid; v < vc; v += UPD_NT) {
        double s = xp[v * n];
        for (int m = 1; m < n; m++) s = s + xp[v * n + m];
        mean[v] = s / (double)n;
      }
      __syncthreads();
      for (int t = tid; t < total; t += UPD_NT) xp[t] = xp[t] - mean[t / n];
      __syncthreads();
      if (TM) {
        const double* tm = transm + (size_t)pl * n;
        for (int vb = 4 * wid; vb < vc; vb += UPD_NT / 8) {
          const int v = min(vb + (lane >> 3), vc - 1);
          double sx = 0.0;
          for (int k = lane & 7; k < n; k += 8) sx = fma(xp[v * n + k], tm[k], sx);
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) sx += __shfl_xor_sync(0xffffffffu, sx, o);
          if ((lane & 7) == 0 && vb + (lane >> 3) < vc) tx[v] = sx;
        }
        __syncthreads();
      }
      for (int t = tid; t < total; t += UPD_NT) {
        const int v = t / n, m = t - v * n;
        const double *x = xp + v * n, *w = W + m * sm;
        double a = 0.0;
        for (int k = 0; k < n; k++) a = fma(x[k], w[k * sk], a);
        if (TM) a = a + tx[v];
        xa[((size_t)(v0 + v) * npts + p) * n + m] = mean[v] + a;
      }
    }
  }
}

template <bool TM>
static int launch_update_point(int ne, int npts, int p0, int cnt, int nv, const double* xb, const double* trans,
                               const double* transm, double* xa, cudaStream_t stream) {
  // a pass of 16 variables, or of 1,024 outputs where that is more; all of them where no fewer CTAs share an SM then
  // (k = 100, 20 variables, merged, 3,000 points: 1,250 us in passes of 16 and 4, 1,163 in one)
  auto bytes = [&](int vc) { return sizeof(double) * ((size_t)ne * (ne | 1) + (size_t)vc * ne + 2 * vc); };
  auto per_sm = [&](int vc) { return 227 * 1024 / (bytes(vc) + 1024); };
  int vc = std::min(nv, std::max(UPD_VC, 1024 / ne));
  if (nv <= 2 * UPD_VC && per_sm(nv) == per_sm(vc)) vc = nv;
  const size_t smem = bytes(vc);
  auto kern = update_point_kernel<TM>;
  const cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (err != cudaSuccess) return cuda_status(err);
  kern<<<cnt, UPD_NT, smem, stream>>>(ne, npts, p0, cnt, nv, vc, xb, trans, transm, xa);
  note_launch();
  return cuda_status(cudaGetLastError());
}

// The plain update of few variables: a warp per batch of rows (variable,
// point), no barrier.  Each lane reads its member's row of trans straight from
// global memory, 64 consecutive bytes at a time where rows are 16-byte aligned;
// x stays in shared memory, no more of it than the batch needs, because the
// rest of the SM's 256 KB is the L1 that holds the lines the lanes are in the
// middle of (with room for 16 rows always: k = 100 0.72 ms instead of 0.27).
// What bounds it is FP64 slots beside the k products of an output: a
// member-order mean costs as many as the products when one lane does it alone,
// so lanes take the rows of the batch.  One variable, 100,000 points of k = 32:
// 0.57 -> 0.22 ms, 20,000 of k = 50: 0.22 -> 0.16, 4,000 of k = 128: 0.75 ->
// 0.16 (before: a CTA per point).  The sums are those of the kernels above in
// the same order, so the results are the same bits.
constexpr int UPR_ROWS = 16;

template <int NVT, bool VEC>
__global__ void __launch_bounds__(UPD_NT, 8) update_rows_kernel(int n, int npts, int p0, int cnt, int pb,
                                                                const double* __restrict__ xb,
                                                                const double* __restrict__ trans,
                                                                const double* __restrict__ transm, double* xa) {
  // pb points of NVT rows each in a batch
  extern __shared__ __align__(16) double su[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, ld = n | 1;
  double* xs = su + (size_t)wid * pb * NVT * (ld + 2);  // [point][variable][ld]
  double* tx = xs + pb * NVT * ld;                      // [point][variable] each
  double* ms = tx + pb * NVT;
  const int nbatch = (cnt + pb - 1) / pb;
  for (int b = blockIdx.x * (UPD_NT / 32) + wid; b < nbatch; b += gridDim.x * (UPD_NT / 32)) {
    const int q0 = b * pb, nq = min(pb, cnt - q0), nr = nq * NVT;
    __syncwarp();
    for (int r = 0; r < nr; r++) {
      const double* src = xb + ((size_t)(r % NVT) * npts + p0 + q0 + r / NVT) * n;
      for (int m = lane; m < n; m += 32) xs[r * ld + m] = src[m];
    }
    __syncwarp();
    double mean = 0.0;
    if (lane < nr) {
      const double* x = xs + lane * ld;
      double s = x[0];
      for (int m = 1; m < n; m++) s = s + x[m];
      mean = s / (double)n;
      ms[lane] = mean;
    }
    for (int r = 0; r < nr; r++) {
      const double mr = __shfl_sync(0xffffffffu, mean, r);
      for (int m = lane; m < n; m += 32) xs[r * ld + m] = xs[r * ld + m] - mr;
    }
    __syncwarp();
    if (transm) {
      for (int rb = 0; rb < nr; rb += 4) {
        const int r = min(rb + (lane >> 3), nr - 1);
        const double* t = transm + (size_t)(q0 + r / NVT) * n;
        double sx = 0.0;
        for (int k = lane & 7; k < n; k += 8) sx = fma(xs[r * ld + k], t[k], sx);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) sx += __shfl_xor_sync(0xffffffffu, sx, o);
        if ((lane & 7) == 0 && rb + (lane >> 3) < nr) tx[r] = sx;
      }
      __syncwarp();
    }
    for (int q = 0; q < nq; q++) {
      const double* x = xs + q * NVT * ld;
      for (int m = lane; m < n; m += 32) {
        const double* w = trans + ((size_t)(q0 + q) * n + m) * n;
        double a[NVT];
#pragma unroll
        for (int v = 0; v < NVT; v++) a[v] = 0.0;
        int k = 0;
        if (VEC) {
          for (; k + 8 <= n; k += 8) {
            double2 t[4];
#pragma unroll
            for (int i = 0; i < 4; i++) t[i] = *reinterpret_cast<const double2*>(w + k + 2 * i);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
              for (int v = 0; v < NVT; v++) {
                a[v] = fma(x[v * ld + k + 2 * i], t[i].x, a[v]);
                a[v] = fma(x[v * ld + k + 2 * i + 1], t[i].y, a[v]);
              }
          }
        }
#pragma unroll 4
        for (; k < n; k++) {
          const double t = w[k];
#pragma unroll
          for (int v = 0; v < NVT; v++) a[v] = fma(x[v * ld + k], t, a[v]);
        }
#pragma unroll
        for (int v = 0; v < NVT; v++)
          xa[((size_t)v * npts + p0 + q0 + q) * n + m] = ms[q * NVT + v] + (transm ? a[v] + tx[q * NVT + v] : a[v]);
      }
    }
  }
}

template <int NVT, bool VEC>
static int launch_update_rows(int ne, int npts, int p0, int cnt, const double* xb, const double* trans,
                              const double* transm, double* xa, cudaStream_t stream) {
  static std::atomic<uint32_t> done{0};
  const cudaError_t err = set_smem_once(update_rows_kernel<NVT, VEC>,
                                        sizeof(double) * (UPD_NT / 32) * (size_t)(UPR_ROWS * (LETKF_MAX_NE + 1) + 2 * UPR_ROWS), done);
  if (err != cudaSuccess) return cuda_status(err);
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  // full batches only where every SM then still has two rounds of warps
  int pb = cnt / (nsm * 64);
  pb = pb < 1 ? 1 : pb > UPR_ROWS / NVT ? UPR_ROWS / NVT : pb;
  const size_t smem = sizeof(double) * (UPD_NT / 32) * (size_t)pb * NVT * ((ne | 1) + 2);
  const int need = (cnt + pb * (UPD_NT / 32) - 1) / (pb * (UPD_NT / 32));
  const int grid = need < nsm * 8 ? need : nsm * 8;
  update_rows_kernel<NVT, VEC><<<grid, UPD_NT, smem, stream>>>(ne, npts, p0, cnt, pb, xb, trans, transm, xa);
  note_launch();
  return cuda_status(cudaGetLastError());
}

template <int MODE, bool BETA>
static int launch_update_as(int ne, int npts, int p0, int cnt, int nv, const double* xb, const double* trans,
                            const double* transm, const double* pao, const RelaxArgs& r, double* xa,
                            cudaStream_t stream) {
  // RTPS of k = 128 leaves room for 15 variables beside W and D
  int vc = nv < UPD_VC ? nv : UPD_VC;
  if (sizeof(double) * upd_smem_doubles(ne, vc, MODE) > 227 * 1024) vc = UPD_VC / 2;
  const size_t smem = sizeof(double) * upd_smem_doubles(ne, vc, MODE);
  auto kern = update_f64_kernel<MODE, BETA, UPD_VC>;
  if constexpr (MODE == 2)
    if (vc < nv && vc < UPD_VC) kern = update_f64_kernel<MODE, BETA, UPD_VC / 2>;
  const cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (err != cudaSuccess) return cuda_status(err);
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  // resident CTAs: shared memory, at most 8 (32 warps cover the FP64 unit's latency)
  int per_sm = (int)((size_t)(220 * 1024) / (smem + 1024));
  per_sm = per_sm < 1 ? 1 : per_sm > 8 ? 8 : per_sm;
  const int grid = cnt < nsm * per_sm ? cnt : nsm * per_sm;
  kern<<<grid, UPD_NT, smem, stream>>>(ne, npts, p0, cnt, nv, xb, trans, transm, pao, r, xa);
  note_launch();
  return cuda_status(cudaGetLastError());
}

// Ensembles of two to eight members: a thread per point and variable with its
// members in registers; no barrier, no shared memory.  A CTA per point has eight
// of its 128 lanes busy per variable, and its passes and barriers to pay for.
// Bound: FP64 and, with many variables, the reads of each point's weights by
// every one of them (L1).  100,000 points in us, a thread per output of a CTA per
// point / the kernels above / here: 2 members, 20 variables, mode 0 with a beta
// array 311 / 597 / 93; 4 members, 20 variables, plain with mean weights 295 / 316 /
// 185, RTPS 5,509 / 1,551 / 385; 8 members, 5 variables, RTPP 737 / 404 / 144.  The plain
// update with merged weights has the point kernel from 5 members on where the
// variables are more than 10 (5 members: 5 variables 133 there / 72 here, 20
// 238 / 277; 8 members 216 / 127, 363 / 477).  The operations are those of the
// kernels above in the same order (sums over the members as their lanes add
// them), so the results are the same bits.
constexpr int UPD_TINY = 8;       // members, at most
constexpr int UPD_TINY_MERGED = 4;  // and with merged weights and more than UPD_TINY_NV variables
constexpr int UPD_TINY_NV = 10;
constexpr int UPT_NT = 128;

// x[0] + .. + x[N-1] as the butterfly of eight lanes, or of a warp, adds them
template <int N>
__device__ __forceinline__ double upt_sum(const double (&x)[N]) {
  double t[N < 4 ? N : 4];
#pragma unroll
  for (int i = 0; i < N && i < 4; i++) t[i] = i + 4 < N ? x[i] + x[i + 4 < N ? i + 4 : 0] : x[i];
  if constexpr (N == 2) return t[0] + t[1];
  if constexpr (N == 3) return (t[0] + t[2]) + t[1];
  if constexpr (N >= 4) return (t[0] + t[2]) + (t[1] + t[3]);
}

template <int N, int MODE>
__global__ void __launch_bounds__(UPT_NT) update_tiny_kernel(int npts, int p0, int cnt, int nv,
                                                             const double* __restrict__ xb,
                                                             const double* __restrict__ trans,
                                                             const double* __restrict__ transm,
                                                             const double* __restrict__ pao, RelaxArgs r, double* xa) {
  const int64_t total = (int64_t)cnt * nv;
  for (int64_t t = (int64_t)blockIdx.x * UPT_NT + threadIdx.x; t < total; t += (int64_t)gridDim.x * UPT_NT) {
    const int v = (int)(t / cnt), pl = (int)(t - (int64_t)v * cnt);
    const size_t at = ((size_t)v * npts + p0 + pl) * N;
    double x[N], y[N], s[N];
#pragma unroll
    for (int m = 0; m < N; m++) x[m] = xb[at + m];
    double mean = x[0];
#pragma unroll
    for (int m = 1; m < N; m++) mean = mean + x[m];
    mean = mean / (double)N;
#pragma unroll
    for (int m = 0; m < N; m++) x[m] = x[m] - mean;
    double tx = 0.0;
    if (transm) {
#pragma unroll
      for (int m = 0; m < N; m++) s[m] = __dmul_rn(x[m], transm[(size_t)pl * N + m]);
      tx = upt_sum<N>(s);
    }
    const double b = r.beta ? r.beta[(size_t)v * npts + p0 + pl] : 1.0;
    double fac = 1.0;
    if (MODE == 2) {
      const double* P = pao + (size_t)pl * N * N;
#pragma unroll
      for (int i = 0; i < N; i++) {  // pairs (i, i + d mod N), as the general kernel's D
        double a = 0.0;
#pragma unroll
        for (int d = 0; 2 * d <= N; d++) {
          const int j = (i + d) % N;
          if (2 * d == N && i > j) continue;
          const double dd = d == 0 ? P[i * N + i] : P[i * N + j] + P[j * N + i];
          a = fma(dd, x[j], a);
        }
        s[i] = __dmul_rn(a, x[i]);
      }
      const double va = upt_sum<N>(s);
#pragma unroll
      for (int i = 0; i < N; i++) s[i] = __dmul_rn(x[i], x[i]);
      const double vg = upt_sum<N>(s);
      if (b != 0.0 && vg > 0.0 && va > 0.0) fac = r.alpha * sqrt(vg / (va * (double)(N - 1))) - r.alpha + 1.0;
      if (r.rtps_infl) r.rtps_infl[(size_t)v * npts + p0 + pl] = fac;
    }
    const double* W = trans + (size_t)pl * N * N;  // W(k, m) at m N + k
#pragma unroll
    for (int m = 0; m < N; m++) {
      double a = 0.0;
#pragma unroll
      for (int k = 0; k < N; k++) a = fma(x[k], W[m * N + k], a);
      if (MODE == 1) a = fma(r.alpha, x[m], __dmul_rn(1.0 - r.alpha, a));  // as the compiler has it above
      if (MODE == 2) a = fac * a;
      if (transm) a = a + tx;
      if (r.beta) a = b == 0.0 ? x[m] : b == 1.0 ? a : b * a + (1.0 - b) * x[m];
      y[m] = mean + a;
    }
    if (r.q_sprd_max > 0.0 && v == r.q_var) {
      const double qm = upt_sum<N>(y) / (double)N;
#pragma unroll
      for (int m = 0; m < N; m++) s[m] = __dmul_rn(y[m] - qm, y[m] - qm);
      const double sp = sqrt(upt_sum<N>(s) / (double)(N - 1)) / qm;
      const double f = r.q_sprd_max / sp;
#pragma unroll
      for (int m = 0; m < N; m++)
        if (sp > r.q_sprd_max) y[m] = qm + (y[m] - qm) * f;
    }
#pragma unroll
    for (int m = 0; m < N; m++) xa[at + m] = y[m];
  }
}

template <int MODE>
static int launch_update_tiny(int ne, int npts, int p0, int cnt, int nv, const double* xb, const double* trans,
                              const double* transm, const double* pao, const RelaxArgs& r, double* xa,
                              cudaStream_t stream) {
  decltype(&update_tiny_kernel<2, MODE>) kern = nullptr;
  switch (ne) {
    case 2: kern = update_tiny_kernel<2, MODE>; break;
    case 3: kern = update_tiny_kernel<3, MODE>; break;
    case 4: kern = update_tiny_kernel<4, MODE>; break;
    case 5: kern = update_tiny_kernel<5, MODE>; break;
    case 6: kern = update_tiny_kernel<6, MODE>; break;
    case 7: kern = update_tiny_kernel<7, MODE>; break;
    case 8: kern = update_tiny_kernel<8, MODE>; break;
  }
  const int64_t need = ((int64_t)cnt * nv + UPT_NT - 1) / UPT_NT;
  kern<<<(unsigned)std::min<int64_t>(need, 1 << 20), UPT_NT, 0, stream>>>(npts, p0, cnt, nv, xb, trans, transm, pao, r,
                                                                          xa);
  note_launch();
  return cuda_status(cudaGetLastError());
}

static int launch_update(int ne, int npts, int p0, int cnt, int nv, const double* xb, const double* trans,
                         const double* transm, const double* pao, const RelaxArgs& r, double* xa,
                         cudaStream_t stream) {
#define UPD_AS(MODE)                                                                                             \
  return r.beta ? launch_update_as<MODE, true>(ne, npts, p0, cnt, nv, xb, trans, transm, pao, r, xa, stream) \
                : launch_update_as<MODE, false>(ne, npts, p0, cnt, nv, xb, trans, transm, pao, r, xa, stream)
  if (ne <= UPD_TINY) {
    if (r.mode == 2) return launch_update_tiny<2>(ne, npts, p0, cnt, nv, xb, trans, transm, pao, r, xa, stream);
    if (r.mode == 1) return launch_update_tiny<1>(ne, npts, p0, cnt, nv, xb, trans, transm, pao, r, xa, stream);
    return launch_update_tiny<0>(ne, npts, p0, cnt, nv, xb, trans, transm, pao, r, xa, stream);
  }
  if (r.mode == 2) UPD_AS(2);
  if (r.mode == 1) UPD_AS(1);
  UPD_AS(0);
#undef UPD_AS
}

int launch_update_f64_range(int ne, int npts_total, int p0, int cnt, int nv, const double* xb, const double* trans,
                            const double* transm, double* xa, cudaStream_t stream) {
  if (ne < 2 || npts_total < 0 || p0 < 0 || cnt < 0 || p0 + cnt > npts_total || nv < 1) return LETKF_ERR_ARG;
  if (ne > LETKF_MAX_NE) return LETKF_ERR_CAPACITY;
  if (cnt == 0) return LETKF_OK;
  const RelaxArgs plain = {0, 0.0, nullptr, -1, 0.0, nullptr};
  if (ne <= (transm || nv <= UPD_TINY_NV ? UPD_TINY : UPD_TINY_MERGED))
    return launch_update(ne, npts_total, p0, cnt, nv, xb, trans, transm, nullptr, plain, xa, stream);
  const bool vec = ne % 2 == 0 && reinterpret_cast<uintptr_t>(trans) % 16 == 0;
#define UPR_LAUNCH(NVT)                                                                                 \
  return vec ? launch_update_rows<NVT, true>(ne, npts_total, p0, cnt, xb, trans, transm, xa, stream) \
             : launch_update_rows<NVT, false>(ne, npts_total, p0, cnt, xb, trans, transm, xa, stream)
  // A warp per batch of rows re-reads x for every member it holds, a CTA per
  // point fills the lanes over all variables.  The lines where they cross are
  // drawn from every n and 1 to 20 variables, 320 MB of weights or 20,000 points;
  // rows / point (before either: a thread per output) in us, merged weights: n =
  // 20, 2 variables 82 / 102 (108), 3 106 / 101 (109); n = 24, 3 122 / 143 (146), 4
  // 150 / 143 (151); n = 32, 4 189 / 213 (336); n = 40, 1 144 / 174 (188), 2 228 /
  // 216 (221); n = 64, 3 274 / 285 (616); n = 72, 2 258 / 280 (298), 3 361 / 326
  // (353); n = 82, 5 503 / 508 (602), 6 599 / 553 (615); n = 128, 6 539 / 993 (1251).
  // With mean weights the same up to n = 54 (n = 8, 3 variables 0.98 / 0.84 of the
  // time before, n = 23, 3 0.60 / 0.68, 4 0.73 / 0.69, n = 44, 2 0.65 / 0.64), then
  // n = 62, 3 0.49 / 0.53, 4 0.50 / 0.50; n = 64, 4 0.44 / 0.47; n = 68, 2 0.53 / 0.60, 3 0.56 / 0.51; n =
  // 77, 5 0.52 / 0.59, 6 0.59 / 0.55; n = 83, 6 0.49 / 0.53.
  const int rows = ne <= 21   ? 2
                   : ne <= 24 ? 3
                   : ne <= 32 ? 4
                   : ne <= 54 ? 1
                   : transm   ? (ne <= 64 ? (ne % 16 ? 3 : 6) : ne <= 71 ? 2 : ne <= 79 ? 5 : 6)
                              : (ne <= 79 ? (ne % 16 ? 2 : 4) : ne <= 82 ? 5 : 6);
  // Few points: a warp takes the same time for the rows of one point as of all
  // that fit, a CTA per point divides them, so up to some waves of its resident
  // CTAs the latter is faster.  rows / point, merged weights (before either) in us: n =
  // 80, 3 variables, 600 points 39 / 33 (50), 1,000 58 / 60 (97); n = 100, 1 variable,
  // 300 27 / 17 (19), 450 28 / 31 (33); 6 variables, 1 point 113 / 33 (33), 600 115 /
  // 80 (82); n = 128, 1 variable, 150 33 / 23 (23), 300 33 / 41 (41), 3 variables, 300
  // 76 / 66 (78), 450 76 / 97 (115); rows that are not 16-byte aligned take longer: n =
  // 127, 1 variable, 450 52 / 50 (52), 600 52 / 69 (76).
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int resident = (int)(227 * 1024 / (sizeof(double) * (size_t)ne * (ne + nv) + 1024));
  const int waves = !vec ? 3 : nv > 2 ? 2 : 1;
  if (nv <= rows && cnt > nsm * std::min(4, waves * resident)) {
    if (nv == 1) UPR_LAUNCH(1);
    if (nv == 2) UPR_LAUNCH(2);
    if (nv == 3) UPR_LAUNCH(3);
    if (nv == 4) UPR_LAUNCH(4);
    if (nv == 5) UPR_LAUNCH(5);
    UPR_LAUNCH(6);
  }
#undef UPR_LAUNCH
  // The general kernel's four sums a thread pay where few CTAs share an SM and W
  // is read without bank conflicts or nearly: n = 128, merged, 7 variables 1,071
  // us against 1,107; with mean weights n = 64, 11 variables 0.96 of the point
  // form's time, n = 88 0.94, n = 96 0.90, n = 112 0.88 (n = 62 1.10, n = 98 1.04).
  if (transm ? ne < 64 || ne % 8 != 0 : ne < 128) {
    if (transm) return launch_update_point<true>(ne, npts_total, p0, cnt, nv, xb, trans, transm, xa, stream);
    return launch_update_point<false>(ne, npts_total, p0, cnt, nv, xb, trans, transm, xa, stream);
  }
  return launch_update(ne, npts_total, p0, cnt, nv, xb, trans, transm, nullptr, plain, xa, stream);
}

int launch_update_f64(int ne, int npts, int nv, const double* xb, const double* trans, const double* transm,
                      double* xa, cudaStream_t stream) {
  return launch_update_f64_range(ne, npts, 0, npts, nv, xb, trans, transm, xa, stream);
}

// relax_beta (scale/letkf/letkf_tools.f90:1182-1220): 0 for the q variables
// above Q_UPDATE_TOP, the boundary-buffer ramp, else 1
__global__ void relax_beta_kernel(int npts, int nv, const double* __restrict__ ri, const double* __restrict__ rj,
                                  const double* __restrict__ rlev, int q_lo, int q_hi, double q_update_top,
                                  double bbw, double dx, double dy, int nlong, int nlatg, int ihalo, int jhalo,
                                  double* beta) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)npts * nv) return;
  const int v = (int)(t / npts), p = (int)(t - (int64_t)v * npts);
  double b = 1.0;
  if (rlev[p] < q_update_top && v >= q_lo && v <= q_hi) {
    beta[t] = 0.0;
    return;
  }
  if (bbw > 0.0) {
    const double d = fmin(fmin(ri[p] - ihalo, nlong + ihalo + 1 - ri[p]) * dx,
                          fmin(rj[p] - jhalo, nlatg + jhalo + 1 - rj[p]) * dy) / bbw;
    if (d < 1.0) b = fmax(d, 0.0);
  }
  beta[t] = b;
}

}  // namespace letkf

using namespace letkf;

extern "C" int letkf_update_relax_f64(int ne, int npts, int nv, const double* xb, const double* trans,
                                      const double* transm, const double* pao, const letkf_relax_desc* rd,
                                      double* xa, double* rtps_infl, void* stream) {
  if (ne < 2 || npts < 0 || nv < 1 || !xb || !trans || !xa || !rd) return LETKF_ERR_ARG;
  if (rd->mode < 0 || rd->mode > 2 || (rd->mode == 2 && !pao)) return LETKF_ERR_ARG;
  if (ne > LETKF_MAX_NE) return LETKF_ERR_CAPACITY;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) {
    cudaGetLastError();
    return LETKF_ERR_NOGPU;
  }
  if (npts == 0) return LETKF_OK;
  RelaxArgs r;
  r.mode = rd->mode;
  r.alpha = rd->alpha;
  r.beta = rd->beta;
  r.q_var = rd->q_var;
  r.q_sprd_max = rd->q_sprd_max;
  r.rtps_infl = rtps_infl;
  return launch_update(ne, npts, 0, npts, nv, xb, trans, transm, pao, r, xa, (cudaStream_t)stream);
}

extern "C" int letkf_relax_beta(int npts, int nv, const double* ri, const double* rj, const double* rlev, int q_lo,
                                int q_hi, double q_update_top, double boundary_buffer_width, double dx, double dy,
                                int nlong, int nlatg, int ihalo, int jhalo, double* beta, void* stream) {
  if (npts < 0 || nv < 1 || (npts > 0 && (!ri || !rj || !rlev || !beta))) return LETKF_ERR_ARG;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) {
    cudaGetLastError();
    return LETKF_ERR_NOGPU;
  }
  const int64_t n = (int64_t)npts * nv;
  if (n == 0) return LETKF_OK;
  relax_beta_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      npts, nv, ri, rj, rlev, q_lo, q_hi, q_update_top, boundary_buffer_width, dx, dy, nlong, nlatg, ihalo, jhalo,
      beta);
  note_launch();
  return cuda_status(cudaGetLastError());
}
