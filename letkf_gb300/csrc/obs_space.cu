// obs_space.cu -- the obs-space clients of the batched core (GFS driver).
//
//  * letkf_obs_analysis: analysis ensemble at observation locations
//    (gfs/letkf/letkf_tools.f90:466-497): with trans the point's merged
//    transform (T + wbar 1^T, RTPP applied as weight_RTPP does, :959-970),
//    obsanal(n, m) = ybar(n) + sum_k obshdxf(n, k) trans(k, m), ybar =
//    obsdat - obsdep, the mean over the members, the q "no update" branch and
//    the relative-spread clip.
//  * letkf_efso: observation sensitivity (gfs/letkf/letkf_tools.f90:547-679)
//    over grid points with their local observation lists.
#include <algorithm>

#include "letkf_common.cuh"

namespace letkf {

constexpr int OSA_NT = 128;
constexpr int OSA_T = 64;       // members and weights of a staged tile
constexpr int OSA_LD = OSA_T + 1;
constexpr int OSA_WARP = 128;   // members of the largest ensemble that a warp takes
constexpr int EFSO_MAX_TERM = 8;
constexpr int EFSO_MAX_NV = 16;
constexpr int EFSO_MC = 16;     // members of a staged tile of 32 observations, or half of them
constexpr int EFSO_FEW = 8;     // members whose rows the lanes read by themselves
constexpr int EFSO_GROUP = 8;   // grid points of a CTA at most

// One CTA per observation location.  Bound: HBM for trans (k^2 doubles, read
// once), as long as the reads are whole lines: tiles of 64 weights x 64
// members go through shared memory (rows of trans are read along the weights,
// the odd row length spreads the transposing stores over the banks), then a
// thread sums half a tile of one member's weights.  A thread walking its own
// member's row in global memory read 32 lines per warp instruction: 20,000
// locations of k = 64 took 0.91 ms, now 0.23.
__global__ void __launch_bounds__(OSA_NT) obs_analysis_kernel(int ne, int n, const double* __restrict__ trans,
                                                               const double* __restrict__ ybar,
                                                               const double* __restrict__ hdxf, double alpha,
                                                               const int* __restrict__ mode, double q_sprd_max,
                                                               double* anal, double* amean) {
  extern __shared__ double so[];
  double* h = so;               // [ne] obshdxf(n, :)
  double* a = h + ne;           // [ne] analysis members
  double* tile = a + ne;        // [OSA_T][OSA_LD] weight k0 + kk of member m0 + m
  double* part = tile + OSA_T * OSA_LD;  // [OSA_T] second half's sums
  const int tid = threadIdx.x, lane = tid & 31;
  const int m = tid % OSA_T, half = tid / OSA_T;
  for (int p = blockIdx.x; p < n; p += gridDim.x) {
    const int md = mode ? mode[p] : 0;
    const double yb = ybar[p];
    const double* tp = trans + (size_t)p * ne * ne;
    __syncthreads();
    for (int i = tid; i < ne; i += OSA_NT) h[i] = hdxf[(size_t)p * ne + i];
    if (md == 1) {
      __syncthreads();
      for (int i = tid; i < ne; i += OSA_NT) a[i] = yb + h[i];
    } else {
      for (int m0 = 0; m0 < ne; m0 += OSA_T) {
        const int nm = min(OSA_T, ne - m0);
        double v = 0.0;
        for (int k0 = 0; k0 < ne; k0 += OSA_T) {
          const int nk = min(OSA_T, ne - k0);
          // all of a thread's part in flight before the tile's last readers are waited for
          double r[OSA_T * OSA_T / OSA_NT];
          const int kk = tid % OSA_T, mm = tid / OSA_T;
          const double* src = tp + (size_t)(m0 + mm) * ne + k0 + kk;
#pragma unroll
          for (int i = 0; i < OSA_T * OSA_T / OSA_NT; i++) {
            const int mi = mm + i * (OSA_NT / OSA_T);
            r[i] = (kk < nk && mi < nm) ? src[(size_t)i * (OSA_NT / OSA_T) * ne] : 0.0;
          }
          __syncthreads();
#pragma unroll
          for (int i = 0; i < OSA_T * OSA_T / OSA_NT; i++) tile[kk * OSA_LD + mm + i * (OSA_NT / OSA_T)] = r[i];
          __syncthreads();
          const int kb = half * (OSA_T / 2), ke = min(nk, kb + OSA_T / 2);
          if (m < nm)
#pragma unroll 4
            for (int kk = kb; kk < ke; kk++) v = fma(h[k0 + kk], tile[kk * OSA_LD + m], v);
        }
        if (half == 1) part[m] = v;
        __syncthreads();
        // RTPP (:959-970) outside the sum: (1 - a) sum_k h(k) w(k, m) + a h(m)
        if (half == 0 && m < nm) {
          v = v + part[m];
          if (alpha != 0.0) v = (1.0 - alpha) * v + alpha * h[m0 + m];
          a[m0 + m] = yb + v;
        }
      }
    }
    __syncthreads();
    if (tid < 32) {
      double s = yb;
      if (md != 1) {
        double t = 0.0;
        for (int i = lane; i < ne; i += 32) t = t + a[i];
        s = warp_sum(t) / (double)ne;
        if (md == 2) {
          double sp = 0.0;
          for (int i = lane; i < ne; i += 32) sp = fma(a[i] - s, a[i] - s, sp);
          sp = sqrt(warp_sum(sp) / (double)(ne - 1)) / s;
          if (sp > q_sprd_max)
            for (int i = lane; i < ne; i += 32) a[i] = s + (a[i] - s) * q_sprd_max / sp;
        }
      }
      if (amean && lane == 0) amean[p] = s;
    }
    __syncthreads();
    for (int i = tid; i < ne; i += OSA_NT) anal[(size_t)p * ne + i] = a[i];
  }
}

// A warp per location, a lane per member (R of them) on its own rows of trans,
// no barrier.  The sums are those of the kernel above in the same order.
// A lane takes 64 consecutive bytes of its row at a time (VEC: by 16 bytes, rows
// aligned), so that the line it is in the middle of stays in L1.  HBM for trans
// bounds it, and the lines' way through L1 up to k = 32.  In us, a CTA per
// location with a thread per member (before the tile) / the tile / here: 20,000
// locations of k = 16 61 / 103 / 48, k = 32 132 / 156 / 68, k = 40 166 / 198 / 134, k =
// 64 324 / 252 / 183, 8,000 of k = 100 242 / 269 / 234, 4,900 of k = 127 196 / 207 / 182.
// From k = 65 a warp alone with its location takes longer than the tile's four
// until the SMs are full of them: 600 locations of k = 100 21 / 21 / 27, 1,000 of k =
// 96 44 / 32 / 27, of k = 101 37 / 39 / 35, of k = 127 47 / 54 / 56.
template <int R, bool VEC>
__global__ void __launch_bounds__(OSA_NT, 8) obs_analysis_warp_kernel(int ne, int n, const double* __restrict__ trans,
                                                                      const double* __restrict__ ybar,
                                                                      const double* __restrict__ hdxf, double alpha,
                                                                      const int* __restrict__ mode, double q_sprd_max,
                                                                      double* anal, double* amean) {
  __shared__ __align__(16) double hs[OSA_NT / 32][32 * R];
  const int lane = threadIdx.x & 31, stride = gridDim.x * (OSA_NT / 32);
  double* h = hs[threadIdx.x >> 5];
  for (int p = blockIdx.x * (OSA_NT / 32) + (threadIdx.x >> 5); p < n; p += stride) {
    const int md = mode ? mode[p] : 0;
    const double yb = ybar[p];
    __syncwarp();
    for (int m = lane; m < ne; m += 32) h[m] = hdxf[(size_t)p * ne + m];
    __syncwarp();
    double a[R], s = yb;
#pragma unroll
    for (int r = 0; r < R; r++) a[r] = yb + (lane + 32 * r < ne ? h[lane + 32 * r] : 0.0);
    if (md != 1) {
      double t = 0.0;
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int m = lane + 32 * r;
        if (m >= ne) continue;
        const double* w = trans + ((size_t)p * ne + m) * ne;
        double v[2] = {0.0, 0.0};  // the even and odd 32s of the weights
#pragma unroll
        for (int q = 0; q < R; q++) {
          const int ke = min(ne, 32 * q + 32);
          int k = 32 * q;
          for (; k + 8 <= ke; k += 8) {  // 64 bytes in flight
            double x[8];
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
              if (VEC) {
                const double2 u = *reinterpret_cast<const double2*>(w + k + i);
                x[i] = u.x;
                x[i + 1] = u.y;
              } else {
                x[i] = w[k + i];
                x[i + 1] = w[k + i + 1];
              }
            }
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
              const double2 hk = *reinterpret_cast<const double2*>(h + k + i);
              v[q & 1] = fma(hk.x, x[i], v[q & 1]);
              v[q & 1] = fma(hk.y, x[i + 1], v[q & 1]);
            }
          }
#pragma unroll 4
          for (; k < ke; k++) v[q & 1] = fma(h[k], w[k], v[q & 1]);
        }
        double b = v[0] + v[1];
        if (alpha != 0.0) b = (1.0 - alpha) * b + alpha * h[m];
        a[r] = yb + b;
        t = t + a[r];
      }
      s = warp_sum(t) / (double)ne;
      if (md == 2) {
        double sp = 0.0;
#pragma unroll
        for (int r = 0; r < R; r++)
          if (lane + 32 * r < ne) sp = fma(a[r] - s, a[r] - s, sp);
        sp = sqrt(warp_sum(sp) / (double)(ne - 1)) / s;
        if (sp > q_sprd_max)
#pragma unroll
          for (int r = 0; r < R; r++) a[r] = s + (a[r] - s) * q_sprd_max / sp;
      }
    }
    if (amean && lane == 0) amean[p] = s;
#pragma unroll
    for (int r = 0; r < R; r++)
      if (lane + 32 * r < ne) anal[(size_t)p * ne + lane + 32 * r] = a[r];
  }
}

struct EfsoTerms {
  int term[EFSO_MAX_NV];
};

// One CTA per group of neighbouring grid points: their work1 in shared memory
// and the entries of all their lists flattened over the lanes, so short lists
// fill the warps.  A lane sums one entry's products over the members (FP64
// pipe: one multiply-add per member and term; the entry's rloc / rdiag, rounded
// once, is applied to the sums), and the rows of the 32 observations of a warp go
// through a tile of 16 members in shared memory, read as whole lines with the
// next tile's loads in flight.  Bound: the FP64 pipe (1.2 TFLOP/s).  A thread
// walking its own observation's row, one point per CTA, two more products per
// member: 30,000 points with 50 local observations of k = 64 and 3 terms took
// 2.55 ms, now 0.78 (FP64 pipe 69 % busy).  (rloc and rdiag loaded ahead of the
// sums hold registers: three terms take 90 instead of 80, one CTA an SM fewer, up
// to 20 % more time where lists are even.)
template <int NTERM, int MC>
__global__ void __launch_bounds__(OSA_NT) efso_djdy_kernel(int ne, int npts, int nv, int group,
                                                            const __grid_constant__ EfsoTerms tv,
                                                            const int64_t* __restrict__ offs,
                                                            const int* __restrict__ idx,
                                                            const double* __restrict__ rdiag,
                                                            const double* __restrict__ rloc,
                                                            const double* __restrict__ hdxa,
                                                            const double* __restrict__ fcst,
                                                            const double* __restrict__ fcer, double* djdy) {
  extern __shared__ double w1[];  // [group][NTERM][ne], then the warps' tiles [MC][33]
  __shared__ int64_t lo[EFSO_GROUP + 1];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  double* tile = w1 + (size_t)group * NTERM * ne + wid * MC * 33;
  const int ngroup = (npts + group - 1) / group;
  for (int g = blockIdx.x; g < ngroup; g += gridDim.x) {
    const int p0 = g * group, np = min(group, npts - p0);
    __syncthreads();
    if (tid <= np) lo[tid] = offs[p0 + tid];
    for (int t = tid; t < np * ne; t += OSA_NT) {
      const int q = t / ne, m = t - q * ne;
      double s[NTERM];
#pragma unroll
      for (int i = 0; i < NTERM; i++) s[i] = 0.0;
      for (int v = 0; v < nv; v++) {
        const double f = fcst[((size_t)v * npts + p0 + q) * ne + m] * fcer[(size_t)v * npts + p0 + q];
#pragma unroll
        for (int i = 0; i < NTERM; i++)
          if (tv.term[v] == i) s[i] = s[i] + f;
      }
#pragma unroll
      for (int i = 0; i < NTERM; i++) w1[((size_t)q * NTERM + i) * ne + m] = s[i];
    }
    __syncthreads();
    const int64_t l0 = lo[0], l1 = lo[np];
    for (int64_t lb = l0 + 32 * wid; lb < l1; lb += OSA_NT) {
      const int64_t l = lb + lane;
      const bool on = l < l1;
      const int ob = on ? idx[l] : -1;
      int q = 0;
      while (q + 1 < np && l >= lo[q + 1]) q++;
      const double* w = w1 + (size_t)q * NTERM * ne;
      double acc[NTERM];
#pragma unroll
      for (int i = 0; i < NTERM; i++) acc[i] = 0.0;
      double wt = 0.0;
      if constexpr (MC == 1) {
        wt = on ? rloc[l] / rdiag[l] : 0.0;
        const double* row = hdxa + (size_t)(on ? ob : 0) * ne;
#pragma unroll 2
        for (int m = 0; m < ne; m++) {
          const double h = on ? row[m] : 0.0;
#pragma unroll
          for (int i = 0; i < NTERM; i++) acc[i] = fma(w[i * ne + m], h, acc[i]);
        }
      } else {
        // RP rows of the tile at a time by MC lanes each, a lane a member
        constexpr int RP = 32 / MC;
        double nx[MC];
        auto load = [&](int m0) {
#pragma unroll
          for (int r = 0; r < MC; r++) {
            const int o = __shfl_sync(0xffffffffu, ob, RP * r + lane / MC);
            const int m = m0 + lane % MC;
            nx[r] = (o >= 0 && m < ne) ? hdxa[(size_t)o * ne + m] : 0.0;
          }
        };
        load(0);
        for (int m0 = 0; m0 < ne; m0 += MC) {
          __syncwarp();
#pragma unroll
          for (int r = 0; r < MC; r++) tile[(lane % MC) * 33 + RP * r + lane / MC] = nx[r];
          __syncwarp();
          if (m0 + MC < ne) load(m0 + MC);
          const int nm = min(MC, ne - m0);
#pragma unroll 4
          for (int m = 0; m < nm; m++) {
            const double h = tile[m * 33 + lane];
#pragma unroll
            for (int i = 0; i < NTERM; i++) acc[i] = fma(w[i * ne + m0 + m], h, acc[i]);
          }
        }
      }
      if (on) {
        if (MC != 1) wt = rloc[l] / rdiag[l];
#pragma unroll
        for (int i = 0; i < NTERM; i++) atomicAdd(&djdy[(size_t)ob * NTERM + i], acc[i] * wt);
      }
    }
  }
}

static int sm_count() {
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nsm;
}

template <int NTERM>
static size_t efso_smem(int ne, int group, int mc) {
  return sizeof(double) * ((size_t)group * NTERM * ne + (mc > 1 ? (OSA_NT / 32) * mc * 33 : 0));
}

template <int NTERM, int MC>
static int launch_efso_as(int ne, int npts, int nv, int group, const EfsoTerms& tv, const int64_t* offs, const int* idx,
                       const double* rdiag, const double* rloc, const double* hdxa, const double* fcst,
                       const double* fcer, double* djdy, cudaStream_t s) {
  const size_t smem = efso_smem<NTERM>(ne, group, MC);
  if (smem > 48 * 1024) {
    const cudaError_t e =
        cudaFuncSetAttribute(efso_djdy_kernel<NTERM, MC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_status(e);
  }
  const int nsm = sm_count();
  const int ngroup = (npts + group - 1) / group;
  const int grid = ngroup < nsm * 8 ? ngroup : nsm * 8;
  efso_djdy_kernel<NTERM, MC><<<grid, OSA_NT, smem, s>>>(ne, npts, nv, group, tv, offs, idx, rdiag, rloc, hdxa, fcst,
                                                     fcer, djdy);
  note_launch();
  return cuda_status(cudaGetLastError());
}

template <int NTERM>
static int launch_efso(int ne, int npts, int nv, const EfsoTerms& tv, const int64_t* offs, const int* idx,
                       const double* rdiag, const double* rloc, const double* hdxa, const double* fcst,
                       const double* fcer, double* djdy, cudaStream_t s) {
  const size_t one = sizeof(double) * (size_t)NTERM * ne;
  // as many points as 24 KB of work1 hold, fewer where that would leave SMs without a group
  const int nsm = sm_count();
  int group = (int)(24 * 1024 / one);
  group = group < 1 ? 1 : group > EFSO_GROUP ? EFSO_GROUP : group;
  const int fill = npts / (nsm * 8);
  if (group > fill) group = fill < 1 ? 1 : fill;
  // no tile where a row is half a line or less (30,000 points with 50 entries, k = 2 / 8,
  // 8 terms: before tiles 156 / 339 us, with one 171 / 283, here 118 / 241)
  if (ne <= EFSO_FEW)
    return launch_efso_as<NTERM, 1>(ne, npts, nv, group, tv, offs, idx, rdiag, rloc, hdxa, fcst, fcer, djdy, s);
  // half a tile where a third CTA shares the SM then: k = 1024, 8 terms, 3,000 points with 50 entries 5.63 -> 3.70
  // ms (4.18 without tiles, three CTAs an SM)
  auto per_sm = [&](int mc) { return 227 * 1024 / (efso_smem<NTERM>(ne, group, mc) + 1024); };
  if (per_sm(EFSO_MC) < 3 && per_sm(EFSO_MC / 2) > per_sm(EFSO_MC))
    return launch_efso_as<NTERM, EFSO_MC / 2>(ne, npts, nv, group, tv, offs, idx, rdiag, rloc, hdxa, fcst, fcer, djdy, s);
  return launch_efso_as<NTERM, EFSO_MC>(ne, npts, nv, group, tv, offs, idx, rdiag, rloc, hdxa, fcst, fcer, djdy, s);
}

__global__ void efso_sense_kernel(int64_t n, int nterm, const double* __restrict__ djdy,
                                  const double* __restrict__ obsdep, double* obsense) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) obsense[i] = djdy[i] * obsdep[i / nterm];
}

static int grid_for(int n) { return std::min(n, 8 * sm_count()); }

static int have_device() {
  int nd = 0;
  if (cudaGetDeviceCount(&nd) != cudaSuccess || nd < 1) {
    cudaGetLastError();
    return 0;
  }
  return 1;
}

}  // namespace letkf

using namespace letkf;

extern "C" int letkf_obs_analysis(int ne, int n, const double* trans, const double* ybar, const double* hdxf,
                                  double relax_alpha, const int* mode, double q_sprd_max, double* anal,
                                  double* anal_mean, void* stream) {
  if (ne < 2 || ne > 4096 || n < 0 || (n > 0 && (!trans || !ybar || !hdxf || !anal))) return LETKF_ERR_ARG;
  if (!have_device()) return LETKF_ERR_NOGPU;
  if (n == 0) return LETKF_OK;
  if (ne <= OSA_T || (ne <= OSA_WARP && n > 6 * sm_count())) {
    const bool vec = ne % 2 == 0 && reinterpret_cast<uintptr_t>(trans) % 16 == 0;
    auto kern = ne <= 32   ? (vec ? obs_analysis_warp_kernel<1, true> : obs_analysis_warp_kernel<1, false>)
                : ne <= 64 ? (vec ? obs_analysis_warp_kernel<2, true> : obs_analysis_warp_kernel<2, false>)
                           : (vec ? obs_analysis_warp_kernel<4, true> : obs_analysis_warp_kernel<4, false>);
    const int need = (int)(((int64_t)n + OSA_NT / 32 - 1) / (OSA_NT / 32));
    kern<<<grid_for(need), OSA_NT, 0, (cudaStream_t)stream>>>(ne, n, trans, ybar, hdxf, relax_alpha, mode, q_sprd_max,
                                                              anal, anal_mean);
    note_launch();
    return cuda_status(cudaGetLastError());
  }
  const size_t smem = sizeof(double) * (2 * (size_t)ne + OSA_T * OSA_LD + OSA_T);
  if (smem > 48 * 1024) {
    const cudaError_t e =
        cudaFuncSetAttribute(obs_analysis_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_status(e);
  }
  obs_analysis_kernel<<<grid_for(n), OSA_NT, smem, (cudaStream_t)stream>>>(ne, n, trans, ybar, hdxf, relax_alpha,
                                                                            mode, q_sprd_max, anal, anal_mean);
  note_launch();
  return cuda_status(cudaGetLastError());
}

extern "C" int letkf_efso(int ne, int npts, int nv, int nterm, const int* term, const int64_t* offs, const int* idx,
                          const double* rdiag, const double* rloc, int nobs, const double* hdxa, const double* fcst,
                          const double* fcer, const double* obsdep, double* djdy, double* obsense, void* stream) {
  if (ne < 2 || npts < 0 || nv < 1 || nv > EFSO_MAX_NV || nterm < 1 || nterm > EFSO_MAX_TERM || nobs < 0 || !term)
    return LETKF_ERR_ARG;
  if (npts > 0 && (!offs || !fcst || !fcer)) return LETKF_ERR_ARG;
  if (nobs > 0 && (!hdxa || !obsdep || !djdy || !obsense)) return LETKF_ERR_ARG;
  EfsoTerms tv;
  for (int v = 0; v < EFSO_MAX_NV; v++) tv.term[v] = v < nv ? term[v] : -1;
  for (int v = 0; v < nv; v++)
    if (tv.term[v] >= nterm) return LETKF_ERR_ARG;
  if ((size_t)nterm * ne * sizeof(double) > 96 * 1024) return LETKF_ERR_CAPACITY;
  if (!have_device()) return LETKF_ERR_NOGPU;
  cudaStream_t s = (cudaStream_t)stream;
  if (nobs == 0) return LETKF_OK;
  int st = cuda_status(cudaMemsetAsync(djdy, 0, sizeof(double) * (size_t)nobs * nterm, s));
  if (st == LETKF_OK && npts > 0) {
#define EFSO_CASE(T) \
  case T: st = launch_efso<T>(ne, npts, nv, tv, offs, idx, rdiag, rloc, hdxa, fcst, fcer, djdy, s); break
    switch (nterm) {
      EFSO_CASE(1);
      EFSO_CASE(2);
      EFSO_CASE(3);
      EFSO_CASE(4);
      EFSO_CASE(5);
      EFSO_CASE(6);
      EFSO_CASE(7);
      EFSO_CASE(8);
    }
#undef EFSO_CASE
  }
  if (st == LETKF_OK) {
    const int64_t tot = (int64_t)nobs * nterm;
    efso_sense_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(tot, nterm, djdy, obsdep, obsense);
    note_launch();
    st = cuda_status(cudaGetLastError());
  }
  return st;
}
