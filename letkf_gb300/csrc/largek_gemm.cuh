// largek_gemm.cuh -- batched tcgen05 GEMM for the large-ensemble core.
//
// One CTA computes a 128 x 128 tile of one point's product with the
// accumulator in tensor memory (128 columns).  Operands are FP32 in global
// memory and enter the tensor core as three-term TF32 splits
// (x = hi + lo, hi = x with the low 13 mantissa bits cleared):
//   acc = A_hi B_hi + A_hi B_lo + A_lo B_hi        (about 1e-6 relative)
// The tile is computed transposed, outᵀ = Yᵀ Xᵀ: the tensor core's A is Yᵀ,
// whose rows the lanes read as whole lines of Y, and is staged in tensor memory
// (a thread has one of its rows; 32 columns a K = 16 stage); its B is X, K-major
// in shared memory (SWIZZLE_NONE core matrices of 8 rows x 16 bytes, 20 KB a
// stage).  What bounded the kernel was shared-memory bandwidth: with both
// operands there a stage wrote 32 KB and its six MMAs read 48 KB (data pipe 94 %
// busy, tensor pipe 27 %), now 16 and 24, and a row per lane of X took a tag
// lookup a lane.  Two stages share a barrier, two such pairs are in flight, and
// two CTAs share an SM (256 TMEM columns each), so that one's MMAs overlap the
// other's global loads.  The tile leaves through shared memory, a row per warp
// request (a row per lane took 32 wavefronts a store).  k = 512, 256 points, one
// product: 580 -> 327 us (tensor memory and tile alone 425); the products and
// their order are the same, and so are the bits.  The Gram (lists of 464 rows a
// point, BF16): 900 -> 470 us, its list entries a pair ahead of the rows and
// nothing waiting on a row before its use.
//
// Modes:
//   LK_GRAM   out = Ywᵀ Y over the point's local rows (K = its L, Yw = w_l y_l):
//             rows of the packed FP32 [nrows][ne] array, or with ridx rows
//             ridx[l] of the observation ensemble (FP32 rows, or BF16 rows16),
//             so that no per-point copies are made however long the list
//   LK_T      out = X Y and e2[b] += ||out - I||²_F   (Newton-Schulz residual)
//   LK_AXPBY  out = alpha X Y + beta D   (alpha, beta per point when alpha_b,
//             beta_b are set;
//             D may be NULL: out = alpha X Y)
// X, Y, D, out are [batch][kp][kp] row-major; B(n, k) = Y[k][n], so no operand
// needs to be symmetric.  Points with active[b] == 0 copy D to out (AXPBY) or
// return (other modes).
#pragma once
#include "letkf_common.cuh"
#include "tc_sm100.cuh"

namespace letkf {

constexpr int LK_NT = 256;
constexpr int LK_TILE = 128;
constexpr int LK_KC = 16;                // K per stage
// B's core matrices lie 32 bytes apart, so that a quarter warp's 16-byte stores
// (two rows of four) fall into different banks
constexpr int LK_LBO = 160, LK_SBO = 4 * LK_LBO;
constexpr int LK_OPER = 16 * LK_SBO;     // one 128 x 16 TF32 operand
constexpr int LK_STAGE = 2 * LK_OPER;    // B_hi, B_lo
constexpr int LK_RING = 4;               // stages: two pairs
constexpr int LK_OUT_LD = LK_TILE + 4;   // floats of a row of the output tile (conflict-free 16-byte columns)
constexpr int LK_BUF = LK_RING * LK_STAGE;
constexpr int LK_SMEM = LK_BUF + 64;
static_assert(LK_BUF >= LK_TILE * LK_OUT_LD * 4, "the tile takes the stages' place");
constexpr uint32_t LK_TMEM_COLS = 256;   // accumulator, then A's stages
constexpr uint32_t LK_TMEM_A = 128;
constexpr uint32_t LK_WAIT = 1u << 22;
// The Gram's K is split over LK_SPLITS CTAs where the tiles alone are less than
// two waves and the mean list is LK_SPLIT_L long: four points of k = 512 with
// 24,000 rows are 64 tiles of 1,500 stages, 6.4 ms; split 1.2.  Shorter
// lists keep one accumulator (and their bits).
constexpr int LK_SPLITS = 6;
constexpr int LK_SPLIT_L = 4096;

enum { LK_GRAM = 0, LK_T = 1, LK_AXPBY = 2 };

struct LkGemmArgs {
  int kp;                 // padded matrix size (multiple of 128)
  int64_t mstride;        // kp * kp
  const float* X;
  const float* Y;
  const float* D;
  float alpha, beta;
  const float* alpha_b;   // [batch] or NULL
  const float* beta_b;    // [batch] or NULL
  float* out;
  float* e2;              // [batch] (LK_T)
  const int* active;      // [batch] or NULL
  // LK_GRAM
  const float* rows;      // [nrows][ne], or [nobs][ne] with ridx
  const __nv_bfloat16* rows16;  // [nobs][ne] BF16 rows (with ridx; rows is then NULL)
  const int* ridx;        // [nrows] observation of each list entry, or NULL (packed rows)
  const float* wts;       // [nrows] weight of each row (rloc / rdiag)
  const int64_t* offs;    // [batch + 1] rows of point b: offs[b] .. offs[b+1]-1
  int ne;
  int nsplit;             // pieces of K, each a CTA's with its own output
  float* outs[LK_SPLITS];
  int* err_flag;
};

// split 4 values into TF32 hi (low 13 mantissa bits cleared) and remainder
__device__ __forceinline__ void lk_split4(const float (&v)[4], float4& hi, float4& lo) {
  float h[4];
#pragma unroll
  for (int j = 0; j < 4; j++) h[j] = __uint_as_float(__float_as_uint(v[j]) & 0xFFFFE000u);
  hi = make_float4(h[0], h[1], h[2], h[3]);
  lo = make_float4(v[0] - h[0], v[1] - h[1], v[2] - h[2], v[3] - h[3]);
}

__device__ __forceinline__ void lk_store(unsigned char* hi_base, unsigned char* lo_base, int r, int kk,
                                         const float (&v)[4]) {
  float4 h, l;
  lk_split4(v, h, l);
  const uint32_t off = (uint32_t)((r >> 3) * LK_SBO + (kk >> 2) * LK_LBO + (r & 7) * 16);
  *reinterpret_cast<float4*>(hi_base + off) = h;
  *reinterpret_cast<float4*>(lo_base + off) = l;
}

template <int MODE>
__global__ void __launch_bounds__(LK_NT, 2) largek_gemm_kernel(LkGemmArgs a) {
  extern __shared__ __align__(1024) unsigned char sm[];
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + LK_BUF);
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(sm + LK_BUF + 16);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nsp = MODE == LK_GRAM ? a.nsplit : 1;
  const int b = blockIdx.z / nsp, sp = blockIdx.z - b * nsp;
  const int m0 = blockIdx.y * LK_TILE, n0 = blockIdx.x * LK_TILE;
  const int kp = a.kp;
  const size_t mo = (size_t)b * a.mstride;
  const bool act = a.active == nullptr || a.active[b] != 0;
  if (!act) {
    if (MODE == LK_AXPBY && a.D) {  // keep the converged state in the output buffer
      for (int t = tid; t < LK_TILE * LK_TILE / 4; t += LK_NT) {
        const int r = t / (LK_TILE / 4), c4 = t % (LK_TILE / 4);
        const size_t idx = mo + (size_t)(m0 + r) * kp + n0 + 4 * c4;
        *reinterpret_cast<float4*>(a.out + idx) = *reinterpret_cast<const float4*>(a.D + idx);
      }
    }
    return;
  }
  int nk;
  int kfirst = 0;  // first stage of this CTA's piece of K
  int64_t r0 = 0;
  int L = 0;
  if (MODE == LK_GRAM) {
    r0 = a.offs[b];
    L = (int)(a.offs[b + 1] - r0);
    nk = (L + LK_KC - 1) / LK_KC;
    if (nsp > 1) {
      const int per = (nk + nsp - 1) / nsp;
      kfirst = min(nk, sp * per);
      nk = min(nk, kfirst + per) - kfirst;
    }
  } else {
    nk = kp / LK_KC;
  }
  if (tid == 0) {
    tc::mbar_init(&mbar[0], 1);
    tc::mbar_init(&mbar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (wid == 0) tc::tmem_alloc(tmem_holder, LK_TMEM_COLS);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tacc = *tmem_holder;
  const uint32_t sbase = tc::smem_u32(sm);
  const uint32_t idesc = tc::idesc_tf32(128, 128);
  // phase parities and stages with MMAs in flight as bit masks (bit = stage
  // buffer): the buffer index is known only at run time, and arrays indexed by
  // it would live in local memory
  uint32_t par = 0u, outst = 0u;
  int tmo = 0;
  const int r = tid & 127, h = tid >> 7;  // staging: row r, K half h (8 values)

  // stage values of this thread, both stages of a pair; the next pair's loads
  // are issued before this pair is split and stored.  A: row r, K half h.  B:
  // in the Gram the same of the weighted rows; else four columns of rows tid / 4
  // and 64 + tid / 4 (a quarter of the sectors' lines that a row per lane
  // touches)
  float va[2][8], vb[2][8];
  // Gram: a lane has an entry of a pair's list rows, loaded a pair ahead of
  // the rows themselves; the weight is applied, and what lies beyond L or ne cleared, where
  // a value is used, so that nothing waits on its load before (those load a
  // valid address: any row serves)
  size_t er = 0;
  float ew = 0.f, nw = 0.f;
  const bool in_a = n0 + r < a.ne, in_b = m0 + r < a.ne;
  const int ca_ = in_a ? n0 + r : 0, cb_ = in_b ? m0 + r : 0;
  auto load_list = [&](int c) {
    const int l = min((kfirst + c) * LK_KC + lane, L - 1);
    er = a.ridx ? (size_t)a.ridx[r0 + l] : (size_t)(r0 + l);
    ew = a.wts[r0 + l];
  };
  auto load_stage = [&](int c, int q, float (&xa)[8], float (&xb)[8]) {
    if (MODE == LK_GRAM) {
      // A(n, l) = y_l[n], B(m, l) = w_l y_l[m]
      size_t at[8];
#pragma unroll
      for (int j = 0; j < 8; j++) at[j] = (size_t)__shfl_sync(0xffffffffu, er, 16 * q + 8 * h + j) * a.ne;
      if (a.rows16) {
        const unsigned short* y16 = reinterpret_cast<const unsigned short*>(a.rows16);
#pragma unroll
        for (int j = 0; j < 8; j++) xa[j] = __uint_as_float((uint32_t)y16[at[j] + ca_]);
#pragma unroll
        for (int j = 0; j < 8; j++) xb[j] = __uint_as_float((uint32_t)y16[at[j] + cb_]);
      } else {
#pragma unroll
        for (int j = 0; j < 8; j++) xa[j] = a.rows[at[j] + ca_];
#pragma unroll
        for (int j = 0; j < 8; j++) xb[j] = a.rows[at[j] + cb_];
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) xa[j] = a.Y[mo + (size_t)(c * LK_KC + h * 8 + j) * kp + n0 + r];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const float4 x = *reinterpret_cast<const float4*>(a.X + mo + (size_t)(m0 + 64 * i + (tid >> 2)) * kp +
                                                          c * LK_KC + 4 * (tid & 3));
        xb[4 * i] = x.x;
        xb[4 * i + 1] = x.y;
        xb[4 * i + 2] = x.z;
        xb[4 * i + 3] = x.w;
      }
    }
  };
  if (MODE == LK_GRAM && nk > 0) load_list(0);
#pragma unroll
  for (int q = 0; q < 2; q++)
    if (q < nk) load_stage(q, q, va[q], vb[q]);
  if (MODE == LK_GRAM && nk > 0) {
    nw = ew;
    load_list(2);
  }

  const uint32_t alane = (uint32_t)(32 * (wid & 3)) << 16;  // a warp's TMEM lanes
  for (int c = 0; c < nk; c += 2) {
    const int buf = (c >> 1) & 1, ns = min(2, nk - c);
    float ca[2][8], cb[2][8];
#pragma unroll
    for (int q = 0; q < 2; q++)
#pragma unroll
      for (int j = 0; j < 8; j++) {
        ca[q][j] = va[q][j];
        cb[q][j] = vb[q][j];
      }
    const float cw = nw;
#pragma unroll
    for (int q = 0; q < 2; q++)
      if (c + 2 + q < nk) load_stage(c + 2 + q, q, va[q], vb[q]);
    if (MODE == LK_GRAM) {
      nw = ew;
      load_list(c + 4);
    }
    if ((outst >> buf) & 1u) {
      if (!tc::mbar_wait(&mbar[buf], (par >> buf) & 1u, LK_WAIT)) tmo = 1;
      par ^= 1u << buf;
      outst &= ~(1u << buf);
    }
    tc::fence_after_sync();
#pragma unroll
    for (int q = 0; q < 2; q++) {
      if (q >= ns) break;
      const int slot = 2 * buf + q;
      unsigned char* st = sm + slot * LK_STAGE;
      if (MODE == LK_GRAM) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const float w = __shfl_sync(0xffffffffu, cw, 16 * q + 8 * h + j);
          const bool in_l = (kfirst + c + q) * LK_KC + 8 * h + j < L;
          if (a.rows16) {
            ca[q][j] = __uint_as_float(__float_as_uint(ca[q][j]) << 16);
            cb[q][j] = __uint_as_float(__float_as_uint(cb[q][j]) << 16);
          }
          ca[q][j] = in_l && in_a ? ca[q][j] : 0.f;
          cb[q][j] = in_l && in_b ? __fmul_rn(w, cb[q][j]) : 0.f;
        }
      }
      float hi[8], lo[8];
#pragma unroll
      for (int j = 0; j < 8; j++) tc::split_tf32(ca[q][j], hi[j], lo[j]);
      const uint32_t at = tacc + alane + LK_TMEM_A + 32 * slot + 8 * h;
      tc::tmem_st8(at, hi);
      tc::tmem_st8(at + 16, lo);
#pragma unroll
      for (int g = 0; g < 2; g++) {
        const float qb[4] = {cb[q][4 * g], cb[q][4 * g + 1], cb[q][4 * g + 2], cb[q][4 * g + 3]};
        if (MODE == LK_GRAM)
          lk_store(st, st + LK_OPER, r, h * 8 + g * 4, qb);
        else
          lk_store(st, st + LK_OPER, 64 * g + (tid >> 2), 4 * (tid & 3), qb);
      }
    }
    tc::tmem_wait_st();
    tc::fence_smem_async();
    tc::fence_before_sync();
    if (__syncthreads_or(tmo)) {  // a bounded wait gave up: issue nothing more
      tmo = 1;
      break;
    }
    if (tid == 0) {
      tc::fence_after_sync();
#pragma unroll
      for (int q = 0; q < 2; q++) {
        if (q >= ns) break;
        const int slot = 2 * buf + q;
        const uint32_t s0 = sbase + slot * LK_STAGE, a0 = tacc + LK_TMEM_A + 32 * slot;
#pragma unroll
        for (int pass = 0; pass < 3; pass++) {
          const uint32_t sa = a0 + (pass == 1 ? 16 : 0);
          const uint32_t sb = s0 + (pass == 2 ? LK_OPER : 0);
#pragma unroll
          for (int s = 0; s < LK_KC / 8; s++)
            tc::mma_tf32_ts(tacc, sa + 8 * s, tc::smem_desc(sb + s * 2 * LK_LBO, LK_LBO, LK_SBO), idesc,
                            (c == 0 && q == 0 && pass == 0 && s == 0) ? 0u : 1u);
        }
      }
      tc::mma_commit(&mbar[buf]);
    }
    outst |= 1u << buf;
  }
  for (int q = 0; q < 2; q++)
    if ((outst >> q) & 1u) {
      if (!tc::mbar_wait(&mbar[q], (par >> q) & 1u, LK_WAIT)) tmo = 1;
      par ^= 1u << q;
      outst &= ~(1u << q);
    }
  tc::fence_after_sync();
  const bool bad = __syncthreads_or(tmo) != 0;
  if (bad) {
    if (tid == 0 && a.err_flag) atomicExch(a.err_flag, 1);
  } else {
    // epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31 (the tile's columns),
    // TMEM columns 64 (w / 4) .. +63 (its rows); then a row per warp request
    float* tile = reinterpret_cast<float*>(sm);
    {
      const int tcol = 32 * (wid & 3) + lane, rb = 64 * (wid >> 2);
      const uint32_t taddr = tacc + alane + (uint32_t)rb;
#pragma unroll 1
      for (int c0 = 0; c0 < 64; c0 += 16) {
        float v[16];
        if (nk > 0) {
          tc::tmem_ld16(taddr + c0, v);
        } else {
#pragma unroll
          for (int j = 0; j < 16; j++) v[j] = 0.f;
        }
#pragma unroll
        for (int j = 0; j < 16; j++) tile[(rb + c0 + j) * LK_OUT_LD + tcol] = v[j];
      }
    }
    __syncthreads();
    const float al = MODE == LK_AXPBY ? (a.alpha_b ? a.alpha_b[b] : a.alpha) : 1.f;
    const float be = MODE == LK_AXPBY ? (a.beta_b ? a.beta_b[b] : a.beta) : 0.f;
    float* out = MODE == LK_GRAM && nsp > 1 ? a.outs[sp] : a.out;
    float e2 = 0.f;
#pragma unroll 4
    for (int row = wid; row < LK_TILE; row += LK_NT / 32) {
      const int col = 4 * lane;
      const size_t at = mo + (size_t)(m0 + row) * kp + n0 + col;
      float4 v = *reinterpret_cast<const float4*>(tile + row * LK_OUT_LD + col);
      if (MODE == LK_AXPBY) {
        if (a.D) {
          const float4 d = *reinterpret_cast<const float4*>(a.D + at);
          // one rounding for the product by alpha, as the compiler had it: bits matter to the iteration's fixed point
          v = make_float4(fmaf(be, d.x, __fmul_rn(al, v.x)), fmaf(be, d.y, __fmul_rn(al, v.y)),
                          fmaf(be, d.z, __fmul_rn(al, v.z)), fmaf(be, d.w, __fmul_rn(al, v.w)));
        } else {
          v = make_float4(al * v.x, al * v.y, al * v.z, al * v.w);
        }
      }
      if (MODE == LK_T) {
        const int dg = m0 + row - n0 - col;  // the diagonal's place in v
        const float d0 = v.x - (dg == 0 ? 1.f : 0.f), d1 = v.y - (dg == 1 ? 1.f : 0.f);
        const float d2 = v.z - (dg == 2 ? 1.f : 0.f), d3 = v.w - (dg == 3 ? 1.f : 0.f);
        e2 = fmaf(d0, d0, fmaf(d1, d1, fmaf(d2, d2, fmaf(d3, d3, e2))));
      }
      *reinterpret_cast<float4*>(out + at) = v;
    }
    if (MODE == LK_T) {
      e2 = warp_sum(e2);
      if (lane == 0) atomicAdd(&a.e2[b], e2);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (wid == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tacc, LK_TMEM_COLS);
  }
}

}  // namespace letkf
