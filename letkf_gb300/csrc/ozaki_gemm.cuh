// ozaki_gemm.cuh -- FP64 products on the BF16 tensor cores by exact digit splitting.
//
// A row of an operand is scaled by a power of two to |x| < 1, rounded to 55
// fractional bits and written as eight signed 7-bit digits (|d| <= 64, exact in
// BF16): x = 2^e sum_i d_i 2^(7 i - 55), i = 0..7.  A product of two such rows is
// sum_(i,j) 2^(7 (i + j) - 110) <d_i, e_j>; the 36 digit products with i + j >=
// 7 are kept.  Those with the same i + j share a power of two and one FP32
// accumulator: over K <= 512 its value is an integer of at most 8 * 512 * 64^2
// = 2^24, so the tensor core's FP32 sum is exact whatever its order, and the
// eight accumulators are joined in integers and rounded to FP64 once per 512
// products; pieces of 512 are added up in FP64, and the tile is written (and
// mirrored, and transposed) once, when its last piece is in.  Of one product
// x y the rounding of the operands loses at most 2^-56 of each row's scale and
// the pairs with i + j <= 6 at most 2^-53 of the two scales' product (7 pairs of
// 2^12 2^-68 and a hundredth of that), a scale being at most twice the row's
// largest element: as good as FP64 for elements near their row's largest, and
// to the same absolute size for smaller ones (K. Ozaki's error-free splitting,
// Ozaki, Ogita, Oishi, Rump 2012).
//
// Bound: BF16 mma.sync (598 TFLOP/s measured here), 36 of them for one FP64
// multiply-add: 16 TFLOP/s where the FP64 pipe has 1.2 and DGEMM reached 0.92.
// A CTA of eight warps has a 64 x 64 tile, a warp 16 x 32 of it with all eight
// accumulators in registers (128 of them), digits staged by cp.async three
// 32-deep stages ahead of 64 KB each: an A fragment set serves four column
// tiles, a B set one warp row, and the fragment loads take a third of the time
// of the products they feed.
#pragma once
#include "letkf_common.cuh"

namespace letkf {

constexpr int OZ_D = 8;           // digits of an operand
constexpr int OZ_TILE = 64;
constexpr int OZ_KC = 32;         // K of a stage
constexpr int OZ_KEXACT = 512;    // K up to which the FP32 sums are exact
constexpr int OZ_NT = 256;
constexpr int OZ_STAGES = 3;
constexpr int OZ_OPER = OZ_D * OZ_TILE * OZ_KC * 2;  // bytes of one operand's stage
constexpr int OZ_OUT_LD = OZ_TILE + 1;
constexpr int OZ_RING = OZ_STAGES * 2 * OZ_OPER;
constexpr int OZ_OUT = OZ_TILE * OZ_OUT_LD * 8;
static_assert(OZ_RING >= OZ_OUT && OZ_RING + OZ_OUT <= 227 * 1024, "shared memory");

// exponent e with |x| < 2^e for the largest magnitude whose bits are mx, as a
// scale 2^e (NaN where a value is not finite)
__device__ __forceinline__ double oz_scale(unsigned long long mx) {
  const int ex = (int)(mx >> 52);
  if (ex == 0x7ff) return NAN;
  return ldexp(1.0, ex < 122 ? -900 : ex - 1022);
}

// the digits of x, |x| < scale, low to high, as BF16 bit patterns; inv55 = 2^55 / scale
__device__ __forceinline__ void oz_digits(double x, double inv55, uint16_t (&d)[OZ_D]) {
  long long v = __double2ll_rn(x * inv55);
#pragma unroll
  for (int i = 0; i < OZ_D - 1; i++) {
    const int q = (int)((v + 64) & 127) - 64;
    d[i] = (uint16_t)(__float_as_uint((float)q) >> 16);
    v = (v - q) >> 7;
  }
  d[OZ_D - 1] = (uint16_t)(__float_as_uint((float)(int)v) >> 16);
}

struct OzGemm {
  int n;                 // rows of A and of B, a multiple of 64 (the output is n x n)
  int K;                 // a multiple of 32
  const uint16_t* A;     // [batch][OZ_D][n][K] digits
  const uint16_t* B;
  const double* sa;      // [batch][n] row scales
  const double* sb;
  double* out;           // [batch or split][n][n] row-major
  double* outT;          // its transpose, or NULL (nsplit 1)
  int64_t obatch;        // elements between the outputs of two points
  int lower;             // only tiles on and below the diagonal
  int mirror;            // and their transposes (a symmetric product)
  int accumulate;        // add to out
  int nsplit;            // K split over this many CTAs, each with its own output
  int64_t osplit;        // elements between their outputs
  const int* skip;       // [batch] or NULL: 1 leaves the point's output alone
  const int* len;        // [batch] or NULL: K of the point is len - k0, the digits past it up to a multiple of 64 are zero
  int k0;
};

__device__ __forceinline__ void oz_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void oz_ldm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

// byte of 16-byte chunk c (0..3) of row r in a [64][32] BF16 stage: rows of 64
// bytes, chunks XORed so that eight rows of one chunk lie on all banks
__device__ __forceinline__ uint32_t oz_off(int r, int c) { return (uint32_t)(r * 64 + ((c ^ ((r >> 1) & 3)) << 4)); }

// MANY: more than one piece of K; the output tile, the sum of the pieces, then
// lies after the stages and not in their place
template <bool MANY>
__global__ void __launch_bounds__(OZ_NT, 1) oz_gemm_kernel(OzGemm g) {
  extern __shared__ __align__(128) unsigned char osm[];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int b = blockIdx.z / g.nsplit, split = blockIdx.z - b * g.nsplit;
  if (g.skip && g.skip[b]) return;
  int ti, tj;
  if (g.lower) {
    int id = blockIdx.x;
    ti = 0;
    while (id > ti) {
      id -= ti + 1;
      ti++;
    }
    tj = id;
  } else {
    const int nt = g.n / OZ_TILE;
    ti = blockIdx.x / nt;
    tj = blockIdx.x - ti * nt;
  }
  const int m0 = ti * OZ_TILE, n0 = tj * OZ_TILE;
  const size_t plane = (size_t)g.n * g.K;  // elements of one digit plane
  const uint16_t* Ab = g.A + (size_t)b * OZ_D * plane + (size_t)m0 * g.K;
  const uint16_t* Bb = g.B + (size_t)b * OZ_D * plane + (size_t)n0 * g.K;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(osm);
  // K is walked in exact pieces; piece p belongs to split p % nsplit
  const int K = g.len ? max(0, min(g.K, (g.len[b] - g.k0 + OZ_KC - 1) / OZ_KC * OZ_KC)) : g.K;
  const int npiece = (K + OZ_KEXACT - 1) / OZ_KEXACT;
  if (g.accumulate && split >= npiece) return;

  auto load = [&](int k0, int stage) {
    // 2 operands x 8 digits x 64 rows x 4 chunks of 16 bytes
    const uint32_t dst = sbase + stage * 2 * OZ_OPER;
#pragma unroll
    for (int i = 0; i < 2 * OZ_D * OZ_TILE * 4 / OZ_NT; i++) {
      const int t = tid + i * OZ_NT;
      const int c = t & 3, r = (t >> 2) & 63, d = (t >> 8) & 7, op = t >> 11;
      const uint16_t* src = (op ? Bb : Ab) + (size_t)d * plane + (size_t)r * g.K + k0 + c * 8;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + op * OZ_OPER + d * OZ_TILE * OZ_KC * 2 +
                                                                     oz_off(r, c)),
                   "l"(src)
                   : "memory");
    }
  };

  float acc[OZ_D][4][4];
  const int wm = (wid & 3) * 16, wn = (wid >> 2) * 32;
  const int row = wm + (lane >> 2), col = wn + 2 * (lane & 3);
  const double* sa = g.sa + (size_t)b * g.n + m0;
  const double* sb = g.sb + (size_t)b * g.n + n0;
  double* out = g.out + (size_t)b * g.obatch + (size_t)split * g.osplit;
  double* tile = reinterpret_cast<double*>(osm + (MANY ? OZ_RING : 0));  // an element is one thread's until the last piece is in
  if (split >= npiece)
    for (int t = tid; t < OZ_TILE * OZ_OUT_LD; t += OZ_NT) tile[t] = 0.0;

  for (int piece = split; piece < npiece; piece += g.nsplit) {
    const int kb = piece * OZ_KEXACT, nst = min(OZ_KEXACT, K - kb) / OZ_KC;
#pragma unroll
    for (int q = 0; q < OZ_D; q++)
#pragma unroll
      for (int t = 0; t < 4; t++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[q][t][e] = 0.f;
    __syncthreads();  // the stages are free
    for (int s = 0; s < OZ_STAGES - 1; s++) {
      if (s < nst) load(kb + s * OZ_KC, s);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int s = 0; s < nst; s++) {
      asm volatile("cp.async.wait_group %0;" ::"n"(OZ_STAGES - 2) : "memory");
      __syncthreads();
      if (s + OZ_STAGES - 1 < nst) load(kb + (s + OZ_STAGES - 1) * OZ_KC, (s + OZ_STAGES - 1) % OZ_STAGES);
      asm volatile("cp.async.commit_group;" ::: "memory");
      const uint32_t as = sbase + (s % OZ_STAGES) * 2 * OZ_OPER, bs = as + OZ_OPER;
#pragma unroll
      for (int kk = 0; kk < OZ_KC / 16; kk++) {
        uint32_t af[OZ_D][4];
#pragma unroll
        for (int d = 0; d < OZ_D; d++)
          oz_ldm4(as + d * OZ_TILE * OZ_KC * 2 + oz_off(wm + (lane & 15), 2 * kk + (lane >> 4)), af[d]);
#pragma unroll
        for (int np = 0; np < 2; np++) {
#pragma unroll
          for (int j = 0; j < OZ_D; j++) {
            // two column tiles of digit j: rows n .. n+7 and n+8 .. n+15, both K halves
            uint32_t bf[4];
            oz_ldm4(bs + j * OZ_TILE * OZ_KC * 2 +
                        oz_off(wn + 16 * np + ((lane >> 4) << 3) + (lane & 7), 2 * kk + ((lane >> 3) & 1)),
                    bf);
#pragma unroll
            for (int i = OZ_D - 1 - j; i < OZ_D; i++) {
              oz_mma(acc[i + j - (OZ_D - 1)][2 * np], af[i], bf[0], bf[1]);
              oz_mma(acc[i + j - (OZ_D - 1)][2 * np + 1], af[i], bf[2], bf[3]);
            }
          }
        }
      }
    }
    // join the accumulators: sum_q acc_q 2^(7 q), two exact integers and one rounding
    if (!MANY) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
    }
#pragma unroll
    for (int t = 0; t < 4; t++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        long long lo = 0, hi = 0;
#pragma unroll
        for (int q = 3; q >= 0; q--) {
          lo = (lo << 7) + (long long)__float2int_rn(acc[q][t][e]);
          hi = (hi << 7) + (long long)__float2int_rn(acc[q + 4][t][e]);
        }
        const double v = fma((double)hi, 268435456.0, (double)lo);  // 2^28
        const int r = row + (e >> 1) * 8, c = col + 8 * t + (e & 1);
        double* sum = tile + r * OZ_OUT_LD + c;
        const double w = v * sa[r] * sb[c] * 4.336808689942018e-19;  // 2^-61
        *sum = !MANY || piece == split ? w : *sum + w;
      }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  for (int t = tid; t < OZ_TILE * OZ_TILE; t += OZ_NT) {
    const int r = t / OZ_TILE, c = t % OZ_TILE;
    const double v = g.mirror && ti == tj && r < c ? tile[c * OZ_OUT_LD + r] : tile[r * OZ_OUT_LD + c];
    double* o = out + (size_t)(m0 + r) * g.n + n0 + c;
    *o = g.accumulate ? *o + v : v;
  }
  if ((g.mirror && ti != tj) || g.outT) {
    double* oT = g.outT ? g.outT + (size_t)b * g.obatch : out;
    for (int t = tid; t < OZ_TILE * OZ_TILE; t += OZ_NT) {
      const int c = t / OZ_TILE, r = t % OZ_TILE;
      double* o = oT + (size_t)(n0 + c) * g.n + m0 + r;
      *o = g.accumulate ? *o + tile[r * OZ_OUT_LD + c] : tile[r * OZ_OUT_LD + c];
    }
  }
}

template <bool MANY>
int oz_launch(const OzGemm& g, int nb, cudaStream_t s) {
  constexpr int bytes = OZ_RING + (MANY ? OZ_OUT : 0);
  static std::atomic<uint32_t> done{0};
  const cudaError_t e = set_smem_once(oz_gemm_kernel<MANY>, bytes, done);
  if (e != cudaSuccess) return cuda_status(e);
  const int nt = g.n / OZ_TILE;
  dim3 grid(g.lower ? nt * (nt + 1) / 2 : nt * nt, 1, nb * g.nsplit);
  oz_gemm_kernel<MANY><<<grid, OZ_NT, bytes, s>>>(g);
  note_launch();
  return cuda_status(cudaGetLastError());
}

inline int oz_gemm(const OzGemm& g, int nb, cudaStream_t s) {
  return g.K > OZ_KEXACT ? oz_launch<true>(g, nb, s) : oz_launch<false>(g, nb, s);
}

}  // namespace letkf
