// Ozaki scheme II contraction on INT8 tensor cores (tcgen05, sm_100a).
//
// C <- alpha * op(A) * op(B) + beta * C for float / double / complex with
// op(A), op(B) in {N, T, C} (the layouts of pgemm_ssb, K-major operands,
// reference src/pgemm_ssb/pgemm_ssb_host.cpp:168-171, of pgemm_sbs and of
// gemm; op(A) = N and op(B) = T, C are read in place, see 2a).
//
// Method (Ozaki, Uchino & Imamura, "Ozaki Scheme II: A GEMM-oriented emulation
// of floating-point matrix multiplication using an integer modular
// technique", 2025), restated here in our own formulation:
//   1. Complex products as two real ones per modulus: the moduli of complex
//      problems have -1 as a square, j^2 = -1 (mod p), and a = ar + i ai goes
//      to u = ar + j ai and v = ar - j ai (mod p). Then U = u_a.u_b and
//      V = v_a.v_b (for A^H, u_a and v_a swapped) are real GEMMs of depth k and
//      Re = (U + V) / 2, Im = (U - V) / (2j) mod p, with the divisions folded
//      into the reconstruction's weights: 32 real products for double (45 with
//      Karatsuba on general moduli), which took the INT8 GEMM from 9.64 to 6.62
//      ms at m = n = 1024, k = 250000 and, with k = 2048, n = 2048 and 200000 rows,
//      from 31.9 to 22.0 ms (reconstruction 9.4 to 8.1 ms); float 27 -> 20. An
//      explicit modulus count other
//      than the default keeps the moduli of real problems (not of that kind)
//      and three products (Karatsuba): P0 = ar.br, P1 = ai.bi, P2 = (ar + s ai).
//      (br + bi), s = -1 for A^H (Re = P0 + P1, Im = P2 - P0 + P1) and +1
//      otherwise (Re = P0 - P1, Im = P2 - P0 - P1).
//   2. Scaling. Every row x (complex: its interleaved reals) is scaled by
//      2^sigma so that ||2^sigma x||_2 < 2^Q and rounded to integers A', B'
//      (exact in double). By Cauchy-Schwarz every entry of the real product,
//      and Re and Im of the complex one, is below 2^(2Q) <= P/4.
//   3. Residues. For pairwise coprime moduli p_t <= 256 with product P, the
//      residues of A', B' mod p_t (symmetric, int8) are multiplied exactly on the
//      INT8 tensor cores with INT32 accumulation (k-chunks of at most 124928
//      so that the sums stay below 2^31), reduced mod p_t and summed over chunks.
//   4. Reconstruction. The Chinese remainder theorem gives X exactly (|X| <=
//      P/4, so the quotient S/P rounds to the right integer without
//      correction); C = 2^(-sigma_i - tau_j) X, then alpha/beta.
// The only rounding is the integer rounding of step 2 (relative to each row's
// 2-norm, 2^-Q) and the final conversion of X to double.
//
// Kernels: oz_row_scale (row norms -> sigma), oz_slice (scaled residues,
// int8, K-major, one plane per modulus and product), oz_slice_mma (the same for
// complex double: ozaki_slice.cuh), oz_row_scale_mn /
// oz_slice_mn (the same for op(A) = N and op(B) = T, C read in place),
// oz_transpose (op(A) = N copied K-major when k is too long for that),
// oz_gemm_pair / oz_gemm
// (tcgen05.mma kind::i8, TMA-fed, TMEM accumulators, warp-specialised
// persistent kernels), oz_reconstruct_tc (CRT sums on the tensor cores) and
// oz_reconstruct (CRT on the CUDA cores), each with
// scaling, alpha/beta and fill-mode tile skipping into C.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "ozaki.cuh"
#include "ozaki_crt.cuh"
#include "ozaki_layout.cuh"
#include "ozaki_slice.cuh"
#include "tcgen05_common.cuh"

namespace splab {
namespace oz {
using namespace tc;

constexpr int BM = 128;       // rows of A per tile (TMEM lanes)
constexpr int BN = 256;       // rows of B per tile (TMEM columns)
constexpr int BKB = 128;      // k bytes per pipeline stage (one 128-byte swizzle atom)
constexpr int STAGES = 4;
constexpr int A_STAGE = BM * BKB;  // 16 KiB
constexpr int B_STAGE = BN * BKB;  // 32 KiB
constexpr int STAGE_BYTES = A_STAGE + B_STAGE;
constexpr int GEMM_THREADS = 192;  // warp 0: TMA, warp 1: MMA, warps 2-5: epilogue
constexpr int GEMM_SMEM = STAGES * STAGE_BYTES + 1024 /*barriers*/ + 1024 /*alignment*/;
// Most k-blocks of 128 bytes per INT32 accumulation: 127/128 * 128 * 128 * k < 2^31
// for the general moduli, 122 * 122 * k < 2^31 for the split ones (p <= 241).
constexpr int kChunkBlocks = 976;        // 976 * 128 = 124928
constexpr int kChunkBlocksSplit = 1127;  // 1127 * 128 = 144256
constexpr unsigned long long kWaitLimitNs = 2000000000ull;  // 2 s bound on any wait

// --------------------------------------------------------------------------
// device helpers

// Instruction descriptor of tcgen05.mma kind::i8: S32 accumulate, signed int8
// A and B, both K-major, M = 128, N = 256.
constexpr uint32_t kIdescI8 = (2u << 4)              // D format S32
                              | (1u << 7)            // A format: signed int8
                              | (1u << 10)           // B format: signed int8
                              | (uint32_t(BN >> 3) << 17)  // N / 8
                              | (uint32_t(BM >> 4) << 24); // M / 16

// the same with an explicit instruction descriptor
__device__ __forceinline__ void umma_i8_desc(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                        uint32_t accumulate) {
  umma_i8_desc(tmem_d, adesc, bdesc, kIdescI8, accumulate);
}


// --------------------------------------------------------------------------
// 1. row scale exponents

// sigma = Q - e (+ 1) for a row with ||row||_2 = f 2^e, f in [0.5, 1) (see Crt::thr).
// Rows of zeros get sigma = 0, rows holding a NaN or an infinity get
// kSigmaNonFinite (the reconstruction then writes NaN where they contribute).
// The sum of squares is kept as S 2^(2E) with E the largest exponent seen
// (rescaled by exact powers of two when it grows), so rows of any finite
// magnitude, 1e-300 or 1e300, neither underflow nor overflow.
constexpr int kSigmaNonFinite = -(1 << 30);

// frexp-style exponent of |v| (v = f 2^e, f in [0.5, 1)); subnormals and
// zero as -1022, infinities and NaN as 1025
__device__ __forceinline__ int exponent_of(double v) {
  const int b = int((__double_as_longlong(v) >> 52) & 0x7FF);
  return (b == 0 ? 1 : b) - 1022;
}

__device__ __forceinline__ void scaled_add(double& S, int& E, double S2, int E2) {
  if (E2 > E) {
    S = ldexp(S, 2 * (E - E2)) + S2;
    E = E2;
  } else {
    S += ldexp(S2, 2 * (E2 - E));
  }
}

// Sum of squares of x[0 .. len), thread t taking t, t + blockDim.x, ...,
// into (S, E, inv): batches of 8 independent loads (memory-level
// parallelism), one exponent check per batch.
template <typename TIn>
__device__ __forceinline__ void ssq_row(const TIn* __restrict__ x, int64_t len, double& S, int& E,
                                        double& inv) {
  const int64_t step = blockDim.x;
  int64_t l = threadIdx.x;
  for (; l + 7 * step < len; l += 8 * step) {
    double v[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) v[b] = double(x[l + b * step]);
    int em = exponent_of(v[0]);
#pragma unroll
    for (int b = 1; b < 8; ++b) em = max(em, exponent_of(v[b]));
    if (em > E) {  // rare: rescale the sum to the new largest exponent
      S = ldexp(S, 2 * (E - em));
      E = em;
      inv = ldexp(1.0, -E);
    }
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const double w = v[b] * inv;
      S = fma(w, w, S);
    }
  }
  for (; l < len; l += step) {
    const double v = double(x[l]);
    const int ev = exponent_of(v);
    if (ev > E) {
      S = ldexp(S, 2 * (E - ev));
      E = ev;
      inv = ldexp(1.0, -E);
    }
    const double w = v * inv;
    S = fma(w, w, S);
  }
}

// Sums of squares of a sample of a row: kRuns runs of run reals, gap apart, each the
// sum (S, E) of 16 consecutive threads of the block's 256, in batches of 8
// independent loads (the runs are short).
constexpr int kRuns = 16;
template <typename TIn>
__device__ __forceinline__ void ssq_sample(const TIn* __restrict__ x, int64_t run, int64_t gap,
                                           double& S, int& E, double& inv) {
  constexpr int gsz = 256 / kRuns;
  static_assert(gsz == 16, "a half warp per run");
  x += int(threadIdx.x) / gsz * gap;
  for (int64_t l = threadIdx.x % gsz; l < run; l += 8 * gsz) {
    double v[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) v[b] = l + b * gsz < run ? double(x[l + b * gsz]) : 0.0;
    int em = exponent_of(v[0]);
#pragma unroll
    for (int b = 1; b < 8; ++b) em = max(em, exponent_of(v[b]));
    if (em > E) {
      S = ldexp(S, 2 * (E - em));
      E = em;
      inv = ldexp(1.0, -E);
    }
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const double w = v[b] * inv;
      S = fma(w, w, S);
    }
  }
  for (int o = gsz / 2; o > 0; o >>= 1) {
    const double S2 = __shfl_xor_sync(0xffffffffu, S, o);
    const int E2 = __shfl_xor_sync(0xffffffffu, E, o);
    scaled_add(S, E, S2, E2);
  }
}

// The runs' sums (ssq_sample) added up into warp 0's (S, E), and the runs' relative
// variance about their mean into its `spread` (1 + spread = kRuns sum_c (S_c / S)^2).
__device__ __forceinline__ void block_sample(double& S, int& E, double& spread, double* redS,
                                             int* redE) {
  if ((threadIdx.x & 15) == 0) {
    redS[threadIdx.x >> 4] = S;
    redE[threadIdx.x >> 4] = E;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const double Sc = redS[threadIdx.x & (kRuns - 1)];  // both half warps alike
    const int Ec = redE[threadIdx.x & (kRuns - 1)];
    S = Sc;
    E = Ec;
    for (int o = kRuns / 2; o > 0; o >>= 1) {
      const double S2 = __shfl_xor_sync(0xffffffffu, S, o);
      const int E2 = __shfl_xor_sync(0xffffffffu, E, o);
      scaled_add(S, E, S2, E2);
    }
    const double part = ldexp(Sc, 2 * (Ec - E)) / S;
    double sq = part * part;
    for (int o = kRuns / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    spread = kRuns * sq - 1.0;
  }
}

// The block's (S, E) summed into thread 0's (blocks of at most 1024 threads)
__device__ __forceinline__ void block_ssq(double& S, int& E, double* redS, int* redE) {
  for (int o = 16; o > 0; o >>= 1) {
    const double S2 = __shfl_xor_sync(0xffffffffu, S, o);
    const int E2 = __shfl_xor_sync(0xffffffffu, E, o);
    scaled_add(S, E, S2, E2);
  }
  if ((threadIdx.x & 31) == 0) {
    redS[threadIdx.x >> 5] = S;
    redE[threadIdx.x >> 5] = E;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const bool have = threadIdx.x < (blockDim.x >> 5);
    S = have ? redS[threadIdx.x] : 0.0;
    E = have ? redE[threadIdx.x] : -2100;
    for (int o = 16; o > 0; o >>= 1) {
      const double S2 = __shfl_xor_sync(0xffffffffu, S, o);
      const int E2 = __shfl_xor_sync(0xffffffffu, E, o);
      scaled_add(S, E, S2, E2);
    }
  }
}

// Bits and threshold of the scale exponents (Crt::q_bits, Crt::thr)
struct ScaleBits {
  int q;
  double thr;
};

// sigma from the exponent-tracked sum of squares S 2^(2E) of a row
__device__ __forceinline__ int sigma_of(double S, int E, ScaleBits b) {
  if (!(S < 1e300)) return kSigmaNonFinite;  // NaN or infinite input
  if (S > 0.0) {
    int e0 = 0;
    const double f = frexp(sqrt(S), &e0);
    return b.q - (e0 + E) + (f < b.thr ? 1 : 0);
  }
  return 0;
}

// Row scale exponents of up to two k-major operands (len reals per row; rows = 0:
// none) in one launch.
struct RowScaleOp {
  const void* X;
  int64_t ld;    // reals between rows
  int rows;
  int* sigma;
  // one-pass scaling: whether the exponent is exact, the sums of squares of the
  // scaled reals, the rows to slice again and their count
  int* exact;
  double* ssq;
  int* list;
  int* count;
};
struct RowScaleParams {
  RowScaleOp op[2];
  int64_t len;
  ScaleBits bits;
  int64_t run, gap;   // kEstimate: runs of `run` reals, `gap` apart
  double lo, hi;      // kRecheck: range of ssq that proves an estimate
  int* status;        // cleared by kExact and kEstimate
};

// kExact: one block per row, the exact exponent. kEstimate: the exponent from a
// sample of the row (the sum of squares of kRuns runs extrapolated to len reals)
// when the estimated norm is clear of the exponents' change (estimate_clear;
// exact[row] = 0), else, and for a zero or non-finite sample, the exact one
// (exact[row] = 1); clears the rows' sums of squares and the counts. kRecheck
// (blocks grid-stride over the rows): a row whose exponent was estimated keeps
// it when its sum of squares at that scale lies within [lo, hi] (the exponent is
// then the exact one, and clear of the rounding of the sum); otherwise (the
// estimate was off, the row is zero or not finite, or the sum lies near the
// exponents' change) it gets its exact exponent and is listed for a second slicing.
enum RowScaleMode { kExact, kEstimate, kRecheck };
template <typename TIn, int MODE>
__global__ void __launch_bounds__(256) oz_row_scale(const __grid_constant__ RowScaleParams P) {
  __shared__ double redS[32];
  __shared__ int redE[32];
  __shared__ int use_estimate;
  const int total = P.op[0].rows + P.op[1].rows;
  if (MODE != kRecheck && blockIdx.x == 0 && threadIdx.x < 3) {
    if (threadIdx.x == 2)
      *P.status = 0;
    else if (MODE == kEstimate && P.op[threadIdx.x].rows > 0)
      *P.op[threadIdx.x].count = 0;
  }
  for (int bi = blockIdx.x; bi < total; bi += gridDim.x) {
    const int which = bi < P.op[0].rows ? 0 : 1;
    const RowScaleOp& op = P.op[which];
    const int row = bi - (which ? P.op[0].rows : 0);
    const TIn* x = static_cast<const TIn*>(op.X) + int64_t(row) * op.ld;
    double S = 0.0, inv = 0.0;  // sum of (v 2^-E)^2, and 2^-E
    int E = -2100;              // below any exponent: the first batch sets it
    if (MODE == kRecheck) {
      const double s = op.ssq[row];
      if (op.exact[row] || (s >= P.lo && s <= P.hi)) continue;  // block-uniform
    }
    if (MODE == kEstimate) {
      double spread = 0.0;
      ssq_sample(x, P.run, P.gap, S, E, inv);
      block_sample(S, E, spread, redS, redE);
      if (threadIdx.x == 0) {
        bool use = false;
        if (S > 0.0 && S < 1e300) {
          int e0 = 0;
          const double f = frexp(sqrt(S * (double(P.len) / (kRuns * double(P.run)))), &e0);
          use = estimate_clear(f, P.bits.thr, spread / (kRuns - 1));
          if (use) op.sigma[row] = P.bits.q - (e0 + E) + (f < P.bits.thr ? 1 : 0);
        }
        op.exact[row] = use ? 0 : 1;
        op.ssq[row] = 0.0;
        use_estimate = use;
      }
      __syncthreads();
      const bool done = use_estimate;
      S = 0.0;
      inv = 0.0;
      E = -2100;
      if (done) continue;  // block-uniform; the next row's first barrier
                           // comes after this row's last read of use_estimate
    }
    ssq_row(x, P.len, S, E, inv);
    block_ssq(S, E, redS, redE);
    if (threadIdx.x == 0) {
      op.sigma[row] = sigma_of(S, E, P.bits);
      if (MODE == kRecheck) op.list[atomicAdd(op.count, 1)] = row;
    }
    __syncthreads();  // redS / redE are reused by the block's next row
  }
}

// --------------------------------------------------------------------------
// 2. residues

// Per-modulus constants of the slicer, each stored twice (both halves of an
// f32x2 operand): -p, 1/p and the digit weights b^i mod p in symmetric form,
// i = 1..4 (digit base b = 2^15 with four digits, else 2^13); with split moduli
// also the weights of the imaginary part, j b^i mod p, i = 0..4 (-j for A^H).
struct SliceConsts {
  int n;
  float p0;  // first modulus (256: residue = low byte of the lowest digit)
  unsigned long long neg_p[kMaxModuli];
  unsigned long long inv_p[kMaxModuli];
  unsigned long long c[kMaxModuli][4];
  unsigned long long cj[kMaxModuli][5];
};

// Residues are computed on the FP32 pipe from digits of the scaled integer
// x = round(2^sigma y), x = sum_i d_i b^i, which are extracted without
// conversion instructions: x = xh 2^h + xl with xh = round(y 2^-h), both read
// as integers from the bits of (value + 1.5 2^52).
//   NDIG 3 and 5 (|x| < 2^39, < 2^62): b = 2^13, h = 26; d_0 = xl mod 2^13
//     (0 .. 8191), d_1 = xl >> 13 (|d_1| <= 4096), xh gives d_2.. the same
//     way (top digit signed); the digit sum below stays under 2^22.
//   NDIG 4 (|x| < 2^58, the default for double): b = 2^15, h = 30, balanced
//     digits (|d_0|, |d_1|, |d_2| <= 2^14 + 1, |d_3| <= 2^13 + 1): one digit
//     fewer; the digit sum stays under 5.3e6 < 2^23.
// For a modulus p the digit sum s = d_0 + sum_i c_i d_i (c_i = b^i mod p in
// symmetric form, |c_i| <= p/2) is exact in FP32, and since |s| < 2^23 the
// quotient rounded from s * fl(1/p) is the nearest integer to s / p (for odd
// p, s / p is at least 1/(2p) away from a half-integer; the product's error is
// below that); r = s - p * nearest(s / p) lies in [-(p-1)/2, (p-1)/2]. For
// p = 256 the weights vanish and r is the low byte of d_0. Each residue is
// produced as the float MAGIC + r, whose low byte is r in two's complement:
// the int8 value without a conversion.
__device__ __forceinline__ float small_int_to_float(int d) {  // |d| < 2^22
  return __int_as_float(0x4B400000 + d) - 12582912.0f;
}

template <int NDIG>
__device__ __forceinline__ void digits13(double y, float (&d)[5]) {
  constexpr double kM52 = 6755399441055744.0;  // 1.5 * 2^52: ulp 1
  constexpr long long kM52Bits = 0x4338000000000000ll;
  if (NDIG == 4) {  // balanced base-2^15 digits, |x| < 2^58
    const double t = fma(y, 1.0 / 1073741824.0, kM52);  // kM52 + round(y 2^-30)
    const double xl_d = fma(t - kM52, -1073741824.0, y);  // exact, |xl_d| <= 2^29
    const int xl = int(__double2loint(xl_d + kM52));
    const int xh = int(__double_as_longlong(t) - kM52Bits);  // |xh| <= 2^28 + 1
    // balanced digits: with u = x + 2^14, d_lo = (u mod 2^15) - 2^14 and
    // d_hi = (x - d_lo) / 2^15 = floor(u / 2^15)
    const int u0 = xl + 0x4000, u2 = xh + 0x4000;
    d[0] = small_int_to_float((u0 & 0x7FFF) - 0x4000);
    d[1] = small_int_to_float(u0 >> 15);
    d[2] = small_int_to_float((u2 & 0x7FFF) - 0x4000);
    d[3] = small_int_to_float(u2 >> 15);
    d[4] = 0.0f;
    return;
  }
  const double t = fma(y, 1.0 / 67108864.0, kM52);  // kM52 + round(y 2^-26)
  const double xl_d = fma(t - kM52, -67108864.0, y);  // exact, |xl_d| <= 2^25
  const int xl = int(__double2loint(xl_d + kM52));  // round(xl_d), two's complement
  const long long xh = __double_as_longlong(t) - kM52Bits;
  d[0] = small_int_to_float(xl & 0x1FFF);
  d[1] = small_int_to_float(xl >> 13);
  if (NDIG == 3) {
    d[2] = small_int_to_float(int(xh));
  } else {
    d[2] = small_int_to_float(int(xh & 0x1FFF));
    d[3] = small_int_to_float(int((xh >> 13) & 0x1FFF));
    d[4] = small_int_to_float(int(xh >> 26));
  }
#pragma unroll
  for (int i = NDIG; i < 5; ++i) d[i] = 0.0f;
}

constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: ulp 1, low mantissa bits hold r

// Type of a slicing thread's reals: float rows with three digits stay in FP32.
template <typename TIn, int NDIG>
using SliceReal = typename std::conditional<sizeof(TIn) == 4 && NDIG == 3, float, double>::type;

// Digits of two floats with |2^sg v| < 2^39 without FP64: the scaled value y is
// exact, d_2 = rint(y 2^-26), d_1 = rint(y_1 2^-13) and d_0 = rint(y_0) with the exact
// remainders y_1 = y - 2^26 d_2 (a multiple of ulp(y), at most 2^25) and y_0 = y_1 -
// 2^13 d_1; so x = round(y), ties to even, as the FP64 digits give it. |d_0|, |d_1| <=
// 2^12, |d_2| <= 2^13. 10 packed operations per two reals and no conversion to double:
// 3072 rows x 400000 floats 2.1 -> 2.0 ms per operand, the call 9.15 -> 8.96 ms;
// complex float 771 x 1003 x 130001 4.30 -> 4.09 ms.
__device__ __forceinline__ unsigned long long digits_f32(unsigned long long v,
                                                         unsigned long long s1,
                                                         unsigned long long s2,
                                                         unsigned long long (&d)[5]) {
  const unsigned long long M = f2_pack(kMagic, kMagic), NM = f2_pack(-kMagic, -kMagic);
  const float h26 = 1.0f / 67108864.0f, h13 = 1.0f / 8192.0f;
  const unsigned long long y = f2_mul(f2_mul(v, s1), s2);
  d[2] = f2_add(f2_fma(y, f2_pack(h26, h26), M), NM);
  const unsigned long long y1 = f2_fma(d[2], f2_pack(-67108864.0f, -67108864.0f), y);
  d[1] = f2_add(f2_fma(y1, f2_pack(h13, h13), M), NM);
  d[0] = f2_add(f2_add(f2_fma(d[1], f2_pack(-8192.0f, -8192.0f), y1), M), NM);
  d[3] = d[4] = 0;
  return y;
}

// The work of one slicing thread once its EL reals (of one row, starting at
// real l0) are loaded: scaling by 2^sg, digits, and for every modulus the
// residues written to res_row + l0 (mode 0) or, in modes 2 and 3, to the three
// or two planes `plane` bytes apart at complex offset l0 / 2. SSQ: the sum of
// squares of the scaled values is handed to on_ssq once the digits are made
// (so that it is not kept in registers through the residue loop).
struct NoSsq {
  __device__ void operator()(double) const {}
};
template <typename TIn, int NDIG, int EL, int NMU, int MODE, bool SSQ = false,
          typename OnSsq = NoSsq>
__device__ __forceinline__ void slice_thread(SliceReal<TIn, NDIG> (&v)[EL], int sg,
                                             int8_t* res_row, int64_t l0, int64_t plane, int s_sum,
                                             int64_t res_mod_stride, const SliceConsts& sc,
                                             OnSsq on_ssq = {}) {
  static_assert(EL == 8 || EL == 16, "8 or 16 reals per thread");
  static_assert(MODE == 0 || MODE == 2 || MODE == 3, "real rows, or complex rows in two forms");
  constexpr int W = EL / 4;  // packed words per modulus
  using V = SliceReal<TIn, NDIG>;
  // 2^sg as a double when representable, else ldexp per element
  const bool direct = sg > -1000 && sg < 1000;
  const double scale = direct ? __longlong_as_double((long long)(sg + 1023) << 52) : 1.0;
  unsigned long long dp[EL / 2][5];  // digits of the element pairs (see below)
  double ssq = 0.0;
  {
    // pairs (2i, 2i + 1) in mode 0; for complex rows the real parts pair up first,
    // then the imaginary parts: (re0, re1), (re2, re3), ..., (im0, im1), ...
    if constexpr (MODE != 0) {
      V u[EL];
#pragma unroll
      for (int i = 0; i < EL / 2; ++i) {
        u[i] = v[2 * i];
        u[EL / 2 + i] = v[2 * i + 1];
      }
#pragma unroll
      for (int i = 0; i < EL; ++i) v[i] = u[i];
    }
    if constexpr (std::is_same<V, float>::value) {
      // 2^sg in two factors (rows of subnormals: sg up to 187), clamped for the rows
      // marked as not finite
      const int h1 = max(-126, min(127, sg >> 1)), h2 = max(-126, min(127, sg - (sg >> 1)));
      const float f1 = __int_as_float((h1 + 127) << 23), f2 = __int_as_float((h2 + 127) << 23);
      unsigned long long sq = 0;
#pragma unroll
      for (int i = 0; i < EL / 2; ++i) {
        const unsigned long long y = digits_f32(f2_pack(v[2 * i], v[2 * i + 1]), f2_pack(f1, f1),
                                                f2_pack(f2, f2), dp[i]);
        if constexpr (SSQ) sq = f2_fma(y, y, sq);
      }
      if constexpr (SSQ) {
        float a, b;
        f2_unpack(sq, a, b);
        ssq = double(a) + double(b);
      }
    } else {
#pragma unroll
      for (int i = 0; i < EL / 2; ++i) {
        float d0[5], d1[5];
        const double y0 = direct ? v[2 * i] * scale : ldexp(v[2 * i], sg);
        const double y1 = direct ? v[2 * i + 1] * scale : ldexp(v[2 * i + 1], sg);
        if constexpr (SSQ) ssq = fma(y1, y1, fma(y0, y0, ssq));
        digits13<NDIG>(y0, d0);
        digits13<NDIG>(y1, d1);
#pragma unroll
        for (int j = 0; j < 5; ++j) dp[i][j] = f2_pack(d0[j], d1[j]);
      }
    }
    if constexpr (SSQ) on_ssq(ssq);
  }
  const unsigned long long M2 = f2_pack(kMagic, kMagic), NM2 = f2_pack(-kMagic, -kMagic);
  int8_t* const out0 = res_row + l0;
  constexpr int H = EL / 4;  // modes 2, 3: pairs of complex elements
  // Mode 3, one modulus: with sr and si the digit sums of re and j im, u = sr +
  // si (accumulated in one chain) and -v = u - 2 sr, each exact in FP32: with
  // four digits of base 2^15 and weights |c| <= h = (p - 1) / 2 <= 120, |u| and
  // |v| <= 2^14 (1 + 6 h) < 1.2e7 < 2^24, and less with the others. V's planes
  // hold -v for both operands, which leaves the products. The quotients are
  // below 49400, so their error (2^-24 relative from 1/p) is below 0.003: the
  // nearest integer or, next to a half, its neighbour, |r| <= 121: one signed
  // byte. 16 operations per complex element and modulus against 19 in mode 2.
  auto modulus_split = [&](const int t) {
    const unsigned long long np = sc.neg_p[t], ip = sc.inv_p[t];
    const unsigned long long TWO = f2_pack(-2.0f, -2.0f);
    unsigned long long ru[H], rv[H];
#pragma unroll
    for (int h = 0; h < H; ++h) {
      unsigned long long sr = f2_fma(sc.c[t][0], dp[h][1], dp[h][0]);
#pragma unroll
      for (int d = 2; d < NDIG; ++d) sr = f2_fma(sc.c[t][d - 1], dp[h][d], sr);
      unsigned long long u = f2_fma(sc.cj[t][0], dp[H + h][0], sr);
#pragma unroll
      for (int d = 1; d < NDIG; ++d) u = f2_fma(sc.cj[t][d], dp[H + h][d], u);
      const unsigned long long v = f2_fma(sr, TWO, u);
      const unsigned long long qu = f2_add(f2_fma(u, ip, M2), NM2);
      const unsigned long long qv = f2_add(f2_fma(v, ip, M2), NM2);
      ru[h] = f2_add(f2_fma(qu, np, u), M2);
      rv[h] = f2_add(f2_fma(qv, np, v), M2);
    }
    int8_t* o = out0 - l0 + l0 / 2 + t * res_mod_stride;  // complex offset l0 / 2
#pragma unroll
    for (int w = 0; w < H / 2; ++w) {
      float a0, a1, a2, a3;
      f2_unpack(ru[2 * w], a0, a1);
      f2_unpack(ru[2 * w + 1], a2, a3);
      *reinterpret_cast<uint32_t*>(o + 4 * w) = pack4(a0, a1, a2, a3);
      f2_unpack(rv[2 * w], a0, a1);
      f2_unpack(rv[2 * w + 1], a2, a3);
      *reinterpret_cast<uint32_t*>(o + plane + 4 * w) = pack4(a0, a1, a2, a3);
    }
  };
  auto modulus = [&](const int t) {
    if constexpr (MODE == 3) {
      modulus_split(t);
      return;
    }
    int8_t* out = out0 + t * res_mod_stride;
    unsigned long long rp2[EL / 2];  // MAGIC + residue of elements 2i, 2i + 1
    unsigned long long ri2[H];       // mode 2: residues of the imaginary pairs, unbiased
    if (t == 0 && sc.p0 == 256.0f) {
#pragma unroll
      for (int i = 0; i < EL / 2; ++i) rp2[i] = f2_add(dp[i][0], M2);
      if constexpr (MODE == 2) {
#pragma unroll
        for (int h = 0; h < H; ++h) ri2[h] = dp[H + h][0];
      }
    } else {
      const unsigned long long np = sc.neg_p[t], ip = sc.inv_p[t];
      const unsigned long long c1 = sc.c[t][0], c2 = sc.c[t][1], c3 = sc.c[t][2],
                               c4 = sc.c[t][3];
#pragma unroll
      for (int i = 0; i < EL / 2; ++i) {
        unsigned long long s2 = f2_fma(c1, dp[i][1], dp[i][0]);
        if (NDIG > 2) s2 = f2_fma(c2, dp[i][2], s2);
        if (NDIG > 3) s2 = f2_fma(c3, dp[i][3], s2);
        if (NDIG > 4) s2 = f2_fma(c4, dp[i][4], s2);
        const unsigned long long q2 = f2_add(f2_fma(s2, ip, M2), NM2);
        // |s| may exceed 2^22 with four digits (s + MAGIC is not exact): r
        // first, then MAGIC + r; both exact. Otherwise one operation fewer.
        if (NDIG == 4 || (MODE == 2 && i >= H)) {
          const unsigned long long r2 = f2_fma(q2, np, s2);
          rp2[i] = f2_add(r2, M2);
          if (MODE == 2 && i >= H) ri2[i - H] = r2;
        } else {
          rp2[i] = f2_fma(q2, np, f2_add(s2, M2));
        }
      }
    }
    float r[EL];
#pragma unroll
    for (int i = 0; i < EL / 2; ++i) f2_unpack(rp2[i], r[2 * i], r[2 * i + 1]);
    uint32_t wu[W];
    if constexpr (MODE == 0) {
#pragma unroll
      for (int q = 0; q < W; ++q)
        wu[q] = pack4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
      if constexpr (W == 4)
        *reinterpret_cast<uint4*>(out) = make_uint4(wu[0], wu[1], wu[2], wu[3]);
      else
        *reinterpret_cast<uint2*>(out) = make_uint2(wu[0], wu[1]);
    } else {
      // rp2[h] = MAGIC + residues of (re_2h, re_2h+1), rp2[H + h] those of the
      // imaginary parts (ri2[h] without MAGIC). Third plane: t = r(re) +
      // s_sum r(im) (|t| < 2^16): MAGIC + t exactly in one FMA, t, its nearest
      // quotient by p and MAGIC + (t - q p) = (MAGIC + t) - q p (for p = 256
      // the residues are unreduced low bytes and the reduction gives the low
      // byte of the sum)
      const unsigned long long np = sc.neg_p[t], ip = sc.inv_p[t];
      const unsigned long long S2 = f2_pack(float(s_sum), float(s_sum));
      unsigned long long sm2[H];
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const unsigned long long tM = f2_fma(S2, ri2[h], rp2[h]);
        const unsigned long long t2 = f2_add(tM, NM2);
        const unsigned long long q2 = f2_add(f2_fma(t2, ip, M2), NM2);
        sm2[h] = f2_fma(q2, np, tM);
      }
      int8_t* o = out0 - l0 + l0 / 2 + t * res_mod_stride;  // complex offset l0 / 2
#pragma unroll
      for (int w = 0; w < H / 2; ++w) {
        float a0, a1, a2, a3;
        f2_unpack(rp2[2 * w], a0, a1);
        f2_unpack(rp2[2 * w + 1], a2, a3);
        *reinterpret_cast<uint32_t*>(o + 4 * w) = pack4(a0, a1, a2, a3);
        f2_unpack(rp2[H + 2 * w], a0, a1);
        f2_unpack(rp2[H + 2 * w + 1], a2, a3);
        *reinterpret_cast<uint32_t*>(o + plane + 4 * w) = pack4(a0, a1, a2, a3);
        f2_unpack(sm2[2 * w], a0, a1);
        f2_unpack(sm2[2 * w + 1], a2, a3);
        *reinterpret_cast<uint32_t*>(o + 2 * plane + 4 * w) = pack4(a0, a1, a2, a3);
      }
    }
  };
  if constexpr (NMU > 0) {
#pragma unroll
    for (int t = 0; t < NMU; ++t) modulus(t);
  } else {
    for (int t = 0; t < sc.n; ++t) modulus(t);
  }
}

// Residues of one operand, written K-major (row stride kp bytes).
// Each thread handles EL (8 or 16) consecutive reals of one row.
// mode 0: real rows: res[t][row][l], l < kp.
// mode 2: complex rows for the three-product (Karatsuba) form: complex element
//         e = (re, im) of row `row` goes to three planes of `rows` x kp bytes,
//         res[t][0][row][e] = r(re), res[t][1][row][e] = r(im) and
//         res[t][2][row][e] = r(re + s_sum im) (residues are linear in the
//         scaled integers, so the third is r(re) + s_sum r(im) reduced mod p).
//         The input row then holds 2 kp reals (kp complex elements).
// mode 3: complex rows with split moduli: res[t][0][row][e] = r(re + j im),
//         res[t][1][row][e] = -r(re - j im).
// TIn: double (|x| < 2^62, five digits) or float (|x| < 2^38, three digits).
// NMU > 0: the moduli in one fully unrolled pass (the per-modulus constants
// become fixed parameter operands); 0: sc.n moduli in a loop.
// MODE (the mode above) is a template parameter so that the unrolled
// modulus loop carries no branch on it.
// The EL reals of one row at real l0 (zeros past len); VEC: 16-byte loads.
template <typename TIn, bool VEC, int EL, typename V>
__device__ __forceinline__ void load_reals(const TIn* __restrict__ x, int64_t l0, int64_t len,
                                           V (&v)[EL]) {
  if (VEC && l0 + EL <= len) {
    if constexpr (sizeof(TIn) == 8) {
#pragma unroll
      for (int i = 0; i < EL / 2; ++i) {
        const double2 t = __ldg(reinterpret_cast<const double2*>(x) + i);
        v[2 * i] = t.x;
        v[2 * i + 1] = t.y;
      }
    } else {
#pragma unroll
      for (int i = 0; i < EL / 4; ++i) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(x) + i);
        v[4 * i] = t.x;
        v[4 * i + 1] = t.y;
        v[4 * i + 2] = t.z;
        v[4 * i + 3] = t.w;
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < EL; ++i) v[i] = (l0 + i < len) ? V(x[i]) : V(0);
  }
}

// Where slice_thread's row starts, for a thread at real l0 of it: pieces of
// kc elements (split moduli) lie G kc apart.
template <int MODE>
__device__ __forceinline__ int8_t* row_base(int8_t* res, const ResidueLayout& lay, int row,
                                            int64_t l0) {
  int8_t* r = res + int64_t(row) * lay.row;
  return MODE == 3 ? r + (lay.at(l0 / 2) - l0 / 2) : r;
}

// SSQ: also adds each row's sum of squares of the scaled values to
// rowssq[row] (one atomic per row and block; blocks of 256 threads).
template <typename TIn, bool VEC, int NDIG, int EL, int NMU, int MODE, bool SSQ = false>
__global__ void __launch_bounds__(256, EL == 8 ? 4 : 2)
    oz_slice(const TIn* __restrict__ X, int64_t ld_doubles, int64_t len, int rows, int64_t kp,
             const int* __restrict__ sigma, int s_sum, int8_t* __restrict__ res,
             ResidueLayout lay, int64_t res_mod_stride, SliceConsts sc,
             double* __restrict__ rowssq) {
  const int64_t groups = (MODE != 0 ? 2 * kp : kp) / EL;
  const int64_t gid = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if constexpr (!SSQ) {
    const int row = int(gid / groups);
    if (row >= rows) return;
    const int64_t l0 = (gid % groups) * EL;
    SliceReal<TIn, NDIG> v[EL];
    load_reals<TIn, VEC, EL>(X + int64_t(row) * ld_doubles + l0, l0, len, v);
    slice_thread<TIn, NDIG, EL, NMU, MODE>(v, sigma[row], row_base<MODE>(res, lay, row, l0), l0,
                                           lay.plane(1), s_sum, res_mod_stride, sc);
  } else {
    // Threads past the last row redo the last row's last groups (the same
    // bytes to the same places) so that every thread takes part in the
    // reductions; their sums count as zero. Aligned segments of W lanes (W
    // the largest power of two dividing groups, at most 32; at least 8,
    // groups being kp / 8 or kp / 16 with kp a multiple of 128) hold one row
    // each: reduced by shuffles, then the block's segments of one row
    // together, one atomic per row and block (atomics from every warp on the
    // few rows the resident blocks share would serialise).
    __shared__ double seg_sum[32];
    __shared__ int seg_row[32];
    const int W = int(groups & -groups) < 32 ? int(groups & -groups) : 32;
    const int nseg = int(blockDim.x) / W;  // blocks of 256 threads: at most 32
    const int row_in = int(gid / groups);
    const int64_t g_in = gid % groups;
    const bool past = row_in >= rows;
    const int row = past ? rows - 1 : row_in;
    const int64_t l0 = (past ? groups - W + (g_in & (W - 1)) : g_in) * EL;
    SliceReal<TIn, NDIG> v[EL];
    load_reals<TIn, VEC, EL>(X + int64_t(row) * ld_doubles + l0, l0, len, v);
    auto on_ssq = [&](double ssq) {
      if (past) ssq = 0.0;
      for (int o = 16; o > 0; o >>= 1)
        if (o < W) ssq += __shfl_xor_sync(0xffffffffu, ssq, o);
      if ((threadIdx.x & (W - 1)) == 0) {
        seg_sum[threadIdx.x / W] = ssq;
        seg_row[threadIdx.x / W] = past ? -1 : row;
      }
    };
    slice_thread<TIn, NDIG, EL, NMU, MODE, true>(v, sigma[row], row_base<MODE>(res, lay, row, l0),
                                                 l0, lay.plane(1), s_sum, res_mod_stride, sc,
                                                 on_ssq);
    __syncthreads();
    if (int(threadIdx.x) < nseg) {
      const int sgi = threadIdx.x, r = seg_row[sgi];
      if (r >= 0 && (sgi == 0 || seg_row[sgi - 1] != r)) {  // first segment of its row
        double t = 0.0;
        for (int u = sgi; u < nseg && seg_row[u] == r; ++u) t += seg_sum[u];
        atomicAdd(rowssq + r, t);
      }
    }
  }
}

// oz_slice over the rows list[0 .. *count - 1] (grid-stride over their
// thread groups): the rows the one-pass check sent back (see kRecheck)
template <typename TIn, bool VEC, int NDIG, int EL, int NMU, int MODE>
__global__ void __launch_bounds__(256, EL == 8 ? 4 : 2)
    oz_slice_rows(const TIn* __restrict__ X, int64_t ld_doubles, int64_t len, int rows,
                  int64_t kp, const int* __restrict__ sigma, int s_sum,
                  int8_t* __restrict__ res, ResidueLayout lay, int64_t res_mod_stride,
                  SliceConsts sc, const int* __restrict__ list, const int* __restrict__ count) {
  const int64_t groups = (MODE != 0 ? 2 * kp : kp) / EL;
  const int64_t total = int64_t(*count) * groups;
  for (int64_t gid = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; gid < total;
       gid += int64_t(gridDim.x) * blockDim.x) {
    const int row = list[gid / groups];
    const int64_t l0 = (gid % groups) * EL;
    SliceReal<TIn, NDIG> v[EL];
    load_reals<TIn, VEC, EL>(X + int64_t(row) * ld_doubles + l0, l0, len, v);
    slice_thread<TIn, NDIG, EL, NMU, MODE>(v, sigma[row], row_base<MODE>(res, lay, row, l0), l0,
                                           lay.plane(1), s_sum, res_mod_stride, sc);
  }
}

// --------------------------------------------------------------------------
// 2a. operands read in place: op(A) = N (A m-major: element (i, kk) at
// X[i + kk ld], the rows of op(A) are the columns of X) and op(B) = T or C
// (B n-major the same way). Instead of a k-major copy the norms read them
// along the rows and the slicer transposes tiles through shared memory.
constexpr int kMnRows = 65536;  // rows from which the norms need no k-slicing

// Row scale exponents of m-major rows, as oz_row_scale computes them: one
// thread per row and k-slice (a warp reads 32 consecutive rows of one kk:
// coalesced), batches of 8 loads in flight. With one k-slice (gridDim.y == 1)
// the thread writes sigma; with several it writes its partial sum (S, E) to
// partS / partE [slice][row] for oz_row_scale_combine.
template <typename TIn, bool CPLX>
__global__ void __launch_bounds__(256) oz_row_scale_mn(const TIn* __restrict__ X, int64_t ld,
                                                       int m, int64_t k, int64_t kspan,
                                                       ScaleBits bits,
                                                       int* __restrict__ sigma,
                                                       double* __restrict__ partS,
                                                       int* __restrict__ partE) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  constexpr int R = CPLX ? 2 : 1;  // reals per element
  const TIn* x = X + int64_t(i) * R;
  const int64_t step = ld * R;  // reals between consecutive kk
  double S = 0.0, inv = 0.0;
  int E = -2100;
  int64_t kk = int64_t(blockIdx.y) * kspan;
  const int64_t kend = min(k, kk + kspan);
  for (; kk + 8 <= kend; kk += 8) {
    double v[8 * R];
#pragma unroll
    for (int b = 0; b < 8; ++b)
#pragma unroll
      for (int c = 0; c < R; ++c) v[b * R + c] = double(x[(kk + b) * step + c]);
    int em = exponent_of(v[0]);
#pragma unroll
    for (int b = 1; b < 8 * R; ++b) em = max(em, exponent_of(v[b]));
    if (em > E) {
      S = ldexp(S, 2 * (E - em));
      E = em;
      inv = ldexp(1.0, -E);
    }
#pragma unroll
    for (int b = 0; b < 8 * R; ++b) {
      const double w = v[b] * inv;
      S = fma(w, w, S);
    }
  }
  for (; kk < kend; ++kk) {
#pragma unroll
    for (int c = 0; c < R; ++c) {
      const double v = double(x[kk * step + c]);
      const int ev = exponent_of(v);
      if (ev > E) {
        S = ldexp(S, 2 * (E - ev));
        E = ev;
        inv = ldexp(1.0, -E);
      }
      const double w = v * inv;
      S = fma(w, w, S);
    }
  }
  if (gridDim.y == 1) {
    sigma[i] = sigma_of(S, E, bits);
  } else {
    partS[int64_t(blockIdx.y) * m + i] = S;
    partE[int64_t(blockIdx.y) * m + i] = E;
  }
}

// sigma of each row from its k-slice partial sums: 32 rows per block, one thread
// of each of its warps (8 to 32) to a row
__global__ void __launch_bounds__(1024) oz_row_scale_combine(const double* __restrict__ partS,
                                                            const int* __restrict__ partE, int m,
                                                            int slices, ScaleBits bits,
                                                            int* __restrict__ sigma) {
  __shared__ double sumS[32][32];
  __shared__ int sumE[32][32];
  const int warps = int(blockDim.x) >> 5;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  double S = 0.0;
  int E = -2100;
  if (i < m)
#pragma unroll 4
    for (int sl = w; sl < slices; sl += warps)
      scaled_add(S, E, partS[int64_t(sl) * m + i], partE[int64_t(sl) * m + i]);
  sumS[w][lane] = S;
  sumE[w][lane] = E;
  __syncthreads();
  if (w != 0 || i >= m) return;
  for (int v = 1; v < warps; ++v) scaled_add(S, E, sumS[v][lane], sumE[v][lane]);
  sigma[i] = sigma_of(S, E, bits);
}

// Raw element of ESZ bytes (a complex or real value of TIn) in shared memory
template <int ESZ> struct RawElem;
template <> struct RawElem<16> { using T = double2; };
template <> struct RawElem<8> { using T = unsigned long long; };
template <> struct RawElem<4> { using T = unsigned int; };

// Residues of m-major rows: a block covers 8 rows (one warp each) and, per row,
// the KT = 32 G elements of one warp row (G = EL / reals per element: 4
// complex or 8 real). The tile is read along i (8 consecutive rows per kk) into
// shared memory and read back along kk; the element index is XOR-swizzled
// within groups of 128 bytes and the row stride is odd, so that the reads are
// free of bank conflicts (the writes at most 2-way, 4-way for real float).
// Each thread then does oz_slice's work (slice_thread) on its EL = 8 reals.
// VEC: 16-byte loads of complex double elements (the base is 16-byte aligned).
// conj: complex elements are conjugated as they are loaded (op(B) = C).
template <typename TIn, bool VEC, int NDIG, int NMU, int MODE>
__global__ void __launch_bounds__(256, 4)
    oz_slice_mn(const TIn* __restrict__ X, int64_t ld, int m, int64_t k, int64_t kp,
                const int* __restrict__ sigma, int s_sum, int conj, int8_t* __restrict__ res,
                ResidueLayout lay, int64_t res_mod_stride, SliceConsts sc) {
  constexpr int EL = 8;
  constexpr int R = MODE != 0 ? 2 : 1;  // reals per element
  constexpr int G = EL / R;             // elements per thread
  constexpr int KT = 32 * G;            // elements per row per tile
  constexpr int ESZ = R * int(sizeof(TIn));
  constexpr int GROUPS = 128 / ESZ;     // elements per 128 bytes of shared memory
  constexpr int RSTR = KT + 1;          // row stride in elements (odd)
  using T = typename RawElem<ESZ>::T;
  __shared__ T tile[8 * RSTR];
  auto swz = [](int kk) { return kk ^ ((kk / G) & (GROUPS - 1)); };
  const int i0 = blockIdx.x * 8;
  const int64_t kk0 = int64_t(blockIdx.y) * KT;
#pragma unroll
  for (int it = 0; it < KT / 32; ++it) {
    const int r = threadIdx.x & 7, kk = (threadIdx.x >> 3) + 32 * it;
    T val;
    if (i0 + r < m && kk0 + kk < k) {
      const int64_t e = int64_t(i0 + r) + (kk0 + kk) * ld;  // element index
      if constexpr (ESZ == 16) {
        if (VEC) {
          val = __ldg(reinterpret_cast<const double2*>(X) + e);
        } else {
          val.x = double(X[2 * e]);
          val.y = double(X[2 * e + 1]);
        }
      } else if constexpr (ESZ == 8 && sizeof(TIn) == 8) {
        val = __double_as_longlong(double(X[e]));
      } else if constexpr (ESZ == 8) {  // complex float
        val = (static_cast<unsigned long long>(__float_as_uint(float(X[2 * e + 1]))) << 32) |
              __float_as_uint(float(X[2 * e]));
      } else {
        val = __float_as_uint(float(X[e]));
      }
    } else {
      if constexpr (ESZ == 16)
        val = make_double2(0.0, 0.0);
      else
        val = 0;
    }
    tile[r * RSTR + swz(kk)] = val;
  }
  __syncthreads();
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int row = i0 + w;
  if (row >= m || kk0 + G * l >= kp) return;
  using V = SliceReal<TIn, NDIG>;
  V v[EL];
#pragma unroll
  for (int q = 0; q < G; ++q) {
    const T e = tile[w * RSTR + swz(G * l + q)];
    if constexpr (ESZ == 16) {
      v[2 * q] = e.x;
      v[2 * q + 1] = conj ? -e.y : e.y;
    } else if constexpr (ESZ == 8 && sizeof(TIn) == 8) {
      v[q] = __longlong_as_double(static_cast<long long>(e));
    } else if constexpr (ESZ == 8) {
      v[2 * q] = V(__uint_as_float(unsigned(e)));
      const V im = V(__uint_as_float(unsigned(e >> 32)));
      v[2 * q + 1] = conj ? -im : im;
    } else {
      v[q] = V(__uint_as_float(e));
    }
  }
  const int64_t l0 = (kk0 + G * l) * R;
  slice_thread<TIn, NDIG, EL, NMU, MODE>(v, sigma[row], row_base<MODE>(res, lay, row, l0), l0,
                                         lay.plane(1), s_sum, res_mod_stride, sc);
}

// --------------------------------------------------------------------------
// 3. INT8 residue GEMM on tcgen05

struct GemmParams {
  int m;             // rows of A per product plane
  int nb;            // rows of B per product plane
  int kblocks;       // kp / 128
  int nchunks;       // k-chunks (choose_gemm)
  int chunk_blocks;  // k-blocks per chunk: ceil(kblocks / nchunks), within the INT32 bound
  int group;         // planes per group, and k-blocks per piece of a plane's row
  int kc_blocks;     // (ResidueLayout: G, kc / 128)
  int nmod;          // products: moduli x nsub (the A/B/R planes in order)
  int nsub;          // products per modulus (Layout::nsub): modulus = product / nsub
  int tiles_m, tiles_n;
  int total_units;   // products * nchunks * tiles
  int* R;            // accumulated residues [product][nb][m] (int32), or
  unsigned char* R8; // bytes [chunk][product][nb][ldr], one plane per k-chunk
  int ldr;           // elements between the columns of a plane, and between planes
  int64_t rplane;
  int* status;       // set to 1 when a bounded wait gave up
  const int* active; // CTA-pair kernel: list of tiles to compute (fill mode), or null = all
  int n_active;
  unsigned long long wait_limit_ns;  // bound on every barrier wait
  int stall_test;    // 1: the producer issues no copies (exercises the bounded waits)
  int p[kMaxModuli];
  int c16[kMaxModuli], off[kMaxModuli];  // division-free v mod p (mod_residue)
  unsigned M[kMaxModuli];
  int epi_split;     // CTA-pair kernel: epilogue warps per TMEM lane quarter (1 or 2)
};

struct Unit {
  int t, c, tm, tn;
};


// Tile raster within one (product, k-chunk): bands of kBandTiles row tiles,
// row tiles fastest within a band. The units in flight at one time cover a
// few row tiles of A and a few column tiles of B, so that each A tile is
// read from DRAM once even when A is much taller than L2 holds (a plain
// row-fastest order re-reads all of A once per column tile).
constexpr int kBandTiles = 8;
__host__ __device__ __forceinline__ void band_tile(int tile, int tiles_m, int tiles_n, int& tm,
                                                   int& tn) {
  const int band_units = kBandTiles * tiles_n;
  const int band = tile / band_units, r = tile - band * band_units;
  const int left = tiles_m - band * kBandTiles;
  const int rows = left < kBandTiles ? left : kBandTiles;
  tm = band * kBandTiles + r % rows;
  tn = r / rows;
}

__device__ __forceinline__ Unit decode_unit(int u, const GemmParams& g) {
  Unit r;
  const int tiles = g.tiles_m * g.tiles_n;
  const int tile = u % tiles;
  const int rest = u / tiles;
  band_tile(tile, g.tiles_m, g.tiles_n, r.tm, r.tn);
  r.c = rest % g.nchunks;
  r.t = rest / g.nchunks;
  return r;
}

__global__ void __launch_bounds__(GEMM_THREADS, 1)
    oz_gemm(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
            const __grid_constant__ GemmParams g) {
  extern __shared__ unsigned char smem_raw[];
  // 1024-byte aligned base for the 128-byte swizzle atoms
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  unsigned char* base_ptr = smem_raw + (base - raw_addr);
  const uint32_t bar_base = base + STAGES * STAGE_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto accf_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + b); };
  auto acce_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + 2 + b); };
  const uint32_t drain_bar = bar_base + 8u * (2 * STAGES + 4);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base_ptr + STAGES * STAGE_BYTES + 256);
  volatile int* abort = reinterpret_cast<volatile int*>(base_ptr + STAGES * STAGE_BYTES + 264);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(accf_bar(b), 1);
      mbar_init(acce_bar(b), 128);
    }
    mbar_init(drain_bar, 1);
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0 && lane == 0) {
    // ---- TMA producer
    int stage = 0;
    uint32_t phase = 0;
    bool ok = g.stall_test == 0;
    for (int u = blockIdx.x; u < g.total_units && ok; u += gridDim.x) {
      const Unit w = decode_unit(u, g);
      const int kb0 = w.c * g.chunk_blocks;
      const int kb1 = min(g.kblocks, kb0 + g.chunk_blocks);
      const int tg = w.t / g.group, tq = w.t - tg * g.group;  // the plane's group, place in it
      int kc = kb0 / g.kc_blocks, kx = kb0 - kc * g.kc_blocks;  // piece, block in it
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort, g.wait_limit_ns)) {
          ok = false;
          break;
        }
        mbar_arrive_expect_tx(full_bar(stage), STAGE_BYTES);
        const uint32_t sa = base + stage * STAGE_BYTES;
        tma_load_5d(sa, &tmA, kx * BKB, tq, kc, w.tm * BM, tg, full_bar(stage));
        tma_load_5d(sa + A_STAGE, &tmB, kx * BKB, tq, kc, w.tn * BN, tg, full_bar(stage));
        if (++kx == g.kc_blocks) {
          kx = 0;
          ++kc;
        }
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (!ok && g.stall_test == 0) {
      // let the copies already issued land before the shared memory goes away
      for (int s = 0; s < STAGES; ++s) {
        const unsigned long long t0 = globaltimer();
        while (!mbar_try_wait(full_bar(s), 0) && !mbar_try_wait(full_bar(s), 1) &&
               globaltimer() - t0 < 1000000ull) {
        }
      }
    }
  } else if (warp == 1 && lane == 0) {
    // ---- MMA issuer
    int stage = 0;
    uint32_t phase = 0;
    uint32_t acc_phase[2] = {0, 0};
    int accb = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < g.total_units && ok; u += gridDim.x) {
      const Unit w = decode_unit(u, g);
      const int kb0 = w.c * g.chunk_blocks;
      const int kb1 = min(g.kblocks, kb0 + g.chunk_blocks);
      if (!mbar_wait(acce_bar(accb), acc_phase[accb] ^ 1u, abort, g.wait_limit_ns)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t d = tmem_base + uint32_t(accb * BN);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(full_bar(stage), phase, abort, g.wait_limit_ns)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sa = base + stage * STAGE_BYTES;
#pragma unroll
        for (int kk = 0; kk < BKB / 32; ++kk) {
          const uint64_t ad = umma_desc_sw128(sa + kk * 32);
          const uint64_t bd = umma_desc_sw128(sa + A_STAGE + kk * 32);
          umma_i8(d, ad, bd, (kb > kb0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(empty_bar(stage));
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (!ok) break;
      umma_commit(accf_bar(accb));
      acc_phase[accb] ^= 1u;
      accb ^= 1;
    }
    if (!ok) {
      // MMAs may still be in flight: wait (bounded) until they retire
      umma_commit(drain_bar);
      const unsigned long long t0 = globaltimer();
      while (!mbar_try_wait(drain_bar, 0) && globaltimer() - t0 < 1000000ull) {
      }
    }
  } else if (warp >= 2) {
    // ---- epilogue: TMEM -> registers -> mod p -> accumulate into R
    const int quarter = warp & 3;  // TMEM lanes 32*quarter .. +31
    const int row = quarter * 32 + lane;
    uint32_t acc_phase[2] = {0, 0};
    int accb = 0;
    for (int u = blockIdx.x; u < g.total_units; u += gridDim.x) {
      const Unit w = decode_unit(u, g);
      // warp-uniform: the TMEM loads below are collective
      if (!__all_sync(0xffffffffu,
                      mbar_wait(accf_bar(accb), acc_phase[accb], abort, g.wait_limit_ns)))
        break;
      tc_fence_after();
      const int mt = w.t / g.nsub;  // modulus of this product
      const int p = g.p[mt], c16 = g.c16[mt], off = g.off[mt];
      const unsigned M = g.M[mt];
      const int i = w.tm * BM + row;
      const int j0 = w.tn * BN;
      int* Rt = g.R + w.t * g.rplane;
      unsigned char* R8t = g.R8 + (int64_t(w.c) * g.nmod + w.t) * g.rplane;
      for (int c0 = 0; c0 < BN; c0 += 32) {
        uint32_t v[32];
        tmem_ld32(tmem_base + (uint32_t(quarter * 32) << 16) + uint32_t(accb * BN + c0), v);
        if (i < g.m) {
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            const int j = j0 + c0 + c;
            if (j < g.nb) {
              const int r = mod_residue(int(v[c]), p, c16, off, M);
              if (g.R8)
                R8t[int64_t(j) * g.ldr + i] = (unsigned char)r;
              else
                atomicAdd(Rt + int64_t(j) * g.ldr + i, r);
            }
          }
        }
      }
      tc_fence_before();
      mbar_arrive(acce_bar(accb));
      acc_phase[accb] ^= 1u;
      accb ^= 1;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort && threadIdx.x == 0) atomicExch(g.status, 1);
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base)
                 : "memory");
  }
}

// --------------------------------------------------------------------------
// 3b. the same GEMM on CTA pairs (tcgen05 cta_group::2)
//
// A cluster of two CTAs computes a 256 x 256 tile: each CTA stages 128 rows of
// A and 128 rows of B per k-block (TMA, no multicast), the even CTA issues
// tcgen05.mma.cta_group::2 (M = 256, N = 256, K = 32) reading both CTAs'
// shared memory, and each CTA's TMEM receives its 128 rows of the tile. Per
// SM this halves the shared-memory operand traffic of the 1-CTA form and
// runs the tensor pipe at its full int8 rate.
//   full[s]  (even CTA): TMA bytes of both CTAs + the even producer's arrival
//   empty[s] (both):     commit of the MMAs, multicast to the pair
//   accf[b]  (both):     commit after a tile's last k-block, multicast
//   acce[b]  (even CTA): 256 epilogue threads of both CTAs, remote arrivals
// NT = 1: pair tile 256 x 256, two accumulator buffers (2 x 256 TMEM
// columns), 6 stages. NT = 2: pair tile 256 x 512 (two MMAs of N = 256 per
// k-step on one A tile: a quarter less L2 -> SMEM traffic per operation), one
// accumulator buffer of 512 columns (drained once per unit), 4 stages.
constexpr int A_STAGE2 = 128 * BKB;  // 16 KiB per CTA
constexpr int B_HALF2 = 128 * BKB;   // 16 KiB per CTA and N = 256 half
template <int NT>
struct PairCfg {
  static constexpr int STAGES = NT == 1 ? 6 : 4;
  static constexpr int STAGE = A_STAGE2 + NT * B_HALF2;
  static constexpr int SMEM = STAGES * STAGE + 1024 + 1024;
  static constexpr int NBUF = NT == 1 ? 2 : 1;
};
constexpr uint32_t kIdescI8Pair = (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(256 >> 3) << 17) |
                                  (uint32_t(256 >> 4) << 24);

__device__ __forceinline__ void umma_i8_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(kIdescI8Pair), "r"(accumulate)
      : "memory");
}
// warp 0: TMA, warp 1: MMA, warps 2-9: epilogue. With g.epi_split = 2 two
// warps per TMEM lane quarter each drain half of the tile's columns: the
// per-value reduction is issue-bound, and one warp per scheduler made it the
// bottleneck when the units are short in k. With long units (the drain hides
// behind the next unit's MMAs) warps 2-5 drain alone and warps 6-9 idle.
constexpr int PAIR_THREADS = 320;
template <int NT>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
    oz_gemm_pair(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ GemmParams g) {
  using P = PairCfg<NT>;
  constexpr int STAGES2 = P::STAGES;
  constexpr int STAGE2_BYTES = P::STAGE;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  unsigned char* base_ptr = smem_raw + (base - raw_addr);
  const uint32_t bar_base = base + STAGES2 * STAGE2_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES2 + s); };
  auto accf_bar = [&](int b) { return bar_base + 8u * (2 * STAGES2 + b); };
  auto acce_bar = [&](int b) { return bar_base + 8u * (2 * STAGES2 + 2 + b); };
  const uint32_t drain_bar = bar_base + 8u * (2 * STAGES2 + 4);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base_ptr + STAGES2 * STAGE2_BYTES + 256);
  volatile int* abort = reinterpret_cast<volatile int*>(base_ptr + STAGES2 * STAGE2_BYTES + 264);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();  // 0: issues the MMAs
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int tiles = g.tiles_m * g.tiles_n;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES2; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(accf_bar(b), 1);
      mbar_init(acce_bar(b), 2 * 4 * g.epi_split);  // one arrival per epilogue warp of the pair
    }
    mbar_init(drain_bar, 1);
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int ntl = g.active ? g.n_active : tiles;
  auto unit_of = [&](int u, int& t, int& c, int& tm, int& tn) {
    const int tl = u % ntl, rest = u / ntl;
    if (g.active) {  // explicit list: tm + tn * tiles_m
      const int tile = g.active[tl];
      tm = tile % g.tiles_m;
      tn = tile / g.tiles_m;
    } else {
      band_tile(tl, g.tiles_m, g.tiles_n, tm, tn);
    }
    c = rest % g.nchunks;
    t = rest / g.nchunks;
  };

  bool aborted = false;
  if (warp == 0 && lane == 0) {
    // ---- TMA producer (both CTAs): 128 rows of A and of B per k-block
    int stage = 0;
    uint32_t phase = 0;
    bool ok = g.stall_test == 0;
    for (int u = pair; u < g.total_units && ok; u += npairs) {
      int t, c, tm, tn;
      unit_of(u, t, c, tm, tn);
      const int kb0 = c * g.chunk_blocks, kb1 = min(g.kblocks, kb0 + g.chunk_blocks);
      const int arow = tm * 256 + int(rank) * 128;
      const int brow = tn * (256 * NT) + int(rank) * 128;
      const int tg = t / g.group, tq = t - tg * g.group;  // the plane's group, place in it
      int kc = kb0 / g.kc_blocks, kx = kb0 - kc * g.kc_blocks;  // piece, block in it
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort, g.wait_limit_ns)) {
          ok = false;
          break;
        }
        const uint32_t fb = map_to_rank(full_bar(stage), 0);
        if (rank == 0) mbar_arrive_expect_tx(full_bar(stage), 2 * STAGE2_BYTES);
        const uint32_t sa = base + stage * STAGE2_BYTES;
        tma_load_5d_pair(sa, &tmA, kx * BKB, tq, kc, arow, tg, fb);
#pragma unroll
        for (int h = 0; h < NT; ++h)
          tma_load_5d_pair(sa + A_STAGE2 + h * B_HALF2, &tmB, kx * BKB, tq, kc, brow + h * 256, tg,
                           fb);
        if (++kx == g.kc_blocks) {
          kx = 0;
          ++kc;
        }
        if (++stage == STAGES2) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    aborted = !ok && g.stall_test == 0;
  } else if (warp == 1 && lane == 0 && rank == 0) {
    // ---- MMA issuer (even CTA)
    int stage = 0;
    uint32_t phase = 0;
    uint32_t acc_phase[2] = {0, 0};
    int accb = 0;
    bool ok = true;
    for (int u = pair; u < g.total_units && ok; u += npairs) {
      int t, c, tm, tn;
      unit_of(u, t, c, tm, tn);
      const int kb0 = c * g.chunk_blocks, kb1 = min(g.kblocks, kb0 + g.chunk_blocks);
      if (!mbar_wait(acce_bar(accb), acc_phase[accb] ^ 1u, abort, g.wait_limit_ns)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t d = tmem_base + uint32_t(accb * 256);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(full_bar(stage), phase, abort, g.wait_limit_ns)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sa = base + stage * STAGE2_BYTES;
#pragma unroll
        for (int kk = 0; kk < BKB / 32; ++kk) {
          const uint64_t adesc = umma_desc_sw128(sa + kk * 32);
#pragma unroll
          for (int h = 0; h < NT; ++h)
            umma_i8_pair(d + uint32_t(h * 256),
                         adesc, umma_desc_sw128(sa + A_STAGE2 + h * B_HALF2 + kk * 32),
                         (kb > kb0 || kk > 0) ? 1u : 0u);
        }
        umma_commit_pair(empty_bar(stage));
        if (++stage == STAGES2) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (!ok) break;
      umma_commit_pair(accf_bar(accb));
      acc_phase[accb] ^= 1u;
      accb = (accb + 1) % P::NBUF;
    }
    if (!ok) {
      asm volatile(
          "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
              drain_bar)
          : "memory");
      const unsigned long long t0 = globaltimer();
      while (!mbar_try_wait(drain_bar, 0) && globaltimer() - t0 < 1000000ull) {
      }
    }
  } else if (warp >= 2 && ((warp - 2) >> 2) < g.epi_split) {
    // ---- epilogue (both CTAs): own TMEM rows -> mod p -> R
    const int quarter = warp & 3;        // TMEM lanes 32*quarter .. +31
    const int half = (warp - 2) >> 2;    // columns half*kCols .. +kCols-1
    const int kCols = 256 * NT / g.epi_split;
    const int row = int(rank) * 128 + quarter * 32 + lane;
    uint32_t acc_phase[2] = {0, 0};
    int accb = 0;
    for (int u = pair; u < g.total_units; u += npairs) {
      int t, c, tm, tn;
      unit_of(u, t, c, tm, tn);
      // warp-uniform: the TMEM loads and the warp's arrival below are collective
      if (!__all_sync(0xffffffffu,
                      mbar_wait(accf_bar(accb), acc_phase[accb], abort, g.wait_limit_ns)))
        break;
      tc_fence_after();
      const int mt = t / g.nsub;  // modulus of this product
      const int p = g.p[mt], c16 = g.c16[mt], off = g.off[mt];
      const unsigned M = g.M[mt];
      const int i = tm * 256 + row;
      const int jw = tn * (256 * NT) + half * kCols;
      const int64_t plane = (g.R8 ? c * g.nmod + t : t) * g.rplane;
      for (int c0 = 0; c0 < kCols; c0 += 32) {
        uint32_t v[32];
        tmem_ld32(tmem_base + (uint32_t(quarter * 32) << 16) +
                      uint32_t(accb * 256 + half * kCols + c0),
                  v);
        const int jb = jw + c0;
        if (i < g.m && jb < g.nb) {
          const int64_t base = plane + int64_t(jb) * g.ldr + i;
          if (jb + 32 <= g.nb) {  // whole group of columns: no per-column test
            if (g.R8) {
              unsigned char* d = g.R8 + base;
#pragma unroll
              for (int cc = 0; cc < 32; ++cc)
                d[int64_t(cc) * g.ldr] = (unsigned char)mod_residue(int(v[cc]), p, c16, off, M);
            } else {
              int* d = g.R + base;
#pragma unroll
              for (int cc = 0; cc < 32; ++cc)
                atomicAdd(d + int64_t(cc) * g.ldr, mod_residue(int(v[cc]), p, c16, off, M));
            }
          } else {
#pragma unroll
            for (int cc = 0; cc < 32; ++cc) {
              if (jb + cc < g.nb) {
                const int r = mod_residue(int(v[cc]), p, c16, off, M);
                if (g.R8)
                  g.R8[base + int64_t(cc) * g.ldr] = (unsigned char)r;
                else
                  atomicAdd(g.R + base + int64_t(cc) * g.ldr, r);
              }
            }
          }
        }
      }
      // the accumulator is drained: one arrival per warp with the default
      // (CTA-scope) semantics on the MMA issuer's barrier; the ordering of the
      // TMEM loads before the next MMAs comes from the tcgen05 fences around
      // the barrier (a cluster-scope release per thread cost membar stalls)
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(map_to_rank(acce_bar(accb), 0));
      acc_phase[accb] ^= 1u;
      accb = (accb + 1) % P::NBUF;
    }
  }

  if (aborted) {
    // copies issued by this CTA may still be landing in shared memory
    const unsigned long long t0 = globaltimer();
    while (globaltimer() - t0 < 2000000ull) {
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort && threadIdx.x == 0) atomicExch(g.status, 1);
  cluster_sync_all();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base)
                 : "memory");
  }
}

// --------------------------------------------------------------------------
// 4. reconstruction

constexpr long long kNaNBits = 0x7FF8000000000000ll;  // quiet NaN

// x * 2^e, correctly rounded: a multiplication by the power of two when the
// result stays normal (|x| is an integer below 2^128 or zero), ldexp otherwise.
__device__ __forceinline__ double scale_pow2(double x, int e) {
  if (e >= -1022 && e <= 895)
    return x * __longlong_as_double((long long)(e + 1023) << 52);
  return ldexp(x, e);
}

// C(i, j) <- alpha * x + beta * C(i, j) (x = xr + i xi for complex types)
template <int DT>
__device__ __forceinline__ void store_c(void* C, int64_t ci, double xr, double xi, double alr,
                                        double ali, double ber, double bei, bool read_c) {
  double outr = alr * xr - ali * xi, outi = alr * xi + ali * xr;
  if constexpr (DT == kC64) {
    double2* c = static_cast<double2*>(C) + ci;
    if (read_c) {
      const double2 old = *c;
      outr += ber * old.x - bei * old.y;
      outi += ber * old.y + bei * old.x;
    }
    *c = make_double2(outr, outi);
  } else if constexpr (DT == kC32) {
    float2* c = static_cast<float2*>(C) + ci;
    if (read_c) {
      const float2 old = *c;
      outr += ber * double(old.x) - bei * double(old.y);
      outi += ber * double(old.y) + bei * double(old.x);
    }
    *c = make_float2(float(outr), float(outi));
  } else if constexpr (DT == kR64) {
    double* c = static_cast<double*>(C) + ci;
    *c = read_c ? fma(ber, *c, outr) : outr;
  } else {
    float* c = static_cast<float*>(C) + ci;
    *c = float(read_c ? fma(ber, double(*c), outr) : outr);
  }
}

// Residues of element (i, j) of the real result (real types) or of Re and Im
// (complex: two product planes per modulus combined by combine_split, or three
// by combine3), for modulus t, summed over the k-chunks. src points at plane 0 of
// modulus t, element (i, j); planes of one product are `plane`, those of one
// k-chunk `chunk` elements apart. off: a multiple of p not below any sum.
template <bool CPLX, bool SPLIT, typename RT>
__device__ __forceinline__ void product_residues(const RT* src, int64_t plane, int chunks,
                                                 int64_t chunk, int off, int conj, int& re,
                                                 int& im) {
  int r[3] = {int(src[0]), CPLX ? int(src[plane]) : 0, CPLX && !SPLIT ? int(src[2 * plane]) : 0};
  if (sizeof(RT) == 1) {  // int32: already summed
    for (int c = 1; c < chunks; ++c) {
      src += chunk;
      r[0] += int(src[0]);
      if (CPLX) r[1] += int(src[plane]);
      if (CPLX && !SPLIT) r[2] += int(src[2 * plane]);
    }
  }
  if (SPLIT) {
    combine_split(r[0], r[1], off, re, im);
  } else if (CPLX) {
    combine3(r[0], r[1], r[2], off, conj, re, im);
  } else {
    re = r[0];
    im = 0;
  }
}

// C(i, j) <- alpha * 2^(-sigma_i - tau_j) * X + beta * C(i, j), X the CRT
// value of the product (complex: of Re and Im). R holds, per product plane,
// int32 sums of per-chunk residues or, per k-chunk and product plane, the
// residues as bytes (RT), columns ldr elements apart. Threads run along i (contiguous in R and C), blocks along j: no
// index division. NM: the number of moduli when fixed at compile time (the
// defaults; the complex ones are the split moduli), 0 for rp.n.
template <int DT, typename RT, int NM>
__global__ void __launch_bounds__(256, 2) oz_reconstruct(const RT* __restrict__ R, int m, int n,
                                                         int64_t plane, int64_t ldr, int chunks,
                                                         const int* __restrict__ sigA,
                                                         const int* __restrict__ sigB, void* C,
                                                         int64_t ldc, double alr, double ali,
                                                         double ber, double bei, int fill,
                                                         int64_t ro, int64_t co, int tile_m,
                                                         int tile_n, ReconParams rp) {
  constexpr bool CPLX = dtype_is_complex(DT);
  constexpr bool SPLIT = CPLX && NM > 0;
  constexpr int NSUB = SPLIT ? 2 : CPLX ? 3 : 1;
  constexpr int NMAX = NM > 0 ? NM : kMaxUsableModuli;
  const int nmod = NM > 0 ? NM : rp.n;
  const bool read_c = (ber != 0.0 || bei != 0.0);
  for (int j = blockIdx.y; j < n; j += gridDim.y) {
    const int tauj = sigB[j];
    const int64_t tj = (j / tile_n) * int64_t(tile_n);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
      if (fill != 0) {
        const int64_t ti = (i / tile_m) * int64_t(tile_m);
        if (!tile_is_active(fill, ti, tj, ::min((int64_t)tile_m, (int64_t)m - ti),
                            ::min((int64_t)tile_n, (int64_t)n - tj), ro, co))
          continue;
      }
      int rr[NMAX], ri[NMAX];
      const RT* src = R + int64_t(j) * ldr + i;
#pragma unroll
      for (int t = 0; t < NMAX; ++t)
        if (t < nmod)
          product_residues<CPLX, SPLIT>(src + t * NSUB * plane, plane, chunks,
                                        NSUB * nmod * plane, rp.off24[t], rp.conj, rr[t], ri[t]);
      const int si = sigA[i];
      const int e = -(si + tauj);
      double xr = scale_pow2(crt_value<NM, false>(rr, rp), e);
      double xi = CPLX ? scale_pow2(crt_value<NM, false, SPLIT>(ri, rp), e) : 0.0;
      if (si == kSigmaNonFinite || tauj == kSigmaNonFinite) xr = xi = __longlong_as_double(kNaNBits);
      store_c<DT>(C, i + int64_t(j) * ldc, xr, xi, alr, ali, ber, bei, read_c);
    }
  }
}

// At(kk, i) <- A(i, kk): op(A) = N operands (A stored m-major) are copied
// k-major so that the row norms and the slicing read them like op(A) = T.
// 32 x 32 tiles through shared memory: reads run along i, writes along kk.
template <typename E>
__global__ void oz_transpose(const E* __restrict__ A, int64_t lda, int m, int64_t k,
                             E* __restrict__ At, int64_t ldat) {
  __shared__ E tile[32][33];
  const int i0 = blockIdx.x * 32;
  for (int64_t k0 = int64_t(blockIdx.y) * 32; k0 < k; k0 += int64_t(gridDim.y) * 32) {
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
      const int i = i0 + threadIdx.x;
      const int64_t kk = k0 + r;
      if (i < m && kk < k) tile[r][threadIdx.x] = A[i + kk * lda];
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
      const int i = i0 + r;
      const int64_t kk = k0 + threadIdx.x;
      if (i < m && kk < k) At[int64_t(i) * ldat + kk] = tile[threadIdx.x][r];
    }
    __syncthreads();
  }
}

// --------------------------------------------------------------------------
// 4b. CRT reconstruction on the tensor cores (byte residues)
//
// By linearity the CRT sum needs no reduction of the product combination:
// with V_k the weight of product plane k, W_t (or the Im weight of a split
// modulus) for the plane's modulus t where the product enters Re or Im with a
// plus sign and P - W_t where it enters with a minus (see combine_split and
// combine3; p_t W_t = 0 mod P), S = sum_k r_k V_k is congruent mod P to the sum
// the CUDA-core kernels form. Written in the bytes of V_k, S = sum_j 256^j S_j with
// S_j = sum_k r_k byte_j(V_k), and for 128 consecutive rows of one column of
// C one tcgen05.mma kind::i8 (unsigned bytes, exact INT32 sums below 2^22)
//   D[128 x NO] = R[128 x KP] . V[KP x NO]
// forms all of them: R is the tile's residue bytes as TMA loads them (one
// 128-byte row per product plane: the MN-major operand layout), V the
// weight bytes (K-major, columns 0-15 for Re, 16-31 for Im). The epilogue
// (one TMEM lane per row of C) combines its 16 sums per part into the four
// 32-bit limb sums of S and finishes with crt_from_limbs, as the CUDA-core
// kernels do: the results are the same doubles.
//
// A work unit is RT_G blocks of 128 rows of one column (the fixed cost of the
// hand-offs below is paid once per unit). Warp 0: TMA producer (4-stage
// ring), warp 1: TMEM allocation and MMA issue (accumulators double-buffered),
// warps 2-5: epilogue (RT_G rows per lane). Every wait is bounded; a give-up
// sets *status.
constexpr int RT_THREADS = 192;
constexpr int RT_STAGES = 4;
constexpr int RT_G = 2;                       // blocks of 128 rows per work unit
constexpr int RT_KP = 64;                     // most planes (K)
constexpr int RT_W_BYTES = 32 * 128;          // weights: 32 rows x 128 B (SW128)
// KP planes per block, padded: 32 or 64. CTAs per SM, within its shared memory and
// its 512 TMEM columns (2 x RT_G x 32 each).
template <int KP>
struct ReconCfg {
  static constexpr int BLOCK = 128 * KP;      // bytes per block of 128 rows
  static constexpr int STAGE = RT_G * BLOCK;  // bytes per stage
  static constexpr int SMEM = RT_STAGES * STAGE + RT_W_BYTES + 256 + 1024;
  static constexpr int CTAS = KP == 32 ? 4 : 3;
  static_assert(CTAS * (SMEM + 1024) <= 228 * 1024 && CTAS * 2 * RT_G * 32 <= 512, "fits an SM");
};

struct ReconTcParams {
  int m, n;
  int row_blocks;         // groups of RT_G blocks of 128 rows: ceil(m / (128 RT_G))
  long long total_units;  // row_blocks * n
  int planes;             // product planes of the residue array (loaded per tile)
  const int* sigA;
  const int* sigB;
  void* C;
  int64_t ldc;
  double alr, ali, ber, bei;
  int fill;
  int64_t ro, co;
  int tile_m, tile_n;
  ReconParams rp;
  unsigned char v[32][RT_KP];  // weight bytes: v[o][k] = byte (o % 16) of V_k for part o / 16
  int* status;
  unsigned long long wait_limit_ns;
};

// UMMA shared-memory descriptor of an MN-major operand in the 128-byte
// swizzle layout: 8-row atoms of 128 bytes along M (one atom covers the 128
// rows of the tile), atoms 1024 B apart along K.
__device__ __forceinline__ uint64_t umma_desc_sw128_mn(uint32_t saddr) {
  uint64_t d = 0;
  d |= uint64_t((saddr >> 4) & 0x3FFFu);  // start address
  d |= uint64_t(1) << 16;                  // leading byte offset (one atom along M: unused)
  d |= uint64_t(1024 >> 4) << 32;          // stride byte offset: 8 K-rows x 128 B
  d |= uint64_t(1) << 46;                  // descriptor version (sm_100)
  d |= uint64_t(2) << 61;                  // layout: 128-byte swizzle
  return d;
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y,
                                            int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

template <int DT, int KP>
__global__ void __launch_bounds__(RT_THREADS, ReconCfg<KP>::CTAS)
    oz_reconstruct_tc(const __grid_constant__ CUtensorMap tmR,
                      const __grid_constant__ ReconTcParams P) {
  constexpr bool CPLX = dtype_is_complex(DT);
  constexpr int RT_BLOCK = ReconCfg<KP>::BLOCK, RT_STAGE = ReconCfg<KP>::STAGE;
  constexpr int NO = CPLX ? 32 : 16;  // output columns of the MMA
  // D S32, A and B unsigned int8, A MN-major, B K-major, N = NO, M = 128
  constexpr uint32_t kIdesc = (2u << 4) | (1u << 15) | (uint32_t(NO >> 3) << 17) |
                              (uint32_t(128 >> 4) << 24);
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  unsigned char* base_ptr = smem_raw + (base - raw_addr);
  const uint32_t w_addr = base + RT_STAGES * RT_STAGE;
  const uint32_t bar_base = w_addr + RT_W_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (RT_STAGES + s); };
  auto accf_bar = [&](int b) { return bar_base + 8u * (2 * RT_STAGES + b); };
  auto acce_bar = [&](int b) { return bar_base + 8u * (2 * RT_STAGES + 2 + b); };
  const uint32_t drain_bar = bar_base + 8u * (2 * RT_STAGES + 4);
  unsigned char* ctl = base_ptr + RT_STAGES * RT_STAGE + RT_W_BYTES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ctl + 8 * (2 * RT_STAGES + 5));
  volatile int* abort = reinterpret_cast<volatile int*>(ctl + 8 * (2 * RT_STAGES + 5) + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // weight bytes into the K-major 128-byte-swizzled B tile (row o, K byte k),
  // and zeros into the plane rows planes .. kp-1 of every stage (TMA writes
  // rows 0 .. planes-1 only)
  {
    unsigned char* wp = base_ptr + RT_STAGES * RT_STAGE;
    for (int idx = threadIdx.x; idx < RT_W_BYTES; idx += RT_THREADS) {
      const int o = idx >> 7, k = idx & 127;
      const unsigned char b = (o < NO && k < KP) ? P.v[o][k] : 0;
      wp[(o >> 3) * 1024 + (o & 7) * 128 + (((k >> 4) ^ (o & 7)) << 4) + (k & 15)] = b;
    }
    const int pad = (KP - P.planes) * 128;  // bytes per block, 16-byte words below
    for (int idx = threadIdx.x; idx < RT_STAGES * RT_G * (pad / 16); idx += RT_THREADS) {
      const int blk = idx / (pad / 16), w16 = idx - blk * (pad / 16);  // blk: stage, block
      *reinterpret_cast<uint4*>(base_ptr + blk * RT_BLOCK + P.planes * 128 + 16 * w16) =
          make_uint4(0u, 0u, 0u, 0u);
    }
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < RT_STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(accf_bar(b), 1);
      mbar_init(acce_bar(b), 4);
    }
    mbar_init(drain_bar, 1);
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // the tensor cores read the weights through the async proxy
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)), "n"(2 * RT_G * 32)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tile_bytes = uint32_t(RT_G * 128 * P.planes);
  bool copies_pending = false;  // the producer gave up with copies possibly in flight

  // unit u = (row block rb, column j), u = rb + j row_blocks: every role walks
  // u = blockIdx.x, + gridDim.x, ... with (rb, j) advanced without division
  const int drb = int(gridDim.x % unsigned(P.row_blocks));
  const int dj = int(gridDim.x / unsigned(P.row_blocks));
  auto next_unit = [&](int& rb, int& j) {
    rb += drb;
    j += dj;
    if (rb >= P.row_blocks) {
      rb -= P.row_blocks;
      ++j;
    }
  };
  const int rb0 = int(blockIdx.x % unsigned(P.row_blocks));
  const int j0 = int(blockIdx.x / unsigned(P.row_blocks));

  if (warp == 0 && lane == 0) {
    // ---- TMA producer: the tile's planes, 128 residue bytes each
    int rb = rb0, j = j0;
    for (long long u = blockIdx.x, it = 0; u < P.total_units;
         u += gridDim.x, ++it, next_unit(rb, j)) {
      const int stage = int(it % RT_STAGES);
      const uint32_t phase = uint32_t((it / RT_STAGES) & 1);
      if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort, P.wait_limit_ns)) {
        copies_pending = true;
        break;
      }
      mbar_arrive_expect_tx(full_bar(stage), tile_bytes);
      // the last group's blocks past m read as zeros (their rows are not stored)
#pragma unroll
      for (int g = 0; g < RT_G; ++g)
        tma_load_3d(base + stage * RT_STAGE + g * RT_BLOCK, &tmR, (rb * RT_G + g) * 128, j, 0,
                    full_bar(stage));
    }
  } else if (warp == 1 && lane == 0) {
    // ---- MMA issuer
    bool ok = true;
    for (long long u = blockIdx.x, it = 0; u < P.total_units; u += gridDim.x, ++it) {
      const int stage = int(it % RT_STAGES);
      const uint32_t phase = uint32_t((it / RT_STAGES) & 1);
      const int b = int(it & 1);
      const uint32_t bpar = uint32_t((it >> 1) & 1);
      if (!mbar_wait(acce_bar(b), bpar ^ 1u, abort, P.wait_limit_ns) ||
          !mbar_wait(full_bar(stage), phase, abort, P.wait_limit_ns)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t sa = base + stage * RT_STAGE;
#pragma unroll
      for (int g = 0; g < RT_G; ++g)
        for (int kb = 0; kb < KP / 32; ++kb)
          umma_i8_desc(tmem_base + uint32_t((b * RT_G + g) * 32),
                       umma_desc_sw128_mn(sa + g * RT_BLOCK + kb * 4096),
                       umma_desc_sw128(w_addr + kb * 32), kIdesc, kb > 0 ? 1u : 0u);
      umma_commit(empty_bar(stage));
      umma_commit(accf_bar(b));
    }
    if (!ok) {
      umma_commit(drain_bar);  // MMAs may be in flight: wait (bounded) until they retire
      const unsigned long long t0 = globaltimer();
      while (!mbar_try_wait(drain_bar, 0) && globaltimer() - t0 < 1000000ull) {
      }
    }
  } else if (warp >= 2) {
    // ---- epilogue: lane quarter (warp % 4), one row of C per lane
    const int quarter = warp & 3;
    const bool read_c = (P.ber != 0.0 || P.bei != 0.0);
    const uint32_t lane_taddr = tmem_base + (uint32_t(quarter * 32) << 16);
    int rb = rb0, j = j0;
    for (long long u = blockIdx.x, it = 0; u < P.total_units;
         u += gridDim.x, ++it, next_unit(rb, j)) {
      const int b = int(it & 1);
      const uint32_t bpar = uint32_t((it >> 1) & 1);
      // the scale exponents load while the accumulator is awaited
      int si[RT_G];
#pragma unroll
      for (int g = 0; g < RT_G; ++g) {
        const int i = (rb * RT_G + g) * 128 + quarter * 32 + lane;
        si[g] = i < P.m ? P.sigA[i] : 0;
      }
      const int tauj = P.sigB[j];
      // warp-uniform: the TMEM loads and the warp's arrival below are collective
      if (!__all_sync(0xffffffffu, mbar_wait(accf_bar(b), bpar, abort, P.wait_limit_ns))) break;
      tc_fence_after();
      __syncwarp();
      uint32_t v[RT_G][32];
#pragma unroll
      for (int g = 0; g < RT_G; ++g)
        tmem_ld32_nowait(lane_taddr + uint32_t((b * RT_G + g) * 32), v[g]);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acce_bar(b));  // the accumulator may be overwritten
#pragma unroll
      for (int g = 0; g < RT_G; ++g) {
        const int i = (rb * RT_G + g) * 128 + quarter * 32 + lane;
        bool active = i < P.m;
        if (active && P.fill != 0) {
          const int64_t ti = (i / P.tile_m) * int64_t(P.tile_m);
          const int64_t tj = (j / P.tile_n) * int64_t(P.tile_n);
          active = tile_is_active(P.fill, ti, tj, ::min((int64_t)P.tile_m, (int64_t)P.m - ti),
                                  ::min((int64_t)P.tile_n, (int64_t)P.n - tj), P.ro, P.co);
        }
        if (active) {
          // limb L of S = sum of S_j 2^(8 (j - 4L)) over j = 4L .. 4L + 3 (below
          // 2^47): two 32-bit shift-adds (each below 2^31) and one wide multiply-add
          auto limb = [&](int j0) {
            const uint32_t a = v[g][j0] + (v[g][j0 + 1] << 8);
            const uint32_t bb = v[g][j0 + 2] + (v[g][j0 + 3] << 8);
            return (unsigned long long)bb * 65536ull + a;
          };
          const int e = -(si[g] + tauj);
          double xr =
              scale_pow2(crt_from_limbs<true>(limb(0), limb(4), limb(8), limb(12), P.rp), e);
          double xi = 0.0;
          if (CPLX)
            xi = scale_pow2(crt_from_limbs<true>(limb(16), limb(20), limb(24), limb(28), P.rp),
                            e);
          if (si[g] == kSigmaNonFinite || tauj == kSigmaNonFinite)
            xr = xi = __longlong_as_double(kNaNBits);
          store_c<DT>(P.C, i + int64_t(j) * P.ldc, xr, xi, P.alr, P.ali, P.ber, P.bei, read_c);
        }
      }
    }
  }

  if (copies_pending) {
    // copies issued by this CTA may still be landing in shared memory
    const unsigned long long t0 = globaltimer();
    while (globaltimer() - t0 < 2000000ull) {
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort && threadIdx.x == 0) atomicExch(P.status, 1);
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "n"(2 * RT_G * 32)
                 : "memory");
  }
}

// --------------------------------------------------------------------------
// host orchestration

int sm_count() {  // read once per device
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return 148;
  }
  if (!cached[dev]) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v < 2)
      v = 148;
    cached[dev] = v;
  }
  return cached[dev];
}

struct Layout {
  int nmod;
  bool split;              // complex with the split moduli
  bool pairs;              // the two planes of a split modulus lie side by side in pieces
  int nsub;                // products per modulus: 1 (real), 2 (split) or 3 (Karatsuba)
  int64_t K2, kp;          // reals per operand row; residue row length (k padded to 128)
  int rowsA, rowsB, nb;    // A rows, B rows, B residue rows per product
  bool at;                 // op(A) = N too long for in-place tiles: A copied k-major
  bool mn;                 // op(A) = N: A read in place (m-major)
  bool mnB;                // op(B) = T or C: B read in place (n-major)
  int ksA, ksB;            // slices of off_partA and off_partB (1: none)
  int nchunks, nt;         // k-chunks and tile width of the GEMM (choose_gemm)
  bool r8;                 // the residues of C are bytes, one plane per product and k-chunk
  int64_t ldR, planeR;     // elements between the columns of a plane and between planes
  int64_t ldAt;            // leading dimension of At (elements of A's type)
  size_t off_sigA, off_sigB, off_resA, off_resB, off_R, off_At, off_status, off_tiles;
  size_t off_partA, off_partB;  // room that is not used (layout_of)
  size_t off_ssq, off_list;     // one-pass row scaling (onepass_operands): scaled sums
                                // of squares, rows sent back and their two counts
  size_t total;
};

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// The moduli's constants, made once: the 16 split ones take the host 15 us.
const Crt& crt_of(const Layout& L) {
  struct Table {
    Crt general[kMaxUsableModuli + 1], split, split_float;
    Table() : split(make_crt_split(kSplitCount)), split_float(make_crt_split(kSplitCountFloat)) {
      for (int n = 1; n <= kMaxUsableModuli; ++n) general[n] = make_crt(n);
    }
  };
  static const Table t;
  if (!L.split) return t.general[L.nmod];
  return L.nmod == kSplitCount ? t.split : t.split_float;
}

// oz_slice_mma's rows for j (`sign` 1) or -j, made once (17 us of host time). V's
// planes hold -v, as oz_slice's.
const SliceRow* split_slice_rows(const Crt& crt, int sign) {
  struct Table {
    SliceRow row[kSlicePlanes];
    Table(const Crt& c, int s) {
      for (int t = 0; t < kSplitCount; ++t) {
        row[2 * t] = make_slice_row(c.p[t], 1, s * c.j[t]);
        row[2 * t + 1] = make_slice_row(c.p[t], -1, s * c.j[t]);
      }
    }
  };
  static const Table plus(crt, 1), minus(crt, -1);
  return sign > 0 ? plus.row : minus.row;
}

// Complex double planes with the split moduli come in pairs: the 32 planes of a
// row are written at once, and as many streams far apart cost the slicer (see
// oz_slice_mma: 1.43 ms with planes apart, 1.16 in pairs), while the GEMM, which
// reads one plane of many rows, slows down once a row's pieces of all planes
// span many pages (m = n = 1024, k = 250000: 6.2 ms apart or in pairs, 6.9 in
// groups of 4, 9.7 of 8). Pieces of 1 KB, or less for rows so short that the
// padding of the last piece could outgrow the workspace of the three-product form
// (45 planes to these 32: up to 3/8 more).
ResidueLayout residue_layout(const Layout& L, int rows) {
  if (!L.pairs) return {rows * L.kp, L.kp, L.kp, 62, 1};
  const int shift = L.kp < 256 ? 7 : L.kp < 2304 ? 8 : 10;
  const int64_t kc = int64_t(1) << shift, row = (L.kp + kc - 1) / kc * 2 * kc;
  return {rows * row, row, kc, shift, 2};
}

size_t residue_bytes(const Layout& L, int rows) {
  const ResidueLayout lay = residue_layout(L, rows);
  return size_t(L.nmod * L.nsub / lay.G) * size_t(lay.group);
}

// Time (us) of the INT8 GEMM over `chunks` k-chunks with pair tiles 256 x 256 nt:
// rounds of work units over the CTA pairs, a unit taking its k-blocks at the measured
// rate (0.44 us per 256 x 256 x 128, 8 % less in the wider tile, which loads A once
// for two MMAs) and its hand-over (the wider tile's single accumulator exposes its
// drain).
double gemm_model_us(const Layout& L, int64_t m, int64_t n, int chunks, int nt, int pairs) {
  const double units = double(L.nmod * L.nsub) * chunks * double((m + 255) / 256) *
                       double((n + 256 * nt - 1) / (256 * nt));
  const double blocks = std::ceil(double(L.kp / BKB) / chunks);
  const double unit = nt == 2 ? blocks * 0.81 + 5.0 : blocks * 0.443 + 1.2;
  return std::ceil(units / pairs) * unit;
}

// k-chunks and tile width of the GEMM. Chunks stay within the exact INT32 bound;
// more of them fill the CTA pairs when there are few units (256 x 256 real double: 15
// units for 74 pairs), as long as all byte planes go to the tensor-core reconstruction.
// Each costs its planes' write and read, and may add at most 4 MB to the workspace
// (complex problems have room for them anyway, see layout_of).
constexpr size_t kMoreChunksBytes = size_t(4) << 20;
void choose_gemm(Layout& L, int64_t m, int64_t n) {
  const int64_t blocks = L.kp / BKB, planes = L.nmod * L.nsub;
  const int64_t limit = L.split ? kChunkBlocksSplit : kChunkBlocks;
  const int least = int(std::max<int64_t>(1, (blocks + limit - 1) / limit));
  const int pairs = std::max(1, sm_count() / 2);
  double best = 0.0;
  L.nchunks = 0;
  for (int c = least; c == least || (c <= blocks / 4 && c * planes <= RT_KP); ++c) {
    const double more = double(c - 1) * planes * m * n;  // bytes
    if (c > least && !L.split && more > kMoreChunksBytes) break;
    for (int nt = 1; nt <= (n >= 512 ? 2 : 1); ++nt) {
      const double t = gemm_model_us(L, m, n, c, nt, pairs) + more / 2.5e6;
      if (L.nchunks == 0 || t < 0.97 * best) {
        best = t;
        L.nchunks = c;
        L.nt = nt;
      }
    }
  }
}

// In-place reading of an m-major operand: the transposing slicer's tiles of
// 128 (complex) or 256 (real) elements along k must fit the grid's y extent.
bool mn_fits(const GemmProblem& p) {
  const int64_t kp = (p.k + BKB - 1) / BKB * BKB;
  const int64_t kt = dtype_is_complex(p.dtype) ? 128 : 256;
  return (kp + kt - 1) / kt <= 65535;
}

// Slices of partial sums of the in-place row norms that the workspace has room for
// (layout_of); the kernels cut finer and keep theirs elsewhere (in_place_slices).
int norm_slices(int64_t rows, int64_t k) {
  if (rows >= kMnRows || k <= 512) return 1;
  const int64_t want = std::min<int64_t>(((int64_t(1) << 18) + rows - 1) / rows, 4096);
  return int(std::max<int64_t>(1, std::min<int64_t>(want, (k + 511) / 512)));
}

Layout layout_of(const GemmProblem& p, int moduli) {
  Layout L{};
  const bool dbl = dtype_is_double(p.dtype), cplx = dtype_is_complex(p.dtype);
  const int def = dbl ? kDefaultModuli : kDefaultModuliFloat;
  const int count = moduli > 0 ? std::min(moduli, kMaxUsableModuli) : def;
  // complex problems at the default precision take the split moduli; another
  // count names that many moduli of the general table
  L.split = cplx && count == def;
  L.nmod = L.split ? (dbl ? kSplitCount : kSplitCountFloat) : count;
  L.nsub = L.split ? 2 : cplx ? 3 : 1;
  L.pairs = L.split && dbl;
  // planes of the three-product form, whose size the workspace keeps (see below)
  const size_t planes = size_t(count) * (cplx ? 3 : 1);
  L.K2 = cplx ? 2 * p.k : p.k;
  L.kp = (p.k + BKB - 1) / BKB * BKB;
  L.rowsA = int(p.m);
  L.rowsB = int(p.n);
  L.nb = int(p.n);
  // op(A) = N and op(B) = T, C: read in place (the tiles of the transposing
  // slicer fit the grid), else A is copied k-major (B is then unsupported)
  L.mn = p.opA == 0 && mn_fits(p);
  L.at = p.opA == 0 && !L.mn;
  L.mnB = p.opB != 0;
  L.ksA = L.mn ? norm_slices(p.m, p.k) : 1;
  L.ksB = L.mnB ? norm_slices(p.n, p.k) : 1;
  choose_gemm(L, p.m, p.n);
  // bytes where the tensor-core reconstruction takes all planes (its columns lie on
  // 16-byte boundaries), else one int32 sum per product
  L.r8 = L.nmod * L.nsub * L.nchunks <= RT_KP;
  L.ldR = L.r8 ? (p.m + 15) / 16 * 16 : p.m;
  // byte planes an odd number of 128-byte lines apart: a box of the reconstruction
  // reads a line of each, which should not fall on few L2 slices
  L.planeR = L.r8 ? ((L.ldR * L.nb + 127) / 128 | 1) * 128 : L.ldR * L.nb;
  L.ldAt = L.at ? (p.k + 7) / 8 * 8 : 0;
  size_t off = 0;
  L.off_sigA = off;
  off = align256(off + sizeof(int) * L.rowsA);
  L.off_sigB = off;
  off = align256(off + sizeof(int) * L.rowsB);
  // The size asked for is that of the three-product form (45 planes to the split form's
  // 32, and int32 sums from the second k-chunk on), of which the planes of the split
  // form's k-chunks take a part: AUTO holds it against a quarter of the device memory,
  // so the problems that the limit turns away are the ones it was measured with.
  const bool one_chunk = (L.kp / BKB + kChunkBlocks - 1) / kChunkBlocks <= 1;
  const size_t reserved = align256(planes * L.rowsA * L.kp) + align256(planes * L.nb * L.kp) +
                          align256((one_chunk ? 1 : sizeof(int)) * planes * L.nb * L.rowsA);
  const size_t start = off;
  L.off_resA = off;
  off = align256(off + residue_bytes(L, L.rowsA));
  L.off_resB = off;
  off = align256(off + residue_bytes(L, L.nb));
  L.off_R = off;
  off = align256(off + (L.r8 ? L.nchunks : sizeof(int)) * size_t(L.nmod) * L.nsub *
                           L.planeR);
  off = std::max(off, start + reserved);
  L.off_At = off;
  off = align256(off + size_t(dtype_bytes(p.dtype)) * size_t(L.rowsA) * size_t(L.ldAt));
  L.off_status = off;
  off = align256(off + 256);
  L.off_tiles = off;
  off = align256(off + sizeof(int) * size_t((L.rowsA + 255) / 256) * ((L.nb + 255) / 256));
  L.off_partA = off;
  // room for partial sums of the in-place norms, part of the size that is asked for;
  // nothing lies here (in_place_slices)
  off = align256(off + (L.ksA > 1 ? size_t(L.ksA) * L.rowsA * (sizeof(double) + sizeof(int)) : 0));
  L.off_partB = off;
  off = align256(off + (L.ksB > 1 ? size_t(L.ksB) * L.rowsB * (sizeof(double) + sizeof(int)) : 0));
  L.off_ssq = off;  // A's rows, then B's
  off = align256(off + sizeof(double) * (size_t(L.rowsA) + L.rowsB));
  L.off_list = off;  // lists of A's and B's rows, their exact flags, the two counts
  off = align256(off + sizeof(int) * (2 * (size_t(L.rowsA) + L.rowsB) + 2));
  L.total = off;
  return L;
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    cudaDriverEntryPointQueryResult q;
    void* f = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  });
  return fn;
}

// Residues of an operand: dims (bytes of a piece, planes of a group, pieces, rows,
// groups), boxes of one k-block of one plane x box_rows rows (rows past the end
// read as zeros).
bool make_map(CUtensorMap* map, void* base, const Layout& L, int rows, int box_rows) {
  auto fn = encode_fn();
  if (!fn) return false;
  const ResidueLayout lay = residue_layout(L, rows);
  const int64_t pieces = lay.row / (lay.G * lay.kc);
  cuuint64_t dims[5] = {cuuint64_t(lay.kc), cuuint64_t(lay.G), cuuint64_t(pieces),
                        cuuint64_t(rows), cuuint64_t(L.nmod * L.nsub / lay.G)};
  cuuint64_t strides[4] = {cuuint64_t(lay.kc), cuuint64_t(lay.G * lay.kc), cuuint64_t(lay.row),
                           cuuint64_t(lay.group)};
  cuuint32_t box[5] = {cuuint32_t(BKB), 1u, 1u, cuuint32_t(box_rows), 1u};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, base, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// Residue bytes of C for the tensor-core reconstruction: dims (m, nb, planes)
// with strides (ldR, planeR) bytes (multiples of 16), boxes of 128 rows x 1 column
// x all planes (rows past m read as zeros), 128-byte swizzle: one 128-byte row per
// plane, the MN-major operand layout.
bool make_map_recon(CUtensorMap* map, void* base, const Layout& L) {
  auto fn = encode_fn();
  if (!fn) return false;
  const int planes = L.nmod * L.nsub * L.nchunks;
  cuuint64_t dims[3] = {cuuint64_t(L.rowsA), cuuint64_t(L.nb), cuuint64_t(planes)};
  cuuint64_t strides[2] = {cuuint64_t(L.ldR), cuuint64_t(L.planeR)};
  cuuint32_t box[3] = {128u, 1u, cuuint32_t(planes)};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}


}  // namespace oz

size_t ozaki_workspace_bytes(const GemmProblem& p, int moduli) {
  if (p.m <= 0 || p.n <= 0) return 0;
  return oz::layout_of(p, moduli).total;
}

bool ozaki_copies_a(const GemmProblem& p) { return p.opA == 0 && !oz::mn_fits(p); }

bool ozaki_supported(const GemmProblem& p) {
  // op(B) = T or C: B is read in place, which needs the slicer's tiles to fit
  return (p.opB == 0 || ((p.opB == 1 || p.opB == 2) && oz::mn_fits(p))) &&
         p.m <= (1 << 24) && p.n <= (1 << 23);
}

namespace {
// Reals per slicing thread: 8 by default (more resident warps), 16 with
// SPLAB_OZAKI_SLICE_EL=16.
int slice_elems() {
  static const int el = [] {
    const char* v = std::getenv("SPLAB_OZAKI_SLICE_EL");
    return (v && std::atoi(v) == 16) ? 16 : 8;
  }();
  return el;
}

// Moduli of the unrolled slicers: the default counts of the input type, real
// (MODE 0) or complex with split moduli (MODE 3); 0 in MODE 2 (always a loop).
template <typename TIn, int MODE>
constexpr int unrolled_moduli() {
  return MODE == 0   ? (sizeof(TIn) == 8 ? oz::kDefaultModuli : oz::kDefaultModuliFloat)
         : MODE == 3 ? (sizeof(TIn) == 8 ? oz::kSplitCount : oz::kSplitCountFloat)
                     : 0;
}

// The default modulus counts over all moduli run unrolled
// (SPLAB_OZAKI_SLICE_UNROLL=0 keeps the loop).
bool slice_unroll() {
  static const bool on = [] {
    const char* v = std::getenv("SPLAB_OZAKI_SLICE_UNROLL");
    return !(v && v[0] == '0');
  }();
  return on;
}

template <typename TIn, bool VEC, int EL, int MODE>
void launch_slice_el(int ndig, unsigned grid, cudaStream_t st, const TIn* X, int64_t ld,
                     int64_t len, int rows, int64_t kp, const int* sig, int s_sign, int8_t* res,
                     const oz::ResidueLayout& lay, int64_t stride, const oz::SliceConsts& sc,
                     double* ssq) {
  using namespace oz;
  constexpr int kNU = unrolled_moduli<TIn, MODE>();
  constexpr int kDigU = sizeof(TIn) == 8 ? 4 : 3;  // digits of the default scaling
  if constexpr (kNU > 0) {
    if (sc.n == kNU && ndig == kDigU && slice_unroll()) {
      if (ssq)
        oz_slice<TIn, VEC, kDigU, EL, kNU, MODE, true><<<grid, 256, 0, st>>>(
            X, ld, len, rows, kp, sig, s_sign, res, lay, stride, sc, ssq);
      else
        oz_slice<TIn, VEC, kDigU, EL, kNU, MODE><<<grid, 256, 0, st>>>(
            X, ld, len, rows, kp, sig, s_sign, res, lay, stride, sc, nullptr);
      return;
    }
  }
  if (ndig <= 3)
    oz_slice<TIn, VEC, 3, EL, 0, MODE><<<grid, 256, 0, st>>>(
        X, ld, len, rows, kp, sig, s_sign, res, lay, stride, sc, nullptr);
  else if (ndig == 4)
    oz_slice<TIn, VEC, 4, EL, 0, MODE><<<grid, 256, 0, st>>>(
        X, ld, len, rows, kp, sig, s_sign, res, lay, stride, sc, nullptr);
  else
    oz_slice<TIn, VEC, 5, EL, 0, MODE><<<grid, 256, 0, st>>>(
        X, ld, len, rows, kp, sig, s_sign, res, lay, stride, sc, nullptr);
}

// ssq (unrolled default scaling only): also the rows' scaled sums of squares
template <typename TIn, bool VEC>
void launch_slice(int ndig, cudaStream_t st, const TIn* X, int64_t ld, int64_t len, int rows,
                  int64_t kp, const int* sig, int mode, int s_sign, int8_t* res,
                  const oz::ResidueLayout& lay, int64_t stride, const oz::SliceConsts& sc,
                  double* ssq) {
  const int el = slice_elems();
  const int64_t kreal = mode != 0 ? 2 * kp : kp;  // reals per row a thread group covers
  const unsigned grid = unsigned((int64_t(rows) * (kreal / el) + 255) / 256);
  auto run = [&](auto el_tag, auto mode_tag) {
    launch_slice_el<TIn, VEC, decltype(el_tag)::value, decltype(mode_tag)::value>(
        ndig, grid, st, X, ld, len, rows, kp, sig, s_sign, res, lay, stride, sc, ssq);
  };
  using E8 = std::integral_constant<int, 8>;
  using E16 = std::integral_constant<int, 16>;
  using M0 = std::integral_constant<int, 0>;
  using M2 = std::integral_constant<int, 2>;
  using M3 = std::integral_constant<int, 3>;
  auto by_mode = [&](auto el_tag) {
    if constexpr (sizeof(TIn) == 4) {  // double: oz_slice_mma
      if (mode == 3) return run(el_tag, M3{});
    }
    if (mode == 2) run(el_tag, M2{});
    else run(el_tag, M0{});
  };
  if (el == 16) by_mode(E16{});
  else by_mode(E8{});
}

// Residues of m-major rows (op(A) = N read in place): oz_slice_mn
template <typename TIn, bool VEC, int MODE>
void launch_slice_mn_v(int ndig, dim3 grid, cudaStream_t st, const TIn* X, int64_t ld, int m,
                       int64_t k, int64_t kp, const int* sig, int s_sign, int conj, int8_t* res,
                       const oz::ResidueLayout& lay, int64_t stride, const oz::SliceConsts& sc) {
  using namespace oz;
  constexpr int kNU = unrolled_moduli<TIn, MODE>();
  constexpr int kDigU = sizeof(TIn) == 8 ? 4 : 3;
  if constexpr (kNU > 0) {
    if (sc.n == kNU && ndig == kDigU && slice_unroll()) {
      oz_slice_mn<TIn, VEC, kDigU, kNU, MODE>
          <<<grid, 256, 0, st>>>(X, ld, m, k, kp, sig, s_sign, conj, res, lay, stride, sc);
      return;
    }
  }
  if (ndig <= 3)
    oz_slice_mn<TIn, VEC, 3, 0, MODE>
        <<<grid, 256, 0, st>>>(X, ld, m, k, kp, sig, s_sign, conj, res, lay, stride, sc);
  else if (ndig == 4)
    oz_slice_mn<TIn, VEC, 4, 0, MODE>
        <<<grid, 256, 0, st>>>(X, ld, m, k, kp, sig, s_sign, conj, res, lay, stride, sc);
  else
    oz_slice_mn<TIn, VEC, 5, 0, MODE>
        <<<grid, 256, 0, st>>>(X, ld, m, k, kp, sig, s_sign, conj, res, lay, stride, sc);
}

template <typename TIn>
void launch_slice_mn(int ndig, cudaStream_t st, const TIn* X, int64_t ld, int m, int64_t k,
                     int64_t kp, const int* sig, int mode, int s_sign, int conj, int8_t* res,
                     const oz::ResidueLayout& lay, int64_t stride, const oz::SliceConsts& sc) {
  const int64_t kt = mode != 0 ? 128 : 256;  // elements per row per tile
  const dim3 grid(unsigned((m + 7) / 8), unsigned((kp + kt - 1) / kt));
  auto run = [&](auto vec_tag, auto mode_tag) {
    launch_slice_mn_v<TIn, decltype(vec_tag)::value, decltype(mode_tag)::value>(
        ndig, grid, st, X, ld, m, k, kp, sig, s_sign, conj, res, lay, stride, sc);
  };
  using T = std::true_type;
  using F = std::false_type;
  // 16-byte element loads for complex double with a 16-byte aligned base
  const bool vec = sizeof(TIn) == 8 && reinterpret_cast<uintptr_t>(X) % 16 == 0;
  if (mode == 3) {
    if (vec) run(T{}, std::integral_constant<int, 3>{});
    else run(F{}, std::integral_constant<int, 3>{});
  } else if (mode == 2) {
    if (vec) run(T{}, std::integral_constant<int, 2>{});
    else run(F{}, std::integral_constant<int, 2>{});
  } else {
    run(F{}, std::integral_constant<int, 0>{});
  }
}

// k-slices of the in-place row norms: threads (one per row and slice) for two
// full loads of the GPU, slices of at least 32 elements (a thread's loads go out in
// batches of 8), and 512 slices or slices of 512 elements (at most 4096, the grid's y
// extent), since each costs a partial sum to add up. The partial sums lie where the
// operand's residues go next. Slices of 512 elements and more throughout had left a
// 1501 x 1207 operand with 24 blocks (39.8 us; now 9.6); up to 4096 slices, added up by
// eight threads a row, took 446 us for both operands of 256 x 256 x 100000 complex
// double NT (161 now, 169 for one of them before) and 463 for 89 x 93 x 122231 complex
// float (126, 339). Up to 64 elements the second launch costs more than it saves (24
// against 17 us).
int in_place_slices(int64_t rows, int64_t k) {
  if (rows >= oz::kMnRows || k <= 64) return 1;
  const int64_t want = (int64_t(oz::sm_count()) * 4096 + rows - 1) / rows;
  const int64_t most = std::min<int64_t>(4096, std::max<int64_t>(512, k / 512));
  return int(std::max<int64_t>(1, std::min({want, (k + 31) / 32, most})));
}

// Row scale exponents of the operands read in place.
template <typename TIn>
void scale_in_place(const oz::Layout& L, const oz::Crt& crt, const GemmProblem& p, bool cplx,
                    int* sigA, int* sigB, int8_t* resA, int8_t* resB, cudaStream_t st) {
  using namespace oz;
  const ScaleBits bits{crt.q_bits, crt.thr};
  auto scale = [&](const void* X, int64_t ld, int rows, int8_t* scratch, int* sig) {
    const int ks = in_place_slices(rows, p.k);
    const int64_t kspan = (p.k + ks - 1) / ks;
    double* partS = reinterpret_cast<double*>(scratch);
    int* partE = reinterpret_cast<int*>(scratch + sizeof(double) * size_t(ks) * rows);
    const dim3 grid(unsigned((rows + 255) / 256), unsigned(ks));
    if (cplx)
      oz_row_scale_mn<TIn, true><<<grid, 256, 0, st>>>(static_cast<const TIn*>(X), ld, rows, p.k,
                                                       kspan, bits, sig, partS, partE);
    else
      oz_row_scale_mn<TIn, false><<<grid, 256, 0, st>>>(static_cast<const TIn*>(X), ld, rows, p.k,
                                                        kspan, bits, sig, partS, partE);
    if (ks > 1) {  // a warp per 16 slices: warp 0 adds up the warps' sums one by one
      const int warps = std::min(32, std::max(8, ks / 16));
      oz_row_scale_combine<<<unsigned((rows + 31) / 32), unsigned(32 * warps), 0, st>>>(
          partS, partE, rows, ks, bits, sig);
    }
  };
  if (L.mn) scale(p.A, p.lda, L.rowsA, resA, sigA);
  if (L.mnB) scale(p.B, p.ldb, L.rowsB, resB, sigB);
}

// Slicer constants of the moduli (s_sign: the sign of j, split moduli), and the
// digit count covering |x| <= 2^Q: 3 of 13 bits, 4 balanced of 15 bits, or 5 of
// 13.
oz::SliceConsts slice_consts(const oz::Layout& L, const oz::Crt& crt, int s_sign, int* ndig_out) {
  using namespace oz;
  SliceConsts sc{};
  sc.n = L.nmod;
  sc.p0 = float(crt.p[0]);
  for (int t = 0; t < L.nmod; ++t) {
    const int pt = crt.p[t];
    sc.neg_p[t] = f2_pack(-float(pt), -float(pt));
    sc.inv_p[t] = f2_pack(1.0f / float(pt), 1.0f / float(pt));
  }
  const int ndig = crt.q_bits + 1 <= 39 ? 3 : (crt.q_bits + 1 <= 58 ? 4 : 5);
  const long long base = ndig == 4 ? 32768 : 8192;
  for (int t = 0; t < L.nmod; ++t) {
    const int pt = crt.p[t];
    auto centred = [pt](long long w) {
      const float c = float(w > pt / 2 ? w - pt : w);
      return f2_pack(c, c);
    };
    const int j = s_sign > 0 ? crt.j[t] : pt - crt.j[t];
    long long w = 1;
    for (int i = 0; i < 5; ++i) {  // w = base^i mod p
      if (i > 0) sc.c[t][i - 1] = centred(w);
      if (L.split) sc.cj[t][i] = centred(w * j % pt);
      w = (w * base) % pt;
    }
  }
  *ndig_out = ndig;
  return sc;
}

// Residues of k-major complex double rows for the split moduli (oz_slice_mma), with
// the rows' scaled sums of squares when ssq is given, or of the listed rows only.
void launch_slice_mma(const oz::Layout& L, const oz::Crt& crt, const double* X, int64_t ld,
                      int rows, const int* sigma, int sign, int8_t* res, double* ssq,
                      const int* list, const int* count, cudaStream_t st) {
  using namespace oz;
  SliceMmaParams P{};
  P.X = X;
  P.ld = ld;
  P.len = L.K2;
  P.rows = rows;
  P.vec = reinterpret_cast<uintptr_t>(X) % 16 == 0 && ld % 2 == 0;
  P.sigma = sigma;
  P.res = res;
  P.lay = residue_layout(L, rows);
  P.ssq = ssq;
  P.list = list;
  P.count = count;
  P.steps_per_row = int(2 * L.kp / kStepReals);
  const int wpr = P.steps_per_row >= 4 ? 4 : 2;  // kp >= 128: at least two steps
  P.warps_per_row = wpr;
  std::copy_n(split_slice_rows(crt, sign), kSlicePlanes, P.row);
  const long long slots = (long long)kSliceBlocks * sm_count();
  const long long steps = (long long)rows * P.steps_per_row;
  // equal segments of a row, of at most 32 steps per warp, and short enough for
  // about eight chunks per block (k = 250000: 6.0 ms for both operands with 16, 5.6
  // with 32; the ring fills anew for each)
  const long long most = std::max<long long>(1, std::min<long long>(32, steps / (32 * slots)));
  const long long segs = (P.steps_per_row + most * wpr - 1) / (most * wpr);
  P.run = int((P.steps_per_row + segs * wpr - 1) / (segs * wpr));
  const long long chunks = ((long long)rows * wpr + 3) / 4 * segs;
  const unsigned grid = unsigned(std::min(slots, chunks));
  if (ssq)
    oz_slice_mma<true><<<grid, 128, 0, st>>>(P);
  else
    oz_slice_mma<false><<<grid, 128, 0, st>>>(P);
}

// Residues of A (which & 1) and B (which & 2).
template <typename TIn>
void slice_operands(const oz::Layout& L, const oz::Crt& crt, const GemmProblem& p, bool cplx,
                    const int* sigA, const int* sigB, int8_t* resA, int8_t* resB, int which,
                    cudaStream_t st, double* ssq) {
  using namespace oz;
  const TIn* A = static_cast<const TIn*>(p.A);
  const TIn* B = static_cast<const TIn*>(p.B);
  double* ssqA = ssq && !L.mn ? ssq : nullptr;
  double* ssqB = ssq && !L.mnB ? ssq + L.rowsA : nullptr;
  const int64_t ldA = cplx ? 2 * p.lda : p.lda;  // in real elements
  const int64_t ldB = cplx ? 2 * p.ldb : p.ldb;
  const int vec_elems = 16 / int(sizeof(TIn));
  const bool vecA = (reinterpret_cast<uintptr_t>(A) % 16 == 0) && (ldA % vec_elems == 0);
  const bool vecB = (reinterpret_cast<uintptr_t>(B) % 16 == 0) && (ldB % vec_elems == 0);
  // complex, split moduli: A's planes take -j for A^H (conj(a) swaps u and v);
  // three products: A's third plane is re(a) - im(a) for A^H (conj(a) b: Im =
  // r2 - r0 + r1) and re(a) + im(a) otherwise, B's is re + im
  const int mode = L.split ? 3 : cplx ? 2 : 0;
  const int sumA = p.opA == 2 ? -1 : 1;
  int ndig = 0;
  const SliceConsts scA = slice_consts(L, crt, sumA, &ndig);
  const SliceConsts sc = slice_consts(L, crt, 1, &ndig);
  const ResidueLayout layA = residue_layout(L, L.rowsA), layB = residue_layout(L, L.nb);
  const int64_t strideA = layA.plane(L.nsub), strideB = layB.plane(L.nsub);
  if constexpr (std::is_same<TIn, double>::value) {
    if (L.pairs) {  // k-major complex double: oz_slice_mma
      if ((which & 1) && !L.mn) {
        launch_slice_mma(L, crt, A, ldA, L.rowsA, sigA, sumA, resA, ssqA, nullptr, nullptr, st);
        which &= ~1;
      }
      if ((which & 2) && !L.mnB) {
        launch_slice_mma(L, crt, B, ldB, L.rowsB, sigB, 1, resB, ssqB, nullptr, nullptr, st);
        which &= ~2;
      }
    }
  }
  if ((which & 1) && L.mn)
    launch_slice_mn<TIn>(ndig, st, A, p.lda, L.rowsA, p.k, L.kp, sigA, mode, sumA, 0, resA,
                         layA, strideA, scA);
  else if ((which & 1) && vecA)
    launch_slice<TIn, true>(ndig, st, A, ldA, L.K2, L.rowsA, L.kp, sigA, mode, sumA, resA,
                            layA, strideA, scA, ssqA);
  else if (which & 1)
    launch_slice<TIn, false>(ndig, st, A, ldA, L.K2, L.rowsA, L.kp, sigA, mode, sumA, resA,
                             layA, strideA, scA, ssqA);
  if ((which & 2) && L.mnB)  // op(B) = T or C: n-major rows, conjugated for C
    launch_slice_mn<TIn>(ndig, st, B, p.ldb, L.rowsB, p.k, L.kp, sigB, mode, 1,
                         p.opB == 2 ? 1 : 0, resB, layB, strideB, sc);
  else if ((which & 2) && vecB)
    launch_slice<TIn, true>(ndig, st, B, ldB, L.K2, L.rowsB, L.kp, sigB, mode, 1, resB, layB, strideB,
                            sc, ssqB);
  else if (which & 2)
    launch_slice<TIn, false>(ndig, st, B, ldB, L.K2, L.rowsB, L.kp, sigB, mode, 1, resB, layB, strideB,
                             sc, ssqB);
}

// One-pass row scaling. The two-pass order reads every row twice: once for
// its norm (the scale exponent), once to slice it. Here the exponent comes
// from a sample of each row (16 evenly spread runs, 1/16 of its reals, the
// sum of squares extrapolated to the whole row) unless the estimate lies too
// near the norms where the exponents change for what the spread of the runs
// says of it (estimate_clear), or the sample is zero or not finite: such rows
// take the exact norm at once. The default slicer also sums the squares of
// the scaled values, and an estimated exponent stands when that sum lies in
// [low^2, 4 low^2), low = thr 2^Q (Crt::thr), with a relative margin at both
// ends far above the rounding of either sum (see launch_row_scale): the
// scaled norm then lies in [low, 2 low), which is what the exact exponent
// gives. Other rows (a sample that misjudged the row) get the exact norm and
// are sliced again. Each row thus ends with the exponent and residues of the
// two-pass order, whatever the order of the atomic sums. Used for each
// k-major operand (an operand read in place keeps its norms) with the default
// modulus count and unrolled slicer and rows of at least kOnePassMinLen reals;
// SPLAB_OZAKI_ONEPASS=0 (read per call) keeps the two-pass order.
//
// It pays from about 256 MB of k-major operands: the norms' second read (6 TB/s)
// against the sample and two more launches (387 x 515 x 60013 complex double, 866
// MB: 150 us of norms, 30 us of estimates and checks); rows of 16384 reals keep 64
// reals per run. Real float rows that short gain nothing (2000 + 2000 rows of 40000: 1.53
// ms against 1.51) and lose 14 % where the rows take their exact norms (1.58 against
// 1.39). Rows of 131072 reals always take it.
constexpr int64_t kOnePassMinLen = 16384, kOnePassLongLen = 131072;
constexpr double kOnePassMinBytes = 256e6;

// The operands scaled in one pass: bit 1 A, bit 2 B (k-major ones only; the
// rows read in place keep their k-sliced norms)
int onepass_operands(const oz::Layout& L, const GemmProblem& p) {
  const char* v = std::getenv("SPLAB_OZAKI_ONEPASS");
  if (v && v[0] == '0') return 0;
  const int nu = dtype_is_double(p.dtype) ? oz::kDefaultModuli : oz::kDefaultModuliFloat;
  const bool unrolled = dtype_is_complex(p.dtype) ? L.split : L.nmod == nu;
  if (p.k <= 0 || !unrolled || !slice_unroll() || L.K2 < kOnePassMinLen) return 0;
  const double bytes = double((L.mn ? 0 : L.rowsA) + (L.mnB ? 0 : L.rowsB)) * double(L.K2) *
                       (dtype_is_double(p.dtype) ? 8 : 4);
  if (L.K2 < kOnePassLongLen && (p.dtype == kR32 || bytes < kOnePassMinBytes)) return 0;
  return (L.mn ? 0 : 1) | (L.mnB ? 0 : 2);
}

// oz_row_scale's operands: the k-major ones, all or none of them scaled in one pass.
// onepass: layout of the lists at `list` (A's rows, B's rows, their exact flags, the
// two counts).
template <typename TIn, int MODE>
void launch_row_scale(const oz::Layout& L, const oz::Crt& crt, const GemmProblem& p, bool cplx,
                      int* sigA, int* sigB, double* ssq, int* list, int* status,
                      cudaStream_t st) {
  using namespace oz;
  RowScaleParams P{};
  const int64_t re = cplx ? 2 : 1;
  int* exact = list + L.rowsA + L.rowsB;
  int* count = exact + L.rowsA + L.rowsB;
  P.op[0] = {p.A, re * p.lda, L.mn ? 0 : L.rowsA, sigA, exact, ssq, list, count};
  P.op[1] = {p.B,          re * p.ldb,     L.mnB ? 0 : L.rowsB, sigB, exact + L.rowsA,
             ssq + L.rowsA, list + L.rowsA, count + 1};
  P.len = L.K2;
  P.bits = {crt.q_bits, crt.thr};
  P.run = (L.K2 / (16 * kRuns) + 7) / 8 * 8;
  P.gap = L.K2 / kRuns;
  // the two sums of squares (norm kernel: runs of K2 / 256 terms per thread, then
  // trees; slicers: at most 128 terms per thread, trees, at most K2 / 128 atomics per
  // row) differ by at most about (K2 / 256 + K2 / 128 + 128) units of 2^-53 relative;
  // the margin is 2^-30, or K2 2^-59 for rows beyond 2^29 reals (float rows: a thread's
  // sum of up to 16 squares is in FP32, 2^-20 at most)
  const double delta = std::max(std::ldexp(1.0, sizeof(TIn) == 4 ? -19 : -30),
                                std::ldexp(double(L.K2), -59));
  const double low = std::ldexp(crt.thr, crt.q_bits);  // scaled norms lie in [low, 2 low)
  P.lo = low * low * (1.0 + delta);
  P.hi = 4.0 * low * low * (1.0 - delta);
  P.status = status;
  const int rows = P.op[0].rows + P.op[1].rows;
  if (rows == 0) return;
  const int grid = MODE == kRecheck ? std::min(rows, 2 * sm_count()) : rows;
  oz_row_scale<TIn, MODE><<<unsigned(grid), 256, 0, st>>>(P);
}

template <typename TIn, bool VEC, int EL, int MODE>
void launch_slice_rows_el(cudaStream_t st, const TIn* X, int64_t ld, int64_t len, int rows,
                          int64_t kp, const int* sig, int s_sign, int8_t* res,
                          const oz::ResidueLayout& lay, int64_t stride, const oz::SliceConsts& sc,
                          const int* list, const int* count) {
  using namespace oz;
  constexpr int kNU = unrolled_moduli<TIn, MODE>();
  constexpr int kDigU = sizeof(TIn) == 8 ? 4 : 3;
  const unsigned grid = unsigned((EL == 8 ? 4 : 2) * sm_count());  // one resident wave
  oz_slice_rows<TIn, VEC, kDigU, EL, kNU, MODE>
      <<<grid, 256, 0, st>>>(X, ld, len, rows, kp, sig, s_sign, res, lay, stride, sc, list, count);
}

// The listed rows of one operand: residues again
template <typename TIn>
void onepass_redo(const oz::Layout& L, const oz::Crt& crt, const TIn* X, int64_t ld, int rows,
                  const int* sig, int s_sign, int8_t* res, const int* list, const int* count,
                  cudaStream_t st) {
  if constexpr (std::is_same<TIn, double>::value) {
    if (L.pairs) {
      launch_slice_mma(L, crt, X, ld, rows, sig, s_sign, res, nullptr, list, count, st);
      return;
    }
  }
  int ndig = 0;
  const oz::SliceConsts sc = slice_consts(L, crt, s_sign, &ndig);
  const oz::ResidueLayout lay = residue_layout(L, rows);
  const int64_t stride = lay.plane(L.nsub);
  const bool vec = reinterpret_cast<uintptr_t>(X) % 16 == 0 && ld % (16 / int(sizeof(TIn))) == 0;
  auto run = [&](auto vec_tag, auto el_tag, auto mode_tag) {
    launch_slice_rows_el<TIn, decltype(vec_tag)::value, decltype(el_tag)::value,
                         decltype(mode_tag)::value>(st, X, ld, L.K2, rows, L.kp, sig, s_sign,
                                                    res, lay, stride, sc, list, count);
  };
  using T = std::true_type;
  using F = std::false_type;
  using E8 = std::integral_constant<int, 8>;
  using E16 = std::integral_constant<int, 16>;
  using M0 = std::integral_constant<int, 0>;
  using M3 = std::integral_constant<int, 3>;
  const bool e16 = slice_elems() == 16;
  auto by_mode = [&](auto vec_tag, auto el_tag) {
    if constexpr (sizeof(TIn) == 4) {
      if (L.split) return run(vec_tag, el_tag, M3{});
    }
    run(vec_tag, el_tag, M0{});
  };
  if (vec) {
    if (e16) by_mode(T{}, E16{});
    else by_mode(T{}, E8{});
  } else {
    if (e16) by_mode(F{}, E16{});
    else by_mode(F{}, E8{});
  }
}

// Check of A's (which & 1) and B's (which & 2) rows after slicing with their
// sums of squares, and the second pass over the rows it lists
template <typename TIn>
void onepass_fixup(const oz::Layout& L, const oz::Crt& crt, const GemmProblem& p, bool cplx,
                   int* sigA, int* sigB, int8_t* resA, int8_t* resB, double* ssq, int* list,
                   int which, cudaStream_t st) {
  using namespace oz;
  int* listA = list;
  int* listB = list + L.rowsA;
  int* cnt = list + 2 * (L.rowsA + L.rowsB);  // A's count, B's count
  launch_row_scale<TIn, kRecheck>(L, crt, p, cplx, sigA, sigB, ssq, list, nullptr, st);
  const int64_t ldA = cplx ? 2 * p.lda : p.lda, ldB = cplx ? 2 * p.ldb : p.ldb;
  if (which & 1)
    onepass_redo<TIn>(L, crt, static_cast<const TIn*>(p.A), ldA, L.rowsA, sigA,
                      p.opA == 2 ? -1 : 1, resA, listA, cnt, st);
  if (which & 2)
    onepass_redo<TIn>(L, crt, static_cast<const TIn*>(p.B), ldB, L.rowsB, sigB, 1, resB,
                      listB, cnt + 1, st);
}

// Tensor-core CRT reconstruction (oz_reconstruct_tc), the default for byte
// residues (at most 64 planes over all k-chunks); SPLAB_OZAKI_RECON_TC=0 (read per
// call) selects the CUDA-core kernel, as do int32 sums. Columns padded to 16 bytes
// let every m take it: 1501 x 2003 real double 76 us on the CUDA cores (uncoalesced
// bytes of 15 planes), 32 us here. True when it applies and its tensor map was made.
bool recon_tc_plan(const oz::Layout& L, unsigned char* R8, CUtensorMap* map) {
  const char* v = std::getenv("SPLAB_OZAKI_RECON_TC");
  if ((v && v[0] == '0') || !R8) return false;
  return oz::make_map_recon(map, R8, L);
}

cudaError_t launch_recon_tc(const GemmProblem& p, const oz::Layout& L, const oz::Crt& crt,
                            const oz::ReconParams& rp, const CUtensorMap& map, const int* sigA,
                            const int* sigB, int* status, cudaStream_t st) {
  using namespace oz;
  const bool cplx = dtype_is_complex(p.dtype);
  const int products = L.nmod * L.nsub, planes = products * L.nchunks;
  static thread_local ReconTcParams P;  // 2.7 KB: kept off the stack
  P = ReconTcParams{};
  P.m = L.rowsA;
  P.n = int(p.n);
  P.row_blocks = (P.m + 128 * RT_G - 1) / (128 * RT_G);
  P.total_units = (long long)P.row_blocks * P.n;
  P.planes = planes;
  P.sigA = sigA;
  P.sigB = sigB;
  P.C = p.C;
  P.ldc = p.ldc;
  P.alr = p.alpha[0];
  P.ali = p.alpha[1];
  P.ber = p.beta[0];
  P.bei = p.beta[1];
  P.fill = p.fill_mode;
  P.ro = p.fill_ro;
  P.co = p.fill_co;
  P.tile_m = BM;
  P.tile_n = cplx ? BN / 2 : BN;
  P.rp = rp;
  // weight bytes: plane k = t * nsub + s takes W_t or P - W_t (the combination
  // of combine_split or combine3 with its signs carried by the weights)
  const unsigned __int128 Pm = (unsigned __int128)crt.P_hi << 64 | crt.P_lo;
  for (int t = 0; t < L.nmod; ++t) {
    const unsigned __int128 W = (unsigned __int128)crt.w_hi[t] << 64 | crt.w_lo[t];
    const unsigned __int128 Wn = Pm - W;
    for (int s = 0; s < L.nsub; ++s) {
      unsigned __int128 vre = W, vim = 0;
      if (L.split) {
        vim = (unsigned __int128)crt.wi_hi[t] << 64 | crt.wi_lo[t];
        if (s == 1) vim = Pm - vim;
      } else if (cplx) {
        if (s == 0) {
          vre = W;
          vim = Wn;
        } else if (s == 1) {
          vre = rp.conj ? W : Wn;
          vim = rp.conj ? W : Wn;
        } else {
          vre = 0;
          vim = W;
        }
      }
      // the planes of all k-chunks of a product alike
      for (int k = t * L.nsub + s; k < planes; k += products)
        for (int o = 0; o < 16; ++o) {
          P.v[o][k] = static_cast<unsigned char>(vre >> (8 * o));
          P.v[16 + o][k] = static_cast<unsigned char>(vim >> (8 * o));
        }
    }
  }
  P.status = status;
  P.wait_limit_ns = kWaitLimitNs;
  auto run = [&](auto kern32, auto kern64) -> cudaError_t {
    const auto kern = planes <= 32 ? kern32 : kern64;
    const int smem = planes <= 32 ? ReconCfg<32>::SMEM : ReconCfg<64>::SMEM;
    const int ctas = planes <= 32 ? ReconCfg<32>::CTAS : ReconCfg<64>::CTAS;
    const cudaError_t ea = set_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
    if (ea != cudaSuccess) return ea;
    const long long grid = std::min<long long>(P.total_units, (long long)ctas * sm_count());
    kern<<<unsigned(grid), RT_THREADS, smem, st>>>(map, P);
    return cudaGetLastError();
  };
  switch (p.dtype) {
    case kC64: return run(oz_reconstruct_tc<kC64, 32>, oz_reconstruct_tc<kC64, 64>);
    case kC32: return run(oz_reconstruct_tc<kC32, 32>, oz_reconstruct_tc<kC32, 64>);
    case kR64: return run(oz_reconstruct_tc<kR64, 32>, oz_reconstruct_tc<kR64, 64>);
    default: return run(oz_reconstruct_tc<kR32, 32>, oz_reconstruct_tc<kR32, 64>);
  }
}

// At <- A k-major (op(A) = N operands); see oz_transpose
cudaError_t transpose_a(const GemmProblem& p, const oz::Layout& L, void* At, cudaStream_t st) {
  const dim3 block(32, 8);
  const dim3 grid(unsigned((p.m + 31) / 32),
                  unsigned(std::min<int64_t>((p.k + 31) / 32, 65535)));
  auto run = [&](auto tag) {
    using E = decltype(tag);
    oz::oz_transpose<E><<<grid, block, 0, st>>>(static_cast<const E*>(p.A), p.lda, int(p.m),
                                                p.k, static_cast<E*>(At), L.ldAt);
  };
  switch (p.dtype) {
    case kC64: run(double2{}); break;
    case kC32: run(float2{}); break;
    case kR64: run(double{}); break;
    default: run(float{}); break;
  }
  return cudaGetLastError();
}
}  // namespace

cudaError_t ozaki_gemm(const GemmProblem& p_in, int moduli, void* ws, size_t ws_bytes,
                       cudaStream_t st) {
  using namespace oz;
  if (!ozaki_supported(p_in)) return cudaErrorNotSupported;
  if (p_in.m <= 0 || p_in.n <= 0) return cudaSuccess;
  const Layout L = layout_of(p_in, moduli);
  if (ws_bytes < L.total || !ws) return cudaErrorInvalidValue;
  const Crt& crt = crt_of(L);
  const bool cplx = dtype_is_complex(p_in.dtype);
  char* w = static_cast<char*>(ws);
  int* sigA = reinterpret_cast<int*>(w + L.off_sigA);
  int* sigB = reinterpret_cast<int*>(w + L.off_sigB);
  int8_t* resA = reinterpret_cast<int8_t*>(w + L.off_resA);
  int8_t* resB = reinterpret_cast<int8_t*>(w + L.off_resB);
  int* R = reinterpret_cast<int*>(w + L.off_R);
  unsigned char* R8 = L.r8 ? reinterpret_cast<unsigned char*>(w + L.off_R) : nullptr;
  int* status = reinterpret_cast<int*>(w + L.off_status);
  // byte residues of C, where they apply, go to the tensor-core reconstruction
  CUtensorMap rmap;
  const bool tc_recon = p_in.k > 0 && recon_tc_plan(L, R8, &rmap);

  cudaError_t e;
  // op(A) = N: everything below reads the k-major copy At as op(A) = T
  GemmProblem p = p_in;
  if (L.at && p.k > 0) {
    p.A = w + L.off_At;
    p.lda = L.ldAt;
    p.opA = 1;
  }
  const bool dbl = dtype_is_double(p.dtype);
  const int onepass = onepass_operands(L, p);
  double* ssq = reinterpret_cast<double*>(w + L.off_ssq);
  int* oplist = reinterpret_cast<int*>(w + L.off_list);
  phase_mark(0, false, st);
  if (L.at && p.k > 0) {
    phase_mark(15, false, st);
    if ((e = transpose_a(p_in, L, w + L.off_At, st)) != cudaSuccess) return e;
    phase_mark(15, true, st);
  }
  // row exponents (the norms of operands read in place first, alone: beside the
  // slicing they measured slower)
  if (p.k > 0) {
    phase_mark(16, false, st);
    if (L.mn && L.mnB) cudaMemsetAsync(status, 0, sizeof(int), st);
    auto exponents = [&](auto tag) {
      using TIn = decltype(tag);
      scale_in_place<TIn>(L, crt, p, cplx, sigA, sigB, resA, resB, st);
      if (onepass)
        launch_row_scale<TIn, kEstimate>(L, crt, p, cplx, sigA, sigB, ssq, oplist, status, st);
      else
        launch_row_scale<TIn, kExact>(L, crt, p, cplx, sigA, sigB, ssq, oplist, status, st);
    };
    if (dbl)
      exponents(double{});
    else
      exponents(float{});
    phase_mark(16, true, st);
  } else {
    cudaMemsetAsync(sigA, 0, sizeof(int) * L.rowsA, st);
    cudaMemsetAsync(sigB, 0, sizeof(int) * L.rowsB, st);
    cudaMemsetAsync(status, 0, sizeof(int), st);
  }
  // byte residues are stored, not accumulated: every element the
  // reconstruction reads is written by the GEMM (k = 0: there is none)
  if (!L.r8 || p.k <= 0)
    cudaMemsetAsync(R, 0, (L.r8 ? 1 : sizeof(int)) * size_t(L.nmod) * L.nsub * L.planeR, st);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if (p.k <= 0) {
    phase_mark(0, true, st);
    phase_mark(1, false, st);
    phase_mark(1, true, st);
  } else {
    // with one-pass scaling the slicer also sums the rows' scaled squares
    double* sums = onepass ? ssq : nullptr;
    auto slice = [&](int which) {
      if (dbl)
        slice_operands<double>(L, crt, p, cplx, sigA, sigB, resA, resB, which, st, sums);
      else
        slice_operands<float>(L, crt, p, cplx, sigA, sigB, resA, resB, which, st, sums);
    };
    CUtensorMap mapA, mapB;
    if (!make_map(&mapA, resA, L, L.rowsA, BM) || !make_map(&mapB, resB, L, L.nb, BN))
      return cudaErrorNotSupported;
    GemmParams g{};
    g.m = L.rowsA;
    g.nb = L.nb;
    g.kblocks = int(L.kp / BKB);
    g.nchunks = L.nchunks;
    // equal chunks (each within the exact INT32 bound): equal work units
    g.chunk_blocks = std::max(1, (g.kblocks + g.nchunks - 1) / std::max(1, g.nchunks));
    g.group = residue_layout(L, 1).G;
    g.kc_blocks = int(residue_layout(L, 1).kc / BKB);
    g.nmod = L.nmod * L.nsub;
    g.nsub = L.nsub;
    g.tiles_m = (L.rowsA + BM - 1) / BM;
    g.tiles_n = (L.nb + BN - 1) / BN;
    g.total_units = g.nmod * g.nchunks * g.tiles_m * g.tiles_n;
    g.R = R;
    g.R8 = R8;
    g.ldr = int(L.ldR);
    g.rplane = L.planeR;
    g.status = status;
    g.wait_limit_ns = kWaitLimitNs;
    g.stall_test = 0;
    if (const char* v = std::getenv("SPLAB_OZAKI_STALL_TEST")) {
      // test hook for the failure path: no copies are issued, every wait runs
      // into a 50 ms bound, the kernel reports SPLAB_ERR_TIMEOUT and returns ("2": only
      // calls with beta = 0, such as the first k-chunk of streamed operands)
      if (v[0] == '1' || (v[0] == '2' && p.beta[0] == 0.0 && p.beta[1] == 0.0)) {
        g.stall_test = 1;
        g.wait_limit_ns = 50000000ull;
      }
    }
    // short units (few k-blocks): two epilogue warps per lane quarter
    g.epi_split = g.chunk_blocks < 128 ? 2 : 1;
    if (const char* v = std::getenv("SPLAB_OZAKI_EPI_SPLIT")) {
      if (v[0] == '1') g.epi_split = 1;
      if (v[0] == '2') g.epi_split = 2;
    }
    for (int t = 0; t < L.nmod; ++t) {
      g.p[t] = crt.p[t];
      const ModMagic mm = make_mod_magic(crt.p[t]);
      g.c16[t] = mm.c16;
      g.off[t] = mm.off;
      g.M[t] = mm.M;
    }
    const char* gk = std::getenv("SPLAB_OZAKI_GEMM");
    const bool pair = !(gk && gk[0] == '1');  // "1sm" selects the single-CTA kernel
    CUtensorMap mapA2, mapB2;
    // pair tile 256 x 512 (one A tile for two MMAs, one 512-column accumulator drained
    // once per unit) or the double-buffered 256 x 256 one (SPLAB_OZAKI_NT=1|2 overrides)
    int nt = L.nt;
    if (const char* v = std::getenv("SPLAB_OZAKI_NT")) {
      if (v[0] == '1') nt = 1;
      if (v[0] == '2') nt = 2;
    }
    const int tile_nb = 256 * nt;
    if (pair) {
      g.tiles_m = (L.rowsA + 255) / 256;
      g.tiles_n = (L.nb + tile_nb - 1) / tile_nb;
      g.total_units = g.nmod * g.nchunks * g.tiles_m * g.tiles_n;
      if (p.fill_mode != 0) {
        // compute only the pair tiles that cover an element the reconstruction
        // writes: its tiles are BM x (BN/2 complex | BN real) of C; a pair tile
        // covers rows r0 .. r1-1 and columns b0 .. b1-1 of C (B rows = columns)
        const int rt_m = BM, rt_n = cplx ? BN / 2 : BN;
        std::vector<int> act;
        for (int tn = 0; tn < g.tiles_n; ++tn)
          for (int tm = 0; tm < g.tiles_m; ++tm) {
            const int64_t r0 = int64_t(tm) * 256, r1 = std::min<int64_t>(r0 + 256, L.rowsA);
            const int64_t b0 = int64_t(tn) * tile_nb, b1 = std::min<int64_t>(b0 + tile_nb, L.nb);
            bool on = false;
            for (int64_t ti = (r0 / rt_m) * rt_m; ti < r1 && !on; ti += rt_m)
              for (int64_t tj = (b0 / rt_n) * rt_n; tj < b1 && !on; tj += rt_n)
                on = tile_is_active(p.fill_mode, ti, tj, std::min<int64_t>(rt_m, p.m - ti),
                                    std::min<int64_t>(rt_n, p.n - tj), p.fill_ro, p.fill_co);
            if (on) act.push_back(tm + tn * g.tiles_m);
          }
        if (act.empty()) act.push_back(0);  // keep the launch well formed
        int* dtiles = reinterpret_cast<int*>(w + L.off_tiles);
        if ((e = cudaMemcpyAsync(dtiles, act.data(), sizeof(int) * act.size(),
                                 cudaMemcpyHostToDevice, st)) != cudaSuccess)
          return e;
        if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;  // host list goes away
        g.active = dtiles;
        g.n_active = int(act.size());
        g.total_units = g.nmod * g.nchunks * g.n_active;
      }
      if ((e = set_dynamic_smem(reinterpret_cast<const void*>(oz_gemm_pair<1>),
                                PairCfg<1>::SMEM)) != cudaSuccess ||
          (e = set_dynamic_smem(reinterpret_cast<const void*>(oz_gemm_pair<2>),
                                PairCfg<2>::SMEM)) != cudaSuccess)
        return e;
      if (!make_map(&mapA2, resA, L, L.rowsA, 128) || !make_map(&mapB2, resB, L, L.nb, 128))
        return cudaErrorNotSupported;
    }
    auto launch_gemm = [&]() -> cudaError_t {
      if (pair) {
        const int pairs = std::max(1, std::min(g.total_units, sm_count() / 2));
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(unsigned(2 * pairs));
        cfg.blockDim = dim3(PAIR_THREADS);
        cfg.dynamicSmemBytes = nt == 2 ? PairCfg<2>::SMEM : PairCfg<1>::SMEM;
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 2;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        return nt == 2 ? cudaLaunchKernelEx(&cfg, oz_gemm_pair<2>, mapA2, mapB2, g)
                       : cudaLaunchKernelEx(&cfg, oz_gemm_pair<1>, mapA2, mapB2, g);
      }
      const cudaError_t ea = set_dynamic_smem(reinterpret_cast<const void*>(oz_gemm), GEMM_SMEM);
      if (ea != cudaSuccess) return ea;
      const int grid = std::min(g.total_units, sm_count());
      oz_gemm<<<grid, GEMM_THREADS, GEMM_SMEM, st>>>(mapA, mapB, g);
      return cudaGetLastError();
    };

    phase_mark(17, false, st);
    slice(1);
    phase_mark(17, true, st);
    phase_mark(18, false, st);
    slice(2);
    phase_mark(18, true, st);
    if (onepass) {
      phase_mark(19, false, st);
      if (dbl)
        onepass_fixup<double>(L, crt, p, cplx, sigA, sigB, resA, resB, ssq, oplist, onepass,
                              st);
      else
        onepass_fixup<float>(L, crt, p, cplx, sigA, sigB, resA, resB, ssq, oplist, onepass,
                             st);
      phase_mark(19, true, st);
    }
    phase_mark(0, true, st);
    phase_mark(1, false, st);
    phase_mark(3, false, st);
    if ((e = launch_gemm()) != cudaSuccess) return e;
    phase_mark(3, true, st);
    phase_mark(1, true, st);
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return e;

  phase_mark(2, false, st);
  ReconParams rp = make_recon(crt);
  rp.conj = p.opA == 2 ? 1 : 0;
  // threads along the rows of C, one block row covering all of them (no
  // partial second pass), blocks along the columns (grid-stride beyond 65535)
  const int threads = 256;
  const unsigned gy = unsigned(std::min<int64_t>(p.n, 65535));
  const unsigned gx = unsigned(std::max<int64_t>(1, (p.m + threads - 1) / threads));
  const bool fixed =
      cplx ? L.split : L.nmod == (dbl ? kDefaultModuli : kDefaultModuliFloat);
  if (tc_recon) {
    if ((e = launch_recon_tc(p, L, crt, rp, rmap, sigA, sigB, status, st)) != cudaSuccess)
      return e;
    phase_mark(2, true, st);
    return cudaGetLastError();
  }
  auto recon = [&](auto kern, const auto* Rsrc) {
    kern<<<dim3(gx, gy), threads, 0, st>>>(Rsrc, L.rowsA, int(p.n), L.planeR, L.ldR,
                                           R8 ? L.nchunks : 1, sigA, sigB, p.C, p.ldc,
                                           p.alpha[0], p.alpha[1], p.beta[0], p.beta[1],
                                           p.fill_mode, p.fill_ro, p.fill_co, BM,
                                           cplx ? BN / 2 : BN, rp);
  };
  using u8 = unsigned char;
  // the default modulus counts run a fully unrolled reconstruction
  auto by_dtype = [&](auto rt_tag, const auto* Rsrc) {
    using RT = decltype(rt_tag);
    switch (p.dtype) {
      case kC64:
        fixed ? recon(oz_reconstruct<kC64, RT, kSplitCount>, Rsrc)
              : recon(oz_reconstruct<kC64, RT, 0>, Rsrc);
        break;
      case kC32:
        fixed ? recon(oz_reconstruct<kC32, RT, kSplitCountFloat>, Rsrc)
              : recon(oz_reconstruct<kC32, RT, 0>, Rsrc);
        break;
      case kR64:
        fixed ? recon(oz_reconstruct<kR64, RT, kDefaultModuli>, Rsrc)
              : recon(oz_reconstruct<kR64, RT, 0>, Rsrc);
        break;
      default:
        fixed ? recon(oz_reconstruct<kR32, RT, kDefaultModuliFloat>, Rsrc)
              : recon(oz_reconstruct<kR32, RT, 0>, Rsrc);
        break;
    }
  };
  if (R8)
    by_dtype(u8{}, R8);
  else
    by_dtype(int{}, R);
  phase_mark(2, true, st);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  return cudaSuccess;
}

OzakiShape ozaki_shape(const GemmProblem& p) {
  const oz::Layout L = oz::layout_of(p, 0);
  return {oz::gemm_model_us(L, p.m, p.n, L.nchunks, L.nt, oz::sm_count() / 2) * 1e-6, L.r8};
}

int* ozaki_status_ptr(const GemmProblem& p, int moduli, void* ws) {
  return reinterpret_cast<int*>(static_cast<char*>(ws) + oz::layout_of(p, moduli).off_status);
}

int ozaki_status(const GemmProblem& p, int moduli, void* ws, cudaStream_t st) {
  const oz::Layout L = oz::layout_of(p, moduli);
  int h = 0;
  cudaMemcpyAsync(&h, static_cast<char*>(ws) + L.off_status, sizeof(int), cudaMemcpyDeviceToHost,
                  st);
  cudaStreamSynchronize(st);
  return h;
}

}  // namespace splab
