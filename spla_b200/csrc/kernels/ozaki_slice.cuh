// Residues of complex double rows for the split moduli (oz_slice_mma): every
// real v of a row is scaled and rounded, x = round(2^sigma v), and the two planes
// of a modulus p take Re + j Im and Re - j Im of it modulo p, one signed byte each,
// K-major.
//
// A plane's value is a digit sum: with x + 2^63 = sum_i b_i 256^i (eight unsigned
// bytes), a x = sum_i (a 256^i mod p) b_i - a 2^63 (mod p). The sums of all 32
// planes are one small integer matrix product, planes x digits by digits x
// elements, and run on the warp-level INT8 tensor instruction mma.m16n8k16
// (u8 x u8, exact s32): K = 16 are the digits of an element's two parts, M = 16
// planes, N eight elements. The sums are reduced mod p by four packed FP32
// operations per two residues (see reduce).
//
// oz_slice (ozaki.cu) forms the digit sums as FP32 chains instead: 305
// instructions per element, its FMA pipe 62 % and issue slots 67 % busy, against
// 193 here (with the sums of squares). m = n = 1024, k = 60000: 1.49 -> 1.16 ms for both operands (5.1
// TB/s read and written); k = 250000, with the sums of squares of the one-pass
// scaling, 7.3 -> 5.6 ms. It stays for the other types and for operands read in
// place, where it measured the same or faster (real double 1.11 against 1.14 ms
// at k = 100000; complex float 1.08 against 1.18 at 60000, where five of its 8
// digits would do; real float 0.63 against 1.07, 18 of 32 rows used; m-major
// 100000 x 2048 complex double 3.0 against 3.3).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#include "ozaki_crt.cuh"
#include "ozaki_layout.cuh"

namespace splab {
namespace oz {

constexpr int kSlicePlanes = 2 * kSplitCount;
static_assert(kSlicePlanes == 32, "two row tiles of 16");
constexpr int kStepReals = 128;    // reals of one row per warp step
constexpr int kSliceBlocks = 4;    // resident blocks of 4 warps per SM
constexpr int kSliceStages = 5;    // steps of a warp's ring of loads

// One plane: the weights of an element's 16 digits and the constants of its
// modulus (see reduce).
struct SliceRow {
  uint32_t w[4];   // digit weights, bytes: real part 0-3, 4-7, imaginary part 0-3, 4-7
  float np, ip;    // -p 2^-127, 2^127 / p
  int off;         // 256 p + (the digits' offset mod p)
};

// Plane of a Re + b Im modulo p.
inline SliceRow make_slice_row(int p, int a, int b) {
  SliceRow r{};
  auto mod = [p](long long v) { return int(((v % p) + p) % p); };
  unsigned char w[16];
  int c = 1;
  for (int j = 0; j < 8; ++j) {  // c = 256^j mod p
    w[j] = static_cast<unsigned char>(mod((long long)c * a));
    w[8 + j] = static_cast<unsigned char>(mod((long long)c * b));
    c = mod(256ll * c);
  }
  std::memcpy(r.w, w, 16);
  r.np = std::ldexp(-float(p), -127);
  r.ip = std::ldexp(1.0f / float(p), 127);
  int o = 1;  // 2^63 mod p
  for (int i = 0; i < 63; ++i) o = mod(2ll * o);
  r.off = 256 * p + mod(-(long long)o * (a + b));
  return r;
}

// D (16 x 8, s32) = W (16 x 16, u8) . X (16 x 8, u8). Lane (g, t) = (lane / 4,
// lane % 4) holds bytes 4 t .. 4 t + 3 of rows g and g + 8 of W and of column g of
// X, and columns 2 t, 2 t + 1 of rows g (d0, d1) and g + 8 (d2, d3) of D.
__device__ __forceinline__ void mma_digits(uint32_t (&d)[4], uint32_t w0, uint32_t w1, uint32_t x) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%7,%7,%7,%7};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(w0), "r"(w1), "r"(x), "r"(0));
}

// A SliceRow in shared memory, its constants in both halves of f32x2 operands
// (48 bytes: the quads' reads of eight rows are free of bank conflicts).
struct alignas(16) SliceRowShared {
  float np[2], ip[2];
  int off[2], pad[2];
  uint32_t w[4];
};

__device__ __forceinline__ void stage_rows(const SliceRow* row, int n, SliceRowShared* tab) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const SliceRow r = row[i];
    SliceRowShared s;
    s.np[0] = s.np[1] = r.np;
    s.ip[0] = s.ip[1] = r.ip;
    s.off[0] = s.off[1] = r.off;
    for (int k = 0; k < 4; ++k) s.w[k] = r.w[k];
    tab[i] = s;
  }
}

// A lane's constants of one row, read for every step and row tile (volatile:
// kept in registers over the loop they would cost a third of the warps).
struct LaneRow {
  unsigned long long np, ip, off;
  uint32_t w;

  __device__ __forceinline__ LaneRow(const SliceRowShared* tab, int r, int t) {
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(tab + r));
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(np), "=l"(ip) : "r"(a));
    asm volatile("ld.shared.b64 %0, [%1 + 16];" : "=l"(off) : "r"(a));
    asm volatile("ld.shared.b32 %0, [%1 + 32];" : "=r"(w) : "r"(a + 4 * t));
  }

  // A pair of digit sums (0 <= s < 2^20) to integers whose low bytes are s plus
  // the digits' offset mod p, without integer conversions: the bits of a small
  // non-negative integer v are those of the (subnormal) float v 2^-149. With
  // v = s + off, q = round(v / p) comes as 3 + q 2^-22 (ulp 2^-22 there) from one
  // FMA, off by the error of 1/p, below 0.001; taking off 3 + 256 2^-22 leaves
  // (q - 256) 2^-22, and v - (q - 256) p = r + 256 p is exact: its low byte is r,
  // |r| <= p/2 + 0.001 p, one signed byte (checked on the CPU for every modulus
  // and digit sum).
  __device__ __forceinline__ void reduce(uint32_t& a, uint32_t& b) const {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(a), "r"(b));
    v = f2_add(v, off);
    constexpr float M = 3.0f, T = 3.0f + 256.0f / 4194304.0f;
    const unsigned long long q = f2_add(f2_fma(v, ip, f2_pack(M, M)), f2_pack(-T, -T));
    const unsigned long long r = f2_fma(q, np, v);
    asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(r));
  }
};

// Position of a lane's reals in a step of 128 reals (64 elements) of a row: unit
// u = 0..3 of lane (g, t) takes real lane_real(g, t) + 8 u. Lanes t = 0, 1 take
// real, t = 2, 3 imaginary parts; even lanes an element of the unit's first column
// tile, odd lanes one of its second. Columns are assigned so that lane t of a quad
// gets the elements 16 t .. 16 t + 15 of the step for each plane.
__host__ __device__ constexpr int lane_real(int g, int t) {
  return 2 * (16 * (g >> 1) + 2 * (t & 1) + (g & 1)) + (t >> 1);
}

// Digits of a step's scaled reals y (by unit), as its column tiles take them.
struct Digits {
  uint32_t a[4], b[4];  // first and second tile of each unit

  __device__ __forceinline__ void set(const double (&y)[4], int t) {
    const bool odd = t & 1;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long x = __double2ll_rn(y[u]);
      const uint32_t lo = uint32_t(x), hi = uint32_t((unsigned long long)x >> 32) ^ 0x80000000u;
      // lane t supplies word t of a pair's digits: even lanes the low, odd lanes the
      // high word of each tile's real, half of which the neighbour holds
      const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);
      a[u] = odd ? got : lo;
      b[u] = odd ? hi : got;
    }
  }
};

// Residues of a step, written to plane 8 j + g at out + j eight (out: the step's
// first byte in plane g).
__device__ __forceinline__ void slice_step(const Digits& x, const SliceRowShared* tab, int8_t* out,
                                           int64_t eight, int g, int t) {
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const LaneRow r0(tab, 16 * m + g, t), r1(tab, 16 * m + 8 + g, t);
    uint32_t o[2][4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      uint32_t da[4], db[4];
      mma_digits(da, r0.w, r1.w, x.a[u]);
      mma_digits(db, r0.w, r1.w, x.b[u]);
      r0.reduce(da[0], da[1]);
      r0.reduce(db[0], db[1]);
      r1.reduce(da[2], da[3]);
      r1.reduce(db[2], db[3]);
      o[0][u] = pack4(da[0], da[1], db[0], db[1]);
      o[1][u] = pack4(da[2], da[3], db[2], db[3]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
      *reinterpret_cast<uint4*>(out + (2 * m + h) * eight + 16 * t) =
          make_uint4(o[h][0], o[h][1], o[h][2], o[h][3]);
  }
}

// 2^sg v: one multiplication when 2^sg is a normal double, else ldexp.
struct RowScale {
  double f;
  int sg;
  bool direct;
  __device__ __forceinline__ explicit RowScale(int s) : sg(s) {
    direct = s > -1000 && s < 1000;
    f = direct ? __longlong_as_double((long long)(s + 1023) << 52) : 1.0;
  }
  __device__ __forceinline__ void apply(double (&v)[4]) const {
    if (!direct) {  // warp-uniform
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = ldexp(v[u], sg);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] *= f;
  }
};

// An operand with k-major rows: row r at X + r ld doubles, len doubles.
struct SliceMmaParams {
  const double* X;
  int64_t ld, len;
  int rows;
  int vec;             // rows on 16-byte boundaries
  const int* sigma;
  int8_t* res;
  ResidueLayout lay;
  double* ssq;         // SSQ: each row's sum of squares of the scaled reals is added
  const int* list;     // rows list[0 .. *count - 1] instead of all (null)
  const int* count;
  int steps_per_row;
  int warps_per_row;   // 1, 2 or 4
  int run;             // steps per warp and chunk
  SliceRow row[kSlicePlanes];
};

// 16 or 8 bytes, the last of them zeros past `valid`
template <int SIZE>
__device__ __forceinline__ void cp_async_bytes(uint32_t dst, const void* src, int valid) {
  if constexpr (SIZE == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(valid));
}

// Place of real l of a step in its stage: the element index XOR-swizzled in groups
// of four, so that a unit's reads (runs of 8 consecutive reals, 32 apart) are free
// of bank conflicts. The units differ in bits 2 and 3 of the element index, which
// are no source of the swizzle: unit u lies at the place of unit 0 XOR 8 u.
__device__ __forceinline__ int stage_place(int l) {
  const int e = l >> 1;
  return 2 * (e ^ (((e >> 4) & 3) << 2)) + (l & 1);
}

// Blocks of 4 warps walk chunks of rows: a segment of `run` x `wpr` consecutive
// steps of each of 4 / wpr rows, wpr warps to a row, interleaved, one step of 128
// reals each at a time. Each warp keeps the copies of its next four steps in
// flight in a ring of its own in shared memory, so that the loads do not depend on
// the registers the residues leave, and has the next step's digits ready (a chain
// of conversions and a shuffle) when it starts on one. Rows of two or three steps
// take two warps each. With SSQ one atomic per warp and segment. Four
// blocks per SM: with more, the few registers spilled per step miss the L1 that
// the stream of loads and stores goes through (60 % slower).
template <bool SSQ>
__global__ void __launch_bounds__(128, kSliceBlocks)
    oz_slice_mma(const __grid_constant__ SliceMmaParams P) {
  __shared__ SliceRowShared tab[kSlicePlanes];
  __shared__ __align__(16) double ring[4][kSliceStages][kStepReals];
  constexpr int STEP = kStepReals * int(sizeof(double));  // bytes
  constexpr int OUT = kStepReals / 2;                     // residues per plane and step
  stage_rows(P.row, kSlicePlanes, tab);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int wpr = P.warps_per_row, rows_per = 4 / wpr;
  const int nrows = P.list ? *P.count : P.rows;
  const int segs = (P.steps_per_row + P.run * wpr - 1) / (P.run * wpr);
  const int64_t chunks = int64_t((nrows + rows_per - 1) / rows_per) * segs;
  const ResidueLayout& lay = P.lay;
  const uint32_t ring0 = static_cast<uint32_t>(__cvta_generic_to_shared(&ring[warp][0][0]));
  const int place = stage_place(lane_real(g, t));

  for (int64_t chunk = blockIdx.x; chunk < chunks; chunk += gridDim.x) {
    const int rg = int(chunk / segs), seg = int(chunk - int64_t(rg) * segs);
    const int ri = rg * rows_per + warp / wpr, s0 = seg * P.run * wpr + warp % wpr;
    const int n = ri < nrows ? min((P.steps_per_row - s0 + wpr - 1) / wpr, P.run) : 0;
    if (n <= 0) continue;  // warp-uniform
    const int row = P.list ? P.list[ri] : ri;
    const double* x = P.X + int64_t(row) * P.ld + int64_t(s0) * kStepReals;
    int64_t left = P.len - int64_t(s0) * kStepReals;  // reals from x to the row's end
    int64_t e = int64_t(s0) * OUT;
    int8_t* const out = P.res + lay.plane(g) + int64_t(row) * lay.row;
    const RowScale scale(P.sigma[row]);
    // copies of step i into its stage; reals past the row's end read as zeros
    auto fetch = [&](int i) {
      if (i < n) {
        const uint32_t dst = ring0 + uint32_t(i % kSliceStages) * STEP;
        if (P.vec && left >= kStepReals) {
#pragma unroll
          for (int c = 0; c < 2; ++c)
            cp_async_bytes<16>(dst + stage_place(2 * lane + 64 * c) * 8, x + 2 * lane + 64 * c, 16);
        } else {  // one real per copy: unaligned rows, and the ragged last step
#pragma unroll 1
          for (int l = lane; l < kStepReals; l += 32)
            cp_async_bytes<8>(dst + stage_place(l) * 8, l < left ? x + l : P.X, l < left ? 8 : 0);
        }
        x += wpr * kStepReals;
        left -= wpr * kStepReals;
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int i = 0; i < kSliceStages - 1; ++i) fetch(i);
    double acc = 0.0;
    Digits cur, next;
    auto digits = [&](int i, Digits& d) {  // of step i, after the ring's next copies
      asm volatile("cp.async.wait_group %0;" ::"n"(kSliceStages - 2) : "memory");
      __syncwarp();  // all lanes' copies of this step; their reads of the last one
      fetch(i + kSliceStages - 1);
      const double* v = &ring[warp][i % kSliceStages][0];
      double y[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) y[u] = v[place ^ (8 * u)];
      scale.apply(y);
      if constexpr (SSQ) acc += fma(y[0], y[0], y[1] * y[1]) + fma(y[2], y[2], y[3] * y[3]);
      d.set(y, t);
    };
    digits(0, cur);
    for (int i = 0; i < n; ++i) {
      if (i + 1 < n) digits(i + 1, next);
      slice_step(cur, tab, out + lay.at(e), lay.eight(), g, t);
      cur = next;
      e += wpr * OUT;
    }
    if constexpr (SSQ) {
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) atomicAdd(P.ssq + row, acc);
    }
    __syncwarp();  // the ring is refilled by the next chunk
  }
}

}  // namespace oz
}  // namespace splab
