// Layout of the Ozaki path's residue planes and the packed FP32 helpers of its
// slicers.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

namespace splab {
namespace oz {

// Where the residues of an operand lie. Planes come in groups of G (1, 2, 4 or 8)
// that lie side by side in pieces of kc = 2^shift bytes: byte e of row r and plane q
// at (q / G) group + r row + at(e) + (q % G) kc. With G = 1 a row is one piece
// (shift 62, row = its length).
struct ResidueLayout {
  int64_t group, row, kc;
  int shift, G;

  // byte e of a row, in the group's first plane
  __host__ __device__ int64_t at(int64_t e) const {
    return (e >> shift) * (G * kc) + (e & ((int64_t(1) << shift) - 1));
  }
  __host__ __device__ int64_t plane(int q) const { return q / G * group + q % G * kc; }
  // from plane q to plane q + 8
  __host__ __device__ int64_t eight() const { return 8 / G * group; }
};

// Two floats in one 64-bit register for the packed FP32 instructions of
// sm_100 (fma/add .f32x2: one instruction, two lanes of work).
__host__ __device__ __forceinline__ unsigned long long f2_pack(float lo, float hi) {
#ifdef __CUDA_ARCH__
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
#else
  uint32_t a, b;
  std::memcpy(&a, &lo, 4);
  std::memcpy(&b, &hi, 4);
  return (static_cast<unsigned long long>(b) << 32) | a;
#endif
}
__device__ __forceinline__ void f2_unpack(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b,
                                                     unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long f2_mul(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long f2_add(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Bytes 0 of a, b, c, d
__device__ __forceinline__ uint32_t pack4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}
__device__ __forceinline__ uint32_t pack4(float a, float b, float c, float d) {
  return pack4(__float_as_uint(a), __float_as_uint(b), __float_as_uint(c), __float_as_uint(d));
}

}  // namespace oz
}  // namespace splab
