// CPU check of the residue product of oz_slice_mma (ozaki_slice.cuh): for both
// planes of every split modulus and both signs of j the digit weights and constants
// of make_slice_row give, for random pairs of scaled integers, the plane's value
// modulo p as one signed byte; and for every digit sum the weights can give, the
// FP32 reduction (fmaf and additions as on the device) leaves a congruent byte.
// Also the places of a step: the lanes' reals are a permutation of the step's 128,
// and a lane's units and quads hold the elements the stores write. Prints "OK
// <cases>".
#include <cmath>
#include <cstdio>
#include <random>

#include "../../spla_b200/csrc/kernels/ozaki_slice.cuh"

using namespace splab::oz;

static float bits_float(int b) {
  float f;
  std::memcpy(&f, &b, 4);
  return f;
}
static int float_bits(float f) {
  int b;
  std::memcpy(&b, &f, 4);
  return b;
}

// The device's reduction of a digit sum: the low byte
static signed char reduce(const SliceRow& r, int s) {
  const float v = bits_float(s + r.off), T = 3.0f + 256.0f / 4194304.0f;
  volatile float q = std::fmaf(v, r.ip, 3.0f);
  q = q - T;
  return static_cast<signed char>(float_bits(std::fmaf(q, r.np, v)) & 255);
}

static long cases = 0;

static bool check(int p, int a, int b, std::mt19937_64& rng) {
  const SliceRow r = make_slice_row(p, a, b);
  unsigned char w[16];
  std::memcpy(w, r.w, 16);
  long hi = 0;
  for (int k = 0; k < 16; ++k) hi += 255L * w[k];
  if (hi + r.off >= 1 << 21) return printf("FAIL range p=%d\n", p), false;
  for (long s = 0; s <= hi; ++s) {
    const int byte = reduce(r, int(s));
    if (((byte - s - r.off) % p + p) % p != 0)
      return printf("FAIL p=%d s=%ld byte %d\n", p, s, byte), false;
    ++cases;
  }
  for (int it = 0; it < 2000; ++it) {
    const int sh = int(rng() % 62);
    const long long x[2] = {(long long)rng() >> (1 + sh), (long long)rng() >> (1 + int(rng() % 62))};
    int v = 0;
    for (int h = 0; h < 2; ++h) {
      const unsigned long long u = (unsigned long long)x[h] ^ 0x8000000000000000ull;
      for (int j = 0; j < 8; ++j) v += int(w[8 * h + j]) * int((u >> (8 * j)) & 255);
    }
    const __int128 want = __int128(a) * x[0] + __int128(b) * x[1];
    if (int(((want - reduce(r, v)) % p + p) % p) != 0)
      return printf("FAIL p=%d a=%d b=%d x=%lld %lld\n", p, a, b, x[0], x[1]), false;
    ++cases;
  }
  return true;
}

static bool places() {
  int seen[kStepReals] = {0};
  for (int g = 0; g < 8; ++g)
    for (int t = 0; t < 4; ++t)
      for (int u = 0; u < 4; ++u) {
        const int l = lane_real(g, t) + 8 * u;
        if (l < 0 || l >= kStepReals || seen[l]++) return false;
        // column g of tile t & 1 of unit u: byte (g & 1) + 2 (t & 1) of word u of quad
        // lane g / 2, whose 16 bytes start at element 16 (g / 2)
        if (l / 2 != 16 * (g / 2) + 4 * u + 2 * (t & 1) + (g & 1) || l % 2 != t / 2) return false;
      }
  return true;
}

int main() {
  std::mt19937_64 rng(7);
  const Crt c = make_crt_split(kSplitCount);
  for (int t = 0; t < c.n; ++t)
    for (int sign : {-1, 1})
      if (!check(c.p[t], 1, sign * c.j[t], rng) || !check(c.p[t], -1, sign * c.j[t], rng)) return 1;
  if (!places()) return printf("FAIL places\n"), 1;
  printf("OK %ld\n", cases);
  return 0;
}
