// CPU check of the split moduli of the Ozaki path's complex products (the
// host/device code of the reconstruction): j^2 = -1 modulo each, the moduli
// pairwise coprime, and random complex integers (Re, Im) with |Re|, |Im| <= P/4,
// given as u = Re + j Im and v = Re - j Im modulo every modulus, reconstructed
// within 1.5 units in the last place from byte residues and from unreduced
// sums (below 2^24). Prints "OK <cases>" on success.
#include <cstdio>
#include <random>

#include "../../spla_b200/csrc/kernels/ozaki_crt.cuh"

using namespace splab::oz;
typedef __int128 i128;

static int mod_pos(i128 x, int p) {
  const int r = int(x % p);
  return r < 0 ? r + p : r;
}
static int gcd(int a, int b) { return b ? gcd(b, a % b) : a; }

template <int N>
static long run() {
  std::mt19937_64 rng(4242 + N);
  const Crt c = make_crt_split(N);
  const ReconParams rp = make_recon(c);
  const Crt general = make_crt(N == kSplitCount ? kDefaultModuli : kDefaultModuliFloat);
  if (c.q_bits < general.q_bits) return -1;  // no less precision than the general moduli
  for (int t = 0; t < N; ++t) {
    if ((c.j[t] * c.j[t] + 1) % c.p[t] != 0) return -2;
    for (int s = 0; s < t; ++s)
      if (gcd(c.p[s], c.p[t]) != 1) return -3;
  }
  const unsigned __int128 P = ((unsigned __int128)c.P_hi << 64) | c.P_lo;
  const i128 quarter = i128(P / 4);
  auto draw = [&](int kind) -> i128 {
    if (kind == 0) return quarter - i128(rng() % 1000);
    if (kind == 1) return -quarter + i128(rng() % 1000);
    if (kind == 2) return i128(int64_t(rng() % 2001)) - 1000;
    return i128((((unsigned __int128)rng() << 64) | rng()) % (unsigned __int128)(2 * quarter + 1)) -
           quarter;
  };
  long cases = 0;
  for (int it = 0; it < 40000; ++it) {
    const i128 re = draw(it % 4), im = draw((it / 4) % 4);
    for (int bytes = 0; bytes < 2; ++bytes) {
      int rr[kMaxModuli], ri[kMaxModuli];
      for (int t = 0; t < N; ++t) {
        const int p = c.p[t], r = mod_pos(re, p), i = mod_pos(im, p);
        int u = (r + c.j[t] * i) % p, v = mod_pos(r - c.j[t] * i, p);
        if (!bytes) {
          u += p * int(rng() % ((1u << 24) / unsigned(p) - 1));
          v += p * int(rng() % ((1u << 24) / unsigned(p) - 1));
        }
        combine_split(u, v, bytes ? p : rp.off24[t], rr[t], ri[t]);
      }
      const double gr = bytes ? crt_value<N, true>(rr, rp) : crt_value<N, false>(rr, rp);
      const double gi =
          bytes ? crt_value<N, true, true>(ri, rp) : crt_value<N, false, true>(ri, rp);
      const double wr = double((long double)re), wi = double((long double)im);
      if (std::fabs(gr - wr) > std::fabs(wr) * 3.4e-16 ||
          std::fabs(gi - wi) > std::fabs(wi) * 3.4e-16) {
        printf("FAIL n=%d it=%d bytes=%d re %.17g/%.17g im %.17g/%.17g\n", N, it, bytes, gr, wr, gi,
               wi);
        return -4;
      }
      ++cases;
    }
  }
  return cases;
}

int main() {
  const long a = run<kSplitCount>(), b = run<kSplitCountFloat>();
  if (a < 0 || b < 0) {
    printf("FAIL %ld %ld\n", a, b);
    return 1;
  }
  printf("OK %ld\n", a + b);
  return 0;
}
