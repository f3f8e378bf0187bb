// Host check of the k-chunks of host-resident operands (stream_chunks.hpp).
#include <cstdio>

#include "../../spla_b200/csrc/host/stream_chunks.hpp"

using namespace spla;

static int failures = 0;
#define CHECK(c)                                        \
  do {                                                  \
    if (!(c)) {                                         \
      std::printf("line %d: %s\n", __LINE__, #c);       \
      ++failures;                                       \
    }                                                   \
  } while (0)

int main() {
  const int64_t edge = 2048;
  const int64_t sizes[] = {1, 17, 64, 256, 1000, 4096, 20000};
  const int64_t ks[] = {1, 63, 64, 65, 256, 4100, 50000, 250000, 3000001};
  for (int64_t m : sizes)
    for (int64_t n : sizes)
      for (int64_t k : ks)
        for (int64_t elem : {4, 8, 16}) {
          const int64_t most = longest_chunk(m, n, k, edge);
          for (bool fp64 : {false, true}) {
            const int64_t c_bytes = elem * m * n;
            const int64_t kc = stream_chunk(m, n, k, edge, elem * (m + n), c_bytes, fp64);
            CHECK(kc >= 1 && kc <= most && most <= k);
            CHECK(kc == k || kc % 64 == 0);
            // a float C is rounded once per chunk: no more chunks than the buffers need
            if (!fp64) CHECK(kc == most);
            // every chunk passes over C: a cut one brings as many bytes
            if (kc < most) CHECK(kc * elem * (m + n) >= c_bytes);
          }
        }
  // one copy in eight is not hidden
  CHECK(stream_chunk(256, 256, 50000, edge, 16 * 512, 16 * 65536, true) == 6272);
  CHECK(stream_chunk(256, 256, 50000, edge, 8 * 512, 8 * 65536, false) == 50000);
  CHECK(stream_chunk(8192, 8192, 512, edge, 16 * 16384, int64_t(16) << 26, true) == 512);
  std::printf(failures ? "FAILED\n" : "OK\n");
  return failures != 0;
}
