// How the k extent of a contraction with host-resident operands is cut into chunks:
// chunk c + 1 is copied while chunk c is contracted. Host code without dependencies.
#pragma once

#include <algorithm>
#include <cstdint>

namespace spla {

// Rows of k, of `most` at the most, in whole k-blocks of 64 (or all of k).
inline int64_t whole_blocks(int64_t rows, int64_t k) {
  rows = (std::min(rows, k) + 63) / 64 * 64;
  return std::min(rows, k);
}

// Largest chunk: four GPU tiles (edge x edge) of the larger operand, at least 256 rows.
inline int64_t longest_chunk(int64_t m, int64_t n, int64_t k, int64_t edge) {
  return whole_blocks(std::max<int64_t>(256, edge * edge * 4 / std::max<int64_t>(1, std::max(m, n))),
                      k);
}

// Chunk of the call. Only the last chunk's contraction is not hidden behind a copy, so
// calls whose products are summed in FP64 and stored as FP64 (`fp64`: DMMA with a double
// type) are cut into at least eight chunks, of 16 MB or more (m = n = 256, k = 50000
// complex double: 8.3 ms as one chunk, 7.6). Others keep the longest chunk, since C
// takes each chunk's product in its own type: a float C would round eight times instead
// of once (128 x 128 x 40000 float, relative to 64 bits: 2.5e-8 as one chunk, 3.8e-8 as
// eight; 1.6e-4 where the chunks cancel), and the Ozaki path's sums, good to 2^-57 of
// the rows' norms, would round to C's 2^-53 at every chunk (1024 x 1024 x 16000 complex
// double 10.25 ms, 9.74 in eight). A chunk brings no fewer bytes than C has, since each
// one's contraction reads and writes all of C (8192 x 8192 x 512 complex double: 5.2 ms
// as one chunk, 15.6 in chunks of 64 rows). row_bytes: bytes copied per row of k.
inline int64_t stream_chunk(int64_t m, int64_t n, int64_t k, int64_t edge, int64_t row_bytes,
                            int64_t c_bytes, bool fp64) {
  const int64_t most = longest_chunk(m, n, k, edge);
  if (!fp64) return most;
  const int64_t bytes = std::max(int64_t(16) << 20, c_bytes);
  const int64_t least = (bytes + row_bytes - 1) / row_bytes;
  return std::min(most, whole_blocks(std::max((k + 7) / 8, least), k));
}

}  // namespace spla
