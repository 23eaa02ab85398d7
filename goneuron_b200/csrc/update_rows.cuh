// update_rows.cuh -- where the rank-one updates of an LSTM's clipped gradient lie.  Plain C++ as well.
#pragma once
#ifdef __CUDACC__
#define GN_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define GN_HOST_DEVICE inline
#endif

namespace gn {

// Updates are numbered in walking order.  Chunk c holds updates c * Kc .. c * Kc + Kc - 1 in rows c * stride + lead onward, zeros in its rows before and behind
// them (the last chunk may be short).
struct UpdateRows {
  long n, Kc, stride, lead, rows;                             // updates; updates and rows of a chunk; rows before its first update; all rows
  struct At { long chunk, r, k; bool update; };               // row `row` is row `r` of its chunk, counted from the chunk's first update, and holds update `k` if `update`
  GN_HOST_DEVICE At at(long row) const {
    const long chunk = row / stride, r = row - chunk * stride - lead, k = chunk * Kc + r;
    return At{chunk, r, k, r >= 0 && r < Kc && k < n};
  }
  GN_HOST_DEVICE long row_of(long k) const { return k / Kc * stride + lead + k % Kc; }
};
// All updates, in chunks of whole groups with `pad` rows of zeros before each
inline UpdateRows update_rows_of_chunks(long n, long Kc, long chunks, long group, long pad) {
  const long stride = pad + (Kc + group - 1) / group * group;
  return UpdateRows{n, Kc, stride, pad, chunks * stride};
}
// One rank's own updates, one after the other: a single chunk
inline UpdateRows update_rows_of_rank(long n) { return UpdateRows{n, n, n, 0, n}; }

}  // namespace gn
