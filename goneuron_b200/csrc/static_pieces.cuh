// static_pieces.cuh -- how gn_op_gemm_nt_static cuts a product whose operand planes do not fit its fixed array at once.  Plain C++.
#pragma once
#include <algorithm>

namespace gn {

// A pass over m rows of A, n rows of B and k contraction indices keeps (m + n) plane rows, padded to whole blocks of 32 indices, and
// a scale per row (B's scales start on a 16-byte boundary).
inline long static_pass_floats(long m, long n, long k) { return (m + n) * ((k + 31) / 32 * 32) + ((m + 3) & ~3L) + n; }
struct StaticPieces { long m, n, k; };
// The documented limit counts rows padded to 8 indices.  A product between the two is walked in pieces of its larger side (every output
// element is then formed as in one pass), in steps that shrink it strictly: to multiples of four as long as there are any.
// One row of each side that still does not fit is walked along the contraction, a piece's result added to the one before.
inline StaticPieces static_pieces(long M, long N, long K, long limit) {
  StaticPieces p{M, N, K};
  while (p.m + p.n > 2 && static_pass_floats(p.m, p.n, p.k) > limit) {
    long& x = p.m >= p.n ? p.m : p.n;
    x = x > 4 ? ((x + 1) / 2 + 3) & ~3L : x / 2;
  }
  if (static_pass_floats(p.m, p.n, p.k) > limit) p.k = std::max(32L, (limit - 4 - p.n) / (p.m + p.n) / 32 * 32);
  return p;
}

// How a pass whose contraction the regular entry point would cut into `splits` slices runs: side by side where the array has room for their partial
// results behind what the pass keeps, else one after the other (contractions of 1024 and more: long accumulator runs truncate more often), else whole:
// slices of a shorter contraction are cut for speed alone, and one after the other they are slower (128 x 3900 over 1000 69 us, whole 51).
enum class StaticSlices { WHOLE, SIDE_BY_SIDE, ONE_BY_ONE };
inline StaticSlices static_slices(int splits, long m, long n, long k, long limit) {
  if (splits <= 1) return StaticSlices::WHOLE;
  const long part = ((m + n) * ((k + 31) / 32 * 32) + ((m + 3) & ~3L) + ((n + 3) & ~3L));
  if (part + splits * m * n <= limit) return StaticSlices::SIDE_BY_SIDE;
  return k >= 1024 ? StaticSlices::ONE_BY_ONE : StaticSlices::WHOLE;
}

}  // namespace gn
