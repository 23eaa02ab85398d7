"""The pieces of gn_op_gemm_nt_static, on the CPU: for every size within the documented limit the plan ends, covers the product and fits."""
import os
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r'''
#include <cstdio>
#include "goneuron_b200/csrc/static_pieces.cuh"
using namespace gn;
static long bad = 0, seen = 0, walked = 0;
static void check(long M, long N, long K) {
  const long limit = 4L << 20;
  if (M <= 0 || N <= 0 || K <= 0 || (M + N) * ((K + 7) / 8 * 8 + 1) > limit) return;
  const StaticPieces p = static_pieces(M, N, K, limit); seen++; walked += p.k < K;
  const bool ok = p.m >= 1 && p.m <= M && p.n >= 1 && p.n <= N && p.k >= 1 && p.k <= K && (p.k == K || p.k % 32 == 0) && static_pass_floats(p.m, p.n, p.k) <= limit;
  if (!ok && bad++ < 5) std::printf("bad %ld %ld %ld -> %ld %ld %ld\\n", M, N, K, p.m, p.n, p.k);
}
int main() {
  const long limit = 4L << 20;
  for (long M = 1; M <= 40; M++) for (long N = 1; N <= 40; N++) { const long top = limit / (M + N); for (long K = top - 80; K <= top + 8; K++) check(M, N, K); }
  for (long K = 1; K <= 200; K++) for (long M : {1L, 2L, 3L, 5L, 100L, 4099L, 60000L, 300001L}) { const long top = limit / ((K + 7) / 8 * 8 + 1) - M; for (long N = top - 9; N <= top; N++) { check(M, N, K); check(N, M, K); } }
  // slices: side by side where their partial results fit, one after the other only where the contraction is long
  for (long M : {1L, 37L, 128L, 256L, 1000L}) for (long N : {1L, 33L, 333L, 2300L, 3900L, 9000L}) for (long K : {512L, 600L, 1000L, 1023L, 1024L, 4000L}) for (int S : {1, 2, 3, 8}) {
    if (static_pass_floats(M, N, K) > limit) continue;
    const bool room = static_pass_floats(M, (N + 3) / 4 * 4, K) - ((N + 3) / 4 * 4 - N) * ((K + 31) / 32 * 32) + S * M * N <= limit;
    const StaticSlices want = S == 1 ? StaticSlices::WHOLE : room ? StaticSlices::SIDE_BY_SIDE : K < 1024 ? StaticSlices::WHOLE : StaticSlices::ONE_BY_ONE;
    if (static_slices(S, M, N, K, limit) != want) { bad++; std::printf("slices %ld %ld %ld %d\\n", M, N, K, S); }
  }
  std::printf("%ld sizes, %ld along the contraction, %ld bad\\n", seen, walked, bad);
  return bad || seen < 10000 || !walked;
}
'''


def test_every_size_of_the_documented_limit_has_a_plan():
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        open(src, "w").write(SRC)
        subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", ROOT, src, "-o", exe])
        r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, r.stdout
