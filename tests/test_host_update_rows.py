"""The rows of an LSTM's updates, on the CPU: what the gather finds in a row is what the placing kernel puts there, every update has one row, and a rank's own
updates lie one after the other."""
import os
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r'''
#include <cstdio>
#include <vector>
#include "goneuron_b200/csrc/update_rows.cuh"
using namespace gn;
static long bad = 0, seen = 0;
static void check(const UpdateRows& u, long chunks) {
  std::vector<int> rows(u.n, 0); seen++;
  for (long row = 0; row < u.rows; row++) {
    const UpdateRows::At at = u.at(row);
    bool ok = at.chunk >= 0 && at.chunk < chunks && at.r >= -u.lead && at.r < u.stride - u.lead;
    if (at.update) { ok = ok && at.k >= 0 && at.k < u.n && at.k / u.Kc == at.chunk && u.row_of(at.k) == row; if (ok) rows[at.k]++; }
    if (!ok && bad++ < 5) std::printf("row %ld of n %ld Kc %ld stride %ld lead %ld\n", row, u.n, u.Kc, u.stride, u.lead);
  }
  for (long k = 0; k < u.n; k++) if (rows[k] != 1 && bad++ < 5) std::printf("update %ld of %ld in %d rows\n", k, u.n, rows[k]);
}
int main() {
  for (long T : {1L, 3L, 13L, 64L}) for (long B : {1L, 2L, 10L, 21L, 64L}) for (long W : {1L, 2L, 4L, 10L}) {
    const long chunk = (B + W - 1) / W, chunks = (B + chunk - 1) / chunk, n = B * T;
    const UpdateRows u = update_rows_of_chunks(n, chunk * T, chunks, 128, 128);
    check(u, chunks);
    for (long c = 0; c < chunks; c++) for (long r = 0; r < 128; r++) bad += u.at(c * u.stride + r).update;      // rows of zeros first
    const UpdateRows own = update_rows_of_rank(n);
    check(own, 1);
    for (long k = 0; k < n; k++) bad += own.row_of(k) != k || own.at(k).k != k || !own.at(k).update;
    // two ranks' rows, each gathered by itself and put one behind the other, are the updates in walking order
    if (B % 2 == 0) { const UpdateRows half = update_rows_of_rank(n / 2); for (int rank = 0; rank < 2; rank++) for (long k = 0; k < n / 2; k++) bad += rank * half.rows + half.row_of(k) != rank * (n / 2) + k; }
  }
  std::printf("%ld layouts, %ld bad\n", seen, bad);
  return bad != 0;
}
'''


def test_every_update_has_its_row():
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        open(src, "w").write(SRC)
        subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", ROOT, src, "-o", exe])
        r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, r.stdout
