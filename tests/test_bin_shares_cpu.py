"""Shares of crowded bins (csrc/bin_shares.cuh) on the CPU, up to the largest record
number: the shares of a bin are its records, each once, no share or step of a
thread wraps, and the further shares fit the histogram's room."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))

CHECK = r"""
#include "bin_shares.cuh"
#include <cstdio>
using namespace arb;

int main() {
  const int64_t top = 0xffffffffLL;
  const int64_t counts[] = {1, 511, 512, 513, 4097, 1000003, 3000000000LL, top - 1025, STAGED_ROWS, top - 1, top};
  const int64_t bins[] = {1, 2, 7, 600, 1215, 1216, 32768, 1000000};
  for (int64_t nq : counts)
    for (int64_t nb : bins) {
      const uint32_t share = bin_share(nb, nq);
      if (share < 512 || (int64_t)share + 1024 > top) return 1;
      // bins that end at the last record, hold the mean, or hold all of them
      const int64_t sizes[] = {1, nq / nb, share, (int64_t)share + 1, 2 * (int64_t)share, nq};
      for (int64_t n : sizes) {
        if (n < 1 || n > nq) continue;
        const int64_t ends[] = {n, nq};
        for (int64_t end : ends) {
          const uint32_t begin = (uint32_t)(end - n), more = bin_more_shares((uint32_t)n, share);
          int64_t at = begin;
          for (int64_t p = 0; p <= more; ++p) {
            const uint32_t t0 = bin_first(begin, (uint32_t)p, share), t1 = bin_end(t0, (uint32_t)end, share);
            if (t0 != at || t1 <= t0 || t1 - t0 > share) {
              std::printf("nq %lld bins %lld n %lld end %lld part %lld: %u to %u\n", (long long)nq, (long long)nb,
                          (long long)n, (long long)end, (long long)p, t0, t1);
              return 2;
            }
            int64_t steps = 0;  // of the last of 256 threads, as the adjoint counts
            for (uint32_t t = t0 + 255; t - t0 < t1 - t0; t += 256) ++steps;
            if (steps != (int64_t)(t1 - t0) / 256) return 5;
            if (nq <= STAGED_ROWS && t1 > 0xffffffffu - 512) return 6;  // and the evaluators: no record past the end wraps
            at = t1;
          }
          if (at != end) return 3;
        }
      }
      // every record in full further shares: the list's words behind the first two
      if (2 + 2 * (nq / share) > 16 * nb + 1 && nq / share > 0) return 4;
    }
  return 0;
}
"""


def test_shares_cover_every_bin(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "shares.cpp"
    src.write_text(CHECK)
    exe = tmp_path / "shares"
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", os.path.join(ROOT, "arbinterp_gb300", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout)
