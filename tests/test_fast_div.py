"""CPU: division by a launch constant as a product (csrc/fast_div.cuh), which the dense stage decodes items and row offsets with: a quotient
one off would be a row of another token.  The host form of the same arithmetic, compiled with g++, against the division."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "baselinebenchmark_b200" / "csrc"
CUDA_INCLUDE = Path("/usr/local/cuda/include")

PROGRAM = r'''
#include "fast_div.cuh"
#include <cstdio>
#include <random>
using namespace moba;
static long checked = 0, wrong = 0;
static void check(int64_t d, int64_t x) {
  if (x < 0 || x > 2147483647) return;
  ++checked;
  if ((int)x / fast_div(d) != (int)(x / d)) ++wrong;
}
static void divisor(int64_t d, std::mt19937& rng) {
  if (d < 1 || d > 2147483647) return;
  for (int64_t x : {(int64_t)0, (int64_t)1, d - 1, d, d + 1, (int64_t)2147483647, (int64_t)2147483646, 2147483647 / d * d, 2147483647 / d * d - 1,
                    (int64_t)1 << 30, ((int64_t)1 << 30) - 1})
    check(d, x);
  for (int i = 0; i < 8; ++i) {
    const int64_t m = (int64_t)(rng() % (uint32_t)(2147483647 / d + 1)) * d;
    check(d, m - 1); check(d, m); check(d, m + 1); check(d, rng() & 0x7fffffff);
  }
}
int main() {
  std::mt19937 rng(1);
  for (int64_t d = 1; d <= 70000; ++d) divisor(d, rng);
  for (int k = 0; k < 31; ++k)
    for (int64_t e = -3; e <= 3; ++e) divisor(((int64_t)1 << k) + e, rng);
  for (int i = 0; i < 100000; ++i) divisor(1 + (int64_t)(rng() & 0x7ffffffe), rng);
  printf("%ld %ld\n", checked, wrong);
}
'''


@pytest.mark.skipif(shutil.which("g++") is None or not (CUDA_INCLUDE / "cuda_runtime.h").exists(),
                    reason="needs g++ and the CUDA headers")
def test_quotients(tmp_path):
    source = tmp_path / "div.cpp"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), "-I", str(CUDA_INCLUDE), str(source), "-o", str(tmp_path / "div")],
                   check=True)
    checked, wrong = map(int, subprocess.run([str(tmp_path / "div")], capture_output=True, text=True, check=True).stdout.split())
    assert checked > 5_000_000 and wrong == 0
