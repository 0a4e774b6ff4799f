"""The division by a launch's constants (host.cuh, Divisor) is the integer division for every 32-bit dividend: edges of the
range and of every quotient's step, for divisors of all sizes, on the CPU with the header's own text."""

import shutil
import subprocess
from pathlib import Path

import pytest

HEADER = Path(__file__).resolve().parents[1] / "foldjax_b200" / "csrc" / "host.cuh"

PROGRAM = """
#include <cstdint>
#include <cstdio>
#include <initializer_list>
#define __host__
#define __device__
#define __forceinline__ inline
%s
static uint32_t state = 12345;
static uint32_t next() { return state = state * 1664525u + 1013904223u; }
int main() {
  long long wrong = 0;
  auto check = [&](uint32_t by) {
    const Divisor d(by);
    auto one = [&](uint32_t x) { wrong += d.quotient(x) != x / by; };
    for (uint32_t x : {0u, 1u, by - 1, by, by + 1, 0x7fffffffu, 0x80000000u, 0xfffffffeu, 0xffffffffu}) one(x);
    for (int i = 0; i < 60; ++i) {
      const uint32_t x = next() >> (i %% 32), multiple = x / by * by;
      one(x);
      one(multiple);
      one(multiple - 1);  // (of nothing: the largest dividend)
    }
  };
  for (uint32_t by = 1; by <= 70000; ++by) check(by);
  for (int bit = 17; bit < 32; ++bit)
    for (int e = -2; e <= 2; ++e) check((1u << bit) + e);
  for (int i = 0; i < 20000; ++i) check(next() | 1u << 16);
  check(0xffffffffu);
  printf("%%lld", wrong);
}
"""


def test_quotients(tmp_path):
    compiler = shutil.which("g++") or shutil.which("c++")
    if compiler is None:
        pytest.skip("no C++ compiler")
    text = HEADER.read_text()
    start = text.index("struct Divisor {")
    source, program = tmp_path / "divisor.cpp", tmp_path / "divisor"
    source.write_text(PROGRAM % text[start:text.index("\n};", start) + 3])
    subprocess.run([compiler, "-std=c++17", "-O2", "-o", str(program), str(source)], check=True)
    assert subprocess.run([str(program)], check=True, capture_output=True, text=True).stdout == "0"
