"""The grid barrier's count modulo 2^32 (engine/barrier_count.h), compiled for
the host: around the rounds where the total of a launch's arrivals passes
2^31 and 2^32, a round is complete with its last arrival and not before, also
for CTAs that are still polling when others have arrived for the next round.
"""
import os
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include "barrier_count.h"
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
int main(int, char **argv) {
  const unsigned ctas = std::strtoul(argv[1], nullptr, 10);
  for (uint64_t total : {uint64_t(0), uint64_t(1) << 31, uint64_t(1) << 32, uint64_t(3) << 31}) {
    const uint64_t near = total / ctas;
    for (uint64_t round = near > 3 ? near - 3 : 1; round < near + 4; round++) {
      const unsigned want = static_cast<unsigned>(round) * ctas;
      // from the round before complete to all but one arrived for the next
      for (uint64_t a = (round - 1) * ctas; a < (round + 1) * ctas; a++)
        if (prgpu::arrivals_reached(static_cast<unsigned>(a), want) != (a >= round * ctas)) {
          std::printf("round %llu arrivals %llu\n", (unsigned long long)round,
                      (unsigned long long)a);
          return 1;
        }
    }
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("barrier")
    src, exe = d / "count.cc", d / "count"
    src.write_text(PROGRAM)
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-I",
                    os.path.join(ROOT, "gapbs_b200", "csrc", "engine"), str(src), "-o", str(exe)],
                   check=True)
    return str(exe)


@pytest.mark.parametrize("ctas", [2, 20, 148, 296])
def test_rounds_around_the_wrap(program, ctas):
    r = subprocess.run([program, str(ctas)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
