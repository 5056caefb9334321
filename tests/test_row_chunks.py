"""The positions that a pulled level of a search takes of a row (row_chunks.h),
compiled for the host: rows that end at the last positions 32 bits hold are
walked once and to their end, as any other."""

import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "pg_warren_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "row_chunks.h"
int main(int argc, char** argv) {
  const uint32_t lo = strtoull(argv[1], 0, 10), hi = strtoull(argv[2], 0, 10);
  for (uint32_t q = 0; q < 8; q++)
    if (wc::in_row(lo, hi, q)) printf("%llu ", (unsigned long long)lo + q);
  int chunks = 0;
  if (hi - lo > 8)
    wc::each_chunk(lo + 8, hi, 32, [&](uint64_t e0) {
      for (uint64_t e = e0; e < e0 + 32 && e < hi; e++) printf("%llu ", (unsigned long long)e);
      return ++chunks == 64;
    });
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    where = tmp_path_factory.mktemp("row_chunks")
    source, binary = where / "rows.cpp", where / "rows"
    source.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-I", CSRC, str(source), "-o", str(binary)], check=True)
    return str(binary)


LAST = 2 ** 32 - 1


@pytest.mark.parametrize("lo,hi", [
    (0, 0), (0, 5), (7, 15), (7, 16), (100, 172), (LAST, LAST), (LAST - 1, LAST),
    (LAST - 5, LAST), (LAST - 8, LAST), (LAST - 9, LAST), (LAST - 40, LAST), (LAST - 41, LAST),
    (LAST - 75, LAST - 3), (LAST - 200, LAST - 31), (LAST - 200, LAST - 32)])
def test_a_row_is_walked_once(program, lo, hi):
    out = subprocess.run([program, str(lo), str(hi)], check=True, capture_output=True, text=True)
    assert [int(p) for p in out.stdout.split()] == list(range(lo, hi))
