"""Which earlier sweep of a round a brick waits for (csrc/oct_wait.h, the function the
round kernel calls), compiled for the CPU: a round of one sweep and a round of full
sweeps own no per-brick bits, so their bricks must not read any (a null pointer
here); for random rounds the answer is the restated definition's."""
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "oct_wait.h"
// rows of "osw first full bits" (bits -1: no array) -> the sweep waited for
int main() {
  int osw, first, bits;
  unsigned full;
  while (std::scanf("%d %d %u %d", &osw, &first, &full, &bits) == 4) {
    uint8_t b[3] = {0, (uint8_t)bits, 0};
    std::printf("%d\n", pdfs::oct_latest(osw, first, full, bits < 0 ? nullptr : b, 1));
  }
}
"""


@pytest.fixture(scope="module")
def latest(tmp_path_factory):
    d = tmp_path_factory.mktemp("oct_wait")
    src, exe = d / "main.cc", d / "main"
    src.write_text(MAIN)
    subprocess.run(["g++", "-O0", "-std=c++17", "-I" + os.path.join(ROOT, "pdfs_gb300", "csrc"), str(src), "-o",
                    str(exe)], check=True)

    def call(rows):
        r = subprocess.run([str(exe)], input="\n".join(" ".join(map(str, t)) for t in rows), text=True,
                           capture_output=True, check=True)
        return [int(x) for x in r.stdout.split()]

    return call


def restated(osw, first, full, bits):
    return max([j for j in range(osw) if full >> j & 1 or bits >> (first + j) % 8 & 1], default=-1)


def test_no_bits_are_read_where_full_sweeps_answer(latest):
    one = [(0, first, 1, -1) for first in range(8)]          # plain sweeps: a round of one
    full = [(j, first, 0xff, -1) for j in range(8) for first in range(8)]
    assert latest(one) == [-1] * 8
    assert latest(full) == [j - 1 for j in range(8) for _ in range(8)]


def test_latest_earlier_sweep(latest):
    r = random.Random(3)
    rows = [(r.randrange(8), r.randrange(8), r.choice([0, 0xff, r.randrange(256)]), r.randrange(256)) for _ in range(4000)]
    assert latest(rows) == [restated(*t) for t in rows]
