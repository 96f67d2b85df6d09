"""Which FP64 exchanges take the int8 tensor cores (i8_rule.h), on both sides of its lines, and the bound behind the
one on n: the digits of the scheme are bytes from -128 to 127 and a group of digit products sums at most seven
pairs of them in 32 bits, so with every digit at -128 the sum still holds for the largest n admitted and no longer for
the first that would wrap."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "i8_rule.h"
int main(int c, char** v) {
  const long n = atol(v[1]), npad = (n + 63) / 64 * 64, kdim = atol(v[2]), noccp = atol(v[3]), kper = atol(v[4]);
  std::printf("%d %d %ld\n", rijk::int8_exchange(npad, kdim), rijk::int8_half_transform(n, npad, kdim, noccp, kper),
              rijk::kMaxDigitSum);
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("rule")
    src, exe = str(d / "r.cpp"), str(d / "r")
    open(src, "w").write(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "nopt_b200", "csrc", "rijk"), src, "-o", exe],
                   check=True, capture_output=True)

    def ask(*a):
        out = subprocess.run([exe] + [str(x) for x in a], check=True, capture_output=True, text=True).stdout
        return [int(x) for x in out.split()]
    return ask


@pytest.mark.parametrize("n,kdim,noccp,kper,k,x", [
    (192, 1 << 20, 16, 1600, 0, 0),       # not more than 192 functions
    (193, 50862, 16, 1600, 0, 0),         # 3 x 256^2 = 196608 and 1e10 / 196608 = 50862.6
    (193, 50863, 16, 1600, 1, 1),
    (300, 70400, 64, 1632, 1, 0),         # parts that split an aux function
    (18720, 16, 16, 16, 1, 1),
    (18721, 16, 16, 16, 1, 0),            # the contraction over n might not be exact
    (40000, 64, 32, 64, 1, 0),
])
def test_lines_of_the_rule(rule, n, kdim, noccp, kper, k, x):
    assert rule(n, kdim, noccp, kper)[:2] == [k, x]


def test_sums_are_exact_up_to_the_bound(rule):
    bound = rule(1, 1, 16, 16)[2]
    worst = lambda n: np.full(7 * n, -128, np.int64) @ np.full(7 * n, -128, np.int64)
    assert worst(bound) < 2 ** 31 - 1
    assert np.int64(np.int32(worst(bound))) == worst(bound)
    assert worst(bound + 5) >= 2 ** 31
