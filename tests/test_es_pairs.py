"""The FP64 spreading's polynomials of the ES kernel (csrc/es_pairs.h, compiled as plain C++) against the
kernel in 50-digit arithmetic."""
import subprocess
from decimal import Decimal, getcontext
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "mp_tools_gb300" / "csrc"
PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include "es_pairs.h"
using namespace mpsq;
int main() {
  for (int w = 3; w <= 16; ++w) {
    const EsPairs t = make_pairs(w, 2.30 * w);
    for (int p = 0; p < (w + 1) / 2 - 1; ++p)
      for (int k = 0; k <= 40; ++k) {                      // as the kernel evaluates a pair
        const double d = -0.5 * w + (k + 0.37) / 41.0, v = std::fma(2.0, d, (double)(w - 1)), v2 = v * v;
        double e = t.e[p][kEven - 1], o = t.o[p][kOdd - 1];
        for (int q = kEven - 2; q >= 0; --q) e = std::fma(e, v2, t.e[p][q]);
        for (int q = kOdd - 2; q >= 0; --q) o = std::fma(o, v2, t.o[p][q]);
        printf("%d %d %a %a %a\n", w, p, d, std::fma(v, o, e), std::fma(-v, o, e));
      }
  }
}
"""


@pytest.fixture(scope="module")
def values(tmp_path_factory):
    d = tmp_path_factory.mktemp("pairs")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(CSRC), "-o", str(d / "main"), str(d / "main.cpp")],
                   check=True)
    rows = subprocess.run([str(d / "main")], check=True, capture_output=True, text=True).stdout.split("\n")
    return [r.split() for r in rows if r]


def test_pairs_against_the_kernel_in_50_digits(values):
    """Bound: the rounding of the value (2^-53 of the peak at most, with that of E and of O before it),
    4e-16; sqrt and exp in double reach 3e-15."""
    getcontext().prec = 50
    worst = Decimal(0)
    for w, p, d, a, b in values:
        w, p, d = int(w), int(p), Decimal(float.fromhex(d))
        beta = Decimal(2.30 * w)
        for cell, got in ((p + 1, a), (w - 2 - p, b)):
            z = (d + cell) * 2 / w
            phi = (beta * ((1 - z * z).sqrt() - 1)).exp()
            worst = max(worst, abs(Decimal(float.fromhex(got)) - phi))
    assert worst < Decimal("4e-16")
