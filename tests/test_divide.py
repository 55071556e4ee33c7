"""Division by a constant through its reciprocal (gdem_divide.cuh) against the
machine's division, bit for bit: random divisors, the leapfrog's own (6, the
masses and inertias of the scenarios), significands next to a power of two,
quotients next to a rounding boundary, zeros of both signs, numbers outside the
range the method covers, infinities and NaN."""
import os
import subprocess
import textwrap
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "pacific_b200" / "csrc"
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"

PROGRAM = textwrap.dedent(r"""
    #include <cstdint>
    #include <cstdio>
    #include <cstring>
    #include <limits>
    #include <random>
    #include "gdem_divide.cuh"
    static bool same(double x, double y) { return std::memcmp(&x, &y, 8) == 0 || (x != x && y != y); }
    int main() {
      std::mt19937_64 g(7);
      auto num = [&](int span) {
        uint64_t m = g() & ((1ull << 52) - 1);
        if (g() % 4 == 0) m = g() % 8;                              // next to a power of two
        if (g() % 4 == 0) m = (1ull << 52) - 1 - g() % 8;
        uint64_t bits = ((uint64_t)(1023 + (int)(g() % (2 * span + 1)) - span) << 52) | m;
        double d;
        std::memcpy(&d, &bits, 8);
        return g() & 1 ? d : -d;
      };
      const double inf = std::numeric_limits<double>::infinity();
      const double own[] = {6., 1.0471975511965977e-05, 4.1887902047863906e-12, 3.2e-17, 8.1e-05};
      long bad = 0, n = 0;
      for (int k = 0; k < 4000; ++k) {
        double b = k < 5 ? own[k] : std::fabs(num(k % 2 ? 40 : 400));
        const double rb = gdem::reciprocalFor(b);
        for (int i = 0; i < 1000; ++i, ++n) {
          double a = num(i % 3 ? 60 : 900);
          if (i % 5 == 0) {                                         // a quotient next to a midpoint
            double q = num(30);
            a = std::fma(b, q, b * q * 1.1102230246251565e-16 * (g() % 2 ? 1. : -1.));
          }
          if (i == 1) a = 0.;
          if (i == 2) a = -0.;
          if (i == 3) a = inf;
          if (i == 4) a = std::numeric_limits<double>::quiet_NaN();
          if (i == 6) a = std::numeric_limits<double>::denorm_min() * (double)(g() % 100);
          if (!same(gdem::divideBy(a, b, rb), a / b) && bad++ < 5)
            std::printf("case %a / %a: %a, not %a\n", a, b, gdem::divideBy(a, b, rb), a / b);
        }
      }
      std::printf("%ld of %ld differ\n", bad, n);
      return bad ? 1 : 0;
    }
""")


def test_division_by_a_constant_is_correctly_rounded(tmp_path):
    if not (CUDA / "cuda_runtime.h").exists():
        pytest.skip("no CUDA headers")
    src = tmp_path / "div.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "div"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{CUDA}", f"-I{CSRC}",
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
