"""div_by (physics.h), the division by a number whose reciprocal is at hand: the
correctly rounded quotient, as IEEE division gives it, over the magnitudes of the
solver's fields, for operands whose quotient lies next to the middle of two
numbers, and for zeros and infinities."""
import pathlib
import shutil
import subprocess

import pytest

SRC = r"""
#include <cmath>
#include <cstdio>
#include <limits>
#include <random>
#include "physics.h"
int main() {
    std::mt19937_64 g(3);
    long bad = 0;
    auto mag = [&](double lo, double hi) { return std::exp(std::uniform_real_distribution<>(std::log(lo), std::log(hi))(g)); };
    auto check = [&](double a, double b) {
        volatile double rb = 1.0 / b, t = a / b;
        const double r = rb;
        bad += gfm::div_by(a, b, r) != t;
    };
    for (int i = 0; i < 500000; ++i) check(mag(1e-150, 1e30) * (g() & 1 ? 1 : -1), mag(1e-6, 1e6));
    for (int i = 0; i < 200000; ++i) {
        const double b = 1.0 + (g() >> 12) * 0x1p-52, q = 1.0 + (g() >> 12) * 0x1p-52, a = b * q;
        check(a, b); check(std::nextafter(a, 0.0), b); check(std::nextafter(a, 9.0), b);
    }
    for (double c : {3.0, 24.0, 1000.0, 1.0e6, 1.5})
        for (int i = 0; i < 50000; ++i) check(mag(1e-30, 1e10), c);
    const double inf = std::numeric_limits<double>::infinity();
    check(0.0, 3.0); check(inf, 3.0); check(-inf, 3.0);
    bad += !std::signbit(gfm::div_by(-0.0, 3.0, 1.0 / 3.0));
    std::printf("%ld\n", bad);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_div_by_is_the_correctly_rounded_quotient(tmp_path):
    csrc = pathlib.Path(__file__).resolve().parent.parent / "gfm_gb300" / "csrc"
    (tmp_path / "d.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{csrc}", "d.cpp", "-o", "d"], cwd=tmp_path, check=True)
    assert subprocess.run(["./d"], cwd=tmp_path, check=True, capture_output=True, text=True).stdout.strip() == "0"
