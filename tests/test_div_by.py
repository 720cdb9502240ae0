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


EDGES = r"""
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include <limits>
#include "physics.h"
int main() {
    long bad = 0;
    const double inf = std::numeric_limits<double>::infinity(), nan = std::nan(""), big = std::numeric_limits<double>::max();
    const double mn = std::numeric_limits<double>::min(), den = std::numeric_limits<double>::denorm_min();
    const double as[] = {0.0, den, mn / 2, std::nextafter(mn, 0.0), mn, std::nextafter(mn, 1.0), 1.0, big / 2, big, inf, nan};
    const double bs[] = {1.0, 3.0, 0.3, 1e-6, 1e6, inf, 0.0, nan};
    for (double a : as)
        for (double b : bs)
            for (double s : {1.0, -1.0}) {
                volatile double rb = 1.0 / b, t = s * a / b;
                const double q = gfm::div_by(s * a, b, rb), want = t;
                const double lo = std::nextafter(want, -inf), hi = std::nextafter(want, inf);
                const bool tiny = std::fabs(a) < std::ldexp(1.0, -969);   // an ulp off at most
                const bool ok = std::isnan(want) ? std::isnan(q) : tiny ? q >= lo && q <= hi : q == want;
                bad += !ok || (want == 0.0 && a == 0.0 && std::signbit(q) != std::signbit(want));
            }
    std::printf("%ld\n", bad);
}
"""


# quotients at the ends of the exponent's range, where the product by the reciprocal
# stays as it is: the device and the host share the expression that decides it
@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_div_by_at_the_ends_of_the_range(tmp_path):
    csrc = pathlib.Path(__file__).resolve().parent.parent / "gfm_gb300" / "csrc"
    (tmp_path / "e.cpp").write_text(EDGES)
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{csrc}", "e.cpp", "-o", "e"], cwd=tmp_path, check=True)
    assert subprocess.run(["./e"], cwd=tmp_path, check=True, capture_output=True, text=True).stdout.strip() == "0"
