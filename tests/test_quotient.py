"""quotient_by (superdca_gb300/csrc/quotient.h), the quotient of k_trial's
softmax weights, against division, compiled with the host compiler: the same
bits for divisors in [1, 4] and dividends from 2^-960 up (random and extreme
significands, quotients next to the midpoint of two doubles), one unit in the
last place below; zero and NaN as division gives them.  No GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>
#include "quotient.h"

int main()
{
    std::mt19937_64 g(20);
    // a significand in [1, 2): random, all zeros, all but a few ones, or nearly 1
    auto sig = [&] {
        uint64_t m = g() >> 12;
        switch (g() % 8) {
        case 0: m = 0; break;
        case 1: m = (1ull << 52) - 1 - g() % 8; break;
        case 2: m = g() % 8; break;
        default: break;
        }
        return 1.0 + std::ldexp((double)m, -52);
    };
    auto divisor = [&] { const double z = sig(); return g() & 1 ? 2.0 * z : z; };
    long apart = 0, middle = 0, low = 0, special = 0;
    for (int i = 0; i < 4000000; ++i) {
        const double z = divisor(), v = std::ldexp(sig(), -(int)(g() % 960));
        apart += sdca::quotient_by(v, z, 1.0 / z) != v / z;
    }
    for (int i = 0; i < 4000000; ++i) {
        // v / z next to q + 2^-53 for a double q in [1, 2), scaled
        const double z = divisor(), q = 1.0 + std::ldexp((double)(g() >> 12), -52);
        const double v = std::ldexp(std::fma(q, z, std::ldexp(z, -53)), -2 - (int)(g() % 900));
        const double w = std::nextafter(v, g() & 1 ? 0.0 : 1.0);
        middle += sdca::quotient_by(v, z, 1.0 / z) != v / z;
        middle += sdca::quotient_by(w, z, 1.0 / z) != w / z;
    }
    for (int i = 0; i < 1000000; ++i) {
        const double z = divisor(), v = std::ldexp(sig(), -960 - (int)(g() % 115)), a = v / z;
        const double b = sdca::quotient_by(v, z, 1.0 / z);
        low += !(b == a || b == std::nextafter(a, 0.0) || b == std::nextafter(a, 1.0));
    }
    special += sdca::quotient_by(0.0, 1.5, 1.0 / 1.5) != 0.0;
    special += !std::isnan(sdca::quotient_by(std::nan(""), 1.5, 1.0 / 1.5));
    special += !std::isnan(sdca::quotient_by(0.5, std::nan(""), 1.0 / std::nan("")));
    std::printf("%ld %ld %ld %ld\n", apart, middle, low, special);
}
"""


def test_quotient_is_the_division(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    src, exe = tmp_path / "quotient.cpp", tmp_path / "quotient"
    src.write_text(SRC)
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I" + os.path.join(ROOT, "superdca_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split() == ["0"] * 4
