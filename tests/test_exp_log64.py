"""The FP64 functions of a node belief (csrc/exp_log64.h), compiled with the
host compiler, against long double.  Bounds: half a unit for the last
rounding, plus what the steps before leave (exp: the remainder's and the
polynomial's rounding, 0.03; log: the remainder's 0.07 and twice 0.125 for
the low parts where the result is at least twice the polynomial; reciprocal:
the cube of the start's error)."""
import json
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cmath>
#include <cstdio>
#include "exp_log64.h"

static double ulps(double got, long double want)
{
    const double w = std::fabs((double)want);
    const long double u = (long double)std::nextafter(w, INFINITY) - w;
    return (double)(std::fabs((long double)got - want) / u);
}

int main()
{
    double we = 0, wl = 0, wr = 0;
    auto e = [&](double x) { we = std::fmax(we, ulps(sdca::exp64(x, sdca::kExpTab), expl((long double)x))); };
    auto l = [&](double z) {
        if (z > 1) wl = std::fmax(wl, ulps(sdca::log64(z, sdca::kLogTab), logl((long double)z)));
        wr = std::fmax(wr, ulps(sdca::rcp64(z), 1.0L / z));
    };
    unsigned long long s = 12345;
    auto uni = [&] { s = s * 6364136223846793005ull + 1442695040888963407ull; return (double)(s >> 11) * 0x1p-53; };
    for (int i = 0; i < 2000000; ++i) {
        e(-uni() * std::exp2(12 * uni() - 3));
        e(-std::exp2(-40 * uni()));
        l(1 + 3 * uni());
        l(1 + std::exp2(-40 * uni()));
    }
    for (int i = 0; i <= 256; ++i) {   // the edges of the intervals
        const double z = i < 128 ? 1 + i / 128.0 : 2 + (i - 128) / 64.0;
        l(z);
        if (z > 1) l(std::nextafter(z, 0.0));
        if (z < 4) l(std::nextafter(z, 9.0));
    }
    for (int k = 0; k < 128 * 700; ++k) {
        const double x = -(k + 0.5) * std::log(2.0) / 128;
        if (x < -699) break;
        e(x);
        e(std::nextafter(x, 0.0));
    }
    const double q = NAN;
    std::printf("{\"exp\": %.4f, \"log\": %.4f, \"rcp\": %.4f, \"exact\": %d, \"nan\": %d, \"low\": %g}\n", we, wl, wr,
                sdca::exp64(0.0, sdca::kExpTab) == 1 && sdca::log64(1.0, sdca::kLogTab) == 0 && sdca::rcp64(1.0) == 1 &&
                    sdca::rcp64(4.0) == 0.25 && sdca::log64(4.0, sdca::kLogTab) == std::log(4.0),
                std::isnan(sdca::exp64(q, sdca::kExpTab)) && std::isnan(sdca::log64(q, sdca::kLogTab)) &&
                    std::isnan(sdca::rcp64(q)),
                std::fmax(sdca::exp64(-1e5, sdca::kExpTab), sdca::exp64(-INFINITY, sdca::kExpTab)));
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_exp_log64_accuracy(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(SRC)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "superdca_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = json.loads(subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout)
    assert r["exact"] == 1 and r["nan"] == 1 and 0 <= r["low"] < 1e-300, r
    assert r["exp"] <= 0.53 and r["log"] <= 0.85 and r["rcp"] <= 0.53, r
