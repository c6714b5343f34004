"""xr::div_const and xr::div_const_scaled (csrc/qp3d_exact.h), the divisions by
a constant that the reference arithmetic's taps take, equal the IEEE division
bit for bit over the ranges their callers keep to: edges and random significands of the dividend at
every exponent, spacings and their squares as divisors."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r'''
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include "qp3d_exact.h"
using namespace qp3d;
static float bits(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
int main(int argc, char **argv)
{
    const float h = strtof(argv[1], nullptr), y = 1.0f / h;
    if (!xr::divisor_in_range(h)) return 2;
    long bad = 0, n = 0;
    uint32_t s = 12345u;
    int elo, ehi;
    frexpf(xr::kDivLo, &elo);
    frexpf(xr::kDivHi, &ehi);
    for (int e = elo - 1; e < ehi; ++e)
        for (int i = 0; i < 60000; ++i) {
            s = s * 1664525u + 1013904223u;
            uint32_t m = i < 64 ? i : i < 128 ? 0x7fffffu - (i - 64) : s >> 9;
            float p = bits(((uint32_t)(e + 127) << 23) | m);
            if (p < xr::kDivLo || p > xr::kDivHi) continue;
            if (i & 1) p = -p;
            if (xr::div_const(p, h, y) != p / h) ++bad;
            ++n;
        }
    // the scaled form: every exponent down to the subnormals, whose quotients
    // round on the subnormal grid
    for (int e = -127; e < ehi; ++e)
        for (int i = 0; i < 60000; ++i) {
            s = s * 1664525u + 1013904223u;
            uint32_t m = i < 64 ? i : i < 128 ? 0x7fffffu - (i - 64) : s >> 9;
            if (e == -127 && (i & 2)) m >>= s >> 28;   // the smallest ones too
            float p = bits(((uint32_t)(e + 127) << 23) | m);
            if (i & 1) p = -p;
            if (fabsf(p) > xr::kDivHi) continue;
            if (xr::div_const_scaled(p, h, y) != p / h) ++bad;
            ++n;
        }
    if (xr::div_const(0.0f, h, y) != 0.0f || xr::div_const(-0.0f, h, y) != 0.0f ||
        xr::div_const_scaled(0.0f, h, y) != 0.0f || xr::div_const_scaled(-0.0f, h, y) != 0.0f)
        ++bad;
    printf("%ld %ld\n", n, bad);
    return bad != 0;
}
'''


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    d = tmp_path_factory.mktemp("div")
    (d / "div.cpp").write_text(SRC)
    out = str(d / "div")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I",
                        os.path.join(ROOT, "gpu-c_3dqmodeling_gb300", "csrc"), str(d / "div.cpp"),
                        "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("h", [10.0, 12.5, 7.3, 2.0, 1.0, 0.3, 2896.3, 2.0 ** -15, 1.9999999])
def test_division_by_a_constant_is_ieee(exe, h):
    h = np.float32(h)
    for d in (h, np.float32(h * h)):
        r = subprocess.run([exe, "%.9g" % d], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, (d, r.stdout)
        assert int(r.stdout.split()[0]) > 10 ** 6
