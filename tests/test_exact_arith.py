"""The decoder's replacements for divisions, restated on the host: the block coordinates' division of
ids below 2^44 by one high multiply, and the recovered coordinates' division by the rounded constants
sqrt(3) and sqrt(5) through the reciprocal with one fused correction (every significand)."""
import os
import shutil
import subprocess

import pytest

SOURCE = r"""
#include "kernels.h"
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
using u64 = unsigned long long;
static u64 udiv44(u64 x, const xnyz::dev::U64Div& d) {
    return (u64)(((unsigned __int128)(x << 20) * d.m44) >> 64) >> d.l44;
}
static float div_const(float x, float d, float y) {
    const float q = x * y;
    return std::fmaf(std::fmaf(-q, d, x), y, q);
}
int main() {
    std::mt19937_64 rng(11);
    long bad = 0;
    for (int i = 0; i < 400; ++i) {
        const u64 d = i < 40 ? (u64)i + 1 : i < 64 ? 1ull << (i - 39) : (rng() >> (39 + rng() % 25)) + 1;
        const auto m = xnyz::dev::make_u64div(d);
        const u64 top = (1ull << 44) - 1;
        for (u64 x : {0ull, 1ull, d - 1, d, d + 1, top, top - 1, top / d * d, top / d * d - 1})
            if (x <= top && udiv44(x, m) != x / d) ++bad;
        for (int k = 0; k < 5000; ++k) {
            const u64 x = (rng() & top) >> (rng() % 44);
            if (udiv44(x, m) != x / d) ++bad;
            const u64 e = x / d * d;
            if (udiv44(e, m) != e / d || (e && udiv44(e - 1, m) != (e - 1) / d)) ++bad;
        }
    }
    for (double k : {3.0, 5.0}) {
        const float d = (float)std::sqrt(k), y = (float)(1.0 / (double)d);
        for (unsigned b = 0x3f800000u; b < 0x40000000u; ++b) {
            float x;
            std::memcpy(&x, &b, 4);
            if (div_const(x, d, y) != x / d || div_const(-x, d, y) != -x / d) ++bad;
        }
        for (int e : {-39, -20, 30, 74}) {
            for (int i = 0; i < 200000; ++i) {
                const float x = std::ldexp((float)((rng() >> 40) | (1 << 23)), e - 23);
                if (div_const(x, d, y) != x / d) ++bad;
            }
        }
        if (div_const(0.0f, d, y) != 0.0f) ++bad;
    }
    std::printf("%ld\n", bad);
    return bad != 0;
}
"""


def test_divisions_by_multiplication(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    src, exe = tmp_path / "div.cpp", tmp_path / "div"
    src.write_text(SOURCE)
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xnyzip_b200", "csrc")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", csrc, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
