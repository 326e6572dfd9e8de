"""Replacements for divisions and roundings, restated on the host: the block coordinates' division of
ids below 2^44 by one high multiply; the recovered coordinates' division by the rounded constants
sqrt(3) and sqrt(5) through the reciprocal with one fused correction, and the quantizers' by any step
with two (every significand); the truncated octahedron's two lattice candidates from the floor."""
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
static float div_any(float x, float d, float y) {
    float q = x * y;
    q = std::fmaf(std::fmaf(-q, d, x), y, q);
    return std::fmaf(std::fmaf(-q, d, x), y, q);
}
static long candidates(float q) {  // as the quantizer defines them, and from floor(q)
    const float e = std::round(q * 0.5f) * 2.0f, o = std::round((q - 1.0f) * 0.5f) * 2.0f + 1.0f;
    const int f = (int)std::floor(q);
    const float e2 = (float)(f + (f & 1)), o2 = q <= 0x1p-25f ? -1.0f : (float)(f | 1);
    return (e != e2) + (o != o2);
}
int main() {
    std::mt19937_64 rng(11);
    long bad = 0;
    for (int i = 0; i < 16; ++i) {
        // 1, just above 1, just below 2, and steps of any significand and size
        const unsigned m = i == 0 ? 0u : i == 1 ? 1u : i == 2 ? 0x7ffffeu : (unsigned)(rng() & 0x7fffffu);
        if (m == 0x7fffffu) continue;
        const unsigned db = (i < 4 ? 127u : 127u - 42u + (unsigned)(rng() % 85)) << 23 | m;
        float d, x;
        std::memcpy(&d, &db, 4);
        const float y = (float)(1.0 / (double)d);
        for (unsigned b = 0x3f800000u; b < 0x40000000u; ++b) {
            std::memcpy(&x, &b, 4);
            if (div_any(x, d, y) != x / d) ++bad;
        }
        for (int e : {-60, -31, 17, 59})
            for (int k = 0; k < 100000; ++k) {
                x = std::ldexp((float)((rng() >> 40) | (1 << 23)), e - 23);
                if (div_any(x, d, y) != x / d) ++bad;
            }
        if (div_any(0.0f, d, y) != 0.0f) ++bad;
    }
    for (unsigned b = 0; b < 0x4b700000u; b += b < 0x3c000000u ? 997u : 13u) {  // 0 to 2^24 - 2^20
        float q;
        std::memcpy(&q, &b, 4);
        bad += candidates(q);
    }
    for (float c = 0x1p-26f; c < 16000000.0f; c = c < 0.5f ? c * 2.0f : c < 4096.0f ? c + 0.5f : c * 1.0009f) {
        const float k = c < 0.5f ? c : std::round(c * 2.0f) * 0.5f;
        for (float q : {k, std::nextafterf(k, 0.0f), std::nextafterf(k, 1e9f)}) bad += candidates(q);
    }
    if (candidates(-0.0f)) ++bad;
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
