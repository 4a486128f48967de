"""The fixed-point conversion of the 7-slice GEMM's epilogue (fixed_pow2, hx_slice.h) on the host: v 2^k rounded
to nearest even, against the long double (64 or more significand bits) result."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "hx_slice.h"
int main()
{
    std::mt19937_64 g(11);
    long bad = 0, refused = 0;
    for (long i = 0; i < 2000000; ++i) {
        long long v = (long long)g() >> (g() % 63 + 1);
        if (i % 7 == 0) v = (1LL << (g() % 62)) - (long long)(g() % 3);             // beside powers of two
        if (i % 11 == 0) v = (long long)((g() >> 11) << 10 | 1ull << 9) >> (g() % 8);   // beside halfway cases
        const int k = i % 13 == 0 ? (int)(g() % 2200) - 1150 : (int)(g() % 200) - 100;
        bool ok = true;
        const double r = tc::fixed_pow2(v, k, ok);
        const double x = (double)std::ldexp((long double)v, k);
        if (!ok) { if (std::fabs(x) > 0x1p-1022 && std::fabs(x) < 1.7e308) ++bad; ++refused; }
        else if (!(r == x)) ++bad;
    }
    printf("%ld %ld\n", bad, refused);
}
"""


def test_fixed_pow2(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "helios_gb300", "csrc"), str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    bad, refused = map(int, subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    assert bad == 0 and refused > 0
