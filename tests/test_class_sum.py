"""The fixed-point sum of the 7-slice GEMM's exact classes and merged class (sum_bits, sum_fixed, hx_slice.h) on the host:
groups of eight counts |n| up to K 2^46.1 with |m| up to 6 K 2^-26, K = 1 to 256, sums that cancel among them. Against
n 2^-32 + m in 128 bits the error stays below 2^-61 of the group's largest value, or below 2^-(33 + cap) where the cap
binds, and no sum leaves 63 bits."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "hx_slice.h"
int main()
{
    std::mt19937_64 g(7);
    long bad = 0, capped = 0;
    for (long i = 0; i < 400000; ++i) {
        const int K = 1 + (int)(g() % 256), cap = 22 - (K > 1 ? 32 - __builtin_clz(K - 1) : 0), down = (int)(g() % 56);
        const long long top = (long long)(K * std::pow(2.0, 46.1));
        long long n[8];
        float m[8];
        unsigned long long u = 0;
        double big = 0;
        for (int e = 0; e < 8; ++e) {
            n[e] = (long long)(g() % (unsigned long long)top) >> (i % 3 ? down : g() % 56);
            if (i % 5 == 0) n[e] = top - (long long)(g() % 4);
            if (i % 17 == 0) n[e] = 0;
            if (g() & 1) n[e] = -n[e];
            m[e] = (float)std::ldexp((double)(long long)(g() >> 12) - 0x1p51, -51) * 6.0f * K * 0x1p-26f / (float)(1ull << (g() % 30));
            if (i % 5 == 0) m[e] = std::copysign(6.0f * K * 0x1p-26f, m[e]);
            u |= (unsigned long long)(n[e] ^ (n[e] >> 63));
            big = std::fmax(big, std::fabs((double)n[e]) * 0x1p-32);
        }
        const int fb = tc::sum_bits(u, cap);
        capped += fb == cap;
        if (fb < 7) ++bad;
        for (int e = 0; e < 8; ++e) {
            const long long v = tc::sum_fixed<32>(n[e], m[e], fb);
            const _Float128 x = (_Float128)n[e] / (_Float128)4294967296.0 + (_Float128)m[e];
            const _Float128 r = (_Float128)v / ((_Float128)4294967296.0 * (_Float128)(1 << fb));
            const double err = std::fabs((double)(r - x));
            if (!(err <= (fb == cap ? std::ldexp(1.0, -33 - cap) : big * 0x1p-61)) || std::llabs(v) >= (1LL << 62) + (1LL << 31)) ++bad;
        }
    }
    printf("%ld %ld\n", bad, capped);
}
"""


def test_sum_fixed(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    r = subprocess.run(["g++", "-O2", "-std=gnu++17", "-I", os.path.join(ROOT, "helios_gb300", "csrc"), str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    bad, capped = map(int, subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    assert bad == 0 and capped > 0
