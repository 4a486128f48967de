"""The step's division by a stored reciprocal (stored_quotient, hx_quotient.h) on the host, against the IEEE division: half a
unit in the last place and a little for ordinary values, and the same infinities, zeros and NaNs where the denominator or the
numerator is zero or infinite."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cstdio>
#include <random>
#include "hx_quotient.h"
static bool same(double x, double y) { return (x != x && y != y) || (x == y && std::signbit(x) == std::signbit(y)); }
int main()
{
    const double inf = INFINITY, v[] = {0.0, -0.0, 1.5, -1.5, 3e-17, -7e300, inf, -inf, NAN};
    long special = 0, bad = 0;
    for (double a : v)
        for (double d : v) {
            const double got = stored_quotient(a, d, 1.0 / d), x = a / d;
            if (!(same(got, x) || std::fabs(got - x) <= 1.1e-16 * std::fabs(x) || (std::fabs(x) < 1e-290 && std::fabs(got) < 1e-290))) {
                printf("%a / %a = %a, not %a\n", a, d, got, x);
                ++special;
            }
        }
    std::mt19937_64 g(3);
    for (long i = 0; i < 2000000; ++i) {
        const double a = std::ldexp((double)(g() >> 11) - 0x1p52, (int)(g() % 120) - 110), d = std::ldexp((double)(g() >> 11) + 1.0, (int)(g() % 60) - 80);
        const double got = stored_quotient(a, -d, 1.0 / -d);
        const long double x = (long double)a / -(long double)d;
        const double ulp = std::nextafter(std::fabs(got), INFINITY) - std::fabs(got);
        if (!(std::fabs((double)(x - got)) <= 0.5001 * ulp)) ++bad;
    }
    printf("%ld %ld\n", special, bad);
}
"""


def test_stored_quotient(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "helios_gb300", "csrc"), str(src),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    assert out.split()[-2:] == ["0", "0"], out
