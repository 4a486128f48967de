"""The slabs of the (T) correction (plan_slabs, hx_slabs.h) on the host: a row of triples fits wherever the integrals and two
rows do (W and the slices of one k-batched operand, v padded to 64 and v^2 to 128), so that no molecule needs more free memory
than slicing term by term takes; the operands of all terms are kept only where they fit as well."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _up(x, m):
    return (x + m - 1) // m * m


def test_no_molecule_needs_more_memory_than_term_by_term(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text('#include <cstdio>\n#include "hx_slabs.h"\nint main() { int N, o, v; double f; while (scanf("%d %d %d %lf", &N, &o, &v, &f) == 4) '
                   '{ SlabPlan p = plan_slabs(N, o, v, f); printf("%d %lld\\n", p.keep ? 1 : 0, p.triples); } }')
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "helios_gb300", "csrc"), str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    asked = []
    for N in (2, 9, 24, 64, 112, 160, 224, 256):
        for o in sorted({1, N // 4, N // 2, 3 * N // 4, N - 1} - {0}):
            v = N - o
            integrals = 8.0 * (o * v ** 3 + o ** 3 * v + N * v * v + 2 * N * o * o)
            row = 8.0 * v ** 3 + 14.0 * _up(v * v, 128) * _up(v, 64)
            kept = 28.0 * (2 * o * v ** 3 + 4 * o ** 3 * v + 6 * (o * v) ** 2)
            least = integrals + 2.0 * o * row
            asked += [(N, o, v, f, o if f >= least else 0, kept + integrals) for f in (1.001 * least, 1.5 * least, least + kept, 5e9, 4e10, 2.8e11)]
    got = subprocess.run([str(exe)], input="".join(f"{N} {o} {v} {f!r}\n" for N, o, v, f, _, _ in asked), capture_output=True, text=True,
                         check=True).stdout.split()
    for k, (N, o, v, f, rows, need) in enumerate(asked):
        keep, triples = int(got[2 * k]), int(got[2 * k + 1])
        if rows and o * (8.0 * v ** 3 + 14.0 * v * v * _up(v, 8)) <= 24e9:
            assert triples >= o, asked[k]
        assert not keep or need < f
    assert any(got[::2][k] == "0" and asked[k][4] for k in range(len(asked))) and "1" in got[::2]
