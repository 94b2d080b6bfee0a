"""The integer float64 product and quotient (csrc/ct_sf64.cuh) against the
processor's, on the host build of the same code: the same bits, or flagged."""

import pathlib
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "numba_celltree_gb300" / "csrc"

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "ct_sf64.cuh"
static std::mt19937_64 g(5);
static double any(int mode) {
    static const double special[] = {0.0, -0.0, 1.0, -1.0, INFINITY, -INFINITY, NAN, 5e-324,
                                     2.2250738585072014e-308, 1.7976931348623157e308, 3.0, 0.1};
    uint64_t b = g(), m = b & 0xfffffffffffffull;
    if (mode == 0) return sf_value(b);
    if (mode == 1) m &= ~((1ull << (g() % 53)) - 1);               // few significant bits
    if (mode == 2) m = (g() & 1) ? m & 0xfff : 0xfffffffffffffull - (m & 0xfff);  // next to a power of two
    if (mode == 4) return special[g() % 12];
    return sf_value((b & 0x8000000000000000ull) | ((uint64_t)(1023 + g() % 60 - 30) << 52) | m);
}
static bool same(double x, double y) { return sf_bits(x) == sf_bits(y) || (x != x && y != y); }
int main() {
    long wrong = 0, needless = 0;
    for (long i = 0; i < 3000000; i++) {
        const double a = any(g() % 5), b = any(g() % 5), p = a * b, q = a / b;
        bool f = false;
        double r = sf_mul(a, b, &f);
        if (!f && !same(r, p)) wrong++;
        if (f && std::isnormal(a) && std::isnormal(b) && std::fabs(p) > 1e-300 && std::fabs(p) < 1e300) {
            if (std::fabs(a) < 1e300 && std::fabs(b) < 1e300) needless++;
        }
        f = false;
        r = sf_div(a, b, &f);
        if (!f && !same(r, q)) wrong++;
        if (f && std::isnormal(a) && std::isnormal(b) && std::fabs(q) > 1e-300 && std::fabs(q) < 1e300) needless++;
        const double t = std::nextafter(p, (g() & 1) ? 1e308 : -1e308);  // a quotient next to a representable one
        f = false;
        r = sf_div(t, b, &f);
        if (!f && !same(r, t / b)) wrong++;
    }
    std::printf("%ld %ld\n", wrong, needless);
    return 0;
}
"""


@pytest.mark.parametrize("rcp_error", [0, 2, -2])
def test_same_bits_as_the_processor(tmp_path, rcp_error):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    cmd = ["g++", "-O2", "-ffp-contract=off", "-I", str(CSRC), str(src), "-o", str(exe)]
    if rcp_error:  # the GPU's reciprocal approximation is off by up to one unit
        cmd.insert(1, f"-DSF_TEST_RCP={rcp_error}")
    subprocess.run(cmd, check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0", "0"]
