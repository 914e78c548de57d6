"""Integer FP64 division, square root, product, conversions and ordering
(csrc/afx_fp64.cuh) against the host's IEEE operations: bit for bit, with the reciprocal seeds off by up
to 3 units in their last place either way."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aeroflex_gb300", "csrc")

SRC = r"""
#include "afx_fp64.cuh"
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
namespace afx { namespace fp64 { int seed_ulps = 0; } }
using namespace afx::fp64;
static bool same(double a, double b) { return (a != a && b != b) || bits_of(a) == bits_of(b); }
int main(int argc, char** argv) {
    seed_ulps = std::atoi(argv[1]);
    std::mt19937_64 g(17 + seed_ulps);
    const double edge[] = {0.0, -0.0, 1.0, -1.0, 1.5, INFINITY, -INFINITY, NAN, 5e-324, -2.5e-308, 2.2250738585072014e-308,
                           1.7976931348623157e308, 0x1.fffffffffffffp-1, 0x1.0000000000001p0, 4.0, 0x1.fffffffffffffp0};
    const int ne = sizeof(edge) / sizeof(edge[0]);
    auto draw = [&]() {
        const int f = (int)(g() & 63);
        uint64_t m = g() & 0x000fffffffffffffull;
        if ((f & 3) == 1) m &= ~((1ull << (g() % 52)) - 1);          // few leading bits
        if ((f & 3) == 2) m |= (1ull << (g() % 52)) - 1;             // ones at the end
        if ((f & 12) == 12) m = (f & 16) ? 0x000fffffffffffffull - (g() & 3) : (g() & 3);  // a binade's ends
        const uint64_t e = (f & 32) ? g() % 2048 : 980 + g() % 90;
        return of_bits((g() & 0x8000000000000000ull) | (e << 52) | m);
    };
    long bad = 0;
    for (long i = 0; i < 2000000; ++i) {
        const double x = i < ne * ne ? edge[i / ne] : draw(), y = i < ne * ne ? edge[i % ne] : draw();
        bad += !same(div(x, y), x / y);
        const Den d = den(y);
        bad += !same(quot(x, d), x / y) || !same(quot(x, twice(d)), x / (2.0 * y));
        bad += !same(root(std::fabs(x)), std::sqrt(std::fabs(x))) || !same(root(x), std::sqrt(x));
        bad += !same(mul(x, y), x * y);
        uint32_t r;
        if (narrow(x, r)) bad += f32_bits((float)x) != r;
        const float xf = (float)x;
        if (std::fabs(xf) >= 1.17549435e-38f || xf == 0.f || xf != xf) bad += !same(widen(f32_bits(xf)), (double)xf);
        bad += less(x, y) != (x < y) || less_equal(x, y) != (x <= y) || less_equal(x, x) != (x <= x);
        const double s = y * y;  // next to exact squares
        if (s > 1e-300 && s < 1e300)
            for (int k = -1; k < 2; ++k) bad += !same(root(of_bits(bits_of(s) + k)), std::sqrt(of_bits(bits_of(s) + k)));
    }
    std::printf("%ld\n", bad);
    return bad != 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("fp64")
    src, exe = d / "t.cpp", d / "t"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("ulps", [-3, 0, 3])
def test_integer_fp64_operations_are_ieee(program, ulps):
    r = subprocess.run([program, str(ulps)], capture_output=True, text=True)
    assert r.returncode == 0, "%s mismatches" % r.stdout.strip()
