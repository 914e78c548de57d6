"""Zero operands of the integer FP64 operations (csrc/afx_fp64.cuh): a zero over
a normal number and a zero times a finite number have IEEE's signed zero and do
not leave the integer path; a zero times an infinity or a NaN does."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aeroflex_gb300", "csrc")

SRC = r"""
#include "afx_fp64.cuh"
#include <cmath>
#include <cstdio>
#include <initializer_list>
namespace afx { namespace fp64 { int seed_ulps = 0; } }
using namespace afx::fp64;
static bool same(double a, double b) { return (a != a && b != b) || bits_of(a) == bits_of(b); }
int main() {
    const double normal[] = {1.0, -3.5, 0x1p-1022, -0x1p1000, 1.7976931348623157e308, 0x1.fffffffffffffp-1};
    const double finite[] = {0.0, -0.0, 5e-324, -2e-308, 1.0, -3.5, 0x1p-1022, 1.7976931348623157e308};
    const double wild[] = {INFINITY, -INFINITY, NAN};
    long bad = 0;
    for (double z : {0.0, -0.0}) {
        for (double y : normal) bad += !same(quot(z, den(y)), z / y);
        for (double y : finite) bad += !same(mul(z, y), z * y) + !same(mul(y, z), y * z);
    }
    const long left = rare_calls;
    for (double z : {0.0, -0.0})
        for (double y : wild) bad += !same(mul(z, y), z * y) + !same(mul(y, z), y * z);
    std::printf("%ld %ld %ld\n", bad, left, rare_calls - left);
    return 0;
}
"""


def test_zero_operands_stay_on_the_integer_path(tmp_path):
    src, exe = tmp_path / "z.cpp", tmp_path / "z"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + CSRC, str(src), "-o", str(exe)], check=True)
    bad, left, wild = map(int, subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    assert (bad, left, wild) == (0, 0, 12)
