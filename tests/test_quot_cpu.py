"""csrc/icp_quot.cuh on the CPU, compiled with g++: quot(a, div_by(b)) equals a / b bit for bit for
random operands, for mantissas at both ends of a binade, for zeros of either sign, subnormals,
infinities and NaN, and on both sides of the exponents at which the operator takes over -- also
where the quotient of two ordinary operands overflows or underflows."""
from __future__ import annotations

import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <limits>
#include <random>
#include <vector>
#include "icp_quot.cuh"
static bool same(double x, double y)
{
    uint64_t a, b;
    std::memcpy(&a, &x, 8);
    std::memcpy(&b, &y, 8);
    return a == b || (x != x && y != y);
}
static long long checked;
static bool check(double a, double b)
{
    ++checked;
    const double got = icp::quot(a, icp::div_by(b)), want = a / b;
    if (same(got, want)) return true;
    printf("%a / %a: %a, operator %a\n", a, b, got, want);
    return false;
}
int main()
{
    std::mt19937_64 g(11);
    const double inf = std::numeric_limits<double>::infinity();
    std::vector<double> v = {0.0, inf, std::numeric_limits<double>::quiet_NaN(), std::numeric_limits<double>::max(),
                             std::numeric_limits<double>::min(), std::numeric_limits<double>::denorm_min(), 1.0, 3.0,
                             3.141592653589793, 6.283185307179586};
    const int edge[] = {-1074, -1022, -1021, -901, -900, -899, -600, -452, -451, -450, -449, -300, -60, -1, 0, 1, 53,
                        300, 448, 449, 450, 451, 600, 899, 900, 901, 1000, 1023};
    for (int e : edge)
        for (double m : {1.0, 1.0 + 0x1p-52, 1.5, 2.0 - 0x1p-52, 2.0 - 0x1p-51, 1.3333333333333333}) v.push_back(std::ldexp(m, e));
    for (double a : v)
        for (double b : v)
            for (int s = 0; s < 4; ++s)
                if (!check(s & 1 ? -a : a, s & 2 ? -b : b)) return 1;
    const auto number = [&](int spread) {
        const uint64_t r = g();
        const double m = 1.0 + (double)(r >> 12) * 0x1p-52;
        const double x = std::ldexp(m, (int)(g() % (2 * spread + 1)) - spread);
        return r & 1 ? -x : x;
    };
    for (int spread : {0, 3, 60, 450, 1023})
        for (int i = 0; i < 3000000; ++i)
            if (!check(number(spread), number(spread))) return 1;
    printf("OK %lld\n", checked);
    return 0;
}
"""


def test_quot_is_the_division_operator(tmp_path):
    src = tmp_path / "quot.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "quot"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(ROOT / "ice_crystal_phase_b200" / "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert int(r.stdout.split()[1]) > 15_000_000
