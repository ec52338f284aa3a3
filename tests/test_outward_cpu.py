"""csrc/icp_outward.cuh on the CPU, compiled with g++: x plus or minus the least subnormal, rounded
outward, is nextafter(x) -- for every sign, exponent and upper half of the significand of binary32
with low halves at both ends and between, and for binary64 at every exponent -- but at an infinity
that it would step away from, which stays.  (A step onto zero may carry the other sign.)"""
from __future__ import annotations

import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include "icp_outward.cuh"
static long long checked;
template <class T, class B> static bool check(B bits)
{
    T x;
    std::memcpy(&x, &bits, sizeof x);
    ++checked;
    const T inf = (T)INFINITY;
    const T up = icp::next_up(x), down = icp::next_down(x);
    const T want_up = x == -inf ? x : std::nextafter(x, inf), want_down = x == inf ? x : std::nextafter(x, -inf);
    const bool ok = x != x ? up != up && down != down
                           : up == want_up && down == want_down;
    if (!ok) printf("%a: up %a (%a), down %a (%a)\n", (double)x, (double)up, (double)want_up, (double)down, (double)want_down);
    return ok;
}
int main()
{
    std::mt19937_64 g(5);
    const uint32_t low[] = {0, 1, 2, 0x7fff, 0x8000, 0xfffe, 0xffff};
    for (uint32_t h = 0; h < 65536; ++h) {
        for (uint32_t l : low)
            if (!check<float>(h << 16 | l)) return 1;
        for (int i = 0; i < 5; ++i)
            if (!check<float>(h << 16 | (uint32_t)(g() & 0xffff))) return 1;
    }
    const uint64_t m = (1ull << 52) - 1, mant[] = {0, 1, 2, m / 2, m / 2 + 1, m - 1, m};
    for (uint64_t e = 0; e < 4096; ++e) {
        for (uint64_t l : mant)
            if (!check<double>(e << 52 | l)) return 1;
        for (int i = 0; i < 50; ++i)
            if (!check<double>(e << 52 | (g() & m))) return 1;
    }
    printf("OK %lld\n", checked);
    return 0;
}
"""


def test_neighbours(tmp_path):
    src = tmp_path / "outward.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "outward"
    subprocess.run(["g++", "-std=c++17", "-O2", "-frounding-math", "-I", str(ROOT / "ice_crystal_phase_b200" / "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert int(r.stdout.split()[1]) > 1_000_000
