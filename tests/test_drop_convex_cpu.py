"""drop_convex_proven (host/icp_drop_host.hpp) on the CPU: the function's own text compiled with a
drop_radius that records where it is evaluated.  Its derivative bounds hold on [-1, 1], so no
interval may be centred outside; the accepted intervals reach mu = 1; and a shape it accepts meets
the conditions at every point of a dense sampling, shapes at the limit included."""
from __future__ import annotations

import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
static double lowest, highest;
static double drop_radius(const double c[8], double mu, double* d1, double* d2)
{
    lowest = std::fmin(lowest, mu);
    highest = std::fmax(highest, mu);
    double t0 = 1, t1 = mu, p0 = 0, p1 = 1, q0 = 0, q1 = 0;
    double r = 1 + c[0] + c[1] * mu, rp = c[1], rpp = 0;
    for (int n = 2; n < 8; ++n) {
        const double t = 2 * mu * t1 - t0, p = 2 * t1 + 2 * mu * p1 - p0, q = 4 * p1 + 2 * mu * q1 - q0;
        r += c[n] * t;
        rp += c[n] * p;
        rpp += c[n] * q;
        t0 = t1; t1 = t; p0 = p1; p1 = p; q0 = q1; q1 = q;
    }
    *d1 = rp;
    *d2 = rpp;
    return r;
}
@FUNCTION@
// least of r, G, Q over a dense sampling
static double least(const double c[8])
{
    double m = 1e300;
    for (int k = 0; k <= 4000; ++k) {
        const double mu = -1.0 + k / 2000.0;
        double rp, rpp;
        const double r = drop_radius(c, mu, &rp, &rpp), s2 = 1 - mu * mu;
        m = std::fmin(m, std::fmin(r, std::fmin(r + mu * rp, r * r + 2 * s2 * rp * rp - r * (s2 * rpp - mu * rp))));
    }
    return m;
}
int main()
{
    std::mt19937_64 gen(7);
    std::normal_distribution<double> normal;
    int accepted = 0, limit = 0;
    for (int i = 0; i < 4000; ++i) {
        double d[8], c[8];
        for (int n = 0; n < 8; ++n) d[n] = normal(gen) * (n ? 0.05 / (n * n) : 0.02);
        double scale = 1;
        if (i % 2) { // scaled to the limit of convexity, then 2 % inside or a hair outside it
            double lo = 0, hi = 1;
            for (int k = 0; k < 24; ++k) {
                const double s = 0.5 * (lo + hi);
                for (int n = 0; n < 8; ++n) c[n] = 4 * s * d[n];
                (least(c) > 0 ? lo : hi) = s;
            }
            scale = 4 * lo * (1 + (i % 4 == 1 ? -0.02 : 1e-5));
        }
        for (int n = 0; n < 8; ++n) c[n] = scale * d[n];
        lowest = 1e300;
        highest = -1e300;
        const bool ok = drop_convex_proven(c);
        if (lowest < -1 || highest > 1) {
            printf("shape %d evaluated at %.17g .. %.17g\n", i, lowest, highest);
            return 1;
        }
        // the last interval's centre is at most half a widest interval from mu = 1
        if (ok && highest < 1 - 1.0 / 64 - 1e-12) {
            printf("shape %d: stops at %.17g\n", i, highest);
            return 1;
        }
        if (ok && !(least(c) > 0)) {
            printf("shape %d accepted with least value %.3g\n", i, least(c));
            return 1;
        }
        accepted += ok;
        limit += ok && i % 2;
    }
    printf("OK %d %d\n", accepted, limit);
    return 0;
}
"""


def test_intervals_stay_within_the_bounds(tmp_path):
    text = (ROOT / "ice_crystal_phase_b200" / "host" / "icp_drop_host.hpp").read_text()
    begin = text.index("inline bool drop_convex_proven")
    function = text[begin:text.index("\n}\n", begin) + 3]
    src = tmp_path / "convex.cpp"
    src.write_text(PROGRAM.replace("@FUNCTION@", function))
    exe = tmp_path / "convex"
    subprocess.run(["g++", "-std=c++17", "-O2", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    accepted, limit = map(int, r.stdout.split()[1:])
    assert accepted > 1000 and limit > 100, r.stdout
