"""Projected area of drops at inclinations where the terminator degenerates (along and across the
axis, a hair off either), against half the integral of |k . n| over a dense grid of the surface."""
from __future__ import annotations

import math

import numpy as np
import pytest


def dense_area(c, k, nchi=20000, npsi=2000):
    """Midpoint rule in the colatitude and the azimuth: about 1e-7."""
    chi = math.pi * (np.arange(nchi) + 0.5) / nchi
    n = np.arange(8)
    r = 1 + np.cos(np.outer(chi, n)) @ np.asarray(c)
    dr = -(np.sin(np.outer(chi, n)) * n) @ np.asarray(c)  # dr / dchi
    # surface r(chi) (sin chi cos psi, -cos chi, sin chi sin psi): normal x area element
    axial = -(r * np.sin(chi)) * (r * np.cos(chi) + dr * np.sin(chi))   # y component
    radial = (r * np.sin(chi)) * (r * np.sin(chi) - dr * np.cos(chi))
    psi = 2 * math.pi * (np.arange(npsi) + 0.5) / npsi
    kt, ky = math.hypot(k[0], k[2]), k[1]
    s = np.abs(kt * radial[:, None] * np.cos(psi)[None, :] + ky * axial[:, None]).sum()
    return 0.5 * s * (math.pi / nchi) * (2 * math.pi / npsi)


@pytest.mark.parametrize("alpha", [0.0, 1e-9, 1e-3, 20.0, 45.0, 89.999, 90.0])
@pytest.mark.parametrize("radius", [0.41, 1.5, 3.0])
def test_area_at_degenerate_inclinations(icp, alpha, radius):
    c = icp.RaindropShape.make(radius).coefficients
    k = (0.0, -1.0, 0.0) if alpha == 90.0 else (math.cos(math.radians(alpha)), -math.sin(math.radians(alpha)), 0.0)
    got = icp.compute_projected_area(c, radius, k) / radius ** 2
    assert abs(got / dense_area(c, k) - 1) <= 1e-6
    # continuous in the inclination, also through the degenerate ones
    near = math.radians(alpha) + (1e-10 if alpha < 45 else -1e-10)
    other = icp.compute_projected_area(c, radius, (math.cos(near), -math.sin(near), 0.0)) / radius ** 2
    assert abs(got / other - 1) <= 1e-9
