"""Focal grids that start on an 8-byte boundary only (all that icp_focal_sample asks for): labels,
results, density and counters equal those of an aligned grid bit for bit."""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import pytest

import rainbow_cases as RC

pytestmark = pytest.mark.gpu


def run(icp, ctx, focal, nt, np_, shift):
    n = nt * np_
    words = np.zeros(18 * n + 2)
    words[shift:shift + 18 * n] = np.ascontiguousarray(focal, dtype=icp.FOCAL_DTYPE).reshape(-1).view(np.float64)
    buf = icp.DeviceArray(ctx, 18 * n + 2).upload(words)
    assert buf.ptr.value % 16 == 0
    ptr = C.c_void_p(buf.ptr.value + 8 * shift)
    cfg = icp.DiffractionConfig(2.0 * math.pi / 180, 4.0, 0.25, 3.0)
    labels = [icp.DeviceArray(ctx, n, np.uint32) for _ in range(2)]
    results = [icp.DeviceArray(ctx, n, icp.DIFFRACTION_DTYPE) for _ in range(2)]
    density = [icp.DeviceArray(ctx, n) for _ in range(2)]
    stats = [icp.DiffractionStats() for _ in range(2)]
    L, ck = icp.LIB, icp.check
    ck(L.icp_rainbow_diffraction(ctx.handle, ptr, nt, np_, C.byref(cfg), labels[0].ptr, results[0].ptr, density[0].ptr,
                                 C.byref(stats[0])))
    ck(L.icp_rainbow_detect(ctx.handle, ptr, nt, np_, C.byref(cfg), labels[1].ptr))
    ck(L.icp_rainbow_filter(ctx.handle, ptr, labels[1].ptr, nt, np_, C.byref(cfg), results[1].ptr, density[1].ptr,
                            C.byref(stats[1])))
    return [a.download().tobytes() for a in (*labels, *results, *density)] + [s.as_dict() for s in stats]


@pytest.mark.parametrize("nt,np_", [(2, 3), (64, 127), (90, 300)])
def test_eight_byte_focal_grid(icp, ctx, nt, np_):
    f = RC.bow_grid(nt, np_, 7, primary_deg=138.0, secondary_deg=129.0, invalid=0.001)
    assert run(icp, ctx, f, nt, np_, 1) == run(icp, ctx, f, nt, np_, 0)
