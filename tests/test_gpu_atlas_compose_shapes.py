"""Cyclic composition at the edges of its kernels' shapes: one cell, rows of less and more than a
thread's cells, each kernel's widest row, entries of one and of two shifts, runs across mask words.
The oracle adds in the same order, so the masses are equal bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import atlas_oracle as AO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,np_", [(1, 1), (3, 2), (2, 5), (2, 31), (2, 33), (5, 161), (2, 1280), (2, 1281),
                                    (300, 45), (2, 2304), (2, 2305), (2, 4096)])
@pytest.mark.parametrize("fill", ["pairs", "runs", "all", "none"])
def test_compose_equals_oracle(icp, ctx, nt, np_, fill):
    if fill == "all" and np_ > 200:
        pytest.skip("the oracle rolls the rows once per weight")
    rng = np.random.default_rng(np_ + nt)
    nodes = 2
    w = np.zeros((nodes, 2, np_))
    if fill == "all":
        w[:] = rng.random(w.shape)
    elif fill != "none":
        for row in w.reshape(-1, np_):
            for _ in range(6):
                n = 2 if fill == "pairs" else int(rng.integers(1, 40))
                at = (int(rng.integers(0, np_)) + np.arange(n)) % np_
                row[at] = rng.random(n) * (rng.random(n) < 0.9)
    mass = rng.random((nodes, nt, np_))
    dm = icp.DeviceArray(ctx, mass.size).upload(mass.reshape(-1))
    dw = icp.DeviceArray(ctx, w.size).upload(w.reshape(-1))
    out = icp.DeviceArray(ctx, nt * np_)
    icp.check(icp.LIB.icp_atlas_compose(ctx.handle, nodes, nt, np_, dm.ptr, dw.ptr, out.ptr))
    assert np.array_equal(out.download().reshape(nt, np_), AO.compose(mass, w))
