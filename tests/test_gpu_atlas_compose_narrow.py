"""Cyclic composition of narrow rows, on both sides of the lines between its kernels, with full, sparse
and empty coupling rows.  The oracle adds in the same order, so the masses are equal bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import atlas_oracle as AO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,np_", [(2, 128), (2, 255), (2, 256), (2, 257), (443, 256), (444, 256), (500, 128), (500, 129),
                                    (500, 200), (591, 256), (592, 256), (592, 128), (592, 129), (3, 1), (3, 32), (3, 33)])
@pytest.mark.parametrize("fill", ["runs", "every second", "one row"])
def test_compose_equals_oracle(icp, ctx, nt, np_, fill):
    rng = np.random.default_rng(np_ + nt)
    nodes = 3
    w = np.zeros((nodes, 2, np_))
    if fill == "every second":  # the most entries that a row can have
        w[1, :, ::2] = rng.random(w[1, :, ::2].shape)
    else:  # rows with and without entries between them
        for row in w.reshape(-1, np_)[:: 1 if fill == "runs" else 4]:
            for _ in range(6):
                n = int(rng.integers(1, 12))
                row[(int(rng.integers(0, np_)) + np.arange(n)) % np_] = rng.random(n)
    mass = rng.random((nodes, nt, np_))
    dm = icp.DeviceArray(ctx, mass.size).upload(mass.reshape(-1))
    dw = icp.DeviceArray(ctx, w.size).upload(w.reshape(-1))
    out = icp.DeviceArray(ctx, nt * np_)
    icp.check(icp.LIB.icp_atlas_compose(ctx.handle, nodes, nt, np_, dm.ptr, dw.ptr, out.ptr))
    assert np.array_equal(out.download().reshape(nt, np_), AO.compose(mass, w))
