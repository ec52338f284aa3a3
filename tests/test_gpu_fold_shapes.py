"""Folded records at candidate counts around the warps of a block: the first candidates of a lattice
alone must give the reference's records of the whole, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from test_folded import NAMES, Z, _device_chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("candidates", [1, 2, 3, 32, 33])
def test_records_of_the_first_candidates(icp, candidates):
    name = NAMES[0]
    want = Z[f"{name}.records"]
    assert len(want) >= candidates
    count = int(want["compact_index"][candidates - 1]) + 1
    with icp.Context(0) as ctx:
        c = _device_chain(icp, ctx, name)
        dv = icp.DeviceArray(ctx, len(c.vertices), icp.VERTEX_DTYPE).upload(c.vertices)
        dp = icp.DeviceArray(ctx, len(c.patches), icp.PATCH_DTYPE).upload(c.patches)
        _, records, n, stats = icp.folded_prepare(ctx, dv, dp, count, c.incident, focal=c.focal)
        got = records.download()
    assert n == stats.candidates == candidates
    assert got.tobytes() == want[:candidates].tobytes()
