"""The patch query's warp-wide forms at the sizes where they can go wrong: direction counts around a
warp, several rays' candidates in one queue, more roots per direction than the counting pass keeps,
boxes that cover every bin, faulty patches and directions.  Bit for bit against the brute-force oracle."""
from __future__ import annotations

import numpy as np
import pytest

import optics_cases as OC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("directions,copies,wide", [(1, 1, 0), (31, 1, 1), (33, 12, 0), (129, 3, 40), (2592, 12, 33)])
def test_query_bit_identical_to_oracle(icp, ctx, oracle, directions, copies, wide):
    v, (w, h, e) = OC.patch_lattice(21)
    _, pa, bx, _ = oracle.patch_build(v, w, h, e)
    pa, bx = np.tile(pa, copies), np.tile(bx, copies)
    pa["patch_id"] = np.arange(len(pa))[::-1]
    rng = np.random.default_rng(directions)
    for k in rng.choice(len(pa), wide, replace=False):     # these patches' caps are the whole sphere
        for a in "xyz":
            bx["min_" + a][k], bx["max_" + a][k] = -2.0, 2.0
    pa["vertex_indices"][len(pa) // 2, 3] = len(v)         # no such vertex
    dirs = np.asarray(icp.query_directions(36, 72, np.float32(OC._K20), np.float32((0, 0, 1)))).reshape(-1, 3)
    dirs = dirs[rng.permutation(len(dirs))[:directions]].copy()
    if directions > 31:
        dirs[7] = np.nan
        dirs[30] *= np.float32(1.3)
    got = icp.patch_query(ctx, v, pa, bx, dirs)
    off, sm, hits = oracle.patch_query(v, pa, bx, dirs)
    assert np.array_equal(got.offsets, off)
    assert got.summaries.tobytes() == sm.tobytes()
    assert got.hits.tobytes() == hits.tobytes()
