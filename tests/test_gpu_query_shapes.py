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


@pytest.mark.parametrize("size", [1e-5, 3e-3, 0.05, 0.5])
def test_caps_cover_poles_and_seam(icp, ctx, oracle, size):
    """Quads of every size at the poles, across the +-pi seam, on bin edges and anywhere, queried inside,
    on their corners and next to them."""
    rng = np.random.default_rng(int(1 / size))
    n = 400
    c = rng.normal(size=(n, 3))
    c[:60] = [0, 0, 1] * rng.choice([-1, 1], (60, 1)) + size * rng.normal(size=(60, 3)) * rng.choice([0, 1], (60, 1))
    c[60:120, 1] = size * rng.normal(size=60)
    c[60:120, 0] = -np.abs(c[60:120, 0])
    row, col = rng.integers(1, 256, 60) * np.pi / 256, rng.integers(0, 512, 60) * np.pi / 256 - np.pi
    c[120:180] = np.stack([np.sin(row) * np.cos(col), np.sin(row) * np.sin(col), np.cos(row)], -1)
    c /= np.linalg.norm(c, axis=1, keepdims=True)
    a = np.cross(c, rng.normal(size=(n, 3)))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    b = np.cross(c, a) * rng.uniform(0.05, 1, (n, 1))
    q = c[:, None] + size * np.stack([-a - b, a - b, b - a, a + b], 1) * rng.uniform(0.6, 1, (n, 4, 1))
    q = (q / np.linalg.norm(q, axis=2, keepdims=True)).astype(np.float32)
    v = np.zeros(4 * n, icp.VERTEX_DTYPE)
    v["direction"] = q.reshape(-1, 3)
    pa, bx = np.zeros(n, icp.PATCH_DTYPE), np.zeros(n, icp.AABB_DTYPE)
    pa["vertex_indices"] = np.arange(4 * n).reshape(n, 4)
    pa["patch_id"], pa["status"] = np.arange(n), 1
    for k, x in enumerate("xyz"):
        bx["min_" + x], bx["max_" + x] = q[:, :, k].min(1) - np.float32(1e-6), q[:, :, k].max(1) + np.float32(1e-6)
    s, t = rng.choice([0.0, 1.0, 0.5, 0.3, -0.01, 1.01], (2, n, 6, 1))
    d = ((1 - s) * q[:, None, 0] + s * q[:, None, 1]) * (1 - t) + ((1 - s) * q[:, None, 2] + s * q[:, None, 3]) * t
    d = np.concatenate([(d / np.linalg.norm(d, axis=2, keepdims=True)).reshape(-1, 3), np.eye(3), -np.eye(3)]).astype(np.float32)
    got = icp.patch_query(ctx, v, pa, bx, d)
    off, sm, hits = oracle.patch_query(v, pa, bx, d)
    assert np.array_equal(got.offsets, off)
    assert got.summaries.tobytes() == sm.tobytes()
    assert got.hits.tobytes() == hits.tobytes()
    assert len(hits) > n
