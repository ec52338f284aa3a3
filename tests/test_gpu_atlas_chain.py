"""Atlas nodes at the ray counts and encounter limits where the trace changes its form: a warp per ray
(16 encounters at a time) up to some thousands of rays, rays spread over the warps above, against the
oracle's node.  Tolerances as for the other nodes: counts exact, the escaped sum to 1e-14."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("subdivisions,hits", [(1, 2048), (2, 1), (2, 15), (2, 16), (2, 17), (2, 33), (5, 2048),
                                               (11, 2048), (11, 17)])
def test_node_matches_oracle(ctx, icp, subdivisions, hits):
    from oracle import oracle as O
    from ice_crystal_phase_b200 import atlas as A

    n, nt, np_ = icp.evaluate_ice_optics(400.0).n, 20, 40
    s = A.settings(0.08, 0.3, n, 2, 1, nt, np_, subdivisions, max_internal_hits=hits)
    rep, mass = icp.AtlasNodeReport(), icp.DeviceArray(ctx, nt * np_)
    rc = icp.LIB.icp_atlas_trace_node(ctx.handle, C.byref(s), 1, 1, mass.ptr, C.byref(rep))
    node = icp.atlas_incident_node(2, 1, 1, 1)
    faces, pts, w = icp.atlas_area_rule(0.08, 0.3, list(node.rule_ki), subdivisions)
    ref, st = O.atlas_node(0.08, 0.3, n, list(node.ki), list(node.e0), list(node.e1), faces, pts, w, nt, np_, max_hits=hits)
    assert (rc == 0) == (st[6] == -1)
    assert (rep.rays, rep.outputs, rep.first_rejected) == (st[2], st[3], st[6])
    assert rep.escaped_mm2 == pytest.approx(st[0], rel=1e-14)
    assert rep.unresolved_mm2 == pytest.approx(st[1], rel=1e-13, abs=1e-18)
    if rc == 0:
        got = mass.download().reshape(nt, np_)
        assert np.array_equal(got > 0, ref > 0)
        assert np.abs(got - ref).sum() / ref.sum() <= 2e-11
