"""Table-II diffraction on grids whose windows stress the filter's tiling: a window wider than one
weight table (full circles near a pole), a partial last block of columns, label masks of a full
circle and of a part of one, both seams.  Oracle and tolerances of test_zzz_gpu_rainbow."""
from __future__ import annotations

import math

import numpy as np
import pytest

import rainbow_cases as RC
from test_zzz_gpu_rainbow import counts, mismatches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,np_,sigma_deg,support,primary,secondary", [
    (9, 3301, 6.0, 4.0, 150.0, 25.0),   # full circles of 1651 offsets: more than one table
    (64, 127, 2.0, 4.0, 138.0, 129.0),  # one block, one column short of full
    (64, 129, 2.0, 4.0, 138.0, 129.0),  # a second block of one column
    (48, 400, 3.0, 8.0, 165.0, 15.0),   # wide support: circles at the poles, parts elsewhere
    (300, 256, 0.7, 4.0, 138.0, 129.0),
    (2, 3, 20.0, 2.0, 90.0, 90.0),
])
def test_windows_match_oracle(icp, ctx, oracle, nt, np_, sigma_deg, support, primary, secondary):
    f = RC.bow_grid(nt, np_, 41, primary_deg=primary, secondary_deg=secondary, invalid=0.0005)
    cfg = (sigma_deg * math.pi / 180, support, 0.25, 0.75 * support)
    out = icp.rainbow_diffraction(ctx, f, nt, np_, icp.DiffractionConfig(*cfg))
    edges = oracle.rainbow_detect(f, nt, np_, cfg)
    assert np.array_equal(out.transitions, edges)
    rng = np.random.default_rng(3)
    pick = np.unique(rng.integers(0, nt * np_, 1500)) if nt * np_ > 3000 else np.arange(nt * np_)
    want = oracle.rainbow_filter_at(f, edges, nt, np_, cfg, pick)
    assert not mismatches(out.results[pick], want), mismatches(out.results[pick], want)
    assert out.stats == counts(out.transitions, out.results)
