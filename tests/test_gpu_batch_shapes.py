"""Batched records at the shapes where the batch's launches change: stored CDFs in two strips, in
more strips and in one launch per record; default chunks of their smallest and largest size; with
and without the graph.  Every record equals the single-record entry's up to the order of the
binary64 histogram sums."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,np_,ct,cp,count,rays", [
    (36, 72, 36, 72, 3, (1, 33, 5000)),                # two strips; chunks of 64
    (180, 360, 90, 180, 5, (2000, 700, 64, 65, 9000)),
    (360, 720, 360, 720, 4, (3000, 1000, 1, 200)),     # more strips per record
    (900, 1800, 900, 1800, 2, (4000, 50)),             # one launch per record
    (35, 75, 7, 25, 2, (40_000, 63)),                  # odd divisors
])
@pytest.mark.parametrize("graph", [False, True])
def test_batch_equals_single_records(icp, ctx, nt, np_, ct, cp, count, rays, graph):
    specs = icp.batched_record_specs(count, seed=5, rays_max=1e6, rays_min=1e3)
    for sp, n in zip(specs, rays):
        sp.rays = n
    s = icp.batch_settings(nt, np_, ct, cp, max_internal_hits=10, use_graph=graph, precision=icp.ICP_FP64)
    out = icp.generate_drop_batch(ctx, specs, s)
    for i, sp in enumerate(specs):
        one = icp.generate_drop_record(ctx, sp.coefficients, sp.radius_mm, sp.interior_index, nt, np_, sp.rays,
                                       seed=sp.seed, inclination_deg=sp.inclination_deg, ct=ct, cp=cp,
                                       max_internal_hits=10, precision=icp.ICP_FP64, wavelength_nm=sp.wavelength_nm,
                                       diffraction=sp.diffraction)
        # sums of the same terms in another order: 1e5 rounding errors of 2^-53 at most
        assert np.allclose(out.phi[i], one.phi, rtol=0, atol=1e-11)
        assert np.allclose(out.theta[i], one.theta, rtol=0, atol=1e-11)
        assert out.reports[i].trace.outputs == one.report.trace.outputs
        assert out.reports[i].projected_area_mm2 == one.report.projected_area_mm2
