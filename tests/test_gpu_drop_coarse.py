"""Drop records on grids of few cells, on both sides of the line where a block keeps the grid in a
shared table: the same exits as straight into the histogram, summed in another order."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp64,nt,np_", [(False, 2, 3), (False, 8, 8), (False, 16, 96), (False, 29, 53), (False, 33, 47),
                                         (True, 2, 3), (True, 16, 32), (True, 27, 19)])
@pytest.mark.parametrize("coefficients", [(0.0,) * 8, (0.0, -0.08, -0.02, 0.005, 0.0, 0.0, 0.0, 0.0)])
def test_table_equals_histogram(icp, ctx, fp64, nt, np_, coefficients):
    rays = 50_001
    out = [icp.generate_drop_record(ctx, list(coefficients), 1.5, 1.335, nt, np_, rays, seed=17, inclination_deg=30.0,
                                    max_internal_hits=20, precision=icp.ICP_FP64 if fp64 else icp.ICP_FP32,
                                    diffraction=False, tuning=icp.Tuning(0, 0, slots, 0)) for slots in (0, 1, 64)]
    for r in out[1:]:
        assert r.report.trace.outputs == out[0].report.trace.outputs
        # the same terms of at most 2^20 in another order, 2^-53 each; the table's are exact
        assert np.allclose(r.phi, out[0].phi, rtol=0, atol=2e-10)
        assert np.allclose(r.theta, out[0].theta, rtol=0, atol=2e-10)
