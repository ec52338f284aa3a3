"""Batched FP32 records over the range of the default chunk: its smallest size, sizes between and its
largest (one block per SM keeps the ray counts small), against chunks of 32 of the same kernel --
the same rays, summed in another order -- and after the autotuner, whose sizes are bounds."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b, rays):
    for i, n in enumerate(rays):
        assert a.reports[i].trace.rays == b.reports[i].trace.rays == n
        assert a.reports[i].trace.outputs == b.reports[i].trace.outputs
        # the same binary64 terms in another order: at most 2^25 of them, 2^-53 each
        assert np.allclose(a.phi[i], b.phi[i], rtol=0, atol=1e-8)
        assert np.allclose(a.theta[i], b.theta[i], rtol=0, atol=1e-8)


@pytest.mark.parametrize("rays", [
    (1, 70_000, 33),                   # chunks of 64
    (900_000, 640_000, 63),            # 148 SMs of 8 warps: 162
    (6_000_000, 5_000_000, 100_001),   # 1024, the largest
])
@pytest.mark.parametrize("graph", [False, True])
def test_default_chunks(icp, ctx, rays, graph):
    specs = icp.batched_record_specs(len(rays), seed=9, rays_max=1e6, rays_min=1e3)
    for sp, n in zip(specs, rays):
        sp.rays = n
    kw = dict(max_internal_hits=4, precision=icp.ICP_FP32, use_graph=graph, blocks_per_sm=1)
    grid = (60, 120, 30, 60)
    _same(icp.generate_drop_batch(ctx, specs, icp.batch_settings(*grid, **kw)),
          icp.generate_drop_batch(ctx, specs, icp.batch_settings(*grid, chunk_rays=32, **kw)), rays)


def test_after_the_autotuner(icp):
    rays = (400_000, 300_000, 77)
    with icp.Context(0) as ctx:
        specs = icp.batched_record_specs(len(rays), seed=9, rays_max=1e6, rays_min=1e3)
        for sp, n in zip(specs, rays):
            sp.rays = n
        kw = dict(max_internal_hits=4, precision=icp.ICP_FP32, use_graph=False)
        plain = icp.generate_drop_batch(ctx, specs, icp.batch_settings(60, 120, 30, 60, **kw))
        tuned = icp.batch_settings(60, 120, 30, 60, **kw)
        assert icp.autotune_drop_batch(ctx, specs, tuned) > 0
        assert tuned.block_threads in (128, 256) and tuned.chunk_rays in (1024, 2048, 8192, 32768)
        _same(icp.generate_drop_batch(ctx, specs, icp.batch_settings(60, 120, 30, 60, **kw)), plain, rays)
        _same(icp.generate_drop_batch(ctx, specs, tuned), plain, rays)
