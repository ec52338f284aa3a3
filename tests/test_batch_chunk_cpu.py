"""The chunk of a batched launch (host/icp_batch_chunk.hpp), compiled with g++: by ray count between
64 and 1024; a given or tuned size bounds it, so that a size tuned on a large batch leaves a small
one its eight chunks per warp and is never larger than asked for."""
from __future__ import annotations

import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "icp_batch_chunk.hpp"
int main(int, char** v)
{
    printf("%u\n", icp::host::batch_chunk((uint32_t)atoll(v[1]), (uint64_t)atoll(v[2]), (uint64_t)atoll(v[3])));
    return 0;
}
"""


@pytest.fixture(scope="module")
def chunk(tmp_path_factory):
    d = tmp_path_factory.mktemp("chunk")
    (d / "chunk.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "ice_crystal_phase_b200" / "host"), str(d / "chunk.cpp"),
                    "-o", str(d / "chunk")], check=True)
    return lambda *a: int(subprocess.run([str(d / "chunk"), *map(str, a)], check=True, capture_output=True, text=True).stdout)


WARPS = 148 * 32


@pytest.mark.parametrize("rays,want", [(1, 64), (160_000, 64), (64 * 8 * WARPS + 8 * WARPS, 65), (16_000_000, 422),
                                       (1024 * 8 * WARPS, 1024), (2 ** 40, 1024)])
def test_by_ray_count(chunk, rays, want):
    assert chunk(0, rays, WARPS) == want


@pytest.mark.parametrize("most", [32, 1024, 2048, 8192, 32768, 65536])
@pytest.mark.parametrize("rays", [1, 160_000, 16_000_000, 110_000_000, 2 ** 40])
def test_given_size_is_a_bound(chunk, most, rays):
    got = chunk(most, rays, WARPS)
    assert got <= most
    if got < most:  # shortened to no less than eight chunks per warp ask for
        assert got == max(64, rays // (8 * WARPS))
    # a tuned size does not starve the warps of any batch
    assert got == 32 or got <= max(64, rays // (8 * WARPS))
