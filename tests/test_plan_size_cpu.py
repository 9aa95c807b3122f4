"""Workspace of plans on large grids (a host calculation, no kernel runs)."""

import ctypes

import pytest


@pytest.fixture(scope="module")
def lib():
    from crocodile_gb300 import _lib, build
    try:
        build.build()
    except RuntimeError as e:  # no nvcc in this environment
        pytest.skip(str(e))
    return _lib


@pytest.mark.parametrize("sep", [1, 0])
@pytest.mark.parametrize("S", [1, 3, 5, 8, 9, 12, 13, 14, 16, 17, 32])
@pytest.mark.parametrize("N", [24000, 32768, 40000, 65536])
@pytest.mark.parametrize("n", [0, 1000, 400000, 2000000, 40000000])
def test_lists_stay_within_the_buckets(lib, N, S, sep, n):
    """At most 2^24 buckets (some more where blocks of 32 x 32 tiles pad a side): 8
    bytes each and 24 for a tile's items, beside 44 bytes for a visibility and 16 for
    an item of 32."""
    kd = lib.KernelDesc(sep, 8, S, 4)
    size = lib.lib().cg_plan_workspace_bytes(lib.CG_PLAN_TILED, n, N, N, ctypes.byref(kd))
    assert 0 < size <= 1.1 * 2 ** 24 * (8 + 24) + n * (44 + 0.5) + 2 ** 20
