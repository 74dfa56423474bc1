"""Kernels that only one of the two libraries has (no GPU: their host entries' names)."""

import pytest


@pytest.mark.parametrize("precision, compiled", [("double", True), ("mixed", False)])
def test_warp_per_track_kernel_is_fp64_only(precision, compiled):
    """The mixed driver takes no steps with its warp's lanes, which would wait for them."""
    from celeritas_gb300.build import build

    with open(build(precision=precision), "rb") as f:
        assert (b"along_charged_warp_kernel" in f.read()) == compiled
