"""The library version, which saved plans are kept by."""
from zorro_gb300 import _lib


def test_version_tells_plans_of_other_kernels_apart():
    """Plans measured on the Stockham transforms (version 100) are not the
    in-place transforms'."""
    assert _lib.load().zr_version() > 100
