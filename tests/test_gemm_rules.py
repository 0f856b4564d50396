"""Host rules of the GEMM dispatch, asked of the built library (no GPU needed)."""
import ctypes
import os

import pytest

from oslo_b200 import ops

TILE = 256


@pytest.fixture(scope="module")
def lib():
    if not os.path.exists(ops.ext_path()):
        pytest.skip("extension not built")
    ops.load_ext(required=True)
    so = ctypes.CDLL(ops.ext_path())
    so.oslo_gemm_split_floats.restype = ctypes.c_longlong
    so.oslo_gemm_split_ranges.argtypes = [ctypes.c_int] * 4 + [ctypes.c_longlong]
    return so


@pytest.mark.parametrize("m, n, k", [(4864, 1024, 8192), (19456, 256, 8192), (768, 768, 8000), (3062, 2048, 8192), (4096, 768, 50264), (38400, 256, 8192)])
def test_ranges_of_k_fit_the_workspace_they_are_given(lib, m, n, k):
    """A workspace sized for one number of SMs and a launch on another (SMs reserved by another thread in between): the cut tiles'
    partial sums never need more than the workspace holds. 76 tiles: 2 are cut on 148 SMs, 6 on 140."""
    tiles = -(-m // TILE) * -(-n // TILE)
    cut = 0
    for sized in (148, 146, 144, 140, 132, 100, 8, 2):
        floats = lib.oslo_gemm_split_floats(m, n, k, sized)
        for sms in (148, 146, 144, 140, 132, 100, 8, 2):
            ranges = lib.oslo_gemm_split_ranges(m, n, k, sms, floats)
            assert ranges >= 1
            if ranges > 1:
                cut += 1
                assert tiles % (sms // 2) * ranges * TILE * TILE <= floats
        if floats:
            assert lib.oslo_gemm_split_ranges(m, n, k, sized, floats) > 1
        assert lib.oslo_gemm_split_ranges(m, n, k, sized, 0) == 1
    assert cut
