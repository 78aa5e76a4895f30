"""CPU test: without a device the standalone stages report the CUDA error that
they met, not a lack of memory."""
import ctypes as C

import pytest

from pbf_gb300 import _capi
from tests.conftest import HAS_GPU


@pytest.mark.skipif(HAS_GPU, reason="checks the no-device path")
def test_standalone_stages_report_the_cuda_error(product_lib):
    buf = [(C.c_uint32 * 4)() for _ in range(3)]
    a, b, c = (C.addressof(x) for x in buf)
    assert product_lib.pbf_find_cells(a, 4, 4, b, c, None) == _capi.PBF_ERR_CUDA
    message = product_lib.pbf_last_error(None)
    assert b"pbf_find_cells" in message and b"memory" not in message
    assert product_lib.pbf_radix_sort(a, b, c, 4, 8, None) == _capi.PBF_ERR_NO_DEVICE
