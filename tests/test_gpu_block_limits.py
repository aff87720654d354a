"""GPU tests of the sizes of the three-body blocks: the scratch of their numbering at counts beyond 32 bits."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def test_scan_scratch_grows_with_the_count():
    from dftd3 import library
    size = getattr(ctypes.CDLL(str(library._LIBPATH)), "_ZN2d319atm_scan_temp_bytesEx")    # d3::atm_scan_temp_bytes
    size.argtypes, size.restype = [ctypes.c_longlong], ctypes.c_size_t
    counts = [1 << 20, 10 ** 9, (1 << 31) - 2, (1 << 31) + 16, 5 * (1 << 29), 1 << 33]
    sizes = [size(n) for n in counts]
    assert 0 < sizes[0] < sizes[1] < sizes[2] <= sizes[3] < sizes[4] < sizes[5]
