"""The exact sampler's quick erf, log and exp equal the header's on every float, and its quick division equals
IEEE division wherever it answers (and answers wherever it says it does)."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fn", [0, 1, 2, 3])
def test_quick_forms_equal_what_they_stand_for(cuda_lib, fn):
    from bamf_gb300 import abi
    f = abi.lib().bamf_parity_math_check
    f.restype, f.argtypes = C.c_int, [C.c_int, C.POINTER(C.c_int64)]
    bad = C.c_int64(-1)
    abi.check(f(fn, C.byref(bad)), "bamf_parity_math_check")
    assert bad.value == 0
