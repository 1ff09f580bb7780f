"""The CPython entry for the shortest calls returns what the same function returns through ctypes."""
import ctypes as C

import pytest


@pytest.mark.parametrize("M,ldc", [(1, 8), (0, 8), (-1, 2**31 - 1)])
def test_call6_status_equals_ctypes(pkg, M, ldc):
    call6 = pkg._load_call6()
    if call6 is None:
        pytest.skip("built without the interpreter's headers")
    L = pkg.lib()
    fn = C.cast(L.inkq_linear, C.c_void_p).value
    want = L.inkq_linear(None, None, None, M, None, ldc)
    assert want != pkg.OK and call6(fn, 0, 0, 0, M, 0, ldc) == want
    with pytest.raises(TypeError):
        call6(fn, 0, 0)
    with pytest.raises(TypeError):
        call6(fn, 0, "w", 0, M, 0, ldc)
