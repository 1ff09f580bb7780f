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


def test_call6_hands_over_every_argument(pkg):
    """Addresses above 2^63, null, and the extremes of the two ints arrive as they were given; so does the status."""
    call6 = pkg._load_call6()
    if call6 is None:
        pytest.skip("built without the interpreter's headers")
    seen = []

    @C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_int)
    def record(*args):
        seen.append(tuple(0 if a is None else a for a in args))
        return -len(seen)

    fn = C.cast(record, C.c_void_p).value
    calls = [(1, 2, 3, 4, 5, 6), (0, 0, 0, 0, 0, 0), (2**64 - 1, 2**63, 2**32, -(2**31), 2**47 + 8, 2**31 - 1)]
    for i, args in enumerate(calls):
        assert call6(fn, *args) == -(i + 1)
    assert seen == calls


@pytest.mark.gpu
@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("M,N,K", [(1, 264, 448), (5, 264, 448), (37, 72, 64)])
def test_linear_gives_the_bits_of_the_ctypes_call(pkg, gpu, scheme, M, N, K):
    """Context.linear (through the CPython entry where it was built) and the same function through ctypes, with a padded ldc."""
    import torch
    w = pkg.synth.weights(N, K, 5)
    wh = gpu.weight(scheme, 1, w["nib"], w["d"], w["m"] if scheme == 0 else None, w["zp"] if scheme == 2 else None)
    x = torch.from_numpy(pkg.synth.activations(M, K, 5)).cuda()
    ldc = N + (8 if M > 1 else 0)
    a, b = (torch.full((M + 1, ldc), -5.0, device="cuda") for _ in range(2))
    gpu.linear(wh, x, M, a, ldc)
    gpu.check(gpu.L.inkq_linear(gpu.h, wh.h, C.c_void_p(x.data_ptr()), M, C.c_void_p(b.data_ptr()), ldc))
    gpu.synchronize()
    assert torch.equal(a, b) and bool((a[:M, :N] != -5.0).any()) and bool((a[M] == -5.0).all()) and bool((a[:, N:] == -5.0).all())
    with pytest.raises(pkg.InkqError) as e:
        gpu.linear(wh, x, M, a, N - 8)
    assert e.value.code == pkg.ERR_INVALID
