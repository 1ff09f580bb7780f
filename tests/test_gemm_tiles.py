"""CPU: the sizes of the GPU tests run every tile of the QGEMM that its rule can choose, so that a change of the table of times cannot
move the choice away from what is tested."""
import ctypes

import pytest

from test_gpu_matmul import TILE_KS, TILE_SIZES

SMS = 148


def tile(pkg, scheme, scale_mode, rows, K, M):
    t = (ctypes.c_int * 3)()
    assert pkg.lib().inkq_debug_gemm_tile(SMS, scheme, scale_mode, rows, K, M, t) == pkg.OK
    return t[0]


@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("scale_mode", [0, 1])
@pytest.mark.parametrize("K", TILE_KS)
def test_gpu_sizes_cover_every_tile_that_is_chosen(pkg, scheme, scale_mode, K):
    """Tiles are multiples of 32 weight rows and of 8 activation rows: the grid holds every choice up to 24576 by 2048."""
    pkg.build()
    chosen = {}
    for rows in range(32, 24576 + 1, 32):
        for M in range(40, 2048 + 1, 8):
            chosen.setdefault(tile(pkg, scheme, scale_mode, rows, K, M), (M, rows))
    tested = {tile(pkg, scheme, scale_mode, n, K, m) for m, n in TILE_SIZES}
    assert {t: size for t, size in chosen.items() if t not in tested} == {}


@pytest.mark.parametrize("bad", [(0, 0, 0, 64, 64, 33), (SMS, -1, 0, 64, 64, 33), (SMS, 3, 0, 64, 64, 33), (SMS, 0, 2, 64, 64, 33), (SMS, 0, 0, 0, 64, 33),
                                 (SMS, 0, 0, 64, 32, 33), (SMS, 0, 0, 64, 64, 32)])
def test_tile_of_bad_arguments_is_refused(pkg, bad):
    pkg.build()
    assert pkg.lib().inkq_debug_gemm_tile(*bad, (ctypes.c_int * 3)()) == pkg.ERR_INVALID
    assert pkg.lib().inkq_debug_gemm_tile(SMS, 0, 0, 64, 64, 33, None) == pkg.ERR_INVALID
