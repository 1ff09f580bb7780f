"""GPU: QGEMV, tensor-core QGEMM and the CUDA-core cross-check, through the C ABI,
against the oracle and the reference's golden outputs.
 - every int32 block dot: exact
 - QGEMM fp32 output: bit-identical to the reference order
 - QGEMV fp32 output: within 5e-4 of the oracle in the measure of conftest.rel_err
   (8 K-slices summed in ascending order; documented in csrc/qgemv.cu); the project
   tolerance is 1e-3
 - fp16 lm_head: within 1e-3 of the exact (double-accumulated) value
"""
import numpy as np
import pytest

from conftest import f16, rel_err

pytestmark = pytest.mark.gpu

GEMV_TOL = 5e-4
SCHEMES = {0: ("A81W41", 2, 1), 1: ("A80W40", 0, 0), 2: ("A80W4Z", 0, 0)}  # scheme -> (name, gemm qmode, gemv qmode)


def setup(pkg, gpu, oracle, scheme, M, N, K, scale_mode, seed=0, qmode=None):
    import torch
    x = pkg.synth.activations(M, K, 50 + seed)
    w = pkg.synth.weights(N, K, seed)
    if scale_mode == 0:
        w["d"] = (w["d"] * np.float32(1.0003)).astype(np.float32)
        w["m"] = (w["m"] * np.float32(0.9997)).astype(np.float32)
    wh = gpu.weight(scheme, scale_mode, w["nib"], w["d"], w["m"], w["zp"])
    act = gpu.act(M, K)
    xd = torch.from_numpy(x).cuda()
    gpu.quantize(act, xd, M, qmode)
    q, d, s = oracle.quantize(x, qmode)
    return x, w, wh, act, (q, d, s)


def oracle_out(oracle, scheme, qds, w, scale_mode, want_dots=False):
    q, d, s = qds
    dw = w["d"] if scale_mode == 0 else f16(w["d"])
    mw = w["m"] if scale_mode == 0 else f16(w["m"])
    return oracle.gemm(scheme, q, d, s if scheme == 0 else None, w["nib"], dw, mw if scheme == 0 else None,
                       w["zp"] if scheme == 2 else None, want_dots=want_dots)


# ------------------------------------------------------------------ QGEMV
@pytest.mark.parametrize("N,K", [(8, 64), (136, 512), (1024, 4096), (4096, 4096), (4096, 12288)])
@pytest.mark.parametrize("scheme", [0, 1, 2])
def test_gemv_matches_oracle(pkg, gpu, oracle, scheme, N, K):
    import torch
    qmode = SCHEMES[scheme][2] if scheme else 1
    x, w, wh, act, qds = setup(pkg, gpu, oracle, scheme, 1, N, K, 1, seed=scheme, qmode=qmode)
    C = torch.full((1, N + 8), -777.0, device="cuda")
    gpu.gemv(act, wh, C)
    gpu.synchronize()
    ref = oracle_out(oracle, scheme, qds, w, 1)
    got = C.cpu().numpy()
    assert np.all(got[0, N:] == -777.0)                      # nothing written past the output
    assert rel_err(got[:, :N], ref) < GEMV_TOL


def test_gemv_matches_reference_golden(pkg, gpu, golden):
    import torch
    g = golden("ref_gemv_a81w41_fp16.npz")
    N, K = g["nib"].shape[0], g["nib"].shape[1] * 2
    wh = gpu.weight(0, 1, g["nib"], g["d"], g["m"])
    act = gpu.act(1, K)
    gpu.quantize(act, torch.from_numpy(g["x"]).cuda(), 1, 1)
    C = torch.empty((1, N), device="cuda")
    gpu.gemv(act, wh, C)
    gpu.synchronize()
    assert rel_err(C.cpu().numpy(), g["C"]) < GEMV_TOL


# ------------------------------------------------------------------ int32 block dots
@pytest.mark.parametrize("tensor_core", [False, True])
@pytest.mark.parametrize("scheme,M,N,K", [(0, 1, 8, 64), (0, 5, 136, 256), (1, 13, 264, 192), (2, 37, 128, 512), (0, 130, 256, 128)])
def test_block_dots_exact(pkg, gpu, oracle, tensor_core, scheme, M, N, K):
    import torch
    qmode = 2 if scheme == 0 else 0
    x, w, wh, act, qds = setup(pkg, gpu, oracle, scheme, M, N, K, 1, seed=3, qmode=qmode)
    dots = torch.full((M, N, K // 32), 123456789, dtype=torch.int32, device="cuda")
    gpu.block_dots(act, wh, dots, tensor_core=tensor_core)
    gpu.synchronize()
    _, ref = oracle_out(oracle, scheme, qds, w, 1, want_dots=True)
    assert np.array_equal(dots.cpu().numpy(), ref)


# ------------------------------------------------------------------ QGEMM
@pytest.mark.parametrize("impl", ["simt", "tc"])
@pytest.mark.parametrize("scheme,scale_mode,M,N,K", [
    (0, 0, 2, 8, 64), (0, 0, 5, 136, 256), (0, 0, 6, 24, 128), (0, 0, 7, 16, 4096), (0, 0, 13, 136, 192),
    (0, 1, 16, 128, 256), (0, 0, 17, 264, 320), (0, 0, 129, 128, 128), (0, 0, 322, 384, 512),
    (1, 1, 6, 32, 256), (1, 1, 150, 200, 448), (2, 1, 5, 16, 64), (2, 1, 257, 136, 256)])
def test_gemm_bit_identical_to_oracle(pkg, gpu, oracle, impl, scheme, scale_mode, M, N, K):
    import torch
    qmode = 2 if scheme == 0 else 0
    x, w, wh, act, qds = setup(pkg, gpu, oracle, scheme, M, N, K, scale_mode, seed=M, qmode=qmode)
    ldc = N + 8
    C = torch.full((M + 1, ldc), -777.0, device="cuda")
    (gpu.gemm if impl == "tc" else gpu.gemm_simt)(act, wh, C, ldc)
    gpu.synchronize()
    got = C.cpu().numpy()
    ref = oracle_out(oracle, scheme, qds, w, scale_mode)
    assert np.all(got[:M, N:] == -777.0) and np.all(got[M] == -777.0)   # guard band untouched
    assert np.array_equal(got[:M, :N].view(np.uint32), ref.view(np.uint32)), f"max abs diff {np.abs(got[:M, :N] - ref).max()}"


@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("scale_mode", [0, 1])
@pytest.mark.parametrize("N,K", [(200, 64), (264, 448), (9736, 320)])     # few and many weight tiles, ragged last tile, partial last stages
def test_gemm_tile_edges(pkg, gpu, scheme, scale_mode, N, K):
    """Both sides of tile widths (8-row steps up to 32 rows, 8- and 16-row steps above) against the CUDA-core kernel."""
    import torch
    w = pkg.synth.weights(N, K, 7)
    if scale_mode == 0:
        w["d"] = (w["d"] * np.float32(1.0003)).astype(np.float32)
    wh = gpu.weight(scheme, scale_mode, w["nib"], w["d"], w["m"] if scheme == 0 else None, w["zp"] if scheme == 2 else None)
    x = torch.from_numpy(pkg.synth.activations(260, K, 7)).cuda()
    act = gpu.act(260, K)
    for M in (2, 8, 9, 16, 17, 24, 25, 32, 33, 48, 49, 64, 65, 127, 129, 260):
        C, ref = torch.full((M + 1, N), -5.0, device="cuda"), torch.empty((M, N), device="cuda")
        gpu.quantize(act, x, M, 2 if scheme == 0 else 0)
        gpu.gemm(act, wh, C, N)
        gpu.gemm_simt(act, wh, ref, N)
        gpu.synchronize()
        assert torch.equal(C[:M], ref) and bool((C[M] == -5.0).all()), M


@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("scale_mode", [0, 1])
@pytest.mark.parametrize("M,N,K", [(33, 504, 576), (257, 1000, 320), (33, 6136, 192), (65, 4096, 576), (49, 6144, 448), (65, 8184, 448), (193, 4096, 320),
                                   (65, 6144, 1088), (97, 6136, 448), (145, 6144, 320), (289, 4088, 320), (321, 4096, 192), (322, 12288, 320),
                                   (49, 24576, 64), (97, 24568, 64), (145, 12288, 192), (289, 8192, 192), (8, 19000, 320), (20, 19000, 192)])
def test_gemm_tile_shapes(pkg, gpu, scheme, scale_mode, M, N, K):
    """Narrow, ordinary and wide layers, ragged in rows, columns and stages."""
    import torch
    w = pkg.synth.weights(N, K, 11)
    wh = gpu.weight(scheme, scale_mode, w["nib"], w["d"], w["m"] if scheme == 0 else None, w["zp"] if scheme == 2 else None)
    x = torch.from_numpy(pkg.synth.activations(M, K, 11)).cuda()
    act = gpu.act(M, K)
    C, ref = torch.full((M + 1, N), -5.0, device="cuda"), torch.empty((M, N), device="cuda")
    gpu.quantize(act, x, M, 2 if scheme == 0 else 0)
    gpu.gemm(act, wh, C, N)
    gpu.gemm_simt(act, wh, ref, N)
    gpu.synchronize()
    assert torch.equal(C[:M], ref) and bool((C[M] == -5.0).all())


@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("scale_mode", [0, 1])
@pytest.mark.parametrize("M,N,K", [(41, 3848, 192), (77, 4088, 1088), (80, 3912, 576), (42, 21976, 64), (2, 18952, 64), (9, 18960, 320), (32, 18952, 576)])
def test_gemm_tiles_of_64_rows(pkg, gpu, scheme, scale_mode, M, N, K):
    """Tiles of 64 weight rows, and 64-row CTAs with up to 32 rows (A81W41 with two: 128-row ones) above 148 weight tiles."""
    test_gemm_tile_shapes(pkg, gpu, scheme, scale_mode, M, N, K)


@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("scale_mode", [0, 1])
@pytest.mark.parametrize("M,N,K", [(41, 6280, 576), (161, 12552, 192), (241, 15808, 64), (1572, 264, 448), (225, 18952, 64), (81, 3096, 576), (33, 9528, 320),
                                   (241, 7072, 192), (261, 4088, 320)])
def test_gemm_tiles_that_one_scheme_or_record_size_takes(pkg, gpu, scheme, scale_mode, M, N, K):
    """Sizes around the borders between tiles."""
    test_gemm_tile_shapes(pkg, gpu, scheme, scale_mode, M, N, K)


# (M, N) that with rows of each length K select every tile that layers of up to 24576 weight rows select with up to 2048 activation rows, in
# every combination of weight scheme and scale records (checked on the CPU by test_gemm_tiles.py).  Ragged in weight and activation rows.
TILE_SIZES = [(1569, 136), (1857, 136), (81, 3096), (125, 3096), (177, 3096), (197, 3096), (201, 3096), (321, 3096), (365, 3096), (389, 3096),
              (401, 3096), (441, 3096), (617, 3096), (821, 3096), (65, 5480), (125, 5480), (149, 5480), (197, 5480), (293, 5480), (341, 5480),
              (365, 5480), (41, 9736), (57, 9736), (321, 11640), (185, 12568), (365, 23960)]
# The longest rows: 129 pairs are more than two rounds of any tile's ring (at most 8 stages of 8 pairs) and leave a ragged last stage, so that
# every slot is refilled and every barrier passes both phases.
TILE_KS = [64, 320, 1088, 64 * 129]


def gemm_tile(gpu, scheme, scale_mode, N, K, M):
    """(index, weight rows, activation rows) of the tile that this device takes"""
    import ctypes
    import torch
    t = (ctypes.c_int * 3)()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    gpu.check(gpu.L.inkq_debug_gemm_tile(sms, scheme, scale_mode, N, K, M, t))
    return tuple(t)


def device_weight(gpu, scheme, scale_mode, N, K):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(N + K)
    nib = torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, device="cuda", generator=g)
    d = torch.rand((N, K // 32), device="cuda", generator=g) * 0.018 + 0.002
    m = torch.rand((N, K // 32), device="cuda", generator=g) * -0.1
    zp = torch.randint(0, 16, (N, K // 32), dtype=torch.uint8, device="cuda", generator=g)
    w = gpu.weight_dev(scheme, scale_mode, N, K, nib, d, m if scheme == 0 else None, zp if scheme == 2 else None)
    gpu.synchronize()
    return w


def assert_gemm_equals_simt(gpu, scheme, w, act, x, M, N):
    import torch
    C, ref = torch.full((M + 1, N), -5.0, device="cuda"), torch.empty((M, N), device="cuda")
    gpu.quantize(act, x, M, 2 if scheme == 0 else 0)
    gpu.gemm(act, w, C, N)
    gpu.gemm_simt(act, w, ref, N)
    gpu.synchronize()
    assert torch.equal(C[:M], ref) and bool((C[M] == -5.0).all()), (M, N)


@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("scale_mode", [0, 1])
@pytest.mark.parametrize("K", TILE_KS)
def test_gemm_every_tile(pkg, gpu, scheme, scale_mode, K):
    """Every tile against the CUDA-core kernel."""
    import torch
    M_max = max(m for m, _ in TILE_SIZES)
    x = torch.randn((M_max, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    act = gpu.act(M_max, K)
    for N in sorted({n for _, n in TILE_SIZES}):
        w = device_weight(gpu, scheme, scale_mode, N, K)
        for M in [m for m, n in TILE_SIZES if n == N]:
            assert_gemm_equals_simt(gpu, scheme, w, act, x, M, N)
        w.close()


@pytest.mark.parametrize("scheme", [1, 2])
@pytest.mark.parametrize("scale_mode", [0, 1])
@pytest.mark.parametrize("cols", range(40, 121, 8))
def test_gemm_tiles_of_schemes_without_mins(pkg, gpu, scheme, scale_mode, cols):
    """128 x 40 to 128 x 120 tiles, 8 warps of 16 rows by all columns: one on every SM, ragged in rows and stages, a column short and full,
    each slot of the ring filled more than twice."""
    import torch
    N, K = 18936, TILE_KS[-1]
    x = torch.randn((cols, K), device="cuda", generator=torch.Generator(device="cuda").manual_seed(cols))
    w, act = device_weight(gpu, scheme, scale_mode, N, K), gpu.act(cols, K)
    for M in (cols - 1, cols):
        assert gemm_tile(gpu, scheme, scale_mode, N, K, M)[1:] == (128, cols)
        assert_gemm_equals_simt(gpu, scheme, w, act, x, M, N)
    w.close()
    test_gemm_tile_shapes(pkg, gpu, scheme, scale_mode, cols - 1, 18936, 448)
    test_gemm_tile_shapes(pkg, gpu, scheme, scale_mode, cols, 18936, 64)


@pytest.mark.parametrize("scale_mode", [0, 1])
@pytest.mark.parametrize("M,N,K", [(88, 18936, 448), (81, 18944, 64), (345, 4088, 1088), (322, 4088, 4160), (352, 4096, 576)])
def test_gemm_tile_with_a_short_column_of_warps(pkg, gpu, scale_mode, M, N, K):
    """128 x 88 tiles of A81W41: their last columns belong to the next tile, which may be ragged."""
    assert gemm_tile(gpu, 0, scale_mode, N, K, M)[1:] == (128, 88)
    test_gemm_tile_shapes(pkg, gpu, 0, scale_mode, M, N, K)


@pytest.mark.parametrize("scheme", [0, 1, 2])
@pytest.mark.parametrize("scale_mode", [0, 1])
@pytest.mark.parametrize("M,N,K", [(4, 20480, 320), (5, 28416, 64), (32, 28416, 576), (5, 28424, 64), (20, 34816, 320), (9, 37888, 64), (2, 37896, 64),
                                   (32, 37896, 576)])
def test_gemm_up_to_32_rows_of_wide_layers(pkg, gpu, scheme, scale_mode, M, N, K):
    """Both sides of three 64-row CTAs on every SM (444 of them) and of two 128-row ones (296), and up to four rows."""
    test_gemm_tile_shapes(pkg, gpu, scheme, scale_mode, M, N, K)


@pytest.mark.parametrize("M", [8, 32])
def test_gemm_up_to_32_rows_needs_no_second_wave(pkg, gpu, M):
    """28416 weight rows are three 64-row CTAs on every SM.  256 rows more would be a fourth on some, a second pass over K: 1.4 and 1.7
    times the time.  As 128-row CTAs they all fit at once: 1.1 and 1.15 times."""
    import torch
    K, best = 4096, []
    for N in (28416, 28672):
        g = torch.Generator(device="cuda")
        g.manual_seed(1)
        ws = [gpu.weight_dev(pkg.A81W41, pkg.SCALES_F16, N, K, torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, device="cuda", generator=g),
                             torch.rand((N, K // 32), device="cuda", generator=g), torch.rand((N, K // 32), device="cuda", generator=g)) for _ in range(3)]
        act, C = gpu.act(M, K), torch.empty((M, N), device="cuda")
        gpu.quantize(act, torch.randn((M, K), device="cuda", generator=g), M, pkg.Q8_1_F32)
        times = []
        for _ in range(8):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            for i in range(30):
                gpu.gemm(act, ws[i % 3], C, N)
            t1.record()
            torch.cuda.synchronize()
            times.append(t0.elapsed_time(t1))
        best.append(min(times[2:]))
        for w in ws:
            w.close()
    assert best[1] < 1.3 * best[0], best


@pytest.mark.parametrize("scheme", [1, 2])
def test_gemm_of_short_rows_costs_no_more_without_mins(pkg, gpu, scheme):
    """Short rows of many tiles per SM: the set-up and the stores of a tile, which do not depend on K, decide between tiles of one and of two
    CTAs per SM.  A layer without mins has less to compute than one with them (0.88 and 0.94 of its time; 1.10 and 1.15 with the tile whose
    time is the least at K = 4096)."""
    import torch
    M, N, K, best = 818, 16832, 384, {}
    for s in (0, scheme):
        g = torch.Generator(device="cuda")
        g.manual_seed(2)
        nib = torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, device="cuda", generator=g)
        d = torch.rand((N, K // 32), device="cuda", generator=g) * 0.018 + 0.002
        zp = torch.randint(0, 16, (N, K // 32), dtype=torch.uint8, device="cuda", generator=g)
        w = gpu.weight_dev(s, pkg.SCALES_F32, N, K, nib, d, d if s == 0 else None, zp if s == 2 else None)
        act, C = gpu.act(M, K), torch.empty((M, N), device="cuda")
        gpu.quantize(act, torch.randn((M, K), device="cuda", generator=g), M, pkg.Q8_1_F32 if s == 0 else pkg.Q8_0_F16)
        times = []
        for _ in range(8):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            for _ in range(30):
                gpu.gemm(act, w, C, N)
            t1.record()
            torch.cuda.synchronize()
            times.append(t0.elapsed_time(t1))
        best[s] = min(times[2:])
        w.close()
    assert best[scheme] < 1.03 * best[0], best


@pytest.mark.parametrize("M", [2, 5, 6, 7, 13])
def test_gemm_matches_reference_golden(pkg, gpu, golden, M):
    import torch
    g = golden("ref_gemm_a81w41_fp32.npz")
    N, K = g["nib"].shape[0], g["nib"].shape[1] * 2
    wh = gpu.weight(0, 0, g["nib"], g["d"], g["m"])
    C = torch.empty((M, N), device="cuda")
    gpu.linear(wh, torch.from_numpy(g[f"x_M{M}"]).cuda(), M, C, N)      # the layer's forward(): quantize + QGEMM
    gpu.synchronize()
    assert np.array_equal(C.cpu().numpy().view(np.uint32), g[f"C_M{M}"].view(np.uint32))


def test_reference_throughput_recipe(pkg, gpu, golden):
    import torch
    g = golden("ref_testlinear_recipe.npz")
    N, K, M = g["nib"].shape[0], g["nib"].shape[1] * 2, g["x"].shape[0]
    wh = gpu.weight(0, 0, g["nib"], g["d"], g["m"])
    C = torch.empty((M, N), device="cuda")
    gpu.linear(wh, torch.from_numpy(g["x"]).cuda(), M, C, N)
    gpu.synchronize()
    assert np.array_equal(C.cpu().numpy().view(np.uint32), g["C"].view(np.uint32))


def test_a80w40_matches_reference_golden(pkg, gpu, golden):
    import torch
    g = golden("ref_a80w40.npz")
    N, K, M = g["nib"].shape[0], g["nib"].shape[1] * 2, g["x"].shape[0]
    wh = gpu.weight(1, 1, g["nib"], g["d"])
    C = torch.empty((M, N), device="cuda")
    gpu.linear(wh, torch.from_numpy(g["x"]).cuda(), M, C, N)
    gpu.synchronize()
    assert np.array_equal(C.cpu().numpy().view(np.uint32), g["C_gemm"].view(np.uint32))
    C1 = torch.empty((1, N), device="cuda")
    gpu.linear(wh, torch.from_numpy(g["x"][:1]).cuda(), 1, C1, N)
    gpu.synchronize()
    assert rel_err(C1.cpu().numpy(), g["C_gemv"]) < GEMV_TOL


# ------------------------------------------------------------------ full benchmark shape, properties + samples
def test_full_prefill_shape(pkg, gpu, oracle):
    """M=322, K=4096, N=12288 (the pp322 gate_proj shape): tensor-core result equals the
    CUDA-core cross-check everywhere and the oracle on sampled outputs; linear_host equals
    the device path; doubling the activations doubles the result exactly (power-of-two linearity)."""
    import torch
    M, N, K = 322, 12288, 4096
    x = pkg.synth.activations(M, K)
    w = pkg.synth.weights(N, K)
    wh = gpu.weight(0, 0, w["nib"], w["d"], w["m"])
    xd = torch.from_numpy(x).cuda()
    C = torch.empty((M, N), device="cuda")
    gpu.linear(wh, xd, M, C, N)
    act = gpu.act(M, K)
    gpu.quantize(act, xd, M, 2)
    C2 = torch.empty((M, N), device="cuda")
    gpu.gemm_simt(act, wh, C2, N)
    gpu.synchronize()
    assert torch.equal(C, C2)
    rng = np.random.default_rng(0)
    rows, cols = rng.integers(0, M, 4000), rng.integers(0, N, 4000)
    rows[:4], cols[:4] = [0, M - 1, 0, M - 1], [0, 0, N - 1, N - 1]
    q, d, s = oracle.quantize(x, 2)
    ref = oracle.gemm_samples(0, q, d, s, w["nib"], w["d"], w["m"], None, rows, cols)
    got = C.cpu().numpy()
    assert np.array_equal(got[rows, cols].view(np.uint32), ref.view(np.uint32))
    Ch = np.empty((M, N), np.float32)
    gpu.linear_host(wh, x, M, Ch, N)
    assert np.array_equal(Ch, got)
    C3 = torch.empty((M, N), device="cuda")
    gpu.linear(wh, xd * 2.0, M, C3, N)
    gpu.synchronize()
    assert torch.equal(C3, C * 2.0)


@pytest.mark.parametrize("scheme", [0, 1])
@pytest.mark.parametrize("M", [37, 97, 130, 322, 1100])
def test_linear_host_row_windows(pkg, gpu, scheme, M):
    """inkq_linear_host works on windows of rows from M = 96 on (activations in, quantizer + QGEMM, finished rows out, on
    three streams): ragged last window and last weight tile, padded host rows (ldc > N); equals the device path bit for
    bit, leaves the padding untouched, and a second call right behind the first does not disturb it."""
    import torch
    N, K, ldc = 1064, 128, 1072           # 9 weight tiles, the last one 40 rows
    w = pkg.synth.weights(N, K, 41)
    wh = gpu.weight(scheme, pkg.SCALES_F16, w["nib"], w["d"], w["m"] if scheme == 0 else None)
    x = pkg.synth.activations(M, K, 41)
    C = torch.empty((M, N), device="cuda")
    gpu.linear(wh, torch.from_numpy(x).cuda(), M, C, N)
    gpu.synchronize()
    Ch = np.full((M, ldc), -7.0, np.float32)
    gpu.linear_host(wh, x, M, Ch, ldc)
    assert np.array_equal(Ch[:, :N], C.cpu().numpy()) and (Ch[:, N:] == -7.0).all()
    x2 = pkg.synth.activations(M, K, 43)
    C2 = torch.empty((M, N), device="cuda")
    Ch2 = np.empty((M, N), np.float32)
    gpu.linear_host(wh, x2, M, Ch2, N)
    gpu.linear(wh, torch.from_numpy(x2).cuda(), M, C2, N)
    gpu.synchronize()
    assert np.array_equal(Ch2, C2.cpu().numpy())


def test_mismatched_quantizer_mode_is_rejected(pkg, gpu, oracle):
    import torch
    x, w, wh, act, _ = setup(pkg, gpu, oracle, 0, 4, 16, 64, 0, qmode=0)   # Q8_0 activations, A81W41 weights
    C = torch.empty((4, 16), device="cuda")
    with pytest.raises(pkg.InkqError) as e:
        gpu.gemm(act, wh, C, 16)
    assert e.value.code == pkg.ERR_INVALID
    with pytest.raises(pkg.InkqError):
        gpu.gemm(act, wh, C, 8)    # ldc < rows


# ------------------------------------------------------------------ weight-only W41 and fp16 lm_head
@pytest.mark.parametrize("M,N,K", [(9, 72, 256), (1, 256, 128), (1, 1064, 512), (1, 4096, 4096), (1, 512, 12288), (1, 6144, 576),   # M == 1: the streaming kernel (many rows, long rows) and the products
                                   # M = 2 .. 16: products in registers, ragged row tiles, fewer and more pairs than warps x depth
                                   (2, 72, 64), (8, 2440, 1088), (10, 136, 8256), (15, 24, 320), (16, 4808, 576), (16, 136, 12288),
                                   (16, 128, 64), (322, 384, 512), (200, 136, 1024), (400, 264, 192),
                                   # enough work items for the two-weight-tiles-per-CTA variant: an odd tile count (the last
                                   # group holds one tile), and two activation tiles of 160 rows
                                   (16, 297 * 128, 64), (300, 74 * 256, 128),
                                   # one and two weight tiles over several waves, tiles of fewer stages than slots, few stages of 256 rows
                                   (33, 297 * 128, 64), (17, 72, 192), (300, 19000, 320), (250, 18904, 448), (500, 38000, 128)])
def test_weight_only_w41(pkg, gpu, oracle, M, N, K):
    """Tensor-core kernel (kind::f16, fp32 accumulation inside tensor memory) and its CUDA-core cross-check against
    the oracle.  The dequantised fp16 weights are identical in all three (one rounding of q*d + m); only the fp32
    summation order differs: k ascending in the oracle and the cross-check, the hardware's in the tensor-core kernel."""
    import torch
    w = pkg.synth.weights(N, K, 4)
    a16 = pkg.synth.activations(M, K, 4).astype(np.float16)
    wh = gpu.weight(3, 1, w["nib"], w["d"], w["m"])
    a_dev = torch.from_numpy(a16).cuda()
    C = torch.full((M + 1, N), 7.0, device="cuda")
    gpu.gemm_w41_f16act(a_dev, M, wh, C, N)
    Cs = torch.empty((M, N), device="cuda")
    gpu.gemm_w41_f16act_simt(a_dev, M, wh, Cs, N)
    gpu.synchronize()
    ref = oracle.gemm_w41_f16act(a16, w["nib"], w["d"], w["m"])
    assert rel_err(Cs.cpu().numpy(), ref) < 1e-5
    # Another summation order moves an fp32 sum of K terms by a few ulps of the terms' magnitude, whatever the size
    # of the result, so the bound is relative to the output's rms (observed 2e-6), not to each element.
    got = C[:M].cpu().numpy()
    assert np.abs(got - ref).max() / np.sqrt(np.mean(ref.astype(np.float64) ** 2)) < 1e-4
    assert bool((C[M] == 7.0).all())                          # nothing stored past row M


def test_weight_only_w41_dequantisation_bits(pkg, gpu, oracle):
    """One-hot fp16 activations read the dequantised weights back out of both GPU kernels: they must be the oracle's
    single rounding of q*d + m bit for bit, also for scales of very different exponents."""
    import torch
    rng = np.random.default_rng(78)
    N, K = 256, 128
    q = rng.integers(0, 16, size=(N, K), dtype=np.uint8)
    d = (rng.uniform(0.5, 2.0, size=(N, K // 32)) * 2.0 ** rng.integers(-12, 4, size=(N, K // 32))).astype(np.float16).astype(np.float32)
    m = (rng.uniform(-2.0, 2.0, size=(N, K // 32)) * 2.0 ** rng.integers(-12, 4, size=(N, K // 32))).astype(np.float16).astype(np.float32)
    nib = pkg.synth.pack_nibbles(q)
    a16 = np.eye(K, dtype=np.float16)
    wh = gpu.weight(3, 1, nib, d, m)
    a_dev = torch.from_numpy(a16).cuda()
    C, Cs = torch.empty((K, N), device="cuda"), torch.empty((K, N), device="cuda")
    gpu.gemm_w41_f16act(a_dev, K, wh, C, N)
    gpu.gemm_w41_f16act_simt(a_dev, K, wh, Cs, N)
    gpu.synchronize()
    ref = oracle.gemm_w41_f16act(a16, nib, d, m)
    assert np.array_equal(C.cpu().numpy(), ref) and np.array_equal(Cs.cpu().numpy(), ref)


@pytest.mark.parametrize("M,N,K", [(1, 1000, 4096), (1, 16, 64), (5, 264, 512),
                                   # warp-level products: one and two passes of rows, ragged row tiles, more and fewer K steps than warps x depth
                                   (2, 1000, 4096), (8, 2408, 2560), (9, 40, 5120), (15, 24, 32), (3, 2400, 544), (4, 72, 40),
                                   (3, 1000, 4160), (1, 24, 544)])
def test_lm_head_f16(pkg, gpu, oracle, M, N, K):
    import torch
    w16 = pkg.synth.lm_head(N, K, 6)
    x = pkg.synth.activations(M, K, 6)
    wh = gpu.f16w(w16)
    C = torch.empty((M, N), device="cuda")
    gpu.f16w_matmul(wh, torch.from_numpy(x).cuda(), M, C, N)
    gpu.synchronize()
    assert rel_err(C.cpu().numpy(), oracle.lmhead_f16w(x, w16)) < 1e-3


@pytest.mark.parametrize("M,K", [(1, 512), (5, 512), (8, 1088), (9, 512), (15, 64), (16, 512), (33, 512), (1, 544), (4, 544)])
@pytest.mark.parametrize("weights", ["finite", "special"])
def test_lm_head_f16_rows_of_any_magnitude(pkg, gpu, M, K, weights):
    """Huge, tiny and subnormal rows keep their precision; infinities and NaNs appear in the outputs where a 64-bit
    evaluation has them.  M < 16 and M >= 16 are different kernels, K % 64 != 0 a third."""
    import torch
    if weights == "special" and M >= 16:
        pytest.skip("infinite weights with 16 and more rows are not part of the contract")
    N = 200
    g = torch.Generator(device="cuda")
    g.manual_seed(M * K)
    w = (torch.randn((N, K), device="cuda", generator=g) * 0.02).half()
    w[11] = 0.0
    if weights == "special":
        w[5, 8], w[6, K - 1], w[7, 3] = float("inf"), float("-inf"), float("nan")
        w[150, 1], w[150, 2] = float("inf"), float("-inf")
    wh = gpu.f16w_dev(w, N, K)
    base = torch.randn((K,), device="cuda", generator=g)
    base[7] = 0.0                                             # of a row without remainder there

    def spiked(**at):
        r = base.clone()
        for i, v in at.items():
            r[int(i[1:])] = v
        return r

    inf = float("inf")
    rows = [spiked(i7=1e34), spiked(i7=2e35), spiked(i7=3.3e38), spiked(i7=-3.4028234663852886e38), base * 1e-30, base * 1e-36, base * 1e-38, base * 1e-41, base * 0.0,
            spiked(i7=inf), spiked(i33=-inf), spiked(i3=inf, i9=-inf), spiked(i3=inf, i9=inf, i12=3e38), spiked(i60=float("nan")), base]
    if K % 64 == 0:                                           # (partial sums of the CUDA-core kernel may overflow here)
        rows += [base * 1e37, base * 1e38]

    def classes(t):
        return torch.where(t.isnan(), 3, torch.where(t == inf, 1, torch.where(t == -inf, 2, 0)))

    C = torch.empty((M, N), device="cuda")
    for i, r in enumerate(rows):
        x = base.repeat(M, 1)
        x[i % M] = r
        gpu.f16w_matmul(wh, x, M, C, N)
        gpu.synchronize()
        ref = x.double() @ w.double().t()
        assert torch.equal(classes(C), classes(ref.float())), (i, int((classes(C) != classes(ref.float())).sum()))
        ok = classes(ref.float()) == 0
        err = torch.where(ok, (C.double() - ref).abs(), 0.0)
        mag = x.double().abs() @ w.double().abs().t()         # sum of |x w|
        # M < 16: an element's split error 2^-23, fp32 sums of at most 32 + K/512 + 16 (CUDA cores: K/32 + 5) rounded or truncated
        # partials; one rounding of a subnormal result, for the CUDA cores of each product.  M >= 16: the hardware's accumulation,
        # as bounded in test_gpu_baseline_shapes.py, 2e-4 of the row's rms (finite rows only)
        if M < 16:
            bound = 2.0 ** -23 * 60 * mag + 2.0 ** -149 * (K if K % 64 else 1)
        else:
            bound = 2e-4 * ref.pow(2).mean(1, keepdim=True).sqrt() + 2.0 ** -149
        assert bool((~ok | (err <= bound)).all()), (i, float(torch.where(ok, err / bound, 0.0).max()))


@pytest.mark.parametrize("M,K", [(1, 64), (8, 64), (9, 64), (16, 64), (2, 40)])
def test_lm_head_f16_refuses_unaligned_activations(pkg, gpu, M, K):
    """Every kernel of the head reads the activations in 16-byte pieces: the host refuses a pointer that does not allow it."""
    import torch
    wh = gpu.f16w(pkg.synth.lm_head(16, K, 6))
    x = torch.zeros((M * K + 4,), device="cuda")
    C = torch.full((M, 16), -5.0, device="cuda")
    before = gpu.launches
    with pytest.raises(pkg.InkqError) as e:
        gpu.f16w_matmul(wh, x[1:], M, C, 16)
    gpu.synchronize()
    assert e.value.code == pkg.ERR_INVALID and gpu.launches == before and bool((C == -5.0).all())
    gpu.f16w_matmul(wh, x[4:], M, C, 16)
    gpu.synchronize()
    assert bool((C == 0.0).all())
