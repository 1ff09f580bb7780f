"""GPU: launches whose shared memory needs the opt-in beyond 48 KB.  The limit counts a kernel's static part too, and it is an
attribute of the function that all contexts and threads of a device share.  Without the opt-in a launch is refused on the
host (an error status), nothing runs."""
import ctypes as C
import importlib.util
import os
import shutil
import sys
import threading

import pytest

pytestmark = pytest.mark.gpu


def P(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("K", [37056, 37120, 37632, 37696])   # dynamic part 46,320 to 47,120 bytes + 768 or 784 static ones
def test_decode_gemv_rows_around_48_kb(pkg, gpu, K):
    import torch
    N = 128
    w = pkg.synth.weights(N, K, 3)
    wh = gpu.weight(pkg.A81W41, pkg.SCALES_F16, w["nib"], w["d"], w["m"])
    act, x = gpu.act(1, K), torch.from_numpy(pkg.synth.activations(1, K, 3)).cuda()
    ref, got = torch.empty((N,), device="cuda"), torch.empty((N,), device="cuda")
    gpu.quantize(act, x, 1, pkg.Q8_1_F16)
    gpu.gemv(act, wh, ref)
    gpu.check(gpu.L.inkq_glue_decode_gemv(gpu.h, wh.h, act.h, P(got), 0, None, C.c_float(0), None, pkg.Q8_1_F16, None))
    gpu.synchronize()
    assert torch.equal(got, ref)


@pytest.mark.parametrize("max_pos", [37600, 38400, 40320])    # scores of a share: the dynamic part is just below 48 KB, 2.6 KB are static
def test_decode_attention_contexts_around_48_kb(pkg, gpu, max_pos):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    nq, past, short = 4, 200, 512
    k, v = (torch.randn((1, short, 128), device="cuda", generator=g).half() for _ in range(2))
    q = torch.randn((1, nq * 128), device="cuda", generator=g)
    pos = torch.tensor([past], dtype=torch.int32, device="cuda")
    out = []
    for n in (short, max_pos):
        kc, vc = (torch.zeros((1, n, 128), dtype=torch.float16, device="cuda") for _ in range(2))
        kc[:, :short], vc[:, :short] = k, v
        o = torch.empty((1, nq * 128), device="cuda")
        gpu.check(gpu.L.inkq_glue_attention(gpu.h, P(q), P(kc), P(vc), P(pos), 1, nq, 1, n, C.c_float(0.088), P(o)))
        gpu.synchronize()
        out.append(o)
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("kind", ["head", "w41"])
def test_threads_with_long_and_short_rows(pkg, gpu, kind):
    """Two threads, each with its own context and stream, call the same kernel with different K."""
    import torch
    N, M, calls = 64, 8, 1500
    errors, wrong = [], []

    def work(K):
        try:
            stream = torch.cuda.Stream()
            ctx = pkg.Context(0, stream.cuda_stream)
            out = torch.empty((M, N), device="cuda")
            x = torch.from_numpy(pkg.synth.activations(M, K, 5)).cuda()
            if kind == "head":
                wh = ctx.f16w(pkg.synth.lm_head(N, K, 6))
            else:
                w = pkg.synth.weights(N, K, 7)
                wh, x = ctx.weight(pkg.W41, pkg.SCALES_F16, w["nib"], w["d"], w["m"]), x.half()
            torch.cuda.synchronize()

            def call():
                if kind == "head":
                    ctx.f16w_matmul(wh, x, M, out, N)
                else:
                    ctx.gemm_w41_f16act(x, M, wh, out, N)

            call()
            ctx.synchronize()
            first = out.clone()
            torch.cuda.synchronize()
            barrier.wait(timeout=60)
            for _ in range(calls):
                call()
            ctx.synchronize()
            if not torch.equal(out, first):
                wrong.append(K)
            ctx.close()
        except Exception as e:                      # noqa: BLE001 - reported by the test's own thread
            errors.append(f"K = {K}: {e}")
            barrier.abort()

    barrier = threading.Barrier(2)
    threads = [threading.Thread(target=work, args=(K,)) for K in (64, 5120)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and not wrong, (errors, wrong)


def test_two_copies_of_the_library_in_one_process(pkg, gpu, tmp_path):
    """Each copy has functions of its own and opts them in itself."""
    import torch
    src = os.path.dirname(os.path.abspath(pkg.__file__))
    for f in os.listdir(src):
        if f.endswith((".py", ".so")):
            shutil.copy(os.path.join(src, f), tmp_path)
    spec = importlib.util.spec_from_file_location("inkq_b200_copy", tmp_path / "__init__.py", submodule_search_locations=[str(tmp_path)])
    copy = importlib.util.module_from_spec(spec)
    sys.modules["inkq_b200_copy"] = copy
    try:
        spec.loader.exec_module(copy)
        N, K, M = 136, 5120, 40
        w, x = pkg.synth.weights(N, K, 7), torch.from_numpy(pkg.synth.activations(M, K, 5)).cuda()
        out = []
        for p, ctx in ((pkg, gpu), (copy, copy.Context(0, torch.cuda.current_stream().cuda_stream))):
            wh, w41, lm = ctx.weight(p.A81W41, p.SCALES_F16, w["nib"], w["d"], w["m"]), ctx.weight(p.W41, p.SCALES_F16, w["nib"], w["d"], w["m"]), ctx.f16w(pkg.synth.lm_head(N, K, 6))
            c = torch.zeros((6, M, N), device="cuda")
            ctx.linear(wh, x, M, c[0], N)
            for i, m in ((1, 8), (2, M)):
                ctx.gemm_w41_f16act(x.half(), m, w41, c[i], N)
            for i, m in ((3, 1), (4, M)):
                ctx.f16w_matmul(lm, x, m, c[i], N)
            ctx.linear(wh, x, 1, c[5], N)
            ctx.synchronize()
            out.append(c)
        assert torch.equal(*out)
    finally:
        del sys.modules["inkq_b200_copy"]
