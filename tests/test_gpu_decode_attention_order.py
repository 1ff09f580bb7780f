"""GPU: the decode attention that starts from the qkv row, called behind kernels that write its caches after they have let
their successor start (csrc/glue_ops.cu): inkq_glue_qkv_attention_quant may read nothing before the kernel in front of it is
done, and inkq_glue_decode_qkv_attention, which reads position and caches early, brings the product it stands behind itself.
Every sequence is run with and without a synchronisation between its calls: the bits are equal."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HD = 128
EPS, SCALE = C.c_float(1e-6), C.c_float(1.0 / np.sqrt(HD))
P = lambda t: C.c_void_p(t.data_ptr())


class Attention:
    """Caches, tables and norm weights of one layer, and its calls."""

    def __init__(self, pkg, gpu, nq, nkv, max_pos, seed):
        import torch
        self.torch, self.pkg, self.gpu, self.nq, self.nkv, self.max_pos = torch, pkg, gpu, nq, nkv, max_pos
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)
        self.width = (nq + 2 * nkv) * HD
        self.qn = torch.rand(HD, device="cuda", generator=self.g) + 0.5
        self.kn = torch.rand(HD, device="cuda", generator=self.g) + 0.5
        ang = torch.rand((max_pos, HD), device="cuda", generator=self.g) * 6.28
        self.cos, self.sin = torch.cos(ang), torch.sin(ang)
        self.kc0 = self.randn(nkv, max_pos, HD).half()
        self.vc0 = self.randn(nkv, max_pos, HD).half()
        self.q = torch.empty((64, nq * HD), device="cuda")
        self.positions = torch.arange(max_pos, dtype=torch.int32, device="cuda")
        self.outs = [gpu.act(1, nq * HD) for _ in range(17)]

    def randn(self, *shape):
        return self.torch.randn(shape, device="cuda", generator=self.g)

    def reset(self):
        self.kc, self.vc = self.kc0.clone(), self.vc0.clone()
        self.torch.cuda.synchronize()

    def _tables(self, pos):
        return P(self.qn), P(self.kn), P(self.cos), P(self.sin), P(self.positions[pos:])

    def append(self, qkv, pos):
        self.gpu.check(self.gpu.L.inkq_glue_qknorm_rope_cache(self.gpu.h, P(qkv), *self._tables(pos), qkv.shape[0], self.nq, self.nkv, self.max_pos,
                                                              EPS, P(self.q), P(self.kc), P(self.vc)))

    def attend(self, row, pos, out):
        self.gpu.check(self.gpu.L.inkq_glue_qkv_attention_quant(self.gpu.h, P(row), *self._tables(pos), self.nq, self.nkv, self.max_pos, EPS, SCALE,
                                                                P(self.kc), P(self.vc), out.h, self.pkg.Q8_1_F16))

    def project_and_attend(self, w, a_in, row, pos, out):
        return self.gpu.L.inkq_glue_decode_qkv_attention(self.gpu.h, w.h, a_in.h, P(row), *self._tables(pos), self.nq, self.nkv, self.max_pos, EPS, SCALE,
                                                         P(self.kc), P(self.vc), out.h, self.pkg.Q8_1_F16)

    def result(self, n):
        self.gpu.synchronize()
        return [self.kc.clone(), self.vc.clone()], [x for o in self.outs[:n] for x in o.export(1)]


def equal(torch, a, b):
    return all(torch.equal(x, y) for x, y in zip(a[0], b[0])) and all(np.array_equal(x, y) for x, y in zip(a[1], b[1]))


@pytest.mark.parametrize("nq,nkv", [(8, 2), (32, 8)])
@pytest.mark.parametrize("pos", [0, 37, 450])
def test_attention_directly_behind_the_cache_append(pkg, gpu, nq, nkv, pos):
    a = Attention(pkg, gpu, nq, nkv, 512, 3)
    T = 48
    qkv = a.randn(T + 1, a.width)
    a.reset()
    a.append(qkv[:T], pos)
    gpu.synchronize()
    a.attend(qkv[T:], pos + T, a.outs[0])
    want = a.result(1)
    assert not a.torch.equal(a.kc[:, pos:pos + T + 1], a.kc0[:, pos:pos + T + 1])
    for _ in range(20):
        a.reset()
        a.append(qkv[:T], pos)
        a.attend(qkv[T:], pos + T, a.outs[0])
        assert equal(a.torch, a.result(1), want)


@pytest.mark.parametrize("nq,nkv", [(8, 2), (8, 8), (32, 8)])
@pytest.mark.parametrize("pos", [0, 100, 640])    # 640: more than one pass of 128 keys per share
def test_attention_calls_in_a_row_for_consecutive_positions(pkg, gpu, nq, nkv, pos):
    """Several tokens scored or verified from one product's [16][...] output: call t + 1 reads the row that call t appends."""
    a = Attention(pkg, gpu, nq, nkv, 1024, 4)
    n = 16
    qkv = a.randn(n, a.width)
    runs = []
    for wait in (True,) + (False,) * 20:
        a.reset()
        for t in range(n):
            a.attend(qkv[t:], pos + t, a.outs[t])
            if wait:
                gpu.synchronize()
        runs.append(a.result(n))
    assert all(equal(a.torch, r, runs[0]) for r in runs[1:])


@pytest.mark.parametrize("nq,nkv", [(8, 2), (32, 8)])
@pytest.mark.parametrize("pos", [0, 2, 130, 640])
def test_projection_and_attention_in_one_call_equal_the_two(pkg, gpu, nq, nkv, pos):
    """Tokens one behind the other without a synchronisation, the appended rows read by the next call; the first call stands
    directly behind the kernel that appends its predecessors' rows."""
    a = Attention(pkg, gpu, nq, nkv, 1024, 5)
    n, K = 6, 1024
    w = pkg.synth.weights(a.width, K, 6)
    wh = gpu.weight(pkg.A81W41, pkg.SCALES_F16, w["nib"], w["d"], w["m"])
    rows, acts = a.torch.empty((n, a.width), device="cuda"), [gpu.act(1, K) for _ in range(n)]
    for h in acts:
        gpu.quantize(h, a.randn(1, K), 1, pkg.Q8_1_F16)
    before = a.randn(32, a.width)
    runs = []
    for one_call in (False,) + (True,) * 10:
        a.reset()
        rows.zero_()
        a.append(before, pos)
        for t in range(n):
            if one_call:
                gpu.check(a.project_and_attend(wh, acts[t], rows[t:], pos + 32 + t, a.outs[t]))
                continue
            gpu.check(gpu.L.inkq_glue_decode_gemv(gpu.h, wh.h, acts[t].h, P(rows[t:]), 0, None, EPS, None, pkg.Q8_1_F16, None))
            gpu.synchronize()
            a.attend(rows[t:], pos + 32 + t, a.outs[t])
            gpu.synchronize()
        caches, outs = a.result(n)
        runs.append((caches + [rows.clone()], outs))
    assert all(equal(a.torch, r, runs[0]) for r in runs[1:])


def test_projection_and_attention_refuses_what_the_two_calls_refuse(pkg, gpu):
    a = Attention(pkg, gpu, 8, 2, 64, 7)
    a.reset()
    row, K = a.randn(1, a.width), 256
    a_in, wrong = gpu.act(1, K), gpu.act(1, K)
    gpu.quantize(a_in, a.randn(1, K), 1, pkg.Q8_1_F16)
    layer = lambda rows, scheme: gpu.weight(scheme, pkg.SCALES_F16, *[pkg.synth.weights(rows, K, 8)[k] for k in ("nib", "d", "m")])
    good = layer(a.width, pkg.A81W41)
    launched = gpu.L.inkq_launch_count(gpu.h)
    for w, act, out in ((layer(a.width - 128, pkg.A81W41), a_in, a.outs[0]),     # not the layer of these heads
                        (layer(a.width, pkg.W41), a_in, a.outs[0]),              # weight-only
                        (good, a_in, wrong),                                     # a row of another length
                        (good, a_in, a_in)):
        if w is not good:
            launched = gpu.L.inkq_launch_count(gpu.h)    # (making the weights launches kernels)
        assert a.project_and_attend(w, act, row, 3, out) == pkg.ERR_INVALID
        assert gpu.L.inkq_launch_count(gpu.h) == launched
    gpu.check(a.project_and_attend(good, a_in, row, 3, a.outs[0]))
