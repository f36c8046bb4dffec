"""The epilogues of the tensor-core products (needs a GPU): every output of a layer's forward and
backward product against float64 at ragged shapes, where the staged pieces meet the matrix edges,
and with outputs that do not start on a 16-byte boundary (the element-wise path)."""

from __future__ import annotations

import ctypes
import math

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

GUARD = 64  # elements past the end of every output that must stay untouched


def _out(rows, cols, dtype, offset):
    buf = torch.full((offset + rows * cols + GUARD,), -7.0, dtype=dtype, device="cuda")
    return buf, buf[offset:offset + rows * cols].view(rows, cols)


def _untouched(buf, offset, n):
    return bool((buf[:offset] == -7.0).all()) and bool((buf[offset + n:] == -7.0).all())


@pytest.mark.parametrize("M,N,K,offset", [(1, 8, 64, 0), (33, 70, 64, 0), (100, 36, 128, 0), (128, 128, 64, 0),
                                          (257, 72, 192, 0), (264, 200, 64, 0), (64, 64, 64, 1), (130, 136, 64, 1)])
def test_every_output_of_a_layer(M, N, K, offset):
    from tissuemc_b200 import surrogate as S

    g = torch.Generator(device="cuda").manual_seed(M * 1000 + N + K)
    X = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    W = (torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    zb, Z = _out(M, N, torch.float32, offset)
    hb, H = _out(M, N, torch.bfloat16, offset)
    tb, HT = _out(N, M, torch.bfloat16, offset)
    S._call("tmc_b200_nn_linear", S._p(X), S._p(W), S._p(bias), S._p(Z), S._p(H), S._p(HT), M, N, K, 1, s)
    z = X.double() @ W.double().T + bias.double()
    assert ((Z.double() - z).abs().max() / z.abs().max()).item() < 2e-6  # float32 sums of exact products
    h = torch.nn.functional.gelu(z, approximate="tanh")
    # half a bf16 step of the value, and the SFU tanh's absolute error (2^-10.9) on x / 2
    assert bool(((H.double() - h).abs() <= 2.0 ** -8 * h.abs() + 3e-4 * z.abs() + 1e-6).all())
    assert torch.equal(HT, H.t())
    for buf in (zb, hb, tb):
        assert _untouched(buf, offset, M * N)

    # backward: dX = (G W) gelu'(Zprev), here with the shapes of the product above
    xb, dX = _out(M, N, torch.bfloat16, offset)
    db, dXT = _out(N, M, torch.bfloat16, offset)
    S._call("tmc_b200_nn_backward_data", S._p(X), S._p(W), S._p(Z), S._p(dX), S._p(dXT), M, N, K, s)
    acc = X.double() @ W.double().T
    zr = Z.double().requires_grad_()
    torch.nn.functional.gelu(zr, approximate="tanh").sum().backward()
    ref = acc * zr.grad
    # half a bf16 step; the tanh's error enters the derivative as e (1/2 + |x u'|) <= 6e-3 for |x| <= 5
    assert bool(((dX.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 6e-3 * acc.abs() + 1e-6).all())
    assert torch.equal(dXT, dX.t())
    for buf in (xb, db):
        assert _untouched(buf, offset, M * N)


@pytest.mark.parametrize("N,K,offset", [(72, 64, 0), (128, 512, 0), (200, 192, 0), (136, 64, 1), (37, 128, 0)])
def test_few_rows_equal_the_same_rows_of_many(N, K, offset):
    """A product of few tiles takes narrower ones: the same bits, and both sides of the rule write no more
    than their matrix. Many rows leave a ragged last tile in either width."""
    from tissuemc_b200 import surrogate as S

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    across = (N + 127) // 128
    last_narrow = sms // 2 // across * 128  # the most rows that still take narrow tiles
    g = torch.Generator(device="cuda").manual_seed(N + K)
    X = torch.randn(last_narrow + 133, K, device="cuda", generator=g).bfloat16()
    W = (torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    got = {}
    for M in (1, 129, last_narrow, last_narrow + 1, last_narrow + 133):
        bufs = [_out(M, N, torch.float32, offset), _out(M, N, torch.bfloat16, offset), _out(N, M, torch.bfloat16, offset),
                _out(M, N, torch.bfloat16, offset), _out(N, M, torch.bfloat16, offset)]
        (_, Z), (_, H), (_, HT), (_, dX), (_, dXT) = bufs
        S._call("tmc_b200_nn_linear", S._p(X), S._p(W), S._p(bias), S._p(Z), S._p(H), S._p(HT), M, N, K, 1, s)
        S._call("tmc_b200_nn_backward_data", S._p(X), S._p(W), S._p(Z), S._p(dX), S._p(dXT), M, N, K, s)
        for buf, _ in bufs:
            assert _untouched(buf, offset, M * N)
        got[M] = Z, H, HT.t(), dX, dXT.t()
    most = got[last_narrow + 133]
    for M, outs in got.items():
        for few, many in zip(outs, most):
            assert torch.equal(few, many[:M])
