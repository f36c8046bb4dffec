"""The passes of a training step that cover all layers in one launch (needs a GPU): the bits of the
single-layer kernels, at ragged shapes."""

from __future__ import annotations

import ctypes

import pytest

import tissuemc_b200 as tmc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _s():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _ptrs(ts):
    return (ctypes.c_void_p * len(ts))(*[t.data_ptr() for t in ts])


def _ints(v):
    return (ctypes.c_int32 * len(v))(*v)


@pytest.mark.parametrize("K,splits", [(64, 1), (192, 3), (4096, 8), (1280, 5)])
def test_weight_gradients_of_several_layers(K, splits):
    from tissuemc_b200 import surrogate as S

    g = torch.Generator(device="cuda").manual_seed(K)
    shapes = [(512, 64), (130, 70), (1, 8), (128, 512), (33, 129)]
    A = [torch.randn(m, K, device="cuda", generator=g).bfloat16() for m, _ in shapes]
    B = [torch.randn(n, K, device="cuda", generator=g).bfloat16() for _, n in shapes]
    D = [torch.full((m * n + 32,), -7.0, device="cuda") for m, n in shapes]
    S._call("tmc_b200_nn_weight_grads", _ptrs(A), _ptrs(B), _ptrs(D), _ints([m for m, _ in shapes]),
            _ints([n for _, n in shapes]), len(shapes), K, splits, _s())
    for a, b, d, (m, n) in zip(A, B, D, shapes, strict=True):
        ref, work = torch.empty(m, n, device="cuda"), torch.empty(splits * m * n, device="cuda")
        S._call("tmc_b200_nn_matmul_f32_splitk", S._p(a), S._p(b), S._p(ref), S._p(work), m, n, K, splits, _s())
        assert torch.equal(d[:m * n].view(m, n), ref) and bool((d[m * n:] == -7.0).all())
        exact = a.double() @ b.double().T
        assert ((ref.double() - exact).abs().max() / exact.abs().max()).item() < 2e-6
    assert tmc.lib().tmc_b200_nn_status(1) == 0
    with pytest.raises(tmc.ConfigError, match="splits"):
        S._call("tmc_b200_nn_weight_grads", _ptrs(A), _ptrs(B), _ptrs(D), _ints([1]), _ints([8]), 1, K, 9, _s())


@pytest.mark.parametrize("M", [1, 31, 128, 129, 700, 4096])
def test_bias_gradients_of_several_layers(M):
    from tissuemc_b200 import surrogate as S

    g = torch.Generator(device="cuda").manual_seed(M)
    cols = [512, 8, 24, 128]
    dZ = [torch.randn(M, n, device="cuda", generator=g).bfloat16() for n in cols]
    db = [torch.full((n + 8,), -7.0, device="cuda") for n in cols]
    S._call("tmc_b200_nn_colsum_multi", _ptrs(dZ), _ptrs(db), _ints(cols), len(cols), M, _s())
    for z, d, n in zip(dZ, db, cols, strict=True):
        ref, work = torch.empty(n, device="cuda"), torch.empty(tmc.lib().tmc_b200_nn_colsum_work(n), device="cuda")
        S._call("tmc_b200_nn_colsum", S._p(z), S._p(ref), M, n, S._p(work), _s())
        assert torch.equal(d[:n], ref) and bool((d[n:] == -7.0).all())


@pytest.mark.parametrize("M,T,ld,k", [(1, 1, 1, 1), (33, 66, 128, 64), (256, 128, 128, 13), (4096, 66, 128, 64)])
def test_loss_with_transposes(M, T, ld, k):
    from tissuemc_b200 import surrogate as S

    g = torch.Generator(device="cuda").manual_seed(M)
    pred, target = (torch.randn(M, c, device="cuda", generator=g) for c in (ld, T))
    X = torch.randn(M, k, device="cuda", generator=g).bfloat16()
    out = [torch.empty(M, ld, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    dZT, XT = torch.empty(ld, M, dtype=torch.bfloat16, device="cuda"), torch.empty(k, M, dtype=torch.bfloat16, device="cuda")
    loss = torch.zeros(2, device="cuda")
    S._call("tmc_b200_nn_mse_transposes", S._p(pred), S._p(target), S._p(out[0]), S._p(dZT), S._p(loss), M, T, ld,
            ctypes.c_float(0.01), S._p(X), S._p(XT), k, _s())
    S._call("tmc_b200_nn_mse", S._p(pred), S._p(target), S._p(out[1]), S._p(loss[1:]), M, T, ld, ctypes.c_float(0.01), _s())
    assert torch.equal(out[0], out[1]) and torch.equal(dZT, out[1].t()) and torch.equal(XT, X.t())
    ref = 0.01 * ((pred[:, :T].double() - target.double()) ** 2).sum().item()
    assert abs(loss[0].item() - ref) <= 1e-5 * ref + 1e-12  # float32 partial sums of at most 17 terms each, then of blocks
